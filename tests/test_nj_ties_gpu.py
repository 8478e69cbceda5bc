"""Neighbor joining where many pairs tie, exactly or within rounding, so that the
picks come from the candidate scan: its list, the lists that overflow, the counts
that stop early, rows split over warps and rows of one to four columns.  Joins,
lengths and statistics against the oracle, in each launch form: equality."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CODE = """
import sys; sys.path.insert(0, 'tests')
import numpy as np
from mestrado_gb300 import Context
from test_nj_range_gpu import _check, _sym
c = Context(10, 2)
for n in (5, 30, 66, 131, 160, 257, 420, 610):
    rng = np.random.default_rng(n)
    f = rng.integers(0, max(2, n // 12), n)
    b = rng.integers(100, 900, (n, n))
    b = np.triu(b) + np.triu(b, 1).T
    _check(c, _sym(np.where(f[:, None] == f[None, :], 0, b[f][:, f])))   # copies of sequences
    _check(c, _sym(1000 + rng.random((n, n))))                           # ties within rounding
    _check(c, _sym(rng.integers(1, 4, (n, n))))
    if n < 400:
        _check(c, _sym(np.full((n, n), 7)))
print('ok')
"""

_FORMS = {
    "one_cta": {"NWG_NJ_CTA_MAX_N": "160"},
    "cluster": {"NWG_NJ_CTA_MAX_N": "0", "NWG_NJ_CLUSTER_MAX_N": "100000"},
    "full_gpu": {"NWG_NJ_CTA_MAX_N": "0", "NWG_NJ_CLUSTER_MAX_N": "0"},
}


@pytest.mark.parametrize("form", list(_FORMS))
def test_ties_match_oracle(form):
    r = subprocess.run([sys.executable, "-c", _CODE], cwd=ROOT, env=dict(os.environ, **_FORMS[form]),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
