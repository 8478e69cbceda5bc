"""The lazy neighbor-joining search where its own machinery can go wrong,
against the oracle, in both team forms (a cluster, the whole GPU): real-valued
and widely scaled matrices (the new row sums in 32-bit and 64-bit units and in
the sequential order), zeros, matrices on which bounds stay tight (additive and
nearly constant ones) or wander (negative, growing values), sizes around whole
CTAs' worth of rows, and more than one rebuild.  Joins, branch lengths and
statistics: equality, in a child process, so that the size thresholds apply."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CODE = """
import sys, numpy as np; sys.path.insert(0, 'tests'); import oracle_py as O
from additive import random_tree_metric
from mestrado_gb300 import Context
c = Context(10, 2)

def check(M):
    M = np.ascontiguousarray(M, np.float32)
    j, st = c.nj(M, stats=True)
    oj, ost = O.nj(M)
    for k in ('rebuilds', 'tie_steps', 'ambiguous_steps'):
        assert st[k] == ost[k], (k, st[k], ost[k])
    for f in ('i', 'j', 'node', 'n', 'd', 'q', 'ti', 'tj', 'len_i', 'len_j'):
        assert np.array_equal(np.array([x[f] for x in oj], j[f].dtype), j[f]), f

def sym(M):
    U = np.triu(M, 1)
    return U + U.T

rng = np.random.default_rng(5)
for n in (2, 3, 15, 16, 17, 33, 151, 152, 153, 305):
    check(sym(rng.integers(-40, 900, (n, n))))
n = 260
check(sym(rng.normal(size=(n, n))))                                     # sequential sums
check(sym(rng.integers(1, 1 << 20, (n, n)) * 2.0 ** -18))               # wide units
check(sym(rng.integers(1, 1 << 22, (n, n)) * 2.0 ** -60))
check(sym(rng.integers(1, 200, (n, n)) * 2.0 ** 90))
check(sym(np.exp(rng.normal(size=(n, n)) * 6)))                         # many magnitudes
check(sym(-rng.integers(0, 500, (n, n))))
check(sym(np.where(rng.random((n, n)) < 0.9, 0, rng.integers(0, 9, (n, n)))))
check(sym(1000 + rng.integers(0, 2, (n, n))))
check(random_tree_metric(410, 3)[0])
check(sym(np.arange(n * n).reshape(n, n) % 977))
check(sym(rng.integers(0, 100000, (700, 700)) / 8))                     # two rebuilds
print('ok')
"""

_FORMS = {
    "cluster": {"NWG_NJ_CTA_MAX_N": "0", "NWG_NJ_SMEM_MAX_N": "0", "NWG_NJ_CLUSTER_MAX_N": "100000"},
    "full_gpu": {"NWG_NJ_CTA_MAX_N": "0", "NWG_NJ_SMEM_MAX_N": "0", "NWG_NJ_CLUSTER_MAX_N": "0"},
}


@pytest.mark.parametrize("form", list(_FORMS))
def test_lazy_search_matches_oracle(form):
    r = subprocess.run([sys.executable, "-c", _CODE], cwd=ROOT, env=dict(os.environ, **_FORMS[form]),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr


def test_compaction_between_rebuilds_matches_oracle():
    # above 2,048 slots the matrix is compacted every eighth of them: three times before the first rebuild here
    code = _CODE[: _CODE.index("rng = ")] + "\nrng = np.random.default_rng(8)\nn = 2200\n" \
        "check(sym(rng.integers(1, 100000, (n, n)) / 8))\nprint('ok')\n"
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
