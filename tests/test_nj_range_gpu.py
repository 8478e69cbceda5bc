"""Neighbor joining on matrices that a float search does not hold or that have no
pair left to join.  Joins, lengths and statistics against the oracle: equality."""
import os
import subprocess
import sys

import numpy as np
import oracle_py as O
import pytest

from mestrado_gb300 import NWGError
from mestrado_gb300._native import NWG_ERR_CUDA

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _sym(M):
    U = np.triu(np.asarray(M, np.float32), 1)
    return np.ascontiguousarray(U + U.T)


def _check(ctx, D):
    j, st = ctx.nj(D, stats=True)
    oj, ost = O.nj(D)
    for k in ("rebuilds", "tie_steps", "ambiguous_steps"):
        assert st[k] == ost[k], k
    for f in ("i", "j", "node", "n", "d", "q", "ti", "tj", "len_i", "len_j"):
        assert np.array_equal(np.array([x[f] for x in oj], j[f].dtype), j[f], equal_nan=True), f


@pytest.mark.parametrize("n,undefined", [(9, 4), (130, 40), (300, 150), (700, 400), (2200, 900)])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_no_pair_left_to_join(ctx, n, undefined, value):
    # the defined taxa join, then no pair has a value: a status, with row sums and
    # compactions of the rest of the job already queued behind the failed pick
    rng = np.random.default_rng(n)
    D = _sym(rng.integers(1, 500, (n, n)))
    D[:undefined, :undefined] = value
    with pytest.raises(NWGError) as e:
        ctx.nj(D)
    assert e.value.status == NWG_ERR_CUDA
    _check(ctx, _sym(rng.integers(1, 500, (640, 640))))


def _overflowing(n, top, seed):
    """Row sums, or q, beyond float, T and q well inside double; sums of two distances inside float."""
    return _sym(np.random.default_rng(seed).integers(1, 1000, (n, n)) * np.float32(top / 1000))


@pytest.mark.parametrize("form", ["default", "cluster", "full_gpu"])
def test_beyond_the_float_search(form):
    code = """
import sys; sys.path.insert(0, 'tests')
import numpy as np, oracle_py as O, pytest
from mestrado_gb300 import Context
from test_nj_range_gpu import _check, _overflowing, _sym
c = Context(10, 2)
for n in (40, 139, 170, 290, 650):
    _check(c, _overflowing(n, 2.0 ** 126, n))            # T and q overflow floats throughout
    _check(c, _overflowing(n, 2.0 ** 116, n))
    _check(c, _overflowing(n, 2.0 ** 112, n))            # exact at first, held by floats once few taxa are left
D = _overflowing(230, 2.0 ** 40, 5)
D[7, 200] = D[200, 7] = 2.0 ** 126                       # one far distance
_check(c, D)
D = _sym(np.random.default_rng(6).integers(1, 900, (210, 210)))
D[5, 5] = np.inf                                         # a row sum is infinite, no distance is
_check(c, D)
rng = np.random.default_rng(7)
for e in (112.2, 112.4, 112.55, 112.7):                  # the largest distance grows past the floats' range on the way
    _check(c, _sym(rng.integers(-1000, 1000, (170, 170)) * np.float32(2.0 ** e / 1000)))
print('ok')
"""
    env = dict(os.environ)
    if form != "default":
        env.update(NWG_NJ_CTA_MAX_N="0", NWG_NJ_CLUSTER_MAX_N="100000" if form == "cluster" else "0")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr


def test_real_valued_distances_cost_what_whole_ones_do(ctx):
    # sums of one join's values in their own units: a sequential sum per join took nine times as long
    rng = np.random.default_rng(2)
    whole, real = _sym(rng.integers(1, 1000, (1200, 1200))), _sym(rng.random((1200, 1200)) * 100)
    for D in (whole, real):
        ctx.nj(D)
    ms = [min(ctx.nj(D, stats=True)[1]["device_ms"] for _ in range(3)) for D in (whole, real)]
    assert ms[1] < 4 * ms[0]
    p = np.sort(rng.random(700)) * 1000
    _check(ctx, _sym(np.abs(p[:, None] - p[None, :])))
    _check(ctx, _sym(rng.random((700, 700)) * 100))
    _check(ctx, _sym(rng.random((330, 330)) * 100))
