"""Neighbor joining on matrices that a float search does not hold or that have no
pair left to join.  Joins, lengths and statistics against the oracle: equality."""
import numpy as np
import oracle_py as O
import pytest

from mestrado_gb300 import NWGError
from mestrado_gb300._native import NWG_ERR_CUDA

pytestmark = pytest.mark.gpu


def _sym(M):
    U = np.triu(np.asarray(M, np.float32), 1)
    return np.ascontiguousarray(U + U.T)


def _check(ctx, D):
    j, st = ctx.nj(D, stats=True)
    oj, ost = O.nj(D)
    for k in ("rebuilds", "tie_steps", "ambiguous_steps"):
        assert st[k] == ost[k], k
    for f in ("i", "j", "node", "n", "d", "q", "ti", "tj", "len_i", "len_j"):
        assert np.array_equal(np.array([x[f] for x in oj], j[f].dtype), j[f]), f


@pytest.mark.parametrize("n,undefined", [(300, 150), (700, 400), (2200, 900)])
def test_no_pair_left_to_join(ctx, n, undefined):
    # the defined taxa join, then no pair has a value: a status, with row sums and
    # compactions of the rest of the job already queued behind the failed pick
    rng = np.random.default_rng(n)
    D = _sym(rng.integers(1, 500, (n, n)))
    D[:undefined, :undefined] = np.nan
    with pytest.raises(NWGError) as e:
        ctx.nj(D)
    assert e.value.status == NWG_ERR_CUDA
    _check(ctx, _sym(rng.integers(1, 500, (640, 640))))
