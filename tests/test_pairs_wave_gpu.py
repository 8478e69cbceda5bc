"""The pair list's wavefront kernels at their edges, against the oracle: rows
around whole bands of both kinds (128 and 256 rows), X shorter than the front,
an odd number of pairs of very unequal X in one word, pairs past the 16-bit
limits (32-bit lanes), gap models, and matrices whose scores need more than
seven bits or are not symmetric.  Scores are whole numbers: equality."""
import os

import numpy as np
import pytest

import oracle_py as O
from mestrado_gb300 import Context, encode

pytestmark = pytest.mark.gpu


def _set(seed, lengths):
    rng = np.random.default_rng(seed)
    letters = np.frombuffer(b"ARNDCQEGHILKMFPSTWYVBZX*", dtype=np.uint8)
    return encode([letters[rng.integers(0, 24, int(n))].tobytes() for n in lengths])


def _check(c, codes, off, pi, pj, go=10, ge=2, sub=None):
    pi, pj = np.asarray(pi, np.int32), np.asarray(pj, np.int32)
    out = c.score_pairs(codes, off, pi, pj)
    assert np.array_equal(out, O.score_list(codes, off, pi, pj, go, ge, os.cpu_count(), sub=sub))


def test_every_edge_against_every_edge(ctx):
    lengths = [1, 2, 7, 8, 9, 31, 32, 33, 63, 127, 128, 129, 200, 255, 256, 257, 300, 511, 513]
    codes, off = _set(1, lengths)
    pi, pj = np.divmod(np.arange(len(lengths) ** 2), len(lengths))
    _check(ctx, codes, off, pi, pj)


@pytest.mark.parametrize("pairs", [[(0, 0)], [(0, 1)], [(1, 0), (0, 0), (2, 1)], [(3, 2)] * 5])
def test_few_pairs(ctx, pairs):
    codes, off = _set(2, [3, 700, 40, 129])
    _check(ctx, codes, off, [p[0] for p in pairs], [p[1] for p in pairs])


def test_16_and_32_bit_pairs_in_one_list(ctx):
    codes, off = _set(3, [2900, 2976, 2977, 3100, 6900, 6901, 7300, 100, 130])
    pi, pj = np.divmod(np.arange(81), 9)
    _check(ctx, codes, off, pi, pj)


def test_identical_sequences_reach_the_16_bit_ceiling(ctx):
    w = b"W" * 2976   # 11 a residue: the highest score that int16 lanes may hold
    codes, off = encode([w, w, w + b"W" * 40, b"W" * 2000])
    pi, pj = np.divmod(np.arange(16), 4)
    _check(ctx, codes, off, pi, pj)


@pytest.mark.parametrize("go,ge", [(0, 0), (2, 5), (11, 1), (60, 3), (900, 400)])
def test_gap_models(go, ge):
    codes, off = _set(go + ge, [1, 40, 128, 150, 256, 390, 600])
    pi, pj = np.divmod(np.arange(49), 7)
    with Context(go, ge) as c:
        _check(c, codes, off, pi, pj, go, ge)


@pytest.mark.parametrize("lo,hi", [(-4, 11), (-60, 67), (-60, 68), (-127, 127), (1, 127), (-100, -1)])
def test_matrices(lo, hi):
    rng = np.random.default_rng(hi - lo)
    sub = rng.integers(lo, hi + 1, 576).astype(np.int8)   # not symmetric
    sub[:2] = lo, hi
    codes, off = _set(abs(hi), [1, 30, 129, 257, 400])
    pi, pj = np.divmod(np.arange(25), 5)
    with Context(10, 2, sub=sub) as c:
        _check(c, codes, off, pi, pj, sub=sub)


def test_empty_list(ctx):
    codes, off = _set(5, [10, 20])
    assert len(ctx.score_pairs(codes, off, [], [])) == 0
