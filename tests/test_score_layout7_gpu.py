"""Layout 7 of the scoring kernel (the recurrence with the extension cost taken
out) where its own parts can go wrong, against the oracle: every rows-per-lane
template and front width; column counts around the staged blocks of 32 columns
and the ramps; bands that end in or before the second Y of a pair; gap models
down to go = ge and beyond its range (go < ge); scores at the top of the 16-bit
range; lengths where the 16-bit or the border's range ends; sets too small to
fill the GPU, which take other templates; the job search over many groups; and
sets with sequences beyond the 16-bit lanes' length, whose lanes move their
values down as they grow (columns and bands around the steps of the move, the
steepest growth, growth of only one of two Y in a word).
Scores are whole numbers: equality."""
import os

import numpy as np
import oracle_py as O
import pytest

from mestrado_gb300 import MODE_BATCHED, MODE_BATCHED_INT32, Context

pytestmark = pytest.mark.gpu
LETTERS = np.frombuffer(b"ARNDCQEGHILKMFPSTWYVBZX*", dtype=np.uint8)


def _seqs(rng, lengths, k=24):
    return [LETTERS[rng.integers(0, k, int(n))].tobytes() for n in lengths]


def _check(seqs, go=10, ge=2, tuning=None, modes=(MODE_BATCHED, MODE_BATCHED_INT32)):
    ref = O.score_all(seqs, go, ge, threads=os.cpu_count())
    with Context(go, ge) as c:
        if tuning:
            c.set_tuning(*tuning)
        for mode in modes:
            assert np.array_equal(c.score_all(seqs, mode=mode), ref), mode


@pytest.mark.parametrize("W", [32, 16, 8, 1])
@pytest.mark.parametrize("R", [4, 8, 12, 16, 18, 20, 22, 24, 26, 28, 30, 32])
def test_templates_at_column_and_row_edges(R, W):
    if W == 1 and (R % 4 or R == 28):
        pytest.skip("one pair per thread: multiples of 4")
    rng = np.random.default_rng(R * 100 + W)
    edges = {1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 39, 40, 47, 48, 63, 64, 65, 95, 96, 97}
    band = R * W
    edges |= {band - 1, band, band + 1, 2 * band + 1} if band <= 512 else {band}
    _check(_seqs(rng, sorted(edges)), tuning=(R, 7, W))


@pytest.mark.parametrize("go,ge", [(10, 2), (11, 1), (0, 0), (5, 5), (1000, 0), (40, 30), (3, 5), (1000, 1000)])
def test_gap_models(go, ge):
    rng = np.random.default_rng(go + ge)
    _check(_seqs(rng, rng.integers(1, 400, 24)), go, ge, tuning=(20, 7, 16))
    _check(_seqs(rng, rng.integers(1, 700, 12)), go, ge)


@pytest.mark.parametrize("go,ge", [(10, 2), (12, 3), (30, 10), (11, 1)])
def test_range_of_the_halves(go, ge):
    # identical runs of the best entry: H and H~ at their largest, beside poor pairs
    rng = np.random.default_rng(ge)
    seqs = [b"W" * 2970, b"W" * 2960, b"W" * 40 + b"P" * 2900, b"P" * 2950] + _seqs(rng, [2800, 33, 1])
    _check(seqs, go, ge, modes=(MODE_BATCHED,))


@pytest.mark.parametrize("go,ge,n", [(12, 3, 5390), (12, 3, 5440), (10, 2, 6899), (11, 1, 7400), (10, 4, 8200)])
def test_lengths_at_the_ends_of_the_ranges(go, ge, n):
    rng = np.random.default_rng(n)
    a = LETTERS[rng.integers(0, 20, n)]
    b = a.copy()
    b[::3] = LETTERS[rng.integers(0, 20, len(b[::3]))]
    _check([a.tobytes(), b[:-60].tobytes(), b"W" * 30] + _seqs(rng, [500]), go, ge, modes=(MODE_BATCHED,))


@pytest.mark.parametrize("n", [1, 2, 3, 33, 34, 260])
def test_small_sets_and_many_groups(n):
    rng = np.random.default_rng(n)
    _check(_seqs(rng, rng.integers(1, 330 if n > 2 else 1500, n), 20))


@pytest.mark.parametrize("go,ge", [(10, 2), (11, 1), (0, 0), (12, 3)])
def test_sets_with_very_long_sequences(go, ge):
    rng = np.random.default_rng(go)
    long = LETTERS[rng.integers(0, 20, 9100)]
    near = long[40:8300].copy()
    near[::4] = LETTERS[rng.integers(0, 20, len(near[::4]))]
    seqs = [b"W" * 7168, b"W" * 7137, b"P" * 7169, long.tobytes(), near.tobytes(), b"W" * 2100 + b"P" * 5000,
            b"W" * 3100, LETTERS[rng.integers(0, 20, 1025)].tobytes()] + _seqs(rng, rng.integers(1, 300, 48), 20)
    ref = O.score_all(seqs, go, ge, threads=os.cpu_count())
    with Context(go, ge) as c:
        D, st = c.score_all(seqs, mode=MODE_BATCHED, stats=True)
        assert np.array_equal(D, ref)
        assert st["pairs_int16"] == len(seqs) * (len(seqs) + 1) // 2   # enough work: no int32 lanes
        # columns short and long against long rows, as a block
        xs = seqs[:4] + seqs[30:]
        assert np.array_equal(c.score_block(xs * 40, seqs[:8])[: len(xs)], ref[np.r_[0:4, 30:len(seqs)]][:, :8])
