"""The progressive alignment's wave form at its edges, against the oracle:
rows around whole bands and around the bands that all warps hold, X shorter
than a front, unequal profiles, and the merges that take the 64-bit form (gap
models with open < extension, and products of the profiles' sequence counts
beyond the 32-bit differences).  Outputs are bytes: equality."""
import numpy as np
import pytest

import oracle_py as O
from mestrado_gb300 import Context

pytestmark = pytest.mark.gpu


def _rand(rng, lengths):
    letters = np.frombuffer(b"ARNDCQEGHILKMFPSTWYVBZX*", dtype=np.uint8)
    return [letters[rng.integers(0, 24, int(n))].tobytes() for n in lengths]


def _mutant(rng, s, p):
    letters = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", dtype=np.uint8)
    a = np.frombuffer(s, np.uint8).copy()
    hit = rng.random(len(a)) < p
    a[hit] = letters[rng.integers(0, 20, int(hit.sum()))]
    keep = rng.random(len(a)) >= p / 4
    keep[0] = True
    return a[keep].tobytes()


@pytest.mark.parametrize("lx", [1, 2, 8, 24, 25, 33, 131])
@pytest.mark.parametrize("ly", [1, 63, 64, 65, 127, 128, 129, 257])
def test_pair_shapes(ctx, lx, ly):
    seqs = _rand(np.random.default_rng(lx * 1000 + ly), [lx, ly])
    assert ctx.msa(seqs, [0], [1]) == O.msa(seqs, [0], [1])


@pytest.mark.parametrize("lx,ly", [(5, 1025), (40, 2050), (300, 1100), (60, 4500), (2100, 70)])
def test_more_rows_than_one_pass(ctx, lx, ly):
    rng = np.random.default_rng(lx + ly)
    y = _rand(rng, [ly])[0]
    seqs = [y[:lx] if lx <= ly else _rand(rng, [lx])[0], y]
    assert ctx.msa(seqs, [0], [1]) == O.msa(seqs, [0], [1])


@pytest.mark.parametrize("go,ge", [(10, 2), (11, 1), (0, 0), (3, 3), (2, 5), (40, 0)])
def test_profiles_and_gap_models(go, ge):
    rng = np.random.default_rng(go * 10 + ge)
    base = _rand(rng, [150, 90])
    seqs = [_mutant(rng, base[k % 2], 0.15) for k in range(13)]
    left, right = [0, 2, 4, 6, 8, 10, 13, 15, 17, 12, 19, 21], [1, 3, 5, 7, 9, 11, 14, 16, 18, 20, 22, 23]
    with Context(go, ge) as c:
        assert c.msa(seqs, left, right) == O.msa(seqs, left, right, go=go, ge=ge)


def test_counts_beyond_32_bit_differences():
    # 520 x 520 sequences at the root: 520 * 520 * (2 * 11 + 4 * 1000) > 2^30
    rng = np.random.default_rng(7)
    seqs = _rand(rng, rng.integers(3, 9, 1040))
    left, right, level, node = [], [], list(range(1040)), 1040
    while len(level) > 1:
        nxt = []
        for k in range(0, len(level) - 1, 2):
            left.append(level[k])
            right.append(level[k + 1])
            nxt.append(node)
            node += 1
        if len(level) % 2:
            nxt.append(level[-1])
        level = sorted(nxt)
    with Context(1000, 1) as c:
        assert c.msa(seqs, left, right) == O.msa(seqs, left, right, go=1000, ge=1)


def _balanced(n):
    left, right, level, node = [], [], list(range(n)), n
    while len(level) > 1:
        nxt = []
        for k in range(0, len(level) - 1, 2):
            left.append(level[k])
            right.append(level[k + 1])
            nxt.append(node)
            node += 1
        if len(level) % 2:
            nxt.append(level[-1])
        level = sorted(nxt)
    return left, right


@pytest.mark.parametrize("n", [26, 600])
def test_column_counts_past_a_byte(ctx, n):
    # 'W' scores 11: row scores pass 127 from 12 sequences on, X's counts pass 255 at the root of 600
    rng = np.random.default_rng(n)
    seqs = [b"W" * int(k) + s for k, s in zip(rng.integers(1, 4, n), _rand(rng, rng.integers(1, 7, n)))]
    left, right = _balanced(n)
    assert ctx.msa(seqs, left, right) == O.msa(seqs, left, right)


def test_row_scores_past_two_bytes(ctx):
    # one sequence against a growing profile: 2,978 'W's in a column still score within 16 bits, 2,979 do not
    n = 2985
    seqs = [b"W" if k % 7 else b"WA" for k in range(n)]
    left, right = [0], [1]
    for k in range(1, n - 1):
        left.append(k + 1)
        right.append(n + k - 1)
    assert ctx.msa(seqs, left, right) == O.msa(seqs, left, right)
