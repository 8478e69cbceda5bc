"""The traceback's pipeline form at its edges, against the oracle: rows around
whole bands of 128 and around the bands that one CTA, several CTAs and a whole
cluster hold, X shorter than the front, launches that give a pair one CTA
(passes over its bands, groups by band count) or several, gap models at and
past the form's limits, and the lengths at which the recurrence's sentinel
comes into play.  Strings and scores: equality."""
import numpy as np
import pytest

import oracle_py as O
from mestrado_gb300 import Context, encode

pytestmark = pytest.mark.gpu
LETTERS = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", dtype=np.uint8)


def _rand(rng, n):
    return LETTERS[rng.integers(0, 20, int(n))].tobytes()


def _mutant(rng, s, p=0.2):
    a = np.frombuffer(s, np.uint8).copy()
    hit = rng.random(len(a)) < p
    a[hit] = LETTERS[rng.integers(0, 20, int(hit.sum()))]
    keep = rng.random(len(a)) >= p / 4
    keep[0] = True
    return a[keep].tobytes()


def _check(c, seqs, px, py, go=10, ge=2, only=None):
    codes, off = encode(seqs)
    out = c.align_pairs(codes, off, px, py)
    for k in range(len(px)) if only is None else only:
        assert out[k] == O.traceback(seqs[px[k]], seqs[py[k]], go, ge), (k, len(seqs[px[k]]), len(seqs[py[k]]))


def test_every_edge_against_every_edge(ctx):
    rng = np.random.default_rng(1)
    base = _rand(rng, 520)
    lengths = [1, 2, 7, 8, 9, 31, 32, 33, 127, 128, 129, 255, 256, 257, 384, 385, 511, 513]
    seqs = [_rand(rng, n) if k % 2 else base[:n] for k, n in enumerate(lengths)]
    px, py = np.divmod(np.arange(len(seqs) ** 2), len(seqs))
    _check(ctx, seqs, px, py)


@pytest.mark.parametrize("lx,ly", [(3, 4200), (40, 4097), (700, 1030), (4200, 5), (1500, 1600)])
def test_one_pair_over_a_cluster(ctx, lx, ly):
    rng = np.random.default_rng(lx)
    y = _rand(rng, ly)
    x = _mutant(rng, y)[:lx] if lx <= ly else _mutant(rng, y) + _rand(rng, lx - ly)
    _check(ctx, [x, y], [0], [1])


@pytest.mark.parametrize("pairs", [130, 300, 800])
def test_many_pairs_in_groups_and_passes(ctx, pairs):
    # one to nine bands: two CTAs a pair (300), one (800: groups of one, two and more bands, three passes)
    rng = np.random.default_rng(pairs)
    seqs = []
    for k in range(pairs):
        y = _rand(rng, rng.choice([30, 100, 128, 200, 256, 300, 520, 1100]) if k else 1100)
        seqs += [_mutant(rng, y, 0.1 + 0.4 * rng.random()), y]
    px, py = np.arange(0, 2 * pairs, 2), np.arange(1, 2 * pairs, 2)
    _check(ctx, seqs, px, py, only=[0, *rng.integers(0, pairs, 120)])


@pytest.mark.parametrize("go,ge", [(0, 0), (2, 2), (11, 1), (4, 1), (58, 58), (120, 58), (58, 59), (2, 5), (300, 64)])
def test_gap_models(go, ge):
    rng = np.random.default_rng(go + ge)
    y = _rand(rng, 300)
    seqs = [y, _mutant(rng, y), _mutant(rng, y, 0.6), _rand(rng, 90), y[:140]]
    px, py = np.divmod(np.arange(25), 5)
    with Context(go, ge) as c:
        _check(c, seqs, px, py, go, ge)


@pytest.mark.parametrize("n", [3270, 3275, 3281])
def test_lengths_at_the_sentinel(n):
    # ge (n + 1) + go passes 32768 between the first two
    rng = np.random.default_rng(n)
    y = _rand(rng, n)
    seqs = [y, _mutant(rng, y)[:60], _rand(rng, 20)]
    with Context(20, 10) as c:
        _check(c, seqs, [0, 1, 0, 2], [1, 0, 2, 0], 20, 10)
