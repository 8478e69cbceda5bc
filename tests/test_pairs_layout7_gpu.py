"""The pair list on the recurrence with the extension cost taken out, against the
oracle: rows around whole bands of 128, 256 and 384 rows and columns around the
staged blocks of 32; gap models at which the profile's bytes are lifted (small
ge), at which they end (2 ge + 11 = 127 and above: the other recurrence) and at
which the borders reach the reference's sentinel.  Whole numbers: equality."""
import os

import numpy as np
import oracle_py as O
import pytest

from mestrado_gb300 import Context, encode

pytestmark = pytest.mark.gpu
LETTERS = np.frombuffer(b"ARNDCQEGHILKMFPSTWYVBZX*", dtype=np.uint8)


def _check(lengths, go, ge, seed=0, k=24):
    rng = np.random.default_rng(seed)
    codes, off = encode([LETTERS[rng.integers(0, k, n)].tobytes() for n in lengths])
    pi, pj = np.divmod(np.arange(len(lengths) ** 2, dtype=np.int32), np.int32(len(lengths)))
    with Context(go, ge) as c:
        out = c.score_pairs(codes, off, pi, pj)
    assert np.array_equal(out, O.score_list(codes, off, pi, pj, go, ge, os.cpu_count()))


def test_band_and_block_edges():
    _check([1, 2, 30, 31, 32, 33, 62, 63, 64, 65, 95, 96, 97, 127, 128, 129, 255, 256, 257, 383, 384, 385, 511, 512,
            513, 767, 768, 769, 1025], 10, 2)


@pytest.mark.parametrize("go,ge", [(0, 0), (9, 0), (11, 1), (10, 2), (7, 7), (1000, 2), (60, 58), (60, 59), (6, 7)])
def test_gap_models(go, ge):
    _check([1, 40, 129, 256, 300, 385, 700], go, ge, go + ge, 20)


def test_borders_at_the_sentinel():
    _check([1500, 1599, 1620, 1700, 40, 300], 700, 20, 3, 20)   # 20 * 1600 + 700 = 32,700
    _check([1500, 1590, 40, 300], 700, 20, 3, 20)
