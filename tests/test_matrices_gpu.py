"""Alignments and the progressive alignment under a caller's matrix: not symmetric,
and with scores at the ends of the signed bytes that the traceback's pipeline
holds with twice the extension added (and one past them).  Bytes: equality with
the oracle."""
import numpy as np
import oracle_py as O
import pytest

from mestrado_gb300 import Context, encode

pytestmark = pytest.mark.gpu
LETTERS = np.frombuffer(b"ARNDCQEGHILKMFPSTWYVBZX*", dtype=np.uint8)


@pytest.mark.parametrize("lo,hi,go,ge", [(-4, 11, 10, 2), (-128, 123, 10, 2), (-128, 124, 10, 2), (-128, 127, 0, 0),
                                         (1, 100, 9, 9), (-100, -1, 3, 1), (-60, 60, 2, 5)])
def test_matrix(monkeypatch, lo, hi, go, ge):
    rng = np.random.default_rng(hi - lo + go)
    sub = rng.integers(lo, hi + 1, 576).astype(np.int8)
    sub[:2] = lo, hi
    seqs = [LETTERS[rng.integers(0, 24, n)].tobytes() for n in (1, 30, 129, 200, 257, 300)]
    codes, off = encode(seqs)
    px, py = np.divmod(np.arange(36, dtype=np.int32), np.int32(6))
    monkeypatch.setattr(O, "blosum", lambda: sub)
    with Context(go, ge, sub=sub) as c:
        out = c.align_pairs(codes, off, px, py)
        for k in range(36):
            assert out[k] == O.traceback(seqs[px[k]], seqs[py[k]], go, ge), (px[k], py[k])
        assert c.msa(seqs, [0, 2, 4, 6, 8], [1, 3, 5, 7, 9]) == O.msa(seqs, [0, 2, 4, 6, 8], [1, 3, 5, 7, 9], go, ge, sub)
