"""A call that fails between forking its launches to side streams and joining them
leaves nothing running: the next call on the context, with other inputs in the
same buffers, gives the oracle's results."""
import os

import numpy as np
import oracle_py as O
import pytest

from mestrado_gb300 import Context, NWGError, encode

pytestmark = pytest.mark.gpu
LETTERS = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", dtype=np.uint8)


def _seqs(seed, n):
    rng = np.random.default_rng(seed)
    return [LETTERS[rng.integers(0, 20, int(k))].tobytes() for k in rng.choice([30, 100, 120, 200, 250, 300, 420, 500], n)]


@pytest.mark.parametrize("seed", range(3))
def test_pair_list(monkeypatch, seed):
    with Context(10, 2) as c:
        for k, fails in ((seed, True), (seed + 50, False)):
            codes, off = encode(_seqs(k, 60))
            pi, pj = (np.random.default_rng(k).integers(0, 60, (2, 8000 if fails else 500))).astype(np.int32)
            if fails:
                monkeypatch.setenv("NWG_INJECT_FORK_ERROR", "1")
                with pytest.raises(NWGError):
                    c.score_pairs(codes, off, pi, pj)
                monkeypatch.delenv("NWG_INJECT_FORK_ERROR")
            else:
                assert np.array_equal(c.score_pairs(codes, off, pi, pj),
                                      O.score_list(codes, off, pi, pj, 10, 2, os.cpu_count()))


@pytest.mark.parametrize("seed", range(3))
def test_traceback(monkeypatch, seed):
    px, py = np.arange(0, 3000, 2, dtype=np.int32), np.arange(1, 3000, 2, dtype=np.int32)
    with Context(10, 2) as c:
        monkeypatch.setenv("NWG_INJECT_FORK_ERROR", "1")
        with pytest.raises(NWGError):
            c.align_pairs(*encode(_seqs(seed, 3000)), px, py)
        monkeypatch.delenv("NWG_INJECT_FORK_ERROR")
        seqs = _seqs(seed + 50, 3000)
        out = c.align_pairs(*encode(seqs), px, py)
        for k in range(0, 1500, 40):
            assert out[k] == O.traceback(seqs[px[k]], seqs[py[k]], 10, 2)
