"""The progressive alignment without the memory for its cell scores: the merges
that find none take the 64-bit form, which needs none, instead of failing the
call.  Rows are bytes: equality with the oracle."""
import numpy as np
import oracle_py as O
import pytest

from mestrado_gb300 import Context

pytestmark = pytest.mark.gpu
LETTERS = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", dtype=np.uint8)


@pytest.mark.parametrize("room", [0, 40000, 200000, 10**9])   # cell scores that fit
@pytest.mark.parametrize("go,ge", [(10, 2), (2, 5)])
def test_no_memory_for_the_scores(monkeypatch, room, go, ge):
    rng = np.random.default_rng(11)
    seqs = [LETTERS[rng.integers(0, 20, int(n))].tobytes() for n in rng.integers(20, 400, 9)]
    left, right = [0, 2, 4, 9, 6, 11, 8, 13], [1, 3, 5, 10, 7, 12, 14, 15]
    with Context(go, ge) as c:
        monkeypatch.setenv("NWG_MSA_INJECT_SCORE_OOM", str(room))
        assert c.msa(seqs, left, right) == O.msa(seqs, left, right, go=go, ge=ge)
        monkeypatch.delenv("NWG_MSA_INJECT_SCORE_OOM")
        assert c.msa(seqs, left, right) == O.msa(seqs, left, right, go=go, ge=ge)
