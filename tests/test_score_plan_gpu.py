"""Plans of sets of uneven lengths: scores against the oracle (whole numbers:
equality), and the launches, of which a set that takes a few milliseconds has one
per length class at most and a set of a fraction of one chain a single one."""
import os

import numpy as np
import oracle_py as O
import pytest

from mestrado_gb300 import Context

pytestmark = pytest.mark.gpu
LETTERS = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", dtype=np.uint8)


@pytest.mark.parametrize("n,median,sigma,launches", [(400, 100, 0.9, 16), (150, 300, 0.6, 14), (16, 300, 0.5, 1)])
@pytest.mark.parametrize("go,ge", [(10, 2), (3, 5)])
def test_uneven_lengths(n, median, sigma, launches, go, ge):
    rng = np.random.default_rng(n)
    lengths = np.clip(np.exp(rng.normal(np.log(median), sigma, n)), 1, 3000).astype(int)
    seqs = [LETTERS[rng.integers(0, 20, k)].tobytes() for k in lengths]
    with Context(go, ge) as c:
        D, st = c.score_all(seqs, stats=True)
        assert np.array_equal(D, O.score_all(seqs, go, ge, threads=os.cpu_count()))
        if go >= ge:
            assert st["launches"] <= 2 + launches   # and the bounds' kernel, the re-run
