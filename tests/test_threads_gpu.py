"""Contexts of their own on two host threads at once, one with large problems and
one with small ones of the same call: results as from one thread."""
import threading
import time

import numpy as np
import pytest

from mestrado_gb300 import Context, encode

pytestmark = pytest.mark.gpu
LETTERS = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", dtype=np.uint8)


def _nj(n):
    U = np.triu(np.random.default_rng(n).integers(1, 1000, (n, n)), 1).astype(np.float32)
    D = np.ascontiguousarray(U + U.T)
    return lambda c: c.nj(D).tobytes()


def _align(columns, pairs):
    rng = np.random.default_rng(columns)
    seqs = [LETTERS[rng.integers(0, 20, columns if k % 2 == 0 else 60)].tobytes() for k in range(2 * pairs)]
    codes, off = encode(seqs)
    px, py = np.arange(0, 2 * pairs, 2, dtype=np.int32), np.arange(1, 2 * pairs, 2, dtype=np.int32)
    return lambda c: c.align_pairs(codes, off, px, py)


@pytest.mark.parametrize("large,small", [(_nj(3000), _nj(610)), (_nj(590), _nj(150)), (_align(42000, 2), _align(50, 2)),
                                         (_align(5000, 40), _nj(140))],
                         ids=["nj", "nj_cluster", "align", "align_and_nj"])
def test_two_contexts_on_two_threads(large, small):
    with Context(10, 2) as c:
        want = [large(c), small(c)]
    end, errors = time.monotonic() + 1.5, []

    def loop(fn, ref):
        try:
            with Context(10, 2) as c:
                while not errors and time.monotonic() < end:
                    assert fn(c) == ref
        except BaseException as e:   # noqa: BLE001 -- the other thread stops, the test fails
            errors.append(e)

    threads = [threading.Thread(target=loop, args=a) for a in zip((large, small), want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
