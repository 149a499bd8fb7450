"""Two engines on two threads: launches of one kernel with different shared memory sizes side by side."""
import threading

import numpy as np
import pytest

import privacyamplification_gb300 as pa
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [pa.DEFAULT_FLAGS | pa.FLAG_EXACT, pa.DEFAULT_FLAGS])
def test_engines_of_different_sizes_side_by_side(pa_lib, flags):
    """Short and long transforms (exact path: one to seven top levels per pass; FP32 passes: tiles of 2 to 64 columns)."""
    sizes = [1 << 19, 1 << 23, 1 << 21, 1 << 25]
    failures = []

    def work(n):
        try:
            v = n // 4 + n // 8
            seed, recv = O.random_block(n, v, n)
            ks, kr = O.key_split(recv, n, v)
            with pa.Engine(max_sample_size=n) as eng:
                eng.set_seed(seed, n, -1)
                want = eng.process(ks, kr, n, v, flags)
                barrier.wait()
                for _ in range(300):
                    if not np.array_equal(eng.process(ks, kr, n, v, flags), want):
                        raise AssertionError("another result")
            if not np.array_equal(want, O.ntt(seed, ks, kr, n, v)):
                raise AssertionError("wrong result")
        except Exception as ex:  # reported by the main thread
            failures.append((n, repr(ex)))
            barrier.abort()

    barrier = threading.Barrier(len(sizes))
    threads = [threading.Thread(target=work, args=(n,)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
