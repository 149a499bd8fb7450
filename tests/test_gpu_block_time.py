"""The device time of a block (pa_stats.gpu_ms) runs from its first kernel's start to its last one's end."""
import numpy as np
import pytest

import privacyamplification_gb300 as pa
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_short_block_time_has_the_seed_count(gpu_engine):
    """The first short block of a seed counts its ones (2^21 bits by eight CTAs, some microseconds): its time is the longer
    one, and the second block's is not cut short by the first's."""
    n, v = 1 << 21, 32
    seed, recv = O.random_block(n, v, 9)
    ks, kr = O.key_split(recv, n, v)
    first, second = [], []
    for _ in range(40):
        gpu_engine.set_seed(seed, n, 2)
        for times in (first, second):
            gpu_engine.process(ks, kr, n, v)
            times.append(gpu_engine.last_stats.gpu_ms)
    assert min(first + second) > 0
    assert np.median(first) > np.median(second) + 0.5e-3, (np.median(first), np.median(second))


@pytest.mark.parametrize("n,v,flags", [(4096, 1536, pa.DEFAULT_FLAGS), (1 << 17, 49152, pa.DEFAULT_FLAGS),
                                       (1 << 18, 98304, pa.DEFAULT_FLAGS), (1 << 18, 98304, pa.DEFAULT_FLAGS | pa.FLAG_EXACT),
                                       (1 << 20, 393216, pa.DEFAULT_FLAGS | pa.FLAG_EXACT), (1 << 22, 1572864, pa.DEFAULT_FLAGS)])
def test_block_time_is_within_the_call(gpu_engine, n, v, flags):
    """Blocks of every path in turn with shorter and longer ones before them: above zero, below the call's own time."""
    import time
    seed, recv = O.random_block(n, v, 3)
    ks, kr = O.key_split(recv, n, v)
    gpu_engine.set_seed(seed, n, -1)
    for _ in range(30):
        t = time.perf_counter()
        gpu_engine.process(ks, kr, n, v, flags)
        wall = (time.perf_counter() - t) * 1e3
        assert 0 < gpu_engine.last_stats.gpu_ms < wall
