"""The exact path's long transforms, 2^21 to 2^27 points (2^26 to 2^30 bits): whole outputs against the exact CPU oracle
up to 2^28 bits, above against the FP32 chunks, which share nothing with it."""
import numpy as np
import pytest

import privacyamplification_gb300 as pa
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DEFAULT = pa.DEFAULT_FLAGS


def inputs(n, v):
    rng = np.random.default_rng(n + v)
    words = lambda k: rng.integers(0, 1 << 32, k, dtype=np.uint64).astype(np.uint32)
    return (words(n // 32), *pa.key_split(words(n // 32 + 1), n, v))


# points: 2^21 (just below), 2^22, 2^22, 2^23, 2^24, 2^24 (ragged), 2^25 (result not compressed)
@pytest.mark.parametrize("n,v,flags", [
    ((1 << 25) - 32, 12582912, DEFAULT), ((1 << 25) + 32, 12582944, DEFAULT), (1 << 26, 25165824, DEFAULT),
    (1 << 27, 50331648, DEFAULT), (1 << 28, 100663296, DEFAULT), ((1 << 27) + 1056, 1 << 26, pa.FLAG_COMPRESS),
    (1 << 28, 1 << 25, pa.FLAG_XOR_KEY_REST)])
def test_whole_output(pa_lib, n, v, flags):
    seed, ks, kr = inputs(n, v)
    with pa.Engine(max_sample_size=n) as eng:
        eng.set_seed(seed, n, -1)
        out = eng.process(ks, kr, n, v, flags | pa.FLAG_EXACT)
        assert eng.last_stats.exact == 1
    assert np.array_equal(out, O.ntt(seed, ks, kr, n, v, flags))


# points: 2^25, 2^26, 2^26 (not compressed), 2^27
@pytest.mark.parametrize("n,v,flags", [
    (1 << 29, 201326592, DEFAULT), (1 << 30, 402653184, DEFAULT), (1 << 29, 1 << 27, 0), (1 << 30, 1 << 26, 0)])
def test_against_the_chunks(pa_lib, n, v, flags):
    seed, ks, kr = inputs(n, v)
    with pa.Engine(max_sample_size=n) as eng:
        eng.set_seed(seed, n, -1)
        exact = eng.process(ks, kr, n, v, flags | pa.FLAG_EXACT)
        assert eng.last_stats.exact == 1
        chunks = eng.process(ks, kr, n, v, flags)
        assert eng.last_stats.exact == 2
    assert np.array_equal(exact, chunks)
