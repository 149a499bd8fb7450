"""Blocks with one result whose integer value is far from its mean (a key that agrees or disagrees with the seed over
many taps).  The value's parity is taken in FP32 arithmetic, and from 2^23 in magnitude on FP32 holds whole numbers only:
a value cannot show its own error, so the block has to be computed again on the exact path.  In a block of 32 results no
other result shares the last butterfly with the large one and betrays the error.  Outputs against the oracle on both
sides of zero and of 2^22, 2^23 and 2^24."""
import numpy as np
import pytest

import privacyamplification_gb300 as pa
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LIMIT = 1 << 23  # FP32 holds whole numbers only from here on


def unpack(words, count):
    return np.unpackbits(words.astype(">u4").view(np.uint8), count=count)


def pack(bits):
    return np.packbits(bits).view(">u4").astype(np.uint32)


def key_for(where, seed_bits, n, h, target):
    """Key bits 0 .. h with (h + 1) // 2 ones, for which the result with seed bits one and zero at the taps `where` is
    `target` plus the even number that the passes remove with the mean (twice the floor of half of it)."""
    ones = (h + 1) // 2
    mean = ones * int(seed_bits.sum()) / n
    hits = target + 2 * int(mean // 2)
    assert 0 <= hits <= where[0].size and ones - hits <= where[1].size
    key = np.zeros(n, np.uint8)
    key[where[0][:hits]] = 1
    key[where[1][:ones - hits]] = 1
    return key


@pytest.mark.parametrize("logn,v", [(26, 32), (26, 1 << 23), (27, 32)])
def test_parity_of_large_values(gpu_engine, logn, v):
    n = 1 << logn
    rng = np.random.default_rng(logn + v)
    edges = [LIMIT >> 1, LIMIT] + ([2 * LIMIT] if logn == 27 else [])
    targets = [s * (e + d) for e in edges for d in (-1, 3) for s in (-1, 1)]
    targets += [-12000001, -10000003, -9000001, -8500003] if v == 32 else [-12000001]
    seed, recv = O.random_block(n, v, logn)
    _, kr = O.key_split(recv, n, v)
    seed_bits = unpack(seed, n)
    at = v // 2
    taps = seed_bits[(at - np.arange(n - v + 1)) % n]
    where = rng.permutation(np.flatnonzero(taps)), rng.permutation(np.flatnonzero(taps == 0))
    oracle = O.NttSeed(seed, n, v) if v > 32 else None
    gpu_engine.set_seed(seed, n, -1)
    for target in targets:
        ks = pack(key_for(where, seed_bits, n, n - v, target))
        out = gpu_engine.process(ks, kr, n, v)
        st = gpu_engine.last_stats
        want = oracle.block(ks, kr) if oracle else O.direct(seed, ks, kr, n, v)
        assert np.array_equal(out, want), (target, st.exact, st.max_residual)
        if abs(target) > LIMIT:  # between 2^22 and 2^23 the rounding error decides
            assert st.exact == 1, (target, st.max_residual)
