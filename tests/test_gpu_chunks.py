"""Blocks above 2^27 bits in 2^27-bit transforms: the FP32 residual is a single chunk's, and whole outputs over the shapes
of the chunk grid (one row, one column, more rows and columns than at v = 3n/8), with kept and own seeds."""
import numpy as np
import pytest

import privacyamplification_gb300 as pa
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DEFAULT = pa.DEFAULT_FLAGS


@pytest.fixture(scope="module")
def engine(pa_lib):
    with pa.Engine(max_sample_size=1 << 29) as eng:
        yield eng


def block(n, v, key):
    rng = np.random.default_rng(key)
    words = rng.integers(0, 1 << 32, n // 32 + 1, dtype=np.uint64).astype(np.uint32)
    return pa.key_split(words, n, v)


def seed_of(n, key):
    return np.random.default_rng(key).integers(0, 1 << 32, n // 32, dtype=np.uint64).astype(np.uint32)


def test_residual_is_that_of_one_chunk(engine):
    """A chunk is a block of 2^27 bits with h = v = 2^26.  The largest error over the 15 chunks of a 2^29-bit block exceeds
    one chunk's by the growth of a maximum only: sqrt(ln(15 2^26) / ln(2^26)) = 1.07 for normal errors; 1.25 allowed."""
    n, v = 1 << 27, 1 << 26
    engine.set_seed(seed_of(n, 1), n, -1)
    engine.process(*block(n, v, 2), n, v)
    assert engine.last_stats.exact == 0
    one = engine.last_stats.max_residual
    n, v = 1 << 29, (1 << 27) + (1 << 26)
    engine.set_seed(seed_of(n, 3), n, 1)
    engine.process(*block(n, v, 4), n, v)
    assert engine.last_stats.exact == 2
    print("residual: one chunk %.4f, 15 chunks %.4f" % (one, engine.last_stats.max_residual))
    assert engine.last_stats.max_residual <= 1.25 * one


# rows x columns of chunks
@pytest.mark.parametrize("n,v,flags,reuse", [
    (1 << 28, 320032, DEFAULT, 1),                             # 1 x 4
    (1 << 28, (1 << 28) - (1 << 20), DEFAULT, 1),              # 4 x 1
    (1 << 28, 1 << 26, pa.FLAG_XOR_KEY_REST, -1),              # 2 x 3, result longer than key_rest
    ((1 << 27) + 32, 1 << 26, DEFAULT, 1),                     # 1 x 2
    ((1 << 28) + (1 << 20) + 96, (1 << 27) + (1 << 26) + 64, DEFAULT, -1)])  # 3 x 2, ragged
def test_whole_output(engine, n, v, flags, reuse):
    seed = seed_of(n, n + v)
    oracle = O.NttSeed(seed, n, v)
    engine.set_seed(seed, n, reuse)
    for key in ((5, 6) if reuse < 0 else (5,)):
        ks, kr = block(n, v, key)
        out = engine.process(ks, kr, n, v, flags)
        assert engine.last_stats.exact == 2 and engine.last_stats.max_residual < 0.1
        assert np.array_equal(out, oracle.block(ks, kr, flags))
    oracle.close()


@pytest.mark.parametrize("v,flags", [((1 << 26) + 32, 0), (1 << 28, DEFAULT), (5 << 26, DEFAULT)])  # 4 x 7, 4 x 4, 5 x 3
def test_more_rows(engine, v, flags):
    """n = 2^29 with an own and with a kept seed, against the exact path; the exact block between two ordinary ones shares
    buffers with the chunks."""
    n = 1 << 29
    seed = seed_of(n, v)
    ks, kr = block(n, v, 7)
    engine.set_seed(seed, n, 1)
    own = engine.process(ks, kr, n, v, flags)
    assert engine.last_stats.exact == 2
    engine.set_seed(seed, n, -1)
    first = engine.process(ks, kr, n, v, flags)
    exact = engine.process(ks, kr, n, v, flags | pa.FLAG_EXACT)
    assert engine.last_stats.exact == 1
    again = engine.process(ks, kr, n, v, flags)
    assert engine.last_stats.exact == 2
    for out in (first, exact, again):
        assert np.array_equal(out, own)


def test_seed_kept_across_lengths(engine):
    """A kept seed's window spectra serve blocks of the same rows and columns only."""
    n = (1 << 28) + 4096
    seed = seed_of(n, 11)
    engine.set_seed(seed, n, -1)
    want = {}
    for v in (100663296, 33554432, 100663328, 100663296):
        ks, kr = block(n, v, v)
        out = engine.process(ks, kr, n, v)
        assert engine.last_stats.exact == 2
        if v not in want:
            want[v] = O.ntt(seed, ks, kr, n, v)
        assert np.array_equal(out, want[v]), v


def test_padded_block_between_one_pass_blocks(engine):
    """A seed of almost 2^27 bits whose block without compression needs chunks: its other blocks' spectrum is not the
    chunks' leftover."""
    n = (1 << 27) - 1024
    seed = seed_of(n, 12)
    engine.set_seed(seed, n, -1)
    for v, flags, path in ((1 << 26, DEFAULT, 0), (1 << 24, 0, 2), (1 << 26, DEFAULT, 0)):
        ks, kr = block(n, v, v + flags)
        out = engine.process(ks, kr, n, v, flags)
        assert engine.last_stats.exact == path
        assert np.array_equal(out, O.ntt(seed, ks, kr, n, v, flags)), (v, flags)


@pytest.mark.parametrize("room", [3.85, 4.4, 5.6])
def test_little_memory(pa_lib, room):
    """Engines beside a tenant that leaves `room` GB: fewer or no row passes held, the same result.  2^28 bits need 3.7 GB and
    take 7.4 where they can."""
    torch = pytest.importorskip("torch")
    n, v = 1 << 28, (1 << 26) + (1 << 25)
    seed = seed_of(n, 13)
    ks, kr = block(n, v, 14)
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - int(room * 1e9), dtype=torch.uint8, device="cuda")
    try:
        with pa.Engine(max_sample_size=n) as eng:
            left, _ = torch.cuda.mem_get_info()
            assert left < room * 1e9 - 3.6e9
            eng.set_seed(seed, n, -1)
            outs = [eng.process(ks, kr, n, v) for _ in range(2)]
            assert eng.last_stats.exact == 2
            print("room %.2f GB: %.2f ms a block" % (room, eng.last_stats.gpu_ms))
            exact = eng.process(ks, kr, n, v, DEFAULT | pa.FLAG_EXACT)
    finally:
        del hog
        torch.cuda.empty_cache()
    want = O.ntt(seed, ks, kr, n, v)
    for out in outs + [exact]:
        assert np.array_equal(out, want)
