"""The exact path (PA_FLAG_EXACT) at the edges of its forms, whole outputs against the exact CPU oracle: the
word-by-word product of short blocks (one and eight result words per CTA, a partial last word, the key's last bit
in a word of its own), its boundary at 2^34 bit products, and every transform length's split into passes (2^16
points and up), with odd sizes, extreme ratios and every flag."""
import numpy as np
import pytest

import privacyamplification_gb300 as pa
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DEFAULT = pa.DEFAULT_FLAGS
# (n, v, flags)
SHORT = [(1024, 32, DEFAULT), (1024, 992, DEFAULT), (1056, 480, 0), (2080, 1024, pa.FLAG_XOR_KEY_REST),
         (19200, 19168, DEFAULT), (19264, 19232, DEFAULT), (65536, 24576, DEFAULT), (65568, 40032, pa.FLAG_COMPRESS),
         (100000, 32, DEFAULT), (262144, 98304, DEFAULT), (262144, 131072, 0)]
# around the boundary: (h + 1) v <= 2^34 is word by word; then 2^16 .. 2^21 points
LONG = [(262144, 131040, DEFAULT), (262176, 131104, DEFAULT), (524288, 196608, DEFAULT), (786432, 32768, 0),
        (1048576, 524288, DEFAULT), (1048608, 524320, DEFAULT), (3000032, 1000032, DEFAULT),
        (4194304, 1572864, pa.FLAG_COMPRESS), (4194336, 4128768, pa.FLAG_XOR_KEY_REST), (8388608, 3145728, DEFAULT),
        (16777248, 6291456, 0), (33554432, 12582912, DEFAULT)]


@pytest.mark.parametrize("n,v,flags", SHORT + LONG)
def test_exact_flag_whole_output(gpu_engine, n, v, flags):
    seed, recv = O.random_block(n, v, n % 9973 + v + flags)
    ks, kr = O.key_split(recv, n, v)
    gpu_engine.set_seed(seed, n, -1)
    out = gpu_engine.process(ks, kr, n, v, flags | pa.FLAG_EXACT)
    assert gpu_engine.last_stats.exact == 1
    assert np.array_equal(out, O.ntt(seed, ks, kr, n, v, flags))


@pytest.mark.parametrize("n", [65536, 1048576])
def test_exact_seed_transform_follows_the_output_length(gpu_engine, n):
    """One static seed, blocks of different v: the exact path's seed transform depends on h and the output length."""
    v1, v2 = n // 4, n // 2
    seed, recv = O.random_block(n, v1, 77)
    gpu_engine.set_seed(seed, n, -1)
    for v, flags in ((v1, DEFAULT), (v2, DEFAULT), (v1, pa.FLAG_XOR_KEY_REST), (v1, DEFAULT)):
        ks, kr = O.key_split(recv, n, v)
        out = gpu_engine.process(ks, kr, n, v, flags | pa.FLAG_EXACT)
        assert np.array_equal(out, O.ntt(seed, ks, kr, n, v, flags))


@pytest.mark.parametrize("n,v,where", [(1024, 384, "key"), (4096, 1536, "seed"), (32768, 12288, "key"),
                                       (32768, 32736, "key_rest"), (20480, 7680, "seed")])
def test_noalloc_output_over_an_input(n, v, where):
    """The result may be written over the seed, the key or key_rest: every input is read first."""
    torch = pytest.importorskip("torch")
    seed, recv = O.random_block(n, v, n + v)
    ks, kr = O.key_split(recv, n, v)
    bufs = {k: torch.from_numpy(np.ascontiguousarray(a, dtype=np.uint32).view(np.int32).copy()).cuda()
            for k, a in (("seed", seed), ("key", ks), ("key_rest", kr))}
    torch.cuda.synchronize()
    pa.process_noalloc(bufs["seed"].data_ptr(), bufs["key"].data_ptr(), bufs["key_rest"].data_ptr(), n, v,
                       bufs[where].data_ptr())
    torch.cuda.synchronize()
    got = bufs[where].cpu().numpy().view(np.uint8)[: v // 8]
    assert np.array_equal(got, O.direct(seed, ks, kr, n, v))


@pytest.mark.parametrize("n,v", [(1024, 32), (1056, 480), (4096, 1536), (10240, 10208), (10304, 10272), (20480, 7680),
                                 (32768, 12288), (65536, 24576), (65568, 40032), (131072, 49152), (196608, 73728),
                                 (262144, 4096)])
def test_short_blocks_by_default(gpu_engine, n, v):
    """Short blocks of pa_process: whole output, zero residual, popcounts of the key and of the placed seed, the second
    block against the kept seed's count."""
    seed, recv = O.random_block(n, v, n + 3 * v)
    ks, kr = O.key_split(recv, n, v)
    gpu_engine.set_seed(seed, n, -1)
    for _ in range(2):
        out = gpu_engine.process(ks, kr, n, v)
        st = gpu_engine.last_stats
        assert np.array_equal(out, O.direct(seed, ks, kr, n, v))
        assert st.exact == 0 and st.max_residual == 0
        assert st.popcount_key == O.popcount(ks, n - v + 1)
        if n & (n - 1) == 0:
            assert st.popcount_seed == O.popcount(seed, n)


def test_short_and_transformed_blocks_share_a_seed(gpu_engine):
    """One seed, blocks on either side of the boundary in turn: the transformed block's spectrum and popcount are not
    disturbed by the short block's, and the other way round."""
    n = 294912
    seed, recv = O.random_block(n, 32, 5)
    gpu_engine.set_seed(seed, n, -1)
    for v in (147456, 4096, 147456, 196608, 4096, 147456):
        ks, kr = O.key_split(recv, n, v)
        out = gpu_engine.process(ks, kr, n, v)
        assert np.array_equal(out, O.ntt(seed, ks, kr, n, v)), v
        assert gpu_engine.last_stats.popcount_key == O.popcount(ks, n - v + 1)


@pytest.mark.parametrize("n,v,exact", [(2097152, 32, 0), (2097152, 2097120, 0), (2097216, 32, 0), (2097248, 2097216, 0),
                                       (1048576, 4096, 0), (4194304, 32, 1), (4194336, 32, 1), (4194368, 4194336, 1)])
def test_long_keys_and_long_results(gpu_engine, n, v, exact):
    """Skewed blocks on either side of the word-by-word product's longest key and result (2^21 bits, exact path 2^22):
    whole output, popcounts of the key and of the seed, which several CTAs count."""
    seed, recv = O.random_block(n, v, n + 5 * v)
    ks, kr = O.key_split(recv, n, v)
    gpu_engine.set_seed(seed, n, 2)
    for _ in range(2):
        out = gpu_engine.process(ks, kr, n, v, DEFAULT | (pa.FLAG_EXACT if exact else 0))
        st = gpu_engine.last_stats
        assert np.array_equal(out, O.ntt(seed, ks, kr, n, v))
        assert st.exact == exact
        if not exact:
            assert st.popcount_key == O.popcount(ks, n - v + 1)
            if n & (n - 1) == 0:
                assert st.popcount_seed == O.popcount(seed, n)
