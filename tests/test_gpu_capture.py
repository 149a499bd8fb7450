"""Captured blocks of the device form: a graph's replay hashes with the seed that the engine holds then, whatever was set
or hashed between capture and replay, and blocks that are not captured are right beside the replays."""
import numpy as np
import pytest

import privacyamplification_gb300 as pa
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DEFAULT = pa.DEFAULT_FLAGS
EXACT = DEFAULT | pa.FLAG_EXACT


@pytest.mark.parametrize("n,v,flags,reuse", [
    (4096, 1536, DEFAULT, -1), (65568, 24576, DEFAULT, -1), (1 << 19, 196608, DEFAULT, -1), (600032, 200032, DEFAULT, -1),
    (600032, 200032, DEFAULT, 1), (1 << 21, 786432, DEFAULT, 1), (2500000, 900000, DEFAULT, -1),
    (1 << 19, 196608, EXACT, -1), (600032, 200032, EXACT, -1)])
def test_replays_follow_the_seed(pa_lib, n, v, flags, reuse):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + v + flags)
    words = lambda k: rng.integers(0, 1 << 32, k, dtype=np.uint64).astype(np.uint32)
    dev = lambda a: torch.from_numpy(a.view(np.int32).copy()).cuda()
    seeds = [words(n // 32) for _ in range(3)]
    ks, kr = O.key_split(words(n // 32 + 1), n, v)
    v2 = v // 2 // 32 * 32  # another placement of the same seed
    ks2, kr2 = O.key_split(words(n // 32 + 1), n, v2)
    plain = flags & ~pa.FLAG_EXACT
    want = lambda seed: O.ntt(seed, ks, kr, n, v, plain)
    d_seeds, d_ks, d_kr, d_ks2, d_kr2 = [dev(s) for s in seeds], dev(ks), dev(kr), dev(ks2), dev(kr2)
    out, out2 = (torch.zeros(x // 8, dtype=torch.uint8, device="cuda") for x in (v, v2))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with pa.Engine(max_sample_size=n) as eng:
        def set_seed(k):
            eng.set_seed_device(d_seeds[k].data_ptr(), n, reuse, stream=stream.cuda_stream)

        def block():
            eng.process_device(d_ks.data_ptr(), d_kr.data_ptr(), n, v, out.data_ptr(), flags, stream=stream.cuda_stream)

        def other():
            eng.process_device(d_ks2.data_ptr(), d_kr2.data_ptr(), n, v2, out2.data_ptr(), flags, stream=stream.cuda_stream)

        def result(o=out):
            torch.cuda.synchronize()
            got = o.cpu().numpy().copy()
            o.zero_()
            torch.cuda.synchronize()
            return got

        set_seed(0)
        block()
        assert np.array_equal(result(), want(seeds[0]))
        set_seed(0)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            block()
        for k in (0, 1, 1):
            set_seed(k)
            torch.cuda.synchronize()
            graph.replay()
            assert np.array_equal(result(), want(seeds[k])), "replay after seed %d" % k
        set_seed(2)
        other()
        torch.cuda.synchronize()
        graph.replay()
        assert np.array_equal(result(), want(seeds[2])), "replay after a block of another length"
        assert np.array_equal(result(out2), O.ntt(seeds[2], ks2, kr2, n, v2, plain))
        set_seed(2)
        other()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        if reuse < 0:  # the same seed, not captured, behind the replay
            other()
            assert np.array_equal(result(out2), O.ntt(seeds[2], ks2, kr2, n, v2, plain)), "block after a replay"
        del graph
        torch.cuda.synchronize()


@pytest.mark.parametrize("n,v", [(4096, 1536), (600032, 200032)])
def test_captured_seed(pa_lib, n, v):
    """The seed's copy in the graph: replays follow the caller's buffer."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    words = lambda k: rng.integers(0, 1 << 32, k, dtype=np.uint64).astype(np.uint32)
    dev = lambda a: torch.from_numpy(a.view(np.int32).copy()).cuda()
    ks, kr = O.key_split(words(n // 32 + 1), n, v)
    d_seed, d_ks, d_kr = dev(words(n // 32)), dev(ks), dev(kr)
    out = torch.zeros(v // 8, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with pa.Engine(max_sample_size=n) as eng:
        def block():
            eng.set_seed_device(d_seed.data_ptr(), n, -1, stream=stream.cuda_stream)
            eng.process_device(d_ks.data_ptr(), d_kr.data_ptr(), n, v, out.data_ptr(), stream=stream.cuda_stream)

        block()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            block()
        for _ in range(2):
            seed = words(n // 32)
            d_seed.copy_(dev(seed))
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), O.ntt(seed, ks, kr, n, v))
            st = eng.sync()
            assert st.popcount_key == O.popcount(ks, n - v + 1)
        # a block that is not captured: its seed is the replayed one
        out.zero_()
        eng.process_device(d_ks.data_ptr(), d_kr.data_ptr(), n, v, out.data_ptr(), stream=stream.cuda_stream)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), O.ntt(seed, ks, kr, n, v))
        if n & (n - 1) == 0:
            assert eng.sync().popcount_seed == O.popcount(seed, n)
        del graph
        torch.cuda.synchronize()


def test_captured_chunks(pa_lib):
    """A block above 2^27 bits: replays with another seed, statistics behind a replay, and ordinary blocks behind those."""
    torch = pytest.importorskip("torch")
    n, v = (1 << 27) + 32, 1 << 26
    rng = np.random.default_rng(28)
    words = lambda k: rng.integers(0, 1 << 32, k, dtype=np.uint64).astype(np.uint32)
    dev = lambda a: torch.from_numpy(a.view(np.int32).copy()).cuda()
    seeds = [words(n // 32) for _ in range(2)]
    ks, kr = O.key_split(words(n // 32 + 1), n, v)
    want = [O.ntt(seed, ks, kr, n, v) for seed in seeds]
    d_seeds, d_ks, d_kr = [dev(s) for s in seeds], dev(ks), dev(kr)
    out = torch.zeros(v // 8, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with pa.Engine(max_sample_size=n) as eng:
        def block(k):
            eng.set_seed_device(d_seeds[k].data_ptr(), n, -1, stream=stream.cuda_stream)
            eng.process_device(d_ks.data_ptr(), d_kr.data_ptr(), n, v, out.data_ptr(), stream=stream.cuda_stream)

        block(0)
        assert eng.sync().gpu_ms > 0
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            eng.process_device(d_ks.data_ptr(), d_kr.data_ptr(), n, v, out.data_ptr(), stream=stream.cuda_stream)
        for k in (1, 0):
            eng.set_seed_device(d_seeds[k].data_ptr(), n, -1, stream=stream.cuda_stream)
            out.zero_()
            torch.cuda.synchronize()
            graph.replay()
            assert eng.sync().exact == 2
            assert np.array_equal(out.cpu().numpy(), want[k])
            out.zero_()
            torch.cuda.synchronize()
            block(1 - k)
            assert eng.sync().gpu_ms > 0
            assert np.array_equal(out.cpu().numpy(), want[1 - k])
        del graph
        torch.cuda.synchronize()
