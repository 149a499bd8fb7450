"""The FP32 transforms of short blocks (up to 2^17 bits), which single blocks do not run (they are multiplied word by word)
and the pool does: structured inputs in batches, grouped, served and in every split, against the oracle."""
import numpy as np
import pytest

import privacyamplification_gb300 as pa
from oracle import oracle as O
from test_gpu_exact import structured_families

pytestmark = pytest.mark.gpu

DEFAULT = pa.DEFAULT_FLAGS


@pytest.fixture()
def engine(pa_lib):
    with pa.Engine(max_sample_size=1 << 18) as eng:
        yield eng


def device(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.uint32).view(np.int32).copy()).cuda()


def run_batch(torch, eng, blocks, n, v, static, flags):
    """Outputs and statistics of blocks (seed, key_start, key_rest) as one batch."""
    keep, outs, jobs = [], [], []
    for seed, ks, kr in blocks:
        sd, k, r = (device(torch, a) for a in (seed, ks, kr))
        out = torch.zeros(v // 8, dtype=torch.uint8, device="cuda")
        sid = eng.seed_cache_add(np.ascontiguousarray(seed), n, v, DEFAULT) if static else -1
        jobs.append(pa.PAJob(None if static else sd.data_ptr(), sid, k.data_ptr(), r.data_ptr(), n, v, DEFAULT,
                             out.data_ptr()))
        keep.append((sd, k, r))
        outs.append(out)
    torch.cuda.synchronize()
    eng.batch_run(jobs, flags)
    stats = eng.batch_sync(len(jobs))
    return [o.cpu().numpy() for o in outs], stats


def structured(n, v):
    fams, keys = structured_families(n, v)
    return {(f, k): (seed, *O.key_split(recv, n, v)) for f, seed in fams.items() for k, recv in keys.items()}


@pytest.mark.parametrize("static", [True, False])
@pytest.mark.parametrize("flags", [0, pa.BATCH_NO_GROUP], ids=["grouped", "single"])
@pytest.mark.parametrize("logn", [10, 12, 14, 15, 16, 17])
def test_structured_blocks_in_batches(engine, logn, flags, static):
    """Up to 2^15 bits a block is one CTA, whose error bound (half the guard's limit) holds for every input."""
    torch = pytest.importorskip("torch")
    n = 1 << logn
    v = n // 4 + n // 8
    blocks = structured(n, v)
    outs, stats = run_batch(torch, engine, list(blocks.values()), n, v, static, flags)
    for (name, blk), out, st in zip(blocks.items(), outs, stats):
        assert np.array_equal(out, O.direct(*blk, n, v)), (name, st.max_residual)
        if logn <= 15:
            assert st.exact == 0 and st.max_residual < 0.125, (name, st.max_residual)


@pytest.mark.parametrize("logn", [10, 15, 17])
def test_structured_blocks_served(engine, logn):
    n = 1 << logn
    v = n // 4 + n // 8
    for name, (seed, ks, kr) in structured(n, v).items():
        out = np.zeros(v // 8, np.uint8)
        args = [np.ascontiguousarray(a) for a in (seed, ks, kr)]
        ticket = engine.submit(pa.PAJob(args[0].ctypes.data, -1, args[1].ctypes.data, args[2].ctypes.data, n, v, DEFAULT,
                                        out.ctypes.data))
        while engine.poll(ticket) is None:
            pass
        assert np.array_equal(out, O.direct(seed, ks, kr, n, v)), name


@pytest.mark.parametrize("static", [True, False])
@pytest.mark.parametrize("log_n", [15, 16])
def test_every_split(engine, log_n, static):
    """Rows of 2^10 and 2^11, columns of 2^5 and 2^6: a random and a structured block."""
    torch = pytest.importorskip("torch")
    n = 1 << (log_n + 1)
    v = n // 4 + n // 8
    seed, recv = O.random_block(n, v, log_n)
    blocks = [(seed, *O.key_split(recv, n, v)), structured(n, v)[("run_1/4", "random")]]
    for log_n2 in range(10, log_n - 4):
        engine.set_split(log_n, log_n2)
        outs, _ = run_batch(torch, engine, blocks, n, v, static, pa.BATCH_NO_GROUP)
        for blk, out in zip(blocks, outs):
            assert np.array_equal(out, O.direct(*blk, n, v)), log_n2
