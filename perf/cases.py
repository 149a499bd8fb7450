"""The engine's work as its callers have it done, as cases that can be timed and compared.

Every case hashes blocks through the public entry points of `privacyamplification_gb300` with the default
flags (XOR with key_rest, compressed output).  Key and seed bits are i.i.d. Bernoulli(1/2) except in the
`guard` kind.  Kinds:

* noalloc: one small block with its own seed on the caller's device buffers (process_noalloc).
* device:  blocks whose data stays in HBM (process_device), the seed set once (static) or per block (own).
* host:    one block from pinned host buffers and back (process), static seed.
* exact:   the same with FLAG_EXACT, the caller's choice of integer arithmetic.
* guard:   the same without the flag on run-structured input (a run of ones in the seed, a key of ones),
           which exceeds the FP32 budget, so the engine detects it and recomputes the block exactly.
* batch:   an uneven mix of blocks as one captured batch (batch_run with BATCH_GRAPH, batch_sync).
* serve:   requests with their own seeds, submitted together and collected as they finish (submit, poll).

Sizes are in bits: n the block (seed) length, v the output length; multiples of 32.
"""
import random

import numpy as np
import torch

import privacyamplification_gb300 as pa

FLAGS = pa.DEFAULT_FLAGS
_shared = {}


def listed():
    return [
        # a short key block of a latency-critical host that owns all device memory
        {"name": "noalloc_4k", "kind": "noalloc", "n": 4096, "v": 1536},
        # the plain method's small block (h = n/2 + n/8, v = n/4 + n/8), a block at a time from the host
        {"name": "host_64k", "kind": "host", "n": 1 << 16, "v": 24576},
        # a megabit block against a seed that is kept
        {"name": "device_1m", "kind": "device", "n": 1 << 20, "v": 393216, "own_seed": False},
        # an odd size, every block with its own seed
        {"name": "device_odd_5m_own", "kind": "device", "n": 5000224, "v": 1600032, "own_seed": True},
        # the reference's default size, static seed: data resident in HBM
        {"name": "device_128m", "kind": "device", "n": 1 << 27, "v": 50331648, "own_seed": False},
        # the same with a fresh seed for every block
        {"name": "device_128m_own", "kind": "device", "n": 1 << 27, "v": 50331648, "own_seed": True},
        # the reference's default size end to end from pinned host memory
        {"name": "host_128m", "kind": "host", "n": 1 << 27, "v": 50331648},
        # integer arithmetic on request, an odd size
        {"name": "exact_odd_3m", "kind": "exact", "n": 3000032, "v": 1000032},
        # structured key material: the guard's recompute
        {"name": "guard_32m", "kind": "guard", "n": 1 << 25, "v": 12582912},
        # the largest block of the precision workload, a fresh seed
        {"name": "device_512m_own", "kind": "device", "n": 1 << 29, "v": 201326592, "own_seed": True},
        # the uneven mix, half of it with cached static seeds, half with own seeds
        {"name": "batch_mix_64", "kind": "batch", "count": 64, "log_lo": 18, "log_hi": 25, "mix": 4},
        # eight requests in flight, each with its own seed
        {"name": "serve_8", "kind": "serve", "count": 8, "log_lo": 20, "log_hi": 27, "mix": 5},
    ]


def _size(rng, lo, hi, ratio=(0.1, 0.9), odd=0.6):
    """(n, v): n log-uniform in [2^lo, 2^hi], a power of two or a multiple of 32."""
    n = int(2 ** rng.uniform(lo, hi)) // 32 * 32
    if rng.random() > odd:
        n = 1 << max(lo, n.bit_length() - 1)
    v = int(n * rng.uniform(*ratio)) // 32 * 32
    return n, min(max(32, v), n - 32)


def draw(rng):
    kind = rng.choice(["noalloc", "device", "device", "device", "host", "exact", "guard", "batch", "serve"])
    if kind == "noalloc":
        n, v = _size(rng, 10, 15)
        return {"kind": kind, "n": n, "v": v}
    if kind == "device":
        n, v = _size(rng, 12, 27)
        return {"kind": kind, "n": n, "v": v, "own_seed": rng.random() < 0.5}
    if kind == "host":
        n, v = _size(rng, 12, 27)
        return {"kind": kind, "n": n, "v": v}
    if kind == "exact":
        n, v = _size(rng, 12, 26)
        return {"kind": kind, "n": n, "v": v}
    if kind == "guard":
        n = 1 << rng.randrange(22, 27)
        return {"kind": kind, "n": n, "v": n // 4 + n // 8}
    if kind == "batch":
        lo = rng.randrange(16, 21)
        return {"kind": kind, "count": rng.randrange(9, 64), "log_lo": lo, "log_hi": rng.randrange(lo + 2, 26),
                "mix": rng.randrange(1 << 20)}
    return {"kind": kind, "count": rng.randrange(3, 9), "log_lo": 20, "log_hi": rng.randrange(23, 28),
            "mix": rng.randrange(1 << 20)}


def _mix(case):
    """The block sizes of a batch or of a set of requests, from the case alone."""
    rng = random.Random(case["mix"])
    sizes = []
    for _ in range(case["count"]):
        n = max(2048, int(2 ** rng.uniform(case["log_lo"], case["log_hi"])) // 1024 * 1024)
        v = max(128, int(n * rng.uniform(0.2, 0.8)) // 128 * 128)
        sizes.append((n, v))
    return sizes


def _blocks(case):
    """(n, v, own seed) of every block of a case."""
    if case["kind"] == "batch":
        return [(n, v, i % 2 == 1) for i, (n, v) in enumerate(_mix(case))]
    if case["kind"] == "serve":
        return [(n, v, True) for n, v in _mix(case)]
    return [(case["n"], case["v"], case["kind"] == "noalloc" or bool(case.get("own_seed")))]


def work(case):
    """Packed bits in and out; the floating-point work of a real transform of length n of the key (and of a
    seed that is used once) and of one inverse."""
    nbytes = flops = 0
    for n, v, own in _blocks(case):
        nbytes += (n - v) // 8 + 4 + v // 8 + n // 8 + v // 8
        flops += (3 if own else 2) * 2.5 * n * (n.bit_length() - 1)
    return {"bytes": nbytes, "flops": int(flops)}


def _words(gen, count):
    return torch.randint(-2 ** 31, 2 ** 31, (count,), dtype=torch.int32, generator=gen, device="cuda")


def _inputs(case, seed):
    """Per block: seed words, key_start words and key_rest words on the GPU."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    blocks = []
    for n, v, _ in _blocks(case):
        sd, ks, kr = _words(gen, n // 32), _words(gen, n // 32), _words(gen, v // 32)
        if case["kind"] == "guard":
            at = random.Random(seed).randrange(n // 64)
            sd.zero_()
            sd[at:at + n // 64] = -1
            ks.fill_(-1)
        blocks.append((sd, ks, kr))
    return blocks


def _host(t):
    """A pinned host copy of words, as numpy sees it (the tensor keeps the memory)."""
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p, p.numpy().view(np.uint32)


def _stream():
    """The stream that a program queues its device-resident blocks on, one after another."""
    if "stream" not in _shared:
        _shared["stream"] = torch.cuda.Stream()
    return _shared["stream"].cuda_stream


def _job(n, v, out, key_start, key_rest, seed_words=0, seed_id=-1):
    return pa.PAJob(seed_words or None, seed_id, key_start, key_rest, n, v, FLAGS, out)


def prepare(case, seed):
    kind = case["kind"]
    blocks = _inputs(case, seed)
    st = {"case": case, "kind": kind}
    if kind in ("noalloc", "device"):
        n, v = case["n"], case["v"]
        st["in"] = blocks[0]
        st["out"] = torch.zeros(pa.output_bytes(n, v, FLAGS), dtype=torch.uint8, device="cuda")
        st["stream"] = _stream()
        torch.cuda.synchronize()
        if kind == "device":
            st["eng"] = pa.Engine(max_sample_size=n)
            if not case["own_seed"]:
                st["eng"].set_seed_device(blocks[0][0].data_ptr(), n, -1, st["stream"])
    elif kind in ("host", "exact", "guard"):
        n, v = case["n"], case["v"]
        sd, ks, kr = (_host(t) for t in blocks[0])
        out = torch.zeros(pa.output_bytes(n, v, FLAGS), dtype=torch.uint8, pin_memory=True)
        st["keep"] = (ks, kr, out)
        st["ks"], st["kr"], st["out"] = ks[1], kr[1], out.numpy()
        torch.cuda.synchronize()
        st["eng"] = pa.Engine(max_sample_size=n)
        st["eng"].set_seed(sd[1], n, -1)
    elif kind == "batch":
        sizes = _blocks(case)
        eng = pa.Engine(max_sample_size=1 << case["log_hi"])
        st["outs"] = [torch.zeros(pa.output_bytes(n, v, FLAGS), dtype=torch.uint8, device="cuda") for n, v, _ in sizes]
        torch.cuda.synchronize()
        jobs = []
        for (n, v, own), (sd, ks, kr), out in zip(sizes, blocks, st["outs"]):
            sid = -1 if own else eng.seed_cache_add(sd.cpu().numpy().view(np.uint32), n, v, FLAGS)
            jobs.append(_job(n, v, out.data_ptr(), ks.data_ptr(), kr.data_ptr(), sd.data_ptr() if own else 0, sid))
        st["keep"], st["jobs"], st["eng"] = blocks, jobs, eng
    else:
        sizes = _blocks(case)
        eng = pa.Engine(max_sample_size=1 << case["log_hi"])
        st["outs"], st["keep"], jobs = [], [], []
        for (n, v, _), words in zip(sizes, blocks):
            sd, ks, kr = (_host(t) for t in words)
            out = torch.zeros(pa.output_bytes(n, v, FLAGS), dtype=torch.uint8, pin_memory=True)
            jobs.append(_job(n, v, out.data_ptr(), ks[0].data_ptr(), kr[0].data_ptr(), sd[0].data_ptr()))
            st["outs"].append(out)
            st["keep"].append((sd, ks, kr))
        torch.cuda.synchronize()
        eng.pool_reserve(1 << case["log_hi"], case["count"])
        st["jobs"], st["eng"] = jobs, eng
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "noalloc":
        sd, ks, kr = st["in"]
        pa.process_noalloc(sd.data_ptr(), ks.data_ptr(), kr.data_ptr(), case["n"], case["v"], st["out"].data_ptr(),
                           FLAGS, st["stream"])
        return st["out"]
    if kind == "device":
        sd, ks, kr = st["in"]
        if case["own_seed"]:
            st["eng"].set_seed_device(sd.data_ptr(), case["n"], 1, st["stream"])
        st["eng"].process_device(ks.data_ptr(), kr.data_ptr(), case["n"], case["v"], st["out"].data_ptr(), FLAGS,
                                 st["stream"])
        return st["out"]
    if kind in ("host", "exact", "guard"):
        flags = FLAGS | (pa.FLAG_EXACT if kind == "exact" else 0)
        return st["eng"].process(st["ks"], st["kr"], case["n"], case["v"], flags, out=st["out"])
    if kind == "batch":
        st["eng"].batch_run(st["jobs"], pa.BATCH_GRAPH)
        st["eng"].batch_sync(len(st["jobs"]))
        return st["outs"]
    eng, waiting, running = st["eng"], list(reversed(st["jobs"])), []
    while waiting or running:
        while waiting:
            ticket = eng.submit(waiting[-1])
            if ticket is None:
                break
            running.append(ticket)
            waiting.pop()
        running = [t for t in running if eng.poll(t) is None]
    return st["outs"]


def _direct(words, n, v):
    """out[i] = parity of sum_j key_start[j] seed[(i - j) mod n], XOR key_rest[i], by a 64-bit transform."""
    sd, ks, kr = (np.unpackbits(np.ascontiguousarray(t.cpu().numpy().view(np.uint32).astype(">u4")).view(np.uint8))
                  for t in words)
    key = np.zeros(n)
    key[:n - v + 1] = ks[:n - v + 1]
    c = np.fft.irfft(np.fft.rfft(key) * np.fft.rfft(sd.astype(np.float64)), n)[:v]
    return np.packbits((np.rint(c).astype(np.int64) & 1).astype(np.uint8) ^ kr)


def exact(case, seed):
    if max(n for n, _, _ in _blocks(case)) > 1 << 23 or case["kind"] in ("batch", "serve"):
        return None
    return _direct(_inputs(case, seed)[0], case["n"], case["v"])
