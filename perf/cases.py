"""Performance cases: the decode work a program gives this library, through
its public entry points, with seeded synthetic content of the benchmark's
distributions (cudec_b200/workload.py).

A case is a batch of `chunks` chunks of `bytes` decompressed bytes each, or,
with `uneven`, of lognormal sizes with that median (the benchmark's mixed
workload: sigma 1.2, copy probability 0.2-0.8 per chunk, 5 % of the chunks
incompressible). `path` names the entry point. Sizes belong to the case;
content belongs to the seed. Every output is bytes or status records, so
results are compared exactly.
"""
import ctypes
import math
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import cudec_b200 as cd
from cudec_b200 import workload as W
from cudec_b200.device import DeviceBatch, _DevView

MIX = ("lz4", "snappy", "zstd", "gdeflate")
MIX_WEIGHTS = (4, 2, 3, 1)  # the serving workload's 40 / 20 / 30 / 10 %


def _case(path, chunks, size, uneven=False, level=0, checksum=False):
    return {"path": path, "chunks": chunks, "bytes": size, "uneven": uneven, "level": level,
            "checksum": checksum}


def listed():
    return [
        # a handful of 4,000-byte records or cache pages: launch and latency
        dict(_case("lz4", 40, 4000), name="lz4_tiny"),
        # the headline batch: 64 KiB blocks of a column, checkpoint or cache
        dict(_case("lz4", 1024, 65536), name="lz4_blocks"),
        # a table scan's pages: Snappy, every size from 256 bytes up
        dict(_case("snappy", 8000, 16384, uneven=True), name="snappy_pages"),
        # a data set's shards at the codec's default level, 1 MiB frames
        dict(_case("zstd", 512, 1 << 20, level=3), name="zstd_default"),
        # archives written once at high level, checksummed, odd frame size
        dict(_case("zstd", 96, 260000, level=19, checksum=True), name="zstd_archive"),
        # one request's few frames: the latency of a single frame
        dict(_case("zstd", 6, 131072, level=3, checksum=True), name="zstd_few"),
        # a level's worth of texture pages
        dict(_case("gdeflate", 4096, 65536, level=6), name="gdeflate_pages"),
        # a few pages for one asset
        dict(_case("gdeflate", 24, 50001, level=6), name="gdeflate_few"),
        # every format in one call, uneven sizes (a plan kept by the program)
        dict(_case("mixed", 10000, 16384, uneven=True, level=3, checksum=True), name="mixed"),
        # compressed chunks in pinned host memory, output in device memory
        dict(_case("stream", 1024, 65536), name="stream_pinned"),
        # a .lz4 file as the lz4 tool writes it: 4 MiB blocks and a content
        # checksum, host memory to host memory
        dict(_case("frame", 16, 4 << 20, checksum=True), name="lz4_file"),
        # eight requests of 64 pages each that arrive together at the server
        dict(_case("serve", 512, 16384, level=3, checksum=True), name="serve_burst"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["lz4", "lz4", "snappy", "snappy", "zstd", "zstd", "gdeflate", "mixed",
                       "stream", "frame", "serve"])
    if path in ("lz4", "snappy"):
        uneven = rng.random() < 0.4
        size = _log(rng, 3000, 30000) if uneven else _log(rng, 600, 2 << 20)
        total = _log(rng, 200000, 200 << 20)
        return _case(path, max(1, min(60000, total // size)), size, uneven)
    if path == "zstd":
        level = rng.choice([1, 3, 3, 19])
        size = _log(rng, 5000, 1 << 20)
        total = _log(rng, 300000, 24 << 20 if level == 19 else 400 << 20)
        return _case(path, max(1, min(20000, total // size)), size, False, level,
                     rng.random() < 0.5)
    if path == "gdeflate":
        size = _log(rng, 4000, 65536)
        total = _log(rng, 300000, 200 << 20)
        return _case(path, max(1, min(8000, total // size)), size, False, 6)
    if path == "mixed":
        return _case(path, _log(rng, 200, 9000), _log(rng, 4000, 18000), True, 3, True)
    if path == "stream":
        size = _log(rng, 4000, 1 << 20)
        total = _log(rng, 1 << 20, 64 << 20)
        return _case(path, max(1, total // size), size)
    if path == "frame":
        size = rng.choice([65536, 262144, 1 << 20, 4 << 20])
        return _case(path, max(1, _log(rng, 1 << 20, 60 << 20) // size), size, False, 0,
                     rng.random() < 0.5)
    return _case(path, 8 * rng.randint(2, 64), 16 * rng.randint(100, 1024), False, 3, True)


def _sizes(case):
    n, size = case["chunks"], case["bytes"]
    if case["uneven"]:
        return W.mixed_sizes(n, 7 + n, size)
    return np.full(n, size, dtype=np.int64)


def _formats(case):
    if case["path"] not in ("mixed", "serve"):
        return [case["path"]] * case["chunks"]
    p = np.asarray(MIX_WEIGHTS, dtype=np.float64)
    rng = np.random.default_rng(11 + case["chunks"])
    return [MIX[k] for k in rng.choice(len(MIX), size=case["chunks"], p=p / p.sum())]


def _page_limited(sizes, formats):
    """A GDeflate chunk is one page: at most 64 KiB."""
    return np.array([min(int(s), 65536) if f == "gdeflate" else int(s)
                     for s, f in zip(sizes, formats)], dtype=np.int64)


def _content(case, seed):
    """(compressed chunks, decompressed sizes, formats)."""
    fmts = _formats(case)
    sizes = _page_limited(_sizes(case), fmts)
    n, level, checksum = len(sizes), case["level"], case["checksum"]
    rng = np.random.default_rng(seed)
    probs = rng.uniform(0.2, 0.8, n) if case["uneven"] else np.full(n, 0.5)
    random_chunk = rng.random(n) < (0.05 if case["uneven"] else 0.0)

    def params(f, p, r):
        if r:
            return W.lz_params(p, True)
        if f == "zstd":
            return W.zstd_params(p, 0.1)
        return W.gdeflate_params(p) if f == "gdeflate" else W.lz_params(p)

    ps = [params(f, float(p), bool(r)) for f, p, r in zip(fmts, probs, random_chunk)]
    buf, offs = W.generate(sizes, ps, param_idx=np.arange(n),
                           seeds=rng.integers(0, 1 << 63, n, dtype=np.uint64))
    raws = [buf[int(o):int(o) + int(s)] for o, s in zip(offs, sizes)]

    def one(k):
        f, r = fmts[k], raws[k]
        if f == "snappy":
            return W.snappy_compress(r)
        if f == "zstd":
            return W.zstd_compress(r, level, 20, checksum)
        if f == "gdeflate":
            return W.gdeflate_compress(r, 6)
        return W.lz4_compress(r)

    with ThreadPoolExecutor(max_workers=min(os.cpu_count() or 1, 32)) as pool:
        comps = list(pool.map(one, range(n), chunksize=max(1, n // 256)))
    return comps, sizes, fmts


def _prepare_stream(case, seed):
    comps, sizes, _ = _content(dict(case, path="lz4"), seed)
    n = len(comps)
    packed = np.frombuffer(b"".join(comps), dtype=np.uint8)
    pinned = torch.from_numpy(packed.copy()).pin_memory()
    lens = np.array([len(c) for c in comps], dtype=np.uint64)
    at = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64)
    slot = (sizes.astype(np.uint64) + 255) // 256 * 256
    to = np.concatenate([[0], np.cumsum(slot)[:-1]]).astype(np.uint64)
    dst = torch.zeros(int(slot.sum()), dtype=torch.uint8, device="cuda")
    return {"ctx": cd.StreamContext(), "pinned": pinned, "dst": dst, "n": n,
            "src_ptrs": at + np.uint64(pinned.data_ptr()), "src_sizes": lens,
            "dst_ptrs": to + np.uint64(dst.data_ptr()), "caps": sizes.astype(np.uint64),
            "records": np.zeros(16 * n, dtype=np.uint8)}


def _prepare_frame(case, seed):
    size = case["bytes"]
    buf, _ = W.generate([size] * case["chunks"], W.lz_params(),
                        seeds=np.random.default_rng(seed).integers(
                            0, 1 << 63, case["chunks"], dtype=np.uint64))
    block_id = {65536: 4, 262144: 5, 1 << 20: 6, 4 << 20: 7}[size]
    frame = W.lz4f_compress(buf, block_id, True, case["checksum"], False, True)
    return {"frame": np.frombuffer(frame, dtype=np.uint8), "out": np.zeros(len(buf), np.uint8),
            "written": ctypes.c_size_t(0)}


def _prepare_serve(case, seed):
    comps, sizes, fmts = _content(case, seed)
    per = len(comps) // 8
    requests = []
    for k in range(8):
        part = slice(k * per, (k + 1) * per)
        cs = comps[part]
        offs = np.concatenate([[0], np.cumsum([len(c) for c in cs])[:-1]])
        requests.append((np.frombuffer(b"".join(cs), dtype=np.uint8), offs,
                         [len(c) for c in cs], sizes[part], fmts[part]))
    total = sum(len(c) for c in comps) + int(sizes.sum())
    return {"server": cd.Server(2 * total + (8 << 20), 4, cd.SERVER_MIXED, 4096),
            "requests": requests, "open": []}


def prepare(case, seed):
    path = case["path"]
    if path == "stream":
        state = _prepare_stream(case, seed)
    elif path == "frame":
        state = _prepare_frame(case, seed)
    elif path == "serve":
        state = _prepare_serve(case, seed)
    else:
        comps, sizes, fmts = _content(case, seed)
        batch = DeviceBatch(comps, sizes)
        state = {"batch": batch}
        if path == "zstd":
            batch.workspace()
        if path == "mixed":
            state["plan"] = cd.MixedPlan()
            state["formats"] = fmts
            state["codes"] = torch.tensor([cd.FORMAT_CODES[f] for f in fmts],
                                          dtype=torch.uint8).cuda()
    state["path"] = path
    return state


def _serve(state):
    server = state["server"]
    for ticket in state["open"]:
        server.release(ticket)
    state["open"] = [server.submit(*r)[1] for r in state["requests"]]
    out = {}
    for k, (ticket, r) in enumerate(zip(state["open"], state["requests"])):
        _, records, ptrs, _ = server.wait(ticket)
        out["records%d" % k] = records.view(np.uint8)
        # equal chunk sizes, a multiple of 16: a request's outputs are one range
        view = _DevView(int(ptrs[0]), int(np.sum(r[3])))
        view.owner = server  # the outputs lie in the server's memory
        out["bytes%d" % k] = torch.as_tensor(view, device="cuda")
    return out


def run(state):
    path = state["path"]
    if path == "serve":
        return _serve(state)
    if path == "stream":
        status = state["ctx"].decode(
            state["src_ptrs"].ctypes.data, state["src_sizes"].ctypes.data,
            state["dst_ptrs"].ctypes.data, state["caps"].ctypes.data, state["n"],
            cd.MEM_DEVICE, state["records"].ctypes.data)
        return {"status": status, "bytes": state["dst"], "records": state["records"]}
    if path == "frame":
        frame, out, written = state["frame"], state["out"], state["written"]
        status = cd.lib().cudec_lz4f_decompress(frame.ctypes.data, len(frame), out.ctypes.data,
                                                len(out), ctypes.byref(written))
        return {"status": status, "bytes": out, "written": written.value}
    batch = state["batch"]
    if path == "mixed":
        stream = torch.cuda.current_stream().cuda_stream
        args = batch.args()
        status = state["plan"].decode(*args[:4], state["codes"].data_ptr(), *args[4:],
                                      stream=stream)
    else:
        status = batch.run(path)
    return {"status": status, "bytes": batch.d_dst, "records": batch.d_results}


# compressed bytes over decompressed bytes of the content, by format
RATIO = {"lz4": 0.55, "snappy": 0.55, "zstd": 0.24, "gdeflate": 0.37}


def work(case):
    """Compressed bytes read once, decompressed bytes written once."""
    fmts = _formats(case)
    sizes = _page_limited(_sizes(case), fmts)
    total = sum(int(s) * (1.0 + RATIO.get(f, RATIO["lz4"])) for s, f in zip(sizes, fmts))
    return {"bytes": total + 16.0 * len(fmts), "flops": 0}


def tolerance(case):
    return "exact"
