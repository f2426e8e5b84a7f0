"""GPU parity of the LZ4 / Snappy batch entries at each width of their CTAs
(512, 256 and 128 threads per chunk, by the batch's chunks per SM), on chunks
whose sizes and tokens sit at the decoder's edges: a region, a tile and the
tiles past it, runs at and past what a lane, a warp and the whole CTA copy.
Every status, byte and untouched tail equals the oracle's.
"""
import random

import pytest

import oracle
from cudec_b200 import workload as W
from cudec_b200.device import DeviceBatch

pytestmark = pytest.mark.gpu

PACK = {"lz4": W.lz4_compress, "snappy": W.snappy_compress}
WANT = {"lz4": oracle.lz4_decode, "snappy": oracle.snappy_decode}


def chunks(n):
    rng = random.Random(n)
    runs = (1, 15, 16, 17, 31, 32, 127, 128, 129, 1023, 1024, 1025, 5000)
    out = []
    for i in range(n):
        size = (1, 52, 53, 6656, 6657, 13312, 26624, 40000)[i % 8]
        kind = i // 8 % 4
        if kind == 0:
            data = W.generate([size], W.lz_params(0.5), seeds=[i])[0].tobytes()
        elif kind == 1:  # runs of random and repeated bytes, each copied again later
            parts = [rng.randbytes(runs[k % 13]) + bytes([k % 7]) * runs[(k + i) % 13]
                     for k in range(60)]
            data = (b"".join(parts) * 2)[:size]
        elif kind == 2:  # few tokens per tile
            data = W.generate([size], W.lz_params(0.02), seeds=[i])[0].tobytes()
        else:
            data = (rng.randbytes(1 + i % 40) * size)[:size]
        out.append(data)
    return out


@pytest.mark.parametrize("fmt", ["lz4", "snappy"])
@pytest.mark.parametrize("n", [32, 200, 500])
def test_widths(cuda, fmt, n):
    import torch
    raws = chunks(n)
    comps = [PACK[fmt](r) for r in raws]
    rng = random.Random(5)
    for i in range(0, n, 11):  # some mutants among them
        b = bytearray(comps[i])
        b[rng.randrange(len(b))] ^= 1 << rng.randrange(8)
        comps[i] = bytes(b)
    caps = [len(r) for r in raws]
    b = DeviceBatch(comps, caps, device=cuda, dst_align=16, dst_skew=3, src_skew=5)
    assert b.run(fmt) == 0
    torch.cuda.synchronize()
    res, dst = b.results(), b.dst_host()
    for i in range(n):
        st, out = WANT[fmt](comps[i], caps[i])
        assert res[i]["status"] == st, (i, res[i], st)
        if st == 0:
            assert res[i]["bytes_written"] == len(out)
            assert b.output(i, dst) == out + b"\xa5" * (caps[i] - len(out)), i


@pytest.mark.parametrize("fmt", ["lz4", "snappy"])
@pytest.mark.parametrize("large", [1, 147, 148, 149, 500])
def test_large_among_many(cuda, fmt, large):
    """Chunks of 256 KiB of capacity and more beside many small ones: up to one
    per SM go to wide CTAs, past that those of 512 KiB and more, and so on."""
    import torch
    n = 500
    raws = [r[:3000] for r in chunks(n)]
    rng = random.Random(large)
    caps = [len(r) for r in raws]
    for j, i in enumerate(rng.sample(range(n), large)):
        caps[i] = (262144, 262145, 524287, 524288, 1 << 20)[j % 5]
        if j < 3:
            raws[i] = W.generate([caps[i]], W.lz_params(0.5), seeds=[j])[0].tobytes()
    comps = [PACK[fmt](r) for r in raws]
    b = bytearray(comps[7])
    b[len(b) // 2] ^= 4
    comps[7] = bytes(b)
    b = DeviceBatch(comps, caps, device=cuda, dst_align=16, dst_skew=3, src_skew=5)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    for _ in range(2):
        assert b.run(fmt, stream) == 0
    stream.synchronize()
    res, dst = b.results(), b.dst_host()
    for i in range(n):
        st, out = WANT[fmt](comps[i], caps[i])
        assert res[i]["status"] == st, (i, res[i], st)
        if st == 0:
            assert res[i]["bytes_written"] == len(out)
            assert b.output(i, dst) == out + b"\xa5" * (caps[i] - len(out)), i


def test_large_among_many_captured(cuda):
    import torch
    raws = [r[:3000] for r in chunks(450)]
    raws[33] = W.generate([300000], W.lz_params(0.5), seeds=[1])[0].tobytes()
    b = DeviceBatch([PACK["lz4"](r) for r in raws], [len(r) for r in raws], device=cuda)
    assert b.run("lz4") == 0
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert b.run("lz4") == 0
    b.d_dst.zero_()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    dst = b.dst_host()
    assert (b.results()["status"] == 0).all()
    for i, r in enumerate(raws):
        assert b.output(i, dst) == r, i


@pytest.mark.parametrize("fmt", ["lz4", "snappy"])
def test_generous_capacities(cuda, fmt):
    """Small pages in slots of 256 KiB: none of so many is large."""
    import torch
    n = 1500
    raws = [r[:2000 + i % 999] for i, r in enumerate(chunks(n))]
    comps = [PACK[fmt](r) for r in raws]
    b = DeviceBatch(comps, [262144] * n, device=cuda, dst_align=16, dst_skew=3, src_skew=5)
    assert b.run(fmt) == 0
    torch.cuda.synchronize()
    res = b.results()
    assert (res["status"] == 0).all()
    assert [int(v) for v in res["bytes_written"]] == [len(r) for r in raws]
    dst = b.dst_host()
    for i, r in enumerate(raws):
        assert b.output(i, dst, len(r) + 64) == r + b"\xa5" * 64, i
