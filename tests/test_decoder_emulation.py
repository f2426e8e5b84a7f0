"""The decoders' device source, run on the CPU.

tests/native/cuda_emul.h runs a CTA's threads as fibers that meet at warp
collectives and barriers (a deadlock, lanes at different collectives, or
threads that disagree on the result fail the run), in an order drawn from a
seed, or with one warp held back until no other can run. The sizes are those where the decoders change their way: LZ4 and Snappy
chunks of one tile and of several at each width of the CTA, batches cut by
long tokens, tiles that few tokens settle; Zstd frames of no, one and more
than one item of 128 sequences, one and several blocks, literal streams shared
by eight lanes or not, runs longer than a lane's own copies; short GDeflate
pages and full ones. Statuses, bytes and untouched memory around them equal
the oracle's; the mutants cover the early ends.
"""
import ctypes
import os
import random
import subprocess

import numpy as np
import pytest

import oracle
from cudec_b200 import workload as W
from lz_blocks import lz4_block, snappy_block

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "cudec_b200", "csrc")


def _build(name):
    out_dir = os.path.join(HERE, "native", "_build")
    os.makedirs(out_dir, exist_ok=True)
    so = os.path.join(out_dir, "lib%s.so" % name)
    src = os.path.join(HERE, "native", name + ".cpp")
    deps = [src, os.path.join(HERE, "native", "cuda_emul.h")] + [
        os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    if not os.path.exists(so) or any(os.path.getmtime(d) > os.path.getmtime(so) for d in deps):
        subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-w",
                        "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, src,
                        "-o", so + ".%d" % os.getpid()], check=True)
        os.replace(so + ".%d" % os.getpid(), so)  # whole, for workers that build at once
    return ctypes.CDLL(so)


@pytest.fixture(scope="module")
def lz():
    lib = _build("lz_emul")
    lib.lz_emulate.argtypes = [ctypes.c_int, ctypes.c_uint32, ctypes.c_void_p, ctypes.c_uint64,
                               ctypes.c_void_p, ctypes.c_uint64, ctypes.c_uint64,
                               ctypes.POINTER(ctypes.c_uint64)]
    lib.lz_ldgs.restype = ctypes.c_uint64
    lib.lz_large.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_uint32, ctypes.c_uint64,
                             ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t,
                             ctypes.c_void_p, ctypes.POINTER(ctypes.c_uint64)]

    def call(fmt, threads):
        return lambda src, n, dst, cap, seed, written: lib.lz_emulate(
            fmt, threads, src, n, dst, cap, seed, written)
    call.lib = lib
    return call


@pytest.fixture(scope="module")
def zstd():
    lib = _build("zstd_emul")
    lib.zstd_emulate.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p,
                                 ctypes.c_uint64, ctypes.c_void_p, ctypes.c_uint64,
                                 ctypes.POINTER(ctypes.c_uint64)]
    slot = np.zeros(128 * 1024, dtype=np.uint8)

    def call(multi):
        def run(src, n, dst, cap, seed, written):
            slot[:] = 0xEE
            return lib.zstd_emulate(multi, src, n, dst, cap, slot.ctypes.data, seed, written)
        return run
    return {"one": call(0), "multi": call(1)}


@pytest.fixture(scope="module")
def gdeflate():
    lib = _build("gdeflate_emul")
    lib.gdeflate_emulate.argtypes = [ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p,
                                     ctypes.c_uint64, ctypes.c_uint64,
                                     ctypes.POINTER(ctypes.c_uint64)]
    return lib.gdeflate_emulate


def starving(order, warp):
    """The seed of order `order` that holds warp `warp` back."""
    return order | (warp + 1) << 8


# What the checks above rest on: two warps of code with a barrier each way.
@pytest.mark.parametrize("kind,why", [
    (0, None), (1, "a thread meets a barrier twice before it completes"),
    (2, "threads state different counts for a barrier"), (3, "deadlock"),
    (4, "lanes of a warp at different collectives")])
def test_emulation(kind, why):
    lib = _build("emul_check")
    lib.emul_check.restype = ctypes.c_char_p
    lib.emul_check.argtypes = [ctypes.c_int, ctypes.c_uint64]
    found = {lib.emul_check(kind, seed) for order in range(8)
             for seed in (order, starving(order, 0), starving(order, 1))}
    assert found == {None} if why is None else why.encode() in found


def check(run, want, comp, cap, seed=0, skew=0, label=None):
    src = np.zeros(len(comp) + 64 + skew, dtype=np.uint8)
    src[32 + skew:32 + skew + len(comp)] = np.frombuffer(comp, dtype=np.uint8)
    dst = np.full(cap + 96, 0xA5, dtype=np.uint8)
    o = 32 + (skew * 7) % 32
    w = ctypes.c_uint64(0)
    st = run(src.ctypes.data + 32 + skew, len(comp), dst.ctypes.data + o, cap, seed,
             ctypes.byref(w))
    want_st, want_out = want(comp, cap)
    assert st == want_st, (label, st, want_st, len(comp), cap, seed)
    assert (dst[:o] == 0xA5).all() and (dst[o + cap:] == 0xA5).all(), (label, "out of bounds")
    if st == 0:
        assert dst[o:o + w.value].tobytes() == want_out, (label, "bytes differ")
        assert (dst[o + w.value:o + cap] == 0xA5).all(), (label, "wrote past bytes_written")


def mutate(rng, comp):
    b = bytearray(comp)
    for _ in range(rng.randrange(1, 4)):
        r = rng.random()
        if r < 0.75:
            b[rng.randrange(len(b))] ^= 1 << rng.randrange(8)
        elif r < 0.9:
            b = b[:rng.randrange(1, len(b) + 1)]
        else:
            b += rng.randbytes(rng.randrange(1, 5))
    return bytes(b)


def contents(size):
    rng = random.Random(size)
    yield W.generate([max(size, 1)], W.zstd_params(), seeds=[size])[0][:size].tobytes()
    yield bytes(size)
    yield rng.randbytes(size)
    yield (b"the quick brown fox jumps over the lazy dog; " * (size // 45 + 1))[:size]
    # long runs of either kind between short ones
    parts = [rng.randbytes(rng.randrange(1, 2500)) + b"x" * rng.randrange(1, 2500)
             for _ in range(size // 2500 + 1)]
    yield (b"".join(parts) + parts[0] * 3)[:size]


def lz_contents(size):
    rng = random.Random(size)
    for p in (0.1, 0.5, 0.9):
        yield W.generate([max(size, 1)], W.lz_params(p), seeds=[size])[0][:size].tobytes()
    words = [rng.randbytes(rng.randrange(3, 12)) for _ in range(200)]
    yield b"".join(rng.choice(words) for _ in range(size // 5 + 1))[:size]


# One tile holds 52 positions per thread.
@pytest.mark.parametrize("threads", [128, 256, 512])
@pytest.mark.parametrize("size", [0, 1, 13, 129, 1025, 6656, 30000])
def test_lz(lz, size, threads):
    rng = random.Random(size)
    datas = list(lz_contents(size)) + list(contents(size))[1:]
    for k, data in enumerate(datas):
        for fmt, pack, want in ((0, W.lz4_compress, oracle.lz4_decode),
                                (1, W.snappy_compress, oracle.snappy_decode)):
            f = pack(data)
            late = rng.randrange(threads // 32)
            check(lz(fmt, threads), want, f, size, starving(k + 1, late), (5 * k + fmt) % 16,
                  (size, k, fmt))
            for m in range(4 if size < 6000 else 1):
                check(lz(fmt, threads), want, mutate(rng, f), size - (m % 2) * size // 2,
                      starving(m, late) if m % 2 else m, 0, (size, k, fmt, m))


def long_tokens(rng, n, share):
    """Sequences of which `share` are longer than 1,024 bytes, by literals or by
    a match from near or far; runs of the others longer than a window."""
    seqs, total = [], 0
    for _ in range(n):
        lit, ml, off = rng.randbytes(rng.randrange(0, 40)), rng.randrange(4, 60), None
        if rng.random() < share:
            size = rng.choice([985, 1024, 1025, 1500, 4000])
            if rng.random() < 0.3:
                lit = rng.randbytes(size)
            else:
                ml = size
        if not seqs:
            lit = rng.randbytes(50)
        total += len(lit)
        off = rng.choice([1, 3, 31, 2000, 5000, 9000, 60000])
        seqs.append((lit, min(off, total, 65535), ml))
        total += ml
    return seqs


# Long tokens one after the other, at a batch's ends and between runs that fill
# more than a window of output.
@pytest.mark.parametrize("threads", [128, 512])
@pytest.mark.parametrize("share", [0.02, 0.1, 1.0])
def test_lz_long_tokens(lz, threads, share):
    rng = random.Random(share)
    for k in range(2):
        n = (130, 600)[k] if share < 0.1 else 40
        seqs = long_tokens(rng, n, share)
        for fmt, pack, want in ((0, lz4_block, oracle.lz4_decode),
                                (1, snappy_block, oracle.snappy_decode)):
            comp = pack(seqs, rng.randbytes((20, 1500)[k]))
            cap = sum(len(lit) + ml for lit, _, ml in seqs) + (20, 1500)[k]
            assert want(comp, cap)[0] == 0
            seed = starving(k, rng.randrange(threads // 32))
            check(lz(fmt, threads), want, comp, cap, seed, (5 * k + fmt) % 16, (share, k, fmt))
            check(lz(fmt, threads), want, mutate(rng, comp), cap, seed, 3, (share, k, fmt, "m"))


def test_lz_long_tokens_share_a_batch(lz):
    # literals and a match each cost a barrier; a batch of its own for every
    # long token was two more
    seqs = [(b"0123456789" * 200, 5000 if i > 5 else 7, 1500) for i in range(30)]
    comp, cap = lz4_block(seqs, bytes(20)), 30 * 3500 + 20
    check(lz(0, 512), oracle.lz4_decode, comp, cap, 1)
    many = lz.lib.lz_barriers()
    comp, cap = lz4_block(seqs[:10], bytes(20)), 10 * 3500 + 20
    check(lz(0, 512), oracle.lz4_decode, comp, cap, 1)
    assert many - lz.lib.lz_barriers() <= 20 * 2 + 40  # and the tiles of 40,000 bytes more


def test_lz_passes_over_a_long_token(lz):
    # 12,000 bytes of extension, some 4,800 of them past the staged input: walked
    # on the chain, in the list, by the ladder and for the copy
    comp = lz4_block([(b"abc", 3, 255 * 12000)], bytes(13))
    check(lz(0, 128), oracle.lz4_decode, comp, 255 * 12000 + 16, 1)
    assert lz.lib.lz_ldgs() < 4.5 * (12000 - 128 * 52 - 512)


def capacities(kind, n):
    rng = random.Random(kind)
    if kind == "alike":
        return [1 << 20] * n
    if kind == "none":
        return [(1 << 18) - 1] * n
    if kind == "at the end":
        return [4096] * (n - n // 2) + [1 << 18] * (n // 2)
    if kind == "few":
        return [rng.choice([1 << 18, 1 << 40, 2**64 - 1]) if i % 211 == 5 else 100
                for i in range(n)]
    return [int(2 ** rng.uniform(10, 23 if kind == "uneven" else 45)) for _ in range(n)]


# Which chunks of a batch a wide CTA takes: those of a size class that holds,
# with the ones above it, no more of them than there are wide CTAs. The wide
# and the narrow CTAs come to the same answer, and the narrow ones read a
# bounded number of capacities for it, not the batch's for each chunk.
@pytest.mark.parametrize("kind", ["alike", "none", "at the end", "few", "uneven", "very uneven"])
@pytest.mark.parametrize("n,wide", [(445, 148), (2000, 148), (2000, 5)])
def test_lz_large_chunks(lz, kind, n, wide):
    caps = capacities(kind, n)
    level = [min(max(c.bit_length() - 18, 0), 16) for c in caps]
    first = next((k for k in range(1, 17) if sum(v >= k for v in level) <= wide), 17)
    want = [i for i in range(n) if level[i] >= first]
    arr = np.array(caps, dtype=np.uint64)
    ask = [i for i in range(n) if level[i]]
    if len(ask) > 150:  # every large one among them
        ask = sorted(set(random.Random(n).sample(ask, 150)) | set(want))
    ask = np.array(ask, dtype=np.uint64)
    chunk = np.zeros(wide, dtype=np.uint64)
    count, reads = ctypes.c_uint32(0), ctypes.c_uint64(0)
    large = np.zeros(max(len(ask), 1), dtype=np.uint8)
    assert lz.lib.lz_large(arr.ctypes.data, n, wide, starving(n % 250, wide % 4),
                           chunk.ctypes.data, ctypes.addressof(count), ask.ctypes.data, len(ask),
                           large.ctypes.data, ctypes.byref(reads)) == 0
    assert sorted(chunk[:count.value].tolist()) == want
    assert [int(i) for i, v in zip(ask, large) if v] == want
    # the CTA's first step and the chunk's own capacity, then what a class reads together
    together = 0 if kind == "alike" else 2 * (wide + 1) * n * len(set(level))
    assert reads.value <= 3 * 128 * len(ask) + together


@pytest.mark.parametrize("size", [0, 1, 40, 1000, 1600, 9000, 131072, 150000])
def test_zstd(zstd, size):
    for k, data in enumerate(contents(size)):
        for level in (1, 19):
            f = W.zstd_compress(data, level, 20, level == 19)
            check(zstd["one"], oracle.zstd_decode, f, size,
                  starving(k, (k + size) % 6) if level == 1 else k, (5 * k + level) % 16,
                  (size, k, level))
    check(zstd["one"], oracle.zstd_decode, f, size + 9, 3, 1, (size, "room"))


# Literals and little else: streams that end anywhere in a window of five
# symbols, and around the length from which eight lanes share one.
def test_zstd_literals(zstd):
    rng = random.Random(3)
    for size in list(range(64, 96)) + list(range(1700, 1712)) + [5000, 5003, 20001]:
        data = bytes(min(int(rng.expovariate(0.2)), 255) for _ in range(size))
        f = W.zstd_compress(data, 1, 20, False)
        check(zstd["one"], oracle.zstd_decode, f, size, size % 251, size % 16, size)
        for k in range(2):
            check(zstd["one"], oracle.zstd_decode, mutate(rng, f), size, k, 0, (size, k))


def test_zstd_mutants(zstd):
    rng = random.Random(11)
    frames = [(W.zstd_compress(d, lv, 20, True), size) for size in (300, 4000, 140000)
              for lv in (1, 19) for d in contents(size)]
    for k in range(240):
        f, cap = frames[k % len(frames)]
        if cap > 100000 and k % 3:
            continue
        cut = rng.choice([0, 0, 1, cap // 2])
        seed = starving(k, rng.randrange(6))
        check(zstd["one"], oracle.zstd_decode, mutate(rng, f), cap - cut, seed, k % 16, k)
        if k % 5 == 0:
            two = f + b"\x50\x2a\x4d\x18\x03\x00\x00\x00abc" + mutate(rng, frames[0][0])
            check(zstd["multi"], oracle.zstd_decode_multi, two, 2 * cap, seed, 0, ("multi", k))


def block(kind, body, size=None, last=False):
    n = len(body) if size is None else size
    return (n << 3 | kind << 1 | last).to_bytes(3, "little") + body


RAW, RLE, COMPRESSED, RESERVED = range(4)
# blocks that decode, of few bytes or none
SMALL = [block(RAW, b"abcd"), block(RAW, b""), block(RLE, b"x", 9), block(RLE, b"x", 0),
         block(COMPRESSED, b"\x18abc\x00")]  # three raw literals, no sequences
# blocks that do not, by the part of the decoder that finds it
FAULTY = {
    "reserved type": block(RESERVED, b""),
    "past the frame": block(RAW, b"ab", 70),
    "no header": b"",
    "no literals header": block(COMPRESSED, b""),
    "literals past the block": block(COMPRESSED, b"\x28ab"),
    "no sequences header": block(COMPRESSED, b"\x18abc"),
    "literals without a table": block(COMPRESSED, b"\x43\xc0\x00zzz\x00"),
    "literals with a bad table": block(COMPRESSED, b"\x42\xc0\x00\xff\x00\x00\x00"),
    "reserved modes": block(COMPRESSED, b"\x18abc\x01\x03\x80"),
    "no sequence table to repeat": block(COMPRESSED, b"\x18abc\x01\xfc\x80"),
    "a code past the last": block(COMPRESSED, b"\x18abc\x01\x40\x3f\x80"),
    "no bitstream": block(COMPRESSED, b"\x18abc\x01\x00"),
    "no padding marker": block(COMPRESSED, b"\x18abc\x01\x00\x00"),
    "bitstream over-read": block(COMPRESSED, b"\x18abc\x01\x00\xff\xff\x07"),
    "an offset past the output": block(COMPRESSED, b"\x18abc\x01\x54\x03\x1f\x00" + b"\xff" * 4),
}


# A fault that ends the frame in its first, second or a later block, with each
# of the six warps as far behind the others as their barriers let it be.
@pytest.mark.parametrize("fault", FAULTY)
def test_zstd_faulty_block(zstd, fault):
    rng = random.Random(fault)
    head = b"\x28\xb5\x2f\xfd\xa0" + (64).to_bytes(4, "little")
    for before in range(4):
        for _ in range(2):
            f = head + b"".join(rng.choice(SMALL) for _ in range(before)) + FAULTY[fault]
            if fault != "no header" and rng.random() < 0.5:
                f += rng.choice(SMALL)
            assert oracle.zstd_decode(f, 64)[0] == 2
            for warp in range(6):
                seed = starving(rng.randrange(256), warp)
                check(zstd["one"], oracle.zstd_decode, f, 64, seed, 0, (f, warp))
                check(zstd["multi"], oracle.zstd_decode_multi, f, 64, seed, 0, (f, warp))


@pytest.mark.parametrize("size", [0, 1, 63, 3000, 20000, 65536])
def test_gdeflate(gdeflate, size):
    rng = random.Random(size)
    pages = list(contents(size))
    pages.append(W.generate([max(size, 1)], W.gdeflate_params(0.8), seeds=[9])[0][:size].tobytes())
    for k, data in enumerate(pages):
        for level in (1, 12):
            f = W.gdeflate_compress(data, level)
            check(gdeflate, oracle.gdeflate_decode, f, size, k, (5 * k + level) % 16,
                  (size, k, level))
            for m in range(3 if size > 5000 else 12):
                check(gdeflate, oracle.gdeflate_decode, mutate(rng, f), size - (m % 2) * size // 2,
                      m, 0, (size, k, level, m))
