"""The content checksum of large frames, hashed while their parts are copied
back: sizes around two parts of 4 MiB, compressed and raw blocks in any order,
lengths that are no multiple of a stripe, flipped checksums and contents.
"""
import numpy as np
import pytest

import cudec_b200 as cd
import oracle
from cudec_b200 import workload as W

pytestmark = pytest.mark.gpu

PART = 4 << 20


def content(n, raw):
    d = W.generate([n], W.lz_params(0.5), seeds=np.array([n], dtype=np.uint64))[0][:n].copy()
    rng = np.random.default_rng(n)
    for at in raw:  # incompressible stretches make raw blocks
        m = min(500000, n - at)
        d[at:at + m] = rng.integers(0, 256, m, dtype=np.uint8)
    return d.tobytes()


@pytest.mark.parametrize("n", [2 * PART - 1, 2 * PART, 2 * PART + 17, 3 * PART + 3])
@pytest.mark.parametrize("raw", [(), (0, 1 << 20, 7 << 20)])
@pytest.mark.parametrize("block", [4, 7])
def test_content_checksum(cuda, n, raw, block):
    d = content(n, raw)
    f = W.lz4f_compress(d, block_size_id=block, content_checksum=True)
    assert cd.lz4f_decompress(f, n) == (0, d)
    for at in (len(f) - 1, len(f) - 4, len(f) - 9):
        g = bytearray(f)
        g[at] ^= 0x10
        want = oracle.lz4f_decode(bytes(g), n)
        got = cd.lz4f_decompress(bytes(g), n)
        assert got[0] == want[0], at
    assert cd.lz4f_decompress(f, n - 1)[0] == oracle.lz4f_decode(f, n - 1)[0]
