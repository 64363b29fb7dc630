"""The allocation-free class map at the edges of its tiles (GPU): ranges from
one block to class arrays of one, two, a tile's and a few tiles' units of 2^16
bits, every word against a plain numpy sieve."""
import ctypes as C

import numpy as np
import pytest

import gbc

pytestmark = pytest.mark.gpu

U30 = (1, 7, 11, 13, 17, 19, 23, 29)
UNIT = 1 << 16


def sieve(lo, hi):
    s = np.ones(hi - lo, dtype=bool)
    s[lo % 2::2] = False
    for p in range(3, int(hi ** 0.5) + 1, 2):
        if all(p % d for d in range(3, int(p ** 0.5) + 1, 2)):
            s[max(p * p, -(-lo // p) * p) - lo::p] = False
    if lo <= 2 < hi:
        s[2 - lo] = True
    s[:max(0, min(2, hi) - lo)] = False
    return s


@pytest.mark.parametrize("q_lo,blocks", [(0, 1), (7, 64), (10**8 + 11, 1), (10**8, UNIT - 64), (10**8 + 29, UNIT - 63),
                                         (10**8, 2 * UNIT - 64), (10**9 + 1, 19 * UNIT + 5), (10**9, 28 * UNIT),
                                         (10**9 + 7, 61 * UNIT - 100)])
def test_map_against_numpy(q_lo, blocks):
    torch = pytest.importorskip("torch")
    base = q_lo // 30 * 30
    q_hi = base + 30 * blocks - 1
    ps = [p for p in range(3, max(int(q_hi ** 0.5) + 400, 80), 2)
          if all(p % d for d in range(3, int(p ** 0.5) + 1, 2))]
    primes = torch.tensor(ps, dtype=torch.int32, device="cuda")
    wpc = (blocks + 64 + UNIT - 1) // UNIT * (UNIT // 32)
    m = torch.full((8 * wpc,), -1, dtype=torch.int32, device="cuda")
    b, nblk, w, err = C.c_uint64(), C.c_uint32(), C.c_uint32(), C.create_string_buffer(256)
    rc = gbc.load().gbc_class_map_noalloc(q_lo, q_hi, primes.data_ptr(), len(ps), ps[-1], m.data_ptr(), m.numel(),
                                          C.byref(b), C.byref(nblk), C.byref(w),
                                          torch.cuda.current_stream().cuda_stream, err, len(err))
    assert rc == 0, err.value
    torch.cuda.synchronize()
    assert (b.value, nblk.value, w.value) == (base, blocks, wpc)
    s = sieve(base, base + 30 * blocks)
    want = np.zeros((8, 4 * wpc), dtype=np.uint8)
    for k, u in enumerate(U30):
        bits = np.packbits(s[u::30], bitorder="little")
        want[k, :len(bits)] = bits
    assert np.array_equal(m.cpu().numpy(), want.reshape(-1).view(np.int32))
