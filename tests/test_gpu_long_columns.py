"""Columns of more than 896 rows, whose groups of 8 do not fit shared memory: a single test asked for such
groups, or whose narrow digits used to need them, and batch slots with narrow digits and with a top
region of more than 8 digits; against Python integers."""
import ctypes as C
import random

import pytest

pytestmark = pytest.mark.gpu


def _mod(v, k, n):
    while v >> n >= k:
        q, r = divmod(v >> n, k)
        v = (v & ((1 << n) - 1)) + q + (r << n)
    return v - (k << n) + 1 if v >= (k << n) - 1 else v


# 10 bits a digit, 5 and 4, and a length whose columns are all so long
@pytest.mark.parametrize("k,n,L,R", [(9357, 700000, 65536, 1024), (187, 340000, 65536, 1024), (3, 280000, 65536, 1024),
                                     (21, 320000, 32000, 1000), (187, 24715281, 4194304, 0)])
def test_single(lib, k, n, L, R):
    from ahnum_gb300.kite import Ctx
    assert R == 0 or lib.kc_set_latency_shape(L, R, 8) == 0
    try:
        rng = random.Random(n)
        a, b = rng.getrandbits(n - 1), rng.getrandbits(n - 1)
        with Ctx(k, n, L) as c:
            x, y = c.num(a), c.num(b)
            assert c.get(x) == a
            if n < 10**7:  # Python's products of the longest numbers take seconds
                c.square(x, 2)
                a = _mod(_mod(a * a, k, n)**2, k, n)
            c.mul(x, y)
            assert c.get(x) == _mod(a * b, k, n)
            assert c.maxerr() < 0.4
    finally:
        lib.kc_set_latency_shape(L, 0, 0)


@pytest.mark.parametrize("k,n,L,R", [(9357, 700000, 65536, 1024), (3, 131000, 65536, 1024), (2**30 - 1, 235000, 65536, 1024),
                                     (2**30 - 1, 235000, 65536, 256)])
def test_batch_slot(lib, k, n, L, R):
    from ahnum_gb300.kite import Batch
    block = 5
    assert lib.kc_set_fft_shape(L, R) == 0
    try:
        with Batch(gerbicz_block=block, gerbicz_blocks=1 << 20) as b:
            slot = b.add_fermat(k, n, 3, L)
            assert slot >= 0
            b.step(3)
            a = (C.c_uint64 * ((n + 127) // 64))()
            assert lib.kc_batch_read(b.h, slot, a) == 0
            v = 1
            for bit in bin(k)[2:]:
                v = _mod(v * v * (3 if bit == "1" else 1), k, n)
            for _ in range(3 * block):
                v = _mod(v * v, k, n)
            assert int.from_bytes(bytes(a), "little") == v
            assert b.result(slot)[1].maxerr < 0.4
    finally:
        lib.kc_set_fft_shape(L, 0)
