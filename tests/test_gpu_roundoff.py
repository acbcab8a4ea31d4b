"""The round-off of random numbers at the length's limit stays below what double-precision transforms had on
the same numbers (24 squarings and a product, largest difference to an integer): lengths whose rows or
columns take three and more odd radices, and digits of 4 bits (k near 2^30); and narrow digits' numbers are
right, read back and in a batch."""
import ctypes as C
import random

import pytest

pytestmark = pytest.mark.gpu

# k, n, L and the largest round-off of the double-precision passes at the same shape
ODD = [(9357, 9009432, 734832, 0.2339), (9357, 11747067, 967680, 0.1410), (9357, 10247149, 839808, 0.2006),
       (9357, 6435445, 518400, 0.1560), (9357, 7765093, 629856, 0.2611), (4501, 12072976, 952560, 0.1665)]
NARROW = [(999999937, 1569822, 373248, 0.3536), (999999937, 1744287, 419904, 0.3456),
          (999999937, 1438948, 338688, 0.2462), (999999937, 1382866, 324000, 0.2555)]


def _mod(v, k, n):
    while v >> n >= k:
        q, r = divmod(v >> n, k)
        v = (v & ((1 << n) - 1)) + q + (r << n)
    return v - (k << n) + 1 if v >= (k << n) - 1 else v


def _largest(k, n, L):
    from ahnum_gb300.kite import Ctx
    with Ctx(k, n, L) as c:
        x = c.num(random.Random(L).getrandbits(n - 1))
        c.reset_maxerr()
        c.square(x, 24)
        c.mul(x, x)
        return c.maxerr()


@pytest.mark.parametrize("k,n,L,double", ODD)
def test_odd_radices(lib, k, n, L, double):
    assert _largest(k, n, L) <= double


@pytest.mark.parametrize("k,n,L,double", NARROW)
def test_narrow_digits(lib, k, n, L, double):
    assert _largest(k, n, L) <= double


# Digits of 4 to 11 bits, k = 1 (no top region) and the largest
@pytest.mark.parametrize("k,n,L", [(1, 5400, 1344), (1, 6720, 1344), (3, 6720, 1344), (2**30 - 1, 9000, 2240), (2**25 - 39, 100001, 13440),
                                   (2**20 - 3, 60000, 6720), (187, 14000, 1344), (187, 13300, 1344), (999999937, 122000, 28672)])
def test_narrow_numbers(lib, k, n, L):
    from ahnum_gb300.kite import Batch, Ctx
    rng = random.Random(n)
    N = (k << n) - 1
    with Ctx(k, n, L) as c:
        patterns = [N // 3, (1 << n) - 1, 1 << (n // 2)]  # times a large k their products need more bits
        for v in [0, 1, 2, N - 1, rng.randrange(N), rng.randrange(N)] + (patterns if k < 1000 else []):
            v %= N
            x, y = c.num(v), c.num(N - 5)
            assert c.get(x) == v
            for count in (1, 2, 20):
                c.square(x, count)
                for _ in range(count):
                    v = _mod(v * v, k, n)
                assert c.get(x) == v
            c.mul(y, x)
            v = _mod(v * (N - 5), k, n)
            assert c.get(y) == v
            c.mul_small(y, 3)
            assert c.get(y) == _mod(3 * v, k, n)
            x.free()
            y.free()
    if L < 5000:
        with Batch(gerbicz_block=7) as b:
            slot = b.add_fermat(k, n, 3, L)
            assert slot >= 0
            b.step(2)
            a = (C.c_uint64 * ((n + 127) // 64))()
            assert lib.kc_batch_read(b.h, slot, a) == 0
            v = pow(3, k, N)
            for _ in range(14):
                v = _mod(v * v, k, n)
            assert int.from_bytes(bytes(a), "little") == v
