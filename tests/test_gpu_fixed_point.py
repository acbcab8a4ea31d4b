"""The fixed-point transforms of the FP64 engine's passes, at the shapes where they can go wrong: every
radix first and not first, transforms of one stage and of the longest rows, the lengths from which
values are scaled once more on the way, each column-group width, long columns in a batch; against
Python integers, with a round-off no larger than the double-precision oracle's on the same input."""
import random

import pytest

pytestmark = pytest.mark.gpu

# k, L, R, G: rows of C = L / 2 / R points, columns of R points
SHAPES = [(3, 64, 2, 8), (9357, 448, 4, 8), (5, 960, 3, 8), (7, 1120, 7, 8), (9999, 1344, 12, 4), (11, 2240, 5, 8),
          (8191, 5376, 14, 2), (3, 6144, 192, 8), (9357, 28672, 56, 2), (9001, 49152, 96, 4), (187, 11760, 49, 8),
          (5, 60000, 75, 8), (3, 65536, 1024, 2), (9357, 65536, 16, 8), (21, 98304, 32, 2), (3, 81920, 512, 8)]


def _n(L, k):
    from ahnum_gb300.tune import safe_bpw
    import math
    return int(L * (safe_bpw(L, k) if L >= 1024 else 21.24 - 0.5 * math.log2(k) - 2))


def _mod(v, k, n):
    """v mod k*2^n-1 for v >= 0, by k*2^n == 1 (Python's own division is quadratic)"""
    while v >> n >= k:
        q, r = divmod(v >> n, k)
        v = (v & ((1 << n) - 1)) + q + (r << n)
    return v - (k << n) + 1 if v >= (k << n) - 1 else v


@pytest.mark.parametrize("k,L,R,G", SHAPES)
def test_shape_against_integers(lib, oracle_mod, k, L, R, G):
    from ahnum_gb300.kite import Ctx
    n = _n(L, k)
    assert lib.kc_set_latency_shape(L, R, G) == 0
    rng = random.Random(L)
    try:
        with Ctx(k, n, L) as c, oracle_mod.OracleCtx(k, n, L) as o:
            N = c.N
            a, b = rng.randrange(N), rng.randrange(N)
            x, y = c.num(a), c.num(b)
            assert c.get(x) == a
            # a square, a product, a sum squared, a product of numbers of very different size, zero
            c.square(x, 3)
            t = a
            for _ in range(3):
                t = _mod(t * t, k, n)
            assert c.get(x) == t
            c.mul(x, y)
            t = _mod(t * b, k, n)
            assert c.get(x) == t
            c.add(x, y)
            c.square(x)
            t = _mod((t + b) ** 2, k, n)
            assert c.get(x) == t
            small = c.num(3)
            c.mul(small, x)
            assert c.get(small) == _mod(3 * t, k, n)
            zero = c.num(0)
            c.square(zero, 2)
            assert c.get(zero) == 0
            c.mul(zero, y)
            assert c.get(zero) == 0
            # round-off: the largest of eight squarings of the same number, engine and oracle
            x, ox = c.num(a), o.num(a)
            c.reset_maxerr()
            o.reset_maxerr()
            c.square(x, 8)
            o.square(ox, 8)
            assert c.get(x) == o.get(ox)
            assert c.maxerr() <= o.maxerr()
    finally:
        lib.kc_set_latency_shape(L, 0, 0)


def test_batch_with_long_columns(lib):
    """a slot whose columns take groups of 4 (1024 rows) beside one with groups of 8"""
    from ahnum_gb300.kite import Batch
    import ctypes as C
    k, n, L = 3, 1100000, 65536
    assert lib.kc_set_fft_shape(L, 1024) == 0
    try:
        with Batch(gerbicz_block=20) as b:
            slots = [(b.add_fermat(k, n, 3, L), k, n), (b.add_fermat(9357, 20000), 9357, 20000)]
            assert all(s[0] >= 0 for s in slots)
            for _ in range(2):
                b.step(1)
            for s, kk, nn in slots:
                arr = (C.c_uint64 * ((nn + 127) // 64))()
                assert lib.kc_batch_read(b.h, s, arr) == 0
                v = sum(int(w) << (64 * i) for i, w in enumerate(arr))
                t = 3**kk
                for _ in range(40):
                    t = _mod(t * t, kk, nn)
                assert v == t
                assert 0 < b.result(s)[1].maxerr < 0.4
    finally:
        lib.kc_set_fft_shape(L, 0)
