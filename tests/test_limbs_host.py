"""Digits to canonical limbs on the host, one pass with a two's-complement sum: against Python integers
at the sizes where it can go wrong (n a multiple of 64 and not, k = 1 and the largest, digits of every
size and sign up to the ends of 64 bits), and back."""
import ctypes as C
import random

import pytest


@pytest.mark.parametrize("k", [1, 3, 9357, 2**30 - 1])
@pytest.mark.parametrize("n,L", [(16, 16), (64, 16), (65, 32), (127, 64), (128, 96), (1000, 64), (4096, 448), (4099, 320)])
def test_digits_to_limbs(lib, k, n, L):
    rng = random.Random(n * L + k)
    bits, w, o, meta = (C.c_uint8 * L)(), (C.c_double * L)(), (C.c_double * L)(), (C.c_uint64 * 8)()
    assert lib.kc_layout(k, n, L, bits, w, o, meta) == 0
    N, nl = k * 2**n - 1, (n + 127) // 64
    out = (C.c_uint64 * nl)()
    cases = [[0] * L, [-1] + [0] * (L - 1), [1] * L, [-(2**63)] * L, [2**63 - 1] * L, [0] * (L - 1) + [-(2**63)]]
    cases += [[rng.randrange(-2**m, 2**m) for _ in range(L)] for m in (1, 8, 20, 40, 51, 63)]
    for d in cases:
        assert lib.kc_digits_to_limbs(k, n, L, (C.c_int64 * L)(*d), out) == 0
        total, s = 0, 0
        for j in range(L):
            total += d[j] << s
            s += bits[j]
        assert sum(int(v) << (64 * i) for i, v in enumerate(out)) == k * total % N
    dd = (C.c_int64 * L)()
    for x in (0, 1, N - 1, rng.randrange(N)):
        limbs = (C.c_uint64 * nl)(*[(x >> (64 * i)) & (2**64 - 1) for i in range(nl)])
        assert lib.kc_limbs_to_digits(k, n, L, limbs, dd) == 0
        assert lib.kc_digits_to_limbs(k, n, L, dd, out) == 0
        assert sum(int(v) << (64 * i) for i, v in enumerate(out)) == x
