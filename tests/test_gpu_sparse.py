"""Numbers with few digits other than zero, as every test starts from: a single digit gives rows and
columns of one modulus, whose inverse transform gathers everything on one element.  Transforms of every
length whose values then reach 2^61 before they are scaled up on the way, as rows and as columns, in a
single test and in a batch; and the lengths on either side, whose last stages grow most (686), or which
are not scaled on the way (343, 256); against Python integers."""
import ctypes as C
import random

import pytest

pytestmark = pytest.mark.gpu

REACH = [288, 315, 320, 420, 525, 560, 640, 672, 700, 1120, 1152, 1280, 1440, 1575]
OTHERS = [256, 343, 350, 490, 512, 686, 1024]
# (L, R, G): the length as columns of R points beside rows of 16, or as rows beside columns of 16
SHAPES = [(32 * n, n, g) for n in REACH + OTHERS if n <= 896 for g in (2, 8)]
SHAPES += [(32 * n, n, 4) for n in (1024,)]
SHAPES += [(32 * n, 16, 8) for n in REACH + OTHERS + [1536, 2048] if n % 8 == 0]
# bits a digit: numbers like 2^(n/2) are k times a periodic pattern, whose spectrum is a few lines; their
# products need some 5 bits more room than random ones (3 with k = 1, where they are sparse)
KS = {1: 17, 3: 14, 9357: 11}


def _mod(v, k, n):
    """v mod k*2^n-1 for v >= 0, by k*2^n == 1"""
    while v >> n >= k:
        q, r = divmod(v >> n, k)
        v = (v & ((1 << n) - 1)) + q + (r << n)
    return v - (k << n) + 1 if v >= (k << n) - 1 else v


def _lucas(P, m, k, n):
    """V_m(P, -1) mod N and V_(m+1)"""
    N = (k << n) - 1
    a, b, i = 2, P, 0
    for bit in bin(m)[2:]:
        s = -1 if i & 1 else 1  # (-1)^i
        mid = (a * b - s * P) % N
        if bit == "1":
            a, b, i = mid, (b * b + 2 * s) % N, 2 * i + 1
        else:
            a, b, i = (a * a - 2 * s) % N, mid, 2 * i
    return a, b


def _numbers(k, n):
    return [0, 1, 2, 3, 5, 11, 25, 81, 100, 243, k, 7 * k, 243 * k, 3**k, 1 << (n // 2), (1 << (n // 2)) + (1 << (n // 2 + 18)),
            1 << (n - 3), (1 << n) - 1, (k << n) - 2, _lucas(3, k, k, n)[0], _lucas(5, k, k, n)[0]]


@pytest.mark.parametrize("L,R,G", SHAPES)
def test_sparse_numbers(lib, L, R, G):
    from ahnum_gb300.kite import Ctx
    assert lib.kc_set_latency_shape(L, R, G) == 0
    wrong = []
    try:
        for k in KS:
            n = KS[k] * L
            rng = random.Random(L + k)
            dense = rng.getrandbits(n - 1)
            with Ctx(k, n, L) as c:
                d = c.num(dense)
                for i, v in enumerate(_numbers(k, n)):
                    v = _mod(v, k, n)
                    x = c.num(v)
                    got, want = [c.get(x)], [v]
                    c.mul(x, d)
                    got.append(c.get(x))
                    want.append(_mod(v * dense, k, n))
                    c.set(x, v)
                    for _ in range(3):
                        c.square(x)
                        v = _mod(v * v, k, n)
                        got.append(c.get(x))
                        want.append(v)
                    if got != want:
                        wrong.append((k, i, [g == w for g, w in zip(got, want)]))
                    x.free()
    finally:
        lib.kc_set_latency_shape(L, 0, 0)
    assert not wrong


@pytest.mark.parametrize("L,R", [(L, R) for L, R, G in SHAPES if G != 2])
def test_starts_in_a_batch(lib, L, R):
    """Fermat starts 3^k, 5^k, 11^k, 25^k and LLR starts V_k(P), squared as a block of 2, and of 3"""
    from ahnum_gb300.kite import Batch
    assert lib.kc_set_fft_shape(L, R) == 0
    wrong = []
    try:
        for block in (2, 3):
            with Batch(gerbicz_block=block, gerbicz_blocks=1 << 20) as b:
                tests = [(k, KS[k] * L + 1, base) for k in KS for base in (3, 5, 11, 25)]
                tests += [(k, 11 * L + 1, 0) for k in (5, 27, 4501)]
                slots = []
                for k, n, base in tests:
                    slots.append(b.add_fermat(k, n, base, L) if base else b.add_llr(k, n, L))
                b.step(1)
                for slot, (k, n, base) in zip(slots, tests):
                    P, factor = C.c_uint32(), C.c_uint64()
                    if not base:
                        lib.kite_llr_choose_P(k, n, C.byref(P), C.byref(factor))
                        if factor.value:
                            continue
                    assert slot >= 0
                    a = (C.c_uint64 * ((n + 127) // 64))()
                    assert lib.kc_batch_read(b.h, slot, a) == 0
                    v = base**k if base else _lucas(P.value, k, k, n)[0] ** 2 + 2
                    for _ in range(block):
                        v = _mod(v, k, n) ** 2 - (0 if base else 2)
                    if int.from_bytes(bytes(a), "little") != _mod(v, k, n):
                        wrong.append((k, base, block))
    finally:
        lib.kc_set_fft_shape(L, 0)
    assert not wrong


# lengths that the library takes by itself, at its own shape: the first squarings of a test
@pytest.mark.parametrize("k,n", [(4501, 2131199), (9357, 4166751), (3, 6090515), (1, 2976221), (3, 11484018), (9999, 8000000),
                                 (9357, 15900000)])
def test_start_of_a_test(lib, k, n):
    from ahnum_gb300.kite import Ctx
    with Ctx(k, n) as c:
        for v in (3**k, 1, 81, _lucas(3, k, k, n)[0]):
            x = c.num(v)
            assert c.get(x) == v
            for _ in range(4):
                c.square(x)
                v = _mod(v * v, k, n)
                assert c.get(x) == v
            x.free()
