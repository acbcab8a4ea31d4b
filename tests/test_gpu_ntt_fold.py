"""Chains of the integer-NTT engine whose reduction runs inside the next squaring's column pass, and the
numbers read back through the GPU's own reduction, against Python integers: both sides of the smallest
n that takes that route, every column length, word boundaries at n (also where the
top word ends an eight), the extreme numbers, constants,
and groups of unequal members."""
import ctypes as C
import random

import pytest

pytestmark = pytest.mark.gpu


def _mod(v, k, n):
    """v mod N by k 2^n == 1"""
    N = k * (1 << n) - 1
    while v > N:
        q, r = divmod(v >> n, k)
        v = (v & ((1 << n) - 1)) + q + (r << n)
    return 0 if v == N else v


class _Engine:
    def __init__(self, k, n):
        from ahnum_gb300 import native
        self.lib, self.k, self.n = native.load(), k, n
        self.e = self.lib.kn_engine_new(k, n, -1)
        assert self.e
        self.x = self.lib.kn_num_alloc(self.e)
        self.nl = self.lib.kn_limbs(self.e)

    def set(self, v):
        a = (C.c_uint64 * self.nl)()
        C.memmove(a, v.to_bytes(8 * self.nl, "little"), 8 * self.nl)
        assert self.lib.kn_set_limbs(self.e, self.x, a) == 0

    def get(self):
        a = (C.c_uint64 * self.nl)()
        assert self.lib.kn_get_limbs(self.e, self.x, a) == 0
        return int.from_bytes(bytes(a), "little")

    def close(self):
        self.lib.kn_num_free(self.e, self.x)
        self.lib.kn_engine_free(self.e)


def _chain(v, k, n, count, c):
    for _ in range(count):
        v = _mod(v * v + c, k, n) if v or c >= 0 else _mod(c % (k * (1 << n) - 1), k, n)
    return v


@pytest.mark.parametrize("k,n", [(1, 8), (3, 349), (3, 399), (3, 400), (5, 450), (2**30 - 1, 401), (9, 800), (2**30 - 1, 1600),
                                 (7, 6350), (4097, 12750), (9999, 50000), (3, 102350), (2**30 - 1, 102400), (1, 409000),
                                 (9357, 369717), (9999, 600000), (11, 1000003), (3, 3300000), (139, 400350), (3795, 355167)])
def test_chain_equals_python(k, n):
    N = k * (1 << n) - 1
    e = _Engine(k, n)
    try:
        rng = random.Random(n)
        starts = [rng.getrandbits(n) % N] if n > 200000 else [0, 1, N - 1, N - 2, (1 << n) - 1, rng.getrandbits(n) % N, rng.getrandbits(n) % N]
        for v in starts:
            for count in (1, 2, 5) if n <= 200000 else (3,):
                for c in (None, -2, 2**62 + 1) if n <= 200000 else (None, -2):
                    e.set(v)
                    assert e.get() == v % N  # k = 1: 2^n - 1 is N
                    if c is None:
                        assert e.lib.kn_square(e.e, e.x, count) == 0
                    elif c >= N or -c >= N:
                        continue
                    else:
                        assert e.lib.kn_square_add(e.e, e.x, count, c) == 0
                    assert e.get() == _chain(v, k, n, count, c or 0) % N
    finally:
        e.close()


@pytest.mark.parametrize("value", ["N", "N+1", "2N+5"])
def test_unreduced_number_reads_reduced(value):
    k, n = 9357, 20011
    N = k * (1 << n) - 1
    v = {"N": N, "N+1": N + 1, "2N+5": 2 * N + 5}[value]
    e = _Engine(k, n)
    try:
        e.set(v)
        assert e.get() == v % N
    finally:
        e.close()


@pytest.mark.parametrize("streams", [1, 3])
def test_group_equals_python(streams):
    from ahnum_gb300.ntt_group import NttGroup
    rng = random.Random(5)
    tests = [(3, 300), (9999, 450)] * (streams == 1) + [(rng.randrange(3, 2**30, 2), rng.randrange(2000, 60000)) for _ in range(7)]
    with NttGroup(tests, streams=streams) as g:
        for count in (1, 8, 11):
            g.square(count)
        for (k, n), e, x in zip(tests, g.engines, g.nums):
            a = (C.c_uint64 * g.lib.kn_limbs(e))()
            assert g.lib.kn_get_limbs(e, x, a) == 0
            assert int.from_bytes(bytes(a), "little") == _chain(3, k, n, 20, 0)


@pytest.mark.parametrize("n,j", [(1000, 4), (20000, 9), (20000, 150), (369717, 5000), (600000, 7)])
def test_carry_through_a_full_word_reads_right(n, j):
    """a number whose words meet a carry into 2^w - 1 when it leaves the Montgomery form: 3 A with the
    words of A chosen so"""
    k = 3
    e = _Engine(k, n)
    try:
        w = e.lib.kn_word_bits(e.e)
        assert (j + 2) * w < n
        full, inv = (1 << w) - 1, pow(3, -1, 1 << w)
        a0 = full                                     # 3 a0: a carry of 2
        a1 = full * inv % (1 << w)                    # 3 a1 = 2^w - 1 (mod 2^w)
        a2 = (full - (3 * a1 >> w)) * inv % (1 << w)  # with a1's carry the next word is full
        a = (a0 << (w * (j - 1))) + (a1 << (w * j)) + (a2 << (w * (j + 1)))
        e.set(3 * a)
        assert e.get() == 3 * a
        assert e.lib.kn_square(e.e, e.x, 2) == 0
        assert e.get() == _chain(3 * a, k, n, 2, 0)
    finally:
        e.close()
