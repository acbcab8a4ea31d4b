"""Squaring chains whose CTAs meet in one cluster, and over the whole GPU, with a neighbour's flag between
the halves of the column pass: chains of odd and even length and past one launch, other operations
between them, and engines of both kinds in several threads, against Python integers."""
import random
import threading

import pytest

pytestmark = pytest.mark.gpu

K = 4095


def _square(v, n, count):
    N = K * (1 << n) - 1
    for _ in range(count):
        v = v * v
        while v > N:
            q, r = divmod(v >> n, K)
            v = (v & ((1 << n) - 1)) + q + (r << n)
    return v % N


def _bits(lib, L):
    from ahnum_gb300.tune import safe_bpw
    return int(L * min(safe_bpw(L, K), 18))


# (L, rows, group width): 2 to 16 items in a cluster of 2 to 16, more over the GPU, several groups per CTA
SHAPES = [(64, 2, 8), (128, 4, 8), (192, 2, 4), (512, 8, 2), (576, 18, 2), (960, 30, 4), (1344, 28, 2), (1344, 6, 2),
          (1536, 24, 8), (3584, 28, 4), (3584, 7, 2), (8192, 2, 2)]


@pytest.mark.parametrize("L,R,G", SHAPES)
def test_chains_equal_python(L, R, G):
    from ahnum_gb300 import native
    from ahnum_gb300.kite import Ctx
    lib = native.load()
    n = _bits(lib, L)
    v, w = random.Random(L).getrandbits(n - 1), random.Random(R).getrandbits(n - 1)
    N = K * (1 << n) - 1
    assert lib.kc_set_latency_shape(L, R, G) == 0
    try:
        with Ctx(K, n, L) as c:
            x, y = c.num(v), c.num(w)
            for count in (1, 2, 3, 514, 1):
                c.square(x, count)
                c.mul(y, x)
                v = _square(v, n, count)
                w = w * v % N
                assert c.get(x) == v
            assert c.get(y) == w
            assert c.maxerr() < 0.4
    finally:
        lib.kc_set_latency_shape(L, 0, 0)


def test_engines_in_threads():
    from ahnum_gb300.kite import Ctx
    sizes = [(512, 700), (1344, 600), (27648, 300), (512, 900), (49152, 200), (221184, 60)]
    from ahnum_gb300 import native
    lib = native.load()
    fails = []

    def one(L, count):
        n = _bits(lib, L)
        v = random.Random(L).getrandbits(n - 1)
        with Ctx(K, n, L) as c:
            x, y = c.num(v), c.num(v)
            for _ in range(3):
                c.square(x, count)
            c.square(y, 3 * count)
            if c.get(x) != c.get(y) or (L < 2000 and c.get(x) != _square(v, n, 3 * count)):
                fails.append(L)

    threads = [threading.Thread(target=one, args=s) for s in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not fails
