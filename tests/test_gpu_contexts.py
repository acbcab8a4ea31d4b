"""Several contexts with work at once: their squarings share the GPU instead of running one after another,
and are right in either form, whatever the count, the addend and how often the round-off is tracked; and
squarings that a caller captures on the engine's stream can be replayed."""
import ctypes as C
import random
import threading
import time

import pytest

pytestmark = pytest.mark.gpu

K = 4095


def _mod(v, k, n):
    while v >> n >= k:
        q, r = divmod(v >> n, k)
        v = (v & ((1 << n) - 1)) + q + (r << n)
    return v - (k << n) + 1 if v >= (k << n) - 1 else v


def _timed(contexts, count):
    def run(c, x):
        c.square(x, count)
        c.sync()

    best = 1e9
    for _ in range(3):
        threads = [threading.Thread(target=run, args=a) for a in contexts]
        t0 = time.perf_counter()
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        best = min(best, time.perf_counter() - t0)
    return best


# one after another, 6 contexts take 6 times as long as one; sharing the GPU they take about 1.5 times
@pytest.mark.parametrize("L", [3584, 28672])
def test_contexts_share_the_gpu(lib, L):
    from ahnum_gb300.kite import Ctx
    cs = [Ctx(K, 12 * L + i, L) for i in range(6)]
    try:
        work = [(c, c.num(random.Random(i).getrandbits(12 * L - 1))) for i, c in enumerate(cs)]
        _timed(work, 64)
        assert _timed(work, 4096) < 3 * _timed(work[:1], 4096)
    finally:
        for c in cs:
            c.close()


# chains of a cluster, of few CTAs and of all, beside a context whose queue is full
@pytest.mark.parametrize("L", [1344, 3584, 28672])
def test_squares_beside_another(lib, L):
    from ahnum_gb300.kite import Ctx
    n, N = 11 * L, K * (1 << (11 * L)) - 1
    rng = random.Random(L)
    v0 = rng.getrandbits(n - 1)
    big = rng.getrandbits(12 * 163840)
    ends = []
    for busy in (False, True):
        with Ctx(K, 12 * 163840 + 1, 163840) as a:
            z = a.num(big)
            e = lib.kc_engine_new(K, n, L, None, None, None, 0, 0, 0, 0, -1)
            assert e
            x = lib.kc_num_alloc(e)
            digits = (C.c_int64 * L)()
            nl = (n + 127) // 64
            limbs = (C.c_uint64 * nl)(*[(v0 >> (64 * i)) & (2**64 - 1) for i in range(nl)])
            assert lib.kc_limbs_to_digits(K, n, L, limbs, digits) == 0
            a.sync()
            if busy:
                a.square(z, 12000)  # 250 ms
            assert lib.kc_from_digits(e, x, digits) == 0
            v = v0
            for every, count, c in ((1, 1, 0), (1, 15, 0), (4, 16, -2), (4, 17, 5), (3, 33, 0), (1, 50, -2), (1, 600, 0)):
                lib.kc_set_roundoff_check(e, every)
                assert (lib.kc_square_add(e, x, count, c) if c else lib.kc_square(e, x, count)) == 0
                if not busy:
                    for _ in range(count):
                        v = _mod(v * v + c, K, n)
            assert lib.kc_to_digits(e, x, digits) == 0
            assert lib.kc_digits_to_limbs(K, n, L, digits, limbs) == 0
            assert lib.kc_maxerr(e) < 0.4
            ends.append(bytes(limbs))
            if not busy:
                assert int.from_bytes(bytes(limbs), "little") == v % N
                a.square(z, 12000)
            ends.append(a.get(z))
            lib.kc_num_free(e, x)
            lib.kc_engine_free(e)
    assert ends[0] == ends[2] and ends[1] == ends[3]


@pytest.mark.parametrize("L", [1344, 3584])
def test_captured_squarings_replay(lib, L):
    torch = pytest.importorskip("torch")
    n = 11 * L
    e = lib.kc_engine_new(K, n, L, None, None, None, 0, 0, 0, 0, -1)
    assert e
    x = lib.kc_num_alloc(e)
    try:
        digits = (C.c_int64 * L)(3)
        assert lib.kc_from_digits(e, x, digits) == 0
        assert lib.kc_square(e, x, 40) == 0 and lib.kc_sync(e) == 0
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(torch.cuda.ExternalStream(lib.kc_stream(e))):
            graph.capture_begin(capture_error_mode="thread_local")
            assert lib.kc_square(e, x, 5) == 0
            graph.capture_end()
            for _ in range(4):
                graph.replay()
        assert lib.kc_square(e, x, 20) == 0
        assert lib.kc_to_digits(e, x, digits) == 0
        limbs = (C.c_uint64 * ((n + 127) // 64))()
        assert lib.kc_digits_to_limbs(K, n, L, digits, limbs) == 0
        v = 3 * K
        for _ in range(80):
            v = _mod(v * v, K, n)
        assert int.from_bytes(bytes(limbs), "little") == v
        assert lib.kc_error(e) == 0
    finally:
        lib.kc_num_free(e, x)
        lib.kc_engine_free(e)
