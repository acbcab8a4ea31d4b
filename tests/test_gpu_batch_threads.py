"""Batches on both sides of the block size's rule: slots whose buffers leave room for many CTAs an SM, and
for fewer than four, alone and together, against Python integers."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _squared(k, n, count):
    N = k * (1 << n) - 1
    v = pow(3, k)
    for _ in range(count + 1):
        while v > N:
            q, r = divmod(v >> n, k)
            v = (v & ((1 << n) - 1)) + q + (r << n)
        if count:
            v = v * v
            count -= 1
    return v % N


# (L, rows): buffers of a column group are 256 bytes a row, of a row pair 64 bytes a column
@pytest.mark.parametrize("shapes", [[(2048, 16)], [(65536, 224)], [(65536, 256)], [(32768, 16)], [(2048, 16), (65536, 256)],
                                    [(2048, 8), (40960, 20), (24576, 96)]])
def test_batch_block_equals_python(shapes):
    from ahnum_gb300 import native
    from ahnum_gb300.kite import Batch
    lib = native.load()
    block, k = 9, 21
    set_ = []
    try:
        for L, R in shapes:
            if (L // 2) % R == 0 and lib.kc_set_fft_shape(L, R) == 0:
                set_.append(L)
        with Batch(gerbicz_block=block, gerbicz_blocks=1 << 20) as b:
            tests = [(k + 2 * i, 17 * L + i) for i, (L, _) in enumerate(shapes)]
            slots = [b.add_fermat(kk, n, 3, L) for (kk, n), (L, _) in zip(tests, shapes)]
            assert min(slots) >= 0
            b.step(1)
            for slot, (kk, n) in zip(slots, tests):
                a = (C.c_uint64 * ((n + 127) // 64))()
                assert lib.kc_batch_read(b.h, slot, a) == 0
                assert int.from_bytes(bytes(a), "little") == _squared(kk, n, block)
    finally:
        for L in set_:
            lib.kc_set_fft_shape(L, 0)
