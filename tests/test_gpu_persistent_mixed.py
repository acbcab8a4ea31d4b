"""The batch's persistent kernel over slots with groups of 4 and of 8 columns together: it runs, and gives
the numbers of the pass launches."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

# (k, n, L, rows of the length or 0): columns of 1024 and 1000 rows take groups of 4
TESTS = [(3, 1000000, 65536, 1024), (9357, 20000, 0, 0), (21, 400000, 32000, 1000), (9001, 662695, 49152, 0)]


@pytest.mark.parametrize("chosen", [TESTS, TESTS[:1], TESTS[1:], TESTS[::2]])
def test_persistent_equals_passes(lib, monkeypatch, chosen):
    from ahnum_gb300.kite import Batch
    out = []
    for persistent in (0, 1):
        monkeypatch.setenv("KITE_GB300_BATCH_PERSISTENT", str(persistent))
        try:
            for _, _, L, R in chosen:
                assert not R or lib.kc_set_fft_shape(L, R) == 0
            with Batch(gerbicz_block=30, gerbicz_blocks=1 << 20) as b:
                slots = [b.add_fermat(k, n, 3, L) for k, n, L, _ in chosen]
                slots.append(b.add_llr(chosen[0][0] + 2, chosen[0][1] + 1, chosen[0][2]))
                assert min(slots) >= 0
                for _ in range(2):
                    b.step(1)
                limbs = []
                for slot, (_, n, _, _) in zip(slots, chosen + [(0, chosen[0][1] + 1, 0, 0)]):
                    a = (C.c_uint64 * ((n + 127) // 64))()
                    if lib.kc_batch_read(b.h, slot, a) == 0:
                        limbs.append(bytes(a))
                assert len(limbs) >= len(chosen)
                out.append(limbs)
                ms, flops = C.c_double(), C.c_double()
                assert lib.kc_batch_profile_steps(b.h, 20, C.byref(ms), C.byref(flops)) == 0
                assert ms.value > 0
        finally:
            for _, _, L, R in chosen:
                if R:
                    lib.kc_set_fft_shape(L, 0)
    assert out[0] == out[1]
