"""The shape that the single-test cost model takes: it gives the numbers of another shape of the same
length bit for bit, from the smallest lengths to those whose items fill the GPU more than once."""
import ctypes as C
import random

import pytest

pytestmark = pytest.mark.gpu


# (L, another shape: rows, group width)
@pytest.mark.parametrize("L,R,G", [(64, 2, 8), (512, 16, 4), (896, 14, 4), (2240, 35, 4), (10240, 128, 8),
                                   (36864, 72, 4), (57344, 112, 8), (163840, 160, 4), (442368, 512, 4)])
def test_model_shape_equals_another(L, R, G):
    from ahnum_gb300 import native
    from ahnum_gb300.kite import Ctx
    from ahnum_gb300.tune import safe_bpw
    lib = native.load()
    k = 9999
    n = int(L * min(safe_bpw(L, k), 20))
    x0 = random.Random(L).getrandbits(n - 1)
    seen, out = [], []
    for shape in (None, (R, G)):
        lib.kc_set_latency_shape(L, 0, 0)
        if shape:
            assert lib.kc_set_latency_shape(L, *shape) == 0
        try:
            e = lib.kc_engine_new(k, n, L, None, None, None, 0, 0, 0, 0, -1)
            assert e
            r, c = C.c_uint32(), C.c_uint32()
            lib.kc_shape(e, C.byref(r), C.byref(c))
            seen.append((r.value, c.value, lib.kc_group_width(e)))
            lib.kc_engine_free(e)
            with Ctx(k, n, L) as g:
                x = g.num(x0)
                g.square(x, 7)
                out.append(g.get(x))
                assert g.maxerr() < 0.4
        finally:
            lib.kc_set_latency_shape(L, 0, 0)
    assert seen[0] != seen[1] and seen[0][0] * seen[0][1] == L // 2
    assert out[0] == out[1]
