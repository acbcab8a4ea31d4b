"""A product that ends exactly half-way between two integers is reported with its full round-off of 0.5:
numbers with one odd digit, halved in the engine's own memory, times 1."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


class _Doubles:
    """The device number at `ptr` for torch."""

    def __init__(self, ptr, count):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (count,), "typestr": "<f8", "version": 3}


@pytest.mark.parametrize("L", [64, 512, 1344])
@pytest.mark.parametrize("value", [1, 3, 7, -5])
@pytest.mark.parametrize("first", [0, 2, 41])
def test_half_is_reported(lib, L, value, first):
    torch = pytest.importorskip("torch")
    e = lib.kc_engine_new(1, 10 * L, L, None, None, None, 0, 0, 0, 0, -1)
    assert e
    x, y = lib.kc_num_alloc(e), lib.kc_num_alloc(e)
    try:
        digits = (C.c_int64 * L)()
        digits[first] = value
        assert lib.kc_from_digits(e, x, digits) == 0
        digits = (C.c_int64 * L)()
        digits[0] = 1
        assert lib.kc_from_digits(e, y, digits) == 0 and lib.kc_sync(e) == 0
        torch.as_tensor(_Doubles(C.cast(x, C.c_void_p).value, L), device="cuda").mul_(0.5)
        torch.cuda.synchronize()
        lib.kc_reset_maxerr(e)
        assert lib.kc_mul(e, x, y) == 0
        assert abs(lib.kc_maxerr(e) - 0.5) < 1e-6
    finally:
        lib.kc_num_free(e, x)
        lib.kc_num_free(e, y)
        lib.kc_engine_free(e)
