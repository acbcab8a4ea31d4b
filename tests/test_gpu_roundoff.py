"""The round-off of random numbers at the length's limit stays below what double-precision transforms had on
the same numbers (24 squarings and a product, largest difference to an integer): lengths whose rows or
columns take three and more odd radices."""
import random

import pytest

pytestmark = pytest.mark.gpu

# k, n, L and the largest round-off of the double-precision passes at the same shape
ODD = [(9357, 9009432, 734832, 0.2339), (9357, 11747067, 967680, 0.1410), (9357, 10247149, 839808, 0.2006),
       (9357, 6435445, 518400, 0.1560), (9357, 7765093, 629856, 0.2611), (4501, 12072976, 952560, 0.1665)]


def _largest(k, n, L):
    from ahnum_gb300.kite import Ctx
    with Ctx(k, n, L) as c:
        x = c.num(random.Random(L).getrandbits(n - 1))
        c.reset_maxerr()
        c.square(x, 24)
        c.mul(x, x)
        return c.maxerr()


@pytest.mark.parametrize("k,n,L,double", ODD)
def test_odd_radices(lib, k, n, L, double):
    assert _largest(k, n, L) <= double
