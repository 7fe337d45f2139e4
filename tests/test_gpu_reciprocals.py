"""The reciprocal and reciprocal square root of the pair and EEQ matrix kernels against CUDA's, over the
ranges that reach them.

Bounds: the estimate is good to 2^-20 at least (its documentation), so the third-order step leaves an error of
order 2^-60 and the result the rounding of its last operations: e is exact to its own rounding, the
correction is below 2^-20 of y, so the final fused multiply-add rounds once (0.5 ulp) on top of an error of
y e of a few 2^-73.  1/x: 0.5 ulp and the library's 0.5.  1/sqrt(x): x y is rounded before it enters e, half
an ulp of e's terms, another 0.5 ulp of the result; with the library's 1 ulp 2 in all.  ulps of the
library's result differ by a factor of two across a power of two."""
import pytest

from curcuma_b200 import _lib

pytestmark = pytest.mark.gpu

N = 20_000_000


# squared distances: from the coincidence limit (1e-20) to pairs a kilometre apart; width sums a_i + a_j
@pytest.mark.parametrize("lo,hi", [(1e-20, 1.0), (0.05, 1e4), (1e4, 1e26), (1e26, 1e300), (1e-300, 1e-20)])
def test_reciprocal_square_root(lo, hi):
    u = _lib.load().gfnff_reciprocal_ulps(0, 1, lo, hi, N)
    assert 0.0 <= u <= 2.0, u


# (r^6 + r0^6)(r^8 + r0^8) of the D4 damping: r0 from 4.8 to some 20 bohr, r up to 50; and the scalars of the
# conjugate gradients, which are checked to lie within 2^-1007 .. 2^1007
@pytest.mark.parametrize("lo,hi", [(1e9, 1e27), (1.0, 1e9), (1e-40, 1.0), (8e-304, 1e-40), (1e27, 1.3e303)])
def test_reciprocal(lo, hi):
    u = _lib.load().gfnff_reciprocal_ulps(0, 0, lo, hi, N)
    assert 0.0 <= u <= 1.0, u
