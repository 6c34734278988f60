"""The amplitudes A^-1 g of the plain form's transform without eigenvectors (zone_sqrt64.cu, 65 <= N
<= 128), which are refined by g - A a: the increments X a that they give at the observations are no
further from the exact ones than the CUDA-core form's (an FP64 eigensolve), in the geometric mean
over the zones. Inputs and reference as in test_gpu_isqrt_amplitudes.py.
"""
import pytest

from test_gpu_isqrt_amplitudes import test_increments_are_as_exact_as_the_eigensolve as _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,N,lo,hi", [("lin", 65, 3, 4), ("lin", 128, 5, 6), ("one", 65, 2, 3),
                                           ("one", 100, 6, 7), ("geom", 100, 2, 3),
                                           ("two", 128, 1.5, 2.5), ("flat", 96, 1, 2)])
def test_increments(shape, N, lo, hi):
    _compare(shape, N, lo, hi)
