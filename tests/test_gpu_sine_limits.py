"""The sine transforms at the edges of the fixed-point sines (k_sine_fixed,
csrc/fp64_kernels.cu), against numpy in 64 bits: weights past float32."""
import numpy as np
import pytest

from test_gpu_sine_fixed import _check

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("step,value", [(3e4, 9e29), (2.0 ** 30, 9e29), (2.0 ** 30, -9e29), (3e4, 1e22),
                                        (2.0 ** 30, 1e20)])
def test_large_weights(step, value):
    """Grids and values that are finite, with products that are not in float32."""
    y = (step * np.arange(300)).astype(F)
    _check((0.5 + 0.25 * np.arange(40)).astype(F), y, np.full(300, value, F))
