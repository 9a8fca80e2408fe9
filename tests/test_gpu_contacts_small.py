"""Contacts around the smallest system that takes the walk over sorted atoms,
and ordered sums of one bucket around what is brought together at a time
(k_atomic_sum, csrc/atomic_kernels.cu)."""
import numpy as np
import pytest

from test_gpu_contacts import _check, _system
from test_gpu_ordered_sum import F, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 894, 895, 896, 1300])
@pytest.mark.parametrize("basis", ["free", "general"])
def test_sizes(oracle_mod, n, basis):
    _check(oracle_mod, _system(n, basis, scale=(n / 4000.0) ** (1 / 3)), reduceDistanceToUpper=True)


@pytest.mark.parametrize("n", [511, 512, 513, 4095, 8191, 8192, 8193, 12289])
def test_one_bucket(n):
    rng = np.random.default_rng(n)
    _run(rng.uniform(0, 2.6, n).astype(F), np.zeros(n, np.int32), 1, 0.0)
