"""The host calls where the device cannot read the caller's arrays
(FRMC_HOST_DIRECT=0: inputs and outputs are copied): the tests of the calls that
read them otherwise, once more in a process with that switch, which is read when
the library's context is made."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("names", [
    ("gpu_cell_pairs", "gpu_cell_lists", "gpu_cell_small", "gpu_cell_blocks_in_range", "gpu_rows_by_value"),
    ("gpu_contacts", "gpu_contacts_small", "gpu_few_rows", "gpu_ordered_sum", "gpu_atomic"),
    ("gpu_coordination", "gpu_coordination_walk"),
    ("gpu_distance_rows", "gpu_sine_fixed", "gpu_sine_limits", "shape_function"),
], ids=["histograms", "contacts", "coordination", "rows_and_sines"])
def test_without_host_reads(names):
    files = [os.path.join(HERE, "test_%s.py" % n) for n in names]
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider", *files],
                       env=dict(os.environ, FRMC_HOST_DIRECT="0"), cwd=os.path.dirname(HERE), capture_output=True,
                       text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-4000:] + r.stderr[-2000:]
    assert " passed" in r.stdout and "skipped" not in r.stdout, r.stdout[-400:]
