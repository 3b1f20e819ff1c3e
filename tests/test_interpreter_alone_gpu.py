"""The vector interpreter without the kernels that take short and normalising graphs off it: it remains the fallback for every
address and form that they do not accept, so the tests of those graphs run on it too (the switches are read once per process)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FILES = ["test_vector_gpu.py", "test_direct_gpu.py", "test_row_kernels_gpu.py", "test_ragged_ring_gpu.py", "test_baseline_shapes_gpu.py"]


@pytest.mark.parametrize("name", FILES)
def test_on_the_interpreter(name):
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider", os.path.join("tests", name)], cwd=ROOT,
                       env=dict(os.environ, DVM_B200_NO_ROW="1", DVM_B200_DIRECT_MAX="0"), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "passed" in r.stdout, r.stdout[-3000:]
