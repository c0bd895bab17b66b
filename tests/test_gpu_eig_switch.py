"""ISVD_GPU_EIG_REFINED=0 (or a device without cluster launches) leaves every eigensolve to the two-sided Jacobi,
in single solves and in batches."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("module", ["test_gpu_batched.py", "test_gpu_svd_start.py"])
def test_without_refinement(module):
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider", os.path.join(HERE, module)],
                       env=dict(os.environ, ISVD_GPU_EIG_REFINED="0"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
