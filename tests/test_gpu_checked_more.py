"""More of the GPU parity tests under the bounds-checked build (see test_gpu_checked.py): the
stress divergence's row pass and the pressure solve on real(8) arrays, whose FP32 transforms
are kernels of their own."""
import os
import subprocess
import sys

import pytest

from overlappingbls_b200 import build
from conftest import ROOT

pytestmark = pytest.mark.gpu

SUBSET = ["tests/test_gpu_divstress.py", "tests/test_gpu_twopass.py", "tests/test_gpu_ops.py"]


def test_line_operations_under_index_checks():
    if os.environ.get("OBL_CHECKED_RUN") == "1":
        pytest.skip("already the child run")
    env = dict(os.environ, OBL_LIB=build.LIB_CHECK, OBL_CHECKED_RUN="1")
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider", *SUBSET,
                        "-k", "not 512 and not 640"],
                       cwd=ROOT, env=env, capture_output=True, text=True, timeout=1200)
    tail = "\n".join(r.stdout.splitlines()[-25:])
    assert r.returncode == 0 and " passed" in tail, tail
