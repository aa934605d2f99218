"""The tiled kernel at the small shapes of its own tests, which the size rule of `ggq_gemv` hands to other kernels by default: the same
tests once more with the rule off.  The switch is read once per process, so they run in a child process."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


def test_the_tiled_kernels_tests_with_the_size_rule_off():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-m", "pytest", os.path.join(root, "tests", "test_tile_gpu.py"), "-q", "-x", "-m", "gpu"],
                       env=dict(os.environ, GGQ_TILE_ALWAYS="1"), cwd=root, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and " passed" in r.stdout, r.stdout[-3000:] + r.stderr[-1000:]
