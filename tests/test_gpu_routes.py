"""Runs routes_gpu.py, whose tests read launches from the profiler, in a fresh process."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


def test_calls_run_the_kernels_they_should():
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-m", "pytest", os.path.join(here, "routes_gpu.py"), "-m", "gpu", "-q", "-p", "no:cacheprovider"], capture_output=True, text=True,
                       cwd=os.path.dirname(here), timeout=900)
    assert r.returncode == 0, r.stdout[-6000:] + r.stderr[-2000:]
