"""The native part of the Python binding as far as it can be reached without a GPU."""
import subprocess
import sys

import pytest
import torch

NO_GPU = pytest.mark.skipif(torch.cuda.is_available(), reason="about a machine without a GPU")


@NO_GPU
def test_current_stream_without_a_gpu_raises():
    code = ("from mooncake_b200 import ep\n"
            "try:\n    ep.current_stream()\n"
            "except RuntimeError:\n    print('raised')\n")
    got = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert got.returncode == 0 and got.stdout.strip() == "raised", got.stderr[-500:]
