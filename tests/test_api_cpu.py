"""The Python layer without a GPU."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("name", ["_cuda_getCurrentRawStream", "_cuda_getDevice"])
def test_stream_without_the_private_names_of_torch(name):
    """A torch without the shortcuts: the module loads, and the current stream is
    asked for by the public call."""
    code = f"""
import torch
if hasattr(torch._C, {name!r}):
    delattr(torch._C, {name!r})
from isai_kernel_gb300 import api

class Stream:
    cuda_stream = 42

torch.cuda.is_initialized = lambda: True
torch.cuda.current_stream = Stream
print(api._s(), api._s(Stream()))
"""
    out = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-500:]
    assert out.stdout.split() == ["42", "42"]
