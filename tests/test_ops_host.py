"""CPU: host logic of the operator bindings that needs no device."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_import_on_a_torch_without_cuda():
    """A torch built without CUDA lacks the raw device and stream calls: the module imports, and asking for a stream goes through
    the public call (which then says what is missing)."""
    code = """
import sys, types
sys.path.insert(0, sys.argv[1])
import torch
for name in ("_cuda_getDevice", "_cuda_getCurrentRawStream"):
    if hasattr(torch._C, name):
        delattr(torch._C, name)
from pet_b200 import ops
torch.cuda.current_stream = lambda: types.SimpleNamespace(cuda_stream=1234)
assert ops._stream() == 1234
print("ok")
"""
    out = subprocess.run([sys.executable, "-c", code, ROOT], capture_output=True, text=True, timeout=240)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stderr[-2000:]
