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


class _Calls:
    """Stands in for the native library: every pointer that a call gets must belong to a copy that is still alive."""

    def __init__(self, copies):
        self.copies, self.names = copies, []

    def __getattr__(self, name):
        def call(*args):
            self.names.append(name)
            alive = {ref().data_ptr() for ref in self.copies if ref() is not None}
            handed = [a for a in args if isinstance(a, int) and a > 1 << 20]
            assert handed and all(a in alive or a in self.outputs for a in handed), name
            assert len(set(handed)) == len(handed), f"{name}: two operands share their memory"
            return 0
        return call


def test_dense_copies_of_operands_outlive_the_call(monkeypatch):
    import types
    import weakref

    import torch
    from pet_b200 import ops
    copies, outputs = [], set()

    def copy_of(t):  # what _f32 does with a view
        c = t.clone()
        copies.append(weakref.ref(c))
        return c

    real_ptr = ops._ptr

    def ptr(t):
        if t is not None and not any(r() is t for r in copies):
            outputs.add(t.data_ptr())
        return real_ptr(t)

    monkeypatch.setattr(ops, "_f32", copy_of)
    monkeypatch.setattr(ops, "_ptr", ptr)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    ctx = ops.Context.__new__(ops.Context)
    ctx.lib, ctx.h, ctx._plans = _Calls(copies), 0, {}
    ctx.lib.outputs = outputs
    x, r = torch.rand(1, 8, 8, 8), torch.rand(1, 8, 8, 8)
    x5, w5 = torch.rand(1, 8, 4, 8, 8), torch.rand(8, 8, 1, 1, 1)
    v8, m = torch.rand(8), torch.rand(1, 64, 64)
    plan = types.SimpleNamespace(h=0, out_shape=(1, 8, 8, 8))
    ctx.conv2d_run(plan, x, v8, residual=r)
    ctx.conv2d_correct(plan, x, r, 0, 2, bias=v8)
    ctx._plans[("conv3d", tuple(x5.shape), tuple(w5.shape), (0, 0, 0), (1, 1, 1), (1, 1, 1), True, "none", "auto")] = \
        types.SimpleNamespace(h=0, out_shape=tuple(x5.shape))
    ctx.conv3d(x5, w5, (0, 0, 0), bias=v8, residual=torch.rand(x5.shape))
    ctx.convtrans_run(plan, x, None, v8)
    mm = types.SimpleNamespace(h=0, out_shape=(1, 64, 64))
    ctx.matmul_run(mm, m, torch.rand(1, 64, 64), torch.rand(64), residual=torch.rand(1, 64, 64))
    ctx.batchnorm(x, v8, torch.rand(8), torch.rand(8), torch.rand(8))
    ctx.layernorm(m, torch.rand(64), torch.rand(64))
    assert len(ctx.lib.names) == 8
