"""The registered ops on CPU, with a stand-in for the layer: calls that something watches go through the dispatcher as those of
any custom op, whatever short way `linear` and `linear_silu` have round it."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from hygemm_vllm import ops


class Layer:
    """A layer reads raw memory: here too, so that a tensor without storage of its own is an error."""
    outputs, k = 3, 4

    def __call__(self, x):
        x.data_ptr()
        return x.detach().sum(1, keepdim=True).expand(-1, 3).contiguous()

    def silu_linear(self, x, math):
        return self(x)


@pytest.fixture(params=["linear", "linear_silu"])
def op(request):
    handle = ops.register_runtime(Layer())
    call = getattr(ops, request.param)
    yield lambda x: call(x, handle, 3) if request.param == "linear" else call(x, handle, 3, 0)
    ops._runtimes.pop(handle)


X = torch.arange(8.).reshape(2, 4)
SUM = X.sum(1, keepdim=True).expand(-1, 3)


def test_an_ordinary_call(op):
    assert torch.equal(op(X), SUM)
    with torch.inference_mode():
        assert torch.equal(op(X.clone()), SUM)


def test_a_gradient_is_refused(op):
    x = X.clone().requires_grad_()
    with pytest.raises(RuntimeError, match="no autograd formula"):
        op(x).sum().backward()


def test_registration():
    for op in (torch.ops.hygemm_vllm.linear.default, torch.ops.hygemm_vllm.linear_silu.default):
        assert torch.Tag.pt2_compliant_tag in op.tags
    assert isinstance(ops.linear, torch.library.CustomOpDef) and isinstance(ops.linear_silu, torch.library.CustomOpDef)
    # in a process of its own: the module again, which defines the ops again, and a library that adds to their namespace
    code = ("import importlib, torch; from hygemm_vllm import ops; importlib.reload(ops); "
            "library = torch.library.Library('hygemm_vllm', 'DEF'); library.define('other(Tensor x) -> Tensor')")
    package = Path(ops.__file__).resolve().parent.parent
    result = subprocess.run([sys.executable, "-c", code], cwd=package, capture_output=True, text=True)
    assert result.returncode == 0, result.stderr[-2000:]
