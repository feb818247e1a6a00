"""The registered ops on CPU, with a stand-in for the layer: calls that something watches go through the dispatcher as those of
any custom op, whatever short way `linear` and `linear_silu` have round it."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch
from torch.fx.experimental.proxy_tensor import make_fx

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


def test_transforms(op):
    assert torch.equal(torch.vmap(op)(torch.stack([X, 2 * X])), torch.stack([SUM, 2 * SUM]))
    assert torch.equal(torch.func.functionalize(op)(X), SUM)
    assert torch.equal(torch.func.jvp(op, (X,), (X,))[0], SUM)


def test_a_gradient_is_refused(op):
    x = X.clone().requires_grad_()
    with pytest.raises(RuntimeError, match="no autograd formula"):
        op(x).sum().backward()
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda x: op(x).sum())(X)


def test_tracers_see_one_op(op):
    for graph in (make_fx(op)(X).graph, make_fx(op, pre_dispatch=True)(X).graph, torch.fx.symbolic_trace(op).graph):
        names = [str(n.target) for n in graph.nodes if n.op == "call_function"]
        assert len(names) == 1 and names[0].startswith("hygemm_vllm.linear"), names
    traced = torch.jit.trace(op, X, check_trace=False)
    assert [n.kind() for n in traced.graph.nodes() if n.kind() != "prim::Constant"][0].startswith("hygemm_vllm::linear")
    assert torch.equal(traced(3 * X), 3 * SUM)
    compiled = torch.compile(lambda x: op(x) + 1, backend="aot_eager", fullgraph=True)
    assert torch.equal(compiled(X), SUM + 1)


def test_modes_and_profiler_see_the_op(op):
    seen = []

    class Mode(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, function, types, args=(), kwargs=None):
            seen.append(str(function))
            return function(*args, **(kwargs or {}))

    with Mode():
        op(X)
    assert any(s.startswith("hygemm_vllm.linear") for s in seen) and not any("data_ptr" in s for s in seen), seen
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as profile:
        op(X)
    assert any(e.key.startswith("hygemm_vllm::linear") for e in profile.key_averages())


def test_a_meta_tensor_gives_a_meta_tensor(op):
    y = op(torch.empty(5, 4, device="meta"))
    assert y.is_meta and y.shape == (5, 3)


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
