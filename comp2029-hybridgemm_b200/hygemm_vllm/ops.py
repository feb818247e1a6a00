"""Opaque torch custom ops of the hybrid linear (no vLLM import needed).

`hygemm_vllm::linear` and `hygemm_vllm::linear_silu` keep the reference's
schemas (quantization.py:18-25, producer.py:27-40 of the reference): the layer
runtime is looked up by an integer handle in `_runtimes`, nothing is mutated,
and the fake implementations give shape/dtype for tracing.

An eager call of a custom op costs about as much host time as the layer itself, so calling `linear` or `linear_silu` on an
ordinary tensor with nothing watching goes straight to the layer.  Everything else goes through the dispatcher: tracing,
modes, functorch transforms, profiling, tensor subclasses and wrappers, tensors that require a gradient (the ops have none,
and say so in the backward pass).
"""
from __future__ import annotations

import torch

_runtimes: dict[int, object] = {}


def register_runtime(runtime) -> int:
    handle = id(runtime)
    _runtimes[handle] = runtime
    return handle


def _linear(x: torch.Tensor, handle: int, outputs: int) -> torch.Tensor:
    return _runtimes[handle](x)


def _linear_fake(x, handle, outputs):
    return x.new_empty((x.shape[0], outputs))


def _silu_linear(runtime, x, math):
    if hasattr(runtime, "silu_linear"):
        return runtime.silu_linear(x, math)
    from .producer import silu_pack
    return runtime.run_packed(*silu_pack(x, math))


def _linear_silu(x: torch.Tensor, handle: int, outputs: int, math: int) -> torch.Tensor:
    runtime = _runtimes[handle]
    if hasattr(runtime, "profile_name") and torch.cuda.is_current_stream_capturing():
        # Same NVTX label as the reference's profiling hook (producer.py:31).
        label = (f"projection|{runtime.profile_name}|O={runtime.outputs}|K={runtime.k}"
                 f"|H={runtime.hi.numel()}|T={x.shape[0]}")
        with torch.cuda.nvtx.range(label):
            return _silu_linear(runtime, x, math)
    return _silu_linear(runtime, x, math)


def _linear_silu_fake(x, handle, outputs, math):
    return x.new_empty((x.shape[0], outputs))


def _plain(x) -> bool:
    """An eager call on an ordinary tensor that nothing traces, transforms, intercepts, records or differentiates."""
    return (not torch.compiler.is_compiling()
            and not torch._C._len_torch_function_stack() and not torch._C._len_torch_dispatch_stack()
            and torch._C._functorch.peek_interpreter_stack() is None and torch._C._get_tracing_state() is None
            and not torch.autograd._profiler_enabled()
            and type(x) is torch.Tensor and not x.requires_grad and not x.is_meta
            and not torch._C._functorch.is_functorch_wrapped_tensor(x) and not torch._is_functional_tensor(x))


class _Op(torch.library.CustomOpDef):
    """A custom op with the short way round the dispatcher; `direct` is its function."""

    def __call__(self, x, *args, **kwargs):
        if _plain(x):
            return self.direct(x, *args, **kwargs)
        return super().__call__(x, *args, **kwargs)


def _define(name, function, fake):
    op = torch.library.custom_op(f"hygemm_vllm::{name}", function, mutates_args=())
    op.register_fake(fake)
    op.__class__ = _Op
    op.direct = function
    return op


linear = _define("linear", _linear, _linear_fake)
linear_silu = _define("linear_silu", _linear_silu, _linear_silu_fake)
