"""Opaque torch custom ops of the hybrid linear (no vLLM import needed).

`hygemm_vllm::linear` and `hygemm_vllm::linear_silu` keep the reference's
schemas (quantization.py:18-25, producer.py:27-40 of the reference): the layer
runtime is looked up by an integer handle in `_runtimes`, nothing is mutated,
and the fake implementations give shape/dtype for tracing.

The ops are registered with the dispatcher directly, and the functions `linear` and `linear_silu` of this module only go
through it where something may be watching (tracing, dispatch modes, tensor subclasses, autograd): an eager call
of an op registered with `torch.library.custom_op` costs about as much host time as the layer itself.
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


_library = torch.library.Library("hygemm_vllm", "DEF")
for _name, _function, _fake in (("linear", _linear, _linear_fake), ("linear_silu", _linear_silu, _linear_silu_fake)):
    _library.define(_name + torch.library.infer_schema(_function, mutates_args=()))
    _library.impl(_name, _function, "CompositeExplicitAutograd")
    torch.library.register_fake(f"hygemm_vllm::{_name}", _fake, lib=_library)


def _plain(x) -> bool:
    """An eager call on an ordinary tensor that nothing traces, intercepts or differentiates."""
    return (not torch.compiler.is_compiling() and type(x) is torch.Tensor and not x.requires_grad
            and not torch._C._len_torch_dispatch_stack())


def linear(x: torch.Tensor, handle: int, outputs: int) -> torch.Tensor:
    return _runtimes[handle](x) if _plain(x) else torch.ops.hygemm_vllm.linear(x, handle, outputs)


def linear_silu(x: torch.Tensor, handle: int, outputs: int, math: int) -> torch.Tensor:
    return _linear_silu(x, handle, outputs, math) if _plain(x) else torch.ops.hygemm_vllm.linear_silu(x, handle, outputs, math)
