"""Matrix products of the model: y = x W^T (+ bias), dx = dy W, dW = dy^T x.

Back ends, chosen once per process (`set_backend`), of the native training step (src/model/gpt2_step.cc) and of the functions below:
  "auto"     (default) this framework's kernel wherever its epilogue saves a pass (GELU and its derivative); of the plain
             products the step gives it the small ones, by their operations, and cuBLAS the large; the functions below
             leave all plain products to cuBLAS
  "tcgen05"  this framework's sm_100a kernel (src/ops/gemm_sm100.cu: TMA -> shared memory ->
             tcgen05.mma with TMEM accumulators) for every product that it supports
  "cublas"   cuBLAS
The step issues its products itself and reports their number through `count`; the functions are for programs that put a model together from Python.
"""
from __future__ import annotations

import os

import torch

_backend = os.environ.get("PICCL_GEMM", "auto")
_counts = {"tcgen05": 0, "cublas": 0}


def set_backend(name: str) -> None:
    global _backend
    assert name in ("auto", "tcgen05", "cublas")
    _backend = name


def backend() -> str:
    return _backend


def backend_code() -> int:
    """The backend as the native training step numbers it."""
    return ("auto", "tcgen05", "cublas").index(_backend)


def counts() -> dict:
    return dict(_counts)


def count(tcgen05: int, cublas: int) -> None:
    """Adds the products of a native training step."""
    _counts["tcgen05"] += tcgen05
    _counts["cublas"] += cublas


def _own_kernel_ok(x, w, out, *others, fused_epilogue: bool = False) -> bool:
    """"auto": the tcgen05 kernel where its fused epilogue saves a pass over the activations (GELU); plain products stay on cuBLAS.
    "tcgen05": wherever supported.  The kernel needs operands that start on a 16-byte boundary."""
    if _backend == "cublas" or (_backend == "auto" and not fused_epilogue):
        return False
    from . import gemm_sm100
    return gemm_sm100.available() and gemm_sm100.supports(x, w, out) and all(t is None or t.data_ptr() % 16 == 0 for t in (x, w, out, *others))


def linear(x: torch.Tensor, w: torch.Tensor, bias, out: torch.Tensor) -> torch.Tensor:
    """out[M, N] = x[M, K] @ w[N, K]^T + bias[N]"""
    if _own_kernel_ok(x, w, out, bias):
        from . import gemm_sm100
        gemm_sm100.gemm(gemm_sm100.NT, gemm_sm100.BIAS, x, w, out, bias=bias)
        _counts["tcgen05"] += 1
        return out
    _counts["cublas"] += 1
    if bias is None:
        return torch.mm(x, w.t(), out=out)
    return torch.addmm(bias, x, w.t(), out=out)


def linear_gelu(x: torch.Tensor, w: torch.Tensor, bias: torch.Tensor, h_out, g_out: torch.Tensor) -> None:
    """h_out = x @ w^T + bias (None: not wanted);  g_out = gelu_tanh(h_out)   — one kernel where the tcgen05 GEMM is usable."""
    if _own_kernel_ok(x, w, g_out, bias, h_out, fused_epilogue=True):
        from . import gemm_sm100
        gemm_sm100.gemm(gemm_sm100.NT, gemm_sm100.GELU, x, w, g_out, bias=bias, pre=h_out)
        _counts["tcgen05"] += 1
        return
    from . import bias_gelu_fwd
    _counts["cublas"] += 1
    h = g_out if h_out is None else h_out
    torch.mm(x, w.t(), out=h)
    bias_gelu_fwd(h, bias, h_out, g_out)


def grad_input(dy: torch.Tensor, w: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """out[M, K] = dy[M, N] @ w[N, K]"""
    _counts["cublas"] += 1
    return torch.mm(dy, w, out=out)


def grad_weight(dy: torch.Tensor, x: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """out[N, K] = dy[M, N]^T @ x[M, K]"""
    _counts["cublas"] += 1
    return torch.mm(dy.t(), x, out=out)
