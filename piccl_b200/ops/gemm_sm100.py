"""Front end of the tcgen05 GEMM (src/ops/gemm_sm100.cu)."""
from __future__ import annotations

import ctypes as C

import torch

from .. import _native as N
from . import _bump, _s

_checked = None


def available() -> bool:
    global _checked
    if _checked is None:
        try:
            lib = N.ops_lib()
            _checked = hasattr(lib, "piccl_ops_gemm_bf16_nt_ex") and torch.cuda.is_available() and torch.cuda.get_device_capability()[0] == 10
        except Exception:
            _checked = False
    return _checked


NT, NN, TN = 0, 1, 2                                   # C = A B^T, A B, A^T B
BIAS, GELU, RESIDUAL, GELU_GRAD = 0, 1, 2, 3           # epilogues, see src/ops/gemm_sm100.cu


def supports(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor) -> bool:
    """Contiguous bf16 operands whose rows are a multiple of 16 bytes."""
    return (x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and out.dtype == torch.bfloat16 and x.is_contiguous() and w.is_contiguous()
            and out.is_contiguous() and x.shape[1] % 8 == 0 and w.shape[1] % 8 == 0 and out.shape[1] % 8 == 0)


_fn: dict = {}


def _native(name: str, argtypes):
    """A function of the library with its argument types declared, so that plain integers pass (half the cost of building ctypes objects)."""
    f = _fn.get(name)
    if f is None:
        f = getattr(N.ops_lib(), name)
        f.argtypes = argtypes
        _fn[name] = f
    return f


_GEMM = [C.c_int] * 2 + [C.c_void_p] * 8 + [C.c_size_t] + [C.c_int] * 3 + [C.c_void_p]
_GEMM_NT = [C.c_void_p] * 5 + [C.c_int] * 4 + [C.c_void_p]


def _ptr(t):
    return None if t is None else t.data_ptr()


def gemm(layout: int, epilogue: int, a: torch.Tensor, b: torch.Tensor, out: torch.Tensor, bias=None, aux=None, pre=None, part: int = 0, ws=None) -> torch.Tensor:
    """The general entry: layouts and epilogues of src/ops/gemm_sm100.cu; `part` is the address of partial_rows(M) x N floats;
    `ws` (uint8, its first 64 KiB zero, one stream at a time) lets deep products with few tiles split K."""
    M, Nn = out.shape
    K = a.shape[0] if layout == TN else a.shape[1]
    rc = _native("piccl_ops_gemm", _GEMM)(layout, epilogue, a.data_ptr(), b.data_ptr(), out.data_ptr(), _ptr(pre), _ptr(bias), _ptr(aux), part or None, _ptr(ws),
                                          ws.numel() if ws is not None else 0, M, Nn, K, _s())
    if rc != 0:
        raise RuntimeError(f"piccl_ops_gemm failed (code {rc}) for layout {layout} epilogue {epilogue} M={M} N={Nn} K={K}")
    _bump()
    return out


def partial_rows(M: int) -> int:
    """Rows of column sums that the GELU_GRAD epilogue leaves: one per 32 rows."""
    return (M + 31) // 32


def gemm_nt(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor, bias=None, gelu: bool = False, pre=None) -> torch.Tensor:
    """out[M, N] = act(x[M, K] @ w[N, K]^T + bias); `pre` (optional) receives the value before the activation"""
    M, K = x.shape
    Nn = w.shape[0]
    rc = _native("piccl_ops_gemm_bf16_nt_ex", _GEMM_NT)(x.data_ptr(), w.data_ptr(), out.data_ptr(), _ptr(pre), _ptr(bias), M, Nn, K, gelu, _s())
    if rc != 0:
        raise RuntimeError(f"piccl_ops_gemm_bf16_nt failed (code {rc}) for M={M} N={Nn} K={K}")
    _bump()
    return out


def gemm_nt_pair(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor, bias=None) -> torch.Tensor:
    """out[M, N] = x[M, K] @ w[N, K]^T + bias on CTA pairs, which is how every product of this module runs."""
    return gemm(NT, BIAS, x, w, out, bias=bias)


def pair_status() -> int:
    """0, or the role whose bounded wait ran out in a GEMM on this device (synchronises the device)."""
    return int(N.ops_lib().piccl_ops_gemm_status())
