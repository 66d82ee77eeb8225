"""Python front ends of the model kernels in libpiccl_ops.so.

Every function launches hand-written CUDA on the current stream and fails
loudly if the native library is missing; there is no PyTorch fallback.  A
process-wide launch counter (`launch_count()`) records how many of these
kernels were started, which the benchmark reports.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from .. import _native as N

_launches = 0


def launch_count() -> int:
    return _launches


def _bump(n: int = 1) -> None:
    global _launches
    _launches += n


def current_stream_ptr(device=None) -> int:
    """The raw handle of the current stream (of the current device), without building a Stream object (0.2 us instead of 3.4)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice() if device is None else device)


_s = current_stream_ptr


def _p(t: Optional[torch.Tensor]) -> C.c_void_p:
    return C.c_void_p(t.data_ptr() if t is not None else 0)


def _chk(rc: int, name: str) -> None:
    if rc != 0:
        raise RuntimeError(f"{name} failed (code {rc})")


def raise_if_a_wait_ran_out() -> None:
    """Raises if a GEMM or attention kernel on the current device gave up on a bounded wait since the last such report: what it should have written is void, and
    so are results computed from it.  Losses of GPT2 are not a number from then on until it is reported here.  Synchronises."""
    words = (C.c_int * 2)()
    _chk(N.ops_lib().piccl_ops_status(words, 1), "status")
    if any(words):
        raise RuntimeError("a kernel gave up on a wait: " + ", ".join(f"{n} (role {w})" for n, w in zip(("GEMM", "attention"), words) if w))


_ws: dict = {}


def _workspace(n_floats: int, device) -> torch.Tensor:
    key = (device, "f32")
    w = _ws.get(key)
    if w is None or w.numel() < n_floats:
        w = torch.empty(max(n_floats, 1 << 20), dtype=torch.float32, device=device)
        _ws[key] = w
    return w


def layernorm_fwd(x, res, gamma, beta, sum_out, y, mean, rstd, eps: float = 1e-5):
    """y = LN(x + res) * gamma + beta; sum_out = x + res (either may be None)."""
    rows, Cc = x.shape
    _chk(N.ops_lib().piccl_ops_ln_fwd(_p(x), _p(res), _p(gamma), _p(beta), _p(sum_out), _p(y), _p(mean), _p(rstd), rows, Cc, C.c_float(eps), C.c_void_p(_s())), "ln_fwd")
    _bump()


class _FinishJob(C.Structure):
    _fields_ = [("part", C.c_void_p), ("out", C.c_void_p), ("nparts", C.c_int), ("C", C.c_int), ("accumulate", C.c_int), ("pad", C.c_int)]


def layernorm_bwd(dy, xin, gamma, mean, rstd, dres, dx, dgamma, dbeta, accumulate: bool = False, rows_per_block: int = 32):
    """dx = dLN(dy) + dres; dgamma / dbeta (bf16) written or accumulated.  `rows_per_block` is taken for callers that pass it: the kernel's
    persistent grid splits the rows by itself."""
    rows, Cc = dy.shape
    n = N.ops_lib().piccl_ops_ln_bwd_parts(rows, Cc)
    ws = _workspace(2 * max(n, 1) * Cc, dy.device)
    _chk(N.ops_lib().piccl_ops_ln_bwd(_p(dy), _p(xin), _p(gamma), _p(mean), _p(rstd), _p(dres), _p(dx), _p(ws), 0, rows, Cc, C.c_void_p(_s())), "ln_bwd")
    jobs = (_FinishJob * 2)(*[(ws.data_ptr() + 4 * i * n * Cc, o.data_ptr(), n, Cc, int(accumulate), 0) for i, o in enumerate((dgamma, dbeta))])
    _chk(N.ops_lib().piccl_ops_finish_parts(jobs, 2, C.c_void_p(_s())), "finish_parts")
    _bump(2)


def bias_gelu_fwd(h, bias, h_out, g):
    rows, Cc = h.shape
    _chk(N.ops_lib().piccl_ops_bias_gelu_fwd(_p(h), _p(bias), _p(h_out), _p(g), C.c_longlong(rows), Cc, C.c_void_p(_s())), "bias_gelu_fwd")
    _bump()


def gelu_bwd(dg, h, dh):
    # element by element: any shape will do, as long as the kernel gets rows of whole 16-byte words
    n = h.numel()
    Cc = h.shape[1] if h.dim() == 2 and h.shape[1] % 8 == 0 else min(n & -n, 2048) or 8
    rows = n // Cc
    _chk(N.ops_lib().piccl_ops_gelu_bwd(_p(dg), _p(h), _p(dh), C.c_void_p(0), C.c_longlong(rows), Cc, C.c_void_p(_s())), "gelu_bwd")
    _bump()


def colsum(x, out, accumulate: bool = False, rows_per_block: int = 256):
    """out[c] (+)= sum_r x[r, c]  (bias gradient)."""
    rows, Cc = x.shape
    nparts = (rows + rows_per_block - 1) // rows_per_block
    ws = _workspace(nparts * Cc, x.device)
    _chk(N.ops_lib().piccl_ops_colsum(_p(x), _p(out), _p(ws), rows, Cc, rows_per_block, int(accumulate), C.c_void_p(_s())), "colsum")
    _bump(2)


def cross_entropy_fwd_bwd(logits, targets, loss_rows, vocab: int, gscale: float):
    """loss_rows[r] = CE(logits[r, :vocab], targets[r]); logits <- d(loss)/d(logits) * gscale, in place."""
    rows, Vp = logits.shape
    _chk(N.ops_lib().piccl_ops_ce_fwd_bwd(_p(logits), _p(targets), _p(loss_rows), rows, vocab, Vp, C.c_float(gscale), C.c_void_p(_s())), "ce_fwd_bwd")
    _bump()


def _attention_operands(batch: int, qkv, out, rows_like=(), floats=()) -> tuple[int, int]:
    """(positions, heads) of packed rows; everything that the kernels do not look at: shapes, types, layout and device."""
    if out.dim() != 2 or out.shape[1] == 0 or out.shape[1] % 64 or batch <= 0 or out.shape[0] == 0 or out.shape[0] % batch:
        raise ValueError(f"attention: {tuple(out.shape)} is not [{batch} * positions, heads * 64]")
    rows, Cc = out.shape
    for t, width in ((qkv, 3 * Cc), (out, Cc), *rows_like):
        if t.numel() != rows * width or t.dtype != torch.bfloat16 or not t.is_contiguous():
            raise ValueError(f"attention: contiguous bf16 [{rows}, {width}] wanted, got {t.dtype} {tuple(t.shape)}")
    S = rows // batch
    heads, pad = Cc // 64, (S + 127) // 128 * 128
    for t, n in ((t, f(S, heads, pad)) for t, f in floats if t is not None):
        if t.numel() < n or t.dtype != torch.float32 or not t.is_contiguous():
            raise ValueError(f"attention: {n} contiguous floats wanted, got {t.dtype} {tuple(t.shape)}")
    for t in (qkv, out, *(t for t, _ in rows_like), *(t for t, _ in floats if t is not None)):
        if not t.is_cuda or t.device != qkv.device:
            raise ValueError("attention: tensors of one CUDA device wanted")
    return S, heads


def attention_fwd(qkv, out, lse, batch: int):
    """Causal attention of packed rows [batch * S, 3 * heads * 64] -> [batch * S, heads * 64]; lse: [batch * heads, S] floats, the logarithm of each row's sum of
    exponentials, which attention_bwd takes, or None."""
    S, heads = _attention_operands(batch, qkv, out, floats=[(lse, lambda S, h, pad: batch * h * S)])
    _chk(N.ops_lib().piccl_ops_attn_fwd(_p(qkv), _p(out), _p(lse), batch, S, heads, C.c_void_p(_s())), "attn_fwd")
    _bump()


def attention_bwd(qkv, out, dout, lse, scratch, dqkv, part, batch: int):
    """dqkv, the gradient of the packed rows, and in part its partial column sums: one row per batch entry and 128 positions.
    lse as attention_fwd leaves it; scratch: 2 * batch * heads * (S rounded up to 128) floats."""
    if lse is None or scratch is None or part is None:
        raise ValueError("attention: the backward pass takes lse, scratch and part")
    S, heads = _attention_operands(batch, qkv, out, [(dout, out.shape[-1]), (dqkv, 3 * out.shape[-1])],
                                   [(lse, lambda S, h, pad: batch * h * S), (scratch, lambda S, h, pad: 2 * batch * h * pad), (part, lambda S, h, pad: batch * (pad // 128) * 3 * h * 64)])
    _chk(N.ops_lib().piccl_ops_attn_bwd(_p(qkv), _p(out), _p(dout), _p(lse), _p(scratch), _p(dqkv), _p(part), batch, S, heads, C.c_void_p(_s())), "attn_bwd")
    _bump(2)


def adamw(p, master, m, v, g, lr: float, b1: float, b2: float, eps: float, wd: float, step: int, gscale: float = 1.0):
    _chk(N.ops_lib().piccl_ops_adamw(_p(p), _p(master), _p(m), _p(v), _p(g), C.c_longlong(p.numel()), C.c_float(lr), C.c_float(b1), C.c_float(b2),
                                     C.c_float(eps), C.c_float(wd), step, C.c_float(gscale), C.c_void_p(_s())), "adamw")
    _bump()


def adamw_devstep(p, master, m, v, g, lr: float, b1: float, b2: float, eps: float, wd: float, step_dev, gscale: float = 1.0):
    """AdamW with the step number in a device int32 tensor (replayable from a CUDA graph)."""
    _chk(N.ops_lib().piccl_ops_adamw_devstep(_p(p), _p(master), _p(m), _p(v), _p(g), C.c_longlong(p.numel()), C.c_float(lr), C.c_float(b1), C.c_float(b2),
                                             C.c_float(eps), C.c_float(wd), _p(step_dev), C.c_float(gscale), C.c_void_p(_s())), "adamw_devstep")
    _bump()


MAX_ADAMW_RUNS = 1024      # runs that the kernel keeps in shared memory (kMaxRuns)


def adamw_runs(p, master, m, v, g, ends, decay_parity: int, lr: float, b1: float, b2: float, eps: float, wd: float, step_dev, ticket):
    """AdamW over flat buffers in one launch: run i ends before pack `ends[i]` of 8 elements (device int32), runs of parity `decay_parity` decay;
    `step_dev` (device int32, steps done so far) is advanced by the launch, `ticket` is a device int32 that holds zero."""
    _chk(N.ops_lib().piccl_ops_adamw_runs(_p(p), _p(master), _p(m), _p(v), _p(g), C.c_longlong(p.numel()), _p(ends), ends.numel(), decay_parity, C.c_float(lr), C.c_float(b1),
                                          C.c_float(b2), C.c_float(eps), C.c_float(wd), _p(step_dev), _p(ticket), C.c_void_p(_s())), "adamw_runs")
    _bump()


def embed_fwd(idx, wte, wpe, out, seq: int):
    rows, Cc = out.shape
    _chk(N.ops_lib().piccl_ops_embed_fwd(_p(idx), _p(wte), _p(wpe), _p(out), rows, seq, Cc, C.c_void_p(_s())), "embed_fwd")
    _bump()


def wpe_bwd(dx, dwpe, batch: int, seq: int, accumulate: bool = False):
    _chk(N.ops_lib().piccl_ops_wpe_bwd(_p(dx), _p(dwpe), batch, seq, seq, dx.shape[1], int(accumulate), C.c_void_p(_s())), "wpe_bwd")
    _bump()


def wte_bwd(idx, dx, stage, dwte):
    rows, Cc = dx.shape
    _chk(N.ops_lib().piccl_ops_wte_bwd(_p(idx), _p(dx), _p(stage), _p(dwte), rows, C.c_longlong(dwte.shape[0]), Cc, C.c_void_p(_s())), "wte_bwd")
    _bump(2)
