"""GPT-2 written against the framework's own kernels, with a hand-scheduled
backward pass.

Why not autograd: the backward pass is where data-parallel communication
overlaps with compute, so the model itself decides when a contiguous range of
the flat gradient buffer is final and hands it to the bucketed all-reduce
(`on_grads_ready`).  Parameters and gradients live in two flat bf16 buffers laid
out in the order in which the backward pass finishes them; buckets are therefore
plain slices and never copied.  fp32 master weights and AdamW moments live in
flat fp32 buffers and are updated by one fused kernel per parameter group.

The step itself is native (src/model/gpt2_step.cc): residual-add + LayerNorm
(forward / backward), GEMMs with fused GELU, bias gradients, embedding, softmax cross
entropy with in-place gradient and AdamW are this framework's CUDA kernels (src/ops);
for heads of 64 columns so are the backward pass of attention and its forward pass in an
evaluation, at the sizes where they are the faster kernels (the rest, and other back ends
that the program asks PyTorch for, goes through PyTorch's fused kernels).

The reference has no model code at all; this module exists for the end-to-end
data-parallel benchmark (GPT-2 medium under bucketed gradient all-reduce).
"""
from __future__ import annotations

import ctypes as C
import math
import threading
import weakref
from dataclasses import dataclass
from typing import Callable, Optional

import torch

from .. import _native as N
from .. import ops
from ..ops import gemm

_READY = C.CFUNCTYPE(None, C.c_longlong)
_MAX_GRAPHS = 8


class _Desc(C.Structure):       # the native step's description of a model (src/model/gpt2_step.cc)
    _fields_ = [(n, C.c_int) for n in ("L", "C", "H", "V", "Vp", "seq_len")] + [("eps", C.c_float), ("pad", C.c_int), ("p", C.c_void_p), ("g", C.c_void_p), ("off", C.c_void_p)]


# What a program may switch between two steps and attention or the library products look at in each call: a step captured under one setting is not
# replayed under another.  (The functions behind the torch.backends properties, which take three times as long: half a microsecond.)
_SETTINGS = [getattr(torch._C, f"_get_{n}") for n in ("cudnn_sdp_enabled", "flash_sdp_enabled", "mem_efficient_sdp_enabled", "math_sdp_enabled", "deterministic_algorithms",
                                                      "cublas_allow_bf16_reduced_precision_reduction")]


def _library_settings() -> tuple:
    return tuple([f() for f in _SETTINGS] + torch._C._get_sdp_priority_order())      # (the order in which attention's back ends are tried)


@dataclass
class GPT2Config:
    vocab_size: int = 50257
    seq_len: int = 1024
    n_layer: int = 24
    n_head: int = 16
    d_model: int = 1024
    ln_eps: float = 1e-5

    @property
    def padded_vocab(self) -> int:
        return (self.vocab_size + 127) // 128 * 128

    @staticmethod
    def medium() -> "GPT2Config":
        return GPT2Config()

    @staticmethod
    def tiny() -> "GPT2Config":
        return GPT2Config(vocab_size=1000, seq_len=128, n_layer=2, n_head=4, d_model=256)


_DECAY = ("w_qkv", "w_o", "w_fc", "w_proj")
_NODECAY = ("ln1_g", "ln1_b", "b_qkv", "b_o", "ln2_g", "ln2_b", "b_fc", "b_proj")


class GPT2:
    def __init__(self, cfg: GPT2Config, device="cuda", seed: int = 0):
        self.cfg = cfg
        self.device = torch.device(device)
        D, L, Vp, S = cfg.d_model, cfg.n_layer, cfg.padded_vocab, cfg.seq_len
        shapes = {"w_qkv": (3 * D, D), "w_o": (D, D), "w_fc": (4 * D, D), "w_proj": (D, 4 * D), "ln1_g": (D,), "ln1_b": (D,),
                  "b_qkv": (3 * D,), "b_o": (D,), "ln2_g": (D,), "ln2_b": (D,), "b_fc": (4 * D,), "b_proj": (D,)}
        # flat order = order in which the backward pass completes gradients
        layout = [("lnf_g", (D,), False), ("lnf_b", (D,), False)]
        for l in reversed(range(L)):
            layout += [(f"h{l}.{n}", shapes[n], True) for n in _DECAY]
            layout += [(f"h{l}.{n}", shapes[n], False) for n in _NODECAY]
        layout += [("wpe", (S, D), True), ("wte", (Vp, D), True)]
        total = sum(math.prod(s) for _, s, _ in layout)
        self.flat_p = torch.zeros(total, dtype=torch.bfloat16, device=self.device)
        self.flat_g = torch.zeros(total, dtype=torch.bfloat16, device=self.device)
        self.p: dict[str, torch.Tensor] = {}
        self.g: dict[str, torch.Tensor] = {}
        self.offset: dict[str, tuple[int, int]] = {}
        self.groups: list[tuple[int, int, bool]] = []     # (begin, end, decay) runs for the optimizer
        off = 0
        for name, shape, decay in layout:
            n = math.prod(shape)
            self.p[name] = self.flat_p[off:off + n].view(shape)
            self.g[name] = self.flat_g[off:off + n].view(shape)
            self.offset[name] = (off, off + n)
            if self.groups and self.groups[-1][2] == decay and self.groups[-1][1] == off:
                self.groups[-1] = (self.groups[-1][0], off + n, decay)
            else:
                self.groups.append((off, off + n, decay))
            off += n
        self.n_params = total
        self._init_weights(seed)
        self.master = self.flat_p.float()
        self.m = torch.zeros_like(self.master)
        self.v = torch.zeros_like(self.master)
        self.step_count = 0
        self.step_dev = torch.zeros(1, dtype=torch.int32, device=self.device)     # the same counter on the device (graph replay)
        # decaying and non-decaying runs alternate; their ends in packs of 8 elements
        self._run_ends = torch.tensor([e // 8 for _, e, _ in self.groups], dtype=torch.int32, device=self.device)
        self._ticket = torch.zeros(1, dtype=torch.int32, device=self.device)
        self._handle = None
        self._arena = None
        self._graphs: dict = {}      # captured steps, at most _MAX_GRAPHS, which share the memory of their attention outputs
        self._graph_pool = None
        self.replays = 0             # steps replayed so far
        self._seen: dict = {}        # how often a step was issued call by call; -1: it cannot be captured
        self._counts = (C.c_longlong * 4)()
        if self.device.type == "cuda":       # PyTorch settles its order of attention's back ends when it is first asked for one; captured steps are known by that order too
            q = torch.empty(1, 1, 8, 64, dtype=torch.bfloat16, device=self.device)
            torch._fused_sdp_choice(q, q, q, None, 0.0, True)

    # ------------------------------------------------------------------ setup
    def _init_weights(self, seed: int) -> None:
        cfg = self.cfg
        gen = torch.Generator(device=self.device).manual_seed(seed)
        for name, t in self.p.items():
            base = name.split(".")[-1]
            if base in ("ln1_g", "ln2_g", "lnf_g"):
                t.fill_(1.0)
            elif base.startswith("b_") or base.endswith("_b"):
                t.zero_()
            else:
                std = 0.02 / math.sqrt(2 * cfg.n_layer) if base in ("w_o", "w_proj") else 0.02
                t.copy_((torch.randn(t.shape, generator=gen, device=self.device, dtype=torch.float32) * std).to(torch.bfloat16))
        self.p["wte"][cfg.vocab_size:].zero_()

    # ------------------------------------------------------------------ forward + backward
    def _native(self):
        if self._handle is None:
            cfg, L = self.cfg, self.cfg.n_layer
            names = ["lnf_g", "lnf_b", "wpe", "wte"] + [f"h{l}.{n}" for l in range(L)
                                                        for n in _DECAY + _NODECAY]
            offs = (C.c_longlong * len(names))(*[self.offset[n][0] for n in names])
            d = _Desc(L, cfg.d_model, cfg.n_head, cfg.vocab_size, cfg.padded_vocab, cfg.seq_len, cfg.ln_eps, 0, self.flat_p.data_ptr(), self.flat_g.data_ptr(), C.cast(offs, C.c_void_p))
            lib = N.model_lib()
            self._handle = lib.piccl_gpt2_create(C.byref(d))
            self._finalizer = weakref.finalize(self, lib.piccl_gpt2_destroy, self._handle)
        return self._handle

    def forward_backward(self, idx: torch.Tensor, targets: torch.Tensor,
                         on_grads_ready: Optional[Callable[[int], None]] = None, loss_only: bool = False) -> torch.Tensor:
        """One training micro-step: returns the mean loss (fp32, on device) and leaves the
        gradients in `flat_g`.  `on_grads_ready(end)` is called whenever flat_g[:end] is final.
        The loss is not a number where a kernel on this device gave up on a bounded wait (the gradients are void then): ops.raise_if_a_wait_ran_out() tells."""
        loss, shared = self._step(idx, targets, on_grads_ready, loss_only)
        return loss.clone() if shared else loss

    def _step(self, idx, targets, on_grads_ready=None, loss_only=False):
        """(loss, whether the tensor is overwritten by the next step)

        A step that comes a third time with the same shape on the same input buffers (a trainer's, which it fills anew for each batch) is captured
        into a CUDA graph and replayed from then on: issued call by call, the launches bound every model of a few hundred columns, and a replay
        also runs the weight gradients on a second stream.  While a capture is open another thread's device-wide synchronisation would fail: there is none
        in a program of several threads.  Inputs elsewhere, a step that reports finished gradients, and one inside somebody else's capture run as before."""
        B, S = idx.shape
        idx = idx.reshape(-1).contiguous()
        targets = targets.reshape(-1).contiguous()
        if idx.dtype != torch.int64 or targets.dtype != torch.int64 or targets.numel() != B * S or S > self.cfg.seq_len:
            raise ValueError("token ids and targets are int64 tensors of one shape, at most seq_len long")
        if self.cfg.d_model % self.cfg.n_head:      # the native step would take heads of d_model // n_head columns
            raise RuntimeError(f"{self.cfg.d_model} columns are not {self.cfg.n_head} heads of one width")
        if on_grads_ready is not None and not loss_only:
            return self._issue(idx, targets, B, S, loss_only, 0, on_grads_ready), False
        key = (idx.data_ptr(), targets.data_ptr(), B, S, loss_only, gemm.backend_code(), _library_settings())
        seen = self._seen.get(key, 0)
        if seen == -1 or torch.cuda.is_current_stream_capturing():
            return self._issue(idx, targets, B, S, loss_only, 0), False
        arena = N.model_lib().piccl_gpt2_arena(self._native())
        if arena != self._arena:                 # a larger shape moved the activations: what was captured before points to the old ones
            self._arena = arena
            self._graphs.clear()
        entry = self._graphs.get(key)
        if entry is None and seen >= 2 and len(self._graphs) < _MAX_GRAPHS and threading.active_count() == 1:
            entry = self._capture(idx, targets, B, S, loss_only)
            if entry is not None:
                self._graphs[key] = entry
            else:
                self._seen[key] = -1             # a part of this step cannot be captured: issued call by call from now on
        elif entry is None:
            if len(self._seen) > 4096:
                self._seen.clear()
            self._seen[key] = min(seen + 1, 2)
        if entry is None:                        # the call before the capture runs what will be captured: libraries set themselves up for it
            return self._issue(idx, targets, B, S, loss_only, int(seen == 1)), False
        graph, loss, counts = entry
        graph.replay()
        self.replays += 1
        ops._bump(counts[0])
        gemm.count(counts[1], counts[2])
        return loss, True

    def _capture(self, idx, targets, B, S, loss_only):
        if not self._graphs:                     # a pool that no graph uses any more cannot be taken up again
            self._graph_pool = torch.cuda.graph_pool_handle()
        graph, cur = torch.cuda.CUDAGraph(), torch.cuda.current_stream()
        stream = torch.cuda.ExternalStream(N.model_lib().piccl_gpt2_capture_stream(self._native()), device=self.device)
        launched, products = ops.launch_count(), gemm.counts()
        stream.wait_stream(cur)
        ok = False
        with torch.cuda.stream(stream):
            graph.capture_begin(pool=self._graph_pool, capture_error_mode="thread_local")
            try:
                loss = self._issue(idx, targets, B, S, loss_only, 1)
                ok = True
            except RuntimeError:
                pass
            finally:                             # also when an interrupt comes here: the stream must not stay in capture
                try:
                    graph.capture_end()
                except RuntimeError:
                    ok = False
        cur.wait_stream(stream)
        after = gemm.counts()
        counts = (ops.launch_count() - launched, after["tcgen05"] - products["tcgen05"], after["cublas"] - products["cublas"])
        ops._bump(-counts[0])                    # the capture itself ran nothing
        gemm.count(-counts[1], -counts[2])
        if not ok or N.model_lib().piccl_gpt2_arena(self._native()) != self._arena:
            return None
        return graph, loss, counts

    def _issue(self, idx, targets, B, S, loss_only, captured, on_grads_ready=None) -> torch.Tensor:
        loss = torch.empty((), dtype=torch.float32, device=self.device)
        raised: list = []
        cb = None
        if on_grads_ready is not None:
            def ready(end):
                try:
                    if not raised:
                        on_grads_ready(end)
                except BaseException as e:      # an exception may not unwind through the native frames: raised again below
                    raised.append(e)
            cb = _READY(ready)
        rc = N.model_lib().piccl_gpt2_run(self._native(), idx.data_ptr(), targets.data_ptr(), B, S, loss.data_ptr(), int(not loss_only), gemm.backend_code(), captured,
                                          C.cast(cb, C.c_void_p) if cb is not None else None, self._counts)
        ops._bump(self._counts[0])
        gemm.count(self._counts[1], self._counts[2])
        if raised:
            raise raised[0]
        if rc != 0:
            raise RuntimeError(f"GPT-2 step failed (code {rc}): {(N.model_lib().piccl_gpt2_error() or b'').decode()}")
        return loss

    # ------------------------------------------------------------------ optimizer
    def optimizer_step(self, lr: float = 3e-4, betas=(0.9, 0.95), eps: float = 1e-8, weight_decay: float = 0.1) -> None:
        """Fused AdamW over the flat buffers in one launch (one per run of parameters in models of more than some 500 layers); the step number lives
        on the device so that it can be replayed."""
        self.step_count += 1
        if len(self.groups) > ops.MAX_ADAMW_RUNS:
            self.step_dev.add_(1)
            for b, e, decay in self.groups:
                ops.adamw_devstep(self.flat_p[b:e], self.master[b:e], self.m[b:e], self.v[b:e], self.flat_g[b:e], lr, betas[0], betas[1], eps, weight_decay if decay else 0.0,
                                  self.step_dev)
            return
        ops.adamw_runs(self.flat_p, self.master, self.m, self.v, self.flat_g, self._run_ends, 0 if self.groups[0][2] else 1, lr, betas[0], betas[1], eps, weight_decay,
                       self.step_dev, self._ticket)

    @torch.no_grad()
    def loss(self, idx: torch.Tensor, targets: torch.Tensor) -> torch.Tensor:
        return self.forward_backward(idx, targets, loss_only=True)

    # ------------------------------------------------------------------ interchange with a plain PyTorch module
    def state_dict(self) -> dict:
        """Parameters under the names of a conventional GPT-2 module (unpadded vocabulary)."""
        cfg = self.cfg
        sd = {"wte.weight": self.p["wte"][:cfg.vocab_size].clone(), "wpe.weight": self.p["wpe"].clone(),
              "ln_f.weight": self.p["lnf_g"].clone(), "ln_f.bias": self.p["lnf_b"].clone()}
        names = {"ln1_g": "ln_1.weight", "ln1_b": "ln_1.bias", "w_qkv": "attn.c_attn.weight", "b_qkv": "attn.c_attn.bias", "w_o": "attn.c_proj.weight",
                 "b_o": "attn.c_proj.bias", "ln2_g": "ln_2.weight", "ln2_b": "ln_2.bias", "w_fc": "mlp.c_fc.weight", "b_fc": "mlp.c_fc.bias",
                 "w_proj": "mlp.c_proj.weight", "b_proj": "mlp.c_proj.bias"}
        for l in range(cfg.n_layer):
            for k, v in names.items():
                sd[f"h.{l}.{v}"] = self.p[f"h{l}.{k}"].clone()
        return sd
