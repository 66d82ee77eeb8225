"""Small, self-terminating workloads for ncu captures (one kernel, a few launches, well under a few GB):

    python benchmarks/profile_cases.py exec      # fused collective executor: 2 virtual ranks, ring all-reduce of 256 MiB fp32
    python benchmarks/profile_cases.py exec8     # the same among 8 virtual ranks, 32 MiB fp32 each
    python benchmarks/profile_cases.py flow      # data flow of a ring all-reduce, 8 virtual ranks, 32 MiB fp32 each
    python benchmarks/profile_cases.py exec_ll   # low-latency all-reduce, 8 virtual ranks, 16 KiB
    python benchmarks/profile_cases.py gemm      # tcgen05 GEMM 8192 x 8192 x 3584 bf16
    python benchmarks/profile_cases.py direct    # DIRECT all-reduce, 8 virtual ranks, 16 MiB fp32
    python benchmarks/profile_cases.py tp        # fused GEMM -> reduce-scatter, 2 virtual ranks, 4096 x 4096 x 2048
    python benchmarks/profile_cases.py ln        # residual-add + LayerNorm forward/backward, 8192 x 1024
    python benchmarks/profile_cases.py ce        # cross entropy forward+backward, 8192 x 50304
    python benchmarks/profile_cases.py nvls      # in-switch all-reduce kernel with the switch emulated: 4 virtual ranks, 64 MiB bf16 each
    python benchmarks/profile_cases.py llf       # low-latency executor: all-gather of 16 KiB per rank, 8 virtual ranks
    python benchmarks/profile_cases.py ag_gemm   # fused all-gather -> GEMM, 2 virtual ranks, 4096 x 2048 x 4096
    python benchmarks/profile_cases.py attention # causal attention forward and backward, 8 x 1024 tokens, 16 heads of 64 columns
    python benchmarks/profile_cases.py elementwise  # AdamW on 128 Mi parameters, bias + GELU forward / backward on 8192 x 4096, embedding 8192 x 1024, column sum

Typical capture (after the same command has exited 0 without ncu):
    ncu --set full --clock-control none -k regex:<kernel> -s 2 -c 2 -o <name> python benchmarks/profile_cases.py <case>
"""
from __future__ import annotations

import sys
from pathlib import Path

import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))


def _group8():
    """Eight ranks with FIFOs of 128 KiB slots for the 18 CTAs that each gets: 1.2 GiB of heaps for FIFOs and low-latency slots instead of 10."""
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    return LoopbackGroup(8, config=make_config(max_cta=18, nslot=4, slot_bytes=128 << 10, scratch_bytes=1 << 20)).slots_only()


def case_exec(ranks: int = 2, count: int = 64 << 20, algo: str = "RING"):
    from piccl_b200.parallel.comm import LoopbackGroup
    n = ranks
    g = LoopbackGroup(n).slots_only() if n == 2 else _group8()
    xs = [torch.ones(count, device="cuda") for _ in range(n)]
    outs = [torch.empty_like(x) for x in xs]
    for _ in range(4):
        g.run("allreduce", xs, outs, count, algo=algo)
    torch.cuda.synchronize()
    assert g.status().aborted == 0
    g.close()


def case_flow():
    n, count = 8, 8 << 20
    g = _group8().slots_only(False)
    xs = [torch.full((count,), float(r + 1), device="cuda") for r in range(n)]
    outs = [torch.empty_like(x) for x in xs]
    for _ in range(4):
        g.run("allreduce", xs, outs, count, algo="RING")
    torch.cuda.synchronize()
    assert g.status().aborted == 0 and float(outs[3][12345]) == n * (n + 1) / 2
    g.close()


def case_gemm():
    from piccl_b200.ops import gemm_sm100
    a = torch.randn(8192, 3584, device="cuda").to(torch.bfloat16)
    b = torch.randn(8192, 3584, device="cuda").to(torch.bfloat16)
    o = torch.empty(8192, 8192, device="cuda", dtype=torch.bfloat16)
    for _ in range(4):
        gemm_sm100.gemm_nt(a, b, o)
    torch.cuda.synchronize()


def case_direct():
    from piccl_b200.parallel.comm import LoopbackGroup
    n, count = 8, 4 << 20
    g = LoopbackGroup(n).slots_only()
    xs = [torch.full((count,), float(r + 1), device="cuda") for r in range(n)]
    outs = [torch.empty_like(x) for x in xs]
    for _ in range(4):
        g.run("allreduce", xs, outs, count, algo="DIRECT")
    torch.cuda.synchronize()
    assert g.status().aborted == 0 and float(outs[3][12345]) == n * (n + 1) / 2
    g.close()


def case_tp():
    from piccl_b200.parallel import tp
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    n, M, N, K = 2, 4096, 4096, 2048
    g = LoopbackGroup(n, config=make_config(tp_bytes=tp.workspace_bytes("gemm_rs", n, M, N, K))).slots_only()
    As = [torch.randn(M, K, device="cuda").to(torch.bfloat16) for _ in range(n)]
    Bs = [torch.randn(N, K, device="cuda").to(torch.bfloat16) for _ in range(n)]
    outs = [torch.empty(M // n, N, device="cuda", dtype=torch.bfloat16) for _ in range(n)]
    for _ in range(4):
        tp.gemm_rs_group(g, As, Bs, outs)
    torch.cuda.synchronize()
    g.close()


def case_nvls():
    """The kernel of the in-switch collectives on one GPU: the multimem instructions are replaced by loops over the virtual
    ranks' windows, everything else (bulk copies, warp groups, counters) is what runs on NVLink multicast windows."""
    from piccl_b200.parallel.comm import LoopbackGroup
    n, count = 4, 32 << 20
    g = LoopbackGroup(n)
    xs = [torch.ones(count, device="cuda", dtype=torch.bfloat16) for _ in range(n)]
    outs = [torch.empty_like(x) for x in xs]
    for _ in range(3):
        g.run("allreduce", xs, outs, count, algo="NVLS")
    torch.cuda.synchronize()
    assert g.status().aborted == 0 and g.stats().nvls_calls == 3 and float(outs[1][777]) == float(n)
    g.close()


def case_llf():
    n, count = 8, 4096
    g = _group8()
    xs = [torch.full((count,), float(r), device="cuda") for r in range(n)]
    outs = [torch.empty(n * count, device="cuda") for _ in range(n)]
    for _ in range(4):
        g.run("allgather", xs, outs, count, algo="RING")
    torch.cuda.synchronize()
    assert g.status().aborted == 0 and float(outs[2][5 * count + 1]) == 5.0
    g.close()


def case_ag_gemm():
    from piccl_b200.parallel import tp
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    n, M, N, K = 2, 4096, 2048, 4096
    g = LoopbackGroup(n, config=make_config(tp_bytes=tp.workspace_bytes("ag_gemm", n, M, N, K))).slots_only()
    As = [torch.randn(M // n, K, device="cuda").to(torch.bfloat16) for _ in range(n)]
    Bs = [torch.randn(N, K, device="cuda").to(torch.bfloat16) for _ in range(n)]
    outs = [torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(n)]
    for _ in range(4):
        tp.ag_gemm_group(g, As, Bs, outs)
    torch.cuda.synchronize()
    assert all(tp.tp_status(h) == 0 for h in g._hs)
    g.close()


def case_elementwise():
    """The memory-bound model kernels of src/ops/elementwise.cu on GPT-2-medium shapes (operands far larger than L2)."""
    from piccl_b200 import ops
    n = 128 << 20
    p = torch.zeros(n, device="cuda", dtype=torch.bfloat16); master = torch.zeros(n, device="cuda")
    m, v = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    g = torch.full((n,), 0.01, device="cuda", dtype=torch.bfloat16)
    T, H, C_ = 8192, 4096, 1024
    h = torch.randn(T, H, device="cuda").bfloat16(); bias = torch.randn(H, device="cuda").bfloat16()
    h_out, act, dh = torch.empty_like(h), torch.empty_like(h), torch.empty_like(h)
    idx = torch.randint(0, 50257, (T,), device="cuda")
    wte = torch.randn(50304, C_, device="cuda").bfloat16(); wpe = torch.randn(1024, C_, device="cuda").bfloat16()
    emb = torch.empty(T, C_, device="cuda", dtype=torch.bfloat16)
    cs = torch.empty(H, device="cuda", dtype=torch.bfloat16)
    for step in range(1, 3):
        ops.adamw(p, master, m, v, g, 3e-4, 0.9, 0.95, 1e-8, 0.1, step)
        ops.bias_gelu_fwd(h, bias, h_out, act)
        ops.gelu_bwd(act, h_out, dh)
        ops.embed_fwd(idx, wte, wpe, emb, 1024)
        ops.colsum(dh, cs)
    torch.cuda.synchronize()
    assert torch.isfinite(cs.float()).all() and float(master.abs().max()) > 0


def case_attention():
    from piccl_b200 import _native as N
    from piccl_b200 import ops
    B, S, H = 8, 1024, 16
    qkv, dout = torch.randn(B * S, 3 * H * 64, device="cuda").bfloat16(), torch.randn(B * S, H * 64, device="cuda").bfloat16()
    out, dqkv, lse = torch.empty_like(dout), torch.empty_like(qkv), torch.empty(B * H, S, device="cuda")
    scratch, part = torch.empty(2 * B * H * S, device="cuda"), torch.empty(B * S // 128, 3 * H * 64, device="cuda")
    for _ in range(4):
        ops.attention_fwd(qkv, out, lse, B)
        ops.attention_bwd(qkv, out, dout, lse, scratch, dqkv, part, B)
    torch.cuda.synchronize()
    assert N.ops_lib().piccl_ops_attn_status() == 0 and torch.isfinite(dqkv.float()).all()


def case_ln():
    from piccl_b200 import ops
    T, C = 8192 * 4, 1024
    x, r = torch.randn(T, C, device="cuda").bfloat16(), torch.randn(T, C, device="cuda").bfloat16()
    g_, b_ = torch.ones(C, device="cuda").bfloat16(), torch.zeros(C, device="cuda").bfloat16()
    s, y = torch.empty_like(x), torch.empty_like(x)
    mean, rstd = torch.empty(T, device="cuda"), torch.empty(T, device="cuda")
    dx, dg, db = torch.empty_like(x), torch.empty_like(g_), torch.empty_like(b_)
    for _ in range(4):
        ops.layernorm_fwd(x, r, g_, b_, s, y, mean, rstd)
        ops.layernorm_bwd(y, s, g_, mean, rstd, r, dx, dg, db)
    torch.cuda.synchronize()


def case_ce():
    from piccl_b200 import ops
    T, V, Vp = 8192, 50257, 50304
    logits = torch.randn(T, Vp, device="cuda").bfloat16()
    tgt = torch.randint(0, V, (T,), device="cuda")
    loss = torch.empty(T, device="cuda")
    for _ in range(4):
        ops.cross_entropy_fwd_bwd(logits, tgt, loss, V, 1.0 / T)
    torch.cuda.synchronize()


if __name__ == "__main__":
    which = sys.argv[1] if len(sys.argv) > 1 else "exec"
    {"exec": case_exec, "flow": case_flow, "exec8": lambda: case_exec(8, 8 << 20), "exec_ll": lambda: case_exec(8, 4096, "PRD"), "gemm": case_gemm, "direct": case_direct, "tp": case_tp, "ln": case_ln, "ce": case_ce, "nvls": case_nvls, "llf": case_llf, "ag_gemm": case_ag_gemm, "attention": case_attention, "elementwise": case_elementwise}[which]()
    print(f"profile case {which} done")
