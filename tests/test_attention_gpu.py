"""The attention kernels (src/ops/attention.cu) against attention in fp64, at the edges of their tiles of 128 rows and steps of 64, forward and backward."""
import sys
from pathlib import Path

import pytest
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
pytestmark = pytest.mark.gpu


def _reference(qkv, dout, B, S, H):
    x = qkv.double().view(B, S, 3, H, 64).requires_grad_(True)
    q, k, v = (x[:, :, i].transpose(1, 2) for i in range(3))
    s = (q @ k.transpose(2, 3)) / 8
    s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    out = (s.softmax(-1) @ v).transpose(1, 2).reshape(B * S, H * 64)
    out.backward(dout.double())
    return out.detach(), torch.logsumexp(s.detach(), -1), x.grad.view(B * S, 3 * H * 64)


def _run(qkv, dout, B, S, H):
    from piccl_b200 import ops
    from piccl_b200 import _native as N
    pad = (S + 127) // 128 * 128
    nan = float("nan")
    out, dqkv = torch.full_like(dout, nan), torch.full_like(qkv, nan)
    lse, scratch = torch.full((B * H, S), nan, device="cuda"), torch.full((2 * B * H * pad,), nan, device="cuda")
    part = torch.full((B * pad // 128, 3 * H * 64), nan, device="cuda")
    ops.attention_fwd(qkv, out, lse, B)
    ops.attention_bwd(qkv, out, dout, lse, scratch, dqkv, part, B)
    assert N.ops_lib().piccl_ops_attn_status() == 0, "a bounded wait ran out"
    return out, lse, dqkv, part


@pytest.mark.parametrize("B,S,H,sigma", [
    (1, 1, 1, 1.0), (2, 63, 3, 1.0), (1, 64, 2, 1.0), (3, 65, 1, 1.0), (2, 127, 4, 1.0), (1, 128, 1, 1.0), (2, 129, 2, 1.0), (2, 191, 1, 1.0), (1, 193, 5, 1.0),
    (3, 777, 2, 1.0), (2, 1000, 2, 6.0),      # steep rows: the maximum rises again and again
    (8, 1024, 16, 1.0),                       # more CTAs than the chip holds at once
])
def test_attention_matches_fp64(B, S, H, sigma):
    gen = torch.Generator(device="cuda").manual_seed(B * S + H)
    qkv = (torch.randn(B * S, 3 * H * 64, generator=gen, device="cuda") * sigma).bfloat16()
    dout = torch.randn(B * S, H * 64, generator=gen, device="cuda").bfloat16()
    out, lse, dqkv, part = _run(qkv, dout, B, S, H)
    want, want_lse, want_d = _reference(qkv, dout, B, S, H)
    # probabilities, score gradients, outputs and gradients are rounded to bf16 (2^-9 each), the sum o * do takes the rounded output
    assert (out.double() - want).norm() <= 2 ** -8 * want.norm()
    assert (lse.view(B, H, S).double() - want_lse).abs().max() <= 1e-4 * max(1.0, sigma * sigma)
    for i in range(3):
        cols = slice(i * H * 64, (i + 1) * H * 64)
        assert (dqkv[:, cols].double() - want_d[:, cols]).norm() <= 2 ** -6 * want_d[:, cols].norm(), i
    sums = dqkv.float().view(B, S, -1)
    tiles = part.view(B, -1, part.shape[1])
    for t in range(tiles.shape[1]):
        w = sums[:, 128 * t:128 * (t + 1)]
        assert (tiles[:, t] - w.sum(1)).abs().max() <= 128 * 2 ** -23 * w.abs().sum(1).max()
    again = _run(qkv, dout, B, S, H)
    assert all(torch.equal(x, y) for x, y in zip((out, lse, dqkv, part), again))


def test_rows_of_one_batch_entry_do_not_see_another():
    """A tile that reaches beyond the last row of a batch entry ends there: infinities in the next entry stay there."""
    B, S, H = 2, 100, 2
    gen = torch.Generator(device="cuda").manual_seed(0)
    qkv = torch.randn(B * S, 3 * H * 64, generator=gen, device="cuda").bfloat16()
    dout = torch.randn(B * S, H * 64, generator=gen, device="cuda").bfloat16()
    clean = _run(qkv, dout, B, S, H)
    qkv[S:] = float("inf")
    dout[S:] = float("inf")
    dirty = _run(qkv, dout, B, S, H)
    assert torch.equal(clean[0][:S], dirty[0][:S]) and torch.equal(clean[2][:S], dirty[2][:S])
    assert not torch.isfinite(dirty[0][S:]).any()


def test_what_is_not_a_number_stays_so():
    """A key that is not a number, on any column of a step, spoils the rows that see it; the output of no row before it (dQ's product multiplies the hidden keys of a step by zero)."""
    B, S, H = 1, 200, 1
    gen = torch.Generator(device="cuda").manual_seed(0)
    dout = torch.randn(B * S, H * 64, generator=gen, device="cuda").bfloat16()
    for key in range(8):
        qkv = torch.randn(B * S, 3 * H * 64, generator=gen, device="cuda").bfloat16()
        clean = _run(qkv, dout, B, S, H)
        qkv[key, 64:128] = float("nan")
        out, lse, dqkv, _ = _run(qkv, dout, B, S, H)
        assert torch.equal(out[:key], clean[0][:key]) and torch.equal(lse[:, :key], clean[1][:, :key]), key
        seen = torch.isfinite(out.float()).all(1)
        assert not seen[key:].any(), key
        assert not torch.isfinite(dqkv[key:, :64].float()).all(1).any(), key


def test_first_use_may_lie_inside_a_callers_capture():
    """In a process whose libraries and other kernels are set up, the first step (evaluation) with heads of 64 columns is captured by its caller."""
    import subprocess
    code = """
import sys, torch
from piccl_b200.models.gpt2 import GPT2, GPT2Config
from piccl_b200 import _native as N
evaluation = sys.argv[1] == "eval"
def model(heads):
    return GPT2(GPT2Config(vocab_size=1000, seq_len=128, n_layer=2, n_head=heads, d_model=256), seed=1)
tok = torch.randint(0, 1000, (4, 129), generator=torch.Generator().manual_seed(0)).cuda()
x, y = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
other = model(2)                           # heads of 128 columns: the same products and launches, attention through PyTorch
other.loss(x, y); other.forward_backward(x, y)
q = torch.randn(4, 4, 128, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
torch.nn.functional.scaled_dot_product_attention(q, q, q, is_causal=True).sum().backward()
torch.cuda.synchronize()
m, g = model(4), torch.cuda.CUDAGraph()
run = m.loss if evaluation else m.forward_backward
with torch.cuda.graph(g):
    loss = run(x, y)
m.flat_g.fill_(float("nan"))
g.replay()
got, grads = float(loss), m.flat_g.clone()
assert abs(float(run(x, y)) - got) <= 1e-5 * got
if not evaluation:                          # the products of a replay may be another back end's
    assert float((m.flat_g.double() - grads.double()).norm()) <= 2 ** -7 * float(grads.double().norm())
assert N.ops_lib().piccl_ops_attn_status() == 0
"""
    for what in ("eval", "train"):
        r = subprocess.run([sys.executable, "-c", code, what], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, (what, r.stderr[-2000:])
