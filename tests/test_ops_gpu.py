"""Model kernels against plain PyTorch fp32 references of the same operation."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _bf(*shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


@pytest.mark.parametrize("C", [256, 768, 1024])
@pytest.mark.parametrize("with_res", [False, True])
def test_layernorm_forward_backward(C, with_res):
    from piccl_b200 import ops
    T = 300
    x, res = _bf(T, C, seed=1), (_bf(T, C, seed=2) if with_res else None)
    gamma, beta = _bf(C, seed=3) * 0.1 + 1, _bf(C, seed=4) * 0.1
    y, s = torch.empty_like(x), torch.empty_like(x)
    mean, rstd = torch.empty(T, device="cuda"), torch.empty(T, device="cuda")
    ops.layernorm_fwd(x, res, gamma, beta, s if with_res else None, y, mean, rstd)
    xin = (x.float() + res.float()).to(torch.bfloat16).float() if with_res else x.float()
    xr = xin.clone().requires_grad_()
    gr, br = gamma.float().requires_grad_(), beta.float().requires_grad_()
    yr = F.layer_norm(xr, (C,), gr, br, 1e-5)
    assert torch.allclose(y.float(), yr, atol=3e-2, rtol=2e-2)
    if with_res:
        assert torch.equal(s.float(), xin)
    assert torch.allclose(mean, xin.mean(1), atol=1e-4)
    dy, dres = _bf(T, C, seed=5), _bf(T, C, seed=6)
    dx, dg, db = torch.empty_like(x), torch.empty_like(gamma), torch.empty_like(beta)
    ops.layernorm_bwd(dy, xin.to(torch.bfloat16), gamma, mean, rstd, dres, dx, dg, db)
    yr.backward(dy.float())
    assert torch.allclose(dx.float(), xr.grad + dres.float(), atol=5e-2, rtol=3e-2)
    assert torch.allclose(dg.float(), gr.grad, atol=0.3, rtol=3e-2)
    assert torch.allclose(db.float(), br.grad, atol=0.3, rtol=3e-2)


def test_bias_gelu_and_colsum():
    from piccl_b200 import ops
    T, C = 500, 1024
    h, b = _bf(T, C, seed=1), _bf(C, seed=2)
    hp, g = torch.empty_like(h), torch.empty_like(h)
    ops.bias_gelu_fwd(h, b, hp, g)
    hr = (h.float() + b.float())
    assert torch.allclose(hp.float(), hr, atol=2e-2, rtol=1e-2)
    hq = hp.float().requires_grad_()
    gr = F.gelu(hq, approximate="tanh")
    assert torch.allclose(g.float(), gr, atol=2e-2, rtol=1e-2)
    dg = _bf(T, C, seed=3)
    dh = torch.empty_like(dg)
    ops.gelu_bwd(dg, hp, dh)
    gr.backward(dg.float())
    assert torch.allclose(dh.float(), hq.grad, atol=2e-2, rtol=2e-2)
    out = torch.empty(C, device="cuda", dtype=torch.bfloat16)
    ops.colsum(dg, out)
    assert torch.allclose(out.float(), dg.float().sum(0), atol=0.3, rtol=2e-2)


def test_cross_entropy_with_padded_vocab():
    from piccl_b200 import ops
    T, V, Vp = 64, 1000, 1024
    logits = _bf(T, Vp, scale=2.0, seed=1)
    ref_in = logits[:, :V].float().clone().requires_grad_()
    tgt = torch.randint(0, V, (T,), device="cuda")
    loss_rows = torch.empty(T, device="cuda")
    ops.cross_entropy_fwd_bwd(logits, tgt, loss_rows, V, 1.0 / T)
    ref = F.cross_entropy(ref_in, tgt, reduction="none")
    assert torch.allclose(loss_rows, ref, atol=1e-3, rtol=1e-3)
    ref.mean().backward()
    assert torch.allclose(logits[:, :V].float(), ref_in.grad, atol=2e-4, rtol=2e-2)
    assert logits[:, V:].abs().sum() == 0


def test_adamw_matches_torch():
    from piccl_b200 import ops
    n = 4096
    p0 = _bf(n, seed=1)
    master = p0.float().clone()
    p = p0.clone()
    m, v = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    ref = torch.nn.Parameter(p0.float().clone())
    opt = torch.optim.AdamW([ref], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    for step in range(1, 4):
        g = _bf(n, seed=10 + step)
        ops.adamw(p, master, m, v, g, 1e-2, 0.9, 0.95, 1e-8, 0.1, step)
        ref.grad = g.float()
        opt.step()
    assert torch.allclose(master, ref.data, atol=1e-5, rtol=1e-4)
    assert torch.allclose(p.float(), ref.data, atol=1e-2, rtol=1e-2)


def test_embedding_forward_backward():
    from piccl_b200 import ops
    B, S, C, V = 3, 16, 256, 100
    idx = torch.randint(0, V, (B * S,), device="cuda")
    wte, wpe = _bf(V, C, seed=1), _bf(S, C, seed=2)
    out = torch.empty(B * S, C, device="cuda", dtype=torch.bfloat16)
    ops.embed_fwd(idx, wte, wpe, out, S)
    ref = wte.float()[idx] + wpe.float().repeat(B, 1)
    assert torch.allclose(out.float(), ref, atol=2e-2, rtol=1e-2)
    dx = _bf(B * S, C, seed=3)
    dwpe = torch.zeros_like(wpe)
    ops.wpe_bwd(dx, dwpe, B, S)
    assert torch.allclose(dwpe.float(), dx.float().view(B, S, C).sum(0), atol=5e-2, rtol=2e-2)
    dwte = torch.zeros_like(wte)
    stage = torch.zeros(V, C, device="cuda")
    ops.wte_bwd(idx, dx, stage, dwte)
    ref_g = torch.zeros(V, C, device="cuda").index_add_(0, idx, dx.float())
    assert torch.allclose(dwte.float(), ref_g, atol=5e-2, rtol=2e-2)


@pytest.mark.parametrize("C,rows", [(256, 1), (256, 6001), (512, 3700), (768, 3001), (1024, 5), (1024, 3001), (2048, 1800)])
def test_layernorm_rows_in_several_rounds(C, rows):
    # more rows than the resident warps (forward) and groups (backward) have at once: rows are prefetched, the last round is partial
    from piccl_b200 import ops
    x, res, gamma, beta = _bf(rows, C, seed=1), _bf(rows, C, seed=2), _bf(C, seed=3) * 0.1 + 1, _bf(C, seed=4) * 0.1
    y, s, mean, rstd = torch.empty_like(x), torch.empty_like(x), torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
    for r in (res, None):
        ops.layernorm_fwd(x, r, gamma, beta, s, y, mean, rstd)
        xin = (x.float() + r.float()).to(torch.bfloat16) if r is not None else x
        assert torch.equal(s, xin)
        xr, gr, br = xin.double().requires_grad_(), gamma.double().requires_grad_(), beta.double().requires_grad_()
        yr = F.layer_norm(xr, (C,), gr, br, 1e-5)
        assert torch.all((y.double() - yr).abs() <= 2 ** -8 * yr.abs() + 1e-4)          # one rounding to bf16, fp32 sums
    if C > 1024:
        return
    dy = _bf(rows, C, seed=5)
    dx, dg, db = torch.empty_like(x), torch.empty_like(gamma), torch.empty_like(beta)
    ops.layernorm_bwd(dy, x, gamma, mean, rstd, None, dx, dg, db)
    yr.backward(dy.double())
    for got, want in ((dx, xr.grad), (dg, gr.grad), (db, br.grad)):
        assert torch.all((got.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-3 * want.abs().max())


@pytest.mark.parametrize("rows,V,Vp", [(3, 5, 8), (40, 1000, 1024), (5, 16400, 16512), (9, 50257, 50304), (2, 120001, 120064)])
def test_cross_entropy_online(rows, V, Vp):
    # vocabularies below and beyond a block's round of 16384 columns and beyond what shared memory holds; logits that rise along the row
    # raise the running maximum all the time
    from ctypes import c_float, c_void_p
    from piccl_b200 import _native as N
    logits = _bf(rows, Vp, scale=3.0, seed=1)
    logits[0] += torch.linspace(-20, 20, Vp, device="cuda").to(torch.bfloat16)
    logits[1, : V // 2] = float("-inf")
    tgt = torch.randint(V // 2, V, (rows,), generator=torch.Generator().manual_seed(2)).cuda()
    tgt[-1] = -100                                          # no target: no loss, no gradient
    ref_in = logits[:, :V].double().requires_grad_()
    ref = F.cross_entropy(ref_in, tgt, reduction="none")
    ref.sum().backward()
    for grad in (0, 1):
        loss, lg = torch.empty(rows, device="cuda"), logits.clone()
        rc = N.ops_lib().piccl_ops_ce(c_void_p(lg.data_ptr()), c_void_p(tgt.data_ptr()), c_void_p(loss.data_ptr()), rows, V, Vp, c_float(0.5), grad, c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        # exponents up to 2^7 carry fp32 rounding of 2^-17; the sum and the logarithm add less
        assert torch.all((loss.double() - ref.detach()).abs() <= 1e-4)
        if not grad:
            assert torch.equal(lg, logits)
            continue
        want = 0.5 * ref_in.grad
        assert torch.all((lg[:, :V].double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5)
        assert lg[:, V:].abs().sum() == 0


@pytest.mark.parametrize("offset", [0.0, 100.0, -400.0, 1000.0])
def test_cross_entropy_does_not_depend_on_an_offset(offset):
    """A common offset of the logits costs no precision: differences of bf16 values are exact in fp32.  Left are the roundings of the exponents (|x - max| log2 e <= 60,
    weighted by the probabilities: below 2^-20), of the exponentials and their sum (2^-22, some 20 additions), of a logarithm up to 11 and of a loss up to 64 (2^-19)."""
    from ctypes import c_float, c_void_p
    from piccl_b200 import _native as N
    rows, V, Vp = 512, 5003, 5120
    gen = torch.Generator(device="cuda").manual_seed(1)
    logits = (torch.randn(rows, Vp, generator=gen, device="cuda") * 4 + offset).bfloat16()
    tgt = torch.randint(0, V, (rows,), generator=gen, device="cuda")
    ref_in = logits[:, :V].double().requires_grad_()
    ref = F.cross_entropy(ref_in, tgt, reduction="none")
    ref.sum().backward()
    for grad in (0, 1):
        loss, lg = torch.empty(rows, device="cuda"), logits.clone()
        rc = N.ops_lib().piccl_ops_ce(c_void_p(lg.data_ptr()), c_void_p(tgt.data_ptr()), c_void_p(loss.data_ptr()), rows, V, Vp, c_float(1.0), grad, c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        assert float((loss.double() - ref.detach()).abs().max()) <= 6e-6
    assert float((lg[:, :V].double() - ref_in.grad).norm()) <= 2 ** -9 * float(ref_in.grad.norm())


@pytest.mark.parametrize("shape", [(4096,), (8,), (4, 8, 64), (16, 12), (3, 40), (0,), (0, 16), (5, 3, 24), (1, 4104)])
def test_gelu_backward_of_any_shape(shape):
    """Vectors, batches of matrices and rows that are no multiple of 16 bytes, in place too; one rounding to bf16 of a value that is exact to a few fp32 roundings."""
    from piccl_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(1)
    h, dg = (torch.randn(shape, generator=gen, device="cuda").bfloat16() for _ in range(2))
    x = h.double().requires_grad_()
    F.gelu(x, approximate="tanh").backward(dg.double())
    dh = torch.empty_like(h)
    ops.gelu_bwd(dg, h, dh)
    assert torch.all((dh.double() - x.grad).abs() <= 2 ** -8 * x.grad.abs() + 2e-6 * dg.double().abs())
    ops.gelu_bwd(dg, h, dg)
    assert torch.equal(dg, dh)
    with pytest.raises(RuntimeError):
        ops.gelu_bwd(torch.ones(12, device="cuda").bfloat16(), torch.ones(12, device="cuda").bfloat16(), torch.ones(12, device="cuda").bfloat16())


def test_layernorm_backward_takes_a_row_split():
    from piccl_b200 import ops
    rows, C = 70, 512
    x, dy, gamma = _bf(rows, C, seed=1), _bf(rows, C, seed=2), _bf(C, seed=3)
    mean, rstd = x.float().mean(1), (x.float().var(1, unbiased=False) + 1e-5).rsqrt()
    got = []
    for split in ((), (False, 16)):
        out = [torch.empty_like(x), torch.empty_like(gamma), torch.empty_like(gamma)]
        ops.layernorm_bwd(dy, x, gamma, mean, rstd, None, *out, *split)
        got.append(out)
    assert all(torch.equal(a, b) for a, b in zip(*got))


def test_partial_rows_of_any_width_and_alignment():
    """Vectors folded together whose rows are not whole pairs, or begin in the middle of one, beside one that is read in pairs; up to more rows than are in flight."""
    import ctypes as C
    from piccl_b200 import _native as N
    from piccl_b200.ops import _FinishJob, _s
    g = torch.Generator(device="cuda").manual_seed(3)
    jobs, want, outs, keep = [], [], [], []
    for n, Cc, shift, acc in [(1, 1, 0, 0), (33, 77, 0, 1), (16, 64, 1, 0), (160, 66, 0, 1), (161, 130, 0, 0), (500, 63, 1, 0)]:
        flat = torch.randn(n * Cc + shift, generator=g, device="cuda")
        part = flat[shift:].view(n, Cc)
        out = torch.randn(Cc, generator=g, device="cuda").bfloat16()
        want.append(part.double().sum(0) + (out.double() if acc else 0))
        outs.append(out)
        keep.append(flat)
        jobs.append((part.data_ptr(), out.data_ptr(), n, Cc, acc, 0))
    assert N.ops_lib().piccl_ops_finish_parts((_FinishJob * len(jobs))(*jobs), len(jobs), C.c_void_p(_s())) == 0
    for w, o, f in zip(want, outs, keep):
        # one rounding to bf16 of the sum, and of each of the fp32 additions
        assert ((o.double() - w).abs() <= 2.0 ** -8 * w.abs() + f.numel() * 2.0 ** -24 * f.abs().max()).all()
