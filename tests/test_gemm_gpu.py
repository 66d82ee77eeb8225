"""tcgen05 GEMM against a plain PyTorch fp32 reference (A @ B^T + bias, optional GELU)."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _bf(*shape, seed=0, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


def _status():
    from piccl_b200 import _native as N
    return N.ops_lib().piccl_ops_gemm_status()


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (128, 256, 64), (256, 256, 256), (128, 384, 128), (1024, 1024, 1024), (384, 3072, 1024), (8192, 1024, 4096), (512, 50304, 1024)])
def test_gemm_matches_fp32_reference(M, N, K):
    from piccl_b200.ops import gemm_sm100
    assert gemm_sm100.available(), "the tcgen05 GEMM must be built and loadable on a B200"
    a, b = _bf(M, K, seed=1), _bf(N, K, seed=2, scale=0.05)
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    gemm_sm100.gemm_nt(a, b, out)
    torch.cuda.synchronize()
    assert _status() == 0
    ref = a.float() @ b.float().t()
    err = (out.float() - ref).abs().max().item()
    assert torch.allclose(out.float(), ref, atol=0.02 * ref.abs().max().item() + 1e-2, rtol=2e-2), f"max abs err {err}"


def test_gemm_bias_and_gelu_epilogue():
    from piccl_b200 import _native as N
    from piccl_b200.ops import gemm_sm100
    M, Nn, K = 512, 1024, 256
    a, b, bias = _bf(M, K, seed=1), _bf(Nn, K, seed=2, scale=0.1), _bf(Nn, seed=3)
    out = torch.empty(M, Nn, device="cuda", dtype=torch.bfloat16)
    gemm_sm100.gemm_nt(a, b, out, bias=bias)
    ref = a.float() @ b.float().t() + bias.float()
    assert torch.allclose(out.float(), ref, atol=5e-2, rtol=2e-2)
    pre = torch.empty_like(out)
    rc = N.ops_lib().piccl_ops_gemm_bf16_nt_ex(C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()), C.c_void_p(out.data_ptr()), C.c_void_p(pre.data_ptr()),
                                               C.c_void_p(bias.data_ptr()), M, Nn, K, 1, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    assert _status() == 0
    assert torch.allclose(pre.float(), ref, atol=5e-2, rtol=2e-2)
    assert torch.allclose(out.float(), F.gelu(pre.float(), approximate="tanh"), atol=2e-2, rtol=2e-2)


def test_gemm_back_to_back_and_unsupported_shapes():
    from piccl_b200 import _native as N
    from piccl_b200.ops import gemm_sm100
    a, b = _bf(256, 512, seed=4), _bf(256, 512, seed=5)
    outs = []
    for _ in range(5):
        o = torch.empty(256, 256, device="cuda", dtype=torch.bfloat16)
        gemm_sm100.gemm_nt(a, b, o)
        outs.append(o)
    torch.cuda.synchronize()
    for o in outs[1:]:
        assert torch.equal(o, outs[0])
    # shapes the kernel does not cover are refused with an error code, not computed wrongly
    rc = N.ops_lib().piccl_ops_gemm_bf16_nt(C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()), C.c_void_p(outs[0].data_ptr()), C.c_void_p(0), 100, 256, 512, 0, C.c_void_p(0))
    assert rc != 0


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (127, 72, 40), (129, 264, 72), (257, 520, 192), (2331, 768, 200)])
@pytest.mark.parametrize("layout,epilogue", [(0, 0), (0, 1), (0, 2), (1, 0), (1, 3), (2, 0)])
def test_gemm_layouts_epilogues_and_edges(M, N, K, layout, epilogue):
    """Ragged tiles of every operand layout and epilogue against fp32.  The result is rounded to bf16 once (2^-9 relative, 2^-8 where
    GELU reads the rounded pre-activation) on top of an fp32 sum, so the error norm stays below 4e-3 of the result's."""
    from piccl_b200.ops import gemm_sm100 as G
    if layout == 2:
        M = (M + 7) // 8 * 8                      # rows of A^T are a multiple of 16 bytes
    a = _bf(M, K, seed=1) if layout != 2 else _bf(K, M, seed=1)
    b = _bf(N, K, seed=2, scale=0.05) if layout == 0 else _bf(K, N, seed=2, scale=0.05)
    bias = _bf(N, seed=3) if epilogue != 3 else None
    aux = _bf(M, N, seed=4) if epilogue >= 2 else None
    guard = torch.full((M + 1, N), float("nan"), device="cuda", dtype=torch.bfloat16)      # the row after the result must stay untouched
    out, pre = guard[:M], (torch.empty(M, N, device="cuda", dtype=torch.bfloat16) if epilogue == 1 else None)
    part = torch.full((G.partial_rows(M), N), float("nan"), device="cuda") if epilogue == 3 else None
    G.gemm(layout, epilogue, a, b, out, bias=bias, aux=aux, pre=pre, part=part.data_ptr() if part is not None else 0)
    torch.cuda.synchronize()
    assert _status() == 0
    ref = (a.float().t() if layout == 2 else a.float()).double() @ (b.float().t() if layout == 0 else b.float()).double()
    if bias is not None:
        ref = ref + bias.double()
    if epilogue == 1:
        assert (pre.double() - ref).norm() <= 4e-3 * ref.norm()
        ref = F.gelu(pre.double(), approximate="tanh")
    if epilogue == 2:
        ref = ref + aux.double()
    if epilogue == 3:
        x = aux.double().requires_grad_()
        F.gelu(x, approximate="tanh").backward(ref)
        ref = x.grad
        assert (part.double().sum(0) - out.double().sum(0)).norm() <= 1e-5 * out.double().abs().sum(0).norm()      # fp32 sums of M values
    assert (out.double() - ref).norm() <= 4e-3 * ref.norm()
    assert torch.isnan(guard[M]).all()


@pytest.mark.parametrize("backend", ["auto", "tcgen05", "cublas"])
@pytest.mark.parametrize("which", ["none", "x", "w", "bias", "h", "out"])
def test_products_of_views_at_any_address(backend, which):
    """An operand or result that starts 2 bytes beyond a 16-byte boundary, at a ragged shape: cuBLAS takes what the kernel cannot.  Bias and GELU by a kernel of their own
    read 16-byte words: there such a view is refused."""
    from piccl_b200.ops import gemm

    def t(name, *shape, scale=1.0):
        n = 1
        for s in shape:
            n *= s
        buf = _bf(n + 8, seed=len(name) + shape[0], scale=scale)
        off = 1 if name == which else 0
        return buf[off:off + n].view(shape)

    M, N, K = 200, 72, 40
    x, w, bias = t("x", M, K), t("w", N, K, scale=0.05), t("bias", N)
    h, out = t("h", M, N), t("out", M, N)
    ref = x.double() @ w.double().t() + bias.double()
    saved = gemm.backend()
    try:
        gemm.set_backend(backend)
        gemm.linear(x, w, bias, out)
        assert (out.double() - ref).norm() <= 4e-3 * ref.norm()            # one rounding to bf16
        if which in ("bias", "h", "out"):
            with pytest.raises(RuntimeError):
                gemm.linear_gelu(x, w, bias, h, out)
            return
        gemm.linear_gelu(x, w, bias, h, out)
        assert (h.double() - ref).norm() <= 8e-3 * ref.norm()              # cuBLAS rounds before the bias is added: two
        want = F.gelu(h.double(), approximate="tanh")
        assert (out.double() - want).norm() <= 4e-3 * want.norm()
    finally:
        gemm.set_backend(saved)
