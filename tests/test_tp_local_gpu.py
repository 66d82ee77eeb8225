"""Tensor-parallel kernels of launches that carry all ranks on one GPU: row blocks of two owners in one pair of CTAs, and products that are exchanged because that is faster."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * scale).to(torch.bfloat16)


# One, three and five row blocks to an owner: an even and an odd number of them in all, tiles of every width, more tiles than pairs of CTAs; one shape that is exchanged outside a capture.
@pytest.mark.parametrize("n,blocks,N,K", [(2, 1, 256, 64), (3, 1, 256, 64), (3, 3, 512, 128), (5, 1, 4096, 64), (7, 1, 1024, 128), (8, 1, 8192, 64), (4, 3, 4096, 128), (2, 5, 2048, 192), (8, 1, 256, 4096)])
def test_row_blocks_of_two_owners(n, blocks, N, K):
    """Against fp64 products: sums of n K products of bf16 values in fp32 err by far less than the result's rounding, half a unit in 2^-8; exchanged partial tiles are rounded
    once each, which is at most 2^-9 of the largest of them, 8 standard deviations of 0.1 sqrt(K).  A captured call, replayed on other operands, always reads them where they are."""
    from piccl_b200.parallel import tp
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    M = 128 * n * blocks
    g = LoopbackGroup(n, config=make_config(max_cta=4, nslot=2, slot_bytes=4096, scratch_bytes=1 << 16, timeout_ms=5000, tp_bytes=tp.workspace_bytes("gemm_rs", n, M, N, K)))
    exchanged = g._lib.piccl_test_tp_width(0, n, M, N, K, torch.cuda.get_device_properties(0).multi_processor_count // 2) == 0
    assert exchanged == (K == 4096)
    As = [_bf(M, K, seed=50 + r) for r in range(n)]
    Bs = [_bf(N, K, seed=60 + r, scale=0.1) for r in range(n)]
    outs = [torch.full((M // n, N), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(n)]

    def check(rounded):
        torch.cuda.synchronize()
        assert all(tp.tp_status(h) == 0 for h in g._hs)
        total = sum(As[r].double() @ Bs[r].double().t() for r in range(n))
        bound = total.abs() * 2.0 ** -8 + n * K * 2.0 ** -20 + (n * 2.0 ** -9 * 8 * 0.1 * K ** 0.5 if rounded else 0.0)
        for r in range(n):
            rows = slice(r * (M // n), (r + 1) * (M // n))
            err = (outs[r].double() - total[rows]).abs()
            assert (err <= bound[rows]).all(), (r, err.max().item())
    for _ in range(2):
        tp.gemm_rs_group(g, As, Bs, outs)
    check(exchanged)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        tp.gemm_rs_group(g, As, Bs, outs)
    for rep in range(2):
        for r in range(n):
            As[r].copy_(_bf(M, K, seed=70 + r + rep))
            outs[r].fill_(float("nan"))
        graph.replay()
        check(False)
    g.close()
