"""The tensor-parallel kernels' tests once more with partial tiles and shards exchanged between the ranks, as between GPUs, and the kernels of a launch that carries all ranks on one GPU."""
import pytest
import torch

from test_tp_gpu import *      # noqa: F401,F403
from test_tp_gpu import _bf, _group, pytestmark      # noqa: F401


@pytest.fixture(autouse=True)
def through_the_workspace(request, monkeypatch):
    from piccl_b200.parallel import comm

    class SlotsOnly(comm.LoopbackGroup):
        def __init__(self, *a, **kw):
            super().__init__(*a, **kw)
            self.slots_only()
    if request.function is not test_all_ranks_in_one_launch:
        monkeypatch.setattr(comm, "LoopbackGroup", SlotsOnly)


# Tiles of 256, 128 and 64 columns by the number of tiles; one, an odd and an even number of row blocks to a rank, more tiles than pairs of CTAs, one k-block to a rank.
@pytest.mark.parametrize("n,blocks,N,K", [(2, 1, 256, 64), (2, 3, 256, 192), (3, 1, 512, 64), (8, 1, 256, 128), (4, 5, 768, 64), (4, 2, 4096, 128), (2, 8, 4096, 320), (8, 3, 1024, 64)])
@pytest.mark.parametrize("which", ["gemm_rs", "ag_gemm"])
def test_all_ranks_in_one_launch(which, n, blocks, N, K):
    """Against fp64 products.  Sums of n K products of bf16 values in fp32 err by far less than the result's rounding to bf16, half a unit in 2^-8; the exchanged form of the same
    call rounds partial tiles too."""
    from piccl_b200.parallel import tp
    M = 128 * n * blocks
    g = _group(n, which, M, N, K)
    rs = which == "gemm_rs"
    As = [_bf(M if rs else M // n, K, seed=50 + r) for r in range(n)]
    Bs = [_bf(N, K, seed=60 + r, scale=0.1) for r in range(n)]
    call = tp.gemm_rs_group if rs else tp.ag_gemm_group

    def run():
        outs = [torch.full((M // n if rs else M, N), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(n)]
        for _ in range(2):
            call(g, As, Bs, outs)
        torch.cuda.synchronize()
        assert all(tp.tp_status(h) == 0 for h in g._hs)
        return outs
    if rs:
        total = sum(As[r].double() @ Bs[r].double().t() for r in range(n))
        want = [total[r * (M // n):(r + 1) * (M // n)] for r in range(n)]
    else:
        want = [torch.cat(As).double() @ Bs[r].double().t() for r in range(n)]
    outs = run()
    for r in range(n):
        err = (outs[r].double() - want[r]).abs()
        assert (err <= want[r].abs() * 2.0 ** -8 + n * K * 2.0 ** -20).all(), (r, err.max().item())
    g.slots_only()
    for r, o in enumerate(run()):
        assert (o.double() - want[r]).norm() <= 2.0 ** -6 * want[r].norm()
        if not rs:
            assert torch.equal(o, outs[r])
    g.close()
