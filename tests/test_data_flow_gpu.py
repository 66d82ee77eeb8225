"""Launches that carry all ranks on one GPU, whose data flow (src/coll/flow.cc) takes the place of the ranks' programs, beside those programs through the slots."""
import itertools

import pytest
import torch

pytestmark = pytest.mark.gpu

ALGOS = ["RING", "K_RING", "RD", "RM", "PRD", "PRM", "DIRECT"]


def _group(n):
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    return LoopbackGroup(n, config=make_config(scratch_bytes=1 << 20, timeout_ms=5000))


def _both(g, coll, xs, n_out, count, **kw):
    """The call's results through the slots and from its data flow."""
    outs = []
    for slots in (True, False):
        g.slots_only(slots)
        outs.append([torch.full((n_out,), 7, device="cuda", dtype=xs[0].dtype) for _ in xs])
        for _ in range(2):
            g.run(coll, xs, outs[-1], count, **kw)
        torch.cuda.synchronize()
        assert g.status().aborted == 0
    return outs


@pytest.mark.parametrize("dtype", [torch.int8, torch.uint8, torch.int32, torch.int64])
@pytest.mark.parametrize("n,k", [(3, 2), (4, 4), (8, 2)])
def test_integers(n, k, dtype):
    """Sums and products that overflow too: the same bits in any order.  Lengths of a few elements, of one block, of several with a remainder and, among them, odd addresses of the blocks."""
    g = _group(n)
    info = torch.iinfo(dtype)
    for coll, count in itertools.product(["allreduce", "reduce_scatter", "reduce"], [3, 4096 + 5, 70001]):
        n_in = count * (n if coll == "reduce_scatter" else 1)
        xs = [torch.randint(info.min, info.max, (n_in,), generator=torch.Generator(device="cuda").manual_seed(r), device="cuda", dtype=dtype) for r in range(n)]
        for algo, op in itertools.product(ALGOS, ["sum", "prod", "max", "min"]):
            a, b = _both(g, coll, xs, count, count, op=op, root=1, algo=algo, k=k)
            assert all(torch.equal(x, y) for x, y in zip(a, b)), (coll, count, algo, op)
    g.close()
