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


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n", [2, 3, 4, 8])
def test_averages_of_small_values(n, dtype):
    """Shares below 2^-14, fp16's normal range, lose bits where they cross between ranks: which do is the same in the data flow, and so it is for thirds, which are rounded in either type.
    Values of 1e-7 to 1, zeros of both signs, the least elements of fp16; lengths that low-latency kernels would take, which round all shares, and longer ones.  The same bits as through the slots."""
    g = _group(n)
    for coll, count in itertools.product(["allreduce", "reduce_scatter", "reduce"], [7, 20011, 600013]):
        n_in = count * (n if coll == "reduce_scatter" else 1)
        xs = []
        for r in range(n):
            gen = torch.Generator(device="cuda").manual_seed(r)
            x = (torch.rand(n_in, generator=gen, device="cuda") * 2 - 1) * 10.0 ** torch.randint(-7, 1, (n_in,), generator=gen, device="cuda")
            xs.append(x.to(dtype))
            xs[-1][::5] = torch.tensor([0.0, -0.0, 2.0 ** -24, -(2.0 ** -24), 3 * 2.0 ** -24], device="cuda", dtype=dtype)[r % 5]
        for algo, k in itertools.product(ALGOS, [2, 8]):
            a, b = _both(g, coll, xs, count, count, op="avg", root=1, algo=algo, k=k)
            assert all(torch.equal(x.view(torch.int16), y.view(torch.int16)) for x, y in zip(a, b)), (coll, count, algo, k)
            if algo in ("RD", "RM", "PRD", "PRM") and coll == "allreduce" and count > 7:       # captured, it is the same call (what the low-latency kernel runs cannot be captured)
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph):
                    g.run(coll, xs, b, count, op="avg", root=1, algo=algo, k=k)
                for y in b:
                    y.zero_()
                graph.replay()
                assert all(torch.equal(x.view(torch.int16), y.view(torch.int16)) for x, y in zip(a, b)), (coll, count, algo, k)
    g.close()


@pytest.mark.parametrize("variable,value", [("PICCL_PROTO", "ll"), ("PICCL_PROTO", "simple"), ("PICCL_MAX_GRID_SIZE", "2"), ("PICCL_MIN_GRID_SIZE", "3")])
def test_a_way_that_is_asked_for_by_name_is_taken(monkeypatch, variable, value):
    """The data path that PICCL_PROTO narrows, and the grid that the reference's variables size, are the executor's."""
    g = _group(4)
    flows = lambda: g._lib.piccl_test_flow_calls(g._hs[0])
    xs = [torch.full((20000,), float(r + 1), device="cuda") for r in range(4)]

    def run():
        outs = [torch.zeros_like(x) for x in xs]
        for algo in ("RING", "PRD"):
            g.run("allreduce", xs, outs, 20000, algo=algo)
        torch.cuda.synchronize()
        assert g.status().aborted == 0 and all(torch.all(o == 10.0) for o in outs)
    try:
        before = flows()
        run()
        assert flows() == before + 2
        monkeypatch.setenv(variable, value)
        g._lib.piccl_env_reload()
        run()
        assert flows() == before + 2
    finally:
        monkeypatch.undo()
        g._lib.piccl_env_reload()
        g.close()


def test_checks_of_the_debug_mode_pass(monkeypatch):
    """PICCL_DEBUG=1 checks fresh programs and data flows against the call's buffers; in place too."""
    monkeypatch.setenv("PICCL_DEBUG", "1")
    g = _group(8)
    g._lib.piccl_env_reload()
    try:
        xs = [torch.full((8 * 30011,), float(r + 1), device="cuda") for r in range(8)]
        for coll, algo in itertools.product(["allreduce", "reduce_scatter", "reduce", "allgather", "broadcast"], ALGOS):
            outs = [torch.zeros(8 * 30011, device="cuda") for _ in xs]
            before = g._lib.piccl_test_flow_calls(g._hs[0])
            g.run(coll, xs, outs, 30011, algo=algo, root=3)
            if coll in ("allgather", "broadcast"):
                g.run(coll, [o[r * 30011:] if coll == "allgather" else o for r, o in enumerate(outs)], outs, 30011, algo=algo, root=3)
            torch.cuda.synchronize()
            assert g.status().aborted == 0 and g._lib.piccl_test_flow_calls(g._hs[0]) > before
            want = {"allgather": 4.0, "broadcast": 4.0}.get(coll, 36.0)
            assert torch.all(outs[3][30011 * 3:30011 * 4] == want) if coll == "allgather" else torch.all(outs[3][:30011] == want)
    finally:
        monkeypatch.undo()
        g._lib.piccl_env_reload()
        g.close()


@pytest.mark.parametrize("coll", ["allreduce", "reduce"])
def test_capture_with_other_buffers_than_the_first_call(coll):
    """The first call's buffers are apart; in the captured one a rank receives into another's send buffer (the ring's sums contain what they overwrite).  The ranks' programs are there although the data flow ran."""
    n, count = 4, 300000
    g = _group(n)
    xs = [torch.randint(-100, 100, (count,), generator=torch.Generator(device="cuda").manual_seed(r), device="cuda").float() for r in range(n)]
    want = [torch.zeros(count, device="cuda") for _ in range(n)]
    flows = g._lib.piccl_test_flow_calls(g._hs[0])
    g.run(coll, xs, want, count, algo="RING", root=1)
    assert g._lib.piccl_test_flow_calls(g._hs[0]) == flows + 1
    ys = [x.clone() for x in xs]
    outs = [torch.zeros(count, device="cuda") for _ in range(n)]
    outs[0 if coll == "allreduce" else 1] = ys[1 if coll == "allreduce" else 2]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        g.run(coll, ys, outs, count, algo="RING", root=1)
    assert g._lib.piccl_test_flow_calls(g._hs[0]) == flows + 1
    graph.replay()
    torch.cuda.synchronize()
    assert g.status().aborted == 0 and torch.equal(outs[1], want[1])
    g.close()


def test_programs_take_over_when_data_flows_are_full():
    """Data flows are kept up to 256 MiB, about 11 KB for an all-gather among eight ranks.  Programs, which have room of their own, run what comes then; what is kept runs on."""
    n, most = 8, 26000
    g = _group(n)
    flows = lambda: g._lib.piccl_test_flow_calls(g._hs[0])
    xs = [torch.full((most,), r, device="cuda", dtype=torch.uint8) for r in range(n)]
    outs = [torch.zeros(n * most, device="cuda", dtype=torch.uint8) for _ in range(n)]
    for count in range(1, most + 1):
        before = flows()
        g.run("allgather", xs, outs, count, algo="RING")
        if flows() == before:
            break
    assert 20000 < count < most, count
    for c, kept in ((count, False), (count + 1, False), (100, True)):
        for o in outs:
            o.zero_()
        before = flows()
        g.run("allgather", xs, outs, c, algo="RING")
        torch.cuda.synchronize()
        assert g.status().aborted == 0 and flows() == before + kept
        assert all(torch.equal(o[:n * c].view(n, c).amin(1), o[:n * c].view(n, c).amax(1)) and o[:n * c:c].tolist() == list(range(n)) for o in outs)
    g.close()


def test_groups_without_the_native_call_path(monkeypatch):
    """As where Python's headers are missing: collectives and products go through ctypes."""
    from piccl_b200 import _native as N
    from piccl_b200.parallel import tp
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    monkeypatch.setattr(N, "fastcall", lambda: None)
    g = LoopbackGroup(2, config=make_config(scratch_bytes=1 << 20, timeout_ms=5000, tp_bytes=tp.workspace_bytes("gemm_rs", 2, 256, 256, 64)))
    xs = [torch.full((5000,), float(r + 1), device="cuda") for r in range(2)]
    outs = [torch.zeros(5000, device="cuda"), None]
    g.run("reduce", xs, outs, 5000, root=0)
    a = [torch.ones(256, 64, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    c = [torch.zeros(128, 256, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    tp.gemm_rs_group(g, a, a, c)
    torch.cuda.synchronize()
    assert g.status().aborted == 0 and torch.all(outs[0] == 3.0) and all(torch.all(x == 128.0) for x in c)
    g.close()


@pytest.mark.parametrize("coll,n,algo,small,large", [("allreduce", 4, "RD", 10001, 60001), ("allreduce", 8, "PRM", 49152, 49153), ("reduce", 8, "K_RING", 8192, 8193)])
def test_small_sums_at_odd_addresses(coll, n, algo, small, large):
    """They stay with the low-latency kernels up to the lines in run_flow, are captured as data flows all the same, and are the same bits whichever runs; two-byte elements, one element into their buffers."""
    g = _group(n)
    flows = lambda: g._lib.piccl_test_flow_calls(g._hs[0])
    for count, flow in ((small, 0), (large, 1)):
        xs = [torch.rand(count + 1, generator=torch.Generator(device="cuda").manual_seed(r), device="cuda").to(torch.bfloat16)[1:] for r in range(n)]
        outs = [[torch.zeros(count + 1, device="cuda", dtype=torch.bfloat16)[1:] for _ in range(n)] for _ in range(2)]
        before = flows()
        g.run(coll, xs, outs[0], count, algo=algo, k=2, root=1)
        assert flows() == before + flow
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            g.run(coll, xs, outs[1], count, algo=algo, k=2, root=1)
        assert flows() == before + flow + 1
        graph.replay()
        torch.cuda.synchronize()
        assert g.status().aborted == 0 and all(torch.equal(x, y) for x, y in zip(*outs))
    g.close()
