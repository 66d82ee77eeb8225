"""Fused executor on one GPU: n virtual ranks in one cooperative launch, compared
with a plain PyTorch fp32 reference of the same collective."""
import itertools

import pytest
import torch

pytestmark = pytest.mark.gpu

ALGOS = ["RING", "K_RING", "RD", "RM", "PRD", "PRM", "DIRECT"]


@pytest.fixture(scope="module")
def groups():
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    cache = {}

    def get(n):
        if n not in cache:
            # small slots so that multi-segment pipelining is exercised with little data
            cache[n] = LoopbackGroup(n, config=make_config(max_cta=8, nslot=2, slot_bytes=4096, scratch_bytes=1 << 20, timeout_ms=5000))
        return cache[n]

    yield get
    for g in cache.values():
        g.close()


def _inputs(n, count, dtype, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if dtype in (torch.int32, torch.int64):
        return [torch.randint(-1000, 1001, (count,), generator=g, device="cuda", dtype=dtype) for _ in range(n)]
    return [(torch.rand(count, generator=g, device="cuda", dtype=torch.float32) * 2 - 1).to(dtype) for _ in range(n)]


def _ref_reduce(xs, op):
    st = torch.stack([x.double() if x.dtype in (torch.int32, torch.int64) else x.float() for x in xs])
    if op == "sum":
        return st.sum(0)
    if op == "prod":
        return st.prod(0)
    if op == "max":
        return st.max(0).values
    if op == "min":
        return st.min(0).values
    return st.mean(0)


def _tol(dtype, n):
    return {torch.float32: 1e-5 * n, torch.float64: 1e-5 * n, torch.bfloat16: 2e-2, torch.float16: 2e-3}.get(dtype, 0.0)


def _check_ok(g):
    torch.cuda.synchronize()
    st = g.status()
    assert st.aborted == 0, f"device wait gave up: code {st.code} rank {st.rank} cta {st.cta} action {st.action} peer {st.peer} seg {st.segment}"


@pytest.mark.parametrize("n", [2, 4, 8])
@pytest.mark.parametrize("algo", ALGOS)
def test_allreduce_fp32(groups, n, algo):
    g = groups(n)
    for count, k in itertools.product([1, 7, 1024, 40000], [2, 4]):
        xs = _inputs(n, count, torch.float32)
        outs = [torch.full_like(x, float("nan")) for x in xs]
        g.run("allreduce", xs, outs, count, op="sum", algo=algo, k=k)
        _check_ok(g)
        ref = _ref_reduce(xs, "sum")
        for r in range(n):
            assert torch.allclose(outs[r].float(), ref, atol=_tol(torch.float32, n), rtol=0), f"n={n} {algo} k={k} count={count} rank {r}"
        # all ranks hold bit-identical results
        for r in range(1, n):
            assert torch.equal(outs[r], outs[0])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.int32, torch.float64, torch.int64])
@pytest.mark.parametrize("op", ["sum", "max", "min", "prod"])
def test_allreduce_dtypes_ops_in_place(groups, dtype, op):
    n = 4
    g = groups(n)
    for algo in ["RING", "PRD", "PRM"]:
        count = 3001
        xs = _inputs(n, count, dtype, seed=1)
        if op == "prod":
            xs = [(x.float().abs() * 0.05 + 0.98).to(dtype) if dtype.is_floating_point else (x % 2 + 1) for x in xs]
        ref = _ref_reduce(xs, op)
        bufs = [x.clone() for x in xs]
        g.run("allreduce", bufs, bufs, count, op=op, algo=algo, k=4)
        _check_ok(g)
        for r in range(n):
            got = bufs[r].double() if not dtype.is_floating_point else bufs[r].float()
            tol = _tol(dtype, n) * (4 if op in ("sum", "prod") else 1)
            assert torch.allclose(got, ref.to(got.dtype), atol=tol, rtol=tol), f"{dtype} {op} {algo} rank {r}"


def test_allreduce_avg(groups):
    n = 4
    g = groups(n)
    xs = _inputs(n, 5000, torch.float32, seed=2)
    outs = [torch.empty_like(x) for x in xs]
    for algo in ["RING", "PRD", "PRM"]:
        g.run("allreduce", xs, outs, 5000, op="avg", algo=algo, k=2)
        _check_ok(g)
        assert torch.allclose(outs[1], _ref_reduce(xs, "avg"), atol=1e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,algo,k", [(2, "RING", -1), (4, "PRD", 2), (8, "K_RING", 4), (3, "PRM", 3), (4, "PRM", 4), (8, "PRM", 8), (6, "RM", 3), (5, "DIRECT", -1)])
def test_averaged_operands(groups, n, algo, k, dtype):
    """Scaled operands alone and beside one, up to three and up to seven others, in small slots: the low-latency kernels, unaligned offsets and the ends of the aligned loops
    (their full rounds: test_averaged_rounds_of_the_default_geometry).  Each of at most three partial sums is rounded to the type once, and so is the scaled operand."""
    eps = 2.0 ** (-24 if dtype == torch.float32 else -9)
    for count in (1, 9, 4096 * 8 + 3, 100003):
        g = groups(n)
        xs = _inputs(n, count, dtype, seed=count)
        outs = [torch.empty_like(x) for x in xs]
        g.run("allreduce", xs, outs, count, op="avg", algo=algo, k=k)
        _check_ok(g)
        for o in outs:
            assert (o.double() - torch.stack(xs).double().mean(0)).abs().max() <= 2 * n * eps


@pytest.mark.parametrize("coll,n,count,dtype,algo,k", [("allreduce", 4, (17 << 20) + 5, torch.bfloat16, "PRD", 2), ("allreduce", 8, (5 << 20) + 3, torch.float32, "RING", -1),
                                                       ("allgather", 4, 4 << 20, torch.int32, "RING", -1), ("reduce_scatter", 2, 5 << 20, torch.float32, "AUTO", -1),
                                                       ("broadcast", 3, (6 << 20) + 1, torch.float32, "RING", -1), ("reduce", 4, (5 << 20) + 7, torch.int32, "AUTO", -1)])
def test_buffers_larger_than_the_cache(coll, n, count, dtype, algo, k):
    """Calls whose buffers crowd L2, where loads and stores carry a priority: twice on the same buffers, the second time with other values."""
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    g = LoopbackGroup(n, config=make_config(timeout_ms=5000))
    try:
        outs = [torch.zeros(count * n if coll == "allgather" else count, dtype=dtype, device="cuda") for _ in range(n)]
        xs = None
        for seed in (1, 2):
            new = _inputs(n, count * n if coll == "reduce_scatter" else count, dtype, seed=seed)
            xs = new if xs is None else [x.copy_(y) for x, y in zip(xs, new)]
            g.run(coll, xs, outs, count, op="sum", root=0, algo=algo, k=k)
            _check_ok(g)
            total = torch.stack(xs).double().sum(0) if coll not in ("allgather", "broadcast") else None
            for r, o in enumerate(outs):
                if coll == "reduce" and r:
                    continue
                want = torch.cat(xs) if coll == "allgather" else xs[0] if coll == "broadcast" else total[r * count:(r + 1) * count] if coll == "reduce_scatter" else total
                if dtype == torch.int32 or total is None:
                    assert torch.equal(o.double(), want.double())
                else:
                    assert (o.double() - want).abs().max() <= n * n * 2.0 ** (-24 if dtype == torch.float32 else -9)
    finally:
        g.close()



@pytest.mark.parametrize("n", [2, 4, 8])
@pytest.mark.parametrize("algo", ALGOS)
def test_allgather(groups, n, algo):
    g = groups(n)
    for count, k, dtype in [(1, 2, torch.float32), (1000, 4, torch.bfloat16), (5003, 2, torch.int32), (33333, 8, torch.uint8)]:
        if dtype == torch.uint8:
            xs = [torch.randint(0, 255, (count,), device="cuda", dtype=dtype) for _ in range(n)]
        else:
            xs = _inputs(n, count, dtype, seed=3)
        outs = [torch.zeros(n * count, device="cuda", dtype=dtype) for _ in range(n)]
        g.run("allgather", xs, outs, count, algo=algo, k=k)
        _check_ok(g)
        ref = torch.cat(xs)
        for r in range(n):
            assert torch.equal(outs[r], ref), f"n={n} {algo} k={k} count={count} rank {r}"
    # in place: the send buffer is the rank's own block of the receive buffer
    count = 2048
    outs = [torch.zeros(n * count, device="cuda") for _ in range(n)]
    xs = []
    for r in range(n):
        outs[r][r * count:(r + 1) * count] = torch.arange(count, device="cuda") + 10000 * r
        xs.append(outs[r][r * count:(r + 1) * count])
    ref = torch.cat([x.clone() for x in xs])
    g.run("allgather", xs, outs, count, algo=algo, k=2)
    _check_ok(g)
    for r in range(n):
        assert torch.equal(outs[r], ref)


@pytest.mark.parametrize("n", [2, 4, 8])
@pytest.mark.parametrize("algo", ALGOS)
def test_reduce_scatter(groups, n, algo):
    g = groups(n)
    for count, k in [(1, 2), (999, 4), (20000, 2)]:
        xs = _inputs(n, n * count, torch.float32, seed=4)
        outs = [torch.zeros(count, device="cuda") for _ in range(n)]
        g.run("reduce_scatter", xs, outs, count, op="sum", algo=algo, k=k)
        _check_ok(g)
        ref = _ref_reduce(xs, "sum")
        for r in range(n):
            assert torch.allclose(outs[r], ref[r * count:(r + 1) * count], atol=_tol(torch.float32, n)), f"n={n} {algo} k={k} count={count} rank {r}"


@pytest.mark.parametrize("n", [2, 4, 8])
@pytest.mark.parametrize("algo", ALGOS)
def test_broadcast_and_reduce(groups, n, algo):
    g = groups(n)
    for count, root, k in [(5, 0, 2), (4097, n - 1, 4), (30000, n // 2, 2)]:
        xs = _inputs(n, count, torch.float32, seed=5)
        outs = [torch.zeros(count, device="cuda") for _ in range(n)]
        g.run("broadcast", xs, outs, count, root=root, algo=algo, k=k)
        _check_ok(g)
        for r in range(n):
            assert torch.equal(outs[r], xs[root]), f"bcast n={n} {algo} root={root} rank {r}"
        outs = [torch.full((count,), -5.0, device="cuda") for _ in range(n)]
        g.run("reduce", xs, outs, count, op="sum", root=root, algo=algo, k=k)
        _check_ok(g)
        assert torch.allclose(outs[root], _ref_reduce(xs, "sum"), atol=_tol(torch.float32, n))
        for r in range(n):
            if r != root:
                assert torch.all(outs[r] == -5.0), "non-root receive buffer must stay untouched"


def test_unaligned_buffers(groups):
    n = 4
    g = groups(n)
    count = 1237
    base = [torch.zeros(count + 8, device="cuda") for _ in range(n)]
    xs = [b[1:1 + count] for b in base]           # 4-byte aligned only
    for i, x in enumerate(xs):
        x.copy_(torch.arange(count, device="cuda") * 0.001 + i)
    outs_base = [torch.zeros(count + 8, device="cuda") for _ in range(n)]
    outs = [b[3:3 + count] for b in outs_base]
    g.run("allreduce", xs, outs, count, op="sum", algo="RING")
    _check_ok(g)
    ref = _ref_reduce([x.clone() for x in xs], "sum")
    for r in range(n):
        assert torch.allclose(outs[r], ref, atol=1e-4)
        assert outs_base[r][:3].abs().sum() == 0 and outs_base[r][3 + count:].abs().sum() == 0


def test_program_cache_and_stats(groups):
    n = 2
    g = groups(n)
    xs = _inputs(n, 4096, torch.float32)
    outs = [torch.empty_like(x) for x in xs]
    before = g.stats(0)
    for _ in range(3):
        g.run("allreduce", xs, outs, 4096, algo="RING")      # FIFO path: compiled programs are cached
    _check_ok(g)
    after = g.stats(0)
    assert after.calls[1] - before.calls[1] == 3
    assert after.program_cache_hits - before.program_cache_hits >= 2
    assert after.launches - before.launches == 3


def test_low_latency_path_matches_fifo_path(groups):
    # small exchange-type all-reduces run the flag-in-data kernel, large ones the FIFO executor: same values
    n = 8
    g = groups(n)
    for algo, k in [("PRD", 2), ("PRM", 8), ("RM", 4), ("RD", 2)]:
        for dtype in (torch.float32, torch.bfloat16):
            small = _inputs(n, 2000, dtype, seed=9)                       # 4-8 KB: low-latency kernel
            outs = [torch.empty_like(x) for x in small]
            before = g.stats(0).program_cache_misses + g.stats(0).program_cache_hits
            g.run("allreduce", small, outs, 2000, algo=algo, k=k)
            _check_ok(g)
            assert g.stats(0).program_cache_misses + g.stats(0).program_cache_hits == before, "expected the low-latency kernel"
            ref = _ref_reduce(small, "sum")
            tol = _tol(dtype, n) * 4
            for r in range(n):
                assert torch.allclose(outs[r].float(), ref, atol=tol, rtol=tol), f"{algo} {dtype} rank {r}"
                assert torch.equal(outs[r], outs[0])


@pytest.mark.parametrize("n", [2, 3, 8])
def test_low_latency_exchange_kernels(groups, n):
    """Small all-gather / reduce-scatter with a one-exchange schedule (DIRECT, PRM with radix = rank count) run the flag-in-data
    kernels of ll_exchange.cu; mixed with low-latency all-reduces back to back, no synchronisation, they share slots and epochs."""
    g = groups(n)
    launches0 = g.stats().launches
    for rep in range(3):
        results = []
        for dtype, op, count in [(torch.float32, "sum", 777), (torch.bfloat16, "avg", 4099), (torch.int32, "max", 1), (torch.float16, "min", 3000), (torch.float64, "prod", 17)]:
            xs = _inputs(n, n * count, dtype, seed=50 + rep)
            if op == "prod":
                xs = [x * 0 + 1 + 0.01 * (r + 1) for r, x in enumerate(xs)]
            outs = [torch.zeros(count, device="cuda", dtype=dtype) for _ in range(n)]
            g.run("reduce_scatter", xs, outs, count, op=op, algo="DIRECT")
            results.append(("rs", dtype, op, count, xs, outs))
            ys = _inputs(n, count, dtype, seed=60 + rep)
            gath = [torch.zeros(n * count, device="cuda", dtype=dtype) for _ in range(n)]
            g.run("allgather", ys, gath, count, algo="PRM", k=8 if n == 8 else n)
            results.append(("ag", dtype, op, count, ys, gath))
            zs = _inputs(n, count, dtype, seed=70 + rep)
            red = [torch.zeros_like(z) for z in zs]
            g.run("allreduce", zs, red, count, op="sum", algo="PRD" if n != 3 else "RING")
            results.append(("ar", dtype, "sum", count, zs, red))
        _check_ok(g)
        for kind, dtype, op, count, xs, outs in results:
            if kind == "ag":
                for r in range(n):
                    assert torch.equal(outs[r], torch.cat(xs)), f"allgather {dtype} {count} rank {r}"
            elif kind == "rs":
                ref = _ref_reduce(xs, op)
                for r in range(n):
                    got = outs[r].double() if dtype in (torch.int32, torch.int64) else outs[r].float()
                    assert torch.allclose(got, ref[r * count:(r + 1) * count].to(got.dtype), atol=_tol(dtype, n), rtol=2e-2), f"reduce_scatter {dtype} {op} {count} rank {r}"
            else:
                ref = _ref_reduce(xs, "sum")
                got = outs[0].double() if dtype in (torch.int32, torch.int64) else outs[0].float()
                assert torch.allclose(got, ref.to(got.dtype), atol=_tol(dtype, n) * 4, rtol=2e-2), f"allreduce {dtype} {count}"
    # unaligned user buffers and an odd number of bytes per rank
    base = [torch.arange(1, 1 + n * 1001 + 1, device="cuda", dtype=torch.uint8) + r for r in range(n)]
    xs = [b[1:1002] for b in base]
    outs_base = [torch.zeros(n * 1001 + 3, device="cuda", dtype=torch.uint8) for _ in range(n)]
    outs = [o[3:] for o in outs_base]
    g.run("allgather", xs, outs, 1001, algo="DIRECT")
    _check_ok(g)
    for r in range(n):
        assert torch.equal(outs[r], torch.cat(xs))
    # every call above was one launch
    assert g.stats().launches - launches0 == 3 * 15 + 1


def test_persistent_launcher_serves_and_leaves():
    # separate process: the launch mode is read from the environment when the library is loaded
    import os
    import subprocess
    import sys
    from pathlib import Path
    env = dict(os.environ, PICCL_LAUNCH="persistent", PICCL_PERSIST_IDLE_US="300")
    r = subprocess.run([sys.executable, str(Path(__file__).parent / "persistent_worker.py")], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "PERSISTENT_OK 45" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]


def test_bounded_wait_reports_instead_of_hanging():
    # a wait for data nobody sends runs into its limit; the kernel returns, the status says where
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    import ctypes as C
    from piccl_b200 import _native as N
    g = LoopbackGroup(1, config=make_config(max_cta=2, nslot=2, slot_bytes=4096, scratch_bytes=1 << 16, timeout_ms=300))
    lib = N.lib()
    t0 = torch.cuda.Event(enable_timing=True); t1 = torch.cuda.Event(enable_timing=True)
    t0.record()
    N.check(lib.piccl_test_unmatched_wait(g._hs[0], 300, torch.cuda.current_stream().cuda_stream), "unmatched wait")
    t1.record()
    torch.cuda.synchronize()
    st = g.status()
    assert st.aborted == 1 and st.code == 2 and st.peer == 0 and st.want == 1 and st.have == 0
    assert 250 < t0.elapsed_time(t1) < 3000
    # the communicator refuses further work instead of running on inconsistent counters
    x = torch.ones(16, device="cuda")
    with pytest.raises(N.PicclError):
        g.run("allreduce", [x], [x], 16)
    # the context is still usable
    assert float((x + 1).sum()) == 32.0
    g.close()


@pytest.mark.parametrize("count", [511, 512, 513, 9215, 9216, 9217, 18 * 512 * 4])
@pytest.mark.parametrize("coll,algo", [("allreduce", "PRM"), ("allgather", "DIRECT"), ("reduce_scatter", "DIRECT"), ("broadcast", "RING"), ("allgather", "RING")])
def test_low_latency_lines_spread_over_ctas(count, coll, algo):
    """Eight ranks leave 18 CTAs each: one line of 8 bytes per thread up to 18 x 256 lines (9216 fp32 elements), several beyond; the executor's low-latency
    variant spreads over up to 16 CTAs.  Sums of eight values below 1 in fp32: each of the seven additions errs by at most 2^-24 x 8."""
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    n = 8
    g = LoopbackGroup(n, config=make_config(max_cta=8, nslot=2, slot_bytes=4096, scratch_bytes=1 << 20, timeout_ms=5000))
    n_in = count * n if coll == "reduce_scatter" else count
    n_out = count * n if coll == "allgather" else count
    for seed in range(3):                                   # both parities of the call epoch
        xs = _inputs(n, n_in, torch.float32, seed=seed)
        outs = [torch.full((n_out,), float("nan"), device="cuda") for _ in range(n)]
        g.run(coll, xs, outs, count, op="sum", algo=algo, k=8)
        _check_ok(g)
        for r in range(n):
            if coll == "allgather":
                assert torch.equal(outs[r], torch.cat(xs))
            elif coll == "broadcast":
                assert torch.equal(outs[r], xs[0])
            else:
                ref = _ref_reduce(xs, "sum")
                ref = ref[r * count:(r + 1) * count] if coll == "reduce_scatter" else ref
                assert torch.allclose(outs[r], ref, atol=7 * 8 * 2.0 ** -24, rtol=0)
    g.close()


@pytest.mark.parametrize("dtype,offset", [(torch.uint8, 3), (torch.bfloat16, 1), (torch.float32, 3), (torch.float64, 1), (torch.bfloat16, 0)])
@pytest.mark.parametrize("coll,algo", [("allgather", "RING"), ("allgather", "PRD"), ("broadcast", "RING"), ("reduce_scatter", "RING"), ("reduce_scatter", "PRD"), ("allreduce", "RING"),
                                       ("allreduce", "PRM"), ("reduce", "RING"), ("allreduce", "DIRECT")])
def test_operands_at_any_address(groups, coll, algo, dtype, offset):
    """Messages too large for the low-latency path with operands that are not 16-byte aligned (a view that starts `offset` elements into its buffer, blocks of
    an odd length): every byte of the result, and the bytes around it untouched.  Whole numbers and byte moves are exact; values are small integers, so sums are too."""
    n, g = 4, groups(4)
    count = 70001 * (4 if dtype == torch.uint8 else 1)
    n_in, n_out = count * (n if coll == "reduce_scatter" else 1), count * (n if coll == "allgather" else 1)
    gen = torch.Generator(device="cuda").manual_seed(7)
    high = 30 if dtype == torch.uint8 else 9
    xs = [torch.randint(0, high, (n_in + 8,), generator=gen, device="cuda").to(dtype)[offset:offset + n_in] for _ in range(n)]
    bufs = [torch.full((n_out + 40,), 77, device="cuda").to(dtype) for _ in range(n)]
    outs = [b[16 + offset:16 + offset + n_out] for b in bufs]
    g.run(coll, xs, outs, count, op="sum", root=1, algo=algo, k=2)
    _check_ok(g)
    total = torch.stack([x.double() for x in xs]).sum(0)
    for r in range(n):
        if coll == "allgather":
            want = torch.cat(xs)
        elif coll == "broadcast":
            want = xs[1]
        elif coll == "reduce_scatter":
            want = total[r * count:(r + 1) * count].to(dtype)
        elif coll == "reduce" and r != 1:
            want = torch.full_like(outs[r], 77)
        else:
            want = total.to(dtype)
        assert torch.equal(outs[r], want), f"rank {r}"
        assert torch.all(bufs[r][:16 + offset] == 77) and torch.all(bufs[r][16 + offset + n_out:] == 77), f"rank {r} wrote outside its buffer"


@pytest.mark.parametrize("n,algo,k", [(2, "RING", 0), (3, "PRM", 3), (4, "PRD", 2), (4, "PRM", 4), (6, "PRM", 6), (7, "DIRECT", 0), (8, "PRM", 8), (8, "K_RING", 4), (8, "PRM", 2)])
def test_rounds_segments_and_windows(n, algo, k):
    """Default geometry (512 threads that move data, 128 KiB segments, two to a window): lengths around a round of four 16-byte packs per thread, around a segment, an odd
    number of segments, and a partial pack; two to eight operands per step.  Whole numbers: exact."""
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    ctas = min(64, 148 // n)
    g = LoopbackGroup(n, config=make_config(scratch_bytes=1 << 20, timeout_ms=5000))
    parts = n if algo == "K_RING" or algo == "RING" or algo == "DIRECT" else 1
    for per_cta in (8192, 8192 - 4, 8192 + 4, 3 * 32768 + 1):        # int32 elements of a CTA's slice
        count = per_cta * ctas * parts - 3
        xs = [torch.randint(-1000, 1001, (count,), generator=torch.Generator(device="cuda").manual_seed(r), dtype=torch.int32, device="cuda") for r in range(n)]
        outs = [torch.empty_like(x) for x in xs]
        want = torch.stack(xs).sum(0, dtype=torch.int32)
        for rep in range(2):
            g.run("allreduce", xs, outs, count, op="sum", algo=algo, k=k)
        _check_ok(g)
        for o in outs:
            assert torch.equal(o, want), (n, algo, per_cta)
        want = torch.stack(xs).max(0).values
        g.run("allreduce", xs, xs, count, op="max", algo=algo, k=k)      # in place
        _check_ok(g)
        for x in xs:
            assert torch.equal(x, want), (n, algo, per_cta)
    g.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,algo,k", [(2, "RING", -1), (8, "RING", -1), (4, "PRD", 2), (3, "PRM", 3), (4, "PRM", 4), (8, "PRM", 8), (8, "K_RING", 4), (5, "DIRECT", -1)])
def test_averaged_rounds_of_the_default_geometry(n, algo, k, dtype):
    """Default geometry (512 threads that move data): CTA slices of whole 16-byte packs, so that every offset is aligned, above the low-latency kernels' sizes and around full rounds of
    one, two, four and eight packs a thread (4096 packs are 1 of 8, 2 of 4 ...), with a segment more and a partial segment.  The scaled operand alone to one destination and to several, beside
    one (to one and two destinations), two and three, four and seven others.  Values and averages of 2, 4 and 8 ranks are multiples of 1 / 64 up to one: exact in each type."""
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    ctas, per_pack = min(64, 148 // n), 16 // torch.tensor([], dtype=dtype).element_size()
    parts = n if algo in ("RING", "K_RING", "DIRECT") else 1
    g = LoopbackGroup(n, config=make_config(scratch_bytes=1 << 20, timeout_ms=5000))
    for packs in (4097, 8191, 8192, 12289):
        count = packs * per_pack * ctas * parts
        xs = [torch.randint(-8, 9, (count,), generator=torch.Generator(device="cuda").manual_seed(packs + r), device="cuda").to(dtype) / 8 for r in range(n)]
        outs = [torch.full_like(x, float("nan")) for x in xs]
        want = sum(x.double() for x in xs) / n
        for rep in range(2):
            g.run("allreduce", xs, outs, count, op="avg", algo=algo, k=k)
        _check_ok(g)
        bound = 0.0 if n in (2, 4, 8) else 2 * n * 2.0 ** -{torch.float32: 24, torch.bfloat16: 9, torch.float16: 11}[dtype]
        for o in outs:
            assert (o.double() - want).abs().max() <= bound, (packs, o.dtype)
        g.run("allreduce", xs, xs, count, op="avg", algo=algo, k=k)      # in place
        _check_ok(g)
        assert all(torch.equal(x, o) for x, o in zip(xs, outs))
    g.close()


@pytest.mark.parametrize("dtype,offset", [(torch.float32, 0), (torch.bfloat16, 0), (torch.bfloat16, 1)])
@pytest.mark.parametrize("coll", ["allreduce", "allgather", "reduce_scatter", "broadcast", "reduce"])
def test_data_flow_is_the_programs_bit_for_bit(coll, dtype, offset):
    """Every algorithm on three, four and eight ranks: the ranks' programs through the slots and the call's data flow, in turn on one communicator, from a captured graph
    too, and with a receive buffer that is another rank's send buffer (programs, whatever was asked for).  Operands are combined and rounded alike: the same bits, also of averages, and of
    maxima of zeros of both signs and values that are not numbers."""
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    for n, k in ((3, 2), (4, 2), (8, 2), (8, 4)):
        g = LoopbackGroup(n, config=make_config(scratch_bytes=1 << 20, timeout_ms=5000))
        count = 40013 if coll in ("allgather", "reduce_scatter") else 180013 * n      # (above the sizes that other kernels take outside a capture)
        n_in, n_out = count * (n if coll == "reduce_scatter" else 1), count * (n if coll == "allgather" else 1)
        ins = {"avg": [x[offset:] for x in _inputs(n, n_in + offset, dtype, seed=3)]}
        odd = torch.tensor([0.0, -0.0, float("nan"), 1.0, -1.0, float("inf"), -float("inf")], device="cuda", dtype=dtype)
        ins["max"] = [odd[torch.randint(0, 7, (n_in + offset,), generator=torch.Generator(device="cuda").manual_seed(r), device="cuda")][offset:] for r in range(n)]
        for algo, op in itertools.product(ALGOS, ["avg", "max"] if coll in ("allreduce", "reduce_scatter", "reduce") else ["avg"]):
            xs, op = ins[op], "sum" if coll in ("allgather", "broadcast") else op
            outs = [[torch.full((n_out + offset,), 7.0, device="cuda", dtype=dtype)[offset:] for _ in range(n)] for _ in range(3)]
            for variant, slots in enumerate((1, 0)):
                for h in g._hs:
                    g._lib.piccl_test_slots_only(h, slots)
                for _ in range(2):
                    g.run(coll, xs, outs[variant], count, op=op, root=1, algo=algo, k=k)
            _check_ok(g)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                g.run(coll, xs, outs[2], count, op=op, root=1, algo=algo, k=k)
            for _ in range(2):
                graph.replay()
            _check_ok(g)
            bits = lambda t: t.clone().view(torch.int16 if dtype == torch.bfloat16 else torch.int32)
            for r in range(n):
                assert torch.equal(bits(outs[0][r]), bits(outs[1][r])) and torch.equal(bits(outs[0][r]), bits(outs[2][r])), (coll, algo, op, n, k, r)
            if n_in == n_out and coll != "broadcast" and op == "avg":       # rank 0 receives into rank 1's send buffer (the ring's sums contain what they overwrite)
                ys = [x.clone() for x in xs]
                zs = [ys[1]] + [torch.full_like(x, 7.0) for x in xs[1:]]
                if coll == "reduce":
                    zs[1], zs[0] = ys[2], zs[1]
                g.run(coll, ys, zs, count, op=op, root=1, algo="RING")
                _check_ok(g)
                g.run(coll, xs, outs[0], count, op=op, root=1, algo="RING")
                _check_ok(g)
                assert torch.equal(zs[1], outs[0][1])
        g.close()


@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float32, torch.float64])
@pytest.mark.parametrize("coll,n,algo,op", [("allgather", 3, "RING", "sum"), ("broadcast", 8, "PRD", "sum"), ("reduce", 2, "RING", "max"), ("reduce_scatter", 4, "DIRECT", "sum"), ("allreduce", 5, "PRM", "avg"), ("allreduce", 4, "PRD", "sum"), ("reduce", 8, "K_RING", "max"),
                                            ("allreduce", 8, "DIRECT", "min")])
def test_slices_of_a_data_flow(coll, n, algo, op, dtype):
    """Blocks of 4 KiB to 64 KiB: one element, a pack and its neighbours, a block and its neighbours, several blocks, a message whose blocks are larger; operands and results
    3 elements into their buffers too.  Small whole numbers: exact but for fifths, whose sum of five rounded operands errs by half a unit each and once more."""
    from piccl_b200.parallel.comm import LoopbackGroup, make_config
    if op == "avg" and dtype == torch.uint8:
        pytest.skip("integers are not averaged")
    g = LoopbackGroup(n, config=make_config(scratch_bytes=1 << 20, timeout_ms=5000))
    esz = torch.tensor([], dtype=dtype).element_size()
    big = 1200001 if coll in ("allgather", "reduce_scatter") else 4200001
    for nbytes, off in itertools.product([esz, 16, 16 + esz, 4096 - esz, 4096, 4096 + esz, 5 * 4096 + 8, big // esz * esz], [0, 3]):
        count = max(1, nbytes // esz)
        n_in, n_out = count * (n if coll == "reduce_scatter" else 1), count * (n if coll == "allgather" else 1)
        gen = torch.Generator(device="cuda").manual_seed(nbytes)
        xs = [torch.randint(0, 9, (n_in + off,), generator=gen, device="cuda").to(dtype)[off:] for _ in range(n)]
        bufs = [torch.full((n_out + off + 8,), 77, device="cuda").to(dtype) for _ in range(n)]
        outs = [b[off:off + n_out] for b in bufs]
        g.run(coll, xs, outs, count, op=op, root=1, algo=algo, k=8)
        _check_ok(g)
        st = torch.stack([x.double() for x in xs])
        total = st.max(0).values if op == "max" else st.min(0).values if op == "min" else st.mean(0) if op == "avg" else st.sum(0)
        for r in range(n):
            want = torch.cat(xs) if coll == "allgather" else xs[1] if coll == "broadcast" else total[r * count:(r + 1) * count] if coll == "reduce_scatter" else total
            if coll == "reduce" and r != 1:
                want = torch.full_like(outs[r], 77)
            bound = 0.0 if op != "avg" else 2 * n * 2.0 ** -{torch.float32: 24, torch.bfloat16: 9, torch.float64: 24}[dtype] * 8       # (1 / 5 is an fp32 factor)
            assert (outs[r].double() - want.double()).abs().max() <= bound, (count, off, r)
            assert torch.all(bufs[r][:off] == 77) and torch.all(bufs[r][off + n_out:] == 77), (count, off, r)
    g.close()
