"""The per-rank action programs executed by real processes over gloo (world size 4 and 3), compared with
torch.distributed's own collectives."""
import os
import sys
from pathlib import Path

import pytest
import torch
import torch.distributed as dist
import torch.multiprocessing as mp

ROOT = Path(__file__).resolve().parent.parent
ALGOS = ["RING", "K_RING", "RD", "RM", "PRD", "PRM", "DIRECT"]


def _worker(rank, world, port, q):
    try:
        sys.path.insert(0, str(ROOT))
        os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port))
        dist.init_process_group("gloo", rank=rank, world_size=world)
        from piccl_b200.parallel.host_exec import host_collective
        count = 37
        for algo in ALGOS:
            for k in (2, 3):
                g = torch.Generator().manual_seed(1000 + rank)
                x = torch.randint(-50, 50, (count,), generator=g, dtype=torch.int64)
                # allreduce
                want = x.clone(); dist.all_reduce(want)
                out = torch.zeros(count, dtype=torch.int64)
                host_collective("allreduce", algo, x, out, count, k=k)
                assert torch.equal(out, want), ("allreduce", algo, k)
                # allgather
                ref = [torch.zeros(count, dtype=torch.int64) for _ in range(world)]
                dist.all_gather(ref, x)
                out = torch.zeros(world * count, dtype=torch.int64)
                host_collective("allgather", algo, x, out, count, k=k)
                assert torch.equal(out, torch.cat(ref)), ("allgather", algo, k)
                # reduce_scatter (max)
                big = torch.randint(-50, 50, (world * count,), generator=g, dtype=torch.int64)
                full = big.clone(); dist.all_reduce(full, op=dist.ReduceOp.MAX)
                out = torch.zeros(count, dtype=torch.int64)
                host_collective("reduce_scatter", algo, big, out, count, k=k, op="max")
                assert torch.equal(out, full[rank * count:(rank + 1) * count]), ("reduce_scatter", algo, k)
                # broadcast / reduce, root = last rank
                root = world - 1
                b = x.clone(); dist.broadcast(b, src=root)
                out = torch.zeros(count, dtype=torch.int64)
                host_collective("broadcast", algo, x, out, count, k=k, root=root)
                assert torch.equal(out, b), ("broadcast", algo, k)
                r = x.clone(); dist.reduce(r, dst=root)
                out = torch.full((count,), -7, dtype=torch.int64)
                host_collective("reduce", algo, x, out, count, k=k, root=root)
                if rank == root:
                    assert torch.equal(out, r), ("reduce", algo, k)
                else:
                    assert torch.all(out == -7)
        dist.barrier()
        dist.destroy_process_group()
        q.put((rank, "ok"))
    except Exception as e:  # noqa: BLE001
        q.put((rank, f"{type(e).__name__}: {e}"))


@pytest.mark.parametrize("world,port", [(4, 29671), (3, 29672)])
def test_programs_over_gloo(world, port):
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    procs = [ctx.Process(target=_worker, args=(r, world, port, q)) for r in range(world)]
    for p in procs:
        p.start()
    results = []
    for _ in range(world):
        results.append(q.get(timeout=240))
    for p in procs:
        p.join(timeout=60)
        if p.is_alive():
            p.terminate()       # this exact child
    assert all(msg == "ok" for _, msg in results), results


def _fault_worker(rank, world, port, q):
    import datetime
    import time
    try:
        sys.path.insert(0, str(ROOT))
        os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port))
        dist.init_process_group("gloo", rank=rank, world_size=world, timeout=datetime.timedelta(seconds=4))
        from piccl_b200.parallel.host_exec import host_collective
        x = torch.ones(16)
        out = torch.zeros(16)
        host_collective("allreduce", "RING", x, out, 16)          # a healthy call first
        assert torch.all(out == world)
        if rank == 1:
            q.put((rank, "left"))                                  # this rank never joins the next collective
            time.sleep(8)
            return
        t0 = time.time()
        try:
            host_collective("allreduce", "RING", x, out, 16)
            q.put((rank, "no error"))
        except Exception as e:  # noqa: BLE001
            q.put((rank, f"error after {time.time() - t0:.1f}s: {type(e).__name__}"))
    except Exception as e:  # noqa: BLE001
        q.put((rank, f"setup failed: {type(e).__name__}: {e}"))


def test_rank_that_never_joins_is_reported_within_the_time_limit():
    """Failure made on the host, no GPU involved: one of two ranks skips a collective; the other one's receive
    ends with an error when the process-group time limit runs out instead of waiting for ever."""
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    procs = [ctx.Process(target=_fault_worker, args=(r, 2, 29673, q)) for r in range(2)]
    for p in procs:
        p.start()
    results = dict(q.get(timeout=120) for _ in range(2))
    for p in procs:
        p.join(timeout=30)
        if p.is_alive():
            p.terminate()
    assert results[1] == "left"
    assert results[0].startswith("error after"), results
    assert float(results[0].split()[2].rstrip("s:")) < 30


def test_tensor_parallel_flags_of_neighbouring_calls_do_not_overlap():
    """A rank may be one call ahead of a peer, of another shape or of the other kernel: no flag of the one call lies where the other's do."""
    import ctypes as C
    import itertools
    from piccl_b200 import _native as N
    lib = N.lib()

    def flags(which, n, M, cols, parity):
        lo, hi = C.c_longlong(), C.c_longlong()
        rc = lib.piccl_tp_flag_range(which, n, M, cols, parity, C.byref(lo), C.byref(hi))
        return (lo.value, hi.value) if rc == 0 else None

    for n in range(1, 9):
        shapes = [(128 * n * b, 256 * c) for b in (1, 2, 3, 8, 16, 61) for c in (1, 5, 32, 128)]
        calls = {s: [[flags(w, n, *s, p) for p in (0, 1)] for w in (0, 1)] for s in shapes}
        usable = [(s, w) for s in shapes for w in (0, 1) if calls[s][w][0] is not None]
        assert len(usable) > len(shapes)
        for (s, w), (t, v) in itertools.product(usable, usable):
            for p, q in itertools.product((0, 1), (0, 1)):
                if (w, p) == (v, q):
                    continue
                a, b = calls[s][w][p], calls[t][v][q]
                assert 0 <= a[0] < a[1] <= 1 << 20
                assert a[1] <= b[0] or b[1] <= a[0], (n, s, w, p, t, v, q)


def test_heads_of_unequal_width_are_refused():
    from piccl_b200.models.gpt2 import GPT2, GPT2Config
    model = GPT2(GPT2Config(vocab_size=100, seq_len=16, n_layer=1, n_head=30, d_model=256), device="cpu")
    idx = torch.zeros(2, 16, dtype=torch.int64)
    for run in (model.loss, model.forward_backward, lambda a, b: model.forward_backward(a, b, on_grads_ready=lambda end: None)):
        with pytest.raises(RuntimeError, match="heads"):
            run(idx, idx)


def test_a_group_call_without_an_operand_is_refused():
    """A rank that receives nothing may have no receive buffer; every rank has something to send, and a missing tensor must not become a null pointer."""
    import struct
    from piccl_b200.parallel.comm import LoopbackGroup

    class Stream:
        cuda_stream = 0

    class Recorder:
        calls = 0

        def piccl_group_collective(self, *args):
            self.calls += 1
            return 0

    g = LoopbackGroup.__new__(LoopbackGroup)
    g._lib, g.nranks, g._hs, g._comms, g._pack = Recorder(), 2, [], b"", struct.Struct("2Q").pack
    a, b, stream = torch.ones(4), torch.ones(4), Stream()
    g.run("reduce", [a, b], [a, None], 4, stream=stream)
    assert g._lib.calls == 1
    with pytest.raises(AttributeError):
        g.run("reduce", [a, None], [a, b], 4, stream=stream)
    assert g._lib.calls == 1


def test_bench_names_the_launch_mode_from_what_happened():
    import bench
    assert bench.replay_share(0, 23) == "issued call by call"
    assert bench.replay_share(21, 23).startswith("21 of 23 steps replayed")
