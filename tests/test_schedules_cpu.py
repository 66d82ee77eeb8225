"""CPU data-flow validation of every collective x algorithm x k x rank count
(the reference ships no such test; its only check is the external OSU validation
run, README.md:40-44)."""
import itertools
import json
import subprocess
import xml.etree.ElementTree as ET
from pathlib import Path

import pytest

from piccl_b200 import schedule as S

COLLS = ["allgather", "allreduce", "broadcast", "reduce", "reduce_scatter"]
ALGOS = ["RING", "K_RING", "RD", "RM", "PRD", "PRM", "DIRECT"]


@pytest.mark.parametrize("coll", COLLS)
@pytest.mark.parametrize("algo", ALGOS)
def test_all_rank_counts_and_radices(coll, algo):
    for n, k, in_place in itertools.product([1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 16], [-1, 2, 3, 4, 8], [False, True]):
        v = S.validate(coll, algo, n, 257, k=k, root=n // 2, in_place=in_place, n_cta=3, seg_elems=32)
        assert v.ok, f"{coll} {algo} n={n} k={k} in_place={in_place}: {v.error}"


@pytest.mark.parametrize("algo", ALGOS)
def test_deferred_counter_updates_never_deadlock(algo):
    """The executor publishes its FIFO counters behind the data it moves (exec_impl.cuh).  Published as late as can be, when the rank is about to block:
    every schedule still terminates with the right data, also with the smallest FIFO."""
    for coll in COLLS:
        for n, k, in_place in itertools.product([2, 3, 4, 6, 8, 9, 16], [-1, 2, 4, 8], [False, True]):
            v = S.validate(coll, algo, n, 257, k=k, root=n - 1, in_place=in_place, n_cta=2, seg_elems=32, fifo_cap=2, deferred=True)
            assert v.ok, f"{coll} {algo} n={n} k={k} in_place={in_place}: {v.error}"


@pytest.mark.parametrize("coll", COLLS)
@pytest.mark.parametrize("algo", ALGOS)
def test_windows_of_segments_never_deadlock(coll, algo):
    """The executor's order with the FIFOs it uses: one segment at a time below four slots, windows of two from there on; one, an odd and an even number of
    segments, counters published at once and as late as can be."""
    for n, k, in_place in itertools.product([2, 3, 4, 6, 7, 8, 9, 16], [-1, 2, 4, 8], [False, True]):
        for fifo, count, deferred in itertools.product([3, 4, 5], [30, 32 * 2 * 3 * n, 257], [False, True]):
            v = S.validate(coll, algo, n, count, k=k, root=n - 1, in_place=in_place, n_cta=2, seg_elems=32, fifo_cap=fifo, deferred=deferred)
            assert v.ok, f"{coll} {algo} n={n} k={k} in_place={in_place} fifo={fifo} count={count} deferred={deferred}: {v.error}"


def test_a_window_needs_its_slots():
    """Two segments to a window with one slot for each: a rank that receives and forwards waits for a slot that only its own later step frees."""
    assert S.validate("allreduce", "RING", 4, 2048, n_cta=1, seg_elems=32, fifo_cap=4, window=2).ok
    v = S.validate("allreduce", "RING", 4, 2048, n_cta=1, seg_elems=32, fifo_cap=2, window=2)
    assert not v.ok and "deadlock" in v.error


@pytest.mark.parametrize("op", ["sum", "prod", "max", "min"])
@pytest.mark.parametrize("integer", [False, True])
def test_ops_exact_for_integers(op, integer):
    for coll, algo in itertools.product(["allreduce", "reduce", "reduce_scatter"], ALGOS):
        v = S.validate(coll, algo, 8, 500, k=4, op=op, integer=integer, n_cta=2, seg_elems=64)
        assert v.ok, f"{coll} {algo} {op}: {v.error}"
        if integer:
            assert v.max_abs_err == 0.0


def test_headline_config_p8_fp32_sum_small_sizes_with_data():
    # allreduce, p = 8, RING / K_RING k=2,4 / PRD / PRM k=2,8, seed-0 uniform[-1,1) fp32 against a serial sum
    for algo, k in [("RING", -1), ("K_RING", 2), ("K_RING", 4), ("PRD", -1), ("PRM", 2), ("PRM", 8)]:
        for nbytes in [8, 64, 4096, 1 << 16, 1 << 20]:
            v = S.validate("allreduce", algo, 8, nbytes // 4, k=k, n_cta=4, seg_elems=4096)
            assert v.ok, f"{algo} k={k} {nbytes} B: {v.error}"
            assert v.max_abs_err < 1e-4


def test_headline_config_large_sizes_symbolic():
    # up to 1 GiB the programs are checked for FIFO order and complete output coverage without data
    for algo, k in [("RING", -1), ("K_RING", 2), ("K_RING", 4), ("PRD", -1), ("PRM", 2), ("PRM", 8)]:
        for nbytes in [1 << 24, 1 << 27, 1 << 30]:
            v = S.validate("allreduce", algo, 8, nbytes // 4, k=k, n_cta=32, symbolic=True)
            assert v.ok, f"{algo} k={k} {nbytes} B: {v.error}"


def test_traffic_matches_cost_model():
    n, count = 8, 8 * 1024
    S_bytes = count * 4
    v = S.validate("allreduce", "RING", n, count, n_cta=1, seg_elems=count)
    assert v.bytes_sent_max_rank == 2 * (n - 1) * S_bytes // n
    v = S.validate("allreduce", "PRD", n, count, n_cta=1, seg_elems=count)
    assert v.bytes_sent_max_rank == 3 * S_bytes
    v = S.validate("allreduce", "PRM", n, count, k=8, n_cta=1, seg_elems=count)
    assert v.bytes_sent_max_rank == 7 * S_bytes
    for algo in ALGOS:
        v = S.validate("allgather", algo, n, count, k=2, n_cta=1, seg_elems=count, elem_size=4)
        assert v.bytes_sent_max_rank == (n - 1) * S_bytes, algo


def test_direct_schedules_move_the_minimum_in_two_exchanges():
    n, count = 8, 7 * 8 * 1024
    S_bytes = count * 4
    # all-reduce: the ring's traffic in 3 steps (contributions out, reduce + sums out, sums stored)
    v = S.validate("allreduce", "DIRECT", n, count, n_cta=1, seg_elems=count)
    assert v.ok and v.bytes_sent_max_rank == 2 * (n - 1) * S_bytes // n
    assert json.loads(S.schedule_json("allreduce", "DIRECT", n, count, 3))["steps"] == 3
    prog = json.loads(S.schedule_json("allreduce", "DIRECT", n, count, 3))["actions"]
    assert [len(a["send"]) for a in prog] == [1] * 7 + [7] + [0] * 7 and [len(a["recv"]) for a in prog] == [0] * 7 + [7] + [1] * 7
    # broadcast: nobody sends more than the message, the root sends it exactly once
    v = S.validate("broadcast", "DIRECT", n, count, root=5, n_cta=1, seg_elems=count)
    assert v.ok and v.bytes_sent_max_rank == S_bytes
    # reduce: each rank sends at most its vector once
    v = S.validate("reduce", "DIRECT", n, count, root=2, n_cta=1, seg_elems=count)
    assert v.ok and v.bytes_sent_max_rank == S_bytes
    # all-gather / reduce-scatter resolve to one exchange with everybody
    r = S.resolve("allgather", "DIRECT", -1, n)
    assert (r.algo, r.k, r.radices) == ("PRM", 8, [8])
    # more than 8 ranks: one action cannot address everybody
    assert S.resolve("allreduce", "DIRECT", -1, 12).algo == "RING"


def test_permutation_oracle_vectors():
    # values of the reference's index formula (src/kernels/permutation_kernel.cu:166-207)
    assert S.permutation_index(0, 8, 2) == [0, 4, 2, 6, 1, 5, 3, 7]
    assert S.permutation_index(1, 8, 2) == [1, 5, 3, 7, 0, 4, 2, 6]
    assert S.permutation_index(3, 8, 2) == [3, 7, 1, 5, 2, 6, 0, 4]
    assert S.permutation_index(7, 8, 2) == [7, 3, 5, 1, 6, 2, 4, 0]
    assert S.permutation_index(5, 8, 8) == [5, 6, 7, 0, 1, 2, 3, 4]
    assert S.permutation_index(4, 9, 3) == [4, 7, 1, 5, 8, 2, 3, 6, 0]
    assert S.permutation_index(8, 9, 3) == [8, 2, 5, 6, 0, 3, 7, 1, 4]
    assert S.permutation_index(6, 16, 4) == [6, 10, 14, 2, 7, 11, 15, 3, 4, 8, 12, 0, 5, 9, 13, 1]
    assert S.permutation_index(5, 16, 2) == [5, 13, 1, 9, 7, 15, 3, 11, 4, 12, 0, 8, 6, 14, 2, 10]
    assert S.permutation_index(1, 8, 4) is None     # 8 is not a power of 4
    assert S.permutation_index(0, 6, 2) is None


def test_direct_placement_equals_permutation_table():
    # the block a permuted-recursive rank holds in receive order q is exactly perm[q]
    for n, b in [(8, 2), (4, 2), (16, 2), (9, 3), (16, 4), (8, 8)]:
        rad = S.resolve("allgather", "PRM", b, n).radices
        assert all(f == b for f in rad)
        for r in range(n):
            assert S.held_blocks(r, len(rad), rad, n, True) == S.permutation_index(r, n, b)


def test_resolve_defines_the_cases_the_reference_leaves_undefined():
    r = S.resolve("allgather", "PRM", 4, 8)          # reference: out-of-bounds writes
    assert sorted(r.radices) == [2, 4] and "mixed" in r.note
    r = S.resolve("allgather", "K_RING", 4, 2)       # reference: silently does nothing
    assert r.k == 2
    r = S.resolve("allreduce", "PRM", -1, 8)         # reference: K unset = -1, undefined behaviour
    assert r.k == 2 and r.radices == [2, 2, 2]
    r = S.resolve("allreduce", "K_RING", 3, 8)       # k does not divide n: plain ring, as the reference
    assert r.k == 8
    r = S.resolve("allreduce", "PRD", -1, 11)        # prime rank count: power-of-two core + followers
    assert r.core == 8
    r = S.resolve("allgather", "RD", -1, 11)
    assert r.algo == "RING"


def test_xml_is_well_formed_with_integer_sizes():
    for coll, algo, k in itertools.product(COLLS, ALGOS, [2, 4]):
        xml = S.schedule_xml(coll, algo, 8, 1024, k=k)
        root = ET.fromstring(xml)
        assert root.tag == "collective" and root.get("nodes") == "8"
        ids = set()
        for t in root.findall("transfer"):
            ids.add(int(t.get("id")))
            assert int(t.get("size")) > 0
            assert 0 <= int(t.get("src")) < 8 and 0 <= int(t.get("dst")) < 8 and t.get("src") != t.get("dst")
        for t in root.findall("transfer"):
            for d in t.get("deps").split(","):
                assert int(d) == -1 or int(d) in ids
        assert len(ids) > 0


def test_xml_transfer_counts():
    n = 8
    count = lambda **kw: len(ET.fromstring(S.schedule_xml(**kw)).findall("transfer"))
    assert count(coll="allgather", algo="RING", nranks=n, count=64) == n * (n - 1)
    assert count(coll="allreduce", algo="RING", nranks=n, count=64 * n) == 2 * n * (n - 1)
    assert count(coll="allreduce", algo="K_RING", nranks=n, count=64 * n, k=2) == 2 * n * (n - 1)
    assert count(coll="allreduce", algo="PRD", nranks=n, count=64) == 3 * n
    assert count(coll="allreduce", algo="PRM", nranks=n, count=64, k=8) == n * (n - 1)
    assert count(coll="broadcast", algo="RING", nranks=n, count=64) == n - 1
    assert count(coll="reduce", algo="PRD", nranks=n, count=64) == n - 1


def test_cache_priorities_are_for_launches_that_carry_every_rank():
    """The executor's evict-first priorities were measured with all ranks on one GPU, where the FIFO's slots and the caller's buffers share its cache."""
    from piccl_b200 import _native as N
    f = N.lib().piccl_test_leave_first
    for coll in N.COLL.values():
        for n in (2, 4, 8):
            assert f(coll, n, n, 1, 1 << 30), (coll, n)
            assert not f(coll, n, 1, 1, 1 << 30), (coll, n)             # one rank per launch, whether or not its GPU has others
            assert not f(coll, n, n, 0, 1 << 30), (coll, n)
            assert not f(coll, n, n // 2, 1, 1 << 30) or n // 2 == n, (coll, n)
            assert not f(coll, n, n, 1, 1 << 16), (coll, n)


def test_results_that_the_cache_can_keep_stay_there():
    """Results of 64 MiB in all are worth more to their reader in the cache than to the call; those beyond its 126 MB leave first, and operands from lower lines on."""
    from piccl_b200 import _native as N
    f, MiB = N.lib().piccl_test_leave_first, 1 << 20
    for coll, n, block, want in [("reduce_scatter", 2, 32, 1), ("broadcast", 4, 16, 1), ("allgather", 4, 4, 1), ("allgather", 2, 26, 1), ("allreduce", 2, 40, 1),
                                 ("allreduce", 8, 12, 1), ("reduce", 4, 32, 1), ("allgather", 4, 8, 3), ("reduce_scatter", 2, 64, 3), ("broadcast", 8, 32, 3), ("allreduce", 4, 25, 3),
                                 ("allreduce", 8, 64, 3), ("reduce", 2, 128, 3), ("allreduce", 8, 8, 0), ("allgather", 8, 1, 0), ("reduce_scatter", 2, 8, 0), ("broadcast", 8, 8, 0)]:
        assert f(N.COLL[coll], n, n, 1, block * MiB) == want, (coll, n, block)


@pytest.mark.parametrize("coll", COLLS)
@pytest.mark.parametrize("algo", ALGOS)
def test_data_flow(coll, algo):
    """What the programs of all ranks compute, as expressions over the send buffers (flow.cc): every algorithm on two to eight ranks has that form and gives the same data, odd
    lengths, strides wider than a block and what may be in place included."""
    for n, k, root in itertools.product(range(2, 9), [-1, 2, 3, 4, 8], [0, 1]):
        for count, in_place in itertools.product([1, 5, 257], [False, True] if coll in ("allgather", "broadcast") else [False]):
            v = S.validate(coll, algo, n, count, k=k, root=root, in_place=in_place, flow=True)
            assert v.ok and v.fifo_entries == 0, f"{coll} {algo} n={n} k={k} count={count} in_place={in_place}: {v.error}"
        if coll in ("allgather", "reduce_scatter"):
            assert S.validate(coll, algo, n, 100, k=k, stride=130, flow=True).ok
        v = S.validate(coll, algo, n, 40, k=k, root=root, op="max", integer=True, flow=True)
        assert v.ok and v.max_abs_err == 0.0


def test_sums_in_place_have_no_data_flow():
    """A rank could overwrite what another is still to read."""
    assert all(not S.validate(c, "RING", 4, 100, in_place=True, flow=True).ok for c in ("allreduce", "reduce", "reduce_scatter"))
    assert not S.validate("allgather", "RING", 9, 100, flow=True).ok


@pytest.fixture(scope="module")
def flow_main(tmp_path_factory):
    out = tmp_path_factory.mktemp("flow") / "flow_main"
    root = Path(__file__).resolve().parent.parent
    cmd = ["g++", "-std=c++17", "-O1", "-g", "-Wall", "-Werror", f"-I{root / 'src' / 'include'}", *map(str, sorted((root / "src" / "coll").glob("*.cc"))), str(root / "tests" / "native" / "flow_main.cc"), "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return lambda what: subprocess.run([str(out), what], capture_output=True, text=True, timeout=120).stdout.strip()


def test_data_flow_of_integers_is_one_fold(flow_main):
    """Nothing is rounded on the way, so the nesting of the programs does not show in the result."""
    assert flow_main("integers") == "OK"


def test_data_flow_of_a_result_with_many_destinations(flow_main):
    assert flow_main("destinations") == "OK"


def test_operations_of_a_data_flow_are_checked(flow_main):
    """What PICCL_DEBUG=1 runs on a fresh data flow, as it checks fresh programs."""
    assert flow_main("checked") == "OK"
