"""The Python front end without its native call path, which needs Python's development headers to be built."""
import struct
import sysconfig

import torch


class _Library:
    """Takes the calls of a group and notes their arguments."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args: self.calls.append((name, args)) or 0


def _group(lib, n=2):
    from piccl_b200.parallel.comm import LoopbackGroup
    g = object.__new__(LoopbackGroup)
    g._lib, g.nranks, g._hs, g._pack, g._comms = lib, n, [], struct.Struct(f"{n}Q").pack, b"\0" * 8 * n
    return g


def test_build_without_python_headers(monkeypatch, tmp_path):
    from piccl_b200 import _native as N, build as B
    assert "_fastcall.so" in B.targets()
    paths = dict(sysconfig.get_paths(), include=str(tmp_path))
    monkeypatch.setattr(sysconfig, "get_paths", lambda *a, **k: paths)
    plan = B.targets()
    assert "_fastcall.so" not in plan and {"piccl.so", "libpiccl_ops.so", "libpiccl_model.so", "piccl_sched", "coll_bench", "loggp_bench"} == set(plan)
    monkeypatch.setattr(N, "_LIB_DIR", tmp_path)
    monkeypatch.setattr(N, "_libs", {})
    assert N.fastcall() is None


def test_calls_through_ctypes(monkeypatch):
    from piccl_b200 import _native as N
    from piccl_b200.parallel import tp
    lib = _Library()
    g = _group(lib)
    xs = [torch.ones(4), torch.ones(4)]
    assert g.table([xs[0], None]) == struct.pack("2Q", xs[0].data_ptr(), 0)
    g.run("reduce", xs, [xs[1], None], 4, op="max", root=0, algo="PRD", stream=type("S", (), {"cuda_stream": 0}))
    name, args = lib.calls[-1]
    assert name == "piccl_group_collective"
    assert args[1:] == (2, N.COLL["reduce"], struct.pack("2Q", *[x.data_ptr() for x in xs]), struct.pack("2Q", xs[1].data_ptr(), 0), 4, N.DTYPE["float32"], N.OP["max"], 0, N.ALGO["PRD"], -1, 0)
    monkeypatch.setattr(N, "fastcall", lambda: None)
    monkeypatch.setattr(tp, "_declare", lambda: lib)
    a = [torch.zeros(256, 64, dtype=torch.bfloat16) for _ in range(2)]
    tp.gemm_rs_group(g, a, a, a, stream=type("S", (), {"cuda_stream": 7}))
    table = struct.pack("2Q", *[x.data_ptr() for x in a])
    assert lib.calls[-1] == ("piccl_gemm_rs_group", (g.handles(), 2, table, table, table, 256, 256, 64, 7))
