"""Performance cases of the framework on one GPU: training and evaluation steps, the tcgen05 matrix product, collectives and the
fused tensor-parallel kernels, each through the call that a user's program makes.

Collectives and tensor-parallel kernels run as virtual ranks of a LoopbackGroup: one cooperative launch that carries every rank's
program.  Requests that would go through the NVSwitch are left out (one GPU has no switch, its emulation says nothing about
speed): AUTO stands for the sizes where it picks a peer-to-peer or low-latency path.
"""
import math

import torch

from piccl_b200.models.gpt2 import GPT2, GPT2Config
from piccl_b200.ops import gemm_sm100
from piccl_b200.parallel import tp
from piccl_b200.parallel.comm import LoopbackGroup, make_config
from piccl_b200.train import DataParallelTrainer

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16, "int32": torch.int32}


def listed():
    return [
        # one optimiser step of the smallest configuration: hundreds of launches of a few microseconds each, the host path counts
        {"name": "train_tiny", "path": "train", "layers": 2, "d_model": 256, "heads": 4, "vocab": 1000, "batch": 4, "seq": 128},
        # a mid-size model on a ragged batch (rows no multiple of any tile), as a last batch or packed documents give it
        {"name": "train_ragged", "path": "train", "layers": 8, "d_model": 768, "heads": 12, "vocab": 50257, "batch": 3, "seq": 777},
        # the headline configuration: GPT-2 medium, 8 x 1024 tokens per GPU, forward, backward, AdamW, loss read back
        {"name": "train_medium", "path": "train", "layers": 24, "d_model": 1024, "heads": 16, "vocab": 50257, "batch": 8, "seq": 1024},
        # validation loss of the same model on a batch of another shape: forward only
        {"name": "eval_medium", "path": "eval", "layers": 24, "d_model": 1024, "heads": 16, "vocab": 50257, "batch": 5, "seq": 1000},
        # the matrix product alone, at the shape of a tensor-parallel shard (compute bound)
        {"name": "linear_8192x8192x3584", "path": "linear", "m": 8192, "n": 8192, "k": 3584, "bias": False, "gelu": False},
        # latency: an all-reduce of 1 KiB among eight ranks (norms, flags, small gradients)
        {"name": "allreduce_1KiB", "path": "coll", "coll": "allreduce", "ranks": 8, "count": 256, "dtype": "fp32", "op": "sum", "algo": "AUTO", "k": -1},
        # a gradient bucket of 25 MB, averaged, with an odd length, by parallel recursive doubling
        {"name": "allreduce_bucket", "path": "coll", "coll": "allreduce", "ranks": 4, "count": 13107199, "dtype": "bf16", "op": "avg", "algo": "PRD", "k": 2},
        # the bandwidth end of the sweep: 64 MiB per rank among eight ranks on the ring
        {"name": "allreduce_64MiB", "path": "coll", "coll": "allreduce", "ranks": 8, "count": 16777216, "dtype": "fp32", "op": "sum", "algo": "RING", "k": -1},
        # parameter gathering: bf16 shards of about 1 MiB in two rings of two ranks
        {"name": "allgather_1MiB", "path": "coll", "coll": "allgather", "ranks": 4, "count": 524301, "dtype": "bf16", "op": "sum", "algo": "K_RING", "k": 2},
        # gradient sharding: fp32 blocks of 32 MiB between two ranks
        {"name": "reduce_scatter_32MiB", "path": "coll", "coll": "reduce_scatter", "ranks": 2, "count": 8388608, "dtype": "fp32", "op": "sum", "algo": "AUTO", "k": -1},
        # tensor-parallel output projection: the benchmark's GEMM -> reduce-scatter, all eight ranks' work
        {"name": "gemm_rs_8", "path": "gemm_rs", "ranks": 8, "m": 8192, "n": 8192, "k": 3584},
        # tensor-parallel input projection of a two-rank group on fewer tokens
        {"name": "ag_gemm_2", "path": "ag_gemm", "ranks": 2, "m": 4096, "n": 2048, "k": 4096},
    ]


# ------------------------------------------------------------------ drawing
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_model(rng, path):
    d = rng.choice([256, 512, 768, 1024])
    c = {"path": path, "layers": rng.randint(2, 24), "d_model": d, "heads": d // 64, "vocab": _log(rng, 1000, 50257), "batch": rng.randint(1, 8),
         "seq": rng.choice([128, 256, 512, 1024, rng.randint(64, 1024), rng.randint(64, 1024)])}
    return c


def _draw_coll(rng):
    coll = rng.choice(["allreduce", "allreduce", "allreduce", "allgather", "reduce_scatter", "broadcast", "reduce"])
    n = rng.choice([2, 4, 8])
    dtype = rng.choice(["fp32", "bf16", "bf16", "fp16", "int32"])
    esz = DTYPES[dtype].itemsize
    per_rank = coll in ("allgather", "reduce_scatter")
    nbytes = _log(rng, 1024, 16 << 20) if per_rank else _log(rng, 8, 64 << 20)
    if rng.random() < 0.5:                       # powers of two, as in a sweep; otherwise any length
        nbytes = 1 << (nbytes.bit_length() - 1)
    op = "sum" if coll in ("allgather", "broadcast") else rng.choice(["sum", "sum", "max"] + (["avg"] if dtype != "int32" else []))
    auto = n == 2 or coll in ("broadcast", "reduce") or nbytes <= (64 << 10)       # nothing AUTO would send through the switch
    algo = rng.choice(["RING", "K_RING", "PRD", "PRM"] + (["AUTO"] * 4 if auto else []))
    return {"path": "coll", "coll": coll, "ranks": n, "count": max(1, nbytes // esz), "dtype": dtype, "op": op, "algo": algo,
            "k": rng.choice([2, 4]) if algo in ("K_RING", "PRM") else -1}


def draw(rng):
    path = rng.choice(["train", "train", "train", "eval", "linear", "coll", "coll", "coll", "coll", "coll", "gemm_rs", "ag_gemm"])
    if path in ("train", "eval"):
        return _draw_model(rng, path)
    if path == "coll":
        return _draw_coll(rng)
    if path == "linear":
        gelu = rng.random() < 0.5
        return {"path": "linear", "m": 128 * _log(rng, 1, 64), "n": 128 * _log(rng, 2, 64), "k": 64 * _log(rng, 4, 64), "bias": gelu or rng.random() < 0.5, "gelu": gelu}
    n = rng.choice([2, 4, 8])
    return {"path": path, "ranks": n, "m": 128 * n * max(1, _log(rng, 4, 64) // n), "n": 256 * _log(rng, 1, 32), "k": 64 * _log(rng, 4, 64)}


# ------------------------------------------------------------------ preparation
_group = {}          # the communicator that the program keeps: the last one used


def _communicator(ranks, tp_bytes=0):
    key = (ranks, tp_bytes)
    if key not in _group:
        _group.clear()
        _group[key] = LoopbackGroup(ranks, config=make_config(tp_bytes=tp_bytes))
    return _group[key]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, *shape, std=1.0):
    return torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=gen)


def _tokens(c, seed):
    # token ids uniform over the vocabulary, in pinned host memory, as a loader hands them over
    tok = torch.randint(0, c["vocab"], (c["batch"], c["seq"] + 1), generator=torch.Generator().manual_seed(seed), dtype=torch.int64)
    return tok[:, :-1].contiguous().pin_memory(), tok[:, 1:].contiguous().pin_memory()


def _config(c):
    return GPT2Config(vocab_size=c["vocab"], seq_len=c["seq"], n_layer=c["layers"], n_head=c["heads"], d_model=c["d_model"])


def prepare(case, seed):
    c, path = case, case["path"]
    if path == "train":
        idx, tgt = _tokens(c, seed)
        return {"path": path, "trainer": DataParallelTrainer(_config(c), seed=seed), "idx": idx, "tgt": tgt}
    if path == "eval":
        idx, tgt = _tokens(c, seed)
        return {"path": path, "model": GPT2(_config(c), seed=seed), "idx": idx.cuda(), "tgt": tgt.cuda()}
    gen = _gen(seed)
    if path == "linear":
        s = {"path": path, "x": _normal(gen, c["m"], c["k"]), "w": _normal(gen, c["n"], c["k"], std=0.02), "bias": None, "pre": None, "gelu": c["gelu"],
             "out": torch.empty(c["m"], c["n"], dtype=torch.bfloat16, device="cuda")}
        if c["bias"]:
            s["bias"] = _normal(gen, c["n"], std=0.02)
        if c["gelu"]:
            s["pre"] = torch.empty_like(s["out"])
        return s
    n = c["ranks"]
    if path in ("gemm_rs", "ag_gemm"):
        group = _communicator(n, tp.workspace_bytes(path, n, c["m"], c["n"], c["k"]))
        rows = c["m"] if path == "gemm_rs" else c["m"] // n
        out = (c["m"] // n, c["n"]) if path == "gemm_rs" else (c["m"], c["n"])
        return {"path": path, "group": group, "a": [_normal(gen, rows, c["k"]) for _ in range(n)], "b": [_normal(gen, c["n"], c["k"], std=0.02) for _ in range(n)],
                "out": [torch.empty(out, dtype=torch.bfloat16, device="cuda") for _ in range(n)]}
    dt, count, coll = DTYPES[c["dtype"]], c["count"], c["coll"]
    n_in = count * n if coll == "reduce_scatter" else count
    n_out = count * n if coll == "allgather" else count

    def values():
        if dt == torch.int32:
            return torch.randint(-1000, 1001, (n_in,), generator=gen, dtype=dt, device="cuda")
        return torch.empty(n_in, dtype=dt, device="cuda").uniform_(-1.0, 1.0, generator=gen)

    return {"path": path, "group": _communicator(n), "send": [values() for _ in range(n)], "recv": [torch.zeros(n_out, dtype=dt, device="cuda") for _ in range(n)],
            "count": count, "coll": coll, "op": c["op"], "algo": c["algo"], "k": c["k"]}


# ------------------------------------------------------------------ one pass
def run(state):
    s, path = state, state["path"]
    if path == "train":
        loss = s["trainer"].step(s["idx"], s["tgt"])
        m = s["trainer"].model
        return {"loss": loss, "grad": m.flat_g, "param": m.flat_p, "master": m.master, "m": m.m, "v": m.v}
    if path == "eval":
        return s["model"].loss(s["idx"], s["tgt"])
    if path == "linear":
        gemm_sm100.gemm_nt(s["x"], s["w"], s["out"], bias=s["bias"], gelu=s["gelu"], pre=s["pre"])
        return [s["out"]] if s["pre"] is None else [s["out"], s["pre"]]
    if path == "gemm_rs":
        tp.gemm_rs_group(s["group"], s["a"], s["b"], s["out"])
        return s["out"]
    if path == "ag_gemm":
        tp.ag_gemm_group(s["group"], s["a"], s["b"], s["out"])
        return s["out"]
    s["group"].run(s["coll"], s["send"], s["recv"], s["count"], op=s["op"], root=0, algo=s["algo"], k=s["k"])
    return s["recv"]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    c, path = case, case["path"]
    if path in ("train", "eval"):
        T, C, L, V = c["batch"] * c["seq"], c["d_model"], c["layers"], c["vocab"]
        params = L * (12 * C * C + 13 * C) + 2 * C + (c["seq"] + (V + 127) // 128 * 128) * C
        forward = 2.0 * T * (12 * L * C * C + C * V) + 2.0 * L * T * c["seq"] * C        # products, and attention under the causal mask
        if path == "eval":
            return {"bytes": 2 * params + 16 * T, "flops": forward}
        # master weights and both moments read and written in fp32, parameters read and written, gradients written in bf16
        return {"bytes": params * (3 * 8 + 4 + 2) + 16 * T, "flops": 3 * forward}
    if path == "linear":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2 * (m * k + n * k + m * n * (2 if c["gelu"] else 1)), "flops": 2.0 * m * n * k}
    r = c["ranks"]
    if path == "gemm_rs":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2 * (r * (m * k + n * k) + m * n), "flops": 2.0 * r * m * n * k}
    if path == "ag_gemm":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2 * (m * k + r * (n * k + m * n)), "flops": 2.0 * r * m * n * k}
    one = c["count"] * DTYPES[c["dtype"]].itemsize
    adds = float(c["count"] * (r - 1))
    return {"allreduce": {"bytes": 2 * r * one, "flops": adds}, "allgather": {"bytes": (r + r * r) * one, "flops": 0},
            "reduce_scatter": {"bytes": (r * r + r) * one, "flops": r * adds}, "broadcast": {"bytes": (1 + r) * one, "flops": 0},
            "reduce": {"bytes": (r + 1) * one, "flops": adds}}[c["coll"]]


def tolerance(case):
    if case["path"] == "train":
        # bf16 products and activations through every layer and back; a first AdamW step is lr * sign(gradient), so an element whose
        # gradient is rounding noise may move the other way by 2 lr; second moments carry twice the gradients' error.  Two back ends of
        # the products differ by 0.75 % in the gradients of a second step, and by 0.8 of their root mean square at the worst element
        return {"rel": 2e-2, "max": 0.95}
    if case["path"] == "eval":
        return {"rel": 1e-3}
    if case["path"] in ("linear", "gemm_rs", "ag_gemm"):
        return {"rel": 1e-2}
    if case["coll"] in ("allgather", "broadcast") or case["op"] == "max" or case["dtype"] == "int32":
        return "exact"
    return {"rel": {"fp32": 1e-5, "fp16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
