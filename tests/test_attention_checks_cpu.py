"""What the attention kernels refuse (no GPU needed: nothing is launched)."""
import pytest
import torch


def _operands(batch=2, S=100, heads=2, dtype=torch.bfloat16):
    rows, Cc, pad = batch * S, heads * 64, (S + 127) // 128 * 128
    f = torch.zeros
    return {"qkv": f(rows, 3 * Cc, dtype=dtype), "out": f(rows, Cc, dtype=dtype), "dout": f(rows, Cc, dtype=dtype), "lse": f(batch * heads, S), "scratch": f(2 * batch * heads * pad),
            "dqkv": f(rows, 3 * Cc, dtype=dtype), "part": f(batch * pad // 128, 3 * Cc), "batch": batch}


@pytest.mark.parametrize("change,why", [
    ({"qkv": torch.zeros(200, 256, dtype=torch.bfloat16)}, "wanted"),                # narrower than q, k and v
    ({"qkv": torch.zeros(199, 384, dtype=torch.bfloat16)}, "wanted"),                # a row short
    ({"qkv": torch.zeros(200, 384)}, "bf16"),
    ({"qkv": torch.zeros(200, 768, dtype=torch.bfloat16)[:, ::2]}, "contiguous"),
    ({"out": torch.zeros(200, 96, dtype=torch.bfloat16)}, "heads"),                  # one head and a half
    ({"batch": 3}, "positions"), ({"batch": 0}, "positions"),
    ({"lse": torch.zeros(4 * 100 - 1)}, "floats"), ({"lse": torch.zeros(4, 100, dtype=torch.float64)}, "floats"),
    ({}, "CUDA"),
])
@pytest.mark.parametrize("backward", [False, True])
def test_operands_that_do_not_fit(change, why, backward):
    from piccl_b200 import ops
    o = {**_operands(), **change}
    with pytest.raises(ValueError, match=why):
        if backward:
            ops.attention_bwd(**o)
        else:
            ops.attention_fwd(o["qkv"], o["out"], o["lse"], o["batch"])


@pytest.mark.parametrize("change", [{"dout": torch.zeros(200, 64, dtype=torch.bfloat16)}, {"dqkv": torch.zeros(100, 384, dtype=torch.bfloat16)}, {"scratch": torch.zeros(2 * 4 * 100)},
                                    {"part": torch.zeros(1, 384)}, {"lse": None}, {"scratch": None}, {"part": None}])
def test_operands_of_the_backward_pass_that_do_not_fit(change):
    from piccl_b200 import ops
    with pytest.raises(ValueError, match="wanted|takes"):
        ops.attention_bwd(**{**_operands(), **change})


def test_null_and_misaligned_addresses_are_refused():
    """The C entries themselves; no address is touched before it is refused."""
    import ctypes as C
    from piccl_b200 import _native as N
    lib = N.ops_lib()
    good = 4096
    p = C.c_void_p
    for i, bad in [(i, b) for i in range(7) for b in (0, good + 2)]:
        a = [good] * 7
        a[i] = bad
        assert lib.piccl_ops_attn_bwd(*[p(x) for x in a], 1, 64, 1, p(0)) == -2, i
    for a in ((0, good, 0), (good, 0, 0), (good + 8, good, 0), (good, good + 2, 0), (good, good, good + 2)):
        assert lib.piccl_ops_attn_fwd(*[p(x) for x in a], 1, 64, 1, p(0)) == -2, a
