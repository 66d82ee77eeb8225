"""The framework's GPT-2 (own kernels, hand-scheduled backward) against a conventional
PyTorch module with the same weights."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pair(n_head=4):
    from benchmarks.torch_gpt2 import TorchGPT2
    from piccl_b200.models.gpt2 import GPT2, GPT2Config
    cfg = GPT2Config.tiny()
    cfg.n_head = n_head
    mine = GPT2(cfg, seed=3)
    ref = TorchGPT2(cfg.vocab_size, cfg.seq_len, cfg.n_layer, cfg.n_head, cfg.d_model).cuda().float()
    sd = {k: v.float() for k, v in mine.state_dict().items()}
    missing = ref.load_state_dict(sd, strict=True)
    assert not missing.missing_keys
    return cfg, mine, ref


def test_loss_and_gradients_match_pytorch():
    cfg, mine, ref = _pair()
    g = torch.Generator().manual_seed(0)
    tok = torch.randint(0, cfg.vocab_size, (4, cfg.seq_len + 1), generator=g).cuda()
    a, b = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
    loss = mine.forward_backward(a, b)
    rl = ref(a, b)
    rl.backward()
    assert abs(float(loss) - float(rl)) < 3e-2, (float(loss), float(rl))
    checks = {"lnf_g": ref.ln_f.weight.grad, "h1.w_fc": ref.h[1].mlp["c_fc"].weight.grad, "h0.w_qkv": ref.h[0].attn["c_attn"].weight.grad,
              "h0.b_qkv": ref.h[0].attn["c_attn"].bias.grad, "h1.ln2_b": ref.h[1].ln_2.bias.grad, "wpe": ref.wpe.weight.grad,
              "h0.w_proj": ref.h[0].mlp["c_proj"].weight.grad, "h1.w_o": ref.h[1].attn["c_proj"].weight.grad}
    for name, rg in checks.items():
        mg = mine.g[name].float()
        rel = (mg - rg).norm() / (rg.norm() + 1e-12)
        assert rel < 5e-2, f"{name}: relative gradient error {float(rel):.4f}"
    mg = mine.g["wte"][:cfg.vocab_size].float()
    rel = (mg - ref.wte.weight.grad).norm() / ref.wte.weight.grad.norm()
    assert rel < 5e-2, f"wte: {float(rel):.4f}"


def test_training_reduces_loss_and_ready_ranges_are_monotonic():
    from piccl_b200.models.gpt2 import GPT2, GPT2Config
    cfg = GPT2Config.tiny()
    m = GPT2(cfg, seed=1)
    g = torch.Generator().manual_seed(0)
    tok = torch.randint(0, cfg.vocab_size, (4, cfg.seq_len + 1), generator=g).cuda()
    a, b = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
    ends = []
    losses = []
    for _ in range(8):
        ends.clear()
        losses.append(float(m.forward_backward(a, b, on_grads_ready=ends.append)))
        m.optimizer_step(lr=1e-3)
    assert ends == sorted(ends) and ends[-1] == m.n_params
    assert losses[-1] < losses[0] - 0.5, losses


@pytest.mark.parametrize("layers,d_model,shapes", [
    (1, 256, [(4, 128)]),
    (5, 256, [(3, 77), (4, 128), (3, 77)]),       # layers take the gradient buffers in turn; a larger batch moves the activations; back to the first one
    (3, 512, [(8, 512)]),                         # products of both back ends
])
def test_replayed_steps_equal_issued_ones(layers, d_model, shapes):
    from piccl_b200.models.gpt2 import GPT2, GPT2Config
    cfg = GPT2Config(vocab_size=1000, seq_len=512, n_layer=layers, n_head=d_model // 64, d_model=d_model)
    replayed, issued = GPT2(cfg, seed=2), GPT2(cfg, seed=2)
    gen = torch.Generator().manual_seed(5)
    for B, S in shapes:
        a, b = torch.empty(B, S, dtype=torch.int64, device="cuda"), torch.empty(B, S, dtype=torch.int64, device="cuda")
        for step in range(6):
            tok = torch.randint(0, cfg.vocab_size, (B, S + 1), generator=gen)
            a.copy_(tok[:, :-1]); b.copy_(tok[:, 1:])
            replayed.flat_g.fill_(float("nan")); issued.flat_g.fill_(float("nan"))
            got = replayed.forward_backward(a, b)
            want = issued.forward_backward(a, b, on_grads_ready=lambda end: None)       # reports gradients: always issued call by call
            assert abs(float(got) - float(want)) <= 1e-5 * float(want)
            for m in (replayed, issued):              # every element is written, also for positions that no token had
                assert not torch.isnan(m.flat_g).any() and not m.g["wpe"][S:].any()
            # every gradient by itself: those of gains and biases are a small part of the whole, and a wait that is missing between the streams may spoil
            # one of them alone.  The sums are the same up to the order of a few (attention and embedding by atomics, products of another back end): at
            # worst another rounding to bf16 (2^-8) of an element in each of the two halves of a layer
            for name, w in issued.g.items():
                d = (replayed.g[name].double() - w.double()).norm()
                assert float(d) <= 2 ** -7 * float(w.double().norm()), (step, name)
            want = issued._issue(a.reshape(-1), b.reshape(-1), B, S, True, 0)
            assert abs(float(replayed.loss(a, b)) - float(want)) <= 1e-5 * float(want)
            replayed.optimizer_step(lr=1e-4 * (step + 1))
            issued.flat_p.copy_(replayed.flat_p)
    assert replayed._graphs, "nothing was captured"


def test_whole_step_graph_outlives_a_larger_evaluation():
    """A step captured with its optimizer keeps the addresses of the activations; an evaluation that outgrows them must leave those to the graph."""
    from piccl_b200.models.gpt2 import GPT2Config
    from piccl_b200.train import DataParallelTrainer
    cfg = GPT2Config.tiny()
    graphed, eager = (DataParallelTrainer(cfg, seed=4, use_graph=g) for g in (True, False))
    gen = torch.Generator().manual_seed(6)

    def batch(B):
        tok = torch.randint(0, cfg.vocab_size, (B, cfg.seq_len + 1), generator=gen)
        return tok[:, :-1].contiguous().pin_memory(), tok[:, 1:].contiguous().pin_memory()

    for step in range(8):
        x, y = batch(4)
        a, b = graphed.step(x, y), eager.step(x, y)
        assert abs(a - b) <= 2e-3 * b, step                      # the two launch modes may take other kernels for a product: bf16 roundings differ
        if step == 4:
            assert graphed._graph is not None and graphed.replayed_steps() == 3
            big = [t.cuda() for t in batch(64)]
            assert abs(float(graphed.model.loss(*big)) - float(eager.model.loss(*big))) <= 2e-3 * b
            torch.cuda.synchronize()
            others = [torch.full((3 << 20,), 77, dtype=torch.uint8, device="cuda") for _ in range(32)]      # what the allocator has free among its large blocks
    torch.cuda.synchronize()
    assert all(bool((t == 77).all()) for t in others)


def test_first_step_inside_a_callers_capture():
    """A model whose very first step is captured by its user: steps issued before the first replay, and replays after them, start from zeroed workspaces."""
    from piccl_b200.models.gpt2 import GPT2, GPT2Config
    cfg = GPT2Config(vocab_size=1000, seq_len=128, n_layer=2, n_head=4, d_model=256)
    tok = torch.randint(0, cfg.vocab_size, (8, cfg.seq_len + 1), generator=torch.Generator().manual_seed(8))
    x, y = tok[:, :-1].contiguous().cuda(), tok[:, 1:].contiguous().cuda()
    known = GPT2(cfg, seed=5)
    want = known.forward_backward(x, y)                            # also sets the libraries up
    fill = [torch.full((64 << 20,), 0x55, dtype=torch.uint8, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    del fill                                                       # what the allocator hands out now is not zero
    model, graph = GPT2(cfg, seed=5), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        loss = model.forward_backward(x, y)
    for issued in (True, False, False, True):
        model.flat_g.fill_(float("nan"))
        if issued:
            loss2 = model.forward_backward(x, y)
        else:
            graph.replay()
            loss2 = loss
        assert abs(float(loss2) - float(want)) <= 1e-5 * float(want)
        for name, g in known.g.items():                            # the same kernels; sums by atomics may round differently
            d = (model.g[name].double() - g.double()).norm()
            assert float(d) <= 2 ** -7 * float(g.double().norm()), (issued, name)


@pytest.mark.parametrize("n_head,seq", [(64, 128), (64, 77), (128, 50), (32, 33)])
def test_narrow_heads(n_head, seq):
    """Heads of 4 and 2 columns, whose gradients no kernel reads in 16-byte words, and of 8, the narrowest that it does; issued and replayed.  bf16 products and
    activations: gradients within 2 % of fp32."""
    cfg, mine, ref = _pair(n_head)
    tok = torch.randint(0, cfg.vocab_size, (3, seq + 1), generator=torch.Generator().manual_seed(0)).cuda()
    a, b = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
    rl = ref(a, b)
    rl.backward()
    for step in range(4):
        mine.flat_g.fill_(float("nan"))
        loss = mine.forward_backward(a, b)
        assert abs(float(loss) - rl.item()) < 1e-2
        for l in range(cfg.n_layer):
            for name, rg in ((f"h{l}.w_qkv", ref.h[l].attn["c_attn"].weight.grad), (f"h{l}.b_qkv", ref.h[l].attn["c_attn"].bias.grad), (f"h{l}.w_o", ref.h[l].attn["c_proj"].weight.grad)):
                assert (mine.g[name].float() - rg).norm() <= 2e-2 * rg.norm(), (step, name)
    assert mine._graphs


def test_optimizer_beyond_the_runs_of_one_launch(monkeypatch):
    """Models with more runs of decaying and other parameters than one launch takes: a launch per run, the same update up to the rounding of a few fp32 operations."""
    from piccl_b200 import ops
    from piccl_b200.models.gpt2 import GPT2, GPT2Config
    cfg = GPT2Config(vocab_size=500, seq_len=32, n_layer=1, n_head=4, d_model=256)
    one, many = GPT2(cfg, seed=1), GPT2(cfg, seed=1)
    for step in range(3):
        g = torch.randn(one.n_params, generator=torch.Generator(device="cuda").manual_seed(step), device="cuda").bfloat16()
        for m in (one, many):
            m.flat_g.copy_(g)
        one.optimizer_step(lr=1e-2)
        with monkeypatch.context() as mp:
            mp.setattr(ops, "MAX_ADAMW_RUNS", 2)
            assert len(many.groups) > 2
            many.optimizer_step(lr=1e-2)
        assert int(one.step_dev) == int(many.step_dev) == step + 1
        for a, b in ((one.master, many.master), (one.m, many.m), (one.v, many.v)):
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-7)
    # and the native call refuses what does not fit
    ends = torch.arange(1, ops.MAX_ADAMW_RUNS + 2, dtype=torch.int32, device="cuda")
    p, f = torch.zeros(8 * ends.numel(), device="cuda", dtype=torch.bfloat16), [torch.zeros(8 * ends.numel(), device="cuda") for _ in range(3)]
    with pytest.raises(RuntimeError):
        ops.adamw_runs(p, *f, p, ends, 0, 1e-3, 0.9, 0.95, 1e-8, 0.1, one.step_dev, one._ticket)


def test_a_captured_step_is_not_replayed_under_other_library_settings():
    """Attention back ends (a context manager) and deterministic algorithms are looked up in each call; a graph holds what was chosen at its capture."""
    from torch.nn.attention import SDPBackend, sdpa_kernel
    from piccl_b200.models.gpt2 import GPT2, GPT2Config
    cfg = GPT2Config.tiny()
    m = GPT2(cfg, seed=1)
    tok = torch.randint(0, cfg.vocab_size, (2, cfg.seq_len + 1), generator=torch.Generator().manual_seed(0)).cuda()
    a, b = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
    for _ in range(4):
        want = float(m.forward_backward(a, b))
    assert m.replays == 2
    with sdpa_kernel(SDPBackend.MATH):
        assert abs(float(m.forward_backward(a, b)) - want) <= 1e-3 * want
    assert m.replays == 2
    torch.use_deterministic_algorithms(True, warn_only=True)
    try:
        assert abs(float(m.forward_backward(a, b)) - want) <= 1e-3 * want
    finally:
        torch.use_deterministic_algorithms(False)
    assert m.replays == 2
    assert float(m.forward_backward(a, b)) == want and m.replays == 3


def test_a_captured_step_is_not_replayed_under_another_order_of_back_ends():
    """The same attention back ends enabled, but another one first."""
    from torch.nn.attention import SDPBackend, sdpa_kernel
    from piccl_b200.models.gpt2 import GPT2, GPT2Config
    cfg = GPT2Config.tiny()
    m = GPT2(cfg, seed=1)
    tok = torch.randint(0, cfg.vocab_size, (2, cfg.seq_len + 1), generator=torch.Generator().manual_seed(0)).cuda()
    a, b = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
    orders = [SDPBackend.CUDNN_ATTENTION, SDPBackend.EFFICIENT_ATTENTION], [SDPBackend.EFFICIENT_ATTENTION, SDPBackend.CUDNN_ATTENTION]
    with sdpa_kernel(orders[0], set_priority=True):
        for _ in range(4):
            want = float(m.forward_backward(a, b))
        grads = m.flat_g.clone()
    assert m.replays == 2
    with sdpa_kernel(orders[1], set_priority=True):
        assert abs(float(m.forward_backward(a, b)) - want) <= 1e-3 * want
    assert m.replays == 2 and not torch.equal(m.flat_g, grads)
    with sdpa_kernel(orders[0], set_priority=True):
        assert float(m.forward_backward(a, b)) == want and m.replays == 3


def test_the_first_model_of_a_process_is_captured_at_its_third_step():
    """In a process that has not asked PyTorch for an attention back end before."""
    import subprocess
    import sys
    from pathlib import Path
    code = ("import torch\nfrom piccl_b200.models.gpt2 import GPT2, GPT2Config\nm = GPT2(GPT2Config.tiny(), seed=1)\nx = torch.zeros(2, 128, dtype=torch.int64, device='cuda')\n"
            "for _ in range(4): m.forward_backward(x, x)\nassert m.replays == 2, m.replays")
    r = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_an_interrupt_during_a_capture_leaves_the_model_usable():
    from piccl_b200.models.gpt2 import GPT2, GPT2Config
    cfg = GPT2Config.tiny()
    m = GPT2(cfg, seed=1)
    tok = torch.randint(0, cfg.vocab_size, (2, cfg.seq_len + 1), generator=torch.Generator().manual_seed(0)).cuda()
    a, b = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
    want = [float(m.forward_backward(a, b)) for _ in range(2)][-1]
    issue = m._issue

    def interrupted(*args):
        issue(*args)
        raise KeyboardInterrupt

    m._issue = interrupted
    with pytest.raises(KeyboardInterrupt):
        m.forward_backward(a, b)
    m._issue = issue
    for _ in range(3):
        assert float(m.forward_backward(a, b)) == want
    torch.cuda.synchronize()
    assert m.replays == 3


@pytest.mark.parametrize("B,S,n_head,own", [(2, 1023, 4, True), (1, 1024, 4, False), (12, 1024, 4, True), (1, 640, 4, True), (1, 768, 4, False), (3, 77, 4, True), (1, 2000, 4, False)])
def test_attention_on_both_sides_of_its_rule(B, S, n_head, own):
    """Backward attention of 64-column heads by own kernels or by cuDNN's, evaluations likewise: the gradients, the training loss and the evaluated loss against PyTorch's plain attention,
    and which of the two ran (two launches in place of one)."""
    from torch.nn.attention import SDPBackend, sdpa_kernel
    from benchmarks.torch_gpt2 import TorchGPT2
    from piccl_b200 import _native as N
    from piccl_b200.models.gpt2 import GPT2, GPT2Config
    layers, D = 3, 64 * n_head
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert bool(N.ops_lib().piccl_ops_attn_pays(1, B, S, n_head, sms)) == own
    fwd = bool(N.ops_lib().piccl_ops_attn_pays(0, B, S, n_head, sms))
    mine = GPT2(GPT2Config(vocab_size=500, seq_len=S, n_layer=layers, n_head=n_head, d_model=D), seed=7)
    ref = TorchGPT2(500, S, layers, n_head, D).cuda().float()
    ref.load_state_dict({k: v.float() for k, v in mine.state_dict().items()})
    tok = torch.randint(0, 500, (B, S + 1), generator=torch.Generator().manual_seed(S)).cuda()
    a, b = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
    with sdpa_kernel(SDPBackend.MATH):
        rl = ref(a, b)
        rl.backward()
    grads = {f"h{l}.{k}": getattr(ref.h[l].attn[v], w).grad for l in range(layers) for k, v, w in
             (("w_qkv", "c_attn", "weight"), ("b_qkv", "c_attn", "bias"), ("w_o", "c_proj", "weight"))}

    def run(evaluate):
        counts = (N.C.c_longlong * 4)()
        mine.flat_g.fill_(float("nan"))
        x, y = a.reshape(-1), b.reshape(-1)
        loss = mine._issue(x, y, B, S, evaluate, 0)
        counts[:] = mine._counts[:]
        return float(loss), counts[0]

    def agree():
        for name, want in grads.items():           # bf16 activations and gradients: 0.6 to 0.9 % from fp32 measured
            assert (mine.g[name].float() - want).norm() <= 2e-2 * want.norm(), name

    loss, launches = run(False)
    agree()
    evaluated, eval_launches = run(True)
    assert abs(loss - rl.item()) < 2e-3 and abs(evaluated - rl.item()) < 2e-3
    with sdpa_kernel(SDPBackend.MATH):             # a back end that the program asks for: nothing of its own
        other, plain = run(False)
        agree()
        other_eval, plain_eval = run(True)
    assert abs(other - loss) < 2e-3 and abs(other_eval - evaluated) < 2e-3
    assert launches - plain == layers * own and eval_launches - plain_eval == layers * fwd


@pytest.mark.parametrize("kind,name", [(0, "GEMM"), (1, "attention")])
def test_a_wait_that_ran_out_is_reported(kind, name):
    """The status word that a kernel sets when it gives up (set here from the host): the loss of a step or an evaluation is not a number, issued, replayed and in a graph of the whole step,
    the trainer raises, and once reported all is as before."""
    from piccl_b200 import _native as N, ops
    from piccl_b200.models.gpt2 import GPT2Config
    from piccl_b200.train import DataParallelTrainer
    cfg = GPT2Config.tiny()
    tok = torch.randint(0, cfg.vocab_size, (2, cfg.seq_len + 1), generator=torch.Generator().manual_seed(0))
    x, y = tok[:, :-1].contiguous().pin_memory(), tok[:, 1:].contiguous().pin_memory()
    xd, yd = x.cuda(), y.cuda()
    for use_graph in (False, True):
        t = DataParallelTrainer(cfg, seed=4, use_graph=use_graph)
        for step in range(6):
            assert t.step(x, y) > 0
            assert N.ops_lib().piccl_ops_test_set_status(kind, 11) == 0
            assert torch.isnan(t.model.loss(xd, yd)) and torch.isnan(t.model.loss(xd, yd))      # stays until it is reported
            with pytest.raises(RuntimeError, match=name):
                t.step(x, y)
            ops.raise_if_a_wait_ran_out()                  # nothing more to report
            assert t.step(x, y) > 0 and float(t.model.loss(xd, yd)) > 0
        assert t.replayed_steps() > 0
