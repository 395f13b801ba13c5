"""sm_100a engine against the PyTorch oracle path of the same model (fp32 weights, fp32 math)."""

import pytest
import torch

pytestmark = pytest.mark.gpu

CFG = dict(num_layers=2, num_heads=4, num_kv_heads=2, emb_dim=512, head_dim=128, vocab_size=4096, ffn_dim=1024)


def relerr(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


def _pair(cfg=CFG, seed=0):
    from torchure_b200.models import Qwen3

    torch.manual_seed(seed)
    fast = Qwen3(**cfg).cuda()
    fast.init_weights()
    # a livelier test than init: non-unit norm gains
    with torch.no_grad():
        for n, p in fast.named_parameters():
            if p.dim() == 1:
                p.add_(torch.randn_like(p) * 0.1)
    slow = Qwen3(**cfg, impl="torch").cuda()
    slow.load_state_dict(fast.state_dict())
    return fast, slow


@pytest.mark.parametrize("fused_ce", [True, False])
def test_forward_backward_matches_oracle(fused_ce):
    from torchure_b200 import ops
    from torchure_b200.objectives import ARObjective
    from torchure_b200.ops import kernels

    fast, slow = _pair()
    ids = torch.randint(0, CFG["vocab_size"], (2, 256), device="cuda")
    batch = {"input_ids": ids, "labels": ids}
    obj = ARObjective(fused_linear_ce=fused_ce, ce_chunk_size=200)
    before = ops.launches()
    loss = obj.compute_loss(fast, batch)
    loss.backward()
    assert ops.launches() - before > 50, "the sm_100a path must be the one that ran"
    ops.force_fallback(True)
    try:
        ref = ARObjective(fused_linear_ce=False).compute_loss(slow, batch)
        ref.backward()
    finally:
        ops.force_fallback(False)
    kernels.check_error()
    assert abs(loss.item() - ref.item()) < 2e-3 * max(1.0, abs(ref.item())), (loss.item(), ref.item())
    for (n, p), (_, q) in zip(fast.named_parameters(), slow.named_parameters()):
        assert p.grad is not None, n
        assert p.grad.dtype == torch.float32 and p.grad.shape == p.shape
        assert relerr(p.grad, q.grad) < 3e-2, (n, relerr(p.grad, q.grad))


def test_hidden_matches_oracle():
    fast, slow = _pair(seed=1)
    ids = torch.randint(0, CFG["vocab_size"], (2, 128), device="cuda")
    with torch.no_grad():
        h = fast(ids, return_final_hidden=True)
        r = slow(ids, return_final_hidden=True)
        assert h.dtype == torch.bfloat16 and h.shape == r.shape
        assert relerr(h, r) < 1e-2
        assert relerr(fast(ids), slow(ids)) < 1e-2


def test_shadow_refresh_after_load_state_dict():
    fast, slow = _pair(seed=2)
    ids = torch.randint(0, CFG["vocab_size"], (1, 128), device="cuda")
    with torch.no_grad():
        a = fast(ids, return_final_hidden=True).clone()
        sd = {k: v * 1.5 if v.dim() == 2 else v for k, v in fast.state_dict().items()}
        fast.load_state_dict(sd)
        slow.load_state_dict(sd)
        b = fast(ids, return_final_hidden=True)
        assert relerr(b, slow(ids, return_final_hidden=True)) < 2e-2
        assert relerr(a, b) > 1e-2


def test_training_steps_track_oracle():
    """3 fused AdamW steps with clipping; shadows are rewritten by the optimizer kernel."""
    from torchure_b200 import ops
    from torchure_b200.core.grad_helper import clip_grad_norm
    from torchure_b200.objectives import ARObjective
    from torchure_b200.optim import build_optimizer

    fast, slow = _pair(seed=3)
    cfg = {"lr": 2e-4, "weight_decay": 0.1, "betas": [0.9, 0.95], "fused": True}
    of, os_ = build_optimizer(fast, "adamw", cfg), build_optimizer(slow, "adamw", dict(cfg, fused=False))
    for p, s in fast.engine().shadow_pairs():
        of.attach_shadow(p, s)
    obj = ARObjective(fused_linear_ce=True, ce_chunk_size=256)

    class M1:
        def size(self, d): return 1
        def coordinate(self, d): return 0
        def get_group(self, d): return None

    losses = []
    for step in range(3):
        ids = torch.randint(0, CFG["vocab_size"], (2, 256), device="cuda", generator=torch.Generator("cuda").manual_seed(step))
        batch = {"input_ids": ids, "labels": ids}
        lf = obj.compute_loss(fast, batch)
        lf.backward()
        clip_grad_norm(list(fast.parameters()), M1(), 1.0)
        of.step(); of.zero_grad()
        ops.force_fallback(True)
        try:
            ls = obj.compute_loss(slow, batch)
            ls.backward()
            clip_grad_norm(list(slow.parameters()), M1(), 1.0)
            os_.step(); os_.zero_grad()
        finally:
            ops.force_fallback(False)
        losses.append((lf.item(), ls.item()))
    for a, b in losses:
        assert abs(a - b) < 5e-3 * max(1.0, abs(b)), losses
    for (n, p), (_, q) in zip(fast.named_parameters(), slow.named_parameters()):
        assert relerr(p, q) < 1e-2, (n, relerr(p, q))


@pytest.mark.parametrize("shape", [(2, 128, 64, 1000, 64), (2, 256, 128, 5000, 512), (2, 1024, 1024, 151936, 1024)])
def test_fused_linear_ce_sm100(shape):
    """loss / dH / dW against hidden @ W^T -> F.cross_entropy in fp32 (tolerances of the reference's own test)."""
    from torchure_b200.loss import fused_linear_cross_entropy

    B, S, D, V, chunk = shape
    torch.manual_seed(0)
    h = torch.randn(B, S, D, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(V, D, device="cuda") * 0.02).requires_grad_()
    y = torch.randint(0, V, (B, S), device="cuda")
    y[torch.rand(B, S, device="cuda") < 0.05] = -100
    loss = fused_linear_cross_entropy(h, w, y, -100, chunk)
    loss.backward()
    h2 = h.detach().float().requires_grad_()
    w2 = w.detach().clone().requires_grad_()
    ref = torch.nn.functional.cross_entropy((h2 @ w2.t()).view(-1, V), y.view(-1), ignore_index=-100)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 2e-3 * max(1.0, ref.item())
    assert relerr(h.grad, h2.grad) < 3e-2
    assert relerr(w.grad, w2.grad) < 3e-2


def test_llama3_runs_on_the_engine_and_matches_oracle():
    """The Llama-3 variant (no QK-norm, theta 5e5, eps 1e-5) on the same kernels, at a head_dim they cover."""
    from torchure_b200 import ops
    from torchure_b200.models import Llama3
    from torchure_b200.objectives import ARObjective
    from torchure_b200.ops import kernels

    cfg = dict(num_layers=2, num_heads=4, num_kv_heads=2, emb_dim=512, vocab_size=4096, ffn_dim=1024)   # head_dim 128
    torch.manual_seed(5)
    fast = Llama3(**cfg).cuda()
    fast.init_weights()
    slow = Llama3(**cfg, impl="torch").cuda()
    slow.load_state_dict(fast.state_dict())
    ids = torch.randint(0, cfg["vocab_size"], (2, 256), device="cuda")
    batch = {"input_ids": ids, "labels": ids}
    before = ops.launches()
    loss = ARObjective(fused_linear_ce=True, ce_chunk_size=256).compute_loss(fast, batch)
    loss.backward()
    assert ops.launches() - before > 40
    ops.force_fallback(True)
    try:
        ref = ARObjective(fused_linear_ce=False).compute_loss(slow, batch)
        ref.backward()
    finally:
        ops.force_fallback(False)
    kernels.check_error()
    assert abs(loss.item() - ref.item()) < 2e-3 * max(1.0, abs(ref.item()))
    for (n, p), (_, q) in zip(fast.named_parameters(), slow.named_parameters()):
        assert relerr(p.grad, q.grad) < 3e-2, (n, relerr(p.grad, q.grad))


def test_uncovered_shapes_are_loud():
    """A sequence length the attention kernels do not cover raises; a head_dim they do not cover runs the PyTorch
    path with a warning: never a silent library kernel on the hot path."""
    from torchure_b200.models import Qwen3

    m = Qwen3(**CFG).cuda()
    m.init_weights()
    with pytest.raises(RuntimeError, match="multiples of 128"):
        m(torch.randint(0, CFG["vocab_size"], (1, 100), device="cuda"))
    small = Qwen3(num_layers=1, num_heads=4, num_kv_heads=2, emb_dim=256, head_dim=64, vocab_size=512, ffn_dim=512).cuda()
    small.init_weights()
    with pytest.warns(UserWarning, match="PyTorch path"):
        out = small(torch.randint(0, 512, (1, 100), device="cuda"))
    assert out.shape == (1, 100, 512)


def test_strided_token_ids():
    """Tokens that are a strided view, one sequence (whose flat form is a view as well) and two: loss and table gradient of
    the copied tokens."""
    from torchure_b200.objectives import ARObjective

    fast, _ = _pair()
    obj = ARObjective(fused_linear_ce=True, ce_chunk_size=200)
    for B in (1, 2):
        wide = torch.randint(0, CFG["vocab_size"], (B, 256), device="cuda")
        got = []
        for ids in (wide[:, ::2], wide[:, ::2].contiguous()):
            fast.zero_grad()
            loss = obj.compute_loss(fast, {"input_ids": ids, "labels": ids})
            loss.backward()
            got.append((loss.item(), fast.token_emb.weight.grad.clone()))
        assert got[0][0] == got[1][0]
        assert relerr(got[0][1], got[1][1]) < 1e-2      # the order of the fp32 dQ additions is open


def test_blocks_and_norms_exchanged_after_the_first_pass():
    """A model whose engine has run: a dropped block and an exchanged norm are those of the next pass."""
    from torchure_b200.models.qwen3 import RMSNorm

    fast, slow = _pair()
    ids = torch.randint(0, CFG["vocab_size"], (1, 128), device="cuda")
    with torch.no_grad():
        assert relerr(fast(ids), slow(ids)) < 2e-2
        for model in (fast, slow):
            model.blocks = model.blocks[:1]
            model.blocks[0].norm1 = RMSNorm(CFG["emb_dim"]).cuda()
            model.blocks[0].norm1.weight.mul_(torch.linspace(-2, 2, CFG["emb_dim"], device="cuda"))
        assert relerr(fast(ids), slow(ids)) < 2e-2


@pytest.mark.parametrize("B,S,qk_norm", [(1, 128, True), (3, 384, False), (2, 1152, True)])
def test_native_block_calls_equal_the_wrappers(monkeypatch, B, S, qk_norm):
    """The block's native forward and backward calls against the same kernels launched one wrapper at a time (what a
    tensor-parallel axis does, here one whose sums are the terms), on both sides of the size up to which launches overlap.
    The forward repeats bit for bit; gradients differ by the order of the fp32 dQ additions, which can flip single bf16
    roundings behind them (2^-9 each).  Neither leaves an element of an output unwritten."""
    from types import SimpleNamespace

    from torchure_b200 import ops
    from torchure_b200.models import build_model
    from torchure_b200.ops import debug, kernels

    native = []
    for name in ("block_forward", "block_backward_mlp", "block_backward_attn"):
        def call(*args, _f=getattr(ops.ext(), name), _name=name):
            native.append(_name)
            return _f(*args)
        monkeypatch.setattr(ops.ext(), name, call)

    torch.manual_seed(0)
    with torch.device("cuda"):
        model = build_model("qwen3_dense" if qk_norm else "llama3_2",
                            dict(num_layers=3, num_heads=4, num_kv_heads=2, emb_dim=640, head_dim=128, vocab_size=1000,
                                 ffn_dim=1096))
        model.init_weights()
    ids = torch.randint(0, 1000, (B, S), device="cuda")
    g = torch.randn(B, S, 640, device="cuda").bfloat16()

    def run():
        model.zero_grad()
        h = model(ids, return_final_hidden=True)
        h.backward(g)
        return h.detach(), {n: p.grad.clone() for n, p in model.named_parameters() if p.grad is not None}

    debug.enable(True)
    try:
        model.engine().tp = SimpleNamespace(all_reduce_=lambda t: t)
        want, want_grads = run()
        assert not native and debug.verify() > 3 * 20
        model.engine().tp = None
        got, got_grads = run()
        assert len(native) == 3 * 3
        names = {n for n, _ in debug._pending}
        assert {"block_forward.qkv", "block_forward.gu", "block_forward.y", "block_backward.dgu", "block_backward.dqkv",
                "block_backward.dq_acc", "block_backward.dx0", "wgrad"} <= names
        assert debug.verify() > 3 * 20
    finally:
        debug.enable(False)
    again, _ = run()
    assert torch.equal(again, got)
    assert torch.equal(got, want) and got_grads.keys() == want_grads.keys() and len(got_grads) > 20
    for n, w in want_grads.items():
        assert ((got_grads[n] - w).norm() / w.norm()).item() < 1e-2, n
    with torch.no_grad():
        for _ in range(20):
            assert torch.equal(model(ids, return_final_hidden=True), want)
    kernels.check_error()


@pytest.mark.parametrize("B,S,layers,qk_norm", [(1, 128, 1, True), (3, 384, 4, False), (2, 1152, 3, True)])
def test_forward_without_gradients_in_one_call(monkeypatch, B, S, layers, qk_norm):
    """The pass without gradients (one native call, the blocks' buffers used again and again) gives the bits of the pass with
    them, for strided ids, an exchanged gain and on another stream; poisoned outputs keep it a block at a time."""
    from torchure_b200 import ops
    from torchure_b200.models import build_model
    from torchure_b200.ops import debug, kernels

    calls = []
    whole = ops.ext().blocks_forward
    monkeypatch.setattr(ops.ext(), "blocks_forward", lambda *a: calls.append(1) or whole(*a))
    torch.manual_seed(1)
    with torch.device("cuda"):
        model = build_model("qwen3_dense" if qk_norm else "llama3_2",
                            dict(num_layers=layers, num_heads=4, num_kv_heads=2, emb_dim=640, head_dim=128, vocab_size=1000,
                                 ffn_dim=1096))
        model.init_weights()
    ids = torch.randint(0, 1000, (S, B), device="cuda").t()
    want = model(ids, return_final_hidden=True).detach()
    assert not calls
    with torch.no_grad():
        for _ in range(20):
            assert torch.equal(model(ids, return_final_hidden=True), want)
        assert len(calls) == 20
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            other = model(ids, return_final_hidden=True)
        side.synchronize()
        assert torch.equal(other, want)
        model.blocks[-1].norm2.weight = torch.nn.Parameter(model.blocks[-1].norm2.weight * 2)
    want = model(ids, return_final_hidden=True).detach()
    with torch.no_grad():
        assert torch.equal(model(ids, return_final_hidden=True), want)
        n = len(calls)
        debug.enable(True)
        try:
            assert torch.equal(model(ids, return_final_hidden=True), want) and debug.verify() > 10
        finally:
            debug.enable(False)
        assert len(calls) == n
    kernels.check_error()


@pytest.mark.parametrize("widths", [(1096, 512, 1096), (512, 2048, 512), (640, 640, 1280)])
@pytest.mark.parametrize("S", [128, 512])
def test_forward_without_gradients_blocks_of_other_widths(widths, S):
    """Blocks whose MLPs differ in width (some were pruned): the pass without gradients gives the bits of the pass with them."""
    from torchure_b200.models import Qwen3
    from torchure_b200.models.qwen3 import SwiGLU
    from torchure_b200.ops import kernels

    torch.manual_seed(1)
    model = Qwen3(num_layers=3, num_heads=4, num_kv_heads=2, emb_dim=640, head_dim=128, vocab_size=1000, ffn_dim=1096)
    for block, width in zip(model.blocks, widths):
        block.ffn = SwiGLU(640, width)
    model = model.cuda()
    model.init_weights()
    ids = torch.randint(0, 1000, (2, S), device="cuda")
    want = model(ids, return_final_hidden=True).detach()
    with torch.no_grad():
        assert torch.equal(model(ids, return_final_hidden=True), want)
    kernels.check_error()


@pytest.mark.parametrize("world,comm_sms", [(1, 16), (2, 16), (8, 40)])
def test_qknorm_backward_is_told_of_communication_ctas(monkeypatch, world, comm_sms):
    """With a gradient sink whose collectives run under the backward pass the QK-norm kernel gets the number of SMs they are
    on, and gives the same gradients."""
    from torchure_b200.ops import kernels

    class Sink:
        def __init__(self, params):
            self.world, self.comm_sms = world, comm_sms
            flat = torch.zeros(sum(p.numel() for p in params), device="cuda")
            self.grads = {p: v.view_as(p) for p, v in zip(params, flat.split([p.numel() for p in params]))}

        def grad_dest(self, p):
            return self.grads[p], False

        def grad_written(self, p):
            pass

    told = []
    plain = kernels.qknorm_rope_bwd_
    monkeypatch.setattr(kernels, "qknorm_rope_bwd_", lambda *a, **k: told.append(k["shared_sms"]) or plain(*a, **k))
    model, _ = _pair(seed=5)
    ids = torch.randint(0, CFG["vocab_size"], (2, 256), device="cuda")
    g = torch.randn(2, 256, CFG["emb_dim"], device="cuda").bfloat16()
    model(ids, return_final_hidden=True).backward(g)
    want = {n: p.grad for n, p in model.named_parameters()}
    model.zero_grad(set_to_none=True)
    sink = Sink(list(model.parameters()))
    model.set_grad_sink(sink)
    model(ids, return_final_hidden=True).backward(g)
    kernels.check_error()
    assert told == ([] if world == 1 else [comm_sms] * CFG["num_layers"])      # one rank: native calls
    for n, p in model.named_parameters():
        if p.dim() == 1 or "proj" in n:
            # gradients behind attention's fp32 additions, whose order differs from run to run
            assert relerr(sink.grads[p], want[n]) < 1e-2, n
