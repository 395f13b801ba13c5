"""tcgen05 flash attention against a plain fp32 softmax(QK^T)V."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


def _inputs(B, S, Hq, Hkv, seed=0, scale=1.0):
    torch.manual_seed(seed)
    hd = 128
    qk = (torch.randn(B * S, (Hq + Hkv) * hd, device="cuda") * scale).bfloat16()
    qkv = torch.randn(B * S, (Hq + 2 * Hkv) * hd, device="cuda").bfloat16()
    return qk, qkv


def _oracle(qk, qkv, B, S, Hq, Hkv):
    from torchure_b200.ops import oracle

    hd = 128
    q = qk[:, :Hq * hd].view(B, S, Hq, hd)
    k = qk[:, Hq * hd:].view(B, S, Hkv, hd)
    v = qkv[:, (Hq + Hkv) * hd:].view(B, S, Hkv, hd)
    o, lse = oracle.attention(q, k, v)
    return o.reshape(B * S, Hq * hd), lse


@pytest.mark.parametrize("B,S,Hq,Hkv,scale", [(1, 128, 2, 1, 1.0), (2, 512, 4, 2, 1.0), (1, 1024, 8, 2, 1.0),
                                              (1, 512, 2, 1, 4.0), (2, 2048, 4, 2, 0.3), (1, 4096, 16, 8, 1.0),
                                              (1, 4096, 32, 8, 1.0)])
def test_attn_fwd(B, S, Hq, Hkv, scale):
    from torchure_b200 import ops
    from torchure_b200.ops import kernels

    qk, qkv = _inputs(B, S, Hq, Hkv, scale=scale)
    o = torch.empty(B * S, Hq * 128, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device="cuda")
    ops.ext().attn_fwd(qk, qkv, o, lse, B, S, Hq, Hkv)
    kernels.check_error()
    ro, rl = _oracle(qk, qkv, B, S, Hq, Hkv)
    assert relerr(o, ro) < 1e-2, relerr(o, ro)
    torch.testing.assert_close(lse, rl, rtol=2e-3, atol=2e-3)


def _grads_oracle(qk, qkv, d_o, B, S, Hq, Hkv):
    """fp32 reference gradients, one (batch, kv head) group at a time so the S x S scores of long sequences fit."""
    from torchure_b200.ops import oracle

    hd, r = 128, Hq // Hkv
    dq = torch.empty(B, S, Hq, hd, device="cuda")
    dk = torch.empty(B, S, Hkv, hd, device="cuda")
    dv = torch.empty(B, S, Hkv, hd, device="cuda")
    qa = qk[:, :Hq * hd].float().view(B, S, Hq, hd)
    ka = qk[:, Hq * hd:].float().view(B, S, Hkv, hd)
    va = qkv[:, (Hq + Hkv) * hd:].float().reshape(B, S, Hkv, hd)
    ga = d_o.float().view(B, S, Hq, hd)
    for b in range(B):
        for g in range(Hkv):
            q = qa[b:b + 1, :, g * r:(g + 1) * r].clone().requires_grad_()
            k = ka[b:b + 1, :, g:g + 1].clone().requires_grad_()
            v = va[b:b + 1, :, g:g + 1].clone().requires_grad_()
            o, _ = oracle.attention(q, k, v)
            o.backward(ga[b:b + 1, :, g * r:(g + 1) * r])
            dq[b, :, g * r:(g + 1) * r], dk[b, :, g], dv[b, :, g] = q.grad[0], k.grad[0, :, 0], v.grad[0, :, 0]
    return dq, dk, dv


@pytest.mark.parametrize("entry", ["attn_bwd_fused", "attn_bwd"])
@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 128, 2, 1), (1, 256, 2, 1), (2, 512, 4, 2), (1, 1024, 8, 2), (1, 384, 2, 1),
                                        (1, 4096, 16, 8), (1, 4096, 32, 8)])
def test_attn_bwd(B, S, Hq, Hkv, entry):
    """Both backward implementations (single pass, two kernels) against fp32 autograd of the dense formula, up to
    the benchmark shapes (16/8 and 32/8 heads at 4096 tokens)."""
    from torchure_b200 import ops
    from torchure_b200.ops import kernels

    hd = 128
    qk, qkv = _inputs(B, S, Hq, Hkv, seed=1)
    o = torch.empty(B * S, Hq * hd, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device="cuda")
    ops.ext().attn_fwd(qk, qkv, o, lse, B, S, Hq, Hkv)
    d_o = torch.randn(B * S, Hq * hd, device="cuda").bfloat16()
    dqkv = torch.zeros(B * S, (Hq + 2 * Hkv) * hd, dtype=torch.bfloat16, device="cuda")
    getattr(ops.ext(), entry)(d_o, qk, qkv, o, lse, dqkv, B, S, Hq, Hkv)
    kernels.check_error()
    rq, rk, rv = _grads_oracle(qk, qkv, d_o, B, S, Hq, Hkv)
    dq = dqkv[:, :Hq * hd].view(B, S, Hq, hd)
    dk = dqkv[:, Hq * hd:(Hq + Hkv) * hd].view(B, S, Hkv, hd)
    dv = dqkv[:, (Hq + Hkv) * hd:].view(B, S, Hkv, hd)
    assert relerr(dv, rv) < 1.5e-2, ("dv", relerr(dv, rv))
    assert relerr(dq, rq) < 1.5e-2, ("dq", relerr(dq, rq))
    assert relerr(dk, rk) < 1.5e-2, ("dk", relerr(dk, rk))


@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv,causal", [(2, 512, 512, 4, 2, True), (1, 256, 768, 4, 2, False),
                                                    (2, 384, 384, 8, 2, False)])
def test_flash_attention_block_pairs(B, Sq, Skv, Hq, Hkv, causal):
    """The block-pair entry points (separate q / k / v tensors, optional full visibility, Sq != Skv) through the
    differentiable ``flash_attention`` op, forward and backward, against the dense fp32 formula."""
    from torchure_b200.ops import kernels
    from torchure_b200.ops.attention import flash_attention, pair_supported

    torch.manual_seed(3)
    q = torch.randn(B, Sq, Hq, 128, device="cuda").bfloat16().requires_grad_()
    k = torch.randn(B, Skv, Hkv, 128, device="cuda").bfloat16().requires_grad_()
    v = torch.randn(B, Skv, Hkv, 128, device="cuda").bfloat16().requires_grad_()
    assert pair_supported(q, k, v)
    out = flash_attention(q, k, v, causal=causal)
    g = torch.randn_like(out)
    out.backward(g)
    kernels.check_error()
    rep = Hq // Hkv
    qf, kf, vf = (t.detach().float().transpose(1, 2).requires_grad_() for t in (q, k, v))
    s = qf @ kf.repeat_interleave(rep, 1).transpose(-1, -2) / 128 ** 0.5
    if causal:
        s = s.masked_fill(~torch.ones(Sq, Skv, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    ref = torch.softmax(s, -1) @ vf.repeat_interleave(rep, 1)
    ref.backward(g.float().transpose(1, 2))
    assert relerr(out, ref.transpose(1, 2)) < 1e-2
    for name, got, want in (("dq", q.grad, qf.grad), ("dk", k.grad, kf.grad), ("dv", v.grad, vf.grad)):
        assert relerr(got, want.transpose(1, 2)) < 1.5e-2, (name, relerr(got, want.transpose(1, 2)))


@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv,causal", [(1, 128, 128, 4, 1, True), (1, 384, 384, 2, 1, True), (1, 1024, 1024, 8, 4, True),
                                                    (2, 1024, 1024, 8, 4, True), (1, 640, 128, 4, 2, False),
                                                    (1, 128, 4096, 8, 1, False), (1, 512, 9472, 2, 1, False)])
def test_backward_with_shared_key_blocks(B, Sq, Skv, Hq, Hkv, causal):
    """Few key blocks: clusters of two and four CTAs share one, with parts of unequal length and (causal) parts without any
    iteration.  Gradients against fp64; dK and dV are summed in a fixed order, so a second run gives the same bits."""
    from torchure_b200.ops import kernels
    from torchure_b200.ops.attention import flash_attention

    torch.manual_seed(5)
    q = torch.randn(B, Sq, Hq, 128, device="cuda").bfloat16().requires_grad_()
    k, v = (torch.randn(B, Skv, Hkv, 128, device="cuda").bfloat16().requires_grad_() for _ in range(2))
    g = torch.randn_like(q)
    grads = []
    for _ in range(2):
        grads.append(torch.autograd.grad(flash_attention(q, k, v, causal=causal), (q, k, v), g))
    kernels.check_error()
    assert torch.equal(grads[0][1], grads[1][1]) and torch.equal(grads[0][2], grads[1][2])
    qf, kf, vf = (t.detach().double().transpose(1, 2).requires_grad_() for t in (q, k, v))
    s = qf @ kf.repeat_interleave(Hq // Hkv, 1).transpose(-1, -2) / 128 ** 0.5
    if causal:
        s = s.masked_fill(~torch.ones(Sq, Skv, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    (torch.softmax(s, -1) @ vf.repeat_interleave(Hq // Hkv, 1)).backward(g.double().transpose(1, 2))
    for name, got, want in zip(("dq", "dk", "dv"), grads[0], (qf.grad, kf.grad, vf.grad)):
        # probabilities, score gradients and the output behind the row statistics are rounded to bf16, as in the tests above
        assert relerr(got, want.transpose(1, 2)) < 1.5e-2, (name, relerr(got, want.transpose(1, 2)))


@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv,causal", [(8, 256, 256, 16, 8, True), (8, 640, 640, 16, 8, True), (4, 128, 1024, 16, 8, False),
                                                    (2, 512, 640, 32, 8, False), (1, 2048, 2048, 16, 8, True)])
def test_backward_on_cta_pairs(B, Sq, Skv, Hq, Hkv, causal):
    """Two key blocks per CTA pair: an even and an odd number of them (the last one's partner is not there), two iterations and
    many.  Gradients against fp64; dK and dV are summed in a fixed order, so a second run gives the same bits."""
    from torchure_b200 import ops
    from torchure_b200.ops import kernels
    from torchure_b200.ops.attention import flash_attention

    assert ops.ext().attn_bwd_on_pairs(B, Sq, Skv, Hq, Hkv, causal)
    torch.manual_seed(6)
    q = torch.randn(B, Sq, Hq, 128, device="cuda").bfloat16().requires_grad_()
    k, v = (torch.randn(B, Skv, Hkv, 128, device="cuda").bfloat16().requires_grad_() for _ in range(2))
    g = torch.randn_like(q)
    grads = [torch.autograd.grad(flash_attention(q, k, v, causal=causal), (q, k, v), g) for _ in range(2)]
    kernels.check_error()
    assert torch.equal(grads[0][1], grads[1][1]) and torch.equal(grads[0][2], grads[1][2])
    qf, kf, vf = (t.detach().double().transpose(1, 2).requires_grad_() for t in (q, k, v))
    s = qf @ kf.repeat_interleave(Hq // Hkv, 1).transpose(-1, -2) / 128 ** 0.5
    if causal:
        s = s.masked_fill(~torch.ones(Sq, Skv, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    (torch.softmax(s, -1) @ vf.repeat_interleave(Hq // Hkv, 1)).backward(g.double().transpose(1, 2))
    for name, got, want in zip(("dq", "dk", "dv"), grads[0], (qf.grad, kf.grad, vf.grad)):
        assert relerr(got, want.transpose(1, 2)) < 1.5e-2, (name, relerr(got, want.transpose(1, 2)))


@pytest.mark.parametrize("Sq,Skv,causal", [(640, 640, True), (256, 640, False)])
def test_backward_on_cta_pairs_inside_larger_tensors(Sq, Skv, causal):
    """Queries and keys at row offsets of larger tensors, statistics and dQ accumulator of a longer sequence, as a step of ring
    attention passes them: the same as on tensors of their own.  Everything outside holds NaN, which must not get in, least of
    all through the partner that the odd last key block does not have."""
    from torchure_b200 import ops
    from torchure_b200.ops import kernels

    E = ops.ext()
    B, Hq, Hkv, pad = 2, 16, 8, 128
    assert E.attn_bwd_on_pairs(B, Sq, Skv, Hq, Hkv, causal)
    torch.manual_seed(7)
    q, g, o = (torch.randn(B, Sq, Hq * 128, device="cuda").bfloat16() for _ in range(3))
    k, v = (torch.randn(B, Skv, Hkv * 128, device="cuda").bfloat16() for _ in range(2))
    lse = torch.full((B, Hq, Sq), 12.0, device="cuda")

    def inside(t):                                      # [B, pad + rows + pad, width], NaN around
        big = torch.full((B, t.shape[1] + 2 * pad, t.shape[2]), float("nan"), dtype=t.dtype, device="cuda")
        big[:, pad:pad + t.shape[1]] = t
        return big.flatten(0, 1)

    def run(qt, kt, vt, gt, rows_q, rows_k, off):
        stats = torch.full((2, B, Hq, rows_q), float("nan"), device="cuda")
        acc = torch.zeros(B, Hq, rows_q, 128, device="cuda")
        nds, nlse2, ref = (torch.empty(n, device="cuda").view(B, Hq, Sq, -1) for n in (B * Hq * Sq, B * Hq * Sq, B * Hq * Sq * 128))
        E.attn_bwd_stats(g.flatten(0, 1), o.flatten(0, 1), lse, nds, nlse2, ref, B, Sq, Hq)
        stats[0, :, :, off:off + Sq], stats[1, :, :, off:off + Sq] = nds.squeeze(-1), nlse2.squeeze(-1)
        dk, dv = (torch.empty(B * Skv, Hkv * 128, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        E.attn_bwd_pair(qt, 0, kt, 0, vt, 0, gt, acc, dk, dv, stats[0], stats[1], B, Sq, Skv, Hq, Hkv, rows_q, off, rows_k, off,
                        rows_q, off, causal)
        kernels.check_error()
        return acc, dk, dv

    a0, dk0, dv0 = run(*(t.flatten(0, 1) for t in (q, k, v, g)), Sq, Skv, 0)
    a1, dk1, dv1 = run(*map(inside, (q, k, v, g)), Sq + 2 * pad, Skv + 2 * pad, pad)
    assert torch.equal(dk0, dk1) and torch.equal(dv0, dv1)
    assert not a1[:, :, :pad].any() and not a1[:, :, pad + Sq:].any()
    # fp32 sums of up to five partial tiles in another order: a few units of 2^-24 of the terms
    assert relerr(a1[:, :, pad:pad + Sq], a0) < 1e-6
