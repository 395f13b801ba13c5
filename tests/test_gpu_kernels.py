"""GPU numerics: each sm_100a kernel against a plain PyTorch fp32 statement of the same op."""

import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


@pytest.fixture(autouse=True)
def _check_kernel_errors():
    yield
    from torchure_b200.ops import kernels

    kernels.check_error()


GEMM_SHAPES = [(128, 256, 64), (256, 512, 128), (384, 768, 1024), (8192, 1024, 2048), (1000, 520, 192),
               (77, 136, 64), (4096, 6144, 1024)]


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_bf16(M, N, K, a_mn, b_mn):
    from torchure_b200.ops import kernels

    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("a transposed operand needs a 16-byte aligned row stride")
    torch.manual_seed(0)
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = torch.randn(N, K, device="cuda").bfloat16()
    ref = a.float() @ b.float().t()
    a_in = a.t().contiguous() if a_mn else a
    b_in = b.t().contiguous() if b_mn else b
    out = kernels.gemm(a_in, b_in, a_mn=a_mn, b_mn=b_mn)
    assert out.dtype == torch.bfloat16 and out.shape == (M, N)
    assert relerr(out, ref) < 5e-3
    # elementwise: bf16 rounding of an fp32-accumulated result
    torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=2e-2 * ref.abs().max().item())


@pytest.mark.parametrize("M,N,K", [(256, 512, 128), (1000, 520, 192), (4096, 1024, 8192)])
def test_gemm_fp32_out_and_accumulate(M, N, K):
    from torchure_b200.ops import kernels

    torch.manual_seed(1)
    a = torch.randn(K, M, device="cuda").bfloat16()  # stored transposed: the wgrad layout
    b = torch.randn(K, N, device="cuda").bfloat16()
    ref = a.float().t() @ b.float()
    out = kernels.gemm(a, b, a_mn=True, b_mn=True, out_dtype=torch.float32)
    assert relerr(out, ref) < 1e-4
    base = torch.randn(M, N, device="cuda")
    acc = base.clone()
    kernels.gemm(a, b, a_mn=True, b_mn=True, out=acc, accumulate=True)
    assert relerr(acc, base + ref) < 1e-4


@pytest.mark.parametrize("tile_n,splits", [(64, 1), (64, 8), (128, 2), (128, 4), (256, 1), (256, 8), (-1, 3), (-1, 7)])
@pytest.mark.parametrize("M,N,K", [(128, 64, 512), (300, 520, 2500), (1, 8, 520), (257, 136, 1000)])
def test_gemm_few_tile_kernels(M, N, K, tile_n, splits):
    """The kernel for few output tiles (K slices summed inside a cluster) and the slices through a workspace, at single
    and ragged tiles and uneven slices: every operand layout, bf16 / fp32 / accumulating outputs, neighbours of a strided
    output untouched, same bits on a second run.  bf16 outputs are within half an ulp (2^-9) of the fp32 sum; fp32 sums
    of K <= 2500 products differ by their order only."""
    from torchure_b200 import ops

    if tile_n < 0 and M <= 128:
        pytest.skip("the pair kernel needs more than 128 rows")
    torch.manual_seed(0)
    pad = lambda n: (n + 7) // 8 * 8
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = torch.randn(N, K, device="cuda").bfloat16()
    ref = a.double() @ b.double().t()

    def stored(t, mn):
        t = t.t() if mn else t
        buf = torch.zeros(t.shape[0], pad(t.shape[1]), dtype=torch.bfloat16, device="cuda")
        buf[:, :t.shape[1]] = t
        return buf[:, :t.shape[1]]

    for mode, a_mn, b_mn in ((0, False, False), (0, False, True), (0, True, True), (1, True, True), (2, True, True),
                             (1, False, False), (2, False, False)):
        if tile_n < 0 and mode == 2:
            continue        # accumulating products split K by reduce-add
        x, y = stored(a, a_mn), stored(b, b_mn)
        dt = torch.bfloat16 if mode == 0 else torch.float32
        base = torch.full((M, pad(N) + 8), 3.0, dtype=dt, device="cuda")
        outs = []
        for _ in range(2):
            buf = base.clone()
            ops.ext().gemm(x, y, buf[:, :N], a_mn, b_mn, mode, splits, tile_n)
            outs.append(buf)
        want = ref + 3.0 if mode == 2 else ref
        assert relerr(outs[0][:, :N].double(), want) < (4e-3 if mode == 0 else 1e-5), (mode, a_mn, b_mn)
        assert (outs[0][:, N:] == 3.0).all(), "columns beyond N"
        assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("M,N,K,tile_n,splits", [(600, 512, 50257, 0, 0), (130, 64, 16400, 0, 0), (300, 520, 2500, 64, 4),
                                                 (1, 8, 520, 128, 2), (257, 136, 1000, 256, 1)])
def test_gemm_transposed_a_row_major_b(M, N, K, tile_n, splits):
    """A [K, M] with B [N, K], bf16 output, at few tiles and a long K: by the plan and on each width of the few-tile kernel.
    The output is rounded to bf16 once (2^-9)."""
    from torchure_b200 import ops

    torch.manual_seed(0)
    pad = lambda n: (n + 7) // 8 * 8
    a = torch.randn(K, pad(M), device="cuda").bfloat16()[:, :M]
    b = torch.randn(N, pad(K), device="cuda").bfloat16()[:, :K]
    out = torch.zeros(M, pad(N), device="cuda", dtype=torch.bfloat16)[:, :N]
    ops.ext().gemm(a, b, out, True, False, 0, splits, tile_n, may_split=True)
    assert relerr(out.double(), a.double().t() @ b.double().t()) < 4e-3


@pytest.mark.parametrize("K", [16384, 19456])       # 2 ffn_dim of the 1B and 4B blocks
def test_block_gradient_rows_do_not_depend_on_their_number(K):
    """The input gradient of a wide block, bf16: a row has the same bits among 128, 256 and 1024 rows."""
    from torchure_b200.ops import kernels

    torch.manual_seed(0)
    dy, w = torch.randn(1024, K, device="cuda").bfloat16(), torch.randn(K, 2048, device="cuda").bfloat16()
    whole = kernels.linear_dgrad(dy, w)
    for M in (128, 256):
        assert torch.equal(kernels.linear_dgrad(dy[:M], w), whole[:M]), M


@pytest.mark.parametrize("M,N,K", [(262, 384, 32245), (600, 512, 50257), (211, 256, 141510), (150, 1024, 20000)])
def test_head_gradient_in_slices_is_no_further_off(M, N, K):
    """dH of a head from softmax gradients, against 64 bits: summing K in slices is at least as close as one long fp32 sum,
    whose additions round K / 64 times as often (both end in a rounding to bf16, 2^-9 / sqrt(3) = 1.1e-3 on average)."""
    from torchure_b200 import ops

    torch.manual_seed(0)
    p = torch.softmax(torch.randn(M, (K + 7) // 8 * 8, device="cuda"), 1)
    p[torch.arange(M), torch.randint(0, K, (M,), device="cuda")] -= 1
    p, w = p.bfloat16()[:, :K], (torch.randn(K, N, device="cuda") * 0.02).bfloat16()
    want = p.double() @ w.double()
    errs = []
    for kw in (dict(splits=1), dict(may_split=True)):
        out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        ops.ext().gemm(p, w, out, False, True, 0, **kw)
        errs.append(((out.double() - want).norm() / want.norm()).item())
    assert errs[1] <= errs[0] * 1.001 and errs[0] < 4e-3, errs


@pytest.mark.parametrize("M,N,K", [(1024, 1024, 2048), (512, 512, 8192), (256, 512, 4096), (128, 128, 4096), (2048, 512, 2048)])
def test_fp32_products_are_as_close_as_the_split_by_reduce_add(M, N, K):
    """Weight gradients with few tiles against 64 bits: whichever kernel the plan takes, no further off than the split that
    adds K slices into C (1 % for the order of the slices); about 1.03e-9 per term of the longest slice."""
    from torchure_b200 import ops
    from torchure_b200.ops import kernels

    torch.manual_seed(0)
    a, b = torch.randn(K, M, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16()
    want = a.double().t() @ b.double()
    err = lambda o: ((o.double() - want).norm() / want.norm()).item()
    got = err(kernels.linear_wgrad(a, b, out_dtype=torch.float32))
    tiles, workers = -(-M // 256) * -(-N // 256), 74
    if M <= 128:
        tiles, workers = -(-N // 256), 148
    splits = min(range(1, 9), key=lambda s: (round(-(-tiles * s // workers) / s + 0.02 * (s - 1), 5), s))
    out = torch.empty(M, N, device="cuda")
    ops.ext().gemm(a, b, out, True, True, 1, splits)
    assert got <= 1.01 * err(out) and got < 1.3e-9 * K / splits + 2e-7, (got, err(out))


@pytest.mark.parametrize("M,D", [(130, 1032), (600, 1280), (1024, 2560), (3000, 2048), (2000, 4096)])
def test_rmsnorm_bwd_of_wide_rows_is_as_close_as_unstaged(M, D):
    """Rows shared by teams of warps against 64 bits, beside the kernels with one warp per row: dx no further off, the gain
    gradient neither, up to the order in which the CTAs' sums are added (mean of eight inputs, 8 %)."""
    from torchure_b200 import ops

    errs = torch.zeros(2, 2, dtype=torch.float64)
    for seed in range(8):
        g = torch.Generator("cuda").manual_seed(seed)
        rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
        x, dh, dx_in, w = rand(M, D), rand(M, D).bfloat16(), rand(M, D), rand(D).abs() + 0.5
        rstd = torch.rsqrt(x.double().pow(2).mean(-1) + 1e-6).float()
        xh, gw = x.double() * rstd.double()[:, None], dh.double() * w.double()
        want = (dx_in.double() + rstd.double()[:, None] * (gw - xh * (gw * xh).mean(-1, keepdim=True)), (dh.double() * xh).sum(0))
        for variant in (0, 1):
            dx, dxb, dw = torch.empty_like(x), torch.empty_like(dh), torch.zeros(D, device="cuda")
            ops.ext().rmsnorm_bwd(dh, x, w, rstd, dx_in, dx, dxb, dw, variant)
            for i, (got, ref) in enumerate(zip((dx, dw), want)):
                errs[variant, i] += (got.double() - ref).norm().cpu() / ref.norm().cpu()
    assert errs[0, 0] <= errs[1, 0] and errs[0, 1] <= 1.08 * errs[1, 1], errs


def test_gemm_with_reserved_sms():
    """Products with most SMs reserved and after the reservation was lifted, in a fresh process whose first launch has it:
    right in both states, and the pairs that the device holds are counted without it."""
    code = """
import torch
from torchure_b200 import ops
from torchure_b200.ops import kernels as K
torch.manual_seed(0)
a, b = torch.randn(2304, 512, device="cuda").bfloat16(), torch.randn(1024, 512, device="cuda").bfloat16()
ref = a.double() @ b.double().t()
outs = []
for free in (120, 16, 0):
    ops.set_compute_sm_reserve(free)
    outs.append(K.gemm(a, b))
    assert (outs[-1].double() - ref).norm() / ref.norm() < 4e-3
assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
wide = K.gemm(a, torch.randn(8192, 512, device="cuda").bfloat16())
assert ops.ext().gemm_pair_capacity() > 40, ops.ext().gemm_pair_capacity()
K.check_error()
"""
    res = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=240)
    assert res.returncode == 0, res.stderr[-1000:]


def test_gemm_strided_views():
    from torchure_b200.ops import kernels

    torch.manual_seed(2)
    big_a = torch.randn(512, 1024, device="cuda").bfloat16()
    big_b = torch.randn(768, 1024, device="cuda").bfloat16()
    big_o = torch.zeros(512, 1536, device="cuda", dtype=torch.bfloat16)
    a, b = big_a[:, 256:768], big_b[:, 256:768]
    out = big_o[:, 512:1280]
    kernels.gemm(a, b, out=out)
    ref = a.float() @ b.float().t()
    assert relerr(out, ref) < 5e-3
    assert big_o[:, :512].abs().sum() == 0 and big_o[:, 1280:].abs().sum() == 0


@pytest.mark.parametrize("M,D", [(64, 512), (1000, 1024), (8192, 1024), (333, 2560)])
def test_add_rmsnorm_fwd_bwd(M, D):
    from torchure_b200.ops import kernels, oracle

    torch.manual_seed(0)
    x = torch.randn(M, D, device="cuda")
    y = (torch.randn(M, D, device="cuda") * 0.5).bfloat16()
    w = torch.rand(D, device="cuda") + 0.5
    x_new, h, rstd = kernels.add_rmsnorm(x, y, w, 1e-6)
    xr = x + y.float()
    torch.testing.assert_close(x_new, xr)
    assert relerr(h, oracle.rmsnorm(xr, w, 1e-6)) < 5e-3
    torch.testing.assert_close(rstd, torch.rsqrt(xr.pow(2).mean(-1) + 1e-6), rtol=1e-5, atol=1e-6)
    # no residual: x passes through
    x2, h2, _ = kernels.add_rmsnorm(x, None, w, 1e-6)
    assert x2 is x and relerr(h2, oracle.rmsnorm(x, w, 1e-6)) < 5e-3
    # backward
    dh = torch.randn(M, D, device="cuda").bfloat16()
    dx_in = torch.randn(M, D, device="cuda")
    dw = torch.zeros(D, device="cuda")
    dx, dxb = kernels.rmsnorm_bwd(dh, xr, w, rstd, dx_in, dw)
    xa = xr.clone().requires_grad_()
    wa = w.clone().requires_grad_()
    oracle.rmsnorm(xa, wa, 1e-6).backward(dh.float())
    assert relerr(dx, xa.grad + dx_in) < 1e-5
    assert relerr(dxb, dx) < 5e-3
    assert relerr(dw, wa.grad) < 1e-4


@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("M,D", [(1, 1032), (7, 2048), (600, 1280), (3000, 2048), (1200, 2056), (333, 3072), (1201, 4096),
                                 (50, 4104)])
def test_rmsnorm_bwd_rows_shared_by_warps(M, D, residual):
    """Rows of more than 1024 columns: two or four warps per row, ragged last slices, fewer rows than teams, the widths on
    both sides of each limit.  fp32 sums of D products against fp64: 2^-24 sqrt(D) is 4e-6 at 4096, 1e-5 allowed; the gain
    gradient sums M rows, 1e-4 as above."""
    from torchure_b200.ops import kernels

    torch.manual_seed(0)
    x, dh = torch.randn(M, D, device="cuda"), torch.randn(M, D, device="cuda").bfloat16()
    w = torch.rand(D, device="cuda") + 0.5
    rstd = torch.rsqrt(x.pow(2).mean(-1) + 1e-6)
    dx_in = torch.randn(M, D, device="cuda") if residual else None
    dw = torch.ones(D, device="cuda")
    dx, dxb = kernels.rmsnorm_bwd(dh, x, w, rstd, dx_in, dw)
    kernels.check_error()
    r, xd, gd = rstd.double()[:, None], x.double(), dh.double()
    xh = xd * r
    want = r * (gd * w.double() - xh * (gd * w.double() * xh).mean(-1, keepdim=True))
    if residual:
        want = want + dx_in.double()
    assert relerr(dx.double(), want) < 1e-5
    assert relerr(dxb, dx) < 5e-3
    assert relerr(dw.double() - 1, (gd * xh).sum(0)) < 1e-4


def test_embedding_gather_norm_and_scatter():
    from torchure_b200.ops import kernels, oracle

    torch.manual_seed(0)
    V, D, M = 1000, 512, 777
    table = torch.randn(V, D, device="cuda")
    ids = torch.randint(0, V, (M,), device="cuda")
    w = torch.rand(D, device="cuda") + 0.5
    x, h, _ = kernels.add_rmsnorm(None, None, w, 1e-6, ids=ids, table=table)
    torch.testing.assert_close(x, table[ids])
    assert relerr(h, oracle.rmsnorm(table[ids], w, 1e-6)) < 5e-3
    dx = torch.randn(M, D, device="cuda")
    dt = torch.zeros(V, D, device="cuda")
    kernels.embedding_bwd_(dx, ids, dt)
    ref = torch.zeros(V, D, device="cuda").index_add_(0, ids, dx)
    torch.testing.assert_close(dt, ref, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("use_norm", [True, False])
def test_qknorm_rope_fwd_bwd(use_norm):
    from torchure_b200.models.qwen3 import RotaryEmbedding
    from torchure_b200.ops import kernels, oracle

    torch.manual_seed(0)
    B, S, Hq, Hkv, hd = 2, 256, 4, 2, 128
    qkv = torch.randn(B * S, (Hq + 2 * Hkv) * hd, device="cuda").bfloat16()
    qw, kw = torch.rand(hd, device="cuda") + 0.5, torch.rand(hd, device="cuda") + 0.5
    cos, sin = RotaryEmbedding(hd).tables(S, "cuda")
    out = kernels.qknorm_rope(qkv, qw, kw, cos, sin, S, Hq, Hkv, 1e-6, use_norm)
    qa = qkv.float().requires_grad_()
    qwa, kwa = qw.clone().requires_grad_(), kw.clone().requires_grad_()
    ref = oracle.qknorm_rope(qa, qwa, kwa, cos, sin, B, S, Hq, Hkv, hd, 1e-6, use_norm)
    assert relerr(out, ref) < 8e-3
    g = torch.randn(B * S, (Hq + 2 * Hkv) * hd, device="cuda").bfloat16()
    ref.backward(g[:, :(Hq + Hkv) * hd].float())
    dqw, dkw = torch.zeros(hd, device="cuda"), torch.zeros(hd, device="cuda")
    d = g.clone()
    kernels.qknorm_rope_bwd_(d, qkv, qw, kw, cos, sin, dqw, dkw, S, Hq, Hkv, 1e-6, use_norm)
    assert relerr(d[:, :(Hq + Hkv) * hd], qa.grad[:, :(Hq + Hkv) * hd]) < 8e-3
    assert torch.equal(d[:, (Hq + Hkv) * hd:], g[:, (Hq + Hkv) * hd:]), "the v columns must pass through"
    if use_norm:
        assert relerr(dqw, qwa.grad) < 5e-3 and relerr(dkw, kwa.grad) < 5e-3


@pytest.mark.parametrize("Hq,Hkv", [(4, 2), (16, 8), (6, 3)])
def test_qknorm_rope_bwd_reads_dq_from_the_fp32_accumulator(Hq, Hkv):
    """dq taken from the head-major fp32 accumulator gives what the q columns of dqkv give when both hold the same
    values, on both row-buffer plans of the kernel; an odd number of k heads leaves half a warp idle in the last pass."""
    from torchure_b200 import ops
    from torchure_b200.models.qwen3 import RotaryEmbedding
    from torchure_b200.ops import kernels

    torch.manual_seed(1)
    B, S, hd = 2, 384, 128
    M = B * S
    qkv = torch.randn(M, (Hq + 2 * Hkv) * hd, device="cuda").bfloat16()
    g = torch.randn(M, (Hq + 2 * Hkv) * hd, device="cuda").bfloat16()
    qw, kw = torch.rand(hd, device="cuda") + 0.5, torch.rand(hd, device="cuda") + 0.5
    cos, sin = RotaryEmbedding(hd).tables(S, "cuda")
    acc = g[:, :Hq * hd].float().view(B, S, Hq, hd).permute(0, 2, 1, 3).contiguous()
    outs = []
    for dq_acc, stages in ((None, 1), (None, 2), (acc, 1), (acc, 2)):
        d = g.clone()
        if dq_acc is not None:
            d[:, :Hq * hd] = 0          # must not be read
        dqw, dkw = torch.zeros(hd, device="cuda"), torch.zeros(hd, device="cuda")
        ops.ext().qknorm_rope_bwd(d, qkv, qw, kw, cos, sin, dqw, dkw, S, Hq, Hkv, 1e-6, True, dq_acc, stages)
        outs.append((d, dqw, dkw))
    kernels.check_error()
    for d, dqw, dkw in outs[1:]:
        assert torch.equal(d, outs[0][0])
        torch.testing.assert_close(dqw, outs[0][1], rtol=1e-4, atol=1e-3)
        torch.testing.assert_close(dkw, outs[0][2], rtol=1e-4, atol=1e-3)


@pytest.mark.parametrize("M,N,K", [(19074, 512, 128), (9600, 904, 72), (20000, 1504, 64), (5000, 4000, 64)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_gemm_tall_outputs_in_groups_of_tile_rows(M, N, K, a_mn, b_mn):
    """Tall outputs go through groups of tile rows: a last group of fewer rows, ragged tiles at both edges, several groups and
    one, every operand order and output mode of the CTA-pair kernel."""
    from torchure_b200.ops import kernels

    torch.manual_seed(8)

    def operand(rows, k_major):
        t = torch.randn(rows, K, device="cuda").bfloat16()
        if k_major:
            return t, t
        wide = torch.zeros(K, (rows + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
        wide[:, :rows] = t.t()
        return t, wide[:, :rows]

    a, a_arg = operand(M, not a_mn)
    b, b_arg = operand(N, not b_mn)
    ref = a.float() @ b.float().t()
    out = kernels.gemm(a_arg, b_arg, a_mn=a_mn, b_mn=b_mn)
    assert relerr(out, ref) < 4e-3                    # rounded to bf16: 2^-9
    if a_mn == b_mn or not a_mn:
        acc = torch.ones(M, N, device="cuda")
        if a_mn == b_mn:
            kernels.gemm(a_arg, b_arg, a_mn=a_mn, b_mn=b_mn, out=acc, accumulate=True)
            assert relerr(acc, ref + 1) < 1e-5
        kernels.gemm(a_arg, b_arg, a_mn=a_mn, b_mn=b_mn, out=acc)
        assert relerr(acc, ref) < 1e-5                # fp32 sums of at most 128 products


@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 8191, 300001])
@pytest.mark.parametrize("share", [0.0, 0.3, 1.0])
def test_ce_count_and_mean(n, share):
    """The number of labels that count (at least one) and the mean loss, against fp64; one element to many per thread."""
    from torchure_b200.ops import kernels

    torch.manual_seed(9)
    y = torch.randint(0, 50, (n,), device="cuda").masked_fill_(torch.rand(n, device="cuda") < share, -100)
    inv = kernels.ce_inverse_count(y, -100, 0.5)
    want = 0.5 / max(1, int((y != -100).sum()))
    assert inv.shape == (1,) and abs(inv.item() / want - 1) < 2e-7
    rows = torch.rand(n, device="cuda") * 12
    mean = kernels.ce_mean(rows, inv)
    # rounded to fp32 three times: the sum, the factor, the product
    assert mean.shape == () and abs(mean.item() / (rows.double().sum().item() * want) - 1) < 3e-7


@pytest.mark.parametrize("Hq,Hkv,M", [(2, 1, 1), (4, 2, 7), (6, 3, 130), (10, 5, 9), (16, 8, 129), (24, 6, 33), (2, 2, 5000)])
@pytest.mark.parametrize("variant", [0, 1, 2])
def test_qknorm_rope_chunks(Hq, Hkv, M, variant):
    """Heads are worked on in chunks of eight (backward: also of four) of one kind or of both, rows by warps that take several:
    chunks that are not full, a kind that fills none, rows that fill no CTA and more rows than warps."""
    from torchure_b200 import ops
    from torchure_b200.models.qwen3 import RotaryEmbedding
    from torchure_b200.ops import kernels, oracle

    torch.manual_seed(2)
    hd = 128
    qkv = torch.randn(M, (Hq + 2 * Hkv) * hd, device="cuda").bfloat16()
    qw, kw = torch.rand(hd, device="cuda") + 0.5, torch.rand(hd, device="cuda") + 0.5
    cos, sin = RotaryEmbedding(hd).tables(M, "cuda")
    qa = qkv.float().requires_grad_()
    qwa, kwa = qw.clone().requires_grad_(), kw.clone().requires_grad_()
    ref = oracle.qknorm_rope(qa, qwa, kwa, cos, sin, 1, M, Hq, Hkv, hd, 1e-6, True)
    assert relerr(kernels.qknorm_rope(qkv, qw, kw, cos, sin, M, Hq, Hkv, 1e-6, True), ref) < 8e-3
    g = torch.randn(M, (Hq + 2 * Hkv) * hd, device="cuda").bfloat16()
    ref.backward(g[:, :(Hq + Hkv) * hd].float())
    acc = g[:, :Hq * hd].float().view(1, M, Hq, hd).permute(0, 2, 1, 3).contiguous()
    for dq_acc in (None, acc):
        d, dqw, dkw = g.clone(), torch.zeros(hd, device="cuda"), torch.zeros(hd, device="cuda")
        ops.ext().qknorm_rope_bwd(d, qkv, qw, kw, cos, sin, dqw, dkw, M, Hq, Hkv, 1e-6, True, dq_acc, variant)
        assert relerr(d[:, :(Hq + Hkv) * hd], qa.grad[:, :(Hq + Hkv) * hd]) < 8e-3
        assert torch.equal(d[:, (Hq + Hkv) * hd:], g[:, (Hq + Hkv) * hd:])
        # the forward of the reference rounds the normalised values to bf16, whose gradient passes unrounded: 5e-3 as above
        assert relerr(dqw, qwa.grad) < 5e-3 and relerr(dkw, kwa.grad) < 5e-3


@pytest.mark.parametrize("Hq,Hkv,M", [(2, 1, 130), (4, 2, 9), (6, 3, 130), (10, 5, 9), (16, 8, 129)])
@pytest.mark.parametrize("variant", [0, 1, 2])
def test_qknorm_rope_bwd_without_eps(Hq, Hkv, M, variant):
    """eps = 0: the halves of a warp that have no head of their own (chunks that are not full) add nothing to the gain gradients."""
    from torchure_b200 import ops
    from torchure_b200.models.qwen3 import RotaryEmbedding
    from torchure_b200.ops import oracle

    torch.manual_seed(3)
    hd = 128
    qkv = torch.randn(M, (Hq + 2 * Hkv) * hd, device="cuda").bfloat16()
    qw, kw = torch.rand(hd, device="cuda") + 0.5, torch.rand(hd, device="cuda") + 0.5
    cos, sin = RotaryEmbedding(hd).tables(M, "cuda")
    qa = qkv.float().requires_grad_()
    qwa, kwa = qw.clone().requires_grad_(), kw.clone().requires_grad_()
    g = torch.randn(M, (Hq + 2 * Hkv) * hd, device="cuda").bfloat16()
    oracle.qknorm_rope(qa, qwa, kwa, cos, sin, 1, M, Hq, Hkv, hd, 0.0, True).backward(g[:, :(Hq + Hkv) * hd].float())
    acc = g[:, :Hq * hd].float().view(1, M, Hq, hd).permute(0, 2, 1, 3).contiguous()
    for dq_acc in (None, acc):
        d, dqw, dkw = g.clone(), torch.zeros(hd, device="cuda"), torch.zeros(hd, device="cuda")
        ops.ext().qknorm_rope_bwd(d, qkv, qw, kw, cos, sin, dqw, dkw, M, Hq, Hkv, 0.0, True, dq_acc, variant)
        # as in test_qknorm_rope_chunks
        assert relerr(d[:, :(Hq + Hkv) * hd], qa.grad[:, :(Hq + Hkv) * hd]) < 8e-3
        assert relerr(dqw, qwa.grad) < 5e-3 and relerr(dkw, kwa.grad) < 5e-3


def test_swiglu_fwd_bwd():
    from torchure_b200.ops import kernels, oracle

    torch.manual_seed(0)
    M, F_ = 1000, 3072
    gu = torch.randn(M, 2 * F_, device="cuda").bfloat16()
    act = kernels.swiglu(gu)
    ga = gu.float().requires_grad_()
    ref = oracle.swiglu(ga)
    assert relerr(act, ref) < 5e-3
    d = torch.randn(M, F_, device="cuda").bfloat16()
    ref.backward(d.float())
    assert relerr(kernels.swiglu_bwd(d, gu), ga.grad) < 5e-3


@pytest.mark.parametrize("M,F,K", [(4096, 1536, 256), (4000, 1544, 192), (2304, 2184, 72), (1100, 3080, 520)])
def test_linear_swiglu_epilogue(M, F, K):
    """The activation in the product's epilogue: the bits of the product followed by the pass over it, with ragged rows,
    ragged last column tiles (whose gate half must not spill into the up half) and a ragged last k block."""
    from torchure_b200 import ops
    from torchure_b200.ops import debug
    from torchure_b200.ops import kernels as k

    torch.manual_seed(0)
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(2 * F, K, device="cuda") * 0.2).bfloat16()
    gu_ref = k.gemm(x, w)
    act_ref = k.swiglu(gu_ref)
    debug.enable(True)
    try:
        before = ops.launches()
        gu, act = k.linear_swiglu(x, w)
        assert ops.launches() - before == 1, "expected the fused kernel"
        none, alone = k.linear_swiglu(x, w, want_gu=False)
        assert none is None
        debug.verify()
    finally:
        debug.enable(False)
    k.check_error()
    assert torch.equal(gu, gu_ref) and torch.equal(act, act_ref) and torch.equal(alone, act_ref)
    # few tiles: another kernel and a pass of its own
    gu, act = k.linear_swiglu(x[:64], w)
    assert torch.equal(act, k.swiglu(gu))


@pytest.mark.parametrize("M,F,K", [(4096, 3856, 2048), (2000, 7696, 2056), (1100, 12304, 2112)])
def test_swiglu_dgrad_epilogue(M, F, K):
    """d(gate) and d(up) in the epilogue of d(act) = dy W against fp64 on the same operands; ragged rows, last column tiles of
    16 columns, a ragged last k block.  Only the results are rounded: 2^-9 relative per element."""
    from torchure_b200 import ops
    from torchure_b200.ops import debug
    from torchure_b200.ops import kernels as k

    torch.manual_seed(0)
    dy, gu = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(M, 2 * F, device="cuda") * 2).bfloat16()
    gu[0, :64] = torch.linspace(-200, 200, 64, device="cuda")
    w = (torch.randn(K, F, device="cuda") * 0.2).bfloat16()
    debug.enable(True)
    try:
        before = ops.launches()
        got = k.swiglu_dgrad(dy, w, gu)
        assert ops.launches() - before == 1, "expected the fused kernel"
        debug.verify()
    finally:
        debug.enable(False)
    k.check_error()
    two = k.swiglu_bwd(k.linear_dgrad(dy, w), gu)
    d, g, u = dy.double() @ w.double(), gu[:, :F].double(), gu[:, F:].double()
    s = torch.sigmoid(g)
    want = torch.cat([d * u * s * (1 + g * (1 - s)), d * g * s], 1)
    err = ((got.double() - want).norm() / want.norm()).item()
    assert err < 2e-3 and err <= ((two.double() - want).norm() / want.norm()).item()
    # few tiles, and few waves of them: the product and a pass of its own
    before = ops.launches()
    assert torch.equal(k.swiglu_dgrad(dy[:1024], w[:, :3072], gu[:1024, :6144].contiguous()),
                       k.swiglu_bwd(k.linear_dgrad(dy[:1024], w[:, :3072]), gu[:1024, :6144].contiguous()))
    assert ops.launches() - before == 4
    assert torch.equal(k.swiglu_dgrad(dy[:64], w, gu[:64]), k.swiglu_bwd(k.linear_dgrad(dy[:64], w), gu[:64]))


@pytest.mark.parametrize("C,V,K", [(512, 50257, 128), (300, 32003, 200), (4096, 2056, 64), (257, 65544, 72)])
def test_gemm_ce_statistics(C, V, K):
    """Loss from the product's epilogue against the loss pass over stored logits and fp64, over ragged vocabularies (last tile
    of 1, 3, 8 columns), ragged rows, ignored and out-of-range labels."""
    from torchure_b200.ops import kernels as k

    torch.manual_seed(0)
    h = torch.randn(C, K, device="cuda").bfloat16()
    w = (torch.randn(V, K, device="cuda") * 0.5).bfloat16()
    y = torch.randint(0, V, (C,), device="cuda")
    y[0], y[1], y[2::7], y[3] = V - 1, 0, -100, V + 5
    logits = torch.zeros(C, (V + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")[:, :V]
    k.gemm(h, w, out=logits)
    target = torch.full((C,), 7.0, device="cuda")
    tiles = k.gemm_ce(h, w, y, target)
    assert tiles is not None, "expected the CTA-pair kernel"
    lse = torch.logsumexp(tiles[..., 0].double() + tiles[..., 1].double().log(), 0)
    # fp32 sums of at most 256 terms (2^-24 x 16 relative), exp2 approximate to 2^-22
    torch.testing.assert_close(lse, torch.logsumexp(logits.double(), 1), rtol=1e-6, atol=2e-6)
    live = (y >= 0) & (y < V)
    assert torch.equal(target[live], logits[live].gather(1, y[live, None])[:, 0].float()) and (target[~live] == 7).all()
    a, b = torch.full((C,), 7.0, device="cuda"), torch.full((C,), 7.0, device="cuda")
    k.ce_loss_tiles(tiles, target, y, a, V, -100)
    k.ce_loss(logits, y, b, -100)
    k.check_error()
    torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)
    assert (a[2::7] == 0).all()


@pytest.mark.parametrize("C,V", [(64, 1000), (300, 5000), (512, 151936), (600, 50264), (130, 32000)])
def test_ce_softmax_grad(C, V):
    from torchure_b200.ops import kernels

    torch.manual_seed(0)
    logits = (torch.randn(C, V, device="cuda") * 2).bfloat16()
    labels = torch.randint(0, V, (C,), device="cuda")
    labels[torch.rand(C, device="cuda") < 0.1] = -100
    n_valid = (labels != -100).sum().clamp_min(1)
    inv = (1.0 / n_valid).float().reshape(1)
    la = logits.float().requires_grad_()
    ref = torch.nn.functional.cross_entropy(la, labels, ignore_index=-100, reduction="sum")
    ref.backward()
    work = logits.clone()
    row_loss = torch.empty(C, device="cuda")
    kernels.ce_softmax_grad_(work, labels, row_loss, inv, -100)
    torch.testing.assert_close(row_loss.sum(), ref.detach(), rtol=1e-4, atol=1e-3)
    assert relerr(work, la.grad / n_valid) < 8e-3
    assert work[labels == -100].abs().sum() == 0


@pytest.mark.parametrize("C,V", [(3, 17), (64, 1000), (130, 32003)])
def test_ce_loss_alone(C, V):
    """The loss of a pass without gradients: the bits of the fused step's, logits untouched, ignored rows zero."""
    from torchure_b200.ops import kernels

    torch.manual_seed(0)
    ld = (V + 7) // 8 * 8
    logits = (torch.randn(C, ld, device="cuda") * 3).bfloat16()[:, :V]
    labels = torch.randint(0, V, (C,), device="cuda")
    labels[::5] = -100
    before = logits.clone()
    alone, fused = torch.full((C,), 7.0, device="cuda"), torch.full((C,), 7.0, device="cuda")
    kernels.ce_loss(logits, labels, alone, -100)
    assert torch.equal(logits, before)
    kernels.ce_softmax_grad_(logits, labels, fused, torch.ones(1, device="cuda"), -100)
    assert torch.equal(alone, fused) and (alone[::5] == 0).all()
    want = torch.nn.functional.cross_entropy(before.float(), labels, reduction="none")
    torch.testing.assert_close(alone, want, rtol=1e-4, atol=1e-4)


def test_linear_ce_without_gradients():
    """no_grad with a weight that requires a gradient: same loss, no gradient work (one product and one loss per chunk)."""
    from torchure_b200 import ops
    from torchure_b200.loss import fused_linear_cross_entropy

    torch.manual_seed(0)
    h = torch.randn(300, 256, device="cuda").bfloat16()
    w = (torch.randn(1000, 256, device="cuda") * 0.05).bfloat16().requires_grad_()
    y = torch.randint(0, 1000, (300,), device="cuda")
    y[3:40] = -100
    full = fused_linear_cross_entropy(h, w, y, -100, 128)
    with torch.no_grad():
        before = ops.launches()
        loss = fused_linear_cross_entropy(h, w, y, -100, 128)
        assert ops.launches() - before == 2 * 3
    assert not loss.requires_grad and torch.equal(loss, full.detach())
    full.backward()
    assert w.grad is not None


def test_product_in_slices_without_room_for_them():
    """A dH whose K slices do not fit the memory that is left runs in one piece."""
    from torchure_b200 import ops
    from torchure_b200.ops import kernels as K

    M, N, V = 1000, 2560, 66000
    kind, _, _, workspace = ops.ext().gemm_plan(M, N, V, b_mn=True, may_split=True)
    assert kind == "slices" and workspace > 16 << 20
    torch.manual_seed(0)
    a, b = torch.randn(M, V, device="cuda").bfloat16(), torch.randn(V, N, device="cuda").bfloat16()
    want, out = K.gemm(a, b, b_mn=True), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    torch.cuda.empty_cache()
    taken = []
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (4 << 20)) / torch.cuda.mem_get_info()[1])
        with pytest.raises(torch.OutOfMemoryError):
            while True:               # free blocks among what earlier tests hold
                taken.append(torch.empty(workspace, dtype=torch.uint8, device="cuda"))
        K.gemm(a, b, b_mn=True, out=out, may_split=True)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        del taken
    assert torch.equal(out, want)
    K.gemm(a, b, b_mn=True, out=out, may_split=True)      # sums of slices round elsewhere: 2^-8 of the value, and rarely
    assert not torch.equal(out, want) and relerr(out, want) < 4e-3
    K.check_error()


@pytest.mark.parametrize("rows", [100, 300])
def test_linear_ce_with_a_count_kept_on_the_host(rows):
    """A normalizer on the CPU gives what the same number on the GPU gives, with and without gradients."""
    from torchure_b200.loss import fused_linear_cross_entropy
    from torchure_b200.ops import kernels

    torch.manual_seed(0)
    h = torch.randn(rows, 256, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(17000, 256, device="cuda") * 0.05).bfloat16()
    y = torch.randint(0, 17000, (rows,), device="cuda")
    want, got = [], []
    for out, n in ((want, torch.tensor(rows // 2, device="cuda")), (got, torch.tensor(rows // 2))):
        with torch.no_grad():
            out.append(fused_linear_cross_entropy(h, w, y, -100, 256, 1.0, n))
        h.grad = None
        loss = fused_linear_cross_entropy(h, w, y, -100, 256, 1.0, n)
        loss.backward()
        out += [loss.detach(), h.grad]
    kernels.check_error()
    for a, b in zip(got, want):
        assert a.is_cuda and torch.equal(a, b)
    with pytest.raises(RuntimeError, match="on the GPU"):
        kernels.ce_mean(torch.zeros(4, device="cuda"), torch.ones(1))


def test_linear_ce_loss_changed_in_place():
    """The loss is a tensor of its own, as on the CPU: a script may divide or add to it before backward, or detach it."""
    from torchure_b200.loss import fused_linear_cross_entropy

    torch.manual_seed(0)
    h = torch.randn(300, 256, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(1000, 256, device="cuda") * 0.05).bfloat16()
    y = torch.randint(0, 1000, (300,), device="cuda")
    plain = fused_linear_cross_entropy(h, w, y, -100, 128)
    plain.backward()
    grad, h.grad = h.grad, None
    loss = fused_linear_cross_entropy(h, w, y, -100, 128)
    loss /= 4
    loss += 1
    assert abs(loss.item() - plain.item() / 4 - 1) < 1e-6      # two roundings to fp32
    loss.backward()
    assert torch.equal(h.grad, grad / 4)                       # a power of two: exact
    loss = fused_linear_cross_entropy(h, w, y, -100, 128)
    loss.detach_()
    assert not loss.requires_grad and torch.equal(loss, plain.detach())


@pytest.mark.parametrize("rows,vocab,chunk,paths", [(1100, 50257, 512, [True, True, False]), (900, 20001, 300, [True] * 3),
                                                    (300, 1000, 128, [False] * 3)])
def test_linear_ce_without_gradients_chunk_by_chunk(monkeypatch, rows, vocab, chunk, paths):
    """Chunks whose logits are not stored (more than 128 rows), a short last one that stores them, and only such: the loss
    of every chunk's rows by themselves, ignored and out-of-range labels among them, is that of the pass with gradients.
    The same logits, summed in another order: 2^-24 x 16 relative per row, as in the test of the statistics."""
    from torchure_b200.loss import fused_linear_cross_entropy
    from torchure_b200.ops import debug
    from torchure_b200.ops import kernels as K

    torch.manual_seed(0)
    h = torch.randn(rows, 256, device="cuda").bfloat16()
    w = (torch.randn(vocab, 256, device="cuda") * 0.2).bfloat16().requires_grad_()
    y = torch.randint(0, vocab, (rows,), device="cuda")
    y[::9] = -100
    y[5] = vocab + 3
    taken, gemm_ce = [], K.gemm_ce
    monkeypatch.setattr(K, "gemm_ce", lambda *a: taken.append(gemm_ce(*a)) or taken[-1])
    for lo in (0, *range(0, rows, chunk)):
        part = y.clone() if not taken else torch.full_like(y, -100)
        part[lo:lo + chunk] = y[lo:lo + chunk]
        full = fused_linear_cross_entropy(h, w, part, -100, chunk)
        before = len(taken)
        with torch.no_grad():
            loss = fused_linear_cross_entropy(h, w, part, -100, chunk)
        assert [t is not None for t in taken[before:]] == paths
        torch.testing.assert_close(loss, full.detach(), rtol=2e-6, atol=0)
    debug.enable(True)
    try:
        with torch.no_grad():
            fused_linear_cross_entropy(h, w, y, -100, chunk)
        assert sum(n == "gemm_ce.stats" for n, _ in debug._pending) == sum(paths)
        debug.verify()
    finally:
        debug.enable(False)


@pytest.mark.parametrize("offset", [0.0, 60.0, 400.0])
def test_loss_without_logits_is_as_close_as_with(offset):
    """Row losses from the product's epilogue and from stored logits against 64 bits on the same rounded logits, whose level
    lies around `offset`: the mean error of 512 rows is no larger (5 %), mostly the rounding of maximum + log."""
    from torchure_b200.ops import kernels as K

    torch.manual_seed(0)
    C, V, D = 512, 40000, 128
    h, w = torch.randn(C, D, device="cuda").bfloat16(), torch.randn(V, D, device="cuda").bfloat16()
    h[:, 0], w[:, 0] = 1, offset
    y = torch.randint(0, V, (C,), device="cuda")
    logits = K.gemm(h, w)
    want = torch.nn.functional.cross_entropy(logits.double(), y, reduction="none")
    stored, fused, target = (torch.empty(C, device="cuda") for _ in range(3))
    K.ce_loss(logits, y, stored, -100)
    K.ce_loss_tiles(K.gemm_ce(h, w, y, target), target, y, fused, V, -100)
    err = lambda t: (t.double() - want).abs().mean().item()
    assert err(fused) <= 1.05 * err(stored), (err(fused), err(stored))


def test_gemm_ce_decides_before_it_allocates():
    from torchure_b200.ops import kernels as K

    h, w = torch.zeros(128, 64, device="cuda").bfloat16(), torch.zeros(1 << 20, 64, device="cuda").bfloat16()
    y, target = torch.zeros(128, dtype=torch.int64, device="cuda"), torch.empty(128, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    assert K.gemm_ce(h, w, y, target) is None and torch.cuda.max_memory_allocated() == before


# statistics from the product (300 rows) and a pass over stored logits (100)
@pytest.mark.parametrize("rows,lo,hi", [(300, 16400, 17000), (100, 16400, 17000), (300, 256, 512), (300, 0, 1), (100, 0, 1)])
def test_linear_ce_without_gradients_infinite_logits(rows, lo, hi):
    """Vocabulary rows whose logits are all -inf (the last tiles of 256 columns, the first ones, one column) add nothing to the
    loss; NaN in the same places makes it NaN."""
    from torchure_b200.loss import fused_linear_cross_entropy

    torch.manual_seed(0)
    h = (torch.rand(rows, 128, device="cuda") + 0.5).bfloat16()
    w = (torch.randn(17000, 128, device="cuda") * 0.1).bfloat16()
    y = torch.randint(512, 16400, (rows,), device="cuda")
    if (lo, hi) == (256, 512):
        w[:256] = -3e38
    w[lo:hi] = -3e38                    # times h beyond the range of fp32
    with torch.no_grad():
        loss = fused_linear_cross_entropy(h, w, y, -100, 300)
        logits = (h.float() @ w.float().t()).bfloat16().double()
        assert (logits == -float("inf")).any()
        # logits rounded to bf16 from sums in another order: single ones differ by 2^-8 of their value, at most 2
        torch.testing.assert_close(loss.double(), torch.nn.functional.cross_entropy(logits, y), rtol=1e-3, atol=0)
        w[lo:hi] = float("nan")
        assert fused_linear_cross_entropy(h, w, y, -100, 300).isnan()


@pytest.mark.parametrize("C,V,shards", [(64, 1024, 2), (300, 5008, 2), (256, 151936, 4)])   # shard rows stay 16-byte aligned
def test_ce_vocabulary_sharded_passes(C, V, shards):
    """The two passes of the loss-parallel CE on column shards of one logits matrix (what the ranks of a
    tensor-parallel axis hold): row statistics per shard, combined as the ranks' all-reduces would, must give the
    log-sum-exp and target logit of the whole row; the gradient pass must give (softmax - onehot) / n."""
    from torchure_b200.ops import kernels

    torch.manual_seed(0)
    logits = (torch.randn(C, V, device="cuda") * 2).bfloat16()
    labels = torch.randint(0, V, (C,), device="cuda")
    labels[torch.rand(C, device="cuda") < 0.1] = -100
    keep = labels != -100
    inv = (1.0 / keep.sum().clamp_min(1)).float().reshape(1)
    la = logits.float().requires_grad_()
    ref = torch.nn.functional.cross_entropy(la, labels, ignore_index=-100, reduction="sum")
    ref.backward()
    per = V // shards
    parts = [logits[:, r * per:(r + 1) * per].contiguous() for r in range(shards)]
    stats = [torch.empty(3, C, device="cuda") for _ in range(shards)]
    for r in range(shards):
        kernels.ce_row_stats_(parts[r], labels, stats[r], r * per, -100)
    mx = torch.stack([s[0] for s in stats]).max(dim=0).values
    sumexp = sum(s[1] * torch.exp(s[0] - mx) for s in stats)
    tgt = sum(s[2] for s in stats)
    lse = mx + torch.log(sumexp)
    torch.testing.assert_close(lse, torch.logsumexp(logits.float(), dim=-1), rtol=1e-5, atol=1e-4)
    want_tgt = logits.float().gather(1, labels.clamp_min(0)[:, None]).squeeze(1) * keep
    torch.testing.assert_close(tgt, want_tgt, rtol=0, atol=0)
    torch.testing.assert_close(((lse - tgt) * keep).sum(), ref.detach(), rtol=1e-4, atol=1e-3)
    for r in range(shards):
        kernels.ce_grad_from_lse_(parts[r], labels, lse, inv, r * per, -100)
        want = la.grad[:, r * per:(r + 1) * per] * inv
        assert relerr(parts[r], want) < 8e-3, r
        assert parts[r][~keep].abs().sum() == 0
    kernels.check_error()


def test_multi_tensor_adamw_norm_scale():
    from torchure_b200.ops import multi_tensor, oracle

    torch.manual_seed(0)
    shapes = [(1024, 1024), (128,), (3, 5, 7), (40000,), (1,)]
    ps = [torch.randn(s, device="cuda") for s in shapes]
    gs = [torch.randn(s, device="cuda") for s in shapes]
    gs[1] = gs[1].bfloat16()
    ms = [torch.randn(s, device="cuda") * 0.1 for s in shapes]
    vs = [torch.rand(s, device="cuda") * 0.1 for s in shapes]
    sh = [torch.empty(s, device="cuda", dtype=torch.bfloat16) if i != 2 else None for i, s in enumerate(shapes)]
    want_sq = sum(g.float().pow(2).sum() for g in gs)
    torch.testing.assert_close(multi_tensor.sq_norm(gs), want_sq, rtol=1e-4, atol=1e-3)
    coef = torch.tensor(0.37, device="cuda")
    refs = [oracle.adamw(p.clone(), g.float() * 0.37, m.clone(), v.clone(), 1e-2, 0.9, 0.95, 1e-8, 0.1, 3)
            for p, g, m, v in zip(ps, gs, ms, vs)]
    multi_tensor.adamw_step(ps, gs, ms, vs, sh, 1e-2, 0.9, 0.95, 1e-8, 0.1, 3, grad_scale=coef)
    for p, m, v, s, (rp, rm, rv) in zip(ps, ms, vs, sh, refs):
        torch.testing.assert_close(p, rp, rtol=1e-5, atol=1e-6)
        torch.testing.assert_close(m, rm, rtol=1e-5, atol=1e-6)
        torch.testing.assert_close(v, rv, rtol=1e-5, atol=1e-6)
        if s is not None:
            torch.testing.assert_close(s.float(), rp, rtol=1e-2, atol=1e-2)
    xs = [torch.randn(s, device="cuda") for s in shapes]
    want = [x * 0.5 for x in xs]
    multi_tensor.scale_(xs, torch.tensor(0.5, device="cuda"))
    for x, wv in zip(xs, want):
        torch.testing.assert_close(x, wv)


def test_multi_tensor_tables_follow_moved_tensors():
    """Tensors of the same sizes at new addresses reuse the table's sizes and upload only their addresses."""
    from torchure_b200.ops import multi_tensor

    torch.manual_seed(0)
    keep = []
    for _ in range(4):
        ts = [torch.randn(n, device="cuda") for n in (5, 40000, 16384, 1)]
        keep.append(ts)
        want = sum(t.double().pow(2).sum() for t in ts)
        torch.testing.assert_close(multi_tensor.sq_norm(ts).double(), want, rtol=1e-5, atol=1e-4)
    multi_tensor.zero_(keep[0])
    assert all((t == 0).all() for t in keep[0]) and all((t != 0).any() for ts in keep[1:] for t in ts)


def test_multi_tensor_tables_belong_to_their_stream():
    """Equal sizes on two streams, at the same and at moved addresses: no device copy is shared, a stream finds its own
    table again, and moved tensors share the sizes of their own stream's table only."""
    from torchure_b200.ops import multi_tensor

    new = lambda: [torch.zeros(n, device="cuda") for n in (7, 40000)]
    first, moved = new(), new()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    here = multi_tensor._table("streams", [first])
    with torch.cuda.stream(side):
        there = multi_tensor._table("streams", [first])
        there_moved = multi_tensor._table("streams", [moved])
        assert multi_tensor._table("streams", [moved]) is there_moved
    assert multi_tensor._table("streams", [first]) is here
    here_moved = multi_tensor._table("streams", [moved])
    copies = lambda tabs: {t.data_ptr() for tab in tabs for t in tab.args()}
    assert not copies([here, here_moved]) & copies([there, there_moved])
    assert here_moved.bt is here.bt and there_moved.bt is there.bt
    torch.cuda.synchronize()


def test_multi_tensor_tables_of_a_capture():
    """A captured step and calls around it on the same and on moved tensors: neither uses the other's tables, replays read
    host bytes that nobody else has been given meanwhile, and these go with the graph."""
    import gc
    import time

    from torchure_b200 import ops
    from torchure_b200.ops import multi_tensor

    sizes = (5, 40000)
    new = lambda v: [torch.full((n,), v, device="cuda") for n in sizes]
    factor = lambda v: torch.tensor(v, device="cuda")
    half, two, one = factor(0.5), factor(2.0), factor(1.0)
    start = ops.ext().graph_keeps()
    a = new(8.0)
    eager = multi_tensor._table("scale", [a], [0, 0])        # a table of these addresses is there before the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        inside = multi_tensor._table("scale", [a], [0, 0])
        multi_tensor.scale_(a, half)
        norm = multi_tensor.sq_norm(a)
        assert multi_tensor._table("scale", [a], [0, 0]) is inside
    assert inside is not eager and multi_tensor._table("scale", [a], [0, 0]) is eager
    assert ops.ext().graph_keeps() == start + 2
    staging = {t.data_ptr() for t in inside.host()}
    b = new(3.0)
    multi_tensor.scale_(b, two)         # moved: replaces the eager table
    multi_tensor.scale_(a, one)         # ... and moved back, before the first replay
    del inside, eager
    multi_tensor._CAPTURES.clear()
    gc.collect()
    torch.cuda.synchronize()
    taken = [torch.zeros(n, dtype=torch.int64).pin_memory() for n in (2, 10) for _ in range(8)]
    assert not staging & {t.data_ptr() for t in taken}
    for want in (4.0, 2.0, 1.0):
        graph.replay()
        torch.cuda.synchronize()
        assert all((t == want).all() for t in a) and all((t == 6.0).all() for t in b)
        assert norm.item() == want * want * sum(sizes)
    graph.reset()
    del graph
    torch.cuda.synchronize()
    for _ in range(200):                # CUDA calls back from a thread of its own
        if ops.ext().graph_keeps() == start:
            break
        time.sleep(0.01)
    assert ops.ext().graph_keeps() == start


def test_bucket_pack():
    from torchure_b200.ops import multi_tensor

    torch.manual_seed(0)
    shapes = [(512, 512), (128,), (30000,)]
    grads = [torch.randn(s, device="cuda") for s in shapes]
    grads[0] = grads[0].bfloat16()
    flat = torch.full((sum(g.numel() for g in grads),), 7.0, device="cuda")
    views, at = [], 0
    for g in grads:
        views.append(flat[at:at + g.numel()].view(g.shape))
        at += g.numel()
    sq = torch.zeros((), device="cuda")
    multi_tensor.bucket_pack(grads, views, False, 1.0, sq)
    want = torch.cat([g.float().flatten() for g in grads])
    torch.testing.assert_close(flat, want)
    torch.testing.assert_close(sq, want.pow(2).sum(), rtol=1e-4, atol=1e-3)
    multi_tensor.bucket_pack(grads, views, True, 0.5, None)
    torch.testing.assert_close(flat, want)  # (x + x) * 0.5


def test_poison_and_verify_mode():
    """Every wrapper output is pre-filled with NaN; a kernel that left any element unwritten would be reported."""
    from torchure_b200.models.qwen3 import RotaryEmbedding
    from torchure_b200.ops import attention, debug, kernels

    debug.enable(True)
    try:
        torch.manual_seed(0)
        M, D, Fd, S, Hq, Hkv = 300, 512, 640, 256, 4, 2   # ragged M and N: edge tiles must be covered too
        x = torch.randn(M, D, device="cuda")
        w = torch.rand(D, device="cuda") + 0.5
        _, h, rstd = kernels.add_rmsnorm(x, (torch.randn(M, D, device="cuda") * 0.1).bfloat16(), w, 1e-6)
        gu = kernels.linear_fwd(h, torch.randn(2 * Fd, D, device="cuda").bfloat16())
        act = kernels.swiglu(gu)
        kernels.swiglu_bwd(torch.randn_like(act), gu)
        kernels.linear_wgrad(torch.randn(M, 2 * Fd, device="cuda").bfloat16(), h, out_dtype=torch.float32)
        kernels.rmsnorm_bwd(torch.randn(M, D, device="cuda").bfloat16(), x, w, rstd, None, torch.zeros(D, device="cuda"))
        qkv = torch.randn(2 * S, (Hq + 2 * Hkv) * 128, device="cuda").bfloat16()
        cos, sin = RotaryEmbedding(128).tables(S, "cuda")
        qk = kernels.qknorm_rope(qkv, w[:128].clone(), w[:128].clone(), cos, sin, S, Hq, Hkv, 1e-6)
        o, state = attention.attn_fwd(qk, qkv, 2, S, Hq, Hkv, 128)
        attention.attn_bwd(torch.randn_like(o), qk, qkv, state, 2, S, Hq, Hkv, 128)
        assert debug.verify() >= 10
        # and the check itself fires: an output that no kernel writes keeps its sentinels
        debug.new_output("never_written", 8, dtype=torch.float32, device="cuda")
        with pytest.raises(RuntimeError, match="never_written"):
            debug.verify()
    finally:
        debug.enable(False)


def test_embedding_scatter_is_exact_and_repeatable():
    """Deterministic multi-source scatter-add against index_add in fp64, with repeated ids inside and across sources;
    two runs give identical bits, and the per-CTA corrections turn the old sum of squares into the new one."""
    from torchure_b200.ops import kernels as K

    torch.manual_seed(0)
    V, D, M = 5000, 1024, 3000
    srcs = []
    for p in range(3):
        ids = torch.randint(0, V, (M,), device="cuda")
        ids[::7] = 11          # a hot row, hit hundreds of times by every source
        srcs.append((ids, torch.randn(M, D, device="cuda")))
    base = torch.randn(V, D, device="cuda")
    want = base.double()
    for ids, rows in srcs:
        want.index_add_(0, ids, rows.double() * 0.25)
    outs = []
    scratch = torch.empty(3 * M, dtype=torch.int64, device="cuda")
    for use_scratch in (None, None, scratch):      # the third run scans a gathered copy of the ids
        t = base.clone()
        delta = torch.zeros(1024, device="cuda")
        K.embedding_scatter_(srcs, t, M, scale=0.25, sq_delta=delta, blocks=592, ids_scratch=use_scratch)
        outs.append(t)
        got_sq = base.double().pow(2).sum() + delta.double().sum()
        assert abs(got_sq.item() - t.double().pow(2).sum().item()) < 1e-4 * t.double().pow(2).sum().item()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    torch.testing.assert_close(outs[0].double(), want, rtol=1e-5, atol=1e-4)


def test_repeat_runs_are_bitwise_stable_under_poison():
    """Race detection for the compute kernels: the deterministic ones (GEMMs with their TMA rings and TMEM double
    buffering, the attention forward, the two-kernel attention backward, norms, RoPE, SwiGLU) must give identical bits
    on every one of many back-to-back launches while every output buffer is pre-filled with NaN; a consumer that
    outruns its producer, a stage recycled too early or a tile left unwritten shows up as a differing or NaN element."""
    from torchure_b200 import ops
    from torchure_b200.models.qwen3 import RotaryEmbedding
    from torchure_b200.ops import debug
    from torchure_b200.ops import kernels as K

    torch.manual_seed(0)
    M, D, F_, Hq, Hkv, hd, S, B = 1024, 512, 1024, 4, 2, 128, 512, 2
    x, y = torch.randn(M, D, device="cuda"), torch.randn(M, D, device="cuda").bfloat16()
    w = torch.rand(D, device="cuda") + 0.5
    h = torch.randn(M, D, device="cuda").bfloat16()
    wqkv = (torch.randn((Hq + 2 * Hkv) * hd, D, device="cuda") * 0.05).bfloat16()
    cos, sin = RotaryEmbedding(hd).tables(S, "cuda")
    gains = torch.rand(hd, device="cuda") + 0.5
    d_o = torch.randn(M, Hq * hd, device="cuda").bfloat16()

    def once():
        outs = list(K.add_rmsnorm(x, y, w, 1e-6))
        qkv = K.linear_fwd(h, wqkv)
        qk = K.qknorm_rope(qkv, gains, gains, cos, sin, S, Hq, Hkv, 1e-6, True)
        o = debug.new_output("o", M, Hq * hd, dtype=torch.bfloat16, device="cuda")
        lse = debug.new_output("lse", B, Hq, S, dtype=torch.float32, device="cuda")
        ops.ext().attn_fwd(qk, qkv, o, lse, B, S, Hq, Hkv)
        dqkv = debug.new_output("dqkv", M, (Hq + 2 * Hkv) * hd, dtype=torch.bfloat16, device="cuda")
        ops.ext().attn_bwd(d_o, qk, qkv, o, lse, dqkv, B, S, Hq, Hkv)      # the deterministic two-kernel backward
        gu = K.linear_fwd(h, torch.cat([wqkv, wqkv])[: 2 * F_])
        outs += [qkv, qk, o, lse, dqkv, K.swiglu(gu), K.linear_dgrad(qkv, wqkv),
                 K.linear_wgrad(qkv, h)]
        return outs

    debug.enable(True)
    try:
        ref = [t.clone() for t in once()]
        for rep in range(40):
            for i, (a, b) in enumerate(zip(once(), ref)):
                assert torch.equal(a, b), (rep, i)
            assert debug.verify() > 0
    finally:
        debug.enable(False)
    K.check_error()


@pytest.mark.parametrize("shared_sms", [0, 16, 148, 1000])
def test_qknorm_rope_bwd_beside_communication(shared_sms):
    """Fewer CTAs, more rows for each: the same gradients (the gains' partials are added in another order)."""
    from torchure_b200.models.qwen3 import RotaryEmbedding
    from torchure_b200.ops import kernels

    torch.manual_seed(4)
    M, Hq, Hkv, hd = 3001, 16, 8, 128
    qkv, g = (torch.randn(M, (Hq + 2 * Hkv) * hd, device="cuda").bfloat16() for _ in range(2))
    w = torch.rand(hd, device="cuda") + 0.5
    cos, sin = RotaryEmbedding(hd).tables(M, "cuda")
    outs = []
    for shared in (0, shared_sms):
        d, dq, dk = g.clone(), torch.zeros(hd, device="cuda"), torch.zeros(hd, device="cuda")
        kernels.qknorm_rope_bwd_(d, qkv, w, w, cos, sin, dq, dk, M, Hq, Hkv, 1e-6, shared_sms=shared)
        outs.append((d, dq, dk))
    assert torch.equal(outs[0][0], outs[1][0])
    # 48000 and 24000 terms in fp32, about 2^-24 x sqrt(terms) of their size
    assert relerr(outs[1][1], outs[0][1]) < 1e-4 and relerr(outs[1][2], outs[0][2]) < 1e-4


@pytest.mark.parametrize("variant", [-1, 3])
def test_qknorm_rope_bwd_refuses_variants_it_does_not_have(variant):
    from torchure_b200 import ops

    t, w, table = torch.zeros(8, 512, device="cuda").bfloat16(), torch.ones(128, device="cuda"), torch.ones(8, 128, device="cuda")
    with pytest.raises(RuntimeError, match="variant"):
        ops.ext().qknorm_rope_bwd(t, t.clone(), w, w, table, table, w.clone(), w.clone(), 8, 2, 1, 1e-6, True, None, variant)
