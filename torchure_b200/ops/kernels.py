"""Thin Python wrappers over the sm_100a kernels (allocation + launch counting); no math here.

Every function launches exactly the kernels its docstring names.  Plain PyTorch statements of the
same operations live in ``ops/oracle.py`` and are what the GPU tests compare against.
"""

from __future__ import annotations

import torch

from torchure_b200 import ops
from torchure_b200.ops import debug
from torchure_b200.ops.debug import new_output

BF16 = torch.bfloat16


def _C():
    ext = ops.ext()
    if ext is None:
        raise RuntimeError("the torchure_b200 CUDA extension is not built (python -m torchure_b200.build)")
    return ext


def check_error() -> None:
    """Synchronise and raise if any kernel recorded an expired wait."""
    word = _C().error_word()
    code = int(word[0].item())
    if code != 0:
        word.zero_()
        names = {1: "GEMM producer waited for a free stage", 2: "GEMM MMA warp waited for a full stage",
                 3: "GEMM MMA warp waited for a free accumulator", 4: "GEMM epilogue waited for an accumulator",
                 5: "a collective waited for a peer flag", 6: "attention pipeline wait",
                 7: "a row staged into shared memory by a bulk copy never arrived"}
        raise RuntimeError(f"sm_100a kernel reported an expired wait: code {code} ({names.get(code, 'unknown')})")


def check_comm_error(rank: int | None = None) -> None:
    """Synchronise and raise if a collective or fused GEMM+collective kernel gave up waiting for a peer."""
    word = _C().comm_error_word()
    code = int(word[0].item())
    if code != 0:
        word.zero_()
        where = "" if rank is None else f" on rank {rank}"
        raise RuntimeError(f"a collective gave up waiting for a peer flag{where} (code {code}); its output is "
                           "incomplete and every later collective bails out until the word is cleared")


# ---- GEMM ---------------------------------------------------------------------------------------
def gemm(a: torch.Tensor, b: torch.Tensor, *, a_mn: bool = False, b_mn: bool = False, out: torch.Tensor | None = None,
         out_dtype=BF16, accumulate: bool = False, splits: int = 0, may_split: bool = False) -> torch.Tensor:
    """out[M,N] (+)= A * B^T on tcgen05 tensor cores, fp32 accumulation.

    a: [M,K] (or [K,M] when a_mn), b: [N,K] (or [K,N] when b_mn); bf16, innermost stride 1.  may_split: a bf16 product
    with few rows and a long K may be summed in slices of K, so that the rounding of a row depends on how many there are.
    """
    M = a.shape[1] if a_mn else a.shape[0]
    N = b.shape[1] if b_mn else b.shape[0]
    if out is None:
        assert not accumulate
        out = new_output("gemm", M, N, dtype=out_dtype, device=a.device)
    mode = 0 if out.dtype == BF16 else (2 if accumulate else 1)
    assert not (accumulate and out.dtype == BF16), "accumulation needs an fp32 output"
    _C().gemm(a, b, out, a_mn, b_mn, mode, splits, 0, may_split)
    ops.count_launch()
    return out


def linear_fwd(x: torch.Tensor, w: torch.Tensor, out=None) -> torch.Tensor:
    """y[M,N] = x[M,K] @ w[N,K]^T"""
    return gemm(x, w, out=out)


def linear_dgrad(dy: torch.Tensor, w: torch.Tensor, out=None, may_split: bool = False) -> torch.Tensor:
    """dx[M,K] = dy[M,N] @ w[N,K]   (w is the MN-major B operand)"""
    return gemm(dy, w, b_mn=True, out=out, may_split=may_split)


def linear_wgrad(dy: torch.Tensor, x: torch.Tensor, out=None, out_dtype=BF16, accumulate=False) -> torch.Tensor:
    """dw[N,K] = dy[M,N]^T @ x[M,K]   (both operands MN-major)"""
    return gemm(dy, x, a_mn=True, b_mn=True, out=out, out_dtype=out_dtype, accumulate=accumulate)


# ---- norms / rope / mlp -----------------------------------------------------------------------------
def add_rmsnorm(x, y, w, eps, *, ids=None, table=None, need_x_out=True):
    """(x_new, h, rstd) with x_new = x + y (or table[ids]); h = rmsnorm(x_new) * w in bf16."""
    if ids is not None:
        M, D = ids.numel(), table.shape[1]
        dev = table.device
    else:
        M, D = x.shape
        dev = x.device
    h = new_output("add_rmsnorm.h", M, D, dtype=BF16, device=dev)
    rstd = new_output("add_rmsnorm.rstd", M, dtype=torch.float32, device=dev)
    x_out = None
    if (y is not None or ids is not None) and need_x_out:
        x_out = new_output("add_rmsnorm.x_out", M, D, dtype=torch.float32, device=dev)
    _C().add_rmsnorm_fwd(x, y, ids, table, w, x_out, h, rstd, eps)
    ops.count_launch()
    return (x_out if x_out is not None else x), h, rstd


def rmsnorm_bwd(dh, x, w, rstd, dx_in, dw, want_bf16=True, dx_out=None):
    """dx = dx_in + d rmsnorm(x)^T dh (fp32), optional bf16 copy; dw += sum_rows(dh * xhat).  `dx_out`: caller-owned
    destination of dx (a symmetric buffer the peers will read)."""
    dx = dx_out if dx_out is not None else new_output("rmsnorm_bwd.dx", x.shape, dtype=x.dtype, device=x.device)
    dxb = new_output("rmsnorm_bwd.dx_bf16", x.shape, dtype=BF16, device=x.device) if want_bf16 else None
    _C().rmsnorm_bwd(dh, x, w, rstd, dx_in, dx, dxb, dw)
    ops.count_launch()
    return dx, dxb


def qknorm_rope(qkv, qw, kw, cos, sin, S, Hq, Hkv, eps, use_norm=True):
    out = new_output("qknorm_rope", qkv.shape[0], (Hq + Hkv) * 128, dtype=BF16, device=qkv.device)
    _C().qknorm_rope_fwd(qkv, qw, kw, cos, sin, out, S, Hq, Hkv, eps, use_norm)
    ops.count_launch()
    return out


def qknorm_rope_bwd_(dqkv, qkv, qw, kw, cos, sin, dqw, dkw, S, Hq, Hkv, eps, use_norm=True, dq_acc=None, shared_sms=0):
    """In place on the q / k columns of dqkv.  `dq_acc` (fp32 [B, Hq, S, 128]): dq is read from there instead of the
    q columns (what the single-pass attention backward leaves behind), saving its conversion pass.  `shared_sms`: SMs that
    CTAs of a communication kernel may be on meanwhile."""
    _C().qknorm_rope_bwd(dqkv, qkv, qw, kw, cos, sin, dqw, dkw, S, Hq, Hkv, eps, use_norm, dq_acc, 0, shared_sms)
    ops.count_launch()
    return dqkv


def swiglu(gu):
    act = new_output("swiglu", gu.shape[0], gu.shape[1] // 2, dtype=BF16, device=gu.device)
    _C().swiglu_fwd(gu, act)
    ops.count_launch()
    return act


def linear_swiglu(x, w, want_gu=True):
    """(gu, act) with gu = x @ w^T (w [2F, K] = gate rows | up rows) and act = silu(gate) * up: one kernel where the product
    runs on CTA pairs, the product and a pass over it otherwise.  gu is None when it is not wanted (no backward pass)."""
    M, F = x.shape[0], w.shape[0] // 2
    act = new_output("linear_swiglu.act", M, F, dtype=BF16, device=x.device)
    gu = new_output("linear_swiglu.gu", M, 2 * F, dtype=BF16, device=x.device) if want_gu else None
    if _C().gemm_swiglu(x, w, gu, act):
        ops.count_launch()
        return gu, act
    gu = gemm(x, w, out=gu)
    _C().swiglu_fwd(gu, act)
    ops.count_launch()
    return gu if want_gu else None, act


def swiglu_bwd(dact, gu):
    dgu = new_output("swiglu_bwd", gu.shape, dtype=gu.dtype, device=gu.device)
    _C().swiglu_bwd(dact, gu, dgu)
    ops.count_launch()
    return dgu


def swiglu_dgrad(dy, w, gu):
    """d(gate) | d(up) [M, 2F] from dy [M, K], the down projection w [K, F] and the stored gu: one kernel where the product
    d(act) = dy @ w runs on CTA pairs with a long k loop, the product and a pass over it otherwise."""
    dgu = new_output("swiglu_dgrad", gu.shape, dtype=gu.dtype, device=gu.device)
    if _C().gemm_swiglu_bwd(dy, w, gu, dgu):
        ops.count_launch()
        return dgu
    _C().swiglu_bwd(linear_dgrad(dy, w), gu, dgu)
    ops.count_launch()
    return dgu


def embedding_bwd_(dx, ids, dtable):
    _C().embedding_bwd(dx, ids, dtable)
    ops.count_launch()
    return dtable


def embedding_scatter_(sources, dtable, M, scale=1.0, sq_delta=None, blocks=592, ids_scratch=None):
    """Deterministic dtable[id] += scale * rows, over `sources` = [(ids (M,) int64, rows (M, D) fp32) or
    (ids address, rows address), ...] in list order; no atomics.  Addresses let a source live on a peer GPU; then pass
    `ids_scratch` (local int64, len(sources) * M): a first kernel copies every source's ids there, because every CTA
    of the scatter scans all of them."""
    ids_ptrs = [s[0] if isinstance(s[0], int) else s[0].data_ptr() for s in sources]
    rows_ptrs = [s[1] if isinstance(s[1], int) else s[1].data_ptr() for s in sources]
    _C().embedding_scatter(ids_ptrs, rows_ptrs, dtable, M, float(scale), sq_delta, blocks, ids_scratch)
    ops.count_launch(2 if ids_scratch is not None else 1)
    return dtable


def ce_softmax_grad_(logits, labels, row_loss, inv_n_valid, ignore_index):
    _C().ce_softmax_grad(logits, labels, row_loss, inv_n_valid, ignore_index)
    ops.count_launch()


def gemm_ce(a, b, labels, target):
    """Partial softmax statistics of the rows of a @ b^T, [ceil(N / 256), M, 2] fp32 (maximum and sum of exponentials per 256
    columns), and the labels' logits in `target`; the product is not stored.  None when the problem runs on another kernel
    than the CTA-pair one (nothing was launched)."""
    stats = _C().gemm_ce(a, b, labels, target, debug.tracker())
    if stats is not None:
        ops.count_launch()
    return stats


def ce_inverse_count(labels, ignore_index, scale):
    """fp32 (1,): scale / max(1, labels that are not ``ignore_index``).  Like ``ce_mean`` not among the counted launches, which are
    those of a chunk."""
    out = new_output("ce_inverse_count", 1, dtype=torch.float32, device=labels.device)
    _C().ce_inverse_count(labels, out, ignore_index, scale)
    return out


def ce_mean(row_loss, inv_n):
    """0-dim fp32: sum(row_loss) * inv_n."""
    out = new_output("ce_mean", (), dtype=torch.float32, device=row_loss.device)     # no view: a caller may change its loss in place
    _C().ce_mean(row_loss, inv_n, out)
    return out


def ce_loss_tiles(tiles, target, labels, row_loss, vocab, ignore_index):
    """``ce_loss`` from the statistics and label logits of ``gemm_ce``."""
    _C().ce_loss_tiles(tiles, target, labels, row_loss, vocab, ignore_index)
    ops.count_launch()


def ce_loss(logits, labels, row_loss, ignore_index):
    """row_loss of ``ce_softmax_grad_`` alone; the logits are left as they are."""
    _C().ce_loss(logits, labels, row_loss, ignore_index)
    ops.count_launch()


def ce_row_stats_(logits, labels, stats, vocab_lo, ignore_index):
    """Vocabulary-sharded CE, first pass: stats (fp32 [3, rows]) <- row maximum, sum of exponentials relative to it,
    target logit (0 when the target lies outside columns [vocab_lo, vocab_lo + V))."""
    _C().ce_row_stats(logits, labels, stats, vocab_lo, ignore_index)
    ops.count_launch()


def ce_grad_from_lse_(logits, labels, lse, inv_n_valid, vocab_lo, ignore_index):
    """Second pass: logits <- (exp(logits - lse[row]) - onehot) * inv_n_valid in place, zeros for ignored rows."""
    _C().ce_grad_from_lse(logits, labels, lse, inv_n_valid, vocab_lo, ignore_index)
    ops.count_launch()


def cast_to_bf16(src, dst=None):
    if dst is None:
        dst = torch.empty(src.shape, dtype=BF16, device=src.device)
    _C().cast_to_bf16(src, dst)
    ops.count_launch()
    return dst


def scale_inplace_(x, scale):
    _C().scale_inplace(x, scale)
    ops.count_launch()
    return x
