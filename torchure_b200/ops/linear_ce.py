"""Chunked fused linear + cross-entropy on sm_100a kernels.

Per chunk of at most ``chunk_size`` rows (``_chunk_rows``; reference algorithm: ``torchure/loss/fused_linear_ce.py:31-93``):

1. ``logits = h_chunk @ W^T``         tcgen05 GEMM, bf16 out (the only (chunk, V) buffer, reused by every chunk)
2. ``ce_softmax_grad``                one kernel: online max/sum, target gather, per-row loss and, in place,
                                      ``dlogits = (softmax - onehot) / n_valid`` in bf16 (zero for ignored rows)
3. ``dH_chunk = dlogits @ W``         tcgen05 GEMM, B operand read MN-major
4. ``dW (+)= dlogits^T @ h_chunk``    tcgen05 GEMM with fp32 output; the first chunk stores, later chunks
                                      accumulate through TMA reduce-add, so there is no separate ``+=`` pass

With the vocabulary sharded over a tensor-parallel axis (``vocab_parallel``) every rank runs steps 1, 3 and 4 on its
V/n rows of the head, and step 2 becomes ``ce_row_stats`` (row maximum, sum of exponentials, target logit of the
rank's columns), two all-reduces over (chunk,)-sized fp32 vectors (maxima; rescaled sums packed with the target
logits) and ``ce_grad_from_lse``; ``dH`` is summed over the axis once after the loop.

Without gradients (``no_grad``, or neither input requires one) steps 3 and 4 fall away, step 1 leaves only the rows'
softmax statistics and label logits (``gemm_ce``) and step 2 combines them; a chunk too small for the CTA-pair kernel
stores its logits and runs ``ce_loss`` over them.

``n_valid`` is counted on the device before the loop, so the mean is folded into step 2 and backward only has
to multiply by the incoming gradient, which a conditional kernel skips when it is exactly 1.
"""

from __future__ import annotations

import torch

from torchure_b200.ops import kernels as K

BF16 = torch.bfloat16


def _chunk_rows(N: int, chunk_size: int, weight_elements: int) -> int:
    """Rows per chunk: as many chunks as ``chunk_size`` asks for, of about equal size, in whole 256-row tiles of the products where
    such a size is no larger than ``chunk_size`` (3000 rows in chunks of at most 1000 stay three of 1000).

    A short last chunk costs nearly what a whole one does, since dW is read and written for it, and ragged ones run tiles that are
    partly empty.  Measured on B200 with only this rule switched, loss head forward and backward, rows x dim x vocabulary (chunk
    size), ``chunk_size`` as it is -> this rule, medians of two runs in us: 4224 x 1024 x 151936 (4096) 4053 -> 3790, 4216 -> 3913;
    4224 x 2048 x 128256 (4096) 6630 -> 5934, 6602 -> 5881; 4097 x 512 x 50257 (4096) 1317 -> 1171, 1096 -> 912; 1531 x 512 x 50257
    (600) 807 -> 760, 745 -> 704; 5000 x 1024 x 100000 (4096), whose last chunk is not that short, 3135 -> 3112, 3416 -> 3262, within
    their spread.  A last chunk of at most 128 rows, which has a kernel of its own, stays where dW (``weight_elements``, this rank's
    in a sharded head) fits the cache (64 MB): 1100 x 512 x 30000 (1000) 252, 258 in equal ones.
    """
    if N <= 0 or chunk_size <= 0:       # refused by the loop over the chunks
        return min(chunk_size, N)
    if 0 < N % chunk_size <= 128 and N > chunk_size and weight_elements <= 1 << 24:
        return chunk_size
    per = -(-N // -(-N // chunk_size))
    per = (per + 255) // 256 * 256
    return min(per if per <= chunk_size else chunk_size, N)


class _LinearCESm100(torch.autograd.Function):
    @staticmethod
    def forward(ctx, hidden, weight, labels, ignore_index, chunk_size, w_bf16, engine, loss_scale, sink_dest,
                normalizer=None, vocab_parallel=None, want_grad=True):
        N, D = hidden.shape
        V_all = w_bf16.shape[0]   # a sharded strategy may have released the fp32 weight's own storage
        v0, V = 0, V_all
        if vocab_parallel is not None:
            # loss-parallel: this rank's logits cover rows [v0, v0 + V) of the head; steps 1, 3 and 4 run on that
            # slice, step 2 becomes statistics -> two small all-reduces -> gradient (see the module docstring)
            from torchure_b200.core.collective import all_reduce
            from torchure_b200.loss.fused_linear_ce import vocab_slice

            v0, V = vocab_slice(V_all, *vocab_parallel)
            w_bf16 = w_bf16[v0:v0 + V]
        dev = hidden.device
        h = hidden if hidden.dtype == BF16 else hidden.to(BF16)
        h, labels = h.contiguous(), labels.contiguous()
        if normalizer is None:
            inv_n = K.ce_inverse_count(labels, ignore_index, loss_scale)
        else:
            inv_n = (loss_scale / normalizer.to(dev).float()).reshape(1)      # read by kernels: a count kept on the host too
        row_loss = torch.empty(N, dtype=torch.float32, device=dev)
        # under no_grad the parameter still counts as an input that needs a gradient; nothing will ever ask for it
        need_dh = want_grad and ctx.needs_input_grad[0]
        need_dw = want_grad and ctx.needs_input_grad[1]
        d_hidden = torch.empty(N, D, dtype=BF16, device=dev) if need_dh else None
        acc0 = False
        if need_dw and sink_dest is not None:
            d_weight, acc0 = sink_dest  # the fused DDP bucket slice of the weight: written in place
        else:
            d_weight = torch.empty(V_all, D, dtype=torch.float32, device=dev) if need_dw else None
        d_weight_all = d_weight
        if vocab_parallel is not None and need_dw:
            if not acc0:    # rows of the other ranks' slices: zero here, filled by the caller's gather over the axis
                d_weight[:v0].zero_()
                d_weight[v0 + V:].zero_()
            d_weight = d_weight[v0:v0 + V]
        chunk = _chunk_rows(N, chunk_size, V * D)      # equal slices of the vocabulary: every rank has the same chunks
        ldl = (V + 7) // 8 * 8
        logits_buf = None       # allocated by the first chunk that keeps its logits
        target = torch.empty(chunk, dtype=torch.float32, device=dev) if not (need_dh or need_dw) else None
        for lo in range(0, N, chunk):
            hi = min(N, lo + chunk)
            hc = h[lo:hi]
            if target is not None and vocab_parallel is None:
                tiles = K.gemm_ce(hc, w_bf16, labels[lo:hi], target[: hi - lo])
                if tiles is not None:       # the logits never leave the chip
                    K.ce_loss_tiles(tiles, target, labels[lo:hi], row_loss[lo:hi], V, ignore_index)
                    continue
            if logits_buf is None:
                logits_buf = torch.empty(chunk, ldl, dtype=BF16, device=dev)
            logits = logits_buf[: hi - lo, :V]
            K.gemm(hc, w_bf16, out=logits)
            if vocab_parallel is None and target is not None:
                K.ce_loss(logits, labels[lo:hi], row_loss[lo:hi], ignore_index)
            elif vocab_parallel is None:
                K.ce_softmax_grad_(logits, labels[lo:hi], row_loss[lo:hi], inv_n, ignore_index)
            else:
                yc = labels[lo:hi]
                stats = torch.empty(3, hi - lo, dtype=torch.float32, device=dev)
                K.ce_row_stats_(logits, yc, stats, v0, ignore_index)
                mx = stats[0].clone()
                all_reduce(mx, *vocab_parallel, "max")
                packed = torch.stack([stats[1] * torch.exp(stats[0] - mx), stats[2]])
                all_reduce(packed, *vocab_parallel, "sum")
                lse = mx + torch.log(packed[0])
                row_loss[lo:hi] = torch.where(yc != ignore_index, lse - packed[1], torch.zeros_like(lse))
                if need_dh or need_dw:
                    K.ce_grad_from_lse_(logits, yc, lse, inv_n, v0, ignore_index)
            if need_dh:
                K.gemm(logits, w_bf16, b_mn=True, out=d_hidden[lo:hi], may_split=True)
            if need_dw:
                K.gemm(logits, hc, a_mn=True, b_mn=True, out=d_weight, accumulate=acc0 or lo > 0)
        if vocab_parallel is not None and need_dh:
            all_reduce(d_hidden, *vocab_parallel, "sum")     # each rank contributed its vocabulary rows
        loss = K.ce_mean(row_loss, inv_n)
        ctx.stash = (d_hidden, d_weight_all)
        ctx.engine = engine
        ctx.in_sink = sink_dest is not None
        ctx.hidden_dtype = hidden.dtype
        return loss

    @staticmethod
    def backward(ctx, grad_out):
        if ctx.stash is None:
            raise RuntimeError("fused_linear_cross_entropy: backward ran twice; its grads are consumed in place")
        d_hidden, d_weight = ctx.stash
        ctx.stash = None
        scale = grad_out.float().reshape(1)
        if d_hidden is not None:
            K.scale_inplace_(d_hidden, scale)
            if ctx.hidden_dtype != BF16:
                d_hidden = d_hidden.to(ctx.hidden_dtype)
        if d_weight is not None:
            if not ctx.in_sink:  # a sink slice may hold earlier micro-batches: the loss must be the root there
                K.scale_inplace_(d_weight, scale)
            eng = ctx.engine
            if eng is not None and eng.expect_tied_grad:
                eng.expect_tied_grad = False
                sink = eng.model._grad_sink
                head = eng.model.lm_head.weight
                if ctx.in_sink and hasattr(sink, "early_table") and sink.early_table(head):
                    # tied embedding under DDP: the dense part of the gradient is complete, reduce it now (under the
                    # whole block backward); the embedding rows are exchanged when the gather's backward has them
                    from torchure_b200.ops.block import EARLY_TABLE

                    sink.grad_written(head)
                    eng.pending_tied_grad = EARLY_TABLE
                else:
                    # hand the buffer to the gather's backward, which adds its rows and returns it
                    eng.pending_tied_grad = d_weight
                d_weight = None
            elif ctx.in_sink:
                eng.model._grad_sink.grad_written(eng.model.lm_head.weight)
                d_weight = None
        return d_hidden, d_weight, None, None, None, None, None, None, None, None, None, None


def linear_ce_sm100(hidden, weight, labels, ignore_index, chunk_size, loss_scale=1.0, normalizer=None,
                    vocab_parallel=None):
    from torchure_b200.ops.block import engine_for_weight

    eng = engine_for_weight(weight)
    sink_dest = None
    if eng is not None:
        eng.refresh()
        w_bf16 = eng.head_shadow
        sink = eng.model._grad_sink
        if sink is not None and weight.requires_grad and torch.is_grad_enabled():
            sink_dest = sink.grad_dest(weight)
    else:
        w_bf16 = K.cast_to_bf16(weight.detach().contiguous()) if weight.dtype != BF16 else weight.detach()
    return _LinearCESm100.apply(hidden, weight, labels, ignore_index, chunk_size, w_bf16, eng, float(loss_scale),
                                sink_dest, normalizer, vocab_parallel, torch.is_grad_enabled())
