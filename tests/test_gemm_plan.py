"""The choice of a kernel for a product (``gemm_plan``), which needs no GPU."""

import subprocess
import sys

import pytest

from torchure_b200 import ops

_C = ops.ext()
pytestmark = pytest.mark.skipif(_C is None, reason="the CUDA extension is not built")

ceil_div = lambda a, b: -(-a // b)
SIZES = [(600, 512, 50257), (130, 64, 151936), (300, 520, 2500), (129, 128, 16384), (256, 256, 4096), (1, 8, 520),
         (128, 1024, 151936), (8192, 1024, 3072)]


@pytest.mark.parametrize("M,N,K", SIZES)
def test_transposed_a_with_row_major_b_is_not_sliced(M, N, K):
    """A [K, M] with B [N, K] exists with bf16 output only: slices of K, which are fp32 products, cannot run it."""
    assert _C.gemm_plan(M, N, K, a_mn=True, b_mn=False, may_split=True)[0] != "slices"


def test_empty_products_are_planned():
    """A size of zero is left to the launcher's argument check (an integer division by zero would end the process, hence
    the child)."""
    code = ("from torchure_b200 import _C\n"
            "for M, N, K in ((256, 0, 8192), (0, 256, 8192), (256, 256, 0), (0, 0, 0), (256, 0, 32768)):\n"
            "    for mode in (0, 1, 2):\n"
            "        kind, _, splits, ws = _C.gemm_plan(M, N, K, out_mode=mode)\n"
            "        assert splits == 1 and ws == 0 and kind != 'slices'\n")
    res = subprocess.run([sys.executable, "-c", "import torch\n" + code], capture_output=True, text=True, timeout=240)
    assert res.returncode == 0, (res.returncode, res.stderr[-500:])


@pytest.mark.parametrize("free", [16, 40, 100])
def test_reserved_sms_stay_free(free):
    """With SMs reserved no product starts more CTAs than the others hold: the kernel for few tiles is not persistent, so its
    tiles have to fit at once (the other kernels take the number of SMs they may use)."""
    sms = 148 - free
    two_waves = 0
    for m in (1, 100, 128, 300, 1024, 1408, 2048, 2304, 4096):
        for n in (64, 512, 1024, 2048, 3072, 6144):
            for k in (64, 512, 4096, 20000):
                for mode in (0, 1):
                    def ctas(**kw):
                        kind, tile, splits, _ = _C.gemm_plan(m, n, k, out_mode=mode, may_split=True, **kw)
                        return -(-m // 128) * -(-n // tile) * splits if kind == "small" else 0
                    assert ctas(num_sms=sms, sms_reserved=True) <= sms, (m, n, k, mode)
                    two_waves += ctas(num_sms=sms) > sms
    assert two_waves > 0


@pytest.mark.parametrize("K", [512, 4096, 16384, 19456, 28672])
@pytest.mark.parametrize("N", [64, 1024, 2048, 2560])
def test_bf16_products_are_split_only_on_request(N, K):
    """A block's product (2 ffn_dim of the input gradient, ffn_dim of the down projection) keeps one order of additions for
    any number of rows; a head's may be split."""
    for M in (1, 128, 129, 256, 600, 1024, 4096):
        assert _C.gemm_plan(M, N, K, b_mn=True)[2] == 1, M


def test_head_products_are_split():
    assert _C.gemm_plan(600, 512, 50257, b_mn=True, may_split=True)[2] > 1
    assert _C.gemm_plan(128, 1024, 151936, b_mn=True, may_split=True)[2] > 1
    assert _C.gemm_plan(600, 512, 8192, b_mn=True, may_split=True)[2] == 1


def test_clusters_of_a_plan_run_at_once():
    """Clusters of 4 and 8 CTAs do not fill every SM: 33 and 15 of them are resident on 148 SMs.  A problem that the few-tile
    kernel could take in one wave of some form is not given to it in two waves of clusters."""
    for m in (128, 256, 512, 1024, 2048):
        for n in (64, 128, 256, 512, 1024):
            for k in (2048, 4096, 8192, 16384, 65536):
                for mode in (1, 2):
                    kind, tile, splits, _ = _C.gemm_plan(m, n, k, a_mn=True, b_mn=True, out_mode=mode)
                    if kind == "small" and splits >= 4:
                        assert -(-m // 128) * -(-n // tile) <= {4: 33, 8: 15}[splits], (m, n, k, mode)


@pytest.mark.parametrize("M,F,K,pays", [(8192, 8192, 2048, True), (4096, 9728, 2560, True), (2048, 9728, 2560, True),
                                        (8192, 2048, 2048, True), (8192, 3072, 1024, False), (2048, 3072, 2048, False),
                                        (512, 9728, 2560, False), (1408, 9728, 2560, False), (256, 9728, 4096, False)])
def test_swiglu_gradient_is_fused_where_it_pays(M, F, K, pays):
    """Long products with enough tiles that the last wave's epilogue, which nothing hides, does not decide."""
    assert _C.gemm_swiglu_bwd_pays(M, F, K, 148) == pays


def test_fp32_products_keep_their_slices_short():
    """The tensor core's fp32 sums lose precision with every term: whichever kernel an fp32 product runs on, its slices of K
    are no longer than those of the split by reduce-add, which gives SM pairs (SMs, up to 128 rows) the least wave time."""
    for m in (64, 128, 256, 512, 1024, 3072, 8192):
        for n in (64, 256, 512, 1024, 2560, 9728):
            for k in (128, 600, 1024, 2048, 4224, 8192, 16384, 50257):
                tile_m, workers = (256, 74) if m > 128 else (128, 148)
                tiles, blocks = ceil_div(m, tile_m) * ceil_div(n, 256), ceil_div(k, 64)
                longest = blocks
                if blocks >= 32 and tiles < 2 * workers:
                    # fp32 arithmetic of the plan: ties within 1e-6 go to fewer slices
                    cost = lambda s: ceil_div(tiles * s, workers) / s + 0.02 * (s - 1)
                    best = min(range(1, min(8, blocks // 8) + 1), key=lambda s: (round(cost(s), 5), s))
                    longest = ceil_div(blocks, best)
                for mode in (1, 2):
                    _, _, splits, _ = _C.gemm_plan(m, n, k, a_mn=True, b_mn=True, out_mode=mode)
                    assert ceil_div(blocks, splits) <= longest, (m, n, k, mode)


@pytest.mark.parametrize("M,N,K", [(4096, 2560, 151936), (2816, 1024, 151936), (4096, 1024, 151936), (8192, 4096, 151936),
                                   (16384, 8192, 151936), (4096, 2560, 9728)])
def test_slices_that_fill_the_waves(M, N, K):
    """A head's dH with many tiles is sliced where the waves are partly empty: within 256 MB, without an empty slice, and on
    request only."""
    assert _C.gemm_plan(M, N, K, b_mn=True)[0] != "slices"
    kind, _, splits, ws = _C.gemm_plan(M, N, K, b_mn=True, may_split=True)
    if kind == "slices":
        assert 1 < splits <= 8 and ws <= 256 << 20
        per = ceil_div(ceil_div(K, 64), splits)
        assert (splits - 1) * per < ceil_div(K, 64)
    assert (kind == "slices") == ((M, N) in ((4096, 2560), (2816, 1024)) and K > 65536)


@pytest.mark.parametrize("weight", [1 << 20, 1 << 28])
def test_chunks_of_the_loss_head(weight):
    """At most ``chunk_size`` rows, no more chunks than it asks for, every row in one; 4097 rows in two chunks of about half."""
    from torchure_b200.ops.linear_ce import _chunk_rows

    for chunk in (1, 100, 255, 256, 257, 512, 600, 1000, 1024, 4096, 10000):
        for n in [1, 2, 127, 128, 129, 255, 256, 257, 511, 513, 600, 1100, 1531, 4096, 4097, 4224, 8192, 30000]:
            rows = _chunk_rows(n, chunk, weight)
            assert 0 < rows <= min(chunk, n) or (rows == chunk and n > chunk), (n, chunk, rows)
            assert ceil_div(n, rows) <= ceil_div(n, chunk), (n, chunk, rows)
    assert _chunk_rows(4097, 4096, 1 << 28) == 2304 and _chunk_rows(1531, 600, 1 << 28) == 512
    assert _chunk_rows(1100, 1000, 1 << 20) == 1000 and _chunk_rows(8192, 4096, 1 << 28) == 4096


def test_chunks_of_a_sharded_loss_head(monkeypatch):
    """With the vocabulary sharded, the products and dW of a chunk cover the rank's rows only: their size decides."""
    import torch

    from torchure_b200.ops import linear_ce

    class Mesh:
        def size(self, dim):
            return 4

        def coordinate(self, dim):
            return 1

    class Seen(Exception):
        pass

    def record(rows, chunk, weight_elements):
        raise Seen(weight_elements)

    monkeypatch.setattr(linear_ce, "_chunk_rows", record)
    h, w = torch.zeros(1100, 64, dtype=torch.bfloat16), torch.zeros(4000, 64, dtype=torch.bfloat16)
    y, one = torch.zeros(1100, dtype=torch.int64), torch.ones(())
    for shard, elements in ((None, 4000 * 64), ((Mesh(), "tp"), 1000 * 64)):
        with pytest.raises(Seen, match=f"^{elements}$"):
            linear_ce._LinearCESm100.apply(h, w, y, -100, 1000, w, None, 1.0, None, one, shard, True)


def test_chunks_that_are_said_to_change():
    """The shapes whose times the rule quotes: it changes those that it is said to speed up, and no others."""
    from torchure_b200.ops.linear_ce import _chunk_rows

    for rows, dim, vocab, chunk, got in ((4224, 1024, 151936, 4096, 2304), (4224, 2048, 128256, 4096, 2304), (4097, 512, 50257, 4096, 2304),
                                         (1531, 512, 50257, 600, 512), (5000, 1024, 100000, 4096, 2560)):
        assert _chunk_rows(rows, chunk, dim * vocab) == got < min(chunk, rows)
    for rows, dim, vocab, chunk in ((3500, 512, 20000, 512), (3000, 2048, 60000, 1000), (1100, 512, 30000, 1000)):
        assert _chunk_rows(rows, chunk, dim * vocab) == chunk
