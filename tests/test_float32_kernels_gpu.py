"""The float32 engine's kernels at the edges of their tiles: every way of cutting the work gives the same bits, and the sums are those of 64 bits
up to their rounding."""
from __future__ import annotations

import math

import pytest
import torch

from test_kernels_gpu import _attention_reference, _paged_case, _rand, dev  # noqa: F401

pytestmark = pytest.mark.gpu

# What a sum of K float32 products may be off by: chains of 64 products, then up to 32 + K / 2048 sums of sums.
EPS = 2.0 ** -24


@pytest.mark.parametrize("dtypes", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("M,N,K", [(17, 64, 64), (64, 65, 320), (65, 1, 2048), (33, 130, 2052), (80, 72, 4160), (18, 70, 77), (50, 66, 3)])
def test_tiled_products(dev, dtypes, M, N, K):
    """Tiles with remainders in every size, one to five groups a slice, groups of one to three chunks, rows that are no whole pieces."""
    from liyab_b200 import ops
    tin, tout = dtypes
    a, w, bias = _rand((M, K), 60, dev, tin), _rand((N, K), 61, dev, tin), _rand((N,), 62, dev)
    out = torch.full((M, N), float("nan"), dtype=tout, device=dev)
    ops.gemm_ffma(a, w, bias, out, M, "none")
    ref = a.double() @ w.double().t() + bias.double()
    bound = EPS * (64 + 32 + K / 2048 + 2) * (a.double().abs() @ w.double().abs().t() + bias.double().abs())
    if tout == torch.bfloat16:
        bound = bound + ref.abs() * 2.0 ** -8
    assert ((out.double() - ref).abs() <= bound).all()
    # The rows by sixteen, which another kernel multiplies where K is whole pieces: the same bits.
    for lo in range(0, M, 16):
        hi = min(M, lo + 16)
        part = torch.empty((hi - lo, N), dtype=tout, device=dev)
        ops.gemm_ffma(a[lo:hi], w, bias, part, hi - lo, "none")
        assert torch.equal(part, out[lo:hi])


@pytest.mark.parametrize("M", [9, 13, 16])
@pytest.mark.parametrize("N,K", [(1, 4), (70, 68), (17, 4160), (2367, 768), (2368, 768), (2377, 3072), (2370, 6400), (1536, 644), (2375, 260),
                                 (1541, 1000), (4738, 1024), (4740, 200)])
def test_products_of_nine_to_sixteen_rows(dev, M, N, K):
    """Sixteen features a block or eight, one chunk a group or several, remainders: the bits of eight rows and one, which another kernel multiplies."""
    from liyab_b200 import ops
    a, w, bias, res = _rand((M, K + 4), 65, dev)[:, :K], _rand((N, K), 66, dev), _rand((N,), 67, dev), _rand((M, N), 68, dev)
    out = res.clone()
    ops.gemm_ffma(a, w, bias, out, M, "none", residual=out)
    ref = a.double() @ w.double().t() + bias.double() + res.double()
    assert ((out.double() - ref).abs() <= EPS * (64 + 32 + K / 2048 + 3) * (a.double().abs() @ w.double().abs().t() + bias.double().abs() + res.double().abs())).all()
    for lo, hi in ((0, 8), (8, M), (M - 1, M)):
        part = res[lo:hi].clone()
        ops.gemm_ffma(a[lo:hi], w, bias, part, hi - lo, "none", residual=part)
        assert torch.equal(part, out[lo:hi])


@pytest.mark.parametrize("M,N,K,pad", [(40, 70, 128, 1), (40, 70, 130, 2), (70, 64, 68, 4)])
def test_tiled_products_of_strided_rows(dev, M, N, K, pad):
    """Rows that lie K + pad apart, so that they are aligned to whole pieces of four or not."""
    from liyab_b200 import ops
    a, w = _rand((M, K + pad), 63, dev)[:, :K], _rand((N, K + pad), 64, dev)[:, :K]
    out, dense = torch.empty((M, N), device=dev), torch.empty((M, N), device=dev)
    ops.gemm_ffma(a, w, None, out, M, "none")
    ops.gemm_ffma(a.contiguous(), w.contiguous(), None, dense, M, "none")
    assert torch.equal(out, dense)


@pytest.mark.parametrize("sinks", [False, True])
@pytest.mark.parametrize("n_head,n_kv_head,page_size,window,lens,q_lens", [
    (12, 12, 16, 0, [1, 15, 16, 17, 33, 300], [1, 15, 16, 17, 33, 290]),           # whole prompts, runs of every length
    (4, 2, 16, 0, [300, 77, 513, 40, 9, 260], [1, 1, 100, 1, 1, 45]),              # portions behind a past, single tokens between them
    (6, 3, 32, -48, [200, 97, 49, 48, 47], [150, 97, 1, 48, 2]),                   # chunks of 48 positions: a run ends with its chunk
    (1, 1, 8, 0, [260], [70])])
def test_runs_of_queries_agree_bit_for_bit_with_single_ones(dev, n_head, n_kv_head, page_size, window, lens, q_lens, sinks):
    from liyab_b200 import ops
    scale = 1.0 / 8.0
    q, cache, tok_seq, positions, table, refs = _paged_case(dev, torch.float32, n_head, n_kv_head, 64, page_size, lens, q_lens, seed=len(lens) + n_head)
    n, sink = q.shape[0], _rand((n_head,), 65, dev) if sinks else None
    runs, single = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    ops.paged_attention_f32_runs(q, cache, tok_seq, positions, table, runs, n, n_head, n_kv_head, page_size, scale, window, sink)
    ops.paged_attention_generic(q, cache, tok_seq, positions, table, single, n, n_head, n_kv_head, 64, page_size, scale, window, sink=sink)
    assert torch.equal(runs, single)
    if window == 0 and not sinks:
        # Float32 weights and sums: a few hundred roundings of values of order one.
        assert (runs.double().cpu() - _attention_reference(refs, n_head, n_kv_head, scale, 0)).abs().max().item() < 2e-5
