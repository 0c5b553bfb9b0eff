"""Steps of few tokens: products whose sixteen rows are two feature groups (up to 8 tokens), and decode attention of single query heads on the 32-bit
units."""
from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import _attention_reference, _paged_case, _rand, dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 5, 8])
@pytest.mark.parametrize("N,K", [(8, 64), (24, 1024), (39, 768), (1192, 1000), (2304, 768), (130, 4096), (1200, 2048)])
def test_products_of_up_to_eight_tokens(dev, M, N, K):
    """One group, odd numbers of groups a pass, several passes, all three reductions: against 64 bits, and the bits of the rows in a launch of sixteen."""
    from liyab_b200 import ops
    a, w, bias = _rand((16, K), 80, dev, torch.bfloat16), _rand((N, K), 81, dev, torch.bfloat16, 0.1), _rand((N,), 82, dev)
    out, whole = (torch.empty((m, N), dtype=torch.float32, device=dev) for m in (M, 16))
    ops.gemm_rows(a[:M], w, bias, out, M)
    ops.gemm_rows(a, w, bias, whole, 16)
    assert torch.equal(out, whole[:M])
    # Sums of K products in eight chains (K / 8 roundings each), and the bias.
    bound = (K / 8 + 16) * 2.0 ** -24 * (a[:M].double().abs() @ w.double().abs().t() + bias.double().abs())
    assert ((out.double() - (a[:M].double() @ w.double().t() + bias.double())).abs() <= bound).all()


@pytest.mark.parametrize("window,splits", [(0, 1), (0, 3), (0, 12), (50, 2)])
@pytest.mark.parametrize("n_head,page_size,n_seq", [(3, 16, 9), (25, 32, 3), (70, 16, 9)])
def test_decode_attention_of_single_heads(dev, n_head, page_size, n_seq, window, splits):
    """Contexts that end in every part of a tile; a key that outweighs the others makes the maximum move late."""
    from liyab_b200 import ops
    lens, scale = [1, 15, 16, 17, 31, 250, 511, 700, 1024][-n_seq:], 0.125
    q, cache, _, positions, table, refs = _paged_case(dev, torch.bfloat16, n_head, n_head, 64, page_size, lens, [1] * n_seq, seed=splits + n_head, boost=(240, 4.0))
    partial = torch.full((n_seq * n_head * splits * 66,), float("nan"), device=dev)
    counters = torch.zeros(n_seq * n_head, dtype=torch.int32, device=dev)
    out = torch.full_like(q, float("nan"))
    ops.decode_attention(q, cache, positions, table, out, partial, counters, n_seq, n_head, n_head, 64, page_size, scale, window, splits, tensor_cores=True)
    ref = _attention_reference(refs, n_head, n_head, scale, window)
    # 32-bit weights and sums of up to 1024 values of order one (a rounding each), and the result in bfloat16.
    assert ((out.double().cpu() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1024 * 2.0 ** -23 * 4).all() and int(counters.abs().sum()) == 0


@pytest.mark.parametrize("n_head,n_seq,splits,max_keys", [
    (25, 9, 1, 0), (25, 16, 1, 0), (16, 32, 1, 0), (12, 64, 1, 0), (25, 48, 1, 0), (16, 96, 1, 0), (24, 80, 1, 0),         # two to thirteen pairs an SM
    (25, 8, 2, 0), (12, 8, 4, 0), (12, 8, 4, 5000), (3, 9, 8, 5000)])                                                        # wide blocks, and ranges in a cluster
def test_decode_attention_of_many_single_heads(dev, n_head, n_seq, splits, max_keys):
    """Every form that the number of pairs chooses: tiles ahead, blocks held to an SM's share of them, blocks of two warps."""
    from liyab_b200 import ops
    lens, scale = ([1, 15, 16, 17, 31, 100, 250, 33, 600] * 11)[:n_seq], 0.125
    q, cache, _, positions, table, refs = _paged_case(dev, torch.bfloat16, n_head, n_head, 64, 16, lens, [1] * n_seq, seed=n_seq, boost=(28, 4.0))
    partial = torch.full((n_seq * n_head * splits * 66,), float("nan"), device=dev)
    counters = torch.zeros(n_seq * n_head, dtype=torch.int32, device=dev)
    out = torch.full_like(q, float("nan"))
    ops.decode_attention(q, cache, positions, table, out, partial, counters, n_seq, n_head, n_head, 64, 16, scale, 0, splits, tensor_cores=True, max_keys=max_keys)
    ref = _attention_reference(refs, n_head, n_head, scale, 0)
    assert ((out.double().cpu() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1024 * 2.0 ** -23 * 4).all() and int(counters.abs().sum()) == 0
    assert ops.device_status() == 0
