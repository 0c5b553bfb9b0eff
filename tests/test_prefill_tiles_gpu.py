"""The tcgen05 prefill attention at the edges of its warps and tiles: portions that fill a part of a tile's warps on contexts of several key
tiles (where warps without rows run ahead of the others), and more requests than one look finds."""
from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import _paged_case, _rand, dev  # noqa: F401

pytestmark = pytest.mark.gpu

EDGES = ([1, 31, 32, 33, 64, 65, 96, 97, 127, 128, 129, 255, 257], [0, 700, 97, 513, 384, 1, 300, 640, 128, 127, 900, 5, 250])
MANY = ([(7 * i) % 40 + 1 + (130 if i % 33 == 0 else 0) for i in range(70)], [(37 * i) % 300 for i in range(70)])


@pytest.mark.parametrize("soft_cap", [0.0, 20.0])
@pytest.mark.parametrize("window", [0, 200])
@pytest.mark.parametrize("new,past,n_head,n_kv_head", [(*EDGES, 3, 3), (*MANY, 4, 2)])
def test_portions_at_the_edges(dev, new, past, n_head, n_kv_head, window, soft_cap):
    from liyab_b200 import ops
    head_dim, page_size, S = 64, 16, len(new)
    q, cache, tok_seq, positions, table, _ = _paged_case(dev, torch.bfloat16, n_head, n_kv_head, head_dim, page_size, [p + n for p, n in zip(past, new)], new,
                                                         seed=S + window)
    starts = torch.tensor([sum(new[:i]) for i in range(S + 1)], dtype=torch.int32, device=dev)
    held = torch.tensor(past, dtype=torch.int32, device=dev)
    sink = _rand((n_head,), 5, dev)
    want = torch.empty_like(q)
    ops.paged_attention_generic(q, cache, tok_seq, positions, table, want, q.shape[0], n_head, n_kv_head, head_dim, page_size, 0.125, window, sink=sink,
                                soft_cap=soft_cap)
    for min_len in (1, 2, 40):
        served = torch.tensor([n >= min_len for n in new for _ in range(n)], device=dev)
        for _ in range(3):
            out = torch.full_like(q, 7.0)
            ops.prefill_attention(q, cache, starts, held, table, out, S, max(new), n_head, n_kv_head, head_dim, page_size, 0.125, window, tcgen05=True, sink=sink,
                                  soft_cap=soft_cap, min_len=min_len)
            assert ops.device_status() == 0
            # Weights and the result in bfloat16 (2^-9 each) on values of order one, as in the kernels' own tests.
            assert (out.float() - want.float())[served].abs().max().item() < 1.5e-2
            assert (out[~served] == 7.0).all()


@pytest.mark.parametrize("soft_cap,slopes", [(0.0, False), (20.0, False), (0.0, True)])
@pytest.mark.parametrize("window", [0, 200])
@pytest.mark.parametrize("new,past", [
    ([1, 300, 1, 1, 45, 1, 1, 1], [0, 20, 15, 16, 700, 512, 1, 930]),
    ([1] * 40 + [200] + [1] * 37, [(53 * i) % 900 for i in range(78)])])
def test_single_tokens_in_the_launch(dev, new, past, window, soft_cap, slopes):
    """Contexts that end in every part of a tile and fill some warps or all, more requests than one look finds, beside a portion."""
    from liyab_b200 import ops
    n_head, page_size, S = 5, 16, len(new)
    q, cache, tok_seq, positions, table, _ = _paged_case(dev, torch.bfloat16, n_head, n_head, 64, page_size, [p + n for p, n in zip(past, new)], new, seed=S + window)
    starts = torch.tensor([sum(new[:i]) for i in range(S + 1)], dtype=torch.int32, device=dev)
    held = torch.tensor(past, dtype=torch.int32, device=dev)
    sink = _rand((n_head,), 6, dev)
    distance = torch.cat([_rand((n_head,), 7, dev).abs() * 0.1, torch.full((n_head,), -1.0, device=dev)]) if slopes else None
    want, out = torch.empty_like(q), torch.full_like(q, float("nan"))
    ops.paged_attention_generic(q, cache, tok_seq, positions, table, want, q.shape[0], n_head, n_head, 64, page_size, 0.125, window, sink=sink, soft_cap=soft_cap,
                                distance=distance)
    ops.prefill_attention(q, cache, starts, held, table, out, S, max(new), n_head, n_head, 64, page_size, 0.125, window, tcgen05=True, sink=sink, soft_cap=soft_cap,
                          distance=distance, min_len=2, singles=True)
    assert ops.device_status() == 0
    # As above; the single tokens' weights stay in 32 bits, their result has one rounding.
    assert (out.float() - want.float()).abs().max().item() < 1.5e-2
