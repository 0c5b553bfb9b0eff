"""Attention of steps that mix prompt portions with single tokens: the portions by the prefill kernels, the single tokens by the decode kernel."""
from __future__ import annotations

import math

import pytest
import torch

from test_kernels_gpu import _attention_reference, _paged_case, _rand, dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tcgen05", [False, True])
@pytest.mark.parametrize("n_head,n_kv_head,page_size,window,lens,q_lens", [
    (4, 4, 16, 0, [300, 1, 77, 513, 16], [1, 1, 40, 1, 16]), (6, 2, 32, 40, [200, 129, 65, 31], [130, 1, 2, 1]), (25, 25, 16, 0, [900, 33, 640], [1, 33, 1])])
def test_portions_and_single_tokens(dev, n_head, n_kv_head, page_size, window, lens, q_lens, tcgen05):
    from liyab_b200 import ops
    scale, head_dim, S = 0.125, 64, len(lens)
    q, cache, tok_seq, positions, table, refs = _paged_case(dev, torch.bfloat16, n_head, n_kv_head, head_dim, page_size, lens, q_lens, seed=S + n_head)
    starts = torch.tensor([sum(q_lens[:i]) for i in range(S + 1)], dtype=torch.int32, device=dev)
    past = torch.tensor([l - n for l, n in zip(lens, q_lens)], dtype=torch.int32, device=dev)
    sink = _rand((n_head,), 97, dev) if n_kv_head != n_head else None
    out = torch.full_like(q, 7.0)
    ops.prefill_attention(q, cache, starts, past, table, out, S, max(q_lens), n_head, n_kv_head, head_dim, page_size, scale, window, tcgen05=tcgen05,
                          sink=sink, min_len=2)
    single = torch.tensor([n == 1 for n in q_lens for _ in range(n)], device=dev)
    assert (out[single] == 7.0).all() and (out[~single] != 7.0).any(dim=1).all()
    portions = out.clone()
    for splits in (1, 3, 12):
        partial = torch.empty(S * n_head * splits * (head_dim + 2), device=dev)
        counters = torch.zeros(S * n_kv_head, dtype=torch.int32, device=dev)
        out = portions.clone()
        ops.decode_attention(q, cache, positions, table, out, partial, counters, S, n_head, n_kv_head, head_dim, page_size, scale, window, splits,
                             tensor_cores=True, sink=sink, q_start=starts)
        assert torch.equal(out[~single], portions[~single]) and (counters == 0).all()
        if sink is None:
            # Probabilities and the result in bfloat16 (2^-9 each), values of order one: as for the kernels by themselves.
            assert (out.double().cpu() - _attention_reference(refs, n_head, n_kv_head, scale, window)).abs().max().item() < 1.5e-2
        else:
            whole = torch.empty_like(q)
            ops.paged_attention_generic(q, cache, tok_seq, positions, table, whole, q.shape[0], n_head, n_kv_head, head_dim, page_size, scale, window, sink=sink)
            assert (out.float() - whole.float()).abs().max().item() < 1.5e-2
