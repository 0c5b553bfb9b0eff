"""Decode attention of 64 or more pairs of a request and a key/value head in two to four ranges: one block of eight or sixteen warps a pair."""
from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import _attention_reference, _paged_case, _rand, dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [2, 3, 4])
@pytest.mark.parametrize("n_head,n_kv_head,page_size,window,n_seq,with_sink", [
    (9, 9, 16, 0, 7, False), (8, 8, 16, 0, 8, False), (32, 8, 32, 0, 8, True), (20, 20, 64, 100, 8, False), (128, 8, 16, 0, 9, False)])
def test_many_pairs(dev, n_head, n_kv_head, page_size, window, n_seq, with_sink, splits):
    from liyab_b200 import ops
    lens = [1, 16, 17, 255, 256, 273, 1024, 600, 40][:n_seq]              # fewer tiles than warps, as many, one more, many
    scale, head_dim = 0.125, 64
    q, cache, tok_seq, positions, table, refs = _paged_case(dev, torch.bfloat16, n_head, n_kv_head, head_dim, page_size, lens, [1] * n_seq, seed=splits + n_head)
    partial = torch.full((n_seq * n_head * splits * (head_dim + 2),), float("nan"), device=dev)
    counters = torch.zeros(n_seq * n_kv_head, dtype=torch.int32, device=dev)
    sink = _rand((n_head,), 98, dev) if with_sink else None
    out = torch.full_like(q, float("nan"))
    ops.decode_attention(q, cache, positions, table, out, partial, counters, n_seq, n_head, n_kv_head, head_dim, page_size, scale, window, splits,
                         tensor_cores=True, sink=sink)
    assert int(counters.abs().sum()) == 0
    # Where contexts may be long, two ranges, or more than 128 pairs, go to clusters of blocks again.
    other = torch.full_like(q, float("nan"))
    ops.decode_attention(q, cache, positions, table, other, partial, counters, n_seq, n_head, n_kv_head, head_dim, page_size, scale, window, splits,
                         tensor_cores=True, sink=sink, max_keys=20_000)
    assert int(counters.abs().sum()) == 0 and (other.float() - out.float()).abs().max().item() < 1.5e-2
    # Probabilities and the result in bfloat16 (2^-9 each), values of order one: as for the blocks of four warps.
    generic = torch.empty_like(q)
    ops.paged_attention_generic(q, cache, tok_seq, positions, table, generic, n_seq, n_head, n_kv_head, head_dim, page_size, scale, window, sink=sink)
    assert (out.float() - generic.float()).abs().max().item() < 1.5e-2
    if sink is None:
        assert (out.double().cpu() - _attention_reference(refs, n_head, n_kv_head, scale, window)).abs().max().item() < 1.5e-2
