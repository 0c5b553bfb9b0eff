"""The tcgen05 prefill attention at the edges of its warps and tiles: portions that fill a part of a tile's warps on contexts of several key
tiles (where warps without rows run ahead of the others), and more requests than one look finds."""
from __future__ import annotations

import numpy as np
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


@pytest.mark.parametrize("form", [{}, {"soft_cap": 3.0}, {"soft_cap": 40.0, "score_bound": 8.0}, {"distance": True}])
def test_one_block_an_sm_has_the_bits_of_two(dev, form):
    """The launch that keeps its blocks apart, alone and with the single tokens: the same sums; capped and biased scores against 64 bits."""
    from liyab_b200 import ops
    lens, q_lens, H, scale = [400, 300, 17, 129, 700], [400, 130, 1, 2, 1], 3, 0.125
    q, cache, _, positions, table, refs = _paged_case(dev, torch.bfloat16, H, H, 64, 16, lens, q_lens, seed=77)
    start = torch.tensor([0] + np.cumsum(q_lens).tolist(), dtype=torch.int32, device=dev)
    past = torch.tensor([l - n for l, n in zip(lens, q_lens)], dtype=torch.int32, device=dev)
    kw = dict(form)
    if kw.pop("distance", False):
        kw["distance"] = torch.tensor([0.4, 0.2, 0.9, 0.5, 2.0, 0.1], device=dev)
    outs = {}
    for singles in (False, True):
        for alone in (False, True):
            out = torch.full_like(q, float("nan"))
            ops.prefill_attention(q, cache, start, past, table, out, len(lens), 448, H, H, 64, 16, scale, 0, tcgen05=True, min_len=2 if singles else 1, singles=singles, alone=alone, **kw)
            outs[singles, alone] = out
    assert ops.device_status() == 0
    assert torch.equal(outs[False, False], outs[False, True]) and torch.equal(outs[True, False], outs[True, True])
    at = 0
    for (qs, k, v, first), n in zip(refs, q_lens):
        back = (torch.arange(n)[:, None] + first - torch.arange(k.shape[0])[None]).double()
        for h in range(H):
            s = qs[:, h] @ k[:, h].t() * scale
            if "soft_cap" in kw:
                s = kw["soft_cap"] * torch.tanh(s / kw["soft_cap"])
            if "distance" in kw:
                d = kw["distance"].double().cpu()
                s = s - d[h] * torch.log1p(d[H + h] * back.clamp(min=0))
            ref = s.masked_fill(back < 0, -float("inf")).softmax(-1) @ v[:, h]
            for out in (outs[False, False], outs[True, False]):
                got = out[at:at + n, h * 64:(h + 1) * 64].double().cpu()
                # Probabilities rounded to bfloat16 (2^-9 of values of up to four), and the result.
                assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -9 * 4).all()
        at += n
