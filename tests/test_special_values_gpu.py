"""Infinities, NaN and values at the ends of the range in the products' and attentions' kernels: they come out where the plain formulas have them, and
nowhere else."""
from __future__ import annotations

import math

import pytest
import torch

from test_kernels_gpu import _paged_case, _rand, dev  # noqa: F401

pytestmark = pytest.mark.gpu
SPECIAL = [float("inf"), -float("inf"), float("nan"), 0.0, -0.0, 3e38, -3e38, 1e20, -1e20, 1e4, -1e4, 88.0, -88.0, 1e-30, -1e-30]


@pytest.mark.parametrize("shared", [False, True])
def test_gelu_of_bfloat16_epilogues(dev, shared):
    """Every row's only non-zero product is its special value, as it is."""
    from liyab_b200 import ops
    M, N, K = 80, 72, 64
    a, w = torch.zeros((M, K), device=dev), torch.zeros((N, K), device=dev)
    a[:, 0] = torch.tensor([SPECIAL[i % len(SPECIAL)] for i in range(M)], device=dev)
    w[:, 0] = 1.0
    a, w = a.to(torch.bfloat16), w.to(torch.bfloat16)
    out = torch.empty((M, N), dtype=torch.bfloat16, device=dev)
    (ops.gemm_pair if shared else ops.gemm_persistent)(a, w, None, out, M, "gelu_tanh")
    want = torch.nn.functional.gelu(a[:, :1].double(), approximate="tanh").expand(M, N)
    finite = want.isfinite()
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.double()[want.isinf()], want[want.isinf()])
    # As in the products' own test: the fast form is off by 1e-6 of the value and the result is rounded to bfloat16.
    assert ((out.double() - want).abs()[finite] <= 2.0 ** -8 * want.abs()[finite] + 1e-30).all()


@pytest.mark.parametrize("M", [8, 13])
def test_rows_that_the_ring_normalises(dev, M):
    """Rows with an infinity, a NaN or a spread past float32's range turn into NaN as the LayerNorm kernel makes them; the others keep their bits."""
    from liyab_b200 import ops
    N, K = 200, 1600
    x, w, gain, offset = _rand((M, K), 40, dev), _rand((N, K), 41, dev, torch.bfloat16, 0.1), _rand((K,), 42, dev), _rand((K,), 43, dev)
    clean, got, normed = (torch.empty((M, n), dtype=t, device=dev) for n, t in ((N, torch.float32), (N, torch.float32), (K, torch.bfloat16)))
    assert ops.gemm_rows_kind(M, N, K, normed=True) == 2
    ops.gemm_rows_normed(x, gain, offset, 1e-5, w, None, clean, M)
    x[1, 3], x[2, K - 1], x[5, 700], x[6] = float("inf"), -float("inf"), float("nan"), x[6] * 1e38
    x[7] = 2.5                                             # no spread at all
    ops.gemm_rows_normed(x, gain, offset, 1e-5, w, None, got, M)
    ops.layernorm(x, gain, offset, 1e-5, normed, M)
    want = normed.double() @ w.double().t()
    keep = torch.tensor([r not in (1, 2, 5, 6, 7) for r in range(M)], device=dev)
    assert torch.equal(got[keep], clean[keep]) and torch.equal(got.isnan(), want.isnan())
    # Eight chains of K / 8 products and one rounding of a normed value that may go either way (2^-8).
    bound = ((K / 8 + 16) * 2.0 ** -24 + 2.0 ** -8) * (normed.double().abs() @ w.double().abs().t())
    assert ((got.double() - want).abs()[7] <= bound[7] + 1e-30).all()


@pytest.mark.parametrize("where", ["query", "key", "value"])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan"), 3e38])
def test_float32_attentions_agree(dev, where, value):
    """The kernel of runs, the one of few pairs and the plain one have the same bits and the same NaN."""
    from liyab_b200 import ops
    n_head, page_size, lens, q_lens, scale = 4, 16, [300, 77, 210], [290, 70, 3], 0.125
    q, cache, tok_seq, positions, table, _ = _paged_case(dev, torch.float32, n_head, n_head, 64, page_size, lens, q_lens, seed=5)
    n = q.shape[0]
    assert n * n_head > 1024
    if where == "query":
        q[40, 10] = q[200, 130] = q[n - 1, 255] = value
    else:
        for seq, at, head in ((0, 17, 1), (0, 299, 0), (1, 3, 2), (2, 100, 3)):
            cache[table[seq, at // page_size].item(), 0 if where == "key" else 1, head, at % page_size, 5] = value
    runs, plain = torch.full_like(q, 7.0), torch.full_like(q, 7.0)
    ops.paged_attention_f32_runs(q, cache, tok_seq, positions, table, runs, n, n_head, n_head, page_size, scale)
    ops.paged_attention_generic(q, cache, tok_seq, positions, table, plain, n, n_head, n_head, 64, page_size, scale, 0)
    same = lambda a, b: torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(nan=1.5), b.nan_to_num(nan=1.5))      # noqa: E731
    assert same(runs, plain) and not (plain.isfinite().all() and not math.isfinite(value))
    for lo, hi in ((30, 60), (190, 210), (n - 4, n)):
        few = torch.full_like(q[lo:hi], 7.0)
        ops.paged_attention_generic(q[lo:hi].contiguous(), cache, tok_seq[lo:hi].contiguous(), positions[lo:hi].contiguous(), table, few, hi - lo, n_head, n_head, 64,
                                    page_size, scale, 0)
        assert same(few, plain[lo:hi])
