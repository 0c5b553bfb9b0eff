"""Products of up to 16 tokens whose weights run through the ring in shared memory: every number of groups a block, of chunks and of tokens at which
the kernel changes, against 64 bits."""
from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import _rand, dev  # noqa: F401

pytestmark = pytest.mark.gpu

SHAPES = [(40, 8192), (1600, 6400), (2368, 4104), (3600, 2056), (4800, 1600), (6400, 1600), (9472, 1032), (9465, 2048), (13, 5000)]


def _bound(a, w, rounding):
    """32-bit sums of K products in eight chains (K / 8 roundings each) and the rounding of what is summed."""
    K = a.shape[1]
    return ((K / 8 + 16) * 2.0 ** -24 + rounding) * (a.abs() @ w.abs().t())


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K", SHAPES)
def test_products(dev, M, N, K):
    from liyab_b200 import ops
    a, w = _rand((M, K + 8), 70, dev, torch.bfloat16)[:, :K], _rand((N, K), 71, dev, torch.bfloat16, 0.1)
    bias, res = _rand((N,), 72, dev), _rand((M, N), 73, dev)
    assert ops.gemm_rows_supports(a, w, M)
    ref = a.double() @ w.double().t()
    bound = _bound(a.double(), w.double(), 0.0) + 2.0 ** -22 * (bias.double().abs() + res.double().abs())
    out = res.clone()
    ops.gemm_rows(a, w, bias, out, M, "none", residual=out)
    assert ((out.double() - (ref + bias.double() + res.double())).abs() <= bound).all()
    half = torch.empty((M, N), dtype=torch.bfloat16, device=dev)
    ops.gemm_rows(a, w, None, half, M)
    assert ((half.double() - ref).abs() <= bound + ref.abs() * 2.0 ** -8).all()
    if M > 1:                      # a row's bits do not depend on how many rows share the launch
        fewer = torch.empty((1, N), dtype=torch.bfloat16, device=dev)
        ops.gemm_rows(a[M - 1:], w, None, fewer, 1)
        assert torch.equal(fewer[0], half[M - 1])


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(40, 1032), (1600, 2048), (4800, 1600), (6400, 1600), (9472, 1280)])
@pytest.mark.parametrize("affine", [True, False])
def test_products_of_normed_rows(dev, M, N, K, affine):
    from liyab_b200 import ops
    x, w, bias = _rand((M, K), 74, dev) * 3.0 + 2.0, _rand((N, K), 75, dev, torch.bfloat16, 0.1), _rand((N,), 76, dev)
    gain, offset = (_rand((K,), 77, dev) * 0.2 + 1.0, _rand((K,), 78, dev) * 0.3) if affine else (None, None)
    d = x.double() - x.double().mean(1, keepdim=True)
    a = d / torch.sqrt((d * d).mean(1, keepdim=True) + 1e-5)
    if affine:
        a = a * gain.double() + offset.double()
    out = torch.empty((M, N), dtype=torch.float32, device=dev)
    ops.gemm_rows_normed(x, gain, offset, 1e-5, w, bias, out, M)
    # The normed rows are rounded to bfloat16 (a value near a rounding boundary may go either way: one unit, 2^-8).
    bound = _bound(a, w.double(), 2.0 ** -8) + 2.0 ** -22 * bias.double().abs()
    assert ((out.double() - (a @ w.double().t() + bias.double())).abs() <= bound).all()


@pytest.mark.parametrize("normed", [False, True])
def test_keys_and_values_go_to_their_pages(dev, normed):
    from liyab_b200 import ops
    M, n_head, n_kv_head, head_dim, page_size, n_pages, K = 11, 24, 8, 64, 16, 5, 1288
    q_dim, kv_dim = n_head * head_dim, n_kv_head * head_dim
    N = q_dim + 2 * kv_dim
    w, bias = _rand((N, K), 79, dev, torch.bfloat16, 0.1), _rand((N,), 80, dev)
    slots = torch.randperm(n_pages * page_size, generator=torch.Generator().manual_seed(1))[:M].to(torch.int32)
    slots[4] = -1
    slots = slots.to(dev)
    want_cache = torch.full((n_pages, 2, n_kv_head, page_size, head_dim), 3.0, dtype=torch.bfloat16, device=dev)
    got_cache, out, got = want_cache.clone(), torch.empty((M, N), dtype=torch.bfloat16, device=dev), torch.empty((M, N), dtype=torch.bfloat16, device=dev)
    kv = (got_cache, slots, q_dim, n_kv_head, head_dim, page_size)
    if normed:
        x = _rand((M, K), 81, dev)
        ops.gemm_rows_normed(x, None, None, 1e-5, w, bias, out, M)
        ops.gemm_rows_normed(x, None, None, 1e-5, w, bias, got, M, kv=kv)
    else:
        x = _rand((M, K), 81, dev, torch.bfloat16)
        ops.gemm_rows(x, w, bias, out, M)
        ops.gemm_rows(x, w, bias, got, M, kv=kv)
    ops.kv_append(out[:, q_dim:q_dim + kv_dim], out[:, q_dim + kv_dim:], slots, want_cache, M, n_kv_head, head_dim, page_size)
    assert torch.equal(got, out) and torch.equal(got_cache, want_cache)
