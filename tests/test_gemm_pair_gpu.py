"""Products in tiles that two SMs make together, at the edges of their tiles, against 64 bits."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import plain_gpt2 as plain
from test_kernels_gpu import _rand, dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [128, 192, 256])
@pytest.mark.parametrize("M,N,K", [(65, 64, 64), (128, 40, 72), (129, 256, 320), (256, 200, 1600), (257, 1000, 200), (700, 520, 328), (2500, 2312, 136)])
def test_products(dev, M, N, K, tile):
    """Less than a tile and several a pair, a second block without tokens, features and strips cut off, fewer k-blocks than stages and more."""
    from liyab_b200 import ops
    a, w = _rand((M, K), 90, dev, torch.bfloat16), _rand((N, K), 91, dev, torch.bfloat16, 0.1)
    bias, res = _rand((N,), 92, dev), _rand((M, N), 93, dev)
    base = a.double() @ w.double().t()
    # 32-bit sums of K products, in whatever order: K roundings at most.
    bound = K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t()) + 2.0 ** -22 * (bias.double().abs() + res.double().abs())
    out = res.clone()
    ops.gemm_pair(a, w, bias, out, M, "none", residual=out, feature_tile=tile)
    assert ((out.double() - (base + bias.double() + res.double())).abs() <= bound).all()
    plain_out = torch.full((M + 1, N), 7.0, device=dev)
    ops.gemm_pair(a, w, None, plain_out, M, "none", feature_tile=tile)
    assert ((plain_out[:M].double() - base).abs() <= bound).all() and (plain_out[M] == 7.0).all()
    half = torch.full((M + 1, -(-N // 8) * 8), 7.0, dtype=torch.bfloat16, device=dev)[:, :N]
    ops.gemm_pair(a, w, bias, half, M, "gelu_tanh", feature_tile=tile)
    want = torch.from_numpy(plain.gelu_tanh((base + bias.double()).cpu().numpy())).to(dev)
    # The slope of GELU is below 1.13; its fast form is off by 1e-6 of the value, and the result is rounded to bfloat16.
    assert ((half[:M].double() - want).abs() <= 1.13 * bound + 2.0 ** -8 * want.abs() + 1e-6).all() and (half[M] == 7.0).all()
    assert ops.device_status() == 0


@pytest.mark.parametrize("M,n_head,n_kv_head,K", [(300, 6, 2, 136), (2500, 25, 25, 136), (19300, 1, 1, 64), (37988, 3, 1, 72)])
def test_keys_and_values_go_to_their_pages(dev, M, n_head, n_kv_head, K):
    """One tile a pair of SMs; several, in other columns; several in the same column, with strips of queries and of keys in one tile: a strip that
    goes to the cache must not let the next tile overwrite queries that are still on their way out."""
    from liyab_b200 import ops
    head_dim, page_size = 64, 16
    n_pages = -(-M // page_size) + 5
    q_dim, kv_dim = n_head * head_dim, n_kv_head * head_dim
    a, w = _rand((M, K), 94, dev, torch.bfloat16), _rand((q_dim + 2 * kv_dim, K), 95, dev, torch.bfloat16, 0.2)
    bias = _rand((q_dim + 2 * kv_dim,), 96, dev)
    slots = np.random.default_rng(5).permutation(n_pages * page_size)[:M].astype(np.int32)
    slots[[3, 200]] = -1
    slot_mapping = torch.from_numpy(slots).to(dev)
    want_cache = torch.full((n_pages, 2, n_kv_head, page_size, head_dim), 3.0, dtype=torch.bfloat16, device=dev)
    want = torch.empty((M, q_dim + 2 * kv_dim), dtype=torch.bfloat16, device=dev)
    ops.gemm_pair(a, w, bias, want, M)
    ops.kv_append(want[:, q_dim:q_dim + kv_dim], want[:, q_dim + kv_dim:], slot_mapping, want_cache, M, n_kv_head, head_dim, page_size)
    for tile in (128, 192, 256):
        got_cache, got = torch.full_like(want_cache, 3.0), torch.empty_like(want)
        ops.gemm_pair(a, w, bias, got, M, feature_tile=tile, kv=(got_cache, slot_mapping, q_dim, n_kv_head, head_dim, page_size))
        assert torch.equal(got[:, :q_dim], want[:, :q_dim]) and torch.equal(got_cache, want_cache)
