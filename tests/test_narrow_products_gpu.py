"""The tcgen05 product for some dozens of tokens: tiles and parts of the reduction with remainders in every size, its cache as a second destination, and
what the plan makes of them."""
from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import _rand, dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 17, 33, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("N,K,features,splits", [
    (8, 8, 8, 1), (104, 200, 24, 1), (256, 256, 64, 2), (768, 768, 32, 4), (1600, 1600, 96, 4), (1000, 4104, 128, 8), (1024, 4096, 64, 8), (384, 3072, 256, 8),
    (264, 640, 256, 1), (512, 6400, 192, 4), (2304, 768, 0, 0), (1600, 6400, 0, 0)])
def test_products(dev, M, N, K, features, splits):
    """Against 64 bits, float32 results with a residual in place and bfloat16 ones with an activation; the same bits on a second call."""
    from liyab_b200 import ops
    a, w = _rand((M, K + 8), 90, dev, torch.bfloat16)[:, :K], _rand((N, K), 91, dev, torch.bfloat16, 0.1)
    bias, res = _rand((N,), 92, dev), _rand((M, N + 8), 93, dev)[:, :N]
    ref = a.double() @ w.double().t() + bias.double()
    # Sums of K products in the tensor core (32-bit accumulators, K / 16 roundings), of up to eight parts, bias and residual.
    bound = (K / 16 + 16) * 2.0 ** -23 * (a.double().abs() @ w.double().abs().t() + bias.double().abs() + res.double().abs())
    outs = []
    for _ in range(2):
        out = res.clone()
        ops.gemm_narrow(a, w, bias, out, M, "none", residual=out, features=features, splits=splits)
        assert ops.device_status() == 0
        assert ((out.double() - ref - res.double()).abs() <= bound).all()
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    half = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=dev)
    ops.gemm_narrow(a, w, bias, half, M, "relu2", features=features, splits=splits)
    want = ref.clamp(min=0) ** 2
    assert ((half.double() - want).abs() <= 2.0 ** -8 * want + 2 * (ref.abs() + bound) * bound).all()


@pytest.mark.parametrize("M", [20, 64, 200])
@pytest.mark.parametrize("n_head,n_kv_head,head_dim,page_size", [(12, 12, 64, 16), (6, 2, 48, 32), (5, 1, 8, 64)])
def test_keys_and_values_go_to_their_pages(dev, M, n_head, n_kv_head, head_dim, page_size):
    from liyab_b200 import ops
    q_dim, kv_dim, K = n_head * head_dim, n_kv_head * head_dim, 512
    N, n_pages = q_dim + 2 * kv_dim, -(-M // page_size) + 2
    a, w, bias = _rand((M, K), 94, dev, torch.bfloat16), _rand((N, K), 95, dev, torch.bfloat16, 0.1), _rand((N,), 96, dev)
    slots = torch.randperm(n_pages * page_size, generator=torch.Generator().manual_seed(M))[:M].int().to(dev)
    slots[3] = -1                                                            # a token that keeps nothing
    cache = torch.full((n_pages, 2, n_kv_head, page_size, head_dim), 7.0, dtype=torch.bfloat16, device=dev)
    out, whole = (torch.full((M, N), 7.0, dtype=torch.bfloat16, device=dev) for _ in range(2))
    ops.gemm_narrow(a, w, bias, out, M, kv=(cache, slots, q_dim, n_kv_head, head_dim, page_size))
    ops.gemm_narrow(a, w, bias, whole, M)
    assert torch.equal(out[:, :q_dim], whole[:, :q_dim]) and (out[:, q_dim:] == 7.0).all()
    want = torch.full_like(cache, 7.0)
    for t, slot in enumerate(slots.tolist()):
        if slot >= 0:
            want[slot // page_size, :, :, slot % page_size] = whole[t, q_dim:].view(2, n_kv_head, head_dim)
    assert torch.equal(cache, want)


def test_refusals(dev):
    from liyab_b200 import ops
    from liyab_b200.status import LiyabError
    a, w, out = _rand((40, 64), 97, dev, torch.bfloat16), _rand((20, 64), 98, dev, torch.bfloat16), torch.zeros((40, 20), device=dev)
    for bad in (lambda: ops.gemm_narrow(a, w, None, out, 40), lambda: ops.gemm_narrow(a, w[:16].clone(), None, out[:, :16], 40, features=12, splits=1),
                lambda: ops.gemm_narrow(a, w[:16].clone(), None, torch.zeros((40, 16), device=dev), 40, features=16, splits=2)):
        with pytest.raises(LiyabError):
            bad()


@pytest.mark.parametrize("activation", ["gelu_tanh", "gelu_erf", "xielu", "relu2"])
@pytest.mark.parametrize("features,splits", [(64, 1), (64, 4)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_activations(dev, activation, features, splits, dtype):
    """Every activation on sums around zero, beside the kernel of the float32 units on the same operands."""
    from liyab_b200 import ops
    M, N, K = 70, 328, 1536
    a, w = _rand((M, K), 100, dev, torch.bfloat16), _rand((N, K), 101, dev, torch.bfloat16, 0.05)
    bias = _rand((N + 2,), 102, dev)                                          # xIELU keeps its two numbers behind the bias
    bias[N:] = torch.tensor([0.8, 0.4], device=dev)
    out, want = (torch.empty((M, N), dtype=t, device=dev) for t in (dtype, torch.float32))
    ops.gemm_narrow(a, w, bias[:N], out, M, activation, features=features, splits=splits)
    ops.gemm_ffma(a, w, bias[:N], want, M, activation)
    assert ops.device_status() == 0
    # The sums' roundings (see test_products) through slopes of up to 2.4 |x| + 1, and the result's own; GELU of bfloat16 results leaves 2^-12 of its argument.
    sums = (K / 16 + 16) * 2.0 ** -23 * (a.double().abs() @ w.double().abs().t() + bias[:N].double().abs())
    x = a.double() @ w.double().t() + bias[:N].double()
    slope = 3 * x.abs().max() + 2
    bound = slope * sums + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20) * want.double().abs() + (2.0 ** -12 * x.abs() if dtype == torch.bfloat16 else 0)
    assert ((out.double() - want.double()).abs() <= bound).all()


@pytest.mark.parametrize("features,splits", [(48, 1), (64, 4), (256, 8)])
def test_special_values_stay_in_their_rows_and_columns(dev, features, splits):
    """Infinities and NaN among activations and weights: the places they reach and no others, like the products of 64-bit numbers."""
    from liyab_b200 import ops
    M, N, K = 70, 512, 2048
    a, w = _rand((M, K), 103, dev, torch.bfloat16), _rand((N, K), 104, dev, torch.bfloat16, 0.1)
    a[3, 5], a[64, K - 1], a[9, 700] = float("inf"), float("nan"), -float("inf")
    w[17, 5], w[511, 40], w[200, 700] = 0.0, float("-inf"), float("nan")
    out = torch.empty((M, N), device=dev)
    ops.gemm_narrow(a, w, None, out, M, features=features, splits=splits)
    ref = a.double() @ w.double().t()
    assert torch.equal(out.isnan(), ref.isnan()) and torch.equal(out == float("inf"), ref == float("inf")) and torch.equal(out == -float("inf"), ref == -float("inf"))
    finite = ref.isfinite()
    assert ((out.double() - ref)[finite].abs() <= 1e-3).all() and ops.device_status() == 0


@pytest.mark.parametrize("M,N,K,narrow", [(40, 768, 768, True), (20, 1600, 6400, True), (20, 768, 768, False), (40, 512, 256, False), (300, 768, 768, False)])
def test_linear_goes_where_a_step_goes(dev, M, N, K, narrow):
    from liyab_b200 import ops
    a, w, bias = _rand((M, K), 105, dev, torch.bfloat16), _rand((N, K), 106, dev, torch.bfloat16, 0.1), _rand((N,), 107, dev)
    out, same = (torch.empty((M, N), dtype=torch.bfloat16, device=dev) for _ in range(2))
    assert ops.gemm_narrow_takes(a, w, out, M) == narrow
    ops.linear(a, w, bias, out, M, "gelu_tanh")
    if narrow:
        ops.gemm_narrow(a, w, bias, same, M, "gelu_tanh")
        assert torch.equal(out, same)
    ref = torch.nn.functional.gelu(a.double() @ w.double().t() + bias.double(), approximate="tanh")
    assert ((out.double() - ref).abs() <= 2.0 ** -7 * ref.abs() + 2e-3).all()
