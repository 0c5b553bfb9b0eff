"""float32 products of up to 8 tokens by whole rows of weights: against 64 bits, and the bits of the kernels that make the same sums another way."""
from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import _rand, dev  # noqa: F401

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24          # chains of 64 products, then up to 32 + K / 2048 sums of sums (see test_float32_kernels_gpu)


@pytest.mark.parametrize("M", [1, 5, 8])
@pytest.mark.parametrize("N,K,stages", [(2304, 768, 2), (2301, 772, 2), (11000, 132, 8), (9999, 4, 8), (768, 3072, 1), (1184, 3072, 1), (9, 2052, 1), (3300, 1600, 3), (1187, 4160, 0),
                                        (300, 1092, 1), (30, 8000, 0)])
def test_products_of_up_to_eight_rows(dev, M, N, K, stages):
    """One group of features a block or many, a ring that wraps, chunks and rows with remainders, one to three chunks a group, a row that does not fit."""
    from liyab_b200 import ops
    assert torch.cuda.get_device_properties(dev).multi_processor_count != 148 or ops.lib().lb_gemm_ffma_stream_stages(M, N, K, 148, None) == stages      # which kernel this is
    a, w, bias, res = _rand((24, K + 4), 65, dev)[:, :K], _rand((N, K), 66, dev), _rand((N,), 67, dev), _rand((24, N), 68, dev)
    out, whole = res[:M].clone(), res.clone()
    ops.gemm_ffma(a[:M], w, bias, out, M, "none", residual=out)
    ops.gemm_ffma(a, w, bias, whole, 24, "none", residual=whole)             # in tiles
    assert torch.equal(out, whole[:M]) and ops.device_status() == 0
    x, y = a[:M].double(), w.double()
    bound = EPS * (64 + 32 + K / 2048 + 3) * (x.abs() @ y.abs().t() + bias.double().abs() + res[:M].double().abs())
    assert ((out.double() - (x @ y.t() + bias.double() + res[:M].double())).abs() <= bound).all()
