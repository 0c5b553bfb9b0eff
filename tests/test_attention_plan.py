"""How a step with prompt portions launches its attentions: the choices whose other side was measured, without a GPU."""
from __future__ import annotations

import ctypes as C
import random

import pytest

from liyab_b200 import _capi

APART, TCGEN05, RUNS, JOINED = 1, 2, 4, 8


def plan(requests, n_head, dtype="bfloat16", n_kv_head=None, head_dim=64, page_size=16, mask=0, sms=148):
    """requests: (tokens held, tokens brought)."""
    start, longest = [0], max(new for _, new in requests)
    for _, new in requests:
        start.append(start[-1] + new)
    bits = C.c_int32(-1)
    _capi.check(_capi.lib().lb_attention_plan(dtype.encode(), n_head, n_kv_head or n_head, head_dim, page_size, mask, sms, len(requests),
                                              (C.c_int32 * len(start))(*start), (C.c_int32 * len(requests))(*[held for held, _ in requests]),
                                              -(-longest // 64) * 64, C.byref(bits)))
    return bits.value


def singles(n, lo, hi):
    r = random.Random(n)
    return [(r.randint(lo, hi), 1) for _ in range(n)]


# Measured in every way a step can be launched (us: with the chosen one, with the best of the others).
@pytest.mark.parametrize("heads,requests,want", [
    # Single tokens among the portion's tiles, where they end before it does and all blocks run at once (14.9 / 14.9, 11.2 / 11.4) ...
    (12, singles(6, 300, 900) + [(700, 200)], TCGEN05), (12, singles(6, 50, 250) + [(300, 300)], TCGEN05),
    # ... by blocks of their own in that launch, where they reach further (8.3 / 11.7, 20.2 / 26.0, 23.5 / 23.0, 18.5 / 18.1, 4.4 / 7.6) ...
    (12, singles(6, 900, 1000) + [(0, 256)], TCGEN05 | JOINED), (25, singles(12, 300, 900) + [(300, 500)], TCGEN05 | JOINED), (12, singles(30, 900, 1000) + [(0, 500)], TCGEN05 | JOINED),
    (25, singles(16, 100, 300) + [(0, 700)], TCGEN05 | JOINED), (12, [(300, 1)] * 6 + [(0, 64)], TCGEN05 | JOINED), (4, [(850, 1)] * 4 + [(0, 300)], TCGEN05 | JOINED),
    # ... or by a launch of their own, where they are many or long (39.0 / 46.0, 10.9 / 16.0, 24.5 / 30.5, 35.0 / 39.1, 13.6 / 20.8, 19.3 / 44.1).
    (25, singles(30, 700, 900) + [(0, 600)], APART | TCGEN05), (25, singles(1, 3000, 3000) + [(0, 100)], APART | TCGEN05), (25, singles(30, 300, 900) + [(0, 130)], APART | TCGEN05),
    (12, singles(60, 900, 1000) + [(0, 130)], APART | TCGEN05), (12, singles(40, 400, 600) + [(0, 2)], APART | TCGEN05), (12, singles(100, 250, 350) + [(0, 64)], APART),
    # Portions alone: the tcgen05 kernel for long ones (16.0 / 35.7 and the like) and, from nineteen requests to twenty, for short ones (13.0 / 16.9, 13.2 / 17.6, 22.5 / 34.0, 20.0 / 21.2,
    # 25.5 / 41.1), the other one for many of less than a tile (14.8 / 21.2, 18.1 / 28.6, 5.3 / 5.7).
    (12, [(0, 1024)], TCGEN05), (12, [(0, 1000)] * 2, TCGEN05), (25, [(0, 1000)] * 2, TCGEN05), (25, [(0, 218), (0, 441), (0, 583), (0, 560), (0, 541)], TCGEN05),
    (25, [(0, 100)] * 19, TCGEN05), (25, [(0, 100)] * 20, TCGEN05), (25, [(350, 64)] * 20, TCGEN05), (16, [(350, 40)] * 20, TCGEN05), (12, [(500, 20)] * 40, TCGEN05),
    (25, [(0, 64)] * 40, 0), (25, [(0, 30)] * 60, 0), (12, [(0, 8)] * 20, 0)])
def test_choices_that_were_measured(heads, requests, want):
    assert plan(requests, heads) == want
    assert plan(requests[::-1], heads) == want          # whatever their order


def test_only_kernels_that_take_the_shape():
    mixed = singles(30, 900, 1000) + [(0, 500)]
    assert plan(mixed, 12, head_dim=128) & TCGEN05 == 0 and plan(mixed, 12, head_dim=128) & APART
    assert plan(mixed, 12, head_dim=32) == 0                     # the decode kernel on the tensor cores takes heads of 64 and 128
    assert plan(mixed, 12, head_dim=40) == 0 and plan(mixed, 34, n_kv_head=2) & APART == 0
    assert plan(mixed, 12, page_size=8) & APART == 0
    assert plan(mixed, 12) & JOINED and plan(mixed, 12, n_kv_head=4) & JOINED == 0 and plan(mixed, 12, head_dim=128) & JOINED == 0     # blocks for single query heads of 64
    assert plan([(100, 1)], 12) in (0, APART, TCGEN05)           # a launch is chosen for any step


@pytest.mark.parametrize("requests,runs", [
    # us by runs / a block a token, 12 heads: 338 / 117, 252 / 57, 167 / 32, 1261 / 213, 104 / 54
    (singles(24, 300, 950) + [(0, 200)], False), ([(699, 1)] * 12 + [(0, 100)], False), ([(599, 1)] * 8 + [(0, 64)], False), ([(2999, 1)] * 24 + [(0, 200)], False),
    ([(99, 1)] * 16 + [(0, 120)], False), ([(899, 1)] * 24 + [(0, 200)], False), ([(999, 1)] * 24 + [(0, 200)], False),
    # 504 / 831, 529 / 1179, 46 / 126, 34 / 122, 19 / 68, 213 / 1420, 28 / 82
    ([(899, 1)] * 100 + [(0, 800)], True), ([(999, 1)] * 120 + [(0, 1000)], True), ([(492, 8)] * 16, True), ([(484, 16)] * 8, True), ([(488, 12)] * 10, True), ([(0, 20)] * 10, True),
    ([(2700, 300)], True), ([(313, 87)], True)])
def test_float32_runs(requests, runs):
    assert plan(requests, 12, dtype="float32") == (RUNS if runs else 0)
    assert plan(requests, 12, dtype="float32", mask=64) == 0 and plan(requests, 12, dtype="float32", head_dim=32) == 0
