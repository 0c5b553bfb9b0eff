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


@pytest.mark.parametrize("heads,requests,want", [
    # The launch for single tokens costs 3 to 5 us: not where they end before the portion does and all blocks run at once (0.93 to 0.98 of the speed) ...
    (12, singles(3, 50, 250) + [(0, 500)], TCGEN05), (12, singles(6, 300, 900) + [(700, 200)], TCGEN05), (12, singles(6, 50, 250) + [(300, 300)], TCGEN05),
    # ... but where they reach further than the portion (1.05 to 1.10), or their blocks would fill the GPU several times (1.15 to 1.6): by blocks of the portion's
    # launch (us in one launch / in two: 20.0 / 25.0 for twelve beside 500 on 300 with 25 heads) or, where those take longer (15.4 /
    # 10.6 for one on 3000 beside 100), by a launch of their own.
    (12, singles(6, 900, 1000) + [(0, 256)], TCGEN05 | JOINED), (25, singles(12, 300, 900) + [(300, 500)], TCGEN05 | JOINED), (12, singles(30, 900, 1000) + [(0, 500)], TCGEN05 | JOINED),
    (25, singles(16, 100, 300) + [(0, 700)], APART | TCGEN05), (25, singles(1, 3000, 3000) + [(0, 100)], APART | TCGEN05),
    # Many blocks without rows: the mma.sync kernel for a short portion (the tcgen05 kernel has 0.82 of its speed there, 0.95 to 0.93 in two launches).
    (12, singles(30, 50, 250) + [(0, 130)], 0), (25, singles(30, 300, 900) + [(0, 130)], APART), (12, singles(60, 900, 1000) + [(0, 130)], APART),
    # Portions alone: the tcgen05 kernel for long ones (0.94 to 0.86 of its speed by the other), the other one for many short ones (0.87 to 0.94).
    (12, [(0, 1024)], TCGEN05), (12, [(0, 1000)] * 2, TCGEN05), (25, [(0, 1000)] * 2, TCGEN05), (25, [(0, 218), (0, 441), (0, 583), (0, 560), (0, 541)], TCGEN05), (25, [(0, 100)] * 20, 0), (25, [(350, 64)] * 20, 0), (16, [(350, 40)] * 20, 0)])
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
