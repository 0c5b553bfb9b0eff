"""How a step with prompt portions launches its attentions: the choices whose other side was measured, without a GPU."""
from __future__ import annotations

import ctypes as C
import random

import pytest

from liyab_b200 import _capi

APART, TCGEN05, RUNS, JOINED, ALONE = 1, 2, 4, 8, 16
SCORES = {"": 0, "cap": 1, "bound": 2, "dist": 3}


def plan(requests, n_head, dtype="bfloat16", n_kv_head=None, head_dim=64, page_size=16, mask=0, sms=148, form=""):
    """requests: (tokens held, tokens brought)."""
    start, longest = [0], max(new for _, new in requests)
    for _, new in requests:
        start.append(start[-1] + new)
    bits = C.c_int32(-1)
    _capi.check(_capi.lib().lb_attention_plan_scores(dtype.encode(), n_head, n_kv_head or n_head, head_dim, page_size, mask, SCORES[form], sms, len(requests),
                                              (C.c_int32 * len(start))(*start), (C.c_int32 * len(requests))(*[held for held, _ in requests]),
                                              -(-longest // 64) * 64, C.byref(bits)))
    return bits.value


def singles(n, lo, hi):
    r = random.Random(n)
    return [(r.randint(lo, hi), 1) for _ in range(n)]


# Measured in every way a step can be launched (us: with the chosen one, with the best of the others).
@pytest.mark.parametrize("heads,requests,want", [
    # Single tokens among the portion's tiles, where they end before it does and all blocks run at once (14.8 / 14.8) ...
    (12, singles(6, 300, 900) + [(700, 200)], TCGEN05),
    # ... by blocks of their own in that launch, where they reach further (11.2 / 11.1, 7.6 / 11.7, 20.2 / 24.3, 18.5 / 18.1, 4.4 / 7.6, 7.2 / 10.4) ...
    (12, singles(6, 50, 250) + [(300, 300)], TCGEN05 | JOINED),
    (12, singles(6, 900, 1000) + [(0, 256)], TCGEN05 | JOINED), (25, singles(12, 300, 900) + [(300, 500)], TCGEN05 | JOINED),
    (25, singles(16, 100, 300) + [(0, 700)], TCGEN05 | JOINED), (12, [(300, 1)] * 6 + [(0, 64)], TCGEN05 | JOINED), (4, [(850, 1)] * 4 + [(0, 300)], TCGEN05 | JOINED),
    # ... or by a launch of their own, where they are many or long (22.3 / 23.5, 40.0 / 46.0, 10.9 / 16.0, 25.1 / 35.4, 35.3 / 43.9, 14.0 / 20.8, 19.3 / 44.1).
    (12, singles(30, 900, 1000) + [(0, 500)], APART | TCGEN05),
    (25, singles(30, 700, 900) + [(0, 600)], APART | TCGEN05), (25, singles(1, 3000, 3000) + [(0, 100)], APART | TCGEN05), (25, singles(30, 300, 900) + [(0, 130)], APART | TCGEN05),
    (12, singles(60, 900, 1000) + [(0, 130)], APART | TCGEN05), (12, singles(40, 400, 600) + [(0, 2)], APART | TCGEN05), (12, singles(100, 250, 350) + [(0, 64)], APART),
    # Portions alone: the tcgen05 kernel for long ones (16.0 / 35.7 and the like) and, from nineteen requests to twenty, for short ones (13.0 / 16.9, 13.2 / 17.6, 22.5 / 34.0, 20.0 / 21.2,
    # 25.5 / 41.1), the other one for many of less than a tile (14.8 / 21.2, 18.1 / 28.6, 5.3 / 5.7).
    (12, [(0, 1024)], TCGEN05), (12, [(0, 1000)] * 2, TCGEN05), (25, [(0, 1000)] * 2, TCGEN05), (25, [(0, 218), (0, 441), (0, 583), (0, 560), (0, 541)], TCGEN05),
    (25, [(0, 100)] * 19, TCGEN05), (25, [(0, 100)] * 20, TCGEN05), (25, [(350, 64)] * 20, TCGEN05), (16, [(350, 40)] * 20, TCGEN05), (12, [(500, 20)] * 40, TCGEN05),
    (25, [(0, 64)] * 40, 0), (25, [(0, 30)] * 60, 0), (12, [(0, 8)] * 20, 0)])
def test_choices_that_were_measured(heads, requests, want):
    assert plan(requests, heads) & ~ALONE == want
    assert plan(requests[::-1], heads) & ~ALONE == want          # whatever their order


# One block an SM where the longest blocks set the time, two elsewhere (us alone / two, the same step with plain scores, capped, and with a penalty by distance).
@pytest.mark.parametrize("heads,requests,alone", [
    (12, [(0, 1000)] * 2, True),           # -, 27.6 / 32.3, 23.7 / 26.5
    (16, [(0, 2048)], True),               # -, 52.4 / 69.6, 45.1 / 54.9
    (25, [(0, 900)], True),                # -, 25.9 / 31.8, 23.2 / 25.8
    (12, [(0, 2048)], True),               # 27.7 / 29.8, 51.2 / 59.4, 43.5 / 47.3
    (25, [(0, 1000)] * 2, False),          # 32.3 / 22.6, 52.3 / 36.2, 45.3 / 31.3
    (12, [(0, 180)] * 8, False),           # 11.6 / 7.3, 14.8 / 10.3, 14.1 / 9.3
    (25, [(0, 218), (0, 441), (0, 583), (0, 560), (0, 541)], False)])
def test_blocks_that_have_an_sm_to_themselves(heads, requests, alone):
    for form in SCORES:
        if form or not alone or requests == [(0, 2048)] and heads == 12:          # the others are close with plain scores
            assert plan(requests, heads, form=form) == TCGEN05 | (ALONE if alone else 0), form


def test_only_kernels_that_take_the_shape():
    mixed = singles(30, 900, 1000) + [(0, 500)]
    assert plan(mixed, 12, head_dim=128) & TCGEN05 == 0 and plan(mixed, 12, head_dim=128) & APART
    assert plan(mixed, 12, head_dim=32) == 0                     # the decode kernel on the tensor cores takes heads of 64 and 128
    assert plan(mixed, 12, head_dim=40) == 0 and plan(mixed, 34, n_kv_head=2) & APART == 0
    assert plan(mixed, 12, page_size=8) & APART == 0
    few = [(300, 1)] * 6 + [(0, 64)]
    assert plan(few, 12) & JOINED and plan(few, 12, n_kv_head=4) & JOINED == 0 and plan(few, 12, head_dim=128) & JOINED == 0     # blocks for single query heads of 64
    assert plan([(100, 1)], 12) & ~ALONE in (0, APART, TCGEN05)           # a launch is chosen for any step


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
