"""Steps of one long portion beside single tokens, through the engine, captured once and replayed with the requests in other places, against the plain model:
with the single tokens in the portion's launch, and with a launch of their own."""
from __future__ import annotations

import numpy as np
import pytest

import plain_gpt2 as plain
from test_attention_plan import ALONE, APART, JOINED, TCGEN05, plan
from tiny_models import random_tokens

pytestmark = pytest.mark.gpu

RAW = dict(model_type="gpt2", n_layer=2, n_embd=256, n_head=4, n_inner=512, vocab_size=640, n_positions=3072, layer_norm_epsilon=1e-5,
           activation_function="gelu_new")
REL_TOL = 2.5e-2
# Tokens held by the long requests, tokens of the portion, how the plan has them launched.  Four heads of 64: single tokens on 850 keys are through before a
# portion of 300; on 2500 a block each takes longer than the portion of 100 and the decode kernel's ranges together.
ROUTES = {"joined": (850, 300, TCGEN05 | JOINED), "apart": (2500, 100, TCGEN05 | APART)}


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    from liyab_b200.weights import write_random_model
    folder = write_random_model(str(tmp_path_factory.mktemp("mixed") / "m"), RAW, seed=11, dtype="bfloat16")
    toks = random_tokens(31, max(held for held, _, _ in ROUTES.values()) + 8, RAW["vocab_size"]), random_tokens(32, 320, RAW["vocab_size"])
    loaded = plain.load_plain_model(folder)
    return folder, toks, [plain.forward_logits(loaded, t) for t in toks]


@pytest.mark.parametrize("route", ROUTES)
def test_a_captured_step_serves_every_arrangement(model, route):
    from liyab_b200.engine import Replayer, StepEntry
    folder, (long, fresh), (want_long, want_fresh) = model
    held, portion, bits = ROUTES[route]
    r = Replayer(folder, "bfloat16", max_tokens=20_000, max_requests=16, cuda_graphs=True, max_step_tokens=2560)
    # Tokens brought by each request, the portion and four more in all and the longest in one bucket; single tokens come to long requests, portions to new ones.
    p = portion
    arrangements = [(p, 1, 1, 1, 1), (1, 1, p, 1, 1), (1, 1, 1, 1, p), (1, p - 1, 1, 2, 1), (4, 1, 1, p - 3, 1), (1, 3, p - 2, 1, 1), (p, 1, 1, 1, 1)]
    before, serial = None, 0
    for turn, lens in enumerate([arrangements[0]] * 2 + arrangements):
        names, entries, wants = [], [], []
        for n in lens:
            name, serial = f"r{serial}", serial + 1
            r.cache.open(name)
            names.append(name)
            if n == 1:
                r.step([StepEntry(name, long[:held])], fetch=False)
                entries.append(StepEntry(name, long[held:held + 1], [0]))
                wants.append(want_long[held])
            else:
                # Eleven wanted rows in every arrangement: all of a short portion's, the others from the long one.
                rows = list(range(n)) if n < 50 else [0, n // 2] + [n - 1] * (9 - sum(m for m in lens if m < 50))
                entries.append(StepEntry(name, fresh[:n], rows))
                wants += [want_fresh[i] for i in rows]
        assert plan([(held if n == 1 else 0, n) for n in lens], RAW["n_head"]) & ~ALONE == bits
        counted = r.counters()
        got = r.step(entries).logits
        after = r.counters()
        if turn == 2:
            before = after["graphs_captured"]
            assert before == counted["graphs_captured"] + 1
        elif turn > 2:
            assert after["graph_steps"] == counted["graph_steps"] + 1 and after["graphs_captured"] == before, lens
        for row, want in zip(got, wants):
            assert np.abs(row - want).max() <= REL_TOL * np.abs(want).max(), (turn, lens)
        for name in names:
            r.cache.close(name)
