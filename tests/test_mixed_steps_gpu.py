"""Steps of one long portion beside single tokens, through the engine: the single tokens' own attention launch, captured once and replayed with the requests in
other places, against the plain model."""
from __future__ import annotations

import numpy as np
import pytest

import plain_gpt2 as plain
from test_attention_plan import APART, plan
from tiny_models import random_tokens

pytestmark = pytest.mark.gpu

# Four heads of 64: single tokens on 850 keys reach four tiles of 128 further than a portion of 300, which is where they are served apart.
RAW = dict(model_type="gpt2", n_layer=2, n_embd=256, n_head=4, n_inner=512, vocab_size=640, n_positions=1024, layer_norm_epsilon=1e-5,
           activation_function="gelu_new")
HELD, REL_TOL = 850, 2.5e-2


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    from liyab_b200.weights import write_random_model
    folder = write_random_model(str(tmp_path_factory.mktemp("mixed") / "m"), RAW, seed=11, dtype="bfloat16")
    toks = random_tokens(31, HELD + 8, RAW["vocab_size"]), random_tokens(32, 320, RAW["vocab_size"])
    loaded = plain.load_plain_model(folder)
    return folder, toks, [plain.forward_logits(loaded, t) for t in toks]


def test_a_captured_step_serves_every_arrangement(model):
    from liyab_b200.engine import Replayer, StepEntry
    folder, (long, fresh), (want_long, want_fresh) = model
    r = Replayer(folder, "bfloat16", max_tokens=12_000, max_requests=16, cuda_graphs=True, max_step_tokens=1024)
    # Tokens brought by each request, 304 in all and the longest in one bucket; single tokens come to long requests, portions to new ones.
    arrangements = [(300, 1, 1, 1, 1), (1, 1, 300, 1, 1), (1, 1, 1, 1, 300), (1, 299, 1, 2, 1), (4, 1, 1, 297, 1), (1, 3, 298, 1, 1), (300, 1, 1, 1, 1)]
    before, serial = None, 0
    for turn, lens in enumerate([arrangements[0]] * 2 + arrangements):
        names, entries, wants = [], [], []
        for n in lens:
            name, serial = f"r{serial}", serial + 1
            r.cache.open(name)
            names.append(name)
            if n == 1:
                r.step([StepEntry(name, long[:HELD])], fetch=False)
                entries.append(StepEntry(name, long[HELD:HELD + 1], [0]))
                wants.append(want_long[HELD])
            else:
                # Eleven wanted rows in every arrangement: all of a short portion's, the others from the long one.
                rows = list(range(n)) if n < 100 else [0, n // 2] + [n - 1] * (9 - sum(m for m in lens if m < 100))
                entries.append(StepEntry(name, fresh[:n], rows))
                wants += [want_fresh[i] for i in rows]
        assert plan([(HELD if n == 1 else 0, n) for n in lens], RAW["n_head"]) & APART
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
