"""Steps beside work on the default stream (another library's kernels): what the engine zeroes and uploads as it goes is there when its own stream uses it, and
nothing is zeroed after that."""
from __future__ import annotations

import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("design", ["revudra", "gekitar", "vosurax", "viresun"])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_first_steps_beside_work_on_the_default_stream(tmp_path, design, dtype):
    """The same bits as an engine that has the GPU to itself, in the steps that create buffers and in those after them."""
    from liyab_b200.engine import Replayer, StepEntry
    m = importlib.import_module(f"{design}_models")
    name = sorted(m.CONFIGS)[0]
    path, config, _ = m.model_folder(str(tmp_path), name)
    toks = np.random.default_rng(6).integers(0, config["vocab"], size=48).astype(int).tolist()
    a = torch.randn((8192, 8192), device="cuda").to(torch.bfloat16)
    b = torch.empty_like(a)

    def run(busy):
        engine = Replayer(path, dtype, 256, max_requests=4)
        engine.cache.open("a")
        rows = []
        for lo, hi in [(0, 40)] + [(i, i + 1) for i in range(40, 48)]:
            torch.cuda.synchronize()
            if busy and lo in (0, 40):
                for _ in range(60):                      # some 50 ms of products on torch's stream, the default one
                    torch.matmul(a, a, out=b)
            rows.append(engine.step([StepEntry("a", toks[lo:hi], list(range(hi - lo)))]).logits)
        torch.cuda.synchronize()
        return np.concatenate(rows)

    want, got = run(False), run(True)
    assert np.isfinite(want).all() and np.array_equal(got, want), np.abs(got - want).max(axis=1)
