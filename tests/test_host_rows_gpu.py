"""The arrays that steps' logits arrive in are ordinary memory to everyone else."""
from __future__ import annotations

import gc

import numpy as np
import pytest
import torch

from tiny_models import CONFIGS, random_tokens, write_model

pytestmark = pytest.mark.gpu


@pytest.fixture()
def engine(tmp_path):
    from liyab_b200.engine import Replayer
    r = Replayer(write_model(str(tmp_path), "D", "bfloat16"), "bfloat16", max_tokens=256)
    r.cache.open("a")
    yield r
    r.close()


def test_an_asynchronous_copy_has_read_its_array(engine):
    """The array is dropped while the copy waits behind other work, and later steps' logits arrive: the copy holds the first step's all the same."""
    from liyab_b200.engine import StepEntry
    toks = random_tokens(3, 12, CONFIGS["D"][0]["vocab_size"])
    first = engine.step([StepEntry("a", toks[:4], [0, 1, 2, 3])]).logits
    assert not torch.from_numpy(first).is_pinned()
    want = first.copy()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)
        there = torch.from_numpy(first).to("cuda", non_blocking=True)
    address = first.ctypes.data
    del first
    gc.collect()
    seen = set()
    for i in (4, 8):
        later = engine.step([StepEntry("a", toks[i:i + 4], [0, 1, 2, 3])]).logits
        seen.add(later.ctypes.data)
        assert not np.array_equal(later, want)
        del later
    torch.cuda.synchronize()
    assert address in seen and np.array_equal(there.cpu().numpy(), want)


def test_arrays_may_die_while_a_stream_is_captured(engine):
    from liyab_b200.engine import StepEntry
    out = engine.step([StepEntry("a", [1, 2], [0, 1])]).logits
    engine.close()
    x = torch.ones(8, device="cuda")
    y = torch.zeros(8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y.add_(x)
        del out                                # its owner is closed: the memory goes back to the system here
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, x)


def test_a_buffer_for_a_device_that_is_not_there_is_refused():
    import ctypes as C
    from liyab_b200 import _capi
    out = C.c_void_p(1)
    assert _capi.lib().lb_host_buffer_create(99, 1 << 16, C.byref(out)) != 0 and not out.value
    assert torch.ones(2, device="cuda").sum().item() == 2.0          # no error is left behind, and the device is the one it was
