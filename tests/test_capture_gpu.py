"""Captured steps of the 32-bit path (the bits of the eager path, results that later steps leave alone), and the streams that captures
and side branches run on (never one and the same)."""
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("name", ["a", "b", "c"])
def test_float32_steps_are_captured_and_their_results_stay(name):
    from infer_b200 import StepEntry
    from test_engine_gpu import _engine
    cfg = H.TINY[name]
    engines = [_engine(name, torch.float32, cuda_graphs=g) for g in (False, True)]
    assert engines[1].use_graphs
    ids = {r: H.random_ids(cfg, 30, 70 + i) for i, r in enumerate("xy")}
    kept = []
    for eng in engines:
        outs = []
        for r in "xy":
            eng.add_request(r)
        outs.append(eng.step([StepEntry(r, ids[r][:20], [19]) for r in "xy"]))
        for t in range(20, 30):
            outs.append(eng.step([StepEntry(r, ids[r][t:t + 1], [0]) for r in "xy"]))
        eng.check_status()
        kept.append(outs)
    assert len(engines[1]._graphs) > 0
    for t, (a, b) in enumerate(zip(*kept)):
        assert torch.equal(a, b), f"step {t}"


def test_streams_of_captures_and_side_branches_differ():
    from infer_b200 import fast_ops
    from infer_b200.parts.block import _side_streams
    device = torch.device(DEV)
    sides = _side_streams(device)
    for _ in range(31):                                  # (torch hands out 32 streams in turn)
        torch.cuda.Stream(device)
    handles = [s.cuda_stream for s in (*sides, fast_ops.capture_stream(device), fast_ops.own_stream(device))]
    assert len(set(handles)) == 4
    assert fast_ops.capture_stream(device) is fast_ops.capture_stream(device)
