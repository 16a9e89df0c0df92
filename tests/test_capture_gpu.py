"""The streams that captures and side branches run on are never one and the same."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


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
