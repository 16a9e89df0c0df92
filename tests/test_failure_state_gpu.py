"""What a kernel that gave up leaves behind (its status word, counts that stay short) is gone once the failure has been reported. The leftovers
are written by hand: no kernel is made to fail."""
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_counts_are_cleared_with_the_status_word():
    from infer_b200 import fast_ops
    from test_engine_gpu import _engine
    eng = _engine("b", torch.bfloat16)
    st = fast_ops.device_state(DEV)
    side = fast_ops.own_stream(DEV)
    fast_ops.register_side_stream(side)
    with torch.cuda.stream(side):
        beside = fast_ops.device_state(DEV)
    assert beside is not st and beside.status is st.status
    x = torch.randn(130, 4096, device=DEV).bfloat16()
    w = (torch.randn(512, 4096, device=DEV) * 0.05).bfloat16()
    assert fast_ops.gemm_choice(130, 512, 4096, st.sm_count)[4] > 0          # its K slices meet through the counters
    want = fast_ops.gemm_tc(x, w, out_dtype=torch.float32)
    grown = st._counters                                          # (a captured graph may hold the address of what a larger call replaced)
    st.counters(grown.numel() + 1)
    where = [t.data_ptr() for t in (grown, st._counters, beside._counters)]
    for t in (grown, st._counters, beside._counters):
        t.fill_(1)
    st.status.fill_(103)
    with pytest.raises(RuntimeError, match="accumulator wait"):
        eng.check_status()
    assert int(st.status) == 0
    for t, at in zip((grown, st._counters, beside._counters), where):
        assert t.data_ptr() == at and not t.any()
    assert torch.equal(fast_ops.gemm_tc(x, w, out_dtype=torch.float32), want)
    eng.check_status()
    # the engine goes on
    cfg = H.TINY["b"]
    from infer_b200 import StepEntry
    eng.add_request("r")
    assert torch.isfinite(eng.step([StepEntry("r", H.random_ids(cfg, 8, 1), [7])])).all()
    eng.check_status()


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_a_device_first_met_inside_a_capture(monkeypatch, mode):
    """The status word and the counters are there, and zero, before the first replay, and no replay touches them."""
    from infer_b200 import fast_ops, ops
    x, w = torch.randn(3, 1536, device=DEV), torch.randn(1536, 1536, device=DEV)
    want = ops.linear_plain(x, w)
    torch.cuda.synchronize()
    monkeypatch.setattr(fast_ops, "_STATES", {})
    graph, out = torch.cuda.CUDAGraph(), torch.empty_like(want)
    with torch.cuda.graph(graph, capture_error_mode=mode):
        ops.linear_plain(x, w, out=out)
    assert len(fast_ops._STATES) == 1
    st = fast_ops.device_state(DEV)
    assert int(st.status) == 0 and not st._counters.any()
    st.status.fill_(7)
    st._counters.fill_(2)
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert int(st.status) == 7 and int(st._counters.min()) == 2
