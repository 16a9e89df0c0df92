"""Matrix products on pairs of SMs (plan codes 1024 + 2 x width) against the plain kernel: one tile, ragged tiles whose second half
of rows or features lies outside, a K tail, more tiles than pairs; bias, residual in place, SwiGLU. The same bound as for the other
tensor-core products: 2e-6 of the conditioning (float sums of at most 3,000 terms in blocks of 16)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("width", [128, 160, 192, 224, 256])
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (129, 16, 72), (257, 496, 64), (300, 272, 72), (1100, 3000, 520), (2048, 1536, 1536), (4000, 4112, 200)])
def test_pairs_match_plain(M, N, K, width):
    from infer_b200 import fast_ops, ops
    g = torch.Generator(device=DEV).manual_seed(M + N + K + width)
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(N, K, device=DEV, generator=g) * 0.05).bfloat16()
    bias, res = torch.randn(N, device=DEV, generator=g), torch.randn(M, N, device=DEV, generator=g)
    cond = x.float().abs() @ w.float().abs().T + 1.0
    st = fast_ops.device_state(DEV)
    plan = (0, 1024 + 2 * width, 1, 0, 0)
    got = fast_ops.gemm_tc(x, w, bias, None, torch.float32, plan=plan)
    assert ((got - ops.linear_plain(x, w, bias, None, torch.float32)).abs() / cond).max().item() < 2e-6
    assert torch.equal(got, fast_ops.gemm_tc(x, w, bias, None, torch.float32, plan=plan))
    own = res.clone()
    fast_ops.gemm_tc(x, w, None, own, torch.float32, out=own, plan=plan)
    assert ((own - ops.linear_plain(x, w, None, res, torch.float32)).abs() / cond).max().item() < 2e-6
    if N % 16 == 0:
        act = fast_ops.gemm_tc(x, w, out_dtype=torch.bfloat16, plan=plan, swiglu=True)
        assert torch.equal(act, fast_ops.gemm_tc(x, w, out_dtype=torch.bfloat16, plan=(0, 128, 1, 0, 0), swiglu=True))
    assert st.status.item() == 0
