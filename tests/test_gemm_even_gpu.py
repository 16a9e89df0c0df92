"""The streaming product with equal runs of stages: tiles that several CTAs share come out like the others, at every way the runs can fall."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# tiles beyond and below the CTAs, a last partial tile, K that ends inside a stage, runs longer than a tile and shorter than a part of one
@pytest.mark.parametrize("N,K,stages", [(5120, 1536, 2), (4999, 2056, 3), (24, 20000, 14), (8, 1544, 2), (40, 640, 5), (3584, 18944, 13), (300, 4096, 16)])
@pytest.mark.parametrize("M", [1, 8, 9, 16])
def test_runs(M, N, K, stages):
    from infer_b200 import fast_ops
    gen = torch.Generator(device=DEV).manual_seed(N + K)
    x = torch.randn(M, K, generator=gen, device=DEV).bfloat16()
    w = (torch.randn(N, K, generator=gen, device=DEV) * 0.03).bfloat16()
    r = torch.randn(M, N, generator=gen, device=DEV)
    size = x.double().abs() @ w.double().abs().T + r.double().abs()
    got = fast_ops.linear_skinny(x, w, None, r, torch.float32, None, even=stages)
    # exact products, float sums: at most K / 16 MMAs and eight warps' sums, a few additions more
    assert ((got.double() - (x.double() @ w.double().T + r.double())).abs() / size).max() <= (K / 16 + 16) * 2.0 ** -23
    for _ in range(3):
        assert torch.equal(fast_ops.linear_skinny(x, w, None, r, torch.float32, None, even=stages), got)      # whoever arrives last
    assert torch.equal(fast_ops.linear_skinny(x[:1].contiguous(), w, None, r[:1].contiguous(), torch.float32, None, even=stages), got[:1])
    st = fast_ops.device_state(torch.device(DEV))
    assert int(st.status) == 0 and int(st._counters.abs().sum()) == 0
    if N % 16 == 0:
        act = fast_ops.linear_skinny(x, w, swiglu=True, even=stages)
        plain = fast_ops.linear_skinny(x, w, swiglu=True, even=0)
        assert (act.float() - plain.float()).abs().max() <= 2.0 ** -7 * plain.float().abs().max()             # two roundings to bfloat16 apart
