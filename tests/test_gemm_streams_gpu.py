"""The streaming product keeps nothing between calls and shares nothing with others: calls on several streams at once, and calls beside counters
that another kernel's wait left raised, give the bits that a call by itself gives."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# K in clusters, in whole rows of several stages, in one stage; tiles beyond and below the CTAs; a last partial tile; K that ends inside a stage
SIZES = [(3584, 18944), (5120, 13824), (5120, 1536), (4999, 2056), (24, 20000), (300, 4096)]


def _operands(M, N, K):
    gen = torch.Generator(device=DEV).manual_seed(M + N + K)
    return (torch.randn(M, K, generator=gen, device=DEV).bfloat16(), (torch.randn(N, K, generator=gen, device=DEV) * 0.03).bfloat16(),
            torch.randn(N, generator=gen, device=DEV), torch.randn(M, N, generator=gen, device=DEV))


@pytest.mark.parametrize("N,K", SIZES)
@pytest.mark.parametrize("M", [1, 8, 9, 16])
def test_nothing_is_left_behind(M, N, K):
    from infer_b200 import fast_ops
    x, w, b, r = _operands(M, N, K)
    size = x.double().abs() @ w.double().abs().T + r.double().abs()
    got = fast_ops.linear_skinny(x, w, None, r, torch.float32)
    # exact products, float sums: at most K / 16 MMAs and eight warps' sums, a few additions more
    assert ((got.double() - (x.double() @ w.double().T + r.double())).abs() / size).max() <= (K / 16 + 16) * 2.0 ** -23
    assert torch.equal(fast_ops.linear_skinny(x[:1].contiguous(), w, None, r[:1].contiguous(), torch.float32), got[:1])
    plain, low = fast_ops.linear_skinny(x, w, b, None, torch.float32), fast_ops.linear_skinny(x, w, b)
    act = fast_ops.linear_skinny(x, w, swiglu=True) if N % 16 == 0 else None
    st = fast_ops.device_state(torch.device(DEV))
    st._counters.fill_(1)
    try:
        for _ in range(3):
            assert torch.equal(fast_ops.linear_skinny(x, w, None, r, torch.float32), got)
        assert torch.equal(fast_ops.linear_skinny(x, w, b, None, torch.float32), plain) and torch.equal(fast_ops.linear_skinny(x, w, b), low)
        assert act is None or torch.equal(fast_ops.linear_skinny(x, w, swiglu=True), act)
        assert int(st._counters.min()) == 1 and int(st._counters.max()) == 1
    finally:
        st._counters.zero_()
    assert int(st.status) == 0


@pytest.mark.parametrize("N,K", SIZES[:2])
def test_two_streams(N, K):
    from infer_b200 import fast_ops
    cases = [_operands(M, N, K) for M in (1, 8)]
    want = [fast_ops.linear_skinny(x, w, None, r, torch.float32) for x, w, _, r in cases]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in cases]
    got = [[], []]
    for _ in range(30):
        for i, (x, w, _, r) in enumerate(cases):
            with torch.cuda.stream(streams[i]):
                got[i].append(fast_ops.linear_skinny(x, w, None, r, torch.float32))
    torch.cuda.synchronize()
    for i in range(2):
        assert all(torch.equal(g, want[i]) for g in got[i])


def test_a_cluster_that_is_asked_for_is_what_runs():
    """At 3584 x 18944 two CTAs share a tile unless the caller says how many do. Sums in another order have other bits."""
    from infer_b200 import fast_ops
    x, w, _, r = _operands(8, *SIZES[0])
    by_cluster = {c: fast_ops.linear_skinny(x, w, None, r, torch.float32, cluster=c) for c in (1, 2, 4)}
    assert torch.equal(fast_ops.linear_skinny(x, w, None, r, torch.float32), by_cluster[2])
    assert not torch.equal(by_cluster[1], by_cluster[2]) and not torch.equal(by_cluster[2], by_cluster[4])
