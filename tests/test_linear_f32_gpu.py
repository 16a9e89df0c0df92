"""The kernels of the 32-bit path's matrix product: every one of them, at the edges of their tiles, gives the same bits, and those lie as
close to the 64-bit product as chains of 16 multiply-adds, one sum and K / 32 more additions allow."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M", [1, 2, 3, 5, 8, 9, 31, 33, 64, 65, 130])
@pytest.mark.parametrize("N,K,odd", [(16, 4, 0), (70, 36, 0), (129, 256, 0), (33, 1540, 0), (2405, 260, 0), (17, 31, 0), (65, 290, 0), (40, 64, 1)])
def test_every_kernel_gives_the_same_bits(M, N, K, odd):
    from infer_b200 import ops
    gen = torch.Generator(device=DEV).manual_seed(M * 1000 + N + K)
    x = torch.randn(M * K + odd, generator=gen, device=DEV)[odd:].view(M, K)         # odd: bases that are not 16-byte aligned
    w = torch.randn(N * K + odd, generator=gen, device=DEV)[odd:].view(N, K)
    b, r = torch.randn(N, generator=gen, device=DEV), torch.randn(M, N, generator=gen, device=DEV)
    want = x.double() @ w.double().T + b.double() + r.double()
    size = x.double().abs() @ w.double().abs().T + b.double().abs() + r.double().abs()
    got = ops.linear_plain(x, w, b, r)
    roundings = 16 + 1 + -(-K // 32) + 2
    assert ((got.double() - want).abs() / size).max() <= roundings * 2.0 ** -24
    for kind in ([1, 2] if M <= 8 else []) + [3, 4, 5]:
        assert torch.equal(ops.linear_plain(x, w, b, r, kind=kind), got), kind
        own = r.clone()
        assert torch.equal(ops.linear_plain(x, w, b, own, out=own, kind=kind), got), kind
    assert torch.equal(ops.linear_plain(x[-1:].contiguous(), w, b, r[-1:].contiguous()), got[-1:])
    x[0, K // 2] = float("inf")
    assert not torch.isfinite(ops.linear_plain(x, w, b, r)[0]).any() and torch.equal(ops.linear_plain(x, w, b, r)[1:], got[1:])


@pytest.mark.parametrize("M,N,K", [(1, 2048, 1536), (3, 40, 64), (8, 4096, 260), (9, 2048, 1536)])
def test_a_matrix_that_the_kernel_before_has_just_written(M, N, K):
    """w is itself a product: nothing of it may be read before the kernel that writes it has ended, whatever was there before."""
    from infer_b200 import ops
    gen = torch.Generator(device=DEV).manual_seed(M + N + K)
    x, a, b = (torch.randn(n, k, generator=gen, device=DEV) for n, k in ((M, K), (N, 1000), (K, 1000)))
    w = ops.linear_plain(a, b)
    torch.cuda.synchronize()
    want = ops.linear_plain(x, w)
    torch.cuda.synchronize()
    for _ in range(20):
        again = torch.full_like(w, float("nan"))
        assert torch.equal(ops.linear_plain(x, ops.linear_plain(a, b, out=again)), want)
    assert torch.equal(ops.linear_plain(x, w, w_ready=True), want)


# (the matrices above of 1024 x 1024 and more go to the tensor cores by themselves: here the kernels of this file are named, or the matrix is smaller)
@pytest.mark.parametrize("M,N,K,kind", [(1, 2048, 1536, 1), (8, 2048, 1536, 2), (9, 2048, 1536, 3), (40, 2048, 1536, 4), (9, 2048, 1536, 5), (9, 900, 1536, 0), (70, 1100, 900, 0)])
def test_every_kernel_waits_for_the_matrix_that_the_kernel_before_writes(M, N, K, kind):
    from infer_b200 import ops
    gen = torch.Generator(device=DEV).manual_seed(M + N + K)
    x, a, b = (torch.randn(n, k, generator=gen, device=DEV) for n, k in ((M, K), (N, 1000), (K, 1000)))
    w = ops.linear_plain(a, b)
    torch.cuda.synchronize()
    want = ops.linear_plain(x, w, kind=kind)
    torch.cuda.synchronize()
    for _ in range(20):
        again = torch.full_like(w, float("nan"))
        assert torch.equal(ops.linear_plain(x, ops.linear_plain(a, b, out=again), kind=kind), want)
    assert torch.equal(ops.linear_plain(x, w, w_ready=True, kind=kind), want)
