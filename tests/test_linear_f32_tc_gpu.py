"""The 32-bit path's product by large matrices, on the tensor cores: close to the 64-bit product, no further off than the multiply-add
kernels, the same bits for a row whatever the other rows are, and the plain product's infinities and NaN."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# whole tiles; K and N that end inside a block and a tile, with rows that are and are not 16-byte aligned; one and eight groups of K
SIZES = [(1024, 1024), (2048, 1536), (1100, 1500), (1025, 1028), (1030, 1031), (1536, 8960), (19000, 1088)]


def _operands(M, N, K, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    make = lambda *s: torch.randn(*s, generator=gen, device=DEV)  # noqa: E731
    return make(M, K), make(N, K) * 0.02, make(N), make(M, N)


@pytest.mark.parametrize("N,K", SIZES)
def test_product(N, K):
    from infer_b200 import ops
    M = 130
    x, w, b, r = _operands(M, N, K, N + K)
    exact, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    got = ops.linear_plain(x, w)
    # in units of 2^-24 of the sum of sizes: four tensor-core additions a block of 64 that may lose two each, a rounding per block
    # and per group, the second accumulators' K / 8 additions at weight 2^-8, and what the three parts leave out
    units = 8 + K / 64 + 8 + K / 8 * 2 / 256 + 3
    assert ((got.double() - exact).abs() / size).max() <= units * 2.0 ** -24
    plain = ops.linear_plain(x, w, kind=3)
    assert (got.double() - exact).norm() <= (plain.double() - exact).norm()
    full = ops.linear_plain(x, w, b, r)
    assert torch.equal(full, (got + b) + r)
    own = r.clone()
    assert torch.equal(ops.linear_plain(x, w, b, own, out=own), full) and torch.equal(own, full)
    for m in (1, 2, 15, 16, 17, 32, 33, 64, 65, 129):                  # every tile of tokens and its edges
        assert torch.equal(ops.linear_plain(x[M - m:].contiguous(), w), got[M - m:]), m
    shifted = torch.empty(M * K + 1, device=DEV)[1:].view(M, K)        # a base that is not 16-byte aligned
    shifted.copy_(x)
    assert torch.equal(ops.linear_plain(shifted, w), got)
    assert ops.linear_plain(x[:0].contiguous(), w).shape == (0, N)


@pytest.mark.parametrize("M", [2, 70])
def test_not_finite(M):
    from infer_b200 import ops
    x, w, _, _ = _operands(M, 1100, 1500, M)
    got = ops.linear_plain(x, w)
    x[0, 3], w[5, 7], w[6, 0] = float("inf"), float("nan"), -float("inf")
    bad = ops.linear_plain(x, w)
    assert torch.equal(torch.nan_to_num(bad[0], nan=3.0), torch.nan_to_num(ops.linear_plain(x, w, kind=3)[0], nan=3.0))
    assert torch.isnan(bad[:, 5]).all() and torch.isinf(bad[1:, 6]).all()
    keep = [n for n in range(1100) if n not in (5, 6)]
    assert torch.equal(bad[1:, keep], got[1:, keep])


@pytest.mark.parametrize("scale", [1e-37, 1e-30, 1e30, 1e36])
def test_ends_of_the_range(scale):
    from infer_b200 import ops
    x, w, _, _ = _operands(20, 1024, 1024, 5)
    x = x * scale
    exact = x.double() @ w.double().T
    assert (ops.linear_plain(x, w).double() - exact).norm() <= (ops.linear_plain(x, w, kind=3).double() - exact).norm()


def test_a_matrix_that_the_kernel_before_has_just_written():
    from infer_b200 import ops
    x, _, _, _ = _operands(3, 8, 1536, 1)
    a, b = _operands(1, 2048, 1000, 2)[1], _operands(1, 1536, 1000, 3)[1]
    w = ops.linear_plain(a, b)
    want = ops.linear_plain(x, w)
    torch.cuda.synchronize()
    for _ in range(20):
        again = torch.full_like(w, float("nan"))
        assert torch.equal(ops.linear_plain(x, ops.linear_plain(a, b, out=again)), want)
    assert torch.equal(ops.linear_plain(x, w, w_ready=True), want)


def test_captured():
    from infer_b200 import ops
    x, w, b, r = _operands(5, 1536, 1536, 9)
    want = ops.linear_plain(x, w, b, r)
    out = torch.empty_like(want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.linear_plain(x, w, b, r, out=out, w_ready=True)
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


# one group, clusters of two and of eight, the last tile of features a repeat of the one before; every tile of tokens
@pytest.mark.parametrize("N,K", [(19000, 1088), (2048, 1536), (1025, 1031), (1536, 8960)])
@pytest.mark.parametrize("M", [1, 5, 20, 70])
def test_not_finite_has_the_bits_of_the_multiply_adds(M, N, K):
    """Rows with a NaN, infinities of one and of both signs, elements that are beyond every bfloat16 number (their results are finite or overflow);
    with bias and with the residual in place."""
    from infer_b200 import ops
    x, w, b, r = _operands(M, N, K, M + N)
    clean = ops.linear_plain(x, w, b, r)
    x[0, K - 1] = float("nan")
    if M > 1:
        x[1, 3], x[2, 7], x[2, 900], x[3, 40:60] = float("inf"), float("inf"), -float("inf"), 3.4e38
    w[N - 1, 5], w[130, 0], w[700, 1] = float("nan"), -float("inf"), 3.4028e38
    got, plain = ops.linear_plain(x, w), ops.linear_plain(x, w, kind=3)
    assert torch.equal(torch.isnan(got), torch.isnan(plain))
    again = (x.abs().nan_to_num(4e38).amax(1) > 3e38)[:, None] | (w.abs().nan_to_num(4e38).amax(1) > 3e38)[None, :]
    assert torch.equal(torch.where(again, got, 0.0).nan_to_num(), torch.where(again, plain, 0.0).nan_to_num())
    full, own = ops.linear_plain(x, w, b, r), r.clone()
    assert torch.equal(torch.nan_to_num(full), torch.nan_to_num((got + b) + r))
    assert torch.equal(torch.nan_to_num(ops.linear_plain(x, w, b, own, out=own)), torch.nan_to_num(full)) and torch.equal(torch.isnan(own), torch.isnan(full))
    kept = [n for n in range(N) if n not in (N - 1, 130, 700)]
    assert torch.equal(full[4:, kept], clean[4:, kept])


def _values(kind, gen, *shape):
    r = torch.randn(*shape, generator=gen, device=DEV)
    if kind == "positive":
        return r.abs()
    if kind in ("wide", "wide positive"):
        r = r * torch.exp(3.0 * torch.randn(*shape, generator=gen, device=DEV))
        return r.abs() if kind == "wide positive" else r
    if kind == "outliers":
        r[:, ::97] *= 300.0
    if kind == "one value":
        r.fill_(1.0038986)                                        # the largest parts: 2^-8 and 2^-17 of the value are left to the second and third
    return r


@pytest.mark.parametrize("kx,kw", [("normal", "normal"), ("outliers", "normal"), ("wide", "normal"), ("wide", "wide"), ("positive", "positive"),
                                   ("wide positive", "wide positive"), ("one value", "one value")])
@pytest.mark.parametrize("N,K", [(1024, 1024), (17920, 1536), (1536, 8960)])
def test_other_operands(N, K, kx, kw):
    """The error's bound holds for operands of one sign, for widely scaled ones and for those of which most is left out; a mean of errors of one
    sign is at most half of what the additions can lose; from K = 3584 on no set of operands is further off than on multiply-adds."""
    from infer_b200 import ops
    gen = torch.Generator(device=DEV).manual_seed(N + K)
    x, w = _values(kx, gen, 40, K), _values(kw, gen, N, K)
    exact, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    off = ops.linear_plain(x, w).double() - exact
    units = 8 + K / 64 + 8 + K / 8 * 2 / 256 + 3                   # as in test_product
    assert (off.abs() / size).max() <= units * 2.0 ** -24
    # four additions a block, each loses up to two units, one on average; what is left out: one more
    assert abs((off / size).mean().item()) <= (8 / 2 + 1 + 1) * 2.0 ** -24
    plain = ops.linear_plain(x, w, kind=3).double() - exact
    if K >= 3584:
        assert off.norm() <= plain.norm() * 1.001
