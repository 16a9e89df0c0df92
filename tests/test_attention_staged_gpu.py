"""Plain attention over float pages: every number of heads that a block takes together gives the bits of the kernel that takes one query
head and waits for its loads, and those are close to float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _oracle(q, kc, vc, table, seg, pos, nh, nkv, window, scale, keep, bias, sink, slopes):
    T, hd = q.shape[0], kc.shape[3]
    out = torch.empty(T, nh, vc.shape[3], dtype=torch.float64, device=q.device)
    for t in range(T):
        p = int(pos[t])
        rows = table[int(seg[t]), :p // 16 + 1].long()
        lo = max(0, p - window + 1) if window else 0
        j = torch.arange(p + 1, device=q.device)
        seen = (j >= lo) | (j < min(keep, lo))
        for h in range(nh):
            g = h // (nh // nkv)
            k, v = (c[rows, g].reshape(-1, c.shape[3])[:p + 1].double() for c in (kc, vc))
            s = k @ q[t, h * hd:(h + 1) * hd].double() * scale
            if bias is not None:
                s = s + bias[(p - j).clamp(max=bias.shape[0] - 1), h].double()
            if slopes is not None:
                s = s - slopes[h].double() * (p - j)
            s = s.masked_fill(~seen, float("-inf"))
            top = s.max() if sink is None else torch.maximum(s.max(), sink[h].double())
            e = torch.exp(s - top)
            out[t, h] = (e @ v) / (e.sum() + (torch.exp(sink[h].double() - top) if sink is not None else 0.0))
    return out.view(T, -1)


# query heads of a kv head: 1 to 8; head and value sizes around the 128 threads; a size that is not of 16-byte pieces takes the other kernel
@pytest.mark.parametrize("nh,nkv,hd,vd", [(4, 4, 64, 64), (4, 2, 128, 128), (6, 2, 32, 160), (4, 1, 100, 20), (5, 1, 64, 64), (12, 2, 128, 128), (7, 1, 128, 128),
                                          (8, 1, 8, 4), (2, 1, 30, 30), (2, 1, 200, 200)])
@pytest.mark.parametrize("window,keep,extra", [(None, 0, ""), (100, 0, "bias"), (50, 7, "sink"), (300, 140, "slopes")])
def test_heads_together(nh, nkv, hd, vd, window, keep, extra):
    from infer_b200 import ops
    gen = torch.Generator(device=DEV).manual_seed(nh * 1000 + hd + keep)
    rand = lambda *s: torch.randn(*s, generator=gen, device=DEV)  # noqa: E731
    segs, per, T = 3, 26, 400                                        # contexts of up to 416 keys: a tile of 128 more than three
    kc, vc = rand(90, nkv, 16, hd), rand(90, nkv, 16, vd)
    table = torch.randperm(90, generator=gen, device=DEV)[:segs * per].view(segs, per).int().contiguous()
    q, seg = rand(T, nh * hd), (torch.arange(T, device=DEV) % segs).int()
    pos = torch.randint(0, per * 16, (T,), generator=gen, device=DEV).int()
    pos[:6] = torch.tensor([0, 127, 128, 255, 256, per * 16 - 1], device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    bias, sink, slopes = (rand(33, nh) if extra == "bias" else None, rand(nh) if extra == "sink" else None,
                          rand(nh).abs() * 0.1 if extra == "slopes" else None)

    def run(a, b, **kw):
        return ops.attention_plain(q[a:b].contiguous(), kc, vc, table, seg[a:b].contiguous(), pos[a:b].contiguous(), nh, nkv, hd, window, 0.1,
                                   v_head_dim=vd, dist_bias=bias, sink=sink, slopes=slopes, keep_first=keep, status=status, **kw)
    full = run(0, T)
    # tokens that are segments of their own, many of them: the kernel that takes a head by itself
    alone = ops.attention_plain(q, kc, vc, table.repeat(T // segs + 1, 1)[:T].contiguous(), torch.arange(T, device=DEV).int(), pos, nh, nkv, hd, window, 0.1,
                                v_head_dim=vd, dist_bias=bias, sink=sink, slopes=slopes, keep_first=keep,
                                single_only=torch.arange(T + 1, device=DEV).int())
    assert torch.equal(alone, full)
    for n in (1, 3, 20, 60, 130):                                    # (few tokens: fewer heads a block)
        assert torch.equal(run(0, n), full[:n]), n
    want = _oracle(q[:12], kc, vc, table, seg[:12], pos[:12], nh, nkv, window, 0.1, keep, bias, sink, slopes)
    # a score's hd products and a sum over up to 416 keys, in float: a few hundred roundings of 2^-24 each
    assert (full[:12].double() - want).abs().max() <= 500 * 2.0 ** -24 * max(1.0, want.abs().max().item())
    assert int(status) == 0


def test_a_page_that_is_not_there():
    from infer_b200 import ops
    q, kc = torch.randn(2, 2 * 64, device=DEV), torch.randn(4, 1, 16, 64, device=DEV)
    table = torch.tensor([[0, 9], [1, 2]], dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    seg, pos = torch.arange(2, device=DEV).int(), torch.tensor([20, 20], device=DEV).int()
    got = ops.attention_plain(q, kc, kc, table, seg, pos, 2, 1, 64, None, 0.1, status=status)
    assert int(status) == 3 and torch.isfinite(got).all()
    fine = ops.attention_plain(q[1:].contiguous(), kc, kc, table[1:].contiguous(), seg[:1], pos[1:].contiguous(), 2, 1, 64, None, 0.1)
    assert torch.equal(got[1:], fine)


@pytest.mark.parametrize("window,keep,extra", [(None, 0, ""), (50, 7, "sink")])
def test_as_many_heads_together_as_fit(window, keep, extra):
    """Six query heads of 144 floats do not fit beside their keys: three do."""
    test_heads_together(12, 2, 144, 144, window, keep, extra)


@pytest.mark.parametrize("nh,nkv,hd", [(4, 4, 64), (12, 2, 128), (14, 2, 64)])
def test_a_few_keys(nh, nkv, hd):
    """Contexts of one tile: only the keys that a token sees are copied. What shared memory held before is not looked at."""
    from infer_b200 import ops
    gen = torch.Generator(device=DEV).manual_seed(nh + hd)
    rand = lambda *s: torch.randn(*s, generator=gen, device=DEV)  # noqa: E731
    T = 24
    kc, vc = rand(T * 8, nkv, 16, hd), rand(T * 8, nkv, 16, hd)
    table = torch.randperm(T * 8, generator=gen, device=DEV).view(T, 8).int().contiguous()
    q, seg = rand(T, nh * hd), torch.arange(T, device=DEV).int()
    pos = torch.tensor([0, 1, 2, 3, 6, 7, 8, 14, 15, 16, 17, 30, 31, 32, 33, 63, 64, 65, 100, 120, 125, 126, 127, 5], device=DEV).int()
    bad_k, bad_v = torch.full_like(kc, float("nan")), torch.full_like(vc, float("nan"))
    for window, keep in ((None, 0), (10, 0), (10, 3)):
        # NaN first, so that keys that are not there would show
        ops.attention_plain(q, bad_k, bad_v, table, seg, pos, nh, nkv, hd, None, 0.1)
        got = ops.attention_plain(q, kc, vc, table, seg, pos, nh, nkv, hd, window, 0.1, keep_first=keep)
        want = _oracle(q, kc, vc, table, seg, pos, nh, nkv, window, 0.1, keep, None, None, None)
        # hd products and a sum over up to 128 keys, in float
        assert (got.double() - want).abs().max() <= 300 * 2.0 ** -24 * max(1.0, want.abs().max().item())
