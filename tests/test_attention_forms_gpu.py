"""The tcgen05 prefill attention of steps whose portions have very different lengths: the scratch in which the parts of query tiles meet."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _step(heads, kv, hd, ends, lens, seed):
    """Tensors of a step: segment i has lens[i] tokens and ends at position ends[i]; all segments read the same cached positions (one set of
    shuffled pages)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    pages = -(-max(ends) // 16)
    kc = torch.randn(pages, kv, 16, hd, device=DEV, generator=g).bfloat16()
    vc = torch.randn(pages, kv, 16, hd, device=DEV, generator=g).bfloat16()
    table = torch.randperm(pages, device=DEV, generator=g).to(torch.int32).expand(len(lens), pages).contiguous()
    q = torch.randn(sum(lens), heads * hd, device=DEV, generator=g).bfloat16()
    start = [0]
    for n in lens:
        start.append(start[-1] + n)
    return (q, kc, vc, table, torch.tensor(start, dtype=torch.int32, device=DEV),
            torch.tensor([e - n for e, n in zip(ends, lens)], dtype=torch.int32, device=DEV))


@pytest.mark.parametrize("lens,end", [([900] + [100] * 10, 8192), ([2, 1, 700, 3, 129, 1, 128, 257], 4000), ([1, 2, 2, 1, 300], 2900)])
@pytest.mark.parametrize("parts", [None, 2, 4])
def test_scratch_of_ragged_portions(lens, end, parts, monkeypatch):
    """Query tiles are shared among CTAs with scratch for the query tiles that exist, and no more than the limit: the same result as whole
    tiles, twice (the counters are back at zero), also where a caller's lengths promise too few tiles."""
    from infer_b200 import fast_ops
    heads, kv, hd = 12, 2, 128
    args = _step(heads, kv, hd, [end - 7 * i for i in range(len(lens))], lens, len(lens))
    st = fast_ops.device_state(DEV)
    st.status.zero_()
    asked = []
    workspace = st.workspace
    monkeypatch.setattr(st, "workspace", lambda n: (asked.append(n), workspace(n))[1])

    def run(split, seg_lens=lens):
        return fast_ops.attention_fast(*args, heads, kv, hd, None, 1 / math.sqrt(hd), 1 in lens, max(lens), end, lens.count(1), n_splits=1,
                                       tc_split=split, seg_lens=seg_lens)
    whole = run(1)
    asked.clear()
    got = run(parts)
    if parts is not None:
        tiles = heads * sum(-(-n // 128) for n in lens if n > 1)
        assert asked == [tiles * parts * (128 * hd + 256)]
    assert all(4 * n <= 4 * fast_ops.PREFILL_PARTS_MAX_FLOATS for n in asked)
    assert torch.equal(got, run(parts))
    assert (got.float() - whole.float()).abs().max() < 1e-2
    if parts is not None:                                                       # (lengths that are not the segments': the rest stays whole)
        assert (run(parts, [max(lens)]).float() - whole.float()).abs().max() < 1e-2
    assert int(st._counters.abs().sum()) == 0
    assert st.status.item() == 0


# ------------------------------------------------------------------------------------------------ the two forms of the kernel

@pytest.fixture(params=[64, 128], ids=["64 keys", "128 keys"])
def form(request, monkeypatch):
    """The kernel that walks over keys 64 or 128 at a time, whatever the plan would take; how often it was asked for."""
    from infer_b200 import fast_ops
    plan, asked = fast_ops.prefill_plan, []

    def pinned(sm_count, n_heads, head_dim, *more):
        asked.append(head_dim)
        return {"IB_HEAD_DIM": head_dim, "IB_ATTN_BN": 128} if request.param == 128 else {"IB_HEAD_DIM": head_dim}, plan(sm_count, n_heads, head_dim, *more)[1]
    monkeypatch.setattr(fast_ops, "prefill_plan", pinned)
    yield request.param
    assert asked


LAYOUTS = [(12, 2, 128), (14, 2, 64)]


@pytest.mark.parametrize("heads,kv,hd", LAYOUTS)
@pytest.mark.parametrize("window", [None, 1, 40, 64, 65, 129, 300])
def test_both_forms_with_windows(form, heads, kv, hd, window):
    """Query tiles and contexts that end on, before and behind the edges of key tiles of either size; windows likewise."""
    from test_attention_gpu import _run
    _run(heads, kv, hd, window, [(0, 2), (0, 63), (0, 64), (0, 65), (0, 128), (1, 128), (64, 129), (127, 257), (300, 17), (5, 1), (63, 2)])


@pytest.mark.parametrize("split", [1, 2, 3, 4])
@pytest.mark.parametrize("heads,kv,hd", LAYOUTS)
def test_both_forms_with_shared_query_tiles(form, heads, kv, hd, split):
    """1 to 17 tiles of 128 keys and twice as many of 64, whole and in parts, twice; with a window that cuts a part's first tile."""
    from infer_b200 import fast_ops
    from test_attention_gpu import _run
    segs = [(0, 1100), (1900, 200), (1, 1), (1530, 2), (500, 1)]
    first = _run(heads, kv, hd, None, segs, 2, seed=5, tc_split=split)
    assert torch.equal(first, _run(heads, kv, hd, None, segs, 2, seed=5, tc_split=split, count_decode=True))
    assert int(fast_ops.device_state(DEV)._counters.abs().sum()) == 0
    _run(heads, kv, hd, 1200, [(700, 900), (2000, 130)], seed=6, tc_split=split)


@pytest.mark.parametrize("window", [None, 33, 130, 300])
@pytest.mark.parametrize("sizes", [(4, 2, 64), (8, 1, 128)])
def test_both_forms_with_distance_bias_and_sink(form, sizes, window):
    import test_fozerax_kernels_gpu as t
    t.test_tensor_core_attention_with_distance_bias_and_sink(sizes, window)


@pytest.mark.parametrize("window,keep", [(None, 0), (150, 40), (128, 3), (300, 200), (40, 130), (520, 1)])
@pytest.mark.parametrize("sizes", [(4, 2, 64), (2, 1, 128)])
def test_both_forms_with_slopes_and_kept_first_keys(form, sizes, window, keep):
    import test_biravik_kernels_gpu as t
    t.test_prompt_portions_on_the_tensor_core_kernel_with_slopes_and_kept_first_keys(sizes, window, keep)
