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
