"""How the prefill attention of a step is laid onto the SMs (host arithmetic): forms and parts at the edges of the rule."""
import pytest

SMS = 148


@pytest.mark.parametrize("heads,lens,ctx,window,form,parts", [
    (12, [512], 512, None, 128, (1,)),                 # few long query tiles, all at once
    (12, [33], 33, None, 64, (1,)),
    (12, [200] * 10, 200, None, 64, (1,)),             # short tiles
    (28, [2048], 2048, None, 64, (1,)),                # many CTAs: two an SM
    (12, [4096], 15873, None, 64, (3, 4)),             # a second round with 88 of 296 places filled, otherwise
    (12, [1024], 9216, None, 64, (3,)),
])
def test_forms_and_parts(heads, lens, ctx, window, form, parts):
    from infer_b200 import fast_ops
    sizes, split = fast_ops.prefill_plan(SMS, heads, 128, lens, ctx, window)
    assert sizes.get("IB_ATTN_BN", 64) == form and sizes["IB_HEAD_DIM"] == 128
    assert split in parts


def test_parts_stay_within_their_scratch_and_the_kernels_limit():
    from infer_b200 import fast_ops
    for heads in (1, 12, 28, 64):
        for n in (2, 130, 1024, 4096, 8192):
            for before in (0, 5000, 30000):
                sizes, split = fast_ops.prefill_plan(SMS, heads, 128, [n], n + before, None)
                assert 1 <= split <= fast_ops.ATTENTION_TC_MAX_SPLIT
                if split > 1 and "IB_ATTN_BN" not in sizes:
                    assert heads * -(-n // 128) * split * (128 * 128 + 256) <= fast_ops.PREFILL_PARTS_MAX_FLOATS


def test_makespan():
    from infer_b200.fast_ops import _makespan
    assert _makespan([3.0, 2.0], 4) == 3.0
    assert _makespan([3.0, 3.0, 2.0, 2.0, 1.0], 2) == 6.0


@pytest.mark.parametrize("heads,lens,ctx", [(12, [3346] + list(range(2, 101, 3)), 26219), (12, [3000] + [30] * 30, 16384), (12, [900] + [100] * 10, 8192),
                                            (28, [512, 2, 2, 2], 9000), (64, [2048] + [2] * 40, 30000)])
def test_scratch_of_ragged_portions_stays_within_its_limit(heads, lens, ctx):
    """What the plan compares with the limit is what a launch asks for: the query tiles that exist, not every portion at the longest one's."""
    from infer_b200 import fast_ops

    class State:
        def workspace(self, n):
            self.floats = n

        def counters(self, n):
            self.n = n
    _, parts = fast_ops.prefill_plan(SMS, heads, 128, lens, ctx, None)
    st = State()
    fast_ops.prefill_scratch(st, heads, 128, fast_ops.prefill_query_tiles(lens), max(parts, 2))
    assert st.n == heads * sum(-(-n // 128) for n in lens)
    assert st.floats == st.n * max(parts, 2) * (128 * 128 + 256)
    assert parts == 1 or st.floats <= fast_ops.PREFILL_PARTS_MAX_FLOATS


@pytest.mark.parametrize("head_dim", [64, 128])
def test_both_forms_are_built_at_the_first_use_of_either(head_dim, monkeypatch):
    from infer_b200 import fast_ops
    from infer_b200.csrc import build
    compiled, loaded = [], []
    monkeypatch.setattr(build, "compile_module", lambda module, defines=None, verbose=False: compiled.append((module, dict(defines))))
    monkeypatch.setattr(fast_ops, "_fn", lambda module, name, argtypes, defines=None: loaded.append(defines))
    fast_ops._build_prefill_forms.cache_clear()
    for _ in range(2):
        fast_ops._prefill_fn("ib_attention_prefill_tc", [], {"IB_HEAD_DIM": head_dim})
    assert sorted(len(d) for m, d in compiled if m == "attn_tc" and d["IB_HEAD_DIM"] == head_dim) == [1, 2] and len(compiled) == 2
    assert loaded == [{"IB_HEAD_DIM": head_dim}] * 2
    fast_ops._build_prefill_forms.cache_clear()


@pytest.mark.parametrize("heads,n,before,singles,parts", [
    (28, 2048, 8192, 0, 3), (28, 2048, 8192, 31, 1), (28, 2048, 8192, 63, 1),        # measured: 402 us, then 614 and 829 in three parts, 579 whole
    (28, 512, 2048, 63, 1),                                                         # 113 us in two parts, 94 whole
    (12, 1024, 8192, 0, 3), (12, 1024, 8192, 31, 3), (12, 1024, 8192, 63, 3),        # 178 us in three parts, 231 whole
    (12, 512, 4096, 63, 3),                                                         # 82 and 90
])
def test_parts_count_the_ctas_that_one_token_segments_leave_idle(heads, n, before, singles, parts):
    from infer_b200 import fast_ops
    assert fast_ops.prefill_plan(SMS, heads, 128, [1] * singles + [n], n + before, None)[1] == parts
