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
