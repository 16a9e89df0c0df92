"""Sizes that the 32-bit product's entry point takes and refuses, asked where there is no device: what is accepted then fails at its launch."""
import pytest
import torch


@pytest.mark.skipif(torch.cuda.is_available(), reason="would launch on operands that do not exist")
@pytest.mark.parametrize("M,N,K,accepted", [(1, 1, 1 << 31, True), (9, 1, (1 << 31) + 4, True), (1, 1 << 31, 4, True), (1, 40, 64, True),
                                            (1, 1, 0, False), (1, 1, 1 << 36, False), (1, 1 << 34, 4, False)])
def test_sizes(M, N, K, accepted):
    from infer_b200.ops import _fn, c_int, c_int64, c_void_p
    f = _fn("lin32", "ib_linear_f32", [c_void_p] * 5 + [c_int64] * 3 + [c_int, c_int, c_int, c_void_p])
    rc = f(None, None, None, None, None, M, N, K, 0, 148, 0, None)
    assert rc == (-2 if accepted else -1)              # IB_ERR_CUDA: there is no device; IB_ERR_ARG: refused
