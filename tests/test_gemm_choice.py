"""Which kernel a tensor-core product of more than 128 rows takes (host arithmetic of ib_gemm_tc_plan and ib_gemm_tc_pairs): the plan for a
single SM a tile, or pairs of SMs (code 1024 + 2 x width) where their estimate is less by more than 2 %."""
import pytest

SMS = 148


def _choice(M, N, K, sms=SMS):
    from infer_b200 import fast_ops
    return fast_ops.gemm_plan(M, N, K, sms), fast_ops.gemm_choice(M, N, K, sms)


@pytest.mark.parametrize("M,N,K,width", [
    (2048, 17920, 1536, 256), (2048, 1536, 8960, 192), (2048, 4608, 3584, 256), (2048, 3584, 18944, 224),    # a 2,048-token prompt, 1.5B and 7B
    (512, 17920, 1536, 256), (512, 4608, 3584, 128), (512, 3584, 3584, 128),                                # portions of 512 tokens
    (640, 2048, 1536, 128), (1024, 1536, 1536, 128), (257, 4608, 3584, 128),                               # where they begin for short products
])
def test_pairs(M, N, K, width):
    plan, choice = _choice(M, N, K)
    assert choice == (0, 1024 + 2 * width, 1, 0, 0) and plan[1] <= 768


@pytest.mark.parametrize("M,N,K", [
    (1, 2048, 1536), (17, 1536, 8960), (128, 37888, 3584),              # up to 128 rows: the weights on the 128-row side
    (129, 1536, 1536), (256, 2048, 1536),                               # K slices as a cluster
    (512, 3584, 18944), (1024, 1536, 8960),                             # K slices of wide tiles
    (257, 17920, 1536), (2048, 2048, 1536), (2048, 1536, 1536),         # one round either way
])
def test_a_single_sm_a_tile(M, N, K):
    plan, choice = _choice(M, N, K)
    assert plan == choice


def test_refused_sizes_and_slices_through_the_workspace_stay():
    assert _choice(300, 1000, 1537) == (None, None)
    for M, N, K in ((129, 16, 512), (200, 500, 1536), (300, 130, 4096), (1000, 100, 1024)):
        plan, choice = _choice(M, N, K)
        assert plan[3] > 0 and choice == plan                           # up to 16 slices that meet in the workspace
    for sms in (1, 0):
        plan, choice = _choice(4096, 4096, 4096, sms)
        assert plan == choice


def test_a_pair_is_chosen_only_below_its_rivals_estimate():
    """Every size of a sweep: a chosen width is one the kernel has, the tile is no wider than what it saves a round for."""
    from infer_b200 import fast_ops
    for M in (129, 255, 256, 257, 511, 513, 700, 1025, 2047, 3000, 8191):
        for N in (16, 130, 1536, 3000, 17920, 37888):
            for K in (64, 72, 1536, 8960):
                choice = fast_ops.gemm_choice(M, N, K, SMS)
                if choice[1] >= 1280:
                    assert choice[1] in (1280, 1344, 1408, 1472, 1536) and choice[2:] == (1, 0, 0)
                    assert fast_ops.gemm_plan(M, N, K, SMS)[3] == 0
