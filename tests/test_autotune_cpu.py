"""The autotuner's candidates hold the work-item sizes that the defaults take, so tuning a plan cannot
leave it slower than its default for want of them."""
from mr_recon_b200.autotune import default_candidates


def test_candidates_reach_the_defaults():
    # the bounds of the default gridding items: 96 to 256 entries in 2D, 512 to 4096 in 3D
    assert {96, 128, 192, 256} <= set(default_candidates(2)["grid_chunk"])
    assert {512, 4096} <= set(default_candidates(3)["grid_chunk"])
