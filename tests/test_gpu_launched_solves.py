"""The solves launched kernel by kernel, on batches that the dispatch sends there: the FP64 CG beyond the nodes of one launch."""
import pytest

import test_gpu_one_launch as one_launch

pytestmark = pytest.mark.gpu


# 54^3 = 157,464 nodes in one point and in 8 (one launch takes 150,000): iterations replayed from a captured graph against
# iterations launched one by one (per-kernel timing on)
@pytest.mark.parametrize("n,ngp", [(53, 1), (26, 8)])
def test_fp64_solve_beyond_one_launch(gpu_lib, n, ngp):
    one_launch.test_one_launch_solve_is_bitwise_the_launched_one(gpu_lib, n, ngp, "damage")
