"""The solves launched kernel by kernel, on batches that the dispatch sends there: the FP64 CG beyond the nodes of one launch and
Newton iterations as CUDA graphs."""
import numpy as np
import pytest

import test_gpu_one_launch as one_launch
from cases import gpu_config
from micropp_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


# 54^3 = 157,464 nodes in one point and in 8 (one launch takes 150,000): iterations replayed from a captured graph against
# iterations launched one by one (per-kernel timing on)
@pytest.mark.parametrize("n,ngp", [(53, 1), (26, 8)])
def test_fp64_solve_beyond_one_launch(gpu_lib, n, ngp):
    one_launch.test_one_launch_solve_is_bitwise_the_launched_one(gpu_lib, n, ngp, "damage")


def test_newton_graphs_of_a_launched_batch_match_unfused(gpu_lib):
    """48 points leave 3 blocks each, too few for one launch.  A Newton iteration as one graph runs the kernels of the
    unfused one in their order, and kernels that set its loop's condition: the handle with graphs counts more launches, which
    shows that it took them (the other way round where only the CG chunks are graphs)."""
    import micropp_gb300 as mg
    n, ngp = 6, 48
    kw = dict(ngp=ngp, elem_type=wl.layers_z(n), mats=((2, 1e7, 0.25, 0, 0, 1e5), (0, 1e8, 0.25, 0, 0, 0),
                                                      (0, 1e7, 0.25, 0, 0, 0)),
              coupling=[1] * ngp, lin_stress=0, calc_ctan_lin=0, **wl.FAST_FORM)
    eps = wl.random_targets(ngp, 4, 2.5e-2)
    handles = [mg.Micropp(gpu_config(n, **kw)) for _ in range(2)]
    handles[1].set_cuda_graphs(False)
    counts = []
    for repeat in range(2):  # the first pass tunes the SpMV's block, which a graph needs
        for g in handles:
            before = g.kernel_launches()
            for gp in range(ngp):
                g.set_strain(gp, eps[gp])
            g.homogenize()
            counts.append(g.kernel_launches() - before)
        a, b = handles
        for gp in range(ngp):
            assert np.array_equal(a.get_stress(gp), b.get_stress(gp)) and np.array_equal(a.u(gp, 1), b.u(gp, 1))
            assert a.newton(gp) == b.newton(gp) and a.status(gp) == b.status(gp) == mg.STATUS_OK
    assert counts[2] > counts[3], counts
