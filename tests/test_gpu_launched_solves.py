"""The solves launched kernel by kernel, on batches that the dispatch sends there: the FP64 CG beyond the nodes of one launch,
Newton iterations as CUDA graphs, and the fast form's error with the headline's solver."""
import numpy as np
import pytest

import test_gpu_fast_error as fast_error
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


@pytest.mark.parametrize("precond", [1, 0], ids=["multigrid", "jacobi"])
def test_fast_form_error_of_a_launched_batch_at_60cubed(gpu_lib, precond):
    """Five RVEs of the headline workload in one handle (1.13 million nodes, one launch takes 950,000), two of them against
    the FP64 solution: the bars of the fast form."""
    import micropp_gb300 as mg
    from micropp_gb300 import accuracy
    n = fast_error.N
    et, xts, targets = wl.damage_layers_rves(n, 32, 2024)
    mats = wl.damage_layers_materials(mg, xts[0])
    fast = accuracy.fast_solution(n, mats, et, 0.5 * targets[:5], targets[:5], dict(wl.FAST_FORM, precond=precond))
    res = accuracy.compare(fast, fp64_solutions(mats, et, targets))
    assert all(status == mg.STATUS_OK for _, _, status in fast)
    assert res["stress"] <= fast_error.TOL_STRESS and res["ctan"] <= fast_error.TOL_CTAN, res


FP64 = []


def fp64_solutions(mats, et, targets):
    from micropp_gb300 import accuracy
    if not FP64:
        FP64.extend(accuracy.fp64_solution(fast_error.N, mats, et, 0.5 * targets[i], targets[i]) for i in range(2))
    return FP64
