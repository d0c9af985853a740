"""FP32 CG solves in one cooperative launch (small batches) against the iterations launched kernel by kernel
(per-kernel timing on).  Each form is within 1e-7 (stress) and 1e-5 (ctan) of the converged FP64 solution, so the two
are within twice that of each other; a solve's sums differ in the last bits, so its iterations by a few at most."""
import numpy as np
import pytest

from cases import gpu_config
from conftest import rel_err
from micropp_gb300 import workloads as wl
from test_gpu_mixed import TOL_CTAN, TOL_STRESS

pytestmark = pytest.mark.gpu

MATS = {"elastic": (0, 1e7, 0.25, 0, 0, 0), "damage": (2, 1e7, 0.25, 0, 0, 1e5), "j2": (1, 1e7, 0.3, 1e5, 1e4, 0)}
AMP = {"elastic": 5e-3, "damage": 2.5e-2, "j2": 5e-3}


# one unit of 32 nodes and less, remainders, many instances (few blocks each, without a block for the coarsest levels), an
# elongated grid whose coarsest level does not fit in one block, several units per block, and both preconditioners
@pytest.mark.parametrize("n,ngp,law,precond", [
    (2, 1, "damage", 0), ((3, 4, 2), 19, "damage", 0), ((7, 4, 9), 3, "j2", 0), (20, 4, "damage", 0),
    (5, 1, "damage", 1), (5, 38, "elastic", 1), ((4, 4, 300), 1, "damage", 1), ((13, 6, 9), 3, "damage", 1),
    (16, 2, "j2", 1), (30, 4, "damage", 1), (45, 1, "damage", 1)])
def test_one_launch_fp32_solve_matches_the_launched_one(gpu_lib, n, ngp, law, precond):
    import micropp_gb300 as mg
    kw = dict(ngp=ngp, mats=(MATS[law], (0, 1e8, 0.25, 0, 0, 0), (0, 1e7, 0.25, 0, 0, 0)), coupling=[2] * ngp,
              lin_stress=0, micro_type=1, geo=(0.2, 0, 0, 0), precision=mg.MIXED, ctan_mode=mg.CTAN_IMPLICIT,
              precond=precond, nr_max_its=30, nr_max_tol=1e-30, nr_rel_tol=1e-8)
    eps = wl.random_targets(ngp, 11, AMP[law])
    out = []
    for timing in (False, True):
        g = mg.Micropp(gpu_config(n, **kw))
        g.set_kernel_timing(timing)
        for gp in range(ngp):
            g.set_strain(gp, eps[gp])
        g.homogenize()
        out.append([(g.get_stress(gp), g.get_ctan(gp), g.newton(gp), g.get_cost(gp), g.status(gp)) for gp in range(ngp)])
        g.close()
    for a, b in zip(*out):
        assert a[4] == b[4] == mg.STATUS_OK and a[2][2] and b[2][2]
        assert rel_err(a[0], b[0]) < 2 * TOL_STRESS
        assert rel_err(a[1], b[1]) < 2 * TOL_CTAN
        assert abs(a[3] - b[3]) <= 2 + 0.1 * b[3]
