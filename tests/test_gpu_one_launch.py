"""Linear solves that run in one cooperative launch (small batches) against the same iterations launched kernel by
kernel (per-kernel timing on): the order of every sum is the same, so the results are bitwise equal."""
import numpy as np
import pytest

from cases import gpu_config
from micropp_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

MATS = {"damage": (2, 1e7, 0.25, 0, 0, 1e5), "j2": (1, 1e7, 0.3, 1e5, 1e4, 0)}


# grids below one unit of 32 nodes, with remainders, with more instances than SMs, with several units per block,
# and just above the size that one launch takes (46^3 nodes)
@pytest.mark.parametrize("n,ngp,law", [(2, 1, "damage"), (3, 160, "damage"), ((7, 4, 9), 3, "j2"), (12, 8, "damage"),
                                       (20, 1, "j2"), (26, 5, "damage"), (46, 1, "damage")])
def test_one_launch_solve_is_bitwise_the_launched_one(gpu_lib, n, ngp, law):
    import micropp_gb300 as mg
    kw = dict(ngp=ngp, mats=(MATS[law], (0, 1e8, 0.25, 0, 0, 0), (0, 1e7, 0.25, 0, 0, 0)), coupling=[1] * ngp,
              lin_stress=0, nr_max_its=4, nr_max_tol=1e-5, micro_type=1, geo=(0.2, 0, 0, 0))
    eps = wl.random_targets(ngp, 11, 2.5e-2 if law == "damage" else 5e-3)
    out = []
    for timing in (False, True):
        g = mg.Micropp(gpu_config(n, **kw))
        g.set_kernel_timing(timing)
        for gp in range(ngp):
            g.set_strain(gp, eps[gp])
        g.homogenize()
        out.append([(g.get_stress(gp), g.u(gp, 1), g.newton(gp), g.get_cost(gp), g.status(gp)) for gp in range(ngp)])
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2:] == b[2:]
