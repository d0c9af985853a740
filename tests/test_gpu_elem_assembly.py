"""The FP64 assembly by element matrices, which works through a ring of element layers: how many layers fit, and so where
its chunks end, depends on the batch, but every entry receives its contributions in a fixed order.  A point of a batch is
therefore bitwise the same point in a handle of its own (the solves' sums do not depend on the batch either).  Sizes:
the smallest grid, blocks of 8 elements that cross layers and end early, and layers so large that the single point takes
two chunks and the batch ten."""
import numpy as np
import pytest

from cases import gpu_config
from micropp_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

MATS = {"damage": (2, 1e7, 0.25, 0, 0, 1e5), "j2": (1, 1e7, 0.3, 1e5, 1e4, 0)}


@pytest.mark.parametrize("n,ngp,law", [(2, 3, "damage"), ((3, 4, 2), 5, "j2"), ((9, 7, 5), 2, "damage"),
                                       ((5, 3, 11), 2, "j2"), ((30, 31, 20), 4, "damage")])
def test_a_point_of_a_batch_is_the_single_point(gpu_lib, n, ngp, law):
    import micropp_gb300 as mg
    kw = dict(mats=(MATS[law], (0, 1e8, 0.25, 0, 0, 0), (0, 1e7, 0.25, 0, 0, 0)), lin_stress=0, calc_ctan_lin=0,
              nr_max_its=2, nr_max_tol=1e-5, micro_type=1, geo=(0.2, 0, 0, 0))
    eps = wl.random_targets(ngp, 3, 2.5e-2 if law == "damage" else 5e-3)

    def results(points):
        g = mg.Micropp(gpu_config(n, ngp=len(points), coupling=[1] * len(points), **kw))
        for gp, e in enumerate(points):
            g.set_strain(gp, e)
        g.homogenize()
        out = [(g.get_stress(gp), g.u(gp, 1), g.newton(gp), g.get_cost(gp)) for gp in range(len(points))]
        g.close()
        return out

    batch = results(eps)
    for gp in range(ngp):
        one = results(eps[gp:gp + 1])[0]
        assert np.array_equal(one[0], batch[gp][0]) and np.array_equal(one[1], batch[gp][1])
        assert one[2:] == batch[gp][2:]
