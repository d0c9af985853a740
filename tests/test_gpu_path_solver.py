"""The load paths' BiCGSTAB in one cooperative launch: on an elastic path the stress is C eps and the strain gradients
are C^T g, with C the handle's linear ctan (six solves of the FP64 CG, another solver).  Both solvers stop at a relative
residual of 1e-12 and the condition numbers are below 1e4, so the results agree to 1e-8; the bar leaves a factor 10."""
import numpy as np
import pytest

from cases import gpu_config
from conftest import rel_err

pytestmark = pytest.mark.gpu

MATS = ((0, 1e7, 0.25, 0, 0, 0), (0, 1e8, 0.25, 0, 0, 0), (0, 1e7, 0.25, 0, 0, 0))


# less than one unit of 32 nodes, remainders, one unit per block, several units per block in turn, and a grid above the
# size that one launch takes
@pytest.mark.parametrize("n", [2, (3, 4, 2), (7, 4, 9), 12, 25, 47, 94])
def test_elastic_path_is_the_linear_ctan(gpu_lib, n):
    import micropp_gb300 as mg
    g = mg.Micropp(gpu_config(n, mats=MATS, coupling=[2], lin_stress=0, micro_type=1, geo=(0.2, 0, 0, 0), nr_max_its=4,
                              nr_max_tol=1e-30, nr_rel_tol=1e-11, cg_rel_tol=1e-12, cg_max_its=20000))
    ctan = g.ctan_lin()
    rng = np.random.default_rng(5)
    strains, grad = rng.uniform(-5e-3, 5e-3, (3, 6)), rng.uniform(-1, 1, (3, 6))
    params = np.array([[m[1], m[2], m[5], m[4], m[3]] for m in MATS])
    # the status is not looked at: on a homogeneous RVE (the smallest grids) the predictor is the solution already, and a
    # residual of rounding errors does not fall
    sigma, _ = g.path_forward(strains, params, 2)
    _, gs, _ = g.path_vjp(grad)
    assert rel_err(sigma, strains @ ctan.T) < 1e-7
    assert rel_err(gs, grad @ ctan) < 1e-7
