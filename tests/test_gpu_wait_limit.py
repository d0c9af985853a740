"""A one-launch solve whose blocks give up waiting: with a limit of one poll the block that arrives first does.  The kernel
returns, the call fails with an error, and the same handle then gives what a handle gives that never stalled."""
import numpy as np
import pytest

from cases import gpu_config
from micropp_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

MATS = ((2, 1e7, 0.25, 0, 0, 1e5), (0, 1e8, 0.25, 0, 0, 0), (0, 1e7, 0.25, 0, 0, 0))
KW = dict(mats=MATS, coupling=[2, 2], ngp=2, lin_stress=0, micro_type=1, geo=(0.2, 0, 0, 0))
EPS = wl.random_targets(2, 8, 2.5e-2)


def results(g):
    out = []
    for f in (0.5, 1.0):
        for gp in range(2):
            g.set_strain(gp, f * EPS[gp])
        g.homogenize()
        out += [(g.get_stress(gp), g.get_ctan(gp), g.u(gp, 1), g.newton(gp), g.get_cost(gp), g.status(gp)) for gp in range(2)]
        g.update_vars()
    return out


@pytest.mark.parametrize("form", ["plain", "jacobi", "multigrid"])
def test_stalled_homogenization_fails_and_the_handle_recovers(gpu_lib, form):
    import micropp_gb300 as mg
    kw = dict(KW, nr_max_its=6) if form == "plain" else dict(KW, **dict(wl.FAST_FORM, precond=int(form == "multigrid")))
    fresh = mg.Micropp(gpu_config(12, **kw))
    g = mg.Micropp(gpu_config(12, **kw))
    g.set_wait_limit(1)
    for gp in range(2):
        g.set_strain(gp, EPS[gp])
    for _ in range(2):
        with pytest.raises(RuntimeError, match="stalled"):
            g.homogenize()
    g.set_wait_limit(0)
    for a, b in zip(results(fresh), results(g)):
        assert all(np.array_equal(x, y) for x, y in zip(a[:3], b[:3])) and a[3:] == b[3:]


def test_stalled_path_fails_and_the_handle_recovers(gpu_lib):
    import micropp_gb300 as mg
    params = np.array([[m[1], m[2], m[5], m[4], m[3]] for m in MATS])
    strains, grad = np.vstack([0.5 * EPS[0], EPS[0]]), np.random.default_rng(1).uniform(-1, 1, (2, 6))

    def handle():
        return mg.Micropp(gpu_config(12, **dict(KW, coupling=[2], ngp=1), calc_ctan_lin=0, nr_max_its=30, nr_max_tol=1e-30,
                                     nr_rel_tol=1e-11, cg_rel_tol=1e-12, cg_max_its=20000))

    def path(h):
        sigma, _ = h.path_forward(strains, params, 1)
        return sigma, *h.path_vjp(grad)

    fresh, g = handle(), handle()
    g.set_wait_limit(1)
    with pytest.raises(RuntimeError, match="stalled"):
        g.path_forward(strains, params, 1)
    g.set_wait_limit(0)
    sigma, _ = g.path_forward(strains, params, 1)
    g.set_wait_limit(1)
    with pytest.raises(RuntimeError, match="stalled"):
        g.path_vjp(grad)
    g.set_wait_limit(0)
    want = path(fresh)
    assert np.array_equal(sigma, want[0])
    assert all(np.array_equal(a, b) for a, b in zip(g.path_vjp(grad), want[1:]))
    assert all(np.array_equal(a, b) for a, b in zip(path(g), want))
