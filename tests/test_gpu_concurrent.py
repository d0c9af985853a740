"""Handles at work at the same time: each one-launch solve leaves SMs to the others.  The count of handles decides how many
blocks a solve takes, never its result: every sum has an order that does not depend on them.  (Jacobi solves of many large
handles in one call are launched kernel by kernel, which rounds the FP64 sums in another order; the sizes here are below.)"""
import ctypes
import threading
import time

import numpy as np
import pytest

from cases import gpu_config
from micropp_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

MATS = {"elastic": (0, 1e7, 0.25, 0, 0, 0), "damage": (2, 1e7, 0.25, 0, 0, 1e5), "j2": (1, 1e7, 0.3, 1e5, 1e4, 0)}
PLAIN = dict(nr_max_its=6, nr_max_tol=1e-5, calc_ctan_lin=0)


def handles(specs, **form):
    """(handle, strains) per (elements, points, law)."""
    import micropp_gb300 as mg
    out = []
    for i, (n, ngp, law) in enumerate(specs):
        kw = dict(ngp=ngp, mats=(MATS[law], (0, 1e8, 0.25, 0, 0, 0), (0, 1e7, 0.25, 0, 0, 0)), lin_stress=0,
                  micro_type=1, geo=(0.2, 0, 0, 0), **form)
        kw.setdefault("coupling", [1] * ngp)
        out.append((mg.Micropp(gpu_config(n, **kw)), wl.random_targets(ngp, 40 + i, 2.5e-2 if law == "damage" else 5e-3)))
    return out


def homogenize(hs):
    """All handles at once; results and seconds."""
    import micropp_gb300 as mg
    lib = mg.load()
    for h, strains in hs:
        for gp, e in enumerate(strains):
            h.set_strain(gp, e)
    arr = (ctypes.POINTER(mg.Handle) * len(hs))(*[ctypes.pointer(h.h) for h, _ in hs])
    t = time.perf_counter()
    lib.micropp3_homogenize_many(arr, len(hs))
    t = time.perf_counter() - t
    assert not lib.micropp3_last_error()
    return [(h.get_stress(gp), h.get_ctan(gp), h.u(gp, 1), h.newton(gp), h.get_cost(gp), h.status(gp))
            for h, s in hs for gp in range(len(s))], t


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a[:3], b[:3])) and a[3:] == b[3:]


def at_once_over_in_turn(hs, repeats=3):
    """Seconds of all handles at once over those of one after the other (least of `repeats`)."""
    for h in hs:
        homogenize([h])
    return min(homogenize(hs)[1] for _ in range(repeats)) / sum(min(homogenize([h])[1] for _ in range(repeats)) for h in hs)


# fewer units than a share has SMs, shares with several units per block and per group of warps, batches, and batches that
# are launched kernel by kernel only when there are so many of them
@pytest.mark.parametrize("specs", [
    [(6, 1, "j2"), ((7, 4, 9), 3, "damage"), (2, 5, "damage")], [(20, 1, "j2")] * 5, [(12, 8, "damage")] * 10,
    [(30, 1, "damage"), (25, 2, "j2"), (30, 2, "damage"), (26, 1, "damage")]])
def test_plain_handles_at_once_are_bitwise_the_lone_ones(gpu_lib, specs):
    hs = handles(specs, **PLAIN)
    lone = [r for h in hs for r in homogenize([h])[0]]
    for _ in range(2):
        assert all(same(a, b) for a, b in zip(lone, homogenize(hs)[0]))
    for h, _ in hs:
        h.close()


def test_plain_handles_overlap(gpu_lib):
    """16 J2 points of 20^3, a handle each: a solve that takes every SM makes the others wait, and all of them at once then
    take as long as one after the other."""
    hs = handles([(20, 1, "j2")] * 16, **PLAIN)
    assert at_once_over_in_turn(hs) < 0.75
    for h, _ in hs:
        h.close()


# FP32 solves with shares of several parts of the sums per block: with and without a block for the coarsest levels, batches
# whose instances have a block each, one and six right-hand sides, and both preconditioners
@pytest.mark.parametrize("precond", [0, 1], ids=["jacobi", "multigrid"])
@pytest.mark.parametrize("specs", [
    [(5, 1, "damage"), ((7, 5, 9), 3, "j2"), (8, 19, "elastic")], [(25, 1, "damage")] * 9, [(16, 8, "damage")] * 5,
    [((13, 17, 23), 2, "j2"), (20, 1, "damage"), (40, 1, "damage"), (12, 16, "damage")]])
def test_fast_handles_at_once_are_bitwise_the_lone_ones(gpu_lib, specs, precond):
    import micropp_gb300 as mg
    form = dict(wl.FAST_FORM, precond=precond, calc_ctan_lin=0)
    hs = [handles([s], **form, coupling=[mg.FE_FULL] * s[1])[0] for s in specs]
    hs = [(h, s * (1 + 0.1 * i)) for i, (h, s) in enumerate(hs)]
    lone = [r for h in hs for r in homogenize([h])[0]]
    for _ in range(2):
        assert all(same(a, b) for a, b in zip(lone, homogenize(hs)[0]))
    for h, _ in hs:
        h.close()


def test_fast_handles_overlap(gpu_lib):
    """13 damage points of 25^3 with the Jacobi preconditioner, a handle each."""
    import micropp_gb300 as mg
    hs = handles([(25, 1, "damage")] * 13, **dict(wl.FAST_FORM, precond=0, calc_ctan_lin=0), coupling=[mg.FE_FULL])
    assert at_once_over_in_turn(hs) < 0.7
    for h, _ in hs:
        h.close()


def paths(hs):
    """A load path and its reverse pass on every handle, each in a thread of its own; results."""
    out = [None] * len(hs)

    def run(i):
        h, strains = hs[i]
        sigma, _ = h.path_forward(np.vstack([0.5 * strains, strains]), PARAMS, 1)
        gp, gs, _ = h.path_vjp(np.random.default_rng(i).uniform(-1, 1, (2, 6)))
        out[i] = (sigma, gp, gs, [h.path_newton(k) for k in range(2)])

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(hs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return out


PARAMS = np.array([[m[1], m[2], m[5], m[4], m[3]] for m in (MATS["damage"], (0, 1e8, 0.25, 0, 0, 0), MATS["elastic"])])


# parts of less than a unit and of one, two and three units at a time, of which a block has one to three
@pytest.mark.parametrize("sizes", [[3, (7, 4, 9), 16, 12], [20, 17, 21], [23, 26]])
def test_paths_at_once_are_bitwise_the_lone_ones(gpu_lib, sizes):
    import micropp_gb300 as mg
    hs = handles([(n, 1, "damage") for n in sizes], coupling=[mg.FE_FULL], calc_ctan_lin=0, nr_max_its=30, nr_max_tol=1e-30,
                 nr_rel_tol=1e-11, cg_rel_tol=1e-12, cg_max_its=20000)
    lone = []
    for i in range(len(hs)):
        h, strains = hs[i]
        sigma, _ = h.path_forward(np.vstack([0.5 * strains, strains]), PARAMS, 1)
        gp, gs, _ = h.path_vjp(np.random.default_rng(i).uniform(-1, 1, (2, 6)))
        lone.append((sigma, gp, gs, [h.path_newton(k) for k in range(2)]))
    for _ in range(2):
        for a, b in zip(lone, paths(hs)):
            assert all(np.array_equal(x, y) for x, y in zip(a[:3], b[:3])) and a[3] == b[3]
    for h, _ in hs:
        h.close()
