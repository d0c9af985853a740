"""The framework's work as timed cases: homogenizations of RVE batches through the Python mirror of the C ABI, the
load-path gradients and the standalone stencil-ELL solve.

A case is a dict of plain values:

  kind    "rve"   one handle: set_strain on every point, homogenize, get_stress and get_ctan
          "many"  handles of several sizes and laws, homogenized together (micropp3_homogenize_many)
          "path"  micropp3_path_forward and micropp3_path_vjp along a cyclic strain path
          "ell"   micropp3_ell_solve_cgpd on device arrays
  form    "plain" the reference algorithm in FP64 (the drop-in); "fast": FP32 solves in FP64-accurate refinement
          with the multigrid; "jacobi": the same with the default (Jacobi) preconditioner
  coupling "full": stress and ctan; "one_way": stress only (ctan stays the linear one, which a program reads once)
  law     of the matrix phase: "elastic", "damage" or "j2"; the second phase is elastic, ten times stiffer
  micro   "sphere" (one, centred), "layers" (4 normal to z) or "spheres" (8, seeded)
  nx, ny, nz elements per axis; ngp points of the handle

Every nonlinear RVE has an accepted history before the timed call, as in a macro time loop; a pass repeats the
macro iteration at the target strain (nothing is accepted, so each pass does the same work).
"""
import ctypes
import math

import numpy as np
import torch

import micropp_gb300 as mg
from micropp_gb300 import workloads as wl

PLAIN = dict(precision=mg.FP64, ctan_mode=mg.CTAN_PERTURB, nr_max_its=12, nr_max_tol=1e-5)
FORMS = {"plain": PLAIN, "fast": wl.FAST_FORM, "jacobi": dict(wl.FAST_FORM, precond=mg.PRECOND_JACOBI)}
# (type, E, nu, Ka, Sy, Xt) of the matrix phase, the strain amplitude and the accepted fractions of the target
LAWS = {
    "elastic": ((0, 1e7, 0.25, 0.0, 0.0, 0.0), 5e-3, ()),
    "damage": ((2, 1e7, 0.25, 0.0, 0.0, 1e5), 2.5e-2, (0.5,)),
    "j2": ((1, 1e7, 0.3, 1e5, 1e4, 0.0), 5e-3, (0.6, 0.8)),
}
STIFF = (0, 1e8, 0.25, 0.0, 0.0, 0.0)


def _rve(name, form, law, micro, n, ngp, coupling="full"):
    nx, ny, nz = (n, n, n) if isinstance(n, int) else n
    c = {"kind": "rve", "form": form, "law": law, "micro": micro, "nx": nx, "ny": ny, "nz": nz, "ngp": ngp,
         "coupling": coupling}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest drop-in call: one linear macro point on a 10^3 RVE, as a macro code makes thousands of
        _rve("plain elastic 10^3", "plain", "elastic", "sphere", 10, 1),
        # a macro element's 8 Gauss points on small damage RVEs, the drop-in with its six perturbed solves
        _rve("plain damage 12^3 x8", "plain", "damage", "layers", 12, 8),
        # the drop-in on a J2 RVE of ordinary size, coupled one way (the reference's default)
        _rve("plain j2 20^3", "plain", "j2", "sphere", 20, 1, "one_way"),
        # the drop-in at the resolution the metric is quoted on, one micro point at a time
        _rve("plain damage 60^3", "plain", "damage", "layers", 60, 1),
        # the fast form on one odd-sized, non-cubic RVE: the latency a macro code sees for a single point
        _rve("fast damage 23x17x31", "fast", "damage", "sphere", (23, 17, 31), 1),
        # a macro element's 8 points on mid-sized RVEs, fast form
        _rve("fast damage 30^3 x8", "fast", "damage", "layers", 30, 8),
        # the same batch with the preconditioner a user gets by default
        _rve("jacobi damage 20^3 x8", "jacobi", "damage", "layers", 20, 8),
        # the headline: 32 damage RVEs of 60^3 in one handle, stress and ctan
        _rve("fast damage 60^3 x32", "fast", "damage", "layers", 60, 32),
        # J2 matrix with 8 spheres, fast form, a fine RVE
        _rve("fast j2 50^3", "fast", "j2", "spheres", 50, 1),
        # uneven RVEs: every (size, micro, law) group a handle of its own, all handles at once
        {"name": "many mixed 20-40", "kind": "many", "form": "fast", "sizes": "20,30,40", "ngp": 2},
        # gradients of a cyclic J2 path: forward pass and reverse pass with checkpoints
        {"name": "path j2 12^3 x4", "kind": "path", "law": "j2", "n": 12, "steps": 4, "every": 2},
        # the linear solver alone, matrix and right-hand side already on the device
        {"name": "ell solve 50x50x50", "kind": "ell", "nx": 50, "ny": 50, "nz": 50},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "fast", "fast", "jacobi", "j2", "many", "path", "ell"])
    law = rng.choice(["elastic", "damage", "j2"])
    micro = rng.choice(["sphere", "layers", "spheres"])
    if kind == "many":
        sizes = sorted(_log_int(rng, 12, 44) for _ in range(3))
        return {"kind": "many", "form": "fast", "sizes": ",".join(map(str, sizes)), "ngp": rng.randint(1, 3)}
    if kind == "path":
        return {"kind": "path", "law": rng.choice(["damage", "j2"]), "n": _log_int(rng, 6, 14),
                "steps": rng.randint(2, 4), "every": rng.randint(1, 3)}
    if kind == "ell":
        return {"kind": "ell", "nx": _log_int(rng, 8, 64), "ny": _log_int(rng, 8, 64), "nz": _log_int(rng, 8, 64)}
    if kind == "plain":
        n, most = _log_int(rng, 6, 40), 64000
    elif kind == "j2":
        n, most, law = _log_int(rng, 10, 56), 200000, "j2"
    else:
        n, most = _log_int(rng, 10, 60), 2000000
        law = law if law != "j2" else "damage"
    coupling = rng.choice(["full", "full", "one_way"])
    if kind == "plain" and law == "j2":
        n, most, coupling = _log_int(rng, 6, 18), 8000, "one_way"
    size = tuple(max(6, n + rng.randint(-3, 3)) for _ in range(3))
    ngp = min(32, max(1, most // (size[0] * size[1] * size[2])))
    return _rve(None, "fast" if kind == "j2" else kind, law, micro, size, _log_int(rng, 1, ngp), coupling)


# ---------------------------------------------------------------------------------------------------------
# microstructures, materials, strains


def _phases(micro, size, seed):
    """Phase of every element, x fastest."""
    if micro == "sphere":
        centres, r = np.array([[0.5, 0.5, 0.5]]), 0.2
    elif micro == "spheres":
        centres, r = wl.sphere_centres(8, 0.12, seed % 1000), 0.12
    z, y, x = np.meshgrid(*[(np.arange(n) + 0.5) / n for n in size[::-1]], indexing="ij")
    if micro == "layers":
        inside = np.min([np.abs(z - c) for c in (0.125, 0.375, 0.625, 0.875)], axis=0) < 0.05
    else:
        inside = np.min([(x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2 for c in centres], axis=0) < r * r
    return inside.astype(np.int32).reshape(-1)


def _materials(law):
    return [mg.material(*LAWS[law][0]), mg.material(*STIFF), mg.material(0, 1e7, 0.25)]


def _size(case):
    return case["nx"], case["ny"], case["nz"]


def _target(law, ngp, seed):
    """Strain targets, each of the law's amplitude in some component so that a nonlinear law is always loaded."""
    t = np.random.default_rng([seed, 7]).uniform(-1.0, 1.0, (ngp, 6))
    return LAWS[law][1] * t / np.max(np.abs(t), axis=1, keepdims=True)


def _groups(case):
    """The handles of a "many" case, as "rve" cases."""
    out = []
    for i, n in enumerate(int(s) for s in case["sizes"].split(",")):
        for j, law in enumerate(("elastic", "damage", "j2")):
            out.append(_rve(None, case["form"], law, ("sphere", "layers")[(i + j) % 2], n, case["ngp"]))
    return out


def _handle(case, seed):
    law, size, ngp = case["law"], _size(case), case["ngp"]
    kw = dict(FORMS[case["form"]], nr_max_its=30 if law == "j2" else FORMS[case["form"]]["nr_max_its"])
    coupling = mg.FE_FULL if case["coupling"] == "full" else mg.FE_ONE_WAY
    h = mg.Micropp(mg.config(size, ngp=ngp, mats=_materials(law), coupling=[coupling] * ngp, lin_stress=0,
                             elem_type=_phases(case["micro"], size, seed), **kw))
    target = _target(law, ngp, seed)
    for f in LAWS[law][2]:
        for gp in range(ngp):
            h.set_strain(gp, f * target[gp])
        h.homogenize()
        h.update_vars()
    return h, target


def _path_case(case, seed):
    law, steps = case["law"], case["steps"]
    k = np.arange(1, steps + 1)
    phase = np.sin(2 * np.pi * k / steps) if law == "j2" else k / steps
    phase = np.where(np.abs(phase) < 0.1, 0.5, phase)
    strains = np.outer((8e-3 if law == "j2" else 2.5e-2) * phase, _target(law, 1, seed)[0] / LAWS[law][1])
    mats = [LAWS[law][0], STIFF, (0, 1e7, 0.25, 0.0, 0.0, 0.0)]
    params = np.array([[m[1], m[2], m[5], m[4], m[3]] for m in mats])
    grad = np.random.default_rng([seed, 9]).uniform(-1.0, 1.0, (steps, 6))
    return strains, params, grad


# ---------------------------------------------------------------------------------------------------------
# the stencil matrix of an elastic two-phase RVE, as a caller of the standalone solve holds it

CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def _bmat(h):
    """Strain matrices (8 Gauss points, 6, 24) of a hex8 element with edges h, and the Gauss weight."""
    g = 0.577350269189626
    B = np.zeros((8, 6, 24))
    for q, cq in enumerate(CORNERS):
        xi = [g if c else -g for c in cq]
        for a, ca in enumerate(CORNERS):
            s = [1.0 if c else -1.0 for c in ca]
            d = [s[i] * (1 + s[(i + 1) % 3] * xi[(i + 1) % 3]) * (1 + s[(i + 2) % 3] * xi[(i + 2) % 3]) / 4 / h[i]
                 for i in range(3)]
            B[q, 0, 3 * a], B[q, 1, 3 * a + 1], B[q, 2, 3 * a + 2] = d
            B[q, 3, 3 * a], B[q, 3, 3 * a + 1] = d[1], d[0]
            B[q, 4, 3 * a], B[q, 4, 3 * a + 2] = d[2], d[0]
            B[q, 5, 3 * a + 1], B[q, 5, 3 * a + 2] = d[2], d[1]
    return B, h[0] * h[1] * h[2] / 8


def _elastic(E, nu):
    lam, mu = nu * E / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    C = np.zeros((6, 6))
    C[:3, :3] = lam
    C[range(6), range(6)] += [2 * mu] * 3 + [mu] * 3
    return C


def _interior(nodes, device):
    m = torch.zeros(nodes[::-1], dtype=torch.bool, device=device)
    m[1:-1, 1:-1, 1:-1] = True
    return m.reshape(-1)


def _ell_apply(vals, x, nodes):
    """A x on interior nodes (0 on the boundary) of the stencil matrix; x: (nodes, 3)."""
    nx, ny, nz = nodes
    nn = nx * ny * nz
    pad = nx * ny + nx + 1
    xp = torch.nn.functional.pad(x, (0, 0, pad, pad))
    y = torch.zeros_like(x)
    v = vals.view(27, 3, 3, -1)[..., :nn]
    for s in range(27):
        off = (s // 9 - 1) * nx * ny + ((s // 3) % 3 - 1) * nx + s % 3 - 1
        y += torch.einsum("ijn,nj->ni", v[s], xp[pad + off:pad + off + nn])
    return y * _interior(nodes, x.device)[:, None]


def _ell_system(case, seed, device):
    nodes = _size(case)
    size = [n - 1 for n in nodes]
    nn, npad = math.prod(nodes), (math.prod(nodes) + 31) // 32 * 32
    B, wg = _bmat([1.0 / n for n in size])
    ke = torch.tensor(np.einsum("gki,kl,glj->ij", B, _elastic(1e7, 0.25), B) * wg, device=device)
    rng = np.random.default_rng([seed, 3])
    stiff = torch.tensor(_phases("spheres", size, seed), device=device).view(size[::-1])
    scale = 1.0 + 9.0 * stiff + torch.tensor(rng.uniform(0.0, 0.2, size[::-1]), device=device)
    full = torch.zeros((27, 3, 3) + tuple(nodes[::-1]), dtype=torch.float64, device=device)
    for a, ca in enumerate(CORNERS):
        for b, cb in enumerate(CORNERS):
            s = 9 * (cb[2] - ca[2] + 1) + 3 * (cb[1] - ca[1] + 1) + cb[0] - ca[0] + 1
            part = full[s, :, :, ca[2]:ca[2] + size[2], ca[1]:ca[1] + size[1], ca[0]:ca[0] + size[0]]
            part += ke[3 * a:3 * a + 3, 3 * b:3 * b + 3, None, None, None] * scale
    vals = torch.zeros((243, npad), dtype=torch.float64, device=device)
    vals[:, :nn] = full.view(243, nn) * _interior(nodes, device)
    # the right-hand side of a Dirichlet problem: the affine field of a random strain on the faces
    z, y, x = torch.meshgrid(*[torch.linspace(0, 1, n, dtype=torch.float64, device=device) for n in nodes[::-1]],
                             indexing="ij")
    e = torch.tensor(rng.uniform(-5e-3, 5e-3, (3, 3)), device=device)
    w = torch.stack([x, y, z], -1).view(nn, 3) @ (e + e.T)
    w = w * ~_interior(nodes, device)[:, None]
    return vals, -_ell_apply(vals, w, nodes)


# ---------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    if case["kind"] == "rve":
        h, target = _handle(case, seed)
        return {"case": case, "handles": [h], "targets": [target]}
    if case["kind"] == "many":
        pairs = [_handle(c, seed + i) for i, c in enumerate(_groups(case))]
        return {"case": case, "handles": [h for h, _ in pairs], "targets": [t for _, t in pairs]}
    if case["kind"] == "path":
        size = (case["n"],) * 3
        h = mg.Micropp(mg.config(size, mats=_materials(case["law"]), coupling=[mg.FE_FULL], lin_stress=0,
                                 calc_ctan_lin=0, elem_type=_phases("sphere", size, seed), nr_max_its=30,
                                 nr_max_tol=1e-30, nr_rel_tol=1e-11, cg_rel_tol=1e-12, cg_max_its=20000))
        return {"case": case, "handles": [h], "path": _path_case(case, seed)}
    vals, b = _ell_system(case, seed, "cuda")
    return {"case": case, "vals": vals, "b": b.reshape(-1).contiguous(), "x": torch.empty(b.numel(), dtype=b.dtype,
                                                                                     device="cuda")}


def _results(h, coupling="full"):
    out = {"stress": np.stack([h.get_stress(gp) for gp in range(h.ngp)])}
    if coupling == "full":
        out["ctan"] = np.stack([h.get_ctan(gp) for gp in range(h.ngp)])
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "ell":
        its = ctypes.c_int()
        nodes = (ctypes.c_int * 3)(*_size(case))
        rc = mg.load().micropp3_ell_solve_cgpd(nodes, state["vals"].data_ptr(), state["b"].data_ptr(),
                                               state["x"].data_ptr(), 1e-8, 1e-50, 5000, ctypes.byref(its),
                                               torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError(f"micropp3_ell_solve_cgpd returned {rc}")
        return {"x": state["x"], "its": its.value}
    hs = state["handles"]
    if case["kind"] == "path":
        strains, params, grad = state["path"]
        sigma, _ = hs[0].path_forward(strains, params, case["every"])
        gp, gs, _ = hs[0].path_vjp(grad)
        # each parameter's gradient per relative change, so that one scale fits all of them
        return {"sigma": sigma, "grad_params": gp * params, "grad_strains": gs}
    for h, target in zip(hs, state["targets"]):
        for gp in range(h.ngp):
            h.set_strain(gp, target[gp])
    if case["kind"] == "many":
        arr = (ctypes.POINTER(mg.Handle) * len(hs))(*[ctypes.pointer(h.h) for h in hs])
        mg.load().micropp3_homogenize_many(arr, len(hs))
        return [_results(h) for h in hs]
    hs[0].homogenize()
    return _results(hs[0], case["coupling"])


def work(case):
    """Bytes: the state of every point (displacements and, where the law has them, the internal variables) read
    and written once, or the stencil matrix read once.  Flops: one evaluation of the element residuals, or one
    product with the matrix; the iterations of the solvers are the framework's own choice."""
    if case["kind"] == "ell":
        nn = math.prod(_size(case))
        return {"bytes": 8.0 * nn * (243 + 6), "flops": 2.0 * 243 * nn}
    if case["kind"] == "many":
        parts = [work(c) for c in _groups(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    size = (case["n"],) * 3 if case["kind"] == "path" else _size(case)
    runs = 2 * case["steps"] if case["kind"] == "path" else case["ngp"]
    elements, nodes = math.prod(size), math.prod(n + 1 for n in size)
    values = {"elastic": 0, "damage": 2, "j2": 7}[case["law"]]
    return {"bytes": runs * 8.0 * 2 * (3 * nodes + 8 * values * elements), "flops": runs * 900.0 * elements}


# ---------------------------------------------------------------------------------------------------------
# the same results in 64 bits: Newton to rounding on the dense or matrix-free tangent, plain torch


class _Fe:
    """Hex8 elements on the unit cube with affine displacements on the faces; nothing of the framework."""

    def __init__(self, size, mats, phases):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        nx, ny, nz = (n + 1 for n in size)
        B, wg = _bmat([1.0 / n for n in size])
        self.B, self.wg = self._t(B), wg
        ez, ey, ex = np.meshgrid(*[np.arange(n) for n in size[::-1]], indexing="ij")
        node = np.stack([(((ez + c[2]) * ny + ey + c[1]) * nx + ex + c[0]).reshape(-1) for c in CORNERS], 1)
        self.dofs = torch.tensor((node[:, :, None] * 3 + np.arange(3)).reshape(len(node), 24), device=self.dev)
        self.ndof = 3 * nx * ny * nz
        z, y, x = np.meshgrid(*[np.linspace(0, 1, n) for n in (nz, ny, nx)], indexing="ij")
        self.xyz = self._t(np.stack([x, y, z], -1).reshape(-1, 3))
        self.free = _interior((nx, ny, nz), self.dev).repeat_interleave(3).double()
        self.phases = torch.tensor(phases, device=self.dev).long()
        self.types = torch.tensor([m[0] for m in mats], device=self.dev)[self.phases]
        self.mats = self._t(np.array(mats)[:, 1:])  # E, nu, Ka, Sy, Xt per phase

    def _t(self, a):
        return torch.tensor(a, dtype=torch.float64, device=self.dev)

    def affine(self, strain):
        """The affine field of a strain (6,) on all nodes, flat."""
        e = strain
        m = torch.stack([torch.stack([e[0], e[3] / 2, e[4] / 2]), torch.stack([e[3] / 2, e[1], e[5] / 2]),
                         torch.stack([e[4] / 2, e[5] / 2, e[2]])])
        return (self.xyz @ m).reshape(-1)

    def strains(self, u):
        return torch.einsum("gki,ei->egk", self.B, u[self.dofs])

    def law(self, eps, h, mats):
        """Stress (e, 8, 6) and updated history (e, 8, 7) of the three laws."""
        E, nu, Ka, Sy, Xt = (mats[:, i][self.phases][:, None] for i in range(5))
        lam, mu = nu * E / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
        tr = eps[..., :3].sum(-1)
        two = self._t([2.0] * 3 + [1.0] * 3)
        one = self._t([1.0] * 3 + [0.0] * 3)
        s = lam[..., None] * tr[..., None] * one + mu[..., None] * two * eps
        out, new = s, h
        dam = (self.types == 2)[:, None]
        if bool(dam.any()):
            sq = E.sqrt()
            prod = (s * eps).sum(-1)
            r = torch.where(prod > 0, prod, torch.ones_like(prod)).sqrt() * (prod > 0)
            r0, q1 = 1e5 / sq, 1e6 / sq
            r1 = r0 + (q1 - r0) / 10.0
            old = torch.maximum(h[..., 0], (Xt / sq).expand_as(r))
            q = torch.where(r < r0, torch.zeros_like(r), torch.where(r < r1, r0 + 10 * (r - r0), q1 + 5 * (r - r1)))
            load = r > old
            D = torch.where(load, 1 - q / torch.where(load, r, torch.ones_like(r)), h[..., 1])
            out = torch.where(dam[..., None], (1 - D)[..., None] * s, out)
            grown = torch.stack([torch.where(load, r, old), D], -1)
            new = torch.cat([torch.where(dam[..., None], grown, new[..., :2]), new[..., 2:]], -1)
        j2 = (self.types == 1)[:, None]
        if bool(j2.any()):
            dev = (eps - h[..., :6]) - one * ((tr - h[..., :3].sum(-1)) / 3)[..., None]
            st = mu[..., None] * two * dev
            n2 = (st * st).sum(-1)
            norm = torch.where(n2 > 0, n2, torch.ones_like(n2)).sqrt()
            f = norm * (n2 > 0) - 0.816496581 * (Sy + Ka * h[..., 6])
            dl = torch.where(f > 0, f, torch.zeros_like(f)) / (2 * mu * (1 + Ka / (3 * mu)))
            dirn = st / norm[..., None]
            k = E / (3 * (1 - 2 * nu))
            sj = st + (k * tr)[..., None] * one - (2 * mu * dl)[..., None] * dirn
            out = torch.where(j2[..., None], sj, out)
            grown = torch.cat([h[..., :6] + dl[..., None] * dirn, (h[..., 6] + 0.816496581 * dl)[..., None]], -1)
            new = torch.where(j2[..., None], grown, new)
        return out, new

    def residual(self, u, h, mats):
        """Unbalanced nodal forces on free unknowns, and the average stress."""
        sig, _ = self.law(self.strains(u), h, mats)
        fe = torch.einsum("gki,egk->ei", self.B, sig) * self.wg
        r = torch.zeros(self.ndof, dtype=torch.float64, device=self.dev).index_add(0, self.dofs.reshape(-1),
                                                                                 fe.reshape(-1))
        return r * self.free, sig.sum((0, 1)) * self.wg

    def tangent(self, u, h, mats):
        """Gauss-point tangents (e, 8, 6, 6) and element matrices (e, 24, 24)."""
        eps = self.strains(u).detach().requires_grad_(True)
        sig, _ = self.law(eps, h.detach(), mats.detach())
        C = torch.stack([torch.autograd.grad(sig[..., i].sum(), eps, retain_graph=i < 5)[0] for i in range(6)], 2)
        return C, torch.einsum("gki,egkl,glj->eij", self.B, C, self.B) * self.wg

    def apply(self, K, x):
        """K x for the columns of x (ndof, m)."""
        ye = torch.einsum("eij,ejm->eim", K, x[self.dofs])
        y = torch.zeros_like(x).index_add(0, self.dofs.reshape(-1), ye.reshape(-1, x.shape[1]))
        return y * self.free[:, None]

    def solve(self, K, b, tol=1e-13):
        """K x = b on the free unknowns (BiCGSTAB with the diagonal, one solve per column of b)."""
        d = torch.zeros(self.ndof, dtype=torch.float64, device=self.dev).index_add(
            0, self.dofs.reshape(-1), torch.diagonal(K, dim1=1, dim2=2).reshape(-1))
        d = torch.where(self.free > 0, 1 / d, torch.zeros_like(d))[:, None]
        x, r = torch.zeros_like(b), b.clone()
        rh, b0 = r.clone(), b.norm(dim=0).clamp_min(1e-300)
        rho = al = om = torch.ones(b.shape[1], dtype=torch.float64, device=self.dev)
        p = v = torch.zeros_like(b)
        div = lambda a, c: torch.where(c != 0, a / torch.where(c != 0, c, torch.ones_like(c)), torch.zeros_like(a))  # noqa: E731
        for it in range(4000):
            new = (rh * r).sum(0)
            p = r + div(new, rho) * div(al, om) * (p - om * v)
            rho = new
            v = self.apply(K, d * p)
            al = div(rho, (rh * v).sum(0))
            s = r - al * v
            t = self.apply(K, d * s)
            om = div((t * s).sum(0), (t * t).sum(0))
            x, r = x + d * (al * p + om * s), s - om * t
            if it % 20 == 19 and bool((r.norm(dim=0) <= tol * b0).all()):
                break
        return x

    def step(self, strain, u, de, h, mats, solve):
        """Newton to rounding at `strain` from u moved with the increment de; returns u."""
        bound = self.affine(strain) * (1 - self.free)
        u = (u + self.affine(de)) * self.free + bound
        r, _ = self.residual(u, h, mats)
        r0 = r.norm()
        for _ in range(40):
            if not bool(r.norm() > 1e-12 * r0):
                break
            du = solve(self.tangent(u, h, mats)[1], -r[:, None])[:, 0]
            t = 1.0
            while True:
                rn, _ = self.residual(u + t * du, h, mats)
                if bool(rn.norm() < r.norm()) or t < 1e-3:
                    break
                t *= 0.5
            if not bool(rn.norm() < r.norm()):
                break
            u, r = u + t * du, rn
        return u


def _exact_rve(case, seed):
    law, size = case["law"], _size(case)
    fe = _Fe(size, [LAWS[law][0], STIFF, (0, 1e7, 0.25, 0.0, 0.0, 0.0)], _phases(case["micro"], size, seed))
    stress, ctan = [], []
    for target in _target(law, case["ngp"], seed):
        u = torch.zeros(fe.ndof, dtype=torch.float64, device=fe.dev)
        h = torch.zeros((len(fe.phases), 8, 7), dtype=torch.float64, device=fe.dev)
        last, kept = fe._t(np.zeros(6)), False
        for f in LAWS[law][2] + (1.0,):
            strain = fe._t(f * target)
            u = fe.step(strain, u, strain - last, h, fe.mats, fe.solve)
            last = strain
            if f < 1.0:
                eps = fe.strains(u)
                new = fe.law(eps, h, fe.mats)[1]
                # J2: the step in which an RVE first yields leaves its history empty (the reference's rule)
                first = law == "j2" and not kept
                kept = kept or not torch.equal(new, h)
                h = h if first else new
        stress.append(fe.residual(u, h, fe.mats)[1])
        C, K = fe.tangent(u, h, fe.mats)
        w = torch.stack([fe.affine(e) for e in torch.eye(6, dtype=torch.float64, device=fe.dev)], 1)
        w = w * (1 - fe.free)[:, None]
        v = w - fe.solve(K, fe.apply(K, w))
        s = torch.einsum("egkl,glj,ejm->km", C, fe.B, v[fe.dofs]) * fe.wg
        ctan.append(s)
    out = {"stress": torch.stack(stress).cpu().numpy(), "ctan": torch.stack(ctan).cpu().numpy()}
    if case["coupling"] == "one_way":
        del out["ctan"]
    elif case["form"] == "plain" and law != "elastic":
        # a forward difference, with a step of 1e-8, of solves that stop at the reference's 1e-3: no 64-bit value
        out["ctan"] = None
    return out


def _exact_path(case, seed):
    size = (case["n"],) * 3
    strains, params, grad = _path_case(case, seed)
    mats = [LAWS[case["law"]][0], STIFF, (0, 1e7, 0.25, 0.0, 0.0, 0.0)]
    fe = _Fe(size, mats, _phases("sphere", size, seed))
    free = torch.nonzero(fe.free)[:, 0]

    def dense(K):
        full = torch.zeros((fe.ndof, fe.ndof), dtype=torch.float64, device=fe.dev)
        i = fe.dofs[:, :, None].expand(-1, 24, 24)
        full.index_put_((i.reshape(-1), i.transpose(1, 2).reshape(-1)), K.reshape(-1), accumulate=True)
        return full[free][:, free]

    def solve(K, b):
        x = torch.zeros_like(b)
        x[free] = torch.linalg.solve(dense(K), b[free])
        return x

    p = fe._t(params).requires_grad_(True)  # E, nu, Xt, Sy, Ka
    e = fe._t(strains).requires_grad_(True)
    m = p[:, [0, 1, 4, 3, 2]]
    h = torch.zeros((len(fe.phases), 8, 7), dtype=torch.float64, device=fe.dev)
    u, last, sigma, loss = torch.zeros(fe.ndof, dtype=torch.float64, device=fe.dev), fe._t(np.zeros(6)), [], 0.0
    for k in range(case["steps"]):
        with torch.no_grad():
            md, hd = m.detach(), h.detach()
        u = fe.step(e[k].detach(), u.detach(), e[k].detach() - last, hd, md, solve)
        last = e[k].detach()
        # one more Newton step with a fixed matrix carries the derivatives of the converged solution
        K = dense(fe.tangent(u, hd, md)[1])
        ud = u * fe.free + fe.affine(e[k]) * (1 - fe.free)
        r, _ = fe.residual(ud, h, m)
        step = torch.linalg.solve(K, r[free][:, None])[:, 0]
        ud = ud - torch.zeros_like(ud).index_add(0, free, step)
        sig = fe.residual(ud, h, m)[1]
        sigma.append(sig.detach())
        loss = loss + (fe._t(grad[k]) * sig).sum()
        h = fe.law(fe.strains(ud), h, m)[1]
    loss.backward()
    return {"sigma": torch.stack(sigma).cpu().numpy(), "grad_params": (p.grad * p.detach()).cpu().numpy(),
            "grad_strains": e.grad.cpu().numpy()}


def _exact_ell(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    nodes = _size(case)
    vals, b = _ell_system(case, seed, dev)
    nn = b.shape[0]
    d = torch.stack([vals[13 * 9 + 4 * i, :nn] for i in range(3)], 1)
    d = torch.where(d != 0, 1 / d, torch.zeros_like(d))
    x, r = torch.zeros_like(b), b.clone()
    p = d * r
    rz, b0 = (r * p).sum(), b.norm()
    for it in range(5000):
        ap = _ell_apply(vals, p, nodes)
        al = rz / (p * ap).sum()
        x, r = x + al * p, r - al * ap
        if it % 20 == 19 and bool(r.norm() < 1e-14 * b0):
            break
        z = d * r
        new = (r * z).sum()
        p, rz = z + new / rz * p, new
    return {"x": x.reshape(-1).cpu().numpy(), "its": None}


def exact(case, seed):
    if case["kind"] == "ell":
        return _exact_ell(case, seed)
    if case["kind"] == "path":
        return _exact_path(case, seed) if case["n"] <= 12 else None
    if case["kind"] == "many":
        return None  # its handles are "rve" cases; together they take too long
    elements = math.prod(_size(case))
    return _exact_rve(case, seed) if elements * case["ngp"] <= 16000 else None
