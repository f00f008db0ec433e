"""The framework's hot calls over the sizes they are used at, for timing and comparing builds.

Each case is one call (or one pair of calls) that a Newton run makes over and over:

* ``tri``:  P1 triangles, p-Laplace or Ginzburg-Landau, a pass of ``assembler.eval``;
* ``he``:   P1 tetrahedra, compressible Neo-Hookean beam, a pass of ``assembler.eval``;
* ``mc``:   plane-strain Mohr-Coulomb slope, P2 / P4 triangles, a pass of ``assembler.eval`` or one
  matrix-free Hessian-vector product (``flags`` = ``"hvp"``);
* ``mc3d``: 3-D Mohr-Coulomb slope, P1 / P2 / P4 tetrahedra, a pass of ``assembler.eval``;
* ``cg``:   the Newton step's linear solve, ``DeviceCG.update`` + ``DeviceCG.solve``;
* ``mlp``:  the warm-start network, one training step or one prediction.

``flags`` names the outputs of an ``eval`` pass: ``e`` energy, ``g`` gradient, ``h`` owned COO Hessian
values.  FP32 element arithmetic is measured through the Hessian with float32 values, which is what it
is selected for (the line search and the convergence test stay on FP64 handles).

``exact`` restates every result in float64 with plain torch: element energies differentiated by
autograd (point by point for Mohr-Coulomb, through the spectral form in 3-D), summed into the COO
pattern by sorted keys.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from fenics_nonlinear_energies_b200 import _lib, meshes
from fenics_nonlinear_energies_b200.assembler import (GLCudaAssembler, HECudaAssembler, PLaplaceCudaAssembler,
                                                      SlopeStability3DCudaAssembler, SlopeStabilityCudaAssembler)
from fenics_nonlinear_energies_b200.newton import DeviceCG
from fenics_nonlinear_energies_b200.warmstart import N_FEATURES, NodalMLP

F64 = torch.float64


def listed():
    return [
        # the reference's p-Laplace grid: a pass of a few microseconds, where launch and latency count
        {"name": "plaplace_128", "kind": "tri", "family": "plaplace", "n": 128, "precision": "fp64", "flags": "egh"},
        # the Ginzburg-Landau configuration of the benchmark, one whole Newton linearisation
        {"name": "gl_1024", "kind": "tri", "family": "gl", "n": 1024, "precision": "fp64", "flags": "egh"},
        # the same grid through the FP32 element path: the Hessian a Newton step solves with
        {"name": "gl_1024_fp32_hessian", "kind": "tri", "family": "gl", "n": 1024, "precision": "fp32", "flags": "h"},
        # line search: some fifteen energy calls per Newton step, on a grid of no round size
        {"name": "gl_701_energy", "kind": "tri", "family": "gl", "n": 701, "precision": "fp64", "flags": "e"},
        # the Neo-Hookean beam configuration (61,440 tets), one whole linearisation
        {"name": "he_160x8x8", "kind": "he", "nx": 160, "ny": 8, "nz": 8, "precision": "fp64", "flags": "egh"},
        # its refinement (491,520 tets): the Hessian callback
        {"name": "he_320x16x16_hessian", "kind": "he", "nx": 320, "ny": 16, "nz": 16, "precision": "fp64",
         "flags": "h"},
        # P4 slope (50,344 elements, 37.7 M COO values), one whole linearisation
        {"name": "mc_p4", "kind": "mc", "degree": 4, "h": 0.16, "precision": "fp64", "flags": "egh"},
        # the same mesh through the FP32 element path
        {"name": "mc_p4_fp32_hessian", "kind": "mc", "degree": 4, "h": 0.16, "precision": "fp32", "flags": "h"},
        # the multigrid smoother's operator: one matrix-free product
        {"name": "mc_p4_hvp", "kind": "mc", "degree": 4, "h": 0.16, "precision": "fp64", "flags": "hvp"},
        # the 3-D slope on P2 tetrahedra at the benchmark's size (61,440 elements)
        {"name": "mc3d_p2", "kind": "mc3d", "degree": 2, "nx": 40, "ny": 16, "nz": 16, "flags": "egh"},
        # a Newton step's linear solve on a Ginzburg-Landau Hessian near its minimiser
        {"name": "cg_gl_512", "kind": "cg", "n": 512},
        # one optimiser step of the warm-start network at its training batch
        {"name": "mlp_train_8192", "kind": "mlp", "rows": 8192, "width": 256, "train": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("tri", "tri", "he", "he", "mc", "mc", "mc3d", "cg", "mlp"))
    if kind == "tri":
        precision = rng.choice(("fp64", "fp64", "fp32"))
        return {"kind": kind, "family": rng.choice(("plaplace", "gl")), "n": _log_int(rng, 17, 1024),
                "precision": precision, "flags": "h" if precision == "fp32" else rng.choice(("egh", "eg", "g", "e", "h"))}
    if kind == "he":
        precision = rng.choice(("fp64", "fp64", "fp32"))
        m = _log_int(rng, 2, 16)
        return {"kind": kind, "nx": m * rng.randint(5, 20), "ny": m, "nz": max(1, m - rng.randint(0, 2)),
                "precision": precision, "flags": "h" if precision == "fp32" else rng.choice(("egh", "eg", "g", "e", "h"))}
    if kind == "mc":
        precision = rng.choice(("fp64", "fp64", "fp32"))
        return {"kind": kind, "degree": rng.choice((2, 4)), "h": round(math.exp(rng.uniform(math.log(0.16), math.log(1.5))), 3),
                "precision": precision, "flags": "h" if precision == "fp32" else rng.choice(("egh", "eg", "e", "h", "hvp"))}
    if kind == "mc3d":
        degree = rng.choice((1, 2, 2, 4))
        m = _log_int(rng, 1, 3 if degree == 4 else 8 if degree == 2 else 10)
        # three layers of hexes: the free degrees of freedom then come in whole blocks of three
        return {"kind": kind, "degree": degree, "nx": m * rng.randint(2, 4), "ny": m, "nz": 3 * rng.randint(1, 2 if m > 2 else 4),
                "flags": rng.choice(("egh", "egh", "h", "eg"))}
    if kind == "cg":
        return {"kind": kind, "n": _log_int(rng, 40, 800)}
    return {"kind": kind, "rows": _log_int(rng, 200, 60000), "width": 256, "train": rng.random() < 0.6}


# ---------------------------------------------------------------------------
# meshes and states (host)
# ---------------------------------------------------------------------------
def _mesh_key(case):
    return tuple((k, case.get(k)) for k in ("kind", "family", "n", "nx", "ny", "nz", "degree", "h"))


@functools.lru_cache(maxsize=32)
def _mesh(key):
    """The problem dictionary of a mesh; a program has it from its mesh file."""
    c = dict(key)
    if c["kind"] == "he":
        return meshes.he_beam_problem(nx=c["nx"], ny=c["ny"], nz=c["nz"])[0]
    if c["kind"] == "mc":
        return meshes.slope_problem(h=c["h"], degree=c["degree"], lam=1.0)
    if c["kind"] == "mc3d":
        return meshes.slope3d_problem(nx=c["nx"], ny=c["ny"], nz=c["nz"], degree=c["degree"], lam=1.0)
    if c["kind"] == "tri" and c["family"] == "plaplace":
        return meshes.plaplace_problem(n=c["n"], seed=0)[0]
    return meshes.gl_problem(n=c["n"])[0]


def _dirichlet_key(case):
    return "u_0_ref" if case["kind"] == "he" else "u_0"


def _full_state(case, seed):
    """All degrees of freedom (Dirichlet ones included) of the state that the pass is taken at."""
    params = _mesh(_mesh_key(case))
    rng = np.random.default_rng([seed, 17])
    free = params["freedofs"]
    if case["kind"] == "he":  # twisted about its axis, as a load step's state, with a small perturbation
        X = params["nodes2coord"]
        a = rng.uniform(0.2, 0.8) * X[:, 0] / X[:, 0].max()
        c, s = np.cos(a), np.sin(a)
        full = np.stack([X[:, 0], c * X[:, 1] + s * X[:, 2], -s * X[:, 1] + c * X[:, 2]], axis=1).ravel()
        full[free] += 1e-5 * rng.standard_normal(free.size)
        return full
    full = np.array(params["u_0"], dtype=np.float64)
    if case["kind"] == "tri":
        full[free] = rng.random(free.size) if case["family"] == "plaplace" else rng.uniform(-0.5, 0.5, free.size)
    elif case["kind"] == "cg":  # a transition layer of the model's width along the boundary
        x, y = params["nodes"][:, 0], params["nodes"][:, 1]
        width = math.sqrt(2.0 * params["eps"])
        layer = np.tanh((1.0 - np.abs(x)) / width) * np.tanh((1.0 - np.abs(y)) / width)
        full[free] = (layer + 0.02 * rng.standard_normal(layer.size))[free]
    elif case["kind"] == "mc":  # a settling slope, elastic and plastic regions side by side
        x, y = params["nodes"][:, 0] / 40.0, params["nodes"][:, 1] / 20.0
        amp, ph = rng.uniform(0.015, 0.03), rng.uniform(0.0, 1.0, 2)
        ux = amp * 4.0 * y * x * (1.0 - x) * (1.0 + 0.3 * np.sin(9.0 * x + 5.0 * y + 6.0 * ph[0]))
        uy = -amp * y * y * (1.0 + 0.3 * np.sin(7.0 * x - 6.0 * y + 6.0 * ph[1]))
        full[free] = np.stack([ux, uy], axis=1).ravel()[free]
    else:
        X = np.asarray(params["nodes"], dtype=np.float64)
        x, y, z = (X / X.max(axis=0)).T
        amp, ph = rng.uniform(0.03, 0.07), rng.uniform(0.0, 1.0, 3)
        u = np.stack([amp * z * x * (1 - x) * np.sin(3.0 * y + 1.0 + ph[0]),
                      amp * z * y * (1 - y) * np.cos(2.0 * x + ph[1]),
                      -amp * z * (1.0 + 0.5 * np.sin(4.0 * x + ph[2]) * np.cos(3.0 * y))], axis=1)
        full[free] = u.ravel()[free]
    return full


def _block(case):
    return {"he": 3, "mc": 2, "mc3d": 3}.get(case["kind"], 1)


def _assembler(case, params):
    fp32 = case.get("precision") == "fp32"
    kw = {"precision": "fp32", "hess_dtype": torch.float32} if fp32 else {}
    cls = {"he": HECudaAssembler, "mc": SlopeStabilityCudaAssembler, "mc3d": SlopeStability3DCudaAssembler,
           "cg": GLCudaAssembler}.get(case["kind"])
    if cls is None:
        cls = PLaplaceCudaAssembler if case["family"] == "plaplace" else GLCudaAssembler
    return cls(params, **kw)


def _mlp_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.randn(case["rows"], N_FEATURES, device="cuda", generator=g)
    T = 0.1 * torch.randn(case["rows"], 3, device="cuda", generator=g)
    return X.to(torch.bfloat16), T


def _mlp_dims(case):
    return (N_FEATURES, case["width"], case["width"], case["width"], 3)


def prepare(case, seed):
    if case["kind"] == "mlp":
        X16, T = _mlp_inputs(case, seed)
        return {"kind": "mlp", "net": NodalMLP(_mlp_dims(case), seed=seed), "X": X16, "T": T, "train": case["train"]}
    params = _mesh(_mesh_key(case))
    asm = _assembler(case, params)
    full = _full_state(case, seed)
    if case["kind"] == "he":
        asm.update_dirichlet(full)
    free, perm = params["freedofs"], asm.layout.perm
    u = torch.as_tensor(full[free][perm], device=asm.device)
    s = {"kind": case["kind"], "asm": asm, "u": u}
    if case["kind"] == "cg":
        _, g, h = asm.eval(u, _lib.FNE_GRAD | _lib.FNE_HESS)
        return dict(s, cg=DeviceCG.for_assembler(asm), b=-g, h=h)
    if case["flags"] == "hvp":
        x = np.random.default_rng([seed, 23]).standard_normal(free.size)
        asm.prepare_matrix_free_operator(u)
        return dict(s, kind="hvp", x=torch.as_tensor(x[perm], device=asm.device))
    flags = 0
    for letter, bit in (("e", _lib.FNE_ENERGY), ("g", _lib.FNE_GRAD), ("h", _lib.FNE_HESS)):
        flags |= bit if letter in case["flags"] else 0
    return dict(s, flags=flags)


def run(state):
    kind = state["kind"]
    if kind == "mlp":
        net = state["net"]
        if not state["train"]:
            return net.forward(state["X"])
        Y = net.forward(state["X"], keep=True)
        diff = Y - state["T"]
        gW, gb = net.backward((2.0 / diff.numel()) * diff)
        net.adam_step(gW, gb, lr=1e-3)
        return {"Y": Y, "gW": gW, "gb": gb, "W": net.W, "b": net.b}
    if kind == "cg":
        state["cg"].update(state["h"])
        x, its = state["cg"].solve(state["b"], rtol=1e-3, maxit=500)
        return {"x": x, "iterations": its}
    if kind == "hvp":
        return state["asm"].matrix_free_mult("matfree_element", state["x"])
    flags = state["flags"]
    e, g, h = state["asm"].eval(state["u"], flags)
    return {k: v for k, v, bit in (("e", e, _lib.FNE_ENERGY), ("g", g, _lib.FNE_GRAD), ("h", h, _lib.FNE_HESS))
            if flags & bit}


# ---------------------------------------------------------------------------
# work: what a pass has to move and compute
# ---------------------------------------------------------------------------
def _sizes(case):
    """(elements, nodes per element, free degrees of freedom, COO values, geometry values per element)."""
    kind = case["kind"]
    if kind in ("tri", "cg"):
        m = case["n"] - 1
        return 2 * case["n"] ** 2, 3, m * m, m * m + 2 * (2 * m * (m - 1) + (m - 1) ** 2), 7
    if kind == "he":
        d = (case["nx"] - 1, case["ny"] + 1, case["nz"] + 1)
        blocks = 0
        for mask in range(1, 8):
            blocks += 2 * math.prod(max(0, d[i] - (mask >> i & 1)) for i in range(3))
        nodes = math.prod(d)
        return 6 * case["nx"] * case["ny"] * case["nz"], 4, 3 * nodes, 9 * (blocks + nodes), 13
    params = _mesh(_mesh_key(case))
    n_el, npe = params["elems_scalar"].shape
    k = case["degree"]
    free = int(params["freedofs"].size)
    if kind == "mc":  # unique node pairs of a triangulation: the pairs on a shared edge count once
        blocks = n_el * npe * npe - 1.5 * n_el * (k + 1) ** 2 + 0.5 * n_el
        geometry = 5 * (params["quad_w"].size if params["det_j"].ndim == 2 else 1)
        return n_el, npe, free, int(4 * blocks), geometry
    face = (k + 1) * (k + 2) // 2
    blocks = n_el * npe * npe - 2.0 * n_el * face ** 2 + 7.0 / 6.0 * n_el * (k + 1) ** 2 - n_el / 6.0
    nq = params["quad_weight"].shape[1]
    return n_el, npe, free, int(9 * blocks), nq * (3 * npe + 6)


def work(case):
    if case["kind"] == "mlp":
        dims, rows = _mlp_dims(case), case["rows"]
        weights = sum(a * b for a, b in zip(dims[:-1], dims[1:]))
        if not case["train"]:
            return {"bytes": rows * (2 * dims[0] + 4 * dims[-1]) + 2 * weights, "flops": 2 * rows * weights}
        # activations written forward and read backward; weights, gradient and two moments in FP32
        acts = rows * sum(dims[1:-1])
        return {"bytes": rows * (2 * dims[0] + 12 * dims[-1]) + 2 * 2 * acts + 30 * weights,
                "flops": 2 * rows * (3 * weights - dims[0] * dims[1])}
    n_el, npe, free, nnz, geometry = _sizes(case)
    if case["kind"] == "cg":  # 100 iterations: the matrix, its columns and twelve vector streams each
        return {"bytes": 100 * (nnz * 12 + free * 96), "flops": 100 * (2 * nnz + 13 * free)}
    real = 4 if case.get("precision") == "fp32" else 8
    flags = case["flags"]
    read = n_el * (4 * npe + real * geometry) + 8 * free
    nq, dim = {"tri": (1, 2), "he": (1, 3), "mc": (19 if case.get("degree") == 4 else 7, 2),
               "mc3d": ({1: 1, 2: 11, 4: 24}.get(case.get("degree"), 1), 3)}[case["kind"]]
    if flags == "hvp":
        return {"bytes": read + 8 * free + n_el * nq * 6 * real, "flops": n_el * nq * (16 * npe + 30)}
    if case["kind"] in ("mc", "mc3d") or (case["kind"] == "tri" and case["family"] == "plaplace"):
        read += 8 * free if "e" in flags or "g" in flags else 0
    wrote = (8 if "e" in flags else 0) + (8 * free if "g" in flags else 0) + (real * nnz if "h" in flags else 0)
    flops = nq * (2 * dim * dim * npe + 60 * dim)
    if "g" in flags:
        flops += nq * 2 * dim * dim * npe
    if "h" in flags:
        flops += nq * npe * (npe + 1) // 2 * 2 * dim ** 4
    return {"bytes": read + wrote, "flops": n_el * flops}


# ---------------------------------------------------------------------------
# float64 results in plain torch
# ---------------------------------------------------------------------------
def _dev(a):
    return torch.as_tensor(np.asarray(a), device="cuda")


def _derivatives(f, x, second=True):
    """Values, gradients and Hessians of ``f`` at the rows of ``x`` (the rows do not interact)."""
    x = x.detach().requires_grad_(True)
    e = f(x)
    g = torch.autograd.grad(e.sum(), x, create_graph=second)[0]
    if not second:
        return e.detach(), g.detach(), None
    H = [torch.autograd.grad(g[:, i].sum(), x, retain_graph=True)[0] for i in range(x.shape[1])]
    return e.detach(), g.detach(), torch.stack(H, dim=1)


def _where(cond, a, b):
    return torch.where(cond, a, b)


def _mc_density(params):
    """Plane-strain Mohr-Coulomb energy density of strains (N, 3): elastic, return to the line, apex."""
    E, nu, c = params["E"], params["nu"], params["cohesion"]
    phi, reg = math.radians(params["phi_deg"]), params["reg"]
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    S11, S12, S33 = (1 - nu * nu) / E, -nu * (1 + nu) / E, 1 / mu
    al, be, kap = 1 + math.sin(phi), 1 - math.sin(phi), 2 * c * math.cos(phi)
    det = S11 * S11 - S12 * S12
    z1, z2 = (S11 * al + S12 * be) / det, (-S12 * al - S11 * be) / det

    def f(eps):
        sx = (lam + 2 * mu) * eps[:, 0] + lam * eps[:, 1]
        sy = lam * eps[:, 0] + (lam + 2 * mu) * eps[:, 1]
        t = mu * eps[:, 2]
        m, d = 0.5 * (sx + sy), 0.5 * (sx - sy)
        r = torch.sqrt(d * d + t * t + reg * reg)
        s1, s2 = m + r, m - r
        elastic = al * s1 - be * s2 - kap <= 0
        lm = (al * s1 - be * s2 - kap) / (al * z1 - be * z2)
        p1, p2 = s1 - lm * z1, s2 - lm * z2
        line = p1 >= p2
        apex = torch.full_like(p1, kap / (al - be))
        p1, p2 = _where(line, p1, apex), _where(line, p2, apex)
        dd, tt = _where(elastic, torch.ones_like(d), d), _where(elastic, torch.zeros_like(t), t)
        rho = torch.sqrt(dd * dd + tt * tt)
        mp, rp = 0.5 * (p1 + p2), 0.5 * (p1 - p2)
        gx, gy, gt = mp + rp * dd / rho, mp - rp * dd / rho, rp * tt / rho

        def psi(a, b, q):
            quad = S11 * (a * a + b * b) + 2 * S12 * a * b + S33 * q * q
            return a * eps[:, 0] + b * eps[:, 1] + q * eps[:, 2] - 0.5 * quad

        return _where(elastic, psi(sx, sy, t), psi(gx, gy, gt))

    return f


def _mc3d_density(c_bar, sp, G, K, la):
    """3-D Mohr-Coulomb energy density of ordered principal strains (N, 3), l1 >= l2 >= l3."""
    def f(z):
        l1, l2, l3 = z[:, 0], z[:, 1], z[:, 2]
        I1 = l1 + l2 + l3
        tr = 2 * la * sp * I1 - c_bar
        f_tr = 2 * G * ((1 + sp) * l1 - (1 - sp) * l3) + tr
        g_sl, g_sr = (l1 - l2) / (1 + sp), (l2 - l3) / (1 - sp)
        g_la, g_ra = (l1 + l2 - 2 * l3) / (3 - sp), (2 * l1 - l2 - l3) / (3 + sp)
        d_s = 4 * la * sp ** 2 + 4 * G * (1 + sp ** 2)
        d_l = 4 * la * sp ** 2 + G * (1 + sp) ** 2 + 2 * G * (1 - sp) ** 2
        d_r = 4 * la * sp ** 2 + 2 * G * (1 + sp) ** 2 + G * (1 - sp) ** 2
        d_a = 4 * K * sp ** 2
        m_s = f_tr / d_s
        m_l = (G * ((1 + sp) * (l1 + l2) - 2 * (1 - sp) * l3) + tr) / d_l
        m_r = (G * (2 * (1 + sp) * l1 - (1 - sp) * (l2 + l3)) + tr) / d_r
        m_a = (2 * K * sp * I1 - c_bar) / d_a
        base, quad = 0.5 * la * I1 ** 2, G * (l1 ** 2 + l2 ** 2 + l3 ** 2)
        el = f_tr <= 0
        sm = m_s <= torch.minimum(g_sl, g_sr)
        left = (g_sl < g_sr) & (m_l >= g_sl) & (m_l <= g_la)
        right = (g_sl > g_sr) & (m_r >= g_sr) & (m_r <= g_ra)
        psi_l = base + G * (l3 ** 2 + 0.5 * (l1 + l2) ** 2) - 0.5 * d_l * m_l ** 2
        psi_r = base + G * (l1 ** 2 + 0.5 * (l2 + l3) ** 2) - 0.5 * d_r * m_r ** 2
        out = _where(right, psi_r, 0.5 * K * I1 ** 2 - 0.5 * d_a * m_a ** 2)
        out = _where(left, psi_l, out)
        out = _where(sm, base + quad - 0.5 * d_s * m_s ** 2, out)
        return _where(el, base + quad, out)

    return f


def _mc3d_points(eps, scalars):
    """Density, stress (N, 6) and tangent (N, 6, 6) at strains (N, 6) through their spectral form."""
    A = torch.empty(eps.shape[0], 3, 3, dtype=F64)
    e = eps.cpu()
    for (i, j), k, s in (((0, 0), 0, 1.0), ((1, 1), 1, 1.0), ((2, 2), 2, 1.0), ((0, 1), 3, 0.5), ((1, 2), 4, 0.5), ((0, 2), 5, 0.5)):
        A[:, i, j] = A[:, j, i] = s * e[:, k]
    w, V = torch.linalg.eigh(A)
    z, V = w.flip(-1).to(eps.device), V.flip(-1).to(eps.device)
    psi, F, FF = _derivatives(_mc3d_density(*scalars), z)

    def voigt(a, b):  # symmetrised a (x) b contracted with the engineering strain components
        return torch.stack([a[:, 0] * b[:, 0], a[:, 1] * b[:, 1], a[:, 2] * b[:, 2],
                            0.5 * (a[:, 0] * b[:, 1] + a[:, 1] * b[:, 0]), 0.5 * (a[:, 1] * b[:, 2] + a[:, 2] * b[:, 1]),
                            0.5 * (a[:, 0] * b[:, 2] + a[:, 2] * b[:, 0])], dim=1)

    M = [voigt(V[:, :, k], V[:, :, k]) for k in range(3)]
    sig = sum(F[:, k, None] * M[k] for k in range(3))
    D = sum(FF[:, k, m, None, None] * M[k][:, :, None] * M[m][:, None, :] for k in range(3) for m in range(3))
    for k, m in ((0, 1), (0, 2), (1, 2)):
        gap = z[:, k] - z[:, m]
        near = gap.abs() <= 1e-13 * z.abs().amax(1)
        c = _where(near, FF[:, k, k] - FF[:, k, m], (F[:, k] - F[:, m]) / _where(near, torch.ones_like(gap), gap))
        S = voigt(V[:, :, k], V[:, :, m])
        D = D + 2.0 * c[:, None, None] * S[:, :, None] * S[:, None, :]
    return psi, sig, D


def _strain_operator(gx, gy, gz=None):
    """Rows (xx, yy, xy) or (xx, yy, zz, xy, yz, xz) of the strain operator from basis gradients (E, nq, n)."""
    E, nq, n = gx.shape
    if gz is None:
        B = torch.zeros(E, nq, 3, 2 * n, dtype=F64, device=gx.device)
        B[:, :, 0, 0::2], B[:, :, 1, 1::2], B[:, :, 2, 0::2], B[:, :, 2, 1::2] = gx, gy, gy, gx
        return B
    B = torch.zeros(E, nq, 6, 3 * n, dtype=F64, device=gx.device)
    B[:, :, 0, 0::3], B[:, :, 1, 1::3], B[:, :, 2, 2::3] = gx, gy, gz
    B[:, :, 3, 0::3], B[:, :, 3, 1::3] = gy, gx
    B[:, :, 4, 1::3], B[:, :, 4, 2::3] = gz, gy
    B[:, :, 5, 0::3], B[:, :, 5, 2::3] = gz, gx
    return B


def _element_results(case, params, v, sl, second):
    """Energies, gradients and Hessians of the elements ``sl`` with nodal values ``v``."""
    kind = case["kind"]
    if kind in ("tri", "cg"):
        dx, dy, vol = (_dev(params[k][sl]) for k in ("dvx", "dvy", "vol"))
        if "p" in params:
            p = params["p"]
            return _derivatives(lambda w: ((w * dx).sum(1) ** 2 + (w * dy).sum(1) ** 2) ** (p / 2) * vol / p, v, second)
        ip, wq, eps = _dev(params["ip"]), _dev(params["w"]), params["eps"]
        return _derivatives(lambda w: vol * (0.5 * eps * ((w * dx).sum(1) ** 2 + (w * dy).sum(1) ** 2)
                                             + (0.25 * ((w @ ip) ** 2 - 1.0) ** 2) @ wq), v, second)
    if kind == "he":
        G = torch.stack([_dev(params[k][sl]) for k in ("dphix", "dphiy", "dphiz")], dim=2)
        vol, C1, D1 = _dev(params["vol"][sl]), params["C1"], params["D1"]

        def f(w):
            F = torch.einsum("eai,eaj->eij", w.reshape(-1, 4, 3), G)
            J = (F[:, 0] * torch.linalg.cross(F[:, 1], F[:, 2])).sum(1)
            return vol * (C1 * ((F * F).sum((1, 2)) - 3.0 - 2.0 * torch.log(J)) + D1 * (J - 1.0) ** 2)

        return _derivatives(f, v, second)
    if kind == "mc":
        inv, det = _dev(params["inv_jac"][sl]), _dev(params["det_j"][sl])
        if inv.ndim == 2:
            inv, det = inv[:, None, :], det[:, None]
        d1, d2 = _dev(params["dhat1"])[None], _dev(params["dhat2"])[None]
        B = _strain_operator(inv[..., 0, None] * d1 + inv[..., 1, None] * d2, inv[..., 2, None] * d1 + inv[..., 3, None] * d2)
        wq = det * _dev(params["quad_w"])[None]
        eps = torch.einsum("eqsi,ei->eqs", B, v)
        psi, sig, D = _derivatives(_mc_density(params), eps.reshape(-1, 3), second)
        m = 3
    else:
        B = _strain_operator(*(_dev(params[k][sl]) for k in ("dphix", "dphiy", "dphiz")))
        wq = _dev(params["quad_weight"][sl])
        eps = torch.einsum("eqsi,ei->eqs", B, v)
        scalars = [float(params[k].flat[0]) for k in ("c_bar", "sin_phi", "shear", "bulk", "lame")]
        psi, sig, D = _mc3d_points(eps.reshape(-1, 6), scalars)
        m = 6
    E, nq = wq.shape
    e = (wq * psi.reshape(E, nq)).sum(1)
    g = torch.einsum("eqsi,eqs->ei", B, wq[..., None] * sig.reshape(E, nq, m))
    if not second:
        return e, g, None
    DB = torch.einsum("eqst,eqti->eqsi", wq[..., None, None] * D.reshape(E, nq, m, m), B)
    n = B.shape[-1]
    return e, g, B.reshape(E, nq * m, n).transpose(1, 2) @ DB.reshape(E, nq * m, n)


class _Exact:
    """Energy, gradient and Hessian values in the framework's ordering: reordered free DOFs, COO rows of the
    free-DOF element graph in their original order."""

    def __init__(self, case, seed, second):
        params = _mesh(_mesh_key(case))
        free, bs = params["freedofs"], _block(case)
        coords = np.asarray(params["nodes2coord" if case["kind"] == "he" else "nodes"])[free[::bs] // bs]
        order = np.lexsort(tuple(coords[:, d] for d in reversed(range(coords.shape[1]))))
        self.perm = torch.as_tensor((bs * order[:, None] + np.arange(bs)).ravel(), device="cuda")
        full = _dev(_full_state(case, seed))
        elems = _dev(params["elems"])
        n, nf = elems.shape[1], int(free.size)
        index = torch.full((full.numel(),), -1, dtype=torch.int64, device="cuda")
        index[_dev(free)] = torch.arange(nf, device="cuda")
        self.nf, self.energy = nf, 0.0
        self.grad = torch.zeros(nf, dtype=F64, device="cuda")
        f = params.get("f", params.get("force"))
        if f is not None:
            f = _dev(f)[_dev(free)]
            self.grad -= f
            self.energy -= float(f @ full[_dev(free)])
        x = None
        if case.get("flags") == "hvp":
            x = torch.zeros_like(full)
            x[_dev(free)] = _dev(np.random.default_rng([seed, 23]).standard_normal(nf))
            self.product = torch.zeros(nf, dtype=F64, device="cuda")
        pattern = second and x is None
        if pattern:
            dof = index[elems]
            key = (dof[:, :, None] * nf + dof[:, None, :])[(dof[:, :, None] >= 0) & (dof[:, None, :] >= 0)]
            key, place = torch.unique(key, return_inverse=True)
            self.rows, self.cols = key // nf, key % nf
            self.hess = torch.zeros(key.numel(), dtype=F64, device="cuda")
            del key
        step, at = max(1, 40_000_000 // (n * n * 8)), 0
        for k in range(0, elems.shape[0], step):
            sl = slice(k, min(k + step, elems.shape[0]))
            dof = index[elems[sl]]
            ok = dof >= 0
            e, g, H = _element_results(case, params, full[elems[sl]], sl, second)
            self.energy += float(e.sum())
            self.grad.index_add_(0, dof[ok], g[ok])
            if x is not None:
                y = torch.einsum("eij,ej->ei", H, x[elems[sl]])
                self.product.index_add_(0, dof[ok], y[ok])
            elif second:
                values = H[ok[:, :, None] & ok[:, None, :]]
                self.hess.index_add_(0, place[at:at + values.numel()], values)
                at += values.numel()


def _exact_cg(case, seed):
    """Jacobi-preconditioned CG from zero to ``|r| <= 1e-3 |b|`` (500 iterations at most)."""
    r = _Exact(case, seed, True)
    A = torch.sparse_coo_tensor(torch.stack((r.rows, r.cols)), r.hess, (r.nf, r.nf)).to_sparse_csr()
    diag = torch.zeros(r.nf, dtype=F64, device="cuda")
    on = r.rows == r.cols
    diag[r.rows[on]] = r.hess[on]
    b = -r.grad
    x, res = torch.zeros_like(b), b.clone()
    z = res / diag.abs()
    p, rz, its = z.clone(), res @ z, 0
    while its < 500:
        its += 1
        Ap = A @ p
        alpha = rz / (p @ Ap)
        x += alpha * p
        res -= alpha * Ap
        if float(res.norm()) <= 1e-3 * float(b.norm()):
            break
        z = res / diag.abs()
        new = res @ z
        p, rz = z + (new / rz) * p, new
    return {"x": x[r.perm], "iterations": None}


def _exact_mlp(case, seed):
    """The network without BF16 rounding, and one Adam step from zero moments.  The biases start from zero, so
    their first step is the sign of each gradient, which the BF16 operands do not settle for the small ones: no
    value stands for them."""
    X16, T = _mlp_inputs(case, seed)
    dims = _mlp_dims(case)
    g = torch.Generator().manual_seed(seed)
    W = [(torch.randn(o, i, generator=g, dtype=torch.float32) * math.sqrt(2.0 / i)).double().cuda().requires_grad_(True)
         for i, o in zip(dims[:-1], dims[1:])]
    b = [torch.zeros(o, dtype=F64, device="cuda", requires_grad=True) for o in dims[1:]]
    h = X16.double()
    for k in range(len(W)):
        h = h @ W[k].T + b[k]
        if k < len(W) - 1:
            h = torch.nn.functional.silu(h)
    if not case["train"]:
        return h.detach()
    grads = torch.autograd.grad(((h - T.double()) ** 2).mean(), W + b)
    new = [(p - 1e-3 * d / (d.abs() + 1e-8)).detach() for p, d in zip(W, grads)]
    return {"Y": h.detach(), "gW": list(grads[:len(W)]), "gb": list(grads[len(W):]), "W": new, "b": None}


def exact(case, seed):
    if case["kind"] == "mlp":
        return _exact_mlp(case, seed)
    if case["kind"] == "cg":
        return _exact_cg(case, seed)
    flags = case["flags"]
    r = _Exact(case, seed, "h" in flags)
    if flags == "hvp":
        return r.product[r.perm]
    out = {}
    if "e" in flags:
        out["e"] = torch.tensor([r.energy], dtype=F64)
    if "g" in flags:
        out["g"] = r.grad[r.perm]
    if "h" in flags:
        out["h"] = r.hess
    return out
