"""Work that a user of this package has it do, as cases to be timed and compared.

A solver calls the builder once or more in every Newton iteration.  The cases are those calls, through
the public entry points, from a 192-triangle slope to one of 277k quadratic tetrahedra:

* ``newton``: F and the regularised tangent K of one Newton iteration
  (``ConstitutiveOperator.build_F_K_regularized_all_free``), handed over on the host (the default: a
  host solver reads F and the CSR values) or left on the device (``host_outputs = False``), in the
  plain (FP64) or the mixed form;
* ``continuation``: the residual and the potential energy of a trial state
  (``build_F_all_free``, ``potential_energy``), what damping and the direct continuation ask for;
* ``bddc``: stresses and tangents of a state, then the regularised matrix of the subdomain that owns
  the lower half of the nodes (``build_bddc_regularized_matrix``);
* ``assemble``: force and tangent from a caller's own stresses and (not symmetric) tangents, a
  material law of the user's (``assemble_owned_force_from_local_stress``,
  ``assemble_owned_tangent_values``).

Meshes, materials and displacements are the package's synthetic slopes (``synthetic.py``); the seed
sets the shear band's amplitude and noise, the strength-reduction factor, and the stresses and tangents
of ``assemble``.
"""

from __future__ import annotations

import math
import random
from functools import lru_cache

import numpy as np
import torch

from slope_stability_petsc4py_gb300 import (
    ConstitutiveOperator,
    assemble_owned_force_from_local_stress,
    assemble_owned_tangent_values,
    prepare_bddc_subdomain_pattern,
    prepare_owned_tangent_pattern,
    synthetic,
)
from slope_stability_petsc4py_gb300.fem import quadrature, reference_gradients

R = 0.1  # regularisation factor of the tangent

# (dim, element): nodes, points per element, CSR entries per dof (about), FP64 operations per element
# of the strain and of the force, and of one plastic point's tangent (about, in flops)
KINDS = {
    (2, "P1"): (3, 1, 14, 60, 100),
    (2, "P2"): (6, 7, 23, 700, 500),
    (2, "P4"): (15, 12, 50, 2900, 2900),
    (3, "P1"): (4, 1, 45, 200, 700),
    (3, "P2"): (10, 11, 83, 1900, 2400),
    (3, "P4"): (35, 24, 209, 31000, 39000),
}
# shear-band displacement (m) that makes about a tenth of the points yield, by material set
AMPLITUDE = {(2, 1): 0.0072, (2, 4): 0.0035, (3, 1): 0.0157, (3, 4): 0.003}


def _case(task, dim, elem, nx, ny, nz, layers=1, form="plain", host=False, **more):
    return dict(task=task, dim=dim, elem=elem, nx=nx, ny=ny, nz=nz, layers=layers, form=form, host=host, **more)


def listed():
    return [
        # a coarse 2D slope, as a first look or a parameter study solves it by the thousand; host hand-off
        _case("newton", 2, "P2", 12, 8, 1, host=True, name="newton_2d_p2_small"),
        # the 2D benchmark slope (20,000 quadratic triangles), solver on the device
        _case("newton", 2, "P2", 100, 100, 1, name="newton_2d_p2"),
        # quartic triangles, layered soil, sides that no tile divides
        _case("newton", 2, "P4", 61, 43, 1, layers=4, name="newton_2d_p4"),
        # a modest 3D slope as the default operator serves it: F and the CSR values on the host
        _case("newton", 3, "P2", 20, 8, 20, host=True, name="newton_3d_p2_host"),
        # the 3D benchmark slope (100,800 quadratic tetrahedra), solver on the device
        _case("newton", 3, "P2", 40, 14, 30, name="newton_3d_p2"),
        # the same in the mixed-precision form
        _case("newton", 3, "P2", 40, 14, 30, form="mixed", name="newton_3d_p2_mixed"),
        # the largest: a refined layered 3D slope, 276,768 quadratic tetrahedra
        _case("newton", 3, "P2", 62, 24, 31, layers=4, name="newton_3d_p2_large"),
        # quartic tetrahedra, layered, sides that no tile divides
        _case("newton", 3, "P4", 19, 7, 13, layers=4, name="newton_3d_p4"),
        # quartic tetrahedra in the mixed form (tensor cores)
        _case("newton", 3, "P4", 14, 6, 10, layers=4, form="mixed", name="newton_3d_p4_mixed"),
        # a trial state of the damping or of the direct continuation on the benchmark slope
        _case("continuation", 3, "P2", 40, 14, 30, name="continuation_3d_p2"),
        # the subdomain matrix of half of a layered slope, for a BDDC preconditioner
        _case("bddc", 3, "P2", 30, 11, 21, layers=4, name="bddc_3d_p2"),
        # a caller's own stresses and tangents
        _case("assemble", 3, "P2", 20, 8, 20, name="assemble_3d_p2"),
    ]


def draw(rng: random.Random):
    task = rng.choice(["newton"] * 6 + ["continuation", "bddc", "assemble"])
    dim, elem = rng.choice([(2, "P1"), (2, "P2"), (2, "P2"), (2, "P4"), (3, "P1"), (3, "P2"), (3, "P2"), (3, "P2"), (3, "P2"),
                            (3, "P4"), (3, "P4")])
    top = {(2, "P1"): 60000, (2, "P2"): 40000, (2, "P4"): 12000, (3, "P1"): 100000, (3, "P2"): 150000, (3, "P4"): 9000}
    cells = math.exp(rng.uniform(math.log(40.0), math.log(top[dim, elem] / (2 if dim == 2 else 6))))
    # sides in random proportions around the slope's own
    if dim == 2:
        nx = max(4, round(math.sqrt(cells * rng.uniform(0.8, 2.5))))
        ny, nz = max(2, round(cells / nx)), 1
    else:
        ny = max(2, round((cells * rng.uniform(0.15, 0.5)) ** (1.0 / 3.0)))
        nx = max(4, round(math.sqrt(cells / ny * rng.uniform(0.8, 2.0))))
        nz = max(2, round(cells / (nx * ny)))
    return _case(task, dim, elem, nx, ny, nz, layers=rng.choice([1, 4]), form=rng.choice(["plain", "plain", "plain", "mixed"]),
                 host=task == "newton" and rng.random() < 0.3)


# ------------------------------------------------------------------------------------------- inputs


@lru_cache(maxsize=4)
def _slope(dim, elem, nx, ny, nz, layers):
    if dim == 2:
        return synthetic.slope_mesh_2d(nx, ny, elem_type=elem, n_layers=layers)
    return synthetic.slope_mesh_3d(nx, ny, nz, elem_type=elem, n_layers=layers)


def _problem(case, seed):
    """Mesh, materials, displacement (dim, n_nodes) and strength-reduction factor."""
    mesh = _slope(case["dim"], case["elem"], case["nx"], case["ny"], case["nz"], case["layers"])
    mats = synthetic.MaterialSet.layered(4, seed=0) if case["layers"] > 1 else synthetic.MaterialSet.homogeneous()
    rng = random.Random(seed)
    amplitude = AMPLITUDE[case["dim"], case["layers"]] * rng.uniform(0.85, 1.25)
    lam = rng.uniform(1.0, 1.2)
    U = synthetic.displacement_field(mesh, mats, amplitude, seed=rng.randrange(1 << 30))
    return mesh, mats, U, lam


def _specs(mats):
    return [dict(c0=float(mats.c0[i]), phi=float(mats.phi[i]), psi=float(mats.psi[i]), young=float(mats.young[i]),
                 poisson=float(mats.poisson[i]), gamma_sat=float(mats.gamma[i]), gamma_unsat=float(mats.gamma[i]))
            for i in range(mats.c0.size)]


def _user_law(mesh, mats, n_q, seed):
    """A caller's stresses and tangents, points first: elastic ones minus a non-associated flow's part
    (D n)(D m)^T / h at a third of the points."""
    dim = mesh.dim
    ns = 6 if dim == 3 else 3
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    mid = torch.as_tensor(np.repeat(mesh.material_id, n_q), device="cuda")
    shear, lame = (torch.as_tensor(np.asarray(v), device="cuda")[mid] for v in (mats.shear, mats.lame))
    D = _elastic(dim, shear, lame)
    n = torch.randn(mid.numel(), 2, ns, dtype=torch.float64, device="cuda", generator=g)
    dn, dm = (torch.einsum("pij,pj->pi", D, n[:, k]) for k in (0, 1))
    h = torch.einsum("pi,pi->p", n[:, 0], dn) + shear
    on = torch.rand(mid.numel(), device="cuda", generator=g) < 1.0 / 3.0
    DS = D - torch.einsum("pi,pj->pij", dn, dm) * (0.4 * on / h)[:, None, None]
    eps = 1e-3 * torch.randn(mid.numel(), ns, dtype=torch.float64, device="cuda", generator=g)
    S = torch.einsum("pij,pj->pi", DS, eps)
    # entry (i, j) of a point's tangent at i + ns * j, the reference's column-major blocks
    return S.contiguous(), DS.transpose(1, 2).reshape(-1, ns * ns).contiguous()


def prepare(case, seed):
    mesh, mats, U, lam = _problem(case, seed)
    specs = _specs(mats)
    if case["task"] == "assemble":
        pattern = prepare_owned_tangent_pattern(mesh.coord, mesh.elem, mesh.q_mask, mesh.material_id, specs, (0, mesh.n_nodes),
                                                elem_type=mesh.elem_type, include_legacy_scatter=False,
                                                include_overlap_B=False, keep_slot_metadata=False)
        S, DS = _user_law(mesh, mats, pattern.n_q, seed)
        return {"task": "assemble", "pattern": pattern, "S": S.T, "DS": DS.T}
    op = ConstitutiveOperator.from_mesh(mesh.coord, mesh.elem, mesh.q_mask, mesh.material_id, specs, elem_type=mesh.elem_type)
    op.tangent_form = case["form"]
    op.host_outputs = bool(case["host"])
    if case["task"] == "bddc":
        op.set_bddc_subdomain_pattern(prepare_bddc_subdomain_pattern(
            mesh.coord, mesh.elem, mesh.q_mask, mesh.material_id, specs, (0, mesh.n_nodes // 2), elem_type=mesh.elem_type,
            overlap_local_int_indices=op.owned_tangent_pattern.local_int_indices, adjacency_source="none"))
        op.reduction(lam)
    return {"task": case["task"], "op": op, "lam": lam, "host": bool(case["host"]),
            "U": U if case["host"] else torch.as_tensor(U, device="cuda")}


def run(state):
    task = state["task"]
    if task == "assemble":
        return {"F": assemble_owned_force_from_local_stress(state["pattern"], state["S"]),
                "K": assemble_owned_tangent_values(state["pattern"], state["DS"])}
    op, U, lam = state["op"], state["U"], state["lam"]
    if task == "newton":
        F, K = op.build_F_K_regularized_all_free(lam, U, R)
        return {"F": F, "K": K.getValuesCSR()[2] if state["host"] else K.values}
    if task == "continuation":
        return {"F": op.build_F_all_free(lam, U), "J": op.potential_energy(U)}
    op.constitutive_problem_stress_tangent(U)
    return {"K": op.build_bddc_regularized_matrix(R).values}


def work(case):
    """Displacements, connectivity, coordinates and materials read; stresses, F and K written."""
    dim, (n_p, n_q, per_dof, flops_el, flops_pl) = case["dim"], KINDS[case["dim"], case["elem"]]
    order = int(case["elem"][1])
    sides = [case["nx"], case["ny"]] + ([case["nz"]] if dim == 3 else [])
    n_el = math.prod(sides) * (2 if dim == 2 else 6)
    n_dof = dim * math.prod(order * s + 1 for s in sides)
    ns, points = (6 if dim == 3 else 3), n_el * n_q
    read = 2 * 8 * n_dof + n_el * (4 * n_p + 8)
    if case["task"] == "continuation":
        return {"bytes": read + 8 * n_dof + 8, "flops": 1.5 * flops_el * n_el + 100 * points}
    if case["task"] == "assemble":
        nld = dim * n_p
        return {"bytes": read + points * 8 * (ns + ns * ns) + 8 * n_dof * (1 + per_dof),
                "flops": 0.5 * flops_el * n_el + points * 2 * dim * (nld * ns + nld * nld)}
    # about an eighth of the points and elements yield
    flops = flops_el * n_el + 60 * points + (600 + flops_pl) * points / 8
    share = 0.5 if case["task"] == "bddc" else 1.0
    return {"bytes": read + 8 * (ns + (dim == 2)) * points + 8 * n_dof * (1 + per_dof) * share, "flops": flops}


# ------------------------------------------------------------------------------ 64-bit values, plain torch


def _elastic(dim, shear, lame):
    ns, nn = (6, 3) if dim == 3 else (3, 2)
    D = torch.zeros(shear.numel(), ns, ns, dtype=torch.float64, device=shear.device)
    D[:, :nn, :nn] = lame[:, None, None]
    for i in range(ns):
        D[:, i, i] += 2.0 * shear if i < nn else shear
    return D


def _reduced(mats, lam):
    """c_bar and sin(phi) of Davis' approach B, per material."""
    phi, psi = np.arctan(np.tan(np.deg2rad(mats.phi)) / lam), np.arctan(np.tan(np.deg2rad(mats.psi)) / lam)
    beta = np.cos(phi) * np.cos(psi) / (1.0 - np.sin(phi) * np.sin(psi))
    phi_r = np.arctan(beta * np.tan(phi))
    return 2.0 * beta * mats.c0 / lam * np.cos(phi_r), np.sin(phi_r)


def _principal_3d(t, I1):
    """Ordered principal values of symmetric tensors t = [11, 22, 33, 12, 23, 13] by invariants."""
    I2 = t[:, 0] * t[:, 1] + t[:, 0] * t[:, 2] + t[:, 1] * t[:, 2] - t[:, 3] ** 2 - t[:, 4] ** 2 - t[:, 5] ** 2
    I3 = (t[:, 0] * t[:, 1] * t[:, 2] - t[:, 2] * t[:, 3] ** 2 - t[:, 1] * t[:, 5] ** 2 - t[:, 0] * t[:, 4] ** 2
          + 2.0 * t[:, 3] * t[:, 4] * t[:, 5])
    Q = torch.clamp((I1 * I1 - 3.0 * I2) / 9.0, min=0.0)
    rad = (-2.0 * I1 ** 3 + 9.0 * I1 * I2 - 27.0 * I3) / 54.0
    safe = torch.where(Q < 1e-30, torch.ones_like(Q), Q)
    theta = torch.where(Q < 1e-30, torch.zeros_like(Q), torch.acos(torch.clamp(rad / safe ** 1.5, -1.0, 1.0)) / 3.0)
    s, third = 2.0 * math.pi / 3.0, I1 / 3.0
    return [-2.0 * Q.sqrt() * torch.cos(theta + a) + third for a in (s, -s, 0.0)]


def _outer(a, b):
    return a[:, :, None] * b[:, None, :]


def _yield_terms(e1, e2, e3, tr, c, s, G, L):
    """Trial yield function and the multipliers, denominators and limits of the plastic branches."""
    f = 2.0 * G * ((1.0 + s) * e1 - (1.0 - s) * e3) + 2.0 * L * s * tr - c
    d = [4.0 * L * s * s + a * G * (1.0 + s) ** 2 + b * G * (1.0 - s) ** 2 for a, b in ((2.0, 2.0), (1.0, 2.0), (2.0, 1.0))]
    lin = 2.0 * L * s * tr - c
    left = (G * ((1.0 + s) * (e1 + e2) - 2.0 * (1.0 - s) * e3) + lin) / d[1]
    right = (G * (2.0 * (1.0 + s) * e1 - (1.0 - s) * (e2 + e3)) + lin) / d[2]
    g_sl, g_sr = (e1 - e2) / (1.0 + s), (e2 - e3) / (1.0 - s)
    lam = [f / d[0], left, right]
    smooth = (f > 0) & (lam[0] <= torch.minimum(g_sl, g_sr))
    is_l = (f > 0) & ~smooth & (g_sl < g_sr) & (left >= g_sl) & (left <= (e1 + e2 - 2.0 * e3) / (3.0 - s))
    is_r = (f > 0) & ~smooth & ~is_l & (g_sl > g_sr) & (right >= g_sr) & (right <= (2.0 * e1 - e2 - e3) / (3.0 + s))
    return f, lam, d, [smooth, is_l, is_r, (f > 0) & ~smooth & ~is_l & ~is_r]


def _return_3d(E, c, s, G, L):
    """Stress (n, 6) and consistent tangent (n, 6, 6)."""
    dev = E.device
    half = torch.tensor([1.0, 1.0, 1.0, 0.5, 0.5, 0.5], dtype=torch.float64, device=dev)
    iota = torch.tensor([1.0, 1.0, 1.0, 0.0, 0.0, 0.0], dtype=torch.float64, device=dev)
    t = E * half
    I1 = t[:, 0] + t[:, 1] + t[:, 2]
    e = _principal_3d(t, I1)
    DS = _elastic(3, G, L)
    S = torch.einsum("pij,pj->pi", DS, E)
    f, lam, den, masks = _yield_terms(*e, I1, c, s, G, L)
    eye, vol = torch.diag(half), torch.outer(iota, iota)
    for kind, mask in enumerate(masks):
        i = torch.nonzero(mask).reshape(-1)
        if i.numel() == 0:
            continue
        T, c_, s_, G_, L_, tr = t[i], c[i], s[i], G[i], L[i], I1[i]
        if kind == 3:
            S[i] = (c_ / (2.0 * s_))[:, None] * iota
            DS[i] = 0.0
            continue
        x = [v[i] for v in e]
        l_, d_ = lam[kind][i], den[kind][i]
        sq = torch.stack([T[:, 0] ** 2 + T[:, 3] ** 2 + T[:, 5] ** 2, T[:, 1] ** 2 + T[:, 3] ** 2 + T[:, 4] ** 2,
                          T[:, 2] ** 2 + T[:, 4] ** 2 + T[:, 5] ** 2,
                          T[:, 0] * T[:, 3] + T[:, 1] * T[:, 3] + T[:, 4] * T[:, 5],
                          T[:, 3] * T[:, 5] + T[:, 1] * T[:, 4] + T[:, 2] * T[:, 4],
                          T[:, 0] * T[:, 5] + T[:, 3] * T[:, 4] + T[:, 2] * T[:, 5]], 1)
        jac = torch.zeros(i.numel(), 6, 6, dtype=torch.float64, device=dev)  # d(t t)/dE
        for a in range(3):
            jac[:, a, a] = 2.0 * T[:, a]
        for a, b, k in ((0, 3, 3), (0, 5, 5), (1, 3, 3), (1, 4, 4), (2, 4, 4), (2, 5, 5)):
            jac[:, a, b] = jac[:, b, a] = T[:, k]
        for a, (m, n) in ((3, (0, 1)), (4, (1, 2)), (5, (0, 2))):
            jac[:, a, a] = 0.5 * (T[:, m] + T[:, n])
        for a, b, k in ((3, 4, 5), (3, 5, 4), (4, 5, 3)):
            jac[:, a, b] = jac[:, b, a] = 0.5 * T[:, k]

        def proj(k):  # eigenprojection of value k and 1 / ((x_k - x_l)(x_k - x_m))
            o = [x[m] for m in range(3) if m != k]
            inv = 1.0 / ((x[k] - o[0]) * (x[k] - o[1]))
            P = inv[:, None] * (sq - (o[0] + o[1])[:, None] * T + (o[0] * o[1])[:, None] * iota)
            return P, inv

        col = lambda v: v[:, None, None]  # noqa: E731
        if kind == 0:
            P, inv = zip(*(proj(k) for k in range(3)))
            p1, m1 = 2.0 * G_ * (1.0 + s_), 2.0 * G_ * (1.0 - s_)
            sv = [L_ * tr + 2.0 * G_ * x[0] - l_ * (2.0 * L_ * s_ + p1), L_ * tr + 2.0 * G_ * x[1] - l_ * 2.0 * L_ * s_,
                  L_ * tr + 2.0 * G_ * x[2] - l_ * (2.0 * L_ * s_ - m1)]
            O = [_outer(P[k], P[k]) for k in range(3)]  # noqa: E741
            ds = col(L_) * vol + col(2.0 * G_) * (O[0] + O[1] + O[2])
            for k in range(3):
                a, b = [m for m in range(3) if m != k]
                dP = col(inv[k]) * (jac - col(x[a] + x[b]) * eye - col(2.0 * x[k] - x[a] - x[b]) * O[k]
                                    - col(x[a] - x[b]) * (O[a] - O[b]))
                ds = ds + col(sv[k]) * dP
            S[i] = sum(sv[k][:, None] * P[k] for k in range(3))
            Dp = p1[:, None] * P[0] - m1[:, None] * P[2] + (2.0 * L_ * s_)[:, None] * iota
        else:
            one = 2 if kind == 1 else 0  # the single value: the smallest (left edge) or the largest (right edge)
            Rp, inv = proj(one)
            Q = iota - Rp
            a, b = [m for m in range(3) if m != one]
            em, xo = x[a] + x[b], x[one]
            if kind == 1:
                sq_, so = (L_ * tr + G_ * em - l_ * (2.0 * L_ * s_ + G_ * (1.0 + s_)),
                           L_ * tr + 2.0 * G_ * xo - l_ * (2.0 * L_ * s_ - 2.0 * G_ * (1.0 - s_)))
                wq, wo = G_ * (1.0 + s_), -2.0 * G_ * (1.0 - s_)
            else:
                sq_, so = (L_ * tr + G_ * em - l_ * (2.0 * L_ * s_ - G_ * (1.0 - s_)),
                           L_ * tr + 2.0 * G_ * xo - l_ * (2.0 * L_ * s_ + 2.0 * G_ * (1.0 + s_)))
                wq, wo = -G_ * (1.0 - s_), 2.0 * G_ * (1.0 + s_)
            S[i] = sq_[:, None] * Q + so[:, None] * Rp
            QT, QR, QQ, RR = _outer(Q, T), _outer(Q, Rp), _outer(Q, Q), _outer(Rp, Rp)
            dP = col(inv) * (jac - col(em) * eye - (QT + QT.transpose(1, 2)) + col(em) * QQ + col(em - 2.0 * xo) * RR
                             + col(xo) * (QR + QR.transpose(1, 2)))
            ds = col(so - sq_) * dP + col(L_) * vol + col(G_) * (QQ + 2.0 * RR)
            Dp = wq[:, None] * Q + wo[:, None] * Rp + (2.0 * L_ * s_)[:, None] * iota
        DS[i] = ds - _outer(Dp, Dp) / col(d_)
    return S, DS


def _return_2d(E, c, s, G, L):
    """In-plane stress (n, 3) and tangent (n, 3, 3) of plane strain."""
    dev, n = E.device, E.shape[0]
    tr2 = E[:, 0] + E[:, 1]
    rad = torch.sqrt((E[:, 0] - E[:, 1]) ** 2 + E[:, 2] ** 2)
    zero = torch.zeros_like(rad)
    vals = torch.stack([0.5 * (tr2 + rad), 0.5 * (tr2 - rad), zero], 1)
    order = torch.tensor([0, 1, 2], device=dev).repeat(n, 1)
    straddle = (vals[:, 0] >= 0) & (vals[:, 1] < 0)
    order[straddle] = torch.tensor([0, 2, 1], device=dev)
    order[vals[:, 0] < 0] = torch.tensor([2, 0, 1], device=dev)
    e = [vals.gather(1, order[:, k:k + 1])[:, 0] for k in range(3)]
    tr = e[0] + e[1] + e[2]
    iota = torch.tensor([1.0, 1.0, 0.0], dtype=torch.float64, device=dev)
    eye = torch.diag(torch.tensor([1.0, 1.0, 0.5], dtype=torch.float64, device=dev))
    DS = _elastic(2, G, L)
    S = torch.einsum("pij,pj->pi", DS, E)
    f, lam, den, masks = _yield_terms(*e, tr, c, s, G, L)
    r = torch.where(rad == 0, torch.ones_like(rad), rad)[:, None]
    P0 = torch.where(rad[:, None] == 0, iota, torch.stack([E[:, 0] - vals[:, 1], E[:, 1] - vals[:, 1], 0.5 * E[:, 2]], 1) / r)
    P1 = iota - P0
    dP0 = torch.where(rad[:, None, None] == 0, zero[:, None, None], (eye - _outer(P0, P0) - _outer(P1, P1)) / r[:, :, None])
    P_all = torch.stack([P0, P1, torch.zeros_like(P0)], 1)
    dP_all = torch.stack([dP0, -dP0, torch.zeros_like(dP0)], 1)
    at = torch.arange(n, device=dev)
    P = [P_all[at, order[:, k]] for k in range(3)]
    dP = [dP_all[at, order[:, k]] for k in range(3)]
    col = lambda v: v[:, None, None]  # noqa: E731
    vol = col(L) * torch.outer(iota, iota)
    for kind, mask in enumerate(masks):
        m2 = mask[:, None]
        if kind == 3:
            S = torch.where(m2, (c / (2.0 * s))[:, None] * iota, S)
            DS = torch.where(col(mask), torch.zeros_like(DS), DS)
            continue
        l_, d_ = lam[kind], den[kind]
        if kind == 0:
            parts, w = [(P[k], dP[k], 2.0 * G) for k in range(3)], [2.0 * G * (1.0 + s), zero, -2.0 * G * (1.0 - s)]
            base = [2.0 * G * e[k] for k in range(3)]
        elif kind == 1:
            parts, w = [(P[0] + P[1], dP[0] + dP[1], G), (P[2], dP[2], 2.0 * G)], [G * (1.0 + s), -2.0 * G * (1.0 - s)]
            base = [G * (e[0] + e[1]), 2.0 * G * e[2]]
        else:
            parts, w = [(P[0], dP[0], 2.0 * G), (P[1] + P[2], dP[1] + dP[2], G)], [2.0 * G * (1.0 + s), -G * (1.0 - s)]
            base = [2.0 * G * e[0], G * (e[1] + e[2])]
        sv = [L * tr + b - l_ * (2.0 * L * s + a) for a, b in zip(w, base)]
        s_new = sum(v[:, None] * p for v, (p, _d, _g) in zip(sv, parts))
        q6 = sum(a[:, None] * p for a, (p, _d, _g) in zip(w, parts)) + (2.0 * L * s)[:, None] * iota
        ds = vol + sum(col(v) * dp + col(g) * _outer(p, p) for v, (p, dp, g) in zip(sv, parts)) - _outer(q6, q6) / col(d_)
        S, DS = torch.where(m2, s_new, S), torch.where(col(mask), ds, DS)
    return S, DS


def _energy(dim, E, c, s, G, K, L):
    """The potential energy density as the reference computes it: its 3D invariants take the engineering
    shears of rows 3..5 as the entries (12), (13), (23), and its sorted 2D triple drops the values that
    change place."""
    if dim == 3:
        t = E[:, [0, 1, 2, 3, 5, 4]]
        tr = E[:, 0] + E[:, 1] + E[:, 2]
        e = _principal_3d(t, tr)
    else:
        tr2, rad = E[:, 0] + E[:, 1], torch.sqrt((E[:, 0] - E[:, 1]) ** 2 + E[:, 2] ** 2)
        a, b, zero = (tr2 + rad) / 2.0, (tr2 - rad) / 2.0, torch.zeros_like(rad)
        e = [torch.where(a < 0, zero, a), torch.where(b < 0, zero, b), zero]
        tr = e[0] + e[1] + e[2]
    f, lam, d, masks = _yield_terms(*e, tr, c, s, G, L)
    vol, el = 0.5 * L * tr * tr, G * (e[0] ** 2 + e[1] ** 2 + e[2] ** 2)
    psi = vol + el
    psi = torch.where(masks[0], psi - 0.5 * d[0] * lam[0] ** 2, psi)
    psi = torch.where(masks[1], vol + G * (e[2] ** 2 + 0.5 * (e[0] + e[1]) ** 2) - 0.5 * d[1] * lam[1] ** 2, psi)
    psi = torch.where(masks[2], vol + G * (e[0] ** 2 + 0.5 * (e[1] + e[2]) ** 2) - 0.5 * d[2] * lam[2] ** 2, psi)
    d_a = 4.0 * K * s * s
    apex = 0.5 * K * tr * tr - 0.5 * d_a * ((2.0 * K * s * tr - c) / d_a) ** 2
    return torch.where(masks[3], apex, psi)


class _Sums:
    """Force and CSR values of a mesh, element by element: rows of every dof, columns of the free ones,
    a constrained row its diagonal alone."""

    def __init__(self, mesh):
        self.dim = mesh.dim
        self.elem = torch.as_tensor(mesh.elem.T.copy(), device="cuda")  # (n_elem, n_p)
        self.free = torch.as_tensor(mesh.q_mask.T.reshape(-1).copy(), device="cuda")  # dof = dim * node + component
        self.coord = torch.as_tensor(mesh.coord, device="cuda")
        xi, wf = quadrature(mesh.dim, mesh.elem_type)
        self.wf = torch.as_tensor(np.asarray(wf, dtype=np.float64), device="cuda")
        self.dhat = torch.as_tensor(np.ascontiguousarray(reference_gradients(mesh.dim, mesh.elem_type)), device="cuda")
        self.n_q, self.n_dof = xi.shape[1], mesh.dim * mesh.coord.shape[1]
        self.chunk = max(1, 200000 // (self.n_q * mesh.elem.shape[0] // 10 + 1))

    def chunks(self):
        """(first element, dofs (n, n_ld), strain operators (n, n_q, ns, n_ld), weights (n, n_q))"""
        dim, ns = self.dim, (6 if self.dim == 3 else 3)
        for e0 in range(0, self.elem.shape[0], self.chunk):
            el = self.elem[e0:e0 + self.chunk]
            J = torch.einsum("den,rnq->eqrd", self.coord[:, el], self.dhat)  # dx_d / dxi_r
            grad = torch.einsum("eqdr,rnq->eqdn", torch.linalg.inv(J), self.dhat)
            B = torch.zeros(el.shape[0], self.n_q, ns, el.shape[1], dim, dtype=torch.float64, device="cuda")
            for k in range(dim):
                B[:, :, k, :, k] = grad[:, :, k]
            for row, (a, b) in zip(range(dim, ns), ((0, 1), (1, 2), (0, 2))):
                B[:, :, row, :, a] = grad[:, :, b]
                B[:, :, row, :, b] = grad[:, :, a]
            dofs = (dim * el[:, :, None] + torch.arange(dim, device="cuda")).reshape(el.shape[0], -1)
            yield e0, dofs, B.reshape(*B.shape[:3], -1), torch.linalg.det(J).abs() * self.wf

    def keys(self, dofs):
        ok = self.free[dofs][:, :, None] & self.free[dofs][:, None, :]
        return dofs[:, :, None] * self.n_dof + dofs[:, None, :], ok

    def pattern(self):
        fixed = torch.nonzero(~self.free).reshape(-1) * (self.n_dof + 1)
        parts = [fixed]
        for e0 in range(0, self.elem.shape[0], self.chunk):
            el = self.elem[e0:e0 + self.chunk]
            key, ok = self.keys((self.dim * el[:, :, None] + torch.arange(self.dim, device="cuda")).reshape(el.shape[0], -1))
            parts.append(torch.unique(key[ok]))
        self.where = torch.unique(torch.cat(parts))
        self.fixed = torch.searchsorted(self.where, fixed)
        return torch.zeros(self.where.numel(), dtype=torch.float64, device="cuda")

    def add(self, values, dofs, B, w, D):
        ns = B.shape[2]
        DB = torch.matmul(D.reshape(*w.shape, ns, ns) * w[:, :, None, None], B)
        Ke = torch.bmm(B.flatten(1, 2).transpose(1, 2), DB.flatten(1, 2))
        key, ok = self.keys(dofs)
        values.index_add_(0, torch.searchsorted(self.where, key[ok]), Ke[ok])


def _submesh(mesh):
    """The elements whose smallest node is in the lower half of the nodes, as a mesh of their own."""
    own = np.flatnonzero(mesh.elem.min(axis=0) < mesh.n_nodes // 2)
    nodes = np.unique(mesh.elem[:, own])
    lid = np.full(mesh.n_nodes, -1, dtype=np.int64)
    lid[nodes] = np.arange(nodes.size)
    return synthetic.SlopeMesh(mesh.dim, mesh.elem_type, np.ascontiguousarray(mesh.coord[:, nodes]), lid[mesh.elem[:, own]],
                               np.ascontiguousarray(mesh.q_mask[:, nodes]), mesh.material_id[own]), nodes


def exact(case, seed):
    mesh, mats, U, lam = _problem(case, seed)
    task, dim = case["task"], case["dim"]
    ns = 6 if dim == 3 else 3
    if task == "assemble":
        S_user, DS_user = _user_law(mesh, mats, quadrature(dim, mesh.elem_type)[0].shape[1], seed)
    if task == "bddc":
        mesh, nodes = _submesh(mesh)
        U = U[:, nodes]
    sums = _Sums(mesh)
    c_bar, sin_phi = _reduced(mats, lam)
    per_material = [torch.as_tensor(np.asarray(v), device="cuda") for v in (c_bar, sin_phi, mats.shear, mats.bulk, mats.lame)]
    mid = torch.as_tensor(mesh.material_id, device="cuda")
    u = torch.as_tensor(U.T.reshape(-1).copy(), device="cuda")
    F = torch.zeros(sums.n_dof, dtype=torch.float64, device="cuda")
    K = None if task == "continuation" else sums.pattern()
    energy = 0.0
    for e0, dofs, B, w in sums.chunks():
        pts = slice(e0 * sums.n_q, (e0 + dofs.shape[0]) * sums.n_q)
        c, s, G, bulk, L = (v[mid[e0:e0 + dofs.shape[0]]].repeat_interleave(sums.n_q) for v in per_material)
        E = torch.einsum("eqsl,el->eqs", B, u[dofs]).reshape(-1, ns)
        if task == "assemble":
            S, DS = S_user[pts], DS_user[pts].reshape(-1, ns, ns).transpose(1, 2)
        else:
            S, DS = (_return_3d if dim == 3 else _return_2d)(E, c, s, G, L)
        F.index_add_(0, dofs.reshape(-1), torch.einsum("eqsl,eqs->el", B, S.reshape(*w.shape, ns) * w[:, :, None]).reshape(-1))
        if task == "continuation":
            energy += float((_energy(dim, E, c, s, G, bulk, L) * w.reshape(-1)).sum())
        elif task == "assemble":
            sums.add(K, dofs, B, w, DS)
        else:
            sums.add(K, dofs, B, w, (1.0 - R) * DS + R * _elastic(dim, G, L))
    if K is not None:
        K[sums.fixed] = 1.0
    if task == "bddc":
        return {"K": K}
    if task == "continuation":
        return {"F": F[sums.free], "J": energy}
    return {"F": F[sums.free] if task == "newton" else F * sums.free, "K": K}
