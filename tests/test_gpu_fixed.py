"""The fixed-point kernels of the plain form (csrc/fixed.cuh) against the oracle, at the sizes and
magnitudes where they can go wrong.

Tolerance: 1e-13 of the largest value.  The fixed-point sums are within 2^-53 of it; the oracle's FP64
sums of some hundred terms, of either sign and up to an order above the result, are within about
100 x 10 x 2^-53 = 1e-13 of theirs."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-13


@pytest.fixture(autouse=True)
def _clean_status(cuda_device):
    from slope_stability_petsc4py_gb300 import _lib

    _lib.device_status(clear=True)
    yield
    assert _lib.device_status(clear=True) == 0


def _pattern(et, dims, dim=3):
    from slope_stability_petsc4py_gb300 import ConstitutiveOperator, synthetic

    mats = synthetic.MaterialSet.layered(4, seed=1)
    mesh = (synthetic.slope_mesh_3d(*dims, elem_type=et, n_layers=4) if dim == 3 else
            synthetic.slope_mesh_2d(*dims, elem_type=et, n_layers=4))
    specs = [dict(c0=float(mats.c0[i]), phi=float(mats.phi[i]), psi=float(mats.psi[i]), young=float(mats.young[i]),
                  poisson=float(mats.poisson[i]), gamma_sat=20.0, gamma_unsat=20.0) for i in range(mats.c0.size)]
    op = ConstitutiveOperator.from_mesh(mesh.coord, mesh.elem, mesh.q_mask, mesh.material_id, specs, elem_type=et)
    return op, op.owned_tangent_pattern


def _plastic_state(op, pat, n_plastic, magnitude, seed):
    """Branch codes with n_plastic points in every element but the first (which has none), moduli and
    symmetric tangents of the given magnitude that differ from the elastic ones at those points."""
    rng = np.random.default_rng(seed)
    n_el, n_q, ns = int(pat.overlap_elements.size), pat.n_q, pat.n_strain
    branch = np.zeros((n_el, n_q), dtype=np.int8)
    for e in range(1, n_el):
        branch[e, rng.choice(n_q, n_plastic, replace=False)] = rng.integers(1, 5, n_plastic)
    idx = pat.local_int_indices
    shear, lame = magnitude * op.shear[idx], magnitude * op.lame[idx]
    nn = 3 if pat.dim == 3 else 2
    D = np.zeros((n_el * n_q, ns, ns))
    D[:, :nn, :nn] = lame[:, None, None]
    for i in range(ns):
        D[:, i, i] += 2.0 * shear if i < nn else shear
    A = rng.standard_normal(D.shape)
    dD = (A + A.transpose(0, 2, 1)) * (shear * 10.0 ** rng.uniform(-3.0, 0.3, shear.size))[:, None, None]
    dD[branch.reshape(-1) == 0] = 0.0
    return branch.reshape(-1), shear, lame, D + dD, dD


@pytest.mark.parametrize("n_plastic,magnitude", [(1, 1.0), (2, 1e-150), (4, 1e150), (5, 1.0), (8, 1e-9), (11, 1e6)])
def test_p2_moment_correction(oracle, n_plastic, magnitude):
    import torch

    from slope_stability_petsc4py_gb300 import _lib
    from slope_stability_petsc4py_gb300.distributed_tangent import _p2_affine_inputs

    op, pat = _pattern("P2", (5, 2, 3))
    d = _p2_affine_inputs(pat)
    branch, shear, lame, DS, dD = _plastic_state(op, pat, n_plastic, magnitude, n_plastic)
    n_el, scale = int(pat.overlap_elements.size), 0.7
    rows = np.ascontiguousarray(DS.transpose(0, 2, 1).reshape(-1, 36))
    dev = {k: torch.as_tensor(v, device="cuda") for k, v in dict(branch=branch, shear=shear, lame=lame, ds=rows).items()}

    def run(ds):
        vals = torch.zeros(pat.nnz, dtype=torch.float64, device="cuda")
        elist = torch.arange(n_el, dtype=torch.int32, device="cuda")
        count = torch.tensor([n_el], dtype=torch.int32, device="cuda")
        _lib.call("ssp_tangent_plastic_correction_p2_moments", _lib.ptr(d["jinv"]), _lib.ptr(d["bary"]), _lib.ptr(ds),
                  _lib.ptr(d["weight"]), _lib.ptr(dev["branch"]), _lib.ptr(dev["shear"]), _lib.ptr(dev["lame"]),
                  _lib.ptr(d["scatter_map"]), n_el, pat.n_q, pat.nnz, scale, _lib.ptr(vals), _lib.ptr(elist),
                  _lib.ptr(count), _lib.stream_handle())
        return vals.cpu().numpy()

    want = oracle.tangent_scatter(3, pat.dphi1, pat.dphi2, pat.dphi3,
                                  np.ascontiguousarray(scale * dD.transpose(0, 2, 1).reshape(-1, 36)),
                                  pat.overlap_assembly_weight, d["scatter_map"].cpu().numpy(), pat.n_q, pat.nnz)
    got = run(dev["ds"])
    assert rel_err(got, want) <= TOL
    # an infinity and a nan stay in their element, in the entries the contraction takes them to
    bad = int(np.flatnonzero(branch)[0])
    ds = dev["ds"].clone()
    ds[bad, 0] = float("inf")
    ds[bad, 21] = float("nan")  # (3, 3)
    out = run(ds)
    smap = d["scatter_map"].cpu().numpy()[bad // pat.n_q]
    assert not np.isfinite(out[smap[smap >= 0]]).all() and np.isnan(out).any()
    others = np.ones(pat.nnz, dtype=bool)
    others[smap[smap >= 0]] = False
    assert np.array_equal(out[others], got[others]) or rel_err(out[others], got[others]) <= TOL


@pytest.mark.parametrize("dims,magnitude,n_q", [((5, 2, 3), 1.0, 11), ((4, 3, 1), 1e-140, 11), ((7, 1, 1), 1e140, 11),
                                                ((4, 2, 2), 1.0, 1), ((4, 2, 2), 1.0, 2), ((4, 2, 2), 1e5, 31), ((4, 2, 2), 1.0, 64)])
def test_p2_strain_and_force(oracle, dims, magnitude, n_q):
    """Element counts that are no multiple of a warp, other point counts (staged and not), magnitudes near
    the ends of FP64's range, and inputs that are not finite."""
    import torch

    from slope_stability_petsc4py_gb300 import _lib
    from slope_stability_petsc4py_gb300.distributed_tangent import _p2_affine_inputs

    op, pat = _pattern("P2", dims)
    d = _p2_affine_inputs(pat)
    rng = np.random.default_rng(n_q)
    n_el = int(pat.overlap_elements.size)
    lam = rng.dirichlet(np.ones(4), n_q) if n_q != 11 else d["bary"].cpu().numpy()
    jinv = d["jinv"].cpu().numpy().reshape(n_el, 3, 3)
    gl = np.concatenate([-jinv.sum(axis=1, keepdims=True), jinv], axis=1)  # (n_el, 4, 3)
    g = np.empty((n_el, n_q, 10, 3))
    for a in range(4):
        g[:, :, a] = (4.0 * lam[None, :, a, None] - 1.0) * gl[:, None, a]
    for a, (i, j) in zip(range(4, 10), ((0, 1), (1, 2), (0, 2), (1, 3), (2, 3), (0, 3))):
        g[:, :, a] = 4.0 * (lam[None, :, i, None] * gl[:, None, j] + lam[None, :, j, None] * gl[:, None, i])
    dphi = [np.ascontiguousarray(g[..., z].reshape(-1, 10)) for z in range(3)]
    u = magnitude * rng.standard_normal(int(pat.overlap_global_dofs.size)) * 10.0 ** rng.uniform(-3.0, 0.0)
    dof = pat.overlap_element_dof_lids
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    bary = dev(lam)

    def strain(u):
        E = torch.full((n_el * n_q, 6), -7.0, dtype=torch.float64, device="cuda")
        ud = dev(u)
        _lib.call("ssp_assemble_overlap_strain_3d_p2_affine", _lib.ptr(d["jinv"]), _lib.ptr(bary), _lib.ptr(ud), u.size,
                  _lib.ptr(d["dof_lids"]), n_el * n_q, n_el, n_q, _lib.ptr(E), _lib.stream_handle())
        return E.cpu().numpy()

    E = strain(u)
    assert rel_err(E, oracle.strain_3d(*dphi, u, dof, n_q)) <= TOL
    S = magnitude * rng.standard_normal((n_el * n_q, 6)) * 10.0 ** rng.uniform(-2.0, 0.0, (n_el * n_q, 1))
    w = rng.uniform(-0.2, 1.0, n_el * n_q)
    rows = d["elem_row"].cpu().numpy()
    n_rows = int(pat.local_matrix_pattern.shape[0])

    def force(S):
        F = torch.full((n_rows,), -7.0, dtype=torch.float64, device="cuda")
        Sd, wd = dev(S), dev(w)
        _lib.call("ssp_assemble_force_element_p2_affine", _lib.ptr(d["jinv"]), _lib.ptr(bary), _lib.ptr(Sd), _lib.ptr(wd),
                  _lib.ptr(d["elem_row"]), n_el, n_q, n_rows, _lib.ptr(F), _lib.stream_handle())
        return F.cpu().numpy()

    bt = ((0, 3, 5), (3, 1, 4), (5, 4, 2))
    want = np.zeros(n_rows)
    ws = (w[:, None] * S).reshape(n_el, n_q, 6)
    for c in range(3):
        f = sum(np.einsum("eqa,eq->ea", g[..., z], ws[..., bt[c][z]]) for z in range(3))
        r = rows.reshape(n_el, 10, 3)[:, :, c]
        np.add.at(want, r[r >= 0], f[r >= 0])
    F = force(S)
    assert rel_err(F, want) <= TOL
    # not finite: the elements of one dof, the rows of one element
    u2 = u.copy()
    u2[dof[0, 4]] = float("nan")
    hit = (dof == dof[0, 4]).any(axis=1).repeat(n_q)
    E2 = strain(u2)
    assert np.isnan(E2[hit]).any() and np.array_equal(E2[~hit], E[~hit])
    S2 = S.copy()
    S2[0, 1] = float("inf")
    F2 = force(S2)
    touched = np.zeros(n_rows, dtype=bool)
    touched[rows[0][rows[0] >= 0]] = True
    assert not np.isfinite(F2[touched]).all() and rel_err(F2[~touched], F[~touched]) <= TOL


@pytest.mark.parametrize("et,dims,kind,n_plastic,magnitude", [
    ("P2", (4, 2, 2), "full", 0, 1.0), ("P2", (4, 2, 2), "symmetric", 0, 1e-150), ("P2", (4, 2, 2), "correction", 1, 1.0),
    ("P2", (4, 2, 2), "correction", 11, 1e150), ("P4", (2, 1, 1), "full", 0, 1e6), ("P4", (2, 1, 1), "symmetric", 0, 1.0),
    ("P4", (2, 2, 1), "correction", 1, 1e-9), ("P4", (2, 2, 1), "correction", 12, 1.0), ("P4", (2, 2, 1), "correction", 13, 1.0), ("P4", (2, 1, 1), "correction", 24, 1.0)])
def test_element_tangents(oracle, et, dims, kind, n_plastic, magnitude):
    import torch

    from slope_stability_petsc4py_gb300 import _lib

    op, pat = _pattern(et, dims)
    d, n_el, scale = pat.device, int(pat.overlap_elements.size), 0.7
    branch, shear, lame, DS, dD = _plastic_state(op, pat, n_plastic, magnitude, n_plastic)
    if kind == "full":
        rng = np.random.default_rng(1)
        DS = DS + 0.5 * shear[:, None, None] * rng.standard_normal(DS.shape)
    dev = {k: torch.as_tensor(np.ascontiguousarray(v), device="cuda") for k, v in dict(
        branch=branch, shear=shear, lame=lame, ds=DS.transpose(0, 2, 1).reshape(-1, 36)).items()}
    geo = [_lib.ptr(d[k]) for k in ("dphi1", "dphi2", "dphi3")]

    def run(ds):
        vals = torch.zeros(pat.nnz, dtype=torch.float64, device="cuda")
        if kind == "correction":
            elist = torch.arange(n_el, dtype=torch.int32, device="cuda")
            count = torch.tensor([n_el], dtype=torch.int32, device="cuda")
            _lib.call("ssp_tangent_plastic_correction", 3, *geo, _lib.ptr(ds), _lib.ptr(d["weight"]), _lib.ptr(dev["branch"]),
                      _lib.ptr(dev["shear"]), _lib.ptr(dev["lame"]), _lib.ptr(d["scatter_map"]), n_el, pat.n_p, pat.n_q,
                      pat.nnz, scale, _lib.ptr(vals), _lib.ptr(elist), _lib.ptr(count), _lib.stream_handle())
        else:
            _lib.call("ssp_tangent_element", 3, int(kind == "symmetric"), *geo, _lib.ptr(ds), _lib.ptr(d["weight"]),
                      _lib.ptr(d["scatter_map"]), n_el, pat.n_p, pat.n_q, pat.nnz, _lib.ptr(vals), 0, _lib.stream_handle())
        return vals.cpu().numpy()

    rows = scale * dD if kind == "correction" else DS
    smap = d["scatter_map"].cpu().numpy()
    want = oracle.tangent_scatter(3, pat.dphi1, pat.dphi2, pat.dphi3, np.ascontiguousarray(rows.transpose(0, 2, 1).reshape(-1, 36)),
                                  pat.overlap_assembly_weight, smap, pat.n_q, pat.nnz)
    got = run(dev["ds"])
    assert rel_err(got, want) <= TOL
    bad = int(np.flatnonzero(branch)[0]) if n_plastic else 3
    ds = dev["ds"].clone()
    ds[bad, 0] = float("inf")
    ds[bad, 21] = float("nan")
    out = run(ds)
    mine = smap[bad // pat.n_q]
    others = np.ones(pat.nnz, dtype=bool)
    others[mine[mine >= 0]] = False
    assert np.isnan(out[mine[mine >= 0]]).any() and rel_err(out[others], got[others]) <= TOL


@pytest.mark.parametrize("et,dims,magnitude", [("P4", (2, 2, 2), 1.0), ("P4", (3, 1, 1), 1e-140), ("P4", (1, 1, 1), 1e140),
                                               ("P2", (4, 2, 3), 1.0)])
def test_affine_strain_and_force(oracle, et, dims, magnitude):
    """The table form (P4's; P2 takes it here for another shape): whole and partly filled groups of elements."""
    import torch

    from slope_stability_petsc4py_gb300 import _lib
    from slope_stability_petsc4py_gb300.fem import reference_gradients

    op, pat = _pattern(et, dims)
    d, n_el, n_q, n_p = pat.device, int(pat.overlap_elements.size), pat.n_q, pat.n_p
    rng = np.random.default_rng(n_el)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    ghat = dev(np.transpose(reference_gradients(3, et), (2, 1, 0)))
    dof = pat.overlap_element_dof_lids
    u = magnitude * (3.0 + rng.standard_normal(int(pat.overlap_global_dofs.size)))
    dphi = [pat.dphi1, pat.dphi2, pat.dphi3]

    def strain(u):
        E, ud = torch.full((n_el * n_q, 6), -7.0, dtype=torch.float64, device="cuda"), dev(u)
        _lib.call("ssp_assemble_overlap_strain_3d_affine", _lib.ptr(d["jinv"]), _lib.ptr(ghat), _lib.ptr(ud), u.size,
                  _lib.ptr(d["dof_lids"]), n_el * n_q, n_el, n_p, n_q, _lib.ptr(E), _lib.stream_handle())
        return E.cpu().numpy()

    E = strain(u)
    assert rel_err(E, oracle.strain_3d(*dphi, u, dof, n_q)) <= TOL
    S = magnitude * rng.standard_normal((n_el * n_q, 6)) * 10.0 ** rng.uniform(-2.0, 0.0, (n_el * n_q, 1))
    rows = d["elem_row"].cpu().numpy()
    n_rows = int(pat.local_matrix_pattern.shape[0])

    def force(S):
        F, Sd = torch.full((n_rows,), -7.0, dtype=torch.float64, device="cuda"), dev(S)
        _lib.call("ssp_assemble_force_element_affine", _lib.ptr(d["jinv"]), _lib.ptr(ghat), _lib.ptr(Sd),
                  _lib.ptr(d["weight"]), _lib.ptr(d["elem_row"]), n_el, n_p, n_q, n_rows, _lib.ptr(F), _lib.stream_handle())
        return F.cpu().numpy()

    bt = ((0, 3, 5), (3, 1, 4), (5, 4, 2))
    want = np.zeros(n_rows)
    ws = (pat.overlap_assembly_weight[:, None] * S).reshape(n_el, n_q, 6)
    for c in range(3):
        f = sum(np.einsum("eqa,eq->ea", dphi[z].reshape(n_el, n_q, n_p), ws[..., bt[c][z]]) for z in range(3))
        r = rows.reshape(n_el, n_p, 3)[:, :, c]
        np.add.at(want, r[r >= 0], f[r >= 0])
    F = force(S)
    assert rel_err(F, want) <= TOL
    u2, S2 = u.copy(), S.copy()
    u2[dof[0, 4]] = float("nan")
    S2[0, 1] = float("inf")
    hit = (dof == dof[0, 4]).any(axis=1).repeat(n_q)
    E2, F2 = strain(u2), force(S2)
    touched = np.zeros(n_rows, dtype=bool)
    touched[rows[0][rows[0] >= 0]] = True
    assert np.isnan(E2[hit]).any() and np.array_equal(E2[~hit], E[~hit])
    assert not np.isfinite(F2[touched]).all() and rel_err(F2[~touched], F[~touched]) <= TOL
