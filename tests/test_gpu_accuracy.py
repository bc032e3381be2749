"""Distance of whole results from sums in extended precision (80 or 128 bits, as the machine has them)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble
BT = ((0, 3, 5), (3, 1, 4), (5, 4, 2))  # strain row of component c's gradient entry z


def _distance(got, want) -> float:
    d = np.asarray(got).astype(LD) - want
    return float(np.sqrt((d * d).sum() / (want * want).sum()))


def _slope(et, dims):
    from slope_stability_petsc4py_gb300 import ConstitutiveOperator, synthetic

    mats = synthetic.MaterialSet.layered(4, seed=1)
    mesh = synthetic.slope_mesh_3d(*dims, elem_type=et, n_layers=4)
    specs = [dict(c0=float(mats.c0[i]), phi=float(mats.phi[i]), psi=float(mats.psi[i]), young=float(mats.young[i]),
                  poisson=float(mats.poisson[i]), gamma_sat=20.0, gamma_unsat=20.0) for i in range(mats.c0.size)]
    op = ConstitutiveOperator.from_mesh(mesh.coord, mesh.elem, mesh.q_mask, mesh.material_id, specs, elem_type=et)
    return mesh, mats, specs, op


@pytest.mark.parametrize("et,dims,seed", [("P2", (6, 3, 4), 1), ("P2", (6, 3, 4), 2), ("P4", (3, 1, 2), 1)])
def test_bddc_regularised_matrix(cuda_device, et, dims, seed):
    """Tolerance: an entry is a handful of element contributions, each within a few tenths of 2^-53 of its element's
    largest, and as many FP64 additions for the elastic values, the same again for the corrections: some eight
    independent roundings of 2^-53 / sqrt(3) in the 2-norm, 1.8e-16, and the tangents' own (1 - r) D + r D_el none
    (the reference takes the rounded DS).  2e-16."""
    from slope_stability_petsc4py_gb300 import prepare_bddc_subdomain_pattern, synthetic

    mesh, mats, specs, op = _slope(et, dims)
    op.host_outputs = False
    op.set_bddc_subdomain_pattern(prepare_bddc_subdomain_pattern(
        mesh.coord, mesh.elem, mesh.q_mask, mesh.material_id, specs, (0, mesh.n_nodes // 2), elem_type=et,
        overlap_local_int_indices=op.owned_tangent_pattern.local_int_indices, adjacency_source="none"))
    op.reduction(1.1)
    op.constitutive_problem_stress_tangent(synthetic.displacement_field(mesh, mats, 0.004, seed=seed))
    r = 0.1
    K = op.build_bddc_regularized_matrix(r).values.cpu().numpy()
    pat = op.bddc_subdomain_pattern
    n_q, n_p = pat.n_q, pat.n_p
    share = float((op._branch != 0).double().mean())
    assert 0.02 < share < 0.9
    DS = np.asarray(op._owned_local_DS).T[pat.overlap_local_positions].reshape(-1, n_q, 6, 6).transpose(0, 1, 3, 2)
    g = np.stack([np.asarray(x).reshape(-1, n_q, n_p) for x in (pat.dphi1, pat.dphi2, pat.dphi3)], -1)
    w = np.asarray(pat.local_assembly_weight).reshape(-1, n_q).astype(LD)
    G, L = (pat.device[k].cpu().numpy().reshape(-1, n_q).astype(LD) for k in ("shear", "lame"))
    want = np.zeros(pat.nnz, LD)
    for e in range(g.shape[0]):
        D_el = np.zeros((n_q, 6, 6), LD)
        D_el[:, :3, :3] = L[e][:, None, None]
        for i in range(6):
            D_el[:, i, i] += (2 if i < 3 else 1) * G[e]
        D = (1 - LD(r)) * DS[e].astype(LD) + LD(r) * D_el
        B = np.zeros((n_q, 6, 3 * n_p), LD)
        for c in range(3):
            for z in range(3):
                B[:, BT[c][z], c::3] = g[e, :, :, z]
        Ke = sum(B[q].T @ ((w[e, q] * D[q]) @ B[q]) for q in range(n_q)).reshape(-1)
        at = pat.scatter_map[e].reshape(-1)
        np.add.at(want, at[at >= 0], Ke[at >= 0])
    want[pat.constrained_diag_positions] = 1.0
    assert _distance(K, want) <= 2e-16


def _components(et, shrink, small):
    """A pattern whose cells are thinned by the powers of ten `shrink` along x, y, z, displacements whose components
    and stresses whose rows and columns are scaled by `small`."""
    from slope_stability_petsc4py_gb300 import ConstitutiveOperator, synthetic

    mats = synthetic.MaterialSet.homogeneous()
    mesh = synthetic.slope_mesh_3d(*((4, 2, 2) if et == "P2" else (2, 1, 2)), elem_type=et)
    coord = mesh.coord * 10.0 ** np.asarray(shrink, dtype=np.float64)[:, None]
    specs = [dict(c0=float(mats.c0[0]), phi=float(mats.phi[0]), psi=float(mats.psi[0]), young=float(mats.young[0]),
                  poisson=float(mats.poisson[0]), gamma_sat=20.0, gamma_unsat=20.0)]
    pat = ConstitutiveOperator.from_mesh(coord, mesh.elem, mesh.q_mask, mesh.material_id, specs,
                                         elem_type=et).owned_tangent_pattern
    rng = np.random.default_rng(5)
    scale = np.asarray(small)
    u = (0.3 + rng.standard_normal((int(pat.overlap_nodes.size), 3))) * scale
    S = rng.standard_normal((pat.n_local_int, 6)) * np.array([scale[a] * scale[b] for a, b in
                                                              ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2))])
    return pat, u.reshape(-1), S


@pytest.mark.parametrize("et", ["P2", "P4"])
@pytest.mark.parametrize("shrink,small", [((0, 0, 0), (1.0, 1.0, 1.0)), ((0, 0, 0), (1.0, 1e-8, 1.0)),
                                          ((0, 0, -3), (1.0, 1.0, 0.0)), ((0, -3, 0), (1.0, 1e-8, 1e-4)),
                                          ((-6, 0, 0), (0.0, 1.0, 1e-12))])
def test_strain_and_force_component_by_component(cuda_device, et, shrink, small):
    """Each strain component and force component to a few ulps of its own terms, whatever the others are.

    An element's terms: for a strain row at a point the sum of |u_a - u_0| |grad phi_a| over its products, for a force
    component the sum of w |sigma| |grad phi_a|, both the largest over the element (one exponent holds its points and
    nodes).  FP64 sums are within some sqrt(30) x 2^-53 of that, the fixed-point ones (2^-56 an operand, of the
    largest difference and table entry, which are up to eight times a term) within about as much: 2^-50."""
    import torch

    from slope_stability_petsc4py_gb300 import _lib
    from slope_stability_petsc4py_gb300.distributed_tangent import _affine_fp64_inputs, _p2_affine_inputs
    from slope_stability_petsc4py_gb300.fem import quadrature, reference_gradients

    pat, u, S = _components(et, shrink, small)
    d = (_p2_affine_inputs if et == "P2" else _affine_fp64_inputs)(pat)
    assert d is not None
    n_el, n_q, n_p = int(pat.overlap_elements.size), pat.n_q, pat.n_p
    n_rows = int(pat.local_matrix_pattern.shape[0])
    jinv = d["jinv"].cpu().numpy().reshape(n_el, 3, 3).astype(LD)
    if et == "P2":  # the kernels' own inputs: barycentric coordinates
        lam = d["bary"].cpu().numpy().astype(LD)
        gl = np.concatenate([-jinv.sum(axis=1, keepdims=True), jinv], axis=1)
        g = np.empty((n_el, n_q, 10, 3), LD)
        for a in range(4):
            g[:, :, a] = (4 * lam[None, :, a, None] - 1) * gl[:, None, a]
        for a, (i, j) in zip(range(4, 10), ((0, 1), (1, 2), (0, 2), (1, 3), (2, 3), (0, 3))):
            g[:, :, a] = 4 * (lam[None, :, i, None] * gl[:, None, j] + lam[None, :, j, None] * gl[:, None, i])
    else:
        gh = np.transpose(reference_gradients(3, et), (2, 1, 0)).astype(LD)  # (n_q, n_p, 3)
        g = sum(gh[None, :, :, k, None] * jinv[:, None, None, k, :] for k in range(3))
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    E, F = (torch.zeros(n, dtype=torch.float64, device="cuda") for n in (6 * n_el * n_q, n_rows))
    ud, Sd = dev(u), dev(S)
    st, more = _lib.stream_handle(), [] if et == "P2" else [n_p]
    kind, table = ("_p2_affine", d["bary"]) if et == "P2" else ("_affine", d["ghat"])
    _lib.call("ssp_assemble_overlap_strain_3d" + kind, _lib.ptr(d["jinv"]), _lib.ptr(table), _lib.ptr(ud), u.size,
              _lib.ptr(d["dof_lids"]), n_el * n_q, n_el, *more, n_q, _lib.ptr(E), st)
    _lib.call("ssp_assemble_force_element" + kind, _lib.ptr(d["jinv"]), _lib.ptr(table), _lib.ptr(Sd), _lib.ptr(d["weight"]),
              _lib.ptr(d["elem_row"]), n_el, *more, n_q, n_rows, _lib.ptr(F), st)
    E, F = E.cpu().numpy().reshape(n_el, n_q, 6).astype(LD), F.cpu().numpy().astype(LD)
    ue = u[pat.overlap_element_dof_lids].reshape(n_el, n_p, 3).astype(LD)
    ue = ue - ue[:, :1]
    H, M = (np.stack([[sum(x[:, None, a, c] * y[:, :, a, z] for a in range(n_p)) for z in range(3)] for c in range(3)])
            for x, y in ((ue, g), (np.abs(ue), np.abs(g))))  # [c][z][e][q]
    for row, (x, y) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2))):
        want, terms = (H[x, x], M[x, x]) if x == y else (H[x, y] + H[y, x], M[x, y] + M[y, x])
        size = terms.max(axis=1, keepdims=True)
        assert np.all(np.abs(E[:, :, row] - want) <= 2.0**-50 * size), (row, float((np.abs(E[:, :, row] - want) / np.maximum(size, 1e-300)).max()))
    ws = pat.overlap_assembly_weight.reshape(n_el, n_q, 1).astype(LD) * S.reshape(n_el, n_q, 6).astype(LD)
    rows = d["elem_row"].cpu().numpy().reshape(n_el, n_p, 3)
    for c in range(3):
        f, terms = (sum((y[:, :, :, z] * x[:, :, None, BT[c][z]]).sum(axis=1) for z in range(3))
                    for x, y in ((ws, g), (np.abs(ws), np.abs(g))))  # (n_el, n_p)
        want, size = np.zeros(n_rows, LD), np.zeros(n_rows, LD)
        r = rows[:, :, c]
        np.add.at(want, r[r >= 0], f[r >= 0])
        np.add.at(size, r[r >= 0], np.broadcast_to(terms.max(axis=1, keepdims=True), r.shape)[r >= 0])
        mine = np.unique(r[r >= 0])
        err = np.abs(F[mine] - want[mine])
        assert np.all(err <= 2.0**-50 * size[mine]), (c, float((err / np.maximum(size[mine], 1e-300)).max()))


@pytest.mark.parametrize("thin", [1.0, 1e-3])
@pytest.mark.parametrize("et,kind", [("P2", "symmetric"), ("P2", "full"), ("P2", "correction"), ("P2", "moments"),
                                     ("P4", "symmetric"), ("P4", "full"), ("P4", "correction")])
def test_element_matrices_in_the_norm(cuda_device, et, kind, thin):
    """Element matrices of distorted, and of 1:1000, elements in the 2-norm.  Gradients, w D and H are within
    2^-57 or 2^-56 of their largest, an entry is rounded to FP64 once, and DS - D_el may cancel two bits: 2^-55 for each
    of three stages and 2^-53 / sqrt(3) are 1.5e-16 together; 3e-16 leaves a factor two for entries below
    the largest.  (FP64 sums are 1.6e-16 to 4.4e-16 away.)"""
    import torch

    from slope_stability_petsc4py_gb300 import _lib
    from slope_stability_petsc4py_gb300.fem import quadrature, reference_gradients

    rng = np.random.default_rng(7)
    n_el, n_p, n_q = (60, 10, 11) if et == "P2" else (8, 35, 24)
    n_ld = 3 * n_p
    nnz = n_el * n_ld * n_ld
    J = (np.eye(3) + 0.4 * rng.uniform(-1, 1, (n_el, 3, 3))) * rng.uniform(0.1, 5, (n_el, 1, 1))
    J[:, 2] *= thin  # dx_i / dxi_j
    jinv = np.linalg.inv(J)  # [k][i]: dxi_k / dx_i
    if kind == "moments":
        xi, _w = quadrature(3, et)
        bary = np.vstack([1 - xi.sum(0), xi]).T
        jl, lam = jinv.astype(LD), bary.astype(LD)
        gl = np.concatenate([-jl.sum(1, keepdims=True), jl], 1)
        g = np.empty((n_el, n_q, 10, 3), LD)
        for a in range(4):
            g[:, :, a] = (4 * lam[None, :, a, None] - 1) * gl[:, None, a]
        for a, (i, j) in zip(range(4, 10), ((0, 1), (1, 2), (0, 2), (1, 3), (2, 3), (0, 3))):
            g[:, :, a] = 4 * (lam[None, :, i, None] * gl[:, None, j] + lam[None, :, j, None] * gl[:, None, i])
    else:
        g = np.einsum("eki,kaq->eqai", jinv, np.asarray(reference_gradients(3, et)))
    G = np.repeat(rng.uniform(5e3, 2e4, (n_el, 1)), n_q, axis=1)
    L = 1.5 * G
    D_el = np.zeros((n_el, n_q, 6, 6), LD)
    D_el[..., :3, :3] = L[..., None, None]
    for i in range(6):
        D_el[..., i, i] += (2 if i < 3 else 1) * G
    V = rng.standard_normal((n_el, n_q, 6, 3))
    DS = D_el.astype(np.float64) - 0.1 * G[..., None, None] * np.einsum("eqik,eqjk->eqij", V, V)
    if kind == "full":
        DS = DS + 0.2 * G[..., None, None] * rng.standard_normal(DS.shape)
    w = rng.uniform(0.5, 1, (n_el, 1)) * rng.uniform(0.05, 0.2, (1, n_q))
    branch = (rng.uniform(size=(n_el, n_q)) < 0.7).astype(np.int8)
    branch[:, 0] = 1
    D = DS.astype(LD)
    if kind in ("correction", "moments"):
        D = (D - D_el) * (branch != 0)[..., None, None]
    want = np.zeros((n_el, n_ld, n_ld), LD)
    for e in range(n_el):
        B = np.zeros((n_q, 6, n_ld), LD)
        for c in range(3):
            for z in range(3):
                B[:, BT[c][z], c::3] = g[e, :, :, z]
        want[e] = sum(B[q].T @ ((LD(w[e, q]) * D[e, q]) @ B[q]) for q in range(n_q))
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    ds, wd, b, sh, la = (dev(a) for a in (DS.swapaxes(-1, -2).reshape(-1, 36), w.reshape(-1), branch.reshape(-1),
                                          G.reshape(-1), L.reshape(-1)))
    emap, elist = torch.arange(nnz, dtype=torch.int32, device="cuda"), torch.arange(n_el, dtype=torch.int32, device="cuda")
    count = dev(np.array([n_el], np.int32))
    K = torch.zeros(nnz, dtype=torch.float64, device="cuda")
    st = _lib.stream_handle()
    if kind == "moments":
        ji, ba = dev(jinv.reshape(n_el, 9)), dev(bary)
        _lib.call("ssp_tangent_plastic_correction_p2_moments", _lib.ptr(ji), _lib.ptr(ba), _lib.ptr(ds), _lib.ptr(wd),
                  _lib.ptr(b), _lib.ptr(sh), _lib.ptr(la), _lib.ptr(emap), n_el, n_q, nnz, 1.0, _lib.ptr(K), _lib.ptr(elist),
                  _lib.ptr(count), st)
    else:
        geo = [dev(g[..., z].reshape(-1, n_p)) for z in range(3)]
        if kind == "correction":
            _lib.call("ssp_tangent_plastic_correction", 3, *(_lib.ptr(x) for x in geo), _lib.ptr(ds), _lib.ptr(wd), _lib.ptr(b),
                      _lib.ptr(sh), _lib.ptr(la), _lib.ptr(emap), n_el, n_p, n_q, nnz, 1.0, _lib.ptr(K), _lib.ptr(elist),
                      _lib.ptr(count), st)
        else:
            _lib.call("ssp_tangent_element", 3, int(kind == "symmetric"), *(_lib.ptr(x) for x in geo), _lib.ptr(ds),
                      _lib.ptr(wd), _lib.ptr(emap), n_el, n_p, n_q, nnz, _lib.ptr(K), 0, st)
    assert _distance(K.cpu().numpy().reshape(want.shape), want) <= 3e-16


@pytest.mark.parametrize("dim,et,dims", [(2, "P1", (40, 30)), (2, "P4", (12, 8)), (3, "P1", (8, 4, 5))])
def test_bddc_matrix_of_fp64_elements(cuda_device, dim, et, dims):
    """Elements whose tangents are FP64 sums: the subdomain matrix is as near the exact sums as the full contraction
    of every point, whose reductions land in another order (up to a twentieth of the distance from run to run: a tenth)."""
    import torch

    from slope_stability_petsc4py_gb300 import ConstitutiveOperator, _lib, prepare_bddc_subdomain_pattern, synthetic
    from slope_stability_petsc4py_gb300.bddc import bddc_tangent_values_device

    mats = synthetic.MaterialSet.layered(4, seed=1)
    mesh = (synthetic.slope_mesh_3d if dim == 3 else synthetic.slope_mesh_2d)(*dims, elem_type=et, n_layers=4)
    specs = [dict(c0=float(mats.c0[i]), phi=float(mats.phi[i]), psi=float(mats.psi[i]), young=float(mats.young[i]),
                  poisson=float(mats.poisson[i]), gamma_sat=20.0, gamma_unsat=20.0) for i in range(mats.c0.size)]
    op = ConstitutiveOperator.from_mesh(mesh.coord, mesh.elem, mesh.q_mask, mesh.material_id, specs, elem_type=et)
    op.host_outputs = False
    op.set_bddc_subdomain_pattern(prepare_bddc_subdomain_pattern(
        mesh.coord, mesh.elem, mesh.q_mask, mesh.material_id, specs, (0, mesh.n_nodes // 2), elem_type=et,
        overlap_local_int_indices=op.owned_tangent_pattern.local_int_indices, adjacency_source="none"))
    op.reduction(1.1)
    op.constitutive_problem_stress_tangent(synthetic.displacement_field(mesh, mats, 0.004, seed=1))
    K = op.build_bddc_tangent_matrix().values.cpu().numpy()
    assert 0.02 < float((op._branch != 0).double().mean()) < 0.9
    pat, ns = op.bddc_subdomain_pattern, 6 if dim == 3 else 3
    n_q, n_p = pat.n_q, pat.n_p
    rows = np.ascontiguousarray(np.asarray(op._owned_local_DS).T[pat.overlap_local_positions])
    full = bddc_tangent_values_device(pat, torch.as_tensor(rows, device="cuda")).cpu().numpy()
    DS = rows.reshape(-1, n_q, ns, ns).transpose(0, 1, 3, 2).astype(LD)
    g = np.stack([np.asarray(x).reshape(-1, n_q, n_p) for x in (pat.dphi1, pat.dphi2, pat.dphi3)[:dim]], -1)
    w = np.asarray(pat.local_assembly_weight).reshape(-1, n_q).astype(LD)
    bt = BT if dim == 3 else ((0, 2), (2, 1))
    want = np.zeros(pat.nnz, LD)
    for e in range(g.shape[0]):
        B = np.zeros((n_q, ns, dim * n_p), LD)
        for c in range(dim):
            for z in range(dim):
                B[:, bt[c][z], c::dim] = g[e, :, :, z]
        Ke = sum(B[q].T @ ((w[e, q] * DS[e, q]) @ B[q]) for q in range(n_q)).reshape(-1)
        at = pat.scatter_map[e].reshape(-1)
        np.add.at(want, at[at >= 0], Ke[at >= 0])
    want[pat.constrained_diag_positions] = 1.0
    assert _distance(K, want) <= 1.1 * _distance(full, want)
