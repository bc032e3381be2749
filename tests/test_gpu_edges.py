"""Calls at the edges of what the kernels' fast forms take: bad row maps, inputs that are not finite, many points
per element, pointers off a 16-byte boundary."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _clean_status(cuda_device):
    from slope_stability_petsc4py_gb300 import _lib

    _lib.device_status(clear=True)
    yield
    assert _lib.device_status(clear=True) == 0


def _pattern(et, dims):
    from slope_stability_petsc4py_gb300 import ConstitutiveOperator, synthetic

    mats = synthetic.MaterialSet.homogeneous()
    mesh = synthetic.slope_mesh_3d(*dims, elem_type=et)
    specs = [dict(c0=float(mats.c0[0]), phi=float(mats.phi[0]), psi=float(mats.psi[0]), young=float(mats.young[0]),
                  poisson=float(mats.poisson[0]), gamma_sat=20.0, gamma_unsat=20.0)]
    return ConstitutiveOperator.from_mesh(mesh.coord, mesh.elem, mesh.q_mask, mesh.material_id, specs,
                                          elem_type=et).owned_tangent_pattern


def _dev(a):
    import torch

    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


BAD_INDEX = 1  # SSP_DEV_BAD_INDEX


@pytest.mark.parametrize("finite", [True, False])
@pytest.mark.parametrize("et", ["P2", "P4"])
def test_bad_row_of_a_force_is_reported(et, finite):
    """A row beyond the force vector is skipped and reported, also in an element with a stress that is not finite."""
    import torch

    from slope_stability_petsc4py_gb300 import _lib
    from slope_stability_petsc4py_gb300.distributed_tangent import _affine_fp64_inputs, _p2_affine_inputs

    pat = _pattern(et, (2, 1, 1))
    d = (_p2_affine_inputs if et == "P2" else _affine_fp64_inputs)(pat)
    n_el, n_q, n_rows = int(pat.overlap_elements.size), pat.n_q, int(pat.local_matrix_pattern.shape[0])
    rows = d["elem_row"].cpu().numpy().reshape(n_el, -1).copy()
    S = np.random.default_rng(1).standard_normal((n_el * n_q, 6))
    if not finite:
        S[n_q + 1, 2] = np.inf

    def force(rows):
        F, Sd, r = torch.empty(n_rows, dtype=torch.float64, device="cuda"), _dev(S), _dev(rows)
        if et == "P2":
            _lib.call("ssp_assemble_force_element_p2_affine", _lib.ptr(d["jinv"]), _lib.ptr(d["bary"]), _lib.ptr(Sd),
                      _lib.ptr(d["weight"]), _lib.ptr(r), n_el, n_q, n_rows, _lib.ptr(F), _lib.stream_handle())
        else:
            _lib.call("ssp_assemble_force_element_affine", _lib.ptr(d["jinv"]), _lib.ptr(d["ghat"]), _lib.ptr(Sd),
                      _lib.ptr(d["weight"]), _lib.ptr(r), n_el, pat.n_p, n_q, n_rows, _lib.ptr(F), _lib.stream_handle())
        return F.cpu().numpy()

    force(rows)
    assert _lib.device_status(clear=True) == 0
    k = int(np.flatnonzero(rows[1] >= 0)[0])
    rows[1, k] = n_rows
    force(rows)
    assert _lib.device_status(clear=True) == BAD_INDEX


def _p2_gradients(jinv, lam):
    """(n_el, n_q, 10, 3) gradients of straight-sided P2 tetrahedra at barycentric points lam (n_q, 4)."""
    gl = np.concatenate([-jinv.sum(axis=1, keepdims=True), jinv], axis=1)
    g = np.empty((jinv.shape[0], lam.shape[0], 10, 3), dtype=jinv.dtype)
    for a in range(4):
        g[:, :, a] = (4 * lam[None, :, a, None] - 1) * gl[:, None, a]
    for a, (i, j) in zip(range(4, 10), ((0, 1), (1, 2), (0, 2), (1, 3), (2, 3), (0, 3))):
        g[:, :, a] = 4 * (lam[None, :, i, None] * gl[:, None, j] + lam[None, :, j, None] * gl[:, None, i])
    return g


@pytest.mark.parametrize("n_q,odd", [(1, False), (11, True), (30, False), (31, False), (2049, False), (2100, True)])
def test_p2_strain_and_force_point_counts_and_alignment(n_q, odd):
    """Any number of points per element, and E and the stresses at any multiple of eight bytes.  Tolerance as in
    the tests of the fixed-point kernels, 1e-13 of the largest value for sums of 30 terms (the strain), and
    sqrt(n_q) times that for the force's sums over the points."""
    import torch

    from slope_stability_petsc4py_gb300 import _lib
    from slope_stability_petsc4py_gb300.distributed_tangent import _p2_affine_inputs

    pat = _pattern("P2", (3, 2, 1))
    d = _p2_affine_inputs(pat)
    rng = np.random.default_rng(n_q)
    n_el, n_rows = int(pat.overlap_elements.size), int(pat.local_matrix_pattern.shape[0])
    lam = rng.dirichlet(np.ones(4), n_q)
    g = _p2_gradients(d["jinv"].cpu().numpy().reshape(n_el, 3, 3), lam)
    dof = pat.overlap_element_dof_lids
    u = rng.standard_normal(int(pat.overlap_global_dofs.size))
    bary, ud = _dev(lam), _dev(u)

    def room(n):
        return torch.full((n + 1,), -7.0, dtype=torch.float64, device="cuda")[1:] if odd else \
            torch.full((n,), -7.0, dtype=torch.float64, device="cuda")

    E = room(n_el * n_q * 6)
    assert E.data_ptr() % 16 == (8 if odd else 0)
    _lib.call("ssp_assemble_overlap_strain_3d_p2_affine", _lib.ptr(d["jinv"]), _lib.ptr(bary), _lib.ptr(ud), u.size,
              _lib.ptr(d["dof_lids"]), n_el * n_q, n_el, n_q, _lib.ptr(E), _lib.stream_handle())
    ue = u[dof].reshape(n_el, 10, 3)
    H = np.einsum("eac,eqaz->eqcz", ue, g)
    want = np.stack([H[..., 0, 0], H[..., 1, 1], H[..., 2, 2], H[..., 0, 1] + H[..., 1, 0], H[..., 1, 2] + H[..., 2, 1],
                     H[..., 0, 2] + H[..., 2, 0]], -1)
    assert rel_err(E.cpu().numpy(), want.reshape(-1)) <= 1e-13
    S = room(n_el * n_q * 6)
    S_host = rng.standard_normal((n_el * n_q, 6))
    S.copy_(torch.as_tensor(S_host.reshape(-1)))
    w = rng.uniform(0.0, 1.0, n_el * n_q)
    wd, F = _dev(w), torch.empty(n_rows, dtype=torch.float64, device="cuda")
    _lib.call("ssp_assemble_force_element_p2_affine", _lib.ptr(d["jinv"]), _lib.ptr(bary), _lib.ptr(S), _lib.ptr(wd),
              _lib.ptr(d["elem_row"]), n_el, n_q, n_rows, _lib.ptr(F), _lib.stream_handle())
    ws = (w[:, None] * S_host).reshape(n_el, n_q, 6)
    bt = ((0, 3, 5), (3, 1, 4), (5, 4, 2))
    rows = d["elem_row"].cpu().numpy().reshape(n_el, 10, 3)
    f = np.stack([sum(np.einsum("eqa,eq->ea", g[..., z], ws[..., bt[c][z]]) for z in range(3)) for c in range(3)], -1)
    want = np.zeros(n_rows)
    np.add.at(want, rows[rows >= 0], f[rows >= 0])
    assert rel_err(F.cpu().numpy(), want) <= 1e-13 * max(1.0, n_q / 11.0) ** 0.5


def test_subnormal_inputs(oracle):
    """Displacements, stresses and tangents among FP64's subnormal numbers count as what they are.  Tolerance: 1e-13
    of the largest value as elsewhere, and a quantum of the subnormal range (5e-324) for each of the roundings to it,
    of which an element's force or tangent has one and an entry a few dozen elements at most."""
    import torch

    from slope_stability_petsc4py_gb300 import _lib
    from slope_stability_petsc4py_gb300.distributed_tangent import _affine_fp64_inputs, _p2_affine_inputs

    tiny, step = 2.0**-1030, 2.0**-44  # a quantum of the subnormal range, 2^-1074, scaled up again
    for et, dims in (("P2", (2, 2, 1)), ("P4", (2, 1, 1))):
        pat = _pattern(et, dims)
        d = (_p2_affine_inputs if et == "P2" else _affine_fp64_inputs)(pat)
        rng = np.random.default_rng(3)
        n_el, n_q, n_p, n_rows = int(pat.overlap_elements.size), pat.n_q, pat.n_p, int(pat.local_matrix_pattern.shape[0])
        u = np.round(rng.standard_normal(int(pat.overlap_global_dofs.size)) * 2.0**40) * 2.0**-40  # exact when scaled
        S = np.round(rng.standard_normal((n_el * n_q, 6)) * 2.0**40) * 2.0**-40
        A = rng.standard_normal((n_el * n_q, 6, 6))
        DS = np.round((A + A.transpose(0, 2, 1)) * 2.0**40) * 2.0**-40
        affine = et == "P4"

        def run(scale):
            E, F = (torch.zeros(n, dtype=torch.float64, device="cuda") for n in (6 * n_el * n_q, n_rows))
            K, Km = (torch.zeros(pat.nnz, dtype=torch.float64, device="cuda") for _ in range(2))
            ud, Sd, Dd = _dev(u * scale), _dev(S * scale), _dev(DS.transpose(0, 2, 1).reshape(-1, 36) * scale)
            st, table = _lib.stream_handle(), d["ghat" if affine else "bary"]
            _lib.call("ssp_assemble_overlap_strain_3d" + ("_affine" if affine else "_p2_affine"), _lib.ptr(d["jinv"]),
                      _lib.ptr(table), _lib.ptr(ud), u.size, _lib.ptr(d["dof_lids"]), n_el * n_q, n_el,
                      *([n_p] if affine else []), n_q, _lib.ptr(E), st)
            _lib.call("ssp_assemble_force_element" + ("_affine" if affine else "_p2_affine"), _lib.ptr(d["jinv"]),
                      _lib.ptr(table), _lib.ptr(Sd), _lib.ptr(d["weight"]), _lib.ptr(d["elem_row"]), n_el,
                      *([n_p] if affine else []), n_q, n_rows, _lib.ptr(F), st)
            geo = [_lib.ptr(d[k]) for k in ("dphi1", "dphi2", "dphi3")]
            _lib.call("ssp_tangent_element", 3, 1, *geo, _lib.ptr(Dd), _lib.ptr(d["weight"]), _lib.ptr(d["scatter_map"]),
                      n_el, n_p, n_q, pat.nnz, _lib.ptr(K), 0, st)
            if et == "P2":
                zero = torch.zeros(n_el * n_q, dtype=torch.float64, device="cuda")
                branch = torch.ones(n_el * n_q, dtype=torch.int8, device="cuda")
                elist, count = torch.arange(n_el, dtype=torch.int32, device="cuda"), _dev(np.array([n_el], np.int32))
                _lib.call("ssp_tangent_plastic_correction_p2_moments", _lib.ptr(d["jinv"]), _lib.ptr(table), _lib.ptr(Dd),
                          _lib.ptr(d["weight"]), _lib.ptr(branch), _lib.ptr(zero), _lib.ptr(zero), _lib.ptr(d["scatter_map"]),
                          n_el, n_q, pat.nnz, 1.0, _lib.ptr(Km), _lib.ptr(elist), _lib.ptr(count), st)
            return [x.cpu().numpy() for x in (E, F, K, Km)]

        for got, want in zip(run(tiny), run(1.0)):
            err = np.abs(got * 2.0**1000 * 2.0**30 - want)
            assert np.all(err <= 1e-13 * np.abs(want).max() + 64 * step)
            assert got.any() or not want.any()
