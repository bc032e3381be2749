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
