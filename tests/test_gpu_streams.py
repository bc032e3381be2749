"""Operators that share a pattern on streams of their own."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _slope(et="P2", dims=(5, 3, 4)):
    from slope_stability_petsc4py_gb300 import ConstitutiveOperator, prepare_bddc_subdomain_pattern, synthetic

    mats = synthetic.MaterialSet.layered(4, seed=1)
    mesh = synthetic.slope_mesh_3d(*dims, elem_type=et, n_layers=4)
    specs = [dict(c0=float(mats.c0[i]), phi=float(mats.phi[i]), psi=float(mats.psi[i]), young=float(mats.young[i]),
                  poisson=float(mats.poisson[i]), gamma_sat=20.0, gamma_unsat=20.0) for i in range(mats.c0.size)]
    op = ConstitutiveOperator.from_mesh(mesh.coord, mesh.elem, mesh.q_mask, mesh.material_id, specs, elem_type=et)
    sub = prepare_bddc_subdomain_pattern(mesh.coord, mesh.elem, mesh.q_mask, mesh.material_id, specs, (0, mesh.n_nodes // 2),
                                         elem_type=et, overlap_local_int_indices=op.owned_tangent_pattern.local_int_indices,
                                         adjacency_source="none")
    return mesh, synthetic.displacement_field(mesh, mats, 0.004, seed=2), op, sub


def _same(op, pattern):
    from slope_stability_petsc4py_gb300 import ConstitutiveOperator

    other = ConstitutiveOperator(B=None, c0=op.c0, phi=op.phi, psi=op.psi, Davis_type=op.Davis_type, shear=op.shear,
                                 bulk=op.bulk, lame=op.lame, WEIGHT=op.WEIGHT, n_strain=op.n_strain, n_int=op.n_int,
                                 dim=op.dim, q_mask=op.q_mask)
    other.set_owned_tangent_pattern(pattern, constitutive_mode="overlap")
    return other


def test_free_rows_are_made_with_the_pattern(cuda_device):
    _mesh, _U, op, sub = _slope()
    pat = op.owned_tangent_pattern
    rows = pat.device["elem_row"].cpu().numpy()
    place = np.full(int(pat.local_matrix_pattern.shape[0]) + 1, -1)
    place[pat.owned_free_local_rows] = np.arange(pat.owned_free_local_rows.size)
    assert np.array_equal(pat.device["elem_free_row"].cpu().numpy(), place[rows])
    assert np.array_equal(sub.device["overlap_positions"].cpu().numpy(), sub.overlap_local_positions)


def test_first_forces_of_two_operators_on_two_streams(cuda_device):
    """A table that operators share is there before either asks for it, whichever stream each is on."""
    import torch

    _mesh, U, op, sub = _slope()
    pat = op.owned_tangent_pattern
    u = torch.as_tensor(U, device="cuda")
    ops = [_same(op, pat) for _ in range(2)]
    for o in ops:
        o.host_outputs = False
        o.set_bddc_subdomain_pattern(sub)
    before = [set(pat.device), set(sub.device)]
    torch.cuda.synchronize()
    F, K = [], []
    for o in ops:
        with torch.cuda.stream(torch.cuda.Stream()):
            F.append(o.build_F_all_free(1.1, u))
            o.constitutive_problem_stress_tangent(u)
            K.append(o.build_bddc_regularized_matrix(0.1).values)
    torch.cuda.synchronize()
    lazy = {"bary"}  # copied from the host in one synchronous call
    assert set(pat.device) - before[0] <= lazy and set(sub.device) == before[1]
    op.host_outputs = False
    op.set_bddc_subdomain_pattern(sub)
    want = op.build_F_all_free(1.1, u)
    op.constitutive_problem_stress_tangent(u)
    K_want = op.build_bddc_regularized_matrix(0.1).values
    free = torch.as_tensor(pat.owned_free_local_rows, device="cuda")
    whole = op.build_F().T.reshape(-1)[free]
    for f in (*F, whole):
        assert float((f - want).abs().max() / want.abs().max()) <= 1e-14
    for k in K:
        assert float((k - K_want).abs().max() / K_want.abs().max()) <= 1e-14


@pytest.mark.parametrize("dims", [(3, 2, 2), (8, 5, 7)])
def test_host_copy_holds_the_values_on_its_stream(cuda_device, monkeypatch, dims):
    """The CSR values stay allocated until their copy to the host has read them, whichever stream it runs on (few
    values: the caller's, many: a side stream)."""
    import torch

    from slope_stability_petsc4py_gb300 import problem

    _mesh, U, op, _sub = _slope(dims=dims)
    few = op.owned_tangent_pattern.nnz < problem.IN_LINE_HOST_VALUES
    assert few == (dims == (3, 2, 2))
    _F, K = op.build_F_K_regularized_all_free(1.1, U, 0.1)
    torch.cuda.synchronize()
    seen, real = [], torch.Tensor.record_stream

    def record(self, stream):
        if self.data_ptr() == K.values.data_ptr():
            seen.append(stream.cuda_stream)
        return real(self, stream)

    monkeypatch.setattr(torch.Tensor, "record_stream", record)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        K.sync_host()
        assert seen == [s.cuda_stream if few else K._copy_stream.cuda_stream]
        host = K.getValuesCSR()[2]
    assert np.array_equal(host, K.values.cpu().numpy())
