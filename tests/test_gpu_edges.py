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
