"""Principal values in the return mapping and the potential energy where they are hardest: exact and close pairs
on either side, spherical strains, and strains beyond the range in which FP32 starts the Newton steps."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

# errors of a few tens of ulps of the trial state (2e-14) are expected of either side
TOL = 1e-12


def _points(amplitude, seed):
    rng = np.random.default_rng(seed)
    gaps = np.array([0.0, 1e-15, 1e-12, 1e-8, 1e-5, 1e-3, 4e-3, 6e-3, 2e-2, 0.3])
    n = 40 * gaps.size
    gap = np.repeat(gaps, 40)
    e = np.zeros((n, 3))
    upper = np.arange(n) % 2 == 0
    e[:, 0] = rng.uniform(-0.3, 0.3, n)
    e[:, 1] = e[:, 0] + gap
    e[:, 2] = e[:, 0] + np.where(upper, -1.0, 1.0) * rng.uniform(0.5, 2.0, n)
    e[::40] = np.where(np.arange(gaps.size) % 2 == 0, 0.7, -0.7)[:, None]  # spherical
    q, _ = np.linalg.qr(rng.standard_normal((n, 3, 3)))
    q[::3] = np.eye(3)  # axis-aligned: pairs exact to the bit
    t = amplitude * np.einsum("nij,nj,nkj->nik", q, e, q)
    E = np.stack([t[:, 0, 0], t[:, 1, 1], t[:, 2, 2], 2 * t[:, 0, 1], 2 * t[:, 1, 2], 2 * t[:, 0, 2]], 1)
    G, nu = rng.uniform(5e3, 2e4, n), rng.uniform(0.2, 0.45, n)
    lame = 2.0 * G * nu / (1.0 - 2.0 * nu)
    return E, amplitude * G * rng.uniform(0.0, 3.0, n), rng.uniform(0.2, 0.7, n), G, lame + 2.0 * G / 3.0, lame


@pytest.mark.parametrize("amplitude", [1e-20, 1e-12, 1e-4, 1e3, 1e20])
def test_returned_stress_is_on_the_yield_surface(cuda_device, amplitude):
    import torch

    from slope_stability_petsc4py_gb300 import _lib

    host = _points(amplitude, 3)
    E, c, s, G, K, L = (torch.as_tensor(np.ascontiguousarray(a), device="cuda") for a in host)
    n = c.numel()
    S = torch.empty((n, 6), dtype=torch.float64, device="cuda")
    branch = torch.empty(n, dtype=torch.int8, device="cuda")
    _lib.call("ssp_constitutive_3d_branch", *(_lib.ptr(a) for a in (E, c, s, G, L)), n, _lib.ptr(S), _lib.ptr(branch),
              _lib.stream_handle())
    S, branch = S.cpu().numpy(), branch.cpu().numpy()
    e, cb, sp, shear, _, lame = host
    m = np.stack([S[:, k] for k in (0, 3, 5, 3, 1, 4, 5, 4, 2)], 1).reshape(n, 3, 3)
    sig = np.linalg.eigvalsh(m)
    f = (1.0 + sp) * sig[:, 2] - (1.0 - sp) * sig[:, 0] - cb
    size = (2.0 * shear + 3.0 * lame) * np.abs(e).max(1) + cb
    plastic = branch != 0
    assert plastic.any() and not plastic.all()
    if amplitude >= 1e-12:  # below sqrt(Q) = 1e-15 the strain counts as spherical
        assert np.all(np.abs(f[plastic]) <= TOL * size[plastic])
        assert np.all(f[~plastic] <= TOL * size[~plastic])
    assert np.all(np.isfinite(S))


@pytest.mark.parametrize("amplitude", [1e-12, 1e-6, 1e-3, 1e3])
def test_energy_of_close_pairs(cuda_device, amplitude):
    import torch

    from oracle import oracle_py as oracle
    from slope_stability_petsc4py_gb300 import _lib

    host = _points(amplitude, 4)
    E, c, s, G, K, L = (torch.as_tensor(np.ascontiguousarray(a), device="cuda") for a in host)
    n = c.numel()
    psi = torch.empty(n, dtype=torch.float64, device="cuda")
    part = torch.empty(_lib.POTENTIAL_PARTIALS + 1, dtype=torch.float64, device="cuda")
    branch = torch.empty(n, dtype=torch.int8, device="cuda")
    w = torch.ones(n, dtype=torch.float64, device="cuda")
    _lib.call("ssp_potential_energy", 3, *(_lib.ptr(a) for a in (E, c, s, G, K, L, w)), n, _lib.ptr(psi),
              _lib.ptr(branch), _lib.ptr(part[:-1]), _lib.ptr(part[-1:]), _lib.stream_handle())
    want = oracle.potential_3d(host[0].T, *host[1:])
    assert rel_err(psi.cpu().numpy(), want) <= TOL
