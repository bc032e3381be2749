"""Kernels that work on lists of points: the screened stresses and energies and the gather of plastic rows,
at list and block sizes where they can go wrong, against the one-pass kernels and plain indexing."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _points(n, plastic, seed):
    """Strains and strengths with about the given share of yielding points, some not finite at the end."""
    rng = np.random.default_rng(seed)
    E = 1e-3 * rng.standard_normal((n, 6))
    G, nu = rng.uniform(5e3, 2e4, n), rng.uniform(0.2, 0.45, n)
    lame = 2.0 * G * nu / (1.0 - 2.0 * nu)
    s = rng.uniform(0.2, 0.7, n)
    c = np.where(rng.uniform(size=n) < plastic, 5.0, 1e4)
    return E, c, s, G, lame + 2.0 * G / 3.0, lame


@pytest.mark.parametrize("n,plastic", [(1, 1.0), (31, 0.0), (33, 0.5), (257, 0.1), (5000, 0.12), (300001, 0.2)])
def test_screened_stress_and_energy(cuda_device, n, plastic):
    import torch

    from oracle import oracle_py as oracle
    from slope_stability_petsc4py_gb300 import _lib

    host = _points(n, plastic, n)
    E, c, s, G, K, L = (torch.as_tensor(a, device="cuda") for a in host)
    st = _lib.stream_handle()
    one, two = (torch.full((n, 6), -7.0, dtype=torch.float64, device="cuda") for _ in range(2))
    scratch = torch.empty(n + 4, dtype=torch.int32, device="cuda")
    mats = [_lib.ptr(a) for a in (c, s, G)]
    _lib.call("ssp_constitutive_3d_s", _lib.ptr(E), *mats, _lib.ptr(K), _lib.ptr(L), n, _lib.ptr(one), st)
    _lib.call("ssp_constitutive_3d_s_screened", _lib.ptr(E), *mats, _lib.ptr(L), n, _lib.ptr(two), _lib.ptr(scratch), st)
    assert rel_err(two.cpu().numpy(), one.cpu().numpy()) <= 1e-14
    psi = torch.empty(n, dtype=torch.float64, device="cuda")
    branch = torch.empty(n, dtype=torch.int8, device="cuda")
    part = torch.empty(_lib.POTENTIAL_PARTIALS + 1, dtype=torch.float64, device="cuda")
    w = torch.rand(n, dtype=torch.float64, device="cuda")
    totals = []
    for _ in range(2):
        _lib.call("ssp_potential_energy", 3, _lib.ptr(E), *mats, _lib.ptr(K), _lib.ptr(L), _lib.ptr(w), n, _lib.ptr(psi),
                  _lib.ptr(branch), _lib.ptr(part[:-1]), _lib.ptr(part[-1:]), st)
        totals.append(float(part[-1].item()))
    assert totals[0] == totals[1]
    ref_psi, ref_branch = oracle.potential_3d(host[0].T, *host[1:], with_branch=True)
    assert np.array_equal(branch.cpu().numpy(), ref_branch)
    assert rel_err(psi.cpu().numpy(), ref_psi) <= 1e-12
    assert abs(totals[0] - float(w.cpu().numpy() @ ref_psi)) <= 1e-12 * float(w.cpu().numpy() @ np.abs(ref_psi))


@pytest.mark.parametrize("n,entries", [(1, 9), (31, 36), (32, 36), (33, 9), (1000, 36)])
def test_gather_plastic_rows(cuda_device, n, entries):
    import torch

    from slope_stability_petsc4py_gb300 import _lib

    rng = np.random.default_rng(n)
    n_src = 2 * n + 3
    branch = rng.integers(0, 3, n_src).astype(np.int8)
    ds = rng.standard_normal((n_src, entries))
    pos = rng.permutation(n_src)[:n].astype(np.int32)
    dev = [torch.as_tensor(a, device="cuda") for a in (branch, ds, pos)]
    b = torch.full((n,), 9, dtype=torch.int8, device="cuda")
    rows = torch.full((n, entries), -7.0, dtype=torch.float64, device="cuda")
    _lib.call("ssp_gather_plastic_rows", *(_lib.ptr(a) for a in dev), n, n_src, entries, _lib.ptr(b), _lib.ptr(rows),
              _lib.stream_handle())
    assert np.array_equal(b.cpu().numpy(), branch[pos])
    want = np.where((branch[pos] != 0)[:, None], ds[pos], -7.0)
    assert np.array_equal(rows.cpu().numpy(), want)


@pytest.mark.parametrize("share", [1, 8])
@pytest.mark.parametrize("n_rows,longest", [(1, 1), (31, 300), (33, 7), (1000, 90), (517, 700), (40000, 3)])
def test_copy_marked_rows(cuda_device, n_rows, longest, share):
    import torch

    from slope_stability_petsc4py_gb300 import _lib

    rng = np.random.default_rng(n_rows)
    lengths = rng.integers(0, longest + 1, n_rows)
    indptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    src = torch.as_tensor(rng.standard_normal(int(indptr[-1]) + 1), device="cuda")[1:] if share == 1 else \
        torch.as_tensor(rng.standard_normal(int(indptr[-1])), device="cuda")  # an odd start: 8-byte copies
    for mark in (np.ones(n_rows), np.zeros(n_rows), rng.uniform(size=n_rows) < 0.5, np.arange(n_rows) % 32 == 31):
        mark = mark.astype(np.uint8)
        dst = torch.full_like(src, -7.0)
        dev = [torch.as_tensor(a, device="cuda") for a in (indptr, mark)]
        _lib.call("ssp_copy_rows_device_share", _lib.ptr(src), *(_lib.ptr(a) for a in dev), n_rows, int(src.numel()),
                  _lib.ptr(dst), share, _lib.stream_handle())
        on = np.repeat(mark != 0, lengths)
        assert np.array_equal(dst.cpu().numpy(), np.where(on, src.cpu().numpy(), -7.0))
