"""Strains that are not finite, or very large, through the elastic screen, the point lists, the energy's queue and the
Newton principal values; the Newton roots and reciprocals themselves."""

from __future__ import annotations

import ctypes
import subprocess

import numpy as np
import pytest

from conftest import rel_err
from test_gpu_lists import _points
from test_gpu_principal import _points as _pairs

pytestmark = pytest.mark.gpu


def _with_bad(n, seed):
    """Points of which some have an infinity or a nan in one entry, spread so that warps mix them with others."""
    E, c, s, G, K, L = _points(n, 0.4, seed)
    rng = np.random.default_rng(seed)
    bad = rng.uniform(size=n) < 0.07
    bad[:3] = bad[-1] = True
    at = np.flatnonzero(bad)
    E_bad = E.copy()
    E_bad[at, rng.integers(0, 6, at.size)] = rng.choice([np.nan, np.inf, -np.inf], at.size)
    return E, E_bad, bad, (c, s, G, K, L)


@pytest.mark.parametrize("n", [4, 130, 20011])
def test_screened_results_with_strains_that_are_not_finite(cuda_device, n):
    import torch

    from oracle import oracle_py as oracle
    from slope_stability_petsc4py_gb300 import _lib

    E, E_bad, bad, host = _with_bad(n, n)
    c, s, G, K, L = (torch.as_tensor(a, device="cuda") for a in host)
    st = _lib.stream_handle()
    mats = [_lib.ptr(a) for a in (c, s, G)]
    one, two, clean = (torch.full((n, 6), -7.0, dtype=torch.float64, device="cuda") for _ in range(3))
    scratch = torch.empty(3 * n + 12, dtype=torch.int32, device="cuda")
    dev = {k: torch.as_tensor(v, device="cuda") for k, v in dict(good=E, bad=E_bad).items()}
    _lib.call("ssp_constitutive_3d_s", _lib.ptr(dev["bad"]), *mats, _lib.ptr(K), _lib.ptr(L), n, _lib.ptr(one), st)
    _lib.call("ssp_constitutive_3d_s_screened", _lib.ptr(dev["bad"]), *mats, _lib.ptr(L), n, _lib.ptr(two), _lib.ptr(scratch), st)
    _lib.call("ssp_constitutive_3d_s", _lib.ptr(dev["good"]), *mats, _lib.ptr(K), _lib.ptr(L), n, _lib.ptr(clean), st)
    one, two, clean = (a.cpu().numpy() for a in (one, two, clean))
    assert np.array_equal(one, two, equal_nan=True)
    assert np.array_equal(one[~bad], clean[~bad])
    # tangents: binned (lists) against one pass in point order
    res = []
    for binned in (False, True):
        S, DS = (torch.full((n, k), -7.0, dtype=torch.float64, device="cuda") for k in (6, 36))
        branch = torch.full((n,), 9, dtype=torch.int8, device="cuda")
        if binned:
            _lib.call("ssp_constitutive_3d_sds_screened", _lib.ptr(dev["bad"]), *mats, _lib.ptr(L), n, _lib.ptr(S), _lib.ptr(DS),
                      _lib.ptr(branch), _lib.ptr(scratch), _lib.BINS_EXACT, None, 0, st)
        else:
            _lib.call("ssp_constitutive_sds_branch", 3, _lib.ptr(dev["bad"]), *mats, _lib.ptr(L), n, _lib.ptr(S), _lib.ptr(DS),
                      _lib.ptr(branch), st)
        res.append([a.cpu().numpy() for a in (S, DS, branch)])
    for a, b in zip(*res):
        assert np.array_equal(a, b, equal_nan=True)
    assert np.array_equal(res[0][0], one, equal_nan=True)
    # energies: the queue's neighbours of a bad point, the branch codes, and the total's nan
    psi, w = (torch.full((n,), v, dtype=torch.float64, device="cuda") for v in (-7.0, 1.0))
    branch = torch.full((n,), 9, dtype=torch.int8, device="cuda")
    part = torch.empty(_lib.POTENTIAL_PARTIALS + 1, dtype=torch.float64, device="cuda")
    _lib.call("ssp_potential_energy", 3, _lib.ptr(dev["bad"]), *mats, _lib.ptr(K), _lib.ptr(L), _lib.ptr(w), n, _lib.ptr(psi),
              _lib.ptr(branch), _lib.ptr(part[:-1]), _lib.ptr(part[-1:]), st)
    with np.errstate(all="ignore"):
        ref_psi, ref_branch = oracle.potential_3d(E_bad.T, *host, with_branch=True)
    psi, branch = psi.cpu().numpy(), branch.cpu().numpy()
    assert np.array_equal(branch, ref_branch)
    assert np.array_equal(np.isnan(psi), np.isnan(ref_psi))
    assert rel_err(psi[~bad], ref_psi[~bad]) <= 1e-12
    assert not np.isfinite(float(part[-1].item()))


@pytest.mark.parametrize("amplitude", [1e60, 1e80, 1e95])
def test_very_large_strains_return_to_the_yield_surface(cuda_device, amplitude):
    """The refinement of a close pair squares the squared strains; where that overflows the pair stays as it was,
    to the accuracy of the invariants (sqrt(2^-53) of the gap near an edge, 1e-7 of the strain at the worst)."""
    import torch

    from slope_stability_petsc4py_gb300 import _lib

    host = _pairs(amplitude, 3)
    E, c, s, G, K, L = (torch.as_tensor(np.ascontiguousarray(a), device="cuda") for a in host)
    n = c.numel()
    S = torch.empty((n, 6), dtype=torch.float64, device="cuda")
    branch = torch.empty(n, dtype=torch.int8, device="cuda")
    _lib.call("ssp_constitutive_3d_branch", *(_lib.ptr(a) for a in (E, c, s, G, L)), n, _lib.ptr(S), _lib.ptr(branch),
              _lib.stream_handle())
    S, branch = S.cpu().numpy() / amplitude, branch.cpu().numpy()
    e, cb, sp, shear, _, lame = host
    assert np.all(np.isfinite(S))
    sig = np.linalg.eigvalsh(np.stack([S[:, k] for k in (0, 3, 5, 3, 1, 4, 5, 4, 2)], 1).reshape(n, 3, 3))
    f = (1.0 + sp) * sig[:, 2] - (1.0 - sp) * sig[:, 0] - cb / amplitude
    size = (2.0 * shear + 3.0 * lame) * (np.abs(e) / amplitude).max(1) + cb / amplitude
    plastic = branch != 0
    assert plastic.any() and not plastic.all()
    tol = 1e-12 if amplitude < 1e77 else 1e-6
    assert np.all(np.abs(f[plastic]) <= tol * size[plastic]) and np.all(f[~plastic] <= tol * size[~plastic])


SOURCE = r"""
#include "mohr_coulomb.cuh"
namespace ssp { __device__ int g_device_status; }
__global__ void helpers(const double *x, int n, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    ssp::roots_newton(x[i], out[3 * i], out[3 * i + 1]);
    out[3 * i + 2] = ssp::recip_newton(x[i]);
}
extern "C" int run(const double *x, int n, double *out) {
    helpers<<<(n + 127) / 128, 128>>>(x, n, out);
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
"""


def test_newton_roots_and_reciprocals(cuda_device, tmp_path):
    """Within 1.5 units in the last place over FP64's normal range, on either side of the ends of the FP32 start,
    and what the CUDA routines give for zeros, subnormal numbers, infinities and nans."""
    import torch

    from slope_stability_petsc4py_gb300 import _lib, build

    src, lib = tmp_path / "helpers.cu", tmp_path / "helpers.so"
    src.write_text(SOURCE)
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-rdc=true", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
                    f"-I{build.CSRC}", "-shared", str(src), "-o", str(lib)], check=True)
    fn = ctypes.CDLL(str(lib)).run
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    rng = np.random.default_rng(1)
    x = 2.0 ** rng.uniform(-1022, 1021, 200000)
    x = np.concatenate([x, 2.0 ** rng.uniform(-115, 115, 400000), 1.0 + np.arange(-2000, 2000) * 2.0**-52])
    ends = 2.0 ** np.array([-110.0, -109.0, 109.0, 110.0])
    x = np.concatenate([x, ends, np.nextafter(ends, 0), np.nextafter(ends, np.inf)])
    special = np.array([0.0, -0.0, 5e-324, 1e-310, np.inf, np.nan, -1.0, -2.0**-200])
    x = np.concatenate([x, special])
    xd = torch.as_tensor(x, device="cuda")
    out = torch.empty((x.size, 3), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert fn(_lib.ptr(xd), x.size, _lib.ptr(out)) == 0
    got = out.cpu().numpy()
    n = x.size - special.size
    xl = x[:n].astype(np.longdouble)
    with np.errstate(over="ignore"):
        want = [np.sqrt(xl), 1 / np.sqrt(xl), 1 / xl]
    for k, w in enumerate(want):
        ulp = np.spacing(np.abs(w).astype(np.float64))
        ok = np.isfinite(w.astype(np.float64)) & (np.abs(w) >= 2.3e-308)
        assert np.all(np.abs(got[:n, k] - w)[ok] <= 1.5 * ulp[ok]), k
    sx = torch.as_tensor(special, device="cuda")
    routines = torch.stack([sx.sqrt(), 1.0 / sx.sqrt(), 1.0 / sx], 1).cpu().numpy()
    assert np.array_equal(got[n:], routines, equal_nan=True)
