"""The TV kernels where their dispatch splits (tv_kernels.cu): the shrink of small
grids (five points' loads at a time, time samples that are no multiple of five)
and of large ones, and the gradient-divergence step with two voxels per thread.

The shrink against NumPy in FP64: its results are sums of at most four FP32 terms
of the size of the input's largest value (2^-24 each), one of them scaled by the
shrink factor, so 16 of them, 1e-6 of the largest value, bound the error; where a
column's sum of squares is compared, twice that.  Reconstructions at the bar of the
other solver tests (1e-4 relative)."""

import ctypes

import numpy as np
import pytest

from oracle import rectv_oracle as orc
from rectv_gpu_gb300.phantom import add_noise, phantom4d, scan_angles

TOL = 1e-6
RHO, LAM0, LAM1 = 0.5, 0.2, 4.0


def _device_shrink(torch, u, uo, psi, mu, n, m, nzp, nchunks):
    from rectv_gpu_gb300 import _lib
    lib = _lib.load()
    sums = torch.zeros(3, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    _lib.check(lib.rectv_shrink_noalloc(*(ctypes.c_void_p(t.data_ptr()) for t in (u, uo, psi, mu)), n, m, nzp, nchunks,
                                        RHO, LAM0, LAM1, ctypes.c_void_p(sums.data_ptr()), None))
    torch.cuda.synchronize()
    return sums.cpu().numpy()


def _grad(u, uo, c, n, m, nzp, nchunks):
    """G of chunk c on its dual grid: [4][nzp+1][m+1][n+1][n+1]"""
    sg = 1.0 / (2.0 * np.cbrt(2.0) * (LAM1 / 2.0))
    lo = uo[c * nzp - 1] if c > 0 else u[c * nzp]
    hi = uo[(c + 1) * nzp] if c < nchunks - 1 else u[(c + 1) * nzp - 1]
    e = np.concatenate([lo[None], u[c * nzp:(c + 1) * nzp], hi[None]])
    e = np.pad(e, ((0, 0), (1, 1), (1, 1), (1, 1)), mode="edge").astype(np.float64)
    f = e[:-1, :-1, :-1, :-1]
    return np.stack([sg * (e[:-1, :-1, :-1, 1:] - f), sg * (e[:-1, :-1, 1:, :-1] - f),
                     sg * LAM1 * (e[:-1, 1:, :-1, :-1] - f), sg * (e[1:, :-1, :-1, :-1] - f)])


def _volumes(seed, n, m, nz, nchunks, nzp):
    rng = np.random.default_rng(seed)
    u, uo = (rng.standard_normal((nz, m, n, n)).astype(np.float32) for _ in range(2))
    mu = rng.standard_normal((4, nchunks, nzp + 1, m + 1, n + 1, n + 1)).astype(np.float32)
    return u, uo, mu


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,nzp,nchunks", [(2, 1, 1, 1), (33, 4, 2, 1), (31, 5, 1, 3), (64, 9, 3, 2), (20, 15, 2, 1),
                                             (160, 4, 5, 2), (161, 3, 9, 1)])
def test_shrink_matches_numpy(lib_built, torch_cuda, n, m, nzp, nchunks):
    torch = torch_cuda
    u, uo, mu = _volumes(n + m, n, m, nzp * nchunks, nchunks, nzp)
    du, duo, dmu = (torch.from_numpy(a).cuda() for a in (u, uo, mu))
    dpsi = torch.zeros_like(dmu)
    sums = _device_shrink(torch, du, duo, dpsi, dmu, n, m, nzp, nchunks)
    psi, mu1 = dpsi.cpu().numpy(), dmu.cpu().numpy()
    want, size = np.zeros(3), 0.0
    for c in range(nchunks):
        h, ho = _grad(u, uo, c, n, m, nzp, nchunks), _grad(uo, uo, c, n, m, nzp, nchunks)
        a = h + mu[:, c] / RHO
        z = np.sqrt((a * a).sum(0))
        p = a * np.where(z <= LAM0 / RHO, 0.0, 1.0 - LAM0 / RHO / np.maximum(z, 1e-300))
        size = max(size, np.abs(a).max(), np.abs(h).max())
        assert np.abs(psi[:, c] - p).max() < TOL * size
        assert np.abs(mu1[:, c] - (mu[:, c] + RHO * h - RHO * p)).max() < TOL * size
        want += [((h - p) ** 2).sum(), ((ho - h) ** 2).sum(), 0.0]
    want[2] = ((u.astype(np.float64) - uo) ** 2).sum()
    assert np.allclose(sums, want, rtol=2 * TOL)


@pytest.mark.gpu
def test_shrink_kernels_agree(lib_built, torch_cuda):
    """Chunk 0 of two chunks (few blocks) and of forty (many) sees the same values."""
    torch = torch_cuda
    n, m, nzp = 48, 7, 2
    u, uo, mu = _volumes(1, n, m, nzp * 40, 40, nzp)
    out = []
    for nchunks in (2, 40):
        du, duo = (torch.from_numpy(a[:nzp * nchunks].copy()).cuda() for a in (u, uo))
        dmu = torch.from_numpy(mu[:, :nchunks].copy()).cuda()
        dpsi = torch.zeros_like(dmu)
        _device_shrink(torch, du, duo, dpsi, dmu, n, m, nzp, nchunks)
        out.append((dpsi[:, 0].cpu().numpy(), dmu[:, 0].cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.gpu
@pytest.mark.parametrize("titer", [1, 3])
def test_two_voxel_step_matches_oracle(lib_built, torch_cuda, titer):
    from rectv_gpu_gb300 import Solver
    n, ntheta, m, nz, nzp, nrot = 200, 24, 3, 8, 4, 4
    theta = scan_angles(ntheta, nrot)
    phi = (np.random.default_rng(3).standard_normal((m, 2 * ntheta)) / np.sqrt(ntheta)).astype(np.float32)
    ops = orc.Operators(n, ntheta, m, theta, phi, n / 2)
    g = add_noise(ops.radonapr(phantom4d(n, nz, m, ntheta, seed=1).astype(np.float64)), 0.01, 1)
    ref = orc.run(g, theta, phi, n / 2, 4e-3, 4.0, 2, titer, nzp)
    with Solver(n, ntheta, m, nz, nzp, 1) as slv:
        slv.set_verbose(False)
        got = slv.recon(g, theta, phi, lambda0=1e-3, lambda1=4.0, niter=2, titer=titer)
    err = np.linalg.norm(got.astype(np.float64) - ref) / np.linalg.norm(ref)
    assert err < 1e-4, err
