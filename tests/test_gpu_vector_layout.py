"""The direction path's vector layout (gather_dir.cu, scatter_dir.cu) where it
can go wrong: every number of time samples per plane (1, 2, 4, 8, 16 values of
a cell, several planes per slice above 16), partly filled planes, the
smallest width, grid sides that are no multiple of the tile, both padded-grid
FFTs, and the ways a tile's work is split over blocks.

Operators against the FP64 oracle at the suite's bar of 2e-5 relative; two
summation orders of the same FP32 terms at 5e-6, as between the per-ray paths.
"""

import numpy as np
import pytest

from oracle import rectv_oracle as orc
from rectv_gpu_gb300.phantom import scan_angles

OP_TOL = 2e-5
ORDER_TOL = 5e-6


def rel(a, b):
    b = np.asarray(b, np.float64)
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


def _phi(ntheta, m, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal((m, 2 * ntheta)) / np.sqrt(ntheta)).astype(np.float32)


CASES = [
    # n, ntheta, m, nz, nrot, centre offset
    (32, 32, 1, 3, 4, 0.0),      # one time sample: 16 slices per plane, three of them live
    (38, 48, 2, 9, 4, 0.5),      # 2n = 76: partial tiles; eight slices per plane, two planes
    (46, 60, 3, 5, 4, -1.0),     # three of four samples live
    (64, 96, 4, 4, 4, 0.0),
    (40, 72, 5, 3, 8, 0.0),      # five of eight samples, an odd slice
    (128, 96, 7, 3, 4, 1.5),     # hand-written padded-grid FFT, 2n = 256
    (256, 64, 4, 1, 8, 0.0),     # 2n = 512 with fused residual-row sizes
    (48, 90, 8, 1, 6, 0.0),
    (128, 96, 9, 1, 4, 0.0),     # nine of 16 values live
    (36, 64, 17, 2, 4, 0.0),     # two planes per slice, one sample in the second
    # mixed-radix grids: every radix of the passes (2n = 108, 88, 104, 140, 120, 144, 200, 272, 76, 960)
    (54, 40, 4, 2, 4, 0.0),
    (44, 40, 16, 1, 4, 0.5),
    (52, 40, 8, 3, 4, 0.0),
    (70, 40, 4, 3, 4, 0.0),
    (60, 40, 12, 1, 4, 0.0),
    (72, 40, 2, 5, 4, -1.5),
    (100, 40, 8, 2, 4, 0.0),
    (136, 40, 8, 2, 4, 0.0),
    (480, 24, 3, 1, 4, 0.0),
    (64, 256, 16, 1, 2, 0.0),    # 128 directions: tiles with several weight tables, split over blocks
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_operators_match_oracle(lib_built, torch_cuda, monkeypatch, case):
    torch = torch_cuda
    from rectv_gpu_gb300 import rectv
    monkeypatch.setenv("RECTV_DIRS", "1")
    n, ntheta, m, nz, nrot, dc = case
    theta, phi, center = scan_angles(ntheta, nrot), _phi(ntheta, m, n + m), n / 2 + dc
    rng = np.random.default_rng(n)
    f = rng.standard_normal((nz, m, n, n)).astype(np.float32)
    g = rng.standard_normal((nz, ntheta, n)).astype(np.float32)
    ops = orc.Operators(n, ntheta, m, theta, phi, center)
    obj = rectv(n, ntheta, m, nz, nz, 1)
    th, ph, df, dg = (torch.from_numpy(a).cuda() for a in (theta, phi, f, g))
    fw, ad = torch.full_like(dg, float("nan")), torch.zeros_like(df)
    torch.cuda.synchronize()
    obj.op_set_geometry(th.data_ptr(), ph.data_ptr(), center)
    assert obj.directions() > 0
    for _ in range(2):  # the second pass meets the first one's buffers
        ad.zero_()
        torch.cuda.synchronize()
        obj.op_radonapr(fw.data_ptr(), df.data_ptr(), nz, 1.0)
        obj.op_radonapradj(ad.data_ptr(), dg.data_ptr(), nz, 1.0)
    fw, ad = fw.cpu().numpy(), ad.cpu().numpy()
    obj.free()
    e = rel(fw, ops.radonapr(f.astype(np.float64), 1.0)), rel(ad, ops.radonapradj(g.astype(np.float64), 1.0))
    assert max(e) < OP_TOL, e


@pytest.mark.gpu
@pytest.mark.parametrize("case", [
    # n, ntheta, m, nz, nzp, nrot: mixed-radix grids and residual rows, an odd number of rows
    (54, 45, 5, 1, 1, 3),
    (84, 36, 16, 3, 1, 4),
])
def test_reconstruction_matches_oracle(lib_built, torch_cuda, case):
    from rectv_gpu_gb300 import Solver
    from rectv_gpu_gb300.phantom import add_noise, phantom4d
    n, ntheta, m, nz, nzp, nrot = case
    theta, phi = scan_angles(ntheta, nrot), _phi(ntheta, m, 2)
    ops = orc.Operators(n, ntheta, m, theta, phi, n / 2)
    g = add_noise(ops.radonapr(phantom4d(n, nz, m, ntheta, seed=1).astype(np.float64)), 0.01, 1)
    ref, hist = orc.run(g, theta, phi, n / 2, 4e-3, 4.0, 3, 3, nzp, return_history=True)
    with Solver(n, ntheta, m, nz, nzp, 1) as slv:
        slv.set_verbose(False)
        got = slv.recon(g, theta, phi, lambda0=1e-3, lambda1=4.0, niter=3, titer=3)
        assert slv.directions() > 0
        h = slv.history()
    assert rel(got, ref) < 1e-4, rel(got, ref)
    assert np.allclose(h["rho"], [x["rho"] for x in hist])


@pytest.mark.gpu
def test_work_split_agrees(lib_built, torch_cuda):
    """Many slices (whole tiles per block, dense tiles in several passes) and
    one slice (dense tiles over four blocks) give the same slice."""
    torch = torch_cuda
    from rectv_gpu_gb300 import rectv
    n, ntheta, m, nz = 64, 256, 16, 160
    theta, phi = scan_angles(ntheta, 4), _phi(ntheta, m, 1)
    gen = torch.Generator(device="cuda").manual_seed(3)
    g = torch.randn((nz, ntheta, n), generator=gen, device="cuda")
    th, ph = torch.from_numpy(theta).cuda(), torch.from_numpy(phi).cuda()
    out = []
    for z in (nz, 1):
        obj = rectv(n, ntheta, m, z, z, 1)
        f = torch.zeros((z, m, n, n), device="cuda")
        gz = g[nz - z:].contiguous()
        torch.cuda.synchronize()
        obj.op_set_geometry(th.data_ptr(), ph.data_ptr(), n / 2)
        obj.op_radonapradj(f.data_ptr(), gz.data_ptr(), z, 1.0)
        out.append(f[-1].cpu().numpy())
        obj.free()
    assert rel(out[0], out[1]) < ORDER_TOL


def test_odd_width_keeps_the_per_ray_kernels(lib_built):
    """Sample k of a ray mirrors sample n - k only for an even detector width."""
    from rectv_gpu_gb300 import plan_directions
    assert plan_directions(scan_angles(64, 8), 64)[0] == 8
    assert plan_directions(scan_angles(64, 8), 65)[0] == 0
    assert plan_directions(scan_angles(64, 8), 30)[0] == 0
