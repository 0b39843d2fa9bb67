"""Both USFFT operators where the oversampled grid's side 2n is no multiple of
the 16-cell tile: the last tile of an axis is 2n mod 16 cells wide, and a
nine-cell stencil that reaches over one narrower than eight touches three tiles
(widths of 1, 2 and 3 mod 8).

Operators against the FP64 oracle at the suite's bar of 2e-5 relative, and
<R u, g> = <u, R* g> to 1e-5 relative.
"""

import numpy as np
import pytest

from oracle import rectv_oracle as orc
from rectv_gpu_gb300.phantom import scan_angles

OP_TOL = 2e-5
DOT_TOL = 1e-5
# every residue of 2n modulo 16, 2, 4 and 6 (one narrow tile) more than once
WIDTHS = [33, 34, 35, 36, 37, 38, 39, 42, 43, 50, 65, 98, 106, 131]


def rel(a, b):
    b = np.asarray(b, np.float64)
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


def _phi(ntheta, m, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal((m, 2 * ntheta)) / np.sqrt(ntheta)).astype(np.float32)


def _check(torch, n, m, nz, ntheta, nrot, dirs):
    from rectv_gpu_gb300 import rectv
    theta, phi, center = scan_angles(ntheta, nrot), _phi(ntheta, m, n + m), n / 2 + 0.5
    rng = np.random.default_rng(n)
    f = rng.standard_normal((nz, m, n, n)).astype(np.float32)
    g = rng.standard_normal((nz, ntheta, n)).astype(np.float32)
    ops = orc.Operators(n, ntheta, m, theta, phi, center)
    obj = rectv(n, ntheta, m, nz, nz, 1)
    th, ph, df, dg = (torch.from_numpy(a).cuda() for a in (theta, phi, f, g))
    fw, ad = torch.zeros_like(dg), torch.zeros_like(df)
    torch.cuda.synchronize()
    obj.op_set_geometry(th.data_ptr(), ph.data_ptr(), center)
    assert (obj.directions() > 0) == dirs
    obj.op_radonapr(fw.data_ptr(), df.data_ptr(), nz, 1.0)
    obj.op_radonapradj(ad.data_ptr(), dg.data_ptr(), nz, 1.0)
    fw, ad = fw.cpu().numpy().astype(np.float64), ad.cpu().numpy().astype(np.float64)
    obj.free()
    e = rel(fw, ops.radonapr(f.astype(np.float64), 1.0)), rel(ad, ops.radonapradj(g.astype(np.float64), 1.0))
    assert max(e) < OP_TOL, e
    a, b = float(np.vdot(fw, g)), float(np.vdot(f, ad))
    assert abs(a - b) < DOT_TOL * np.linalg.norm(fw) * np.linalg.norm(g), (a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [3, 8, 16])  # FP32 scatter, tensor-core scatter of half and whole sample groups
@pytest.mark.parametrize("n", WIDTHS)
def test_per_ray(lib_built, torch_cuda, monkeypatch, n, m):
    monkeypatch.setenv("RECTV_DIRS", "0")
    _check(torch_cuda, n, m, 2, 96, 4, False)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [n for n in WIDTHS if n % 2 == 0])
def test_directions(lib_built, torch_cuda, monkeypatch, n):
    monkeypatch.delenv("RECTV_DIRS", raising=False)
    _check(torch_cuda, n, 8, 2, 96, 4, True)


@pytest.mark.gpu
@pytest.mark.parametrize("dirs", ["0", "1"])
def test_reconstruction(lib_built, torch_cuda, monkeypatch, dirs):
    from rectv_gpu_gb300 import Solver
    from rectv_gpu_gb300.phantom import add_noise, phantom4d
    monkeypatch.setenv("RECTV_DIRS", dirs)
    n, ntheta, m, nz, nrot = 50, 45, 5, 1, 3
    theta, phi = scan_angles(ntheta, nrot), _phi(ntheta, m, 2)
    ops = orc.Operators(n, ntheta, m, theta, phi, n / 2)
    g = add_noise(ops.radonapr(phantom4d(n, nz, m, ntheta, seed=1).astype(np.float64)), 0.01, 1)
    ref, hist = orc.run(g, theta, phi, n / 2, 4e-3, 4.0, 3, 3, nz, return_history=True)
    with Solver(n, ntheta, m, nz, nz, 1) as slv:
        slv.set_verbose(False)
        got = slv.recon(g, theta, phi, lambda0=1e-3, lambda1=4.0, niter=3, titer=3)
        h = slv.history()
    assert rel(got, ref) < 1e-4, rel(got, ref)
    assert np.allclose(h["rho"], [x["rho"] for x in hist])


@pytest.mark.parametrize("n", [34, 42, 50, 98, 106])
def test_widths_of_2_mod_8_share_directions(lib_built, n):
    from rectv_gpu_gb300 import plan_directions
    assert plan_directions(scan_angles(64, 8), n)[0] == 8
