"""The per-ray operators where the oversampled grid's side 2n is less than two
tiles: stencils wrap into the tile they start in (widths up to 15), cover the
grid more than once (up to 4), and footprints reach past its second copy (2).

Against the FP64 oracle at the suite's bar of 2e-5 relative."""

import numpy as np
import pytest

from oracle import rectv_oracle as orc

pytestmark = pytest.mark.gpu
OP_TOL = 2e-5


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def _case(torch, n, m):
    from rectv_gpu_gb300 import rectv
    ntheta, nz = 24, 2
    rng = np.random.default_rng(100 * n + m)
    theta = np.sort(rng.uniform(0, np.pi, ntheta)).astype(np.float32)
    phi = (rng.standard_normal((m, 2 * ntheta)) / np.sqrt(ntheta)).astype(np.float32)
    f = rng.standard_normal((nz, m, n, n)).astype(np.float32)
    g = rng.standard_normal((nz, ntheta, n)).astype(np.float32)
    ops = orc.Operators(n, ntheta, m, theta, phi, n / 2)
    obj = rectv(n, ntheta, m, nz, nz, 1)
    th, ph, df, dg = (torch.from_numpy(a).cuda() for a in (theta, phi, f, g))
    fw, ad = torch.zeros_like(dg), torch.zeros_like(df)
    torch.cuda.synchronize()
    obj.op_set_geometry(th.data_ptr(), ph.data_ptr(), n / 2)
    obj.op_radonapr(fw.data_ptr(), df.data_ptr(), nz, 1.0)
    obj.op_radonapradj(ad.data_ptr(), dg.data_ptr(), nz, 1.0)
    fw, ad = fw.cpu().numpy(), ad.cpu().numpy()
    obj.free()
    return (rel(fw, ops.radonapr(f.astype(np.float64), 1.0)), rel(ad, ops.radonapradj(g.astype(np.float64), 1.0)))


@pytest.mark.parametrize("m", [1, 3, 8, 16])
@pytest.mark.parametrize("n", list(range(2, 17)) + [24])
def test_forward(lib_built, torch_cuda, n, m):
    e = _case(torch_cuda, n, m)
    assert e[0] < OP_TOL, e


@pytest.mark.parametrize("m", [1, 3, 8, 16])
@pytest.mark.parametrize("n", list(range(2, 17)) + [24])
def test_adjoint(lib_built, torch_cuda, n, m):
    e = _case(torch_cuda, n, m)
    assert e[1] < OP_TOL, e
