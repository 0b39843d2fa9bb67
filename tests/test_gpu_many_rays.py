"""Directions of more rays than the adjoint's mixing takes at a time (64): later
groups of rays add to the stored sums.  Operators against the FP64 oracle at the
suite's bar of 2e-5 relative."""

import numpy as np
import pytest

from oracle import rectv_oracle as orc
from rectv_gpu_gb300.phantom import scan_angles

pytestmark = pytest.mark.gpu
OP_TOL = 2e-5


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("m,nz", [(1, 2), (4, 3), (16, 1), (17, 1)])
@pytest.mark.parametrize("ndir,nrays", [(4, 64), (4, 65), (3, 130)])
def test_operators(lib_built, torch_cuda, ndir, nrays, m, nz):
    torch = torch_cuda
    from rectv_gpu_gb300 import rectv
    n, ntheta = 64, ndir * nrays
    theta = scan_angles(ntheta, nrays)
    rng = np.random.default_rng(m)
    phi = (rng.standard_normal((m, 2 * ntheta)) / np.sqrt(ntheta)).astype(np.float32)
    f = rng.standard_normal((nz, m, n, n)).astype(np.float32)
    g = rng.standard_normal((nz, ntheta, n)).astype(np.float32)
    ops = orc.Operators(n, ntheta, m, theta, phi, n / 2)
    obj = rectv(n, ntheta, m, nz, nz, 1)
    th, ph, df, dg = (torch.from_numpy(a).cuda() for a in (theta, phi, f, g))
    fw, ad = torch.zeros_like(dg), torch.zeros_like(df)
    torch.cuda.synchronize()
    obj.op_set_geometry(th.data_ptr(), ph.data_ptr(), n / 2)
    assert obj.directions() == ndir
    obj.op_radonapr(fw.data_ptr(), df.data_ptr(), nz, 1.0)
    obj.op_radonapradj(ad.data_ptr(), dg.data_ptr(), nz, 1.0)
    fw, ad = fw.cpu().numpy(), ad.cpu().numpy()
    obj.free()
    e = rel(fw, ops.radonapr(f.astype(np.float64), 1.0)), rel(ad, ops.radonapradj(g.astype(np.float64), 1.0))
    assert max(e) < OP_TOL, e
