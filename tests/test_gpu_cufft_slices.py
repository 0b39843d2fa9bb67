"""Grids on cuFFT: the images of a 2D call are those of the slices there are.

Width 1030 (2n has the prime factor 103): one image takes 16 n (n + 2) bytes."""

import numpy as np
import pytest

from rectv_gpu_gb300.phantom import scan_angles

pytestmark = pytest.mark.gpu
N, NTHETA = 1030, 24


def _operators(torch, m, u, g):
    from rectv_gpu_gb300 import rectv
    nz, n = u.shape[0], u.shape[-1]
    theta = scan_angles(NTHETA, 1)
    phi = np.random.default_rng(m).standard_normal((m, 2 * NTHETA)).astype(np.float32)
    obj = rectv(n, NTHETA, m, nz, nz, 1)
    held = obj.device_bytes()
    th, ph = torch.from_numpy(theta).cuda(), torch.from_numpy(phi).cuda()
    fw, ad = torch.zeros_like(g), torch.zeros_like(u)
    torch.cuda.synchronize()
    obj.op_set_geometry(th.data_ptr(), ph.data_ptr(), n / 2)
    obj.op_radonapr(fw.data_ptr(), u.data_ptr(), nz, 1.0)
    obj.op_radonapradj(ad.data_ptr(), g.data_ptr(), nz, 1.0)
    fw, ad = fw.cpu(), ad.cpu()
    obj.free()
    return fw, ad, held


def test_one_slice_holds_one_slice(lib_built, torch_cuda):
    from rectv_gpu_gb300 import rectv
    img = 16 * N * (N + 2)
    obj, own = rectv(N, NTHETA, 1, 1, 1, 1), rectv(1024, NTHETA, 1, 1, 1, 1)
    held, ref = obj.device_bytes(), own.device_bytes()
    obj.free()
    own.free()
    assert held < 1.05 * ref + 2 * img, (held, ref)  # everything else grows by 2 %


# width 262 (prime factor 131): 3 of 5 slices per call, 12 of 22
@pytest.mark.parametrize("n,m,nz", [(N, 1, 3), (N, 3, 5), (N, 4, 6), (N, 9, 3), (262, 16, 5), (262, 3, 22)])
def test_slices_of_a_call_agree_with_one(lib_built, torch_cuda, n, m, nz):
    """Several calls per batch, the last one partly filled: every slice is what it is alone."""
    torch = torch_cuda
    gen = torch.Generator(device="cuda").manual_seed(m)
    u = torch.randn((nz, m, n, n), generator=gen, device="cuda")
    g = torch.randn((nz, NTHETA, n), generator=gen, device="cuda")
    fw, ad, _ = _operators(torch, m, u, g)
    for z in range(nz):
        f1, a1, _ = _operators(torch, m, u[z:z + 1].contiguous(), g[z:z + 1].contiguous())
        assert float((fw[z] - f1[0]).norm() / f1.norm()) < 1e-6
        assert float((ad[z] - a1[0]).norm() / a1.norm()) < 5e-6
