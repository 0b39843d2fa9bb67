"""Results of more than 4 MB whose pages are faulted in beside the GPU's work
(host_pages.h): the ingest's copy part by part, with frame counts that are no
multiple of the eight frames per thread, and a reconstruction with slices behind
the last chunk."""

import numpy as np
import pytest

from rectv_gpu_gb300.phantom import scan_angles


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint16, np.float32])
@pytest.mark.parametrize("shape", [(1003, 3, 517), (7, 2, 130000), (9, 1, 33)])
def test_ingest_parts(lib_built, dtype, shape):
    """-log((v - d) / w) of FP32 operations on operands within 2^16 and quotients
    above 1/8: five roundings and logf's, 2^-21 absolute."""
    from rectv_gpu_gb300.ingest import preprocess
    rng = np.random.default_rng(1)
    data = rng.integers(6000, 30000, shape).astype(dtype)
    dark = rng.integers(100, 200, (3,) + shape[1:]).astype(dtype)
    flat = rng.integers(30000, 40000, (5,) + shape[1:]).astype(dtype)
    d, f = dark.mean(0, dtype=np.float64), flat.mean(0, dtype=np.float64)
    want = -np.log((data - d) / (1e-3 + f - d)).swapaxes(0, 1)
    assert np.abs(preprocess(data, dark, flat) - want).max() < 2.0 ** -21


@pytest.mark.gpu
def test_reconstruction_result(lib_built, torch_cuda):
    torch = torch_cuda
    from rectv_gpu_gb300 import Solver
    from rectv_gpu_gb300.rectv import rectv
    n, ntheta, m, nz, nzp = 200, 24, 3, 11, 5
    theta = scan_angles(ntheta, 4)
    rng = np.random.default_rng(2)
    phi = (rng.standard_normal((m, 2 * ntheta)) / np.sqrt(ntheta)).astype(np.float32)
    g = rng.random((nz, ntheta, n)).astype(np.float32)
    with Solver(n, ntheta, m, nz, nzp, 1) as slv:
        slv.set_verbose(False)
        got = slv.recon(g, theta, phi, lambda0=1e-3, lambda1=4.0, niter=1, titer=2)
    obj = rectv(n, ntheta, m, nz, nzp, 1)
    obj.set_verbose(False)
    dg, dt, dp = (torch.from_numpy(a).cuda() for a in (g, theta, phi))
    out = torch.zeros((nz, m, n, n), device="cuda")
    torch.cuda.synchronize()
    obj.setup_device(dg.data_ptr(), dt.data_ptr(), dp.data_ptr(), n / 2, 4e-3, 4.0, 2)
    obj.iterate(1)
    obj.result_device(out.data_ptr())
    obj.synchronize()
    obj.free()
    want = out.cpu().numpy()
    want[10:] = 0
    assert np.allclose(got, want, rtol=0, atol=1e-5 * np.abs(want).max())
    assert not got[10:].any()
