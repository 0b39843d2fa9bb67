"""A slice's results do not depend on its neighbours' values: with a slice made
10000 times brighter, or one value of it NaN, the other slices keep every bit.

The operators act on each slice alone (radonapr / radonapradj of the
reference, src/cuda/operators.cu), and with one slice per chunk so does an
outer iteration from zero (its halos are zero)."""

import numpy as np
import pytest

from rectv_gpu_gb300.phantom import scan_angles

pytestmark = pytest.mark.gpu

# padded-grid FFTs: power of two, mixed radix (even and odd width), cuFFT
WIDTHS = [128, 54, 55, 46]


def _phi(ntheta, m):
    rng = np.random.default_rng(m)
    return (rng.standard_normal((m, 2 * ntheta)) / np.sqrt(ntheta)).astype(np.float32)


def _spoiled(a, z):
    bright, nan = a.clone(), a.clone()
    bright[z] *= 1e4
    nan[z].view(-1)[7] = float("nan")
    return bright, nan


@pytest.mark.parametrize("dirs", ["0", "1"])
@pytest.mark.parametrize("m", [1, 2, 3, 8, 16, 17])
@pytest.mark.parametrize("n", WIDTHS)
def test_operators(lib_built, torch_cuda, monkeypatch, n, m, dirs):
    torch = torch_cuda
    from rectv_gpu_gb300 import rectv
    monkeypatch.setenv("RECTV_DIRS", dirs)
    ntheta, nz, z = 48, 5, 2
    gen = torch.Generator(device="cuda").manual_seed(n + m)
    u = torch.randn((nz, m, n, n), generator=gen, device="cuda")
    g = torch.randn((nz, ntheta, n), generator=gen, device="cuda")
    theta, phi = torch.from_numpy(scan_angles(ntheta, 4)).cuda(), torch.from_numpy(_phi(ntheta, m)).cuda()
    obj = rectv(n, ntheta, m, nz, nz, 1)
    torch.cuda.synchronize()
    obj.op_set_geometry(theta.data_ptr(), phi.data_ptr(), n / 2)

    def ops(uu, gg):
        fw, ad = torch.zeros_like(g), torch.zeros_like(u)
        torch.cuda.synchronize()
        obj.op_radonapr(fw.data_ptr(), uu.data_ptr(), nz, 1.0)
        obj.op_radonapradj(ad.data_ptr(), gg.data_ptr(), nz, 1.0)
        torch.cuda.synchronize()
        return fw, ad

    ref = ops(u, g)
    for us, gs in zip(_spoiled(u, z), _spoiled(g, z)):
        got = ops(us, gs)
        for a, b in zip(got, ref):
            for i in range(nz):
                if i != z:
                    assert torch.equal(a[i], b[i]), i
    obj.free()


@pytest.mark.parametrize("ntheta", [45, 48])  # an odd count: a slice's last row has no partner
@pytest.mark.parametrize("n,m", [(54, 5), (54, 1), (128, 8), (256, 8), (46, 4)])
def test_outer_iteration_of_single_slice_chunks(lib_built, torch_cuda, n, m, ntheta):
    torch = torch_cuda
    from rectv_gpu_gb300 import rectv
    nz, z = 3, 1
    gen = torch.Generator(device="cuda").manual_seed(n)
    g = torch.randn((nz, ntheta, n), generator=gen, device="cuda")
    theta, phi = torch.from_numpy(scan_angles(ntheta, 3)).cuda(), torch.from_numpy(_phi(ntheta, m)).cuda()
    obj = rectv(n, ntheta, m, nz, 1, 1)
    obj.set_verbose(False)

    def run(gg):
        f = torch.empty((nz, m, n, n), device="cuda")
        torch.cuda.synchronize()
        obj.setup_device(gg.data_ptr(), theta.data_ptr(), phi.data_ptr(), n / 2, 4e-3, 4.0, 3)
        obj.iterate(1)
        obj.result_device(f.data_ptr())
        torch.cuda.synchronize()
        return f

    ref = run(g)
    bright, nan = g.clone(), g.clone()
    bright[z] *= 1e4
    nan[z, -1] = float("nan")
    nan[z, 0] = float("nan")
    for gg in (bright, nan):
        got = run(gg)
        for i in (0, 2):
            assert torch.equal(got[i], ref[i]), i
    obj.free()
