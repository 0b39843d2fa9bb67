"""The estimate of a problem's device memory against what a handle holds: grids
on cuFFT, grids and rows on the hand-written transforms, one slice, few and
many time samples, and scans that revisit directions (whose mixing buffer the
engine adds from the angles)."""

import numpy as np
import pytest

from rectv_gpu_gb300.phantom import scan_angles
from rectv_gpu_gb300.rectv import estimate_bytes

CASES = [
    # n, ntheta, m, nz, nzp
    (458, 96, 16, 4, 2),    # 2n = 4 * 229: cuFFT
    (1030, 48, 16, 2, 1),   # 2n > 2048
    (1030, 48, 1, 1, 1),    # one slice of one time sample
    (262, 96, 2, 3, 3),     # cuFFT, eight slices per plane
    (262, 640, 9, 4, 4),    # rows larger than the images
    (131, 96, 20, 2, 1),    # odd width, two planes per slice
    (26, 2000, 3, 2, 2),
    (504, 96, 8, 4, 2),
    (128, 96, 16, 4, 2),
    (256, 720, 4, 8, 4),
]


def _phi(ntheta, m):
    rng = np.random.default_rng(ntheta)
    return (rng.standard_normal((m, 2 * ntheta)) / np.sqrt(ntheta)).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("nrot", [1, 8])  # no repeated direction; eight rays per direction
@pytest.mark.parametrize("case", CASES)
def test_engine_estimate_covers_the_handle(lib_built, torch_cuda, case, nrot):
    from rectv_gpu_gb300 import engine
    n, ntheta, m, nz, nzp = case
    g = np.zeros((nz, ntheta, n), np.float32)
    with engine.Engine() as eng:
        i = eng.submit(g, scan_angles(ntheta, nrot), _phi(ntheta, m), nzp=nzp, niter=1, titer=1)
        eng.run()
        info = eng.info(i)
    assert info["status"] == "done", info
    est, held = info["est_bytes"], info["bytes"]
    assert held <= est <= 2 * held + (64 << 20), (est / 1e6, held / 1e6)


def test_cufft_images_are_counted(lib_built):
    """Width 1030: 2n has the prime factor 103, so the padded images of a slice
    (16 n (n + 2) bytes per time sample) and as much work area count."""
    m = 16
    grow = estimate_bytes(1030, 48, m, 1, 1) - estimate_bytes(1024, 48, m, 1, 1)
    assert grow > 2 * m * 16 * 1030 * 1032
