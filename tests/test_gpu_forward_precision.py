"""Rounding of the forward operator on the direction path against its 64-bit
evaluation, on the forward projections of perf/cases.py: no further off than
with whole rows and every position's own stencil (bounds: that form's errors on
these inputs, two seeds each)."""

import importlib.util
import os

import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # n, ntheta, m, nz, errors of the whole-row form at seeds 1 and 2
    (1024, 2880, 16, 3, (2.2451e-07, 2.1222e-07)),
    (504, 2400, 8, 2, (4.2814e-07, 4.2094e-07)),
    (512, 1440, 16, 2, (2.3470e-07, 1.7893e-07)),
]


@pytest.mark.parametrize("n,ntheta,m,nz,bounds", CASES)
def test_forward(lib_built, torch_cuda, n, ntheta, m, nz, bounds):
    torch = torch_cuda
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "perf", "cases.py")
    spec = importlib.util.spec_from_file_location("perf_cases", path)
    cases = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(cases)
    c = dict(kind="forward", n=n, ntheta=ntheta, m=m, nz=nz, nzp=nz, nrot=8, cal=1.0)
    for seed, bound in zip((1, 2), bounds):
        st = cases.prepare(c, seed)
        assert st["obj"].directions() > 0
        g = cases.run(st)
        torch.cuda.synchronize()
        ref = cases.exact(c, seed)
        err = float((g.double() - ref).norm() / ref.norm())
        st["obj"].free()
        assert err < bound, (seed, err, bound)
