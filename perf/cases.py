"""Performance cases of the 4D tomography framework.

Each case is one pass through a public entry point as a user's program calls
it: a whole reconstruction on host arrays (``Solver.recon``), outer iterations
of a device-resident session (``setup_device`` / ``iterate`` /
``result_device``), the forward and adjoint operators on device arrays, the
filtered backprojection, the detector-frame ingest, and the allocation-free
shrink step.  Sizes are those of the repository's own configurations and
tests (the reference's foam and tao scans, the benchmark's geometry, the
oracle's golden configuration) with fewer slices where a whole volume would
not fit the card several times; ``draw`` spreads the same families over their
ranges, ragged sizes among them.

Inputs: sinograms are the line integrals of seeded moving ellipsoids at each
projection's own time (the object the temporal model describes) with 1 %
Gaussian noise; volumes are such ellipsoids rasterised at the m time samples
with 1 % noise; frames are uint16 counts of an attenuated beam.

``exact`` evaluates the same quantities in 64 bits with plain torch.
"""

import ctypes
import math

import numpy as np
import torch

from rectv_gpu_gb300 import _lib, Solver, rectv, takephi
from rectv_gpu_gb300.ingest import preprocess

LAMBDA0, LAMBDA1 = 1e-3, 4.0  # regularisation of the benchmark and of the golden configuration
PI_USFFT = 3.1415926535       # the transform's own constant (kernels_radonusfft.cuh:1)
GATHER_FLOPS = 81 * 4         # one complex sample: 81 taps, two multiply-adds each

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def _session(name, n, ntheta, m, nz, nzp, nrot, cal, niter):
    return dict(name=name, kind="session", n=n, ntheta=ntheta, m=m, nz=nz, nzp=nzp, nrot=nrot, cal=cal,
                titer=4, niter=niter)


def listed():
    return [
        # the ADMM end-of-iteration step on a caller's own small buffers: the smallest call, launch latency
        dict(name="shrink 64", kind="shrink", n=64, m=8, nzp=8, nchunks=1),
        # a whole small reconstruction on host arrays (the golden configuration): many short launches
        dict(name="recon 64", kind="recon", n=64, ntheta=256, m=8, nz=8, nzp=8, nrot=4, cal=1.0, titer=4, niter=32),
        # a preview reconstruction on host arrays: copies, set-up and a few iterations
        dict(name="recon 256", kind="recon", n=256, ntheta=720, m=16, nz=16, nzp=8, nrot=8, cal=1.0, titer=4,
             niter=4),
        # the foam scan (n = 504, 8 time samples, angles that return every half-turn)
        _session("foam 504", 504, 2400, 8, 16, 8, 8, 1.0, 2),
        # the tao scan (n = 480, measured angles with a calibration factor: no direction repeats), 8 of its slices
        _session("tao 480", 480, 1440, 16, 8, 8, 16, 0.9977, 1),
        # the 512 configuration (two of its four chunks)
        _session("iterate 512", 512, 1440, 16, 16, 8, 8, 1.0, 2),
        # the benchmark's geometry, one chunk of its four: the largest
        _session("iterate 1024", 1024, 2880, 16, 16, 16, 8, 1.0, 2),
        # a dynamic scan with few time samples
        _session("few samples 256", 256, 720, 4, 8, 8, 4, 1.0, 2),
        # forward projection of a time-resolved volume (simulation, residual checks), odd number of slices
        dict(name="forward 1024", kind="forward", n=1024, ntheta=2880, m=16, nz=3, nzp=3, nrot=8, cal=1.0),
        # backprojection with the adjoint (gradient of the data term)
        dict(name="adjoint 1024", kind="adjoint", n=1024, ntheta=2880, m=16, nz=3, nzp=3, nrot=8, cal=1.0),
        # filtered backprojection of a stack of sinograms on host arrays (previews, warm starts)
        dict(name="fbp 512", kind="fbp", n=512, ntheta=1440, m=8, nz=8, nzp=8, nrot=8, cal=1.0),
        # detector frames to sinograms: uint16 host frames with dark and flat fields
        dict(name="ingest 480", kind="ingest", n=480, ntheta=1440, nz=16, nflat=10, ndark=10, u16=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed families: sizes over the logarithm of their
    ranges, detector widths even (any even number, powers of two now and then),
    odd numbers of angles, time samples and slices among them."""
    kind = rng.choice(["session", "session", "session", "recon", "recon", "forward", "adjoint", "fbp", "ingest",
                       "shrink"])
    if kind == "shrink":
        return dict(kind=kind, n=2 * _log(rng, 16, 256), m=rng.randint(1, 20), nzp=rng.randint(1, 16),
                    nchunks=rng.randint(1, 2))
    if kind == "ingest":
        return dict(kind=kind, n=_log(rng, 64, 1024), ntheta=_log(rng, 32, 720), nz=_log(rng, 2, 24),
                    nflat=rng.randint(1, 12), ndark=rng.randint(1, 12), u16=rng.random() < 0.7)
    # detector width: powers of two, round sizes, any even size
    shape = rng.random()
    if shape < 0.35:
        n = 2 ** rng.randint(6, 10)
    elif shape < 0.7:
        n = 8 * _log(rng, 8, 128)
    else:
        n = 2 * _log(rng, 24, 512)
    m = rng.choice([8, 16, 16, 16, rng.randint(1, 7), rng.randint(9, 20)])
    nrot = rng.choice([4, 8, 8, 16])
    # multi-rotation scans (angles return each half-turn) or calibrated angles (they do not)
    cal = 1.0 if rng.random() < 0.7 else round(rng.uniform(0.99, 0.9995), 4)
    per = _log(rng, max(8, n // 8), max(9, (3 * n) // 8))  # angles per half-turn
    ntheta = min(2880, per * nrot + (rng.randint(0, 3) if cal != 1.0 else 0))
    if cal == 1.0:
        ntheta -= ntheta % nrot
    # slices: up to the work of the largest listed case
    most = max(1, int(16 * (1024 / n) ** 2 * (16 / m) / 2))
    nzp = rng.randint(1, min(8, most))
    nz = nzp * rng.randint(1, max(1, min(4, most // nzp)))
    c = dict(kind=kind, n=n, ntheta=ntheta, m=m, nz=nz, nzp=nzp, nrot=nrot, cal=cal)
    if kind in ("forward", "adjoint", "fbp"):
        c["nz"] = c["nzp"] = min(nz, 8, max(1, int(3 * (1024 / n) ** 2)))
    else:
        c["titer"] = rng.choice([2, 4, 4])
        c["niter"] = rng.randint(1, 2) if kind == "session" else rng.randint(1, 4)
    if kind == "recon" and n * n * m * nz > 16 * 16 * 512 * 512:  # host volumes of at most 256 MB
        c["nz"] = c["nzp"] = max(1, (16 * 16 * 512 * 512) // (n * n * m * 2))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _theta(c):
    a = np.linspace(0, c["nrot"] * np.pi, c["ntheta"], endpoint=False) * c["cal"]
    return a.astype(np.float32)


def _phi(c):
    n2, m = c["ntheta"], c["m"]
    if n2 % 2 == 0 and m % 2 == 0:
        return takephi(n2, m)
    # the same Fourier basis for odd counts
    k = np.arange(n2) - n2 // 2
    i = np.arange(m) - m // 2
    a = 2 * np.pi * np.outer(i, k) / n2
    phi = np.zeros((m, 2 * n2), np.float32)
    phi[:, ::2] = np.cos(a) / np.sqrt(n2)
    phi[:, 1::2] = np.sin(a) / np.sqrt(n2)
    return phi


def _ellipsoids(n, nz, seed):
    """Ten seeded moving ellipsoids: centre (z, y, x), semi-axes, density,
    in-plane angle, displacement (y, x) over the scan."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(10):
        c0 = rng.uniform(-0.3, 0.3, 3) * np.array([nz, n, n])
        ax = np.maximum(rng.uniform(0.05, 0.3, 3) * np.array([max(nz, 8), n, n]), 0.75)
        d = rng.normal(size=2)
        out.append((c0, ax, rng.uniform(0.1, 1.0), rng.uniform(0, np.pi),
                    d / (np.linalg.norm(d) + 1e-12) * rng.uniform(0, 0.1 * n)))
    return out


def _noise(g, seed, dev):
    gen = torch.Generator(device=dev).manual_seed(int(seed) + 7)
    return g + 0.01 * g.abs().max() * torch.randn(g.shape, generator=gen, device=dev, dtype=torch.float32)


def _sinograms(c, seed, dev="cuda"):
    """g [nz, ntheta, n] float32 on the device: line integrals at each
    projection's own time, in the operator's scale."""
    n, nz, nt = c["n"], c["nz"], c["ntheta"]
    th = torch.as_tensor(_theta(c), device=dev, dtype=torch.float32)[:, None]
    frac = (torch.arange(nt, device=dev, dtype=torch.float32) / nt)[:, None]
    s = (torch.arange(n, device=dev, dtype=torch.float32) - n // 2)[None, :]
    g = torch.zeros((nz, nt, n), device=dev)
    for c0, ax, dens, ang, disp in _ellipsoids(n, nz, seed):
        cy, cx = float(c0[1]) + frac * float(disp[0]), float(c0[2]) + frac * float(disp[1])
        sn, cs = torch.sin(th), torch.cos(th)
        d = s - (cx * sn + cy * cs)
        ca, sa = math.cos(ang), math.sin(ang)
        r2 = (float(ax[2]) * (ca * sn - sa * cs)) ** 2 + (float(ax[1]) * (sa * sn + ca * cs)) ** 2
        for z in range(nz):
            h = 1.0 - ((z - nz / 2 + 0.5 - float(c0[0])) / float(ax[0])) ** 2
            if h <= 0:
                continue
            k2 = r2 * h  # semi-axes of the slice's ellipse shrink with sqrt(h)
            g[z] += 2 * dens * h * float(ax[1] * ax[2]) * torch.sqrt(torch.clamp(k2 - d * d, min=0)) / k2
    return _noise(g * math.sqrt(c["m"] / (n * nt)), seed, dev).contiguous()


def _volume(c, seed, dev="cuda"):
    """u [nz, m, n, n] float32 on the device: the ellipsoids at the m time samples."""
    n, nz, m = c["n"], c["nz"], c["m"]
    x = torch.arange(n, dtype=torch.float32, device=dev) - n / 2 + 0.5
    z = (torch.arange(nz, dtype=torch.float32, device=dev) - nz / 2 + 0.5).view(nz, 1, 1)
    u = torch.zeros((nz, m, n, n), device=dev)
    for c0, ax, dens, ang, disp in _ellipsoids(n, nz, seed):
        ca, sa = math.cos(ang), math.sin(ang)
        for j in range(m):
            dy = (x - (float(c0[1]) + j / m * float(disp[0]))).view(1, n, 1)
            dx = (x - (float(c0[2]) + j / m * float(disp[1]))).view(1, 1, n)
            inside = ((z - float(c0[0])) / float(ax[0])) ** 2 + ((ca * dy - sa * dx) / float(ax[1])) ** 2 + \
                ((sa * dy + ca * dx) / float(ax[2])) ** 2 <= 1.0
            u[:, j] += dens * inside
    return _noise(u, seed, dev).contiguous()


def _frames(c, seed):
    """uint16 or float32 detector frames [ntheta, nz, n], dark and flat fields."""
    rng = np.random.default_rng(seed)
    n, nz, nt = c["n"], c["nz"], c["ntheta"]
    beam = 20000.0 * (0.8 + 0.2 * np.cos(np.linspace(-1, 1, n)))[None, :] * np.ones((nz, 1))
    dark = rng.integers(90, 110, (c["ndark"], nz, n))
    flat = beam[None] + 100 + rng.integers(-100, 100, (c["nflat"], nz, n))
    absorb = np.exp(-rng.uniform(0.05, 2.0, (nt, 1, 1)) * np.exp(-np.linspace(-2, 2, n) ** 2)[None, None, :])
    data = beam[None] * absorb + 100 + rng.integers(-60, 60, (nt, nz, n))
    t = np.uint16 if c["u16"] else np.float32
    return tuple(np.ascontiguousarray(a).astype(t) for a in (data, dark, flat))


def _shrink_inputs(c, seed):
    n, m, nz = c["n"], c["m"], c["nzp"] * c["nchunks"]
    cc = dict(n=n, m=m, nz=nz)
    u = _volume(cc, seed)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 99)
    old = u + 0.02 * torch.randn(u.shape, generator=gen, device="cuda")
    gp = (n + 1) * (n + 1) * (m + 1) * (c["nzp"] + 1) * c["nchunks"]
    mu = 2e-3 * torch.randn(4 * gp, generator=gen, device="cuda")
    return u, old, mu


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "ingest":
        return dict(kind=k, frames=_frames(c, seed))
    if k == "shrink":
        u, old, mu = _shrink_inputs(c, seed)
        st = dict(kind=k, case=c, u=u, old=old, mu=mu, psi=torch.empty_like(mu),
                  sums=torch.zeros(3, dtype=torch.float64, device="cuda"))
        torch.cuda.synchronize()
        return st
    theta, phi, n = _theta(c), _phi(c), c["n"]
    dims = (n, c["ntheta"], c["m"], c["nz"], c["nzp"], 1)
    if k in ("recon", "fbp"):
        slv = Solver(*dims)
        slv.set_verbose(False)
        return dict(kind=k, case=c, slv=slv, theta=theta, phi=phi, g=_sinograms(c, seed).cpu().numpy())
    obj = rectv(*dims)
    obj.set_verbose(False)
    st = dict(kind=k, case=c, obj=obj, theta=torch.from_numpy(theta).cuda(), phi=torch.from_numpy(phi).cuda())
    shape = (c["nz"], c["m"], n, n)
    if k == "session":
        st["g"] = _sinograms(c, seed)
        st["f"] = torch.empty(shape, device="cuda")
    elif k == "forward":
        st["f"] = _volume(c, seed)
        st["g"] = torch.empty((c["nz"], c["ntheta"], n), device="cuda")
    else:
        st["g"] = _sinograms(c, seed)
        st["f"] = torch.empty(shape, device="cuda")
        st["stream"] = torch.cuda.ExternalStream(obj.stream)
    torch.cuda.synchronize()
    # the handle keeps the geometry of the scan
    obj.op_set_geometry(st["theta"].data_ptr(), st["phi"].data_ptr(), n / 2)
    return st


def run(state):
    st, k = state, state["kind"]
    if k == "ingest":
        return preprocess(*st["frames"])
    c = st["case"]
    if k == "shrink":
        def p(t):
            return ctypes.c_void_p(t.data_ptr())
        _lib.check(_lib.load().rectv_shrink_noalloc(
            p(st["u"]), p(st["old"]), p(st["psi"]), p(st["mu"]), c["n"], c["m"], c["nzp"], c["nchunks"], 0.5,
            LAMBDA0 * LAMBDA1, LAMBDA1, p(st["sums"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return {"psi": st["psi"], "mu": st["mu"], "sums": st["sums"]}
    if k == "recon":
        return st["slv"].recon(st["g"], st["theta"], st["phi"], lambda0=LAMBDA0, lambda1=LAMBDA1, niter=c["niter"],
                               titer=c["titer"])
    if k == "fbp":
        return st["slv"].fbp(st["g"], st["theta"])
    obj = st["obj"]
    if k == "session":
        obj.setup_device(st["g"].data_ptr(), st["theta"].data_ptr(), st["phi"].data_ptr(), c["n"] / 2,
                         LAMBDA0 * LAMBDA1, LAMBDA1, c["titer"])
        obj.iterate(c["niter"])
        obj.result_device(st["f"].data_ptr())
        return st["f"]
    if k == "forward":
        obj.op_radonapr(st["g"].data_ptr(), st["f"].data_ptr(), c["nz"], 1.0)
        return st["g"]
    with torch.cuda.stream(st["stream"]):  # the operator adds into f on the handle's stream
        st["f"].zero_()
    obj.op_radonapradj(st["f"].data_ptr(), st["g"].data_ptr(), c["nz"], 1.0)
    return st["f"]


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------


def _transform_work(n, ntheta, m, nz, nrot, cal):
    """(bytes, flops) of one forward or adjoint transform: volume and data once,
    the half-plane spectra written and read once; padded 2D FFTs, row FFTs,
    the interpolation of every distinct position."""
    P = 2 * n
    dirs = -(-ntheta // nrot) if cal == 1.0 else ntheta
    b = 4.0 * n * n * m * nz + 4.0 * n * ntheta * nz + 2 * 8.0 * P * (n + 1) * m * nz
    f = m * nz * (n / 2 + n + 1) * 5.0 * P * math.log2(P) + nz * ntheta * 2.5 * n * math.log2(n)
    return b, f + GATHER_FLOPS * float(dirs) * n * m * nz + 8.0 * ntheta * n * m * nz


def work(case):
    c, k = case, case["kind"]
    if k == "ingest":
        e = 2 if c["u16"] else 4
        px = c["nz"] * c["n"]
        return {"bytes": px * (e * (c["ntheta"] + c["nflat"] + c["ndark"]) + 4.0 * c["ntheta"]),
                "flops": px * 4.0 * c["ntheta"]}
    if k == "shrink":
        gp = float((c["n"] + 1) ** 2 * (c["m"] + 1) * (c["nzp"] + 1) * c["nchunks"])
        u = float(c["n"] ** 2 * c["m"] * c["nzp"] * c["nchunks"])
        return {"bytes": 8 * u + 48 * gp, "flops": 80 * gp}
    n, m, nz = c["n"], c["m"], c["nz"]
    if k == "fbp":  # one static image per slice
        b, f = _transform_work(n, c["ntheta"], 1, nz, c["nrot"], c["cal"])
        return {"bytes": b, "flops": f}
    b, f = _transform_work(n, c["ntheta"], m, nz, c["nrot"], c["cal"])
    if k in ("forward", "adjoint"):
        return {"bytes": b, "flops": f}
    U = float(n * n * m * nz)
    gp = float((n + 1) ** 2 * (m + 1) * (c["nzp"] + 1) * (nz // c["nzp"]))
    # inner step: both transforms, u in and out with one dual array read; outer step: shrink and dual update
    inner = 2 * b + 4.0 * U + 16 * gp
    return {"bytes": c["niter"] * (c["titer"] * inner + 8 * U + 48 * gp),
            "flops": c["niter"] * (c["titer"] * (2 * f + 60 * U) + 80 * gp)}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
F64, C128 = torch.float64, torch.complex128


class _Radon64:
    """The temporal-basis Radon transform and its adjoint in float64: padded
    FFT of every time sample, 9x9 Gaussian interpolation at the polar points,
    mixing over the time samples, row FFT."""

    def __init__(self, n, ntheta, m, theta, phi, center, dev):
        self.n, self.ntheta, self.m, self.dev = n, ntheta, m, dev
        P = self.P = 2 * n
        mu = float(np.float32(-math.log(float(np.float32(1e-3))) / (2.0 * n * n)))
        th = torch.as_tensor(theta, device=dev).to(F64)
        q = (torch.arange(n, device=dev, dtype=F64) - n // 2) / n
        pos = []
        for v in (torch.sin(th)[:, None] * q, torch.cos(th)[:, None] * q):
            v = torch.where(v >= 0.5, torch.full_like(v, 0.5 - 1e-5), v)
            pos.append(v[:, 1:].reshape(-1))  # sample k = 0 is never used
        self.ix, self.w = [], []
        for v in pos:
            f = torch.floor(2 * n * v)
            taps = [f + i for i in range(-4, 5)]
            self.ix.append([torch.remainder(t.long() + n, P) for t in taps])
            self.w.append([torch.exp(-PI_USFFT ** 2 / mu * (t / P - v) ** 2) for t in taps])
        self.cw = PI_USFFT / mu / n
        k = torch.arange(n, device=dev, dtype=F64)
        self.sgn = 1.0 - 2.0 * ((k + 1) % 2)  # (-1)^(k+1)
        self.shift = torch.exp(-2j * PI_USFFT * (center - n / 2) * (k - n / 2) / n)
        x = k - n // 2
        d = torch.exp(mu * x * x)
        self.deapod = d[:, None] * d[None, :] / (4.0 * n * n)
        X = torch.arange(P, device=dev)
        self.mod2 = (1.0 - 2.0 * ((X[:, None] + X[None, :]) % 2)).to(F64)
        self.scale = 1.0 / math.sqrt(float(n) * ntheta)
        if phi is not None:
            ph = torch.complex(torch.as_tensor(phi[:, ::2], device=dev).to(F64),
                               torch.as_tensor(phi[:, 1::2], device=dev).to(F64))
            tj = torch.as_tensor((np.arange(m) * ntheta) // m, device=dev)
            self.K = ntheta / math.sqrt(m) * torch.einsum("it,ij->tj", ph, torch.conj(ph[:, tj]))

    def _slices(self, nz):
        per = max(1, int(6e9 / (self.P * self.P * self.m * 16.0)))  # slices per group of images
        return [slice(z, min(nz, z + per)) for z in range(0, nz, per)]

    def forward(self, u):
        g = torch.empty((u.shape[0], self.ntheta, self.n), dtype=F64, device=self.dev)
        for s in self._slices(u.shape[0]):
            g[s] = self._forward(u[s])
        return g

    def _forward(self, u):
        n, P, nt, m = self.n, self.P, self.ntheta, self.m
        nz = u.shape[0]
        a = torch.zeros((nz * m, P, P), dtype=F64, device=self.dev)
        h = n // 2
        a[:, h:h + n, h:h + n] = u.reshape(nz * m, n, n) * self.deapod
        F = torch.fft.fft2(a * self.mod2) * self.mod2
        Z = torch.view_as_real(F.reshape(nz * m, P * P).t().contiguous()).reshape(P * P, -1)
        del a, F
        npts = nt * (n - 1)
        S = torch.zeros((npts, Z.shape[1]), dtype=F64, device=self.dev)
        for lo in range(0, npts, 1 << 19):
            r = slice(lo, min(npts, lo + (1 << 19)))
            for b in range(9):
                row = self.ix[1][b][r] * P
                for c in range(9):
                    S[r].addcmul_(Z.index_select(0, row + self.ix[0][c][r]), (self.w[0][c][r] * self.w[1][b][r])[:, None])
        del Z
        S = torch.view_as_complex(S.reshape(nt, n - 1, nz, m, 2)) * self.cw
        rows = torch.zeros((nz, nt, n), dtype=C128, device=self.dev)
        rows[:, :, 1:] = torch.einsum("tkzj,tj->ztk", S, self.K)
        return (torch.fft.ifft(rows * self.shift * self.sgn) * n * self.sgn * self.scale).real

    def adjoint(self, g, filt=None):
        f = torch.empty((g.shape[0], self.m, self.n, self.n), dtype=F64, device=self.dev)
        for s in self._slices(g.shape[0]):
            f[s] = self._adjoint(g[s], filt)
        return f

    def _adjoint(self, g, filt):
        n, P, nt, m = self.n, self.P, self.ntheta, self.m
        nz = g.shape[0]
        E = torch.fft.fft((g * self.sgn).to(C128)) * self.sgn * torch.conj(self.shift) * self.cw
        if filt is not None:
            E = E * filt
        E = torch.view_as_real(E[:, :, 1:].permute(1, 2, 0).contiguous())  # [t, k, z, 2]
        E = torch.view_as_complex(E)
        npts = nt * (n - 1)
        Z = torch.zeros((P * P, nz * m * 2), dtype=F64, device=self.dev)
        per = max(1, (1 << 19) // (n - 1))
        for t0 in range(0, nt, per):
            t1 = min(nt, t0 + per)
            r = slice(t0 * (n - 1), min(npts, t1 * (n - 1)))
            if filt is None:
                v = E[t0:t1, :, :, None] * torch.conj(self.K[t0:t1])[:, None, None, :]
            else:
                v = E[t0:t1, :, :, None]
            v = torch.view_as_real(v.contiguous()).reshape(-1, nz * m * 2)
            for b in range(9):
                row = self.ix[1][b][r] * P
                for c in range(9):
                    Z.index_add_(0, row + self.ix[0][c][r], v * (self.w[0][c][r] * self.w[1][b][r])[:, None])
        F = torch.view_as_complex(Z.reshape(P, P, nz * m, 2)).permute(2, 0, 1).contiguous()
        del Z
        a = torch.fft.ifft2(F * self.mod2).real * float(P * P) * self.mod2
        h = n // 2
        return (a[:, h:h + n, h:h + n] * self.deapod * self.scale).reshape(nz, m, n, n)


def _gradient64(fm, lo, hi, l1):
    """Forward differences of the chunk fm [nzp + 2, m, n, n] (halo slabs used when lo / hi) on the dual grid."""
    nzp, m, n = fm.shape[0] - 2, fm.shape[1], fm.shape[2]
    dev = fm.device
    ix = torch.clamp(torch.arange(n + 2, device=dev) - 1, 0, n - 1)
    it = torch.clamp(torch.arange(m + 2, device=dev) - 1, 0, m - 1)
    iz = torch.clamp(torch.arange(nzp + 2, device=dev) - 1, -lo, nzp - 1 + hi) + 1
    e = fm[iz][:, it][:, :, ix][:, :, :, ix]
    s = 1.0 / (2.0 * 2.0 ** (1 / 3) * (l1 / 2.0))
    b = e[:-1, :-1, :-1, :-1]
    return torch.stack([(e[:-1, :-1, :-1, 1:] - b) * s, (e[:-1, :-1, 1:, :-1] - b) * s,
                        (e[:-1, 1:, :-1, :-1] - b) * s * l1, (e[1:, :-1, :-1, :-1] - b) * s])


def _divergence64(h, l1):
    s = 1.0 / (4.0 * 2.0 ** (1 / 3) * (l1 / 2.0))
    c = h[:, 1:, 1:, 1:, 1:]
    return s * ((h[0, 1:, 1:, 1:, :-1] - c[0]) + (h[1, 1:, 1:, :-1, 1:] - c[1]) +
                l1 * (h[2, 1:, :-1, 1:, 1:] - c[2]) + (h[3, :-1, 1:, 1:, 1:] - c[3]))


def _shrink64(h, mu, lam0, rho):
    p = h + mu / rho
    za = torch.sqrt((p * p).sum(0, keepdim=True))
    thr = lam0 / rho
    return torch.where(za <= thr, torch.zeros_like(p), p * (1 - thr / torch.where(za > 0, za, torch.ones_like(za))))


def _halo(u, old, z0, nzp, nz):
    fm = torch.zeros((nzp + 2,) + u.shape[1:], dtype=F64, device=u.device)
    fm[1:-1] = u[z0:z0 + nzp]
    lo, hi = int(z0 > 0), int(z0 + nzp < nz)
    if lo:
        fm[0] = old[z0 - 1]
    if hi:
        fm[-1] = old[z0 + nzp]
    return fm, lo, hi


def _admm64(c, g, theta, phi, dev):
    n, m, nzp = c["n"], c["m"], c["nzp"]
    nz = (c["nz"] // nzp) * nzp
    lam0, l1 = LAMBDA0 * LAMBDA1, LAMBDA1
    R = _Radon64(n, c["ntheta"], m, theta, phi, n / 2, dev)
    g = g.to(F64)
    f = torch.zeros((c["nz"], m, n, n), dtype=F64, device=dev)
    psi = [torch.zeros((4, nzp + 1, m + 1, n + 1, n + 1), dtype=F64, device=dev) for _ in range(nz // nzp)]
    mu = [torch.zeros_like(p) for p in psi]
    rho = 0.5
    for _ in range(c["niter"]):
        new, rs, ss = f.clone(), 0.0, 0.0
        for i in range(nz // nzp):
            fm, lo, hi = _halo(f, f, i * nzp, nzp, nz)
            h0 = _gradient64(fm, lo, hi, l1)
            for _ in range(c["titer"]):
                h = rho * (_gradient64(fm, lo, hi, l1) - psi[i]) + mu[i]
                d = _divergence64(h, l1)
                del h
                d += R.adjoint(R.forward(fm[1:-1]) - g[i * nzp:(i + 1) * nzp])
                fm[1:-1] -= 0.5 * d
                del d
            h = _gradient64(fm, lo, hi, l1)
            psi[i] = _shrink64(h, mu[i], lam0, rho)
            mu[i] = mu[i] + rho * (h - psi[i])
            rs += float(((h - psi[i]) ** 2).sum())
            ss += float(((h0 - h) ** 2).sum()) * rho * rho
            new[i * nzp:(i + 1) * nzp] = fm[1:-1]
            del h, h0, fm
        f = new
        rho = rho * 2 if rs > 10 * ss else (rho * 0.5 if ss > 10 * rs else rho)
    return f


def _slow(c):
    """Whether the 64-bit reconstruction takes more than about 20 seconds."""
    steps = c["niter"] * c["titer"]
    return steps * (3.0 * c["ntheta"] * c["n"] + 4.0 * c["n"] ** 2) * c["m"] * c["nz"] > 3e10


def exact(case, seed):
    c, k = case, case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if k == "ingest":
        data, dark, flat = (a.astype(np.float64) for a in _frames(c, seed))
        d = dark.mean(0)
        return np.ascontiguousarray((-np.log((data - d) / (1e-3 + flat.mean(0) - d))).swapaxes(0, 1))
    if k == "shrink":
        u, old, mu = (a.to(F64) for a in _shrink_inputs(c, seed))
        n, m, nzp, nch = c["n"], c["m"], c["nzp"], c["nchunks"]
        rho, lam0 = 0.5, LAMBDA0 * LAMBDA1
        mu = mu.reshape(4, nch, nzp + 1, m + 1, n + 1, n + 1)
        psi, out, sums = torch.empty_like(mu), torch.empty_like(mu), torch.zeros(3, dtype=F64, device=mu.device)
        for i in range(nch):
            fm, lo, hi = _halo(u, old, i * nzp, nzp, nzp * nch)
            h = _gradient64(fm, lo, hi, LAMBDA1)
            fo, lo, hi = _halo(old, old, i * nzp, nzp, nzp * nch)
            ho = _gradient64(fo, lo, hi, LAMBDA1)
            psi[:, i] = _shrink64(h, mu[:, i], lam0, rho)
            out[:, i] = mu[:, i] + rho * (h - psi[:, i])
            sums += torch.stack([((h - psi[:, i]) ** 2).sum(), ((ho - h) ** 2).sum(),
                                 ((fm[1:-1] - fo[1:-1]) ** 2).sum()])
        return {"psi": psi.reshape(-1), "mu": out.reshape(-1), "sums": sums}
    theta, n = _theta(c), c["n"]
    if k == "fbp":
        R = _Radon64(n, c["ntheta"], 1, theta, None, n / 2, dev)
        r = (torch.arange(n, dtype=F64, device=dev) - n // 2) / n
        w = torch.where(r == 0, torch.zeros_like(r), 4 * n * torch.sin(r.abs()))
        f = R.adjoint(_sinograms(c, seed, dev).to(F64), w)[:, 0] * (PI_USFFT / 4)
        return f * (4 * r[None, :] ** 2 + 4 * r[:, None] ** 2 < 1)
    if k in ("session", "recon"):
        if _slow(c):
            return None
        return _admm64(c, _sinograms(c, seed, dev), theta, _phi(c), dev)
    R = _Radon64(n, c["ntheta"], c["m"], theta, _phi(c), n / 2, dev)
    if k == "forward":
        return R.forward(_volume(c, seed, dev).to(F64))
    return R.adjoint(_sinograms(c, seed, dev).to(F64))
