"""Performance cases of the holotomography framework.

Each case is one use of the framework through its public entry points: a
propagation, a Radon transform or its adjoint, a filtered back-projection, a
B-spline shift or back-projection, the differentiable data term with its
backward pass, and whole Bilinear-Hessian reconstructions (holotomography and
near-field ptychography).  ``listed()`` gives the fixed cases, ``draw(rng)``
one more of the same ranges.  Sizes are those of the repository's benchmark,
tests and serving workload, and odd ones between them.

``exact`` restates the operators in 64 bits with plain torch.
"""
import math
import types

import numpy as np
import torch

from holotomocupy_b200 import Propagation, Rec, RecNFP, Shift, Tomo
from holotomocupy_b200.autograd import DataFidelity

WAVELENGTH, VOXEL = 7.3e-11, 20e-9
DISTANCES = (3e-3, 4e-3, 5e-3, 6e-3)
MASK = 0.9
RHO = (1, 0.05, 0.02)      # variable scalings of obj, prb, pos
NFP_RHO = (1, 0.5, 0.1)    # of proj, prb, pos
DEV = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one small field through the propagator, as an interactive script or a probe update calls it:
        # three launches and their latency
        {"name": "prop_128", "kind": "prop", "n": 128, "nz": 128, "batch": 1, "adjoint": False},
        # a chunk of large-detector images through the propagator
        {"name": "prop_2048", "kind": "prop", "n": 2048, "nz": 2048, "batch": 16, "adjoint": False},
        # projections of a slab of the 512^3 volume at all 900 angles
        {"name": "radon_512", "kind": "radon", "op": "R", "n": 512, "nz": 64, "ntheta": 900, "real": False},
        # back-projection of a ragged last slab at a size that is not a power of two
        {"name": "radon_adj_384", "kind": "radon", "op": "RT", "n": 384, "nz": 37, "ntheta": 671, "real": False},
        # a few slices of the large-detector volume
        {"name": "radon_2048", "kind": "radon", "op": "R", "n": 2048, "nz": 20, "ntheta": 1800, "real": False},
        # conventional reconstruction of real phase projections
        {"name": "fbp_256", "kind": "radon", "op": "fbp", "n": 256, "nz": 250, "ntheta": 361, "real": True},
        # a stack of real coefficient images resampled onto an odd detector (prefilter and stencil)
        {"name": "shift_real", "kind": "shift", "op": "S", "n": 450, "nz": 501, "npsi": 512, "nzpsi": 512,
         "batch": 90, "real": True},
        # the single-distance initial guess: images of one magnification spread onto the object grid
        {"name": "sback_512", "kind": "sback", "n": 512, "nz": 512, "npsi": 512, "nzpsi": 512, "batch": 128,
         "mag": 0.8},
        # the differentiable data term and its gradients, angles in two chunks
        {"name": "fidelity_256", "kind": "fidelity", "n": 256, "nobj": 256, "ntheta": 90, "ndist": 4, "chunk": 45},
        # the smallest request of the serving mix: launches count
        {"name": "bh_128", "kind": "bh", "n": 128, "ntheta": 180, "ndist": 4, "niter": 4, "real": False},
        # the headline reconstruction's lines, images and slices, at a quarter of its angles
        {"name": "bh_512", "kind": "bh", "n": 512, "ntheta": 225, "ndist": 4, "niter": 4, "real": False},
        # near-field ptychography: one projection under a scanned probe
        {"name": "nfp_512", "kind": "nfp", "n": 512, "nobj": 768, "ntheta": 96, "niter": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["prop", "prop", "radon", "radon", "radon", "shift", "sback", "fidelity", "bh", "bh", "nfp"])
    if kind == "prop":
        sizes = [64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048]
        n, nz = rng.choice(sizes), rng.choice(sizes)
        return {"kind": kind, "n": n, "nz": nz, "batch": _log_int(rng, 1, max(1, (1 << 26) // (n * nz))),
                "adjoint": rng.random() < 0.5}
    if kind == "radon":
        n = rng.choice([64, 96, 128, 192, 256, 384, 512, 768, 1024, 2048])
        op = rng.choice(["R", "RT", "fbp"])
        ntheta = _log_int(rng, max(16, n // 4), 2 * n if n < 1024 else n)
        return {"kind": kind, "op": op, "n": n, "nz": _log_int(rng, 1, min(n, max(2, (1 << 25) // (n * n)))),
                "ntheta": ntheta, "real": rng.random() < 0.3}
    if kind == "shift":
        npsi, nzpsi = rng.choice([64, 128, 256, 384, 512, 768, 1024]), rng.choice([64, 128, 256, 384, 512, 768, 1024])
        n, nz = max(8, npsi - rng.randrange(0, npsi // 4)), max(8, nzpsi - rng.randrange(0, nzpsi // 4))
        return {"kind": kind, "op": rng.choice(["S", "adj"]), "n": n, "nz": nz, "npsi": npsi, "nzpsi": nzpsi,
                "batch": _log_int(rng, 1, max(1, (1 << 25) // (npsi * nzpsi))), "real": rng.random() < 0.5}
    if kind == "sback":
        npsi, nzpsi = rng.choice([128, 256, 384, 512, 768]), rng.choice([128, 256, 384, 512, 768])
        return {"kind": kind, "n": npsi - rng.randrange(0, npsi // 4), "nz": nzpsi - rng.randrange(0, nzpsi // 4),
                "npsi": npsi, "nzpsi": nzpsi, "batch": _log_int(rng, 1, max(1, (1 << 25) // (npsi * nzpsi))),
                "mag": round(rng.uniform(0.6, 1.0), 3)}
    if kind == "fidelity":
        n = rng.choice([64, 128, 256])
        nobj = rng.choice([s for s in (64, 128, 192, 256, 384) if n <= s <= 1.5 * n])
        ntheta = _log_int(rng, 16, 96)
        return {"kind": kind, "n": n, "nobj": nobj, "ntheta": ntheta, "ndist": rng.choice([1, 2, 4]),
                "chunk": rng.choice([ntheta, (ntheta + 1) // 2, (ntheta + 2) // 3])}
    if kind == "bh":
        n = rng.choice([64, 128, 256, 384, 512])
        return {"kind": kind, "n": n, "ntheta": _log_int(rng, n // 4, min(225, 7 * n // 4)), "ndist": rng.choice([2, 3, 4]),
                "niter": rng.choice([3, 4]), "real": n <= 256 and rng.random() < 0.4}
    n = rng.choice([128, 256, 512])
    return {"kind": kind, "n": n, "nobj": 3 * n // 2, "ntheta": _log_int(rng, 16, 128), "niter": rng.choice([3, 4])}


# ------------------------------------------------------------------ the inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1000 + seed)


def _smooth(shape, g, coarse=16):
    """Smooth random images or volumes in about [-2, 2] (the last two axes, and
    the first as well for a volume, interpolated from a coarse grid)."""
    batch, ny, nx = shape
    cy, cx = max(2, ny // coarse), max(2, nx // coarse)
    low = torch.randn(batch, 1, cy, cx, generator=g, device=DEV)
    return torch.nn.functional.interpolate(low, size=(ny, nx), mode="bilinear", align_corners=False)[:, 0]


def _volume(n, g):
    low = torch.rand(1, 1, max(4, n // 16), max(4, n // 16), max(4, n // 16), generator=g, device=DEV)
    v = torch.nn.functional.interpolate(low, size=(n, n, n), mode="trilinear", align_corners=False)[0, 0]
    ax = torch.linspace(-1, 1, n, device=DEV)
    return v * (ax[:, None] ** 2 + ax[None, :] ** 2 < 0.6)


def _object(n, g):
    """k dx (-delta + i delta / 50), delta up to 1e-6, inside a cylinder."""
    d = _volume(n, g) * (2 * math.pi / WAVELENGTH * VOXEL * 1e-6)
    return torch.complex(-d, d / 50)


def _wave(shape, g):
    """Detector-plane waves: amplitude near 1, smooth phase, fine noise."""
    amp = 1 + 0.1 * torch.randn(shape, generator=g, device=DEV)
    return torch.polar(amp, 0.5 * _smooth(shape, g))


def _amplitudes(shape, g):
    """Measured amplitudes: fringes of 10 % and photon noise of 1 %."""
    out = torch.empty(shape, device=DEV)
    for i in range(shape[0]):
        out[i] = 1 + 0.1 * _smooth(shape[1:], g, 8) + 0.01 * torch.randn(shape[1:], generator=g, device=DEV)
    return out.clamp_(min=0.05)


def _theta(ntheta):
    return np.linspace(0, np.pi, ntheta, endpoint=False).astype("float32")


def _probe(ndist, n, g):
    return torch.polar(1 + 0.05 * _smooth((ndist, n, n), g), 0.1 * _smooth((ndist, n, n), g))


def _positions(shape, amp, g):
    return amp * (2 * torch.rand(shape, generator=g, device=DEV) - 1)


def _inputs(c, seed):
    g = _gen(seed)
    k = c["kind"]
    if k == "prop":
        return {"x": _wave((c["batch"], c["nz"], c["n"]), g)}
    if k == "radon":
        n = c["n"]
        if c["op"] == "R":
            x = _smooth((c["nz"], n, n), g)
            return {"x": x if c["real"] else torch.complex(x, _smooth((c["nz"], n, n), g) / 50)}
        shape = (c["ntheta"], c["nz"], n)
        x = torch.randn(shape, generator=g, device=DEV) * 0.05 + torch.linspace(-1, 1, n, device=DEV).neg().cos()
        return {"x": x if c["real"] else torch.complex(x, 0.05 * torch.randn(shape, generator=g, device=DEV))}
    if k in ("shift", "sback"):
        b = c["batch"]
        coef, img = (b, c["nzpsi"], c["npsi"]), (b, c["nz"], c["n"])
        noise = lambda s: 0.02 * torch.randn(s, generator=g, device=DEV)
        field = lambda s: _smooth(s, g) + noise(s)
        r = _positions((b, 2), 2.0, g)
        if k == "sback":
            return {"x": torch.complex(field(img), noise(img)), "r": r}
        m = 1 - 0.05 * torch.rand(b, generator=g, device=DEV)
        x = field(coef) if c["real"] else torch.complex(field(coef), noise(coef))
        out = {"x": x, "r": r, "m": m}
        if c["op"] == "adj":
            out["g"] = field(img) if c["real"] else torch.complex(field(img), noise(img))
        return out
    if k == "nfp":
        n, no, nt = c["n"], c["nobj"], c["ntheta"]
        p = 0.3 * _smooth((1, no, no), g)[0]
        return {"proj": torch.complex(-p, p / 50), "prb": _probe(1, n, g)[0], "pos": _positions((nt, 2), 4.0, g),
                "data": _amplitudes((nt, 1, n, n), g)[:, 0]}
    n, nt, nd = c["n"], c["ntheta"], c["ndist"]
    obj = _object(c.get("nobj", n), g)
    return {"obj": obj.real.contiguous() if c.get("real") else obj, "prb": _probe(nd, n, g),
            "pos": _positions((nt, nd, 2), 2.0, g), "data": _amplitudes((nt, nd, n, n), g)}


def _rec_args(c):
    n, nt, nd = c["n"], c["ntheta"], c["ndist"]
    return types.SimpleNamespace(
        theta=_theta(nt), ndist=nd, ntheta=nt, nz=n, n=n, nzobj=n, nobj=n,
        obj_dtype="float32" if c["real"] else "complex64", mask=MASK, lam_prbfit=0.0, rho=list(RHO),
        niter=c["niter"], nchunk=n, vis_step=-1, err_step=-1, start_iter=0, distance=np.array(DISTANCES[:nd]),
        wavelength=WAVELENGTH, voxelsize=VOXEL, norm_magnifications=np.ones(nd))


def prepare(c, seed):
    s = _inputs(c, seed)
    s["case"] = c
    k = c["kind"]
    if k == "prop":
        s["op"] = Propagation(c["n"], c["nz"], c["batch"], 1, WAVELENGTH, VOXEL, np.array(DISTANCES[:1]))
    elif k == "radon":
        s["op"] = Tomo(c["n"], c["nz"], _theta(c["ntheta"]), MASK)
    elif k in ("shift", "sback"):
        s["op"] = Shift(c["n"], c["npsi"], c["nz"], c["nzpsi"], "float32" if c.get("real") else "complex64")
    elif k == "fidelity":
        s["op"] = DataFidelity.create(c["n"], c["n"], c["nobj"], c["nobj"], _theta(c["ntheta"]), c["ndist"], WAVELENGTH,
                                      VOXEL, np.array(DISTANCES[:c["ndist"]]), MASK, c["chunk"])
        s["mag"] = torch.ones(c["ntheta"], c["ndist"], device=DEV)
        for name in ("obj", "prb", "pos"):
            s[name].requires_grad_(True)
    elif k == "bh":
        s["op"] = Rec(_rec_args(c))
        s["op"].data.copy_(s["data"])
    else:
        n, no = c["n"], c["nobj"]
        s["op"] = RecNFP(types.SimpleNamespace(
            distance=np.array(DISTANCES[1:2]), wavelength=WAVELENGTH, voxelsize=VOXEL, ntheta=c["ntheta"], nz=n, n=n,
            nzobj=no, nobj=no, obj_dtype="complex64", rho=list(NFP_RHO), niter=c["niter"], nchunk=c["ntheta"],
            vis_step=-1, err_step=-1, start_iter=0))
        s["op"].data.copy_(s["data"])
    return s


def run(s):
    c, op = s["case"], s["op"]
    k = c["kind"]
    if k == "prop":
        return op.DT(s["x"], 0) if c["adjoint"] else op.D(s["x"], 0)
    if k == "radon":
        return getattr(op, c["op"])(s["x"])
    if k == "shift":
        coef = op.coeff(s["x"])
        if c["op"] == "S":
            return op.curlySc(coef, s["r"], s["m"])
        return op.dcurlySadjc(coef, s["r"], s["m"], s["g"])
    if k == "sback":
        return op.curlySback(s["x"], s["r"], c["mag"])
    if k == "fidelity":
        f = op(s["obj"], s["prb"], s["pos"], s["mag"], s["data"])
        return [f.detach()] + list(torch.autograd.grad(f, [s["obj"], s["prb"], s["pos"]]))
    names = ("obj", "prb", "pos") if k == "bh" else ("proj", "prb", "pos")
    for name in names:          # a reconstruction starts from its initial guess
        op.vars[name].copy_(s[name])
    if k == "bh":
        op.shrink_nd.zero_()    # where BH() leaves the magnifications it used
    op.BH(mode="graph")
    return {name: op.vars[name] for name in names}


# ------------------------------------------------------- what a pass cannot do without
def _fft(n):
    return 5 * math.log2(n)


def _radon_flops(n, nz, ntheta):
    # the padded 2-D transform, the 9 x 9 window of every polar sample, the detector transform
    return nz * (6 * n * n * _fft(2 * n) + ntheta * n * (81 * 4 + _fft(n)))


def _cascade_flops(n, nimg, directions):
    # a propagation is two passes of cosine transforms along each axis; a stencil is 4 + 4 taps on complex samples
    prop = 4 * _fft(n) + 8
    return nimg * n * n * ((2 + directions) * prop + (2 + directions) * 3 * 32 + 100)


def work(c):
    k, it = c["kind"], 4 if c.get("real") else 8
    if k == "prop":
        pix = c["batch"] * c["nz"] * c["n"]
        return {"bytes": 16 * pix + 8 * c["nz"] * c["n"], "flops": pix * (2 * _fft(c["n"]) + 2 * _fft(c["nz"]) + 8)}
    if k == "radon":
        n, nz, nt = c["n"], c["nz"], c["ntheta"]
        fl = _radon_flops(n, nz, nt) + (nz * nt * n * 2 * _fft(n) if c["op"] == "fbp" else 0)
        return {"bytes": it * nz * n * (n + nt), "flops": fl}
    if k == "shift":
        coef, img = c["batch"] * c["nzpsi"] * c["npsi"], c["batch"] * c["nz"] * c["n"]
        fl = coef * 2 * (_fft(c["npsi"]) + _fft(c["nzpsi"])) + img * 2 * 16 * it / 4
        if c["op"] == "adj":
            return {"bytes": it * (2 * coef + img), "flops": fl + img * 4 * 16 * it / 4}
        return {"bytes": it * (coef + img), "flops": fl}
    if k == "sback":
        coef, img = c["batch"] * c["nzpsi"] * c["npsi"], c["batch"] * c["nz"] * c["n"]
        return {"bytes": 8 * (coef + img), "flops": coef * (64 + 2 * (_fft(c["npsi"]) + _fft(c["nzpsi"])))}
    if k == "fidelity":
        n, no, nt, nd = c["n"], c["nobj"], c["ntheta"], c["ndist"]
        return {"bytes": 16 * no ** 3 + 4 * nt * nd * n * n + 16 * nd * n * n,
                "flops": 2 * _radon_flops(no, no, nt) + _cascade_flops(n, nt * nd, 0)}
    if k == "bh":
        n, nt, nd = c["n"], c["ntheta"], c["ndist"]
        return {"bytes": 2 * it * n ** 3 + 4 * nt * nd * n * n + 16 * nd * n * n,
                "flops": c["niter"] * (2 * _radon_flops(n, n, nt) + _cascade_flops(n, nt * nd, 2))}
    n, no, nt = c["n"], c["nobj"], c["ntheta"]
    return {"bytes": 16 * no * no + 4 * nt * n * n + 16 * n * n, "flops": c["niter"] * _cascade_flops(n, nt, 2)}


def tolerance(c):
    k = c["kind"]
    # about four times the distance from exact() seen over the ranges: 32-bit transforms and sums, and 32-bit sample
    # positions -- in the shifts, more so where they weigh a noisy image, and in the adjoint Radon transform, where a
    # position next to a cell boundary may place its window one cell on; a reconstruction carries each iteration's
    # rounding into the next
    if k == "radon":
        return {"rel": 2e-6 if c["op"] == "R" else 2.5e-5}
    if k == "shift":
        return {"rel": 8e-6 if c["op"] == "S" else 4.5e-5}
    return {"rel": {"prop": 8e-7, "sback": 2e-6, "fidelity": 2.5e-5, "bh": 1e-5, "nfp": 4e-6}[k]}


# ------------------------------------------------------------ the operators in 64 bits
def _fresnel(n, nz, distance):
    fx = np.fft.fftfreq(2 * n, d=VOXEL).astype("float32")
    fy = np.fft.fftfreq(2 * nz, d=VOXEL).astype("float32")
    fx, fy = np.meshgrid(fx, fy)
    h = np.exp(-1j * np.pi * WAVELENGTH * np.float64(distance) * (fx ** 2 + fy ** 2)) / float(4 * n * nz)
    return torch.from_numpy(h.astype("complex64")).to(DEV).to(torch.complex128)


def _mirror(n):
    i = torch.arange(2 * n, device=DEV) - n // 2
    i = torch.where(i < 0, -1 - i, i)
    return torch.where(i >= n, 2 * n - 1 - i, i)


def _prop64(x, h, adjoint=False):
    nz, n = x.shape[-2:]
    iy, ix = _mirror(nz), _mirror(n)
    if not adjoint:
        y = torch.fft.ifft2(torch.fft.fft2(x[..., iy, :][..., ix]) * h, norm="forward")
        return y[..., nz // 2:nz // 2 + nz, n // 2:n // 2 + n]
    p = torch.nn.functional.pad(x, (n // 2, n - n // 2, nz // 2, nz - nz // 2))
    y = torch.fft.ifft2(torch.fft.fft2(p) * h.conj(), norm="forward")
    y = torch.zeros(y.shape[:-2] + (nz, 2 * n), dtype=y.dtype, device=DEV).index_add_(-2, iy, y)
    return torch.zeros(y.shape[:-1] + (n,), dtype=y.dtype, device=DEV).index_add_(-1, ix, y)


def _mask64(n):
    t = np.linspace(-1, 1, n)
    x, y = np.meshgrid(t, t)
    disc = (x ** 2 + y ** 2 < MASK).astype("float32")
    g = np.exp(-400 * (x ** 2 + y ** 2))
    f = lambda a: np.fft.fftshift(np.fft.fft2(np.fft.fftshift(a)))
    m = np.fft.fftshift(np.fft.ifft2(np.fft.fftshift(f(disc) * f(g)))).real.astype("float32")
    return m / np.amax(m)


class _Radon64:
    """The gridded Radon transform (window half-width 4) and its adjoint; a
    64-bit volume [nz, n, n] to projections [ntheta, nz, n] and back."""

    def __init__(self, n, ntheta, norm_ntheta=None, first=0):
        full = norm_ntheta or ntheta
        self.n, self.ntheta = n, ntheta
        mu = -math.log(1e-3) / (2 * n * n)
        t = np.linspace(-0.5, 0.5, n, endpoint=False).astype("float32")
        dx, dy = np.meshgrid(t, t)
        phi = np.exp((mu * (n * n) * (dx * dx + dy * dy)).astype("float32")) * np.float32(1 - n % 4)
        phi = (phi.astype("float64") * _mask64(n).astype("float64") / (n * np.sqrt(n * full))).astype("float32")
        th = _theta(full)[first:first + ntheta].astype("float64")
        rho = (np.arange(n) - n // 2).astype("float32") / np.float32(n)
        # sample positions as the 32-bit values that place the window
        x0 = torch.from_numpy((rho[None, :] * np.cos(th).astype("float32")[:, None]).astype("float64")).to(DEV)
        y0 = torch.from_numpy((-rho[None, :] * np.sin(th).astype("float32")[:, None]).astype("float64")).to(DEV)
        self.phi = torch.from_numpy(phi).to(DEV).double()
        self.x0, self.y0, self.mu = x0.reshape(-1), y0.reshape(-1), mu
        self.bx, self.by = torch.floor(2 * n * self.x0).long() - 4, torch.floor(2 * n * self.y0).long() - 4
        i = torch.arange(2 * n, device=DEV)
        self.sign = (1.0 - 2.0 * (i % 2)).double()
        self.window = slice(n // 2, n // 2 + n)

    def _taps(self):
        n, mu = self.n, self.mu
        for j in range(9):
            y = self.by + j
            wy = math.pi / mu * torch.exp(-math.pi ** 2 / mu * (y.double() / (2 * n) - self.y0) ** 2)
            for i in range(9):
                x = self.bx + i
                wx = torch.exp(-math.pi ** 2 / mu * (x.double() / (2 * n) - self.x0) ** 2)
                yield ((n + y) % (2 * n)) * 2 * n + (n + x) % (2 * n), wx * wy

    def R(self, u):
        n, nz, s, w = self.n, u.shape[0], self.sign, self.window
        p = torch.zeros(nz, 2 * n, 2 * n, dtype=torch.complex128, device=DEV)
        p[:, w, w] = u * self.phi * s[w, None] * s[None, w]
        f = torch.fft.fft2(p) * s[:, None] * s[None, :]
        f = f.reshape(nz, -1).t().contiguous()
        acc = torch.zeros(self.ntheta * n, nz, dtype=torch.complex128, device=DEV)
        for idx, wt in self._taps():
            acc += wt[:, None] * f[idx]
        t = acc.reshape(self.ntheta, n, nz).transpose(1, 2) / n * s[:n]
        return torch.fft.ifft(t) * s[:n] / 4

    def RT(self, d):
        n, nz, s, w = self.n, d.shape[1], self.sign, self.window
        t = torch.fft.fft(d * s[:n]) * s[:n] / n / (4 * n)
        t = torch.view_as_real(t.transpose(1, 2).reshape(-1, nz).contiguous()).reshape(-1, 2 * nz)
        f = torch.zeros(4 * n * n, 2 * nz, dtype=torch.float64, device=DEV)
        for idx, wt in self._taps():
            f.index_add_(0, idx, wt[:, None] * t)
        f = torch.view_as_complex(f.reshape(-1, nz, 2)).t().reshape(nz, 2 * n, 2 * n)
        p = torch.fft.ifft2(f * s[:, None] * s[None, :]) * (4 * n * n)
        return p[:, w, w] * self.phi * s[w, None] * s[None, w]


class _RadonFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, u, op):
        ctx.op = op
        return op.R(u)

    @staticmethod
    def backward(ctx, g):
        return ctx.op.RT(g), None


def _coeff64(x):
    """The periodic cubic B-spline prefilter over the last two axes."""
    sy, sx = (1 / (4 + 2 * torch.cos(2 * math.pi * torch.arange(k, device=DEV).double() / k)) for k in x.shape[-2:])
    y = torch.fft.ifft2(torch.fft.fft2(x) * sy[:, None] * sx[None, :])
    return y if x.is_complex() else y.real


def _taps64(x, size):
    """Indices, clamped into range, and weights of the four taps at x (0 outside)."""
    i = torch.floor(x.detach())
    d, e = x - i, 1 - (x - i)
    w = [e ** 3, 4 - 6 * d * d + 3 * d ** 3, 4 - 6 * e * e + 3 * e ** 3, d ** 3]
    for j in range(4):
        p = i.long() + j - 1
        yield p.clamp(0, size - 1), torch.where((p >= 0) & (p < size), w[j], torch.zeros_like(x))


def _shift64(c, r, m, nz, n):
    """c [B, nzpsi, npsi] at the detector pixels shifted by r [B, 2] (y, x) and scaled by m [B]."""
    nzp, npx = c.shape[1:]
    at = lambda k, big, sh: (m[:, None] * (torch.arange(k, device=DEV).double() - k // 2) - sh[:, None]
                             + (m[:, None] - 1) / 2) + big // 2
    rows = cols = 0
    for p, w in _taps64(at(nz, nzp, r[:, 0]), nzp):
        rows = rows + w[:, :, None] * torch.gather(c, 1, p[:, :, None].expand(-1, -1, npx))
    for p, w in _taps64(at(n, npx, r[:, 1]), npx):
        cols = cols + w[:, None, :] * torch.gather(rows, 2, p[:, None, :].expand(-1, nz, -1))
    return cols


def _sback64(g, r, m, nzp, npx):
    """Detector images spread with the B-spline stretched by m."""
    b, nz, n = g.shape
    mf = torch.tensor(m, dtype=torch.float32, device=DEV)
    half = (mf - 1) / 2

    def axis(k, big, sh):
        # the position and the tap range in 32 bits (they decide which taps there are)
        p = (torch.arange(k, device=DEV) - k // 2).double()
        x = ((mf.double() * p[None, :] - sh.double()[:, None]).float() + half) + float(big // 2)
        i = torch.floor(x)
        d = x - i
        return i.long(), d, torch.ceil(d - 2 * mf), torch.trunc(d + 2 * mf)

    def phi(t):
        a = t.abs()
        return torch.where(a <= 1, 4 - 6 * a * a + 3 * a ** 3, (2 - a).clamp(min=0) ** 3)

    iy, dy, y0, y1 = axis(nz, nzp, r[:, 0])
    ix, dx, x0, x1 = axis(n, npx, r[:, 1])
    span = range(-3, 5)
    rows = torch.zeros(b, nzp, n, dtype=torch.complex128, device=DEV)
    for j in span:
        p = iy + j
        w = phi((dy.double() - j) / m) * ((j >= y0) & (j < y1) & (p >= 0) & (p < nzp))
        rows.scatter_add_(1, p.clamp(0, nzp - 1)[:, :, None].expand(-1, -1, n), w[:, :, None] * g)
    out = torch.zeros(b, nzp, npx, dtype=torch.complex128, device=DEV)
    for j in span:
        p = ix + j
        w = phi((dx.double() - j) / m) * ((j >= x0) & (j < x1) & (p >= 0) & (p < npx))
        out.scatter_add_(2, p.clamp(0, npx - 1)[:, None, :].expand(-1, nzp, -1), w[:, None, :] * rows)
    sym = []
    for k in (nzp, npx):
        f = 2 * math.pi * torch.arange(k, device=DEV).double() / k
        sym.append(4 + sum(2 * phi(torch.tensor(q / m, dtype=torch.float64)).item() * torch.cos(q * f) for q in range(1, 5)))
    return torch.fft.ifft2(torch.fft.fft2(out) / sym[0][:, None] / sym[1][None, :])


def _misfit64(c, prb, pos, data, tables):
    """sum (|D_k(prb_k exp(i S c))| - d)^2 over the angles [B] and distances of one chunk."""
    out = 0
    n = prb.shape[-1]
    for k, h in enumerate(tables):
        x22 = _shift64(c, pos[:, k], torch.ones(len(c), device=DEV).double(), prb.shape[-2], n)
        out = out + ((_prop64(prb[k] * torch.exp(1j * x22), h).abs() - data[:, k]) ** 2).sum()
    return out


def _forms64(v, y, z, data, tables, nall):
    """Gradients over (c, prb, pos) at v, or, with directions y and z, the
    Hessian forms [yy, yz as the solver pairs it, zz, yz symmetric], one chunk
    of angles at a time.  c is [B, nzobj, nobj], or one array for all angles."""
    c, prb, pos = v
    shared = c.ndim == 2
    gc, gprb, gpos, forms = [], 0, [], np.zeros(4)
    step = max(1, (1 << 22) // (prb.shape[-1] * prb.shape[-2] * len(tables)))
    for a in range(0, len(pos), step):
        sl = slice(a, a + step)
        nb = len(pos[sl])
        at = lambda t: t.expand(nb, -1, -1) if shared else t[sl]
        if y is None:
            w = [t.detach().clone().requires_grad_(True) for t in (c if shared else c[sl], prb, pos[sl])]
            f = _misfit64(w[0].expand(nb, -1, -1) if shared else w[0], w[1], w[2], data[sl], tables) / nall
            dc, dp, dr = torch.autograd.grad(f, w)
            gc.append(dc)
            gprb, gpos = gprb + dp, gpos + [dr]
            continue
        st = torch.zeros(2, dtype=torch.float64, device=DEV, requires_grad=True)
        move = lambda i, pick: pick(v[i]) + st[0] * pick(y[i]) + st[1] * pick(z[i])
        f = _misfit64(move(0, at), move(1, lambda t: t), move(2, lambda t: t[sl]), data[sl], tables) / nall
        g = torch.autograd.grad(f, st, create_graph=True)[0]
        hyy, hyz = torch.autograd.grad(g[0], st, retain_graph=True)[0].tolist()
        hzz = torch.autograd.grad(g[1], st)[0][1].item()
        # the solver's mixed form pairs the coefficients of each direction with its own positions
        own = cross = 0.0
        for k, h in enumerate(tables):
            one = torch.ones(nb, device=DEV).double()
            sh = lambda cc, rr: _shift64(cc, rr, one, prb.shape[-2], prb.shape[-1])
            x22 = sh(at(c), pos[sl][:, k]).detach().requires_grad_(True)
            fk = ((_prop64(prb[k] * torch.exp(1j * x22), h).abs() - data[sl][:, k]) ** 2).sum() / nall
            y22 = torch.autograd.grad(fk, x22)[0]
            q = []
            for d in (y, z):
                rr = pos[sl][:, k].detach().clone().requires_grad_(True)
                q.append(torch.autograd.grad((y22.conj() * sh(at(d[0]), rr)).real.sum(), rr)[0])
            ry, rz = y[2][sl][:, k], z[2][sl][:, k]
            own += ((q[0] * ry).sum() + (q[1] * rz).sum()).item()
            cross += ((q[0] * rz).sum() + (q[1] * ry).sum()).item()
        forms += np.array([hyy, hyz + own - cross, hzz, hyz])
    if y is not None:
        return forms
    return (sum(gc) if shared else torch.cat(gc)), gprb, torch.cat(gpos)


def _solve64(names, v, to_coef, from_coef, data, tables, rho, niter):
    """niter Bilinear-Hessian iterations over v (a dict of 64-bit arrays, the
    first of names being the object or projection)."""
    o = names[0]
    eta = None
    nall = data.numel()
    pack = lambda d: (to_coef(d[o]), d["prb"], d["pos"])
    dot = lambda a, b: (a.conj() * b).real.sum().item() if a.is_complex() else (a * b).sum().item()
    for _ in range(niter):
        gc, gprb, gpos = _forms64(pack(v), None, None, data, tables, nall)
        grad = dict(zip(names, (from_coef(gc), gprb, gpos)))
        grad = {k: t * rho[k] ** 2 for k, t in grad.items()}
        hgg, hge, hee, hsym = _forms64(pack(v), pack(grad), pack(eta if eta is not None else grad), data, tables, nall)
        beta = 0.0 if eta is None else hge / hee
        eta = {k: -t if eta is None else beta * eta[k] - t for k, t in grad.items()}
        top = -sum(dot(grad[k], eta[k]) / rho[k] ** 2 for k in names)
        alpha = top / (hgg if beta == 0.0 else beta * beta * hee - 2 * beta * hsym + hgg)
        v = {k: t + alpha * eta[k] for k, t in v.items()}
    return v


def _wide(t):
    return t.to(torch.complex128) if t.is_complex() else t.double()


def exact(c, seed):
    k = c["kind"]
    # in 64 bits with plain operations these take longer than a check should (or more memory than the card has)
    if (k == "bh" and c["n"] ** 3 * c["ntheta"] > 128 ** 3 * 200) or (k == "nfp" and c["n"] ** 2 * c["ntheta"] > 1 << 25):
        return None
    s = {name: _wide(t) for name, t in _inputs(c, seed).items()}
    if k == "prop":
        h = _fresnel(c["n"], c["nz"], DISTANCES[0])
        return torch.cat([_prop64(x[None], h, c["adjoint"]) for x in s["x"]])
    if k == "radon":
        op = _Radon64(c["n"], c["ntheta"])
        x, out = s["x"], []
        if c["op"] == "fbp":
            f = np.abs(np.fft.fftfreq(c["n"]).astype("float32")) * 4 * c["n"]
            x = torch.fft.ifft(torch.fft.fft(x) * torch.from_numpy(f).to(DEV).double())
            x = x.real if c["real"] else x
        step = max(1, 32 * 512 // c["n"])
        for z in range(0, c["nz"], step):
            out.append(op.R(x[z:z + step].to(torch.complex128)) if c["op"] == "R"
                       else op.RT(x[:, z:z + step].to(torch.complex128)))
        out = torch.cat(out, dim=1 if c["op"] == "R" else 0)
        if c["op"] == "fbp":
            out = out * float(np.float32(math.sqrt(c["n"] / c["ntheta"])))
        return out.real if c["real"] else out
    if k == "shift":
        coef = _coeff64(s["x"])
        if c["op"] == "S":
            return _shift64(coef, s["r"], s["m"], c["nz"], c["n"])
        r = s["r"].requires_grad_(True)
        coef.requires_grad_(True)
        f = (s["g"].conj() * _shift64(coef, r, s["m"], c["nz"], c["n"])).real.sum()
        gpos = torch.autograd.grad(f, r)[0]
        u = torch.zeros_like(coef).requires_grad_(True)
        v = _shift64(u, r.detach(), s["m"], c["nz"], c["n"])
        return [torch.autograd.grad(v, u, s["g"])[0], gpos]
    if k == "sback":
        return _sback64(s["x"], s["r"], c["mag"], c["nzpsi"], c["npsi"])
    if k == "fidelity":
        tables = [_fresnel(c["n"], c["n"], d) for d in DISTANCES[:c["ndist"]]]
        total, grads, nall = 0.0, [0, 0, []], s["data"].numel()
        for a in range(0, c["ntheta"], 16):
            sl = slice(a, a + 16)
            nb = len(s["pos"][sl])
            op = _Radon64(c["nobj"], nb, c["ntheta"], a)
            w = [s["obj"].detach(), s["prb"].detach().clone(), s["pos"][sl].detach().clone()]
            for t in w:
                t.requires_grad_(True)
            f = _misfit64(_coeff64(_RadonFn.apply(w[0], op)), w[1], w[2], s["data"][sl], tables) / nall
            g = torch.autograd.grad(f, w)
            total += f.item()
            grads = [grads[0] + g[0], grads[1] + g[1], grads[2] + [g[2]]]
        return [torch.tensor(total, dtype=torch.float64), grads[0], grads[1], torch.cat(grads[2])]
    if k == "nfp":
        tables = [_fresnel(c["n"], c["n"], DISTANCES[1])]
        v = {"proj": s["proj"], "prb": s["prb"][None], "pos": s["pos"][:, None]}
        v = _solve64(("proj", "prb", "pos"), v, _coeff64, _coeff64, s["data"][:, None], tables,
                     dict(zip(("proj", "prb", "pos"), NFP_RHO)), c["niter"])
        return {"proj": v["proj"], "prb": v["prb"][0], "pos": v["pos"][:, 0]}
    tables = [_fresnel(c["n"], c["n"], d) for d in DISTANCES[:c["ndist"]]]
    op = _Radon64(c["n"], c["ntheta"])
    norm = float(np.float32(np.sqrt(c["n"] / c["ntheta"])))
    keep = (lambda t: t.real) if c["real"] else (lambda t: t)
    mask = torch.from_numpy(_mask64(c["n"])).to(DEV).double()
    v = {"obj": s["obj"] / norm * mask, "prb": s["prb"], "pos": s["pos"]}
    v = _solve64(("obj", "prb", "pos"), v, lambda u: _coeff64(keep(op.R(u.to(torch.complex128)))),
                 lambda g: keep(op.RT(_coeff64(g).to(torch.complex128))), s["data"], tables,
                 dict(zip(("obj", "prb", "pos"), RHO)), c["niter"])
    return {"obj": v["obj"] * norm, "prb": v["prb"], "pos": v["pos"]}
