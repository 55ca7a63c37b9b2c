"""The workloads whose speed this package is held to: sizes, inputs, one pass, and its value in 64 bits.

``listed()`` names the fixed cases and ``draw(rng)`` makes others of the same ranges.  A case is a dict of plain
values:

    op       project | backproject | grad | osem | mlem | batch
    nx, nz   image nx x nx x nz (views nx x nz)
    px, pz   PSF support
    nview    views of the plan, over ``arc`` degrees
    step     the call takes every step-th view (project, backproject, grad); the number of subsets (osem)
    niter    EM iterations
    psf      gauss        depth-dependent Gaussians of a circular orbit, one stack for every view
             contour      the same on a body-contouring orbit: a stack of its own for every view
             penetration  Gaussian core with a radial exponential tail (septal penetration): not separable
    method   two (bilinear rotation) | one (three shears)

``prepare`` makes the inputs (ellipsoid phantom and body attenuation map for a 4.8 mm voxel, Poisson data with a
background of 5 % of the mean) and the plan that a program keeps; ``run`` is one call of the public API on them;
``exact`` is the same system model in 64 bits, in plain torch.
"""
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DY = 4.8  # mm
MU = 0.0096  # soft tissue, 1/mm
DEVICE = "cuda"


def _package():
    """The package directory ``spectrecon.jl_b200`` imported as ``spectrecon_b200``."""
    name = "spectrecon_b200"
    if name not in sys.modules:
        folder = os.path.join(ROOT, "spectrecon.jl_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ---------------------------------------------------------------- the cases

def _case(name, op, nx, nz, px, nview, step=1, niter=0, pz=None, psf="gauss", method="two", arc=360):
    return dict(name=name, op=op, nx=nx, nz=nz, px=px, pz=px if pz is None else pz, nview=nview, step=step,
                niter=niter, psf=psf, method=method, arc=arc)


def listed():
    return [
        # one transaxial slice, the 2-D example: the smallest call, bound by launches
        _case("slice_project", "project", 128, 1, 11, 80, pz=1),
        # one OS-EM-sized subset of the small study, as a program's own iteration calls it
        _case("subset_project_64", "project", 64, 64, 11, 64, step=8),
        # a training step through the projector at the reference's own timing size: forward and gradient
        _case("grad_64", "grad", 64, 40, 19, 60),
        # the small study, ML-EM on host arrays through the reference-shaped call
        _case("mlem_host_64", "mlem", 64, 64, 11, 64, niter=16),
        # all views of the clinical 128 x 128 x 80 study: simulating a scan
        _case("project_128", "project", 128, 80, 37, 120),
        # the adjoint of one subset of that study
        _case("backproject_128", "backproject", 128, 80, 37, 120, step=8),
        # the whole OS-EM reconstruction of that study
        _case("osem_128", "osem", 128, 80, 37, 120, step=8, niter=4),
        # a matrix that no tile divides, 180 degree cardiac arc, anisotropic PSF: OS-EM on odd sizes
        _case("osem_ragged", "osem", 90, 53, 21, 66, step=6, niter=2, pz=17, arc=180),
        # high-energy collimator: measured PSFs that are not separable, forward and adjoint
        _case("grad_penetration_128", "grad", 128, 80, 37, 120, step=8, psf="penetration"),
        # the shear rotation, a subset forward and adjoint
        _case("grad_shear_96", "grad", 96, 48, 21, 90, step=6, method="one"),
        # several patients of different sizes at once, body-contouring orbits among them
        dict(_case("batch_mixed", "batch", 0, 0, 0, 0, niter=2), jobs=5, mix=3),
        # whole-body matrix at high resolution: one OS-EM iteration of the large study
        _case("osem_256", "osem", 256, 200, 65, 128, step=16, niter=1),
    ]


def _odd(rng, lo, hi):
    """An odd number of [lo, hi], spread over its logarithm."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(max(lo, hi))))))
    return max(lo, min(hi, v // 2 * 2 + 1))


def _job(rng, largest):
    """Sizes, PSF and subsets of one drawn study."""
    if rng.random() < 0.5:
        nx = rng.choice([n for n in (64, 96, 128, 256) if n <= largest])
    else:
        nx = 2 * int(round(math.exp(rng.uniform(math.log(16), math.log(largest / 2)))))
    nz = 1 if rng.random() < 0.08 else int(round(math.exp(rng.uniform(math.log(8), math.log(max(10, 0.9 * nx))))))
    px = _odd(rng, 5, min(65, nx * 3 // 10 | 1))
    pz = 1 if nz == 1 else (px if rng.random() < 0.7 else _odd(rng, 3, px))
    nview, step = rng.choice([(32, 4), (60, 6), (60, 10), (64, 8), (66, 11), (90, 9), (90, 15), (120, 8), (120, 24),
                              (128, 16)])
    kinds = ["gauss"] * 13 + ["contour"] * 2 + ["penetration"] * 5
    psf = rng.choice(kinds) if nx <= 128 else "gauss"
    return dict(nx=nx, nz=nz, px=px, pz=pz, nview=nview, step=step, psf=psf, method="two",
                arc=rng.choice([180, 360, 360]))


def draw(rng):
    op = rng.choice(["project", "project", "backproject", "backproject", "grad", "grad", "osem", "osem", "osem",
                     "mlem", "batch"])
    if op == "batch":
        return dict(op=op, nx=0, nz=0, px=0, pz=0, nview=0, step=1, niter=rng.choice([1, 2]), psf="gauss",
                    method="two", arc=360, jobs=rng.randint(2, 5), mix=rng.randint(100, 10 ** 6))
    c = dict(op=op, niter=0, **_job(rng, 128 if op == "mlem" else 256))
    if op in ("project", "backproject", "grad") and rng.random() < 0.4:
        c["step"] = 1
    if op == "osem":
        c["niter"] = rng.choice([1, 2, 4])
    if op == "mlem":
        c["niter"], c["step"] = rng.choice([2, 4, 16]), 1
    if c["nx"] <= 128 and rng.random() < 0.12:
        c["method"] = "one"
    share = 0.5 if c["psf"] == "gauss" and c["method"] == "two" else 0.1  # the general paths do more for one voxel
    most = share * max(work(x)["flops"] for x in listed())
    while work(c)["flops"] > most and (c["niter"] > 1 or c["nview"] > 32):
        if c["niter"] > 1:
            c["niter"] //= 2
        else:
            c["nview"], c["step"] = 32, min(c["step"], 4)
    return c


def _jobs(case):
    """The studies of a case: itself, or the jobs of a batch."""
    if case["op"] != "batch":
        return [case]
    rng = random.Random(case["mix"])
    got = []
    for _ in range(case["jobs"]):
        j = _job(rng, 128)
        j.update(nz=rng.randint(24, 80), psf=rng.choice(["gauss", "gauss", "gauss", "contour"]), op="osem",
                 niter=case["niter"])
        j["pz"] = j["px"]
        got.append(j)
    return got


def work(case):
    """Bytes (each input and output once) and operations of one pass: per view and voxel four bilinear taps, the
    attenuation, and the PSF -- its separable taps, or two 2-D transforms of the padded plane."""
    nbytes = flops = 0.0
    for c in _jobs(case):
        nx, nz, px, pz = c["nx"], c["nz"], c["px"], c["pz"]
        vox, view = nx * nx * nz, nx * nz
        conv = 2 * (px + pz)
        if c["psf"] == "penetration":
            n = (nx + px - 1) * (nz + pz - 1)
            conv = min(2 * px * pz, (5 * n * math.log2(n) + 2 * n) / view)
        if c["op"] in ("osem", "mlem"):
            passes = c["nview"] * (1 + 2 * c["niter"])  # sensitivities; forward and adjoint of every iteration
            nbytes += 4 * (3 * vox + 2 * c["nview"] * view)  # mu-map, start, result; data, background
        else:
            n = len(range(0, c["nview"], c["step"]))
            both = c["op"] == "grad"
            passes = n * (1 + both)
            nbytes += 4 * ((2 + both) * vox + (1 + both) * n * view)
        stacks = c["nview"] if c["psf"] == "contour" else 1
        nbytes += 4 * stacks * nx * (px * pz if c["psf"] == "penetration" else px + pz)
        flops += passes * vox * (8 + 1 + conv)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------- inputs

def _gauss(n, fwhm):
    """Rows of normalised Gaussians, one for each full width (pixels)."""
    r = np.arange(n) - (n - 1) / 2
    w = np.exp(-0.5 * (r / (np.asarray(fwhm, np.float64)[..., None] / math.sqrt(math.log(256.0)))) ** 2)
    return w / w.sum(-1, keepdims=True)


def _fwhm(c):
    """Full widths along the depth: 1 pixel at the collimator, p / 6 far from it."""
    return 1.0, max(1.5, c["px"] / 6.0)


def _psfs(c):
    """(psfs[px, pz, ny, nview] in float32) of a case whose PSFs are given as an array."""
    lo, hi = _fwhm(c)
    depth = np.linspace(lo, hi, c["nx"])
    if c["psf"] == "contour":  # the detector follows an elliptic body: nearer at the front than at the sides
        ang = 2 * np.pi * np.arange(c["nview"]) / c["nview"]
        f = depth[None, :] + 0.15 * (hi - lo) * (1 - np.cos(2 * ang))[:, None]
        a, b = _gauss(c["px"], f), _gauss(c["pz"], f)
        h = (a[:, :, None, :] * b[:, :, :, None]).astype(np.float32)  # [view, y, pz, px]
        return h.transpose(3, 2, 1, 0)
    a, b = _gauss(c["px"], depth), _gauss(c["pz"], depth)
    x, z = np.arange(c["px"]) - (c["px"] - 1) / 2, np.arange(c["pz"]) - (c["pz"] - 1) / 2
    r = np.sqrt(x[None, :] ** 2 + z[:, None] ** 2)
    tail = np.exp(-r[None] / (2.0 * depth[:, None, None]))
    h = a[:, None, :] * b[:, :, None] + 0.15 * tail / tail.sum((1, 2), keepdims=True)
    h = (h / h.sum((1, 2), keepdims=True)).astype(np.float32)
    h = np.broadcast_to(h, (c["nview"],) + h.shape)  # one stack, repeated over the views
    return np.ascontiguousarray(h).transpose(3, 2, 1, 0)


def _angles(c):
    """View angles (float32): the plan's default for a full circle."""
    turn = float(np.float32(2 * np.pi)) * c["arc"] / 360.0
    return (np.arange(c["nview"]) / c["nview"] * turn).astype(np.float32)


def _phantom(c, seed):
    """Emission image and attenuation map, float32 on the GPU as [z, y, x]."""
    nx, nz = c["nx"], c["nz"]
    rng = np.random.default_rng(seed)
    t = torch.arange(nx, device=DEVICE, dtype=torch.float32) - (nx - 1) / 2
    x, y = t[None, None, :], t[None, :, None]
    z = (torch.arange(nz, device=DEVICE, dtype=torch.float32) - (nz - 1) / 2)[:, None, None]
    image = torch.zeros((nz, nx, nx), device=DEVICE)
    image += 0.1 * (x * x + y * y <= (0.45 * nx) ** 2)
    body = (x / (0.42 * nx)) ** 2 + (y / (0.34 * nx)) ** 2 <= 1
    mu = torch.zeros_like(image) + MU * body
    for i in range(8):
        cx, cy, cz = rng.uniform(-0.3, 0.3, 3) * (nx, nx, nz)
        ax, ay, az = np.maximum(rng.uniform(0.08, 0.3, 3) * (nx, nx, nz), 0.6)
        phi, value = rng.uniform(0, np.pi), rng.uniform(0.5, 2.0)
        u, v = math.cos(phi) * (x - cx) + math.sin(phi) * (y - cy), math.cos(phi) * (y - cy) - math.sin(phi) * (x - cx)
        inside = (u / ax) ** 2 + (v / ay) ** 2 + ((z - cz) / az) ** 2 <= 1
        image += value * inside
        if i < 2:  # bone and lung
            mu = torch.where(inside & body, (0.015, 0.004)[i], mu)
    return image, mu


def _plan(c, mu):
    S = _package()
    mumap = np.asfortranarray(mu.cpu().numpy().transpose(2, 1, 0))
    angles = None if c["arc"] == 360 else _angles(c)
    if c["psf"] == "gauss":
        lo, hi = _fwhm(c)
        return S.SPECTplan.gauss(mumap, DY, c["nview"], px=c["px"], pz=c["pz"], fwhm_start=lo, fwhm_end=hi,
                                 viewangle=angles, interpmeth=c["method"])
    return S.SPECTplan(mumap, _psfs(c), DY, viewangle=angles, interpmeth=c["method"])


def _index(c):
    return None if c["step"] == 1 else np.arange(0, c["nview"], c["step"], dtype=np.int32)


def _julia(t):
    """A contiguous tensor as the column-major array of the reversed shape that the package takes."""
    return t.permute(*reversed(range(t.dim())))


def _inputs(c, seed):
    """Everything but the plan, on the GPU, as [view, z, x] and [z, y, x]."""
    image, mu = _phantom(c, seed)
    s = {"mu": mu}
    gen = torch.Generator(DEVICE).manual_seed(int(seed))
    if c["op"] in ("project", "grad"):
        s["image"] = image
    if c["op"] == "grad":  # what a loss sends back
        n = len(range(0, c["nview"], c["step"]))
        s["dy"] = torch.randn((n, c["nz"], c["nx"]), device=DEVICE, generator=gen)
    if c["op"] in ("backproject", "osem", "mlem"):
        views = range(0, c["nview"], c["step"]) if c["op"] == "backproject" else range(c["nview"])
        mean = _Model(c, mu, torch.float32).project(image, views).clamp_(min=0)
        bg = 0.05 * mean.mean()
        scale = 4.0 / (1.05 * mean.mean())  # about four counts in a detector bin
        s["y"] = torch.poisson((mean + bg) * scale, generator=gen) / scale
        s["bg"] = torch.zeros_like(mean) + bg
        s["x0"] = torch.ones_like(image)
    return s


def prepare(case, seed):
    S = _package()
    states = []
    for k, c in enumerate(_jobs(case)):
        s = _inputs(c, seed + 1000 * k)
        s["plan"] = _plan(c, s.pop("mu"))
        s["index"] = _index(c)
        if c["op"] == "project":
            n = len(range(0, c["nview"], c["step"]))
            s["out"] = torch.empty((n, c["nz"], c["nx"]), device=DEVICE)
        if c["op"] in ("backproject", "osem"):
            s["out"] = torch.empty((c["nz"], c["nx"], c["nx"]), device=DEVICE)
        if c["op"] == "osem":
            s["blocks"], s["niter"] = S.Ablock(s["plan"], c["step"]), c["niter"]
        if c["op"] == "mlem":  # host arrays in the reference's layout
            for key in ("x0", "y", "bg"):
                s[key] = np.asfortranarray(_julia(s[key]).cpu().numpy())
            s["niter"] = c["niter"]
        else:
            s = {key: _julia(v) if torch.is_tensor(v) else v for key, v in s.items()}
        if c["op"] == "grad":
            import spectrecon_b200.operator as operator

            s["operator"] = operator.SPECTOperator(s["plan"], s["index"])
            s["project_ad"] = operator.project_ad
        states.append(s)
    if case["op"] != "batch":
        return {"op": case["op"], **states[0]}
    batch = S.Batch([s["plan"] for s in states], [c["step"] for c in _jobs(case)], [c["niter"] for c in _jobs(case)])
    for k, s in enumerate(states):
        batch.set_job(k, s["out"], s["x0"], s["y"], s["bg"])
    return {"op": "batch", "batch": batch, "jobs": states}


def run(state):
    S = _package()
    op = state["op"]
    if op == "project":
        return S.project_(state["out"], state["image"], state["plan"], index=state["index"])
    if op == "backproject":
        return S.backproject_(state["out"], state["y"], state["plan"], index=state["index"])
    if op == "osem":
        return S.osem_(state["out"], state["x0"], state["y"], state["bg"], state["blocks"], niter=state["niter"])
    if op == "mlem":
        return S.mlem(state["x0"], state["y"], state["bg"], state["plan"], niter=state["niter"])
    if op == "grad":
        x = state["image"].detach().requires_grad_(True)
        y = state["project_ad"](x, state["operator"])
        y.backward(state["dy"])
        return y.detach(), x.grad
    state["batch"].run()
    return [s["out"] for s in state["jobs"]]


# ---------------------------------------------------------------- the same in plain torch

class _Model:
    """The system model of a case in plain torch: rotation about z, attenuation, replicate-boundary convolution with
    the PSF of every depth plane, depth sum, and the transpose of that.  Images are [z, y, x], views [view, z, x]."""

    def __init__(self, c, mu, dtype):
        self.c, self.dtype = c, dtype
        self.nx, self.nz = c["nx"], c["nz"]
        self.hx, self.hz = (c["px"] - 1) // 2, (c["pz"] - 1) // 2
        self.size = (self.nz + 2 * self.hz, self.nx + 2 * self.hx)  # no output wraps at these
        self.angles = _angles(c).astype(np.float64)
        self.mu = mu.to(dtype)
        self.spectra, self.psfs = {}, None if c["psf"] == "gauss" else _psfs(c)

    def _spectrum(self, v):
        key = v if self.c["psf"] == "contour" else 0
        if key not in self.spectra:
            if self.psfs is None:
                f = np.linspace(*_fwhm(self.c), self.nx)
                a, b = _gauss(self.c["px"], f), _gauss(self.c["pz"], f)
                h = a[:, None, :] * b[:, :, None]
            else:
                h = self.psfs[:, :, :, key].transpose(2, 1, 0)
            k = torch.zeros((self.nx,) + self.size, dtype=self.dtype, device=DEVICE)
            k[:, :self.c["pz"], :self.c["px"]] = torch.from_numpy(np.ascontiguousarray(h, np.float64)).to(k)
            self.spectra = {key: torch.fft.rfft2(torch.roll(k, (-self.hz, -self.hx), (1, 2)))}
        return self.spectra[key]

    # ---- rotation
    def _bilinear(self, v):
        """Rows of the image (as [y x, z]) and their weights for the four taps of every rotated-grid point."""
        n, th = self.nx, float(self.angles[v])
        phi, c0 = 2 * math.pi - th, (n - 1) / 2
        cs, sn = (1.0, 0.0) if th == 0 else (math.cos(phi), math.sin(phi))
        t = torch.arange(n, dtype=torch.float64, device=DEVICE) - c0
        s1 = c0 + cs * t[None, :] - sn * t[:, None]
        s2 = c0 + sn * t[None, :] + cs * t[:, None]
        f1, f2 = s1.floor(), s2.floor()
        for d1 in (0, 1):
            for d2 in (0, 1):
                j1, j2 = f1 + d1, f2 + d2
                w = (1 - (s1 - j1).abs()) * (1 - (s2 - j2).abs())
                ok = (j1 >= 0) & (j1 < n) & (j2 >= 0) & (j2 < n)
                row = (j2.clamp(0, n - 1) * n + j1.clamp(0, n - 1)).long()
                yield row.reshape(-1), torch.where(ok, w, torch.zeros_like(w)).reshape(-1, 1).to(self.dtype)

    def _shears(self, v):
        """(quarter turns, None) or (quarter turns, the lines' indices and weights along x, y, x)."""
        th, pad = float(self.angles[v]), math.ceil(1 + self.nx * math.sqrt(2) / 2 - self.nx / 2)
        m = math.floor(0.5 + th / (math.pi / 2)) % 4
        rest = th - m * (math.pi / 2)
        if abs(rest) <= math.sqrt(2.0 ** -23) * max(abs(th), m * math.pi / 2):
            return pad, m, None
        L = self.nx + 2 * pad

        def lines(slope):
            shift = (torch.arange(L, dtype=torch.float64, device=DEVICE) - (L - 1) / 2)[:, None] * slope
            lo = shift.floor()
            at = torch.arange(L, device=DEVICE)[None, :] + lo.long()
            return at.clamp(0, L - 1), (at + 1).clamp(0, L - 1), (shift - lo).to(self.dtype)

        return pad, m, (lines(math.tan(rest / 2)), lines(-math.sin(rest)), lines(math.tan(rest / 2)))

    @staticmethod
    def _turn(a, m):
        """m quarter turns in the plane's last two dimensions: (x, y) -> (L - 1 - y, x)."""
        for _ in range(m % 4):
            a = a.transpose(-1, -2).flip(-1)
        return a

    @staticmethod
    def _shear(a, line, along_x, adjoint):
        i0, i1, t = line
        if not along_x:
            a = a.transpose(-1, -2)
        i0, i1 = i0.expand_as(a), i1.expand_as(a)
        if adjoint:
            out = torch.zeros_like(a).scatter_add_(-1, i0, (1 - t) * a).scatter_add_(-1, i1, t * a)
        else:
            out = (1 - t) * a.gather(-1, i0) + t * a.gather(-1, i1)
        return out if along_x else out.transpose(-1, -2)

    def _rotate(self, a, v):
        if self.c["method"] == "two":
            rows = a.reshape(self.nz, -1).t().contiguous()
            out = sum(w * rows[r] for r, w in self._bilinear(v))
            return out.t().reshape(self.nz, self.nx, self.nx)
        if self.angles[v] == 0:
            return a
        pad, m, lines = self._shears(v)
        a = self._turn(torch.nn.functional.pad(a, (pad,) * 4), m)
        for k, line in enumerate(lines or ()):
            a = self._shear(a, line, k != 1, False)
        return a[:, pad:pad + self.nx, pad:pad + self.nx]

    def _rotate_adjoint(self, a, v):
        if self.c["method"] == "two":
            rows = a.reshape(self.nz, -1).t().contiguous()
            out = torch.zeros_like(rows)
            for r, w in self._bilinear(v):
                out.index_add_(0, r, w * rows)
            return out.t().reshape(self.nz, self.nx, self.nx)
        if self.angles[v] == 0:
            return a
        pad, m, lines = self._shears(v)
        a = torch.nn.functional.pad(a, (pad,) * 4)
        for k, line in reversed(list(enumerate(lines or ()))):
            a = self._shear(a, line, k != 1, True)
        return self._turn(a, -m)[:, pad:pad + self.nx, pad:pad + self.nx]

    def _attenuation(self, v):
        """exp(-dy (sum of mu in front, half of its own)) on the rotated grid, as [y, z, x]."""
        mu = self._rotate(self.mu, v).transpose(0, 1)
        return torch.exp(-float(np.float32(DY)) * (mu.cumsum(0) - 0.5 * mu))

    # ---- projector
    def project(self, image, views):
        image, got = image.to(self.dtype), []
        for v in views:
            a = self._rotate(image, v).transpose(0, 1) * self._attenuation(v)
            a = torch.nn.functional.pad(a[None], (self.hx, self.hx, self.hz, self.hz), mode="replicate")[0]
            f = (torch.fft.rfft2(a) * self._spectrum(v)).sum(0)
            a = torch.fft.irfft2(f, s=self.size)
            got.append(a[self.hz:self.hz + self.nz, self.hx:self.hx + self.nx])
        return torch.stack(got)

    def backproject(self, y, views):
        out = torch.zeros((self.nz, self.nx, self.nx), dtype=self.dtype, device=DEVICE)
        for k, v in enumerate(views):
            a = torch.nn.functional.pad(y[k].to(self.dtype), (self.hx, self.hx, self.hz, self.hz))
            a = torch.fft.irfft2(torch.fft.rfft2(a)[None] * self._spectrum(v), s=self.size)
            for dim, h, n in ((1, self.hz, self.nz), (2, self.hx, self.nx)):  # padding folds into the edges
                body = a.narrow(dim, h, n).clone()
                body.narrow(dim, 0, 1).add_(a.narrow(dim, 0, h).sum(dim, keepdim=True))
                body.narrow(dim, n - 1, 1).add_(a.narrow(dim, h + n, h).sum(dim, keepdim=True))
                a = body
            out += self._rotate_adjoint((a * self._attenuation(v)).transpose(0, 1).contiguous(), v)
        return out

    def osem(self, x, y, bg, nblocks, niter):
        x, y, bg = x.to(self.dtype), y.to(self.dtype), bg.to(self.dtype)
        subsets = [range(b, self.c["nview"], nblocks) for b in range(nblocks)]
        sens = []
        for s in subsets:
            a = self.backproject(torch.ones_like(y[:len(s)]), s)
            sens.append(torch.where(a == 0, torch.full_like(a, math.inf), a))
        for _ in range(niter):
            for s, a in zip(subsets, sens):
                at = torch.tensor(list(s), device=DEVICE)
                x = x * (self.backproject(y[at] / (self.project(x, s) + bg[at]), s) / a)
        return x


def exact(case, seed):
    """What ``run`` returns for these inputs, in 64 bits."""
    got = []
    for k, c in enumerate(_jobs(case)):
        s = _inputs(c, seed + 1000 * k)
        m = _Model(c, s["mu"], torch.float64)
        views = range(0, c["nview"], c["step"])
        if c["op"] == "project":
            got.append(_julia(m.project(s["image"], views)))
        elif c["op"] == "backproject":
            got.append(_julia(m.backproject(s["y"], views)))
        elif c["op"] == "grad":
            return _julia(m.project(s["image"], views)), _julia(m.backproject(s["dy"], views))
        else:
            got.append(_julia(m.osem(s["x0"], s["y"], s["bg"], c["step"] if c["op"] == "osem" else 1, c["niter"])))
    if case["op"] == "batch":
        return got
    return got[0].cpu().numpy() if case["op"] == "mlem" else got[0]
