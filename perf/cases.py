"""The calls that programs make of nemaktis_gb300, as cases to time and to check.

Four kinds of call:

  backend     the drop-in entry of the nemaktis package, bpm_backend.run_backend_{without,with}_mask, on host
              arrays in FP64 (its default), or api.run / api.run_batch with precision="fp32";
  plan        api.Plan: settings and director laid out once, then execute + download per pass;
  microscope  OpticalFields / FieldViewer: refocus the fields and form the spectrum again (FP64);
  lines       nbpm_periodic_tridiag_solve: batched periodic tridiagonal line solves on device arrays (FP64).

The fields of an FP32 run are 32-bit numbers that the entry point widens into the caller's complex128 array;
such cases hand them on as complex64, which loses nothing.

exact() propagates the same inputs in 64 bits with plain torch: the operators of each slab are written down
entry by entry and the periodic tridiagonal lines are solved by cyclic reduction.
"""
import ctypes
import math

import numpy as np
import torch

from nemaktis_gb300 import _lib, api, bpm_backend, microscope, workloads

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # the smallest call of a nemaktis script: one wavelength at normal incidence on a small cell
        {"name": "backend_tn_64_fp64", "kind": "backend", "precision": "fp64", "director": "twisted",
         "nx": 64, "ny": 64, "nz": 40, "nl": 1, "nq": 1},
        # the same cell in the FP32 mode
        {"name": "backend_tn_64_fp32", "kind": "backend", "precision": "fp32", "director": "twisted",
         "nx": 64, "ny": 64, "nz": 40, "nl": 1, "nq": 1},
        # a Q-tensor simulation on an odd mesh, a few colours, tilted illumination
        {"name": "backend_odd_fp64", "kind": "backend", "precision": "fp64", "director": "qtensor",
         "nx": 97, "ny": 75, "nz": 33, "nl": 3, "nq": 7},
        # a masked droplet with its interface formula, as light_propagator passes it
        {"name": "backend_droplet_fp64", "kind": "backend", "precision": "fp64", "director": "droplet",
         "nx": 128, "ny": 128, "nz": 64, "nl": 1, "nq": 1},
        # a small request of the serving mix: small mesh, many colours and angles
        {"name": "plan_small_many_fp32", "kind": "plan", "precision": "fp32", "director": "smooth",
         "nx": 64, "ny": 64, "nz": 32, "nl": 8, "nq": 7},
        # a white-light micrograph under Koehler illumination in the reference's precision
        {"name": "plan_koehler_fp64", "kind": "plan", "precision": "fp64", "director": "defects",
         "nx": 256, "ny": 256, "nz": 16, "nl": 3, "nq": 13},
        # the headline benchmark: white-light Koehler micrograph, FP32 batched
        {"name": "plan_koehler_fp32", "kind": "plan", "precision": "fp32", "director": "defects",
         "nx": 256, "ny": 256, "nz": 64, "nl": 16, "nq": 13},
        # a large droplet, one propagation: few slots on a large mesh
        {"name": "plan_droplet_512_fp32", "kind": "plan", "precision": "fp32", "director": "droplet",
         "nx": 512, "ny": 512, "nz": 128, "nl": 1, "nq": 1},
        # the largest transverse mesh of the benchmark's uneven samples
        {"name": "plan_1024_fp32", "kind": "plan", "precision": "fp32", "director": "smooth",
         "nx": 1024, "ny": 1024, "nz": 24, "nl": 2, "nq": 7},
        # several samples of uneven size in one call
        {"name": "batch_uneven_fp32", "kind": "backend", "precision": "fp32", "director": "smooth",
         "nx": 256, "ny": 256, "nz": 24, "nl": 2, "nq": 7, "samples": 3},
        # moving the focus of a micrograph
        {"name": "microscope_256", "kind": "microscope", "precision": "fp64",
         "nx": 256, "ny": 256, "nl": 4, "nq": 19},
        # the line solve as a primitive of its own
        {"name": "lines_512", "kind": "lines", "precision": "fp64", "nx": 513, "ny": 2048},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _size(rng, a, b):
    """A mesh size: any up to 200 points; larger meshes are chosen with small factors for their Fourier transforms."""
    n = _log(rng, a, b)
    while n > 200 and _largest_factor(n) > 23:
        n -= 1
    return n


def _largest_factor(n):
    p = 2
    while p * p <= n:
        if n % p:
            p += 1
        else:
            n //= p
    return n


def draw(rng):
    kind = rng.choice(["backend", "backend", "backend", "plan", "plan", "plan", "plan", "microscope", "lines"])
    if kind == "lines":
        return {"kind": kind, "precision": "fp64", "nx": _log(rng, 48, 1025), "ny": _log(rng, 64, 4096)}
    if kind == "microscope":
        return {"kind": kind, "precision": "fp64", "nx": _size(rng, 64, 360), "ny": _size(rng, 64, 360),
                "nl": rng.randint(1, 4), "nq": rng.choice([1, 7, 19])}
    precision = rng.choice(["fp64", "fp32"])
    c = {"kind": kind, "precision": precision,
         "director": rng.choice(["twisted", "qtensor", "droplet", "smooth", "defects"])}
    if kind == "backend":
        c.update(nx=_size(rng, 40, 200), ny=_size(rng, 40, 200), nz=rng.randint(12, 64), nl=rng.randint(1, 6),
                 nq=rng.randint(1, 13))
        if rng.random() < 0.2:
            c.update(samples=rng.randint(2, 3), director="smooth")
    else:
        c.update(nx=_size(rng, 48, 1024), ny=_size(rng, 48, 1024), nz=rng.randint(12, 96), nl=rng.randint(1, 16),
                 nq=rng.randint(1, 19))
    # at most the work of the largest listed case of the precision: fewer colours, angles and planes until it is
    most = 6e7 if precision == "fp64" else 1.0e9
    while _voxel_steps(c) > most:
        k = max(("nl", "nq", "nz"), key=lambda n: c[n] / {"nl": 3, "nq": 3, "nz": 12}[n])
        c[k] = max(1, c[k] * 3 // 4)
    return c


# ---- what a case stands for: mesh, colours, angles, director ---------------------------------------------

SPACING = 0.25


def _dims(case):
    """Mesh of each sample of the case (a batch's samples get smaller one by one)."""
    n = case.get("samples", 1)
    return [(max(24, case["nx"] * (n - i) // n), max(24, case["ny"] * (n - i) // n), case["nz"]) for i in range(n)]


def _voxel_steps(case):
    return sum(x * y * (z - 1) for x, y, z in _dims(case)) * case["nl"] * case["nq"] * 2


def _wavelengths(case):
    return [0.55] if case["nl"] == 1 else [0.4 + 0.4 * i / (case["nl"] - 1) for i in range(case["nl"])]


def _wavevectors(nq):
    """The first nq points of a hexagonal condenser grid of two rings at NA 0.25."""
    q = [(0.0, 0.0)]
    for r in (1, 2):
        q += [(0.125 * r * math.cos(k * math.pi / (3 * r)), 0.125 * r * math.sin(k * math.pi / (3 * r)))
              for k in range(6 * r)]
    return q[:nq]


def _no(lam):
    return 1.52 + 0.008 / lam**2


def _ne(lam):
    return 1.74 + 0.008 / lam**2


# the aperture passes between the Fourier modes of the round meshes, so that none lies on its edge
NHOST, NA = 1.55, 0.4137


def _radius2(dims):
    r = 0.39 * SPACING * (min(dims) - 1) + 0.0123457
    return round(r * r, 5)


def _mesh(dims):
    ax = [(torch.arange(n, dtype=torch.float64, device=DEV) - 0.5 * (n - 1)) * SPACING for n in dims]
    return ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]


def _director(kind, dims, seed):
    """Director (Nz, Ny, Nx, 3) or Q-tensor (.., 6), float64, and the mask values or None."""
    g = torch.Generator().manual_seed(int(seed))
    rnd = lambda *s: torch.rand(*s, generator=g, dtype=torch.float64).tolist()  # noqa: E731
    x, y, z = _mesh(dims)
    span = [SPACING * max(1, n - 1) for n in dims]

    def waves(n, shortest):  # a smooth random scalar: plane waves with wavelengths of at least `shortest` um
        s = torch.zeros(dims[::-1], dtype=torch.float64, device=DEV)
        for a, b, c, p, w in zip(*(rnd(n) for _ in range(5))):
            k = [2 * math.pi / shortest * (2 * v - 1) / math.sqrt(3) for v in (a, b, c)]
            s += (0.3 + w) * torch.cos(k[0] * x + k[1] * y + k[2] * z + 2 * math.pi * p)
        return s / math.sqrt(n)

    mask = None
    if kind in ("smooth", "qtensor"):
        v = torch.stack([waves(8, 4.0) for _ in range(3)], -1)
        n = v / v.norm(dim=-1, keepdim=True).clamp_min(1e-9)
        if kind == "qtensor":
            s = 0.6 + 0.1 * torch.tanh(waves(4, 6.0))
            n0, n1, n2 = n.unbind(-1)
            n = torch.stack([s * (1.5 * a * b - (0.5 if a is b else 0.0)) for a, b in
                             ((n0, n0), (n1, n1), (n2, n2), (n0, n1), (n0, n2), (n1, n2))], -1)
    elif kind == "twisted":
        phi = 0.5 * math.pi * (z / span[2] + 0.5) + 0.02 * waves(6, 3.0)
        t = 0.05 * waves(8, 3.0)
        n = torch.stack([phi.cos() * t.cos(), phi.sin() * t.cos(), t.sin()], -1)
    elif kind == "defects":
        phi = torch.zeros(1, dims[1], dims[0], dtype=torch.float64, device=DEV)
        for k, (a, b) in enumerate(zip(rnd(8), rnd(8))):
            phi = phi + (0.5 if k % 2 == 0 else -0.5) * torch.atan2(y - 0.8 * (b - 0.5) * span[1], x - 0.8 * (a - 0.5) * span[0])
        n = torch.stack([phi.cos(), phi.sin(), torch.zeros_like(phi)], -1).expand(dims[2], -1, -1, -1)
    else:  # cholesteric droplet
        phase = 2 * math.pi * rnd(1)[0]
        r = (x * x + y * y + z * z).sqrt().clamp_min(1e-9)
        rho = (x * x + y * y).sqrt().clamp_min(1e-9)
        psi = 2 * math.pi * r / 5.0 + phase
        rh = [c.expand(r.shape) / r for c in (x, y, z)]
        az = [(-y / rho).expand(r.shape), (x / rho).expand(r.shape), torch.zeros_like(r)]
        cr = [az[1] * rh[2] - az[2] * rh[1], az[2] * rh[0] - az[0] * rh[2], az[0] * rh[1] - az[1] * rh[0]]
        mask = (_radius2(dims) - x * x - y * y - z * z).expand(r.shape)
        n = torch.stack([psi.cos() * a + psi.sin() * b for a, b in zip(rh, cr)], -1)
        n = torch.where((mask >= 0)[..., None], n, torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device=DEV))
        mask = mask.contiguous()
    return n.contiguous(), mask


def _samples(case, seed):
    """What a program hands to the backend: settings, director, mask, formula and result array per sample."""
    out = []
    for i, dims in enumerate(_dims(case)):
        lc, mask = _director(case["director"], dims, seed * 16 + i)
        js = workloads.settings_json(
            dims, (SPACING,) * 3, _wavelengths(case), _wavevectors(case["nq"]), no="1.52+0.008/lambda^2",
            ne="1.74+0.008/lambda^2", nhost=repr(NHOST), NA=NA,
            lc_type="Q-tensor" if case["director"] == "qtensor" else "Director")
        s = {"json": js, "lc": lc.cpu().numpy(), "mask": None if mask is None else mask.cpu().numpy(),
             "formula": None if mask is None else "%.5f-x^2-y^2-z^2" % _radius2(dims)}
        shape = (case["nl"], case["nq"], 4, dims[1], dims[0])
        if case["kind"] == "plan":  # kept for many passes: page-locked
            s["pinned"] = torch.zeros(shape, dtype=torch.complex128, pin_memory=DEV == "cuda")
            s["E"] = s["pinned"].numpy()
        else:
            s["E"] = np.zeros(shape, np.complex128)
        out.append(s)
    return out


# ---- one pass ----------------------------------------------------------------------------------------------

def prepare(case, seed):
    state = {"kind": case["kind"], "precision": case["precision"]}
    if case["kind"] == "lines":
        state["lines"] = _line_systems(case, seed)
        state["x"] = torch.zeros_like(state["lines"][3])
        state["lib"] = _lib.load()
    elif case["kind"] == "microscope":
        q = _wavevectors(case["nq"])
        of = microscope.OpticalFields(
            wavelengths=_wavelengths(case), max_NA_objective=NA, max_NA_condenser=0.25, wavevectors=q,
            N_radial_wavevectors=_rings(case["nq"]), mesh_dimensions=(case["nx"], case["ny"]),
            mesh_lengths=(SPACING * (case["nx"] - 1), SPACING * (case["ny"] - 1)))
        of.vals = _micro_fields(case, seed).cpu().numpy()
        v = microscope.FieldViewer(of)
        v.polariser, v.analyser, v.analyser_angle = True, True, 80.0
        v.NA_condenser = 0.25 if case["nq"] > 1 else 0.0
        state["viewer"] = v
    else:
        state["samples"] = _samples(case, seed)
        if case["kind"] == "plan":
            s = state["samples"][0]
            state["plan"] = api.Plan([{k: s[k] for k in ("json", "lc", "mask", "formula", "E")}], case["precision"])
            state["plan"].upload()
        else:
            bpm_backend.set_strict(True)
    return state


def run(state):
    kind, fp32 = state["kind"], state["precision"] == "fp32"
    if kind == "lines":
        a = [ctypes.c_void_p(t.data_ptr()) for t in state["lines"]]
        x = state["x"]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(state["lib"].nbpm_periodic_tridiag_solve(x.shape[1], x.shape[0], *a, ctypes.c_void_p(x.data_ptr()), stream))
        return x
    if kind == "microscope":
        v = state["viewer"]
        v.z_focus = 3.0
        v.update_image()
        return v.get_spectrum()
    samples = state["samples"]
    if kind == "plan":
        state["plan"].execute()
        state["plan"].download()
        E = samples[0]["pinned"].to(DEV, non_blocking=True)  # the fields go on to torch code on the GPU
        return E.to(torch.complex64) if fp32 else E
    if len(samples) > 1:
        api.run_batch(samples, precision=state["precision"])
    elif fp32:
        s = samples[0]
        api.run(s["json"], s["lc"], s["E"], mask=s["mask"], formula=s["formula"], precision="fp32")
    else:
        s = samples[0]
        if s["mask"] is None:
            bpm_backend.run_backend_without_mask(s["json"], s["lc"].ravel(), s["E"])
        else:
            bpm_backend.run_backend_with_mask(s["json"], s["formula"], s["lc"].ravel(), s["mask"].ravel(), s["E"])
    return [s["E"].astype(np.complex64) if fp32 else s["E"] for s in samples]


def work(case):
    """Each input and output once; the operations of the discretisation: per propagated point and slab 96 stencil
    taps and 60 line-solve steps, 8 phase products (complex multiply-adds) and, for tilted waves, 32 real ones x 2."""
    if case["kind"] == "lines":
        n = case["nx"] * case["ny"]
        return {"bytes": 5 * 16 * n, "flops": 8 * 8 * n}
    if case["kind"] == "microscope":
        n, planes = case["nx"] * case["ny"], case["nl"] * case["nq"] * 4
        fft = 2 * 5 * n * math.log2(n) * planes
        return {"bytes": 16 * n * planes + 8 * n * case["nl"], "flops": fft + 40 * n * planes}
    vs = _voxel_steps(case)
    fd = 6 if case["director"] == "qtensor" else 3
    nvox = sum(x * y * z for x, y, z in _dims(case))
    field = sum(x * y for x, y, z in _dims(case)) * case["nl"] * case["nq"] * 4
    per = 8 * (96 + 60 + 8) + (128 if case["nq"] > 1 else 0)
    return {"bytes": nvox * 8 * (fd + (case["director"] == "droplet")) + 16 * field, "flops": per * vs}


def _rings(nq):
    return {1: 1, 7: 2, 19: 3}[nq]


def _micro_fields(case, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    shape = (case["nl"], case["nq"], 4, case["ny"], case["nx"])
    r = torch.randn(shape, generator=g, dtype=torch.float64, device=DEV)
    return torch.complex(r, torch.randn(shape, generator=g, dtype=torch.float64, device=DEV))


def _line_systems(case, seed):
    """Periodic systems like those of the implicit half-steps: i * mu * (second difference with varying weights)."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    shape = (case["ny"], case["nx"])
    rnd = lambda: torch.randn(shape, generator=g, dtype=torch.float64, device=DEV)  # noqa: E731
    a, b = 0.15 * (1 + 0.2 * rnd()), 0.15 * (1 + 0.2 * rnd())
    inf, sup = torch.complex(0.02 * rnd(), -a), torch.complex(0.02 * rnd(), -b)
    mid = torch.complex(1 + 0.02 * rnd(), a + b)
    return inf, mid, sup, torch.complex(rnd(), rnd())


# ---- the same in 64 bits, in plain torch -----------------------------------------------------------------

def exact(case, seed):
    if case["kind"] == "lines":
        inf, mid, sup, rhs = _line_systems(case, seed)
        x = _Lines(inf[:, :-1], mid[:, :-1], sup[:, :-1]).solve(rhs[:, :-1])
        return torch.cat([x, x[:, :1]], 1)
    if case["kind"] == "microscope":
        return _exact_spectrum(case, seed)
    if _voxel_steps(case) > 2.2e9:
        return None
    out = []
    for i, dims in enumerate(_dims(case)):
        E = [_propagate(case, dims, seed * 16 + i, lam) for lam in _wavelengths(case)]
        out.append(torch.stack(E))
    return out[0] if case["kind"] == "plan" else out


class _Lines:
    """Periodic tridiagonal systems along the last axis, inf_i x_{i-1} + mid_i x_i + sup_i x_{i+1} = b_i, by cyclic
    reduction: every step doubles the distance of the coupled neighbours and squares the size of the coupling."""

    def __init__(self, inf, mid, sup):
        self.r0 = 1 / mid
        a, c, s = inf * self.r0, sup * self.r0, 1
        self.steps = []
        while max(a.abs().max().item(), c.abs().max().item()) > 1e-18:
            if len(self.steps) > 16:
                raise ValueError("not reducible")
            am, cm, ap, cp = (torch.roll(v, sh, -1) for v, sh in ((a, s), (c, s), (a, -s), (c, -s)))
            r = 1 / (1 - a * cm - c * ap)
            self.steps.append((s, -a * r, r, -c * r))
            a, c, s = -a * am * r, -c * cp * r, 2 * s

    def solve(self, b):
        b = b * self.r0
        for s, fa, r, fc in self.steps:
            b = fa * torch.roll(b, s, -1) + r * b + fc * torch.roll(b, -s, -1)
        return b


def _eps_planes(case, dims, seed, lam):
    """Per plane iz: the nine quantities of the voxels that the operators are made from; and nref."""
    lc, mask = _director(case["director"], dims, seed)
    ep, ea = _no(lam) ** 2, _ne(lam) ** 2 - _no(lam) ** 2
    if lc.shape[-1] == 3:
        n = lc.unbind(-1)
        e = [ep + ea * n[0] ** 2, ep + ea * n[1] ** 2, ep + ea * n[2] ** 2, ea * n[0] * n[1], ea * n[0] * n[2], ea * n[1] * n[2]]
    else:
        Q = lc.unbind(-1)
        e = [ep + ea / 3 + 2 * ea / 3 * Q[k] for k in range(3)] + [2 * ea / 3 * Q[k] for k in (3, 4, 5)]
    if mask is not None:
        inside = mask >= 0
        host = torch.tensor(NHOST**2, dtype=torch.float64, device=DEV)
        e = [torch.where(inside, v, host if k < 3 else 0 * host) for k, v in enumerate(e)]
    xx, yy, xy = e[0] - e[4] ** 2 / e[2], e[1] - e[5] ** 2 / e[2], e[3] - e[4] * e[5] / e[2]
    tr, det = 0.5 * (xx + yy), xx * yy - xy * xy
    r2 = tr * tr - det
    r = r2.clamp_min(0).sqrt()
    neff = torch.where(r2 < 1e-8, tr.sqrt(), ((tr + r).sqrt() + (tr - r).clamp_min(0).sqrt()) / 2)
    planes = {"xx": xx, "yy": yy, "xy": xy, "sxx": neff + (xx - yy) / (4 * neff), "syy": neff + (yy - xx) / (4 * neff),
              "sxy": xy / (2 * neff), "vx": e[4] / e[2], "vy": e[5] / e[2], "iz": 1 / e[2]}
    return planes, neff.mean().item(), mask


def _z_weights(dims, mask):
    """Weights of a slab's two planes where the droplet's surface crosses it: bisection to 1e-3 of the spacing."""
    x, y, _ = _mesh(dims)
    f = lambda z: _radius2(dims) - x[0] ** 2 - y[0] ** 2 - z * z  # noqa: E731
    out = []
    for iz in range(dims[2] - 1):
        zi = (iz - 0.5 * (dims[2] - 1)) * SPACING
        lo = torch.full(mask.shape[1:], zi, dtype=torch.float64, device=DEV)
        hi = torch.full_like(lo, (iz + 1 - 0.5 * (dims[2] - 1)) * SPACING)
        fl = f(lo)
        cross = fl * f(hi) <= 0
        z, live = lo.clone(), cross.clone()
        while True:
            live = live & ((hi - lo).abs() >= 1e-3 * SPACING)
            if not live.any():
                break
            mid = 0.5 * (lo + hi)
            fm = f(mid)
            z = torch.where(live, mid, z)
            live = live & (fm != 0)
            down = live & (fm * fl < 0)
            up = live & ~(fm * fl < 0)
            hi = torch.where(down, mid, hi)
            lo, fl = torch.where(up, mid, lo), torch.where(up, fm, fl)
        w0 = (z - zi) / SPACING
        half = torch.full_like(w0, 0.5)
        out.append((torch.where(cross, w0, half), torch.where(cross, 1 - w0, half)))
    return out


def _propagate(case, dims, seed, lam):
    """Screen fields (Nq, 4, Ny, Nx) of one wavelength."""
    Nx, Ny, Nz = dims
    k0 = 2 * math.pi / lam
    h = k0 * SPACING
    P, nref, mask = _eps_planes(case, dims, seed, lam)
    weights = None if mask is None else _z_weights(dims, mask)
    q = _wavevectors(case["nq"])
    # entrance: polarisations x and y through the input Fresnel operator; (Nq, 2 pol) fields of 2 components
    def fresnel(iz):
        return P["sxx"][iz], P["syy"][iz], P["sxy"][iz]

    sxx, syy, sxy = fresnel(0)
    det = (1 + sxx) * (1 + syy) - sxy**2
    jin = [2 * (1 + syy) / det, -2 * sxy / det, 2 * (1 + sxx) / det]
    f0 = torch.stack([jin[0], jin[1]]).to(torch.complex128).repeat(len(q), 1, 1).contiguous()
    f1 = torch.stack([jin[1], jin[2]]).to(torch.complex128).repeat(len(q), 1, 1).contiguous()
    shift = _Shift(q, dims, nref, h)
    for iz in range(Nz - 1):
        A = {k: v[iz] for k, v in P.items()}
        B = {k: v[iz + 1] for k, v in P.items()}
        w = (0.5, 0.5) if weights is None else weights[iz]
        ph = _phase(A, B, w, h, _no(lam))
        op = _Slab(A, B, h, Nx, Ny)
        f0, f1 = shift(f0, f1)
        f0, f1 = ph[0] * f0 + ph[2] * f1, ph[2] * f0 + ph[1] * f1
        f0, f1 = op.step(f0, f1)
        f0, f1 = ph[0] * f0 + ph[2] * f1, ph[2] * f0 + ph[1] * f1
        f0, f1 = shift(f0, f1)
    sxx, syy, sxy = fresnel(Nz - 1)
    det = (1 + sxx) * (1 + syy) - sxy**2
    f0, f1 = (2 * (1 - (1 + syy) / det) * f0 + 2 * sxy / det * f1, 2 * (1 - (1 + sxx) / det) * f1 + 2 * sxy / det * f0)
    # screen: the aperture of the objective in Fourier space
    freq = lambda n: torch.fft.fftfreq(n, SPACING, dtype=torch.float64, device=DEV) * 2 * math.pi / k0  # noqa: E731
    E = torch.stack([f0, f1], 1).reshape(len(q), 4, Ny, Nx)
    for i, (qx, qy) in enumerate(q):
        kx, ky = freq(Nx) + qx, freq(Ny) + qy
        open_ = (kx[None, :] ** 2 + ky[:, None] ** 2).sqrt() < NA
        E[i] = torch.fft.ifft2(torch.fft.fft2(E[i]) * open_)
    return E


def _phase(A, B, w, h, no):
    """exp(i d) of the symmetric 2x2 phase d of half a slab: its xx, yy and xy entries."""
    dxx = 0.5 * h * (w[0] * A["sxx"] + w[1] * B["sxx"] - no)
    dyy = 0.5 * h * (w[0] * A["syy"] + w[1] * B["syy"] - no)
    dxy = 0.5 * h * (w[0] * A["sxy"] + w[1] * B["sxy"])
    m, d = (dxx + dyy) / 2, (dxx - dyy) / 2
    r = (dxy**2 + d**2).sqrt()
    sinc = torch.where(r < 1e-8, torch.ones_like(r), r.sin() / r.clamp_min(1e-30))
    e, c = torch.exp(1j * m), r.cos()
    return e * (c + 1j * d * sinc), e * (c - 1j * d * sinc), e * 1j * dxy * sinc


class _Shift:
    """Translation of tilted waves by half a slab: four-point cubic interpolation with period N - 1, and their phase."""

    def __init__(self, q, dims, nref, h):
        self.q, self.px, self.py = q, dims[0] - 1, dims[1] - 1
        self.par = []
        for qx, qy in q:
            t = []
            for v in (qx, qy):
                s = -v / (2 * nref)
                m = math.floor(s)
                u = s - m
                t.append((m, (-u * (1 - u) ** 2 / 2, (1 - u) * (1 + u - 1.5 * u * u), u * (1 + 4 * u - 3 * u * u) / 2, -u * u * (1 - u) / 2)))
            a = -h * (qx * qx + qy * qy) / (4 * nref)
            self.par.append((t[0], t[1], complex(math.cos(a), math.sin(a))))

    @staticmethod
    def _axis(f, dim, period, m, w):
        n = f.shape[dim]
        i = torch.arange(n, device=f.device)
        return sum(wk * f.index_select(dim, (i + m - 1 + k) % period) for k, wk in enumerate(w))

    def __call__(self, *fs):
        out = []
        for f in fs:
            f = f.clone()
            for i, ((mx, wx), (my, wy), ph) in enumerate(self.par):
                g = self._axis(f[2 * i:2 * i + 2], 2, self.px, mx, wx)
                f[2 * i:2 * i + 2] = ph * self._axis(g, 1, self.py, my, wy)
            out.append(f)
        return out


class _Slab:
    """The diffraction operator of one slab, R = i W + (D S^-1 + S^-1 D) / 4, as stencil entries, and its
    alternating-direction step with two Woodbury iterates. The last row and column repeat the first."""

    def __init__(self, A, B, h, Nx, Ny):
        self.Nx, self.Ny = Nx, Ny
        dev = A["xx"].device
        iy, ix = torch.arange(Ny, device=dev), torch.arange(Nx, device=dev)
        nb = lambda i, n: {0: i, 1: torch.where(i == n - 2, 0, i + 1).clamp_max(n - 1),  # noqa: E731
                           -1: torch.where(i == 0, n - 2, i - 1)}
        self.X, self.Y = nb(ix, Nx), nb(iy, Ny)
        # the weights of the first derivative reach the neighbour across the repeated point
        nq = lambda i, n: {0: i, 1: torch.where(i == n - 1, 1, (i + 1).clamp_max(n - 1)),  # noqa: E731
                           -1: torch.where(i == 0, n - 2, i - 1)}
        QX, QY = nq(ix, Nx), nq(iy, Ny)
        self.fx, self.fy = torch.where(ix == Nx - 1, 0, ix), torch.where(iy == Ny - 1, 0, iy)
        avg = {k: (A[k] + B[k]) / 2 for k in A}
        det = avg["sxx"] * avg["syy"] - avg["sxy"] ** 2
        S = (avg["syy"] / det, avg["sxx"] / det, -avg["sxy"] / det)
        v = (A["vx"] + B["vx"], A["vy"] + B["vy"])
        ez, mu = avg["iz"], h / 2
        at = lambda t, y, x: t[y][:, x]  # noqa: E731
        rowx, rowy = (ix < Nx - 1)[None, :], (iy < Ny - 1)[:, None]

        def entry(D, y, x, dd, b, ok):
            """mu R of the four blocks for the neighbour at (y, x), D = ((D00, D01), (D10, D11))."""
            C = [at(s, y, x) for s in S]
            z = torch.zeros_like(S[0])
            D = [z + d for d in D]
            re = [D[0] * C[0] + D[1] * C[2] + S[0] * D[0] + S[2] * D[2],
                  D[0] * C[2] + D[1] * C[1] + S[0] * D[1] + S[2] * D[3],
                  D[2] * C[0] + D[3] * C[2] + S[2] * D[0] + S[1] * D[2],
                  D[2] * C[2] + D[3] * C[1] + S[2] * D[1] + S[1] * D[3]]
            im = [0, 0, 0, 0]
            if dd:
                for a in (0, 1):
                    im[2 * a + b] = im[2 * a + b] + dd * v[a]
                    im[2 * b + a] = im[2 * b + a] + dd * at(v[a], y, x)
            return [torch.where(ok, mu / 4 * torch.complex(z - i, z + r), 0j) for r, i in zip(re, im)]

        self.dx, self.dy, self.dd = {}, {}, {}
        c = {s: 0.5 * (at(ez, iy, QX[s]) + ez) / h**2 for s in (-1, 1)}
        c[0] = -c[-1] - c[1]
        for s in (-1, 0, 1):
            K = at(avg["xx"], iy, self.X[s]), at(avg["xy"], iy, self.X[s])
            self.dx[s] = entry((c[s] * K[0], c[s] * K[1], 0, (1.0, -2.0, 1.0)[s + 1] / h**2), iy, self.X[s], 0.5 * s / h, 0, rowx)
        c = {s: 0.5 * (at(ez, QY[s], ix) + ez) / h**2 for s in (-1, 1)}
        c[0] = -c[-1] - c[1]
        for s in (-1, 0, 1):
            K = at(avg["yy"], self.Y[s], ix), at(avg["xy"], self.Y[s], ix)
            self.dy[s] = entry(((1.0, -2.0, 1.0)[s + 1] / h**2, 0, c[s] * K[1], c[s] * K[0]), self.Y[s], ix, 0.5 * s / h, 1, rowy)
        for sy in (-1, 1):
            for sx in (-1, 1):
                g = -sx * sy / (4 * h**2)
                d01 = sx * sy * at(ez, iy, QX[sx]) / (4 * h**2)
                d10 = sx * sy * at(ez, QY[sy], ix) / (4 * h**2)
                y, x = self.Y[sy], self.X[sx]
                kxx, kyy, kxy = (at(avg[k], y, x) for k in ("xx", "yy", "xy"))
                self.dd[sy, sx] = entry((d01 * kxy, g + d01 * kyy, g + d10 * kxx, d10 * kxy), y, x, 0, 0, rowx & rowy)
        n, m = Nx - 1, Ny - 1
        self.lx = [_Lines(-self.dx[-1][b][:, :n], 1 - self.dx[0][b][:, :n], -self.dx[1][b][:, :n]) for b in (0, 3)]
        self.ly = [_Lines(*(t.T.contiguous() for t in (-self.dy[-1][b][:m], 1 - self.dy[0][b][:m], -self.dy[1][b][:m])))
                   for b in (0, 3)]

    def _dx(self, b, f):
        return sum(self.dx[s][b] * f.index_select(2, self.X[s]) for s in (-1, 0, 1))

    def _dy(self, b, f):
        return sum(self.dy[s][b] * f.index_select(1, self.Y[s]) for s in (-1, 0, 1))

    def _dd(self, b, f):
        return sum(self.dd[sy, sx][b] * f.index_select(1, self.Y[sy]).index_select(2, self.X[sx])
                   for sy in (-1, 1) for sx in (-1, 1))

    def _fold(self, t, y=True, x=True):
        if y:
            t = t.index_select(1, self.fy)
        return t.index_select(2, self.fx) if x else t

    def _solve_x(self, c, b):
        x = self.lx[c].solve(b[..., :-1])
        return torch.cat([x, x[..., :1]], -1)

    def _solve_y(self, c, b):
        x = self.ly[c].solve(b[:, :-1].transpose(1, 2)).transpose(1, 2)
        return torch.cat([x, x[:, :1]], 1)

    def step(self, f0, f1):
        t0 = f0 + self._fold(self._dy(0, f0) + self._dy(1, f1), x=False)
        t1 = f1 + self._fold(self._dy(3, f1) + self._dd(3, f1) + self._dy(2, f0) + self._dd(2, f0))
        t0, t1 = self._solve_x(0, t0), self._solve_x(1, t1)
        f0, f1 = t0, t1
        for _ in range(2):
            t0, t1 = (self._solve_x(0, self._fold(self._dx(1, t1) + self._dd(1, t1) + self._dd(0, t0))),
                      self._solve_x(1, self._fold(self._dx(2, t0), y=False)))
            f0, f1 = f0 + t0, f1 + t1
        t0 = f0 + self._fold(self._dx(0, f0) + self._dd(0, f0) + self._dx(1, f1) + self._dd(1, f1))
        t1 = f1 + self._fold(self._dx(3, f1) + self._dx(2, f0), y=False)
        t0, t1 = self._solve_y(0, t0), self._solve_y(1, t1)
        f0, f1 = t0, t1
        for _ in range(2):
            t0, t1 = (self._solve_y(0, self._fold(self._dy(1, t1), x=False)),
                      self._solve_y(1, self._fold(self._dy(2, t0) + self._dd(2, t0) + self._dd(3, t1))))
            f0, f1 = f0 + t0, f1 + t1
        return f0, f1


def _exact_spectrum(case, seed):
    """Focus by 3 um through the objective's filter, polariser at 0 and analyser at 80 degrees, Koehler average."""
    V = _micro_fields(case, seed)
    Nx, Ny, nq = case["nx"], case["ny"], case["nq"]
    q = _wavevectors(nq)
    w = _koehler_weights(0.25, _rings(nq), nq)
    a = math.radians(80.0)
    out = torch.zeros(Ny, Nx, case["nl"], dtype=torch.float64, device=DEV)
    for l, lam in enumerate(_wavelengths(case)):
        k0 = 2 * math.pi / lam
        kx = torch.fft.fftfreq(Nx, SPACING, dtype=torch.float64, device=DEV) * 2 * math.pi
        ky = torch.fft.fftfreq(Ny, SPACING, dtype=torch.float64, device=DEV) * 2 * math.pi
        for i, wi in enumerate(w):
            k2 = (kx[None, :] + k0 * q[i][0]) ** 2 + (ky[:, None] + k0 * q[i][1]) ** 2
            arg = (k0**2 - k2).clamp_min(0).sqrt() - k0
            theta = torch.atan2(arg.sin(), arg.cos())
            filt = torch.where(k2 < (NA * k0) ** 2, torch.exp(3j * theta), 0j)
            F = torch.fft.ifft2(torch.fft.fft2(V[l, i]) * filt)
            # polariser along x keeps the fields of input x (components 0 and 1); the analyser projects on its axis
            out[:, :, l] += wi * 0.5 * (math.cos(a) * F[0] + math.sin(a) * F[1]).abs() ** 2
    return torch.flip(out, (0,)).cpu().numpy()


def _koehler_weights(NA, rings, nq):
    """Weights of the condenser's rings for a linear interpolation between them (none for a single wave)."""
    if nq == 1:
        return [1.0]
    d, rmax = NA / (rings - 1), rings - 1
    F = lambda v, p: v - math.atanh(v) - p * math.log(1 - v * v) / 2  # noqa: E731
    first = lambda r: 1 + 3 * r * (r - 1)  # noqa: E731
    w = [0.0] * first(rmax + 1)
    if rmax == 1:
        w[0] = (F(NA, d) - F(0, d)) / d
        w[1:7] = [(F(0, 0) - F(NA, 0)) / (6 * d)] * 6
    else:
        w[0] = (F(d, d) - F(0, d)) / d
        for r in range(1, rmax):
            top = NA if r == rmax - 1 else (r + 1) * d
            v = (F(top, (r + 1) * d) + F((r - 1) * d, (r - 1) * d) - 2 * F(r * d, r * d)) / (6 * r * d)
            w[first(r):first(r + 1)] = [v] * (6 * r)
        w[first(rmax):] = [(F((rmax - 1) * d, (rmax - 1) * d) - F(NA, (rmax - 1) * d)) / (6 * rmax * d)] * (6 * rmax)
    return [2 / NA**2 * v for v in w]
