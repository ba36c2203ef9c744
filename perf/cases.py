"""Performance cases of the space-charge library: what a user's program has it do.

Each case is one pass through the public entry points (src_b200/scgpu.py, the
C ABI of include/scgpu.h):

  solve    PoissonSolver::computePotential on a device buffer
  image    computePotential(rho, hr, zshift): the image charge's potential
  fields   PartBunch::computeSelfFields: host arrays in, host arrays out
  job      a tracking job: upload a bunch, step it, download it (optionally a
           statistics record every `stat_every` steps, energy bins, a DC beam)
  batch    an optimizer's generation: bunches of uneven sizes join a batch,
           step together in rounds, are read back and leave

Bunches are the Gaussian recipe of the single-bunch workloads (1 nC,
sigma = 1, 1, 2 mm, beta*gamma 10), the photoinjector's and the DC beam's
stand-ins, and the batched workload's distributions, drawn on the GPU from
the case's seed.  `exact` restates the same physics in 64-bit torch
operations (torch.fft, index_add) without the library.
"""
import ctypes
import math

import numpy as np
import torch

from src_b200 import scgpu

C_LIGHT = 299792458.0
MASS_EV = 0.51099892e6
CHARGE = -1.0
COUPLING = 1.0 / (4 * 3.14159265358979323846 * 8.854187817e-12)
DT = 1e-12
BBOXINCR = 2.0
MESHES = [n for n in range(12, 129) if max(p for p in range(2, 2 * n + 1) if (2 * n) % p == 0 and all(p % q for q in range(2, p))) <= 5]


def listed():
    return [
        # smallest call: a coarse solver's potential, launch latency
        {"name": "solve 16^3", "kind": "solve", "nx": 16, "ny": 16, "nz": 16},
        # a mesh whose axes differ and are no powers of two
        {"name": "solve 40x20x60", "kind": "solve", "nx": 40, "ny": 20, "nz": 60},
        # the finest mesh of the benchmark workloads
        {"name": "solve 128^3", "kind": "solve", "nx": 128, "ny": 128, "nz": 128},
        # a self-field call of a host-side tracker (arrays in host memory)
        {"name": "fields 1e5 32^3", "kind": "fields", "n": 100_000, "nx": 32, "ny": 32, "nz": 32},
        # the smallest job of the optimizer's mix, an odd particle count, mixed form
        {"name": "job 10007 16^3 mixed", "kind": "job", "n": 10_007, "nx": 16, "ny": 16, "nz": 16, "mixed": True,
         "steps": 100, "bz": 0.0, "stat_every": 0, "bins": 0, "dc": False},
        # the 100-step single-bunch workload with a statistics record every ten steps
        {"name": "job 1e5 32^3", "kind": "job", "n": 100_000, "nx": 32, "ny": 32, "nz": 32, "mixed": False,
         "steps": 100, "bz": 0.0, "stat_every": 10, "bins": 0, "dc": False},
        # the benchmark's workload, FP64
        {"name": "job 1e6 64^3", "kind": "job", "n": 1_000_000, "nx": 64, "ny": 64, "nz": 64, "mixed": False,
         "steps": 100, "bz": 0.0, "stat_every": 0, "bins": 0, "dc": False},
        # the same in the mixed form
        {"name": "job 1e6 64^3 mixed", "kind": "job", "n": 1_000_000, "nx": 64, "ny": 64, "nz": 64, "mixed": True,
         "steps": 100, "bz": 0.0, "stat_every": 0, "bins": 0, "dc": False},
        # the large workload: 1e7 particles in a solenoid field, mixed form
        {"name": "job 1e7 128^3 mixed bz", "kind": "job", "n": 10_000_000, "nx": 128, "ny": 128, "nz": 128,
         "mixed": True, "steps": 60, "bz": 0.2, "stat_every": 0, "bins": 0, "dc": False},
        # a photoinjector bunch: ten energy bins with image charges
        {"name": "photoinjector 1e6 64^3", "kind": "job", "n": 1_000_000, "nx": 64, "ny": 64, "nz": 64,
         "mixed": False, "steps": 5, "bz": 0.0, "stat_every": 0, "bins": 10, "dc": False},
        # a coasting beam with periodic z
        {"name": "dc 3e5 48x48x64", "kind": "job", "n": 300_001, "nx": 48, "ny": 48, "nz": 64, "mixed": False,
         "steps": 50, "bz": 0.0, "stat_every": 0, "bins": 0, "dc": True},
        # uneven bunches stepping together, mixed form (the batched workload's distributions)
        {"name": "batch 12 mixed", "kind": "batch", "count": 12, "mixed": True, "rounds": 5, "steps": 8, "jobs_seed": 7},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, lo=12, hi=128):
    """A supported mesh size, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((m for m in MESHES if lo <= m <= hi), key=lambda m: abs(math.log(m / v)))


def draw(rng):
    kind = rng.choice(["solve", "image", "fields", "job", "job", "job", "job", "bins", "dc", "batch"])
    if kind in ("solve", "image"):
        return {"kind": kind, "nx": _mesh(rng), "ny": _mesh(rng), "nz": _mesh(rng)}
    if kind == "fields":
        return {"kind": "fields", "n": _log_int(rng, 1e4, 1e6), "nx": _mesh(rng, 16, 64), "ny": _mesh(rng, 16, 64),
                "nz": _mesh(rng, 16, 64)}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(3, 24), "mixed": rng.random() < 0.5, "rounds": rng.randint(2, 5),
                "steps": rng.randint(2, 12), "jobs_seed": rng.randrange(1 << 20)}
    c = {"kind": "job", "n": _log_int(rng, 1e4, 2e6), "nx": _mesh(rng, 16), "ny": _mesh(rng, 16), "nz": _mesh(rng, 16),
         "mixed": rng.random() < 0.5, "steps": rng.randint(20, 100), "bz": rng.choice([0.0, 0.0, 0.2]),
         "stat_every": rng.choice([0, 0, 10]), "bins": 0, "dc": False}
    if kind == "bins":
        c.update(n=_log_int(rng, 1e4, 1e6), nx=_mesh(rng, 16, 64), ny=_mesh(rng, 16, 64), nz=_mesh(rng, 16, 64),
                 bins=rng.randint(2, 12), steps=rng.randint(3, 10), bz=0.0, stat_every=0)
    if kind == "dc":
        c.update(dc=True, nz=2 * _mesh(rng, 12, 64), n=_log_int(rng, 1e4, 1e6), steps=rng.randint(20, 50))
    return c


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) * 1_000_003 + 17)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=_device(), dtype=torch.float64)


def _gaussian(g, n, sigma=(1e-3, 1e-3, 2e-3), bg_z=10.0, rel_spread=1e-3, bg_perp=1e-3):
    s = torch.tensor(sigma, dtype=torch.float64, device=_device())
    R = _randn(g, n, 3) * s
    P = _randn(g, n, 3) * bg_perp
    P[:, 2] = bg_z + P[:, 2] / bg_perp * (bg_z * rel_spread)
    return R, P


def _photoinjector(g, n, nbins):
    """Shortly after emission from a cathode at z = 0: bins by slices of z, the head fastest."""
    R = _randn(g, n, 3) * torch.tensor([1e-3, 1e-3, 0.8e-3], dtype=torch.float64, device=_device())
    R[:, 2] = R[:, 2].clamp(-4e-3, 4e-3) + 5e-3
    P = _randn(g, n, 3) * 1e-3
    order = torch.argsort(-R[:, 2], stable=True)
    bins = torch.empty(n, dtype=torch.int32, device=_device())
    bins[order] = (torch.arange(n, device=_device()) * nbins // n).to(torch.int32)
    bg = 1.5 - bins.double() / max(nbins - 1, 1)
    P[:, 2] = bg * (1.0 + P[:, 2])
    return R, P, bins


def _period():
    return 2e-2


def _dc(g, n, period):
    R, P = _gaussian(g, n, sigma=(1e-3, 1e-3, 1e-3))
    R[:, 2] = (torch.rand(n, generator=g, device=_device(), dtype=torch.float64) - 0.5) * (period * 1.05)
    return R, P


def _job_inputs(case, seed):
    g = _gen(seed)
    if case["bins"]:
        return _photoinjector(g, case["n"], case["bins"])
    if case["dc"]:
        return (*_dc(g, case["n"], _period()), None)
    return (*_gaussian(g, case["n"]), None)


def _solve_inputs(case, seed):
    """A Gaussian charge cloud with particle noise in the middle of the mesh."""
    g = _gen(seed)
    axes = [torch.linspace(-3.5, 3.5, case[k], dtype=torch.float64, device=_device()) for k in ("nz", "ny", "nx")]
    z, y, x = torch.meshgrid(*axes, indexing="ij")
    rho = -1e-3 * torch.exp(-0.5 * (x * x + y * y + z * z)) * (1.0 + 0.1 * _randn(g, *x.shape))
    hr = tuple(float(v) for v in 1e-4 * (0.8 + 0.4 * torch.rand(3, generator=g, device=_device(), dtype=torch.float64)))
    return rho, hr, -(case["nz"] + 6.37) * hr[2]


def _batch_jobs(case):
    r = np.random.default_rng(case["jobs_seed"])
    jobs = []
    for _ in range(case["count"]):
        jobs.append({"n": int(round(math.exp(r.uniform(math.log(1e4), math.log(5e5))))),
                     "mesh": int(r.choice([16, 32, 48, 64])), "sigma": [float(v) for v in r.uniform(0.5e-3, 3e-3, 3)],
                     "q": float(r.uniform(0.1, 2.0)) * 1e-9, "bg": float(r.uniform(2.0, 20.0))})
    return jobs


def _pinned(t):
    """Page-locked host memory, as a tracker that hands its arrays to a GPU keeps them."""
    t = t.cpu().contiguous()
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def _pinned_empty(n):
    return torch.empty((n, 3), dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("solve", "image"):
        rho, hr, zshift = _solve_inputs(case, seed)
        s["ctx"] = scgpu.Context((case["nx"], case["ny"], case["nz"]), bboxincr=BBOXINCR)
        s["stream"] = torch.cuda.Stream()
        s["ctx"].set_stream(s["stream"].cuda_stream)
        s["rho"], s["buf"] = rho, torch.empty_like(rho)
        s["hr"], s["zshift"] = (ctypes.c_double * 3)(*hr), zshift
        torch.cuda.synchronize()
    elif kind == "fields":
        g = _gen(seed)
        R, P = _gaussian(g, case["n"], sigma=(1e-3, 1e-3, 2e-2))
        s["R"], s["P"] = R.cpu().numpy(), P.cpu().numpy()
        s["ctx"] = scgpu.Context((case["nx"], case["ny"], case["nz"]), bboxincr=BBOXINCR)
    elif kind == "job":
        R, P, bins = _job_inputs(case, seed)
        s["R"], s["P"] = _pinned(R), _pinned(P)
        s["R1"], s["P1"] = _pinned_empty(case["n"]), _pinned_empty(case["n"])
        s["bins"] = None if bins is None else bins.cpu().numpy()
        s["ctx"] = scgpu.Context((case["nx"], case["ny"], case["nz"]),
                                 precision=scgpu.MIXED if case["mixed"] else scgpu.PLAIN_FP64, bboxincr=BBOXINCR)
        if case["dc"]:
            s["ctx"].set_periodic_z(True)
            s["ctx"].set_beam_frequency(C_LIGHT / _period())
        if case["stat_every"]:
            s["stats"] = np.empty((case["steps"] // case["stat_every"], scgpu.NSTATS))
    else:
        g = _gen(seed)
        s["jobs"] = _batch_jobs(case)
        s["in"], s["out"] = [], []
        for j in s["jobs"]:
            R, P = _gaussian(g, j["n"], sigma=j["sigma"], bg_z=j["bg"])
            s["in"].append((_pinned(R), _pinned(P)))
            s["out"].append((_pinned_empty(j["n"]), _pinned_empty(j["n"])))
        s["batch"] = scgpu.Batch(precision=scgpu.MIXED if case["mixed"] else scgpu.PLAIN_FP64)
    return s


def _q_macro(case):
    return -1e-9 / case["n"]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("solve", "image"):
        L, ctx = scgpu.lib(), s["ctx"]
        with torch.cuda.stream(s["stream"]):
            s["buf"].copy_(s["rho"])
        p = ctypes.cast(s["buf"].data_ptr(), ctypes.POINTER(ctypes.c_double))
        if kind == "solve":
            rc = L.scgpu_compute_potential_device(ctx.h, p, s["hr"])
        else:
            rc = L.scgpu_compute_potential_image_device(ctx.h, p, s["hr"], ctypes.c_double(s["zshift"]))
        ctx._check(rc, kind)
        return {"phi": s["buf"]}
    if kind == "fields":
        Ef, Bf, q = s["ctx"].compute_self_fields(s["R"], s["P"], _q_macro(case), DT)
        return {"E": Ef, "B": Bf, "q": q}
    if kind == "job":
        ctx = s["ctx"]
        ctx.upload(s["R"], s["P"], DT, _q_macro(case), MASS_EV, charge=CHARGE, coupling=COUPLING, bz_ext=case["bz"])
        if case["bins"]:
            ctx.set_energy_bins(s["bins"], case["bins"])
        out = {}
        every = case["stat_every"]
        if every:
            for k in range(case["steps"] // every):
                ctx.track(every - 1)
                ctx.track(1, s["stats"][k:k + 1])
            ctx.track(case["steps"] % every)
            out["stats"] = s["stats"]
        else:
            ctx.track(case["steps"])
        out["R"], out["P"] = ctx.download(s["R1"], s["P1"])
        return out
    b = s["batch"]
    slots = []
    for j, (R, P) in zip(s["jobs"], s["in"]):
        slots.append(b.add((j["mesh"],) * 3, R, P, DT, -j["q"] / j["n"], MASS_EV, bboxincr=BBOXINCR, charge=CHARGE,
                           coupling=COUPLING, ref_P=(0.0, 0.0, j["bg"])))
    for _ in range(case["rounds"]):
        b.track(case["steps"])
    out = {}
    for i, (slot, (R, P)) in enumerate(zip(slots, s["out"])):
        b.member(slot).download(R, P)
        b.remove(slot)
        out["R%02d" % i], out["P%02d" % i] = R, P
    return out


# -------------------------------------------------------------------- work
def _solve_work(nx, ny, nz):
    """The charge read and the potential written once; the pruned doubled-grid
    transforms (rho forward, phi inverse, cosine transforms of G: together
    about the work of two full real transforms) and about 200 operations per
    point of the Green's function."""
    m = nx * ny * nz
    v = 8 * m
    return 16 * m, 2 * 2.5 * v * math.log2(max(v, 2)) * 0.6 + 200 * (nx + 2) * (ny + 2) * (nz + 2)


def work(case):
    kind = case["kind"]
    if kind in ("solve", "image"):
        by, fl = _solve_work(case["nx"], case["ny"], case["nz"])
        return {"bytes": by, "flops": fl}
    if kind == "fields":
        by, fl = _solve_work(case["nx"], case["ny"], case["nz"])
        return {"bytes": by + 96 * case["n"], "flops": fl + 150 * case["n"]}
    if kind == "job":
        by, fl = _solve_work(case["nx"], case["ny"], case["nz"])
        k = max(1, 2 * case["bins"])
        # a step reads and writes positions and momenta once
        return {"bytes": case["steps"] * (96 * case["n"] + k * by) + 192 * case["n"],
                "flops": case["steps"] * (k * fl + 400 * case["n"])}
    by = fl = 0
    steps = case["rounds"] * case["steps"]
    for j in _batch_jobs(case):
        b1, f1 = _solve_work(j["mesh"], j["mesh"], j["mesh"])
        by += steps * (96 * j["n"] + b1) + 192 * j["n"]
        fl += steps * (f1 + 400 * j["n"])
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------------------- exact
def _antiderivative(nr, hr, z0):
    x, y, z = (torch.arange(nr[d] + 2, dtype=torch.float64, device=_device()) * hr[d] - hr[d] / 2 for d in range(3))
    z = (z + z0)[:, None, None]
    y, x = y[None, :, None], x[None, None, :]
    r = torch.sqrt(x * x + y * y + z * z)
    t = -z * z * torch.atan(x * y / (z * r)) / 2 - y * y * torch.atan(x * z / (y * r)) / 2
    t = t - x * x * torch.atan(y * z / (x * r)) / 2
    t = t + y * z * torch.log(x + r) + x * z * torch.log(y + r) + x * y * torch.log(z + r)
    return t / (hr[0] * hr[1] * hr[2])


def _corners(t):
    for d in range(3):
        t = t.diff(dim=d)
    return t


def _mirror(g, dim, n):
    """Offsets 0..n along dim to the 2n offsets of the doubled axis."""
    return torch.cat([g, g.narrow(dim, 1, n - 1).flip(dim)], dim)


def _potential(rho, hr, zshift=None, periodic=False):
    """rho [nz, ny, nx]; the convolution with the integrated Green's function
    on the doubled grid (zshift: the image charge's, z flipped)."""
    nz, ny, nx = rho.shape
    nr = (nx, ny, nz)
    if zshift is None:
        g = _corners(_antiderivative(nr, hr, 0.0))
        g[0, 0, 0] = g[1, 0, 0]
        g = g[:nz] if periodic else _mirror(g, 0, nz)
    else:
        ga = _corners(_antiderivative(nr, hr, zshift))
        gb = _corners(_antiderivative(nr, hr, zshift - nz * hr[2]))
        g = torch.cat([ga, gb[1:nz]], 0)
    g = _mirror(_mirror(g, 1, ny), 2, nx)
    shape = g.shape
    phi = torch.fft.irfftn(torch.fft.rfftn(rho, s=shape) * torch.fft.rfftn(g), s=shape)[:nz, :ny, :nx]
    return phi.clone() if zshift is None else -phi.flip(0)


def _quaternion(u, ref=(0.0, 0.0, 1.0)):
    lu, lr = math.sqrt(sum(v * v for v in u)), math.sqrt(sum(v * v for v in ref))
    u, ref = [v / lu for v in u], [v / lr for v in ref]
    ax = [u[1] * ref[2] - u[2] * ref[1], u[2] * ref[0] - u[0] * ref[2], u[0] * ref[1] - u[1] * ref[0]]
    na = math.sqrt(sum(v * v for v in ax))
    if na < 1e-12:
        return (1.0, 0.0, 0.0, 0.0)
    ca = math.sqrt(0.5 * (1 + sum(a * b for a, b in zip(u, ref))))
    sa = math.sqrt(1 - ca * ca)
    return (ca, *(sa * v / na for v in ax))


def _rotation(q):
    w, x, y, z = q
    return torch.tensor([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (w * y + x * z)],
                         [2 * (w * z + x * y), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                         [2 * (x * z - w * y), 2 * (w * x + y * z), 1 - 2 * (x * x + y * y)]],
                        dtype=torch.float64, device=_device())


def _grad(phi, h):
    """-grad phi, one-sided at the faces: [nz, ny, nx, 3]."""
    out = []
    for d, dim in ((0, 2), (1, 1), (2, 0)):
        p = phi.movedim(dim, 0)
        e = torch.empty_like(p)
        e[1:-1] = p[2:] - p[:-2]
        e[0] = -p[2] + 4 * p[1] - 3 * p[0]
        e[-1] = p[-3] - 4 * p[-2] + 3 * p[-1]
        out.append(-(e * (0.5 / h[d])).movedim(0, dim))
    return torch.stack(out, -1)


def _boundp(R, nr, period):
    lo, hi = R.amin(0).tolist(), R.amax(0).tolist()
    h = [0.0] * 3
    for d in range(3):
        if d == 2 and period:
            hi[d] = lo[d] + period
        else:
            e = BBOXINCR / 100 * (hi[d] - lo[d])
            lo[d], hi[d] = lo[d] - e, hi[d] + e
        h[d] = (hi[d] - lo[d]) / (nr[d] - 1)
    return h, [lo[d] - h[d] / 2 for d in range(3)]


def _stencil(R, nr, h, org):
    """Corner nodes and weights of every particle; planes outside z get the periodic image and a flag."""
    u = (R - R.new_tensor(org)) / R.new_tensor(h) - 0.5
    f = torch.floor(u)
    d, base = u - f, f.long()
    for c in range(8):
        o = (c & 1, (c >> 1) & 1, c >> 2)
        w = 1.0
        for a in range(3):
            w = w * (d[:, a] if o[a] else 1 - d[:, a])
        k = base[:, 2] + o[2]
        inside = (k >= 0) & (k < nr[2])
        yield base[:, 0] + o[0] + nr[0] * (base[:, 1] + o[1] + nr[1] * (k % nr[2])), w, inside


def _deposit(R, q, nr, h, org):
    rho = torch.zeros(nr[0] * nr[1] * nr[2], dtype=torch.float64, device=R.device)
    for node, w, inside in _stencil(R, nr, h, org):
        rho.index_add_(0, node, w * inside * q)
    return rho.view(nr[2], nr[1], nr[0])


def _gather(R, E, nr, h, org):
    E = E.reshape(-1, E.shape[-1])
    out = torch.zeros((R.shape[0], E.shape[1]), dtype=torch.float64, device=R.device)
    for node, w, _ in _stencil(R, nr, h, org):
        out += w[:, None] * E[node]
    return out


def _self_fields(R, P, q, nr, bins=None, nbins=0, period=0.0):
    """computeSelfFields in the beam frame (R is wrapped in place for a DC beam): E, B per particle."""
    h, org = _boundp(R, nr, period)
    if period:
        top = org[2] + h[2] * nr[2]
        z = R[:, 2]
        z.copy_(torch.where(z < org[2], top - (org[2] - z), torch.where(z >= top, org[2] + (z - top), z)))
    F = torch.zeros((nr[2], nr[1], nr[0], 6), dtype=torch.float64, device=R.device)
    for b in range(max(nbins, 1)):
        sel = bins == b if nbins else None
        if nbins:
            gz = float(torch.sqrt(1 + (P[sel] ** 2).sum(1)).mean())
        else:
            gz = math.sqrt(float(P[:, 2].mean()) ** 2 + 1)
        hs = (h[0], h[1], h[2] * gz)
        vol = hs[0] * hs[1] * hs[2]
        rho = _deposit(R[sel] if nbins else R, q, nr, h, org) / vol
        scale = torch.tensor([gz, gz, 1 / gz], dtype=torch.float64, device=R.device) * vol * COUPLING
        bc = math.sqrt(gz * gz - 1) / gz / C_LIGHT
        for image in range(2 if nbins else 1):
            zs = -(2 * org[2] + nr[2] * h[2]) * gz if image else None
            E = _grad(_potential(rho, hs, zs, period > 0), h) * scale
            sign = -1.0 if image else 1.0
            F[..., :3] += E
            F[..., 3] -= sign * bc * E[..., 1]
            F[..., 4] += sign * bc * E[..., 0]
    f = _gather(R, F, nr, h, org)
    return f[:, :3].contiguous(), f[:, 3:].contiguous()


def _push(R, P, dt):
    return R + (0.5 * C_LIGHT * dt) * P / torch.sqrt(1 + (P * P).sum(1, keepdim=True))


def _kick(P, E, B, dt):
    ke = 0.5 * dt * CHARGE * C_LIGHT / MASS_EV
    P = P + ke * E
    g = torch.sqrt(1 + (P * P).sum(1, keepdim=True))
    t = (0.5 * dt * CHARGE * C_LIGHT ** 2 / MASS_EV) / g * B
    w = P + torch.linalg.cross(P, t)
    P = P + torch.linalg.cross(w, 2.0 / (1.0 + (t * t).sum(1, keepdim=True)) * t)
    return P + ke * E


def _moments(R, P):
    v = torch.stack([R[:, 0], P[:, 0], R[:, 1], P[:, 1], R[:, 2], P[:, 2]], 1)
    m = v.T @ v
    return [*v.sum(0).tolist(), *(float(m[i, j]) for i in range(6) for j in range(i + 1)),
            float(torch.sqrt(1 + (P * P).sum(1)).sum())]


def _track(R, P, q, nr, steps, bz=0.0, ref_pz=10.0, bins=None, nbins=0, period=0.0, stat_every=0):
    ref_R = torch.zeros((1, 3), dtype=torch.float64, device=R.device)
    ref_P = torch.tensor([[0.0, 0.0, ref_pz]], dtype=torch.float64, device=R.device)
    path, stats = 0.0, []
    for k in range(steps):
        R = _push(R, P, DT)
        M = _rotation([v * s for v, s in zip(_quaternion(P.mean(0).tolist()), (1, -1, -1, -1))])  # beam -> reference
        org = torch.tensor([0.0, 0.0, path], dtype=torch.float64, device=R.device)
        R = R @ M + org
        E, B = _self_fields(R, P, q, nr, bins, nbins, period)
        R, E, B = (R - org) @ M.T, E @ M.T, B @ M.T
        B[:, 2] += bz
        P = _kick(P, E, B, DT)
        R = _push(R, P, DT)
        zero = torch.zeros_like(ref_P)
        bref = zero.clone()
        bref[0, 2] = bz
        ref_R = _push(ref_R, ref_P, DT)
        ref_P = _kick(ref_P, zero, bref, DT)
        ref_R = _push(ref_R, ref_P, DT)
        path += float(ref_R.norm())
        U = _rotation(_quaternion(ref_P[0].tolist()))
        R, P = (R - ref_R) @ U.T, P @ U.T
        ref_R, ref_P = (ref_R - ref_R) @ U.T, ref_P @ U.T
        if stat_every and (k + 1) % stat_every == 0:
            stats.append(_moments(R, P))
    return R, P, stats


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "image"):
        rho, hr, zshift = _solve_inputs(case, seed)
        return {"phi": _potential(rho, hr, zshift if kind == "image" else None)}
    if kind == "fields":
        R, P = _gaussian(_gen(seed), case["n"], sigma=(1e-3, 1e-3, 2e-2))
        E, B = _self_fields(R, P, _q_macro(case), (case["nx"], case["ny"], case["nz"]))
        return {"E": E.cpu().numpy(), "B": B.cpu().numpy(), "q": _q_macro(case)}
    if kind == "job":
        R, P, bins = _job_inputs(case, seed)
        R, P, stats = _track(R, P, _q_macro(case), (case["nx"], case["ny"], case["nz"]), case["steps"], case["bz"],
                             bins=bins, nbins=case["bins"], period=_period() if case["dc"] else 0.0,
                             stat_every=case["stat_every"])
        out = {"R": R.cpu().numpy(), "P": P.cpu().numpy()}
        if stats:
            out["stats"] = np.array(stats)
        return out
    g = _gen(seed)
    out = {}
    jobs = _batch_jobs(case)
    bunches = [_gaussian(g, j["n"], sigma=j["sigma"], bg_z=j["bg"]) for j in jobs]
    for i, (j, (R, P)) in enumerate(zip(jobs, bunches)):
        R, P, _ = _track(R, P, -j["q"] / j["n"], (j["mesh"],) * 3, case["rounds"] * case["steps"], ref_pz=j["bg"])
        out["R%02d" % i], out["P%02d" % i] = R.cpu().numpy(), P.cpu().numpy()
    return out
