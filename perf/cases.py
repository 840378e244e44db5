"""Workloads of the sky-map projection, from the smallest call to the largest.

Every case is one call that a program makes through the Python package or the
C ABI: a single map (``Renderer.render``), a batch of observers
(``render_batch``), the chunked file flow (``MapGenerator.start``), the
allocation-free render (``dmann_render_noalloc``), the gradient of a map
(``Renderer.adjoint``) and the differentiable map of a training loop
(``autograd.sky_map``).

Particles are an NFW host (rs 20 kpc, r200 400 kpc) with NFW subhalos holding
a tenth of them, observed from 8 kpc: the synthetic set of
``annmap.synth.nfw_halo``, drawn here on the GPU.  ``n_total`` says how many
particles the whole simulation has: the n particles of a call are a random
sample of it, so they have its densities, smoothing lengths and disc sizes
(``n == n_total`` renders the whole set).  Names give the particle count, the
Nside and the precision form.
"""
import ctypes as C
import math
import os
import sys
import tempfile

import numpy as np
import torch

_PKG = os.path.join("dm-annihilation-cxx_gb300", "pywrapper")
for _base in (os.getcwd(), os.path.dirname(os.path.dirname(os.path.abspath(__file__)))):
    if os.path.isdir(os.path.join(_base, _PKG)):
        sys.path.insert(0, os.path.join(_base, _PKG))
        break

import annmap  # noqa: E402
from annmap import _lib, autograd, synth  # noqa: E402

MASS = 4.1e3          # Msun, at 2^24 particles
FIELDS = ("x", "y", "z", "m", "rho", "h")


# ------------------------------------------------------------------ the cases
def _case(name, op, n, n_total, nside, precision, *, subs=0, near=0, law="ann_nosom", observers=1, chunk=0):
    c = {"op": op, "n": n, "n_total": n_total, "nside": nside, "precision": precision, "subs": subs,
         "near": near, "law": law, "observers": observers, "chunk": chunk}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the first thousand particles of a large snapshot on a coarse map:
        # the "test" key of an info file, a quick look, a unit test
        _case("look 1k ns64", "render", 1000, 1 << 24, 64, "comp", subs=100),
        # a small halo on a coarse map of its own resolution, odd counts
        _case("halo 20k ns96", "render", 20011, 1 << 20, 96, "comp", subs=6),
        # the whole small configuration: 1,048,576 particles at Nside 512
        _case("nfw 1M ns512", "render", 1 << 20, 1 << 20, 512, "comp"),
        # the headline configuration: 16,777,216 particles, 100 subhalos, Nside 2048
        _case("nfw 16M ns2048", "render", 1 << 24, 1 << 24, 2048, "comp", subs=100),
        # one chunk of the large-map configuration: Nside 4096, some particles
        # within 0.5 kpc of the observer with discs up to the whole sky
        _case("near 2M ns4096", "render", 2000003, 1 << 27, 4096, "comp", subs=500, near=150),
        # a large set on a coarse map: discs of a few to some hundred pixels
        _case("coarse 8M ns128", "render", 1 << 23, 1 << 23, 128, "comp", subs=50),
        # six observers with mixed Nside over one particle set, one batch call
        _case("batch 1M x6", "batch", 1 << 20, 1 << 23, 512, "comp", subs=50, observers=6),
        # the reference program's flow: a particle file on disk read in chunks
        # (host memory in, host map out), a velocity-dependent flux law
        _case("file 1.5M ns512 somv", "file", 1500007, 1 << 24, 512, "comp", subs=100, law="ann_somv",
              chunk=400000),
        # the plain FP64 form, the reference's arithmetic, on a sample of the small configuration
        _case("plain 16k ns512", "render", 1 << 14, 1 << 20, 512, "plain"),
        # the gradient of a map for a training loop, FP32 weights
        _case("adjoint 1M ns512", "adjoint", 1 << 20, 1 << 22, 512, "comp", subs=20),
        # forward and backward of the differentiable map at its default precision (FP64)
        _case("sky_map 4k ns512 f64", "grad", 4096, 1 << 22, 512, "plain", subs=20),
        # a plug-in that may not allocate device memory
        _case("noalloc 100k ns256", "noalloc", 100003, 1 << 20, 256, "comp", subs=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["render", "render", "render", "render", "batch", "file", "plain", "adjoint", "grad", "noalloc"])
    total = rng.choice([1 << 20, 1 << 22, 1 << 23, 1 << 24, 1 << 27])
    subs = rng.choice([0, 6, 20, 50, 100])
    n = lambda lo, hi: min(total, _log(rng, lo, hi) | 1)   # odd counts  # noqa: E731
    if op == "render":
        nside = _log(rng, 64, 4096)
        # the particle budget keeps the pixels visited below the largest listed case's
        px = 17000.0 * (nside / 512.0) ** 2 * (2.0 ** 20 / total) ** (2.0 / 3.0)
        law = rng.choice(["ann_nosom", "ann_nosom", "decay", "ann_pwave"])
        return _case(None, "render", n(800, max(2000, min(1 << 24, int(2e11 / px)))), total, nside, "comp", subs=subs,
                     near=rng.choice([0, 0, 20]), law=law)
    if op == "batch":
        return _case(None, "batch", n(20000, 1 << 20), 1 << 23, rng.choice([128, 256, 512]), "comp", subs=subs,
                     observers=rng.randint(2, 8))
    if op == "file":
        return _case(None, "file", n(50000, 2000000), total, _log(rng, 64, 512), "comp", subs=subs,
                     law=rng.choice(["ann_nosom", "ann_somv", "ann_somv2"]), chunk=_log(rng, 50000, 1000000))
    if op == "plain":
        return _case(None, "render", n(500, 1 << 14), total, _log(rng, 32, 512), "plain", subs=subs)
    if op == "adjoint":
        return _case(None, "adjoint", n(3000, 1 << 20), 1 << 22, _log(rng, 64, 512), "comp", subs=subs,
                     law=rng.choice(["ann_nosom", "decay"]))
    if op == "grad":
        return _case(None, "grad", n(500, 4096), 1 << 22, _log(rng, 64, 512), "plain", subs=subs)
    return _case(None, "noalloc", n(1000, 200000), max(total, 1 << 20), _log(rng, 32, 256), "comp", subs=subs)


# ------------------------------------------------------------------ particles
def _mu(x):
    return torch.log1p(x) - x / (1.0 + x)


def _iso(g, n):
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    ph = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)
    s = torch.sqrt((1 - u * u).clamp_min(0))
    return torch.stack([s * torch.cos(ph), s * torch.sin(ph), u], 1)


def _nfw(g, n, rs, mass, centre, m):
    """n particles of an NFW halo of concentration synth.CONC that holds `mass`."""
    grid = torch.cat([torch.zeros(1, device="cuda", dtype=torch.float64),
                      torch.logspace(-6, math.log10(synth.CONC), 8192, device="cuda", dtype=torch.float64)])
    mg = _mu(grid)
    q = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * mg[-1]
    k = torch.searchsorted(mg, q).clamp(1, len(grid) - 1)
    x = grid[k - 1] + (grid[k] - grid[k - 1]) * ((q - mg[k - 1]) / (mg[k] - mg[k - 1]))
    x = x.clamp_min(1e-6)
    rho_s = mass / (4 * math.pi * rs ** 3 * float(mg[-1]))
    rho = rho_s / (x * (1 + x) ** 2)
    rho = rho * torch.exp(0.3 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
    pos = torch.as_tensor(centre, device="cuda", dtype=torch.float64)[None] + _iso(g, n) * (x * rs)[:, None]
    return pos, rho, (32.0 * m / (4.0 * math.pi / 3.0 * rho)) ** (1.0 / 3.0)


def _particles(case, seed):
    """Float32 CUDA tensors x, y, z, m, rho, h (and sigmav) and the particle mass."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + 17)
    n, near, total, subs = case["n"], case["near"], case["n_total"], case["subs"]
    m = MASS if total <= 1 << 24 else MASS * (1 << 24) / total
    n_halo = n - near
    n_sub = int(0.1 * n_halo) if subs else 0
    n_host = n_halo - n_sub
    m_host = (0.9 if subs else 1.0) * total * m
    parts = [_nfw(g, n_host, synth.RS_HOST, m_host, (0.0, 0.0, 0.0), m)]
    if subs:
        msub = 10.0 ** (6.0 + 3.0 * torch.rand(subs, generator=g, device="cuda", dtype=torch.float64))
        c = _iso(g, subs) * (synth.SUB_RMAX * torch.rand(subs, generator=g, device="cuda", dtype=torch.float64)
                             ** (1.0 / 3.0))[:, None]
        count = torch.bincount(torch.multinomial(msub / msub.sum(), max(1, n_sub), replacement=True, generator=g),
                               minlength=subs).tolist() if n_sub else [0] * subs
        share = (msub / msub.sum()).tolist()
        for j, (ms, cc) in enumerate(zip(msub.tolist(), c.tolist())):
            if count[j]:
                rs = synth.R200_HOST * (ms / m_host) ** (1.0 / 3.0) / synth.CONC
                parts.append(_nfw(g, count[j], rs, share[j] * 0.1 * total * m, cc, m))
    if near:
        obs = torch.tensor(synth.default_observer(), device="cuda", dtype=torch.float64)
        d = 0.5 * torch.rand(near, generator=g, device="cuda", dtype=torch.float64) ** (1.0 / 3.0)
        pos = obs[None] + _iso(g, near) * d[:, None]
        rr = pos.norm(dim=1) / synth.RS_HOST
        rho = m_host / (4 * math.pi * synth.RS_HOST ** 3 * (math.log(21.0) - 20.0 / 21.0)) / (rr * (1 + rr) ** 2)
        parts.append((pos, rho, (32.0 * m / (4.0 * math.pi / 3.0 * rho)) ** (1.0 / 3.0)))
    pos, rho, h = (torch.cat([p[k] for p in parts]) for k in range(3))
    perm = torch.randperm(n, generator=g, device="cuda")
    f = lambda t: t[perm].to(torch.float32).contiguous()  # noqa: E731
    out = {"x": f(pos[:, 0]), "y": f(pos[:, 1]), "z": f(pos[:, 2]),
           "m": torch.full((n,), m, device="cuda", dtype=torch.float32), "rho": f(rho), "h": f(h)}
    # velocity dispersion in code units: 0 to 300 km/s, and a few at rest
    if case["law"] in ("ann_somv", "ann_somv2", "ann_pwave"):
        par = _params(case, m)
        v = 300.0 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64) ** 2
        out["sigmav"] = (v * 1e5 / par.codeunits.velocity_to_cgs).to(torch.float32)
    return out, m


def _params(case, m, obs=None, nside=None):
    """The parameters of an info file: 1 kpc code length, masses in Msun."""
    obs = obs or synth.default_observer()
    return annmap.Parameters(text="\n".join([
        "Omega_M = 0.238", "h100 = 0.73", "Lbox_in_Mpc = 0.001", "mass_to_Msun = 1", f"particle_masses = {m!r}",
        "centerpos = 0 0 0", "align_vec = 0 0 1", "obs_pos = " + " ".join(repr(float(v)) for v in obs),
        f"nside = {nside or case['nside']}"]) + "\n")


def _observers(case, seed):
    """(observer, Nside) of a batch: uniform on the 8 kpc sphere, Nside / 2, Nside, 2 Nside in turn."""
    ns = case["nside"]
    return synth.batched_observers(case["observers"], seed=int(seed), nsides=(ns // 2, ns, 2 * ns))


def _prec(case):
    return annmap.COMP_F32 if case["precision"] == "comp" else annmap.PLAIN_F64


def _gmap(case, seed):
    """dL/dmap of a pixelwise loss: random signs and sizes."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 3)
    return torch.randn(12 * case["nside"] ** 2, generator=g, device="cuda", dtype=torch.float64)


class _File:
    """A native particle file that goes away with the state."""

    def __init__(self, parts):
        fd, self.path = tempfile.mkstemp(suffix=".bin")
        os.close(fd)
        host = {k: v.cpu().numpy() for k, v in parts.items()}
        annmap.write_native(self.path, {k: host[k] for k in FIELDS},
                            {"sigmav": host["sigmav"]} if "sigmav" in host else None)

    def __del__(self):
        try:
            os.unlink(self.path)
        except OSError:
            pass


def prepare(case, seed):
    parts, m = _particles(case, seed)
    s = {"case": case, "parts": parts, "par": _params(case, m)}
    op, ns = case["op"], case["nside"]
    if op == "file":
        s["file"] = _File(parts)
        del s["parts"]
        return s
    if op == "grad":
        s["parts"] = {k: v.requires_grad_() for k, v in parts.items()}
        s["opos"] = torch.tensor(s["par"].params.opos, dtype=torch.float64, requires_grad=True)
        s["gmap"] = _gmap(case, seed)
        return s
    if op == "noalloc":
        s["lib"] = _lib.load()
        s["out"] = torch.zeros(12 * ns * ns, device="cuda", dtype=torch.float64)
        s["rot"] = (C.c_double * 9)(*s["par"].rot_flat())
        s["op"] = (C.c_double * 3)(*s["par"].params.opos)
        return s
    s["r"] = annmap.Renderer(0)
    s["r"].set_params(s["par"], case["law"])
    if op == "batch":
        s["frames"], s["nsides"] = [], []
        for obs, k in _observers(case, seed):
            p = _params(case, m, obs, k)
            s["frames"].append((p.rotmatrix, p.params.opos))
            s["nsides"].append(k)
        s["outs"] = [torch.zeros(12 * k * k, device="cuda", dtype=torch.float64) for k in s["nsides"]]
    elif op == "adjoint":
        s["gmap"] = _gmap(case, seed)
    else:
        s["out"] = torch.zeros(12 * ns * ns, device="cuda", dtype=torch.float64)
    return s


def run(s):
    case = s["case"]
    op, ns, prec = case["op"], case["nside"], _prec(case)
    if op == "render":
        return s["r"].render(s["parts"], ns, prec, out=s["out"])
    if op == "batch":
        return s["r"].render_batch(s["parts"], s["frames"], s["nsides"], prec, outs=s["outs"])
    if op == "file":
        reader = annmap.DataReader(s["file"].path)
        reader.setBuf(case["chunk"])
        reader.open()
        gen = annmap.MapGenerator(s["par"], reader, precision=prec, flux_model=case["law"])
        gen.start()
        reader.close()
        return gen.getMap()
    if op == "adjoint":
        g, go = s["r"].adjoint(s["parts"], ns, s["gmap"], precision=prec)
        return {"grad": g, "observer": go}
    if op == "grad":
        p = s["parts"]
        for t in (*p.values(), s["opos"]):
            t.grad = None
        par = s["par"]
        mp = autograd.sky_map(*[p[k] for k in FIELDS], s["opos"], nside=ns, unit_factor=par.unit_factor,
                              hires_threshold=par.hires_threshold)
        mp.backward(s["gmap"])
        return {"map": mp.detach(), "grads": [p[k].grad for k in FIELDS], "observer": s["opos"].grad}
    st = s["lib"].dmann_render_noalloc(
        *[C.c_void_p(s["parts"][k].data_ptr()) for k in FIELDS], case["n"], ns, s["rot"], s["op"],
        s["par"].unit_factor, s["par"].hires_threshold, C.c_void_p(s["out"].data_ptr()), 0,
        C.c_void_p(torch.cuda.current_stream().cuda_stream) if torch.cuda.current_stream().cuda_stream else None)
    if st != _lib.OK:
        raise RuntimeError("dmann_render_noalloc: %d" % st)
    return s["out"]


# ------------------------------------------------------------------ the work
def _views(case, seed):
    if case["op"] == "batch":
        return _observers(case, seed)
    return [(synth.default_observer(), case["nside"])]


def _pixels(case):
    """Pixels of all discs of one pass (cap areas of a sample of the particles)."""
    n = min(case["n"], 50000)
    near = max(1, case["near"] * n // case["n"]) if case["near"] else 0
    parts, m = _particles(dict(case, n=n, near=near, law="ann_nosom"), 1)
    tot = 0.0
    for obs, ns in _views(case, 1):
        o = torch.tensor(obs, device="cuda", dtype=torch.float64)
        d = (torch.stack([parts["x"], parts["y"], parts["z"]], 1).double() - o).norm(dim=1)
        ar = parts["h"].double() / d
        px = 12 * ns * ns * torch.sin(ar.clamp(max=math.pi / 2)) ** 2
        if near:   # weight the near-observer particles by their share of the call
            px = px.sort().values
            tot += float(px[:-near].mean()) * (case["n"] - case["near"]) + float(px[-near:].mean()) * case["near"]
        else:
            tot += float(px.clamp_min(1.0).mean()) * case["n"]
    return tot


def work(case):
    """Bytes: each input read once, each output written once.  Operations per
    disc pixel: a weight is the squared distance (8), the exponential (2) and
    its share of the disc's sum (1); the render multiplies and adds it into
    the map (2); the gradient adds the tangent sums (30)."""
    px = _pixels(case)
    maps = sum(8.0 * 12 * ns * ns for _, ns in _views(case, 1))
    n, op = case["n"], case["op"]
    flops = {"adjoint": 41.0, "grad": 54.0}.get(op, 13.0) * px
    inputs = (48.0 if op == "file" else 24.0) * n + (4.0 * n if case["law"] == "ann_pwave" else 0.0)
    grads = {"adjoint": 48.0 * n, "grad": 24.0 * n}.get(op, 0.0)
    return {"bytes": inputs + grads + maps * (2.0 if op == "grad" else 1.0), "flops": flops}


# ------------------------------------------------------------------ 64-bit values
def _rings(nside, r):
    """z, sin(theta), pixels, first pixel and half-pixel shift of RING rings r (1 .. 4 nside - 1)."""
    npix = 12 * nside * nside
    rd = r.double()
    north, south = r < nside, r > 3 * nside
    i = torch.where(north, r, torch.where(south, 4 * nside - r, torch.full_like(r, nside)))
    id_ = i.double()
    cap = 1.0 - id_ * id_ * (4.0 / npix)
    z = torch.where(north, cap, torch.where(south, -cap, (2 * nside - rd) * (8.0 * nside / npix)))
    t = id_ * id_ * (4.0 / npix)
    st = torch.where(north | south, torch.sqrt(t * (2 - t)), torch.sqrt((1 - z) * (1 + z)))
    nr = 4 * i
    start = torch.where(north, 2 * i * (i - 1),
                        torch.where(south, npix - 2 * i * (i + 1), 2 * nside * (nside - 1) + (r - nside) * 4 * nside))
    shift = torch.where(north | south | (((r - nside) & 1) == 0), 0.5, 0.0)
    return z, st, nr, start, shift


def _ring_above(nside, z):
    az = z.abs()
    eq = (nside * (2 - 1.5 * z)).long()
    cap = (nside * torch.sqrt((3 * (1 - az)).clamp_min(0))).long()
    return torch.where(az <= 2.0 / 3.0, eq, torch.where(z > 0, cap, 4 * nside - cap - 1))


def _centre_pixel(nside, z, st, phi):
    npix = 12 * nside * nside
    tt = torch.remainder(phi * (2 / math.pi), 4.0)
    za = z.abs()
    t1, t2 = nside * (0.5 + tt), nside * z * 0.75
    jp, jm = (t1 - t2).long(), (t1 + t2).long()
    ir = nside + 1 + jp - jm
    ks = 1 - (ir & 1)
    ip = torch.remainder((jp + jm - nside + ks + 1 + 8 * nside) >> 1, 4 * nside)
    eq = 2 * nside * (nside - 1) + (ir - 1) * 4 * nside + ip
    tp = tt - tt.floor()
    tmp = torch.where(za < 0.99, nside * torch.sqrt((3 * (1 - za)).clamp_min(0)), nside * st / torch.sqrt((1 + za) / 3))
    jp, jm = (tp * tmp).long(), ((1 - tp) * tmp).long()
    ir = jp + jm + 1
    ip = torch.minimum((tt * ir).long(), 4 * ir - 1)
    cap = torch.where(z > 0, 2 * ir * (ir - 1) + ip, npix - 2 * ir * (ir + 1) + ip)
    return torch.where(za <= 2.0 / 3.0, eq, cap)


def _flux(case, par, p, d):
    law = case["law"]
    mass, dens = p["m"].double(), p["rho"].double()
    if law == "decay":
        return par.flux_unit_factor(law) * mass / (4 * math.pi * d * d)
    f = par.flux_unit_factor(law) * dens * mass / (4 * math.pi * d * d)
    if law == "ann_nosom":
        return f
    v = p["sigmav"].double() * par.codeunits.velocity_to_cgs
    c = 2.99792458e10
    if law == "ann_somv":
        return f * c / (v / 1e5).clamp_min(1.0) / 1e4
    if law == "ann_somv2":
        return f * (c / (v / 1e5).clamp_min(5.0)) ** 2 / 1e8
    return f * (v / c) ** 2


def _expand(start, count):
    """(owner, start[owner] + 0, 1, ... count[owner] - 1) of every owner."""
    own = torch.repeat_interleave(torch.arange(len(count), device="cuda"), count)
    first = torch.cumsum(count, 0) - count
    return own, start[own] + (torch.arange(len(own), device="cuda") - first[own])


def _exact_view(case, par, parts, nside, gmap=None):
    """One map in 64 bits, or with gmap the [6, n] gradients of sum(gmap * map)."""
    f64 = torch.float64
    npix = 12 * nside * nside
    dom = 4 * math.pi / npix
    rot = torch.tensor(par.rotmatrix, device="cuda", dtype=f64)
    u = torch.stack([parts[k] for k in "xyz"], 1).double() - torch.tensor(par.params.opos, device="cuda", dtype=f64)
    d = u.norm(dim=1)
    flux = _flux(case, par, parts, d)
    w = (u @ rot) / d[:, None]                       # rot^T u / d
    nv = torch.stack([-w[:, 0], -w[:, 1], w[:, 2]], 1)   # phi is shifted by pi
    cz = nv[:, 2].clamp(-1, 1)
    st0 = torch.hypot(nv[:, 0], nv[:, 1])
    theta = torch.atan2(st0, cz)
    phi = torch.remainder(torch.atan2(nv[:, 1], nv[:, 0]), 2 * math.pi)
    ar = parts["h"].double() / d
    R = 2 * ar
    cpix = _centre_pixel(nside, cz, st0, phi)
    single = R < math.acos(1 - dom / (2 * 3.141592))
    allsky = R >= math.pi
    lo_lat, hi_lat = theta - R, theta + R
    irmin = torch.where(allsky, 1, _ring_above(nside, torch.cos(lo_lat)) + 1)
    irmax = torch.where(allsky, 0, _ring_above(nside, torch.cos(hi_lat)))
    r0 = torch.where(allsky | ((lo_lat <= 0) & (irmin > 1)), 1, irmin).clamp_min(1)
    r1 = torch.where(allsky | ((hi_lat >= math.pi) & (irmax + 1 < 4 * nside)), 4 * nside - 1, irmax)
    r1 = r1.clamp_max(4 * nside - 1)
    est = (npix * torch.sin(ar.clamp(max=math.pi / 2)) ** 2 + 4 * (r1 - r0 + 1)).clamp_min(1)
    est[single] = 1
    out = torch.zeros(npix, device="cuda", dtype=f64) if gmap is None else torch.zeros(6, len(d), device="cuda", dtype=f64)
    edges = torch.cumsum(est, 0)
    i0 = 0
    while i0 < len(d):   # a few 10^7 pixels at a time
        base = float(edges[i0 - 1]) if i0 else 0.0
        i1 = max(i0 + 1, int(torch.searchsorted(edges, base + 4e7)))
        sl = slice(i0, i1)
        th, ph, a, rr = theta[sl], phi[sl], ar[sl], R[sl]
        nring = torch.where(single[sl], 0, (r1[sl] - r0[sl] + 1).clamp_min(0))
        po, ring = _expand(r0[sl], nring)
        z, st, nr, start, shift = _rings(nside, ring)
        full = allsky[sl][po] | (ring < irmin[sl][po]) | (ring > irmax[sl][po])
        x = (torch.cos(rr)[po] - z * cz[sl][po]) / st0[sl][po]
        ysq = 1 - z * z - x * x
        dphi = torch.atan2(torch.sqrt(ysq.clamp_min(0)), x)
        fnr = nr.double() / (2 * math.pi)
        lo = torch.floor(fnr * (ph[po] - dphi) - shift).long() + 1
        hi = torch.floor(fnr * (ph[po] + dphi) - shift).long()
        cnt = torch.where(full, nr, torch.where(ysq > 0, (hi - lo + 1).clamp_min(0), 0))
        lo = torch.where(full, 0, lo)
        ro, k = _expand(lo, cnt)
        pp = po[ro]
        npx = torch.bincount(pp, minlength=i1 - i0)
        disc = (npx >= 2) & ~single[sl]
        dp = (k.double() + shift[ro]) / fnr[ro] - ph[pp]
        pix = start[ro] + torch.remainder(k, nr[ro])
        thr = torch.atan2(st, z)
        sdt, sdp = torch.sin(0.5 * (thr[ro] - th[pp])), torch.sin(0.5 * dp)
        hav = (sdt * sdt + st[ro] * torch.sin(th)[pp] * sdp * sdp).clamp(0, 1)
        al = 2 * torch.atan2(torch.sqrt(hav), torch.sqrt(1 - hav))
        wt = torch.exp(-0.5 * (al / a[pp]) ** 2 / 0.333)
        add = lambda v: torch.zeros(i1 - i0, device="cuda", dtype=f64).index_add_(0, pp, v)  # noqa: E731
        S = add(wt).clamp_min(1e-300)
        F = flux[sl]
        if gmap is None:
            out.index_add_(0, pix, torch.where(disc[pp], wt / S[pp] * F[pp], 0.0))
            out.index_add_(0, cpix[sl], torch.where(disc, 0.0, F))
        else:
            G = gmap / dom
            Gb = torch.where(disc, add(G[pix] * wt) / S, G[cpix[sl]])
            q = torch.where(disc[pp], (G[pix] - Gb[pp]) * wt, 0.0)
            # the unit tangent from the particle towards the pixel, in its (e_theta, e_phi), times alpha
            sa = torch.sin(al)
            f = torch.where(sa > 1e-300, al / sa, 1.0)
            et = torch.sin(thr[ro] - th[pp]) - 2 * torch.cos(th)[pp] * st[ro] * sdp * sdp
            ep = st[ro] * torch.sin(dp)
            vt, vp, T = add(q * f * et), add(q * f * ep), add(q * al * al)
            ct, s0, cp, sp = torch.cos(th), torch.sin(th), torch.cos(ph), torch.sin(ph)
            K = F / (0.333 * S * a * a)
            V = torch.stack([ct * cp * vt - sp * vp, ct * sp * vt + cp * vp, -s0 * vt], 1) * K[:, None]
            KT = torch.where(disc, K * T, 0.0)
            DV = torch.stack([-V[:, 0], -V[:, 1], V[:, 2]], 1) * disc[:, None]
            uh, dd = u[sl] / d[sl][:, None], d[sl]
            gp = -((2 * Gb * F + KT) / dd)[:, None] * uh + (DV @ rot.T) / dd[:, None]
            out[:3, sl] = gp.T
            out[3, sl] = Gb * F / parts["m"][sl].double()
            out[4, sl] = 0.0 if case["law"] == "decay" else Gb * F / parts["rho"][sl].double()
            out[5, sl] = KT / parts["h"][sl].double()
        i0 = i1
    return out / dom if gmap is None else out


def exact(case, seed):
    if _pixels(case) > 2.5e10:
        return None
    parts, m = _particles(case, seed)
    op = case["op"]
    par = _params(case, m)
    if op == "batch":
        return [_exact_view(case, _params(case, m, obs, ns), parts, ns) for obs, ns in _observers(case, seed)]
    if op == "adjoint":
        return {"grad": _exact_view(case, par, parts, case["nside"], _gmap(case, seed)), "observer": None}
    if op == "grad":
        g = _exact_view(case, par, parts, case["nside"], _gmap(case, seed))
        return {"map": _exact_view(case, par, parts, case["nside"]), "grads": list(g), "observer": None}
    return _exact_view(case, par, parts, case["nside"])
