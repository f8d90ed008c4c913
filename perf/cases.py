"""The work that users of conan_b200 have it do, as cases that can be timed.

A case is a dict of plain values; `kind` names the entry point:

  deposit   conan_deposit_static: CIC density of device displacements, for
            callers inside their own loop (latency counts)
  run       Gravity.run from a potential in host memory, then the state
            (the `run` tool up to a snapshot); FP32 states go on to a torch
            program on the GPU as float32 tensors, FP64 states stay doubles
  model     DiffPM forward: device white noise -> final density
  grad      DiffPM forward and backward through torch.autograd
  ensemble  Ensemble.run: boxes of mixed sizes in one graph launch, then
            every member's state as float32
  fof       FoF.run_device: friends-of-friends tags of device positions
  ic        generate_random_field and compute_potential on host arrays (the
            `ic` tool)
  cic       cic on host arrays (the `cic` tool)

`exact` is the same physics in 64-bit torch, written from the formulas.
"""
import ctypes as C
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import conan_b200 as cb
from conan_b200 import _lib
from conan_b200.autograd import DiffPM
from conan_b200.ensemble import Ensemble

DEV = "cuda"
H0, OMEGA_M, OMEGA_L = 68.5, 1.0, 0.0  # the solver's default cosmology


# ------------------------------------------------------------------ cases --

def listed():
    return [
        # the smallest call: a 64^3 density inside someone else's step
        dict(name="deposit_3d_64", kind="deposit", dim=3, mbits=6, f=1, rms=1.5),
        # the plain 2D method as the reference runs it: FP64, 100 steps
        dict(name="run_2d_256_fp64", kind="run", dim=2, mbits=8, f=1, L=50.0, ns=-1.0, precision="fp64",
             gradient="fd4", periodic=False, a0=0.02, da=0.0098, n=100),
        # an ordinary 3D run on the product path: 128^3, 50 steps
        dict(name="run_3d_128", kind="run", dim=3, mbits=7, f=1, L=100.0, ns=-2.0, precision="fp32",
             gradient="fd4", periodic=False, a0=0.02, da=0.0096, n=50),
        # a larger 3D run with its snapshot
        dict(name="run_3d_256", kind="run", dim=3, mbits=8, f=1, L=250.0, ns=-1.5, precision="fp32",
             gradient="fd4", periodic=False, a0=0.05, da=0.01125, n=40),
        # the throughput box, device to device: 512^3 particles and cells
        dict(name="model_3d_512", kind="model", dim=3, mbits=9, f=1, L=500.0, ns=-1.5, a0=0.05, da=0.03, n=6),
        # a force mesh finer than the particle lattice: 256^3 particles, 512^3 cells
        dict(name="model_3d_256_f2", kind="model", dim=3, mbits=8, f=2, L=250.0, ns=-1.5, a0=0.05, da=0.0475, n=6),
        # field-level inference: gradient of a density loss, 128^3
        dict(name="grad_3d_128", kind="grad", dim=3, mbits=7, f=1, L=100.0, ns=-2.0, a0=0.05, da=0.0296875, n=16,
             every=8),
        # the same on a larger box with fewer steps
        dict(name="grad_3d_256", kind="grad", dim=3, mbits=8, f=1, L=250.0, ns=-1.5, a0=0.05, da=0.0475, n=6, every=3),
        # an ensemble of mixed sizes, 40 steps, one graph launch
        dict(name="ensemble_6", kind="ensemble", n5=2, n6=2, n7=2, L=100.0, a0=0.05, a_end=0.525, n=40),
        # halo finding on a snapshot on the device; the count is no power of two
        dict(name="fof_3d_6m", kind="fof", dim=3, np=6000001, b=0.2, share=0.5),
        # initial conditions as the `ic` tool makes them: 128^3, FP64, seeded noise
        dict(name="ic_3d_128", kind="ic", dim=3, mbits=7, L=100.0, ns=-2.0, scale_free=True, smooth=True),
        # the `cic` tool on a snapshot: 128^3 particles, 256^3 mesh
        dict(name="cic_3d_128_f2", kind="cic", dim=3, mbits=7, f=2, sub=1, L=100.0),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["deposit", "run", "run", "model", "model", "grad", "grad", "ensemble", "fof", "fof", "ic", "cic"])
    ns = round(rng.uniform(-2.5, -1.0), 2)
    if kind == "deposit":
        dim = rng.choice([2, 3, 3])
        mbits = rng.randint(5, 9) if dim == 2 else rng.randint(4, 7)
        f = 1 if (mbits + 1) * dim > 21 else rng.choice([1, 1, 2])
        return dict(kind=kind, dim=dim, mbits=mbits, f=f, rms=round(_log(rng, 0.1, 4.0), 3))
    if kind == "run":
        dim = rng.choice([2, 3, 3, 3])
        mbits = rng.randint(6, 10) if dim == 2 else rng.randint(5, 8)
        precision = rng.choice(["fp32", "fp32", "fp64"])
        f = rng.choice([1, 1, 2]) if mbits * dim < 23 else 1
        n = rng.randint(4, 40 if mbits * dim < 23 else 20)
        a0 = round(rng.uniform(0.02, 0.06), 4)
        return dict(kind=kind, dim=dim, mbits=mbits, f=f, L=round(_log(rng, 40.0, 400.0), 2), ns=ns,
                    precision=precision, gradient=rng.choice(["fd4", "fd4", "fd4", "spectral"]),
                    periodic=rng.choice([False, True]), a0=a0, da=round((rng.uniform(0.2, 0.5) - a0) / n, 5), n=n)
    if kind in ("model", "grad"):
        mbits = rng.randint(6, 8) if kind == "model" else rng.randint(5, 8)
        f = rng.choice([1, 1, 2]) if mbits < 8 else 1
        n = rng.randint(3, 10) if kind == "model" else rng.randint(2, 8)
        a0 = round(rng.uniform(0.03, 0.06), 4)
        c = dict(kind=kind, dim=3, mbits=mbits, f=f, L=round(_log(rng, 60.0, 400.0), 2), ns=ns, a0=a0,
                 da=round(rng.uniform(0.01, 0.04), 5), n=n)
        if kind == "grad":
            c["every"] = rng.randint(1, 8)
        return c
    if kind == "ensemble":
        return dict(kind=kind, n5=rng.randint(1, 8), n6=rng.randint(0, 4), n7=rng.randint(0, 2),
                    L=round(_log(rng, 60.0, 200.0), 2), a0=0.05, a_end=round(rng.uniform(0.2, 0.5), 3),
                    n=rng.randint(5, 40))
    if kind == "fof":
        return dict(kind=kind, dim=rng.choice([2, 3, 3]), np=int(_log(rng, 2.0e4, 8.0e6)) | 1,
                    b=round(rng.uniform(0.1, 0.3), 3), share=round(rng.uniform(0.2, 0.6), 2))
    if kind == "ic":
        dim = rng.choice([2, 3, 3])
        return dict(kind=kind, dim=dim, mbits=rng.randint(6, 10) if dim == 2 else rng.randint(5, 7),
                    L=round(_log(rng, 40.0, 400.0), 2), ns=ns, scale_free=rng.choice([True, False]),
                    smooth=rng.choice([True, False]))
    return dict(kind=kind, dim=3, mbits=rng.randint(5, 7), f=rng.choice([1, 2]), sub=rng.choice([1, 1, 2]),
                L=round(_log(rng, 40.0, 400.0), 2))


# ------------------------------------------- the physics in 64-bit torch --

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _noise(case, seed, dtype=torch.float64):
    n = 1 << case["mbits"]
    return torch.randn(n ** case["dim"], generator=_gen(seed), device=DEV, dtype=dtype)


def _axes(n, dim, half=True):
    """Integer wave numbers per axis k (0 fastest), shaped to broadcast over a half spectrum."""
    out = []
    for k in range(dim):
        i = torch.arange(n // 2 + 1 if half and k == 0 else n, device=DEV, dtype=torch.float64)
        w = torch.where(i > n // 2, i - n, i)
        out.append(w.reshape([-1 if d == dim - 1 - k else 1 for d in range(dim)]))
    return out


def _filter(n, dim, L, ns, scale_free, with_s, scale):
    ks = _axes(n, dim)
    k2 = sum(k * k for k in ks)
    k2 = torch.where(k2 > 0, k2, torch.ones_like(k2))
    if not scale_free:  # CDM transfer function at physical k (Omega0 = 0.32, H0 = 69)
        k = k2.sqrt() * (2 * math.pi / L)
        q = k * (2.7255 / 2.7) ** 2 / (0.32 * 0.69)
        l0 = torch.log(2 * 2.718281828459045 + 1.8 * q)
        t0 = l0 / (l0 + (14.2 + 731.0 / (1 + 62.5 * q)) * q * q)
        f = torch.sqrt(1122670 * k ** ns * t0 * t0)
    else:
        f = torch.sqrt((k2.sqrt() * (2 * math.pi / n)) ** ns)
        if with_s:
            t = scale * n / L
            for k in ks:
                f = f * torch.exp(t * (torch.cos(k * (2 * math.pi / n)) - 1))
    f.view(-1)[0] = 0.0
    return f


def _grf(noise, dim, n, L, ns, scale_free=True, smooth=False, scale=8.0, sigma=0.83):
    shape = (n,) * dim
    W = torch.fft.rfftn(noise.reshape(shape))
    if not scale_free:
        return torch.fft.irfftn(W * _filter(n, dim, L, ns, False, False, scale), s=shape) / (L / n) ** (dim / 2)
    var = torch.fft.irfftn(W * _filter(n, dim, L, ns, True, True, scale), s=shape).square().mean()
    return torch.fft.irfftn(W * _filter(n, dim, L, ns, True, smooth, scale), s=shape) * (sigma / var.sqrt())


def _potential(dens, dim, n, L, amp=1.0):
    k2 = sum(k * k for k in _axes(n, dim))
    g = torch.where(k2 > 0, -amp * (L / (2 * math.pi)) ** 2 / torch.where(k2 > 0, k2, torch.ones_like(k2)),
                    torch.zeros_like(k2))
    return torch.fft.irfftn(torch.fft.rfftn(dens) * g, s=dens.shape)


def _fd4(f, k):
    ax = f.dim() - 1 - k
    return (torch.roll(f, 2, ax) - torch.roll(f, -2, ax)) / 12 + (torch.roll(f, -1, ax) - torch.roll(f, 1, ax)) * (2 / 3)


def _lattice(n, dim, f):
    i = torch.arange(n ** dim, device=DEV)
    return [((i // n ** k) % n) * f for k in range(dim)]


def _corners(org, nf, dim):
    for b in range(1 << dim):
        idx = 0
        for k in range(dim - 1, -1, -1):
            idx = idx * nf + (org[k] + ((b >> k) & 1)) % nf
        yield b, idx


def _weight(fr, b, dim):
    w = 1.0
    for k in range(dim):
        w = w * (fr[k] if (b >> k) & 1 else 1 - fr[k])
    return w


def _density(d, q, nf, dim, mass):
    """CIC density contrast of displacements d (force cells) from lattice points q."""
    org = [q[k] + torch.floor(d[k].detach()).long() for k in range(dim)]
    fr = [d[k] - torch.floor(d[k].detach()) for k in range(dim)]
    rho = torch.zeros(nf ** dim, device=DEV, dtype=torch.float64)
    for b, idx in _corners(org, nf, dim):
        rho = rho.index_add(0, idx, _weight(fr, b, dim))
    return rho * mass - 1


def _adot(a):
    return H0 * a * math.sqrt(OMEGA_L + OMEGA_M * a ** -3 + (1 - OMEGA_M - OMEGA_L) * a ** -2)


def _kick(d, p, q, n, f, dim, L, a, da, periodic, spectral):
    nf = n * f
    res = L / nf
    delta = _density(d, q, nf, dim, float(f) ** dim).reshape((nf,) * dim)
    phi = _potential(delta, dim, nf, L, 1.5 * OMEGA_M * H0 * H0 / a)
    if spectral:
        F = torch.fft.rfftn(phi)
        G = []
        for k, w in enumerate(_axes(nf, dim)):
            w = torch.where(w.abs() * 2 == nf, torch.zeros_like(w), w) * (2 * math.pi / nf)
            G.append(torch.fft.irfftn(F * w * 1j, s=phi.shape).reshape(-1))
    else:
        G = [_fd4(phi, k).reshape(-1) for k in range(dim)]
    org, fr = [], []
    for k in range(dim):
        fl = torch.floor(d[k].detach())
        o, r = q[k] + fl.long(), d[k] - fl
        if not periodic:  # the reference's gather truncates unwrapped coordinates toward zero
            up = (o < 0) & (r.detach() != 0)
            o, r = o + up.long(), r - up.double()
        org.append(o)
        fr.append(r)
    F = [0.0] * dim
    for b, idx in _corners(org, nf, dim):
        w = _weight(fr, b, dim)
        for k in range(dim):
            F[k] = F[k] + G[k].index_select(0, idx) * w
    ck = (da / _adot(a)) / (res * res)
    return [p[k] - F[k] * ck for k in range(dim)]


def _steps(phi, n, f, dim, L, a0, da, steps, periodic=False, spectral=False, save=False):
    """Zel'dovich start from the potential phi and `steps` leapfrog steps: d, p in force cells, q."""
    res_m, res_f = L / n, L / (n * f)
    q = _lattice(n, dim, f)
    u = [_fd4(phi, k).reshape(-1) for k in range(dim)]
    d = [x * (-a0 / (res_m * res_f)) for x in u]
    p = [x * (-(a0 + da / 2) / (res_m * res_f)) for x in u]

    def step(a, *dp):
        d, p = list(dp[:dim]), list(dp[dim:])
        cd = da / (a * a * _adot(a))
        d = [d[k] + p[k] * cd for k in range(dim)]
        p = _kick(d, p, q, n, f, dim, L, a + da / 2, da, periodic, spectral)
        return (*d, *p)

    a = a0
    for _ in range(steps):
        out = checkpoint(step, a, *d, *p, use_reentrant=False) if save else step(a, *d, *p)
        d, p = list(out[:dim]), list(out[dim:])
        a += da
    return d, p, q


def _state(d, p, q, res, dim):
    X = torch.stack([(q[k] + d[k]) * res for k in range(dim)], 1)
    return X, torch.stack([p[k] * res for k in range(dim)], 1)


def _zeldovich(case, seed, rms):
    """Displacements of a correlated field in lattice cells (rms per axis)."""
    n, dim = 1 << case["mbits"], case["dim"]
    phi = _potential(_grf(_noise(case, seed), dim, n, 100.0, -2.0), dim, n, 100.0)
    u = [_fd4(phi, k).reshape(-1) for k in range(dim)]
    s = rms / torch.stack([x.square().mean() for x in u]).mean().sqrt()
    return [x * s for x in u]


def _philox_normals(n, seed):
    """Unit normals of Philox4x32-10 (Salmon et al., SC'11) and Box-Muller, pairs (2j, 2j+1)."""
    j = np.arange(n // 2, dtype=np.uint64)
    m32 = np.uint64(0xFFFFFFFF)
    c = [j & m32, j >> np.uint64(32), np.full_like(j, 0x636F6E61), np.zeros_like(j)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = [((((c[i] << np.uint64(32)) | c[i + 1]) >> np.uint64(11)).astype(np.float64) + 0.5) * 2.0 ** -53 for i in (0, 2)]
    r, t = np.sqrt(-2.0 * np.log(u[0])), 2.0 * np.pi * u[1]
    return torch.from_numpy(np.stack([r * np.cos(t), r * np.sin(t)], 1).reshape(-1)).to(DEV)


# -------------------------------------------------------- inputs and runs --

def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _ic_header(case):
    return {"dim": case["dim"], "mbits": case["mbits"], "size": case["L"], "ns": case["ns"],
            "smooth": case["smooth"], "scale-free": case["scale_free"], "scale": 8.0, "sigma": 0.83,
            "Omega0": 0.32, "H0": 69.0}


def _members(case, seed):
    ns = [-2.5, -2.0, -1.5, -1.0]
    out = []
    for mbits, count in ((5, case["n5"]), (6, case["n6"]), (7, case["n7"])):
        for _ in range(count):
            i = len(out)
            out.append((mbits, case["L"], ns[(seed + 3 * i) % 4], 1000 + 64 * (seed % 1000003) + i))
    return out


def _diff(case):
    return DiffPM(dim=case["dim"], mbits=case["mbits"], L_box=case["L"], ns=case["ns"], a0=case["a0"], da=case["da"],
                  n=case["n"], checkpoint_every=case.get("every", 8), f=case["f"])


def _points(case, seed):
    """Clustered positions in a unit-density box: a share in cuspy halos of power-law masses, the rest uniform."""
    n, dim, g = case["np"], case["dim"], _gen(seed)
    L = n ** (1.0 / dim)
    nh = max(4, n // 300)
    mass = (1 - torch.rand(nh, generator=g, device=DEV, dtype=torch.float64)).pow(-0.9).clamp(max=1.0e3)
    cum = torch.cumsum(mass, 0)
    ncl = int(case["share"] * n)
    h = torch.searchsorted(cum, torch.rand(ncl, generator=g, device=DEV, dtype=torch.float64) * cum[-1]).clamp(max=nh - 1)
    ball = 4 * math.pi / 3 if dim == 3 else math.pi
    R = (mass * (ncl / cum[-1]) / (200 * ball)).pow(1.0 / dim)
    centre = torch.rand(nh, dim, generator=g, device=DEV, dtype=torch.float64) * L
    v = torch.randn(ncl, dim, generator=g, device=DEV, dtype=torch.float64)
    r = torch.rand(ncl, 1, generator=g, device=DEV, dtype=torch.float64).pow(0.6)
    X = torch.rand(n, dim, generator=g, device=DEV, dtype=torch.float64) * L
    X[:ncl] = centre[h] + v / v.norm(dim=1, keepdim=True) * r * R[h].unsqueeze(1)
    return X[torch.randperm(n, generator=g, device=DEV)].contiguous(), L


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    n = 1 << case["mbits"] if "mbits" in case else 0
    if kind == "deposit":
        d = [(x * case["f"]).float() for x in _zeldovich(case, seed, case["rms"])]
        s.update(d=d, out=torch.empty((n * case["f"]) ** case["dim"], device=DEV))
    elif kind == "run":
        dim = case["dim"]
        dens = _grf(_noise(case, seed), dim, n, case["L"], case["ns"])
        s["phi"] = _pinned(_potential(dens, dim, n, case["L"]).reshape(-1)).numpy()
        s["G"] = cb.Gravity(dim, n, case["f"], case["L"], precision=case["precision"], gradient=case["gradient"],
                            periodic_gather=case["periodic"])
        s["X"], s["P"] = (torch.empty(n ** dim, dim, dtype=torch.float64, pin_memory=True) for _ in range(2))
    elif kind in ("model", "grad"):
        s["model"] = _diff(case)
        s["noise"] = _noise(case, seed, torch.float32)
        if kind == "grad":
            # a target of the same kind of field, on the force mesh
            t = _noise({"mbits": case["mbits"], "dim": 3}, seed + 500009, torch.float32).reshape(n, n, n)
            for ax in range(3):
                t = t.repeat_interleave(case["f"], dim=ax)
            s["target"] = t.reshape(-1).contiguous()
        else:
            s["out"] = torch.empty((n * case["f"]) ** 3, device=DEV)
    elif kind == "ensemble":
        s["ens"] = Ensemble(_members(case, seed), a0=case["a0"], a_end=case["a_end"], steps=case["n"], autotune=False)
        s["ens"].init()
    elif kind == "fof":
        s["X"], L = _points(case, seed)
        s["tags"] = torch.empty(case["np"], dtype=torch.int64, device=DEV)
        s["fof"] = cb.FoF(case["dim"], case["np"], L, case["b"])
    elif kind == "ic":
        s["H"] = _ic_header(case)
        s["noise"] = _noise(case, seed).cpu().numpy()
    else:
        q = _lattice(n, 3, 1)
        d = _zeldovich(case, seed, 1.5)
        s["X"] = (torch.stack([q[k] + d[k] for k in range(3)], 1) * (case["L"] / n)).cpu().numpy()
    return s


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "deposit":
        d = [C.c_void_p(x.data_ptr()) for x in s["d"]] + [None]
        _lib.check(_lib.lib().conan_deposit_static(case["dim"], 1 << case["mbits"], case["f"], d[0], d[1], d[2],
                                                   C.c_void_p(s["out"].data_ptr()),
                                                   C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return s["out"]
    if kind == "run":
        s["G"].run(s["phi"], case["a0"], case["da"], case["n"], every=case["n"])
        s["G"].state_into(s["X"].numpy(), s["P"].numpy())
        if case["precision"] == "fp64":
            return [s["X"], s["P"]]
        return [x.to(DEV, non_blocking=True).float() for x in (s["X"], s["P"])]
    if kind == "model":
        s["model"].forward_raw(s["noise"], s["out"])
        return s["out"]
    if kind == "grad":
        noise = s["noise"].requires_grad_(True)
        delta = s["model"](noise)
        loss = (delta - s["target"]).square().mean()
        return [delta.detach(), torch.autograd.grad(loss, noise)[0]]
    if kind == "ensemble":
        s["ens"].run()
        return [torch.from_numpy(x).float() for i in range(len(s["ens"].members)) for x in s["ens"].state(i)]
    if kind == "fof":
        groups = s["fof"].run_device(s["X"].data_ptr(), s["tags"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return [s["tags"], groups]
    if kind == "ic":
        dens = cb.generate_random_field(s["H"], noise=s["noise"])
        return [dens, cb.compute_potential(s["H"], dens)]
    n = 1 << case["mbits"]
    return cb.cic(s["X"], case["dim"], n, case["L"], f=case["f"], sub_sample=case["sub"])


def exact(case, seed):
    kind = case["kind"]
    n = 1 << case["mbits"] if "mbits" in case else 0
    if kind == "fof":
        return None  # whole numbers
    if kind == "deposit":
        d = [(x * case["f"]).float().double() for x in _zeldovich(case, seed, case["rms"])]
        q = _lattice(n, case["dim"], case["f"])
        return _density(d, q, n * case["f"], case["dim"], float(case["f"]) ** case["dim"])
    if kind == "run":
        dim = case["dim"]
        phi = _potential(_grf(_noise(case, seed), dim, n, case["L"], case["ns"]), dim, n, case["L"])
        with torch.no_grad():
            d, p, q = _steps(phi, n, case["f"], dim, case["L"], case["a0"], case["da"], case["n"], case["periodic"],
                             case["gradient"] == "spectral")
        return list(_state(d, p, q, case["L"] / (n * case["f"]), dim))
    if kind in ("model", "grad"):
        noise = _noise(case, seed, torch.float32).double()
        if kind == "grad":
            noise.requires_grad_(True)
        with torch.set_grad_enabled(kind == "grad"):
            phi = _potential(_grf(noise, 3, n, case["L"], case["ns"]), 3, n, case["L"])
            d, _, q = _steps(phi, n, case["f"], 3, case["L"], case["a0"], case["da"], case["n"], save=kind == "grad")
            delta = _density(d, q, n * case["f"], 3, float(case["f"]) ** 3)
        if kind == "model":
            return delta
        t = _noise({"mbits": case["mbits"], "dim": 3}, seed + 500009, torch.float32).reshape(n, n, n)
        for ax in range(3):
            t = t.repeat_interleave(case["f"], dim=ax)
        loss = (delta - t.reshape(-1).double()).square().mean()
        return [delta.detach(), torch.autograd.grad(loss, noise)[0]]
    if kind == "ensemble":
        out = []
        with torch.no_grad():
            for mbits, L, ns, sd in _members(case, seed):
                m = 1 << mbits
                phi = _potential(_grf(_philox_normals(m ** 3, sd), 3, m, L, ns), 3, m, L)
                da = (case["a_end"] - case["a0"]) / case["n"]
                out += _state(*_steps(phi, m, 1, 3, L, case["a0"], da, case["n"]), L / m, 3)
        return out
    if kind == "ic":
        dim = case["dim"]
        dens = _grf(_noise(case, seed), dim, n, case["L"], case["ns"], case["scale_free"], case["smooth"])
        return [dens.reshape(-1), _potential(dens, dim, n, case["L"]).reshape(-1)]
    q, d = _lattice(n, 3, 1), _zeldovich(case, seed, 1.5)
    sub, nf, L = case["sub"], n * case["f"], case["L"]
    if sub == 1:
        x = [(q[k] + d[k]) * case["f"] for k in range(3)]
        mass = 1.0
    else:  # linear interpolation of the displacement on a finer grid
        ns = n * sub
        j = _lattice(ns, 3, 1)
        org, fr = [i // sub for i in j], [(i % sub).double() / sub for i in j]
        v = [0.0] * 3
        for b, idx in _corners(org, n, 3):
            w = _weight(fr, b, 3)
            v = [v[k] + d[k][idx] * w for k in range(3)]
        x = [(j[k].double() / sub + v[k]) * case["f"] for k in range(3)]
        mass = (ns / nf) ** -3.0
    zero = [torch.zeros_like(x[0], dtype=torch.int64)] * 3
    return (_density(x, zero, nf, 3, 1.0) + 1) * mass


def work(case):
    """Bytes and operations of one pass: per leapfrog step, positions, momenta and the mesh once per phase that
    needs all of them before the next can start; host data once."""
    kind = case["kind"]
    n = 1 << case["mbits"] if "mbits" in case else 0
    dim = case.get("dim", 3)
    npart, ncell = n ** dim, (n * case.get("f", 1)) ** dim

    def step(npart, ncell, w, dim):  # state in and out, positions again for the deposit, mesh in and out of each transform
        return npart * w * dim * 5 + ncell * w * 6, npart * (1 << dim) * 6 * dim + ncell * (5 * math.log2(ncell) + 6 * dim)

    if kind == "deposit":
        return {"bytes": 4 * (dim * npart + ncell), "flops": npart * (1 << dim) * 4}
    if kind == "run":
        w = 8 if case["precision"] == "fp64" else 4
        b, fl = step(npart, ncell, w, dim)
        return {"bytes": case["n"] * b + 8 * npart * (1 + 2 * dim), "flops": case["n"] * fl}
    if kind in ("model", "grad"):
        b, fl = step(npart, ncell, 4, dim)
        k = case["n"] * (1 if kind == "model" else 1 + 2)  # backward: the state again and its adjoint
        return {"bytes": k * b + 4 * (2 * npart + ncell), "flops": k * fl}
    if kind == "ensemble":
        b = fl = 0
        for mbits, count in ((5, case["n5"]), (6, case["n6"]), (7, case["n7"])):
            m = 1 << (3 * mbits)
            x, y = step(m, m, 4, 3)
            b, fl = b + count * (case["n"] * x + 48 * m), fl + count * case["n"] * y
        return {"bytes": b, "flops": fl}
    if kind == "fof":
        return {"bytes": case["np"] * 8 * (dim + 1), "flops": case["np"] * 60}
    if kind == "ic":
        return {"bytes": npart * 8 * 4, "flops": npart * (10 * math.log2(npart) + 20)}
    return {"bytes": 8 * (3 * npart + ncell), "flops": 24 * (n * case["sub"]) ** 3}
