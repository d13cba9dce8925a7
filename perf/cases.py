"""Work that users of the library have it do, as cases to time and to compare.

A case is a dict of plain values.  Its "kind" names what one pass calls:

  cycle     gev_step (or gev_step_lightcone): one cycle of the main loop of a
            run whose state stays on the device
  stages    the same cycle through the separate entry points, in the order of a
            host code that keeps the reference's unfused calls
  spectrum  gev_power_spectrum: the P(k) written at the output times of a run
  grad      the differentiable run and its gradient (forward and backward
            through the autograd function)
  pm        the differentiable run, forward only
  poisson   gev_poisson_noalloc: a host code's own potential solve on its own
            device arrays

Grids are the ones the library accepts, up to the 512^3 box of the main
configuration; cells are 5 Mpc/h wide, as in all of the repository's
configurations.  Particle counts need not be N^3.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gevolution-2.0_b200", "python"))

import gevb200 as gev  # noqa: E402
from gevb200 import pm as gevpm  # noqa: E402
from gevb200.ics import C_LIGHT, hconf, linear_pk  # noqa: E402

OM, OL, CELL = 0.32, 0.68, 5.0
F64 = torch.float64
TAU0 = 1.0                     # conformal time of a run's first cycle (only differences to it matter)


def listed():
    return [
        # the smallest call: a host code's Poisson solve at a coarse grid, bound by launches
        {"name": "poisson 32 mixed", "kind": "poisson", "N": 32, "fp64": False},
        # the coarse validation box, FP64, at its start
        {"name": "cycle 64 fp64", "kind": "cycle", "N": 64, "np": 64 ** 3, "fp64": True, "z": 100.0,
         "parabolic": False, "tensor": False, "lightcone": False},
        # a development box late in its run: clustered particles, dense tiles
        {"name": "cycle 128 mixed late", "kind": "cycle", "N": 128, "np": 128 ** 3, "fp64": False, "z": 0.2,
         "parabolic": False, "tensor": False, "lightcone": False},
        # the FP64 drop-in configuration
        {"name": "cycle 256 fp64", "kind": "cycle", "N": 256, "np": 256 ** 3, "fp64": True, "z": 30.0,
         "parabolic": False, "tensor": False, "lightcone": False},
        # every optional field of the metric: parabolic B_i and evolved h_ij
        {"name": "cycle 256 mixed tensor", "kind": "cycle", "N": 256, "np": 256 ** 3, "fp64": False, "z": 10.0,
         "parabolic": True, "tensor": True, "lightcone": False},
        # a grid of 3 x 128, an odd number of particles, late: two multi-box pencils, ragged buckets
        {"name": "cycle 384 mixed late", "kind": "cycle", "N": 384, "np": 43046721, "fp64": False, "z": 0.5,
         "parabolic": False, "tensor": False, "lightcone": False},
        # the headline run: 512^3 with one lightcone shell per cycle
        {"name": "cycle 512 mixed lightcone", "kind": "cycle", "N": 512, "np": 512 ** 3, "fp64": False, "z": 100.0,
         "parabolic": False, "tensor": False, "lightcone": True},
        # the unfused call sequence, tracers fewer than cells
        {"name": "stages 128 mixed", "kind": "stages", "N": 128, "np": 1771561, "fp64": False, "z": 2.0},
        # the spectrum of a mixed-precision run
        {"name": "spectrum 256 mixed", "kind": "spectrum", "N": 256, "np": 256 ** 3, "fp64": False, "z": 1.0,
         "bins": 256},
        # the differentiable configuration: 128^3, 32 steps from z = 50 to 0, checkpoints every 8
        {"name": "grad 128 mixed", "kind": "grad", "N": 128, "np": 128 ** 3, "fp64": False, "steps": 32, "every": 8},
        # a small FP64 gradient, as gradient checks and fits use it
        {"name": "grad 32 fp64", "kind": "grad", "N": 32, "np": 32 ** 3, "fp64": True, "steps": 10, "every": 4},
        # a forward-only run of the differentiable path
        {"name": "pm 64 fp64", "kind": "pm", "N": 64, "np": 64 ** 3, "fp64": True, "steps": 16, "every": 16},
    ]


def _count(rng, N, most):
    """A particle count between N^3 / 3 and most N^3, hardly ever round."""
    return max(1, int(N ** 3 * math.exp(rng.uniform(math.log(1 / 3), math.log(most)))) | 1)


def draw(rng):
    kind = rng.choice(["cycle"] * 5 + ["stages", "spectrum", "grad", "pm", "poisson"])
    z = round(math.exp(rng.uniform(0.0, math.log(101.0))) - 1.0, 3)
    fp64 = rng.random() < 0.4
    if kind == "poisson":
        return {"kind": kind, "N": rng.choice([16, 32, 64, 128]), "fp64": fp64}
    if kind in ("grad", "pm"):
        N = rng.choice([16, 32, 64, 128])
        steps = rng.randint(1, 32)
        return {"kind": kind, "N": N, "np": _count(rng, N, 1.0), "fp64": fp64, "steps": steps,
                "every": rng.randint(1, steps)}
    if kind in ("spectrum", "stages"):
        N = rng.choice([16, 32, 64, 128, 256])
        c = {"kind": kind, "N": N, "np": _count(rng, N, 2.0 if N < 256 else 1.0), "fp64": fp64, "z": z}
        if kind == "spectrum":
            c["bins"] = rng.randint(16, 1024)
        return c
    N = rng.choice([16, 32, 64, 128, 256] + ([] if fp64 else [384]))
    return {"kind": kind, "N": N, "np": _count(rng, N, 2.0 if N < 256 else 1.0), "fp64": fp64, "z": z,
            "parabolic": rng.random() < 0.3, "tensor": rng.random() < 0.3,
            "lightcone": N >= 256 and z > 30.0 and rng.random() < 0.5}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def growth(a):
    """Linear growth D(a), normalised to a at early times (Carroll, Press & Turner 1992)."""
    om = OM / (OM + OL * a ** 3)
    ol = 1.0 - om
    return a * 2.5 * om / (om ** (4.0 / 7.0) - ol + (1.0 + 0.5 * om) * (1.0 + ol / 70.0))


def wavenumbers(N):
    kf = torch.fft.fftfreq(N, d=1.0 / N, device="cuda", dtype=F64)
    kh = torch.fft.rfftfreq(N, d=1.0 / N, device="cuda", dtype=F64)
    return kf[:, None, None], kf[None, :, None], kh[None, None, :]


def fourpig(N):
    return 1.5 * (CELL * N) ** 2 / C_LIGHT ** 2


def box(N, count, a, seed, clumps):
    """Particles and potential of a box at scale factor a on the GPU: Zel'dovich
    displacements of `count` particles spread evenly over the cell centres.
    With clumps, particles within a few cells of random centres (one per 8^3
    cells) have collapsed towards them, as they have late in a run.  Returns
    unwrapped positions [count, 3] and momenta in box units and the potential
    [N, N, N] (z, y, x), as FP64 values that single precision represents for
    all but the positions, and the undisplaced sites."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    kz, ky, kx = wavenumbers(N)
    W = torch.fft.rfftn(torch.randn((N, N, N), generator=g, device="cuda", dtype=torch.float32).to(F64))
    n2 = kx * kx + ky * ky + kz * kz
    n2[0, 0, 0] = 1.0
    # sqrt(P(k)) from a table over ln |n|
    t = np.linspace(0.0, math.log(N), 2048)
    amp = torch.from_numpy(np.sqrt(linear_pk(np.exp(t) * 2 * math.pi / (CELL * N), 1.0) / CELL ** 3)).cuda()
    at = 0.5 * torch.log(n2) / (t[1] - t[0])
    lo = at.floor().clamp_(0, 2046)
    at -= lo
    lo = lo.long()
    W *= torch.lerp(amp[lo], amp[lo + 1], at) * growth(a)
    del at, lo
    W[0, 0, 0] = 0.0
    sites = (torch.arange(count, device="cuda") * N ** 3) // count
    cells = torch.stack([sites % N, (sites // N) % N, sites // (N * N)], dim=1).to(F64) + 0.5
    if count != N ** 3:
        cells += torch.rand((count, 3), generator=g, device="cuda", dtype=F64) - 0.5
    pos = torch.empty((count, 3), device="cuda", dtype=F64)
    q = torch.empty((count, 3), device="cuda", dtype=F64)
    om_a = OM / (OM + OL * a ** 3)
    vel = a * om_a ** 0.55 * hconf(a, fourpig(N), OM, OL)
    for c, k in enumerate((kx, ky, kz)):
        psi = torch.fft.irfftn(W * (1j / (2 * math.pi)) * (k / n2), s=(N, N, N)).reshape(-1)[sites]
        q[:, c] = vel * psi
        pos[:, c] = cells[:, c] / N + psi
        del psi
    lap = sum((2.0 * N * torch.sin(math.pi * k / N)) ** 2 for k in (kx, ky, kz))
    H = hconf(a, fourpig(N), OM, OL)
    W *= -(fourpig(N) / a) * OM / (lap + 3.0 * (H * H + fourpig(N) * OM / a))
    phi = torch.fft.irfftn(W, s=(N, N, N)).float().to(F64)
    del W, lap, n2
    if clumps:
        nb = N // 8
        centre = torch.rand((nb ** 3, 3), generator=g, device="cuda", dtype=F64) * 8.0
        radius = 4.0 * a * torch.rand(nb ** 3, generator=g, device="cuda", dtype=F64).sqrt() + 1e-3
        p = pos * N
        b = torch.floor(p / 8.0)
        bi = b.long() % nb
        bi = bi[:, 0] + nb * (bi[:, 1] + nb * bi[:, 2])
        r = p - 8.0 * b - centre[bi]
        f = (r.norm(dim=1) / radius[bi]).clamp_(max=1.0)
        pos += r * (f * f - 1.0)[:, None] / N
        q += (1e-3 * a) * (1.0 - f)[:, None] * torch.randn((count, 3), generator=g, device="cuda", dtype=F64)
        del p, b, bi, r, f
    return pos, q.float().to(F64), phi, cells / N


def cycle_start(case):
    """Scale factor, time step and cosmology of a cycle case.  The step limit
    shrinks with the grid so that a state stays close to its epoch however many
    cycles of a small box are run."""
    N, a = case["N"], 1.0 / (1.0 + case["z"])
    cosmo = gev.Cosmo(OM, OL, 0.0, fourpig(N), 48.0, 0.04 * (N / 512.0) ** 2, 200.0, CELL * N)
    dtau = min(48.0 / N, cosmo.steplimit / hconf(a, fourpig(N), OM, OL))
    return a, dtau, cosmo


class Held(dict):
    """The outputs that a library context holds in device memory, each read
    through the library's getters when it is looked up (a program leaves them
    on the device from cycle to cycle)."""

    def __init__(self, readers, **values):
        super().__init__({**dict.fromkeys(readers), **values})
        self.readers = readers

    def __getitem__(self, key):
        return self.readers[key]() if key in self.readers else super().__getitem__(key)


def held_particles(s):
    """Displacements from the sites and momenta, in ID order."""
    pos, q, ids = (torch.from_numpy(x).cuda() for x in s["ctx"].get_particles())
    d = torch.empty_like(pos)
    d[ids] = pos - s["sites"][ids]
    out = torch.empty_like(q)
    out[ids] = q
    return {"displacement": d - torch.round(d), "momentum": out}


def held_lightcone(s):
    """The shell's particles in ID order: whether each crossed, and where and how fast."""
    pos, vel, ids = (torch.from_numpy(x).cuda() for x in s["ctx"].lightcone_fetch(s["crossed"]))
    n = s["case"]["np"]
    out = {"crossed": torch.zeros(n, dtype=torch.uint8, device="cuda"),
           "pos": torch.zeros((n, 3), device="cuda"), "vel": torch.zeros((n, 3), device="cuda")}
    out["crossed"][ids] = 1
    out["pos"][ids] = pos
    out["vel"][ids] = vel
    return out


def device_field(s, field):
    return torch.from_numpy(s["ctx"].get_field(field)).cuda()


def prepare(case, seed):
    N, kind = case["N"], case["kind"]
    prec = gev.FP64 if case["fp64"] else gev.MIXED
    real = F64 if case["fp64"] else torch.float32
    if kind == "poisson":
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        src = torch.randn((N, N, N), generator=g, device="cuda", dtype=torch.float32).to(real)
        return {"case": case, "src": src, "phi": torch.empty_like(src), "prec": prec}
    if kind in ("grad", "pm"):
        a0 = 1.0 / 51.0
        x0, q0, _, _ = box(N, case["np"], a0, seed, False)
        coef, _ = gevpm.schedule(N, fourpig(N), OM, OL, a0, 1.0, case["steps"])
        s = {"case": case, "x0": x0, "q0": q0, "coef": coef,
             "pm": gevpm.PM(N, case["np"], OM / case["np"], prec, checkpoint_every=case["every"])}
        if kind == "grad":
            s["run"] = gevpm.run_function()
            g = torch.Generator(device="cuda")
            g.manual_seed(int(seed) + 1)
            s["target"] = torch.randn(N ** 3, generator=g, device="cuda", dtype=torch.float32).to(F64)
            x0.requires_grad_(True)
            q0.requires_grad_(True)
        else:
            s["delta"] = torch.empty(N ** 3, dtype=F64, device="cuda")
            s["x"], s["q"] = torch.empty_like(x0), torch.empty_like(q0)
        return s
    a, dtau, cosmo = cycle_start({**case, "z": case["z"]})
    pos, q, phi, sites = box(N, case["np"], a, seed, case["z"] < 3.0)
    pos = torch.remainder(pos, 1.0)
    host = (pos.cpu().numpy(), q.cpu().numpy(), np.arange(case["np"], dtype=np.int64))
    phi = phi.cpu().numpy().ravel()
    del pos, q
    if case["np"] > 10 ** 8:
        torch.cuda.empty_cache()      # the context allocates outside torch's pool
    ctx = gev.Context(N, precision=prec, capacity=case["np"], boxsize=CELL * N,
                      vector_method=gev.VECTOR_PARABOLIC if case.get("parabolic") else gev.VECTOR_ELLIPTIC,
                      tensor=case.get("tensor", False))
    ctx.set_particles(*host, OM / case["np"])
    ctx.set_field(gev.FIELD_PHI, phi)
    s = {"case": case, "ctx": ctx, "sites": sites, "cosmo": cosmo,
         "state": gev.State(a, TAU0, dtau, dtau, 1, 0.0, 0.0, 0.0)}
    if case.get("lightcone"):
        # a full-sky shell around the box corner whose surface starts 0.98 box lengths out
        s["lc"] = gev.LightconeArgs((0.0, 0.0, 0.0), (1.0 / math.sqrt(3.0),) * 3, -1.0, (1.0, 0.3), TAU0 + 0.98, 1, 0)
        s["lc_cap"] = case["np"] // 5
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["case"]["kind"]
    if kind == "poisson":
        N = s["case"]["N"]
        rc = gev.poisson_noalloc(N, s["prec"], s["src"].data_ptr(), s["phi"].data_ptr(), float(N), 1.0,
                                 torch.cuda.current_stream().cuda_stream)
        assert rc == gev.GEV_OK
        return s["phi"]
    if kind == "grad":
        s["x0"].grad = s["q0"].grad = None
        delta = s["run"].apply(s["x0"], s["q0"], s["pm"], s["coef"])
        ((delta - s["target"]) ** 2).sum().backward()
        return {"delta": delta.detach(), "gx": s["x0"].grad, "gq": s["q0"].grad}
    if kind == "pm":
        s["pm"].forward(s["coef"], s["x0"], s["q0"], s["delta"], s["x"], s["q"])
        return {"delta": s["delta"], "x": s["x"], "q": s["q"]}
    ctx = s["ctx"]
    if kind == "spectrum":
        kb, pw, ks, ps, oc = ctx.power_spectrum(s["case"]["bins"])
        # the scatters are roots of differences that cancel in bins of one |k|: as second moments they are well defined
        return Held({"density": lambda: device_field(s, gev.FIELD_SOURCE)}, k=kb, power=pw, krms=np.hypot(kb, ks),
                    prms=np.hypot(pw, ps), count=oc)
    if kind == "stages":
        return run_stages(s)
    st = s["state"]
    readers = {"phi": lambda: device_field(s, gev.FIELD_PHI), "chi": lambda: device_field(s, gev.FIELD_CHI),
               "B": lambda: device_field(s, gev.FIELD_BI), "particles": lambda: held_particles(s)}
    if s["case"]["tensor"]:
        readers["hij"] = lambda: device_field(s, gev.FIELD_HIJ_FT)
    if s["case"]["lightcone"]:
        s["crossed"] = ctx.step_lightcone(s["cosmo"], st, s["lc"], s["lc_cap"])
        readers["lightcone"] = lambda: held_lightcone(s)
    else:
        ctx.step(s["cosmo"], st)
    return Held(readers, scalars=np.array([st.a, st.dtau, st.T00hom, st.phi_hom, st.maxvel]))


def run_stages(s):
    """The cycle as a host code with the reference's call sequence makes it
    (main.cu:608-1283): one call per projection, solve, kick and drift."""
    ctx, st, N = s["ctx"], s["state"], s["case"]["N"]
    fpg, dx, a = s["cosmo"].fourpiG, 1.0 / N, s["state"].a
    H = hconf(a, fpg, OM, OL)
    ctx.project(gev.PROJ_T00 | gev.PROJ_TIJ, a, 1.0, True)
    t00 = ctx.prepare_T00(OM, 3.0 * H * dx * dx / st.dtau_old, fpg * dx * dx / a, 3.0 * H * H * dx * dx)
    _, hom = ctx.solve_phi(False, 0.0, 0.0, 0.0, 0.0, 1.0 / (dx * dx), 3.0 * H / st.dtau_old)
    ctx.solve_chi(2.0 * fpg * dx * dx / a)
    ctx.project(gev.PROJ_T0I, 1.0, 1.0, True)
    ctx.solve_B(fpg * dx * dx, 0.0)
    v = ctx.kick(0.5 * (st.dtau + st.dtau_old), a, a * a * N, 3)
    a = gev.rungekutta4bg(a, fpg, s["cosmo"], 0.5 * st.dtau)
    ctx.drift(st.dtau, a, a * a * N, 3)
    st.a = gev.rungekutta4bg(a, fpg, s["cosmo"], 0.5 * st.dtau)
    st.tau += st.dtau
    return Held({"phi": lambda: device_field(s, gev.FIELD_PHI), "chi": lambda: device_field(s, gev.FIELD_CHI),
                 "B": lambda: device_field(s, gev.FIELD_BI), "particles": lambda: held_particles(s)},
                scalars=np.array([st.a, st.dtau, t00 * dx ** 3, hom, v / math.sqrt(v * v + 1.0)]))


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how exact it is
# ---------------------------------------------------------------------------
def work(case):
    N, kind = case["N"], case["kind"]
    n3, R = N ** 3, 8 if case["fp64"] else 4
    fft = 2.5 * n3 * math.log2(n3)
    if kind == "poisson":
        return {"bytes": 2 * n3 * R, "flops": 2 * fft + 6 * n3}
    n = case["np"]
    if kind in ("grad", "pm"):
        # positions and momenta in and out of every step; the gradient runs the steps
        # once more from the checkpoints and once backwards
        step = {"bytes": 96 * n, "flops": 2 * fft + 250 * n}
        runs = 3 if kind == "grad" else 1
        return {"bytes": runs * case["steps"] * step["bytes"] + runs * 8 * n3, "flops": runs * case["steps"] * step["flops"]}
    if kind == "spectrum":
        return {"bytes": 28 * n + 8 * n3, "flops": fft + 30 * n + 60 * n3}
    # the particle state in and out, phi and chi in, phi, chi and B_i out
    transforms = 12 if case.get("parabolic") else 15
    w = {"bytes": 2 * n * (12 + 24 + 3 * R) + 7 * n3 * R, "flops": transforms * fft + 600 * n + 300 * n3}
    if case.get("tensor"):
        w["bytes"] += 24 * n3 * R     # h_ij and h_ij' in and out
        w["flops"] += 400 * n3
    if case.get("parabolic"):
        w["bytes"] += 6 * n3 * R      # the B_i spectrum in and out
    return w


def tolerance(case):
    """About four times (FP32) the error of the outputs against exact(); "max" where
    single values can be further off: a particle at a cell face or at the edge
    of the shell falls on either side of it."""
    kind, fp64 = case["kind"], case["fp64"]
    if kind == "poisson":
        return {"rel": 1e-14 if fp64 else 1e-6}
    if kind == "spectrum":
        return {"rel": 1e-11 if fp64 else 1e-7}
    if kind == "grad":
        return {"rel": 1e-10, "max": 1e-6} if fp64 else {"rel": 1e-3, "max": 0.5}
    if kind == "pm":
        return {"rel": 1e-11, "max": 1e-8} if fp64 else {"rel": 2e-5, "max": 1e-2}
    if fp64:
        return {"rel": 1e-11, "max": 1e-7}
    # early boxes are nearly uniform: B_i is what remains of sources that cancel (1.7e-4 at 512^3, z = 100)
    return {"rel": 1e-4 if case["z"] < 10.0 else 7e-4, "max": 0.9 if case.get("lightcone") else 3e-2, "differ": 1e-6}


# ---------------------------------------------------------------------------
# the same results in 64 bits from torch alone
# ---------------------------------------------------------------------------
CHUNK = 1 << 23


def rfft3(f):
    return torch.fft.rfftn(f)


def irfft3(F, N):
    """Unnormalised inverse; the imaginary parts of kx = 0 and N/2 do not count."""
    F = torch.fft.ifft(torch.fft.ifft(F, dim=0, norm="forward"), dim=1, norm="forward")
    return torch.fft.irfft(F, n=N, dim=2, norm="forward")


def k_tables(N):
    i = torch.arange(N, device="cuda", dtype=F64)
    gk = 2.0 * N * torch.sin(math.pi * i / N)
    ks = gk * torch.exp(-1j * math.pi * i / N)
    h = N // 2 + 1
    g = (gk ** 2)[:h][None, None, :], (gk ** 2)[None, :, None], (gk ** 2)[:, None, None]
    k = ks[:h][None, None, :], ks[None, :, None], ks[:, None, None]
    return g, k, g[0] + g[1] + g[2]


def poisson(src, N, coeff, modif):
    g, _, k2 = k_tables(N)
    F = rfft3(src) * (coeff / -float(N) ** 3)
    den = k2 + modif
    F = torch.where(den != 0.0, F / torch.where(den != 0.0, den, 1.0), 0.0)
    return irfft3(F, N), F[0, 0, 0].real


class Stencil:
    """Cells and in-cell offsets of some particles, and field values around them."""

    def __init__(self, x, N):
        p = x * N
        c = torch.floor(p)
        self.N, self.d, self.c = N, p - c, c.long() % N

    def site(self, dx, dy, dz):
        N, c = self.N, self.c
        return (c[:, 0] + dx) % N + N * ((c[:, 1] + dy) % N + N * ((c[:, 2] + dz) % N))

    def w(self, axis, b):
        return self.d[:, axis] if b else 1.0 - self.d[:, axis]

    def corners(self):
        for k in range(8):
            b = (k >> 2) & 1, (k >> 1) & 1, k & 1
            yield b, self.w(0, b[0]) * self.w(1, b[1]) * self.w(2, b[2])

    def face(self, f, i, shift=0, order=(0, 0, 0)):
        """f interpolated over the two axes other than i, at cell + shift along i (and + order)."""
        u, v = [k for k in range(3) if k != i]
        out = 0.0
        for bu in (0, 1):
            for bv in (0, 1):
                o = list(order)
                o[i] += shift
                o[u] += bu
                o[v] += bv
                out = out + self.w(u, bu) * self.w(v, bv) * f[self.site(*o)]
        return out

    def line(self, f, axis, shift=(0, 0, 0)):
        """f interpolated along one axis at cell + shift."""
        out = 0.0
        for b in (0, 1):
            o = list(shift)
            o[axis] += b
            out = out + self.w(axis, b) * f[self.site(*o)]
        return out


def unit(i):
    return tuple(int(k == i) for k in range(3))


def deposit(x, q, m, phi, a, N):
    """T00, Tij (00,01,02,11,12,22) and the T0i sums without their potential factor."""
    T = torch.zeros((10, N ** 3), device="cuda", dtype=F64)
    for o in range(0, len(x), CHUNK):
        s, v = Stencil(x[o:o + CHUNK], N), q[o:o + CHUNK]
        f2 = (v * v).sum(dim=1)
        e = torch.sqrt(f2 + a * a)
        f = 3.0 * e + f2 / e
        g = (0.5 * f * f + f2 / (1.0 + f2 / (a * a))) / e
        pint = sum(w * phi[s.site(*b)] for b, w in s.corners())
        fac = (1.0 + (4.0 + a * a / (e * e)) * pint) * (m / a) / e
        for b, w in s.corners():
            i = s.site(*b)
            ph = phi[i]
            T[0].index_add_(0, i, w * (e + f * ph + g * ph * ph) * (m / a))
            for row, c in ((1, 0), (4, 1), (6, 2)):
                T[row].index_add_(0, i, w * fac * v[:, c] * v[:, c])
        for row, c1, c2 in ((2, 0, 1), (3, 0, 2), (5, 1, 2)):
            u = 3 - c1 - c2
            for b in (0, 1):
                T[row].index_add_(0, s.site(*(b * n for n in unit(u))), s.w(u, b) * fac * v[:, c1] * v[:, c2])
        for c in range(3):
            u1, u2 = [k for k in range(3) if k != c]
            for b1 in (0, 1):
                for b2 in (0, 1):
                    b = tuple(b1 * x1 + b2 * x2 for x1, x2 in zip(unit(u1), unit(u2)))
                    T[7 + c].index_add_(0, s.site(*b), s.w(u1, b1) * s.w(u2, b2) * m * v[:, c])
    return T


def up(f, *axes):
    """f(x + e_i) for each axis i given (x, y, z = 0, 1, 2) of a [z, y, x] field."""
    for i in axes:
        f = torch.roll(f, -1, 2 - i)
    return f


def down(f, i):
    return torch.roll(f, 1, 2 - i)


def metric(T, phi, chi, case, a, dtau, N):
    """The field solves of one cycle: phi, chi, B_i, mean T00, phi's k = 0 mode."""
    fpg, dx2 = fourpig(N), 1.0 / (N * N)
    H = hconf(a, fpg, OM, OL)
    c, c2, c3 = 3.0 * H * dx2 / dtau, fpg * dx2 / a, 3.0 * H * H * dx2
    src = T[0].view(N, N, N)
    r = c2 * (src - OM) * (1.0 - 2.0 * phi * (1.0 - phi)) + (c3 * (1.0 - 3.0 * phi) - c) * phi - c3 * chi
    for i in range(3):
        r = r + 0.125 * (down(phi, i) - up(phi, i)) ** 2
    phi, hom = poisson(r, N, float(N * N), 3.0 * H / dtau)
    coeff = 2.0 * fpg * dx2 / a
    g, k, k2 = k_tables(N)
    safe = torch.where(k2 > 0.0, k2, 1.0)
    S = {}
    for row, (i, j) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
        if i == j:
            f = 0.5 * (up(phi, i) - down(phi, i)) ** 2
        else:
            u, v = up(phi, i) - phi, up(phi, j) - phi
            w = (up(phi, i, j) - up(phi, i)) - v
            f = 2.0 * u * v + w * (u + v + 0.5 * w)
        S[i, j] = S[j, i] = rfft3(f + coeff * T[1 + row].view(N, N, N))
    F = 0.0
    for i in range(3):
        F = F + (k2 - 3.0 * g[i]) * S[i, i]
        F = F - 6.0 * k[i] * k[(i + 1) % 3] * S[i, (i + 1) % 3]
    chi = irfft3(torch.where(k2 > 0.0, F / (2.0 * safe * safe * N), 0.0), N)
    B = torch.empty((3, N ** 3), device="cuda", dtype=F64)
    if case.get("parabolic"):
        fac = -2j * a * a * dtau / (safe * safe)
        for i in range(3):
            u, v = [m for m in range(3) if m != i]
            F = k[i].conj() * ((g[u] + g[v]) * S[i, i] - g[u] * S[u, u] - g[v] * S[v, v] - 2.0 * k[u] * k[v] * S[u, v])
            F = F + (g[u] + g[v] - g[i]) * (k[u] * S[i, u] + k[v] * S[i, v])
            B[i] = irfft3(torch.where(k2 > 0.0, fac * F, 0.0), N).reshape(-1)
    else:
        S = [rfft3((1.0 + phi + up(phi, i)) * T[7 + i].view(N, N, N)) for i in range(3)]
        long = (k[0] * S[0] + k[1] * S[1] + k[2] * S[2]) / safe
        for i in range(3):
            F = (S[i] - k[i].conj() * long) * (4.0 * fpg * dx2) / safe
            B[i] = irfft3(torch.where(k2 > 0.0, F, 0.0), N).reshape(-1)
    return phi, chi, B, float(src.mean()), float(hom)


def kick_drift(x, q, phi, chi, B, a, ad, dtau, N):
    """update_q at a, then update_pos at ad, in place; returns max |q| / a."""
    vmax = 0.0
    for o in range(0, len(x), CHUNK):
        s, v = Stencil(x[o:o + CHUNK], N), q[o:o + CHUNK].clone()
        f2 = (v * v).sum(dim=1)
        e2 = f2 + a * a
        ph = sum(w * phi[s.site(*b)] for b, w in s.corners())
        t = ph / e2
        t = 4.0 * t * f2 + (1.0 + a * a * t) * (f2 + e2) / e2
        grad = []
        for i in range(3):
            n = unit(i)
            gr = 0.0
            for b, w in s.corners():
                hi, lo = (tuple(x1 + sg * x2 for x1, x2 in zip(b, n)) for sg in (1, -1))
                gr = gr + 0.5 * w * (phi[s.site(*hi)] - phi[s.site(*lo)])
            gr = gr * t - (s.face(chi, i, 1) - s.face(chi, i))
            pb = (s.d[:, i] - 1.0) * s.face(B[i], i, -1) + (1.0 - 2.0 * s.d[:, i]) * s.face(B[i], i)
            pb = (pb + s.d[:, i] * s.face(B[i], i, 1)) * v[:, i]
            for j in range(3):
                if j != i:
                    m = 3 - i - j
                    pb = pb + (s.line(B[j], m, n) - s.line(B[j], m)) * v[:, j]
            grad.append(gr + pb / (a * a * N) / torch.sqrt(e2))
        v -= dtau * N * torch.sqrt(e2)[:, None] * torch.stack(grad, dim=1)
        q[o:o + CHUNK] = v
        f2 = (v * v).sum(dim=1)
        vmax = max(vmax, float(f2.max()) / (a * a))
        e2 = f2 + ad * ad
        ch = sum(w * chi[s.site(*b)] for b, w in s.corners())
        u = (1.0 + (3.0 - f2 / e2) * ph - ch) / torch.sqrt(e2)
        shift = torch.stack([s.face(B[i], i) for i in range(3)], dim=1) / (ad * ad * N)
        x[o:o + CHUNK] += dtau * (v * u[:, None] + shift)
    return math.sqrt(vmax)


def background(a, dtau, fpg):
    """One Runge-Kutta step of the scale factor."""
    f = lambda y: y * hconf(y, fpg, OM, OL)  # noqa: E731
    k1 = f(a)
    k2 = f(a + 0.5 * dtau * k1)
    k3 = f(a + 0.5 * dtau * k2)
    return a + dtau * (k1 + 2.0 * k2 + 2.0 * k3 + f(a + dtau * k3)) / 6.0


def exact_cycle(case, seed):
    N = case["N"]
    a, dtau, cosmo = cycle_start(case)
    x, q, phi, sites = box(N, case["np"], a, seed, case["z"] < 3.0)
    m = OM / case["np"] * float(N) ** 3
    T = deposit(x, q, m, phi.view(-1), a, N)
    phi, chi, B, t00, hom = metric(T, phi, torch.zeros_like(phi), case, a, dtau, N)
    del T
    ah = background(a, 0.5 * dtau, cosmo.fourpiG)
    v = kick_drift(x, q, phi.reshape(-1), chi.reshape(-1), B, a, ah, dtau, N)
    a = background(ah, 0.5 * dtau, cosmo.fourpiG)
    step = dtau if case["kind"] == "stages" else min(48.0 / N, cosmo.steplimit / hconf(a, cosmo.fourpiG, OM, OL))
    d = x - sites
    out = {"phi": phi, "chi": chi, "B": B.view(3, N, N, N),
           "particles": {"displacement": d - torch.round(d), "momentum": q},
           "scalars": np.array([a, step, t00, hom, v / math.sqrt(v * v + 1.0)])}
    if case.get("tensor"):
        out["hij"] = None
    if case.get("lightcone"):
        out["lightcone"] = None
    return out


def exact_spectrum(case, seed):
    N, nb = case["N"], case["bins"]
    x = box(N, case["np"], 1.0 / (1.0 + case["z"]), seed, case["z"] < 3.0)[0]
    rho = contrast(x, N, OM / case["np"] * float(N) ** 3)
    F = rfft3(rho.view(N, N, N))
    i = torch.arange(N, device="cuda", dtype=F64)
    i = torch.minimum(i, N - i)
    t = (2.0 * math.pi) * i
    lin = t * t
    sinc = torch.where(i > 0, torch.sin(math.pi * i / N) * N / (math.pi * torch.where(i > 0, i, 1.0)), 1.0)
    h = N // 2 + 1
    k2 = (lin[None, None, :h] + lin[None, :, None]) + lin[:, None, None]
    s = (sinc[None, None, :h] * sinc[None, :, None] * sinc[:, None, None]) ** 2
    p = F.real ** 2 + F.imag ** 2
    sk = torch.sqrt(k2)
    kmax = math.sqrt(3.0 * float(lin[N // 2]))
    b = torch.floor(nb * sk / torch.full_like(sk, kmax)).long().reshape(-1)
    wt = torch.full((N, N, h), 2.0, device="cuda", dtype=F64)
    wt[:, :, 0] = wt[:, :, N // 2] = 1.0
    wt[0, 0, 0] = 0.0
    b = b.clamp_(max=nb)
    acc = []
    for v in (sk, k2, p * k2 * sk / s, p * p * k2 ** 3 / s / s, torch.ones_like(k2)):
        acc.append(torch.zeros(nb + 1, device="cuda", dtype=F64).index_add_(0, b, (wt * v).reshape(-1))[:nb])
    n = torch.clamp(acc[4], min=1.0)
    return {"density": rho.view(N, N, N), "k": acc[0] / n, "power": acc[2] / n, "krms": torch.sqrt(acc[1] / n),
            "prms": torch.sqrt(acc[3] / n), "count": None}


def contrast(x, N, m):
    """CIC density of particles of mass m (per cell volume)."""
    s = Stencil(x, N)
    rho = torch.zeros(N ** 3, device="cuda", dtype=F64)
    for b, w in s.corners():
        rho = rho.index_add(0, s.site(*b), m * w)
    return rho


def pm_step(x, q, N, m, kq, kx, pc):
    psi = poisson(contrast(x, N, m).view(N, N, N), N, pc, 0.0)[0]
    s = Stencil(x, N)
    g = []
    for i in range(3):
        f = (0.5 * (up(psi, i) - down(psi, i))).reshape(-1)
        g.append(sum(w * f[s.site(*b)] for b, w in s.corners()))
    q = q - kq * torch.stack(g, dim=1)
    return x + kx * q, q


def exact_pm(case, seed):
    from torch.utils.checkpoint import checkpoint

    N, n = case["N"], case["np"]
    x0, q0, _, _ = box(N, n, 1.0 / 51.0, seed, False)
    coef, _ = gevpm.schedule(N, fourpig(N), OM, OL, 1.0 / 51.0, 1.0, case["steps"])
    m = OM / n * float(N) ** 3
    back = case["kind"] == "grad"
    x0.requires_grad_(back)
    q0.requires_grad_(back)
    x, q = x0, q0
    for kq, kx, pc in coef.reshape(-1, 3):
        x, q = checkpoint(pm_step, x, q, N, m, float(kq), float(kx), float(pc), use_reentrant=False)
    delta = contrast(x, N, float(N) ** 3 / n) - 1.0
    if not back:
        return {"delta": delta, "x": x, "q": q}
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 1)
    target = torch.randn(N ** 3, generator=g, device="cuda", dtype=torch.float32).to(F64)
    ((delta - target) ** 2).sum().backward()
    return {"delta": delta.detach(), "gx": x0.grad, "gq": q0.grad}


def exact(case, seed):
    if case["kind"] == "poisson":
        src = prepare(case, seed)["src"].to(F64)
        return poisson(src, case["N"], float(case["N"]), 1.0)[0]
    if case["kind"] in ("grad", "pm"):
        return exact_pm(case, seed)
    return exact_spectrum(case, seed) if case["kind"] == "spectrum" else exact_cycle(case, seed)
