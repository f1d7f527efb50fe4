"""The work a program has this library do, as cases that can be timed and compared.

Every case goes through the public entry points (`latfield2_b200.Context`,
`autodiff.pm_chain_loss` and, for device pointers that the Python wrapper does
not take, the C ABI).  A case is a dict of plain values:

  op       what one pass does (below)
  n0 n1 n2 lattice sites per dim; npart particles
  dist     uniform | clumps | lognormal (how the particles are placed)
  mode     fixed | fp32 | plain (deposit mode of the context)
  mass/ids per-particle masses / carried IDs
  steps    chain: kick-drift steps per pass; operator stencil | pm
  family   moments: ngp | full;  halo, real: layout of the caller's fields

  step     gather-kick, drift, rebin and the density (lf2_step)
  cycle    the same as separate calls, as updateVel (with its max |v|),
           moveParticles and two projections (density, momentum) run
  moments  the projections of a state: density, momentum and stress (ngp), or
           the staggered momentum and stress (full)
  pm       Poisson force of the density, then a step: a self-gravitating run
  coupled  an application with its own halo'd fields on the GPU: force in,
           step, density out with its halo filled
  load     a new set of particles into a context and its first density
  chain    loss and gradients of the differentiable multi-step chain

Sizes are those of the benchmark and the tests (64^3 to 512^3, about one
particle per cell) with velocities of 0.01 box units and time steps of
0.1 * 64 / n, so that a particle moves 0.06 cells per step.
"""
import math

import numpy as np
import torch

import latfield2_b200 as L
from latfield2_b200.autodiff import pm_chain_loss

MODES = {"fixed": L.DEPOSIT_FIXED64, "fp32": L.DEPOSIT_FP32, "plain": L.DEPOSIT_FP32_PLAIN}
PM_COUPLING = 0.03     # forces of the size of the benchmark's force field
CHAIN_COUPLING = 4 * math.pi


def _case(name, op, n, npart=None, dist="uniform", mode="fixed", **more):
    n = (n,) * 3 if isinstance(n, int) else n
    c = {"op": op, "n0": n[0], "n1": n[1], "n2": n[2],
         "npart": npart if npart else n[0] * n[1] * n[2], "dist": dist, "mode": mode,
         "mass": False, "ids": False}
    c.update(more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the benchmark's headline: the largest run of one GPU that its users quote
        _case("step_512_lognormal", "step", 512, dist="lognormal"),
        # the middle configuration, in the context's default deposit mode
        _case("step_256_clumps_fp32", "step", 256, dist="clumps", mode="fp32"),
        # the smallest configuration: launches and latency count
        _case("step_64_fp32", "step", 64, mode="fp32"),
        # a lattice that no tile divides, individual masses and IDs, the reference's call order
        _case("cycle_ragged_masses", "cycle", (150, 141, 133), dist="clumps", mass=True, ids=True),
        # the reference's call order at the middle size
        _case("cycle_256", "cycle", 256, dist="lognormal"),
        # T00, T0i and Tij of a relativistic code, every step
        _case("moments_ngp_256", "moments", 256, dist="lognormal", family="ngp"),
        # the staggered momentum and stress, default mode
        _case("moments_full_256_fp32", "moments", 256, dist="clumps", mode="fp32", family="full"),
        # a self-gravitating run
        _case("pm_256", "pm", 256, dist="lognormal"),
        # host code on the GPU that keeps double fields with a halo of 2
        _case("coupled_256_double", "coupled", 256, dist="lognormal", halo=2, real=8),
        # initial conditions or a restart
        _case("load_256_ids", "load", 256, dist="clumps", ids=True),
        # the differentiable chain's own configuration (forward and backward)
        _case("chain_stencil_128", "chain", 128, mode="fp32", operator="stencil", steps=8),
        # one step of it with the Poisson force and fixed-point deposits
        _case("chain_pm_256", "chain", 256, dist="clumps", operator="pm", steps=1),
    ]


def draw(rng):
    op = rng.choice(["step", "step", "cycle", "moments", "pm", "coupled", "load", "chain"])
    cubic = op in ("pm", "chain") or rng.random() < 0.5
    # sites per dim, spread over the logarithm; the costlier passes end sooner
    top = {"step": 480, "cycle": 320, "moments": 240, "pm": 384, "coupled": 320, "load": 288,
           "chain": 160}[op]

    def size():
        v = int(round(math.exp(rng.uniform(math.log(32), math.log(top)))))
        return v - v % 4 if rng.random() < 0.4 else v
    a = size()
    if cubic:
        n = (a - a % 2 if op in ("pm", "chain") else a,) * 3
    else:
        n = (a,) + tuple(max(32, min(top, int(round(a * rng.uniform(0.7, 1.3))))) for _ in range(2))
    sites = n[0] * n[1] * n[2]
    npart = int(sites * math.exp(rng.uniform(math.log(0.25), math.log(1.2))))
    mode = rng.choice(["fixed", "fixed", "fp32", "fp32", "plain"])
    c = _case(None, op, n, npart, rng.choice(["uniform", "clumps", "lognormal"]), mode)
    if op in ("step", "cycle", "load", "moments"):
        c["mass"] = rng.random() < 0.3
        c["ids"] = op != "moments" and rng.random() < 0.4
    if op == "moments":
        c["family"] = rng.choice(["ngp", "full"])
    if op == "coupled":
        c["halo"] = rng.choice([1, 2])
        c["real"] = rng.choice([4, 8])
    if op == "chain":
        c["operator"] = rng.choice(["stencil", "pm"])
        c["steps"] = rng.choice([1, 2, 4, 8])
        c["mode"] = rng.choice(["fixed", "fp32"])
    return c


# ------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _gaussian(n, g):
    """Real Gaussian field, P(k) ~ k^-2, unit variance, shape (n2, n1, n0)."""
    wk = torch.fft.rfftn(torch.randn(n[2], n[1], n[0], generator=g, device="cuda"))
    k = [torch.fft.fftfreq(m, device="cuda") * m for m in (n[2], n[1])]
    k.append(torch.fft.rfftfreq(n[0], device="cuda") * n[0])
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    f = torch.fft.irfftn(wk * torch.where(k2 > 0, k2.clamp_min(1e-12).rsqrt(), 0.0 * k2),
                         s=(n[2], n[1], n[0]))
    return (f - f.mean()) / f.std()


def _particles(case, seed):
    """int32 cells, FP32 in-cell offsets and velocities (box units)."""
    n = (case["n0"], case["n1"], case["n2"])
    npart = case["npart"]
    g = _gen(1000 + seed)
    if case["dist"] == "lognormal":  # rho ~ exp(2 delta - 2), cells drawn from it
        rho = torch.exp(2.0 * _gaussian(n, g).double() - 2.0).reshape(-1)
        # integer weights, whose running sum is the same bits in every run
        cdf = torch.cumsum((rho * 1048576.0).to(torch.int64), 0).double()
        u = torch.rand(npart, generator=g, device="cuda", dtype=torch.float64) * cdf[-1]
        cell = torch.searchsorted(cdf, u).clamp_max(rho.numel() - 1)
        off = torch.rand(npart, 3, generator=g, device="cuda")
    else:
        pos = torch.rand(npart, 3, generator=g, device="cuda", dtype=torch.float64)
        if case["dist"] == "clumps":  # half of them in 64 Gaussian clumps
            m = npart // 2
            centre = torch.rand(64, 3, generator=g, device="cuda", dtype=torch.float64)
            at = torch.randint(0, 64, (m,), generator=g, device="cuda")
            pos[:m] = torch.remainder(centre[at] + 0.01 * torch.randn(
                m, 3, generator=g, device="cuda", dtype=torch.float64), 1.0)
            pos = pos[torch.randperm(npart, generator=g, device="cuda")]
        u = pos * torch.tensor(n, dtype=torch.float64, device="cuda")
        fl = torch.floor(u)
        off = (u - fl).float()
        c = fl.to(torch.int64)
        for d in range(3):
            c[:, d].clamp_(0, n[d] - 1)
        cell = c[:, 0] + n[0] * (c[:, 1] + n[1] * c[:, 2])
    off = off.clamp_(0.0, 1.0 - 2.0 ** -24)
    vel = 0.01 * torch.randn(npart, 3, generator=g, device="cuda")
    return cell.to(torch.int32).contiguous(), off.contiguous(), vel.contiguous()


def _masses(case, seed):
    if not case["mass"]:
        return None
    u = torch.rand(case["npart"], generator=_gen(2000 + seed), device="cuda")
    return ((0.9 + 0.2 * u) / case["npart"]).contiguous()


def _force(n, seed):
    """Central differences of a Gaussian field, rms 0.01, shape (3, n2, n1, n0)."""
    phi = _gaussian(n, _gen(3000 + seed))
    F = torch.stack([0.5 * (torch.roll(phi, -1, a) - torch.roll(phi, 1, a)) for a in (2, 1, 0)])
    return (F * (0.01 / F.std())).contiguous()


def _to_reference(F, halo, real):
    """(comps, n2, n1, n0) -> the reference's layout (z, y, x, comps) with its halo, zeros there."""
    t = torch.float64 if real == 8 else torch.float32
    c, n2, n1, n0 = F.shape
    out = torch.zeros(n2 + 2 * halo, n1 + 2 * halo, n0 + 2 * halo, c, dtype=t, device="cuda")
    out[halo:halo + n2, halo:halo + n1, halo:halo + n0] = F.permute(1, 2, 3, 0)
    return out


def _chain_inputs(case, seed):
    n, npart = (case["n0"],) * 3, case["npart"]
    cell, off, vel = _particles(case, seed)
    c = cell.to(torch.int64)
    pos = torch.stack([c % n[0], (c // n[0]) % n[0], c // (n[0] * n[0])], 1).double()
    pos = (pos + off.double()) / n[0]
    g = _gen(4000 + seed)
    m = (1.0 + 0.1 * (2 * torch.rand(npart, generator=g, device="cuda", dtype=torch.float64) - 1))
    S = 0.02 * torch.randn(81, generator=g, device="cuda", dtype=torch.float64)
    w = torch.randn(n[0] ** 3, generator=g, device="cuda", dtype=torch.float64)
    return pos, vel.double(), m / npart, S if case["operator"] == "stencil" else None, w


def _dt(case):
    return 0.1 * 64.0 / case["n0"]


def prepare(case, seed):
    n = (case["n0"], case["n1"], case["n2"])
    ctx = L.Context(n, box=1.0, mode=MODES[case["mode"]])
    s = {"case": case, "ctx": ctx, "dt": _dt(case)}
    if case["op"] == "chain":
        s["leaves"] = [t if t is None else t.requires_grad_(True) for t in _chain_inputs(case, seed)]
        return s
    cell, off, vel = _particles(case, seed)
    mass = _masses(case, seed)
    ids = torch.arange(case["npart"], device="cuda") if case["ids"] else None
    gm = 0.0 if mass is not None else 1.0 / case["npart"]
    if case["op"] == "load":
        s["set"] = (cell, off, vel, mass, gm, ids)
    else:
        ctx.set_particles(cell, off, vel, mass=mass, global_mass=gm, ids=ids)

    def field(comps):
        t = torch.zeros(comps, n[2], n[1], n[0], device="cuda")
        return t, ctx.field(comps, t)
    s["rho"] = field(1)
    if case["op"] == "moments":
        s["vec"], s["ten"] = field(3), field(6)
    elif case["op"] == "cycle":
        s["vec"] = field(3)
    if case["op"] in ("step", "cycle", "pm", "coupled"):
        s["F"] = field(3)
    if case["op"] in ("step", "cycle"):
        s["F"][0].copy_(_force(n, seed))
    elif case["op"] == "pm":
        ctx.deposit_scalar(s["rho"][1])
    elif case["op"] == "coupled":
        s["F_in"] = _to_reference(_force(n, seed), case["halo"], case["real"])
        h = 2 * case["halo"]
        s["rho_out"] = torch.zeros(n[2] + h, n[1] + h, n[0] + h, dtype=s["F_in"].dtype, device="cuda")
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case, ctx, dt = s["case"], s["ctx"], s["dt"]
    op = case["op"]
    if op == "step":
        ctx.step(s["F"][1], dt, dt, s["rho"][1])
        return {"rho": s["rho"][0]}
    if op == "cycle":
        max_v = ctx.gather_kick(s["F"][1], dt, want_max_v=True)
        ctx.drift_rebin(dt)
        ctx.deposit_scalar(s["rho"][1])
        ctx.deposit_vector(s["vec"][1])
        return {"rho": s["rho"][0], "momentum": s["vec"][0], "max_v": max_v}
    if op == "moments":
        if case["family"] == "full":
            ctx.deposit_vector_cic(s["vec"][1])
            ctx.deposit_vecvec_cic(s["ten"][1])
            return {"momentum": s["vec"][0], "stress": s["ten"][0]}
        ctx.deposit_scalar(s["rho"][1])
        ctx.deposit_vector(s["vec"][1])
        ctx.deposit_symtensor(s["ten"][1])
        return {"rho": s["rho"][0], "momentum": s["vec"][0], "stress": s["ten"][0]}
    if op == "pm":
        ctx.pm_force(s["rho"][1], s["F"][1], PM_COUPLING)
        ctx.step(s["F"][1], dt, dt, s["rho"][1])
        return {"force": s["F"][0], "rho": s["rho"][0]}
    if op == "coupled":
        s["F"][1].import_(s["F_in"], halo=case["halo"])
        ctx.step(s["F"][1], dt, dt, s["rho"][1])
        out = s["rho_out"]
        L._lib.check(ctx.h, L.load().lf2_field_export(
            ctx.h, s["rho"][1].h, out.data_ptr(), case["halo"], case["real"], 1, L._lib.PTR_DEVICE),
            "field_export")
        return {"rho": out}
    if op == "load":
        cell, off, vel, mass, gm, ids = s["set"]
        ctx.set_particles(cell, off, vel, mass=mass, global_mass=gm, ids=ids)
        ctx.deposit_scalar(s["rho"][1])
        return {"rho": s["rho"][0]}
    pos, vel, m, S, w = s["leaves"]
    loss = pm_chain_loss(ctx, pos, vel, m, S, w, steps=case["steps"], dt=dt, checkpoint_every=2,
                         operator=case["operator"], coupling=CHAIN_COUPLING)
    leaves = [t for t in s["leaves"] if t is not None]
    grads = torch.autograd.grad(loss, leaves)
    return {"loss": loss.detach(), "grads": list(grads)}


# ---------------------------------------------------------- necessary work
def work(case):
    """Each input read once, each output written once (a particle: cell,
    offsets and velocity, 28 bytes, with its mass and ID where it has them)."""
    sites, npart, op = case["n0"] * case["n1"] * case["n2"], case["npart"], case["op"]
    state = 28 + (4 if case["mass"] else 0) + (8 if case["ids"] else 0)
    extra = 4 if case["mass"] else 0
    if op == "step":
        b, f = npart * 2 * state + sites * 16, npart * 130
    elif op == "cycle":
        b, f = npart * 2 * state + sites * 28, npart * 200
    elif op == "moments" and case["family"] == "ngp":
        b, f = npart * (28 + extra) + sites * 40, npart * 200
    elif op == "moments":
        b, f = npart * (28 + extra) + sites * 36, npart * 300
    elif op == "pm":
        b, f = npart * 2 * state + sites * 20, npart * 130 + sites * 5 * math.log2(sites)
    elif op == "coupled":
        b, f = npart * 2 * state + sites * (12 + case["real"] * 4), npart * 130
    elif op == "load":
        b, f = npart * 2 * state + sites * 4, npart * 50
    else:  # positions, velocities and masses in, their gradients out, w and its gradient
        b = npart * 112 + sites * 16
        f = case["steps"] * (npart * 500 + sites * (27 * 3 * 6 if case["operator"] == "stencil" else 300))
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    if case["op"] == "chain":
        # FP32 state through every step; CIC gradients jump at cell faces, and
        # a particle within rounding of a face may land on its other side
        # (1e-3, single particles 2 of the rms, against 64 bits)
        return {"rel": 4e-3, "max": 0.9}
    if case["op"] == "pm":
        # differences of an FP32 potential: 1e-5 against 64 bits at 352^3
        return {"rel": 4e-5, "max": 5e-4}
    if case["mode"] == "fixed":
        return "exact"  # integer sums: the same bits in any order
    if case["mode"] == "fp32":
        # compensated sums: 6e-8, single sites 3e-6 of the rms, against 64 bits
        return {"rel": 2.4e-7, "max": 1.3e-5}
    return {"rel": 2e-6, "max": 5e-5}


# --------------------------------------------------------- the same in 64 bits
CHUNK = 1 << 24


def _corner_sites(n, c, shift=(0, 0, 0)):
    x = torch.remainder(c[0] + shift[0], n[0])
    y = torch.remainder(c[1] + shift[1], n[1])
    z = torch.remainder(c[2] + shift[2], n[2])
    return x + n[0] * (y + n[1] * z)


def _split(n, cell):
    c = cell.to(torch.int64)
    return [c % n[0], (c // n[0]) % n[1], c // (n[0] * n[1])]


def _bits(q):
    return (q >> 2) & 1, (q >> 1) & 1, q & 1


def _spread(out, n, c, f, value, dims=(True, True, True)):
    """out += value spread with CIC weights along the dims asked for, the
    cell's own vertex along the others."""
    for q in range(8):
        b = _bits(q)
        if any(b[d] and not dims[d] for d in range(3)):
            continue
        w = value
        for d in range(3):
            if dims[d]:
                w = w * (f[d] if b[d] else 1.0 - f[d])
        out.index_add_(0, _corner_sites(n, c, b), w)


def _staggered(c, f, dims):
    """Cell and offset on the grid moved by half a cell along the dims."""
    c2, f2 = list(c), list(f)
    for d in range(3):
        if dims[d]:
            s = f[d] - 0.5
            up = s >= 0
            c2[d] = torch.where(up, c[d], c[d] - 1)
            f2[d] = torch.where(up, s, s + 1.0)
    return c2, f2


def _projection64(n, vol, kind, c, f, v, m):
    """Adds of one chunk: a function of the output (comps, sites)."""
    def into(out):
        mv = m / vol
        pairs = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))
        if kind == "rho":
            _spread(out[0], n, c, f, mv)
        elif kind == "vec":
            for i in range(3):
                _spread(out[i], n, c, f, mv * v[i], [d != i for d in range(3)])
        elif kind == "ten":
            for k, (i, j) in enumerate(pairs):
                _spread(out[k], n, c, f, mv * v[i] * v[j],
                        [True] * 3 if i == j else [d not in (i, j) for d in range(3)])
        elif kind == "vec_cic":
            for i in range(3):
                c2, f2 = _staggered(c, f, [d == i for d in range(3)])
                _spread(out[i], n, c2, f2, mv * v[i])
        else:
            for k, (i, j) in enumerate(pairs):
                c2, f2 = (c, f) if i == j else _staggered(c, f, [d in (i, j) for d in range(3)])
                _spread(out[k], n, c2, f2, mv * v[i] * v[j])
    return into


COMPS = {"rho": 1, "vec": 3, "ten": 6, "vec_cic": 3, "ten_cic": 6}


def _poisson64(rho, n, coupling):
    """F (3, sites): lap7(phi) = coupling (rho - mean), F = -grad phi."""
    m, res = n[0], 1.0 / n[0]
    K = torch.fft.rfftn(rho.reshape(m, m, m))
    k = torch.arange(m, dtype=torch.float64, device="cuda")
    s2 = torch.sin(math.pi * k / m) ** 2
    lam = s2[:, None, None] + s2[None, :, None] + s2[None, None, :m // 2 + 1]
    lam[0, 0, 0] = 1.0
    G = -0.25 * coupling * res * res / lam
    G[0, 0, 0] = 0.0
    phi = torch.fft.irfftn(K * G, s=(m, m, m))
    return torch.stack([((torch.roll(phi, 1, a) - torch.roll(phi, -1, a)) / (2 * res)).reshape(-1)
                        for a in (2, 1, 0)])


def _move64(n, res, c, f, v, F, dt):
    """Kick with the CIC gather of F (3, sites) (None: no move), then drift."""
    a = [torch.zeros_like(f[0]) for _ in range(3)]
    for q in range(8):
        b = _bits(q)
        w = torch.ones_like(f[0])
        for d in range(3):
            w = w * (f[d] if b[d] else 1.0 - f[d])
        s = _corner_sites(n, c, b)
        for i in range(3):
            a[i] += w * F[i][s].double()
    c2, f2, v2 = [], [], []
    for d in range(3):
        v2.append(v[d] + dt * a[d])
        u = f[d] + dt / res * v2[d]
        fl = torch.floor(u)
        c2.append(torch.remainder(c[d] + fl.to(torch.int64), n[d]))
        f2.append(u - fl)
    return c2, f2, v2


def _chain64(case, seed):
    pos, vel, m, S, w = _chain_inputs(case, seed)
    leaves = [t.requires_grad_(True) for t in (pos, vel, m, S, w) if t is not None]
    n, res, dt = (case["n0"],) * 3, 1.0 / case["n0"], _dt(case)

    def corners(x):
        u = x / res
        fl = torch.floor(u).detach()
        f, ci = u - fl, fl.to(torch.int64).unbind(1)
        for q in range(8):
            b = _bits(q)
            wt = torch.ones_like(f[:, 0])
            for d in range(3):
                wt = wt * (f[:, d] if b[d] else 1.0 - f[:, d])
            yield _corner_sites(n, ci, b), wt

    def density(x):
        rho = torch.zeros(n[0] ** 3, dtype=torch.float64, device="cuda")
        for s, wt in corners(x):
            rho = rho.index_add(0, s, wt * m / res ** 3)
        return rho
    x, v = pos, vel
    for _ in range(case["steps"]):
        rho = density(x)
        if S is None:
            F = _poisson64(rho, n, CHAIN_COUPLING)
        else:
            r = rho.reshape(n[2], n[1], n[0])
            acc = [0.0, 0.0, 0.0]
            for o in range(27):
                sh = torch.roll(r, (1 - o // 9, 1 - (o // 3) % 3, 1 - o % 3), (0, 1, 2))
                acc = [acc[i] + S[27 * i + o] * sh for i in range(3)]
            F = torch.stack([t.reshape(-1) for t in acc])
        G = sum((wt * F[:, s] for s, wt in corners(x)), torch.zeros(3, case["npart"], device="cuda",
                                                                    dtype=torch.float64))
        v = v + dt * G.t()
        x = x + dt * v
    loss = torch.dot(w, density(x))
    return {"loss": loss.detach(), "grads": [t.detach() for t in torch.autograd.grad(loss, leaves)]}


def exact(case, seed):
    op = case["op"]
    if op == "chain":
        if case["steps"] * case["npart"] > 1 << 25:
            return None  # autograd in 64 bits would not fit
        return _chain64(case, seed)
    n = (case["n0"], case["n1"], case["n2"])
    sites, res, dt = n[0] * n[1] * n[2], 1.0 / case["n0"], _dt(case)
    cell, off, vel = _particles(case, seed)
    mass = _masses(case, seed)
    kinds = {"step": ["rho"], "cycle": ["rho", "vec"], "pm": ["rho"], "coupled": ["rho"],
             "load": ["rho"]}.get(op) or (["vec_cic", "ten_cic"] if case["family"] == "full"
                                          else ["rho", "vec", "ten"])

    def project(kinds, F, dt):
        out = {k: torch.zeros(COMPS[k], sites, dtype=torch.float64, device="cuda") for k in kinds}
        top = 0.0
        for p in range(0, case["npart"], CHUNK):
            e = min(case["npart"], p + CHUNK)
            c = _split(n, cell[p:e])
            f = list(off[p:e].double().unbind(1))
            v = list(vel[p:e].double().unbind(1))
            m = mass[p:e].double() if mass is not None else torch.full_like(f[0], 1.0 / case["npart"])
            if F is not None:
                c, f, v = _move64(n, res, c, f, v, F, dt)
            top = max(top, float((v[0] ** 2 + v[1] ** 2 + v[2] ** 2).max()))
            for k in kinds:
                _projection64(n, res ** 3, k, c, f, v, m)(out[k])
        return {k: t.reshape(COMPS[k], n[2], n[1], n[0]) for k, t in out.items()}, math.sqrt(top)

    F = None
    if op in ("step", "cycle", "coupled"):
        F = _force(n, seed).reshape(3, -1)
    elif op == "pm":
        rho0, _ = project(["rho"], None, dt)
        F = _poisson64(rho0["rho"].reshape(-1), n, PM_COUPLING)
    got, top = project(kinds, F, dt)
    if op == "cycle":
        return {"rho": got["rho"], "momentum": got["vec"], "max_v": np.float64(top)}
    if op == "pm":
        return {"force": F.reshape(3, n[2], n[1], n[0]), "rho": got["rho"]}
    if op == "moments" and case["family"] == "full":
        return {"momentum": got["vec_cic"], "stress": got["ten_cic"]}
    if op == "moments":
        return {"rho": got["rho"], "momentum": got["vec"], "stress": got["ten"]}
    if op == "coupled":
        h = case["halo"]
        at = [torch.remainder(torch.arange(-h, n[d] + h, device="cuda"), n[d]) for d in (2, 1, 0)]
        r = got["rho"][0]
        return {"rho": r[at[0]][:, at[1]][:, :, at[2]]}
    return {"rho": got["rho"]}
