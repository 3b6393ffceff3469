"""The work that is timed: calls of the package's public entry points over the sizes, types and options they are used with.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes what a program holds before
the call, ``run`` is one pass, ``work`` the bytes and operations a pass cannot do without, and ``exact`` the outputs in 64
bits from plain torch. The kinds of case:

level     RK4 steps of one periodic box (``PeriodicLevel.advance``)
dropin    one RK4 step stage by stage on AMReX-layout boxes with ghosts, as a host with its own RK driver runs it
diag      the post-timestep pass: string count, pierced list, energies, velocities
ensemble  RK4 steps of independent boxes of uneven sizes
gradient  a smooth string-core loss after an evolution, with its gradients (forward and backward)
twolevel  coarse steps of a refined level, each with two subcycled fine steps on the tagged patches

Fields are Gaussian random fields cut off at a wavelength of ``cut`` cells, psi of rms R(tau) and Pi smaller: the initial
data of a string simulation, which a seed alone determines. The clock stands at the same step in every pass.
"""
import math

import numpy as np
import torch

import axion_strings_adaptive_gb300 as axs
from axion_strings_adaptive_gb300 import adjoint, amr

DX, DT, LAMBDA0 = 0.5, 0.1, 2.0
ENSEMBLE_SIZES = (32, 48, 64, 96, 128)
TYPES = {"f32": torch.float32, "f64": torch.float64}


def listed():
    return [
        # the plain configuration: a fat-string FP64 run of a small box, where launches and latency count
        dict(name="level 64^3 f64", kind="level", dtype="f64", nx=64, ny=64, nz=64, steps=10, c0=1.0, a_inv=2.0, tau=1.0, cut=4),
        # a host that calls the level hook once per step, physical strings, a mid-sized box
        dict(name="level 256^3 f32 one step", kind="level", dtype="f32", nx=256, ny=256, nz=256, steps=1, c0=0.0, a_inv=2.0, tau=1.0, cut=8),
        # a box whose sides suit no tile, matter domination
        dict(name="level 200x150x90 f32", kind="level", dtype="f32", nx=200, ny=150, nz=90, steps=4, c0=1.0, a_inv=1.5, tau=2.0, cut=8),
        # the production configuration: Moore strings on a large box
        dict(name="level 512^3 f32", kind="level", dtype="f32", nx=512, ny=512, nz=512, steps=4, c0=2.0, a_inv=2.0, tau=1.0, cut=8),
        # its FP64 counterpart, which a precision study runs beside it
        dict(name="level 256^3 f64", kind="level", dtype="f64", nx=256, ny=256, nz=256, steps=2, c0=2.0, a_inv=2.0, tau=1.0, cut=8),
        # the drop-in hooks on one AMReX box with the reference's ghost width
        dict(name="dropin 128^3 f32", kind="dropin", dtype="f32", nx=128, ny=128, nz=128, ng=3, c0=0.0, a_inv=2.0, tau=1.0, cut=8),
        # the same in FP64 on a ragged box
        dict(name="dropin 97x75x50 f64", kind="dropin", dtype="f64", nx=97, ny=75, nz=50, ng=3, c0=1.0, a_inv=2.0, tau=1.0, cut=8),
        # the post-timestep diagnostics as the reference computes them, with the pierced list
        dict(name="diag 256^3 f32", kind="diag", dtype="f32", nx=256, ny=256, nz=256, cells32=False, pierced=True, scheme=1, c0=1.0, a_inv=2.0, tau=10.0, cut=16),
        # the same sums with FP32 per-cell terms on the production box, counts only
        dict(name="diag 512^3 f32 cells", kind="diag", dtype="f32", nx=512, ny=512, nz=512, cells32=True, pierced=False, scheme=1, c0=2.0, a_inv=2.0, tau=10.0, cut=32),
        # a batch of seeded realisations of uneven sizes
        dict(name="ensemble 24 boxes f32", kind="ensemble", dtype="f32", boxes=24, layout=7, steps=8, c0=1.0, a_inv=2.0, tau=1.0, cut=8),
        # gradients through an evolution with checkpoints
        dict(name="gradient 128^3 f32", kind="gradient", dtype="f32", nx=128, ny=128, nz=128, steps=40, every=20, c0=1.0, a_inv=2.0, tau=1.0, cut=8),
        # a refined level: patches on the blocks along strings, as many as a dense network refines
        dict(name="twolevel 256^3 f32", kind="twolevel", dtype="f32", nx=256, ny=256, nz=256, block=16, layout=3, share=0.4, steps=1, c0=0.0, a_inv=2.0, tau=1.0, cut=64),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _box(rng, lo, hi, mult, least=8):
    """A box of lo^3 to hi^3 cells: half of them cubes of whole 16s or 32s, half of any shape (nx a multiple of mult)."""
    n = _log(rng, lo, hi)
    if rng.random() < 0.5:
        s = int(rng.choice((16, 32)))
        n = max(s, int(n) // s * s)
        return dict(nx=n, ny=n, nz=n)
    a, b = _log(rng, 0.7, 1.4), _log(rng, 0.7, 1.4)
    # the product of the three sides stays n^3
    sides = [max(least, round(n * f)) for f in (a, b, 1.0 / (a * b))]
    return dict(nx=max(mult, sides[0] // mult * mult), ny=sides[1], nz=sides[2])


def draw(rng):
    kind = rng.choice(("level", "level", "level", "dropin", "diag", "ensemble", "gradient", "twolevel"))
    dtype = "f64" if rng.random() < 0.3 else "f32"
    c0 = float(rng.choice((0.0, 1.0, 2.0)))
    # physical strings (c0 = 0) shrink against the grid: it resolves them early on only
    case = dict(kind=kind, dtype=dtype, c0=c0, a_inv=float(rng.choice((2.0, 2.0, 1.5))) if c0 else 2.0,
                tau=round(_log(rng, 1.0, 10.0 if c0 else 1.5), 3), cut=int(rng.choice((4, 8, 16, 32))))
    if kind == "level":
        case |= _box(rng, 48, 210 if dtype == "f64" else 440, 2 if dtype == "f64" else 4)
        case["steps"] = rng.randint(1, 3 if dtype == "f64" else 6)
    elif kind == "dropin":
        case |= _box(rng, 24, 96 if dtype == "f64" else 256, 1) | dict(ng=rng.choice((2, 3, 4)))
    elif kind == "diag":
        f32 = dtype == "f32"
        cells32 = f32 and rng.random() < 0.5
        case |= _box(rng, 48, 400 if cells32 else 230, 4) | dict(cells32=cells32, pierced=rng.random() < 0.5, scheme=rng.choice((0, 1, 2)),
                                                                             cut=int(rng.choice((16, 32))))
    elif kind == "ensemble":
        case |= dict(boxes=rng.randint(3, 20 if dtype == "f32" else 5), layout=rng.randint(0, 9999), steps=rng.randint(1, 8 if dtype == "f32" else 2))
    elif kind == "gradient":
        case |= _box(rng, 24, 110 if dtype == "f32" else 48, 4) | dict(steps=rng.randint(8, 30), every=rng.randint(4, 16))
    else:
        case["dtype"] = "f32" if rng.random() < 0.8 else "f64"
        n = int(rng.choice((64, 96, 128) if case["dtype"] == "f64" else (64, 96, 128, 160, 192, 224)))
        case |= dict(nx=n, ny=n, nz=int(rng.choice((64, 96, n))), block=16, layout=rng.randint(0, 9999), share=round(rng.uniform(0.1, 0.5), 2),
                     steps=rng.randint(1, 2), cut=int(rng.choice((32, 48, 64))))
    return case


# ------------------------------------------------------------------------------------------------ inputs
def _dtype(case):
    return TYPES[case["dtype"]]


def _radius(case, tau):
    b = case["a_inv"] - 1.0
    return tau ** (1.0 / b) / b


def _field(n, cut, rms, dtype, gen):
    """One random component (nz, ny, nx) of modes of wavelength over `cut` cells."""
    nx, ny, nz = n
    f = torch.fft.rfftn(torch.randn((nz, ny, nx), generator=gen, device="cuda", dtype=dtype))
    k2 = (torch.fft.fftfreq(nz, device="cuda")[:, None, None] ** 2 + torch.fft.fftfreq(ny, device="cuda")[None, :, None] ** 2 +
          torch.fft.rfftfreq(nx, device="cuda")[None, None, :] ** 2)
    f *= (k2 < max(1.0 / cut, 2.5 / min(n)) ** 2) & (k2 > 0)
    f = torch.fft.irfftn(f, s=(nz, ny, nx))
    return f.mul_(rms * math.sqrt(f.numel()) / f.norm())


def _state(case, n, gen):
    R = _radius(case, case["tau"])
    out = torch.empty((4, n[2], n[1], n[0]), dtype=_dtype(case), device="cuda")
    for c in range(4):
        out[c] = _field(n, case["cut"], R * (math.sqrt(0.5) if c < 2 else 0.2), _dtype(case), gen)
    return out


def _dims(case):
    """The sizes of an ensemble's cubes, uniform over the set."""
    r = np.random.RandomState(case["layout"])
    return [(int(s),) * 3 for s in r.choice(ENSEMBLE_SIZES, case["boxes"])]


def _blocks(case):
    """The refined blocks (x, y, z): along the zeros of a smooth random field, `share` of all."""
    nb = [case[a] // case["block"] for a in ("nz", "ny", "nx")]
    f = np.random.RandomState(case["layout"]).standard_normal(nb)
    for d in range(3):
        f = f + np.roll(f, 1, d) + np.roll(f, -1, d)
    near = np.argsort(np.abs(f).reshape(-1), kind="stable")[:max(1, int(case["share"] * f.size))]
    return np.stack(np.unravel_index(np.sort(near), nb), 1)[:, ::-1]


def _fields(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["kind"] == "ensemble":
        return [_state(case, n, gen) for n in _dims(case)]
    return _state(case, (case["nx"], case["ny"], case["nz"]), gen)


def prepare(case, seed):
    kind, dt = case["kind"], _dtype(case)
    bg = axs.Background.expanding(case["a_inv"], case["c0"], lambda0=LAMBDA0)
    s = dict(case=case, bg=bg)
    v = _fields(case, seed)
    if kind == "ensemble":
        s["e"] = e = axs.Ensemble(_dims(case), DX, dtype=dt)
        for b, x in enumerate(v):
            e.set_box(b, x)
        e.fill_ghosts()
        return s
    n = (case["nx"], case["ny"], case["nz"])
    if kind in ("level", "diag", "twolevel"):
        s["level"] = lv = axs.PeriodicLevel(n, DX, dtype=dt, pierced_capacity=None if kind == "diag" else 1)
        lv.set_state(v)
    if kind == "twolevel":
        s["two"] = amr.TwoLevel(lv, case["block"])
        s["two"].set_blocks(_blocks(case))
    if kind == "dropin":
        s["u"], s["stage"] = (axs.new_fab(n, case["ng"], dtype=dt) for _ in range(2))
        s["k"] = [axs.new_fab(n, 0, dtype=dt) for _ in range(4)]
        axs.valid(s["u"], case["ng"]).copy_(v)
    if kind == "gradient":
        s["x"] = v.requires_grad_()
        s["lam"] = torch.tensor(LAMBDA0, device="cuda", dtype=dt, requires_grad=True)
        s["spec"] = adjoint.EvolutionSpec(dx=DX, dt=DT, nsteps=case["steps"], tau_i=case["tau"], a_inv=case["a_inv"],
                                          c0=case["c0"], checkpoint_every=case["every"])
    return s


# ------------------------------------------------------------------------------------------------ one pass
def _dropin_step(s):
    """GRTeclyn's classic RK4 on the drop-in hooks: stage times t, t + dt/2, t + dt/2, t + dt."""
    case, bg, u, st, k = s["case"], s["bg"], s["u"], s["stage"], s["k"]
    ng, tau = case["ng"], case["tau"]
    src = u
    for i, c in enumerate((0.0, 0.5, 0.5, 1.0)):
        if i:
            axs.lincomb(axs.valid(st, ng), axs.valid(u, ng), c * DT, k[i - 1], 0)
            src = st
        axs.fill_periodic_ghosts(src, ng)
        axs.eval_rhs(src, k[i], ng, 0, DX, bg.rhs_coeffs(tau + c * DT))
    axs.rk4_combine(axs.valid(u, ng), axs.valid(u, ng), *k, 0, DT)
    return axs.valid(u, ng)


def _patch_cells(p):
    """The valid cells of every patch, (4, patches, z, y, x), as a view of the arena."""
    lay, n = p.layout, p.n
    return p.state.as_strided((4, p.npatches, n, n, n), (lay.plane_elems, lay.patch_elems, lay.kstride, lay.jstride, 1),
                              p.state.storage_offset() + lay.z_offset * lay.kstride + lay.y_offset * lay.jstride + lay.x_offset)


def run(s):
    case, bg = s["case"], s["bg"]
    kind, tau = case["kind"], case["tau"]
    if kind == "level":
        s["level"].advance(bg, tau, 0.0, DT, case["steps"])
        return s["level"].valid_view()
    if kind == "dropin":
        return _dropin_step(s)
    if kind == "diag":
        d = s["level"].diagnostics(bg, tau, case["scheme"], 0.8, want_list=case["pierced"], per_cell_fp32=case["cells32"])
        out = dict(count=d.n_p_plain, weighted=d.n_p_weighted, corners=d.vel_count, energy=np.array(d.energy_sums), velocity=d.vel_sum)
        if case["pierced"]:
            # a map of the pierced faces (entry 4 cell + plane; the list comes in any order)
            out["pierced"] = torch.zeros(4 * s["level"].n_cells, dtype=torch.uint8, device="cuda").index_fill_(0, d.pierced, 1)
        return out
    if kind == "ensemble":
        s["e"].advance(bg, tau, 0.0, DT, case["steps"])
        return [s["e"].box_view(b) for b in range(case["boxes"])]
    if kind == "gradient":
        loss = adjoint.string_core_loss(s["x"], s["lam"], s["spec"])
        g = torch.autograd.grad(loss, (s["x"], s["lam"]))
        return dict(loss=loss.detach(), state=g[0], lam=g[1])
    s["two"].advance(bg, tau, 0.0, DT, case["steps"])
    return dict(coarse=s["level"].valid_view(), fine=_patch_cells(s["two"].patches))


def work(case):
    """Bytes: the state in and out of each step (of each call, where the caller sees its result). Operations: a Laplacian
    takes 25, a step 8 of them and about 80 more per site; an adjoint step reads two states and takes twice that."""
    es = 4 if case["dtype"] == "f32" else 8
    if case["kind"] == "ensemble":
        cells = sum(n[0] ** 3 for n in _dims(case))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    step_bytes, step_flops = 8 * es * cells, 280 * cells
    kind = case["kind"]
    if kind == "dropin":
        return dict(bytes=92 * es * cells, flops=280 * cells)
    if kind == "diag":
        return dict(bytes=4 * es * cells, flops=200 * cells)
    if kind == "gradient":
        return dict(bytes=case["steps"] * (step_bytes + 12 * es * cells), flops=3 * case["steps"] * step_flops)
    if kind == "twolevel":
        fine = 2 * 8 * case["share"]  # two fine steps, eight fine cells to a refined coarse one
        return dict(bytes=case["steps"] * (1 + fine) * step_bytes, flops=case["steps"] * (1 + fine) * step_flops)
    return dict(bytes=case["steps"] * step_bytes, flops=case["steps"] * step_flops)


# ------------------------------------------------------------------------------------------------ in 64 bits
def _lap(f):
    out = -7.5 * f
    for d in (-1, -2, -3):
        out += (4.0 / 3.0) * (f.roll(1, d) + f.roll(-1, d)) - (1.0 / 12.0) * (f.roll(2, d) + f.roll(-2, d))
    return out / DX ** 2


def _coeffs(case, tau, lam0):
    b = case["a_inv"] - 1.0
    R = _radius(case, tau)
    return (1.0 - b) / (b * b * tau * tau), lam0 * (R * b) ** (-2.0 * case["c0"]), R


def _rhs(case, y, tau, lam0):
    kappa, lam, R = _coeffs(case, tau, lam0)
    mod = y[0] * y[0] + y[1] * y[1]
    pot = kappa - 0.5 * lam * (mod - R * R)
    return torch.stack((y[2], y[3], _lap(y[0]) + pot * y[0], _lap(y[1]) + pot * y[1]))


def _rk4(case, y, t, lam0):
    tau = case["tau"] + t
    k1 = _rhs(case, y, tau, lam0)
    k2 = _rhs(case, y + 0.5 * DT * k1, tau + 0.5 * DT, lam0)
    acc = k1 + 2.0 * k2
    k3 = _rhs(case, y + 0.5 * DT * k2, tau + 0.5 * DT, lam0)
    acc = acc + 2.0 * k3
    k4 = _rhs(case, y + DT * k3, tau + DT, lam0)
    return y + (DT / 6.0) * (acc + k4)


def _evolved(case, y, steps):
    for i in range(steps):
        y = _rk4(case, y, i * DT, LAMBDA0)
    return y


def _diff(f, d):
    return (8.0 * (f.roll(-1, d) - f.roll(1, d)) - (f.roll(-2, d) - f.roll(2, d))) / (12.0 * DX)


def _energies(case, y):
    """The 14 sums of the energy pass: each density, and the density times the masking weight; the weights; the cells."""
    _, lam, R = _coeffs(case, case["tau"], LAMBDA0)
    b = case["a_inv"] - 1.0
    rpr = 1.0 / (b * case["tau"])
    mod = y[0] ** 2 + y[1] ** 2
    c1, c2 = y[2] - rpr * y[0], y[3] - rpr * y[1]
    grad = torch.zeros_like(mod)
    phase = torch.zeros_like(mod)
    for d in (-1, -2, -3):
        g1, g2 = _diff(y[0], d), _diff(y[1], d)
        grad += g1 * g1 + g2 * g2
        phase += ((y[0] * g2 - y[1] * g1) / mod) ** 2
    pot = 0.25 * lam * (mod - R * R) ** 2 / R ** 4
    rows = [(c1 * c1 + c2 * c2 + grad) / R ** 4 + pot, ((y[0] * y[3] - y[2] * y[1]) / mod / R) ** 2, phase / R ** 2,
            (y[0] * c1 + y[1] * c2) ** 2 / mod / R ** 4, (grad - mod * phase) / R ** 4, pot]
    m = mod.sqrt() / R
    w = torch.ones_like(m) if case["scheme"] == 0 else (1.0 + (m - 1.0) / math.sqrt(2.0)) ** 2 if case["scheme"] == 1 else (m >= 0.8).double()
    sums = [float(x) for r in rows for x in (r.sum(), (r * w).sum())]
    return np.array(sums + [float(w.sum()), float(mod.numel())])


def exact(case, seed):
    kind = case["kind"]
    v = _fields(case, seed)
    if kind == "level":
        return _evolved(case, v.double(), case["steps"])
    if kind == "dropin":
        return _evolved(case, v.double(), 1)
    if kind == "diag":
        out = dict(count=None, weighted=None, corners=None, energy=_energies(case, v.double()), velocity=None)
        return out | (dict(pierced=None) if case["pierced"] else {})
    if kind == "ensemble":
        return [_evolved(case, x.double(), case["steps"]) for x in v]
    if kind == "twolevel":
        return dict(coarse=_evolved(case, v.double(), case["steps"]), fine=None)
    from torch.utils.checkpoint import checkpoint
    x = v.double().requires_grad_()
    lam = torch.tensor(LAMBDA0, dtype=torch.float64, device="cuda", requires_grad=True)
    y = x
    for i in range(case["steps"]):
        y = checkpoint(_rk4, case, y, i * DT, lam, use_reentrant=False)
    R = _radius(case, case["tau"] + case["steps"] * DT)
    mod = y[0] ** 2 + y[1] ** 2
    loss = torch.exp(-mod / (R * R) / 0.1).sum() + (((y[0] * y[3] - y[2] * y[1]) / mod / R) ** 2).mean()
    g = torch.autograd.grad(loss, (x, lam))
    return dict(loss=loss.detach(), state=g[0], lam=g[1])
