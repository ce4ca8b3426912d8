"""The work that programs built on this framework have it do, as measurable cases.

A case is a dict of plain values; ``prepare`` makes what a program holds before
the call (a context with its fields, potential, laser and time step, or a batch),
``run`` makes one pass through the public Python entry points, ``exact`` gives
the same outputs from plain torch in 64 bits, and ``work`` the bytes and
operations that a pass cannot do without.

Kinds of work (``path``):

  block     one output interval of a real-time program: nk Strang steps
            (``Solver.block``).  ``step`` is the sequence's tag: freeprop with a
            potential ("nl"), bragg_ad ("bragg"), the three-level bragg_ad
            ("double_bragg"), the two-species one ("bragg_ds"), the numerical
            three-state step ("raman")
  sobmin    part of a ground-state descent (``Solver.sob_run``)
  observe   what a program prints per output point: particle numbers, <x>, <p>
            and the Rabi populations
  exchange  a program that owns its fields as host arrays: upload, a block,
            download
  sweep     many small bragg runs side by side (``Batch``), fields read at the end

Grids have power-of-two axes (the framework takes no others); raggedness is in
the axis ratios, in axes of 2 to 16 points, and in the number of steps.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from atus2_b200 import (PREC_FP64, PREC_MIXED, STEP_BRAGG_AD, STEP_BRAGG_DS_AD, STEP_DOUBLE_BRAGG_AD, STEP_NL,
                        STEP_NUMERICAL_RAMAN, Batch, Laser, Solver, binfmt)

DT = 1e-3
KIND = {"nl": STEP_NL, "bragg": STEP_BRAGG_AD, "double_bragg": STEP_DOUBLE_BRAGG_AD, "bragg_ds": STEP_BRAGG_DS_AD,
        "raman": STEP_NUMERICAL_RAMAN}
NCOMP = {"nl": 1, "bragg": 2, "double_bragg": 3, "bragg_ds": 4, "raman": 3}
PULSED = ("bragg", "double_bragg", "bragg_ds")
# box length and coarsest spacing per dimension, as the programs' input files have them
BOX = {1: (200.0, 0.05), 2: (128.0, 0.0625), 3: (64.0, 0.25)}
G_NL = {1: 10.0, 2: 1.0, 3: 100.0}
SOB_STEP, SOB_EPS = 4e-4, 1e-10
RABI_K0, RABI_THR = (0.0, 4.0, 8.0, 12.0), 1.5


def _block(name, step, nx, ny=1, nz=1, *, nk, mixed=False):
    return dict(name=name, path="block", step=step, nx=nx, ny=ny, nz=nz, nk=nk, mixed=mixed)


def listed():
    return [
        # a short interferometer run in 1D: the smallest call, all latency
        _block("bragg_1d_512", "bragg", 512, nk=10),
        # the 1D trap run (4096 points on [-100, 100)): the field fits on chip
        _block("rt_1d_4096", "nl", 4096, nk=200),
        # a long 1D axis: expanding clouds need fine spacing over a long box
        _block("rt_1d_1m", "nl", 1 << 20, nk=10),
        # the 2D double slit
        _block("slit_2d_2048", "nl", 2048, 2048, nk=20),
        # three momentum states on an ordinary 2D grid, two outputs' worth of steps
        _block("double_bragg_2d", "double_bragg", 512, 256, nk=20),
        # a 3D test run: small fields, many launches
        _block("bragg_3d_64", "bragg", 64, 64, 64, nk=10),
        # the full-size 3D Bragg pulse, both precisions
        _block("bragg_3d_256", "bragg", 256, 256, 256, nk=10),
        _block("bragg_3d_256_mixed", "bragg", 256, 256, 256, nk=10, mixed=True),
        # ground state at the usual size: one outer chunk of the descent
        dict(name="sobmin_3d_128", path="sobmin", nx=128, ny=128, nz=128, iters=65),
        # observables of an elongated cloud
        dict(name="observe_3d", path="observe", nx=256, ny=128, nz=64, ncomp=2),
        # host arrays in and out around a short block
        dict(name="exchange_2d", path="exchange", step="bragg", nx=512, ny=512, nz=1, nk=20, mixed=False),
        # a parameter sweep over uneven grids
        dict(name="sweep_mixed", path="sweep", count=48, lg_min=10, lg_max=14, n2d=256, nk=100, mixed=True),
    ]


def _split(rng, total, dim, top):
    """Axis exponents of a dim-D grid of 2**total points, each between 1 and top."""
    while True:
        e = [rng.randint(1, top) for _ in range(dim - 1)]
        last = total - sum(e)
        if 1 <= last <= top:
            e.append(last)
            rng.shuffle(e)
            return [1 << k for k in e] + [1] * (3 - dim)


def draw(rng):
    path = rng.choice(["block"] * 8 + ["sobmin", "observe", "exchange", "sweep"])
    if path == "sweep":
        return dict(path=path, count=rng.randint(3, 48), lg_min=rng.randint(10, 12), lg_max=rng.randint(12, 14),
                    n2d=rng.choice([64, 128, 256]), nk=rng.randint(10, 100), mixed=rng.random() < 0.7)
    if path == "sobmin":
        n = _split(rng, rng.randint(12, 21), 3, 8)
        return dict(path=path, nx=n[0], ny=n[1], nz=n[2], iters=rng.randint(2, 65))
    if path == "observe":
        dim = rng.randint(1, 3)
        n = _split(rng, rng.randint(6, 22) if dim > 1 else rng.randint(6, 20), dim, 20 if dim == 1 else 11)
        return dict(path=path, nx=n[0], ny=n[1], nz=n[2], ncomp=rng.randint(1, 4))
    dim = rng.randint(1, 3)
    step = rng.choice(["nl", "nl", "bragg", "bragg", "double_bragg", "bragg_ds", "raman"])
    mixed = rng.random() < 0.35
    if path == "exchange":
        step, mixed = "bragg", False
    top = {1: 20, 2: 12, 3: 9}[dim]
    most = {"raman": 19, "bragg_ds": 20, "double_bragg": 21}.get(step, 23)
    total = rng.randint(3, min(most, {1: 20, 2: 22, 3: 23}[dim]))
    if path == "exchange":
        total = min(total, 20)
    n = _split(rng, total, dim, top)
    # a pass costs at most about what the largest listed one does
    nk = int(math.exp(rng.uniform(0.0, math.log(100.0))))
    cap = (256**3 * 2 * 10) // ((1 << total) * NCOMP[step] * (16 if step == "raman" else 2))
    return dict(path=path, step=step, nx=n[0], ny=n[1], nz=n[2], nk=max(1, min(nk, cap)), mixed=mixed)


# ------------------------------------------------------------------ inputs
def _shape(case):
    n = [case["nx"], case["ny"], case["nz"]]
    dim = 3 if n[2] > 1 else 2 if n[1] > 1 else 1
    return tuple(n[:dim])


def _header(shape, lengths):
    return binfmt.make_header(len(shape), list(shape), [-0.5 * L for L in lengths], [0.5 * L for L in lengths], dt=DT)


def _lengths(shape):
    most, coarse = BOX[len(shape)]
    return [min(most, n * coarse) for n in shape]


def _axes(h, shape, coords):
    """Per-axis coordinates as broadcastable FP64 CUDA tensors."""
    out = []
    for a in range(len(shape)):
        v = torch.from_numpy(coords(h, a)).cuda()
        out.append(v.reshape([-1 if b == a else 1 for b in range(len(shape))]))
    return out


def _fields(h, shape, ncomp, rnd):
    """Normalised packets: a cloud of random width and position with a momentum
    along x and 1e-6 noise; further states are weaker copies, kicked."""
    X = _axes(h, shape, binfmt.x_coords)
    lengths = [float(h["d" + ax]) * n for ax, n in zip("xyz", shape)]
    gen = torch.Generator(device="cuda").manual_seed(rnd.randrange(1 << 30))
    width = [L / 16 * rnd.uniform(0.8, 1.3) for L in lengths]
    centre = [L / 16 * rnd.uniform(-1.0, 1.0) for L in lengths]
    k = rnd.uniform(1.5, 2.5)
    base = torch.ones(shape, dtype=torch.float64, device="cuda")
    for x, w, c in zip(X, width, centre):
        base = base * torch.exp(-0.5 * ((x - c) / w) ** 2)
    psi = []
    for c in range(ncomp):
        p = base * (1.0, 0.5, 0.3, 0.2)[c] * torch.exp(1j * ((k + 0.5 * c) * X[0]))
        p = p + 1e-6 * torch.randn(shape, dtype=torch.complex128, device="cuda", generator=gen)
        psi.append(p)
    vol = float(np.prod([float(h["d" + ax]) for ax in "xyz"[: len(shape)]]))
    norm = math.sqrt(vol * sum(float(p.abs().square().sum()) for p in psi))
    return [p / norm for p in psi]


def _potential(h, shape, rnd):
    """The programs' potentials: a trap in 1D and 3D, the double slit in 2D."""
    X = _axes(h, shape, binfmt.x_coords)
    w = rnd.uniform(0.8, 1.2)
    if len(shape) == 2:
        x, y = X
        wall = (x.abs() < 0.5) & ~(((y - 4).abs() < w) | ((y + 4).abs() < w))
        return torch.where(wall, 200.0, 0.0).to(torch.float64)
    V = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for x in X:
        V = V + 0.5 * (w * x) * (w * x)
    return V


def _matrix(ncomp, rnd):
    """Interaction strengths of hyperfine states: nearly equal, symmetric."""
    g = np.zeros((ncomp, ncomp))
    for i in range(ncomp):
        for j in range(i + 1):
            g[i, j] = g[j, i] = 100.0 * (1.0 - 0.05 * rnd.random())
    return g


class _Device:
    """A context's field as the CUDA array it is; the tensor made from it keeps
    the context, which owns the memory, alive."""

    def __init__(self, solver, c):
        self.solver = solver
        self.__cuda_array_interface__ = {"data": (solver.device_ptr(c), False), "shape": tuple(solver.shape) + (2,),
                                         "typestr": "<f4" if solver.precision == PREC_MIXED else "<f8", "version": 2}


def _view(s, c):
    raw = torch.as_tensor(_Device(s, c), device="cuda")
    return torch.view_as_complex(raw)


def _envelope(t0, nk):
    """AMP_T of the nk potential steps of a block: a train of Gaussian pulses."""
    t = t0 + DT * (np.arange(nk) + 1.0)
    return np.exp(-((t % 2.0 - 1.0) ** 2) / (2 * 0.5**2))


def _laser(step, rnd):
    kw = dict(Amp=[4.0 * rnd.uniform(0.8, 1.2), 3.0], laser_k=[8.0, 0.0], laser_domh=[rnd.uniform(12.0, 16.0), 0.0])
    if step == "bragg_ds":
        kw["DeltaL"] = [0.0, 0.5, 0.0, 0.25]
    return kw


def _problem(case, seed):
    """Everything that defines a case's inputs, made from the seed alone."""
    import random

    rnd = random.Random(seed)
    shape = _shape(case)
    step = case.get("step", "bragg")
    ncomp = case.get("ncomp", NCOMP[step])
    p = dict(shape=shape, step=step, ncomp=ncomp, header=_header(shape, _lengths(shape)))
    p["psi"] = _fields(p["header"], shape, ncomp, rnd)
    p["V"] = _potential(p["header"], shape, rnd) if step == "nl" else None
    p["gs"] = np.array([[G_NL[len(shape)] * rnd.uniform(0.9, 1.1)]]) if step == "nl" else _matrix(ncomp, rnd)
    p["laser"], p["laser2"] = _laser(step, rnd), _laser(step, rnd)
    return p


def _trap(case, seed):
    """A ground-state problem: anisotropic trap, Thomas-Fermi start."""
    import random

    rnd = random.Random(seed)
    shape = _shape(case)
    lengths = [min(32.0, 0.25 * n) for n in shape]
    h = _header(shape, lengths)
    X = _axes(h, shape, binfmt.x_coords)
    om = [1.0, rnd.uniform(0.5, 4.0), rnd.uniform(0.5, 4.0)]
    g = 10.0 ** rnd.uniform(1.0, 3.3)
    V = sum(0.5 * (w * x) ** 2 for w, x in zip(om, X)).expand(shape).contiguous()
    mu = 0.5 * (15.0 * g * om[1] * om[2] / (4 * math.pi)) ** 0.4 + 0.5 * sum(om)
    psi = torch.sqrt(torch.clamp(mu - V, min=0.0) / g) + 1e-3 * torch.exp(-V)
    return dict(shape=shape, header=h, V=V, g=g, psi=psi.to(torch.complex128))


def _instances(case, seed):
    """Instances of a sweep: grids in a fixed round, parameters from the seed."""
    import random

    rnd = random.Random(seed)
    grids = [(1, 1 << k) for k in range(case["lg_min"], case["lg_max"] + 1)] + [(2, case["n2d"])]
    out = []
    for i in range(case["count"]):
        dim, n = grids[i % len(grids)]
        L = 128.0 if dim == 1 else 32.0
        h = _header((n,) * dim, [L] * dim)
        om, delta, g, T = rnd.uniform(2, 20), rnd.uniform(-4, 4), rnd.uniform(0, 200), rnd.uniform(0.5, 3)
        kw = dict(Amp=[om / 2, om / 2], laser_k=[8.0, 0], laser_domh=[delta, 0])
        out.append(dict(header=h, alpha=0.5, gs=[g] * 4, kw=kw, laser=Laser.make(**kw), pulse=(T / 2, T / 6),
                        bragg_stable=True, width=rnd.uniform(0.8, 1.2), shape=(n,) * dim))
    return out


def _sweep_field(d):
    xs = np.meshgrid(*[binfmt.x_coords(d["header"], a) for a in range(len(d["shape"]))], indexing="ij")
    p = np.exp(-0.5 * sum(x * x for x in xs) / d["width"] ** 2).astype(np.complex128)
    vol = float(np.prod([d["header"]["d" + ax] for ax in "xyz"[: len(d["shape"])]]))
    return p / np.sqrt(vol * np.sum(np.abs(p) ** 2))


_STREAM = None


def _solver(header, ncomp, mixed):
    """A context on the program's own CUDA stream."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    s = Solver(header, ncomp, PREC_MIXED if mixed else PREC_FP64)
    s.set_stream(_STREAM.cuda_stream)
    return s


def _context(p, mixed):
    s = _solver(p["header"], p["ncomp"], mixed)
    dim = len(p["shape"])
    for c in range(p["ncomp"]):
        s.set_alpha(c, [0.5] * dim)
    s.set_gs(p["gs"])
    if p["V"] is not None:
        s.set_potential(0, p["V"].cpu().numpy())
    s.set_laser(Laser.make(**p["laser"]))
    if p["step"] == "bragg_ds":
        s.set_species2(Laser.make(**p["laser2"]))
    s.set_dt(DT)
    return s


def prepare(case, seed):
    path = case["path"]
    if path == "sweep":
        insts = _instances(case, seed)
        b = Batch(insts, PREC_MIXED if case["mixed"] else PREC_FP64, DT)
        for i, d in enumerate(insts):
            f = _sweep_field(d)
            b.set_psi(i, 0, f)
            b.set_psi(i, 1, np.zeros_like(f))
        b.tune(10)
        return dict(case=case, batch=b)
    if path == "sobmin":
        p = _trap(case, seed)
        s = _solver(p["header"], 1, False)
        s.set_gs([p["g"]])
        s.set_potential(0, p["V"].cpu().numpy())
        _view(s, 0).copy_(p["psi"])
        s.sob_init([0.5], SOB_STEP)
        torch.cuda.synchronize()
        return dict(case=case, solver=s, out=_view(s, 0))
    p = _problem(case, seed)
    s = _context(p, case.get("mixed", False))
    st = dict(case=case, solver=s)
    if path == "exchange":
        st["host"] = [f.cpu().numpy() for f in p["psi"]]
        return st
    st["out"] = [_view(s, c) for c in range(p["ncomp"])]
    for v, f in zip(st["out"], p["psi"]):
        v.copy_(f)
    torch.cuda.synchronize()
    return st


# ------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    path = case["path"]
    if path == "sweep":
        b = state["batch"]
        b.run(case["nk"])
        # complex64 fields come back as complex64, complex128 ones as they are
        kind = np.complex64 if case["mixed"] else np.complex128
        return np.concatenate([b.psi(i, c).ravel() for i in range(b.count) for c in range(2)]).astype(kind, copy=False)
    s = state["solver"]
    if path == "sobmin":
        iters, res = s.sob_run(SOB_EPS, case["iters"])
        return dict(iters=iters, res=res, psi=state["out"])
    if path == "observe":
        dim = s.dim
        k0 = [[k] + [0.0] * (dim - 1) for k in RABI_K0]
        return dict(n=[s.particle_number(c) for c in range(s.ncomp)],
                    x=[s.expval_position(c) for c in range(s.ncomp)],
                    p=[s.expval_momentum(c) for c in range(s.ncomp)], rabi=s.rabi_integrals(k0, RABI_THR))
    if path == "exchange":
        for c, f in enumerate(state["host"]):
            s.set_psi(c, f)
    F = _envelope(s.t, case["nk"]) if case["step"] in PULSED else None
    s.block(case["nk"], KIND[case["step"]], F=F)
    if path == "exchange":
        return [s.psi(c) for c in range(s.ncomp)]
    return state["out"]


# ------------------------------------------------------------------ bytes and operations
def work(case):
    path = case["path"]
    if path == "sweep":
        flops = pts = 0.0
        for d in _grids(case):
            n = float(np.prod(d))
            pts += n
            flops += n * 2 * (10.0 * math.log2(n) + 60.0)
        return {"bytes": 2.0 * 2 * pts * (8 if case["mixed"] else 16), "flops": flops * case["nk"]}
    n = float(np.prod(_shape(case)))
    fft = 5.0 * math.log2(n)
    if path == "sobmin":
        return {"bytes": n * (16 + 8 + 16), "flops": n * case["iters"] * (4 * fft + 40.0)}
    if path == "observe":
        return {"bytes": n * 16 * case["ncomp"], "flops": n * case["ncomp"] * (fft + 15.0)}
    nc = NCOMP[case["step"]]
    point = {"nl": 25.0, "bragg": 60.0, "double_bragg": 80.0, "bragg_ds": 60.0, "raman": 300.0}[case["step"]]
    size = 8 if case["mixed"] else 16
    return {"bytes": n * (2 * nc * size + (8 if case["step"] == "nl" else 0)),
            "flops": n * nc * case["nk"] * (2 * fft + 20.0 + point)}


def _grids(case):
    grids = [(1 << k,) for k in range(case["lg_min"], case["lg_max"] + 1)] + [(case["n2d"],) * 2]
    return [grids[i % len(grids)] for i in range(case["count"])]


# ------------------------------------------------------------------ the same in plain torch
def _kinetic(h, shape, dt):
    K = _axes(h, shape, binfmt.k_coords)
    return torch.exp(-1j * dt * 0.5 * sum(k * k for k in K))


def _two_level(a, b, V11, V22, W):
    """exp(-i dt [[V11, W], [W, V22]]) on (a, b), W real."""
    m, d = 0.5 * (V11 + V22), 0.5 * (V11 - V22)
    r = torch.sqrt(d * d + W * W)
    sinc = DT * torch.sinc(DT * r / math.pi)
    cos, e = torch.cos(DT * r), torch.exp(-1j * DT * m)
    return e * ((cos - 1j * sinc * d) * a - 1j * sinc * W * b), e * ((cos + 1j * sinc * d) * b - 1j * sinc * W * a)


def _potential_step(step, psi, V, gs, L, L2, x, t1, F):
    rho = [p.real**2 + p.imag**2 for p in psi]
    phi = [sum(float(gs[i][j]) * rho[j] for j in range(len(psi))) for i in range(len(psi))]

    def cosine(kw, sign=1.0):
        return F * kw["Amp"][0] * torch.cos(sign * kw["laser_k"][0] * x - kw["laser_domh"][0] * t1)

    if step == "nl":
        return [psi[0] * torch.exp(-1j * DT * (V + phi[0]))]
    if step == "bragg":
        return list(_two_level(psi[0], psi[1], phi[0], phi[1], cosine(L)))
    if step == "bragg_ds":
        phi = [p - d for p, d in zip(phi, L["DeltaL"])]
        return [*_two_level(psi[0], psi[1], phi[0], phi[1], cosine(L)),
                *_two_level(psi[2], psi[3], phi[2], phi[3], cosine(L2))]
    if step == "double_bragg":
        # states 2 and 3 share V22: one combination of them couples to state 1,
        # the orthogonal one only takes its phase
        Wp, Wm = cosine(L), cosine(L, -1.0)
        W = torch.sqrt(Wp * Wp + Wm * Wm)
        up, um = torch.where(W > 0, Wp / W, 1.0), torch.where(W > 0, Wm / W, 0.0)
        bright, dark = up * psi[1] + um * psi[2], um * psi[1] - up * psi[2]
        a, bright = _two_level(psi[0], bright, phi[0], phi[1], W)
        dark = dark * torch.exp(-1j * DT * phi[1])
        return [a, up * bright + um * dark, um * bright - up * dark]
    # raman: three-state Hermitian exponential
    A = torch.zeros(psi[0].shape + (3, 3), dtype=torch.complex128, device="cuda")
    for i in range(3):
        A[..., i, i] = phi[i] + (L["laser_domh"][0] if i == 2 else 0.0)
    e = torch.exp(1j * L["laser_k"][0] * x)
    A[..., 0, 2], A[..., 1, 2] = 0.5 * L["Amp"][0] * e, 0.5 * L["Amp"][1] * e.conj()
    A[..., 2, 0], A[..., 2, 1] = A[..., 0, 2].conj(), A[..., 1, 2].conj()
    out = torch.matrix_exp(-1j * DT * A) @ torch.stack(psi, -1)[..., None]
    return [out[..., i, 0] for i in range(3)]


def _strang(psi, h, shape, nk, potential):
    """half, (V, full)^(nk-1), V, half; potential(psi, t1, j) is one V step."""
    half, full = _kinetic(h, shape, 0.5 * DT), _kinetic(h, shape, DT)
    psi = [torch.fft.ifftn(torch.fft.fftn(p) * half) for p in psi]
    for j in range(nk):
        psi = potential(psi, DT * (j + 1.0), j)
        factor = half if j == nk - 1 else full
        psi = [torch.fft.ifftn(torch.fft.fftn(p) * factor) for p in psi]
    return psi


def _sob_exact(case, seed):
    p = _trap(case, seed)
    h, shape, V, g = p["header"], p["shape"], p["V"], p["g"]
    ar = float(np.prod([float(h["d" + ax]) for ax in "xyz"[: len(shape)]]))
    k2 = sum(k * k for k in _axes(h, shape, binfmt.k_coords)) * 0.5
    S = 1.0 / (1.0 + k2)
    dot = lambda a, b: float((a.real * b.real + a.imag * b.imag).sum())  # noqa: E731
    psi = p["psi"] / math.sqrt(ar * dot(p["psi"], p["psi"]))
    res = math.inf
    iters = 0
    while res > SOB_EPS and iters < case["iters"]:
        f = torch.fft.fftn(psi)
        lap = torch.fft.ifftn(f * -k2)
        spsi = torch.fft.ifftn(f * S)
        grad = torch.fft.ifftn(torch.fft.fftn(-lap + (V + g * psi.abs().square()) * psi) * S)
        grad = grad - (dot(psi, grad) / dot(psi, spsi)) * spsi
        res = ar * dot(grad, grad)
        N = ar * dot(psi, psi)
        if abs(N - 1.0) > 1e-5:
            psi = psi / math.sqrt(N)
        psi = psi - SOB_STEP * grad
        iters += 1
    return dict(iters=None, res=res, psi=psi)


def _observe_exact(case, seed):
    p = _problem(case, seed)
    h, shape = p["header"], p["shape"]
    dim = len(shape)
    X, K = _axes(h, shape, binfmt.x_coords), _axes(h, shape, binfmt.k_coords)
    ar = float(np.prod([float(h["d" + ax]) for ax in "xyz"[:dim]]))
    ark = float(np.prod([float(h["dk" + ax]) for ax in "xyz"[:dim]]))
    out = dict(n=[], x=[], p=[])
    for c, f in enumerate(p["psi"]):
        rho = f.abs().square()
        hat = torch.fft.fftn(f).abs().square() * (ar / (2 * math.pi) ** (dim / 2)) ** 2
        out["n"].append(ar * float(rho.sum()))
        out["x"].append(np.array([ar * float((x * rho).sum()) for x in X]))
        out["p"].append(np.array([ark * float((k * hat).sum()) for k in K]))
        if c == 0:
            # a point inside a ball does not advance the bin of the balls after it
            bins = torch.zeros(shape, dtype=torch.int64, device="cuda")
            sums = [0.0] * len(RABI_K0)
            for k0 in RABI_K0:
                r2 = (K[0] - k0) ** 2
                for k in K[1:]:
                    r2 = r2 + k * k
                inside = (torch.sqrt(r2) < RABI_THR).expand(shape)
                for j in range(len(sums)):
                    sums[j] += ark * float(hat[inside & (bins == j)].sum())
                bins = torch.where(inside, bins, bins + 1)
            out["rabi"] = np.array(sums)
    return out


def exact(case, seed):
    path = case["path"]
    if path == "sobmin":
        return _sob_exact(case, seed)
    if path == "observe":
        return _observe_exact(case, seed)
    if path == "sweep":
        got = []
        for d in _instances(case, seed):
            tc, sigma = d["pulse"]
            x = _axes(d["header"], d["shape"], binfmt.x_coords)[0]
            a = torch.from_numpy(_sweep_field(d)).cuda()
            gs = np.array(d["gs"]).reshape(2, 2)

            def step(psi, t1, j, d=d, x=x, gs=gs, tc=tc, sigma=sigma):
                F = math.exp(-((t1 - tc) ** 2) / (2 * sigma * sigma))
                return _potential_step("bragg", psi, None, gs, d["kw"], None, x, t1, F)

            psi = _strang([a, torch.zeros_like(a)], d["header"], d["shape"], case["nk"], step)
            got += [f.reshape(-1) for f in psi]
        return torch.cat(got)
    p = _problem(case, seed)
    x = _axes(p["header"], p["shape"], binfmt.x_coords)[0]
    F = _envelope(0.0, case["nk"]) if p["step"] in PULSED else np.ones(case["nk"])

    def step(psi, t1, j):
        return _potential_step(p["step"], psi, p["V"], p["gs"], p["laser"], p["laser2"], x, t1, float(F[j]))

    return _strang(p["psi"], p["header"], p["shape"], case["nk"], step)
