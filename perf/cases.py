"""The work that users of picpp_gb300 have it do, one case per kind of run.

A case is a dict of plain values.  "kind" names the entry points it goes
through:

  explicit   buneman_step: the whole Buneman/Tristan Yee step, then the field
             dump of a diagnostics interval
  implicit   implicit_step: moments, field solve, mover, then the field dump
             (and the particles, in the order of their numbers, where the run
             keeps trajectories)
  shock      implicit_step of a reflecting-wall box that is fed through the
             open boundary with append_particles before every step
  solve      maxwell_solve of a given system in host memory
  gradient   nn_loss_grad: forward and backward pass of the learned
             preconditioner's network
  moments    updateDensityParameters and updateEnergy, with their download

Dumps go to pinned host memory through the C ABI and are kept in the
precision of the run's particles: a run with FP32 particles and fields
writes its fields in single precision.
"""
import ctypes
import math

import numpy as np
import torch

import picpp_gb300 as P
from picpp_gb300 import initstate as I

FOUR_PI = 4.0 * math.pi


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # electron-positron Weibel pairs on a plane, FP64 throughout, reference
        # GMRES, trajectories kept: the smallest stated run, bound by launches
        dict(name="weibel_32x32x1_f64", kind="implicit", setup="pairs", nx=32, ny=32, nz=1, ppc=32, steps=5,
             f64=True, compat=0, solver="reference", particles=True),
        # the class's default pressure placement (the reference's own), FP64, on
        # a box of ragged extents: what a parity run against the reference does
        dict(name="parity_26x20x18_f64", kind="implicit", setup="beams", nx=26, ny=20, nz=18, ppc=16, steps=2,
             f64=True, compat=1, solver="reference", particles=True),
        # explicit electron-proton plasma, FP32, a small box in steps of a short
        # diagnostics interval: launch latency and a part-filled GPU
        dict(name="explicit_32_f32", kind="explicit", nx=32, ny=32, nz=32, ppc=16, steps=20, f64=False, smooth=0),
        # the headline explicit workload: 128^3, 16 particles per cell and
        # species, sorted every 5 steps
        dict(name="explicit_128_f32", kind="explicit", nx=128, ny=128, nz=128, ppc=16, steps=5, f64=False, smooth=0),
        # the all-FP64 explicit run that the FP32 one is compared with
        dict(name="explicit_64_f64", kind="explicit", nx=64, ny=64, nz=64, ppc=16, steps=5, f64=True, smooth=0),
        # a box whose extents no power-of-two tile divides well, with the
        # current smoothed twice a step
        dict(name="explicit_100x60x54_f32_smooth", kind="explicit", nx=100, ny=60, nz=54, ppc=9, steps=5, f64=False,
             smooth=2),
        # relativistic counter-streaming beams, FP32 push and FP64 GMRES(30), the
        # box size that the solver's training data are recorded on
        dict(name="beams_64x64x16_f32", kind="implicit", setup="beams", nx=64, ny=64, nz=16, ppc=64, steps=2,
             f64=False, compat=0, solver="restarted", particles=False),
        # the headline implicit workload: 537 million particles, the
        # mixed-precision field solve
        dict(name="beams_256x256x64_f32_mixed", kind="implicit", setup="beams", nx=256, ny=256, nz=64, ppc=64,
             steps=1, f64=False, compat=0, solver="mixed", particles=False),
        # reflecting-wall shock: three species, injection every step
        dict(name="shock_512x64x4_f32", kind="shock", nx=512, ny=64, nz=4, steps=1),
        # a field solve alone, FP64 GMRES(30) on host arrays
        dict(name="solve_128x128x32_f64", kind="solve", nx=128, ny=128, nz=32, solver="restarted"),
        # one gradient of the network's loss: its forward and backward pass
        dict(name="gradient_4x16x64x64", kind="gradient", batch=4, nx=64, ny=64, nz=16),
        # the density, energy and bulk-velocity moments of a diagnostics step
        dict(name="moments_64_f32", kind="moments", nx=64, ny=64, nz=64, ppc=16, f64=False),
    ]


def _between(rng, lo, hi):
    """A whole number of [lo, hi], even over the logarithm, odd ones among them."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _fit(n, ppc, most):
    """ppc, lowered until two species on n cells hold no more than `most` particles."""
    return max(1, min(ppc, int(most // (2 * n))))


def draw(rng):
    kind = rng.choice(["explicit", "explicit", "explicit64", "pairs", "parity", "beams", "beams", "shock", "solve",
                       "gradient", "moments"])
    if kind in ("explicit", "explicit64"):
        f64 = kind == "explicit64"
        hi = 64 if f64 else 128
        nx, ny, nz = (_between(rng, 16, hi) for _ in range(3))
        ppc = _fit(nx * ny * nz, _between(rng, 4, 32), 8e6 if f64 else 6e7)
        return dict(kind="explicit", nx=nx, ny=ny, nz=nz, ppc=ppc, steps=5, f64=f64, smooth=rng.choice([0, 0, 1, 2]))
    if kind == "pairs":
        return dict(kind="implicit", setup="pairs", nx=_between(rng, 16, 96), ny=_between(rng, 16, 96), nz=1,
                    ppc=_between(rng, 8, 64), steps=rng.choice([2, 3, 5]), f64=True, compat=0, solver="reference",
                    particles=True)
    if kind == "parity":
        nx, ny, nz = (_between(rng, 8, 32) for _ in range(3))
        return dict(kind="implicit", setup="beams", nx=nx, ny=ny, nz=nz, ppc=_between(rng, 2, 16),
                    steps=rng.choice([1, 2]), f64=True, compat=1, solver="reference", particles=True)
    if kind == "beams":
        nx, ny, nz = _between(rng, 16, 128), _between(rng, 16, 128), _between(rng, 8, 64)
        return dict(kind="implicit", setup="beams", nx=nx, ny=ny, nz=nz, ppc=_fit(nx * ny * nz, _between(rng, 8, 64), 3e7),
                    steps=rng.choice([1, 2]), f64=False, compat=0, solver=rng.choice(["restarted", "mixed"]),
                    particles=False)
    if kind == "shock":
        return dict(kind="shock", nx=_between(rng, 48, 512), ny=_between(rng, 8, 64), nz=_between(rng, 4, 8), steps=1)
    if kind == "solve":
        return dict(kind="solve", nx=_between(rng, 16, 128), ny=_between(rng, 16, 128), nz=_between(rng, 8, 48),
                    solver=rng.choice(["restarted", "reference"]))
    if kind == "gradient":
        return dict(kind="gradient", batch=_between(rng, 1, 4), nx=4 * _between(rng, 4, 16), ny=4 * _between(rng, 4, 16),
                    nz=4 * _between(rng, 2, 4))
    nx, ny, nz = (_between(rng, 16, 96) for _ in range(3))
    return dict(kind="moments", nx=nx, ny=ny, nz=nz, ppc=_fit(nx * ny * nz, _between(rng, 4, 32), 1.6e7), f64=False)


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed, k):
    g = torch.Generator(device=_device())
    g.manual_seed((int(seed) * 1009 + k) & 0x7FFFFFFF)
    return g


def _rand(n, g):
    """Uniform values of [0, 1) that single precision holds, in double."""
    return torch.rand(n, generator=g, device=g.device, dtype=torch.float32).double()


def _juttner(n, theta, mass, gamma, sign, g):
    """Maxwell-Juttner momenta of temperature theta, boosted along x by the
    flipping method; values that single precision holds."""
    umax = math.sqrt((1.0 + 40.0 * theta) ** 2 - 1.0)
    u = torch.linspace(0.0, umax, 20001, dtype=torch.float64, device=g.device)
    pdf = u * u * torch.exp(-(torch.sqrt(1.0 + u * u) - 1.0) / theta)
    cdf = torch.cat([torch.zeros(1, dtype=torch.float64, device=g.device), torch.cumsum(0.5 * (pdf[1:] + pdf[:-1]), 0)])
    cdf = cdf / cdf[-1].clone()
    r = _rand(n, g)
    at = torch.clamp(torch.searchsorted(cdf, r, right=True), 1, 20000)
    s = u[at - 1] + (u[at] - u[at - 1]) * (r - cdf[at - 1]) / torch.clamp(cdf[at] - cdf[at - 1], min=1e-300)
    cos_t, phi = 2.0 * _rand(n, g) - 1.0, 2.0 * math.pi * _rand(n, g)
    sin_t = torch.sqrt(torch.clamp(1.0 - cos_t * cos_t, min=0.0))
    px, py, pz = s * cos_t, s * sin_t * torch.cos(phi), s * sin_t * torch.sin(phi)
    if gamma > 1.0:
        beta = math.sqrt(1.0 - 1.0 / (gamma * gamma))
        lor = torch.sqrt(1.0 + px * px + py * py + pz * pz)
        px = torch.where(-beta * sign * px / lor > _rand(n, g), -px, px)
        px = gamma * (px + sign * beta * lor)
    return tuple((p * mass).float().double() for p in (px, py, pz))


def _species(cells, ppc, q, m, w, theta, gamma, sign, g):
    """ppc particles in every cell of `cells`, offsets uniform in the cell."""
    n = cells.numel() * ppc
    cell = cells.repeat_interleave(ppc)
    off = [_rand(n, g) for _ in range(3)]
    if sign == 0:   # half each way
        sign = 1.0 - 2.0 * (torch.arange(n, device=g.device) % 2).double()
    p = _juttner(n, theta, m, gamma, sign, g)
    return dict(q=q, m=m, w=w, cell=cell, ox=off[0], oy=off[1], oz=off[2], px=p[0], py=p[1], pz=p[2])


def _plasma(case, seed):
    """(box, species on the device, uniform B0) of a periodic case."""
    nx, ny, nz, ppc = case["nx"], case["ny"], case["nz"], case["ppc"]
    n_e = 1.0 / FOUR_PI
    setup = case.get("setup", "protons")
    if setup == "protons":   # electrons and protons of mass 100, magnetised along x
        box = I.Box(nx, ny, nz, 0.1, 0.1, 0.1, 0.045)
        kinds = [(-1.0, 1.0, 0.1, 1.0, 1.0), (1.0, 100.0, 1e-3, 1.0, 1.0)]
        B0 = (math.sqrt(FOUR_PI * 0.1 * n_e * 101.0), 0.0, 0.0)
    elif setup == "pairs":   # electron-positron pairs drifting at +-0.5 c
        box = I.Box(nx, ny, nz, 0.2, 0.2, 0.2, 0.1, theta=0.5)
        gam = 1.0 / math.sqrt(0.75)
        kinds = [(-1.0, 1.0, 0.01, gam, 0), (1.0, 1.0, 0.01, gam, 0)]
        B0 = (0.0, 0.0, 0.0)
    else:                    # electron-ion beams of Lorentz factor 10 along +-x
        box = I.Box(nx, ny, nz, 0.5, 0.5, 0.5, 0.5, theta=0.5)
        kinds = [(-1.0, 1.0, 0.01, 10.0, 0), (1.0, 25.0, 0.01 / 25.0, 10.0, 0)]
        B0 = (0.0, 0.0, math.sqrt(FOUR_PI * 0.01 * n_e * 26.0 * 10.0))
    w = I.density_weight(box, n_e, ppc)
    if _filled(case):
        return box, [dict(q=q, m=m, w=w, theta=th, gamma=gam) for q, m, th, gam, _ in kinds], B0
    cells = torch.arange(box.ncells, dtype=torch.int32, device=_device())
    return box, [_species(cells, ppc, q, m, w, th, gam, sign, _generator(seed, s))
                 for s, (q, m, th, gam, sign) in enumerate(kinds)], B0


def _filled(case):
    """Boxes too large to build on the host are filled by the library."""
    return 2 * case["nx"] * case["ny"] * case["nz"] * case["ppc"] > 1e8


def _pinned(t):
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    p.copy_(t)
    return p


def _upload(sim, s, sp):
    host = {k: _pinned(sp[k]).numpy() for k in ("cell", "ox", "oy", "oz", "px", "py", "pz")}
    sim.upload_particles(s, host)


def _uniform(box, B0):
    E, B = np.zeros((3, box.nz, box.ny, box.nx)), np.zeros((3, box.nz, box.ny, box.nx))
    for d in range(3):
        B[d] = B0[d]
    return E, B


def _opts(name):
    return {"reference": P.solve_opts(P.GMRES_REFERENCE, max_iter=50, tol=1e-8),
            "restarted": P.solve_opts(P.GMRES_RESTARTED, restart=30, max_iter=600, tol=1e-8),
            "mixed": P.solve_opts(P.FGMRES_MIXED, restart=30, max_iter=600, tol=1e-8, inner=12)}[name]


class _Dump:
    """The dump of a run: pinned buffers that a diagnostics interval fills."""

    def __init__(self, box, f64, counts=()):
        pin = torch.cuda.is_available()
        self.box, self.f64 = box, f64
        self.field = [torch.empty((3, box.nz, box.ny, box.nx), dtype=torch.float64, pin_memory=pin) for _ in range(3)]
        self.parts = [[torch.empty(n, dtype=torch.float64, pin_memory=pin) for _ in range(6)] +
                      [torch.empty(n, dtype=torch.int32, pin_memory=pin) for _ in range(2)] for n in counts]

    def fields(self, sim):
        at = [ctypes.cast(f.data_ptr(), ctypes.POINTER(ctypes.c_double)) for f in self.field]
        sim._ck(sim.L.pic_download_fields(sim.ctx, *at))
        return [f.clone() if self.f64 else f.to(torch.float32) for f in self.field]

    def particles(self, sim):
        """Momenta and positions of every species, in the order of the particles' numbers."""
        got, n, b = [], ctypes.c_long(), self.box
        for s, a in enumerate(self.parts):
            at = [ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double)) for t in a[:6]]
            whole = [ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_int)) for t in a[6:]]
            sim._ck(sim.L.pic_download_particles(sim.ctx, s, ctypes.byref(n), whole[0], *at, whole[1]))
            cell, ids = a[6].long(), a[7].long()
            pos = [(cell % b.nx + a[0]) * b.dx, (cell // b.nx % b.ny + a[1]) * b.dy, (cell // (b.nx * b.ny) + a[2]) * b.dz]
            out = torch.empty((6, n.value), dtype=torch.float64)
            out[:, ids] = torch.stack(pos + a[3:6])
            got.append(out)
        return got


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return _prepare_solve(case, seed)
    if kind == "gradient":
        return _prepare_gradient(case, seed)
    if kind == "shock":
        return _prepare_shock(case, seed)
    box, species, B0 = _plasma(case, seed)
    real = P.F64 if case["f64"] else P.F32
    if kind == "implicit":
        sim = P.GpuSimulation(box, P.IMPLICIT, particle_real=real, pressure_compat=case["compat"], sort_every=1,
                              tile=(0, 0, 0))
    else:
        sim = P.GpuSimulation(box, P.BUNEMAN, particle_real=real, sort_every=5, tile=(0, 0, 0),
                              smoothing_count=case.get("smooth", 0))
    n = box.ncells * case["ppc"]
    for s, sp in enumerate(species):
        sim.add_species(sp["q"], sp["m"], sp["w"], n)
        if _filled(case):
            sim.fill_species(s, case["ppc"], 2 * seed + s, sp["theta"], sp["gamma"], True)
        else:
            _upload(sim, s, sp)
    sim.upload_fields(*_uniform(box, B0))
    state = dict(case=case, sim=sim)
    if kind == "moments":
        sim.buneman_step(1)
        return state
    state["dump"] = _Dump(box, case["f64"], [n, n] if case.get("particles") else ())
    if kind == "implicit":
        state["opts"] = _opts(case["solver"])
    return state


def _prepare_shock(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    specs, E0, B0, v0 = I.shock_parameters(0.5)
    box = I.Box(nx, ny, nz, 0.5, 0.5, 0.5, 0.4, theta=0.5)
    sim = P.GpuSimulation(box, P.IMPLICIT, particle_real=P.F32, pressure_compat=0, sort_every=1, tile=(0, 0, 0),
                          boundary_x=P.BOUNDARY_WALL_OPEN, e_right=tuple(E0), b_right=tuple(B0))
    cells = torch.arange(box.ncells, dtype=torch.int32, device=_device())
    cells = cells[cells % nx < nx - 2]
    for s, (q, m, n, ppc, th) in enumerate(specs):
        w = I.density_weight(box, n, ppc)
        sim.add_species(q, m, w, 2 * ppc * cells.numel() + 12000 * ny * nz)
        _upload(sim, s, _species(cells, ppc, q, m, w, th, 1.5, -1.0, _generator(seed, s)))
    sim.upload_fields(*I.wall_fields(nx, ny, nz, E0, B0))
    # what enters in the next steps, drawn before them
    source = I.Injector(box, specs, 1.5, seed=seed)
    return dict(case=case, sim=sim, dump=_Dump(box, False), opts=_opts("restarted"), inject=[source.step() for _ in range(6)], at=0)


def _system(case, seed):
    """A system of the kind the beams give: mu near -0.2 on the diagonal, with
    the particles' noise, and a right part with structure on all scales."""
    g = _generator(seed, 9)
    n = case["nx"] * case["ny"] * case["nz"]
    shape = (case["nz"], case["ny"], case["nx"])
    noise = torch.randn((9, n), generator=g, device=g.device, dtype=torch.float32).double()
    mu = 0.01 * noise
    for d in (0, 4, 8):
        mu[d] = -0.2 + 0.05 * noise[d]
    rhs = torch.randn((3, n), generator=g, device=g.device, dtype=torch.float32).double()
    x = torch.arange(case["nx"], device=g.device, dtype=torch.float64) * (2 * math.pi / case["nx"])
    wave = torch.sin(x).expand(shape).reshape(-1)
    for d in range(3):
        rhs[d] += 3.0 * wave * (d + 1)
    return mu, rhs


def _prepare_solve(case, seed):
    box = I.Box(case["nx"], case["ny"], case["nz"], 0.5, 0.5, 0.5, 0.5, theta=0.5)
    sim = P.GpuSimulation(box, P.IMPLICIT, particle_real=P.F64, pressure_compat=0, tile=(0, 0, 0))
    mu, rhs = (_pinned(t.reshape(-1)).numpy() for t in _system(case, seed))
    return dict(case=case, sim=sim, mu=mu, rhs=rhs, opts=_opts(case["solver"]))


# the network's layers: name, input and output channels, level
_LAYERS = [("e0a", 16, 16), ("e0b", 16, 16), ("e1a", 16, 32), ("e1b", 32, 32), ("e2a", 32, 64), ("e2b", 64, 64),
           ("d1a", 96, 32), ("d1b", 32, 32), ("d0a", 48, 16), ("d0b", 16, 16), ("head", 16, 16)]


def _network(case, seed):
    """Weights (He-normal, small biases), input and target of one batch."""
    rng = np.random.default_rng(seed)
    parts = []
    for name, ci, co in _LAYERS:
        real_in, real_out = 6 if name == "e0a" else ci, 3 if name == "head" else co
        W, b = np.zeros((27, co, ci), dtype=np.float32), np.zeros(co, dtype=np.float32)
        W[:, :real_out, :real_in] = rng.standard_normal((27, real_out, real_in)) * math.sqrt(2.0 / (27 * real_in))
        b[:real_out] = 0.05 * rng.standard_normal(real_out)
        parts += [W.reshape(-1), b]
    params = np.concatenate(parts + [np.ones(1, dtype=np.float32)])
    shape = (case["batch"], case["nz"], case["ny"], case["nx"])
    x0 = np.zeros(shape + (16,), dtype=np.float32)
    x0[..., :3] = rng.standard_normal(shape + (3,), dtype=np.float32)
    x0[..., 3:6] = -0.3 * rng.random(shape + (3,), dtype=np.float32)
    return params, x0, rng.standard_normal(shape + (3,), dtype=np.float32)


def _prepare_gradient(case, seed):
    box = I.Box(8, 8, 8, 0.5, 0.5, 0.5, 0.5)
    sim = P.GpuSimulation(box, P.IMPLICIT, particle_real=P.F64, pressure_compat=0)
    params, x0, target = _network(case, seed)
    sim.nn_set_params(params)
    return dict(case=case, sim=sim, x0=x0, target=target)


# ------------------------------------------------------------------ one pass
def run(state):
    case, sim = state["case"], state["sim"]
    kind = case["kind"]
    if kind == "explicit":
        sim.buneman_step(case["steps"])
        return state["dump"].fields(sim)
    if kind == "implicit":
        for _ in range(case["steps"]):
            sim.implicit_step(state["opts"])
        return state["dump"].fields(sim) + state["dump"].particles(sim)
    if kind == "shock":
        for s, new in enumerate(state["inject"][state["at"] % len(state["inject"])]):
            sim.append_particles(s, new)
        state["at"] += 1
        sim.implicit_step(state["opts"])
        return state["dump"].fields(sim)
    if kind == "solve":
        return sim.maxwell_solve(state["mu"], state["rhs"], state["opts"])[0]
    if kind == "gradient":
        loss, grad = sim.nn_loss_grad(state["x0"], state["target"])
        return [np.float32(loss), grad]
    sim.updateDensityParameters()
    out = [a.astype(np.float32) for s in range(2) for a in sim.download_density(s)]
    return out + [sim.updateEnergy().astype(np.float32)]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind, n = case["kind"], case["nx"] * case["ny"] * case["nz"]
    if kind == "gradient":
        vox = case["batch"] * n
        lvl = {"e0a": 0, "e0b": 0, "e1a": 1, "e1b": 1, "e2a": 2, "e2b": 2, "d1a": 1, "d1b": 1, "d0a": 0, "d0b": 0, "head": 0}
        flops = sum(3 * 2 * 27 * ci * co / 8 ** lvl[k] for k, ci, co in _LAYERS) * vox   # forward, two products back
        return {"bytes": 76.0 * vox + 8.0 * sum(27 * ci * co + co for _, ci, co in _LAYERS), "flops": flops}
    # a field solve: mu, the right part and the solution; about 17 Arnoldi
    # steps of the operator (63 operations a node) and Gram-Schmidt
    solve = (120.0 * n, 17.0 * (63 + 3 * 4 * 9) * n)
    if kind == "solve":
        return {"bytes": solve[0], "flops": solve[1]}
    if kind == "shock":
        parts, size, steps = n * 72, 4, 1
    else:
        parts, size, steps = 2 * n * case["ppc"], 8 if case["f64"] else 4, case.get("steps", 1)
    one = 4 + 6 * size   # cell, offsets, momenta
    if kind == "moments":
        return {"bytes": float(parts * one + 11 * 8 * n), "flops": 80.0 * parts}
    if kind == "explicit":   # particles read and written, E, B read and written, J
        return {"bytes": float(steps * (2 * one * parts + (12 * size + 24) * n)), "flops": 330.0 * parts * steps}
    # particles read for the moments, read and written by the mover; E, B in and
    # out, 19 moments
    return {"bytes": steps * (3.0 * one * parts + (96 + 2 * 19 * 8) * n + solve[0]), "flops": steps * (1100.0 * parts + solve[1])}


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    """What run() returns for a new state, in plain torch in 64 bits."""
    kind = case["kind"]
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind == "solve":
        box = I.Box(case["nx"], case["ny"], case["nz"], 0.5, 0.5, 0.5, 0.5, theta=0.5)
        mu, rhs = _system(case, seed)
        g = _Grid(box)
        return g.solve(mu.reshape(9, *g.shape), rhs.reshape(3, *g.shape)).reshape(-1).cpu().numpy()
    # the wall box's boundary rows and the reference's pressure placement are
    # the library's own conventions; the largest box would take minutes
    if kind == "shock" or case.get("compat") or _filled(case):
        return None
    box, species, B0 = _plasma(case, seed)
    g = _Grid(box)
    E = torch.zeros((3,) + g.shape, dtype=torch.float64, device=_device())
    B = E + torch.tensor(B0, dtype=torch.float64, device=_device()).view(3, 1, 1, 1)
    parts = [_Particles(box, sp) for sp in species]
    if kind == "implicit":
        for _ in range(case["steps"]):
            E, B, J = g.implicit_step(parts, E, B)
        out = [t.cpu() for t in (E, B, J)]
        return out + ([p.phase_space().cpu() for p in parts] if case["particles"] else [])
    for _ in range(1 if kind == "moments" else case["steps"]):
        E, B, J = g.explicit_step(parts, E, B, case.get("smooth", 0))
    if kind == "explicit":
        return [t.cpu() for t in (E, B, J)]
    return g.density(parts, E, B)


class _Particles:
    def __init__(self, box, sp):
        self.box, self.q, self.m, self.w = box, sp["q"], sp["m"], sp["w"]
        c = sp["cell"].long()
        self.c = [c % box.nx, c // box.nx % box.ny, c // (box.nx * box.ny)]
        self.u = [sp["ox"], sp["oy"], sp["oz"]]
        self.p = [sp["px"], sp["py"], sp["pz"]]

    def chunks(self, most=1 << 23):
        n = self.p[0].numel()
        for a in range(0, n, most):
            yield slice(a, min(n, a + most))

    def phase_space(self):
        d = (self.box.dx, self.box.dy, self.box.dz)
        return torch.stack([(self.c[a] + self.u[a]) * d[a] for a in range(3)] + self.p)


def _cross(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


class _Grid:
    """The method on a periodic box: arrays [component, k, j, i]."""

    def __init__(self, box):
        self.box = box
        self.n = (box.nx, box.ny, box.nz)
        self.d = (box.dx, box.dy, box.dz)
        self.shape = (box.nz, box.ny, box.nx)
        self.vol = box.dx * box.dy * box.dz

    def at(self, f, i=0, j=0, k=0):
        """f shifted so that the value of (i, j, k) further on stands at each place."""
        for s, dim in ((i, -1), (j, -2), (k, -3)):
            if s:
                f = torch.roll(f, -s, dim)
        return f

    def index(self, i, j, k):
        return ((k % self.n[2]) * self.n[1] + j % self.n[1]) * self.n[0] + i % self.n[0]

    # -------------------------------------------------------------- weights
    def node(self, axis, c, u):
        if self.n[axis] == 1:
            return [(c, torch.ones_like(u))]
        return [(c, 1.0 - u), (c + 1, u)]

    def centre(self, axis, c, u):
        if self.n[axis] == 1:
            return [(c, torch.ones_like(u))]
        low = u < 0.5
        first = torch.where(low, c - 1, c)
        up = torch.where(low, u + 0.5, u - 0.5)
        return [(first, 1.0 - up), (first + 1, up)]

    def spread(self, wx, wy, wz):
        for i, a in wx:
            for j, b in wy:
                for k, c in wz:
                    yield self.index(i, j, k), a * b * c

    def gather(self, fields, wx, wy, wz):
        out = [0.0] * len(fields)
        for at, w in self.spread(wx, wy, wz):
            for d, f in enumerate(fields):
                out[d] = out[d] + f.reshape(-1)[at] * w
        return out

    # -------------------------------------------------------------- explicit
    def b_half(self, E, B):
        dx, dy, dz = self.d
        f = self.box.cfix * self.box.dt / 2.0
        ddx = lambda a: (self.at(a, i=1) - a) / dx   # noqa: E731
        ddy = lambda a: (self.at(a, j=1) - a) / dy   # noqa: E731
        ddz = lambda a: (self.at(a, k=1) - a) / dz   # noqa: E731
        rot = torch.stack([ddy(E[2]) - ddz(E[1]), ddz(E[0]) - ddx(E[2]), ddx(E[1]) - ddy(E[0])])
        return B - rot * f

    def e_step(self, E, B, J):
        dx, dy, dz = self.d
        ddx = lambda a: (a - self.at(a, i=-1)) / dx   # noqa: E731
        ddy = lambda a: (a - self.at(a, j=-1)) / dy   # noqa: E731
        ddz = lambda a: (a - self.at(a, k=-1)) / dz   # noqa: E731
        rot = torch.stack([ddy(B[2]) - ddz(B[1]), ddz(B[0]) - ddx(B[2]), ddx(B[1]) - ddy(B[0])])
        return E + (self.box.cfix * rot - FOUR_PI * J) * self.box.dt

    def advance(self, p, sl, axis, move):
        """x += move (in cells), with the periodic wrap."""
        un = p.u[axis][sl] + move
        s = torch.floor(un)
        un = un - s
        over = un >= 1.0
        c = p.c[axis][sl] + s.long() + over.long()
        return torch.where(over, un - 1.0, un), c % self.n[axis]

    def push(self, p, sl, E, B):
        dt, m = self.box.dt, p.m
        nd = [self.node(a, p.c[a][sl], p.u[a][sl]) for a in range(3)]
        ce = [self.centre(a, p.c[a][sl], p.u[a][sl]) for a in range(3)]
        e = [self.gather([E[0]], ce[0], nd[1], nd[2])[0], self.gather([E[1]], nd[0], ce[1], nd[2])[0],
             self.gather([E[2]], nd[0], nd[1], ce[2])[0]]
        b = [self.gather([B[0]], nd[0], ce[1], ce[2])[0], self.gather([B[1]], ce[0], nd[1], ce[2])[0],
             self.gather([B[2]], ce[0], ce[1], nd[2])[0]]
        dp = [x * (p.q * dt * 0.5) for x in e]
        mom = [p.p[a][sl] + dp[a] for a in range(3)]
        bs = p.q * dt / (2.0 * m) / torch.sqrt(_dot(mom, mom) / (m * m) + 1.0)
        f = 2.0 / torch.sqrt(1.0 + bs * bs * _dot(b, b))
        half = _cross(mom, b)
        half = [mom[a] + half[a] * bs for a in range(3)]
        turn = _cross(half, b)
        mom = [mom[a] + (turn[a] * (f * bs) + dp[a]) for a in range(3)]
        gam = torch.sqrt(_dot(mom, mom) / (m * m) + 1.0)
        v = [x / (m * gam) for x in mom]
        for a in range(3):
            p.p[a][sl] = mom[a]
            p.u[a][sl], p.c[a][sl] = self.advance(p, sl, a, v[a] * dt / self.d[a])
        return v

    def zigzag(self, p, sl, v, J):
        dt = self.box.dt
        fcd = p.q * p.w / self.vol
        shift, old, rel, new = [], [], [], []
        for a in range(3):
            X = p.u[a][sl] * self.d[a]
            before = X - v[a] * dt
            if self.n[a] == 1:
                s = torch.zeros_like(p.c[a][sl])
            else:
                s = torch.floor(before / self.d[a]).long()
            r = torch.where(s == 0, (X + before) / 2, torch.clamp(s, min=0).double() * self.d[a])
            shift.append(s), old.append(before), rel.append(r), new.append(X)
        for first in (True, False):
            if first:
                F = [fcd * (rel[a] - old[a]) / dt for a in range(3)]
                W = [(old[a] + rel[a]) / (2 * self.d[a]) - shift[a] for a in range(3)]
                c = [p.c[a][sl] + shift[a] for a in range(3)]
            else:
                F = [fcd * (new[a] - rel[a]) / dt for a in range(3)]
                W = [(new[a] + rel[a]) / (2 * self.d[a]) for a in range(3)]
                c = [p.c[a][sl] for a in range(3)]
            pair = [self.node(a, c[a], W[a]) for a in range(3)]
            here = [[(c[a], 1.0)] for a in range(3)]
            for a in range(3):
                use = [here[b] if b == a else pair[b] for b in range(3)]
                for at, w in self.spread(*use):
                    J[a].view(-1).index_add_(0, at, F[a] * w)

    def smooth(self, f):
        for dim, n in ((-1, self.n[0]), (-2, self.n[1]), (-3, self.n[2])):
            if n > 1:
                f = 0.5 * f + 0.25 * (torch.roll(f, 1, dim) + torch.roll(f, -1, dim))
        return f

    def explicit_step(self, parts, E, B, smooth):
        B = self.b_half(E, B)
        J = torch.zeros_like(E)
        for p in parts:
            for sl in p.chunks():
                self.zigzag(p, sl, self.push(p, sl, E, B), J)
        B = self.b_half(E, B)
        for _ in range(smooth):
            J = self.smooth(J)
        return self.e_step(E, B, J), B, J

    def density(self, parts, E, B):
        out, rho, energy = [], 0.0, torch.zeros(6, dtype=torch.float64)
        for p in parts:
            conc, en, vel = (torch.zeros((k,) + self.shape, dtype=torch.float64, device=E.device) for k in (1, 1, 3))
            for sl in p.chunks():
                mom = [x[sl] for x in p.p]
                lor = torch.sqrt(_dot(mom, mom) / (p.m * p.m) + 1.0)
                use = [self.centre(a, p.c[a][sl], p.u[a][sl]) for a in range(3)]
                for at, w in self.spread(*use):
                    w = w * (p.w / self.vol)
                    conc.view(-1).index_add_(0, at, w)
                    en.view(-1).index_add_(0, at, w * lor * p.m)
                    for d in range(3):
                        vel[d].view(-1).index_add_(0, at, w * mom[d])
                energy[0] += float(((lor - 1) * p.m * p.w).sum())
                for d in range(3):
                    energy[3 + d] += float(mom[d].sum() * p.w)
            rho = rho + p.q * conc
            vel = torch.where(en > 0, vel / torch.where(en > 0, en, torch.ones_like(en)), torch.zeros_like(vel))
            out.append([conc.reshape(-1), en.reshape(-1), vel.reshape(3, -1)])
        energy[1] = float((E * E).sum()) * self.vol / (8 * math.pi)
        energy[2] = float((B * B).sum()) * self.vol / (8 * math.pi)
        return [t.cpu() for three in out for t in three + [rho.reshape(-1)]] + [energy]

    # -------------------------------------------------------------- implicit
    def alpha(self, p, v, gam, e, b):
        """The rotation tensor, rows of three."""
        beta = 0.5 * p.q * self.box.dt / p.m
        G = beta * _dot(e, v) + gam
        bs = beta / G
        den = G * (1 + bs * bs * _dot(b, b))
        al = [[((1.0 if i == j else 0.0) + bs * bs * b[i] * b[j]) / den for j in range(3)] for i in range(3)]
        for i, j, l, s in ((0, 1, 2, 1), (1, 2, 0, 1), (2, 0, 1, 1), (1, 0, 2, -1), (2, 1, 0, -1), (0, 2, 1, -1)):
            al[i][j] = al[i][j] + s * bs * b[l] / den
        return al

    def state(self, p, sl, E, B):
        mom = [x[sl] for x in p.p]
        gam = torch.sqrt(_dot(mom, mom) / (p.m * p.m) + 1.0)
        v = [x / (p.m * gam) for x in mom]
        nd = [self.node(a, p.c[a][sl], p.u[a][sl]) for a in range(3)]
        ce = [self.centre(a, p.c[a][sl], p.u[a][sl]) for a in range(3)]
        e, b = self.gather(list(E), *nd), self.gather(list(B), *ce)
        return mom, gam, v, nd, ce, b, self.alpha(p, v, gam, e, b)

    def deposit(self, parts, E, B):
        bx = self.box
        J, mu, rho, Pi = (torch.zeros((k,) + self.shape, dtype=torch.float64, device=E.device) for k in (3, 9, 1, 9))
        for p in parts:
            omega = p.w * bx.theta * bx.dt * bx.dt * 2 * math.pi * p.q * p.q / p.m
            for sl in p.chunks(1 << 22):
                mom, gam, v, nd, ce, b, al = self.state(p, sl, E, B)
                rv = [gam * _dot(al[a], v) for a in range(3)]
                for at, w in self.spread(*nd):
                    w = w / self.vol
                    for d in range(3):
                        J[d].view(-1).index_add_(0, at, rv[d] * (p.q * p.w * w))
                        for c in range(3):
                            mu[3 * d + c].view(-1).index_add_(0, at, al[d][c] * (-omega * w))
                for at, w in self.spread(*ce):
                    w = w * (p.q * p.w / self.vol)
                    rho[0].view(-1).index_add_(0, at, w)
                    for d in range(3):
                        for c in range(d, 3):
                            Pi[3 * d + c].view(-1).index_add_(0, at, w * rv[d] * rv[c])
        for d, c in ((1, 0), (2, 0), (2, 1)):
            Pi[3 * d + c] = Pi[3 * c + d]
        return J, mu, rho[0], Pi

    def step(self, axis):
        return {"i" if axis == 0 else "j" if axis == 1 else "k": 1}

    def ddn(self, f, axis):
        """Derivative at nodes of a cell-centred field: the averages over the two other axes."""
        if self.n[axis] == 1:
            return torch.zeros_like(f)
        for a in range(3):
            if a != axis:
                f = 0.5 * (f + self.at(f, **{k: -s for k, s in self.step(a).items()}))
        return (f - self.at(f, **{k: -s for k, s in self.step(axis).items()})) / self.d[axis]

    def ddc(self, f, axis):
        """Derivative at cell centres of a node-centred field."""
        if self.n[axis] == 1:
            return torch.zeros_like(f)
        for a in range(3):
            if a != axis:
                f = 0.5 * (f + self.at(f, **self.step(a)))
        return (self.at(f, **self.step(axis)) - f) / self.d[axis]

    def operator(self, mu, x):
        K = (self.box.theta * self.box.dt) ** 2 * self.box.cfix ** 2
        u = torch.stack([sum(mu[3 * a + b] * x[b] for b in range(3)) for a in range(3)])
        y = x - u
        names = "ijk"
        for a in range(3):
            for ax in range(3):
                if self.n[ax] == 1:
                    continue
                one = names[ax]
                y[a] += K / self.d[ax] ** 2 * (2 * x[a] - self.at(x[a], **{one: 1}) - self.at(x[a], **{one: -1}))
                if ax == a:
                    y[a] += K / self.d[a] ** 2 * (self.at(u[a], **{one: 1}) + self.at(u[a], **{one: -1}) - 2 * u[a])
                elif self.n[a] > 1:
                    two, f = names[a], u[ax]
                    y[a] += K / (4 * self.d[a] * self.d[ax]) * (
                        self.at(f, **{one: 1, two: 1}) + self.at(f, **{one: -1, two: -1}) -
                        self.at(f, **{one: -1, two: 1}) - self.at(f, **{one: 1, two: -1}))
        return y

    def solve(self, mu, rhs, tol=2e-15, most=120):
        """GMRES from zero, restarted on the true residual."""
        x, top = torch.zeros_like(rhs), float(rhs.norm())
        for _ in range(6):
            r = rhs - self.operator(mu, x)
            beta = float(r.norm())
            if beta <= tol * top:
                break
            V, H = [(r / beta).reshape(-1)], np.zeros((most + 1, most))
            g = np.zeros(most + 1)
            g[0] = beta
            cs, sn, k = [], [], 0
            for k in range(most):
                w = self.operator(mu, V[k].view(rhs.shape)).reshape(-1)
                A = torch.stack(V)
                h = A @ w
                w = w - h @ A
                h2 = A @ w
                w = w - h2 @ A
                col = np.append((h + h2).cpu().numpy(), float(w.norm()))
                V.append(w / col[-1])
                for q in range(k):
                    col[q], col[q + 1] = cs[q] * col[q] + sn[q] * col[q + 1], cs[q] * col[q + 1] - sn[q] * col[q]
                t = math.hypot(col[k], col[k + 1])
                cs.append(col[k] / t), sn.append(col[k + 1] / t)
                H[:k + 1, k] = np.append(col[:k], t)
                g[k + 1], g[k] = -sn[k] * g[k], cs[k] * g[k]
                if abs(g[k + 1]) <= 1e-9 * beta or abs(g[k + 1]) <= tol * top:
                    break
            k += 1
            y = np.linalg.solve(H[:k, :k], g[:k])
            x = x + (torch.as_tensor(y, device=x.device) @ torch.stack(V[:k])).view(rhs.shape)
        return x

    def implicit_step(self, parts, E, B):
        bx = self.box
        J, mu, rho, Pi = self.deposit(parts, E, B)
        if min(self.n) > 1:   # the pressure's divergence acts in three dimensions only
            J = J - bx.eta * bx.dt * torch.stack([sum(self.ddn(Pi[3 * a + c], a) for a in range(3)) for c in range(3)])
        rho = rho - bx.dt * bx.theta * sum(self.ddc(J[a], a) for a in range(3))
        td, cf = bx.theta * bx.dt, bx.cfix
        rot = torch.stack([self.ddn(B[2], 1) - self.ddn(B[1], 2), self.ddn(B[0], 2) - self.ddn(B[2], 0),
                           self.ddn(B[1], 0) - self.ddn(B[0], 1)])
        grad = torch.stack([self.ddn(rho, a) for a in range(3)])
        rhs = E + (rot * cf - J * FOUR_PI) * td - grad * (cf * cf * td * td * FOUR_PI)
        Et = self.solve(mu, rhs)
        rot = torch.stack([self.ddc(Et[2], 1) - self.ddc(Et[1], 2), self.ddc(Et[0], 2) - self.ddc(Et[2], 0),
                           self.ddc(Et[1], 0) - self.ddc(Et[0], 1)])
        for p in parts:
            for sl in p.chunks(1 << 22):
                self.move(p, sl, E, B, Et)
        return (Et - E * (1 - bx.theta)) / bx.theta, B - rot * (cf * bx.dt), J

    def move(self, p, sl, E, B, Et):
        bx = self.box
        dt, eta, m = bx.dt, bx.eta, p.m
        mom, gam, v, nd, ce, b, al = self.state(p, sl, E, B)
        e = self.gather(list(Et), *nd)
        beta, qdt = 0.5 * p.q * dt / m, p.q * dt
        vxb = _cross(v, b)
        new = [mom[a] + (e[a] + vxb[a]) * qdt for a in range(3)]
        p2 = _dot(new, new)
        slow = torch.where(p2 < 1e-4 * m * m, torch.ones_like(p2), torch.sqrt(p2 + m * m) / m)
        mv = [v[a] * (1 - eta) + new[a] / (m * slow) * eta for a in range(3)]
        vh = [gam * _dot(al[a], v) for a in range(3)]
        most = 1e-14 * torch.sqrt(_dot(mom, mom))
        diff = [mom[a] - new[a] for a in range(3)]
        on = torch.sqrt(_dot(diff, diff)) > most
        far = [x * (eta * dt) for x in mv]
        for _ in range(3):
            if not bool(on.any()):
                break
            nv = [vh[a] + _dot(al[a], e) * beta for a in range(3)]
            nf = [x * (eta * dt) for x in nv]
            at = [self.advance(p, sl, a, nf[a] / self.d[a]) for a in range(3)]
            ne = self.gather(list(Et), *[self.node(a, at[a][1], at[a][0]) for a in range(3)])
            nb = self.gather(list(B), *[self.centre(a, at[a][1], at[a][0]) for a in range(3)])
            nxb = _cross(nv, nb)
            nn = [mom[a] + (ne[a] + nxb[a]) * qdt for a in range(3)]
            dm = [new[a] - nn[a] for a in range(3)]
            df = [far[a] - nf[a] for a in range(3)]
            keep = lambda x, y: [torch.where(on, x[a], y[a]) for a in range(3)]   # noqa: E731
            e, mv, far, new = keep(ne, e), keep(nv, mv), keep(nf, far), keep(nn, new)
            on = on & (torch.sqrt(_dot(dm, dm)) > most) & (torch.sqrt(_dot(df, df)) > 1e-8 * bx.dx)
        for a in range(3):
            p.u[a][sl], p.c[a][sl] = self.advance(p, sl, a, mv[a] * dt / self.d[a])
            p.p[a][sl] = new[a]


def _exact_gradient(case, seed):
    params, x0, target = _network(case, seed)
    dev = _device()
    conv, pool = torch.nn.functional.conv3d, torch.nn.functional.avg_pool3d
    up = lambda x: torch.nn.functional.interpolate(x, scale_factor=2, mode="nearest")   # noqa: E731
    at, net, flat = 0, {}, []
    for name, ci, co in _LAYERS:
        W = torch.tensor(params[at:at + 27 * ci * co], dtype=torch.float64, device=dev, requires_grad=True)
        b = torch.tensor(params[at + 27 * ci * co:at + 27 * ci * co + co], dtype=torch.float64, device=dev, requires_grad=True)
        at += 27 * ci * co + co
        net[name] = (W.view(3, 3, 3, co, ci).permute(3, 4, 0, 1, 2), b)
        flat += [W, b]
    ch = lambda x: torch.tensor(x, dtype=torch.float64, device=dev).permute(0, 4, 1, 2, 3)   # noqa: E731
    cv = lambda name, x: conv(x, net[name][0], net[name][1], padding=1)   # noqa: E731
    e0 = cv("e0b", cv("e0a", ch(x0)))
    e1 = cv("e1b", cv("e1a", pool(e0, 2)))
    e2 = cv("e2b", cv("e2a", pool(e1, 2)))
    d1 = cv("d1b", cv("d1a", torch.cat([up(e2), e1], 1)))
    d0 = cv("d0b", cv("d0a", torch.cat([up(d1), e0], 1)))
    loss = (cv("head", d0)[:, :3] - ch(target)).square().mean()
    grad = torch.autograd.grad(loss, flat)
    return [float(loss.detach()), torch.cat(list(grad) + [torch.zeros(1, dtype=torch.float64, device=dev)]).cpu().numpy()]
