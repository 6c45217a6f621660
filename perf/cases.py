"""The work that users of this framework have it do, as measurable cases
through its public entry points.

  frame    frames of the simulation loop: a few substeps (Sim.step), then the
           statistics (Sim.read_stats), on a burning pool
  vcycles  the stand-alone pressure solver with the reference's fixed V-cycles
  cg       the stand-alone pressure solver with MGPCG, FP32 or BF16 storage,
           to a tolerance
  net      the learned warm start's forward pass (Net.forward)
  grad     loss and gradients of the learned stage on a batch of crops
           (Net.loss_grad), the work of a training step
  render   one path-traced frame of a burning pool (Renderer.render_device),
           with light caches or with pure path tracing
  develop  one traced image to 8-bit sRGB (Developer.develop)

`listed()` gives the cases that stand for these, `draw(rng)` others of the
same ranges, `prepare(case, seed)` what a program holds before the call,
`run(state)` one pass, `work(case)` the bytes and operations it cannot do
without and `exact(case, seed)` the outputs in 64 bits from plain torch.
"""
import math
import os

import numpy as np
import torch
import torch.nn.functional as F

from pyro_b200 import _abi
from pyro_b200.develop import Developer
from pyro_b200.learned import SPEC, Net
from pyro_b200.poisson import PoissonSolver
from pyro_b200.post import Camera
from pyro_b200.render import Renderer
from pyro_b200.scene import Domain, Ignition, Object, Scene, SimCfg
from pyro_b200.sim import Sim

DEV = "cuda"
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(_abi.__file__)), "weights",
                       "warmstart.pnet")
FPS = 30.0


def listed():
    return [
        # The small pool at 8 cm (scenes/pool_small_8cm.toml's 32 x 80 x 32
        # grid): a frame is two substeps and its statistics, bound by
        # launches and the latency of small levels.
        dict(name="frame_8cm", kind="frame", nx=32, ny=80, nz=32, dx=0.08, substeps=2,
             solver="vcycle"),
        # The headline scene, the 2 cm pool (scenes/pool_2cm.toml): a 1/30 s
        # frame of six substeps with the reference's four V-cycles each.
        dict(name="frame_2cm", kind="frame", nx=160, ny=320, nz=160, dx=0.02, substeps=6,
             solver="vcycle"),
        # The 4 cm pool on the exact grid of its 3.0 x 7.3 x 3.0 m domain,
        # which does not halve evenly: three substeps with BF16 MGPCG to 1e-4
        # (the solver such grids need).
        dict(name="frame_odd_cg", kind="frame", nx=75, ny=183, nz=75, dx=0.04, substeps=3,
             solver="mgpcg_bf16"),
        # The pressure solver by itself with the reference's scheme, four
        # V-cycles on the grid of the 5 cm pallet stack.
        dict(name="vcycles_pallets", kind="vcycles", nx=128, ny=240, nz=128, dx=0.05, cycles=4),
        # MGPCG in FP32 to 1e-6 on the 256^3 case with 5 % solid boxes, the
        # largest solve.
        dict(name="cg_fp32_256", kind="cg", nx=256, ny=256, nz=256, dx=0.02, mode="mgpcg",
             tol=1e-6),
        # BF16 MGPCG to 1e-4 on the exact 2 cm grid (odd coarse rows).
        dict(name="cg_bf16_odd", kind="cg", nx=150, ny=365, nz=150, dx=0.02,
             mode="mgpcg_bf16", tol=1e-4),
        # The learned warm start's forward pass on the 2 cm pool's grid.
        dict(name="net_2cm", kind="net", nx=160, ny=320, nz=160, nb=1, dx=0.02),
        # ... and on the small pool's, where launches count.
        dict(name="net_8cm", kind="net", nx=32, ny=80, nz=32, nb=1, dx=0.08),
        # One training batch: two crops of 128^3, as the training loop draws.
        dict(name="grad_2x128", kind="grad", nx=128, ny=128, nz=128, nb=2, dx=0.02),
        # A default frame of the path tracer: 1280 x 720, light caches.
        dict(name="render_cache", kind="render", nx=80, ny=160, nz=80, dx=0.04, width=1280,
             height=720, spp=16, mode="cache"),
        # The same flame with pure path tracing, at preview size.
        dict(name="render_path", kind="render", nx=80, ny=160, nz=80, dx=0.04, width=640,
             height=360, spp=8, mode="path"),
        # A traced 1280 x 720 image to 8-bit sRGB with glare.
        dict(name="develop_720p", kind="develop", width=1280, height=720),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: grids from the small pool to the 2 cm one, ragged sizes
    where the path takes them (the reference's V-cycles need dimensions of a
    multiple of 16, as its scene loader makes them)."""
    kind = rng.choice(["frame", "frame", "vcycles", "cg", "cg", "net", "grad", "render",
                       "develop"])
    if kind == "frame":
        w = _log(rng, 24, 150)
        h = rng.randint(int(1.6 * w), int(2.2 * w))
        solver = rng.choice(["vcycle", "vcycle", "mgpcg", "mgpcg_bf16"])
        if solver == "vcycle":
            w, h = (w + 15) // 16 * 16, (h + 15) // 16 * 16
        return dict(kind=kind, nx=w, ny=h, nz=w, dx=round(3.2 / w, 4),
                    substeps=rng.randint(1, 3), solver=solver)
    if kind == "vcycles":
        d = [max(2, round(_log(rng, 32, 224) / 16)) * 16 for _ in range(3)]
        return dict(kind=kind, nx=d[0], ny=d[1], nz=d[2], dx=0.05, cycles=rng.randint(1, 4))
    if kind == "cg":
        d = [_log(rng, 20, 220) for _ in range(3)]
        return dict(kind=kind, nx=d[0], ny=d[1], nz=d[2], dx=0.02,
                    mode=rng.choice(["mgpcg", "mgpcg_bf16"]), tol=rng.choice([1e-4, 1e-6]))
    if kind == "net":
        d = [_log(rng, 12, 200) for _ in range(3)]
        return dict(kind=kind, nx=d[0], ny=d[1], nz=d[2], nb=rng.randint(1, 2), dx=0.02)
    if kind == "grad":
        d = [_log(rng, 16, 128) for _ in range(3)]
        return dict(kind=kind, nx=d[0], ny=d[1], nz=d[2], nb=rng.randint(1, 2), dx=0.02)
    if kind == "render":
        w = rng.randint(32, 80)
        return dict(kind=kind, nx=w, ny=2 * w, nz=w, dx=round(3.2 / w, 4),
                    width=rng.randint(160, 900), height=rng.randint(120, 540),
                    spp=rng.randint(2, 12), mode=rng.choice(["cache", "cache", "path"]))
    return dict(kind="develop", width=rng.randint(160, 1280), height=rng.randint(120, 720))


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _noise(g, shape, cells):
    """Smooth noise of unit variance with features of `cells` cells."""
    lo = [max(2, int(math.ceil(n / cells)) + 1) for n in shape]
    a = torch.randn([1, 1] + lo, generator=g, device=DEV)
    a = F.interpolate(a, size=list(shape), mode="trilinear", align_corners=True)[0, 0]
    return a / a.std().clamp_min(1e-6)


def _scene(case):
    nx, ny, nz, dx = case["nx"], case["ny"], case["nz"], case["dx"]
    cx, cz = 0.5 * nx * dx, 0.5 * nz * dx
    sc = Scene(domain=Domain([nx * dx, ny * dx, nz * dx], dx),
               sim=SimCfg(vorticity=6.0, fps=FPS),
               ignition=Ignition(pos=[cx, 0.12, cz], radius=0.3, flux=30000.0, temp=1300.0,
                                 until=4.0),
               objects=[Object(kind="pool", material="heptane", center=[cx, 0.0, cz],
                               radius=0.5, depth=max(0.08, dx))])
    sc.dims_override = [nx, ny, nz]
    return sc


def _burning(case, sim, seed):
    """A burning plume above the pool: hot core with fuel at its base, oxygen
    drawn down, soot and smoke above, a buoyant jet with turbulence."""
    g = _gen(seed)
    nx, ny, nz, dx = case["nx"], case["ny"], case["nz"], case["dx"]
    shape = (nz, ny, nx)

    def axes(s, off):
        return [((torch.arange(n, device=DEV) + o) * dx) for n, o in zip(s, off)]

    z, y, x = axes(shape, (0.5, 0.5, 0.5))
    cx, cz = 0.5 * nx * dx, 0.5 * nz * dx
    top = ny * dx
    width = 0.35 + 0.12 * y / top * 4.0
    sway = 0.15 * torch.sin(3.0 * y + 6.28 * float(torch.rand(1, generator=g, device=DEV)))
    r2 = ((x[None, None, :] - cx - sway[None, :, None]) ** 2 + (z[:, None, None] - cz) ** 2)
    core = torch.exp(-r2 / (width ** 2)[None, :, None])
    fade = torch.exp(-(y / (0.55 * top)) ** 2)[None, :, None]
    n1 = _noise(g, shape, max(2.0, 0.12 / dx))
    n2 = _noise(g, shape, max(2.0, 0.3 / dx))
    body = (core * fade * (1.0 + 0.35 * n1 + 0.2 * n2)).clamp(0.0, 1.2)
    s0 = torch.zeros(shape + (4,), device=DEV)
    s0[..., 0] = 293.0 + 1500.0 * body
    s0[..., 1] = 0.25 * body * torch.exp(-y / 0.8)[None, :, None]
    s0[..., 2] = 0.233 * (1.0 - 0.9 * body.clamp(0.0, 1.0))
    s0[..., 3] = 0.004 * body * (1.0 + 0.5 * n2).clamp(0.0, 2.0)
    s1 = torch.zeros(shape + (4,), device=DEV)
    s1[..., 0] = 0.006 * body.sqrt()
    s1[..., 1] = 1.5e6 * body * (body > 0.25)
    s1[..., 2] = 2.0 * body * n1
    sim.write_field(_abi.F_S0, s0.cpu().numpy())
    sim.write_field(_abi.F_S1, s1.cpu().numpy())
    fshape = (nz + 1, ny + 1, nx + 1)
    z, y, x = axes(fshape, (0.5, 0.0, 0.5))
    jet = torch.exp(-((x[None, None, :] - cx) ** 2 + (z[:, None, None] - cz) ** 2) / 0.25)
    rise = (3.5 * torch.sqrt(y / top).clamp(0.0, 1.0))[None, :, None] * jet
    for f, base, amp in ((_abi.F_U, 0.0, 0.8), (_abi.F_V, rise, 0.8), (_abi.F_W, 0.0, 0.8)):
        t = amp * _noise(g, fshape, max(2.0, 0.25 / dx)) * (0.15 + jet) + base
        t[:, 0, :] = 0.0
        sim.write_field(f, t.to(torch.float32).contiguous().cpu().numpy())


class _Borrowed:
    """A device array of the library as torch sees it; it keeps the object
    that owns the memory alive."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f4",
                                             data=(int(ptr), False), version=3)


def _boxes(case, seed):
    """Flags with 5 % of the cells solid in random boxes, and a zero-mean
    right-hand side on the fluid cells."""
    rng = np.random.default_rng(int(seed) + 1)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    f = torch.zeros((nz, ny, nx), dtype=torch.int32, device=DEV)
    count, target = 0, 0.05 * nx * ny * nz
    while count < target:
        e = [int(rng.integers(2, min(21, max(3, d // 4)))) for d in (nz, ny, nx)]
        o = [int(rng.integers(0, d - q + 1)) for d, q in zip((nz, ny, nx), e)]
        f[o[0]:o[0] + e[0], o[1]:o[1] + e[1], o[2]:o[2] + e[2]] = 1
        count += 0.9 * e[0] * e[1] * e[2]
    b = torch.randn(f.shape, generator=_gen(seed), device=DEV)
    fl = f == 0
    b = torch.where(fl, b - b[fl].double().mean().float(), torch.zeros_like(b)).contiguous()
    return f, b


def _divergence(case, seed):
    """What the network sees: right-hand sides like those of a flame (strong
    in a plume, weak elsewhere) and a solid mask."""
    nx, ny, nz, nb = case["nx"], case["ny"], case["nz"], case["nb"]
    g = _gen(seed)
    bs, fs = [], []
    for k in range(nb):
        n = _noise(g, (nz, ny, nx), 4.0)
        env = torch.exp(0.8 * _noise(g, (nz, ny, nx), 24.0))
        f = (_noise(g, (nz, ny, nx), 12.0) > 2.0).to(torch.int32)
        bs.append(torch.where(f == 1, torch.zeros_like(n), 50.0 * n * env))
        fs.append(f)
    return torch.stack(bs).contiguous(), torch.stack(fs).contiguous()


SOLVERS = {"vcycle": _abi.SOLVER_VCYCLE, "mgpcg": _abi.SOLVER_MGPCG,
           "mgpcg_bf16": _abi.SOLVER_MGPCG_BF16}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "render"):
        sc = _scene(case)
        if kind == "render":
            cx = 0.5 * case["nx"] * case["dx"]
            sc.render.width, sc.render.height = case["width"], case["height"]
            sc.render.mode = case["mode"]
            sc.render.camera, sc.render.target = [cx, 1.5, -6.0], [cx, 2.0, cx]
        sim = Sim(sc)
        _burning(case, sim, seed)
        if kind == "render":
            r = Renderer(sc, sim)
            return dict(kind=kind, sim=sim, renderer=r, spp=case["spp"],
                        frame=int(seed) % 1000)
        if case["solver"] != "vcycle":
            sim.set_solver(SOLVERS[case["solver"]], 1e-4, 100)
        return dict(kind=kind, sim=sim, n=case["substeps"],
                    dt=1.0 / FPS / max(1, round(6 * 0.02 / case["dx"])), views={})
    if kind in ("vcycles", "cg"):
        f, b = _boxes(case, seed)
        ps = PoissonSolver((case["nx"], case["ny"], case["nz"]), case["dx"], 0)
        torch.cuda.synchronize()
        ps.set_flags(f.data_ptr())
        mode = SOLVERS["vcycle" if kind == "vcycles" else case["mode"]]
        return dict(kind=kind, ps=ps, f=f, b=b, phi=torch.zeros_like(b), mode=mode,
                    tol=case.get("tol", 1e-3), iters=case.get("cycles", 200),
                    stream=torch.cuda.ExternalStream(ps.stream()))
    if kind in ("net", "grad"):
        b, f = _divergence(case, seed)
        net = Net.load(WEIGHTS)
        if kind == "grad":
            net.set_loss(0.0, 1.0)
        torch.cuda.synchronize()
        return dict(kind=kind, net=net, b=b, f=f, phi=torch.zeros_like(b),
                    dims=(case["nx"], case["ny"], case["nz"]), nb=case["nb"], h=case["dx"])
    g = _gen(seed)
    w, h = case["width"], case["height"]
    a = torch.exp(1.5 * _noise(g, (2, h, w), 12.0)[:1] - 3.0) * 16.0
    a = a * torch.exp(4.0 * (_noise(g, (2, h, w), 40.0)[:1] - 1.0)).clamp(max=40.0)
    acc = torch.empty((h * w, 4), device=DEV)
    for k, c in enumerate((1.0, 0.45, 0.15)):
        acc[:, k] = (c * a * (1.0 + 0.1 * torch.rand(a.shape, generator=g, device=DEV))).view(-1)
    acc[:, 3] = 16.0
    torch.cuda.synchronize()
    return dict(kind=kind, dev=Developer(w, h), cam=Camera(True, 0.0, 0.04), accum=acc)


# ------------------------------------------------------------------- run
def run(state):
    kind = state["kind"]
    if kind == "frame":
        sim, n = state["sim"], state["n"]
        for s in range(n):
            sim.step(state["dt"], s == n - 1)
        st = sim.read_stats()
        nx, ny, nz = sim.dims
        out = {"stats": st.raw}
        for name, f, shape in (("s0", _abi.F_S0, (nz, ny, nx, 4)),
                               ("s1", _abi.F_S1, (nz, ny, nx, 4)),
                               ("sol", _abi.F_SOL, (nz, ny, nx, 4)),
                               ("u", _abi.F_U, (nz + 1, ny + 1, nx + 1)),
                               ("v", _abi.F_V, (nz + 1, ny + 1, nx + 1)),
                               ("w", _abi.F_W, (nz + 1, ny + 1, nx + 1)),
                               ("phi", _abi.F_PHI, (nz, ny, nx))):
            p = sim.device_ptr(f)[0]
            if p not in state["views"]:
                state["views"][p] = torch.as_tensor(_Borrowed(p, shape, sim), device=DEV)
            out[name] = state["views"][p]
        return out
    if kind in ("vcycles", "cg"):
        with torch.cuda.stream(state["stream"]):
            state["phi"].zero_()
        state["ps"].solve(state["b"].data_ptr(), state["phi"].data_ptr(), state["mode"],
                          state["tol"], state["iters"], allow_cap=True)
        return state["phi"]
    if kind == "net":
        state["net"].forward(state["b"].data_ptr(), state["f"].data_ptr(), state["dims"],
                             state["nb"], state["h"], state["phi"].data_ptr(),
                             stream=torch.cuda.current_stream().cuda_stream)
        return state["phi"]
    if kind == "grad":
        loss, grad = state["net"].loss_grad(
            state["b"].data_ptr(), state["f"].data_ptr(), state["phi"].data_ptr(),
            state["dims"], state["nb"], state["h"],
            stream=torch.cuda.current_stream().cuda_stream)
        return {"loss": loss, "grad": grad}
    if kind == "render":
        state["renderer"].render_device(state["sim"], state["frame"], state["spp"])
        return state["renderer"].accum
    return state["dev"].develop(state["cam"], state["accum"].data_ptr(), 1.0 / FPS)


# ------------------------------------------------------------------ work
def work(case):
    kind = case["kind"]
    if kind == "develop":
        n = case["width"] * case["height"]
        # the image in, 8-bit RGB out; six box sums, curve and dither per value
        return dict(bytes=n * (16 + 3), flops=n * 3 * 80)
    cells = case["nx"] * case["ny"] * case["nz"] * case.get("nb", 1)
    if kind == "frame":
        # per substep: s0, s1, sol, velocities and pressure in and out, and
        # the surface terms out; stencils, traces, chemistry and the solve
        return dict(bytes=case["substeps"] * cells * 148, flops=case["substeps"] * cells * 3000)
    if kind == "vcycles":
        # flags, b and phi in, phi out; eight colour passes, residual and
        # transfers per cell and cycle over the level sum 8/7
        return dict(bytes=cells * 16, flops=case["cycles"] * cells * 90)
    if kind == "cg":
        its = 5 if case["tol"] > 1e-5 else 10
        return dict(bytes=cells * 16, flops=its * cells * 130)
    if kind in ("net", "grad"):
        per = sum(2.0 * 27 * ci * co / 8 ** lvl for ci, co, lvl, _ in SPEC)
        if kind == "net":
            return dict(bytes=cells * 12, flops=cells * per)
        return dict(bytes=cells * 8, flops=3 * cells * per)
    px = case["width"] * case["height"]
    # the fields in, the image out; a march of a few hundred samples a ray
    return dict(bytes=cells * 64 + px * 16, flops=px * case["spp"] * 20000)


# ----------------------------------------------------------------- exact
def _neigh(p):
    """Sum of the six neighbours with zeros outside, (z, y, x)."""
    s = torch.zeros_like(p)
    s[:, :, :-1] += p[:, :, 1:]
    s[:, :, 1:] += p[:, :, :-1]
    s[:, :-1] += p[:, 1:]
    s[:, 1:] += p[:, :-1]
    s[:-1] += p[1:]
    s[1:] += p[:-1]
    return s


def _counts(fluid):
    """Neighbours that count: fluid ones and the Dirichlet sides and top."""
    c = _neigh(fluid)
    c[:, :, 0] += 1
    c[:, :, -1] += 1
    c[:, -1] += 1
    c[0] += 1
    c[-1] += 1
    return c


class _Level:
    def __init__(self, solid, h):
        self.fluid = (~solid).double()
        self.solid, self.h2 = solid, h * h
        self.cnt = _counts(self.fluid)
        z, y, x = (torch.arange(n, device=DEV) for n in solid.shape)
        par = (x[None, None, :] + y[None, :, None] + z[:, None, None]) & 1
        ok = ~solid & (self.cnt >= 0.5)
        self.col = [ok & (par == c) for c in range(2)]
        self.den = self.cnt.clamp_min(0.5)

    def smooth(self, p, b, iters, om):
        for _ in range(iters):
            for c in range(2):
                q = (_neigh(p * self.fluid) - self.h2 * b) / self.den
                p = torch.where(self.col[c], p * (1.0 - om) + q * om, p)
        return p

    def resid(self, p, b):
        return (b - (_neigh(p * self.fluid) - self.cnt * p) / self.h2) * self.fluid


def _children(a):
    """Sums over 2x2x2 children (the dimensions padded to even)."""
    nz, ny, nx = a.shape
    a = F.pad(a, (0, nx & 1, 0, ny & 1, 0, nz & 1))
    nz, ny, nx = a.shape
    return a.view(nz // 2, 2, ny // 2, 2, nx // 2, 2).sum(dim=(1, 3, 5))


def _prolong(pc, fluid_c, shape):
    idx, wts = [], []
    for n, m in zip(shape, pc.shape):
        g = (torch.arange(n, device=DEV).double() + 0.5) * 0.5 - 0.5
        i0 = torch.floor(g)
        fr = g - i0
        idx.append([(i0.long() + o).clamp(0, m - 1) for o in (0, 1)])
        wts.append([1.0 - fr, fr])
    acc = torch.zeros(shape, dtype=torch.float64, device=DEV)
    ws = torch.zeros_like(acc)
    val = pc * fluid_c
    for k in range(8):
        o = (k >> 2 & 1, k >> 1 & 1, k & 1)
        w = (wts[0][o[0]][:, None, None] * wts[1][o[1]][None, :, None] *
             wts[2][o[2]][None, None, :])

        def at(a):
            return (a.index_select(0, idx[0][o[0]]).index_select(1, idx[1][o[1]])
                    .index_select(2, idx[2][o[2]]))

        acc += w * at(val)
        ws += w * at(fluid_c)
    return torch.where(ws > 1e-4, acc / ws.clamp_min(1e-4), torch.zeros_like(acc))


def _exact_vcycles(case, seed):
    f, b = _boxes(case, seed)
    lv, solid, h = [], f == 1, float(np.float32(case["dx"]))
    for _ in range(4):
        lv.append(_Level(solid, h))
        if min(solid.shape) < 16:
            break
        cnt = _children((~solid).double())
        solid, h = cnt == 0, 2.0 * h
    p = torch.zeros(f.shape, dtype=torch.float64, device=DEV)

    def cycle(l, p, b):
        if l == len(lv) - 1:
            return lv[l].smooth(p, b, 80, float(np.float32(1.6)))
        p = lv[l].smooth(p, b, 2, 1.0)
        n = _children(lv[l].fluid)
        bc = _children(lv[l].resid(p, b)) / n.clamp_min(1.0)
        pc = cycle(l + 1, torch.zeros_like(bc), bc)
        p = p + _prolong(pc, lv[l + 1].fluid, p.shape) * lv[l].fluid
        return lv[l].smooth(p, b, 2, 1.0)

    for _ in range(case["cycles"]):
        p = cycle(0, p, b.double())
    return p


def _exact_cg(case, seed):
    """A phi = b on the fluid cells connected to an open face, by Jacobi-PCG
    in 64 bits to 1e-11; the others keep the zero guess."""
    f, b = _boxes(case, seed)
    fluid = (f == 0).double()
    reach = torch.zeros_like(fluid)
    for s in ((slice(None), slice(None), 0), (slice(None), slice(None), -1),
              (slice(None), -1), (0,), (-1,)):
        reach[s] = fluid[s]
    n = -1.0
    while float(reach.sum()) != n:
        n = float(reach.sum())
        for _ in range(32):
            reach = ((reach + _neigh(reach)) > 0).double() * fluid
    cnt = _counts(reach)
    h2 = float(np.float32(case["dx"])) ** 2
    rhs = -b.double() * reach * h2
    dinv = reach / cnt.clamp_min(1.0)
    x = torch.zeros_like(rhs)
    r = rhs.clone()
    z = dinv * r
    p = z.clone()
    rz = (r * z).sum()
    stop = 1e-11 * float(rhs.norm())
    for it in range(6000):
        q = (cnt * p - _neigh(p)) * reach
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        if it % 25 == 24 and float(r.norm()) <= stop:
            break
        z = dinv * r
        rz, old = (r * z).sum(), rz
        p = z + (rz / old) * p
    return x


class _Conv(torch.autograd.Function):
    """3x3x3 convolution, padding 1, on (nb, z, y, x, c) in 64 bits with
    weights (co, 27, ci), tap by tap."""

    @staticmethod
    def forward(ctx, x, w, b):
        ctx.save_for_backward(x, w)
        nb, nz, ny, nx, c = x.shape
        xp = F.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        y = b.expand(nb * nz * ny * nx, -1).clone()
        for t in range(27):
            dz, dy, dx = t // 9, t // 3 % 3, t % 3
            s = xp[:, dz:dz + nz, dy:dy + ny, dx:dx + nx].reshape(-1, c)
            y.addmm_(s, w[:, t].t())
        return y.view(nb, nz, ny, nx, -1)

    @staticmethod
    def backward(ctx, g):
        x, w = ctx.saved_tensors
        nb, nz, ny, nx, c = x.shape
        xp = F.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        gp = torch.zeros_like(xp)
        gw = torch.zeros_like(w)
        gf = g.reshape(-1, g.shape[-1])
        for t in range(27):
            dz, dy, dx = t // 9, t // 3 % 3, t % 3
            sl = (slice(None), slice(dz, dz + nz), slice(dy, dy + ny), slice(dx, dx + nx))
            gw[:, t] = gf.t() @ xp[sl].reshape(-1, c)
            gp[sl] += (gf @ w[:, t]).view(nb, nz, ny, nx, c)
        return gp[:, 1:-1, 1:-1, 1:-1].contiguous(), gw, gf.sum(0)


def _pool(x):
    nz, ny, nx = x.shape[1:4]
    pad = (0, 0, 0, nx & 1, 0, ny & 1, 0, nz & 1)

    def s(a):
        a = F.pad(a, pad)
        nb, z, y, w, c = a.shape
        return a.view(nb, z // 2, 2, y // 2, 2, w // 2, 2, c).sum(dim=(2, 4, 6))

    return s(x) / s(torch.ones_like(x[:1, ..., :1]))


def _up(x, like):
    for d in (1, 2, 3):
        x = x.repeat_interleave(2, dim=d)
    return x[:, :like.shape[1], :like.shape[2], :like.shape[3]]


def _net64(params, b, f):
    """The network in 64 bits: output (nb, z, y, x), normalised b, rms."""
    ws, bs, o = [], [], 0
    for ci, co, _, _ in SPEC:
        ws.append(params[o:o + co * 27 * ci].view(co, 27, ci))
        o += co * 27 * ci
    for _, co, _, _ in SPEC:
        bs.append(params[o:o + co])
        o += co
    fluid = (f != 1).double()
    n = fluid.sum(dim=(1, 2, 3)).clamp_min(1.0)
    rms = ((b.double() ** 2 * fluid).sum(dim=(1, 2, 3)) / n).sqrt()
    bh = b.double() * fluid / rms.clamp_min(1e-300)[:, None, None, None]

    def conv(x, l):
        y = _Conv.apply(x, ws[l], bs[l])
        return y.relu() if SPEC[l][3] else y

    e0 = conv(conv(torch.stack([bh, 1.0 - fluid], -1), 0), 1)
    e1 = conv(conv(_pool(e0), 2), 3)
    e2 = conv(conv(_pool(e1), 4), 5)
    d1 = conv(torch.cat([_up(e2, e1), e1], -1), 6)
    d0 = conv(torch.cat([_up(d1, e0), e0], -1), 7)
    return conv(d0, 8)[..., 0], bh, rms, fluid


def _exact_net(case, seed):
    b, f = _divergence(case, seed)
    p, scale = Net.read_file(WEIGHTS)
    params = torch.from_numpy(p).to(DEV).double()
    grad = case["kind"] == "grad"
    params.requires_grad_(grad)
    h = float(np.float32(case["dx"]))
    with torch.set_grad_enabled(grad):
        out, bh, rms, fluid = _net64(params, b, f)
        if not grad:
            return out * scale * h * h * rms[:, None, None, None] * fluid
        # the mean squared normalised residual on the inner fluid cells
        lo = []
        for v in range(out.shape[0]):
            s = F.pad(out[v] * fluid[v], (1, 1, 1, 1, 1, 1))
            c = F.pad(fluid[v], (1, 1, 1, 1, 1, 1))

            def six(a):
                return (a[1:-1, 1:-1, 2:] + a[1:-1, 1:-1, :-2] + a[1:-1, 2:, 1:-1] +
                        a[1:-1, :-2, 1:-1] + a[2:, 1:-1, 1:-1] + a[:-2, 1:-1, 1:-1])

            lo.append(bh[v] - scale * (six(s) - six(c) * out[v]))
        inner = torch.zeros_like(fluid)
        inner[:, 1:-1, 1:-1, 1:-1] = fluid[:, 1:-1, 1:-1, 1:-1]
        loss = (torch.stack(lo) ** 2 * inner).sum() / inner.sum()
        loss.backward()
    return {"loss": loss.detach(), "grad": params.grad}


def exact(case, seed):
    """The outputs in 64 bits.  A whole substep and the Monte Carlo images
    have none: a restatement of the first is a second framework, and the
    samples of the second follow single-precision branch decisions.  The
    developed image is bytes."""
    if case["kind"] == "vcycles":
        return _exact_vcycles(case, seed)
    if case["kind"] == "cg":
        return _exact_cg(case, seed)
    if case["kind"] in ("net", "grad"):
        return _exact_net(case, seed)
    return None
