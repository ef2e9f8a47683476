"""The work this framework is used for, as cases that can be timed and compared.

A case is a dict of plain values; its "path" says which public entry points it goes through:

  stepper   ``Stepper``: a pack of meshblocks, its interiors loaded from a packed array (device,
            or pinned host memory), k full RK steps, the interiors stored, the clock read
  refined   ``amr.AmrStepper``: the same on a statically refined 2D mesh of uneven blocks
  ensemble  ``ensemble.EnsembleStepper``: independent problems stepped together
  driver    ``hydro.Driver``: the reference's kernel-by-kernel path (per pack or per meshblock)
  rollout   ``adjoint.Adjoint``: a fixed-dt rollout with checkpoints and its reverse sweep
  rollouts  ``adjoint.EnsembleAdjoint``: the same over an ensemble

``exact`` restates the scheme in plain torch FP64 on whole grids (no meshblocks): ConsToPrim,
donor cell / PLM / PPM, HLLE / HLLC / LHLLC, the RK stages, gravity, passive scalars, the CFL
policy, and for refined meshes one array per level with restriction, prolongation and flux
correction; torch.autograd differentiates it for the rollouts.
"""
import math
import random

import numpy as np
import torch

from apophis_gb300 import adjoint, amr, ensemble, hydro
from apophis_gb300.mesh import MeshConfig
from apophis_gb300.stepper import Stepper

GHOSTS = {"dc": 1, "plm": 2, "ppm": 3}
PERIODIC = ("periodic", "periodic")
# (gam0, gam1, beta) per stage of the low-storage integrators
STAGES = {"rk1": [(0.0, 1.0, 1.0)], "rk2": [(0.0, 1.0, 1.0), (0.5, 0.5, 0.5)],
          "rk3": [(0.0, 1.0, 1.0), (0.25, 0.75, 0.25), (2.0 / 3.0, 1.0 / 3.0, 2.0 / 3.0)],
          "vl2": [(0.0, 1.0, 0.5), (0.0, 1.0, 1.0)]}


def _uniform(path, flow, mesh, block, ng, recon, rsolver, integrator, steps, exact=True, **more):
    mesh, block = tuple(mesh) + (1,) * (3 - len(mesh)), tuple(block) + (1,) * (3 - len(block))
    c = {"path": path, "flow": flow, "ng": ng, "recon": recon, "rsolver": rsolver,
         "integrator": integrator, "steps": steps, "exact": exact, "scalars": 0, "host": False}
    for d in range(3):
        c["n%d" % (d + 1)], c["b%d" % (d + 1)] = mesh[d], block[d]
    c.update(more)
    return c


def listed():
    def named(name, c):
        return dict(c, name=name)

    return [
        # a one-dimensional shock tube in one small block, the regression suites' problem: a
        # step is a handful of launches and grid barriers, so latency decides
        named("sod1d", _uniform("stepper", "sod", (256,), (256,), 2, "plm", "hlle", "rk2", 16)),
        # the linear-wave convergence run (vl2 + plm + hllc): one 3D block, few cells per SM
        named("wave3d", _uniform("stepper", "wave", (64, 32, 32), (64, 32, 32), 2, "plm", "hllc", "vl2", 8)),
        # the headline workload: 3D Kelvin-Helmholtz, 64 blocks of 64^3, PPM + HLLC, in the
        # arithmetic that reproduces the reference's bits; a production run's step
        named("kh3d_256", _uniform("stepper", "kh", (256,) * 3, (64,) * 3, 4, "ppm", "hllc", "rk2", 1)),
        # a medium 3D run in the fast arithmetic whose state lives in pinned host memory
        # (a host code that loads it before and stores it after every call)
        named("kh3d_128_host", _uniform("stepper", "kh", (128,) * 3, (64,) * 3, 4, "ppm", "hllc", "rk2", 1,
                                        exact=False, host=True)),
        # odd block sides, three ghost layers, dyes, LHLLC and RK3: the shapes nobody tuned for
        named("kh3d_ragged", _uniform("stepper", "kh", (99, 70, 45), (33, 35, 45), 3, "ppm", "lhllc", "rk3", 1,
                                      scalars=2)),
        # 2D production grid of the differentiable configuration, forward only, fast arithmetic
        named("kh2d_512", _uniform("stepper", "kh", (512, 512), (64, 64), 2, "plm", "hlle", "rk2", 4, exact=False)),
        # the statically refined Rayleigh-Taylor pack: 1440 blocks of 32^2 and 16^2, gravity
        named("rt2d_refined", {"path": "refined", "n1": 256, "n2": 768, "block0": 32, "blockf": 16, "ng": 4,
                               "recon": "ppm", "rsolver": "hllc", "integrator": "rk2", "steps": 2, "exact": True}),
        # 64 independent blast waves on grids of 128^2 to 512^2, each with its own gas and clock
        named("blasts_64", {"path": "ensemble", "members": 64, "largest": 512, "block": 64, "ng": 4,
                            "recon": "ppm", "rsolver": "hllc", "integrator": "rk2", "steps": 1, "exact": True}),
        # the reference's own kernel granularity through the drop-in entry points, per pack
        named("driver_kh3d", _uniform("driver", "kh", (128,) * 3, (64,) * 3, 4, "ppm", "hllc", "rk2", 1,
                                      per_block=False)),
        # and per meshblock, as a host code that loops over its blocks: many small launches
        named("driver_rt2d_blocks", _uniform("driver", "rt", (64, 192), (32, 32), 4, "ppm", "hllc", "rk2", 1,
                                             per_block=True)),
        # gradient of a 2D rollout (PLM + HLLE, the differentiable configuration) with
        # checkpoints: forward, recomputation and reverse sweep
        named("rollout_kh2d", _uniform("rollout", "kh", (512, 512), (64, 64), 2, "plm", "hlle", "rk2", 4,
                                       exact=False, every=2)),
        # gradients of a few blast waves at once with PPM + HLLC
        named("rollouts_blast", {"path": "rollouts", "members": 8, "largest": 256, "block": 64, "ng": 4,
                                 "recon": "ppm", "rsolver": "hllc", "integrator": "rk2", "steps": 2, "every": 2,
                                 "exact": False}),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["stepper", "stepper", "stepper", "stepper", "refined", "ensemble", "driver", "driver",
                       "rollout", "rollouts"])
    recon = rng.choice(["ppm", "ppm", "ppm", "plm", "plm", "dc"])
    ng = rng.choice([g for g in (1, 2, 3, 4) if g >= GHOSTS[recon] and (g > 1 or recon == "dc")])
    rsolver = rng.choice(["hllc", "hllc", "hllc", "hlle", "lhllc"])
    integrator = rng.choice(["rk2", "rk2", "rk2", "vl2", "rk3"] + ["rk1"] * (recon == "dc"))
    common = {"recon": recon, "ng": ng, "rsolver": rsolver, "integrator": integrator}
    if path in ("stepper", "driver"):
        ndim = rng.choice([1, 2, 2, 3, 3, 3])
        most = {1: 8192, 2: 1 << 20, 3: 1 << 22}[ndim] >> (2 if path == "driver" else 0)
        while True:
            block = [_log_int(rng, *{1: (32, 400), 2: (12, 128), 3: (10, 72)}[ndim]) for _ in range(ndim)]
            mesh = [b * _log_int(rng, 1, 8) for b in block]
            if math.prod(mesh) <= most:
                break
        flow = rng.choice({1: ["sod"], 2: ["kh", "kh", "rt", "blast"], 3: ["kh", "kh", "wave"]}[ndim])
        steps = max(1, min(16, (1 << 20) // math.prod(mesh))) if path == "stepper" else 1
        more = {"scalars": rng.choice([0, 0, 0, 1, 2, 3])}
        if path == "driver":
            more["per_block"] = math.prod(m // b for m, b in zip(mesh, block)) <= 16 and rng.random() < 0.5
        else:
            more["host"] = rng.random() < 0.25
        return _uniform(path, flow, mesh, block, steps=steps, exact=rng.random() < 0.7, **common, **more)
    if path == "refined":
        n1 = 32 * rng.randint(2, 8)
        return dict(common, path=path, n1=n1, n2=3 * n1, block0=32, blockf=16,
                    steps=rng.randint(1, 4), exact=rng.random() < 0.7)
    if path == "ensemble":
        return dict(common, path=path, members=_log_int(rng, 2, 64), largest=64 * rng.randint(2, 8),
                    block=64 // rng.choice([1, 2]), steps=1, exact=rng.random() < 0.7)
    common["rsolver"] = rng.choice(["hllc", "hlle"])
    steps = rng.randint(1, 4)
    if path == "rollout":
        block = _log_int(rng, 16, 64)
        return _uniform(path, "kh", (block * rng.randint(2, 8), block * rng.randint(2, 8)), (block, block),
                        steps=steps, exact=False, every=rng.randint(1, steps), **common)
    return dict(common, path=path, members=rng.randint(2, 8), largest=32 * rng.randint(2, 8), block=32,
                steps=steps, every=rng.randint(1, steps), exact=False)


# ---- inputs ---------------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _noise(gen, shape):
    return 2.0 * torch.rand(shape, generator=gen, dtype=torch.float64, device=gen.device) - 1.0


def _generator(seed):
    return torch.Generator(_device()).manual_seed(1_000_003 * int(seed) + 17)


def _cons(rho, vx, vy, vz, p, gm1, dyes=()):
    rho, vx, vy, vz, p = torch.broadcast_tensors(rho, vx, vy, vz, p)
    e = p / gm1 + 0.5 * rho * (vx * vx + vy * vy + vz * vz)
    return torch.stack([rho, rho * vx, rho * vy, rho * vz, e] + [rho * s for s in dyes])


def _mesh(case):
    """The MeshConfig of a uniform case."""
    flow = case["flow"]
    nx = tuple(case["n%d" % d] for d in (1, 2, 3))
    ndim = 3 if nx[2] > 1 else 2 if nx[1] > 1 else 1
    kw = {"sod": dict(bc=(("outflow", "outflow"), PERIODIC, PERIODIC), gamma=1.4, cfl=0.4),
          "kh": dict(gamma=5.0 / 3.0, cfl=0.3), "blast": dict(gamma=1.4, cfl=0.3),
          "wave": dict(gamma=5.0 / 3.0, cfl=0.3),
          "rt": dict(xmax=(0.5, 1.5, 1.0), bc=(PERIODIC, ("reflecting", "reflecting"), PERIODIC),
                     gravity=(0.0, -0.1, 0.0), gamma=1.4, cfl=0.4)}[flow]
    return MeshConfig(ndim=ndim, mesh_nx=nx, block_nx=tuple(case["b%d" % d] for d in (1, 2, 3)), ng=case["ng"],
                      recon=case["recon"], rsolver=case["rsolver"], integrator=case["integrator"],
                      nscalars=case["scalars"], name="perf_" + flow, **kw)


def _grid(cfg):
    ax = [(torch.arange(n, dtype=torch.float64, device=_device()) + 0.5) * dx for n, dx in zip(cfg.mesh_nx, cfg.dx)]
    return ax[0].view(1, 1, -1), ax[1].view(1, -1, 1), ax[2].view(-1, 1, 1)


def _state(case, cfg, seed):
    """The conserved state (nvar, nz, ny, nx) on the whole mesh."""
    x, y, z = _grid(cfg)
    gen = _generator(seed)
    shape = cfg.mesh_nx[::-1]
    w = _noise(gen, (8,)).tolist()
    zero = torch.zeros(shape, dtype=torch.float64, device=x.device)
    two_pi = 2.0 * math.pi
    if case["flow"] == "sod":  # diaphragm near the middle, states a few per cent around Sod's
        left = x < 0.5 + 0.05 * w[0]
        rho = torch.where(left, 1.0 + 0.05 * w[1], 0.125 * (1.0 + 0.05 * w[2])) + zero
        vx, vy, vz = zero, zero, zero
        p = torch.where(left, 1.0 + 0.05 * w[3], 0.1 * (1.0 + 0.05 * w[4])) + zero
    elif case["flow"] == "wave":  # a small sound wave across the box
        s = 1e-6 * torch.sin(two_pi * (x + y + z) + 3.0 * w[0])
        rho, p = 1.0 + s, (1.0 + cfg.gamma * s) / cfg.gamma
        vx, vy, vz = s / math.sqrt(3.0), s / math.sqrt(3.0), s / math.sqrt(3.0)
    elif case["flow"] == "blast":
        rho, vx, vy, vz, p = _blast(x, y, zero, 0.2 + 0.1 * w[0], gen)
    elif case["flow"] == "rt":  # heavy over light fluid, hydrostatic, perturbed at the interface
        xc, yc = x - 0.25, y - 0.75
        rho = torch.where(yc < 0.0, 1.0, 2.0) + 0.01 * _noise(gen, shape)
        vy = 0.01 * (1.0 + torch.cos(4 * math.pi * xc + w[0])) * (1.0 + torch.cos(3 * math.pi * yc)) / 4.0 + zero
        vx, vz = 1e-3 * _noise(gen, shape), zero
        p = 1.0 / cfg.gamma - 0.1 * torch.where(yc < 0.0, 1.0, 2.0) * yc + zero
    else:  # Kelvin-Helmholtz: a dense band moving against its surroundings, noise in the velocities
        band = (y - 0.5).abs() < 0.25
        rho = torch.where(band, 2.0, 1.0) + 0.02 * torch.cos(two_pi * (x + y + z) + w[1]) + zero
        vx = torch.where(band, 0.5, -0.5) + 1e-3 * _noise(gen, shape)
        vy = 0.01 * torch.sin(4.0 * math.pi * x + w[0]) + 1e-3 * _noise(gen, shape)
        vz = 1e-3 * _noise(gen, shape) if cfg.ndim == 3 else zero
        p = 2.5 + 0.05 * torch.cos(two_pi * (x - 2.0 * y + z) + w[2]) + zero
    q = y if cfg.ndim >= 2 else x
    dyes = [0.5 * (torch.tanh((q - 0.25) / 0.05) - torch.tanh((q - 0.75) / 0.05)) + zero,
            0.5 + 0.25 * torch.sin(two_pi * x + w[3]) * torch.cos(two_pi * y) * torch.cos(two_pi * z)]
    return _cons(rho, vx, vy, vz, p, cfg.gm1, [dyes[k % 2] for k in range(cfg.nscalars)])


def _blast(x, y, zero, r0, gen):
    """A blast some way out: hot expanding gas inside r0 of the centre of the unit square, a
    slightly uneven ambient gas outside."""
    r = torch.sqrt((x - 0.5) ** 2 + (y - 0.5) ** 2) + zero
    hot = r < r0
    rho = torch.where(hot, 0.3 + 1.5 * (r / r0) ** 4, 1.0) + 0.02 * _noise(gen, zero.shape)
    v = torch.where(hot, 1.5 / r0, 0.0)
    p = torch.where(hot, 3.0, 0.1) * (1.0 + 0.02 * torch.cos(9.0 * (x + 2.0 * y)))
    return rho, v * (x - 0.5), v * (y - 0.5), zero, p


def _to_blocks(u, cfg):
    """(nvar, nz, ny, nx) -> packed interiors (nblocks, nvar, b3, b2, b1), blocks x-fastest."""
    b, nb, nv = cfg.block_nx, cfg.blocks_per_dim, u.shape[0]
    v = u.reshape(nv, nb[2], b[2], nb[1], b[1], nb[0], b[0]).permute(1, 3, 5, 0, 2, 4, 6)
    return v.reshape(cfg.nblocks, nv, b[2], b[1], b[0]).contiguous()


def _with_ghosts(blocks, cfg):
    out = torch.zeros(cfg.pack_shape(blocks.shape[1]), dtype=torch.float64, device=blocks.device)
    sk, sj, si = cfg.interior
    out[:, :, sk, sj, si] = blocks
    return out


def _members(case, seed):
    """The ensemble's meshes (sizes by the case alone) and the members' states."""
    sizes = random.Random(case["members"] * 1009 + case["largest"])
    r = random.Random(int(seed))
    gen = _generator(seed)
    cfgs, states = [], []
    for m in range(case["members"]):
        n = case["block"] * sizes.randint(max(1, case["largest"] // case["block"] // 4),
                                          case["largest"] // case["block"])
        cfg = MeshConfig(ndim=2, mesh_nx=(n, n, 1), block_nx=(case["block"], case["block"], 1), ng=case["ng"],
                         recon=case["recon"], rsolver=case["rsolver"], integrator=case["integrator"],
                         gamma=r.uniform(1.4, 5.0 / 3.0), cfl=0.3, name="perf_blast_m%d" % m)
        x, y, _ = _grid(cfg)
        zero = torch.zeros((1, n, n), dtype=torch.float64, device=x.device)
        cfgs.append(cfg)
        states.append(_cons(*_blast(x, y, zero, r.uniform(0.15, 0.35), gen), cfg.gm1))
    return cfgs, states


def _refined(case, seed):
    """The refined mesh and its state, block after block (packed interiors, flat)."""
    cfg, _ = amr.rt2d_amr(nx=case["n1"], ny=case["n2"], block0=case["block0"], blockf=case["blockf"],
                          ng=case["ng"], recon=case["recon"], rsolver=case["rsolver"], integrator=case["integrator"])
    xs, ys = zip(*(cfg.cell_centers(b) for b in range(cfg.nblocks)))
    x, y = (torch.from_numpy(np.concatenate([a.reshape(-1) for a in v])).to(_device()) for v in (xs, ys))
    gen = _generator(seed)
    w = _noise(gen, (2,)).tolist()
    xc, yc = x - 0.25, y - 0.75
    rho = torch.where(yc < 0.0, 1.0, 2.0)
    p = 1.0 / cfg.gamma - 0.1 * rho * yc
    vy = 0.01 * (1.0 + torch.cos(4 * math.pi * xc + w[0])) * (1.0 + torch.cos(3 * math.pi * yc)) / 4.0
    vx = 1e-3 * _noise(gen, x.shape)
    u = _cons(rho + 0.01 * _noise(gen, x.shape), vx, vy, torch.zeros_like(x), p, cfg.gm1)
    parts, at = [], 0
    for B in cfg.blocks:
        n = B.nx[0] * B.nx[1]
        parts.append(u[:, at:at + n].reshape(-1))
        at += n
    return cfg, torch.cat(parts)


def _max_dt(cfgs, states):
    """A common dt for a fixed schedule: 0.8 of the members' smallest CFL estimate."""
    return [0.8 * float(_estimate(s, c.dx, c.ndim, c.gm1, c.cfl)) for c, s in zip(cfgs, states)]


def prepare(case, seed):
    path, s = case["path"], {"case": case}
    if path == "refined":
        cfg, packed = _refined(case, seed)
        host, flat, at = packed.cpu().numpy(), np.zeros(cfg.flat_size()), 0
        for b, B in enumerate(cfg.blocks):
            n, g = 5 * B.nx[0] * B.nx[1], cfg.ng
            cfg.block_view(flat, b)[:, 0, g:-g, g:-g] = host[at:at + n].reshape(5, B.nx[1], B.nx[0])
            at += n
        s.update(stepper=amr.AmrStepper(cfg, flat, exact=case["exact"]), src=packed, dst=torch.empty_like(packed))
        return s
    if path in ("ensemble", "rollouts"):
        cfgs, states = _members(case, seed)
        ens = ensemble.Ensemble(cfgs, [1e9] * len(cfgs))  # no end time in reach
        blocks = [_to_blocks(u, c) for u, c in zip(states, cfgs)]
        flat = ens.pack([_with_ghosts(b, c).cpu().numpy() for b, c in zip(blocks, cfgs)])
        if path == "ensemble":
            src = torch.cat([b.reshape(-1) for b in blocks])
            s.update(stepper=ensemble.EnsembleStepper(ens, flat, exact=case["exact"]), src=src,
                     dst=torch.empty_like(src))
            return s
        lam = [_with_ghosts(b, c).reshape(-1) for b, c in zip(_directions(cfgs, seed), cfgs)]
        s.update(adjoint=adjoint.EnsembleAdjoint(ens), u0=torch.from_numpy(flat).to("cuda"), lam=torch.cat(lam),
                 dts=[_max_dt(cfgs, states)] * case["steps"], ng=case["ng"],
                 view=(ens.nblocks, 5, 1, case["block"] + 2 * case["ng"], case["block"] + 2 * case["ng"]))
        return s
    cfg = _mesh(case)
    u = _state(case, cfg, seed)
    blocks = _to_blocks(u, cfg)
    pack = _with_ghosts(blocks, cfg)
    if path == "driver":
        s["driver"] = hydro.Driver(cfg, pack.cpu().numpy(), exact=case["exact"], per_block=case["per_block"])
        return s
    if path == "rollout":
        s.update(adjoint=adjoint.Adjoint(cfg), u0=pack, lam=_with_ghosts(_directions([cfg], seed)[0], cfg),
                 dts=_max_dt([cfg], [u]) * case["steps"], ng=case["ng"], view=cfg.pack_shape(5))
        return s
    s.update(stepper=Stepper(cfg, cons=pack, exact=case["exact"]), src=blocks, dst=torch.empty_like(blocks))
    if case["host"]:
        s.update(src=blocks.cpu().pin_memory(), dst=torch.empty(blocks.shape, dtype=torch.float64).pin_memory())
    return s


def _directions(cfgs, seed):
    """The adjoint of a rollout's final state: what a loss would hand to the reverse sweep."""
    gen = _generator(int(seed) + 500_009)
    return [_to_blocks(torch.randn((5, 1) + c.mesh_nx[1::-1], generator=gen, dtype=torch.float64, device=gen.device), c)
            for c in cfgs]


# ---- one pass -------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    if "stepper" in state:  # load the interiors, step, store them, read the clock
        st = state["stepper"]
        st.load_interiors(state["src"])
        st.step(case["steps"])
        st.store_interiors(state["dst"])
        clock = st.member_status() if case["path"] == "ensemble" else st.status()
        out = {"state": state["dst"]}
        for k in ("time", "dt", "ncycle"):
            v = clock[k]
            out[k] = torch.tensor(v, dtype=torch.int64 if k == "ncycle" else torch.float64) if isinstance(v, list) else v
        return out
    if "driver" in state:
        d = state["driver"]
        d.run(nsteps=case["steps"])
        return {"cons": d.md.cons, "time": d.time, "dt": d.dt, "ncycle": d.ncycle}
    A, g = state["adjoint"], state["ng"]
    if case["path"] == "rollouts":
        u = A.forward_members(state["u0"], state["dts"], checkpoint_every=case["every"])
    else:
        u = A.forward(state["u0"], state["dts"], checkpoint_every=case["every"])
    lam = A.backward(state["lam"])
    # ghost cells of the final state are scratch: its interior is the output
    return {"state": u.view(state["view"])[:, :, 0, g:-g, g:-g], "gradient": lam}


# ---- what a pass cannot do without ----------------------------------------------------------
def _zones(case):
    if case["path"] in ("ensemble", "rollouts"):
        sizes = random.Random(case["members"] * 1009 + case["largest"])
        k = case["largest"] // case["block"]
        return sum((case["block"] * sizes.randint(max(1, k // 4), k)) ** 2 for _ in range(case["members"]))
    if case["path"] == "refined":
        cfg, _ = amr.rt2d_amr(nx=case["n1"], ny=case["n2"], block0=case["block0"], blockf=case["blockf"])
        return cfg.zones()
    return case["n1"] * case["n2"] * case["n3"]


def work(case):
    """The state read once and written once (for a rollout also the adjoint), and the
    arithmetic of the scheme: per zone, stage and direction the reconstruction of each variable,
    one Riemann solve and the flux differences; per stage ConsToPrim and the update.  A reverse
    step counts twice the forward's arithmetic on top of the forward."""
    ndim = 2 if case["path"] in ("ensemble", "rollouts", "refined") else \
        3 if case["n3"] > 1 else 2 if case["n2"] > 1 else 1
    nv, zones = 5 + case.get("scalars", 0), _zones(case)
    recon = {"dc": 0, "plm": 7, "ppm": 45}[case["recon"]]
    riemann = {"hlle": 85, "hllc": 105, "lhllc": 120}[case["rsolver"]]
    stage = ndim * (recon * nv + riemann + 3 * nv) + 25 + 6 * nv
    flops = zones * stage * len(STAGES[case["integrator"]]) * case["steps"]
    size = 8.0 * nv * zones
    if case["path"] in ("rollout", "rollouts"):
        return {"bytes": 4 * size, "flops": 3.0 * flops}
    return {"bytes": 2 * size, "flops": float(flops)}


# ---- the scheme in plain torch --------------------------------------------------------------
C2 = 2.99792458e10 ** 2


def _primitives(u, gm1):
    rho = u[0]
    v = [u[k] / rho for k in (1, 2, 3)]
    e_k = 0.5 * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) / rho
    return [rho] + v + [gm1 * (u[4] - e_k)] + [u[k] / rho for k in range(5, u.shape[0])]


def _estimate(u, dx, ndim, gm1, cfl, where=None):
    w = _primitives(u, gm1)
    lam = torch.sqrt(C2 * (gm1 + 1.0) / (1.0 + (w[4] / (gm1 * w[0]) + C2) * w[0] / w[4]))
    m = None
    for d in range(ndim):
        c = dx[d] / (w[1 + d].abs() + lam)
        m = c if m is None else torch.minimum(m, c)
    return cfl * (m if where is None else m[where]).min()


def _pad(u, axis, g, bc):
    """g ghost cells on both sides of axis of (nvar, nz, ny, nx), boundaries bc = (low, high)."""
    n, normal = u.shape[axis], 4 - axis  # the momentum along the axis

    def ghost(side):
        if bc[side] == "periodic":
            return u.narrow(axis, n - g if side == 0 else 0, g)
        if bc[side] == "outflow":
            return torch.cat([u.narrow(axis, 0 if side == 0 else n - 1, 1)] * g, axis)
        v = u.narrow(axis, 0 if side == 0 else n - g, g).flip(axis)
        return torch.cat([v[:normal], -v[normal:normal + 1], v[normal + 1:]])

    return torch.cat([ghost(0), u, ghost(1)], axis)


def _ppm_faces(q, ax):
    """Left and right states of faces 0..n from n + 6 cells along ax."""
    n = q.shape[ax] - 6

    def cells(lo, count, a=q):  # a's entries from cell lo on, a starting at cell -3
        return a.narrow(ax, lo + 3, count)

    m, c, p = cells(-3, n + 4), cells(-2, n + 4), cells(-1, n + 4)
    slope, curve = 0.5 * (p - m), (m + p) - 2.0 * c
    at = lambda a, lo, count: a.narrow(ax, lo + 2, count)  # noqa: E731  (a starting at cell -2)
    a, b = cells(-2, n + 3), cells(-1, n + 3)  # the cells on both sides of faces -1..n+1
    ca, cb = at(curve, -2, n + 3), at(curve, -1, n + 3)
    mean = 0.5 * (a + b)
    face = mean + (at(slope, -2, n + 3) - at(slope, -1, n + 3)) / 6.0
    bend = 3.0 * (a + b - 2.0 * face)
    same = ((bend < 0) == (ca < 0)) & ((bend < 0) == (cb < 0))
    small = torch.minimum(1.25 * torch.minimum(ca.abs(), cb.abs()), bend.abs())
    small = torch.where(same, torch.where(bend < 0, -small, small), torch.zeros_like(small))
    face = torch.where((face - a) * (b - face) < 0, mean - small / 6.0, face)
    lo, hi = face.narrow(ax, 0, n + 2), face.narrow(ax, 1, n + 2)
    m2, m1, c, p1, p2 = (cells(k, n + 2) for k in (-3, -2, -1, 0, 1))
    k1, k0, k2 = (at(curve, k, n + 2) for k in (-2, -1, 0))
    d2 = 6.0 * (lo + hi - 2.0 * c)
    down, up = c - lo, hi - c
    extremum = ~(down * up > 0) | ~((p1 - c) * (c - m1) > 0)
    same = ((d2 < 0) == (k1 < 0)) & ((d2 < 0) == (k0 < 0)) & ((d2 < 0) == (k2 < 0))
    small = torch.minimum(1.25 * torch.minimum(torch.minimum(k1.abs(), k0.abs()), k2.abs()), d2.abs())
    small = torch.where(same, torch.where(d2 < 0, -small, small), torch.zeros_like(small))
    top = torch.stack([m2.abs(), m1.abs(), c.abs(), p1.abs(), p2.abs()]).amax(0)
    large = d2.abs() > 1e-12 * top
    rho = torch.where(large, small / torch.where(large, d2, torch.ones_like(d2)), torch.zeros_like(d2))
    cut = rho <= 1.0 - 1e-12
    right = torch.where(extremum, torch.where(cut, c - rho * down, lo),
                        torch.where(down.abs() >= 2.0 * up.abs(), c - 2.0 * up, lo))
    left = torch.where(extremum, torch.where(cut, c + rho * up, hi),
                       torch.where(up.abs() >= 2.0 * down.abs(), c + 2.0 * down, hi))
    return left.narrow(ax, 0, n + 1), right.narrow(ax, 1, n + 1)


def _faces(q, ax, recon):
    """Left and right states of faces 0..n of q, which holds GHOSTS[recon] ghost cells along ax."""
    if recon == "ppm":
        return _ppm_faces(q, ax)
    n = q.shape[ax] - 2 * GHOSTS[recon]
    if recon == "dc":
        return q.narrow(ax, 0, n + 1), q.narrow(ax, 1, n + 1)
    m, c, p = (q.narrow(ax, k, n + 2) for k in (0, 1, 2))
    a, b = c - m, p - c
    rising = a * b > 0
    d = torch.where(rising, a * b / torch.where(rising, a + b, torch.ones_like(a)), torch.zeros_like(a))
    return (c + d).narrow(ax, 0, n + 1), (c - d).narrow(ax, 1, n + 1)


def _riemann(solver, wl, wr, gm1):
    """Fluxes (mass, normal, two transverse momenta, energy) of states (rho, vn, vt1, vt2, p)."""
    gamma = gm1 + 1.0
    (rl, ul, pl), (rr, ur, pr) = (wl[0], wl[1], wl[4]), (wr[0], wr[1], wr[4])

    def sound(r, p):
        return torch.sqrt(C2 * gamma * p / (p * (1.0 + 1.0 / gm1) + r * C2))

    def fluxes(w, b):
        r, u, v, z, p = w
        e = p / gm1 + 0.5 * r * (u * u + v * v + z * z)
        s = u - b
        return [r * s, r * u * s + p, r * v * s, r * z * s, e * s + p * u]

    one = torch.ones_like(pl)
    cl, cr = sound(rl, pl), sound(rr, pr)
    mid = 0.5 * (pl + pr) - 0.5 * (ur - ul) * (0.5 * (rl + rr)) * (0.5 * (cl + cr)) * one
    if solver == "hlle":
        k = (gamma + 1.0) / math.sqrt(2.0 * gamma)
        sl = ul - cl * torch.where(mid > pl, 1.0 + k * (mid / pl - 1.0), one)
        sr = ur + cr * torch.where(mid > pr, 1.0 + k * (mid / pr - 1.0), one)
        bp, bm = sr.clamp_min(0.0), sl.clamp_max(0.0)
        fl, fr = fluxes(wl, bm), fluxes(wr, bp)
        moves = (bp != 0) | (bm != 0)
        t = torch.where(moves, 0.5 * (bp + bm) / torch.where(moves, bp - bm, one), torch.zeros_like(bp))
        return [0.5 * (a + b) + (a - b) * t for a, b in zip(fl, fr)]
    if solver == "lhllc":
        speed = [torch.sqrt(w[1] * w[1] + w[2] * w[2] + w[3] * w[3]) for w in (wl, wr)]
        chi = torch.maximum(*speed)
        mid = 0.5 * (pl + pr) - 0.5 * (ur - ul) * (0.5 * (rl + rr)) * (0.5 * (cl + cr)) * (chi * (2.0 - chi))
    k = (gamma + 1.0) / (2.0 * gamma)
    sl = ul - cl * torch.sqrt(torch.where(mid > pl, 1.0 + k * (mid / pl - 1.0), one))
    sr = ur + cr * torch.sqrt(torch.where(mid > pr, 1.0 + k * (mid / pr - 1.0), one))
    bp, bm = torch.where(sr > 0, sr, 1e-20 * one), torch.where(sl < 0, sl, -1e-20 * one)
    tl, tr = pl + (ul - sl) * rl * ul, pr + (ur - sr) * rr * ur
    ml, mr = rl * (ul - sl), -(rr * (ur - sr))
    star, cp = (tl - tr) / (ml + mr), (ml * tr + mr * tl) / (ml + mr)
    cp = torch.where(cp > 0, cp, torch.zeros_like(cp))
    right = star >= 0  # the contact moves right: the left state is upwind
    edge = torch.where(right, bm, bp)
    share = star / torch.where(right, star - bm, star - bp)
    push = -edge / torch.where(right, star - bm, star - bp)
    f = [share * torch.where(right, a, b) for a, b in zip(fluxes(wl, bm), fluxes(wr, bp))]
    f[1] = f[1] + push * cp
    f[4] = f[4] + push * cp * star
    return f


def _sweep(u, d, bc, recon, solver, gm1):
    """Fluxes (nvar, ..) through faces 0..n along dimension d of the cells u, which hold
    GHOSTS[recon] ghost cells along it when bc is None."""
    ax = 3 - d
    if bc is not None:
        u = _pad(u, ax, GHOSTS[recon], bc)
    states = [_faces(q, ax - 1, recon) for q in _primitives(u, gm1)]
    order = [0, 1 + d, 1 + (d + 1) % 3, 1 + (d + 2) % 3, 4]
    f = _riemann(solver, [states[k][0] for k in order], [states[k][1] for k in order], gm1)
    out = [None] * 5
    for k, x in zip(order, f):
        out[k] = x
    return torch.stack(out + [out[0] * torch.where(out[0] >= 0, l, r) for l, r in states[5:]])


def _kick(new, u, gravity, beta_dt, gm1):
    """The constant-gravity source of a stage from the stage's input state u."""
    if gravity is None:
        return new
    rho, mom = u[0], sum(g * u[1 + k] / u[0] for k, g in enumerate(gravity))
    add = [torch.zeros_like(rho)] + [g * rho * beta_dt for g in gravity] + [mom * rho * beta_dt]
    return new + torch.stack(add + [torch.zeros_like(rho)] * (u.shape[0] - 5))


def _step(u, cfg, dt):
    """One RK step of the whole uniform mesh."""
    start, vl2 = u, cfg.integrator == "vl2"
    for i, (g0, g1, beta) in enumerate(STAGES[cfg.integrator]):
        recon = "dc" if vl2 and i == 0 else cfg.recon
        rate = torch.zeros_like(u)
        for d in range(cfg.ndim):
            f = _sweep(u, d, cfg.bc[d], recon, cfg.rsolver, cfg.gm1)
            n = u.shape[3 - d]
            rate = rate - (f.narrow(3 - d, 1, n) - f.narrow(3 - d, 0, n)) / cfg.dx[d]
        u = _kick(g0 * u + g1 * start + beta * dt * rate, u, cfg.gravity, beta * dt, cfg.gm1)
    return u


def _advance(u, cfg, steps):
    """(state, time, next dt) after CFL steps."""
    t, dt = 0.0, float(_estimate(u, cfg.dx, cfg.ndim, cfg.gm1, cfg.cfl))
    for _ in range(steps):
        u = _step(u, cfg, dt)
        t, dt = t + dt, min(2.0 * dt, float(_estimate(u, cfg.dx, cfg.ndim, cfg.gm1, cfg.cfl)))
    return u, t, dt


class _Levels:
    """A refined mesh as one array per level: leaf cells, the cells on the transverse edges of
    their blocks, and the packed position of every leaf cell."""

    def __init__(self, cfg):
        self.cfg, levels = cfg, max(B.level for B in cfg.blocks) + 1
        shapes = [(cfg.base_nx[1] << k, cfg.base_nx[0] << k) for k in range(levels)]
        at = [np.full(s, -1, np.int64) for s in shapes]
        edge = [[np.zeros(s, bool) for s in shapes] for _ in range(2)]  # of the block along x, y
        off = 0
        for B in cfg.blocks:
            j, i = (slice(B.origin[k], B.origin[k] + B.nx[k]) for k in (1, 0))
            n = B.nx[0] * B.nx[1]
            at[B.level][j, i] = np.arange(off, off + n).reshape(B.nx[1], B.nx[0])
            e = np.zeros((B.nx[1], B.nx[0]), bool)
            e[:, 0] = e[:, -1] = True
            edge[0][B.level][j, i] = e
            e = np.zeros((B.nx[1], B.nx[0]), bool)
            e[0] = e[-1] = True
            edge[1][B.level][j, i] = e
            off += n
        to = lambda a: torch.from_numpy(a).to(_device())  # noqa: E731
        self.at, self.edge = [to(a) for a in at], [[to(a) for a in v] for v in edge]
        self.leaf = [a >= 0 for a in self.at]
        self.dx = [tuple((cfg.xmax[d] - cfg.xmin[d]) / cfg.base_nx[d] / 2 ** k for d in range(2)) + (1.0,)
                   for k in range(levels)]
        # cells under four leaf cells of the next level
        self.under = [self._quads(self.leaf[k + 1]).all(0) if k + 1 < levels else torch.zeros_like(self.leaf[k])
                      for k in range(levels)]

    @staticmethod
    def _quads(a):
        return torch.stack([a[..., j::2, i::2] for j in (0, 1) for i in (0, 1)])

    def spread(self, cells):
        """(5, cells) in packed order -> one (5, 1, ny, nx) array per level (1 outside leaves)."""
        return [torch.where(m, cells[:, a.clamp_min(0)], torch.ones((), dtype=torch.float64, device=m.device))[:, None]
                for a, m in zip(self.at, self.leaf)]

    def gather(self, levels):
        out = torch.empty((5, sum(int(m.sum()) for m in self.leaf)), dtype=torch.float64, device=levels[0].device)
        for u, a, m in zip(levels, self.at, self.leaf):
            out[:, a[m]] = u[:, 0][:, m]
        return out

    def filled(self, levels, d):
        """Every level's cells with those across coarse-fine faces along d filled in."""
        ax = 3 - d
        means = [self._quads(levels[k + 1]).mean(0) if k + 1 < len(levels) else levels[k] for k in range(len(levels))]
        out = []
        for k, u in enumerate(levels):
            v = torch.where(self.leaf[k], u, torch.where(self.under[k], means[k], u))
            if k > 0:
                c = torch.where(self.leaf[k - 1], levels[k - 1],
                                torch.where(self.under[k - 1], means[k - 1], levels[k - 1]))

                def slope(axis):
                    a, b = c - c.roll(1, axis), c.roll(-1, axis) - c
                    return torch.where(a * b > 0, torch.where(a.abs() < b.abs(), a, b), torch.zeros_like(a))

                sx, sy = slope(3), slope(2)
                if d == 0:
                    sy = torch.where(self.edge[1][k - 1], torch.zeros_like(sy), sy)
                else:
                    sx = torch.where(self.edge[0][k - 1], torch.zeros_like(sx), sx)
                fine = torch.empty_like(u)
                for j in (0, 1):
                    for i in (0, 1):
                        fine[..., j::2, i::2] = c + (0.25 if i else -0.25) * sx + (0.25 if j else -0.25) * sy
                v = torch.where(self.leaf[k] | self.under[k], v, fine)
            out.append(_pad(v, ax, 3, self.cfg.bc[d]))
        return out

    def rates(self, levels, recon):
        cfg, rate = self.cfg, [torch.zeros_like(u) for u in levels]
        for d in range(2):
            ax = 3 - d
            full = self.filled(levels, d)
            cut = 3 - GHOSTS[recon]
            flux = [_sweep(u.narrow(ax, cut, u.shape[ax] - 2 * cut), d, None, recon, cfg.rsolver, cfg.gm1) for u in full]
            for k in range(len(levels)):
                f, n = flux[k], levels[k].shape[ax]
                if k + 1 < len(levels):  # the mean of the two fine fluxes through a coarse face
                    g = flux[k + 1]
                    g = g[..., ::2] if d == 0 else g[..., ::2, :]
                    g = 0.5 * (g[..., ::2, :] + g[..., 1::2, :]) if d == 0 else 0.5 * (g[..., ::2] + g[..., 1::2])
                    pad = lambda m: torch.cat([m.narrow(ax - 2, n - 1, 1), m, m.narrow(ax - 2, 0, 1)], ax - 2)  # noqa: E731
                    leaf, under = pad(self.leaf[k]), pad(self.under[k])
                    at = lambda m, o: m.narrow(ax - 2, o, n + 1)  # noqa: E731
                    meets = (at(leaf, 0) & at(under, 1)) | (at(under, 0) & at(leaf, 1))
                    f = torch.where(meets, g, f)
                rate[k] = rate[k] - (f.narrow(ax, 1, n) - f.narrow(ax, 0, n)) / self.dx[k][d]
        return rate

    def estimate(self, levels):
        return min(float(_estimate(u, self.dx[k], 2, self.cfg.gm1, self.cfg.cfl, self.leaf[k][None]))
                   for k, u in enumerate(levels))

    def advance(self, cells, steps):
        cfg, levels = self.cfg, self.spread(cells)
        t, dt = 0.0, self.estimate(levels)
        for _ in range(steps):
            start = levels
            for i, (g0, g1, beta) in enumerate(STAGES[cfg.integrator]):
                rates = self.rates(levels, "dc" if cfg.integrator == "vl2" and i == 0 else cfg.recon)
                new = []
                for u, u0, r, m in zip(levels, start, rates, self.leaf):
                    v = _kick(g0 * u + g1 * u0 + beta * dt * r, u, cfg.gravity, beta * dt, cfg.gm1)
                    new.append(torch.where(m, v, u))
                levels = new
            t, dt = t + dt, min(2.0 * dt, self.estimate(levels))
        return self.gather(levels), t, dt


def _rolled(cfg, u, dt, lam, steps):
    """(final state, gradient) of a fixed-dt rollout, the gradient by torch.autograd."""
    u = u.clone().requires_grad_(True)
    out = u
    for _ in range(steps):
        out = _step(out, cfg, dt)
    return out.detach(), torch.autograd.grad(out, u, lam)[0]


def _from_blocks(v, cfg):
    b, nb = cfg.block_nx, cfg.blocks_per_dim
    return v.reshape(nb[2], nb[1], nb[0], v.shape[1], b[2], b[1], b[0]).permute(3, 0, 4, 1, 5, 2, 6).reshape(
        v.shape[1], cfg.mesh_nx[2], cfg.mesh_nx[1], cfg.mesh_nx[0])


def exact(case, seed):
    path, steps = case["path"], case["steps"]
    if path == "refined":
        cfg, packed = _refined(case, seed)
        at, cells = 0, []
        for B in cfg.blocks:
            n = B.nx[0] * B.nx[1]
            cells.append(packed[at:at + 5 * n].view(5, n))
            at += 5 * n
        u, t, dt = _Levels(cfg).advance(torch.cat(cells, 1), steps)
        parts, at = [], 0
        for B in cfg.blocks:
            n = B.nx[0] * B.nx[1]
            parts.append(u[:, at:at + n].reshape(-1))
            at += n
        return {"state": torch.cat(parts), "time": t, "dt": dt, "ncycle": steps}
    if path in ("ensemble", "rollouts"):
        cfgs, states = _members(case, seed)
        if path == "ensemble":
            done = [_advance(u, c, steps) for c, u in zip(cfgs, states)]
            return {"state": torch.cat([_to_blocks(r[0], c).reshape(-1) for c, r in zip(cfgs, done)]),
                    "time": torch.tensor([r[1] for r in done], dtype=torch.float64),
                    "dt": torch.tensor([r[2] for r in done], dtype=torch.float64),
                    "ncycle": torch.full((len(cfgs),), steps, dtype=torch.int64)}
        lam = [_from_blocks(b, c) for b, c in zip(_directions(cfgs, seed), cfgs)]
        done = [_rolled(c, u, dt, m, steps) for c, u, dt, m in zip(cfgs, states, _max_dt(cfgs, states), lam)]
        return {"state": torch.cat([_to_blocks(r[0], c) for c, r in zip(cfgs, done)])[:, :, 0],
                "gradient": torch.cat([_with_ghosts(_to_blocks(r[1], c), c).reshape(-1) for c, r in zip(cfgs, done)])}
    cfg = _mesh(case)
    u = _state(case, cfg, seed)
    if path == "rollout":
        lam = _from_blocks(_directions([cfg], seed)[0], cfg)
        u, grad = _rolled(cfg, u, _max_dt([cfg], [u])[0], lam, steps)
        return {"state": _to_blocks(u, cfg)[:, :, 0], "gradient": _with_ghosts(_to_blocks(grad, cfg), cfg)}
    u, t, dt = _advance(u, cfg, steps)
    if path == "stepper":
        return {"state": _to_blocks(u, cfg), "time": t, "dt": dt, "ncycle": steps}
    for d in range(cfg.ndim):  # the driver's arrays, ghost cells filled
        u = _pad(u, 3 - d, cfg.ng, cfg.bc[d])
    for d in range(3):
        g = cfg.ng if d < cfg.ndim else 0
        u = u.unfold(3 - d, cfg.block_nx[d] + 2 * g, cfg.block_nx[d])
    # (nvar, nb3, nb2, nb1, ni, nj, nk) -> (nblocks, nvar, nk, nj, ni)
    cons = u.permute(1, 2, 3, 0, 6, 5, 4).reshape(cfg.pack_shape(cfg.nvar))
    return {"cons": cons, "time": t, "dt": dt, "ncycle": steps}
