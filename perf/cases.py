"""Performance cases of the particle path: what a user's program has it do,
through the public entry points (Simulation, Batch, trace_device).

A universe case is one call of the reference's simulateSteps as the drop-in
makes it: the particles go up from pinned host memory, the fields with them,
`steps` timesteps run, and what the program reads afterwards comes back
(fields, current and charge density, per-cell counts; the particles in the
caller's order where the program follows them). So every pass starts from the
same inputs, whatever ran before. The push's autotuner has chosen its shape
in prepare(), as a program's first steps let it.

Case fields: `kind` "universe" | "ensemble" | "tracer"; the rest are sizes,
policies and options by name (see _universe, _ensemble, _tracer)."""
import math
import random

import numpy as np
import torch

import allscale_ipic3d_gb300 as ipg
from allscale_ipic3d_gb300 import abi, tracer

_U64 = (1 << 64) - 1


def _universe(name, **kw):
    """A universe of n^3 cells of width `width`, `ppc` particles per cell (on
    average), `steps` timesteps per pass."""
    c = dict(kind="universe", name=name, n=8, width=1.0, ppc=64, steps=10, fp32=False, mover="field",
             solver="static", project=True, bc="periodic", species=1, load="uniform", vth=0.01, drift=0.0, dt=0.05,
             dipole=False, inject=False, div8=False, div_vol=False, si_units=False, particles_back=False)
    c.update(kw)
    return c


def _ensemble(name, **kw):
    c = dict(kind="ensemble", name=name, universes=64, sizes=12345, steps=50, fp32=True)
    c.update(kw)
    return c


def _tracer(name, **kw):
    c = dict(kind="tracer", name=name, particles=20000, T=40, S=10, R=16)
    c.update(kw)
    return c


def listed():
    return [
        # the small E x B drift run (8^3 x 64 ppc, 100 steps) in the default
        # FP64: a parameter study's single call, where latency counts
        _universe("exb_8_fp64", n=8, ppc=64, steps=100, dt=0.1, particles_back=True),
        # the .inp driver's own policies (dipole mover, static fields,
        # reflecting walls, planet) at tiny.inp's grid, in the reference's FP64
        _universe("inp_16_fp64", n=16, ppc=256, steps=20, mover="dipole", project=False, bc="reflect",
                  si_units=True, particles_back=True),
        # the headline magnetosphere run: FP32, 100 steps between outputs
        _universe("dipole_32_fp32", n=32, ppc=256, steps=100, fp32=True, solver="leapfrog", bc="outflow", species=2,
                  vth=0.005, drift=0.02, dipole=True, inject=True),
        # the same run in FP64 (what the FP32 run's error is stated against)
        _universe("dipole_32_fp64", n=32, ppc=256, steps=5, solver="leapfrog", bc="outflow", species=2,
                  vth=0.005, drift=0.02, dipole=True, inject=True),
        # uneven load: half uniform, half a Gaussian blob, so that cells hold
        # from a hundred to thousands of particles
        _universe("uneven_48_fp32", n=48, ppc=152, steps=50, fp32=True, solver="leapfrog", species=2, load="blob",
                  vth=0.02),
        # few particles per cell on an odd grid: the field solve, placement
        # and launches weigh as much as the push
        _universe("sparse_59_fp32", n=59, ppc=16, steps=100, fp32=True, solver="leapfrog", species=2, vth=0.02),
        # the forward solver with the reference's normalisations (/ vol, / 8)
        # on cells of another width, odd grid, FP64
        _universe("forward_21_fp64", n=21, width=0.5, ppc=33, steps=20, solver="forward", species=2, div8=True,
                  div_vol=True, dt=0.02),
        # many small independent runs at once: 64 periodic universes of
        # 8^3 .. 24^3 cells with 16 .. 256 particles per cell
        _ensemble("ensemble_64_fp32"),
        # the reference's :U:N benchmark policies (electrons, dipole mover
        # without external field, reflecting walls), N = 4M, FP32
        _universe("udist_32_fp32", n=32, width=10.0, ppc=128, steps=100, fp32=True, mover="dipole", project=False,
                  bc="reflect", vth=0.2, dt=0.15, particles_back=True),
        # a host program that keeps the particles and calls every timestep:
        # the whole state up, one headline step, the whole state back
        _universe("roundtrip_32_fp32", n=32, ppc=256, steps=1, fp32=True, solver="leapfrog", bc="outflow", species=2,
                  vth=0.005, drift=0.02, dipole=True, particles_back=True),
        # the standalone tracer: a short run, and pic_tracer's default run
        _tracer("tracer_20k"),
        _tracer("tracer_16m", particles=16000000, T=150, S=10, R=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(["field", "field", "field", "dipole_mover", "ensemble", "tracer"])
    if kind == "tracer":
        T = rng.randrange(20, 160)
        n = _log_int(rng, 5000, 8000000)
        c = _tracer("", particles=n, T=T, S=rng.choice([5, 7, 10]), R=rng.choice([16, 24, 33, 64]))
    elif kind == "ensemble":
        c = _ensemble("", universes=rng.randrange(3, 48), sizes=rng.randrange(1 << 20), fp32=rng.random() < 0.7)
        c["steps"] = rng.randrange(10, 60) if c["fp32"] else rng.randrange(2, 6)
    else:
        n = _log_int(rng, 5, 48)
        ppc = _log_int(rng, 8, 256)
        ppc = max(4, min(ppc, 12000000 // n ** 3))
        fp32 = rng.random() < 0.5
        steps = max(1, min(100, int((4e9 if fp32 else 1.5e8) / (n ** 3 * ppc))))
        steps = max(1, int(steps * rng.uniform(0.5, 1.0)))
        if kind == "dipole_mover":
            si = rng.random() < 0.5
            c = _universe("", n=n, ppc=ppc, steps=steps, fp32=fp32 and not si, mover="dipole", project=False,
                          bc="reflect", si_units=si, width=rng.choice([1.0, 2.5, 10.0]), vth=0.2, dt=0.1,
                          particles_back=True)
        else:
            dipole = rng.random() < 0.4 and n >= 10
            c = _universe("", n=n, ppc=ppc, steps=steps, fp32=fp32,
                          solver=rng.choice(["static", "leapfrog", "forward"]), species=rng.choice([1, 2]),
                          vth=rng.choice([0.005, 0.01, 0.02]), dt=rng.choice([0.03, 0.05]),
                          width=1.0 if dipole else rng.choice([1.0, 0.75]),
                          bc=rng.choice(["outflow", "reflect"]) if dipole else rng.choice(["periodic", "reflect"]),
                          load=rng.choice(["uniform", "blob"]), dipole=dipole, drift=0.02 if dipole else 0.0,
                          div8=rng.random() < 0.3, particles_back=rng.random() < 0.5)
            c["inject"] = dipole and c["bc"] == "outflow" and rng.random() < 0.5 and not c["particles_back"]
    del c["name"]
    return c


# ---- inputs ------------------------------------------------------------------------
CHARGE = 1e-3  # of a cell's worth of one species: plasma frequency 0.03


def _props(case):
    n = case["n"]
    if case["si_units"]:  # the .inp driver's universe: Earth, SI units, 10 planet radii across
        p = tracer.tracer_props(n)
        w = 10.0 * p.planet_radius / n
        return abi.Props.make(size=(n,) * 3, cell_width=(w,) * 3, dt=0.01, speed_of_light=p.speed_of_light,
                              planet_radius=p.planet_radius, origin=(-n * w / 2.0,) * 3, external_b=(0, 0, 3.07e-5))
    w = case["width"]
    if case["dipole"]:  # |B| = 0.5 at 4 cells, the 2 innermost masked
        return abi.Props.make(size=(n,) * 3, cell_width=(w,) * 3, dt=case["dt"], planet_radius=2.0 * w,
                              origin=(-n * w / 2.0,) * 3, external_b=(0.0, 0.0, 4.0))
    return abi.Props.make(size=(n,) * 3, cell_width=(w,) * 3, dt=case["dt"])


def _species(case):
    """[(q, q/m, thermal speed)]"""
    if case["si_units"]:
        qom = tracer.ELEMENTARY_CHARGE / tracer.PROTON_MASS
        return [(tracer.ELEMENTARY_CHARGE, qom, tracer.speed_scale(_props(case)))]
    if case["mover"] == "dipole":
        return [(-1.0, -25.0, case["vth"])]
    per = max(1, case["ppc"] // case["species"])
    q = CHARGE / per
    if case["species"] == 1:
        return [(-q, -1.0, case["vth"])]
    ion = case["vth"] if case["dipole"] else case["vth"] / 10.0
    return [(-q, -1.0, case["vth"]), (q, 0.01, ion)]


def _config(case):
    faces = {"periodic": [abi.BC_PERIODIC] * 3, "reflect": [abi.BC_REFLECT] * 3,
             "outflow": [abi.BC_OPEN, abi.BC_PERIODIC, abi.BC_PERIODIC]}[case["bc"]]
    flags = abi.F_USE_GRAPH
    flags |= abi.F_REFRESH_NODE_B if case["solver"] == "leapfrog" else 0
    flags |= abi.F_J_DIV8 if case["div8"] else 0
    flags |= abi.F_GATHER_DIV_VOL if case["div_vol"] else 0
    flags |= abi.F_DIPOLE_IN_GATHER if case["dipole"] else 0
    flags |= abi.F_TRACK_IDS if case["particles_back"] else 0
    kw = {}
    if case["inject"]:
        flags |= abi.F_INJECT_LOW_X
        q, qom, vth = _species(case)[0]
        kw = dict(inject_per_cell=case["ppc"] / case["species"] * case["drift"] * case["dt"] / case["width"],
                  inject_q=q, inject_qom=qom, inject_drift=(case["drift"], 0.0, 0.0), inject_vth=(vth,) * 3,
                  seed=12345)
    return abi.Config.make(
        precision=abi.FP32 if case["fp32"] else abi.FP64,
        mover=abi.MOVER_DIPOLE if case["mover"] == "dipole" else abi.MOVER_FIELD,
        solver={"static": abi.SOLVER_STATIC, "leapfrog": abi.SOLVER_LEAPFROG, "forward": abi.SOLVER_FORWARD}[
            case["solver"]],
        projector=abi.PROJECT_CIC if case["project"] else abi.PROJECT_NONE, bc_low=faces, bc_high=faces, flags=flags,
        **kw)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _particles(props, counts, species, drift, g):
    """(N, 8) records on the GPU, grouped by cell: position uniform in the
    cell, velocity Maxwellian, species drawn per particle."""
    n = props.shape[0]
    cell = torch.repeat_interleave(torch.arange(n ** 3, device="cuda"), counts)
    N = int(cell.numel())
    rec = torch.empty((N, 8), dtype=torch.float64, device="cuda")
    r = torch.rand((N, 3), generator=g, dtype=torch.float64, device="cuda")
    for a, idx in enumerate((cell // (n * n), (cell // n) % n, cell % n)):
        rec[:, a] = props.origin[a] + (idx + r[:, a]) * props.cell_width[a]
    sp = torch.tensor(species, dtype=torch.float64, device="cuda")
    which = torch.randint(len(species), (N,), generator=g, device="cuda")
    rec[:, 3:6] = torch.randn((N, 3), generator=g, dtype=torch.float64, device="cuda") * sp[which, 2:3]
    rec[:, 3] += drift
    rec[:, 6:8] = sp[which, 0:2]
    return rec


def _universe_inputs(case, seed):
    """(props, particle records on the GPU, counts per cell on the GPU, field
    grid, cell-centred B grid)."""
    g = _generator(seed)
    props = _props(case)
    n = case["n"]
    nc = n ** 3
    if case["load"] == "blob":  # half uniform, half in a Gaussian blob off the centre
        half = case["ppc"] // 2
        centre = torch.tensor([0.62, 0.56, 0.5], dtype=torch.float64, device="cuda") * n
        at = torch.randn((half * nc, 3), generator=g, dtype=torch.float64, device="cuda") * (n * 0.1) + centre
        at = at.floor().long() % n
        counts = torch.bincount((at[:, 0] * n + at[:, 1]) * n + at[:, 2], minlength=nc) + (case["ppc"] - half)
    else:
        counts = torch.full((nc,), case["ppc"], dtype=torch.int64, device="cuda")
    rec = _particles(props, counts, _species(case), case["drift"], g)
    field = np.zeros(abi.field_shape(props))
    bc = np.zeros(abi.bcfield_shape(props))
    if case["mover"] == "field":
        tilt = float(torch.rand(1, generator=g, dtype=torch.float64, device="cuda"))
        if not case["dipole"]:
            field[..., 3], field[..., 5] = 0.05 * tilt, 0.1
            bc[..., 0], bc[..., 2] = 0.05 * tilt, 0.1
        if case["solver"] == "static":
            field[..., 1] = 0.01
    return props, rec, counts, field, bc


def _pinned(rec):
    """The records in pinned host memory, as the reference's Particle array."""
    host = torch.empty(rec.shape, dtype=torch.float64, pin_memory=True)
    host.copy_(rec)
    return host, host.numpy().reshape(-1).view(abi.PARTICLE_DTYPE)


def _upload_first(sim, props, species, parts, counts):
    """A universe's first upload: a particle of each species first, so that
    the large upload finds its species known (the device path)."""
    few = np.zeros(len(species), abi.PARTICLE_DTYPE)
    few["position"] = np.array(props.origin) + 0.5 * np.array(props.cell_width)
    few["q"], few["qom"] = [s[0] for s in species], [s[1] for s in species]
    c0 = np.zeros(props.ncells, np.uint64)
    c0[0] = len(few)
    sim.upload_particles(few, c0)
    sim.upload_particles(parts, counts)


def _let_it_tune(sim):
    for _ in range(100):
        sim.step(1)
        if not sim.push_shape()["tuning"]:
            break


class _Universe:
    def __init__(self, case, seed):
        self.case = case
        props, rec, counts, self.field, self.bc = _universe_inputs(case, seed)
        self.host, self.parts = _pinned(rec)
        self.counts = counts.cpu().numpy().astype(np.uint64)
        species = _species(case)
        if case["fp32"]:  # the shape is kept per workload: the run's own universe starts at step 0
            with ipg.Simulation(props, _config(case)) as probe:
                probe.upload_fields(self.field, self.bc)
                _upload_first(probe, props, species, self.parts, self.counts)
                _let_it_tune(probe)
        self.sim = ipg.Simulation(props, _config(case))
        _upload_first(self.sim, props, species, self.parts, self.counts)
        self.back = None
        if case["particles_back"]:
            room = len(self.parts)
            self.back_host = torch.empty((room, 8), dtype=torch.float64, pin_memory=True)
            self.back = (self.back_host.numpy().reshape(-1).view(abi.PARTICLE_DTYPE),
                         np.zeros(props.ncells, np.uint64))
            self.ids_host = torch.zeros(room, dtype=torch.int32, pin_memory=True)
            self.ids = self.ids_host.numpy().view(np.uint32)

    def run(self):
        case, sim, out = self.case, self.sim, {}
        sim.upload_fields(self.field, self.bc)
        sim.upload_particles(self.parts, self.counts)
        sim.step(case["steps"])
        if self.back is not None:
            p, counts, _ = sim.download_particles(out=self.back, ids=self.ids)
            k = len(p)
            # back in the caller's order, on the GPU, where its analysis goes on
            at = self.ids_host[:k].to("cuda", non_blocking=True).long()
            mine = torch.zeros((len(self.parts), 8), dtype=torch.float64, device="cuda")
            mine[at] = self.back_host[:k].to("cuda", non_blocking=True)
            out["particles"] = mine
            out["counts"] = counts.astype(np.int64)
        else:
            out["counts"] = sim.cell_counts().astype(np.int64)
        if case["project"]:
            f, b, J, rho = sim.download_fields()
            out["J"], out["rho"] = J, rho
            if case["solver"] != "static":
                out["field"], out["bcfield"] = f, b
        return out


class _Ensemble:
    SIZES, PPC = (8, 12, 16, 20, 24), (16, 32, 64, 128, 256)

    @classmethod
    def params(cls, case):
        r = random.Random(case["sizes"])
        return [(r.choice(cls.SIZES), r.choice(cls.PPC), r.uniform(0.005, 0.02)) for _ in range(case["universes"])]

    @classmethod
    def inputs(cls, case, seed, i, n, ppc, vth):
        g = _generator(seed * 1000 + i)
        props = abi.Props.make(size=(n,) * 3, dt=0.1)
        counts = torch.full((n ** 3,), ppc, dtype=torch.int64, device="cuda")
        species = [(-1.0 / ppc, -1.0, vth)]
        rec = _particles(props, counts, species, 0.0, g)
        d = torch.randn(6, generator=g, dtype=torch.float64, device="cuda").cpu().numpy()
        m = torch.rand(2, generator=g, dtype=torch.float64, device="cuda").cpu().numpy()
        B = d[:3] / np.linalg.norm(d[:3]) * (0.02 + 0.18 * m[0])
        E = d[3:] / np.linalg.norm(d[3:]) * 0.02 * m[1]
        field = np.zeros(abi.field_shape(props))
        field[..., 0:3], field[..., 3:6] = E, B
        bc = np.zeros(abi.bcfield_shape(props))
        bc[...] = B
        return props, rec, counts, field, bc, species

    def __init__(self, case, seed):
        self.case = case
        cfg = abi.Config.make(precision=abi.FP32 if case["fp32"] else abi.FP64, mover=abi.MOVER_FIELD,
                              projector=abi.PROJECT_CIC, bc=abi.BC_PERIODIC, flags=abi.F_USE_GRAPH)
        made = [self.inputs(case, seed, i, *p) for i, p in enumerate(self.params(case))]
        self.batch = ipg.Batch([m[0] for m in made], cfg)
        self.keep, self.sets = [], []
        for i, (props, rec, counts, field, bc, species) in enumerate(made):
            host, parts = _pinned(rec)
            u = self.batch.universe(i)
            c = counts.cpu().numpy().astype(np.uint64)
            u.upload_fields(field, bc)
            _upload_first(u, props, species, parts, c)
            self.keep.append(host)
            self.sets.append((u, parts, c))
        if case["fp32"]:
            _let_it_tune(self.batch)

    def run(self):
        for u, parts, counts in self.sets:
            u.upload_particles(parts, counts)
        self.batch.step(self.case["steps"])
        J, rho, n = [], [], []
        for u, _, _ in self.sets:
            _, _, j, r = u.download_fields()
            J.append(j.reshape(-1))
            rho.append(r.reshape(-1))
            n.append(u.cell_counts().astype(np.int64))
        return {"J": np.concatenate(J), "rho": np.concatenate(rho), "counts": np.concatenate(n)}


class _Tracer:
    def __init__(self, case, seed):
        self.case, self.props = case, tracer.tracer_props(case["R"])
        g = _generator(seed)
        N = case["particles"]
        low, hig = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in tracer.particle_box(self.props))
        self.rec = torch.empty((N, 8), dtype=torch.float64, device="cuda")
        self.rec[:, 0:3] = low + torch.rand((N, 3), generator=g, dtype=torch.float64, device="cuda") * (hig - low)
        self.rec[:, 3:6] = torch.randn((N, 3), generator=g, dtype=torch.float64, device="cuda") * float(
            tracer.speed_scale(self.props))
        self.rec[:, 6] = tracer.ELEMENTARY_CHARGE
        self.rec[:, 7] = tracer.ELEMENTARY_CHARGE / tracer.PROTON_MASS
        self.frames = case["T"] // case["S"] + 1
        self.counts = torch.empty((self.frames,) + self.props.shape, dtype=torch.int32, device="cuda")

    def run(self):
        self.counts.zero_()
        ipg.trace_device(self.props, self.rec.data_ptr(), self.case["particles"], self.case["T"] + 1, self.case["S"],
                         self.frames, self.counts.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return self.counts


def prepare(case, seed):
    return {"universe": _Universe, "ensemble": _Ensemble, "tracer": _Tracer}[case["kind"]](case, seed)


def run(state):
    return state.run()


def work(case):
    """Per pass: the caller's records read once, the particle state read and
    written once a step in the path's precision, the fields and moments of
    the grid once a step where they take part, the outputs written once. The
    tracer's particles stay on the chip between its steps. flops: the
    arithmetic of a particle step in its cheapest form."""
    if case["kind"] == "tracer":
        N, cells = case["particles"], case["R"] ** 3
        return {"bytes": 64 * N + 4 * cells * (case["T"] // case["S"] + 1), "flops": 90 * N * (case["T"] + 1)}
    if case["kind"] == "ensemble":
        sets = [(n ** 3, ppc * n ** 3, (n + 1) ** 3) for n, ppc, _ in _Ensemble.params(case)]
        cells, N, nodes = (sum(s[k] for s in sets) for k in range(3))
        field, solver, dipole, back, project = True, "static", False, False, True
    else:
        n = case["n"]
        cells, nodes, N = n ** 3, (n + 1) ** 3, n ** 3 * case["ppc"]
        field, solver, dipole = case["mover"] == "field", case["solver"], case["dipole"] or case["mover"] == "dipole"
        back, project = case["particles_back"], case["project"]
    e = 4 if case["fp32"] else 8
    step = 12 * e * N + (6 * e * nodes if field else 0) + (64 * nodes if project else 0)
    step += 18 * 8 * nodes if solver != "static" else 0
    flops = 45 + (84 if field else 0) + (25 if dipole else 0) + (70 if project else 0)
    once = 64 * N + 8 * cells + (64 * N if back else 0) + (32 * nodes if project else 0)
    once += 2 * 96 * nodes if solver != "static" else 0
    return {"bytes": once + case["steps"] * step, "flops": case["steps"] * N * flops}


# ---- the same timesteps in plain 64-bit torch -----------------------------------------
def _signed(v):
    v &= _U64
    return v - (1 << 64) if v >> 63 else v


def _fmix(k):
    """MurmurHash3's 64-bit finaliser on int64 tensors (wrapping products)."""
    k = k ^ ((k >> 33) & 0x7FFFFFFF)
    k = k * _signed(0xFF51AFD7ED558CCD)
    k = k ^ ((k >> 33) & 0x7FFFFFFF)
    k = k * _signed(0xC4CEB9FE1A85EC53)
    return k ^ ((k >> 33) & 0x7FFFFFFF)


class _Plain:
    """The timestep of one universe on FP64 arrays, written from the method:
    trilinear gather, Boris with sub-cycles, walls, planet, migration by cell
    index, cloud-in-cell densities, leapfrog / forward fields."""

    def __init__(self, props, rec, counts, field, bc, o):
        self.p, self.o, self.n = props, o, props.shape[0]
        dev = rec.device
        n = self.n
        cell = torch.repeat_interleave(torch.arange(n ** 3, device=dev), counts)
        self.N = rec.shape[0]
        # in mixed order: neighbours in the list then add to different nodes
        self.id = torch.randperm(self.N, generator=_generator(1), device=dev)
        cell, rec = cell[self.id], rec[self.id]
        self.c = [cell // (n * n), (cell // n) % n, cell % n]
        self.x = [rec[:, a].clone() for a in range(3)]
        self.v = [rec[:, 3 + a].clone() for a in range(3)]
        self.q, self.qom = rec[:, 6].clone(), rec[:, 7].clone()
        self.w, self.org = [float(v) for v in props.cell_width], [float(v) for v in props.origin]
        self.vol = self.w[0] * self.w[1] * self.w[2]
        self.f = torch.as_tensor(field, device=dev).clone()
        self.b = torch.as_tensor(bc, device=dev).clone()
        self.J = torch.zeros((n + 1,) * 3 + (3,), dtype=torch.float64, device=dev)
        self.rho = torch.zeros((n + 1,) * 3, dtype=torch.float64, device=dev)
        self.t = 0
        if o["project"]:
            self.project()

    def frac(self, a):
        return (self.x[a] - (self.org[a] + self.c[a] * self.w[a])) / self.w[a]

    def corners(self):
        r = [self.frac(a) for a in range(3)]
        for i in range(2):
            for j in range(2):
                for k in range(2):
                    yield (i, j, k), (r[0] if i else 1 - r[0]) * (r[1] if j else 1 - r[1]) * (r[2] if k else 1 - r[2])

    def project(self):
        n = self.n
        s = torch.zeros(((n + 1) ** 3, 4), dtype=torch.float64, device=self.f.device)
        qv = torch.stack([self.q * v for v in self.v] + [self.q], 1)
        for (i, j, k), fac in self.corners():
            s.index_add_(0, ((self.c[0] + i) * (n + 1) + self.c[1] + j) * (n + 1) + self.c[2] + k, qv * fac[:, None])
        s = s.reshape(n + 1, n + 1, n + 1, 4)
        for a in range(3):  # a boundary node stands for its image too
            both = s.select(a, 0) + s.select(a, n)
            s.select(a, 0).copy_(both)
            s.select(a, n).copy_(both)
        s = s / self.vol
        if self.o["div8"]:
            s = s / 8.0
        self.J, self.rho = s[..., :3].clone(), s[..., 3].clone()

    def solve(self):
        for g, m in ((self.f, self.n + 3), (self.b, self.n + 2)):  # ghost faces
            e, i = m - 1, slice(1, m - 1)
            g[0, i, i], g[e, i, i] = g[e - 1, i, i].clone(), g[1, i, i].clone()
            g[i, 0, i], g[i, e, i] = g[i, e - 1, i].clone(), g[i, 1, i].clone()
            g[i, i, 0], g[i, i, e] = g[i, i, e - 1].clone(), g[i, i, 1].clone()
        n, dt, c, (wx, wy, wz) = self.n, float(self.p.dt), float(self.p.speed_of_light), self.w
        u, d = slice(1, n + 2), slice(0, n + 1)    # a node's own cell and the one before
        E = self.f[..., 0:3]
        if self.o["solver"] == "leapfrog":
            B, Bx, By, Bz = self.b[u, u, u], self.b[d, u, u], self.b[u, d, u], self.b[u, u, d]
            D = B - Bx, B - By, B - Bz
        else:
            def diff(a):  # difference along a, mean over the other two axes
                tot = 0
                for i in (u, d):
                    for j in (u, d):
                        s1, s0 = [i, j], [i, j]
                        s1.insert(a, u)
                        s0.insert(a, d)
                        tot = tot + 0.25 * (self.b[tuple(s1)] - self.b[tuple(s0)])
                return tot
            D = diff(0), diff(1), diff(2)
        curl = torch.stack([D[1][..., 2] / wy - D[2][..., 1] / wz, D[2][..., 0] / wz - D[0][..., 2] / wx,
                            D[0][..., 1] / wx - D[1][..., 0] / wy], -1)
        E[u, u, u] += dt * ((c * c if self.o["solver"] == "leapfrog" else c) * curl - self.J)
        u, d = slice(2, n + 2), slice(1, n + 1)
        if self.o["solver"] == "leapfrog":
            D = E[u, d, d] - E[d, d, d], E[d, u, d] - E[d, d, d], E[d, d, u] - E[d, d, d]
        else:
            def diff_e(a):
                tot = 0
                for i in (u, d):
                    for j in (u, d):
                        s1, s0 = [i, j], [i, j]
                        s1.insert(a, u)
                        s0.insert(a, d)
                        tot = tot + 0.25 * (E[tuple(s1)] - E[tuple(s0)])
                return tot
            D = diff_e(0), diff_e(1), diff_e(2)
        curl = torch.stack([D[1][..., 2] / wy - D[2][..., 1] / wz, D[2][..., 0] / wz - D[0][..., 2] / wx,
                            D[0][..., 1] / wx - D[1][..., 0] / wy], -1)
        self.b[d, d, d] -= (1.0 if self.o["solver"] == "leapfrog" else c) * dt * curl
        u, d = slice(1, n + 2), slice(0, n + 1)
        self.f[u, u, u, 3:6] = 0.125 * sum(self.b[i, j, k] for i in (u, d) for j in (u, d) for k in (u, d))

    def push(self):
        p, o, n, dt = self.p, self.o, self.n, float(self.p.dt)
        E = B = torch.zeros((1, 3), dtype=torch.float64, device=self.f.device)
        if o["field"]:
            EB = 0
            flat = self.f[..., :6].reshape(-1, 6)
            for (i, j, k), fac in self.corners():
                EB = EB + flat[((self.c[0] + i + 1) * (n + 3) + self.c[1] + j + 1) * (n + 3) + self.c[2] + k + 1] * \
                    fac[:, None]
            if o["div_vol"]:
                EB = EB / self.vol
            E, B = EB[:, :3], EB[:, 3:]
        if o["dipole"]:
            x, y, z = self.x
            f = -float(p.external_b[2]) * float(p.planet_radius) ** 3 / (x * x + y * y + z * z) ** 2.5
            B = B + torch.stack([3 * x * z * f, 3 * y * z * f, (2 * z * z - x * x - y * y) * f], 1)
        B2 = (B * B).sum(1)
        ratio = dt * 4.0 * self.qom.abs() * B2 / (math.pi * float(p.speed_of_light))
        ns = (ratio.floor().clamp(max=99).nan_to_num(0) + 1).expand(len(self.qom))
        dts = dt / ns
        k = (self.qom * 0.5 * dts)[:, None]
        t = k * B
        s = 2 * t / (1 + (t * t).sum(1, keepdim=True))
        v, x = torch.stack(self.v, 1), torch.stack(self.x, 1)
        for m in range(int(ns.max()) if len(ns) else 0):
            on = (ns > m)[:, None]
            vm = v + k * E
            vp = vm + torch.linalg.cross(vm, t)
            vn = vm + torch.linalg.cross(vp, s) + k * E
            v = torch.where(on, vn, v)
            x = torch.where(on, x + v * dts[:, None], x)
        drop = torch.zeros(len(v), dtype=torch.bool, device=v.device)
        flip = drop.clone()
        mid = [self.org[a] + self.c[a] * self.w[a] + self.w[a] / 2 for a in range(3)]
        half = [w / 2 for w in self.w]
        for a in range(3):
            rel = x[:, a] - mid[a]
            lo, hi = (self.c[a] == 0) & (rel < -half[a]), (self.c[a] == n - 1) & (rel > half[a])
            if o["bc"][a] == "open":
                drop |= lo | hi
            elif o["bc"][a] == "reflect":
                flip |= lo | hi
                x[:, a] = torch.where(lo, x[:, a] + half[a], torch.where(hi, x[:, a] - half[a], x[:, a]))
        v = torch.where(flip[:, None], -v, v)
        drop |= sum((x[:, a] - float(p.object_center[a])) ** 2 for a in range(3)) <= float(p.planet_radius) ** 2
        for a in range(3):
            rel = x[:, a] - mid[a]
            step = (rel > half[a]).long() - (rel < -half[a]).long()
            to = self.c[a] + step
            if o["bc"][a] == "periodic":
                L = n * self.w[a]
                x[:, a] = torch.where(to < 0, x[:, a] + L, torch.where(to >= n, x[:, a] - L, x[:, a]))
            self.c[a] = to % n
        keep = ~drop
        self.x, self.v = [x[keep, a] for a in range(3)], [v[keep, a] for a in range(3)]
        self.c = [c[keep] for c in self.c]
        self.q, self.qom, self.id = self.q[keep], self.qom[keep], self.id[keep]

    def inject(self, cfg):
        """Counter-based draws keyed by (seed, step, face cell, draw)."""
        n, dev = self.n, self.f.device
        cell = torch.arange(n * n, device=dev)
        k0 = _fmix(torch.tensor([_signed(cfg.seed ^ (self.t * 0x9E3779B97F4A7C15 & _U64))], device=dev))

        def u(cells, d):
            key = _fmix(k0 ^ (cells * _signed(0xD1B54A32D192ED03) + d))
            return ((key >> 11) & ((1 << 53) - 1)).double() * 2.0 ** -53

        many = (cfg.inject_per_cell + u(cell, 0)).floor().long()
        for m in range(int(many.max())):
            c = cell[many > m]
            r = [u(c, 1 + 8 * m + t) for t in range(7)]
            g1, g2 = (-2 * (1 - r[3]).log()).sqrt(), (-2 * (1 - r[5]).log()).sqrt()
            normal = [g1 * (2 * math.pi * r[4]).cos(), g1 * (2 * math.pi * r[4]).sin(),
                      g2 * (2 * math.pi * r[6]).cos()]
            at = [torch.zeros_like(c), c // n, c % n]
            for a in range(3):
                self.x[a] = torch.cat([self.x[a], self.org[a] + (at[a] + r[a]) * self.w[a]])
                self.v[a] = torch.cat([self.v[a], cfg.inject_drift[a] + cfg.inject_vth[a] * normal[a]])
                self.c[a] = torch.cat([self.c[a], at[a]])
            self.q = torch.cat([self.q, torch.full_like(r[0], cfg.inject_q)])
            self.qom = torch.cat([self.qom, torch.full_like(r[0], cfg.inject_qom)])
            self.id = torch.cat([self.id, torch.full_like(c, -1)])

    def steps(self, count, cfg=None):
        for _ in range(count):
            if self.o["solver"] != "static":
                self.solve()
            self.push()
            if cfg is not None:
                self.inject(cfg)
            if self.o["project"]:
                self.project()
            self.t += 1

    def in_order(self):
        mine = torch.zeros((self.N, 8), dtype=torch.float64, device=self.f.device)
        mine[self.id] = torch.stack(self.x + self.v + [self.q, self.qom], 1)
        return mine


def exact(case, seed):
    if case["kind"] == "tracer":
        return None  # counts only
    if case["kind"] == "ensemble":
        J, rho = [], []
        for i, par in enumerate(_Ensemble.params(case)):
            props, rec, counts, field, bc, _ = _Ensemble.inputs(case, seed, i, *par)
            o = dict(field=True, dipole=False, solver="static", project=True, div8=False, div_vol=False,
                     bc=["periodic"] * 3)
            s = _Plain(props, rec, counts, field, bc, o)
            s.steps(case["steps"])
            J.append(s.J.reshape(-1))
            rho.append(s.rho.reshape(-1))
        return {"J": torch.cat(J), "rho": torch.cat(rho), "counts": None}
    props, rec, counts, field, bc = _universe_inputs(case, seed)
    o = dict(field=case["mover"] == "field", dipole=case["dipole"] or case["mover"] == "dipole",
             solver=case["solver"], project=case["project"], div8=case["div8"], div_vol=case["div_vol"],
             bc=["open", "periodic", "periodic"] if case["bc"] == "outflow" else [case["bc"]] * 3)
    s = _Plain(props, rec, counts, field, bc, o)
    s.steps(case["steps"], _config(case) if case["inject"] else None)
    out = {"counts": None}
    if case["particles_back"]:
        out["particles"] = s.in_order()
    if case["project"]:
        out["J"], out["rho"] = s.J, s.rho
        if case["solver"] != "static":
            out["field"], out["bcfield"] = s.f, s.b
    return out
