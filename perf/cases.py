"""Performance cases of the PIC + DSMC framework, driven through its public entry points.

listed() names the cases, draw() gives others of the same ranges, prepare() builds what a user's
program holds before the call (a world with its species, solver and fields, or device arrays), and
run() is one pass of that program: a stretch of the time loop up to the diagnostics it reads, a
Poisson solve of a given charge density, or the sampling of a density or of gas properties.
work() states the bytes and operations a pass cannot do without, and exact() what run() returns
on new inputs in 64-bit arithmetic, in plain torch.

What the cases stand for:
  loop     pic_step() as the ch4/v3 driver calls it (collisions, push, deposit, charge density,
           Poisson, E, sort and merge checks), with the per-step diagnostics of runtime_diags.csv
  trace    the same loop with the field solve switched off, as the v3 driver ships: electrons and
           ions pushed through a frozen field, their moving-average density read every 20 steps
  poisson  a cold solve of a charge density the caller holds, and the potential read back
  moments  velocity moments of a neutral gas sampled over some steps, then its gas properties
  density  number density of the caller's own device arrays (no device allocation)
  dsmc     particle-particle collisions of a neutral gas, then its sums and cell counts
"""
import importlib
import math

import numpy as np
import torch

pic = importlib.import_module("engineering-degree-in-plasma-simulations_gb300")

EV_K = pic.QE / pic.KB
LOTZ = dict(A=2.107e-17, b=1.0, c=0.18, I=12.06)  # O2 ionisation, as the benchmark's discharges
TRACE_STEPS = 20  # one period of Field::updateMovingAverage
MOMENT_STEPS = 4
DSMC_CALLS = 4


# the physics of the discharges: box side, anode, background density, time step
DISCHARGE = dict(side=0.02, volts=500.0, gas=1e21, dt=2e-12, fields=True)
LARGE = dict(side=0.04, volts=1000.0, gas=2e21, dt=1e-12, fields=False)


def listed():
    return [
        # plain electrostatic PIC, 21^3 nodes with Dirichlet walls and 80 000 + 80 000 particles, the
        # reference's own SOR solver: the smallest loop, where launches and waits count
        dict(name="loop_plain_21", what="loop", ni=21, nj=21, nk=21, n=80_000, instances=0, solver="gs", steps=10,
             fields=True),
        # the electrode discharge (500 V, O2 background) with collisions and the learned solver
        dict(name="loop_discharge_64", what="loop", ni=64, nj=64, nk=256, n=2_000_000, instances=0,
             solver="learned", steps=20, **DISCHARGE),
        # 16 stacked discharges of 32 x 32 x 128 nodes with uneven particle counts
        dict(name="loop_ensemble_16", what="loop", ni=32, nj=32, nk=128, n=300_000, instances=16, solver="learned",
             steps=10, **DISCHARGE),
        # the large discharge, 100 M + 100 M particles: diagnostics of every step, no field output
        dict(name="loop_large", what="loop", ni=256, nj=256, nk=512, n=100_000_000, instances=0, solver="learned",
             steps=10, **LARGE),
        # electrons and ions through a frozen field on a ragged grid
        dict(name="trace_ragged", what="trace", ni=97, nj=113, nk=129, n=16_000_000),
        # cold solves: the reference's small grid with E; the default PCG on an odd box (rows of 129
        # nodes); SOR; the learned preconditioner on the 256^3 blob charge
        dict(name="poisson_pcg_31", what="poisson", ni=31, nj=31, nk=51, solver="pcg", periodic=False, field=True),
        dict(name="poisson_pcg_129", what="poisson", ni=129, nj=129, nk=129, solver="pcg", periodic=False, field=False),
        dict(name="poisson_gs_65", what="poisson", ni=65, nj=65, nk=97, solver="gs", periodic=False, field=False),
        dict(name="poisson_learned_256", what="poisson", ni=256, nj=256, nk=256, solver="learned", periodic=True,
             field=False),
        # gas diagnostics of a neutral flow
        dict(name="moments_64", what="moments", ni=65, nj=65, nk=65, n=8_000_000),
        # a plugin's density field from its own arrays, in cell order as a particle code keeps them
        dict(name="density_100", what="density", ni=101, nj=101, nk=101, n=10_000_000, ordered=True),
        # rarefied gas, 16 particles per cell
        dict(name="dsmc_128", what="dsmc", ni=129, nj=129, nk=129, ppc=16),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["plain", "discharge", "ensemble", "trace", "pcg", "gs", "learned", "moments", "density", "dsmc"])
    if kind == "plain":
        return dict(what="loop", ni=size(11, 41), nj=size(11, 41), nk=size(11, 51), n=size(10_000, 300_000),
                    instances=0, solver=rng.choice(["gs", "pcg"]), steps=10, fields=True)
    if kind == "discharge":
        return dict(what="loop", ni=size(24, 128), nj=size(24, 128), nk=size(48, 256), n=size(100_000, 10_000_000),
                    instances=0, solver="learned", steps=rng.randint(5, 20), **DISCHARGE)
    if kind == "ensemble":
        return dict(what="loop", ni=size(17, 33), nj=size(17, 33), nk=size(32, 128), n=size(20_000, 400_000),
                    instances=rng.randint(3, 24), solver="learned", steps=rng.randint(5, 10), **DISCHARGE)
    if kind == "trace":
        return dict(what="trace", ni=size(16, 128), nj=size(16, 128), nk=size(16, 160), n=size(50_000, 20_000_000))
    if kind in ("pcg", "gs", "learned"):
        lo, hi = {"pcg": (17, 144), "gs": (17, 80), "learned": (32, 200)}[kind]
        per = kind == "learned" or rng.random() < 0.4
        return dict(what="poisson", ni=size(lo, hi), nj=size(lo, hi), nk=size(lo, hi), solver=kind, periodic=per,
                    field=rng.random() < 0.5)
    if kind == "moments":
        return dict(what="moments", ni=size(9, 97), nj=size(9, 97), nk=size(9, 97), n=size(20_000, 10_000_000))
    if kind == "density":
        return dict(what="density", ni=size(9, 101), nj=size(9, 101), nk=size(9, 101), n=size(1_000, 12_000_000),
                    ordered=rng.random() < 0.7)
    return dict(what="dsmc", ni=size(9, 129), nj=size(9, 129), nk=size(9, 129), ppc=rng.randint(4, 32))


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
class State:
    """A world and what a pass needs with it; the world is closed with the state."""

    def __init__(self, case, world=None, **more):
        self.case, self.world = case, world
        self.__dict__.update(more)

    def __del__(self):
        if self.world is not None:
            self.world.close()


def gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def shape(case):
    return case["ni"], case["nj"], case["nk"]


def sigma_tables():
    """Synthetic O2 collision table: elastic 6e-20/sqrt(1+E/10eV) m^2 plus Lotz ionisation."""
    E = np.geomspace(0.01, 1e5, 400)
    x = E / LOTZ["I"]
    ion = np.where(E > LOTZ["I"], LOTZ["A"] * np.log(np.maximum(x, 1)) / (E * LOTZ["I"]) *
                   (1 - LOTZ["b"] * np.exp(-LOTZ["c"] * (x - 1))), 0.0)
    return E, 6e-20 / np.sqrt(1 + E / 10.0) + ion


def prepare(case, seed):
    return {"loop": prepare_loop, "trace": prepare_trace, "poisson": prepare_poisson, "moments": prepare_moments,
            "density": prepare_density, "dsmc": prepare_dsmc}[case["what"]](case, seed)


def prepare_loop(case, seed):
    nn = shape(case)
    if case["solver"] != "learned":
        return prepare_plain(case, seed)
    inst, n = case["instances"], case["n"]
    nx = max(nn[0], nn[1]) - 1
    L = (case["side"] * (nn[0] - 1) / nx, case["side"] * (nn[1] - 1) / nx, 0.08)
    dz = L[2] / (nn[2] - 1)
    nk = nn[2] * max(1, inst)
    W = pic.World(nn[0], nn[1], nk, (0.0, 0.0, 0.0), (L[0], L[1], (nk - 1) * dz))
    W.set_boundaries((1, 1, 0), (1,) * 6, (0, 0, 0, 0, 0.0, 0.0 if inst else case["volts"]))
    if inst:
        W.set_slabs(np.zeros(inst), np.linspace(200.0, 800.0, inst))
    W.setTime(case["dt"], 1 << 30)
    band = 1e13 * L[0] * L[1] * 0.4 * L[2]  # real particles of an instance at 1e13 m^-3
    if inst:
        r = np.random.default_rng(seed)
        counts = np.exp(r.uniform(np.log(n / 30.0), np.log(3.0 * n), inst)).astype(np.int64)
    else:
        counts = np.array([n])
    w_mean = float(np.median(band / counts))
    cap = int(counts.sum() * 1.25) + 8192
    bound = cap * w_mean * 400.0
    e = pic.Species("e-", pic.ME, -pic.QE, W, w_mean, capacity=cap, weight_bound=bound)
    i = pic.Species("O2+", 32 * pic.AMU, pic.QE, W, w_mean, capacity=cap, weight_bound=bound)
    for k, c in enumerate(counts):
        z0 = k * nn[2] * dz
        lo, hi = (0.0, 0.0, z0 + 0.3 * L[2]), (L[0], L[1], z0 + 0.7 * L[2])
        e.loadUniform(lo, hi, int(c), 2.0 * EV_K, band / c, 0.5, seed=2 * (1000 * seed + k) + 1)
        i.loadUniform(lo, hi, int(c), 0.03 * EV_K, band / c, 0.5, seed=2 * (1000 * seed + k) + 2)
    tE, tS = sigma_tables()
    M = pic.MC_MEX_Ionization(e, i, W, case["gas"], 300.0, 32 * pic.AMU, LOTZ["I"], tE, tS, sigma_ion_kind=1,
                              sigma_ion_params=(LOTZ["A"], LOTZ["b"], LOTZ["c"], 0.0), seed=seed + 1)
    if inst:
        M.set_slab_density(np.geomspace(5e20, 2e21, inst))
    S = pic.PotentialSolver(W, 20000, 1e-6, pic.SOLVER_LEARNED, stop=pic.STOP_REL_CHARGE)
    S.setWarmStart(pic.WARM_EXTRAPOLATE)
    S.setWarmJacobi(0)
    W.configure_loop(solve_each_step=True, sort_every=20, merge_every=20, merge_after=0, merge_min=64)
    S.solve(raise_on_fail=True)
    S.computeEF()
    # the preconditioner's level gains from the first steps' solves
    lp = pic.LearnedPreconditioner(W)
    lp.collect(True)
    for _ in range(3):
        W.step()
    lp.collect(False)
    lp.calibrate()
    for _ in range(3):
        W.step()
    W.synchronize()
    return State(case, W, species=(e, i), mcc=M, solver=S)


def prepare_plain(case, seed):
    nn = shape(case)
    W = pic.World(*nn, (0.0, 0.0, 0.0), tuple(0.01 * (k - 1) for k in nn))
    W.dirichletBoundries(0.0)
    W.setTime(5e-12, 1 << 30)
    n = case["n"]
    L = W.xm - W.x0
    w = 1e11 * float(np.prod(L)) / n
    cap = n + 4096
    e = pic.Species("e-", pic.ME, -pic.QE, W, w, capacity=cap)
    i = pic.Species("O+", 16 * pic.AMU, pic.QE, W, w, capacity=cap)
    e.loadUniform(W.x0, W.xm, n, EV_K, w, 0.0, seed=2 * seed + 1)
    i.loadUniform(W.x0, W.xm, n, 0.1 * EV_K, w, 0.0, seed=2 * seed + 2)
    if case["solver"] == "gs":
        S = pic.PotentialSolver(W, 10000, 1e-4, pic.GS, omega=1.4, stop=pic.STOP_ABS_RMS)
    else:
        S = pic.PotentialSolver(W, 10000, 1e-6, pic.PCG)
    W.configure_loop(solve_each_step=True, sort_every=20)
    for _ in range(3):
        W.step()
    W.synchronize()
    return State(case, W, species=(e, i), mcc=None, solver=S)


def trace_world(case):
    return (0.0, 0.0, 0.0), tuple(1e-3 * (k - 1) for k in shape(case))


def trace_field(case):
    """The frozen field on the nodes (FP32 values): a standing wave that confines along z."""
    ni, nj, nk = shape(case)
    x, y, z = (torch.arange(k, device="cuda", dtype=torch.float64) / (k - 1) for k in (ni, nj, nk))
    tau = 2 * math.pi
    E = torch.empty(nk, nj, ni, 3, device="cuda", dtype=torch.float64)
    E[..., 0] = 50.0 * torch.sin(tau * x)[None, None, :] * torch.cos(math.pi * z)[:, None, None]
    E[..., 1] = 50.0 * torch.sin(tau * y)[None, :, None] * torch.cos(math.pi * z)[:, None, None]
    E[..., 2] = 80.0 * torch.sin(math.pi * z)[:, None, None] * torch.cos(tau * x)[None, None, :]
    return E.reshape(-1, 3).float()


TRACE_SPECIES = (("e-", pic.ME, -pic.QE, 2.0), ("O2+", 32 * pic.AMU, pic.QE, 0.03))
TRACE_DT = 5e-12


def trace_particles(case, seed, k):
    """Positions, velocities and lognormal weights of species k, in cell order."""
    g = gen(10 * seed + k)
    n = case["n"]
    x0, xm = trace_world(case)
    L = torch.tensor(xm, device="cuda", dtype=torch.float64)
    pos = torch.rand(n, 3, device="cuda", dtype=torch.float64, generator=g) * L
    c = (pos / 1e-3).floor().long()
    order = torch.argsort((c[:, 2] * (case["nj"] - 1) + c[:, 1]) * (case["ni"] - 1) + c[:, 0])
    pos = pos[order].contiguous()
    del c, order
    _, mass, _, T = TRACE_SPECIES[k]
    vth = math.sqrt(pic.QE * T / mass)
    vel = torch.randn(n, 3, device="cuda", generator=g).mul_(vth).double()
    w = torch.exp(0.5 * torch.randn(n, device="cuda", generator=g) - 0.125).mul_(50.0).double()
    return pos, vel, w


def prepare_trace(case, seed):
    x0, xm = trace_world(case)
    W = pic.World(*shape(case), x0, xm)
    W.set_boundaries((1, 1, 0), (1,) * 6, (0.0,) * 6)
    W.setTime(TRACE_DT, 1 << 30)
    W.ef = trace_field(case).double().cpu().numpy()
    W.configure_loop(solve_each_step=False, sort_every=20)
    sp = [pic.Species(name, mass, q, W, 50.0, capacity=case["n"] + 1024) for name, mass, q, _ in TRACE_SPECIES]
    parts = [trace_particles(case, seed, k) for k in range(len(sp))]
    torch.cuda.synchronize()
    W.add_particles_batch(sp, *zip(*parts), rewind=False, sort=False)
    return State(case, W, species=sp)


def blob_rho(case, seed):
    """Seeded sum of 8-64 Gaussian blobs (amplitude +-1e-3 C/m^3, widths 2-20 cells), FP32 values."""
    nn = shape(case)
    r = np.random.default_rng(seed)
    ax = [torch.arange(k, device="cuda", dtype=torch.float64) for k in nn]
    rho = torch.zeros(nn[2], nn[1], nn[0], device="cuda", dtype=torch.float64)
    for _ in range(int(r.integers(8, 65))):
        c = r.uniform(0, 1, 3) * (np.array(nn) - 1)
        wd = r.uniform(2, min(20.0, 0.25 * min(nn)))
        amp = r.uniform(-1e-3, 1e-3)
        lo = np.maximum(0, np.floor(c - 4 * wd)).astype(int)
        hi = np.minimum(np.array(nn), np.ceil(c + 4 * wd + 1)).astype(int)
        gx, gy, gz = [torch.exp(-0.5 * ((ax[d][lo[d]:hi[d]] - float(c[d])) / wd) ** 2) for d in range(3)]
        rho[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]] += amp * gz[:, None, None] * gy[None, :, None] * gx[None, None, :]
    return rho.float()


POISSON_DX, POISSON_V = 1.5625e-4, 1000.0


def prepare_poisson(case, seed):
    nn = shape(case)
    per = int(case["periodic"])
    W = pic.World(*nn, (0.0, 0.0, 0.0), tuple(POISSON_DX * (k - 1) for k in nn))
    W.set_boundaries((per, per, 0), (1,) * 6, (0, 0, 0, 0, 0.0, POISSON_V))
    phi0 = W.phi
    omega = 2.0 / (1.0 + math.sin(math.pi / (max(nn) - 1)))
    method = {"gs": pic.GS, "pcg": pic.PCG, "learned": pic.SOLVER_LEARNED}[case["solver"]]
    S = pic.PotentialSolver(W, 100000, 1e-8, method, omega=omega, stop=pic.STOP_REL_CHARGE)
    if case["solver"] == "learned":
        lp = pic.LearnedPreconditioner(W)
        lp.collect(True)
        W.rho = blob_rho(case, seed + 7001).double().cpu().numpy().ravel()
        S.solve(raise_on_fail=True)
        lp.collect(False)
        lp.calibrate()
    return State(case, W, solver=S, rho=blob_rho(case, seed).double().cpu().numpy().ravel(), phi0=phi0)


MOMENT_M, MOMENT_T, MOMENT_DT = 16 * pic.AMU, 300.0, 2e-7


def moment_particles(case, seed):
    """A drifting gas at 300 K in a periodic box, FP32 velocities, one weight."""
    g = gen(seed)
    n = case["n"]
    _, xm = trace_world(case)
    L = torch.tensor(xm, device="cuda", dtype=torch.float64)
    pos = torch.rand(n, 3, device="cuda", dtype=torch.float64, generator=g) * L
    vel = torch.randn(n, 3, device="cuda", generator=g).mul_(math.sqrt(pic.KB * MOMENT_T / MOMENT_M))
    vel[:, 0] += 300.0
    vel[:, 1] += 200.0 * torch.sin(2 * math.pi * pos[:, 2] / L[2]).float()
    return pos, vel.double(), torch.full((n,), 1e6, device="cuda", dtype=torch.float64)


def prepare_moments(case, seed):
    x0, xm = trace_world(case)
    W = pic.World(*shape(case), x0, xm)
    W.set_boundaries((1, 1, 1), (0,) * 6, (0.0,) * 6)
    W.setTime(MOMENT_DT, 1 << 30)
    sp = pic.Species("O", MOMENT_M, 0.0, W, 1e6, capacity=case["n"] + 1024)
    pos, vel, w = moment_particles(case, seed)
    torch.cuda.synchronize()
    W.add_particles_batch([sp], [pos], [vel], [w], rewind=False, sort=True)
    return State(case, W, species=[sp])


def density_arrays(case, seed):
    """The caller's arrays: cell and in-cell offsets, velocity and weight (float4 each)."""
    g = gen(seed)
    n = case["n"]
    c = [torch.randint(0, k - 1, (n,), device="cuda", generator=g, dtype=torch.int32) for k in shape(case)]
    if case["ordered"]:
        order = torch.argsort((c[2].long() * case["nj"] + c[1]) * case["ni"] + c[0])
        c = [a[order] for a in c]
    pos = torch.rand(n, 4, device="cuda", generator=g)
    pos.view(torch.int32)[:, 3] = c[0] | (c[1] << 9) | (c[2] << 18)
    vel = torch.randn(n, 4, device="cuda", generator=g)
    vel[:, 3] = 20.0 * torch.exp(0.5 * torch.randn(n, device="cuda", generator=g))
    return pos, vel, c


DENSITY_SCALE, DENSITY_L = 2.0**20, 0.05


def prepare_density(case, seed):
    pos, vel, _ = density_arrays(case, seed)
    out = torch.empty(case["nk"], case["nj"], case["ni"], device="cuda")
    torch.cuda.synchronize()
    return State(case, None, lib=pic.library(), pos=pos, vel=vel, out=out, x0=np.zeros(3),
                 xm=np.full(3, DENSITY_L), periodic=np.array([1, 1, 0], np.int32))


def prepare_dsmc(case, seed):
    nn = shape(case)
    W = pic.World(*nn, (0.0, 0.0, 0.0), tuple(1e-3 * (k - 1) for k in nn))
    W.set_boundaries((1, 1, 1), (0,) * 6, (0.0,) * 6)
    W.setTime(1e-6, 1 << 30)
    n = int(W.num_cells * case["ppc"])
    sp = pic.Species("O", 16 * pic.AMU, 0.0, W, 1e12 / case["ppc"], capacity=n + 1024)
    sp.loadUniform(W.x0, W.xm, n, 300.0, sp.mpw0, 0.0, seed=seed + 1)
    D = pic.DSMC_MEX(sp, W, seed=seed + 1)
    for _ in range(3):  # (sigma v)_max settles
        D.apply(1e-6)
    W.synchronize()
    return State(case, W, species=[sp], dsmc=D)


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
def run(state):
    case, W = state.case, state.world
    what = case["what"]
    if what == "loop":
        # a row of runtime_diags.csv per step: micro count, momentum and kinetic energy of each
        # species, the field energy; the file keeps seven digits
        rows = np.empty((case["steps"], 11), np.float32)
        for k in range(case["steps"]):
            W.step()
            rows[k, :5] = state.species[0].sums()
            rows[k, 5:10] = state.species[1].sums()
            rows[k, 10] = W.getPE()
        if not case["fields"]:
            return {"diags": rows}
        return {"diags": rows, "phi": W.phi.astype(np.float32), "rho": W.rho.astype(np.float32)}
    if what == "trace":
        for _ in range(TRACE_STEPS):
            W.step()
            for s in state.species:
                s.updateAverages()
        return [s.den_avg.astype(np.float32) for s in state.species]
    if what == "poisson":
        W.rho = state.rho
        W.phi = state.phi0
        state.solver.solve(raise_on_fail=True)
        out = {"phi": W.phi.astype(np.float32)}
        if case["field"]:
            state.solver.computeEF()
            out["ef"] = W.ef.astype(np.float32)
        return out
    if what == "moments":
        sp = state.species[0]
        sp.clearSamples()
        for _ in range(MOMENT_STEPS):
            sp.sampleMoments()
            sp.advance(MOMENT_DT, deposit=False)
        sp.sortIndexes()  # the gas moved: back into cell order
        vel, T = sp.computeGasProperties()
        return {"vel": vel.astype(np.float32), "T": T.astype(np.float32)}
    if what == "density":
        rc = state.lib.pic_number_density_noalloc(
            case["ni"], case["nj"], case["nk"], state.x0.ctypes.data, state.xm.ctypes.data, state.periodic.ctypes.data,
            state.pos.data_ptr(), state.vel.data_ptr(), case["n"], DENSITY_SCALE, state.out.data_ptr(),
            torch.cuda.current_stream().cuda_stream)
        if rc != pic.PIC_OK:
            raise RuntimeError("pic_number_density_noalloc: %d" % rc)
        return state.out
    sp = state.species[0]
    for _ in range(DSMC_CALLS):
        state.dsmc.apply(1e-6)
    return {"sums": sp.sums(), "counts": sp.computeMacroParticlesCount()}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def work(case):
    """Bytes: particles 60 B a push (32 read, 28 written), 8 B of id where collisions are drawn,
    20 B a node and species of E and density; 8 B a node of rho and phi in and out of every solve's
    iteration at the method's minimum (12 B a sweep, 40 B a PCG and 56 B a learned iteration) for
    the iterations that such a solve takes; host arrays 8 B a value."""
    nn = shape(case)
    nv = nn[0] * nn[1] * nn[2]
    what = case["what"]
    if what == "loop":
        inst = max(1, case["instances"])
        n, nodes, steps = 2 * case["n"] * inst, nv * inst, case["steps"]
        per_node = {"gs": 12.0 * 25, "pcg": 40.0 * 20, "learned": 56.0 * 10}[case["solver"]] + 2 * 20.0 + 4 + 24 + 2 * 24
        b = steps * (60.0 * n + 16.0 * n + (4.0 * n if case["solver"] == "learned" else 0.0) + per_node * nodes)
        f = steps * (120.0 * n + {"gs": 350.0, "pcg": 400.0, "learned": 1500.0}[case["solver"]] * nodes)
        return {"bytes": b, "flops": f}
    if what == "trace":
        n = 2 * case["n"]
        return {"bytes": TRACE_STEPS * (60.0 * n + 2 * (20.0 + 12.0) * nv) + 2 * 8.0 * nv, "flops": TRACE_STEPS * 120.0 * n}
    if what == "poisson":
        m = max(nn)
        its = {"gs": 6.0 * m, "pcg": 6.0 * m, "learned": 40.0}[case["solver"]]
        per, fl = {"gs": (12.0, 14.0), "pcg": (40.0, 24.0), "learned": (56.0, 130.0)}[case["solver"]]
        return {"bytes": nv * (its * per + 4 * 24.0 + 3 * 8.0 + (24.0 if case["field"] else 0.0)),
                "flops": nv * (its * fl + 4 * 160.0)}
    if what == "moments":
        n = case["n"]
        return {"bytes": MOMENT_STEPS * (32.0 * n + 60.0 * n + 7 * 8.0 * nv) + 80.0 * n + 7 * 4.0 * nv + 32.0 * nv,
                "flops": MOMENT_STEPS * 200.0 * n}
    if what == "density":
        return {"bytes": 20.0 * case["n"] + 4.0 * nv, "flops": 32.0 * case["n"]}
    cells = (nn[0] - 1) * (nn[1] - 1) * (nn[2] - 1)
    n = cells * case["ppc"]
    return {"bytes": DSMC_CALLS * 32.0 * n + 16.0 * n + 4.0 * cells, "flops": DSMC_CALLS * 60.0 * n}


# ------------------------------------------------------------------------------------------
# 64-bit answers
# ------------------------------------------------------------------------------------------
def exact(case, seed):
    what = case["what"]
    if what == "trace":
        return exact_trace(case, seed)
    if what == "poisson":
        return exact_poisson(case, seed)
    if what == "moments":
        return exact_moments(case, seed)
    if what == "density":
        return exact_density(case, seed)
    return None  # the loop's stochastic state, and collisions drawn in an order of its own


def corners(nn, c, f):
    """(node, weight) of the eight corners of cells c (n, 3) at offsets f (n, 3)."""
    for k in range(8):
        b = [(k >> d) & 1 for d in range(3)]
        w = 1.0
        for d in range(3):
            w = w * (f[:, d] if b[d] else 1.0 - f[:, d])
        yield ((c[:, 2] + b[2]) * nn[1] + c[:, 1] + b[1]) * nn[0] + c[:, 0] + b[0], w


def node_density(acc, nn, periodic, cell_volume):
    """Weights summed on the nodes -> number density (periodic copies folded, half cells at walls)."""
    a = acc.reshape(nn[2], nn[1], nn[0]).clone()
    for d in range(3):
        ax = 2 - d
        lo, hi = a.select(ax, 0), a.select(ax, nn[d] - 1)
        if periodic[d]:
            s = lo + hi
            lo.copy_(s)
            hi.copy_(s)
        else:
            lo.mul_(2.0)
            hi.mul_(2.0)
    return a.reshape(-1) / cell_volume


def exact_trace(case, seed):
    nn = shape(case)
    nc = torch.tensor([k - 1 for k in nn], device="cuda", dtype=torch.float64)
    E = trace_field(case).double()
    nv = nn[0] * nn[1] * nn[2]
    out = []
    for k, (_, mass, q, _) in enumerate(TRACE_SPECIES):
        pos, vel, w = trace_particles(case, seed, k)
        avg = torch.zeros(nv, device="cuda", dtype=torch.float64)
        piece = 2_000_000
        for a in range(0, case["n"], piece):
            x, v, ww = pos[a:a + piece] / 1e-3, vel[a:a + piece].clone(), w[a:a + piece]
            for _ in range(TRACE_STEPS):
                c = torch.minimum(x.floor(), nc - 1).long()
                f = x - c
                e = 0.0
                for node, wt in corners(nn, c, f):
                    e = e + E[node] * wt[:, None]
                v = v + (q / mass * TRACE_DT) * e
                x = x + v * (TRACE_DT / 1e-3)
                x[:, :2] = torch.remainder(x[:, :2], nc[:2])
                live = (x[:, 2] >= 0) & (x[:, 2] < nc[2])
                if not bool(live.all()):
                    x, v, ww = x[live], v[live], ww[live]
                c = torch.minimum(x.floor(), nc - 1).long()
                for node, wt in corners(nn, c, x - c):
                    avg.index_add_(0, node, wt * ww)
        out.append(node_density(avg / TRACE_STEPS, nn, (1, 1, 0), 1e-9))
        del pos, vel, w
    return out


def exact_poisson(case, seed):
    """The discrete system solved by sine transforms between walls and Fourier transforms along
    periodic axes."""
    nn = shape(case)
    per = case["periodic"]
    eps0 = pic.EPS0
    h2 = POISSON_DX**2
    rho = blob_rho(case, seed).double()
    if per:
        b = rho[1:-1, :-1, :-1] / eps0
    else:
        b = rho[1:-1, 1:-1, 1:-1] / eps0
    b = b.clone()
    b[-1] += POISSON_V / h2

    def sine(a, ax):  # DST-I along an axis
        m = a.shape[ax]
        z = torch.zeros([1 if d == ax else a.shape[d] for d in range(3)], device=a.device, dtype=a.dtype)
        ext = torch.cat([z, a, z, -a.flip(ax)], ax)
        return torch.fft.fft(ext, dim=ax).narrow(ax, 1, m).mul(0.5j)

    def both(a, forward):
        a = a.to(torch.complex128)
        for ax in range(3):
            if per and ax > 0:
                a = torch.fft.fft(a, dim=ax) if forward else torch.fft.ifft(a, dim=ax)
            else:
                m = a.shape[ax]
                a = sine(a, ax)
                if not forward:
                    a = a * (2.0 / (m + 1))
        return a

    lam = 0.0
    for ax in range(3):
        m = b.shape[ax]
        t = torch.arange(m, device="cuda", dtype=torch.float64)
        ang = 2 * math.pi * t / m if (per and ax > 0) else math.pi * (t + 1) / (m + 1)
        lam = lam + ((2.0 - 2.0 * torch.cos(ang)) / h2).reshape([m if d == ax else 1 for d in range(3)])
    x = both(both(b, True) / lam, False).real
    phi = torch.zeros(nn[2], nn[1], nn[0], device="cuda", dtype=torch.float64)
    phi[-1] = POISSON_V
    if per:
        phi[1:-1, :-1, :-1] = x
        phi[:, -1, :] = phi[:, 0, :]
        phi[:, :, -1] = phi[:, :, 0]
    else:
        phi[1:-1, 1:-1, 1:-1] = x
        phi[:, :, 0] = phi[:, :, -1] = 0.0  # the x walls, then the y walls, are set before the z walls
        phi[:, 0, :] = phi[:, -1, :] = 0.0
    out = {"phi": phi.reshape(-1)}
    if case["field"]:
        E = torch.zeros(nn[2], nn[1], nn[0], 3, device="cuda", dtype=torch.float64)
        for d in range(3):
            p = phi.movedim(2 - d, 0)
            e = torch.empty_like(p)
            e[1:-1] = p[:-2] - p[2:]
            if per and d < 2:
                e[0] = p[-2] - p[1]
                e[-1] = e[0]
            else:
                e[0] = 3 * p[0] - 4 * p[1] + p[2]
                e[-1] = -(p[-3] - 4 * p[-2] + 3 * p[-1])
            E[..., d] = (e / (2 * POISSON_DX)).movedim(0, 2 - d)
        out["ef"] = E.reshape(-1, 3)
    return out


def exact_moments(case, seed):
    nn = shape(case)
    nc = torch.tensor([k - 1 for k in nn], device="cuda", dtype=torch.float64)
    nv = nn[0] * nn[1] * nn[2]
    pos, vel, w = moment_particles(case, seed)
    m = torch.zeros(7, nv, device="cuda", dtype=torch.float64)
    x = pos / 1e-3
    for k in range(MOMENT_STEPS):
        y = torch.remainder(x + vel * (k * MOMENT_DT / 1e-3), nc)
        c = torch.minimum(y.floor(), nc - 1).long()
        for node, wt in corners(nn, c, y - c):
            ww = wt * w
            m[0].index_add_(0, node, ww)
            for d in range(3):
                m[1 + d].index_add_(0, node, ww * vel[:, d])
                m[4 + d].index_add_(0, node, ww * vel[:, d] ** 2)
    n = torch.where(m[0] > 0, m[0], torch.ones_like(m[0]))
    u = m[1:4] / n
    T = MOMENT_M / (2 * pic.KB) * (m[4:7] / n - u**2).sum(0)
    return {"vel": u.t().contiguous(), "T": T}


def exact_density(case, seed):
    nn = shape(case)
    pos, vel, c = density_arrays(case, seed)
    acc = torch.zeros(nn[0] * nn[1] * nn[2], device="cuda", dtype=torch.float64)
    w = vel[:, 3].double()
    cc = torch.stack([a.long() for a in c], 1)
    for node, wt in corners(nn, cc, pos[:, :3].double()):
        acc.index_add_(0, node, wt * w)
    vol = 1.0
    for k in nn:
        vol *= DENSITY_L / (k - 1)
    return node_density(acc, nn, (1, 1, 0), vol).reshape(nn[2], nn[1], nn[0])
