"""The workloads that the framework's speed is judged on.

Every case is a run as a user's program makes one: a solver built from a
config and a mesh, its state set from the host, so many Runge-Kutta steps, the
state read back (or one right-hand side and the dQ read back; or a burst of
requests through the serving loop).  A pass restarts from the same state, so
passes are alike however often they are repeated.

The kinds, each over the sizes its users run:

  tgv      the Taylor-Green vortex, one calorically perfect gas, kepaec
  mix      two or three calorically perfect species, MUSCL or kepaec
  react    H2/air (9 species) or CH4/O2 (12), thermally perfect, kinetic
           theory, finite-rate chemistry
  layer    the transcritical O2/H2 mixing layer, Peng-Robinson, double flux
  channel  the channel with an inflow, an exit and two walls, two species
  pool     independent reactors and 1-D domains through the serving pool

``exact`` works the same answer out in plain torch, float64, on one global
padded grid; it shares nothing with the library but the inputs (meshes,
fields, the stored tables of species data).
"""

import math
import os

import numpy as np
import torch

import peregrine_b200 as pg
from peregrine_b200 import cases as library
from peregrine_b200 import native, serving
from peregrine_b200.mesher import CubeMesher

NG = 2
RU = 8314.46261815324
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

LISTED = [
    # the smallest run: one 32^3 block, launches and latency count
    dict(name="tgv-32", kind="tgv", nx=32, ny=32, nz=32, bi=1, bj=1, bk=1, simulator="navier-stokes",
         integrator="rk4", controller="fixed", jostle=0.0, steps=10, op="step"),
    # the production size: 128^3 in 27 uneven blocks
    dict(name="tgv-128-27blocks", kind="tgv", nx=128, ny=128, nz=128, bi=3, bj=3, bk=3, simulator="navier-stokes",
         integrator="rk4", controller="fixed", jostle=0.0, steps=20, op="step"),
    # inviscid, odd extents, uneven blocks, the step size taken from the flow
    dict(name="tgv-euler-cfl-ragged", kind="tgv", nx=61, ny=75, nz=47, bi=2, bj=1, bk=2, simulator="euler",
         integrator="tvd-rk3", controller="cfl", jostle=0.0, steps=10, op="step"),
    # a grid that is no lattice of boxes: every metric array is read
    dict(name="tgv-curvilinear-64", kind="tgv", nx=64, ny=64, nz=64, bi=2, bj=2, bk=1, simulator="navier-stokes",
         integrator="rk4", controller="fixed", jostle=0.1, steps=10, op="step"),
    # a right-hand side alone, as a caller with its own integrator asks for it
    dict(name="mix-rhs-40", kind="mix", nx=40, ny=40, nz=40, bi=2, bj=2, bk=2, species=3, primary="hllc",
         recon="muscl", simulator="navier-stokes", integrator="rk4", jostle=0.0, steps=1, op="rhs"),
    # two species on a curvilinear grid of odd extents
    dict(name="mix-curvilinear-53", kind="mix", nx=53, ny=45, nz=61, bi=1, bj=2, bk=1, species=2, primary="hllc",
         recon="muscl", simulator="navier-stokes", integrator="tvd-rk3", jostle=0.1, steps=5, op="step"),
    # the reacting field at its full size
    dict(name="react-h2-96", kind="react", gas="h2o2_gri30", nx=96, ny=96, nz=96, bi=1, bj=1, bk=1, primary="hllc",
         recon="muscl", integrator="tvd-rk3", steps=5, op="step"),
    # a small ragged reacting box in two blocks
    dict(name="react-h2-ragged", kind="react", gas="h2o2_gri30", nx=37, ny=29, nz=23, bi=2, bj=1, bk=1,
         primary="hllc", recon="muscl", integrator="tvd-rk3", steps=5, op="step"),
    # the widest mechanism: 12 species, 38 reactions
    dict(name="react-ch4-48", kind="react", gas="ch4_o2_ffcmy", nx=48, ny=48, nz=48, bi=1, bj=2, bk=1, primary="hllc",
         recon="muscl", integrator="tvd-rk3", steps=3, op="step"),
    # the real gas with the double flux, eight uneven blocks
    dict(name="layer-256x128x4", kind="layer", nx=256, ny=128, nz=4, bi=8, integrator="tvd-rk3", steps=20, op="step"),
    # a bounded domain under the cfl controller
    dict(name="channel-192x96x96", kind="channel", nx=192, ny=96, nz=96, bi=2, bj=2, bk=2, steps=5, op="step"),
    # a burst of requests served by one pool
    dict(name="pool-32", kind="pool", requests=32, nmin=64, nmax=2048, steps=20),
]


def listed():
    return [dict(c) for c in LISTED]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("tgv", "tgv", "mix", "react", "react", "layer", "channel", "pool"))
    if kind == "tgv":
        c = dict(nx=size(16, 112), ny=size(16, 112), nz=size(16, 112), bi=rng.randint(1, 3), bj=rng.randint(1, 2),
                 bk=rng.randint(1, 3), simulator=rng.choice(("navier-stokes", "navier-stokes", "euler")),
                 integrator=rng.choice(("rk4", "tvd-rk3", "rk2")), controller=rng.choice(("fixed", "cfl")),
                 jostle=rng.choice((0.0, 0.0, 0.1)), steps=rng.randint(5, 15), op=rng.choice(("step", "step", "rhs")))
    elif kind == "mix":
        primary = rng.choice(("hllc", "kepaec", "rusanov"))
        c = dict(nx=size(16, 80), ny=size(16, 80), nz=size(16, 80), bi=rng.randint(1, 2), bj=rng.randint(1, 3),
                 bk=rng.randint(1, 2), species=rng.randint(2, 3), primary=primary,
                 recon="constant" if primary == "kepaec" else "muscl",
                 simulator=rng.choice(("navier-stokes", "navier-stokes", "euler")),
                 integrator=rng.choice(("rk4", "tvd-rk3")), jostle=rng.choice((0.0, 0.0, 0.1)),
                 steps=rng.randint(2, 8), op=rng.choice(("step", "step", "rhs")))
    elif kind == "react":
        gas = rng.choice(("h2o2_gri30", "h2o2_gri30", "ch4_o2_ffcmy"))
        primary = rng.choice(("hllc", "hllc", "kepaec"))
        c = dict(gas=gas, nx=size(12, 64), ny=size(12, 64), nz=size(12, 64), bi=rng.randint(1, 2),
                 bj=rng.randint(1, 2), bk=rng.randint(1, 2), primary=primary,
                 recon="constant" if primary == "kepaec" else "muscl", integrator="tvd-rk3",
                 steps=rng.randint(1, 5), op=rng.choice(("step", "step", "rhs")))
    elif kind == "layer":
        c = dict(nx=size(48, 320), ny=size(32, 160), nz=rng.randint(2, 6), bi=rng.randint(1, 8),
                 integrator="tvd-rk3", steps=rng.randint(5, 20), op="step")
    elif kind == "channel":
        c = dict(nx=size(24, 128), ny=size(24, 96), nz=size(16, 96), bi=rng.randint(1, 2), bj=rng.randint(1, 2),
                 bk=rng.randint(1, 2), steps=rng.randint(2, 6), op="step")
    else:
        c = dict(requests=rng.randint(1, 40), nmin=rng.randint(32, 96), nmax=rng.randint(256, 2048),
                 steps=rng.randint(5, 25))
    return dict(kind=kind, **c)


###############################################################################
# meshes, configs and fields: the inputs, from the seed alone
###############################################################################
TWO_PI = 2.0 * math.pi
REACT_DX = 1e-4     # m a cell
LAYER_DX = 2e-5


def cuts(n, blocks, seed):
    """n cells in so many blocks of uneven widths."""
    if blocks == 1:
        return [n]
    rng = np.random.default_rng(seed)
    share = rng.uniform(0.8, 1.2, blocks)
    out = np.maximum(4, np.floor(n * share / share.sum())).astype(int)
    while out.sum() > n:
        out[np.argmax(out)] -= 1
    out[np.argmin(out)] += n - out.sum()
    return [int(x) for x in out]


def mesh_of(case):
    kind = case["kind"]
    n = [case["nx"], case["ny"], case["nz"]]
    b = [case["bi"], case.get("bj", 1), case.get("bk", 1)]
    cells = [cuts(n[a], b[a], 10 + a) for a in range(3)]
    if kind in ("tgv", "mix"):
        lengths = [TWO_PI] * 3
    elif kind == "react":
        lengths = [REACT_DX * m for m in n]
    elif kind == "layer":
        lengths = [LAYER_DX * m for m in n]
    else:
        lengths = list(library.CHANNEL_LENGTHS)
    if kind == "channel":
        return CubeMesher(mbdims=b, cells=cells, lengths=lengths, periodic=[False, False, True],
                          bcnames={1: "inflow", 2: "exit", 3: "floor", 4: "lid"})
    return CubeMesher(mbdims=b, cells=cells, lengths=lengths, periodic=[True] * 3, jostle=case.get("jostle", 0.0))


def config_of(case):
    kind = case["kind"]
    if kind == "tgv":
        return library.tgv_config(case["simulator"], case["integrator"], "batched")
    if kind == "mix":
        return library.mixing_config(case["simulator"], case["integrator"], case["primary"], case["recon"],
                                     "koren" if case["recon"] == "muscl" else None, case["species"], "batched")
    if kind == "react":
        return library.reacting_config("navier-stokes", case["integrator"], case["primary"], case["recon"],
                                       "koren" if case["recon"] == "muscl" else None, True, case["gas"], "batched")
    if kind == "layer":
        return library.mixing_layer_config("pr", "euler-df", case["integrator"], "batched")
    return library.channel_config("batched")


def centres(case):
    """The uniform lattice's cell centres, three arrays that broadcast."""
    n = [case["nx"], case["ny"], case["nz"]]
    L = mesh_of(dict(case, jostle=0.0)).lengths
    x = [(np.arange(m) + 0.5) * (ln / m) for m, ln in zip(n, L)]
    return x[0][:, None, None], x[1][None, :, None], x[2][None, None, :]


def table(case):
    """A stored table set: the species data of a gas, read as a file."""
    name = case["gas"] if case["kind"] == "react" else "h2o2_gri30" if case["kind"] == "pool" else "o2_h2_pr"
    with np.load(os.path.join(ROOT, "peregrine_b200", "data", f"{name}.npz")) as z:
        return {k: z[k] for k in z.files}


def composition(tab, gas):
    """Stoichiometric H2/air or CH4/O2, by mass."""
    names = [str(s) for s in tab["spnames"]]
    moles = {"H2": 2.0, "O2": 1.0, "N2": 3.76} if gas == "h2o2_gri30" else {"CH4": 1.0, "O2": 2.0}
    Y = np.array([moles.get(s, 0.0) for s in names]) * tab["MW"]
    return Y / Y.sum()


def fields(case, seed):
    """Primitives p, u, v, w, T, Y... over the whole lattice, (nx, ny, nz, ne)."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    x, y, z = centres(case)
    n = (case["nx"], case["ny"], case["nz"])
    if kind == "tgv":
        _, g = library.tgv_gas()
        q = np.empty(n + (5,))
        U0, rho0 = g["U0"], g["rho0"]
        q[..., 0] = library.P0 + rho0 * U0 ** 2 / 16.0 * (np.cos(2 * x) + np.cos(2 * y)) * (np.cos(2 * z) + 2.0)
        q[..., 1] = U0 * np.sin(x) * np.cos(y) * np.cos(z)
        q[..., 2] = -U0 * np.cos(x) * np.sin(y) * np.cos(z)
        q[..., 3] = 0.0
        q[..., 1:4] += 1e-2 * U0 * rng.standard_normal(n + (3,))
        q[..., 4] = library.T0 * q[..., 0] / library.P0
        return q
    if kind == "mix":
        # waves with a step in pressure, temperature and composition
        ns = case["species"]
        ph = rng.uniform(0.0, TWO_PI, 8)
        step = (x > math.pi).astype(float)
        q = np.empty(n + (4 + ns,))
        q[..., 0] = library.P0 * (1.0 + 0.2 * np.sin(x + ph[0]) * np.cos(y + ph[1]) + 0.5 * step)
        q[..., 1] = 150.0 * np.sin(x + ph[2]) * np.cos(z + ph[3])
        q[..., 2] = 60.0 * np.cos(y + ph[4])
        q[..., 3] = 45.0 * np.sin(z + ph[5]) * np.cos(x)
        q[..., 1:4] += 5.0 * rng.standard_normal(n + (3,))
        q[..., 4] = library.T0 * (1.0 + 0.2 * np.cos(x + ph[6]) * np.sin(z + ph[7]) + 0.4 * step)
        for s in range(ns - 1):
            q[..., 5 + s] = (0.6 - 0.2 * step) / (ns - 1) * (1.0 + 0.3 * np.sin((s + 1) * x + y + ph[s]))
        return q
    if kind == "react":
        # hot spots and a swirling velocity in the fresh mixture, radicals in traces
        tab = table(case)
        Y = composition(tab, case["gas"])
        ns = len(Y)
        L = [REACT_DX * m for m in n]
        T0, dT = (1000.0, 400.0) if case["gas"] == "h2o2_gri30" else (1400.0, 300.0)
        T = np.full(n, T0)
        for _ in range(4):
            c, a = rng.uniform(0.0, 1.0, 3) * L, rng.uniform(0.5, 1.0) * dT
            d = [v - cc for v, cc in zip((x, y, z), c)]
            d = [v - ln * np.round(v / ln) for v, ln in zip(d, L)]
            T += a * np.exp(-0.5 * (d[0] ** 2 + d[1] ** 2 + d[2] ** 2) / (8.0 * REACT_DX) ** 2)
        q = np.zeros(n + (4 + ns,))
        for _ in range(6):
            k = rng.integers(1, 4, 3) * rng.choice([-1, 1], 3)
            kv = TWO_PI * k / np.array(L)
            a = np.cross(kv, rng.normal(0.0, 1.0, 3))
            wave = np.cos(kv[0] * x + kv[1] * y + kv[2] * z + rng.uniform(0.0, TWO_PI))
            for m in range(3):
                q[..., 1 + m] += a[m] * wave
        q[..., 1:4] *= 10.0 / np.sqrt(np.mean(q[..., 1:4] ** 2))
        q[..., 0] = library.P0
        q[..., 4] = T
        for s in range(ns - 1):
            q[..., 5 + s] = Y[s] if Y[s] > 0.0 else 1e-5 * rng.uniform(0.5, 1.0, n)
        return q
    if kind == "layer":
        Ly, d, dU = LAYER_DX * n[1], 4.0 * LAYER_DX, 50.0
        f = 0.5 * (np.tanh((y - 0.25 * Ly) / d) - np.tanh((y - 0.75 * Ly) / d))
        q = np.zeros(n + (6,))
        q[..., 0] = 6e6
        q[..., 1] = -0.5 * dU + dU * f + 0.01 * dU * rng.standard_normal(n)
        q[..., 2] = 0.01 * dU * rng.standard_normal(n)
        q[..., 4] = 300.0 + (120.0 - 300.0) * f
        q[..., 5] = np.clip(f, 0.0, 1.0)
        return q
    # the channel: a developed profile with noise
    h = library.CHANNEL_LENGTHS[1]
    q = np.zeros(n + (6,))
    q[..., 0] = library.P0
    q[..., 1] = 30.0 + 30.0 * 4.0 * (y / h) * (1.0 - y / h)
    q[..., 1:4] += 2.0 * rng.standard_normal(n + (3,))
    q[..., 4] = 300.0 + 10.0 * np.cos(300.0 * z)
    q[..., 5] = 0.5 + 0.1 * np.sin(TWO_PI * x / library.CHANNEL_LENGTHS[0])
    return q


def step_size(case):
    """A step well inside the scheme's bound (the cfl cases take their own)."""
    kind = case["kind"]
    n = (case["nx"], case["ny"], case["nz"])
    if kind == "tgv":
        return 0.4 * TWO_PI / max(n) / 400.0
    if kind == "mix":
        return 0.3 * TWO_PI / max(n) / 1000.0
    if kind == "react":
        return 2e-8
    return 2e-9


CFL = 0.5


def places(mesh):
    """Each block's slices of the global lattice, in block order."""
    out = []
    for k in range(mesh.mbdims[2]):
        for j in range(mesh.mbdims[1]):
            for i in range(mesh.mbdims[0]):
                out.append(tuple(slice(int(mesh.starts[a][m]), int(mesh.starts[a][m + 1]))
                                 for a, m in enumerate((i, j, k))))
    return out


###############################################################################
# the pass
###############################################################################
def prepare(case, seed):
    if case["kind"] == "pool":
        return prepare_pool(case, seed)
    cfg, mesh = config_of(case), mesh_of(case)
    mb = pg.get_solver(cfg, mesh, pg.get_backend("cuda", cfg))
    q = fields(case, seed)
    prims = [np.asfortranarray(q[at]) for at in places(mesh)]
    mb.set_prims(prims)
    n = mb.ncells * mb.ne
    start = torch.empty(n, dtype=torch.float64, pin_memory=True)
    result = torch.empty(n, dtype=torch.float64, pin_memory=True)
    native.call("pgb_state_get", mb.case, 0, native_ptr(start), n)
    # the result's parts: every component of every block where that is few
    # arrays, else every block
    parts, at = [], 0
    split = len(mb.mesh_blocks) * mb.ne <= 60
    for b in mb.mesh_blocks:
        m = int(np.prod(b.cells))
        rows = result[at:at + m * mb.ne].view(mb.ne, m)
        parts += list(rows) if split else [rows]
        at += m * mb.ne
    return dict(kind=case["kind"], op=case["op"], mb=mb, prims=prims, start=start, result=result, parts=parts, n=n,
                dt=step_size(case), steps=case["steps"], cfl=cfl_of(case))


def cfl_of(case):
    return CFL if case["kind"] == "channel" or case.get("controller") == "cfl" else None


def native_ptr(t):
    import ctypes

    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def prepare_pool(case, seed):
    cfg = library.reacting_config("navier-stokes", "tvd-rk3", "hllc", "muscl", "koren", True)
    proto = pg.get_solver(cfg, library.reacting_mesh(4), pg.get_backend("cuda", cfg))
    reqs = pool_requests(case, seed)
    for r in reqs:
        if r.kind == "1d":
            serving.box_metrics(r.cells, r.lengths)
    pool = serving.Pool(proto, 2_000_000, 512)
    return dict(kind="pool", proto=proto, pool=pool, requests=reqs)


def pool_requests(case, seed):
    """The stream's kinds and sizes are the case's; what each request holds
    (composition, temperature, pressure, where its hot spot sits) the seed's."""
    tab = table(case)
    names = [str(s) for s in tab["spnames"]]
    reqs = serving.requests(case["requests"], 0.0, names, tab["MW"], seed=case["requests"], steps=case["steps"],
                            nmin=case["nmin"], nmax=case["nmax"])
    rng = np.random.default_rng(seed)
    for r in reqs:
        q = r.prims
        if r.kind == "0d":
            q[..., 0], q[..., 4] = rng.uniform(1.0, 40.0) * serving.ATM, rng.uniform(900.0, 1400.0)
            q[..., 5:] = serving.h2_air(names, tab["MW"], rng.uniform(0.5, 2.0))[:-1]
        else:
            x = np.arange(r.cells[0]) + 0.5 - r.cells[0] * rng.uniform(0.3, 0.7)
            q[..., 4] = (1000.0 + rng.uniform(300.0, 500.0) * np.exp(-0.5 * (x / 8.0) ** 2))[:, None, None]
    return reqs


POOL_DT = 2e-8


def run(state):
    if state["kind"] == "pool":
        reqs = serving.Server(state["pool"], POOL_DT).run(state["requests"], 3)
        return [r.result for r in reqs]
    mb = state["mb"]
    if state["kind"] == "layer":
        mb.set_prims(state["prims"])  # the frozen planes are formed anew from primitives
    else:
        native.call("pgb_state_set", mb.case, 0, native_ptr(state["start"]), state["n"])
    out = 0
    if state["op"] == "rhs":
        mb.rhs()
        out = mb.nregs - 1
    elif state["cfl"]:
        mb.tme = 0.0
        mb.step_cfl(state["cfl"], 1e-2, state["steps"])
    else:
        mb.step(state["dt"], state["steps"])
    native.call("pgb_state_get", mb.case, out, native_ptr(state["result"]), state["n"])
    return state["parts"]


STAGES = {"rk2": 2, "tvd-rk3": 3, "rk4": 4}
# register reads and writes over a step's stages
TRAFFIC = {"rk2": 2 + 3, "tvd-rk3": 2 + 3 + 3, "rk4": 3 + 5 + 5 + 4}


def work(case):
    """The registers' traffic and the floating-point work of the right-hand
    sides, with the state carried in and out once."""
    if case["kind"] == "pool":
        mean = (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        cells = case["requests"] * 0.5 * (1.0 + 4.0 * mean)
        return dict(bytes=8.0 * 13 * cells * (2 + case["steps"] * TRAFFIC["tvd-rk3"]),
                    flops=cells * case["steps"] * 3 * 9000.0)
    integrator = "tvd-rk3" if case["kind"] == "channel" else case["integrator"]
    ns = {"tgv": 1, "layer": 2, "channel": 2}.get(case["kind"]) or case.get("species") or \
        {"h2o2_gri30": 9, "ch4_o2_ffcmy": 12}[case["gas"]]
    cells = float(case["nx"] * case["ny"] * case["nz"])
    per = {"tgv": 650.0 if case.get("simulator") == "navier-stokes" else 200.0, "mix": 900.0, "channel": 800.0,
           "layer": 600.0, "react": 9000.0 if ns == 9 else 13000.0}[case["kind"]]
    if case["op"] == "rhs":
        return dict(bytes=8.0 * (4 + ns) * cells * 2, flops=cells * per)
    return dict(bytes=8.0 * (4 + ns) * cells * (2 + case["steps"] * TRAFFIC[integrator]),
                flops=cells * per * case["steps"] * STAGES[integrator])


# 64-bit arithmetic throughout.  Measured against the sums below, largest of
# an output: a step 3e-13 (the smallest component of a calorically perfect
# run), 3e-10 where temperature comes of a Newton on fits whose terms cancel;
# a right-hand side is a difference of far larger fluxes.
TOLERANCE = {
    "tgv": (3e-12, 1e-11),
    "mix": (3e-12, 1e-11),
    "react": (2e-9, 1e-7),
    "layer": (5e-10, None),
    "channel": (3e-12, None),
    "pool": (2e-9, None),
}


def tolerance(case):
    return {"rel": TOLERANCE[case["kind"]][1 if case.get("op") == "rhs" else 0]}


###############################################################################
# the same answers in plain torch, float64, on one padded global lattice
###############################################################################
def device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def tt(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=device())


class Grid:
    """The global lattice's metrics from its nodes, halo 2; arrays [..., i, j, k]."""

    def __init__(self, n, nodes):
        self.n = n
        X = nodes.permute(3, 0, 1, 2)  # (3, X+1, Y+1, Z+1)

        def corner(hi, axes=(0, 1, 2)):
            s = [slice(None)] * 4
            for a, h in zip(axes, hi):
                s[1 + a] = slice(1, None) if h else slice(None, -1)
            return X[tuple(s)]

        allc = [(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)]
        self.xcc = sum(corner(h) for h in allc) / 8.0
        self.S, self.xf = [], []
        for a in range(3):
            p = ((a + 1) % 3, (a + 2) % 3)
            c00, c01, c10, c11 = (corner(h, p) for h in ((0, 0), (0, 1), (1, 0), (1, 1)))
            self.S.append(0.5 * torch.cross(c10 - c01, c11 - c00, dim=0))
            self.xf.append(0.25 * (c00 + c01 + c10 + c11))
        diag = corner((1, 1, 1)) - corner((0, 0, 0))
        high = self.S[0][:, 1:] + self.S[1][:, :, 1:] + self.S[2][:, :, :, 1:]
        self.vol = (diag * high).sum(0) / 3.0
        e = []
        for a in range(3):
            d = 0.0
            for h in allc:
                if h[a]:
                    lo = list(h)
                    lo[a] = 0
                    d = d + 0.25 * (corner(h) - corner(lo))
            e.append(d)
        rows = [torch.cross(e[1], e[2], dim=0), torch.cross(e[2], e[0], dim=0), torch.cross(e[0], e[1], dim=0)]
        self.J = torch.stack(rows) / self.vol  # (3 axes, 3 directions, ...)

    def inner(self, f):
        return f[..., NG:-NG, NG:-NG, NG:-NG]

    def at(self, f, A, o):
        """f on the cells o along axis A from each face's high-side cell."""
        s = [slice(NG, NG + m) for m in self.n]
        s[A] = slice(NG + o, NG + o + self.n[A] + 1)
        return f[(Ellipsis, *s)]

    def step(self, f, A, o):
        s = [slice(NG, NG + m) for m in self.n]
        s[A] = slice(NG + o, NG + o + self.n[A])
        return f[(Ellipsis, *s)]

    def faces(self, F, A):
        """Low faces less high faces."""
        lo, hi = [slice(None)] * F.dim(), [slice(None)] * F.dim()
        lo[1 + A], hi[1 + A] = slice(None, -1), slice(1, None)
        return F[tuple(lo)] - F[tuple(hi)]


def global_grid(case):
    mesh = mesh_of(case)
    n = (case["nx"], case["ny"], case["nz"])
    nodes = np.zeros(tuple(m + 1 + 2 * NG for m in n) + (3,))
    blocks = mesh.make_blocks(NG)
    at = places(mesh)
    # halos first, every block's own nodes over them
    for inner in (False, True):
        for b, s in zip(blocks, at):
            if inner:
                nodes[tuple(slice(NG + x.start, NG + x.stop + 1) for x in s)] = b.nodes[NG:-NG, NG:-NG, NG:-NG]
            else:
                nodes[tuple(slice(x.start, x.stop + 1 + 2 * NG) for x in s)] = b.nodes
    # the rest of the halo: periodic images
    for a in range(3):
        if mesh.periodic[a]:
            p, L = np.moveaxis(nodes, a, 0), np.eye(3)[a] * mesh.lengths[a]
            m = n[a]
            for h in range(NG):
                p[h] = p[h + m] - L
                p[NG + m + 1 + h] = p[NG + 1 + h] + L
    return mesh, Grid(n, tt(nodes))


class Ideal:
    """The ideal gases: calorically or thermally perfect."""

    def __init__(self, cfg=None, tab=None):
        if tab is not None:
            self.MW = tt(tab["MW"])
            self.ns = len(self.MW)
            self.cppolyR, self.hpoly, self.h298 = tt(tab["cppolyR"]), tt(tab["hpoly"]), tt(tab["h298"])
            self.mupoly, self.kappapoly = tt(tab["mupoly"]), tt(tab["kappapoly"])
            self.lewis = tt(tab["lewis"])
            self.tpg = True
        else:
            sp = list(cfg["mixture"]["species"].values())
            self.MW = tt([s["MW"] for s in sp])
            self.ns = len(sp)
            self.cp0 = tt([s["cp0"] for s in sp])
            self.href = tt([s.get("dHf298", 0.0) / s["MW"] - 298.15 * s["cp0"] for s in sp])
            self.mu0, self.kappa0 = tt([s.get("mu0", 0.0) for s in sp]), tt([s.get("kappa0", 1.0) for s in sp])
            self.lewis = tt([s.get("lewis", 1.0) for s in sp])
            self.tpg = False
        self.R = RU / self.MW

    def mix(self, w, Y):
        return torch.einsum("s,s...->...", w, Y)

    def cp_h(self, T, Y):
        if not self.tpg:
            cp = self.mix(self.cp0, Y)
            return cp, cp * T + self.mix(self.href, Y)
        u, cp, hp = torch.log(T), 0.0, 0.0
        cc = torch.einsum("st,s...->t...", self.cppolyR, Y)
        hc = 0.0
        for m in reversed(range(cc.shape[0])):
            cp = cp * u + cc[m]
            hc = cc[m] - (m + 1) * hc
            hp = hp * u + hc
        return cp, hp * T + self.mix(self.h298 * self.R, Y)

    def h_species(self, T):
        if not self.tpg:
            return torch.stack([c * T + h for c, h in zip(self.cp0, self.href)])
        return torch.stack([horner(p, torch.log(T)) * T * RU / m + h * RU / m
                            for p, h, m in zip(self.hpoly, self.h298, self.MW)])

    def state(self, Q, T=None):
        rho = Q[0]
        vel = Q[1:4] / rho
        Yc = Q[5:] / rho
        Y = torch.cat([Yc, (1.0 - Yc.sum(0))[None]])
        e = Q[4] / rho - 0.5 * (vel ** 2).sum(0)
        R = self.mix(self.R, Y)
        if self.tpg:
            T = torch.full_like(rho, 1200.0) if T is None else T
            for _ in range(12):
                cp, h = self.cp_h(T, Y)
                T = T + (e - (h - R * T)) / (cp - R)
            cp, _ = self.cp_h(T, Y)
        else:
            cp, h0 = self.mix(self.cp0, Y), self.mix(self.href, Y)
            T = (e - h0) / (cp - R)
        return self.finish(dict(rho=rho, vel=vel, Y=Y, e=e, T=T, cp=cp, R=R))

    def finish(self, s):
        s["p"] = s["rho"] * s["R"] * s["T"]
        s["gamma"] = s["cp"] / (s["cp"] - s["R"])
        s["c"] = torch.sqrt(s["gamma"] * s["R"] * s["T"])
        return s

    def from_pT(self, p, T, vel, Y):
        R = self.mix(self.R, Y)
        cp, h = self.cp_h(T, Y)
        return self.finish(dict(rho=p / (R * T), vel=vel, Y=Y, e=h - R * T, T=T, cp=cp, R=R))

    def Q(self, p, vel, T, Yc):
        s = self.from_pT(p, T, vel, torch.cat([Yc, (1.0 - Yc.sum(0))[None]]))
        rho = s["rho"]
        return torch.cat([rho[None], rho * vel, (rho * (s["e"] + 0.5 * (vel ** 2).sum(0)))[None], rho * Yc])

    def transport(self, s, T=None):
        """mu, kappa and rho D over rho per species; h per species."""
        Y, T = s["Y"].clone(), s["T"] if T is None else T
        Y[-1] = Y[-1].clamp(min=0.0)
        mole = Y / self.MW[(slice(None),) + (None,) * T.dim()]
        X = mole / mole.sum(0)
        if self.tpg:
            u, sT = torch.log(T), torch.sqrt(T)
            mu = torch.stack([(horner(p, u) * torch.sqrt(sT)) ** 2 for p in self.mupoly])
            kap = torch.stack([horner(p, u) * sT for p in self.kappapoly])
        else:
            mu = torch.stack([m + 0.0 * T for m in self.mu0])
            kap = torch.stack([k + 0.0 * T for k in self.kappa0])
        total = 0.0
        for a in range(self.ns):
            phi = 0.0
            for b in range(self.ns):
                r = 1.0 + torch.sqrt(mu[a] / mu[b]) * (self.MW[b] / self.MW[a]) ** 0.25
                phi = phi + r ** 2 / torch.sqrt(8.0 * (1.0 + self.MW[a] / self.MW[b])) * X[b]
            total = total + mu[a] * X[a] / phi
        kappa = 0.5 * ((X * kap).sum(0) + 1.0 / (X / kap).sum(0))
        D = torch.stack([kappa / (s["rho"] * s["cp"] * le) for le in self.lewis])
        return total, kappa, D


def horner(poly, u):
    out = 0.0
    for c in reversed(range(len(poly))):
        out = out * u + poly[c]
    return out


class Chemistry:
    def __init__(self, tab, gas):
        self.t, self.gas = tab, gas
        self.gpoly = tt(tab["gpoly"])

    def rates(self, rho, Yc, T):
        """Net production rates of the carried species, kg / m^3 / s."""
        t, ns = self.t, self.gas.ns
        Yc = (Yc / rho).clamp(0.0, 1.0)
        last = (1.0 - Yc.sum(0)).clamp(min=0.0)
        Y = torch.cat([Yc / Yc.sum(0).clamp(min=1.0), last[None]])
        c = [rho * Y[s] / self.gas.MW[s] for s in range(ns)]
        ctot = sum(c)
        u, Ti = torch.log(T), 1.0 / T
        g = [horner(self.gpoly[s], u) + self.gas.h298[s] * Ti for s in range(ns)]
        floor = float(t["logcfloor"])
        logc = [torch.log(x.clamp(min=1e-300)).clamp(min=floor) for x in c]
        cG = [x.clamp(min=0.0) * torch.exp(y) for x, y in zip(c, g)]
        lpRuT = float(t["logprefRu"]) - u
        tb = []
        for j in range(len(t["tbdefeff"])):
            m = float(t["tbdefeff"][j]) * ctot
            for i in range(int(t["tb_neff"][j])):
                m = m + float(t["tbeffdev"][j][i]) * c[int(t["tb_effsp"][j][i])]
            tb.append(m)
        omega = [torch.zeros_like(rho) for _ in range(ns)]

        def side(k, sp, nu):
            return [(int(a), float(b)) for a, b in zip(t[sp][k], t[nu][k]) if b != 0.0]

        for k in range(int(t["rxn_nr"])):
            kind = int(t["rxn_kind"][k])
            lk = float(t["rxn_logA"][k]) + float(t["rxn_b"][k]) * u - float(t["rxn_EaR"][k]) * Ti
            lk = lk + torch.zeros_like(rho)
            M = tb[int(t["rxn_tb"][k])] if kind else None
            if kind >= 2:
                lpr = torch.log(M.clamp(min=1e-300)) + float(t["rxn_logprA"][k]) + float(t["rxn_prb"][k]) * u \
                    - float(t["rxn_prEaR"][k]) * Ti
                pr = torch.exp(lpr)
                factor = pr / (1.0 + pr)
            if kind == 3:
                poly = t["rxnlfcpoly"][int(t["rxn_troeidx"][k])]
                tf = (u - float(t["troeuc"])) * float(t["troeuhinv"])
                lfc = horner([float(x) for x in poly], tf)
                C, N = -0.4 - 0.67 * lfc, 0.75 - 1.27 * lfc
                a = lpr / math.log(10.0) + C
                b = N - 0.14 * a
                lk = lk + lfc / (1.0 + (a / b) ** 2) * math.log(10.0)
            nusum = float(t["rxn_nusum"][k])
            if int(t["rxn_product"][k]):
                react, prod = side(k, "rxn_reactsp", "rxn_reactnu"), side(k, "rxn_prodsp", "rxn_prodnu")
                K = torch.exp(lk - sum(nu * g[s] for s, nu in react))
                K = K * M if kind == 1 else K * factor if kind >= 2 else K
                fwd, rev = K, K * torch.exp(-nusum * lpRuT)
                for s, nu in react:
                    fwd = fwd * cG[s] ** nu
                for s, nu in prod:
                    rev = rev * cG[s] ** nu
            else:
                lk = lk + torch.log(M.clamp(min=1e-300)) if kind == 1 else lk + torch.log(factor) if kind >= 2 else lk
                net = [(int(a), float(b)) for a, b in zip(t["rxn_netsp"][k], t["rxn_netnu"][k]) if b != 0.0]
                lrp = lk + sum(o * logc[s] for s, o in side(k, "rxn_fwdsp", "rxn_fwdorder"))
                fwd = torch.exp(lrp)
                rev = torch.exp(lrp - nusum * lpRuT + sum(nu * (g[s] + logc[s]) for s, nu in net))
            rp = fwd - rev if int(t["rxn_reversible"][k]) else fwd
            for s, nu, w in zip(t["rxn_netsp"][k], t["rxn_netnu"][k], t["rxn_netnuMW"][k]):
                if nu != 0.0:
                    omega[int(s)] = omega[int(s)] + float(w) * rp
        return torch.stack(omega[:-1])


def koren(l, c, r):
    """Half the koren-limited slope at c."""
    a, b = c - l, r - c
    s = torch.where(b < 0.0, -1.0, 1.0)
    a, m = s * a, b.abs()
    lim = torch.minimum(torch.minimum(2.0 * a, (2.0 * m + a) / 3.0), 2.0 * m).clamp(min=0.0)
    return torch.where(b == 0.0, torch.zeros_like(b), 0.5 * s * lim)


class Flow:
    """The right-hand side of the ideal gases on the lattice."""

    def __init__(self, grid, gas, primary, recon, viscous, chemistry=None, wrap=(True, True, True), bcs=None,
                 index=None, damping=1.0):
        self.g, self.gas, self.primary, self.recon, self.viscous = grid, gas, primary, recon, viscous
        self.chem, self.wrap, self.bcs, self.index, self.damping = chemistry, wrap, bcs, index, damping

    def pad(self, f):
        """Interior values to the full lattice; periodic axes wrapped, the others repeated."""
        for a in range(3):
            d = f.dim() - 3 + a
            n = f.shape[d]
            if self.index is not None and a == 0:
                f = f.index_select(d, self.index)
                continue
            idx = torch.arange(-NG, n + NG, device=f.device)
            f = f.index_select(d, idx % n if self.wrap[a] else idx.clamp(0, n - 1))
        return f

    def rhs(self, Qi, t=0.0):
        g, gas = self.g, self.gas
        Q = self.pad(Qi)
        T0 = getattr(self, "T", None)
        s = gas.state(Q, T0)
        if gas.tpg:
            self.T = s["T"]
        if self.bcs is not None:
            Q = self.bcs.halo(Q, s, t)
            s = gas.state(Q)
        if self.viscous:
            mu, kappa, D = gas.transport(s)
            hs = gas.h_species(s["T"])
            rows = torch.cat([s["vel"], s["T"][None], s["Y"][:-1]])
            d = [0.5 * (g.step(rows, a, 1) - g.step(rows, a, -1)) for a in range(3)]
            J = g.inner(g.J)
            grads = torch.stack([sum(d[a] * J[a, e] for a in range(3)) for e in range(3)], 1)
            G = self.pad(grads)
        dQ = torch.zeros_like(Qi)
        if self.chem is not None:
            dQ[5:] = self.chem.rates(Qi[0], Qi[5:], g.inner(s["T"]))
        for A in range(3):
            S = g.at(g.S[A], A, 0)
            F = self.advective(s, S, A)
            if self.viscous:
                xf, xL, xR = g.at(g.xf[A], A, 0), g.at(g.xcc, A, -1), g.at(g.xcc, A, 0)
                F = F + self.diffusive(s, rows, G, mu, kappa, D, hs, S, xf, xL, xR, A)
            if self.bcs is not None:
                self.bcs.walls(F, s, A, S, t)
            dQ = dQ + g.faces(F, A) / g.inner(g.vol)
        return dQ

    def sides(self, s, A):
        at = self.g.at
        out = []
        if self.recon == "constant":
            for o in (-1, 0):
                out.append({k: at(s[k], A, o) for k in ("p", "rho", "e", "c", "vel", "Y", "T", "cp", "gamma")})
            return out
        for o, sign in ((-1, 1.0), (0, -1.0)):
            def face(f):
                l, c, r = (at(f, A, o - 1), at(f, A, o), at(f, A, o + 1)) if sign > 0 else \
                    (at(f, A, o + 1), at(f, A, o), at(f, A, o - 1))
                # the slope limited against the difference across the face
                return c + koren(l, c, r)

            Yc = face(s["Y"][:-1])
            Y = torch.cat([Yc, (1.0 - Yc.sum(0))[None]])
            out.append(self.gas.from_pT(face(s["p"]), face(s["T"]), face(s["vel"]), Y))
        return out

    def advective(self, s, S, A):
        L, R = self.sides(s, A)
        dot = lambda v: (v * S).sum(0)  # noqa: E731
        if self.primary == "kepaec":
            vf = 0.5 * (L["vel"] + R["vel"])
            C = 0.5 * (L["rho"] + R["rho"]) * dot(vf)
            th = [x["cp"] / x["gamma"] * x["T"] for x in (L, R)]
            pf = 0.5 * (L["p"] + R["p"])
            K = 0.5 * C * (L["vel"] * R["vel"]).sum(0)
            P = 0.5 * (L["p"] * dot(R["vel"]) + R["p"] * dot(L["vel"]))
            ef = 2.0 * th[0] * th[1] / (th[0] + th[1]) + 0.5 * (L["e"] - th[0] + R["e"] - th[1])
            Yf = 0.5 * (L["Y"] + R["Y"])[:-1]
            return torch.cat([C[None], C * vf + pf * S, (ef * C + K + P)[None], C * Yf])
        area = torch.sqrt(dot(S))
        nrm = S / area
        un = [(x["vel"] * nrm).sum(0) for x in (L, R)]
        full = []
        for x, u in zip((L, R), un):
            E = x["rho"] * (x["e"] + 0.5 * (x["vel"] ** 2).sum(0))
            U = torch.cat([x["rho"][None], x["rho"] * x["vel"], E[None], x["rho"] * x["Y"][:-1]])
            F = U * u
            F[1:4] += x["p"] * nrm
            F[4] += x["p"] * u
            full.append((U, F, E))
        if self.primary == "rusanov":
            lam = torch.maximum(un[0].abs() + L["c"], un[1].abs() + R["c"])
            return 0.5 * area * (full[0][1] + full[1][1] - lam * (full[1][0] - full[0][0]))
        SL, SR = un[0] - L["c"], un[1] + R["c"]
        mL, mR = L["rho"] * (SL - un[0]), R["rho"] * (SR - un[1])
        Ss = (R["p"] - L["p"] + mL * un[0] - mR * un[1]) / (mL - mR)
        star = []
        for x, u, sx, (U, F, E) in zip((L, R), un, (SL, SR), full):
            k = x["rho"] * (sx - u) / (sx - Ss)
            V = torch.cat([k[None], k * (x["vel"] + (Ss - u) * nrm),
                           (k * (E / x["rho"] + (Ss - u) * (Ss + x["p"] / (x["rho"] * (sx - u)))))[None],
                           k * x["Y"][:-1]])
            star.append(F + sx * (V - U))
        F = torch.where(SL >= 0.0, full[0][1], torch.where(Ss >= 0.0, star[0], torch.where(SR >= 0.0, star[1],
                                                                                         full[1][1])))
        return F * area

    def diffusive(self, s, rows, G, mu, kappa, D, hs, S, xf, xL, xR, A):
        at = self.g.at
        nrm = S / torch.sqrt((S * S).sum(0))
        damp = self.damping / torch.sqrt((((xR - xL) * nrm) ** 2).sum(0)) * nrm
        gL, gR = at(G, A, -1), at(G, A, 0)
        wl = at(rows, A, -1) + (gL * (xf - xL)).sum(1)
        wr = at(rows, A, 0) + (gR * (xf - xR)).sum(1)
        grad = 0.5 * (gL + gR) + damp * (wr - wl)[:, None]
        mean = lambda f: 0.5 * (at(f, A, -1) + at(f, A, 0))  # noqa: E731
        m, k = mean(mu), mean(kappa)
        du = grad[0:3]  # [component, direction]
        div = du[0, 0] + du[1, 1] + du[2, 2]
        tau = -m * (du + du.transpose(0, 1))
        for d in range(3):
            tau[d, d] = tau[d, d] + 2.0 / 3.0 * m * div
        force = (tau * S).sum(1)
        energy = -k * (grad[3] * S).sum(0) + (mean(s["vel"]) * force).sum(0)
        rho = mean(s["rho"])
        gY = (grad[4:] * S).sum(1)
        gY = torch.cat([gY, -gY.sum(0, keepdim=True)])
        Df, h, Y = mean(D), mean(hs), mean(s["Y"])
        flux = -rho * Df * gY + Y * (rho * (Df * gY).sum(0))
        energy = energy + (flux * h).sum(0)
        return torch.cat([torch.zeros_like(energy)[None], force, energy[None], flux[:-1]])

    def combined(self, Qi):
        """The largest combined CFL number per unit step."""
        s, g = self.gas.state(Qi), self.g
        inv, conv = 0.0, 0.0
        for A in range(3):
            S, xf = g.at(g.S[A], A, 0), g.at(g.xf[A], A, 0)
            n = S / torch.sqrt((S * S).sum(0))
            lo, hi = [slice(None)] * 4, [slice(None)] * 4
            lo[1 + A], hi[1 + A] = slice(None, -1), slice(1, None)
            lo, hi = tuple(lo), tuple(hi)
            d = torch.sqrt(((xf[hi] - xf[lo]) ** 2).sum(0))
            inv = inv + 1.0 / d ** 2
            conv = conv + (0.5 * (n[lo] + n[hi]) * s["vel"]).sum(0).abs() / d
        return float((s["c"] * torch.sqrt(inv) + conv).max())


class Channel:
    """The channel's boundary cells and wall faces."""

    def __init__(self, cfg, grid, gas):
        self.cfg, self.g, self.gas = cfg, grid, gas
        self.h = library.CHANNEL_LENGTHS[1]

    def inflow(self, t):
        g = self.g
        x = g.xf[0][:, NG, NG:-NG, NG:-NG]
        y, z = x[1], x[2]
        u = 60.0 * (y / self.h) * (1.0 - y / self.h) * 4.0 + 5.0 * math.sin(2000.0 * t)
        return torch.stack([u, torch.zeros_like(u), 2.0 * torch.sin(300.0 * z)]), \
            300.0 + 20.0 * torch.cos(300.0 * z), torch.full_like(u, 0.6)[None]

    def halo(self, Q, s, t):
        Q = Q.clone()
        nx, ny, _ = self.g.n
        J, K = slice(NG, -NG), slice(NG, -NG)
        for layer in range(NG):
            # the inflow: its values, the pressure extrapolated
            i0 = NG
            vel, T, Y = self.inflow(t)
            p = 2.0 * s["p"][i0, J, K] - s["p"][i0 + min(layer + 1, nx - 1), J, K]
            Q[:, NG - 1 - layer, J, K] = self.gas.Q(p, vel, T, Y)
            # the exit: its pressure, the velocity extrapolated where it leaves
            i0 = NG + nx - 1
            im, im1 = i0 - min(layer, nx - 1), i0 - min(layer + 1, nx - 1)
            v0, vm, vm1 = (s["vel"][:, i, J, K] for i in (i0, im, im1))
            back = vm.clone()
            back[0] = -back[0]
            vel = torch.where(v0[0] > 0.0, 2.0 * v0 - vm1, back)
            Q[:, NG + nx + layer, J, K] = self.gas.Q(torch.full_like(v0[0], library.P0), vel, s["T"][i0, J, K],
                                                     s["Y"][:-1, i0, J, K])
            # the floor: held at rest and at 320 K
            I = slice(NG, -NG)
            j = NG + min(layer, ny - 1)
            Q[:, I, NG - 1 - layer, K] = self.gas.Q(s["p"][I, j, K], -s["vel"][:, I, j, K],
                                                    torch.full_like(s["p"][I, j, K], 320.0), s["Y"][:-1, I, j, K])
            # the lid: moving, adiabatic
            j = NG + ny - 1 - min(layer, ny - 1)
            rho, vel = s["rho"][I, j, K], s["vel"][:, I, j, K]
            vh = tt([20.0, 0.0, 0.0])[:, None, None] * 2.0 - vel
            q = Q[:, I, j, K].clone()
            q[1:4] = rho * vh
            q[4] = q[4] + 0.5 * rho * ((vh ** 2).sum(0) - (vel ** 2).sum(0))
            Q[:, I, NG + ny + layer, K] = q
        # the periodic images of the cells just set
        n = self.g.n[2]
        Q[..., :NG], Q[..., NG + n:] = Q[..., n:n + NG].clone(), Q[..., NG:2 * NG].clone()
        return Q

    def walls(self, F, s, A, S, t):
        if A != 1:
            return
        g, ny = self.g, self.g.n[1]
        I, K = slice(NG, -NG), slice(NG, -NG)
        for low in (True, False):
            j, f, out = (NG, 0, -1.0) if low else (NG + ny - 1, ny, 1.0)
            Sf = S[:, :, f]
            area = torch.sqrt((Sf * Sf).sum(0))
            n = Sf / area
            vel, p, rho, c = s["vel"][:, I, j, K], s["p"][I, j, K], s["rho"][I, j, K], s["c"][I, j, K]
            pw = (p + rho * c * out * (vel * n).sum(0)).clamp(min=0.0)
            cell = {k: (v[:, I, j, K] if v.dim() == 4 else v[I, j, K]) for k, v in s.items()}
            if low:
                wall, Tw = torch.zeros(3, dtype=torch.float64, device=F.device), 320.0
                at = self.gas.from_pT(p, torch.full_like(p, Tw), vel, cell["Y"])
                mu, kappa, _ = self.gas.transport(at)
                dT = Tw - cell["T"]
            else:
                wall = tt([20.0, 0.0, 0.0])
                mu, kappa, _ = self.gas.transport(cell)
                dT = torch.zeros_like(p)
            xf, xc = g.xf[1][:, I, NG + f, K], g.xcc[:, I, j, K]
            dn = ((xc - xf) * n).sum(0).abs()
            dun = out * (wall[:, None, None] - vel) / dn
            div = (dun * n).sum(0)
            tS = -mu * area * (dun + div * n / 3.0)
            F[:, :, f] = 0.0
            F[1:4, :, f] = pw * Sf + tS
            F[4, :, f] = (wall[:, None, None] * tS).sum(0) - kappa * out * dT / dn * area


class Cubic:
    """The Peng-Robinson gas with the double flux (inviscid, kepaec)."""

    def __init__(self, grid, tab):
        self.g = grid
        self.ideal = Ideal(tab=tab)
        self.MW = self.ideal.MW
        f = lambda k: float(tab[k])  # noqa: E731
        self.u, self.w, self.sg, self.ep = f("cubicu"), f("cubicw"), f("cubicsigma"), f("cubiceps")
        for k in ("cubicsqrtac", "cubicb", "cubicda", "cubicmTc", "cubiconepm", "vshift"):
            setattr(self, k, tt(tab[k]))

    def mixture(self, Y):
        moles = Y / self.MW[:, None, None, None]
        MW = 1.0 / moles.sum(0)
        return moles * MW, MW

    def attraction(self, X, T):
        sT = torch.sqrt(T)
        root = [self.cubicsqrtac[n] * (self.cubiconepm[n] - sT * self.cubicmTc[n]).abs() for n in range(2)]
        S1 = sum(X[n] * root[n] for n in range(2))
        S2 = sum(X[n] * self.cubicda[n] for n in range(2))
        return root, S1, S2, S1 ** 2, -S1 * S2 / sT

    def density(self, p, T, Y):
        """The cubic's root of least Gibbs energy."""
        X, MW = self.mixture(Y)
        b, c = (sum(X[n] * k[n] for n in range(2)) for k in (self.cubicb, self.vshift))
        _, _, _, a, _ = self.attraction(X, T)
        A, B = a * p / (RU * T) ** 2, b * p / (RU * T)
        z2 = -(1.0 + B - self.u * B)
        z1 = A + self.w * B ** 2 - self.u * B - self.u * B ** 2
        z0 = -(A * B + self.w * B ** 2 * (1.0 + B))
        Qc = (z2 ** 2 - 3.0 * z1) / 9.0
        Rc = (2.0 * z2 ** 3 - 9.0 * z2 * z1 + 27.0 * z0) / 54.0
        M = Rc ** 2 - Qc ** 3
        S = -torch.sign(Rc) * (Rc.abs() + torch.sqrt(M.clamp(min=0.0))) ** (1.0 / 3.0)
        one = S + Qc / S - z2 / 3.0
        sq = torch.sqrt(Qc.clamp(min=1e-300))
        th = torch.acos((Rc / (Qc * sq)).clamp(-1.0, 1.0)) / 3.0
        best, gb = None, None
        for k in (0.0, 2.0 * math.pi / 3.0, -2.0 * math.pi / 3.0):
            Z = -2.0 * sq * torch.cos(th + k) - z2 / 3.0
            gibbs = Z - 1.0 - torch.log((Z - B).clamp(min=1e-300)) + A / (B * (self.sg - self.ep)) * \
                torch.log(((Z + self.ep * B) / (Z + self.sg * B)).clamp(min=1e-300))
            gibbs = torch.where(Z > B, gibbs, torch.full_like(gibbs, 1e300))
            best, gb = (Z, gibbs) if best is None else (torch.where(gibbs < gb, Z, best), torch.minimum(gibbs, gb))
        Z = torch.where(M > 0.0, one, best)
        return p * MW / (RU * T * (Z - c * p / (RU * T)))

    def point(self, rho, Y, T):
        """The gas at a volume and temperature."""
        o = {}
        X, MW = self.mixture(Y)
        b, cm = (sum(X[n] * k[n] for n in range(2)) for k in (self.cubicb, self.vshift))
        root, S1, S2, a, da = self.attraction(X, T)
        v = MW / rho + cm
        D = (v + self.sg * b) * (v + self.ep * b)
        I = torch.log((v + self.sg * b) / (v + self.ep * b)) / ((self.sg - self.ep) * b)
        cpi, hi = self.ideal.cp_h(T, Y)
        R = RU / MW
        p = RU * T / (v - b) - a / D
        dpdT = RU / (v - b) - da / D
        dpdv = -RU * T / (v - b) ** 2 + a * (2.0 * v + (self.sg + self.ep) * b) / D ** 2
        d2a = 0.5 * (S2 ** 2 - da) / T
        e = hi - R * T - (a - T * da) * I / MW
        cv = cpi - R + T * d2a * I / MW
        o.update(p=p, e=e, cv=cv, dpdT=dpdT, dpdrho=-dpdv * MW / rho ** 2, MW=MW, X=X, v=v, b=b, cm=cm, a=a, da=da,
                 S1=S1, S2=S2, root=root, D=D, I=I, T=T, rho=rho, Y=Y, d2a=d2a, dpdv=dpdv)
        return o

    def T_of_e(self, rho, Y, e, T):
        for _ in range(12):
            o = self.point(rho, Y, T)
            T = T - (o["e"] - e) / o["cv"]
        return T

    def T_of_p(self, rho, Y, p, T):
        for _ in range(12):
            o = self.point(rho, Y, T)
            T = T - (o["p"] - p) / o["dpdT"]
        return T

    def plane(self, o):
        """The tangent plane of rho e in p, rho and rho Y."""
        rho, T, Y = o["rho"], o["T"], o["Y"]
        theta = rho * o["cv"] / o["dpdT"]
        # d(rho e) at fixed T and Y, then moved to fixed p
        epsY = o["e"] - (T * o["dpdT"] - o["p"]) / rho - theta * o["dpdrho"]
        # partial enthalpies and the density's derivative in Y_0 at fixed p, T:
        # by the chain rule on molar volume, covolume and attraction per mole
        h = self.partial_h(o)
        dpdrho_T = o["dpdrho"]
        rho_T = -o["dpdT"] / dpdrho_T
        dMW = -o["MW"] ** 2 * (1.0 / self.MW[0] - 1.0 / self.MW[1])
        dX = [dMW / self.MW[n] * Y[n] + o["MW"] / self.MW[n] * (1.0 if n == 0 else -1.0) for n in range(2)]
        db, dc = (sum(dX[n] * k[n] for n in range(2)) for k in (self.cubicb, self.vshift))
        dS1 = sum(dX[n] * o["root"][n] for n in range(2))
        dam = 2.0 * o["S1"] * dS1
        dv = dMW / rho + dc
        v, b = o["v"], o["b"]
        vs, ve = v + self.sg * b, v + self.ep * b
        dD = (dv + self.sg * db) * ve + vs * (dv + self.ep * db)
        dpdY = -RU * T * (dv - db) / (v - b) ** 2 - dam / o["D"] + o["a"] * dD / o["D"] ** 2
        rho_Y = -dpdY / dpdrho_T
        cp = o["cv"] + T * o["dpdT"] ** 2 / (rho ** 2 * dpdrho_T)
        zeta = h[0] - h[1] - cp / rho_T * rho_Y
        eps = epsY - zeta * Y[0]
        kappa = rho * o["e"] - epsY * rho - theta * o["p"]
        return dict(theta=theta, eps=eps, kappa=kappa, zeta=zeta)

    def partial_h(self, o):
        """Partial enthalpies per mass: d(n h)/dn_k at fixed p, T, from the
        residual A = (a - T a') n I, differentiated at fixed volume and moved
        to fixed pressure."""
        T, v, b, X = o["T"], o["v"], o["b"], o["X"]
        hs = self.ideal.h_species(T)
        MW, vol = o["MW"], o["v"]
        w = o["a"] - T * o["da"]
        sT = torch.sqrt(T)
        vs, ve = v + self.sg * b, v + self.ep * b
        H = None
        out = []
        for k in range(2):
            # per mole of mixture at total moles 1: d/dn_k with the molar
            # translated volume V = n v fixed
            dS1 = o["root"][k] - o["S1"]
            dS2 = self.cubicda[k] - o["S2"]
            da = 2.0 * o["S1"] * dS1
            dda = -(dS1 * o["S2"] + o["S1"] * dS2) / sT
            db = self.cubicb[k] - b
            dv = self.vshift[k] - o["cm"] - (v - o["cm"])
            # molar residual internal energy u = -w I(v, b)
            dI_v = -1.0 / (vs * ve)
            dI_b = (self.sg / vs - self.ep / ve) / ((self.sg - self.ep) * b) - o["I"] / b
            du = -(da - T * dda) * o["I"] - w * (dI_v * dv + dI_b * db)
            u_k = -w * o["I"] + du
            # p's derivative at fixed volume
            dD = (dv + self.sg * db) * ve + vs * (dv + self.ep * db)
            p_k = -RU * T * (dv - db) / (v - b) ** 2 - da / o["D"] + o["a"] * dD / o["D"] ** 2
            # the partial molar volume and the internal pressure
            v_k = -p_k / o["dpdv"]
            pi = T * o["dpdT"] - o["p"]
            ideal = hs[k] * self.MW[k] - RU * T
            out.append((ideal + u_k + pi * v_k + o["p"] * v_k) / self.MW[k])
        return out

    def run(self, q, dt, steps):
        """q interior primitives (ne, ...): Q after the steps of TVD-RK3."""
        Yc = q[5:]
        Y = torch.cat([Yc, 1.0 - Yc])
        rho = self.density(q[0], q[4], Y)
        o = self.point(rho, Y, q[4])
        Q = torch.cat([rho[None], rho * q[1:4], (rho * (o["e"] + 0.5 * (q[1:4] ** 2).sum(0)))[None], rho * Yc])
        T = q[4]
        plane = None

        def split(Q):
            return Q[0], Q[1:4] / Q[0], torch.cat([Q[5:] / Q[0], 1.0 - Q[5:] / Q[0]])

        def freeze(Q, T, plane):
            rho, vel, Y = split(Q)
            if plane is None:
                T = self.T_of_e(rho, Y, Q[4] / rho - 0.5 * (vel ** 2).sum(0), T)
            else:
                T = self.T_of_p(rho, Y, self.p_of(Q, plane), T)
            o = self.point(rho, Y, T)
            Q = Q.clone()
            Q[4] = rho * (o["e"] + 0.5 * (vel ** 2).sum(0))
            return Q, T, self.plane(o)

        Q, T, plane = freeze(Q, T, None)
        for _ in range(steps):
            Q, T, plane = freeze(Q, T, plane)
            P = {k: self.pad(v) for k, v in plane.items()}
            Q1 = Q + dt * self.rhs(Q, P)
            Q1 = 0.25 * Q1 + 0.75 * Q + 0.25 * dt * self.rhs(Q1, P)
            Q = 2.0 / 3.0 * Q1 + 1.0 / 3.0 * Q + 2.0 / 3.0 * dt * self.rhs(Q1, P)
        return Q

    def p_of(self, Q, P):
        return (Q[4] - 0.5 * (Q[1:4] ** 2).sum(0) / Q[0] - P["eps"] * Q[0] - P["zeta"] * Q[5] - P["kappa"]) / P["theta"]

    def pad(self, f):
        for a in range(3):
            d = f.dim() - 3 + a
            n = f.shape[d]
            f = f.index_select(d, torch.arange(-NG, n + NG, device=f.device) % n)
        return f

    def rhs(self, Qi, P):
        g = self.g
        Q = self.pad(Qi)
        vel, rho, Y, p = Q[1:4] / Q[0], Q[0], Q[5] / Q[0], self.p_of(Q, P)
        dQ = 0.0
        for A in range(3):
            at = lambda f, o: g.at(f, A, o)  # noqa: E731
            S = g.at(g.S[A], A, 0)
            vL, vR, pL, pR, rL, rR, YL, YR = (at(f, o) for f in (vel, p, rho, Y) for o in (-1, 0))
            vf = 0.5 * (vL + vR)
            C = 0.5 * (rL + rR) * (S * vf).sum(0)
            K = 0.5 * C * (vL * vR).sum(0)
            Pj = 0.5 * (pL * (vR * S).sum(0) + pR * (vL * S).sum(0))
            E = []
            for o in (-1, 0):
                th, ep, ka, ze = (at(P[k], o) for k in ("theta", "eps", "kappa", "zeta"))
                tL, tR = (th * pL + ka) / rL, (th * pR + ka) / rR
                E.append((ep + 0.5 * ze * (YL + YR) + 2.0 * tL * tR / (tL + tR)) * C + K + Pj)
            F = torch.cat([C[None], C * vf + 0.5 * (pL + pR) * S, E[0][None], (0.5 * (YL + YR) * C)[None]])
            d = g.faces(F, A)
            # the energy: the right cell's plane on a cell's low faces, the left's on its high ones
            lo, hi = [slice(None)] * 3, [slice(None)] * 3
            lo[A], hi[A] = slice(None, -1), slice(1, None)
            d[4] = E[1][tuple(lo)] - E[0][tuple(hi)]
            dQ = dQ + d / g.inner(g.vol)
        return dQ


def advance(flow, Q, integrator, dt, steps, cfl=None, dtmax=None):
    t = 0.0
    for _ in range(steps):
        h = min(cfl / flow.combined(Q), dtmax) if cfl else dt
        if integrator == "rk4":
            k1 = flow.rhs(Q, t)
            k2 = flow.rhs(Q + 0.5 * h * k1, t + 0.5 * h)
            k3 = flow.rhs(Q + 0.5 * h * k2, t + 0.5 * h)
            k4 = flow.rhs(Q + h * k3, t + h)
            Q = Q + h / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        elif integrator == "rk2":
            Q1 = Q + h * flow.rhs(Q, t)
            Q = 0.5 * Q1 + 0.5 * Q + 0.5 * h * flow.rhs(Q1, t + h)
        else:
            Q1 = Q + h * flow.rhs(Q, t)
            Q1 = 0.25 * Q1 + 0.75 * Q + 0.25 * h * flow.rhs(Q1, t + h)
            Q = 2.0 / 3.0 * Q1 + 1.0 / 3.0 * Q + 2.0 / 3.0 * h * flow.rhs(Q1, t + 0.5 * h)
        t += h
    return Q


def exact(case, seed):
    torch.backends.cuda.matmul.allow_tf32 = False
    if case["kind"] == "pool":
        return exact_pool(case, seed)
    mesh, grid = global_grid(case)
    cfg = config_of(case)
    q = tt(fields(case, seed)).permute(3, 0, 1, 2).contiguous()
    if case["kind"] == "layer":
        out = Cubic(grid, table(case)).run(q, step_size(case), case["steps"])
    else:
        tab = table(case) if case["kind"] == "react" else None
        gas = Ideal(cfg, tab)
        viscous = cfg["simulation"]["simulator"] == "navier-stokes"
        chem = Chemistry(tab, gas) if tab is not None else None
        bcs = Channel(cfg, grid, gas) if case["kind"] == "channel" else None
        adv = cfg["adv-flux"]
        flow = Flow(grid, gas, adv["primary"], adv["recon"], viscous, chem, tuple(mesh.periodic), bcs,
                    damping=float(cfg["diff-flux"]["values"].get("alpha", 1.0)))
        Q = gas.Q(q[0], q[1:4], q[4], q[5:])
        if case["op"] == "rhs":
            out = flow.rhs(Q)
        else:
            out = advance(flow, Q, cfg["time-integration"]["integrator"], step_size(case), case["steps"],
                          cfl_of(case), 1e-2)
    parts, at = [], places(mesh)
    split = len(at) * out.shape[0] <= 60
    for s in at:
        # components outermost, i fastest, as the library's state arrays
        rows = out[(slice(None), *s)].permute(0, 3, 2, 1).reshape(out.shape[0], -1)
        parts += list(rows) if split else [rows]
    return parts


def exact_pool(case, seed):
    tab = table(case)
    gas = Ideal(tab=tab)
    chem = Chemistry(tab, gas)
    reqs = pool_requests(case, seed)
    out = [None] * len(reqs)
    steps = case["steps"]
    zero = [r for r in reqs if r.kind == "0d"]
    if zero:
        # the reactors: every one a cell
        q = tt(np.stack([r.prims[0, 0, 0] for r in zero], -1))[..., None, None]
        Q = gas.Q(q[0], q[1:4], q[4], q[5:])

        class Box:
            @staticmethod
            def rhs(Q, t):
                d = torch.zeros_like(Q)
                d[5:] = chem.rates(Q[0], Q[5:], gas.state(Q)["T"])
                return d

        Q = advance(Box, Q, "tvd-rk3", POOL_DT, steps)
        for k, r in enumerate(zero):
            out[r.rid] = Q[:, k, 0, 0].expand(2, 2, 2, -1)
    one = [r for r in reqs if r.kind == "1d"]
    if one:
        # the 1-D domains end to end along i, each with its own periodic halo
        # between it and the next
        dx = one[0].lengths[0] / one[0].cells[0]
        length = sum(r.cells[0] + 2 * NG for r in one)
        src, at, spans = [], 0, []
        for r in one:
            m = r.cells[0]
            src += [at + NG + (x % m) for x in range(-NG, m + NG)]
            spans.append(slice(at, at + m))
            at += m + 2 * NG
        n = length - 2 * NG
        index = torch.as_tensor(src, device=device()) - NG  # into the lattice's interior
        ax = [np.arange(-NG, m + 1 + NG) * dx for m in (n, 2, 2)]
        grid = Grid((n, 2, 2), tt(np.stack(np.meshgrid(*ax, indexing="ij"), -1)))
        q = np.zeros((n, 2, 2, gas.ns + 4))
        q[...] = one[0].prims[0, 0, 0]
        for r, s in zip(one, spans):
            q[s] = r.prims
        q = tt(q).permute(3, 0, 1, 2).contiguous()
        flow = Flow(grid, gas, "hllc", "muscl", True, chem, index=index)
        Q = advance(flow, gas.Q(q[0], q[1:4], q[4], q[5:]), "tvd-rk3", POOL_DT, steps)
        for r, s in zip(one, spans):
            out[r.rid] = Q[:, s].permute(1, 2, 3, 0)
    return out
