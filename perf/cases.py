"""The calls this library is used for, as cases that a benchmark can draw, prepare, run and check.

A case is a dict of plain values; `prepare` makes its inputs and handles, `run` is one pass through the public
Python entry points (m2c_b200.gpu), `work` its unavoidable bytes and operations, and `exact` the same outputs from
plain torch / numpy in 64 bits where the computation has such a value (single-material runs, Riemann star states,
the warm-start network's gradient; the two-material runs have none that is quick to compute).

Kinds:
  residual  one residual of a small subdomain, read back to the host (SpaceOperator::ComputeResidual's replacement)
  run       upload, a number of steps (or to a final time), download: one output interval of a single-material run
  bubbles   the same with air bubbles in water, a level set and the exact interface Riemann problems
  step      one step of the drop-in integrator: upload, advance by dt, download, on ordinary host arrays
  plane     a box cut by a resting plane: one-sided Riemann problems on every cut face
  tubes     a batch of uneven two-material shock tubes: create, advance, download
  riemann   exact Riemann problems of per-problem material pairs, host arrays in and out
  gradient  loss and gradient of the warm-start network on one training batch
"""
import ctypes as C
import math

import numpy as np
import torch

from m2c_b200 import abi, cases, gpu

FLUX = {"hllc": abi.FLUX_HLLC, "roe": abi.FLUX_ROE, "llf": abi.FLUX_LLF}
LIMITER = {"vanalbada": abi.LIM_VANALBADA, "minmod": abi.LIM_GENMINMOD, "none": abi.LIM_NONE}
PRECISION = {"fp64": abi.PREC_FP64, "mixed": abi.PREC_MIXED}
BOUNDARY = {
    "periodic": (abi.BC_PERIODIC,) * 6,
    "walls": (abi.BC_SYMMETRY,) * 6,
    # a channel: inflow and outflow along x, two kinds of wall across y, symmetry in z
    "channel": (abi.BC_INLET, abi.BC_OUTLET, abi.BC_SLIPWALL, abi.BC_STICKWALL, abi.BC_SYMMETRY, abi.BC_SYMMETRY),
}
BASE = (1.0, 0.0, 0.0, 0.0, 1.0 / 1.4)  # the box's mean state: ideal gas, sound speed 1


def listed():
    return [
        # one residual of a small piece of a domain: latency, the smallest call a host integrator makes
        dict(name="residual_24x20x18", kind="residual", nx=24, ny=20, nz=18, bc="channel", mesh="stretched", flux="hllc",
             limiter="vanalbada", precision="fp64"),
        # the standard 1D validation run, all its steps to t = 0.2: launches and host round trips
        dict(name="sod_400", kind="run", field="sod", nx=400, ny=1, nz=1, bc="sod", mesh="uniform", flux="hllc",
             limiter="vanalbada", rk=2, precision="fp64", steps=100000, t_max=0.2),
        # a development-size box, too small to fill the chip
        dict(name="box_64_mixed", kind="run", field="fourier", nx=64, ny=64, nz=64, bc="channel", mesh="uniform",
             flux="hllc", limiter="vanalbada", rk=2, precision="mixed", steps=40, t_max=0.0),
        # the FP64 path on an odd-sized, stretched channel: ragged tiles on every axis
        dict(name="channel_161x97x131_fp64", kind="run", field="fourier", nx=161, ny=97, nz=131, bc="channel",
             mesh="stretched", flux="hllc", limiter="vanalbada", rk=3, precision="fp64", steps=10, t_max=0.0),
        # the single-material production box
        dict(name="box_256_mixed", kind="run", field="fourier", nx=256, ny=256, nz=256, bc="periodic", mesh="uniform",
             flux="roe", limiter="minmod", rk=3, precision="mixed", steps=10, t_max=0.0),
        # one step as the drop-in integrator makes it, host arrays in the reference's layout
        dict(name="dropin_step_64_fp64", kind="step", nx=64, ny=64, nz=64, nbubbles=1, rk=3, precision="fp64"),
        # a single collapsing bubble in FP64, odd-sized; two reinitialisations
        dict(name="bubble_101x96x90_fp64", kind="bubbles", nx=101, ny=96, nz=90, nbubbles=1, rk=3, precision="fp64",
             steps=20),
        # the headline workload at the size whose inputs are quick to make: bubble cluster at first shock contact,
        # one reinitialisation
        dict(name="cluster_256_mixed", kind="bubbles", nx=256, ny=256, nz=256, nbubbles=16, rk=3, precision="mixed",
             steps=10),
        # a box cut by an embedded plane
        dict(name="plane_96_mixed", kind="plane", nx=96, ny=96, nz=96, rk=3, precision="mixed", steps=5),
        # the batched shock tubes
        dict(name="tubes_1024", kind="tubes", ntubes=1024, lmin=100, lmax=2000, rk=2, steps=40),
        # labelling a training set for the warm start
        dict(name="riemann_100000", kind="riemann", n=100000),
        # one batch of the warm start's training: forward and backward
        dict(name="gradient_8192", kind="gradient", n=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["residual", "run", "run", "run", "bubbles", "bubbles", "step", "plane", "tubes", "riemann",
                       "gradient"])
    if kind == "residual":
        n = [_log_int(rng, 8, 96) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], bc=rng.choice(["periodic", "walls", "channel"]),
                    mesh=rng.choice(["uniform", "stretched"]), flux=rng.choice(["hllc", "roe", "llf"]),
                    limiter=rng.choice(["vanalbada", "minmod"]), precision=rng.choice(["fp64", "mixed"]))
    if kind == "run" and rng.random() < 0.25:
        return dict(kind=kind, field="sod", nx=_log_int(rng, 64, 2000), ny=1, nz=1, bc="sod", mesh="uniform",
                    flux=rng.choice(["hllc", "roe", "llf"]), limiter=rng.choice(["vanalbada", "minmod"]),
                    rk=rng.choice([2, 3]), precision="fp64", steps=100000, t_max=round(rng.uniform(0.05, 0.2), 3))
    if kind == "run":
        precision = rng.choice(["fp64", "mixed"])
        n = [_log_int(rng, 24, 160 if precision == "fp64" else 224) for _ in range(3)]
        return dict(kind=kind, field="fourier", nx=n[0], ny=n[1], nz=n[2],
                    bc=rng.choice(["periodic", "walls", "channel"]), mesh=rng.choice(["uniform", "uniform", "stretched"]),
                    flux=rng.choice(["hllc", "roe", "llf"]), limiter=rng.choice(["vanalbada", "minmod"]),
                    rk=rng.choice([2, 3]), precision=precision, steps=rng.randint(5, 15), t_max=0.0)
    if kind in ("bubbles", "step"):
        precision = rng.choice(["fp64", "mixed"])
        n = _log_int(rng, 32, (96 if kind == "step" else 128) if precision == "fp64" else 176)
        c = dict(kind=kind, nx=n + rng.randint(0, 7), ny=n + rng.randint(0, 7), nz=n + rng.randint(0, 7),
                 nbubbles=rng.choice([1, 4, 16]) if n >= 96 else 1, rk=rng.choice([2, 3]), precision=precision)
        if kind == "bubbles":
            c["steps"] = rng.randint(3, 15)
        return c
    if kind == "plane":
        n = [_log_int(rng, 24, 128) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], rk=rng.choice([2, 3]),
                    precision=rng.choice(["fp64", "mixed"]), steps=rng.randint(2, 6))
    if kind == "tubes":
        lmin = rng.randint(20, 200)
        return dict(kind=kind, ntubes=_log_int(rng, 8, 1024), lmin=lmin, lmax=lmin * rng.randint(2, 8),
                    rk=rng.choice([2, 3]), steps=rng.randint(5, 30))
    if kind == "riemann":
        return dict(kind=kind, n=_log_int(rng, 100, 100000))
    return dict(kind=kind, n=_log_int(rng, 64, 65536))


# ----------------------------------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def _coordinates(g):
    return [torch.tensor(c, dtype=torch.float64, device=_device()) for c in abi.cell_centres(g)]


def _ghosted(inner):
    """[c, nz, ny, nx] on the device -> pinned host array in the reference's ghosted layout, ghosts zero."""
    c, nz, ny, nx = inner.shape
    full = torch.zeros((nz + 2, ny + 2, nx + 2, c), dtype=torch.float64, device=inner.device)
    full[1:-1, 1:-1, 1:-1] = inner.permute(1, 2, 3, 0)
    host = _pinned(full.shape if c > 1 else full.shape[:3])
    torch.from_numpy(host).copy_(full if c > 1 else full[..., 0])
    return host


def _single(case):
    """Grid, scheme and materials of a single-material case."""
    shape = (case["nx"], case["ny"], case["nz"])
    if case["bc"] == "sod":
        bc = (abi.BC_INLET, abi.BC_OUTLET) + (abi.BC_SYMMETRY,) * 4
    else:
        bc = BOUNDARY[case["bc"]]
    g = abi.grid(*shape, bc=bc, inlet=BASE, outlet=BASE)
    if case["mesh"] == "stretched":
        cases.stretch(g, seed=3)
    s = abi.scheme(flux=FLUX[case["flux"]], limiter=LIMITER[case["limiter"]], minmod_coeff=1.0,
                   rk_order=case.get("rk", 2), cfl=0.5 if case["bc"] == "sod" else 0.4,
                   precision=PRECISION[case["precision"]])
    return g, s, [abi.material(1.4, 0.0)]


def _sod_states(seed):
    r = np.random.default_rng(seed)
    left = (1.0 * r.uniform(0.9, 1.1), 0.0, 0.0, 0.0, 1.0 * r.uniform(0.9, 1.1))
    right = (0.125 * r.uniform(0.9, 1.1), 0.0, 0.0, 0.0, 0.1 * r.uniform(0.9, 1.1))
    return left, right


def _field(case, g, seed):
    """Interior primitive state [5, nz, ny, nx] on the device."""
    if case.get("field") == "sod":
        left, right = _sod_states(seed)
        x = _coordinates(g)[0]
        lo, hi = (torch.tensor(v, dtype=torch.float64, device=x.device) for v in (left, right))
        return torch.where(x < 0.5, lo[:, None], hi[:, None])[:, None, None, :].contiguous()
    # smooth seeded Fourier modes about BASE: 1% in density and pressure, a solenoidal velocity of RMS Mach 0.3
    r = np.random.default_rng(seed)
    X, Y, Z = _coordinates(g)

    def wave():
        while True:
            k = r.integers(-6, 7, 3)
            if 1 <= np.linalg.norm(k) <= 6:
                break
        tp = 2 * math.pi
        return k, torch.cos(tp * (float(k[2]) * Z[:, None, None] + float(k[1]) * Y[None, :, None] +
                                  float(k[0]) * X[None, None, :]) + r.uniform(0, tp))

    V = torch.zeros((5, len(Z), len(Y), len(X)), dtype=torch.float64, device=X.device)
    for _ in range(6):
        V[0] += wave()[1]
        V[4] += wave()[1]
    for c in (0, 4):
        V[c] = BASE[c] * (1.0 + 0.01 * V[c] / math.sqrt(3.0))
    for _ in range(6):
        k, w = wave()
        b = np.cross(k, r.normal(size=3))
        for d in range(3):
            V[1 + d] += float(b[d]) * w
    V[1:4] *= 0.3 / math.sqrt(float((V[1:4] ** 2).sum(0).mean()))
    return V


def _bubble_setup(case, seed):
    """Bubbles in a 2 cm cube of water with a planar shock about to reach the nearest of them: grid, scheme,
    materials, level set, and the interior state, material IDs and signed distance on the device."""
    L = 0.02
    n = (case["nx"], case["ny"], case["nz"])
    rho1, u1 = cases.post_shock_sg(1000.0, 1.0e5, 1.0e9, **cases.WATER)
    g = abi.grid(*n, x=(0.0, L), y=(0.0, L), z=(0.0, L), bc=(abi.BC_INLET, abi.BC_OUTLET) + (abi.BC_SYMMETRY,) * 4,
                 inlet=(rho1, u1, 0.0, 0.0, 1.0e9), outlet=(1000.0, 0.0, 0.0, 0.0, 1.0e5))
    s = abi.scheme(flux=abi.FLUX_HLLC, limiter=abi.LIM_VANALBADA, rk_order=case["rk"], cfl=0.4,
                   precision=PRECISION[case["precision"]])
    mats = [abi.material(**cases.WATER), abi.material(**cases.AIR)]
    ls = abi.levelset(material_id=1, reinit_frequency=10)
    r, h = np.random.default_rng(seed), L / min(n)
    if case["nbubbles"] == 1:
        centres, radii = [L * (0.5 + 0.02 * r.uniform(-1, 1, 3))], [2.0e-3 * r.uniform(0.9, 1.1)]
    else:
        centres, radii = [], []
        while len(centres) < case["nbubbles"]:
            q = r.uniform(0.5e-3, 1.5e-3)
            c = r.uniform(q + 2 * h, L - q - 2 * h, 3)
            c[0] = r.uniform(0.0075 + q + 2 * h, L - q - 2 * h)
            if all(np.linalg.norm(c - c2) >= q + q2 + 2 * h for c2, q2 in zip(centres, radii)):
                centres.append(c)
                radii.append(q)
    X, Y, Z = _coordinates(g)
    phi = torch.full((n[2], n[1], n[0]), math.inf, dtype=torch.float64, device=X.device)
    for c, q in zip(centres, radii):
        d2 = (Z[:, None, None] - c[2]) ** 2 + (Y[None, :, None] - c[1]) ** 2 + (X[None, None, :] - c[0]) ** 2
        phi = torch.minimum(phi, d2.sqrt_() - q)
    front = min(c[0] - q for c, q in zip(centres, radii)) - 2 * L / n[0]
    shocked, air = (X < front)[None, None, :].expand_as(phi), phi < 0
    V = torch.zeros((5,) + tuple(phi.shape), dtype=torch.float64, device=X.device)
    for c, (post, water, gas) in {0: (rho1, 1000.0, 1.2), 1: (u1, 0.0, 0.0), 4: (1.0e9, 1.0e5, 1.0e5)}.items():
        V[c] = torch.where(air, gas, torch.where(shocked, post, water).double())
    return g, s, mats, ls, V, air.double(), phi


def _riemann_inputs(n, seed):
    """n problems of the batched tubes' distribution that the solver solves (others are redrawn, as the tubes'
    set-up does): material table, left and right states, normals."""
    r, s = np.random.default_rng(seed), cases.tube_scheme()
    keep = [[], [], [], []]
    have = 0
    while have < n:
        m = n - have + 64 + n // 16
        gamma = r.uniform(1.2, 7.0, (m, 2))
        pinf = np.where(r.random((m, 2)) < 0.25, 0.0, 10.0 ** r.uniform(6.0, 9.0, (m, 2)))
        VL, VR = cases.tube_states(m, r)
        VL[:, 2:4], VR[:, 2:4] = r.uniform(-20.0, 20.0, (m, 2)), r.uniform(-20.0, 20.0, (m, 2))
        dirs = r.normal(size=(m, 3))
        dirs /= np.linalg.norm(dirs, axis=1)[:, None]
        err = gpu.riemann_batch_pairs(s, abi.material_table(gamma.ravel(), pinf.ravel()), VL, VR, dirs)[6]
        ok = err == 0
        for k, a in zip(keep, (np.stack([gamma, pinf], 2), VL, VR, dirs)):
            k.append(a[ok])
        have += int(ok.sum())
    mat, VL, VR, dirs = (np.ascontiguousarray(np.concatenate(k)[:n]) for k in keep)
    return s, mat, VL, VR, dirs


def _tube_inputs(case, seed):
    """Tubes none of which meets a non-physical state in the case's steps (those that do are redrawn), and the tuning
    measured for them. The lengths belong to the case, the materials and states to the seed."""
    n, s = case["ntubes"], cases.tube_scheme(rk_order=case["rk"])
    lens = np.random.default_rng(n).integers(case["lmin"], case["lmax"] + 1, n).astype(np.int32)
    r = np.random.default_rng(seed)
    mats, (VL, VR) = np.empty((n, 2), object), cases.tube_states(n, r)
    flat = lambda at: [m for t in at for m in mats[t]]  # noqa: E731
    new = np.arange(n)
    while len(new):
        for t in new:
            mats[t] = cases.stiffened_gas_pair(r), cases.stiffened_gas_pair(r)
        VL[new], VR[new] = cases.tube_states(len(new), r)
        bad = gpu.tube_rejects(s)(flat(new), VL[new], VR[new])
        go = new[~bad]
        if len(go):
            b = gpu.Batch(s, lens[go], flat(go), VL[go], VR[go], 512, 256, 1)
            b.time_steps(case["steps"], check_errors=False)
            bad[~bad] = b.tube_errors() != 0
            b.close()
        new = new[bad]
    b = gpu.Batch(s, lens, flat(range(n)), VL, VR)
    tuning = b.tuning()
    b.close()
    return s, lens, flat(range(n)), VL, VR, tuning


def _plane_faces(nx, ny, nz):
    jj, kk = np.meshgrid(np.arange(ny), np.arange(nz), indexing="ij")
    f = np.zeros((ny * nz, 4), np.int32)
    f[:, 1], f[:, 2], f[:, 3] = nx // 2, jj.ravel(), kk.ravel()
    return f


def _gradient_inputs(n, seed):
    r = np.random.default_rng(seed)
    X = r.normal(size=(n, gpu.Mlp.NIN)).astype(np.float32)
    return X, (np.tanh(X[:, 0] - 0.5 * X[:, 3]) + 0.1 * r.normal(size=n)).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": dict(case)}
    if kind in ("residual", "run"):
        g, s, mats = _single(case)
        if case.get("field") == "sod":
            left, right = _sod_states(seed)
            g.inlet, g.outlet = (C.c_double * 5)(*left), (C.c_double * 5)(*right)
        st["V"] = _ghosted(_field(case, g, seed))
        st["solver"] = gpu.Solver(g, s, mats)
        st["out"] = _pinned(st["V"].shape)
        st["solver"].upload(st["V"])
    elif kind in ("bubbles", "step"):
        g, s, mats, ls, V, ID, phi = _bubble_setup(case, seed)
        st["in"] = [_ghosted(V), _ghosted(ID[None]), _ghosted(phi[None])]
        del V, ID, phi
        st["out"] = [_pinned(a.shape) for a in st["in"]]
        if kind == "step":  # the host code's own arrays: not pinned
            st["in"], st["out"] = [a.copy() for a in st["in"]], [np.zeros(a.shape) for a in st["in"]]
        st["solver"] = gpu.Solver(g, s, mats, ls)
        st["solver"].upload(*st["in"])
        st["dt"] = st["solver"].compute_dt()
    elif kind == "plane":
        full = dict(case, bc="periodic", mesh="uniform", flux="roe", limiter="minmod", field="fourier")
        g, s, mats = _single(full)
        st["V"] = _ghosted(_field(full, g, seed))
        st["solver"] = gpu.Solver(g, s, mats)
        st["solver"].set_wall_faces(_plane_faces(case["nx"], case["ny"], case["nz"]))
        st["out"] = _pinned(st["V"].shape)
    elif kind == "tubes":
        st["tubes"] = _tube_inputs(case, seed)
    elif kind == "riemann":
        st["s"], mat, st["VL"], st["VR"], st["dirs"] = _riemann_inputs(case["n"], seed)
        st["mats"] = abi.material_table(np.ascontiguousarray(mat[:, :, 0]).ravel(),
                                        np.ascontiguousarray(mat[:, :, 1]).ravel())
    else:
        st["net"] = gpu.Mlp(seed=seed)
        st["X"], st["y"] = _gradient_inputs(case["n"], seed)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "residual":
        return {"R": st["solver"].residual()}
    if kind in ("run", "plane"):
        sol = st["solver"]
        sol.t = 0.0
        sol.upload(st["V"])
        _, t = sol.run(case["steps"], case.get("t_max", 0.0) or math.inf)
        sol.download(out_V=st["out"], with_id=False)
        return {"V": st["out"], "t": t}
    if kind == "bubbles":
        sol = st["solver"]
        sol.t = 0.0
        sol.upload(*st["in"])
        _, t = sol.run(case["steps"])
        V, ID, phi = sol.download(*st["out"])
        return {"V": V, "ID": ID.astype(np.int8), "phi": phi, "t": t}
    if kind == "step":
        sol = st["solver"]
        sol.t, sol.step = 0.0, 0
        sol.upload(*st["in"])
        sol.advance(st["dt"])
        V, ID, phi = sol.download(*st["out"])
        return {"V": V, "ID": ID, "phi": phi}
    if kind == "tubes":
        s, lens, mats, VL, VR, tuning = st["tubes"]
        b = gpu.Batch(s, lens, mats, VL, VR, **tuning)
        b.run(case["steps"])
        V, ID, t = b.download()
        b.close()
        return {"V": V[0].base, "ID": ID[0].base, "t": t}
    if kind == "riemann":
        Vs, mid, Vsm, Vsp, it, ev, err = gpu.riemann_batch_pairs(st["s"], st["mats"], st["VL"], st["VR"], st["dirs"])
        return {"Vs": Vs, "id": mid, "Vsm": Vsm, "Vsp": Vsp, "iterations": it, "evaluations": ev, "err": err}
    loss, grad = st["net"].loss_grad(st["X"], st["y"])
    return {"loss": np.float32(loss), "grad": grad}


# ----------------------------------------------------------------------------------------------------------------
# work
# ----------------------------------------------------------------------------------------------------------------
STAGE_FLOPS = 650.0  # per cell and stage: 15 limited slopes, 6 face checks, 3 fluxes, the update


def _sod_steps(case):
    return 0.88 * case["nx"] * case["t_max"] / 0.2  # about 350 steps of CFL 0.5 for 400 cells to t = 0.2


def work(case):
    kind = case["kind"]
    if kind == "riemann":
        # in: two states, normal, two materials; out: three states and four integers. A solve evaluates both waves
        # at about five trial pressures.
        return {"bytes": case["n"] * (13 * 8 + 2 * 40 + 15 * 8 + 16), "flops": case["n"] * 5 * 2 * 100.0}
    if kind == "gradient":
        p = 16 * 64 + 2 * 64 * 64 + 64
        return {"bytes": case["n"] * 17 * 4 + 2 * gpu.Mlp.NPARAM * 4, "flops": 6.0 * p * case["n"]}
    if kind == "tubes":
        cells = case["ntubes"] * 0.5 * (case["lmin"] + case["lmax"])
        vec = {1: 2, 2: 5, 3: 8}[case["rk"]]
        return {"bytes": cells * (48.0 * vec * case["steps"] + 2 * 44), "flops": cells * 250.0 * case["rk"] * case["steps"]}
    cells = float(case["nx"] * case["ny"] * case["nz"])
    if kind == "residual":
        return {"bytes": cells * 80.0, "flops": cells * STAGE_FLOPS}
    steps = 1 if kind == "step" else (_sod_steps(case) if case.get("field") == "sod" else case["steps"])
    vec = {1: 2, 2: 5, 3: 8}[case["rk"]]
    per = 48.0 if kind in ("bubbles", "step") else 40.0  # state vector, with phi where there is a level set
    io = 2 * (per + (8.0 if kind in ("bubbles", "step") else 0.0))
    return {"bytes": cells * (per * vec * steps + io), "flops": cells * STAGE_FLOPS * case["rk"] * steps}


# ----------------------------------------------------------------------------------------------------------------
# 64-bit values
# ----------------------------------------------------------------------------------------------------------------
def _axis_coefficients(w, periodic):
    dm = torch.roll(w, 1)
    dp = torch.roll(w, -1)
    if not periodic:
        dm[0], dp[-1] = w[0], w[-1]
    return (dm + w) / (w + dp), 2.0 * w / (w + dp)


class _Box:
    """The scheme (MUSCL, limiter, flux, RK with a CFL step) on one ideal gas, written with whole-array operations."""

    def __init__(self, case, g, s):
        self.dev = _device()
        self.gam = 1.4
        self.flux, self.limiter, self.alpha, self.delta = case["flux"], case["limiter"], s.minmod_coeff, s.roe_delta
        self.bc = list(g.bc)
        self.ghost = {abi.BC_INLET: list(g.inlet), abi.BC_OUTLET: list(g.outlet)}
        self.n = (g.nx, g.ny, g.nz)
        mesh = getattr(g, "_mesh", {})
        span = ((g.x0, g.xmax), (g.y0, g.ymax), (g.z0, g.zmax))
        self.w, self.A, self.B, self.K = [], [], [], []
        for a in range(3):
            w = mesh[a][1] if a in mesh else np.full(self.n[a], (span[a][1] - span[a][0]) / self.n[a])
            w = torch.tensor(w, dtype=torch.float64, device=self.dev)
            A, B = _axis_coefficients(w, self.bc[2 * a] == abi.BC_PERIODIC)
            K = torch.zeros_like(A)
            for i, (p, q) in enumerate(zip(A.tolist(), B.tolist())):
                k = 2
                while q > 2.0 / (1.0 + ((k - 1.0) / k) ** (k - 1) / k) * min(p, 1.0):
                    k += 1
                K[i] = k
            self.w.append(w)
            self.A.append(A)
            self.B.append(B)
            self.K.append(K)

    def sound(self, V):
        return torch.sqrt(self.gam * V[4] / V[0])

    def cons(self, V):
        q = V[1] ** 2 + V[2] ** 2 + V[3] ** 2
        return torch.stack([V[0], V[0] * V[1], V[0] * V[2], V[0] * V[3], V[4] / (self.gam - 1.0) + 0.5 * V[0] * q])

    def prim(self, U):
        u = U[1:4] / U[0]
        p = (self.gam - 1.0) * (U[4] - 0.5 * U[0] * (u ** 2).sum(0))
        return torch.stack([U[0], u[0], u[1], u[2], p])

    def physical(self, V, d):
        F = self.cons(V)
        F[4] += V[4]
        F *= V[1 + d]
        F[1 + d] += V[4]
        return F

    def roe_average(self, L, R):
        a, b = torch.sqrt(L[0]), torch.sqrt(R[0])
        return lambda x, y: (a * x + b * y) / (a + b)

    def hat(self, L, R, d):
        """Generalized Roe averages of the ideal gas (dp/drho = (gamma-1) e, Gamma = gamma-1), with the eps of the
        scheme: density, internal energy, dp/drho, Gamma and sound speed."""
        avg, g1, eps = self.roe_average(L, R), self.gam - 1.0, 1.0e-10
        rho = torch.sqrt(L[0] * R[0])
        eL, eR = L[4] / (g1 * L[0]), R[4] / (g1 * R[0])
        diff = (R[1 + d] - L[1 + d]) / (torch.sqrt(L[0]) + torch.sqrt(R[0]))
        pr = avg(L[4] / L[0], R[4] / R[0]) + 0.5 * diff ** 2
        e = avg(eL, eR)
        dr, de, dp = R[0] - L[0], eR - eL, R[4] - L[4]
        wr, we = dr ** 2 / rho ** 2, de ** 2 / e ** 2
        den, pa, ga = wr + we + eps, avg(g1 * eL, g1 * eR), g1
        dpdr = ((we + eps) * pa + (dp - ga * rho * de) * dr / rho ** 2) / den
        G = ((wr + eps) * ga + (dp - pa * dr) * de / (rho * e ** 2)) / den
        return rho, e, dpdr, G, torch.sqrt(dpdr + G * pr)

    def numerical(self, L, R, d):
        cL, cR = self.sound(L), self.sound(R)
        if self.flux == "llf":
            a = torch.maximum(L[1 + d].abs() + cL, R[1 + d].abs() + cR)
            return 0.5 * (self.physical(L, d) + self.physical(R, d) - a * (self.cons(R) - self.cons(L)))
        avg = self.roe_average(L, R)
        rho, e, dpdr, G, c = self.hat(L, R, d)
        if self.flux == "hllc":
            uL, uR, u = L[1 + d], R[1 + d], avg(L[1 + d], R[1 + d])
            sL, sR = torch.minimum(uL - cL, u - c), torch.maximum(uR + cR, u + c)
            star = (R[4] - L[4] + L[0] * uL * (sL - uL) - R[0] * uR * (sR - uR)) / \
                   (L[0] * (sL - uL) - R[0] * (sR - uR))

            def side(V, S):
                U, v = self.cons(V), V[1 + d]
                k = torch.stack([torch.ones_like(v), V[1], V[2], V[3],
                                 U[4] / V[0] + (star - v) * (star + V[4] / (V[0] * (S - v)))])
                k[1 + d] = star
                return self.physical(V, d) + S * (k * (V[0] * (S - v) / (S - star)) - U)

            F = torch.where(star >= 0, side(L, sL), side(R, sR))
            F = torch.where(sL >= 0, self.physical(L, d), F)
            return torch.where(sR <= 0, self.physical(R, d), F)
        g1 = self.gam - 1.0
        H = avg(*[V[4] / (g1 * V[0]) + 0.5 * (V[1] ** 2 + V[2] ** 2 + V[3] ** 2) + V[4] / V[0] for V in (L, R)])
        vel = [avg(L[1 + i], R[1 + i]) for i in range(3)]
        un, dn, D = vel[d], R[1 + d] - L[1 + d], R - L
        lam = [un - c, un, un + c]
        tol = self.delta * torch.maximum(lam[0], torch.maximum(un.abs(), lam[2].abs()))
        lam = [torch.where(x.abs() < tol, (x * x + tol * tol) / (2 * tol), x).abs() for x in lam]
        F = 0.5 * (self.physical(L, d) + self.physical(R, d))
        one, q = torch.ones_like(un), vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2
        for sign, l in ((-1.0, lam[0]), (1.0, lam[2])):
            k = torch.stack([one, vel[0], vel[1], vel[2], H + sign * un * c])
            k[1 + d] = un + sign * c
            F -= 0.5 * l * (D[4] + sign * rho * c * dn) / (2 * c * c) * k
        F -= 0.5 * lam[1] * (D[0] - D[4] / (c * c)) * torch.stack([one, *vel, e + 0.5 * q - dpdr / G])
        for i in range(3):
            if i != d:
                w = 0.5 * lam[1] * rho * D[1 + i]
                F[1 + i] -= w
                F[4] -= w * vel[i]
        return F

    def ghost_of(self, inner, a, side):
        """The state beyond a boundary, for the inner neighbour `inner` (cell or face state)."""
        bc = self.bc[2 * a + side]
        if bc in self.ghost:
            g = torch.tensor(self.ghost[bc], dtype=torch.float64, device=self.dev)
            return g.reshape([5] + [1] * (inner.dim() - 1)).expand_as(inner).clone()
        out = inner.clone()
        if bc == abi.BC_STICKWALL:
            out[1:4] = -out[1:4]
        else:
            out[1 + a] = -out[1 + a]
        return out

    def along(self, x, a):
        s = [1, 1, 1]
        s[2 - a] = -1
        return x.reshape(s)

    def slope(self, dl, dr, a):
        if self.limiter == "none":
            return 0.5 * (dl + dr)
        A, B = self.along(self.A[a], a), self.along(self.B[a], a)
        if self.limiter == "minmod":
            mid = B / (A + 1.0) * (dl + dr)
            low = torch.minimum(self.alpha * dl, torch.minimum(mid, self.alpha * dr))
            high = torch.maximum(self.alpha * dl, torch.maximum(mid, self.alpha * dr))
            zero = torch.zeros_like(dl)
            return torch.where((dl > 0) & (dr > 0), low, torch.where((dl < 0) & (dr < 0), high, zero))
        on = (dl * dr > 0) & (dl * dr >= 1.0e-16)
        K = self.along(self.K[a], a)
        if bool((self.K[a] == 2).all()):
            p0, p1 = dl * dl, dr * dr
        else:
            p0, p1 = torch.pow(dl.abs(), K), torch.pow(dr.abs(), K)
            odd = K % 2 == 1
            p0, p1 = torch.where(odd, p0 * dl.sign(), p0), torch.where(odd, p1 * dr.sign(), p1)
        return torch.where(on, B * (dr * p0 + dl * p1) / torch.where(on, p0 + A * p1, torch.ones_like(p0)),
                           torch.zeros_like(p0))

    def residual(self, V):
        out = torch.zeros_like(V)
        for a in range(3):
            if self.n[a] == 1:
                continue  # a single cell between mirror walls: its two fluxes cancel
            d = 3 - a
            first, last = V.narrow(d, 0, 1), V.narrow(d, self.n[a] - 1, 1)
            per = self.bc[2 * a] == abi.BC_PERIODIC
            lo, hi = (last, first) if per else (self.ghost_of(first, a, 0), self.ghost_of(last, a, 1))
            diff = torch.diff(torch.cat([lo, V, hi], d), dim=d)
            s = self.slope(diff.narrow(d, 0, self.n[a]), diff.narrow(d, 1, self.n[a]), a)
            del diff
            minus, plus = V - 0.5 * s, V + 0.5 * s
            del s
            m0, p1 = minus.narrow(d, 0, 1), plus.narrow(d, self.n[a] - 1, 1)
            glo, ghi = (p1, m0) if per else (self.ghost_of(m0, a, 0), self.ghost_of(p1, a, 1))
            F = self.numerical(torch.cat([glo, plus], d), torch.cat([minus, ghi], d), a)
            del minus, plus
            out -= torch.diff(F, dim=d) / self.along(self.w[a], a)
        return out

    def step_size(self, V, cfl):
        c = self.sound(V)
        return cfl * min(float((self.along(self.w[a], a) / (V[1 + a].abs() + c)).min()) for a in range(3))

    def run(self, V, steps, t_max, cfl, rk):
        t, k = 0.0, 0
        while k < steps and t < t_max:
            dt = self.step_size(V, cfl)
            if t + dt > t_max:
                dt = t_max - t
            t += dt
            U0 = self.cons(V)
            U = U0 + dt * self.residual(V)
            if rk == 2:
                U = 0.5 * U0 + 0.5 * U + 0.5 * dt * self.residual(self.prim(U))
            elif rk == 3:
                U = 0.75 * U0 + 0.25 * U + 0.25 * dt * self.residual(self.prim(U))
                U = U0 / 3.0 + 2.0 / 3.0 * U + 2.0 / 3.0 * dt * self.residual(self.prim(U))
            V = self.prim(U)
            k += 1
        return V, t

    def with_ghosts(self, V):
        """The host layout: one ghost layer by the boundary rule on the faces, zeros on edges and corners."""
        full = torch.zeros((V.shape[1] + 2, V.shape[2] + 2, V.shape[3] + 2, 5), dtype=torch.float64, device=self.dev)
        full[1:-1, 1:-1, 1:-1] = V.permute(1, 2, 3, 0)
        for a in range(3):
            d = 3 - a
            for side in (0, 1):
                edge = V.narrow(d, 0 if side == 0 else self.n[a] - 1, 1)
                if self.bc[2 * a] == abi.BC_PERIODIC:
                    edge = V.narrow(d, self.n[a] - 1 if side == 0 else 0, 1)
                else:
                    edge = self.ghost_of(edge, a, side)
                at = [slice(1, -1)] * 3
                at[2 - a] = slice(0, 1) if side == 0 else slice(-1, None)
                full[tuple(at)] = edge.permute(1, 2, 3, 0)
        return full.cpu().numpy()


def _star_states(mat, VL, VR, dirs):
    """Exact star states of stiffened-gas Riemann problems: bisection on the pressure in the closed wave curves."""
    g, P = mat[:, :, 0], mat[:, :, 1]
    side = []
    for q, V in ((0, VL), (1, VR)):
        side.append((V[:, 0], (V[:, 1:4] * dirs).sum(1), V[:, 4] + P[:, q], g[:, q], P[:, q]))

    def wave(s, p):
        """Velocity change across the wave and the density behind it."""
        rho, _, k, gam, pinf = s
        x = np.maximum(p + pinf, 1e-300) / k
        c = np.sqrt(gam * k / rho)
        shock = x > 1
        with np.errstate(invalid="ignore", over="ignore"):
            f = np.where(shock, k * (x - 1) * np.sqrt(2.0 / (rho * k * ((gam + 1) * x + gam - 1))),
                         2 * c / (gam - 1) * (x ** ((gam - 1) / (2 * gam)) - 1))
            r = np.where(shock, rho * ((gam + 1) * x + gam - 1) / ((gam - 1) * x + gam + 1), rho * x ** (1 / gam))
        return f, r

    # pressures measured from the smaller stiffness: p + S > 0 is where both curves exist
    S = np.minimum(P[:, 0], P[:, 1])
    lo = np.full(len(S), -400.0)
    hi = np.full(len(S), 80.0)
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        p = np.exp(mid) - S
        f = wave(side[0], p)[0] + wave(side[1], p)[0] + side[1][1] - side[0][1]
        lo, hi = np.where(f < 0, mid, lo), np.where(f < 0, hi, mid)
    p = np.exp(0.5 * (lo + hi)) - S
    (fl, rl), (fr, rr) = wave(side[0], p), wave(side[1], p)
    u = 0.5 * (side[0][1] - fl + side[1][1] + fr)
    out = []
    for V, s, r in ((VL, side[0], rl), (VR, side[1], rr)):
        W = np.empty_like(V)
        W[:, 0], W[:, 4] = r, p
        W[:, 1:4] = V[:, 1:4] + (u - s[1])[:, None] * dirs
        out.append(W)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("residual", "run"):
        g, s, _ = _single(case)
        if case.get("field") == "sod":
            left, right = _sod_states(seed)
            g.inlet, g.outlet = (C.c_double * 5)(*left), (C.c_double * 5)(*right)
        box = _Box(case, g, s)
        V = _field(case, g, seed)
        if kind == "residual":
            R = np.zeros((case["nz"] + 2, case["ny"] + 2, case["nx"] + 2, 5))
            R[1:-1, 1:-1, 1:-1] = box.residual(V).permute(1, 2, 3, 0).cpu().numpy()
            return {"R": R}
        V, t = box.run(V, case["steps"], case["t_max"] or math.inf, s.cfl, case["rk"])
        return {"V": box.with_ghosts(V), "t": t}
    if kind == "riemann":
        _, mat, VL, VR, dirs = _riemann_inputs(case["n"], seed)
        Vsm, Vsp = _star_states(mat, VL, VR, dirs)
        # the state at xi = 0 inside a fan is interpolated by the solver, and the rest are counts
        return {"Vs": None, "id": None, "Vsm": Vsm, "Vsp": Vsp, "iterations": None, "evaluations": None, "err": None}
    if kind == "gradient":
        X, y = (torch.tensor(a, dtype=torch.float64) for a in _gradient_inputs(case["n"], seed))
        p = torch.tensor(gpu.Mlp(seed=seed).params()[0], dtype=torch.float64, requires_grad=True)
        h, at = X, 0
        for rows, cols in ((64, 16), (64, 64), (64, 64), (1, 64)):
            W, b = p[at:at + rows * cols].reshape(rows, cols), p[at + rows * cols:at + rows * cols + rows]
            at += rows * cols + rows
            h = h @ W.T + b
            h = torch.tanh(h) if rows > 1 else h[:, 0]
        loss = ((h - y) ** 2).mean()
        loss.backward()
        return {"loss": float(loss), "grad": p.grad.numpy()}
    return None
