"""Performance cases: the work a user of this framework has it do, through its public
entry points (``HiDEMLib``, ``HiDEMBatch``, ``Surrogate``), over the range of sizes, types
and options it is used with.

A case is a dict of plain values. ``listed()`` names the fixed ones, ``draw(rng)`` gives more
of the same ranges, ``prepare(case, seed)`` makes what a caller holds before the call,
``run(state)`` is one pass, ``work(case)`` the bytes and operations the pass cannot do
without, ``exact(case, seed)`` the same outputs in 64-bit arithmetic, written with torch alone.

The particle sets are FCC lattices at d = 1 m with seeded positions, increments, rotations,
link-end history and broken links, as a run that has been going for a while holds them: the
bonds are intact but for a seeded fraction, about half of the bonded neighbours overlap.
"""
from __future__ import annotations

import math

import numpy as np
import torch

SQRT2 = math.sqrt(2.0)
DEV = "cuda"
SETTLE_INPUTS, SETTLE_BANDS = 82, 4  # the settling network's shape (82 lattice inputs, 4 bands)

# Every run parameter the passes depend on (the ice-block configuration's material).
MATERIAL = dict(dt=1e-4, scale=1.0, E=1e9, beamWidth=0.6, damping=9100.0, dampingRotation=9100.0,
                attractDistance=0.0, attractScaleForce=0.0, maxLoad=5e-4, bendBreak=0.01,
                breakTime=0.0, g=9.81, rhoIce=910.0, rhoWater=1030.0, waterLevel=-1.0e3,
                airDrag=1.0, waterDrag=10.0, bedDrag=1000.0, bedStiffness=2e8, bedInteract=2.0,
                searchDistanceScale=1.2, maxRadius=0.5, bedHeight=0.0, bedFriction=1.0,
                useFixed=0, useBed=0, useFrontPressure=0)
FIXED, FRONT = 0x40, 0x80

POSITION = ("xCord", "yCord", "zCord")
THETA = ("xTheta", "yTheta", "zTheta")
DIFF = ("xDiff", "yDiff", "zDiff", "uDiff", "vDiff", "wDiff")
CT = ("CT0", "CT1", "CT2", "CT3", "CT4", "CT5")


# --------------------------------------------------------------------------- the cases

def listed():
    steps = lambda name, cells, precision, n, setting="block": dict(  # noqa: E731
        name=name, kind="steps", nx=cells[0], ny=cells[1], nz=cells[2], precision=precision,
        setting=setting, steps=n)
    return [
        # the smallest run a user makes: a 256-sphere block, ten steps and the state back
        # (launches, host work and latency)
        steps("block_256", (4, 4, 4), "mixed", 10),
        # the ice-block configuration: 32,000 spheres, bottom layer fixed, in air
        steps("block_32k", (20, 20, 20), "mixed", 20),
        # an odd-sized block in plain double precision
        steps("block_9k_fp64", (13, 19, 9), "fp64", 20),
        # the headline configuration: the 5.7M-particle calving slab on a bed, water line and
        # front pressure, mixed precision; the whole state back after forty steps
        steps("slab_5.7M", (283, 71, 71), "mixed", 40, "slab"),
        # the same slab in plain double precision
        steps("slab_5.7M_fp64", (283, 71, 71), "fp64", 20, "slab"),
        # a slab confined by a fjord-shaped collision mesh (the MeshConstrainedDem setting)
        steps("fjord_800k", (113, 42, 42), "mixed", 20, "fjord"),
        # the timestep through the reference's separate operator calls, as a sample main
        # drives it (gridService, computePartForce, applyForce, linkUpdate, finalizeTs)
        dict(name="split_37k", kind="split", nx=37, ny=23, nz=11, precision="mixed",
             setting="block", steps=10),
        # a neighbour-structure rebuild (cells, contact list, link ends) and the first forces
        dict(name="rebuild_800k", kind="rebuild", nx=113, ny=42, nz=42, precision="mixed",
             setting="slab"),
        # an ensemble of uneven blocks advanced together (5k to 80k particles each)
        dict(name="ensemble_32", kind="ensemble", blocks=32, n_min=5000, n_max=80000,
             precision="mixed", steps=20),
        # a whole job from the caller's pinned host arrays: upload, twenty steps, download
        dict(name="job_200k", kind="job", nx=71, ny=35, nz=20, precision="mixed", setting="slab",
             steps=20),
        # the warm start's predictions for the particles of a tongue, rows on the device
        dict(name="predict_262k", kind="predict", rows=262144 + 77, inputs=SETTLE_INPUTS,
             bands=SETTLE_BANDS),
        # ten training steps of the warm start's network at its settling batch
        dict(name="train_8192", kind="train", batch=8192, rows=65536, inputs=SETTLE_INPUTS,
             bands=SETTLE_BANDS, steps=10),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _cells(rng, n, flat):
    """Unit cells of a block or slab of about n particles."""
    base = (n / 4.0) ** (1.0 / 3.0)
    sx, sy = (rng.uniform(1.5, 3.0), rng.uniform(0.7, 1.2)) if flat else (rng.uniform(0.7, 1.5), rng.uniform(0.7, 1.5))
    nx, ny = max(2, round(base * sx)), max(2, round(base * sy))
    return nx, ny, max(2, round(n / (4.0 * nx * ny)))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "split", "rebuild", "ensemble", "job",
                       "predict", "train"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind in ("steps", "split", "rebuild", "job"):
        top = {"steps": 3e6, "split": 1e6, "rebuild": 2e6, "job": 5e5}[kind]
        n = _log_uniform(rng, 300, top)
        setting = rng.choice(["block", "slab", "fjord"] if kind in ("steps", "split") and n > 2e4 else ["block", "slab"])
        nx, ny, nz = _cells(rng, n, setting != "block")
        case = dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision, setting=setting)
        if kind != "rebuild":
            case["steps"] = rng.choice([1, 5, 10, 20, 25])
        return case
    if kind == "ensemble":
        return dict(kind="ensemble", blocks=rng.randint(3, 40), n_min=2000, n_max=rng.randint(10000, 80000),
                    precision=precision, steps=rng.choice([10, 15, 20]))
    inputs, bands = rng.choice([(5, 8), (82, 4), (82, 4), (98, 4), (40, 4)])
    if kind == "predict":
        return dict(kind="predict", rows=int(_log_uniform(rng, 1000, 2e6)), inputs=inputs, bands=bands)
    return dict(kind="train", batch=128 * rng.randint(8, 256), rows=rng.randint(40000, 200000),
                inputs=inputs, bands=bands, steps=rng.choice([1, 5, 10]))


# --------------------------------------------------------------------------- inputs

def _lp(case):
    return torch.float32 if case["precision"] == "mixed" else torch.float64


def _params(case):
    P = dict(MATERIAL)
    if case["setting"] == "block":
        P["useFixed"] = 1
    else:
        # flat bed half a diameter below the lowest centres, water line at 0.9 of the height,
        # front pressure on the x-max face
        P.update(useBed=1, bedHeight=0.5, bedFriction=0.3, useFrontPressure=1,
                 waterLevel=0.9 * case["nz"] * SQRT2)
        if case["setting"] == "fjord":
            P["bedInteract"] = 0.25
    return P


def _inputs(case, seed):
    """Particles and links of a lattice case, in input order, as tensors on the GPU."""
    nx, ny, nz, lp = case["nx"], case["ny"], case["nz"], _lp(case)
    gen = torch.Generator(device=DEV).manual_seed(1000003 * (seed % 1000003) + 17)
    n = 4 * nx * ny * nz
    i = torch.arange(n, device=DEV)
    s, c, j, k = i % 4, (i // 4) % nx, (i // (4 * nx)) % ny, i // (4 * nx * ny)
    site = torch.tensor([[0, 0, 0], [1, 1, 0], [1, 0, 1], [0, 1, 1]], device=DEV)
    h = [2 * c + site[s, 0], 2 * j + site[s, 1], 2 * k + site[s, 2]]  # half-cell coordinates
    uniform = lambda scale, count, dtype: (  # noqa: E731
        torch.rand(count, generator=gen, device=DEV, dtype=torch.float64) * 2 - 1).mul_(scale).to(dtype)
    x = [h[q].double() * (SQRT2 / 2) + uniform(1e-3, n, torch.float64) for q in range(3)]
    p = dict(zip(POSITION, x))
    p.update({f: uniform(1e-4, n, lp) for f in THETA})
    p.update({f: uniform(1e-6, n, lp) for f in DIFF})
    p["radius"] = torch.full((n,), 0.5, device=DEV, dtype=lp)
    p["type"] = torch.zeros(n, device=DEV, dtype=torch.uint8)
    if case["setting"] == "block":
        p["type"][h[2] == 0] = FIXED
    else:
        p["type"][h[0] == 2 * nx - 1] = FRONT
    # the twelve nearest neighbours, each pair once: end A the lower index
    parity = torch.tensor([[[0, -1], [-1, 3]], [[-1, 2], [1, -1]]], device=DEV)  # [x][y][z]
    lim = (2 * nx, 2 * ny, 2 * nz)
    pairs = []
    for o in ((1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1), (0, 1, 1), (0, 1, -1)):
        t = [h[q] + o[q] for q in range(3)]
        ok = torch.ones(n, dtype=torch.bool, device=DEV)
        for q in range(3):
            ok &= (t[q] >= 0) & (t[q] < lim[q])
        t = [v[ok] for v in t]
        other = 4 * ((t[2] // 2 * ny + t[1] // 2) * nx + t[0] // 2) + parity[t[0] % 2, t[1] % 2, t[2] % 2]
        a = i[ok]
        pairs.append(torch.minimum(a, other) * n + torch.maximum(a, other))
    key = torch.sort(torch.cat(pairs)).values
    del pairs
    A, B = key // n, key % n
    L = A.numel()
    length = torch.sqrt(sum((x[q][A] - x[q][B]) ** 2 for q in range(3)))
    l = dict(globalKeyEndA=A, globalKeyEndB=B, initialLen=length.to(lp),
             state=(torch.rand(L, generator=gen, device=DEV) >= 0.01).to(torch.uint8))
    l.update({f: uniform(1e3, 2 * L, lp) for f in CT})
    return p, l


def _fjord_mesh(case, precision):
    from hidem_b200 import abi, workloads
    top = [case[q] * SQRT2 for q in ("nx", "ny", "nz")]
    lo, hi = (-0.55, -0.55), (top[0] + 0.55, top[1] + 0.55, top[2] + 5.0)
    v, nrm = workloads.container_mesh(lo, hi, lambda xx, yy: -0.55 - 0.002 * (xx - lo[0]),
                                      max(1, round(top[0] / 4.0)), max(1, round(top[1] / 4.0)),
                                      walls=("x-", "y-", "y+"))
    return abi.mesh(v, nrm, 8.0, precision, mesh_force=1e5, mesh_drag=1000.0)


def _context(case, p, l):
    from hidem_b200 import abi
    from hidem_b200.hidemlib import HiDEMLib
    precision = abi.PREC_MIXED if case["precision"] == "mixed" else abi.PREC_FP64
    lib = HiDEMLib(abi.default_params(**_params(case), precision=precision))
    if p is not None:
        torch.cuda.synchronize()
        lib.set_particles(p)
        lib.set_links(l)
    if case["setting"] == "fjord":
        mesh, _keep = _fjord_mesh(case, precision)
        lib.set_collision_mesh(mesh)
    return lib


def _readback(n, L, lp, device=DEV, pin=False):
    make = lambda count, dtype: torch.empty(count, dtype=dtype, device=device, pin_memory=pin)  # noqa: E731
    p = {f: make(n, torch.float64) for f in POSITION}
    p.update({f: make(n, lp) for f in THETA + DIFF})
    l = {"state": make(L, torch.uint8)}
    l.update({f: make(2 * L, lp) for f in CT})
    return p, l


def _block_cases(case, seed):
    """The blocks of an ensemble: sizes log-uniform, each with inputs of its own."""
    rng = np.random.default_rng(7)  # the sizes are the case's, the contents the seed's
    n = np.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]), size=case["blocks"]))
    for q, e in enumerate(np.maximum(1, np.rint(np.cbrt(n / 4.0))).astype(int)):
        yield dict(case, kind="steps", setting="block", nx=int(e), ny=int(e), nz=int(e)), 1009 * seed + q


def _network(case, seed):
    """Parameters of a network as one flat array in the library's order, and input rows."""
    gen = torch.Generator(device=DEV).manual_seed(seed + 5)
    rand = lambda *shape: torch.rand(*shape, generator=gen, device=DEV) * 2 - 1  # noqa: E731
    k = max(128, -(-case["inputs"] * (1 + 2 * case["bands"]) // 128) * 128)
    params = []
    for _ in range(4):
        params += [rand(256, k) * math.sqrt(6.0 / k), rand(256) * 0.1]
        k = 256
    params += [rand(3, 256) * math.sqrt(3.0 / 256), rand(3) * 0.1]
    return params, rand(case["rows"], case["inputs"])


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("predict", "train"):
        from hidem_b200 import surrogate as sg
        params, rows = _network(case, seed)
        over = dict(inputs=case["inputs"], fourier_bands=case["bands"], seed=seed)
        if kind == "train":
            over["batch"] = case["batch"]
        net = sg.Surrogate(sg.default_config(**over))
        net.set_params(torch.cat([w.reshape(-1) for w in params]).cpu().numpy())
        if kind == "train":
            targets = torch.tanh(rows[:, :3] + 0.5 * rows[:, 1:4] * rows[:, 2:5])
            net.set_data(rows.cpu().numpy(), targets.cpu().numpy())
            return dict(case=case, net=net)
        out = torch.empty(case["rows"], 3, device=DEV)
        torch.cuda.synchronize()
        return dict(case=case, net=net, rows=rows, out=out)
    if kind == "ensemble":
        from hidem_b200.hidemlib import HiDEMBatch
        libs = []
        for c, s in _block_cases(case, seed):
            libs.append(_context(c, *_inputs(c, s)))
        P, K = _readback(sum(b.n for b in libs), sum(b.L for b in libs), _lp(case))
        views, i, j = [], 0, 0
        for b in libs:
            views.append(({f: v[i:i + b.n] for f, v in P.items()},
                          {f: (v[2 * j:2 * (j + b.L)] if f in CT else v[j:j + b.L]) for f, v in K.items()}))
            i, j = i + b.n, j + b.L
        return dict(case=case, libs=libs, batch=HiDEMBatch(libs), views=views, out={**P, **K})
    p, l = _inputs(case, seed)
    n, L = p["xCord"].numel(), l["state"].numel()
    if kind == "job":
        host = lambda d: {f: v.cpu().pin_memory() for f, v in d.items()}  # noqa: E731
        links = host({f: v for f, v in l.items() if f not in CT})
        P, _ = _readback(n, 1, _lp(case), device="cpu", pin=True)
        return dict(case=case, lib=_context(case, None, None), particles=host(p), links=links, out=P)
    state = dict(case=case, lib=_context(case, p, l), step=0)
    if kind != "rebuild":
        state["P"], state["K"] = _readback(n, L, _lp(case))
    return state


# --------------------------------------------------------------------------- one pass

class _DeviceArray:
    """A device array of a context's view, for torch.as_tensor."""

    def __init__(self, ptr, count, typestr):
        self.__cuda_array_interface__ = dict(shape=(count,), typestr=typestr, data=(ptr, False), version=3)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "steps":
        lib = state["lib"]
        lib.step(case["steps"])
        return {**lib.get_particles(state["P"]), **lib.get_links(state["K"])}
    if kind == "split":
        lib = state["lib"]
        for _ in range(case["steps"]):
            lib.gridService()
            lib.computePartForce()
            lib.applyForce()
            if lib.breakActive(state["step"]):
                lib.linkUpdate()
            lib.finalizeTs()
            state["step"] += 1
        return {**lib.get_particles(state["P"]), **lib.get_links(state["K"])}
    if kind == "rebuild":
        lib = state["lib"]
        lib.regenerate()
        lib.computePartForce()
        lib.synchronize()
        v = lib.device_view()
        real = "<f4" if case["precision"] == "mixed" else "<f8"
        return dict(force=torch.as_tensor(_DeviceArray(v.force, 6 * v.n, real), device=DEV),
                    order=torch.as_tensor(_DeviceArray(v.input_index, v.n, "<i4"), device=DEV),
                    counts=torch.as_tensor(_DeviceArray(v.counts, v.n, "<i4"), device=DEV))
    if kind == "ensemble":
        state["batch"].step(case["steps"])
        for lib, (p, l) in zip(state["libs"], state["views"]):
            lib.get_particles(p)
            lib.get_links(l)
        return state["out"]
    if kind == "job":
        lib = state["lib"]
        lib.set_timestep(0)
        lib.set_particles(state["particles"])
        lib.set_links(state["links"])
        lib.step(case["steps"])
        return lib.get_particles(state["out"])
    if kind == "predict":
        state["net"].predict_device(state["rows"].data_ptr(), case["rows"], state["out"].data_ptr())
        return state["out"]
    loss = state["net"].train(case["steps"])
    return dict(params=state["net"].get_params(), loss=loss)


# --------------------------------------------------------------------------- its least work

def _lattice_counts(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = 4 * nx * ny * nz
    planes = lambda a, b, c: 2 * (2 * a - 1) * (2 * b - 1) * c  # noqa: E731 (face diagonals of one plane family)
    return n, planes(nx, ny, nz) + planes(nx, nz, ny) + planes(ny, nz, nx)


def _step_work(n, L, lp):
    """One timestep: each particle's record read and written, each link end's history read and
    written with its partner and state, each link's length, the contact list."""
    S = 2 * L
    b = n * (2 * (24 + 10 * lp) + 1) + S * (12 * lp + 5) + L * lp + S * 4
    f = S * 230.0 + S * 40.0 + n * 90.0
    return b, f


def work(case):
    kind = case["kind"]
    if kind in ("predict", "train"):
        k = max(128, -(-case["inputs"] * (1 + 2 * case["bands"]) // 128) * 128)
        weights = 256 * k + 3 * 256 * 256 + 3 * 256
        if kind == "predict":
            return dict(bytes=4.0 * case["rows"] * (case["inputs"] + 3) + 2.0 * weights,
                        flops=2.0 * case["rows"] * weights)
        back = 2.0 * (3 * 256 * 256 + 3 * 256) + 2.0 * weights
        return dict(bytes=case["steps"] * (4.0 * case["batch"] * (case["inputs"] + 3) + 24.0 * weights),
                    flops=case["steps"] * case["batch"] * (2.0 * weights + back))
    lp = 4 if case["precision"] == "mixed" else 8
    if kind == "ensemble":
        total = [0.0, 0.0]
        for c, _ in _block_cases(case, 0):
            n, L = _lattice_counts(c)
            b, f = _step_work(n, L, lp)
            total[0] += case["steps"] * b + n * (24 + 9 * lp) + L * (1 + 12 * lp)
            total[1] += case["steps"] * f
        return dict(bytes=total[0], flops=total[1])
    n, L = _lattice_counts(case)
    b, f = _step_work(n, L, lp)
    if kind == "rebuild":
        # cells and records moved, the contact list written, each link end's data moved
        return dict(bytes=n * (2 * (24 + 10 * lp) + 20) + 2 * L * (14 * lp + 20) + b, flops=f + 2.0 * L * 30)
    out = n * (24 + 9 * lp) + L * (1 + 12 * lp) if kind != "job" else n * (24 + 9 * lp)
    up = n * (24 + 10 * lp + 1) + L * (16 + lp + 1) if kind == "job" else 0
    return dict(bytes=case["steps"] * b + out + up, flops=case["steps"] * f)


# --------------------------------------------------------------------------- in 64 bits

def _forces(P, x, th, d, r, A, B, state, cts, cand):
    """Contact, damping and beam forces on every particle; the link ends' history advances."""
    n = r.numel()
    F = [torch.zeros(n, device=DEV, dtype=torch.float64) for _ in range(6)]
    inv = 1.0 / P["dt"]
    a, b = cand
    dx = [x[q][a] - x[q][b] for q in range(3)]
    dist = torch.sqrt(dx[0] ** 2 + dx[1] ** 2 + dx[2] ** 2)
    rs = r[a] + r[b]
    touch = dist < rs
    a, b, dx, dist, rs = a[touch], b[touch], [v[touch] for v in dx], dist[touch], rs[touch]
    C = torch.sqrt((rs - dist) ** 3) * (P["E"] * P["scale"])
    for q in range(6):
        c = P["damping"] if q < 3 else P["dampingRotation"]
        t = -c * ((d[q][a] - d[q][b]) * inv)
        if q < 3:
            t = t + C * dx[q] / dist
        F[q].index_add_(0, a, t)
        F[q].index_add_(0, b, -t)
    W = P["beamWidth"] * P["scale"]
    W2, W4, E = W * W, W ** 4, P["E"]
    G = E / 2
    on = (state != 0).double()
    for end, (s_, o_) in enumerate(((A, B), (B, A))):
        X, Y, Z = (x[q][s_] - x[q][o_] for q in range(3))
        xy = X * X + Y * Y
        D2 = xy + Z * Z
        iL, iP = 1 / torch.sqrt(D2), 1 / torch.sqrt(xy)
        LI = torch.sqrt(D2)
        T = [X * iL, Y * iL, Z * iL, -Y * iP, X * iP, -(Z * X) * iL * iP, -(Z * Y) * iL * iP, xy * iL * iP]
        local = lambda u, v, w: (T[0] * u + T[1] * v + T[2] * w, T[3] * u + T[4] * v,  # noqa: E731
                                 T[5] * u + T[6] * v + T[7] * w)
        ds, do = [d[q][s_] for q in range(6)], [d[q][o_] for q in range(6)]
        B0, B1, B2 = local(*ds[:3])
        B3, B4, B5 = local(*ds[3:])
        B6, B7, B8 = local(*do[:3])
        B9, B10, B11 = local(*do[3:])
        K0, K1, K5 = E * W2 * iL, E * W4 / LI ** 3, E * W4 / (2 * LI ** 2)
        K2, K3, K4 = G * W4 * iL / 6, E * W4 * iL / 3, E * W4 * iL / 6
        ct = [c[end::2] for c in cts]
        ct[0] += K0 * (B0 - B6)
        ct[1] += K1 * (B1 - B7) + K5 * (B5 + B11)
        ct[2] += K1 * (B2 - B8) - K5 * (B4 + B10)
        ct[3] += K2 * (B3 - B9)
        ct[4] += K5 * (B8 - B2) + K3 * B4 + K4 * B10
        ct[5] += K5 * (B1 - B7) + K3 * B5 + K4 * B11
        back = lambda u, v, w: (T[0] * u + T[3] * v + T[5] * w, T[1] * u + T[4] * v + T[6] * w,  # noqa: E731
                                T[2] * u + T[7] * w)
        turned = back(*ct[:3]) + back(*ct[3:])
        for q in range(6):
            c = P["damping"] if q < 3 else P["dampingRotation"]
            F[q].index_add_(0, s_, (-c * ((ds[q] - do[q]) * inv) - turned[q]) * on)
    return F


def _integrate(P, x, th, d, r, kind, F):
    dt, z = P["dt"], x[2]
    dia = 2 * r
    mass = P["rhoIce"] * dia ** 3
    inertia = mass * dia * dia / 6
    above = z > P["waterLevel"]
    drag = torch.where(above, P["airDrag"], P["waterDrag"]).double()
    zF = F[2] + torch.where(above, -P["g"], (P["rhoWater"] - P["rhoIce"]) / P["rhoIce"] * P["g"]) * mass
    xF = F[0]
    if P["useBed"]:
        near = z + r - P["bedHeight"] < P["bedInteract"]
        drag = torch.where(near, min(P["bedDrag"] * P["bedFriction"], 1e5 * P["scale"] ** 2), drag)
        zF = zF + P["bedStiffness"] * (P["bedHeight"] - (z + r)).clamp_min(0)
    if P["useFrontPressure"]:
        push = ((kind & FRONT) != 0) & (z < P["waterLevel"])
        xF = xF - torch.where(push, P["rhoWater"] * P["g"] * (P["waterLevel"] - z) * dia * dia, 0.0)
    free = torch.ones_like(r)
    if P["useFixed"]:
        free = ((kind & FIXED) == 0).double()
    f = [xF, F[1], zF, F[3], F[4], F[5]]
    D = drag / (2 * dt)
    for q in range(6):
        m = (mass if q < 3 else inertia) / (dt * dt)
        d[q] = (f[q] + m * d[q] - D * d[q]) / (m + D) * free
    for q in range(3):
        x[q] = x[q] + d[q]
        th[q] = th[q] + d[3 + q]


def _break(P, x, th, A, B, state, L0):
    S = torch.sqrt(sum((x[q][A] - x[q][B]) ** 2 for q in range(3)))
    bend = torch.stack([(th[q][A] - th[q][B]).abs() for q in range(3)]).amax(0)
    state[(S - L0) / L0 + P["bendBreak"] * bend >= P["maxLoad"]] = 0


def _state64(case, seed):
    p, l = _inputs(case, seed)
    x, th, d = ([p[f].double() for f in fs] for fs in (POSITION, THETA, DIFF))
    cts = [l[f].double() for f in CT]
    if case["kind"] == "job":  # a fresh job hands over no history
        cts = [torch.zeros_like(c) for c in cts]
    return p, x, th, d, p["radius"].double(), l["globalKeyEndA"], l["globalKeyEndB"], l["state"], l["initialLen"].double(), cts


def _after_steps(case, seed):
    P = _params(case)
    p, x, th, d, r, A, B, state, L0, cts = _state64(case, seed)
    for t in range(case["steps"]):
        F = _forces(P, x, th, d, r, A, B, state, cts, (A, B))
        _integrate(P, x, th, d, r, p["type"], F)
        if t * P["dt"] > P["breakTime"]:
            _break(P, x, th, A, B, state, L0)
    out = dict(zip(POSITION + THETA + DIFF, x + th + d))
    if case["kind"] != "job":
        out.update(zip(CT, cts), state=None)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "train" or case.get("setting") == "fjord":
        return None
    if kind == "predict":
        params, u = _network(case, seed)
        W = [w.double() for w in params]
        outs = []
        for rows in u.double().split(1 << 17):
            X = torch.zeros(rows.shape[0], W[0].shape[1], device=DEV, dtype=torch.float64)
            nin = case["inputs"]
            X[:, :nin] = rows
            for f in range(case["bands"]):
                a = 2.0 ** f * math.pi * rows
                X[:, nin * (1 + 2 * f):nin * (3 + 2 * f)] = torch.stack([torch.sin(a), torch.cos(a)], 2).flatten(1)
            for q in range(4):
                X = torch.nn.functional.silu(X @ W[2 * q].T + W[2 * q + 1])
            outs.append(X @ W[8].T + W[9])
        return torch.cat(outs)
    if kind == "ensemble":
        parts = [_after_steps(c, s) for c, s in _block_cases(case, seed)]
        return {f: None if parts[0][f] is None else torch.cat([q[f] for q in parts]) for f in parts[0]}
    if kind == "rebuild":
        P = _params(case)
        p, x, th, d, r, A, B, state, L0, cts = _state64(case, seed)
        F = _forces(P, x, th, d, r, A, B, state, cts, (A, B))
        h = P["searchDistanceScale"] * 2 * P["maxRadius"]
        if case["precision"] == "mixed":  # the particle diameter is a 32-bit number there, 1.0
            h = P["searchDistanceScale"] * float(np.float32(P["maxRadius"]) * np.float32(2))
        cell = [torch.floor((x[q] - x[q].min()) / h).long() for q in range(3)]
        dim = [int(c.max()) + 1 for c in cell]
        order = torch.sort(cell[0] + dim[0] * (cell[1] + dim[1] * cell[2]), stable=True).indices
        return dict(force=torch.cat([f[order] for f in F]), order=None, counts=None)
    return _after_steps(case, seed)
