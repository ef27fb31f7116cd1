"""The work measured: calls of the public API on synthetic scenes.

Every case is one call pattern of a program that uses the library: a block of
time steps of a scene whose state stays on the GPU, a batch of specimens, one
gradient, one step through the per-stage functions, or a block of steps with
its output rows and a frame.  Scenes are seeded: jittered lattices whose
overlaps are pushed apart until neighbours just touch, with small random
velocities and spins, at the sizes of the repository's benchmark and tests
(settling pile of 4,096 disks, 65,536 to 4,194,304 disks "plain at scale",
specimens of 256 to 8,192 disks, the 16,384-disk incline).
"""
import math

import numpy as np
import torch

import demso_b200 as D
from demso_b200 import scenes
from demso_b200.output import render_params

RMEAN, RMAX = 1.0e-3, 1.1e-3


def listed():
    return [
        # the settling pile, stepped as one cluster launch per call
        dict(name="pile_cluster_4k", kind="step", n=4096, phi=0.75, vel=0.05, mats=1,
             attract=0.0, radii="uniform", steps=100, resident=True, accel=False),
        # a mid-size scene on the general path, where latency counts
        dict(name="plain_65k", kind="step", n=65536, phi=0.55, vel=0.05, mats=1, attract=0.0,
             radii="lognormal", steps=50, resident=False, accel=False),
        # a dense flowing packing of ragged size, acceleration kept for output
        dict(name="dense_1m", kind="step", n=1000003, phi=0.80, vel=0.1, mats=1, attract=0.0,
             radii="uniform", steps=20, resident=False, accel=True),
        # the headline size
        dict(name="plain_4m", kind="step", n=4194304, phi=0.55, vel=0.05, mats=1, attract=0.0,
             radii="lognormal", steps=20, resident=False, accel=False),
        # three cohesive materials
        dict(name="cohesive_250k", kind="step", n=250007, phi=0.78, vel=0.1, mats=3, attract=20.0,
             radii="uniform", steps=20, resident=False, accel=False),
        # a fast dilute gas: many disks change cell on every step
        dict(name="gas_131k", kind="step", n=131071, phi=0.30, vel=3.0, mats=2, attract=0.0,
             radii="uniform", steps=20, resident=False, accel=False),
        # the reference's control particle ploughing through a packing
        dict(name="control_200k", kind="control", n=200000, phi=0.78, vel=0.05, mats=1,
             radii="uniform", steps=20),
        # many small specimens as bins in shared memory, one launch per call
        dict(name="batch_resident_512", kind="batch", specimens=512, nmin=256, nmax=8192, mats=1,
             phi=0.5, vel=0.1, steps=20, resident=True),
        # two-material specimens stepped together on the general path
        dict(name="batch_two_materials_256", kind="batch", specimens=256, nmin=256, nmax=8192,
             mats=2, phi=0.6, vel=0.1, steps=20, resident=False),
        # one gradient of a differentiable scene: forward with checkpoints, backward
        dict(name="gradient_16k", kind="adjoint", n=16384, phi=0.72, vel=0.05, steps=100,
             every=50),
        # one step through the reference's five stage functions on the caller's buffers
        dict(name="stages_1m", kind="stages", n=1048576, phi=0.78, vel=0.1, mats=1),
        # the headless runner: steps with followed rows, then a frame
        dict(name="output_262k", kind="output", n=262144, phi=0.75, vel=0.05, mats=2, steps=20,
             follow=64, height=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "control", "batch", "adjoint", "stages", "output"])
    if kind == "step":
        resident = rng.random() < 0.25
        mats = 1 if resident else rng.choice([1, 1, 2, 3])
        attract = 0.0 if resident else rng.choice([0.0, 0.0, 20.0])
        n = _log(rng, 500, 8000) if resident else _log(rng, 3000, 500000 if attract else 2000000)
        return dict(kind="step", n=n, phi=round(rng.uniform(0.3, 0.8), 3),
                    vel=round(rng.uniform(0.02, 1.0), 3), mats=mats, attract=attract,
                    radii=rng.choice(["uniform", "lognormal"]), steps=rng.randint(10, 30),
                    resident=resident, accel=rng.random() < 0.3)
    if kind == "control":
        return dict(kind="control", n=_log(rng, 5000, 1000000), phi=round(rng.uniform(0.5, 0.8), 3),
                    vel=0.05, mats=rng.choice([1, 2]), radii="uniform", steps=rng.randint(5, 30))
    if kind == "batch":
        mats = rng.choice([1, 2])
        return dict(kind="batch", specimens=_log(rng, 16, 600), nmin=256, nmax=8192, mats=mats,
                    phi=round(rng.uniform(0.4, 0.75), 3), vel=0.1, steps=rng.randint(5, 30),
                    resident=mats == 1 and rng.random() < 0.5)
    if kind == "adjoint":
        steps = rng.randint(40, 120)
        return dict(kind="adjoint", n=_log(rng, 1000, 40000), phi=round(rng.uniform(0.6, 0.78), 3),
                    vel=0.05, steps=steps, every=rng.randint(15, 60))
    if kind == "stages":
        return dict(kind="stages", n=_log(rng, 5000, 3000000), phi=round(rng.uniform(0.4, 0.8), 3),
                    vel=0.1, mats=rng.choice([1, 2]))
    return dict(kind="output", n=_log(rng, 4000, 1000000), phi=round(rng.uniform(0.4, 0.8), 3),
                vel=0.05, mats=rng.choice([1, 3]), steps=rng.randint(5, 30),
                follow=rng.randint(1, 200), height=rng.randint(400, 1600))


# -- scenes ------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _materials(mats, attract, e=0.5):
    return [scenes.pair_material(kn=1e5 * (1 + m), mu=0.5 - 0.1 * m, zeta=0.3 + 0.05 * m,
                                 e_boundary=e, attraction=attract * (m + 1)) for m in range(mats)]


def _packing(n, phi, vel, mats, attract, radii, seed):
    """A System and its state on the GPU: n disks on a hexagonal lattice at
    area fraction `phi`, jittered, with overlaps relaxed away."""
    g = _gen(seed)
    cuda = dict(device="cuda", dtype=torch.float64)
    if radii == "lognormal":
        r = RMEAN * torch.exp(0.15 * torch.randn(n, generator=g, **cuda))
        r = r.clamp(0.6e-3, 1.6e-3)
        rmax = 1.6e-3
    else:
        r = 0.9e-3 + 0.2e-3 * torch.rand(n, generator=g, **cuda)
        rmax = RMAX
    r = r.float().double()
    er2 = float((r * r).mean())
    a = math.sqrt(math.pi * er2 / (phi * math.sqrt(3.0) / 2.0))  # lattice pitch
    cols = max(2, int(round(math.sqrt(n * math.sqrt(3.0) / 2.0))))
    rows = -(-n // cols)
    Lx, Ly = (cols + 0.5) * a, (rows + 1.0) * a * math.sqrt(3.0) / 2.0 + 0.3 * a
    k = torch.arange(rows * cols, device="cuda")
    y, x = k // cols, k % cols
    p = torch.stack([(x + 0.5 + 0.5 * (y & 1)) * a, (y + 0.7) * a * math.sqrt(3.0) / 2.0], 1)
    p = p.double()
    free = max(0.0, a - 2.0 * RMEAN)
    p += (torch.rand(p.shape, generator=g, **cuda) - 0.5) * (0.2e-3 + 0.8 * free)
    rr = torch.zeros(rows * cols, **cuda)
    rr[:n] = 0.9995 * r  # neighbours end up pressed together by about a micrometre
    p[n:] = -1.0  # sites without a disk
    p, rr = p.view(rows, cols, 2), rr.view(rows, cols)
    odd = (torch.arange(rows, device="cuda") & 1).view(rows, 1) == 1
    for _ in range(25):
        move = torch.zeros_like(p)
        for dy, dx in ((0, 1), (0, -1), (1, 0), (1, 1), (-1, 0), (-1, 1)):
            if dy:  # the two neighbours above or below: shifted by the row's offset
                ev = torch.roll(p, (-dy, 1 - dx), (0, 1)), torch.roll(rr, (-dy, 1 - dx), (0, 1))
                od = torch.roll(p, (-dy, -dx), (0, 1)), torch.roll(rr, (-dy, -dx), (0, 1))
                q = torch.where(odd[..., None], od[0], ev[0])
                rq = torch.where(odd, od[1], ev[1])
            else:
                q, rq = torch.roll(p, -dx, 1), torch.roll(rr, -dx, 1)
            d = p - q
            dist = d.norm(dim=2).clamp_min(1e-12)
            over = (rr + rq - dist).clamp_min(0.0) * ((rr > 0) & (rq > 0))
            move += d * (0.5 * over / dist)[..., None]
        p = p + 0.8 * move
        p[..., 0] = torch.minimum(torch.maximum(p[..., 0], rr), Lx - rr)
        p[..., 1] = torch.minimum(torch.maximum(p[..., 1], rr), Ly - rr)
    gx, gy = scenes.grid_2r(Lx, rmax), scenes.grid_2r(Ly, rmax)
    ms = _materials(mats, attract)
    sys = D.System(Lx=Lx, Ly=Ly, gx=gx, gy=gy, dt=2e-6, gravity=(0.0, -9.81),
                   knWall=ms[0].normalStiffness, ktWall=ms[0].shearStiffness, materials=ms)
    st = dict(pos=p.view(-1, 2)[:n].float(), radius=r.float())
    return sys, _finish(st, n, vel, mats, g)


def _finish(st, n, vel, mats, g):
    f = dict(device="cuda", dtype=torch.float32, generator=g)
    r = st["radius"].double()
    st["vel"] = torch.randn((n, 2), **f) * vel
    st["theta"] = torch.rand(n, **f) * 6.28
    st["omega"] = torch.randn(n, **f) * 20.0
    st["mass"] = (scenes.RHO * math.pi * r * r * scenes.THICK).float()
    st["id"] = torch.arange(n, dtype=torch.int32, device="cuda")
    st["type"] = (torch.randint(0, mats, (n,), device="cuda", generator=g, dtype=torch.int32)
                  if mats > 1 else None)
    return {k: (v.contiguous() if v is not None else None) for k, v in st.items()}


def _specimens(case, seed):
    """Specimens of log-uniform size, each in its own square box."""
    g = _gen(seed)
    rng = np.random.default_rng(int(seed) + 5)
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    # the sizes are the case's, not the seed's: evenly spread over their logarithm
    num = case["specimens"]
    counts = [int(math.exp(lo + (hi - lo) * (k + 0.5) / num)) for k in range(num)]
    counts = [counts[(k * 7) % num] if math.gcd(7, num) == 1 else counts[k] for k in range(num)]
    specs, pos, rad = [], [], []
    for c in counts:
        r = rng.uniform(0.9e-3, 1.1e-3, c)
        side = int(math.ceil(math.sqrt(c)))
        pitch = math.sqrt(math.pi * 1.0033e-6 / case["phi"])
        ij = np.stack([np.arange(c) % side, np.arange(c) // side], 1)
        jit = 0.4 * max(0.0, pitch - 2 * RMEAN)
        pos.append((ij + 0.5) * pitch + rng.uniform(-jit, jit, (c, 2)))
        rad.append(r)
        L = side * pitch
        k = float(np.exp(rng.uniform(np.log(5e4), np.log(5e5))))
        ms = [scenes.pair_material(kn=k * (1 + m), mu=float(rng.uniform(0.2, 0.8)),
                                   zeta=float(rng.uniform(0.1, 0.5))) for m in range(case["mats"])]
        gr = scenes.grid_2r(L, RMAX)
        specs.append((D.System(Lx=L, Ly=L, gx=gr, gy=gr, dt=2e-6, gravity=(0.0, -9.81),
                               knWall=ms[0].normalStiffness, ktWall=ms[0].shearStiffness,
                               materials=ms), c))
    up = lambda a: torch.from_numpy(np.concatenate(a).astype(np.float32)).cuda()
    st = dict(pos=up(pos), radius=up(rad))
    return specs, _finish(st, sum(counts), case["vel"], case["mats"], g)


def _control(sys, rc=0.03):
    """A large disk just above the packing's top row, pressed into it."""
    return dict(pos=(0.25 * sys.Lx, sys.Ly + rc - 3.2e-3), radius=rc, material=0,
                drift=(0.0, -2e-5))


def _load(sim, st):
    sim.set_state(st["pos"], st["vel"], st["theta"], st["omega"], st["radius"], st["mass"],
                  st["id"], st["type"])


def _scene(case, seed):
    return _packing(case["n"], case["phi"], case["vel"], case.get("mats", 1),
                    case.get("attract", 0.0), case.get("radii", "uniform"), seed)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        specs, st = _specimens(case, seed)
        sim = D.Batch(specs, flags=D.CTX_PRESSURE | (D.CTX_RESIDENT if case["resident"] else 0))
        _load(sim, st)
        return dict(case=case, sim=sim)
    sys, st = _scene(case, seed)
    n = case["n"]
    if kind == "stages":
        z = lambda *s: torch.zeros(s, device="cuda", dtype=torch.float32)
        zi = lambda *s: torch.zeros(s, device="cuda", dtype=torch.int32)
        other = {k: (torch.zeros_like(v) if v is not None else None) for k, v in st.items()}
        return dict(case=case, sys=sys, a=st, b=other, loc=zi(n), hash=zi(n), index=zi(n),
                    start=zi(sys.num_cells), end=zi(sys.num_cells), acc=z(n, 2), alpha=z(n),
                    pressure=z(n),
                    scratch=torch.empty(D.sort_scratch_bytes(n, sys.key_bits), dtype=torch.uint8,
                                        device="cuda"))
    flags = D.CTX_PRESSURE
    if case.get("resident"):
        flags |= D.CTX_RESIDENT
    if case.get("accel") or kind in ("adjoint", "output"):
        flags |= D.CTX_ACCEL
    sim = D.Simulation(sys, capacity=n, flags=flags)
    _load(sim, st)
    state = dict(case=case, sim=sim)
    if kind == "control":
        sim.set_control(**_control(sys))
    if kind == "adjoint":
        state["init"] = st
        state["lam"] = [torch.empty((n, 2), device="cuda"), torch.empty((n, 2), device="cuda"),
                        torch.empty(n, device="cuda")]
    if kind == "output":
        state["ids"] = np.linspace(0, n - 1, case["follow"]).astype(np.uint32)
        state["rows"] = torch.empty((case["steps"], case["follow"], 12), dtype=torch.float32,
                                    pin_memory=True)
        state["params"] = render_params(sys.Lx, sys.Ly, [(255.0, 80.0 * (m + 1), 40.0)
                                                         for m in range(case["mats"])],
                                        case["height"])
        state["image"] = torch.empty((state["params"].imageDIMy, state["params"].imageDIMx, 4),
                                     dtype=torch.uint8, device="cuda")
    return state


_FIELDS = ("pos", "vel", "theta", "omega", "radius", "mass", "id", "type")


def _state(sim):
    """The state a program reads back: the fields the context's flags keep."""
    got = sim.get_state()
    keep = _FIELDS + ("loc",)
    if sim.flags & D.CTX_PRESSURE:
        keep += ("pressure",)
    if sim.flags & D.CTX_ACCEL:
        keep += ("acc", "alpha")
    return {k: got[k] for k in keep if got[k] is not None}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("step", "batch"):
        sim = state["sim"]
        sim.step(case["steps"])
        return _state(sim)
    if kind == "control":
        sim = state["sim"]
        sim.step(case["steps"])
        pos, reaction = sim.control()
        return dict(_state(sim), control=list(pos), reaction=list(reaction))
    if kind == "adjoint":
        sim, st, lam = state["sim"], state["init"], state["lam"]
        _load(sim, st)
        sim.adjoint_forward(case["steps"], case["every"])
        v = sim.state_view()
        ids = v["id"].long()
        # loss: squared distance of the final positions from the first ones, and kinetic energy
        lam[0].zero_()
        lam[0][ids] = 2e6 * (v["pos"] - st["pos"][ids])
        lam[1][ids] = v["mass"][:, None] * v["vel"] * 1e3
        lam[2].zero_()
        grad = sim.adjoint_backward(*lam)
        return dict(lam_pos=lam[0], lam_vel=lam[1], lam_omega=lam[2], grad=grad)
    if kind == "stages":
        s, n, sys, a, b = state, case["n"], state["sys"], state["a"], state["b"]
        D.calcHash(sys, a["pos"], s["index"], s["hash"], n)
        D.sortParticles(s["hash"], s["index"], n, sys.key_bits, s["scratch"])
        D.reorderDataAndFindCellStart(
            sys, s["start"], s["end"], b["pos"], b["vel"], b["theta"], b["omega"], b["radius"],
            b["mass"], b["id"], s["loc"], b["type"], s["hash"], s["index"], a["pos"], a["vel"],
            a["theta"], a["omega"], a["radius"], a["mass"], a["id"], a["type"], n, sys.num_cells)
        D.collide(sys, b["pos"], b["vel"], s["acc"], b["omega"], s["alpha"], b["type"],
                  b["radius"], b["mass"], s["start"], s["end"], n, sys.num_cells, s["pressure"])
        D.integrateSystem(sys, b["pos"], b["vel"], s["acc"], b["theta"], b["omega"], s["alpha"],
                          b["type"], b["radius"], b["mass"], s["pressure"], n)
        state["a"], state["b"] = b, a
        out = {k: b[k] for k in _FIELDS if b[k] is not None}
        return dict(out, acc=s["acc"], alpha=s["alpha"], pressure=s["pressure"], loc=s["loc"],
                    hash=s["hash"], index=s["index"], start=s["start"], end=s["end"])
    sim = state["sim"]
    sim.step_followed(case["steps"], state["ids"], state["rows"])
    sim.render(state["params"], state["image"])
    torch.cuda.current_stream().synchronize()  # the rows are written out on the host
    return dict(_state(sim), rows=state["rows"], image=state["image"])


def _count(case):
    if case["kind"] != "batch":
        return case["n"]
    num, lo, hi = case["specimens"], math.log(case["nmin"]), math.log(case["nmax"])
    return sum(int(math.exp(lo + (hi - lo) * (k + 0.5) / num)) for k in range(num))


def work(case):
    """Per disk and step: position, velocity, angle and spin in and out
    (48 B), radius and mass in (8 B), the type where there is one; about 150
    operations (candidate tests, one or two contacts, integration)."""
    n, kind = _count(case), case["kind"]
    per = 56.0 + (4.0 if case.get("mats", 1) > 1 else 0.0)
    if kind == "stages":  # the sorted copy, its cells, accelerations and the new state
        return dict(bytes=n * (36.0 + 56.0 + 16.0 + 48.0), flops=n * 150.0)
    steps = case["steps"]
    if kind == "adjoint":  # forward, forward again while recording, and the reverse
        return dict(bytes=n * steps * (2 * per + 64.0 + 40.0), flops=n * steps * 900.0)
    b, f = n * steps * per, n * steps * 150.0
    if kind == "output":
        b += 48.0 * case["follow"] * steps + 4.0 * case["height"] ** 2
    return dict(bytes=b, flops=f)


# -- the same in 64 bits -----------------------------------------------------
def exact(case, seed):
    """One step in float64 for the stage functions.  The other cases run tens
    of steps: a contact force is a large stiffness times a difference of
    nearly equal numbers, so the rounding of float32 positions moves their
    forces by tens of per cent within a few steps, and 64-bit values of those
    trajectories (and of the gradient, whose branches are the float
    trajectory's own) say nothing about them."""
    if case["kind"] != "stages":
        return None
    sys, st = _scene(case, seed)
    n, K = case["n"], len(sys.materials)
    f32 = lambda x: float(np.float32(x))
    t64 = lambda a: torch.tensor(a, device="cuda", dtype=torch.float64)
    # sorted by cell, which is defined in float32
    p = st["pos"]
    Lx, Ly = f32(sys.Lx), f32(sys.Ly)
    cx = torch.floor(p[:, 0] * sys.gx / torch.tensor(Lx, device="cuda")).long() & (sys.gx - 1)
    cy = torch.floor(p[:, 1] * sys.gy / torch.tensor(Ly, device="cuda")).long() & (sys.gy - 1)
    order = torch.argsort(cy * sys.gx + cx, stable=True)
    cx, cy = cx[order], cy[order]
    p, v, th, w, r, m = (st[k][order].double() for k in
                         ("pos", "vel", "theta", "omega", "radius", "mass"))
    t = st["type"][order].long() if st["type"] is not None else torch.zeros(n, device="cuda").long()
    mat = {k: t64([f32(getattr(q, k)) for q in sys.materials]) for k in
           ("normalStiffness", "shearStiffness", "normalDamping", "frictionCoefficient",
            "boundaryDamping")}
    ser = lambda a, b: a * b / (a + b)
    pair = lambda a: ser(a[:, None], a[None, :])
    kn, kt, cn = (pair(mat[k]) for k in ("normalStiffness", "shearStiffness", "normalDamping"))
    mu = (mat["frictionCoefficient"][:, None] + mat["frictionCoefficient"][None, :]) / 2.0
    dt, g = f32(sys.dt), t64([f32(x) for x in sys.gravity])
    I = 2.0 * m * r * r / 5.0
    # every disk against the disks of its 3 x 3 cells
    key = cy * sys.gx + cx
    count = torch.bincount(key, minlength=sys.num_cells)
    first = torch.cumsum(count, 0) - count
    me = torch.arange(n, device="cuda")
    F, M, pr = torch.zeros_like(p), torch.zeros_like(r), torch.zeros_like(r)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            h = ((cy + dy) & (sys.gy - 1)) * sys.gx + ((cx + dx) & (sys.gx - 1))
            for k in range(int(count[h].max())):
                i = me[count[h] > k]
                j = first[h[i]] + k
                near = ((p[j] - p[i]).norm(dim=1) < r[i] + r[j]) & (i != j)
                i, j = i[near], j[near]
                q = (t[i], t[j])
                rel = p[j] - p[i]
                dist = rel.norm(dim=1)
                nx = rel / dist[:, None]
                tx = torch.stack([-nx[:, 1], nx[:, 0]], 1)
                rv = v[j] - v[i]
                vn = (rv * nx).sum(1)
                vt = rv - vn[:, None] * nx
                fn = -kn[q] * (r[i] + r[j] - dist) + torch.where(vn < 0, cn[q] * vn, 0.0)
                vc = vt - (r[i] * w[i] + r[j] * w[j])[:, None] * tx
                ft, lim = kt[q][:, None] * vc * dt, mu[q] * fn.abs()
                slip = ft.norm(dim=1) >= lim
                ft = torch.where(slip[:, None], lim[:, None] * vc / vc.norm(dim=1)[:, None], ft)
                ft = torch.where((mu[q] != 0)[:, None], ft, 0.0)
                F.index_add_(0, i, fn[:, None] * nx + ft)
                M.index_add_(0, i, r[i] * (ft * tx).sum(1))
                pr.index_add_(0, i, fn.abs())
    acc, alpha = F / m[:, None], M / I
    v = v + (g + acc) * dt
    p = p + v * dt
    w = w + alpha * dt
    th = th + w * dt
    turn = 2 * math.pi
    th = torch.where((th > turn) | (th < 0), th - turn * torch.floor(th / turn), th)
    eb = mat["boundaryDamping"][t]
    for axis, L, sides in ((0, Lx, 2), (1, Ly, 1)):  # side walls, top
        out = p[:, axis] > L - r
        p[:, axis] = torch.where(out, L - r, p[:, axis])
        v[:, axis] = torch.where(out, -eb * v[:, axis], v[:, axis])
        if sides == 2:
            out = p[:, axis] < r
            p[:, axis] = torch.where(out, r, p[:, axis])
            v[:, axis] = torch.where(out, -eb * v[:, axis], v[:, axis])
    low = p[:, 1] < r  # the floor: normal (0, -1), tangent (1, 0)
    ktw = ser(mat["shearStiffness"], f32(sys.ktWall))[t]
    fn = torch.stack([-m * g[0], -m * g[1] - torch.where(
        v[:, 1] < 0, mat["normalDamping"][t] * v[:, 1], 0.0)], 1).norm(dim=1)
    vc = -v[:, 0] - r * w
    ft, lim = ktw * vc * dt, mat["frictionCoefficient"][t] * fn
    ft = torch.where(ft.abs() >= lim, lim * torch.sign(vc), ft)
    aw, wa = torch.where(low, ft / m, 0.0), torch.where(low, r * ft / I, 0.0)
    v[:, 0] += aw * dt
    p[:, 0] += aw * dt * dt
    w, th = w + wa * dt, th + wa * dt * dt
    v[:, 1] = torch.where(low, -eb * v[:, 1], v[:, 1])
    p[:, 1] = torch.where(low, r, p[:, 1])
    pr = (pr + torch.where(low, fn, 0.0)) / (4 * math.pi * r * r)
    out = dict(pos=p, vel=v, theta=th, omega=w, radius=r, mass=m, id=None, acc=acc, alpha=alpha,
               pressure=pr, loc=None, hash=None, index=None, start=None, end=None)
    return dict(out, type=None) if K > 1 else out
