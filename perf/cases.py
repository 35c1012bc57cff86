"""What a program does with this framework, as cases that can be timed and compared.

A pass is what such a program does once per frame, control interval or
rollout: (a reset,) step(n), and the state read back through the public
Python API (titan_gb300.Sim).  A case is a dict of plain values:

    kind     "scene"    one scene, stepped on and read each pass
             "rollout"  one scene, set to a request's initial state and spring
                        parameters, stepped and read each pass (how a pooled
                        engine is used again for the next request)
             "requests" several scenes of uneven sizes, each on its own
                        handle and stream, all in flight at once
    prec     "f64" | "f32" | "f32c"        integ  "euler" | "verlet" | "rk2"
    nx ny nz masses per axis of a lattice (26-neighbourhood springs); or
    bodies, side_lo, side_hi: independent bodies with a ground plane each; or
    bodies = requests with mass counts between mass_lo and mass_hi
    steps    steps of one pass              drop, act  share of the springs
             removed / actuated             damping    spring damping
    extras   fixed masses at one end, external forces and drag
    contact  start at the ground plane (else above it)
    read     "state"   get_state() into new arrays
             "pinned"  get_state() into page-locked arrays kept by the caller
             "device"  export_vertices() into a float32 CUDA tensor, and
                       get_state() of the velocities
    energy   the energies and momenta of diagnostics() are read too
"""
import math

import numpy as np
import torch

TWO_PI = 2.0 * math.pi
G = (0.0, 0.0, -9.81)


def _case(name, kind="scene", prec="f64", integ="euler", nx=0, ny=0, nz=0, bodies=0, side_lo=0, side_hi=0, mass_lo=0,
          mass_hi=0, steps=100, drop=0.0, act=0.0, damping=0.1, extras=False, contact=True, ball=False, dt=1e-4,
          read="state", energy=False):
    c = {k: v for k, v in locals().items() if k != "name"}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the reference's robot (5^3 masses on a frictional plane, the drop-in
        # precision) in a control loop that reads the state every millisecond
        _case("cube5_f64_10", prec="f64", nx=5, ny=5, nz=5, steps=10, damping=0.0),
        # the same robot in the fast precision, one frame of 100 steps a read
        _case("cube5_f32c_100", prec="f32c", nx=5, ny=5, nz=5, steps=100, damping=0.0),
        # one soft robot of a design study in the drop-in precision: a pooled
        # engine takes the next parameters, rolls out and is read
        _case("rollout9_f64", kind="rollout", prec="f64", nx=9, ny=9, nz=9, steps=200, drop=0.05, act=0.3),
        # the same for a larger design in the fast precision (many tiles)
        _case("rollout23_f32c", kind="rollout", prec="f32c", nx=23, ny=23, nz=23, steps=200, drop=0.05, act=0.3),
        # a cantilever of odd extents: one end fixed, loads, drag, a ball
        _case("beam_f64", prec="f64", nx=61, ny=11, nz=7, steps=50, extras=True, contact=False, ball=True),
        # the higher-order integrators at a middling size
        _case("block_rk2_f64", prec="f64", integ="rk2", nx=24, ny=19, nz=27, steps=20, act=0.2),
        _case("block_verlet_f32c", prec="f32c", integ="verlet", nx=38, ny=41, nz=33, steps=100, act=0.2, read="pinned"),
        # populations of small bodies of uneven sizes: training in the fast
        # precision with the positions left on the GPU, checks in FP64
        _case("bodies1024_f32c", prec="f32c", bodies=1024, side_lo=3, side_hi=12, steps=50, drop=0.05, act=0.3,
              read="device"),
        _case("bodies96_f64", prec="f64", bodies=96, side_lo=3, side_hi=9, steps=50, drop=0.05, act=0.3),
        # rollout requests of very uneven sizes in flight together
        _case("requests24_f32c", kind="requests", prec="f32c", bodies=24, mass_lo=27, mass_hi=60000, steps=200, drop=0.05,
              act=0.3),
        # one large lattice: the drop-in precision with its energies, and the
        # fast precision at a million masses
        _case("lattice70_f64", prec="f64", nx=70, ny=70, nz=70, steps=10, act=0.2, ball=True, read="pinned", energy=True),
        _case("lattice100_f32c", prec="f32c", nx=100, ny=100, nz=100, steps=100, act=0.2, ball=True, read="pinned"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["scene", "scene", "scene", "rollout", "bodies", "requests"])
    prec = rng.choice(["f64", "f64", "f32c", "f32c", "f32"])
    cap = 90e6 if prec != "f64" else 3.5e6  # mass-steps of a pass
    damping = rng.choice([0.0, 0.1, 0.1])
    act, drop = rng.choice([0.0, 0.2, 0.3]), rng.choice([0.0, 0.05])
    if kind == "requests":
        n = rng.randint(4, 24)
        hi = int(_log(rng, 2000, 60000 if prec != "f64" else 10000))
        return _case(None, kind="requests", prec=prec, bodies=n, mass_lo=27, mass_hi=hi,
                     steps=max(10, int(min(300, cap / (n * hi / 4)))), drop=0.05, act=act)
    if kind == "bodies":
        n = int(_log(rng, 8, 1024 if prec != "f64" else 256))
        lo = rng.randint(3, 6)
        hi = rng.randint(lo, 12 if prec != "f64" else 9)
        steps = int(_log(rng, 5, 100))
        return _case(None, prec=prec, bodies=n, side_lo=lo, side_hi=hi, steps=max(2, min(steps, int(cap / (n * hi ** 3)))),
                     drop=drop, act=act, damping=damping, read=rng.choice(["state", "pinned", "device"]))
    n = _log(rng, 27, 700000 if prec != "f64" else 300000)
    if kind == "rollout":
        n = min(n, 60000)
    # sides of uneven extents around the cube root
    a, b = _log(rng, 0.5, 2.0), _log(rng, 0.5, 2.0)
    s = n ** (1.0 / 3.0)
    nx, ny = max(2, round(s * a)), max(2, round(s * b))
    nz = max(2, round(n / (nx * ny)))
    steps = max(2, min(int(_log(rng, 5, 400)), int(cap / (nx * ny * nz))))
    integ = rng.choice(["euler", "euler", "euler", "verlet", "rk2"]) if kind == "scene" else "euler"
    if integ == "rk2":
        steps = max(1, steps // 2)
    return _case(None, kind=kind, prec=prec, integ=integ, nx=nx, ny=ny, nz=nz, steps=steps, drop=drop, act=act, damping=damping,
                 extras=kind == "scene" and rng.random() < 0.2, contact=rng.random() < 0.7, ball=rng.random() < 0.3,
                 read=rng.choice(["state", "pinned", "device"]) if kind == "scene" else "state",
                 energy=kind == "scene" and rng.random() < 0.2)


# ------------------------------------------------------------------ inputs --
_FORWARD = [(di, dj, dk) for di in (-1, 0, 1) for dj in (-1, 0, 1) for dk in (-1, 0, 1) if (di, dj, dk) > (0, 0, 0)]


def _lattice(nx, ny, nz, spacing, bottom):
    """A lattice's masses in (i, j, k) order and its springs in the order of their left ends."""
    i, j, k = (a.reshape(-1) for a in np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"))
    pos = np.stack([(i - (nx - 1) / 2) * spacing, (j - (ny - 1) / 2) * spacing, bottom + k * spacing], 1)
    n = nx * ny * nz
    other = np.full((n, len(_FORWARD)), -1, np.int32)
    here = np.arange(n)
    for q, (di, dj, dk) in enumerate(_FORWARD):
        ok = (i + di < nx) & (0 <= j + dj) & (j + dj < ny) & (0 <= k + dk) & (k + dk < nz)
        other[:, q] = np.where(ok, here + (di * ny + dj) * nz + dk, -1)
    left = np.repeat(here.astype(np.int32), len(_FORWARD)).reshape(n, -1)[other >= 0]
    return pos, left, other[other >= 0]


def _springs(sc, design, rng, c):
    """Stiffness, damping and actuation of the springs that stay (which ones do, and which are actuated, is the design's)."""
    if c["drop"]:
        stay = design.random(sc["left"].size) >= c["drop"]
        sc["left"], sc["right"] = sc["left"][stay], sc["right"][stay]
    ns = sc["left"].size
    d = sc["pos"][sc["left"]] - sc["pos"][sc["right"]]
    sc["rest"] = np.sqrt((d * d).sum(1))
    sc["damping"] = np.full(ns, c["damping"])
    sc["type"] = np.zeros(ns, np.int32)
    if c["act"]:
        on = design.random(ns) < c["act"]
        sc["type"][on] = design.integers(2, 4, int(on.sum()))
    _parameters(sc, rng)


def _parameters(sc, rng):
    """One request's spring constants, actuation and velocities on a design."""
    ns, on = sc["left"].size, sc["type"] >= 2
    sc["k"] = np.exp(rng.uniform(math.log(1e3), math.log(1e5), ns))
    sc["amp"] = np.where(on, 0.1, 0.2)
    sc["phase"] = np.where(on, rng.uniform(0.0, TWO_PI, ns), 0.0)
    sc["omega"] = np.where(on, TWO_PI / rng.uniform(0.1, 1.0, ns), 0.0)
    sc["vel"] = rng.normal(scale=0.01, size=sc["pos"].shape)
    sc["vel"][:, 2] -= 0.05


def _one(c, design, rng, nx, ny, nz):
    """One lattice scene."""
    spacing = 0.1 if max(nx, ny, nz) < 30 else 0.05
    pos, left, right = _lattice(nx, ny, nz, spacing, 0.0005 if c["contact"] else 0.3)
    sc = {"pos": pos, "left": left, "right": right, "m": np.full(len(pos), 0.1), "planes": [((0.0, 0.0, 1.0), 0.0, 0.5, 0.5)],
          "balls": [((0.0, 0.0, -2.5), 2.0)] if c["ball"] else []}
    if c["extras"]:
        n = len(pos)
        end = pos[:, 0] == pos[:, 0].min()
        sc["fixed"] = end.astype(np.uint8)
        sc["ext"] = np.where(rng.random(n)[:, None] < 0.1, rng.normal(scale=0.5, size=(n, 3)), 0.0)
        sc["drag"] = np.where(rng.random(n) < 0.1, 1.0, 0.0)
    _springs(sc, design, rng, c)
    return sc


def _population(c, design, rng):
    """Independent bodies on a grid, each with its own ground plane."""
    pos, left, right, ptr, planes = [], [], [], [0], []
    sides = design.integers(c["side_lo"], c["side_hi"] + 1, c["bodies"])
    made = {int(s): _lattice(int(s), int(s), int(s), 0.1, 0.0005 if c["contact"] else 0.3) for s in set(sides.tolist())}
    grid = int(math.ceil(math.sqrt(c["bodies"])))
    for b, s in enumerate(sides.tolist()):
        p, le, ri = made[s]
        pos.append(p + np.array([(b % grid) * 2.0, (b // grid) * 2.0, 0.0]))
        left.append(le + ptr[-1])
        right.append(ri + ptr[-1])
        ptr.append(ptr[-1] + len(p))
        mu = float(rng.uniform(0.3, 0.8))
        planes.append(((0.0, 0.0, 1.0), 0.0, mu, mu))
    sc = {"pos": np.concatenate(pos), "left": np.concatenate(left).astype(np.int32),
          "right": np.concatenate(right).astype(np.int32), "m": np.full(ptr[-1], 0.1), "planes": [], "balls": [],
          "body_ptr": np.array(ptr, np.int64), "body_planes": planes}
    _springs(sc, design, rng, c)
    return sc


def _scenes(c, seed):
    # sizes and topology are the case's, values are the seed's
    design, rng = np.random.default_rng(c["steps"]), np.random.default_rng([int(seed), c["steps"]])
    if c["kind"] == "requests":
        n = np.exp(design.uniform(math.log(c["mass_lo"]), math.log(c["mass_hi"]), c["bodies"]))
        n[:2] = c["mass_lo"], c["mass_hi"]
        return [_one(c, design, rng, s, s, s) for s in np.maximum(2, np.round(np.cbrt(n))).astype(int).tolist()]
    if c["bodies"]:
        return [_population(c, design, rng)]
    sc = _one(c, design, rng, c["nx"], c["ny"], c["nz"])
    if c["kind"] == "rollout":  # the next request on the design: other parameters
        sc = dict(sc, first={k: sc[k] for k in ("k", "phase", "omega", "vel")})
        _parameters(sc, rng)
    return [sc]


def _masses_springs(c):
    """Masses and springs of a case (of the expected sizes, where they are drawn)."""
    def lattice(x, y, z):
        pairs = sum((x - abs(a)) * (y - abs(b)) * (z - abs(d)) for a, b, d in _FORWARD)
        return np.array([x * y * z, pairs * (1.0 - c["drop"])])
    if c["kind"] == "requests":
        lo, hi = math.log(c["mass_lo"]), math.log(c["mass_hi"])
        at = [max(2, round(math.exp(lo + (hi - lo) * (q + 0.5) / c["bodies"]) ** (1 / 3))) for q in range(c["bodies"])]
        return sum(lattice(s, s, s) for s in at)
    if c["bodies"]:
        sides = range(c["side_lo"], c["side_hi"] + 1)
        return sum(lattice(s, s, s) for s in sides) * (c["bodies"] / len(sides))
    return lattice(c["nx"], c["ny"], c["nz"])


def work(c):
    n, ns = _masses_springs(c)
    real = 8 if c["prec"] == "f64" else 4
    record = {"f64": 48, "f32": 32, "f32c": 48}[c["prec"]]
    # per step: every mass's state read and written, its mass and flags; every
    # spring's constants and ends, an actuated one's amplitude and phase
    once = n * (2 * record + real + 1) + ns * (3 * real + 8) + c["act"] * ns * 2 * real
    passes = c["steps"] * (2 if c["integ"] == "rk2" else 1)
    # what is larger than the L2 comes from memory again in every step
    moved = once * (passes if once > 126e6 else 1) + n * 48
    if c["kind"] == "rollout":
        moved += n * 48 + ns * 3 * 8
    flops = passes * (ns * (29 + (17 if c["damping"] else 0) + 20 * c["act"]) + n * 60 + 6 * ns)
    return {"bytes": float(moved), "flops": float(flops)}


# ------------------------------------------------------------------- a pass --
def prepare(case, seed):
    import titan_gb300 as tg

    c = dict(case)
    sims, scenes = [], _scenes(c, seed)
    prec = {"f64": tg.FP64, "f32": tg.FP32, "f32c": tg.FP32C}[c["prec"]]
    for sc in scenes:
        sim = tg.Sim(prec)
        sim.set_time_step(c["dt"])
        sim.set_global_acc(G)
        if c["integ"] != "euler":
            sim.set_integrator({"verlet": tg.VERLET, "rk2": tg.RK2}[c["integ"]])
        sim.set_masses(sc["pos"], sc["m"], vel=sc.get("first", sc)["vel"], ext=sc.get("ext"), fixed=sc.get("fixed"),
                       drag=sc.get("drag"))
        f = sc.get("first", sc)
        sim.set_springs(sc["left"], sc["right"], f["k"], sc["rest"], damping=sc["damping"], type=sc["type"],
                        omega=f["omega"], amp=sc["amp"], phase=f["phase"])
        for n, off, fk, fs in sc["planes"]:
            sim.add_plane(n, off, fk, fs)
        for at, r in sc["balls"]:
            sim.add_ball(at, r)
        if "body_ptr" in sc:
            sim.set_bodies(sc["body_ptr"])
            for b, (n, off, fk, fs) in enumerate(sc["body_planes"]):
                sim.set_body_plane(b, n, off, fk, fs)
        sim.start()
        sims.append(sim)
    st = {"case": c, "sims": sims, "scenes": scenes}
    n = len(scenes[0]["pos"])
    if c["read"] == "pinned":
        st["out"] = {k: tg.pinned_empty((n, 3)) for k in ("pos", "vel")}
    if c["read"] == "device":
        st["vertices"] = torch.empty((n, 3), dtype=torch.float32, device="cuda")
    return st


def run(st):
    c, sims = st["case"], st["sims"]
    if c["kind"] == "requests":
        for sim in sims:
            sim.step(c["steps"])
        got = [sim.get_state() for sim in sims]
        return [[g["pos"], g["vel"]] for g in got]
    sim = sims[0]
    if c["kind"] == "rollout":
        sc = st["scenes"][0]
        sim.set_mass_state(None, pos=sc["pos"], vel=sc["vel"])
        sim.set_spring_params(None, k=sc["k"], omega=sc["omega"], phase=sc["phase"])
        sim.set_time(0.0)
    sim.step(c["steps"])
    if c["read"] == "device":
        sim.export_vertices(device_ptr=st["vertices"].data_ptr())
        got = [st["vertices"], sim.get_state(pos=False)["vel"]]
    else:
        g = sim.get_state(out=st.get("out"))
        got = [g["pos"], g["vel"]]
    if c["energy"]:
        d = sim.diagnostics()
        got += [np.array([d["spring_pe"], d["kinetic"], d["gravity_pe"], d["total"]]), d["linear"], d["angular"]]
    return got


# ------------------------------------------------------------------ in 64 bits --
def _dot(a, b):
    return (a * b).sum(1, keepdim=True)


def _norm(a):
    return a.square().sum(1, keepdim=True).sqrt()


def _plane(F, x, v, n, off, fk, fs):
    """A contact plane (rows of n, off, fk, fs per mass): friction against the force so far, then the push out."""
    disp = _dot(x, n) - off
    fn = n * _dot(F, n)
    vp = v - n * _dot(v, n)
    vn = _norm(vp)
    moving = F - vp * (fk * _norm(fn)) / vn.clamp_min(1e-300)
    held = torch.where(fs * _norm(fn) > _norm(F - fn), fn, F)
    out = torch.where(vn > 1e-16, moving, held) + n * (-disp * 20000.0)
    return torch.where(disp < 0, out, F)


def _simulate(sc, c, dev):
    t = lambda a, kind=torch.float64: torch.as_tensor(np.ascontiguousarray(a)).to(dev, kind)  # noqa: E731
    x, v, m = t(sc["pos"]), t(sc["vel"]), t(sc["m"]).unsqueeze(1)
    left, right = t(sc["left"], torch.int64), t(sc["right"], torch.int64)
    k, rest, damping = (t(sc[q]).unsqueeze(1) for q in ("k", "rest", "damping"))
    on = np.nonzero(sc["type"] >= 2)[0]
    sign = t(np.where(sc["type"][on] == 2, -1.0, 1.0) * sc["amp"][on]).unsqueeze(1)
    om, ph, on = t(sc["omega"][on]).unsqueeze(1), t(sc["phase"][on]).unsqueeze(1), t(on, torch.int64)
    g = t(G).unsqueeze(0)
    free = torch.ones_like(m) if "fixed" not in sc else (t(sc["fixed"]) == 0).double().unsqueeze(1)
    if "body_ptr" in sc:
        per = np.repeat(np.arange(len(sc["body_planes"])), np.diff(sc["body_ptr"]))
        planes = [tuple(t([p[q] for p in sc["body_planes"]]).reshape(len(sc["body_planes"]), -1)[t(per, torch.int64)]
                        for q in range(4))]
    else:
        planes = [(t(n).unsqueeze(0), off, fk, fs) for n, off, fk, fs in sc["planes"]]

    def acceleration(x, v, T):
        d = x[right] - x[left]
        r = _norm(d)
        u = d / r
        goal = rest
        if len(on):
            goal = rest.clone()
            goal[on] = rest[on] * (1.0 + sign * torch.sin(om * T + ph))
        f = u * (k * (goal - r))
        if c["damping"]:
            f = f + u * (_dot(v[left] - v[right], u) * damping)
        F = torch.zeros_like(x)
        F.index_add_(0, right, f)
        F.index_add_(0, left, f, alpha=-1)
        F = F + g * m
        if "ext" in sc:
            F = F + t(sc["ext"])
        if "body_ptr" not in sc:
            for p in planes:
                F = _plane(F, x, v, *p)
        for at, rad in sc["balls"]:
            e = x - t(at).unsqueeze(0)
            dist = _norm(e)
            F = torch.where(dist <= rad, F + 20000.0 * e / dist, F)
        if "body_ptr" in sc:
            F = _plane(F, x, v, *planes[0])
        if "drag" in sc:
            F = F - v * _norm(v) * t(np.trunc(sc["drag"])).unsqueeze(1)
        return F / m

    T, dt, before = 0.0, c["dt"], torch.zeros_like(x)
    for _ in range(c["steps"]):
        a = acceleration(x, v, T)
        if c["integ"] == "rk2":
            xm, vm = x + free * (0.5 * dt) * v, v + free * (0.5 * dt) * a
            a = acceleration(xm, vm, T + 0.5 * dt)
            x, v = x + free * dt * vm, v + free * dt * a
        elif c["integ"] == "verlet":
            v = v + free * 0.5 * (before + a) * dt
            x = x + free * (v * dt + 0.5 * a * dt * dt)
            before = a
        else:
            v = v + free * a * dt
            x = x + free * v * dt
        T += dt
    got = [x, v]
    if c["energy"]:
        stretch = _norm(x[left] - x[right]) - rest
        p = v * m
        pe, ke, gr = (k * stretch.square() / 2).sum(), (m * v.square() / 2).sum(), (m * 9.81 * x[:, 2:]).sum()
        spin = torch.stack([p[:, 1] * x[:, 2] - p[:, 2] * x[:, 1], x[:, 0] * p[:, 2] - p[:, 0] * x[:, 2],
                            p[:, 0] * x[:, 1] - p[:, 1] * x[:, 0]], 1)
        got += [torch.stack([pe, ke, gr, pe + ke + gr]), p.sum(0), spin.sum(0)]
    return [q.cpu().numpy() for q in got]


def exact(case, seed):
    c = dict(case)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    got = [_simulate(sc, c, dev) for sc in _scenes(c, seed)]
    if c["kind"] == "requests":
        return got
    return got[0]
