"""The work that a user of the engine has it do, as cases that can be timed.

listed() holds one case per kind of use; draw() gives others of the same
ranges.  prepare() builds a seeded packing on the engine (what a program
holds before its time loop), run() is one pass through the public entry
points, exact() the same pass in plain 64-bit torch where the result is a
computed number (spheres: every contact is a closed form).  For the other
shapes the closest points are what a GJK with tolerances of its own stops at,
which no independent 64-bit evaluation gives, so exact() is None there.

A pass of a stepping case is a rollout: the initial state goes in (the FP64
modes: gb_load_state from a state kept on the device; the mixed mode: from
pinned host buffers), the system advances by some steps in one call, and the
state it reached is read in place.  Every pass of a system so does the same
work, however often it is repeated.
"""
import math

import numpy as np
import torch

from grains3dgpu_b200 import abi, adjoint, engine, scenes

PREC = {"mixed": abi.GB_MIXED, "fp64": abi.GB_FP64, "strict": abi.GB_FP64_STRICT}
GJK = {"jh": abi.GB_GJK_JH, "sv": abi.GB_GJK_SV, "nesterov": abi.GB_GJK_NESTEROV}
LAW = {"hooke": abi.GB_LAW_HOOKE, "history": abi.GB_LAW_HOOKE_HISTORY}
INTEGRATOR = {"euler": abi.GB_FIRST_ORDER_EXPLICIT, "verlet": abi.GB_VELOCITY_VERLET}


def _case(kind, n, precision, steps, gjk="jh", law="history", integrator="euler", name=None):
    c = {"kind": kind, "n": n, "precision": precision, "steps": steps, "gjk": gjk, "law": law,
         "integrator": integrator}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest runs: a desktop-size column, a save interval of twenty
        # steps a call; launches and latency decide
        _case("column", 2000, "mixed", 20, gjk="sv", name="column_2k_mixed"),
        # the same kind of column all in FP64
        _case("column", 10_007, "fp64", 10, gjk="sv", name="column_10k_fp64"),
        # the headline: a million polydisperse superquadrics as a dense bed
        _case("bed", 1_000_000, "mixed", 10, name="bed_1M_mixed"),
        # a laboratory-size bed in the all-FP64 mode
        _case("bed", 130_003, "fp64", 10, name="bed_130k_fp64"),
        # the same grains before they settle: hardly a candidate pair
        _case("dilute", 500_000, "mixed", 20, name="dilute_500k_mixed"),
        # crushed rock: convex polyhedra of 8-32 vertices
        _case("polyhedra", 100_003, "mixed", 20, gjk="sv", name="polyhedra_100k_mixed"),
        # dense spheres, every lattice neighbour in contact: the FP64 mode with
        # the reference's law, and the mixed mode with the tangential history
        _case("spheres", 400_009, "fp64", 10, law="hooke", name="spheres_400k_fp64"),
        _case("spheres", 1_000_000, "mixed", 10, name="spheres_1M_mixed"),
        # the rotating drum's mix of spheres, cubes and superquadrics, packed
        _case("drum", 400_001, "mixed", 10, gjk="sv", name="drum_400k_mixed"),
        # gradients through a trajectory: calibration of the law's parameters
        _case("adjoint", 50_021, "fp64", 6, law="hooke", name="adjoint_50k_fp64"),
        # the drop-in behind a host code's ComponentManager: the state in and
        # out every step and the three calls on their own, in the parity mode
        _case("exchange", 20_011, "strict", 1, law="hooke", name="exchange_20k_strict"),
        # grains among fixed pegs (binned obstacles), velocity Verlet
        _case("pegs", 12_007, "fp64", 20, law="hooke", integrator="verlet", name="pegs_12k_fp64"),
    ]


# kind: smallest and largest n, precisions, GJK variants, laws, integrators, steps
RANGES = {
    "column": (300, 60_000, ("mixed", "fp64"), ("sv", "nesterov"), ("history",), ("euler", "verlet"), (10, 20)),
    "bed": (5000, 1_000_000, ("mixed", "fp64"), ("jh",), ("history",), ("euler", "verlet"), (5, 10)),
    "dilute": (10_000, 1_000_000, ("mixed", "fp64"), ("jh",), ("history",), ("euler",), (10, 20)),
    "polyhedra": (3000, 200_000, ("mixed", "fp64"), ("jh", "sv"), ("history",), ("euler",), (10, 20)),
    "spheres": (3000, 1_000_000, ("mixed", "fp64"), ("jh",), ("hooke", "history"), ("euler", "verlet"), (5, 10)),
    "drum": (8000, 500_000, ("mixed", "fp64"), ("sv",), ("history",), ("euler",), (5, 10)),
    "adjoint": (200, 100_000, ("fp64",), ("jh",), ("hooke",), ("euler", "verlet"), (3, 6)),
    "exchange": (500, 60_000, ("fp64", "strict", "mixed"), ("jh",), ("hooke",), ("euler",), (1,)),
    "pegs": (500, 60_000, ("mixed", "fp64", "strict"), ("jh",), ("hooke",), ("euler", "verlet"), (10, 20)),
}
# the FP64 modes' largest packings cost as much per step as a larger mixed one
FP64_CAP = {"bed": 250_000, "spheres": 400_000, "dilute": 500_000, "drum": 200_000, "polyhedra": 120_000}


def draw(rng):
    kind = rng.choice(sorted(RANGES))
    lo, hi, precs, gjks, laws, integs, steps = RANGES[kind]
    prec = rng.choice(precs)
    if prec != "mixed":
        hi = min(hi, FP64_CAP.get(kind, hi))
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.7:
        n |= 1  # mostly odd sizes
    gjk, k = rng.choice(gjks), rng.choice(steps)
    if gjk == "nesterov" and prec != "mixed":
        k = 5  # its longest pairs run to the iteration cap
    return _case(kind, min(n, hi), prec, k, gjk=gjk, law=rng.choice(laws),
                 integrator=rng.choice(integs))


# ---- the packings ---------------------------------------------------------------
def _box(n, pitch, margin, aspect=1.0, headroom=0.0):
    """A box whose jittered lattice holds n sites, about `aspect` times as high
    as wide, with `headroom` above them."""
    m = max(3, int(math.ceil((n / aspect) ** (1.0 / 3.0))))
    nz = int(math.ceil(n / (m * m)))
    side = 2 * margin + (m - 0.5) * pitch
    return (side, side, 2 * margin + (nz - 0.5) * pitch + headroom)


def _polyhedra(n, seed, pitch=2.13e-3, radius=1.05e-3):
    """n grains of 512 convex polyhedra (hulls of 8-32 points on ellipsoids),
    each scaled to the same circumscribed radius so that lattice neighbours
    come within their crusts and no cores intersect."""
    lib = engine.load()

    def centroid(v):
        c, vol = np.zeros(3), abi.C.c_double(0.0)
        lib.convex_hull_centroid(abi.dptr(np.ascontiguousarray(v)), v.shape[0], abi.dptr(c),
                                 abi.C.byref(vol))
        return c

    s = scenes.polyhedra_box(seed=seed, n=512, hull_centroid=centroid)
    for rb in s.rbs:
        v = s.vertices[rb["first_vertex"]:rb["first_vertex"] + rb["n_vertices"]]
        v *= radius / np.linalg.norm(v, axis=1).max()
    rng = np.random.default_rng(seed)
    box = _box(n, pitch, 1.6e-3, headroom=0.01)
    pos, _ = scenes.lattice(box, pitch, 1.6e-3, n, rng, 0.01e-3)
    tr = np.zeros((n, 12))
    tr[:, :9] = scenes.random_rotations(rng, n)
    tr[:, 9:] = pos
    vel = np.zeros((n, 6))
    vel[:, :3] = rng.normal(0.0, 0.05, size=(n, 3))
    vel[:, 3:] = rng.normal(0.0, 5.0, size=(n, 3))
    walls, wtr = scenes.box_walls(box)
    cfg = dict(s.config, n_particles=n, max_coordinate=box)
    return scenes.Scene("polyhedra", cfg, s.rbs, s.vertices,
                        rng.integers(0, 512, n).astype(np.uint32), tr, vel, walls, wtr,
                        s.contact_models)


def _column(n, seed, pitch, tilt):
    box = _box(n, pitch, 1.6e-3, headroom=0.01)
    s = scenes.superquadric_column(seed=seed, n=n, box=box, pitch=pitch, jitter=0.02e-3, tilt=tilt)
    rng = np.random.default_rng(seed + 1)
    s.velocities[:, :3] = rng.normal(0.0, 0.05, size=(n, 3))
    s.velocities[:, 3:] = rng.normal(0.0, 5.0, size=(n, 3))
    return s


def _drum(n, seed):
    """The rotating drum's grains packed until lattice neighbours touch, as in
    a drum that has turned for a while: a 2.05 mm lattice with little jitter,
    grains of about that width turned by up to 0.1 rad per axis, so that many
    crusts meet while the cores stay apart."""
    pitch, margin = 2.05e-3, 1.7e-3
    s = scenes.rotating_drum(seed=seed, n=n, margin=margin, v_sigma=0.1, pitch=pitch)
    s.rbs[0]["p"][0] = 1.03e-3
    s.vertices *= 0.85 / 0.8
    s.rbs[2]["p"][:3] *= 0.93
    rng = np.random.default_rng(seed + 1)
    x = s.transforms[:, 9:]
    first = np.array([1e-3 + margin, 2e-3, 1e-3 + margin])  # a site of the drum's lattice
    x -= 0.75 * (x - first - pitch * np.round((x - first) / pitch))
    q = np.concatenate([np.ones((n, 1)), rng.uniform(-0.05, 0.05, (n, 3))], 1)
    s.transforms[:, :9] = scenes.quat_to_matrix(q / np.linalg.norm(q, axis=1, keepdims=True))
    s.velocities[:, 3:] = rng.normal(0.0, 5.0, size=(n, 3))
    return s


def _spheres(n, seed):
    """The sphere bed with its grains' places drawn from the seed."""
    box = _box(n, 2.05e-3, 1.6e-3, headroom=0.03)
    s = scenes.sphere_bed(seed=seed, n=n, box=box)
    rng = np.random.default_rng(seed + 1)
    s.transforms[:, 9:] += rng.uniform(-0.02e-3, 0.02e-3, size=(n, 3))
    s.transforms[:, :9] = scenes.random_rotations(rng, n)
    return s


def _scene(case, seed):
    n, kind = case["n"], case["kind"]
    seed = 1 + seed % (1 << 30)
    if kind == "column":  # dense: neighbours within the crusts' reach
        return _column(n, seed, 2.13e-3, 0.05), abi.GB_FLAG_CRUST_BOUNDS
    if kind == "bed":
        if n >= 500_000:  # the headline's own box
            return scenes.polydisperse_bed(seed=seed, n=n), 0
        return scenes.polydisperse_bed(seed=seed, n=n, box=_box(n, 2.2e-3, 2.5e-3, 0.7, 0.2)), 0
    if kind == "dilute":
        side = 0.3 * (n / 1e6) ** (1.0 / 3.0)
        return scenes.polydisperse_superquadrics(seed=seed, n=n, box=(side, side, 4 * side)), 0
    if kind == "polyhedra":
        return _polyhedra(n, seed), abi.GB_FLAG_CRUST_BOUNDS
    if kind in ("spheres", "adjoint"):
        return _spheres(n, seed), 0
    if kind == "drum":
        return _drum(n, seed), abi.GB_FLAG_CRUST_BOUNDS
    if kind == "exchange":  # the reference's GJK on randomly turned, touching grains
        return _column(n, seed, 2.05e-3, None), 0
    pegs = 40 + n // 40
    s = scenes.peg_board(seed=seed, n=n, pegs=pegs,
                         box=_box(n + pegs, 2.05e-3, 1.2e-3, headroom=0.003))
    s.contact_models = [dict(m, etat=3000.0, muc=0.05) for m in s.contact_models]
    return s, 0


# ---- the states and the passes --------------------------------------------------
class _DeviceRows:
    """`rows` x n values of one of the engine's device arrays.  A tensor made of
    it holds it, and it the engine that owns the memory."""

    def __init__(self, system, name, rows, dtype):
        self.system = system
        p = abi.C.c_void_p()
        system._check(system.lib.device_pointer(system.ctx, name, abi.C.byref(p)), "device_pointer")
        self.__cuda_array_interface__ = {"shape": (rows, system.n), "typestr": dtype,
                                         "data": (p.value, False), "version": 2}


def _views(system, precision):
    t = "<f4" if precision == "mixed" else "<f8"
    rows = {"pos": (b"pos_x", 3, "<f8"), "rot": (b"rotation", 8 if precision == "mixed" else 9, t),
            "vel": (b"vel_x", 3, t), "omega": (b"omega_x", 3, t)}
    return {k: torch.as_tensor(_DeviceRows(system, *v), device="cuda") for k, v in rows.items()}


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    scene, flags = _scene(case, seed)
    kw = dict(contact_law=LAW[case["law"]], gjk_variant=GJK[case["gjk"]],
              integrator=INTEGRATOR[case["integrator"]], flags=flags)
    dev = torch.cuda.current_device()
    if case["kind"] == "adjoint":
        s.sim = adjoint.Simulation(scene, precision=PREC[case["precision"]], device=dev, **kw)
        put = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
        s.x, s.v, s.w = (put(scene.transforms[:, 9:]), put(scene.velocities[:, :3]),
                         put(scene.velocities[:, 3:]))
        s.laws = s.sim.law_tensor()
        s.weights = _weights(case, seed)
        return s
    s.system = scenes.System(engine.load(), scene, precision=PREC[case["precision"]], device=dev, **kw)
    if case["kind"] == "exchange":
        s.tr, s.kin = scene.transforms.copy(), scene.velocities.copy()
        s.contacts = np.zeros(s.system.n, np.int32)
        return s
    stream = torch.cuda.current_stream().cuda_stream
    s.system._check(s.system.lib.set_stream(s.system.ctx, abi.C.c_void_p(stream)), "set_stream")
    s.views = _views(s.system, case["precision"])
    if case["precision"] == "mixed":
        pin = lambda a: torch.tensor(a).pin_memory().numpy()  # noqa: E731
        s.tr, s.kin = pin(scene.transforms), pin(scene.velocities)
    else:
        s.state = torch.empty((18, s.system.n), dtype=torch.float64, device="cuda")
        s.system._check(s.system.lib.save_state(s.system.ctx, abi.C.c_void_p(s.state.data_ptr())),
                        "save_state")
    torch.cuda.synchronize()
    return s


def _weights(case, seed):
    g = torch.Generator().manual_seed(int(seed) + 3)
    return [torch.randn((case["n"], 3), generator=g, dtype=torch.float64).cuda() for _ in range(3)]


def run(s):
    case = s.case
    if case["kind"] == "adjoint":
        leaves = [t.detach().clone().requires_grad_(True) for t in (s.x, s.v, s.w, s.laws)]
        out = adjoint.trajectory(s.sim, *leaves, case["steps"], 3)
        loss = sum((w * o).sum() for w, o in zip(s.weights, out))
        loss.backward()
        return {"x": out[0].detach(), "v": out[1].detach(), "w": out[2].detach(),
                "grad_x": leaves[0].grad, "grad_v": leaves[1].grad, "grad_w": leaves[2].grad,
                "grad_laws": leaves[3].grad}
    if case["kind"] == "exchange":
        # GrainsCPU::simulate's loop body with the state owned by the host
        y = s.system
        y.set_transforms(s.tr)
        y.set_velocities(s.kin)
        s.contacts[:] = 0
        y.detect(s.contacts)
        torces = y.torces()
        y.add_external_forces()
        y.move()
        return {"transforms": y.transforms(), "velocities": y.velocities(), "torces": torces,
                "contacts": s.contacts.copy()}
    y = s.system
    if case["precision"] == "mixed":
        y.set_transforms(s.tr)
        y.set_velocities(s.kin)
    else:
        y._check(y.lib.load_state(y.ctx, abi.C.c_void_p(s.state.data_ptr())), "load_state")
    if case["integrator"] == "verlet":
        y._check(y.lib.set_integrator_phase(y.ctx, 0), "set_integrator_phase")
    y.step(case["steps"])
    return s.views


# ---- what a pass cannot do without ------------------------------------------------
# ordered candidate pairs per grain, and flops an unordered one cannot do
# without: a closed-form sphere contact ~150; a pair of other shapes its
# bounding boxes and one support each, ~300
PAIRS = {"column": 8.0, "bed": 7.7, "dilute": 0.02, "polyhedra": 4.0, "spheres": 4.0, "drum": 7.0,
         "adjoint": 4.0, "exchange": 12.0, "pegs": 4.0}


def work(case):
    n, steps = case["n"], case["steps"]
    mixed = case["precision"] == "mixed"
    state = 24 + (56 if mixed else 120)  # position, orientation, velocities
    per_step = 2.0 * state * n
    if case["kind"] in ("bed", "dilute"):  # every grain its own shape and inertia
        per_step += (100 + 64 if mixed else 176 + 128) * n
    else:
        per_step += 4.0 * n
    flops = steps * n * (150.0 + 0.5 * PAIRS[case["kind"]]
                         * (150.0 if case["kind"] in ("spheres", "adjoint", "pegs") else 300.0))
    if case["kind"] == "adjoint":
        return {"bytes": 2.0 * steps * per_step, "flops": 3.0 * flops}
    if case["kind"] == "exchange":
        return {"bytes": 2.0 * 144 * n + 48 * n + per_step, "flops": flops}
    return {"bytes": 144.0 * n + steps * per_step, "flops": flops}


def tolerance(case):
    # About four times what the modes differ by among themselves (FP64 against
    # FP64 in another operation order; mixed against FP64).  Spheres are
    # closed forms: FP64 carries every sum in 64 bits, the mixed mode keeps
    # velocities and forces in FP32.  Other shapes: a contact's witness points
    # are where GJK's tolerance stops it, which moves with rounding -- little
    # for the reference's Johnson GJK on superquadrics, more for the
    # signed-volume one on nearly parallel faces and for polyhedra.
    mixed = case["precision"] == "mixed"
    if case["kind"] in ("spheres", "adjoint", "pegs"):
        return {"rel": 1e-5, "max": 1e-3} if mixed else {"rel": 1e-9}
    if case["kind"] in ("bed", "dilute", "exchange"):
        return {"rel": 1e-6, "max": 1e-4, "differ": 0.0} if mixed else {"rel": 1e-9, "max": 1e-6}
    if case["kind"] == "polyhedra":
        return {"rel": 5e-3, "max": 0.9}
    return {"rel": 2e-4, "max": 0.05}


# ---- spheres in plain 64-bit torch ------------------------------------------------
def _pairs(x, reach):
    """Ordered pairs (a, b), a != b, of centres closer than `reach`."""
    n = x.shape[0]
    c = torch.floor((x - x.min(0).values) / reach).to(torch.int64) + 1
    dim = c.max(0).values + 2
    key = (c[:, 2] * dim[1] + c[:, 1]) * dim[0] + c[:, 0]
    skey, order = torch.sort(key)
    found = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                k = key + (dz * dim[1] + dy) * dim[0] + dx
                lo, hi = torch.searchsorted(skey, k), torch.searchsorted(skey, k, right=True)
                for j in range(int((hi - lo).max()) if n else 0):
                    a = torch.nonzero(lo + j < hi).squeeze(1)
                    b = order[lo[a] + j]
                    near = ((x[b] - x[a]).square().sum(1) < reach * reach) & (a != b)
                    found.append(torch.stack([a[near], b[near]]))
    p = torch.cat(found, 1)
    return p[:, torch.argsort(p[0] * n + p[1])]


def _cross(a, b):
    return torch.cross(a, b, dim=1)


def _norm(a):
    return a.square().sum(1, keepdim=True).sqrt()


def _force(history, law, dt, vec, rel, m1, m2, arm, xi):
    """A contact's force and torque on its first body, and the new tangential
    spring: the Hooke law of the reference, or the spring-dashpot with history.
    m2 None: a wall."""
    kn, en, etat, muc, kt = law
    c = torch.log(en) / torch.sqrt(math.pi ** 2 + torch.log(en) ** 2)
    nrm = vec / _norm(vec)
    vn = (rel * nrm).sum(1, keepdim=True) * nrm
    vt = rel - vn
    if history:
        ms = m1 if m2 is None else m1 * m2 / (m1 + m2)
        fn = kn * vec + 2.0 * c * torch.sqrt(kn * ms) * vn
        xi = xi - (xi * nrm).sum(1, keepdim=True) * nrm + dt * vt
        gt = 2.0 * etat * ms
        ft = -kt * xi - gt * vt
        cap, size = muc * _norm(fn), _norm(ft)
        slides = size > cap
        ft = torch.where(slides, cap / torch.where(slides, size, torch.ones_like(size)) * ft, ft)
        xi = torch.where(slides, (-1.0 / kt) * (ft + gt * vt), xi)
    else:
        if m2 is None:
            ms, omega = 0.5 * m1, 2.0 * torch.sqrt(kn / (0.5 * m1))
        else:
            ms = m1 * m2 / (m1 + m2)
            omega = torch.sqrt(kn / ms)
        fn = kn * vec + 2.0 * omega * c * ms * vn
        ft = -2.0 * etat * ms * vt
        size = ft.square().sum(1, keepdim=True)
        cap = muc * _norm(fn)
        slides = size > cap * cap
        nvt = torch.where(slides, vt, torch.ones_like(vt))
        ft = torch.where(slides, -cap * vt / _norm(nvt), ft)
    return fn + ft, _cross(arm, fn + ft), xi


class _Spheres:
    """Spheres of one size on planar walls and among spherical pegs."""

    def __init__(self, case, scene, laws=None):
        put = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64).cuda()  # noqa: E731
        self.history, self.verlet = case["law"] == "history", case["integrator"] == "verlet"
        self.dt = scene.config["dt"]
        self.g = put(np.array(scene.config["gravity"], float))
        self.r = float(scene.rbs[0]["p"][0])
        self.m = float(scene.rbs[0]["density"]) * 4.0 / 3.0 * math.pi * self.r ** 3
        self.inertia = 0.4 * self.m * self.r ** 2
        self.m_t = put(np.array(self.m))
        wall = scene.obstacles["type"] == abi.GB_RECTANGLE
        tr = scene.obstacle_transforms
        self.normals, self.origins = put(tr[wall][:, [2, 5, 8]]), put(tr[wall][:, 9:])
        self.pegs, self.peg_r = put(tr[~wall][:, 9:]), float(scene.obstacles["p"][~wall][:, 0].max()) if (~wall).any() else 0.0
        # materials: grains 0, walls and pegs 1
        keys = ("kn", "en", "etat", "muc", "kt")
        self.laws = put(np.array([[m[k] for k in keys] for m in scene.contact_models]))
        if laws is not None:  # kn, en, etat, muc as differentiable inputs
            self.laws = torch.cat([laws, self.laws[:, 4:]], 1)
        self.xi = self.xi_key = None
        self.started = False

    def step(self, x, v, w):
        n, dt, r = x.shape[0], self.dt, self.r
        F, T = torch.zeros_like(x), torch.zeros_like(x)
        with torch.no_grad():
            a, b = _pairs(x.detach(), 2 * r)
        # grains on grains
        d = x[b] - x[a]
        dist = _norm(d)
        u, overlap = d / dist, dist - 2 * r
        pt = x[a] + (r + 0.5 * overlap) * u
        arm = pt - x[a]
        if self.history:
            rel = (v[a] + _cross(w[a], arm)) - (v[b] + _cross(w[b], pt - x[b]))
        else:  # the reference's lever arm: the contact point itself
            rel = (v[a] + _cross(w[a], pt)) - (v[b] + _cross(w[b], pt))
        xi, key = torch.zeros_like(d), a * n + b
        if self.history and self.xi_key is not None:
            at = torch.searchsorted(self.xi_key, key).clamp(max=len(self.xi_key) - 1)
            xi = torch.where((self.xi_key[at] == key)[:, None], self.xi[at], xi)
        f, t, self.xi = _force(self.history, self.laws[0], dt, overlap * u, rel, self.m_t, self.m_t,
                               arm, xi)
        self.xi_key = key
        F, T = F.index_add(0, a, f), T.index_add(0, a, t)
        # grains on walls, met as planes
        for nw, ow in zip(self.normals, self.origins):
            e = x - ow
            side = torch.sign((e * nw).sum(1, keepdim=True))
            s = side * (e * nw).sum(1, keepdim=True) - r
            hit = torch.nonzero(s[:, 0] < 0).squeeze(1)
            rn, sh = (side * nw)[hit], s[hit]
            pt = x[hit] - (r + 0.5 * sh) * rn
            arm = pt - x[hit]
            rel = v[hit] + _cross(w[hit], arm if self.history else pt)
            f, t, _ = _force(self.history, self.laws[1], dt, -sh * rn, rel, self.m_t, None, arm,
                             torch.zeros_like(rn))
            F, T = F.index_add(0, hit, f), T.index_add(0, hit, t)
        # grains on pegs
        for p in self.pegs:
            d = p - x
            hit = torch.nonzero(_norm(d)[:, 0] < r + self.peg_r).squeeze(1)
            if not len(hit):
                continue
            d = d[hit]
            dist = _norm(d)
            overlap = dist - r - self.peg_r
            pt = x[hit] + (r + 0.5 * overlap) * d / dist
            arm = pt - x[hit]
            rel = v[hit] + _cross(w[hit], arm if self.history else pt)
            f, t, _ = _force(self.history, self.laws[1], dt, overlap * d / dist, rel, self.m_t, None,
                             arm, torch.zeros_like(d))
            F, T = F.index_add(0, hit, f), T.index_add(0, hit, t)
        acc, alpha = F / self.m + self.g, T / self.inertia
        if self.verlet:
            h = dt if self.started else 0.5 * dt
            v, w = v + h * acc, w + h * alpha
            x, turn = x + dt * v, w
        else:
            x, turn = x + dt * v, w
            v, w = v + dt * acc, w + dt * alpha
        self.started = True
        return x, v, w, turn


def _rotate(R, w, dt):
    """exp(dt [w]x) R."""
    th = _norm(w)[:, :, None] * dt
    k = w / _norm(w).clamp(min=1e-300)
    z = torch.zeros_like(k[:, 0])
    K = torch.stack([z, -k[:, 2], k[:, 1], k[:, 2], z, -k[:, 0], -k[:, 1], k[:, 0], z], 1).view(-1, 3, 3)
    half = torch.sin(0.5 * th)
    return R + (torch.sin(th) * K + 2.0 * half * half * (K @ K)) @ R


def exact(case, seed):
    if case["kind"] not in ("spheres", "adjoint", "pegs"):
        return None
    scene, _ = _scene(case, seed)
    put = lambda a: torch.tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    x, v, w = put(scene.transforms[:, 9:]), put(scene.velocities[:, :3]), put(scene.velocities[:, 3:])
    if case["kind"] == "adjoint":
        laws = torch.tensor([[m[k] for k in adjoint.LAW_PARAMS] for m in scene.contact_models],
                            dtype=torch.float64)
        leaves = [t.requires_grad_(True) for t in (x, v, w, laws)]
        model = _Spheres(case, scene, leaves[3].cuda())
        for _ in range(case["steps"]):
            x, v, w, _ = model.step(x, v, w)
        loss = sum((k * o).sum() for k, o in zip(_weights(case, seed), (x, v, w)))
        grads = torch.autograd.grad(loss, leaves)
        return {"x": x.detach(), "v": v.detach(), "w": w.detach(), "grad_x": grads[0],
                "grad_v": grads[1], "grad_w": grads[2], "grad_laws": grads[3]}
    R = put(scene.transforms[:, :9]).view(-1, 3, 3)
    model = _Spheres(case, scene)
    for _ in range(case["steps"]):
        x, v, w, turn = model.step(x, v, w)
        R = _rotate(R, turn, model.dt)
    # the mixed mode keeps a quaternion in two FP32 parts: no single 64-bit value
    rot = None if case["precision"] == "mixed" else R.reshape(-1, 9).T.contiguous()
    return {"pos": x.T.contiguous(), "rot": rot, "vel": v.T.contiguous(), "omega": w.T.contiguous()}
