"""The narrow phase's unordered FP32 cull, its mirror records and the
sphere-only pass, against the FP64 oracle at list lengths around a warp's
batch of 32 pairs: mixtures of shapes (spheres of two radii, boxes,
polyhedra: supports without transcendental functions, so FP64-strict is bit
exact) and packings of spheres alone."""
import numpy as np
import pytest

from grains3dgpu_b200 import abi, scenes

from conftest import rel_err, share_props
from test_gpu_parity import pair

pytestmark = pytest.mark.gpu

SPHERES = (0, 1)
MIXTURE = (0, 1, 2, 3)


def packing(n, bodies, seed=3):
    """n grains of the given bodies on a 1.9 mm lattice, randomly turned by up
    to 0.3 rad, moving."""
    m = max(2, int(np.ceil(n ** (1 / 3))))
    side = 3.2e-3 + (m + 1) * 1.9e-3
    s = scenes.superquadric_column(seed=seed, n=n, pitch=1.9e-3, box=(side, side, side + 2e-3),
                                   shape="box", tilt=0.3)
    rng = np.random.default_rng(seed)
    rbs = np.zeros(4, scenes.RB_DTYPE)
    rbs["density"] = 2500.0
    rbs["crust"] = [5e-5, 4e-5, 5e-5, 4e-5]
    rbs["type"] = [abi.GB_SPHERE, abi.GB_SPHERE, abi.GB_BOX, abi.GB_POLYHEDRON]
    rbs["p"][0, 0], rbs["p"][1, 0] = 1.1e-3, 0.9e-3
    rbs["p"][2, :3] = [0.8e-3, 0.7e-3, 0.9e-3]
    rbs[3]["n_vertices"] = 8
    h = 0.85e-3
    s.vertices = np.array([[x * h, y * h, z * h] for x in (-1, 1) for y in (-1, 1)
                           for z in (-1, 1)])
    s.rbs = rbs
    s.rb_ids = rng.choice(bodies, size=n).astype(np.uint32)
    if set(bodies) == set(SPHERES):
        s.rbs, s.vertices = rbs[:2].copy(), np.zeros((0, 3))
    s.config["n_rigid_bodies"] = len(s.rbs)
    s.velocities = rng.normal(0.0, 0.1, (n, 6))
    s.contact_models = [dict(m, etat=0.3) for m in s.contact_models]
    return s


@pytest.mark.parametrize("variant", [abi.GB_GJK_JH, abi.GB_GJK_SV])
@pytest.mark.parametrize("n", [2, 11, 33, 400])
def test_mixture_single_step_bit_exact(gb, oracle, n, variant):
    g, o = pair(gb, oracle, packing(n, MIXTURE), gjk_variant=variant)
    g.detect()
    o.detect()
    assert np.array_equal(g.dump(abi.GB_DUMP_CONTACT_PAIRS), o.dump(abi.GB_DUMP_CONTACT_PAIRS))
    assert np.array_equal(g.dump(abi.GB_DUMP_CONTACT_INFO), o.dump(abi.GB_DUMP_CONTACT_INFO),
                          equal_nan=True)
    assert np.array_equal(g.torces(), o.torces(), equal_nan=True)
    if n == 400:
        assert g.stats().contacts > 0


def test_basis_off_orthonormal_takes_the_fp64_path(gb, oracle):
    """A basis scaled by 1 + 1e-3 is outside what the FP32 certificates
    assume; its pairs must reach the FP64 solve and agree all the same."""
    s = packing(200, (2, 3))
    s.transforms[:, :9] *= 1.001
    g, o = pair(gb, oracle, s, gjk_variant=abi.GB_GJK_SV)
    g.detect()
    o.detect()
    assert g.stats().gjk_fp64_calls == g.stats().candidate_pairs > 0
    assert np.array_equal(g.dump(abi.GB_DUMP_CONTACT_PAIRS), o.dump(abi.GB_DUMP_CONTACT_PAIRS))
    assert np.array_equal(g.torces(), o.torces(), equal_nan=True)


@pytest.mark.parametrize("law", [abi.GB_LAW_HOOKE, abi.GB_LAW_HOOKE_HISTORY])
@pytest.mark.parametrize("n", [2, 33, 257])
def test_spheres_alone(gb, oracle, n, law):
    """The sphere-only pass over a few steps: FP64-strict repeats the oracle,
    the FP64 and mixed modes follow it within their rounding.  The torque of a
    normal force is pure rounding, eps r F, so a contact and step may turn the
    0.9 mm sphere by eps r F dt / I: with F up to kn (0.3 mm) = 3 N and
    I = 2.5e-12 kg m2 that is 2.6e-4 rad/s in FP32 (eps 1.2e-7) and 5e-13 in
    FP64, of largest velocities of 0.1-0.3: 1e-3 and 1e-10 leave the FP32
    bound times one contact and the FP64 one times many."""
    for precision, tol in ((abi.GB_FP64_STRICT, 1e-14), (abi.GB_FP64, 1e-10), (abi.GB_MIXED, 1e-3)):
        g, o = pair(gb, oracle, packing(n, SPHERES), precision=precision, contact_law=law)
        for _ in range(2):
            for y in (g, o):
                y.detect()
                y.add_external_forces()
                y.move()
        g.step(2)
        o.step(2)
        assert np.array_equal(g.dump(abi.GB_DUMP_CONTACT_PAIRS), o.dump(abi.GB_DUMP_CONTACT_PAIRS))
        assert rel_err(g.velocities(), o.velocities()) <= tol
        if n > 2:
            assert g.stats().contacts > 0


def big_grain(shape, first, n=1350, seed=9):
    """One large grain among n small ones that touch it: small spheres (and a
    tenth boxes) on the shell of a large sphere, or small boxes lying on the
    faces of a large box.  The large grain is the first or the last particle,
    which decides in whose list the other's record is looked up."""
    rng = np.random.default_rng(seed)
    R, r = 4e-3, 0.2e-3
    rbs = np.zeros(4, scenes.RB_DTYPE)
    rbs["density"] = 2500.0
    rbs["crust"] = 5e-5
    rbs["type"] = [abi.GB_SPHERE, abi.GB_SPHERE, abi.GB_BOX, abi.GB_BOX]
    rbs["p"][0, 0], rbs["p"][1, 0] = R, r
    rbs["p"][2, :3], rbs["p"][3, :3] = R, r
    if shape == "sphere":
        k = np.arange(n) + 0.5
        phi, z = np.pi * (1 + 5 ** 0.5) * k, 1 - 2 * k / n
        u = np.stack([np.sqrt(1 - z * z) * np.cos(phi), np.sqrt(1 - z * z) * np.sin(phi), z], 1)
        pos = u * (R + r * rng.uniform(0.8, 1.05, n))[:, None]
        ids = np.where(rng.random(n) < 0.1, 3, 1)
    else:
        m = int(np.ceil(np.sqrt(n / 6)))
        s = (np.arange(m) - (m - 1) / 2) * (2 * (R - r) / (m - 1))
        u, v = (x.ravel() for x in np.meshgrid(s, s, indexing="ij"))
        h = R + r + rng.uniform(0.5e-5, 0.9e-4, (6, m * m))
        faces = []
        for f in range(6):
            q = np.zeros((m * m, 3))
            q[:, f % 3] = h[f] * (1 if f < 3 else -1)
            q[:, (f + 1) % 3], q[:, (f + 2) % 3] = u, v
            faces.append(q)
        pos = np.concatenate(faces)[:n]
        ids = np.full(n, 3)
    rot = np.tile(np.eye(3).ravel(), (n + 1, 1))
    ang = rng.uniform(-0.05, 0.05, n + 1)
    rot[:, 0], rot[:, 1], rot[:, 3], rot[:, 4] = np.cos(ang), -np.sin(ang), np.sin(ang), np.cos(ang)
    at = 0 if first else n
    side = 0.03
    tr = np.zeros((n + 1, 12))
    tr[:, :9] = rot
    tr[:, 9:] = np.insert(pos, at, 0.0, axis=0) + 0.5 * side
    ids = np.insert(ids, at, 0 if shape == "sphere" else 2).astype(np.uint32)
    walls, wtr = scenes.box_walls((side,) * 3)
    cfg = dict(n_particles=n + 1, n_rigid_bodies=4, n_obstacles=6, n_materials=2,
               origin=(0, 0, 0), max_coordinate=(side,) * 3, dt=1e-6, gravity=(0, 0, -9.81))
    vel = rng.normal(0.0, 0.05, (n + 1, 6))
    return scenes.Scene("big-grain", cfg, rbs, np.zeros((0, 3)), ids, tr, vel, walls, wtr,
                        [scenes.law(etat=0.3)] * 3)


@pytest.mark.parametrize("first", [True, False])
@pytest.mark.parametrize("shape", ["sphere", "box"])
def test_mirror_records_of_a_long_list(gb, oracle, shape, first):
    """Records looked up in a list of a thousand (the closed form of two
    spheres, the queue of the FP64 GJK): both orders of every contact, bit for
    bit."""
    s = big_grain(shape, first)
    kw = dict(gjk_variant=abi.GB_GJK_SV, contact_law=abi.GB_LAW_HOOKE)
    g = scenes.System(gb, s, precision=abi.GB_FP64_STRICT, **kw,
                      flags=abi.GB_FLAG_CRUST_BOUNDS | abi.GB_FLAG_RECORD_CONTACT_INFO)
    o = scenes.System(oracle, s, flags=abi.GB_FLAG_CRUST_BOUNDS, **kw)
    share_props(g, o, oracle)
    g.detect()
    o.detect()
    contacts = g.dump(abi.GB_DUMP_CONTACT_PAIRS)
    big = 0 if first else s.n - 1
    assert (contacts[:, 0] == big).sum() > 300
    assert np.array_equal(contacts, o.dump(abi.GB_DUMP_CONTACT_PAIRS))
    assert np.array_equal(g.dump(abi.GB_DUMP_CONTACT_INFO), o.dump(abi.GB_DUMP_CONTACT_INFO),
                          equal_nan=True)
    assert np.array_equal(g.torces(), o.torces(), equal_nan=True)


@pytest.mark.parametrize("variant", [abi.GB_GJK_JH, abi.GB_GJK_SV])
def test_mixture_of_several_rounds(gb, oracle, variant):
    """A list several times as long as the cull's threads (five blocks of 128 a
    multiprocessor: 94,720 records at a time), so that what a stage leaves in a
    warp's queues is carried over from round to round."""
    g, o = pair(gb, oracle, packing(40_000, MIXTURE), gjk_variant=variant)
    g.detect()
    o.detect()
    assert g.stats().candidate_pairs > 300_000
    assert np.array_equal(g.dump(abi.GB_DUMP_CONTACT_PAIRS), o.dump(abi.GB_DUMP_CONTACT_PAIRS))
    assert np.array_equal(g.dump(abi.GB_DUMP_CONTACT_INFO), o.dump(abi.GB_DUMP_CONTACT_INFO),
                          equal_nan=True)
    assert np.array_equal(g.torces(), o.torces(), equal_nan=True)


def loose_boxes(n=20_000, stretch=1.2, crust=2e-4):
    """Boxes alone, far enough apart that nearly all of them meet in their
    crusts; no polyhedron in the table of bodies."""
    s = packing(n, (2,))
    s.rbs, s.vertices = s.rbs[:3].copy(), np.zeros((0, 3))
    s.rbs["crust"] = crust
    s.config["n_rigid_bodies"] = 3
    s.config["max_coordinate"] = tuple(stretch * x for x in s.config["max_coordinate"])
    for a in (s.transforms[:, 9:], s.obstacle_transforms[:, 9:], s.obstacles["p"]):
        a *= stretch
    return s


@pytest.mark.parametrize("variant", [abi.GB_GJK_SV, abi.GB_GJK_NESTEROV])
def test_long_queue_of_signed_volume_solves(gb, oracle, variant):
    """More FP64 solves than a wave of four-lane pairs holds (at most four
    blocks of 128 a multiprocessor: 18,944), which the two-lane form takes:
    FP64-strict bit for bit as the oracle; in the mixed mode the same contacts,
    and forces within 1e-5 but for the grains whose cores all but intersect."""
    s = loose_boxes()
    kw = dict(gjk_variant=variant, flags=abi.GB_FLAG_CRUST_BOUNDS)
    o = scenes.System(oracle, s, **kw)
    g, m, f = (scenes.System(gb, s, precision=p, **kw)
               for p in (abi.GB_FP64_STRICT, abi.GB_MIXED, abi.GB_FP64))
    share_props(g, o, oracle)
    for y in (o, g, m, f):
        y.detect()
    assert min(y.stats().gjk_fp64_calls for y in (g, m, f)) > 20_000
    want = o.dump(abi.GB_DUMP_CONTACT_PAIRS)
    assert want.shape[0] > 20_000
    for y in (g, m, f):
        assert np.array_equal(y.dump(abi.GB_DUMP_CONTACT_PAIRS), want)
    assert np.array_equal(g.torces(), o.torces(), equal_nan=True)
    a, b = (y.dump(abi.GB_DUMP_CONTACT_FORCES)[:, :3] for y in (m, f))
    ok = np.isfinite(a).all(1) & np.isfinite(b).all(1)
    assert ok.mean() > 0.97
    err = np.linalg.norm(a[ok] - b[ok], axis=1) / np.linalg.norm(b[ok], axis=1)
    assert np.quantile(err, 0.99) <= 1e-5


@pytest.mark.parametrize("large", [True, False])
def test_mixed_sums_of_long_and_short_lists(gb, large):
    """The mixed mode's per-particle sums in both forms of that pass: a grain
    twenty times as large as the median body, with a thousand contacts (the
    plain loop), and a mixture of like sizes (single records).  Forces against
    the FP64 mode's: sums of n FP32 values of at most the largest contact
    force each, within n 2^-24 of their sum and the contacts' own 1e-6."""
    s = big_grain("sphere", False) if large else packing(400, MIXTURE)
    m, f = (scenes.System(gb, s, precision=p) for p in (abi.GB_MIXED, abi.GB_FP64))
    m.detect()
    f.detect()
    pairs = f.dump(abi.GB_DUMP_CONTACT_PAIRS)
    assert np.array_equal(m.dump(abi.GB_DUMP_CONTACT_PAIRS), pairs)
    force = np.linalg.norm(f.dump(abi.GB_DUMP_CONTACT_FORCES)[:, :3], axis=1)
    count = np.bincount(pairs[:, 0], minlength=s.n)
    total = np.bincount(pairs[:, 0], force, minlength=s.n)
    assert count.max() > 900 if large else 3 < count.max() < 64
    inside = np.all((s.transforms[:, 9:] > 3e-3)
                    & (s.transforms[:, 9:] < np.array(s.config["max_coordinate"]) - 3e-3), axis=1)
    err = np.linalg.norm(m.torces()[:, :3] - f.torces()[:, :3], axis=1)
    assert np.all(err[inside] <= (count * 2.0 ** -24 + 1e-6)[inside] * total[inside])
