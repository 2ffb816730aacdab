"""The narrow phase's unordered FP32 cull, its mirror records and the
sphere-only pass, against the FP64 oracle at list lengths around a warp's
batch of 32 pairs: mixtures of shapes (spheres of two radii, boxes,
polyhedra: supports without transcendental functions, so FP64-strict is bit
exact) and packings of spheres alone."""
import numpy as np
import pytest

from grains3dgpu_b200 import abi, scenes

from conftest import rel_err
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
