"""Failure detection on the GPU, with no GPU fault: every wait in the
engine's kernels is bounded and reports a status, and bad input is reported
by the host call.

* The one-pass scans wait for their predecessor tiles' sums (a decoupled
  look-back) for at most GB_DEBUG_SCAN_SPIN_LIMIT polls (2^20 by default).
  With the limit at 0 the wait runs out as soon as a predecessor is still
  working; the step then reports GB_E_CUDA, every later kernel of the step
  returns at entry (no kernel uses the stalled scan's offsets), the state is
  the one before the step, and a context made without the knob steps on.
* A non-finite particle state is reported as GB_E_NONFINITE and a centre
  outside the linked-cell grid as GB_E_OUT_OF_DOMAIN (host-injected).
"""
import numpy as np
import pytest

from grains3dgpu_b200 import abi, scenes

from test_gpu_cull import packing

pytestmark = pytest.mark.gpu


def test_scan_wait_that_runs_out_is_reported(gb, monkeypatch):
    scene = scenes.polydisperse_superquadrics(n=1_000_000)  # ~500 tiles per scan
    monkeypatch.setenv("GB_DEBUG_SCAN_SPIN_LIMIT", "0")
    s = scenes.System(gb, scene, precision=abi.GB_MIXED)
    monkeypatch.delenv("GB_DEBUG_SCAN_SPIN_LIMIT")
    tr0, kin0 = s.transforms(), s.velocities()
    statuses = [gb.step(s.ctx, 1) for _ in range(3)]
    assert abi.GB_E_CUDA in statuses, statuses
    assert all(st in (abi.GB_OK, abi.GB_E_CUDA) for st in statuses)
    if all(st == abi.GB_E_CUDA for st in statuses):
        assert np.array_equal(s.transforms(), tr0) and np.array_equal(s.velocities(), kin0)
    s.close()
    fresh = scenes.System(gb, scene, precision=abi.GB_MIXED)
    assert gb.step(fresh.ctx, 2) == abi.GB_OK
    assert np.isfinite(fresh.transforms()).all()
    fresh.close()


def test_nonfinite_state_is_reported(gb):
    scene = scenes.superquadric_column(n=1500, pitch=2.05e-3)
    for prec in (abi.GB_MIXED, abi.GB_FP64):
        s = scenes.System(gb, scene, precision=prec)
        tr = scene.transforms.copy()
        tr[17, 10] = np.nan
        s.set_transforms(tr)
        assert gb.detect_collision_and_compute_contact_forces(s.ctx, None) == abi.GB_E_NONFINITE
        kin = scene.velocities.copy()
        kin[3, 0] = np.inf
        s.set_transforms(scene.transforms)
        s.set_velocities(kin)
        assert gb.step(s.ctx, 1) == abi.GB_E_NONFINITE
        s.close()


def test_out_of_domain_is_reported(gb):
    scene = scenes.superquadric_column(n=1500, pitch=2.05e-3)
    s = scenes.System(gb, scene, precision=abi.GB_FP64)
    tr = scene.transforms.copy()
    tr[5, 9] = -0.5  # half a metre outside the box
    s.set_transforms(tr)
    assert gb.detect_collision_and_compute_contact_forces(s.ctx, None) == abi.GB_E_OUT_OF_DOMAIN
    assert gb.step(s.ctx, 1) == abi.GB_E_OUT_OF_DOMAIN
    s.set_transforms(scene.transforms)
    assert gb.step(s.ctx, 1) == abi.GB_OK
    s.close()


def _rb_pointer(rbs):
    return rbs.ctypes.data_as(abi.C.POINTER(abi.RigidBodyDesc))


def _refused_tables(rbs, nmat):
    """Tables of as many bodies that gb_set_rigid_bodies refuses, each for a
    body after ones of other types than the scene's, or for its grid."""
    n = len(rbs)

    def table(kinds, last=None, **fields):
        t = rbs.copy()
        t["type"] = kinds
        t["p"] = 1e-3
        t["n_vertices"] = t["first_vertex"] = 0
        if last is not None:
            t["type"][-1] = last
        for k, v in fields.items():
            t[k][-1] = v
        return t

    tiny = table(abi.GB_SPHERE)
    tiny["p"] = 1e-13  # more linked cells than the grid can have
    for first in (abi.GB_SPHERE, abi.GB_BOX):
        yield table(first, material=nmat), abi.GB_E_INVALID_ARG
        yield table(first, last=abi.GB_CONE), abi.GB_E_UNSUPPORTED
        yield (table(first, last=abi.GB_POLYHEDRON, n_vertices=8, first_vertex=10 ** 6),
               abi.GB_E_INVALID_ARG)
    assert n > 1
    yield tiny, abi.GB_E_INVALID_ARG


@pytest.mark.parametrize("precision", [abi.GB_FP64_STRICT, abi.GB_MIXED])
@pytest.mark.parametrize("bodies", [(0, 1), (2, 3), (0, 2)])
def test_refused_bodies_leave_the_context_as_it_was(gb, bodies, precision):
    """A refused gb_set_rigid_bodies changes nothing: the steps after it are
    those of a context that never saw the call, whatever shapes the refused
    table held."""
    scene = packing(150, bodies)
    seen = scenes.System(gb, scene, precision=precision)
    twin = scenes.System(gb, scene, precision=precision)
    for s in (seen, twin):
        s.step(2)
    verts = np.ascontiguousarray(scene.vertices, dtype=np.float64)
    for rbs, status in _refused_tables(scene.rbs, scene.config["n_materials"]):
        assert gb.set_rigid_bodies(seen.ctx, _rb_pointer(rbs),
                                   abi.dptr(verts) if verts.size else None,
                                   verts.shape[0]) == status
        assert bytes(seen.rb_props(1)) == bytes(twin.rb_props(1))
        for s in (seen, twin):
            s.step(2)
        assert np.array_equal(seen.transforms(), twin.transforms())
        assert np.array_equal(seen.velocities(), twin.velocities())
        a, b = seen.stats(), twin.stats()
        assert (a.cell_size, a.n_cells, a.contacts) == (b.cell_size, b.n_cells, b.contacts)


def test_refused_obstacles_leave_the_context_as_it_was(gb):
    """After refused obstacles (shrunk pegs elsewhere, the last one of an
    unknown material), bodies set again -- which makes the obstacle bins
    anew -- meet the obstacles of a context that never saw the call."""
    scene = scenes.peg_board()
    seen, twin = (scenes.System(gb, scene, precision=abi.GB_FP64) for _ in range(2))
    obs = np.ascontiguousarray(scene.obstacles).copy()
    obs["p"] *= 0.1
    obs["material"][-1] = scene.config["n_materials"]
    tr = np.ascontiguousarray(scene.obstacle_transforms, dtype=np.float64) + 0.01
    assert gb.set_obstacles(seen.ctx, _rb_pointer(obs), abi.dptr(tr)) == abi.GB_E_INVALID_ARG
    rbs = np.ascontiguousarray(scene.rbs)
    for s in (seen, twin):
        assert gb.set_rigid_bodies(s.ctx, _rb_pointer(rbs), None, 0) == abi.GB_OK
        s.step(2)
    assert seen.stats().obstacle_contacts == twin.stats().obstacle_contacts > 100
    assert np.array_equal(seen.transforms(), twin.transforms())


def test_refused_contact_models_leave_the_context_as_it_was(gb):
    """The adjoint reads the laws' host copy: after refused laws (other
    stiffnesses, a negative one last) its gradients are those of a context
    that never saw the call."""
    import torch
    scene = scenes.sphere_bed()
    n, nl = scene.n, len(scene.contact_models)
    adj = torch.ones((9, n), dtype=torch.float64, device="cuda")
    out = []
    for refused in (False, True):
        s = scenes.System(gb, scene, precision=abi.GB_FP64)
        if refused:
            laws = [dict(m, kn=2.0 * m["kn"]) for m in scene.contact_models]
            laws[-1]["kn"] = -1.0
            assert gb.set_contact_models(s.ctx, abi.contact_model_array(laws)) \
                == abi.GB_E_INVALID_ARG
        prev = torch.empty_like(adj)
        grad = torch.zeros(4 * nl, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        ptr = [abi.C.cast(abi.C.c_void_p(t.data_ptr()), abi._D) for t in (adj, prev, grad)]
        assert gb.adjoint_step(s.ctx, *ptr) == abi.GB_OK
        out.append((prev.cpu().numpy(), grad.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert np.abs(out[0][1]).max() > 0.0


@pytest.mark.parametrize("law,fails", [(abi.GB_LAW_HOOKE, "work"),
                                       (abi.GB_LAW_HOOKE_HISTORY, "work"),
                                       (abi.GB_LAW_HOOKE_HISTORY, "list")])
def test_growth_without_memory_is_reported(gb, law, fails):
    """A contact set too large for the device (a header that claims so; nothing
    past it is read) makes the pair arrays' growth fail.  The call says so, no
    array of the failed growth is read, and the steps after it, springs of
    the history law included, are those of a context that never saw it."""
    import torch
    scene = packing(150, (0, 1))
    kw = dict(precision=abi.GB_FP64_STRICT, contact_law=law,
              flags=abi.GB_FLAG_RECORD_CONTACT_INFO)
    seen, twin = (scenes.System(gb, scene, **kw) for _ in range(2))
    for s in (seen, twin):
        s.step(3)
    before = seen.dump(abi.GB_DUMP_CONTACT_PAIRS)
    # bytes per record of the list (58 with the springs) and of the other
    # arrays (144 with the contact information), half as many records again
    total = torch.cuda.get_device_properties(0).total_memory
    pairs = int(1.25 * total / (1.5 * (58 if fails == "list" else 144)))
    buf = torch.zeros(4096, dtype=torch.int64, device="cuda")
    buf[0], buf[1] = scene.n, pairs
    torch.cuda.synchronize()
    assert gb.load_contacts(seen.ctx, buf.data_ptr()) == abi.GB_E_OUT_OF_MEMORY
    if fails == "list":
        assert np.array_equal(seen.dump(abi.GB_DUMP_CONTACT_PAIRS), before)
    else:
        count = abi.C.c_int64(0)
        assert gb.debug_dump(seen.ctx, abi.GB_DUMP_CONTACT_PAIRS, None, 0,
                             abi.C.byref(count)) == abi.GB_E_NOT_READY
    for s in (seen, twin):
        assert s.step(3) == abi.GB_OK
    assert np.array_equal(seen.dump(abi.GB_DUMP_CONTACT_INFO), twin.dump(abi.GB_DUMP_CONTACT_INFO))
    assert np.array_equal(seen.transforms(), twin.transforms())
    assert np.array_equal(seen.velocities(), twin.velocities())


def test_springs_survive_growth(gb):
    """The pair arrays grow in a step whose history holds springs: most grains
    are far apart at first and come into one packing afterwards, so that the
    candidates pass the capacity while earlier contacts last.  The trajectory
    is that of a context that never grew, and not that of one without the
    springs."""
    scene = packing(400, (0, 1))
    dense = scene.transforms.copy()
    top = scene.config["max_coordinate"][2]
    scene.config["max_coordinate"] = (*scene.config["max_coordinate"][:2], 1.0)
    tr = scene.obstacle_transforms
    tr[np.isclose(tr[:, 11], top), 11] = 1.0
    apart = dense.copy()
    up = np.argsort(dense[:, 11], kind="stable")[100:]
    apart[up, 11] = 0.03 + 3e-3 * np.arange(len(up))
    scene.transforms = apart
    ends = []
    for capacity, history in ((1, True), (100_000, True), (100_000, False)):
        s = scenes.System(gb, scene, precision=abi.GB_FP64_STRICT, pair_capacity=capacity,
                          contact_law=abi.GB_LAW_HOOKE_HISTORY)
        s.step(5)
        assert 0 < s.stats().contacts <= s.stats().candidate_pairs < 1024
        kin = s.velocities()
        lower = s.transforms()
        if not history:
            s = scenes.System(gb, scene, precision=abi.GB_FP64_STRICT,
                              contact_law=abi.GB_LAW_HOOKE_HISTORY)
            s.set_velocities(kin)
        lower[up] = dense[up]
        s.set_transforms(lower)
        s.step(3)
        assert s.stats().candidate_pairs > 1024
        ends.append((s.transforms(), s.velocities()))
    assert all(np.array_equal(a, b) for a, b in zip(ends[0], ends[1]))
    assert not np.array_equal(ends[1][1], ends[2][1])
