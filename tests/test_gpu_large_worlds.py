"""Worlds beyond the sizes the kernels keep in registers, and world counts at the default schedule's
borders, bit for bit against the oracle (parity build)."""

import numpy as np
import pytest
import torch

from newton_custom_contact_b200 import CollisionPipeline, SolverXPBD, _lib, scenes
from newton_custom_contact_b200.schedule import default_mode

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _exact_build():
    with _lib.build("exact"):
        yield


def _substeps(model, info, orc, substeps, schedule=None):
    pipe = CollisionPipeline(model)
    if schedule is not None:
        pipe.set_step_schedule(schedule[1], mode=schedule[0])
    solver = SolverXPBD(model, iterations=4)
    dt = info["dt"] / info["substeps"]
    a, b, contacts = model.state(), model.state(), pipe.contacts()
    q, qd = model.host("body_q").copy(), model.host("body_qd").copy()
    f = np.zeros((model.body_count, 6), np.float32)
    for _ in range(substeps):
        pipe.collide(a, contacts)
        solver.step(a, b, None, contacts, dt)
        a, b = b, a
        segs = orc.collide(model, pipe.layout, q)
        q, qd, _ = orc.step(model, pipe.layout, solver.params(), q, qd, f, segs, dt)
    table = orc.contacts_table(model, pipe.layout, segs)
    n = int(contacts.rigid_contact_count.item())
    assert n == table.shape[0] and n > 0
    for name, cols in (("point0", slice(4, 7)), ("point1", slice(7, 10)), ("normal", slice(10, 13)),
                       ("offset0", slice(13, 16)), ("offset1", slice(16, 19))):
        got = getattr(contacts, f"rigid_contact_{name}")[:n].cpu().numpy()
        assert np.array_equal(got.view(np.uint32), np.asarray(table[:, cols], np.float32).view(np.uint32)), name
    assert np.array_equal(a.body_q.cpu().numpy().view(np.uint32), q.view(np.uint32))
    assert np.array_equal(a.body_qd.cpu().numpy().view(np.uint32), qd.view(np.uint32))


@pytest.mark.parametrize("bodies", [64, 127, 128, 129, 200])
def test_world_sizes(cuda, orc, bodies):
    # 128 bodies: 8256 pairs, one more than the eight chunks a warp keeps; 200: most are tested again
    model, info = scenes.scene_c2(seed=bodies, worlds=2, nmin=bodies, nmax=bodies, device=cuda)
    _substeps(model, info, orc, 2)


@pytest.mark.parametrize("schedule", [("batch", 256), ("groups", 128), ("groups", 64), ("groups_compact", 32)])
def test_full_and_partial_solve_rounds(cuda, orc, schedule):
    # stacks rest on each other: 4 contacts per box, so 16 boxes hold about two rounds of a warp, and the
    # wider groups' rounds stay partial
    model, info = scenes.scene_c5(seed=4, worlds=5, height=16, device=cuda)
    info = dict(info, dt=info["dt"] * info["substeps"])
    _substeps(model, info, orc, 6, schedule)


def test_default_schedule_by_world_count():
    sms = 148
    for worlds, bodies, want in ((1, 64, 256), (296, 128, 256), (297, 128, 128), (592, 32, 128), (593, 32, 64),
                                 (1184, 64, 64), (1185, 64, 32), (1185, 65, 64), (2368, 128, 64), (2369, 128, 32)):
        assert default_mode(bodies, worlds, sms)[1] == want, (worlds, bodies)
    # 32 threads cannot hold 200 bodies: the smallest group that does
    assert default_mode(200, 5000, sms) == ("groups_compact", 64)
    assert default_mode(600, 5000, sms) == ("batch", None)


@pytest.mark.parametrize("grid", [1, 2, 7])
def test_narrow_phase_with_few_ctas(cuda, grid):
    """More queue items than threads: the analytic kernel's ordered tiles and the MPR/GJK kernel's loop give
    the contacts of the default grids, where every item has a thread (or two)."""
    import ctypes as C

    model, info = scenes.scene_c2(seed=21, worlds=24, nmin=8, nmax=90, device=cuda)
    pipe, solver = CollisionPipeline(model), SolverXPBD(model, iterations=4)
    a, b, want, got = model.state(), model.state(), pipe.contacts(), pipe.contacts()
    for _ in range(12 * info["substeps"]):
        pipe.collide(a, want)
        solver.step(a, b, None, want, info["dt"] / info["substeps"])
        a, b = b, a
    pipe.collide(a, want)
    lib, desc, stream = _lib.load(), pipe.desc(), C.c_void_p(_lib.stream_handle(model.device))
    seg, pub = pipe.seg_struct(got), pipe.public_struct(got)
    _lib.check("nb_collide", lib.nb_collide(C.byref(desc), C.c_void_p(a.body_q.data_ptr()), C.byref(seg), grid, stream))
    _lib.check("nb_publish_contacts", lib.nb_publish_contacts(C.byref(desc), C.byref(seg), C.byref(pub), stream))
    n = int(want.rigid_contact_count.item())
    assert n > 128 * grid and int(got.rigid_contact_count.item()) == n and pipe.status(got) == 0
    for k in ("shape0", "shape1", "point0", "point1", "offset0", "offset1", "normal", "margin0", "margin1"):
        x, y = getattr(want, f"rigid_contact_{k}")[:n], getattr(got, f"rigid_contact_{k}")[:n]
        assert torch.equal(x, y), k
