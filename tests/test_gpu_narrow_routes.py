"""The narrow phase's routes by item count (csrc/nb_collide.cu): an item per thread or ordered tiles in the
analytic kernel, items shared by two warps or taken in a loop in the MPR/GJK kernel, and the kernels fitted to
many bodies.  The queues' lengths are read from the device's counters, so that a case cannot miss its route."""

import ctypes as C

import numpy as np
import pytest
import torch

from newton_custom_contact_b200 import CollisionPipeline, SolverXPBD, _lib, scenes

pytestmark = pytest.mark.gpu

THREADS, SHARED = 128, 64  # items per CTA: one per thread, or one per two threads


def _landed(cuda, **scene):
    model, info = scenes.scene_c2(device=cuda, **scene)
    pipe, solver = CollisionPipeline(model), SolverXPBD(model, iterations=4)
    a, b, contacts = model.state(), model.state(), pipe.contacts()
    for _ in range(12 * info["substeps"]):
        pipe.collide(a, contacts)
        solver.step(a, b, None, contacts, info["dt"] / info["substeps"])
        a, b = b, a
    return model, pipe, a, contacts


def _same_as_oracle(model, pipe, a, contacts, orc):
    segs = orc.collide(model, pipe.layout, a.body_q.cpu().numpy())
    table = orc.contacts_table(model, pipe.layout, segs)
    n = int(contacts.rigid_contact_count.item())
    assert n == table.shape[0] and n > 0 and pipe.status(contacts) == 0
    for name, cols in (("point0", slice(4, 7)), ("point1", slice(7, 10)), ("normal", slice(10, 13)),
                       ("offset0", slice(13, 16)), ("offset1", slice(16, 19))):
        got = getattr(contacts, f"rigid_contact_{name}")[:n].cpu().numpy()
        assert np.array_equal(got.view(np.uint32), np.asarray(table[:, cols], np.float32).view(np.uint32)), name


@pytest.mark.parametrize("grid,tiles,loop", [(1, True, True), (3, True, True), (0, False, False)])
def test_items_beyond_the_threads(cuda, orc, grid, tiles, loop):
    model, pipe, a, contacts = _landed(cuda, seed=21, worlds=24, nmin=8, nmax=90)
    lib, stream = _lib.load(), C.c_void_p(_lib.stream_handle(model.device))
    seg, pub, desc = pipe.seg_struct(contacts), pipe.public_struct(contacts), pipe.desc()
    _lib.check("nb_collide", lib.nb_collide(C.byref(desc), C.c_void_p(a.body_q.data_ptr()), C.byref(seg), grid, stream))
    counter = contacts._seg["work_counter"].tolist()
    analytic, gjk = counter[2], counter[5] + counter[6]
    ctas = grid or 4 * torch.cuda.get_device_properties(cuda).multi_processor_count  # at least 4 per SM by default
    assert gjk > 0 and (analytic > ctas * THREADS) == tiles and (gjk > ctas * SHARED) == loop, (analytic, gjk)
    _lib.check("nb_publish_contacts", lib.nb_publish_contacts(C.byref(desc), C.byref(seg), C.byref(pub), stream))
    _same_as_oracle(model, pipe, a, contacts, orc)


def test_kernels_for_many_bodies(cuda, orc):
    bodies = 4 * THREADS * torch.cuda.get_device_properties(cuda).multi_processor_count
    model, pipe, a, contacts = _landed(cuda, seed=5, worlds=bodies // 6 + 1, nmin=6, nmax=6)
    assert model.body_count > bodies
    pipe.collide(a, contacts)
    _same_as_oracle(model, pipe, a, contacts, orc)
