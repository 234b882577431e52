"""Publishing by a warp and by a CTA per world (csrc/nb_collide.cu publish_by_warps): the public rows and the
solver records, bit for bit against the oracle (parity build), and a capacity below the contact count."""

import numpy as np
import pytest
import torch

from newton_custom_contact_b200 import CollisionPipeline, SolverXPBD, scenes
from newton_custom_contact_b200._abi import NB_STATUS_CONTACT_OVERFLOW

pytestmark = pytest.mark.gpu

ROWS = ("shape0", "shape1", "point0", "point1", "normal", "offset0", "offset1", "margin0", "margin1")


def _landed(worlds, lo, hi, cuda, frames=10):
    model, info = scenes.scene_c2(seed=worlds, worlds=worlds, nmin=lo, nmax=hi, device=cuda)
    pipe, solver = CollisionPipeline(model), SolverXPBD(model, iterations=4)
    dt = info["dt"] / info["substeps"]
    a, b, contacts = model.state(), model.state(), pipe.contacts()
    for _ in range(frames * info["substeps"]):
        pipe.collide(a, contacts)
        solver.step(a, b, None, contacts, dt)
        a, b = b, a
    pipe.collide(a, contacts)
    return model, pipe, solver, a, contacts, dt


# worlds, bodies: up to 32 pairs per world (one round of a warp), a CTA, a warp's rounds past one and two
# waves of CTAs, and worlds of 5,000 pairs on average
@pytest.mark.parametrize("worlds,lo,hi", [(1, 1, 1), (7, 2, 6), (300, 2, 6), (300, 8, 24), (1300, 8, 20), (2400, 24, 26),
                                          (3, 90, 110)])
def test_contacts_and_records(cuda, orc, worlds, lo, hi):
    model, pipe, solver, a, contacts, dt = _landed(worlds, lo, hi, cuda)
    q, qd = a.body_q.cpu().numpy(), a.body_qd.cpu().numpy()
    segs = orc.collide(model, pipe.layout, q)
    table = orc.contacts_table(model, pipe.layout, segs)
    n = int(contacts.rigid_contact_count.item())
    assert n == table.shape[0] and (n > 0 or worlds == 1) and pipe.status(contacts) == 0
    for name, cols in (("point0", slice(4, 7)), ("point1", slice(7, 10)), ("normal", slice(10, 13)),
                       ("offset0", slice(13, 16)), ("offset1", slice(16, 19))):
        got = getattr(contacts, f"rigid_contact_{name}")[:n].cpu().numpy()
        assert np.array_equal(got.view(np.uint32), np.asarray(table[:, cols], np.float32).view(np.uint32)), name
    out = model.state()
    solver.step(a, out, None, contacts, dt)
    f = np.zeros((model.body_count, 6), np.float32)
    q, qd, _ = orc.step(model, pipe.layout, solver.params(), q, qd, f, segs, dt)
    assert np.array_equal(out.body_q.cpu().numpy().view(np.uint32), q.view(np.uint32))
    assert np.array_equal(out.body_qd.cpu().numpy().view(np.uint32), qd.view(np.uint32))


@pytest.mark.parametrize("worlds,lo,hi", [(400, 2, 6), (1300, 8, 20)])
def test_capacity_below_the_count(cuda, worlds, lo, hi):
    model, _, _, a, full, _ = _landed(worlds, lo, hi, cuda)
    n = int(full.rigid_contact_count.item())
    cap = n // 2 + 1
    pipe = CollisionPipeline(model, rigid_contact_max=cap)
    small = pipe.contacts()
    pipe.collide(a, small)
    assert int(small.rigid_contact_count.item()) == n and pipe.status(small) & NB_STATUS_CONTACT_OVERFLOW
    for name in ROWS:
        assert torch.equal(getattr(small, f"rigid_contact_{name}"), getattr(full, f"rigid_contact_{name}")[:cap])
    assert torch.equal(small._seg["rec"], full._seg["rec"][:cap])
