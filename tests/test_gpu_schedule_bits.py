"""The step's schedules against each other and the default schedule at its borders.

Product build: a plain step gives the same bits on every schedule (with per-contact forces, with restitution and
with joints too), so that the default rule, which goes by world count, does not show in results.  Parity build:
world counts on both sides of the rule's borders, bit for bit against the oracle.
"""

import numpy as np
import pytest
import torch

from newton_custom_contact_b200 import CollisionPipeline, SolverXPBD, scenes
from newton_custom_contact_b200.schedule import candidate_schedules, default_mode

pytestmark = pytest.mark.gpu


def _scene(name, cuda):
    if name == "arms":
        return scenes.scene_c3(seed=3, worlds=9, device=cuda)
    return scenes.scene_c2(seed=2, worlds=40, nmin=8, nmax=70, device=cuda)


@pytest.mark.product_build
@pytest.mark.parametrize("name", ["mixed", "forces", "restitution", "arms"])
def test_product_build_same_bits_on_every_schedule(cuda, name):
    model, info = _scene(name, cuda)
    if name == "forces":
        model.request_contact_attributes("force")
    pipe = CollisionPipeline(model)
    solver = SolverXPBD(model, iterations=6, enable_restitution=name == "restitution")
    dt = info["dt"] / info["substeps"]
    a, b, contacts = model.state(), model.state(), pipe.contacts()
    for _ in range(12 * info["substeps"]):
        pipe.collide(a, contacts)
        solver.step(a, b, None, contacts, dt)
        a, b = b, a
    pipe.collide(a, contacts)
    assert int(contacts.rigid_contact_count.item()) > model.body_count // 2
    want = None
    for mode, group in candidate_schedules(model):
        pipe.set_step_schedule(group, mode=mode)
        solver.step(a, b, None, contacts, dt)
        got = [b.body_q.clone(), b.body_qd.clone()]
        if name == "forces":
            solver.update_contacts(contacts)
            got.append(contacts.force.clone())
        want = want or got
        assert all(torch.equal(x, y) for x, y in zip(got, want)), (mode, group)


@pytest.mark.parametrize("past", [0, 1])
@pytest.mark.parametrize("waves", [2, 4, 8, 16])
def test_world_counts_at_the_rules_borders(cuda, orc, waves, past):
    worlds = waves * torch.cuda.get_device_properties(cuda).multi_processor_count + past
    model, info = scenes.scene_c2(seed=waves, worlds=worlds, nmin=1, nmax=9, device=cuda)
    group = {2: (256, 128), 4: (128, 64), 8: (64, 32), 16: (32, 32)}[waves][past]
    assert default_mode(model.max_world_bodies, worlds)[1] == group
    pipe, solver = CollisionPipeline(model), SolverXPBD(model, iterations=4)
    dt = info["dt"] / info["substeps"]
    a, b, contacts = model.state(), model.state(), pipe.contacts()
    for _ in range(10 * info["substeps"]):
        pipe.collide(a, contacts)
        solver.step(a, b, None, contacts, dt)
        a, b = b, a
    pipe.collide(a, contacts)
    q, qd = a.body_q.cpu().numpy(), a.body_qd.cpu().numpy()
    segs = orc.collide(model, pipe.layout, q)
    assert int(contacts.rigid_contact_count.item()) == int(segs.world_count.sum()) > worlds
    solver.step(a, b, None, contacts, dt)
    assert pipe._schedule.group_threads == group
    f = np.zeros((model.body_count, 6), np.float32)
    q, qd, _ = orc.step(model, pipe.layout, solver.params(), q, qd, f, segs, dt)
    assert np.array_equal(b.body_q.cpu().numpy().view(np.uint32), q.view(np.uint32))
    assert np.array_equal(b.body_qd.cpu().numpy().view(np.uint32), qd.view(np.uint32))
