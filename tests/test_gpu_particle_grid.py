"""The particle neighbour search's two forms (csrc/nb_particles.cu: entries in bucket order, linked lists)
against the numpy oracle, bit for bit in the parity build: particle counts at the edges of the bucket
counts, rows that wrap around the table, particles far from the origin, and scratch too small for the
sorted form."""

import numpy as np
import pytest
import torch

from newton_custom_contact_b200 import CollisionPipeline, ModelBuilder, SolverXPBD, _lib, particles
from oracle import oracle_particles as op

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _exact_build():
    with _lib.build("exact"):
        yield


def _cloud(count, spread, offset, seed, radii=(0.01, 0.02), cuda=None):
    rng = np.random.default_rng(seed)
    b = ModelBuilder()
    for k in range(count):
        p = np.asarray(offset) + rng.uniform(-spread, spread, 3)
        b.add_particle(tuple(p), tuple(rng.normal(0.0, 0.2, 3)), float(rng.uniform(0.01, 0.05)),
                       radius=float(rng.uniform(*radii)), flags=0 if k % 11 == 5 else 1)
    model = b.finalize(device=cuda)
    model.particle_cohesion = 0.002
    return model


def _compare(model, grid_size=None, iterations=3, dt=1.0 / 240.0):
    solver = SolverXPBD(model, iterations=iterations)
    ps = solver._particles
    if grid_size is not None:
        ps.grid_size = grid_size
        ps.grid_head = torch.full((2 * grid_size,), -1, dtype=torch.int32, device=model.device)
    a, b = model.state(), model.state()
    contacts = CollisionPipeline(model).contacts()
    q, qd = model.host("particle_q").copy(), model.host("particle_qd").copy()
    none = op.soft_collide(model._host, q, None, 0.01, 0)
    for _ in range(2):
        solver.step(a, b, contacts=contacts, control=None, dt=dt)
        a, b = b, a
        q, qd = op.step(model._host, particles.params(model), q, qd, None, none, dt, iterations, 0.9, False)
    assert ps.status() == 0
    act = (model.host("particle_flags") & 1) != 0
    for got, want in ((a.particle_q, q), (a.particle_qd, qd)):
        got = got.cpu().numpy()[act].view(np.uint32)
        assert np.array_equal(got, np.ascontiguousarray(want[act], np.float32).view(np.uint32))


@pytest.mark.parametrize("count", [2, 7, 8, 9, 31, 64, 1023, 1024, 1025, 2500, 4096, 4097])
def test_counts_at_the_bucket_edges(cuda, count):
    # about 4 particles per cell of 42 mm
    _compare(_cloud(count, 0.5 * 0.026 * count ** (1.0 / 3.0), (0.1, -0.2, 0.3), count, cuda=cuda))


@pytest.mark.parametrize("offset", [(-3.3, 81.0, 5.0), (0.0, 0.0, -250.0)])
def test_far_from_the_origin(cuda, offset):
    _compare(_cloud(400, 0.1, offset, 3, cuda=cuda))


def test_one_large_among_small_particles(cuda):
    # the cells have the large particle's size: long candidate lists, most of them out of reach
    model = _cloud(1200, 0.12, (0.0, 0.0, 0.0), 5, radii=(0.002, 0.004), cuda=cuda)
    h = model.host("particle_radius")
    h[7] = 0.03
    model.particle_radius.copy_(torch.from_numpy(h))
    model.particle_max_radius = 0.03
    h_q = model.host("particle_q")
    h_q[7] = (0.5, 0.5, 0.5)  # away from the cloud: its own contacts would exceed the neighbour limit
    model.particle_q.copy_(torch.from_numpy(h_q))
    _compare(model)


@pytest.mark.parametrize("grid_size", [64, 1024, 2048, 4096])
def test_small_scratch_takes_the_lists(cuda, grid_size):
    # 900 particles: sorted from 2048 (ranges and entries fit), linked lists below
    _compare(_cloud(900, 0.13, (0.0, 0.0, 0.0), 9, cuda=cuda), grid_size=grid_size)


@pytest.mark.parametrize("count", [900, 2300, 4500])
def test_many_candidates_within_reach(cuda, count):
    # small particles beside one large one: dozens to hundreds of candidates of a particle pass the packed distance,
    # so the list of candidates fills and is tested several times, at every phase of its rounds
    model = _cloud(count, 0.09, (0.02, -0.03, 0.05), count, radii=(0.001, 0.0025), cuda=cuda)
    h, h_q = model.host("particle_radius"), model.host("particle_q")
    h[7] = 0.05
    h_q[7] = (0.7, 0.7, 0.7)  # away from the cloud: its own contacts would exceed the neighbour limit
    model.particle_radius.copy_(torch.from_numpy(h))
    model.particle_q.copy_(torch.from_numpy(h_q))
    model.particle_max_radius = 0.05
    reach = h[0] + model.particle_max_radius + model.particle_cohesion
    near = np.linalg.norm(h_q[:, None] - h_q[None, :200], axis=2) < reach
    assert near.sum(axis=0).max() > 64
    _compare(model)
