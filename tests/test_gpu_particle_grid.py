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


def _rows(rows, cuda):
    """A model without gravity of (position, radius) rows: mass 0.02, particle_max_radius 0.02 and cohesion
    2 mm, so cells of 42 mm, whatever the rows' radii."""
    b = ModelBuilder(gravity=0.0)
    for p, r in rows:
        b.add_particle(tuple(float(c) for c in p), (0.0, 0.0, 0.0), 0.02, radius=r)
    model = b.finalize(device=cuda)
    model.particle_max_radius = 0.02
    model.particle_cohesion = 0.002
    return model


@pytest.mark.parametrize("pairs", [12, 2100])  # one block's grid, and the three kernels'
def test_neighbour_radius_beyond_the_maximum(cuda, pairs):
    # Each pair lies in one cell, overlapping by 4 mm, with the large particle outside of the small one's
    # reach by particle_max_radius: a candidate of its cell all the same
    rows = []
    for k in range(pairs):
        o = 0.042 * 5.0 * np.array([k % 13, (k // 13) % 13, k // 169])
        rows += [(o + (0.008, 0.021, 0.021), 0.002), (o + (0.036, 0.021, 0.021), 0.03)]
    _compare(_rows(rows, cuda), iterations=2)


def test_own_radius_beyond_the_maximum(cuda):
    # Reach 2.4 cells around a cell's middle: five cells per axis, two rounds of rows, candidates told
    # apart by their cells.  The small particles do not see the large one, so only its own correction is
    # the oracle's.
    rng = np.random.default_rng(2)
    d = rng.normal(size=(24, 3))
    d *= (rng.uniform(0.05, 0.08, 24) / np.linalg.norm(d, axis=1))[:, None]
    d = np.concatenate([d, 0.08 * np.eye(3), -0.08 * np.eye(3)])  # cells 2 and -2
    far = rng.uniform(-0.2, 0.2, (200, 3))
    far = far[np.linalg.norm(far, axis=1) > 0.09]
    model = _rows([((0.021, 0.021, 0.021), 0.08)] + [(0.021 + p, 0.002) for p in d] +
                  [(0.021 + p, 0.0005) for p in far], cuda)
    solver, a, b = SolverXPBD(model, iterations=1), model.state(), model.state()
    solver.step(a, b, contacts=CollisionPipeline(model).contacts(), control=None, dt=1.0 / 240.0)
    q, qd = model.host("particle_q"), model.host("particle_qd")
    none = op.soft_collide(model._host, q, None, 0.01, 0)
    want = op.step(model._host, particles.params(model), q, qd, None, none, 1.0 / 240.0, 1, 0.9, False)[0][0]
    assert solver._particles.status() == 0 and not np.array_equal(want, q[0])
    assert np.array_equal(b.particle_q[0].cpu().numpy().view(np.uint32), want.astype(np.float32).view(np.uint32))


@pytest.mark.parametrize("axis,far", [(0, 1.0e9), (1, 1.0e9), (2, 1.0e9), (0, -1.0e9), (2, -3.0e38)])
def test_cells_beyond_an_int(cuda, axis, far):
    # one coordinate's cell is the largest or smallest int; the particles touch in the other two
    p = np.random.default_rng(6).uniform(-0.06, 0.06, (24, 3))
    p[:, axis] = far
    _compare(_rows([(row, 0.015) for row in p], cuda), iterations=2)


@pytest.mark.parametrize("count", [2047, 2048, 2049, 3071, 3072, 3073])
def test_counts_at_the_border_of_one_block(cuda, count):
    _compare(_cloud(count, 0.5 * 0.026 * count ** (1.0 / 3.0), (0.1, -0.2, 0.3), count, cuda=cuda))


@pytest.mark.parametrize("count", [9, 1000, 5000])
def test_scratch_off_an_eight_byte_boundary(cuda, count):
    model = _cloud(count, 0.5 * 0.026 * count ** (1.0 / 3.0), (0.1, -0.2, 0.3), count, cuda=cuda)
    solver = SolverXPBD(model, iterations=3)
    ps = solver._particles
    buf = torch.full((2 * ps.grid_size + 2,), -7, dtype=torch.int32, device=cuda)
    ps.grid_head = buf[1:-1]
    a, b, contacts = model.state(), model.state(), CollisionPipeline(model).contacts()
    solver.step(a, b, contacts=contacts, control=None, dt=1.0 / 240.0)
    q, qd = model.host("particle_q"), model.host("particle_qd")
    none = op.soft_collide(model._host, q, None, 0.01, 0)
    want = op.step(model._host, particles.params(model), q, qd, None, none, 1.0 / 240.0, 3, 0.9, False)[0]
    act = (model.host("particle_flags") & 1) != 0
    assert np.array_equal(b.particle_q.cpu().numpy()[act].view(np.uint32), want[act].astype(np.float32).view(np.uint32))
    assert int(buf[0]) == -7 and int(buf[-1]) == -7
