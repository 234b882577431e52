"""Work that programs have this framework do, as cases to measure: collide, solve, whole substeps,
gradients, particles and the learned warm start, from one small world to thousands.

A case is a dict of plain values.  ``prepare`` builds what a program holds before the call (model,
pipeline, solver, buffers and the bodies' or particles' state), ``run`` is one pass through the public
entry points, ``exact`` the same result in 64-bit torch where the path has one.

The model and its pipeline are built once per scene and kept, as a program keeps them; the state comes
from the seed: bodies start with velocities of their own and fall for some frames, so that every pass
meets piles with the contacts a running simulation has.  That fall runs on the library's parity build,
whose results do not depend on how the compiler fuses multiply-adds.
"""

import functools
import math
import os

import numpy as np
import torch

import newton_custom_contact_b200 as newton
from newton_custom_contact_b200 import CollisionPipeline, SolverXPBD, _lib, adjoint, scenes
from newton_custom_contact_b200.warmstart import WarmStart, WarmStartNet

MODEL_SEED = 1
DISTINCT_WORLDS = 256   # larger scenes repeat these worlds (with velocities of their own)
DISTINCT_ARMS = 32


def listed():
    return [
        # one world of 64 boxes, the scene a first program writes: ten substeps of one frame, in one call
        dict(name="frame_boxes_1", kind="frame", scene="boxes", worlds=1, nmin=64, nmax=64, frames=20, substeps=10,
             iterations=4, graph=False),
        # the same scene stepped by hand: contacts are read between collide and step (a control loop)
        dict(name="substep_boxes_1", kind="substep", scene="boxes", worlds=1, nmin=64, nmax=64, frames=20,
             iterations=4, broad="explicit"),
        # a few dozen environments, an evaluation run
        dict(name="substep_mixed_37", kind="substep", scene="mixed", worlds=37, nmin=8, nmax=101, frames=22,
             iterations=8, broad="explicit"),
        # a captured frame of a training batch
        dict(name="frame_mixed_1024", kind="frame", scene="mixed", worlds=1024, nmin=8, nmax=128, frames=20,
             substeps=2, iterations=8, graph=True),
        # contact generation of the benchmark's batch, every body in the pile's reach
        dict(name="collide_mixed_4096", kind="collide", scene="mixed", worlds=4096, nmin=8, nmax=128, frames=24,
             broad="explicit"),
        # the solve of the same batch on those contacts
        dict(name="step_mixed_4096", kind="step", scene="mixed", worlds=4096, nmin=8, nmax=128, frames=24,
             iterations=8, force=False),
        # contacts matched to the previous substep's and replayed (sticky), as grasping uses it
        dict(name="match_boxes_300", kind="match", scene="boxes", worlds=300, nmin=64, nmax=64, frames=20,
             mode="sticky"),
        # articulated arms with drives and limits among loose boxes
        dict(name="step_arms_256", kind="arms", worlds=256, frames=12, iterations=8),
        # gradients of a short rollout of box stacks with respect to state and forces
        dict(name="grad_stacks_256", kind="grad", worlds=256, height=16, substeps=4, iterations=8, checkpoint=16),
        # a cloth and a hundred thousand loose particles landing on static shapes
        dict(name="particles_110k", kind="particles", cloth=100, loose=100000, radius=0.01, settle=60, iterations=8),
        # a small cloth with some particles on it
        dict(name="particles_3k", kind="particles", cloth=47, loose=801, radius=0.02, settle=60, iterations=4),
        # the solve with the learned warm start in place of most iterations
        dict(name="warm_mixed_512", kind="warm", scene="mixed", worlds=512, nmin=8, nmax=128, frames=22,
             iterations=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["substep", "substep", "collide", "step", "step", "frame", "match", "arms", "grad", "particles",
                       "particles", "warm"])
    if kind == "arms":
        return dict(kind=kind, worlds=_log_int(rng, 1, 256), frames=rng.randint(4, 14),
                    iterations=rng.choice([2, 4, 8]))
    if kind == "grad":
        return dict(kind=kind, worlds=_log_int(rng, 1, 256), height=rng.randint(3, 16), substeps=rng.randint(1, 4),
                    iterations=rng.choice([2, 4, 8]), checkpoint=rng.choice([1, 4, 16]))
    if kind == "particles":
        return dict(kind=kind, cloth=_log_int(rng, 3, 100), loose=_log_int(rng, 20, 100000),
                    radius=rng.choice([0.01, 0.02]), settle=rng.randint(30, 70), iterations=rng.choice([2, 4, 8]))
    scene = rng.choice(["mixed", "mixed", "boxes"])
    worlds = _log_int(rng, 1, 4096 if scene == "mixed" else 1024)
    hi = rng.randint(13, 128) if scene == "mixed" else 64
    case = dict(kind=kind, scene=scene, worlds=worlds, nmin=min(8, hi) if scene == "mixed" else 64, nmax=hi,
                frames=rng.randint(12, 24))
    if kind == "substep":
        case.update(iterations=rng.choice([2, 4, 8]), broad=rng.choice(["explicit", "explicit", "nxn", "sap"]))
    elif kind == "collide":
        case.update(broad=rng.choice(["explicit", "nxn", "sap"]))
    elif kind == "step":
        case.update(iterations=rng.choice([1, 2, 4, 8]), force=rng.random() < 0.3)
    elif kind == "frame":
        case.update(worlds=min(worlds, 1024), substeps=rng.randint(1, 3), iterations=rng.choice([2, 4, 8]),
                    graph=rng.random() < 0.5)
    elif kind == "match":
        case.update(worlds=min(worlds, 600), mode=rng.choice(["latest", "sticky"]))
    else:
        case.update(worlds=min(worlds, 1024), iterations=rng.choice([1, 2, 3]))
    return case


# ---------------------------------------------------------------- scenes
@functools.lru_cache(maxsize=1)
def _pile(scene, worlds, nmin, nmax, broad):
    """(model, pipeline, dt) of `worlds` piles of free bodies over a ground plane."""
    if scene == "boxes" and worlds == 1:
        model, info = scenes.scene_c1(seed=MODEL_SEED, device="cuda")
    else:
        base = min(worlds, DISTINCT_WORLDS)
        if scene == "boxes":
            host, info = scenes.scene_c1_batch(seed=MODEL_SEED, worlds=base, device="cpu")
        else:
            host, info = scenes.scene_c2(seed=MODEL_SEED, worlds=base, nmin=nmin, nmax=nmax, device="cpu")
        counts = np.bincount(host.host("body_world"), minlength=base)
        start = np.concatenate([[0], np.cumsum(counts)])
        pick = np.arange(worlds) % base
        body = np.concatenate([np.arange(start[w], start[w + 1]) for w in pick])
        model = scenes.assemble_free_bodies(
            np.repeat(np.arange(worlds), counts[pick]), host.host("shape_type")[1:][body],
            host.host("shape_scale")[1:][body], host.host("body_q")[body], host.host("shape_material_mu")[1:][body],
            worlds, device="cuda")
    return model, CollisionPipeline(model, broad_phase=broad), info["dt"] / info["substeps"], info["substeps"]


@functools.lru_cache(maxsize=1)
def _arms(worlds):
    """Arms among boxes: (model, pipeline, dt, substeps, the driven joints' targets)."""
    model, info = scenes.scene_c3(seed=MODEL_SEED, worlds=worlds, device="cuda")
    rev = np.nonzero(model.host("joint_type") == int(newton.JointType.REVOLUTE))[0]
    target = np.zeros(model.joint_dof_count, np.float32)
    target[model.host("joint_qd_start")[rev]] = 0.5 * np.sin(np.asarray(info["phases"]).reshape(-1))
    return model, CollisionPipeline(model), info["dt"] / info["substeps"], info["substeps"], target


@functools.lru_cache(maxsize=1)
def _particles(cloth, loose, radius):
    extent = max(0.3, math.sqrt(loose / 1.0e5) * radius / 0.01)
    model, _ = scenes.scene_particles(seed=MODEL_SEED, cloth=cloth, loose=loose, radius=radius, device="cuda",
                                      loose_extent=extent, loose_height=(0.33, 1.2))
    return model, CollisionPipeline(model), 1.0 / 240.0


def _state(model, seed, sigma):
    """The model's state with normally distributed body velocities."""
    g = torch.Generator(device="cpu").manual_seed(int(seed))
    s = model.state()
    s.body_qd.add_((sigma * torch.randn(s.body_qd.shape, generator=g)).to(s.body_qd.device))
    return s


def _fall(model, pipe, state, dt, substeps, iterations=8, control=None):
    """`state` after `substeps` substeps, on the parity build."""
    with _lib.build("exact"):
        solver, contacts, a, b = SolverXPBD(model, iterations=iterations), pipe.contacts(), state, model.state()
        for _ in range(substeps):
            pipe.collide(a, contacts)
            solver.step(a, b, control, contacts, dt)
            a, b = b, a
        return a


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "particles":
        model, pipe, dt = _particles(case["cloth"], case["loose"], case["radius"])
        a = model.state()
        g = torch.Generator(device="cpu").manual_seed(int(seed))
        a.particle_qd.add_((0.1 * torch.randn(a.particle_qd.shape, generator=g)).cuda())
        a = _fall(model, pipe, a, dt, case["settle"])
        st.update(solver=SolverXPBD(model, iterations=case["iterations"]), b=model.state())
    elif kind == "arms":
        model, pipe, dt, per_frame, target = _arms(case["worlds"])
        control = model.control()
        control.joint_target_pos.copy_(torch.from_numpy(target))
        a = _fall(model, pipe, _state(model, seed, 0.05), dt, case["frames"] * per_frame, control=control)
        st.update(solver=SolverXPBD(model, iterations=case["iterations"]), b=model.state(), control=control)
    elif kind == "grad":
        model, info = scenes.scene_c5(seed=int(seed), worlds=case["worlds"], height=case["height"], device="cuda")
        pipe, dt = CollisionPipeline(model), info["dt"]
        solver = SolverXPBD(model, iterations=case["iterations"])
        a = model.state()
        g = torch.Generator(device="cpu").manual_seed(int(seed) + 1)
        rollout = adjoint.Rollout(pipe, solver, dt, case["checkpoint"])
        st.update(solver=solver, rollout=rollout, f=a.body_f.requires_grad_(), q=a.body_q.requires_grad_(),
                  qd=a.body_qd.requires_grad_(), gq=torch.randn(a.body_q.shape, generator=g).cuda(),
                  gqd=torch.randn(a.body_qd.shape, generator=g).cuda())
    else:
        key = (case["scene"], case["worlds"], case["nmin"], case["nmax"])
        model, pipe, dt, per_frame = _pile(*key, case.get("broad", "explicit"))
        a = _fall(model, pipe, _state(model, seed, 0.3), dt, case["frames"] * per_frame)
        if kind == "match":
            pipe = CollisionPipeline(model, contact_matching=case["mode"])
            st["next"] = _fall(model, pipe, _copy(model, a), dt, 1)
        if kind in ("step", "frame", "substep", "warm"):
            st.update(solver=SolverXPBD(model, iterations=case["iterations"]), b=model.state())
        if kind == "warm":
            net = os.path.join(os.path.dirname(newton.__file__), "data", "warmstart_c2.npz")
            st["solver"].warm_start = WarmStart(WarmStartNet.load(net, device="cuda"), iterations=case["iterations"])
    st.update(model=model, pipe=pipe, dt=dt, a=a)
    if kind == "step" and case["force"]:
        model.request_contact_attributes("force")
        st["contacts"] = pipe.contacts()
        model._requested_contact_attributes.discard("force")  # the model is shared with cases without forces
    elif kind != "grad":
        st["contacts"] = pipe.contacts()
    if kind in ("step", "arms", "warm"):
        pipe.collide(a, st["contacts"])
    if kind == "frame":
        st["x"] = model.state()
        if case["graph"]:
            torch.cuda.synchronize()
            side = torch.cuda.Stream()
            with torch.cuda.stream(side):
                _frame(st)  # loads the library before the capture
            torch.cuda.synchronize()
            st["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(st["graph"]):
                _frame(st)
    torch.cuda.synchronize()
    return st


def _copy(model, state):
    s = model.state()
    s.assign(state)
    return s


def _contacts_of(c):
    return {"count": c.rigid_contact_count, "shape0": c.rigid_contact_shape0, "shape1": c.rigid_contact_shape1,
            "point0": c.rigid_contact_point0, "point1": c.rigid_contact_point1, "offset0": c.rigid_contact_offset0,
            "offset1": c.rigid_contact_offset1, "normal": c.rigid_contact_normal, "margin0": c.rigid_contact_margin0,
            "margin1": c.rigid_contact_margin1}


def _frame(st):
    """A frame from the prepared state: the substeps in one call, or one by one where it is captured."""
    x, y = st["x"], st["b"]
    x.assign(st["a"])
    if not st["case"]["graph"]:
        st["solver"].step_substeps(x, y, st["contacts"], st["dt"], st["case"]["substeps"])
        return y
    for _ in range(st["case"]["substeps"]):
        x.clear_forces()
        st["pipe"].collide(x, st["contacts"])
        st["solver"].step(x, y, None, st["contacts"], st["dt"])
        x, y = y, x
    return x


# ---------------------------------------------------------------- run
def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "collide":
        st["pipe"].collide(st["a"], st["contacts"])
        return _contacts_of(st["contacts"])
    if kind == "match":
        st["pipe"].reset_contact_matching()
        st["pipe"].collide(st["a"], st["contacts"])
        st["pipe"].collide(st["next"], st["contacts"])
        return dict(_contacts_of(st["contacts"]), match=st["contacts"].rigid_contact_match_index)
    if kind in ("step", "arms", "warm"):
        st["solver"].step(st["a"], st["b"], st.get("control"), st["contacts"], st["dt"])
        out = {"q": st["b"].body_q, "qd": st["b"].body_qd}
        if st["contacts"].force is not None:
            st["solver"].update_contacts(st["contacts"], st["b"])
            out["force"] = st["contacts"].force
        return out
    if kind == "substep":
        st["a"].clear_forces()
        st["pipe"].collide(st["a"], st["contacts"])
        st["solver"].step(st["a"], st["b"], None, st["contacts"], st["dt"])
        return dict(_contacts_of(st["contacts"]), q=st["b"].body_q, qd=st["b"].body_qd)
    if kind == "frame":
        if case["graph"]:
            st["graph"].replay()
            last = st["x"] if case["substeps"] % 2 == 0 else st["b"]
        else:
            last = _frame(st)
        return {"q": last.body_q, "qd": last.body_qd}
    if kind == "grad":
        q, qd = adjoint.simulate(st["pipe"], st["solver"], st["q"], st["qd"], st["f"], substeps=case["substeps"],
                                 dt=st["dt"], checkpoint_every=case["checkpoint"], rollout=st["rollout"])
        grads = torch.autograd.grad([q, qd], [st["q"], st["qd"], st["f"]], [st["gq"], st["gqd"]])
        return {"q": q.detach(), "qd": qd.detach(), "grad_q": grads[0], "grad_qd": grads[1], "grad_f": grads[2]}
    st["pipe"].collide(st["a"], st["contacts"])
    st["solver"].step(st["a"], st["b"], None, st["contacts"], st["dt"])
    c = st["contacts"]
    return {"q": st["b"].particle_q, "qd": st["b"].particle_qd, "count": c.soft_contact_count,
            "particle": c.soft_contact_particle, "shape": c.soft_contact_shape, "body_pos": c.soft_contact_body_pos,
            "normal": c.soft_contact_normal}


# ---------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass: inputs read once, outputs written once; the contact counts are
    those of the settled piles (per body about 3 in mixed piles, 5 among boxes)."""
    kind = case["kind"]
    if kind == "particles":
        P = case["cloth"] ** 2 + case["loose"]
        springs, edges = 4 * case["cloth"] ** 2, case["cloth"] ** 2
        per = 4 * 30 + 12 * 40  # soft contacts' tests; about 12 neighbours, 40 operations each
        return {"bytes": P * (36 + 24 + 20) + springs * 24 + edges * 28,
                "flops": case["iterations"] * (P * per + springs * 60 + edges * 250)}
    if kind == "arms":
        B, J = case["worlds"] * 35, case["worlds"] * 7
        it = case["iterations"]
        return {"bytes": B * 224 + 2 * B * 80 + J * 150, "flops": it * (B * 300 + 2 * B * 200 + J * 1500)}
    if kind == "grad":
        B, n, it = case["worlds"] * case["height"], case["substeps"], case["iterations"]
        return {"bytes": B * (19 * 4 + 13 * 4 + 13 * 4 + 19 * 4 + 96),
                "flops": n * B * (it * (3 * (300 + 4 * 400)) + 2 * 5 * 2000)}
    box = case["scene"] == "boxes"
    n = 64.0 if box else 0.5 * (case["nmin"] + case["nmax"])
    B, pairs = case["worlds"] * n, case["worlds"] * (n * n / 2 if box else (n * n + (case["nmax"] - case["nmin"]) ** 2 / 12) / 2)
    C = B * (5.0 if box else 3.0)
    collide = {"bytes": B * (44 + 28) + 4 * pairs + 84 * C, "flops": 6 * pairs + 1000 * C}
    it = case.get("iterations", 0)
    step = {"bytes": B * 224 + C * 80, "flops": B * (300 + 300 * it) + it * C * (60 + 150)}
    if kind == "collide":
        return collide
    if kind == "match":
        return {"bytes": 2 * collide["bytes"] + 2 * C * 60, "flops": 2 * collide["flops"]}
    if kind == "step":
        return {"bytes": step["bytes"] + (24 * C if case["force"] else 0), "flops": step["flops"]}
    if kind == "warm":
        return {"bytes": step["bytes"] + 24 * C, "flops": step["flops"] + 45000 * C}
    k = case.get("substeps", 1)
    return {"bytes": 224 * B + 4 * pairs + (84 * C if kind == "substep" else 0),
            "flops": k * (collide["flops"] + step["flops"])}


# ---------------------------------------------------------------- exact
def _rotate(q, v):
    u, w = q[..., :3], q[..., 3:]
    return v + 2.0 * torch.cross(u, torch.cross(u, v, dim=-1) + w * v, dim=-1)


def _unrotate(q, v):
    return _rotate(torch.cat([-q[..., :3], q[..., 3:]], -1), v)


def _advance(q, w, dt):
    """q + dt / 2 * (w, 0) * q, normalised."""
    u, s = q[..., :3], q[..., 3:]
    d = torch.cat([s * w + torch.cross(w, u, dim=-1), -(w * u).sum(-1, keepdim=True)], -1)
    q = q + 0.5 * dt * d
    return q / q.norm(dim=-1, keepdim=True)


def _mv(m, v):
    return torch.einsum("bij,bj->bi", m, v)


def _unit(v):
    n = v.norm(dim=-1, keepdim=True)
    return torch.where(n > 0, v / n.clamp_min(1e-300), torch.zeros_like(v))


def _rest(v):
    return torch.where(v.norm(dim=-1, keepdim=True) < 1e-4, torch.zeros_like(v), v)


def _exact_step(st):
    """One XPBD substep of free bodies on the prepared contacts, in 64 bits; row B of every body array
    stands for the static world."""
    m, c, dt, it = st["model"], st["contacts"], st["dt"], st["case"]["iterations"]
    B = m.body_count
    d = lambda t, *s: t.double().reshape(-1, *s) if s else t.double()  # noqa: E731
    pad = lambda t: torch.cat([t, torch.zeros_like(t[:1])])  # noqa: E731
    im, I, iI = pad(d(m.body_inv_mass)), pad(d(m.body_inertia, 3, 3)), pad(d(m.body_inv_inertia, 3, 3))
    x, r, v, w = d(st["a"].body_q)[:, :3], d(st["a"].body_q)[:, 3:], d(st["a"].body_qd)[:, :3], d(st["a"].body_qd)[:, 3:]
    # integration (centres of mass at the body origins)
    v = v + d(m.gravity)[m.body_world.clamp_min(0).long()] * dt
    wb = _unrotate(r, w)
    w = _rotate(r, wb + dt * _mv(iI[:B], -torch.cross(wb, _mv(I[:B], wb), dim=-1)))
    x, r = x + v * dt, _advance(r, w, dt)
    n = int(c.rigid_contact_count)
    sa, sb = c.rigid_contact_shape0[:n].long(), c.rigid_contact_shape1[:n].long()
    a, b = (torch.where(k < 0, torch.full_like(k, B), k) for k in (m.shape_body.long()[sa], m.shape_body.long()[sb]))
    mu, mut, mur = (0.5 * (d(t)[sa] + d(t)[sb])[:, None] for t in
                    (m.shape_material_mu, m.shape_material_mu_torsional, m.shape_material_mu_rolling))
    nrm, thick = d(c.rigid_contact_normal[:n]), d(c.rigid_contact_margin0[:n] + 0.0) + d(c.rigid_contact_margin1[:n])
    pa, pb, oa, ob = (d(t[:n]) for t in (c.rigid_contact_point0, c.rigid_contact_point1, c.rigid_contact_offset0,
                                         c.rigid_contact_offset1))
    one = torch.tensor([[0.0, 0.0, 0.0, 1.0]], dtype=torch.float64, device=x.device)

    def lam(err, ja, jb, lin, Ra, Rb, aa, bb):
        """-0.8 err / (dt (J M^-1 J^T)) of one constraint row (angular parts ja, jb; unit linear part or none)."""
        k = lin * (im[aa] + im[bb])[:, None]
        for j, R, i in ((ja, Ra, aa), (jb, Rb, bb)):
            u = _unrotate(R, j)
            k = k + (u * _mv(iI[i], u)).sum(-1, keepdim=True)
        return -0.8 * torch.where(k > 0, err / (dt * k).clamp_min(1e-300), err)

    force = torch.zeros(n, 6, dtype=torch.float64, device=x.device)
    for _ in range(it):
        X, R, W = pad(x), torch.cat([r, one]), pad(w)
        depth = (nrm * (X[b] + _rotate(R[b], pb) - X[a] - _rotate(R[a], pa))).sum(-1) - thick
        on = torch.nonzero((a != b) & (depth < 0))[:, 0]
        A, Bb, N, D = a[on], b[on], nrm[on], depth[on][:, None]
        Ra, Rb = R[A], R[Bb]
        ra, rb = _rotate(Ra, pa[on]), _rotate(Rb, pb[on])
        ja, jb = -torch.cross(ra, N, dim=-1), torch.cross(rb, N, dim=-1)
        ln = lam(D, ja, jb, 1.0, Ra, Rb, A, Bb)
        la, lb, ta, tb = -N * ln, N * ln, ja * ln, jb * ln
        ra, rb = _rotate(Ra, pa[on] + oa[on]), _rotate(Rb, pb[on] + ob[on])
        slip = X[Bb] + rb - X[A] - ra
        slip = slip - (slip * N).sum(-1, keepdim=True) * N
        t, err = _unit(slip), slip.norm(dim=-1, keepdim=True)
        ja, jb = -torch.cross(ra, t, dim=-1), torch.cross(rb, t, dim=-1)
        lf = torch.where((err > 0) & (mu[on] > 0), torch.maximum(lam(err, ja, jb, 1.0, Ra, Rb, A, Bb), -ln * mu[on]),
                         torch.zeros_like(err))
        la, lb, ta, tb = la - t * lf, lb + t * lf, ta + ja * lf, tb + jb * lf
        om = W[Bb] - W[A]
        e = (om * N).sum(-1, keepdim=True) * dt
        cap = ln * mut[on]
        lt = torch.where(e != 0, torch.minimum(torch.maximum(lam(e, -N, N, 0.0, Ra, Rb, A, Bb), -cap), cap),
                         torch.zeros_like(e))
        ta, tb = ta - N * lt, tb + N * lt
        om = om - (om * N).sum(-1, keepdim=True) * N
        e, u = om.norm(dim=-1, keepdim=True) * dt, _unit(om)
        lr = torch.where(e > 0, torch.maximum(lam(e, -u, u, 0.0, Ra, Rb, A, Bb), -ln * mur[on]), torch.zeros_like(e))
        ta, tb = ta - u * lr, tb + u * lr
        lin, ang = torch.zeros_like(X), torch.zeros_like(X)
        lin.index_add_(0, A, la).index_add_(0, Bb, lb)
        ang.index_add_(0, A, ta).index_add_(0, Bb, tb)
        cnt = torch.zeros(B + 1, dtype=torch.float64, device=x.device)
        cnt.index_add_(0, A, torch.ones_like(cnt[A])).index_add_(0, Bb, torch.ones_like(cnt[Bb]))
        cnt[B] = 0.0
        ca, cb = cnt[A], cnt[Bb]
        wt = torch.where(ca == 0, 1.0 / cb, torch.where(cb == 0, 1.0 / ca, 2.0 / (ca + cb)))[:, None]
        force[on] += wt * torch.cat([la, ta], -1)
        k = 1.0 / cnt[:B, None].clamp_min(1.0)
        dv = lin[:B] * im[:B, None] * k
        wb, dwb = _unrotate(r, w), _mv(iI[:B], _unrotate(r, ang[:B] * k))
        tq = torch.cross(dwb, _mv(I[:B], wb + dwb), dim=-1) + torch.cross(wb, _mv(I[:B], dwb), dim=-1)
        dw = _rotate(r, dwb - dt * _mv(iI[:B], tq))
        x, r, v, w = x + dv * dt, _advance(r, dw, dt), _rest(v + dv), _rest(w + dw)
    out = {"q": torch.cat([x, r], -1), "qd": torch.cat([v, w], -1)}
    if c.force is not None:
        out["force"] = torch.zeros(c.force.shape, dtype=torch.float64, device=x.device)
        out["force"][:n] = force / dt
    return out


def _pairs_within(x, reach, h):
    """(i, j), i != j, of points at most about `reach` <= h apart, by cells of size h."""
    cell = torch.floor(x / h).long()
    cell = cell - cell.min(0).values + 1
    dim = cell.max(0).values + 2
    key = (cell[:, 0] * dim[1] + cell[:, 1]) * dim[2] + cell[:, 2]
    key, order = torch.sort(key)
    found = []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                want = key + (dx * dim[1] + dy) * dim[2] + dz
                lo, hi = torch.searchsorted(key, want), torch.searchsorted(key, want, right=True)
                i = torch.repeat_interleave(torch.arange(len(x), device=x.device), hi - lo)
                j = torch.arange(len(i), device=x.device) - torch.repeat_interleave((hi - lo).cumsum(0) - (hi - lo), hi - lo) + lo[i]
                i, j = order[i], order[j]
                near = (i != j) & ((x[i] - x[j]).norm(dim=-1) <= reach[i] + reach[j])
                found.append((i[near], j[near]))
    return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])


def _exact_particles(st):
    """The particle substep in 64 bits: soft contacts as the path's own collide lists them (points and
    normals of static shapes), neighbours, springs and bending edges."""
    m, s, dt = st["model"], st["a"], st["dt"]
    st["pipe"].collide(s, st["contacts"])
    c = st["contacts"]
    n = int(c.soft_contact_count)
    d = lambda t: t.double()  # noqa: E731
    act = ((m.particle_flags & 1) != 0)[:, None]
    im, rad = d(m.particle_inv_mass)[:, None], d(m.particle_radius)
    x0, v = d(s.particle_q), d(s.particle_qd)
    v0 = v
    v = v + dt * d(m.gravity)[0] * (im > 0)
    x = torch.where(act, x0 + v * dt, x0)
    v = torch.where(act, v, v0)
    cp, pos, nrm = c.soft_contact_particle[:n].long(), d(c.soft_contact_body_pos[:n]), d(c.soft_contact_normal[:n])
    cmu = 0.5 * (m.soft_contact_mu + d(m.shape_material_mu)[c.soft_contact_shape[:n].long()])[:, None]
    sp = m.spring_indices.long().reshape(-1, 2)
    ke, kd, rest = d(m.spring_stiffness)[:, None], d(m.spring_damping)[:, None], d(m.spring_rest_length)[:, None]
    ed, ep = m.edge_indices.long(), d(m.edge_bending_properties)

    def friction(mu, lam, vt):
        return _unit(vt) * torch.maximum(mu * lam, -vt.norm(dim=-1, keepdim=True) * dt)

    for _ in range(st["case"]["iterations"]):
        delta = torch.zeros_like(x)
        pen = (nrm * (x[cp] - pos)).sum(-1, keepdim=True) - rad[cp][:, None]
        wc, vc = im[cp], v[cp]
        vt = vc - nrm * (nrm * vc).sum(-1, keepdim=True)
        on = (pen <= m.particle_adhesion) & (wc > 0)
        soft = (friction(cmu, pen, vt) - nrm * pen) * 0.9  # inverse mass over itself
        delta.index_add_(0, cp, torch.where(on, soft, torch.zeros_like(soft)))
        reach = rad + 0.5 * m.particle_cohesion
        ids = torch.nonzero(act[:, 0])[:, 0]
        i, j = _pairs_within(x[ids], reach[ids], 2.0 * float(reach.max()))
        i, j = ids[i], ids[j]
        dx = x[i] - x[j]
        dist = dx.norm(dim=-1, keepdim=True)
        err, wsum, nn = dist - rad[i][:, None] - rad[j][:, None], im[i] + im[j], dx / dist
        vr = v[i] - v[j]
        vt = vr - nn * (nn * vr).sum(-1, keepdim=True)
        f = (friction(m.particle_mu, err, vt) - nn * err) / wsum.clamp_min(1e-300) * im[i] * 0.9
        delta.index_add_(0, i, torch.where(wsum > 0, f, torch.zeros_like(f)))
        dx, dv = x[sp[:, 0]] - x[sp[:, 1]], v[sp[:, 0]] - v[sp[:, 1]]
        ln = dx.norm(dim=-1, keepdim=True)
        nn, al, ga = dx / ln, 1.0 / (ke * dt * dt), kd / (ke * dt)
        wa, wb = im[sp[:, 0]], im[sp[:, 1]]
        lam = -(ln - rest + ga * dt * (nn * dv).sum(-1, keepdim=True)) / ((1.0 + ga) * (wa + wb) + al)
        delta.index_add_(0, sp[:, 0], nn * wa * lam).index_add_(0, sp[:, 1], -nn * wb * lam)
        x1, x2, x3, x4 = (x[ed[:, k]] for k in range(4))
        n1, n2, e = torch.cross(x3 - x1, x4 - x1, dim=-1), torch.cross(x4 - x2, x3 - x2, dim=-1), x4 - x3
        el = e.norm(dim=-1, keepdim=True)
        n1, n2, e = _unit(n1), _unit(n2), e / el
        dot = lambda p, q: (p * q).sum(-1, keepdim=True)  # noqa: E731
        ang = torch.atan2(dot(torch.cross(n1, n2, dim=-1), e), dot(n1, n2)) - d(m.edge_rest_angle)[:, None]
        grads = [-n1 * el, -n2 * el, -n1 * dot(x1 - x4, e) - n2 * dot(x2 - x4, e),
                 -n1 * dot(x3 - x1, e) - n2 * dot(x3 - x2, e)]
        den = sum(im[ed[:, k]] * dot(g, g) for k, g in enumerate(grads))
        al, ga = 1.0 / (ep[:, :1] * dt * dt), ep[:, 1:] / (ep[:, :1] * dt)
        gv = dt * sum(dot(g, v[ed[:, k]]) for k, g in enumerate(grads))
        lam = -(ang + ga * gv) / ((1.0 + ga) * den + al)
        for k, g in enumerate(grads):
            delta.index_add_(0, ed[:, k], g * im[ed[:, k]] * lam)
        x = torch.where(act, x + delta, x)
        v = torch.where(act, (x - x0) / dt, v)
    return {"q": x, "qd": v, "count": None, "particle": None, "shape": None, "body_pos": None, "normal": None}


def exact(case, seed):
    """64-bit results of the substeps that have them: the solve on given contacts and the particle
    substep.  Contact generation and rollouts pick features by tests that another precision decides
    otherwise."""
    if case["kind"] == "step":
        return _exact_step(prepare(case, seed))
    if case["kind"] == "particles":
        return _exact_particles(prepare(case, seed))
    return None
