"""The framework's work, as its users have it do it, in cases that can be timed.

Every case goes through a public entry point: the implicit cloth step
(``capi.Cloth.step_into``: assembly, PCG solve, update), its batched form, the
step with a contact operator, the cloth VBD step (``capi.Vbd.step_cloth``) and
the training step of the learned warm start's network (``learned.Trainer``).

A cloth is a triangulated nx x ny grid, one metre along its longer side, with
+-1% jitter of the rest positions, areal density 0.1 kg/m^2, Baraff-Witkin
stretch k = 1e4 and one spring per edge, pinned at its two top corners; it is
met in mid-motion: low-frequency waves in and out of plane (strains of a
percent or two, stretched and compressed regions) and smooth velocities.  For
the fixed 50 iterations it is held taut instead (2% over its rest shape): 50
iterations on slack cloth end so far from convergence that FP32 rounding alone
moves them by percents.  A pass is one time step of dt = 1/60 from that state
into the other state buffers, so that every pass solves the same system.

``exact`` restates the discretisation in FP64 torch: element gradients and
Hessians, lumped masses, pins, contacts, the linear solve, the VBD sweeps, the
network and its gradient.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ai-phyiscs_b200"))

from chysx import capi, learned, scenes  # noqa: E402

DT = 1.0 / 60.0
GRAVITY = (0.0, -9.81, 0.0)
DENSITY = 0.1
K_STRETCH = 1.0e4
K_SHEAR = 5.0e3
K_BEND = 5.0e-3
K_PIN = 1.0e6
DET_EPS = 1.0e-12
# ground plane and a box standing out of it, under part of the cloth
PLANE = ((0.0, 1.0, 0.0), -0.985)
BOX = ((0.1, 0.96, -0.1), (0.2, 0.03, 0.15))
STATIC = dict(thickness=0.01, k=1.0e4, mu=0.3, eps=1.0e-4)
# self-contact between two sheets 7 mm apart at a 10 mm thickness
GAP, THICK, K_CONTACT, MU_CONTACT, EPS_CONTACT = 0.007, 0.010, 1.0e3, 0.2, 1.0e-4
VBD_ITERATIONS = 10
VBD_MU, VBD_LAMBDA, VBD_DAMP, VBD_BEND, VBD_BEND_DAMP = 2.0e3, 2.0e3, 1.0e-3, 5.0e-3, 1.0e-3


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _step(nx, ny, solver, extra="", **more):
    return dict(kind="step", nx=nx, ny=ny, solver=solver, extra=extra, **more)


def listed():
    return [
        # the smallest: one 10 x 10 patch with every default of the reference (50 iterations, previous dx):
        # a game's flag or a unit of many, bound by latency and launches
        dict(name="patch10_default", **_step(10, 10, "default")),
        # a small garment: shear, bending (general 3x3 blocks), ground and box with friction, to 1e-6
        dict(name="garment61x47", **_step(61, 47, "plain", "garment")),
        # a middling cloth with the learned warm start and the two-level preconditioner
        dict(name="grid128_learned", **_step(128, 128, "learned")),
        # the 256 x 256 plain-method configuration with the reference's fixed 50 iterations
        dict(name="grid256_default", **_step(256, 256, "default")),
        # the same to 1e-6 with the two-level preconditioner (the benchmark's headline)
        dict(name="grid256_twolevel", **_step(256, 256, "twolevel")),
        # a large ragged cloth, fixed 50 iterations: rows stream from memory
        dict(name="grid801x643_default", **_step(801, 643, "default")),
        # the largest grid configuration, to 1e-6 with the two-level preconditioner
        dict(name="grid1024_twolevel", **_step(1024, 1024, "twolevel")),
        # many uneven instances in one launch, each to its own 1e-6 (the batched configuration, a quarter of it)
        dict(name="batch128", kind="batch", count=128, lo=16, hi=128),
        # two sheets in contact: a detector's list folded into the system every step, to 1e-6 with block-Jacobi
        dict(name="sheets160_contact", kind="contact", nx=160, ny=160),
        # cloth VBD, the second solver: small, and large and ragged
        dict(name="vbd64", kind="vbd", nx=64, ny=64),
        dict(name="vbd701x513", kind="vbd", nx=701, ny=513),
        # one training step of the warm-start network at its own batch size
        dict(name="train8192", kind="train", rows=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    nx = _log_int(rng, lo, hi)
    return nx, max(4, int(round(nx * rng.uniform(0.6, 1.0))))


def draw(rng):
    kind = rng.choice(["default", "default", "twolevel", "twolevel", "garment", "learned", "batch", "contact", "vbd",
                       "vbd", "train"])
    if kind == "default":
        return _step(*_sides(rng, 8, 1024), "default")
    if kind == "twolevel":
        return _step(*_sides(rng, 64, 1024), "twolevel")
    if kind == "garment":
        return _step(*_sides(rng, 12, 90), "plain", "garment")
    if kind == "learned":
        return _step(*_sides(rng, 48, 250), "learned")
    if kind == "batch":
        lo = rng.randint(10, 40)
        return dict(kind="batch", count=_log_int(rng, 4, 128), lo=lo, hi=rng.randint(lo + 8, 128))
    if kind == "contact":
        nx, ny = _sides(rng, 24, 300)
        return dict(kind="contact", nx=nx, ny=ny)
    if kind == "vbd":
        nx, ny = _sides(rng, 10, 700)
        return dict(kind="vbd", nx=nx, ny=ny)
    return dict(kind="train", rows=_log_int(rng, 200, 60000))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _waves(rng, uv, amp, out):
    """Adds six low-frequency modes of amplitude `amp` per component (uv in metres)."""
    for _ in range(6):
        f = rng.uniform(-2.0, 2.0, 2)
        ph = rng.uniform(0.0, 2.0 * math.pi)
        w = np.sin(2.0 * math.pi * (uv[:, 0] * f[0] + uv[:, 1] * f[1]) + ph)
        out += w[:, None] * (rng.standard_normal(3) * np.asarray(amp) / math.sqrt(6.0))[None]


def _sheet(rng, nx, ny, spacing=None, y=1.0, taut=False):
    """Rest positions, mid-motion positions and velocities, triangles of one grid."""
    h = 1.0 / (max(nx, ny) - 1) if spacing is None else spacing
    pos, tris = scenes.grid_mesh(nx, ny, y=y, spacing=h, origin=(-0.5 * h * (nx - 1), -0.5 * h * (ny - 1)))
    rest = pos + rng.uniform(-0.01 * h, 0.01 * h, pos.shape)
    uv = pos[:, [0, 2]]
    cur = rest.copy()
    in_plane = 2.0e-4 if taut else 1.0e-3
    _waves(rng, uv, (in_plane, 1.0e-2, in_plane), cur)
    cur[:, [0, 2]] *= (1.02, 1.02) if taut else (1.0, 1.005)
    vel = np.zeros_like(pos)
    _waves(rng, uv, (0.05, 0.3, 0.05), vel)
    vel[:, 1] -= 0.2
    return rest.astype(np.float32), cur.astype(np.float32), vel.astype(np.float32), tris.astype(np.int32)


def _n_edges(nx, ny):
    return (nx - 1) * ny + nx * (ny - 1) + (nx - 1) * (ny - 1)


def _log_uniform(rng, lo, hi, n):
    return np.exp(rng.uniform(math.log(lo), math.log(hi), n)).astype(np.float32)


def _problem(case, seed):
    """The host arrays of a cloth-step case."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        # the same sides for every seed: shapes belong to the case
        sides = np.random.default_rng(case["count"]).integers(case["lo"], case["hi"] + 1, case["count"])
        parts, offs, ks, kt, pins = [], [0], [], [], []
        for s in sides:
            s = int(s)
            rest, cur, vel, tris = _sheet(rng, s, s, spacing=1.0 / s)
            parts.append((rest, cur, vel, tris + offs[-1]))
            ks.append(_log_uniform(rng, 1.0e2, 1.0e4, _n_edges(s, s)))
            kt.append(np.full(tris.shape[0], _log_uniform(rng, 1.0e3, 1.0e5, 1)[0], np.float32))
            corners = np.array([0, s - 1, (s - 1) * s, s * s - 1])
            pins.append(offs[-1] + np.sort(rng.choice(corners, int(rng.integers(1, 5)), replace=False)))
            offs.append(offs[-1] + s * s)
        rest, cur, vel, tris = (np.concatenate([p[k] for p in parts]) for k in range(4))
        q = dict(rest=rest, cur=cur, vel=vel, tris=tris, k_spring=np.concatenate(ks), k_stretch=np.concatenate(kt),
                 pins=np.concatenate(pins), offsets=np.asarray(offs, np.int32))
    elif case["kind"] == "contact":
        nx, ny = case["nx"], case["ny"]
        rest, cur, vel, tris = _sheet(rng, nx, ny)
        n = rest.shape[0]
        up = np.array([0.0, GAP, 0.0], np.float32)
        jit = rng.uniform(-0.1, 0.1, (n, 3)).astype(np.float32) * (0.3 / (max(nx, ny) - 1))
        vel2 = vel + rng.uniform(-0.02, 0.02, 3).astype(np.float32)
        q = dict(rest=np.concatenate([rest, rest + up]), cur=np.concatenate([cur, cur + up + jit]),
                 vel=np.concatenate([vel, vel2]), tris=np.concatenate([tris, tris + n]).astype(np.int32),
                 k_spring=_log_uniform(rng, 1.0e2, 1.0e4, 2 * _n_edges(nx, ny)), k_stretch=K_STRETCH,
                 pins=np.array([(ny - 1) * nx, ny * nx - 1, n + (ny - 1) * nx, n + ny * nx - 1]))
        # vertex-face contacts: a third of the lower vertices against a face of the upper sheet around them
        v = np.flatnonzero(rng.uniform(size=n) < 1.0 / 3.0)
        i, j = np.minimum(v % nx, nx - 2), np.minimum(v // nx, ny - 2)
        f0 = n + j * nx + i
        bary = rng.dirichlet((2.0, 2.0, 2.0), v.size)
        pairs = np.stack([v, f0, f0 + 1, f0 + nx + 1], 1).astype(np.int32)
        nrm = np.array([0.0, -1.0, 0.0]) + rng.uniform(-0.05, 0.05, (v.size, 3))
        nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
        w = np.zeros((v.size, 8), np.float32)
        w[:, 0] = 1.0
        w[:, 1:4] = -bary
        w[:, 4:7] = nrm
        w[:, 7] = THICK - GAP + rng.uniform(-0.001, 0.001, v.size)
        slip = rng.uniform(-3.0e-4, 3.0e-4, (v.size, 3))
        slip -= np.sum(slip * nrm, 1, keepdims=True) * nrm
        u = np.concatenate([slip, np.linalg.norm(slip, axis=1, keepdims=True)], 1).astype(np.float32)
        q.update(pairs=pairs, weights=w, slips=u)
    else:
        nx, ny = case["nx"], case["ny"]
        rest, cur, vel, tris = _sheet(rng, nx, ny, taut=case["solver"] == "default")
        q = dict(rest=rest, cur=cur, vel=vel, tris=tris, k_spring=_log_uniform(rng, 1.0e2, 1.0e4, _n_edges(nx, ny)),
                 k_stretch=K_STRETCH, pins=np.array([(ny - 1) * nx, ny * nx - 1]))
    q["pins"] = q["pins"].astype(np.int32)
    q["pin_targets"] = q["cur"][q["pins"]].copy()
    return q


def _solver(case):
    """(max_iter, rel_tol, warm_start) of a cloth-step case."""
    if case["kind"] == "batch" or case.get("solver") == "twolevel":
        return 30000, 1.0e-6, "zero"
    if case["kind"] == "contact" or case.get("solver") == "plain":
        return 30000, 1.0e-6, "zero"
    if case.get("solver") == "learned":
        return 30000, 1.0e-6, "learned"
    return 50, 0.0, "previous"


def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _prepare_step(case, seed):
    q = _problem(case, seed)
    n = q["rest"].shape[0]
    st = dict(n=n, pos=_gpu(q["rest"]), vel=_gpu(q["vel"]), inv_mass=torch.ones(n, device="cuda"))
    st["pos_out"], st["vel_out"] = torch.empty_like(st["pos"]), torch.empty_like(st["vel"])
    s = capi.Cloth()
    s.set_material(density=DENSITY, gravity=GRAVITY)
    s.set_external_buffers(st["pos"].data_ptr(), st["vel"].data_ptr(), n, st["inv_mass"].data_ptr())
    s.set_mesh(q["tris"])
    if "offsets" in q:
        s.set_instances(q["offsets"])
    s.set_options(True, False, DET_EPS)
    s.redistribute_mass(DENSITY, st["inv_mass"].data_ptr(), n)
    s.build_springs(q["k_spring"])
    s.build_fem_stretch(q["k_stretch"])
    if case.get("extra") == "garment":
        s.build_fem_shear(K_SHEAR)
        s.build_bending(K_BEND)
        s.add_static_plane(*PLANE)
        s.add_static_box(*BOX)
        s.set_static_contact(STATIC["thickness"], STATIC["k"], STATIC["mu"], STATIC["eps"])
    s.set_pins(q["pins"], q["pin_targets"], K_PIN)
    if case["kind"] == "contact":
        for k in ("pairs", "weights", "slips"):
            st[k] = _gpu(q[k])
        st["count"] = torch.tensor([q["pairs"].shape[0]], dtype=torch.int32, device="cuda")
        s.set_contact_op(st["pairs"].data_ptr(), st["weights"].data_ptr(), st["count"].data_ptr(),
                         q["pairs"].shape[0], K_CONTACT, slips=st["slips"].data_ptr(), friction_mu=MU_CONTACT,
                         friction_epsilon=EPS_CONTACT)
    max_iter, tol, warm = _solver(case)
    if warm == "learned":
        params, _ = learned.load()
        s.set_network(params)
    if case["kind"] == "batch" or case.get("solver") in ("twolevel", "learned"):
        s.set_row_order(1)
        s.set_preconditioner("chebyshev_coarse", 7, 60.0)
    s.set_solver(max_iter, tol, warm)
    st["sim"] = s
    # the frame before this one, as a running simulation has behind it: the plan is laid out, and the
    # previous dx is there for the solves that start from it
    cur = _gpu(q["cur"])
    st["pos"].copy_(cur - DT * st["vel"])
    s.step_into(DT, st["pos"].data_ptr(), st["vel"].data_ptr(), st["pos_out"].data_ptr(), st["vel_out"].data_ptr())
    torch.cuda.synchronize()
    st["pos"].copy_(cur)
    return st


def _vbd_problem(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    rest, cur, vel, tris = _sheet(rng, nx, ny)
    x = rest.astype(np.float64)
    e1, e2 = x[tris[:, 1]] - x[tris[:, 0]], x[tris[:, 2]] - x[tris[:, 0]]
    l1 = np.linalg.norm(e1, axis=1)
    nrm = np.cross(e1, e2)
    area = 0.5 * np.linalg.norm(nrm, axis=1)
    b = np.cross(nrm / (2.0 * area)[:, None], e1 / l1[:, None])
    u, v = np.einsum("ij,ij->i", e2, e1) / l1, np.einsum("ij,ij->i", e2, b)
    poses = np.stack([1.0 / l1, -u / (l1 * v), np.zeros_like(l1), 1.0 / v], 1)

    def at(i, j):
        return (j * nx + i).ravel()

    # interior edges (o0, o1, v2, v3): quad diagonals, then the edges along x and along z
    i, j = np.meshgrid(np.arange(nx - 1), np.arange(ny - 1), indexing="xy")
    hinges = [np.stack([at(i, j + 1), at(i + 1, j), at(i, j), at(i + 1, j + 1)], 1)]
    i, j = np.meshgrid(np.arange(nx - 1), np.arange(1, ny - 1), indexing="xy")
    hinges.append(np.stack([at(i + 1, j + 1), at(i, j - 1), at(i, j), at(i + 1, j)], 1))
    i, j = np.meshgrid(np.arange(1, nx - 1), np.arange(ny - 1), indexing="xy")
    hinges.append(np.stack([at(i - 1, j), at(i + 1, j + 1), at(i, j), at(i, j + 1)], 1))
    edges = np.concatenate(hinges).astype(np.int32)
    mass = np.zeros(x.shape[0])
    np.add.at(mass, tris.ravel(), np.repeat(area * DENSITY / 3.0, 3))
    inv_mass = 1.0 / mass
    inv_mass[[(ny - 1) * nx, ny * nx - 1]] = 0.0
    xe = [x[edges[:, k]] for k in range(4)]
    ii = np.arange(nx * ny)
    return dict(pos=cur, vel=vel, inv_mass=inv_mass.astype(np.float32), tris=tris, poses=poses.astype(np.float32),
                areas=area.astype(np.float32),
                mats=np.tile(np.array([VBD_MU, VBD_LAMBDA, VBD_DAMP], np.float32), (tris.shape[0], 1)), edges=edges,
                rest_angle=np.zeros(edges.shape[0], np.float32),
                rest_length=np.linalg.norm(xe[3] - xe[2], axis=1).astype(np.float32),
                props=np.tile(np.array([VBD_BEND, VBD_BEND_DAMP], np.float32), (edges.shape[0], 1)),
                # 2 x 2 colouring of the grid: vertices of one element or hinge differ in the parity of i or j
                colors=((ii % nx) % 2 + 2 * ((ii // nx) % 2)).astype(np.int32))


def _prepare_vbd(case, seed):
    q = _vbd_problem(case, seed)
    n = q["pos"].shape[0]
    s = capi.Vbd()
    s.set_coloring(q["colors"])
    s.build_tri_adjacency(q["tris"], n)
    s.build_edge_adjacency(q["edges"], n)
    st = {k: _gpu(v) for k, v in q.items() if k != "colors"}
    st.update(sim=s, n=n, x=st["pos"].clone(), v=st["vel"].clone())
    _run_vbd(st)
    torch.cuda.synchronize()
    return st


def _run_vbd(st):
    # a rollout's step: from the saved state
    st["x"].copy_(st["pos"])
    st["v"].copy_(st["vel"])
    p = {k: st[k].data_ptr() for k in ("x", "v", "inv_mass", "tris", "poses", "areas", "mats", "edges", "rest_angle",
                                       "rest_length", "props")}
    st["sim"].step_cloth(p["x"], p["v"], p["inv_mass"], st["n"], p["tris"], p["poses"], p["areas"], p["mats"],
                         st["tris"].shape[0], p["edges"], p["rest_angle"], p["rest_length"], p["props"],
                         st["edges"].shape[0], GRAVITY, DT, VBD_ITERATIONS)
    return st["x"], st["v"]


def _train_problem(case, seed):
    rng = np.random.default_rng(seed)
    rows = case["rows"]
    mu_in, sd_in = 0.1 * rng.standard_normal(20), rng.uniform(0.5, 2.0, 20)
    mu_out, sd_out = 0.1 * rng.standard_normal(3), rng.uniform(0.5, 1.5, 3)
    params = learned.init_params(rng, mu_in, sd_in, mu_out, sd_out)
    feats = (mu_in + sd_in * rng.standard_normal((rows, 20))).astype(np.float32)
    # targets the features explain in part, as velocity changes are
    mix = rng.standard_normal((20, 3)) / math.sqrt(20.0)
    targs = np.tanh(((feats - mu_in) / sd_in) @ mix) + 0.3 * rng.standard_normal((rows, 3))
    targs = (mu_out + sd_out * targs).astype(np.float32)
    m1 = (1.0e-3 * rng.standard_normal(params.size)).astype(np.float32)
    m2 = (1.0e-5 * rng.uniform(0.5, 2.0, params.size)).astype(np.float32)
    return params, feats, targs, m1, m2


TRAIN_STEP, TRAIN_LR = 100, 2.0e-3


def _prepare_train(case, seed):
    params, feats, targs, m1, m2 = _train_problem(case, seed)
    t = learned.Trainer(params, case["rows"])
    t.m1.copy_(_gpu(m1))
    t.m2.copy_(_gpu(m2))
    t.t = TRAIN_STEP
    return dict(trainer=t, feats=_gpu(feats), targs=_gpu(targs))


def prepare(case, seed):
    if case["kind"] == "vbd":
        return _prepare_vbd(case, seed)
    if case["kind"] == "train":
        return _prepare_train(case, seed)
    return _prepare_step(case, seed)


def run(state):
    if "trainer" in state:
        t = state["trainer"]
        loss = t.step(state["feats"], state["targs"], TRAIN_LR)
        return dict(loss=loss, params=t.p, grad=t.g, m1=t.m1, m2=t.m2)
    if "x" in state:
        return _run_vbd(state)
    state["sim"].step_into(DT, state["pos"].data_ptr(), state["vel"].data_ptr(), state["pos_out"].data_ptr(),
                           state["vel_out"].data_ptr())
    return state["pos_out"], state["vel_out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _size(case):
    if case["kind"] == "batch":
        s = 0.5 * (case["lo"] + case["hi"])
        return int(case["count"] * (s * s + (case["hi"] - case["lo"]) ** 2 / 12.0))
    return case["nx"] * case["ny"] * (2 if case["kind"] == "contact" else 1)


def work(case):
    if case["kind"] == "train":
        per_row = 2 * (20 * 64 + 2 * 64 * 64 + 64 * 3)
        return dict(bytes=case["rows"] * 23 * 4 + 4 * 4 * 9900 + 3 * 4 * 9900, flops=3 * per_row * case["rows"])
    n = _size(case)
    if case["kind"] == "vbd":
        # state in and out, 2 triangles (indices, rest data, material) and 3 hinges per vertex, every sweep once;
        # about 300 flops for each of a vertex's 6 triangle and 12 hinge terms
        return dict(bytes=n * (7 * 4 + 6 * 4 + 2 * 44 + 3 * 32), flops=VBD_ITERATIONS * n * 18 * 300)
    # state, inverse mass, 2 triangles and 3 springs with their rest data; 3x3 products of 6 blocks and the diagonal
    # and ten vector operations per row and iteration, for the fixed count or (to 1e-6) a nominal 300
    its = _solver(case)[0] if _solver(case)[1] == 0.0 else 300
    return dict(bytes=n * (13 * 4 + 2 * 52 + 3 * 20), flops=n * (its * (7 * 18 + 60) + 4000))


def tolerance(case):
    if case["kind"] == "train":
        # BF16 operands and FP32 sums: the gradient lies 2.7e-3 from FP64, and so would another kernel's
        return {"rel": 1.0e-2, "max": 0.4}
    if case["kind"] == "vbd":
        # FP32 throughout: velocities 4e-6 from FP64
        return {"rel": 2.0e-5, "max": 1.0e-3}
    if _solver(case)[1] == 0.0:
        # 50 iterations: resident and streamed kernels, whose sums run in other orders, differ by up to 3.2e-7, and
        # on a patch so small that 50 is close to its Krylov space by up to 2.9e-4 (10 x 10)
        return {"rel": 1.2e-3, "max": 0.05} if _size(case) < 4000 else {"rel": 4.0e-6, "max": 4.0e-4}
    # solves to 1e-6 with other kernels, CTA sizes and preconditioners: up to 6.4e-5 (max 0.08)
    return {"rel": 2.5e-4, "max": 0.35}


# ---------------------------------------------------------------------------
# the same in FP64
# ---------------------------------------------------------------------------
EXACT_ROWS = 300000  # above this a converged FP64 solve takes too long


def _d(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", torch.float64 if np.asarray(a).dtype.kind == "f" else torch.int64)


def _norm(a):
    return a.norm(dim=1, keepdim=True)


def _outer(a, b):
    return a[:, :, None] * b[:, None, :]


class _System:
    """b - A x of one step in FP64: 3x3 blocks gathered as (row, col, block) triples."""

    def __init__(self, n):
        self.n, self.rows, self.cols, self.blocks = n, [], [], []
        self.g = torch.zeros(n, 3, dtype=torch.float64, device="cuda")

    def add(self, r, c, blk):
        self.rows.append(r)
        self.cols.append(c)
        self.blocks.append(blk)

    def grad(self, r, v):
        self.g.index_add_(0, r, v)

    def finish(self):
        r, c, blk = torch.cat(self.rows), torch.cat(self.cols), torch.cat(self.blocks)
        key, inv = torch.unique(r * self.n + c, return_inverse=True)
        b = torch.zeros(key.numel(), 9, dtype=torch.float64, device="cuda").index_add_(0, inv, blk.reshape(-1, 9))
        del r, c, blk, inv
        self.rows = self.cols = self.blocks = None
        r, c, b = key // self.n, key % self.n, b.reshape(-1, 3, 3)
        d = torch.zeros(self.n, 3, 3, dtype=torch.float64, device="cuda")
        on = r == c
        d[r[on]] = b[on]
        q = torch.arange(3, device="cuda")
        rr = (3 * r[:, None, None] + q[None, :, None]).expand(-1, 3, 3).reshape(-1)
        cc = (3 * c[:, None, None] + q[None, None, :]).expand(-1, 3, 3).reshape(-1)
        a = torch.sparse_coo_tensor(torch.stack([rr, cc]), b.reshape(-1), (3 * self.n, 3 * self.n)).to_sparse_csr()
        return a, torch.linalg.inv(d)


def _rest_shape(x, tris, turn):
    a, b, c = (x[tris[:, k]] for k in range(3))
    ab, ac = b - a, c - a
    lab = ab.norm(dim=1)
    uc = (ab * ac).sum(1) / lab
    vc = torch.sqrt(torch.clamp((ac * ac).sum(1) - uc * uc, min=0.0))
    i00, i01, i11 = 1.0 / lab, -uc / (lab * vc), 1.0 / vc
    ct, s = math.cos(turn), math.sin(turn)
    return torch.stack([i00 * ct - i01 * s, i00 * s + i01 * ct, -i11 * s, i11 * ct], 1), 0.5 * lab * vc


def _add_stretch(sys_, x, tris, dm, area, k):
    a, b = x[tris[:, 1]] - x[tris[:, 0]], x[tris[:, 2]] - x[tris[:, 0]]
    ke = (area * k)[:, None]
    ds, ms, gs = [], [], []
    for w in range(2):
        f = a * dm[:, w:w + 1] + b * dm[:, 2 + w:3 + w]
        l = _norm(f).clamp(min=1.0e-6)
        u, c = f / l, l - 1.0
        s = torch.where(c > 0.0, ke * c / l, torch.zeros_like(c))
        ms.append((ke - s)[:, :, None] * _outer(u, u) + s[:, :, None] * torch.eye(3, dtype=torch.float64, device="cuda"))
        gs.append(u * c * ke)
        ds.append([-dm[:, w] - dm[:, 2 + w], dm[:, w], dm[:, 2 + w]])
    for p in range(3):
        sys_.grad(tris[:, p], gs[0] * ds[0][p][:, None] + gs[1] * ds[1][p][:, None])
        for q in range(3):
            sys_.add(tris[:, p], tris[:, q], (ds[0][p] * ds[0][q])[:, None, None] * ms[0] +
                     (ds[1][p] * ds[1][q])[:, None, None] * ms[1])


def _bend(x0, x1, x2, x3):
    e, e2, e3 = x1 - x0, x2 - x0, x3 - x0
    n1, n2 = torch.linalg.cross(e2, e), torch.linalg.cross(e, e3)
    n1, n2 = n1 / _norm(n1), n2 / _norm(n2)
    le = _norm(e)
    th = torch.atan2((torch.linalg.cross(n1, n2) * e / le).sum(1).clamp(-1, 1), (n1 * n2).sum(1))
    w1, w2 = (e * e2).sum(1, keepdim=True) / le ** 2, (e * e3).sum(1, keepdim=True) / le ** 2
    g1, g2 = 1.0 / _norm(e2 - e * w1), 1.0 / _norm(e3 - e * w2)
    return th, [n1 * ((w1 - 1.0) * g1) + n2 * ((w2 - 1.0) * g2), n1 * (-w1 * g1) + n2 * (-w2 * g2), n1 * g1, n2 * g2]


def _dihedrals(tris):
    """(v0, v1 hinge as one triangle walks it, v2 its third vertex, v3 the other triangle's)."""
    t = np.asarray(tris, np.int64)
    u = np.concatenate([t[:, 0], t[:, 1], t[:, 2]])
    v = np.concatenate([t[:, 1], t[:, 2], t[:, 0]])
    w = np.concatenate([t[:, 2], t[:, 0], t[:, 1]])
    key = np.minimum(u, v) * (t.max() + 1) + np.maximum(u, v)
    o = np.argsort(key, kind="stable")
    first = np.flatnonzero(key[o][1:] == key[o][:-1])
    p, q = o[first], o[first + 1]
    return np.stack([u[p], v[p], w[p], w[q]], 1)


def _static(x, vel, dt, sys_):
    """Deepest static contact of every particle: gradient, block, and (depth, normal) for the cone."""
    th, k, mu, eps = STATIC["thickness"], *(float(np.float32(STATIC[q])) for q in ("k", "mu", "eps"))
    th = float(np.float32(th))
    nrm = torch.tensor(PLANE[0], dtype=torch.float64, device="cuda").expand_as(x).clone()
    best = (th - (x @ nrm[0] + float(np.float32(PLANE[1])))).clamp(min=0.0)
    c = torch.tensor(np.asarray(BOX[0], np.float32), dtype=torch.float64, device="cuda")
    h = torch.tensor(np.asarray(BOX[1], np.float32), dtype=torch.float64, device="cuda")
    rel = x - c
    sg = torch.where(rel >= 0, 1.0, -1.0).to(torch.float64)
    d = rel.abs() - h
    inside = (d <= 0).all(1)
    face = torch.nn.functional.one_hot(d.argmax(1), 3).to(torch.float64)
    cl = d.clamp(min=0.0)
    dist = cl.norm(dim=1)
    nb = torch.where(inside[:, None], face * sg, cl * sg / dist.clamp(min=1.0e-300)[:, None])
    depth = th - torch.where(inside, d.max(1).values, dist)
    deeper = depth > best
    nrm = torch.where(deeper[:, None], nb, nrm)
    best = torch.where(deeper, depth, best)
    on = best > 0.0
    r = torch.nonzero(on)[:, 0]
    n, dp = nrm[r], best[r][:, None]
    dx = vel[r] * dt
    ut = dx - n * (n * dx).sum(1, keepdim=True)
    un = _norm(ut)
    al = mu * (k * dp) * torch.where(un > eps, 1.0 / un.clamp(min=1e-300), (-un / eps + 2.0) / eps)
    sys_.grad(r, n * (-k * dp) - ut * al)
    nn = _outer(n, n)
    sys_.add(r, r, k * nn + al[:, :, None] * (torch.eye(3, dtype=torch.float64, device="cuda") - nn))
    return r, n, dp


def _cone(b, contact):
    r, n, dp = contact
    k, mu = float(np.float32(STATIC["k"])), float(np.float32(STATIC["mu"]))
    f0 = b[r] - n * (k * dp)
    fn0 = (f0 * n).sum(1, keepdim=True)
    fn, ft = (-fn0).clamp(min=0.0), f0 - n * fn0
    l = _norm(ft)
    cut = torch.where(l <= mu * fn, torch.ones_like(l), mu * fn / l.clamp(min=1.0e-300))
    b = b.clone()
    b[r] = torch.where((fn > 0) & (l > 0), b[r] - ft * cut, b[r])
    return b


def _assemble(case, q, x, vel):
    n = x.shape[0]
    dt = float(np.float32(DT))
    s = _System(n)
    tris, rest = _d(q["tris"]), _d(q["rest"])
    edges = _edges(q["tris"])
    ex, ey = _d(edges[:, 0]), _d(edges[:, 1])
    k = _d(q["k_spring"])[:, None]
    rl = _norm(rest[ex] - rest[ey])
    d = x[ex] - x[ey]
    l = _norm(d)
    dh, a = d / l, k * rl / l
    s.grad(ex, dh * (k * (l - rl)))
    s.grad(ey, -dh * (k * (l - rl)))
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    h = torch.where(l < rl, torch.zeros_like(l), k - a)[:, :, None] * eye + a[:, :, None] * _outer(dh, dh)
    for p, c, sg in ((ex, ex, 1.0), (ey, ey, 1.0), (ex, ey, -1.0), (ey, ex, -1.0)):
        s.add(p, c, sg * h)
    kt = torch.full((tris.shape[0],), q["k_stretch"], dtype=torch.float64, device="cuda") if np.ndim(q["k_stretch"]) == 0 else _d(q["k_stretch"])
    dm, area = _rest_shape(rest, tris, 0.0)
    area = area.float().double()
    _add_stretch(s, x, tris, dm, area, kt)
    garment = case.get("extra") == "garment"
    if garment:
        dm, _ = _rest_shape(rest, tris, 0.25 * math.pi)
        _add_stretch(s, x, tris, dm, area, torch.full_like(kt, K_SHEAR))
        v = [_d(c) for c in _dihedrals(q["tris"]).T]
        t0, _ = _bend(*(rest[c] for c in v))
        th, ga = _bend(*(x[c] for c in v))
        kb = float(np.float32(K_BEND))
        for p in range(4):
            s.grad(v[p], kb * (th - t0)[:, None] * ga[p])
            for c in range(4):
                s.add(v[p], v[c], kb * _outer(ga[p], ga[c]))
    if case["kind"] == "contact":
        pr, w, u = _d(q["pairs"]), _d(q["weights"]), _d(q["slips"])
        nrm, dp, kc = w[:, 4:7], w[:, 7:8], K_CONTACT
        eps = float(np.float32(EPS_CONTACT))
        un = u[:, 3:4]
        al = float(np.float32(MU_CONTACT)) * kc * dp * torch.where(un > eps, 1.0 / un.clamp(min=1e-300), (-un / eps + 2.0) / eps)
        nn = _outer(nrm, nrm)
        hc = (kc - al)[:, :, None] * nn + al[:, :, None] * eye
        for p in range(4):
            s.grad(pr[:, p], w[:, p:p + 1] * (-kc * dp * nrm - al * u[:, :3]))
            for c in range(4):
                s.add(pr[:, p], pr[:, c], (w[:, p] * w[:, c])[:, None, None] * hc)
    pins, tg = _d(q["pins"]), _d(q["pin_targets"])
    s.grad(pins, K_PIN * (x[pins] - tg))
    s.add(pins, pins, (K_PIN * eye).expand(pins.numel(), 3, 3))
    x0, x1, x2 = (rest[tris[:, c]] for c in range(3))
    ta = 0.5 * torch.linalg.cross(x1 - x0, x2 - x0).norm(dim=1)
    m = torch.zeros(n, dtype=torch.float64, device="cuda")
    for c in range(3):
        m.index_add_(0, tris[:, c], ta * (float(np.float32(DENSITY)) / 3.0))
    rows = torch.arange(n, device="cuda")
    s.add(rows, rows, (m / dt ** 2)[:, None, None] * eye)
    contact = _static(x, vel, dt, s) if garment else None
    grav = torch.tensor(np.asarray(GRAVITY, np.float32), dtype=torch.float64, device="cuda")
    b = (vel / dt + grav) * m[:, None] - s.g
    if contact is not None:
        b = _cone(b, contact)
    a, minv = s.finish()
    return a, minv, b


def _edges(tris):
    """Sorted unique undirected edges."""
    t = np.asarray(tris, np.int64)
    u = np.concatenate([t[:, 0], t[:, 1], t[:, 2]])
    v = np.concatenate([t[:, 1], t[:, 2], t[:, 0]])
    n = t.max() + 1
    key = np.unique(np.minimum(u, v) * n + np.maximum(u, v))
    return np.stack([key // n, key % n], 1)


def _pcg(a, minv, b, x, iters, tol):
    """Block-Jacobi PCG: `iters` iterations, or (tol > 0) to ||r|| <= tol ||b||."""
    def spmv(p):
        return (a @ p.reshape(-1)).reshape(-1, 3)

    def prec(r):
        return torch.bmm(minv, r[:, :, None])[:, :, 0]

    r = b - spmv(x)
    z = prec(r)
    p = z.clone()
    rho = (r * z).sum()
    stop = tol * tol * float((b * b).sum())
    for k in range(iters):
        ap = spmv(p)
        alpha = rho / (p * ap).sum()
        x = x + alpha * p
        r = r - alpha * ap
        if tol > 0.0 and k % 50 == 49 and float((r * r).sum()) <= stop:
            break
        z = prec(r)
        new = (r * z).sum()
        p = z + (new / rho) * p
        rho = new
    return x


def _exact_step(case, seed):
    q = _problem(case, seed)
    n = q["rest"].shape[0]
    max_iter, tol, warm = _solver(case)
    if tol > 0.0 and n > EXACT_ROWS:
        return None
    vel = _d(q["vel"])
    x = _d(q["cur"])
    dx = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    if warm == "previous":
        prev = torch.from_numpy(q["cur"]).cuda() - DT * torch.from_numpy(q["vel"]).cuda()
        a, minv, b = _assemble(case, q, prev.double(), vel)
        dx = _pcg(a, minv, b, dx, max_iter, 0.0)
        del a
    a, minv, b = _assemble(case, q, x, vel)
    dx = _pcg(a, minv, b, dx, max_iter if tol == 0.0 else 60000, 1.0e-11 if tol > 0.0 else 0.0)
    return x + dx, dx / float(np.float32(DT))


def _exact_vbd(case, seed):
    q = _vbd_problem(case, seed)
    dt = float(np.float32(DT))
    d = {k: _d(v) for k, v in q.items()}
    n = q["pos"].shape[0]
    grav = torch.tensor(np.asarray(GRAVITY, np.float32), dtype=torch.float64, device="cuda")
    xp = d["pos"]
    free = (d["inv_mass"] > 0)[:, None]
    vn = d["vel"] + grav * dt
    y = torch.where(free, xp + vn * dt, xp)
    x = y.clone()
    m = torch.where(d["inv_mass"] > 0, 1.0 / d["inv_mass"].clamp(min=1e-30), torch.zeros_like(d["inv_mass"]))
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    jobs = []
    for c in range(4):
        mine = (d["colors"] == c) & (d["inv_mass"] > 0)
        jobs.append((torch.nonzero(mine)[:, 0],
                     [torch.nonzero(mine[d["tris"][:, k]])[:, 0] for k in range(3)],
                     [torch.nonzero(mine[d["edges"][:, k]])[:, 0] for k in range(4)]))
    mu, la, dm_ = (float(np.float32(v)) for v in (VBD_MU, VBD_LAMBDA, VBD_DAMP))
    bk, bd = (float(np.float32(v)) for v in (VBD_BEND, VBD_BEND_DAMP))
    lam = la + mu
    alpha = 1.0 + mu / lam

    def damp(kd, g, rate, area, f, h):
        return f - g * (kd * rate * area), h + (kd / dt * area)[:, :, None] * _outer(g, g)

    for _ in range(VBD_ITERATIONS):
        for verts, tri_jobs, edge_jobs in jobs:
            f = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
            h = torch.zeros(n, 3, 3, dtype=torch.float64, device="cuda")
            for w, t in enumerate(tri_jobs):
                tv = d["tris"][t]
                xs, ps = [x[tv[:, k]] for k in range(3)], [xp[tv[:, k]] for k in range(3)]
                dm, ar = d["poses"][t], d["areas"][t][:, None]
                e1, e2 = xs[1] - xs[0], xs[2] - xs[0]
                f0, f1 = e1 * dm[:, 0:1] + e2 * dm[:, 2:3], e1 * dm[:, 1:2] + e2 * dm[:, 3:4]
                q0, q1 = ((-(dm[:, 0:1] + dm[:, 2:3]), -(dm[:, 1:2] + dm[:, 3:4])), (dm[:, 0:1], dm[:, 1:2]),
                          (dm[:, 2:3], dm[:, 3:4]))[w]
                nr = torch.linalg.cross(f0, f1)
                j = _norm(nr).clamp(min=1.0e-10)
                wv = f1 * q0 - f0 * q1
                dj = torch.linalg.cross(wv, nr / j)
                vol = lam * (j - alpha)
                fo = ((f0 * q0 + f1 * q1) * mu + dj * vol) * (-ar)
                r = vol.clamp(min=0.0) / j
                hh = ((mu * (q0 * q0 + q1 * q1) + r * (wv * wv).sum(1, keepdim=True)) * ar)[:, :, None] * eye
                hh = hh + ((lam - r) * ar)[:, :, None] * _outer(dj, dj) - (r * ar)[:, :, None] * _outer(wv, wv)
                g00, g11 = 0.5 * ((f0 * f0).sum(1, keepdim=True) - 1.0), 0.5 * ((f1 * f1).sum(1, keepdim=True) - 1.0)
                g01 = 0.5 * (f0 * f1).sum(1, keepdim=True)
                gn = torch.sqrt(g00 ** 2 + g11 ** 2 + 2.0 * g01 ** 2)
                u1, u2 = (e1 - (ps[1] - ps[0])) / dt, (e2 - (ps[2] - ps[0])) / dt
                a0, a1 = u1 * dm[:, 0:1] + u2 * dm[:, 2:3], u1 * dm[:, 1:2] + u2 * dm[:, 3:4]
                s00, s11 = (f0 * a0).sum(1, keepdim=True), (f1 * a1).sum(1, keepdim=True)
                s01 = 0.5 * ((f0 * a1).sum(1, keepdim=True) + (f1 * a0).sum(1, keepdim=True))
                gd = (f0 * g00 + f1 * g01) * (q0 / gn) + (f0 * g01 + f1 * g11) * (q1 / gn)
                fo, hh = damp(mu * dm_, gd, (g00 * s00 + g11 * s11 + 2.0 * g01 * s01) / gn, ar, fo, hh)
                fo, hh = damp(la * dm_, f0 * q0 + f1 * q1, s00 + s11, ar, fo, hh)
                f.index_add_(0, tv[:, w], fo)
                h.index_add_(0, tv[:, w], hh)
            for w, e in enumerate(edge_jobs):
                ev = d["edges"][e]
                xs, ps = [x[ev[:, k]] for k in range(4)], [xp[ev[:, k]] for k in range(4)]
                eg = xs[3] - xs[2]
                n1 = torch.linalg.cross(xs[2] - xs[0], xs[3] - xs[0])
                n2 = torch.linalg.cross(xs[3] - xs[1], xs[2] - xs[1])
                q1, q2, le = (n1 * n1).sum(1, keepdim=True), (n2 * n2).sum(1, keepdim=True), _norm(eg)
                ok = ((torch.sqrt(q1) >= 1.0e-6) & (torch.sqrt(q2) >= 1.0e-6) & (le >= 1.0e-6)).double()
                t = eg / le
                a, b = n1 / q1, n2 / q2
                l12 = torch.sqrt(q1 * q2)
                th = torch.atan2((torch.linalg.cross(n1, n2) * t).sum(1, keepdim=True) / l12,
                                 (n1 * n2).sum(1, keepdim=True) / l12)

                def along(p, o):
                    return ((xs[p] - xs[o]) * t).sum(1, keepdim=True)

                g = [a * (-le), b * (-le), a * (-along(0, 3)) - b * along(1, 3), a * along(0, 2) + b * along(1, 2)]
                k = bk * d["rest_length"][e][:, None] * ok
                fo = g[w] * (-k * (th - d["rest_angle"][e][:, None]))
                hh = k[:, :, None] * _outer(g[w], g[w])
                rate = sum((g[c] * (xs[c] - ps[c])).sum(1, keepdim=True) for c in range(4)) / dt
                fo, hh = damp(bd, g[w], rate, k, fo, hh)
                f.index_add_(0, ev[:, w], fo)
                h.index_add_(0, ev[:, w], hh)
            md = (m[verts] / dt ** 2)[:, None]
            fv = f[verts] + (y[verts] - x[verts]) * md
            hv = h[verts] + md[:, :, None] * eye
            x[verts] = x[verts] + torch.linalg.solve(hv, fv[:, :, None])[:, :, 0]
    return x, (x - xp) / dt


def _exact_train(case, seed):
    params, feats, targs, m1, m2 = _train_problem(case, seed)
    p = _d(params)
    f, t = _d(feats), _d(targs)
    mu_in, sd_in, mu_out, sd_out = p[:20], p[20:40], p[40:43], p[43:46]
    w = p[46:].clone().requires_grad_(True)
    layers, k = [], 0
    for a, b in ((20, 64), (64, 64), (64, 64), (64, 3)):
        layers.append((w[k:k + a * b].reshape(a, b), w[k + a * b:k + a * b + b]))
        k += a * b + b
    h = (f - mu_in) / sd_in
    for n, (mat, bias) in enumerate(layers):
        h = h @ mat + bias
        if n < 3:
            h = torch.nn.functional.gelu(h)
    loss = ((h - (t - mu_out) / sd_out) ** 2).mean()
    loss.backward()
    g = torch.cat([torch.zeros(46, dtype=torch.float64, device="cuda"), w.grad])
    a1, a2 = _d(m1), _d(m2)
    n1, n2 = a1.clone(), a2.clone()
    n1[46:] = 0.9 * a1[46:] + 0.1 * g[46:]
    n2[46:] = 0.999 * a2[46:] + 0.001 * g[46:] ** 2
    step = TRAIN_STEP + 1
    out = p.clone()
    out[46:] -= TRAIN_LR * (n1[46:] / (1.0 - 0.9 ** step)) / (torch.sqrt(n2[46:] / (1.0 - 0.999 ** step)) + 1.0e-8)
    return dict(loss=float(loss.detach()), params=out, grad=g, m1=n1, m2=n2)


def exact(case, seed):
    if case["kind"] == "vbd":
        return _exact_vbd(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return _exact_step(case, seed)
