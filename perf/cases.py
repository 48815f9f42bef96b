"""Performance cases of the SAP contact step.

Each case is one call, or one short run of calls, that a program using this
framework makes through its public entry points: whole steps (SolverSAP), the
free motion with the contact rows (SapContactJacobian), the contact solve
alone in its three layouts (one DOF count, one count per world, tree-blocked),
contact generation, and a training step of the warm-start network.

`listed()` names the cases, `draw()` takes more from the same ranges.  Inputs
are synthetic and come from a seed: the robots, contact counts, penetrations,
friction and stiffness ranges are those of the scenes in
sap_warp_b200/models.py and sap_warp_b200/scenes.py.  `exact()` computes the
same outputs in plain FP64 torch (dense Newton to the rounding floor).
"""

from __future__ import annotations

import math

import numpy as np
import torch

from sap_warp_b200 import models, scenes
from sap_warp_b200._solve import ContactSolveBuffers, blocked_contact_solve, contact_solve, make_options
from sap_warp_b200.collision import ContactGenerator, ShapeSet
from sap_warp_b200.runtime import SAP_JOINT_FREE, SapState
from sap_warp_b200.solver import SapContactJacobian, SolverSAP
from sap_warp_b200.warmstart import FeatureNorm, TrainBuffers, WarmStartMLP

DT = 2.0e-3
F64, F32, I32 = torch.float64, torch.float32, torch.int32
CUDA = torch.device("cuda:0")


# ---- the cases ------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # one robot in a control or teleoperation loop: eight eager steps from
        # a given state, where launches and host work are what is waited for
        dict(name="rollout-humanoid-1", kind="rollout", robot="humanoid", worlds=1, steps=8, precision="fp64",
             warm_start="previous_velocity", graph=False),
        # sampling or policy training: a batch of humanoids rolled out from
        # given states, two steps per captured graph, the fastest settings
        dict(name="rollout-humanoid-4096", kind="rollout", robot="humanoid", worlds=4096, steps=8, precision="fp32",
             warm_start="learned", graph=True),
        # manipulation: an arm gripping one of eight stacked boxes, worlds of
        # several trees (tree-blocked layout), reference settings
        dict(name="rollout-arm-boxes-512", kind="rollout", robot="arm_boxes", boxes=8, worlds=512, steps=2,
             precision="fp64", warm_start="previous_velocity", graph=False),
        # free motion and contact rows of the batch, as a program with a
        # solver of its own takes them
        dict(name="rows-humanoid-4096", kind="rows", robot="humanoid", worlds=4096, precision="fp64",
             point="contact_midpoint", weight="diag_delassus"),
        # the same on a small batch of another robot and in the other modes
        dict(name="rows-quadruped-250", kind="rows", robot="quadruped", worlds=250, precision="fp64",
             point="witness_point", weight="body_inertia"),
        # the contact solve alone: the reference's method on the headline batch
        dict(name="solve-35x4096-fp64", kind="solve", dofs=35, contacts=32, worlds=4096, precision="fp64",
             line_search="armijo_decay"),
        # ... with the FP32 Hessian on quadrupeds, a batch size that is no
        # multiple of anything, the exact line search
        dict(name="solve-18x3001-fp32", kind="solve", dofs=18, contacts=16, worlds=3001, precision="fp32",
             line_search="exact_root"),
        # ... on a robot without a specialised kernel
        dict(name="solve-27x777-fp64", kind="solve", dofs=27, contacts=24, worlds=777, precision="fp64",
             line_search="monotone_decay"),
        # an uneven batch in one launch: arms with a box (13 DOFs), quadrupeds
        # (18) and humanoids (35), each world at its own DOF count
        dict(name="solve-uneven-6000-fp32", kind="uneven", worlds=6000, contacts=64, precision="fp32",
             line_search="armijo_decay"),
        # clutter: worlds of 64 stacked free boxes, 384 DOFs, about 400 contacts
        dict(name="solve-boxes64-296-fp32", kind="boxes", boxes=64, contacts=448, worlds=296, precision="fp32",
             line_search="armijo_decay"),
        # contacts of stacked boxes found anew from the pose
        dict(name="contacts-boxes64-256", kind="contacts", boxes=64, worlds=256),
        # training the warm-start network, at the batch its training uses
        dict(name="train-8192", kind="train", batch=8192),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["rollout", "rollout", "rows", "solve", "solve", "solve", "uneven", "boxes", "contacts", "train"])
    precision = rng.choice(["fp64", "fp32"])
    search = rng.choice(["armijo_decay", "armijo_decay", "monotone_decay", "exact_root"])
    if kind == "rollout":
        robot = rng.choice(["humanoid", "quadruped", "arm_boxes"])
        c = dict(kind=kind, robot=robot, worlds=_log_int(rng, 1, 512 if robot == "arm_boxes" else 4000),
                 steps=rng.randint(1, 3) if robot == "arm_boxes" else rng.randint(2, 7), precision=precision,
                 warm_start=rng.choice(["previous_velocity", "previous_impulses", "learned"]), graph=False)
        if robot == "arm_boxes":
            c["boxes"] = rng.randint(4, 9)
            c["warm_start"] = rng.choice(["previous_velocity", "previous_impulses"])
        elif rng.random() < 0.5:
            c["steps"], c["graph"] = 2 * rng.randint(1, 3), True
        return c
    if kind == "rows":
        return dict(kind=kind, robot=rng.choice(["humanoid", "quadruped", "arm_boxes"]), boxes=rng.randint(2, 7),
                    worlds=_log_int(rng, 16, 800), precision="fp64",
                    point=rng.choice(["contact_midpoint", "witness_point"]),
                    weight=rng.choice(["diag_delassus", "body_inertia"]))
    if kind == "solve":
        return dict(kind=kind, dofs=rng.choice([35, 18, rng.randint(7, 44)]), contacts=rng.randint(6, 32),
                    worlds=_log_int(rng, 4, 4096), precision=precision, line_search=search)
    if kind == "uneven":
        return dict(kind=kind, worlds=_log_int(rng, 48, 6000), contacts=rng.randint(24, 64), precision=precision,
                    line_search=search)
    if kind == "boxes":
        boxes = rng.randint(12, 64)
        return dict(kind=kind, boxes=boxes, contacts=7 * boxes, worlds=_log_int(rng, 8, 296), precision=precision,
                    line_search=search)
    if kind == "contacts":
        return dict(kind=kind, boxes=rng.randint(8, 64), worlds=_log_int(rng, 4, 256))
    return dict(kind="train", batch=_log_int(rng, 200, 20000))


# ---- inputs ----------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device=CUDA)
    g.manual_seed(int(seed))
    return g


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device=CUDA, dtype=F64)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=CUDA, dtype=F64)


def _scene(case: dict, seed: int):
    """(model, state, control, contacts, contact slots per world) of a rollout or rows case."""
    if case["robot"] == "arm_boxes":
        model, state, control, contacts = models.box_scene(case["worlds"], seed, CUDA, boxes=case["boxes"],
                                                           sites=(3, 5), arm=True)[:4]
        slots = 14 * case["boxes"]
    else:
        lo, hi = (8, 32) if case["robot"] == "humanoid" else (4, 16)
        model, state, control, contacts, _ = models.rollout_scene(case["robot"], case["worlds"], seed, CUDA,
                                                                  contacts=(lo, hi))
        slots = hi
    revolute = (model.joint_armature > 0).to(F64)  # the actuated joints: small torques
    control.joint_f.copy_(0.5 * revolute * _normal(_gen(seed), revolute.numel()))
    return model, state, control, contacts, slots


def _like(state: SapState) -> SapState:
    return SapState(joint_q=state.joint_q.clone(), joint_qd=state.joint_qd.clone(), body_q=state.body_q.clone(),
                    body_f=None if state.body_f is None else state.body_f.clone())


def _problem_of(tree: "Tree", q, body0, body1, counts, g, C: int, mu=(0.3, 1.0)) -> dict:
    """Dense stage-2 arrays of E worlds at coordinates q: contacts between
    body0 (or the ground, -1) and body1 at points within 5 cm of body1."""
    E, n = q.shape[0], tree.n
    pos, R, S = tree.poses(q)
    A = tree.mass_matrix(pos, R, S)
    world = torch.arange(E, device=CUDA)[:, None]
    d = _normal(g, E, C, 3)
    r = _uniform(g, 0.0, 0.05, E, C, 1) * d / d.norm(dim=-1, keepdim=True)
    x = pos[world, body1] + torch.einsum("ecij,ecj->eci", R[world, body1], r)
    nrm = _normal(g, E, C, 3)
    ground = (body0 < 0)[..., None]
    nrm = torch.where(ground, torch.tensor([0.0, 0.0, 1.0], dtype=F64, device=CUDA) + 0.1 * nrm, nrm)
    J = _rows(tree, S, body0, body1, x, x, _frame(nrm / nrm.norm(dim=-1, keepdim=True)))
    live = (torch.arange(C, device=CUDA)[None] < counts[:, None])
    J = J * live[..., None, None]
    v_star = 0.5 * _normal(g, E, n)
    z = lambda a: (a * live).contiguous()
    one = torch.ones(E, C, dtype=F64, device=CUDA)
    return dict(contact_count=counts.to(I32), dynamics_matrix=A.contiguous(), jacobian=J.contiguous(),
                phi0=z(_uniform(g, -2.0e-3, 0.0, E, C)), w_eff=z(_delassus_weight(J, A)), mu=z(_uniform(g, *mu, E, C)),
                stiffness=z(1.0e5 * one), tau_d=z(0.01 * one), v_star=v_star.reshape(-1).contiguous(),
                v0=(v_star + 0.01 * _normal(g, E, n)).reshape(-1).contiguous(),
                dt=torch.full((E,), DT, dtype=F64, device=CUDA))


def _chain_problem(dofs: int, E: int, C: int, counts, seed: int) -> dict:
    """A floating-base chain of dofs - 6 revolute joints per world, contacts
    against the ground on its distal half (the shape of the humanoid scenes)."""
    rng = np.random.default_rng(seed)
    g = _gen(seed)
    tree = Tree.of_template(models.world_template("humanoid", rng), bodies=min(dofs - 5, 30))
    if dofs > 35:  # longer chains than the humanoid's
        tree = tree.extended(dofs - 35, rng)
    q = torch.zeros(E, tree.nq, dtype=F64, device=CUDA)
    q[:, :3] = _uniform(g, -1.0, 1.0, E, 3)
    h = _normal(g, E, 4)
    q[:, 3:7] = h / h.norm(dim=-1, keepdim=True)
    q[:, 7:] = _uniform(g, -1.0, 1.0, E, tree.nq - 7)
    body1 = torch.randint(tree.B // 2, tree.B, (E, C), generator=g, device=CUDA)
    return _problem_of(tree, q, torch.full_like(body1, -1), body1, counts, g, C)


def _arm_box_problem(E: int, C: int, counts, seed: int) -> dict:
    """A fixed-base seven-joint arm whose last link grips a free box."""
    rng = np.random.default_rng(seed)
    g = _gen(seed)
    tree = Tree.of_template(models.world_template("arm_box", rng))
    q = torch.zeros(E, tree.nq, dtype=F64, device=CUDA)
    q[:, :7] = _uniform(g, -1.0, 1.0, E, 7)
    q[:, 13] = 1.0
    q[:, 7:10] = tree.poses(q)[0][:, 6] + 0.03 * _normal(g, E, 3)
    h = _normal(g, E, 4)
    q[:, 10:14] = h / h.norm(dim=-1, keepdim=True)
    body1 = torch.full((E, C), 7, device=CUDA)
    return _problem_of(tree, q, torch.full_like(body1, 6), body1, counts, g, C)


def _uneven_problem(case: dict, seed: int):
    """(the three homogeneous problems, the one batch they make)."""
    E, C = case["worlds"], case["contacts"]
    sizes = [E // 3, E // 3, E - 2 * (E // 3)]
    rng = np.random.default_rng(seed)
    poisson = lambda k: torch.as_tensor(np.clip(rng.poisson(12.0, size=k), 1, C), device=CUDA)
    parts = [_arm_box_problem(sizes[0], 8, torch.as_tensor(rng.integers(2, 9, size=sizes[0]), device=CUDA), seed),
             _chain_problem(18, sizes[1], C, poisson(sizes[1]), seed + 1),
             _chain_problem(35, sizes[2], C, poisson(sizes[2]), seed + 2)]
    n = 35
    A = torch.zeros(E, n * n, dtype=F64, device=CUDA)
    J = torch.zeros(E, C * 3 * n, dtype=F64, device=CUDA)
    out = {k: torch.zeros(E, C, dtype=F64, device=CUDA) for k in ("phi0", "w_eff", "mu", "stiffness", "tau_d")}
    out |= {k: torch.zeros(E, n, dtype=F64, device=CUDA) for k in ("v_star", "v0")}
    dofs = torch.zeros(E, dtype=I32, device=CUDA)
    e0 = 0
    for p in parts:
        k, m = p["dynamics_matrix"].shape[:2]
        c = p["phi0"].shape[1]
        rows = slice(e0, e0 + k)
        A[rows, :m * m] = p["dynamics_matrix"].reshape(k, -1)
        J[rows, :c * 3 * m] = p["jacobian"].reshape(k, -1)
        for name in ("phi0", "w_eff", "mu", "stiffness", "tau_d"):
            out[name][rows, :c] = p[name]
        for name in ("v_star", "v0"):
            out[name][rows, :m] = p[name].reshape(k, m)
        dofs[rows] = m
        e0 += k
    count = torch.cat([p["contact_count"] for p in parts])
    work = dofs.to(F64) ** 3 / 3 + count * dofs.to(F64) ** 2
    batch = dict(contact_count=count, dynamics_matrix=A, jacobian=J, dof_count=dofs,
                 world_order=torch.argsort(-work, stable=True).to(I32),
                 dt=torch.full((E,), DT, dtype=F64, device=CUDA),
                 **{k: v.reshape(-1) if k in ("v_star", "v0") else v for k, v in out.items()})
    return parts, batch


def _boxes_problem(case: dict, seed: int) -> dict:
    """Tree-blocked arrays of worlds of stacked boxes: up to 24 different
    stacks, repeated over the batch with velocities, penetrations and friction
    of each world's own."""
    E, T, C = case["worlds"], case["boxes"], case["contacts"]
    few = max(3, T // 4)
    base = scenes.box_stack_problem(min(E, 24), seed, boxes=T, max_contacts=C, sites=(few - few // 4, few + few // 4))
    g = _gen(seed)
    k = base.num_envs
    idx = torch.arange(E, device=CUDA) % k
    t = lambda a, dt=F64: torch.as_tensor(a, dtype=dt).to(CUDA)[idx].contiguous()
    count = t(base.contact_count, I32)
    live = (torch.arange(C, device=CUDA)[None] < count[:, None]).to(F64)
    fall = t((base.v_star - base.v0).reshape(k, -1))
    v0 = 0.05 * _normal(g, E, 6 * T)
    return dict(contact_count=count, tree_mass=t(base.tree_mass), jacobian=t(base.jacobian),
                contact_tree=t(base.contact_tree, I32), phi0=_uniform(g, -2.0e-3, 0.0, E, C) * live,
                w_eff=t(base.w_eff), mu=_uniform(g, 0.3, 1.0, E, C) * live, stiffness=t(base.stiffness),
                tau_d=t(base.tau_d), v_star=(v0 + fall).reshape(-1), v0=v0.reshape(-1), dt=t(base.dt))


def _box_poses(case: dict, seed: int):
    """(model, joint coordinates, shapes) of worlds of stacked boxes over a ground plane."""
    E, T = case["worlds"], case["boxes"]
    rng = np.random.default_rng(seed)
    few = max(3, T // 4)
    _, _, _, _, _, host = models.box_scene(min(E, 12), seed, CUDA, boxes=T, sites=(few - few // 4, few + few // 4))
    idx = np.arange(E) % host["q"].shape[0]
    q, dims = host["q"][idx].reshape(E, T, 7), host["dims"][idx].reshape(E * T, 3)
    q[..., :3] += rng.normal(scale=2.0e-4, size=(E, T, 3))
    tpl = host["tpl"]
    model = models.to_model(tpl, models.replicate(tpl, E, rng), q.reshape(E, -1), CUDA)
    X = np.zeros((E * T + 1, 7))
    X[:, 6] = 1.0
    X[:-1, 2] = 0.5 * dims[:, 2]
    scale = np.zeros((E * T + 1, 3))
    scale[:-1] = 0.5 * dims
    shapes = ShapeSet(num_worlds=E, shapes_per_world=T, num_global_shapes=1,
                      shape_type=np.concatenate([np.full(E * T, 2), [0]]).astype(np.int32), shape_scale=scale,
                      shape_X_bs=X, shape_body=np.concatenate([np.arange(E * T), [-1]]).astype(np.int32))
    return model, torch.as_tensor(q.reshape(-1), dtype=F64, device=CUDA), shapes


def _train_data(case: dict, seed: int):
    """(parameters, standardised inputs, targets) of one training batch."""
    g = _gen(seed)
    raw = torch.randn(case["batch"], 12, generator=g, device=CUDA, dtype=F32)
    mix = torch.randn(12, 3, generator=g, device=CUDA, dtype=F32) / 3.0
    target = torch.tanh(raw @ mix) + 0.1 * torch.randn(case["batch"], 3, generator=g, device=CUDA, dtype=F32)
    return raw, target.contiguous()


# ---- what a program holds before the call ------------------------------------------
class _State:
    pass


def prepare(case: dict, seed: int):
    s = _State()
    s.case, kind = case, case["kind"]
    if kind == "rollout":
        s.model, s.start, s.control, s.contacts, slots = _scene(case, seed)
        s.solver = SolverSAP(s.model, max_rigid_contact=slots, contact_preset_variant="drake",
                             hessian_precision=case["precision"], warm_start=case["warm_start"])
        s.a, s.b = _like(s.start), _like(s.start)
        s.graph = s.solver.capture_steps(s.a, s.b, s.control, s.contacts, DT) if case["graph"] else None
    elif kind == "rows":
        s.model, s.start, s.control, s.contacts, slots = _scene(case, seed)
        s.rows = SapContactJacobian(s.model, max_rigid_contact=slots, contact_point_mode=case["point"],
                                    contact_weight_mode=case["weight"], tree_blocked=False)
        s.rows.set_dt(DT)
    elif kind in ("solve", "uneven"):
        if kind == "solve":
            s.arrays = _solve_inputs(case, seed)
            n = case["dofs"]
        else:
            s.arrays, n = _uneven_problem(case, seed)[1], 35
        s.buffers = ContactSolveBuffers(case["worlds"], n, case["contacts"], CUDA)
        s.options = _options(case)
    elif kind == "boxes":
        s.arrays = _boxes_problem(case, seed)
        s.buffers = ContactSolveBuffers(case["worlds"], 6 * case["boxes"], case["contacts"], CUDA)
        s.options = _options(case)
    elif kind == "contacts":
        s.model, s.q, shapes = _box_poses(case, seed)
        view = SapContactJacobian(s.model, max_rigid_contact=1).view
        s.generator = ContactGenerator(shapes, view, capacity=16 * case["boxes"] * case["worlds"], gap=1.0e-3)
    else:
        raw, s.target = _train_data(case, seed)
        s.x = FeatureNorm.identity().encode(raw)
        s.mlp = WarmStartMLP(CUDA, seed=seed)
        s.buffers = TrainBuffers(case["batch"], CUDA)
    return s


def _options(case: dict):
    """The reference's tolerances; monotone_decay, whose own cost test stops
    far from the minimum, with the cost tolerance of the other searches."""
    return make_options(case["line_search"], hessian_precision=case["precision"],
                        linear_solve_precision=case["precision"],
                        cost_rel_tol=1.0e-15 if case["line_search"] == "monotone_decay" else None)


def _solve_inputs(case: dict, seed: int) -> dict:
    E, C = case["worlds"], case["contacts"]
    counts = torch.randint(max(1, C // 4), C + 1, (E,), generator=_gen(seed + 7), device=CUDA)
    return _chain_problem(case["dofs"], E, C, counts, seed)


def run(s):
    kind = s.case["kind"]
    if kind == "rollout":
        s.solver.reset_runtime_state()
        s.a.joint_q.copy_(s.start.joint_q)
        s.a.joint_qd.copy_(s.start.joint_qd)
        a, b = s.a, s.b
        if s.graph is not None:
            for _ in range(s.case["steps"] // 2):
                s.graph.replay()
        else:
            for _ in range(s.case["steps"]):
                s.solver.step(a, b, s.control, s.contacts, DT)
                a, b = b, a
        return {"joint_q": a.joint_q, "joint_qd": a.joint_qd}
    if kind == "rows":
        r = s.rows.compute(s.start, s.contacts, control=s.control)
        return {"v_star": s.rows.v_star, "A": r.dynamics_matrix_env, "J": r.contact_env_jacobian,
                "phi0": r.contact_env_phi0, "w": r.contact_env_w_eff, "mu": r.contact_env_mu,
                "stiffness": r.contact_env_stiffness, "count": r.contact_env_count}
    if kind in ("solve", "uneven"):
        b = contact_solve(**s.arrays, buffers=s.buffers, options=s.options)
        return {"v": b.v, "gamma": b.contact_gamma, "cost": b.cost, "converged": b.converged}
    if kind == "boxes":
        b = blocked_contact_solve(**s.arrays, buffers=s.buffers, options=s.options, trees_per_env=s.case["boxes"])
        return {"v": b.v, "gamma": b.contact_gamma, "cost": b.cost, "converged": b.converged}
    if kind == "contacts":
        c = s.generator.generate(s.q)
        return {"count": c.rigid_contact_count, "shape0": c.rigid_contact_shape0, "shape1": c.rigid_contact_shape1,
                "point0": c.rigid_contact_point0d, "point1": c.rigid_contact_point1d,
                "normal": c.rigid_contact_normald, "point1_f32": c.rigid_contact_point1}
    loss = s.mlp.train_step(s.x, s.target, s.buffers, lr=1.0e-3)
    return {"loss": loss, "grad": s.mlp.grad, "params": s.mlp.params}


# ---- the work no implementation can leave out ---------------------------------------
def _solve_work(E: float, n: float, C: float, newton: float) -> tuple[float, float]:
    """Bytes and FP64 operations of E dense solves with C contacts on average:
    each input read and each output written once; per Newton iteration the
    Hessian, its factor, and the products with A and J."""
    b = 8 * (n * n + 3 * C * n + 3 * n + 5 * C) + 8 * (n + 3 * C)
    f = newton * (6 * C * n * n + n ** 3 / 3 + 6 * n * n + 18 * C * n)
    return E * b, E * f


def work(case: dict) -> dict:
    kind, E = case["kind"], case.get("worlds", 0)
    if kind in ("rollout", "rows"):
        if case["robot"] == "arm_boxes":
            B, n, C = 7 + case["boxes"], 7 + 6 * case["boxes"], 7.5 * case["boxes"]
            row, a = 14.0, 49 * (1 + case["boxes"])
        else:
            B, n, C = (30, 35, 20) if case["robot"] == "humanoid" else (13, 18, 10)
            row, a = n, n * n
        if kind == "rows":
            row, a = n, n * n
        state = 8 * (2 * n + 1) * 2
        model = 8 * B * (3 + 7 + 7 + 13 + 1) + 8 * C * 11
        rows = 8 * (a + 3 * C * row + 5 * C + n)
        f = 60.0 * B + 12 * n * n + 40 * C * row + n ** 3 / 3
        if kind == "rows":
            return {"bytes": E * (state + model + rows), "flops": E * f}
        # a step reads the state, model and contacts and writes the new state
        steps = case["steps"]
        newton = 4 if case["robot"] != "arm_boxes" else 12
        return {"bytes": steps * E * (state + model), "flops": steps * E * (f + newton * (6 * C * row * row + a * 10))}
    if kind == "solve":
        b, f = _solve_work(E, case["dofs"], 0.625 * case["contacts"], 4)
        return {"bytes": b, "flops": f}
    if kind == "uneven":
        parts = [_solve_work(E / 3, n, C, 4) for n, C in ((13, 5), (18, 12), (35, 12))]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if kind == "boxes":
        T = case["boxes"]
        C = 6.2 * T
        b = 8 * (36 * T + 36 * C + 3 * 6 * T + 5 * C) + 8 * (6 * T + 3 * C)
        return {"bytes": E * b, "flops": E * 40.0 * (C * 6 * 12 * 12 + T * 6 ** 3 * 4)}
    if kind == "contacts":
        T = case["boxes"]
        return {"bytes": E * (T * 8 * (7 + 7 + 10) + 6.5 * T * (13 * 8 + 8)), "flops": E * T * T / 2 * 30.0}
    params = 12 * 128 + 2 * 128 * 128 + 3 * 128 + 3 * 128 + 3
    return {"bytes": case["batch"] * (16 * 2 + 3 * 4) + params * 4 * 7, "flops": 6.0 * case["batch"] * params}


# ---- the same in plain FP64 torch ------------------------------------------------------
def _cross(a, b):
    return torch.linalg.cross(*torch.broadcast_tensors(a, b))


def _quat_matrix(q):
    """Rotation matrices of the quaternions (x, y, z, w)."""
    x, y, z, w = (q / q.norm(dim=-1, keepdim=True)).unbind(-1)
    return torch.stack([torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], -1),
                        torch.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], -1),
                        torch.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1)], -2)


def _axis_matrix(axis, angle):
    h = 0.5 * angle
    return _quat_matrix(torch.cat([axis * torch.sin(h)[..., None], torch.cos(h)[..., None]], -1))


def _frame(nrm):
    """Rows (t1, t2, n): the axis of the smallest component of n leads."""
    a = nrm.abs()
    i = a.argmin(-1)
    u = torch.gather(nrm, -1, i[..., None])[..., 0]
    mag = torch.sqrt(1 - u * u)
    r = 1 / mag
    s = -r * u
    x, y, z = nrm.unbind(-1)
    o = torch.zeros_like(x)
    pick = lambda p, q, t: torch.where((i == 0)[..., None], p, torch.where((i == 1)[..., None], q, t))
    st = lambda *c: torch.stack(c, -1)
    t1 = pick(st(o, -r * z, r * y), st(r * z, o, -r * x), st(-r * y, r * x, o))
    t2 = pick(st(mag, s * y, s * z), st(s * x, mag, s * z), st(s * x, s * y, mag))
    return torch.stack([t1, t2, nrm], -2)


class Tree:
    """One world's bodies: revolute joints (one per body) and free ones, each
    body's frame at its joint; masses may differ between worlds."""

    def __init__(self, parent, free, axis, X_p, mass, inertia, com, armature):
        t = lambda a: torch.as_tensor(np.asarray(a), dtype=F64, device=CUDA)
        self.parent, self.free = [int(p) for p in parent], [bool(f) for f in free]
        self.B = len(self.parent)
        self.axis, self.X_p = t(axis), t(X_p)  # axis per body (unused where free)
        self.mass, self.inertia, self.com = t(mass), t(inertia), t(com)  # (B, ..) or (E, B, ..)
        self.armature = t(armature)
        self.ds, self.qs, d, q = [], [], 0, 0
        for f in self.free:
            self.ds.append(d)
            self.qs.append(q)
            d, q = d + (6 if f else 1), q + (7 if f else 1)
        self.n, self.nq = d, q
        anc = np.zeros((self.B, d))
        for b in range(self.B):
            k = b
            while k >= 0:
                anc[b, self.ds[k]:self.ds[k] + (6 if self.free[k] else 1)] = 1.0
                k = self.parent[k]
        self.anc = t(anc)

    @classmethod
    def of_template(cls, tpl: dict, bodies: int | None = None) -> "Tree":
        B = bodies or tpl["bodies_per_world"]
        free = tpl["joint_type"][:B] == SAP_JOINT_FREE
        n = int(tpl["joint_qd_start"][B])
        axis = [tpl["joint_axis"][tpl["joint_qd_start"][b]] for b in range(B)]
        return cls(tpl["joint_parent"][:B], free, axis, tpl["joint_X_p"][:B], tpl["body_mass"][:B],
                   tpl["body_inertia"][:B], tpl["body_com"][:B], tpl["joint_armature"][:n])

    @classmethod
    def of_model(cls, m) -> "Tree":
        E = int(m.world_count)
        B, n = int(m.body_count) // E, int(m.joint_dof_count) // E
        ds = m.joint_qd_start[:B].cpu().numpy()
        return cls(m.joint_parent[:B].cpu().numpy(), m.joint_type[:B].cpu().numpy() == SAP_JOINT_FREE,
                   m.joint_axis[:n].cpu().numpy()[ds], m.joint_X_p[:B].cpu().numpy(),
                   m.body_mass.reshape(E, B).cpu().numpy(), m.body_inertia.reshape(E, B, 3, 3).cpu().numpy(),
                   m.body_com.reshape(E, B, 3).cpu().numpy(), m.joint_armature[:n].cpu().numpy())

    def extended(self, more: int, rng) -> "Tree":
        """The chain with `more` links like its last one appended."""
        c = lambda a: a.cpu().numpy()
        axis = rng.normal(size=(more, 3))
        axis /= np.linalg.norm(axis, axis=1, keepdims=True)
        rep = lambda a: np.concatenate([c(a), np.repeat(c(a)[-1:], more, 0)])
        return Tree(self.parent + list(range(self.B - 1, self.B - 1 + more)), self.free + [False] * more,
                    np.concatenate([c(self.axis), axis]), rep(self.X_p), rep(self.mass), rep(self.inertia),
                    rep(self.com), rep(self.armature))

    def poses(self, q):
        """Body origins (E, B, 3), rotations (E, B, 3, 3) and the motion
        subspace columns (E, n, 6), [omega; velocity at the world origin]."""
        E = q.shape[0]
        pos, R, S = [], [], torch.zeros(E, self.n, 6, dtype=F64, device=CUDA)
        eye = torch.eye(3, dtype=F64, device=CUDA)
        for b in range(self.B):
            k, d = self.qs[b], self.ds[b]
            Xp, Xr = self.X_p[b, :3].expand(E, 3), _quat_matrix(self.X_p[b, 3:]).expand(E, 3, 3)
            if self.parent[b] >= 0:
                p = self.parent[b]
                Xp, Xr = pos[p] + torch.einsum("eij,ej->ei", R[p], Xp), R[p] @ Xr
            if self.free[b]:
                w = Xr
                Xp, Xr = Xp + torch.einsum("eij,ej->ei", Xr, q[:, k:k + 3]), Xr @ _quat_matrix(q[:, k + 3:k + 7])
                for a in range(3):
                    e = torch.einsum("eij,j->ei", w, eye[a])
                    S[:, d + a, :3], S[:, d + a, 3:] = e, _cross(Xp, e)
                    S[:, d + 3 + a, 3:] = e
            else:
                w = torch.einsum("eij,j->ei", Xr, self.axis[b])
                S[:, d, :3], S[:, d, 3:] = w, _cross(Xp, w)
                Xr = Xr @ _axis_matrix(self.axis[b].expand(E, 3), q[:, k])
            pos.append(Xp)
            R.append(Xr)
        return torch.stack(pos, 1), torch.stack(R, 1), S

    def inertias(self, pos, R):
        """6 x 6 spatial inertias about the world origin (E, B, 6, 6)."""
        E, B = pos.shape[:2]
        m = self.mass.expand(E, B)
        c = pos + torch.einsum("ebij,ebj->ebi", R, self.com.expand(E, B, 3))
        eye = torch.eye(3, dtype=F64, device=CUDA)
        cx = torch.linalg.cross(c[..., None, :].expand(E, B, 3, 3), eye.expand(E, B, 3, 3)).transpose(-1, -2)  # [c]x
        I = torch.zeros(E, B, 6, 6, dtype=F64, device=CUDA)
        I[..., :3, :3] = R @ self.inertia.expand(E, B, 3, 3) @ R.transpose(-1, -2) + m[..., None, None] * (
            (c * c).sum(-1)[..., None, None] * eye - c[..., :, None] * c[..., None, :])
        I[..., :3, 3:] = m[..., None, None] * cx
        I[..., 3:, :3] = -m[..., None, None] * cx
        I[..., 3:, 3:] = m[..., None, None] * eye
        return I

    def mass_matrix(self, pos, R, S):
        A = torch.diag_embed(self.armature.expand(pos.shape[0], self.n).clone())
        I = self.inertias(pos, R)
        for b in range(self.B):
            Jb = S * self.anc[b][:, None]
            A += Jb @ I[:, b] @ Jb.transpose(1, 2)
        return 0.5 * (A + A.transpose(1, 2))

    def free_motion(self, q, qd, joint_f, gravity, dt):
        """(v*, A, body origins, rotations, S) of one step."""
        E = q.shape[0]
        pos, R, S = self.poses(q)
        A = self.mass_matrix(pos, R, S)
        I = self.inertias(pos, R)
        vj = S * qd[..., None]
        V = torch.einsum("bn,enk->ebk", self.anc, vj)
        bias = torch.zeros(E, self.B, 6, dtype=F64, device=CUDA)
        for b in range(self.B):
            d = self.ds[b]
            if self.free[b]:
                w, v = qd[:, d:d + 3], qd[:, d + 3:d + 6]
                bias[:, b, 3:] = _cross(v, w)
            elif self.parent[b] >= 0:
                Vp, s = V[:, self.parent[b]], vj[:, d]
                bias[:, b, :3] = _cross(Vp[:, :3], s[:, :3])
                bias[:, b, 3:] = _cross(Vp[:, :3], s[:, 3:]) + _cross(Vp[:, 3:], s[:, :3])
        up = torch.stack([self.anc[:, d] for d in self.ds], 1)  # (B, B): whether a body is an ancestor-or-self
        acc = torch.einsum("bk,ekr->ebr", up, bias)
        acc[..., 3:] -= gravity[:, None]
        h = torch.einsum("ebij,ebj->ebi", I, V)
        f = torch.einsum("ebij,ebj->ebi", I, acc)
        f[..., :3] += _cross(V[..., :3], h[..., :3]) + _cross(V[..., 3:], h[..., 3:])
        f[..., 3:] += _cross(V[..., :3], h[..., 3:])
        tau = joint_f - torch.einsum("enk,bn,ebk->en", S, self.anc, f)
        vdot = torch.linalg.solve(A, tau)
        return qd + dt * vdot, A, pos, R, S

    def integrate(self, q, v, dt):
        out = q.clone()
        for b in range(self.B):
            k, d = self.qs[b], self.ds[b]
            if not self.free[b]:
                out[:, k] = q[:, k] + dt * v[:, d]
                continue
            out[:, k:k + 3] = q[:, k:k + 3] + dt * v[:, d + 3:d + 6]
            h, w = q[:, k + 3:k + 7], v[:, d:d + 3]
            dq = torch.cat([h[:, 3:] * w + _cross(w, h[:, :3]), -(w * h[:, :3]).sum(-1, keepdim=True)], -1)
            h = h + 0.5 * dt * dq
            out[:, k + 3:k + 7] = h / h.norm(dim=-1, keepdim=True)
        return out


def _rows(tree, S, body0, body1, x0, x1, frame):
    """Contact rows (E, C, 3, n); body -1 is the static world."""
    J = 0.0
    for sign, body, x in ((-1.0, body0, x0), (1.0, body1, x1)):
        on = tree.anc[body.clamp(min=0)] * (body >= 0)[..., None] * sign  # (E, C, n)
        vel = S[:, None, :, 3:] + _cross(S[:, None, :, :3], x[:, :, None, :])
        J = J + torch.einsum("ecri,ecni,ecn->ecrn", frame, vel, on)
    return J


def _delassus_weight(J, A):
    d = 1.0 / torch.diagonal(A, dim1=1, dim2=2).clamp(min=1e-12)
    W = torch.einsum("ecrn,en,ecsn->ecrs", J, d, J)
    return (W.flatten(-2).norm(dim=-1) / 3.0).clamp(min=1e-12)


def _scene_rows(tree, model, contacts, C, pos, R, S, A, point, weight):
    """The per-world contact slots (flat order) at the given poses."""
    E, B = pos.shape[:2]
    N = int(contacts.rigid_contact_count.item())
    sh0, sh1 = contacts.rigid_contact_shape0[:N].long(), contacts.rigid_contact_shape1[:N].long()
    g0, g1 = model.shape_body[sh0].long(), model.shape_body[sh1].long()
    world = torch.where(g0 >= 0, g0, g1) // B
    order = torch.argsort(world, stable=True)
    world = world[order]
    count = torch.bincount(world, minlength=E)
    slot = torch.arange(N, device=CUDA) - (torch.cumsum(count, 0) - count)[world]
    keep = slot < C
    order, world, slot = order[keep], world[keep], slot[keep]

    def put(a, fill=0):
        out = torch.full((E, C) + a.shape[1:], fill, dtype=a.dtype, device=CUDA)
        out[world, slot] = a[order]
        return out

    local = lambda b: torch.where(b >= 0, b % B, b)
    b0, b1 = put(local(g0), -1), put(local(g1), -1)
    ev = torch.arange(E, device=CUDA)[:, None]
    at = lambda b, x: torch.where((b >= 0)[..., None], pos[ev, b.clamp(min=0)] + torch.einsum(
        "ecij,ecj->eci", R[ev, b.clamp(min=0)], x), x)
    x0, x1 = at(b0, put(contacts.rigid_contact_point0d[:N])), at(b1, put(contacts.rigid_contact_point1d[:N]))
    nrm = put(contacts.rigid_contact_normald[:N])
    live = put(torch.ones(N, dtype=F64, device=CUDA))
    nrm = torch.where((live > 0)[..., None], nrm, torch.tensor([0.0, 0.0, 1.0], dtype=F64, device=CUDA))
    nrm = nrm / nrm.norm(dim=-1, keepdim=True)
    F = _frame(nrm)
    k0, k1 = put(model.shape_material_ke[sh0]), put(model.shape_material_ke[sh1])
    m0, m1 = put(model.shape_material_mu[sh0]), put(model.shape_material_mu[sh1])
    t0, t1 = put(model.shape_material_tau[sh0]), put(model.shape_material_tau[sh1])
    den = (k0 + k1).clamp(min=1e-300)
    mid = (k0 / den)[..., None] * x0 + (k1 / den)[..., None] * x1
    p0, p1 = (mid, mid) if point == "contact_midpoint" else (x0, x1)
    J = _rows(tree, S, b0, b1, p0, p1, F) * live[..., None, None]
    if weight == "diag_delassus":
        w = _delassus_weight(J, A)
    else:
        w = 0.0
        for b, x in ((b0, x0), (b1, x1)):
            k = b.clamp(min=0)
            mass, Ib = tree.mass.expand(E, B)[ev, k], tree.inertia.expand(E, B, 3, 3)[ev, k]
            Rb = R[ev, k]
            r = x - pos[ev, k] - torch.einsum("ecij,ecj->eci", Rb, tree.com.expand(E, B, 3)[ev, k])
            cb = torch.einsum("ecij,ecri->ecrj", Rb, _cross(r[:, :, None], F))
            inv = 1.0 / torch.diagonal(Ib, dim1=-2, dim2=-1).clamp(min=1e-12)
            w = w + (b >= 0) * (1.0 / mass[..., None] + (cb * cb * inv[:, :, None]).sum(-1)).sum(-1)
        w = (w / 3.0).clamp(min=1e-12)
    return dict(contact_count=count.to(I32), dynamics_matrix=A, jacobian=J, phi0=((x1 - x0) * nrm).sum(-1) * live,
                w_eff=w * live, mu=2 * m0 * m1 / (m0 + m1).clamp(min=1e-300) * live, stiffness=k0 * k1 / den * live,
                tau_d=(t0 + t1) * live)


def _project(p, vc, want):
    """Regularized friction-cone projection at contact velocities vc (E, C, 3):
    impulses, costs and (want) the 3 x 3 derivatives."""
    y = torch.stack([-vc[..., 0] / p["rt"], -vc[..., 1] / p["rt"], (p["vhat"] - vc[..., 2]) / p["rn"]], -1)
    yt, yn, mu = y[..., :2], y[..., 2], p["mu"]
    yr = torch.sqrt((yt * yt).sum(-1) + 1.0e-14)
    t = yt / yr[..., None]
    live = p["live"]
    stick = live & (yr <= mu * yn)
    slide = live & ~stick & (-p["mu_hat"] * yr < yn) & (yn < yr / mu)
    gn = (yn + p["mu_hat"] * yr) * p["factor"]
    zero = torch.zeros_like(yn)
    g = torch.where(stick[..., None], y, torch.where(
        slide[..., None], torch.cat([(mu * gn)[..., None] * t, gn[..., None]], -1), torch.zeros_like(y)))
    cost = 0.5 * (p["rt"] * (g[..., :2] ** 2).sum(-1) + p["rn"] * g[..., 2] ** 2)
    if not want:
        return g, cost, None
    G = torch.zeros(*yn.shape, 3, 3, dtype=F64, device=vc.device)
    P = t[..., :, None] * t[..., None, :]
    eye = torch.eye(2, dtype=F64, device=vc.device)
    D = mu[..., None, None] * ((gn / yr)[..., None, None] * (eye - P) + (p["mu_hat"] * p["factor"])[..., None, None] * P)
    pick = lambda a, b: torch.where(stick, a, torch.where(slide, b, zero))
    for i in range(2):
        for j in range(2):
            G[..., i, j] = pick(eye[i, j] / p["rt"], D[..., i, j] / p["rt"])
        G[..., i, 2] = pick(zero, mu * p["factor"] * t[..., i] / p["rn"])
        G[..., 2, i] = pick(zero, p["mu_hat"] * p["factor"] * t[..., i] / p["rt"])
    G[..., 2, 2] = pick(1 / p["rn"], p["factor"] / p["rn"])
    return g, cost, G


def _minimize(a: dict, v0=None):
    """(v, gamma, cost) at the minimum of the stage-2 objective: dense Newton
    with a line search by bisection, until no world improves."""
    A, J = a["dynamics_matrix"], a["jacobian"]
    E, n = A.shape[:2]
    C = J.shape[1]
    vs = a["v_star"].reshape(E, n)
    w = a["w_eff"].clamp(min=1e-12)
    dt = a["dt"].reshape(E, 1)
    rn = torch.maximum(w / (4 * math.pi ** 2), 1.0 / (dt * torch.where(a["stiffness"] > 0, a["stiffness"], 1.0)
                                                       * (dt + a["tau_d"])))
    rt = 1.0e-3 * w
    mu = a["mu"]
    p = dict(rt=rt, rn=rn, vhat=-a["phi0"] / (dt + a["tau_d"]), mu=mu.clamp(min=1e-300), mu_hat=mu * rt / rn,
             factor=1.0 / (1.0 + mu * mu * rt / rn),
             live=torch.arange(C, device=CUDA)[None] < a["contact_count"][:, None])
    Jf = J.reshape(E, 3 * C, n)
    mul = lambda M, x: torch.bmm(M, x[..., None])[..., 0]
    v = (vs if v0 is None else v0.reshape(E, n)).clone()
    best, stall = torch.full((E,), math.inf, dtype=F64, device=CUDA), 0
    scale = 1.0 / torch.sqrt(torch.diagonal(A, dim1=1, dim2=2))
    keep = v.clone()
    for _ in range(400):
        vc = mul(Jf, v).reshape(E, C, 3)
        g, _, G = _project(p, vc, True)
        ares, jg = mul(A, v - vs), torch.einsum("eki,ek->ei", Jf, g.reshape(E, -1))
        grad = ares - jg
        size = (scale * grad).norm(dim=1) / torch.maximum((scale * mul(A, v)).norm(dim=1),
                                                          (scale * jg).norm(dim=1)).clamp(min=1e-300)
        better = size < 0.9 * best
        keep = torch.where((size < best)[:, None], v, keep)
        best = torch.minimum(best, size)
        stall = 0 if bool((better & (size > 1e-14)).any()) else stall + 1
        if stall >= (4 if bool((best < 1e-11).all()) else 40):
            break
        GJ = torch.einsum("ecij,ecjn->ecin", G, J).reshape(E, 3 * C, n)
        H = A + torch.bmm(Jf.transpose(1, 2), GJ)
        L = torch.linalg.cholesky(0.5 * (H + H.transpose(1, 2)))
        dv = -torch.cholesky_solve(grad[..., None], L)[..., 0]
        dvc = mul(Jf, dv).reshape(E, C, 3)
        q1, q2 = (dv * ares).sum(1), (dv * mul(A, dv)).sum(1)

        def slope(al):
            gl, _, _ = _project(p, vc + al[:, None, None] * dvc, False)
            return q1 + al * q2 - (gl * dvc).sum((1, 2))

        one = torch.ones(E, dtype=F64, device=CUDA)
        noise = 1e-14 * (q1.abs() + q2.abs())
        full = slope(one) <= noise  # still downhill at the full step: take it
        lo, hi = torch.zeros_like(one), one.clone()
        if not bool(full.all()):
            for _ in range(45):
                mid = 0.5 * (lo + hi)
                down = slope(mid) < 0
                lo, hi = torch.where(down, mid, lo), torch.where(down, hi, mid)
        al = torch.where(full | (best < 1e-10), one, 0.5 * (lo + hi))
        v = v + al[:, None] * dv
    v = keep
    vc = mul(Jf, v).reshape(E, C, 3)
    g, c, _ = _project(p, vc, False)
    cost = 0.5 * ((v - vs) * mul(A, v - vs)).sum(1) + c.sum(1)
    return v, g, cost


def _dense_boxes(a: dict, T: int, worlds) -> dict:
    """The tree-blocked problem of some worlds in the dense layout."""
    pick = lambda k: a[k][worlds]
    tm, Jb, ct = pick("tree_mass"), pick("jacobian"), pick("contact_tree").long()
    E, C = Jb.shape[:2]
    A = torch.zeros(E, T, 6, T, 6, dtype=F64, device=CUDA)
    i = torch.arange(T, device=CUDA)
    A[:, i, :, i, :] = tm.transpose(0, 1)
    J = torch.zeros(E, C, 3, T, 6, dtype=F64, device=CUDA)
    for s in range(2):
        e, c = torch.nonzero(ct[..., s] >= 0, as_tuple=True)
        J[e, c, :, ct[e, c, s]] += Jb[e, c, :, 6 * s:6 * s + 6]
    out = {k: pick(k) for k in ("contact_count", "phi0", "w_eff", "mu", "stiffness", "tau_d", "dt")}
    return dict(out, dynamics_matrix=A.reshape(E, 6 * T, 6 * T), jacobian=J.reshape(E, C, 3, 6 * T),
                v_star=a["v_star"].reshape(-1, 6 * T)[worlds])


def exact(case: dict, seed: int):
    kind, E = case["kind"], case.get("worlds", 0)
    if kind == "rollout":
        model, state, control, contacts, C = _scene(case, seed)
        tree = Tree.of_model(model)
        q, qd = state.joint_q.reshape(E, -1).clone(), state.joint_qd.reshape(E, -1).clone()
        for _ in range(case["steps"]):
            vs, A, pos, R, S = tree.free_motion(q, qd, control.joint_f.reshape(E, -1), model.gravity.reshape(E, 3), DT)
            a = _scene_rows(tree, model, contacts, C, pos, R, S, A, "contact_midpoint", "diag_delassus")
            qd = _minimize(dict(a, v_star=vs, dt=torch.full((E,), DT, dtype=F64, device=CUDA)), v0=qd)[0]
            q = tree.integrate(q, qd, DT)
        return {"joint_q": q.reshape(-1), "joint_qd": qd.reshape(-1)}
    if kind == "rows":
        model, state, control, contacts, C = _scene(case, seed)
        tree = Tree.of_model(model)
        q, qd = state.joint_q.reshape(E, -1), state.joint_qd.reshape(E, -1)
        vs, A, pos, R, S = tree.free_motion(q, qd, control.joint_f.reshape(E, -1), model.gravity.reshape(E, 3), DT)
        a = _scene_rows(tree, model, contacts, C, pos, R, S, A, case["point"], case["weight"])
        return {"v_star": vs.reshape(-1), "A": A, "J": a["jacobian"], "phi0": a["phi0"], "w": a["w_eff"],
                "mu": a["mu"], "stiffness": a["stiffness"], "count": a["contact_count"]}
    if kind == "solve":
        v, g, cost = _minimize(_solve_inputs(case, seed))
        return {"v": v.reshape(-1), "gamma": g, "cost": cost, "converged": None}
    if kind == "uneven":
        V = torch.zeros(E, 35, dtype=F64, device=CUDA)
        G = torch.zeros(E, case["contacts"], 3, dtype=F64, device=CUDA)
        costs, e0 = [], 0
        for p in _uneven_problem(case, seed)[0]:
            v, g, cost = _minimize(p)
            V[e0:e0 + len(v), :v.shape[1]] = v
            G[e0:e0 + len(v), :g.shape[1]] = g
            costs.append(cost)
            e0 += len(v)
        return {"v": V.reshape(-1), "gamma": G, "cost": torch.cat(costs), "converged": None}
    if kind == "boxes":
        a = _boxes_problem(case, seed)
        parts = [_minimize(_dense_boxes(a, case["boxes"], slice(e, e + 148))) for e in range(0, E, 148)]
        v, g, cost = (torch.cat([p[i] for p in parts]) for i in range(3))
        return {"v": v.reshape(-1), "gamma": g, "cost": cost, "converged": None}
    if kind == "train":
        raw, target = _train_data(case, seed)
        x = raw.to(torch.bfloat16).to(F64)
        p = WarmStartMLP(CUDA, seed=seed).params.to(F64)
        shapes = [(128, 12), (128,), (128, 128), (128,), (128, 128), (128,), (3, 128), (3,)]
        parts = [t.reshape(s) for t, s in zip(p.split([math.prod(s) for s in shapes]), shapes)]
        for t in parts:
            t.requires_grad_(True)
        h = x
        for k in range(3):
            h = torch.nn.functional.gelu(h @ parts[2 * k].T + parts[2 * k + 1], approximate="tanh")
        loss = ((h @ parts[6].T + parts[7] - target.to(F64)) ** 2).sum()
        # the network's gradient is the mean squared error's
        grad = torch.cat([t.reshape(-1) for t in torch.autograd.grad(loss / target.numel(), parts)])
        return {"loss": loss.detach().reshape(1), "grad": grad, "params": None}
    return None  # contacts: counts and closed-form points, held to the type's bound
