"""The plans of the solves beyond test_gpu_solve_sizes' cases: the DOF sweep with
the FP32 factor (its own panel strides and instantiations) and with
monotone_decay, worlds that fill an SM with the FP32 factor, the box counts
around the 512-thread launch in both precisions, and the launches per size class
of a large uneven batch with candidate starts, a kept factor, a guess, drives,
limits and worlds without contacts, against the same worlds in small batches;
and a tree-blocked candidate start that is rejected.

Tolerances: FP32 directions and monotone_decay (here with the other searches'
cost tolerance) may take other paths than the oracle, so up to half of a batch may be loose in
assert_parity, which then checks that each of those is stationary.  Wide box
worlds are checked to be stationary by themselves, path or not
(test_gpu_far_start's check).  Between the launches of an uneven batch as in
test_gpu_solve_sizes: the same arithmetic per world.
"""

import numpy as np
import pytest
import torch

from sap_warp_b200 import scenes
from sap_warp_b200._solve import (ContactSolveBuffers, DofTermArrays, blocked_contact_solve,
                                  blocked_problem_to_device, contact_solve, make_options)
from tests.test_gpu_blocked import run_blocked
from tests.test_gpu_contact_solve import assert_parity, run_gpu
from tests.test_gpu_far_start import check_reported
from tests.test_gpu_solve_sizes import _uneven, leading_dofs

pytestmark = pytest.mark.gpu
FP32 = dict(hessian_precision="fp32", linear_solve_precision="fp32")


@pytest.mark.parametrize("n", [1, 5, 6, 7, 8, 9, 13, 16, 17, 18, 31, 32, 33, 35, 36, 40, 41, 59, 60])
@pytest.mark.parametrize("variant", ["armijo_decay", "exact_root"])
def test_dof_counts_with_fp32_factor(cuda_device, oracle, n, variant):
    prob = leading_dofs(n, 8, [1, 2, 3, 4, 5, 8, 12, 13])
    assert_parity(prob, run_gpu(prob, cuda_device, variant, **FP32), oracle.solve(prob, variant), max_loose_frac=0.5)


@pytest.mark.parametrize("n", [1, 6, 8, 9, 13, 18, 32, 33, 35, 41, 60])
def test_dof_counts_with_monotone_decay(cuda_device, oracle, n):
    prob = leading_dofs(n, 8, [1, 2, 3, 4, 5, 8, 12, 13])
    gpu = run_gpu(prob, cuda_device, "monotone_decay", cost_rel_tol=1.0e-15, cost_abs_tol=1.0e-30)
    ref = oracle.solve(prob, "monotone_decay", cost_rel_tol=1.0e-15, cost_abs_tol=1.0e-30)
    assert_parity(prob, gpu, ref, max_loose_frac=0.5)


@pytest.mark.parametrize("n, contacts", [(41, 112), (55, 128)])
def test_worlds_that_fill_an_sm_with_fp32_factor(cuda_device, oracle, n, contacts):
    prob = scenes.humanoid_contact_problem(6, seed=420 + n, revolute=n - 6, contacts=(contacts // 2, contacts),
                                           max_contacts=contacts)
    assert_parity(prob, run_gpu(prob, cuda_device, "armijo_decay", **FP32), oracle.solve(prob, "armijo_decay"),
                  max_loose_frac=0.5)


@pytest.mark.parametrize("boxes", [59, 60, 63])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("variant", ["armijo_decay", "exact_root"])
def test_wide_box_worlds_are_stationary(cuda_device, boxes, precision, variant):
    bp = scenes.box_stack_problem(12, seed=480 + boxes, boxes=boxes)
    gpu = run_blocked(bp, cuda_device, variant, hessian_precision=precision, linear_solve_precision=precision)
    check_reported(bp.to_dense(), gpu, 1e-6)


def _ldlt(A):
    """The kept factor's form of A = L D L^T: L_ik d_k below the diagonal, d on it."""
    H = A.copy()
    for k in range(len(H)):
        H[k + 1:, k + 1:] -= np.outer(H[k + 1:, k], H[k + 1:, k]) / H[k, k]
    return np.tril(H)


def _extras(kind, arrays, dofs, n, C, device):
    """The problem's optional arrays for `kind`, as functions of a slice of worlds."""
    W = dofs.numel()
    gen = torch.Generator(device=device).manual_seed(7)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=device, dtype=torch.float64)
    v0 = arrays["v0"].reshape(W, n)
    if kind == "candidates":
        vc, g0 = v0[None] + 0.02 * rnd(2, W, n), 0.05 * rnd(3, W, C, 3).abs()
        g0[:, ::4] = 0.0  # worlds whose sets are all zero
        return lambda sl: dict(v_candidates=vc[:, sl].contiguous(), gamma0=g0[:, sl].contiguous())
    if kind == "factor":
        A, d = arrays["dynamics_matrix"].cpu().numpy(), dofs.cpu().numpy()
        F, made = np.zeros_like(A), {}
        for e in range(W):
            k = int(d[e])
            m = A[e, :k * k]
            key = (k, m.tobytes())
            if key not in made:
                made[key] = _ldlt(m.reshape(k, k)).reshape(-1)
            F[e, :k * k] = made[key]
        F = torch.as_tensor(F, device=device)
        g0, base = 0.05 * rnd(1, W, C, 3).abs(), v0 + 0.01 * rnd(W, n)
        return lambda sl: dict(gamma0=g0[:, sl].contiguous(), dynamics_factor=F[sl].contiguous(),
                               gamma0_base=base[sl].reshape(-1).contiguous())
    guess, q = v0 + 0.1 * rnd(W, n), 0.3 * rnd(W, n)
    mode = (torch.rand(W, n, generator=gen, device=device) < 0.5).to(torch.int32)

    def terms(sl):
        E = sl.stop - sl.start
        full = lambda x, dt: torch.full((E * n,), x, dtype=dt, device=device)
        idx = torch.arange(E * n, dtype=torch.int32, device=device)
        f32, f64 = torch.float32, torch.float64
        t = DofTermArrays(has_pd=1, has_limits=1, dof_coord_index=idx, dof_target_index=idx,
                          limit_supported=full(1, torch.int32), joint_target_mode=mode[sl].reshape(-1).contiguous(),
                          joint_target_ke=full(40.0, f32), joint_target_kd=full(2.0, f32),
                          joint_effort_limit=full(30.0, f32), joint_limit_lower=full(-0.3, f64),
                          joint_limit_upper=full(0.3, f64), joint_limit_ke=full(1.0e4, f64),
                          joint_limit_kd=full(10.0, f64), joint_q=q[sl].reshape(-1).contiguous(),
                          joint_target_pos=full(0.1, f32), joint_target_vel=full(0.0, f32), joint_act=full(0.0, f32))
        return dict(dof_terms=t, v_guess=guess[sl].reshape(-1).clone(),
                    v_guess_active=torch.ones(1, dtype=torch.int32, device=device))

    return terms


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["candidates", "factor", "guess, drives and limits"])
def test_class_launches_with_every_start_and_term(cuda_device, precision, kind):
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    W = 16 * sms + 5
    arrays, dofs, n, C = _uneven(W, (35, 18, 13, 6, 9, 24, 41), cuda_device)
    arrays["contact_count"][::10] = 0
    extras = _extras(kind, arrays, dofs, n, C, cuda_device)
    opts = make_options("armijo_decay", hessian_precision=precision, linear_solve_precision=precision)

    def run(sl):
        buf = ContactSolveBuffers(sl.stop - sl.start, n, C, cuda_device)
        cut = {k: a.reshape(W, -1)[sl].contiguous() if a.numel() != W else a[sl].contiguous()
               for k, a in arrays.items()}
        cut = {k: a.reshape(-1) if k in ("v_star", "v0") else a for k, a in cut.items()}
        contact_solve(**cut, **extras(sl), buffers=buf, options=opts, dof_count=dofs[sl].contiguous())
        torch.cuda.synchronize()
        return buf

    whole = run(slice(0, W))
    assert bool(whole.converged.all()) and not bool(whole.status.any())
    if kind == "candidates":
        assert int(whole.warm_start_accepted.max()) > 0
    vw = whole.v.reshape(W, n)
    tol = 1e-9 if precision == "fp64" else 1e-6
    for s in range(0, W, 500):
        sl = slice(s, min(s + 500, W))
        part = run(sl)
        vp = part.v.reshape(-1, n)
        err = (vw[sl] - vp).abs().amax(1) / vp.abs().amax(1)
        assert float(err.max()) <= tol, float(err.max())
        for name in ("newton_iterations", "converged", "warm_start_accepted"):
            assert torch.equal(getattr(whole, name)[sl], getattr(part, name)), name
        live = torch.arange(C, device=cuda_device)[None] < arrays["contact_count"][sl][:, None]
        assert not bool(part.contact_gamma[~live].any()) and not bool(whole.contact_gamma[sl][~live].any())


@pytest.mark.parametrize("boxes", [8, 30, 63])
@pytest.mark.parametrize("threads", [0, 128, 256])
def test_rejected_tree_blocked_candidate_leaves_the_plain_start(cuda_device, boxes, threads):
    """Starting impulses far too large are evaluated and rejected: the solve
    goes on from the plain start, which other threads save than overwrite, and
    gives the bits of a solve without candidate."""
    bp = scenes.box_stack_problem(24, seed=500 + boxes, boxes=boxes)
    t = blocked_problem_to_device(bp, cuda_device)
    g0 = torch.full((bp.num_envs, bp.max_contacts, 3), 1.0e3, dtype=torch.float64, device=cuda_device)
    out = []
    for gamma0 in (None, g0):
        buf = ContactSolveBuffers(bp.num_envs, bp.dof_per_env, bp.max_contacts, cuda_device)
        blocked_contact_solve(buffers=buf, options=make_options("armijo_decay", threads_per_cta=threads),
                              trees_per_env=bp.trees_per_env, tree_dofs=bp.tree_dofs, gamma0=gamma0, **t)
        torch.cuda.synchronize()
        out.append(buf)
    assert not bool(out[1].warm_start_accepted.any())
    for name in ("v", "contact_gamma", "newton_iterations", "status"):
        assert torch.equal(getattr(out[0], name), getattr(out[1], name)), name
