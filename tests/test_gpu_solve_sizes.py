"""The dense solve at the sizes where its tiles and classes end: DOF counts
around the 8 x 8 Hessian blocks, the factorization's column blocks and the
32 lanes of its backward substitution, the specialised counts and their
neighbours, contact counts around the four-row steps; and large uneven
batches, which run one launch per size class, against the same worlds in
small ones, which run in one; and worlds that fill an SM's shared memory,
which run eight warps by default; and free-box worlds around the 360 DOFs
from which the tree-blocked solve runs 512 threads, against 256 (two answers
that may take different paths, as in test_gpu_blocked's full-size worlds).

Tolerances as in test_gpu_contact_solve (same iterates as the oracle up to
rounding); between the two launches of an uneven batch the worlds run the
same arithmetic, so only its order within a product may differ: 1e-9
relative in FP64, three decimal orders below the solve's own tolerance; with the
FP32 factor, whose directions carry 1e-7, that tolerance itself (1e-6).
"""

import numpy as np
import pytest
import torch

from sap_warp_b200 import scenes
from sap_warp_b200._solve import ContactSolveBuffers, contact_solve, make_options, problem_to_device
from tests.test_gpu_blocked import run_blocked
from tests.test_gpu_contact_solve import assert_parity, run_gpu

pytestmark = pytest.mark.gpu


def leading_dofs(n: int, worlds: int, counts) -> scenes.ContactProblemArrays:
    """The leading n DOFs of a 60-DOF chain's problem: A's leading block, J's
    first n columns, contacts on its last bodies."""
    p = scenes.humanoid_contact_problem(worlds, seed=300 + n, revolute=54, contacts=(1, 13), max_contacts=13,
                                        counts=np.asarray(counts, np.int32))
    E, B = worlds, p.bodies_per_env
    q = scenes.ContactProblemArrays(**{f: getattr(p, f) for f in p.__dataclass_fields__})
    q.dof_per_env = n
    q.dynamics_matrix = np.ascontiguousarray(p.dynamics_matrix[:, :n, :n])
    q.jacobian = np.ascontiguousarray(p.jacobian[..., :n])
    q.v_star = np.ascontiguousarray(p.v_star.reshape(E, -1)[:, :n]).reshape(-1)
    q.v0 = np.ascontiguousarray(p.v0.reshape(E, -1)[:, :n]).reshape(-1)
    q.body_dof_count = np.full(E * B, n, np.int32)
    q.w_eff = scenes.diag_delassus_weight(q.jacobian, q.dynamics_matrix) * (q.w_eff > 0)
    return q


@pytest.mark.parametrize("n", [1, 3, 5, 6, 7, 8, 9, 13, 16, 17, 18, 31, 32, 33, 35, 36, 40, 41, 59, 60])
@pytest.mark.parametrize("variant", ["armijo_decay", "exact_root"])
def test_dof_counts_match_oracle(cuda_device, oracle, n, variant):
    prob = leading_dofs(n, 8, [1, 2, 3, 4, 5, 8, 12, 13])
    gpu = run_gpu(prob, cuda_device, variant)
    ref = oracle.solve(prob, variant)
    assert_parity(prob, gpu, ref)
    np.testing.assert_array_equal(gpu["converged"], ref["converged"])


@pytest.mark.parametrize("n, contacts", [(41, 96), (55, 112)])
def test_worlds_that_fill_an_sm_match_oracle(cuda_device, oracle, n, contacts):
    prob = scenes.humanoid_contact_problem(6, seed=400 + n, revolute=n - 6, contacts=(contacts // 2, contacts),
                                           max_contacts=contacts)
    gpu = run_gpu(prob, cuda_device, "armijo_decay")
    assert_parity(prob, gpu, oracle.solve(prob, "armijo_decay"))
    four = run_gpu(prob, cuda_device, "armijo_decay", threads_per_cta=128)
    assert_parity(prob, gpu, four)


@pytest.mark.parametrize("boxes", [59, 60, 63])
@pytest.mark.parametrize("variant", ["armijo_decay", "exact_root"])
def test_wide_box_worlds_match_256_threads(cuda_device, boxes, variant):
    bp = scenes.box_stack_problem(4, seed=460 + boxes, boxes=boxes)
    gpu = run_blocked(bp, cuda_device, variant)
    narrow = run_blocked(bp, cuda_device, variant, threads_per_cta=256)
    np.testing.assert_array_equal(gpu["converged"], narrow["converged"])
    np.testing.assert_array_equal(gpu["status"], 0)
    assert_parity(bp.to_dense(), gpu, narrow, max_loose_frac=0.5)


def _uneven(worlds: int, dofs, device):
    """Worlds of the given DOF counts in turn (compact, 41-DOF slots)."""
    n, C = 41, 6
    rng = np.random.default_rng(11)
    d = np.asarray([dofs[i % len(dofs)] for i in range(worlds)], np.int32)
    A, J = np.zeros((worlds, n * n)), np.zeros((worlds, C * 3 * n))
    v = np.zeros((worlds, n))
    few = {k: leading_dofs(k, 16, rng.integers(1, C + 1, size=16)) for k in dofs}
    per = {f: np.zeros((worlds, C)) for f in ("phi0", "w_eff", "mu", "stiffness", "tau_d")}
    count = np.zeros(worlds, np.int32)
    for e in range(worlds):
        q, k, i = few[int(d[e])], int(d[e]), e % 16
        A[e, :k * k] = q.dynamics_matrix[i].reshape(-1)
        J[e, :C * 3 * k] = q.jacobian[i, :C].reshape(-1)
        v[e, :k] = q.v_star.reshape(16, k)[i] + rng.normal(scale=0.05, size=k)
        count[e] = q.contact_count[i]
        for f in per:
            per[f][e] = getattr(q, f)[i, :C]
    t = lambda a, dt=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=device)
    arrays = dict(contact_count=t(count, torch.int32), dynamics_matrix=t(A), jacobian=t(J), v_star=t(v.reshape(-1)),
                  v0=t(v.reshape(-1)), dt=t(np.full(worlds, 2.0e-3)), **{f: t(a) for f, a in per.items()})
    return arrays, t(d, torch.int32), n, C


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_large_uneven_batch_equals_its_worlds_in_small_ones(cuda_device, precision):
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    W = 16 * sms + 1  # one world past the batches that run in one launch
    arrays, dofs, n, C = _uneven(W, (35, 18, 13, 6, 9, 24, 41), cuda_device)
    opts = make_options("armijo_decay", hessian_precision=precision, linear_solve_precision=precision)
    order = torch.argsort(dofs, descending=True, stable=True).to(torch.int32)

    def run(sl, wo=None):
        E = sl.stop - sl.start
        buf = ContactSolveBuffers(E, n, C, cuda_device)
        cut = {k: (a.reshape(W, -1)[sl].contiguous() if a.numel() != W else a[sl].contiguous())
               for k, a in arrays.items()}
        cut = {k: a.reshape(-1) if k in ("v_star", "v0") else a for k, a in cut.items()}
        contact_solve(**cut, buffers=buf, options=opts, world_order=wo, dof_count=dofs[sl].contiguous())
        torch.cuda.synchronize()
        return buf

    whole = run(slice(0, W), order)
    assert bool(whole.converged.all())
    vw = whole.v.reshape(W, n)
    tol = 1e-9 if precision == "fp64" else 1e-6
    for s in range(0, W, 500):
        sl = slice(s, min(s + 500, W))
        part = run(sl)
        vp = part.v.reshape(-1, n)
        err = (vw[sl] - vp).abs().amax(1) / vp.abs().amax(1)
        assert float(err.max()) <= tol, float(err.max())
        assert torch.equal(whole.newton_iterations[sl], part.newton_iterations)
