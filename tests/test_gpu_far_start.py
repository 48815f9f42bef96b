"""The dense solve from starts far from the solution: the contact velocities
and A (v - v*) move along the line searches, so what is reported -- the
gradient norm, the impulses, convergence -- has to belong to the returned
velocity whatever the iterates went through.

Tolerance: gradient and impulses are formed here in numpy at the returned v.
Moved at most seven steps from values formed at up to four times the present
size (in the norm of diag(A)), each step at most twice that size, their error
is below 7 * 8 + 1 times that of a sum of n products, numpy's own is one more:
64 n eps times |A| |v - v*| and |J| |v|, with |v_j| <= ||v||_D / sqrt(A_jj),
and through the projection's steepest slope, the inverse regularization.
"""

import numpy as np
import pytest

from sap_warp_b200 import scenes
from tests import sap_numpy as sn
from tests.test_gpu_contact_solve import run_gpu

pytestmark = pytest.mark.gpu


def check_reported(prob, g, rel_tol):
    n, E = prob.dof_per_env, prob.num_envs
    V, vs = g["v"].reshape(E, n), prob.v_star.reshape(E, n)
    unit = 64 * n * np.finfo(float).eps
    assert np.all(g["converged"] == 1) and np.all(g["status"] == 0)
    for e in range(E):
        c = int(prob.contact_count[e])
        A, J = prob.dynamics_matrix[e], prob.jacobian[e, :c]
        par = [getattr(prob, f)[e] for f in ("phi0", "w_eff", "mu", "stiffness", "tau_d")]
        _, grad, gamma, _ = sn.objective(V[e], A, vs[e], prob.jacobian[e], *par, c)
        rt, rn, _ = sn.contact_constants(par[0][:c], par[1][:c], par[2][:c], par[3][:c], par[4][:c])
        d = np.diag(A)
        s = 1.0 / np.sqrt(d)
        size = lambda x: np.sqrt(np.sum(d * x * x))
        dgamma = (np.abs(J) @ s) * size(V[e]) / np.stack([rt, rt, rn], -1)
        dgrad = (np.abs(A) @ s) * size(V[e] - vs[e]) + np.einsum("crj,cr->j", np.abs(J), dgamma)
        floor = unit * np.linalg.norm(s * dgrad)
        norm = np.linalg.norm(s * grad)
        assert abs(norm - g["grad_norm"][e]) <= floor
        np.testing.assert_array_less(np.abs(gamma - g["contact_gamma"][e, :c]), unit * dgamma.max() + 1e-300)
        scale = max(np.linalg.norm(s * (A @ V[e])), np.linalg.norm(s * np.einsum("crj,cr->j", J, gamma)))
        assert norm <= 1.0e-14 + rel_tol * scale * (1.0 + 1.0e-9) + floor


@pytest.mark.parametrize("n", [18, 31, 35])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("variant, rel_tol", [("armijo_decay", 1e-6), ("exact_root", 1e-6), ("exact_root", 1e-11)])
@pytest.mark.parametrize("size", [1.0e2, 1.0e6, 1.0e10])
def test_reports_belong_to_the_returned_velocity(cuda_device, n, precision, variant, rel_tol, size):
    prob = scenes.humanoid_contact_problem(16, seed=77 + n, revolute=n - 6, contacts=(4, 13), max_contacts=13)
    guess = prob.v_star + size * np.random.default_rng(3).normal(size=prob.v_star.shape)
    g = run_gpu(prob, cuda_device, variant, v_guess=guess, guess_active=True, optimality_rel_tol=rel_tol,
                hessian_precision=precision, linear_solve_precision=precision)
    check_reported(prob, g, rel_tol)
