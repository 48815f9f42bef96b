"""Pivots beyond the range of the fast reciprocal (2^126 with the FP32 factor):
worlds so heavy that H's diagonal ends just below FP32's largest number are
solved like any other, by the dense and the tree-blocked kernel.  Checked as
in test_gpu_far_start (same tolerance): the reported state is stationary."""

import numpy as np
import pytest

from sap_warp_b200 import scenes
from tests.test_gpu_blocked import run_blocked
from tests.test_gpu_contact_solve import run_gpu
from tests.test_gpu_far_start import check_reported

pytestmark = pytest.mark.gpu


def heavy(diag) -> float:
    """The mass factor that puts the largest diagonal entry at 3e38."""
    return 3.0e38 / float(np.max(diag))


@pytest.mark.parametrize("n", [6, 13, 18, 24, 35, 47])
def test_dense_worlds(cuda_device, n):
    prob = scenes.humanoid_contact_problem(8, seed=500 + n, revolute=n - 6, contacts=(2, 9), max_contacts=9)
    k = heavy(np.diagonal(prob.dynamics_matrix, axis1=1, axis2=2))
    prob.dynamics_matrix = prob.dynamics_matrix * k
    prob.w_eff = prob.w_eff / k
    rng = np.random.default_rng(n)
    guess = prob.v_star + 0.01 * rng.normal(size=prob.v_star.shape)
    g = run_gpu(prob, cuda_device, "armijo_decay", v_guess=guess, guess_active=True, hessian_precision="fp32",
                linear_solve_precision="fp32")
    check_reported(prob, g, 1e-6)


@pytest.mark.parametrize("boxes", [8, 60])
def test_tree_blocked_worlds(cuda_device, boxes):
    bp = scenes.box_stack_problem(3, seed=520 + boxes, boxes=boxes)
    k = heavy(np.diagonal(bp.tree_mass, axis1=2, axis2=3))
    bp.tree_mass = bp.tree_mass * k
    bp.w_eff = bp.w_eff / k
    bp.v0 = bp.v_star + 0.01 * np.random.default_rng(boxes).normal(size=bp.v_star.shape)
    g = run_blocked(bp, cuda_device, "armijo_decay", hessian_precision="fp32", linear_solve_precision="fp32")
    check_reported(bp.to_dense(), g, 1e-6)
