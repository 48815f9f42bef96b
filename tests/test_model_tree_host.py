"""The model view refuses a model whose bodies do not hang off the ground: a
body among its own ancestors.  On the host only: no kernel runs on such a model."""

import dataclasses

import numpy as np
import pytest
import torch

from sap_warp_b200 import models
from sap_warp_b200.solver import _ModelView


def _model(worlds=3, uneven=False):
    rng = np.random.default_rng(5)
    made = []
    for kind in ("quadruped", "arm_boxes") if uneven else ("quadruped",):
        tpl = models.world_template(kind, rng, boxes=2)
        g = models.replicate(tpl, worlds, rng)
        made.append(models.to_model(tpl, g, models.random_joint_q(tpl, rng, worlds), "cpu"))
    return models.concat_models(made) if uneven else made[0]


@pytest.mark.parametrize("uneven", (False, True))
def test_trees_are_accepted(uneven):
    _ModelView(_model(uneven=uneven))


@pytest.mark.parametrize("uneven", (False, True))
@pytest.mark.parametrize("case", ("own parent", "pair", "whole chain", "last world"))
def test_cycles_are_refused(case, uneven):
    m = _model(uneven=uneven)
    view = _ModelView(m)
    parent, child = m.joint_parent.clone(), m.joint_child
    # a joint whose parent is a body (not the ground), and that body's joint
    j = int(torch.nonzero(parent >= 0)[-1 if case == "last world" else 0])
    above = int(torch.nonzero(child == parent[j])[0])
    if case in ("own parent", "last world"):
        parent[j] = child[j]
    elif case == "pair":
        parent[above] = child[j]
    else:  # the root hangs from the deepest body below it
        root = j
        while parent[root] >= 0:
            root = int(torch.nonzero(child == parent[root])[0])
        tip = child[j]
        while bool((parent == tip).any()):
            tip = child[int(torch.nonzero(parent == tip)[-1])]
        parent[root] = tip
    m = dataclasses.replace(m, joint_parent=parent)
    assert view.W > 1
    with pytest.raises(ValueError, match="cycle"):
        _ModelView(m)


def test_parents_outside_the_world_are_the_ground():
    """As in the free motion: a parent of another world is no ancestor."""
    m = _model()
    Bw = int(m.body_count) // int(m.world_count)
    parent = m.joint_parent.clone()
    root = int(torch.nonzero(m.joint_child == 0)[0])
    parent[root] = Bw  # world 1's root body
    root1 = int(torch.nonzero(m.joint_child == Bw)[0])
    parent[root1] = 0
    m = dataclasses.replace(m, joint_parent=parent)
    _ModelView(m)
