"""Trainer.rescale on a trainer that has evaluated before: its captured evaluation holds the radial
scaling by value and must not outlive it.  The trials of a trainer of at most five frames run on the
trainer itself, so nothing else makes it capture again."""
import os

import numpy as np
import pytest

from conftest import load_json
from superlinear_gb300.synth import read_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["static_l2k3o2_c2", "effect_l3k4r2o2"])
def test_loss_after_rescale_of_a_captured_trainer(engine_lib, golden, name):
    import superlinear_gb300 as sg
    data = load_json(os.path.join(golden, "linear", name + "__rescale.json"))
    model = sg.Model(os.path.join(golden, "models", data["model"]))
    frames = read_cfg(os.path.join(golden, "frames", data["frames"]))

    def trainer():
        return sg.Trainer(sg.Engine(model, 0, sg.FP64), frames, *data["weights"], weighting=data["weighting"], gate_x_l2=0.0)

    tr = trainer()
    for _ in range(2):  # eager and captured, then replayed
        tr.loss_grad(model.params())
    before = model.scaling
    p, s, _ = tr.rescale(model.params())
    assert abs(s / before - 1) > 1e-3
    loss, grad = tr.loss_grad(p)
    model.scaling = s
    model.set_params(p)
    loss0, grad0 = trainer().loss_grad(p)
    assert loss == loss0
    np.testing.assert_array_equal(grad, grad0)
