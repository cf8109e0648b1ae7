"""Parameters replaced in a running engine, against a new engine for the same parameters, and caller
edges in any order.

The in-place path keeps the device buffers and copies the rank weights into every program image; both
engines then run the same kernels on the same tables, whose sums are ordered: E/F/virial are equal.
The gradient's FP64 sums meet in no fixed order (1e-12); an FP32 engine's parts are rounded to 24 bits
before they meet (1e-6 of the norm)."""
import os

import numpy as np
import pytest

import superlinear_gb300 as sg
from conftest import rel_err
from superlinear_gb300._lib import Sus2Error
from superlinear_gb300.synth import lattice_frame

pytestmark = pytest.mark.gpu
MODELS = os.path.join(os.path.dirname(__file__), "golden", "models")


@pytest.mark.parametrize("precision", [sg.FP32, sg.FP64])
@pytest.mark.parametrize("name,species", [("static_l3k4o2", 1), ("effect_l3k4r2o2", 1), ("effect_l5k8r2o2_c3", 3)])
def test_update_params_in_place(name, species, precision):
    rng = np.random.default_rng(5)
    path = os.path.join(MODELS, name + ".sus2")
    frames = [lattice_frame("diamond", (2, 2, 1 + s), 5.43, 0.08, rng, species=species) for s in range(3)]
    n = sum(len(f.types) for f in frames)
    weights = rng.standard_normal(n), rng.standard_normal((n, 3)), rng.standard_normal((3, 9))
    model = sg.Model(path)
    eng = sg.Engine(model, precision=precision)
    eng.set_static_split(True)  # the split passes' programs are in use before the update
    eng.calc_efs(frames)
    eng.combination_grad(frames, *weights)
    for _ in range(2):
        p = np.asarray(model.params())
        model.set_params(p * (1 + 0.02 * rng.standard_normal(p.size)))
        model.scaling = model.scaling * 1.1
        eng.update_params()
        new = sg.Engine(model, precision=precision)
        for split in (False, True):
            for e in (eng, new):
                e.set_static_split(split)
            for x, y in zip(eng.calc_efs(frames), new.calc_efs(frames)):
                np.testing.assert_array_equal(x, y)
        a, b = eng.combination_grad(frames, *weights), new.combination_grad(frames, *weights)
        assert rel_err(a, b) < (1e-6 if precision == sg.FP32 else 1e-12)


@pytest.mark.parametrize("precision", [sg.FP32, sg.FP64])
@pytest.mark.parametrize("name", ["static_l3k4o2", "effect_l3k4r2o2"])
def test_caller_edges_any_order(name, precision):
    frame = lattice_frame("diamond", (4, 4, 4), 5.43, 0.08, np.random.default_rng(3))  # no image repeats a pair
    eng = sg.Engine(sg.Model(os.path.join(MODELS, name + ".sus2")), precision=precision)
    eng.calc_efs([frame])
    ci, cj, d = eng.edges()
    n = len(frame.types)
    want = eng.efs_edges(n, frame.types, ci, cj, d)
    assert eng.edge_count() == len(ci)
    o = np.random.default_rng(1).permutation(len(ci))
    for x, y in zip(eng.efs_edges(n, frame.types, ci[o], cj[o], d[o]), want):
        np.testing.assert_array_equal(x, y)
    # an edge that is refused leaves the engine's edges and its next results as they were
    for k, (i, j, v) in enumerate([(n, 0, (1.0, 0, 0)), (0, n, (1.0, 0, 0)), (-1, 0, (1.0, 0, 0)), (0, 1, (0, 0, 0)),
                                   (0, 1, (np.nan, 0, 0)), (0, 1, (1e160, 0, 0))]):
        bad = [ci.copy(), cj.copy(), d.copy()]
        at = (len(ci) - 1) * k // 5
        bad[0][at], bad[1][at], bad[2][at] = i, j, v
        with pytest.raises(Sus2Error, match="index out of range" if k < 3 else "length"):
            eng.efs_edges(n, frame.types, *bad)
        assert eng.edge_count() == len(ci)
    empty = eng.efs_edges(n, frame.types, ci[:0], cj[:0], d[:0])
    assert np.all(np.isfinite(empty[0])) and eng.edge_count() == 0
    for x, y in zip(eng.efs_edges(n, frame.types, ci, cj, d), want):
        np.testing.assert_array_equal(x, y)
