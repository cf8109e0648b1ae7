"""A frame's results do not depend on the frames it is evaluated with, also where the batch runs the
split passes (by its number of centres) and the frame alone the fused ones."""
import os

import numpy as np
import pytest

from superlinear_gb300.synth import Frame, lattice_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["static_l2k3o2_c2", "static_l3k4o2", "effect_l3k4r2o2", "effect_l4k8r2o3", "effect_l5k8r2o2_c3"])
def test_frame_alone_and_in_a_large_batch(engine_lib, golden, name):
    import superlinear_gb300 as sg
    model = sg.Model(os.path.join(golden, "models", name + ".sus2"))
    rng = np.random.default_rng(23)
    species = model.dims["C"]
    # image-scan and cell-list frames of uneven neighbour counts, and enough centres around them for
    # the split passes of every model (40 per SM and more)
    frames = [lattice_frame("diamond", (2, 2, 3), 3.7, 0.15, rng, species=species),
              lattice_frame("fcc", (5, 5, 6), 3.9, 0.2, rng, species=species),
              lattice_frame("bcc", (3, 2, 2), 3.1, 0.1, rng, species=species),
              Frame(np.eye(3) * 30.0, rng.uniform(0, 6, (7, 3)), rng.integers(0, species, 7)),
              lattice_frame("diamond", (10, 10, 10), 3.6, 0.1, rng, species=species)]
    eng = sg.Engine(model, 0, sg.FP32)
    e, f, v, s = eng.calc_efs(frames)
    at = 0
    for k, fr in enumerate(frames[:4]):
        n = fr.natoms
        e1, f1, v1, s1 = sg.Engine(model, 0, sg.FP32).calc_efs([fr])
        np.testing.assert_array_equal(s1, s[at:at + n])
        np.testing.assert_array_equal(f1, f[at:at + n])
        np.testing.assert_array_equal(v1[0], v[k])
        assert e1[0] == e[k]
        at += n


@pytest.mark.parametrize("name", ["effect_l3k4r2o2", "effect_l4k8r2o3", "effect_l5k8r2o2_c3"])
def test_effect_split_is_bitwise_the_fused_form(engine_lib, golden, name):
    import superlinear_gb300 as sg
    model = sg.Model(os.path.join(golden, "models", name + ".sus2"))
    fr = lattice_frame("diamond", (3, 4, 5), 3.7, 0.2, np.random.default_rng(4), species=model.dims["C"])
    eng = sg.Engine(model, 0, sg.FP32)
    results = []
    for split in (False, True):
        eng.set_static_split(split)
        results.append(eng.calc_efs([fr]))
    for x, y in zip(*results):
        np.testing.assert_array_equal(x, y)
