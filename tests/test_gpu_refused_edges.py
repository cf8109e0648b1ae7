"""A caller edge list that is refused leaves the engine as it was: its geometry holds the species it
was given on the device, which a later stage and the autotuner read."""
import os

import numpy as np
import pytest

from superlinear_gb300.synth import lattice_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("larger", [False, True])
def test_refused_list_between_the_stages(engine_lib, golden, larger):
    import superlinear_gb300 as sg
    model = sg.Model(os.path.join(golden, "models", "effect_l3k4r2o2.sus2"))
    fr = lattice_frame("diamond", (3, 3, 3), 3.9, 0.1, np.random.default_rng(8), species=2)
    n = fr.natoms
    src = sg.Engine(model, 0, sg.FP64)
    src.calc_efs([fr])
    ei, ej, d = src.edges()

    def staged(between):
        eng = sg.Engine(model, 0, sg.FP64)
        eng.stage_begin(n, fr.types, ei, ej, d)
        between(eng)
        eng.stage_outer()
        return eng.stage_finish(n, n)

    def refuse(eng):
        k = 50 if larger else 1
        bad = np.concatenate([ej] * k)
        bad[-1] = k * n
        with pytest.raises(sg.Sus2Error, match="index out of range"):
            eng.efs_edges(k * n, np.tile(1 - fr.types, k), np.concatenate([ei] * k), bad, np.concatenate([d] * k))

    for x, y in zip(staged(refuse), staged(lambda eng: None)):
        np.testing.assert_array_equal(x, y)
