"""set_static_split(None) gives the choice between the fused and the split passes back to the number of
centres (40 per SM and more run split, Static)."""
import os

import numpy as np
import pytest

from superlinear_gb300.synth import lattice_frame

pytestmark = pytest.mark.gpu


def test_split_choice_back_to_the_number_of_centres(engine_lib, golden):
    import superlinear_gb300 as sg
    rng = np.random.default_rng(1)
    eng = sg.Engine(sg.Model(os.path.join(golden, "models", "static_l3k4o2.sus2")), 0, sg.FP32)
    for on in (True, False):
        eng.set_static_split(on)
        eng.set_static_split(None)
        for frames, split in (([lattice_frame("diamond", (2, 2, 2), 3.6, 0.1, rng)], False), ([lattice_frame("diamond", (10, 10, 9), 3.6, 0.1, rng)], True)):
            eng.calc_efs(frames)
            assert eng.pass_shapes()["static"]["split"] == split
