"""A caller's stream may end before the engine takes new parameters."""
import ctypes
import os

import numpy as np
import pytest

from superlinear_gb300.synth import lattice_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_update_params_after_the_callers_stream_is_gone(engine_lib, golden, precision):
    torch = pytest.importorskip("torch")
    import superlinear_gb300 as sg
    rt = torch.cuda.cudart()
    model = sg.Model(os.path.join(golden, "models", "effect_l3k4r2o2.sus2"))
    fr = lattice_frame("diamond", (2, 2, 2), 3.7, 0.1, np.random.default_rng(2), species=2)
    eng = sg.Engine(model, 0, precision)
    stream = ctypes.c_void_p()
    assert int(rt.cudaStreamCreate(ctypes.addressof(stream))) == 0
    eng.set_stream(stream.value)
    for _ in range(3):
        eng.calc_efs([fr])
    assert int(rt.cudaStreamDestroy(stream.value)) == 0
    model.set_params(np.asarray(model.params()) * 1.01)
    eng.update_params()
    for x, y in zip(eng.calc_efs([fr]), sg.Engine(model, 0, precision).calc_efs([fr])):
        np.testing.assert_array_equal(x, y)
