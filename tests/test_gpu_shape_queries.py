"""Engine.pass_shapes tells the form that ran, also where the number of centres chose it."""
import os

import numpy as np
import pytest

from superlinear_gb300.synth import lattice_frame

pytestmark = pytest.mark.gpu


def boxes(count, reps, species):
    rng = np.random.default_rng(count)
    return [lattice_frame("diamond", reps, 3.6, 0.1, rng, species=species) for _ in range(count)]


@pytest.mark.parametrize("name", ["static_l3k4o2", "effect_l3k4r2o2"])
def test_pass_shapes_without_tuning(engine_lib, golden, name):
    torch = pytest.importorskip("torch")
    import superlinear_gb300 as sg
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    model = sg.Model(os.path.join(golden, "models", name + ".sus2"))
    species = model.dims["C"]
    # five centres per SM: blocks of four warps put eight on some SMs, blocks of two at most six
    few = boxes(5 * sms // 8, (1, 1, 1), species)
    many = boxes(40 * sms // 512 + 1, (4, 4, 4), species)
    eng = sg.Engine(model, 0, sg.FP32)

    def shapes(frames):
        eng.calc_efs(frames)
        found = {(sh["split"], sh["warps_per_block"]) for sh in eng.pass_shapes().values()}
        assert len(found) == 1
        return found.pop()

    assert shapes(many)[0] and not shapes(few)[0]
    assert shapes(few)[1] == 2
    for _ in range(3):  # eager, captured, replayed
        assert shapes(many)[0]
    eng.set_static_split(True)
    assert shapes(few)[0]
    eng.set_static_split(False)
    assert not shapes(many)[0]
    # an FP64 engine has no split form
    eng = sg.Engine(model, 0, sg.FP64)
    eng.set_static_split(True)
    assert shapes(few) == (False, 2)
