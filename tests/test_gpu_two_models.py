"""Host threads that take gradients of two models on one GPU: the models need different amounts of
shared memory of the same kernels."""
import os
import threading

import numpy as np
import pytest

from superlinear_gb300.synth import lattice_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_gradients_of_two_models_at_once(engine_lib, golden, precision):
    import superlinear_gb300 as sg
    failed, start = [], threading.Barrier(2)

    def work(name):
        try:
            model = sg.Model(os.path.join(golden, "models", name + ".sus2"))
            fr = [lattice_frame("diamond", (1, 1, 2), 3.7, 0.1, np.random.default_rng(3), species=model.dims["C"])]
            rng = np.random.default_rng(1)
            w = rng.standard_normal(16), rng.standard_normal((16, 3)), rng.standard_normal((1, 9))
            want = sg.Engine(model, 0, precision).combination_grad(fr, *w)
            eng = sg.Engine(model, 0, precision)
            eng.combination_grad(fr, *w)
            start.wait()
            got = [eng.combination_grad(fr, *w) for _ in range(1000)]  # (nothing else between the calls)
            for g in got:
                np.testing.assert_array_equal(g, want)
        except BaseException as error:  # noqa: BLE001 (reported by the test's thread)
            start.abort()
            failed.append(error)

    threads = [threading.Thread(target=work, args=(name,)) for name in ("effect_l3k4r2o2", "effect_l5k8r2o2_c3")]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
