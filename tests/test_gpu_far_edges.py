"""A caller's edge far beyond the cutoff contributes nothing, however long it is: also where its
components overflow the FP32 record."""
import os

import numpy as np
import pytest

from superlinear_gb300.synth import lattice_frame
from test_zz_no_alloc import call_noalloc, csr_rows

pytestmark = pytest.mark.gpu

FAR = [(20.0, 0, 0), (1e20, -1e19, 3), (1e38, 2e38, -1e38), (0, -1e40, 1e39), (1e149, -2.0, 0)]
# the far edge joins the sums as zeros and may move their batches of 32: the rounding of ~100-term sums
BAR = (1e-12, 2e-6)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", ["static_l3k4o2", "effect_l3k4r2o2"])
def test_far_edges(engine_lib, golden, name, precision):
    torch = pytest.importorskip("torch")
    import superlinear_gb300 as sg
    model = sg.Model(os.path.join(golden, "models", name + ".sus2"))
    fr = lattice_frame("diamond", (3, 3, 3), 5.43, 0.1, np.random.default_rng(6), species=model.dims["C"])
    n = fr.natoms
    eng = sg.Engine(model, 0, precision)
    eng.calc_efs([fr])
    ei, ej, d = eng.edges()
    want = eng.efs_edges(n, fr.types, ei, ej, d)

    def check(got):
        for x, y in zip(got, want):
            x, y = np.asarray(x), np.asarray(y)
            assert np.all(np.isfinite(x)) and np.linalg.norm(x - y) <= BAR[precision] * (np.linalg.norm(y) + np.linalg.norm(want[2]))

    for k, far in enumerate(FAR):
        at = np.searchsorted(ei, 7 + k)  # one more edge of centre 7 + k
        args = np.insert(ei, at, 7 + k), np.insert(ej, at, 100), np.insert(d, at, far, axis=0)
        for split in (False, True):
            eng.set_static_split(split)
            check(eng.efs_edges(n, fr.types, *args))
        if precision == sg.FP32 and name.startswith("static"):
            rc, e, f, v, s = call_noalloc(torch, engine_lib, eng, n, fr.types, csr_rows(args[0], n), *args[1:])
            assert rc == 0
            check((e, s, f, v))
