"""FP64 passes keep their edges' functions for the adjoint up to 128 edges per centre and, in the gate
passes, up to 8,192 centres; past either they are evaluated again.  Dense frames on both sides of 128
edges against the FP64 oracle, and a box of 8,200 centres against half of it (its periodic image:
equal forces).  FP64 sums of some 1e3 terms: 1e-10, as the other FP64 comparisons."""
import os

import numpy as np
import pytest

from conftest import rel_err
from superlinear_gb300.synth import Frame, lattice_frame

pytestmark = pytest.mark.gpu
MODELS = os.path.join(os.path.dirname(__file__), "golden", "models")
TOL = 1e-10


@pytest.mark.parametrize("name,species", [("static_l3k4o2", 1), ("effect_l3k4r2o2", 1), ("effect_l5k8r2o2_c3", 3)])
def test_dense_frames(engine_lib, oracle_lib, name, species):
    import superlinear_gb300 as sg
    path = os.path.join(MODELS, name + ".sus2")
    rng = np.random.default_rng(2)
    frames = [lattice_frame("fcc", (2, 2, 2), a, 0.05, rng, species=species) for a in (2.5, 2.53, 2.58, 2.9)]
    om, eng = oracle_lib.OracleModel(path), sg.Engine(sg.Model(path), 0, sg.FP64)
    want = [om.efs(fr.cell, fr.positions, fr.types) for fr in frames]
    e, f, v, s = eng.calc_efs(frames)
    counts = np.bincount(eng.edges()[0])
    assert counts.min() < 96 and counts.max() > 128
    assert rel_err(e, np.array([w[0] for w in want])) < TOL
    assert rel_err(f, np.concatenate([w[1] for w in want])) < TOL
    assert rel_err(v, np.array([w[2] for w in want])) < TOL


def test_gate_rows_past_the_limit(engine_lib):
    import superlinear_gb300 as sg
    half = lattice_frame("diamond", (5, 5, 21), 3.567, 0.08, np.random.default_rng(4))  # 4,200 atoms
    cell = np.diag([2.0, 1.0, 1.0]) @ half.cell
    box = Frame(cell, np.concatenate([half.positions, half.positions + half.cell[0]]), np.concatenate([half.types] * 2))
    assert half.natoms <= 8192 < box.natoms
    eng = sg.Engine(sg.Model(os.path.join(MODELS, "effect_l3k4r2o2.sus2")), 0, sg.FP64)
    e1, f1, v1, _ = eng.calc_efs([half])
    e2, f2, v2, _ = eng.calc_efs([box])
    assert rel_err(f2, np.concatenate([f1, f1])) < TOL
    assert rel_err(e2, 2 * e1) < TOL and rel_err(v2, 2 * v1) < TOL
