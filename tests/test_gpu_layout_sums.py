"""Virials and site energies of every moment-item layout (tests/test_gpu_shapes.py) in FP32, fused and
split, against the FP64 oracle; with a frame of one atom and centres of 31 to 33 neighbours."""
import numpy as np
import pytest

from superlinear_gb300.synth import Frame, lattice_frame
from test_gpu_shapes import FP32_ENERGY, FP32_FORCE, SHAPES, write_model

pytestmark = pytest.mark.gpu
CUTOFF = 5.0  # of write_model
# sites: twice (products of two moments) the rounding of a sum that cancels to a thirtieth of its terms
SITE = 4 * FP32_ENERGY


def one_centre(neighbours, C, rng):
    """A centre with so many neighbours, on a shell, in a box too wide for images."""
    u = rng.normal(size=(neighbours, 3))
    shell = u / np.linalg.norm(u, axis=1)[:, None] * rng.uniform(2.5, 4.8, (neighbours, 1))
    return Frame(np.eye(3) * 40.0, np.vstack([np.zeros(3), shell]) + 20.0, rng.integers(0, C, neighbours + 1))


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "L%d_K%d_C%d_B%d_%s_%s_%g" % (s[:4] + (("static", "effect")[s[4]],) + s[5:]))
def test_virials_and_sites_of_every_layout(engine_lib, oracle_lib, tmp_path, shape):
    import superlinear_gb300 as sg
    L, K, C, B, gated, smap, angular = shape
    path = write_model(tmp_path / "m.sus2", L, K, C, B, gated, smap, angular, seed=31 * L + K)
    rng = np.random.default_rng(11)
    frames = [Frame(np.array([[0, 2.2, 2.2], [2.2, 0, 2.2], [2.2, 2.2, 0]]), rng.uniform(0, 2, (1, 3)), rng.integers(0, C, 1)),
              one_centre(31, C, rng), one_centre(32, C, rng), one_centre(33, C, rng),
              lattice_frame("fcc", (2, 2, 3), 3.9, 0.1, rng, species=C)]
    om = oracle_lib.OracleModel(path)
    eng = sg.Engine(sg.Model(path), 0, sg.FP32)
    eng.calc_efs(frames)
    counts = np.bincount(eng.edges()[0], minlength=sum(f.natoms for f in frames))
    assert [counts[k] for k in (1, 33, 66)] == [31, 32, 33] and counts[0] > 0
    for split in (False, True):
        eng.set_static_split(split)
        e, f, v, s = eng.calc_efs(frames)
        at = 0
        for k, fr in enumerate(frames):
            n = fr.natoms
            e0, f0, v0, s0 = om.efs(fr.cell, fr.positions, fr.types)[:4]
            scale = np.linalg.norm(v0) + CUTOFF * np.linalg.norm(f0)
            assert np.linalg.norm(v[k] - v0) <= FP32_FORCE * scale
            assert np.max(np.abs(s[at:at + n] - s0) / (1.0 + np.abs(s0))) <= SITE
            at += n
