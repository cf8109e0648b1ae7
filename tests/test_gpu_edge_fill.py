"""Cell-list edges against a direct search in FP64: neighbour counts on both sides of the sort's
register (32 per place) and shared-memory (64 or 128 edges) limits, a skewed cell, atoms whole cells
away from home.  The edge set and its order are exact; FP64 components differ by the grouping of
x_j + n.cell - x_i (~10 roundings of 1e3 A: 1e-12), FP32 ones by one rounding of a component below
5 A (2.4e-7, doubled for the double-float parts)."""
import os

import numpy as np
import pytest

import superlinear_gb300 as sg
from superlinear_gb300.synth import Frame

pytestmark = pytest.mark.gpu
MODEL = os.path.join(os.path.dirname(__file__), "golden", "models", "static_l3k4o2.sus2")
RC = 5.0


def direct(pos, cell):
    inv = np.linalg.inv(cell)
    off = np.floor(pos @ inv)
    home = pos - off @ cell
    out = []
    for n in np.ndindex(3, 3, 3):
        shift = (np.array(n) - 1.0) @ cell
        d = home[None] + shift - home[:, None]
        hit = (d ** 2).sum(-1) < RC * RC
        if n == (1, 1, 1):
            np.fill_diagonal(hit, False)
        i, j = np.nonzero(hit)
        out.append((i, j, d[i, j]))
    i, j, d = (np.concatenate(x) for x in zip(*out))
    o = np.lexsort((j, i))
    return i[o], j[o], d[o]


@pytest.mark.parametrize("precision", [sg.FP32, sg.FP64])
@pytest.mark.parametrize("mean", [12, 31, 63, 96, 128, 190])
def test_edges_match_direct_search(mean, precision):
    rng = np.random.default_rng(mean)
    cell = np.array([[17.0, 0, 0], [1.5, 16.5, 0], [-2.0, 1.0, 18.0]])
    n = int(mean * abs(np.linalg.det(cell)) / (4 / 3 * np.pi * RC ** 3)) + 1
    if n <= 512:  # (the cell list starts above 512 atoms)
        cell = cell * (513 / n) ** (1 / 3)
        n = 520
    pos = rng.random((n, 3)) @ cell + rng.integers(-20, 21, (n, 3)) @ cell
    eng = sg.Engine(sg.Model(MODEL), precision=precision)
    eng.calc_efs([Frame(cell, pos, np.zeros(n, np.int32))])
    ci, cj, d = eng.edges()
    wi, wj, wd = direct(pos, cell)
    counts = np.bincount(wi, minlength=n)
    assert counts.min() <= mean <= counts.max()
    np.testing.assert_array_equal(ci, wi)
    np.testing.assert_array_equal(cj, wj)
    assert np.abs(d - wd).max() < (1e-12 if precision == sg.FP64 else 5e-7)


def direct_images(pos, cell):
    """As direct(), with as many images as the cell needs, ordered by (i, j, n) of the given positions."""
    inv = np.linalg.inv(cell)
    off = np.floor(pos @ inv)
    home = pos - off @ cell
    span = [int(np.ceil(RC * np.linalg.norm(inv[:, q]))) + 1 for q in range(3)]
    out = []
    for n in np.ndindex(*(2 * s + 1 for s in span)):
        n = np.array(n) - span
        d = home[None] + n @ cell - home[:, None]
        hit = (d ** 2).sum(-1) < RC * RC
        if not n.any():
            np.fill_diagonal(hit, False)
        i, j = np.nonzero(hit)
        out.append((i, j, d[i, j], n - off[j] + off[i]))
    i, j, d, n = (np.concatenate(x) for x in zip(*out))
    o = np.lexsort((n[:, 2], n[:, 1], n[:, 0], j, i))
    return i[o], j[o], d[o]


# (cell widths, atoms, cells away from home): images of one pair, the self images of a lone atom, counts past
# the staged and the register limits, a thin cell of more than 1,024 atoms (two-word order), ranges
# close to the packable limit
SMALL = [((2.6, 2.6, 2.6), 1, 0), ((3.5, 3.5, 3.5), 8, 0), ((3.0, 3.0, 3.0), 10, 3), ((7.1, 7.1, 7.1), 64, 2),
         ((9.0, 11.0, 14.0), 333, 1), ((12.0, 20.0, 60.0), 1100, 1), ((4.0, 4.0, 30.0), 40, 29)]


@pytest.mark.parametrize("precision", [sg.FP32, sg.FP64])
@pytest.mark.parametrize("case", range(len(SMALL)))
def test_image_edges_match_direct_search(case, precision):
    widths, n, away = SMALL[case]
    rng = np.random.default_rng(case)
    cell = np.diag(widths) + np.array([[0, 0, 0], [0.1, 0, 0], [-0.2, 0.15, 0]]) * widths[0]
    grid = np.stack(np.unravel_index(rng.permutation(12 ** 3)[:n], (12, 12, 12)), -1) / 12.0  # no close pairs
    pos = (grid + rng.uniform(0, 0.02, (n, 3)) + rng.integers(-away, away + 1, (n, 3))) @ cell
    eng = sg.Engine(sg.Model(MODEL), precision=precision)
    eng.calc_efs([Frame(cell, pos, np.zeros(n, np.int32))])
    ci, cj, d = eng.edges()
    wi, wj, wd = direct_images(pos, cell)
    np.testing.assert_array_equal(ci, wi)
    np.testing.assert_array_equal(cj, wj)
    assert np.abs(d - wd).max() < (1e-12 if precision == sg.FP64 else 5e-7)
