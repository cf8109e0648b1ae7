"""Every moment-item layout of the per-atom passes against the FP64 oracle.

The passes map (radial channel k, harmonic lm) items to lanes by L (groups of (L + 1)^2 lanes side by
side up to L = 4, one group and a tail of items at L = 5) and run one of two slot counts by K; rows
of gate signals travel as 16-byte units or value by value, by F = K (L + 1).  Models of small
product graphs (scalars sum_m A_klm A_k'lm and their products) are written here for the corners of
those rules: K = 1, the last K of the short slot count, the first of the long one, K = 8, each
scaling map, one and two cutoffs, basis sizes 8 (compiled) and others (generic)."""
import numpy as np
import pytest

from conftest import rel_err
from superlinear_gb300.sus2_format import format_list
from superlinear_gb300.synth import lattice_frame

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-10
# ~100-term FP32 sums (2^-24 each) whose terms cancel to about a thirtieth of their size
FP32_FORCE = 2e-5      # relative norm
FP32_ENERGY = 1e-6     # eV/atom, absolute
GRAD_TOL = (1e-10, 1e-4)  # relative norm, FP64 plain and FP32 bulk

# (L, K, species, basis size, gated, scaling map, angular cutoff / max cutoff)
SHAPES = [
    (0, 1, 1, 8, False, "K", 1.0), (0, 8, 2, 8, True, "K", 1.0), (1, 3, 2, 8, True, "pair", 1.0),
    (1, 8, 1, 5, False, "L", 1.0), (2, 1, 2, 8, True, "K", 0.8), (2, 3, 1, 8, True, "LK", 1.0),
    (2, 4, 2, 8, True, "K", 1.0), (2, 8, 1, 8, False, "K", 1.0), (3, 1, 1, 8, True, "L", 0.7),
    (3, 3, 2, 8, True, "K", 1.0), (3, 4, 3, 16, True, "K", 1.0), (3, 5, 1, 8, True, "K", 1.0),
    (4, 1, 2, 8, True, "LK", 1.0), (4, 4, 1, 8, True, "K", 0.8), (4, 5, 2, 7, True, "K", 1.0),
    (5, 1, 1, 8, True, "K", 1.0), (5, 4, 2, 8, True, "K", 1.0), (5, 5, 1, 8, False, "pair", 0.9),
    (5, 7, 1, 8, True, "K", 1.0),
]


def write_model(path, L, K, C, B, gated, scaling_map, angular, seed):
    rng = np.random.default_rng(seed)
    H, F = (L + 1) ** 2, K * (L + 1)
    basic = [(k, l, m) for k in range(K) for l in range(L + 1) for m in range(-l, l + 1)]
    index = {b: i for i, b in enumerate(basic)}
    products, scalars, node = [], [], len(basic)
    for l in range(L + 1):
        for k in range(K):
            for k2 in {k, (k + 1) % K}:
                for m in range(-l, l + 1):
                    products.append((index[k, l, m], index[k2, l, m], node, 1.0 / (2 * l + 1)))
                scalars.append(node)
                node += 1
    for a in range(0, len(scalars) - 1, 2):  # a second level
        products.append((scalars[a], scalars[a + 1], node, 0.5))
        scalars.append(node)
        node += 1
    scalars += [index[k, 0, 0] for k in range(K)]
    S = len(scalars)
    nblk = {"pair": 1, "L": L + 1, "K": K}.get(scaling_map, F)
    warp = np.empty((nblk, 2, C * C))
    warp[:, 0], warp[:, 1] = rng.uniform(2.5, 3.5, (nblk, C * C)), rng.uniform(1.5, 2.5, (nblk, C * C))
    radial = rng.uniform(-0.5, 0.5, (F, B + C))
    radial[:, B:] = rng.uniform(0.5, 1.5, (F, C))
    f = ["MTP", "version = 1.8.0", "potential_name = shape", "scaling = 1.0e-02", f"L = {L}",
         f"scaling_map = {scaling_map}", f"species_count = {C}", "potential_tag = SUS2-SH", f"sh_l_max = {L}",
         f"sh_k_max = {K}", "sh_body_order = 4", "sh_parity = even", "radial_basis_type = RBChebyshev_sss",
         "min_dist = 1.5", "max_dist = 5.0", f"angular_max_dist = {5.0 * angular}", f"radial_basis_size = {B}",
         f"radial_funcs_count = {F}", f"shift_coeffs = {format_list(rng.uniform(-1.5, -0.5, C))}",
         f"scal_coeffs = {format_list(warp.ravel())}", "radial_coeffs", "0-0"]
    f += [format_list(row) for row in radial]
    f += [f"alpha_moments_count = {node}", f"alpha_index_basic_count = {len(basic)}",
          f"alpha_index_basic = {format_list(np.array(basic).ravel(), 3)}", "alpha_index_times_count = 0",
          "alpha_index_times = {}", f"sh_product_count = {len(products)}",
          f"sh_products = {format_list(np.array(products).ravel(), 4)}", f"alpha_scalar_moments = {S}",
          f"alpha_moment_mapping = {format_list(scalars, 1)}", "readout_mode = species"]
    if gated:
        f += ["two_layer_gate_enabled = true", "two_layer_gate_mode = mu-scalar-full",
              "two_layer_gate_radial_mode = shared-radial", f"two_layer_gate_scalar_indices = {format_list(range(S), 1)}",
              f"two_layer_gate_radial_coeffs = {format_list(rng.uniform(-0.5, 0.5, F * B))}",
              f"two_layer_gate_additive_coeffs = {format_list(rng.uniform(0.05, 0.15, C * F))}",
              f"two_layer_gate_type_coeffs = {format_list(rng.uniform(0.5, 1.5, C * F))}",
              f"two_layer_gate_weights = {format_list(rng.uniform(-1, 1, F * S) / S)}"]
    f += [f"species_coeffs = {format_list(np.ones(C))}", f"moment_coeffs = {format_list(rng.uniform(-1, 1, C * S) / S)}"]
    path.write_text("\n".join(f) + "\n")
    return str(path)


def frames(C, seed):
    """A frame of one atom, one whose centres have just under, at and above multiples of 32
    neighbours, and one larger than a warp's block."""
    rng = np.random.default_rng(seed)
    return [lattice_frame("bcc", (1, 1, 1), 3.4, 0.05, rng, species=C),
            lattice_frame("diamond", (1, 1, 2), 3.9, 0.15, rng, species=C),
            lattice_frame("fcc", (2, 3, 3), 3.9, 0.1, rng, species=C)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "L%d_K%d_C%d_B%d_%s_%s_%g" % (s[:4] + (("static", "effect")[s[4]],) + s[5:]))
def test_efs_and_gradient_of_every_layout(engine_lib, oracle_lib, tmp_path, shape):
    import superlinear_gb300 as sg
    L, K, C, B, gated, smap, angular = shape
    path = write_model(tmp_path / "m.sus2", L, K, C, B, gated, smap, angular, seed=17 * L + K)
    om, model, frs = oracle_lib.OracleModel(path), sg.Model(path), frames(C, 5)
    want = [om.efs(fr.cell, fr.positions, fr.types) for fr in frs]
    e0, f0, v0, s0 = (np.array([w[0] for w in want]), np.concatenate([w[1] for w in want]),
                      np.array([w[2] for w in want]), np.concatenate([w[3] for w in want]))
    rng = np.random.default_rng(3)
    n = [fr.natoms for fr in frs]
    ew, fw, sw = rng.normal(size=sum(n)), rng.normal(size=(sum(n), 3)), rng.normal(size=(len(frs), 3, 3))
    at, g0 = 0, 0.0
    for fr, w in zip(frs, sw):
        g0 = g0 + om.grad(fr.cell, fr.positions, fr.types, ew[at:at + fr.natoms], fw[at:at + fr.natoms], w)
        at += fr.natoms
    for prec in (sg.FP64, sg.FP32):
        g = sg.Engine(model, 0, prec)
        for split in ((None, False, True) if prec == sg.FP32 and B == 8 else (None,)):
            if split is not None:
                g.set_static_split(split)
            e, f, v, s = g.calc_efs(frs)
            if prec == sg.FP64:
                assert max(rel_err(e, e0), rel_err(f, f0), rel_err(v, v0), rel_err(s, s0)) < FP64_TOL
            else:
                assert np.linalg.norm(f - f0) <= FP32_FORCE * np.linalg.norm(f0)
                assert np.max(np.abs(e - e0) / n) <= FP32_ENERGY
        grad = g.combination_grad(frs, ew, fw, sw)
        assert np.linalg.norm(grad - g0) <= GRAD_TOL[prec == sg.FP32] * np.linalg.norm(g0)


def test_staged_evaluation_keeps_the_form_it_began_in(engine_lib, tmp_path):
    """The split gate passes keep their values in another layout than the fused ones: a switch
    between begin and finish takes effect with the next evaluation."""
    import superlinear_gb300 as sg
    path = write_model(tmp_path / "m.sus2", 3, 4, 2, 8, True, "K", 1.0, 5)
    fr = frames(2, 9)[2]
    g = sg.Engine(sg.Model(path), 0, sg.FP32)
    e0, f0, _, _ = g.calc_efs([fr])
    ei, ej, d = g.edges()
    for begin in (False, True):
        g.set_static_split(begin)
        g.stage_begin(fr.natoms, fr.types, ei, ej, d)
        g.set_static_split(not begin)
        g.stage_outer()
        e, s, f, v = g.stage_finish(fr.natoms, fr.natoms)
        assert np.linalg.norm(f - f0) <= FP32_FORCE * np.linalg.norm(f0)
        assert abs(e - e0[0]) / fr.natoms <= FP32_ENERGY
