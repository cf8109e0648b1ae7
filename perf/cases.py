"""The measured workloads: what a user of this framework has it do, through its public entry points.

Five kinds of work over the models under tests/golden/models, on the lattices that the tests and the
benchmark use (diamond boxes with Gaussian displacements; uneven fcc / bcc / diamond frames):

  md        repeated E / F / virial steps of one box through ``Engine.calc_efs_device`` (positions and
            outputs stay on the GPU), as a molecular-dynamics driver calls it
  host      one ``Engine.calc_efs`` call over frames held as host arrays (calc-efs)
  edges     ``Engine.efs_edges`` over a caller's neighbour list with ghosts (pair_style sus2/embedded)
  train     ``Trainer.loss_grad`` over labelled frames resident on the GPU: objective and gradient
  autograd  ``autograd.efs_device`` forward and backward: parameters -> E, F, virial -> gradient

An FP32 engine's results carry 32-bit accuracy in 64-bit arrays; they are handed on as float32, the
type such a program goes on with.  An FP64 engine's stay float64.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

import superlinear_gb300 as sg
from superlinear_gb300 import autograd as sg_autograd
from superlinear_gb300.synth import Frame

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MODELS = os.path.join(ROOT, "tests", "golden", "models")

# name -> (species, L, K, basis size, cutoff / A, gated)
_MODELS = {
    "static_l2k3o2_c2": (2, 2, 3, 8, 4.5, False),
    "static_l3k4o2": (1, 3, 4, 8, 5.0, False),
    "effect_l3k4r2o2": (2, 3, 4, 8, 5.0, True),
    "effect_l4k8r2o3": (2, 4, 8, 8, 5.5, True),
    "effect_l5k8r2o2_c3": (3, 5, 8, 8, 5.0, True),
}
_BASIS = {
    "fcc": ((0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0)),
    "bcc": ((0, 0, 0), (.5, .5, .5)),
    "diamond": ((0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0),
                (.25, .25, .25), (.25, .75, .75), (.75, .25, .75), (.75, .75, .25)),
}
DIAMOND_A = 3.567   # A, the benchmark's lattice constant
WEIGHTS = (1.0, 0.01, 0.001)  # energy, force, stress: the example training profile's
GATE_X_L2 = 1e-4    # the Trainer's default


def listed():
    return [
        # one small configuration evaluated at once, as an interactive or per-molecule caller does:
        # launches, copies and latency
        {"name": "static_host_64", "kind": "host", "model": "static_l3k4o2", "bits": 32, "count": 1,
         "nmin": 64, "nmax": 64},
        # the benchmark's MD step: 4,096 carbon atoms
        {"name": "static_md_4096", "kind": "md", "model": "static_l3k4o2", "bits": 32, "n1": 8, "n2": 8, "n3": 8},
        # a large single-species MD box
        {"name": "static_md_32768", "kind": "md", "model": "static_l3k4o2", "bits": 32, "n1": 16, "n2": 16, "n3": 16},
        # the reference-precision MD step
        {"name": "static_md_4096_fp64", "kind": "md", "model": "static_l3k4o2", "bits": 64, "n1": 8, "n2": 8, "n3": 8},
        # one domain of a pair-style run: 1,728 owned atoms, ghosts around, the driver's edge list
        {"name": "static_edges_1728", "kind": "edges", "model": "static_l2k3o2_c2", "bits": 32, "n1": 6, "n2": 6, "n3": 6},
        # a two-species Effect box of odd extents
        {"name": "effect_l3_md_1400", "kind": "md", "model": "effect_l3k4r2o2", "bits": 32, "n1": 5, "n2": 5, "n3": 7},
        # the large Effect model on a mid-sized box
        {"name": "effect_l4_md_8000", "kind": "md", "model": "effect_l4k8r2o3", "bits": 32, "n1": 10, "n2": 10, "n3": 10},
        # the benchmark's large Effect box
        {"name": "effect_l4_md_110592", "kind": "md", "model": "effect_l4k8r2o3", "bits": 32, "n1": 24, "n2": 24, "n3": 24},
        # calc-efs over a batch of uneven frames from host memory
        {"name": "effect_l3_host_64x", "kind": "host", "model": "effect_l3k4r2o2", "bits": 32, "count": 64,
         "nmin": 8, "nmax": 216},
        # the benchmark's training batch: loss and gradient
        {"name": "train_l3_256x", "kind": "train", "model": "effect_l3k4r2o2", "bits": 32, "count": 256,
         "nmin": 8, "nmax": 216},
        # three-species training on the largest angular order
        {"name": "train_l5_96x", "kind": "train", "model": "effect_l5k8r2o2_c3", "bits": 32, "count": 96,
         "nmin": 16, "nmax": 512},
        # reference-precision fitting from torch
        {"name": "autograd_l3_12x_fp64", "kind": "autograd", "model": "effect_l3k4r2o2", "bits": 64, "count": 12,
         "nmin": 8, "nmax": 216},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("md", "md", "host", "edges", "train", "autograd"))
    bits = 32 if rng.random() < 0.75 else 64
    if kind == "md":
        model = rng.choice(("static_l2k3o2_c2", "static_l3k4o2", "effect_l3k4r2o2", "effect_l4k8r2o3"))
        # conventional cells, spread over the logarithm; FP64 boxes an eighth of the atoms
        cells = _log_int(rng, 8, 13000 if bits == 32 else 1000)
        n1 = max(1, int(round(cells ** (1 / 3) * rng.uniform(0.7, 1.2))))
        n2 = max(1, int(round((cells / n1) ** 0.5 * rng.uniform(0.8, 1.2))))
        return {"kind": kind, "model": model, "bits": bits, "n1": n1, "n2": n2, "n3": max(1, round(cells / (n1 * n2)))}
    if kind == "edges":
        return {"kind": kind, "model": rng.choice(("static_l2k3o2_c2", "static_l3k4o2")), "bits": bits,
                "n1": rng.randint(1, 9), "n2": rng.randint(1, 9), "n3": rng.randint(2, 9)}
    model = rng.choice(("effect_l3k4r2o2", "effect_l5k8r2o2_c3") if kind != "host" else
                       ("static_l2k3o2_c2", "static_l3k4o2", "effect_l3k4r2o2", "effect_l4k8r2o3"))
    most = {"host": 200, "train": 300, "autograd": 60}[kind]
    if bits == 64 or model == "effect_l5k8r2o2_c3":
        most //= 6
    nmax = rng.choice((64, 128, 216))
    return {"kind": kind, "model": model, "bits": bits, "count": _log_int(rng, 1, most), "nmin": rng.choice((4, 8, 16)),
            "nmax": nmax}


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------

def _model_path(case):
    return os.path.join(MODELS, case["model"] + ".sus2")


def _lattice(kind, reps, a, sigma, species, rng):
    grid = np.stack(np.meshgrid(*(np.arange(n) for n in reps), indexing="ij"), -1).reshape(-1, 1, 3)
    pos = ((grid + np.array(_BASIS[kind])[None]).reshape(-1, 3)) * a
    pos = pos + rng.normal(0.0, sigma, pos.shape)
    return np.diag([n * a for n in reps]).astype(np.float64), pos, rng.integers(0, species, len(pos)).astype(np.int32)


def _box(case, seed):
    rng = np.random.default_rng([seed, 1])
    return _lattice("diamond", (case["n1"], case["n2"], case["n3"]), DIAMOND_A, 0.08, _MODELS[case["model"]][0], rng)


def _frames(case, seed):
    """Uneven frames: sizes over the range's logarithm (the case's own), lattice constants 2.9 - 4.3 A."""
    rng = np.random.default_rng([seed, 2])
    size_rng = np.random.default_rng([case["count"], case["nmin"], case["nmax"]])
    sizes = {k: [(len(b) * n1 * n2 * n3, (n1, n2, n3)) for n1 in range(1, 7) for n2 in range(n1, 7) for n3 in range(n2, 7)]
             for k, b in _BASIS.items()}
    out = []
    for q in range(case["count"]):
        kind = ("diamond", "fcc", "bcc")[q % 3]
        target = math.exp(size_rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        reps = min(sizes[kind], key=lambda s: (abs(s[0] - target), s[1][2] - s[1][0]))[1]
        a = DIAMOND_A if case["count"] == 1 else rng.uniform(2.9, 4.3)
        out.append(_lattice(kind, tuple(rng.permutation(reps)), a, 0.08, _MODELS[case["model"]][0], rng))
    return out


def _labels(frames, seed):
    """Energy, force and stress labels of the size such frames have (eV, eV / A, eV)."""
    rng = np.random.default_rng([seed, 3])
    out = []
    for _, pos, _ in frames:
        n = len(pos)
        s = rng.normal(0.0, 0.05 * n, (3, 3))
        out.append((-0.4 * n + rng.normal(0.0, 0.02 * n), rng.normal(0.0, 0.5, (n, 3)), 0.5 * (s + s.T)))
    return out


def _params(base, seed):
    return base * (1.0 + 0.02 * np.random.default_rng([seed, 4]).normal(size=base.size))


def _weights(natoms, seed):
    """Upstream gradients of (E, F, virial), as a loss written in torch sends them."""
    rng = np.random.default_rng([seed, 5])
    return (rng.normal(0, 1, len(natoms)), rng.normal(0, 0.1, (int(sum(natoms)), 3)), rng.normal(0, 0.01, (len(natoms), 6)))


def _domain(case, seed):
    """One domain of a decomposed box: owned atoms first, then the ghosts within the cutoff of the
    domain, and the owned centres' directed edges."""
    species, rc = _MODELS[case["model"]][0], _MODELS[case["model"]][4]
    rng = np.random.default_rng([seed, 6])
    reps, shell = (case["n1"], case["n2"], case["n3"]), 2
    grid = np.stack(np.meshgrid(*(np.arange(-shell, n + shell) for n in reps), indexing="ij"), -1).reshape(-1, 1, 3)
    site = (grid + np.array(_BASIS["diamond"])[None]).reshape(-1, 3)
    inside = ((site >= 0) & (site < np.array(reps))).all(1)
    order = np.concatenate([np.flatnonzero(inside), np.flatnonzero(~inside)])
    site, owned = site[order], int(inside.sum())
    pos = site * DIAMOND_A + rng.normal(0.0, 0.08, site.shape)
    types = rng.integers(0, species, len(pos)).astype(np.int32)
    ei, ej = [], []
    for a in range(0, owned, 256):
        d2 = ((pos[a:min(a + 256, owned), None, :] - pos[None, :, :]) ** 2).sum(-1)
        i, j = np.nonzero((d2 < rc * rc) & (d2 > 0))
        ei.append(i + a)
        ej.append(j)
    ei, ej = np.concatenate(ei).astype(np.int32), np.concatenate(ej).astype(np.int32)
    return owned, types, ei, ej, pos[ej] - pos[ei]


class _Labelled(Frame):
    def __init__(self, frame, label):
        super().__init__(*frame, energy=label[0], forces=label[1], stress=label[2])


def prepare(case, seed):
    model = sg.Model(_model_path(case))
    engine = sg.Engine(model, 0, sg.FP32 if case["bits"] == 32 else sg.FP64)
    state = {"kind": case["kind"], "engine": engine, "bits": case["bits"]}
    if case["kind"] == "md":
        cell, pos, types = _box(case, seed)
        n = len(pos)
        state.update(natoms=np.array([n], np.int32), cells=cell[None], pos=torch.from_numpy(pos).cuda(),
                     types=torch.from_numpy(types).cuda(), out=torch.empty(7 + 4 * n, dtype=torch.float64, device="cuda"))
    elif case["kind"] == "host":
        state["frames"] = [Frame(*f) for f in _frames(case, seed)]
    elif case["kind"] == "edges":
        state["domain"] = _domain(case, seed)
    elif case["kind"] == "train":
        frames = _frames(case, seed)
        state["trainer"] = sg.Trainer(engine, [_Labelled(f, y) for f, y in zip(frames, _labels(frames, seed))], *WEIGHTS)
        state["params"] = _params(model.params(), seed)
    else:
        frames = _frames(case, seed)
        natoms = np.array([len(f[1]) for f in frames], np.int32)
        state.update(natoms=natoms, cells=np.stack([f[0] for f in frames]),
                     pos=torch.from_numpy(np.concatenate([f[1] for f in frames])).cuda(),
                     types=torch.from_numpy(np.concatenate([f[2] for f in frames])).cuda(),
                     params=torch.from_numpy(_params(model.params(), seed)),
                     weights=[torch.from_numpy(w).cuda() for w in _weights(natoms, seed)])
    return state


def _efs(e, f, v, s):
    return {"energy": e, "forces": f, "virial": v, "site": s}


def run(state):
    kind, engine = state["kind"], state["engine"]
    host = np.float32 if state["bits"] == 32 else np.float64
    if kind == "md":
        out, n = state["out"], int(state["natoms"][0])
        at = out.data_ptr()
        engine.calc_efs_device(state["natoms"], state["cells"], state["pos"].data_ptr(), state["types"].data_ptr(), at,
                               at + 8, at + 8 * (1 + 3 * n), at + 8 * (7 + 3 * n))
        out = out.float() if state["bits"] == 32 else out
        return _efs(out[:1], out[1:1 + 3 * n].view(n, 3), out[1 + 3 * n:7 + 3 * n], out[7 + 3 * n:])
    if kind == "host":
        return _efs(*(x.astype(host, copy=False) for x in engine.calc_efs(state["frames"])))
    if kind == "edges":
        e, s, f, v = engine.efs_edges(*state["domain"])
        return _efs(np.array([e], host), f.astype(host, copy=False), v.astype(host, copy=False), s.astype(host, copy=False))
    if kind == "train":
        loss, grad = state["trainer"].loss_grad(state["params"])
        return {"loss": np.array([loss], host), "grad": grad.astype(host, copy=False)}
    p = state["params"].clone().requires_grad_(True)
    e, f, v = sg_autograd.efs_device(p, engine, state["natoms"], state["cells"], state["pos"], state["types"])
    we, wf, wv = state["weights"]
    ((e * we).sum() + (f * wf).sum() + (v * wv).sum()).backward()
    outs = {"energy": e.detach(), "forces": f.detach(), "virial": v.detach(), "grad": p.grad}
    return {k: x.float() for k, x in outs.items()} if state["bits"] == 32 else outs


def _atoms(case):
    """(atoms, mean number density / A^-3), expected."""
    if case["kind"] in ("md", "edges"):
        return 8 * case["n1"] * case["n2"] * case["n3"], 8 / DIAMOND_A ** 3
    lo, hi = case["nmin"], case["nmax"]
    mean = lo if lo == hi else (hi - lo) / math.log(hi / lo)
    if case["count"] == 1:
        return mean, 8 / DIAMOND_A ** 3
    # mean of 1 / a^3 over the lattice constants, thirds of 8-, 4- and 2-atom cells
    return case["count"] * mean, (14 / 3) * (2.9 ** -2 - 4.3 ** -2) / (2 * (4.3 - 2.9))


def work(case):
    """Per edge and pass: the harmonics (4 H) and their gradient contraction (8 H), the warped
    Chebyshev values and slopes (5 B + 30 per radial channel), the radial functions and their
    slopes (4 B + 8 each), the moment sums and their adjoints (2 and 4 per moment); the Effect model
    has two passes and the gate signal (6 per function); a parameter gradient repeats the forward
    with tangents and adds its reverse (4 times the value-and-force work)."""
    species, L, K, B, rc, gated = _MODELS[case["model"]]
    n, rho = _atoms(case)
    edges = n * rho * 4 / 3 * math.pi * rc ** 3
    H, F = (L + 1) ** 2, K * (L + 1)
    one = 12 * H + K * (5 * B + 30) + F * (4 * B + 8) + 6 * K * H
    flops = edges * ((2 * one + 6 * F) if gated else one)
    nbytes = n * (24 + 4 + 32)
    if case["kind"] == "edges":
        nbytes += edges * 32
    if case["kind"] in ("train", "autograd"):
        flops *= 5
        nbytes += n * 32
    return {"bytes": float(nbytes), "flops": float(flops)}


# ------------------------------------------------------------------------------------------------
# the same quantities in 64 bits, from the definitions, in plain torch
# ------------------------------------------------------------------------------------------------

class _Sus2:
    """A .sus2 file's fields and the tables that the evaluation needs."""

    def __init__(self, path):
        self.f, rows, depth, key = {}, [], 0, None
        with open(path) as fh:
            for line in fh.read().splitlines()[1:]:
                line = line.strip()
                if not line:
                    continue
                if depth:
                    self.f[key] += " " + line
                elif "=" in line:
                    key, value = (x.strip() for x in line.split("=", 1))
                    self.f[key] = value
                elif line.startswith("{"):
                    rows.append(line)
                    continue
                else:
                    continue
                depth += line.count("{") - line.count("}")
        self.f["radial_coeffs"] = ",".join(rows)
        self.C, self.L, self.K, self.B, self.F, self.M, self.S = (int(self.f[k]) for k in (
            "species_count", "sh_l_max", "sh_k_max", "radial_basis_size", "radial_funcs_count", "alpha_moments_count",
            "alpha_scalar_moments"))
        self.H, self.rc, self.scaling = (self.L + 1) ** 2, float(self.f["max_dist"]), float(self.f["scaling"])
        self.gated = self.f.get("two_layer_gate_enabled") == "true"
        self.basic = self.num("alpha_index_basic", int).reshape(-1, 3)
        self.prod = self.num("sh_products").reshape(-1, 4)
        self.scalar = self.num("alpha_moment_mapping", int)
        C, K, F, L = self.C, self.K, self.F, self.L
        names = [("shift_coeffs", (C,)), ("scal_coeffs", (K, 2, C, C)), ("radial_coeffs", (F, self.B + C))]
        if self.gated:
            self.gate = self.num("two_layer_gate_scalar_moment_indices", int)
            if not len(self.gate):
                self.gate = self.scalar[self.num("two_layer_gate_scalar_indices", int)]
            self.grank = int(self.f["two_layer_gate_k_rank"])
            names.append(("two_layer_gate_radial_coeffs", (F, self.B)))
            if self.f.get("two_layer_gate_scaling_mode", "shared-scaling") == "decoupled":
                names.append(("two_layer_gate_scaling_coeffs", (K, 2, C, C)))
            names += [("two_layer_gate_additive_coeffs", (C, F)), ("two_layer_gate_type_coeffs", (C, F)),
                      ("two_layer_gate_weights", (F, len(self.gate))),
                      ("two_layer_gate_k_rank_weights", (L + 1, self.grank, K))]
        self.rank = int(self.f["outer_k_rank"])
        names += [("outer_k_rank1_weights", (L + 1, self.rank, K)), ("species_coeffs", (C,)), ("moment_coeffs", (C, self.S))]
        self.names = names
        self.vector = np.concatenate([self.num(k).reshape(-1) for k, _ in names])

    def num(self, key, kind=float):
        text = self.f.get(key, "").replace("{", " ").replace("}", " ").replace(",", " ")
        return np.array([kind(float(x)) for x in text.split()], dtype=np.float64 if kind is float else np.int64)

    def split(self, vector):
        out, at = {}, 0
        for name, shape in self.names:
            n = int(np.prod(shape))
            out[name] = vector[at:at + n].view(shape)
            at += n
        return out


def _harmonics(u, L):
    """Real Y_lm on unit vectors, [E, (L + 1)^2], index l^2 + l + m."""
    cos, sin = [torch.ones_like(u[:, 0])], [torch.zeros_like(u[:, 0])]
    for m in range(L):
        cos.append(u[:, 0] * cos[m] - u[:, 1] * sin[m])
        sin.append(u[:, 0] * sin[m] + u[:, 1] * cos[m])
    out = [None] * (L + 1) ** 2
    for m in range(L + 1):
        before, p = torch.zeros_like(u[:, 2]), torch.full_like(u[:, 2], float(math.prod(range(1, 2 * m, 2))))
        for l in range(m, L + 1):
            if l > m:
                before, p = p, ((2 * l - 1) * u[:, 2] * p - (l + m - 1) * before) / (l - m)
            norm = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            if m == 0:
                out[l * l + l] = norm * p
            else:
                out[l * l + l + m] = math.sqrt(2) * norm * p * cos[m]
                out[l * l + l - m] = math.sqrt(2) * norm * p * sin[m]
    return torch.stack(out, 1)


def _moments(m, d, ei, n, pair, coeff, scal, weight):
    """A[i, k, h] = sum_e weight[e, mu] R_mu(r_e) Y_h(d_e), mu = k (L + 1) + l(h)."""
    r = d.norm(dim=1)
    Y = _harmonics(d / r[:, None], m.L)
    slope, shift = (scal[:, q].reshape(m.K, -1)[:, pair].t() for q in (0, 1))
    xi = torch.tanh(slope * (r[:, None] - shift) / 2)
    T = [torch.ones_like(xi), xi]
    while len(T) < m.B:
        T.append(2 * xi * T[-1] - T[-2])
    radial = torch.einsum("ekb,klb->ekl", torch.stack(T[:m.B], 2), coeff.view(m.K, m.L + 1, m.B))
    radial = radial * (m.scaling * (r - m.rc) ** 2)[:, None, None] * weight.view(-1, m.K, m.L + 1)
    l_of = torch.tensor([l for l in range(m.L + 1) for _ in range(2 * l + 1)], device=d.device)
    return torch.zeros(n, m.K, m.H, dtype=d.dtype, device=d.device).index_add(0, ei, radial[:, :, l_of] * Y[:, None, :])


def _graph(m, A, rank, begin, first, last, w):
    """Basic moments, rank contraction and the products [first, last): node values [n, M]."""
    dev, n = A.device, A.shape[0]
    k, l, mm = (torch.from_numpy(np.ascontiguousarray(m.basic[:, q])).to(dev) for q in range(3))
    v = torch.zeros(n, m.M, dtype=A.dtype, device=dev)
    v = v.index_add(1, torch.arange(len(k), device=dev), A[:, k, l * l + l + mm])
    for a in range(rank):
        dst = begin + rank * (m.H - (l + 1) ** 2) + (rank - 1 - a) * (2 * l + 1) + mm + l
        v = v.index_add(1, dst, v[:, :len(k)] * w[l, a, k])
    level, steps = np.zeros(m.M, int), {}
    rows = m.prod[first:last]
    made = {}
    for a, b, out, _ in rows:  # a node's level is one above its deepest factor's
        made[int(out)] = max(made.get(int(out), 0), level[int(a)] + 1, level[int(b)] + 1)
        level[int(out)] = made[int(out)]
    for row in rows:
        steps.setdefault(level[int(row[2])], []).append(row)
    for lv in sorted(steps):
        t = torch.from_numpy(np.array(steps[lv])).to(dev)
        a, b, out = (t[:, q].long() for q in range(3))
        v = v.index_add(1, out, t[:, 3] * v[:, a] * v[:, b])
    return v


def _energy(m, p, d, ei, ej, types, n):
    """(site energies [n], gate signals [n, F] or None, node values) from edge vectors d."""
    f = m.f
    ti, tj = types[ei], types[ej]
    pair = ti * m.C + tj
    tau = p["radial_coeffs"][:, m.B:].t()
    h, source = None, tau[tj]
    begin = int(f["outer_k_rank1_product_begin"])
    if m.gated:
        g = p["two_layer_gate_type_coeffs"]
        A = _moments(m, d, ei, n, pair, p["two_layer_gate_radial_coeffs"], p.get("two_layer_gate_scaling_coeffs", p["scal_coeffs"]),
                     g[ti] * g[tj])
        v = _graph(m, A, m.grank, int(f["two_layer_gate_k_rank_basic_begin"]), int(f["two_layer_gate_k_rank_product_begin"]),
                   int(f["two_layer_gate_k_rank_product_end"]), p["two_layer_gate_k_rank_weights"])
        h = v[:, torch.from_numpy(m.gate).to(d.device)] @ p["two_layer_gate_weights"].t()
        source = source + p["two_layer_gate_additive_coeffs"][tj] * h[ej]
    A = _moments(m, d, ei, n, pair, p["radial_coeffs"][:, :m.B], p["scal_coeffs"], tau[ti] * source)
    v = _graph(m, A, m.rank, int(f["outer_k_rank1_basic_begin"]), begin, len(m.prod), p["outer_k_rank1_weights"])
    lin = p["moment_coeffs"][types]
    site = p["species_coeffs"][types] + p["shift_coeffs"][types] + (lin * v[:, torch.from_numpy(m.scalar).to(d.device)]).sum(1)
    return site, h


def _edges(frames, rc, dev):
    """Directed edges of a batch of orthogonal periodic frames: (i, j, d, frame of i)."""
    I, J, D, Fr, base = [], [], [], [], 0
    for q, (cell, pos, _) in enumerate(frames):
        x, box = torch.from_numpy(pos).to(dev), torch.from_numpy(np.diag(cell).copy()).to(dev)
        n = len(pos)
        x = x - torch.floor(x / box) * box
        reach = [int(math.ceil(rc / b)) for b in np.diag(cell)]
        once = all(b > 2 * rc for b in np.diag(cell))
        shifts = [(0, 0, 0)] if once else [(a, b, c) for a in range(-reach[0], reach[0] + 1)
                                           for b in range(-reach[1], reach[1] + 1) for c in range(-reach[2], reach[2] + 1)]
        step = max(1, (1 << 24) // n)
        for a in range(0, n, step):
            diff = x[None] - x[a:a + step, None]
            if once:
                diff = diff - torch.round(diff / box) * box
            for s in shifts:
                v = diff + torch.tensor(s, dtype=x.dtype, device=dev) * box
                r2 = v.square().sum(-1)
                i, j = torch.nonzero((r2 < rc * rc) & (r2 > 1e-12), as_tuple=True)
                I.append(i + a + base)
                J.append(j + base)
                D.append(v[i, j])
                Fr.append(torch.full_like(i, q))
        base += n
    return torch.cat(I), torch.cat(J), torch.cat(D), torch.cat(Fr)


def _evaluate(m, p, frames, dev, graph):
    """E, F, virial, site energies and gate signals of a batch; with `graph`, differentiable in p."""
    ei, ej, d, _ = _edges(frames, m.rc, dev)
    types = torch.from_numpy(np.concatenate([f[2] for f in frames])).long().to(dev)
    n = len(types)
    frame_of = torch.repeat_interleave(torch.arange(len(frames), device=dev),
                                       torch.tensor([len(f[1]) for f in frames], device=dev))
    d.requires_grad_(True)
    site, h = _energy(m, p, d, ei, ej, types, n)
    g, = torch.autograd.grad(site.sum(), d, create_graph=graph)
    F = torch.zeros(n, 3, dtype=d.dtype, device=dev).index_add(0, ei, g).index_add(0, ej, -g)
    w = -torch.stack([d[:, a] * g[:, b] for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))], 1)
    zero = torch.zeros(len(frames), dtype=d.dtype, device=dev)
    E = zero.index_add(0, frame_of, site)
    V = torch.zeros(len(frames), 6, dtype=d.dtype, device=dev).index_add(0, frame_of[ei], w)
    return E, F, V, site, h, (ej, types, frame_of)


def _groups(frames, m, most):
    """The batch in runs of frames of about `most` edges."""
    group, size = [], 0.0
    for f in frames:
        e = len(f[1]) ** 2 / abs(np.linalg.det(f[0])) * 4 / 3 * math.pi * m.rc ** 3
        if group and size + e > most:
            yield group
            group, size = [], 0.0
        group.append(f)
        size += e
    if group:
        yield group


def _objective(m, p, frames, labels, dev):
    """The training objective's sum over these frames (energy, force, stress and gate-x terms)."""
    E, F, V, _, h, (ej, types, frame_of) = _evaluate(m, p, frames, dev, True)
    wE, wF, wS = WEIGHTS
    F0 = torch.from_numpy(np.concatenate([y[1] for y in labels])).to(dev)
    loss = wF * (F - F0).square().sum()
    S = V[:, [0, 3, 4, 3, 1, 5, 4, 5, 2]]
    n = torch.tensor([float(len(f[1])) for f in frames], dtype=E.dtype, device=dev)
    S0 = torch.from_numpy(np.stack([y[2].reshape(9) for y in labels])).to(dev)
    E0 = torch.tensor([y[0] for y in labels], dtype=E.dtype, device=dev)
    loss = loss + (wS * (S - S0).square().sum(1) / n).sum() + (wE * (E - E0).square() / n).sum()
    if m.gated:
        # per frame: coeff / (neighbour types present x F x edges of that neighbour type) x (alpha h)^2
        key = frame_of[ej] * m.C + types[ej]
        count = torch.bincount(key, minlength=len(frames) * m.C).view(-1, m.C)
        active = (count > 0).sum(1)
        norm = GATE_X_L2 / (active[:, None] * m.F * count.clamp(min=1)).double()
        x = p["two_layer_gate_additive_coeffs"][types] * h
        degree = torch.bincount(ej, minlength=len(types)).double()
        loss = loss + (norm[frame_of, types] * degree * x.square().sum(1)).sum()
    return loss


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n, rho = _atoms(case)
    m = _Sus2(_model_path(case))
    edges = n * rho * 4 / 3 * math.pi * m.rc ** 3
    # boxes whose evaluation in 64 bits takes long
    if edges * (2 * m.K * m.H if m.gated else m.K * m.H) > 5e8:
        return None
    vec = torch.from_numpy(m.vector).to(dev)
    if case["kind"] == "edges":
        owned, types, ei, ej, d = _domain(case, seed)
        ei, ej = (torch.from_numpy(x).long().to(dev) for x in (ei, ej))
        d = torch.from_numpy(d).to(dev).requires_grad_(True)
        t = torch.from_numpy(types).long().to(dev)
        site, _ = _energy(m, m.split(vec), d, ei, ej, t, len(types))
        site = site[:owned]
        g, = torch.autograd.grad(site.sum(), d)
        F = torch.zeros(len(types), 3, dtype=d.dtype, device=dev).index_add(0, ei, g).index_add(0, ej, -g)
        w = -torch.stack([(d[:, a] * g[:, b]).sum() for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))])
        return {k: x.detach().cpu() for k, x in _efs(site.sum().view(1), F, w, site).items()}
    if case["kind"] in ("md", "host"):
        frames = [_box(case, seed)] if case["kind"] == "md" else _frames(case, seed)
        parts = [[x.detach().cpu() for x in _evaluate(m, m.split(vec), g, dev, False)[:4]] for g in _groups(frames, m, 2e5)]
        E, F, V, S = (torch.cat(x) for x in zip(*parts))
        return _efs(E, F, V.view(6) if case["kind"] == "md" else V, S)
    frames = _frames(case, seed)
    vec = torch.from_numpy(_params(m.vector, seed)).to(dev).requires_grad_(True)
    grad = torch.zeros_like(vec)
    at, total, parts = 0, 0.0, []
    if case["kind"] == "train":
        labels = _labels(frames, seed)
        for group in _groups(frames, m, 1e5):
            loss = _objective(m, m.split(vec), group, labels[at:at + len(group)], dev) / len(frames)
            grad += torch.autograd.grad(loss, vec)[0]
            total += float(loss.detach())
            at += len(group)
        return {"loss": torch.tensor([total], dtype=torch.float64), "grad": grad.cpu()}
    we, wf, wv = (torch.from_numpy(w).to(dev) for w in _weights([len(f[1]) for f in frames], seed))
    atom = 0
    for group in _groups(frames, m, 1e5):
        E, F, V = _evaluate(m, m.split(vec), group, dev, True)[:3]
        k = len(F)
        J = (E * we[at:at + len(group)]).sum() + (F * wf[atom:atom + k]).sum() + (V * wv[at:at + len(group)]).sum()
        grad += torch.autograd.grad(J, vec)[0]
        parts.append([x.detach().cpu() for x in (E, F, V)])
        at, atom = at + len(group), atom + k
    E, F, V = (torch.cat(x) for x in zip(*parts))
    return {"energy": E, "forces": F, "virial": V, "grad": grad.cpu()}
