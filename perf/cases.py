"""The work that programs have this solver do, as measurable cases.

A cluster solver is called in a few ways, and each has its cases here:

  apply    y = H x on device vectors (with or without the three dot products of a
           Krylov step), the Hamiltonian plugin point that an outer eigensolver
           or time evolution drives
  host     y += H x on host vectors, the plugin point as the C++ library calls it
  solve    new instances of a model at new parameters: ground state, Green
           function, G on Matsubara frequencies (one CDMFT or VCA point, a batch
           of bath points, a cluster with a point group)
  batch    many small clusters of uneven size in one call, every sector
  omega    the (frequency, wavevector) sum of the Potthoff functional (VCA)
  hybrid   the CDMFT host function on a wavevector grid
  mixed    y = H x in the symmetry-adapted basis of a cluster with a point group
  train    epochs of the VCA surrogate (BF16 tensor-core products, FP32 Adam)

Everything but the surrogate is FP64. Sizes are those of this repository's
workloads, tests and benchmark, and generic ones between them.
"""
from __future__ import annotations

import ctypes
import itertools
import math

import numpy as np
import torch

import pyqcm_b200 as qed
from pyqcm_b200 import lattice, surrogate
from pyqcm_b200 import workloads as W

_count = itertools.count(1)  # model names and instance labels are process-global

BETA = 50.0


# ---------------------------------------------------------------- the cases ----

def listed():
    return [
        # the smallest product: one 8-site chain at half filling, 4900 states; launches count
        {"name": "apply_chain8", "kind": "apply", "nx": 8, "ny": 1, "up": 4, "dn": 4, "tp": False, "neel": False,
         "bath": 0, "dots": False},
        # the Krylov product of the standard CDMFT cluster, 2x2 plaquette + 8 bath orbitals, 853776
        # states: every hybridisation is a hopping amplitude of its own
        {"name": "apply_bath12", "kind": "apply", "nx": 2, "ny": 2, "up": 6, "dn": 6, "tp": False, "neel": False,
         "bath": 8, "dots": True},
        # the largest: the 4x4 cluster with t' at half filling, 1.66e8 states
        {"name": "apply_4x4", "kind": "apply", "nx": 4, "ny": 4, "up": 8, "dn": 8, "tp": True, "neel": False,
         "bath": 0, "dots": False},
        # odd sizes: 15 sites, one hole away from half filling, rows of 6435, a staggered field
        # that makes the two spins different, with the dot products
        {"name": "apply_3x5_odd", "kind": "apply", "nx": 3, "ny": 5, "up": 7, "dn": 7, "tp": True, "neel": True,
         "bath": 0, "dots": True},
        # host vectors through the plugin point: 2x7, 1.18e7 states
        {"name": "host_2x7", "kind": "host", "nx": 2, "ny": 7, "up": 7, "dn": 7, "tp": True, "neel": False, "bath": 0},
        # one CDMFT point: the plaquette with 8 bath orbitals at new bath parameters
        {"name": "solve_bath12", "kind": "solve", "nx": 2, "ny": 2, "up": 6, "dn": 6, "tp": False, "neel": False,
         "bath": 8, "sym": False, "n": 1, "nz": 256},
        # one point of a larger cluster through its point group: 3x4 with both mirrors, 12 sites
        {"name": "solve_3x4_c2v", "kind": "solve", "nx": 3, "ny": 4, "up": 6, "dn": 6, "tp": True, "neel": False,
         "bath": 0, "sym": True, "n": 1, "nz": 256},
        # uneven clusters of 4 to 10 sites with every sector, one batched call
        {"name": "batch_random", "kind": "batch", "n": 64, "nz": 64},
        # one evaluation of the VCA integrand on 2x5 clusters, both spins
        {"name": "omega_2x5", "kind": "omega", "ny": 5, "neel": True, "nw": 64, "side": 64, "poles": 480},
        # one CDMFT host function, plaquette with bath, default grid of 32 x 32 wavevectors
        {"name": "hybrid_2x2", "kind": "hybrid", "ny": 2, "neel": False, "bath": 8, "nw": 64, "side": 32,
         "poles": 360},
        # the product in the symmetry-adapted basis of a 14-site ladder, 2.9e6 states
        {"name": "mixed_2x7", "kind": "mixed", "nx": 2, "ny": 7, "up": 7, "dn": 7, "tp": True, "irrep": 0},
        # the VCA surrogate: 20 epochs over 4096 points in batches of 256
        {"name": "train_4096", "kind": "train", "points": 4096, "batch": 256, "epochs": 20},
    ]


#: lattices of 4 to 16 sites that apply, host and mixed cases are drawn from
SHAPES = [(2, 2), (2, 3), (3, 2), (8, 1), (2, 4), (3, 3), (10, 1), (2, 5), (11, 1), (3, 4), (12, 1), (2, 6), (13, 1),
          (2, 7), (14, 1), (3, 5), (4, 4)]

#: the geometries of the random clusters (workloads.random_batch)
BATCH_SHAPES = [(2, 2), (2, 3), (2, 4), (8, 1), (10, 1)]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _filled(rng, lo, hi, shapes, most=16):
    """A lattice and a filling whose sector is near a log-uniform dimension in [lo, hi]."""
    want = _log(rng, lo, hi)
    near = []
    for nx, ny in shapes:
        n = nx * ny
        if n > most:
            continue
        for up in range(1, n):
            for dn in range(1, n):
                d = math.comb(n, up) * math.comb(n, dn)
                if want / 1.6 <= d <= want * 1.6 and d <= hi:
                    near.append((nx, ny, up, dn))
    return rng.choice(near) if near else (8, 1, 4, 4)


def draw(rng):
    kind = rng.choices(["apply", "bath", "host", "solve", "batch", "omega", "hybrid", "mixed", "train"],
                       [30, 12, 8, 13, 8, 9, 9, 8, 3])[0]
    flag = lambda p=0.5: rng.random() < p  # noqa: E731
    if kind == "apply":
        nx, ny, up, dn = _filled(rng, 3e3, 1.656e8, SHAPES)
        return {"kind": "apply", "nx": nx, "ny": ny, "up": up, "dn": dn, "tp": flag() and ny > 1 and nx > 1,
                "neel": flag(0.4), "bath": 0, "dots": flag()}
    if kind == "bath":
        bath = rng.choice([4, 8, 8])
        n = 4 + bath
        return {"kind": "apply", "nx": 2, "ny": 2, "up": n // 2 - rng.randint(0, 2), "dn": n // 2 - rng.randint(0, 2),
                "tp": flag(0.2), "neel": False, "bath": bath, "dots": flag()}
    if kind == "host":
        nx, ny, up, dn = _filled(rng, 1e4, 1.2e7, SHAPES, 14)
        return {"kind": "host", "nx": nx, "ny": ny, "up": up, "dn": dn, "tp": flag() and ny > 1 and nx > 1,
                "neel": flag(0.3), "bath": 0}
    if kind == "solve":
        form = rng.choice(["bath", "cluster", "sym"])
        if form == "bath":
            bath = rng.choice([4, 8, 8])
            n = 4 + bath
            return {"kind": "solve", "nx": 2, "ny": 2, "up": n // 2, "dn": n // 2, "tp": flag(0.2), "neel": False,
                    "bath": bath, "sym": False, "n": rng.choice([1, 1, 2, 3, 5]), "nz": rng.choice([64, 100, 256])}
        nx, ny = rng.choice([(2, 4), (2, 5), (9, 1), (11, 1), (2, 6)] if form == "cluster" else [(2, 4), (2, 5), (2, 6)])
        up = nx * ny // 2
        return {"kind": "solve", "nx": nx, "ny": ny, "up": up, "dn": nx * ny - up - (form == "cluster" and flag(0.3)),
                "tp": ny > 1, "neel": form == "cluster" and flag(0.3), "bath": 0, "sym": form == "sym", "n": 1,
                "nz": rng.choice([64, 100, 256])}
    if kind == "batch":
        return {"kind": "batch", "n": round(_log(rng, 5, 64)), "nz": rng.choice([32, 64])}
    if kind == "omega":
        return {"kind": "omega", "ny": rng.randint(1, 6), "neel": flag(0.7), "nw": rng.choice([16, 33, 64]),
                "side": rng.choice([16, 25, 32, 48, 64]), "poles": 2 * round(_log(rng, 30, 300))}
    if kind == "hybrid":
        return {"kind": "hybrid", "ny": rng.randint(1, 4), "neel": flag(0.3), "bath": rng.choice([4, 8]),
                "nw": rng.choice([20, 31, 64, 100]), "side": rng.choice([12, 16, 32, 33]),
                "poles": 2 * round(_log(rng, 30, 300))}
    if kind == "mixed":
        nx, ny = rng.choice([(2, 4), (2, 5), (3, 4), (2, 6), (2, 7)])
        n = nx * ny
        return {"kind": "mixed", "nx": nx, "ny": ny, "up": n // 2 - rng.randint(0, 1), "dn": n // 2 - rng.randint(0, 1),
                "tp": flag(), "irrep": rng.randint(0, 3)}
    return {"kind": "train", "points": rng.choice([600, 1024, 2048, 3000]), "batch": rng.choice([64, 128, 256]),
            "epochs": rng.randint(3, 12)}


# ------------------------------------------------------------ the programs ----

class _Held:
    """What a program keeps between calls; its instances are erased with it."""

    def __init__(self, case):
        self.case = case
        self.labels = []

    def __del__(self):
        for name in ("H", "net"):
            self.__dict__.pop(name, None)
        for label in self.labels:
            try:
                qed.erase_model_instance(label)
            except Exception:
                pass


def _mirrors(nx, ny):
    """The two mirrors of an nx x ny cluster as site permutations (1-based)."""
    site = lambda x, y: 1 + x + nx * y  # noqa: E731
    return [[site(nx - 1 - x, y) for y in range(ny) for x in range(nx)],
            [site(x, ny - 1 - y) for y in range(ny) for x in range(nx)]]


def _problem(case, rng):
    """The cluster of an apply, host, solve or mixed case; interaction, chemical
    potential, t', field and bath are drawn."""
    U = float(rng.uniform(4.0, 10.0))
    if case.get("bath"):
        nb = case["bath"]
        per = nb // 4
        n = 4 + nb
        prob = W.hubbard_cluster(2, 2, tp=float(rng.uniform(0.1, 0.4)) if case["tp"] else None, U=U)
        ops = {}
        for op, (typ, el) in prob.operators.items():  # spin-down orbitals follow the bath
            ops[op] = (typ, [(r + (nb if r >= 4 else 0), c + (nb if c >= 4 else 0), v) for r, c, v in el])
        prob.operators = ops
        prob.n_bath = nb
        for b in range(nb):
            prob.operators[f"eb{b}"] = ("one-body", [(4 + b, 4 + b, 1.0), (4 + b + n, 4 + b + n, 1.0)])
            prob.operators[f"tb{b}"] = ("one-body", [(b // per, 4 + b, 1.0), (b // per + n, 4 + b + n, 1.0)])
            prob.params[f"eb{b}"] = float(rng.uniform(-2, 2))
            prob.params[f"tb{b}"] = float(rng.uniform(0.1, 1))
    else:
        prob = W.hubbard_cluster(case["nx"], case["ny"], tp=float(rng.uniform(0.1, 0.4)) if case["tp"] else None, U=U,
                                 M=float(rng.uniform(0.05, 0.3)) if case.get("neel") else None)
    prob.params["mu"] = U / 2 + float(rng.uniform(-0.5, 0.5))
    up, dn = case["up"], case["dn"]
    prob.sectors = f"R{case.get('irrep', 0)}:N{up + dn}:S{up - dn}"
    if case["kind"] == "mixed" or case.get("sym"):
        prob.generators = _mirrors(case["nx"], case["ny"])
    return prob


def _define(prob, fmt):
    """The model of a problem, its Hamiltonian format settled by a first instance."""
    k = next(_count)
    name = f"perf{k}"
    qed.load_problem(prob, 500000 + k, model_name=name, fmt=fmt)
    qed.erase_model_instance(500000 + k)
    return name


def _instance(held, name, prob):
    label = 600000 + next(_count)
    qed.new_model_instance(name, prob.params, prob.sectors, label)
    held.labels.append(label)
    return label


def _vector(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    return v / v.norm()


def _lehmann(rng, L, M):
    """Poles and residues as a solved insulating cluster has them: a gap around
    zero, complete residues (V V^T = 1)."""
    e = np.concatenate([-np.sort(rng.uniform(0.4, 9.0, M // 2))[::-1], np.sort(rng.uniform(0.4, 9.0, M - M // 2))])
    v = np.linalg.qr(rng.standard_normal((M, L)))[0].T
    return e, np.ascontiguousarray(v)


def _lattice_problem(case, rng):
    """2 x ny clusters tiling the square lattice, with a Weiss field or a bath."""
    ny, nb = case["ny"], case.get("bath", 0)
    n = 2 * ny
    U = float(rng.uniform(4, 10))
    prob = W.square_lattice_vca(2, ny, U=U, M1=float(rng.uniform(0.05, 0.3)) if case["neel"] else 0.0,
                                mu1=U / 2 + float(rng.uniform(-0.3, 0.3)), superlattice=[(2, 0, 0), (ny % 2, ny, 0)])
    if not case["neel"]:
        prob.density_waves = []
        for k in ("M", "M_1"):
            prob.params.pop(k)
    if nb:
        no = n + nb
        prob.n_bath = nb
        for b in range(nb):
            prob.cluster_operators[f"eb{b}"] = ("one-body", [(n + b, n + b, 1.0), (n + b + no, n + b + no, 1.0)])
            prob.cluster_operators[f"tb{b}"] = ("one-body", [(b % n, n + b, 1.0), (b % n + no, n + b + no, 1.0)])
            prob.params[f"eb{b}_1"] = float(rng.uniform(-2, 2))
            prob.params[f"tb{b}_1"] = float(rng.uniform(0.1, 1))
        prob.sectors = f"R0:N{no}:S0"
    poles = [_lehmann(rng, n, case["poles"]) for _ in range(2 if case["neel"] else 1)]
    return prob, poles


def _frequencies(case):
    if case["kind"] == "hybrid":
        return (2 * np.arange(case["nw"]) + 1) * math.pi / BETA
    return W.regular_frequency_grid(2.0, case["nw"] // 2, case["nw"] - case["nw"] // 2)[0]


def _load_poles(label, poles):
    """A solved state of the instance, as reading a checkpoint leaves it."""
    lib, dp = qed.lib(), ctypes.POINTER(ctypes.c_double)
    check = qed._check
    check(lib.qed_instance_load_begin(label, -1.0, 0, 4 if len(poles) == 2 else 0))
    i = ctypes.c_int()
    check(lib.qed_instance_load_state(label, b"R0:N0:S0", -1.0, 1.0, ctypes.byref(i)))
    for sd, (e, v) in enumerate(poles):
        vt = np.ascontiguousarray(v.T)  # column-major L x M
        check(lib.qed_instance_load_qmatrix(label, i.value, sd, v.shape[0], v.shape[1], e.ctypes.data_as(dp),
                                            vt.ctypes.data_as(dp)))
    check(lib.qed_instance_load_end(label))


def _training_set(case, rng):
    x = rng.uniform(-1, 1, (case["points"], 4)).astype(np.float32)
    t = (np.sin(2 * x[:, 0]) + 0.5 * x[:, 1] * x[:, 2] + 0.3 * np.cos(3 * x[:, 3])).astype(np.float32)
    return x, t


def prepare(case, seed):
    s = _Held(case)
    rng = np.random.default_rng([seed, 7])
    kind = case["kind"]
    if kind in ("apply", "host", "mixed"):
        prob = _problem(case, rng)
        name = _define(prob, "E" if kind == "mixed" else "F")
        label = _instance(s, name, prob)
        s.H = (qed.MixedHamiltonian if kind == "mixed" else qed.Hamiltonian)(label, prob.sectors)
        s.x = _vector(s.H.dim, seed)
        if kind == "host":
            s.x = s.x.cpu().pin_memory().numpy()
            s.y = torch.zeros(s.H.dim, dtype=torch.float64).pin_memory().numpy()
        else:
            s.y = torch.zeros_like(s.x)
            s.dots = torch.zeros(3, dtype=torch.float64, device="cuda")
    elif kind == "solve":
        s.jobs = []
        for _ in range(case["n"]):
            prob = _problem(case, rng)
            s.jobs.append((_define(prob, "E" if case["sym"] else "F"), prob))
        s.z = W.matsubara(case["nz"], BETA)
    elif kind == "batch":
        models, s.jobs = {}, []
        for i in range(case["n"]):  # the geometries in turn, so that every seed has the same work
            prob = W.random_batch(1, seed=int(rng.integers(1 << 31)), geoms=[BATCH_SHAPES[i % len(BATCH_SHAPES)]])[0]
            if prob.name not in models:
                models[prob.name] = _define(prob, "F")
            s.jobs.append((models[prob.name], prob))
        s.z = W.matsubara(case["nz"], BETA)
    elif kind in ("omega", "hybrid"):
        prob, poles = _lattice_problem(case, rng)
        k = next(_count)
        model = lattice.LatticeModel(prob, cluster_model=f"perf{k}")
        s.inst = model.instance(600000 + k)
        s.labels.append(s.inst.label)
        _load_poles(s.inst.label, poles)
        s.freqs = _frequencies(case)
    else:
        s.x, s.t = _training_set(case, rng)
        s.net = surrogate.MLP(4, 256, seed=int(rng.integers(1 << 31)))
        s.order = int(rng.integers(1 << 31))
    return s


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "apply":
        stream = torch.cuda.current_stream().cuda_stream
        if case["dots"]:
            s.H.apply_dots_device(s.x.data_ptr(), s.y.data_ptr(), s.dots.data_ptr(), stream)
            return s.y, s.dots
        s.H.apply_device(s.x.data_ptr(), s.y.data_ptr(), stream)
        return s.y
    if kind == "host":
        s.H.mult_add(s.x, s.y)
        return s.y
    if kind == "mixed":
        qed._check(qed.lib().qed_mixed_hamiltonian_apply_device(
            s.H.h, ctypes.c_void_p(s.x.data_ptr()), ctypes.c_void_p(s.y.data_ptr()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return s.y
    if kind in ("solve", "batch"):
        labels = []
        for name, prob in s.jobs:
            label = 600000 + next(_count)
            qed.new_model_instance(name, prob.params, prob.sectors, label)
            labels.append(label)
        if len(labels) > 1:
            qed.Green_function_solve_batch(labels)
        else:
            qed.ground_state_solve(labels[0])
            qed.Green_function_solve(labels[0])
        energy = np.array([qed.ground_state_solve(label)[0] for label in labels])
        G = np.concatenate([qed.Green_function(s.z, label=label).ravel() for label in labels])
        for label in labels:
            qed.erase_model_instance(label)
        return energy, G
    if kind == "omega":
        return s.inst.sef_integrand(s.freqs, (case["side"], case["side"]))
    if kind == "hybrid":
        return lattice.CDMFT_host(s.inst, s.freqs, case["side"])
    return s.net.train(s.x, s.t, case["epochs"], batch=case["batch"], seed=s.order), s.net.get_params()


# --------------------------------------------------------------- their work ----

def _bonds(case):
    """Undirected hops per spin of a cluster or plaquette with bath."""
    if case.get("bath"):
        return 4 + (2 if case["tp"] else 0) + case["bath"]
    nn, nnn = W.lattice_bonds(case["nx"], case["ny"], diagonal=case["tp"])
    return len(nn) + len(nnn)


def _product(case):
    """(states, flops) of one product H x: a multiply and an add per hop and diagonal entry."""
    n = 4 + case["bath"] if case.get("bath") else case["nx"] * case["ny"]
    up, dn = case["up"], case["dn"]
    D = math.comb(n, up) * math.comb(n, dn)
    hops = sum(2 * _bonds(case) * math.comb(n - 2, k - 1) / math.comb(n, k) for k in (up, dn))
    return D, 2.0 * D * (hops + 1)


def work(case):
    kind = case["kind"]
    if kind in ("apply", "host"):
        D, flops = _product(case)
        return {"bytes": 16.0 * D, "flops": flops}
    if kind == "mixed":  # a quarter of the states; the matrix elements follow from the state
        D, flops = _product(case)
        return {"bytes": 4.0 * D, "flops": flops / 4}
    if kind == "solve":
        # about 70 Lanczos steps, twice (energy, vector), and two Krylov bases of about 35 blocks of
        # n_sites vectors: one product and its vectors each
        D, flops = _product(case)
        share = 4 if case["sym"] else 1
        steps = 140 + 70 * case["nx"] * case["ny"]
        return {"bytes": case["n"] * steps * 16.0 * D / share, "flops": case["n"] * steps * flops / share}
    if kind == "batch":  # states of every sector of a mean cluster, about 30 steps each
        mean = sum(4.0 ** n for n in (4, 6, 8, 8, 10)) / 5
        return {"bytes": case["n"] * mean * 30 * 16.0, "flops": case["n"] * mean * 30 * 20.0}
    if kind in ("omega", "hybrid"):
        n, spins = 2 * case["ny"], 2 if case["neel"] else 1
        points = spins * case["nw"] * case["side"] ** 2
        per = 8.0 / 3 * n ** 3 if kind == "omega" else 8.0 * n ** 3  # a complex LU, an inverse
        return {"bytes": spins * (case["nw"] * n * n * 32.0 + case["poles"] * (n + 1) * 8.0),
                "flops": points * per + spins * case["nw"] * case["poles"] * n * n * 4.0}
    weights = 4 * 256 + 2 * 256 * 256 + 256
    steps = case["epochs"] * -(-case["points"] // case["batch"])
    return {"bytes": case["points"] * 20.0 + steps * weights * 24.0, "flops": 6.0 * case["epochs"] * case["points"] * weights}


# ---------------------------------------------------- the values in 64 bits ----

def _strings(n, k):
    s = np.array(sorted(sum(1 << i for i in c) for c in itertools.combinations(range(n), k)), dtype=np.int64)
    return s


def _popcount(v):
    v = np.asarray(v, dtype=np.int64)
    return sum((v >> i) & 1 for i in range(32))


def _hops(strings, n, t):
    """[(targets, sources, signed amplitudes)] of one spin, one entry per directed bond."""
    out = []
    for r in range(n):
        for c in range(n):
            if r == c or t[r, c] == 0.0:
                continue
            src = np.nonzero(((strings >> c) & 1 == 1) & ((strings >> r) & 1 == 0))[0]
            lo, hi = min(r, c), max(r, c)
            between = ((1 << hi) - 1) & ~((2 << lo) - 1)
            sign = 1 - 2 * (_popcount(strings[src] & between) & 1)
            dst = np.searchsorted(strings, strings[src] ^ (1 << c) ^ (1 << r))
            out.append((dst, src, t[r, c] * sign))
    return out


def _one_body(prob):
    """(t_up, t_dn, U per site) of a problem."""
    n = prob.n_orb
    t = np.zeros((2, n, n))
    U = np.zeros(n)
    for op, (typ, el) in prob.operators.items():
        p = prob.params.get(op, 0.0)
        for r, c, v in el:
            if typ == "interaction":
                U[r] += p * v
            else:
                s = r // n
                t[s, r % n, c % n] += p * v
                if r != c:
                    t[s, c % n, r % n] += p * v
    return t[0], t[1], U


def _apply_exact(prob, up, dn, x):
    """H x of a whole (up, dn) sector in torch; x[dn, up]."""
    n, dev = prob.n_orb, x.device
    tu, td, U = _one_body(prob)
    su, sd = _strings(n, up), _strings(n, dn)
    put = lambda a, d=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=d, device=dev)  # noqa: E731
    occ = lambda s: np.stack([(s >> i) & 1 for i in range(n)], 1).astype(np.float64)  # noqa: E731
    ou, od = put(occ(su)), put(occ(sd))
    y = (od * put(U)) @ ou.T
    y += (ou @ put(np.diag(tu)))[None, :] + (od @ put(np.diag(td)))[:, None]
    y *= x
    for dst, src, a in _hops(sd, n, td):
        y.index_add_(0, put(dst, torch.int64), x[put(src, torch.int64)] * put(a)[:, None])
    xt, yt = x.T.contiguous(), torch.zeros_like(x.T)
    for dst, src, a in _hops(su, n, tu):
        yt.index_add_(0, put(dst, torch.int64), xt[put(src, torch.int64)] * put(a)[:, None])
    return y + yt.T


def _mixed_exact(case, prob, seed):
    """H x in the basis of orbit representatives (the smallest state of each orbit,
    in increasing order): x is spread over the orbits, the whole sector's H is
    applied, and the representatives are read back."""
    n, up, dn = case["nx"] * case["ny"], case["up"], case["dn"]
    gens = [np.array(g) - 1 for g in _mirrors(case["nx"], case["ny"])]
    su, sd = _strings(n, up), _strings(n, dn)

    def image(strings, perm):  # (index of the permuted string, fermion sign)
        new = sum(((strings >> i) & 1) << int(perm[i]) for i in range(n))
        swaps = sum(((strings >> i) & 1) * ((strings >> j) & 1) for i in range(n) for j in range(i + 1, n)
                    if perm[i] > perm[j])
        return np.searchsorted(strings, new), 1 - 2 * (np.asarray(swaps) & 1)

    dev, du, D = "cuda", len(su), len(su) * len(sd)
    rep = torch.arange(D, device=dev)
    sign = torch.ones(D, dtype=torch.float64, device=dev)
    null = torch.zeros(D, dtype=torch.bool, device=dev)
    fixed = torch.ones(D, dtype=torch.float64, device=dev)
    me = torch.arange(D, device=dev)
    for a, b in ((1, 0), (0, 1), (1, 1)):
        perm = np.arange(n)
        if a:
            perm = gens[0][perm]
        if b:
            perm = gens[1][perm]
        chi = (-1) ** (a * (case["irrep"] & 1) + b * (case["irrep"] >> 1))
        iu, gu = image(su, perm)
        idn, gd = image(sd, perm)
        to = (torch.as_tensor(idn, device=dev)[:, None] * du + torch.as_tensor(iu, device=dev)[None, :]).reshape(-1)
        ph = chi * (torch.as_tensor(gd, device=dev)[:, None] * torch.as_tensor(gu, device=dev)[None, :]).reshape(-1)
        null |= (to == me) & (ph < 0)
        fixed += (to == me).double()
        less = to < rep
        rep = torch.where(less, to, rep)
        sign = torch.where(less, ph.double(), sign)
    null = null | null[rep]
    basis = torch.nonzero((rep == me) & ~null).reshape(-1)
    length = 4.0 / fixed[basis]
    full = torch.zeros(D, dtype=torch.float64, device=dev)
    full[basis] = _vector(len(basis), seed) / length.sqrt()
    full = torch.where(null, torch.zeros_like(full), full[rep] * sign)
    y = _apply_exact(prob, up, dn, full.reshape(len(sd), du)).reshape(-1)
    return y[basis] * length.sqrt()


def _lattice_exact(case, seed):
    prob, poles = _lattice_problem(case, np.random.default_rng([seed, 7]))
    ny, n = case["ny"], 2 * case["ny"]
    pos = {(x, y): x + 2 * y for y in range(ny) for x in range(2)}
    p = prob.params
    inter = []  # (site, site, R, amplitude) of the hops that leave the cluster
    for (x, y), s in pos.items():
        for dx, dy in ((1, 0), (0, 1), (-1, 0), (0, -1)):
            X, Y = x + dx, y + dy
            R2 = Y // ny
            X, Y = X - R2 * (ny % 2), Y - R2 * ny
            R1 = X // 2
            X -= 2 * R1
            if R1 or R2:
                inter.append((s, pos[X, Y], R1, R2, -p["t"]))
    w, side = _frequencies(case), case["side"]
    off = 0.5 if case["kind"] == "hybrid" else 0.0
    kx, ky = (a.ravel() for a in np.meshgrid((np.arange(side) + off) / side, (np.arange(side) + off) / side,
                                             indexing="ij"))
    Vk = np.zeros((side * side, n, n), dtype=np.complex128)
    for r, c, R1, R2, a in inter:
        Vk[:, r, c] += a * np.exp(2j * np.pi * (kx * R1 + ky * R2))
    z = 1j * w
    out = []
    for sd, (e, v) in enumerate(poles):
        G = np.einsum("am,wm,bm->wab", v, 1.0 / (z[:, None] - e[None, :]), v, optimize=True)
        V0 = np.zeros((len(w), n, n), dtype=np.complex128)
        diag = np.full(n, p["mu_1"] - p["mu"], dtype=np.float64)
        if case["neel"]:
            diag -= p["M_1"] * (1 - 2 * sd) * np.array([(-1.0) ** (x + y) for y in range(ny) for x in range(2)])
        V0 += np.diag(diag)
        gamma = np.zeros_like(V0)
        for b in range(case.get("bath", 0)):
            gamma[:, b % n, b % n] += p[f"tb{b}_1"] ** 2 / (z - p[f"eb{b}_1"])
        V0 -= gamma
        if case["kind"] == "omega":
            out.append(np.array([np.mean(np.linalg.slogdet((V0[i] + Vk) @ G[i] - np.eye(n))[1]) for i in range(len(w))]))
        else:
            P = np.array([np.mean(G[i] @ np.linalg.inv(np.eye(n) - (V0[i] + Vk) @ G[i]), axis=0) for i in range(len(w))])
            out.append(np.linalg.inv(P) - gamma - np.linalg.inv(G))
    if case["kind"] == "hybrid":
        return out
    return out[0] + out[1] if len(out) == 2 else 2.0 * out[0]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("apply", "host", "mixed"):
        rng = np.random.default_rng([seed, 7])
        prob = _problem(case, rng)
        if kind == "mixed":
            return _mixed_exact(case, prob, seed)
        n = prob.n_orb
        du, dd = math.comb(n, case["up"]), math.comb(n, case["dn"])
        x = _vector(du * dd, seed).reshape(dd, du)
        y = _apply_exact(prob, case["up"], case["dn"], x)
        if kind == "host":
            return y.reshape(-1).cpu().numpy()
        if case["dots"]:
            return y.reshape(-1), torch.stack([(x * y).sum(), (y * y).sum(), (x * x).sum()])
        return y.reshape(-1)
    if kind in ("omega", "hybrid"):
        return _lattice_exact(case, seed)
    # whole solves: a sector of 1e4 to 1e6 states, its Krylov bases and poles take minutes in numpy;
    # training: the order of the points is drawn in the library
    return None
