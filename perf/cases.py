"""Timed cases of the evaluation engine, each one pass through a public entry
point, with the inputs a program holds beforehand and the 64-bit values its
results should have.

The potentials are the repository's: "abx3" (5 elements, 280 symmetry
functions each, the benchmark's), "example" (the 8-atom molecule's) and "prz"
(softplus and ReLU layers, non-integer zeta).  Structures are ABX3 supercells
with the benchmark's strain and jitter, the same with vacancies (odd atom
counts), the example molecule, and clusters cut from the cell.

Results of the mixed-precision form carry 32-bit accuracy and are handed on
as 32-bit values; everything else is 64-bit.
"""
import itertools
import os
import shutil
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import __graft_entry__  # noqa: E402

__graft_entry__.load_package()
from hdnnp_b200 import engine, plan, server, workloads as W  # noqa: E402

GOLDEN = os.path.join(ROOT, "tests", "golden")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference's own caller: one small molecule per host call, once per MD step
        {"name": "call_molecule8", "kind": "call", "pot": "example", "precision": "fp64", "shape": "molecule"},
        # one defective unit-cell multiple per host call (odd atom count), energy, forces and stress
        {"name": "call_cell47", "kind": "call", "pot": "abx3", "precision": "fp64", "shape": "cell",
         "nx": 2, "ny": 2, "nz": 1, "vacancies": 1},
        # the 768-atom cell per host call in mixed precision
        {"name": "call_cell768_mixed", "kind": "call", "pot": "abx3", "precision": "mixed", "shape": "cell",
         "nx": 4, "ny": 4, "nz": 4, "vacancies": 0},
        # a data set of unequal cells and molecules in one host call (rescoring, active learning)
        {"name": "batch96", "kind": "batch", "pot": "abx3", "precision": "fp64", "structs": 96, "molecules": 7},
        # the same for a potential with non-integer zeta and other activations
        {"name": "batch24_prz", "kind": "batch", "pot": "prz", "precision": "fp64", "structs": 24, "molecules": 2},
        # uncertainty of one configuration: mean and spread of three networks on one cell
        {"name": "committee3_cell190", "kind": "committee", "pot": "abx3", "precision": "fp64", "members": 3,
         "nx": 4, "ny": 2, "nz": 2, "vacancies": 2},
        # a short trajectory of the example molecule on the device
        {"name": "md_molecule8", "kind": "md", "pot": "example", "precision": "fp64", "shape": "molecule",
         "steps": 100, "skin": 0.0, "dt": 20.0},
        # one step of a relaxation of the 768-atom cell through a resident plan
        {"name": "plan_cell768", "kind": "plan", "pot": "abx3", "precision": "fp64", "structs": 1,
         "nx": 4, "ny": 4, "nz": 4},
        # ten MD steps of the strained 49,152-atom cell with a Verlet skin
        {"name": "md_cell49152_mixed", "kind": "md", "pot": "abx3", "precision": "mixed", "shape": "cell",
         "nx": 16, "ny": 16, "nz": 16, "steps": 10, "skin": 1.0, "dt": 0.5},
        # one evaluation of every walker of a served ensemble (continuous batching)
        {"name": "serve64_mixed", "kind": "serve", "pot": "abx3", "precision": "mixed", "walkers": 64},
        # the benchmark's batch through a resident plan, in both precisions
        {"name": "plan4096", "kind": "plan", "pot": "abx3", "precision": "fp64", "structs": 4096,
         "nx": 0, "ny": 0, "nz": 0},
        {"name": "plan4096_mixed", "kind": "plan", "pot": "abx3", "precision": "mixed", "structs": 4096,
         "nx": 0, "ny": 0, "nz": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "batch", "batch", "plan", "plan", "plan", "md", "committee", "serve"])
    prec = rng.choice(["fp64", "fp64", "mixed"])
    cell = {"nx": rng.randint(1, 4), "ny": rng.randint(1, 4), "nz": rng.randint(1, 4), "vacancies": rng.randint(0, 3)}
    if kind == "call":
        shape = rng.choice(["molecule", "cluster", "cell", "cell", "cell"])
        if shape == "molecule":
            return {"kind": "call", "pot": "example", "precision": "fp64", "shape": shape}
        if shape == "cluster":
            return {"kind": "call", "pot": "abx3", "precision": "fp64", "shape": shape, "atoms": rng.randint(5, 90)}
        return {"kind": "call", "pot": rng.choice(["abx3", "abx3", "prz"]), "precision": prec, "shape": shape, **cell}
    if kind == "batch":
        n = _log_int(rng, 2, 400)
        return {"kind": "batch", "pot": rng.choice(["abx3", "abx3", "abx3", "prz"]), "precision": prec, "structs": n,
                "molecules": rng.randint(0, max(1, n // 8))}
    if kind == "plan":
        if rng.random() < 0.4:
            n = _log_int(rng, 1, 9)
            return {"kind": "plan", "pot": "abx3", "precision": prec, "structs": 1, "nx": n, "ny": rng.randint(1, 6),
                    "nz": rng.randint(1, 6)}
        return {"kind": "plan", "pot": "abx3", "precision": prec, "structs": _log_int(rng, 2, 3000), "nx": 0, "ny": 0,
                "nz": 0}
    if kind == "md":
        if rng.random() < 0.5:
            return {"kind": "md", "pot": "example", "precision": "fp64", "shape": "molecule",
                    "steps": rng.randint(10, 200), "skin": 0.0, "dt": 20.0}
        return {"kind": "md", "pot": "abx3", "precision": prec, "shape": "cell", "nx": rng.randint(2, 10),
                "ny": rng.randint(2, 10), "nz": rng.randint(2, 10), "steps": rng.randint(2, 10),
                "skin": rng.choice([0.0, 1.0]), "dt": 0.5}
    if kind == "committee":
        return {"kind": "committee", "pot": "abx3", "precision": prec, "members": rng.randint(2, 4), **cell}
    return {"kind": "serve", "pot": "abx3", "precision": prec, "walkers": _log_int(rng, 2, 128)}


# ------------------------------------------------------------------ inputs
def _cell(rng, n, strain=0.05, jitter=0.15, vacancies=0):
    """An n[0] x n[1] x n[2] ABX3 supercell: affine strain, jitter, atoms removed."""
    c = W.abx3_cell()
    g = np.array(list(itertools.product(*[range(k) for k in n])), float)
    pos = (g @ c["lat"].T)[:, None, :] + c["pos"][None]
    T = np.eye(3) + rng.uniform(-strain, strain, (3, 3))
    pos = pos.reshape(-1, 3) @ T.T
    pos = pos + rng.normal(0.0, jitter, pos.shape)
    keep = np.ones(len(pos), bool)
    keep[rng.permutation(len(pos))[:vacancies]] = False
    return {"Z": np.tile(c["Z"], len(g))[keep].astype(np.int32), "pos": pos[keep],
            "lat": T @ (c["lat"] * np.array(n, float)[None, :])}


def _cluster(rng, n):
    """The n atoms of a jittered supercell nearest to its centre, as a molecule."""
    s = _cell(rng, (3, 3, 3), 0.02, 0.1)
    o = np.argsort(((s["pos"] - s["lat"].sum(axis=1) / 2) ** 2).sum(axis=1), kind="stable")[:n]
    return {"Z": s["Z"][o], "pos": s["pos"][o], "lat": None}


def _molecule(rng):
    s = W.read_xyz(os.path.join(GOLDEN, "example", "input.xyz"))
    s["pos"] = s["pos"] + rng.normal(0.0, 0.05, s["pos"].shape)
    return s


def _structures(case, seed):
    """Sizes are the case's; strain, jitter and vacancies are the seed's."""
    rng, sizes = np.random.default_rng([11, int(seed)]), np.random.default_rng(4)
    kind = case["kind"]
    if kind == "batch":
        out = [_cell(rng, tuple(sizes.integers(1, 5, 3)), vacancies=int(sizes.integers(0, 3)))
               for _ in range(case["structs"] - case["molecules"])]
        return out + [_molecule(rng) for _ in range(case["molecules"])]
    if kind == "serve":
        shapes = W.walker_shapes()
        return [_cell(rng, shapes[int(sizes.integers(len(shapes)))], 0.0, 0.1) for _ in range(case["walkers"])]
    if kind == "plan" and not case["nx"]:
        return [_cell(rng, tuple(sizes.integers(1, 5, 3))) for _ in range(case["structs"])]
    if case.get("shape") == "molecule":
        return [_molecule(rng)]
    if case.get("shape") == "cluster":
        return [_cluster(rng, case["atoms"])]
    n = (case["nx"], case["ny"], case["nz"])
    if kind == "md":
        return [_cell(rng, n, 0.03, 0.02)]
    return [_cell(rng, n, vacancies=case.get("vacancies", 0))]


class _State:
    def __init__(self):
        self.close = []

    def __del__(self):
        for c in self.close:
            try:
                c()
            except Exception:
                pass


def _precision(case):
    return engine.HDNNP_PREC_MIXED if case["precision"] == "mixed" else engine.HDNNP_PREC_FP64


def _member_seeds(case, seed):
    return [None] + [1000 * int(seed) + k for k in range(1, case["members"])]


def _write_member(directory, wseed):
    for f in ("input.nn", "scaling.data"):
        shutil.copy(os.path.join(GOLDEN, "abx3", f), directory)
    W.write_abx3_weights(directory, seed=wseed)


def prepare(case, seed):
    s = _State()
    s.case, kind = case, case["kind"]
    structs = _structures(case, seed)
    s.pot = engine.Hdnnp.from_runner(os.path.join(GOLDEN, case["pot"]))
    prec = _precision(case)
    s.pot.set_precision(prec)
    s.single = (lambda a: np.asarray(a, np.float32)) if case["precision"] == "mixed" else (lambda a: a)
    if kind in ("call", "committee"):
        x = structs[0]
        s.ats = engine.AtStruct(x["Z"], x["pos"], x["lat"])
    if kind == "committee":
        s.members = [s.pot]
        for ws in _member_seeds(case, seed)[1:]:
            with tempfile.TemporaryDirectory() as d:
                _write_member(d, ws)
                s.members.append(engine.Hdnnp.from_runner(d))
            s.members[-1].set_precision(prec)
        s.close += [m.close for m in s.members[1:]]
    if kind == "batch":
        off, Z, pos, lat, per = W.concat(structs)
        s.arrays = (off, Z, np.ascontiguousarray(pos), per, np.concatenate([m.ravel(order="F") for m in lat]))
    if kind in ("plan", "md"):
        kw = {}
        if kind == "md":
            m, p = W.maxwell_boltzmann(structs[0]["Z"], 140.0 if case["pot"] == "example" else 300.0, int(seed) + 17)
            kw = {"masses": m, "momenta": p, "dt": case["dt"], "steps_per_launch": case["steps"], "skin": case["skin"]}
        s.stream = torch.cuda.Stream()
        s.plan = plan.Plan(s.pot, structs, precision=prec, **kw)
        s.pos = torch.from_numpy(np.concatenate([x["pos"] for x in structs])).pin_memory()
        if kind == "md":
            s.start = (s.plan.pos.clone(), s.plan.mom.clone(), s.plan.F.clone())
        torch.cuda.synchronize()
        s.close.append(s.plan.close)
    if kind == "serve":
        s.server = server.Server(s.pot, max_batch_atoms=131072, workers=2, precision=prec)
        s.walkers = [s.server.add_walker(x["Z"], x["pos"], x["lat"]) for x in structs]
        s.close.append(s.server.close)
    s.close.append(s.pot.close)
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case, kind, f = s.case, s.case["kind"], s.single
    if kind == "call":
        E, F, L = s.pot.energy_and_forces(s.ats, dEdLat=s.ats.periodic)
        return {"energy": E, "forces": f(F), "dEdLat": None if L is None else f(L)}
    if kind == "committee":
        E, F, L, sd = s.pot.committee_energy_and_forces(s.members, s.ats, dEdLat=True)
        return {"energy": E, "forces": f(F), "dEdLat": f(L), "std": f(np.float64(sd))}
    if kind == "batch":
        o = s.pot.eval_batch_arrays(*s.arrays)
        return {k: f(o[k]) for k in ("energy", "forces", "dEdLat")}
    if kind == "serve":
        tickets = [s.server.submit(w, server.REQ_EVAL) for w in s.walkers]
        r = [s.server.wait(t) for t in tickets]
        return {"energy": f(np.array([x[0] for x in r])), "forces": f(np.concatenate([x[1] for x in r])),
                "dEdLat": f(np.array([x[2] for x in r]))}
    p = s.plan
    with torch.cuda.stream(s.stream):
        if kind == "md":  # a trajectory from the same starting point
            p.pos.copy_(s.start[0])
            p.mom.copy_(s.start[1])
            p.F.copy_(s.start[2])
        else:  # this step's positions from the host
            p.pos.copy_(s.pos, non_blocking=True)
        p.launch(s.stream.cuda_stream)
        p.sync(s.stream.cuda_stream)
        out = {"energy": p.E, "forces": p.F}
        if kind == "md":
            out.update(positions=p.pos, momenta=p.mom)
        else:
            out["dEdLat"] = p.L
        return {k: v.float() for k, v in out.items()} if case["precision"] == "mixed" else out


# ------------------------------------------------------------------ least work
# per atom: neighbour entries, contributing angular pairs, radial and angular terms
_DENSE = {"abx3": (49.9, 543.0, 399.0), "prz": (49.9, 543.0, 279.0), "example": (7.0, 21.0, 28.0)}
_NET = {"abx3": 280 * 25 + 25 * 25 + 25, "prz": 195 * 16 + 16 * 12 + 12, "example": 27 * 10 + 10 * 10 + 10}


def _atoms(case):
    kind = case["kind"]
    if kind == "batch":
        return 185 * (case["structs"] - case["molecules"]) + 8 * case["molecules"]
    if kind == "serve":
        return 900 * case["walkers"]
    if kind == "plan" and not case["nx"]:
        return 187 * case["structs"]
    if case.get("shape") == "molecule":
        return 8
    if case.get("shape") == "cluster":
        return case["atoms"]
    return 12 * case["nx"] * case["ny"] * case["nz"] - case.get("vacancies", 0)


def work(case):
    n, steps = _atoms(case), case.get("steps", 1)
    entries, pairs, g2 = _DENSE[case["pot"]]
    if case.get("shape") == "cluster":
        entries, pairs = min(entries, n - 1.0), min(pairs, n * n / 2.0)
    members = case.get("members", 1)
    # values and gradients: geometry per entry, both passes per pair, radial terms, forward and backward network
    flops = n * steps * (entries * 87 + pairs * 351 + g2 * 19 + members * 4 * _NET[case["pot"]])
    # positions, numbers and (MD) momenta in, forces, energies and (MD) positions and momenta out
    return {"bytes": n * (28 + 24 + (96 if case["kind"] == "md" else 0)), "flops": flops}


# ------------------------------------------------------------------ 64-bit values
def _read_potential(directory):
    """input.nn, scaling.data and weights.NNN.data in plain numpy."""
    sym = {"H": 1, "C": 6, "N": 7, "I": 53, "Pb": 82}
    sfs, acts, nodes, flags, ae = {}, [], [], set(), {}
    for line in open(os.path.join(directory, "input.nn")):
        w = line.split("#")[0].split()
        if not w:
            continue
        if w[0] == "elements":
            els = sorted(sym[x] for x in w[1:])
        elif w[0] == "global_hidden_layers_short":
            hidden = int(w[1])
        elif w[0] == "global_nodes_short":
            nodes = [int(x) for x in w[1:1 + hidden]] + [1]
        elif w[0] == "global_activation_short":
            acts = w[1:2 + hidden]
        elif w[0] in ("scale_symmetry_functions", "center_symmetry_functions"):
            flags.add(w[0][:5])
        elif w[0] == "atom_energy":
            ae[sym[w[1]]] = float(w[2])
        elif w[0] == "symfunction_short" and w[2] == "2":
            eta, rs, rc = (float(x) for x in w[4:7])
            key = "%2d%9.5f%9.5f%9.5f%3d" % (2, rc, eta, rs, sym[w[3]])
            sfs.setdefault(sym[w[1]], []).append((key, (2, sym[w[3]], 0, eta, rs, 0.0, rc)))
        elif w[0] == "symfunction_short":
            eta, lam, zeta, rc = (float(x) for x in w[5:9])
            key = "%2d%9.5f%9.5f%9.5f%9.5f%3d%3d" % (3, rc, eta, zeta, lam + 10.0, sym[w[3]], sym[w[4]])
            sfs.setdefault(sym[w[1]], []).append((key, (3, sym[w[3]], sym[w[4]], eta, lam, zeta, rc)))
    rows = [x.split() for x in open(os.path.join(directory, "scaling.data")) if x.split()]
    pot, at = {}, 0
    for z in els:
        f = [v for _, v in sorted(sfs[z], key=lambda kv: kv[0])]
        s = np.array([[float(x) for x in r[2:5]] for r in rows[at:at + len(f)]])
        at += len(f)
        v = np.array([float(x.split()[0]) for x in open(os.path.join(directory, "weights.%03d.data" % z)) if x.split()])
        net, o, nin = [], 0, len(f)
        for n, a in zip(nodes, acts):
            net.append((v[o:o + nin * n].reshape(nin, n).T.copy(), v[o + nin * n:o + nin * n + n], a))
            o, nin = o + nin * n + n, n
        pot[z] = {"sfs": f, "mean": s[:, 2] if "cente" in flags else 0 * s[:, 2],
                  "width": s[:, 1] - s[:, 0] if "scale" in flags else 0 * s[:, 2] + 1.0, "net": net,
                  "e0": ae.get(z, 0.0), "rc": f[0][6]}
    return pot


def _entries(structs, rc, dev):
    """Neighbour entries (centre, neighbour, relative vector) of all structures by brute force over images."""
    I, J, D, first = [], [], [], 0
    for s in structs:
        n = len(s["Z"])
        pos = torch.tensor(s["pos"], device=dev)
        shifts = np.zeros((1, 3))
        if s["lat"] is not None:
            h = torch.tensor(s["lat"], device=dev)
            f = torch.linalg.solve(h, pos.T).T
            pos = (f - torch.floor(f)) @ h.T
            k = np.ceil(rc * np.linalg.norm(np.linalg.inv(s["lat"]), axis=1)).astype(int) + 1
            shifts = np.array(list(itertools.product(*[range(-m, m + 1) for m in k])), float) @ s["lat"].T
        for sh in shifts:
            t = torch.tensor(sh, device=dev)
            d = pos[:, None, :] - (pos[None, :, :] + t)
            m = (d * d).sum(-1) < rc * rc
            if not sh.any():
                m.fill_diagonal_(False)
            i, j = torch.nonzero(m, as_tuple=True)
            I.append(i + first)
            J.append(j + first)
            D.append(d[i, j])
        first += n
    I, J, D = torch.cat(I), torch.cat(J), torch.cat(D)
    o = torch.argsort(I, stable=True)
    return I[o], J[o], D[o]


def _exact_structs(pots, structs, dev):
    """Per structure the members' energies, mean forces and mean dE/dh (lists over members collapsed)."""
    pot = pots[0]
    rc = max(p["rc"] for p in pot.values())
    Z = torch.tensor(np.concatenate([s["Z"] for s in structs]).astype(np.int64), device=dev)
    N = len(Z)
    I, J, D = _entries(structs, rc, dev)
    cnt = torch.bincount(I, minlength=N)
    start = torch.cumsum(cnt, 0) - cnt
    T = lambda a: torch.tensor(np.asarray(a, float), device=dev)  # noqa: E731
    atomE = torch.zeros(len(pots), N, dtype=torch.float64, device=dev)
    gD = torch.zeros_like(D)
    i0 = 0
    while i0 < N:  # chunks of centres, bounded by their candidate pairs
        c2 = torch.cumsum((cnt[i0:] * (cnt[i0:] - 1)) // 2, 0)
        i1 = i0 + max(1, int((c2 <= 1500000).sum()))
        e0, e1 = int(start[i0]), int(start[i1 - 1] + cnt[i1 - 1])
        d = D[e0:e1].clone().requires_grad_(True)
        ci, zj = I[e0:e1] - i0, Z[J[e0:e1]]
        zc = Z[i0:i1]
        r = torch.sqrt((d * d).sum(-1))
        # ordered candidate pairs a < b of the entries of one centre
        m = cnt[i0:i1][ci]
        pos_in = torch.arange(e1 - e0, device=dev) - (start[i0:i1] - e0)[ci]
        rep = m - 1 - pos_in
        a = torch.repeat_interleave(torch.arange(e1 - e0, device=dev), rep)
        b = a + 1 + torch.arange(len(a), device=dev) - torch.repeat_interleave(torch.cumsum(rep, 0) - rep, rep)
        with torch.no_grad():
            near = ((d[a] - d[b]) ** 2).sum(-1) < rc * rc
        a, b = a[near], b[near]
        total = torch.zeros((), dtype=torch.float64, device=dev)
        for z, p in pot.items():
            mine = zc == z
            if not bool(mine.any()):
                continue
            row = torch.cumsum(mine.long(), 0) - 1
            G = torch.zeros(int(mine.sum()), len(p["sfs"]), dtype=torch.float64, device=dev)
            fcut = lambda x: torch.tanh(torch.clamp(1.0 - x / p["rc"], min=0.0)) ** 3  # noqa: E731
            by = {}
            for k, f in enumerate(p["sfs"]):
                by.setdefault((f[0],) + tuple(sorted(f[1:3])), []).append(k)
            for (typ, z1, z2), ks in by.items():
                f = [p["sfs"][k] for k in ks]
                if typ == 2:
                    sel = torch.nonzero(mine[ci] & (zj == z2)).flatten()
                    x = r[sel]
                    v = torch.exp(-T([q[3] for q in f]) * (x[:, None] - T([q[4] for q in f])) ** 2) * fcut(x)[:, None]
                    at = row[ci[sel]]
                else:
                    sel = torch.nonzero(mine[ci[a]] & (((zj[a] == z1) & (zj[b] == z2)) |
                                                       ((zj[a] == z2) & (zj[b] == z1)))).flatten()
                    pa, pb = a[sel], b[sel]
                    s2 = ((d[pa] - d[pb]) ** 2).sum(-1)
                    ra, rb = r[pa], r[pb]
                    cos = ((d[pa] * d[pb]).sum(-1) / (ra * rb))[:, None]
                    ze = T([q[5] for q in f])
                    v = 2.0 ** (1.0 - ze) * torch.clamp(1.0 + T([q[4] for q in f]) * cos, min=1e-300) ** ze
                    v = v * torch.exp(-T([q[3] for q in f]) * (ra * ra + rb * rb + s2)[:, None])
                    v = v * (fcut(ra) * fcut(rb) * fcut(torch.sqrt(s2)))[:, None]
                    at = row[ci[pa]]
                G[:, torch.tensor(ks, device=dev)] = torch.zeros(len(G), len(ks), dtype=torch.float64,
                                                                 device=dev).index_add(0, at, v)
            x0 = (G - T(p["mean"])) / T(p["width"])
            for q, other in enumerate(pots):
                x = x0
                for w, bias, act in other[z]["net"]:
                    x = x @ T(w).T + T(bias)
                    x = (torch.tanh(x) if act == "t" else torch.nn.functional.softplus(x, threshold=1e9) if act == "p"
                         else torch.relu(x) if act == "r" else x)
                atomE[q, i0:i1][mine] = x[:, 0].detach() + other[z]["e0"]
                total = total + x.sum() / len(pots)
        gD[e0:e1] = torch.autograd.grad(total, d)[0]
        i0 = i1
    F = torch.zeros(N, 3, dtype=torch.float64, device=dev).index_add(0, J, gD).index_add(0, I, -gD)
    off = np.concatenate([[0], np.cumsum([len(s["Z"]) for s in structs])])
    E = [atomE[:, off[k]:off[k + 1]].sum(1).cpu().numpy() for k in range(len(structs))]
    L = []
    for k, s in enumerate(structs):
        sel = (I >= int(off[k])) & (I < int(off[k + 1]))
        if s["lat"] is None:
            L.append(None)
        else:
            frac = D[sel] @ torch.linalg.inv(torch.tensor(s["lat"], device=dev)).T
            L.append((gD[sel].T @ frac).cpu().numpy())
    return E, F.cpu().numpy(), L


def exact(case, seed):
    kind = case["kind"]
    if kind == "md" or _atoms(case) > 20000:
        return None  # a trajectory has no closed value; too long
    structs = _structures(case, seed)
    pots = [_read_potential(os.path.join(GOLDEN, case["pot"]))]
    if kind == "committee":
        for ws in _member_seeds(case, seed)[1:]:
            with tempfile.TemporaryDirectory() as d:
                _write_member(d, ws)
                pots.append(_read_potential(d))
    E, F, L = _exact_structs(pots, structs, torch.device("cuda" if torch.cuda.is_available() else "cpu"))
    if kind == "call":
        return {"energy": float(E[0][0]), "forces": F, "dEdLat": L[0]}
    if kind == "committee":
        return {"energy": float(E[0].mean()), "forces": F, "dEdLat": L[0], "std": E[0].std()}
    energy = np.array([e[0] for e in E])
    if kind == "serve":
        return {"energy": energy, "forces": F, "dEdLat": np.array(L)}
    if kind == "batch":  # flat, column-major; a molecule has none
        return {"energy": energy, "forces": F,
                "dEdLat": np.concatenate([np.zeros(9) if m is None else m.ravel(order="F") for m in L])}
    return {"energy": energy, "forces": F, "dEdLat": np.stack([m.ravel(order="F") for m in L])}
