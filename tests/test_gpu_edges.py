"""Edges of the neighbour-list and symmetry-function kernels' loops: cells with
more atoms than a warp has lanes and more candidates than it stages, images of
an atom itself, slab tables that are too long, molecules among cells; more
than eight elements and radial functions; the two launches of a pass, by
neighbour count, for every grid shape in both precisions."""
import itertools

import numpy as np
import pytest

from conftest import ABX3_DIR
from test_gpu_sf_forms import structures, write_potential

pytestmark = pytest.mark.gpu


def crowd(rng, n, size):
    """A molecule of n atoms in a box of that edge, no two within 0.6 Bohr."""
    pos = np.zeros((0, 3))
    while len(pos) < n:
        p = rng.uniform(0, size, 3)
        if len(pos) == 0 or ((pos - p) ** 2).sum(1).min() > 0.36:
            pos = np.vstack([pos, p])
    return {"Z": rng.choice([1, 6, 7, 53, 82], n).astype(np.int32), "pos": pos, "lat": None}


def list_batch(W):
    rng = np.random.default_rng(9)
    s = [W.strain(W.supercell(W.abx3_cell(), n), rng.uniform(-0.05, 0.05, (3, 3)))
         for n in ((1, 1, 1), (2, 1, 1), (3, 2, 1), (4, 4, 2))]
    for x in s:
        x["pos"] = x["pos"] + rng.normal(0, 0.1, x["pos"].shape)
    s.insert(1, crowd(rng, 5, 4.0))
    s.insert(3, crowd(rng, 60, 6.5))    # one cell, two groups of lanes
    s.append(crowd(rng, 200, 7.0))      # one cell of 200: seven groups, two windows of candidates
    s.append(crowd(rng, 150, 13.0))     # eight cells, more than 128 candidates in 32 of them
    # 60 atoms in one corner of a large periodic cell
    c = crowd(rng, 60, 6.5)
    c["lat"] = np.diag([30.0, 24.0, 21.0])
    s.append(c)
    # three atoms in a cell of 5 Bohr: many images, a slab table that is too long
    s.append({"Z": np.array([1, 6, 7], np.int32), "pos": np.array([[0.1, 0.2, 0.3], [2.6, 2.4, 0.2], [0.4, 2.5, 2.7]]),
              "lat": np.array([[5.0, 0.2, 0.0], [0.0, 5.1, 0.3], [0.1, 0.0, 4.9]])})
    return s


def test_list_forms_on_crowded_cells(pkg, W):
    """A thread per atom, a warp per atom and a warp per cell: the same lists
    entry for entry, and the same results bit for bit."""
    from hdnnp_b200 import engine

    pot = engine.Hdnnp.from_runner(ABX3_DIR)
    try:
        structs = list_batch(W)
        n = sum(len(s["Z"]) for s in structs)
        out = {}
        for v in (1, -1, 2):
            pot.set_option("nei_warp", v)
            pot.eval_batch(structs)  # counted lists
            r = pot.eval_batch(structs)  # one-pass lists
            cnt = pot.fetch("nei_count", n, np.int32)
            m = int(cnt.sum())
            out[v] = [cnt] + [pot.fetch(k, m, np.int32) for k in ("nei_index", "nei_shift", "nei_rev")] + \
                [r[k] for k in ("energy", "forces", "dEdLat")]
        assert out[2][0].max() >= 199 and out[2][0].min() >= 4
        for v in (-1, 2):
            assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(out[1], out[v]))
    finally:
        pot.close()


@pytest.mark.parametrize("skin", [0.0, 1.0])
def test_plan_by_cells(pkg, W, skin):
    """A plan large enough for the warp-per-cell search, with crowded cells
    and molecules: against the eager call with a warp per atom, bit for bit
    without a skin, within rounding with one (the lists' order differs)."""
    import torch

    from hdnnp_b200 import engine, plan

    rng = np.random.default_rng(4)
    structs = list_batch(W)
    while sum(len(s["Z"]) for s in structs) < 12400:
        s = W.supercell(W.abx3_cell(), tuple(rng.integers(2, 5, 3)))
        s["pos"] = s["pos"] + rng.normal(0, 0.1, s["pos"].shape)
        structs.append(s)
    pot = engine.Hdnnp.from_runner(ABX3_DIR)
    try:
        pot.set_option("nei_warp", 1)
        pot.eval_batch(structs)
        ref = pot.eval_batch(structs)
        with plan.Plan(pot, structs, skin=skin) as p:
            p.launch()
            p.sync()
            torch.cuda.synchronize()
            E, F = p.E.cpu().numpy(), p.F.cpu().numpy().reshape(-1, 3)
        if skin == 0.0:
            assert np.array_equal(E, ref["energy"]) and np.array_equal(F, ref["forces"].reshape(-1, 3))
        else:
            top = np.abs(ref["forces"]).max()
            assert np.abs(E - ref["energy"]).max() <= 1e-10 * np.abs(ref["energy"]).max()
            assert np.abs(F - ref["forces"].reshape(-1, 3)).max() <= 1e-11 * max(1.0, top)
    finally:
        pot.close()


TEN = {1: "H", 6: "C", 7: "N", 8: "O", 9: "F", 14: "Si", 15: "P", 16: "S", 17: "Cl", 53: "I"}


def ten_element_potential(d, radial):
    """Ten elements, `radial` functions per neighbour element, 2 x 2 x 2 angular ones per pair."""
    rows, n = [], 0
    for c in TEN.values():
        n = 0
        for e in TEN.values():
            for k in range(radial):
                rows.append(f"symfunction_short {c} 2 {e} {0.02 + 0.05 * (k % 4):.4f} {0.7 * k:.4f} 12.0000")
                n += 1
        for a, b in itertools.combinations_with_replacement(TEN.values(), 2):
            for eta, lam, z in itertools.product((0.001, 0.01), (-1.0, 1.0), (1, 4)):
                rows.append(f"symfunction_short {c} 3 {a} {b} {eta:.4f} {lam:.1f} {z:.1f} 12.0000")
                n += 1
    (d / "input.nn").write_text("\n".join([
        "number_of_elements 10", "elements " + " ".join(TEN.values()), "global_hidden_layers_short 2",
        "global_nodes_short 9 7", "global_activation_short t t l", "cutoff_type 2", "scale_symmetry_functions",
        "center_symmetry_functions"] + rows) + "\n")
    rng = np.random.default_rng(radial)
    (d / "scaling.data").write_text("\n".join(
        f"{e + 1} {k + 1} 0.0 {rng.uniform(3, 9):.6f} {rng.uniform(0, 1):.6f}" for e in range(10) for k in range(n))
        + "\n-1.0 1.0\n")
    for z in TEN:
        v = np.concatenate([rng.normal(0, 1 / np.sqrt(i), i * o + o) for i, o in ((n, 9), (9, 7), (7, 1))])
        (d / f"weights.{z:03d}.data").write_text("\n".join(f"{x:.12e}" for x in v) + "\n")


@pytest.mark.parametrize("radial", [8, 9, 17])
def test_ten_elements_many_radial_functions(pkg, orc, tmp_path, radial):
    """Against the FP64 oracle, with the tolerances of the grid shapes' test."""
    from hdnnp_b200 import engine

    ten_element_potential(tmp_path, radial)
    model = orc.Model(str(tmp_path))
    pot = engine.Hdnnp.from_runner(str(tmp_path))
    try:
        rng = np.random.default_rng(radial)
        n = 45
        g = np.array(list(itertools.product(range(4), repeat=3)), float)[:n] * 4.6
        s = {"Z": rng.choice(list(TEN), n).astype(np.int32), "pos": g + rng.normal(0, 0.4, g.shape),
             "lat": np.diag([18.4, 18.4, 18.4]) + rng.uniform(-0.5, 0.5, (3, 3))}
        ref = model.eval(s["Z"], s["pos"], s["lat"])
        top = max(1.0, np.abs(ref["forces"]).max())
        for prec, lim in (("FP64", 1e-9), ("MIXED", 1e-4)):
            pot.set_precision(getattr(engine, "HDNNP_PREC_" + prec))
            out = pot.eval_batch([s])
            assert abs(out["energy"][0] - ref["energy"]) <= 0.1 * lim * max(1.0, abs(ref["energy"]))
            assert np.abs(out["forces"].reshape(-1, 3) - ref["forces"].reshape(-1, 3)).max() <= lim * top
            d = out["dEdLat"].reshape(3, 3, order="F") - ref["dEdLat"]
            assert np.abs(d).max() <= lim * max(1.0, np.abs(ref["dEdLat"]).max())
    finally:
        pot.close()


@pytest.mark.parametrize("prec", ["FP64", "MIXED"])
@pytest.mark.parametrize("etas, zetas", [((0.001, 0.01), (1, 2, 4, 16)), ((0.004,), (1, 4)), ((0.003, 0.3), (1, 3, 5, 6)),
                                         ((0.001, 0.004, 0.02, 0.2), (1, 2, 6, 9)),
                                         ((0.002, 0.009), (1, 2, 3, 4, 5, 8, 12, 16)), ((0.001, 0.01), (1, 2.5, 6.3))])
def test_two_launches_equal_one(pkg, W, tmp_path, etas, zetas, prec):
    """Centres listed for the second launch (all, some, none of the dense
    structure's, whose counts are 96-111) and those of the first: the bits of
    one launch for all."""
    from hdnnp_b200 import engine

    write_potential(tmp_path, etas, zetas)
    pot = engine.Hdnnp.from_runner(str(tmp_path))
    try:
        pot.set_option("small_eval", 0)
        pot.set_precision(getattr(engine, "HDNNP_PREC_" + prec))
        structs = structures(W)
        pot.set_option("sf_split", -1)
        one = pot.eval_batch(structs)
        for split in (8, 48, 104, 112):
            pot.set_option("sf_split", split)
            two = pot.eval_batch(structs)
            for k in ("energy", "forces", "dEdLat"):
                assert np.array_equal(one[k], two[k]), (split, k)
    finally:
        pot.close()
