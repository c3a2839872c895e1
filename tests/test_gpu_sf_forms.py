"""The product-space symmetry-function kernels over the forms their launch
accepts, against the FP64 oracle: grids of one, two and four etas and up to
eight zetas (accumulator tiles, several passes over the partner elements),
exponents inside and beyond the range of the form without range tests, centre
elements without functions for some element pairs; centres without pairs and
with more pairs than the pair list holds (the oracle's batch is small enough
for one launch; test_gpu_edges.py compares the two launches of a pass with
one, bit for bit).  Scaling, collinear atoms, the dense batch's launches, the
second stream.

FP64: |dE| <= 1e-10 |E|, max |dF|, |d dE/dh| <= 1e-9 times the largest force
(at least 1).  Mixed precision: 1e-4 of the largest force, the FP32 rounding
(6e-8) of some 500 pairs' terms through networks with summed weights of ~10."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SYM = {1: "H", 6: "C", 7: "N", 53: "I", 82: "Pb"}


def write_potential(d, etas, zetas, missing=False, radial=(0.002, 0.05, 0.4), rs=(0.0, 1.5, 4.0), seed=5):
    """5 elements, G2 for every neighbour element and G4 on the grid; with
    `missing`, N centres have no functions for pairs with I and Pb centres no
    radial functions for C."""
    rows, n = [], {}
    for c in SYM:
        k = 0
        for e in SYM:
            for eta, r in zip(radial, rs):
                if not (missing and c == 82 and e == 6):
                    rows.append(f"symfunction_short {SYM[c]} 2 {SYM[e]} {eta:.6f} {r:.4f} 12.0000")
                    k += 1
        for a, b in itertools.combinations_with_replacement(SYM, 2):
            if missing and c == 7 and 53 in (a, b):
                continue
            for eta in etas:
                for lam in (-1.0, 1.0):
                    for z in zetas:
                        rows.append(f"symfunction_short {SYM[c]} 3 {SYM[a]} {SYM[b]} {eta:.6f} {lam:.1f} {z:.1f} 12.0000")
                        k += 1
        n[c] = k
    (d / "input.nn").write_text("\n".join([
        "number_of_elements 5", "elements " + " ".join(SYM.values()), "global_hidden_layers_short 2",
        "global_nodes_short 9 7", "global_activation_short t t l", "cutoff_type 2", "scale_symmetry_functions",
        "center_symmetry_functions"] + rows) + "\n")
    rng = np.random.default_rng(seed)
    sc = [f"{ie + 1} {k + 1} 0.0 {rng.uniform(3, 9):.6f} {rng.uniform(0, 1):.6f}" for ie, z in enumerate(SYM)
          for k in range(n[z])]
    (d / "scaling.data").write_text("\n".join(sc) + "\n-1.0 1.0\n")
    for z in SYM:
        v = []
        for i, o in ((n[z], 9), (9, 7), (7, 1)):
            v += list(rng.normal(0, 1 / np.sqrt(i), i * o + o))
        (d / f"weights.{z:03d}.data").write_text("\n".join(f"{x:.12e}" for x in v) + "\n")


def structures(W):
    rng = np.random.default_rng(3)
    dense = W.strain(W.supercell(W.abx3_cell(), (2, 2, 2)), -0.2 * np.eye(3))  # ~100 neighbours, ~2,000 pairs
    out = [W.strain(W.supercell(W.abx3_cell(), (2, 1, 1)), rng.uniform(-0.05, 0.05, (3, 3))), dense]
    for s in out:
        s["pos"] = s["pos"] + rng.normal(0, 0.1, s["pos"].shape)
    # centres with no pair, one neighbour, three neighbours
    out.append({"Z": np.array([7, 53, 6, 1], np.int32), "lat": None,
                "pos": np.array([[0.0, 0, 0], [4, 1, 0.5], [1, 11.2, 2], [7, 3, 13.5]])})
    out.append({"Z": np.array([82, 1, 53, 1, 7], np.int32), "lat": None,
                "pos": np.array([[0.0, 0, 0], [3, 1, 0.2], [1, 3, 2.5], [-2, 2, 4], [2.5, -2, -3]])})
    return out


@pytest.mark.parametrize("etas, zetas, missing", [
    ((0.001, 0.01), (1, 2, 4, 16), False),
    ((0.001, 0.01), (1, 2, 4, 16), True),
    ((0.004,), (1, 4), True),
    ((0.003, 0.3), (1, 3, 5, 6), False),
    ((0.001, 0.004, 0.02, 0.2), (1, 2, 6, 9), True),
    ((0.002, 0.009), (1, 2, 3, 4, 5, 8, 12, 16), True),
])
def test_forms_against_oracle(pkg, orc, W, tmp_path, etas, zetas, missing):
    from hdnnp_b200 import engine

    write_potential(tmp_path, etas, zetas, missing)
    model = orc.Model(str(tmp_path))
    pot = engine.Hdnnp.from_runner(str(tmp_path))
    try:
        pot.set_option("small_eval", 0)
        structs = structures(W)
        for prec, lim in ((engine.HDNNP_PREC_FP64, 1e-9), (engine.HDNNP_PREC_MIXED, 1e-4)):
            pot.set_precision(prec)
            out = pot.eval_batch(structs)
            at = 0
            for k, s in enumerate(structs):
                ref = model.eval(s["Z"], s["pos"], s["lat"])
                n = len(s["Z"])
                top = max(1.0, np.abs(ref["forces"]).max())
                assert abs(out["energy"][k] - ref["energy"]) <= (1e-10 if lim == 1e-9 else 1e-5) * max(1.0, abs(ref["energy"]))
                assert np.abs(out["forces"][at:at + n] - ref["forces"]).max() <= lim * top
                if s["lat"] is not None:
                    d = out["dEdLat"][9 * k:9 * k + 9].reshape(3, 3, order="F") - ref["dEdLat"]
                    assert np.abs(d).max() <= lim * max(1.0, np.abs(ref["dEdLat"]).max())
                at += n
    finally:
        pot.close()


def test_forms_need_no_list(pkg, W, tmp_path):
    """A structure evaluated in one launch, and split into launches by
    neighbour count, bit for bit."""
    from hdnnp_b200 import engine

    write_potential(tmp_path, (0.001, 0.01), (1, 2, 4, 16))
    pot = engine.Hdnnp.from_runner(str(tmp_path))
    try:
        s = structures(W)[1]
        res = []
        for split in (-1, 32, 64, 97):
            pot.set_option("sf_split", split)
            res.append(pot.energy_and_forces(engine.AtStruct(s["Z"], s["pos"], s["lat"]), dEdLat=True))
        for r in res[1:]:
            assert r[0] == res[0][0] and np.array_equal(r[1], res[0][1]) and np.array_equal(r[2], res[0][2])
    finally:
        pot.close()


def test_value_at_its_mean_scales_to_zero(pkg, tmp_path):
    """(value - mean) / (max - min) with the mean set to the value: the
    difference is formed first, so the scaled function is exactly zero."""
    from hdnnp_b200 import engine

    Z = np.array([1, 6, 7, 53, 82], np.int32)  # an atom of every element
    pos = np.array([[0.0, 0, 0], [3, 1, 0.2], [1, 3, 2.5], [-2, 2, 4], [2.5, -2, -3]])
    scaling = tmp_path / "scaling.data"
    write_potential(tmp_path, (0.001, 0.01), (1, 2, 4, 16))

    def values():
        pot = engine.Hdnnp.from_runner(str(tmp_path))
        try:
            pot.set_option("small_eval", 0)
            pot.energy_and_forces(engine.AtStruct(Z, pos, None))
            nsf = max(pot.nsf.values())
            return pot.fetch("G", len(Z) * nsf).reshape(len(Z), nsf), [pot.nsf[int(z)] for z in Z]
        finally:
            pot.close()

    n = [sum(1 for x in scaling.read_text().splitlines() if x.split()[0] == str(k + 1) and len(x.split()) == 5)
         for k in range(5)]
    rows = [(e + 1, k + 1) for e in range(5) for k in range(n[e])]
    scaling.write_text("\n".join(f"{e} {k} 0.0 1.0 0.0" for e, k in rows) + "\n-1.0 1.0\n")
    raw, nsf = values()
    assert nsf == n and np.count_nonzero(raw[:, : min(n)]) > 500
    w = np.random.default_rng(2).uniform(0.1, 3.0, len(rows))
    scaling.write_text("\n".join(f"{e} {k} 0.0 {x:.17g} {raw[e - 1, k - 1]:.17g}" for (e, k), x in zip(rows, w))
                       + "\n-1.0 1.0\n")
    scaled, _ = values()
    for a in range(5):
        assert np.count_nonzero(scaled[a, : n[a]]) == 0


@pytest.mark.parametrize("small, generic, prec", [(1, 0, "FP64"), (0, 0, "FP64"), (0, 1, "FP64"), (0, 0, "MIXED")])
def test_collinear_atoms_with_noninteger_zeta(pkg, tmp_path, small, generic, prec):
    """1 + lambda cos of three atoms in a line is zero up to the sign of its
    rounding: finite results, equal to those of a bend of 1e-4 Bohr (the
    energy changes by about its square, the forces by its curvature)."""
    from hdnnp_b200 import engine

    write_potential(tmp_path, (0.001, 0.01), (1, 2.5, 6.3))
    pot = engine.Hdnnp.from_runner(str(tmp_path))
    try:
        pot.set_option("small_eval", small)
        pot.set_option("generic_sf", generic)
        pot.set_precision(getattr(engine, "HDNNP_PREC_" + prec))
        rng = np.random.default_rng(0)
        zs = sorted(int(z) for z in pot.nsf)
        for k in range(60):
            v = np.array([1.0, 0, 0]) if k % 4 < 2 else rng.normal(size=3)
            v /= np.linalg.norm(v)
            w = np.cross(v, rng.normal(size=3))
            w /= np.linalg.norm(w)
            d1, d2 = rng.uniform(1.5, 4.0, 2)
            pos = np.array([-d1 * v, 0 * v, (d1 if k % 2 else d2) * v])
            Z = rng.choice(zs, 3).astype(np.int32)
            E, F, _ = pot.energy_and_forces(engine.AtStruct(Z, pos))
            assert np.isfinite(E) and np.isfinite(F).all(), k
            pos[1] += 1e-4 * w
            E1, F1, _ = pot.energy_and_forces(engine.AtStruct(Z, pos))
            assert abs(E - E1) <= (1e-6 if prec == "FP64" else 1e-4), k
            assert np.abs(F - F1).max() <= 1e-3 * max(1.0, np.abs(F).max()), k
    finally:
        pot.close()


def test_dense_batch_fills_the_gpu(pkg, W, tmp_path):
    """19,200 atoms of which nearly all have more neighbours than the first
    launch takes: the two launches of the default are as fast as one launch
    for all (within 20 %, best of 10 each)."""
    from hdnnp_b200 import engine

    write_potential(tmp_path, (0.001, 0.01), (1, 2, 4, 16))
    pot = engine.Hdnnp.from_runner(str(tmp_path))
    try:
        rng = np.random.default_rng(1)
        structs = []
        for _ in range(200):
            s = W.strain(W.supercell(W.abx3_cell(), (2, 2, 2)), -0.2 * np.eye(3))
            s["pos"] = s["pos"] + rng.normal(0, 0.1, s["pos"].shape)
            structs.append(s)
        for prec in (engine.HDNNP_PREC_FP64, engine.HDNNP_PREC_MIXED):
            pot.set_precision(prec)
            best = {}
            pot.set_profiling(False)
            pot.eval_batch(structs)
            pot.set_profiling(True)
            for split in (0, -1):
                pot.set_option("sf_split", split)
                pot.eval_batch(structs)
                for _ in range(10):
                    pot.eval_batch(structs[:1])  # the profile of a call is collected by the next one
                    pot.profile(reset=True)
                    pot.eval_batch(structs)
                    pot.eval_batch(structs[:1])
                    ms = pot.profile()[0]
                    best[split] = min(best.get(split, 1e9), ms["sf_values"] + ms["sf_gradients"])
            assert best[0] <= 1.2 * best[-1], best
    finally:
        pot.close()


@pytest.mark.parametrize("prec", ["FP64", "MIXED"])
def test_second_stream_only_where_it_is_used(pkg, W, prec):
    """A context makes its second stream when a batch first runs in two
    launches: not for one cell (all its warps fit on the GPU), and not for a
    batch when the option asks for one launch; the results are the same."""
    from conftest import ABX3_DIR

    from hdnnp_b200 import engine

    pot = engine.Hdnnp.from_runner(ABX3_DIR)
    try:
        pot.set_precision(getattr(engine, "HDNNP_PREC_" + prec))
        batch = W.config_c4(n_struct=96)

        def made():
            return int(pot.fetch("side_stream", 1, np.int32)[0])

        pot.eval_batch(batch[:1])
        assert made() == 0
        pot.set_option("sf_split", -1)
        one = pot.eval_batch(batch)
        assert made() == 0
        pot.set_option("sf_split", 0)
        two = pot.eval_batch(batch)
        assert made() == 1
        for k in ("energy", "forces", "dEdLat"):
            assert np.array_equal(one[k], two[k])
    finally:
        pot.close()
