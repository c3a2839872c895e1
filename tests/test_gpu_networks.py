"""FP64 network kernels (forward, dE/dG) against the layers in numpy, on the
symmetry functions the device computed: tiles of 8 atoms that are partly
filled (one atom, one tile less / plus one atom, elements with fewer atoms
than a tile), and batches on either side of the line between the per-tile and
the weights-resident kernel, with rows of even (abx3, 280) and odd (prz, 195)
length.

Tolerance: eps times the terms of the longest sum times the largest sum of
absolute products, carried through the later layers by their largest absolute
row / column sums (activations are 1-Lipschitz)."""
import numpy as np
import pytest

from conftest import ABX3_DIR, EXAMPLE_DIR, PRZ_DIR

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def layers(net, x):
    """Energies, dE/dG and their rounding bounds for the rows of x."""
    ys, ds, grow = [x], [], 1.0
    scale = 1.0
    for w, b, a in net:
        c = ys[-1] @ w.T + b
        scale = max(scale, (np.abs(ys[-1]) @ np.abs(w).T + np.abs(b)).max())
        y = np.tanh(c) if a == "t" else np.logaddexp(0.0, c) if a == "p" else np.maximum(c, 0.0) if a == "r" else c
        d = 1 - y * y if a == "t" else 1 / (1 + np.exp(-c)) if a == "p" else (c > 0) * 1.0 if a == "r" else 1 + 0 * c
        ys.append(y)
        ds.append(d)
        grow *= max(1.0, np.abs(w).sum(1).max(), np.abs(w).sum(0).max()) if len(ys) > 2 else 1.0
    g = ds[-1]
    for k in range(len(net) - 1, 0, -1):
        g = (g @ net[k][0]) * ds[k - 1]
    tol = 4 * EPS * x.shape[1] * scale * grow
    return ys[-1][:, 0], g @ net[0][0], tol, tol * max(1.0, np.abs(net[0][0]).max()) * grow


@pytest.mark.parametrize("pot_dir, natoms", [(EXAMPLE_DIR, 8), (EXAMPLE_DIR, 1), (ABX3_DIR, 7), (ABX3_DIR, 9),
                                             (ABX3_DIR, 97), (PRZ_DIR, 65), (ABX3_DIR, 18936), (ABX3_DIR, 18945),
                                             (PRZ_DIR, 18951)])
def test_networks(pkg, W, pot_dir, natoms):
    from hdnnp_b200 import engine

    pot = engine.Hdnnp.from_runner(pot_dir)
    try:
        pot.set_option("small_eval", 0)
        rng = np.random.default_rng(natoms)
        if pot_dir == EXAMPLE_DIR:
            s = W.read_xyz(EXAMPLE_DIR + "/input.xyz")
        else:
            s = W.supercell(W.abx3_cell(), (12, 12, 11) if natoms > 1000 else (3, 3, 1))
            s["pos"] = s["pos"] + rng.normal(0, 0.1, s["pos"].shape)
        Z, pos = s["Z"][:natoms], s["pos"][:natoms]
        pot.energy_and_forces(engine.AtStruct(Z, pos, s["lat"]))
        nsf = max(pot.nsf.values())
        G = pot.fetch("G", natoms * nsf).reshape(natoms, nsf)
        D = pot.fetch("dEdG", natoms * nsf).reshape(natoms, nsf)
        E = pot.fetch("atom_energy", natoms)
        e0 = pot.flags()["atomenergies"]
        for z in np.unique(Z):
            m, n = Z == z, pot.nsf[int(z)]
            e, g, te, tg = layers(pot.network(int(z)), G[m][:, :n])
            e = e + e0[int(z) - 1]
            assert np.abs(E[m] - e).max() <= te + 4 * EPS * np.abs(e).max()
            assert np.abs(D[m][:, :n] - g).max() <= tg
    finally:
        pot.close()


@pytest.mark.parametrize("pot_dir", [ABX3_DIR, PRZ_DIR])
def test_alone_equals_in_the_large_batch(pkg, W, pot_dir):
    """The per-tile and the weights-resident kernel give an atom the same bits."""
    from hdnnp_b200 import engine

    pot = engine.Hdnnp.from_runner(pot_dir)
    try:
        rng = np.random.default_rng(8)
        small = W.strain(W.supercell(W.abx3_cell(), (2, 2, 1)), rng.uniform(-0.05, 0.05, (3, 3)))
        small["pos"] = small["pos"] + rng.normal(0, 0.15, small["pos"].shape)
        big = W.supercell(W.abx3_cell(), (12, 12, 11))
        big["pos"] = big["pos"] + rng.normal(0, 0.1, big["pos"].shape)
        alone = pot.eval_batch([small])
        both = pot.eval_batch([big, small])
        n = len(small["Z"])
        assert both["energy"][1] == alone["energy"][0]
        assert np.array_equal(both["forces"][-n:], alone["forces"])
        assert np.array_equal(both["dEdLat"][9:], alone["dEdLat"])
    finally:
        pot.close()


def deep_potential(W, directory, hidden):
    import os
    import shutil

    from hdnnp_b200 import engine

    W.write_abx3_input(str(directory), hidden=hidden)
    W.write_abx3_weights(str(directory), hidden=hidden, seed=len(hidden))
    shutil.copy(os.path.join(ABX3_DIR, "scaling.data"), str(directory))
    return engine.Hdnnp.from_runner(str(directory))


@pytest.mark.parametrize("hidden", [(30, 30), (25, 25, 25), (32, 32, 32), (25, 25, 25, 25), (30, 30, 30, 30), (7, 32, 17),
                                    (32,) * 7])
def test_networks_of_other_shapes(pkg, W, tmp_path, hidden):
    """Networks with more weights than leave room for ten warps of the
    resident kernel (eight to six, or the per-tile kernel), widths that are no
    multiple of a tile: against numpy, and an atom's bits in a small batch."""
    pot = deep_potential(W, tmp_path, hidden)
    try:
        rng = np.random.default_rng(len(hidden))
        big = W.supercell(W.abx3_cell(), (12, 12, 11))
        big["pos"] = big["pos"] + rng.normal(0, 0.1, big["pos"].shape)
        small = W.supercell(W.abx3_cell(), (2, 1, 1))
        small["pos"] = small["pos"] + rng.normal(0, 0.1, small["pos"].shape)
        alone = pot.eval_batch([small])
        both = pot.eval_batch([big, small])
        n = len(small["Z"])
        assert both["energy"][1] == alone["energy"][0] and np.array_equal(both["forces"][-n:], alone["forces"])
        Z = np.concatenate([big["Z"], small["Z"]])
        nsf = max(pot.nsf.values())
        G = pot.fetch("G", len(Z) * nsf).reshape(len(Z), nsf)
        D = pot.fetch("dEdG", len(Z) * nsf).reshape(len(Z), nsf)
        E = pot.fetch("atom_energy", len(Z))
        e0 = pot.flags()["atomenergies"]
        for z in np.unique(Z):
            m, k = Z == z, pot.nsf[int(z)]
            e, g, te, tg = layers(pot.network(int(z)), G[m][:, :k])
            e = e + e0[int(z) - 1]
            assert np.abs(E[m] - e).max() <= te + 4 * EPS * np.abs(e).max()
            assert np.abs(D[m][:, :k] - g).max() <= tg
    finally:
        pot.close()


def test_time_of_a_third_hidden_layer(pkg, W, tmp_path):
    """40,272 atoms: a third hidden layer of 25 is under a tenth of the
    multiplications; it costs at most 35 % of the network stage (best of 10)."""
    ms = {}
    structs = W.config_c4(n_struct=200)
    for hidden in ((25, 25), (25, 25, 25)):
        d = tmp_path / str(len(hidden))
        d.mkdir()
        pot = deep_potential(W, d, hidden)
        try:
            pot.eval_batch(structs)
            pot.set_profiling(True)
            for _ in range(10):
                pot.eval_batch(structs[:1])  # the profile of a call is collected by the next one
                pot.profile(reset=True)
                pot.eval_batch(structs)
                pot.eval_batch(structs[:1])
                t = pot.profile()[0]["mlp"]
                ms[hidden] = min(ms.get(hidden, 1e9), t)
        finally:
            pot.close()
    assert ms[(25, 25, 25)] <= 1.35 * ms[(25, 25)], ms
