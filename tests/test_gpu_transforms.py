"""Transform passes of two register stages and the int32 deposits, at the sizes where they can
go wrong, against the FP64 oracle.

Tolerances: forces max_p |df_p| / max(|f_p|, f_rms) <= 1e-5 and pair energies 1e-5 relative
(FP32 deposit, transforms of at most 256 points per axis and gather: a few hundred roundings of
6e-8, added in quadrature); deterministic deposits are exact integer sums, so results that
differ only in how a tile is summed are equal bit for bit.
"""
import numpy as np
import pytest

import oracle
import tild_b200
from conftest import force_error, spec_to_system
from tild_b200 import synth

pytestmark = pytest.mark.gpu


def make_box(spec, **opts):
    o = {"write_files": 0}
    o.update(opts)
    b = tild_b200.box_from_spec(spec, options=o)
    b.command("endBox")
    return b


def species_system(nsp, grid, seed=5):
    """Short chains of nsp species with every pair interacting: nsp density fields and force groups."""
    rng = np.random.default_rng(seed)
    L = np.array([0.45 * g for g in grid])
    x = synth.random_walk_chains(rng, 60, 6, L, 0.6)
    types = rng.integers(0, nsp, size=len(x)).astype(np.int32)
    names = ["A", "B", "C", "D"][:nsp]
    pots = [dict(kind="gaussian", I=a, J=b, A=1.0 + 0.3 * i + 0.2 * j, sigma=0.7)
            for i, a in enumerate(names) for j, b in enumerate(names) if i <= j]
    return synth.SystemSpec("species", L, grid, x, types, names, synth.chain_bonds(60, 6), np.repeat(np.arange(60), 6),
                            potentials=pots, order=3, seed=seed)


# one-stage lines (5, 7, 11, 13), uneven factors, the longest lines (256, 240, 225, 208), and axes
# that keep the mixed-radix path (17, 34, 250) beside ones that do not
@pytest.mark.parametrize("grid", [(6, 8, 9), (5, 7, 11), (13, 10, 12), (14, 15, 16), (22, 26, 33), (49, 18, 20), (64, 9, 8),
                                  (256, 8, 6), (8, 240, 6), (6, 8, 225), (208, 7, 6), (17, 16, 12), (16, 34, 12), (12, 8, 250)])
@pytest.mark.parametrize("nsp", [1, 2, 3, 4])
def test_transforms_match_oracle(grid, nsp):
    if nsp > 2 and max(grid) > 100:
        pytest.skip("field counts are covered on the smaller grids")
    spec = species_system(nsp, grid)
    sysm = spec_to_system(spec)
    fref, inter = oracle.forces(sysm, prec=64)
    eref = np.array(oracle.pair_energies(sysm, inter["dens"]))
    with make_box(spec) as b:
        assert force_error(b.forces(), fref) <= 1e-5
        e = np.array(b.thermo()["potentials"])
        assert np.all(np.abs(e - eref) <= 1e-5 * np.abs(eref).max())
        k, s, n = b.structure_factor("A", 8, 5.0)
        kr, sr, nr = oracle.structure_factor(sysm, inter["dens"]["A"][0], 8, 5.0)
        assert np.array_equal(n, nr) and np.allclose(s, sr, rtol=1e-4, atol=1e-9)


# every radix of either stage along every axis: k x k points for k = 3 .. 16, 3 x 2, 5 x 1, and
# 2 x 2 (of the order-2 box)
EDGES = [4, 5, 6, 9, 16, 25, 36, 49, 64, 81, 100, 121, 144, 169, 196, 225, 256]


def two_stage_factors(n):
    r1 = next(r for r in range(1, 17) if r * r >= n and n % r == 0)
    return r1, n // r1


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("nsp", [1, 2, 3, 4])
def test_every_radix_of_both_stages_matches_oracle(axis, nsp):
    factors = [two_stage_factors(n) for n in EDGES]
    assert {a for a, _ in factors} == set(range(2, 17)) and {b for _, b in factors} == set(range(1, 17))
    for n in EDGES:
        grid = [6, 8]
        grid.insert(axis, n)
        spec = species_system(nsp, tuple(grid), seed=n)
        spec.order = 2 if n == 4 else 3
        sysm = spec_to_system(spec)
        fref, inter = oracle.forces(sysm, prec=64)
        eref = np.array(oracle.pair_energies(sysm, inter["dens"]))
        with make_box(spec) as b:
            assert force_error(b.forces(), fref) <= 1e-5, n
            assert np.all(np.abs(np.array(b.thermo()["potentials"]) - eref) <= 1e-5 * np.abs(eref).max()), n


@pytest.mark.parametrize("charge", [1.0, 0.5, 2.5])
@pytest.mark.parametrize("deterministic", [0, 1])
def test_deposit_coefficients_match_oracle(charge, deterministic):
    # charges of +-1 (one conversion for both fields), other magnitudes (one each), and zero
    spec = synth.small_system(seed=31, charges=True, n_free=200)
    spec.charges = (spec.charges * np.float32(charge)).astype(np.float32)
    spec.potentials = [dict(kind="gaussian", I="all", J="all", A=1.5, sigma=0.7), dict(kind="charges", lB=1.0, sigma=0.5)]
    fref, _ = oracle.forces(spec_to_system(spec), prec=64)
    with make_box(spec, deterministic=deterministic) as b:
        assert force_error(b.forces(), fref) <= 1e-5


@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_deterministic_sums_do_not_depend_on_the_tile(order):
    # 80,000 particles on 16^3: tiles of 8 bricks hold 10,000 (two int32 words per point), of
    # 32 bricks 40,000 (past the bound of the words: 64-bit box), of 64 do not fit (global)
    rng = np.random.default_rng(order)
    n, L = 80000, 7.0
    x = rng.uniform(0.0, L, size=(n, 3))
    types = rng.integers(0, 2, size=n)
    pots = [dict(kind="gaussian", I="A", J="A", A=0.01, sigma=0.7), dict(kind="gaussian", I="A", J="B", A=0.02, sigma=0.7)]
    spec = synth.SystemSpec("dense", [L] * 3, [16] * 3, x, types, ["A", "B"], [], np.arange(n), potentials=pots, order=order)
    out = []
    for codes in (8, 32, 64):
        with make_box(spec, deterministic=1, deposit_codes=codes) as b:
            out.append(b.forces())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    # against the oracle for the continuous splines only: the order-4 weights (s^4 for s^3) jump
    # at cell edges by up to 1e-2, and of 240,000 uniform coordinates some lie within FP32
    # rounding (about 1e-6 of a cell) of an edge and fall in the other cell there
    if order < 4:
        fref, _ = oracle.forces(spec_to_system(spec), prec=64)
        assert force_error(out[0], fref) <= 1e-5


def test_structure_factor_of_long_x_and_z_lines():
    # x and z far past the two-stage lengths beside a y axis of 4 = 2 x 2: nz hp^2 >= 2^32, past
    # the two-stage y pass's column division.  Spacings of 20 in y and z put the columns of the
    # x Nyquist index, the last of a row, in shells of their own.
    grid, L = [3910, 4, 1200], [0.4 * 3910, 20.0 * 4, 20.0 * 1200]
    rng = np.random.default_rng(3)
    n = 3000
    x = rng.uniform(0.0, 1.0, size=(n, 3)) * L
    spec = synth.SystemSpec("rod", L, grid, x, np.zeros(n, np.int32), ["A"], [], np.arange(n),
                            potentials=[dict(kind="gaussian", I="A", J="A", A=0.1, sigma=0.7)], order=1)
    with make_box(spec, sort_interval=0) as b:
        rho = b.density("A")
        k, s, c = b.structure_factor("A", 1963, 7.87)
    kr, sr, cr = oracle.structure_factor(spec_to_system(spec), rho, 1963, 7.87)
    assert np.array_equal(c, cr) and np.allclose(k, kr, rtol=1e-9) and np.allclose(s, sr, rtol=1e-4, atol=0.0)


def default_deposit_box(x, q, pots, order, **opts):
    """A box of 88^3 points whose default deposit tiles are 16 bricks of 4^3 cells."""
    n = len(x)
    spec = synth.SystemSpec("tiles", [88.0] * 3, [88] * 3, x, np.zeros(n, np.int32), ["A"], [], np.arange(n), charges=q,
                            potentials=pots, order=order)
    b = make_box(spec, tile_codes=8, **opts)
    t = b.describe()["tiles"]
    assert (t["deposit_codes"], t["deposit_threads"]) == (16, 128)
    return spec, b


def test_dense_default_deposit_tiles_keep_the_finest_scale():
    # Order 1: int32 sums at 2^24 per unit weight take 115 particles of charge 1.  Charges +1 at
    # s = 1/256 and 5/256 of a cell and -1 twice at 3/256, alike in y and z: every weight is a
    # multiple of 2^-24 and the four cancel point by point, in sums at 2^24 exactly, while at
    # 2^23 the odd multiples round.  100 of them in each half of one 16-brick tile.
    rng = np.random.default_rng(9)
    x, q = [], []
    for half in (0, 8):
        for _ in range(25):
            c = rng.integers(1, 7, size=3) + [half, 0, 0]
            yz = (2 * rng.integers(-60, 60, size=2) + 1) / 256.0
            for s, v in ((1, 1.0), (5, 1.0), (3, -1.0), (3, -1.0)):
                x.append(c + 0.5 + np.array([s / 256.0, yz[0], yz[1]]))
                q.append(v)
    spec, b = default_deposit_box(np.array(x), np.array(q, np.float32), [dict(kind="charges", lB=1.0, sigma=0.5)], 1)
    with b:
        assert np.array_equal(b.forces(), np.zeros_like(spec.x))


@pytest.mark.parametrize("counts", [(100, 100), (300, 40), (0, 900), (1500, 1200)])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_dense_default_deposit_tiles_match_oracle(order, counts):
    # the halves of one tile at each fixed-point scale, empty, and past all scales (FP32)
    rng = np.random.default_rng(sum(counts) + order)
    x = np.concatenate([rng.uniform(0.0, 8.0, size=(n, 3)) + [8.0 * h, 0.0, 0.0] for h, n in enumerate(counts)] +
                       [rng.uniform(0.0, 88.0, size=(500, 3))])
    if order == 4:   # away from cell edges, where the order-4 weights jump (see above)
        x = np.floor(x) + 0.05 + 0.9 * (x - np.floor(x))
        x = np.where(np.abs(x - np.floor(x) - 0.5) < 0.02, x + 0.04, x)
    spec, b = default_deposit_box(x, None, [dict(kind="gaussian", I="A", J="A", A=0.5, sigma=0.7)], order)
    with b:
        f = b.forces()
    fref, _ = oracle.forces(spec_to_system(spec), prec=64)
    assert force_error(f, fref) <= 1e-5


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("nsp,deterministic", [(1, 1), (2, 0), (3, 0), (3, 1)])
def test_large_deposit_boxes_launch_for_each_kernel(order, nsp, deterministic):
    # deposit tiles of 64 bricks (16 for three fields in 64 bits): boxes past the 48 KB that a
    # kernel has without opting in, alone, in a batch, and after the field count has dropped
    spec = species_system(nsp, (32, 32, 32), seed=order)
    spec.order = order
    if order == 4:   # away from cell edges, where the order-4 weights jump (see above)
        h = spec.L[0] / 32
        c = np.floor(spec.x / h)
        spec.x = ((c + 0.1 + 0.3 * (spec.x / h - c)) * h).astype(np.float32)
    opts = dict(deterministic=deterministic, tile_codes=8, deposit_codes=16 if nsp == 3 and deterministic else 64)
    fref, _ = oracle.forces(spec_to_system(spec), prec=64)
    with make_box(spec, **opts) as b:
        assert force_error(b.forces(), fref) <= 1e-5
        if nsp > 1:
            for _ in range(nsp):   # the interactions of the first species: one field fewer
                b.modify("potential remove 1")
            rest = list(spec.potentials)[nsp:]
            sub, _ = oracle.forces(spec_to_system(synth.SystemSpec(
                "rest", spec.L, spec.grid, spec.x, spec.types, spec.species, spec.bonds, spec.mol, potentials=rest,
                order=order)), prec=64)
            assert force_error(b.forces(), sub) <= 1e-5
    if nsp < 3:
        with make_box(spec, **opts) as b:
            b.step(2)
            alone = b.positions()
        with make_box(spec, **opts) as b, tild_b200.Batch() as batch:
            batch.add(b)
            batch.step(2)
            d = b.positions() - alone
            batch.close()
        assert np.abs(d - np.round(d / spec.L) * spec.L).max() <= (0.0 if deterministic else 1e-3)


@pytest.mark.parametrize("n,codes", [(80, 8), (88, 16)])
def test_default_deposit_tiles_on_either_side_of_the_tile_count(n, codes):
    # 500 and 726 tiles of 16 bricks: below and above four CTAs per SM
    rng = np.random.default_rng(n)
    spec = synth.SystemSpec("t", [float(n)] * 3, [n] * 3, rng.uniform(0.0, n, size=(1000, 3)), np.zeros(1000, np.int32), ["A"],
                            [], np.arange(1000), potentials=[dict(kind="gaussian", I="A", J="A", A=0.5, sigma=0.7)], order=3)
    with make_box(spec, tile_codes=8) as b:
        assert b.describe()["tiles"]["deposit_codes"] == codes
    with make_box(spec, tile_codes=8, deterministic=1) as b:
        assert b.describe()["tiles"]["deposit_codes"] == 8


def test_batch_of_two_stage_and_mixed_radix_boxes_with_dense_tiles():
    # a replica whose default 16-brick tiles are dense (halves), one of two-stage lines on
    # smaller tiles, and one on the mixed-radix path, two force groups each, in fast mode: the
    # same kernels as alone, sums in another order (FP32 rounding carried through five steps)
    rng = np.random.default_rng(17)
    pots = [dict(kind="gaussian", I=a, J=c, A=v, sigma=0.7) for a, c, v in (("A", "A", 1.0), ("A", "B", 1.5), ("B", "B", 1.0))]
    specs = []
    for g, dense in ((88, 700), (32, 0), (34, 0)):
        x = np.concatenate([rng.uniform(0.0, 8.0, size=(dense, 3)), rng.uniform(0.0, g, size=(2000, 3))])
        m = len(x)
        specs.append(synth.SystemSpec("b%d" % g, [float(g)] * 3, [g] * 3, x, np.arange(m) % 2, ["A", "B"], [], np.arange(m),
                                      potentials=pots, order=3, seed=g))
    alone = []
    for s in specs:
        with make_box(s, tile_codes=8) as b:
            b.step(5)
            alone.append(b.positions())
    boxes = [make_box(s, tile_codes=8) for s in specs]
    assert [b.describe()["tiles"]["deposit_codes"] for b in boxes] == [16, 8, 8]
    with tild_b200.Batch() as batch:
        for b in boxes:
            batch.add(b)
        batch.step(5)
    for b, x, s in zip(boxes, alone, specs):
        d = b.positions() - x
        assert np.abs(d - np.round(d / s.L) * s.L).max() <= 1e-4
        b.close()
