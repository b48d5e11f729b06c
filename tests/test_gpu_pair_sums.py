"""The matrix-free pair sums (tea.cu) against BD_BOX's restatement (the
oracle), at sizes where the work split changes: tile edges, one bead over,
odd numbers of tiles, jobs of several column and row tiles; and the converged
split of the lattice sums (ewald_fast.cuh) against the reference's own sums in
FP64, over what decides between the two."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

from bd_box_b200 import decks, engine  # noqa: E402


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 64, 65, 95, 97, 161])
def test_drift_and_noise_at_tile_edges(n, deck_dir):
    import pyoracle
    d = decks.read_deck(decks.write_chain_deck(deck_dir, f"pairs{n}", n, seed=50 + n, hydro="geyer"))
    o = pyoracle.Oracle(d)
    g = np.random.default_rng(n).standard_normal(3 * n)
    F = o.forces()[0]
    dt = d.prm["dt"]
    df, tea = o.df(F, dt), o.tea(g, dt)
    tea = tea[0] if isinstance(tea, tuple) else tea
    s = engine.System(d, precision=engine.PREC_FP64, noise=engine.NOISE_HOST)
    # 3N additions of ~1 ulp each side
    assert rel(s.compute_Rf(), df) <= 1e-13
    assert rel(s.compute_r(g), tea) <= 1e-13
    m = engine.System(d, precision=engine.PREC_MIXED, noise=engine.NOISE_HOST)
    assert rel(m.compute_Rf(), df) <= 2e-6
    assert rel(m.compute_r(g), tea) <= 2e-6


@pytest.mark.parametrize("sizes", [(2, 33, 700, 64, 31), tuple(range(600, 900, 6)), (1500,) * 6 + (1441, 1409)])
def test_mixed_batch_follows_fp64(sizes, deck_dir):
    """Batches whose jobs hold 1, 2 and more column tiles, with and without
    row-tile pairs (odd and even tile counts)."""
    ds = [decks.read_deck(decks.write_chain_deck(deck_dir, f"b{n}", n, seed=n, hydro="geyer")) for n in sorted(set(sizes))]
    by_n = {d.n: d for d in ds}
    batch = [by_n[n] for n in sizes]
    n3 = 3 * sum(sizes)
    g = np.random.default_rng(1).standard_normal(n3)
    out = {}
    for p in (engine.PREC_FP64, engine.PREC_MIXED):
        s = engine.System(batch, precision=p, noise=engine.NOISE_HOST)
        out[p] = s.compute_Rf(), s.compute_r(g)
        s.close()
    for a, b in zip(out[engine.PREC_MIXED], out[engine.PREC_FP64]):
        assert np.isfinite(a).all()
        assert rel(a, b) <= 1e-6


def test_jobs_of_several_column_tiles(deck_dir):
    """39,600 tile pairs: jobs of 2 column tiles on two row tiles in FP32, of 4
    in FP64 (their row sums take two records, or one FP64). Each segment as it
    is alone, where a job is half a tile pair."""
    ds = [decks.read_deck(decks.write_chain_deck(deck_dir, f"jt{n}", n, seed=n, hydro="geyer")) for n in (1300, 1281)]
    batch = [ds[0]] * 45 + [ds[1]]
    rng = np.random.default_rng(8)
    g = rng.standard_normal(3 * sum(d.n for d in batch))
    for prec, tol in ((engine.PREC_FP64, 1e-13), (engine.PREC_MIXED, 1e-6)):
        s = engine.System(batch, precision=prec, noise=engine.NOISE_HOST)
        rf, rs = s.compute_Rf(), s.compute_r(g)
        s.close()
        for k in (0, 17, 44, 45):
            lo = 3 * 1300 * k
            sl = slice(lo, lo + 3 * batch[k].n)
            a = engine.System(batch[k], precision=prec, noise=engine.NOISE_HOST)
            assert rel(rf[sl], a.compute_Rf()) <= tol
            assert rel(rs[sl], a.compute_r(g[sl])) <= tol
            a.close()


@pytest.mark.parametrize("method", ["beenakker", "smith"])
@pytest.mark.parametrize("r", [2, 3, 4, 5])
@pytest.mark.parametrize("kind", ["plain", "radii", "outside", "overlap"])
def test_lattice_sums_mixed_against_fp64(method, r, kind, deck_dir):
    """R = 4 and 5 take the converged split where it holds; other radii than
    bead 0's, beads outside the box and overlapping pairs go back to the
    reference's sums, pair by pair."""
    n = 97
    d = decks.read_deck(decks.write_suspension_deck(deck_dir, f"lat_{method}{r}", n, seed=3, ewald_r=r,
                                                    extra={"ewald_method": method}))
    d.coord = d.coord.copy()
    if kind == "radii":
        d.coord[::3, 3] *= 0.7
    elif kind == "outside":
        d.coord[5, 0] += d.box[0]
        d.coord[40, 2] -= 2 * d.box[0]
    elif kind == "overlap":
        d.coord[11, :3] = d.coord[60, :3] + [0.9, 0.4, -0.3]
    g = np.random.default_rng(4).standard_normal(3 * n)
    s64 = engine.System(d, precision=engine.PREC_FP64, noise=engine.NOISE_HOST)
    mix = engine.System(d, precision=engine.PREC_MIXED, noise=engine.NOISE_HOST)
    assert rel(mix.compute_Rf(), s64.compute_Rf()) <= 2e-6
    if kind in ("plain", "radii"):   # the others make eps, hence TEA, meaningless
        assert rel(mix.compute_r(g), s64.compute_r(g)) <= 4e-6


@pytest.mark.parametrize("method", ["beenakker", "smith"])
def test_lattice_sums_fp64_against_oracle(method, deck_dir):
    import pyoracle
    d = decks.read_deck(decks.write_suspension_deck(deck_dir, f"lo_{method}", 40, seed=9, ewald_r=5,
                                                    extra={"ewald_method": method}))
    o = pyoracle.Oracle(d)
    s = engine.System(d, precision=engine.PREC_FP64, noise=engine.NOISE_HOST)
    for i, j in ((0, 1), (7, 30), (39, 2), (5, 5)):
        a, b = s.compute_Dij(i, j), np.asarray(o.tile(max(i, j), min(i, j))).reshape(3, 3)
        assert np.abs(a - b).max() <= 1e-13 * np.abs(o.tile(0, 0)).max()


# R, Smith's ewald_alpha (0: Beenakker), box lengths; at each of them the
# Gaussian recurrence along a row of images overflows if it is used
@pytest.mark.parametrize("r,alpha,boxes", [(4, 0.0, 120), (3, 0.0, 120), (3, 1.7724538509055159, 120), (3, 4.8, 16),
                                           (2, 6.0, 11), (5, 3.4, 40), (0, 1.7724538509055159, 300)])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_lattice_sums_fp64_far_outside_the_box(r, alpha, boxes, axis, deck_dir):
    """Steps wrap positions, callers need not: a bead many box lengths away in
    either direction has the oracle's tile, which sums image by image."""
    import pyoracle
    extra = {"ewald_method": "smith", "ewald_alpha": alpha} if alpha else {}
    d = decks.read_deck(decks.write_suspension_deck(deck_dir, f"far{r}_{boxes}", 24, seed=5, ewald_r=r, extra=extra))
    d.coord = d.coord.copy()
    d.coord[3, axis] += boxes * d.box[0]
    d.coord[17, axis] -= boxes * d.box[0]
    o = pyoracle.Oracle(d)
    s = engine.System(d, precision=engine.PREC_FP64, noise=engine.NOISE_HOST)
    scale = np.abs(o.tile(0, 0)).max()
    for i, j in ((3, 0), (17, 0), (17, 3), (5, 1)):
        a, b = s.compute_Dij(i, j), np.asarray(o.tile(i, j)).reshape(3, 3)
        # phases 2 pi k v carry v's rounding: 2 pi R |v| ulps of weights ~ 1
        assert np.abs(a - b).max() <= 2e-16 * 8 * np.pi * (r + 1) * (2 * boxes + 1) * scale
    assert np.isfinite(s.compute_Rf()).all()
    assert np.isfinite(s.compute_r(np.random.default_rng(r).standard_normal(72))).all()


@pytest.mark.parametrize("prec,far", [(engine.PREC_FP64, 1e155), (engine.PREC_MIXED, 1e20)])
@pytest.mark.parametrize("hydro", ["geyer", "cholesky"])
def test_a_bead_whose_distance_squared_overflows(prec, far, hydro, deck_dir):
    """Its tiles with all other beads vanish: everyone else moves as without it."""
    n = 70
    d = decks.read_deck(decks.write_chain_deck(deck_dir, f"far_{hydro}", n, seed=6, hydro=hydro))
    for k, w, m in (("bond", 2, 3), ("angle", 3, 2), ("angle_cos", 3, 2), ("dihe", 4, 2), ("dihe_angle", 4, 2)):
        setattr(d, k + "_pairs", np.zeros((0, w), np.int32))
        setattr(d, k + "_parms", np.zeros((0, m)))
    d.coord = d.coord.copy()
    out = []
    for x in (300.0, far):
        d.coord[n - 1, :3] = (x, -x, 0.5 * x)
        s = engine.System(d, precision=prec, noise=engine.NOISE_HOST)
        out.append((s.compute_D() if hydro == "cholesky" else s.compute_Rf()))
        s.close()
    near, gone = out
    assert np.isfinite(gone).all()
    if hydro == "cholesky":
        assert np.array_equal(gone[:-3, :-3], near[:-3, :-3])
        assert np.abs(gone[-3:, :-3]).max() <= 1e-15 * np.abs(gone).max()
    else:   # no force acts on the far bead, nor does it change the others' drift
        assert rel(gone[:-3], near[:-3]) <= (1e-13 if prec == engine.PREC_FP64 else 1e-6)


@pytest.mark.parametrize("first", [1.0, 3e4])
def test_close_pairs_beside_a_large_bead(first, deck_dir):
    """The grid on which the mixed path's separations are exact follows the
    least radius: with a first bead 1.5e4 times as large as the others, whose
    neighbours are a few of their radii away, every separation still rounds
    like one FP32 operation."""
    n = 64
    d = decks.read_deck(decks.write_chain_deck(deck_dir, f"big{int(first)}", n, seed=4, hydro="geyer"))
    d.coord = d.coord.copy()
    d.coord[:, :3] *= 0.7
    d.coord[0] = (5e4, 5e4, 5e4, first)
    out = {}
    for p in (engine.PREC_FP64, engine.PREC_MIXED):
        s = engine.System(d, precision=p, noise=engine.NOISE_HOST)
        out[p] = s.compute_r(np.random.default_rng(2).standard_normal(3 * n)).reshape(n, 3)
        s.close()
    assert rel(out[engine.PREC_MIXED][1:], out[engine.PREC_FP64][1:]) <= 1e-6
