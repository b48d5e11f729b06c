"""The lattice sums' own erfcx, 1/sqrt and Gaussian (rpy_tile.cuh) over their
range, one image at a time: with R = 0 a pair's Smith tile is a single image
and no reciprocal vector, a closed form of erfc(x) and exp(-x^2), x = alpha r."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

from bd_box_b200 import decks, engine  # noqa: E402

L, RADIUS = 64.0, 1.0 / 256   # coordinates are multiples of 1/16: r/L and its square are exact in FP32 too


@pytest.mark.parametrize("alpha", [0.25, 1.0, 1.75, 4.5, 20.0])
@pytest.mark.parametrize("prec", [engine.PREC_FP64, engine.PREC_MIXED])
def test_one_image(alpha, prec, deck_dir):
    from scipy.special import erfcx
    n = 80
    box = {k: f"{L:.6f}" for k in ("xbox", "ybox", "zbox")}
    d = decks.read_deck(decks.write_suspension_deck(
        deck_dir, f"im{alpha}", n, seed=2, ewald_r=0, radius=RADIUS,
        extra={"ewald_method": "smith", "ewald_alpha": alpha, "hydro": "cholesky", **box}))
    d.coord = d.coord.copy()
    rng = np.random.default_rng(int(4 * alpha))
    # half the beads over the whole box, half near its middle: r/L from 0.001 to 1.7
    x = rng.integers(-512, 512, size=(n, 3)) / 16
    x[::2] = rng.integers(-24, 25, size=(n // 2, 3)) / 16
    d.coord[:, :3] = x
    s = engine.System(d, precision=prec, noise=engine.NOISE_HOST)
    D = s.compute_D().reshape(n, 3, n, 3).transpose(0, 2, 1, 3)
    s.close()
    i, j = np.triu_indices(n, 1)
    v = (x[i] - x[j]) / L
    r2 = np.sum(v * v, axis=1)
    keep = r2 > 0
    if prec == engine.PREC_MIXED:   # images beyond erfc(4.45) are dropped there
        keep &= alpha * alpha * r2 < 4.4 ** 2
    i, j, v, r2 = i[keep], j[keep], v[keep], r2[keep]
    assert len(i) > 100 and (prec == engine.PREC_MIXED or np.sqrt(r2).max() > 1)
    r, a, s2 = np.sqrt(r2), d.prm["ewald_alpha"], (RADIUS / L) ** 2
    g = np.exp(-(np.longdouble(a) ** 2) * r2.astype(np.longdouble))   # (its argument in 64 bits)
    er = g * erfcx(a * r) / r
    e = 2 * a * 0.5641895835 * g                                     # BD_BOX's 10 digits of 1/sqrt(pi)
    sq = (er + e) / r2
    A = 0.75 * er + 0.5 * s2 * sq
    B = (0.75 * (er + e) - 0.5 * s2 * (3 * sq + 2 * a * a * e)) / r2
    pre = 0.00010537375739171604 * d.prm["T"] / (d.prm["visc"] * d.prm["vfactor"]) / L
    want = pre * (A[:, None, None] * np.eye(3) + B[:, None, None] * v[:, :, None] * v[:, None, :])
    size = np.abs(want).max(axis=(1, 2))
    err = np.abs(D[i, j] - want).max(axis=(1, 2)) / size
    x2 = a * a * r2
    if prec == engine.PREC_FP64:
        # about 20 operations, and the rounding of the exponent, x^2 ulps
        ok = size > 1e-290
        assert (err[ok] <= 2.3e-16 * (24 + 2 * x2[ok].astype(float))).all()
    else:
        # the exponent's rounding is put back: no growth with x^2
        assert (err <= 6e-8 * 24).all(), err.max() / 6e-8


def test_constants_do_not_bias_the_mean(deck_dir):
    """The polynomials' constants are rounded alike in every image, so a
    constant that is off by ulps shifts the tensor's mean, which TEA's eps is.
    Beenakker's tiles of 250 pairs against 40 digits: single errors of 3.4e-15
    of the tiles' size leave 6.5e-16 in their mean (three standard errors),
    and the constants, half an ulp each of numbers up to 2.5 where a tile's sum
    is 0.2, up to 7e-16."""
    mp = pytest.importorskip("mpmath")
    R, n = 2, 60
    d = decks.read_deck(decks.write_suspension_deck(deck_dir, "bias", n, seed=3, ewald_r=R,
                                                    extra={"hydro": "cholesky"}))
    s = engine.System(d, precision=engine.PREC_FP64, noise=engine.NOISE_HOST)
    D = s.compute_D()
    s.close()
    box = mp.mpf(float(d.box[0]))
    root_pi = mp.mpf(1.77245385090551602729)   # as the reference spells it
    pre = 0.00010537375739171604 * d.prm["T"] / (d.prm["visc"] * d.prm["vfactor"])
    rng = np.random.default_rng(0)
    err, size = [], []
    with mp.workdps(40):
        a = root_pi / box
        for _ in range(250):
            i, j = sorted(rng.choice(n, 2, replace=False))
            r = [mp.mpf(float(d.coord[i, k])) - mp.mpf(float(d.coord[j, k])) for k in range(3)]
            s2 = mp.mpf(float(d.coord[i, 3] ** 2 + d.coord[j, 3] ** 2)) / 2
            tr, sq = mp.mpf(0), 0.0
            for h, f, g in np.ndindex(2 * R + 1, 2 * R + 1, 2 * R + 1):
                m = (h - R, f - R, g - R)
                if sum(q * q for q in m) > R * R:
                    continue
                x2 = sum((r[k] + box * m[k]) ** 2 for k in range(3))
                x, ex = mp.sqrt(x2), mp.exp(-a * a * x2) / root_pi
                er = mp.erfc(a * x)
                A = (a * s2 / x2 + 14 * a**3 * s2 - 4.5 * a - 20 * a**5 * s2 * x2 + 3 * a**3 * x2
                     + 4 * a**7 * s2 * x2**2) * ex + er * (0.75 / x + s2 / (2 * x * x2))
                B = (-3 * a * s2 / x2 - 2 * a**3 * s2 + 1.5 * a + 16 * a**5 * s2 * x2 - 3 * a**3 * x2
                     - 4 * a**7 * s2 * x2**2) * ex + er * (0.75 / x - 3 * s2 / (2 * x * x2))
                tr += 3 * A + B   # (the reciprocal weights are exp(-pi L^2) here)
            t = D[3 * i:3 * i + 3, 3 * j:3 * j + 3]
            err.append(float(mp.mpf(float(t[0, 0])) + mp.mpf(float(t[1, 1])) + mp.mpf(float(t[2, 2])) - pre * tr))
            size.append(np.mean(t * t))
    assert abs(np.mean(err)) <= 1.4e-15 * np.sqrt(np.mean(size))
