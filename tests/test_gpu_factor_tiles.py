"""The tiled Cholesky factorisation at sizes around its 128-column panels, from
a matrix of one block (no panel below it, no update) up, against LAPACK's
factor of the same D in 64 bits, and the captured refresh at those sizes."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

from bd_box_b200 import decks, engine  # noqa: E402


# 3N = 15, 60, 126 | 129, 255 | 258, 384 | 387, 771, 1155: 1, 2, 3, 4, 7 and 10 blocks
@pytest.mark.parametrize("n", [5, 20, 42, 43, 85, 86, 128, 129, 257, 385])
@pytest.mark.parametrize("prec", [engine.PREC_FP64, engine.PREC_MIXED])
def test_factor_at_block_edges(n, prec, deck_dir):
    d = decks.read_deck(decks.write_chain_deck(deck_dir, f"ft{n}", n, seed=n, hydro="cholesky"))
    g = np.random.default_rng(n).standard_normal(3 * n)
    s = engine.System(d, precision=prec, refresh=1, noise=engine.NOISE_HOST)
    D = s.compute_D()
    Rs = np.asarray(s.compute_r(g)).ravel()
    s.close()
    ref = np.sqrt(2 * d.prm["dt"]) * (np.linalg.cholesky(D) @ g)
    # backward error of a Cholesky factor, 3N eps |D|, times D's condition
    # number; eps 2^-53, or 2^-22 where L is stored in FP32 and updated from
    # split halves
    w = np.linalg.eigvalsh(D)
    eps = 2.0 ** -53 if prec == engine.PREC_FP64 else 2.0 ** -22
    assert np.linalg.norm(Rs - ref) <= 3 * n * eps * w[-1] / w[0] * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [20, 42, 43, 129])
def test_captured_refresh_at_block_edges(n, deck_dir):
    d = decks.read_deck(decks.write_chain_deck(deck_dir, f"fc{n}", n, seed=n, hydro="cholesky"))
    x0 = decks.read_deck(decks.write_chain_deck(deck_dir, f"fc{n}", n, seed=n, hydro="cholesky")).coord[:, :3]
    g = np.random.default_rng(n).standard_normal((8, 3 * n))
    out = []
    for prec in (engine.PREC_FP64, engine.PREC_MIXED):
        s = engine.System(d, precision=prec, refresh=4, noise=engine.NOISE_HOST)
        s.step(8, g)
        out.append(np.asarray(s.get_coord()).reshape(n, -1)[:, :3] - x0)
        s.close()
    assert np.linalg.norm(out[1] - out[0]) <= 1e-5 * np.linalg.norm(out[0])
