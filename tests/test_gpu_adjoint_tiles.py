"""The adjoint's dense products (inverse of the factor, 128 x 128 tiles) at
sizes around their tiles, and its checkpoints: what a segment keeps and what
is computed again must give the same gradient."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

from bd_box_b200 import decks, engine  # noqa: E402


def make(n, deck_dir):
    d = decks.read_deck(decks.write_chain_deck(deck_dir, f"at{n}", n, seed=n, hydro="cholesky",
                                               extra={"cutoff_c": 1000, "cutoff_lj": 1000}))
    rng = np.random.default_rng(n)
    pairs = np.array([rng.choice(n, 2, replace=False) for _ in range(16)], dtype=np.int32)
    return d, pairs, rng.uniform(10, 60, size=16), rng


# 3N = 129, 255, 258, 513, 771: padded to 2, 2, 3, 5 and 7 tiles of 128
@pytest.mark.parametrize("n", [20, 43, 85, 86, 171, 257])
def test_gradient_at_tile_edges(n, deck_dir):
    d, pairs, targets, rng = make(n, deck_dir)
    K, out = 3, {}
    for prec in (engine.PREC_FP64, engine.PREC_MIXED):
        s = engine.System(d, precision=prec, refresh=1, seed=7)
        out[prec] = s.adjoint(K, 2, pairs, targets)
        s.close()
    (l64, gx, gp), (l32, mx, mp) = out[engine.PREC_FP64], out[engine.PREC_MIXED]
    assert abs(l32 - l64) <= 1e-7 * abs(l64)
    assert np.linalg.norm(mx - gx) <= 1e-5 * np.linalg.norm(gx)
    assert np.linalg.norm(mp - gp) <= 1e-4 * np.linalg.norm(gp)
    # FP64 against a central difference along a random direction: error
    # h^2 of a third derivative and 1e-16 loss / h
    v = rng.standard_normal((n, 3))
    v /= np.linalg.norm(v)
    h, f = 1e-4, []
    for sign in (1, -1):
        s = engine.System(d, precision=engine.PREC_FP64, refresh=1, seed=7)
        c = d.coord.copy()
        c[:, :3] += sign * h * v
        s.set_coord(c)
        s.step(K)
        x = s.get_coord()[:, :3]
        r = np.linalg.norm(x[pairs[:, 1]] - x[pairs[:, 0]], axis=1)
        f.append(np.mean((r - targets) ** 2))
        s.close()
    fd = (f[0] - f[1]) / (2 * h)
    assert abs(fd - np.sum(gx * v)) <= 1e-6 * np.linalg.norm(gx)


@pytest.mark.parametrize("prec", [engine.PREC_FP64, engine.PREC_MIXED])
def test_checkpoints_give_the_same_gradient(prec, deck_dir):
    d, pairs, targets, _ = make(60, deck_dir)
    got = []
    for ck in (1, 2, 3, 5, 8):
        s = engine.System(d, precision=prec, refresh=1, seed=9)
        got.append(s.adjoint(5, ck, pairs, targets))
        x = s.get_coord()
        s.close()
        s = engine.System(d, precision=prec, refresh=1, seed=9)
        s.step(5)
        assert np.abs(s.get_coord() - x).max() <= 1e-9   # left at the final positions
        s.close()
    for loss, gx, gp in got[1:]:
        # a recomputed segment starts from re-sorted cells: force sums in
        # another order
        assert abs(loss - got[0][0]) <= 1e-12 * abs(loss)
        tol = 1e-10 if prec == engine.PREC_FP64 else 1e-6
        assert np.linalg.norm(gx - got[0][1]) <= tol * np.linalg.norm(gx)
        assert np.linalg.norm(gp - got[0][2]) <= tol * np.linalg.norm(gp)


@pytest.mark.parametrize("prec", [engine.PREC_FP64, engine.PREC_MIXED])
@pytest.mark.parametrize("K,ck", [(6, 2), (5, 3), (3, 8)])
def test_kept_and_recomputed_matrices_agree(prec, K, ck, deck_dir):
    """With no room to keep a segment's matrices and forces the reverse pass
    computes them again from the positions."""
    d, pairs, targets, _ = make(60, deck_dir)
    got = []
    for keep in (-1, 0):
        s = engine.System(d, precision=prec, refresh=1, seed=9)
        s.set_adjoint_keep(keep)
        got.append(s.adjoint(K, ck, pairs, targets) + (s.get_coord(),))
        s.close()
    (l0, gx0, gp0, x0), (l1, gx1, gp1, x1) = got
    # forces from cells sorted anew: sums in another order
    assert abs(l1 - l0) <= 1e-12 * abs(l0)
    tol = 1e-10 if prec == engine.PREC_FP64 else 1e-6
    assert np.linalg.norm(gx1 - gx0) <= tol * np.linalg.norm(gx0)
    assert np.linalg.norm(gp1 - gp0) <= tol * np.linalg.norm(gp0)
    assert np.abs(x1 - x0).max() <= 1e-9


def test_scratch_is_two_matrices(deck_dir):
    """At 48 tiles the pieces of S go in two rounds; FP64 and mixed agree, and
    the call takes the room the header states: 2 (3N)^2 elements and 0.3 GB."""
    import threading
    import torch
    n = 2048
    d, pairs, targets, _ = make(n, deck_dir)
    out = {}
    for prec in (engine.PREC_FP64, engine.PREC_MIXED):
        s = engine.System(d, precision=prec, refresh=1, seed=7)
        s.set_adjoint_keep(0)
        s.adjoint(1, 1, pairs, targets)   # the system's own buffers are made
        s.set_coord(d.coord)
        torch.cuda.synchronize()
        before, least, done = torch.cuda.mem_get_info()[0], [], threading.Event()

        def watch():
            while not done.is_set():
                least.append(torch.cuda.mem_get_info()[0])

        t = threading.Thread(target=watch)
        t.start()
        out[prec] = s.adjoint(3, 3, pairs, targets)
        done.set()
        t.join()
        s.close()
        el = 8 if prec == engine.PREC_FP64 else 4
        assert before - min(least) <= 2.2 * (3 * n) ** 2 * el + 3e8
    (l64, gx, _), (l32, mx, _) = out[engine.PREC_FP64], out[engine.PREC_MIXED]
    assert abs(l32 - l64) <= 1e-7 * abs(l64)
    assert np.linalg.norm(mx - gx) <= 1e-5 * np.linalg.norm(gx)
