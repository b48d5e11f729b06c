"""The non-bonded kernel where its per-bead lists overflow what a warp holds: a
bead with more than 8 bonded neighbours (1-2 pairs scaled, so each must be
recognised) and with more than 10 bonded slots (bonds, angles and dihedrals),
alone in a small segment and among the cells of a larger one."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

from bd_box_b200 import decks, engine  # noqa: E402
import pyoracle  # noqa: E402


@pytest.mark.parametrize("n,arms", [(40, 8), (40, 9), (40, 12), (700, 12), (700, 33)])
@pytest.mark.parametrize("angles", [False, True])
def test_star_against_oracle(n, arms, angles, deck_dir):
    d = decks.read_deck(decks.write_chain_deck(deck_dir, f"star{n}_{arms}", n, seed=n + arms, hydro="none",
                                               extra={"bond_lj_scale": 0.5, "bond_c_scale": 0.25}))
    hub = n // 2
    rng = np.random.default_rng(arms)
    # the hub's nearest beads are its arms, so that the scaled pairs lie within the cutoffs
    near = np.argsort(np.linalg.norm(d.coord[:, :3] - d.coord[hub, :3], axis=1))[1:]
    chained = {hub - 1, hub + 1}
    arm = [int(b) for b in near if int(b) not in chained][:arms - 2]
    pairs = [(hub, b) if rng.random() < 0.5 else (b, hub) for b in arm]
    d.bond_pairs = np.vstack([d.bond_pairs, np.array(pairs, np.int32).reshape(-1, 2)]).astype(np.int32)
    d.bond_parms = np.vstack([d.bond_parms, np.tile([6.0, 1e4, 2.0], (len(arm), 1))])
    if angles:
        d.angle_pairs = np.array([[arm[k], hub, arm[k + 1]] for k in range(len(arm) - 1)], np.int32)
        d.angle_parms = np.tile([1.9, 3.0], (len(arm) - 1, 1))
        d.dihe_angle_pairs = np.array([[hub, arm[k], arm[k + 1], arm[k + 2]] for k in range(3)], np.int32)
        d.dihe_angle_parms = np.tile([0.6, 2.0], (3, 1))
    o = pyoracle.Oracle(d)
    Fo, Eo, repo, co = o.forces()
    s = engine.System(d, precision=engine.PREC_FP64, noise=engine.NOISE_HOST)
    F, E, rep, c = s.compute_forces()
    assert rep == repo and c == co
    assert np.abs(F - Fo).max() <= 1e-12 * np.abs(Fo).max()
    for k in range(1, 9):
        assert abs(E[k] - Eo[k]) <= 1e-10 * max(abs(Eo[k]), 1e-12), (k, E[k], Eo[k])
    # without energies another instance of the kernel runs
    assert np.array_equal(s.compute_forces(energies=False)[0], F)
    s.close()
