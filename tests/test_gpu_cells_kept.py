"""When cells are sorted again, at sizes whose skin test runs over the whole
GPU (2,048 beads and more, k_moved): beads are moved by steps, which keep the
sort until one has left the skin (set_coord always sorts afresh). Forces and
pair counts against the oracle at every position, and the kept order itself:
sums in another order than a fresh sort's show that the sort was kept, the
fresh sort's bits that it was not."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

from bd_box_b200 import decks, engine  # noqa: E402
import pyoracle  # noqa: E402

DENSE = {"cutoff_lj": 8, "hydro": "none"}   # cells of ~8.8 A, 16 beads each at phi = 0.1


def suspension(d, name, n, box=None):
    extra = dict(DENSE)
    if box:
        extra.update({k: f"{box:.6f}" for k in ("xbox", "ybox", "zbox")})
    return decks.read_deck(decks.write_suspension_deck(d, name, n, seed=n, phi=0.1, extra=extra))


def chain(d, name, n):
    return decks.read_deck(decks.write_chain_deck(d, name, n, seed=n, hydro="none", dt=0.005))


def case(kind, d):
    """The decks of a system, and the segments whose beads leave the skin."""
    if kind == "dense":
        return [suspension(d, "kd", 2304)], {0}
    if kind == "chain":
        return [chain(d, "kc", 2500)], {0}
    if kind == "batch":
        return [chain(d, f"kb{n}", n) for n in (900, 700, 800)], {1}
    if kind == "dense_batch":   # unequal segments in one box
        box = float(suspension(d, "ks", 1800).box[0])
        return [suspension(d, f"kd{n}", n, box) for n in (500, 1800, 300)], {2}
    return [chain(d, "kl", 17000)], {0}   # above the shared-memory sort


@pytest.mark.parametrize("kind", ["dense", "chain", "batch", "dense_batch", "large"])
def test_sort_is_kept_until_a_bead_leaves_the_skin(kind, tmp_path):
    ds, leave = case(kind, str(tmp_path))
    s = engine.System(ds if len(ds) > 1 else ds[0], precision=engine.PREC_FP64, noise=engine.NOISE_HOST)
    fresh = engine.System(ds if len(ds) > 1 else ds[0], precision=engine.PREC_FP64, noise=engine.NOISE_HOST)
    oracles = [pyoracle.Oracle(d) for d in ds]
    lo = np.cumsum([0] + [d.n for d in ds])
    rng = np.random.default_rng(3)
    n = s.n

    def check(kept, resorted):
        x = s.get_coord()
        F, _, rep, c = s.compute_forces()
        want, count, flag = [], np.zeros(2, dtype=np.int64), 0
        for k, o in enumerate(oracles):
            o.set_coord(x[lo[k]:lo[k + 1]])
            Fo, _, repo, co = o.forces()
            want.append(Fo)
            count += co
            flag |= repo
        want = np.concatenate(want)
        assert c == tuple(count) and rep == flag
        assert np.abs(F - want).max() <= 1e-12 * np.abs(want).max()
        fresh.set_coord(x)
        G = fresh.compute_forces()[0]
        for k in range(len(ds)):
            same = np.array_equal(F[3 * lo[k]:3 * lo[k + 1]], G[3 * lo[k]:3 * lo[k + 1]])
            if k in kept:
                assert not same, f"segment {k} was sorted again within its skin"
            if k in resorted:
                assert same, f"segment {k} was not sorted again"

    # the skin is 0.5 or a tenth of the reach, half of it is the limit
    prm = ds[0].prm
    radius = ds[0].coord[0, 3]
    unit = np.sqrt(2 * prm["dt"] * 0.00010537375739171604 * prm["T"] / (prm["visc"] * prm["vfactor"]) / radius)
    every = set(range(len(ds)))
    small = rng.uniform(-1, 1, size=3 * n) * 0.05 / unit     # within 0.05 A a coordinate
    s.step(1, small)
    check(every, set())
    big = rng.uniform(-1, 1, size=3 * n) * 0.02 / unit
    for k in leave:   # all beads of the segment by the same 6 A (no new overlaps)
        big[3 * lo[k]:3 * lo[k + 1]] += np.tile([4.0, 3.5, -2.8], lo[k + 1] - lo[k]) / unit
    s.step(1, big)
    check(every - leave, leave)
    if kind != "large":   # (the oracle's all pairs of 17,000 beads take seconds)
        s.step(1, rng.uniform(-1, 1, size=3 * n) * 0.02 / unit)
        check(every, set())
    s.close()
    fresh.close()
