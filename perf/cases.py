"""The measured workloads of the framework: the work its users have it do,
through its public entry points, over the range of sizes, precisions and
options that its configurations, tests and benchmark use.

A case is a dict of plain values. ``kind`` picks the entry point:

* ``product``  bdb_stored_matvec_noalloc: D.F and L.X from a stored matrix on
               buffers that the caller owns (device pointers, no set-up);
* ``step``     System.step: Ermak-McCammon steps, then the positions read back,
               as a driver that follows BD_BOX's main loop does;
* ``igt``      System.step_igt: the predictor-corrector, positions read back;
* ``drift``    System.compute_Rf and System.compute_r at fixed positions:
               D.F and the random displacement by themselves;
* ``forces``   System.compute_forces with energies and pair counts;
* ``adjoint``  System.adjoint: a loss's gradient back through the steps.

``prec`` is 64 (everything in FP64) or 32 (the mixed path). Chains are
self-avoiding walks with the benchmark's force field (harmonic bonds, LJ,
Debye-Hueckel); suspensions are spheres at volume fraction 0.1 in a periodic
box, inserted at random without overlaps.

``exact`` computes the same outputs in plain torch and numpy in 64 bits.
"""
import ctypes
import math
import os
import random
import tempfile

import numpy as np
import torch

from bd_box_b200 import decks, engine

KB, KB_8PI, KB_6PI = 0.001986248532617, 0.00007903031804378703, 0.00010537375739171604
PIF = float(np.float32(math.pi))


def f32(x):
    """A .prm value as BD_BOX reads it (rounded to float)."""
    return float(np.float32(x))


# ------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest call: the per-step products of a host that owns all
        # device memory, at the entry point's largest size
        {"name": "product_1024", "kind": "product", "n": 1024},
        # BD_BOX's own loop on a small protein-sized chain: one step a call,
        # Gaussians from the host, positions back; FP64 TEA
        {"name": "tea_chain_96_fp64", "kind": "step", "n": 96, "hydro": "geyer", "prec": 64, "k": 1, "refresh": 1,
         "host": True},
        # the plain method: D and its Cholesky factor rebuilt every step, FP64
        {"name": "chol_chain_512_fp64", "kind": "step", "n": 512, "hydro": "cholesky", "prec": 64, "k": 1,
         "refresh": 1, "host": False},
        # the headline workload: D and L rebuilt every ten steps, mixed precision
        {"name": "chol_chain_4096_mixed", "kind": "step", "n": 4096, "hydro": "cholesky", "prec": 32, "k": 10,
         "refresh": 10, "host": False},
        # the FP64 path at a size that is no multiple of any tile
        {"name": "chol_chain_2001_fp64", "kind": "step", "n": 2001, "hydro": "cholesky", "prec": 64, "k": 10,
         "refresh": 10, "host": False},
        # predictor-corrector on a ragged chain, two factorisations a step
        {"name": "igt_chain_1001_mixed", "kind": "igt", "n": 1001, "hydro": "cholesky", "prec": 32, "k": 1,
         "host": False},
        # 256 independent chains of 64 to 1024 beads advanced together, TEA
        {"name": "replicas_256_mixed", "kind": "step", "n": 64, "n_max": 1024, "replicas": 256, "hydro": "geyer",
         "prec": 32, "k": 10, "refresh": 1, "host": False},
        # the periodic suspension (Beenakker sums, TEA) of the benchmark
        {"name": "ewald_4096_mixed", "kind": "step", "n": 4096, "hydro": "geyer", "ewald": "beenakker", "r": 4,
         "prec": 32, "k": 1, "refresh": 1, "host": False},
        # Smith's sums in FP64: D.F and TEA noise at given Gaussians
        {"name": "smith_777_fp64", "kind": "drift", "n": 777, "hydro": "geyer", "ewald": "smith", "r": 3, "prec": 64},
        # D.F and TEA noise of one free-space chain in FP64, matrix-free
        {"name": "tea_chain_3000_fp64", "kind": "drift", "n": 3000, "hydro": "geyer", "prec": 64},
        # forces, energies and pair counts of a dense system that needs the
        # multi-CTA cell sort
        {"name": "forces_20000", "kind": "forces", "n": 20000, "hydro": "none", "prec": 64, "ewald": "none"},
        # gradient of a pair-distance loss through ten steps, mixed precision
        {"name": "adjoint_1024_mixed", "kind": "adjoint", "n": 1024, "hydro": "cholesky", "prec": 32, "k": 10,
         "checkpoint": 5},
    ]


def draw(rng: random.Random):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["product", "step_tea", "step_chol", "step_chol", "igt", "replicas", "ewald", "drift", "forces",
                       "adjoint"])
    prec = rng.choice([32, 64])
    if kind == "product":
        return {"kind": "product", "n": size(16, 1024)}
    if kind == "step_tea":
        return {"kind": "step", "n": size(32, 4096 if prec == 32 else 2500), "hydro": "geyer", "prec": prec,
                "k": rng.choice([1, 10]), "refresh": 1, "host": rng.random() < 0.5}
    if kind == "step_chol":
        return {"kind": "step", "n": size(40, 4096 if prec == 32 else 2000), "hydro": "cholesky", "prec": prec,
                "k": rng.choice([1, 10]), "refresh": rng.choice([1, 10]) if prec == 32 else 10,
                "host": rng.random() < 0.5}
    if kind == "igt":
        return {"kind": "igt", "n": size(40, 2500 if prec == 32 else 1000), "hydro": "cholesky", "prec": prec, "k": 1,
                "host": rng.random() < 0.5}
    if kind == "replicas":
        lo = size(16, 200)
        return {"kind": "step", "n": lo, "n_max": lo + size(10, 800 if prec == 32 else 300),
                "replicas": size(3, 256 if prec == 32 else 64), "hydro": "geyer", "prec": prec,
                "k": rng.choice([1, 10]), "refresh": 1, "host": False}
    if kind == "ewald":
        return {"kind": "step", "n": size(50, 4000 if prec == 32 else 1200), "hydro": "geyer",
                "ewald": rng.choice(["beenakker", "smith"]), "r": rng.choice([2, 3, 4, 5]), "prec": prec,
                "k": rng.choice([1, 2]), "refresh": 1, "host": rng.random() < 0.5}
    if kind == "drift":
        per = rng.random() < 0.5
        return {"kind": "drift", "n": size(50, 1000 if per else 3000), "hydro": "geyer",
                "ewald": rng.choice(["beenakker", "smith"]) if per else "", "r": rng.choice([2, 3, 4]), "prec": prec}
    if kind == "forces":
        per = rng.random() < 0.6
        return {"kind": "forces", "n": size(60, 20000 if per else 4096), "hydro": "none", "prec": 64,
                "ewald": "none" if per else ""}
    return {"kind": "adjoint", "n": size(40, 1024 if prec == 32 else 500), "hydro": "cholesky", "prec": prec,
            "k": rng.choice([3, 6, 10]), "checkpoint": rng.choice([2, 5])}


# --------------------------------------------------------------- geometry

def _walks(sizes, seed):
    """Self-avoiding walks of the given sizes, grown side by side: steps of
    3.8 A, non-consecutive beads at least 4 A apart (of 16 directions the
    first that fits). Returns one (n, 3) array per walk."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    nw, nmax, tries = len(sizes), max(sizes), 16
    g = np.random.default_rng(seed)
    pos = torch.zeros((nw, nmax, 3), dtype=torch.float64, device=dev)
    rows = torch.arange(nw, device=dev)
    score = torch.arange(tries, 0, -1, dtype=torch.float64, device=dev) * 1e6
    block = max(1, (1 << 22) // (nw * tries * 3))
    for i in range(1, nmax):
        at = (i - 1) % block
        if at == 0:
            d = torch.from_numpy(g.standard_normal((min(block, nmax - i), nw, tries, 3))).to(dev)
            d = 3.8 * d / d.norm(dim=3, keepdim=True)
        cand = pos[:, i - 1:i, :] + d[at]
        if i > 1:
            near = torch.full((nw, tries), 1e9, dtype=torch.float64, device=dev)
            gap = torch.cdist(cand, pos[:, :i - 1, :], compute_mode="donot_use_mm_for_euclid_dist")
            near = gap.amin(dim=2)
            pick = torch.where(near >= 4.0, score + 4.0, near).argmax(dim=1)
            pos[:, i, :] = cand[rows, pick]
        else:
            pos[:, i, :] = cand[:, 0]
    out = pos.cpu().numpy()
    return [out[w, :n].copy() for w, n in enumerate(sizes)]


def _suspension(n, seed):
    """n unit spheres at volume fraction 0.1 in a cubic box, inserted one
    after another at uniform positions, overlapping ones rejected."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    L = f32("%.6f" % (n * 4.0 / 3.0 * math.pi / 0.1) ** (1.0 / 3.0))
    m = 2 * n + 64
    cand = np.random.default_rng(seed).uniform(-L / 2, L / 2, size=(m, 3))
    c = torch.from_numpy(cand).to(dev)
    clash = [[] for _ in range(m)]
    for b in range(0, m, 512):
        d = c[b:b + 512, None, :] - c[None, :, :]
        d -= L * torch.round(d / L)
        hit = torch.nonzero((d * d).sum(dim=2) < 4.02).cpu().numpy()
        for i, j in hit:
            if j < i + b:
                clash[i + b].append(int(j))
    ok, kept = np.zeros(m, dtype=bool), []
    for i in range(m):
        if not any(ok[j] for j in clash[i]):
            ok[i] = True
            kept.append(i)
            if len(kept) == n:
                return cand[kept], L
    raise RuntimeError("suspension too dense")


PRM = {"T": 293, "visc": 0.01, "vfactor": 14.4, "bdsteps": 1000, "algorithm": "ermak_const", "epsilon_c": 78.54,
       "kappa_c": 0.1, "gamma_c": 331.842, "alpha_lj": 4, "lj_6_term": "yes", "bond_lj_scale": 0, "bond_c_scale": 0,
       "check_overlap": "no", "nb_list": "bucket_space", "geyer_on_the_fly": "yes"}


def _inputs(case, seed):
    """(list of bead-system dicts, .prm keys): everything made from the seed."""
    prm = dict(PRM, hydro=case.get("hydro", "none"), rand_seed=1 + seed % 30000)
    if case.get("ewald"):
        pos, L = _suspension(case["n"], seed)
        n = len(pos)
        charged = case["kind"] == "forces"
        prm.update(dt=0.005, bc="periodic", xbox="%.6f" % L, ybox="%.6f" % L, zbox="%.6f" % L,
                   elec="yes" if charged else "no", cutoff_c=12, cutoff_lj=-1)
        if case["ewald"] != "none":
            prm.update(ewald_method=case["ewald"], ewald_real=case["r"], ewald_recip=case["r"])
        q = np.random.default_rng(seed + 7919).choice([-1.0, 1.0], size=n) if charged else np.zeros(n)
        return [{"pos": pos, "radius": 1.0, "q": q, "lj": (1.0, 0.5), "bonds": 0, "L": L}], prm
    prm.update(dt=0.01, bc="none", elec="yes", cutoff_c=12, cutoff_lj=12)
    g = np.random.default_rng(seed + 17)
    sizes = [case["n"]]
    if case.get("replicas"):
        sizes = [int(v) for v in decks.replica_sizes(case["replicas"], case["n"], case["n_max"])]
    return [{"pos": p, "radius": 2.0, "q": g.choice([-1.0, 1.0], size=len(p)), "lj": (2.0, 0.1), "bonds": len(p) - 1,
             "L": 0.0} for p in _walks(sizes, seed)], prm


def _decks(case, seed):
    systems, keys = _inputs(case, seed)
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "case.prm")
        with open(path, "w") as f:
            f.writelines("%s %s\n" % kv for kv in keys.items())
        prm = decks.read_prm(path)
    out = []
    for s in systems:
        n, b = len(s["pos"]), s["bonds"]
        none = {w: np.zeros((0, k), dtype=t) for w, k, t in (
            ("angle_pairs", 3, np.int32), ("angle_parms", 2, float), ("angle_cos_pairs", 3, np.int32),
            ("angle_cos_parms", 2, float), ("dihe_pairs", 4, np.int32), ("dihe_parms", 2, float),
            ("dihe_angle_pairs", 4, np.int32), ("dihe_angle_parms", 2, float))}
        out.append(decks.Deck(
            prm=prm, coord=np.column_stack([s["pos"], np.full(n, s["radius"])]), Q=s["q"],
            LJ=np.tile(np.array(s["lj"]), (n, 1)), masses=np.ones(n), ids=np.arange(1, n + 1, dtype=np.int32),
            bond_pairs=np.column_stack([np.arange(b), np.arange(b) + 1]).astype(np.int32).reshape(-1, 2),
            bond_parms=np.tile(np.array([3.8, 1e10, 10.0]), (b, 1)).reshape(-1, 3),
            box=np.full(4, s["L"]) * np.array([1, 1, 1, 0]),
            inv_L=np.full(4, 1 / s["L"] if s["L"] else 0.0) * np.array([1, 1, 1, 0]),
            ewald=int(bool(s["L"]) and case.get("hydro") not in (None, "none")),
            max_force_cutoff=12.01 if prm["elec"] else 2.3, **none))
    return out


def _gauss(case, seed, n3, count):
    return np.random.default_rng(seed + 23).standard_normal((count, n3))


def _loss(case, seed, n):
    g = np.random.default_rng(seed + 31)
    a = g.integers(0, n, size=128)
    b = (a + g.integers(1, n, size=128)) % n
    return np.column_stack([a, b]).astype(np.int32), g.uniform(10, 60, size=128)


def _product_inputs(case, seed):
    """A stored matrix as the Cholesky path keeps it (D above the diagonal,
    its factor below), of a random symmetric positive definite D."""
    n3 = 3 * case["n"]
    ld = (n3 + 3) // 4 * 4
    g = torch.Generator().manual_seed(seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    a = torch.randn((n3, 32), generator=g, dtype=torch.float64).to(dev) / 16
    D = a @ a.T * 0.05
    D.diagonal().add_(0.1)
    M = torch.zeros((n3, ld), dtype=torch.float32, device=dev)
    M[:, :n3] = (torch.triu(D, 1) + torch.linalg.cholesky(D)).float()
    v = torch.randn((2, n3), generator=g, dtype=torch.float64).to(dev)
    return M, D.diagonal().clone(), v[0].contiguous(), v[1].contiguous()


# ------------------------------------------------------- the measured calls

def prepare(case, seed):
    if case["kind"] == "product":
        M, dD, F, X = _product_inputs(case, seed)
        return {"kind": "product", "lib": engine.load_library(), "M": M, "dD": dD, "F": F, "X": X,
                "Rf": torch.empty_like(F), "Rs": torch.empty_like(X)}
    ds = _decks(case, seed)
    host = case.get("host", False)
    s = engine.System(ds if len(ds) > 1 else ds[0],
                      precision=engine.PREC_FP64 if case["prec"] == 64 else engine.PREC_MIXED,
                      refresh=case.get("refresh", 1), noise=engine.NOISE_HOST if host else engine.NOISE_PHILOX,
                      seed=seed + 5)
    if case["kind"] == "step" and case["n"] >= 4000:
        s.autotune(True)   # as the benchmark runs these sizes
    st = {"kind": case["kind"], "sys": s, "k": case.get("k", 1), "turn": 0, "checkpoint": case.get("checkpoint", 1)}
    if host or case["kind"] == "drift":
        # sixteen Gaussian vectors, then their negatives, so that repeated
        # passes do not push the beads one way
        per = st["k"] * (2 if case["kind"] == "igt" else 1)
        g = _gauss(case, seed, s.n3, 16 * per).reshape(16, per * s.n3)
        st["gauss"] = np.concatenate([g, -g])
    if case["kind"] == "adjoint":
        st["x0"] = s.get_coord()
        st["pairs"], st["targets"] = _loss(case, seed, s.n)
    return st


def run(st):
    kind = st["kind"]
    if kind == "product":
        M = st["M"]
        p = ctypes.c_void_p
        rc = st["lib"].bdb_stored_matvec_noalloc(
            p(M.data_ptr()), st["F"].numel(), M.shape[1], p(st["dD"].data_ptr()), p(st["F"].data_ptr()),
            p(st["X"].data_ptr()), 0.017, p(st["Rf"].data_ptr()), p(st["Rs"].data_ptr()),
            p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise engine.BDBError(rc, st["lib"].bdb_last_error().decode())
        return {"Rf": st["Rf"], "Rs": st["Rs"]}
    s = st["sys"]
    g = None
    if "gauss" in st:
        g = st["gauss"][st["turn"] % len(st["gauss"])]
        st["turn"] += 1
    if kind == "step":
        flag = s.step(st["k"], g)
        return {"coord": s.get_coord(), "flag": flag}
    if kind == "igt":
        flag = s.step_igt(st["k"], g)
        return {"coord": s.get_coord(), "flag": flag}
    if kind == "drift":
        return {"Rf": s.compute_Rf(), "Rs": s.compute_r(g)}
    if kind == "forces":
        F, E, flag, counts = s.compute_forces()
        return {"F": F, "E": E, "flag": flag, "pairs_c": counts[0], "pairs_lj": counts[1]}
    # a training step: the gradient at the given starting positions
    s.set_coord(st["x0"])
    loss, gx, gp = s.adjoint(st["k"], st["checkpoint"], st["pairs"], st["targets"])
    return {"loss": loss, "grad_coord": gx, "grad_params": gp}


# ------------------------------------------------------------------- work

def work(case):
    kind = case["kind"]
    if kind == "product":
        n3 = 3 * case["n"]
        return {"bytes": 4.0 * n3 * n3 + 8.0 * 5 * n3, "flops": 3.0 * n3 * n3}
    el = 8.0 if case["prec"] == 64 else 4.0
    n, k = case["n"], case.get("k", 1)
    n3 = 3.0 * n
    if case.get("replicas"):
        lo, hi = case["n"], case["n_max"]
        beads = case["replicas"] * (lo + hi) / 2
        pairs = case["replicas"] * ((hi ** 3 - lo ** 3) / (3.0 * max(1, hi - lo))) / 2
    else:
        beads, pairs = n, n * (n - 1) / 2
    io = 8.0 * beads * (4 + 4)
    near = 60.0   # pairs within the cutoffs, per bead
    force = 40.0 * near / 2 * beads
    if kind == "forces":
        return {"bytes": 8.0 * beads * (4 + 1 + 2 + 3), "flops": 40.0 * beads * (173 / 2 if case["ewald"] else 20)}
    # a tile, its products with two vectors both ways and its squared rows
    tile = 47.0 + 2 * 45
    if case.get("ewald") and case["ewald"] != "none":
        m = 4.0 / 3.0 * math.pi * case["r"] ** 3
        # per lattice image and reciprocal pair: the scalar functions (20) and
        # the six tile entries (12); half of the reciprocal sphere
        tile += 32.0 * m + 14.0 * m / 2
    if case["hydro"] == "geyer":
        steps = k if kind == "step" else 2
        return {"bytes": io + steps * 8.0 * beads * 12, "flops": steps * (tile * pairs + force)}
    chol = n3 ** 3 / 3 + 30.0 * pairs
    if kind == "step":
        # the factor of the call's refreshes, and the stored products of each step
        ref = k / case["refresh"]
        return {"bytes": io + k * el * n3 * n3 + ref * el * n3 * n3, "flops": ref * chol + k * (3.0 * n3 * n3 + force)}
    if kind == "igt":
        return {"bytes": io + 5 * el * n3 * n3, "flops": 2 * chol + 4.0 * n3 * n3 + force}
    # adjoint: the forward pass, its repetition and, per step backwards, the
    # factor and two triangular solves of a full matrix
    back = chol + 2 * n3 ** 3 + 200.0 * pairs
    return {"bytes": io + k * 6 * el * n3 * n3, "flops": k * (3 * chol + 2 * n3 ** 3 + 200.0 * pairs + 2 * force)}


def tolerance(case):
    """About four times what the paths were seen to differ from exact() by on
    B200. The positions are compared whole (extents of ~100 A against steps
    of ~0.1 A), so their bounds are the steps' errors times that ratio."""
    kind = case["kind"]
    if kind == "product":
        return {"rel": 1e-15, "max": 1e-14}   # seen 2.5e-16, 8e-16
    if kind in ("step", "igt"):
        if case["prec"] == 64:
            return {"rel": 1e-15, "max": 1e-13}   # seen 9e-17, 4e-16
        return {"rel": 1.2e-8, "max": 1e-7} if case.get("ewald") else {"rel": 2e-9, "max": 2e-8}   # seen 3e-9; 5e-10
    if kind == "drift":
        if case["prec"] == 64:
            return {"rel": 2e-14, "max": 1.2e-13}   # seen 5e-15, 3e-14
        return {"rel": 2.4e-6, "max": 1.2e-5}   # seen 5.6e-7, 2.9e-6
    if kind == "forces":
        return {"rel": 5e-15, "max": 1e-13}   # seen 1.3e-15, 2e-14
    if case["prec"] == 64:
        return {"rel": 2e-14, "max": 2e-13}   # seen 5e-15
    return {"rel": 6e-6, "max": 1e-5}   # seen 1.4e-6 (of the four scale factors), 2e-6


# ------------------------------------------------------------------ exact

def _philox_gauss(seed, stream, n3):
    """Unit Gaussians of the device stream: Philox-4x32-10 (Salmon, Moraes,
    Dror, Shaw, SC'11), counter (pair, stream), and Box-Muller."""
    np_ = (n3 + 1) // 2
    mask = np.uint64(0xFFFFFFFF)
    c = [np.arange(np_, dtype=np.uint64), np.full(np_, stream & 0xFFFFFFFF, dtype=np.uint64),
         np.full(np_, stream >> 32, dtype=np.uint64), np.full(np_, 0x42444242, dtype=np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & mask, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1),
             p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    d = [v.astype(np.float64) for v in (c[0] >> np.uint64(5), c[1] >> np.uint64(6), c[2] >> np.uint64(5),
                                        c[3] >> np.uint64(6))]
    u0, u1 = (d[0] * 67108864.0 + d[1] + 0.5) / 2.0 ** 53, (d[2] * 67108864.0 + d[3]) / 2.0 ** 53
    r = np.sqrt(-2 * np.log(u0))
    z = np.empty(2 * np_)
    z[0::2], z[1::2] = r * np.cos(2 * np.pi * u1), r * np.sin(2 * np.pi * u1)
    return z[:n3]


class _Exact:
    """One bead system in 64-bit torch, on the GPU where there is one."""

    def __init__(self, case, system, keys):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.case, self.s = case, system
        self.n = len(system["pos"])
        self.dt = f32(keys["dt"])
        self.kT = KB * f32(keys["T"])
        vis = f32(keys["visc"]) * f32(keys["vfactor"])
        self.Dii, self.Dij = KB_6PI * f32(keys["T"]) / vis, KB_8PI * f32(keys["T"]) / vis
        self.L, self.a = system["L"], system["radius"]
        self.elec = keys["elec"] == "yes"
        self.kappa, self.eps_c, self.gamma = f32(0.1), f32(78.54), f32(331.842)
        self.q = self.t(system["q"])
        self.x = self.t(system["pos"])

    def t(self, a):
        return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=self.dev)

    # forces, energies, pair counts; sc: scale factors (LJ epsilon, LJ sigma, bond H, Debye length)
    def forces(self, x, sc=None, rows=2048):
        sc = [1.0] * 4 if sc is None else sc
        n, (half, eps) = self.n, self.s["lj"]
        F, e_c, e_lj, n_c, n_lj = [], 0.0, 0.0, 0, 0
        j = torch.arange(n, device=self.dev)
        sig = 2 * half * sc[1]
        kap = self.kappa / sc[3]
        g = self.gamma / self.eps_c
        lim = 12.0 if self.s["bonds"] else f32(1.122462) * 2 * half
        for b in range(0, n, rows):
            i = torch.arange(b, min(n, b + rows), device=self.dev)
            d = x[i][:, None, :] - x[None, :, :]
            if self.L:
                d = d - self.L * torch.floor(d / self.L + 0.5)
            rr = (d * d).sum(dim=2)
            other = i[:, None] != j[None, :]
            r = torch.sqrt(torch.where(other, rr, torch.ones_like(rr)))
            act = other
            if self.s["bonds"]:
                act = act & ((i[:, None] - j[None, :]).abs() != 1)
            near_c, near_lj = other & (r <= 12.0) & self.elec, other & (r <= lim)
            n_c, n_lj = n_c + int(near_c.sum()), n_lj + int(near_lj.sum())
            qq = self.q[i][:, None] * self.q[None, :]
            ex = torch.exp(-kap * r)
            m_c, m_lj = (near_c & act).double(), (near_lj & act).double()
            s6 = (sig / r) ** 6
            lj = 4.0 * eps * sc[0]
            Fm = m_c * g * qq * (1 + kap * r) * ex / (r * r) + m_lj * lj * 6 * s6 * (2 * s6 - 1) / r
            F.append((Fm / r)[:, :, None].mul(d).sum(dim=1))
            e_c = e_c + (m_c * g * qq * ex / r).sum() / 2
            e_lj = e_lj + (m_lj * lj * s6 * (s6 - 1)).sum() / 2
        F = torch.cat(F)
        e_b = 0.0
        if self.s["bonds"]:
            d = x[1:] - x[:-1]
            r = d.norm(dim=1)
            H, m2, r0, rm = 10.0 * sc[2], 1e20, 3.8, 1e10
            f = (H * (r0 - r) / (1 - r * r / m2) / r)[:, None] * d
            z = torch.zeros((1, 3), dtype=torch.float64, device=self.dev)
            F = F + torch.cat([z, f]) - torch.cat([f, z])
            # the energy's logarithms cancel to 1e-20 of their arguments at
            # this rmax: no 64-bit value
            e_b = None
        return F, (e_b, e_lj, e_c), (n_c // 2, n_lj // 2)

    # tiles D_ij as (n, n) planes {xx, yy, zz, xy, xz, yz}, diagonal tiles zero
    def planes(self, x):
        n, a = self.n, self.a
        eye = torch.eye(n, dtype=torch.bool, device=self.dev)
        d = [x[:, k][:, None] - x[:, k][None, :] for k in range(3)]
        rr = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
        rr = torch.where(eye, torch.ones_like(rr), rr)
        r = torch.sqrt(rr)
        over = (r < 2 * a) & ~eye
        far = (~eye).double()
        ab = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
        # far field and overlap form
        A, B = self.Dij / r * (1 + 2 * a * a / rr / 3), self.Dij / r * (1 - 2 * a * a / rr)
        Ao, Bo = self.Dii / a * (1 - 9 * r / (32 * a)), self.Dii / a * 3 * r / (32 * a)
        ewald = self.case.get("ewald")
        if not ewald:
            A, B = torch.where(over, Ao, A) * far, torch.where(over, Bo, B) * far / rr
            return [B * d[p] * d[q] + (A if p == q else 0.0) for p, q in ab], self.Dii / a
        ov = over.double()
        A, B = (Ao - A) * ov, (Bo - B) * ov / rr
        t = [B * d[p] * d[q] + (A if p == q else 0.0) for p, q in ab]
        e, self_d = self._lattice(d, eye, ewald)
        return [(t[k] + self.Dii * e[k]) * far for k in range(6)], self_d

    def _lattice(self, d, eye, method):
        """The Ewald sums over |m| <= R of Beenakker (J. Chem. Phys. 85, 1581
        (1986)) or Smith (Physica A 150, 474 (1988)) with BD_BOX's constants."""
        L, a, R, sp = self.L, self.a, self.case["r"], math.sqrt(math.pi)
        ab = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
        s2 = a * a
        ball = [(h, f, g) for h in range(-R, R + 1) for f in range(-R, R + 1) for g in range(-R, R + 1)
                if h * h + f * f + g * g <= R * R]
        fl = np.float32
        two, four2, six = float(2 * fl(PIF)), float(4 * fl(PIF) * fl(PIF)), float(6 * fl(PIF))
        out = [torch.zeros_like(d[0]) for _ in range(6)]
        if method == "beenakker":
            al = 1.77245385090551602729 / L
            sp = 1.77245385090551602729
            a3, a5, a7 = al ** 3, al ** 5, al ** 7
        else:
            al = 1.77245385090551602729
            sp = 1 / 0.5641895835
        for m in ball:
            v = [d[k] * (-1 if method == "beenakker" else 1) + L * m[k] for k in range(3)]
            if method == "smith":
                v = [d[k] / L + m[k] for k in range(3)]
            rr = v[0] ** 2 + v[1] ** 2 + v[2] ** 2
            live = (rr != 0).double()
            rr = torch.where(rr == 0, torch.ones_like(rr), rr)
            r = torch.sqrt(rr)
            ex, er = torch.exp(-al * al * rr) / sp, torch.erfc(al * r)
            if method == "beenakker":
                A = (al * s2 / rr + 14 * a3 * s2 - 4.5 * al - 20 * a5 * s2 * rr + 3 * a3 * rr + 4 * a7 * s2 * rr * rr) * ex \
                    + er * (0.75 / r + 0.5 * s2 / (r * rr))
                B = (-3 * al * s2 / rr - 2 * a3 * s2 + 1.5 * al + 16 * a5 * s2 * rr - 3 * a3 * rr
                     - 4 * a7 * s2 * rr * rr) * ex + er * (0.75 / r - 1.5 * s2 / (r * rr))
            else:
                so, sq = er / r, (er + 2 * al * r * ex) / (r * rr)
                preO, preQ = 0.75 / L, 0.5 * s2 / L ** 3
                A = preO * so + preQ * sq
                B = preO * (so + 2 * al * ex) + preQ * (-3 * sq - 4 * al ** 3 * ex)
            A, B = A * live, B * live / rr
            for k, (p, q) in enumerate(ab):
                out[k] += B * v[p] * v[q] + (A if p == q else 0.0)
        w = [d[k] / L for k in range(3)]
        pif2 = float(-(fl(PIF) * fl(PIF)))
        for m in ball:
            kk = float(m[0] ** 2 + m[1] ** 2 + m[2] ** 2)
            if kk == 0 or m < (0, 0, 0):
                continue   # k and -k contribute alike: one of the two, doubled
            cs = torch.cos(two * (w[0] * m[0] + w[1] * m[1] + w[2] * m[2]))
            e = [c / math.sqrt(kk) for c in m]
            if method == "beenakker":
                k2, ia2 = kk * four2, 1 / (al * al)
                P = (1 + ia2 * k2 / 4 * (1 + ia2 * k2 / 2)) * six * math.exp(-ia2 * k2 / 4) / k2
                f = 2 * (P - s2 * k2 / 3 * P) / L ** 3
                for k, (p, q) in enumerate(ab):
                    out[k] += f * ((1.0 if p == q else 0.0) - e[p] * e[q]) * cs
            else:
                mp = pif2 / (al * al)
                w_ = math.exp(mp * kk)
                ci = 4 * 0.75 / L * w_ / (PIF * kk)
                ce = ci * (mp * kk - 1) + s2 / L ** 3 * float(4 * fl(PIF)) * w_
                for k, (p, q) in enumerate(ab):
                    out[k] += (ce * e[p] * e[q] + (ci if p == q else 0.0)) * cs
        # self tile
        own = out[0][0, 0]
        if method == "beenakker":
            c = -6 * al / sp + 40 * a3 * a * a / (3 * sp)
        else:
            c3 = (al * a / L) ** 3 / sp / 3
            c = -(0.75 / L * 1.5 * al * a / sp / L + 0.5 * a * a / L ** 3 * c3)
        return out, [float(self.Dii / a + self.Dii * (c + out[k][0, 0])) for k in range(3)]

    def dense(self, t):
        n = self.n
        D = torch.stack([torch.stack([t[0], t[3], t[4]], -1), torch.stack([t[3], t[1], t[5]], -1),
                         torch.stack([t[4], t[5], t[2]], -1)], 1).reshape(3 * n, 3 * n)
        return D + self.Dii / self.a * torch.eye(3 * n, dtype=torch.float64, device=self.dev)

    def tea(self, x, F, g):
        """(Rf, Rs) without a stored tensor: D.F and the Geyer-Winter noise."""
        t, own = self.planes(x)
        own = own if isinstance(own, list) else [own] * 3
        rows = ((0, 3, 4), (3, 1, 5), (4, 5, 2))
        d, n3 = self.Dii / self.a, 3 * self.n
        X = g * math.sqrt(2 * self.dt / d)
        mul = lambda v: torch.stack([sum(t[r[k]] @ v[:, k] for k in range(3)) for r in rows], 1)  # noqa: E731
        Rf = self.dt / self.kT * (mul(F) + F * self.t(own))
        eps = sum((1.0 if k < 3 else 2.0) * float(t[k].sum()) for k in range(6)) / 2
        eps = min(1.0, eps / n3 / (n3 - 1) * 2)
        aa = (n3 - 1) * eps * eps - (n3 - 2) * eps
        beta = 0.5 if abs(aa) < f32(1e-7) else (1 - math.sqrt(1 - aa)) / aa
        C = torch.stack([sum((t[r[k]] ** 2).sum(dim=1) for k in range(3)) for r in rows], 1) / d
        Rs = (beta * mul(X) + d * X) / torch.sqrt(1 + C * beta * beta / d)
        return Rf, Rs

    def wrap(self, x):
        return x - self.L * torch.floor(x / self.L + 0.5) if self.L else x


def _gaussians(case, seed, n3, count):
    if case.get("host"):
        return list(_gauss(case, seed, n3, 16 * count)[:count])
    return [_philox_gauss(seed + 5, k, n3) for k in range(count)]


def exact(case, seed):
    if case["kind"] == "product":
        M, dD, F, X = _product_inputs(case, seed)
        n3 = F.numel()
        M = M[:, :n3].double()
        U = torch.triu(M, 1)
        return {"Rf": 0.017 * (U @ F + U.T @ F + dD * F), "Rs": torch.tril(M) @ X}
    systems, keys = _inputs(case, seed)
    sys_ = [_Exact(case, s, keys) for s in systems]
    n3 = 3 * sum(e.n for e in sys_)
    kind = case["kind"]
    if kind == "forces":
        F, (e_b, e_lj, e_c), counts = sys_[0].forces(sys_[0].x)
        if systems[0]["bonds"]:
            E = None
        else:
            E = np.zeros(9)
            E[6], E[7] = float(e_lj), float(e_c)
        return {"F": F.reshape(-1).cpu().numpy(), "E": E, "flag": None, "pairs_c": None, "pairs_lj": None}
    if kind == "adjoint":
        return _exact_adjoint(case, seed, sys_[0])
    if kind == "drift":
        e = sys_[0]
        F, _, _ = e.forces(e.x)
        g = e.t(_gauss(case, seed, n3, 16)[0]).reshape(-1, 3)
        Rf, Rs = e.tea(e.x, F, g)
        return {"Rf": Rf.reshape(-1).cpu().numpy(), "Rs": Rs.reshape(-1).cpu().numpy()}
    k = case["k"]
    gs = _gaussians(case, seed, n3, k * (2 if kind == "igt" else 1))
    out, first = [], 0
    for e in sys_:
        sl = slice(first, first + 3 * e.n)
        first += 3 * e.n
        x, Lc = e.x, None
        sq = math.sqrt(2 * e.dt)
        for i in range(k):
            F, _, _ = e.forces(x)
            if case["hydro"] == "geyer":
                Rf, Rs = e.tea(x, F, e.t(gs[i][sl]).reshape(-1, 3))
                x = e.wrap(x + Rf + Rs)
                continue
            c = e.dt / e.kT
            if kind == "igt":
                D = e.dense(e.planes(x)[0])
                d1 = c * (D @ F.reshape(-1))
                xp = x + (d1 + torch.linalg.cholesky(D) @ (sq * e.t(gs[2 * i][sl]))).reshape(-1, 3)
                Dp = e.dense(e.planes(xp)[0])
                d2 = c * (Dp @ e.forces(xp)[0].reshape(-1))
                Lc = torch.linalg.cholesky((D + Dp) / 2)
                x = x + ((d1 + d2) / 2 + Lc @ (sq * e.t(gs[2 * i + 1][sl]))).reshape(-1, 3)
                continue
            if Lc is None or i % case["refresh"] == 0:
                D = e.dense(e.planes(x)[0])
                Lc = torch.linalg.cholesky(D)
            x = x + (c * (D @ F.reshape(-1)) + Lc @ (sq * e.t(gs[i][sl]))).reshape(-1, 3)
        out.append(np.column_stack([x.cpu().numpy(), np.full(e.n, e.a)]))
    return {"coord": np.concatenate(out), "flag": None}


def _exact_adjoint(case, seed, e):
    """The same gradient by torch's automatic differentiation in 64 bits."""
    pairs, targets = _loss(case, seed, e.n)
    x0 = e.x.clone().requires_grad_(True)
    sc = torch.ones(4, dtype=torch.float64, device=e.dev, requires_grad=True)
    c, sq, x = e.dt / e.kT, math.sqrt(2 * e.dt), x0
    for k in range(case["k"]):
        F, _, _ = e.forces(x, sc)
        D = e.dense(e.planes(x)[0])
        X = sq * e.t(_philox_gauss(seed + 5, k, 3 * e.n))
        x = x + (c * (D @ F.reshape(-1)) + torch.linalg.cholesky(D) @ X).reshape(-1, 3)
    p = torch.as_tensor(pairs.astype(np.int64), device=e.dev)
    r = (x[p[:, 1]] - x[p[:, 0]]).norm(dim=1)
    loss = ((r - e.t(targets)) ** 2).mean()
    gx, gp = torch.autograd.grad(loss, [x0, sc])
    return {"loss": float(loss.detach()), "grad_coord": gx.cpu().numpy(), "grad_params": gp.cpu().numpy()}
