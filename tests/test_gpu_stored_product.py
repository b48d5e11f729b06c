"""The stored-matrix products (k_strip_mv, k_mv_finish) at sizes around the
edges of their strips (32 rows) and tiles (128 columns), through the
allocation-free entry point (FP32 matrix) and an FP64 system. Padding columns
hold NaN: nothing outside the matrix may be read into a sum."""
import ctypes as C

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

from bd_box_b200 import decks, engine  # noqa: E402


@pytest.mark.parametrize("n3", [1, 3, 31, 32, 33, 127, 128, 129, 160, 255, 385, 1000, 3071, 3072])
@pytest.mark.parametrize("null_stream", [False, True])
def test_noalloc_product_at_edges(n3, null_stream):
    import torch
    rng = np.random.default_rng(n3)
    ld = (n3 + 3) // 4 * 4 + 8
    Mh = np.full((n3, ld), np.nan, dtype=np.float32)
    Mh[:, :n3] = rng.standard_normal((n3, n3))
    dD, F, X = rng.standard_normal((3, n3))
    M = Mh[:, :n3].astype(np.float64)
    U = np.triu(M, 1)
    want_f = 0.3 * (U @ F + U.T @ F + dD * F)
    want_s = np.tril(M) @ X
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (Mh, dD, F, X)]
    out = torch.full((2, n3), float("nan"), dtype=torch.float64, device="cuda")
    lib = engine.load_library()
    torch.cuda.synchronize()
    stream = None if null_stream else C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        rc = lib.bdb_stored_matvec_noalloc(t[0].data_ptr(), n3, ld, t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(),
                                           0.3, out[0].data_ptr(), out[1].data_ptr(), stream)
        assert rc == 0, lib.bdb_last_error().decode()
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    # sums of 3N FP64 products of entries ~1: 2 sqrt(3N) ulps is generous
    bound = 4e-16 * np.sqrt(n3) * (np.abs(M).sum(axis=1).max() + 1)
    assert np.abs(got[0] - want_f).max() <= bound
    assert np.abs(got[1] - want_s).max() <= bound


@pytest.mark.parametrize("n,warps", [(11, 16), (43, 8), (43, 64), (86, 16), (128, 32), (171, 1)])
def test_fp64_stored_products(n, warps, deck_dir):
    import pyoracle
    d = decks.read_deck(decks.write_chain_deck(deck_dir, f"sp{n}", n, seed=n, hydro="cholesky"))
    o = pyoracle.Oracle(d)
    g = np.random.default_rng(n).standard_normal(3 * n)
    dt = d.prm["dt"]
    s = engine.System(d, precision=engine.PREC_FP64, noise=engine.NOISE_HOST)
    s.set_tuning(mv_warps_per_sm=warps)
    df = o.df(o.forces()[0], dt)
    D = s.compute_D()
    rs = np.linalg.cholesky(D) @ (g * np.sqrt(2 * dt))
    assert np.abs(s.compute_Rf() - df).max() <= 1e-12 * np.abs(df).max()
    assert np.abs(s.compute_r(g) - rs).max() <= 1e-12 * np.abs(rs).max()


@pytest.mark.parametrize("n3", [1, 2, 3, 30, 33, 127, 129, 255, 1023, 3069, 3071])
def test_noalloc_matrix_ends_with_its_last_element(n3):
    """A caller's matrix may end with the last column of its last row; beyond
    it nothing may be read."""
    import torch
    rng = np.random.default_rng(n3)
    ld = (n3 + 3) // 4 * 4
    flat = np.full(n3 * ld, np.nan, dtype=np.float32)
    M = rng.standard_normal((n3, n3)).astype(np.float32)
    for r in range(n3):
        flat[r * ld:r * ld + n3] = M[r]
    dD, F, X = rng.standard_normal((3, n3))
    M = M.astype(np.float64)
    U = np.triu(M, 1)
    t = [torch.from_numpy(a).cuda() for a in (flat[:(n3 - 1) * ld + n3].copy(), dD, F, X)]
    out = torch.full((2, n3), float("nan"), dtype=torch.float64, device="cuda")
    lib = engine.load_library()
    torch.cuda.synchronize()
    rc = lib.bdb_stored_matvec_noalloc(t[0].data_ptr(), n3, ld, t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(),
                                       1.0, out[0].data_ptr(), out[1].data_ptr(), None)
    assert rc == 0, lib.bdb_last_error().decode()
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    bound = 4e-16 * np.sqrt(n3) * (np.abs(M).sum(axis=1).max() + 1)   # as above
    assert np.abs(got[0] - (U @ F + U.T @ F + dD * F)).max() <= bound
    assert np.abs(got[1] - np.tril(M) @ X).max() <= bound
