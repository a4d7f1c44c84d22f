"""The banded Cholesky's factor and solves at the edges of its tiles, through the C entry points: band
matrices of 0, 1, 2 and more tile bands, ragged last tiles, bands as wide as the matrix."""
import ctypes as C

import numpy as np
import pytest
import scipy.linalg as sl
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu


def _band_matrix(n, bw, seed):
    """A symmetric band matrix whose diagonal dominates (condition below 10), as CSR."""
    rng = np.random.default_rng(seed)
    d = [rng.uniform(-1.0, 1.0, n - k) for k in range(1, bw + 1)]
    off = sp.diags(d, list(range(1, bw + 1)), shape=(n, n)) if bw else sp.csr_matrix((n, n))
    A = off + off.T
    row = np.asarray(abs(A).sum(axis=1)).ravel()
    return sp.csr_matrix(A + sp.diags(1.2 * row.max() + 1.0 + rng.uniform(0.0, 1.0, n)))


def _assembled(A, bw):
    """(feab_band, its storage, stream) of the CSR matrix A with its rows in order."""
    from feab200 import _lib as L
    dev = torch.device("cuda")
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a, dtype=dt)).to(dev)  # noqa: E731
    n = A.shape[0]
    rp, ci, va = t(A.indptr, np.int32), t(A.indices, np.int32), t(A.data, np.float64)
    csr = L.CSR(n, n, int(A.nnz), rp.data_ptr(), ci.data_ptr(), va.data_ptr(), None, None)
    iperm = torch.arange(n, dtype=torch.int32, device=dev)
    storage = torch.full((int(L.lib.feab_band_bytes(n, bw)),), 77, dtype=torch.uint8, device=dev)
    band = L.Band(0, 0, 0, 0, storage.data_ptr())
    st = L.stream_ptr(dev)
    assert L.lib.feab_band_assemble(C.byref(csr), L.dptr(iperm), bw, C.byref(band), st) == L.FEAB_OK
    return band, storage, st


def _solve(band, b, st):
    from feab200 import _lib as L
    bt = torch.zeros(64 * band.n_tiles, dtype=torch.float64, device="cuda")
    bt[:len(b)] = torch.as_tensor(b).cuda()
    x, w = torch.empty_like(bt), torch.empty_like(bt)
    assert L.lib.feab_band_solve(C.byref(band), L.dptr(bt), L.dptr(x), L.dptr(w), st) == L.FEAB_OK
    x = x.cpu().numpy()
    assert not x[len(b):].any()
    return x[:len(b)]


@pytest.mark.parametrize("n,bw", [(1, 0), (63, 0), (64, 20), (65, 1), (64, 63), (128, 64), (130, 65), (200, 128),
                                  (500, 129), (449, 192), (700, 699), (1500, 257)])
def test_band_factor_and_solve(n, bw):
    from feab200 import _lib as L
    A = _band_matrix(n, bw, 100 * n + bw)
    band, storage, st = _assembled(A, bw)
    piv = (C.c_double * 2)()
    assert L.lib.feab_band_cholesky(C.byref(band), piv, st) == L.FEAB_OK
    full = np.linalg.cholesky(A.toarray())
    # a backward-stable factorisation of a matrix with condition number below 10: n eps each way
    tol = 40.0 * max(n, 64) * 2.0 ** -53
    assert abs(piv[0] / np.diag(full).min() ** 2 - 1.0) < tol and abs(piv[1] / np.diag(full).max() ** 2 - 1.0) < tol
    nt, bands = band.n_tiles, band.bands
    tiles = storage[256:256 + nt * (bands + 1) * 4096 * 8].view(torch.float64).reshape(nt, bands + 1, 64, 64).cpu().numpy()
    got = np.zeros((64 * nt, 64 * nt))
    for i in range(nt):
        for d in range(min(bands, i) + 1):
            got[64 * i:64 * i + 64, 64 * (i - d):64 * (i - d) + 64] = tiles[i, d]
    assert np.abs(got[:n, :n] - full).max() < tol * np.abs(full).max()
    rng = np.random.default_rng(n)
    for _ in range(2):
        b = rng.standard_normal(n)
        want = sl.cho_solve((full, True), b)
        assert np.linalg.norm(_solve(band, b, st) - want) < tol * np.linalg.norm(want)


@pytest.mark.parametrize("bands", [8, 9, 16, 17, 33, 65, 128, 129])
def test_wide_band_solve(bands):
    """Both sides of each form of the solve: a few diagonals, the outermost at the band's edge."""
    from feab200 import _lib as L
    bw = 64 * bands
    n = bw + 200
    rng = np.random.default_rng(bands)
    off = sp.diags([rng.uniform(-1.0, 1.0, n - k) for k in (1, 65, bw // 2 + 3, bw)], [1, 65, bw // 2 + 3, bw],
                   shape=(n, n))
    A = sp.csr_matrix(off + off.T + sp.diags(10.0 + rng.uniform(0.0, 1.0, n)))
    band, storage, st = _assembled(A, bw)
    assert band.bands == bands
    piv = (C.c_double * 2)()
    assert L.lib.feab_band_cholesky(C.byref(band), piv, st) == L.FEAB_OK
    b = rng.standard_normal(n)
    x = _solve(band, b, st)
    # condition number below 10, as above
    assert np.linalg.norm(b - A @ x) < 40.0 * n * 2.0 ** -53 * np.linalg.norm(b)
