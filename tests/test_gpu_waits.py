"""What a bounded wait on the device that runs out reports."""
import numpy as np
import pytest
import torch
import wait_limits

pytestmark = pytest.mark.gpu


def _declare(lib, *names):
    from feab200 import _lib as L
    for n in names:
        f = getattr(lib, n)
        f.restype, f.argtypes = L.SIGNATURES[n]


def test_eigensolver(tmp_path, monkeypatch):
    from feab200 import _lib as L
    from feab200.pod import PodBasis
    lib = wait_limits.build(tmp_path, "feab_gram.cu")
    if lib is None:
        pytest.skip("no nvcc")
    _declare(lib, "feab_symeig_jacobi")
    rng = np.random.default_rng(1)
    B = rng.standard_normal((64, 64))
    A = torch.as_tensor(B @ B.T).cuda()
    w, V = torch.zeros(64, dtype=torch.float64, device="cuda"), torch.zeros((64, 64), dtype=torch.float64, device="cuda")
    sweeps = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = lib.feab_symeig_jacobi(L.dptr(A), 64, L.dptr(w), L.dptr(V), 40, L.dptr(sweeps), L.stream_ptr(A.device))
    assert rc == L.FEAB_OK and int(sweeps) == -1 and bool(w.isnan().all()) and bool(V.isnan().all())
    # without vectors nothing waits
    rc = lib.feab_symeig_jacobi(L.dptr(A), 64, L.dptr(w), None, 40, L.dptr(sweeps), L.stream_ptr(A.device))
    assert rc == L.FEAB_OK and int(sweeps) > 0 and not bool(w.isnan().any())
    # the callers that read the result raise
    monkeypatch.setattr(L.lib, "feab_symeig_jacobi", lib.feab_symeig_jacobi)
    with pytest.raises(RuntimeError, match="timed out"):
        PodBasis().fit(torch.as_tensor(rng.standard_normal((500, 64))).cuda(), n_modes=3)
    monkeypatch.undo()
    assert PodBasis().fit(torch.as_tensor(rng.standard_normal((500, 64))).cuda(), n_modes=3).V.shape == (500, 3)
