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


def _cantilever(shape):
    import feab200
    mesh = feab200.box_mesh(2.0, 0.4, 0.4, *shape)
    fs = feab200.FESystem(mesh, feab200.Hex8Solid3D(), sparse=True)
    fs.assemble_stiffness(feab200.D_solid3d(feab200.Material(E=1.0, nu=0.3)), vectorized=True)
    fs.fix_dofs(mesh.nodes_on_plane(0, 0.0), (0, 1, 2))
    fs.add_nodal_force(mesh.nodes_on_plane(0, 2.0), 2, 1.0)
    return fs


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


@pytest.mark.parametrize("shape", [(6, 2, 2), (24, 8, 8), (40, 12, 12)])
def test_band_solve(tmp_path, monkeypatch, shape):
    """Bands of 1, 5 and 9 tiles: clusters of 8 and of 16 CTAs."""
    import ctypes as C
    from feab200 import _lib as L
    from feab200 import torch_sparse_solver as ts
    lib = wait_limits.build(tmp_path, "feab_band.cu")
    if lib is None:
        pytest.skip("no nvcc")
    _declare(lib, "feab_band_solve", "feab_band_solve_flag")
    fs = _cantilever(shape)
    mesh = fs.mesh
    want = np.asarray(fs.solve_static())
    fac = fs.reduced_operator(want32=False).direct_factor(coords=mesh.nodes)
    st = L.stream_ptr(torch.device("cuda"))
    b = torch.ones(fac.op.n, dtype=torch.float64, device="cuda")
    x = fac.solve(b)
    fac.check()
    with monkeypatch.context() as m:
        m.setattr(L.lib, "feab_band_solve_flag", lib.feab_band_solve_flag)
        assert bool(fac.solve(b).isnan().any())
        with pytest.raises(L.FeabError, match="timed out"):
            fac.check()
        fac.check()                                                # said once
        fac.solve(b)
        torch.cuda.synchronize()
        with pytest.raises(L.FeabError, match="timed out"):
            fac.solve(b)
        with pytest.raises(L.FeabError, match="timed out"):
            fs.solve_static()
        with pytest.raises(L.FeabError, match="timed out"):
            ts.fesystem_solve_static_torch(fs, method="dense")
    # without a flag of its own a solve sets the header's
    header = fac.storage[32:36].view(torch.int32)
    bp = torch.zeros(fac.padded, dtype=torch.float64, device="cuda")
    bp[:fac.op.n] = 1.0
    xp, work = torch.empty_like(bp), torch.empty_like(bp)
    for fn, flag in ((L.lib.feab_band_solve, 0), (lib.feab_band_solve, 1)):
        assert fn(C.byref(fac.band), L.dptr(bp), L.dptr(xp), L.dptr(work), st) == L.FEAB_OK
        assert int(header) == flag and bool(xp.isnan().any()) == bool(flag)
    assert torch.equal(fac.solve(b), x)
    assert np.array_equal(np.asarray(fs.solve_static()), want)


def test_ring_of_the_sliced_pcg(tmp_path, monkeypatch):
    """44,649 nodes: beyond the resident solve, so that step A streams through its ring."""
    from feab200 import _lib as L
    lib = wait_limits.build(tmp_path, "feab_pcg.cu", "feab_sell.cu", "feab_scan.cu")
    if lib is None:
        pytest.skip("no nvcc")
    _declare(lib, "feab_pcg_solve")
    fs = _cantilever((40, 32, 32))
    for precision, tol in (("fp64", 1e-10), ("mixed", 1e-9)):
        want = np.asarray(fs.solve_static(method="pcg", precision=precision, tol=tol))
        with monkeypatch.context() as m:
            m.setattr(L.lib, "feab_pcg_solve", lib.feab_pcg_solve)
            with pytest.raises(L.FeabError):
                fs.solve_static(method="pcg", precision=precision, tol=tol)
            assert fs.last_solve_info.status == L.FEAB_CUDA_ERROR
        assert np.array_equal(np.asarray(fs.solve_static(method="pcg", precision=precision, tol=tol)), want)


def test_pair_records_of_the_block_pcg(tmp_path, monkeypatch):
    """One problem that takes several chunks and two that take one: all report the error, none hangs."""
    import oracle as O
    from feab200 import _lib as L
    from feab200.batched import ProblemBatch, block_pcg
    lib = wait_limits.build(tmp_path, "feab_block_pcg.cu")
    if lib is None:
        pytest.skip("no nvcc")
    _declare(lib, "feab_block_pcg_solve")
    probs = []
    rng = np.random.default_rng(3)
    for sh in ((30, 6, 5), (3, 2, 2), (2, 1, 1)):
        X, el = O.box_mesh(1.0, 0.5, 0.3, *sh)
        probs.append((X, el, O.D_solid3d(5.0, 0.3), O.fixed_dofs_on_plane(X, 0, 0.0), rng.standard_normal((3 * len(X), 16))))
    b = ProblemBatch(probs)
    op, B = b.assemble(), b.rhs_panel()
    kw = dict(max_groups=8, tune=False, node_tiles=True)
    for precision in ("fp64", "mixed"):
        for K in (8, 16):
            Bk = B[:, :K].contiguous()
            args = (op, b.row_bounds, Bk, [K, 3, K])
            want, res = block_pcg(*args, tol=1e-9, precision=precision, tile_width=K, **kw)
            assert (res.status == 0).all()
            with monkeypatch.context() as m:
                m.setattr(L.lib, "feab_block_pcg_solve", lib.feab_block_pcg_solve)
                with pytest.raises(L.FeabError):
                    block_pcg(*args, tol=1e-9, precision=precision, tile_width=K, **kw)
            got, res = block_pcg(*args, tol=1e-9, precision=precision, tile_width=K, **kw)
            assert (res.status == 0).all() and torch.equal(got, want)
