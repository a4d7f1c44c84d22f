"""The one-block eigensolver over its sizes and scales, and the panel product over its tile edges."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("k", [1, 2, 3, 5, 31, 32, 33, 63, 64])
@pytest.mark.parametrize("kind", ["spd", "indefinite", "clustered", "diagonal", "huge", "tiny", "zero"])
def test_symeig(k, kind):
    from feab200.pod import symeig
    rng = np.random.default_rng(k)
    A = rng.standard_normal((k, k))
    if kind in ("spd", "huge", "tiny"):
        A = A @ A.T * {"spd": 1.0, "huge": 1e200, "tiny": 1e-200}[kind]
    elif kind == "indefinite":
        A = A + A.T
    elif kind == "clustered":
        Q = np.linalg.qr(A)[0]
        A = (Q * np.where(np.arange(k) % 3 == 0, 2.0, 1.0)) @ Q.T
    elif kind == "diagonal":
        A = np.diag(rng.permutation(k) - 1.0)
    else:
        A = np.zeros((k, k))
    A = 0.5 * (A + A.T)
    w, V = symeig(torch.as_tensor(A).cuda())
    w, V = w.cpu().numpy(), V.cpu().numpy()
    size = np.linalg.norm(A) if kind not in ("huge", "tiny") else np.abs(A).max() * k
    # ten sweeps of rotations, each a relative error of a few eps on the entries it turns
    tol = 40.0 * max(k, 4) * EPS
    assert np.all(np.diff(w) <= 0.0)
    assert np.abs(w - np.sort(np.linalg.eigvalsh(A))[::-1]).max() <= tol * size
    assert np.abs(V.T @ V - np.eye(k)).max() <= tol
    assert np.abs(A @ V - V * w).max() <= tol * size


@pytest.mark.parametrize("n,k,m", [(1, 1, 1), (5, 3, 64), (127, 64, 7), (128, 64, 8), (129, 7, 9), (1000, 64, 16),
                                   (1000, 33, 17), (40000, 64, 64)])
def test_panel_small(n, k, m):
    from feab200.panel import panel_small, panel_small_f32
    g = torch.Generator(device="cuda").manual_seed(n + k + m)
    Y = torch.randn((n, 70), generator=g, dtype=torch.float64, device="cuda")[:, 2:2 + k]    # rows 70 apart
    V = torch.randn((k, m), generator=g, dtype=torch.float64, device="cuda")
    for Yi, fn in ((Y, panel_small), (Y.float(), panel_small_f32)):
        Z = fn(Yi, V)
        Yd = Yi.double()
        bound = 2 * k * EPS * (Yd.abs() @ V.abs())
        assert Z.shape == (n, m) and bool(((Z - Yd @ V).abs() <= bound).all())


@pytest.mark.parametrize("k", [17, 64])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_fit_does_not_depend_on_the_layout_of_the_snapshots(k, dtype):
    from feab200.pod import PodBasis
    g = torch.Generator(device="cuda").manual_seed(k)
    wide = torch.randn((3001, k + 5), generator=g, dtype=dtype, device="cuda")
    X = wide[:, 3:3 + k].contiguous()
    base = PodBasis().fit(X, n_modes=5)
    before = X.clone()
    for other in (wide[:, 3:3 + k], X.t().contiguous().t(), X.cpu()):
        p = PodBasis().fit(other, n_modes=5)
        assert np.array_equal(p.singular_values, base.singular_values) and torch.equal(p.V, base.V)
    assert torch.equal(X, before)


@pytest.mark.parametrize("k", [1, 3, 32, 63, 64])
@pytest.mark.parametrize("where", ["first", "middle", "all"])
def test_symeig_writes_every_output_where_a_value_is_nan(k, where):
    """A diagonal matrix with NaN among its entries needs no rotation: its entries come out, each once, and
    the unit vectors in the same order."""
    from feab200 import _lib as L
    d = np.random.default_rng(k).permutation(k) + 1.0
    d[{"first": slice(0, 1), "middle": slice(k // 3, k // 3 + 2), "all": slice(None)}[where]] = np.nan
    A = torch.as_tensor(np.diag(d)).cuda()
    w = torch.full((k,), 1e9, dtype=torch.float64, device="cuda")
    V = torch.full((k, k), 1e9, dtype=torch.float64, device="cuda")
    assert L.lib.feab_symeig_jacobi(L.dptr(A), k, L.dptr(w), L.dptr(V), 40, None, L.stream_ptr(A.device)) == L.FEAB_OK
    w, V = w.cpu().numpy(), V.cpu().numpy()
    assert np.array_equal(np.sort(w), np.sort(d), equal_nan=True)
    assert np.array_equal(np.sort(V, axis=0)[-1], np.ones(k)) and np.array_equal(V.sum(0), np.ones(k))
    assert np.array_equal(d[V.argmax(0)], w, equal_nan=True)
