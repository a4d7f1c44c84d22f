"""The resident PCG (whole solve in one kernel) at the edges of its range, against the step kernels
on the CSR: sizes on both sides of one cluster (48 slices of 32 nodes), of one row per thread (5
slices per SM) and of the largest operator it takes (8 slices per SM); shuffled node numbers, whose
column offsets need 32 bits and whose rows refer to more of p than shared memory holds; a solve that
needs more iterations than one launch runs."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _operator(nx, ny, nz, shuffle=False, size=(2.0, 0.4, 0.4)):
    from feab200.device import DeviceMesh
    nodes, el = O.box_mesh(*size, nx, ny, nz)
    if shuffle:
        new = np.random.default_rng(3).permutation(len(nodes))     # old node -> new node
        moved = np.empty_like(nodes)
        moved[new] = nodes
        nodes, el = moved, new[el]
    dm = DeviceMesh(nodes, el)
    return dm.assemble(dm.element_stiffness(O.D_solid3d(210e9, 0.3)), dm.pattern(O.fixed_dofs_on_plane(nodes, 0, 0.0)),
                       want32=False)


def _check(op, tol, precision="fp64", **kw):
    from feab200.device import pcg_solve
    b = torch.as_tensor(np.random.default_rng(7).standard_normal(op.n)).cuda()
    x, info = pcg_solve(op, b, tol=tol, precision=precision, **kw)
    again, info2 = pcg_solve(op, b, tol=tol, precision=precision, **kw)
    assert info.status == 0 and info.iters == info2.iters and torch.equal(x, again)
    p = op.pattern
    row = torch.repeat_interleave(torch.arange(op.n, device="cuda"), (p.row_ptr[1:] - p.row_ptr[:-1]).long())
    xc = x[p.col_idx.long()]
    Kx = torch.zeros_like(b).index_add_(0, row, op.vals64 * xc)
    size = torch.zeros_like(b).index_add_(0, row, (op.vals64 * xc).abs())
    bn = float(b.norm())
    # the recurrence's residual is below tol; the true one differs by the rounding of each step's
    # update of r and x, at most (row terms + steps) eps |K| |x|
    assert float((b - Kx).norm()) <= (tol + EPS * (81 + 4 * info.iters) * float(size.norm()) / bn) * bn
    want, ref = pcg_solve(op, b, tol=tol, precision="fp64", layout="csr", use_dinv=kw.get("use_dinv", True))
    return info, ref


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 4), (20, 4, 4), (31, 6, 6), (33, 6, 6), (43, 9, 10), (72, 18, 17),
                                   (73, 19, 17), (84, 20, 20), (88, 21, 20)])
def test_resident_solve(shape, precision):
    op = _operator(*shape)
    info, ref = _check(op, 1e-9, precision)
    if precision == "fp64":   # the same recurrence, other sums (mixed: other values and residual replacements)
        assert abs(info.iters - ref.iters) <= 2 + ref.iters // 25


def test_shuffled_nodes_fit_with_wide_columns():
    op = _operator(64, 16, 16, shuffle=True)
    _check(op, 1e-9)


def test_shuffled_nodes_beyond_shared_memory():
    op = _operator(80, 20, 20, shuffle=True)
    info, ref = _check(op, 1e-9)
    assert abs(info.iters - ref.iters) <= 2 + ref.iters // 25


def test_more_iterations_than_one_launch():
    op = _operator(600, 1, 1, size=(60.0, 0.1, 0.1))
    info, _ = _check(op, 1e-6, use_dinv=False)
    assert info.iters > 4096 and info.graph_launches > 1


def test_start_vector_and_iteration_limit():
    from feab200 import _lib as L
    from feab200.device import pcg_solve
    op = _operator(20, 4, 4)
    b = torch.as_tensor(np.random.default_rng(8).standard_normal(op.n)).cuda()
    x, info = pcg_solve(op, b, tol=1e-10)
    half, cut = pcg_solve(op, b, tol=1e-10, maxiter=info.iters // 2)
    assert cut.status == L.FEAB_NOT_CONVERGED and cut.iters == info.iters // 2
    same, warm = pcg_solve(op, b, tol=1e-10, x0=x)
    assert warm.status == 0 and warm.iters <= 2
    rest, more = pcg_solve(op, b, tol=1e-10, x0=half)
    assert more.status == 0 and float((rest - x).norm() / x.norm()) < 1e-6


def test_solves_after_memory_went_back_to_the_driver():
    """A cached graph outlives the workspace it was captured with."""
    from feab200.batched import block_pcg
    from feab200.device import pcg_solve
    for shape in ((20, 4, 4), (20, 4, 5), (20, 4, 4)):
        op = _operator(*shape)
        b = torch.as_tensor(np.random.default_rng(9).standard_normal(op.n)).cuda()
        x, info = pcg_solve(op, b, tol=1e-9, layout="csr", lanes_per_group=8)
        X, res = block_pcg(op, [0, op.n], b[:, None].repeat(1, 16), [16], tol=1e-9, tune=False)
        assert info.status == 0 and (res.status == 0).all()
        assert float((X - x[:, None]).norm() / X.norm()) < 1e-6
        del op, b, x, X
        torch.cuda.empty_cache()
