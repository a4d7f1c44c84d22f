"""The sliced PCG step through the ring of bulk copies (operators beyond the resident solve's 8 slices per SM) against
the step kernels on the CSR: sizes just past that limit, with a last slice that is full, short or of one group, with
fewer slices than warps and with more than one slice per warp, and nodes of which only some DOFs are free."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _operator(nx, ny, nz, partial=False):
    from feab200.device import DeviceMesh
    nodes, el = O.box_mesh(2.0, 0.4, 0.4, nx, ny, nz)
    fixed = O.fixed_dofs_on_plane(nodes, 0, 0.0)
    if partial:     # single DOFs of nodes all over the mesh
        rng = np.random.default_rng(5)
        fixed = np.union1d(fixed, rng.choice(3 * len(nodes), len(nodes) // 5, replace=False))
    dm = DeviceMesh(nodes, el)
    return dm.assemble(dm.element_stiffness(O.D_solid3d(210e9, 0.3)), dm.pattern(fixed), want32=False)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,partial", [((79, 21, 21), False), ((81, 21, 21), False), ((85, 21, 21), True),
                                           ((160, 31, 31), False)])
def test_ring_solve(shape, partial, precision):
    from feab200.device import pcg_solve
    op = _operator(*shape, partial=partial)
    b = torch.as_tensor(np.random.default_rng(7).standard_normal(op.n)).cuda()
    tol = 1e-8
    x, info = pcg_solve(op, b, tol=tol, precision=precision)
    again, info2 = pcg_solve(op, b, tol=tol, precision=precision)
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
    if precision == "fp64":   # the same recurrence, other sums
        _, ref = pcg_solve(op, b, tol=tol, precision="fp64", layout="csr")
        assert abs(info.iters - ref.iters) <= 2 + ref.iters // 25
