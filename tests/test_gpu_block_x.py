"""X of the block PCG where the last step's part comes in behind the loop: solves cut off by the iteration limit, and
columns that are done before the first step or before the others, against single solves on the CSR."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


def _operator(nx, ny, nz):
    from feab200.device import DeviceMesh
    nodes, el = O.box_mesh(2.0, 0.4, 0.4, nx, ny, nz)
    dm = DeviceMesh(nodes, el)
    return dm.assemble(dm.element_stiffness(O.D_solid3d(210e9, 0.3)), dm.pattern(O.fixed_dofs_on_plane(nodes, 0, 0.0)),
                       want32=False)


@pytest.mark.parametrize("k,tiles", [(1, False), (2, False), (4, True), (8, True), (16, True), (16, False), (64, True)])
@pytest.mark.parametrize("steps", [1, 3])
def test_cut_off_solve(k, tiles, steps):
    from feab200.batched import block_pcg
    from feab200.device import pcg_solve
    op = _operator(17, 5, 6)
    cols = max(1, k - 1)
    B = torch.zeros((op.n, k), dtype=torch.float64, device="cuda")
    B[:, :cols] = torch.as_tensor(np.random.default_rng(k).standard_normal((op.n, cols))).cuda()
    if cols > 2:
        B[:, 1] = 0.0                     # done before the first step
    X, res = block_pcg(op, [0, op.n], B, [cols], tol=1e-12, maxiter=steps, max_groups=64, tile_width=k, node_tiles=tiles)
    for c in range(cols):
        want, info = pcg_solve(op, B[:, c].contiguous(), tol=1e-12, maxiter=steps, layout="csr")
        assert int(res.iters[0, c]) == info.iters
        # the same few steps with other orders of summation: some 100 roundings each, and a step multiplies
        # an error in the direction by at most |D^-1 K| |K^-1 D| of the steps so far (below 1e4 here)
        assert float((X[:, c] - want).norm()) <= 1e4 * 100 * steps * 2.0 ** -53 * float(want.norm())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_columns_that_end_at_different_steps(precision):
    from feab200.batched import block_pcg
    op = _operator(17, 5, 6)
    rng = np.random.default_rng(2)
    B = torch.as_tensor(rng.standard_normal((op.n, 16))).cuda()
    B[:, 3] = 1.0                         # smooth: another step count
    tol = 1e-9
    X, res = block_pcg(op, [0, op.n], B, [16], tol=tol, precision=precision, max_groups=64, tile_width=16,
                       node_tiles=True)
    assert not res.status.any()
    p = op.pattern
    row = torch.repeat_interleave(torch.arange(op.n, device="cuda"), (p.row_ptr[1:] - p.row_ptr[:-1]).long())
    for c in range(16):
        xc = X[p.col_idx.long(), c]
        Kx = torch.zeros_like(B[:, c]).index_add_(0, row, op.vals64 * xc)
        size = torch.zeros_like(Kx).index_add_(0, row, (op.vals64 * xc).abs())
        steps = int(res.iters[0, c])
        # the recurrence's residual is below tol; the true one differs by the rounding of each step's update
        bound = tol * float(B[:, c].norm()) + 2.0 ** -53 * (81 + 4 * steps) * float(size.norm())
        assert float((B[:, c] - Kx).norm()) <= bound
