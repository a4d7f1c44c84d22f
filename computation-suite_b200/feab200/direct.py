"""Direct solve of the reduced system on the GPU: a banded tile Cholesky factorisation.

The reference's default static solve (FESystem.solve_static with method=None on a sparse
system) is FESystem._sparse_lu_solve (fea_engine/src/fea_engine/solver.py:1681-1724): SuperLU's
splu of K_ff, a singularity test on its pivots (min |U_ii| < tol max |U_ii|, tol 1e-10), then
lu.solve.  K_ff is SPD, so its LU factorisation without pivoting is the Cholesky factorisation
K_ff = L L^T with U_ii = L_ii^2; the same pivot test is made on the Cholesky pivots.

The free DOFs are renumbered node by node, layer by layer along the axis with most layers of nodes or in
reverse Cuthill-McKee order of the node graph (on the host, as SuperLU's column ordering is in the
reference), so that the band of the renumbered K_ff is narrow; the band is factored and solved on the GPU with the
feab_band_* kernels (64 x 64 tiles).  The factor of an operator is computed once and reused for
every right-hand side.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from . import _lib as L

PIVOT_TOL = 1e-10        # the reference's _sparse_lu_solve default
TILE = 64


def node_order(op):
    """Reverse Cuthill-McKee order of the node row groups of op (int64 array of group ids).
    The node graph is formed on the device from each group's column list; its edges go to the
    host for SciPy's reverse_cuthill_mckee."""
    import scipy.sparse as sp
    from scipy.sparse.csgraph import reverse_cuthill_mckee
    p = op.pattern
    dev = op.vals64.device
    gp = p.group_ptr.to(torch.int64)
    G = gp.numel() - 1
    sizes = gp[1:] - gp[:-1]
    row_group = torch.repeat_interleave(torch.arange(G, device=dev), sizes)
    rp = p.row_ptr.to(torch.int64)
    starts, lens = rp[gp[:-1]], rp[gp[:-1] + 1] - rp[gp[:-1]]
    src = torch.repeat_interleave(torch.arange(G, device=dev), lens)
    off = torch.arange(int(lens.sum()), device=dev) - torch.repeat_interleave(torch.cumsum(lens, 0) - lens, lens)
    nbr = row_group[p.col_idx.to(torch.int64)[torch.repeat_interleave(starts, lens) + off]]
    keep = torch.ones_like(nbr, dtype=torch.bool)
    keep[1:] = (nbr[1:] != nbr[:-1]) | (src[1:] != src[:-1])   # the DOFs of one neighbour are adjacent
    src, nbr = src[keep].cpu().numpy(), nbr[keep].cpu().numpy()
    g = sp.csr_matrix((np.ones(src.size, np.int8), (src, nbr)), shape=(G, G))
    return np.asarray(reverse_cuthill_mckee(g, symmetric_mode=True), dtype=np.int64)


def coordinate_order(op, coords):
    """Node row groups sorted by their node's coordinate along the mesh's longest extent (then
    the other two): on an elongated mesh the band is about one cross-section of nodes wide."""
    X = np.asarray(coords, dtype=float)
    fm = op.pattern.free_map
    dof_of_row = torch.nonzero(fm >= 0).flatten().cpu().numpy()
    gp = op.pattern.group_ptr.cpu().numpy().astype(np.int64)
    key = X[dof_of_row[gp[:-1]] // 3]
    ax = np.argsort(np.ptp(key, axis=0))          # ascending extent: the longest axis is last
    return np.lexsort((key[:, ax[0]], key[:, ax[1]], key[:, ax[2]])).astype(np.int64)


def layer_order(op, coords, sample=2048):
    """Node row groups sorted layer by layer along the axis with most layers, within a layer by the other
    two, and the number of layers: the coordinates in units of the mesh's own spacing along each
    axis (the mean length of the longer edges of some nodes), rounded.  Unlike the coordinates
    themselves, whole layers stay together when the nodes are not exactly in their planes, so the
    band is one cross-section of nodes wide and not two; and the smallest cross-section is the one across
    the axis of most layers, whatever its length.  On the operator's device."""
    order, n_layers = _layers(op, coords, sample)
    return order, int(n_layers[2])


def _spread(G, count, dev):
    """`count` of the indices 0 .. G - 1, evenly spread, the last among them.  In FP64: FP32 numbers are whole
    multiples of 2 from 2^24 on, and the last could be G."""
    return torch.linspace(0, G - 1, count, dtype=torch.float64, device=dev).to(torch.int64)


def _layers(op, coords, sample=2048):
    """The order of layer_order, and the layers along the three axes, ascending."""
    p = op.pattern
    dev = op.vals64.device
    gp, rp = p.group_ptr.to(torch.int64), p.row_ptr.to(torch.int64)
    G = gp.numel() - 1
    dof = torch.nonzero(p.free_map >= 0).flatten()
    key = torch.as_tensor(np.ascontiguousarray(coords, dtype=float)).to(dev)[dof[gp[:-1]] // 3]
    some = _spread(G, min(G, int(sample)), dev)
    start = rp[gp[some]]
    lens = rp[gp[some] + 1] - start
    src = torch.repeat_interleave(torch.arange(some.numel(), device=dev), lens)
    col = torch.arange(src.numel(), device=dev) + (start - torch.cumsum(lens, 0) + lens)[src]
    nbr = torch.searchsorted(gp, p.col_idx[col].to(torch.int64), right=True) - 1
    d = (key[nbr] - key[some[src]]).abs()
    long = d > 0.5 * d.amax(0)
    h = torch.where(long, d, torch.zeros_like(d)).sum(0) / long.sum(0).clamp_min(1)
    lo = key.amin(0)
    q = ((key - lo) / torch.where(h > 0, h, torch.ones_like(h))).round().to(torch.int64)
    n_layers = (q.amax(0) + 1).cpu().numpy()
    ax = np.argsort(n_layers, kind="stable")      # fewest first: neighbours within a layer stay closest
    code = (q[:, ax[2]] * int(n_layers[ax[1]]) + q[:, ax[1]]) * int(n_layers[ax[0]]) + q[:, ax[0]]
    return torch.argsort(code, stable=True), n_layers[ax]


def dof_permutation(op, order):
    """iperm (old reduced row -> new row, int32 device tensor) for the node order `order`."""
    dev = op.vals64.device
    gp = op.pattern.group_ptr.to(torch.int64)
    order = torch.as_tensor(order).to(dev)
    sz = gp[1:] - gp[:-1]
    first = torch.empty_like(sz)
    first[order] = torch.cumsum(sz[order], 0) - sz[order]
    group = torch.repeat_interleave(torch.arange(sz.numel(), device=dev), sz, output_size=op.n)
    return (first[group] + torch.arange(op.n, device=dev) - gp[group]).to(torch.int32)


def narrowest_order(op, coords, width):
    """(iperm, bandwidth, name) of the node order with the narrowest band; width(iperm) is an order's band.
    coords: the mesh's node coordinates (N, 3), if known: the ordering in layers is then tried first, and
    unless its band is known to be about as narrow as any, the ordering by coordinates and reverse
    Cuthill-McKee beside it."""
    best = None

    def consider(name, order):
        nonlocal best
        iperm = dof_permutation(op, order)
        bw = int(width(iperm))
        if best is None or bw < best[1]:
            best = (iperm, bw, name)

    done = False
    if coords is not None:
        order, n_layers = _layers(op, coords)
        consider("axis", order)
        # No order's band is narrower than the rows divided by the steps between the two nodes farthest
        # apart.  On a whole box these are the layers of its longest axis; within half as much again (a layer
        # and the line of nodes beside the next one's nearest) the other orders are not tried: reverse
        # Cuthill-McKee takes 30 ms of host time at 96x24x24 elements and is 1.2 to 2.7 times as wide on boxes.
        # A box has a node in every place of the lattice and every one of its 27 neighbours; a bent, branched,
        # slit or graded mesh lacks some, and its farthest nodes may be many layers apart.
        nl = n_layers.astype(np.float64)
        G = op.pattern.n_groups
        box = G >= 0.99 * np.prod(nl) > 0 and op.pattern.nnz >= 0.99 * (op.n / G) ** 2 * np.prod(3 * nl - 2)
        done = box and best[1] <= 1.5 * op.n / nl[2] + 6
    if not done:
        if coords is not None:
            consider("axis", coordinate_order(op, coords))
        consider("rcm", node_order(op))
    return best


class BandCholesky:
    """K_ff = L L^T on the device, in the renumbered order.  Raises MemoryError when the band
    would take more than `max_fraction` of the device's free memory."""

    def __init__(self, op, coords=None, max_fraction=0.6):
        """coords: the mesh's node coordinates (N, 3), if known, for the order (see narrowest_order)."""
        self.op = op
        dev = op.vals64.device
        if op.pattern.group_ptr is None:
            raise ValueError("the direct solve needs node row groups (an assembled K_ff)")
        csr = op.csr_struct()
        scratch = torch.zeros(2, dtype=torch.int32, device=dev)

        def width(iperm):
            bw = C.c_int32(0)
            rc = L.lib.feab_band_width(C.byref(csr), L.dptr(iperm), L.dptr(scratch), C.byref(bw), L.stream_ptr(dev))
            L.raise_for(rc, "band width")
            return bw.value

        self.iperm, self.bandwidth, self.ordering = narrowest_order(op, coords, width)
        nbytes = int(L.lib.feab_band_bytes(op.n, self.bandwidth))
        free, _ = torch.cuda.mem_get_info(dev)
        if nbytes > max_fraction * free:
            raise MemoryError(f"banded Cholesky of n={op.n} (bandwidth {self.bandwidth}) needs {nbytes / 1e9:.1f} GB, "
                              f"more than {max_fraction:.0%} of the {free / 1e9:.1f} GB free on the device")
        self.storage = torch.empty(nbytes, dtype=torch.uint8, device=dev)
        self.band = L.Band(0, 0, 0, 0, self.storage.data_ptr())
        rc = L.lib.feab_band_assemble(C.byref(csr), L.dptr(self.iperm), self.bandwidth, C.byref(self.band),
                                      L.stream_ptr(dev))
        L.raise_for(rc, "band assembly")
        piv = (C.c_double * 2)()
        rc = L.lib.feab_band_cholesky(C.byref(self.band), piv, L.stream_ptr(dev))
        self.pivots = (float(piv[0]), float(piv[1]))
        if rc == L.FEAB_NOT_SPD:
            raise np.linalg.LinAlgError("banded Cholesky: a pivot <= 0 -- K_ff is not SPD")
        L.raise_for(rc, "banded Cholesky")
        self.padded = int(self.band.n_tiles) * TILE
        self._error = torch.zeros(1, dtype=torch.int32, pin_memory=True)     # set by a solve whose wait timed out

    @property
    def near_singular(self):
        """The reference's test on the factor's pivots: min < 1e-10 max."""
        lo, hi = self.pivots
        return not (lo >= PIVOT_TOL * hi)

    def solve(self, b):
        """x = K_ff^{-1} b (b: (n,) host or device array; returns an FP64 device tensor).  Asynchronous.
        Where a bounded wait times out on the device x is NaN, and check() or the next solve raises."""
        self._raise_if_timed_out()
        op = self.op
        dev = op.vals64.device
        b = torch.as_tensor(b, dtype=torch.float64).to(dev).reshape(-1)
        if b.numel() != op.n:
            raise ValueError(f"b must have {op.n} entries, got {b.numel()}")
        bp = torch.zeros(self.padded, dtype=torch.float64, device=dev)
        bp[self.iperm.long()] = b
        xp = torch.empty_like(bp)
        work = torch.empty_like(bp)
        rc = L.lib.feab_band_solve_flag(C.byref(self.band), L.dptr(bp), L.dptr(xp), L.dptr(work), L.dptr(self._error),
                                        L.stream_ptr(dev))
        L.raise_for(rc, "banded Cholesky solve")
        return xp[self.iperm.long()]

    def check(self):
        """Waits for the solves on the current stream; raises when a bounded wait of one timed out."""
        torch.cuda.current_stream(self.op.vals64.device).synchronize()
        self._raise_if_timed_out()

    def _raise_if_timed_out(self):
        if int(self._error[0]):
            self._error.zero_()
            L.raise_for(L.FEAB_CUDA_ERROR, "banded Cholesky solve: a bounded wait timed out on the device")
