"""POD basis of a snapshot panel on the GPU (rom_engine/src/rom_engine/pod.py:100-176).

``PodBasis.fit`` keeps the reference's signature and rank rule (n_modes / energy_threshold,
_select_rank pod.py:163-176).  The FP64 economy SVD of the reference (pod.py:140-147) is
replaced by the method of snapshots: the 64 x 64 Gram matrix X^T X, its FP64 eigenvalues by a
Jacobi solver on a cluster of three CTAs (feab_symeig_jacobi), singular values sqrt(lambda), and modes
U = X V / sigma.  Three Gram kernels; the default ``gram="auto"`` takes the int8 one for FP32
snapshots and the FP64 one for FP64 snapshots (whose values carry more bits than seven 7-bit
digits keep):

* ``gram="int8"``: the tensor cores with exact products (seven signed 7-bit digits per
  value, tcgen05.mma kind::i8 with int32 accumulation, FP64 combination; feab_gram_int8) --
  FP64-level accuracy at tensor-core speed; at 1,382,976 x 64 its singular values agree with the
  FP64 Gram's to 1.4e-9 and it runs in 0.81 ms against 1.2 ms;
* ``gram="fp64"``: FP64 accumulation on the CUDA cores (feab_gram_fp64), which keeps trailing
  singular values of fast-decaying snapshot spectra (sigma_10 / sigma_1 ~ 1e-4 for elastic
  solutions) to FP32-input accuracy;
* ``gram="bf16x3"``: the tensor cores (split-bf16 x3 products, FP32 accumulate, FP64 across
  chunks; feab_gram_bf16x3) -- resolves eigenvalues down to ~1e-6 of the largest, i.e. the
  leading singular values only.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from . import _lib as L
from .device import cuda_device
from .panel import panel_small, panel_small_f32

MAX_SNAPSHOTS = 64


def gram_bf16x3(X, check=True, workspace=None):
    """G = X^T X (FP64, 64 x 64) of a device panel X (n x 64, FP32, row major).  With
    check=False the call stays asynchronous and returns (G, error_flag): the device flag is
    non-zero if a bounded wait timed out, and the caller reads it later."""
    X = X.contiguous()
    if X.dtype != torch.float32 or X.ndim != 2 or X.shape[1] != MAX_SNAPSHOTS:
        raise ValueError("gram_bf16x3 needs an (n, 64) float32 device panel")
    dev = X.device
    n = X.shape[0]
    wbytes = int(L.lib.feab_gram_workspace_bytes(n, MAX_SNAPSHOTS))
    ws = workspace if workspace is not None and workspace.numel() >= wbytes else torch.empty(wbytes, dtype=torch.uint8,
                                                                                               device=dev)
    G = torch.empty((MAX_SNAPSHOTS, MAX_SNAPSHOTS), dtype=torch.float64, device=dev)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    rc = L.lib.feab_gram_bf16x3(L.dptr(X), n, MAX_SNAPSHOTS, L.dptr(G), L.dptr(ws), wbytes, L.dptr(err),
                                L.stream_ptr(dev))
    L.raise_for(rc, "gram_bf16x3")
    if not check:
        return G, err
    if int(err.item()):
        raise RuntimeError("gram_bf16x3: a bounded wait timed out on the device")
    return G


def gram_int8(X, check=True, workspace=None):
    """G = X^T X (FP64, 64 x 64) of a device panel X (n x 64, FP32, row major) on the tensor cores
    with exact integer digit products (feab_gram_int8): FP64-level accuracy.  With check=False
    the call stays asynchronous and returns (G, error_flag) as gram_bf16x3 does."""
    X = X.contiguous()
    if X.dtype != torch.float32 or X.ndim != 2 or X.shape[1] != MAX_SNAPSHOTS:
        raise ValueError("gram_int8 needs an (n, 64) float32 device panel")
    dev = X.device
    n = X.shape[0]
    wbytes = int(L.lib.feab_gram_workspace_bytes(n, MAX_SNAPSHOTS))
    ws = workspace if workspace is not None and workspace.numel() >= wbytes else torch.empty(wbytes, dtype=torch.uint8,
                                                                                               device=dev)
    G = torch.empty((MAX_SNAPSHOTS, MAX_SNAPSHOTS), dtype=torch.float64, device=dev)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    rc = L.lib.feab_gram_int8(L.dptr(X), n, MAX_SNAPSHOTS, L.dptr(G), L.dptr(ws), wbytes, L.dptr(err),
                              L.stream_ptr(dev))
    L.raise_for(rc, "gram_int8")
    if not check:
        return G, err
    if int(err.item()):
        raise RuntimeError("gram_int8: a bounded wait timed out on the device")
    return G


def gram_fp64(X, workspace=None):
    """G = X^T X (FP64, 64 x 64) accumulated in FP64 for a device panel X (n x 64, FP32 or
    FP64, row major).  Asynchronous on the current stream."""
    X = X.contiguous()
    if X.dtype not in (torch.float32, torch.float64) or X.ndim != 2 or X.shape[1] != MAX_SNAPSHOTS:
        raise ValueError("gram_fp64 needs an (n, 64) float32 or float64 device panel")
    dev = X.device
    n = X.shape[0]
    wbytes = int(L.lib.feab_gram_workspace_bytes(n, MAX_SNAPSHOTS))
    ws = workspace if workspace is not None and workspace.numel() >= wbytes else torch.empty(wbytes, dtype=torch.uint8,
                                                                                               device=dev)
    G = torch.empty((MAX_SNAPSHOTS, MAX_SNAPSHOTS), dtype=torch.float64, device=dev)
    rc = L.lib.feab_gram_fp64(L.dptr(X), X.element_size(), n, MAX_SNAPSHOTS, L.dptr(G), L.dptr(ws), wbytes,
                              L.stream_ptr(dev))
    L.raise_for(rc, "gram_fp64")
    return G


def symeig(G, vectors=True, max_sweeps=40):
    """Eigenvalues (descending) and eigenvectors of a symmetric FP64 device matrix (k <= 64).  Asynchronous:
    all are NaN if a bounded wait timed out on the device (PodBasis.fit and solve_modal raise then)."""
    return _symeig(G, vectors, max_sweeps)[:2]


def _symeig(G, vectors=True, max_sweeps=40):
    """symeig's results and the device int of the sweeps, -1 after a wait that timed out."""
    k = G.shape[0]
    A = G.contiguous().clone()
    w = torch.empty(k, dtype=torch.float64, device=G.device)
    V = torch.empty((k, k), dtype=torch.float64, device=G.device) if vectors else None
    sweeps = torch.zeros(1, dtype=torch.int32, device=G.device)
    rc = L.lib.feab_symeig_jacobi(L.dptr(A), k, L.dptr(w), L.dptr(V), int(max_sweeps), L.dptr(sweeps),
                                  L.stream_ptr(G.device))
    L.raise_for(rc, "symeig_jacobi")
    return w, V, sweeps


def _check_symeig(sweeps):
    if int(sweeps.item()) < 0:
        raise RuntimeError("symeig_jacobi: a bounded wait timed out on the device")


def _select_rank(S, n_modes, energy_threshold):
    candidates = []
    if n_modes is not None:
        candidates.append(min(int(n_modes), len(S)))
    if energy_threshold is not None:
        energy = S ** 2
        total = np.sum(energy)
        if total <= 0:
            candidates.append(1)
        else:
            cum = np.cumsum(energy) / total
            candidates.append(min(int(np.searchsorted(cum, energy_threshold) + 1), len(S)))
    return max(1, min(candidates))


class PodBasis:
    def __init__(self):
        self.V = None
        self.singular_values = None
        self.n_modes = None
        self.mass_weighted = False
        self.M = None

    def fit(self, snapshots, n_modes=None, energy_threshold=None, M=None, device=None, gram="auto"):
        if n_modes is None and energy_threshold is None:
            raise ValueError("fit() needs at least one of n_modes, energy_threshold")
        if M is not None:
            raise NotImplementedError("PodBasis.fit: mass-weighted POD is not on the GPU path")
        dev = snapshots.device if torch.is_tensor(snapshots) and snapshots.is_cuda else cuda_device(device)
        X = torch.as_tensor(snapshots).to(dev)
        if X.ndim != 2:
            raise ValueError(f"snapshots must be 2-D (n_dof, n_snapshots), got shape {tuple(X.shape)}")
        n, k = X.shape
        if k > MAX_SNAPSHOTS:
            raise NotImplementedError(f"PodBasis.fit: at most {MAX_SNAPSHOTS} snapshots per panel on the GPU path")
        if gram not in ("auto", "fp64", "bf16x3", "int8"):
            raise ValueError("gram must be 'auto', 'fp64', 'bf16x3' or 'int8'")
        if gram == "auto":
            gram = "int8" if X.dtype == torch.float32 else "fp64"
        dt = torch.float64 if gram == "fp64" else torch.float32
        if k == MAX_SNAPSHOTS and X.dtype == dt and X.is_contiguous() and X.data_ptr() % 16 == 0:
            Xp = X                                           # a whole panel as the Gram kernels read it
        else:
            Xp = torch.zeros((n, MAX_SNAPSHOTS), dtype=dt, device=dev)
            Xp[:, :k] = X.to(dt)
        G = {"bf16x3": gram_bf16x3, "int8": gram_int8, "fp64": gram_fp64}[gram](Xp)
        w, V, sweeps = _symeig(G)
        S = torch.sqrt(torch.clamp(w[: min(k, n)], min=0.0))
        S_host = S.cpu().numpy()
        if np.isnan(S_host).any():                           # NaN snapshots, or no result
            _check_symeig(sweeps)
        r = _select_rank(S_host, n_modes, energy_threshold)
        Vk = V[:k, :r]                                       # eigenvectors of the k x k Gram block
        inv = torch.where(S[:r] > 0, 1.0 / S[:r], torch.zeros_like(S[:r]))
        # method of snapshots: U = X V / sigma, as one panel product (V scaled by 1 / sigma first)
        W = (Vk * inv[None, :]).contiguous()
        if X.dtype == torch.float32 and X.stride(1) == 1 and X.stride(0) >= k:
            self.V = panel_small_f32(X, W)                   # the values widen to FP64 in the kernel
        else:
            self.V = panel_small(X.to(torch.float64), W)
        self.singular_values = S_host
        self.n_modes = r
        return self

    def energy_captured(self):
        energy = self.singular_values ** 2
        total = np.sum(energy)
        return 1.0 if total <= 0 else float(np.sum(energy[: self.n_modes]) / total)
