"""The work that a user of feab200 has it do, as cases that can be timed.

Every case is a cantilever: a hex8 box over 2.0 x 0.4 x 0.4 m, clamped on x = 0 and loaded on its
tip, with the interior nodes moved by up to 5 % of the element size (the sizes, loads and moduli of
``feab200.cantilever``).  The kinds:

- ``static``       a new model from host arrays: FESystem, assemble_stiffness, fix_dofs,
                   solve_static(method="pcg"); with ``grad`` also the compliance gradient dC/drho;
- ``load``         one more load on a model that is kept (solve_static_device, method="pcg");
- ``direct``       a new model solved with the default solve_static(), the banded Cholesky;
- ``direct_load``  one more load on a factor that is kept;
- ``batch``        many models of uneven size, each with some load cases (ProblemBatch.solve);
- ``panel``        many load cases of one model (solve_static_batched);
- ``simp``         one step of a SIMP design loop: u(rho) and its backward through
                   torch.autograd, the sensitivity filter and the optimality-criteria update;
- ``stress``       nodal stress, von Mises and element stress of a displacement on the device;
- ``pod``          a POD basis of a panel of snapshots on the device.

``exact`` computes the same in FP64 with plain torch: element matrices by einsum, K applied element
by element, conjugate gradients to round-off.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "computation-suite_b200"))

import feab200  # noqa: E402
from feab200 import cantilever, topopt  # noqa: E402
from feab200.mesh import jitter_interior  # noqa: E402
from feab200.pod import PodBasis  # noqa: E402

LX, LY, LZ = 2.0, 0.4, 0.4
# A program that solves again and again keeps the device memory that it has used: the cases allocate
# from one pool, which gives nothing back to the driver between two solves.
_POOL = []
PENAL, RHO_MIN, VOLUME = 3.0, 1e-9, 0.5


# ----------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest model of the tests and of the documentation: launches and host work
        dict(name="static_20x4x4", kind="static", nx=20, ny=4, nz=4, precision="fp64", tol=1e-10, grad=False),
        # an ordinary model with odd sides, in mixed precision
        dict(name="static_37x11x9_mixed", kind="static", nx=37, ny=11, nz=9, precision="mixed", tol=1e-9, grad=False),
        # the headline workload: assembly, solve and gradient at 131,072 elements
        dict(name="step_128x32x32_mixed", kind="static", nx=128, ny=32, nz=32, precision="mixed", tol=1e-9,
             grad=True),
        # load stepping on a kept model, in FP64
        dict(name="load_64x16x16", kind="load", nx=64, ny=16, nz=16, precision="fp64", tol=1e-10),
        # the default static solve, a small odd model and a large one
        dict(name="direct_33x9x8", kind="direct", nx=33, ny=9, nz=8),
        dict(name="direct_96x24x24", kind="direct", nx=96, ny=24, nz=24),
        # another load on a kept factor
        dict(name="direct_load_64x16x16", kind="direct_load", nx=64, ny=16, nz=16),
        # models of uneven size with 4 to 16 load cases each
        dict(name="batch_64_mixed", kind="batch", problems=64, nx_max=48, ny_max=16, precision="mixed", tol=1e-9),
        # 64 load cases of one model, as for a set of snapshots
        dict(name="panel_64x16x16_64", kind="panel", nx=64, ny=16, nz=16, loads=64, precision="fp64", tol=1e-10),
        # one step of topology optimisation, forward and backward
        dict(name="simp_47x15x16", kind="simp", nx=47, ny=15, nz=16, precision="fp64", tol=1e-10),
        # the step after the solve at the headline's size
        dict(name="stress_128x32x32", kind="stress", nx=128, ny=32, nz=32),
        # 64 snapshots of the headline's 418,176 free DOFs
        dict(name="pod_418176x64", kind="pod", n=418176, snapshots=64, dtype="float32", modes=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, nx_lo, nx_hi, side_lo, side_hi):
    """An elongated box: sides of about a quarter of its length, odd ones among them."""
    nx = _log_int(rng, nx_lo, nx_hi)
    side = [min(side_hi, max(side_lo, int(round(nx * rng.uniform(0.18, 0.32))))) for _ in range(2)]
    return dict(nx=nx, ny=side[0], nz=side[1])


def draw(rng):
    kind = rng.choice(["static", "static", "load", "load", "direct", "direct_load", "batch", "panel", "simp", "stress",
                       "pod"])
    precision = rng.choice(["fp64", "mixed"])
    tol = 1e-10 if precision == "fp64" else 1e-9
    if kind == "static":
        return dict(kind=kind, precision=precision, tol=tol, grad=rng.random() < 0.5, **_box(rng, 10, 120, 3, 30))
    if kind == "load":
        return dict(kind=kind, precision=precision, tol=tol, **_box(rng, 10, 120, 3, 30))
    if kind == "direct":
        return dict(kind=kind, **_box(rng, 10, 88, 3, 22))
    if kind == "direct_load":
        return dict(kind=kind, **_box(rng, 10, 80, 3, 20))
    if kind == "batch":
        return dict(kind=kind, problems=_log_int(rng, 8, 60), nx_max=rng.randint(16, 44), ny_max=rng.randint(6, 15),
                    precision=precision, tol=tol)
    if kind == "panel":
        return dict(kind=kind, loads=_log_int(rng, 3, 64), precision=precision, tol=tol, **_box(rng, 10, 60, 3, 15))
    if kind == "simp":
        return dict(kind=kind, precision="fp64", tol=1e-10, **_box(rng, 10, 72, 3, 20))
    if kind == "stress":
        return dict(kind=kind, **_box(rng, 10, 128, 3, 32))
    return dict(kind=kind, n=_log_int(rng, 4000, 1200000), snapshots=rng.randint(12, 64),
                dtype=rng.choice(["float32", "float64"]), modes=rng.randint(4, 12))


# ----------------------------------------------------------------------------- inputs
def _mesh(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return jitter_interior(feab200.box_mesh(LX, LY, LZ, nx, ny, nz), 0.1, seed, h=(LX / nx, LY / ny, LZ / nz))


def _D(E=210e9, nu=0.3):
    return feab200.D_solid3d(feab200.Material(E=E, nu=nu))


def _tip_loads(mesh, seed, k=None):
    """Consistent loads of a random z traction per tip node, N(0, 1e6) Pa on a mean of -1e6 Pa."""
    rng = np.random.default_rng([seed, 7])
    tip = mesh.nodes_on_plane(0, LX)
    t = np.zeros((len(mesh.nodes), 1 if k is None else k))
    t[tip] = -1.0e6 + 1.0e6 * rng.standard_normal((len(tip), t.shape[1]))
    F = cantilever.nodal_tip_load(mesh, LX, t)
    return F[:, 0] if k is None else F


def _clamp(mesh):
    return mesh.nodes_on_plane(0, 0.0)


def _system(mesh, D):
    fs = feab200.FESystem(mesh, feab200.Hex8Solid3D(), sparse=True)
    fs.assemble_stiffness(D, vectorized=True)
    fs.fix_dofs(_clamp(mesh), (0, 1, 2))
    return fs


def _batch_models(case, seed):
    # the sizes are the case's, the moduli, loads and node positions the seed's
    sizes = np.random.default_rng([case["problems"], case["nx_max"], case["ny_max"]])
    rng = np.random.default_rng([seed, 11])
    out = []
    for p in range(case["problems"]):
        nx, s = int(sizes.integers(8, case["nx_max"] + 1)), int(sizes.integers(4, case["ny_max"] + 1))
        k = int(sizes.integers(4, 17))
        mesh = _mesh(dict(nx=nx, ny=s, nz=s), int(rng.integers(1 << 30)))
        D = _D(E=float(np.exp(rng.normal(np.log(210e9), 0.3))))
        F = cantilever.uniform_tip_load(mesh, LX, 1.0)[:, None] * rng.normal(0.0, 1.0e6, k)[None, :]
        out.append((mesh.nodes, mesh.elements, D, cantilever.clamped_dofs(mesh), F))
    return out


def _snapshots(case, seed):
    """Snapshots of a decaying spectrum: smooth fields with amplitudes that fall by a factor a mode."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, k = case["n"], case["snapshots"]
    x = torch.linspace(0.0, 1.0, n, dtype=torch.float64, device="cuda")
    C = torch.randn((16, k), generator=g, dtype=torch.float64, device="cuda")
    X = torch.zeros((n, k), dtype=torch.float64, device="cuda")
    for m in range(16):
        X += torch.sin((m + 1) * math.pi * x)[:, None] * (0.7 ** m * C[m])[None, :]
    X += 1e-3 * torch.randn((n, k), generator=g, dtype=torch.float64, device="cuda")
    return (1e-3 * X).to(getattr(torch, case["dtype"]))


def _displacement(mesh, seed):
    """A smooth bending field with a little noise, as a solve gives it."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.as_tensor(mesh.nodes).cuda()
    x, y, z = X[:, 0] / LX, X[:, 1] / LY, X[:, 2] / LZ
    a = 1e-3 * torch.randn(6, generator=g, dtype=torch.float64, device="cuda")
    u = torch.stack([a[0] * x * z + a[1] * x * x * y, a[2] * x * x * torch.cos(3 * z) + a[3] * y * y,
                     a[4] * x ** 3 + a[5] * torch.sin(4 * x) * z], dim=1)
    u += 1e-6 * torch.randn(u.shape, generator=g, dtype=torch.float64, device="cuda") * x[:, None]
    return u.reshape(-1).contiguous()


def _keep_memory():
    if not _POOL:
        pool = torch.cuda.MemPool()
        _POOL.extend((pool, torch.cuda.use_mem_pool(pool)))
        _POOL[1].__enter__()


def prepare(case, seed):
    _keep_memory()
    kind = case["kind"]
    s = dict(case=case)
    if kind == "batch":
        s["models"] = _batch_models(case, seed)
        s["batch"] = feab200.ProblemBatch(s["models"])
        s["batch"].assemble()
        return s
    if kind == "pod":
        s["X"] = _snapshots(case, seed)
        return s
    mesh = s["mesh"] = _mesh(case, seed)
    s["D"] = _D(E=1.0) if kind == "simp" else _D()
    if kind == "panel":
        s["F"] = _tip_loads(mesh, seed, case["loads"])
    elif kind == "simp":
        s["F"] = cantilever.uniform_tip_load(mesh, LX, -1.0)
    elif kind != "stress":
        s["F"] = _tip_loads(mesh, seed)
    rng = np.random.default_rng([seed, 13])
    s["rho"] = rng.uniform(0.3, 1.0, len(mesh.elements))
    if kind in ("load", "direct_load", "panel", "stress"):
        fs = s["system"] = _system(mesh, s["D"])
        op = fs.reduced_operator(want32=False)
        if kind == "load":
            op.sell_operator(case["precision"])
        elif kind == "direct_load":
            s["factor"] = op.direct_factor(coords=mesh.nodes)
            s["b"] = torch.as_tensor(s["F"][fs.free_dofs]).cuda()
        elif kind == "stress":
            s["U"] = _displacement(mesh, seed)
    if kind == "simp":
        fs = feab200.FESystem(mesh, feab200.Hex8Solid3D(), sparse=True)
        fs.fix_dofs(_clamp(mesh), (0, 1, 2))
        free = fs.free_dofs
        dm = fs.device_mesh
        s["problem"] = topopt.SimpProblem(dm, s["D"], free, penal=PENAL, rho_min=RHO_MIN, tol=case["tol"],
                                          precision=case["precision"])
        s["f"] = torch.as_tensor(s["F"][free]).cuda()
        s["rho_t"] = torch.as_tensor(s["rho"]).cuda().requires_grad_(True)
        s["H"] = topopt.build_filter_weights(topopt.element_centroids(dm), _radius(case))
    return s


def _radius(case):
    return 1.5 * max(LX / case["nx"], LY / case["ny"], LZ / case["nz"])


# ----------------------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "static":
        fs = _system(s["mesh"], s["D"])
        fs.F[:] = s["F"]
        U = fs.solve_static(method="pcg", tol=case["tol"], precision=case["precision"])
        out = {"u": np.asarray(U)}
        if case["grad"]:
            stack, conn = topopt.unit_stiffness_stack(fs, s["D"])
            out["dc"] = topopt.compliance_sensitivity_closed_form(stack, conn, 3, out["u"], s["rho"], PENAL, RHO_MIN)
        return out
    if kind == "load":
        fs = s["system"]
        fs.F[:] = s["F"]
        return {"u": fs.solve_static_device(method="pcg", tol=case["tol"], precision=case["precision"])}
    if kind == "direct":
        fs = _system(s["mesh"], s["D"])
        fs.F[:] = s["F"]
        return {"u": np.asarray(fs.solve_static())}
    if kind == "direct_load":
        return {"u": s["factor"].solve(s["b"])}
    if kind == "batch":
        U, _ = s["batch"].solve(tol=case["tol"], precision=case["precision"])
        return {"u": U}
    if kind == "panel":
        return {"u": feab200.solve_static_batched(s["system"], s["F"], tol=case["tol"], precision=case["precision"])}
    if kind == "simp":
        rho = s["rho_t"]
        u = s["problem"](rho, s["f"])
        c = torch.dot(s["f"], u)
        with torch.autograd.set_multithreading_enabled(False):   # backward on this thread, from the same pool
            (dc,) = torch.autograd.grad(c, rho)
        dcf = topopt.apply_sensitivity_filter(s["H"], rho.detach(), dc)
        new = topopt.oc_update(rho.detach(), dcf, VOLUME, move=0.2, rho_min_bound=1e-3)
        return {"u": u.detach(), "dc": dc, "filtered": dcf, "rho": new}
    if kind == "stress":
        fs = s["system"]
        return {"stress": fs.stress_tensor(s["U"]), "mises": fs.von_mises_tensor(s["U"]),
                "elements": fs.stress_tensor(s["U"], at="elements")}
    pod = PodBasis().fit(s["X"], n_modes=case["modes"])
    return {"sigma": pod.singular_values, "V": pod.V}


# ----------------------------------------------------------------------------- the work of a pass
def _sizes(case):
    """(elements, nodes, free DOFs, entries of K_ff) of a box clamped on one x face."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    blocks = (3 * nx - 2) * (3 * ny + 1) * (3 * nz + 1)   # pairs of neighbouring nodes off the clamped face
    return nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1), 3 * nx * (ny + 1) * (nz + 1), 9 * blocks


def _steps(case):
    """Iterations of Jacobi-PCG on these cantilevers: about ten for each element of the length."""
    return 10.0 * max(case["nx"], 3 * case["ny"], 3 * case["nz"])


def _cg(case, k=1):
    """Bytes and flops of a PCG solve of k loads: each step reads K once (8-byte values, or 6-byte
    ones in mixed precision) and passes over x, r, p and the product."""
    _, _, n, nnz = _sizes(case)
    value = 6.0 if case["precision"] == "mixed" else 8.0
    it = _steps(case)
    return it * (nnz * value + nnz / 3.0 * 2.0 + 9.0 * 8.0 * n * k), it * k * (2.0 * nnz + 12.0 * n)


def _assembly(case):
    E, N, n, nnz = _sizes(case)
    return 24.0 * N + 32.0 * E + 12.0 * nnz, E * 8.0 * 36.0 * 162.0


def work(case):
    kind = case["kind"]
    if kind == "pod":
        size = 4 if case["dtype"] == "float32" else 8
        n, k, m = case["n"], case["snapshots"], case["modes"]
        return {"bytes": n * (k * size * 2.0 + 8.0 * m), "flops": 2.0 * n * k * (k / 2.0 + m)}
    if kind == "batch":
        sizes = np.random.default_rng([case["problems"], case["nx_max"], case["ny_max"]])
        total = {"bytes": 0.0, "flops": 0.0}
        for _ in range(case["problems"]):
            nx, s = int(sizes.integers(8, case["nx_max"] + 1)), int(sizes.integers(4, case["ny_max"] + 1))
            k = int(sizes.integers(4, 17))
            b, f = _cg(dict(case, nx=nx, ny=s, nz=s), k)
            total["bytes"] += b
            total["flops"] += f
        return total
    E, N, n, nnz = _sizes(case)
    if kind in ("static", "direct"):
        b, f = _assembly(case)
        if kind == "static":
            c = _cg(case)
        else:
            # the band of an ordering along the length is one cross-section of nodes wide
            w = 3.0 * (case["ny"] + 2) * (case["nz"] + 1)
            c = (8.0 * n * w * 3.0, n * w * w + 4.0 * n * w)
        return {"bytes": b + c[0], "flops": f + c[1]}
    if kind == "direct_load":
        w = 3.0 * (case["ny"] + 2) * (case["nz"] + 1)
        return {"bytes": 2.0 * 8.0 * n * w, "flops": 4.0 * n * w}
    if kind == "simp":
        b, f = _assembly(case)
        c = _cg(case)
        return {"bytes": 2.0 * (b + c[0]), "flops": 2.0 * (f + c[1])}
    if kind == "stress":
        return {"bytes": 3.0 * (48.0 * N + 32.0 * E) + 56.0 * N + 48.0 * E, "flops": 3.0 * E * 8.0 * 700.0}
    c = _cg(case, case.get("loads", 1))
    return {"bytes": c[0], "flops": c[1]}


# ----------------------------------------------------------------------------- 64-bit values
_CORNERS = ((-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1))


def _gauss_points(X, conn):
    """(N (8,), dN (E, 8, 3), weight * |J| (E,)) at each of the 2 x 2 x 2 Gauss points."""
    c = torch.tensor(_CORNERS, dtype=torch.float64, device=X.device)
    a = 1.0 / math.sqrt(3.0)
    for p in _CORNERS:
        q = torch.tensor(p, dtype=torch.float64, device=X.device) * a
        t = 1.0 + c * q
        Nv = t.prod(1) / 8.0
        d = torch.stack([c[:, 0] * t[:, 1] * t[:, 2], c[:, 1] * t[:, 0] * t[:, 2], c[:, 2] * t[:, 0] * t[:, 1]]) / 8.0
        J = torch.einsum("ia,eaj->eij", d, X[conn])
        yield Nv, torch.linalg.solve(J, d.expand(len(conn), 3, 8)).transpose(1, 2), torch.linalg.det(J)


def _B(dN):
    B = torch.zeros((dN.shape[0], 6, 8, 3), dtype=torch.float64, device=dN.device)
    x, y, z = dN.unbind(2)
    B[:, 0, :, 0], B[:, 1, :, 1], B[:, 2, :, 2] = x, y, z
    B[:, 3, :, 0], B[:, 3, :, 1] = y, x
    B[:, 4, :, 1], B[:, 4, :, 2] = z, y
    B[:, 5, :, 0], B[:, 5, :, 2] = z, x
    return B.reshape(-1, 6, 24)


class _Exact:
    """K_ff applied element by element, and conjugate gradients to round-off."""

    def __init__(self, mesh, D, scale=None):
        self.X = torch.as_tensor(mesh.nodes).cuda()
        self.conn = torch.as_tensor(mesh.elements).cuda()
        D = torch.as_tensor(D).cuda()
        ke = torch.zeros((len(self.conn), 24, 24), dtype=torch.float64, device="cuda")
        for _, dN, w in _gauss_points(self.X, self.conn):
            B = _B(dN)
            ke += torch.einsum("esa,st,etb->eab", B, D, B * w[:, None, None])
        self.unit = ke
        self.ke = ke if scale is None else ke * scale[:, None, None]
        self.dof = (3 * self.conn[:, :, None] + torch.arange(3, device="cuda")).reshape(len(self.conn), 24)
        self.free = torch.ones(3 * len(self.X), dtype=torch.float64, device="cuda")
        ids = torch.as_tensor(mesh.nodes_on_plane(0, 0.0)).cuda()
        self.free.view(-1, 3)[ids] = 0.0

    def apply(self, p):
        y = torch.zeros_like(p)
        y.index_add_(0, self.dof.reshape(-1), (self.ke @ p[self.dof]).reshape(-1, p.shape[1]))
        return y * self.free[:, None]

    def solve(self, F):
        b = torch.as_tensor(F).cuda().reshape(len(self.free), -1) * self.free[:, None]
        d = torch.zeros_like(self.free).index_add_(0, self.dof.reshape(-1), torch.diagonal(self.ke, dim1=1, dim2=2)
                                                   .reshape(-1))
        x = torch.zeros_like(b)
        norm = b.norm(dim=0).clamp_min(1e-300)
        for tol in (1e-11, 1e-4, 1e-3):   # the solve, then corrections of its residual
            r = b - self.apply(x)
            first = r.norm(dim=0).clamp_min(1e-300)
            e = torch.zeros_like(b)
            z = r / d[:, None]
            p = z
            rz = (r * z).sum(0)
            for it in range(20000):
                q = self.apply(p)
                alpha = rz / (p * q).sum(0).clamp_min(1e-300)
                e += alpha * p
                r = r - alpha * q
                if it % 10 == 9 and bool((r.norm(dim=0) <= tol * torch.maximum(first, 1e-4 * norm * tol)).all()):
                    break
                z = r / d[:, None]
                new = (r * z).sum(0)
                p = z + (new / rz.clamp_min(1e-300)) * p
                rz = new
            x += e
        return x

    def energy(self, u, v):
        """u_e^T K0_e v_e of the unscaled element matrices."""
        return torch.einsum("ea,eab,eb->e", u[self.dof], self.unit, v[self.dof])


def exact(case, seed):
    kind = case["kind"]
    if kind == "pod":
        X = _snapshots(case, seed).double()
        # the modes are fixed up to their sign: no value for them
        return {"sigma": torch.linalg.svdvals(torch.linalg.qr(X, mode="r").R).cpu().numpy(), "V": None}
    if kind == "batch":
        out = []
        for nodes, elements, D, _, F in _batch_models(case, seed):
            out.append(_Exact(feab200.Mesh(nodes=nodes, elements=elements), D).solve(F).cpu().numpy())
        return {"u": out}
    mesh = _mesh(case, seed)
    if kind == "stress":
        return _exact_stress(mesh, _D(), _displacement(mesh, seed))
    rho = torch.as_tensor(np.random.default_rng([seed, 13]).uniform(0.3, 1.0, len(mesh.elements))).cuda()
    if kind == "simp":
        K = _Exact(mesh, _D(E=1.0), RHO_MIN + (1.0 - RHO_MIN) * rho ** PENAL)
        u = K.solve(cantilever.uniform_tip_load(mesh, LX, -1.0))[:, 0]
        dc = -PENAL * (1.0 - RHO_MIN) * rho ** (PENAL - 1.0) * K.energy(u, u)
        centre = K.X[K.conn].mean(1)
        filtered = torch.empty_like(dc)
        for a in range(0, len(dc), 2048):
            h = torch.clamp(_radius(case) - (centre[a:a + 2048, None] - centre[None]).norm(dim=2), min=0.0)
            r = rho[a:a + 2048]
            filtered[a:a + 2048] = (h @ (rho * dc)) / torch.clamp(torch.clamp(r, min=1e-9) * h.sum(1), min=1e-9)
        # the update stops within a tolerance of its multiplier: no exact value for the new densities
        return {"u": u[K.free > 0], "dc": dc, "filtered": filtered, "rho": None}
    K = _Exact(mesh, _D())
    if kind == "panel":
        return {"u": K.solve(_tip_loads(mesh, seed, case["loads"])).cpu().numpy()}
    u = K.solve(_tip_loads(mesh, seed))[:, 0]
    if kind == "load":
        return {"u": u}
    if kind == "direct_load":
        return {"u": u[K.free > 0]}
    out = {"u": u.cpu().numpy()}
    if case.get("grad"):
        out["dc"] = (-PENAL * (1.0 - RHO_MIN) * rho ** (PENAL - 1.0) * K.energy(u, u)).cpu().numpy()
    return out


def _exact_stress(mesh, D, U):
    X, conn, D = torch.as_tensor(mesh.nodes).cuda(), torch.as_tensor(mesh.elements).cuda(), torch.as_tensor(D).cuda()
    dof = (3 * conn[:, :, None] + torch.arange(3, device="cuda")).reshape(len(conn), 24)
    num = torch.zeros((len(X), 6), dtype=torch.float64, device="cuda")
    den = torch.zeros(len(X), dtype=torch.float64, device="cuda")
    mean = torch.zeros((len(conn), 6), dtype=torch.float64, device="cuda")
    vol = torch.zeros(len(conn), dtype=torch.float64, device="cuda")
    for Nv, dN, w in _gauss_points(X, conn):
        s = torch.einsum("st,eta,ea->es", D, _B(dN), U[dof])
        wn = Nv[None, :] * w[:, None]
        num.index_add_(0, conn.reshape(-1), (wn[:, :, None] * s[:, None, :]).reshape(-1, 6))
        den.index_add_(0, conn.reshape(-1), wn.reshape(-1))
        mean += w[:, None] * s
        vol += w
    s = num / den[:, None]
    a, b, c, d, e, f = s.unbind(1)
    mises = torch.sqrt(0.5 * ((a - b) ** 2 + (b - c) ** 2 + (c - a) ** 2) + 3.0 * (d * d + e * e + f * f))
    return {"stress": s, "mises": mises, "elements": mean / vol[:, None]}
