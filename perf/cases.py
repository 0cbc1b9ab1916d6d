"""The measured cases: what programs that use this package have it do, through its public entry points.

Every case is a dict of plain values; ``kind`` names the call that a pass makes:

* ``solve``        one load case of an assembled cantilever or I-beam, numpy in and out
                   (``solve_c3d10_pcg``);
* ``multi``        several load cases at once (``solve_c3d10_multi`` on numpy arrays, or
                   ``SolidSystem.solve_multi_device`` on CUDA tensors);
* ``design``       one step of a stiffness optimisation: compliance and its gradients for new
                   moduli (``ComplianceProblem``: assembly, solve, adjoint), with the AMG hierarchy
                   kept or rebuilt;
* ``assemble``     the stiffness matrix of new moduli that are already on the GPU;
* ``apply``        the products of a caller's own Krylov loop: K x in FP64 and in FP32;
* ``recover``      internal forces and stresses of a displacement field;
* ``frame_newton`` a geometrically nonlinear beam frame (``solve_nonlinear_jfnk``);
* ``frame_solve``  one load case of a linear space frame (``FrameSystem.solve``).

``exact`` evaluates the same outputs densely in 64 bits with torch alone, up to the sizes where a
dense factorisation is quick.
"""

from __future__ import annotations

import dataclasses
import functools

import numpy as np
import torch

from wnfea_b200 import _lib
from wnfea_b200.autograd import ComplianceProblem
from wnfea_b200.beam import frame_linear_system, solve_nonlinear_jfnk
from wnfea_b200.frames import generate_frame_grid, generate_space_frame
from wnfea_b200.mesh import (generate_c3d10_ibeam_structured, generate_c3d10_kuhn_block, generate_c3d10_pressure_block,
                             tip_load_cases)
from wnfea_b200.solid_solver import assemble_c3d10_sparse_3dof, solve_c3d10_multi, solve_c3d10_pcg

#: Largest system that exact() factorises densely.
EXACT_DOFS = 24_000


# ----------------------------------------------------------------------------------------
# cases
# ----------------------------------------------------------------------------------------
def listed():
    return [
        # a small part solved as a newcomer calls it, every argument at its default (point Jacobi, FP64, 1e-6):
        # some hundred iterations of microseconds of work
        {"name": "solve_default", "kind": "solve", "mesh": "bar", "nx": 20, "ny": 2, "nz": 2,
         "preconditioner": "jacobi", "precision": "fp64", "rtol": 1e-6},
        # the same part with the multigrid preconditioner, as interactive checks of small parts use it: latency
        {"name": "solve_small", "kind": "solve", "mesh": "bar", "nx": 20, "ny": 2, "nz": 2,
         "preconditioner": "amg", "precision": "fp64", "rtol": 1e-8},
        # the benchmark's I-beam (1,012,755 DOFs) in its mixed precision: the framework's headline call
        {"name": "solve_ibeam", "kind": "solve", "mesh": "ibeam", "slices": 315,
         "preconditioner": "amg", "precision": "mixed_fp32", "rtol": 1e-8},
        # an ordinary beam (about 300,000 DOFs), all in FP64
        {"name": "solve_fp64", "kind": "solve", "mesh": "ibeam", "slices": 97,
         "preconditioner": "amg", "precision": "fp64", "rtol": 1e-8},
        # the load book of one structure: the benchmark's 32 tip load cases at once, on the GPU
        {"name": "multi_32", "kind": "multi", "mesh": "ibeam", "slices": 315, "cases": 32,
         "precision": "mixed_fp32", "rtol": 1e-8, "host": False},
        # a handful of load cases of a modest part, numpy in and out
        {"name": "multi_5", "kind": "multi", "mesh": "bar", "nx": 41, "ny": 9, "nz": 7, "cases": 5,
         "precision": "fp64", "rtol": 1e-8, "host": True},
        # one step of a graded-modulus design loop on the 162,000-element block, hierarchy kept
        {"name": "design_step", "kind": "design", "nx": 60, "ny": 30, "nz": 15,
         "precision": "mixed_fp32", "rebuild": False},
        # the first evaluation of a new matrix, hierarchy built on the way
        {"name": "design_rebuild", "kind": "design", "nx": 31, "ny": 17, "nz": 9,
         "precision": "fp64", "rebuild": True},
        # the matrix of new moduli for a caller who keeps the mesh (a material or topology sweep)
        {"name": "assemble", "kind": "assemble", "mesh": "ibeam", "slices": 315},
        # a caller's own iteration around the assembled matrix (eigenvalues, dynamics)
        {"name": "apply", "kind": "apply", "mesh": "ibeam", "slices": 157},
        # post-processing of a displacement field: reactions (internal forces) and stresses
        {"name": "recover", "kind": "recover", "mesh": "ibeam", "slices": 315},
        # the 10 x 10 frame under large displacements, ten load increments
        {"name": "frame_newton", "kind": "frame_newton", "nx": 10, "ny": 10, "steps": 10},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "multi", "multi", "design", "design", "assemble", "apply", "recover",
                       "frame_newton", "frame_solve"])
    if kind == "solve":
        how = rng.choice(["default", "amg", "amg", "amg"])
        if how == "default":
            return {"kind": kind, "mesh": "bar", "nx": _log(rng, 5, 40), "ny": rng.randint(1, 5),
                    "nz": rng.randint(1, 5), "preconditioner": rng.choice(["jacobi", "block_jacobi"]),
                    "precision": "fp64", "rtol": 1e-6}
        case = {"kind": kind, "preconditioner": "amg", "precision": rng.choice(["fp64", "mixed_fp32"]), "rtol": 1e-8}
        if rng.random() < 0.5:
            return {**case, "mesh": "bar", "nx": _log(rng, 8, 90), "ny": _log(rng, 2, 16), "nz": _log(rng, 2, 16)}
        return {**case, "mesh": "ibeam", "slices": _log(rng, 20, 310)}
    if kind == "multi":
        case = {"kind": kind, "cases": rng.choice([2, 3, 7, 16, 29, 32]), "rtol": 1e-8,
                "precision": rng.choice(["fp64", "mixed_fp32"]), "host": rng.random() < 0.5}
        if rng.random() < 0.5:
            return {**case, "mesh": "bar", "nx": _log(rng, 8, 60), "ny": _log(rng, 2, 12), "nz": _log(rng, 2, 12)}
        return {**case, "mesh": "ibeam", "slices": _log(rng, 20, 200)}
    if kind == "design":
        return {"kind": kind, "nx": _log(rng, 6, 60), "ny": _log(rng, 4, 28), "nz": _log(rng, 3, 15),
                "precision": rng.choice(["fp64", "mixed_fp32"]), "rebuild": rng.random() < 0.3}
    if kind in ("assemble", "apply", "recover"):
        if rng.random() < 0.3:
            return {"kind": kind, "mesh": "bar", "nx": _log(rng, 4, 90), "ny": rng.randint(1, 12),
                    "nz": rng.randint(1, 12)}
        return {"kind": kind, "mesh": "ibeam", "slices": _log(rng, 10, 310)}
    if kind == "frame_newton":
        return {"kind": kind, "nx": rng.randint(4, 13), "ny": rng.randint(4, 13), "steps": rng.randint(3, 10)}
    return {"kind": kind, "nx": _log(rng, 6, 32), "ny": _log(rng, 6, 32), "nz": _log(rng, 6, 32),
            "precision": rng.choice(["fp64", "mixed_fp32"])}


# ----------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _mesh(mesh, *size):
    if mesh == "ibeam":
        return generate_c3d10_ibeam_structured(n_slices=size[0], length=4.0 * size[0] / 315)[0]
    nx, ny, nz = size
    if mesh == "bar":  # cells of 0.05 m, the cantilever of 20 x 2 x 2 of them among the sizes
        return generate_c3d10_kuhn_block(0.05 * nx, 0.05 * ny, 0.05 * nz, nx, ny, nz)[0]
    return generate_c3d10_pressure_block(nx / 30, ny / 30, nz / 30, nx, ny, nz)[0]


def _model(case):
    """The case's model, a fresh object around the (kept) host mesh."""
    if case["kind"] == "design":
        m = _mesh("block", case["nx"], case["ny"], case["nz"])
    elif case["mesh"] == "ibeam":
        m = _mesh("ibeam", case["slices"])
    else:
        m = _mesh("bar", case["nx"], case["ny"], case["nz"])
    return dataclasses.replace(m)


def _fixed(model):
    """Fixed DOFs of a solid model whose supports clamp whole nodes."""
    ids = np.array([s.node_id for s in model.supports], dtype=np.int64)
    return (3 * ids[:, None] + np.arange(3)).ravel()


def _loads(model, n, seed):
    """n tip load cases (columns) of random direction and 10 to 100 kN, zero on the fixed DOFs."""
    F = tip_load_cases(model.mesh_nodes, n, seed=seed)
    F[_fixed(model)] = 0.0
    return F


def _moduli(n, seed):
    """Per-element moduli, log-uniform over 1 to 210 GPa."""
    return np.exp(np.random.default_rng(seed).uniform(np.log(1e9), np.log(210e9), n))


def _field(model, seed):
    """Nodal displacements of a bent, twisted and locally disturbed body (millimetres), node-major."""
    rng = np.random.default_rng(seed)
    x = model.mesh_nodes - model.mesh_nodes.mean(axis=0)
    x = x / np.abs(x).max()
    a = rng.standard_normal((3, 10))
    p = np.column_stack([np.ones(len(x)), x, x**2, x[:, 0] * x[:, 1], x[:, 1] * x[:, 2], x[:, 2] * x[:, 0]])
    return (1e-3 * (p @ a.T) + 1e-6 * rng.standard_normal(x.shape)).ravel()


def _frame(case, seed):
    if case["kind"] == "frame_newton":
        return generate_frame_grid(case["nx"], case["ny"], seed=seed)
    return generate_space_frame(case["nx"], case["ny"], case["nz"], seed=seed)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind in ("solve", "multi"):
        model = _model(case)
        K, _, _ = assemble_c3d10_sparse_3dof(model)
        if kind == "solve":
            F = _loads(model, 1, seed)[:, 0].copy()
        else:
            F = _loads(model, case["cases"], seed)
            if not case["host"]:
                F = torch.from_numpy(F).cuda()
                state["U"] = torch.empty_like(F)
        if case.get("preconditioner", "amg") == "amg":
            K.system.amg_setup()
        return {**state, "K": K, "F": F}
    if kind == "design":
        model = _model(case)
        problem = ComplianceProblem.from_model(model, precision=case["precision"], reuse_hierarchy=not case["rebuild"])
        F = np.zeros((len(model.mesh_nodes), 3))
        ids = np.array([ld.node_id for ld in model.loads])
        F[ids] = np.array([[ld.fx, ld.fy, ld.fz] for ld in model.loads])
        F = torch.from_numpy(F.ravel()).cuda()
        E = torch.from_numpy(_moduli(problem.n_el, seed)).cuda()
        if not case["rebuild"]:  # the loop's earlier steps have built the hierarchy, for other moduli
            problem.solve(E * torch.from_numpy(1 + 0.1 * np.random.default_rng(seed + 1).random(problem.n_el)).cuda(), F)
        return {**state, "problem": problem, "E": E.requires_grad_(True), "F": F.requires_grad_(True)}
    if kind in ("assemble", "apply", "recover"):
        model = _model(case)
        K, _, _ = assemble_c3d10_sparse_3dof(model)
        s = K.system
        u = torch.from_numpy(_field(model, seed)).cuda()
        if kind == "assemble":
            E = torch.from_numpy(_moduli(s.n_el, seed)).cuda()
            return {**state, "K": K, "props": torch.stack([E, torch.full_like(E, 0.3)], dim=1).contiguous(),
                    "values": _device_values(s)}
        if kind == "apply":
            return {**state, "K": K, "x": u, "x32": u.float(), "y": torch.empty_like(u),
                    "y32": torch.empty_like(u, dtype=torch.float32)}
        f8 = functools.partial(torch.empty, dtype=torch.float64, device="cuda")
        return {**state, "K": K, "u": u, "f": f8(3 * s.n_nodes), "sig": f8(s.n_el, 6), "vm": f8(s.n_el),
                "nodal": f8(s.n_nodes)}
    model = _frame(case, seed)
    if kind == "frame_newton":
        return {**state, "model": model}
    frame, system, F = frame_linear_system(model)
    system.amg_setup()
    return {**state, "frame": frame, "system": system, "F": F}


class _Borrowed:
    """A device array of a handle, as torch takes it in."""

    def __init__(self, address, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (address, False), "version": 3,
                                         "strides": None}


def _device_values(system):
    """The handle's assembled FP64 values as a CUDA tensor (9, nnzb), entry (i, j) in row 3 i + j."""
    import ctypes

    p = [ctypes.c_void_p() for _ in range(5)]
    _lib.call("wn_solid_device_arrays", system.handle, *map(ctypes.byref, p))
    return torch.as_tensor(_Borrowed(p[0].value, (9, system.nnzb)), device="cuda")


# ----------------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        return solve_c3d10_pcg(state["K"], state["F"], rtol=case["rtol"], preconditioner=case["preconditioner"],
                               precision=case["precision"])[0]
    if kind == "multi":
        if case["host"]:
            return solve_c3d10_multi(state["K"], state["F"], rtol=case["rtol"], precision=case["precision"])[0]
        state["K"].system.solve_multi_device(state["F"], state["U"], rtol=case["rtol"],
                                             precision=0 if case["precision"] == "fp64" else 1)
        return state["U"]
    if kind == "design":
        E, F = state["E"], state["F"]
        C = state["problem"].compliance(E, F)
        gE, gF = torch.autograd.grad(C, (E, F))
        return {"C": C.detach(), "dE": gE, "dF": gF}
    if kind == "frame_newton":
        return solve_nonlinear_jfnk(state["model"], n_load_steps=case["steps"], verbose=False)
    if kind == "frame_solve":
        return state["system"].solve(state["F"], precision=case["precision"])[0]
    h = state["K"].system.handle
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "assemble":
        _lib.call("wn_assemble_c3d10_device", h, state["props"].data_ptr(), 1, stream)
        return state["values"]
    if kind == "apply":
        _lib.call("wn_spmv_solid_device", h, 0, state["x"].data_ptr(), state["y"].data_ptr(), stream)
        _lib.call("wn_spmv_solid_device", h, 1, state["x32"].data_ptr(), state["y32"].data_ptr(), stream)
        return {"y": state["y"], "y32": state["y32"]}
    _lib.call("wn_fint_c3d10_device", h, state["u"].data_ptr(), state["f"].data_ptr(), stream)
    _lib.call("wn_stress_c3d10_device", h, state["u"].data_ptr(), state["sig"].data_ptr(), state["vm"].data_ptr(),
              state["nodal"].data_ptr(), stream)
    return {"f": state["f"], "sig": state["sig"], "vm": state["vm"], "nodal": state["nodal"]}


# ----------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=32)
def _blocks(*key):
    """Number of 3x3 blocks of a mesh's matrix."""
    m = _mesh(*key)
    conn = torch.from_numpy(m.solid_elements.astype(np.int64))
    conn = conn.cuda() if torch.cuda.is_available() else conn
    pair = conn[:, :, None] * len(m.mesh_nodes) + conn[:, None, :]
    return int(torch.unique(pair.reshape(-1)).numel())


def work(case):
    """Inputs read once, outputs written once; one product with the matrix where there is one."""
    kind = case["kind"]
    if kind == "frame_newton":
        n, e = case["nx"] * case["ny"], 2 * case["nx"] * case["ny"] - case["nx"] - case["ny"]
        return {"bytes": 8.0 * (6 * n * 2 + 18 * e), "flops": case["steps"] * 2 * (6 * n) ** 3 / 3}
    if kind == "frame_solve":
        n = case["nx"] * case["ny"] * case["nz"]
        blocks = 7 * n - 2 * (n // case["nx"] + n // case["ny"] + n // case["nz"])
        return {"bytes": blocks * (36 * 8 + 4.0) + 6 * n * 16, "flops": 72.0 * blocks}
    key = ("block", case["nx"], case["ny"], case["nz"]) if kind == "design" else (
        ("ibeam", case["slices"]) if case["mesh"] == "ibeam" else ("bar", case["nx"], case["ny"], case["nz"]))
    m = _mesh(*key)
    n, e = len(m.mesh_nodes), len(m.solid_elements)
    element_in = 24.0 * n + e * (40 + 16)
    if kind == "recover":
        return {"bytes": element_in + 24 * n + 24 * n + e * 56 + 8 * n, "flops": 2.0 * e * 4 * (30 * 9 + 36 + 180)}
    b = _blocks(*key)
    if kind == "assemble":
        return {"bytes": element_in + 72.0 * b, "flops": e * 100 * 4 * 20.0}
    if kind == "apply":
        return {"bytes": b * (72 + 36 + 4.0) + 3 * n * 24, "flops": 36.0 * b}
    k = case.get("cases", 1)
    solve = {"bytes": b * 76.0 + 3 * n * 16 * k, "flops": 18.0 * b * k}
    if kind == "design":
        return {"bytes": solve["bytes"] + element_in + 72.0 * b + 24 * n + 8 * e, "flops": solve["flops"] + e * 8000.0}
    return solve


# ----------------------------------------------------------------------------------------
# the same outputs in 64 bits, from torch alone
# ----------------------------------------------------------------------------------------
def _element_fields(x):
    """dN/dx (M, 4, 3, 10) and w |J| (M, 4) of ten-node tetrahedra with coordinates x (M, 10, 3)."""
    a, b = (5 - 5**0.5) / 20, (5 + 3 * 5**0.5) / 20
    at = torch.tensor([[a, a, a], [b, a, a], [a, b, a], [a, a, b]], dtype=x.dtype, device=x.device)

    def shape(p):
        L = torch.cat([1 - p.sum()[None], p])
        pairs = ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))
        return torch.stack([*(L * (2 * L - 1)), *(4 * L[i] * L[j] for i, j in pairs)])

    dN = torch.stack([torch.autograd.functional.jacobian(shape, p).T for p in at])  # (4, 3, 10)
    J = torch.einsum("gkn,mnj->mgkj", dN, x)
    return torch.einsum("mgij,gjn->mgin", torch.linalg.inv(J), dN), torch.linalg.det(J) / 24


def _strain_operator(d):
    """B (M, 4, 6, 30), rows xx, yy, zz, xy, yz, zx, from dN/dx."""
    B = d.new_zeros(*d.shape[:2], 6, 10, 3)
    for row, parts in enumerate((((0, 0),), ((1, 1),), ((2, 2),), ((0, 1), (1, 0)), ((1, 2), (2, 1)), ((2, 0), (0, 2)))):
        for axis, comp in parts:
            B[:, :, row, :, comp] = d[:, :, axis]
    return B.reshape(*d.shape[:2], 6, 30)


def _elasticity(E, nu):
    C = E.new_zeros(len(E), 6, 6)
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    C[:, :3, :3] = lam[:, None, None]
    for i in range(3):
        C[:, i, i] += 2 * mu
        C[:, 3 + i, 3 + i] = mu
    return C


class _Dense:
    """Element matrices of a model and what follows from them."""

    def __init__(self, model, E, nu=0.3):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.x = torch.from_numpy(model.mesh_nodes).to(dev)
        self.conn = torch.from_numpy(model.solid_elements.astype(np.int64)).to(dev)
        self.n, self.dev = len(self.x), dev
        self.E = torch.as_tensor(E, dtype=torch.float64, device=dev).expand(len(self.conn))
        self.nu = nu
        self.dofs = (3 * self.conn[:, :, None] + torch.arange(3, device=dev)).reshape(len(self.conn), 30)
        fixed = torch.zeros(3 * self.n, dtype=torch.bool, device=dev)
        fixed[torch.from_numpy(_fixed(model)).to(dev)] = True
        self.fixed = fixed

    def parts(self, step=8192):
        for i in range(0, len(self.conn), step):
            s = slice(i, i + step)
            d, w = _element_fields(self.x[self.conn[s]])
            yield s, _strain_operator(d), w, _elasticity(self.E[s], self.nu)

    def element_matrices(self, s, B, w, C):
        Ke = torch.einsum("mg,mgki,mgkj->mij", w, B, torch.einsum("mkl,mglj->mgkj", C, B))
        return 0.5 * (Ke + Ke.transpose(1, 2))

    def clamp(self, Ke, s):
        f = self.fixed[self.dofs[s]]
        return Ke.masked_fill(f[:, :, None] | f[:, None, :], 0.0)

    def factor(self):
        K = torch.zeros(9 * self.n * self.n, dtype=torch.float64, device=self.dev)
        for s, *p in self.parts():
            at = self.dofs[s][:, :, None] * (3 * self.n) + self.dofs[s][:, None, :]
            K.index_add_(0, at.reshape(-1), self.clamp(self.element_matrices(s, *p), s).reshape(-1))
        K = K.view(3 * self.n, 3 * self.n)
        K.diagonal()[self.fixed] = 1.0
        return torch.linalg.cholesky(K)

    def solve(self, F):
        return torch.cholesky_solve(F.to(self.dev), self.factor())

    def stresses(self, u):
        """Internal forces, Gauss-point stresses (M, 4, 6)."""
        f = torch.zeros_like(u)
        sig = []
        for s, B, w, C in self.parts():
            t = torch.einsum("mkl,mglj,mj->mgk", C, B, u[self.dofs[s]])
            f.index_add_(0, self.dofs[s].reshape(-1), torch.einsum("mg,mgki,mgk->mi", w, B, t).reshape(-1))
            sig.append(t)
        return f, torch.cat(sig)

    def block_values(self):
        """Values (9, blocks) over the sorted block pattern, clamped rows and columns made identity."""
        pair = self.conn[:, :, None] * self.n + self.conn[:, None, :]
        keys, slot = torch.unique(pair.reshape(-1), return_inverse=True)
        slot = slot.reshape(len(self.conn), 100)
        V = torch.zeros(len(keys), 9, dtype=torch.float64, device=self.dev)
        for s, *p in self.parts():
            Ke = self.clamp(self.element_matrices(s, *p), s).reshape(-1, 10, 3, 10, 3).transpose(2, 3)
            V.index_add_(0, slot[s].reshape(-1), Ke.reshape(-1, 9))
        diag = torch.searchsorted(keys, torch.arange(self.n, device=self.dev) * (self.n + 1))
        for c in range(3):
            on = self.fixed[c::3]
            V[diag[on], 4 * c] = 1.0
        return keys, V.T.contiguous()


def _beam_force(ue, v0, eref, L0, props):
    """Co-rotational force (12) of one beam with end displacements ue (12)."""
    u1, t1, u2, t2 = ue.split(3)
    e1, e2, _ = eref.split(3)
    du = u2 - u1
    v = v0 + du
    L = v.norm()
    r1 = v / L
    w, c = torch.linalg.cross(e1, r1), e1 @ r1  # the rotation of e1 onto r1: w = sin * axis
    r2 = c * e2 + torch.linalg.cross(w, e2) + w * (w @ e2) / (1 + c)
    tw = 0.5 * ((t1 + t2) @ r1)
    r2 = r2 * torch.cos(tw) + torch.linalg.cross(r1, r2) * torch.sin(tw)
    r3 = torch.linalg.cross(r1, r2)
    E, G, A, Iy, Iz, J = props
    stretch = (2 * (v0 @ du) + du @ du) / (L + L0)
    y, z = (r3 @ du) / L, (r2 @ du) / L
    ty1, tz1, ty2, tz2 = r2 @ t1 + y, r3 @ t1 - z, r2 @ t2 + y, r3 @ t2 - z
    N, T = E * A / L0 * stretch, G * J / L0 * (r1 @ (t2 - t1))
    My1, My2 = E * Iy / L0 * (4 * ty1 + 2 * ty2), E * Iy / L0 * (2 * ty1 + 4 * ty2)
    Mz1, Mz2 = E * Iz / L0 * (4 * tz1 + 2 * tz2), E * Iz / L0 * (2 * tz1 + 4 * tz2)
    f = -N * r1 - (My1 + My2) / L * r3 + (Mz1 + Mz2) / L * r2
    return torch.cat([f, -T * r1 + My1 * r2 + Mz1 * r3, -f, T * r1 + My2 * r2 + Mz2 * r3])


def _frame_solution(model, steps):
    """Displacements of a frame of equal bars, by Newton's method with the exact tangent (steps = 0: linear)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.from_numpy(model.mesh_nodes).to(dev)
    el = torch.from_numpy(model.mesh_elements.astype(np.int64)).to(dev)
    mat, sec = next(iter(model.materials.values())), next(iter(model.sections.values()))
    p = [mat.youngs_modulus, mat.shear_modulus, sec.area, sec.iy, sec.iz, sec.j]
    props = torch.tensor(p, dtype=torch.float64, device=dev).expand(len(el), 6)
    v0 = x[el[:, 1]] - x[el[:, 0]]
    L0 = v0.norm(dim=1)
    e1 = v0 / L0[:, None]
    up = torch.where((e1[:, 2:].abs() < 0.9), x.new_tensor([0.0, 0.0, 1.0]), x.new_tensor([0.0, 1.0, 0.0]))
    e2 = torch.linalg.cross(up, e1)
    e2 = e2 / e2.norm(dim=1, keepdim=True)
    args = (v0, torch.cat([e1, e2, torch.linalg.cross(e1, e2)], dim=1), L0, props)
    dofs = (6 * el[:, :, None] + torch.arange(6, device=dev)).reshape(-1, 12)
    n = 6 * len(x)
    F = x.new_zeros(n)
    for ld in model.loads:
        F[6 * ld.node_id:6 * ld.node_id + 6] += x.new_tensor(ld.force_vector)
    free = torch.ones(n, dtype=torch.bool, device=dev)
    for s in model.supports:
        free[6 * s.node_id:6 * s.node_id + 6] = False
    force = torch.func.vmap(lambda ue, *a: _beam_force(ue, a[0], a[1], a[2], a[3].unbind()))
    tangent = torch.func.vmap(torch.func.jacfwd(lambda ue, *a: _beam_force(ue, a[0], a[1], a[2], a[3].unbind())))

    def step(U, lam):
        R = x.new_zeros(n).index_add_(0, dofs.reshape(-1), force(U[dofs], *args).reshape(-1)) - lam * F
        K = x.new_zeros(n * n)
        K.index_add_(0, (dofs[:, :, None] * n + dofs[:, None, :]).reshape(-1), tangent(U[dofs], *args).reshape(-1))
        K = K.view(n, n)
        d = x.new_zeros(n)
        d[free] = torch.linalg.solve(K[free][:, free], -R[free])
        return d

    U = x.new_zeros(n)
    if steps == 0:
        return step(U, 1.0)
    for lam in np.linspace(1.0 / steps, 1.0, steps):
        for _ in range(25):
            d = step(U, float(lam))
            U = U + d
            if d.norm() <= 1e-12 * U.norm():
                break
    return U


def exact(case, seed):
    kind = case["kind"]
    if kind in ("frame_newton", "frame_solve"):
        model = _frame(case, seed)
        if 6 * len(model.mesh_nodes) > EXACT_DOFS:
            return None
        return _frame_solution(model, case["steps"] if kind == "frame_newton" else 0).cpu().numpy()
    model = _model(case)
    if kind == "recover":
        sys_ = _Dense(model, 2.1e11)
        u = torch.from_numpy(_field(model, seed)).to(sys_.dev)
        f, sig = sys_.stresses(u)
        a, b, c, p, q, r = sig.unbind(-1)
        vm = (0.5 * ((a - b)**2 + (b - c)**2 + (c - a)**2 + 6 * (p**2 + q**2 + r**2))).sqrt().mean(1)
        flat = sys_.conn.reshape(-1)
        total = torch.zeros(sys_.n, dtype=torch.float64, device=sys_.dev).index_add_(0, flat, vm.repeat_interleave(10))
        return {"f": f, "sig": sig.mean(1), "vm": vm, "nodal": total / torch.bincount(flat, minlength=sys_.n)}
    if kind == "assemble":
        return _Dense(model, _moduli(len(model.solid_elements), seed)).block_values()[1]
    if kind == "apply":
        sys_ = _Dense(model, 2.1e11)
        keys, V = sys_.block_values()
        rows, cols = keys // sys_.n, keys % sys_.n
        y = []
        for x in (torch.from_numpy(_field(model, seed)), torch.from_numpy(_field(model, seed)).float().double()):
            t = torch.einsum("ijb,bj->bi", V.view(3, 3, -1), x.to(sys_.dev).view(-1, 3)[cols])
            y.append(torch.zeros(sys_.n, 3, dtype=torch.float64, device=sys_.dev).index_add_(0, rows, t).reshape(-1))
        return {"y": y[0], "y32": y[1]}
    if 3 * len(model.mesh_nodes) > EXACT_DOFS:
        return None
    if kind == "design":
        E = _moduli(len(model.solid_elements), seed)
        sys_ = _Dense(model, E)
        F = np.zeros((len(model.mesh_nodes), 3))
        F[[ld.node_id for ld in model.loads]] = [[ld.fx, ld.fy, ld.fz] for ld in model.loads]
        F = torch.from_numpy(F.ravel()).to(sys_.dev).masked_fill(sys_.fixed, 0.0)
        u = sys_.solve(F[:, None])[:, 0]
        dE = []
        for s, *p in sys_.parts():
            ue = u[sys_.dofs[s]]
            dE.append(-torch.einsum("mi,mij,mj->m", ue, sys_.element_matrices(s, *p), ue) / sys_.E[s])
        return {"C": F @ u, "dE": torch.cat(dE), "dF": (2 * u).masked_fill(sys_.fixed, 0.0)}
    F = torch.from_numpy(_loads(model, case.get("cases", 1), seed))
    U = _Dense(model, 2.1e11).solve(F)
    return (U[:, 0] if kind == "solve" else U).cpu().numpy()
