"""Cases that show how fast the framework does its users' work, from the smallest call to the largest.

Each case is a piece of a simulation's inner loop on tetrahedralised cubes (side k, z = 0 pinned,
3 k (k+1)^2 free variables), through the C ABI or the Python factorizer:

newton   a Newton step: assemble the element Hessians, factor, solve (values and vectors on the device)
batch    the same for many independent meshes of uneven size as one block-diagonal system
solve    further right-hand sides against a factor that is kept (load cases, time steps on a linear model)
host     the drop-in call on host arrays: a shifted factorization and a solve
product  assemble and multiply (a Krylov iteration or a line search, which need no factor)
pcg      assemble and solve by the PCG with the learned preconditioner

The mesh, its analysis and the factorizer are what a program keeps over its steps: they are made once
for a case. The values (element stiffness) and the vectors are made from the seed.
"""
import ctypes
import math
from collections import OrderedDict

import numpy as np
import torch

from meshfemsparse_b200 import _lib, fem
from meshfemsparse_b200.factorizer import B200Factorizer
from meshfemsparse_b200.hessian import BlockCSCHessian, SystemAssembler
from meshfemsparse_b200.learned import LearnedPreconditioner

FULL_DEVICE = _lib.MFS_SOLVE_FULL | _lib.MFS_DEVICE_POINTERS
F64 = torch.float64


def listed():
    return [
        # the benchmark's configuration 2, the largest: one Newton step, four right-hand sides, FP32 with refinement
        {"name": "newton_f32_k64", "kind": "newton", "k": 64, "nrhs": 4, "prec": "f32", "graphs": False},
        # a step of the 48-sided load ramp with the default factorizer: FP64, one right-hand side
        {"name": "newton_f64_k48", "kind": "newton", "k": 48, "nrhs": 1, "prec": "f64", "graphs": False},
        # a middling mesh of odd side
        {"name": "newton_f32_k33", "kind": "newton", "k": 33, "nrhs": 3, "prec": "f32", "graphs": False},
        # configuration 1's mesh, replayed from a CUDA graph as an interactive simulation has it
        {"name": "newton_f32_k20_graph", "kind": "newton", "k": 20, "nrhs": 1, "prec": "f32", "graphs": True},
        # configuration 1 itself: FP64
        {"name": "newton_f64_k20", "kind": "newton", "k": 20, "nrhs": 1, "prec": "f64", "graphs": False},
        # the smallest: a coarse model, where latency and launches count
        {"name": "newton_f64_k7", "kind": "newton", "k": 7, "nrhs": 1, "prec": "f64", "graphs": False},
        # configuration 3 at a fifth of its count: meshes of 1,000 to 50,000 variables, eight right-hand sides
        {"name": "batch_f32_48", "kind": "batch", "count": 48, "nrhs": 8, "prec": "f32", "mesh_seed": 3},
        # load cases on a kept factor: many right-hand sides at once ...
        {"name": "solve_f32_k48_r32", "kind": "solve", "k": 48, "nrhs": 32, "prec": "f32"},
        # ... and one at a time
        {"name": "solve_f64_k40_r1", "kind": "solve", "k": 40, "nrhs": 1, "prec": "f64"},
        # the reference's drop-in call: numpy in, numpy out, H + sigma I
        {"name": "host_f64_k24", "kind": "host", "k": 24, "nrhs": 2, "prec": "f64", "sigma": 1e-3},
        # matrix products between factorizations on the largest mesh
        {"name": "product_k64", "kind": "product", "k": 64, "nrhs": 1},
        # the learned preconditioner's PCG on the load ramp's material
        {"name": "pcg_k24", "kind": "pcg", "k": 24, "nrhs": 1},
    ]


def draw(rng):
    def side(lo, hi):   # spread over the logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["newton", "newton", "newton", "batch", "solve", "solve", "host", "product", "pcg"])
    prec = rng.choice(["f32", "f64"])
    if kind == "newton":
        return {"kind": kind, "k": side(6, 56 if prec == "f32" else 44), "nrhs": rng.choice([1, 1, 2, 3, 4, 8]),
                "prec": prec, "graphs": rng.random() < 0.25}
    if kind == "batch":
        return {"kind": kind, "count": side(4, 48), "nrhs": rng.choice([1, 3, 8]), "prec": prec,
                "mesh_seed": rng.randrange(1000)}
    if kind == "solve":
        return {"kind": kind, "k": side(8, 44), "nrhs": rng.choice([1, 1, 2, 5, 8, 13, 32]), "prec": prec}
    if kind == "host":
        return {"kind": kind, "k": side(6, 30), "nrhs": rng.choice([1, 2, 5]), "prec": prec,
                "sigma": rng.choice([0.0, 1e-3, 1e-1])}
    if kind == "product":
        return {"kind": kind, "k": side(8, 60), "nrhs": rng.choice([1, 2, 4])}
    return {"kind": kind, "k": side(6, 28), "nrhs": rng.choice([1, 2])}


# ---------------------------------------------------------------- meshes and factorizers
def sides(case):
    """The cubes' sides: one, or a batch's (sides log-uniform so that variables span 1,000 to 50,000)."""
    if case["kind"] != "batch":
        return [case["k"]]
    rng = np.random.default_rng(case["mesh_seed"])
    return [int(round(math.exp(v))) for v in rng.uniform(math.log(7), math.log(24), size=case["count"])]


class Mesh:
    """A case's mesh, analysis and factorizer, and on the GPU what its element matrices are made of."""

    def __init__(self, case):
        nodes, tets, pins, off = [], [], [], 0
        for m, k in enumerate(sides(case)):
            p, t = fem.tet_cube(k, jitter=0.1, seed=m)
            nodes.append(p)
            tets.append(t + off)
            pins.append(fem.bottom_pins(p) + 3 * off)
            off += p.shape[0]
        nodes, tets, pins = np.concatenate(nodes), np.concatenate(tets), np.concatenate(pins)
        self.n = 3 * nodes.shape[0]
        grads, volume = fem.shape_gradients(nodes, tets)
        dev = torch.device("cuda")
        self.grads, self.volume = torch.as_tensor(grads, device=dev), torch.as_tensor(volume, device=dev)
        self.dofs = (3 * torch.as_tensor(tets, device=dev)[:, :, None] + torch.arange(3, device=dev)).reshape(-1, 12)
        self.free = torch.ones(self.n, dtype=torch.bool, device=dev)
        self.free[torch.as_tensor(pins, device=dev)] = False
        self.pattern = SystemAssembler(nodes.shape[0]).blockSparsityPattern(tets)
        f32 = case.get("prec") == "f32"
        # refined a little past the default 1e-10, so that the solution and not the stopping point is what comes out
        self.fac = B200Factorizer(f32, refine=f32, refine_tol=1e-11, use_graphs=bool(case.get("graphs")))
        self.fac.factorizeSymbolic(self.pattern, pins)
        self.fac.setElements(tets)
        if case["kind"] == "solve":
            ke = self.stiffness(0)
            torch.cuda.synchronize()
            assemble(self.fac, ke)
            _lib.check(_lib.load().mfs_numeric(self.fac._h, None, None, 0.0, 0), self.fac._h)
        if case["kind"] == "pcg":
            # as before training: the work of an iteration does not depend on the weights
            self.net = LearnedPreconditioner(seed=0)

    def stiffness(self, seed):
        """(elements, 12, 12) linear-elastic stiffness, Young's modulus log-uniform in [0.1, 10] per element, nu 0.35."""
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        E = torch.exp(math.log(10.0) * (2 * torch.rand(self.volume.numel(), generator=gen, device="cuda", dtype=F64) - 1))
        nu = 0.35
        lam, mu = E * self.volume * nu / ((1 + nu) * (1 - 2 * nu)), E * self.volume / (2 * (1 + nu))
        g = self.grads
        ke = torch.empty(g.shape[0], 4, 3, 4, 3, device="cuda", dtype=F64)
        for a in range(4):
            for b in range(4):
                outer = g[:, a, :, None] * g[:, b, None, :]
                k = lam[:, None, None] * outer + mu[:, None, None] * outer.transpose(1, 2)
                k.diagonal(dim1=1, dim2=2).add_((mu * (g[:, a] * g[:, b]).sum(1))[:, None])
                ke[:, a, :, b, :] = k
        ke = ke.reshape(-1, 12, 12)
        return (0.5 * (ke + ke.transpose(1, 2))).contiguous()

    def vectors(self, seed, nrhs):
        """nrhs loads as rows, standard normal, zero on the pinned variables."""
        gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
        return torch.randn(nrhs, self.n, generator=gen, device="cuda", dtype=F64) * self.free


_kept = OrderedDict()


def mesh_of(case):
    """The case's mesh; the last two are kept."""
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "nrhs", "sigma")))
    if key not in _kept:
        while len(_kept) >= 2:
            _kept.popitem(last=False)
        _kept[key] = Mesh(case)
    _kept.move_to_end(key)
    return _kept[key]


def pointer(t):
    return ctypes.c_void_p(t.data_ptr())


def assemble(fac, ke, out=None):
    _lib.check(_lib.load().mfs_assemble(fac._h, pointer(ke), None if out is None else pointer(out),
                                        _lib.MFS_DEVICE_POINTERS), fac._h)


# ---------------------------------------------------------------- the cases
def prepare(case, seed):
    mesh, kind, nrhs = mesh_of(case), case["kind"], case["nrhs"]
    state = {"case": case, "mesh": mesh, "fac": mesh.fac, "b": mesh.vectors(seed, nrhs)}
    state["x"] = torch.empty_like(state["b"])
    if kind != "solve":
        state["ke"] = mesh.stiffness(seed)
    if kind == "product":
        state["ax"] = torch.empty(9 * mesh.pattern.nz, device="cuda", dtype=F64)
    if kind == "host":
        torch.cuda.synchronize()
        p = mesh.pattern
        ax = torch.empty(9 * p.nz, device="cuda", dtype=F64)
        assemble(mesh.fac, state.pop("ke"), ax)
        state["H"] = BlockCSCHessian(p.numBlocks, p.Ap, p.Ai, 3, ax.cpu().numpy())
        state["b"] = np.ascontiguousarray(state["b"].T.cpu().numpy())
        del state["x"]
    torch.cuda.synchronize()
    return state


def run(state):
    case, fac = state["case"], state["fac"]
    lib, h, kind, nrhs = _lib.load(), fac._h, case["kind"], case["nrhs"]
    if kind == "host":
        fac.factorizeNumericWithShift(state["H"], case["sigma"])
        return fac.solveMultiRHS(state["b"])
    b, x = state["b"], state["x"]
    n = b.shape[1]
    if kind == "solve":
        _lib.check(lib.mfs_solve(h, pointer(b), pointer(x), nrhs, n, FULL_DEVICE), h)
        return x
    if kind == "product":
        assemble(fac, state["ke"], state["ax"])
        _lib.check(lib.mfs_apply(h, pointer(b), pointer(x), nrhs, n, FULL_DEVICE), h)
        return {"values": state["ax"], "y": x}
    assemble(fac, state["ke"])
    if kind == "pcg":
        iterations = ctypes.c_int32()
        _lib.check(lib.mfs_pcg_solve(h, state["mesh"].net._p, None, pointer(b), pointer(x), nrhs, n, FULL_DEVICE, 6000,
                                     1e-13, ctypes.byref(iterations)), h)
        return x
    _lib.check(lib.mfs_numeric(h, None, None, 0.0, 0), h)
    _lib.check(lib.mfs_solve(h, pointer(b), pointer(x), nrhs, n, FULL_DEVICE), h)
    return x


def work(case):
    """Sizes from the mesh; the factor's entries and operations by fits to nested dissection on these cubes (within 4 %)."""
    f32, nrhs = case.get("prec") == "f32", case["nrhs"]
    n = ke = blocks = entries = ops = 0
    for k in sides(case):
        m, nodes = 3 * k * (k + 1) ** 2, (k + 1) ** 3
        n += m
        ke += 6 * k ** 3 * 144 * 8
        blocks += nodes + 3 * k * (k + 1) ** 2 + 3 * k * k * (k + 1) + k ** 3      # nodes and edges
        entries += m ** (4 / 3) * (1.85 * math.log(m) - 2.9)
        ops += m ** 2 * (1.45 * math.log(m) + 2.3)
    values, vectors, size = 72 * blocks, 8 * n * nrhs, 4 if f32 else 8
    solve = {"bytes": 2 * size * entries + 2 * vectors, "flops": 4 * entries * nrhs}
    kind = case["kind"]
    if kind == "solve":
        return solve
    product = {"bytes": values + 2 * vectors, "flops": 36 * blocks * nrhs}
    if kind == "product":
        return {"bytes": ke + values + product["bytes"], "flops": ke / 8 + product["flops"]}
    if kind == "pcg":
        its = 45 * max(sides(case))   # about; an iteration: H, G and its transpose
        return {"bytes": ke + 3 * its * product["bytes"], "flops": 3 * its * product["flops"]}
    start = 2 * values if kind == "host" else ke + values
    return {"bytes": start + size * entries + solve["bytes"], "flops": ops + solve["flops"]}


# ---------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    mesh, kind = mesh_of(case), case["kind"]
    b = mesh.vectors(seed, case["nrhs"])
    ke = mesh.stiffness(0 if kind == "solve" else seed)
    sigma, free = case.get("sigma", 0.0), mesh.free
    every = mesh.dofs.reshape(-1)

    def times(v):
        out = torch.empty_like(v)
        for r in range(v.shape[0]):
            parts = torch.bmm(ke, v[r][mesh.dofs][:, :, None]).reshape(-1)
            out[r] = torch.zeros_like(v[r]).index_add_(0, every, parts) * free
        return out + sigma * v

    if kind == "product":
        return {"values": None, "y": times(b)}
    if ke.shape[0] * case["nrhs"] > 1.6e6 and case["nrhs"] > 1:
        return None   # over 20 seconds
    # conjugate gradients with the diagonal, started again on the true residual until that no longer falls
    diag = torch.zeros(mesh.n, device="cuda", dtype=F64).index_add_(0, every, ke.diagonal(dim1=1, dim2=2).reshape(-1)) + sigma
    inv = torch.where(free, 1 / diag, torch.zeros_like(diag))
    x = torch.zeros_like(b)
    norm = b.norm(dim=1, keepdim=True)
    for _ in range(3):
        r = b - times(x)
        z = r * inv
        p, rz, start = z.clone(), (r * z).sum(1, keepdim=True), r.norm(dim=1, keepdim=True)
        for it in range(20000):
            q = times(p)
            alpha = rz / (p * q).sum(1, keepdim=True).clamp_min(1e-300)
            x += alpha * p
            r -= alpha * q
            if it % 32 == 31 and bool((r.norm(dim=1, keepdim=True) <= torch.maximum(1e-8 * start, 1e-17 * norm)).all()):
                break
            z = r * inv
            new = (r * z).sum(1, keepdim=True)
            p = z + (new / rz.clamp_min(1e-300)) * p
            rz = new
    return x.T.contiguous() if kind == "host" else x
