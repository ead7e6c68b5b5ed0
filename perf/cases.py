"""The work a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values.  ``listed()`` gives the fixed ones, ``draw(rng)`` one more of
the same ranges, ``prepare(case, seed)`` what a program holds before the call (mesh arrays, DOF
table, coefficients, an assembled matrix), ``run(state)`` one pass through the public entry points
with its outputs, ``work(case)`` the bytes and operations of a pass, ``exact(case, seed)`` the
outputs as plain torch computes them in 64 bits.

The kinds of work:

* ``assemble``: a new mesh comes in (mesh adaption, a moving mesh): the space, the pattern, the
  matrix and the right-hand side, handed back as FreeFEM's sorted CSR;
* ``terms``: the same for a varf with coefficients and sources that are functions of the point
  (advection, reaction, a Robin boundary);
* ``script``: a whole script, mesh to solution: space, matrix, right-hand side, CG;
* ``cg``: u[] = A^-1*b on a kept matrix (time steps, several loads), FP64 or double-float SpMV;
* ``mixed``: the same with the FP32 inner solver and FP64 refinement;
* ``gmres``: a nonsymmetric system (advection);
* ``adjoint``: loss and gradient of an inverse problem: numeric reassembly, forward solve, transpose
  solve, element sensitivities;
* ``batch``: many small problems with new coefficients: numeric reassembly and one batched solve.

Meshes are squares and cubes cut into simplices with every interior vertex moved at random, as
unstructured as a mesh with this connectivity can be; coefficients are lognormal per element.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "freefem-sources_gb300"))
import ffgpu  # noqa: E402
from ffgpu import adjoint as ff_adjoint  # noqa: E402
from ffgpu import batch as ff_batch  # noqa: E402
from ffgpu import expr as ff_expr  # noqa: E402

F64, I32, I64 = torch.float64, torch.int32, torch.int64


def listed():
    return [
        # the smallest calls, where host work and launches count: a coarse mesh of an adaption loop
        dict(name="assemble_p1_square33", kind="assemble", fe="P1", dim=2, nx=33, ny=47, nz=0),
        # heat conduction in 3D, one material value per tetrahedron
        dict(name="assemble_p1_cube96", kind="assemble", fe="P1", dim=3, nx=96, ny=96, nz=96),
        # linear elasticity on a block, the densest rows FreeFEM's P2 spaces give
        dict(name="assemble_p2vec_cube22", kind="assemble", fe="P2vec", dim=3, nx=22, ny=23, nz=21),
        # advection-diffusion-reaction with coefficients of the point, P2, a Robin wall
        dict(name="terms_p2_cube20", kind="terms", fe="P2", dim=3, nx=20, ny=19, nz=21),
        # the tutorial script at an ordinary size, mesh to solution
        dict(name="script_p1_square256", kind="script", fe="P1", dim=2, nx=256, ny=256, nz=0),
        # one time step's solve on a large 3D heat problem
        dict(name="cg_p1_cube120", kind="cg", fe="P1", dim=3, nx=120, ny=120, nz=120, mode=0),
        # one load case on a kept elasticity matrix, FP64 and with the double-float SpMV
        dict(name="cg_p2vec_cube24", kind="cg", fe="P2vec", dim=3, nx=24, ny=24, nz=24, mode=0),
        dict(name="cg_p2vec_cube17_df", kind="cg", fe="P2vec", dim=3, nx=17, ny=16, nz=15, mode=1),
        # the large heat problem where FP32 inner iterations pay
        dict(name="mixed_p1_cube120", kind="mixed", fe="P1", dim=3, nx=120, ny=120, nz=120),
        # a nonsymmetric system, FreeFEM's default restart length never reached
        dict(name="gmres_p1_square90", kind="gmres", fe="P1", dim=2, nx=90, ny=101, nz=0),
        # one step of an inverse problem
        dict(name="adjoint_p1_square200", kind="adjoint", fe="P1", dim=2, nx=200, ny=211, nz=0),
        # a parameter study over many small domains
        dict(name="batch_p1_200", kind="batch", fe="P1", dim=2, nprob=200, nmin=16, nmax=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["assemble", "assemble", "terms", "script", "cg", "cg", "mixed", "gmres", "adjoint", "batch"])
    if kind == "batch":
        nmin = rng.randint(12, 40)
        return dict(kind=kind, fe="P1", dim=2, nprob=_log(rng, 3, 200), nmin=nmin, nmax=nmin + rng.randint(0, 80))
    if kind == "assemble":
        fe, dim, hi = rng.choice([("P1", 2, 900), ("P1", 3, 88), ("P2", 2, 300), ("P2", 3, 32), ("P2vec", 3, 20)])
    elif kind == "terms":
        fe, dim, hi = rng.choice([("P1", 2, 300), ("P1", 3, 44), ("P2", 2, 120), ("P2", 3, 18)])
    elif kind == "cg":
        fe, dim, hi = rng.choice([("P1", 2, 400), ("P1", 3, 110), ("P2", 3, 24), ("P2vec", 3, 20)])
    elif kind == "mixed":
        fe, dim, hi = rng.choice([("P1", 2, 300), ("P1", 3, 110), ("P2", 3, 24)])
    else:
        fe, dim, hi = "P1", 2, {"script": 250, "gmres": 90, "adjoint": 190}[kind]
    lo = 5 if dim == 2 else 3
    n = _log(rng, lo, hi / 1.1)
    size = [max(lo, int(round(n * rng.uniform(0.85, 1.1)))) for _ in range(dim)] + [0] * (3 - dim)
    case = dict(kind=kind, fe=fe, dim=dim, nx=size[0], ny=size[1], nz=size[2])
    if kind == "cg":
        case["mode"] = 1 if fe != "P1" and rng.random() < 0.4 else 0
    return case


# ------------------------------------------------------------------ inputs (plain torch)
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _grid(*n):
    """Indices of an n[0] x n[1] (x n[2]) grid, the first running fastest."""
    r = torch.meshgrid(*[torch.arange(k, device="cuda") for k in reversed(n)], indexing="ij")
    return [a.reshape(-1) for a in reversed(r)]


def _square(nx, ny, gen, jitter=0.2):
    i, j = _grid(nx + 1, ny + 1)
    X = torch.stack([i.double() / nx, j.double() / ny], 1)
    move = (torch.rand(X.shape, generator=gen, device="cuda", dtype=F64) * 2 - 1) * jitter
    move *= torch.tensor([1.0 / nx, 1.0 / ny], device="cuda", dtype=F64)
    move[(i == 0) | (i == nx) | (j == 0) | (j == ny)] = 0
    a, b = _grid(nx, ny)
    i0 = a + b * (nx + 1)
    E = torch.stack([i0, i0 + 1, i0 + nx + 2, i0, i0 + nx + 2, i0 + nx + 1], 1).reshape(-1, 3)
    ib, jb, w = torch.arange(nx, device="cuda"), torch.arange(ny, device="cuda"), nx + 1
    be = torch.cat([torch.stack([ib, ib + 1], 1), torch.stack([nx + jb * w, nx + jb * w + w], 1),
                    torch.stack([ib + ny * w, ib + ny * w + 1], 1), torch.stack([jb * w, jb * w + w], 1)])
    bl = torch.cat([torch.full((k,), l, device="cuda") for k, l in ((nx, 1), (ny, 2), (nx, 3), (ny, 4))])
    return X + move, E.to(I32), be.to(I32), bl.to(I32)


# the six tetrahedra around the long diagonal of a hexahedron, corner = a + 2 b + 4 c
_HEX = [[0, 1, 3, 7], [0, 5, 1, 7], [0, 3, 2, 7], [0, 2, 6, 7], [0, 4, 5, 7], [0, 6, 4, 7]]


def _cube(nx, ny, nz, gen, jitter=0.1):
    i, j, k = _grid(nx + 1, ny + 1, nz + 1)
    X = torch.stack([i.double() / nx, j.double() / ny, k.double() / nz], 1)
    move = (torch.rand(X.shape, generator=gen, device="cuda", dtype=F64) * 2 - 1) * jitter
    move *= torch.tensor([1.0 / nx, 1.0 / ny, 1.0 / nz], device="cuda", dtype=F64)
    # bits 1 2 4 8 16 32: on x=0, x=1, y=0, y=1, z=0, z=1
    side = ((i == 0) + 2 * (i == nx) + 4 * (j == 0) + 8 * (j == ny) + 16 * (k == 0) + 32 * (k == nz)).to(I64)
    move[side > 0] = 0
    a, b, c = _grid(nx, ny, nz)
    w, h = nx + 1, (nx + 1) * (ny + 1)
    corner = torch.stack([(a + p) + (b + q) * w + (c + r) * h for r in (0, 1) for q in (0, 1) for p in (0, 1)], 1)
    E = corner[:, torch.tensor(_HEX, device="cuda")].reshape(-1, 4)
    be, bl = [], []
    for f in ((1, 2, 3), (0, 3, 2), (0, 1, 3), (0, 2, 1)):
        fv = E[:, list(f)]
        common = side[fv[:, 0]] & side[fv[:, 1]] & side[fv[:, 2]]
        for bit, label in ((1, 4), (2, 2), (4, 1), (8, 3), (16, 5), (32, 6)):
            at = common == bit
            be.append(fv[at])
            bl.append(torch.full((be[-1].shape[0],), label, device="cuda"))
    return X + move, E.to(I32), torch.cat(be).to(I32), torch.cat(bl).to(I32)


_EDGES = {2: [[1, 2], [2, 0], [0, 1]], 3: [[0, 1], [0, 2], [0, 3], [1, 2], [1, 3], [2, 3]]}


def _edge_keys(E, nv, dim):
    a, b = (E.long()[:, [e[s] for e in _EDGES[dim]]] for s in (0, 1))
    return torch.minimum(a, b) * (nv + 1) + torch.maximum(a, b)


def _p2_nodes(E, nv, dim):
    """P2 nodes (vertices, then edges, of every element) numbered by first encounter."""
    keys = torch.cat([E.long() * (nv + 1) + nv, _edge_keys(E, nv, dim)], 1)
    u, inv = torch.unique(keys, return_inverse=True)
    n = u.numel()
    inv = inv.reshape(-1)
    first = torch.full((n,), inv.numel(), device="cuda").scatter_reduce_(0, inv, torch.arange(inv.numel(), device="cuda"), "amin")
    rank = torch.empty_like(first)
    rank[torch.argsort(first)] = torch.arange(n, device="cuda")
    return rank[inv].reshape(keys.shape).to(I32), n


def _inputs(case, seed):
    """Mesh, DOF table and coefficients of a case, from the seed alone."""
    gen = _gen(seed)
    s = dict(case=case, dim=case["dim"])
    if case["kind"] == "batch":
        sizes = np.random.default_rng(12345 + case["nprob"]).integers(case["nmin"], case["nmax"] + 1, case["nprob"])
        parts = [_square(int(n), int(n), gen) for n in sizes]
        s["nv"] = np.array([p[0].shape[0] for p in parts], np.int32)
        s["nt"] = np.array([p[1].shape[0] for p in parts], np.int32)
        s["X"], s["E"] = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
        off = np.concatenate([[0], np.cumsum(s["nv"].astype(np.int64))])
        s["voff"] = off
        s["on"] = torch.zeros(int(off[-1]), dtype=torch.uint8, device="cuda")
        s["on"][torch.cat([p[2].long().reshape(-1) + int(o) for p, o in zip(parts, off)])] = 1
        s["kappa"] = torch.exp(torch.randn(s["E"].shape[0], generator=gen, device="cuda", dtype=F64))
        return s
    if case["dim"] == 2:
        s["X"], s["E"], s["be"], s["bl"] = _square(case["nx"], case["ny"], gen)
    else:
        s["X"], s["E"], s["be"], s["bl"] = _cube(case["nx"], case["ny"], case["nz"], gen)
    nv, nt = s["X"].shape[0], s["E"].shape[0]
    if case["fe"] == "P1":
        s["nodes"], s["nn"] = s["E"], nv
    else:
        s["nodes"], s["nn"] = _p2_nodes(s["E"], nv, case["dim"])
    s["bs"] = 3 if case["fe"] == "P2vec" else 1
    s["n"] = s["nn"] * s["bs"]
    s["kappa"] = torch.exp(torch.randn(nt, generator=gen, device="cuda", dtype=F64))
    s["f"] = 1.0 + 0.5 * torch.randn(nt * s["bs"], generator=gen, device="cuda", dtype=F64)
    s["E_nu"] = (1.0 + float(torch.rand((), generator=gen, device="cuda")), 0.25 + 0.1 * float(torch.rand((), generator=gen, device="cuda")))
    if case["kind"] == "terms":
        s["w"] = 0.3 * torch.randn(nv, generator=gen, device="cuda", dtype=F64)
    if case["kind"] in ("cg", "mixed", "gmres"):
        s["b"] = torch.randn(s["n"], generator=gen, device="cuda", dtype=F64) * s["n"] ** -0.5
    if case["kind"] == "adjoint":
        x, y = s["X"][:, 0], s["X"][:, 1]
        s["u_obs"] = 0.05 * torch.sin(math.pi * x) * torch.sin(math.pi * y) * (1 + 0.01 * torch.randn(nv, generator=gen, device="cuda", dtype=F64))
    return s


# Dirichlet sides of a case.  Assemblies use FreeFEM's tgv = -2 (exact elimination of rows and
# columns), so that no 1e30 hides the other entries; the solves use the default tgv = 1e30.
def _sides(case):
    if case["kind"] == "terms":
        return ()
    if case["fe"] == "P2vec":
        return (4,)
    return (1, 2, 3, 4) if case["dim"] == 2 else (1, 2, 3, 4, 5, 6)


def _varf(s):
    case = s["case"]
    on = _sides(case)
    tgv = -2.0 if case["kind"] == "assemble" else 1e30
    if case["fe"] == "P2vec":
        E, nu = s["E_nu"]
        return ffgpu.varf_elasticity(E=E, nu=nu, f=(0.0, 0.1, -1.0), on=on, tgv=tgv)
    if case["kind"] == "assemble":
        return ffgpu.varf_diffusion(kappa=s["kappa"], f=s["f"], on=on, tgv=tgv, c_mass=0.5 if case["fe"] == "P2" else 0.0)
    if case["kind"] == "terms":
        x, y = ff_expr.x, ff_expr.y
        w = ff_expr.fe("P1", s["w"])
        terms = [("id", "dx", 1.0 + y * w), ("id", "dy", ff_expr.sin(3.0 * x)), ("id", "id", 2.0 + w * w)]
        return ffgpu.varf_diffusion(kappa=s["kappa"], f=ff_expr.exp(-x) * (1.0 + w), terms=terms,
                                    bterms=(ffgpu.BoundaryTerm(labels=(1, 2), robin=3.0, g=0.5),))
    if case["kind"] == "gmres":
        return ffgpu.varf_diffusion(kappa=s["kappa"], f=s["f"], on=on, terms=[("id", "dx", 20.0), ("id", "dy", -7.0)])
    return ffgpu.varf_diffusion(kappa=s["kappa"], f=s["f"], on=on)


def _host_space(s):
    """The FreeFEM space as a script holds it (host mesh and DOF table)."""
    case = s["case"]
    Th = ffgpu.Mesh(case["dim"], *[s[k].cpu().numpy() for k in ("X", "E", "be", "bl")])
    return ffgpu.FESpace(Th, case["fe"], dof=None if case["fe"] == "P1" else s["nodes"].cpu().numpy())


def _space(s):
    """The mesh, the DOF table and the boundary on the device, from resident arrays."""
    return ffgpu.DeviceSpace(s["Vh"], coords=s["X"], elems=s["E"], dof=s["dof"], belems=s["be"], blabel=s["bl"])


# ------------------------------------------------------------------ the passes
def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        s["B"] = ff_batch.Batch(arrays=(s["nv"], s["nt"], s["X"], s["E"], s["on"]))
        s["x"] = torch.empty(int(s["voff"][-1]), dtype=F64, device="cuda")
        torch.cuda.synchronize()
        return s
    s["Vh"] = _host_space(s)
    if case["fe"] == "P2vec":
        n3 = 3 * s["nodes"]
        s["dof"] = torch.cat([n3, n3 + 1, n3 + 2], 1).contiguous()
    else:
        s["dof"] = None if case["fe"] == "P1" else s["nodes"]
    s["rhs"] = torch.zeros(s["n"], dtype=F64, device="cuda")
    torch.cuda.synchronize()
    if kind in ("cg", "mixed", "gmres"):
        s["space"] = _space(s)
        s["A"] = ffgpu.matrix(_varf(s), s["space"], solver="GMRES" if kind == "gmres" else "CG", eps=1e-10, rhs_out=s["rhs"])
        # one load: the assembled source plus a random one off the Dirichlet rows
        s["load"] = s["rhs"] + torch.where(_dirichlet(s), 0.0, s["b"])
    elif kind == "adjoint":
        s["P"] = ff_adjoint.DiffusionProblem(s["Vh"], eps=1e-12)
    torch.cuda.synchronize()
    return s


def _csr(A):
    """[I,J,C] = A on the device, through the C ABI's export."""
    rp = torch.empty(A.n + 1, dtype=I32, device="cuda")
    cl = torch.empty(A.nnz, dtype=I32, device="cuda")
    vl = torch.empty(A.nnz, dtype=F64, device="cuda")
    code = ffgpu.lib().ffgpu_matrix_csr(A.h, rp.data_ptr(), cl.data_ptr(), vl.data_ptr())
    if code:
        raise RuntimeError(ffgpu.lib().ffgpu_last_error())
    return rp, cl, vl


def _from_zero(s):
    """u[] = 0 before the solve; the library works on a stream of its own, so a program lets
    torch finish the fill before it hands the array over."""
    u = torch.zeros(s["n"], dtype=F64, device="cuda")
    torch.cuda.current_stream().synchronize()
    return u


def run(s):
    kind = s["case"]["kind"]
    if kind in ("assemble", "terms"):
        A = ffgpu.matrix(_varf(s), _space(s), rhs_out=s["rhs"])
        rp, cl, vl = _csr(A)
        return {"rowptr": rp, "col": cl, "val": vl, "b": s["rhs"]}
    if kind == "script":
        A = ffgpu.matrix(_varf(s), _space(s), eps=1e-10, rhs_out=s["rhs"])
        return {"b": s["rhs"], "u": A.solve(s["rhs"], out=_from_zero(s))}
    if kind == "cg":
        return {"u": s["A"].solve(s["load"], out=_from_zero(s), spmv_mode=s["case"]["mode"])}
    if kind == "mixed":
        return {"u": s["A"].solve_mixed(s["load"], out=_from_zero(s))}
    if kind == "gmres":
        return {"u": s["A"].solve(s["load"], out=_from_zero(s))}
    if kind == "adjoint":
        loss, gk, gf, u, lam = s["P"].value_and_grad(s["kappa"], 1.0, s["u_obs"])
        return {"loss": loss, "grad_kappa": gk, "grad_f": gf, "u": u, "lam": lam}
    s["B"].assemble(s["kappa"], f=1.0)
    return {"x": s["B"].solve(eps=1e-10, out=s["x"])}


# ------------------------------------------------------------------ work of a pass
def _counts(case):
    """(elements, vertices, DOFs, stored entries, boundary elements) of a case."""
    if case["kind"] == "batch":
        n = np.random.default_rng(12345 + case["nprob"]).integers(case["nmin"], case["nmax"] + 1, case["nprob"]).astype(float)
        return 2 * (n ** 2).sum(), ((n + 1) ** 2).sum(), ((n + 1) ** 2).sum(), (7 * (n + 1) ** 2 - 8 * n - 6).sum(), 4 * n.sum()
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["dim"] == 2:
        nt, nv, nbe = 2 * nx * ny, (nx + 1) * (ny + 1), 2 * (nx + ny)
        edges = 3 * nx * ny + nx + ny
        if case["fe"] == "P1":
            return nt, nv, nv, nv + 2 * edges, nbe
        return nt, nv, nv + edges, 11.5 * (nv + edges), nbe
    nt, nv, nbe = 6 * nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1), 4 * (nx * ny + ny * nz + nx * nz)
    edges = 7 * nx * ny * nz + 3 * (nx * ny + ny * nz + nx * nz) + nx + ny + nz
    if case["fe"] == "P1":
        return nt, nv, nv, nv + 2 * edges, nbe
    nn = nv + edges
    return (nt, nv, 3 * nn, 9 * 28.0 * nn, nbe) if case["fe"] == "P2vec" else (nt, nv, nn, 28.0 * nn, nbe)


def work(case):
    """Assembly: the mesh, the DOF table and the coefficients read, the CSR and b written, the
    element matrices' products.  Solves: a Krylov method has to apply the matrix once per
    iteration; the iteration counts grow with the mesh width (about 2.3/h in 2D, 5/h in 3D with
    lognormal coefficients, 57/h for elasticity to 1e-10)."""
    nt, nv, n, nnz, nbe = _counts(case)
    dim, kind = case["dim"], case["kind"]
    loc = (dim + 1) if case["fe"] == "P1" else (6 if dim == 2 else 10)
    bs = 3 if case["fe"] == "P2vec" else 1
    asm_b = 8.0 * dim * nv + 4.0 * (dim + 1) * nt + (4.0 * loc * bs * nt if case["fe"] != "P1" else 0) + 8.0 * nt * (2 if bs == 1 else 0)
    asm_b += 4.0 * (dim + 1) * nbe + 12.0 * nnz + 4.0 * n + 8.0 * n
    asm_f = nt * (loc * bs) ** 2 * (2.0 * dim + 2.0)
    if kind == "assemble":
        return {"bytes": asm_b, "flops": asm_f}
    if kind == "terms":
        return {"bytes": asm_b + 8.0 * nv, "flops": nt * (14 if dim == 3 else 7) * (3 * 2.0 * loc * loc + 40.0)}
    # solves: values, column numbers and vectors once per iteration
    width = max(case.get("nx", 0), case.get("ny", 0), case.get("nz", 0), case.get("nmax", 0))
    per_b, per_f = (8.0 if kind != "mixed" and kind != "batch" else 4.0) * nnz + 4.0 * nnz / (bs * bs) + 40.0 * n, 2.0 * nnz + 10.0 * n
    its = width * (57.0 if bs == 3 else (5.0 if dim == 3 else 2.6) * (2.0 if case["fe"] == "P2" else 1.0))
    if kind == "script":
        return {"bytes": asm_b - 12.0 * nnz + its * per_b, "flops": asm_f + its * per_f}
    if kind == "adjoint":
        return {"bytes": 2.4 * its * per_b, "flops": 2.4 * its * per_f}
    if kind == "gmres":
        return {"bytes": its * (per_b + 4.0 * its * n), "flops": its * (per_f + 2.0 * its * n)}
    return {"bytes": its * per_b, "flops": its * per_f}


# ------------------------------------------------------------------ plain torch in 64 bits
def _dirichlet(s):
    """The DOFs of on(sides) as a mask."""
    case = s["case"]
    mask = torch.zeros(s["nn"], dtype=torch.bool, device="cuda")
    sides = _sides(case)
    if sides:
        be = s["be"].long()[torch.isin(s["bl"], torch.tensor(sides, device="cuda", dtype=I32))]
        if case["fe"] == "P1":
            mask[be.reshape(-1)] = True
        else:
            nv, nvk = s["X"].shape[0], case["dim"] + 1
            on = torch.zeros(nv, dtype=torch.bool, device="cuda")
            on[be.reshape(-1)] = True
            nodes = s["nodes"].long()
            mask[nodes[:, :nvk][on[s["E"].long()]]] = True
            pairs = [[0, 1]] if case["dim"] == 2 else [[0, 1], [1, 2], [0, 2]]
            bk = torch.cat([torch.minimum(be[:, a], be[:, b]) * (nv + 1) + torch.maximum(be[:, a], be[:, b]) for a, b in pairs])
            mask[nodes[:, nvk:][torch.isin(_edge_keys(s["E"], nv, case["dim"]), bk)]] = True
    return mask.repeat_interleave(s["bs"])


def _geometry(s):
    """Measures and barycentric gradients of the elements."""
    P = s["X"][s["E"].long()]
    J = P[:, 1:] - P[:, :1]
    G = torch.linalg.inv(J).transpose(1, 2)
    G = torch.cat([-G.sum(1, keepdim=True), G], 1)
    return torch.linalg.det(J) / math.factorial(s["dim"]), G


def _basis(fe, dim, G, lam):
    """Values (nq, loc) and gradients (nt, nq, loc, dim) of the local basis at barycentric points."""
    nq = lam.shape[0]
    if fe == "P1":
        return lam, G[:, None].expand(-1, nq, -1, -1)
    a, b = ([e[k] for e in _EDGES[dim]] for k in (0, 1))
    val = torch.cat([lam * (2 * lam - 1), 4 * lam[:, a] * lam[:, b]], 1)
    gv = (4 * lam - 1)[None, :, :, None] * G[:, None]
    ge = 4 * (lam[None, :, a, None] * G[:, None, b] + lam[None, :, b, None] * G[:, None, a])
    return val, torch.cat([gv, ge], 2)


def _rule(dim):
    """The varfs' default rules: 7 points on triangles, 14 on tetrahedra, degree 5."""
    if dim == 2:
        q = math.sqrt(15.0)
        pts, w = [[1 / 3] * 3], [0.225]
        for a, b, c in (((6 - q) / 21, (9 + 2 * q) / 21, (155 - q) / 1200), ((6 + q) / 21, (9 - 2 * q) / 21, (155 + q) / 1200)):
            pts += [[b, a, a], [a, b, a], [a, a, b]]
            w += [c] * 3
    else:
        pts, w = [], []
        for a, b, c in ((0.7217942490673263207930282587889082, 0.0927352503108912264023239137370306, 0.0122488405193936582572850342477212 * 6),
                        (0.067342242210098170607962798709629, 0.310885919263300609797345733763457, 0.0187813209530026417998642753888810 * 6)):
            pts += [[a if i == k else b for i in range(4)] for k in range(4)]
            w += [c] * 4
        a, b = 0.454496295874350350508119473720660, 0.045503704125649649491880526279339
        pts += [[a if i in (k, l) else b for i in range(4)] for k in range(4) for l in range(k + 1, 4)]
        w += [7.09100346284691107301157135337624e-3 * 6] * 6
    return torch.tensor(pts, dtype=F64, device="cuda"), torch.tensor(w, dtype=F64, device="cuda")


def _volume(s, terms, kappa):
    """Element matrices of int(kappa grad u.grad v) + int(coef op_i(v) op_j(u)), by the rule."""
    case = s["case"]
    meas, G = _geometry(s)
    lam, w = _rule(case["dim"])
    if case["fe"] == "P1" and not terms:
        return (kappa * meas)[:, None, None] * (G @ G.transpose(1, 2))
    val, grad = _basis(case["fe"], case["dim"], G, lam)
    ops = lambda o: val[None].expand(grad.shape[0], -1, -1) if o == 0 else grad[..., o - 1]  # noqa: E731
    K = torch.zeros(grad.shape[0], val.shape[1], val.shape[1], dtype=F64, device="cuda")
    for d in range(case["dim"]):
        K += torch.einsum("t,q,tqi,tqj->tij", kappa * meas, w, grad[..., d], grad[..., d])
    for i, j, c in terms:
        K += torch.einsum("tq,tqi,tqj->tij", c * meas[:, None] * w, ops(i), ops(j))
    return K


def _elasticity(s):
    E, nu = s["E_nu"]
    mu, la = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
    meas, G = _geometry(s)
    lam, w = _rule(3)
    _, grad = _basis("P2", 3, G, lam)
    g = torch.einsum("t,q,tqia,tqjb->tiajb", meas, w, grad, grad)
    K = la * g + mu * g.permute(0, 1, 4, 3, 2)
    tr = torch.einsum("tiaja->tij", g)
    for c in range(3):
        K[:, :, c, :, c] += mu * tr
    return K


def _points(s):
    lam, _ = _rule(s["dim"])
    return lam, torch.einsum("qi,tid->tqd", lam, s["X"][s["E"].long()])


def _system(s):
    """(rows, columns, values, b) of a case, coalesced, before the Dirichlet sides."""
    case = s["case"]
    meas, G = _geometry(s)
    nodes, n = s["nodes"].long(), s["n"]
    lam, w = _rule(case["dim"])
    val = _basis(case["fe"] if s["bs"] == 1 else "P2", case["dim"], G[:1], lam)[0]
    if s["bs"] == 3:
        K = _elasticity(s)
        dof = 3 * nodes[:, :, None] + torch.arange(3, device="cuda")
        K, dof = K.reshape(K.shape[0], 30, 30), dof.reshape(-1, 30)
        load = torch.einsum("t,q,qi,c->tic", meas, w, val, torch.tensor([0.0, 0.1, -1.0], dtype=F64, device="cuda")).reshape(-1, 30)
    else:
        dof, terms, f = nodes, [], s.get("f")
        if case["kind"] == "assemble" and case["fe"] == "P2":
            terms = [(0, 0, torch.full((1, 1), 0.5, dtype=F64, device="cuda"))]
        if case["kind"] == "gmres":
            terms = [(0, 1, torch.full((1, 1), 20.0, dtype=F64, device="cuda")), (0, 2, torch.full((1, 1), -7.0, dtype=F64, device="cuda"))]
        if case["kind"] == "terms":
            lam, x = _points(s)
            wq = torch.einsum("qi,ti->tq", lam, s["w"][s["E"].long()])
            terms = [(0, 1, 1.0 + x[..., 1] * wq), (0, 2, torch.sin(3.0 * x[..., 0])), (0, 0, 2.0 + wq * wq)]
            load = torch.einsum("tq,qi->ti", torch.exp(-x[..., 0]) * (1.0 + wq) * meas[:, None] * w, val)
        else:
            load = torch.einsum("t,q,qi->ti", (1.0 if case["kind"] == "adjoint" else f) * meas, w, val)
        K = _volume(s, terms, s["kappa"])
    r = dof[:, :, None].expand_as(K).reshape(-1)
    c = dof[:, None, :].expand_as(K).reshape(-1)
    v = K.reshape(-1)
    b = torch.zeros(n, dtype=F64, device="cuda").index_add_(0, dof.reshape(-1), load.reshape(-1))
    if case["kind"] == "terms":
        # int over the sides 1 and 2 of 3 u v + 0.5 v
        at = (s["bl"] == 1) | (s["bl"] == 2)
        be = s["be"].long()[at]
        size, bd, M, m = _wall(s, be)
        r = torch.cat([r, bd[:, :, None].expand(-1, -1, bd.shape[1]).reshape(-1)])
        c = torch.cat([c, bd[:, None, :].expand(-1, bd.shape[1], -1).reshape(-1)])
        v = torch.cat([v, (3.0 * size[:, None, None] * M).reshape(-1)])
        b.index_add_(0, bd.reshape(-1), (0.5 * size[:, None] * m).reshape(-1))
    key, inv = torch.unique(r * n + c, return_inverse=True)
    v = torch.zeros(key.numel(), dtype=F64, device="cuda").index_add_(0, inv, v)
    return key // n, key % n, v, b


def _wall(s, be):
    """Sizes, nodes, unit mass matrix and unit load of boundary edges or faces."""
    dim = s["dim"]
    P = s["X"][be]
    if dim == 2:
        size = (P[:, 1] - P[:, 0]).norm(dim=1)
        t, w = np.polynomial.legendre.leggauss(4)
        lam = torch.tensor(np.stack([(1 - t) / 2, (1 + t) / 2], 1), device="cuda")
        w = torch.tensor(w / 2, device="cuda")
        edges = [[0, 1]]
    else:
        size = 0.5 * torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]).norm(dim=1)
        lam, w = _rule(2)
        edges = [[0, 1], [1, 2], [0, 2]]
    val, dofs = lam, be
    if s["case"]["fe"] != "P1":
        nv, nvk = s["X"].shape[0], dim + 1
        a, b = ([e[k] for e in edges] for k in (0, 1))
        val = torch.cat([lam * (2 * lam - 1), 4 * lam[:, a] * lam[:, b]], 1)
        vnode = torch.zeros(nv, dtype=I64, device="cuda")
        vnode[s["E"].long()] = s["nodes"].long()[:, :nvk]
        ek = _edge_keys(s["E"], nv, dim).reshape(-1)
        order = torch.argsort(ek)
        bk = torch.minimum(be[:, a], be[:, b]) * (nv + 1) + torch.maximum(be[:, a], be[:, b])
        pos = order[torch.searchsorted(ek[order], bk.reshape(-1).contiguous())]
        dofs = torch.cat([vnode[be], s["nodes"].long()[:, nvk:].reshape(-1)[pos].reshape(bk.shape)], 1)
    return size, dofs, torch.einsum("q,qi,qj->ij", w, val, val), torch.einsum("q,qi->i", w, val)


def _solve(r, c, v, n, b, fixed, symmetric=True):
    """A u = b with u = 0 on the fixed DOFs: CG to the last bits, or a dense solve."""
    free = ~(fixed[r] | fixed[c])
    new = torch.cumsum((~fixed).long(), 0) - 1
    m = int((~fixed).sum())
    r, c, v, f = new[r[free]], new[c[free]], v[free], b[~fixed]
    if not symmetric:
        A = torch.zeros(m, m, dtype=F64, device="cuda")
        A[r, c] = v
        x = torch.linalg.solve(A, f)
        x += torch.linalg.solve(A, f - A @ x)
    else:
        ptr = torch.searchsorted(r.contiguous(), torch.arange(m + 1, device="cuda"))
        A = torch.sparse_csr_tensor(ptr, c, v, (m, m))
        d = torch.zeros(m, dtype=F64, device="cuda")
        d[r[r == c]] = 1.0 / v[r == c]
        x = torch.zeros_like(f)
        for _ in range(3):   # CG, started again on the true residual
            g = f - A @ x
            z = d * g
            h, gz = z, g @ z
            stop = gz * (1e-26 if _ == 0 else 1e-8)
            for it in range(20000):
                q = A @ h
                a = gz / (h @ q)
                x = x + a * h
                g = g - a * q
                z = d * g
                new_gz = g @ z
                if it % 32 == 31 and not float(new_gz) > float(stop):
                    break
                h = z + (new_gz / gz) * h
                gz = new_gz
    u = torch.zeros(n, dtype=F64, device="cuda")
    u[~fixed] = x
    return u


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        s["nn"] = s["n"] = int(s["voff"][-1])
        s["bs"] = 1
        first = torch.as_tensor(np.repeat(s["voff"][:-1], s["nt"]), device="cuda")
        s["E"] = (s["E"].long() + first[:, None]).to(I32)
        s["nodes"] = s["E"]
        s["f"] = torch.ones(s["E"].shape[0], dtype=F64, device="cuda")
        r, c, v, b = _system(s)
        return {"x": _solve(r, c, v, s["n"], b, s["on"].bool())}
    r, c, v, b = _system(s)
    fixed = _dirichlet(s)
    n = s["n"]
    if kind in ("assemble", "terms"):
        gone = fixed[r] | fixed[c]
        v = torch.where(gone, torch.where(r == c, 1.0, 0.0).to(F64), v)
        return {"rowptr": None, "col": None, "val": v, "b": torch.where(fixed, 0.0, b)}
    if kind == "adjoint":
        u = _solve(r, c, v, n, b, fixed)
        meas, G = _geometry(s)
        el = s["E"].long()
        d = u - s["u_obs"]
        local = (d[el].sum(1, keepdim=True) + d[el]) * meas[:, None] / 12.0
        Mr = torch.zeros(n, dtype=F64, device="cuda").index_add_(0, el.reshape(-1), local.reshape(-1))
        lam = _solve(r, c, v, n, Mr, fixed)
        # a Dirichlet row of A is tgv u_i = 0: its multiplier takes M (u - u_obs) / tgv
        K = G @ G.transpose(1, 2)
        gk = -meas * torch.einsum("ti,tij,tj->t", lam[el], K, u[el])
        return {"loss": float(0.5 * d @ Mr), "grad_kappa": gk, "grad_f": meas * lam[el].sum(1) / 3.0, "u": u, "lam": lam}
    if kind == "script":
        return {"b": torch.where(fixed, 0.0, b), "u": _solve(r, c, v, n, b, fixed)}
    load = torch.where(fixed, 0.0, b + s["b"])
    return {"u": _solve(r, c, v, n, load, fixed, symmetric=kind != "gmres")}
