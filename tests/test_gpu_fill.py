"""The pattern and the numeric fill (pattern_kernel, p1_elem_kernel, fill_kernel) where they change
shape: fewer rows than a warp holds, a hub node whose long row shrinks the blocks, the two forms
of the fill (complete element matrices or terms to add), and every tgv < 0 variant.

Bars: pattern and numbering equal to the oracle's, values to 1e-12 of the larger of the entry and
1e-3 of its row's largest (the assembly's bar), a reassembly bit for bit.
"""
import numpy as np
import pytest

import ffgpu
import ffo
from ffgpu.fespace import FESpace
from ffgpu.mesh import Mesh, cube, square

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_built():
    from ffgpu.build import build
    build()
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    ffgpu.context(0)
    yield


def fan(n):
    """n triangles around one hub."""
    t = 2 * np.pi * np.arange(n) / n
    X = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(t), np.sin(t)], 1) * (1 + 0.1 * np.cos(5 * t))[:, None]])
    i = np.arange(n)
    E = np.stack([0 * i, 1 + i, 1 + (i + 1) % n], 1)
    return Mesh(2, X, E.astype(np.int32), np.stack([1 + i, 1 + (i + 1) % n], 1).astype(np.int32), np.ones(n, np.int32))


def cone(n):
    """n tetrahedra around one edge."""
    F = fan(n)
    X = np.concatenate([np.c_[F.coords, np.zeros(n + 1)], [[0.1, 0.0, 1.0]]])
    E = np.c_[F.elems, np.full(n, n + 1)]
    return Mesh(3, X, E.astype(np.int32), F.elems.copy(), np.ones(n, np.int32))


def one(dim):
    X = np.concatenate([np.zeros((1, dim)), np.eye(dim)]) + 0.05 * np.arange(dim + 1)[:, None]
    return Mesh(dim, X, np.arange(dim + 1, dtype=np.int32)[None], np.arange(dim, dtype=np.int32)[None], np.ones(1, np.int32))


MESHES = {"one2": one(2), "one3": one(3), "fan128": fan(128), "fan9": fan(9), "cone25": cone(25), "cone100": cone(100),
          "square1": square(1), "square3x2": square(3, 2), "cube1": cube(1), "cube3x1x2": cube(3, 1, 2)}


def _close(A, Ao):
    rp, cl, v = A.csr()
    ro, co, vo = Ao.csr()
    assert np.array_equal(rp, ro) and np.array_equal(cl, co)
    row = np.repeat(np.arange(rp.size - 1), np.diff(rp))
    top = np.zeros(rp.size - 1)
    np.maximum.at(top, row, np.abs(vo))
    assert np.all(np.abs(v - vo) <= 1e-12 * np.maximum(np.abs(vo), 1e-3 * top[row]))


@pytest.mark.parametrize("kind", ["P1", "P2", "P2vec"])
@pytest.mark.parametrize("name", sorted(MESHES))
def test_edges_against_the_oracle(name, kind):
    Th = MESHES[name]
    nn = {"P1": Th.dim + 1, "P2": 10 if Th.dim == 3 else 6, "P2vec": 10}[kind]
    if kind == "P2vec" and Th.dim == 2:
        pytest.skip("[P2,P2,P2] is provided on tetrahedra")
    if int(np.bincount(Th.elems.ravel()).max()) * nn > 512:
        pytest.skip("above the supported node valence")
    Vh = FESpace(Th, kind)
    kappa = np.exp(np.random.Generator(np.random.PCG64(1)).standard_normal(Th.nt))
    forms = [dict(kappa=kappa), dict(kappa=kappa, c_mass=0.7)] if kind != "P2vec" else [{}]
    for f in forms:
        va = ffgpu.varf_elasticity(E=1.3, nu=0.2) if kind == "P2vec" else ffgpu.varf_diffusion(**f)
        A = ffgpu.matrix(va, Vh)
        Ao = (ffo.assemble(Th, Vh, form="elasticity", E=1.3, nu=0.2) if kind == "P2vec"
              else ffo.assemble(Th, Vh, kappa=f["kappa"], mass=f.get("c_mass", 0.0)))
        _close(A, Ao)
        v = A.csr()[2]
        A.reassemble(va)
        assert np.array_equal(A.csr()[2], v)


@pytest.mark.parametrize("kind", ["P1", "P2"])
def test_added_terms_are_the_sum_of_their_matrices(kind):
    """The general form of the fill: a mass coefficient at points plus general terms on top of the
    stiffness equals the matrices of the parts (exact sums of at most three rounded terms)."""
    Th = cube(3, 2, 2)
    Vh = FESpace(Th, kind)
    kappa = np.exp(np.random.Generator(np.random.PCG64(2)).standard_normal(Th.nt))
    c = lambda x, y, z: 1.0 + x * y  # noqa: E731
    t = [("id", "dx", 2.0)]
    whole = ffgpu.matrix(ffgpu.varf_diffusion(kappa=kappa, c_mass=c, terms=t), Vh).csr()
    parts = [ffgpu.matrix(v, Vh).csr() for v in (ffgpu.varf_diffusion(kappa=kappa), ffgpu.varf_diffusion(c_stiff=0.0, c_mass=c),
                                                 ffgpu.varf_diffusion(c_stiff=0.0, terms=t))]
    for p in parts:
        assert np.array_equal(p[0], whole[0]) and np.array_equal(p[1], whole[1])
    total = sum(p[2] for p in parts)
    scale = sum(np.abs(p[2]) for p in parts).max()
    # each entry sums at most 24 elements of three rounded terms: (3 * 24 + 3) ulp of the largest
    assert np.abs(whole[2] - total).max() <= 75 * 2.2e-16 * scale


@pytest.mark.parametrize("kind", ["P1", "P2vec"])
@pytest.mark.parametrize("tgv", [1e30, -1, -2, -3, -10, -20, -30])
def test_dirichlet_variants(kind, tgv):
    """HashMatrix::SetBC: rows unit (0 from -10 on), off-diagonals zero unless -3/-30, the columns
    too for -2/-20/-3/-30 (with the diagonal for -20/-30)."""
    Th = cube(2, 3, 2)
    Vh = FESpace(Th, kind)
    make = lambda **k: ffgpu.varf_elasticity(**k) if kind == "P2vec" else ffgpu.varf_diffusion(c_mass=0.3, **k)  # noqa: E731
    rp, cl, v = ffgpu.matrix(make(), Vh).csr()
    got = ffgpu.matrix(make(on=(1, 4), tgv=tgv), Vh).csr()[2]
    on = Vh.on((1, 4)).astype(bool)
    row = np.repeat(np.arange(rp.size - 1), np.diff(rp))
    diag = row == cl
    want = v.copy()
    if tgv > 0:
        want[diag & on[row]] = tgv
    else:
        if tgv not in (-3, -30):
            want[on[row] & ~diag] = 0.0
        want[on[row] & diag] = 0.0 if tgv <= -10 else 1.0
        if tgv in (-2, -3, -20, -30):
            want[on[cl] & (~diag | (tgv <= -20))] = 0.0
    assert np.array_equal(got, want)
