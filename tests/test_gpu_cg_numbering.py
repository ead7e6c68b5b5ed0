"""How a scalar CG solve runs, by pattern: the in-kernel loops and the launches per iteration on both sides
of their lines -- column ranges, long rows, rows of unequal length, sizes -- for meshes numbered along
the grid and at random.

Every solve against the launches per iteration (FFGPU_CLUSTER_CG=0) and its residual with scipy;
iteration counts within 2, the same bits on a second solve and on a second matrix.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import ffgpu
from ffgpu import mesh
from ffgpu.fespace import FESpace

pytestmark = pytest.mark.gpu

THREE, TWO, BAND, WIDE, LOOP = 1, 2, 4, 5, 6


@pytest.fixture(scope="module", autouse=True)
def _lib_built():
    from ffgpu.build import build
    build()
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    ffgpu.context(0)
    yield


def _grid(*shape):
    """Five- or seven-point matrix with lognormal couplings, symmetric positive definite."""
    n = int(np.prod(shape))
    idx = np.arange(n).reshape(shape)
    rng = np.random.Generator(np.random.PCG64(n))
    i, j = [], []
    for d in range(len(shape)):
        a, b = np.take(idx, range(shape[d] - 1), d).ravel(), np.take(idx, range(1, shape[d]), d).ravel()
        i.append(a)
        j.append(b)
    i, j = np.concatenate(i), np.concatenate(j)
    w = np.exp(rng.standard_normal(i.size))
    K = sp.coo_matrix((-w, (i, j)), (n, n))
    K = K + K.T
    return (K + sp.diags(-np.asarray(K.sum(1)).ravel() + 0.01)).tocsr()


def _renumber(S, width=None):
    """Rows and columns renumbered at random, in pieces of ``width``."""
    n = S.shape[0]
    rng = np.random.Generator(np.random.PCG64(1))
    p = np.arange(n)
    for o in range(0, n, width or n):
        p[o:o + (width or n)] = rng.permutation(p[o:o + (width or n)])
    return S[p][:, p]


def _long_row(S, k):
    n = S.shape[0]
    c = np.unique(np.linspace(1, n - 1, k).astype(int))
    T = sp.coo_matrix((np.full(c.size, 1e-3 / c.size), (np.zeros(c.size, int), c)), (n, n))
    return S + T + T.T


def _check(S, path, monkeypatch, trans=False):
    S = S.tocsr()
    S.sort_indices()
    args = S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data
    A = ffgpu.matrix_from_csr(*args, eps=1e-9)
    b = np.random.Generator(np.random.PCG64(3)).standard_normal(S.shape[0])
    u = A.solve(b, trans=trans)
    its = A.stats.iterations
    assert A.layout_code(6) == path
    assert np.array_equal(A.solve(b, trans=trans), u)
    B = ffgpu.matrix_from_csr(*args, eps=1e-9)
    assert np.array_equal(B.solve(b, trans=trans), u)
    monkeypatch.setenv("FFGPU_CLUSTER_CG", "0")
    v = B.solve(b, trans=trans)
    assert B.layout_code(6) in (THREE, TWO) and abs(B.stats.iterations - its) <= 2
    d = S.diagonal()
    for x in (u, v):
        r = S @ x - b
        # the stopping test, (r, C r) < eps^2 (r0, C r0), with room for the recurrence's drift
        assert r @ (r / d) <= 4 * 1e-18 * (b @ (b / d))


@pytest.mark.parametrize("m,width,path", [(20, None, BAND), (44, None, BAND), (48, None, WIDE), (70, None, WIDE), (165, None, WIDE), (255, None, WIDE),
                                          (277, 4000, WIDE), (401, None, WIDE), (401, 2000, BAND), (540, None, WIDE)])
def test_square_grids_numbered_at_random(m, width, path, monkeypatch):
    """Rows per block 64 (one block and several), 192, 448, 512, 1088 and 1920; ranges of 15 and 18 columns per
    thread around the line at 16, and 31 and 62 around the one by entries."""
    _check(_renumber(_grid(m, m), width), path, monkeypatch)


def test_transposed_and_nonsymmetric_values(monkeypatch):
    S = _renumber(_grid(90, 91)).tocoo()
    S.data = S.data * (1 + 1e-3 * np.sin(np.arange(S.nnz)))
    S = S.tocsr()
    _check(0.5 * (S + S.T), WIDE, monkeypatch, trans=True)


def test_cubes_along_the_grid_and_at_random(monkeypatch):
    _check(_grid(59, 60, 61), BAND, monkeypatch)          # 33 columns and 38 entries per thread
    monkeypatch.delenv("FFGPU_CLUSTER_CG")
    _check(_renumber(_grid(30, 31, 29)), WIDE, monkeypatch)


@pytest.mark.parametrize("k,path", [(60, WIDE), (88, WIDE), (120, TWO), (400, THREE)])
def test_one_long_row(k, path, monkeypatch):
    """The longest row the wide form takes is 96; with 400 entries the layout has eight lanes per row, more partial
    sums than the two-launch iteration holds."""
    S = _long_row(_grid(300, 301), k)
    if path == THREE:
        S = S.tocsr()
        S.sort_indices()
        A = ffgpu.matrix_from_csr(S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data, eps=1e-9)
        b = np.random.Generator(np.random.PCG64(3)).standard_normal(S.shape[0])
        monkeypatch.setenv("FFGPU_CLUSTER_CG", "0")
        u = A.solve(b)
        assert A.layout_code() in (1, 2, 4, 8) and A.layout_code(6) in (TWO, THREE)
        assert np.linalg.norm(S @ u - b) <= 1e-6 * np.linalg.norm(b)
        monkeypatch.delenv("FFGPU_CLUSTER_CG")
        v = A.solve(b)
        assert np.linalg.norm(S @ v - b) <= 1e-6 * np.linalg.norm(b)
        return
    _check(S, path, monkeypatch)


def test_long_row_of_a_small_system_is_staged(monkeypatch):
    _check(_long_row(_grid(60, 61), 500), BAND, monkeypatch)


@pytest.mark.parametrize("n,kinds", [((9, 8, 10), (BAND,)), ((20, 21, 19), (BAND, WIDE))])
def test_rows_of_unequal_length(n, kinds, monkeypatch):
    """P2 on tetrahedra, rows of 10 to 65 entries: 32 consecutive rows padded to the longest fit the SMs on the
    smaller mesh, on the larger one they are taken by length."""
    Vh = FESpace(mesh.cube(*n), "P2")
    A = ffgpu.matrix(ffgpu.varf_diffusion(f=1.0, on=(1, 2), c_mass=1.0, tgv=-2), Vh)
    rp, cl, vl = A.csr()
    S = sp.csr_matrix((vl, cl, rp))
    x = np.random.Generator(np.random.PCG64(3)).standard_normal(S.shape[0])
    A.solve(x, eps=1e-9)
    assert A.layout_code(6) in kinds
    _check(S, A.layout_code(6), monkeypatch)
    monkeypatch.delenv("FFGPU_CLUSTER_CG")
    _check(_renumber(S), WIDE, monkeypatch)


def test_streamed_where_the_numbering_is_local(monkeypatch):
    """P1 on 62^3 cells past the SMs' shared memory: streamed along the grid, launches numbered at random."""
    Th = mesh.cube(62)
    A = ffgpu.matrix(ffgpu.varf_diffusion(f=1.0, on=(1, 2), c_mass=1.0, tgv=-2), FESpace(Th, "P1"))
    rp, cl, vl = A.csr()
    S = sp.csr_matrix((vl, cl, rp))
    A = ffgpu.matrix_from_csr(rp, cl, vl, eps=1e-9)
    A.solve(np.ones(A.n))
    # (where the layout tuner takes block CSR, which it hardly does here, the launches run)
    _check(S, LOOP if A.layout_code() >= 64 else THREE, monkeypatch)
    monkeypatch.delenv("FFGPU_CLUSTER_CG")
    _check(_renumber(S), THREE, monkeypatch)
