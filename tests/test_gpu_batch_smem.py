"""The batched solver in shared memory (batch_sm_kernel) at the edges of its dispatch and its packed
rows: problems smaller than a warp, row counts around multiples of 32 and of the CTA, long rows
(a hub node), the largest problem that fits next to small ones, and one that does not (the
general kernel).

Each problem against a sparse direct solution of its own matrix; eps = 1e-10 on the residual leaves
errors far below the 1e-8 the batched solver is held to elsewhere.
"""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

import ffgpu
from ffgpu import batch, mesh
from ffgpu.fespace import FESpace
from ffgpu.mesh import Mesh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_built():
    from ffgpu.build import build
    build()
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    ffgpu.context(0)
    yield


def _fan(n):
    t = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(t), np.sin(t)], 1)
    X = np.concatenate([[[0.0, 0.0]], 0.5 * ring, ring])
    i, j = np.arange(n), (np.arange(n) + 1) % n
    E = np.concatenate([np.stack([0 * i, 1 + i, 1 + j], 1), np.stack([1 + i, 1 + n + i, 1 + n + j], 1),
                        np.stack([1 + i, 1 + n + j, 1 + j], 1)])
    return Mesh(2, X, E.astype(np.int32), np.stack([1 + n + i, 1 + n + j], 1).astype(np.int32), np.ones(n, np.int32))


def _check(meshes, seed=0):
    rng = np.random.Generator(np.random.PCG64(seed))
    kappas = [np.exp(rng.standard_normal(m.nt)) for m in meshes]
    B = batch.Batch(meshes)
    for _ in range(2):   # the second assembly keeps the packed pattern
        B.assemble(kappas, f=1.0)
        x = B.solve(eps=1e-10)
    assert np.array_equal(B.solve(eps=1e-10), x)
    for m, k, xp in zip(meshes, kappas, B.split(x)):
        b = np.empty(m.nv)
        A = ffgpu.matrix(ffgpu.varf_diffusion(kappa=k, f=1.0, on=(1, 2, 3, 4), tgv=-2), FESpace(m, "P1"), rhs_out=b)
        rp, cl, vl = A.csr()
        u = spl.spsolve(sp.csc_matrix(sp.csr_matrix((vl, cl, rp), (m.nv, m.nv))), b)
        assert np.linalg.norm(xp - u) <= 1e-8 * np.linalg.norm(u)
    return B


def test_small_and_odd_problems():
    sq = [mesh.square(a, b) for a, b in ((2, 2), (3, 3), (4, 5), (7, 3), (30, 30), (31, 31), (32, 31), (45, 22))]
    _check(sq + [_fan(9), _fan(120)])


def test_largest_that_fits_and_one_that_does_not():
    B = _check([mesh.square(137, 137), mesh.square(5, 6), mesh.square(64, 64)])
    assert B.tuned()[0] == 1024
    _check([mesh.square(138, 139), mesh.square(5, 6)])


@pytest.mark.parametrize("n", [67, 68, 95, 96])
def test_sizes_around_the_smaller_ctas(n):
    """4 624 to 4 761 rows: four CTAs of 256 threads; to 9 409: two of 512."""
    _check([mesh.square(n, n), mesh.square(n // 2, n)], seed=n)
