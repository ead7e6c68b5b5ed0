"""FGMRES where its kernels change shape: 32, 64, 128 and 256 rows per block of the update (by the
size), sub-tiles of 512 elements with a remainder, columns longer than a block of the back
substitution and than the staged Hessenberg column, restarts.

Bar: the residual FreeFEM's test promises, ||b - A u|| < eps ||b|| off the tgv rows; the recurrence's
estimate and the true residual part by rounding only, so 10 eps leaves a wide margin at eps = 1e-10.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import ffgpu
from ffgpu.fespace import FESpace
from ffgpu.mesh import square

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_built():
    from ffgpu.build import build
    build()
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    ffgpu.context(0)
    yield


@pytest.mark.parametrize("n,restart", [(2, 1000), (15, 1000), (70, 1000), (71, 40), (98, 1000), (98, 3), (139, 1000), (200, 1000), (200, 150)])
def test_residual(n, restart):
    Th = square(n, n + 1)
    Vh = FESpace(Th, "P1")
    b = np.empty(Vh.ndof)
    a = ffgpu.varf_diffusion(f=1.0, on=(1, 2, 3, 4), terms=[("id", "dx", 25.0), ("id", "dy", -8.0)])
    A = ffgpu.matrix(a, Vh, solver="GMRES", eps=1e-10, dim_krylov=restart, itmax=40000, rhs_out=b)
    u = A.solve(b)
    rp, cl, vl = A.csr()
    S = sp.csr_matrix((vl, cl, rp), (A.n, A.n))
    free = S.diagonal() < 1e20
    assert np.linalg.norm((b - S @ u)[free]) <= 1e-9 * np.linalg.norm(b)
    assert np.array_equal(A.solve(b), u)


def test_long_column():
    """More than 1024 iterations in one cycle (the staged column's length) and 512 (the threads of the
    back substitution): Poisson with a rough coefficient, restart 1500."""
    Th = square(150)
    Vh = FESpace(Th, "P1")
    kappa = np.exp(2.5 * np.random.Generator(np.random.PCG64(1)).standard_normal(Th.nt))
    b = np.empty(Vh.ndof)
    A = ffgpu.matrix(ffgpu.varf_diffusion(kappa=kappa, f=1.0, on=(1, 2, 3, 4)), Vh, solver="GMRES", eps=1e-10,
                     dim_krylov=1500, rhs_out=b)
    u = A.solve(b)
    assert A.stats.iterations > 1024
    rp, cl, vl = A.csr()
    S = sp.csr_matrix((vl, cl, rp), (A.n, A.n))
    free = S.diagonal() < 1e20
    assert np.linalg.norm((b - S @ u)[free]) <= 1e-9 * np.linalg.norm(b)


def test_one_vector_cycles():
    """Restarts after every step: the cycle's only step is finished by the step that is not taken."""
    Th = square(2, 3)
    Vh = FESpace(Th, "P1")
    b = np.empty(Vh.ndof)
    A = ffgpu.matrix(ffgpu.varf_diffusion(f=1.0, on=(1, 2, 3, 4)), Vh, solver="GMRES", eps=1e-10, dim_krylov=1,
                     itmax=40000, rhs_out=b)
    u = A.solve(b)
    rp, cl, vl = A.csr()
    S = sp.csr_matrix((vl, cl, rp), (A.n, A.n))
    free = S.diagonal() < 1e20
    assert np.linalg.norm((b - S @ u)[free]) <= 1e-9 * np.linalg.norm(b)
