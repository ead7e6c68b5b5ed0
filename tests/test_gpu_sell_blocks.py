"""The 3x3-block SELL layout: four lanes per row and one block of 32 warps per SM (single chunks per
unit), and the one-lane form with units of eight above 300 000 block rows, for every kernel that
reads it -- FP64, double-float and FP32 products, both assignments, all row loops, A and A'.

y = A x against scipy on the exported matrix: a row sums at most 3 x 195 products in another order,
so 600 ulp of the row's absolute sum.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import ffgpu
from ffgpu.fespace import FESpace
from ffgpu.mesh import cube

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_built():
    from ffgpu.build import build
    build()
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    ffgpu.context(0)
    yield


def _elasticity(n):
    Vh = FESpace(cube(*n), "P2vec")
    b = np.empty(Vh.ndof)
    A = ffgpu.matrix(ffgpu.varf_elasticity(on=(4,), tgv=-2), Vh, eps=1e-10, rhs_out=b)
    rp, cl, vl = A.csr()
    return A, b, sp.csr_matrix((vl, cl, rp), (A.n, A.n))


@pytest.mark.parametrize("n", [(1, 1, 1), (2, 1, 3), (5, 4, 6)])
@pytest.mark.parametrize("code", range(64, 72))
def test_products_and_solutions_of_every_layout(n, code):
    A, b, S = _elasticity(n)
    u = A.solve(b, spmv_layout=code)
    assert A.layout_code() == code
    assert np.linalg.norm(S @ u - b) <= 1e-8 * np.linalg.norm(b)
    x = np.random.Generator(np.random.PCG64(1)).standard_normal(A.n)
    assert np.all(np.abs(A.mult(x) - S @ x) <= 600 * 2.2e-16 * (abs(S) @ np.abs(x)) + 1e-300)
    t = A.solve(b, trans=True, spmv_layout=code)
    assert np.linalg.norm(t - u) <= 1e-8 * np.linalg.norm(u)
    if code < 68:
        d = A.solve(b, spmv_mode=1, spmv_layout=code)
        assert np.linalg.norm(d - u) <= 1e-8 * np.linalg.norm(u)


def test_mixed_precision_on_the_block_layout():
    A, b, S = _elasticity((4, 5, 3))
    u = A.solve_mixed(b)
    assert np.linalg.norm(S @ u - b) <= 1e-8 * np.linalg.norm(b)


def test_one_lane_per_row_above_the_limit():
    """340 071 block rows: products of the device space's matrix against its rigid translations and
    against the block-CSR kernel (a fixed layout) on the same matrix."""
    import torch
    sp_ = ffgpu.device_space("P2vec", 3, 34, 35, 35)
    b = torch.zeros(sp_.Vh.ndof, dtype=torch.float64, device="cuda")
    A = ffgpu.matrix(ffgpu.varf_elasticity(on=(4,)), sp_, eps=1e-4, rhs_out=b)
    assert A.n // 3 > 300000
    x = torch.sin(torch.arange(A.n, device="cuda", dtype=torch.float64))
    A.solve(b, spmv_layout=65)
    y = A.mult(x)
    A.solve(b, spmv_layout=4)
    z = A.mult(x)
    free = z.abs() < 1e20
    assert float((y - z)[free].abs().max()) <= 600 * 2.2e-16 * float(z[free].abs().max()) * 40


@pytest.mark.parametrize("n", [(9, 10, 11), (14, 14, 13)])
def test_small_block_matrices_take_block_csr(n):
    """9 177 and 22 707 block rows: past the size that is tuned, below the one where SELL is timed."""
    A, b, S = _elasticity(n)
    u = A.solve(b)
    assert A.layout_code() in (1, 2, 4, 8)
    assert np.linalg.norm(S @ u - b) <= 1e-8 * np.linalg.norm(b)
