"""The 3x3-block layout where chunks go round the SMs in units of eight (from 4864 chunks on) with a
remainder, and with one lane per row (above 300 000 block rows): every kernel that walks it -- stride
and staged, FP64, double-float and FP32.

Solutions by their residual, against the exported matrix or the block-CSR product: eps = 1e-8 bounds the
preconditioned residual; the plain one is within the square root of the diagonal's spread (below 100
here) of it, 1e-6.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import ffgpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_built():
    from ffgpu.build import build
    build()
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    ffgpu.context(0)
    yield


def _elasticity(*n):
    import torch
    S = ffgpu.device_space("P2vec", 3, *n)
    b = torch.zeros(S.Vh.ndof, dtype=torch.float64, device="cuda")
    A = ffgpu.matrix(ffgpu.varf_elasticity(on=(4,), tgv=-2), S, eps=1e-8, rhs_out=b)
    return A, b, S


@pytest.mark.parametrize("mode,code", [(0, 65), (0, 67), (0, 71), (1, 65), (1, 67), (2, 0)])
def test_units_of_eight(mode, code):
    A, b, S = _elasticity(17, 16, 17)
    assert 38912 < A.n // 3 < 300000 and -(-(A.n // 3) // 8) % 8 and -(-(A.n // 3) // 8) >= 4864
    rp, cl, vl = A.csr()
    M = sp.csr_matrix((vl, cl, rp), (A.n, A.n))
    x = np.random.Generator(np.random.PCG64(1)).standard_normal(A.n)
    if mode == 2:
        u = A.solve_mixed(b)
    else:
        u = A.solve(b, spmv_mode=mode, spmv_layout=code)
        assert A.layout_code(mode) == code
    r = M @ u.cpu().numpy() - b.cpu().numpy()
    assert np.linalg.norm(r) <= 1e-6 * float(b.norm())
    if mode == 0:
        assert np.all(np.abs(A.mult(x) - M @ x) <= 600 * 2.2e-16 * (abs(M) @ np.abs(x)) + 1e-300)


@pytest.mark.parametrize("mode,code", [(0, 71), (1, 67), (2, 0)])
def test_one_lane_per_row(mode, code):
    A, b, S = _elasticity(34, 35, 35)
    assert A.n // 3 > 300000
    B = ffgpu.matrix(ffgpu.varf_elasticity(on=(4,), tgv=-2), S, eps=1e-2)
    B.solve(b, spmv_layout=4)   # block CSR
    if mode == 2:
        u = A.solve_mixed(b)
    else:
        u = A.solve(b, spmv_mode=mode, spmv_layout=code)
        assert A.layout_code(mode) == code
    assert float((B.mult(u) - b).norm() / b.norm()) <= 1e-6
