"""The FP32 layout of the mixed-precision solver is timed for each numbering: a matrix of a mesh numbered at
random does not take the choice made for the same mesh numbered along the grid."""
import numpy as np
import pytest
import scipy.sparse as sp

import ffgpu
from ffgpu import mesh
from ffgpu.fespace import FESpace

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_built():
    from ffgpu.build import build
    build()
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    ffgpu.context(0)
    yield


def test_each_numbering_is_timed(monkeypatch, capfd):
    Th = mesh.cube(37, 38, 39)   # 59 280 rows: random neighbours are more than 2^15 apart
    A = ffgpu.matrix(ffgpu.varf_diffusion(f=1.0, on=(1, 2), c_mass=1.0, tgv=-2), FESpace(Th, "P1"))
    rp, cl, vl = A.csr()
    S = sp.csr_matrix((vl, cl, rp), (A.n, A.n))
    p = np.random.Generator(np.random.PCG64(2)).permutation(A.n)
    b = np.random.Generator(np.random.PCG64(3)).standard_normal(A.n)
    monkeypatch.setenv("FFGPU_VERBOSE", "1")
    timed = []
    for q in (np.arange(A.n), p, p):
        T = S[q][:, q].tocsr()
        T.sort_indices()
        M = ffgpu.matrix_from_csr(T.indptr.astype(np.int32), T.indices.astype(np.int32), T.data, eps=1e-8)
        capfd.readouterr()
        u = M.solve_mixed(b[q])
        timed.append("FP32 SpMV tuner" in capfd.readouterr().err)
        assert np.linalg.norm(T @ u - b[q]) <= 1e-6 * np.linalg.norm(b)
    assert timed == [True, True, False]
