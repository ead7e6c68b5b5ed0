"""The initial residual of a CG solve is summed in the order of the matrix's own SpMV layout, whatever
ran before: a warm-started solve gives the same bits the first and the second time, on a matrix that
was reassembled, and on another matrix of the same shape, for A and A', on every size class of the
scalar loops (untimed layout, tuned layout, vectors streamed).  So does a product after a solve.
"""
import numpy as np
import pytest

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


@pytest.mark.parametrize("kind,Th", [("P1", mesh.square(30, 23)), ("P1", mesh.square(151, 140)), ("P2", mesh.cube(9, 8, 10)),
                                     ("P1", mesh.cube(59, 60, 62))], ids=["untimed", "tuned", "tuned_p2", "streamed"])
def test_warm_start_gives_the_same_bits(kind, Th):
    Vh = FESpace(Th, kind)
    rng = np.random.Generator(np.random.PCG64(7))
    kappa, x0, b = np.exp(rng.standard_normal(Th.nt)), rng.standard_normal(Vh.ndof), rng.standard_normal(Vh.ndof)
    a = ffgpu.varf_diffusion(kappa=kappa, f=1.0, on=(1, 2), c_mass=1.0)
    S = ffgpu.DeviceSpace(Vh)
    A = ffgpu.matrix(a, S, eps=1e-6)
    want, prod = {}, {}
    for trans in (False, True):
        want[trans] = A.solve(b, x0=x0, trans=trans)
        assert np.array_equal(A.solve(b, x0=x0, trans=trans), want[trans]), "second solve"
        prod[trans] = A.mult(x0, trans=trans)
    A.reassemble(a)
    B = ffgpu.matrix(a, S, eps=1e-6)
    for M, what in ((A, "reassembled"), (B, "another matrix of the shape")):
        for trans in (False, True):
            assert np.array_equal(M.solve(b, x0=x0, trans=trans), want[trans]), what
            assert np.array_equal(M.mult(x0, trans=trans), prod[trans]), what + ", product"
