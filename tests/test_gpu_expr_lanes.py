"""The terms kernel (terms_kernel) at the edges of its lanes: element counts that leave a warp
part empty, and so many terms that a warp's coefficients are taken in several chunks of points.

A form of many terms equals the sum of its terms' matrices: each entry sums at most 24 elements of
`count` terms of 14 points, so the two differ by rounding of at most 24 * 14 * count ulp of the largest sum.
"""
import numpy as np
import pytest

import ffgpu
from ffgpu.expr import cos, exp, x, y
from ffgpu.fespace import FESpace
from ffgpu.mesh import cube, square

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_built():
    from ffgpu.build import build
    build()
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    ffgpu.context(0)
    yield


@pytest.mark.parametrize("count", [1, 5, 16])
@pytest.mark.parametrize("kind", ["P1", "P2"])
@pytest.mark.parametrize("Th", [square(1, 1), square(5, 3), cube(1), cube(1, 2, 1)], ids=["tri2", "tri30", "tet6", "tet12"])
def test_many_terms_are_the_sum_of_their_matrices(Th, kind, count):
    Vh = FESpace(Th, kind)
    ops = ["id", "dx", "dy"] + (["dz"] if Th.dim == 3 else [])
    coef = [1.0 + x * y, 2.0, exp(-x), cos(y) - x]
    terms = [(ops[(3 * k) % len(ops)], ops[(k + k // 4) % len(ops)], coef[k % 4]) for k in range(count)]
    whole = ffgpu.matrix(ffgpu.varf_diffusion(c_stiff=0.0, terms=terms), Vh).csr()[2]
    parts = [ffgpu.matrix(ffgpu.varf_diffusion(c_stiff=0.0, terms=[t]), Vh).csr()[2] for t in terms]
    scale = sum(np.abs(p) for p in parts).max()
    assert np.abs(whole - sum(parts)).max() <= 24 * 14 * count * 2.2e-16 * scale

