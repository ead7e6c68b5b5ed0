"""Short restarts of FGMRES: a full cycle of m steps launches the kernels of m steps (four launches frame a
cycle, five make a step), the host-driven loop gives the graph's bits, and the solution is the oracle's.
"""
import numpy as np
import pytest

import ffgpu
import ffo
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


@pytest.mark.parametrize("m", [1, 2, 3, 7])
@pytest.mark.parametrize("n", [6, 40])
def test_short_restarts(n, m, monkeypatch):
    Th = mesh.square(n, n + 1)
    Vh = FESpace(Th, "P1")
    kappa = np.exp(0.3 * np.random.Generator(np.random.PCG64(4)).standard_normal(Th.nt))
    c = 400.0 * n / 6   # a strong mass term: restarts converge in tens of cycles
    Ao = ffo.assemble(Th, Vh, kappa=kappa, mass=c)
    bo = ffo.rhs(Th, Vh, f=1.0)
    ffo.setbc(Ao, bo, Vh.on((1, 2, 3, 4)))
    uo, ito, conv, _ = ffo.fgmres(Ao, bo, eps=1e-10, restart=m)
    assert conv
    b = np.empty(Vh.ndof)
    A = ffgpu.matrix(ffgpu.varf_diffusion(kappa=kappa, c_mass=c, f=1.0, on=(1, 2, 3, 4)), Vh, solver="GMRES", eps=1e-10,
                     dim_krylov=m, rhs_out=b)
    u = A.solve(b)
    l0 = ffgpu.kernel_launches()
    assert np.array_equal(A.solve(b), u)
    launches, it = ffgpu.kernel_launches() - l0, A.stats.iterations
    cycles = it // m + 1
    # a step more where the last cycle stops early; the start of the solve
    assert launches <= 4 * cycles + 5 * (it + 2) + 8, (launches, it, cycles)
    assert abs(it - ito) <= max(2, 0.05 * ito)
    assert np.linalg.norm(u - uo) <= 1e-8 * np.linalg.norm(uo)
    monkeypatch.setenv("FFGPU_CG_GRAPH", "0")
    assert np.array_equal(A.solve(b), u)
