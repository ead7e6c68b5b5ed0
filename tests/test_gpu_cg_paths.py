"""Which way a scalar CG solve runs, and the two-launch iteration that FFGPU_CLUSTER_CG=0 selects.

The in-kernel loops are the default, so the two-launch iteration (cg_kca_sell and K_b storing C G) is
solved here with them switched off, with the bars of the other CG paths: 1e-12 of the three-launch path,
iteration counts within 1, two launches per iteration, the host-driven loop's bits, for A and A'.
"""
import numpy as np
import pytest

import ffgpu
from ffgpu import mesh
from ffgpu.fespace import FESpace

pytestmark = pytest.mark.gpu

THREE, TWO, BAND, LOOP = 1, 2, 4, 6


@pytest.fixture(scope="module", autouse=True)
def _lib_built():
    from ffgpu.build import build
    build()
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    ffgpu.context(0)
    yield


def _matrix(Th, kind="P1"):
    Vh = FESpace(Th, kind)
    kappa = np.exp(np.random.Generator(np.random.PCG64(5)).standard_normal(Th.nt))
    b = np.empty(Vh.ndof)
    return ffgpu.matrix(ffgpu.varf_diffusion(kappa=kappa, f=1.0, on=(1, 2, 3, 4)), Vh, eps=1e-10, rhs_out=b), b


def _counted(A, b, **kw):
    A.solve(b, **kw)   # set-up, tuning, graph
    l0 = ffgpu.kernel_launches()
    u = A.solve(b, **kw)
    return u, ffgpu.kernel_launches() - l0, A.stats.iterations


@pytest.mark.parametrize("Th,kind", [(mesh.square(64), "P1"), (mesh.square(150, 149), "P1"), (mesh.square(40), "P2"),
                                     (mesh.cube(10), "P1"), (mesh.cube(12, 13, 11), "P2")])
@pytest.mark.parametrize("trans", [False, True])
def test_two_launch_iteration(Th, kind, trans, monkeypatch):
    A, b = _matrix(Th, kind)
    if trans:
        b = np.random.Generator(np.random.PCG64(2)).standard_normal(A.n)
    monkeypatch.setenv("FFGPU_CLUSTER_CG", "0")
    u, launches, it = _counted(A, b, trans=trans)
    assert A.layout_code(6) == TWO
    assert 2 * it <= launches <= 2 * it + 24, (launches, it)
    monkeypatch.setenv("FFGPU_CG_GRAPH", "0")
    assert np.array_equal(_counted(A, b, trans=trans)[0], u)
    monkeypatch.delenv("FFGPU_CG_GRAPH")
    monkeypatch.setenv("FFGPU_CG_FUSE", "0")
    v, launches3, it3 = _counted(A, b, trans=trans)
    assert A.layout_code(6) == THREE and launches3 >= 3 * it3 and abs(it - it3) <= 1
    assert np.linalg.norm(u - v) <= 1e-12 * np.linalg.norm(v)


@pytest.mark.parametrize("n", [2, 9, 93, 138, 140, 196, 198, 277, 280, 395, 556])
def test_squares_along_the_grid_stay_on_the_sms(n):
    """Every instance of the loop: 64, 128 / 160, 256 / 288, 512 / 544, 1056 and 2048 rows per block."""
    A, b = _matrix(mesh.square(n))
    A.solve(b)
    assert A.layout_code(6) == BAND


def test_past_the_last_size_the_matrix_is_streamed():
    A, b = _matrix(mesh.square(561, 557))
    A.solve(b)
    # (block CSR, should the layout tuner take it, runs with launches)
    assert A.layout_code(6) == (LOOP if A.layout_code() >= 64 else THREE)


@pytest.mark.parametrize("n,full", [(28, False), (32, True)])
def test_p2_is_streamed_where_the_passes_are_full(n, full, monkeypatch):
    """P2 past the SMs' shared memory: 5 788 chunks of 32 rows over 4 864 warps (0.60 of two passes), 8 583 (0.88)."""
    import torch
    S = ffgpu.device_space("P2", 3, n, n, n)
    b = torch.zeros(S.Vh.ndof, dtype=torch.float64, device="cuda")
    A = ffgpu.matrix(ffgpu.varf_diffusion(f=1.0, on=(1, 2), c_mass=0.5), S, rhs_out=b, eps=1e-9)
    u = A.solve(b)
    it = A.stats.iterations
    assert A.layout_code(6) == (LOOP if full or A.layout_code() >= 64 else THREE)
    assert torch.equal(A.solve(b), u)
    monkeypatch.setenv("FFGPU_CLUSTER_CG", "0")
    v = A.solve(b)
    assert A.layout_code(6) == THREE and abs(A.stats.iterations - it) <= 2
    assert float((u - v).norm() / v.norm()) <= 1e-8
