"""The CG loops inside one cooperative kernel (cg_band and cg_loop, ffgpu_persist.cu) at the edges of
their dispatch: one block, the row counts where the threads per block and rows per thread change, the
last size cg_band takes, and what cg_loop takes: wide column ranges, larger systems, odd sizes.

Bars: the ones of the other CG paths -- 1e-9 against the launches per iteration (FFGPU_CG_FUSE=0)
and the oracle, iteration counts within 2, the same bits on a second solve.
"""
import os

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


def _matrix(Th, kind="P1", **kw):
    Vh = FESpace(Th, kind)
    kappa = np.exp(np.random.Generator(np.random.PCG64(3)).standard_normal(Th.nt))
    on = (1, 2, 3, 4) if Th.dim == 2 else (1, 2, 3, 4, 5, 6)
    b = np.empty(Vh.ndof)
    A = ffgpu.matrix(ffgpu.varf_diffusion(kappa=kappa, f=1.0, on=on), Vh, rhs_out=b, **kw)
    return A, b


def _solve(A, b, env=None, **kw):
    old = {k: os.environ.get(k) for k in (env or {})}
    os.environ.update(env or {})
    try:
        A.solve(b, **kw)
        l0 = ffgpu.kernel_launches()
        u = A.solve(b, **kw)
        return u, ffgpu.kernel_launches() - l0, A.stats.iterations
    finally:
        for k, v in old.items():
            os.environ.pop(k) if v is None else os.environ.__setitem__(k, v)


# rows per block 64 (1, 2 and 139 blocks), 128/160, 256/288, 512/544, 1056, 2048
@pytest.mark.parametrize("n", [2, 9, 93, 138, 140, 196, 198, 277, 280, 395, 556])
def test_loop_against_launches(n):
    A, b = _matrix(mesh.square(n), eps=1e-10)
    u, l, it = _solve(A, b)
    assert l < 12, l                                      # one kernel for all iterations
    assert np.array_equal(A.solve(b), u)
    u3, l3, it3 = _solve(A, b, env={"FFGPU_CG_FUSE": "0"})
    assert l3 >= 3 * it3
    assert abs(it - it3) <= 2
    assert np.linalg.norm(u - u3) <= 1e-9 * np.linalg.norm(u3)


@pytest.mark.parametrize("kind,Th", [("P1", mesh.cube(9, 7, 8)), ("P2", mesh.square(30, 17)), ("P2", mesh.cube(4))])
@pytest.mark.parametrize("trans", [False, True])
def test_loop_against_oracle(kind, Th, trans):
    A, b = _matrix(Th, kind, eps=1e-10)
    rp, cl, vl = A.csr()
    c = np.random.Generator(np.random.PCG64(2)).standard_normal(A.n)
    u, l, it = _solve(A, c, trans=trans)
    assert l < 12, l
    x = np.zeros(A.n)
    import scipy.sparse as sp
    S = sp.csr_matrix((vl, cl, rp), (A.n, A.n))
    S = S.T.tocsr() if trans else S
    # Jacobi-PCG as FreeFEM runs it: x = b/tgv on tgv rows, stop at (g, Cg) < eps^2 (g0, Cg0)
    d = 1.0 / S.diagonal()
    tgv = S.diagonal() == 1e30
    x[tgv] = c[tgv] / 1e30
    g = S @ x - c
    h = -d * g
    gcg = float(g @ (d * g))
    eps2 = 1e-20 * gcg
    its = 0
    while True:
        q = S @ h
        rho = -float(g @ h) / float(h @ q)
        x += rho * h
        g += rho * q
        new = float(g @ (d * g))
        h = (new / gcg) * h - d * g
        gcg = new
        its += 1
        if gcg < eps2:
            break
    assert abs(it - its) <= 2
    assert np.linalg.norm(u - x) <= 1e-9 * np.linalg.norm(x)


def test_loop_iteration_limit_and_converged_start():
    A, b = _matrix(mesh.square(60), eps=1e-10, itmax=5)
    with pytest.raises(ffgpu.FFGPUError) as ei:
        A.solve(b)
    assert ei.value.code == -3 and A.stats.iterations == 5
    A.itmax = 0
    z = np.zeros(A.n)
    assert np.array_equal(A.solve(z), z) and A.stats.iterations == 0


def test_wide_pattern_streams_and_a_fixed_layout_keeps_the_launches():
    A, b = _matrix(mesh.square(200), eps=1e-10)
    rp, cl, vl = A.csr()
    import scipy.sparse as sp
    p = np.random.Generator(np.random.PCG64(4)).permutation(A.n)
    S = sp.csr_matrix((vl, cl, rp), (A.n, A.n))[p][:, p].tocsr()
    S.sort_indices()
    B = ffgpu.matrix_from_csr(S.indptr, S.indices, S.data, eps=1e-10)
    u, l, it = _solve(A, b)
    v, lw, itw = _solve(B, b[p])                          # a block of the permuted rows touches every column
    assert l < 12 and lw < 12 and abs(it - itw) <= 2
    assert np.linalg.norm(v - u[p]) <= 1e-9 * np.linalg.norm(u)
    assert np.array_equal(B.solve(b[p]), v)
    t, lt, _ = _solve(B, b[p], trans=True)
    assert lt < 12 and np.linalg.norm(t - v) <= 1e-9 * np.linalg.norm(v)
    w, lf, itf = _solve(A, b, spmv_layout=64)
    assert lf >= 2 * itf
    assert np.linalg.norm(w - u) <= 1e-9 * np.linalg.norm(u)


@pytest.mark.parametrize("kind,dim,n", [("P1", 3, (59, 60, 61)), ("P1", 2, (557, 561)), ("P2", 3, (20, 21, 19)), ("P1", 3, (95, 96, 94))])
def test_streaming_loop_against_launches(kind, dim, n):
    import torch
    S = ffgpu.device_space(kind, dim, *n)
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    kappa = torch.exp(torch.randn(S.Vh.Th.nt, generator=g, device="cuda", dtype=torch.float64))
    b = torch.zeros(S.Vh.ndof, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    A = ffgpu.matrix(ffgpu.varf_diffusion(kappa=kappa, on=(1, 2, 3, 4)), S, eps=1e-10, rhs_out=b)
    bh = b.cpu().numpy()
    u, l, it = _solve(A, bh)
    assert l < 12, l
    assert np.array_equal(A.solve(bh), u)
    u3, l3, it3 = _solve(A, bh, env={"FFGPU_CG_FUSE": "0"})
    assert l3 >= 3 * it3 and abs(it - it3) <= 2
    assert np.linalg.norm(u - u3) <= 1e-8 * np.linalg.norm(u3)
