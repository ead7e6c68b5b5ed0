"""The FP32 inner product with the matrix staged through shared memory, against the FP64 solution and
the other layouts: rows shorter and longer than a stage (16 slots) and than the ring (32), one
chunk, a last pass that only some warps have, 32-bit columns.

Bar: the mixed path's own, 1e-8 relative (its outer loop stops on the FP64 residual)."""
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
    ffgpu.context(0)
    yield


def shuffled(Th, seed):
    """The mesh with its vertices renumbered at random (column differences past 16 bits)."""
    p = np.random.Generator(np.random.PCG64(seed)).permutation(Th.nv)
    X = np.empty_like(Th.coords)
    X[p] = Th.coords
    return mesh.Mesh(Th.dim, X, p[Th.elems].astype(np.int32), p[Th.belems].astype(np.int32), Th.blabel)


CASES = {
    "one_chunk": (lambda: mesh.square(3, 4), "P1"),
    "p1_2d": (lambda: mesh.square(57, 61), "P1"),
    "p1_3d": (lambda: mesh.cube(23), "P1"),
    "p1_3d_passes": (lambda: mesh.cube(62), "P1"),
    "p2_3d": (lambda: mesh.cube(9), "P2"),
    "wide_columns": (lambda: shuffled(mesh.square(200), 1), "P1"),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_layouts_agree(name, monkeypatch):
    make, fe = CASES[name]
    Th = make()
    Vh = FESpace(Th, fe)
    labels = (1, 2, 3, 4) if Th.dim == 2 else (1, 2, 3, 4, 5, 6)
    sol = {}
    for code in (69, 65, 66, 67):
        b = np.empty(Vh.ndof)
        A = ffgpu.matrix(ffgpu.varf_diffusion(f=1.0, on=labels), Vh, eps=1e-10, rhs_out=b)
        monkeypatch.setenv("FFGPU_IR_LAYOUT", str(code))
        u = A.solve_mixed(b, eps=1e-10)
        assert A.layout_code(2) == code
        assert np.array_equal(A.solve_mixed(b, eps=1e-10), u)
        sol[code] = u
        if code == 69:
            ref = A.solve(b)
    for code, u in sol.items():
        assert np.linalg.norm(u - ref) <= 1e-8 * np.linalg.norm(ref), code
