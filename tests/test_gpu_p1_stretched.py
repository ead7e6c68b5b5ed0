"""P1 element matrices on stretched elements (boundary layers, thin plates).

Separate triangles or tetrahedra cut from boxes of aspect 1 to 1e4 along one axis, with moved corners and
every choice of first vertex: the assembled entries are the element matrices.  Each entry is compared
with the exact rational value, its error relative to sqrt(K_ii K_jj).

Bar: four times the worst error that FreeFEM's own formula -- measure times the product of the
barycentric gradients, Mesh3dn.hpp:126-136 -- has on the same elements in FP64.
"""
from fractions import Fraction

import numpy as np
import pytest

import ffgpu
from ffgpu import mesh
from ffgpu.fespace import FESpace

pytestmark = pytest.mark.gpu

_HEX = [[0, 1, 3, 7], [0, 5, 1, 7], [0, 3, 2, 7], [0, 2, 6, 7], [0, 4, 5, 7], [0, 6, 4, 7]]


@pytest.fixture(scope="module", autouse=True)
def _lib_built():
    from ffgpu.build import build
    build()
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    ffgpu.context(0)
    yield


def _cross(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


def _gradients(P, one):
    """Barycentric gradients and the measure, in the arithmetic of P's numbers."""
    d = len(P[0])
    if d == 2:
        e = [[P[(i + 2) % 3][k] - P[(i + 1) % 3][k] for k in range(2)] for i in range(3)]
        det = e[2][0] * -e[1][1] + e[2][1] * e[1][0]
        return [[-v[1] / det, v[0] / det] for v in e], det / (2 * one)
    V = [[P[i + 1][k] - P[0][k] for k in range(3)] for i in range(3)]
    N = [_cross(V[1], V[2]), _cross(V[2], V[0]), _cross(V[0], V[1])]
    det = sum(a * b for a, b in zip(V[0], N[0]))
    G = [[v / det for v in n] for n in N]
    return [[-(a + b + c) for a, b, c in zip(*G)]] + G, det / (6 * one)


def _matrix(P, one):
    G, m = _gradients(P, one)
    return [[m * sum(a * b for a, b in zip(gi, gj)) for gj in G] for gi in G]


@pytest.mark.parametrize("aspect", [1.0, 1e2, 1e4])
@pytest.mark.parametrize("dim", [2, 3])
def test_entries_of_stretched_elements(dim, aspect):
    rng = np.random.Generator(np.random.PCG64(11))
    nt, nv = 240, dim + 1
    scale = np.array([1.0] * (dim - 1) + [aspect])
    X = np.empty((nt, nv, dim))
    for t in range(nt):
        if dim == 2:
            C = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], float) + rng.uniform(-.2, .2, (4, 2))
            P = C[np.roll([0, 1, 2], t % 3)]
        else:
            C = np.array([[k & 1, (k >> 1) & 1, k >> 2] for k in range(8)], float) + rng.uniform(-.1, .1, (8, 3))
            P = C[np.roll(_HEX[t % 6], t % 4)]
        P = (P + rng.integers(0, 20, dim)) * scale / 20
        V = P[1:] - P[0]
        X[t] = P if np.linalg.det(V) > 0 else P[[0, 2, 1, 3][:nv]]
    E = np.arange(nt * nv, dtype=np.int32).reshape(nt, nv)
    Th = mesh.Mesh(dim, X.reshape(-1, dim).copy(), E, E[:1, :dim].copy(), np.ones(1, np.int32))
    A = ffgpu.matrix(ffgpu.varf_diffusion(f=1.0), FESpace(Th, "P1"))
    rp, cl, vl = A.csr()
    K = vl.reshape(nt, nv, nv)
    worst = bar = 0.0
    for t in range(nt):
        exact = _matrix([[Fraction(float(x)) for x in p] for p in X[t]], Fraction(1))
        form = _matrix([[float(x) for x in p] for p in X[t]], 1.0)
        for i in range(nv):
            for j in range(nv):
                s = float(exact[i][i] * exact[j][j]) ** 0.5
                worst = max(worst, abs(float(Fraction(float(K[t, i, j])) - exact[i][j])) / s)
                bar = max(bar, abs(float(Fraction(form[i][j]) - exact[i][j])) / s)
    assert worst <= 4 * bar, (worst / 2.2e-16, bar / 2.2e-16)
