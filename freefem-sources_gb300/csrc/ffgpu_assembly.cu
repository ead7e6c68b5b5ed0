// ffgpu_assembly.cu -- mesh/FE-space upload, symbolic pattern and numeric assembly.
//
// Design (GB300): FreeFEM walks elements and scatters each element matrix into a hash
// matrix (problem.cpp:1096-1103, HashMatrix.cpp:1295-1332).  Here every matrix row gathers the
// contributions of the elements incident to its node:
//   pattern (once per matrix): a warp per row collects the nodes of the incident elements in a
//                    small hash table, ranks the distinct ones, and notes for every incidence
//                    the rank of each of the element's nodes in the row (pattern_kernel);
//   scan:            row pointer;
//   element pass:    the element matrices -- P1 in closed form (p1_elem_kernel), P2 from the
//                    tensor cores (ffgpu_elemtc.cu), coefficients at quadrature points from
//                    their own kernels;
//   fill:            a group of lanes per row adds the rows of the element matrices in ascending
//                    element order (the reference's summation order) into shared memory at the
//                    noted ranks, applies tgv, and writes the row once, coalesced.
// No atomics and no colouring are needed on the value path: each value is written once and
// no read-modify-write of the matrix happens.  A numeric reassembly repeats the last two only.
// For [P2]^3 the pattern is stored as 3x3 blocks (DOF = 3*node + c, FESpacen.hpp:582),
// which is the same (i,j) set as FreeFEM's MatriceMorse and 2/3 of the index traffic.
#include <math.h>
#include <string.h>

#include <algorithm>

#include "ffgpu_internal.cuh"

namespace ffgpu {

// ------------------------------------------------------------------ small device utils
// binary search of v in the sorted list s[0..n)
__device__ __forceinline__ int find_sorted(const int *s, int n, int v) {
    int lo = 0, hi = n - 1;
    while (lo <= hi) {
        int mid = (lo + hi) >> 1;
        int w = s[mid];
        if (w == v) return mid;
        if (w < v) lo = mid + 1; else hi = mid - 1;
    }
    return -1;
}

// ------------------------------------------------------------------ space construction
__global__ void build_nodes_kernel(const int32_t *dof, int nt, int ndofK, int nn, int bs,
                                   int ndof, int32_t *nodes, int *status) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)nt * nn) return;
    int k = (int)(t / nn), i = (int)(t % nn);
    const int32_t *d = dof + (int64_t)k * ndofK;
    int v0 = d[i];
    if (v0 < 0 || v0 >= ndof) { dev_fail(status, kDevBadIndex); nodes[t] = 0; return; }
    if (bs == 1) { nodes[t] = v0; return; }
    int node = v0 / bs;
    bool ok = (v0 % bs) == 0;
    for (int c = 1; c < bs; ++c) ok = ok && d[c * nn + i] == bs * node + c;
    if (!ok) dev_fail(status, kDevBadDofLayout);
    nodes[t] = node;
}

// four numbers per thread, in one load where the array (a caller's, maybe) is aligned for it
__global__ void check_elems_kernel(const int32_t *elems, int64_t m, int nv, int *status) {
    const int64_t t = 4 * (blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
    bool bad = false;
    if (t + 4 <= m && (reinterpret_cast<uintptr_t>(elems) & 15) == 0) {
        const int4 v = *reinterpret_cast<const int4 *>(elems + t);
        bad = min(min(v.x, v.y), min(v.z, v.w)) < 0 || max(max(v.x, v.y), max(v.z, v.w)) >= nv;
    } else {
        for (int64_t i = t; i < m && i < t + 4; ++i) bad |= elems[i] < 0 || elems[i] >= nv;
    }
    if (bad) dev_fail(status, kDevBadIndex);
}

// incidences per node, and the arrival number of each slot at its node: the fill needs no atomics
// (a node number out of range is skipped here: the status word, read with the counts, has it)
__global__ void inc_count_kernel(const int32_t *nodes, int64_t m, int nnodes, int32_t *cnt, uint16_t *at) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < m && (unsigned)nodes[t] < (unsigned)nnodes) at[t] = (uint16_t)min(atomicAdd(&cnt[nodes[t]], 1), 65535);
}

__global__ void inc_fill_kernel(const int32_t *nodes, int64_t m, const int32_t *ptr, const uint16_t *at, int32_t *inc) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < m) inc[ptr[nodes[t]] + at[t]] = (int32_t)t;
}

// Each node's incidence list by slot, i.e. by element number (the reference's element order): the
// place of a slot is the number of smaller ones.  G lanes per node (8 up to 8 slots a node on
// average, as 2D meshes have, else 32); lists longer than G lanes hold are counted from memory.  (A bitonic sort by
// a warp per node of the longest list's length: 632 us for the 21 M slots of 96^3 cells; this, 158 us.)
template <int G>
__global__ void __launch_bounds__(256) inc_sort_kernel(const int32_t *__restrict__ ptr, int nnodes,
                                                       const int32_t *__restrict__ in, int32_t *__restrict__ inc) {
    const int sub = threadIdx.x & (G - 1);
    const unsigned mask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) & ~(G - 1));
    const int64_t per = (int64_t)gridDim.x * (blockDim.x / G);
    for (int64_t a = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G; a < nnodes; a += per) {
        const int b = ptr[a], n = ptr[a + 1] - b;
        if (n <= G) {
            const int key = sub < n ? in[b + sub] : 0x7fffffff;
            int r = 0;
            for (int k = 0; k < n; ++k) r += __shfl_sync(mask, key, k, G) < key;
            if (sub < n) inc[b + r] = key;
        } else {
            for (int i = sub; i < n; i += G) {
                const int key = in[b + i];
                int r = 0;
                for (int k = 0; k < n; ++k) r += in[b + k] < key;
                inc[b + r] = key;
            }
        }
    }
}

// ------------------------------------------------------------------ geometry
// meas and barycentric gradients: Triangle::H (fem.hpp:321-324), Tet::Gradlambda
// (Mesh3dn.hpp:126-136), tet volume det(AB,AC,AD)/6 (Mesh3dn.hpp:70)
__global__ void geometry_kernel(const double *X, const int32_t *elems, int nt, int dim,
                                const double *kappa, double c_stiff, double *geo) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nt) return;
    double *g = geo + (int64_t)k * kGeoStride;
    double G[4][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    double meas;
    if (dim == 2) {
        const int32_t *v = elems + 3 * (int64_t)k;
        double P[3][2];
        for (int i = 0; i < 3; ++i) { P[i][0] = X[2 * (int64_t)v[i]]; P[i][1] = X[2 * (int64_t)v[i] + 1]; }
        double area = ((P[1][0] - P[0][0]) * (P[2][1] - P[0][1]) - (P[1][1] - P[0][1]) * (P[2][0] - P[0][0])) * 0.5;
        for (int i = 0; i < 3; ++i) {
            int i1 = (i + 1) % 3, i2 = (i + 2) % 3;
            double ex = P[i2][0] - P[i1][0], ey = P[i2][1] - P[i1][1];
            G[i][0] = -ey / (2 * area);
            G[i][1] = ex / (2 * area);
        }
        meas = area;
    } else {
        const int32_t *v = elems + 4 * (int64_t)k;
        double A[3], V[3][3];
        for (int d = 0; d < 3; ++d) A[d] = X[3 * (int64_t)v[0] + d];
        for (int i = 0; i < 3; ++i)
            for (int d = 0; d < 3; ++d) V[i][d] = X[3 * (int64_t)v[i + 1] + d] - A[d];
        double c23[3] = {V[1][1] * V[2][2] - V[1][2] * V[2][1], V[1][2] * V[2][0] - V[1][0] * V[2][2],
                         V[1][0] * V[2][1] - V[1][1] * V[2][0]};
        double c31[3] = {V[2][1] * V[0][2] - V[2][2] * V[0][1], V[2][2] * V[0][0] - V[2][0] * V[0][2],
                         V[2][0] * V[0][1] - V[2][1] * V[0][0]};
        double c12[3] = {V[0][1] * V[1][2] - V[0][2] * V[1][1], V[0][2] * V[1][0] - V[0][0] * V[1][2],
                         V[0][0] * V[1][1] - V[0][1] * V[1][0]};
        double vol = (V[0][0] * c23[0] + V[0][1] * c23[1] + V[0][2] * c23[2]) / 6.;
        double det1 = 1. / (6. * vol);
        for (int d = 0; d < 3; ++d) {
            G[1][d] = c23[d] * det1;
            G[2][d] = c31[d] * det1;
            G[3][d] = c12[d] * det1;
            G[0][d] = -G[1][d] - G[2][d] - G[3][d];
        }
        meas = vol;
    }
    g[0] = meas;
    g[1] = (kappa ? kappa[k] : 1.0) * c_stiff;
    g[2] = 0; g[3] = 0;
    for (int i = 0; i < 4; ++i)
        for (int d = 0; d < 3; ++d) g[4 + 3 * i + d] = G[i][d];
}

// ------------------------------------------------------------------ element entries
// P2 gradients are linear: grad(phi_i) = sum_a lambda_a C_i[a], with
//   vertex i: C_i[i] = 3 g_i, C_i[a != i] = -g_i            (grad = (4 lambda_i - 1) g_i)
//   edge (p,q): C_i[p] = 4 g_q, C_i[q] = 4 g_p, else 0      (grad = 4(lambda_p g_q + lambda_q g_p))
// (P012_3d.cpp:199-277; 2D: FESpace.cpp:1219-1300 with edge i opposite vertex i), and
//   int_K lambda_a lambda_b = |K| (1 + delta_ab) / ((d+1)(d+2)),
// so int_K d_alpha(phi_i) d_beta(phi_j) = m (sum_a C_i[a].al C_j[a].be + S_i.al S_j.be),
// m = |K|/((d+1)(d+2)), S_i = sum_a C_i[a].  This integrates the degree-2 integrand
// exactly, as FreeFEM's default rules (T_5, Tet_5) do.
struct V3 {
    double x, y, z;
};
__device__ __forceinline__ V3 v3(const double *p) { return V3{__ldg(p), __ldg(p + 1), __ldg(p + 2)}; }
__device__ __forceinline__ V3 operator*(double a, V3 v) { return V3{a * v.x, a * v.y, a * v.z}; }
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return V3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ double comp(V3 v, int c) { return c == 0 ? v.x : (c == 1 ? v.y : v.z); }

// local edge e -> vertices (p,q): tets {01,02,03,12,13,23}, triangles edge i opposite vertex i
template <int DIM>
__device__ __forceinline__ void edge_vertices(int e, int &p, int &q) {
    if (DIM == 3) {
        p = e < 3 ? 0 : (e < 5 ? 1 : 2);
        q = e < 3 ? e + 1 : (e == 3 ? 2 : 3);
    } else {
        p = (e + 1) % 3;
        q = (e + 2) % 3;
    }
}

// One P2 basis function J in the two-gradient form used below, with no divergent branches:
//   C_J[a] = c1(a) g_p1 + c2(a) g_p2,   S_J = sum_a C_J[a] = d1 g_p1 + d2 g_p2
//   vertex j:   p1 = p2 = j, c1(a) = (a == j ? 3 : -1), c2 = 0,  d1 = 3 - dim, d2 = 0
//   edge (r,s): p1 = s, p2 = r, c1(a) = 4 [a == r], c2(a) = 4 [a == s], d1 = d2 = 4
// (grad(phi_j) = (4 lambda_j - 1) g_j and grad(4 lambda_r lambda_s) = 4 (lambda_r g_s + lambda_s g_r)).
template <int DIM>
struct P2Basis {
    int p1, p2;
    bool vtx;
    __device__ __forceinline__ explicit P2Basis(int J) {
        vtx = J <= DIM;
        int r = 0, s = 0;
        edge_vertices<DIM>(vtx ? 0 : J - DIM - 1, r, s);
        p1 = vtx ? J : s;
        p2 = vtx ? J : r;
    }
    __device__ __forceinline__ double c1(int a) const {
        return vtx ? (a == p1 ? 3.0 : -1.0) : (a == p2 ? 4.0 : 0.0);
    }
    __device__ __forceinline__ double c2(int a) const { return vtx ? 0.0 : (a == p1 ? 4.0 : 0.0); }
    __device__ __forceinline__ double d1() const { return vtx ? 3.0 - DIM : 4.0; }
    __device__ __forceinline__ double d2() const { return vtx ? 0.0 : 4.0; }
};

// P2 mass matrix of the element, int_K phi_i phi_j = |K| kP2Mass*[i][j] / den (exact integrals
// of the degree-4 products of the vertex functions l(2l-1) and edge functions 4 l_p l_q,
// int_K l^a = |K| d! prod a_i! / (d + |a|)!), local order as the P2 basis above
__device__ __constant__ signed char kP2Mass2[6][6] = {{6, -1, -1, -4, 0, 0},  {-1, 6, -1, 0, -4, 0},
                                                     {-1, -1, 6, 0, 0, -4},  {-4, 0, 0, 32, 16, 16},
                                                     {0, -4, 0, 16, 32, 16}, {0, 0, -4, 16, 16, 32}};
__device__ __constant__ signed char kP2Mass3[10][10] = {
    {6, 1, 1, 1, -4, -4, -4, -6, -6, -6},   {1, 6, 1, 1, -4, -6, -6, -4, -4, -6},
    {1, 1, 6, 1, -6, -4, -6, -4, -6, -4},   {1, 1, 1, 6, -6, -6, -4, -6, -4, -4},
    {-4, -4, -6, -6, 32, 16, 16, 16, 16, 8}, {-4, -6, -4, -6, 16, 32, 16, 16, 8, 16},
    {-4, -6, -6, -4, 16, 16, 32, 8, 16, 16}, {-6, -4, -4, -6, 16, 16, 8, 32, 16, 16},
    {-6, -4, -6, -4, 16, 8, 16, 16, 32, 16}, {-6, -6, -4, -4, 8, 16, 16, 16, 16, 32}};

template <int DIM>
__device__ __forceinline__ double p2_mass(int i, int j) {
    return DIM == 3 ? kP2Mass3[i][j] * (1.0 / 420.0) : kP2Mass2[i][j] * (1.0 / 180.0);
}

// The 3x3 matrix (1/m) int_K d_a(phi_I) d_b(phi_J) = sum_c C_I[c]_a C_J[c]_b + S_I,a S_J,b as a sum
// of at most three outer products u_k (x) w_k:
//   I vertex i:   u = g_i,  w = 4 C_J[i] - (d-2) S_J                    (rank 1)
//   I edge (p,q): 4 g_q (x) C_J[p] + 4 g_p (x) C_J[q] + S_I (x) S_J    (rank 3)
// The I type is the same on every lane of a warp (a row's node is either a vertex or an edge
// of all its elements); the J side is evaluated without branches.
template <int DIM>
struct P2Pair {
    V3 u0, w0, u1, w1, u2, w2;
    bool vertex;
    __device__ __forceinline__ P2Pair(const double *G, int I, int Jidx) {
        const P2Basis<DIM> J(Jidx);
        const V3 g1 = v3(G + 3 * J.p1), g2 = v3(G + 3 * J.p2);
        vertex = I <= DIM;
        if (vertex) {
            u0 = v3(G + 3 * I);
            // 4 C_J[i] - (d-2) S_J, with the coefficients selected, not branched on
            const double a1 = 4.0 * J.c1(I) - (DIM - 2) * J.d1(), a2 = 4.0 * J.c2(I) - (DIM - 2) * J.d2();
            w0 = a1 * g1 + a2 * g2;
            u1 = w1 = u2 = w2 = V3{0.0, 0.0, 0.0};
        } else {
            int p, q;
            edge_vertices<DIM>(I - DIM - 1, p, q);
            const V3 gp = v3(G + 3 * p), gq = v3(G + 3 * q);
            u0 = 4.0 * gq; w0 = J.c1(p) * g1 + J.c2(p) * g2;
            u1 = 4.0 * gp; w1 = J.c1(q) * g1 + J.c2(q) * g2;
            u2 = 4.0 * (gp + gq); w2 = J.d1() * g1 + J.d2() * g2;
        }
    }
    __device__ __forceinline__ double g(int a, int b) const {
        double t = comp(u0, a) * comp(w0, b);
        if (!vertex) t += comp(u1, a) * comp(w1, b) + comp(u2, a) * comp(w2, b);
        return t;
    }
    __device__ __forceinline__ double trace() const {
        double t = u0.x * w0.x + u0.y * w0.y + u0.z * w0.z;
        if (!vertex) t += u1.x * w1.x + u1.y * w1.y + u1.z * w1.z + u2.x * w2.x + u2.y * w2.y + u2.z * w2.z;
        return t;
    }
};

// int_K phi_i for the linear form with a constant source on the element
template <int DIM, int ORDER>
__device__ __forceinline__ double basis_integral(double meas, int i) {
    if (ORDER == 1) return meas / (DIM + 1);
    if (DIM == 3) return i < 4 ? -meas / 20.0 : meas / 5.0;
    return i < 3 ? 0.0 : meas / 3.0;
}

// ------------------------------------------------------------------ P1 element matrices
// Products and sums with their roundings spelled out where two kernels have to form the same
// bits (the measure enters the matrix kernel and the linear form).
__device__ __forceinline__ double det2(double a, double b, double c, double d) { return fma(a, d, -__dmul_rn(b, c)); }

// Vertex coordinates of an element relative to its first vertex: V[i] = P[i+1] - P[0]
template <int DIM>
__device__ __forceinline__ void edge_vectors(const double *__restrict__ X, const int32_t *__restrict__ v, double V[DIM][DIM]) {
    double A[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) A[d] = __ldg(X + (int64_t)DIM * v[0] + d);
#pragma unroll
    for (int i = 0; i < DIM; ++i)
#pragma unroll
        for (int d = 0; d < DIM; ++d) V[i][d] = __dsub_rn(__ldg(X + (int64_t)DIM * v[i + 1] + d), A[d]);
}
// det of the edge vectors (DIM! times the measure) and, in 3D, the cross product V1 x V2
__device__ __forceinline__ double edge_det(const double V[2][2], double *) { return det2(V[0][0], V[0][1], V[1][0], V[1][1]); }
__device__ __forceinline__ double edge_det(const double V[3][3], double *c) {
    c[0] = det2(V[1][1], V[1][2], V[2][1], V[2][2]);
    c[1] = det2(V[1][2], V[1][0], V[2][2], V[2][0]);
    c[2] = det2(V[1][0], V[1][1], V[2][0], V[2][1]);
    return fma(V[0][2], c[2], fma(V[0][1], c[1], __dmul_rn(V[0][0], c[0])));
}
template <int DIM>
__device__ __forceinline__ double measure_of(double det) { return __dmul_rn(det, DIM == 2 ? 0.5 : 1.0 / 6.0); }

__device__ __forceinline__ void store4(double *p, double a, double b, double c, double d) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// Element matrices of int(c_stiff kappa grad u.grad v + c_mass u v) on P1, one thread each:
//   grad phi_i = N_i / det with N_i the inward normals (cross products of edges), so
//   K_ij = (kappa c_stiff / (DIM! det)) N_i.N_j, one dot product per pair.
// Row la of element e at out[(e * (DIM + 1) + la) * 4], four doubles wide (32-byte stores; the
// row fill reads one sector).  FP64 issue bounds it (a warp's fused multiply-add
// takes 64 cycles of its sub-partition, an add or multiply 76): about 90 FP64 operations per tetrahedron against about 60 for the gradients
// alone, and none of the products is left to the row fill (5.3 M tetrahedra: 0.84 ms).
template <int DIM>
__global__ void __launch_bounds__(256) p1_elem_kernel(const double *__restrict__ X, const int32_t *__restrict__ elems, int nt,
                                                      const double *__restrict__ kappa, double c_stiff, double c_mass,
                                                      double *__restrict__ out, double *__restrict__ measure) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= nt) return;
    constexpr int NV = DIM + 1;
    int32_t v[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = __ldg(elems + e * NV + i);
    double V[DIM][DIM], c[3];
    edge_vectors<DIM>(X, v, V);
    const double det = edge_det(V, c);
    const double meas = measure_of<DIM>(det);
    if (measure) measure[e] = meas;
    if (!out) return;
    const double w = (kappa ? kappa[e] : 1.0) * c_stiff / (DIM == 2 ? 2.0 * det : 6.0 * det);
    double K[NV][NV];
    if constexpr (DIM == 2) {
        // edges opposite the vertices: e0 = P2 - P1, e1 = -V1, e2 = V0; every entry a product of its own (row
        // sums would carry the rounding of the largest entry: 600 eps of an entry at aspect 1e4 instead of 3)
        const double x0 = __ldg(X + 2 * (int64_t)v[2]) - __ldg(X + 2 * (int64_t)v[1]);
        const double y0 = __ldg(X + 2 * (int64_t)v[2] + 1) - __ldg(X + 2 * (int64_t)v[1] + 1);
        K[0][1] = -w * fma(x0, V[1][0], y0 * V[1][1]);
        K[0][2] = w * fma(x0, V[0][0], y0 * V[0][1]);
        K[1][2] = -w * fma(V[1][0], V[0][0], V[1][1] * V[0][1]);
        K[0][0] = w * fma(x0, x0, y0 * y0);
        K[1][1] = w * fma(V[1][0], V[1][0], V[1][1] * V[1][1]);
        K[2][2] = w * fma(V[0][0], V[0][0], V[0][1] * V[0][1]);
    } else {
        // N1 = V1 x V2 (c), N2 = V2 x V0, N3 = V0 x V1
        const double p0 = det2(V[2][1], V[2][2], V[0][1], V[0][2]), p1 = det2(V[2][2], V[2][0], V[0][2], V[0][0]),
                     p2 = det2(V[2][0], V[2][1], V[0][0], V[0][1]);
        const double q0 = det2(V[0][1], V[0][2], V[1][1], V[1][2]), q1 = det2(V[0][2], V[0][0], V[1][2], V[1][0]),
                     q2 = det2(V[0][0], V[0][1], V[1][0], V[1][1]);
        K[1][1] = w * fma(c[2], c[2], fma(c[1], c[1], c[0] * c[0]));
        K[2][2] = w * fma(p2, p2, fma(p1, p1, p0 * p0));
        K[3][3] = w * fma(q2, q2, fma(q1, q1, q0 * q0));
        K[1][2] = w * fma(c[2], p2, fma(c[1], p1, c[0] * p0));
        K[1][3] = w * fma(c[2], q2, fma(c[1], q1, c[0] * q0));
        K[2][3] = w * fma(p2, q2, fma(p1, q1, p0 * q0));
        // N0 from the zero sum of the N_i; its products by themselves: as row sums they would carry the
        // rounding of the largest entry (needles and flat elements: 3e4 eps of an entry instead of 70)
        const double n0 = -(c[0] + p0 + q0), n1 = -(c[1] + p1 + q1), n2 = -(c[2] + p2 + q2);
        K[0][0] = w * fma(n2, n2, fma(n1, n1, n0 * n0));
        K[0][1] = w * fma(n2, c[2], fma(n1, c[1], n0 * c[0]));
        K[0][2] = w * fma(n2, p2, fma(n1, p1, n0 * p0));
        K[0][3] = w * fma(n2, q2, fma(n1, q1, n0 * q0));
    }
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int j = 0; j < i; ++j) K[i][j] = K[j][i];
    if (c_mass != 0.0) {
        const double m = c_mass * meas * (DIM == 3 ? 1.0 / 20.0 : 1.0 / 12.0);
#pragma unroll
        for (int i = 0; i < NV; ++i)
#pragma unroll
            for (int j = 0; j < NV; ++j) K[i][j] += i == j ? 2.0 * m : m;
    }
    double *o = out + e * NV * 4;
#pragma unroll
    for (int i = 0; i < NV; ++i) store4(o + 4 * i, K[i][0], K[i][1], K[i][2], DIM == 3 ? K[i][NV - 1] : 0.0);
}

// ------------------------------------------------------------------ pattern
// Warp per row.  The candidates (all nodes of the incident elements, in incidence order) go into
// a hash table of H >= their number entries, so each distinct node is kept once; the rank of
// a node is the count of smaller ones (an O(degree^2 / 32) loop of broadcast reads: shorter than a
// sort up to the degrees FE meshes have).  tmpcol: the row's sorted columns at inc_ptr[a] * NN;
// rmap: rank of node lb of incidence t at t * NN + lb; drank: rank of the row's own node.
template <int NN>
__global__ void __launch_bounds__(128) pattern_kernel(int nnodes, const int32_t *__restrict__ inc_ptr,
                                                      const int32_t *__restrict__ inc, const int32_t *__restrict__ nodes,
                                                      int logH, int32_t *__restrict__ deg, int32_t *__restrict__ tmpcol,
                                                      uint16_t *__restrict__ rmap, int32_t *__restrict__ drank, int *status) {
    extern __shared__ int sh_pat[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, H = 1 << logH;
    int *tab = sh_pat + w * 3 * H, *lst = tab + H;
    uint16_t *sl = reinterpret_cast<uint16_t *>(lst + H), *lsl = sl + H;
    for (int a = blockIdx.x * 4 + w; a < nnodes; a += gridDim.x * 4) {
        const int b = inc_ptr[a], m = (inc_ptr[a + 1] - b) * NN;
        if (m > kCandMax) { if (lane == 0) { dev_fail(status, kDevCandOverflow); deg[a] = 0; } continue; }
        for (int i = lane; i < H; i += 32) tab[i] = -1;
        __syncwarp();
        for (int p = lane; p < m; p += 32) {
            const int t = p / NN, i = p - t * NN;
            const int v = __ldg(nodes + __ldg(inc + b + t) / NN * NN + i);
            int h = (int)(((unsigned)v * 2654435761u) >> (32 - logH));
            for (;;) {
                const int old = atomicCAS(tab + h, -1, v);
                if (old == -1 || old == v) break;
                h = (h + 1) & (H - 1);
            }
            sl[p] = (uint16_t)h;
        }
        __syncwarp();
        int u = 0;
        for (int c = 0; c < H; c += 32) {
            const int v = tab[c + lane];
            const unsigned bal = __ballot_sync(0xffffffffu, v >= 0);
            if (v >= 0) {
                const int i = u + __popc(bal & ((1u << lane) - 1u));
                lst[i] = v;
                lsl[i] = (uint16_t)(c + lane);
            }
            u += __popc(bal);
        }
        __syncwarp();
        bool self = false;
        for (int i = lane; i < u; i += 32) {
            const int v = lst[i];
            int r = 0;
#pragma unroll 4
            for (int k = 0; k < u; ++k) r += lst[k] < v;
            tmpcol[(int64_t)b * NN + r] = v;
            tab[lsl[i]] = r;
            if (v == a) { drank[a] = r; self = true; }
        }
        self = __any_sync(0xffffffffu, self);
        __syncwarp();   // the ranks in tab are read by other lanes (a vote orders no memory)
        for (int p = lane; p < m; p += 32) rmap[(int64_t)b * NN + p] = (uint16_t)tab[sl[p]];
        if (lane == 0) {
            deg[a] = u;
            if (!self) { drank[a] = 0; dev_fail(status, kDevNotFound); }
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------ fill + numeric pass
struct FillArgs {
    int nnodes;
    const int32_t *inc_ptr, *inc;
    const int32_t *nodes;
    const double *geo;        // element geometry (only where the fill itself forms or scales entries)
    const int32_t *browptr;
    int32_t *bcol;
    const uint16_t *rmap;     // rank in its row of every node of every incidence (pattern_kernel)
    const int32_t *tmpcol;    // first numeric pass: the rows' columns and own ranks as pattern_kernel
    const int32_t *drank;     //   left them, copied to bcol / diagpos; NULL later
    int32_t *diagpos;         // block index of the diagonal block
    double *val;
    const double *kloc;       // element stiffness matrices, row la of element e at (e * NN + la) * krs, or NULL
    int krs;
    const double *mloc;       // element mass matrices of a coefficient at quadrature points, or NULL
    const double *tloc;       // element matrices of the general volume terms (ffgpu_varf.terms), or NULL
    const double *lame;       // per-element (lambda, mu) of the elasticity form, or NULL
    const double *eloc;       // [P2]^3 element blocks from the tensor cores (ffgpu_elemtc.cu), or NULL
    double c_mass;            // mass term to add (has_mass); none where kloc includes it
    int has_mass;
    double lam, mu;           // elasticity
    const uint8_t *onbc;
    double tgv;
    int tgv_rows;             // tgv > 0 and there is an on(...)
    int neg;                  // tgv < 0 and there is an on(...): the NegTgv bits of the variant
    int max_deg;
    int *status;
    // boundary terms (NULL bptr: none): node -> codes b*NN + il, element matrices
    const int32_t *bptr, *blist, *bel_elem;
    const double *bmat;
};

enum NegTgv { kNegOn = 1, kNegKeepRow = 2, kNegZeroCol = 4, kNegZeroColDiag = 8, kNegZeroDiag = 16 };

static int neg_tgv_bits(double tgv) {
    if (!(tgv < 0)) return 0;
    const auto is = [&](double v) { return fabs(tgv + v) < 1e-10; };
    int bits = kNegOn;
    if (is(3.0) || is(30.0)) bits |= kNegKeepRow;
    if (is(2.0) || is(20.0) || is(3.0) || is(30.0)) bits |= kNegZeroCol;
    if (tgv < -19.0) bits |= kNegZeroColDiag;
    if (tgv < -9.0) bits |= kNegZeroDiag;
    return bits;
}

// Numeric fill.  FE: 1 = P1 scalar, 2 = P2 scalar, 3 = [P2]^3 elasticity.
// A group of GL lanes owns a row, RW rows per warp: lane lb of a scalar group adds entry (la, lb)
// of one incident element after the other to the row in shared memory; a [P2]^3 group has a lane
// per (lb, component) and adds three values.  The nodes of one element are distinct, so the lanes
// of a step never meet on an entry, and every FP64 add is issued by all the rows of the warp at
// once: FP64 issue (76 cycles per warp add and sub-partition, however many lanes are
// active) bounds the fill, and a step per incident element is the fewest adds there are.
// The form this replaces gave the row one copy per concurrent element and summed the copies:
// 21 warp adds per P1 row in 3D instead of 3.  PLAIN: the element matrices are complete (kloc or
// eloc and nothing to add); the general form keeps its tests out of that loop.  On 96^3 cells (912 673 rows, 13.4 M entries), the
// products moved to p1_elem_kernel (0.84 ms): 3.27 -> 0.30 ms.  (With the tests on tgv and c_mass
// as FP64 compares in the loops it took 1.6 ms: a compare costs as much as an add.)
template <int DIM, int FE, bool PLAIN>
__global__ void __launch_bounds__(256) fill_kernel(FillArgs A) {
    constexpr int nvk = DIM + 1;
    constexpr int NN = FE == 1 ? nvk : (DIM == 3 ? 10 : 6);
    constexpr int BS = FE == 3 ? 3 : 1;
    constexpr int BS2 = BS * BS;
    constexpr int GL = NN * BS, RW = 32 / GL;
    constexpr int STEP = 4;          // incident elements whose loads are in flight together
    extern __shared__ __align__(16) double sh_fill[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int warps = blockDim.x >> 5;
    double *rows = sh_fill + (int64_t)w * RW * A.max_deg * BS2;
    const int grp = lane / GL, sub = lane - grp * GL;
    const int lb = sub / BS, c = sub - lb * BS;

    for (int64_t a0 = ((int64_t)blockIdx.x * warps + w) * RW; a0 < A.nnodes; a0 += (int64_t)gridDim.x * warps * RW) {
        const int a = (int)a0 + grp;
        const bool act = grp < RW && a < A.nnodes;
        const int last = (int)min((int64_t)A.nnodes, a0 + RW);
        const int rb0 = A.browptr[a0], total = (A.browptr[last] - rb0) * BS2;
        const int rb = act ? A.browptr[a] : rb0, deg = act ? A.browptr[a + 1] - rb : 0;
        double *acc = rows + (int64_t)(rb - rb0) * BS2;
        for (int q = lane; q < total; q += 32) rows[q] = 0.0;
        const int ib = act ? A.inc_ptr[a] : 0, ie = act ? A.inc_ptr[a + 1] : 0;
        const int steps = __reduce_max_sync(0xffffffffu, ie - ib);
        __syncwarp();
        for (int s0 = 0; s0 < steps; s0 += STEP) {
            double v[STEP][BS];
            int rk[STEP];
#pragma unroll
            for (int u = 0; u < STEP; ++u) {
                const int t = ib + s0 + u;
                rk[u] = -1;
                if (t >= ie) continue;
                const int64_t sl = __ldg(A.inc + t);   // e * NN + la
                rk[u] = __ldg(A.rmap + (int64_t)t * NN + lb);
                if (PLAIN) {
                    const double *src = FE == 3 ? A.eloc + (sl * NN + lb) * 9 + 3 * c : A.kloc + sl * A.krs + lb;
#pragma unroll
                    for (int q = 0; q < BS; ++q) v[u][q] = __ldg(src + q);
                    continue;
                }
                const int64_t e = sl / NN;
                const int la = (int)(sl - e * NN);
                const double *ge = A.geo + e * kGeoStride;
                if (FE <= 2) {
                    double x;
                    if (A.kloc) {
                        x = __ldg(A.kloc + sl * A.krs + lb);
                    } else {
                        // P2 without the tensor-core element matrices
                        x = __ldg(ge + 1) * (__ldg(ge) * (DIM == 3 ? 1.0 / 20.0 : 1.0 / 12.0)) *
                            (FE == 2 ? P2Pair<DIM>(ge + 4, la, lb).trace() : 0.0);
                    }
                    if (A.has_mass) {
                        const double meas = __ldg(ge);
                        x += FE == 1 ? A.c_mass * meas * (DIM == 3 ? 1.0 / 20.0 : 1.0 / 12.0) * (la == lb ? 2.0 : 1.0)
                                     : A.c_mass * meas * p2_mass<DIM>(la, lb);
                    }
                    if (A.mloc) x += __ldg(A.mloc + sl * NN + lb);
                    if (A.tloc) x += __ldg(A.tloc + sl * NN + lb);
                    v[u][0] = x;
                } else {
                    const P2Pair<DIM> P(ge + 4, la, lb);
                    const double m = __ldg(ge) * (1.0 / 20.0), tr = P.trace();
                    const double lam = A.lame ? __ldg(A.lame + 2 * e) : A.lam;
                    const double mu = A.lame ? __ldg(A.lame + 2 * e + 1) : A.mu;
#pragma unroll
                    for (int q = 0; q < BS; ++q) {
                        double x = lam * P.g(c, q) + mu * P.g(q, c);
                        if (q == c) x += mu * tr;
                        v[u][q] = m * x;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < STEP; ++u) {
                if (rk[u] >= 0) {
#pragma unroll
                    for (int q = 0; q < BS; ++q) acc[rk[u] * BS2 + c * BS + q] += v[u][q];
                }
                __syncwarp();   // the next element's lanes may meet this one's entries
            }
        }
        // ---- the row's columns: copied out by the first pass, where on(...) looks them up later
        const int32_t *cs = A.tmpcol ? A.tmpcol + (int64_t)ib * NN : A.bcol + rb;
        if (A.tmpcol)
            for (int r = sub; r < deg; r += GL) A.bcol[rb + r] = cs[r];
        const int self = act ? (A.tmpcol ? A.drank[a] : A.diagpos[a] - rb) : 0;
        if (A.tmpcol && act && sub == 0) A.diagpos[a] = rb + self;
        // ---- boundary terms, boundary element by boundary element, after the volume sum
        if (A.bptr && A.bmat) {
            const int p0 = act ? A.bptr[a] : 0, p1 = act ? A.bptr[a + 1] : 0;
            const int nb = __reduce_max_sync(0xffffffffu, p1 - p0);
            for (int s = 0; s < nb; ++s) {
                if (p0 + s < p1) {
                    const int code = A.blist[p0 + s];
                    const int bb = code / NN, il = code - bb * NN;
                    const int cn = A.nodes[(int64_t)A.bel_elem[bb] * NN + lb];
                    const int r = find_sorted(cs, deg, cn);
                    if (r < 0) dev_fail(A.status, kDevNotFound);
                    else acc[r * BS2 + c * BS + c] += A.bmat[((int64_t)bb * NN + il) * NN + lb];
                }
                __syncwarp();
            }
        }
        // ---- Dirichlet rows (tgv > 0): diagonal := tgv
        if (act && sub < BS && A.tgv_rows && A.onbc[(int64_t)a * BS + sub])
            acc[self * BS2 + sub * BS + sub] = A.tgv;
        __syncwarp();
        // tgv < 0 (HashMatrix::SetBC, HashMatrix.cpp:1195-1238): Dirichlet rows get a unit
        // diagonal (0 when tgv <= -10) and, except for -3/-30, zero off-diagonals; for
        // -2/-20/-3/-30 the Dirichlet columns are zeroed too (the diagonal also for -20/-30).
        // (the tests on tgv are made on the host: FP64 compares would cost more than the sums)
        if (A.neg) {
            for (int q = sub; q < deg * BS2; q += GL) {
                const int k = q / BS2, r = (q % BS2) / BS, cp = q % BS;
                const int col = cs[k];
                const bool diag = col == a && r == cp;
                const bool mine = A.onbc[(int64_t)a * BS + r];
                const bool gone = (mine && !(A.neg & kNegKeepRow) && !diag) ||
                                  ((A.neg & kNegZeroCol) && (!diag || (A.neg & kNegZeroColDiag)) && A.onbc[(int64_t)col * BS + cp]);
                if (gone) acc[q] = 0.0;
                else if (mine && diag) acc[q] = A.neg & kNegZeroDiag ? 0.0 : 1.0;
            }
            __syncwarp();
        }
        for (int q = lane; q < total; q += 32) A.val[(int64_t)rb0 * BS2 + q] = rows[q];
        __syncwarp();
    }
}

// linear form (real[int] b = a(0,Vh), alone or beside the matrix): per node, sum over incident
// elements; measure[e * mstride] is the measure of element e
template <int DIM, int FE>
__global__ void rhs_kernel(int nnodes, const int32_t *inc_ptr, const int32_t *inc, const double *measure, int mstride, const double *fP0,
                           const double *fint, double f0, double f1, double f2, const uint8_t *onbc,
                           const double *g,
                           double tgv, double *rhs, const int32_t *bptr, const int32_t *blist,
                           const double *brhs) {
    constexpr int BS = FE == 3 ? 3 : 1;
    // element p of the node goes to partial p % SLOTS, partials summed in order
    constexpr int NN = FE == 1 ? DIM + 1 : (DIM == 3 ? 10 : 6);
    constexpr int SLOTS = 32 / NN;
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)nnodes * BS) return;
    int a = (int)(t / BS), c = (int)(t % BS);
    double part[SLOTS];
#pragma unroll
    for (int sl = 0; sl < SLOTS; ++sl) part[sl] = 0.0;
    const int ib = inc_ptr[a], ie = inc_ptr[a + 1];
    for (int p0 = ib; p0 < ie; p0 += SLOTS) {
#pragma unroll
        for (int sl = 0; sl < SLOTS; ++sl) {
            const int p = p0 + sl;
            if (p < ie) {
                const int e = inc[p] / NN, l = inc[p] - e * NN;
                double meas = measure[(int64_t)e * mstride];
                double f = fP0 ? fP0[(int64_t)e * BS + c] : (c == 0 ? f0 : (c == 1 ? f1 : f2));
                const double add = fint ? fint[((int64_t)e * NN + l) * BS + c]
                                        : __dmul_rn(__dmul_rn(meas, f), FE == 1 ? 1.0 / (DIM + 1)
                                                                                : basis_integral<DIM, 2>(1.0, l));
                part[sl] = __dadd_rn(part[sl], add);
            }
        }
    }
    double s = part[0];
#pragma unroll
    for (int sl = 1; sl < SLOTS; ++sl) s += part[sl];
    if (bptr)   // boundary terms, in boundary-element order, after the volume terms
        for (int p = bptr[a]; p < bptr[a + 1]; ++p) {
            const int code = blist[p];
            const int bb = code / NN, il = code - bb * NN;
            s += brhs[((int64_t)bb * BS + c) * NN + il];
        }
    if (onbc && onbc[t]) s = (tgv > 0 ? tgv : 1.0) * (g ? g[t] : 0.0);
    rhs[t] = s;
}

// ------------------------------------------------------------------ CSR export
// a scalar matrix is stored as the CSR it exports: one launch for the three arrays
__global__ void __launch_bounds__(256) copy_csr_kernel(int nr, int64_t nnz, const int32_t *__restrict__ rp,
                                                       const int32_t *__restrict__ cl, const double *__restrict__ vl,
                                                       int32_t *__restrict__ orp, int32_t *__restrict__ ocl,
                                                       double *__restrict__ ovl) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x, t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (int64_t t = t0; t < nr; t += step) orp[t] = rp[t];
#pragma unroll 4
    for (int64_t t = t0; t < nnz; t += step) {
        ocl[t] = cl[t];
        ovl[t] = __ldcs(vl + t);
    }
}

// [P2]^3 blocks to scalar rows: a warp per block row, lanes along each scalar row (a scalar
// matrix is stored as the CSR it exports, ffgpu_matrix_csr copies it).  A thread per block row,
// its writes scattered over the warp's rows, took 567 us for 24.7 M entries; this, 104 us.
__global__ void __launch_bounds__(256) export_bsr3_kernel(int nb, const int32_t *__restrict__ browptr,
                                                          const int32_t *__restrict__ bcol, const double *__restrict__ val,
                                                          int32_t *__restrict__ rowptr, int32_t *__restrict__ col,
                                                          double *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t a = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (a >= nb) return;
    const int64_t b0 = browptr[a], deg = browptr[a + 1] - b0;
    if (lane < 3) rowptr[3 * a + lane] = (int32_t)(9 * b0 + 3 * lane * deg);
    if (lane == 3 && a == nb - 1) rowptr[3 * (int64_t)nb] = (int32_t)(9 * (int64_t)browptr[nb]);
    for (int c = 0; c < 3; ++c) {
        const int64_t r0 = 9 * b0 + 3 * c * deg;
        for (int64_t q = lane; q < 3 * deg; q += 32) {
            const int64_t k = q / 3, cp = q - 3 * k;
            col[r0 + q] = 3 * bcol[b0 + k] + (int)cp;
            out[r0 + q] = val[(b0 + k) * 9 + 3 * c + cp];
        }
    }
}

// ------------------------------------------------------------------ on(labels): DOF marking
// AssembleBC (problem.cpp:9881-10034) marks the DOFs of the boundary elements carrying one of
// the labels.  On the device: (1) vertices of the selected boundary elements, (2) vertex nodes
// of those vertices, (3) edge nodes whose two endpoints lie on one common selected boundary
// element (scanning the vertex -> boundary-element incidence of one endpoint).
__device__ __forceinline__ bool label_selected(int lab, int nlabels, const int32_t *labels) {
    for (int k = 0; k < nlabels; ++k)
        if (labels[k] == lab) return true;
    return false;
}

__global__ void bmark_vertices_kernel(int nbe, int bdim, const int32_t *belems, const int32_t *blabel,
                                      int nlabels, const int32_t *labels, uint8_t *vmark) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nbe || !label_selected(blabel[b], nlabels, labels)) return;
    for (int k = 0; k < bdim; ++k) vmark[belems[(int64_t)b * bdim + k]] = 1;
}

__device__ __forceinline__ void mark_node(uint8_t *onbc, int node, int bs, int comp_mask) {
    for (int c = 0; c < bs; ++c)
        if (comp_mask == 0 || (comp_mask >> c) & 1) onbc[(int64_t)node * bs + c] = 1;
}

// P1 without a DOF table: the nodes are the vertices (the same mask from the boundary elements
// alone; onbc is zero before)
__global__ void bmark_p1_kernel(int nbe, int bdim, const int32_t *belems, const int32_t *blabel, int nlabels,
                                const int32_t *labels, uint8_t *onbc) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nbe || !label_selected(blabel[b], nlabels, labels)) return;
    for (int k = 0; k < bdim; ++k) onbc[belems[(int64_t)b * bdim + k]] = 1;
}

template <int DIM>
__global__ void bmark_nodes_kernel(int nt, int nn, const int32_t *elems, const int32_t *nodes, const uint8_t *vmark,
                                   const int32_t *bv_ptr, const int32_t *bv_elem, const int32_t *belems,
                                   const int32_t *blabel, int nlabels, const int32_t *labels, int bs,
                                   int comp_mask, uint8_t *onbc) {
    constexpr int NV = DIM + 1;
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)nt * nn) return;
    int e = (int)(t / nn), i = (int)(t % nn);
    const int32_t *v = elems + (int64_t)e * NV;
    if (i < NV) {
        if (vmark[v[i]]) mark_node(onbc, nodes[t], bs, comp_mask);
        return;
    }
    int p, q;
    edge_vertices<DIM>(i - NV, p, q);
    int a = v[p], b = v[q];
    if (!vmark[a] || !vmark[b]) return;
    for (int k = bv_ptr[a]; k < bv_ptr[a + 1]; ++k) {
        int f = bv_elem[k];
        if (!label_selected(blabel[f], nlabels, labels)) continue;
        const int32_t *fv = belems + (int64_t)f * DIM;
        bool has_b = false;
        for (int j = 0; j < DIM; ++j) has_b |= fv[j] == b;
        if (has_b) { mark_node(onbc, nodes[t], bs, comp_mask); return; }
    }
}

// (vertex numbers out of range are skipped; the status word has them)
__global__ void bcount_kernel(int nbe, int bdim, int nv, const int32_t *belems, int32_t *cnt) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < (int64_t)nbe * bdim && (unsigned)belems[t] < (unsigned)nv) atomicAdd(&cnt[belems[t]], 1);
}

__global__ void bfill_kernel(int nbe, int bdim, int nv, const int32_t *belems, const int32_t *ptr, int32_t *cursor,
                             int32_t *out) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)nbe * bdim) return;
    int v = belems[t];
    if ((unsigned)v >= (unsigned)nv) return;
    out[ptr[v] + atomicAdd(&cursor[v], 1)] = (int32_t)(t / bdim);
}

__global__ void row_degree_kernel(int n, const int32_t *rp, int32_t *deg) {
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a < n) deg[a] = rp[a + 1] - rp[a];
}

// diagonal block of each row of a sorted CSR (-1 if absent)
__global__ void diagpos_kernel(int n, const int32_t *rp, const int32_t *col, int32_t *pos) {
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n) return;
    int lo = rp[a], hi = rp[a + 1] - 1, p = -1;
    while (lo <= hi) {
        int mid = (lo + hi) >> 1;
        int c = col[mid];
        if (c == a) { p = mid; break; }
        if (c < a) lo = mid + 1; else hi = mid - 1;
    }
    pos[a] = p;
}

static int grid_for(int64_t n, int block) { return (int)((n + block - 1) / block); }

int space_bc_mask_device(ffgpu_space *S, int nlabels, const int32_t *labels, int comp_mask, uint8_t *onbc) {
    FFGPU_CHECK(S->belems, FFGPU_EINVAL, "on(labels): the space has no boundary elements (ffgpu_space_set_boundary)");
    FFGPU_CHECK(nlabels > 0 && nlabels <= 64 && labels, FFGPU_EINVAL, "on(labels): 1..64 labels expected");
    ffgpu_ctx *ctx = S->ctx;
    cudaStream_t s = ctx->stream;
    DevIn<int32_t> lab(labels, nlabels, ctx);
    FFGPU_TRY(lab.err);
    FFGPU_CUDA(cudaMemsetAsync(onbc, 0, S->ndof, s));
    if (S->nodes == S->elems && !(comp_mask && !(comp_mask & 1))) {
        bmark_p1_kernel<<<grid_for(S->nbe, 256), 256, 0, s>>>(S->nbe, S->dim, S->belems, S->blabel, nlabels, lab.d, onbc);
        return launch_check(ctx, "bmark_p1");
    }
    FFGPU_CUDA(cudaMemsetAsync(S->vmark, 0, S->nv, s));
    bmark_vertices_kernel<<<grid_for(S->nbe, 256), 256, 0, s>>>(S->nbe, S->dim, S->belems, S->blabel, nlabels,
                                                                 lab.d, S->vmark);
    FFGPU_TRY(launch_check(ctx, "bmark_vertices"));
    int64_t m = (int64_t)S->nt * S->nn;
    if (S->dim == 2)
        bmark_nodes_kernel<2><<<grid_for(m, 256), 256, 0, s>>>(S->nt, S->nn, S->elems, S->nodes, S->vmark, S->bv_ptr,
                                                               S->bv_elem, S->belems, S->blabel, nlabels, lab.d,
                                                               S->bs, comp_mask, onbc);
    else
        bmark_nodes_kernel<3><<<grid_for(m, 256), 256, 0, s>>>(S->nt, S->nn, S->elems, S->nodes, S->vmark, S->bv_ptr,
                                                               S->bv_elem, S->belems, S->blabel, nlabels, lab.d,
                                                               S->bs, comp_mask, onbc);
    return launch_check(ctx, "bmark_nodes");
}

}  // namespace ffgpu

using namespace ffgpu;

// ------------------------------------------------------------------ helpers on the host
static int fill_launch(ffgpu_space *S, FillArgs &fa) {
    ffgpu_ctx *ctx = S->ctx;
    const int bs2 = S->bs * S->bs, rw = 32 / (S->nn * S->bs);
    // a row above this degree has always been refused
    FFGPU_CHECK((size_t)4 * (kCandMax * sizeof(int) + (size_t)(32 / S->nn) * fa.max_deg * bs2 * sizeof(double)) <= 200 * 1024,
                FFGPU_EMESH, "row degree %d too large for shared memory", fa.max_deg);
    const bool plain = (S->fe == FFGPU_FE_P2VEC3 ? fa.eloc : fa.kloc) && !fa.has_mass && !fa.mloc && !fa.tloc;
    void (*kern)(FillArgs) = nullptr;
    if (S->dim == 2 && S->fe == FFGPU_FE_P1) kern = plain ? fill_kernel<2, 1, true> : fill_kernel<2, 1, false>;
    if (S->dim == 3 && S->fe == FFGPU_FE_P1) kern = plain ? fill_kernel<3, 1, true> : fill_kernel<3, 1, false>;
    if (S->dim == 2 && S->fe == FFGPU_FE_P2) kern = plain ? fill_kernel<2, 2, true> : fill_kernel<2, 2, false>;
    if (S->dim == 3 && S->fe == FFGPU_FE_P2) kern = plain ? fill_kernel<3, 2, true> : fill_kernel<3, 2, false>;
    if (S->dim == 3 && S->fe == FFGPU_FE_P2VEC3) kern = plain ? fill_kernel<3, 3, true> : fill_kernel<3, 3, false>;
    FFGPU_CHECK(kern, FFGPU_EINVAL, "unsupported element (dim %d, fe %d)", S->dim, S->fe);
    // warps per block: 8, fewer where rows are long (48 KB of row buffers a block keep the SM full)
    const size_t per_warp = (size_t)rw * fa.max_deg * bs2 * sizeof(double);
    int warps = 8;
    while (warps > 1 && warps * per_warp > 48 * 1024) warps >>= 1;
    const size_t smem = warps * per_warp;
    const int64_t need = ((int64_t)S->nnodes + warps * rw - 1) / (warps * rw);
    FFGPU_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<(int)std::min<int64_t>(kNumSM * 32, std::max<int64_t>(1, need)), warps * 32, smem, ctx->stream>>>(fa);
    return launch_check(ctx, "fill_kernel");
}

static int pattern_launch(ffgpu_space *S, int32_t *deg, int32_t *tmpcol, uint16_t *rmap, int32_t *drank) {
    ffgpu_ctx *ctx = S->ctx;
    int logH = 5;
    while ((1 << logH) < S->max_inc * S->nn && logH < 9) ++logH;   // kCandMax = 512 candidates at most
    const size_t smem = (size_t)4 * 3 * sizeof(int) << logH;
    const int grid = std::min(kNumSM * 16, std::max(1, (S->nnodes + 3) / 4));
#define FFGPU_PATTERN(NN)                                                                                        \
    pattern_kernel<NN><<<grid, 128, smem, ctx->stream>>>(S->nnodes, S->inc_ptr, S->inc, S->nodes, logH, deg, \
                                                         tmpcol, rmap, drank, ctx->d_status)
    switch (S->nn) {
        case 3: FFGPU_PATTERN(3); break;
        case 4: FFGPU_PATTERN(4); break;
        case 6: FFGPU_PATTERN(6); break;
        default: FFGPU_PATTERN(10); break;
    }
#undef FFGPU_PATTERN
    return launch_check(ctx, "pattern_kernel");
}

static int rhs_launch(ffgpu_space *S, const double *measure, int mstride, const double *fP0, const double *fint,
                      const double *f, const uint8_t *mask, const double *g, double tgv, double *rhs,
                      const BoundaryTerms &bt) {
    auto k = rhs_kernel<2, 1>;
    if (S->dim == 3 && S->fe == FFGPU_FE_P1) k = rhs_kernel<3, 1>;
    if (S->dim == 2 && S->fe == FFGPU_FE_P2) k = rhs_kernel<2, 2>;
    if (S->dim == 3 && S->fe == FFGPU_FE_P2) k = rhs_kernel<3, 2>;
    if (S->dim == 3 && S->fe == FFGPU_FE_P2VEC3) k = rhs_kernel<3, 3>;
    k<<<grid_for((int64_t)S->ndof, 256), 256, 0, S->ctx->stream>>>(S->nnodes, S->inc_ptr, S->inc, measure,
                                                                   mstride, fP0, fint, f[0], f[1], f[2], mask, g, tgv, rhs,
                                                                   bt.rhs ? bt.ptr : nullptr, bt.list, bt.rhs);
    return launch_check(S->ctx, "rhs_kernel");
}

// P1 element matrices (out) and measures, either may be NULL
static int p1_elem_launch(ffgpu_space *S, const double *kappa, double c_stiff, double c_mass, double *out, double *measure) {
    auto k = S->dim == 2 ? p1_elem_kernel<2> : p1_elem_kernel<3>;
    k<<<grid_for(S->nt, 256), 256, 0, S->ctx->stream>>>(S->coords, S->elems, S->nt, kappa, c_stiff, c_mass, out, measure);
    return launch_check(S->ctx, "p1_elem_kernel");
}

static int varf_check(const ffgpu_space *S, const ffgpu_varf *v) {
    FFGPU_CHECK(v, FFGPU_EINVAL, "varf is NULL");
    if (v->form == FFGPU_FORM_ELASTICITY)
        FFGPU_CHECK(S->fe == FFGPU_FE_P2VEC3, FFGPU_EINVAL, "elasticity needs the [P2,P2,P2] space");
    else
        FFGPU_CHECK(v->form == FFGPU_FORM_DIFFUSION && S->fe != FFGPU_FE_P2VEC3, FFGPU_EINVAL,
                    "unsupported form %d for this space", v->form);
    return FFGPU_OK;
}

static int run_geometry(ffgpu_space *S, const ffgpu_varf *v, double *geo) {
    ffgpu_ctx *ctx = S->ctx;
    DevIn<double> kap(v->kappa, v->kappa ? S->nt : 0, ctx);
    FFGPU_TRY(kap.err);
    double cs = v->form == FFGPU_FORM_DIFFUSION ? v->c_stiff : 1.0;
    geometry_kernel<<<grid_for(S->nt, 256), 256, 0, ctx->stream>>>(S->coords, S->elems, S->nt, S->dim,
                                                                   kap.d, cs, geo);
    return launch_check(ctx, "geometry_kernel");
}

// the varf needs the element geometry (measure, gradients) beyond the P1 element matrices
static bool needs_geometry(const ffgpu_space *S, const ffgpu_varf *v) {
    return S->fe != FFGPU_FE_P1 || v->f_qp || v->mass_qp || v->stiff_qp || v->f_expr || v->nterms > 0;
}

// Measures and gradients of the elements in M->geo.  P1 reads nothing else there, so it is formed
// once per matrix and only when something asks for it; P2 also keeps kappa in it.
int ffgpu::matrix_geometry(ffgpu_matrix *M, const ffgpu_varf *v) {
    ffgpu_space *S = M->space;
    if (M->geo && S->fe == FFGPU_FE_P1) return FFGPU_OK;
    if (!M->geo && dalloc(M->ctx, (void **)&M->geo, sizeof(double) * kGeoStride * S->nt) != cudaSuccess) {
        set_error("element geometry: device allocation failed");
        return FFGPU_ENOMEM;
    }
    return run_geometry(S, v, M->geo);
}

// tmpcol, drank: what pattern_kernel left (first numeric pass of a matrix), else NULL
static int numeric_pass(ffgpu_matrix *M, const ffgpu_varf *v, const ffgpu_bc *bc, double *rhs,
                        const int32_t *tmpcol, const int32_t *drank) {
    ffgpu_space *S = M->space;
    ffgpu_ctx *ctx = S->ctx;
    FFGPU_TRY(varf_check(S, v));
    int bs = S->bs;
    DevIn<double> fP0(v->f, v->f ? (size_t)S->nt * bs : 0, ctx);
    DevIn<double> kap(v->kappa, v->kappa && S->fe == FFGPU_FE_P1 ? S->nt : 0, ctx);
    DevIn<uint8_t> onbc(bc ? bc->onbc : nullptr, bc && bc->onbc ? S->ndof : 0, ctx);
    DevIn<double> gv(bc ? bc->g : nullptr, bc && bc->g ? S->ndof : 0, ctx);
    DevOut<double> rh(rhs, rhs ? S->ndof : 0, ctx, false);
    FFGPU_TRY(fP0.err); FFGPU_TRY(kap.err); FFGPU_TRY(onbc.err); FFGPU_TRY(gv.err); FFGPU_TRY(rh.err);
    if (needs_geometry(S, v)) FFGPU_TRY(matrix_geometry(M, v));
    const uint8_t *mask = onbc.d;
    if (bc && !bc->onbc && bc->nlabels > 0) {
        if (!M->bcmask) FFGPU_CUDA(dalloc(ctx, (void **)&M->bcmask, S->ndof));
        FFGPU_TRY(space_bc_mask_device(S, bc->nlabels, bc->labels, bc->comp_mask, M->bcmask));
        mask = M->bcmask;
    }
    FillArgs fa;
    memset(&fa, 0, sizeof(fa));
    fa.nnodes = S->nnodes;
    fa.inc_ptr = S->inc_ptr; fa.inc = S->inc;
    fa.nodes = S->nodes; fa.geo = M->geo; fa.browptr = M->browptr;
    fa.bcol = M->bcol; fa.rmap = M->rmap; fa.tmpcol = tmpcol; fa.drank = drank;
    fa.diagpos = M->diagpos;
    fa.val = M->val;
    fa.c_mass = v->form == FFGPU_FORM_DIFFUSION && !v->mass_qp ? v->c_mass : 0.0;
    if (v->form == FFGPU_FORM_ELASTICITY) {
        fa.mu = v->E / (2 * (1 + v->nu));
        fa.lam = v->E * v->nu / ((1 + v->nu) * (1 - 2 * v->nu));
    }
    fa.onbc = mask; fa.tgv = bc ? bc->tgv : 0.0;
    fa.tgv_rows = mask && fa.tgv > 0;
    fa.neg = mask ? neg_tgv_bits(fa.tgv) : 0;
    fa.max_deg = M->max_deg; fa.status = ctx->d_status;
    DevIn<double> lame(v->form == FFGPU_FORM_ELASTICITY ? v->lame : nullptr, (size_t)S->nt * 2, ctx);
    FFGPU_TRY(lame.err);
    fa.lame = lame.d;
    double *fint = nullptr, *mloc = nullptr, *kloc = nullptr, *tloc = nullptr, *eloc = nullptr, *meas = nullptr;
    int frc = rh.d ? source_prepare(S, v, M->geo, &fint) : FFGPU_OK;
    if (!frc) frc = mass_prepare(S, v, M->geo, &mloc);
    if (!frc) frc = stiff_prepare(S, v, M->geo, &kloc);
    if (!frc) frc = terms_prepare(S, v, M->geo, &tloc);
    fa.kloc = kloc;
    fa.krs = S->nn;
    if (!frc && S->fe == FFGPU_FE_P1) {
        // P1: closed form, the mass term included; only the measures where the stiffness comes
        // from values at quadrature points
        if (rh.d && dalloc(ctx, (void **)&meas, sizeof(double) * S->nt)) frc = FFGPU_ENOMEM;
        if (!frc && !kloc && dalloc(ctx, (void **)&eloc, sizeof(double) * 4 * S->nn * S->nt)) frc = FFGPU_ENOMEM;
        if (frc) set_error("assembly: allocation of the element matrices failed");
        if (!frc && (eloc || meas)) frc = p1_elem_launch(S, kap.d, v->c_stiff, fa.c_mass, eloc, meas);
        if (eloc) { fa.kloc = eloc; fa.krs = 4; fa.c_mass = 0.0; }
    } else if (!frc && !kloc && (S->fe == FFGPU_FE_P2VEC3 || v->c_stiff != 0.0)) {
        // P2 stiffness / [P2]^3 elasticity with an element-constant coefficient: the element
        // matrices from the tensor cores (a coefficient at the rule's points keeps its own path)
        frc = elem_tc_prepare(S, M->geo, fa.lam, fa.mu, lame.d, &eloc);
        if (S->fe == FFGPU_FE_P2 && eloc) fa.kloc = eloc;
        if (S->fe == FFGPU_FE_P2VEC3) fa.eloc = eloc;
    }
    fa.has_mass = fa.c_mass != 0.0;
    fa.mloc = mloc;
    fa.tloc = tloc;
    BoundaryTerms bt;
    if (!frc) frc = boundary_prepare(S, v, rh.d != nullptr, true, bt);
    if (!frc) {
        fa.bptr = bt.ptr; fa.blist = bt.list; fa.bel_elem = bt.bel_elem; fa.bmat = bt.mat;
        frc = fill_launch(S, fa);
        if (!frc && rh.d)
            frc = rhs_launch(S, meas ? meas : M->geo, meas ? 1 : kGeoStride, fP0.d, fint, v->f_const, mask, gv.d, fa.tgv,
                             rh.d, bt);
        boundary_release(S, bt);
    }
    dfree(ctx, fint);
    dfree(ctx, mloc);
    dfree(ctx, kloc);
    dfree(ctx, tloc);
    dfree(ctx, eloc);
    dfree(ctx, meas);
    FFGPU_TRY(frc);
    FFGPU_TRY(check_device_status(ctx, "assembly"));
    FFGPU_TRY(rh.finish());
    // the solver data of a previous numeric state are stale; so is a cached CG graph, which
    // holds the addresses of the derived value arrays
    M->ntgv = -1;
    if (M->val_t) { dfree(ctx, M->val_t); M->val_t = nullptr; }
    if (M->val32) { dfree(ctx, M->val32); M->val32 = nullptr; }
    if (M->valx) { dfree(ctx, M->valx); M->valx = nullptr; }
    if (M->valx_t) { dfree(ctx, M->valx_t); M->valx_t = nullptr; }
    sell_release_values(M);
    direct_invalidate(M);
    if (M->cg_exec) { cudaGraphExecDestroy(M->cg_exec); M->cg_exec = nullptr; }
    return FFGPU_OK;
}

extern "C" {

int ffgpu_space_create(ffgpu_ctx *ctx, int dim, int nv, const double *coords, int nt,
                       const int32_t *elems, int fe, int ndofK, const int32_t *dof, int ndof,
                       ffgpu_space **out) {
    FFGPU_CHECK(ctx && out && coords && elems && (dof || fe == FFGPU_FE_P1), FFGPU_EINVAL,
                "ffgpu_space_create: NULL argument");
    FFGPU_CHECK(dof || ndof == nv, FFGPU_EINVAL,
                "ffgpu_space_create: P1 without a DOF table needs ndof == nv (got %d, nv %d)", ndof, nv);
    FFGPU_CHECK(dim == 2 || dim == 3, FFGPU_EINVAL, "dim must be 2 or 3");
    FFGPU_CHECK(nv > 0 && nt > 0 && ndof > 0, FFGPU_EINVAL, "empty mesh or space");
    int nvk = dim + 1, nn, bs;
    if (fe == FFGPU_FE_P1) { nn = nvk; bs = 1; }
    else if (fe == FFGPU_FE_P2) { nn = dim == 3 ? 10 : 6; bs = 1; }
    else if (fe == FFGPU_FE_P2VEC3) { FFGPU_CHECK(dim == 3, FFGPU_EINVAL, "[P2]^3 needs dim 3"); nn = 10; bs = 3; }
    else { set_error("unknown finite element %d", fe); return FFGPU_EINVAL; }
    FFGPU_CHECK(ndofK == nn * bs, FFGPU_EINVAL, "ndofK %d does not match the element (%d)", ndofK, nn * bs);
    FFGPU_CHECK(ndof % bs == 0, FFGPU_EINVAL, "ndof %d not a multiple of %d", ndof, bs);
    FFGPU_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    ffgpu_space *S = new ffgpu_space();
    memset(S, 0, sizeof(*S));
    S->ctx = ctx; S->dim = dim; S->nvk = nvk; S->nv = nv; S->nt = nt; S->fe = fe; S->nn = nn;
    S->bs = bs; S->ndofK = ndofK; S->ndof = ndof; S->nnodes = ndof / bs;
    int64_t m = (int64_t)nt * nn;
    int rc = FFGPU_OK;
    int32_t *cnt = nullptr, *unsorted = nullptr;
    uint16_t *at = nullptr;
    {
        DevIn<int32_t> D(dof, dof ? (size_t)nt * ndofK : 0, ctx);   // NULL (P1): the vertices
        if (D.err) { rc = D.err; goto fail; }
        if (dalloc(ctx, (void **)&S->coords, sizeof(double) * nv * dim) ||
            dalloc(ctx, (void **)&S->elems, sizeof(int32_t) * nt * nvk) ||
            (dof && dalloc(ctx, (void **)&S->nodes, sizeof(int32_t) * m)) ||
            dalloc(ctx, (void **)&S->inc_ptr, sizeof(int32_t) * (S->nnodes + 1)) ||
            dalloc(ctx, (void **)&S->inc, sizeof(int32_t) * m) ||
            dalloc(ctx, (void **)&cnt, sizeof(int32_t) * (S->nnodes + 1)) ||
            dalloc(ctx, (void **)&at, sizeof(uint16_t) * m) || dalloc(ctx, (void **)&unsorted, sizeof(int32_t) * m)) {
            set_error("ffgpu_space_create: device allocation failed");
            rc = FFGPU_ENOMEM; goto fail;
        }
        if (!dof) S->nodes = S->elems;   // P1 without a table: the nodes are the vertices
        // host or device arrays, copied straight into the space's own buffers
        if (cudaMemcpyAsync(S->coords, coords, sizeof(double) * nv * dim, cudaMemcpyDefault, s) ||
            cudaMemcpyAsync(S->elems, elems, sizeof(int32_t) * nt * nvk, cudaMemcpyDefault, s)) {
            set_error("ffgpu_space_create: copy of the mesh failed");
            rc = FFGPU_ECUDA; goto fail;
        }
        check_elems_kernel<<<grid_for(((int64_t)nt * nvk + 3) / 4, 256), 256, 0, s>>>(S->elems, (int64_t)nt * nvk, nv,
                                                                                       ctx->d_status);
        if ((rc = launch_check(ctx, "check_elems"))) goto fail;
        if (dof) {
            build_nodes_kernel<<<grid_for(m, 256), 256, 0, s>>>(D.d, nt, ndofK, nn, bs, ndof, S->nodes, ctx->d_status);
            if ((rc = launch_check(ctx, "build_nodes"))) goto fail;
        }
    }
    cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (S->nnodes + 1), s);
    inc_count_kernel<<<grid_for(m, 256), 256, 0, s>>>(S->nodes, m, S->nnodes, cnt, at);
    if ((rc = launch_check(ctx, "inc_count"))) goto fail;
    if ((rc = device_max_status(ctx, cnt, S->nnodes, nullptr, "ffgpu_space_create", &S->max_inc, nullptr))) goto fail;
    {
        // the bounds of the pattern pass (which also keep the arrival numbers in 16 bits)
        int P = 1;
        while (P < S->max_inc) P <<= 1;
        if ((size_t)4 * P * sizeof(long long) > 200 * 1024 || (int64_t)S->max_inc * nn > kCandMax) {
            set_error("node valence %d too high (at most %d candidate neighbours)", S->max_inc, kCandMax);
            rc = FFGPU_EMESH; goto fail;
        }
    }
    if ((rc = device_scan_i32(ctx, cnt, S->inc_ptr, S->nnodes))) goto fail;
    inc_fill_kernel<<<grid_for(m, 256), 256, 0, s>>>(S->nodes, m, S->inc_ptr, at, unsorted);
    if ((rc = launch_check(ctx, "inc_fill"))) goto fail;
    if (m <= (int64_t)8 * S->nnodes)
        inc_sort_kernel<8><<<min(kNumSM * 64, grid_for((int64_t)S->nnodes * 8, 256)), 256, 0, s>>>(S->inc_ptr, S->nnodes,
                                                                                                    unsorted, S->inc);
    else
        inc_sort_kernel<32><<<min(kNumSM * 64, grid_for((int64_t)S->nnodes * 32, 256)), 256, 0, s>>>(S->inc_ptr, S->nnodes,
                                                                                                      unsorted, S->inc);
    if ((rc = launch_check(ctx, "inc_sort"))) goto fail;
    dfree(ctx, at);
    dfree(ctx, unsorted);
    at = nullptr;
    unsorted = nullptr;
    dfree(ctx, cnt);
    cnt = nullptr;
    if (cudaStreamSynchronize(s) != cudaSuccess) {
        set_error("ffgpu_space_create: %s", cudaGetErrorString(cudaGetLastError()));
        rc = FFGPU_ECUDA; goto fail;
    }
    *out = S;
    return FFGPU_OK;
fail:
    dfree(ctx, cnt);
    dfree(ctx, at);
    dfree(ctx, unsorted);
    ffgpu_space_destroy(S);
    return rc;
}

int ffgpu_space_destroy(ffgpu_space *S) {
    if (!S) return FFGPU_OK;
    cudaStreamSynchronize(S->ctx->stream);
    dfree(S->ctx, S->coords);
    if (S->nodes != S->elems) dfree(S->ctx, S->nodes);
    dfree(S->ctx, S->elems);
    dfree(S->ctx, S->inc_ptr); dfree(S->ctx, S->inc);
    dfree(S->ctx, S->belems); dfree(S->ctx, S->blabel); dfree(S->ctx, S->bv_ptr); dfree(S->ctx, S->bv_elem); dfree(S->ctx, S->vmark);
    dfree(S->ctx, S->bel_elem); dfree(S->ctx, S->bel_face);
    delete S;
    return FFGPU_OK;
}

int ffgpu_space_set_boundary(ffgpu_space *S, int nbe, const int32_t *belems, const int32_t *blabel) {
    FFGPU_CHECK(S && nbe > 0 && belems && blabel, FFGPU_EINVAL, "ffgpu_space_set_boundary: bad argument");
    ffgpu_ctx *ctx = S->ctx;
    FFGPU_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    const int bdim = S->dim;   // vertices per boundary element
    dfree(ctx, S->belems); dfree(ctx, S->blabel); dfree(ctx, S->bv_ptr); dfree(ctx, S->bv_elem); dfree(ctx, S->vmark);
    dfree(ctx, S->bel_elem); dfree(ctx, S->bel_face);
    S->belems = S->blabel = S->bv_ptr = S->bv_elem = S->bel_elem = S->bel_face = nullptr;
    S->vmark = nullptr;
    S->nbe = nbe;
    int32_t *cnt = nullptr;
    if (dalloc(ctx, (void **)&S->belems, sizeof(int32_t) * nbe * bdim) ||
        dalloc(ctx, (void **)&S->blabel, sizeof(int32_t) * nbe) ||
        dalloc(ctx, (void **)&S->bv_ptr, sizeof(int32_t) * (S->nv + 1)) ||
        dalloc(ctx, (void **)&S->bv_elem, sizeof(int32_t) * nbe * bdim) ||
        dalloc(ctx, (void **)&S->vmark, S->nv) ||
        dalloc(ctx, (void **)&cnt, sizeof(int32_t) * (S->nv + 1))) {
        set_error("ffgpu_space_set_boundary: device allocation failed");
        dfree(ctx, cnt);
        return FFGPU_ENOMEM;
    }
    FFGPU_CUDA(cudaMemcpyAsync(S->belems, belems, sizeof(int32_t) * nbe * bdim, cudaMemcpyDefault, s));
    FFGPU_CUDA(cudaMemcpyAsync(S->blabel, blabel, sizeof(int32_t) * nbe, cudaMemcpyDefault, s));
    check_elems_kernel<<<grid_for(((int64_t)nbe * bdim + 3) / 4, 256), 256, 0, s>>>(S->belems, (int64_t)nbe * bdim, S->nv,
                                                                                     ctx->d_status);
    FFGPU_TRY(launch_check(ctx, "check_belems"));
    cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (S->nv + 1), s);
    bcount_kernel<<<grid_for((int64_t)nbe * bdim, 256), 256, 0, s>>>(nbe, bdim, S->nv, S->belems, cnt);
    int rc = launch_check(ctx, "bcount");
    if (!rc) rc = device_scan_i32(ctx, cnt, S->bv_ptr, S->nv);
    if (!rc) {
        cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (S->nv + 1), s);
        bfill_kernel<<<grid_for((int64_t)nbe * bdim, 256), 256, 0, s>>>(nbe, bdim, S->nv, S->belems, S->bv_ptr, cnt,
                                                                         S->bv_elem);
        rc = launch_check(ctx, "bfill");
    }
    if (!rc) rc = check_device_status(ctx, "ffgpu_space_set_boundary");
    dfree(ctx, cnt);
    if (!rc && cudaStreamSynchronize(s) != cudaSuccess) { set_error("ffgpu_space_set_boundary failed"); rc = FFGPU_ECUDA; }
    return rc;
}

int ffgpu_space_bc_mask(ffgpu_space *S, int nlabels, const int32_t *labels, int comp_mask, uint8_t *onbc) {
    FFGPU_CHECK(S && onbc, FFGPU_EINVAL, "ffgpu_space_bc_mask: NULL argument");
    cudaStream_t s = S->ctx->stream;
    FFGPU_CUDA(cudaSetDevice(S->ctx->device));
    DevOut<uint8_t> m(onbc, S->ndof, S->ctx, false);
    FFGPU_TRY(m.err);
    FFGPU_TRY(space_bc_mask_device(S, nlabels, labels, comp_mask, m.d));
    FFGPU_TRY(m.finish());
    FFGPU_CUDA(cudaStreamSynchronize(s));
    return FFGPU_OK;
}

int ffgpu_matrix_assemble(ffgpu_space *S, const ffgpu_varf *v, const ffgpu_bc *bc, double *rhs,
                          ffgpu_matrix **out) {
    FFGPU_CHECK(S && out, FFGPU_EINVAL, "ffgpu_matrix_assemble: NULL argument");
    FFGPU_TRY(varf_check(S, v));
    ffgpu_ctx *ctx = S->ctx;
    cudaStream_t s = ctx->stream;
    FFGPU_CUDA(cudaSetDevice(ctx->device));
    ffgpu_matrix *M = new ffgpu_matrix();
    memset(M, 0, sizeof(*M));
    M->ctx = ctx; M->space = S; M->bs = S->bs; M->nb = S->nnodes; M->n = S->ndof;
    M->ntgv = -1; M->csr_lanes = 0;
    int rc = FFGPU_OK;
    int32_t *deg = nullptr, *tmpcol = nullptr, *drank = nullptr;
    const size_t cand = (size_t)S->nt * S->nn * S->nn;   // nodes of all incidences
    if (dalloc(ctx, (void **)&M->browptr, sizeof(int32_t) * (M->nb + 1)) ||
        dalloc(ctx, (void **)&deg, sizeof(int32_t) * (M->nb + 1)) ||
        dalloc(ctx, (void **)&drank, sizeof(int32_t) * M->nb) ||
        dalloc(ctx, (void **)&tmpcol, sizeof(int32_t) * cand) ||
        dalloc(ctx, (void **)&M->rmap, sizeof(uint16_t) * cand)) {
        set_error("ffgpu_matrix_assemble: device allocation failed");
        rc = FFGPU_ENOMEM; goto fail;
    }
    // symbolic: the rows' columns and degrees, row pointer
    if ((rc = pattern_launch(S, deg, tmpcol, M->rmap, drank))) goto fail;
    if ((rc = device_scan_i32(ctx, deg, M->browptr, M->nb))) goto fail;
    {
        int32_t nnzb = 0;
        if ((rc = device_max_status(ctx, deg, M->nb, M->browptr + M->nb, "pattern", &M->max_deg, &nnzb))) goto fail;
        M->nnzb = nnzb;
        M->nnz = M->nnzb * M->bs * M->bs;
    }
    // SpMV row order: block rows grouped by degree so that the lanes of a warp share trip counts
    if (dalloc(ctx, (void **)&M->rowperm, sizeof(int32_t) * M->nb)) {
        set_error("ffgpu_matrix_assemble: device allocation failed");
        rc = FFGPU_ENOMEM; goto fail;
    }
    if ((rc = device_order_by_key_desc(ctx, deg, M->nb, M->max_deg, M->rowperm))) goto fail;
    dfree(ctx, deg);
    deg = nullptr;
    if (dalloc(ctx, (void **)&M->bcol, sizeof(int32_t) * M->nnzb) ||
        dalloc(ctx, (void **)&M->diagpos, sizeof(int32_t) * M->nb) ||
        dalloc(ctx, (void **)&M->val, sizeof(double) * M->nnz)) {
        set_error("ffgpu_matrix_assemble: allocation of %lld values failed", (long long)M->nnz);
        rc = FFGPU_ENOMEM; goto fail;
    }
    if ((rc = numeric_pass(M, v, bc, rhs, tmpcol, drank))) goto fail;
    dfree(ctx, tmpcol);
    dfree(ctx, drank);
    *out = M;
    return FFGPU_OK;
fail:
    dfree(ctx, deg);
    dfree(ctx, tmpcol);
    dfree(ctx, drank);
    ffgpu_matrix_destroy(M);
    return rc;
}

int ffgpu_matrix_reassemble(ffgpu_matrix *M, const ffgpu_varf *v, const ffgpu_bc *bc, double *rhs) {
    FFGPU_CHECK(M && M->space, FFGPU_EINVAL, "ffgpu_matrix_reassemble: matrix has no FE space");
    FFGPU_CUDA(cudaSetDevice(M->ctx->device));
    return numeric_pass(M, v, bc, rhs, nullptr, nullptr);
}

int ffgpu_rhs_assemble(ffgpu_space *S, const ffgpu_varf *v, const ffgpu_bc *bc, double *rhs) {
    FFGPU_CHECK(S && v && rhs, FFGPU_EINVAL, "ffgpu_rhs_assemble: NULL argument");
    FFGPU_TRY(varf_check(S, v));
    ffgpu_ctx *ctx = S->ctx;
    cudaStream_t s = ctx->stream;
    FFGPU_CUDA(cudaSetDevice(ctx->device));
    // P1 with a source per element needs the measures only
    const bool full = S->fe != FFGPU_FE_P1 || v->f_qp || v->f_expr;
    double *geo = nullptr;
    FFGPU_CUDA(dalloc(ctx, (void **)&geo, sizeof(double) * (full ? kGeoStride : 1) * S->nt));
    int rc = full ? run_geometry(S, v, geo) : p1_elem_launch(S, nullptr, 0.0, 0.0, nullptr, geo);
    {
        DevIn<double> fP0(v->f, v->f ? (size_t)S->nt * S->bs : 0, ctx);
        DevIn<uint8_t> onbc(bc ? bc->onbc : nullptr, bc && bc->onbc ? S->ndof : 0, ctx);
        DevIn<double> gv(bc ? bc->g : nullptr, bc && bc->g ? S->ndof : 0, ctx);
        DevOut<double> rh(rhs, S->ndof, ctx, false);
        if (!rc) rc = fP0.err ? fP0.err : (onbc.err ? onbc.err : (gv.err ? gv.err : rh.err));
        uint8_t *lmask = nullptr;
        const uint8_t *mask = onbc.d;
        if (!rc && bc && !bc->onbc && bc->nlabels > 0) {
            if (dalloc(ctx, (void **)&lmask, S->ndof) != cudaSuccess) rc = FFGPU_ENOMEM;
            if (!rc) rc = space_bc_mask_device(S, bc->nlabels, bc->labels, bc->comp_mask, lmask);
            mask = lmask;
        }
        BoundaryTerms bt;
        double *fint = nullptr;
        if (!rc) rc = source_prepare(S, v, geo, &fint);
        if (!rc) rc = boundary_prepare(S, v, true, false, bt);
        if (!rc)
            rc = rhs_launch(S, geo, full ? kGeoStride : 1, fP0.d, fint, v->f_const, mask, gv.d, bc ? bc->tgv : 0.0, rh.d, bt);
        boundary_release(S, bt);
        dfree(ctx, fint);
        if (!rc) rc = rh.finish();
        if (lmask) dfree(ctx, lmask);
    }
    dfree(ctx, geo);
    cudaStreamSynchronize(s);
    return rc;
}

int ffgpu_matrix_from_csr(ffgpu_ctx *ctx, int n, int64_t nnz, const int32_t *rowptr,
                          const int32_t *col, const double *val, ffgpu_matrix **out) {
    FFGPU_CHECK(ctx && out && rowptr && col && val && n > 0 && nnz > 0, FFGPU_EINVAL,
                "ffgpu_matrix_from_csr: bad argument");
    FFGPU_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    ffgpu_matrix *M = new ffgpu_matrix();
    memset(M, 0, sizeof(*M));
    M->ctx = ctx; M->bs = 1; M->nb = n; M->n = n; M->nnzb = nnz; M->nnz = nnz; M->ntgv = -1;
    if (dalloc(ctx, (void **)&M->browptr, sizeof(int32_t) * (n + 1)) ||
        dalloc(ctx, (void **)&M->bcol, sizeof(int32_t) * nnz) ||
        dalloc(ctx, (void **)&M->diagpos, sizeof(int32_t) * n) ||
        dalloc(ctx, (void **)&M->val, sizeof(double) * nnz)) {
        set_error("ffgpu_matrix_from_csr: device allocation failed");
        ffgpu_matrix_destroy(M);
        return FFGPU_ENOMEM;
    }
    cudaMemcpyAsync(M->browptr, rowptr, sizeof(int32_t) * (n + 1), cudaMemcpyDefault, s);
    cudaMemcpyAsync(M->bcol, col, sizeof(int32_t) * nnz, cudaMemcpyDefault, s);
    cudaMemcpyAsync(M->val, val, sizeof(double) * nnz, cudaMemcpyDefault, s);
    {
        int32_t first = -1, last = -1;
        cudaMemcpyAsync(&first, M->browptr, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(&last, M->browptr + n, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
        FFGPU_CUDA(cudaStreamSynchronize(s));
        if (first != 0 || last != nnz) {
            set_error("rowptr inconsistent with nnz");
            ffgpu_matrix_destroy(M);
            return FFGPU_EINVAL;
        }
        int32_t *deg = nullptr;
        FFGPU_CUDA(dalloc(ctx, (void **)&deg, sizeof(int32_t) * n));
        row_degree_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, M->browptr, deg);
        int rc = launch_check(ctx, "row_degree");
        if (!rc) rc = device_max_i32(ctx, deg, n, &M->max_deg);
        if (!rc && dalloc(ctx, (void **)&M->rowperm, sizeof(int32_t) * n)) { set_error("allocation failed"); rc = FFGPU_ENOMEM; }
        if (!rc) rc = device_order_by_key_desc(ctx, deg, n, M->max_deg, M->rowperm);
        dfree(ctx, deg);
        if (rc) { ffgpu_matrix_destroy(M); return rc; }
    }
    diagpos_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, M->browptr, M->bcol, M->diagpos);
    FFGPU_TRY(launch_check(ctx, "diagpos"));
    FFGPU_CUDA(cudaStreamSynchronize(s));
    *out = M;
    return FFGPU_OK;
}

int ffgpu_matrix_destroy(ffgpu_matrix *M) {
    if (!M) return FFGPU_OK;
    cudaStreamSynchronize(M->ctx->stream);
    if (M->cg_exec) cudaGraphExecDestroy(M->cg_exec);
    direct_release(M);
    dfree(M->ctx, M->browptr); dfree(M->ctx, M->bcol); dfree(M->ctx, M->diagpos); dfree(M->ctx, M->rowperm); dfree(M->ctx, M->val);
    dfree(M->ctx, M->geo); dfree(M->ctx, M->bcmask); dfree(M->ctx, M->rmap);
    dfree(M->ctx, M->band_perm);
    dfree(M->ctx, M->diag_inv); dfree(M->ctx, M->wcl); dfree(M->ctx, M->vec); dfree(M->ctx, M->val_t);
    dfree(M->ctx, M->val32); dfree(M->ctx, M->valx); dfree(M->ctx, M->valx_t); dfree(M->ctx, M->hx); dfree(M->ctx, M->ks);
    sell_release(M);
    delete M;
    return FFGPU_OK;
}

int ffgpu_matrix_info(const ffgpu_matrix *M, int *n, int64_t *nnz, int *bs) {
    FFGPU_CHECK(M, FFGPU_EINVAL, "ffgpu_matrix_info: NULL matrix");
    if (n) *n = M->n;
    if (nnz) *nnz = M->nnz;
    if (bs) *bs = M->bs;
    return FFGPU_OK;
}

int ffgpu_matrix_csr(const ffgpu_matrix *M, int32_t *rowptr, int32_t *col, double *val) {
    FFGPU_CHECK(M && rowptr && col && val, FFGPU_EINVAL, "ffgpu_matrix_csr: NULL argument");
    ffgpu_ctx *ctx = M->ctx;
    cudaStream_t s = ctx->stream;
    FFGPU_CUDA(cudaSetDevice(ctx->device));
    if (M->bs == 1 && is_device_ptr(rowptr) && is_device_ptr(col) && is_device_ptr(val)) {
        const int64_t per = 4 * 256;
        copy_csr_kernel<<<(int)std::min<int64_t>((M->nnz + per - 1) / per + 1, 16 * kNumSM), 256, 0, s>>>(
            M->n + 1, M->nnz, M->browptr, M->bcol, M->val, rowptr, col, val);
        FFGPU_TRY(launch_check(ctx, "copy_csr"));
        FFGPU_CUDA(cudaStreamSynchronize(s));
        return FFGPU_OK;
    }
    if (M->bs == 1) {
        // stored as exported: copied to the caller's arrays, host or device
        FFGPU_CUDA(cudaMemcpyAsync(rowptr, M->browptr, sizeof(int32_t) * ((size_t)M->n + 1), cudaMemcpyDefault, s));
        FFGPU_CUDA(cudaMemcpyAsync(col, M->bcol, sizeof(int32_t) * M->nnz, cudaMemcpyDefault, s));
        FFGPU_CUDA(cudaMemcpyAsync(val, M->val, sizeof(double) * M->nnz, cudaMemcpyDefault, s));
        FFGPU_CUDA(cudaStreamSynchronize(s));
        return FFGPU_OK;
    }
    DevOut<int32_t> rp(rowptr, M->n + 1, ctx, false);
    DevOut<int32_t> cl(col, M->nnz, ctx, false);
    DevOut<double> vl(val, M->nnz, ctx, false);
    FFGPU_TRY(rp.err); FFGPU_TRY(cl.err); FFGPU_TRY(vl.err);
    export_bsr3_kernel<<<grid_for((int64_t)M->nb * 32, 256), 256, 0, s>>>(M->nb, M->browptr, M->bcol, M->val, rp.d, cl.d,
                                                                       vl.d);
    FFGPU_TRY(launch_check(ctx, "export_bsr3"));
    FFGPU_TRY(rp.finish()); FFGPU_TRY(cl.finish()); FFGPU_TRY(vl.finish());
    FFGPU_CUDA(cudaStreamSynchronize(s));
    return FFGPU_OK;
}

}  // extern "C"
