// ffgpu_gmres.cu -- FreeFEM's right-preconditioned FGMRES (CG.cpp:348-517, driven by
// SolverGMRES::dosolver, VirtualSolverCG.hpp:195-257) on the device.
//
// FreeFEM's Arnoldi step orthogonalises w = A C v_it against v_0..v_it by modified Gram-Schmidt:
//   for i = 0..it: H(i,it) = (w, v_i); w -= H(i,it) v_i
// i.e. 2(it+1) dependent passes over n-vectors.  Here the same coefficients come from ONE pass:
// with s_i = (w_0, v_i) (the unmodified w) and the Gram entries G(i,j) = (v_i, v_j), j < i,
// modified Gram-Schmidt's coefficients are the solution of the unit lower-triangular system
//   h_i = s_i - sum_{j<i} h_j G(i,j)
// (low-synchronisation MGS, Swirydowicz, Langou, Ananthan, Yang & Thomas, Numer. Linear Algebra
// Appl. 28 (2021)).  The new Gram row G(it, .) = (v_it, v_j) is formed in the same pass as s.
// The recurrence is evaluated to first order in the Gram entries, h = s - L s with L the strictly
// lower Gram triangle: the dropped terms are O(|L|^2 |s|), below the rounding of s itself while
// the basis is orthonormal to working accuracy, and the coefficients then come from a parallel
// matrix-vector product instead of a sequential substitution (GB300 runs ~2 FP64 FMAs per clock
// per SM: O(it^2) sequential work in one block cost more than the whole step at it ~ 500).
// One Arnoldi step is five kernels, none with a host round trip:
//   gm_prep    v_it *= 1/||w_prev|| (FreeFEM's Vi[it] = (1/aux) w), vp = C v_it (Jacobi)
//   SpMV       w = A vp
//   gm_dots    s = V' w and the Gram row in one pass over V: blocks are (slab of the vectors'
//              elements) x (group of basis vectors), w and v_it of a slab staged in shared
//              memory, one warp reduction per pair of sums and sub-tile, the last block of a group
//              sums its slabs; one more block finishes step it - 1: the new rotation, Q's two
//              changed rows, the residual estimate |g_it|, FreeFEM's stopping tests
//   gm_coef    h = s - L s (a warp per row, all SMs)
//   gm_update  v_{it+1} = w - V h, ||v_{it+1}||^2 by blocks, and the earlier rotations applied to h
//              as u = Q h with their product Q (a warp per row)
// and the Arnoldi loop of one restart cycle is a CUDA-graph `while` node.  The host reads the
// scalars once per restart cycle.  All reductions sum in a fixed order (warp order inside a
// block, block order across blocks), so results are reproducible run to run.
//
// No kernel ends with one block that works alone: gm_dots ends with one per vector group, the norm
// is summed where it is read, and the rotation (a chain of square roots and divisions) runs beside
// the next step's dot products, at the price of that step's first three kernels once per solve,
// when it says stop.  The last step of a full cycle is finished by the back substitution's block, so that a
// short restart pays for no step of its own (90 x 90 cells, 400 steps, dim_krylov 1: 29.5 -> 25.8 ms, with last
// blocks 26.2; dim_krylov 3: 16.4 -> 15.0, 18.8).  (9282 rows, 381 steps: 16.7 ms with last blocks in gm_dots and gm_update,
// 14.3 ms now; the FP64 products alone are 3.4 ms, the rest is latency inside the five kernels).
// Sums of gm_dots' slabs by every block of gm_coef instead: 16.2 ms.
// A rotation after the other (FreeFEM's loop) is a chain of 2 it dependent FP64 operations, 64 to
// 76 cycles each on GB300: 14 us at it = 190.  The product Q costs it^2 multiplications over all SMs.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "ffgpu_gridsync.cuh"
#include "ffgpu_sell.cuh"

namespace ffgpu {

constexpr int kGmThreads = 256;
constexpr int kGmWarps = kGmThreads / 32;
constexpr int kGmSub = 512;                  // elements of w and v_it staged per sub-tile of gm_dots
constexpr int kGmMaxSlabs = 32;              // slabs of gm_dots (partials summed by its last block)
constexpr int kGmBack = 512;                 // threads of the back substitution
constexpr int kGmHs = 1024;                  // Hessenberg columns up to this length stay in shared memory

struct GmScal {
    double normb, relres, eps;
    int it, iter, itmax, m, conv, stop, steps, itf;
    int next;                                // the step of gm_prep and gm_dots (gm_coef sets it; `it` is gm_coef's and gm_update's)
    unsigned ticket;
};

struct GmArgs {
    int n, m;
    int64_t vs;
    int nslab, ngrp;                         // gm_dots grid: nslab x ngrp blocks
    int64_t slab_len;                        // elements per slab (a multiple of kGmSub)
    double *V, *Vp, *vpc, *w, *x;
    const double *b, *dinv;
    const uint8_t *wcl;
    int use_wcl;
    int rows;                                // rows of a block of gm_update / gm_xupd
    int nupd;                                // blocks of gm_update (parts of nrm)
    int *tick;                               // gm_dots: blocks of a vector group that are done
    double *R, *Q, *u, *g, *y, *Gm, *h, *red, *part, *nrm;   // R: column it of the triangle at it * (m + 1)
    GmScal *sc;
    cudaGraphConditionalHandle cond;
    int in_graph;
};

__device__ __noinline__ void gm_set_cond(cudaGraphConditionalHandle c, unsigned v) { cudaGraphSetConditional(c, v); }

// Last-block protocol for a vector of K partial sums per block: part[k * gridDim.x + block].
// Returns true in the last block to finish (all its threads), after red[k] = sum over blocks in
// block order (one warp per k, lanes striding the blocks, fixed shuffle tree).
__device__ bool gm_last_block(const double *mine, int K, double *part, double *red, unsigned *ticket) {
    __shared__ bool s_last;
    for (int k = threadIdx.x; k < K; k += blockDim.x) part[(int64_t)k * gridDim.x + blockIdx.x] = mine[k];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return false;
    __threadfence();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = warp; k < K; k += blockDim.x >> 5) {
        double s = 0;
        for (int b = lane; b < (int)gridDim.x; b += 32) s += __ldcg(part + (int64_t)k * gridDim.x + b);
        s = warp_sum(s);
        if (lane == 0) red[k] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) *ticket = 0u;
    return true;
}

// block sum of one value per thread into sh[0] (sh: kGmWarps doubles + 1)
__device__ double gm_block_sum(double v, double *sh) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    v = warp_sum(v);
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int w = 0; w < kGmWarps; ++w) t += sh[w];
        sh[kGmWarps] = t;
    }
    __syncthreads();
    return sh[kGmWarps];
}

// ||b||, the tgv rows left out (FreeFEM zeroes them in wi before mysnrm2); initialises the scalars
__global__ void __launch_bounds__(kGmThreads) gm_init(GmArgs a, double eps, int itmax) {
    __shared__ double sh[kGmWarps + 1];
    double s = 0;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < a.n; k += (int64_t)gridDim.x * blockDim.x) {
        const double v = (a.use_wcl && a.wcl[k]) ? 0.0 : a.b[k];
        s = fma(v, v, s);
    }
    const double t = gm_block_sum(s, sh);
    if (gm_last_block(&t, 1, a.part, a.red, &a.sc->ticket) && threadIdx.x == 0) {
        GmScal *c = a.sc;
        c->normb = sqrt(a.red[0]);
        c->relres = 1e100;
        c->eps = eps;
        c->iter = 0;
        c->itmax = itmax;
        c->m = a.m;
        c->conv = 0;
        c->steps = 0;
    }
}

// start of a restart cycle: V[0] holds A x; r = -(A x - b) into V[0], g[0] = ||r||
__global__ void __launch_bounds__(kGmThreads) gm_resid(GmArgs a) {
    __shared__ double sh[kGmWarps + 1];
    double s = 0;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < a.n; k += (int64_t)gridDim.x * blockDim.x) {
        const double r = -(a.V[k] - a.b[k]);
        a.V[k] = r;
        s = fma(r, r, s);
    }
    const double t = gm_block_sum(s, sh);
    if (gm_last_block(&t, 1, a.part, a.red, &a.sc->ticket) && threadIdx.x == 0) {
        GmScal *c = a.sc;
        const double g0 = sqrt(a.red[0]);
        a.g[0] = g0;
        a.Q[0] = 1.0;
        if (c->normb < 1.e-20 || c->eps < 0) c->normb = 1.;
        c->it = 0;
        c->next = 0;
        c->stop = 0;
        // an exact initial guess: FreeFEM would divide by zero here; the solve is converged
        if (g0 == 0.0) {
            c->conv = 1;
            c->stop = 1;
            c->relres = 0.0;
            c->itf = -1;
            if (a.in_graph) gm_set_cond(a.cond, 0);
        }
    }
}

// ||v_it||^2 before its scaling, in every thread of the block (kGmThreads or more): the sum of gm_update's
// parts (at most 4 * kNumSM of them)
__device__ __forceinline__ double gm_norm2(const GmArgs &a) {
    __shared__ double sh[kGmWarps];
    static_assert(4 * kNumSM <= 3 * kGmThreads && kGmWarps == 8, "parts per thread");
    double v[3];
#pragma unroll
    for (int u = 0; u < 3; ++u) {
        const int b = threadIdx.x + u * kGmThreads;
        v[u] = b < a.nupd && threadIdx.x < kGmThreads ? __ldcg(a.nrm + b) : 0.0;
    }
    double t = warp_sum((v[0] + v[1]) + v[2]);
    if ((threadIdx.x & 31) == 0 && threadIdx.x < kGmThreads) sh[threadIdx.x >> 5] = t;
    __syncthreads();
    t = sh[threadIdx.x & 7];
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// v_it *= 1/||.|| (FreeFEM: Vi[it] = (1./aux)*wi), vp = C v_it into Vp[it] and the SpMV input
__global__ void __launch_bounds__(kGmThreads) gm_prep(GmArgs a) {
    const int it = a.sc->next;
    double *v = a.V + it * a.vs, *vp = a.Vp + it * a.vs;
    const double inv = it == 0 ? 1. / a.g[0] : 1. / sqrt(gm_norm2(a));
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < a.n; k += (int64_t)gridDim.x * blockDim.x) {
        const double vk = inv * v[k];
        v[k] = vk;
        const double p = a.dinv[k] * vk;
        vp[k] = p;
        a.vpc[k] = p;
    }
}

// the end of step it: the new rotation, the triangle's column, Q, the stopping tests (one block; in_loop: of
// a kernel inside the while node)
__device__ void gm_finish(const GmArgs &a, int it, bool in_loop) {
    __shared__ double rot[2];
    const int ld = a.m + 1;
    GmScal *c = a.sc;
    // what the chain below reads is under way during the norm's sum
    const double hd = a.u[it], g0 = a.g[it], normb = c->normb, eps = c->eps;
    const int itmax = c->itmax, iter = c->iter, steps = c->steps;
    const double aux = sqrt(gm_norm2(a));
    if (threadIdx.x == 0) {
        const double hs1 = aux;
        const double sq = sqrt(hd * hd + hs1 * hs1);
        const double c0 = hd / sq, s0 = hs1 / sq;
        rot[0] = c0;
        rot[1] = s0;
        a.R[(int64_t)it * ld + it] = c0 * hd + s0 * hs1;
        a.g[it + 1] = -s0 * g0;
        a.g[it] = c0 * g0;
        const double relres = fabs(-s0 * g0);
        c->relres = relres;
        c->steps = steps + 1;
        c->itf = it;
        bool stop = false;
        if (relres / normb < fabs(eps)) {
            c->conv = 1;
            stop = true;
        } else if (it > itmax) {
            stop = true;                       // FreeFEM: `if (it > nbitermx) break;`
        } else {
            c->it = it + 1;                    // the loop increment it++, iter++
            c->iter = iter + 1;
            if (it + 1 >= a.m) { stop = true; c->itf = a.m - 1; }
        }
        c->stop = stop;
        if (stop && a.in_graph && in_loop) gm_set_cond(a.cond, 0);
    }
    __syncthreads();
    // the column of the triangle, and Q with the new rotation of its rows it and it + 1
    double *q0 = a.Q + (int64_t)it * (ld + 1), *q1 = q0 + ld + 1;
    for (int i = threadIdx.x; i <= it + 1; i += blockDim.x) {
        if (i < it) a.R[(int64_t)it * ld + i] = a.u[i];
        if (!in_loop) continue;   // no step comes after
        const double q = i <= it ? q0[i] : 0.0;
        q0[i] = i <= it ? rot[0] * q : rot[1];
        q1[i] = i <= it ? -rot[1] * q : rot[0];
    }
}

// s_i = (w, v_i), i <= it, and the Gram row (v_it, v_j), j < it, in one pass over V.
// Block (slab, group): the elements [slab * slab_len, +slab_len) of the vectors i = group +
// ngrp * r; per sub-tile of kGmSub elements w and v_it are staged in shared memory and each warp
// runs its vectors over the sub-tile (16 elements per lane, then one warp reduction for both sums).
// A vector's elements are loaded before the products of the one before it (the first vector's
// before the staging).
// Partials part[(2 i + c) * nslab + slab]: c = 0 for s, 1 for the Gram row; the last block of a
// vector group sums them in slab order (a half warp per sum).
__global__ void __launch_bounds__(kGmThreads) gm_dots(GmArgs a) {
    extern __shared__ __align__(16) double smd[];
    double *wsh = smd, *vsh = smd + kGmSub, *acc = smd + 2 * kGmSub;
    const int it = a.sc->next;
    if (blockIdx.x == 0) {
        if (it > 0) gm_finish(a, it - 1, true);
        return;
    }
    const int ni = it + 1, K = 2 * ni;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int blk = blockIdx.x - 1;
    const int slab = blk % a.nslab, grp = blk / a.nslab;
    for (int k = threadIdx.x; k < K; k += blockDim.x) acc[k] = 0;
    const double *vit = a.V + it * a.vs;
    const int64_t e0 = (int64_t)slab * a.slab_len;
    const int64_t e1 = e0 + a.slab_len < a.n ? e0 + a.slab_len : (int64_t)a.n;
    for (int64_t t0 = e0; t0 < e1; t0 += kGmSub) {
        const int len = e1 - t0 < kGmSub ? (int)(e1 - t0) : kGmSub;
        const int len2 = len & ~1;   // pairs of elements as 16-byte loads; an odd last element apart
        constexpr int NP = kGmSub / 64;
        int i = grp + a.ngrp * warp;
        double2 q[NP], nx[NP];
        const auto load = [&](double2 *d, int iv) {
            const double *vi = a.V + iv * a.vs + t0;   // 16-byte aligned: vs and t0 are even
#pragma unroll
            for (int u = 0; u < NP; ++u)
                if (2 * lane + 64 * u < len2) d[u] = __ldcs(reinterpret_cast<const double2 *>(vi + 2 * lane + 64 * u));
        };
        if (i < ni) load(q, i);
        __syncthreads();   // the previous sub-tile's readers are done (and acc is zeroed)
        for (int e = threadIdx.x; e < len; e += blockDim.x) {
            wsh[e] = a.w[t0 + e];
            vsh[e] = vit[t0 + e];
        }
        __syncthreads();
        while (i < ni) {
            const int in = i + a.ngrp * kGmWarps;
            if (in < ni) load(nx, in);
            double ts = 0, tl = 0;
#pragma unroll
            for (int u = 0; u < NP; ++u) {
                const int e = 2 * lane + 64 * u;
                if (e < len2) {
                    const double2 w2 = *reinterpret_cast<const double2 *>(wsh + e);
                    const double2 v2 = *reinterpret_cast<const double2 *>(vsh + e);
                    ts = fma(q[u].x, w2.x, ts);
                    tl = fma(q[u].x, v2.x, tl);
                    ts = fma(q[u].y, w2.y, ts);
                    tl = fma(q[u].y, v2.y, tl);
                }
            }
            if (len2 < len && lane == 0) {
                const double qo = __ldcs(a.V + i * a.vs + t0 + len2);
                ts = fma(qo, wsh[len2], ts);
                tl = fma(qo, vsh[len2], tl);
            }
            const double p = warp_sum_pair(ts, tl);   // vector i belongs to this warp
            if ((lane & 15) == 0) acc[lane ? ni + i : i] += p;
#pragma unroll
            for (int u = 0; u < NP; ++u) q[u] = nx[u];
            i = in;
        }
    }
    __syncwarp();   // a warp reads back its own vectors' sums
    for (int i = grp + a.ngrp * warp; i < ni; i += a.ngrp * kGmWarps)
        if (lane < 2) a.part[(2 * (int64_t)i + lane) * a.nslab + slab] = acc[lane * ni + i];
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(a.tick + grp, 1) == a.nslab - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    static_assert(kGmMaxSlabs == 32, "two slabs per lane of a half warp");
    const int l16 = lane & 15, c = lane >> 4;
    for (int i = grp + a.ngrp * warp; i < ni; i += a.ngrp * kGmWarps) {
        const double *p = a.part + (2 * (int64_t)i + c) * a.nslab;
        double t = l16 < a.nslab ? __ldcg(p + l16) : 0.0;
        if (l16 + 16 < a.nslab) t += __ldcg(p + l16 + 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) a.red[i] = t;                                        // s
        if (lane == 16 && i < it) a.Gm[(int64_t)it * (a.m + 1) + i] = t;   // Gram row of v_it
    }
    if (threadIdx.x == 0) a.tick[grp] = 0;
}

// modified Gram-Schmidt's coefficients of this step to first order in the Gram entries:
// h_i = s_i - sum_{j<i} G(i,j) s_j (a warp per row, rows over the whole grid)
__global__ void __launch_bounds__(kGmThreads) gm_coef(GmArgs a) {
    if (a.sc->stop) return;
    const int it = a.sc->it;
    const int ni = it + 1, ld = a.m + 1;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.sc->next = ni;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = blockIdx.x * kGmWarps + warp; i < ni; i += gridDim.x * kGmWarps) {
        const double *gi = a.Gm + (int64_t)i * ld;
        double t = 0;
#pragma unroll 8
        for (int j = lane; j < i; j += 32) t = fma(__ldcg(gi + j), __ldcg(a.red + j), t);
        t = warp_sum(t);
        if (lane == 0) a.h[i] = __ldcg(a.red + i) - t;
    }
}

// sum_i c_i V_i[k] over the vectors i = grp, grp + ngrp, ... < ni, onto t (negated coefficients where
// SUB): the loads of 16 vectors are issued before their products, and the next 16 before the
// products of these (two batches in flight)
template <bool SUB>
__device__ __forceinline__ double gm_combine(double t, const double *c, const double *V, int64_t vs, int64_t k, int grp,
                                             int ngrp, int ni) {
    const int m = (ni - grp + ngrp - 1) / ngrp;   // vectors of this group
    const double *v = V + (int64_t)grp * vs + k;
    const int64_t step = (int64_t)ngrp * vs;
    const auto mad = [&](int j, double q) {
        const double cj = c[grp + j * ngrp];
        t = fma(SUB ? -cj : cj, q, t);
    };
    int j = 0;
    if (m >= 16) {
        double q[16], r[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) q[u] = __ldcs(v + u * step);
        for (; j + 32 <= m; j += 16) {
#pragma unroll
            for (int u = 0; u < 16; ++u) r[u] = __ldcs(v + (j + 16 + u) * step);
#pragma unroll
            for (int u = 0; u < 16; ++u) mad(j + u, q[u]);
#pragma unroll
            for (int u = 0; u < 16; ++u) q[u] = r[u];
        }
#pragma unroll
        for (int u = 0; u < 16; ++u) mad(j + u, q[u]);
        j += 16;
    }
#pragma unroll 8
    for (; j < m; ++j) mad(j, __ldcs(v + j * step));
    return t;
}

// v_{it+1} = w - sum_i h_i v_i and ||v_{it+1}||^2 by blocks; u = Q h.  A block takes a.rows elements at a time, 256 / rows threads each on a
// part of the vectors, so that small systems use all SMs (n = 9282, it = 190: 37 blocks of one
// thread per element took 53.5 us with the rotations, 8.9 us now).
__global__ void __launch_bounds__(kGmThreads) gm_update(GmArgs a) {
    __shared__ double hs[kGmHs], pt[kGmThreads];
    __shared__ double sh[kGmWarps + 1];
    if (a.sc->stop) return;
    const int it = a.sc->it;
    const int ni = it + 1, ld = a.m + 1;
    // the cycle is full: no step comes after this one (gm_back finishes it)
    if (ni == a.m && a.in_graph && blockIdx.x == 0 && threadIdx.x == 0) gm_set_cond(a.cond, 0);
    const double *hh = a.h;
    if (ni <= kGmHs) {
        for (int i = threadIdx.x; i < ni; i += blockDim.x) hs[i] = a.h[i];
        hh = hs;
    }
    __syncthreads();
    double *vn = a.V + (it + 1) * a.vs;
    const int rows = a.rows, ngrp = kGmThreads / rows, grp = threadIdx.x / rows, r = threadIdx.x - grp * rows;
    double s = 0;
    for (int64_t k0 = (int64_t)blockIdx.x * rows; k0 < a.n; k0 += (int64_t)gridDim.x * rows) {
        const int64_t k = k0 + r;
        double t = 0;
        if (k < a.n) t = gm_combine<true>(grp == 0 ? a.w[k] : 0.0, hh, a.V, a.vs, k, grp, ngrp, ni);
        if (ngrp > 1) {
            __syncthreads();
            pt[threadIdx.x] = t;
            __syncthreads();
            if (grp == 0)
                for (int q = 1; q < ngrp; ++q) t += pt[q * rows + r];
        }
        if (grp == 0 && k < a.n) {
            vn[k] = t;
            s = fma(t, t, s);
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = blockIdx.x * kGmWarps + warp; i < ni; i += gridDim.x * kGmWarps) {
        const double *q = a.Q + (int64_t)i * (ld + 1);
        double t = 0;
        const int len = min(ni, i + 2);   // row i ends at its rotation
        for (int j = lane; j < len; j += 32) t = fma(__ldcg(q + j), hh[j], t);
        t = warp_sum(t);
        if (lane == 0) a.u[i] = t;
    }
    const double tot = gm_block_sum(s, sh);
    if (threadIdx.x == 0) a.nrm[blockIdx.x] = tot;
}

// y = R^-1 g on the it+1 leading rows, column by column: y_i, then g_j -= R(j,i) y_i for all j < i
// at once, with the next column's loads under way (one block; a warp per row's dot product took
// 750 us for 381 rows; the whole solve: 31.2 -> 16.7 ms)
__global__ void __launch_bounds__(kGmBack) gm_back(GmArgs a) {
    extern __shared__ __align__(16) double smb[];
    if (!a.sc->stop) {           // a full cycle
        gm_finish(a, a.m - 1, false);
        __syncthreads();
    }
    const int it = a.sc->itf;
    if (it < 0) return;
    const int ld = a.m + 1, t = threadIdx.x;
    double *gs = smb, *rinv = smb + it + 1;
    for (int i = t; i <= it; i += kGmBack) {
        gs[i] = a.g[i];
        rinv[i] = 1.0 / a.R[(int64_t)i * ld + i];
    }
    double next = t < it ? a.R[(int64_t)it * ld + t] : 0.0;
    __syncthreads();
    for (int i = it; i >= 0; --i) {
        const double *col = a.R + (int64_t)i * ld;
        const double cur = next;
        next = i > 0 && t < i - 1 ? a.R[(int64_t)(i - 1) * ld + t] : 0.0;
        const double yi = gs[i] * rinv[i];
        if (t == 0) a.y[i] = yi;
        if (t < i) gs[t] = fma(-cur, yi, gs[t]);
        for (int j = t + kGmBack; j < i; j += kGmBack) gs[j] = fma(-col[j], yi, gs[j]);
        __syncthreads();
    }
}

// x = (sum_i y_i Vp_i) + x  (FreeFEM: wi = 0; wi += y_i Vpi[i]; uni = wi + x0)
__global__ void __launch_bounds__(kGmThreads) gm_xupd(GmArgs a) {
    __shared__ double pt[kGmThreads];
    const int it = a.sc->itf;
    if (it < 0) return;
    const int rows = a.rows, ngrp = kGmThreads / rows, grp = threadIdx.x / rows, r = threadIdx.x - grp * rows;
    for (int64_t k0 = (int64_t)blockIdx.x * rows; k0 < a.n; k0 += (int64_t)gridDim.x * rows) {
        const int64_t k = k0 + r;
        double t = k < a.n ? gm_combine<false>(0.0, a.y, a.Vp, a.vs, k, grp, ngrp, it + 1) : 0.0;
        if (ngrp > 1) {
            __syncthreads();
            pt[threadIdx.x] = t;
            __syncthreads();
            if (grp == 0)
                for (int q = 1; q < ngrp; ++q) t += pt[q * rows + r];
        }
        if (grp == 0 && k < a.n) a.x[k] = t + a.x[k];
    }
}

__global__ void gm_x0_kernel(int n, double *x, const double *b, const uint8_t *wcl, double tgv) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n && wcl[i]) x[i] = b[i] / tgv;
}

// grids: vector kernels resident and capped by the work; the dot kernel by tiles
static int gm_vec_grid(int64_t n) {
    return (int)std::max<int64_t>(1, std::min<int64_t>(4 * kNumSM, (n + kGmThreads - 1) / kGmThreads));
}
// rows of a block of gm_update: 256 where that gives every SM a block, else fewer (at least a warp)
// with the vectors split over the threads left
static int gm_rows(int64_t n) {
    int rows = kGmThreads;
    while (rows > 32 && (n + rows - 1) / rows < kNumSM) rows >>= 1;
    return rows;
}
// gm_dots: sub-tiles of kGmSub elements grouped into at most kGmMaxSlabs slabs, and enough
// vector groups for about two blocks per SM
static void gm_dot_shape(int64_t n, int &nslab, int &ngrp, int64_t &slab_len) {
    const int64_t nsub = std::max<int64_t>(1, (n + kGmSub - 1) / kGmSub);
    const int64_t per = (nsub + kGmMaxSlabs - 1) / kGmMaxSlabs;
    nslab = (int)((nsub + per - 1) / per);
    slab_len = per * kGmSub;
    // at most two blocks per SM (a block is 8 warps and ~49 KB of shared memory): a third block on
    // some SMs sets the kernel's time while most SMs idle
    ngrp = std::max(1, (2 * kNumSM) / nslab);
}
static int gm_coef_grid(int m) { return std::max(1, std::min(kNumSM, (m + 1 + kGmWarps - 1) / kGmWarps)); }

// one right-hand side; b, x device pointers of length n (x: initial guess, then solution)
int gmres_one(ffgpu_matrix *A, const double *b, double *x, int trans, const ffgpu_solver_params *prm,
              ffgpu_solver_stats *st) {
    ffgpu_ctx *ctx = A->ctx;
    cudaStream_t s = ctx->stream;
    const int n = A->n;
    // FreeFEM's default restart (Data_Sparse_Solver::NbSpace, VirtualSolver.hpp:79)
    const int m = prm->dim_krylov > 0 ? prm->dim_krylov : 1000;
    const int itmax = prm->itmax > 0 ? prm->itmax : n;
    const double tgv = prm->tgv > 0 ? prm->tgv : 1e30;
    const size_t dsmem = sizeof(double) * (2 * (size_t)kGmSub + 2 * (size_t)(m + 1));
    FFGPU_CHECK(sizeof(double) * (4096 + 2 * (size_t)(m + 1)) <= 200 * 1024, FFGPU_EINVAL, "gmres: dim_krylov %d above the supported 10000", m);
    const int64_t vs = vstride(n);
    int nslab = 1, ngrp = 1;
    int64_t slab_len = kGmSub;
    gm_dot_shape(n, nslab, ngrp, slab_len);
    const int rows = gm_rows(n);
    const int Gv = gm_vec_grid(n), Gd = 1 + nslab * ngrp, Gc = gm_coef_grid(m);
    const int Gu = (int)std::max<int64_t>(1, std::min<int64_t>(4 * kNumSM, ((int64_t)n + rows - 1) / rows));
    const size_t bsmem = sizeof(double) * 2 * ((size_t)m + 1);
    // workspace: V (m+1 vectors), Vp (m), the SpMV input and output, the small arrays
    // R, Q, u g y, Gram, h, red, part, nrm, tick, then the scalars (in doubles, rounded up)
    const size_t nscal = (sizeof(GmScal) + sizeof(double) - 1) / sizeof(double);
    const size_t ntick = ((size_t)ngrp + 1) / 2;   // one counter per vector group of gm_dots
    const size_t npart = std::max(2 * (size_t)(m + 1) * nslab, (size_t)Gv);
    const size_t small = (size_t)(m + 2) * (m + 1) + (size_t)(m + 2) * (m + 2) + 3 * (size_t)(m + 2) +
                         (size_t)(m + 1) * (m + 1) + (size_t)(m + 2) + 2 * (size_t)(m + 1) + npart + (size_t)Gu + ntick + nscal;
    double *ws = nullptr;
    const size_t nvec = (size_t)(2 * m + 3);
    FFGPU_CUDA(dalloc(ctx, (void **)&ws, sizeof(double) * (nvec * vs + small)));
    GmArgs a;
    memset(&a, 0, sizeof(a));
    a.n = n; a.m = m; a.vs = vs;
    a.nslab = nslab; a.ngrp = ngrp; a.slab_len = slab_len;
    a.V = ws; a.Vp = ws + (size_t)(m + 1) * vs; a.vpc = a.Vp + (size_t)m * vs; a.w = a.vpc + vs;
    double *sm = a.w + vs;
    a.rows = rows;
    a.nupd = Gu;
    a.R = sm; sm += (size_t)(m + 2) * (m + 1);
    a.Q = sm; sm += (size_t)(m + 2) * (m + 2);
    a.u = sm; sm += m + 2;
    a.g = sm; sm += m + 2;
    a.y = sm; sm += m + 2;
    a.Gm = sm; sm += (size_t)(m + 1) * (m + 1);
    a.h = sm; sm += m + 2;
    a.red = sm; sm += 2 * (m + 1);
    a.part = sm; sm += npart;
    a.nrm = sm; sm += Gu;
    a.tick = reinterpret_cast<int *>(sm); sm += ntick;
    a.sc = reinterpret_cast<GmScal *>(sm);
    sm += nscal;
    if ((size_t)(sm - ws) != nvec * vs + small) {
        dfree(ctx, ws);
        FFGPU_CHECK(false, FFGPU_EINVAL, "gmres: workspace layout mismatch");
    }
    a.x = x; a.b = b; a.dinv = A->diag_inv; a.wcl = A->wcl; a.use_wcl = A->ntgv > 0;
    FFGPU_CUDA(cudaMemsetAsync(a.sc, 0, sizeof(GmScal), s));
    FFGPU_CUDA(cudaMemsetAsync(a.tick, 0, sizeof(int) * ngrp, s));
    FFGPU_CUDA(cudaFuncSetAttribute((const void *)gm_dots, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dsmem));
    FFGPU_CUDA(cudaFuncSetAttribute((const void *)gm_back, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsmem));
    int rc = FFGPU_OK;
    cudaGraphExec_t exec = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    if (A->ntgv > 0) {
        gm_x0_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, x, b, A->wcl, tgv);   // SetInitWithBC
        rc = launch_check(ctx, "gmres x0");
    }
    if (!rc) {
        gm_init<<<Gv, kGmThreads, 0, s>>>(a, prm->eps, itmax);
        rc = launch_check(ctx, "gmres init");
    }
    // the SpMV's launch data (SELL partition) are set up by this first call, before the capture
    if (!rc) rc = spmv(A, a.vpc, a.w, trans, s);
    const bool host_loop = getenv("FFGPU_CG_GRAPH") && getenv("FFGPU_CG_GRAPH")[0] == '0';
    if (!rc && !host_loop) {
        // graph of one restart cycle: [A x -> V0, residual, while(!stop){prep, SpMV, dots, coef, update},
        // back substitution, x update]
        cudaGraph_t graph = nullptr;
        cudaGraphConditionalHandle cond;
        cudaError_t e = cudaGraphCreate(&graph, 0);
        if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&cond, graph, 1, cudaGraphCondAssignDefault);
        GmArgs ag = a;
        ag.cond = cond;
        ag.in_graph = 1;
        cudaGraphNode_t pre_last = nullptr, wnode = nullptr;
        cudaGraph_t body = nullptr;
        // prologue: captured into the parent graph
        if (e == cudaSuccess) e = cudaStreamBeginCaptureToGraph(s, graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            int r2 = spmv(A, x, a.V, trans, s);
            gm_resid<<<Gv, kGmThreads, 0, s>>>(ag);
            cudaError_t ec = cudaStreamEndCapture(s, &graph);
            if (r2 || ec != cudaSuccess) e = ec != cudaSuccess ? ec : cudaErrorUnknown;
        }
        // the while node after the prologue's last node
        if (e == cudaSuccess) {
            size_t nn = 0;
            e = cudaGraphGetNodes(graph, nullptr, &nn);
            std::vector<cudaGraphNode_t> nodes(nn);
            if (e == cudaSuccess) e = cudaGraphGetNodes(graph, nodes.data(), &nn);
            // the prologue is a chain; its sink is the node with no dependents
            for (size_t i = 0; e == cudaSuccess && i < nn; ++i) {
                size_t nd = 0;
                e = cudaGraphNodeGetDependentNodes(nodes[i], nullptr, nullptr, &nd);
                if (e == cudaSuccess && nd == 0) pre_last = nodes[i];
            }
            alignas(cudaGraphNodeParams) unsigned char cp_buf[sizeof(cudaGraphNodeParams)];
            memset(cp_buf, 0, sizeof(cp_buf));
            cudaGraphNodeParams *cp = reinterpret_cast<cudaGraphNodeParams *>(cp_buf);
            cp->type = cudaGraphNodeTypeConditional;
            cp->conditional.handle = cond;
            cp->conditional.type = cudaGraphCondTypeWhile;
            cp->conditional.size = 1;
            if (e == cudaSuccess) e = cudaGraphAddNode(&wnode, graph, &pre_last, nullptr, 1, cp);
            if (e == cudaSuccess) body = cp->conditional.phGraph_out[0];
        }
        if (e == cudaSuccess) e = cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            gm_prep<<<Gv, kGmThreads, 0, s>>>(ag);
            int r2 = spmv(A, a.vpc, a.w, trans, s);
            gm_dots<<<Gd, kGmThreads, dsmem, s>>>(ag);
            gm_coef<<<Gc, kGmThreads, 0, s>>>(ag);
            gm_update<<<Gu, kGmThreads, 0, s>>>(ag);
            cudaError_t ec = cudaStreamEndCapture(s, &body);
            if (r2 || ec != cudaSuccess) e = ec != cudaSuccess ? ec : cudaErrorUnknown;
        }
        if (e == cudaSuccess) e = cudaStreamBeginCaptureToGraph(s, graph, &wnode, nullptr, 1, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            gm_back<<<1, kGmBack, bsmem, s>>>(ag);
            gm_xupd<<<Gu, kGmThreads, 0, s>>>(ag);
            e = cudaStreamEndCapture(s, &graph);
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
        if (graph) cudaGraphDestroy(graph);
        if (e != cudaSuccess) {
            set_error("gmres graph: %s", cudaGetErrorString(e));
            cudaGetLastError();
            rc = FFGPU_ECUDA;
        }
    }
    GmScal hs;
    memset(&hs, 0, sizeof(hs));
    int cycles = 0;
    int64_t steps_seen = 0;
    while (!rc) {
        if (host_loop) {
            // the same kernels launched from the host, for profilers that do not trace conditional
            // graph nodes; the stop flag is read after every Arnoldi step
            if ((rc = spmv(A, x, a.V, trans, s))) break;
            gm_resid<<<Gv, kGmThreads, 0, s>>>(a);
            for (;;) {
                if ((rc = launch_check(ctx, "gmres resid"))) break;
                FFGPU_CUDA(cudaMemcpyAsync(&hs, a.sc, sizeof(hs), cudaMemcpyDeviceToHost, s));
                FFGPU_CUDA(cudaStreamSynchronize(s));
                if (hs.stop || hs.next >= m) break;
                gm_prep<<<Gv, kGmThreads, 0, s>>>(a);
                if ((rc = spmv(A, a.vpc, a.w, trans, s))) break;
                gm_dots<<<Gd, kGmThreads, dsmem, s>>>(a);   // may say stop: the two kernels below then return
                gm_coef<<<Gc, kGmThreads, 0, s>>>(a);
                gm_update<<<Gu, kGmThreads, 0, s>>>(a);
                ctx->launches += 4;
            }
            if (rc) break;
            gm_back<<<1, kGmBack, bsmem, s>>>(a);
            gm_xupd<<<Gu, kGmThreads, 0, s>>>(a);
            ctx->launches += 2;
        } else {
            FFGPU_CUDA(cudaGraphLaunch(exec, s));
        }
        FFGPU_CUDA(cudaMemcpyAsync(&hs, a.sc, sizeof(hs), cudaMemcpyDeviceToHost, s));
        cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            set_error("gmres: %s", cudaGetErrorString(e));
            rc = FFGPU_ECUDA;
            break;
        }
        ++cycles;
        // a stop inside the cycle is found in the step after it
        const int64_t steps = hs.steps - steps_seen;
        if (!host_loop) ctx->launches += 4 + 5 * (steps >= m || hs.itf < 0 ? steps : steps + 1);
        steps_seen = hs.steps;
        if (hs.conv) break;
        if (hs.iter > itmax) break;
    }
    cudaEventRecord(e1, s);
    cudaStreamSynchronize(s);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (exec) cudaGraphExecDestroy(exec);
    dfree(ctx, ws);
    cudaStreamSynchronize(s);
    if (rc) return rc;
    if (getenv("FFGPU_VERBOSE"))
        fprintf(stderr, "ffgpu: fgmres %d iterations, %d restart cycles, relative residual %.3e\n", hs.iter, cycles,
                hs.relres / hs.normb);
    if (st) {
        st->iterations = hs.iter;
        st->converged = hs.conv != 0;
        st->residual = hs.relres / hs.normb;
        st->elapsed_ms += ms;
    }
    return hs.conv ? FFGPU_OK : FFGPU_ENOCONV;
}

}  // namespace ffgpu
