// ffgpu_persist.cu -- the CG loop of ffgpu_solve_cg inside one cooperative kernel.
//
// FreeFEM's ConjugueGradient (src/femlib/CG.cpp:196-265) as ffgpu_solve.cu describes it, in two
// forms.  cg_loop, further down, streams the matrix.  cg_band is for scalar systems whose rows
// touch a narrow range of columns (2D meshes, small 3D ones).  One block per SM owns
// consecutive rows for the whole solve:
//   * its rows of the matrix in shared memory (values FP64, columns as 16-bit numbers relative
//     to the first column the block touches), x, g and 1/A_ii in registers;
//   * per iteration it forms the direction h' = gamma h - C g once for every column it touches
//     (its own rows and the halo), from the h and C g the owners left in L2, multiplies from
//     shared memory, and takes part in two exchanges (ffgpu_gridsync.cuh): (g,h'), (h',A h')
//     and (g, C g).
// So nothing of the matrix moves after the start, and an iteration is two trips through L2.
// The launches of the two-kernel loop spend an iteration on kernel boundaries, a chain of
// dependent L2 reads and FP64 reductions over many more warps than the sums need.
#include <stdlib.h>
#include <string.h>

#include <algorithm>

#include "ffgpu_gridsync.cuh"
#include "ffgpu_sell.cuh"

namespace ffgpu {

struct BandArgs {
    int n, rows;                 // rows per block
    const int32_t *rp, *col;
    const double *val, *dinv;
    double *x, *g, *h0, *h1, *cg;
    KrylovScalars *ks;
    GridSync gs;
    int range_cap;               // doubles of the staged direction
};

// What a block needs: the column range of its rows and the slots of its row groups (32 rows
// padded to the longest).  need[0]: widest range, need[1]: most slots (both over the blocks).
__global__ void __launch_bounds__(128) band_need_kernel(int n, int rows, const int32_t *__restrict__ rp,
                                                        const int32_t *__restrict__ col, int *need) {
    __shared__ int lo, hi, slots;
    if (threadIdx.x == 0) { lo = 0x7fffffff; hi = -1; slots = 0; }
    __syncthreads();
    const int r0 = blockIdx.x * rows, r1 = min(n, r0 + rows);
    for (int base = r0; base < r1; base += blockDim.x) {
        const int r = base + threadIdx.x;
        int L = 0;
        if (r < r1) {
            const int b = rp[r], e = rp[r + 1];
            L = e - b;
            int cl = r, ch = r;   // the row itself is staged too
            for (int k = b; k < e; ++k) { cl = min(cl, col[k]); ch = max(ch, col[k]); }
            atomicMin(&lo, cl);
            atomicMax(&hi, ch);
        }
        L = __reduce_max_sync(0xffffffffu, L);
        if ((threadIdx.x & 31) == 0) atomicAdd(&slots, L);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(need, hi - lo + 1);
        atomicMax(need + 1, slots);
    }
}

// RPT rows per thread, NT threads.  Row r0 + u * NT + t belongs to thread t.
// FP64 instructions set the floor (one per 64 cycles and sub-partition): about 16 per group of
// 32 rows and iteration on a 2D P1 mesh.
template <int NT, int RPT>
__global__ void __launch_bounds__(NT, 1) cg_band(BandArgs A) {
    constexpr int NW = NT / 32;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[kGsRed<NW>];
    __shared__ int s_lo, s_hi, s_base[RPT * NW + 1];
    if (A.ks->done) return;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int r0 = blockIdx.x * A.rows, r1 = min(A.n, r0 + A.rows);
    double *hs = reinterpret_cast<double *>(smraw);
    if (t == 0) { s_lo = 0x7fffffff; s_hi = -1; }
    __syncthreads();
    double x[RPT], g[RPT], z[RPT], d[RPT];
    int len[RPT];
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
        const int r = r0 + u * NT + t;
        const bool own = r < r1;
        int L = 0;
        x[u] = g[u] = z[u] = d[u] = 0.0;
        if (own) {
            const int b = A.rp[r], e = A.rp[r + 1];
            L = e - b;
            int cl = r, ch = r;
            for (int k = b; k < e; ++k) { cl = min(cl, A.col[k]); ch = max(ch, A.col[k]); }
            atomicMin(&s_lo, cl);
            atomicMax(&s_hi, ch);
            x[u] = A.x[r]; g[u] = A.g[r]; d[u] = A.dinv[r];
        }
        len[u] = __reduce_max_sync(0xffffffffu, L);
        if (lane == 0) s_base[u * NW + w] = len[u];
    }
    __syncthreads();
    if (t == 0) {
        int s = 0;
        for (int i = 0; i < RPT * NW; ++i) { const int L = s_base[i]; s_base[i] = s; s += L; }
        s_base[RPT * NW] = s;
    }
    __syncthreads();
    const int lo = s_lo, nc = s_hi - lo + 1;
    double *mv = hs + A.range_cap;
    uint16_t *mc = reinterpret_cast<uint16_t *>(mv + (size_t)s_base[RPT * NW] * 32);
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
        const int r = r0 + u * NT + t;
        const int b = r < r1 ? A.rp[r] : 0, L = r < r1 ? A.rp[r + 1] - b : 0;
        const int base = s_base[u * NW + w] * 32 + lane;
        for (int j = 0; j < len[u]; ++j) {
            mv[base + 32 * j] = j < L ? A.val[b + j] : 0.0;
            mc[base + 32 * j] = (uint16_t)(j < L ? A.col[b + j] - lo : 0);
        }
    }
    const double eps2 = A.ks->eps2;
    const int itmax = A.ks->itmax;
    double gcg = A.ks->gcg, gcgp = gcg, gamma = 1.0, rho = 0.0, sgh = 0.0, shq = 0.0;
    int iter = 0, conv = 0, k = 0;
    bool good = true;
    const double *hold = A.h0;
    double *hnew = A.h1;
    for (;;) {
        // ---- the direction on every column the block touches (the loads of four in flight)
        for (int c0 = t; c0 < nc; c0 += 4 * NT) {
            double hv[4], cv[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int c = c0 + q * NT;
                hv[q] = c < nc ? __ldcg(hold + lo + c) : 0.0;
                cv[q] = c < nc && iter ? __ldcg(A.cg + lo + c) : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int c = c0 + q * NT;
                if (c < nc) hs[c] = fma(gamma, hv[q], -cv[q]);
            }
        }
        __syncthreads();
        // ---- q = A h' from shared memory, the rows' products side by side
        double y[RPT], ho[RPT];
        double pa = 0.0, pb = 0.0;
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
            const int r = r0 + u * NT + t;
            const int base = s_base[u * NW + w] * 32 + lane;
            double s = 0.0;
#pragma unroll 4
            for (int j = 0; j < len[u]; ++j) s = fma(mv[base + 32 * j], hs[mc[base + 32 * j]], s);
            y[u] = s;
            ho[u] = 0.0;
            if (u * NT < A.rows) {               // uniform: groups past the rows do no FP64 work
                ho[u] = r < r1 ? hs[r - lo] : 0.0;
                if (r < r1) __stcg(hnew + r, ho[u]);
                pa = fma(g[u], ho[u], pa);
                pb = fma(ho[u], y[u], pb);
            }
        }
        if (!gs_sum2<NW, false>(A.gs, k++, pa, pb, red)) { good = false; break; }
        sgh = pa;
        shq = pb;
        rho = -pa / pb;
        // ---- x += rho h', g += rho q, C g
        double pc = 0.0, none = 0.0;
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
            if (u * NT < A.rows) {
                const int r = r0 + u * NT + t;
                x[u] = fma(rho, ho[u], x[u]);
                g[u] = fma(rho, y[u], g[u]);
                z[u] = __dmul_rn(d[u], g[u]);
                if (r < r1) __stcg(A.cg + r, z[u]);
                pc = fma(g[u], z[u], pc);
            }
        }
        if (!gs_sum2<NW, true>(A.gs, k++, pc, none, red)) { good = false; break; }
        gcgp = gcg;
        gcg = pc;
        gamma = gcg / gcgp;
        ++iter;
        conv = gcg < eps2;
        if (conv || iter >= itmax) break;
        double *const swap = const_cast<double *>(hold);
        hold = hnew;
        hnew = swap;
    }
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
        const int r = r0 + u * NT + t;
        if (r < r1) A.x[r] = x[u];
    }
    if (blockIdx.x == 0 && t == 0) {
        KrylovScalars *ks = A.ks;
        ks->gcg = gcg; ks->gcgp = gcgp; ks->gamma = gamma; ks->rho = rho; ks->s_gh = sgh; ks->s_hq = shq;
        ks->iter = iter;
        ks->converged = conv;
        ks->done = good ? 1 : 2;
    }
}

// ------------------------------------------------------------------ larger scalar systems
// The same loop for matrices that stream from L2 or HBM: one block of 32 warps per SM, the SELL-32
// copy in its stride assignment with the batched row loop, three exchanges per iteration --
//   q = A h, (h,q)              [q visible]      rho
//   x += rho h, g += rho q, z = C g, (g,z)       gamma, FreeFEM's stopping test
//   h = gamma h - z, (g,h)      [h visible]
// -- on vectors each block owns a contiguous piece of; the pieces of g and z stay in shared memory.
// Against the three launches per iteration it saves their starts, tails and last-block sums.
// Per iteration, launches and loop: P1 on 60^3 cells 31.2 and 29.2 us, 90^3 60.2 and 50.2, 120^3 105.9
// and 98.4 (102 with g and z in L2); on 140^3, where two pieces no longer fit, 152 and 153; P2 on 24 x
// 23 x 22 40.9 and 33.9; P1 on 700^2 39.3 and 34.3.  3x3 blocks (24^3 cells: 90.3 and 91.4) and
// double-float products (17 x 16 x 15: 39.3 and 49.9) are no faster and keep the launches.
struct LoopArgs {
    int n, per;                  // elements of a block, even
    SellArgs S;
    const double *val, *dinv;
    double *x, *g, *h, *q, *z;
    KrylovScalars *ks;
    GridSync gs;
};

template <bool C16>
__global__ void __launch_bounds__(1024, 1) cg_loop(LoopArgs A) {
    extern __shared__ __align__(16) double smd[];
    __shared__ double buf[1024 + 16];
    if (A.ks->done) return;
    const int t = threadIdx.x, lane = t & 31;
    const int e0 = blockIdx.x * A.per, ne = max(0, min(A.per, A.n - e0)), np = ne >> 1;
    double *const xs = A.x + e0, *const hs = A.h + e0, *const gs = smd, *const zs = smd + A.per;
    const double *const ds = A.dinv + e0;
    for (int i = t; i < ne; i += 1024) gs[i] = A.g[e0 + i];
    __syncthreads();
    const double eps2 = A.ks->eps2;
    const int itmax = A.ks->itmax;
    double gcg = A.ks->gcg, gcgp = gcg, gamma = 1.0, rho = 0.0, sgh = A.ks->s_gh, shq = 0.0;
    int iter = 0, conv = 0, k = 0;
    bool good = true;
    const double *const hg = A.h;
    for (;;) {
        // ---- q = A h, (h, q)
        double part = 0.0;
        sell_for_chunks<kSellStride, 1>(A.S, [&](int c, int a, int L, int64_t sr) {
            double y[1];
            sell_row64<1, C16, 2, true>(A.S, A.val, hg, L, sr, lane, a, y);
            if (a >= 0) {
                __stcg(A.q + a, y[0]);
                part = fma(__ldca(hg + a), y[0], part);
            }
        });
        if (!gs_sum_wide<true>(A.gs, k++, part, buf)) { good = false; break; }
        shq = part;
        rho = -sgh / shq;
        // ---- x += rho h, g += rho q, z = C g, (g, z)
        part = 0.0;
#pragma unroll 2
        for (int j = t; j < np; j += 1024) {
            const double2 qv = __ldcg(reinterpret_cast<const double2 *>(A.q + e0) + j);
            const double2 hv = __ldcg(reinterpret_cast<const double2 *>(hs) + j), dv = reinterpret_cast<const double2 *>(ds)[j];
            double2 xv = reinterpret_cast<double2 *>(xs)[j], gv = reinterpret_cast<double2 *>(gs)[j];
            xv.x = fma(rho, hv.x, xv.x); xv.y = fma(rho, hv.y, xv.y);
            gv.x = fma(rho, qv.x, gv.x); gv.y = fma(rho, qv.y, gv.y);
            reinterpret_cast<double2 *>(xs)[j] = xv;
            reinterpret_cast<double2 *>(gs)[j] = gv;
            const double2 zv = make_double2(__dmul_rn(dv.x, gv.x), __dmul_rn(dv.y, gv.y));
            reinterpret_cast<double2 *>(zs)[j] = zv;
            part = fma(gv.x, zv.x, part);
            part = fma(gv.y, zv.y, part);
        }
        if ((ne & 1) && t == 0) {
            const int j = ne - 1;
            xs[j] = fma(rho, __ldcg(hs + j), xs[j]);
            const double gv = fma(rho, __ldcg(A.q + e0 + j), gs[j]);
            gs[j] = gv;
            zs[j] = __dmul_rn(ds[j], gv);
            part = fma(gv, zs[j], part);
        }
        if (!gs_sum_wide<false>(A.gs, k++, part, buf)) { good = false; break; }
        gcgp = gcg;
        gcg = part;
        gamma = gcg / gcgp;
        ++iter;
        conv = gcg < eps2;
        if (conv || iter >= itmax) break;
        // ---- h = gamma h - z, (g, h)
        part = 0.0;
#pragma unroll 2
        for (int j = t; j < np; j += 1024) {
            const double2 gv = reinterpret_cast<const double2 *>(gs)[j], zv = reinterpret_cast<const double2 *>(zs)[j];
            double2 hv = __ldcg(reinterpret_cast<const double2 *>(hs) + j);
            hv.x = fma(gamma, hv.x, -zv.x);
            hv.y = fma(gamma, hv.y, -zv.y);
            __stcg(reinterpret_cast<double2 *>(hs) + j, hv);
            part = fma(gv.x, hv.x, part);
            part = fma(gv.y, hv.y, part);
        }
        if ((ne & 1) && t == 0) {
            const int j = ne - 1;
            const double hv = fma(gamma, __ldcg(hs + j), -zs[j]);
            __stcg(hs + j, hv);
            part = fma(gs[j], hv, part);
        }
        if (!gs_sum_wide<true>(A.gs, k++, part, buf)) { good = false; break; }
        sgh = part;
    }
    if (blockIdx.x == 0 && t == 0) {
        KrylovScalars *ks = A.ks;
        ks->gcg = gcg; ks->gcgp = gcgp; ks->gamma = gamma; ks->rho = rho; ks->s_gh = sgh; ks->s_hq = shq;
        ks->iter = iter;
        ks->converged = conv;
        ks->done = good ? 1 : 2;
    }
}

// ------------------------------------------------------------------ host side
constexpr int kBandOneBlock = 512;
// Rows per block: a multiple of 32, all SMs, at least 64 (a shorter block costs more exchange than
// it saves FP64 time).
static int band_rows(int n) {
    // one block needs no exchange: 4.9 us per iteration for 441 rows, 5.8 with seven blocks
    if (n <= kBandOneBlock) return (n + 31) / 32 * 32;
    const int per = (n + kNumSM - 1) / kNumSM;
    return std::max(64, (per + 31) / 32 * 32);
}
// threads and rows per thread by the rows of a block: 128 threads (one warp per sub-partition)
// keep the block sums short; 256 from 512 rows on, where registers run out
static void *band_fn(int rows, int *nt) {
    *nt = rows <= 512 ? 128 : 256;
    if (rows <= 128) return (void *)cg_band<128, 1>;
    if (rows <= 256) return (void *)cg_band<128, 2>;
    if (rows <= 512) return (void *)cg_band<128, 4>;
    if (rows <= 1024) return (void *)cg_band<256, 4>;
    return (void *)cg_band<256, 8>;
}
constexpr int kBandMaxRows = 2048;
constexpr size_t kBandSmem = 224 * 1024;   // of the 227 KB a block may have: the static arrays too

static size_t band_smem(const ffgpu_matrix *A) {
    return sizeof(double) * (((size_t)A->band_range + 1) & ~(size_t)1) + (size_t)A->band_slots * 32 * (sizeof(double) + sizeof(uint16_t));
}

// Whether the in-kernel loop takes this matrix: a rule on the pattern and the device, never on
// timings.  The pattern's needs are measured once (band_need_kernel).
bool band_cg_fits(ffgpu_matrix *A) {
    ffgpu_ctx *ctx = A->ctx;
    if (!ctx->coop || !ctx->d_sync || A->bs != 1) return false;
    const int rows = band_rows(A->n);
    if (rows > kBandMaxRows) return false;
    if (A->band_range == 0) {
        cudaStream_t s = ctx->stream;
        int need[2] = {0, 0};
        A->band_range = -1;
        if (cudaMemsetAsync(ctx->d_iscratch, 0, sizeof(need), s) != cudaSuccess) return false;
        band_need_kernel<<<(A->n + rows - 1) / rows, 128, 0, s>>>(A->n, rows, A->browptr, A->bcol, ctx->d_iscratch);
        if (launch_check(ctx, "band_need") != FFGPU_OK) return false;
        if (cudaMemcpyAsync(need, ctx->d_iscratch, sizeof(need), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            return false;
        A->band_range = need[0];
        A->band_slots = need[1];
    }
    return A->band_range > 0 && A->band_range < 65536 && band_smem(A) <= kBandSmem;
}

// The loop from the state cg_init leaves (x, g, h, Krylov scalars); h2, cg: two more work
// vectors.  x receives the solution.
int band_cg_run(ffgpu_matrix *A, int trans, double *x, double *g, double *h, double *h2, double *cg, cudaStream_t s) {
    ffgpu_ctx *ctx = A->ctx;
    const int rows = band_rows(A->n);
    int nt = 0;
    void *fn = band_fn(rows, &nt);
    const size_t smem = band_smem(A);
    BandArgs a;
    memset(&a, 0, sizeof(a));
    a.n = A->n; a.rows = rows;
    a.rp = A->browptr; a.col = A->bcol;
    a.val = trans ? A->val_t : A->val;
    a.dinv = A->diag_inv;
    a.x = x; a.g = g; a.h0 = h; a.h1 = h2; a.cg = cg;
    a.ks = A->ks;
    a.gs.slots = (ulonglong2 *)ctx->d_sync;
    a.range_cap = (A->band_range + 1) & ~1;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return kLoopRefused;
    }
    FFGPU_CUDA(cudaMemsetAsync(ctx->d_sync, 0xff, kGsBytes, s));
    void *args[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3((A->n + rows - 1) / rows), dim3(nt), args, smem, s);
    if (e != cudaSuccess) {
        cudaGetLastError();   // nothing ran: the caller takes the launches per iteration
        return kLoopRefused;
    }
    return launch_check(ctx, "cg_band");
}

constexpr size_t kLoopSmem = 190 * 1024;   // the rest of the SM's 256 KB is the L1 the gathers go through
static int loop_piece(int n) { return ((n + kNumSM - 1) / kNumSM + 1) & ~1; }
// Whether the streaming loop takes the system: a rule on sizes and the device.
bool loop_cg_fits(const ffgpu_matrix *A) {
    return A->ctx->coop && A->ctx->d_sync && A->bs == 1 && 2 * sizeof(double) * (size_t)loop_piece(A->n) <= kLoopSmem;
}

// The loop from the state cg_init leaves; z: a work vector.
int loop_cg_run(ffgpu_matrix *A, int trans, double *x, double *g, double *h, double *q, double *z, cudaStream_t s) {
    ffgpu_ctx *ctx = A->ctx;
    FFGPU_TRY(sell_values(A, trans ? kSell64T : kSell64));
    LoopArgs a;
    memset(&a, 0, sizeof(a));
    a.n = A->n;
    a.per = loop_piece(A->n);
    a.S = sell_args(A);
    a.val = trans ? A->sval_t : A->sval;
    a.dinv = A->diag_inv;
    a.x = x; a.g = g; a.h = h; a.q = q; a.z = z;
    a.ks = A->ks;
    a.gs.slots = (ulonglong2 *)ctx->d_sync;
    const size_t smem = 2 * sizeof(double) * (size_t)a.per;
    void *fn = A->scol16 ? (void *)cg_loop<true> : (void *)cg_loop<false>;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return kLoopRefused;
    }
    FFGPU_CUDA(cudaMemsetAsync(ctx->d_sync, 0xff, kGsBytes, s));
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel(fn, dim3(kNumSM), dim3(1024), args, smem, s) != cudaSuccess) {
        cudaGetLastError();
        return kLoopRefused;
    }
    return launch_check(ctx, "cg_loop");
}

}  // namespace ffgpu
