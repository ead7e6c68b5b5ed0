// ffgpu_persist.cu -- the CG loop of ffgpu_solve_cg inside one cooperative kernel.
//
// FreeFEM's ConjugueGradient (src/femlib/CG.cpp:196-265) as ffgpu_solve.cu describes it, in two
// forms.  cg_loop, further down, streams the matrix.  cg_band is for scalar systems whose matrix
// fits the SMs' shared memory.  One block per SM owns consecutive rows for the whole solve:
//   * its rows of the matrix in shared memory (values FP64, columns as 16-bit numbers relative
//     to the first column the block touches), x, g and 1/A_ii in registers;
//   * per iteration it forms the direction h' = gamma h - C g once for every column it touches
//     (its own rows and the halo), from the h and C g the owners left in L2, multiplies from
//     shared memory, and takes part in two exchanges (ffgpu_gridsync.cuh): (g,h'), (h',A h')
//     and (g, C g).
// So nothing of the matrix moves after the start, and an iteration is two trips through L2.
// Where the rows touch a wide range of columns (a mesh numbered at random), forming h' for all of
// it would cost more than the rest: the WIDE form gathers the pair (h, C g) of each entry from L2.
// Rows of unequal length (P2) are taken in the order of their length within a block where 32
// consecutive rows padded to the longest would not fit.
// The launches of the two-kernel loop spend an iteration on kernel boundaries, a chain of
// dependent L2 reads and FP64 reductions over many more warps than the sums need.
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <type_traits>

#include "ffgpu_gridsync.cuh"
#include "ffgpu_sell.cuh"

namespace ffgpu {

constexpr int kWideBatch = 8;    // gathers of a row in flight (WIDE)

struct BandArgs {
    int n, rows;                 // rows per block
    const int32_t *rp, *col;
    const double *val, *dinv;
    double *x, *g, *h0, *h1, *cg;
    double2 *pair;               // WIDE: (h, C g) of every row
    const uint16_t *perm;        // rows of a block by length (NULL: as numbered), relative to its first
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

// The rows of each block by decreasing length (ties as numbered) and the slots of their groups: the place
// of a row is the number of rows before it.
__global__ void __launch_bounds__(256) band_sort_kernel(int n, int rows, const int32_t *__restrict__ rp,
                                                        uint16_t *__restrict__ perm, int *need) {
    extern __shared__ int sh_len[];
    int *sorted = sh_len + rows;
    const int r0 = blockIdx.x * rows, m = min(n, r0 + rows) - r0;
    for (int i = threadIdx.x; i < m; i += blockDim.x) sh_len[i] = rp[r0 + i + 1] - rp[r0 + i];
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int L = sh_len[i];
        int rank = 0;
        for (int k = 0; k < m; ++k) rank += sh_len[k] > L || (sh_len[k] == L && k < i);
        perm[r0 + rank] = (uint16_t)i;
        sorted[rank] = L;
    }
    __syncthreads();
    int slots = 0;
    for (int q = threadIdx.x * 32; q < m; q += blockDim.x * 32) slots += sorted[q];
    slots = __reduce_add_sync(0xffffffffu, slots);
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) atomicAdd(&total, slots);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(need, total);
}

// RPT rows per thread, NT threads.  Row u * NT + t of the block's order belongs to thread t.
// FP64 instructions set the floor (one per 64 to 76 cycles and sub-partition): about 16 per group of
// 32 rows and iteration on a 2D P1 mesh.
template <int NT, int RPT, bool WIDE>
__global__ void __launch_bounds__(NT, 1) cg_band(BandArgs A) {
    constexpr int NW = NT / 32;
    using Col = std::conditional_t<WIDE, int32_t, uint16_t>;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[kGsRed<NW>];
    __shared__ int s_lo, s_hi, s_base[RPT * NW + 1];
    if (A.ks->done) return;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int r0 = blockIdx.x * A.rows, r1 = min(A.n, r0 + A.rows);
    double *hs = reinterpret_cast<double *>(smraw);
    if (t == 0) { s_lo = 0x7fffffff; s_hi = -1; }
    __syncthreads();
    double x[RPT], g[RPT], z[RPT], d[RPT], ho[RPT];
    int len[RPT], row[RPT];      // row: -1 past the block's rows
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
        const int p = r0 + u * NT + t;
        const int r = p >= r1 ? -1 : A.perm ? r0 + A.perm[p] : p;
        int L = 0;
        row[u] = r;
        x[u] = g[u] = z[u] = d[u] = ho[u] = 0.0;
        if (r >= 0) {
            const int b = A.rp[r], e = A.rp[r + 1];
            L = e - b;
            if (!WIDE) {
                int cl = r, ch = r;
                for (int k = b; k < e; ++k) { cl = min(cl, A.col[k]); ch = max(ch, A.col[k]); }
                atomicMin(&s_lo, cl);
                atomicMax(&s_hi, ch);
            }
            x[u] = A.x[r]; g[u] = A.g[r]; d[u] = A.dinv[r];
            if (WIDE) {
                ho[u] = A.h0[r];
                __stcg(A.pair + r, make_double2(ho[u], 0.0));
            }
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
    const int lo = WIDE ? 0 : s_lo, nc = WIDE ? 0 : s_hi - lo + 1;
    double *mv = hs + A.range_cap;
    Col *mc = reinterpret_cast<Col *>(mv + (size_t)s_base[RPT * NW] * 32);
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
        const int r = row[u];
        const int b = r >= 0 ? A.rp[r] : 0, L = r >= 0 ? A.rp[r + 1] - b : 0;
        const int base = s_base[u * NW + w] * 32 + lane;
        for (int j = 0; j < len[u]; ++j) {
            mv[base + 32 * j] = j < L ? A.val[b + j] : 0.0;
            mc[base + 32 * j] = (Col)(j < L ? A.col[b + j] - lo : WIDE ? max(r, 0) : 0);
        }
    }
    const double eps2 = A.ks->eps2;
    const int itmax = A.ks->itmax;
    double gcg = A.ks->gcg, gcgp = gcg, gamma = 1.0, rho = 0.0, sgh = 0.0, shq = 0.0;
    int iter = 0, conv = 0, k = 0;
    bool good = true;
    const double *hold = A.h0;
    double *hnew = A.h1;
    if (WIDE) {                  // all pairs are there before the first gather
        double a = 0.0, b = 0.0;
        good = gs_sum2<NW, true>(A.gs, k++, a, b, red);
    }
    while (good) {
        if (!WIDE) {
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
        }
        // ---- q = A h', the rows' products side by side
        double y[RPT];
        double pa = 0.0, pb = 0.0;
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
            const int r = row[u];
            const int base = s_base[u * NW + w] * 32 + lane;
            double s = 0.0;
            if (WIDE) {
                // the pairs of a batch of entries, then the products
                for (int j = 0; j < len[u]; j += kWideBatch) {
                    double2 p[kWideBatch];
#pragma unroll
                    for (int q = 0; q < kWideBatch; ++q)
                        if (j + q < len[u]) p[q] = __ldcg(A.pair + mc[base + 32 * (j + q)]);
#pragma unroll
                    for (int q = 0; q < kWideBatch; ++q)
                        if (j + q < len[u]) s = fma(mv[base + 32 * (j + q)], fma(gamma, p[q].x, -p[q].y), s);
                }
            } else {
#pragma unroll 4
                for (int j = 0; j < len[u]; ++j) s = fma(mv[base + 32 * j], hs[mc[base + 32 * j]], s);
            }
            y[u] = s;
            if (u * NT < A.rows) {               // uniform: groups past the rows do no FP64 work
                if (WIDE) {
                    ho[u] = fma(gamma, ho[u], -z[u]);
                } else {
                    ho[u] = r >= 0 ? hs[r - lo] : 0.0;
                    if (r >= 0) __stcg(hnew + r, ho[u]);
                }
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
                const int r = row[u];
                x[u] = fma(rho, ho[u], x[u]);
                g[u] = fma(rho, y[u], g[u]);
                z[u] = __dmul_rn(d[u], g[u]);
                if (r >= 0) {
                    if (WIDE) __stcg(A.pair + r, make_double2(ho[u], z[u]));   // every block has gathered
                    else __stcg(A.cg + r, z[u]);
                }
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
    for (int u = 0; u < RPT; ++u)
        if (row[u] >= 0) A.x[row[u]] = x[u];
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
constexpr int kBandRange = 64;
constexpr int kWideThreads = 256;
// longest row of the wide form: its warp gathers the row's slots alone, about 0.1 us each (120^2 cells and one
// row of 60, 100 and 120 entries: 14.6, 19.0 and 21.7 us per iteration, with launches 16.2, 19.0, 20.1)
constexpr int kWideDeg = 96;
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
static int band_threads(int rows) { return rows <= 512 ? 128 : 256; }
static void *band_fn(int rows, bool wide, int *nt) {
    if (wide) {
        *nt = kWideThreads;
        if (rows <= kWideThreads) return (void *)cg_band<kWideThreads, 1, true>;
        if (rows <= 2 * kWideThreads) return (void *)cg_band<kWideThreads, 2, true>;
        if (rows <= 4 * kWideThreads) return (void *)cg_band<kWideThreads, 4, true>;
        return (void *)cg_band<kWideThreads, 8, true>;
    }
    *nt = band_threads(rows);
    if (rows <= 128) return (void *)cg_band<128, 1, false>;
    if (rows <= 256) return (void *)cg_band<128, 2, false>;
    if (rows <= 512) return (void *)cg_band<128, 4, false>;
    if (rows <= 1024) return (void *)cg_band<256, 4, false>;
    return (void *)cg_band<256, 8, false>;
}
constexpr int kBandMaxRows = 2048;
constexpr size_t kBandSmem = 224 * 1024;   // of the 227 KB a block may have: the static arrays too

static size_t band_smem(int range, int slots, bool wide) {
    const size_t entries = (size_t)slots * 32;
    return wide ? entries * (sizeof(double) + sizeof(int32_t))
                : sizeof(double) * (((size_t)range + 1) & ~(size_t)1) + entries * (sizeof(double) + sizeof(uint16_t));
}

// Whether the in-kernel loop takes this matrix, and how: a rule on the pattern and the device, never on
// timings.  The pattern's needs are measured once (band_need_kernel, band_sort_kernel).
bool band_cg_fits(ffgpu_matrix *A) {
    ffgpu_ctx *ctx = A->ctx;
    if (!ctx->coop || !ctx->d_sync || A->bs != 1) return false;
    const int rows = band_rows(A->n), blocks = (A->n + rows - 1) / rows;
    if (rows > kBandMaxRows) return false;
    if (A->band_kind != kBandUnknown) return A->band_kind != kBandNone;
    cudaStream_t s = ctx->stream;
    int need[2] = {0, 0};
    A->band_kind = kBandNone;
    if (cudaMemsetAsync(ctx->d_iscratch, 0, sizeof(need), s) != cudaSuccess) return false;
    band_need_kernel<<<blocks, 128, 0, s>>>(A->n, rows, A->browptr, A->bcol, ctx->d_iscratch);
    if (launch_check(ctx, "band_need") != FFGPU_OK) return false;
    if (cudaMemcpyAsync(need, ctx->d_iscratch, sizeof(need), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return false;
    A->band_range = need[0];
    // Staging costs about 0.10 us per column and thread and iteration, gathering 0.25 us more per entry and thread
    // than shared memory does: staged up to twice as many columns as the wide form has entries per thread.  Per
    // iteration, staged and wide: 300^2 numbered at random in pieces, 31 columns and 12 entries a thread,
    // 12.8 and 12.4 us; 500^2, 62 and 32: 19.3 and 20.7; 400^2, 62 and 21: 17.8 and 16.7; 60^3, 34 and 39: 16.5
    // and 18.7.  (Staged without a limit: 165^2 numbered at random, 213 and 5: 31.4 us; wide 8.6, launches 14.0.)
    // Up to kBandRange columns per thread it is still ahead of the launches where a long row rules out the wide form.
    const int64_t cols = need[0] / band_threads(rows), entries = A->nnz / ((int64_t)blocks * kWideThreads);
    const bool wide = A->max_deg <= kWideDeg;
    const bool staged = cols <= std::max<int64_t>(16, 2 * entries) || (!wide && cols <= kBandRange);
    const auto take = [&](int slots) {
        A->band_slots = slots;
        if (staged && band_smem(need[0], slots, false) <= kBandSmem) A->band_kind = kBandStaged;
        else if (wide && band_smem(0, slots, true) <= kBandSmem) A->band_kind = kBandWide;
        return A->band_kind != kBandNone;
    };
    if (take(need[1])) return true;
    // by length, if the entries alone could fit
    if (!(staged || wide) || A->nnz / blocks * 10 > (int64_t)kBandSmem) return false;
    if (dalloc(ctx, (void **)&A->band_perm, sizeof(uint16_t) * (size_t)A->n) != cudaSuccess) return false;
    int slots = 0;
    if (cudaMemsetAsync(ctx->d_iscratch, 0, sizeof(int), s) == cudaSuccess) {
        band_sort_kernel<<<blocks, 256, 2 * sizeof(int) * rows, s>>>(A->n, rows, A->browptr, A->band_perm, ctx->d_iscratch);
        if (launch_check(ctx, "band_sort") == FFGPU_OK &&
            cudaMemcpyAsync(&slots, ctx->d_iscratch, sizeof(int), cudaMemcpyDeviceToHost, s) == cudaSuccess &&
            cudaStreamSynchronize(s) == cudaSuccess && take(slots))
            return true;
    }
    dfree(ctx, A->band_perm);
    A->band_perm = nullptr;
    return false;
}

// The loop from the state cg_init leaves (x, g, h, Krylov scalars); h2, cg: two more work
// vectors, pair: two vectors side by side.  x receives the solution.
int band_cg_run(ffgpu_matrix *A, int trans, double *x, double *g, double *h, double *h2, double *cg, double *pair,
                cudaStream_t s) {
    ffgpu_ctx *ctx = A->ctx;
    const int rows = band_rows(A->n);
    const bool wide = A->band_kind == kBandWide;
    int nt = 0;
    void *fn = band_fn(rows, wide, &nt);
    const size_t smem = band_smem(A->band_range, A->band_slots, wide);
    BandArgs a;
    memset(&a, 0, sizeof(a));
    a.n = A->n; a.rows = rows;
    a.rp = A->browptr; a.col = A->bcol;
    a.val = trans ? A->val_t : A->val;
    a.dinv = A->diag_inv;
    a.x = x; a.g = g; a.h0 = h; a.h1 = h2; a.cg = cg;
    a.ks = A->ks;
    a.gs.slots = (ulonglong2 *)ctx->d_sync;
    a.range_cap = wide ? 0 : (A->band_range + 1) & ~1;
    a.pair = reinterpret_cast<double2 *>(pair);
    a.perm = A->band_perm;
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
// Whether the streaming loop takes the system (sell: its tuned layout is SELL): a rule on sizes, the numbering (16-bit
// column differences) and the device.  Per iteration, loop and launches: P1 along the grid, 60^3 cells 30.2 and
// 32.5 us, 118^3 94 and 105, 1300^2 69.6 and 73.3; numbered at random 38.7 and 35.6, 191 and 148, 103 and 90.6: one
// block per SM has fewer gathers in flight.
// Where the tuner took block CSR, rows are long or of unequal length, and the loop's warps have to have chunks of
// 32 rows alike: it runs where their passes are 0.65 full or more (P2 on 28^3 cells, 0.60: 44.0 and 43.5; 29^3, 0.66:
// 44.4 and 45.4; 30^3, 0.73: 45.1 and 49.0; 32^3, 0.88: 46.1 and 58.3), the longest row is no more than its warp
// can walk beside the others (one of 120 entries in 80^3 58.4 and 71.6, of 250 83.3 and 73.3) and little is padding.
constexpr int kLoopDeg = 128;
bool loop_cg_fits(ffgpu_matrix *A, bool sell) {
    if (!A->ctx->coop || !A->ctx->d_sync || A->bs != 1 || 2 * sizeof(double) * (size_t)loop_piece(A->n) > kLoopSmem) return false;
    if (sell) return A->scol16;
    const int64_t chunks = (A->n + 31) / 32, warps = 32 * kNumSM, passes = (chunks + warps - 1) / warps;
    if (A->max_deg > kLoopDeg || 20 * chunks < 13 * warps * passes) return false;
    return sell_prepare(A) == FFGPU_OK && A->scol16 && 4 * A->nslot * 32 <= 5 * A->nnz;
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
