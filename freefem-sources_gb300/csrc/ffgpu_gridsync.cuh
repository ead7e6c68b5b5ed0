// ffgpu_gridsync.cuh -- sums over all blocks of one cooperative launch, used by the Krylov loops
// that stay inside one kernel.
//
// An exchange is one all-to-all: every block stores its partial sums (16 bytes) into every block's
// inbox and reads its own, so the totals need no counter, no last block and no second trip to
// L2, and no line is polled by more than one SM.  A probe of 148 blocks of 4 warps, block sums
// included: 4.0 us with one array of slots polled by all, 2.9 us with 4 to 32 copies of it,
// 2.8 us with the inboxes (half of that FP64 instructions of the two sums).
// A slot holds kGsEmpty until the partial arrives; a value that would have these bits is a NaN
// and is sent as the canonical one.  The reader empties a slot when it has read it.  Exchange k
// uses the inboxes k & 3.  An exchange that publishes (template argument) makes what the block
// wrote before it visible to every block after it; one that does not costs no fence.  Of any two
// exchanges in a row at least one publishes, so between the emptying of a slot and its next
// use, four exchanges on, lies a publishing one of the reader's that the sender has seen.
// Every wait is bounded: after kGsPolls reads of a slot the sum reports failure to the whole block,
// which leaves its loop, and so do the others when their own waits run out.
// FP64 on GB300 issues one warp instruction per 64 cycles (fused multiply-add) or 76 (add, multiply) and SM
// sub-partition, whatever lanes are active, so the sums are arranged for few instructions: pairs of sums share a warp (lanes
// 0-15 one, 16-31 the other), and four warps, one per sub-partition, read the slots.
#pragma once
#include "ffgpu_internal.cuh"

namespace ffgpu {

constexpr unsigned long long kGsEmpty = 0xffffffffffffffffull;
constexpr int kGsPolls = 1 << 22;      // about 2 s of polling
// many blocks wait before they poll: the polling slows the partials that are still on their way
// (CG on 130^2 and 256^2 cells, per iteration with two exchanges: 7.14 -> 6.4 and 9.42 -> 8.8 us; seven
// blocks lose 0.3 us by it)
constexpr int kGsPatient = 32;
constexpr unsigned kGsWaitNs = 500;
constexpr int kGsMaxBlocks = 160;      // four warps send and read, at most two slots per lane
constexpr size_t kGsBytes = (size_t)4 * kGsMaxBlocks * kGsMaxBlocks * 16;

struct GridSync {
    ulonglong2 *slots;    // 4 x kGsMaxBlocks inboxes x kGsMaxBlocks senders, all kGsEmpty at launch
};
// doubles of shared memory of the sums over NW warps (two halves, used in turn)
template <int NW>
constexpr int kGsRed = 2 * (2 * NW + 8);

template <bool ACQUIRE>
__device__ __forceinline__ ulonglong2 gs_load(const ulonglong2 *p) {
    ulonglong2 v;
    if (ACQUIRE)
        asm volatile("ld.acquire.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    else
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void gs_store(ulonglong2 *p, ulonglong2 v) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(v.x), "l"(v.y) : "memory");
}
__device__ __forceinline__ unsigned long long gs_bits(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return b == kGsEmpty ? 0x7fffffffffffffffull : b;
}

// lanes 0-15: the warp's sum of a; lanes 16-31: of b (five FP64 instructions for both)
__device__ __forceinline__ double warp_sum_pair(double a, double b) {
    const bool hi = threadIdx.x & 16;
    double keep = hi ? b : a;
    const double send = hi ? a : b;
    keep += __shfl_xor_sync(0xffffffffu, send, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) keep += __shfl_xor_sync(0xffffffffu, keep, o);
    return keep;
}

// Totals of (a, b) over all threads of all blocks, in a fixed order; the same bits in every
// thread.  PUBLISH: whatever the block stored to global memory before is visible to every block
// after (other blocks' data have to be read past L1).  k: the number of the exchange, 0, 1, ...;
// red: kGsRed<NW> doubles of shared memory.  Returns false in every thread of the block when a
// wait ran out.
template <int NW, bool PUBLISH>
__device__ __forceinline__ bool gs_sum2(const GridSync &G, int k, double &a, double &b, double *red) {
    static_assert(NW >= 4 && NW <= 16 && (NW & (NW - 1)) == 0, "4, 8 or 16 warps");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned full = 0xffffffffu;
    red += (k & 1) * (2 * NW + 8);   // the last sum's readers may still be at theirs
    double p = warp_sum_pair(a, b);
    if ((lane & 15) == 0) red[(lane >> 4) * NW + w] = p;
    __syncthreads();
    const int nb = gridDim.x;
    const double *src = red;
    int cnt = NW;
    bool ok = true;
    if (nb > 1) {
        ulonglong2 *const all = G.slots + (size_t)(k & 3) * kGsMaxBlocks * kGsMaxBlocks;
        if (w < 4) {
            // each sending warp finishes the block's sum itself (no barrier in between)
            double v = lane < 2 * NW ? red[lane] : 0.0;
#pragma unroll
            for (int o = NW / 2; o > 0; o >>= 1) v += __shfl_xor_sync(full, v, o);
            const double va = __shfl_sync(full, v, 0), vb = __shfl_sync(full, v, NW);
            const ulonglong2 out = make_ulonglong2(gs_bits(va), gs_bits(vb));
            if (PUBLISH) __threadfence();
            for (int d = w * 32 + lane; d < nb; d += 128) gs_store(all + (size_t)d * kGsMaxBlocks + blockIdx.x, out);
            ulonglong2 *const box = all + (size_t)blockIdx.x * kGsMaxBlocks;
            const int per = (nb + 3) >> 2;            // at most 64
            const int i0 = w * per + lane, i1 = i0 + 32;
            const bool h0 = lane < per && i0 < nb, h1 = lane + 32 < per && i1 < nb;
            ulonglong2 s0 = make_ulonglong2(0, 0), s1 = make_ulonglong2(0, 0);
            bool m0 = h0, m1 = h1;
            int left = kGsPolls;
            if (nb >= kGsPatient) __nanosleep(kGsWaitNs);
            while (m0 || m1) {
                if (m0) s0 = gs_load<PUBLISH>(box + i0);
                if (m1) s1 = gs_load<PUBLISH>(box + i1);
                m0 = m0 && (s0.x == kGsEmpty || s0.y == kGsEmpty);
                m1 = m1 && (s1.x == kGsEmpty || s1.y == kGsEmpty);
                if (--left == 0) break;
            }
            ok = !(m0 || m1);
            if (h0) gs_store(box + i0, make_ulonglong2(kGsEmpty, kGsEmpty));
            if (h1) gs_store(box + i1, make_ulonglong2(kGsEmpty, kGsEmpty));
            __syncwarp();
            double ta = __longlong_as_double((long long)s0.x), tb = __longlong_as_double((long long)s0.y);
            if (per > 32) {
                ta += __longlong_as_double((long long)s1.x);
                tb += __longlong_as_double((long long)s1.y);
            }
            p = warp_sum_pair(ta, tb);
            if ((lane & 15) == 0) red[2 * NW + (lane >> 4) * 4 + w] = p;
        }
        src = red + 2 * NW;
        cnt = 4;
    }
    if (__syncthreads_or(!ok)) return false;
    const double *mine = src + (lane >> 4) * cnt;
    double t = mine[0];
    for (int i = 1; i < cnt; ++i) t += mine[i];
    a = __shfl_sync(full, t, 0);
    b = __shfl_sync(full, t, 16);
    return true;
}

// Total of one value per thread over all threads of all blocks of 32 warps, as gs_sum2.  The block's
// 1024 values are summed by four warps, eight per lane, through shared memory: 15 FP64
// instructions on each sub-partition where a shuffle tree in every warp takes 40.
// buf: 1024 + 16 doubles.
template <bool PUBLISH>
__device__ __forceinline__ bool gs_sum_wide(const GridSync &G, int k, double &a, double *buf) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double *part = buf + 1024, *tot = part + 8;   // part: two halves used in turn, tot likewise
    part += (k & 1) * 4;
    tot += (k & 1) * 4;
    buf[threadIdx.x] = a;
    __syncthreads();
    const int nb = gridDim.x;
    bool ok = true;
    if (w < 4) {
        double v = buf[w * 256 + lane];
#pragma unroll
        for (int i = 1; i < 8; ++i) v += buf[w * 256 + 32 * i + lane];
        v = warp_sum(v);
        if (lane == 0) part[w] = v;
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const double mine = (part[0] + part[1]) + (part[2] + part[3]);
        double t = mine;
        if (nb > 1) {
            ulonglong2 *const all = G.slots + (size_t)(k & 3) * kGsMaxBlocks * kGsMaxBlocks;
            const ulonglong2 out = make_ulonglong2(gs_bits(mine), 0);
            if (PUBLISH) __threadfence();
            for (int d = w * 32 + lane; d < nb; d += 128) gs_store(all + (size_t)d * kGsMaxBlocks + blockIdx.x, out);
            ulonglong2 *const box = all + (size_t)blockIdx.x * kGsMaxBlocks;
            const int per = (nb + 3) >> 2;
            const int i0 = w * per + lane, i1 = i0 + 32;
            const bool h0 = lane < per && i0 < nb, h1 = lane + 32 < per && i1 < nb;
            ulonglong2 s0 = make_ulonglong2(0, 0), s1 = make_ulonglong2(0, 0);
            bool m0 = h0, m1 = h1;
            int left = kGsPolls;
            if (nb >= kGsPatient) __nanosleep(kGsWaitNs);
            while (m0 || m1) {
                if (m0) s0 = gs_load<PUBLISH>(box + i0);
                if (m1) s1 = gs_load<PUBLISH>(box + i1);
                m0 = m0 && s0.x == kGsEmpty;
                m1 = m1 && s1.x == kGsEmpty;
                if (--left == 0) break;
            }
            ok = !(m0 || m1);
            if (h0) gs_store(box + i0, make_ulonglong2(kGsEmpty, kGsEmpty));
            if (h1) gs_store(box + i1, make_ulonglong2(kGsEmpty, kGsEmpty));
            __syncwarp();
            t = __longlong_as_double((long long)s0.x);
            if (per > 32) t += __longlong_as_double((long long)s1.x);
            t = warp_sum(t);
        } else if (w) {
            t = 0.0;
        }
        if (lane == 0) tot[w] = t;
    }
    if (__syncthreads_or(!ok)) return false;
    a = (tot[0] + tot[1]) + (tot[2] + tot[3]);
    return true;
}

}  // namespace ffgpu
