// Pieces of the one-launch CG kernels (persist.cu, persist_batch.cu): mailboxes,
// grid-wide exchanges and CTA sums.
#pragma once

#include "internal.cuh"

namespace ogb {

namespace {

constexpr int PARTS = 4;                  // threads per node row
constexpr int MAX_CTAS = 160;             // five mailboxes per lane of a warp
constexpr int PERSIST_SPIN = 1 << 20;     // polls before a wait gives up
constexpr int WAIT_TIMEOUT = 5;           // PcgScal::done of a wait that gave up
constexpr int BUDGET = 512;               // iterations of a launch
constexpr int SMEM_LIMIT = 227 * 1024;
constexpr int STATIC_SMEM = 12 * 1024;    // the kernels' own shared arrays, rounded up

// A value and the exchange it belongs to, moved as one 16-byte access.
struct __align__(16) Mail {
    double value;
    unsigned long long epoch;
};

__device__ __forceinline__ void post(Mail *m, double v, unsigned long long epoch)
{
    const unsigned __int128 b = (unsigned __int128)epoch << 64 | (unsigned long long)__double_as_longlong(v);
    asm volatile("st.relaxed.gpu.global.b128 [%0], %1;" ::"l"(m), "q"(b) : "memory");
}

__device__ __forceinline__ bool collect(const Mail *m, double &v, unsigned long long epoch)
{
    unsigned __int128 b;
    asm volatile("ld.relaxed.gpu.global.b128 %0, [%1];" : "=q"(b) : "l"(m) : "memory");
    v = __longlong_as_double((long long)(unsigned long long)b);
    return (unsigned long long)(b >> 64) == epoch;
}

// Grid-wide sums of NV values of every CTA, by its first warp: the CTA posts its
// value to a mailbox of every CTA and polls its own mailboxes. A mailbox is polled
// by one CTA only (slots polled by all CTAs took 6 us an exchange), and the value
// and its epoch travel in one 16-byte access, so nothing is cleared and an exchange
// of values alone needs no fence. Two sets alternate: a CTA posts exchange n + 2 after
// it has everyone's n + 1, posted after their senders had read n. ORDER: what any
// thread of any CTA wrote before is visible to the warp after (and to its CTA after
// the next __syncthreads). False when a wait gave up.
//
// The CTAs first .. first + G - 1 of the launch exchange with each other; MV: values
// a mailbox row has room for.
template <int NV, bool ORDER, int MV>
__device__ __forceinline__ bool exchange(Mail *mail, unsigned long long epoch, int first, int G, const double (&mine)[NV],
                                         double (&sum)[NV])
{
    constexpr int PER = MAX_CTAS / 32;
    const int lane = threadIdx.x & 31, total = gridDim.x, me = blockIdx.x - first;
    if (G == 1) {   // one CTA: its own sums (what its threads wrote is ordered by its barriers)
#pragma unroll
        for (int v = 0; v < NV; ++v) sum[v] = mine[v];
        return true;
    }
    Mail *set = mail + (size_t)(epoch & 1) * MV * total * total;
    if (ORDER) asm volatile("fence.acq_rel.gpu;" ::: "memory");
#pragma unroll
    for (int k = 0; k < PER; ++k)
        if (lane + 32 * k < G)
#pragma unroll
            for (int v = 0; v < NV; ++v) post(set + ((size_t)(first + lane + 32 * k) * total + me) * MV + v, mine[v], epoch);
    // (four values at a time: their mailboxes stay in registers)
    bool fine = true;
#pragma unroll
    for (int v0 = 0; v0 < NV; v0 += 4) {
        constexpr int C = NV < 4 ? NV : 4;
        double got[C][PER];
        bool all;
        int spin = 0;
        do {
            all = true;
#pragma unroll
            for (int k = 0; k < PER; ++k)
#pragma unroll
                for (int v = 0; v < C; ++v) {
                    got[v][k] = 0.0;
                    if (v0 + v < NV && lane + 32 * k < G)
                        all &= collect(set + ((size_t)blockIdx.x * total + lane + 32 * k) * MV + v0 + v, got[v][k], epoch);
                }
            all = __all_sync(0xffffffffu, all);
        } while (!all && ++spin < PERSIST_SPIN);
        fine &= all;
#pragma unroll
        for (int v = 0; v < C; ++v)
            if (v0 + v < NV) sum[v0 + v] = ((got[v][0] + got[v][1]) + (got[v][2] + got[v][3])) + got[v][4];
    }
    if (ORDER) asm volatile("fence.acq_rel.gpu;" ::: "memory");
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int v = 0; v < NV; ++v) sum[v] += __shfl_xor_sync(0xffffffffu, sum[v], o);
    return fine;
}

// Fixed-order sums over the CTA of NV values per thread held in `in` (count entries
// each, `stride` apart), for the first warp. Up to four warps per value, so that the
// FP64 additions of a thousand values do not queue up in every warp's shuffles.
template <int NV, class T>
__device__ __forceinline__ void cta_sum(const T *in, int count, int stride, double (&out)[NV], double *warp_sums)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int per = nw >= 4 * NV ? 4 : nw >= NV ? 1 : 0;   // warps per value (0: one warp takes all)
    __syncthreads();
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        if (per ? warp / per != v : warp != 0) continue;
        const int q = per ? warp % per : 0, np = per ? per : 1;
        double s = 0.0;
        for (int i = lane + 32 * q; i < count; i += 32 * np) s += (double)in[v * stride + i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) warp_sums[4 * v + q] = s;
    }
    __syncthreads();
    if (warp == 0)
#pragma unroll
        for (int v = 0; v < NV; ++v)
            out[v] = per == 4 ? (warp_sums[4 * v] + warp_sums[4 * v + 1]) + (warp_sums[4 * v + 2] + warp_sums[4 * v + 3])
                              : warp_sums[4 * v];
}

}  // namespace
}  // namespace ogb
