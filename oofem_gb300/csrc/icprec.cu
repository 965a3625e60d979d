// Incomplete-Cholesky preconditioner of the IML solver (lsprecond 4,
// CompCol_ICPreconditioner, src/core/iml/icprecond.C:40-226).
//
// Factorization (host, once per matrix version, as the reference does it on
// its host): the lower triangle of the symmetric matrix by columns -- column k
// holds rows >= k, the diagonal first; for the symmetric pattern stored here
// that is row k of the CSR restricted to columns >= k -- then the reference's
// ICFactor loop (icprecond.C:133-163) kept step for step: the diagonal takes a
// square root, the column is divided by it, and the columns of the rows below
// are updated by the same nested search over row indices. That search only
// matches at the last entry of column k (its successor test reads into the next
// column), so the factor it produces is not a textbook IC(0); parity requires
// the same loop, not a cleaner one.
//
// Application (device): ICSolve (icprecond.C:166-190), a forward and a backward
// substitution, runs by rows as a dataflow inside one thread-block cluster
// (k_tri_flow below): no barrier between levels, a row starts when the last
// value it needs arrives. A row's products are summed in a fixed order (by the
// schedule, not by column), so z = M^-1 r is bitwise reproducible and equals the
// reference's to rounding.
//
// lsprecond 2 (CompCol_ILUPreconditioner, src/core/iml/iluprecond.C:75-193,
// 265-289) is built the same way: the matrix split by columns into a strictly
// lower L (unit diagonal implied) and an upper U with the diagonal last, the
// reference's factorization loop, and its solves L w = x and U y = w.
#include <math.h>
#include <math_constants.h>

#include <algorithm>
#include <vector>

#include "internal.cuh"

namespace ogb {

namespace {

// ---------------------------------------------------------------- device solves
// Both triangular solves and r.z in one launch of one thread-block cluster.
//
// The rows are grouped on the host into units of up to four consecutive rows, each
// depending on the one before (the DOFs of a node, or of a node and a half), the
// units sorted by their dependency level and dealt round-robin to the warps of the
// cluster. A warp takes its units in that order; a unit's row is held by eight
// lanes. The solution vector is replicated in the shared memory of every CTA and
// starts as a NaN pattern no arithmetic produces; a lane polls its own CTA's copy
// until the entry has arrived, and the warp that finishes a row stores it to all
// copies through distributed shared memory. Every unit waits only on units before
// it in the order and all warps are resident, so some warp can always go on.
// What bounds it is the chain of dependent rows: per unit one remote store, the
// last product, three shuffle sums of eight lanes and the unit's own 4 x 4
// triangle (rows' values by shuffle). A row's entries are sorted by when they
// become ready, so all but the last are summed while the warp would wait, and the
// next unit's coefficients are loaded meanwhile.
// Systems whose vector does not fit the shared memory of a CTA (LOCAL false,
// FLOW_LOCAL_MAX rows) keep it in global memory, preset to the same pattern, and
// poll it through L2.
//
// Measured (GB300, 33 x 7 x 6 hexes, 5.5 k rows, 71 node levels): forward plus
// backward solve and r.z 116 us; the previous form, one cluster barrier, one round
// of L2 gathers and a 40-long chain of differences per scalar level (213 levels),
// 2,370 us without r.z.
constexpr int FLOW_THREADS = 512;
constexpr int FLOW_KP = 8;             // entries per lane loaded ahead
constexpr int FLOW_ROWS = 4;           // rows of a unit at most
constexpr int FLOW_LOCAL_MAX = 28800;  // rows of a shared-memory copy (8 bytes each of 227 KB)
constexpr int FLOW_SPIN = 1 << 20;     // polls before a wait gives up
constexpr unsigned long long FLOW_EMPTY = 0xffffffffffffffffull;

struct FlowView {
    int nunits;
    const int4 *unit;       // first row in processing order, rows, slots per lane, first slot / 32
    const double *coef;     // per unit and row: its entries in the unit's earlier rows (3), 1 / diagonal
    const int *col;         // slot k of lane l at 32 k + l (-1: none)
    const double *val;
};

template <bool LOCAL>
__device__ __forceinline__ unsigned long long flow_load(const double *x)
{
    unsigned long long b;
    if (LOCAL)
        asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];"
                     : "=l"(b)
                     : "r"((uint32_t)__cvta_generic_to_shared(x))
                     : "memory");
    else
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b) : "l"(x) : "memory");
    return b;
}

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n"
                 "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// One substitution over F's units. in: right-hand side; x: the vector of this solve
// (LOCAL: the CTA's copy), out: its global copy; rdot: r of the fused r.z (or null).
template <bool LOCAL, bool REV>
__device__ __forceinline__ void flow_solve(const FlowView &F, int n, const double *in, double *x, double *out,
                                           const double *rdot, double &dot, uint32_t rank, uint32_t nranks, bool &dead)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 3, sub = lane & 7;
    const int first = (int)rank + (int)nranks * warp, stride = (int)nranks * (FLOW_THREADS / 32);
    int4 u = make_int4(0, 0, 0, 0);
    int c[FLOW_KP];
    double v[FLOW_KP], bi = 0.0, ri = 0.0;
    double4 cf = make_double4(0, 0, 0, 0);
    auto fetch = [&](int p, int4 &nu, int (&nc)[FLOW_KP], double (&nv)[FLOW_KP], double &nb, double &nr, double4 &ncf) {
        nu = make_int4(0, 0, 0, 0);
        if (p < F.nunits) nu = __ldg(F.unit + p);
#pragma unroll
        for (int k = 0; k < FLOW_KP; ++k) {
            const bool on = k < nu.z;
            nc[k] = on ? __ldg(F.col + 32 * ((size_t)nu.w + k) + lane) : -1;
            nv[k] = on ? __ldg(F.val + 32 * ((size_t)nu.w + k) + lane) : 0.0;
        }
        nb = nr = 0.0;
        if (g < nu.y) {
            const int i = REV ? n - 1 - (nu.x + g) : nu.x + g;
            nb = __ldcg(in + i);
            if (rdot) nr = __ldg(rdot + i);
            const double2 *cp = reinterpret_cast<const double2 *>(F.coef + (size_t)p * 16 + g * 4);
            const double2 a = __ldg(cp), b = __ldg(cp + 1);
            ncf = make_double4(a.x, a.y, b.x, b.y);
        } else {
            ncf = make_double4(0, 0, 0, 0);
        }
    };
    fetch(first, u, c, v, bi, ri, cf);
    for (int p = first; p < F.nunits; p += stride) {
        int4 nu;
        int nc[FLOW_KP];
        double nv[FLOW_KP], nb, nr;
        double4 ncf;
        fetch(p + stride, nu, nc, nv, nb, nr, ncf);
        double s = 0.0;
        unsigned long long b[FLOW_KP];
#pragma unroll
        for (int k = 0; k < FLOW_KP; ++k) b[k] = c[k] >= 0 ? flow_load<LOCAL>(x + c[k]) : 0ull;
        auto take = [&](unsigned long long bits, int col, double val) {
            int spin = 0;
            while (__any_sync(0xffffffffu, bits == FLOW_EMPTY) && !dead) {
                if (bits == FLOW_EMPTY) bits = flow_load<LOCAL>(x + col);
                if (++spin > FLOW_SPIN) dead = true;   // the same count in every lane: a uniform exit
            }
            s = fma(val, __longlong_as_double((long long)bits), s);
        };
#pragma unroll
        for (int k = 0; k < FLOW_KP; ++k)
            if (k < u.z) take(b[k], c[k], v[k]);
        for (int k = FLOW_KP; k < u.z; ++k) {
            const int ck = __ldg(F.col + 32 * ((size_t)u.w + k) + lane);
            const double vk = __ldg(F.val + 32 * ((size_t)u.w + k) + lane);
            take(ck >= 0 ? flow_load<LOCAL>(x + ck) : 0ull, ck, vk);
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        double t = bi - s;
        const double tri[3] = {cf.x, cf.y, cf.z};
#pragma unroll
        for (int j = 0; j < FLOW_ROWS - 1; ++j)
            if (j + 1 < u.y) {
                const double xj = __shfl_sync(0xffffffffu, t * cf.w, 8 * j);
                if (g > j) t = fma(-tri[j], xj, t);
            }
        double xi = t * cf.w;
        if (g < u.y) {
            const int i = REV ? n - 1 - (u.x + g) : u.x + g;
            unsigned long long bits = (unsigned long long)__double_as_longlong(xi);
            if (bits == FLOW_EMPTY) bits = 0x7ff8000000000000ull;
            if (LOCAL) {
                const uint32_t a = (uint32_t)__cvta_generic_to_shared(x + i);
                for (uint32_t q = sub; q < nranks; q += 8) {
                    uint32_t ra;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(q));
                    asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(ra), "l"(bits) : "memory");
                }
                if (sub == 0) out[i] = xi;
            } else if (sub == 0) {
                asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(out + i), "l"(bits) : "memory");
            }
            if (sub == 0) dot += ri * xi;
        }
        u = nu;
        cf = ncf;
        bi = nb;
        ri = nr;
#pragma unroll
        for (int k = 0; k < FLOW_KP; ++k) {
            c[k] = nc[k];
            v[k] = nv[k];
        }
    }
}

// z = M^-1 r (forward into work, backward into z) and, with sc, r.z -> rho, beta
// (none in the first iteration) as IML's CG takes them.
template <bool LOCAL>
__global__ void __launch_bounds__(FLOW_THREADS, 1) k_tri_flow(int n, FlowView F, FlowView B, const double *r, double *work,
                                                             double *z, PcgScal *sc, int *status)
{
    if (sc && (sc->done || sc->reliable)) return;   // the same for every CTA of the cluster
    extern __shared__ double xs[];
    __shared__ double wsum[FLOW_THREADS / 32], csum[16];
    uint32_t rank, nranks;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(nranks));
    bool dead = false;
    double dot = 0.0, none = 0.0;
    auto clear = [&]() {
        if (LOCAL)
            for (int i = threadIdx.x; i < n; i += FLOW_THREADS) xs[i] = __longlong_as_double((long long)FLOW_EMPTY);
        cluster_barrier();
    };
    clear();
    flow_solve<LOCAL, false>(F, n, r, LOCAL ? xs : work, work, nullptr, none, rank, nranks, dead);
    cluster_barrier();   // every copy complete and read before it is cleared
    clear();
    flow_solve<LOCAL, true>(B, n, work, LOCAL ? xs : z, z, r, dot, rank, nranks, dead);
    if (dead) atomicCAS(status, DS_OK, DS_TIMEOUT);
    // r.z: lanes, warps, then CTAs, each in index order
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_down_sync(0xffffffffu, dot, o);
    if (lane == 0) wsum[warp] = dot;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < FLOW_THREADS / 32; ++w) t += wsum[w];
        uint32_t ra;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                     : "=r"(ra)
                     : "r"((uint32_t)__cvta_generic_to_shared(csum + rank)), "r"(0u));
        asm volatile("st.relaxed.cluster.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(dead ? CUDART_NAN : t) : "memory");
    }
    cluster_barrier();   // also: no CTA leaves while another may still store to it
    if (!sc || rank != 0 || threadIdx.x != 0) return;
    double rz = 0.0;
    for (uint32_t q = 0; q < nranks; ++q) rz += csum[q];
    if (!isfinite(rz) || !(rz > 0.0)) {
        sc->done = 2;
        return;
    }
    sc->beta = sc->iters == 0 ? 0.0 : rz / sc->rho;
    sc->rho = rz;
    sc->zcoef = 1.0;
}

// ---------------------------------------------------------------- host schedule
// Units, their order and the slot of every entry for one triangular solve given by
// rows (ptr, col); reversed: rows run from n - 1 down (entries in later rows).
// Kept as long as the structure stays the same; the values are filled in per factor.
void flow_schedule(FlowSched &S, int n, bool rev, const std::vector<int64_t> &ptr, const std::vector<int> &col)
{
    if (S.n == n && S.ptr == ptr && S.col == col) return;
    S.n = n;
    S.ptr = ptr;
    S.col = col;
    const auto row = [&](int t) { return rev ? n - 1 - t : t; };
    // rows of a unit at most: two to four, whichever gives the shorter chain of
    // units (a unit's cost grows by one shuffle and two FP64 operations per row)
    std::vector<int> start, unit_of(n), lev;
    double best = 0.0;
    for (int cap = 2; cap <= FLOW_ROWS; ++cap) {
        std::vector<int> st, uo(n), lv;
        int nlev = 0;
        for (int t = 0; t < n;) {
            int len = 1;
            while (len < cap && t + len < n) {   // the next row needs the one before it, or neither needs any
                const int i = row(t + len), prev = row(t + len - 1);
                bool link = ptr[i] == ptr[i + 1] && ptr[prev] == ptr[prev + 1];
                for (int64_t e = ptr[i]; e < ptr[i + 1] && !link; ++e) link = col[e] == prev;
                if (!link) break;
                ++len;
            }
            const int id = (int)st.size();
            st.push_back(t);
            int l = 0;
            for (int q = t; q < t + len; ++q) uo[row(q)] = id;
            for (int q = t; q < t + len; ++q)
                for (int64_t e = ptr[row(q)]; e < ptr[row(q) + 1]; ++e)
                    if (uo[col[e]] != id) l = std::max(l, lv[uo[col[e]]] + 1);
            lv.push_back(l);
            nlev = std::max(nlev, l + 1);
            t += len;
        }
        const double cost = nlev * (600.0 + 110.0 * cap);
        if (cap == 2 || cost < best) {
            best = cost;
            st.push_back(n);
            start.swap(st);
            unit_of.swap(uo);
            lev.swap(lv);
        }
    }
    const int nu = (int)lev.size();
    int nlev = 0;
    for (int l : lev) nlev = std::max(nlev, l + 1);
    std::vector<int> pos(nu), order(nu), fill(nlev + 1, 0);
    for (int l : lev) fill[l + 1]++;
    for (int l = 0; l < nlev; ++l) fill[l + 1] += fill[l];
    for (int q = 0; q < nu; ++q) {
        pos[q] = fill[lev[q]]++;
        order[pos[q]] = q;
    }
    // every row's entries in the order in which their columns become ready: the
    // units in order hand themselves to the rows that use them (transposed lists)
    const int64_t nz = ptr[n];
    std::vector<int> erow(nz), tp(n + 1, 0), te(nz), sorted(nz);
    for (int i = 0; i < n; ++i)
        for (int64_t e = ptr[i]; e < ptr[i + 1]; ++e) {
            erow[e] = i;
            tp[col[e] + 1]++;
        }
    for (int i = 0; i < n; ++i) tp[i + 1] += tp[i];
    {
        std::vector<int> f(tp.begin(), tp.end() - 1);
        for (int64_t e = 0; e < nz; ++e) te[f[col[e]]++] = (int)e;
    }
    std::vector<int64_t> next(ptr.begin(), ptr.end() - 1);
    for (int p = 0; p < nu; ++p)
        for (int t = start[order[p]]; t < start[order[p] + 1]; ++t)
            for (int k = tp[row(t)]; k < tp[row(t) + 1]; ++k) {
                const int e = te[k];
                if (unit_of[erow[e]] != order[p]) sorted[next[erow[e]]++] = e;
            }
    // slots: entry q of a row in lane q % 8 of the row's eight lanes, slot q / 8;
    // entries inside the unit go to its triangle
    S.unit.assign((size_t)nu * 4, 0);
    S.csrc.assign((size_t)nu * 16, -1);
    S.slot_col.clear();
    S.slot_src.clear();
    for (int p = 0; p < nu; ++p) {
        const int q = order[p], t0 = start[q], len = start[q + 1] - t0;
        int slots = 0;
        for (int g = 0; g < len; ++g) {
            const int i = row(t0 + g);
            slots = std::max<int>(slots, (int)((next[i] - ptr[i] + 7) / 8));
        }
        const size_t base = S.slot_col.size();
        S.unit[4 * (size_t)p] = t0;
        S.unit[4 * (size_t)p + 1] = len;
        S.unit[4 * (size_t)p + 2] = slots;
        S.unit[4 * (size_t)p + 3] = (int)(base / 32);
        S.slot_col.resize(base + 32 * (size_t)slots, -1);
        S.slot_src.resize(base + 32 * (size_t)slots, -1);
        for (int g = 0; g < len; ++g) {
            const int i = row(t0 + g);
            for (int64_t k = ptr[i]; k < next[i]; ++k) {
                const int o = (int)(k - ptr[i]);
                const size_t at = base + 32 * (size_t)(o / 8) + 8 * g + o % 8;
                S.slot_col[at] = col[sorted[k]];
                S.slot_src[at] = sorted[k];
            }
            for (int64_t e = ptr[i]; e < ptr[i + 1]; ++e)
                if (unit_of[col[e]] == q) {
                    const int j = (rev ? n - 1 - col[e] : col[e]) - t0;
                    S.csrc[16 * (size_t)p + 4 * g + j] = (int)e;
                }
        }
    }
    S.uploaded = false;
}

// Fills the values of one solve into its schedule and uploads it. unit_diag: the
// diagonal is an implied one.
int flow_upload(FlowSched &S, cudaStream_t s, bool rev, const std::vector<double> &val, const std::vector<double> &dg,
                bool unit_diag)
{
    const size_t nu = S.unit.size() / 4, ns = S.slot_col.size();
    std::vector<double> coef(nu * 16, 0.0), v(ns, 0.0);
    for (size_t p = 0; p < nu; ++p)
        for (int g = 0; g < S.unit[4 * p + 1]; ++g) {
            for (int j = 0; j < g; ++j) {
                const int e = S.csrc[16 * p + 4 * g + j];
                if (e >= 0) coef[16 * p + 4 * g + j] = val[e];
            }
            const int t = S.unit[4 * p] + g;
            coef[16 * p + 4 * g + 3] = unit_diag ? 1.0 : 1.0 / dg[rev ? S.n - 1 - t : t];
        }
    for (size_t k = 0; k < ns; ++k)
        if (S.slot_src[k] >= 0) v[k] = val[S.slot_src[k]];
    auto up = [&](auto &dst, const auto &src) -> int {
        using T = typename std::decay_t<decltype(src)>::value_type;
        OGB_CHECK(dst.alloc(src.empty() ? 1 : src.size()));
        if (!src.empty())
            OGB_CUDA(cudaMemcpyAsync(dst.p, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice, s));
        return OGB_OK;
    };
    if (!S.uploaded) {
        OGB_CHECK(up(S.d_unit, S.unit));
        OGB_CHECK(up(S.d_col, S.slot_col));
        S.uploaded = true;
    }
    OGB_CHECK(up(S.d_coef, coef));
    OGB_CHECK(up(S.d_val, v));
    OGB_CUDA(cudaStreamSynchronize(s));   // the host arrays are freed on return
    return OGB_OK;
}

}  // namespace

namespace {

// Device copy of a factor given by its forward / backward rows and diagonal.
int upload_factor(ogb_mtrx *m, int kind, const std::vector<int64_t> &fp, const std::vector<int> &fc,
                  const std::vector<double> &fv, const std::vector<int64_t> &bp, const std::vector<int> &bc,
                  const std::vector<double> &bv, const std::vector<double> &dg)
{
    IcFactor &F = m->ic;
    cudaStream_t s = m->ctx->stream;
    const int n = (int)dg.size();
    F.version = -1;
    flow_schedule(F.fwd, n, false, fp, fc);
    flow_schedule(F.bwd, n, true, bp, bc);
    OGB_CHECK(flow_upload(F.fwd, s, false, fv, dg, kind == 2));
    OGB_CHECK(flow_upload(F.bwd, s, true, bv, dg, false));
    OGB_CHECK(F.work.alloc(n > 0 ? n : 1));
    F.n = n;
    F.kind = kind;
    F.version = m->version;
    return OGB_OK;
}

// The matrix by rows on the host (npad rows, identity padding included).
int host_csr(ogb_mtrx *m, std::vector<int64_t> &rp, std::vector<int> &ci, std::vector<double> &va)
{
    cudaStream_t s = m->ctx->stream;
    const int n = m->npad;
    const int64_t ntot = m->nnz + (m->npad - m->neq);
    rp.resize(n + 1);
    ci.resize(ntot);
    va.resize(ntot);
    OGB_CUDA(cudaMemcpyAsync(rp.data(), m->rowptr.p, (n + 1) * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    OGB_CUDA(cudaMemcpyAsync(ci.data(), m->colind.p, ntot * sizeof(int), cudaMemcpyDeviceToHost, s));
    OGB_CUDA(cudaMemcpyAsync(va.data(), m->val.p, ntot * sizeof(double), cudaMemcpyDeviceToHost, s));
    OGB_CUDA(cudaStreamSynchronize(s));
    return OGB_OK;
}

int build_ilu(ogb_mtrx *m)
{
    std::vector<int64_t> rp;
    std::vector<int> ci;
    std::vector<double> va;
    OGB_CHECK(host_csr(m, rp, ci, va));
    const int n = m->npad;
    // column i of the (symmetric) matrix = row i: L takes rows > i, U rows <= i
    // (CompCol_ILUPreconditioner::initialize, iluprecond.C:75-130)
    std::vector<int> lp(n + 1, 0), up_(n + 1, 0);
    for (int i = 0; i < n; ++i) {
        int l = 0, u = 0;
        for (int64_t j = rp[i]; j < rp[i + 1]; ++j) (ci[j] > i ? l : u) += 1;
        lp[i + 1] = lp[i] + l;
        up_[i + 1] = up_[i] + u;
    }
    std::vector<int> lr(lp[n]), ur(up_[n]);
    std::vector<double> lv(lp[n]), uv(up_[n]);
    for (int i = 0; i < n; ++i) {
        int a = lp[i], b = up_[i];
        for (int64_t j = rp[i]; j < rp[i + 1]; ++j) {
            if (ci[j] > i) {
                lr[a] = ci[j];
                lv[a++] = va[j];
            } else {
                ur[b] = ci[j];
                uv[b++] = va[j];
            }
        }
        if (up_[i + 1] == up_[i] || ur[up_[i + 1] - 1] != i)
            return fail(OGB_E_ZERODIAG, "ILU preconditioner: diagonal not found");
    }
    // the factorization loop (iluprecond.C:134-167)
    for (int i = 0; i < n - 1; ++i) {
        double multiplier = uv[up_[i + 1] - 1];
        for (int j = lp[i]; j < lp[i + 1]; ++j) lv[j] /= multiplier;
        for (int j = up_[i + 1]; j < up_[i + 2] - 1; ++j) {
            multiplier = uv[j];
            int qn = j + 1, rn = lp[i + 1], pn;
            for (pn = lp[ur[j]]; pn < lp[ur[j] + 1] && lr[pn] <= i + 1; ++pn) {
                while (qn < up_[i + 2] && ur[qn] < lr[pn]) ++qn;
                if (qn < up_[i + 2] && lr[pn] == ur[qn]) uv[qn] -= multiplier * lv[pn];
            }
            for (; pn < lp[ur[j] + 1]; ++pn) {
                while (rn < lp[i + 2] && lr[rn] < lr[pn]) ++rn;
                if (rn < lp[i + 2] && lr[pn] == lr[rn]) lv[rn] -= multiplier * lv[pn];
            }
        }
    }
    // forward rows: (c, L_ic) from the columns c < i, c ascending
    std::vector<int64_t> fp(n + 1, 0);
    for (int c = 0; c < n; ++c)
        for (int t = lp[c]; t < lp[c + 1]; ++t) fp[lr[t] + 1]++;
    for (int i = 0; i < n; ++i) fp[i + 1] += fp[i];
    std::vector<int> fc(fp[n]);
    std::vector<double> fv(fp[n]);
    {
        std::vector<int64_t> fill(fp.begin(), fp.end() - 1);
        for (int c = 0; c < n; ++c)
            for (int t = lp[c]; t < lp[c + 1]; ++t) {
                const int64_t e = fill[lr[t]]++;
                fc[e] = c;
                fv[e] = lv[t];
            }
    }
    // backward rows: (c, U_rc) from the columns c > r, c descending; the diagonal
    std::vector<int64_t> bp(n + 1, 0);
    for (int c = 0; c < n; ++c)
        for (int t = up_[c]; t < up_[c + 1] - 1; ++t) bp[ur[t] + 1]++;
    for (int i = 0; i < n; ++i) bp[i + 1] += bp[i];
    std::vector<int> bc(bp[n]);
    std::vector<double> bv(bp[n]), dg(n);
    {
        std::vector<int64_t> fill(bp.begin(), bp.end() - 1);
        for (int c = n - 1; c >= 0; --c) {
            dg[c] = uv[up_[c + 1] - 1];
            for (int t = up_[c]; t < up_[c + 1] - 1; ++t) {
                const int64_t e = fill[ur[t]]++;
                bc[e] = c;
                bv[e] = uv[t];
            }
        }
    }
    return upload_factor(m, 2, fp, fc, fv, bp, bc, bv, dg);
}

}  // namespace

int build_ic(ogb_mtrx *m)
{
    IcFactor &F = m->ic;
    if (F.version == m->version && F.kind == m->precond) return OGB_OK;
    if (m->precond == 2) return build_ilu(m);
    const int n = m->npad;
    std::vector<int64_t> rp;
    std::vector<int> ci;
    std::vector<double> va;
    OGB_CHECK(host_csr(m, rp, ci, va));
    // lower triangle by columns (CompCol_ICPreconditioner::initialize, icprecond.C:64-107)
    std::vector<int> pntr(n + 1, 0);
    for (int k = 0; k < n; ++k) {
        int c = 0;
        for (int64_t j = rp[k]; j < rp[k + 1]; ++j) c += ci[j] >= k;
        pntr[k + 1] = pntr[k] + c;
    }
    const int nz = pntr[n];
    std::vector<int> indx(nz);
    std::vector<double> val(nz);
    for (int k = 0; k < n; ++k) {
        int t = pntr[k];
        for (int64_t j = rp[k]; j < rp[k + 1]; ++j)
            if (ci[j] >= k) {
                indx[t] = ci[j];
                val[t] = va[j];
                ++t;
            }
        if (pntr[k] == pntr[k + 1] || indx[pntr[k]] != k) return fail(OGB_E_ZERODIAG, "IC preconditioner: diagonal not found");
    }
    // ICFactor (icprecond.C:133-163), the same loop nest. indx gets one sentinel
    // entry: the successor test of the last entry of the last column reads one
    // past the end there.
    indx.push_back(n);
    for (int k = 0; k < n - 1; ++k) {
        const int d = pntr[k];
        const double z = val[d] = sqrt(val[d]);
        for (int i = d + 1; i < pntr[k + 1]; ++i) val[i] /= z;
        for (int i = d + 1; i < pntr[k + 1]; ++i) {
            const double zi = val[i];
            const int h = indx[i];
            int g = i;
            for (int j = pntr[h]; j < pntr[h + 1]; ++j)
                for (; g < pntr[k + 1] && indx[g + 1] <= indx[j]; ++g)
                    if (indx[g] == indx[j]) val[j] -= zi * val[g];
        }
    }
    if (n > 0) val[pntr[n - 1]] = sqrt(val[pntr[n - 1]]);
    indx.pop_back();
    // forward rows: entries (c, L_ic) from the columns c < i, c ascending
    std::vector<int64_t> fp(n + 1, 0);
    for (int c = 0; c < n; ++c)
        for (int t = pntr[c] + 1; t < pntr[c + 1]; ++t) fp[indx[t] + 1]++;
    for (int i = 0; i < n; ++i) fp[i + 1] += fp[i];
    std::vector<int> fc(fp[n]);
    std::vector<double> fv(fp[n]);
    {
        std::vector<int64_t> fill(fp.begin(), fp.end() - 1);
        for (int c = 0; c < n; ++c)
            for (int t = pntr[c] + 1; t < pntr[c + 1]; ++t) {
                const int64_t e = fill[indx[t]]++;
                fc[e] = c;
                fv[e] = val[t];
            }
    }
    // backward rows: row i's own column below the diagonal, rows ascending
    std::vector<int64_t> bp(n + 1, 0);
    for (int i = 0; i < n; ++i) bp[i + 1] = bp[i] + (pntr[i + 1] - pntr[i] - 1);
    std::vector<int> bc(bp[n]);
    std::vector<double> bv(bp[n]), dg(n);
    for (int i = 0; i < n; ++i) {
        dg[i] = val[pntr[i]];
        for (int t = pntr[i] + 1; t < pntr[i + 1]; ++t) {
            bc[bp[i] + (t - pntr[i] - 1)] = indx[t];
            bv[bp[i] + (t - pntr[i] - 1)] = val[t];
        }
    }
    return upload_factor(m, 4, fp, fc, fv, bp, bc, bv, dg);
}

// z = M^-1 r and, with sc, r.z -> rho and beta (see k_tri_flow). The cluster is 16
// CTAs where the device takes that size, else 8.
int launch_ic_solve(ogb_mtrx *m, const double *r, double *z, PcgScal *sc)
{
    IcFactor &F = m->ic;
    cudaStream_t s = m->ctx->stream;
    const bool local = F.n <= FLOW_LOCAL_MAX;
    const void *fn = local ? (const void *)k_tri_flow<true> : (const void *)k_tri_flow<false>;
    const size_t smem = local ? (size_t)F.n * sizeof(double) : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(FLOW_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (!F.cluster || F.cluster_local != local) {
        OGB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        if (local)
            OGB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          FLOW_LOCAL_MAX * (int)sizeof(double)));
        int fits = 0;
        cfg.gridDim = dim3(16);
        cfg.dynamicSmemBytes = local ? FLOW_LOCAL_MAX * sizeof(double) : 0;
        attr[0].val.clusterDim.x = 16;
        if (cudaOccupancyMaxActiveClusters(&fits, fn, &cfg) != cudaSuccess) {
            cudaGetLastError();
            fits = 0;
        }
        F.cluster = fits > 0 ? 16 : 8;
        F.cluster_local = local;
        cfg.dynamicSmemBytes = smem;
    }
    cfg.gridDim = dim3(F.cluster);
    attr[0].val.clusterDim.x = F.cluster;
    if (!local) {   // the vectors start as FLOW_EMPTY
        OGB_CUDA(cudaMemsetAsync(F.work.p, 0xff, (size_t)F.n * sizeof(double), s));
        OGB_CUDA(cudaMemsetAsync(z, 0xff, (size_t)F.n * sizeof(double), s));
    }
    auto view = [](const FlowSched &S) {
        return FlowView{(int)(S.unit.size() / 4), reinterpret_cast<const int4 *>(S.d_unit.p), S.d_coef.p, S.d_col.p, S.d_val.p};
    };
    const FlowView fv = view(F.fwd), bv = view(F.bwd);
    int *status = m->ctx->status.p;
    if (local) OGB_CUDA(cudaLaunchKernelEx(&cfg, k_tri_flow<true>, F.n, fv, bv, r, F.work.p, z, sc, status));
    else OGB_CUDA(cudaLaunchKernelEx(&cfg, k_tri_flow<false>, F.n, fv, bv, r, F.work.p, z, sc, status));
    count_launch(m->ctx);
    OGB_CUDA(cudaGetLastError());
    return OGB_OK;
}

}  // namespace ogb
