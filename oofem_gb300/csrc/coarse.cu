// Coarse part of the mixed solve's preconditioner: z = B^-1 r + W Ac^-1 W^T r.
//
// Block Jacobi alone leaves CG to carry the smooth, nearly rigid motions of a mesh
// through it one element per iteration (about eleven iterations per element of a
// cantilever's length). The active nodes are therefore grouped into boxes, W spans
// the rigid motions of each box (translations and rotations about its centre, zero on
// prescribed DOFs), and Ac = W^T K64 W, a few hundred equations, is inverted once per
// matrix version. The sum of the two corrections is symmetric and positive definite
// like each of them, so CG, the FP64 residual replacements and the convergence test
// on the FP64 residual stay as they are; only the search directions are better.
// Iterations without -> with it, and the solve with set-up (GB300): 290 x 58 x 58 hexes
// to 1e-8 3,300 -> 350, 660 -> 112 ms; 101 x 21 x 19 to 1e-9 1,760 -> 150, 31 (one launch)
// -> 9.6 ms; 40^3-cell tets to 1e-11 710 -> 140, 24.6 -> 11.5 ms.
//
// Everything is deterministic: Ac is summed in 64-bit integers (fixed point scaled by
// K's largest diagonal entry), so the order of the atomic additions does not matter;
// W^T r is summed per box in a fixed order.
#include <math.h>

#include <algorithm>

#include "internal.cuh"
#include "reduce.cuh"

namespace ogb {

namespace {

constexpr int GJ = 32;             // block of the inversion
constexpr double COARSE_SOFTEST = 3e-7;
constexpr int AC_BITS = 42;        // fixed point of Ac: 2^42 per largest diagonal entry of K (2^18 terms an entry fit)

template <int ND>
struct Modes {
    static constexpr int NM = ND == 3 ? 6 : 3;
};

// Rows of W for a node: w[d][m] is motion m at DOF d; x the node's position in its
// box (scaled), free DOFs in `mask`.
template <int ND, class R>
__device__ __forceinline__ void rigid(const R (&x)[ND], int mask, R (&w)[ND][Modes<ND>::NM])
{
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
        for (int m = 0; m < Modes<ND>::NM; ++m) w[d][m] = 0;
#pragma unroll
    for (int d = 0; d < ND; ++d) w[d][d] = 1;
    if constexpr (ND == 3) {
        w[1][3] = -x[2]; w[2][3] = x[1];
        w[0][4] = -x[2]; w[2][4] = x[0];
        w[0][5] = -x[1]; w[1][5] = x[0];
    } else {
        w[0][2] = -x[1]; w[1][2] = x[0];
    }
#pragma unroll
    for (int d = 0; d < ND; ++d)
        if (!(mask >> d & 1))
#pragma unroll
            for (int m = 0; m < Modes<ND>::NM; ++m) w[d][m] = 0;
}

template <int ND>
__device__ __forceinline__ void load_rel(const float *__restrict__ rel, int64_t n, int64_t a, float (&x)[ND])
{
#pragma unroll
    for (int d = 0; d < ND; ++d) x[d] = rel[d * n + a];
}

// Largest diagonal entry of K (as the bits of a positive double).
template <int ND>
__global__ void k_max_diag(int nact, const int64_t *__restrict__ diag, const double *__restrict__ val, unsigned long long *out)
{
    double v = 0.0;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nact; a += gridDim.x * blockDim.x) {
        const int64_t slot = diag[a];
        const int r = (int)(slot & 31);
        const double *vb = val + (slot - r) * (ND * ND) + r;
#pragma unroll
        for (int d = 0; d < ND; ++d) v = fmax(v, fabs(vb[32 * (d * ND + d)]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(v));
}

// Rows that add to Ac: a row whose neighbours all lie in its own box with all DOFs
// free adds nothing (K times a rigid motion is zero there). About a fifth of a large
// mesh is left; the list of them keeps warps full of rows that have work.
__global__ void k_coarse_need(int nact, const int64_t *__restrict__ sl_ptr, const int *__restrict__ sl_width,
                              const int *__restrict__ col, const int *__restrict__ box, const int *__restrict__ mask, int full,
                              int64_t *__restrict__ flag)
{
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a > nact) return;
    bool need = false;
    if (a < nact) {
        const int s = a >> 5, r = a & 31, w = sl_width[s], I = box[a];
        const int64_t base = sl_ptr[s];
        for (int k = 0; k < w && !need; ++k) {
            const int B = col[base + 32 * k + r];
            need = box[B] != I || mask[B] != full;
        }
    }
    flag[a] = need ? 1 : 0;
}

__global__ void k_coarse_list(int nact, const int64_t *__restrict__ pos, int *__restrict__ list)
{
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a < nact && pos[a + 1] > pos[a]) list[pos[a]] = a;
}

// Ac += W_a^T K_aB W_B over the blocks of row a, a thread per listed row. The blocks
// are taken box by box (a row meets few), so a box pair costs one product with W_a^T
// and one round of atomic additions. The translations of W need no arithmetic, the
// rotations two terms per entry.
template <int ND>
__global__ void __launch_bounds__(128) k_coarse_matrix(int nlist, const int *__restrict__ list, const int64_t *__restrict__ sl_ptr,
                                                       const int *__restrict__ sl_width, const int *__restrict__ col,
                                                       const double *__restrict__ val, const int *__restrict__ box,
                                                       const float *__restrict__ rel, const int *__restrict__ mask,
                                                       int64_t nrows, int nc, const unsigned long long *__restrict__ maxd,
                                                       unsigned long long *A)
{
    constexpr int NM = Modes<ND>::NM;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nlist) return;
    const int a = list[t], s = a >> 5, r = a & 31, w = sl_width[s], I = box[a];
    const int64_t base = sl_ptr[s];
    const double scale = ldexp(1.0, AC_BITS) / __longlong_as_double((long long)*maxd);
    float xf[ND];
    double wa[ND][NM];
    load_rel<ND>(rel, nrows, a, xf);
    {
        double xa[ND];
#pragma unroll
        for (int d = 0; d < ND; ++d) xa[d] = xf[d];
        rigid<ND, double>(xa, mask[a], wa);
    }
    int J = I;   // own box first, then the others in increasing order
    for (;;) {
        double T[ND][NM];
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int m = 0; m < NM; ++m) T[d][m] = 0.0;
        int next = 0x7fffffff;
        for (int k = 0; k < w; ++k) {
            const int B = col[base + 32 * k + r], q = box[B];
            if (q != J) {
                if (q != I && (J == I || q > J)) next = min(next, q);
                continue;
            }
            const double *vk = val + (base + 32 * (int64_t)k) * (ND * ND) + r;
            load_rel<ND>(rel, nrows, B, xf);
            const int mb = mask[B];
            double xb[ND];
#pragma unroll
            for (int d = 0; d < ND; ++d) xb[d] = xf[d];
#pragma unroll
            for (int i = 0; i < ND; ++i) {
                double K[ND];
#pragma unroll
                for (int j = 0; j < ND; ++j) {
                    K[j] = (mb >> j & 1) ? vk[32 * (i * ND + j)] : 0.0;
                    T[i][j] += K[j];
                }
                if constexpr (ND == 3) {
                    T[i][3] += K[2] * xb[1] - K[1] * xb[2];
                    T[i][4] += K[2] * xb[0] - K[0] * xb[2];
                    T[i][5] += K[1] * xb[0] - K[0] * xb[1];
                } else {
                    T[i][2] += K[1] * xb[0] - K[0] * xb[1];
                }
            }
        }
#pragma unroll
        for (int m = 0; m < NM; ++m)
#pragma unroll
            for (int n = 0; n < NM; ++n) {
                double c = 0.0;
                if (m < ND) {
                    c = wa[m < ND ? m : 0][m] * T[m < ND ? m : 0][n];
                } else {
#pragma unroll
                    for (int d = 0; d < ND; ++d) c = fma(wa[d][m], T[d][n], c);
                }
                const long long f = __double2ll_rn(c * scale);
                if (f) atomicAdd(A + (size_t)(I * NM + m) * nc + J * NM + n, (unsigned long long)f);
            }
        if (next == 0x7fffffff) break;
        J = next;
    }
}

// Ac in FP64 on whole blocks of GJ, symmetric; motions no DOF takes part in (a box of
// one node has no rotations) get a unit diagonal, and a shift of 1e-8 keeps boxes
// with dependent motions (nodes on a line) positive definite.
__global__ void k_coarse_convert(int nc, int ncp, const long long *__restrict__ F, const unsigned long long *__restrict__ maxd,
                                 double *__restrict__ A)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)ncp * ncp) return;
    const int i = (int)(t / ncp), j = (int)(t % ncp);
    double v = i == j ? 1.0 : 0.0;
    if (i < nc && j < nc) {
        const double unit = __longlong_as_double((long long)*maxd) * ldexp(1.0, -AC_BITS);
        v = 0.5 * ((double)F[(size_t)i * nc + j] + (double)F[(size_t)j * nc + i]) * unit;
        if (i == j) v = v > 0.0 ? v * (1.0 + 1e-8) : 1.0;
    }
    A[t] = v;
}

// Block Gauss-Jordan inversion, step k: D = inverse of the diagonal block (one CTA),
// then every tile of the next iterate from this one:
//   (k, k): D;  (k, j): D A_kj;  (i, k): -A_ik D;  (i, j): A_ij - A_ik D A_kj.
// In the diagonal step a warp holds rows warp + 8 q and the pivot's owner publishes its
// scaled row, as in the direct solver's diagonal block (with a division in each of 32
// warps the step took 76 us).
__global__ void __launch_bounds__(NTHREADS) k_gj_diag(int n, int k, const double *__restrict__ A, double *__restrict__ D)
{
    __shared__ double W[2][GJ];
    const int c = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double e[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) e[q] = A[(size_t)(k * GJ + warp + 8 * q) * n + k * GJ + c];
    auto publish = [&](int p, double &row) {   // row p's warp: the row becomes its part of the inverse
        const double d = 1.0 / __shfl_sync(0xffffffffu, row, p);
        row = c == p ? d : row * d;
        W[p & 1][c] = row;
    };
    if (warp == 0) publish(0, e[0]);
#pragma unroll
    for (int pq = 0; pq < 4; ++pq)
#pragma unroll 1
        for (int pw = 0; pw < 8; ++pw) {
            const int p = pw + 8 * pq;
            __syncthreads();
            const double w = W[p & 1][c];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int q = (h + (pw == 7 ? pq + 1 : pq)) & 3, r = warp + 8 * q;   // the next pivot's row first
                if (r == p) continue;
                const double f = __shfl_sync(0xffffffffu, e[q], p);
                e[q] = fma(-f, w, c == p ? 0.0 : e[q]);
                if (r == p + 1) publish(r, e[q]);
            }
        }
#pragma unroll
    for (int q = 0; q < 4; ++q) D[(warp + 8 * q) * GJ + c] = e[q];
}

__global__ void __launch_bounds__(NTHREADS) k_gj_update(int n, int k, const double *__restrict__ A, const double *__restrict__ D,
                                                        double *__restrict__ B)
{
    __shared__ double L[GJ][GJ + 1], R[GJ][GJ + 1], M[GJ][GJ + 1];
    const int i = blockIdx.y, j = blockIdx.x, c = threadIdx.x & 31, r0 = threadIdx.x >> 5;
    for (int r = r0; r < GJ; r += 8) {
        M[r][c] = D[r * GJ + c];
        if (i != k) L[r][c] = A[(size_t)(i * GJ + r) * n + k * GJ + c];
        if (j != k) R[r][c] = A[(size_t)(k * GJ + r) * n + j * GJ + c];
    }
    __syncthreads();
    double p[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) p[q] = 0.0;
    if (j != k) {   // D A_kj
#pragma unroll 8
        for (int e = 0; e < GJ; ++e)
#pragma unroll
            for (int q = 0; q < 4; ++q) p[q] = fma(M[r0 + 8 * q][e], R[e][c], p[q]);
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) p[q] = M[r0 + 8 * q][c];
    }
    if (i != k) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            M[r0 + 8 * q][c] = p[q];
            p[q] = j != k ? A[(size_t)(i * GJ + r0 + 8 * q) * n + j * GJ + c] : 0.0;
        }
        __syncthreads();
#pragma unroll 8
        for (int e = 0; e < GJ; ++e)
#pragma unroll
            for (int q = 0; q < 4; ++q) p[q] = fma(-L[r0 + 8 * q][e], M[e][c], p[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) B[(size_t)(i * GJ + r0 + 8 * q) * n + j * GJ + c] = p[q];
}

// Partial sums of W^T r: CTA u sums the rows list[first .. last) of one box; a
// thread's terms in FP32 (a dozen rows), FP64 from there.
template <int ND>
__global__ void __launch_bounds__(NTHREADS) k_coarse_restrict(const int *__restrict__ part, const int *__restrict__ list,
                                                              const float *__restrict__ rel, const int *__restrict__ mask,
                                                              int64_t nrows, const float *__restrict__ r,
                                                              double *__restrict__ out, const PcgScal *sc, int always)
{
    if (!always && (sc->done || sc->reliable)) return;
    constexpr int NM = Modes<ND>::NM;
    const int lo = part[blockIdx.x], hi = part[blockIdx.x + 1];
    float v[NM];
#pragma unroll
    for (int m = 0; m < NM; ++m) v[m] = 0.f;
#pragma unroll 3
    for (int k = lo + threadIdx.x; k < hi; k += NTHREADS) {
        const int64_t a = list[k];
        float x[ND], w[ND][NM];
        load_rel<ND>(rel, nrows, a, x);
        rigid<ND, float>(x, mask[a], w);
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const float rd = r[a * ND + d];
#pragma unroll
            for (int m = 0; m < NM; ++m) v[m] = fmaf(w[d][m], rd, v[m]);
        }
    }
    double s[NM];
    block_sum_t<NM, float>(v, s);
    if (threadIdx.x == 0)
#pragma unroll
        for (int m = 0; m < NM; ++m) out[(size_t)blockIdx.x * NM + m] = s[m];
}

// c = Ac^-1 w, a warp per row (w = the parts of each box added in order), w.c, and in
// the last block the scalars of the iteration: r.z = r.z1 + w.c (r.z1, of the block
// Jacobi part, is in sc->rho_old), then as finish_update32 / finish_replace.
__global__ void __launch_bounds__(NTHREADS) k_coarse_solve(int nc, int ncp, int nm, const int *__restrict__ box_part,
                                                           const double *__restrict__ parts, const double *__restrict__ inv,
                                                           double *__restrict__ c, double *part, unsigned int *count,
                                                           PcgScal *sc, int maxit, int replace, int first)
{
    if (!replace && (sc->done || sc->reliable)) return;
    extern __shared__ double w[];
    for (int i = threadIdx.x; i < ncp; i += NTHREADS) {
        double s = 0.0;
        if (i < nc) {
            const int b = i / nm, m = i % nm;
            for (int u = box_part[b]; u < box_part[b + 1]; ++u) s += parts[(size_t)u * nm + m];
        }
        w[i] = s;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, row = blockIdx.x * (NTHREADS / 32) + (threadIdx.x >> 5);
    double v[1] = {0.0};
    if (row < nc) {
        const double *q = inv + (size_t)row * ncp;
        double s = 0.0;
#pragma unroll 12
        for (int j = lane; j < ncp; j += 32) s = fma(__ldg(q + j), w[j], s);
        s = warp_sum(s);
        if (lane == 0) {
            c[row] = s;
            v[0] = s * w[row];
        }
    }
    block_sum<1>(v);
    if (!publish_partials<1>(v, part, count)) return;
    double t[1];
    final_sums<1>(part, t);
    if (threadIdx.x != 0) return;
    *count = 0;
    const double rz = sc->rho_old + t[0];
    if (replace) {
        if (!isfinite(rz) || !(rz > 0.0)) {
            sc->done = 2;
        } else {
            sc->beta = first ? 0.0 : rz / sc->rho;
            sc->zcoef = 1.0;
            sc->rho = rz;
        }
        return;
    }
    const double rr = sc->rnorm2;
    sc->iters += 1;
    if (!isfinite(rr) || !isfinite(rz)) {
        sc->done = 2;
    } else if (rr <= sc->drop2 * sc->rmax2 || rr <= sc->tol2 || !(rz > 0.0) || sc->iters >= maxit || sc->iters >= sc->cycle_end) {
        sc->reliable = 1;
    } else {
        sc->beta = rz / sc->rho;
        sc->rho = rz;
        sc->zcoef = 1.0;
    }
}

// p = z + W c + beta p.
template <int ND>
__global__ void __launch_bounds__(NTHREADS) k_coarse_pupdate(int64_t nact, const float *__restrict__ z, float *__restrict__ p,
                                                             const int *__restrict__ box, const float *__restrict__ rel,
                                                             const int *__restrict__ mask, int64_t nrows,
                                                             const double *__restrict__ c, const PcgScal *sc)
{
    if (sc->done || sc->reliable) return;
    constexpr int NM = Modes<ND>::NM;
    const float beta = (float)sc->beta;
    for (int64_t a = (int64_t)blockIdx.x * NTHREADS + threadIdx.x; a < nact; a += (int64_t)gridDim.x * NTHREADS) {
        float x[ND], w[ND][NM], cc[NM];
        load_rel<ND>(rel, nrows, a, x);
        rigid<ND, float>(x, mask[a], w);
        const double *q = c + (size_t)box[a] * NM;
#pragma unroll
        for (int m = 0; m < NM; ++m) cc[m] = (float)__ldg(q + m);
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            float zz = z[a * ND + d];
#pragma unroll
            for (int m = 0; m < NM; ++m) zz = fmaf(w[d][m], cc[m], zz);
            p[a * ND + d] = fmaf(beta, p[a * ND + d], zz);
        }
    }
}

}  // namespace

// From COARSE_MIN_NODES active nodes on: below, the one-launch iterations without it are
// as fast (17^3-cell tets, 5.8 k nodes: 4.9 ms with it, about 4.5 ms in one launch;
// 40 x 11 x 9 hexes, 4.9 k nodes: 4.8 against about 9 ms).
bool coarse_wanted(const ogb_ctx *ctx, const SellMat &S)
{
    return ctx->persist && S.ninst == 1 && S.nact >= COARSE_MIN_NODES && S.xyz.p != nullptr;
}

// Boxes of the active nodes (host, once per structure): equal boxes of the bounding
// box. More boxes mean fewer iterations (they follow the box's width in elements) and
// a larger Ac, whose inversion takes 0.4 ms for 288 equations and 4 ms for 1,200; whole
// solves, ms, at one box per 5,000 / 600 / 300 nodes: 129 k DOFs 11.9 / 9.6 / 11.2, 1.2 M
// DOFs 71 / 51 / 70 (caps 160 / 200 / 320), quads 200 x 200 22.5 / 20.9 / 14.0.
static int build_boxes(ogb_ctx *ctx, SellMat &S)
{
    Coarse &C = S.coarse;
    cudaStream_t s = ctx->stream;
    const int n = S.nact, nd = S.nd;
    const int64_t nrows = (int64_t)S.nslices * 32;
    C.tried = true;
    C.ok = false;
    std::vector<double> x((size_t)nd * nrows);
    OGB_CUDA(cudaMemcpyAsync(x.data(), S.xyz.p, x.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
    OGB_CUDA(cudaStreamSynchronize(s));
    double lo[3], len[3], vol = 1.0;
    int dims = 0;
    for (int d = 0; d < nd; ++d) {
        const auto mm = std::minmax_element(x.begin() + d * nrows, x.begin() + d * nrows + n);
        lo[d] = *mm.first;
        len[d] = *mm.second - *mm.first;
        if (!(len[d] >= 0.0) || !std::isfinite(len[d])) return OGB_OK;
        if (len[d] > 0.0) {
            vol *= len[d];
            ++dims;
        }
    }
    if (dims == 0) return OGB_OK;
    // The smooth search directions that the coarse part brings must be resolved by the
    // FP32 operator: the softest one, bending of the whole mesh, has about
    // (h / L)^2 (width / L)^2 of the largest stiffness, which has to stand clear of the
    // FP32 rounding (6e-8). 160 x 5 x 5 hexes (4e-8) do not converge with it,
    // 290 x 58 x 58 (5e-7) do.
    double longest = 0.0, width = 0.0;
    for (int d = 0; d < nd; ++d) longest = std::max(longest, len[d]);
    width = longest;
    for (int d = 0; d < nd; ++d)
        if (len[d] > 0.0) width = std::min(width, len[d]);
    const double he = pow(vol / n, 1.0 / dims);
    if (pow(he / longest, 2) * pow(width / longest, 2) < COARSE_SOFTEST) return OGB_OK;
    const double want = nd == 3 ? std::min(200.0, std::max(48.0, n / 600.0)) : std::min(320.0, std::max(48.0, n / 125.0)), h = pow(vol / want, 1.0 / dims);
    int k[3] = {1, 1, 1};
    for (int d = 0; d < nd; ++d) k[d] = (int)std::min(256.0, std::max(1.0, std::round(len[d] / h)));
    const int64_t cells = (int64_t)k[0] * k[1] * k[2];
    if (cells > 2048) return OGB_OK;
    std::vector<int> cell(n), box(nrows, 0), id(cells, -1), count;
    for (int a = 0; a < n; ++a) {
        int q = 0;
        for (int d = nd - 1; d >= 0; --d) {
            const int i = len[d] > 0.0 ? std::min(k[d] - 1, (int)((x[d * nrows + a] - lo[d]) / len[d] * k[d])) : 0;
            q = q * k[d] + i;
        }
        cell[a] = q;
        if (id[q] < 0) {
            id[q] = (int)count.size();
            count.push_back(0);
        }
        box[a] = id[q];
        count[id[q]]++;
    }
    const int nb = (int)count.size();
    std::vector<double> cen((size_t)nb * nd, 0.0);
    for (int a = 0; a < n; ++a)
        for (int d = 0; d < nd; ++d) cen[(size_t)box[a] * nd + d] += x[d * nrows + a];
    std::vector<float> rel((size_t)nd * nrows, 0.f);
    for (int d = 0; d < nd; ++d)
        for (int a = 0; a < n; ++a)
            rel[d * nrows + a] = (float)((x[d * nrows + a] - cen[(size_t)box[a] * nd + d] / count[box[a]]) / h);
    // the boxes' rows, and CTAs of at most PART_ROWS of them
    constexpr int PART_ROWS = 1536;
    std::vector<int> start(nb + 1, 0), list(n), part, bp(nb + 1, 0);
    for (int i = 0; i < nb; ++i) start[i + 1] = start[i] + count[i];
    std::vector<int> fill(start.begin(), start.end() - 1);
    for (int a = 0; a < n; ++a) list[fill[box[a]]++] = a;
    for (int i = 0; i < nb; ++i) {
        bp[i] = (int)part.size();
        for (int q = start[i]; q < start[i + 1]; q += PART_ROWS) part.push_back(q);
    }
    bp[nb] = (int)part.size();
    C.nparts = (int)part.size();
    part.push_back(n);
    C.nm = nd == 3 ? 6 : 3;
    C.nc = nb * C.nm;
    C.ncp = (int)ceil_div(C.nc, GJ) * GJ;
    auto up = [&](auto &dst, const auto &src) -> int {
        OGB_CHECK(dst.alloc(src.size()));
        OGB_CUDA(cudaMemcpyAsync(dst.p, src.data(), src.size() * sizeof(src[0]), cudaMemcpyHostToDevice, s));
        return OGB_OK;
    };
    OGB_CHECK(up(C.box, box));
    OGB_CHECK(up(C.rel, rel));
    OGB_CHECK(up(C.list, list));
    OGB_CHECK(up(C.part, part));
    OGB_CHECK(up(C.box_part, bp));
    OGB_CUDA(cudaStreamSynchronize(s));
    OGB_CHECK(C.fixed.alloc((size_t)C.nc * C.nc));
    OGB_CHECK(C.maxd.alloc(1));
    OGB_CHECK(C.a.alloc((size_t)C.ncp * C.ncp));
    OGB_CHECK(C.b.alloc((size_t)C.ncp * C.ncp));
    OGB_CHECK(C.d.alloc(GJ * GJ));
    OGB_CHECK(C.parts.alloc((size_t)C.nparts * C.nm));
    OGB_CHECK(C.c.alloc(C.ncp));
    // the rows that add to Ac
    {
        DBuf<int64_t> flag;
        OGB_CHECK(flag.alloc(n + 1));
        OGB_CHECK(C.need.alloc(n));
        k_coarse_need<<<(unsigned)ceil_div(n + 1, 256), 256, 0, s>>>(n, S.sl_ptr.p, S.sl_width.p, S.col.p, C.box.p, S.free_mask.p,
                                                                    (1 << nd) - 1, flag.p);
        int64_t total = 0;
        OGB_CHECK(exclusive_scan_i64(ctx, flag.p, flag.p, n + 1, &total));
        k_coarse_list<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(n, flag.p, C.need.p);
        count_launch(ctx, 2);
        OGB_CUDA(cudaGetLastError());
        OGB_CUDA(cudaStreamSynchronize(s));   // flag is freed
        C.nlist = (int)total;
    }
    C.version = -1;
    C.ok = true;
    return OGB_OK;
}

// Boxes and Ac^-1 of the current FP64 values (S.coarse.ok false: not usable here).
int refresh_coarse(ogb_ctx *ctx, SellMat &S, int64_t version)
{
    Coarse &C = S.coarse;
    if (!C.tried) OGB_CHECK(build_boxes(ctx, S));
    if (!C.ok || C.version == version) return OGB_OK;
    cudaStream_t s = ctx->stream;
    const int64_t nrows = (int64_t)S.nslices * 32;
    OGB_CUDA(cudaMemsetAsync(C.fixed.p, 0, (size_t)C.nc * C.nc * sizeof(long long), s));
    OGB_CUDA(cudaMemsetAsync(C.maxd.p, 0, sizeof(unsigned long long), s));
    const unsigned g = (unsigned)ceil_div(C.nlist > 0 ? C.nlist : 1, 128);
    unsigned long long *F = reinterpret_cast<unsigned long long *>(C.fixed.p);
    if (S.nd == 3) {
        k_max_diag<3><<<num_sms() * 2, 256, 0, s>>>(S.nact, S.diag.p, S.v64.p, C.maxd.p);
        k_coarse_matrix<3><<<g, 128, 0, s>>>(C.nlist, C.need.p, S.sl_ptr.p, S.sl_width.p, S.col.p, S.v64.p, C.box.p, C.rel.p, S.free_mask.p,
                                             nrows, C.nc, C.maxd.p, F);
    } else {
        k_max_diag<2><<<num_sms() * 2, 256, 0, s>>>(S.nact, S.diag.p, S.v64.p, C.maxd.p);
        k_coarse_matrix<2><<<g, 128, 0, s>>>(C.nlist, C.need.p, S.sl_ptr.p, S.sl_width.p, S.col.p, S.v64.p, C.box.p, C.rel.p, S.free_mask.p,
                                             nrows, C.nc, C.maxd.p, F);
    }
    const int64_t nn = (int64_t)C.ncp * C.ncp;
    k_coarse_convert<<<(unsigned)ceil_div(nn, 256), 256, 0, s>>>(C.nc, C.ncp, C.fixed.p, C.maxd.p, C.a.p);
    double *A = C.a.p, *B = C.b.p;
    const int nb = C.ncp / GJ;
    for (int k = 0; k < nb; ++k) {
        k_gj_diag<<<1, NTHREADS, 0, s>>>(C.ncp, k, A, C.d.p);
        k_gj_update<<<dim3(nb, nb), NTHREADS, 0, s>>>(C.ncp, k, A, C.d.p, B);
        std::swap(A, B);
    }
    C.inv = A;
    count_launch(ctx, 3 + 2 * nb);
    OGB_CUDA(cudaGetLastError());
    C.version = version;
    return OGB_OK;
}

// After the update (replace 0) or a residual replacement (1): c = Ac^-1 W^T r, the
// iteration's scalars, p = z + W c + beta p.
int launch_coarse(ogb_ctx *ctx, SellMat &S, const float *r, const float *z, float *p, double *part, unsigned int *count,
                  PcgScal *sc, int maxit, int replace, int first)
{
    Coarse &C = S.coarse;
    cudaStream_t s = ctx->stream;
    const int64_t nrows = (int64_t)S.nslices * 32;
    const int g = (int)ceil_div(C.nc, NTHREADS / 32), gp = (int)std::min<int64_t>(ceil_div(S.nact, NTHREADS), (int64_t)num_sms() * 8);
    if (S.nd == 3) k_coarse_restrict<3><<<C.nparts, NTHREADS, 0, s>>>(C.part.p, C.list.p, C.rel.p, S.free_mask.p, nrows, r, C.parts.p, sc, replace);
    else k_coarse_restrict<2><<<C.nparts, NTHREADS, 0, s>>>(C.part.p, C.list.p, C.rel.p, S.free_mask.p, nrows, r, C.parts.p, sc, replace);
    k_coarse_solve<<<g, NTHREADS, C.ncp * sizeof(double), s>>>(C.nc, C.ncp, C.nm, C.box_part.p, C.parts.p, C.inv, C.c.p, part, count, sc,
                                                               maxit, replace, first);
    if (S.nd == 3) k_coarse_pupdate<3><<<gp, NTHREADS, 0, s>>>(S.nact, z, p, C.box.p, C.rel.p, S.free_mask.p, nrows, C.c.p, sc);
    else k_coarse_pupdate<2><<<gp, NTHREADS, 0, s>>>(S.nact, z, p, C.box.p, C.rel.p, S.free_mask.p, nrows, C.c.p, sc);
    count_launch(ctx, 3);
    return OGB_OK;
}

}  // namespace ogb
