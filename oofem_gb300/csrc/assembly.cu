// Deterministic assembly by gathering (K4 matrix, K5 vector).
//
// The reference scatters element matrices into the global matrix inside an
// OpenMP critical section (EngngModel::assemble engngm.C:889-1037 ->
// CompCol::assemble compcol.C:275-316). Here every node block (A,B) of the
// pattern owns the list of (element, a, b) contributions in ascending element
// order, so one thread sums an entry in the same order as the serial
// reference loop: no floating-point atomics, bitwise reproducible.
#include "internal.cuh"

namespace ogb {

namespace {

// The CSR values and the node-block SELL copy (FP64 and FP32: every entry of the
// ND x ND block, with prescribed rows/columns zero and an identity diagonal for
// prescribed DOFs of active nodes) in the order of the copy's slots, a thread per entry
// of a block, SLOT_GROUPS x 32 slots per CTA. Bound by the sectors that pass L1 and
// L2: the entries of a block's contribution are read by consecutive lanes, and the copy,
// whose planes hold one entry of 32 rows, is written through shared memory in whole lines
// (a thread per block read 72-byte pieces and wrote single values 2,304 bytes apart:
// 398 us for 138 k hexes, 102 x 38 x 38 nodes; this: 201 us). The four groups'
// chains list -> element value run side by side in a thread.
constexpr int SLOT_GROUPS = 4;
template <int ND>
__global__ void __launch_bounds__(32 * ND * ND) k_gather_slots(
    int64_t nslots, int nnpe, const int *__restrict__ slot_blk, const int *__restrict__ blk_node,
    const int *__restrict__ nb_col, const int *__restrict__ nb_coloff, const int64_t *__restrict__ cb_ptr,
    const uint32_t *__restrict__ cb, const int *__restrict__ eq, const double *__restrict__ ke,
    const int64_t *__restrict__ rowptr, double *__restrict__ val, double *__restrict__ v64, float *__restrict__ v32)
{
    constexpr int E = ND * ND, SLOTS = 32 * SLOT_GROUPS;
    __shared__ int64_t first[SLOTS], rowpos[ND][SLOTS];   // rowpos: CSR position of the block's row, -1: prescribed
    __shared__ int count[SLOTS], free_cols[SLOTS];        // free_cols: -1: no block; bit ND: diagonal block
    __shared__ double st[E][33];
    const int t = threadIdx.x;
    const int64_t s0 = (int64_t)blockIdx.x * SLOTS;
    for (int h = t; h < SLOTS; h += 32 * E) {
        const int k = s0 + h < nslots ? slot_blk[s0 + h] : -1;
        int64_t c0 = 0;
        int n = 0, mask = -1;
        if (k >= 0) {
            const int A = blk_node[k], B = nb_col[k], off = nb_coloff[k];
            c0 = cb_ptr[k];
            n = (int)(cb_ptr[k + 1] - c0);
            mask = A == B ? 1 << ND : 0;
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                const int ra = eq[(size_t)A * ND + d];
                rowpos[d][h] = ra > 0 ? rowptr[ra - 1] + off : -1;
                if (eq[(size_t)B * ND + d] > 0) mask |= 1 << d;
            }
        }
        first[h] = c0;
        count[h] = n;
        free_cols[h] = mask;
    }
    __syncthreads();
    const int b = t / E, en = t % E, i = en / ND, j = en % ND;
    double s[SLOT_GROUPS];
    int n = 0;
#pragma unroll
    for (int q = 0; q < SLOT_GROUPS; ++q) {
        s[q] = 0.0;
        n = max(n, count[32 * q + b]);
    }
    for (int c = 0; c < n; ++c)
#pragma unroll
        for (int q = 0; q < SLOT_GROUPS; ++q)
            if (c < count[32 * q + b]) {
                const uint32_t w = cb[first[32 * q + b] + c];
                s[q] += ke[(((size_t)(w >> 6) * nnpe + ((w >> 3) & 7u)) * nnpe + (w & 7u)) * E + en];
            }
#pragma unroll
    for (int q = 0; q < SLOT_GROUPS; ++q) {
        const int h = 32 * q + b, mask = free_cols[h];
        if (mask >= 0) {
            const int64_t pos = rowpos[i][h];
            const bool on = pos >= 0 && (mask >> j & 1);
            if (on) val[pos + __popc(mask & ((1 << j) - 1))] = s[q];
            st[en][b] = on ? s[q] : (mask >> ND & 1) && i == j ? 1.0 : 0.0;
        }
        __syncthreads();
        const int lane = t & 31, plane = t >> 5;
        if (free_cols[32 * q + lane] >= 0) {   // padding slots keep their zero or identity block
            const int64_t o = (s0 + 32 * q) * E + t;
            v64[o] = st[plane][lane];
            v32[o] = (float)st[plane][lane];
        }
        __syncthreads();
    }
}

// f[A] = sum over incident (element, a) in ascending element order of fe[e][a].
template <int ND>
__global__ void __launch_bounds__(NTHREADS) k_gather_nodes(int nnodes, int nnpe, const int64_t *__restrict__ inc_ptr,
                                                           const uint32_t *__restrict__ inc,
                                                           const double *__restrict__ fe, double *__restrict__ f)
{
    int A = blockIdx.x * blockDim.x + threadIdx.x;
    if (A >= nnodes) return;
    double s[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) s[d] = 0.0;
    for (int64_t k = inc_ptr[A]; k < inc_ptr[A + 1]; ++k) {
        uint32_t w = inc[k];
        int e = (int)(w >> 3), a = (int)(w & 7u);
        const double *src = fe + ((size_t)e * nnpe + a) * ND;
#pragma unroll
        for (int d = 0; d < ND; ++d) s[d] += src[d];
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) f[(size_t)A * ND + d] = s[d];
}

// Difference form of the FP32 SELL copy: the diagonal slot of every row
// receives the FP64 block row sum S_A = sum_B K_AB (see k_sell_spmv DIFF);
// padding rows hold one identity block, whose row sum is itself.
template <int ND>
__global__ void __launch_bounds__(NTHREADS) k_sell_rowsum(int nrows, const int64_t *__restrict__ sl_ptr,
                                                          const int *__restrict__ sl_width,
                                                          const int64_t *__restrict__ diag,
                                                          const double *__restrict__ v64, float *__restrict__ v32)
{
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= nrows) return;
    int s = a >> 5, r = a & 31;
    const double *vp = v64 + sl_ptr[s] * (ND * ND) + r;
    double S[ND * ND];
#pragma unroll
    for (int e = 0; e < ND * ND; ++e) S[e] = 0.0;
    for (int k = 0; k < sl_width[s]; ++k)
#pragma unroll
        for (int e = 0; e < ND * ND; ++e) S[e] += vp[(int64_t)k * 32 * ND * ND + 32 * e];
    int64_t slot = diag[a];
    float *out = v32 + (slot - r) * (ND * ND) + r;
#pragma unroll
    for (int e = 0; e < ND * ND; ++e) out[32 * e] = (float)S[e];
}

}  // namespace

int launch_gather_matrix(ogb_model *md, ogb_mtrx *m)
{
    ogb_ctx *ctx = md->ctx;
    if (!m->has_sell) return fail(OGB_E_STATE, "matrix was not built from this model (ogb_model_build_matrix)");
    const SellMat &S = m->sell;
    const unsigned nb = (unsigned)ceil_div(S.nslots, 32 * SLOT_GROUPS);
    if (md->ndofpn == 3)
        k_gather_slots<3><<<nb, 32 * 9, 0, ctx->stream>>>(S.nslots, md->nnpe, S.slot_blk.p, md->blk_node.p, md->nb_col.p,
                                                          md->nb_coloff.p, md->cb_ptr.p, md->cb.p, md->eq.p, md->ke.p,
                                                          m->rowptr.p, m->val.p, S.v64.p, S.v32.p);
    else
        k_gather_slots<2><<<nb, 32 * 4, 0, ctx->stream>>>(S.nslots, md->nnpe, S.slot_blk.p, md->blk_node.p, md->nb_col.p,
                                                          md->nb_coloff.p, md->cb_ptr.p, md->cb.p, md->eq.p, md->ke.p,
                                                          m->rowptr.p, m->val.p, S.v64.p, S.v32.p);
    if (ctx->mixed_diff) {
        const int nrows = S.nslices * 32;   // instances of a batch interleave active and padding rows
        unsigned nbr = (unsigned)ceil_div(nrows, NTHREADS);
        if (S.nd == 3)
            k_sell_rowsum<3><<<nbr, NTHREADS, 0, ctx->stream>>>(nrows, S.sl_ptr.p, S.sl_width.p, S.diag.p, S.v64.p,
                                                                S.v32.p);
        else
            k_sell_rowsum<2><<<nbr, NTHREADS, 0, ctx->stream>>>(nrows, S.sl_ptr.p, S.sl_width.p, S.diag.p, S.v64.p,
                                                                S.v32.p);
        count_launch(ctx);
    }
    m->sell.v32_version = m->version + 1;   // FP32 copy written together with FP64
    count_launch(ctx);
    OGB_CUDA(cudaGetLastError());
    m->version++;
    return OGB_OK;
}

int launch_gather_vector(ogb_model *md, double *f_node)
{
    ogb_ctx *ctx = md->ctx;
    unsigned nb = (unsigned)ceil_div(md->nnodes, NTHREADS);
    if (md->ndofpn == 3)
        k_gather_nodes<3><<<nb, NTHREADS, 0, ctx->stream>>>(md->nnodes, md->nnpe, md->inc_ptr.p, md->inc.p, md->fe.p,
                                                            f_node);
    else
        k_gather_nodes<2><<<nb, NTHREADS, 0, ctx->stream>>>(md->nnodes, md->nnpe, md->inc_ptr.p, md->inc.p, md->fe.p,
                                                            f_node);
    count_launch(ctx);
    OGB_CUDA(cudaGetLastError());
    return OGB_OK;
}

}  // namespace ogb
