// Latent attention: what stands between the projections and the attention core when keys and values are kept as one
// low-rank latent per token.
//
// A token's cache row is [c | r]: the latent c (rank values, RMS-normed with a weight) and one turning key part r (dr
// values, turned by the token's position) that all heads share.  A head's plain key would be Wuk c and its value Wuv c;
// neither is ever formed for cached tokens.  The score q_plain . (Wuk c) equals (Wuk^T q_plain) . c, so the query is
// carried into the latent's space once per token and head (a batch of small products, one per head) and attention runs
// over the rows themselves with ONE key/value head of size rank + dr whose values are the leading rank columns of its
// keys; the head's result, a weighted sum of latents, is brought to value space by Wuv afterwards (again one small
// product per head).  A layer that shares another layer's latents runs the same steps without writing rows.
//
// latent_prepare: one block per token.  From the float projections p (row stride ldp): the plain part of every query
// head goes to q_plain [T, H, dk] (the operand of the products with Wuk^T); the turning part, turned in pairs
// (2i, 2i + 1) by float(pos) * inv_freq[i], goes to columns rank .. rank + dr of q_full [T, H, rank + dr]; and, when the
// layer writes rows, c = rmsnorm(p[c_off : c_off + rank]) * c_w and the turned p[c_off + rank : + dr] go into the
// token's place in the pages (pages[page][0][position in page][rank + dr]).
#include "common.cuh"

//
// BY4 (head parts, rows and their offsets in multiples of four, on 16 bytes): a thread takes four neighbouring values of the queries, whose
// loads, and those of the latent, are under way together before anything waits.  What bounds it is the bytes: p is read once.  Measured on B200,
// 4,096 tokens, 16 heads of 128 + 64, rank 512 (us): a value at a time 57, by fours 32 (90 MB: 14).
template <typename TQ, typename TC, bool BY4>
__global__ void __launch_bounds__(256, 6)
latent_prepare_kernel(const float* __restrict__ p, int ldp, int q_off, int c_off, const float* __restrict__ c_w, float eps,
                      TQ* __restrict__ q_plain, TQ* __restrict__ q_full, TC* __restrict__ k_pages, const int* __restrict__ token_seq,
                      const int* __restrict__ token_pos, const int* __restrict__ table, int table_stride,
                      const float* __restrict__ inv_freq, int H, int dk, int dr, int rank, int page_size, int n_pages,
                      int write_cache, int* status) {
    extern __shared__ __align__(16) float cs[];          // [dr/2] cos, [dr/2] sin
    __shared__ float red[32];
    ik_pdl_wait();
    IK_AFTER_WAIT(p);
    IK_AFTER_WAIT(token_seq);
    IK_AFTER_WAIT(token_pos);
    IK_AFTER_WAIT(table);
    ik_pdl_launch_dependents();
    const int t = blockIdx.x, half = dr / 2, pos = token_pos[t], hd = rank + dr;
    const float* row = p + (size_t)t * ldp;
    const int per = dk + dr;
    constexpr int EARLY = 4;                             // fours of the queries a thread asks for before the latent's sum
    float4 ahead[EARLY];
    if (BY4) {
        #pragma unroll
        for (int k = 0; k < EARLY; k++) {
            const int e = 4 * ((int)threadIdx.x + k * 256);
            if (e < H * per) ahead[k] = ik_ld4(row, q_off + e);
        }
    }
    for (int i = threadIdx.x; i < dr; i += 256) {        // (cosines and sines by threads of their own: each is a long chain)
        const float ang = __fmul_rn((float)pos, inv_freq[i < half ? i : i - half]);
        cs[i] = i < half ? cosf(ang) : sinf(ang);
    }
    float rc = 1.f;
    size_t page_off = 0;
    bool page_ok = false;
    if (write_cache) {
        float ss = 0.f;
        for (int i = threadIdx.x; i < rank; i += 256) { const float v = row[c_off + i]; ss = fmaf(v, v, ss); }
        ss = ik_block_sum<256>(ss, red);
        rc = 1.0f / sqrtf(ss / (float)rank + eps);
        const int page = table[(size_t)token_seq[t] * table_stride + pos / page_size];
        page_ok = page >= 0 && page < n_pages;
        if (!page_ok) { if (threadIdx.x == 0) ik_set_status(status, IK_STATUS_WRITE_NO_PAGE); }
        else page_off = (size_t)page * page_size + (pos % page_size);
    }
    __syncthreads();
    if (BY4) {
        auto four = [&](int e, const float4& v) {
            const int head = e / per, i = e - head * per;
            if (i < dk) { ik_st4(q_plain, ((size_t)t * H + head) * dk + i, v); return; }
            const int f = (i - dk) >> 1;
            const float c0 = cs[f], s0 = cs[half + f], c1 = cs[f + 1], s1 = cs[half + f + 1];
            const float4 turned = make_float4(__fsub_rn(__fmul_rn(v.x, c0), __fmul_rn(v.y, s0)), __fadd_rn(__fmul_rn(v.y, c0), __fmul_rn(v.x, s0)),
                                              __fsub_rn(__fmul_rn(v.z, c1), __fmul_rn(v.w, s1)), __fadd_rn(__fmul_rn(v.w, c1), __fmul_rn(v.z, s1)));
            ik_st4(q_full, ((size_t)t * H + head) * hd + rank + i - dk, turned);
        };
        #pragma unroll
        for (int k = 0; k < EARLY; k++) {
            const int e = 4 * ((int)threadIdx.x + k * 256);
            if (e < H * per) four(e, ahead[k]);
        }
        for (int e = 4 * ((int)threadIdx.x + EARLY * 256); e < H * per; e += 1024) four(e, ik_ld4(row, q_off + e));
    }
    for (int e = threadIdx.x; !BY4 && e < H * per; e += 256) {
        const int head = e / per, i = e - head * per;
        const float val = row[q_off + e];
        if (i < dk) { ik_st(q_plain, ((size_t)t * H + head) * dk + i, val); continue; }
        const int ii = i - dk, f = ii >> 1;
        const bool first = (ii & 1) == 0;
        const float other = row[q_off + (first ? e + 1 : e - 1)];
        const float c = cs[f], s = cs[half + f];
        // (u, v) -> (u c - v s, v c + u s); `first` holds u
        const float turned = first ? __fsub_rn(__fmul_rn(val, c), __fmul_rn(other, s)) : __fadd_rn(__fmul_rn(val, c), __fmul_rn(other, s));
        ik_st(q_full, ((size_t)t * H + head) * hd + rank + ii, turned);
    }
    if (!page_ok) return;
    TC* dst = k_pages + page_off * hd;
    for (int i = threadIdx.x; i < rank; i += 256) ik_st(dst, i, row[c_off + i] * rc * c_w[i]);
    for (int ii = threadIdx.x; ii < dr; ii += 256) {
        const int f = ii >> 1;
        const bool first = (ii & 1) == 0;
        const float val = row[c_off + rank + ii], other = row[c_off + rank + (first ? ii + 1 : ii - 1)];
        const float c = cs[f], s = cs[half + f];
        ik_st(dst, rank + ii, first ? __fsub_rn(__fmul_rn(val, c), __fmul_rn(other, s)) : __fadd_rn(__fmul_rn(val, c), __fmul_rn(other, s)));
    }
}

IK_EXPORT int ik_latent_prepare(const float* p, int ldp, int q_off, int c_off, const float* c_w, float eps, void* q_plain, void* q_full,
                                int q_dtype, void* k_pages, int cache_dtype, const int* token_seq, const int* token_pos,
                                const int* table, int table_stride, const float* inv_freq, int T, int H, int dk, int dr, int rank,
                                int page_size, int n_pages, int write_cache, int* status, cudaStream_t stream) {
    // H = 0: the queries are made elsewhere (behind a latent of their own) and only the row is written; dr = 0: no turning part
    if (T < 0 || H < 0 || (H > 0 && (dk <= 0 || !q_plain || (dr > 0 && !q_full))) || dr < 0 || (dr & 1) || rank <= 0 || page_size <= 0 ||
        (dr > 0 && !inv_freq))
        return IK_BAD_ARGUMENT;
    if (write_cache && (!c_w || !k_pages)) return IK_BAD_ARGUMENT;
    if (T == 0) return IK_OK;
    const size_t smem = (size_t)dr * sizeof(float);
    const bool by4 = H > 0 && dk % 4 == 0 && dr % 4 == 0 && rank % 4 == 0 && ldp % 4 == 0 && q_off % 4 == 0 &&
                     (((uintptr_t)p | (uintptr_t)q_plain | (uintptr_t)q_full) % 16) == 0;
#define IK_LP(TQ, TC)                                                                                                            \
    IK_RETURN_IF_ERROR(ik_launch(by4 ? latent_prepare_kernel<TQ, TC, true> : latent_prepare_kernel<TQ, TC, false>, T, 256, smem, stream, p, ldp, q_off, c_off, c_w, eps, (TQ*)q_plain,   \
                                 (TQ*)q_full, (TC*)k_pages, token_seq, token_pos, table, table_stride, inv_freq, H, dk, dr, rank,  \
                                 page_size, n_pages, write_cache, status))
    if (q_dtype == IK_F32 && cache_dtype == IK_F32) IK_LP(float, float);
    else if (q_dtype == IK_BF16 && cache_dtype == IK_BF16) IK_LP(__nv_bfloat16, __nv_bfloat16);
    else return IK_BAD_ARGUMENT;
#undef IK_LP
    IK_LAUNCH_STATUS();
}
