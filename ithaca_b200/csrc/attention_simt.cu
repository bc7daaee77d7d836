// Attention over the paged cache on the CUDA cores, for prefill and decode alike.
//
// One block per (query token, NG heads that share a kv head: a key's and a value's row is read once for all of them, and the
// weighted sums of all their values keep every thread busy).  A head's arithmetic and its order are the same whatever NG.  Keys run from j0 to the token's own position
// (causal by loop bound; j0 > 0 only under a window), in tiles of 128 that start at
// absolute multiples of 128 (the tiles of the first `keep` keys, which stay visible behind the window, come first), so the order in which a query's keys are reduced depends
// only on its position, not on how the tokens were cut into steps or batched.
// Scores, the running maximum, the sum and the output are float; exp is the accurate
// function.  This is the 32-bit path's attention (prompts without options of head sizes 64 and 128 run in attention_rows.cu, with the
// same bits) and the fallback for head sizes the tensor-core kernels do not take.  Options: a cap on the scores, s <- cap * tanh(s / cap) after the scale
// (cap 0 = none), value heads of another size than the key heads (hdv), values that are the leading hdv columns of the
// key rows themselves (v_pages = k_pages with ldv = hd: a latent that serves as key and value), and a sink: one more
// key of score 0 that carries no value, so that the weights are exp(s_j) / (1 + sum exp(s_j)).  Under a window the first
// `keep` keys of the sequence may stay visible to every later query.  With key_scales (scales[page][kv head][position in page])
// every score is multiplied by its key's number, for keys that are stored as projected because they are the values too and whose
// norm is a factor.  With slopes [nh] a score loses slope * (i - j), behind the cap.
#include <math.h>
#define IK_FAMILY 4
#include "common.cuh"

namespace {

constexpr int TILE = 128;       // keys per tile = threads per block
constexpr int MAX_R = 4;        // head dims per thread: head_dim <= 512

template <typename TQ, typename TC, typename TO, int NG>
__global__ void __launch_bounds__(TILE)
attention_simt_kernel(const TQ* __restrict__ q, const TC* __restrict__ k_pages, const TC* __restrict__ v_pages,
                      TO* __restrict__ out, const int* __restrict__ token_seq, const int* __restrict__ token_pos,
                      const int* __restrict__ table, int table_stride, int nh, int nkv, int hd, int hdv, int ldv, float scale,
                      float softcap, int window, int keep, int sink, const float* __restrict__ sink_v, const float* __restrict__ key_scales,
                      const float* __restrict__ slopes, int page_size, int n_pages, int* status, int vec) {
    ik_pdl_wait();
    ik_pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char smem[];
    size_t* row = (size_t*)smem;              // [TILE] row of key j in the pages (page, kv head, place), times the head size = its offset
    float* sc = (float*)(row + TILE);         // [NG][TILE]
    float* red = sc + NG * TILE;              // [NG][4] a warp's share of a maximum or a sum
    float* qs = red + 4 * NG;                 // [NG][hd]

    const int t = blockIdx.x, h0 = blockIdx.y * NG, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = h0 / (nh / nkv);
    const int pos = token_pos[t], seq = token_seq[t];
    const int j0 = (window > 0 && pos + 1 > window) ? pos + 1 - window : 0;

    const TQ* qrow = q + ((size_t)t * nh + h0) * hd;
    for (int i = tid; i < NG * hd; i += TILE) qs[i] = ik_ld(qrow, i);

    // the sink stands at the head of the running softmax: a maximum of 0 whose weight exp(0 - 0) = 1 is already in the sum
    // (with sink_v the sink's score is the head's own number instead of 0; it is not scaled)
    float m[NG], l[NG], o[MAX_R];
    #pragma unroll
    for (int g = 0; g < NG; g++) { m[g] = sink ? (sink_v ? sink_v[h0 + g] : 0.f) : -INFINITY; l[g] = sink ? 1.f : 0.f; }
    #pragma unroll
    for (int r = 0; r < MAX_R; r++) o[r] = 0.f;
    __syncthreads();

    // every tile visited holds at least one visible key
    const int kept_tiles = (keep + TILE - 1) / TILE;
    for (int tile = keep > 0 ? 0 : j0 / TILE; tile * TILE <= pos; tile = tile + 1 >= kept_tiles ? max(tile + 1, j0 / TILE) : tile + 1) {
        const int base = tile * TILE, j = base + tid;
        const bool valid = (j >= j0 || j < keep) && j <= pos;
        float s[NG];
        #pragma unroll
        for (int g = 0; g < NG; g++) s[g] = -INFINITY;
        size_t off = 0;
        if (valid) {
            const int page = table[(size_t)seq * table_stride + j / page_size];
            if (page < 0 || page >= n_pages) {
                ik_set_status(status, IK_STATUS_READ_NO_PAGE);
                off = 0;
            } else {
                off = ((size_t)page * nkv + kvh) * page_size + (j % page_size);
            }
            const TC* kr = k_pages + off * hd;
            float dot[NG];
            #pragma unroll
            for (int g = 0; g < NG; g++) dot[g] = 0.f;
            if (vec) {                                         // hd a multiple of 4, rows on the boundary of four values
                #pragma unroll 4
                for (int i = 0; i < hd; i += 4) {
                    const float4 k4 = ik_ld4(kr, i);
                    #pragma unroll
                    for (int g = 0; g < NG; g++) {
                        const float4 q4 = *reinterpret_cast<const float4*>(qs + g * hd + i);
                        dot[g] = fmaf(q4.x, k4.x, dot[g]);
                        dot[g] = fmaf(q4.y, k4.y, dot[g]);
                        dot[g] = fmaf(q4.z, k4.z, dot[g]);
                        dot[g] = fmaf(q4.w, k4.w, dot[g]);
                    }
                }
            } else {
                for (int i = 0; i < hd; i++) {
                    const float k1 = ik_ld(kr, i);
                    #pragma unroll
                    for (int g = 0; g < NG; g++) dot[g] = fmaf(qs[g * hd + i], k1, dot[g]);
                }
            }
            #pragma unroll
            for (int g = 0; g < NG; g++) {
                s[g] = dot[g] * scale;
                if (key_scales) s[g] *= key_scales[off];
                if (softcap > 0.f) s[g] = softcap * tanhf(s[g] / softcap);
                if (slopes) s[g] = fmaf(-slopes[h0 + g], (float)(pos - j), s[g]);
            }
        }
        row[tid] = off;
        // maximum and sum over the tile: lanes by shuffles, then the four warps in their order
        #pragma unroll
        for (int g = 0; g < NG; g++) {
            float v = s[g];
            #pragma unroll
            for (int d = 16; d > 0; d >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
            if (lane == 0) red[4 * g + warp] = v;
        }
        __syncthreads();
        float alpha[NG], p[NG];
        #pragma unroll
        for (int g = 0; g < NG; g++) {
            const float m_new = fmaxf(m[g], fmaxf(fmaxf(red[4 * g], red[4 * g + 1]), fmaxf(red[4 * g + 2], red[4 * g + 3])));
            p[g] = valid ? expf(s[g] - m_new) : 0.f;
            sc[g * TILE + tid] = p[g];
            alpha[g] = expf(m[g] - m_new);                     // 0 on the first tile (m = -inf)
            m[g] = m_new;
        }
        __syncthreads();                                       // the maxima have been read
        #pragma unroll
        for (int g = 0; g < NG; g++) {
            float v = p[g];
            #pragma unroll
            for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
            if (lane == 0) red[4 * g + warp] = v;
        }
        __syncthreads();                                       // publishes the sums, sc[] and row[]
        #pragma unroll
        for (int g = 0; g < NG; g++) {
            float sum = 0.f;
            #pragma unroll
            for (int w = 0; w < 4; w++) sum += red[4 * g + w];
            l[g] = l[g] * alpha[g] + sum;
        }
        const int n_in_tile = min(TILE, pos - base + 1);
        #pragma unroll
        for (int r = 0; r < MAX_R; r++) {
            const int x = tid + r * TILE;                      // value i of head g
            if (x < NG * hdv) {
                const int g = NG == 1 ? 0 : x / hdv, i = x - g * hdv;
                float mult = alpha[0];
                #pragma unroll
                for (int e = 1; e < NG; e++) mult = g == e ? alpha[e] : mult;
                float acc = o[r] * mult;
                const float* pg = sc + g * TILE;
                #pragma unroll 8
                for (int jj = 0; jj < n_in_tile; jj++) {
                    const float pj = pg[jj];
                    const float vj = ik_ld(v_pages + row[jj] * ldv, i);
                    if (pj != 0.f) acc = fmaf(pj, vj, acc);
                }
                o[r] = acc;
            }
        }
        __syncthreads();                                       // sc[] and row[] are rewritten by the next tile
    }
    TO* orow = out + ((size_t)t * nh + h0) * hdv;
    #pragma unroll
    for (int r = 0; r < MAX_R; r++) {
        const int x = tid + r * TILE;
        if (x < NG * hdv) {
            const int g = NG == 1 ? 0 : x / hdv;
            float sum = l[0];
            #pragma unroll
            for (int e = 1; e < NG; e++) sum = g == e ? l[e] : sum;
            ik_st(orow, x, o[r] * (1.0f / sum));
        }
    }
}

}  // namespace

IK_EXPORT int ik_attention_simt(const void* q, int q_dtype, const void* k_pages, const void* v_pages, int cache_dtype,
                                void* out, int out_dtype, const int* token_seq, const int* token_pos, const int* table,
                                int table_stride, int T, int nh, int nkv, int hd, int hdv, int ldv, float scale, float softcap, int window, int keep,
                                int sink, const float* sink_v, const float* key_scales, const float* slopes, int page_size, int n_pages, int* status,
                                cudaStream_t stream) {
    if (ldv < hdv) return IK_BAD_ARGUMENT;
    if (T < 0 || nh <= 0 || nkv <= 0 || nh % nkv || hd <= 0 || hdv <= 0 || hdv > TILE * MAX_R || page_size <= 0 || softcap < 0.f || keep < 0) return IK_BAD_ARGUMENT;
    if (q_dtype != out_dtype) return IK_BAD_ARGUMENT;
    if (T == 0) return IK_OK;
    // Heads per block: as many of a kv head's as there are in fours or twos, as long as their values fit the threads, their queries the shared memory, and the
    // blocks still go four times around the SMs (300 tokens, float32, one head / these: 32 heads of 64 on 8 kv heads 620 / 144 us,
    // 200 tokens, 16 heads of 128 on 4 336 / 109).
    const int group = nh / nkv;
    auto bytes = [&](int n) { return TILE * sizeof(size_t) + (size_t)n * (TILE + 4 + hd) * sizeof(float); };    // of shared memory
    int ng = 1;
    for (int n = 4; n > 1; n /= 2)
        if (ng == 1 && group % n == 0 && n * hdv <= TILE * MAX_R && (long long)T * nh / n >= 4LL * ik_sm_count() && bytes(n) <= 48 * 1024) ng = n;
    const int size = cache_dtype == IK_F32 ? 4 : 2;
    const int vec = hd % 4 == 0 && ((uintptr_t)k_pages % (4 * size)) == 0;
    dim3 grid(T, nh / ng);
    const size_t smem = bytes(ng);
#define IK_ATT_N(TQ, TC, NG)                                                                                          \
    IK_RETURN_IF_ERROR(ik_launch(attention_simt_kernel<TQ, TC, TQ, NG>, grid, TILE, smem, stream, (const TQ*)q, (const TC*)k_pages, (const TC*)v_pages, \
        (TQ*)out, token_seq, token_pos, table, table_stride, nh, nkv, hd, hdv, ldv, scale, softcap, window, keep, sink, sink_v, key_scales, slopes, page_size, n_pages, status, vec))
#define IK_ATT(TQ, TC)                                                                                                \
    do {                                                                                                              \
        if (ng == 4) IK_ATT_N(TQ, TC, 4);                                                                             \
        else if (ng == 2) IK_ATT_N(TQ, TC, 2);                                                                        \
        else IK_ATT_N(TQ, TC, 1);                                                                                     \
    } while (0)
    if (q_dtype == IK_F32 && cache_dtype == IK_F32) IK_ATT(float, float);
    else if (q_dtype == IK_BF16 && cache_dtype == IK_BF16) IK_ATT(__nv_bfloat16, __nv_bfloat16);
    else if (q_dtype == IK_F32 && cache_dtype == IK_BF16) IK_ATT(float, __nv_bfloat16);
    else if (q_dtype == IK_BF16 && cache_dtype == IK_F32) IK_ATT(__nv_bfloat16, float);
    else return IK_BAD_ARGUMENT;
#undef IK_ATT
#undef IK_ATT_N
    IK_LAUNCH_STATUS();
}
