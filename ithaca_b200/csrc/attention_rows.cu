// 32-bit attention of prompts over the paged cache on the CUDA cores, head sizes 64 and 128: what attention_simt.cu computes for one token a block,
// for 64 rows (tokens x heads that share a kv head) a block.  Every row's arithmetic and its order are attention_simt.cu's: scores are
// sums in ascending place, keys come in tiles of 128 at absolute multiples of 128, a tile's sum is a butterfly over 32 keys four times over, a
// value's sum runs in ascending key.  So a token has the same bits in a prompt, in a piece of one and in a decode step, whichever kernel takes it.
//
// A block's tokens may belong to several sequences: neighbours of one sequence are a run, and runs follow one another.  Of a run's tile, keys
// and then values go through one buffer of shared memory; a thread holds 4 x 8 scores, later 4 rows x 4 (8) values, in registers.  A row
// that a tile has nothing for (before its window, behind its position) is left alone.
// What bounds it: reads of 16 bytes from shared memory, an SM returns one warp's in four cycles (12 for 128 multiply-adds of a score, 8 for 64 of a value),
// then the latencies between barriers, which two blocks an SM cover in part.  Which steps come here: ops.attention_rows_pay.
// Measured on B200, 32 heads of 64 on 8 kv heads (us, attention_simt.cu / this): prompts of 300, 130 and 35 119 / 60, 700 behind 300 748 / 204, 2,000
// 3,046 / 748; 40 heads of 128 on 40 390 / 139, 3,015 / 490.  (32 rows and 128 threads a block, butterflies a row 77 and 949; 8 x 8 scores a
// thread, 128 threads 79 and 913: a warp to a scheduler waits for itself.)
#include <math.h>
#include <type_traits>
#define IK_FAMILY 4
#include "common.cuh"

namespace {

constexpr int TILE = 128, ROWS = 64, THREADS = 256, PLD = ROWS + 4, WARP_ROWS = ROWS / (THREADS / 32);

template <int HD> constexpr int rows_floats() { return TILE * (HD + 4) + ROWS * (HD + 4) + TILE * PLD + 2 * ROWS + 2 * TILE; }

template <int HD>
__global__ void __launch_bounds__(THREADS, 2)
attention_rows_kernel(const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages, float* __restrict__ out,
                      const int* __restrict__ token_seq, const int* __restrict__ token_pos, const int* __restrict__ table, int table_stride, int T,
                      int nh, int nkv, int heads, float scale, int window, int page_size, int n_pages, int* status) {
    constexpr int LD = HD + 4, VC = HD / 64;                  // rows of keys and queries; fours of values a thread
    extern __shared__ __align__(16) float sm[];
    float* const kv = sm;                                     // [TILE][LD]: keys, then values
    float* const qs = kv + TILE * LD;                         // [ROWS][LD]
    float* const ps = qs + ROWS * LD;                         // [TILE][PLD]: a key's scores, then weights, by row
    float* const factor = ps + TILE * PLD;                    // [ROWS] what a tile's maximum makes of the sums before it; at the end 1 / sum
    int* const row_pos = (int*)(factor + ROWS);               // [ROWS] position, -1: a row that is not there
    size_t* const place = (size_t*)(row_pos + ROWS);          // [TILE] row of key j in the pages (page, kv head, place)
    ik_pdl_wait();
    IK_AFTER_WAIT(q);
    IK_AFTER_WAIT(k_pages);
    IK_AFTER_WAIT(v_pages);
    IK_AFTER_WAIT(token_seq);
    IK_AFTER_WAIT(token_pos);
    IK_AFTER_WAIT(table);
    ik_pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tx = tid & 15, ty = tid >> 4;
    const int tokens = ROWS / heads, t0 = blockIdx.x * tokens, h0 = blockIdx.y * heads, kvh = h0 / (nh / nkv);
    const int n_tok = min(tokens, T - t0);
    // row r: token r / heads, head r % heads
    for (int i = tid; i < ROWS * (HD / 4); i += THREADS) {
        const int r = i / (HD / 4), c = 4 * (i % (HD / 4)), t = r / heads;
        *reinterpret_cast<float4*>(qs + r * LD + c) =
            t < n_tok ? ik_ld4(q, ((size_t)(t0 + t) * nh + h0 + r % heads) * HD + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (tid < ROWS) row_pos[tid] = tid / heads < n_tok ? token_pos[t0 + tid / heads] : -1;
    constexpr int GROUPS = WARP_ROWS / 4;                     // of four rows; a lane keeps the maximum and the sum of row lane / 8 of each
    float m[GROUPS], l[GROUPS];
    #pragma unroll
    for (int i = 0; i < GROUPS; i++) { m[i] = -INFINITY; l[i] = 0.f; }
    float o[4][4 * VC];                                       // rows 4 ty .., values 4 tx .. (and 64 + 4 tx ..)
    #pragma unroll
    for (int i = 0; i < 4; i++)
        #pragma unroll
        for (int c = 0; c < 4 * VC; c++) o[i][c] = 0.f;
    __syncthreads();

    for (int a = 0; a < n_tok;) {                             // a run: tokens t0 + a .. t0 + b - 1
        const int seq = token_seq[t0 + a];
        int b = a + 1, least = row_pos[a * heads], most = least;
        while (b < n_tok && token_seq[t0 + b] == seq) {
            least = min(least, row_pos[b * heads]);
            most = max(most, row_pos[b * heads]);
            b++;
        }
        const int row_lo = a * heads, row_hi = b * heads;
        // (the pages before the first key that any of the run's rows sees may have been given back)
        const int seen = window > 0 && least + 1 > window ? least + 1 - window : 0, first = seen / TILE;
        for (int tile = first; tile * TILE <= most; tile++) {
            const int base = tile * TILE, n_keys = min(TILE, most - base + 1);
            if (tid < n_keys) {
                const int page = base + tid < seen ? 0 : table[(size_t)seq * table_stride + (base + tid) / page_size];
                size_t off = 0;
                if (page < 0 || page >= n_pages) ik_set_status(status, IK_STATUS_READ_NO_PAGE);
                else if (base + tid >= seen) off = ((size_t)page * nkv + kvh) * page_size + (base + tid) % page_size;
                place[tid] = off;
            }
            __syncthreads();
            auto bring = [&](const float* pages) {            // the tile's rows, zeros behind the last; whether all of this thread's are finite
                constexpr int EACH = TILE * (HD / 4) / THREADS;
                bool finite = true;
                #pragma unroll
                for (int k = 0; k < EACH; k += 8) {
                    float4 v[8];
                    #pragma unroll
                    for (int e = 0; e < 8; e++) {
                        const int i = tid + (k + e) * THREADS, r = i / (HD / 4), c = 4 * (i % (HD / 4));
                        v[e] = r < n_keys ? ik_ld4(pages, place[r] * HD + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                    #pragma unroll
                    for (int e = 0; e < 8; e++) {
                        const int i = tid + (k + e) * THREADS, r = i / (HD / 4), c = 4 * (i % (HD / 4));
                        finite = finite && fmaxf(fmaxf(fabsf(v[e].x), fabsf(v[e].y)), fmaxf(fabsf(v[e].z), fabsf(v[e].w))) < INFINITY &&
                                 v[e].x == v[e].x && v[e].y == v[e].y && v[e].z == v[e].z && v[e].w == v[e].w;
                        *reinterpret_cast<float4*>(kv + r * LD + c) = v[e];
                    }
                }
                return finite;
            };
            bring(k_pages);
            __syncthreads();
            {                                                 // scores of rows 4 ty .., keys tx + 16 j
                float s[4][8] = {};
                auto scores = [&](auto most_keys) {
                    #pragma unroll 2
                    for (int d = 0; d < HD; d += 4) {
                        float4 q4[4];
                        #pragma unroll
                        for (int i = 0; i < 4; i++) q4[i] = ik_ld4(qs, (4 * ty + i) * LD + d);
                        #pragma unroll
                        for (int j = 0; j < decltype(most_keys)::value / 16; j++) {
                            const float4 k4 = ik_ld4(kv, (tx + 16 * j) * LD + d);
                            #pragma unroll
                            for (int i = 0; i < 4; i++) {
                                s[i][j] = fmaf(q4[i].x, k4.x, s[i][j]);
                                s[i][j] = fmaf(q4[i].y, k4.y, s[i][j]);
                                s[i][j] = fmaf(q4[i].z, k4.z, s[i][j]);
                                s[i][j] = fmaf(q4[i].w, k4.w, s[i][j]);
                            }
                        }
                    }
                };
                if (n_keys > 48) scores(std::integral_constant<int, TILE>());
                else scores(std::integral_constant<int, 48>());
                #pragma unroll
                for (int j = 0; j < 8; j++)
                    ik_st4(ps, (tx + 16 * j) * PLD + 4 * ty, make_float4(s[0][j] * scale, s[1][j] * scale, s[2][j] * scale, s[3][j] * scale));
            }
            __syncthreads();                                  // the keys have been read, the scores are there
            const bool finite = bring(v_pages);
            // Weights: four rows of a warp at a time, lane's keys lane + 32 c.  Maxima and sums over the lanes by exchanges that halve what a lane holds
            // (the same additions as a butterfly per row and 32 keys, a third of the shuffles): lane 8 r .. ends with row r's maximum, lane
            // 8 r + 2 c with the sum of row r's keys 32 c ...  Without branches; what a row that is not visited comes to is dropped.
            #pragma unroll
            for (int g = 0; g < GROUPS; g++) {
                const int r0 = warp * WARP_ROWS + 4 * g, mine = lane >> 3;
                const int4 p4 = *reinterpret_cast<const int4*>(row_pos + r0);
                const int pos[4] = {p4.x, p4.y, p4.z, p4.w};
                int j0[4];
                bool visited[4];
                #pragma unroll
                for (int r = 0; r < 4; r++) {
                    j0[r] = window > 0 && pos[r] + 1 > window ? pos[r] + 1 - window : 0;
                    visited[r] = r0 + r >= row_lo && r0 + r < row_hi && base <= pos[r] && base + TILE > j0[r];
                }
                float s[4][4], v[4];                          // [c][row]
                #pragma unroll
                for (int c = 0; c < 4; c++) {
                    const float4 s4 = ik_ld4(ps, (lane + 32 * c) * PLD + r0);
                    s[c][0] = s4.x; s[c][1] = s4.y; s[c][2] = s4.z; s[c][3] = s4.w;
                    const int j = base + lane + 32 * c;
                    #pragma unroll
                    for (int r = 0; r < 4; r++) {
                        if (!(j >= j0[r] && j <= pos[r])) s[c][r] = -INFINITY;
                        v[r] = c ? fmaxf(v[r], s[c][r]) : s[c][r];
                    }
                }
                const bool u16 = lane & 16, u8 = lane & 8, u4 = lane & 4, u2 = lane & 2;
                #pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float theirs = __shfl_xor_sync(0xffffffffu, u16 ? v[i] : v[i + 2], 16);
                    v[i] = fmaxf(u16 ? v[i + 2] : v[i], theirs);
                }
                {
                    const float theirs = __shfl_xor_sync(0xffffffffu, u8 ? v[0] : v[1], 8);
                    v[0] = fmaxf(u8 ? v[1] : v[0], theirs);
                }
                #pragma unroll
                for (int d = 4; d > 0; d >>= 1) v[0] = fmaxf(v[0], __shfl_xor_sync(0xffffffffu, v[0], d));
                const bool seen = mine == 0 ? visited[0] : mine == 1 ? visited[1] : mine == 2 ? visited[2] : visited[3];
                const float m_new = fmaxf(m[g], v[0]);
                #pragma unroll
                for (int r = 0; r < 4; r++) {
                    const float top = __shfl_sync(0xffffffffu, m_new, 8 * r);
                    #pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const int j = base + lane + 32 * c;
                        s[c][r] = visited[r] && j >= j0[r] && j <= pos[r] ? expf(s[c][r] - top) : 0.f;
                    }
                }
                #pragma unroll
                for (int c = 0; c < 4; c++) ik_st4(ps, (lane + 32 * c) * PLD + r0, make_float4(s[c][0], s[c][1], s[c][2], s[c][3]));
                #pragma unroll
                for (int c = 0; c < 4; c++) {
                    #pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const float theirs = __shfl_xor_sync(0xffffffffu, u16 ? s[c][i] : s[c][i + 2], 16);
                        s[c][i] = (u16 ? s[c][i + 2] : s[c][i]) + theirs;
                    }
                    const float theirs = __shfl_xor_sync(0xffffffffu, u8 ? s[c][0] : s[c][1], 8);
                    s[c][0] = (u8 ? s[c][1] : s[c][0]) + theirs;
                }
                #pragma unroll
                for (int c = 0; c < 2; c++) {
                    const float theirs = __shfl_xor_sync(0xffffffffu, u4 ? s[c][0] : s[c + 2][0], 4);
                    s[c][0] = (u4 ? s[c + 2][0] : s[c][0]) + theirs;
                }
                {
                    const float theirs = __shfl_xor_sync(0xffffffffu, u2 ? s[0][0] : s[1][0], 2);
                    s[0][0] = (u2 ? s[1][0] : s[0][0]) + theirs;
                }
                s[0][0] += __shfl_xor_sync(0xffffffffu, s[0][0], 1);
                float sum = 0.f;
                #pragma unroll
                for (int c = 0; c < 4; c++) sum += __shfl_sync(0xffffffffu, s[0][0], (lane & 24) + 2 * c);
                const float alpha = seen ? expf(m[g] - m_new) : 1.f;
                l[g] = seen ? l[g] * alpha + sum : l[g];
                m[g] = seen ? m_new : m[g];
                if ((lane & 7) == 0) factor[r0 + mine] = alpha;
            }
            // weights and values are there.  A key a row does not see has a weight of 0 and leaves the sum as it is, unless its value is not finite:
            // then, and only then, every product is asked whether it is wanted.
            const bool plain = __syncthreads_and(finite);
            #pragma unroll
            for (int i = 0; i < 4; i++) {
                const float f = factor[4 * ty + i];
                #pragma unroll
                for (int c = 0; c < 4 * VC; c++) o[i][c] *= f;
            }
            auto values = [&](auto asked) {
                #pragma unroll 4
                for (int jj = 0; jj < n_keys; jj++) {
                    const float4 w4 = ik_ld4(ps, jj * PLD + 4 * ty);
                    const float w[4] = {w4.x, w4.y, w4.z, w4.w};
                    #pragma unroll
                    for (int c = 0; c < VC; c++) {
                        const float4 v4 = ik_ld4(kv, jj * LD + 64 * c + 4 * tx);
                        #pragma unroll
                        for (int i = 0; i < 4; i++)
                            if (!decltype(asked)::value || w[i] != 0.f) {
                                o[i][4 * c] = fmaf(w[i], v4.x, o[i][4 * c]);
                                o[i][4 * c + 1] = fmaf(w[i], v4.y, o[i][4 * c + 1]);
                                o[i][4 * c + 2] = fmaf(w[i], v4.z, o[i][4 * c + 2]);
                                o[i][4 * c + 3] = fmaf(w[i], v4.w, o[i][4 * c + 3]);
                            }
                    }
                }
            };
            if (plain) values(std::false_type());
            else values(std::true_type());
            __syncthreads();                                  // the buffer, the weights and the factors are rewritten
        }
        a = b;
    }
    #pragma unroll
    for (int g = 0; g < GROUPS; g++)
        if ((lane & 7) == 0) factor[warp * WARP_ROWS + 4 * g + (lane >> 3)] = 1.0f / l[g];
    __syncthreads();
    #pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = 4 * ty + i, t = r / heads;
        if (t >= n_tok) continue;
        const float f = factor[r];
        #pragma unroll
        for (int c = 0; c < VC; c++)
            ik_st4(out, ((size_t)(t0 + t) * nh + h0 + r % heads) * HD + 64 * c + 4 * tx,
                   make_float4(o[i][4 * c] * f, o[i][4 * c + 1] * f, o[i][4 * c + 2] * f, o[i][4 * c + 3] * f));
    }
}

template <int HD>
int launch_rows(const float* q, const float* k, const float* v, float* out, const int* token_seq, const int* token_pos, const int* table, int table_stride,
                int T, int nh, int nkv, float scale, int window, int page_size, int n_pages, int* status, cudaStream_t stream) {
    // heads of a kv head in a block: as many as divide them, up to eight (a key then meets the rows of four tokens)
    const int group = nh / nkv;
    int heads = 1;
    while (heads < 8 && group % (2 * heads) == 0) heads *= 2;
    constexpr int smem = rows_floats<HD>() * (int)sizeof(float);
    IK_RETURN_IF_ERROR(cudaFuncSetAttribute(attention_rows_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const int tokens = ROWS / heads;
    IK_RETURN_IF_ERROR(ik_launch(attention_rows_kernel<HD>, dim3((T + tokens - 1) / tokens, nh / heads), THREADS, smem, stream, q, k, v, out, token_seq,
                                 token_pos, table, table_stride, T, nh, nkv, heads, scale, window, page_size, n_pages, status));
    IK_LAUNCH_STATUS();
}

}  // namespace

// As ik_attention_simt for float queries and pages without options but a window.  IK_UNSUPPORTED for other head sizes and rows off 16 bytes.
IK_EXPORT int ik_attention_rows(const float* q, const float* k_pages, const float* v_pages, float* out, const int* token_seq, const int* token_pos,
                                const int* table, int table_stride, int T, int nh, int nkv, int hd, float scale, int window, int page_size,
                                int n_pages, int* status, cudaStream_t stream) {
    if (T < 0 || nh <= 0 || nkv <= 0 || nh % nkv || hd <= 0 || page_size <= 0) return IK_BAD_ARGUMENT;
    if (((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)out) % 16 || nh > 65535) return IK_UNSUPPORTED;
    if (T == 0) return IK_OK;
    if (hd == 64) return launch_rows<64>(q, k_pages, v_pages, out, token_seq, token_pos, table, table_stride, T, nh, nkv, scale, window, page_size, n_pages, status, stream);
    if (hd == 128) return launch_rows<128>(q, k_pages, v_pages, out, token_seq, token_pos, table, table_stride, T, nh, nkv, scale, window, page_size, n_pages, status, stream);
    return IK_UNSUPPORTED;
}
