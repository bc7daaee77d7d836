// Latent attention of prompts with the keys and values of every head formed from the cached rows.
//
// Carried into the rows' space, a score costs rank + turning part products and a value rank more (512 + 64 + 512); formed per head
// they cost head size + turning part and head size (128 + 64 + 128), plus once per key and head the products that form them.
// With some hundred new tokens behind a key the second way is the cheaper one by far, so prompts go this way: the cached latents
// are gathered into one matrix (latent_gather_kernel), one product gives all heads' plain keys and values, and the kernel
// below runs attention over them; the turning part of a key, which all heads share, is read from the cached rows themselves.
//
// The attention: a block owns 2 x 128 queries of one head of one sequence and walks the keys 64 at a time; both tiles of queries
// read the same copies of keys and values.  As in attention_bf16.cu a tile's scores lie in two TMEM buffers of 64 columns, the
// softmax threads (one per query) write P over the scores it came from, and O += P V accumulates in TMEM:
//   warp 0      TMA: the queries once, then keys one step ahead of values, three stages each
//   warp 1      tcgen05.mma (the warp stays together and elects the lane that issues)
//   warps 2..5  softmax of the first tile, warps 6..9 of the second
// TMEM: scores 2 x 2 x 64 columns, outputs 2 x 128.  What bounds a step is the products of a score 64 columns wide, which the
// tensor core takes at half its rate (12 x 64 + 4 x 64 cycles per tile), beside a softmax warp's chain; two tiles keep either busy
// while the other waits.
// Measured on B200: 4,096 tokens, 16 heads, rank 512 + 64: attention over the cached rows 1,713 us -> 107 us (805 TFLOP/s of what is left),
// 7 us for the gathering and 64 us for the product in front of it; the layer 2,056 -> 348 us.
// All waits are bounded (tc_common.cuh).
#include <math.h>
#define IK_FAMILY 4
#include "tc_common.cuh"

namespace {

typedef __nv_bfloat16 bf16;
constexpr int HDV = 128, PAGE = 64, BM = 128, NS = 3;          // head size of plain keys and values; keys a step; queries a tile; stages
constexpr int THREADS = 320;
constexpr int O_COL = 256;
template <int TURN> struct Cfg {                               // TURN: 64 turning columns beside the plain ones
    static constexpr int KB = 2 + TURN;                        // 64-wide boxes of a key
    static constexpr int Q_BYTES = KB * BM * 128, K_BYTES = KB * PAGE * 128, V_BYTES = 2 * PAGE * 128;
    static constexpr int SMEM = 2 * Q_BYTES + NS * (K_BYTES + V_BYTES) + 512;
};

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&p);
}
// Where a sequence's keys begin in the gathered matrix: every sequence's rows are padded to whole steps.
__device__ __forceinline__ int key_base(const int* kv_lens, int b) {
    int base = 0;
    for (int i = 0; i < b; i++) base += (kv_lens[i] + PAGE - 1) / PAGE * PAGE;
    return base;
}

template <int TURN>
__global__ void __launch_bounds__(THREADS, 1)
latent_prompt_kernel(const __grid_constant__ CUtensorMap map_qp, const __grid_constant__ CUtensorMap map_qt, const __grid_constant__ CUtensorMap map_kv,
                     const __grid_constant__ CUtensorMap map_rows, bf16* __restrict__ out, const int* __restrict__ cu_seqlens,
                     const int* __restrict__ kv_lens, const int* __restrict__ table, int table_stride, int H, int hd, int rank, float scale_log2e,
                     int window, int n_pages, int* status) {
    typedef Cfg<TURN> C;
    extern __shared__ __align__(1024) unsigned char smem[];
    ik_pdl_wait();
    ik_pdl_launch_dependents();
    // late tiles see the most keys: they are started first
    const int linear = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z), per_tile = gridDim.y * gridDim.z;
    const int tile = gridDim.x - 1 - linear / per_tile, h = (linear % per_tile) % gridDim.y, b = (linear % per_tile) / gridDim.y;
    const int q_begin = cu_seqlens[b], n_new = cu_seqlens[b + 1] - q_begin;
    const int row0 = tile * 2 * BM;
    if (row0 >= n_new) return;
    if (ik_status_has(status, IK_STATUS_GEMM_TIMEOUT)) return;
    const int kv_len = kv_lens[b], start = kv_len - n_new;
    if (smem_u32(smem) & 1023) {
        if (threadIdx.x == 0) ik_set_status(status, IK_STATUS_SMEM_ALIGN);
        return;
    }
    // steps [first, last] of either tile, counted from the first tile's first
    int rows[2], pos_lo[2], first[2], last[2];
    const int j_lo0 = window > 0 ? max(0, start + row0 + 1 - window) : 0, p_lo = j_lo0 / PAGE;
    #pragma unroll
    for (int t = 0; t < 2; t++) {
        rows[t] = max(0, min(BM, n_new - row0 - t * BM));
        pos_lo[t] = start + row0 + t * BM;
        first[t] = (window > 0 ? max(0, pos_lo[t] + 1 - window) : 0) / PAGE - p_lo;
        last[t] = rows[t] > 0 ? (pos_lo[t] + rows[t] - 1) / PAGE - p_lo : -1;
    }
    const int n_iter = max(last[0], last[1]) + 1;

    unsigned char* Qs = smem;                                  // [2][Q_BYTES]
    unsigned char* Ks = Qs + 2 * C::Q_BYTES;
    unsigned char* Vs = Ks + NS * C::K_BYTES;
    uint64_t* q_full = (uint64_t*)(Vs + NS * C::V_BYTES);
    uint64_t* k_full = q_full + 1;
    uint64_t* v_full = k_full + NS;
    uint64_t* k_free = v_full + NS;
    uint64_t* v_free = k_free + NS;
    uint64_t* s_full = v_free + NS;                            // [tile][buffer]
    uint64_t* p_ready = s_full + 4;                            // [tile][buffer]
    uint64_t* pv_done = p_ready + 4;                           // [tile]
    uint64_t* o_done = pv_done + 2;                            // [tile] used once
    uint32_t* tmem_slot = (uint32_t*)(o_done + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < NS; s++) { mbar_init(k_full + s, 1); mbar_init(v_full + s, 1); mbar_init(k_free + s, 1); mbar_init(v_free + s, 1); }
        for (int i = 0; i < 4; i++) { mbar_init(s_full + i, 1); mbar_init(p_ready + i, 128); }
        for (int t = 0; t < 2; t++) { mbar_init(pv_done + t, 1); mbar_init(o_done + t, 1); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    auto wait_all = [&](uint64_t* bar, uint32_t parity, int site, int i) {
        return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, status, IK_WAIT_LIMIT_NS, site, i)) != 0;
    };

    if (warp == 0) {
        const int base = key_base(kv_lens, b) + p_lo * PAGE;
        if (elect_one()) {
            mbar_expect_tx(q_full, (rows[1] > 0 ? 2 : 1) * C::Q_BYTES);
            for (int t = 0; t < (rows[1] > 0 ? 2 : 1); t++) {
                const int y = q_begin + row0 + t * BM;
                for (int bx = 0; bx < 2; bx++) tma_load_2d(Qs + t * C::Q_BYTES + bx * (BM * 128), &map_qp, h * HDV + bx * 64, y, q_full);
                if (TURN) tma_load_2d(Qs + t * C::Q_BYTES + 2 * (BM * 128), &map_qt, h * hd + rank, y, q_full);
            }
        }
        __syncwarp();
        int armed_k = 0, armed_v = 0;
        for (int i = 0; i <= n_iter; i++) {
            if (i < n_iter) {
                const int s = i % NS;
                if (!wait_all(k_free + s, ((i / NS) & 1) ^ 1, 51, i)) break;
                int page = 0;
                if (TURN) {
                    page = table[(size_t)b * table_stride + p_lo + i];
                    if (page < 0 || page >= n_pages) { ik_set_status(status, IK_STATUS_READ_NO_PAGE); page = 0; }
                }
                if (elect_one()) {
                    unsigned char* dst = Ks + s * C::K_BYTES;
                    mbar_expect_tx(k_full + s, C::K_BYTES);
                    for (int bx = 0; bx < 2; bx++) tma_load_2d(dst + bx * (PAGE * 128), &map_kv, h * HDV + bx * 64, base + i * PAGE, k_full + s);
                    if (TURN) tma_load_2d(dst + 2 * (PAGE * 128), &map_rows, rank, page * PAGE, k_full + s);
                }
                __syncwarp();
                armed_k = i + 1;
            }
            if (i > 0) {
                const int s = (i - 1) % NS;
                if (!wait_all(v_free + s, (((i - 1) / NS) & 1) ^ 1, 52, i)) break;
                if (elect_one()) {
                    mbar_expect_tx(v_full + s, C::V_BYTES);
                    for (int bx = 0; bx < 2; bx++)
                        tma_load_2d(Vs + s * C::V_BYTES + bx * (PAGE * 128), &map_kv, (H + h) * HDV + bx * 64, base + (i - 1) * PAGE, v_full + s);
                }
                __syncwarp();
                armed_v = i;
            }
        }
        if (*abort_flag && lane == 0) {                        // leave no copy in flight
            const long long c0 = wait_clock();
            while (!mbar_test(q_full, 0) && !wait_ran_out(c0, 2000000ull)) {}
            for (int i = max(0, armed_k - NS); i < armed_k; i++) {
                const long long c1 = wait_clock();
                while (!mbar_test(k_full + i % NS, (i / NS) & 1) && !wait_ran_out(c1, 2000000ull)) {}
            }
            for (int i = max(0, armed_v - NS); i < armed_v; i++) {
                const long long c1 = wait_clock();
                while (!mbar_test(v_full + i % NS, (i / NS) & 1) && !wait_ran_out(c1, 2000000ull)) {}
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc_qk = umma_idesc(PAGE), idesc_pv = umma_idesc(HDV, 1);
        bool ok = wait_all(q_full, 0, 53, 0);
        auto issue_qk = [&](int i) -> bool {
            const int s = i % NS;
            if (!wait_all(k_full + s, (i / NS) & 1, 54, i)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t k_addr = smem_u32(Ks + s * C::K_BYTES);
            if (elect_one()) {
                #pragma unroll
                for (int t = 0; t < 2; t++) {
                    if (i < first[t] || i > last[t]) continue;
                    const int buf = (i - first[t]) & 1;
                    const uint32_t q_addr = smem_u32(Qs + t * C::Q_BYTES);
                    #pragma unroll
                    for (int j = 0; j < 4 * C::KB; j++)
                        umma(tmem + (2 * t + buf) * PAGE, umma_desc(q_addr + (j / 4) * (BM * 128) + (j % 4) * 32),
                             umma_desc(k_addr + (j / 4) * (PAGE * 128) + (j % 4) * 32), idesc_qk, j != 0);
                    umma_commit(s_full + 2 * t + buf);
                }
                umma_commit(k_free + s);                       // the stage is free once these products have read it
            }
            __syncwarp();
            return true;
        };
        if (ok) ok = issue_qk(0);
        for (int i = 0; i < n_iter && ok; i++) {
            if (i + 1 < n_iter) { ok = issue_qk(i + 1); if (!ok) break; }     // runs while step i is in the softmax
            const int s = i % NS;
            ok = wait_all(v_full + s, (i / NS) & 1, 56, i);
            if (!ok) break;
            const uint32_t v_addr = smem_u32(Vs + s * C::V_BYTES);
            #pragma unroll
            for (int t = 0; t < 2; t++) {
                if (!ok || i < first[t] || i > last[t]) continue;
                const int c = i - first[t], buf = c & 1;
                ok = wait_all(p_ready + 2 * t + buf, (c >> 1) & 1, 55, i);
                if (!ok) continue;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
                    #pragma unroll
                    for (int j = 0; j < PAGE / 16; j++)
                        umma_ts(tmem + O_COL + t * HDV, tmem + (2 * t + buf) * PAGE + j * 8, umma_desc_mn(v_addr + j * 2048, PAGE * 128), idesc_pv, (c | j) != 0);
                    umma_commit(pv_done + t);
                    if (i == last[t]) umma_commit(o_done + t);
                }
                __syncwarp();
            }
            if (ok && elect_one()) umma_commit(v_free + s);
            __syncwarp();
        }
    } else {
        const int t = warp >= 6, quarter = warp & 3, r = quarter * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16), s_col = 2 * t * PAGE, o_col = O_COL + t * HDV;
        const int my_rows = rows[t], my_lo = pos_lo[t], my_first = first[t], n = last[t] - my_first + 1, pos_hi = my_lo + my_rows - 1;
        const bool row_valid = r < my_rows;
        const int pos_r = my_lo + r;
        float m = -INFINITY, l = 0.f;
        bool ok = my_rows > 0;
        for (int c = 0; c < n && ok; c++) {
            const int p = p_lo + my_first + c, buf = c & 1;
            ok = mbar_wait(s_full + 2 * t + buf, (c >> 1) & 1, abort_flag, status, IK_WAIT_LIMIT_NS, 57, c);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float sc[PAGE];
            #pragma unroll
            for (int c0 = 0; c0 < PAGE; c0 += 16) tmem_ld16_issue(lane_base + s_col + buf * PAGE + c0, sc + c0);
            tmem_ld_wait();
            const bool need_mask = (p * PAGE + PAGE - 1 > my_lo) || (window > 0 && p * PAGE < pos_hi + 1 - window);
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            if (need_mask) {
                #pragma unroll
                for (int e = 0; e < PAGE; e++) {
                    const int j = p * PAGE + e;
                    const bool in = row_valid && j <= pos_r && (window <= 0 || j > pos_r - window);
                    sc[e] = in ? sc[e] : -INFINITY;
                    mx4[e & 3] = fmaxf(mx4[e & 3], sc[e]);
                }
            } else {
                #pragma unroll
                for (int e = 0; e < PAGE; e += 2) mx4[(e >> 1) & 3] = max3(mx4[(e >> 1) & 3], sc[e], sc[e + 1]);
            }
            // the reference of the exponentials follows the running maximum only when that has moved by more than 8
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2e;
            float alpha = 1.f;
            if (mx > m + 8.f) {
                alpha = ik_ex2(m - mx);                        // 0 on the first step (m = -inf)
                m = mx;
            }
            const float m_use = m == -INFINITY ? 0.f : m;
            float sum4[4] = {0.f, 0.f, 0.f, 0.f};
            #pragma unroll
            for (int e = 0; e < PAGE; e += 2) {
                float a0, a1;
                fma_f32x2(a0, a1, sc[e], sc[e + 1], scale_log2e, -m_use);
                sc[e] = ik_ex2(a0);
                sc[e + 1] = ik_ex2(a1);
                add_f32x2(sum4[e & 2], sum4[(e & 2) + 1], sc[e], sc[e + 1]);
            }
            l = l * alpha + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
            if (c > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
                // O is at rest between the product of the step before (waited for here; its barrier has completed c - 1 or c
                // phases) and this step's, which waits for this thread
                ok = mbar_wait(pv_done + t, (c - 1) & 1, abort_flag, status, IK_WAIT_LIMIT_NS, 58, c);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                #pragma unroll
                for (int c0 = 0; c0 < HDV; c0 += 32) {
                    float v[32];
                    tmem_ld16_issue(lane_base + o_col + c0, v);
                    tmem_ld16_issue(lane_base + o_col + c0 + 16, v + 16);
                    tmem_ld_wait();
                    #pragma unroll
                    for (int e = 0; e < 32; e++) v[e] *= alpha;
                    tmem_st16(lane_base + o_col + c0, *reinterpret_cast<float(*)[16]>(v));
                    tmem_st16(lane_base + o_col + c0 + 16, *reinterpret_cast<float(*)[16]>(v + 16));
                }
            }
            #pragma unroll
            for (int c0 = 0; c0 < PAGE / 2; c0 += 16) {
                uint32_t pk[16];
                #pragma unroll
                for (int e = 0; e < 16; e++) pk[e] = pack2(sc[2 * (c0 + e)], sc[2 * (c0 + e) + 1]);
                tmem_st16_bits(lane_base + s_col + buf * PAGE + c0, pk);
            }
            tmem_st_wait();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(p_ready + 2 * t + buf);
        }
        if (ok && mbar_wait(o_done + t, 0, abort_flag, status, IK_WAIT_LIMIT_NS, 59, n)) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const float inv = 1.0f / l;
            bf16* orow = out + ((size_t)(q_begin + row0 + t * BM + r) * H + h) * HDV;
            #pragma unroll
            for (int c0 = 0; c0 < HDV; c0 += 16) {
                float v[16];
                tmem_ld16(lane_base + o_col + c0, v);
                if (row_valid) {
                    uint4 w0, w1;
                    w0.x = pack2(v[0] * inv, v[1] * inv);   w0.y = pack2(v[2] * inv, v[3] * inv);
                    w0.z = pack2(v[4] * inv, v[5] * inv);   w0.w = pack2(v[6] * inv, v[7] * inv);
                    w1.x = pack2(v[8] * inv, v[9] * inv);   w1.y = pack2(v[10] * inv, v[11] * inv);
                    w1.z = pack2(v[12] * inv, v[13] * inv); w1.w = pack2(v[14] * inv, v[15] * inv);
                    *reinterpret_cast<uint4*>(orow + c0) = w0;
                    *reinterpret_cast<uint4*>(orow + c0 + 8) = w1;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u) : "memory");
    }
}

// The cached latents of all sequences' keys, one after another: row key_base(b) + j holds the leading `rank` columns of key j of
// sequence b, and zeros where the last step of a sequence has no key.  Pages that lie wholly behind the window of the step's first
// query are passed over: they may have been given back, and their rows are never read.
__global__ void __launch_bounds__(256)
latent_gather_kernel(const bf16* __restrict__ rows, const int* __restrict__ cu_seqlens, const int* __restrict__ kv_lens, const int* __restrict__ table,
                     int table_stride, bf16* __restrict__ out, int hd, int rank, int window, int n_pages, int* status) {
    ik_pdl_wait();
    ik_pdl_launch_dependents();
    const int b = blockIdx.y, p = blockIdx.x, len = kv_lens[b];
    if (p * PAGE >= len) return;
    const int first = len - (cu_seqlens[b + 1] - cu_seqlens[b]);               // position of the sequence's first query
    if (window > 0 && (p + 1) * PAGE <= first + 1 - window) return;
    int page = table[(size_t)b * table_stride + p];
    const bool there = page >= 0 && page < n_pages;
    if (!there) {
        if (threadIdx.x == 0) ik_set_status(status, IK_STATUS_READ_NO_PAGE);
        page = 0;
    }
    bf16* dst = out + ((size_t)key_base(kv_lens, b) + p * PAGE) * rank;
    const int quads = rank / 8;
    for (int i = threadIdx.x; i < PAGE * quads; i += 256) {
        const int r = i / quads, w = i % quads;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (there && p * PAGE + r < len) v = *reinterpret_cast<const uint4*>(rows + ((size_t)page * PAGE + r) * hd + 8 * w);
        *reinterpret_cast<uint4*>(dst + (size_t)r * rank + 8 * w) = v;
    }
}

template <int TURN>
int launch_prompt(const CUtensorMap& qp, const CUtensorMap& qt, const CUtensorMap& kv, const CUtensorMap& rows, void* out, const int* cu_seqlens,
                  const int* kv_lens, const int* table, int table_stride, int B, int max_new, int H, int hd, int rank, float scale, int window,
                  int n_pages, int* status, cudaStream_t stream) {
    const cudaError_t e = cudaFuncSetAttribute(latent_prompt_kernel<TURN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<TURN>::SMEM);
    if (e != cudaSuccess) return (int)e;
    IK_RETURN_IF_ERROR(ik_launch(latent_prompt_kernel<TURN>, dim3((max_new + 2 * BM - 1) / (2 * BM), H, B), THREADS, Cfg<TURN>::SMEM, stream, qp, qt, kv, rows,
                                 (bf16*)out, cu_seqlens, kv_lens, table, table_stride, H, hd, rank, scale * 1.4426950408889634f, window, n_pages,
                                 status));
    IK_LAUNCH_STATUS();
}

}  // namespace

// Gathers the latents (columns 0 .. rank - 1 of the rows [n_pages][64][hd]) of B sequences' keys into out [sum of lengths rounded up to 64, rank].
IK_EXPORT int ik_latent_gather(const void* rows, const int* cu_seqlens, const int* kv_lens, const int* table, int table_stride, void* out, int B,
                               int max_kv_len, int hd, int rank, int window, int n_pages, int* status, cudaStream_t stream) {
    if (B < 0 || max_kv_len < 0 || rank <= 0 || hd < rank || n_pages <= 0) return IK_BAD_ARGUMENT;
    if (hd % 8 || rank % 8 || ((uintptr_t)rows | (uintptr_t)out) % 16 || B > 65535) return IK_UNSUPPORTED;
    if (B == 0 || max_kv_len == 0) return IK_OK;
    IK_RETURN_IF_ERROR(ik_launch(latent_gather_kernel, dim3((max_kv_len + PAGE - 1) / PAGE, B), 256, 0, stream, (const bf16*)rows, cu_seqlens,
                                 kv_lens, table, table_stride, (bf16*)out, hd, rank, window, n_pages, status));
    IK_LAUNCH_STATUS();
}

// q_plain [T, H * 128], q_full [T, H * hd] (turning parts in each head's columns rank .. hd - 1; hd - rank is 64 or 0), kv [n_keys, 2 * H * 128]: all heads'
// plain keys, then their values, in the rows' order of ik_latent_gather; rows: the cached rows, for the keys' turning parts.  out [T, H * 128].
IK_EXPORT int ik_latent_prompt(const void* q_plain, const void* q_full, const void* kv, const void* rows, void* out, const int* cu_seqlens,
                               const int* kv_lens, const int* table, int table_stride, int T, int B, int max_new, int n_keys, int H, int hd, int rank,
                               float scale, int window, int n_pages, int* status, cudaStream_t stream) {
    if (T < 0 || B < 0 || max_new < 0 || n_keys < 0 || H <= 0 || rank <= 0 || hd < rank || n_pages <= 0 || scale <= 0.f) return IK_BAD_ARGUMENT;
    const int turn = hd - rank;
    if ((turn != 0 && turn != 64) || hd % 8 || rank % 8 || B > 65535 || H > 65535 ||
        ((uintptr_t)q_plain | (uintptr_t)q_full | (uintptr_t)kv | (uintptr_t)rows | (uintptr_t)out) % 16) return IK_UNSUPPORTED;
    if (T == 0 || B == 0) return IK_OK;
    CUtensorMap qp, qt = {}, mkv, mrows = {};
    int st = ik_make_map(&qp, q_plain, T, H * HDV, H * HDV, BM);
    if (st != IK_OK) return st;
    st = ik_make_map(&mkv, kv, n_keys, 2 * H * HDV, 2 * H * HDV, PAGE);
    if (st != IK_OK) return st;
    if (turn) {
        st = ik_make_map(&qt, q_full, T, H * hd, H * hd, BM);
        if (st != IK_OK) return st;
        st = ik_make_map(&mrows, rows, (unsigned long long)n_pages * PAGE, hd, hd, PAGE);
        if (st != IK_OK) return st;
        return launch_prompt<1>(qp, qt, mkv, mrows, out, cu_seqlens, kv_lens, table, table_stride, B, max_new, H, hd, rank, scale, window, n_pages, status, stream);
    }
    return launch_prompt<0>(qp, qt, mkv, mrows, out, cu_seqlens, kv_lens, table, table_stride, B, max_new, H, hd, rank, scale, window, n_pages, status, stream);
}

// Sites: 51, 52 = loader for a free stage of keys / values, 53 = issuer for the queries, 54 keys, 55 probabilities, 56 values, 57 = softmax for
// scores, 58 for the product before, 59 for the last.
IK_EXPORT int ik_latent_prompt_take_wait_record(int* out4) { return ik_take_wait_record(out4); }
