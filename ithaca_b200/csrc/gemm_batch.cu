// bfloat16 product on the fifth-generation tensor cores for a decoding batch or a short prompt (up to 128 tokens):
//   Y[M, N] (+)= X[M, K] * W[N, K]^T,  X and W bfloat16 with K contiguous, float accumulation in TMEM.
//
// Such a product is the bytes of W.  Two blocks (a cluster of two neighbouring SMs, cta_group::2) take 256 features x 64 or 128 tokens: each holds 128
// rows of W (TMEM lanes are features) and half of the tokens' rows, so a K step brings 16 KB of W and 4 or 8 KB of X into an SM; a block
// that works alone (gemm_tcgen05.cu) brings 8 or 16 KB of X, which at 128 tokens doubles what the SM takes in.
//
// Few tiles: S = 2 or 4 pairs, a cluster of 2 S blocks, share one tile, each a slice of K.  Every pair then finishes one S-th of the tokens: the blocks
// send one another the sums of the tokens that are not theirs (distributed shared memory, 16 bytes a store) and add what they got in the
// order of the slices.  So the exchange and the epilogue are shared out too, with no scratch and no second kernel.
// Otherwise whole tiles, dealt round robin; two accumulators, one is drained while the other fills.  A last round that is half empty costs
// little, since half of the SMs still draw the memory's full rate.
//
// What bounds it: the bytes of W, and beside them the start, the first latency and the end of a short kernel.
// Measured on B200 (us, replayed graphs over weights larger than L2 together; the ways of gemm_tcgen05.cu before / this / cuBLAS), 64 tokens: gate/up
// 28672 x 4096 51.8 / 43.0 / 41.5 (35.9 for its bytes), down 4096 x 14336 30.9 / 25.5 / 24.4, q/k/v 6144 x 4096 19.4 / 13.8 / 11.8, o 4096 x 4096 17.0 / 11.5 / 10.1,
// gate/up 16384 x 2048 22.1 / 16.0 / 12.5; 128 tokens: 65.4 / 47.0 / 48.0, 35.9 / 29.1 / 25.2, 26.6 / 15.8 / 12.2, 19.8 / 13.8 / 10.3, 28.7 / 17.5 / 13.6; 17 tokens: 43.5 /
// 41.2 / 40.1, 25.2 / 24.3 / 24.0, 15.4 / 13.7 / 11.9.  Of that, the activations in an instance of their own: where every result asked for its kind, eight
// tokens of a tile took 0.65 us to leave (1024 x 512 for 128 tokens 8.7 -> 5.3).
//
// Every wait is bounded like those of gemm_tcgen05.cu.
#include <type_traits>
#define IK_FAMILY 8
#include "tc_common.cuh"
#include "rope_store.cuh"

namespace {

typedef __nv_bfloat16 bf16;
constexpr int BK = 64, EPI_WARPS = 8, THREADS = 128 + 32 * EPI_WARPS, MOST_STAGES = 12, BUDGET = 215 * 1024, MOST_SMEM = BUDGET + 1536;
constexpr int A_BYTES = 128 * BK * 2;
template <int BN, int CG> constexpr int stage_bytes() { return A_BYTES + BN / CG * BK * 2; }
enum { OUT_F32 = 0, OUT_BF16 = 1, OUT_JOIN = 2, OUT_ROPE = 3, OUT_ACT = 4 };

struct BatchArgs {
    void* Y;
    int M, N, ldy, nkb, per, slices, tiles, stages, accumulate;
    int* status;
    IkGlu join;
    IkRopeStore rope;
};

template <int CG> __device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    if (CG == 2)
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                     :: "r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                     :: "r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
template <int CG> __device__ __forceinline__ void product(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t acc) {
    if (CG == 2)
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t}"
                     :: "r"(d), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(acc) : "memory");
    else
        umma_halves(d, a_lo, b_lo, hi, idesc, acc);
}
// Arrives on the barrier (at the same place in both blocks of the pair whose first has cluster rank `first`) once the products issued so far are done.
template <int CG> __device__ __forceinline__ void commit(uint64_t* bar, uint32_t first) {
    if (CG == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                     :: "r"(smem_u32(bar)), "h"((uint16_t)(3u << first)) : "memory");
    else
        umma_commit(bar);
}
// TMEM changes hands: the tcgen05 fences on both sides order it, so the arrival orders no other memory between the blocks (see gemm_split.cu).
__device__ __forceinline__ void arrive_in_cluster(uint32_t addr) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" :: "r"(addr) : "memory"); }
__device__ __forceinline__ void store_in_cluster(uint32_t addr, const float* v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" :: "r"(addr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
}
// mbar_wait for what threads of other blocks have stored here before they arrived.
__device__ __forceinline__ bool wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, int site, int info) {
    if (mbar_test_cluster(bar, parity)) return true;
    const long long c0 = wait_clock();
    for (int spin = 0;; spin++) {
        if (mbar_test_cluster(bar, parity)) return true;
        if ((spin & 63) == 63) {
            if (*abort_flag) return false;
            if (wait_ran_out(c0, IK_WAIT_LIMIT_NS)) {
                note_wait_gave_up(site, info, (int)parity);
                *abort_flag = 1;
                ik_set_status(status, IK_STATUS_GEMM_TIMEOUT);
                return false;
            }
        }
    }
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    #pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}

template <int BN, int CG, int OUT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_batch_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ BatchArgs g) {
    constexpr int STAGE = stage_bytes<BN, CG>(), FEATURES = 128 * CG;
    typedef typename std::conditional<OUT == OUT_F32, float, bf16>::type TY;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int nst = g.stages, S = g.slices, CW = BN / S;
    const int ld_got = CW + 4;                                         // floats of a lane's row of what a block got: no bank twice
    float* const got = (float*)(tiles + nst * STAGE);                  // [S - 1][128 lanes][ld_got]
    uint64_t* full = (uint64_t*)(got + (size_t)(S - 1) * 128 * ld_got);
    uint64_t* empty = full + MOST_STAGES;
    uint64_t* acc_full = empty + MOST_STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* got_full = acc_empty + 2;
    uint32_t* tmem_slot = (uint32_t*)(got_full + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t crank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
    const uint32_t rank = CG == 2 ? crank & 1 : 0, head = crank - rank;    // place in the pair, cluster rank of the pair's first block
    const int slice = (int)crank / CG;
    int* const status = g.status;
    const int first = (int)blockIdx.x / (CG * S), step = (int)gridDim.x / (CG * S);
    const int k_lo = slice * g.per, k_hi = min(g.nkb, k_lo + g.per);

    if (threadIdx.x == 0) {
        for (int s = 0; s < nst; s++) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        for (int b = 0; b < 2; b++) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, CG * EPI_WARPS); }
        mbar_init(got_full, S > 1 ? (S - 1) * EPI_WARPS : 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&map_x) : "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&map_w) : "memory");
    }
    if (warp == 1) {
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tmem_slot)), "r"(2u * BN) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tmem_slot)), "r"(2u * BN) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    cluster_sync();                                    // every block's barriers exist before another arrives on them

    // Weights are written by no kernel: those of the first stages are asked for before the wait for the kernel before.
    int pre = 0;
    if (threadIdx.x == 0) {
        for (int u = first; u < g.tiles && pre < nst; u += step)
            for (int i = k_lo; i < k_hi && pre < nst; i++, pre++) {
                if (rank == 0) mbar_expect_tx(full + pre, CG * STAGE);
                load_tile<CG>(smem_u32(tiles + pre * STAGE), &map_w, i * BK, u * FEATURES + (int)rank * 128, cluster_addr(smem_u32(full + pre), head));
            }
    }
    ik_pdl_wait();
    ik_pdl_launch_dependents();

    if (warp == 0) {
        int it = 0, s = 0;
        uint32_t phase = 1;                            // of the next wait for a free stage
        bool ok = true;
        const int n_pre = __shfl_sync(0xffffffffu, pre, 0);
        const uint32_t full0 = cluster_addr(smem_u32(full), head);
        for (int u = first; ok && u < g.tiles; u += step)
            for (int i = k_lo; i < k_hi; i++, it++) {
                if (it >= n_pre) {
                    ok = __all_sync(0xffffffffu, mbar_wait(empty + s, phase, abort_flag, status, IK_WAIT_LIMIT_NS, 1, it));
                    if (!ok) break;
                }
                if (elect_one()) {
                    const uint32_t bar = full0 + s * 8, a = smem_u32(tiles + s * STAGE);
                    if (it >= n_pre) {
                        if (rank == 0) mbar_expect_tx(full + s, CG * STAGE);
                        load_tile<CG>(a, &map_w, i * BK, u * FEATURES + (int)rank * 128, bar);
                    }
                    load_tile<CG>(a + A_BYTES, &map_x, i * BK, (int)rank * (BN / CG), bar);
                }
                __syncwarp();
                if (++s == nst) { s = 0; phase ^= 1; }
            }
        if (*abort_flag && rank == 0 && lane == 0) {   // leave no copy in flight: the stages armed last
            for (int i = max(0, it - nst); i < it; i++) {
                const long long c0 = wait_clock();
                while (!mbar_test(full + i % nst, (i / nst) & 1) && !wait_ran_out(c0, 2000000ull)) {}
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(FEATURES >> 4) << 24);
            const uint32_t hi = umma_desc_hi(), lo0 = umma_desc_lo(smem_u32(tiles));
            int it = 0, lt = 0, s = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int u = first; ok && u < g.tiles; u += step, lt++) {
                const int buf = lt & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(acc_empty + buf, ((lt >> 1) & 1) ^ 1, abort_flag, status, IK_WAIT_LIMIT_NS, 2, lt));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int i = k_lo; i < k_hi; i++, it++) {
                    ok = __all_sync(0xffffffffu, mbar_wait(full + s, phase, abort_flag, status, IK_WAIT_LIMIT_NS, 3, it));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_lo = lo0 + (uint32_t)s * (STAGE >> 4), b_lo = a_lo + (A_BYTES >> 4);
                    if (elect_one()) {
                        #pragma unroll
                        for (int j = 0; j < BK / 16; j++) product<CG>(tmem + buf * BN, a_lo + 2 * j, b_lo + 2 * j, hi, idesc, (uint32_t)(i != k_lo || j != 0));
                        commit<CG>(empty + s, head);
                    }
                    __syncwarp();
                    if (++s == nst) { s = 0; phase ^= 1; }
                }
                if (ok && elect_one()) commit<CG>(acc_full + buf, head);
                __syncwarp();
            }
        }
    } else if (warp >= 4) {
        const int quarter = warp & 3, half = (warp - 4) >> 2, row = quarter * 32 + lane;
        const bool odd = lane & 1;
        TY* const Y = (TY*)g.Y;
        int lt = 0;
        for (int u = first; u < g.tiles; u += step, lt++) {
            const int buf = lt & 1, f = u * FEATURES + (int)rank * 128 + row, wide = CW / 2, c_lo = slice * CW + half * wide;    // this warp's tokens
            const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + buf * BN;
            // what the results meet: asked for before the sums are waited for, and for the next eight tokens before these are stored
            float old[8] = {};
            auto load_old = [&](int c) {
                #pragma unroll
                for (int i = 0; i < 8; i++) old[i] = f < g.N && c + i < g.M ? ik_ld(Y, (size_t)(c + i) * g.ldy + f) : 0.f;
            };
            const IkRopeStore& e = g.rope;
            const int f0 = f & ~1, hd_of = OUT == OUT_ROPE ? f0 / e.hd : 0, r0 = OUT == OUT_ROPE ? f0 - hd_of * e.hd : 0;
            const bool is_q = OUT == OUT_ROPE && hd_of < e.nh, rotated = OUT == OUT_ROPE && hd_of < e.nh + e.nkv;
            float2 cs[4] = {};
            auto load_rope = [&](int c) {
                #pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int m = c + (odd ? 4 : 0) + i;
                    cs[i] = make_float2(1.f, 0.f);
                    if (rotated && f < g.N && m < g.M)
                        asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(cs[i].x), "=f"(cs[i].y) : "l"(e.cos_sin + ((size_t)m * (e.hd >> 1) + (r0 >> 1)) * 2));
                }
            };
            int at_lo = -1, at_hi = -1;                // cache rows of the warp's tokens lane and 32 + lane
            if (OUT == OUT_ROPE) {
                if (lane < wide) at_lo = ik_rope_cache_row(e, c_lo + lane, g.M);
                if (32 + lane < wide) at_hi = ik_rope_cache_row(e, c_lo + 32 + lane, g.M);
            }
            if (OUT == OUT_F32 && g.accumulate) load_old(c_lo);
            if (OUT == OUT_ROPE) load_rope(c_lo);
            if (!mbar_wait(acc_full + buf, (lt >> 1) & 1, abort_flag, status, IK_WAIT_LIMIT_NS, 4, lt)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (S > 1) {                               // (one tile a cluster)
                for (int d = 1; d < S; d++) {
                    const int to = (slice + d) % S;
                    const uint32_t theirs = cluster_addr(smem_u32(got + ((size_t)(slice < to ? slice : slice - 1) * 128 + row) * ld_got), CG * to + rank);
                    int c = half * wide;
                    for (; c + 16 <= (half + 1) * wide; c += 16) {
                        float v[16];
                        tmem_ld16_issue(acc + to * CW + c, v);
                        tmem_ld_wait();
                        #pragma unroll
                        for (int i = 0; i < 16; i += 4) store_in_cluster(theirs + 4 * (c + i), v + i);
                    }
                    for (; c < (half + 1) * wide; c += 8) {
                        float v[8];
                        tmem_ld8(acc + to * CW + c, v);
                        store_in_cluster(theirs + 4 * c, v);
                        store_in_cluster(theirs + 4 * c + 16, v + 4);
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(cluster_addr(smem_u32(got_full), CG * to + rank));       // releases the warp's stores
                }
                if (!wait_cluster(got_full, 0, abort_flag, status, 5, lt)) break;
            }
            #pragma unroll 1
            for (int c = c_lo; c < c_lo + wide && c < g.M; c += 8) {
                const bool more = c + 8 < c_lo + wide && c + 8 < g.M;
                float had[8], v[8];
                float2 turn[4];
                #pragma unroll
                for (int i = 0; i < 8; i++) had[i] = old[i];
                #pragma unroll
                for (int i = 0; i < 4; i++) turn[i] = cs[i];
                if (OUT == OUT_F32 && g.accumulate && more) load_old(c + 8);
                if (OUT == OUT_ROPE && more) load_rope(c + 8);
                tmem_ld8(acc + c, v);
                if (S > 1) {
                    float t[8];
                    #pragma unroll
                    for (int i = 0; i < 8; i++) t[i] = 0.f;
                    for (int s = 0; s < S; s++) {
                        if (s == slice) {
                            #pragma unroll
                            for (int i = 0; i < 8; i++) t[i] += v[i];
                            continue;
                        }
                        const float* p = got + ((size_t)(s < slice ? s : s - 1) * 128 + row) * ld_got + c - slice * CW;
                        const float4 a = ik_ld4(p, 0), b = ik_ld4(p, 4);
                        t[0] += a.x; t[1] += a.y; t[2] += a.z; t[3] += a.w; t[4] += b.x; t[5] += b.y; t[6] += b.z; t[7] += b.w;
                    }
                    #pragma unroll
                    for (int i = 0; i < 8; i++) v[i] = t[i];
                }
                if (OUT == OUT_F32) {
                    if (g.accumulate) {
                        #pragma unroll
                        for (int i = 0; i < 8; i++) v[i] += had[i];
                    }
                    if (f < g.N) {
                        #pragma unroll
                        for (int i = 0; i < 8; i++)
                            if (c + i < g.M) ik_st(Y, (size_t)(c + i) * g.ldy + f, v[i]);
                    }
                } else if (OUT == OUT_BF16 || OUT == OUT_ACT) {
                    if (f < g.N) {
                        #pragma unroll
                        for (int i = 0; i < 8; i++)
                            if (c + i < g.M) ik_st(Y, (size_t)(c + i) * g.ldy + f, OUT == OUT_ACT ? ik_glu_act(g.join, v[i]) : v[i]);
                    }
                } else {
                    // lanes (2j, 2j + 1) hold gate j and up j, or a rotary pair: the even lane takes tokens 0 .. 3, the odd one 4 .. 7
                    const float bias0 = OUT == OUT_ROPE && e.bias && f < g.N ? e.bias[f0] : 0.f, bias1 = OUT == OUT_ROPE && e.bias && f < g.N ? e.bias[f0 + 1] : 0.f;
                    #pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float other = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 4], 1);
                        const float a = odd ? other : v[i], b = odd ? v[i + 4] : other;
                        const int m = c + (odd ? 4 : 0) + i;
                        int at = -1;
                        if (OUT == OUT_ROPE) at = __shfl_sync(0xffffffffu, c - c_lo < 32 ? at_lo : at_hi, (m - c_lo) & 31);
                        if (f >= g.N || m >= g.M) continue;
                        if (OUT == OUT_JOIN) {
                            ik_st(Y, (size_t)m * g.ldy + (f >> 1), ik_glu_join_fast(g.join, a, b));
                        } else {
                            const float x = a + bias0, y = b + bias1;
                            const __nv_bfloat162 packed = __floats2bfloat162_rn(x * turn[i].x - y * turn[i].y, x * turn[i].y + y * turn[i].x);
                            if (is_q) *reinterpret_cast<__nv_bfloat162*>(e.q_out + ((size_t)m * e.nh + hd_of) * e.hd + r0) = packed;
                            else if (at >= 0)
                                *reinterpret_cast<__nv_bfloat162*>((rotated ? e.k_pages : e.v_pages) +
                                    ((size_t)at + (size_t)(hd_of - e.nh - (rotated ? 0 : e.nkv)) * e.page_size) * e.hd + r0) = packed;
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_in_cluster(cluster_addr(smem_u32(acc_empty + buf), head));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();                                    // no block leaves, or gives its TMEM back, while another still works with it
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(2u * BN) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(2u * BN) : "memory");
    }
}

template <int BN, int CG, int OUT>
int launch_batch(const CUtensorMap& mx, const CUtensorMap& mw, BatchArgs& g, cudaStream_t stream) {
    constexpr int STAGE = stage_bytes<BN, CG>();
    auto kern = gemm_batch_kernel<BN, CG, OUT>;
    const int room = (g.slices - 1) * 128 * (BN / g.slices + 4) * 4;
    g.stages = (BUDGET - room) / STAGE;
    if (g.stages > MOST_STAGES) g.stages = MOST_STAGES;
    const int smem = g.stages * STAGE + room + 1024 + 512;
    // the most of any call, not this one's: another thread may launch the same instance for another share in between
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST_SMEM);
    if (e != cudaSuccess) return (int)e;
    const int most = ik_sm_count() / CG;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(g.slices > 1 ? CG * g.slices * g.tiles : CG * (g.tiles < most ? g.tiles : most)));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CG * g.slices; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (ik_pdl_mask() & IK_FAMILY) ? 2 : 1;
    IK_RETURN_IF_ERROR(cudaLaunchKernelEx(&cfg, kern, mx, mw, g));
    return (int)cudaGetLastError();
}

struct Share { int cg, slices; };                                      // blocks to a tile, slices of K

// Clusters of four blocks that find room at once with all of the shared memory each: fewer than a quarter of the SMs, since a cluster lies within one
// group of them (asked for once per device).
int clusters_of_four() {
    static int cached[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (cached[dev] == 0) {
        auto kern = gemm_batch_kernel<128, 1, OUT_F32>;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 4; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(4 * 64); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = MOST_SMEM;
        cfg.attrs = attr; cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST_SMEM) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
            (void)cudaGetLastError();
            n = ik_sm_count() / 5;
        }
        cached[dev] = n;
    }
    return cached[dev];
}

// Four slices of 128 features where they find room for all tiles at once and K is long, two of 256 likewise, else whole tiles.  us on B200 for 64 tokens,
// whole pairs / two slices of pairs / four of single blocks: 4096 x 4096 15.7 / 12.7 / 11.3, 4096 x 14336 46 / 30 / 26, 3072 x 2048 11.0 / 9.4 / 8.6, 6144 x 4096
// 16.6 / 13.9 / 22.5 (two rounds), 5120 x 5120 21 / 16 / 24; K of 512, 1024 x 512 4.2 / 4.8 / 5.3.  Four slices of pairs (clusters of eight) come to what four
// of single blocks do up to twelve tiles; more such clusters do not find room together (4096 x 4096 20.6).
Share share_for(int N, int nkb) {
    if (nkb >= 24 && (N + 127) / 128 <= clusters_of_four()) return {1, 4};
    if (nkb >= 16 && (N + 255) / 256 <= clusters_of_four()) return {2, 2};
    return {2, 1};
}

int batch_impl(const void* X, const void* W, void* Y, int y_dtype, int M, int N, int K, int ldx, int ldw, int ldy, int accumulate, IkGlu join,
               int way, int* status, const IkRopeStore* rope, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || K <= 0 || ldx < K || ldw < K || (!rope && ldy < (join ? N / 2 : N))) return IK_BAD_ARGUMENT;
    if ((join && ((N & 1) || accumulate)) || (join.act && accumulate)) return IK_BAD_ARGUMENT;
    if (y_dtype != IK_F32 && y_dtype != IK_BF16) return IK_BAD_ARGUMENT;
    if (M > 128 || K % 8 || ldx % 8 || ldw % 8 || ((uintptr_t)X % 16) || ((uintptr_t)W % 16)) return IK_UNSUPPORTED;
    if (!rope && (y_dtype == IK_F32 ? join || join.act : accumulate)) return IK_UNSUPPORTED;
    BatchArgs g = {};
    g.Y = Y; g.M = M; g.N = N; g.ldy = ldy; g.accumulate = accumulate; g.status = status; g.join = join;
    if (rope) g.rope = *rope;
    g.nkb = (K + BK - 1) / BK;
    if (ik_sm_count() < 2) return IK_UNSUPPORTED;
    const Share share = way ? Share{way >> 4, way & 15} : share_for(N, g.nkb);
    g.slices = share.slices;
    if ((share.cg != 1 && share.cg != 2) || (g.slices != 1 && g.slices != 2 && g.slices != 4)) return IK_BAD_ARGUMENT;
    g.tiles = (N + 128 * share.cg - 1) / (128 * share.cg);
    g.per = (g.nkb + g.slices - 1) / g.slices;
    if ((g.slices - 1) * g.per >= g.nkb) return IK_UNSUPPORTED;      // (a slice of nothing)
    const int bn = M <= 64 ? 64 : 128;
    CUtensorMap mx, mw;
    int st = ik_make_map(&mx, X, M, K, ldx, bn / share.cg);
    if (st != IK_OK) return st;
    st = ik_make_map(&mw, W, N, K, ldw, 128);
    if (st != IK_OK) return st;
    const int out = rope ? OUT_ROPE : y_dtype == IK_F32 ? OUT_F32 : join ? OUT_JOIN : join.act ? OUT_ACT : OUT_BF16;
#define IK_BATCH(OUT)                                                                                                              \
    case OUT:                                                                                                                     \
        if (share.cg == 2) return bn == 64 ? launch_batch<64, 2, OUT>(mx, mw, g, stream) : launch_batch<128, 2, OUT>(mx, mw, g, stream); \
        return bn == 64 ? launch_batch<64, 1, OUT>(mx, mw, g, stream) : launch_batch<128, 1, OUT>(mx, mw, g, stream)
    switch (out) {
        IK_BATCH(OUT_F32);
        IK_BATCH(OUT_BF16);
        IK_BATCH(OUT_JOIN);
        IK_BATCH(OUT_ACT);
        IK_BATCH(OUT_ROPE);
    }
#undef IK_BATCH
    return IK_BAD_ARGUMENT;
}

}  // namespace

// Arguments as ik_gemm_wide; way: 16 * blocks to a tile (1, 2) + slices of K (1, 2, 4), 0 = chosen.  Up to 128 tokens.
IK_EXPORT int ik_gemm_batch(const void* X, const void* W, void* Y, int y_dtype, int M, int N, int K, int ldx, int ldw, int ldy, int accumulate,
                            int swiglu, float glu_alpha, float glu_limit, float glu_shift, int way, int* status, cudaStream_t stream) {
    return batch_impl(X, W, Y, y_dtype, M, N, K, ldx, ldw, ldy, accumulate, IkGlu(swiglu, glu_alpha, glu_limit, glu_shift), way, status, nullptr, stream);
}

// As ik_gemm_qkv_rope_tcgen05.
IK_EXPORT int ik_gemm_qkv_rope_batch(const void* X, const void* W, int M, int N, int K, int ldx, int ldw, int way, int* status,
                                     const IkRopeStore* rope, cudaStream_t stream) {
    if (!rope || !rope->q_out || (rope->hd & 1) || N != (rope->nh + 2 * rope->nkv) * rope->hd) return IK_BAD_ARGUMENT;
    return batch_impl(X, W, nullptr, IK_F32, M, N, K, ldx, ldw, N, 0, IkGlu(), way, status, rope, stream);
}

// Sites: 1 = loader for a free stage, 2 = issuer for a drained accumulator, 3 = issuer for a loaded stage, 4 = epilogue, 5 = the other slices' sums.
IK_EXPORT int ik_gemm_batch_take_wait_record(int* out4) { return ik_take_wait_record(out4); }
