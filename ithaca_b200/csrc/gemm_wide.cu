// bfloat16 product on the fifth-generation tensor cores for many tokens (prompts):
//   Y[M, N] (+)= X[M, K] * W[N, K]^T,  X and W bfloat16 with K contiguous, float accumulation in TMEM.
//
// Two blocks (a cluster of two neighbouring SMs) compute one tile of 256 tokens x bn features (bn = 128, 192 or 256) with
// tcgen05.mma.cta_group::2: block r holds the accumulator of tokens 128 r .. 128 r + 127 (one TMEM lane per token, one
// column per feature), its own 128 rows of X and half of the tile's rows of W; the instruction reads the other half from
// the neighbour.  What bounds such a product is, next to the tensor pipe, what an SM takes in per K step: 32 KB here
// (128 x 64 of X and 128 x 64 of W) against 48 KB for a block that works alone on 128 x 256 (gemm_tcgen05.cu).  Grouped
// products whose token tiles have 128 rows run the same kernel with one block to a tile (CG = 1: a neighbour would belong to
// another matrix).
//
// Tokens are TMEM lanes, so a thread of the epilogue holds neighbouring features of one token: gate and up, or the two
// members of a rotary pair, meet in one thread without shuffles, and results leave through shared memory as TMA stores of
// 32 tokens x 64 or 128 bytes (adding into Y: as TMA
// reductions, one per element, so that Y is never read by the SM; a sum below 2^-126 may become zero).  Eight warps drain an
// accumulator (each 32 lanes of every other chunk of columns) while the next tile fills the other one.
//
// Measured on B200 against gemm_tcgen05.cu's pair mode (us, replayed graphs over weights larger than L2 together; cuBLAS beside):
// 2,048 tokens: gate/up 28672 x 4096 370 -> 293 (315), down 4096 x 14336 184 -> 159 (148), q/k/v 6144 x 4096 78 -> 71 (68),
// o 4096 x 4096 60 -> 49 (46), gate/up 16384 x 2048 185 -> 88 (95); 8,192 tokens: gate/up 16384 x 2048 714 -> 356 (367).  With K = 2,048
// the old epilogue (four warps, 2-byte stores, pairs joined by shuffles) took longer than a tile's 32 K steps.
//
// Roles of a block's twelve warps: warp 0 loads (TMA), warp 1 allocates TMEM and, in the block of rank 0, issues the
// products (both keep their warp together and elect a lane where they issue), warps 4..11 are the epilogue.  Barriers: "full"
// (rank 0's; the bytes of both blocks' copies are counted there), "empty" and "accumulator full" (in both blocks, by one commit
// that arrives in both), "accumulator empty" (rank 0's; one arrival per epilogue warp of both blocks).  No copy goes to more
// than one block.
//
// Every wait is bounded like those of gemm_tcgen05.cu: on expiry the status word and the block's abort flag are set, every
// role leaves its loop, the leader waits (bounded) for the copies in flight, both blocks meet, and TMEM is freed.
#define IK_FAMILY 8
#include "tc_common.cuh"
#include "rope_store.cuh"

namespace {

typedef __nv_bfloat16 bf16;
constexpr int BK = 64, THREADS = 384, EPI_WARPS = 8;
constexpr int ROWS = 128;                                          // tokens of a block's part of a tile
constexpr int A_BYTES = ROWS * BK * 2;
constexpr int STAGING = 4096;                                      // per epilogue warp
template <int CG> struct Cfg {
    static constexpr int B_BYTES = 256 / CG * BK * 2;
    static constexpr int STAGE = A_BYTES + B_BYTES;
    static constexpr int STAGES = 196608 / STAGE;                  // 6 of 32 KB, or 4 of 48 KB
    static constexpr int SMEM = STAGES * STAGE + EPI_WARPS * STAGING + 1024 + 256;
};
enum { OUT_F32 = 0, OUT_ADD = 1, OUT_BF16 = 2, OUT_JOIN = 3, OUT_ROPE = 4, OUT_ACT = 5 };

struct WideArgs {
    int M, N, K, bn, tiles_m, tiles_n, units;
    int* status;
    const int* groups;                                             // grouped: the matrix of every token tile, or -1
    IkGlu join;
    IkRopeStore rope;
};

template <int CG> __device__ __forceinline__ void load_tile(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    if (CG == 2)
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                     :: "r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                     :: "r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
template <int CG> __device__ __forceinline__ void product(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t acc) {
    if (CG == 2)
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t}"
                     :: "r"(d), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(acc) : "memory");
    else
        umma_halves(d, a_lo, b_lo, hi, idesc, acc);
}
// Arrives on the barrier (at the same place in both blocks of a pair) once the products issued so far are done.
template <int CG> __device__ __forceinline__ void commit(uint64_t* bar) {
    if (CG == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                     :: "r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
    else
        umma_commit(bar);
}
// mbar_wait for a barrier that threads of the other block arrive on.
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
__device__ __forceinline__ void st_shared16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" :: "r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&p);
}
template <int KIND> __device__ __forceinline__ void activate(float* v) {
    #pragma unroll
    for (int i = 0; i < 64; i++) v[i] = ik_plain_act_value(v[i], KIND);
}
template <bool ADD> __device__ __forceinline__ void store_tile(const CUtensorMap* map, uint32_t src, int x, int y) {
    if (ADD)
        asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
                     :: "l"(map), "r"(src), "r"(x), "r"(y) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];"
                     :: "l"(map), "r"(src), "r"(x), "r"(y) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// The tiles of a cluster in order: units cluster, cluster + clusters, ...  Plain: bands of eight token tiles, weight tiles
// outside, so that the clusters at work at one time share about eight token tiles and nine weight tiles, whose K steps come
// from L2 once fetched.  Grouped: the weight tiles of a token tile follow one another (see gemm_tcgen05.cu).
struct Tiles {
    int unit, step, units, tiles_m, tiles_n;
    const int* groups;
    int mt, nt, group;
    __device__ bool next() {
        for (;; unit += step) {
            if (unit >= units) return false;
            group = 0;
            if (groups) {
                mt = unit / tiles_n;
                nt = unit - mt * tiles_n;
                asm volatile("ld.global.s32 %0, [%1];" : "=r"(group) : "l"(groups + mt) : "memory");
                if (group < 0) continue;
            } else {
                const int band = unit / (8 * tiles_n), in = unit - band * 8 * tiles_n;
                const int high = min(8, tiles_m - band * 8);
                nt = in / high;
                mt = band * 8 + (in - nt * high);
            }
            unit += step;
            return true;
        }
    }
};

template <int CG, int OUT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_y,
                 const __grid_constant__ WideArgs g) {
    typedef Cfg<CG> C;
    constexpr int NST = C::STAGES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* staging = tiles + NST * C::STAGE;
    uint64_t* full = (uint64_t*)(staging + EPI_WARPS * STAGING);
    uint64_t* empty = full + NST;
    uint64_t* acc_full = empty + NST;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = CG == 2 ? blockIdx.x & 1 : 0;
    int* const status = g.status;
    if (CG == 1 && ik_status_has(status, IK_STATUS_GEMM_TIMEOUT)) return;       // (a pair goes on to its barriers; its waits are bounded)
    const int bn = g.bn, nkb = (g.K + BK - 1) / BK;
    const uint32_t bytes = A_BYTES + bn / CG * BK * 2;                 // what a K step brings into one block

    if (threadIdx.x == 0) {
        for (int s = 0; s < NST; s++) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        for (int b = 0; b < 2; b++) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, CG * EPI_WARPS); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&map_x) : "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&map_w) : "memory");
        if (OUT != OUT_ROPE) asm volatile("prefetch.tensormap [%0];" :: "l"(&map_y) : "memory");
    }
    if (warp == 1) {
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    if (CG == 2) cluster_sync();                       // both blocks' barriers exist before either is arrived on from outside
    const Tiles first = {(int)(blockIdx.x / CG), (int)(gridDim.x / CG), g.units, g.tiles_m, g.tiles_n, g.groups, 0, 0, 0};

    // Weights are written by no kernel: those of the first stages are asked for before the wait for the kernel before.
    int pre = 0;
    if (threadIdx.x == 0 && !g.groups) {
        Tiles t = first;
        while (pre < NST && t.next())
            for (int i = 0; i < nkb && pre < NST; i++, pre++) {
                if (rank == 0) mbar_expect_tx(full + pre, CG * bytes);
                load_tile<CG>(tiles + pre * C::STAGE + A_BYTES, &map_w, i * BK, t.nt * bn + (int)rank * (bn / CG), cluster_addr(smem_u32(full + pre), 0));
            }
    }
    ik_pdl_wait();
    ik_pdl_launch_dependents();

    if (warp == 0) {
        int it = 0, s = 0;
        uint32_t phase = 1;                            // of the next wait for a free stage
        bool ok = true;
        const int n_pre = __shfl_sync(0xffffffffu, pre, 0);
        const uint32_t full0 = cluster_addr(smem_u32(full), 0);
        for (Tiles t = first; ok && t.next();) {
            const int m0 = t.mt * (CG * ROWS) + (int)rank * ROWS, n0 = t.group * g.N + t.nt * bn + (int)rank * (bn / CG);
            for (int i = 0; i < nkb; i++, it++) {
                unsigned char* a = tiles + s * C::STAGE;
                if (it >= n_pre) {
                    ok = __all_sync(0xffffffffu, mbar_wait(empty + s, phase, abort_flag, status, IK_WAIT_LIMIT_NS, 1, it));
                    if (!ok) break;
                }
                if (elect_one()) {
                    const uint32_t bar = full0 + s * 8;
                    if (it >= n_pre) {
                        if (rank == 0) mbar_expect_tx(full + s, CG * bytes);
                        load_tile<CG>(a + A_BYTES, &map_w, i * BK, n0, bar);
                    }
                    load_tile<CG>(a, &map_x, i * BK, m0, bar);
                }
                __syncwarp();
                if (++s == NST) { s = 0; phase ^= 1; }
            }
        }
        if (*abort_flag && rank == 0 && lane == 0) {   // leave no copy in flight: the stages armed last
            for (int i = max(0, it - NST); i < it; i++) {
                const long long c0 = wait_clock();
                while (!mbar_test(full + i % NST, (i / NST) & 1) && !wait_ran_out(c0, 2000000ull)) {}
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(CG * 128 >> 4) << 24);
            const uint32_t hi = umma_desc_hi(), lo0 = umma_desc_lo(smem_u32(tiles));
            int it = 0, lt = 0, s = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (Tiles t = first; ok && t.next(); lt++) {
                const int buf = lt & 1;
                ok = __all_sync(0xffffffffu, wait_cluster(acc_empty + buf, ((lt >> 1) & 1) ^ 1, abort_flag, status, 2, lt));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + buf * 256;
                for (int i = 0; i < nkb; i++, it++) {
                    ok = __all_sync(0xffffffffu, mbar_wait(full + s, phase, abort_flag, status, IK_WAIT_LIMIT_NS, 3, it));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_lo = lo0 + (uint32_t)s * (C::STAGE >> 4), b_lo = a_lo + (A_BYTES >> 4);
                    if (elect_one()) {
                        #pragma unroll
                        for (int j = 0; j < BK / 16; j++) product<CG>(acc, a_lo + 2 * j, b_lo + 2 * j, hi, idesc, (i | j) != 0);
                        commit<CG>(empty + s);
                    }
                    __syncwarp();
                    if (++s == NST) { s = 0; phase ^= 1; }
                }
                if (ok && elect_one()) commit<CG>(acc_full + buf);
                __syncwarp();
            }
        }
    } else if (warp >= 4) {
        const int quarter = warp & 3, half = (warp - 4) >> 2;
        const uint32_t stage = smem_u32(staging) + (warp - 4) * STAGING;
        constexpr int CHUNK = OUT <= OUT_ADD ? 32 : 64;                // columns of the accumulator that leave together
        int lt = 0;
        for (Tiles t = first; t.next(); lt++) {
            const int buf = lt & 1, n0 = t.nt * bn, m0 = t.mt * (CG * ROWS) + (int)rank * ROWS + quarter * 32;
            int cache_row = -1;
            if (OUT == OUT_ROPE) cache_row = ik_rope_cache_row(g.rope, m0 + lane, g.M);
            if (!mbar_wait(acc_full + buf, (lt >> 1) & 1, abort_flag, status, IK_WAIT_LIMIT_NS, 4, lt)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + buf * 256;
            #pragma unroll 1
            for (int c0 = half * CHUNK; c0 < bn; c0 += 2 * CHUNK) {
                const int f = n0 + c0;
                if (f >= g.N || m0 >= g.M) break;
                float v[CHUNK];
                if (OUT == OUT_ROPE) {
                    const IkRopeStore& e = g.rope;
                    const int head = f / e.hd, r0 = f - head * e.hd;           // (64 columns lie in one head)
                    const bool is_q = head < e.nh, rotated = head < e.nh + e.nkv;
                    float cs[64];
                    const int m = min(m0 + lane, g.M - 1);
                    if (rotated) {
                        const float* src = e.cos_sin + ((size_t)m * (e.hd >> 1) + (r0 >> 1)) * 2;
                        #pragma unroll
                        for (int i = 0; i < 16; i++)
                            asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];"
                                         : "=f"(cs[4 * i]), "=f"(cs[4 * i + 1]), "=f"(cs[4 * i + 2]), "=f"(cs[4 * i + 3]) : "l"(src + 4 * i));
                    }
                    #pragma unroll
                    for (int i = 0; i < 4; i++) tmem_ld16_issue(acc + c0 + 16 * i, v + 16 * i);
                    tmem_ld_wait();
                    if (e.bias) {
                        #pragma unroll
                        for (int i = 0; i < 64; i++) v[i] += __ldg(e.bias + f + i);
                    }
                    uint32_t out[32];
                    #pragma unroll
                    for (int i = 0; i < 32; i++) {
                        const float a = v[2 * i], b = v[2 * i + 1];
                        out[i] = rotated ? pack2(a * cs[2 * i] - b * cs[2 * i + 1], a * cs[2 * i + 1] + b * cs[2 * i]) : pack2(a, b);
                    }
                    __syncwarp();                                       // the rows of the chunk before have been read
                    #pragma unroll
                    for (int j = 0; j < 8; j++)
                        st_shared16(stage + lane * 128 + ((j ^ (lane & 7)) << 4), out[4 * j], out[4 * j + 1], out[4 * j + 2], out[4 * j + 3]);
                    __syncwarp();
                    // four tokens' 128 bytes per instruction
                    bf16* const kv = (rotated ? e.k_pages : e.v_pages) + (size_t)(is_q ? 0 : head - e.nh - (rotated ? 0 : e.nkv)) * e.page_size * e.hd + r0;
                    const int seg = lane & 7;
                    #pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int row = 4 * i + (lane >> 3);
                        const int at = __shfl_sync(0xffffffffu, cache_row, row);
                        uint4 w;
                        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w)
                                     : "r"(stage + row * 128 + ((seg ^ (row & 7)) << 4)));
                        if (is_q) {
                            if (m0 + row < g.M)
                                *reinterpret_cast<uint4*>(e.q_out + ((size_t)(m0 + row) * e.nh + head) * e.hd + r0 + seg * 8) = w;
                        } else if (at >= 0) {
                            *reinterpret_cast<uint4*>(kv + (size_t)at * e.hd + seg * 8) = w;
                        }
                    }
                    continue;
                }
                #pragma unroll
                for (int i = 0; i < CHUNK / 16; i++) tmem_ld16_issue(acc + c0 + 16 * i, v + 16 * i);
                tmem_ld_wait();
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");    // the chunk before has left the staging room
                __syncwarp();
                if (OUT <= OUT_ADD) {
                    #pragma unroll
                    for (int j = 0; j < 8; j++)
                        st_shared16(stage + lane * 128 + ((j ^ (lane & 7)) << 4), __float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]),
                                    __float_as_uint(v[4 * j + 2]), __float_as_uint(v[4 * j + 3]));
                } else if (OUT == OUT_BF16 || OUT == OUT_ACT) {
                    // the activation has an instance of its own and its kind is chosen once a chunk: chosen for every value, the
                    // code of 64 hyperbolic tangents stood between plain ones (us on B200, 16-bit results without activation:
                    // 2048 x 2048 x 2048 23.7 -> 15.6, 2048 x 16384 x 2048 102 -> 91, 513 x 8192 x 256 23.8 -> 7.8; gelu 27 -> 19, 120 -> 99)
                    if (OUT == OUT_ACT) {
                        if (g.join.act == 1) activate<0>(v);
                        else if (g.join.act == 2) activate<1>(v);
                        else activate<2>(v);
                    }
                    uint32_t out[32];
                    #pragma unroll
                    for (int i = 0; i < 32; i++) out[i] = pack2(v[2 * i], v[2 * i + 1]);
                    #pragma unroll
                    for (int j = 0; j < 8; j++)
                        st_shared16(stage + lane * 128 + ((j ^ (lane & 7)) << 4), out[4 * j], out[4 * j + 1], out[4 * j + 2], out[4 * j + 3]);
                } else {                                               // columns (2j, 2j + 1) are gate j and up j: rows of 32 results, 64-byte swizzle
                    uint32_t out[16];
                    #pragma unroll
                    for (int i = 0; i < 16; i++)
                        out[i] = pack2(ik_glu_join_fast(g.join, v[4 * i], v[4 * i + 1]), ik_glu_join_fast(g.join, v[4 * i + 2], v[4 * i + 3]));
                    #pragma unroll
                    for (int j = 0; j < 4; j++)
                        st_shared16(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4), out[4 * j], out[4 * j + 1], out[4 * j + 2], out[4 * j + 3]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) store_tile<OUT == OUT_ADD>(&map_y, stage, OUT == OUT_JOIN ? f >> 1 : f, m0);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_addr(smem_u32(acc_empty + buf), 0));
        }
        if (OUT != OUT_ROPE && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (CG == 2) cluster_sync();                       // neither block leaves, or gives its TMEM back, while the other still works
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u) : "memory");
    }
}

// rows x cols matrix, cols contiguous; box = 32 rows x box_cols elements (box_cols * size = the swizzle's width); writes
// outside the matrix are left out.
int make_out_map(CUtensorMap* map, void* base, bool f32, unsigned long long rows, int cols, unsigned long long ld, int box_cols) {
    IkEncodeTiled enc = ik_encode_fn();
    if (!enc) return IK_UNSUPPORTED;
    const int size = f32 ? 4 : 2;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * size};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, 32u};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols * size == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? IK_OK : IK_BAD_ARGUMENT;
}

template <int CG, int OUT>
int launch_wide(const CUtensorMap& mx, const CUtensorMap& mw, const CUtensorMap& my, const WideArgs& g, cudaStream_t stream) {
    auto kern = gemm_wide_kernel<CG, OUT>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<CG>::SMEM);
    if (e != cudaSuccess) return (int)e;
    const int most = ik_sm_count() / CG;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(CG * (g.units < most ? g.units : most)));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = Cfg<CG>::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CG; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (ik_pdl_mask() & IK_FAMILY) ? 2 : 1;
    IK_RETURN_IF_ERROR(cudaLaunchKernelEx(&cfg, kern, mx, mw, my, g));
    return (int)cudaGetLastError();
}

// Features of a tile: of 256, 192 and 128 the one whose tiles take the least time in whole rounds over the pairs of SMs.
// A K step of a tile takes 0.34, 0.27 or 0.225 us (measured, all SMs at work): the loads and the issuing thread bind where the
// tensor pipe (0.27, 0.2, 0.135 us) does not.
int wide_width(long long tiles_m, int N, int pairs) {
    int best = 256;
    long long best_cost = -1;
    for (int bn = 256; bn >= 128; bn -= 64) {
        const long long rounds = (tiles_m * ((N + bn - 1) / bn) + pairs - 1) / pairs;
        const long long cost = rounds * (bn == 256 ? 340 : bn == 192 ? 270 : 225);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = bn; }
    }
    return best;
}

// A grouped plan has a tile to spare for every group, since any group may end in one that is partly filled; on average half of them are
// in use.  Counted in full they chose the width for work that is not there (us on B200, 8 experts, 4,096 x 14,336, 300 tokens of 2
// experts each 205 -> 157, 2,048 tokens 626 -> 431; 16 of 1,024 x 512, 600 tokens 10.1 -> 8.6).
int tiles_in_use(int tiles, int n_groups) { return tiles - n_groups / 2 > 1 ? tiles - n_groups / 2 : 1; }

int wide_impl(const void* X, const void* W, void* Y, int y_dtype, int M, int N, int K, int ldx, int ldw, int ldy, int accumulate,
              IkGlu join, const int* groups, int n_groups, int tile_rows, int bn, int* status, const IkRopeStore* rope, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || K <= 0 || ldx < K || ldw < K || (!rope && ldy < (join ? N / 2 : N))) return IK_BAD_ARGUMENT;
    if ((join && ((N & 1) || accumulate)) || (join.act && accumulate)) return IK_BAD_ARGUMENT;
    if (y_dtype != IK_F32 && y_dtype != IK_BF16) return IK_BAD_ARGUMENT;
    if (K % 8 || ldx % 8 || ldw % 8 || ((uintptr_t)X % 16) || ((uintptr_t)W % 16)) return IK_UNSUPPORTED;
    const bool f32 = y_dtype == IK_F32;
    int out;
    if (rope) {
        if (rope->hd % 64 || ((uintptr_t)rope->q_out % 16) || ((uintptr_t)rope->k_pages % 16) || ((uintptr_t)rope->v_pages % 16) ||
            ((uintptr_t)rope->cos_sin % 16)) return IK_UNSUPPORTED;
        out = OUT_ROPE;
    } else {
        // results leave as TMA tiles: 16-byte rows
        if (((uintptr_t)Y % 16) || ((long long)ldy * (f32 ? 4 : 2)) % 16) return IK_UNSUPPORTED;
        if (f32 ? (join || join.act) : accumulate) return IK_UNSUPPORTED;
        out = f32 ? (accumulate ? OUT_ADD : OUT_F32) : join ? OUT_JOIN : join.act ? OUT_ACT : OUT_BF16;
    }
    if (groups && tile_rows != 128 && tile_rows != 256) return IK_UNSUPPORTED;
    const int cg = groups && tile_rows == 128 ? 1 : 2;
    WideArgs g = {};
    g.M = M; g.N = N; g.K = K; g.status = status; g.groups = groups; g.join = join;
    if (rope) g.rope = *rope;
    g.tiles_m = (M + cg * ROWS - 1) / (cg * ROWS);
    const int pairs = ik_sm_count() / cg;
    if (pairs < 1) return IK_UNSUPPORTED;
    g.bn = bn ? bn : wide_width(tiles_in_use(g.tiles_m, groups ? n_groups : 0), N, pairs);
    if (g.bn != 128 && g.bn != 192 && g.bn != 256) return IK_BAD_ARGUMENT;
    g.tiles_n = (N + g.bn - 1) / g.bn;
    if ((long long)g.tiles_m * g.tiles_n > 0x3fffffff) return IK_UNSUPPORTED;
    g.units = g.tiles_m * g.tiles_n;
    CUtensorMap mx, mw, my = {};
    int st = ik_make_map(&mx, X, M, K, ldx, ROWS);
    if (st != IK_OK) return st;
    st = ik_make_map(&mw, W, (unsigned long long)N * n_groups, K, ldw, g.bn / cg);
    if (st != IK_OK) return st;
    if (!rope) {
        st = make_out_map(&my, Y, f32, M, join ? N / 2 : N, ldy, out == OUT_BF16 || out == OUT_ACT ? 64 : 32);
        if (st != IK_OK) return st;
    }
    if (cg == 1) {
        switch (out) {
            case OUT_F32: return launch_wide<1, OUT_F32>(mx, mw, my, g, stream);
            case OUT_BF16: return launch_wide<1, OUT_BF16>(mx, mw, my, g, stream);
            case OUT_JOIN: return launch_wide<1, OUT_JOIN>(mx, mw, my, g, stream);
            case OUT_ACT: return launch_wide<1, OUT_ACT>(mx, mw, my, g, stream);
            default: return IK_UNSUPPORTED;
        }
    }
    switch (out) {
        case OUT_F32: return launch_wide<2, OUT_F32>(mx, mw, my, g, stream);
        case OUT_ADD: return launch_wide<2, OUT_ADD>(mx, mw, my, g, stream);
        case OUT_BF16: return launch_wide<2, OUT_BF16>(mx, mw, my, g, stream);
        case OUT_JOIN: return launch_wide<2, OUT_JOIN>(mx, mw, my, g, stream);
        case OUT_ACT: return launch_wide<2, OUT_ACT>(mx, mw, my, g, stream);
        default: return launch_wide<2, OUT_ROPE>(mx, mw, my, g, stream);
    }
}

}  // namespace

// Arguments as ik_gemm_tcgen05 without scratch and sharing; bn: features of a tile (128, 192, 256; 0 = chosen).
// IK_UNSUPPORTED where results cannot leave as TMA tiles (rows of Y not on 16 bytes) or the epilogue is another one.
IK_EXPORT int ik_gemm_wide(const void* X, const void* W, void* Y, int y_dtype, int M, int N, int K, int ldx, int ldw, int ldy,
                           int accumulate, int swiglu, float glu_alpha, float glu_limit, float glu_shift, int bn, int* status,
                           cudaStream_t stream) {
    return wide_impl(X, W, Y, y_dtype, M, N, K, ldx, ldw, ldy, accumulate, IkGlu(swiglu, glu_alpha, glu_limit, glu_shift), nullptr, 1, 0,
                     bn, status, nullptr, stream);
}

// As ik_gemm_tcgen05_grouped for token tiles of 128 or 256 rows.
IK_EXPORT int ik_gemm_wide_grouped(const void* X, const void* W, void* Y, int y_dtype, const int* tile_group, int n_groups, int tile_rows,
                                   int M, int N, int K, int ldx, int ldw, int ldy, int swiglu, int* status, cudaStream_t stream) {
    if (!tile_group || n_groups < 1 || tile_rows < 1 || M % tile_rows) return IK_BAD_ARGUMENT;
    if (M == 0) return IK_OK;
    return wide_impl(X, W, Y, y_dtype, M, N, K, ldx, ldw, ldy, 0, IkGlu(swiglu, 1.f, 0.f, 0.f), tile_group, n_groups, tile_rows, 0,
                     status, nullptr, stream);
}

// As ik_gemm_qkv_rope_tcgen05, for heads of a multiple of 64.
IK_EXPORT int ik_gemm_qkv_rope_wide(const void* X, const void* W, int M, int N, int K, int ldx, int ldw, int bn, int* status,
                                    const IkRopeStore* rope, cudaStream_t stream) {
    if (!rope || !rope->q_out || (rope->hd & 1) || N != (rope->nh + 2 * rope->nkv) * rope->hd) return IK_BAD_ARGUMENT;
    return wide_impl(X, W, nullptr, IK_F32, M, N, K, ldx, ldw, N, 0, IkGlu(), nullptr, 1, 0, bn, status, rope, stream);
}

// The width of tiles that is chosen for `tiles` token tiles (of which a grouped plan of n_groups keeps some to spare) on so many SMs or pairs.
IK_EXPORT int ik_gemm_wide_tile_width(int tiles, int n_groups, int N, int pairs) {
    if (tiles <= 0 || n_groups < 0 || N <= 0 || pairs <= 0) return 0;
    return wide_width(tiles_in_use(tiles, n_groups), N, pairs);
}

// Sites: 1 = loader for a free stage, 2 = issuer for a drained accumulator, 3 = issuer for a loaded stage, 4 = epilogue.
IK_EXPORT int ik_gemm_wide_take_wait_record(int* out4) { return ik_take_wait_record(out4); }
