// Product of the 32-bit path with 16-bit weights on the fifth-generation tensor cores:
//   Y[M, N] (+)= X[M, K] * W[N, K]^T,  X and Y float, W bfloat16, K contiguous.
//
// A float is the sum of three bfloat16 numbers without a remainder (its 24 significant bits in three eights), and a product of two
// bfloat16 numbers is a float without rounding.  So X goes to the tensor core as three planes, each multiplied by W, and nothing is lost
// before the sums.  (The small planes are stored 2^7 and 2^15 times too large, and what has been summed is scaled down where the next plane's
// products begin, so that a small number's last bits do not fall below 2^-133, the least bfloat16; only the last bit of a number below 2^-125
// does.)  The sums are what the error comes from: tcgen05.mma drops the bits that do not fit when it adds to its accumulator, always towards zero, so a long chain of them leans.  Here a chain is 64 k: eight instructions for
// the two small planes, then four for the large one.  The chain's sum is taken out of TMEM and added to a float in registers,
// rounded to nearest, while the next chains run in other columns of TMEM.  Slices of K, cut by K alone, join in their order what Y
// holds: a row of Y has the same bits whatever other rows are in the call, whatever tile takes it, and whether the slices run one after another in one
// block or side by side.
// Error against 64 bits (2-norm; gemm_simt.cu / this): normal X and W, K = 256 2.9e-7 / 0.9e-7, 2,048 8.1e-7 / 1.3e-7, 14,336 2.2e-6 /
// 1.4e-7; all positive 2.5e-7 / 1.0e-7, 6.2e-7 / 1.1e-7, 1.8e-6 / 1.0e-7; X over several powers of e 2.8e-7 / 1.2e-7, 8.4e-7 / 1.6e-7, 2.3e-6 / 1.6e-7.
// (Chains of 128 k, the planes in turn: 3.3e-7, and 9e-7 where all is positive.)
//
// Two blocks (a cluster of two neighbouring SMs) compute 256 features x bn tokens (bn = 32, 64, 128, 256) with cta_group::2: each
// holds 128 rows of W (TMEM lanes) and half of the tokens' rows of the three planes.  A stage of 64 k brings 16 KB of W and 192 bytes a
// token into a block for 12 products: W is read once for the three planes.  Lanes are features, so a warp stores 32
// neighbouring features of a token at a time.
// What bounds it: with many tokens the tensor pipe (three times the operations of a 16-bit product; at work 86 % of the cycles with 2,048 tokens x 16384 x
// 2048), with few the bytes of W and the start.
// Measured on B200 (us in replayed graphs, with the kernels that form the planes and add the slices; gemm_simt.cu / this): 2,048 tokens x 16384 x
// 2048 2,446 / 276 (498 TFLOP/s), 2048 x 8192 1,443 / 179; 465 tokens 737 / 76, 475 / 47; 1 token 177 / 15, 302 / 17; 128256 x 2048 for 3 tokens 861 / 84.
#include <type_traits>
#define IK_FAMILY 8
#include "tc_common.cuh"

namespace {

typedef __nv_bfloat16 bf16;
constexpr int BK = 64;
constexpr int A_BYTES = 128 * BK * 2;
constexpr int MAX_SLICES = 8;
constexpr int MID_SCALE = 7, LOW_SCALE = 15;          // powers of two by which the small planes are stored too large
template <int BN> struct Cfg {
    static constexpr int PLANE = BN / 2 * BK * 2;                  // a block's half of the tokens, one plane
    static constexpr int STAGE = A_BYTES + 3 * PLANE;
    static constexpr int STAGES = 204800 / STAGE;                  // 9, 7, 5, 3
    static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
    static constexpr int BUFS = BN == 256 ? 2 : 4;                 // K steps in TMEM
    static constexpr int TMEM = BUFS * BN;                         // columns (128 to 512)
    static constexpr int EPI_WARPS = BN == 256 ? 16 : 8;           // so that a thread's sums stay in registers
    static constexpr int THREADS = 128 + 32 * EPI_WARPS;
};

struct SplitArgs {
    float* Y;                                                      // results, or the slices' sums [slice][M][N]
    int M, N, ldy, nkb, slices, per, tiles_m, units, side_by_side, accumulate;
    int* status;
};

__device__ __forceinline__ void load_pair_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 :: "r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void load_pair_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 :: "r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
// D = A B + D 2^-SCALE (acc = 0: D = A B).
template <int SCALE>
__device__ __forceinline__ void product_pair(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t acc) {
    if (SCALE)
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p, %6;\n\t}"
                     :: "r"(d), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(acc), "n"(SCALE) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t}"
                     :: "r"(d), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(acc) : "memory");
}
// Arrives on the barrier (at the same place in both blocks) once the products issued so far are done.
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 :: "r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
// Arrives on a barrier of a block of the cluster.  What is handed over is TMEM, ordered by the tcgen05 fences on both sides, so neither the
// arrival nor the wait for it orders other memory between the blocks: a release and an acquire at cluster scope there, once
// a K step, made a step last 0.9 to 1.0 us whatever its width.
__device__ __forceinline__ void arrive_in_cluster(uint32_t addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" :: "r"(addr) : "memory");
}

// A unit of work: a tile and the slices of K that it takes (all, or one where they run side by side).  Token tiles follow one another, so
// that pairs at work at one time read the same weights.
struct Unit {
    int mt, nt, s0, s1;
    __device__ Unit(const SplitArgs& g, int u) {
        const int rest = u / g.tiles_m;
        mt = u - rest * g.tiles_m;
        if (g.side_by_side) { nt = rest / g.slices; s0 = rest - nt * g.slices; s1 = s0 + 1; }
        else { nt = rest; s0 = 0; s1 = g.slices; }
    }
};

template <int BN>
__global__ void __launch_bounds__(Cfg<BN>::THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ SplitArgs g) {
    typedef Cfg<BN> C;
    constexpr int NST = C::STAGES, PLANE = C::PLANE, BUFS = C::BUFS, EPI_WARPS = C::EPI_WARPS;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(tiles + NST * C::STAGE);
    uint64_t* empty = full + NST;
    uint64_t* acc_full = empty + NST;
    uint64_t* acc_empty = acc_full + BUFS;
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + BUFS);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = blockIdx.x & 1;
    int* const status = g.status;
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NST; s++) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        for (int b = 0; b < BUFS; b++) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, 2 * EPI_WARPS); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&map_x) : "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&map_w) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tmem_slot)), "r"((uint32_t)C::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    cluster_sync();                                    // both blocks' barriers exist before either is arrived on from outside

    // Weights are written by no kernel: those of the first stages are asked for before the wait for the kernel before.
    int pre = 0;
    if (threadIdx.x == 0) {
        for (int u = first; u < g.units && pre < NST; u += step) {
            const Unit t(g, u);
            for (int i = t.s0 * g.per; i < min(g.nkb, t.s1 * g.per) && pre < NST; i++, pre++) {
                if (rank == 0) mbar_expect_tx(full + pre, 2 * C::STAGE);
                load_pair_2d(smem_u32(tiles + pre * C::STAGE), &map_w, i * BK, t.nt * 256 + (int)rank * 128, cluster_addr(smem_u32(full + pre), 0));
            }
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
        for (int u = first; ok && u < g.units; u += step) {
            const Unit t(g, u);
            const int n0 = t.nt * 256 + (int)rank * 128, m0 = t.mt * BN + (int)rank * (BN / 2);
            for (int i = t.s0 * g.per; i < min(g.nkb, t.s1 * g.per); i++, it++) {
                if (it >= n_pre) {
                    ok = __all_sync(0xffffffffu, mbar_wait(empty + s, phase, abort_flag, status, IK_WAIT_LIMIT_NS, 1, it));
                    if (!ok) break;
                }
                if (elect_one()) {
                    const uint32_t bar = full0 + s * 8, a = smem_u32(tiles + s * C::STAGE);
                    if (it >= n_pre) {
                        if (rank == 0) mbar_expect_tx(full + s, 2 * C::STAGE);
                        load_pair_2d(a, &map_w, i * BK, n0, bar);
                    }
                    load_pair_3d(a + A_BYTES, &map_x, i * BK, m0, 0, bar);
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
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
            const uint32_t hi = umma_desc_hi(), lo0 = umma_desc_lo(smem_u32(tiles));
            int it = 0, s = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int u = first; ok && u < g.units; u += step) {
                const Unit t(g, u);
                for (int i = t.s0 * g.per; i < min(g.nkb, t.s1 * g.per); i++, it++) {
                    const int buf = it % BUFS;
                    ok = __all_sync(0xffffffffu, mbar_wait(acc_empty + buf, ((it / BUFS) & 1) ^ 1, abort_flag, status, IK_WAIT_LIMIT_NS, 2, it)) &&
                         __all_sync(0xffffffffu, mbar_wait(full + s, phase, abort_flag, status, IK_WAIT_LIMIT_NS, 3, it));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t acc = tmem + buf * BN, a_lo = lo0 + (uint32_t)s * (C::STAGE >> 4), b_lo = a_lo + (A_BYTES >> 4);
                    if (elect_one()) {
                        // the small planes first: their sums are far below the last bit of the large one's
                        auto product = [&](auto scale, int p, int j) {
                            product_pair<decltype(scale)::value>(acc, a_lo + 2 * j, b_lo + p * (PLANE >> 4) + 2 * j, hi, idesc, (uint32_t)(p != 2 || j != 0));
                        };
                        product(std::integral_constant<int, 0>(), 2, 0);
                        #pragma unroll
                        for (int j = 1; j < BK / 16; j++) product(std::integral_constant<int, 0>(), 2, j);
                        product(std::integral_constant<int, LOW_SCALE - MID_SCALE>(), 1, 0);
                        #pragma unroll
                        for (int j = 1; j < BK / 16; j++) product(std::integral_constant<int, 0>(), 1, j);
                        product(std::integral_constant<int, MID_SCALE>(), 0, 0);
                        #pragma unroll
                        for (int j = 1; j < BK / 16; j++) product(std::integral_constant<int, 0>(), 0, j);
                        commit_pair(empty + s);
                        commit_pair(acc_full + buf);
                    }
                    __syncwarp();
                    if (++s == NST) { s = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp >= 4) {
        constexpr int COLS = 4 * BN / EPI_WARPS;                        // tokens of a thread
        const int quarter = warp & 3, part = (warp - 4) >> 2;
        const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + part * COLS;
        int it = 0;
        bool ok = true;
        for (int u = first; ok && u < g.units; u += step) {
            const Unit t(g, u);
            const int f = t.nt * 256 + (int)rank * 128 + quarter * 32 + lane, m0 = t.mt * BN + part * COLS;
            const size_t ld = g.side_by_side ? g.N : g.ldy;
            float* const y = g.Y + (g.side_by_side ? (size_t)t.s0 * g.M * g.N : 0) + m0 * ld + f;
            for (int sl = t.s0; ok && sl < t.s1; sl++) {
                float sum[COLS];
                #pragma unroll
                for (int j = 0; j < COLS; j++) sum[j] = 0.f;
                const int k1 = min(g.nkb, (sl + 1) * g.per);
                for (int i = sl * g.per; i < k1; i++, it++) {
                    const int buf = it % BUFS;
                    ok = mbar_wait(acc_full + buf, (it / BUFS) & 1, abort_flag, status, IK_WAIT_LIMIT_NS, 4, it);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    #pragma unroll
                    for (int c = 0; c < COLS; c += 16) {
                        float v[16];
                        tmem_ld16_issue(acc + buf * BN + c, v);
                        tmem_ld_wait();
                        #pragma unroll
                        for (int j = 0; j < 16; j++) sum[c + j] += v[j];
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) arrive_in_cluster(cluster_addr(smem_u32(acc_empty + buf), 0));
                }
                if (!ok || f >= g.N) continue;
                // the slice joins what the slices before it (and Y) came to
                const bool first_of_all = g.side_by_side || (sl == 0 && !g.accumulate);
                float* at = y;
                #pragma unroll
                for (int c = 0; c < COLS; c += 8) {
                    asm volatile("" : "+l"(at));                        // (one address at a time, not one for each of the thread's tokens)
                    float old[8];
                    if (!first_of_all) {
                        #pragma unroll
                        for (int j = 0; j < 8; j++) old[j] = m0 + c + j < g.M ? at[j * ld] : 0.f;
                    }
                    #pragma unroll
                    for (int j = 0; j < 8; j++)
                        if (m0 + c + j < g.M) at[j * ld] = first_of_all ? sum[c + j] : old[j] + sum[c + j];
                    at += 8 * ld;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();                                    // neither block leaves, or gives its TMEM back, while the other still works
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"((uint32_t)C::TMEM) : "memory");
    }
}

// The leading eight significant bits of a float, cut off and not rounded: a large float does not become infinite, and the planes have one sign.  Where
// nothing would be left for the next plane, one step less: no plane of a float from 2^-117 on is zero, so that an infinite weight gives the
// infinity it gives beside the number itself, and not 0 * inf.
__device__ __forceinline__ float leading(float v) {
    const uint32_t bits = __float_as_uint(v), h = bits & 0xffff0000u;
    return __uint_as_float(h == bits && (h & 0x7fff0000u) > 0x10000u ? h - 0x10000u : h);
}
// The three planes of eight neighbouring floats of a row; infinities and NaN are the same in all three.
__global__ void __launch_bounds__(256) split_planes_kernel(const float* __restrict__ X, bf16* __restrict__ planes, int M, int K, size_t ldx, int vec) {
    ik_pdl_wait();
    IK_AFTER_WAIT(X);
    ik_pdl_launch_dependents();
    const int per_row = K / 8;
    const size_t at = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (at >= (size_t)M * per_row) return;
    const size_t m = at / per_row;
    const int k = (int)(at - m * per_row) * 8;
    const float* x = X + m * ldx + k;
    float v[8];
    if (vec) {
        const float4 a = *reinterpret_cast<const float4*>(x), b = *reinterpret_cast<const float4*>(x + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
        #pragma unroll
        for (int i = 0; i < 8; i++) v[i] = x[i];
    }
    uint32_t out[3][4];
    #pragma unroll
    for (int i = 0; i < 8; i += 2) {
        uint32_t part[2][3];
        #pragma unroll
        for (int e = 0; e < 2; e++) {
            const uint32_t bits = __float_as_uint(v[i + e]);
            if ((bits & 0x7f800000u) != 0x7f800000u) {
                const float h = leading(v[i + e]), rest = (v[i + e] - h) * (float)(1 << MID_SCALE), mid = leading(rest);
                part[e][0] = __float_as_uint(h);
                part[e][1] = __float_as_uint(mid);
                part[e][2] = __float_as_uint((rest - mid) * (float)(1 << (LOW_SCALE - MID_SCALE))) & 0xffff0000u;
            } else {                                                   // (a NaN whose mark lies in the bits that are cut off)
                part[e][0] = part[e][1] = part[e][2] = (bits & 0xffff0000u) | ((bits & 0x7fffffu) ? 0x400000u : 0u);
            }
        }
        #pragma unroll
        for (int p = 0; p < 3; p++) out[p][i / 2] = (part[0][p] >> 16) | part[1][p];
    }
    #pragma unroll
    for (int p = 0; p < 3; p++)
        *reinterpret_cast<uint4*>(planes + ((size_t)p * M + m) * K + k) = make_uint4(out[p][0], out[p][1], out[p][2], out[p][3]);
}

// What Y held and the slices' sums, in order.
template <typename V>
__global__ void __launch_bounds__(256) split_sum_kernel(const float* __restrict__ partial, float* __restrict__ Y, int M, int N, int ldy, int slices, int accumulate) {
    constexpr int W = sizeof(V) / 4;
    ik_pdl_wait();
    IK_AFTER_WAIT(partial);
    ik_pdl_launch_dependents();
    const int per_row = N / W;
    const size_t at = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (at >= (size_t)M * per_row) return;
    const size_t m = at / per_row;
    const int n = (int)(at - m * per_row) * W;
    V part[MAX_SLICES];
    #pragma unroll
    for (int s = 0; s < MAX_SLICES; s++)
        if (s < slices) part[s] = *reinterpret_cast<const V*>(partial + ((size_t)s * M + m) * N + n);
    V old = {};
    V* y = reinterpret_cast<V*>(Y + m * ldy + n);
    if (accumulate) old = *y;
    #pragma unroll
    for (int i = 0; i < W; i++) {
        float t = (&reinterpret_cast<const float&>(part[0]))[i];
        if (accumulate) t = (&reinterpret_cast<const float&>(old))[i] + t;
        #pragma unroll
        for (int s = 1; s < MAX_SLICES; s++)
            if (s < slices) t += (&reinterpret_cast<const float&>(part[s]))[i];
        (&reinterpret_cast<float&>(old))[i] = t;
    }
    *y = old;
}

template <int BN>
int launch_split(const CUtensorMap& mx, const CUtensorMap& mw, const SplitArgs& g, cudaStream_t stream) {
    auto kern = gemm_split_kernel<BN>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::SMEM);
    if (e != cudaSuccess) return (int)e;
    const int most = ik_sm_count() / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * (g.units < most ? g.units : most)));
    cfg.blockDim = dim3(Cfg<BN>::THREADS);
    cfg.dynamicSmemBytes = Cfg<BN>::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (ik_pdl_mask() & IK_FAMILY) ? 2 : 1;
    IK_RETURN_IF_ERROR(cudaLaunchKernelEx(&cfg, kern, mx, mw, g));
    return (int)cudaGetLastError();
}

// How K is cut: into slices of at least 32 K steps, eight of them at most, whatever M and N are.
void cut(int K, int& nkb, int& per, int& slices) {
    nkb = (K + BK - 1) / BK;
    const int want = nkb / 32 < 1 ? 1 : nkb / 32 > MAX_SLICES ? MAX_SLICES : nkb / 32;
    per = (nkb + want - 1) / want;
    slices = (nkb + per - 1) / per;
}

struct Plan { int bn, side_by_side; };

// Tokens of a tile, and whether the slices of K run side by side (with a second kernel that adds them): what takes the least time in
// whole rounds over the pairs of SMs.  Nanoseconds a K step with all SMs at work, measured: 1,150 with 256 tokens a tile, 580 with 128, 365 with 64, 300 with 32.
Plan plan(int M, int N, int K, int pairs) {
    int nkb, per, slices;
    cut(K, nkb, per, slices);
    Plan best = {256, 0};
    long long best_ns = -1;
    for (int bn = 256; bn >= 32; bn /= 2) {
        const long long step = bn == 256 ? 1150 : bn == 128 ? 580 : bn == 64 ? 365 : 300;
        const long long tiles = (long long)((N + 255) / 256) * ((M + bn - 1) / bn);
        for (int side = 0; side < (slices > 1 ? 2 : 1); side++) {
            const long long rounds = (tiles * (side ? slices : 1) + pairs - 1) / pairs;
            const long long ns = rounds * (side ? per : nkb) * step + (side ? 2000 + (slices + 1ll) * M * N / 1000 : 0);
            if (best_ns < 0 || ns < best_ns) { best_ns = ns; best = {bn, side}; }
        }
    }
    return best;
}

}  // namespace

// Floats of scratch for the slices' sums that ik_gemm_split wants for these sizes (0 = none).
IK_EXPORT long long ik_gemm_split_scratch(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    int nkb, per, slices;
    cut(K, nkb, per, slices);
    return plan(M, N, K, ik_sm_count() / 2).side_by_side ? (long long)slices * M * N : 0;
}

// planes: 3 * M * K bfloat16 of scratch; partial: as ik_gemm_split_scratch says.  force: 0 = as chosen, or 2 * bn + (slices side by
// side) with scratch of slices * M * N floats.  IK_UNSUPPORTED where rows are not on 16 bytes.
IK_EXPORT int ik_gemm_split(const float* X, const void* W, float* Y, void* planes, float* partial, int M, int N, int K, int ldx, int ldw, int ldy,
                            int accumulate, int force, int* status, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || ldx < K || ldw < K || ldy < N) return IK_BAD_ARGUMENT;
    if (K % 8 || ldw % 8 || ((uintptr_t)W % 16) || ((uintptr_t)planes % 16)) return IK_UNSUPPORTED;
    if (M == 0) return IK_OK;
    const int pairs = ik_sm_count() / 2;
    if (pairs < 1) return IK_UNSUPPORTED;
    SplitArgs g = {};
    cut(K, g.nkb, g.per, g.slices);
    Plan p = force ? Plan{force >> 1, force & 1} : plan(M, N, K, pairs);
    if ((p.bn != 32 && p.bn != 64 && p.bn != 128 && p.bn != 256) || !planes || (p.side_by_side && !partial)) return IK_BAD_ARGUMENT;
    g.M = M; g.N = N; g.ldy = ldy; g.status = status;
    g.side_by_side = p.side_by_side;
    g.Y = p.side_by_side ? partial : Y;
    g.accumulate = p.side_by_side ? 0 : accumulate;
    g.tiles_m = (M + p.bn - 1) / p.bn;
    const long long units = (long long)g.tiles_m * ((N + 255) / 256) * (p.side_by_side ? g.slices : 1);
    if (units > 0x3fffffff) return IK_UNSUPPORTED;
    g.units = (int)units;

    CUtensorMap mx, mw;
    int st = ik_make_map(&mw, W, N, K, ldw, 128);
    if (st != IK_OK) return st;
    IkEncodeTiled enc = ik_encode_fn();
    if (!enc) return IK_UNSUPPORTED;
    cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)M, 3};
    cuuint64_t strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)M * K * 2};
    cuuint32_t box[3] = {64u, (cuuint32_t)p.bn / 2, 3u};
    cuuint32_t estr[3] = {1, 1, 1};
    if (enc(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, planes, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return IK_BAD_ARGUMENT;

    const size_t quads = (size_t)M * (K / 8);
    IK_RETURN_IF_ERROR(ik_launch_family(IK_FAMILY_ELEMENTWISE, split_planes_kernel, dim3((unsigned)((quads + 255) / 256)), dim3(256), 0, stream, X, (bf16*)planes, M, K,
                                        (size_t)ldx, (int)(ldx % 4 == 0 && (uintptr_t)X % 16 == 0)));
    st = p.bn == 256 ? launch_split<256>(mx, mw, g, stream) : p.bn == 128 ? launch_split<128>(mx, mw, g, stream) : p.bn == 64 ? launch_split<64>(mx, mw, g, stream) : launch_split<32>(mx, mw, g, stream);
    if (st != IK_OK || !p.side_by_side) return st;
    const bool vec = N % 4 == 0 && ldy % 4 == 0 && (uintptr_t)Y % 16 == 0 && (uintptr_t)partial % 16 == 0;
    const size_t pieces = (size_t)M * (vec ? N / 4 : N);
    const dim3 grid((unsigned)((pieces + 255) / 256));
    if (vec) IK_RETURN_IF_ERROR(ik_launch_family(IK_FAMILY_ELEMENTWISE, split_sum_kernel<float4>, grid, dim3(256), 0, stream, (const float*)partial, Y, M, N, ldy, g.slices, accumulate));
    else IK_RETURN_IF_ERROR(ik_launch_family(IK_FAMILY_ELEMENTWISE, split_sum_kernel<float>, grid, dim3(256), 0, stream, (const float*)partial, Y, M, N, ldy, g.slices, accumulate));
    IK_LAUNCH_STATUS();
}

// Sites: 1 = loader for a free stage, 2 = issuer for a drained accumulator, 3 = issuer for a loaded stage, 4 = epilogue.
IK_EXPORT int ik_gemm_split_take_wait_record(int* out4) { return ik_take_wait_record(out4); }
