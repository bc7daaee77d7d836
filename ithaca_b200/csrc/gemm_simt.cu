// Plain matrix product on the CUDA cores: Y[M, N] (+)= X[M, K] * W[N, K]^T.
//
// This is the 32-bit path's product for 32-bit weights, for K < 256 and for rows off 16 bytes (gemm_split.cu takes the others), and the fallback for
// shapes the 16-bit tensor-core kernels refuse.  Operands are converted to float when loaded; every output element is one
// float accumulator that adds its K products in ascending k, whatever M and N are, so a
// row of Y does not depend on which other rows are in the call.  No split along K, no
// atomics, no reduced-precision matrix mode.  A batch of products of equal shape (one per head, say) runs as one
// launch: product b reads X + b * bx, W + b * bw and writes Y + b * by.
#define IK_FAMILY 2
#include "common.cuh"

namespace {

constexpr int BK = 16;

// Four neighbouring values of k of one row (zeros past K or the last row), as they are stored: turned into floats only when they go
// to shared memory, since a conversion next to the load would wait for the load.
template <typename T> struct Quad { typedef float4 type; };
template <> struct Quad<__nv_bfloat16> { typedef uint2 type; };
__device__ __forceinline__ float4 as_floats(const float4& v) { return v; }
__device__ __forceinline__ float4 as_floats(const uint2& r) {
    return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
}
__device__ __forceinline__ float4 one_by_one(const float* p, int n) {
    return make_float4(p[0], n > 1 ? p[1] : 0.f, n > 2 ? p[2] : 0.f, n > 3 ? p[3] : 0.f);
}
__device__ __forceinline__ uint2 one_by_one(const __nv_bfloat16* p, int n) {
    const unsigned short* q = reinterpret_cast<const unsigned short*>(p);
    return make_uint2(q[0] | (n > 1 ? (unsigned)q[1] << 16 : 0u), (n > 2 ? (unsigned)q[2] : 0u) | (n > 3 ? (unsigned)q[3] << 16 : 0u));
}
template <typename T> __device__ __forceinline__ typename Quad<T>::type ld_k4(const T* row, bool there, int k, int K, bool vec) {
    typename Quad<T>::type v = {};
    if (there && k < K) v = vec ? *reinterpret_cast<const typename Quad<T>::type*>(row + k) : one_by_one(row + k, K - k);   // (vec: K is a multiple of 4)
    return v;
}
__device__ __forceinline__ uint64_t pair(float lo, float hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ void fma_pair(uint64_t& d, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }

// A thread's products are TM x TN of a BM x BN tile, in groups of four neighbouring rows and columns, so that a step of k costs TM / 4 + TN / 4
// reads of 16 bytes from shared memory for TM * TN multiply-adds, which go in pairs of neighbouring columns (fma.rn.f32x2: each
// half rounds as fmaf does).  Tiles of BK steps lie [k][row] in shared memory, rows exchanged in eights by k (row ^ 8 (k / 4)): the
// transposing stores of a warp (8 rows x 4 quads of k) then meet all banks once.  The next D tiles are on their way into registers
// while one is computed, two tiles of shared memory, one barrier a tile.
// What bounds it is the multiply-adds, one per product and in order.  Measured on B200 (float X, bfloat16 W; us, a thread's 4 x 4
// products with scalar loads -> this): 465 tokens x 16384 x 2048 1,225 -> 729, x 2048 x 8192 866 -> 544; 2,048 tokens x 16384 x 2048
// 4,611 -> 2,465 (56 TFLOP/s); 1 token x 2048 x 8192 631 -> 317.
template <typename TX, typename TW, typename TY, int BM, int BN, int TM, int TN, int D>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), BM == 128 ? 2 : 3)
gemm_simt_kernel(const TX* __restrict__ X, const TW* __restrict__ W, TY* __restrict__ Y, int M, int N, int K,
                 int ldx, int ldw, int ldy, int accumulate, size_t bx, size_t bw, size_t by, int vec_x, int vec_w) {
    constexpr int NT = (BM / TM) * (BN / TN), NX = BN / TN, QX = BM * 4 / NT, QW = BN * 4 / NT;
    static_assert(BM * 4 % NT == 0 && BN * 4 % NT == 0 && TM % 4 == 0 && TN % 4 == 0, "whole quads a thread");
    X += blockIdx.z * bx;
    W += blockIdx.z * bw;
    Y += blockIdx.z * by;
    ik_pdl_wait();
    IK_AFTER_WAIT(X);                 // the tokens are the kernel before's results; this kernel takes no weight early
    ik_pdl_launch_dependents();
    __shared__ __align__(16) float xs[2][BK][BM];
    __shared__ __align__(16) float ws[2][BK][BN];
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN, tid = threadIdx.x;
    const int tx = tid % NX, ty = tid / NX;                       // tx -> n, ty -> m
    uint64_t acc[TM][TN / 2];                                     // columns (2 j, 2 j + 1)
    #pragma unroll
    for (int i = 0; i < TM; i++)
        #pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[i][j] = 0;
    typedef typename Quad<TX>::type RX;
    typedef typename Quad<TW>::type RW;
    RX rx[D][QX];
    RW rw[D][QW];
    auto fetch = [&](int k0, RX (&x)[QX], RW (&w)[QW]) {
        #pragma unroll
        for (int l = 0; l < QX; l++) {
            const int r = (tid + l * NT) >> 2, k = k0 + 4 * (tid & 3);
            x[l] = ld_k4(X + (size_t)min(m0 + r, M - 1) * ldx, m0 + r < M, k, K, vec_x);
        }
        #pragma unroll
        for (int l = 0; l < QW; l++) {
            const int r = (tid + l * NT) >> 2, k = k0 + 4 * (tid & 3);
            w[l] = ld_k4(W + (size_t)min(n0 + r, N - 1) * ldw, n0 + r < N, k, K, vec_w);
        }
    };
    auto store = [&](int buf, const RX (&x)[QX], const RW (&w)[QW]) {
        const int q = tid & 3;
        #pragma unroll
        for (int l = 0; l < QX; l++) {
            const int r = ((tid + l * NT) >> 2) ^ (8 * q);
            const float4 v = as_floats(x[l]);
            xs[buf][4 * q][r] = v.x; xs[buf][4 * q + 1][r] = v.y; xs[buf][4 * q + 2][r] = v.z; xs[buf][4 * q + 3][r] = v.w;
        }
        #pragma unroll
        for (int l = 0; l < QW; l++) {
            const int r = ((tid + l * NT) >> 2) ^ (8 * q);
            const float4 v = as_floats(w[l]);
            ws[buf][4 * q][r] = v.x; ws[buf][4 * q + 1][r] = v.y; ws[buf][4 * q + 2][r] = v.z; ws[buf][4 * q + 3][r] = v.w;
        }
    };
    #pragma unroll
    for (int d = 0; d < D; d++) fetch(d * BK, rx[d], rw[d]);
    store(0, rx[0], rw[0]);
    fetch(D * BK, rx[0], rw[0]);                                  // (past K: zeros, no access)
    __syncthreads();
    constexpr int U = D > 1 ? D : 2;                              // unrolled so that a tile's buffers are known at compile time
    static_assert(U % 2 == 0, "two tiles of shared memory");
    for (int k0 = 0; k0 < K; k0 += U * BK) {
        #pragma unroll
        for (int d = 0; d < U; d++) {                             // tile k0 / BK + d, in buffer d & 1; registers (d + 1) % D hold the next
            if (k0 + d * BK >= K) break;
            #pragma unroll
            for (int kk = 0; kk < BK; kk++) {
                float a[TM];
                uint64_t b[TN / 2];
                #pragma unroll
                for (int g = 0; g < TM / 4; g++) {
                    const float4 v = *reinterpret_cast<const float4*>(&xs[d & 1][kk][(g * (BM / (TM / 4)) + ty * 4) ^ (8 * (kk >> 2))]);
                    a[4 * g] = v.x; a[4 * g + 1] = v.y; a[4 * g + 2] = v.z; a[4 * g + 3] = v.w;
                }
                #pragma unroll
                for (int g = 0; g < TN / 4; g++) {
                    const float4 v = *reinterpret_cast<const float4*>(&ws[d & 1][kk][(g * (BN / (TN / 4)) + tx * 4) ^ (8 * (kk >> 2))]);
                    b[2 * g] = pair(v.x, v.y); b[2 * g + 1] = pair(v.z, v.w);
                }
                #pragma unroll
                for (int i = 0; i < TM; i++) {
                    const uint64_t aa = pair(a[i], a[i]);
                    #pragma unroll
                    for (int j = 0; j < TN / 2; j++) fma_pair(acc[i][j], aa, b[j]);
                }
            }
            store((d + 1) & 1, rx[(d + 1) % D], rw[(d + 1) % D]);
            fetch(k0 + (d + 1 + D) * BK, rx[(d + 1) % D], rw[(d + 1) % D]);
            __syncthreads();
        }
    }
    #pragma unroll
    for (int i = 0; i < TM; i++) {
        const int m = m0 + (i / 4) * (BM / (TM / 4)) + ty * 4 + i % 4;
        if (m >= M) continue;
        #pragma unroll
        for (int j = 0; j < TN; j++) {
            const int n = n0 + (j / 4) * (BN / (TN / 4)) + tx * 4 + j % 4;
            if (n >= N) continue;
            const size_t o = (size_t)m * ldy + n;
            float v = __uint_as_float((unsigned)(acc[i][j / 2] >> (32 * (j & 1))));
            if (accumulate) v += ik_ld(Y, o);
            ik_st(Y, o, v);
        }
    }
}

template <typename TX, typename TW, typename TY, int BM, int BN, int TM, int TN, int D>
int launch_tile(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw, int ldy, int accumulate,
                cudaStream_t stream, int batch, size_t bx, size_t bw, size_t by) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
    const int vec_x = K % 4 == 0 && ldx % 4 == 0 && bx % 4 == 0 && (uintptr_t)X % (4 * sizeof(TX)) == 0;
    const int vec_w = K % 4 == 0 && ldw % 4 == 0 && bw % 4 == 0 && (uintptr_t)W % (4 * sizeof(TW)) == 0;
    IK_RETURN_IF_ERROR(ik_launch(gemm_simt_kernel<TX, TW, TY, BM, BN, TM, TN, D>, grid, (BM / TM) * (BN / TN), 0, stream, (const TX*)X, (const TW*)W, (TY*)Y, M, N,
                                 K, ldx, ldw, ldy, accumulate, bx, bw, by, vec_x, vec_w));
    IK_LAUNCH_STATUS();
}

// Larger tiles read less from shared memory per multiply-add, smaller ones fill the SMs' last round better: the tile whose rounds
// take least, in units of 32 x 32 products, the smaller ones counted a twelfth and a quarter dearer.
template <typename TX, typename TW, typename TY>
int launch(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw, int ldy, int accumulate,
           cudaStream_t stream, int batch = 1, size_t bx = 0, size_t bw = 0, size_t by = 0) {
    const long long sms = ik_sm_count();
    auto rounds = [&](int bm, int bn) { return ((long long)((N + bn - 1) / bn) * ((M + bm - 1) / bm) * batch + sms - 1) / sms; };
    const long long large = rounds(128, 128) * 192, middle = rounds(128, 64) * 104, small = rounds(64, 64) * 60;
    if (large <= middle && large <= small)
        return launch_tile<TX, TW, TY, 128, 128, 8, 8, 1>(X, W, Y, M, N, K, ldx, ldw, ldy, accumulate, stream, batch, bx, bw, by);
    if (middle <= small)
        return launch_tile<TX, TW, TY, 128, 64, 8, 4, 2>(X, W, Y, M, N, K, ldx, ldw, ldy, accumulate, stream, batch, bx, bw, by);
    return launch_tile<TX, TW, TY, 64, 64, 4, 4, 4>(X, W, Y, M, N, K, ldx, ldw, ldy, accumulate, stream, batch, bx, bw, by);
}

}  // namespace

// Padding zeros in K contribute exact zeros, and a k beyond K is never added to a real
// product's partial sum out of order: the accumulation order of the real terms is 0..K-1.
IK_EXPORT int ik_gemm_simt(const void* X, int x_dtype, const void* W, int w_dtype, void* Y, int y_dtype, int M, int N,
                           int K, int ldx, int ldw, int ldy, int accumulate, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || ldx < K || ldw < K || ldy < N) return IK_BAD_ARGUMENT;
    if (M == 0) return IK_OK;
    const int code = x_dtype * 4 + w_dtype * 2 + y_dtype;
    switch (code) {
        case 0: return launch<float, float, float>(X, W, Y, M, N, K, ldx, ldw, ldy, accumulate, stream);
        case 1: return launch<float, float, __nv_bfloat16>(X, W, Y, M, N, K, ldx, ldw, ldy, accumulate, stream);
        case 2: return launch<float, __nv_bfloat16, float>(X, W, Y, M, N, K, ldx, ldw, ldy, accumulate, stream);
        case 3: return launch<float, __nv_bfloat16, __nv_bfloat16>(X, W, Y, M, N, K, ldx, ldw, ldy, accumulate, stream);
        case 4: return launch<__nv_bfloat16, float, float>(X, W, Y, M, N, K, ldx, ldw, ldy, accumulate, stream);
        case 5: return launch<__nv_bfloat16, float, __nv_bfloat16>(X, W, Y, M, N, K, ldx, ldw, ldy, accumulate, stream);
        case 6: return launch<__nv_bfloat16, __nv_bfloat16, float>(X, W, Y, M, N, K, ldx, ldw, ldy, accumulate, stream);
        case 7: return launch<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(X, W, Y, M, N, K, ldx, ldw, ldy, accumulate, stream);
    }
    return IK_BAD_ARGUMENT;
}

// `batch` products of one shape in one launch (strides between them in elements).  x and y have one type (the activations'),
// w its own.
IK_EXPORT int ik_gemm_simt_batched(const void* X, int x_dtype, const void* W, int w_dtype, void* Y, int y_dtype, int M, int N,
                                   int K, int ldx, int ldw, int ldy, int batch, unsigned long long bx, unsigned long long bw,
                                   unsigned long long by, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || ldx < K || ldw < K || ldy < N || batch <= 0 || batch > 65535) return IK_BAD_ARGUMENT;
    if (M == 0) return IK_OK;
    const int code = x_dtype * 4 + w_dtype * 2 + y_dtype;
    switch (code) {
        case 0: return launch<float, float, float>(X, W, Y, M, N, K, ldx, ldw, ldy, 0, stream, batch, bx, bw, by);
        case 2: return launch<float, __nv_bfloat16, float>(X, W, Y, M, N, K, ldx, ldw, ldy, 0, stream, batch, bx, bw, by);
        case 4: return launch<__nv_bfloat16, float, float>(X, W, Y, M, N, K, ldx, ldw, ldy, 0, stream, batch, bx, bw, by);
        case 6: return launch<__nv_bfloat16, __nv_bfloat16, float>(X, W, Y, M, N, K, ldx, ldw, ldy, 0, stream, batch, bx, bw, by);
        case 7: return launch<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(X, W, Y, M, N, K, ldx, ldw, ldy, 0, stream, batch, bx, bw, by);
    }
    return IK_BAD_ARGUMENT;
}
