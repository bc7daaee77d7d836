// The gated delta rule for prompts, 64 tokens at a time (the 16-bit path; every number here is float, as in delta.cu).
//
// Within a chunk, with G_t the product of the decays up to token t and M[t, s] = b_t (G_t / G_s) (k_t . k_s) for s < t, the
// corrections u_t of all tokens solve a triangular system: (I + M) U = b (V - G (K S)), S the state before the chunk.  So
//   U = T (V - G (K S)) with T = (I + M)^-1 diag(b);   O = G (Q S) + P U with P[t, s] = (G_t / G_s) (q_t . k_s), s <= t;
//   S <- G_end S + K^T ((G_end / G) U).
// delta_chunk_prepare_kernel forms T and P of every chunk and head side by side; delta_chunk_kernel walks a sequence's chunks with
// a slice of a head's columns per block: five small products a chunk in place of 64 dependent steps.  The tokens' chain is what
// bounds the token-by-token kernel (0.37 to 0.4 us a token; which sequences of a step go which way: ops.delta_chunks_from); the chunks' chain is
// bound by the walk's products and the latencies between them.
// Measured on B200, 16 heads of 128 over two prompts of 3,000 and 1,910 tokens: token by token 2,776 us (the layer), in chunks 594 us with the walk's float
// products on the CUDA cores, which read half of 16 bytes from shared memory per four multiply-adds, and 424 us with these on the tensor cores: 80 us for T
// and P, 7.4 us a chunk for the walk.
#include <math_constants.h>
#include "common.cuh"

namespace {

constexpr int C = 64;                                    // tokens of a chunk
constexpr int TLD = C + 4;                               // row stride of T and P in shared memory
// A chunk's floats beside T and P: G [64], G_end / G [64], G_end, padding, the diagonals of T [64] and P [64].
constexpr int VEC_T = 132, VEC_P = VEC_T + C, VEC = VEC_P + C;

// SOME: only sequences of at least `least` (> 0) tokens are walked, and their chunks numbered, in the order of the sequences.  Otherwise all
// are, and chunk j of sequence b has the number cu_seqlens[b] / 64 + b + j (instances of their own: the walk takes 2 % longer where its
// sequence is looked for).
__device__ __forceinline__ int chunk_base(const int* cu_seqlens, int b) { return cu_seqlens[b] / C + b; }
struct Walked {
    int b, chunk0;                                       // the sequence (-1: there is none), the number of its first chunk
};
// The i-th walked sequence, or (BY_CHUNK) the one that chunk number i belongs to.  Every warp looks by itself, 32 sequences at a time.
template <bool BY_CHUNK>
__device__ __forceinline__ Walked walked_sequence(const int* cu_seqlens, int n_seqs, int least, int i) {
    const int lane = threadIdx.x & 31;
    for (int b0 = 0, seen = 0, chunks = 0; b0 < n_seqs; b0 += 32) {
        const int b = b0 + lane, n = b < n_seqs ? cu_seqlens[b + 1] - cu_seqlens[b] : 0;
        const bool mine = n >= least;
        const int own = mine ? (n + C - 1) / C : 0;
        int upto = own;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int before = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += before;
        }
        const unsigned all = __ballot_sync(0xffffffffu, mine);
        const bool it = mine && (BY_CHUNK ? i < chunks + upto && i >= chunks + upto - own : seen + __popc(all & ((1u << lane) - 1)) == i);
        const int found = __reduce_max_sync(0xffffffffu, it ? b : -1);
        if (found >= 0) return {found, __reduce_max_sync(0xffffffffu, it ? chunks + upto - own : -1)};
        seen += __popc(all);
        chunks += __shfl_sync(0xffffffffu, upto, 31);
    }
    return {-1, 0};
}

__device__ __forceinline__ void copy16(float* dst, const float* src, bool there) {           // zeros where there is nothing
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ float4 at4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// One block per (chunk, value head).
template <int DK, bool SOME>
__global__ void __launch_bounds__(256, 3)
delta_chunk_prepare_kernel(const float* __restrict__ u, int ldu, int q_off, int k_off, const float* __restrict__ bg, float* __restrict__ scratch,
                           float* __restrict__ vecs, const int* __restrict__ cu_seqlens, int n_seqs, int least, int H, int G) {
    constexpr int LD = DK + 4;
    extern __shared__ __align__(16) float sm[];
    float* const Ks = sm;                                // [64][LD]
    float* const Qs = Ks + C * LD;
    // M, then T, lie where K and Q were once their products are in registers: three blocks an SM instead of two (us on B200, 3,000 + 1,910 tokens, 16
    // heads of 128: 86 -> 78)
    constexpr int ROOM = 2 * C * LD > 2 * C * TLD ? 2 * C * LD : 2 * C * TLD;
    float* const Ms = sm;                                // [64][TLD]
    float* const Ts = Ms + C * TLD;
    double* const logs = (double*)(sm + ROOM);           // [64] sums of the decays' logarithms
    float* const beta = (float*)(logs + C);              // [64]
    ik_pdl_wait();
    IK_AFTER_WAIT(u);
    IK_AFTER_WAIT(bg);
    IK_AFTER_WAIT(cu_seqlens);
    ik_pdl_launch_dependents();
    const int tid = threadIdx.x, h = blockIdx.y, f = blockIdx.x;
    Walked seq = {0, 0};
    if (SOME) {
        seq = walked_sequence<true>(cu_seqlens, n_seqs, least, f);
        if (seq.b < 0) return;
    } else {
        for (int high = n_seqs - 1; seq.b < high;) {         // the last sequence whose first chunk is not behind this one
            const int mid = (seq.b + high + 1) >> 1;
            if (chunk_base(cu_seqlens, mid) <= f) seq.b = mid;
            else high = mid - 1;
        }
        seq.chunk0 = chunk_base(cu_seqlens, seq.b);
    }
    const int t0 = cu_seqlens[seq.b] + (f - seq.chunk0) * C, n = min(C, cu_seqlens[seq.b + 1] - t0);
    if (n <= 0) return;
    const int kvh = h / (H / G);
    for (int i = tid; i < 2 * C * (DK / 4); i += 256) {
        const int r = i / (DK / 4), w = i % (DK / 4), t = r & (C - 1);
        copy16((r < C ? Ks : Qs) + t * LD + 4 * w, u + (size_t)(t0 + min(t, n - 1)) * ldu + (r < C ? k_off : q_off) + kvh * DK + 4 * w, t < n);
    }
    copies_commit();
    if (tid < C) {
        beta[tid] = tid < n ? bg[((size_t)(t0 + tid) * 2) * H + h] : 0.f;
        // a decay of 0 counts as e^-10000: 0 again wherever it is met
        const float g = tid < n ? bg[((size_t)(t0 + tid) * 2 + 1) * H + h] : 1.f;
        logs[tid] = g == 0.f ? -10000.0 : log((double)g);
    }
    __syncthreads();
    if (tid < 32) {                                      // prefix sums, two tokens a lane
        double a = logs[2 * tid], c = a + logs[2 * tid + 1], sum = c;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double before = __shfl_up_sync(0xffffffffu, sum, o);
            if (tid >= o) sum += before;
        }
        const double earlier = __shfl_up_sync(0xffffffffu, sum, 1);
        logs[2 * tid] = tid ? earlier + a : a;
        logs[2 * tid + 1] = tid ? earlier + c : c;
    }
    copies_wait();
    __syncthreads();
    float* const vec = vecs + ((size_t)f * H + h) * VEC;
    if (tid < C) {
        vec[VEC_T + tid] = beta[tid];
        vec[tid] = expf((float)logs[tid]);
        vec[C + tid] = expf((float)(logs[C - 1] - logs[tid]));     // (tokens that are not there have a decay of 1)
        if (tid == 0) vec[2 * C] = expf((float)logs[C - 1]);
    }
    // k . k and q . k of 4 x 4 tokens a thread: rows ti + 16 i, columns tj + 16 j
    const int tj = tid & 15, ti = tid >> 4;
    float kk[4][4] = {}, qk[4][4] = {};
    #pragma unroll 2
    for (int d = 0; d < DK; d += 4) {
        float4 kc[4];
        #pragma unroll
        for (int j = 0; j < 4; j++) kc[j] = at4(Ks + (tj + 16 * j) * LD + d);
        #pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 kr = at4(Ks + (ti + 16 * i) * LD + d), qr = at4(Qs + (ti + 16 * i) * LD + d);
            #pragma unroll
            for (int j = 0; j <= i; j++) {               // (columns 16 j .. lie past row 16 i + 15 for j > i)
                kk[i][j] = fmaf(kr.x, kc[j].x, fmaf(kr.y, kc[j].y, fmaf(kr.z, kc[j].z, fmaf(kr.w, kc[j].w, kk[i][j]))));
                qk[i][j] = fmaf(qr.x, kc[j].x, fmaf(qr.y, kc[j].y, fmaf(qr.z, kc[j].z, fmaf(qr.w, kc[j].w, qk[i][j]))));
            }
        }
    }
    float* const outT = scratch + ((size_t)f * H + h) * 2 * C * C;
    float* const outP = outT + C * C;
    __syncthreads();                                     // K and Q have been read
    #pragma unroll
    for (int i = 0; i < 4; i++)
        #pragma unroll
        for (int j = 0; j < 4; j++) {
            const int t = ti + 16 * i, s = tj + 16 * j;
            const float ratio = s <= t ? expf((float)(logs[t] - logs[s])) : 0.f;
            outP[t * C + s] = s < t ? ratio * qk[i][j] : 0.f;
            if (s == t) vec[VEC_P + t] = qk[i][j];
            Ms[t * TLD + s] = s < t ? beta[t] * ratio * kk[i][j] : 0.f;
        }
    __syncthreads();
    // X = (I + M)^-1 by blocks of 16: the diagonal blocks column by column, then a block row at a time
    if (tid < C) {
        const int blk = tid >> 4, c = tid & 15;
        float x[16];
        #pragma unroll
        for (int r = 0; r < 16; r++) {
            float a = r == c ? 1.f : 0.f;
            #pragma unroll
            for (int s = 0; s < r; s++) a = fmaf(-Ms[(blk * 16 + r) * TLD + blk * 16 + s], x[s], a);
            x[r] = a;
            Ts[(blk * 16 + r) * TLD + blk * 16 + c] = a;
        }
    }
    __syncthreads();
    for (int i = 1; i < 4; i++) {                        // X[i, j] = -X[i, i] sum_k M[i, k] X[k, j], j < i; the sums over M's own block row i
        float a[3] = {0.f, 0.f, 0.f};
        #pragma unroll
        for (int j = 0; j < 3; j++)
            if (j < i)
                for (int s = 16 * j; s < 16 * i; s++) a[j] = fmaf(Ms[(16 * i + ti) * TLD + s], Ts[s * TLD + 16 * j + tj], a[j]);
        __syncthreads();
        #pragma unroll
        for (int j = 0; j < 3; j++)
            if (j < i) Ms[(16 * i + ti) * TLD + 16 * j + tj] = a[j];
        __syncthreads();
        #pragma unroll
        for (int j = 0; j < 3; j++)
            if (j < i) {
                float x = 0.f;
                #pragma unroll
                for (int s = 0; s < 16; s++)                  // (a later token's infinities never meet a zero here)
                    if (s <= ti) x = fmaf(-Ts[(16 * i + ti) * TLD + 16 * i + s], Ms[(16 * i + s) * TLD + 16 * j + tj], x);
                Ts[(16 * i + ti) * TLD + 16 * j + tj] = x;
            }
        __syncthreads();
    }
    for (int i = tid; i < C * C; i += 256) {                 // (0, not 0 * beta, above the diagonal: the walk reads whole blocks of 16)
        const int t = i / C, s = i % C;
        outT[i] = s < t ? Ts[t * TLD + s] * beta[s] : 0.f;
    }
}

// The five products of a chunk run on the tensor cores (mma.sync, bfloat16) with every float as the sum of three bfloat16 numbers, h + m + l, which
// hold its 24 bits: h h' + (h m' + m h' + m m' + h l' + l h'), the small terms in sums of their own; what is left out is under 2^-23 of a
// product.  Sums of the large terms leave the tensor core every 16 products and are added as floats (it drops bits towards zero).  What a strong decay leaves
// of a sum, a token's own term of T (..) and P U and the last token's of K^T E, is no part of those sums: it is multiplied and added as floats, one
// rounding to nearest.  Numbers of 3.3e38 and more count as infinite, bits below 2^-133 go.
//
// Everything is transposed, columns of the state first: a warp's sums [columns][tokens or keys' components] are then, lane by lane, what it has to
// leave as the first operand of the next product, and K, Q, T and P are second operands as they lie (K once more, transposed by the load, for the state).
// Eight warps share the tokens of each product (8 each; warps w and w + 4 meet the long and the short rows of the triangles on one scheduler) and the
// state (DK / 8 components each, floats in registers); its planes and those of V - G (K S) and of U pass through shared memory.  Four more
// warps bring the next chunk's K, Q, T and P as planes: they hold them in registers until the place is free.
//
// One block per (16 MT columns of a head, value head, walked sequence).  Bound by what its latencies leave between three barriers a chunk, then by the tensor
// pipe: about 14,000 cycles a chunk with MT = 2, of which counters show the pipe at work for 5,600 (2 cycles an instruction and SM) and 31 % of the issue slots
// taken; a quarter fewer with MT = 1 (eight warps to bring in place of four, or a matrix asked for
// ahead, change nothing).  Distance to 64 bits over prompts of 1,000 and 1,500 tokens, 8 heads of 128 (2-norm, results and states, float products
// on the CUDA cores / these): decays around 0.1 2.07e-7 3.7e-8 / 2.07e-7 3.7e-8, 0.5 2.09e-7 4.7e-8 / 2.09e-7 5.1e-8, 0.8 to 1 2.32e-7 1.01e-7 / 2.15e-7
// 0.85e-7, 0.97 2.48e-7 1.28e-7 / 2.12e-7 0.92e-7, near one 4.39e-7 4.09e-7 / 1.93e-7 1.56e-7.  (With those terms in the sums too: 2.23e-7 9.3e-8 around 0.1,
// and 1 % less time.)
template <int DK, int MT>
struct Walk {
    static constexpr int LDK = DK + 8, LDT = C + 8;      // row strides of the planes (rows on 16 bytes, 8 of them over all banks)
    static constexpr int NT = DK / 64, KS = DK / 16;     // 8-wide pieces of the state a warp owns; steps of 16 components
    static constexpr int K = 0, Q = K + 3 * C * LDK * 2, T = Q + 3 * C * LDK * 2, P = T + 3 * C * LDT * 2;
    static constexpr int S = P + 3 * C * LDT * 2;        // first operands: [step][plane][MT][lane] 16 bytes
    static constexpr int R = S + KS * 3 * MT * 512, U = R + 4 * 3 * MT * 512, E = U + 4 * 3 * MT * 512;
    static constexpr int FIRST = E + 4 * 3 * MT * 512;   // [16 MT] the first token of a chunk that is not finite in a column (C: none)
    static constexpr int LAST = FIRST + 16 * MT * 4;     // [16 MT] (G_end / G) U of the chunk's last token
    static constexpr int BYTES = LAST + 16 * MT * 4;
};
constexpr int MULTIPLIERS = 256, BRINGERS = 128, ALL = MULTIPLIERS + BRINGERS;
// barriers 1 to 4: K, Q, T, P are there; 5 to 8: they have been read; 9: the multipliers among themselves
__device__ __forceinline__ void bar_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(ALL) : "memory"); }
__device__ __forceinline__ void bar_wait(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(ALL) : "memory"); }
__device__ __forceinline__ void bar_multipliers() { asm volatile("bar.sync 9, %0;" ::"n"(MULTIPLIERS) : "memory"); }
__device__ __forceinline__ bool bar_any(bool mine) {     // a barrier of the multipliers that also says whether any of them said so
    int any;
    asm volatile("{ .reg .pred p, q; setp.ne.s32 p, %1, 0; barrier.red.or.pred q, 9, %2, p; selp.s32 %0, 1, 0, q; }"
                 : "=r"(any) : "r"((int)mine), "n"(MULTIPLIERS) : "memory");
    return any;
}
__device__ __forceinline__ unsigned two_bf16(float x, float y) {          // x in the lower half
    unsigned r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
    return r;
}
__device__ __forceinline__ void planes(float x, float y, unsigned& h, unsigned& m, unsigned& l) {
    h = two_bf16(x, y);
    x -= __uint_as_float(h << 16);
    y -= __uint_as_float(h & 0xffff0000u);
    m = two_bf16(x, y);
    l = two_bf16(x - __uint_as_float(m << 16), y - __uint_as_float(m & 0xffff0000u));
}
__device__ __forceinline__ void mma(float (&d)[4], const uint4& a, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
// One step of 16: the terms but the largest into lo; that is added to hi.
template <int MT>
__device__ __forceinline__ void mma_planes(float (&hi)[MT][4], float (&lo)[MT][4], const uint4 (&a)[MT][3], const unsigned (&b)[3][2]) {
    constexpr int AP[5] = {2, 0, 1, 1, 0}, BP[5] = {0, 2, 1, 0, 1};
    #pragma unroll
    for (int i = 0; i < 5; i++)
        #pragma unroll
        for (int mt = 0; mt < MT; mt++) mma(lo[mt], a[mt][AP[i]], b[BP[i]][0], b[BP[i]][1]);
    float h[MT][4] = {};
    #pragma unroll
    for (int mt = 0; mt < MT; mt++) mma(h[mt], a[mt][0], b[0][0], b[0][1]);
    #pragma unroll
    for (int mt = 0; mt < MT; mt++)
        #pragma unroll
        for (int c = 0; c < 4; c++) hi[mt][c] += h[mt][c];
}
template <int MT>
__device__ __forceinline__ void first_operand(uint4 (&a)[MT][3], const char* from, int step, int lane) {
    #pragma unroll
    for (int mt = 0; mt < MT; mt++)
        #pragma unroll
        for (int p = 0; p < 3; p++) a[mt][p] = *reinterpret_cast<const uint4*>(from + (((step * 3 + p) * MT + mt) * 32 + lane) * 16);
}
// A warp's sums c of an 8-wide piece, as half of a step's first operand.
template <int MT>
__device__ __forceinline__ void leave(char* to, int piece, int mt, int lane, const float (&c)[4]) {
    uint2 h, m, l;
    planes(c[0], c[1], h.x, m.x, l.x);
    planes(c[2], c[3], h.y, m.y, l.y);
    char* at = to + ((piece >> 1) * 3 * MT + mt) * 512 + lane * 16 + (piece & 1) * 8;
    *reinterpret_cast<uint2*>(at) = h;
    *reinterpret_cast<uint2*>(at + MT * 512) = m;
    *reinterpret_cast<uint2*>(at + 2 * MT * 512) = l;
}
// Two 8 x 8 pieces of a second operand whose rows are the results' (n), or (TRANS) the sum's (k).
template <bool TRANS>
__device__ __forceinline__ void second_operand(unsigned (&b)[2], unsigned at) {
    if (TRANS) asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(b[0]), "=r"(b[1]) : "r"(at) : "memory");
    else asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(b[0]), "=r"(b[1]) : "r"(at) : "memory");
}

// A matrix of 64 rows of `width` floats, n of them there (zeros else), as planes with rows of `ld`: read into registers, then left.
template <int WIDTH, int LD>
struct Bring {
    static constexpr int N = C * WIDTH / 8 / BRINGERS;
    uint4 h[N], m[N], l[N];
    __device__ __forceinline__ void read(const float* from, size_t stride, int n, int tid) {
        #pragma unroll
        for (int i = 0; i < N; i++) {
            const int r = (tid + i * BRINGERS) / (WIDTH / 8), w = (tid + i * BRINGERS) % (WIDTH / 8);
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
            if (r < n) {
                x = at4(from + (size_t)r * stride + 8 * w);
                y = at4(from + (size_t)r * stride + 8 * w + 4);
            }
            planes(x.x, x.y, h[i].x, m[i].x, l[i].x);
            planes(x.z, x.w, h[i].y, m[i].y, l[i].y);
            planes(y.x, y.y, h[i].z, m[i].z, l[i].z);
            planes(y.z, y.w, h[i].w, m[i].w, l[i].w);
        }
    }
    __device__ __forceinline__ void leave(char* to, int tid) const {
        #pragma unroll
        for (int i = 0; i < N; i++) {
            const int r = (tid + i * BRINGERS) / (WIDTH / 8), w = (tid + i * BRINGERS) % (WIDTH / 8);
            char* at = to + (r * LD + 8 * w) * 2;
            *reinterpret_cast<uint4*>(at) = h[i];
            *reinterpret_cast<uint4*>(at + C * LD * 2) = m[i];
            *reinterpret_cast<uint4*>(at + 2 * C * LD * 2) = l[i];
        }
    }
};

template <int DK, int MT, bool SOME>
__global__ void __launch_bounds__(ALL, 1)
delta_chunk_kernel(const float* __restrict__ u, int ldu, int q_off, int k_off, int v_off, const float* __restrict__ scratch, const float* __restrict__ vecs,
                   float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ cu_seqlens,
                   const int* __restrict__ kv_lens, float* __restrict__ out, int n_seqs, int least, int H, int G, int dv) {
    typedef Walk<DK, MT> W;
    constexpr int NT = W::NT, KS = W::KS;
    extern __shared__ __align__(16) char sb[];
    ik_pdl_wait();
    IK_AFTER_WAIT(u);
    IK_AFTER_WAIT(scratch);
    IK_AFTER_WAIT(vecs);
    IK_AFTER_WAIT(slots);
    IK_AFTER_WAIT(cu_seqlens);
    IK_AFTER_WAIT(kv_lens);
    ik_pdl_launch_dependents();
    Walked seq = {(int)blockIdx.z, 0};
    if (SOME) {
        seq = walked_sequence<false>(cu_seqlens, n_seqs, least, blockIdx.z);
        if (seq.b < 0) return;
    }
    const int b = seq.b, h = blockIdx.y, col0 = blockIdx.x * 16 * MT;
    const int lo = cu_seqlens[b], hi = cu_seqlens[b + 1], end = kv_lens[b], start = end - (hi - lo);
    if (!SOME && hi <= lo) return;
    const int kvh = h / (H / G);
    const int f0 = SOME ? seq.chunk0 : chunk_base(cu_seqlens, b), n_chunks = (hi - lo + C - 1) / C;
    const float* const tp = scratch + ((size_t)f0 * H + h) * 2 * C * C;
    const size_t tp_step = (size_t)H * 2 * C * C;

    if (threadIdx.x >= MULTIPLIERS) {                    // bring
        const int tid = threadIdx.x - MULTIPLIERS;
        for (int j = 0; j < n_chunks; j++) {
            const int t0 = lo + j * C, n = min(C, hi - t0);
            {
                Bring<DK, W::LDK> x;
                x.read(u + (size_t)t0 * ldu + q_off + kvh * DK, ldu, n, tid);
                if (j) bar_wait(6);
                x.leave(sb + W::Q, tid);
                bar_arrive(2);
            }
            {
                Bring<C, W::LDT> x;
                x.read(tp + j * tp_step, C, C, tid);
                if (j) bar_wait(7);
                x.leave(sb + W::T, tid);
                bar_arrive(3);
            }
            {
                Bring<DK, W::LDK> x;
                x.read(u + (size_t)t0 * ldu + k_off + kvh * DK, ldu, n, tid);
                if (j) bar_wait(5);
                x.leave(sb + W::K, tid);
                bar_arrive(1);
            }
            {
                Bring<C, W::LDT> x;
                x.read(tp + j * tp_step + C * C, C, C, tid);
                if (j) bar_wait(8);
                x.leave(sb + W::P, tid);
                bar_arrive(4);
            }
        }
        return;
    }

    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane >> 2, pair = 2 * (lane & 3);
    int* const first = (int*)(sb + W::FIRST);
    float* const last = (float*)(sb + W::LAST);
    if (threadIdx.x < 16 * MT) first[threadIdx.x] = C;
    const size_t per = (size_t)H * DK * dv;
    const float* const st_in = state + ((size_t)slots[b] * 2 + ((start - 1) & 1)) * per + (size_t)h * dv * DK;
    float* const st_out = state + ((size_t)slots[b] * 2 + ((end - 1) & 1)) * per + (size_t)h * dv * DK;
    // element c of a lane's sums: column 16 mt + row + 8 (c / 2), token or component pair + c % 2 of the warp's piece
    auto column = [&](int mt, int c) { return col0 + 16 * mt + row + 8 * (c >> 1); };
    float S[NT][MT][4];
    #pragma unroll
    for (int i = 0; i < NT; i++)
        #pragma unroll
        for (int mt = 0; mt < MT; mt++)
            #pragma unroll
            for (int c = 0; c < 4; c++)
                S[i][mt][c] = start > 0 && column(mt, c) < dv ? st_in[(size_t)column(mt, c) * DK + 8 * (w * NT + i) + pair + (c & 1)] : 0.f;
    const unsigned base = (unsigned)__cvta_generic_to_shared(sb);
    // where this lane's rows of second operands begin: tokens 8 w + .., pieces of 8 along the row; (K for the state) tokens .., the warp's components
    const unsigned by_token = ((8 * w + (lane & 7)) * W::LDK + 8 * ((lane >> 3) & 1)) * 2, by_row = ((8 * w + (lane & 7)) * W::LDT + 8 * ((lane >> 3) & 1)) * 2;
    const unsigned by_component = ((lane & 15) * W::LDK + 8 * w * NT) * 2;

    float v[MT][4], g[2], e[2], t_own[2], p_own[2], g_end;   // this chunk's, asked for a chunk ahead
    auto ask = [&](int j) {
        const int t0 = lo + j * C + 8 * w + pair;
        #pragma unroll
        for (int mt = 0; mt < MT; mt++)
            #pragma unroll
            for (int c = 0; c < 4; c++)
                v[mt][c] = t0 + (c & 1) < hi && column(mt, c) < dv ? u[(size_t)(t0 + (c & 1)) * ldu + v_off + (size_t)h * dv + column(mt, c)] : 0.f;
        const float* ve = vecs + ((size_t)(f0 + j) * H + h) * VEC;
        #pragma unroll
        for (int c = 0; c < 2; c++) {
            g[c] = ve[8 * w + pair + c];
            e[c] = ve[C + 8 * w + pair + c];
            t_own[c] = ve[VEC_T + 8 * w + pair + c];
            p_own[c] = ve[VEC_P + 8 * w + pair + c];
        }
        g_end = ve[2 * C];
    };
    ask(0);
    auto leave_state = [&]() {
        #pragma unroll
        for (int i = 0; i < NT; i++)
            #pragma unroll
            for (int mt = 0; mt < MT; mt++) leave<MT>(sb + W::S, w * NT + i, mt, lane, S[i][mt]);
    };
    leave_state();
    bar_multipliers();
    for (int j = 0; j < n_chunks; j++) {
        // K S and Q S (products and sums rounded one by one: as many columns a block as there are, the bits are the same)
        float ks[MT][4] = {}, qs[MT][4] = {};
        {
            float klo[MT][4] = {}, qlo[MT][4] = {};
            bar_wait(2);
            bar_wait(1);
            #pragma unroll
            for (int s = 0; s < KS; s++) {
                uint4 a[MT][3];
                unsigned kb[3][2], qb[3][2];
                first_operand<MT>(a, sb + W::S, s, lane);
                #pragma unroll
                for (int p = 0; p < 3; p++) {
                    second_operand<false>(kb[p], base + W::K + by_token + (p * C * W::LDK + 16 * s) * 2);
                    second_operand<false>(qb[p], base + W::Q + by_token + (p * C * W::LDK + 16 * s) * 2);
                }
                mma_planes<MT>(ks, klo, a, kb);
                mma_planes<MT>(qs, qlo, a, qb);
            }
            #pragma unroll
            for (int mt = 0; mt < MT; mt++)
                #pragma unroll
                for (int c = 0; c < 4; c++) { ks[mt][c] += klo[mt][c]; qs[mt][c] = __fmul_rn(g[c & 1], qs[mt][c] + qlo[mt][c]); }
            if (j + 1 < n_chunks) bar_arrive(6);
        }
        // V - G (K S).  What is not finite must not meet the zeros of earlier tokens' rows in a product: it goes in as 0.  Its own token's results, and
        // the state if that is the last token, have its terms apart; behind its token the column's results and its state are NaN.
        bool bad = false;
        float x[MT][4];
        auto finite = [&](float& r) {
            if (!(fabsf(r) < 3.3e38f)) { bad = true; return 0.f; }
            return r;
        };
        auto remember = [&](const float (&r)[MT][4]) {
            #pragma unroll
            for (int mt = 0; mt < MT; mt++)
                #pragma unroll
                for (int c = 0; c < 4; c++)
                    if (!(fabsf(r[mt][c]) < 3.3e38f)) atomicMin(first + column(mt, c) - col0, 8 * w + pair + (c & 1));
            bar_multipliers();
        };
        #pragma unroll
        for (int mt = 0; mt < MT; mt++) {
            float r[4];
            #pragma unroll
            for (int c = 0; c < 4; c++) {
                x[mt][c] = fmaf(-g[c & 1], ks[mt][c], v[mt][c]);
                r[c] = finite(x[mt][c]);
            }
            leave<MT>(sb + W::R, w, mt, lane, r);
        }
        const float e0 = e[0], e1 = e[1], to0 = t_own[0], to1 = t_own[1], po0 = p_own[0], po1 = p_own[1], ge = g_end;
        const int n_last = min(C, hi - lo - j * C) - 1;
        if (j + 1 < n_chunks) ask(j + 1);
        bool any = bar_any(bad);
        if (any) remember(x);
        // U = T (..): a row meets its own and earlier steps of 16 tokens
        {
            float hi4[MT][4] = {}, lo4[MT][4] = {};
            bar_wait(3);
            #pragma unroll
            for (int s = 0; s < 4; s++)
                if (s <= w >> 1) {
                    uint4 a[MT][3];
                    unsigned tb[3][2];
                    first_operand<MT>(a, sb + W::R, s, lane);
                    #pragma unroll
                    for (int p = 0; p < 3; p++) second_operand<false>(tb[p], base + W::T + by_row + (p * C * W::LDT + 16 * s) * 2);
                    mma_planes<MT>(hi4, lo4, a, tb);
                }
            if (j + 1 < n_chunks) bar_arrive(7);
            bad = false;
            #pragma unroll
            for (int mt = 0; mt < MT; mt++) {
                float r[4], re[4];
                #pragma unroll
                for (int c = 0; c < 4; c++) {
                    x[mt][c] = fmaf((c & 1) ? to1 : to0, x[mt][c], hi4[mt][c] + lo4[mt][c]);
                    r[c] = finite(x[mt][c]);
                    re[c] = __fmul_rn((c & 1) ? e1 : e0, r[c]);
                    if (8 * w + pair + (c & 1) == n_last) {
                        last[column(mt, c) - col0] = __fmul_rn((c & 1) ? e1 : e0, x[mt][c]);
                        re[c] = 0.f;
                    }
                }
                leave<MT>(sb + W::U, w, mt, lane, r);
                leave<MT>(sb + W::E, w, mt, lane, re);
            }
        }
        if (bar_any(bad)) {
            any = true;
            remember(x);
        }
        // O = G (Q S) + P U
        {
            float hi4[MT][4] = {}, lo4[MT][4] = {};
            bar_wait(4);
            #pragma unroll
            for (int s = 0; s < 4; s++)
                if (s <= w >> 1) {
                    uint4 a[MT][3];
                    unsigned pb[3][2];
                    first_operand<MT>(a, sb + W::U, s, lane);
                    #pragma unroll
                    for (int p = 0; p < 3; p++) second_operand<false>(pb[p], base + W::P + by_row + (p * C * W::LDT + 16 * s) * 2);
                    mma_planes<MT>(hi4, lo4, a, pb);
                }
            if (j + 1 < n_chunks) bar_arrive(8);
            const int t0 = lo + j * C + 8 * w + pair;
            #pragma unroll
            for (int mt = 0; mt < MT; mt++)
                #pragma unroll
                for (int c = 0; c < 4; c++) {
                    float o = fmaf((c & 1) ? po1 : po0, x[mt][c], qs[mt][c] + (hi4[mt][c] + lo4[mt][c]));
                    if (any && 8 * w + pair + (c & 1) > first[column(mt, c) - col0]) o = CUDART_NAN_F;
                    if (t0 + (c & 1) < hi && column(mt, c) < dv) out[(size_t)(t0 + (c & 1)) * H * dv + (size_t)h * dv + column(mt, c)] = o;
                }
        }
        // the state: S <- G_end S + K^T ((G_end / G) U)
        {
            float hi4[NT][MT][4] = {}, lo4[NT][MT][4] = {};
            #pragma unroll
            for (int s = 0; s < 4; s++) {
                uint4 a[MT][3];
                first_operand<MT>(a, sb + W::E, s, lane);
                #pragma unroll
                for (int i = 0; i < NT; i++) {
                    unsigned kb[3][2];
                    #pragma unroll
                    for (int p = 0; p < 3; p++) second_operand<true>(kb[p], base + W::K + by_component + ((p * C + 16 * s) * W::LDK + 8 * i) * 2);
                    mma_planes<MT>(hi4[i], lo4[i], a, kb);
                }
            }
            float k_last[NT][2], u_last[MT][2];              // the last token's key (its planes' sum is the float) and (G_end / G) U
            #pragma unroll
            for (int i = 0; i < NT; i++) {
                const char* at = sb + W::K + (n_last * W::LDK + 8 * (w * NT + i) + pair) * 2;
                const unsigned h = *reinterpret_cast<const unsigned*>(at), m = *reinterpret_cast<const unsigned*>(at + C * W::LDK * 2),
                               l = *reinterpret_cast<const unsigned*>(at + 2 * C * W::LDK * 2);
                k_last[i][0] = __uint_as_float(h << 16) + (__uint_as_float(m << 16) + __uint_as_float(l << 16));
                k_last[i][1] = __uint_as_float(h & 0xffff0000u) + (__uint_as_float(m & 0xffff0000u) + __uint_as_float(l & 0xffff0000u));
            }
            #pragma unroll
            for (int mt = 0; mt < MT; mt++)
                #pragma unroll
                for (int c = 0; c < 2; c++) u_last[mt][c] = last[16 * mt + row + 8 * c];
            if (j + 1 < n_chunks) bar_arrive(5);
            #pragma unroll
            for (int i = 0; i < NT; i++)
                #pragma unroll
                for (int mt = 0; mt < MT; mt++)
                    #pragma unroll
                    for (int c = 0; c < 4; c++) {
                        S[i][mt][c] = fmaf(k_last[i][c & 1], u_last[mt][c >> 1], fmaf(ge, S[i][mt][c], hi4[i][mt][c] + lo4[i][mt][c]));
                        if (any && first[column(mt, c) - col0] < n_last) S[i][mt][c] = CUDART_NAN_F;
                    }
        }
        if (j + 1 < n_chunks) {
            leave_state();                               // (last read before the barrier behind V - G (K S))
            bar_multipliers();
            if (any && threadIdx.x < 16 * MT) first[threadIdx.x] = C;      // (next touched behind the next barrier)
        }
    }
    #pragma unroll
    for (int i = 0; i < NT; i++)
        #pragma unroll
        for (int mt = 0; mt < MT; mt++)
            #pragma unroll
            for (int c = 0; c < 4; c++)
                if (column(mt, c) < dv) st_out[(size_t)column(mt, c) * DK + 8 * (w * NT + i) + pair + (c & 1)] = S[i][mt][c];
}

template <int DK, int MT, bool SOME>
int walk(const float* u, int ldu, int q_off, int k_off, int v_off, const float* scratch, const float* vecs, float* state, const int* slots,
         const int* cu_seqlens, const int* kv_lens, float* out, int B, int least, int n_walked, int H, int G, int dv, cudaStream_t stream) {
    constexpr size_t smem = Walk<DK, MT>::BYTES;
    const cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel<DK, MT, SOME>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    IK_RETURN_IF_ERROR(ik_launch(delta_chunk_kernel<DK, MT, SOME>, dim3((dv + 16 * MT - 1) / (16 * MT), H, n_walked), ALL, smem, stream, u, ldu, q_off, k_off,
                                 v_off, scratch, vecs, state, slots, cu_seqlens, kv_lens, out, B, least, H, G, dv));
    IK_LAUNCH_STATUS();
}

template <int DK, bool SOME>
int chunks(const float* u, int ldu, int q_off, int k_off, int v_off, const float* bg, float* scratch, float* state, const int* slots,
           const int* cu_seqlens, const int* kv_lens, float* out, int B, int least, int n_walked, int n_chunks, int H, int G, int dv,
           cudaStream_t stream) {
    float* vecs = scratch + (size_t)n_chunks * H * 2 * C * C;
    constexpr size_t smem = (2 * C * (DK + 4) + C) * sizeof(float) + C * sizeof(double);          // (DK is at least 64: M and T fit)
    const cudaError_t e = cudaFuncSetAttribute(delta_chunk_prepare_kernel<DK, SOME>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    IK_RETURN_IF_ERROR(ik_launch(delta_chunk_prepare_kernel<DK, SOME>, dim3(n_chunks, H), 256, smem, stream, u, ldu, q_off, k_off, bg, scratch, vecs,
                                 cu_seqlens, B, least, H, G));
    // 32 columns a block do a third fewer loads per multiply-add; 16 where that leaves more than half of the SMs idle
    if (2LL * n_walked * H * ((dv + 31) / 32) <= ik_sm_count())
        return walk<DK, 1, SOME>(u, ldu, q_off, k_off, v_off, scratch, vecs, state, slots, cu_seqlens, kv_lens, out, B, least, n_walked, H, G, dv, stream);
    return walk<DK, 2, SOME>(u, ldu, q_off, k_off, v_off, scratch, vecs, state, slots, cu_seqlens, kv_lens, out, B, least, n_walked, H, G, dv, stream);
}

}  // namespace

// Floats of scratch for B sequences of T tokens together; 0 where the chunks do not apply (short prompts, key sizes other than 64 and
// 128, value sizes that are no multiple of 4): ik_delta_rule runs those.
IK_EXPORT long long ik_delta_chunks_scratch(int T, int B, int max_new, int H, int dk, int dv) {
    if (T <= 0 || B <= 0 || B > 65535 || H > 65535 || max_new < C || (dk != 64 && dk != 128) || dv % 4) return 0;
    return (long long)(T / C + B) * H * (2 * C * C + VEC);
}

// As ik_delta_rule, a chunk of tokens at a time, for the sequences that bring at least `least` tokens (the others are left alone): at
// most n_walked of them, of at most n_chunks chunks together, for which scratch has room.  least 1: all of them, n_walked = B and n_chunks =
// T / 64 + B.  IK_UNSUPPORTED where rows of q, k or v are not on 16 bytes.
IK_EXPORT int ik_delta_chunks(const float* u, int ldu, int q_off, int k_off, int v_off, const float* bg, float* state, const int* slots,
                              const int* cu_seqlens, const int* kv_lens, float* out, float* scratch, int T, int B, int least, int n_walked,
                              int n_chunks, int H, int G, int dk, int dv, cudaStream_t stream) {
    if (T < 0 || B < 0 || least <= 0 || n_walked < 0 || n_chunks < 0 || n_walked > 65535 || H <= 0 || G <= 0 || H % G || dv <= 0 || !state || !bg ||
        !scratch) return IK_BAD_ARGUMENT;
    if (least == 1 && (n_walked != B || n_chunks != T / C + B)) return IK_BAD_ARGUMENT;
    if (T == 0 || B == 0 || n_walked == 0 || n_chunks == 0) return IK_OK;
    if (ldu % 4 || q_off % 4 || k_off % 4 || v_off % 4 || dv % 4 || ((uintptr_t)u | (uintptr_t)out | (uintptr_t)scratch) % 16) return IK_UNSUPPORTED;
#define IK_CHUNKS(DK)                                                                                                                       \
    if (dk == DK)                                                                                                                           \
        return (least == 1 ? chunks<DK, false> : chunks<DK, true>)(u, ldu, q_off, k_off, v_off, bg, scratch, state, slots, cu_seqlens, kv_lens, out, B, \
                                                                   least, n_walked, n_chunks, H, G, dv, stream)
    IK_CHUNKS(128);
    IK_CHUNKS(64);
#undef IK_CHUNKS
    return IK_UNSUPPORTED;
}
