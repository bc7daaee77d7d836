// The gated delta rule for prompts, 64 tokens at a time (the 16-bit path; every number here is float, as in delta.cu).
//
// Within a chunk, with G_t the product of the decays up to token t and M[t, s] = b_t (G_t / G_s) (k_t . k_s) for s < t, the
// corrections u_t of all tokens solve a triangular system: (I + M) U = b (V - G (K S)), S the state before the chunk.  So
//   U = T (V - G (K S)) with T = (I + M)^-1 diag(b);   O = G (Q S) + P U with P[t, s] = (G_t / G_s) (q_t . k_s), s <= t;
//   S <- G_end S + K^T ((G_end / G) U).
// delta_chunk_prepare_kernel forms T and P of every chunk and head side by side; delta_chunk_kernel walks a sequence's chunks with
// a slice of a head's columns per block: five small products a chunk in place of 64 dependent steps.  The tokens' chain is what
// bounds the token-by-token kernel (0.37 to 0.4 us a token; which sequences of a step go which way: ops.delta_chunks_from); the chunks' chain is bound by the walk's
// reads from shared memory (half a 16-byte read per four multiply-adds and thread, and an SM returns 128 bytes of reads a cycle)
// beside its multiply-adds, about 8,200 cycles a chunk and block at full rate.
// Measured on B200: a layer 2,048 wide with 16 heads of 128 over two prompts of 3,000 and fewer tokens 2,776 -> 790 us (the rule itself
// 2,240 -> 600: 89 us of T and P, 509 us of the walk, 10.8 us a chunk; with 512 threads, each half the results, the walk took 606).
#include "common.cuh"

namespace {

constexpr int C = 64;                                    // tokens of a chunk
constexpr int TLD = C + 4;                               // row stride of T and P in shared memory
constexpr int VEC = 132;                                 // floats of a chunk's decays: G [64], G_end / G [64], G_end, padding

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
            outP[t * C + s] = s <= t ? ratio * qk[i][j] : 0.f;
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
    for (int i = tid; i < C * C; i += 256) {
        const int t = i / C, s = i % C;
        outT[i] = (s >> 4) <= (t >> 4) ? Ts[t * TLD + s] * beta[s] : 0.f;
    }
}

// One block per (columns of a head, value head, walked sequence); DS columns.  A thread owns 4 columns of one or two rows of the chunk's
// products (ty and 63 - ty: the triangular products then take every warp equally long), and 4 columns of DK / RG neighbouring
// rows of the state (in registers; shared memory holds a copy to read from).
template <int DK, int DS>
struct Walk {
    static constexpr int CG = DS / 4, RG = 256 / CG, LD = DK + 4;
    static constexpr int RK = C / RG, RS = DK / RG;      // rows of K (and of Q), and of the state, a thread owns
    static constexpr int FLOATS = 4 * C * LD + C * TLD + 2 * C * TLD + 3 * C * DS + DK * DS + 2 * VEC;
};

template <int DK, int DS, bool SOME>
__global__ void __launch_bounds__(256, 1)
delta_chunk_kernel(const float* __restrict__ u, int ldu, int q_off, int k_off, int v_off, const float* __restrict__ scratch, const float* __restrict__ vecs,
                   float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ cu_seqlens,
                   const int* __restrict__ kv_lens, float* __restrict__ out, int n_seqs, int least, int H, int G, int dv) {
    typedef Walk<DK, DS> W;
    constexpr int LD = W::LD, RG = W::RG, RK = W::RK, RS = W::RS;
    extern __shared__ __align__(16) float sm[];
    float* const KQ = sm;                                // [2][K, Q][64][LD]
    float* const Ts = KQ + 4 * C * LD;                   // [64][TLD]
    float* const Ps = Ts + C * TLD;                      // [2][64][TLD]
    float* const Vs = Ps + 2 * C * TLD;                  // [64][DS]
    float* const Us = Vs + C * DS;                       // [64][DS]: V - G (K S), then U
    float* const Es = Us + C * DS;                       // [64][DS]: (G_end / G) U
    float* const Ss = Es + C * DS;                       // [DK][DS]
    float* const vec = Ss + DK * DS;                     // [2][VEC]
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
    const int tid = threadIdx.x, b = seq.b, h = blockIdx.y, col0 = blockIdx.x * DS;
    const int lo = cu_seqlens[b], hi = cu_seqlens[b + 1], end = kv_lens[b], start = end - (hi - lo);
    if (!SOME && hi <= lo) return;
    const int tx = tid % W::CG, ty = tid / W::CG, kvh = h / (H / G);
    const int col = col0 + 4 * tx, k0 = RS * ty;
    auto row = [&](int i) { return i == 0 ? ty : C - 1 - ty; };
    static_assert(RK * RG == C && RK <= 2, "a thread's rows");
    const bool live = col < dv;                          // dv is a multiple of 4
    const size_t per = (size_t)H * DK * dv;
    const float* st_in = state + ((size_t)slots[b] * 2 + ((start - 1) & 1)) * per + ((size_t)h * dv + (live ? col : 0)) * DK + k0;
    float* st_out = state + ((size_t)slots[b] * 2 + ((end - 1) & 1)) * per + ((size_t)h * dv + (live ? col : 0)) * DK + k0;
    const int f0 = SOME ? seq.chunk0 : chunk_base(cu_seqlens, b), n_chunks = (hi - lo + C - 1) / C;

    auto bring_kq = [&](int j) {
        float* dst = KQ + (j & 1) * 2 * C * LD;
        const int t0 = lo + j * C, n = min(C, hi - t0);
        for (int i = tid; i < 2 * C * (DK / 4); i += 256) {
            const int r = i / (DK / 4), w = i % (DK / 4), t = r & (C - 1);
            copy16(dst + r * LD + 4 * w, u + (size_t)(t0 + min(t, n - 1)) * ldu + (r < C ? k_off : q_off) + kvh * DK + 4 * w, t < n);
        }
        const float* p = scratch + ((size_t)(f0 + j) * H + h) * 2 * C * C + C * C;
        for (int i = tid; i < C * (C / 4); i += 256) copy16(Ps + (j & 1) * C * TLD + (i / (C / 4)) * TLD + 4 * (i % (C / 4)), p + 4 * i, true);
        const float* ve = vecs + ((size_t)(f0 + j) * H + h) * VEC;
        if (tid < VEC / 4) copy16(vec + (j & 1) * VEC + 4 * tid, ve + 4 * tid, true);
    };
    auto bring_tv = [&](int j) {
        const int t0 = lo + j * C, n = min(C, hi - t0);
        const float* p = scratch + ((size_t)(f0 + j) * H + h) * 2 * C * C;
        for (int i = tid; i < C * (C / 4); i += 256) copy16(Ts + (i / (C / 4)) * TLD + 4 * (i % (C / 4)), p + 4 * i, true);
        for (int i = tid; i < C * W::CG; i += 256) {
            const int t = i / W::CG, w = col0 + 4 * (i % W::CG);
            copy16(Vs + 4 * i, u + (size_t)(t0 + min(t, n - 1)) * ldu + v_off + h * dv + min(w, dv - 4), t < n && w < dv);
        }
    };
    bring_kq(0);
    bring_tv(0);
    copies_commit();
    float S[RS][4];                                      // [row k0 + r][column c]
    #pragma unroll
    for (int c = 0; c < 4; c++)
        #pragma unroll
        for (int r = 0; r < RS; r++) S[r][c] = live && start > 0 ? st_in[(size_t)c * DK + r] : 0.f;

    for (int j = 0; j < n_chunks; j++) {
        #pragma unroll
        for (int r = 0; r < RS; r++) *reinterpret_cast<float4*>(Ss + (k0 + r) * DS + 4 * tx) = make_float4(S[r][0], S[r][1], S[r][2], S[r][3]);
        copies_wait();
        __syncthreads();                                 // this chunk's K, Q, P, T, V and the state are there
        if (j + 1 < n_chunks) { bring_kq(j + 1); copies_commit(); }
        const float* K = KQ + (j & 1) * 2 * C * LD;
        const float* P = Ps + (j & 1) * C * TLD;
        const float* gam = vec + (j & 1) * VEC;
        // K S and Q S
        float ks[RK][4] = {}, qs[RK][4] = {};
        #pragma unroll 2
        for (int d = 0; d < DK; d += 4) {
            float4 s[4], a;
            #pragma unroll
            for (int e = 0; e < 4; e++) s[e] = at4(Ss + (d + e) * DS + 4 * tx);
            #pragma unroll
            for (int i = 0; i < 2 * RK; i++) {
                a = at4(K + ((i < RK ? 0 : C) + row(i % RK)) * LD + d);
                float (&acc)[4] = i < RK ? ks[i % RK] : qs[i % RK];
                const float av[4] = {a.x, a.y, a.z, a.w};
                #pragma unroll
                for (int e = 0; e < 4; e++) {
                    acc[0] = fmaf(av[e], s[e].x, acc[0]); acc[1] = fmaf(av[e], s[e].y, acc[1]);
                    acc[2] = fmaf(av[e], s[e].z, acc[2]); acc[3] = fmaf(av[e], s[e].w, acc[3]);
                }
            }
        }
        #pragma unroll
        for (int i = 0; i < RK; i++) {
            const int t = row(i);
            const float4 v = at4(Vs + t * DS + 4 * tx);
            const float g = gam[t];
            *reinterpret_cast<float4*>(Us + t * DS + 4 * tx) = make_float4(fmaf(-g, ks[i][0], v.x), fmaf(-g, ks[i][1], v.y),
                                                                           fmaf(-g, ks[i][2], v.z), fmaf(-g, ks[i][3], v.w));
        }
        __syncthreads();
        // U = T (...), then O = G (Q S) + P U: lower triangles.  A row meets its own and earlier tokens only (not zeros times
        // later ones: their infinities would show).
        auto lower = [&](const float* A, float (&acc)[RK][4]) {
            #pragma unroll
            for (int i = 0; i < RK; i++) {
                const int t = row(i);
                const float* a = A + t * TLD;
                #pragma unroll 4
                for (int s = 0; s < (t & ~3); s += 4) {
                    const float4 a4 = at4(a + s);
                    const float av[4] = {a4.x, a4.y, a4.z, a4.w};
                    #pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const float4 x = at4(Us + (s + e) * DS + 4 * tx);
                        acc[i][0] = fmaf(av[e], x.x, acc[i][0]); acc[i][1] = fmaf(av[e], x.y, acc[i][1]);
                        acc[i][2] = fmaf(av[e], x.z, acc[i][2]); acc[i][3] = fmaf(av[e], x.w, acc[i][3]);
                    }
                }
                for (int s = t & ~3; s <= t; s++) {
                    const float w = a[s];
                    const float4 x = at4(Us + s * DS + 4 * tx);
                    acc[i][0] = fmaf(w, x.x, acc[i][0]); acc[i][1] = fmaf(w, x.y, acc[i][1]);
                    acc[i][2] = fmaf(w, x.z, acc[i][2]); acc[i][3] = fmaf(w, x.w, acc[i][3]);
                }
            }
        };
        float un[RK][4] = {};
        lower(Ts, un);
        __syncthreads();                                 // everybody has read the right-hand sides, T and V
        #pragma unroll
        for (int i = 0; i < RK; i++) {
            const int t = row(i);
            const float e = gam[C + t];
            *reinterpret_cast<float4*>(Us + t * DS + 4 * tx) = make_float4(un[i][0], un[i][1], un[i][2], un[i][3]);
            *reinterpret_cast<float4*>(Es + t * DS + 4 * tx) = make_float4(e * un[i][0], e * un[i][1], e * un[i][2], e * un[i][3]);
        }
        if (j + 1 < n_chunks) { bring_tv(j + 1); copies_commit(); }
        __syncthreads();
        const int t0 = lo + j * C;
        #pragma unroll
        for (int i = 0; i < RK; i++) {
            const float g = gam[row(i)];
            #pragma unroll
            for (int c = 0; c < 4; c++) qs[i][c] *= g;
        }
        lower(P, qs);
        #pragma unroll
        for (int i = 0; i < RK; i++) {
            const int t = t0 + row(i);
            if (live && t < hi) *reinterpret_cast<float4*>(out + (size_t)t * H * dv + (size_t)h * dv + col) = make_float4(qs[i][0], qs[i][1], qs[i][2], qs[i][3]);
        }
        // the state: S <- G_end S + K^T E
        const float g_end = gam[2 * C];
        #pragma unroll
        for (int r = 0; r < RS; r++)
            #pragma unroll
            for (int c = 0; c < 4; c++) S[r][c] *= g_end;
        #pragma unroll 4
        for (int t = 0; t < C; t++) {
            const float4 x = at4(Es + t * DS + 4 * tx);
            float a[RS];
            if (RS == 4) { const float4 a4 = at4(K + t * LD + k0); a[0] = a4.x; a[1 % RS] = a4.y; a[2 % RS] = a4.z; a[3 % RS] = a4.w; }
            else if (RS == 2) { const float2 a2 = *reinterpret_cast<const float2*>(K + t * LD + k0); a[0] = a2.x; a[1 % RS] = a2.y; }
            else a[0] = K[t * LD + k0];
            #pragma unroll
            for (int r = 0; r < RS; r++) {
                S[r][0] = fmaf(a[r], x.x, S[r][0]); S[r][1] = fmaf(a[r], x.y, S[r][1]);
                S[r][2] = fmaf(a[r], x.z, S[r][2]); S[r][3] = fmaf(a[r], x.w, S[r][3]);
            }
        }
        // (the copy of the state is written anew before the next barrier; it was last read before the one after K S)
    }
    if (live) {
        #pragma unroll
        for (int c = 0; c < 4; c++)
            #pragma unroll
            for (int r = 0; r < RS; r++) st_out[(size_t)c * DK + r] = S[r][c];
    }
}

template <int DK, int DS, bool SOME>
int walk(const float* u, int ldu, int q_off, int k_off, int v_off, const float* scratch, const float* vecs, float* state, const int* slots,
         const int* cu_seqlens, const int* kv_lens, float* out, int B, int least, int n_walked, int H, int G, int dv, cudaStream_t stream) {
    constexpr size_t smem = Walk<DK, DS>::FLOATS * sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel<DK, DS, SOME>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    IK_RETURN_IF_ERROR(ik_launch(delta_chunk_kernel<DK, DS, SOME>, dim3((dv + DS - 1) / DS, H, n_walked), 256, smem, stream, u, ldu, q_off, k_off, v_off,
                                 scratch, vecs, state, slots, cu_seqlens, kv_lens, out, B, least, H, G, dv));
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
        return walk<DK, 16, SOME>(u, ldu, q_off, k_off, v_off, scratch, vecs, state, slots, cu_seqlens, kv_lens, out, B, least, n_walked, H, G, dv, stream);
    return walk<DK, 32, SOME>(u, ldu, q_off, k_off, v_off, scratch, vecs, state, slots, cu_seqlens, kv_lens, out, B, least, n_walked, H, G, dv, stream);
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
