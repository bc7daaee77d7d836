// Mixers that carry a state of fixed size from token to token: a short causal convolution with bias and
// activation, the selective scan, and linear attention with a constant decay per head.
//
// All of them work on the step's token-major batch: sequence b brings tokens cu_seqlens[b] .. cu_seqlens[b+1] - 1,
// which sit at positions kv_lens[b] - n_b .. kv_lens[b] - 1; its state lives in slot slots[b].  A sequence whose
// first token sits at position 0 starts from zeros whatever its slot holds.
//
// State that a step replaces (the scan's and the linear attention's) is kept twice, by the parity of the
// position it belongs to: a step that ends at position e reads the copy of parity (first - 1) & 1 and writes
// the copy of parity e & 1.  A decode step therefore never overwrites what it read, so running the same step
// again (a captured graph replayed after its warm-up run, a step launched ahead and dropped) gives the same
// state.  The convolution's history is a ring of `taps` positions, position p in place p mod taps, with the same
// property.
//
// Everything is float: decays, step sizes, softplus, exponentials, states and their sums.  Only the inputs that
// come out of a projection or a convolution may be 16-bit.
#include "common.cuh"

__device__ __forceinline__ float ik_silu(float x) { return x / (1.0f + expf(-x)); }
// ... as a result of the given type: what is rounded to 16 bits anyway takes the hardware's approximate exponential and quotient
// (relative error near 1e-6)
template <typename TO> __device__ __forceinline__ float ik_silu_for(float x) {
    return sizeof(TO) == 2 ? __fdividef(x, 1.0f + __expf(-x)) : ik_silu(x);
}
__device__ __forceinline__ float ik_sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float ik_softplus(float x) { return x > 20.0f ? x : log1pf(expf(x)); }

// ------------------------------------------------------------------ causal convolution
// y[p, c] = act(b[c] + sum_j w[j, c] * u[p - taps + 1 + j, c]), u = 0 before the sequence's start.  u of this step's
// tokens comes from x (row stride ldx), older ones from the ring.  w is tap-major [taps, C].
// inline_ring: every sequence brings one token, so the kernel also writes u[p] into the ring (nobody reads that place
// in this step); otherwise conv_ring_kernel does it afterwards.
template <typename TO>
__global__ void __launch_bounds__(256)
causal_conv_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ w, const float* __restrict__ bias,
                   float* __restrict__ ring, const int* __restrict__ slots, const int* __restrict__ cu_seqlens,
                   const int* __restrict__ token_seq, const int* __restrict__ token_pos, TO* __restrict__ out,
                   int T, int C, int taps, int act, int inline_ring) {
    ik_pdl_wait();
    IK_AFTER_WAIT(x);
    IK_AFTER_WAIT(slots);
    IK_AFTER_WAIT(cu_seqlens);
    IK_AFTER_WAIT(token_seq);
    IK_AFTER_WAIT(token_pos);
    ik_pdl_launch_dependents();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)T * C) return;
    const int t = (int)(idx / C), c = (int)(idx - (size_t)t * C);
    const int b = token_seq[t], pos = token_pos[t], first = cu_seqlens[b];
    const float* rg = ring ? ring + (size_t)slots[b] * taps * C : nullptr;
    float acc = bias ? bias[c] : 0.f;
    for (int j = 0; j < taps; j++) {
        const int back = taps - 1 - j;                   // the input `back` positions ago
        if (back > pos) continue;                        // before the sequence's start
        float u;
        if (t - back >= first) u = x[(size_t)(t - back) * ldx + c];
        else u = rg[(size_t)((pos - back) % taps) * C + c];
        acc = fmaf(w[(size_t)j * C + c], u, acc);
    }
    if (inline_ring && ring) ring[((size_t)slots[b] * taps + pos % taps) * C + c] = x[(size_t)t * ldx + c];
    ik_st(out, idx, act ? ik_silu_for<TO>(acc) : acc);
}

// The same for four neighbouring channels per thread (channel counts and row distances that are multiples of four,
// aligned pointers): 16-byte accesses, and a token's few index computations once per four results.
template <typename TO>
__global__ void __launch_bounds__(256)
causal_conv4_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ w, const float* __restrict__ bias,
                    float* __restrict__ ring, const int* __restrict__ slots, const int* __restrict__ cu_seqlens,
                    const int* __restrict__ token_seq, const int* __restrict__ token_pos, TO* __restrict__ out,
                    int T, int C, int taps, int act, int inline_ring) {
    ik_pdl_wait();
    IK_AFTER_WAIT(x);
    IK_AFTER_WAIT(slots);
    IK_AFTER_WAIT(cu_seqlens);
    IK_AFTER_WAIT(token_seq);
    IK_AFTER_WAIT(token_pos);
    ik_pdl_launch_dependents();
    const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4, t = blockIdx.x;
    if (c >= C) return;
    const int b = token_seq[t], pos = token_pos[t], first = cu_seqlens[b];
    const float* rg = ring ? ring + (size_t)slots[b] * taps * C : nullptr;
    float4 acc = bias ? ik_ld4(bias, c) : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = 0; j < taps; j++) {
        const int back = taps - 1 - j;
        if (back > pos) continue;
        const float4 u = t - back >= first ? ik_ld4(x, (size_t)(t - back) * ldx + c) : ik_ld4(rg, (size_t)((pos - back) % taps) * C + c);
        const float4 wj = ik_ld4(w, (size_t)j * C + c);
        acc.x = fmaf(wj.x, u.x, acc.x); acc.y = fmaf(wj.y, u.y, acc.y); acc.z = fmaf(wj.z, u.z, acc.z); acc.w = fmaf(wj.w, u.w, acc.w);
    }
    if (inline_ring && ring) ik_st4(ring, ((size_t)slots[b] * taps + pos % taps) * C + c, ik_ld4(x, (size_t)t * ldx + c));
    if (act) { acc.x = ik_silu_for<TO>(acc.x); acc.y = ik_silu_for<TO>(acc.y); acc.z = ik_silu_for<TO>(acc.z); acc.w = ik_silu_for<TO>(acc.w); }
    ik_st4(out, (size_t)t * C + c, acc);
}

// The same for prompts: a thread takes RUN neighbouring tokens of its four channels and keeps the inputs behind the current
// one in registers, so an input is read once (and TAPS - 1 more at the run's start and where a sequence begins) instead of TAPS
// times.  The sum of a token runs in the same order as above.  What bounds it is the bytes, as long as enough blocks have their loads under way: runs of
// eight in 118 registers (two blocks an SM) took 41 us for 4,910 tokens of 3,072 channels in float and 36 of 4,096 in 16 bits, of four in 80 37 and 36,
// of four in 64 (four blocks) 31 and 30, of two 40 and 41 (18 for the bytes).
template <typename TO, int TAPS, int RUN>
__global__ void __launch_bounds__(256, 4)
causal_conv4_run_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ w, const float* __restrict__ bias,
                        const float* __restrict__ ring, const int* __restrict__ slots, const int* __restrict__ cu_seqlens,
                        const int* __restrict__ token_seq, const int* __restrict__ token_pos, TO* __restrict__ out, int T, int C, int act) {
    ik_pdl_wait();
    IK_AFTER_WAIT(x);
    IK_AFTER_WAIT(ring);
    IK_AFTER_WAIT(slots);
    IK_AFTER_WAIT(cu_seqlens);
    IK_AFTER_WAIT(token_seq);
    IK_AFTER_WAIT(token_pos);
    ik_pdl_launch_dependents();
    const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4, t0 = blockIdx.x * RUN;
    if (c >= C) return;
    float4 now[RUN], wj[TAPS], past[TAPS - 1];
    #pragma unroll
    for (int r = 0; r < RUN; r++) now[r] = t0 + r < T ? ik_ld4(x, (size_t)(t0 + r) * ldx + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    #pragma unroll
    for (int j = 0; j < TAPS; j++) wj[j] = ik_ld4(w, (size_t)j * C + c);
    const float4 b4 = bias ? ik_ld4(bias, c) : make_float4(0.f, 0.f, 0.f, 0.f);
    int seq = -1;
    #pragma unroll
    for (int r = 0; r < RUN; r++) {
        const int t = t0 + r;
        if (t >= T) break;
        const int b = token_seq[t];
        if (r == 0 || b != seq) {                          // the inputs behind this token: of this step, older ones, or none
            const int pos = token_pos[t], first = cu_seqlens[b];
            seq = b;
            #pragma unroll
            for (int j = 0; j < TAPS - 1; j++) {
                const int back = TAPS - 1 - j;
                past[j] = back > pos ? make_float4(0.f, 0.f, 0.f, 0.f)
                        : t - back >= first ? ik_ld4(x, (size_t)(t - back) * ldx + c)
                                            : ik_ld4(ring, ((size_t)slots[b] * TAPS + (pos - back) % TAPS) * C + c);
            }
        }
        float4 acc = b4;
        #pragma unroll
        for (int j = 0; j < TAPS; j++) {
            const float4 u = j < TAPS - 1 ? past[j] : now[r];
            acc.x = fmaf(wj[j].x, u.x, acc.x); acc.y = fmaf(wj[j].y, u.y, acc.y); acc.z = fmaf(wj[j].z, u.z, acc.z); acc.w = fmaf(wj[j].w, u.w, acc.w);
        }
        #pragma unroll
        for (int j = 0; j < TAPS - 1; j++) past[j] = j < TAPS - 2 ? past[j + 1] : now[r];
        if (act) { acc.x = ik_silu_for<TO>(acc.x); acc.y = ik_silu_for<TO>(acc.y); acc.z = ik_silu_for<TO>(acc.z); acc.w = ik_silu_for<TO>(acc.w); }
        ik_st4(out, (size_t)t * C + c, acc);
    }
}

// The last `taps` inputs of every sequence go into its ring.
__global__ void __launch_bounds__(256)
conv_ring_kernel(const float* __restrict__ x, int ldx, float* __restrict__ ring, const int* __restrict__ slots,
                 const int* __restrict__ cu_seqlens, const int* __restrict__ kv_lens, int C, int taps) {
    ik_pdl_wait();
    IK_AFTER_WAIT(x);
    IK_AFTER_WAIT(slots);
    IK_AFTER_WAIT(cu_seqlens);
    IK_AFTER_WAIT(kv_lens);
    ik_pdl_launch_dependents();
    const int b = blockIdx.y;
    const int lo = cu_seqlens[b], hi = cu_seqlens[b + 1], end = kv_lens[b];
    const int n = min(taps, hi - lo);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n * C; i += gridDim.x * blockDim.x) {
        const int k = i / C, c = i - k * C;              // the k-th of the last n tokens
        const int t = hi - n + k, pos = end - n + k;
        ring[((size_t)slots[b] * taps + pos % taps) * C + c] = x[(size_t)t * ldx + c];
    }
}

IK_EXPORT int ik_causal_conv(const float* x, int ldx, const float* w, const float* bias, float* ring, const int* slots,
                             const int* cu_seqlens, const int* kv_lens, const int* token_seq, const int* token_pos,
                             void* out, int out_dtype, int T, int B, int C, int taps, int act, int one_token_each,
                             cudaStream_t stream) {
    if (T < 0 || B < 0 || C <= 0 || taps <= 0 || ldx < C || (taps > 1 && !ring)) return IK_BAD_ARGUMENT;
    if (T == 0) return IK_OK;
    const size_t total = (size_t)T * C;
    const int blocks = (int)((total + 255) / 256);
    const int inl = one_token_each && taps > 1;
    const bool by4 = C % 4 == 0 && ldx % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0 && (uintptr_t)out % 16 == 0 &&
                     (!bias || (uintptr_t)bias % 16 == 0) && (!ring || (uintptr_t)ring % 16 == 0);
    if (by4 && (out_dtype == IK_F32 || out_dtype == IK_BF16)) {
        const int threads = C / 4 >= 256 ? 256 : ((C / 4 + 31) / 32) * 32;
        const dim3 grid(T, (C / 4 + threads - 1) / threads);
        constexpr int RUN = 4;
        const bool runs = !inl && taps >= 2 && taps <= 4 && (long long)T * grid.y >= 64LL * ik_sm_count();   // enough blocks either way
#define IK_CONV_RUN(TO, TAPS)                                                                                                       \
    IK_RETURN_IF_ERROR(ik_launch(causal_conv4_run_kernel<TO, TAPS, RUN>, dim3((T + RUN - 1) / RUN, grid.y), threads, 0, stream, x, ldx, w, bias, \
                                 (const float*)ring, slots, cu_seqlens, token_seq, token_pos, (TO*)out, T, C, act))
        if (runs && out_dtype == IK_F32) { if (taps == 2) IK_CONV_RUN(float, 2); else if (taps == 3) IK_CONV_RUN(float, 3); else IK_CONV_RUN(float, 4); }
        else if (runs) { if (taps == 2) IK_CONV_RUN(__nv_bfloat16, 2); else if (taps == 3) IK_CONV_RUN(__nv_bfloat16, 3); else IK_CONV_RUN(__nv_bfloat16, 4); }
        else
#undef IK_CONV_RUN
        if (out_dtype == IK_F32)
            IK_RETURN_IF_ERROR(ik_launch(causal_conv4_kernel<float>, grid, threads, 0, stream, x, ldx, w, bias, ring, slots, cu_seqlens,
                                         token_seq, token_pos, (float*)out, T, C, taps, act, inl));
        else
            IK_RETURN_IF_ERROR(ik_launch(causal_conv4_kernel<__nv_bfloat16>, grid, threads, 0, stream, x, ldx, w, bias, ring, slots,
                                         cu_seqlens, token_seq, token_pos, (__nv_bfloat16*)out, T, C, taps, act, inl));
    } else if (out_dtype == IK_F32)
        IK_RETURN_IF_ERROR(ik_launch(causal_conv_kernel<float>, blocks, 256, 0, stream, x, ldx, w, bias, ring, slots, cu_seqlens,
                                     token_seq, token_pos, (float*)out, T, C, taps, act, inl));
    else if (out_dtype == IK_BF16)
        IK_RETURN_IF_ERROR(ik_launch(causal_conv_kernel<__nv_bfloat16>, blocks, 256, 0, stream, x, ldx, w, bias, ring, slots,
                                     cu_seqlens, token_seq, token_pos, (__nv_bfloat16*)out, T, C, taps, act, inl));
    else
        return IK_BAD_ARGUMENT;
    if (taps > 1 && !inl) {
        const dim3 grid(min(64, (taps * C + 255) / 256), B);
        IK_RETURN_IF_ERROR(ik_launch(conv_ring_kernel, grid, 256, 0, stream, x, ldx, ring, slots, cu_seqlens, kv_lens, C, taps));
    }
    IK_LAUNCH_STATUS();
}

// ------------------------------------------------------------------ selective scan
// Per channel c and state n:  S[c, n] <- exp(dt_c A[c, n]) S[c, n] + dt_c u_c B_n;  y_c = sum_n S[c, n] C_n + D_c u_c;
// out = y * silu(z).  dt = softplus(dt_raw + dt_bias).  B_n, C_n are columns of `bc` (row stride ldbc), z of `z`
// (row stride ldz).  L lanes (a power of two) share a channel: lane l holds states l, l + L, ... (NPT of them at most);
// their sums are added by shuffles in a fixed order.  One block row per sequence, tokens in order.
//
// The tokens go through shared memory in tiles: while a tile is computed, the next tile's inputs are on their way
// into registers; softplus and silu are applied when a tile is stored, by all threads at once, so that the
// token-by-token chain holds only the exponential and the multiply-adds.  What is computed for a token does not
// depend on where tiles begin.  FAST (16-bit inputs): exponentials and the gate's sigmoid are the hardware's
// approximations.
template <bool FAST> __device__ __forceinline__ float ik_silu_as(float x) {
    return FAST ? x * __frcp_rn(1.0f + __expf(-x)) : x / (1.0f + expf(-x));
}

// A load that is issued where it stands (the compiler may otherwise sink it to its first use, behind the tile's arithmetic).
__device__ __forceinline__ float ik_ld_now(const float* p) { float v; asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p)); return v; }
// The 16-bit value stays as it was loaded until ik_raw_float turns it into a float where it is used: a conversion next to
// the load would wait for the load.
__device__ __forceinline__ unsigned short ik_ld_now(const __nv_bfloat16* p) {
    unsigned short v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ik_raw_float(float v) { return v; }
__device__ __forceinline__ float ik_raw_float(unsigned short v) { return __uint_as_float((unsigned)v << 16); }
template <typename T> struct IkRaw { typedef float type; };
template <> struct IkRaw<__nv_bfloat16> { typedef unsigned short type; };
template <bool FAST> __device__ __forceinline__ float ik_softplus_as(float x) {
    return x > 20.0f ? x : (FAST ? __logf(1.0f + __expf(x)) : log1pf(expf(x)));
}

// NPT states a thread, L lanes a channel, TT tokens a tile: all fixed at compile time, so that the tile's layout and the
// sum over lanes are constants.  Lane l holds states l*NPT .. l*NPT + NPT - 1; the L*NPT >= N places beyond N are padding
// (A = 0, B = C = 0: they stay zero and add nothing), which spares every guard in the token loop.
// One state's step, S <- exp(dt a) S + dt x B.  16-bit path: float, with the hardware's exponential.  float32 path: the
// factor and the update are formed in double and rounded to float once, so that a step's error is half a unit in the last
// place and has no bias that could add up over thousands of steps (the state itself stays a float).
template <bool FAST> __device__ __forceinline__ float ik_scan_step(float S, float dt, float x, float a, float B) {
    if (FAST) return fmaf(__expf(dt * a), S, dt * x * B);
    return (float)fma(exp((double)dt * (double)a), (double)S, (double)dt * (double)x * (double)B);
}

// Prompts of the 16-bit path are cut into pieces of `piece` tokens that run side by side (token by token a prompt is a chain:
// with one sequence there are hardly two warps a scheduler, each waiting for itself).  MODE 1 runs every piece but a sequence's
// last from a zero state and leaves its end state and the sum of its step sizes in scratch; scan_carry_kernel turns the end
// states into the pieces' states at entry, S <- exp(a * sum dt) S + S_piece; MODE 2 runs the pieces from there and writes the
// results.  MODE 0: whole sequences.  Pieces have flat numbers: piece j of sequence b is cu_seqlens[b] / piece + b + j, of
// which there are at most T / piece + B.
// Which steps go this way: ops.scan_pieces_pay, and ops.scan_pieces_beat_stream where whole sequences run in selective_scan_stream_kernel.  Measured on
// B200, 4,096 channels of 16 states: prompts of 3,000 and 1,910 tokens 685 us with a shuffle tree per token, 399 with the sums of a channel's lanes
// exchanged L tokens at a time (below), 380 in pieces as well, 193 in the stream kernel.
struct ScanPieces {
    int piece;                                        // tokens; 0 = whole sequences
    int n_seqs;
    float* states;                                    // [flat piece][inner][N]: end states, then states at entry
    float* sums;                                      // [flat piece][inner]: sums of the step sizes
};
__device__ __forceinline__ int scan_piece_base(const int* cu_seqlens, int b, int piece) { return cu_seqlens[b] / piece + b; }

template <typename TU, typename TO, bool FAST, int NPT, int L, int TT, int MODE>
__global__ void __launch_bounds__(128)
selective_scan_kernel(const TU* __restrict__ u, const float* __restrict__ dt_raw, const float* __restrict__ dt_bias,
                      const float* __restrict__ A, const float* __restrict__ bc, int ldbc, int b_off, int c_off,
                      const float* __restrict__ Dv, const float* __restrict__ z, int ldz, float* __restrict__ state,
                      const int* __restrict__ slots, const int* __restrict__ cu_seqlens, const int* __restrict__ kv_lens,
                      TO* __restrict__ out, int inner, int N, ScanPieces pieces) {
    constexpr int CH = 128 / L, NPAD = L * NPT, W = 3 * CH + 2 * NPAD, PER_TILE = TT * W;
    constexpr int KX = (TT * CH + 127) / 128, KB = (TT * 2 * NPAD + 127) / 128;      // staged values a thread
    extern __shared__ __align__(16) float sm[];      // [2][TT][W]: x, dt, silu(z) per channel; B (padded), C (padded)
    ik_pdl_wait();
    IK_AFTER_WAIT(u);
    IK_AFTER_WAIT(dt_raw);
    IK_AFTER_WAIT(bc);
    IK_AFTER_WAIT(z);
    IK_AFTER_WAIT(slots);
    IK_AFTER_WAIT(cu_seqlens);
    IK_AFTER_WAIT(kv_lens);
    ik_pdl_launch_dependents();
    int b = blockIdx.y;
    if (MODE != 0) {                                         // the sequence of this flat piece: the last whose first piece is not behind it
        int low = 0, high = pieces.n_seqs - 1;
        while (low < high) {
            const int mid = (low + high + 1) >> 1;
            if (scan_piece_base(cu_seqlens, mid, pieces.piece) <= (int)blockIdx.y) low = mid;
            else high = mid - 1;
        }
        b = low;
    }
    const int l = threadIdx.x & (L - 1), ch = threadIdx.x / L;
    const int c0 = blockIdx.x * CH, c = c0 + ch;
    const bool live = c < inner;
    const int cc = live ? c : inner - 1;                     // idle lanes follow along (the shuffles need them)
    const int seq_lo = cu_seqlens[b], seq_hi = cu_seqlens[b + 1], end = kv_lens[b], start = end - (seq_hi - seq_lo);
    const int lo = MODE == 0 ? seq_lo : seq_lo + ((int)blockIdx.y - scan_piece_base(cu_seqlens, b, pieces.piece)) * pieces.piece;
    const int hi = MODE == 0 ? seq_hi : min(seq_hi, lo + pieces.piece);
    if (hi <= lo || (MODE == 1 && hi == seq_hi)) return;
    float* const carried = MODE == 0 ? nullptr : pieces.states + ((size_t)blockIdx.y * inner + cc) * N;
    float* st_in = state + ((size_t)slots[b] * 2 + ((start - 1) & 1)) * inner * N + (size_t)cc * N;
    float* st_out = state + ((size_t)slots[b] * 2 + ((end - 1) & 1)) * inner * N + (size_t)cc * N;
    float S[NPT], a[NPT];
    #pragma unroll
    for (int r = 0; r < NPT; r++) {
        const int n = l * NPT + r;
        a[r] = n < N ? A[(size_t)cc * N + n] : 0.f;
        if (MODE == 0) S[r] = (n < N && start > 0) ? st_in[n] : 0.f;
        else S[r] = MODE == 2 && n < N ? carried[n] : 0.f;
    }
    float dt_sum = 0.f;
    const float dskip = Dv ? Dv[cc] : 0.f;
    typename IkRaw<TU>::type rx[KX];
    float rd[KX], rz[KX], rb[KB], bias_k[KX];
    #pragma unroll
    for (int k = 0; k < KX; k++) {
        const int col = c0 + ((threadIdx.x + k * 128) % CH);
        bias_k[k] = (dt_bias && col < inner) ? dt_bias[col] : 0.f;
    }
    auto fetch = [&](int t0) {
        #pragma unroll
        for (int k = 0; k < KX; k++) {
            const int e = threadIdx.x + k * 128, tt = e / CH, col = c0 + e % CH;
            const int t = min(t0 + tt, hi - 1);
            rx[k] = 0;
            rd[k] = rz[k] = 0.f;
            if (tt < TT && col < inner) {
                rx[k] = ik_ld_now(u + (size_t)t * inner + col);
                rd[k] = ik_ld_now(dt_raw + (size_t)t * inner + col);
                if (MODE != 1 && z) rz[k] = ik_ld_now(z + (size_t)t * ldz + col);
            }
        }
        #pragma unroll
        for (int k = 0; k < KB; k++) {
            const int e = threadIdx.x + k * 128, tt = e / (2 * NPAD), n2 = e % (2 * NPAD), n = n2 % NPAD;
            const int t = min(t0 + tt, hi - 1);
            rb[k] = 0.f;
            if (tt < TT && n < N && (MODE != 1 || n2 < NPAD)) rb[k] = ik_ld_now(bc + (size_t)t * ldbc + (n2 < NPAD ? b_off : c_off) + n);
        }
    };
    auto store = [&](int buf) {
        float* tile = sm + buf * PER_TILE;
        #pragma unroll
        for (int k = 0; k < KX; k++) {
            const int e = threadIdx.x + k * 128, tt = e / CH, w = e % CH;
            if (tt < TT) {
                tile[tt * W + w] = ik_raw_float(rx[k]);
                tile[tt * W + CH + w] = ik_softplus_as<FAST>(rd[k] + bias_k[k]);
                if (MODE != 1) tile[tt * W + 2 * CH + w] = ik_silu_as<FAST>(rz[k]);
            }
        }
        #pragma unroll
        for (int k = 0; k < KB; k++) {
            const int e = threadIdx.x + k * 128, tt = e / (2 * NPAD), n2 = e % (2 * NPAD);
            if (tt < TT) tile[tt * W + 3 * CH + n2] = rb[k];
        }
    };
    fetch(lo);
    store(0);
    __syncthreads();
    int buf = 0;
    for (int t0 = lo; t0 < hi; t0 += TT, buf ^= 1) {
        if (t0 + TT < hi) fetch(t0 + TT);
        const int n_here = min(TT, hi - t0);
        const float* tile = sm + buf * PER_TILE;
        // the tile's tokens in order; a token's sum over this lane's states stays in a register, the lanes' sums are added
        // for the whole tile afterwards (the shuffles are off the token-by-token chain)
        float acc[TT];
        #pragma unroll
        for (int tt = 0; tt < TT; tt++) {
            const float* row = tile + tt * W;
            const float dt = row[CH + ch], x = row[ch];
            float bv[NPT], cv[NPT];
            if (NPT % 4 == 0) {
                #pragma unroll
                for (int r = 0; r < NPT; r += 4) {
                    const float4 b4 = *reinterpret_cast<const float4*>(row + 3 * CH + l * NPT + r);
                    const float4 c4 = *reinterpret_cast<const float4*>(row + 3 * CH + NPAD + l * NPT + r);
                    bv[r] = b4.x; bv[r + 1] = b4.y; bv[r + 2] = b4.z; bv[r + 3] = b4.w;
                    cv[r] = c4.x; cv[r + 1] = c4.y; cv[r + 2] = c4.z; cv[r + 3] = c4.w;
                }
            } else {
                #pragma unroll
                for (int r = 0; r < NPT; r++) { bv[r] = row[3 * CH + l * NPT + r]; cv[r] = row[3 * CH + NPAD + l * NPT + r]; }
            }
            float a0 = 0.f, a1 = 0.f;
            if (tt < n_here) {
                #pragma unroll
                for (int r = 0; r < NPT; r++) {
                    S[r] = ik_scan_step<FAST>(S[r], dt, x, a[r], bv[r]);
                    if (MODE == 1) continue;
                    if (r & 1) a1 = fmaf(S[r], cv[r], a1);
                    else a0 = fmaf(S[r], cv[r], a0);
                }
                if (MODE == 1) dt_sum += dt;
            }
            acc[tt] = a0 + a1;
        }
        // Sums over a channel's lanes, L tokens at a time: each exchange halves what a lane still holds, so that lane i ends with
        // token i's sum (the same additions as a butterfly per token, a quarter of the shuffles) and finishes that token.
        constexpr int GRP = TT % L == 0 ? L : 1;
        #pragma unroll
        for (int t4 = 0; MODE != 1 && t4 < TT; t4 += GRP) {
            float v[GRP];
            #pragma unroll
            for (int i = 0; i < GRP; i++) v[i] = acc[t4 + i];
            if (GRP == L) {
                #pragma unroll
                for (int o = L >> 1; o > 0; o >>= 1) {
                    const bool upper = l & o;
                    #pragma unroll
                    for (int i = 0; i < o; i++) {
                        const float theirs = __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[(i + o) % GRP], o);
                        v[i] = (upper ? v[(i + o) % GRP] : v[i]) + theirs;
                    }
                }
            } else {
                #pragma unroll
                for (int o = L >> 1; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
            }
            const int tt = GRP == L ? t4 + l : t4;
            if ((GRP == L || l == 0) && live && tt < n_here) {
                const float* row = tile + tt * W;
                float y = fmaf(dskip, row[ch], v[0]);
                if (z) y *= row[2 * CH + ch];
                ik_st(out, (size_t)(t0 + tt) * inner + c, y);
            }
        }
        if (t0 + TT < hi) store(buf ^ 1);
        __syncthreads();
    }
    if (live && (MODE != 2 || hi == seq_hi)) {
        #pragma unroll
        for (int r = 0; r < NPT; r++) {
            const int n = l * NPT + r;
            if (n < N) (MODE == 1 ? carried : st_out)[n] = S[r];
        }
        if (MODE == 1 && l == 0) pieces.sums[(size_t)blockIdx.y * inner + c] = dt_sum;
    }
}

// Whole sequences of the 16-bit path with up to 64 states, the work shared between the warps of a block.  Two teams of four warps take turns to bring
// tiles of TT tokens through registers into one of four places in shared memory (step sizes, their products with the inputs, gates, B, C) and to write the
// results of the tile before; the four last warps do nothing but the recurrence, a thread four states of a channel, L lanes a channel, CH channels a
// block, two states per instruction where the hardware has one (mul and fma of f32x2).  So neither waits for the other's latency: a token
// takes 40 ns with a block to an SM, and with more the reads from shared memory (10 to 14 cycles a warp and token), the exponentials (four a
// cycle and scheduler) and the issue slots bind about evenly (counters, 1,000 + 640 tokens, 4,096 channels of 16 states: 53, 61 and 54 %).  Tokens that are not there have a step size and an
// input of 0: a factor of 1 and nothing added.
// Measured on B200, 4,096 channels of 16 states (us, the kernel above / this): one prompt of 200 25 / 10, of 3,000 341 / 125, 3,000 + 1,910 399 / 193,
// eight of 2,000 790 / 437.  One team alone took 231 for 3,000 + 1,910 (a tile's softplus, gates and stores are 225 instructions of one
// warp in sequence); two states a thread and twice the warps 220; with the sums of four tokens stored before the next four's reads 221.
template <int L, int CH, int TT>
struct StreamTile {
    static constexpr int NPAD = 4 * L, QC = CH / 4, WORKERS = CH * L;
    // A row of pairs (step size, its product with x; x, gate) is a token's channels: channel 4 q + i in place i QC + q (of 32, q ^ 4 for
    // i >= 2), rows 2 QC floats further apart than they are long, and the rows of sums likewise: four channels a thread on one side, a few
    // neighbouring ones a warp on the other, neither meets a bank twice.
    static constexpr int ROW = 2 * CH + 2 * QC, YLD = CH == 32 ? CH + 8 : CH + 4;
    static constexpr int BC = TT * ROW, XG = BC + 2 * TT * NPAD, Y = XG + TT * ROW, FLOATS = Y + TT * YLD;         // places of B and C, of x and gate, of the sums
    static __device__ __forceinline__ int place(int tt, int q, int i) { return tt * ROW + 2 * (i * QC + (CH == 32 ? q ^ (4 * (i >> 1)) : q)); }
};
__device__ __forceinline__ uint64_t ik_pack2(float lo, float hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ float2 ik_unpack2(uint64_t v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ uint64_t ik_mul2(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t ik_fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ uint64_t ik_exp2_2(uint64_t v) {
    float2 x = ik_unpack2(v);
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(x.x));
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(x.y));
    return ik_pack2(x.x, x.y);
}

template <typename TO, int L, int CH, int TT, bool VEC>
__global__ void __launch_bounds__(256 + CH * L, VEC ? 2 : 1)
selective_scan_stream_kernel(const __nv_bfloat16* __restrict__ u, const float* __restrict__ dt_raw, const float* __restrict__ dt_bias,
                             const float* __restrict__ A, const float* __restrict__ bc, int ldbc, int b_off, int c_off,
                             const float* __restrict__ Dv, const float* __restrict__ z, int ldz, float* __restrict__ state,
                             const int* __restrict__ slots, const int* __restrict__ cu_seqlens, const int* __restrict__ kv_lens,
                             TO* __restrict__ out, int inner, int N) {
    typedef StreamTile<L, CH, TT> Tile;
    constexpr int NPAD = Tile::NPAD, YLD = Tile::YLD, ALL = 128 + Tile::WORKERS;
    extern __shared__ __align__(16) float sm[];              // [4][FLOATS]
    ik_pdl_wait();
    IK_AFTER_WAIT(u);
    IK_AFTER_WAIT(dt_raw);
    IK_AFTER_WAIT(bc);
    IK_AFTER_WAIT(z);
    IK_AFTER_WAIT(slots);
    IK_AFTER_WAIT(cu_seqlens);
    IK_AFTER_WAIT(kv_lens);
    ik_pdl_launch_dependents();
    const int b = blockIdx.y, c0 = blockIdx.x * CH;
    const int lo = cu_seqlens[b], hi = cu_seqlens[b + 1], end = kv_lens[b], start = end - (hi - lo);
    if (hi <= lo) return;
    const int n_tiles = (hi - lo + TT - 1) / TT;
    // barriers 1 to 4: a place is filled; 5 to 8: its sums are there (one side arrives, the other waits)
    if (threadIdx.x < 256) {
        const int tid = threadIdx.x & 127, team = threadIdx.x >> 7;
        constexpr int QC = Tile::QC, Q = TT * QC;            // four neighbouring channels of a token: places in a tile
        constexpr int QB = TT * 2 * NPAD / 4, KB = QB / 128; // four neighbouring values of B or C
        static_assert(Q <= 128 && QB % 128 == 0 && TT % L == 0, "a tile's values and the threads that bring them");
        const int tt = tid / QC, w = 4 * (tid % QC), col = c0 + w;
        const bool mine = tid < Q;
        float bias[4], skip[4];
        #pragma unroll
        for (int i = 0; i < 4; i++) {
            const int cc = min(col + i, inner - 1);
            bias[i] = dt_bias ? dt_bias[cc] : 0.f;
            skip[i] = Dv ? Dv[cc] : 0.f;
        }
        struct Values { uint2 u; float4 d, z, b[KB]; };      // of a tile, on their way
        // VEC: four values are four neighbours in memory.  No branch stands between these loads and their use two tiles later (a value that
        // two branches may have set is moved where they meet, and the move waits for the load); what is not there is replaced where it is stored.
        auto fetch = [&](Values& r, int t0) {
            const int t = min(t0 + tt, hi - 1);
            if (VEC) {
                const int at = min(col, inner - 4);
                asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(r.u.x), "=r"(r.u.y) : "l"(u + (size_t)t * inner + at));
                asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.d.x), "=f"(r.d.y), "=f"(r.d.z), "=f"(r.d.w) : "l"(dt_raw + (size_t)t * inner + at));
                asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.z.x), "=f"(r.z.y), "=f"(r.z.z), "=f"(r.z.w) : "l"(z + (size_t)t * ldz + at));
            } else {
                unsigned v[4];
                #pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int at = min(col + i, inner - 1);
                    v[i] = ik_ld_now(u + (size_t)t * inner + at);
                    (&r.d.x)[i] = ik_ld_now(dt_raw + (size_t)t * inner + at);
                    (&r.z.x)[i] = z ? ik_ld_now(z + (size_t)t * ldz + at) : 0.f;
                }
                r.u = make_uint2(v[0] | v[1] << 16, v[2] | v[3] << 16);
            }
            #pragma unroll
            for (int k = 0; k < KB; k++) {
                const int e = tid + k * 128, n2 = 4 * (e % (NPAD / 2)), n = n2 % NPAD;
                const float* p = bc + (size_t)min(t0 + e / (NPAD / 2), hi - 1) * ldbc + (n2 < NPAD ? b_off : c_off);
                if (VEC) asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.b[k].x), "=f"(r.b[k].y), "=f"(r.b[k].z), "=f"(r.b[k].w) : "l"(p + n));
                else {
                    #pragma unroll
                    for (int i = 0; i < 4; i++) (&r.b[k].x)[i] = ik_ld_now(p + min(n + i, N - 1));
                }
            }
        };
        auto finish = [&](int j) {                           // tile j's results
            const float* tile = sm + (j & 3) * Tile::FLOATS;
            asm volatile("bar.sync %0, %1;" :: "r"(5 + (j & 3)), "n"(ALL) : "memory");
            const int t = lo + j * TT + tt;
            if (!mine || t >= hi) return;
            float y[4];
            const float4 sum = *reinterpret_cast<const float4*>(tile + Tile::Y + tt * YLD + w);
            #pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 xg = *reinterpret_cast<const float2*>(tile + Tile::XG + Tile::place(tt, tid % QC, i));
                y[i] = fmaf(skip[i], xg.x, (&sum.x)[i]);
                if (z) y[i] *= xg.y;
            }
            TO* o = out + (size_t)t * inner + col;
            if (VEC) {
                if (col < inner) ik_st4(o, 0, make_float4(y[0], y[1], y[2], y[3]));
            } else {
                #pragma unroll
                for (int i = 0; i < 4; i++)
                    if (col + i < inner) ik_st(o, i, y[i]);
            }
        };
        Values r;
        fetch(r, lo + team * TT);
        for (int j = team; j < n_tiles; j += 2) {
            float* tile = sm + (j & 3) * Tile::FLOATS;       // (free: the results of tile j - 4 have been read, by this team)
            if (mine) {
                const bool there = lo + j * TT + tt < hi;
                if (!there) r.u = make_uint2(0u, 0u);
                #pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float x = __uint_as_float(((i & 1) ? (i < 2 ? r.u.x : r.u.y) & 0xffff0000u : (i < 2 ? r.u.x : r.u.y) << 16));
                    const float dt = there ? ik_softplus_as<true>((&r.d.x)[i] + bias[i]) : 0.f;
                    *reinterpret_cast<float2*>(tile + Tile::place(tt, tid % QC, i)) = make_float2(dt, dt * x);
                    *reinterpret_cast<float2*>(tile + Tile::XG + Tile::place(tt, tid % QC, i)) = make_float2(x, ik_silu_as<true>((&r.z.x)[i]));
                }
            }
            #pragma unroll
            for (int k = 0; k < KB; k++) {
                const int e = tid + k * 128, n = 4 * (e % (NPAD / 2)) % NPAD;
                const bool there = lo + j * TT + e / (NPAD / 2) < hi;
                #pragma unroll
                for (int i = 0; i < 4; i++)
                    if (!there || (!VEC && n + i >= N)) (&r.b[k].x)[i] = 0.f;
                *reinterpret_cast<float4*>(tile + Tile::BC + 4 * e) = r.b[k];
            }
            asm volatile("bar.arrive %0, %1;" :: "r"(1 + (j & 3)), "n"(ALL) : "memory");
            fetch(r, lo + (j + 2) * TT);
            if (j >= 2) finish(j - 2);
        }
        if (n_tiles > team) finish(n_tiles - 1 - ((n_tiles - 1 - team) & 1));
    } else {
        const int tid = threadIdx.x - 256, l = tid & (L - 1), ch = tid / L, c = c0 + ch, cc = min(c, inner - 1);   // (idle lanes follow along: the shuffles need them)
        const float* st_in = state + ((size_t)slots[b] * 2 + ((start - 1) & 1)) * inner * N + (size_t)cc * N;
        float* st_out = state + ((size_t)slots[b] * 2 + ((end - 1) & 1)) * inner * N + (size_t)cc * N;
        uint64_t S[2], a[2];                                 // states 4 l .. 4 l + 3; a in powers of two
        #pragma unroll
        for (int r = 0; r < 2; r++) {
            float s[2], e[2];
            #pragma unroll
            for (int i = 0; i < 2; i++) {
                const int n = 4 * l + 2 * r + i;
                const float p = n < N ? A[(size_t)cc * N + n] * 1.44269504f : 0.f;
                e[i] = p < -3.4e38f ? -3.4e38f : p;          // (an A of minus infinity: a step size of 0 still leaves the state alone; NaN stays)
                s[i] = n < N && start > 0 ? st_in[n] : 0.f;
            }
            S[r] = ik_pack2(s[0], s[1]);
            a[r] = ik_pack2(e[0], e[1]);
        }
        for (int j = 0; j < n_tiles; j++) {
            float* tile = sm + (j & 3) * Tile::FLOATS;
            asm volatile("bar.sync %0, %1;" :: "r"(1 + (j & 3)), "n"(ALL) : "memory");
            // all of the tile's sums before the first is stored: a store in between would hold up the reads behind it
            float v[TT];
            #pragma unroll
            for (int tt = 0; tt < TT; tt++) {
                const float2 d = *reinterpret_cast<const float2*>(tile + Tile::place(tt, ch >> 2, ch & 3));           // step size, its product with x
                const float* row = tile + Tile::BC + tt * 2 * NPAD + 4 * l;
                const ulonglong2 B = *reinterpret_cast<const ulonglong2*>(row), Cv = *reinterpret_cast<const ulonglong2*>(row + NPAD);
                const uint64_t dd = ik_pack2(d.x, d.x), dx = ik_pack2(d.y, d.y);
                S[0] = ik_fma2(ik_exp2_2(ik_mul2(dd, a[0])), S[0], ik_mul2(dx, B.x));
                S[1] = ik_fma2(ik_exp2_2(ik_mul2(dd, a[1])), S[1], ik_mul2(dx, B.y));
                const float2 sum = ik_unpack2(ik_fma2(S[1], Cv.y, ik_mul2(S[0], Cv.x)));
                v[tt] = sum.x + sum.y;
            }
            // the lanes' sums, L tokens at a time: lane i ends with token i's (as above)
            #pragma unroll
            for (int o = L >> 1; o > 0; o >>= 1) {
                const bool upper = l & o;
                #pragma unroll
                for (int t4 = 0; t4 < TT; t4 += L)
                    #pragma unroll
                    for (int i = 0; i < o; i++) {
                        const float theirs = __shfl_xor_sync(0xffffffffu, upper ? v[t4 + i] : v[t4 + i + o], o);
                        v[t4 + i] = (upper ? v[t4 + i + o] : v[t4 + i]) + theirs;
                    }
            }
            #pragma unroll
            for (int t4 = 0; t4 < TT; t4 += L) tile[Tile::Y + (t4 + l) * YLD + ch] = v[t4];
            asm volatile("bar.arrive %0, %1;" :: "r"(5 + (j & 3)), "n"(ALL) : "memory");
        }
        if (c < inner) {
            #pragma unroll
            for (int r = 0; r < 2; r++) {
                const float2 s = ik_unpack2(S[r]);
                const int n = 4 * l + 2 * r;
                if (n < N) st_out[n] = s.x;
                if (n + 1 < N) st_out[n + 1] = s.y;
            }
        }
    }
}

// The states with which a sequence's pieces begin, one thread per channel and state.
__global__ void __launch_bounds__(256)
scan_carry_kernel(const float* __restrict__ A, const float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ cu_seqlens,
                  const int* __restrict__ kv_lens, int inner, int N, ScanPieces pieces) {
    ik_pdl_wait();
    ik_pdl_launch_dependents();
    const int b = blockIdx.y, i = blockIdx.x * 256 + threadIdx.x, all = inner * N;
    if (i >= all) return;
    const int n_new = cu_seqlens[b + 1] - cu_seqlens[b], start = kv_lens[b] - n_new, f0 = scan_piece_base(cu_seqlens, b, pieces.piece);
    const int n = (n_new + pieces.piece - 1) / pieces.piece, c = i / N;
    const float a = A[i];
    float S = start > 0 && n > 0 ? state[((size_t)slots[b] * 2 + ((start - 1) & 1)) * all + i] : 0.f;
    float* mine = pieces.states + (size_t)f0 * all + i;
    const float* sums = pieces.sums + (size_t)f0 * inner + c;
    for (int j0 = 0; j0 < n; j0 += 8) {                      // eight pieces' loads in flight together
        float own[8], sum[8];
        #pragma unroll
        for (int j = 0; j < 8; j++) {
            const bool has = j0 + j + 1 < n;                 // the last piece leaves nothing
            own[j] = has ? mine[(size_t)(j0 + j) * all] : 0.f;
            sum[j] = has ? sums[(size_t)(j0 + j) * inner] : 0.f;
        }
        #pragma unroll
        for (int j = 0; j < 8; j++) {
            if (j0 + j < n) mine[(size_t)(j0 + j) * all] = S;
            S = fmaf(__expf(a * sum[j]), S, own[j]);
        }
    }
}

// One token per sequence (a decode step): no tiles; every thread reads its own inputs and its NPT states, advances them and
// writes them to the other parity's copy.  The arithmetic and its order are those of the kernel above, so a token gives
// the same float32 bits whichever kernel runs it.
template <typename TU, typename TO, bool FAST, int NPT, int L>
__global__ void __launch_bounds__(128)
selective_scan_decode_kernel(const TU* __restrict__ u, const float* __restrict__ dt_raw, const float* __restrict__ dt_bias,
                             const float* __restrict__ A, const float* __restrict__ bc, int ldbc, int b_off, int c_off,
                             const float* __restrict__ Dv, const float* __restrict__ z, int ldz, float* __restrict__ state,
                             const int* __restrict__ slots, const int* __restrict__ cu_seqlens, const int* __restrict__ kv_lens,
                             TO* __restrict__ out, int inner, int N) {
    constexpr int CH = 128 / L;
    ik_pdl_wait();
    IK_AFTER_WAIT(u);
    IK_AFTER_WAIT(dt_raw);
    IK_AFTER_WAIT(bc);
    IK_AFTER_WAIT(z);
    IK_AFTER_WAIT(slots);
    IK_AFTER_WAIT(cu_seqlens);
    IK_AFTER_WAIT(kv_lens);
    ik_pdl_launch_dependents();
    const int b = blockIdx.y, l = threadIdx.x & (L - 1), c = blockIdx.x * CH + threadIdx.x / L;
    const bool live = c < inner;
    const int cc = live ? c : inner - 1;
    const int t = cu_seqlens[b], end = kv_lens[b], start = end - 1;
    const float* st_in = state + ((size_t)slots[b] * 2 + ((start - 1) & 1)) * inner * N + (size_t)cc * N;
    float* st_out = state + ((size_t)slots[b] * 2 + ((end - 1) & 1)) * inner * N + (size_t)cc * N;
    const float x = ik_ld(u, (size_t)t * inner + cc);
    const float dt = ik_softplus_as<FAST>(dt_raw[(size_t)t * inner + cc] + (dt_bias ? dt_bias[cc] : 0.f));
    const float* row = bc + (size_t)t * ldbc;
    float S[NPT], a0 = 0.f, a1 = 0.f;
    #pragma unroll
    for (int r = 0; r < NPT; r++) {
        const int n = l * NPT + r;
        if (n < N) {
            const float ar = A[(size_t)cc * N + n];
            S[r] = start > 0 ? st_in[n] : 0.f;
            S[r] = ik_scan_step<FAST>(S[r], dt, x, ar, row[b_off + n]);
            if (r & 1) a1 = fmaf(S[r], row[c_off + n], a1);
            else a0 = fmaf(S[r], row[c_off + n], a0);
            if (live) st_out[n] = S[r];
        }
    }
    float v = a0 + a1;
    #pragma unroll
    for (int o = L >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (l == 0 && live) {
        float y = fmaf(Dv ? Dv[cc] : 0.f, x, v);
        if (z) y *= ik_silu_as<FAST>(z[(size_t)t * ldz + cc]);
        ik_st(out, (size_t)t * inner + c, y);
    }
}

// Tokens of a piece, 0 = whole sequences: pieces pay where the longest sequence is several of them.  As long as about
// twelve blocks an SM come together (each piece costs scratch), of 64 to 512 tokens.  A grid's second dimension ends at 65,535.
static int scan_piece_tokens(int T, int B, int max_new, int inner, int N) {
    if (N > 64 || max_new < 192) return 0;
    int piece = 512;
    const long long across = (inner + 31) / 32;
    while (piece > 64 && across * (T / piece) < 12LL * ik_sm_count()) piece /= 2;
    return max_new >= 3 * piece && T / piece + B <= 65535 ? piece : 0;
}

// Whether whole sequences of the 16-bit path run with the work shared between a block's warps.  Its blocks are large: where most sequences bring a few
// tokens, starting them costs more than the longer sequences gain.  Microseconds, fitted on B200 for 1 to 64 sequences of 1 to 3,000 tokens,
// 1,024 to 8,192 channels, 16 to 64 states; blocks are those of a sequence per SM (the other kernel / this): 4,096 channels of 16 states, 64 sequences
// of 2 tokens 33 / 59, of 20 75 / 90, of 100 275 / 217, one of 200 beside 63 of 1 44 / 64, one of 1,000 179 / 83.
static bool scan_streams(int T, int B, int max_new, int inner, int N) {
    if (N > 64) return false;
    const double longest = max_new > 0 ? max_new : T / (double)B;
    const int ch = N <= 16 ? 32 : N <= 32 ? 16 : 8;
    const double blocks = (inner + ch - 1) / ch / (double)ik_sm_count();
    const double chain = 0.113 * longest, all = 0.48 * B * blocks + (N <= 32 ? 0.042 : 0.038) * T * blocks;
    const double other = fmax(chain, all) + 0.5 * fmin(chain, all);
    const double here = fmax(0.043 * longest, 1.07 * B * blocks + (N <= 32 ? 0.031 : 0.034) * T * blocks);
    return B * blocks < 2.0 || here <= other;                    // (two blocks an SM start together)
}

template <typename TU, typename TO, bool FAST>
static int launch_scan(const void* u, const float* dt_raw, const float* dt_bias, const float* A, const float* bc, int ldbc, int b_off,
                       int c_off, const float* Dv, const float* z, int ldz, float* state, const int* slots, const int* cu_seqlens,
                       const int* kv_lens, void* out, int T, int B, int inner, int N, int one_token_each, int max_new, float* scratch,
                       cudaStream_t stream) {
    // four states a thread (eight from 65 states on), as many lanes a channel as that takes, tiles as long as a thread's
    // staging registers allow
#define IK_SCAN_AT(NPT, L, TT, MODE, ROWS)                                                                                      \
    IK_RETURN_IF_ERROR(ik_launch(selective_scan_kernel<TU, TO, FAST, NPT, L, TT, MODE>, dim3((inner + 128 / (L) - 1) / (128 / (L)), ROWS), 128, \
                                 (size_t)2 * (TT) * (3 * (128 / (L)) + 2 * (L) * (NPT)) * sizeof(float), stream,                \
                                 (const TU*)u, dt_raw, dt_bias, A, bc, ldbc, b_off, c_off, Dv, z, ldz, state, slots, cu_seqlens,  \
                                 kv_lens, (TO*)out, inner, N, pieces))
#define IK_SCAN_DECODE(NPT, L)                                                                                                  \
    IK_RETURN_IF_ERROR(ik_launch(selective_scan_decode_kernel<TU, TO, FAST, NPT, L>, dim3((inner + 128 / (L) - 1) / (128 / (L)), B), 128, 0, stream, (const TU*)u, dt_raw,   \
                                 dt_bias, A, bc, ldbc, b_off, c_off, Dv, z, ldz, state, slots, cu_seqlens, kv_lens, (TO*)out, inner, N))
#define IK_SCAN(NPT, L, TT)                                                                                                     \
    do {                                                                                                                        \
        if (one_token_each) IK_SCAN_DECODE(NPT, L);                                                                             \
        else IK_SCAN_AT(NPT, L, TT, 0, B);                                                                                      \
    } while (0)
#define IK_SCAN_PIECES(NPT, L, TT)                                                                                              \
    do {                                                                                                                        \
        const int rows = T / pieces.piece + B;                                                                                  \
        IK_SCAN_AT(NPT, L, TT, 1, rows);                                                                                        \
        IK_RETURN_IF_ERROR(ik_launch(scan_carry_kernel, dim3((inner * N + 255) / 256, B), 256, 0, stream, A, (const float*)state, slots, \
                                     cu_seqlens, kv_lens, inner, N, pieces));                                                   \
        IK_SCAN_AT(NPT, L, TT, 2, rows);                                                                                        \
    } while (0)
    ScanPieces pieces = {0, B, nullptr, nullptr};
    if constexpr (FAST) {
        const int piece = one_token_each || !scratch ? 0 : scan_piece_tokens(T, B, max_new, inner, N);
        if (piece > 0) {
            pieces.piece = piece;
            pieces.states = scratch;
            pieces.sums = scratch + (size_t)(T / piece + B) * inner * N;
            if (N <= 16) IK_SCAN_PIECES(4, 4, 16);
            else if (N <= 32) IK_SCAN_PIECES(4, 8, 16);
            else IK_SCAN_PIECES(4, 16, 16);
            IK_LAUNCH_STATUS();
        }
    }
    if constexpr (FAST) {
        if (!one_token_each && scan_streams(T, B, max_new, inner, N)) {
            const bool vec = inner % 4 == 0 && z && ldz % 4 == 0 && ldbc % 4 == 0 && b_off % 4 == 0 && c_off % 4 == 0 && (N == 16 || N == 32 || N == 64) &&
                             (((uintptr_t)dt_raw | (uintptr_t)z | (uintptr_t)bc | (2 * (uintptr_t)u)) % 16) == 0 && ((uintptr_t)out % (4 * sizeof(TO))) == 0;
#define IK_SCAN_STREAM_AT(L, CH, VEC)                                                                                           \
    IK_RETURN_IF_ERROR(cudaFuncSetAttribute(selective_scan_stream_kernel<TO, L, CH, 16, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                                            4 * (int)sizeof(float) * StreamTile<L, CH, 16>::FLOATS));                           \
    IK_RETURN_IF_ERROR(ik_launch(selective_scan_stream_kernel<TO, L, CH, 16, VEC>, dim3((inner + (CH) - 1) / (CH), B), 256 + (CH) * (L), \
                                 4 * sizeof(float) * StreamTile<L, CH, 16>::FLOATS, stream, (const __nv_bfloat16*)u, dt_raw, dt_bias, A, bc, ldbc, b_off, \
                                 c_off, Dv, z, ldz, state, slots, cu_seqlens, kv_lens, (TO*)out, inner, N))
#define IK_SCAN_STREAM(L, CH)                                                                                                   \
    do {                                                                                                                        \
        if (vec) { IK_SCAN_STREAM_AT(L, CH, true); }                                                                            \
        else { IK_SCAN_STREAM_AT(L, CH, false); }                                                                               \
    } while (0)
            if (N <= 16) IK_SCAN_STREAM(4, 32);
            else if (N <= 32) IK_SCAN_STREAM(8, 16);
            else IK_SCAN_STREAM(16, 8);
#undef IK_SCAN_STREAM
#undef IK_SCAN_STREAM_AT
            IK_LAUNCH_STATUS();
        }
    }
    // up to 16 states, a decode step of the 16-bit path: two states a thread while four would leave the SMs with fewer than two warps a
    // scheduler.  The float32 path keeps one shape whatever the batch, so that its sums never depend on what else a step brings.
    if (FAST && one_token_each && N <= 16 && (long long)((inner + 31) / 32) * B * 4 < 8LL * ik_sm_count()) {
        IK_SCAN_DECODE(2, 8);
        IK_LAUNCH_STATUS();
    }
    if (N <= 16) IK_SCAN(4, 4, 16);
    else if (N <= 32) IK_SCAN(4, 8, 16);
    else if (N <= 64) IK_SCAN(4, 16, 16);
    else if (N <= 128) IK_SCAN(8, 16, 8);
    else if (N <= 256) IK_SCAN(8, 32, 4);
    else return IK_UNSUPPORTED;
#undef IK_SCAN
#undef IK_SCAN_DECODE
    IK_LAUNCH_STATUS();
}

// Floats of scratch that ik_selective_scan wants for these sizes (0: none): bfloat16 inputs in several pieces.
IK_EXPORT long long ik_selective_scan_scratch(int u_dtype, int T, int B, int max_new, int inner, int N, int one_token_each) {
    if (u_dtype != IK_BF16 || one_token_each || T <= 0 || B <= 0) return 0;
    const int piece = scan_piece_tokens(T, B, max_new, inner, N);
    return piece ? (long long)(T / piece + B) * inner * (N + 1) : 0;
}

// scratch: ik_selective_scan_scratch floats, or null (every sequence is then run token by token).  max_new: the longest sequence's tokens.
IK_EXPORT int ik_selective_scan(const void* u, int u_dtype, const float* dt_raw, const float* dt_bias, const float* A,
                                const float* bc, int ldbc, int b_off, int c_off, const float* Dv, const float* z, int ldz,
                                float* state, const int* slots, const int* cu_seqlens, const int* kv_lens, void* out,
                                int out_dtype, int T, int B, int inner, int N, int one_token_each, int max_new, float* scratch,
                                cudaStream_t stream) {
    if (T < 0 || B < 0 || inner <= 0 || N <= 0 || !state || b_off < 0 || c_off < 0 || ldbc < N) return IK_BAD_ARGUMENT;
    if (T == 0 || B == 0) return IK_OK;
    if (one_token_each && T != B) return IK_BAD_ARGUMENT;
#define IK_ARGS u, dt_raw, dt_bias, A, bc, ldbc, b_off, c_off, Dv, z, ldz, state, slots, cu_seqlens, kv_lens, out, T, B, inner, N, one_token_each, max_new, scratch, stream
    if (u_dtype == IK_F32 && out_dtype == IK_F32) return launch_scan<float, float, false>(IK_ARGS);
    if (u_dtype == IK_BF16 && out_dtype == IK_BF16) return launch_scan<__nv_bfloat16, __nv_bfloat16, true>(IK_ARGS);
    if (u_dtype == IK_F32 && out_dtype == IK_BF16) return launch_scan<float, __nv_bfloat16, false>(IK_ARGS);
    if (u_dtype == IK_BF16 && out_dtype == IK_F32) return launch_scan<__nv_bfloat16, float, true>(IK_ARGS);
#undef IK_ARGS
    return IK_BAD_ARGUMENT;
}

// ------------------------------------------------------------------ linear attention with a constant decay per head
// Per head h with decay a_h:  S <- a_h S + k v^T (S is dk x dv);  o = S^T q.  q, k, v are columns of the projections'
// output `p` (row stride ldp), each passed through silu when act is set (act 2: with the hardware's approximate
// exponential and reciprocal, for the 16-bit path).  A block holds 32 columns of one head's S for one sequence: thread
// (j, part) keeps rows part*R .. part*R + R - 1 of column j in registers, one warp per part, up to 16 of them.  The
// tokens go through shared memory in tiles (q, k and the block's 32 columns of v, activation applied when a tile is
// stored); while a tile is computed the next one is on its way into registers, every warp fetching whole token rows.
// The parts' sums of a column are added in part order, once per tile.  What is computed for a token does not depend on
// where tiles begin.  FULL: dk = parts * RMAX and RMAX is a multiple of 4: no row is guarded and q, k come from shared
// memory four at a time.
constexpr int LA_ROWS = 2;         // token rows a warp stages per tile, at most

// LA_PER_ROW: 32-wide pieces of a staged row (2 dk + 32 values): 9 up to dk = 128, 17 up to 256
template <int RMAX, bool FULL, int LA_PER_ROW>
__global__ void __launch_bounds__(512)
decay_attention_kernel(const float* __restrict__ p, int ldp, int q_off, int k_off, int v_off, const float* __restrict__ decay,
                       float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ cu_seqlens,
                       const int* __restrict__ kv_lens, float* __restrict__ out, int H, int dk, int dv, int R, int act, int TT) {
    extern __shared__ __align__(16) float sm[];          // [2][TT][2 dk + 32]: q, k, v;  [2][TT][parts][32] partial sums
    ik_pdl_wait();
    IK_AFTER_WAIT(p);
    IK_AFTER_WAIT(slots);
    IK_AFTER_WAIT(cu_seqlens);
    IK_AFTER_WAIT(kv_lens);
    ik_pdl_launch_dependents();
    const int b = blockIdx.x, h = blockIdx.y, j = threadIdx.x, part = threadIdx.y, parts = blockDim.y;
    const int col0 = blockIdx.z * 32, col = col0 + j;
    const bool live = col < dv;
    const int ccol = live ? col : dv - 1;
    const int tid = part * 32 + j, nthreads = parts * 32, W = 2 * dk + 32, per_tile = TT * W;
    float* partial = sm + 2 * per_tile;
    const int lo = cu_seqlens[b], hi = cu_seqlens[b + 1], end = kv_lens[b], start = end - (hi - lo);
    if (hi <= lo) return;
    const float a = decay[h];
    const size_t per = (size_t)H * dk * dv;
    const float* st_in = state + ((size_t)slots[b] * 2 + ((start - 1) & 1)) * per + (size_t)h * dk * dv;
    float* st_out = state + ((size_t)slots[b] * 2 + ((end - 1) & 1)) * per + (size_t)h * dk * dv;
    float S[RMAX];
    #pragma unroll
    for (int r = 0; r < RMAX; r++) {
        const int i = part * R + r;
        S[r] = (r < R && i < dk && start > 0) ? st_in[(size_t)i * dv + ccol] : 0.f;
    }
    // staging: warp `part` fetches token rows part, part + parts, ...; lane j the columns j, j + 32, ... of a row
    float regs[LA_ROWS][LA_PER_ROW];
    auto fetch = [&](int t0) {
        #pragma unroll
        for (int rr = 0; rr < LA_ROWS; rr++) {
            const int tt = part + parts * rr;
            const float* row = p + (size_t)min(t0 + tt, hi - 1) * ldp;
            #pragma unroll
            for (int kk = 0; kk < LA_PER_ROW; kk++) {
                const int w = j + 32 * kk;
                regs[rr][kk] = 0.f;
                if (tt >= TT || w >= W) continue;
                if (w < dk) regs[rr][kk] = row[q_off + h * dk + w];
                else if (w < 2 * dk) regs[rr][kk] = row[k_off + h * dk + w - dk];
                else if (col0 + w - 2 * dk < dv) regs[rr][kk] = row[v_off + h * dv + col0 + w - 2 * dk];
            }
        }
    };
    auto store = [&](int buf) {
        #pragma unroll
        for (int rr = 0; rr < LA_ROWS; rr++) {
            const int tt = part + parts * rr;
            #pragma unroll
            for (int kk = 0; kk < LA_PER_ROW; kk++) {
                const int w = j + 32 * kk;
                if (tt < TT && w < W) sm[buf * per_tile + tt * W + w] = regs[rr][kk];
            }
        }
        if (!act) return;
        // the activation on what this thread has just stored, in a loop that is not unrolled (one copy of its code)
        for (int tt = part; tt < TT; tt += parts) {
            float* row = sm + buf * per_tile + tt * W;
            #pragma unroll 1
            for (int w = j; w < W; w += 32) row[w] = act == 2 ? ik_silu_as<true>(row[w]) : ik_silu_as<false>(row[w]);
        }
    };
    fetch(lo);
    store(0);
    __syncthreads();
    int buf = 0;
    for (int t0 = lo; t0 < hi; t0 += TT, buf ^= 1) {
        if (t0 + TT < hi) fetch(t0 + TT);
        const int n_here = min(TT, hi - t0);
        for (int tt = 0; tt < n_here; tt++) {
            const float* q = sm + buf * per_tile + tt * W + part * R;
            const float* k = q + dk;
            const float v = sm[buf * per_tile + tt * W + 2 * dk + j];
            float acc0 = 0.f, acc1 = 0.f;
            if (FULL) {
                #pragma unroll
                for (int r = 0; r < RMAX; r += 4) {
                    const float4 kk = *reinterpret_cast<const float4*>(k + r), qq = *reinterpret_cast<const float4*>(q + r);
                    S[r] = fmaf(a, S[r], kk.x * v);         acc0 = fmaf(S[r], qq.x, acc0);
                    S[r + 1] = fmaf(a, S[r + 1], kk.y * v); acc1 = fmaf(S[r + 1], qq.y, acc1);
                    S[r + 2] = fmaf(a, S[r + 2], kk.z * v); acc0 = fmaf(S[r + 2], qq.z, acc0);
                    S[r + 3] = fmaf(a, S[r + 3], kk.w * v); acc1 = fmaf(S[r + 3], qq.w, acc1);
                }
            } else {
                #pragma unroll
                for (int r = 0; r < RMAX; r++) {
                    if (r < R && part * R + r < dk) {
                        S[r] = fmaf(a, S[r], k[r] * v);
                        if (r & 1) acc1 = fmaf(S[r], q[r], acc1);
                        else acc0 = fmaf(S[r], q[r], acc0);
                    }
                }
            }
            const float acc = acc0 + acc1;
            if (parts > 1) partial[((buf * TT + tt) * parts + part) * 32 + j] = acc;
            else if (live) out[(size_t)(t0 + tt) * H * dv + h * dv + col] = acc;
        }
        if (t0 + TT < hi) store(buf ^ 1);
        __syncthreads();
        if (parts > 1) {
            for (int e = tid; e < n_here * 32; e += nthreads) {
                const int tt = e >> 5, jj = e & 31;
                if (col0 + jj >= dv) continue;
                float o = 0.f;
                for (int pp = 0; pp < parts; pp++) o += partial[((buf * TT + tt) * parts + pp) * 32 + jj];
                out[(size_t)(t0 + tt) * H * dv + h * dv + col0 + jj] = o;
            }
        }
    }
    if (live) {
        #pragma unroll
        for (int r = 0; r < RMAX; r++) {
            const int i = part * R + r;
            if (r < R && i < dk) st_out[(size_t)i * dv + col] = S[r];
        }
    }
}

// One token per sequence (a decode step): no tiles and few registers, so that several blocks share an SM and the state
// streams.  q and k pass the activation once per block (shared memory), every thread advances its R rows of its column
// and writes them to the other parity's copy.  The arithmetic and its order are those of the kernel above.
template <int RMAX>
__global__ void __launch_bounds__(512)
decay_attention_decode_kernel(const float* __restrict__ p, int ldp, int q_off, int k_off, int v_off, const float* __restrict__ decay,
                              float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ cu_seqlens,
                              const int* __restrict__ kv_lens, float* __restrict__ out, int H, int dk, int dv, int R, int act) {
    extern __shared__ __align__(16) float sm[];          // [2 dk] q, k;  [parts][32] partial sums
    ik_pdl_wait();
    IK_AFTER_WAIT(p);
    IK_AFTER_WAIT(slots);
    IK_AFTER_WAIT(cu_seqlens);
    IK_AFTER_WAIT(kv_lens);
    ik_pdl_launch_dependents();
    const int b = blockIdx.x, h = blockIdx.y, j = threadIdx.x, part = threadIdx.y, parts = blockDim.y;
    const int col0 = blockIdx.z * 32, col = col0 + j;
    const bool live = col < dv;
    const int ccol = live ? col : dv - 1;
    const int tid = part * 32 + j, nthreads = parts * 32;
    float* partial = sm + 2 * dk;
    const int t = cu_seqlens[b], end = kv_lens[b], start = end - 1;
    const size_t per = (size_t)H * dk * dv;
    const float* st_in = state + ((size_t)slots[b] * 2 + ((start - 1) & 1)) * per + (size_t)h * dk * dv;
    float* st_out = state + ((size_t)slots[b] * 2 + ((end - 1) & 1)) * per + (size_t)h * dk * dv;
    float S[RMAX];
    #pragma unroll
    for (int r = 0; r < RMAX; r++) {
        const int i = part * R + r;
        S[r] = (r < R && i < dk && start > 0) ? st_in[(size_t)i * dv + ccol] : 0.f;
    }
    const float* row = p + (size_t)t * ldp;
    for (int e = tid; e < 2 * dk; e += nthreads) {
        const float x = e < dk ? row[q_off + h * dk + e] : row[k_off + h * dk + e - dk];
        sm[e] = act == 2 ? ik_silu_as<true>(x) : act ? ik_silu_as<false>(x) : x;
    }
    float v = row[v_off + h * dv + ccol];
    v = act == 2 ? ik_silu_as<true>(v) : act ? ik_silu_as<false>(v) : v;
    const float a = decay[h];
    __syncthreads();
    const float* q = sm + part * R;
    const float* k = q + dk;
    float acc0 = 0.f, acc1 = 0.f;
    #pragma unroll
    for (int r = 0; r < RMAX; r++) {
        if (r < R && part * R + r < dk) {
            S[r] = fmaf(a, S[r], k[r] * v);
            if (r & 1) acc1 = fmaf(S[r], q[r], acc1);
            else acc0 = fmaf(S[r], q[r], acc0);
            if (live) st_out[(size_t)(part * R + r) * dv + col] = S[r];
        }
    }
    const float acc = acc0 + acc1;
    if (parts == 1) {
        if (live) out[(size_t)t * H * dv + h * dv + col] = acc;
        return;
    }
    partial[part * 32 + j] = acc;
    __syncthreads();
    if (part == 0 && live) {
        float o = 0.f;
        for (int pp = 0; pp < parts; pp++) o += partial[pp * 32 + j];
        out[(size_t)t * H * dv + h * dv + col] = o;
    }
}

IK_EXPORT int ik_decay_attention(const float* p, int ldp, int q_off, int k_off, int v_off, const float* decay, float* state,
                                 const int* slots, const int* cu_seqlens, const int* kv_lens, float* out, int T, int B, int H,
                                 int dk, int dv, int act, int one_token_each, cudaStream_t stream) {
    if (T < 0 || B < 0 || H <= 0 || dk <= 0 || dv <= 0 || !state || !decay) return IK_BAD_ARGUMENT;
    if (T == 0 || B == 0) return IK_OK;
    if (dk > 256) return IK_UNSUPPORTED;
    if (one_token_each && T != B) return IK_BAD_ARGUMENT;
    int parts = (dk + 7) / 8;                       // eight rows a thread ...
    if (parts > 16) parts = 16;                     // ... sixteen from 129 rows on
    const int R = (dk + parts - 1) / parts, W = 2 * dk + 32;
    int TT = LA_ROWS * parts;
    if (TT > 16) TT = 16;
    const bool full = dk == parts * R && (R == 8 || R == 16) && ldp % 4 == 0;
    const dim3 grid(B, H, (dv + 31) / 32), block(32, parts);
    if (one_token_each) {
        const size_t smem1 = (size_t)(2 * dk + parts * 32) * sizeof(float);
        if (R <= 8)
            IK_RETURN_IF_ERROR(ik_launch(decay_attention_decode_kernel<8>, grid, block, smem1, stream, p, ldp, q_off, k_off, v_off, decay, state,
                                         slots, cu_seqlens, kv_lens, out, H, dk, dv, R, act));
        else
            IK_RETURN_IF_ERROR(ik_launch(decay_attention_decode_kernel<16>, grid, block, smem1, stream, p, ldp, q_off, k_off, v_off, decay, state,
                                         slots, cu_seqlens, kv_lens, out, H, dk, dv, R, act));
        IK_LAUNCH_STATUS();
    }
    const size_t smem = (size_t)(2 * TT * W + 2 * TT * parts * 32) * sizeof(float);
    if (smem > 160 * 1024) return IK_UNSUPPORTED;
#define IK_LA(RMAX, FULL, PER_ROW)                                                                                               \
    do {                                                                                                                         \
        static bool raised = false;                                                                                              \
        if (smem > 48 * 1024 && !raised) {                                                                                       \
            IK_RETURN_IF_ERROR(cudaFuncSetAttribute(decay_attention_kernel<RMAX, FULL, PER_ROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                    160 * 1024));                                                                \
            raised = true;                                                                                                       \
        }                                                                                                                        \
        IK_RETURN_IF_ERROR(ik_launch(decay_attention_kernel<RMAX, FULL, PER_ROW>, grid, block, smem, stream, p, ldp, q_off, k_off, v_off, \
                                     decay, state, slots, cu_seqlens, kv_lens, out, H, dk, dv, R, act, TT));                      \
    } while (0)
    if (full && R == 8) IK_LA(8, true, 9);
    else if (full) IK_LA(16, true, 17);
    else if (R <= 8) IK_LA(8, false, 9);
    else IK_LA(16, false, 17);
#undef IK_LA
    IK_LAUNCH_STATUS();
}
