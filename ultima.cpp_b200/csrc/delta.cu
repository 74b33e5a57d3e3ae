// The gated delta-rule mixer: a recurrent layer whose state is, for every head, a matrix S [D, E]
// (D key channels, E value channels) in float32, plus the last inputs of a short causal convolution.
//
// For one token of one head, with unit vectors q (scaled) and k, a value v, a write strength b in
// (0, 1) and a decay a[d] in (0, 1) for every key channel:
//     S[d, :] *= a[d];   u = b * (v - S^T k);   S += k u^T;   o = S^T q
// so the read-out sees the token's own write.  Every column of S evolves on its own, which is what
// the scan kernel uses: a group of eight lanes holds one column, tokens are taken in order.
//
// Four kernels, for prompts and single tokens alike (a step's tokens of one sequence are rows
// seq_start[s] .. seq_start[s + 1] of the packed batch; state rows are slot numbers):
//   delta_prepare      short convolution + SiLU of q, k, v; unit vectors; write strength; decay
//   conv_state_update  the convolution's last inputs, carried to the next step
//   delta_scan         the recurrence
//   delta_finish       per-head RMS norm of o, weight, output gate (sigmoid or SiLU of the gate's sums)
// The decay is one number a head and key channel (its sums come in a matrix of their own, ``dpre``), or one
// number a head whose sums are a column range of the projection row (``a_off`` >= 0; the bias then has one
// entry a head).
// Everything is float32 (long prompts: two products on the tensor cores, a float32 operand as three bfloat16 parts, and sums over a few
// tokens in float64; see delta_chunks_kernel); the projections come in as float32 sums of the products (for few tokens as the
// partial sums of K slices, which the kernels add up as they read).
#include "common.cuh"
#include "tc_common.cuh"
#include <stdlib.h>
#include <type_traits>

constexpr int MAX_TAPS = 16;

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float softplusf_(float x) { return x > 20.f ? x : log1pf(expf(x)); }

struct DeltaShape {
    int H, G, D, E;          // heads, q/k heads, key size, value size
    int taps;                // convolution length (the last tap is the current token's)
    int q_off, k_off, v_off, b_off;   // columns of a projection row
    int a_off;               // >= 0: one decay a head, its sums in the H columns from here on; < 0: one a key channel, from dpre
    long long ldp;           // row stride of the projections
    int n_parts;             // the projection row is the sum of this many partial results ...
    long long part_stride;   // ... this many elements apart
};

__device__ __forceinline__ float proj_at(const float* __restrict__ p, const DeltaShape& s, long long t, int c) {
    float v = 0.f;
    for (int i = 0; i < s.n_parts; ++i) v += p[i * s.part_stride + t * s.ldp + c];
    return v;
}

// One warp a (token, unit); units of a token: G query heads, G key heads, H value heads (which also
// make the head's write strength and decay).  ``update_state`` (only when every sequence brings ONE token, so
// that a channel's state has this lane as its only reader): the convolution's state moves on here, and
// conv_state_update is not launched.
__global__ void __launch_bounds__(128)
delta_prepare_kernel(const float* __restrict__ p, DeltaShape s, const float* __restrict__ conv_w,
                     float* conv_state, int update_state, const float* __restrict__ dpre,
                     const float* __restrict__ dt_bias, const float* __restrict__ a_log,
                     const int* __restrict__ tok_seq, const int* __restrict__ seq_start,
                     const int* __restrict__ seq_slot, float* __restrict__ qn, float* __restrict__ kn,
                     float* __restrict__ vc, float* __restrict__ beta, float* __restrict__ dec,
                     int n_tokens, float unit_eps, float q_scale) {
    pdl_trigger();
    pdl_wait();
    const int units = 2 * s.G + s.H;
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= (long long)n_tokens * units) return;
    const int t = (int)(wid / units), unit = (int)(wid % units);
    const int seq = tok_seq[t];
    const int r = t - seq_start[seq];
    const int K = s.taps - 1;
    const int C = 2 * s.G * s.D + s.H * s.E;
    float* st = conv_state + (long long)seq_slot[seq] * K * C;

    auto conv_silu = [&](int c) -> float {
        float acc = 0.f;
        for (int j = K; j >= 0; --j) {                 // oldest input first
            const float w = conv_w[(long long)c * s.taps + (s.taps - 1 - j)];
            const float x = (r - j >= 0) ? proj_at(p, s, t - j, c) : st[(long long)(K + r - j) * C + c];
            acc = fmaf(w, x, acc);
            if (update_state && j < K) st[(long long)(K - 1 - j) * C + c] = x;     // r = 0: the input j back becomes j + 1 back
        }
        return acc * sigmoidf_(acc);
    };

    if (unit < 2 * s.G) {
        const bool is_q = unit < s.G;
        const int head = is_q ? unit : unit - s.G;
        const int c0 = (is_q ? s.q_off : s.k_off) + head * s.D;      // q_off = 0 and k_off = G * D: columns are channels
        float vals[8];
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int d = lane + 32 * i;
            vals[i] = d < s.D ? conv_silu(c0 + d) : 0.f;
            ss += vals[i] * vals[i];
        }
        ss = warp_sum(ss);
        const float inv = (is_q ? q_scale : 1.0f) / sqrtf(ss + unit_eps);
        float* o = (is_q ? qn : kn) + (long long)t * s.G * s.D + head * s.D;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int d = lane + 32 * i;
            if (d < s.D) o[d] = vals[i] * inv;
        }
        return;
    }
    const int h = unit - 2 * s.G;
    for (int e = lane; e < s.E; e += 32)
        vc[(long long)t * s.H * s.E + h * s.E + e] = conv_silu(s.v_off + h * s.E + e);
    if (lane == 0) beta[(long long)t * s.H + h] = sigmoidf_(proj_at(p, s, t, s.b_off + h));
    const float rate = expf(a_log[h]);
    if (s.a_off >= 0) {
        const float a = expf(-rate * softplusf_(proj_at(p, s, t, s.a_off + h) + dt_bias[h]));
        for (int d = lane; d < s.D; d += 32) dec[(long long)t * s.H * s.D + h * s.D + d] = a;
        return;
    }
    for (int d = lane; d < s.D; d += 32) {
        const long long c = (long long)t * s.H * s.D + h * s.D + d;
        dec[c] = expf(-rate * softplusf_(dpre[c] + dt_bias[h * s.D + d]));
    }
}

// The same for heads of 64 or 128 (keys and values) and up to four taps: a warp a unit and a run of up to WALK tokens, a lane
// two or four neighbouring channels.  Inputs are asked for two tokens ahead and a token's earlier inputs stay in
// registers (a warp a token and unit read every input once a tap, one number a lane); decays are units of their own, since their
// exponentials and logarithms are the longer part.  2,048 tokens, 16 heads on 4 of 128: 123 -> 38 us (85 MB).
constexpr int WALK = 8;

template <int V>
__device__ __forceinline__ void row_piece(const float* __restrict__ p, const DeltaShape& s, long long t, int c, float* x) {
    load_vec<float, V>(p + t * s.ldp + c, x);
    for (int i = 1; i < s.n_parts; ++i) {
        float y[V];
        load_vec<float, V>(p + i * s.part_stride + t * s.ldp + c, y);
#pragma unroll
        for (int v = 0; v < V; ++v) x[v] += y[v];
    }
}

// ``dst``: the unit's columns of the output at this lane, rows ``ld`` apart.  NORM: unit vectors times ``scale``.
template <int V, bool NORM>
__device__ __forceinline__ void walk_channels(const float* __restrict__ p, const DeltaShape& s, const float* __restrict__ conv_w,
                                              float* conv_state, int update_state, const int* __restrict__ tok_seq,
                                              const int* __restrict__ seq_start, const int* __restrict__ seq_slot, int t0, int n,
                                              int c, int C, float* dst, long long ld, float unit_eps, float scale) {
    const int K = s.taps - 1;
    float x[V], next[2][V], w[V][4], hist[3][V];         // hist[j]: the input j + 1 back; w[v][i]: weight of the input 3 - i back
    row_piece<V>(p, s, t0, c, next[0]);
    row_piece<V>(p, s, t0 + min(1, n - 1), c, next[1]);
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
        for (int i = 0; i < 4; ++i) w[v][i] = i >= 3 - K ? conv_w[(long long)(c + v) * s.taps + i - (3 - K)] : 0.f;
    int seq = -1;
    // (rolled up: eight copies of the sigmoid's code a channel do not fit the instruction cache)
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        const int t = t0 + i, now = tok_seq[t];
#pragma unroll
        for (int v = 0; v < V; ++v) { x[v] = next[0][v]; next[0][v] = next[1][v]; }
        row_piece<V>(p, s, t0 + min(i + 2, n - 1), c, next[1]);
        if (now != seq) {                                  // the run's first token, or another sequence's first one
            seq = now;
            const int r = t - seq_start[seq];
            const float* st = conv_state + (long long)seq_slot[seq] * K * C + c;
#pragma unroll
            for (int j = 1; j <= 3; ++j) {
                if (j > K) {
#pragma unroll
                    for (int v = 0; v < V; ++v) hist[j - 1][v] = 0.f;
                } else if (r - j >= 0) row_piece<V>(p, s, t - j, c, hist[j - 1]);
                else load_vec<float, V>(st + (long long)(K + r - j) * C, hist[j - 1]);
            }
            if (update_state) {                            // one token a sequence: the input j back becomes j + 1 back
                float* sw = conv_state + (long long)seq_slot[seq] * K * C + c;
                if (K > 0) store_vec<float, V>(sw + (long long)(K - 1) * C, x);
                if (K > 1) store_vec<float, V>(sw + (long long)(K - 2) * C, hist[0]);
                if (K > 2) store_vec<float, V>(sw + (long long)(K - 3) * C, hist[1]);
            }
        }
        float y[V], ss = 0.f;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            float acc = 0.f;
            if (K >= 3) acc = fmaf(w[v][0], hist[2][v], acc);
            if (K >= 2) acc = fmaf(w[v][1], hist[1][v], acc);
            if (K >= 1) acc = fmaf(w[v][2], hist[0][v], acc);
            acc = fmaf(w[v][3], x[v], acc);
            y[v] = acc * sigmoidf_(acc);
            ss = fmaf(y[v], y[v], ss);
            hist[2][v] = hist[1][v];
            hist[1][v] = hist[0][v];
            hist[0][v] = x[v];
        }
        if constexpr (NORM) {
            const float inv = scale / sqrtf(warp_sum(ss) + unit_eps);
#pragma unroll
            for (int v = 0; v < V; ++v) y[v] *= inv;
        }
        store_vec<float, V>(dst + (long long)t * ld, y);
    }
}

template <int VD, int VE>
__global__ void __launch_bounds__(128)
delta_prepare_rows_kernel(const float* __restrict__ p, DeltaShape s, const float* __restrict__ conv_w,
                          float* conv_state, int update_state, const float* __restrict__ dpre,
                          const float* __restrict__ dt_bias, const float* __restrict__ a_log,
                          const int* __restrict__ tok_seq, const int* __restrict__ seq_start,
                          const int* __restrict__ seq_slot, float* __restrict__ qn, float* __restrict__ kn,
                          float* __restrict__ vc, float* __restrict__ beta, float* __restrict__ dec,
                          int n_tokens, int walk, float unit_eps, float q_scale) {
    pdl_trigger();
    pdl_wait();
    constexpr int D = VD * 32, E = VE * 32;
    const int units = 2 * s.G + 2 * s.H;
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int unit = (int)(wid % units);
    const long long first = wid / units * walk;
    if (first >= n_tokens) return;
    const int t0 = (int)first, n = min(walk, n_tokens - t0);
    const int C = 2 * s.G * D + s.H * E;
    if (unit < 2 * s.G) {
        const bool is_q = unit < s.G;
        const int head = is_q ? unit : unit - s.G, o = head * D + lane * VD;
        walk_channels<VD, true>(p, s, conv_w, conv_state, update_state, tok_seq, seq_start, seq_slot, t0, n,
                                (is_q ? s.q_off : s.k_off) + o, C, (is_q ? qn : kn) + o, (long long)s.G * D, unit_eps, is_q ? q_scale : 1.0f);
    } else if (unit < 2 * s.G + s.H) {
        const int h = unit - 2 * s.G, o = h * E + lane * VE;
        if (lane < n) beta[(long long)(t0 + lane) * s.H + h] = sigmoidf_(proj_at(p, s, t0 + lane, s.b_off + h));
        walk_channels<VE, false>(p, s, conv_w, conv_state, update_state, tok_seq, seq_start, seq_slot, t0, n,
                                 s.v_off + o, C, vc + o, (long long)s.H * E, 0.f, 1.f);
    } else {
        const int h = unit - 2 * s.G - s.H, o = h * D + lane * VD;
        const float rate = expf(a_log[h]);
        if (s.a_off >= 0) {
            for (int i = 0; i < n; ++i) {
                const long long t = t0 + i;
                const float a = expf(-rate * softplusf_(proj_at(p, s, t, s.a_off + h) + dt_bias[h]));
                float y[VD];
#pragma unroll
                for (int v = 0; v < VD; ++v) y[v] = a;
                store_vec<float, VD>(dec + t * s.H * D + o, y);
            }
            return;
        }
        float bias[VD], next[VD];
        load_vec<float, VD>(dt_bias + o, bias);
        load_vec<float, VD>(dpre + (long long)t0 * s.H * D + o, next);
#pragma unroll 1
        for (int i = 0; i < n; ++i) {
            float y[VD];
#pragma unroll
            for (int v = 0; v < VD; ++v) y[v] = next[v];
            load_vec<float, VD>(dpre + (long long)(t0 + min(i + 1, n - 1)) * s.H * D + o, next);
#pragma unroll
            for (int v = 0; v < VD; ++v) y[v] = expf(-rate * softplusf_(y[v] + bias[v]));
            store_vec<float, VD>(dec + (long long)(t0 + i) * s.H * D + o, y);
        }
    }
}

// One thread a (sequence, channel): the last taps - 1 inputs of what the state held followed by the step's.
__global__ void conv_state_update_kernel(const float* __restrict__ p, DeltaShape s, float* __restrict__ conv_state,
                                         const int* __restrict__ seq_start, const int* __restrict__ seq_slot,
                                         int n_seqs, int C, int taps) {
    pdl_trigger();
    pdl_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)n_seqs * C) return;
    const int b = (int)(i / C), c = (int)(i % C);
    const int K = taps - 1;
    const int first = seq_start[b], n = seq_start[b + 1] - first;
    float* st = conv_state + (long long)seq_slot[b] * K * C;
    float tmp[MAX_TAPS];
    for (int k = 0; k < K; ++k) {
        const int rel = n - K + k;
        tmp[k] = rel >= 0 ? proj_at(p, s, first + rel, c) : st[(long long)(K + rel) * C + c];
    }
    for (int k = 0; k < K; ++k) st[(long long)k * C + c] = tmp[k];
}

// The recurrence.  A block of 128 threads takes 128 / LANES value channels of one head of one sequence;
// LANES (8, 16 or 32) lanes hold one column of S, lane p the key channels of the float4 chunks p,
// p + LANES, ...: the lanes of a column read consecutive bytes of shared memory in one instruction, and a
// dot product over the key channels ends in log2(LANES) exchanges.  Tokens come through shared memory a
// few at a time, the next few asked for (cp.async) while these are worked on.
//
// The kernel is bound by latency, not by bytes or arithmetic: a token's update depends on the one before
// it through a chain of multiply, dot product, exchanges and update, and a warp issues in order.  The
// read-out o = S^T q is off that chain: its partial sums go to shared memory and are added up once for
// the tokens of a stage, and the loop over a full stage's tokens is unrolled.

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// The same recurrence for keys of 64 or 128 and values in sixteens (every array on a 16-byte boundary), prompts and single
// tokens alike, so that a sequence has the same bits however it is cut.
//
// Bound by the chain from token to token; everything else is kept off it.  Against the kernel below: the dot product is taken of the
// state as it is with a * k (a product that waits for nothing), so the decay runs beside the chain's exchanges and not before
// them; pairs of key channels go through packed float32 instructions (half the issue slots: a scheduler has one warp here); eight
// tokens' read-outs are summed over a column's eight lanes by seven exchanges with no way through shared memory; v and the
// write strength come straight to registers a stage ahead; one barrier a stage of eight tokens instead of two.
// 2,048 tokens, 16 heads of 128 x 128: 695 -> 491 us.
__device__ __forceinline__ uint64_t pair_of(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpair(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

template <int D>
__global__ void __launch_bounds__(128)
delta_scan_pairs_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vc,
                        const float* __restrict__ beta, const float* __restrict__ dec, float* __restrict__ out,
                        float* __restrict__ S, const int* __restrict__ seq_start, const int* __restrict__ seq_slot,
                        int H, int G, int E, int below) {
    constexpr int TT = 8;                                 // tokens a stage: as many as a column has lanes
    constexpr int NC = D / 32;                            // float4 chunks a lane: chunks p, p + 8, ... of the key channels
    constexpr int BUFS = 3;
    __shared__ __align__(16) float ring[BUFS][TT][3][D];  // a token's q, k and decay
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, col = tid >> 3, p = tid & 7;
    const int h = blockIdx.y, b = blockIdx.z, g = h / (H / G);
    const int j = blockIdx.x * 16 + col;
    const int t0 = seq_start[b], t1 = seq_start[b + 1];
    if (t0 >= t1 || t1 - t0 >= below) return;             // (longer sequences: another kernel's)
    float* Sh = S + ((long long)seq_slot[b] * H + h) * D * E + j;
    uint64_t s[2 * NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int d = (c * 8 + p) * 4;
        s[2 * c] = pair_of(Sh[(long long)d * E], Sh[(long long)(d + 1) * E]);
        s[2 * c + 1] = pair_of(Sh[(long long)(d + 2) * E], Sh[(long long)(d + 3) * E]);
    }
    // this thread's 16-byte pieces of a stage: piece tid + 128 i of TT x 3 x D / 4
    constexpr int PIECES = TT * 3 * D / 4 / 128;
    auto fetch = [&](int base) {
        const int buf = ((base - t0) / TT) % BUFS;
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const int c = tid + 128 * i, tt = c / (3 * D / 4), arr = (c / (D / 4)) % 3, d = (c % (D / 4)) * 4;
            const long long t = base + tt;
            const float* src = arr == 0 ? qn + (t * G + g) * D : arr == 1 ? kn + (t * G + g) * D : dec + (t * H + h) * D;
            if (t < t1) cp_async16(&ring[buf][tt][arr][d], src + d);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const float* vsrc = vc + (long long)h * E + j;
    float bn[TT], vn[TT];                                 // the stage ahead: write strengths and values
    auto fetch_values = [&](int base) {
#pragma unroll
        for (int tt = 0; tt < TT; ++tt) {
            const long long t = min(base + tt, t1 - 1);
            bn[tt] = beta[t * H + h];
            vn[tt] = vsrc[t * H * E];
        }
    };
    fetch(t0);
    fetch(t0 + TT);                                       // (an empty group where there is nothing)
    fetch_values(t0);
    for (int base = t0; base < t1; base += TT) {
        const int n = min(TT, t1 - base);
        const int buf = ((base - t0) / TT) % BUFS;
        float bb[TT], bv[TT], op[TT];
#pragma unroll
        for (int tt = 0; tt < TT; ++tt) { bb[tt] = -bn[tt]; bv[tt] = bn[tt] * vn[tt]; op[tt] = 0.f; }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                  // the stage is there; the one asked for next lies where the stage before was
        fetch(base + 2 * TT);
        fetch_values(min(base + TT, t1 - 1));
        auto token = [&](int tt) {
            const ulonglong2* q4 = reinterpret_cast<const ulonglong2*>(ring[buf][tt][0]);
            const ulonglong2* k4 = reinterpret_cast<const ulonglong2*>(ring[buf][tt][1]);
            const ulonglong2* a4 = reinterpret_cast<const ulonglong2*>(ring[buf][tt][2]);
            uint64_t k[2 * NC], a[2 * NC], part[4];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const ulonglong2 kk = k4[c * 8 + p], aa = a4[c * 8 + p];
                k[2 * c] = kk.x; k[2 * c + 1] = kk.y;
                a[2 * c] = aa.x; a[2 * c + 1] = aa.y;
            }
#pragma unroll
            for (int i = 0; i < 2 * NC; ++i) {            // (a s)^T k = s^T (a k)
                const uint64_t ak = mul2(a[i], k[i]);
                part[i & 3] = i < 4 ? mul2(s[i], ak) : fma2(s[i], ak, part[i & 3]);
            }
            const float2 d2 = unpair(add2(add2(part[0], part[1]), add2(part[2], part[3])));
            float dot = d2.x + d2.y;
#pragma unroll
            for (int w = 1; w < 8; w <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, w);
            const float u = fmaf(bb[tt], dot, bv[tt]);    // b (v - dot)
            const uint64_t uu = pair_of(u, u);
            uint64_t o2[2];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const ulonglong2 q = q4[c * 8 + p];
                s[2 * c] = fma2(k[2 * c], uu, mul2(a[2 * c], s[2 * c]));
                s[2 * c + 1] = fma2(k[2 * c + 1], uu, mul2(a[2 * c + 1], s[2 * c + 1]));
                o2[0] = c == 0 ? mul2(s[2 * c], q.x) : fma2(s[2 * c], q.x, o2[0]);
                o2[1] = c == 0 ? mul2(s[2 * c + 1], q.y) : fma2(s[2 * c + 1], q.y, o2[1]);
            }
            const float2 o = unpair(add2(o2[0], o2[1]));
            op[tt] = o.x + o.y;
        };
        if (n == TT) {
#pragma unroll
            for (int tt = 0; tt < TT; ++tt) token(tt);
        } else {
#pragma unroll
            for (int tt = 0; tt < TT; ++tt)
                if (tt < n) token(tt);
        }
        // eight tokens over eight lanes: lane p ends with token p's sum
#pragma unroll
        for (int w = 4; w > 0; w >>= 1) {
#pragma unroll
            for (int i = 0; i < w; ++i) {
                const float send = p & w ? op[i] : op[i + w], keep = p & w ? op[i + w] : op[i];
                op[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
            }
        }
        if (p < n) out[((long long)(base + p) * H + h) * E + j] = op[0];
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int d = (c * 8 + p) * 4;
        const float2 x = unpair(s[2 * c]), y = unpair(s[2 * c + 1]);
        Sh[(long long)d * E] = x.x;
        Sh[(long long)(d + 1) * E] = x.y;
        Sh[(long long)(d + 2) * E] = y.x;
        Sh[(long long)(d + 3) * E] = y.y;
    }
}

// The recurrence four tokens at a time, for prompts of runs whose sums need not have one order however a sequence is cut
// (16-bit activations).  With g_i the product of the decays up to token i of the four (a number a key channel), everything that
// four tokens ask of the state can be asked of the state before them:
//     u_i = b_i (v_i - S^T (g_i k_i) - sum_{j<i} c_ij u_j),     c_ij = sum_d k_j (a_{j+1} .. a_i) k_i
//     o_i = S^T (g_i q_i) + sum_{j<=i} e_ij u_j,                e_ij = sum_d k_j (a_{j+1} .. a_i) q_i
//     S  <- g_4 S + sum_j (a_{j+1} .. a_4) k_j u_j^T
// so the chain from token to token has one round of exchanges for four of them, and an element of the state takes 13 operations
// instead of 20.  All products are of decays in (0, 1]: nothing is divided and nothing grows.  What does not depend on the state
// is made by a kernel of its own, once for a head's columns: a record of 13 rows of D numbers (g_i k_i, g_i q_i, the writes' keys,
// g_4) and eight rows of four (c_i0, c_i1, c_i2, b_i; e_i0 .. e_i3) for every four tokens and head.  A sequence's last record is filled up
// with tokens that write nothing (k = q = 0, a = 1, b = 0).
// 2,048 tokens, 16 heads of 128 x 128: 491 (the kernel above) -> 12 + 271 us.
constexpr int DELTA_RECORD_BUFS = 6;        // records in shared memory: five are on their way, some 2 us ahead
template <int D> struct DeltaRecord { static constexpr int FLOATS = 13 * D + 32; };

// Records of the sequences before sequence b: at most this many, so it is b's first record's place.  Sequences with fewer than min_new
// tokens are passed over (the kernel above takes them), so a sequence's kernel, and with it its rounding, follows its own tokens
// and not what shares the step; of those with 32 tokens or more, n have at most n / 4 + 1 and so floor(9 n / 32) records, however
// many shorter sequences lie between.
constexpr int DELTA_LONG = 32;
__device__ __forceinline__ int first_record(const int* seq_start, int b, int min_new) {
    return min_new >= DELTA_LONG ? (int)(9LL * seq_start[b] >> 5) : (seq_start[b] + 3 * b) >> 2;
}

template <int D>
__global__ void __launch_bounds__(128)
delta_records_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ beta,
                     const float* __restrict__ dec, float* __restrict__ rec, const int* __restrict__ seq_start, int H, int G, int min_new,
                     int below) {
    pdl_trigger();
    pdl_wait();
    constexpr int V = D / 32;
    const int b = blockIdx.y, lane = threadIdx.x & 31;
    const int unit = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, h = unit % H, nb = unit / H, g = h / (H / G);
    const int t0 = seq_start[b] + 4 * nb, n = min(4, seq_start[b + 1] - t0);
    if (n <= 0 || seq_start[b + 1] - seq_start[b] < min_new || seq_start[b + 1] - seq_start[b] >= below) return;
    float* r = rec + ((long long)(first_record(seq_start, b, min_new) + nb) * H + h) * DeltaRecord<D>::FLOATS;
    float k[4][V], q[4][V], a[4][V], bt[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        bt[i] = 0.f;
#pragma unroll
        for (int v = 0; v < V; ++v) { k[i][v] = q[i][v] = 0.f; a[i][v] = 1.f; }
        if (i < n) {
            const long long t = t0 + i;
            load_vec<float, V>(kn + (t * G + g) * D + lane * V, k[i]);
            load_vec<float, V>(qn + (t * G + g) * D + lane * V, q[i]);
            load_vec<float, V>(dec + (t * H + h) * D + lane * V, a[i]);
            bt[i] = beta[t * H + h];
        }
    }
    float c[4][4], e[4][4], row[V], p[V];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] = e[i][j] = 0.f;
#pragma unroll
    for (int v = 0; v < V; ++v) p[v] = 1.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {                          // g_i, and with it the rows the state is asked with
#pragma unroll
        for (int v = 0; v < V; ++v) { p[v] *= a[i][v]; row[v] = p[v] * k[i][v]; }
        store_vec<float, V>(r + i * D + lane * V, row);
#pragma unroll
        for (int v = 0; v < V; ++v) row[v] = p[v] * q[i][v];
        store_vec<float, V>(r + (4 + i) * D + lane * V, row);
    }
    store_vec<float, V>(r + 12 * D + lane * V, p);
#pragma unroll
    for (int j = 0; j < 4; ++j) {                          // k_j on its way through the decays behind it
#pragma unroll
        for (int v = 0; v < V; ++v) { row[v] = k[j][v]; e[j][j] = fmaf(row[v], q[j][v], e[j][j]); }
#pragma unroll
        for (int i = j + 1; i < 4; ++i)
#pragma unroll
            for (int v = 0; v < V; ++v) {
                row[v] *= a[i][v];
                c[i][j] = fmaf(row[v], k[i][v], c[i][j]);
                e[i][j] = fmaf(row[v], q[i][v], e[i][j]);
            }
        store_vec<float, V>(r + (8 + j) * D + lane * V, row);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            if (j < i) c[i][j] = warp_sum(c[i][j]);
            e[i][j] = warp_sum(e[i][j]);
        }
    if (lane == 0) {
        float4* coef = reinterpret_cast<float4*>(r + 13 * D);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            coef[i] = make_float4(c[i][0], c[i][1], c[i][2], bt[i]);
            coef[4 + i] = make_float4(e[i][0], e[i][1], e[i][2], e[i][3]);
        }
    }
}

// One warp a scheduler walks a chain, so a load whose number is used at once costs its whole latency: the places of the loads from
// shared memory are therefore written out (the compiler put them next to their uses: 425 us against 348).  The rows that the next record asks
// the state with are fetched behind this record's update, the update's rows ahead of the exchanges.
__device__ __forceinline__ void lds_pairs(uint64_t& x, uint64_t& y, const float* p) {
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ float4 lds_four(const float* p) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"((uint32_t)__cvta_generic_to_shared(p)));
    return v;
}
__device__ __forceinline__ float2 lds_two(const float* p) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"((uint32_t)__cvta_generic_to_shared(p)));
    return v;
}

// Sixteen lanes hold two neighbouring columns of the state, lane p the key channels of the float4 chunks p, p + 16, ...: what bounds
// the kernel next is the width of the way from shared memory to the registers (a load of sixteen bytes takes a warp four turns,
// whether its lanes read the same bytes or not), and two columns share a lane's loads (eight
// lanes and one column: 348 us; sixteen and one, with two warps a scheduler: 370; this: 277).  Sixteen sums (four askings and four read-outs
// of two columns) meet by fifteen exchanges that leave lane p with sum p.
template <int D>
__global__ void __launch_bounds__(128)
delta_scan_records_kernel(const float* __restrict__ rec, const float* __restrict__ vc, float* __restrict__ out, float* __restrict__ S,
                          const int* __restrict__ seq_start, const int* __restrict__ seq_slot, int H, int E, int min_new, int below) {
    constexpr int NC = D / 64, REC = DeltaRecord<D>::FLOATS, STAGE = REC + 64, BUFS = DELTA_RECORD_BUFS;
    extern __shared__ __align__(16) float ring[];          // [BUFS][STAGE]: a record and its four tokens' values of the block's columns
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, col = (tid >> 4) * 2, p = tid & 15;
    const int h = blockIdx.y, b = blockIdx.z;
    const int j = blockIdx.x * 16 + col;
    const int t0 = seq_start[b], t1 = seq_start[b + 1], n_rec = (t1 - t0 + 3) >> 2;
    if (n_rec <= 0 || t1 - t0 < min_new || t1 - t0 >= below) return;
    float* Sh = S + ((long long)seq_slot[b] * H + h) * D * E + j;
    uint64_t s[2][2 * NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const long long d = (c * 16 + p) * 4;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            s[k][2 * c] = pair_of(Sh[d * E + k], Sh[(d + 1) * E + k]);
            s[k][2 * c + 1] = pair_of(Sh[(d + 2) * E + k], Sh[(d + 3) * E + k]);
        }
    }
    // this thread's pieces of a record, and the pointer that walks over them
    const float* src = rec + ((long long)first_record(seq_start, b, min_new) * H + h) * REC + tid * 4;
    const float* vsrc = vc + (long long)h * E + blockIdx.x * 16 + (tid & 3) * 4;
    const long long rstep = (long long)H * REC, vstep = (long long)H * E;
    int fetched = 0, fbuf = 0;
    auto fetch = [&]() {                                   // the next record, or nothing behind the last
        if (fetched < n_rec) {
            float* to = ring + fbuf * STAGE + tid * 4;
#pragma unroll
            for (int i = 0; i < (REC + 511) / 512; ++i)
                if (tid * 4 + i * 512 < REC) cp_async16(to + i * 512, src + i * 512);
            if (tid < 16)                                  // (a token past the end: the last one's values, which its write leaves out)
                cp_async16(ring + fbuf * STAGE + REC + tid * 4, vsrc + min(t0 + 4 * fetched + (tid >> 2), t1 - 1) * vstep);
            src += rstep;
        }
        ++fetched;
        fbuf = fbuf + 1 == BUFS ? 0 : fbuf + 1;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int r = 0; r < BUFS; ++r) fetch();
    uint64_t ask[8][2 * NC];
    auto load_ask = [&](const float* R) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int c = 0; c < NC; ++c) lds_pairs(ask[i][2 * c], ask[i][2 * c + 1], R + i * D + (c * 16 + p) * 4);
    };
    asm volatile("cp.async.wait_group %0;" ::"n"(BUFS - 1) : "memory");
    __syncthreads();
    load_ask(ring);
    const float* R = ring;
    const int tok = (p & 7) >> 1;                          // lanes 8 to 15: token and column of the read-out they end with
    float* op = out + ((long long)(t0 + tok) * H + h) * E + j + (p & 1);
    int left = p >= 8 ? t1 - t0 - tok : 0;                 // tokens from this lane's own of the record on
    // ``part``: a sequence's last record with n_tok tokens, in a copy of its own behind the loop (asked in the loop it cost a tenth)
    auto record = [&](auto part, int n_tok) {
        float m[16];                                       // 2 i + k: S_k^T (g_i k_i); 8 + 2 i + k: S_k^T (g_i q_i)
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                uint64_t x = mul2(s[k][0], ask[i][0]), y = mul2(s[k][1], ask[i][1]);
#pragma unroll
                for (int c = 1; c < NC; ++c) { x = fma2(s[k][2 * c], ask[i][2 * c], x); y = fma2(s[k][2 * c + 1], ask[i][2 * c + 1], y); }
                const float2 t = unpair(add2(x, y));
                m[2 * i + k] = t.x + t.y;
            }
        // what the update reads, asked for ahead of the exchanges
        uint64_t w[5][2 * NC];
        float4 cf[4];
        float2 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) { cf[i] = lds_four(R + 13 * D + 4 * i); v[i] = lds_two(R + REC + 16 * i + col); }
#pragma unroll
        for (int i = 0; i < 5; ++i)
#pragma unroll
            for (int c = 0; c < NC; ++c) lds_pairs(w[i][2 * c], w[i][2 * c + 1], R + (8 + i) * D + (c * 16 + p) * 4);
        const float4 e = lds_four(R + 13 * D + 16 + 4 * tok);
#pragma unroll
        for (int x = 8; x > 0; x >>= 1)
#pragma unroll
            for (int i = 0; i < x; ++i) {
                const float send = p & x ? m[i] : m[i + x], keep = p & x ? m[i + x] : m[i];
                m[i] = keep + __shfl_xor_sync(0xffffffffu, send, x);
            }
        float u[2][4];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            float d[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) d[i] = (k ? v[i].y : v[i].x) - __shfl_sync(0xffffffffu, m[0], 2 * i + k, 16);
            u[k][0] = cf[0].w * d[0];
            u[k][1] = cf[1].w * fmaf(-cf[1].x, u[k][0], d[1]);
            u[k][2] = cf[2].w * fmaf(-cf[2].y, u[k][1], fmaf(-cf[2].x, u[k][0], d[2]));
            u[k][3] = cf[3].w * fmaf(-cf[3].z, u[k][2], fmaf(-cf[3].y, u[k][1], fmaf(-cf[3].x, u[k][0], d[3])));
            if (decltype(part)::value) {                   // past the end nothing is written, also where the token before wrote an infinity
#pragma unroll
                for (int i = 1; i < 4; ++i)
                    if (i >= n_tok) u[k][i] = 0.f;
            }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
#pragma unroll
            for (int c = 0; c < 2 * NC; ++c) s[k][c] = mul2(w[4][c], s[k][c]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint64_t uu = pair_of(u[k][i], u[k][i]);
#pragma unroll
                for (int c = 0; c < 2 * NC; ++c) s[k][c] = fma2(w[i][c], uu, s[k][c]);
            }
        }
        asm volatile("cp.async.wait_group %0;" ::"n"(BUFS - 2) : "memory");
        __syncthreads();                                   // the next record is there, and nobody reads this one any more
        fetch();
        R = R == ring + (BUFS - 1) * STAGE ? ring : R + STAGE;
        load_ask(R);                                       // (behind the last record: numbers that nothing uses)
        const bool odd = p & 1;
        const float u0 = odd ? u[1][0] : u[0][0], u1 = odd ? u[1][1] : u[0][1], u2 = odd ? u[1][2] : u[0][2], u3 = odd ? u[1][3] : u[0][3];
        float o = fmaf(e.w, u3, fmaf(e.z, u2, fmaf(e.y, u1, fmaf(e.x, u0, m[0]))));
        if (!isfinite(o)) {                                // zero times a later token's infinite write: such writes are left out
            o = fmaf(e.x, u0, m[0]);
            if (tok > 0) o = fmaf(e.y, u1, o);
            if (tok > 1) o = fmaf(e.z, u2, o);
            if (tok > 2) o = fmaf(e.w, u3, o);
        }
        if (left > 0) *op = o;
        op += 4 * vstep;
        left -= 4;
    };
    const int n_full = (t1 - t0) >> 2;
#pragma unroll 1
    for (int r = 0; r < n_full; ++r) record(std::false_type{}, 4);
    if (n_full < n_rec) record(std::true_type{}, t1 - t0 - 4 * n_full);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const long long d = (c * 16 + p) * 4;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float2 x = unpair(s[k][2 * c]), y = unpair(s[k][2 * c + 1]);
            Sh[d * E + k] = x.x;
            Sh[(d + 1) * E + k] = x.y;
            Sh[(d + 2) * E + k] = y.x;
            Sh[(d + 3) * E + k] = y.y;
        }
    }
}

// The recurrence sixteen tokens at a time, for prompts of runs whose sums need not have one order however a sequence is cut
// (16-bit activations).  With g_i the product of the decays up to token i of the sixteen (a number a key channel), everything that
// the tokens ask of the state can be asked of the state S before them:
//     u_i = b_i (v_i - S^T (g_i k_i) - sum_{j<i} c_ij u_j),     c_ij = sum_d k_j (a_{j+1} .. a_i) k_i
//     o_i = S^T (g_i q_i) + sum_{j<=i} e_ij u_j,                e_ij = sum_d k_j (a_{j+1} .. a_i) q_i
//     S  <- g_16 S + sum_j w_j u_j^T,                           w_j = (a_{j+1} .. a_16) k_j
// u_i is linear in the values and in S, so the sums over j are worked off ahead, row by row:
//     kb_i = b_i (g_i k_i - sum_{j<i} c_ij kb_j)     vb_i = b_i (v_i - sum_{j<i} c_ij vb_j)     u_i = vb_i - S^T kb_i
//     qb_i = g_i q_i - sum_{j<=i} e_ij kb_j          ob_i = sum_{j<=i} e_ij vb_j                o_i = ob_i + S^T qb_i
// (a published rearrangement: Yang, Wang, Zhang, Shen and Kim, "Parallelizing linear transformers with the delta rule over sequence
// length", 2024).
// All products are of decays in (0, 1]: nothing is divided and nothing grows.  The chain from sixteen tokens to the next is two
// small products, S^T [kb qb] and w u^T, which run on the tensor cores: a float32 operand as three bfloat16 parts, six products a term
// (as in gemm_f32_tc.cu), float32 sums.  What does not depend on the state is made by a kernel of its own, once for a head's columns:
// a record of the three parts of kb, qb and w (48 rows of D), g_16, and vb and ob of every sixteen columns, for each sixteen
// tokens and head.  A sequence's last record is filled up with tokens that write nothing (k = q = 0, a = 1, b = 0).
// Rows are worked off from the first, so what a token brings reaches no token before it.
// 2,048 tokens, 16 heads of 128 x 128: 279 us four tokens at a time -> 187 (70 for the records, 117 for the scan); four sequences of 512:
// 203 -> 191; 8 heads of 64 x 64: 189 -> 100.  Below some 300 tokens the records' kernel weighs more than the shorter chain gives.
constexpr int DELTA_CHUNK = 16;
constexpr int DELTA_ROWS = 3 * DELTA_CHUNK;                 // kb, qb, w
template <int D> struct DeltaChunk {
    static constexpr int PLANE = DELTA_ROWS * D;           // bfloat16 numbers of one part; sixteen bytes c of row r lie at c ^ (r % 8)
    static constexpr int HEAD = 3 * PLANE / 2 + D;         // floats ahead of the columns: the parts and g_16
    static constexpr int VB = 8 * 40, COLS = VB + 16 * DELTA_CHUNK;    // floats of sixteen columns: vb [pair of tokens: 40][column][2], ob [token][column]
    __host__ __device__ static constexpr long long floats(int E) { return HEAD + (long long)(E / 16) * COLS; }
};

// A portion of the work: the sequences from ``seq`` on (as many as the grid has), of each the tokens from ``first`` on (a multiple of
// sixteen), at most ``most`` records; sequences with fewer than ``min_new`` tokens are left alone.  The state carries over from portion to
// portion, so the sums and their bits are those of the whole; a long step then needs no more scratch than its caller has.
// ``places``: the records a head that there is room for.
struct DeltaPortion { int seq, first, most, min_new; long long places; };

// The records of the portion that lie before sequence b's, counted by each warp.
__device__ __forceinline__ long long first_chunk(const int* seq_start, int b, const DeltaPortion& q) {
    int sum = 0;
    for (int i = q.seq + (threadIdx.x & 31); i < b; i += 32) {
        const int n = seq_start[i + 1] - seq_start[i];
        if (n >= q.min_new && n > q.first) sum += min(q.most, (n - q.first + DELTA_CHUNK - 1) / DELTA_CHUNK);
    }
    return __reduce_add_sync(0xffffffffu, sum);
}

__device__ __forceinline__ void split_bf16(float x, float y, uint32_t* part) {
    auto pack = [](float a, float b) { __nv_bfloat162 v = __floats2bfloat162_rn(a, b); return *reinterpret_cast<uint32_t*>(&v); };
    auto low = [](uint32_t v) { return __uint_as_float(v << 16); };
    auto high = [](uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); };
    part[0] = pack(x, y);
    x -= low(part[0]); y -= high(part[0]);
    part[1] = pack(x, y);
    part[2] = pack(x - low(part[1]), y - high(part[1]));
}

// One block of D / 2 threads a record, a thread two key channels, then two columns.  What bounds it: the triangles' numbers on their way
// from shared memory (two turns for eight bytes, though every lane reads the same), which two channels share; before that 256 sums over
// the channels, 32 of which meet by 31 exchanges a warp.  The triangles are worked off in 64 bits: in 32 the rounding of sixteen rows
// in a row was half of the recurrence's error (outputs of 2,048 tokens against 64 bits, 2-norm: 1.35e-7, 9.9e-8 so, 1.15e-7 four tokens at a
// time, 1.12e-7 token by token).
template <int D>
__global__ void __launch_bounds__(D / 2)
delta_chunks_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vc, const float* __restrict__ beta,
                    const float* __restrict__ dec, float* __restrict__ rec, const int* __restrict__ seq_start, int H, int G, int E,
                    DeltaPortion po, int* __restrict__ error) {
    pdl_trigger();
    pdl_wait();
    constexpr int C = DELTA_CHUNK, WARPS = D / 64, N = D / 2;
    __shared__ float sums[WARPS][8][32];
    __shared__ __align__(16) double cm[C][C], em[C][C];    // c_ij and e_ij
    __shared__ __align__(16) float rows[DELTA_ROWS * D];   // kb, qb and w, then the columns
    static_assert(D / 16 * DeltaChunk<D>::COLS <= DELTA_ROWS * D, "the columns' place");
    const int b = po.seq + blockIdx.y, h = blockIdx.x % H, nb = blockIdx.x / H, g = h / (H / G), tid = threadIdx.x, lane = tid & 31;
    const int t0 = seq_start[b] + po.first + C * nb, n = min(C, seq_start[b + 1] - t0);
    if (n <= 0 || seq_start[b + 1] - seq_start[b] < po.min_new) return;
    const long long place = first_chunk(seq_start, b, po) + nb;
    if (place >= po.places) {                              // (a caller that counted wrong: the scan raises it too and writes nothing)
        if (tid == 0 && error) atomicExch(error, 1);
        return;
    }
    float* r = rec + (place * H + h) * DeltaChunk<D>::floats(E);
    float2 k[C], q[C], a[C];
    float bt[C];
#pragma unroll
    for (int i = 0; i < C; ++i) {
        k[i] = q[i] = make_float2(0.f, 0.f);
        bt[i] = 0.f;
        a[i] = make_float2(1.f, 1.f);
        if (i < n) {
            const long long t = t0 + i;
            k[i] = reinterpret_cast<const float2*>(kn + (t * G + g) * D)[tid];
            q[i] = reinterpret_cast<const float2*>(qn + (t * G + g) * D)[tid];
            a[i] = reinterpret_cast<const float2*>(dec + (t * H + h) * D)[tid];
            bt[i] = beta[t * H + h];
        }
    }
    // columns j and 15 - j of both triangles are 32 sums
#pragma unroll
    for (int j = 0; j < C / 2; ++j) {
        float m[32];
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const int jj = side ? C - 1 - j : j, base = side ? 31 - 2 * j : 0;
            float2 row = k[jj];
#pragma unroll
            for (int i = jj; i < C; ++i) {
                if (i > jj) {
                    row.x *= a[i].x; row.y *= a[i].y;
                    m[base + C - jj + i - jj - 1] = fmaf(row.x, k[i].x, row.y * k[i].y);
                }
                m[base + i - jj] = fmaf(row.x, q[i].x, row.y * q[i].y);
            }
        }
#pragma unroll
        for (int x = 16; x > 0; x >>= 1)
#pragma unroll
            for (int i = 0; i < x; ++i) {
                const float send = lane & x ? m[i] : m[i + x], keep = lane & x ? m[i + x] : m[i];
                m[i] = keep + __shfl_xor_sync(0xffffffffu, send, x);
            }
        sums[tid >> 5][j][lane] = m[0];
    }
    auto put = [&](int row, float x, float y) { reinterpret_cast<float2*>(rows + row * D)[tid] = make_float2(x, y); };
    float2 t = make_float2(1.f, 1.f);
#pragma unroll
    for (int j = C - 1; j >= 0; --j) {                     // w_j: k_j through the decays behind it
        put(2 * C + j, k[j].x * t.x, k[j].y * t.y);
        t.x *= a[j].x; t.y *= a[j].y;
    }
    reinterpret_cast<float2*>(r + 3 * DeltaChunk<D>::PLANE / 2)[tid] = t;
    __syncthreads();
    for (int v = tid; v < 256; v += N) {
        const int j = v >> 5, first = 31 - 2 * j;          // (sums of column j, then of column 15 - j; of each e, then c)
        const int jj = (v & 31) < first ? j : C - 1 - j, at = (v & 31) < first ? v & 31 : (v & 31) - first;
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) x += sums[w][j][v & 31];
        if (at < C - jj) em[jj + at][jj] = x;
        else cm[jj + 1 + at - (C - jj)][jj] = x;
    }
    __syncthreads();
    double px = 1.0, py = 1.0, bx[C], by[C];
#pragma unroll
    for (int i = 0; i < C; ++i) {
        px *= a[i].x; py *= a[i].y;
        double x = px * k[i].x, y = py * k[i].y, u = px * q[i].x, v = py * q[i].y;
#pragma unroll
        for (int j = 0; j < i; ++j) { const double c = cm[i][j]; x = fma(-c, bx[j], x); y = fma(-c, by[j], y); }
        bx[i] = bt[i] * x;
        by[i] = bt[i] * y;
        put(i, (float)bx[i], (float)by[i]);
#pragma unroll
        for (int j = 0; j <= i; ++j) { const double e = em[i][j]; u = fma(-e, bx[j], u); v = fma(-e, by[j], v); }
        put(C + i, (float)u, (float)v);
    }
    __syncthreads();
    for (int i = tid; i < DELTA_ROWS * D / 8; i += N) {    // eight channels of a row into sixteen bytes of each part
        const int row = i / (D / 8), c = i % (D / 8);
        const float4 x = reinterpret_cast<const float4*>(rows)[2 * i], y = reinterpret_cast<const float4*>(rows)[2 * i + 1];
        uint32_t p0[3], p1[3], p2[3], p3[3];
        split_bf16(x.x, x.y, p0); split_bf16(x.z, x.w, p1); split_bf16(y.x, y.y, p2); split_bf16(y.z, y.w, p3);
        uint4* dst = reinterpret_cast<uint4*>(r) + row * (D / 8) + (c ^ (row & 7));
#pragma unroll
        for (int p = 0; p < 3; ++p) dst[p * (DeltaChunk<D>::PLANE / 8)] = make_uint4(p0[p], p1[p], p2[p], p3[p]);
    }
    __syncthreads();
    for (int c0 = 0; c0 < E; c0 += D) {
        const int cl = 2 * tid & 15, width = min(D, E - c0);
        if (2 * tid < width) {
            float* col = rows + (tid >> 3) * DeltaChunk<D>::COLS;
            float2 vi[C];
#pragma unroll
            for (int i = 0; i < C; ++i)
                vi[i] = i < n ? *reinterpret_cast<const float2*>(vc + ((t0 + i) * (long long)H + h) * E + c0 + 2 * tid) : make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < C; ++i) {
                double x = vi[i].x, y = vi[i].y, u = 0.0, v = 0.0;
#pragma unroll
                for (int j = 0; j < i; ++j) { const double c = cm[i][j]; x = fma(-c, bx[j], x); y = fma(-c, by[j], y); }
                bx[i] = bt[i] * x;                         // vb_i
                by[i] = bt[i] * y;
#pragma unroll
                for (int j = 0; j <= i; ++j) { const double e = em[i][j]; u = fma(e, bx[j], u); v = fma(e, by[j], v); }
                if (i & 1) *reinterpret_cast<float4*>(col + (i >> 1) * 40 + cl * 2) = make_float4((float)bx[i - 1], (float)bx[i], (float)by[i - 1], (float)by[i]);
                *reinterpret_cast<float2*>(col + DeltaChunk<D>::VB + i * 16 + cl) = make_float2((float)u, (float)v);
            }
        }
        __syncthreads();
        float4* dst = reinterpret_cast<float4*>(r + DeltaChunk<D>::HEAD + (long long)(c0 >> 4) * DeltaChunk<D>::COLS);
        for (int i = tid; i < width / 16 * (DeltaChunk<D>::COLS / 4); i += N) dst[i] = reinterpret_cast<const float4*>(rows)[i];
        __syncthreads();
    }
}

__device__ __forceinline__ void mma_bf16_16816(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void bulk_copy(float* dst, const float* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t* r, const void* p) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(p);
    if (TRANS) asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
    else asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}

// A block takes sixteen columns of a head's state, transposed: rows are columns of S, and each of four warps holds a quarter of the key
// channels in the layout of an MMA's result, which is that of its left operand two tiles at a time.  S^T [kb qb] is summed over the
// warps through shared memory; then every warp has all of u and updates its own channels.  What bounds it is the chain: some 1,700
// cycles a record for 435 instructions a warp, 72 of them MMAs, one warp a scheduler.
constexpr int DELTA_CHUNK_BUFS = 4;                              // records in shared memory
template <int D> constexpr int delta_scan_smem() {
    return (DELTA_CHUNK_BUFS * (DeltaChunk<D>::HEAD + DeltaChunk<D>::COLS) + 2 * 4 * 16 * 40) * (int)sizeof(float) + DELTA_CHUNK_BUFS * 8 + 16;
}
// Four warps that compute and one that has the records copied.  (By cp.async, from the computing warps or from others, the copies took 800
// of 2,000 cycles a record: they go through the same units as the loads from shared memory.)
constexpr int DELTA_SCAN_THREADS = 160;
template <int D>
__global__ void __launch_bounds__(DELTA_SCAN_THREADS)
delta_scan_chunks_kernel(const float* __restrict__ rec, float* __restrict__ out, float* __restrict__ S, const int* __restrict__ seq_start,
                          const int* __restrict__ seq_slot, int H, int E, DeltaPortion po, int* __restrict__ error) {
    constexpr int C = DELTA_CHUNK, NT = D / 32, KS = D / 64, STAGE = DeltaChunk<D>::HEAD + DeltaChunk<D>::COLS, XROW = 40;
    extern __shared__ __align__(128) float ring[];         // [BUFS][STAGE], then the warps' sums [2][4][16 columns][XROW]
    float* xch = ring + DELTA_CHUNK_BUFS * STAGE;
    uint64_t* full = reinterpret_cast<uint64_t*>(xch + 2 * 4 * 16 * XROW);
    volatile int* err = reinterpret_cast<volatile int*>(full + DELTA_CHUNK_BUFS);
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, row = lane >> 2, quad = lane & 3;
    const int h = blockIdx.y, b = po.seq + blockIdx.z, col0 = blockIdx.x * 16;
    const int t0 = seq_start[b] + po.first, T = min(seq_start[b + 1] - t0, C * po.most), n_rec = (T + C - 1) / C;
    if (T <= 0 || seq_start[b + 1] - seq_start[b] < po.min_new) return;
    const long long place = first_chunk(seq_start, b, po);
    if (place + n_rec > po.places) {
        if (tid == 0 && error) atomicExch(error, 1);
        return;
    }
    const long long step = (long long)H * DeltaChunk<D>::floats(E);
    if (tid == 128) {
        for (int i = 0; i < DELTA_CHUNK_BUFS; ++i) mbar_init(&full[i], 1);
        *err = 0;
        fence_barrier_init();
    }
    if (warp == 4) {                                       // records on their way: BUFS - 1
        const float* src = rec + (place * H + h) * DeltaChunk<D>::floats(E);
        const float* csrc = src + DeltaChunk<D>::HEAD + blockIdx.x * DeltaChunk<D>::COLS;
        int fetched = 0;
        auto fetch = [&]() {                               // the next record, or nothing behind the last
            if (fetched >= n_rec) return;
            uint64_t* bar = &full[fetched % DELTA_CHUNK_BUFS];
            float* to = ring + fetched % DELTA_CHUNK_BUFS * STAGE;
            mbar_expect_tx(bar, STAGE * 4);
            bulk_copy(to, src, DeltaChunk<D>::HEAD * 4, bar);
            bulk_copy(to + DeltaChunk<D>::HEAD, csrc, DeltaChunk<D>::COLS * 4, bar);
            src += step;
            csrc += step;
            ++fetched;
        };
        if (lane == 0) {
            for (int r = 0; r < DELTA_CHUNK_BUFS - 1; ++r) fetch();
            mbar_wait(&full[0], 0, err);
        }
        __syncwarp();
        __syncthreads();
        for (int rc = 0; rc < n_rec; ++rc) {
            if (lane == 0 && rc + 1 < n_rec) mbar_wait(&full[(rc + 1) % DELTA_CHUNK_BUFS], (uint32_t)(((rc + 1) / DELTA_CHUNK_BUFS) & 1), err);
            __syncwarp();
            __syncthreads();                               // (the one in the computing warps' loop: nobody reads the record before this one)
            if (lane == 0 && !*err) fetch();
        }
        if (lane == 0 && *err) {                           // the copies in flight land before the block's memory goes
            const long long since = clock64();
            for (int r = max(0, fetched - DELTA_CHUNK_BUFS); r < fetched; ++r)
                while (!mbar_try_wait(&full[r % DELTA_CHUNK_BUFS], (r / DELTA_CHUNK_BUFS) & 1)) if (clock64() - since > WAIT_LIMIT_CYCLES / 4) break;
            if (error) atomicExch(error, 1);
        }
        return;
    }
    float* Sh = S + ((long long)seq_slot[b] * H + h) * D * E + col0;
    const int ch0 = warp * (D / 4) + 2 * quad;             // channels ch0 + 8 i and the next, of columns row and row + 8
    float s[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x) s[i][x] = Sh[(long long)(ch0 + 8 * i + (x & 1)) * E + row + (x >> 1) * 8];
    __syncthreads();
    // the smallest products first: (part of the left operand, part of the right one)
    constexpr int PA[6] = {2, 1, 0, 1, 0, 0}, PB[6] = {0, 1, 2, 0, 1, 0};
    float* op = out + ((long long)(t0 + 2 * (tid >> 4)) * H + h) * E + col0 + (tid & 15);    // this thread's two read-outs
    uint32_t kb[3][KS][2][4];                              // the next record's askings: sixteen tokens (kb, qb) x sixteen channels
    auto load_asks = [&](const float* at) {
        const uint8_t* planes = reinterpret_cast<const uint8_t*>(at);
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int rr = i * 16 + (lane >> 4) * 8 + (lane & 7), c = warp * (D / 32) + 2 * ks + ((lane >> 3) & 1);
                    ldmatrix4<false>(kb[p][ks][i], planes + p * (2 * DeltaChunk<D>::PLANE) + rr * (2 * D) + ((c ^ (rr & 7)) << 4));
                }
    };
    load_asks(ring);
    int buf = 0;
#pragma unroll 1
    for (int rc = 0; rc < n_rec; ++rc) {
        const float* R = ring + buf * STAGE;
        const uint8_t* planes = reinterpret_cast<const uint8_t*>(R);
        // ---- S^T [kb qb] over this warp's channels ----
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[i][x] = 0.f;
        uint32_t sa[KS][3][4];
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                uint32_t part[3];
                split_bf16(s[2 * ks + (x >> 1)][(x & 1) * 2], s[2 * ks + (x >> 1)][(x & 1) * 2 + 1], part);
#pragma unroll
                for (int p = 0; p < 3; ++p) sa[ks][p][x] = part[p];
            }
#pragma unroll
        for (int j = 0; j < 5; ++j)
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    mma_bf16_16816(acc[i], sa[ks][PA[j]], kb[PB[j]][ks][i >> 1][(i & 1) * 2], kb[PB[j]][ks][i >> 1][(i & 1) * 2 + 1]);
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float hh[4] = {0.f, 0.f, 0.f, 0.f};
                mma_bf16_16816(hh, sa[ks][0], kb[0][ks][i >> 1][(i & 1) * 2], kb[0][ks][i >> 1][(i & 1) * 2 + 1]);
#pragma unroll
                for (int x = 0; x < 4; ++x) acc[i][x] += hh[x];
            }
        float* xw = xch + ((rc & 1) * 4 + warp) * 16 * XROW;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            *reinterpret_cast<float2*>(xw + row * XROW + 8 * i + 2 * quad) = make_float2(acc[i][0], acc[i][1]);
            *reinterpret_cast<float2*>(xw + (row + 8) * XROW + 8 * i + 2 * quad) = make_float2(acc[i][2], acc[i][3]);
        }
        // what the update reads, asked for ahead of the exchange
        uint32_t wf[3][NT / 2][4];
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int i = 0; i < NT / 2; ++i) {             // sixteen tokens x sixteen channels, transposed
                const int rr = 2 * C + ((lane >> 3) & 1) * 8 + (lane & 7), c = warp * (D / 32) + 2 * i + (lane >> 4);
                ldmatrix4<true>(wf[p][i], planes + p * (2 * DeltaChunk<D>::PLANE) + rr * (2 * D) + ((c ^ (rr & 7)) << 4));
            }
        float u[8];                                        // columns row and row + 8, tokens 2 quad, 2 quad + 1, the same of the second eight
#pragma unroll
        for (int x = 0; x < 4; ++x)
            *reinterpret_cast<float2*>(u + 2 * x) = *reinterpret_cast<const float2*>(R + DeltaChunk<D>::HEAD + ((x >> 1) * 4 + quad) * 40 + (row + (x & 1) * 8) * 2);
        const float* ob = R + DeltaChunk<D>::HEAD + DeltaChunk<D>::VB + (tid >> 4) * 32 + (tid & 15);
        float2 o = make_float2(ob[0], ob[16]);             // column tid % 16, tokens 2 (tid / 16) and the next
        float2 gd[NT];
#pragma unroll
        for (int i = 0; i < NT; ++i) gd[i] = *reinterpret_cast<const float2*>(R + 3 * DeltaChunk<D>::PLANE / 2 + ch0 + 8 * i);
        __syncthreads();                                   // the sums and the next record are there
        buf = buf + 1 == DELTA_CHUNK_BUFS ? 0 : buf + 1;
        const float* xr = xch + (rc & 1) * 4 * 16 * XROW;
#pragma unroll
        for (int x = 0; x < 4; ++x) {                      // (column row or row + 8, first or second eight tokens)
            float2 m = make_float2(0.f, 0.f);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const float2 v = *reinterpret_cast<const float2*>(xr + (w * 16 + row + (x & 1) * 8) * XROW + (x >> 1) * 8 + 2 * quad);
                m.x += v.x; m.y += v.y;
            }
            u[(x >> 1) * 4 + (x & 1) * 2] -= m.x;
            u[(x >> 1) * 4 + (x & 1) * 2 + 1] -= m.y;
        }
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float2 v = *reinterpret_cast<const float2*>(xr + (w * 16 + (tid & 15)) * XROW + C + 2 * (tid >> 4));
            o.x += v.x; o.y += v.y;
        }
        const int left = T - rc * C;                       // tokens from the record's first on
        if (left < C) {                                    // past the end nothing is written, whatever the state holds
#pragma unroll
            for (int x = 0; x < 8; ++x)
                if ((x >> 2) * 8 + 2 * quad + (x & 1) >= left) u[x] = 0.f;
        }
        // ---- S <- g S + w u^T ----
        bool finite = true;
#pragma unroll
        for (int x = 0; x < 8; ++x) finite &= fabsf(u[x]) < 3.3e38f;
        float add[NT][4];
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int x = 0; x < 4; ++x) add[i][x] = 0.f;
        if (__all_sync(0xffffffffu, finite)) {
            uint32_t ua[3][4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                uint32_t part[3];
                split_bf16(u[(x >> 1) * 4 + (x & 1) * 2], u[(x >> 1) * 4 + (x & 1) * 2 + 1], part);
#pragma unroll
                for (int p = 0; p < 3; ++p) ua[p][x] = part[p];
            }
            float hm[NT][4], hh[NT][4];                    // three chains a tile: the sixth largest products, the next, the largest
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int x = 0; x < 4; ++x) hm[i][x] = hh[i][x] = 0.f;
            auto product = [&](float (&d)[NT][4], int j) {
#pragma unroll
                for (int i = 0; i < NT; ++i) mma_bf16_16816(d[i], ua[PA[j]], wf[PB[j]][i >> 1][(i & 1) * 2], wf[PB[j]][i >> 1][(i & 1) * 2 + 1]);
            };
            product(add, 0); product(hm, 3); product(hh, 5); product(add, 1); product(hm, 4); product(add, 2);
            load_asks(ring + buf * STAGE);                 // (behind the last record: numbers that nothing uses)
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int x = 0; x < 4; ++x) add[i][x] = (add[i][x] + hm[i][x]) + hh[i][x];
        } else {                                           // an infinite write has no three parts: token by token, from the parts of w
            load_asks(ring + buf * STAGE);
#pragma unroll 1
            for (int t = 0; t < C; ++t) {
                float u0 = 0.f, u1 = 0.f;
#pragma unroll
                for (int x = 0; x < 8; x += 4)
#pragma unroll
                    for (int y = 0; y < 2; ++y) {
                        const float p0 = __shfl_sync(0xffffffffu, u[x + y], (lane & 28) + ((t & 7) >> 1));
                        const float p1 = __shfl_sync(0xffffffffu, u[x + 2 + y], (lane & 28) + ((t & 7) >> 1));
                        if ((t >> 3) * 4 == x && (t & 1) == y) { u0 = p0; u1 = p1; }
                    }
                if (t >= left) break;
                const int rr = 2 * C + t;
#pragma unroll
                for (int i = 0; i < NT; ++i)
#pragma unroll
                    for (int y = 0; y < 2; ++y) {
                        const int ch = ch0 + 8 * i + y;
                        float w = 0.f;
#pragma unroll
                        for (int p = 2; p >= 0; --p)
                            w += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(planes + p * (2 * DeltaChunk<D>::PLANE) + rr * (2 * D) +
                                                                                          (((ch >> 3) ^ (rr & 7)) << 4) + (ch & 7) * 2));
                        add[i][y] = fmaf(w, u0, add[i][y]);
                        add[i][2 + y] = fmaf(w, u1, add[i][2 + y]);
                    }
            }
        }
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            s[i][0] = fmaf(gd[i].x, s[i][0], add[i][0]);
            s[i][1] = fmaf(gd[i].y, s[i][1], add[i][1]);
            s[i][2] = fmaf(gd[i].x, s[i][2], add[i][2]);
            s[i][3] = fmaf(gd[i].y, s[i][3], add[i][3]);
        }
        if (2 * (tid >> 4) < left) op[0] = o.x;
        if (2 * (tid >> 4) + 1 < left) op[(long long)H * E] = o.y;
        op += (long long)C * H * E;
    }
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x) Sh[(long long)(ch0 + 8 * i + (x & 1)) * E + row + (x >> 1) * 8] = s[i][x];
}

// VEC: sizes are multiples of 4 and every array starts on a 16-byte boundary, so tokens are fetched in
// 16-byte copies, each thread keeping the same one or two places of a token's row for the whole launch.
//
// GEN: the generalised rule, in which a token removes along its unit key u at a rate of its own for every key channel and
// writes its raw key: with c = S_old^T u,  S[d, :] = w[d] S_old[d, :] - rem[d] c + kraw[d] v,  o = S^T q.  ``kn`` then holds
// u, ``dec`` holds w, ``rem`` = rate * u and ``kraw`` come as two more arrays of the keys' shape, and ``beta`` is not read.
template <int R, int SCAN_LANES, bool VEC, bool GEN>
__global__ void __launch_bounds__(128)
delta_scan_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vc,
                  const float* __restrict__ beta, const float* __restrict__ dec, float* __restrict__ out,
                  float* __restrict__ S, const int* __restrict__ seq_start, const int* __restrict__ seq_slot,
                  int H, int G, int D, int E, const float* __restrict__ rem, const float* __restrict__ kraw) {
    static_assert(R % 4 == 0, "a lane holds whole float4 chunks");
    constexpr int SCAN_COLS = 128 / SCAN_LANES;
    constexpr int DP = SCAN_LANES * R;
    constexpr int NC = R / 4;                             // chunks a lane
    constexpr int TT = DP <= 128 ? 8 : 4;                 // tokens a stage
    __shared__ __align__(16) float sq[2][TT][DP], sk[2][TT][DP], sa[2][TT][DP];
    __shared__ __align__(16) float sr[GEN ? 2 : 1][GEN ? TT : 1][GEN ? DP : 4], sw[GEN ? 2 : 1][GEN ? TT : 1][GEN ? DP : 4];
    __shared__ __align__(16) float sv[2][TT][SCAN_COLS];
    __shared__ float sb[2][TT];
    __shared__ float so[TT][128];                          // the read-out's partial sums, [token][lane of the column][column]
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x;
    const int col = tid / SCAN_LANES, p = tid % SCAN_LANES;
    const int h = blockIdx.y, b = blockIdx.z;
    const int g = h / (H / G);
    const int j = blockIdx.x * SCAN_COLS + col;
    const int t0 = seq_start[b], t1 = seq_start[b + 1];
    if (t0 >= t1) return;
    float* Sh = S + ((long long)seq_slot[b] * H + h) * D * E;
    float s[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int d = ((i >> 2) * SCAN_LANES + p) * 4 + (i & 3);
        s[i] = (d < D && j < E) ? Sh[(long long)d * E + j] : 0.f;
    }
    // columns past the sizes are constants that no copy ever touches
    for (int idx = tid; idx < 2 * TT * DP; idx += blockDim.x) {
        const int d = idx % DP;
        if (d >= D) {
            (&sq[0][0][0])[idx] = 0.f; (&sk[0][0][0])[idx] = 0.f; (&sa[0][0][0])[idx] = 1.f;
            if (GEN) { (&sr[0][0][0])[idx] = 0.f; (&sw[0][0][0])[idx] = 0.f; }
        }
    }
    for (int idx = tid; idx < 2 * TT * SCAN_COLS; idx += blockDim.x)
        if (blockIdx.x * SCAN_COLS + idx % SCAN_COLS >= E) (&sv[0][0][0])[idx] = 0.f;

    // this thread's places in a token's [q | k | decay] row of 3 * D / 4 chunks (VEC)
    constexpr int NARR = GEN ? 5 : 3, NSL = GEN ? 3 : 2;          // arrays of the keys' shape; places a thread may hold
    int my_arr[NSL], my_d[NSL];
    for (int sl = 0; sl < NSL; ++sl) { my_arr[sl] = -1; my_d[sl] = 0; }
    if (VEC) {
        const int d4 = D >> 2;
        for (int sl = 0; sl < NSL; ++sl) {
            const int c = tid + sl * (int)blockDim.x;
            if (c < NARR * d4) { my_arr[sl] = c / d4; my_d[sl] = (c % d4) * 4; }
        }
    }
    const float* qrow = qn + (long long)g * D;
    const float* krow = kn + (long long)g * D;
    const float* arow = dec + (long long)h * D;
    const float* vrow = vc + (long long)h * E + blockIdx.x * SCAN_COLS;

    auto fetch = [&](int base, int buf) {
        const int n = min(TT, t1 - base);
        if (VEC) {
            for (int tt = 0; tt < n; ++tt) {
                const long long t = base + tt;
#pragma unroll
                for (int sl = 0; sl < NSL; ++sl) {
                    const int d = my_d[sl];
                    if (my_arr[sl] == 0) cp_async16(&sq[buf][tt][d], qrow + t * G * D + d);
                    else if (my_arr[sl] == 1) cp_async16(&sk[buf][tt][d], krow + t * G * D + d);
                    else if (my_arr[sl] == 2) cp_async16(&sa[buf][tt][d], arow + t * H * D + d);
                    else if (GEN && my_arr[sl] == 3) cp_async16(&sr[GEN ? buf : 0][GEN ? tt : 0][d], rem + (t * G + g) * D + d);
                    else if (GEN && my_arr[sl] == 4) cp_async16(&sw[GEN ? buf : 0][GEN ? tt : 0][d], kraw + (t * G + g) * D + d);
                }
            }
            if (tid < n * (SCAN_COLS / 4)) {
                const int tt = tid / (SCAN_COLS / 4), c = (tid % (SCAN_COLS / 4)) * 4;
                if (blockIdx.x * SCAN_COLS + c < E) cp_async16(&sv[buf][tt][c], vrow + (long long)(base + tt) * H * E + c);
            }
            if (!GEN && tid >= 64 && tid < 64 + n) cp_async4(&sb[buf][tid - 64], beta + (long long)(base + tid - 64) * H + h);
            asm volatile("cp.async.commit_group;" ::: "memory");
            return;
        }
        for (int idx = tid; idx < n * D; idx += blockDim.x) {
            const int tt = idx / D, d = idx % D;
            const long long t = base + tt;
            cp_async4(&sq[buf][tt][d], qn + (t * G + g) * D + d);
            cp_async4(&sk[buf][tt][d], kn + (t * G + g) * D + d);
            cp_async4(&sa[buf][tt][d], dec + (t * H + h) * D + d);
            if (GEN) {
                cp_async4(&sr[GEN ? buf : 0][GEN ? tt : 0][d], rem + (t * G + g) * D + d);
                cp_async4(&sw[GEN ? buf : 0][GEN ? tt : 0][d], kraw + (t * G + g) * D + d);
            }
        }
        for (int idx = tid; idx < n * SCAN_COLS; idx += blockDim.x) {
            const int tt = idx / SCAN_COLS, c = idx % SCAN_COLS;
            const int jj = blockIdx.x * SCAN_COLS + c;
            if (jj < E) cp_async4(&sv[buf][tt][c], vc + ((long long)(base + tt) * H + h) * E + jj);
        }
        if (!GEN && tid < n) cp_async4(&sb[buf][tid], beta + (long long)(base + tid) * H + h);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    fetch(t0, 0);
    int buf = 0;
    for (int base = t0; base < t1; base += TT, buf ^= 1) {
        const int n = min(TT, t1 - base);
        if (base + TT < t1) {
            fetch(base + TT, buf ^ 1);                    // (that buffer's readers passed the barrier at the end of the last round)
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        auto token = [&](int tt) {
            const float4* a4 = reinterpret_cast<const float4*>(sa[buf][tt]);
            const float4* k4 = reinterpret_cast<const float4*>(sk[buf][tt]);
            const float4* q4 = reinterpret_cast<const float4*>(sq[buf][tt]);
            if constexpr (GEN) {
                const float4* r4 = reinterpret_cast<const float4*>(sr[buf][tt]);
                const float4* w4 = reinterpret_cast<const float4*>(sw[buf][tt]);
                float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c = 0; c < NC; ++c) {                     // c = S_old^T u
                    const float4 u4 = k4[c * SCAN_LANES + p];
                    part[0] = fmaf(s[4 * c + 0], u4.x, part[0]);
                    part[1] = fmaf(s[4 * c + 1], u4.y, part[1]);
                    part[2] = fmaf(s[4 * c + 2], u4.z, part[2]);
                    part[3] = fmaf(s[4 * c + 3], u4.w, part[3]);
                }
                float dot = (part[0] + part[1]) + (part[2] + part[3]);
#pragma unroll
                for (int w = 1; w < SCAN_LANES; w <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, w);
                const float v = sv[buf][tt][col];
                float op[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float4 a = a4[c * SCAN_LANES + p], rm = r4[c * SCAN_LANES + p], kw = w4[c * SCAN_LANES + p];
                    const float4 q = q4[c * SCAN_LANES + p];
                    s[4 * c + 0] = fmaf(kw.x, v, fmaf(-rm.x, dot, a.x * s[4 * c + 0]));
                    s[4 * c + 1] = fmaf(kw.y, v, fmaf(-rm.y, dot, a.y * s[4 * c + 1]));
                    s[4 * c + 2] = fmaf(kw.z, v, fmaf(-rm.z, dot, a.z * s[4 * c + 2]));
                    s[4 * c + 3] = fmaf(kw.w, v, fmaf(-rm.w, dot, a.w * s[4 * c + 3]));
                    op[0] = fmaf(s[4 * c + 0], q.x, op[0]);
                    op[1] = fmaf(s[4 * c + 1], q.y, op[1]);
                    op[2] = fmaf(s[4 * c + 2], q.z, op[2]);
                    op[3] = fmaf(s[4 * c + 3], q.w, op[3]);
                }
                so[tt][p * SCAN_COLS + col] = (op[0] + op[1]) + (op[2] + op[3]);
                return;
            }
            float4 kk[NC];
            float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float4 a = a4[c * SCAN_LANES + p];
                kk[c] = k4[c * SCAN_LANES + p];
                s[4 * c + 0] *= a.x; s[4 * c + 1] *= a.y; s[4 * c + 2] *= a.z; s[4 * c + 3] *= a.w;
                part[0] = fmaf(s[4 * c + 0], kk[c].x, part[0]);
                part[1] = fmaf(s[4 * c + 1], kk[c].y, part[1]);
                part[2] = fmaf(s[4 * c + 2], kk[c].z, part[2]);
                part[3] = fmaf(s[4 * c + 3], kk[c].w, part[3]);
            }
            float dot = (part[0] + part[1]) + (part[2] + part[3]);
#pragma unroll
            for (int w = 1; w < SCAN_LANES; w <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, w);
            const float u = sb[buf][tt] * (sv[buf][tt][col] - dot);
            float op[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float4 q = q4[c * SCAN_LANES + p];
                s[4 * c + 0] = fmaf(kk[c].x, u, s[4 * c + 0]);
                s[4 * c + 1] = fmaf(kk[c].y, u, s[4 * c + 1]);
                s[4 * c + 2] = fmaf(kk[c].z, u, s[4 * c + 2]);
                s[4 * c + 3] = fmaf(kk[c].w, u, s[4 * c + 3]);
                op[0] = fmaf(s[4 * c + 0], q.x, op[0]);
                op[1] = fmaf(s[4 * c + 1], q.y, op[1]);
                op[2] = fmaf(s[4 * c + 2], q.z, op[2]);
                op[3] = fmaf(s[4 * c + 3], q.w, op[3]);
            }
            so[tt][p * SCAN_COLS + col] = (op[0] + op[1]) + (op[2] + op[3]);      // summed over the lanes behind the loop
        };
        if (n == TT) {
#pragma unroll
            for (int tt = 0; tt < TT; ++tt) token(tt);
        } else {
            for (int tt = 0; tt < n; ++tt) token(tt);
        }
        __syncthreads();
        if (tid < n * SCAN_COLS) {                            // one thread a (token, column): the lanes' partial sums in lane order
            const int tt = tid / SCAN_COLS, c = tid % SCAN_COLS;
            const int jj = blockIdx.x * SCAN_COLS + c;
            float o = 0.f;
#pragma unroll
            for (int l = 0; l < SCAN_LANES; ++l) o += so[tt][l * SCAN_COLS + c];
            if (jj < E) out[((long long)(base + tt) * H + h) * E + jj] = o;
        }
        __syncthreads();                                  // this buffer is asked for again in the next round
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int d = ((i >> 2) * SCAN_LANES + p) * 4 + (i & 3);
        if (d < D && j < E) Sh[(long long)d * E + j] = s[i];
    }
}

// One warp a (token, head): o / rms(o) * w * gate(z), z the gate's sums: H * E columns of rows ``ldz`` apart, the sum
// of ``n_parts`` parts; gate: sigmoid(z), or (``silu_gate``) z * sigmoid(z).
template <typename TO>
__global__ void __launch_bounds__(128)
delta_finish_kernel(const float* __restrict__ o, const float* __restrict__ z, long long ldz, int n_parts, long long part_stride,
                    int silu_gate, const float* __restrict__ w, TO* __restrict__ out, int n_tokens, int H, int E, float eps,
                    int w_heads) {
    pdl_trigger();
    pdl_wait();
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= (long long)n_tokens * H) return;
    const long long t = wid / H;
    const int h = (int)(wid % H);
    const float* orow = o + (t * H + h) * E;
    float ss = 0.f;
    for (int e = lane; e < E; e += 32) { const float v = orow[e]; ss += v * v; }
    ss = warp_sum(ss);
    const float inv = inv_rms(ss, (float)E, eps);
    const float* zrow = z + t * ldz + (long long)h * E;
    if (w_heads) w += (long long)h * E;                   // a weight for every head instead of one shared by the heads
    for (int e = lane; e < E; e += 32) {
        float zv = 0.f;
        for (int i = 0; i < n_parts; ++i) zv += zrow[i * part_stride + e];
        const float g = silu_gate ? zv * sigmoidf_(zv) : sigmoidf_(zv);
        out[(t * H + h) * E + e] = from_f32<TO>(orow[e] * inv * w[e] * g);
    }
}

// The generalised delta rule's inputs, one warp a (token, head).  A projection row holds r, k, v (H heads of D) and the
// removal rate's sums at their columns; ``wpre`` [T, H * D] holds the decay's sums (the low-rank product's result).
//   u = k / sqrt(sum k^2 + unit_eps);  rem = sigmoid(a + a_bias) * u;  w = exp(-decay_scale * sigmoid(wpre + w0))
// r, u, raw k, rem, w and v go out as [T, H * D] float32 each, the scan's operands.
__global__ void __launch_bounds__(128)
gdelta_prepare_kernel(const float* __restrict__ p, long long ldp, int n_parts, long long part_stride, int r_off, int k_off,
                      int v_off, int a_off, const float* __restrict__ a_bias, const float* __restrict__ wpre,
                      const float* __restrict__ w0, float* __restrict__ rn, float* __restrict__ un, float* __restrict__ kraw,
                      float* __restrict__ rem, float* __restrict__ dec, float* __restrict__ vc, int n_tokens, int H, int D,
                      float unit_eps, float decay_scale) {
    pdl_trigger();
    pdl_wait();
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= (long long)n_tokens * H) return;
    const long long t = wid / H;
    const int h = (int)(wid % H);
    auto at = [&](int c) -> float {
        float v = 0.f;
        for (int i = 0; i < n_parts; ++i) v += p[i * part_stride + t * ldp + c];
        return v;
    };
    float kv[8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int d = lane + 32 * i;
        kv[i] = d < D ? at(k_off + h * D + d) : 0.f;
        ss += kv[i] * kv[i];
    }
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss + unit_eps);
    const long long base = (t * H + h) * D;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int d = lane + 32 * i;
        if (d >= D) continue;
        const int c = h * D + d;
        const float u = kv[i] * inv;
        un[base + d] = u;
        kraw[base + d] = kv[i];
        rem[base + d] = sigmoidf_(at(a_off + c) + a_bias[c]) * u;
        dec[base + d] = expf(-decay_scale * sigmoidf_(wpre[base + d] + w0[c]));
        rn[base + d] = at(r_off + c);
        vc[base + d] = at(v_off + c);
    }
}

UB_API int ub_gdelta_prepare(const float* p, long long ldp, int n_parts, long long part_stride, int r_off, int k_off, int v_off,
                             int a_off, const float* a_bias, const float* wpre, const float* w0, float* rn, float* un,
                             float* kraw, float* rem, float* dec, float* vc, int n_tokens, int H, int D, float unit_eps,
                             float decay_scale, cudaStream_t st) {
    if (n_tokens <= 0) return 0;
    if (H <= 0 || D <= 0 || D > 256 || n_parts < 1) return UB_ERR_ARG;
    const long long warps = (long long)n_tokens * H;
    return (int)ub_launch_dependent(gdelta_prepare_kernel, dim3((unsigned)((warps + 3) / 4)), dim3(128), 0, st, p, ldp, n_parts,
                                    part_stride, r_off, k_off, v_off, a_off, a_bias, wpre, w0, rn, un, kraw, rem, dec, vc,
                                    n_tokens, H, D, unit_eps, decay_scale);
}

// ---------------------------------------------------------------------------------------
// shape: [H, G, D, E, taps, q_off, k_off, v_off, b_off, a_off] (10 ints)
static int read_shape(const int* shape, long long ldp, int n_parts, long long part_stride, DeltaShape& s) {
    s.H = shape[0]; s.G = shape[1]; s.D = shape[2]; s.E = shape[3]; s.taps = shape[4];
    s.q_off = shape[5]; s.k_off = shape[6]; s.v_off = shape[7]; s.b_off = shape[8]; s.a_off = shape[9];
    s.ldp = ldp; s.n_parts = n_parts; s.part_stride = part_stride;
    if (s.H <= 0 || s.G <= 0 || s.H % s.G || s.D <= 0 || s.D > 256 || s.E <= 0 || s.taps < 1 || s.taps > MAX_TAPS ||
        s.H > 65535 || n_parts < 1) return UB_ERR_ARG;
    // the convolution's state is indexed by projection column: q, k, v are the row's first columns
    if (s.q_off != 0 || s.k_off != s.G * s.D || s.v_off != 2 * s.G * s.D) return UB_ERR_ARG;
    return 0;
}

UB_API int ub_delta_prepare(const float* p, long long ldp, int n_parts, long long part_stride, const int* shape,
                            const float* conv_w, float* conv_state, int update_state, const float* dpre,
                            const float* dt_bias, const float* a_log, const int* tok_seq,
                            const int* seq_start, const int* seq_slot, float* qn, float* kn, float* vc, float* beta,
                            float* dec, int n_tokens, float unit_eps, float q_scale, cudaStream_t st) {
    if (n_tokens <= 0) return 0;
    DeltaShape s;
    if (int rc = read_shape(shape, ldp, n_parts, part_stride, s)) return rc;
    auto aligned = [](const void* a) { return ((uintptr_t)a & 15) == 0; };
    if ((s.D == 64 || s.D == 128) && (s.E == 64 || s.E == 128) && s.taps <= 4 && ldp % 4 == 0 && part_stride % 4 == 0 &&
        aligned(p) && aligned(conv_state) && aligned(dpre) && aligned(dt_bias) && aligned(qn) && aligned(kn) && aligned(vc) && aligned(dec)) {
        // few tokens: a warp each, so that the chip has warps to run
        const int walk = n_tokens <= 256 ? 1 : WALK;
        const long long w = (long long)((n_tokens + walk - 1) / walk) * (2 * s.G + 2 * s.H);
        auto kern = s.D == 128 ? (s.E == 128 ? delta_prepare_rows_kernel<4, 4> : delta_prepare_rows_kernel<4, 2>)
                               : (s.E == 128 ? delta_prepare_rows_kernel<2, 4> : delta_prepare_rows_kernel<2, 2>);
        return (int)ub_launch_dependent(kern, dim3((unsigned)((w + 3) / 4)), dim3(128), 0, st, p, s, conv_w, conv_state, update_state,
                                        dpre, dt_bias, a_log, tok_seq, seq_start, seq_slot, qn, kn, vc, beta, dec, n_tokens, walk,
                                        unit_eps, q_scale);
    }
    const long long warps = (long long)n_tokens * (2 * s.G + s.H);
    const unsigned grid = (unsigned)((warps + 3) / 4);
    return (int)ub_launch_dependent(delta_prepare_kernel, dim3(grid), dim3(128), 0, st, p, s, conv_w, conv_state, update_state, dpre, dt_bias,
                                    a_log, tok_seq, seq_start, seq_slot, qn, kn, vc, beta, dec, n_tokens, unit_eps, q_scale);
}

UB_API int ub_conv_state_update(const float* p, long long ldp, int n_parts, long long part_stride, float* conv_state,
                                const int* seq_start, const int* seq_slot, int n_seqs, int C, int taps, cudaStream_t st) {
    if (n_seqs <= 0 || taps <= 1) return 0;
    if (taps > MAX_TAPS || n_parts < 1) return UB_ERR_ARG;
    DeltaShape s = {};
    s.ldp = ldp; s.n_parts = n_parts; s.part_stride = part_stride;
    const long long n = (long long)n_seqs * C;
    return (int)ub_launch_dependent(conv_state_update_kernel, dim3((unsigned)((n + 127) / 128)), dim3(128), 0, st, p, s,
                                    conv_state, seq_start, seq_slot, n_seqs, C, taps);
}

// below: sequences of that many tokens and more are left alone (0: none; with sizes that delta_scan_pairs_kernel takes only).
UB_API int ub_delta_scan(const float* qn, const float* kn, const float* vc, const float* beta, const float* dec, float* out,
                         float* S, const int* seq_start, const int* seq_slot, int n_seqs, int n_tokens, int H, int G, int D,
                         int E, int sm_count, const float* rem, const float* kraw, int below, cudaStream_t st) {
    if (n_seqs <= 0) return 0;
    const bool gen = rem != nullptr;
    if (gen != (kraw != nullptr)) return UB_ERR_ARG;
    if (H <= 0 || G <= 0 || H % G || D <= 0 || D > 256 || E <= 0 || H > 65535 || n_seqs > 65535) return UB_ERR_ARG;
    const bool vec = D % 4 == 0 && E % 4 == 0 &&
        (((uintptr_t)qn | (uintptr_t)kn | (uintptr_t)vc | (uintptr_t)dec | (uintptr_t)rem | (uintptr_t)kraw) & 15) == 0;
    const bool dep = n_tokens <= n_seqs;                   // (see below)
    if (vec && !gen && (D == 64 || D == 128) && E % 16 == 0) {
        const dim3 pg(E / 16, H, n_seqs);
        auto kern = D == 64 ? delta_scan_pairs_kernel<64> : delta_scan_pairs_kernel<128>;
        return (int)ub_launch_ordered(dep, kern, pg, dim3(128), 0, st, qn, kn, vc, beta, dec, out, S, seq_start, seq_slot, H, G, E, below > 0 ? below : 0x7fffffff);
    }
    if (below > 0) return UB_ERR_ARG;                      // (sizes that only this kernel takes)
    // lanes a column: eight, and more (fewer values and a shorter chain a thread) only while the launch still has
    // no more than about one warp for every scheduler and every lane gets a whole float4 chunk; measured at 2,048
    // tokens, 16 heads, sizes of 128: 346 / 372 / 405 ns a token with 8 / 16 / 32 lanes, at sizes of 64: 322 / 296
    static const int forced = getenv("ULTIMA_SCAN_LANES") ? atoi(getenv("ULTIMA_SCAN_LANES")) : 0;    // for measurements
    const long long budget = 4LL * (sm_count > 0 ? sm_count : 148);
    auto warps_with = [&](int l) { return (long long)n_seqs * H * ((E * l + 127) / 128) * 4; };
    int lanes = 8;
    while (lanes < 32 && lanes * 2 * 4 <= ((D + 3) / 4) * 4 && warps_with(lanes * 2) <= budget) lanes <<= 1;
    if (forced == 8 || forced == 16 || forced == 32) lanes = forced;
    while (lanes > 8 && lanes * 4 > ((D + 3) / 4) * 4) lanes >>= 1;
    const int cols = 128 / lanes;
    const dim3 grid((E + cols - 1) / cols, H, n_seqs), block(128);
    const int per_lane = (D + lanes - 1) / lanes;          // key channels a lane, rounded up to whole chunks
    const int R = per_lane <= 4 ? 4 : per_lane <= 8 ? 8 : per_lane <= 16 ? 16 : 32;
    cudaError_t e = cudaErrorInvalidValue;
    // A step that brings more than one token a sequence starts as an ordinary launch, behind the end of the kernels before
    // it.  As a programmatic dependent its few CTAs (one for an SM or fewer, each busy for the whole step) are placed while
    // the kernel before drains, on the SMs that happen to have room first, several to an SM: measured, a prompt of 2,048
    // tokens with four such layers took 8.2 ms so and 6.6 ms with every CTA on an SM of its own.
#define GO2(RR, LL, VV, GG) ub_launch_ordered(dep, delta_scan_kernel<RR, LL, VV, GG>, grid, block, 0, st, qn, kn, vc, beta, dec, out, S, seq_start, seq_slot, H, G, D, E, rem, kraw)
#define GO(RR, LL) e = gen ? (vec ? GO2(RR, LL, true, true) : GO2(RR, LL, false, true)) : (vec ? GO2(RR, LL, true, false) : GO2(RR, LL, false, false))
    if (lanes == 32) { if (R == 4) GO(4, 32); else if (R == 8) GO(8, 32); else return UB_ERR_ARG; }
    else if (lanes == 16) { if (R == 4) GO(4, 16); else if (R == 8) GO(8, 16); else if (R == 16) GO(16, 16); else return UB_ERR_ARG; }
    else { if (R == 4) GO(4, 8); else if (R == 8) GO(8, 8); else if (R == 16) GO(16, 8); else GO(32, 8); }
#undef GO
#undef GO2
    return (int)e;
}

// The recurrence four tokens at a time (see delta_records_kernel); ``rec``: scratch, ((n_tokens + 3 n_seqs) / 4 + 1) * H
// records (9 n_tokens / 32 * H from min_new 32 on); max_new: the longest sequence's tokens; sequences with fewer than min_new
// or, with below > 0, with below or more are left alone.
UB_API int ub_delta_scan_records(const float* qn, const float* kn, const float* vc, const float* beta, const float* dec, float* out,
                                 float* S, float* rec, const int* seq_start, const int* seq_slot, int n_seqs, int n_tokens, int max_new,
                                 int min_new, int below, int H, int G, int D, int E, cudaStream_t st) {
    if (n_seqs <= 0 || n_tokens <= 0 || max_new <= 0) return 0;
    if (below <= 0) below = 0x7fffffff;
    if (min_new < 1 || H <= 0 || G <= 0 || H % G || (D != 64 && D != 128) || E <= 0 || E % 16 || H > 65535 || n_seqs > 65535) return UB_ERR_ARG;
    if (((uintptr_t)qn | (uintptr_t)kn | (uintptr_t)dec | (uintptr_t)rec | (uintptr_t)vc) & 15) return UB_ERR_ARG;
    const long long warps = (long long)((min(max_new, below) + 3) / 4) * H;
    const dim3 rg((unsigned)((warps + 3) / 4), n_seqs), sg(E / 16, H, n_seqs);
    cudaError_t e = D == 64 ? ub_launch_dependent(delta_records_kernel<64>, rg, dim3(128), 0, st, qn, kn, beta, dec, rec, seq_start, H, G, min_new, below)
                            : ub_launch_dependent(delta_records_kernel<128>, rg, dim3(128), 0, st, qn, kn, beta, dec, rec, seq_start, H, G, min_new, below);
    if (e != cudaSuccess) return (int)e;
    // (an ordinary launch, as the scan above for prompts: see there)
    const size_t smem = DELTA_RECORD_BUFS * sizeof(float) * (13 * D + 32 + 64);
    e = D == 64 ? ub_launch_ordered(false, delta_scan_records_kernel<64>, sg, dim3(128), smem, st, rec, vc, out, S, seq_start, seq_slot, H, E, min_new, below)
                : ub_launch_ordered(false, delta_scan_records_kernel<128>, sg, dim3(128), smem, st, rec, vc, out, S, seq_start, seq_slot, H, E, min_new, below);
    return (int)e;
}

// A portion of the recurrence sixteen tokens at a time (see delta_chunks_kernel, DeltaPortion): n_seqs sequences from ``seq`` on, of those
// that bring min_new tokens or more the tokens from ``first`` on, at most ``most`` records of sixteen each.  ``rec``: scratch of rec_floats numbers, H (73 D + 36 E) a
// record; max_new: the longest sequence's tokens.  ``error`` (or null) is raised when a wait ran out of time or the scratch is too small.
UB_API int ub_delta_scan_chunks(const float* qn, const float* kn, const float* vc, const float* beta, const float* dec, float* out,
                                 float* S, float* rec, long long rec_floats, const int* seq_start, const int* seq_slot, int seq,
                                 int n_seqs, int max_new, int min_new, int first, int most, int H, int G, int D, int E, int* error,
                                 cudaStream_t st) {
    if (n_seqs <= 0 || max_new <= first) return 0;
    if (min_new < 1 || H <= 0 || G <= 0 || H % G || (D != 64 && D != 128) || E <= 0 || E % 16 || H > 65535 || n_seqs > 65535) return UB_ERR_ARG;
    if (((uintptr_t)qn | (uintptr_t)kn | (uintptr_t)dec | (uintptr_t)rec | (uintptr_t)vc) & 15) return UB_ERR_ARG;
    const long long places = rec_floats / (H * (D == 64 ? DeltaChunk<64>::floats(E) : DeltaChunk<128>::floats(E)));
    if (seq < 0 || first < 0 || first % DELTA_CHUNK || most < 1 || places < 1) return UB_ERR_ARG;
    most = min(most, (max_new - first + DELTA_CHUNK - 1) / DELTA_CHUNK);
    const long long records = (long long)most * H;
    if (records > 0x7fffffffll) return UB_ERR_ARG;
    const DeltaPortion po{seq, first, most, min_new, places};
    const dim3 rg((unsigned)records, n_seqs), sg(E / 16, H, n_seqs);
    cudaError_t e = D == 64 ? ub_launch_dependent(delta_chunks_kernel<64>, rg, dim3(32), 0, st, qn, kn, vc, beta, dec, rec, seq_start, H, G, E, po, error)
                            : ub_launch_dependent(delta_chunks_kernel<128>, rg, dim3(64), 0, st, qn, kn, vc, beta, dec, rec, seq_start, H, G, E, po, error);
    if (e != cudaSuccess) return (int)e;
    static UbAllowSmem allow64, allow128;
    const int smem = D == 64 ? delta_scan_smem<64>() : delta_scan_smem<128>();
    e = D == 64 ? allow64(delta_scan_chunks_kernel<64>, smem) : allow128(delta_scan_chunks_kernel<128>, smem);
    if (e != cudaSuccess) return (int)e;
    // (an ordinary launch, as the scan above for prompts: see there)
    e = D == 64 ? ub_launch_ordered(false, delta_scan_chunks_kernel<64>, sg, dim3(DELTA_SCAN_THREADS), smem, st, rec, out, S, seq_start, seq_slot, H, E, po, error)
                : ub_launch_ordered(false, delta_scan_chunks_kernel<128>, sg, dim3(DELTA_SCAN_THREADS), smem, st, rec, out, S, seq_start, seq_slot, H, E, po, error);
    return (int)e;
}

UB_API int ub_delta_finish(const float* o, const float* z, long long ldz, int n_parts, long long part_stride, int silu_gate,
                           const float* w, void* out, int out_dtype, int n_tokens, int H, int E, float eps, int w_heads,
                           cudaStream_t st) {
    if (n_tokens <= 0) return 0;
    if (n_parts < 1) return UB_ERR_ARG;
    const long long warps = (long long)n_tokens * H;
    const unsigned grid = (unsigned)((warps + 3) / 4);
    cudaError_t e;
    if (out_dtype == UB_F32)
        e = ub_launch_dependent(delta_finish_kernel<float>, dim3(grid), dim3(128), 0, st, o, z, ldz, n_parts, part_stride, silu_gate, w, (float*)out, n_tokens, H, E, eps, w_heads);
    else if (out_dtype == UB_BF16)
        e = ub_launch_dependent(delta_finish_kernel<__nv_bfloat16>, dim3(grid), dim3(128), 0, st, o, z, ldz, n_parts, part_stride, silu_gate, w, (__nv_bfloat16*)out, n_tokens, H, E, eps, w_heads);
    else return UB_ERR_UNSUPPORTED;
    return (int)e;
}
