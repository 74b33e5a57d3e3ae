// Attention in float32 throughout, over the paged float32 cache (pages of 64 positions): softmax(q k * scale) v, causal, with an
// optional window, for head sizes 64 and 128.  Further options and other sizes are attn_simple.cu's.
//
// A block takes up to BR rows, a row being one token and one query head of a key head's group, so that a page of keys and values is
// fetched once for all of them.  Scores of a page on the FMA units from shared memory (keys and queries 16 bytes at a time),
// the running maximum and sum a row, then the weighted values.
//
// The order of a row's sums depends on the key range alone: a page of 64 positions (counted from the sequence's start) has a
// maximum and sums of its own, and pages are merged in their order.  So prompts (a block walks the pages of its rows) and
// single tokens (pages shared out over blocks, the merge in a kernel of its own) give the same bits, however a sequence was
// cut into steps.
//
// It restates the reference's per-token loop (src/model/qwen_block.cpp:94-135), as attn_simple.cu does.  What bounds it: a
// prompt's FMAs; with one token a sequence, the latency of a page's fetch and two passes (about 6 us), which is why pages are
// shared out until the chip is full (four sequences at 340 positions, 16 heads on 4: 162 us with attn_simple.cu, 27 us with
// four pages in a row a block, 13 and 3 us for the merge so).
#include <type_traits>
#include "common.cuh"

constexpr int PG = 64;                       // keys a page

struct AttnF32 {
    const float* q; long long ldq;
    const float* kc; const float* vc;
    float* out; long long ldo;
    const int* seq_start; const int* seq_before; const int* table;
    int pages_per_seq, ring, nh, nkv, window;
    float scale;
    float* part;              // split: [token, head, place][HD + 2]: weighted values, maximum, sum
    int places;               // split: pages the scratch holds a row (page g in place g % places): as many as a sequence's
                              // tokens of the step see together
    int z;                    // split: blocks that share a row's pages
};

template <int BR, int HD> struct AttnSmem {
    static constexpr int LD = HD + 4, LDP = PG + 4;
    static constexpr int FLOATS = (BR + 2 * PG) * LD + BR * LDP;
    static constexpr int TOTAL = FLOATS * 4;
};

// m, l, acc <- the merge of (m, l, acc) with a later page's (sm, sl, sacc)
template <int N>
__device__ __forceinline__ void merge_page(float& m, float& l, float* acc, float sm, float sl, const float* sacc) {
    if (sm == -INFINITY && sl == 0.f) return;                // nothing visible in the page
    const float mn = fmaxf(m, sm);
    const float a = m == -INFINITY ? 0.f : expf(m - mn), b = expf(sm - mn);
    l = fmaf(l, a, sl * b);
#pragma unroll
    for (int c = 0; c < N; ++c) acc[c] = fmaf(acc[c], a, sacc[c] * b);
    m = mn;
}

template <int BR, int HD, bool SPLIT>
__global__ void __launch_bounds__(256)
attn_f32_kernel(AttnF32 p) {
    using S = AttnSmem<BR, HD>;
    extern __shared__ __align__(16) float attn_smem[];
    float* sq = attn_smem;                                   // [BR][LD]
    float* sk = sq + BR * S::LD;                             // [PG][LD]
    float* sv = sk + PG * S::LD;                             // [PG][LD]
    float* sp = sv + PG * S::LD;                             // [BR][LDP]: a page's weights
    constexpr int RT = BR / 16;                              // rows a thread: ty + 16 i
    constexpr int KT = PG / 16;                              // keys a thread: tx + 16 j
    constexpr int CT = HD / 16;                              // output columns a thread: 4 tx + 64 c ...
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;                  // a row's sixteen threads are half a warp
    pdl_trigger();
    pdl_wait();
    const int step = SPLIT ? p.z : 1;
    const int seq = blockIdx.z / step;
    const int kvh = blockIdx.y, group = p.nh / p.nkv;
    const int t_first = p.seq_start[seq], n_new = p.seq_start[seq + 1] - t_first, before = p.seq_before[seq];
    const int n_rows = n_new * group;
    const int r0 = blockIdx.x * BR;
    if (r0 >= n_rows) return;
    const int last_row = min(r0 + BR, n_rows) - 1;
    const int pos_lo = before + r0 / group, pos_hi = before + last_row / group;
    const int key_lo = p.window > 0 ? max(0, pos_lo - p.window + 1) : 0;
    const int page_end = pos_hi / PG + 1;
    int page = key_lo / PG + blockIdx.z % step;
    if (page >= page_end) return;
    int my_pos[RT], my_lo[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int my = r0 + ty + 16 * i;
        my_pos[i] = my < n_rows ? before + my / group : -1;
        my_lo[i] = p.window > 0 ? max(0, my_pos[i] - p.window + 1) : 0;
    }
    // keys and values outside the block's range are zero in shared memory: what a page holds there may be anything
    auto load_page = [&](const float* cache, float* dst, int pg) {
        const int li = (pg * PG) % p.ring;
        const float* src = cache + ((long long)p.table[(long long)seq * p.pages_per_seq + li / PG] * p.nkv + kvh) * PG * HD;
#pragma unroll
        for (int i = 0; i < PG * HD / 4 / 256; ++i) {
            const int e = tid + i * 256, key = e / (HD / 4), c = (e % (HD / 4)) * 4;
            const int pos = pg * PG + key;
            cp16(dst + key * S::LD + c, src + key * HD + c, pos >= key_lo && pos <= pos_hi);
        }
        cp_commit();
    };
    for (int e = tid; e < BR * HD / 4; e += 256) {
        const int r = e / (HD / 4), c = (e % (HD / 4)) * 4, gr = r0 + r;
        const bool ok = gr < n_rows;
        cp16(sq + r * S::LD + c, p.q + (ok ? (long long)(t_first + gr / group) * p.ldq + (long long)(kvh * group + gr % group) * HD + c : 0), ok);
    }
    load_page(p.kc, sk, page);                               // (one group with the queries)
    load_page(p.vc, sv, page);
    float m[RT], l[RT], acc[SPLIT ? 1 : RT][CT];             // a row's sums over the pages so far
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
        if constexpr (!SPLIT) {
#pragma unroll
            for (int c = 0; c < CT; ++c) acc[i][c] = 0.f;
        }
    }
    for (; page < page_end; page += step) {
        cp_wait<1>();                                        // the page's keys
        __syncthreads();
        float s[RT][KT], sm[RT], sl[RT], sacc[RT][CT];       // the page's scores, maxima, sums
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int j = 0; j < KT; ++j) s[i][j] = 0.f;
#pragma unroll 4
        for (int d = 0; d < HD; d += 4) {
            float4 qv[RT];
#pragma unroll
            for (int i = 0; i < RT; ++i) qv[i] = *reinterpret_cast<const float4*>(sq + (ty + 16 * i) * S::LD + d);
#pragma unroll
            for (int j = 0; j < KT; ++j) {
                const float4 kv = *reinterpret_cast<const float4*>(sk + (tx + 16 * j) * S::LD + d);
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    s[i][j] = fmaf(qv[i].x, kv.x, s[i][j]);
                    s[i][j] = fmaf(qv[i].y, kv.y, s[i][j]);
                    s[i][j] = fmaf(qv[i].z, kv.z, s[i][j]);
                    s[i][j] = fmaf(qv[i].w, kv.w, s[i][j]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < KT; ++j) {
                const int pos = page * PG + tx + 16 * j;
                s[i][j] = pos <= my_pos[i] && pos >= my_lo[i] ? s[i][j] * p.scale : -INFINITY;
                mx = fmaxf(mx, s[i][j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            float ps = 0.f;
#pragma unroll
            for (int j = 0; j < KT; ++j) {
                // (the maximum passes over NaN: where every visible score of the page is one, the weights carry it)
                const float w = mx == -INFINITY ? (s[i][j] == -INFINITY ? 0.f : s[i][j]) : expf(s[i][j] - mx);
                sp[(ty + 16 * i) * S::LDP + tx + 16 * j] = w;
                ps += w;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
            sl[i] = ps;
            sm[i] = mx;
#pragma unroll
            for (int c = 0; c < CT; ++c) sacc[i][c] = 0.f;
        }
        __syncthreads();                                     // the keys are read: the next page's may come
        if (page + step < page_end) load_page(p.kc, sk, page + step);
        else cp_commit();
        cp_wait<1>();                                        // the page's values
        __syncthreads();
        auto add_values = [&](auto edge) {
            constexpr int UNROLL = decltype(edge)::value ? 1 : 4;
#pragma unroll UNROLL
            for (int k = 0; k < PG; k += 4) {
                float4 w[RT];
#pragma unroll
                for (int i = 0; i < RT; ++i) w[i] = *reinterpret_cast<const float4*>(sp + (ty + 16 * i) * S::LDP + k);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                    for (int c = 0; c < CT; c += 4) {
                        const float4 v = *reinterpret_cast<const float4*>(sv + (k + kk) * S::LD + tx * 4 + c * 16);
#pragma unroll
                        for (int i = 0; i < RT; ++i) {
                            const int pos = page * PG + k + kk;
                            if (decltype(edge)::value && (pos > my_pos[i] || pos < my_lo[i])) continue;
                            const float wk = kk == 0 ? w[i].x : kk == 1 ? w[i].y : kk == 2 ? w[i].z : w[i].w;
                            sacc[i][c] = fmaf(wk, v.x, sacc[i][c]);
                            sacc[i][c + 1] = fmaf(wk, v.y, sacc[i][c + 1]);
                            sacc[i][c + 2] = fmaf(wk, v.z, sacc[i][c + 2]);
                            sacc[i][c + 3] = fmaf(wk, v.w, sacc[i][c + 3]);
                        }
                    }
            }
        };
        // where the page holds keys that some row of the block does not see, such a row leaves their values out: a weight of zero would
        // bring it another token's infinity or NaN
        const bool edge = pos_lo != pos_hi && (min(page * PG + PG - 1, pos_hi) > pos_lo || (p.window > 0 && page * PG <= pos_hi - p.window));
        if (edge) add_values(std::true_type{});
        else add_values(std::false_type{});
        __syncthreads();                                     // values and weights are read
        if (page + step < page_end) load_page(p.vc, sv, page + step);
        else cp_commit();
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            if constexpr (SPLIT) {
                if (my_pos[i] < 0) continue;
                const int my = r0 + ty + 16 * i;
                float* o = p.part + (((long long)(t_first + my / group) * p.nh + kvh * group + my % group) * p.places + page % p.places) * (HD + 2);
#pragma unroll
                for (int c = 0; c < CT; ++c) o[tx * 4 + (c / 4) * 64 + c % 4] = sacc[i][c];
                if (tx == 0) { o[HD] = sm[i]; o[HD + 1] = sl[i]; }
            } else {
                merge_page<CT>(m[i], l[i], acc[i], sm[i], sl[i], sacc[i]);
            }
        }
    }
    if constexpr (!SPLIT) {
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            if (my_pos[i] < 0) continue;
            const int my = r0 + ty + 16 * i;
            const float inv = 1.0f / l[i];
            float* o = p.out + (long long)(t_first + my / group) * p.ldo + (long long)(kvh * group + my % group) * HD;
#pragma unroll
            for (int c = 0; c < CT; c += 4)
                *reinterpret_cast<float4*>(o + tx * 4 + c * 16) =
                    make_float4(acc[i][c] * inv, acc[i][c + 1] * inv, acc[i][c + 2] * inv, acc[i][c + 3] * inv);
        }
    }
}

// The merge of a row's pages: one warp a (token, head), eight pages asked for at a time.
template <int HD>
__global__ void __launch_bounds__(128)
attn_f32_merge_kernel(AttnF32 p, const int* __restrict__ tok_pos, int n_tokens) {
    pdl_trigger();
    pdl_wait();
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= (long long)n_tokens * p.nh) return;
    const long long t = wid / p.nh;
    const int head = (int)(wid % p.nh);
    const int pos = tok_pos[t], lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
    constexpr int CT = HD / 32;
    float m = -INFINITY, l = 0.f, acc[CT];
#pragma unroll
    for (int c = 0; c < CT; ++c) acc[c] = 0.f;
    const int end = pos / PG + 1;
    for (int g0 = lo / PG; g0 < end; g0 += 8) {
        float sm[8], sl[8], sacc[8][CT];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float* o = p.part + (wid * p.places + min(g0 + i, end - 1) % p.places) * (HD + 2);
            sm[i] = g0 + i < end ? o[HD] : -INFINITY;
            sl[i] = g0 + i < end ? o[HD + 1] : 0.f;
#pragma unroll
            for (int c = 0; c < CT; ++c) sacc[i][c] = o[lane + 32 * c];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) merge_page<CT>(m, l, acc, sm[i], sl[i], sacc[i]);
    }
    const float inv = 1.0f / l;
    float* o = p.out + t * p.ldo + (long long)head * HD;
#pragma unroll
    for (int c = 0; c < CT; ++c) o[lane + 32 * c] = acc[c] * inv;
}

template <int BR, int HD, bool SPLIT>
static int launch(const AttnF32& p, int n_seqs, int max_new, cudaStream_t st) {
    auto kern = attn_f32_kernel<BR, HD, SPLIT>;
    constexpr int smem = AttnSmem<BR, HD>::TOTAL;
    static UbAllowSmem allow;
    if (cudaError_t e = allow(kern, smem)) return (int)e;
    const int group = p.nh / p.nkv;
    const long long z = SPLIT ? (long long)n_seqs * p.z : n_seqs;
    dim3 grid((unsigned)(((long long)max_new * group + BR - 1) / BR), p.nkv, (unsigned)z);
    if (grid.y > 65535 || z > 65535) return UB_ERR_ARG;
    return (int)ub_launch_dependent(kern, grid, dim3(256), smem, st, p);
}

template <int HD>
static int go(const AttnF32& p, int n_seqs, int max_new, int n_tokens, const int* tok_pos, cudaStream_t st) {
    const bool few = (long long)max_new * (p.nh / p.nkv) <= 16;
    if (!p.part) return few ? launch<16, HD, false>(p, n_seqs, max_new, st) : launch<64, HD, false>(p, n_seqs, max_new, st);
    const int rc = few ? launch<16, HD, true>(p, n_seqs, max_new, st) : launch<64, HD, true>(p, n_seqs, max_new, st);
    if (rc) return rc;
    const long long warps = (long long)n_tokens * p.nh;
    return (int)ub_launch_dependent(attn_f32_merge_kernel<HD>, dim3((unsigned)((warps + 3) / 4)), dim3(128), 0, st, p, tok_pos, n_tokens);
}

// q: [T, *] float32, heads side by side, row stride ldq; out likewise; caches [pages, kv heads, 64, head size].  ``part`` (float32
// [T, heads, places, head size + 2] or null): scratch for the pages' sums, at least as many places as pages that a sequence's
// tokens of the step see together; ``z`` blocks share a row's pages then.
UB_API int ub_attn_f32(const void* q, long long ldq, const void* kc, const void* vc, void* out, long long ldo, const int* seq_start,
                       const int* seq_before, const int* tok_pos, const int* table, int pages_per_seq, int ring, int n_seqs, int max_new,
                       int n_tokens, int nh, int nkv, int hd, int window, float scale, void* part, int places, int z, cudaStream_t st) {
    if (n_tokens <= 0 || n_seqs <= 0 || max_new <= 0) return 0;
    if (nkv <= 0 || nh % nkv || ring <= 0 || ring % PG || ldq % 4 || ldo % 4 || ((uintptr_t)q & 15) || ((uintptr_t)out & 15)) return UB_ERR_ARG;
    if (((uintptr_t)kc & 15) || ((uintptr_t)vc & 15) || (part && (places <= 0 || z <= 0))) return UB_ERR_ARG;
    AttnF32 p{(const float*)q, ldq, (const float*)kc, (const float*)vc, (float*)out, ldo, seq_start, seq_before, table, pages_per_seq,
              ring, nh, nkv, window, scale, (float*)part, places, z};
    if (hd == 64) return go<64>(p, n_seqs, max_new, n_tokens, tok_pos, st);
    if (hd == 128) return go<128>(p, n_seqs, max_new, n_tokens, tok_pos, st);
    return UB_ERR_ARG;
}
