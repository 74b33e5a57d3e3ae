// Matrix product of float32 operands on the tensor cores: out[t, n] = sum_k A[t, k] * W[n, k], for any number of tokens.  Many are
// taken by tcgen05.mma (below), few by mma.sync (further down), with the same bits.
//
// The tensor cores have no float32 product, but a float32 number is the exact sum of three bfloat16 numbers, x = h + m + l (h is x rounded,
// m what is left rounded, l the rest: 8 + 8 + 8 significant bits), and a product of two bfloat16 numbers is exact in float32.  (The parts of
// a number below 2^-110 would reach below the smallest bfloat16, 2^-133: operands are multiplied by 2^24 ahead of the split, so that
// every part of every float32 is a normal number, and sums by 2^-48 behind it, which changes no other bit.)  So
//   x y = h h' + (h m' + m h') + (h l' + m m' + l h') + (m l' + l m' + l l'),
// (a published method: Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial intelligence datatype for higher-precision computations",
// 2019), of which the last three are below 2^-26 of x y and are left out.  What remains is rounding while products are added, so tensor
// memory never holds a long sum: a block of 64 terms of K is summed from zero, the small products first (their sums are then too small
// for their rounding to matter), and the blocks are added in order by ordinary float32 additions in registers.  K is cut into up
// to four slices of whole blocks, a chain each, which are added in their order: the order of an output's sum depends on K alone.
// A sum that comes out infinite or NaN is formed again with float32 FMA: an infinite operand, or one of 2^104 or more, has no such parts.
//
// The tokens' parts are made once, by a kernel of their own, and copied by TMA for each of the weight tiles; the weights pass a CTA once a
// 128 tokens and are split where they are needed (their planes would be half as large again as they are).
//
// One CTA takes 128 weight rows (the gate product: 64 of each matrix) and 128 tokens.  Warps 0-7 load the weights' next block of 64
// columns, two blocks ahead, split it and write the three bfloat16 planes to shared memory (128-byte swizzle, two stages).  Warps 8-15 add
// finished blocks to their sums (three buffers in tensor memory), and in turn one of them issues the 24 MMAs of the next block: an issuing
// warp stands for as long as the block before it is multiplied, and with three buffers its share of the sums may come that much later.
// (One warp that issued all blocks left the tensor cores idle for 1,000 of 2,500 cycles a block; a warp of its own would make
// seventeen and leave each 96 registers for 128.)  Where the tiles are too few for the chip a cluster of four CTAs takes a
// tile, a slice of K each, and the slices meet through distributed shared memory: same bits.
//
// What bounds it: shared memory, 1.2 us (2,250 cycles) a block, of which the MMAs' operands are 1,540 cycles (as long as the MMAs
// themselves take) and the planes' way in 770.  With one issuing lane and both operands split by the loading warps it was 1.65 us.
// Against the forms of gemm_f32.cu, inputs not in the L2: 780 tokens, N 6,144, K 2,048: 609 -> 132 us (149 TFLOP/s; 190 at 1.65 us a
// block); N 2,048, K 6,144: 569 -> 125 (185); 200 tokens, N 2,048, K 2,048: 74 -> 23 (29).  The relative error
// against 64 bits (2-norm, normal inputs): K 1,024 9.7e-8 for 2.1e-7; K 2,048 1.0e-7 for 2.9e-7; K 6,144 1.3e-7 for 5.0e-7.
#include <cooperative_groups.h>
#include <float.h>
#include "common.cuh"
#include "tc_common.cuh"

namespace cg = cooperative_groups;

enum : int { EPI_STORE = 0, EPI_ADD = 1, EPI_SWIGLU = 2 };

constexpr int BM = 128;                      // weight rows a tile (MMA M)
constexpr int BN = 128;                      // tokens a tile (MMA N, or fewer in the last one)
constexpr int BK = 64;                       // terms a block: 128 bytes of bfloat16
constexpr int SLICES = 4;
constexpr int PLANE = 128 * BK * 2;          // bytes of one plane of one operand's block
constexpr int STAGE = 6 * PLANE;             // h, m, l of the weights, then of the tokens
constexpr int STAGES = 2;
constexpr int SMEM = STAGES * STAGE + 1024 + 256;
constexpr int THREADS = 512;
constexpr int ACCS = 3;                      // buffers in tensor memory
constexpr int TOTAL_COL = ACCS * BN;         // columns of tensor memory in which the slices before are kept
constexpr int TMEM_COLS = 512;
constexpr float SCALE_IN = 0x1p24f, SCALE_OUT = 0x1p-48f;

struct F32TcParams {
    const float* a; const float* w; const float* w2; float* out;
    int M, N, K;
    long long lda, ldw, ldo;
    int* error;
};

// The sum again with float32 FMA (slices and order as in gemm_f32.cu).
__device__ __noinline__ float plain_sum(const float* a, const float* w, int K) {
    const int len = max(64, ((K + 7) / 8 + 31) / 32 * 32);
    float total = 0.f;
    for (int k0 = 0; k0 < K; k0 += len) {
        float s = 0.f;
        for (int k = k0; k < min(K, k0 + len); ++k) s = fmaf(a[k], w[k], s);
        total += s;
    }
    return total;
}

// A sum as it came out of the tensor cores, or again with FMA.
__device__ __forceinline__ float result(float s, const float* a, const float* w, int K) {
    return fabsf(s) <= FLT_MAX ? s * SCALE_OUT : plain_sum(a, w, K);
}

// Four numbers times SCALE_IN, two at a time (one at a time the loading warps hold the MMAs up: 681 tokens 1 % slower).
__device__ __forceinline__ float4 scaled(float4 v) {
    float4 r;
    asm("{\n\t.reg .b64 a, b, s;\n\tmov.b64 a, {%4, %5};\n\tmov.b64 b, {%6, %7};\n\tmov.b64 s, {%8, %8};\n\t"
        "mul.rn.f32x2 a, a, s;\n\tmul.rn.f32x2 b, b, s;\n\tmov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
        : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "f"(SCALE_IN));
    return r;
}

// Two scaled numbers' three parts, each two bfloat16 in a register (the differences two numbers at a time).
__device__ __forceinline__ void split2(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
    auto pack = [](uint64_t v) {
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
        __nv_bfloat162 r = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<uint32_t*>(&r);
    };
    auto pair = [](uint32_t a, uint32_t b) { uint64_t v; asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(a), "r"(b)); return v; };
    auto less = [&](uint64_t v, uint32_t part) {             // v - part
        uint64_t d;
        const uint32_t one = __float_as_uint(-1.f);
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(pair(part << 16, part & 0xFFFF0000u)), "l"(pair(one, one)), "l"(v));
        return d;
    };
    uint64_t v = pair(__float_as_uint(x), __float_as_uint(y));
    h = pack(v);
    v = less(v, h);
    m = pack(v);
    l = pack(less(v, m));
}

// Four numbers of a row into the three planes at ``dst`` (the planes lie PLANE bytes apart).
__device__ __forceinline__ void put_split(uint8_t* dst, float4 v) {
    uint2 h, m, l;
    split2(v.x, v.y, h.x, m.x, l.x);
    split2(v.z, v.w, h.y, m.y, l.y);
    *reinterpret_cast<uint2*>(dst) = h;
    *reinterpret_cast<uint2*>(dst + PLANE) = m;
    *reinterpret_cast<uint2*>(dst + 2 * PLANE) = l;
}

// The tokens' three planes, [3][M][ldp] with ldp a multiple of 8, of which TMA copies tiles: split once for all weight tiles.
__global__ void __launch_bounds__(256)
split_planes_kernel(const float* __restrict__ a, __nv_bfloat16* __restrict__ planes, int M, int quads, long long lda, int ldp) {
    pdl_trigger();
    pdl_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)M * quads) return;
    const int t = (int)(i / quads), c = (int)(i % quads) * 4;
    const float4 v = scaled(*reinterpret_cast<const float4*>(a + t * lda + c));
    uint2 h, m, l;
    split2(v.x, v.y, h.x, m.x, l.x);
    split2(v.z, v.w, h.y, m.y, l.y);
    __nv_bfloat16* dst = planes + (long long)t * ldp + c;
    const long long plane = (long long)M * ldp;
    *reinterpret_cast<uint2*>(dst) = h;
    *reinterpret_cast<uint2*>(dst + plane) = m;
    *reinterpret_cast<uint2*>(dst + 2 * plane) = l;
}

template <int EPI, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap planes, F32TcParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(smem + STAGES * STAGE);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;             // [ACCS]
    uint64_t* acc_empty = acc_full + ACCS;           // [ACCS]
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + ACCS);
    volatile int* err = (volatile int*)(tmem_slot + 1);

    constexpr int FEATURES = EPI == EPI_SWIGLU ? BM / 2 : BM;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = SPLIT ? (int)(blockIdx.x % SLICES) : 0;
    const int n0 = (SPLIT ? blockIdx.x / SLICES : blockIdx.x) * FEATURES, t0 = blockIdx.y * BN;
    const int nkb = (p.K + BK - 1) / BK;
    const int per = (nkb + SLICES - 1) / SLICES;     // blocks a slice
    const int kb0 = SPLIT ? min(nkb, rank * per) : 0, kb1 = SPLIT ? min(nkb, kb0 + per) : nkb;
    const int nt = min(BN, (p.M - t0 + 15) / 16 * 16);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 9); mbar_init(&empty[s], 1); }
        for (int b = 0; b < ACCS; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8); }
        *err = 0;
        fence_barrier_init();
    }
    if (warp == 0) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
    if (threadIdx.x == 0) prefetch_tmap(&planes);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();

    float sum[BN / 2];                               // (warps 8-15: a weight row's sums over half of the tokens)
    bool ok = true;
    int armed = 0;                                   // (thread 0: blocks whose tokens' copies have been issued)
    if (warp < 8) {
        // ---------------- weights: load and split; a thread has 4 columns of rows r0, r0 + 16, ..., two blocks ahead ----------------
        const int r0 = threadIdx.x >> 4, col = (threadIdx.x & 15) * 4;
        uint8_t* dst0 = smem + r0 * 128 + ((((threadIdx.x & 15) >> 1) ^ (r0 & 7)) << 4) + (threadIdx.x & 1) * 8;
        const float* wsrc = p.w + (long long)(n0 + r0) * p.ldw + col;
        const float* wsrc2 = EPI == EPI_SWIGLU ? p.w2 + (long long)(n0 + r0) * p.ldw + col : wsrc + 64 * p.ldw;
        float4 wv[2][8];
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        auto load_w = [&](float4 (&v)[8], int kb) {
            const bool in = kb * BK + col < p.K;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int f = EPI == EPI_SWIGLU ? r0 + 16 * (i & 3) : r0 + 16 * i;
                const float* src = (i < 4 ? wsrc : wsrc2) + 16 * (i & 3) * p.ldw + (long long)kb * BK;
                v[i] = in && n0 + f < p.N ? *reinterpret_cast<const float4*>(src) : zero;
            }
        };
        bool go = true;
        auto block = [&](float4 (&v)[8], int kb) {
            const int i0 = kb - kb0, s = i0 % STAGES;
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = scaled(v[i]);             // (ahead of the wait: what follows it holds up the MMAs)
            go = warp_wait(&empty[s], (uint32_t)(((i0 / STAGES) & 1) ^ 1), err);
            if (!go) return;
            if (threadIdx.x == 0) {                  // the tokens' planes, 128 tokens of all three
                mbar_expect_tx(&full[s], 3 * PLANE);
                tma_load_3d(smem + s * STAGE + 3 * PLANE, &planes, &full[s], kb * BK, t0, 0);
                armed = i0 + 1;
            }
            uint8_t* dst = dst0 + s * STAGE;
#pragma unroll
            for (int i = 0; i < 8; ++i) put_split(dst + i * 16 * 128, v[i]);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
            if (kb + 2 < kb1) load_w(v, kb + 2);
        };
        if (kb0 < kb1) load_w(wv[0], kb0);           // the weights are no kernel's output
        if (kb0 + 1 < kb1) load_w(wv[1], kb0 + 1);
        pdl_wait();
        for (int kb = kb0; kb < kb1 && go; kb += 2) {
            block(wv[0], kb);
            if (go && kb + 1 < kb1) block(wv[1], kb + 1);
        }
    } else {
        // ---------------- sums: warps 8-11 the first half of the tokens, 12-15 the second ----------------
        const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) & 1) * (BN / 2);
        pdl_wait();
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        auto issue = [&](int i0) {                       // a whole warp: the MMAs of block i0
            const int s = i0 % STAGES, buf = i0 % ACCS;
            if (!warp_wait(&acc_empty[buf], (uint32_t)(((i0 / ACCS) & 1) ^ 1), err)) return;
            if (!warp_wait(&full[s], (uint32_t)((i0 / STAGES) & 1), err)) return;
            tc_fence_after();
            const uint64_t da = make_desc(smem_u32(smem + s * STAGE)), db = make_desc(smem_u32(smem + s * STAGE + 3 * PLANE));
            // (weights' part, tokens' part): the smallest products first
            constexpr int PA[6] = {2, 1, 0, 1, 0, 0}, PB[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
            for (int j = 0; j < 6; ++j)
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    warp_mma_bf16(tmem_base + buf * BN, da + (uint64_t)((PA[j] * PLANE + k * 32) >> 4),
                                  db + (uint64_t)((PB[j] * PLANE + k * 32) >> 4), idesc, j + k > 0 ? 1u : 0u);
            warp_commit(&empty[s]);
            warp_commit(&acc_full[buf]);
        };
        if (warp == 8 && kb0 < kb1) issue(0);
#pragma unroll
        for (int c = 0; c < BN / 2; ++c) sum[c] = 0.f;
        int in_slice = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
            const int i0 = kb - kb0, buf = i0 % ACCS;
            if (warp - 8 == ((i0 + 1) & 7) && kb + 1 < kb1) issue(i0 + 1);
            ok = warp_wait(&acc_full[buf], (uint32_t)((i0 / ACCS) & 1), err);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t r[32];
                tmem_ld32(lane_addr + buf * BN + h * 32, r);
                tmem_ld_wait();
                if (h == 1) {                            // the buffer is free before its last half has been added
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[buf]);
                }
#pragma unroll
                for (int c = 0; c < 32; ++c) sum[h * 32 + c] += __uint_as_float(r[c]);
            }
            if (!SPLIT && (++in_slice == per || kb + 1 == kb1)) {
                // a slice's end: the slices before it wait in tensor memory
                const bool first = kb + 1 <= per, last = kb + 1 == kb1;
                if (first && last) break;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t r[32];
                    if (!first) {
                        tmem_ld32(lane_addr + TOTAL_COL + h * 32, r);
                        tmem_ld_wait();
#pragma unroll
                        for (int c = 0; c < 32; ++c) sum[h * 32 + c] = __uint_as_float(r[c]) + sum[h * 32 + c];
                    }
                    if (!last) {
#pragma unroll
                        for (int c = 0; c < 32; ++c) { r[c] = __float_as_uint(sum[h * 32 + c]); sum[h * 32 + c] = 0.f; }
                        tmem_st32(lane_addr + TOTAL_COL + h * 32, r);
                    }
                }
                if (!last) tmem_st_wait();
                in_slice = 0;
            }
        }
    }
    // ---------------- results: by way of shared memory (the planes have been read for the last time) ----------------
    float* xch = (float*)smem;                           // [token][weight row]
    if (warp >= 8) {
        const int row = (warp & 3) * 32 + lane, half = (warp >> 2) & 1;
#pragma unroll
        for (int c = 0; c < BN / 2; ++c) xch[(half * (BN / 2) + c) * BM + row] = sum[c];
    }
    tc_fence_before();
    if constexpr (SPLIT) cg::this_cluster().sync();
    else __syncthreads();
    if (!*err) {
        const int slices = (nkb + per - 1) / per;
        constexpr int SHARE = SPLIT ? BN / SLICES : BN;  // this CTA's share of the tile's tokens
        constexpr int TOKENS = THREADS / FEATURES;       // tokens that the block takes at a time
        const int f = threadIdx.x % FEATURES, n = n0 + f;
        auto sum_of = [&](int tok, int col, const float* w) {
            float s;
            if constexpr (SPLIT) {
                s = 0.f;
                for (int i = 0; i < slices; ++i) s += cg::this_cluster().map_shared_rank(xch, i)[tok * BM + col];
            } else {
                s = xch[tok * BM + col];
            }
            return result(s, p.a + (long long)(t0 + tok) * p.lda, w + (long long)n * p.ldw, p.K);
        };
        constexpr int GROUP = SHARE / TOKENS < 8 ? SHARE / TOKENS : 8;      // results whose old values are asked for together
#pragma unroll 1
        for (int c0 = 0; c0 < SHARE / TOKENS; c0 += GROUP) {
            const int tok0 = rank * (SPLIT ? SHARE : 0) + threadIdx.x / FEATURES + c0 * TOKENS;
            float* o = p.out + (long long)(t0 + tok0) * p.ldo + n;
            float old[GROUP];
            if (EPI == EPI_ADD) {
#pragma unroll
                for (int c = 0; c < GROUP; ++c)
                    old[c] = n < p.N && t0 + tok0 + c * TOKENS < p.M ? o[(long long)c * TOKENS * p.ldo] : 0.f;
            }
#pragma unroll
            for (int c = 0; c < GROUP; ++c) {
                const int tok = tok0 + c * TOKENS;
                if (n >= p.N || t0 + tok >= p.M) continue;
                float v = sum_of(tok, f, p.w);
                if (EPI == EPI_ADD) v = old[c] + v;
                if (EPI == EPI_SWIGLU) v = v / (1.0f + expf(-v)) * sum_of(tok, FEATURES + f, p.w2);
                o[(long long)c * TOKENS * p.ldo] = v;
            }
        }
    }
    if (threadIdx.x == 0 && *err) {                      // the copies in flight land before the block's memory goes
        const long long since = clock64();
        for (int i = max(0, armed - STAGES); i < armed; ++i)
            while (!mbar_try_wait(&full[i % STAGES], (uint32_t)((i / STAGES) & 1))) if (clock64() - since > WAIT_LIMIT_CYCLES / 4) break;
    }
    if constexpr (SPLIT) cg::this_cluster().sync();      // nobody's sums go while another CTA reads them
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
    if (threadIdx.x == 0 && *err) atomicExch(p.error, 1);
}

// ---------------------------------------------------------------------------------------
// few tokens: the same sums by mma.sync
// ---------------------------------------------------------------------------------------
// A tile of 128 weight rows leaves the chip idle for a handful of tokens, and tensor memory, barriers and planes cost 9 us before the first
// result.  mma.sync (m16n8k16) adds sixteen products to its accumulator as tcgen05.mma does, with the same bits (the tests hold every
// form to that), so the same six products in the same order of sixteens, blocks of 64 and slices give the sums of the kernel above, and a
// token's result does not depend on how many tokens share the step.  Within sixteen terms the order does not matter, so a lane takes four
// neighbours of a row, 16 bytes, which it alone copies to shared memory (cp.async, two or three blocks ahead) and reads from there.
// A block takes 16 weight rows (the gate product: 8 of each matrix).  One, two or four warps take a slice of K: one adds its blocks up in
// registers; more leave the results of eight blocks in shared memory at a time and add them in order.
// What bounds it: with many rows the bytes; else the chain of a block of 64 (splitting, then 24 MMAs one after another: 1.1 us with a warp a
// scheduler), for which few rows get more warps.  Against the few-row kernel of gemm_f32.cu, inputs not in the L2, 4 tokens: N 2,048, K 6,144: 18.9 us -> 13.6;
// N 32,768, K 2,048: 52.9 -> 51.2 (5.2 TB/s); gate product of N 6,144, K 2,048: 23.5 -> 22.6; N 3,072, K 2,048: 7.8 -> 8.6; 16 tokens, in
// that order: 26.6 -> 18.4, 124 -> 65, 49.6 -> 28.2, 18.1 -> 13.5.  (With the weights in registers, a block ahead: 20.3, 50.8, 28.1, 9.0 with 4 tokens.)
constexpr int FEW_PIECE = 16 * 8;            // results of 16 weight rows and 8 tokens
constexpr int FEW_GROUP = 8;                 // blocks of a slice whose results meet at a time
template <int NT, int P> struct Few {
    static constexpr int STAGES = P == 1 && NT == 1 ? 3 : 2;             // blocks on their way, a warp
    static constexpr int STAGE = (8 + 4 * NT) * 128;     // floats: eight 16-byte pieces a lane of the weights, four of each eight tokens
    static constexpr int RING = 4 * P * STAGES * STAGE;
    static constexpr int TOTAL = (RING + SLICES * (P == 1 ? 1 : FEW_GROUP) * NT * FEW_PIECE) * 4;
};

__device__ __forceinline__ void mma_16816(float* d, const uint32_t* a, const uint32_t* b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <int EPI, int NT, int P>            // NT: eights of tokens; P: warps a slice
__global__ void __launch_bounds__(128 * P, P == 1 ? 3 : P == 2 && NT == 1 ? 2 : 1)
gemm_f32_few_mma_kernel(F32TcParams p) {
    using F = Few<NT, P>;
    extern __shared__ __align__(16) float few_smem[];
    constexpr int FEATURES = EPI == EPI_SWIGLU ? 8 : 16, MINE = FEW_GROUP / P;       // blocks of a group that a warp takes
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int slice = warp / P, part = warp % P;
    float* ring = few_smem + warp * F::STAGES * F::STAGE + lane * 4;     // (a lane's own pieces, 512 bytes apart)
    float* few = few_smem + F::RING;                 // [slice][block of the group][eight tokens][weight row][token]
    const int blocks_t = (p.M + 8 * NT - 1) / (8 * NT);      // neighbours share weights
    const int n0 = (int)(blockIdx.x / blocks_t) * FEATURES, t0 = (int)(blockIdx.x % blocks_t) * 8 * NT;
    const int nkb = (p.K + BK - 1) / BK, per = (nkb + SLICES - 1) / SLICES;
    const int lo = min(nkb, slice * per), hi = min(nkb, lo + per);
    // this warp's blocks: MINE neighbours of every group of FEW_GROUP (P == 1: all)
    auto block_of = [&](int i) { return P == 1 ? lo + i : lo + i / MINE * FEW_GROUP + part * MINE + i % MINE; };
    pdl_trigger();
    const bool ok0 = n0 + g < p.N, ok1 = EPI == EPI_SWIGLU ? ok0 : n0 + 8 + g < p.N;
    const float* w0 = p.w + (long long)(ok0 ? n0 + g : 0) * p.ldw;
    const float* w1 = EPI == EPI_SWIGLU ? p.w2 + (long long)(ok1 ? n0 + g : 0) * p.ldw : p.w + (long long)(ok1 ? n0 + 8 + g : 0) * p.ldw;
    auto load_w = [&](int i) {
        const int kb = block_of(i);
        if (kb >= hi) return;
        float* to = ring + i % F::STAGES * F::STAGE;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int c = kb * BK + k * 16 + 4 * t;
            const bool in = c < p.K;
            cp16(to + 2 * k * 128, w0 + (in ? c : 0), ok0 && in);
            cp16(to + (2 * k + 1) * 128, w1 + (in ? c : 0), ok1 && in);
        }
    };
    auto load_a = [&](int i) {
        const int kb = block_of(i);
        if (kb >= hi) return;
        float* to = ring + i % F::STAGES * F::STAGE + 8 * 128;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const int m = t0 + 8 * j + g;
            const float* at = p.a + (long long)(m < p.M ? m : 0) * p.lda;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int c = kb * BK + k * 16 + 4 * t;
                const bool in = c < p.K;
                cp16(to + (4 * j + k) * 128, at + (in ? c : 0), m < p.M && in);
            }
        }
    };
    // the weights are no kernel's output: the ring fills before the kernel in front has ended
#pragma unroll
    for (int i = 0; i < F::STAGES; ++i) load_w(i);
    pdl_wait();
#pragma unroll
    for (int i = 0; i < F::STAGES; ++i) {            // (the first group brings the weights of all stages)
        load_a(i);
        cp_commit();
    }
    float sum[P == 1 ? 4 * NT : 4 * NT / P];         // (P == 1: as the MMAs leave them; else this thread's outputs of the slice)
#pragma unroll
    for (int x = 0; x < (int)(sizeof(sum) / 4); ++x) sum[x] = 0.f;
    const int who = threadIdx.x % (32 * P);
    float* mine = few + slice * FEW_GROUP * NT * FEW_PIECE;
    const int groups = P == 1 ? 1 : (hi - lo + FEW_GROUP - 1) / FEW_GROUP;
    for (int gr = 0; gr < groups; ++gr) {
        const int i0 = P == 1 ? 0 : gr * MINE, i1 = P == 1 ? hi - lo : i0 + MINE;
#pragma unroll 1
        for (int i = i0; i < i1; ++i) {
            if (block_of(i) >= hi) break;
            cp_wait<F::STAGES - 1>();
            const float* v = ring + i % F::STAGES * F::STAGE;
            uint32_t a[4][3][4], b[NT][4][3][2];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float4 x = scaled(*reinterpret_cast<const float4*>(v + 2 * k * 128));
                const float4 y = scaled(*reinterpret_cast<const float4*>(v + (2 * k + 1) * 128));
                split2(x.x, x.y, a[k][0][0], a[k][1][0], a[k][2][0]);
                split2(y.x, y.y, a[k][0][1], a[k][1][1], a[k][2][1]);
                split2(x.z, x.w, a[k][0][2], a[k][1][2], a[k][2][2]);
                split2(y.z, y.w, a[k][0][3], a[k][1][3], a[k][2][3]);
            }
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float4 x = scaled(*reinterpret_cast<const float4*>(v + (8 + 4 * j + k) * 128));
                    split2(x.x, x.y, b[j][k][0][0], b[j][k][1][0], b[j][k][2][0]);
                    split2(x.z, x.w, b[j][k][0][1], b[j][k][1][1], b[j][k][2][1]);
                }
            load_w(i + F::STAGES);
            load_a(i + F::STAGES);
            cp_commit();
            // (weights' part, tokens' part): the smallest products first, as above
            constexpr int PA[6] = {2, 1, 0, 1, 0, 0}, PB[6] = {0, 1, 2, 0, 1, 0};
            float d[NT][4] = {};
#pragma unroll
            for (int y = 0; y < 6; ++y)
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int j = 0; j < NT; ++j) mma_16816(d[j], a[k][PA[y]], b[j][k][PB[y]]);
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                if constexpr (P == 1) {
#pragma unroll
                    for (int x = 0; x < 4; ++x) sum[4 * j + x] += d[j][x];
                } else {
                    float* to = mine + ((i - i0 + part * MINE) * NT + j) * FEW_PIECE + g * 8 + 2 * t;
                    *reinterpret_cast<float2*>(to) = make_float2(d[j][0], d[j][1]);
                    *reinterpret_cast<float2*>(to + 64) = make_float2(d[j][2], d[j][3]);
                }
            }
        }
        if constexpr (P > 1) {                       // the slice's warps add the group's blocks up in order
            asm volatile("bar.sync %0, %1;" ::"r"(1 + slice), "n"(32 * P) : "memory");
            const int n = min(FEW_GROUP, hi - lo - gr * FEW_GROUP);
#pragma unroll
            for (int x = 0; x < 4 * NT / P; ++x)
#pragma unroll
                for (int k = 0; k < FEW_GROUP; ++k)
                    if (k < n) sum[x] += mine[k * NT * FEW_PIECE + x * 32 * P + who];
            asm volatile("bar.sync %0, %1;" ::"r"(1 + slice), "n"(32 * P) : "memory");
        }
    }
    // the slices' sums: [slice][eight tokens][weight row][token], in a place of their own each
    constexpr int STRIDE = (P == 1 ? 1 : FEW_GROUP) * NT * FEW_PIECE;
    if constexpr (P == 1) {
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            float* to = few + slice * STRIDE + j * FEW_PIECE + g * 8 + 2 * t;
            *reinterpret_cast<float2*>(to) = make_float2(sum[4 * j], sum[4 * j + 1]);
            *reinterpret_cast<float2*>(to + 64) = make_float2(sum[4 * j + 2], sum[4 * j + 3]);
        }
    } else {
#pragma unroll
        for (int x = 0; x < 4 * NT / P; ++x) mine[x * 32 * P + who] = sum[x];
    }
    __syncthreads();
    const int slices = (nkb + per - 1) / per;
    for (int o = threadIdx.x; o < FEATURES * 8 * NT; o += 128 * P) {
        const int f = o % FEATURES, tok = o / FEATURES, n = n0 + f, m = t0 + tok;
        if (n >= p.N || m >= p.M) continue;
        auto sum_of = [&](int row, const float* w) {
            const float* at = few + (tok >> 3) * FEW_PIECE + row * 8 + (tok & 7);
            float s = 0.f;
            for (int i = 0; i < slices; ++i) s += at[i * STRIDE];
            return result(s, p.a + (long long)m * p.lda, w + (long long)n * p.ldw, p.K);
        };
        float* out = p.out + (long long)m * p.ldo + n;
        float v = sum_of(f, p.w);
        if (EPI == EPI_ADD) v = *out + v;
        if (EPI == EPI_SWIGLU) v = v / (1.0f + expf(-v)) * sum_of(8 + f, p.w2);
        *out = v;
    }
}

template <int EPI, int NT, int P>
static int launch_few(const F32TcParams& p, cudaStream_t st) {
    auto kern = gemm_f32_few_mma_kernel<EPI, NT, P>;
    constexpr int smem = Few<NT, P>::TOTAL;
    static UbAllowSmem allow;
    if (cudaError_t e = allow(kern, smem)) return (int)e;
    const int features = EPI == EPI_SWIGLU ? 8 : 16;
    const long long blocks = (long long)((p.N + features - 1) / features) * ((p.M + 8 * NT - 1) / (8 * NT));
    if (blocks > 0x7fffffffll) return UB_ERR_ARG;
    return (int)ub_launch_dependent(kern, dim3((unsigned)blocks), dim3(128 * P), smem, st, p);
}

template <int EPI>
static int launch_few(const F32TcParams& p, int warps, cudaStream_t st) {
    if (p.M <= 8) return warps == 1 ? launch_few<EPI, 1, 1>(p, st) : warps == 2 ? launch_few<EPI, 1, 2>(p, st) : launch_few<EPI, 1, 4>(p, st);
    return warps == 1 ? launch_few<EPI, 2, 1>(p, st) : launch_few<EPI, 2, 2>(p, st);
}

template <int EPI, bool SPLIT>
static int launch(const CUtensorMap& planes, const F32TcParams& p, cudaStream_t st) {
    auto kern = gemm_f32_tc_kernel<EPI, SPLIT>;
    static UbAllowSmem allow;
    if (cudaError_t e = allow(kern, SMEM)) return (int)e;
    const int features = EPI == EPI_SWIGLU ? BM / 2 : BM;
    dim3 grid((p.N + features - 1) / features, (p.M + BN - 1) / BN);
    if (grid.y > 65535) return UB_ERR_ARG;
    if (!SPLIT) return (int)ub_launch_dependent(kern, grid, dim3(THREADS), SMEM, st, planes, p);
    grid.x *= SLICES;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];                             // an ordinary launch: clusters take no part in dependent launches
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = SLICES; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kern, planes, p);
}

// ``form``: 0 whole tiles, 1 a cluster of four CTAs a tile, a slice of K each; 2, 3 and 4 the kernel of few tokens with one, two and four
// warps a slice (four: up to 8 tokens).  All give the same bits.  ``planes`` (forms 0 and 1): scratch of 3 M ldp bfloat16
// numbers, ldp = K rounded up to a multiple of 8, 16-byte aligned.  ``error`` is raised when a wait ran out of time.
UB_API int ub_gemm_f32_tc(const void* A, const void* W, const void* W2, void* out, void* planes, int M, int N, int K, long long lda,
                          long long ldw, long long ldo, int epi, int form, int* error, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 || lda % 4 || ldw % 4 || ((uintptr_t)A & 15) || ((uintptr_t)W & 15) || ((uintptr_t)W2 & 15)) return UB_ERR_ARG;
    if ((epi == EPI_SWIGLU && !W2) || epi < EPI_STORE || epi > EPI_SWIGLU || form < 0 || form > 4 || (form == 4 && M > 8)) return UB_ERR_ARG;
    const F32TcParams p{(const float*)A, (const float*)W, (const float*)W2, (float*)out, M, N, K, lda, ldw, ldo, error};
    if (form >= 2) {
        const int warps = 1 << (form - 2);
        if (epi == EPI_STORE) return launch_few<EPI_STORE>(p, warps, st);
        return epi == EPI_ADD ? launch_few<EPI_ADD>(p, warps, st) : launch_few<EPI_SWIGLU>(p, warps, st);
    }
    if (!error || !planes || ((uintptr_t)planes & 15)) return UB_ERR_ARG;
    static const EncodeTiledFn encode = tensor_map_encoder();
    if (!encode) return UB_ERR_UNSUPPORTED;
    const int ldp = (K + 7) / 8 * 8;
    CUtensorMap map;
    cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)M, 3};
    cuuint64_t strides[2] = {(cuuint64_t)ldp * 2, (cuuint64_t)M * ldp * 2};
    cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)BN, 3}, estr[3] = {1, 1, 1};
    if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, planes, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return UB_ERR_ARG;
    const long long quads = (long long)M * (K / 4);
    if (int e = (int)ub_launch_dependent(split_planes_kernel, dim3((unsigned)((quads + 255) / 256)), dim3(256), 0, st, (const float*)A,
                                         (__nv_bfloat16*)planes, M, K / 4, lda, ldp)) return e;
    if (epi == EPI_STORE) return form ? launch<EPI_STORE, true>(map, p, st) : launch<EPI_STORE, false>(map, p, st);
    if (epi == EPI_ADD) return form ? launch<EPI_ADD, true>(map, p, st) : launch<EPI_ADD, false>(map, p, st);
    return form ? launch<EPI_SWIGLU, true>(map, p, st) : launch<EPI_SWIGLU, false>(map, p, st);
}
