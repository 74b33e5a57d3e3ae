// Matrix product of float32 operands on the CUDA cores: out[t, n] = sum_k A[t, k] * W[n, k], float32 FMA.
//
// The true 32-bit path's products with small matrices (large ones: gemm_f32_tc.cu).  Rows of A and W start on
// 16-byte boundaries and K is a multiple of 4; everything else, and every mix with bfloat16, is gemm_simt.cu's.
//
// The order of an output's sum depends on K alone: K is cut into at most eight slices (``slice_len``), a slice is one chain
// of FMAs in k order, and the slices' sums are added in their order.  So a token's result does not depend on what else is in the
// batch, and eight slices of one output can be summed side by side where a product has few tokens.
//
// Three forms:
//   few rows (up to 16 tokens): bound by the weights' bytes.  A block takes 16 weight rows, its eight warps a slice of K each;
//      a warp streams its 16 rows through a ring of its own with cp.async (no block barrier in the loop) and a lane holds the sums of two
//      rows and of every fourth token.
//   tiles of 128 columns and 32, 64 or 128 tokens, K whole: bound by the FMA units; 8 columns a thread and up to 8 tokens.
//   the tiles of 32 and 64 tokens with a cluster of eight blocks, a slice each, where the tiles are too few for the chip; the slices' sums meet
//      through distributed shared memory.
//
// Measured against gemm_simt.cu (64 x 64 tiles, scalar loads, one chain): 4 tokens, N 2,048, K 6,144: 931 -> 18 us; N 32,768, K 2,048:
// 683 -> 54 us (5.0 TB/s); 681 tokens, the gate product of N 6,144, K 2,048: 1,390 -> 890 us (39 TFLOP/s; the FMA pipe is 62 %
// busy, registers' read ports and two warps a scheduler hold the rest), N 2,048, K 6,144: 824 -> 486 us.
#include <cooperative_groups.h>
#include "common.cuh"

namespace cg = cooperative_groups;

enum : int { EPI_STORE = 0, EPI_ADD = 1, EPI_SWIGLU = 2 };
constexpr int MAX_SLICES = 8;

__host__ __device__ inline int slice_len(int K) {
    const int per = ((K + MAX_SLICES - 1) / MAX_SLICES + 31) / 32 * 32;
    return per < 64 ? 64 : per;
}

__device__ __forceinline__ float chain4(float4 a, float4 w, float s) {
    s = fmaf(a.x, w.x, s);
    s = fmaf(a.y, w.y, s);
    s = fmaf(a.z, w.z, s);
    return fmaf(a.w, w.w, s);
}

struct F32Params {
    const float* a; const float* w; const float* w2; float* out;
    int M, N, K;
    long long lda, ldw, ldo;
};

template <int EPI>
__device__ __forceinline__ void put(const F32Params& p, int m, int n, float s, float u) {
    float* o = p.out + (long long)m * p.ldo + n;
    if (EPI == EPI_STORE) *o = s;
    else if (EPI == EPI_ADD) *o += s;
    else *o = s / (1.0f + expf(-s)) * u;
}

// ---------------------------------------------------------------------------------------
// few rows
// ---------------------------------------------------------------------------------------
constexpr int FR_ROWS = 16;                  // weight rows a block (the gate product: 8 of each matrix)
constexpr int FR_K = 32;                     // k columns a stage: 128 bytes a row
constexpr int FR_LD = FR_K + 4;              // eight rows' 16-byte pieces then lie in different banks
constexpr int FR_STAGES = 4;

template <int MPL> struct FewSmem {
    static constexpr int STAGE = (FR_ROWS + 4 * MPL) * FR_LD;                     // floats a warp and stage
    static constexpr int TOTAL = (8 * FR_STAGES * STAGE + MAX_SLICES * FR_ROWS * 4 * MPL) * 4;
};

template <int MPL, int EPI>
__global__ void __launch_bounds__(256)
gemm_f32_few_kernel(F32Params p) {
    using S = FewSmem<MPL>;
    extern __shared__ __align__(16) float few_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* ring = few_smem + warp * FR_STAGES * S::STAGE;
    float* red = few_smem + 8 * FR_STAGES * S::STAGE;            // [slice][row][token]
    constexpr int FEATURES = EPI == EPI_SWIGLU ? FR_ROWS / 2 : FR_ROWS;
    constexpr int TOKENS = 4 * MPL;
    const int n0 = blockIdx.x * FEATURES;
    const int len = slice_len(p.K);
    const int ks = min(p.K, warp * len), ke = min(p.K, ks + len);
    const int steps = (ke - ks + FR_K - 1) / FR_K;
    pdl_trigger();

    // a lane copies 16-byte piece (lane & 7) of rows (lane >> 3) + 4 i
    const int piece = (lane & 7) * 4, row0 = lane >> 3;
    const float* wsrc[FR_ROWS / 4];
    bool wok[FR_ROWS / 4];
#pragma unroll
    for (int i = 0; i < FR_ROWS / 4; ++i) {
        const int rr = row0 + 4 * i;
        const int n = n0 + (EPI == EPI_SWIGLU ? rr % FEATURES : rr);
        wok[i] = n < p.N;
        const float* base = EPI == EPI_SWIGLU && rr >= FEATURES ? p.w2 : p.w;
        wsrc[i] = base + (long long)(wok[i] ? n : 0) * p.ldw;
    }
    auto load_w = [&](int s) {
        float* st = ring + (s % FR_STAGES) * S::STAGE;
        const int k = ks + s * FR_K + piece;
        const bool in = k < ke;
#pragma unroll
        for (int i = 0; i < FR_ROWS / 4; ++i) cp16(st + (row0 + 4 * i) * FR_LD + piece, wsrc[i] + (in ? k : 0), wok[i] && in);
    };
    auto load_a = [&](int s) {
        float* st = ring + (s % FR_STAGES) * S::STAGE + FR_ROWS * FR_LD;
        const int k = ks + s * FR_K + piece;
#pragma unroll
        for (int i = 0; i < MPL; ++i) {
            const int m = row0 + 4 * i;
            const bool ok = m < p.M && k < ke;
            cp16(st + m * FR_LD + piece, p.a + (ok ? (long long)m * p.lda + k : 0), ok);
        }
    };
    // the weights are no kernel's output: the ring fills before the kernel in front has ended
#pragma unroll
    for (int s = 0; s < FR_STAGES - 1; ++s)
        if (s < steps) load_w(s);
    pdl_wait();
    // (the first group brings the weights of all these stages)
#pragma unroll
    for (int s = 0; s < FR_STAGES - 1; ++s) {
        if (s < steps) load_a(s);
        cp_commit();
    }
    const int r = lane >> 2, ml = lane & 3;
    float acc[2][MPL];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < MPL; ++j) acc[i][j] = 0.f;
    for (int s = 0; s < steps; ++s) {
        cp_wait<FR_STAGES - 2>();
        __syncwarp();
        const float* st = ring + (s % FR_STAGES) * S::STAGE;
#pragma unroll
        for (int k = 0; k < FR_K; k += 4) {
            float4 wv[2], av[MPL];
#pragma unroll
            for (int i = 0; i < 2; ++i) wv[i] = *reinterpret_cast<const float4*>(st + (r + 8 * i) * FR_LD + k);
#pragma unroll
            for (int j = 0; j < MPL; ++j) av[j] = *reinterpret_cast<const float4*>(st + (FR_ROWS + ml + 4 * j) * FR_LD + k);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < MPL; ++j) acc[i][j] = chain4(av[j], wv[i], acc[i][j]);
        }
        __syncwarp();                                    // every lane has read the stage that is filled next
        const int next = s + FR_STAGES - 1;
        if (next < steps) { load_w(next); load_a(next); }
        cp_commit();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < MPL; ++j) red[(warp * FR_ROWS + r + 8 * i) * TOKENS + ml + 4 * j] = acc[i][j];
    __syncthreads();
    const int slices = (p.K + len - 1) / len;
    for (int o = threadIdx.x; o < FEATURES * TOKENS; o += 256) {
        const int f = o % FEATURES, m = o / FEATURES;
        if (m >= p.M || n0 + f >= p.N) continue;
        float s = red[f * TOKENS + m], u = EPI == EPI_SWIGLU ? red[(f + FEATURES) * TOKENS + m] : 0.f;
        for (int i = 1; i < slices; ++i) {
            s += red[(i * FR_ROWS + f) * TOKENS + m];
            if (EPI == EPI_SWIGLU) u += red[(i * FR_ROWS + f + FEATURES) * TOKENS + m];
        }
        put<EPI>(p, m, n0 + f, s, u);
    }
}

// ---------------------------------------------------------------------------------------
// tiles
// ---------------------------------------------------------------------------------------
constexpr int TL_N = 128;                    // columns a tile (the gate product: 64 of each matrix)
constexpr int TL_K = 32;
constexpr int TL_LD = TL_K + 4;
constexpr int TL_STAGES = 3;

template <int BM> struct TileSmem {
    static constexpr int STAGE = (BM + TL_N) * TL_LD;
    static constexpr int RING = TL_STAGES * STAGE;
    static constexpr int TOTAL = (RING > BM * TL_N ? RING : BM * TL_N) * 4;
};

template <int BM, int EPI, bool SPLIT>
__global__ void __launch_bounds__(256, BM == 32 ? 2 : 1)
gemm_f32_tile_kernel(F32Params p) {
    using S = TileSmem<BM>;
    extern __shared__ __align__(16) float tile_smem[];
    constexpr int MT = BM / 16;                              // tokens a thread
    constexpr int FEATURES = EPI == EPI_SWIGLU ? TL_N / 2 : TL_N;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);
    const int rank = SPLIT ? (int)(blockIdx.x % MAX_SLICES) : 0;
    const int n0 = (SPLIT ? blockIdx.x / MAX_SLICES : blockIdx.x) * FEATURES, m0 = blockIdx.y * BM;
    const int len = slice_len(p.K);
    const int ks = SPLIT ? min(p.K, rank * len) : 0, ke = SPLIT ? min(p.K, ks + len) : p.K;
    const int steps = (ke - ks + TL_K - 1) / TL_K;
    const int steps_slice = len / TL_K;
    pdl_trigger();

    const int piece = (tid & 7) * 4, row0 = tid >> 3;        // 32 rows a pass over the block
    const float* wsrc[TL_N / 32];
    bool wok[TL_N / 32];
#pragma unroll
    for (int i = 0; i < TL_N / 32; ++i) {
        const int rr = row0 + 32 * i;
        const int n = n0 + (EPI == EPI_SWIGLU ? rr % FEATURES : rr);
        wok[i] = n < p.N;
        wsrc[i] = (EPI == EPI_SWIGLU && rr >= FEATURES ? p.w2 : p.w) + (long long)(wok[i] ? n : 0) * p.ldw;
    }
    auto load_w = [&](int s) {
        float* st = tile_smem + (s % TL_STAGES) * S::STAGE + BM * TL_LD;
        const int k = ks + s * TL_K + piece;
        const bool in = k < ke;
#pragma unroll
        for (int i = 0; i < TL_N / 32; ++i) cp16(st + (row0 + 32 * i) * TL_LD + piece, wsrc[i] + (in ? k : 0), wok[i] && in);
    };
    auto load_a = [&](int s) {
        float* st = tile_smem + (s % TL_STAGES) * S::STAGE;
        const int k = ks + s * TL_K + piece;
#pragma unroll
        for (int i = 0; i < BM / 32; ++i) {
            const int m = m0 + row0 + 32 * i;
            const bool ok = m < p.M && k < ke;
            cp16(st + (row0 + 32 * i) * TL_LD + piece, p.a + (ok ? (long long)m * p.lda + k : 0), ok);
        }
    };
#pragma unroll
    for (int s = 0; s < TL_STAGES - 1; ++s)
        if (s < steps) load_w(s);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < TL_STAGES - 1; ++s) {
        if (s < steps) load_a(s);
        cp_commit();
    }
    float acc[MT][8], total[SPLIT ? 1 : MT][8];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            acc[i][j] = 0.f;
            if constexpr (!SPLIT) total[i][j] = 0.f;
        }
    int in_slice = 0;
    for (int s = 0; s < steps; ++s) {
        cp_wait<TL_STAGES - 2>();
        __syncthreads();                                     // the stage is there, and the one filled next has been read
        const int next = s + TL_STAGES - 1;
        if (next < steps) { load_w(next); load_a(next); }
        cp_commit();
        const float* sa = tile_smem + (s % TL_STAGES) * S::STAGE;
        const float* sw = sa + BM * TL_LD;
#pragma unroll
        for (int k = 0; k < TL_K; k += 4) {
            float4 av[MT];
#pragma unroll
            for (int i = 0; i < MT; ++i) av[i] = *reinterpret_cast<const float4*>(sa + (ty + 16 * i) * TL_LD + k);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 wv = *reinterpret_cast<const float4*>(sw + (tx + 16 * j) * TL_LD + k);
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i][j] = chain4(av[i], wv, acc[i][j]);
            }
        }
        if constexpr (!SPLIT) {
            if (++in_slice == steps_slice || s + 1 == steps) {
#pragma unroll
                for (int i = 0; i < MT; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        total[i][j] += acc[i][j];
                        acc[i][j] = 0.f;
                    }
                in_slice = 0;
            }
        }
    }
    if constexpr (!SPLIT) {
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int m = m0 + ty + 16 * i;
            if (m >= p.M) continue;
#pragma unroll
            for (int j = 0; j < (EPI == EPI_SWIGLU ? 4 : 8); ++j) {
                const int n = n0 + tx + 16 * j;
                if (n < p.N) put<EPI>(p, m, n, total[i][j], EPI == EPI_SWIGLU ? total[i][(j + 4) & 7] : 0.f);
            }
        }
    } else {
        cg::cluster_group cluster = cg::this_cluster();
        __syncthreads();                                     // the ring is read for the last time
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) tile_smem[(ty + 16 * i) * TL_N + tx + 16 * j] = acc[i][j];
        cluster.sync();
        const int slices = (p.K + len - 1) / len;
        constexpr int ROWS = BM / MAX_SLICES;                // this block's share of the tile's tokens
        for (int o = tid; o < ROWS * FEATURES; o += 256) {
            const int row = rank * ROWS + o / FEATURES, f = o % FEATURES;
            const int m = m0 + row, n = n0 + f;
            if (m >= p.M || n >= p.N) continue;
            float s = 0.f, u = 0.f;
            for (int i = 0; i < slices; ++i) {
                const float* other = cluster.map_shared_rank(tile_smem, i) + row * TL_N + f;
                s += other[0];
                if (EPI == EPI_SWIGLU) u += other[FEATURES];
            }
            put<EPI>(p, m, n, s, u);
        }
        cluster.sync();                                      // nobody's sums go while another block reads them
    }
}

template <int MPL, int EPI>
static int launch_few(const F32Params& p, cudaStream_t st) {
    auto kern = gemm_f32_few_kernel<MPL, EPI>;
    constexpr int smem = FewSmem<MPL>::TOTAL;
    static UbAllowSmem allow;
    if (cudaError_t e = allow(kern, smem)) return (int)e;
    const int features = EPI == EPI_SWIGLU ? FR_ROWS / 2 : FR_ROWS;
    return (int)ub_launch_dependent(kern, dim3((p.N + features - 1) / features), dim3(256), smem, st, p);
}

template <int BM, int EPI, bool SPLIT>
static int launch_tile(const F32Params& p, cudaStream_t st) {
    auto kern = gemm_f32_tile_kernel<BM, EPI, SPLIT>;
    constexpr int smem = TileSmem<BM>::TOTAL;
    static UbAllowSmem allow;
    if (cudaError_t e = allow(kern, smem)) return (int)e;
    const int features = EPI == EPI_SWIGLU ? TL_N / 2 : TL_N;
    dim3 grid((p.N + features - 1) / features, (p.M + BM - 1) / BM);
    if (grid.y > 65535) return UB_ERR_ARG;
    if (!SPLIT) return (int)ub_launch_dependent(kern, grid, dim3(256), smem, st, p);
    grid.x *= MAX_SLICES;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];                             // an ordinary launch: clusters take no part in dependent launches
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = MAX_SLICES; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kern, p);
}

template <int EPI>
static int go(const F32Params& p, int form, cudaStream_t st) {
    switch (form) {
        case 0: return p.M <= 4 ? launch_few<1, EPI>(p, st) : p.M <= 8 ? launch_few<2, EPI>(p, st) : launch_few<4, EPI>(p, st);
        case 32: return launch_tile<32, EPI, false>(p, st);
        case 64: return launch_tile<64, EPI, false>(p, st);
        case 128: return launch_tile<128, EPI, false>(p, st);
        case -32: return launch_tile<32, EPI, true>(p, st);
        case -64: return launch_tile<64, EPI, true>(p, st);
    }
    return UB_ERR_ARG;
}

// form: 0 the kernel of few rows (M up to 16); 32, 64, 128 tiles of that many tokens; -32, -64: the same with a cluster a tile.
UB_API int ub_gemm_f32(const void* A, const void* W, const void* W2, void* out, int M, int N, int K, long long lda, long long ldw,
                       long long ldo, int epi, int form, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 || lda % 4 || ldw % 4 || ((uintptr_t)A & 15) || ((uintptr_t)W & 15) || ((uintptr_t)W2 & 15)) return UB_ERR_ARG;
    if (form == 0 && M > 16) return UB_ERR_ARG;
    if (epi == EPI_SWIGLU && !W2) return UB_ERR_ARG;
    const F32Params p{(const float*)A, (const float*)W, (const float*)W2, (float*)out, M, N, K, lda, ldw, ldo};
    if (epi == EPI_STORE) return go<EPI_STORE>(p, form, st);
    if (epi == EPI_ADD) return go<EPI_ADD>(p, form, st);
    if (epi == EPI_SWIGLU) return go<EPI_SWIGLU>(p, form, st);
    return UB_ERR_ARG;
}
