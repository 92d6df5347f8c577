// C[M, N] = A[M, K] * W[N, K]^T in true float32: FMA on the CUDA cores, no tensor-core
// mode of reduced precision.  It is the matrix product of the float32 path, but for the tokens of longer rows, whose wide products
// gemm_f32_tc.cu takes (exact splits of the operands on the tensor cores; the caller chooses, acorninfer_b200/kernels/ops.py).
//
// Every kernel of this file sums an output element in one order: K is cut into eight ranges of ceil(K / 128) * 16, a range is a
// chain acc = fma(a[k], w[k], acc) from 0 in the order of k, and the result is T0 + T1 + ... + T7 from the left.  So a
// row's bits do not depend on the kernel that ran, on M, on the other rows or on the tile sizes.  The ranges are what lets
// eight warps (decode) or eight CTAs (prompts with few tiles) work on one output tile: one chain over all of K = 6,144
// takes 12.5 us in dependent multiply-adds alone, where the weights of N = 2,048 columns stream in 7.6 us.
//
// A, W: float32 row-major, K contiguous, with row strides lda, ldw; C row stride ldc.
//   rows kernel   up to 16 rows (decode; at many widths up to 32, in two launches): a block takes up to 16 or 32 columns and all
//                 rows, a warp one range of K with a ring of cp.async stages of its own (no block barrier): bound by reading W
//                 once and by the reads of shared memory;
//   tile kernel   more rows: 64 x 128 a block; a cluster of eight shares a tile's ranges where the tiles
//                 alone leave the device idle: bound by the multiply-adds and the reads of shared memory that feed them;
//   plain kernel  64 x 64 a block, scalar loads: operands that are not 16-byte aligned.
#include "mma_helpers.cuh"

#include <cooperative_groups.h>
namespace cg = cooperative_groups;

// a range of K: a multiple of 16, so that no k-step of a kernel crosses from one into the next
#define K_RANGES 8
__host__ __device__ __forceinline__ int k_range(int K) { return (K + 16 * K_RANGES - 1) / (16 * K_RANGES) * 16; }

// ------------------------------------------------------------------ plain kernel

#define PL_BM 64
#define PL_BN 64
#define PL_BK 16

__global__ void __launch_bounds__(256) gemm_f32_kernel(const float* __restrict__ A, int64_t lda,
                                                       const float* __restrict__ W, int64_t ldw,
                                                       float* __restrict__ C, int64_t ldc, int M, int N, int K) {
    __shared__ float As[PL_BK][PL_BM + 4];
    __shared__ float Ws[PL_BK][PL_BN + 4];
    const int m0 = blockIdx.y * PL_BM, n0 = blockIdx.x * PL_BN;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // 16 x 16 threads
    float acc[4][4] = {}, total[4][4] = {};
    const int range = k_range(K);
    for (int k0 = 0; k0 < K; k0 += PL_BK) {
        if (k0 > 0 && k0 % range == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    total[i][j] += acc[i][j];
                    acc[i][j] = 0.f;
                }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int idx = threadIdx.x + e * 256;
            const int row = idx >> 4, kk = idx & 15;
            const int k = k0 + kk;
            As[kk][row] = (m0 + row < M && k < K) ? A[(int64_t)(m0 + row) * lda + k] : 0.f;
            Ws[kk][row] = (n0 + row < N && k < K) ? W[(int64_t)(n0 + row) * ldw + k] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < PL_BK; ++kk) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n < N) C[(int64_t)m * ldc + n] = total[i][j] + acc[i][j];
        }
    }
}

// ------------------------------------------------------------------ rows kernel

#define RS_BK 32
#define RS_LD (RS_BK + 4)       // row stride in shared memory: 16-byte reads of 8 neighbouring rows hit 8 groups of banks
#define RS_THREADS (32 * K_RANGES)

// R rows and CPL columns a lane, 2 R rows and 16 CPL columns a block, of which a tile of the NARROW form uses `width`.
template <int R, int CPL> constexpr int rs_stages() { return R >= 7 && CPL == 2 ? 3 : 4; }     // what shared memory holds
template <int R, int CPL> constexpr int rs_ring() { return K_RANGES * rs_stages<R, CPL>() * (16 * CPL + 2 * R) * RS_LD; }
// the ranges' sums: with one column a lane in the place of the rings, with two behind them, for two tiles
template <int R, int CPL> constexpr int rs_smem() {
    return (rs_ring<R, CPL>() + (CPL == 2 ? 2 * K_RANGES * 2 * R * 16 * CPL : 0)) * (int)sizeof(float);
}

// With two columns a lane a row of A that was read serves two weights, but a block takes 32 columns: for wide matrices only.
// A block then walks the tiles of its share one behind the other, and the next tile's weights are under way while the ranges'
// sums of the one before are added: a block that ends with its tile spends a third of its time on filling and emptying its
// rings (6 rows, N = 12,288, K = 2,048: 31 -> 25 us).
// The reads of A and W from shared memory that feed the multiply-adds set the pace (R + CPL reads of 16 bytes a lane for 4 R CPL
// multiply-adds), so there is a form for each number of rows a lane: at most one row is read that is not there (two for two rows).
// Measured (B200, us, forms for 4, 8 and 16 rows only / this), 6 rows: N = 4,096, K = 2,048 11.5 / 8.5; N = 2,048, K = 6,144 19.6 / 14.2; N = 12,288, K = 2,048
// 26.4 / 24.9 (4.0 TB/s); N = 151,936, K = 1,024 134 / 122 (5.1 TB/s); one row of the last 107 / 98 (6.4 TB/s).
template <int R, int CPL, bool NARROW>
__global__ void __launch_bounds__(RS_THREADS) gemm_f32_rows_kernel(const float* __restrict__ A, int64_t lda,
                                                                   const float* __restrict__ W, int64_t ldw,
                                                                   float* __restrict__ C, int64_t ldc, int M, int N, int K, int width) {
    extern __shared__ __align__(16) float rs_buf[];
    constexpr int BN = 16 * CPL, ROWS = BN + 2 * R, STAGE = ROWS * RS_LD, STAGES = rs_stages<R, CPL>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int col = lane & 15, row0 = (lane >> 4) * R;
    const int range = k_range(K), kbeg = min(K, warp * range), kend = min(K, kbeg + range);
    const int nk = (kend - kbeg + RS_BK - 1) / RS_BK;
    const int step = NARROW ? width : BN;        // columns from a tile to the next
    const int tiles = (int)(((unsigned int)N + step - 1) / step);
    const int mine = CPL == 2 ? (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 1;   // tiles of this block
    float* ring = rs_buf + warp * STAGES * STAGE;

    int ltile = 0, lkb = 0, fill = 0;            // the next stage to load: of which tile of this block, where in K, into which slot
    auto load = [&]() {
        if (ltile < mine && nk > 0) {
            const int n0 = ((int)blockIdx.x + ltile * (int)gridDim.x) * step, cols = NARROW ? min(width, N - n0) : N - n0;
            float* dst = ring + fill * STAGE;
#pragma unroll
            for (int e = 0; e < (ROWS + 3) / 4; ++e) {           // rows of W, then of A; 8 lanes take 128 bytes of a row
                const int row = e * 4 + (lane >> 3), seg = (lane & 7) * 4, k = kbeg + lkb * RS_BK + seg;
                if (ROWS % 4 != 0 && row >= ROWS) break;         // in the last turn
                const bool of_w = e < BN / 4;
                const bool valid = k < kend && (of_w ? (NARROW ? row < cols : n0 + row < N) : row - BN < M);
                const float* src = of_w ? W + (int64_t)(n0 + row) * ldw + k : A + (int64_t)(row - BN) * lda + k;
                cp_async_16(smem_addr(dst + row * RS_LD + seg), valid ? src : W, valid);
            }
            if (++lkb == nk) { lkb = 0; ++ltile; }
            fill = fill + 1 == STAGES ? 0 : fill + 1;
        }
        cp_async_commit();
    };

    // the first weights on their way to L2 while the kernel before this one ends (W may be its result: not read yet)
#pragma unroll
    for (int e = 0; e < CPL * (STAGES - 1) / 2; ++e) {
        const int c = (lane + 32 * e) % BN, n = (int)blockIdx.x * step + c, k = kbeg + ((lane + 32 * e) / BN) * RS_BK;
        if (k < kend && (!NARROW || c < width) && n < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(W + (int64_t)n * ldw + k));
    }
    pdl_wait();
    pdl_trigger();
    for (int s = 0; s < STAGES - 1; ++s) load();
    int stage = 0;
    for (int it = 0; it < mine; ++it) {
        const int n0 = ((int)blockIdx.x + it * (int)gridDim.x) * step, cols = NARROW ? min(width, N - n0) : N - n0;
        float acc[R][CPL];
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int c = 0; c < CPL; ++c) acc[i][c] = 0.f;
        for (int kb = 0; kb < nk; ++kb) {
            cp_async_wait<STAGES - 2>();         // this lane's copies of the stage have landed
            __syncwarp();                        // all lanes' have, and all are done with the stage before
            load();
            const float* wrow = ring + stage * STAGE + col * RS_LD;
            const float* arow = ring + stage * STAGE + (BN + row0) * RS_LD;
            stage = stage + 1 == STAGES ? 0 : stage + 1;
#pragma unroll
            for (int kk = 0; kk < RS_BK; kk += 4) {
                float4 w[CPL];
#pragma unroll
                for (int c = 0; c < CPL; ++c) w[c] = *reinterpret_cast<const float4*>(wrow + 16 * c * RS_LD + kk);
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    const float4 a = *reinterpret_cast<const float4*>(arow + i * RS_LD + kk);
#pragma unroll
                    for (int c = 0; c < CPL; ++c) {
                        acc[i][c] = fmaf(a.x, w[c].x, acc[i][c]);
                        acc[i][c] = fmaf(a.y, w[c].y, acc[i][c]);
                        acc[i][c] = fmaf(a.z, w[c].z, acc[i][c]);
                        acc[i][c] = fmaf(a.w, w[c].w, acc[i][c]);
                    }
                }
            }
        }
        float* parts = rs_buf;                   // [ranges][2 R][BN]
        if (CPL == 2) {
            parts += rs_ring<R, CPL>() + (it & 1) * K_RANGES * 2 * R * BN;
        } else {
            cp_async_wait<0>();
            __syncthreads();                     // the rings are free
        }
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int c = 0; c < CPL; ++c) parts[(warp * 2 * R + row0 + i) * BN + 16 * c + col] = acc[i][c];
        __syncthreads();                         // the one barrier of a tile: its sums were read before the next tile's barrier
        for (int o = threadIdx.x; o < 2 * R * BN; o += RS_THREADS) {
            const int r = o / BN, c = o % BN;
            if (r >= M || (NARROW ? c >= cols : n0 + c >= N)) continue;
            float v = parts[o];
#pragma unroll
            for (int q = 1; q < K_RANGES; ++q) v += parts[q * 2 * R * BN + o];
            C[(int64_t)r * ldc + n0 + c] = v;
        }
    }
    cp_async_wait<0>();
}

// ------------------------------------------------------------------ tile kernel

#define TL_BM 64
#define TL_BN 128
#define TL_BK 16
#define TL_THREADS 128
#define TL_SMEM ((2 * TL_BK * (TL_BM + TL_BN) + TL_BM * TL_BN) * (int)sizeof(float))

// acc += (a, a) * w on a pair of columns
__device__ __forceinline__ void fma_pair(float2& acc, unsigned long long a, float2 w) {
    unsigned long long r = *reinterpret_cast<unsigned long long*>(&acc);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(r) : "l"(a), "l"(*reinterpret_cast<unsigned long long*>(&w)));
    acc = *reinterpret_cast<float2*>(&r);
}

// A thread holds 8 rows x 8 columns in packed pairs: four 16-byte reads of shared memory feed 64 multiply-adds, and the packed
// instructions leave half of the issue slots to them.  Four lanes bring 64 bytes of a row; shared memory is [k][row], rows
// exchanged in groups of eight by k / 4, so that neither those writes nor the reads meet in a bank.
// SPLIT: a cluster of eight CTAs shares an output tile, each takes one range of K, and each adds up and writes an eighth of
// the tile's rows.
// Bound by the multiply-adds and the reads of shared memory about equally (2,048 rows, N = 4,096, K = 1,024: the multiply-add
// pipe 67 % busy, the shared memory pipe 70 %; 47 TFLOP/s, where a loop of nothing but packed multiply-adds runs at 73).
// Measured (B200): the 112 products of a 777-token prompt at Qwen3-0.6B sizes: with one chain over K and tiles of 128 x 128
// 32.8 ms; tiles of 64 x 64, 4 x 8 a thread, one multiply-add an instruction, rows as in memory 20.6 ms; this 18.8 ms.
template <bool SPLIT>
__global__ void __launch_bounds__(TL_THREADS, 3) gemm_f32_tile_kernel(const float* __restrict__ A, int64_t lda,
                                                                      const float* __restrict__ W, int64_t ldw,
                                                                      float* __restrict__ C, int64_t ldc, int M, int N,
                                                                      int K) {
    constexpr int BM = TL_BM, BN = TL_BN;
    extern __shared__ __align__(16) float tl_buf[];
    float* As = tl_buf;                                          // [2][BK][BM]
    float* Ws = As + 2 * TL_BK * BM;                             // [2][BK][BN]
    float* total = Ws + 2 * TL_BK * BN;                          // the ranges' sum so far, [element][thread]; SPLIT: [row][column]
    const int part = SPLIT ? blockIdx.x % K_RANGES : 0;
    const int m0 = blockIdx.y * BM, n0 = (SPLIT ? blockIdx.x / K_RANGES : blockIdx.x) * BN;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);     // columns 4 tx .., 64 + ..; rows 4 ty .., 32 + ..
    const int range = k_range(K);
    const int kbeg = SPLIT ? min(K, part * range) : 0, kend = SPLIT ? min(K, kbeg + range) : K;
    const int nt = (kend - kbeg + TL_BK - 1) / TL_BK;
    const int lrow = threadIdx.x >> 2, lseg = threadIdx.x & 3;   // brings k 4 lseg .. of rows lrow + 32 e
    float4 ra[BM / 32], rw[BN / 32];

    auto fetch = [&](int t) {                                    // rows beyond the matrix: another row's values, never written
        const int k = kbeg + t * TL_BK + 4 * lseg;
#pragma unroll
        for (int e = 0; e < BM / 32; ++e)
            ra[e] = k < kend ? *reinterpret_cast<const float4*>(A + (int64_t)min(m0 + lrow + 32 * e, M - 1) * lda + k) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int e = 0; e < BN / 32; ++e)
            rw[e] = k < kend ? *reinterpret_cast<const float4*>(W + (int64_t)min(n0 + lrow + 32 * e, N - 1) * ldw + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto stash = [&](int buf) {
        float* a = As + (buf * TL_BK + 4 * lseg) * BM + (lrow ^ (lseg << 3));
        float* w = Ws + (buf * TL_BK + 4 * lseg) * BN + (lrow ^ (lseg << 3));
#pragma unroll
        for (int e = 0; e < BM / 32; ++e) {
            a[32 * e] = ra[e].x; a[BM + 32 * e] = ra[e].y; a[2 * BM + 32 * e] = ra[e].z; a[3 * BM + 32 * e] = ra[e].w;
        }
#pragma unroll
        for (int e = 0; e < BN / 32; ++e) {
            w[32 * e] = rw[e].x; w[BN + 32 * e] = rw[e].y; w[2 * BN + 32 * e] = rw[e].z; w[3 * BN + 32 * e] = rw[e].w;
        }
    };

    float2 acc[8][4];                            // [row][pair of columns]
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
    pdl_wait();
    pdl_trigger();
    if (nt > 0) {
        fetch(0);
        stash(0);
    }
    __syncthreads();
    bool folded = false;
    for (int t = 0; t < nt; ++t) {
        const int buf = t & 1;
        if (t + 1 < nt) fetch(t + 1);            // in flight while this tile is multiplied
        if (!SPLIT && t > 0 && (t * TL_BK) % range == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float2* p = reinterpret_cast<float2*>(total) + (i * 4 + j) * TL_THREADS + threadIdx.x;
                    float2 v = folded ? *p : make_float2(0.f, 0.f);
                    v.x += acc[i][j].x;
                    v.y += acc[i][j].y;
                    *p = v;
                    acc[i][j] = make_float2(0.f, 0.f);
                }
            folded = true;
        }
#pragma unroll
        for (int kk = 0; kk < TL_BK; ++kk) {
            const float* a_at = As + (buf * TL_BK + kk) * BM;
            const float* w_at = Ws + (buf * TL_BK + kk) * BN;
            float2 w[4];
            unsigned long long a[8];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const float4 v = *reinterpret_cast<const float4*>(w_at + ((64 * c + 4 * tx) ^ ((kk >> 2) << 3)));
                w[2 * c] = make_float2(v.x, v.y);
                w[2 * c + 1] = make_float2(v.z, v.w);
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float4 v = *reinterpret_cast<const float4*>(a_at + ((32 * r + 4 * ty) ^ ((kk >> 2) << 3)));
                asm("mov.b64 %0, {%1, %1};" : "=l"(a[4 * r]) : "f"(v.x));
                asm("mov.b64 %0, {%1, %1};" : "=l"(a[4 * r + 1]) : "f"(v.y));
                asm("mov.b64 %0, {%1, %1};" : "=l"(a[4 * r + 2]) : "f"(v.z));
                asm("mov.b64 %0, {%1, %1};" : "=l"(a[4 * r + 3]) : "f"(v.w));
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) fma_pair(acc[i][j], a[i], w[j]);
        }
        if (t + 1 < nt) stash(buf ^ 1);          // the other buffer was last read before the barrier below, a tile ago
        __syncthreads();
    }
    if (SPLIT) {
        cg::cluster_group cluster = cg::this_cluster();
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int c = 0; c < 2; ++c)
                *reinterpret_cast<float4*>(total + (4 * ty + (i & 3) + 32 * (i >> 2)) * BN + 64 * c + 4 * tx) =
                    make_float4(acc[i][2 * c].x, acc[i][2 * c].y, acc[i][2 * c + 1].x, acc[i][2 * c + 1].y);
        cluster.sync();
        const float4* mine = reinterpret_cast<const float4*>(total);
#pragma unroll 2
        for (int o = threadIdx.x; o < BM / K_RANGES * BN / 4; o += TL_THREADS) {
            const int row = part * (BM / K_RANGES) + o / (BN / 4), c = (o % (BN / 4)) * 4, at = (row * BN + c) / 4;
            if (m0 + row >= M) break;
            float4 p[K_RANGES];
#pragma unroll
            for (int q = 0; q < K_RANGES; ++q) p[q] = cluster.map_shared_rank(mine, q)[at];
            float v[4] = {p[0].x, p[0].y, p[0].z, p[0].w};
#pragma unroll
            for (int q = 1; q < K_RANGES; ++q) { v[0] += p[q].x; v[1] += p[q].y; v[2] += p[q].z; v[3] += p[q].w; }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (n0 + c + e < N) C[(int64_t)(m0 + row) * ldc + n0 + c + e] = v[e];
        }
        cluster.sync();                          // a CTA's shared memory stays until all have read it
        return;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + 4 * ty + (i & 3) + 32 * (i >> 2);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float2 v = acc[i][j];
            if (folded) {
                const float2 p = reinterpret_cast<const float2*>(total)[(i * 4 + j) * TL_THREADS + threadIdx.x];
                v.x = p.x + v.x;
                v.y = p.y + v.y;
            }
            const int n = n0 + 64 * (j >> 1) + 4 * tx + 2 * (j & 1);
            if (m < M && n < N) C[(int64_t)m * ldc + n] = v.x;
            if (m < M && n + 1 < N) C[(int64_t)m * ldc + n + 1] = v.y;
        }
    }
}

// ------------------------------------------------------------------ host side

static_assert(PL_BM == TL_BM, "the plain and the tile kernel cover the same rows a grid");

// Shared memory that leaves no room for a second block on the SM.  A launch of no more blocks than SMs asks for it: its blocks come
// while those of the kernel before it end, and two would go to the SMs that are free first, while others stay without (a decode step
// of 6 rows at Qwen3-1.7B sizes: 3,042 -> 2,938 us).
#define RS_ALONE (116 * 1024)

template <int R, int CPL, bool NARROW>
static int launch_rows_of(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N, int K, int width,
                          cudaStream_t stream) {
    static AcornPerDevice configured;
    if (!configured.seen()) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_rows_kernel<R, CPL, NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             rs_smem<R, CPL>() < RS_ALONE ? RS_ALONE : rs_smem<R, CPL>());
        if (e != cudaSuccess) return (int)e;
        configured.mark();
    }
    const int sms = acorn_sms(), tiles = (int)(((int64_t)N + width - 1) / width);
    const int smem = tiles <= sms && rs_smem<R, CPL>() < RS_ALONE ? RS_ALONE : rs_smem<R, CPL>();
    return acorn_launch(gemm_f32_rows_kernel<R, CPL, NARROW>, dim3(CPL == 2 && sms < tiles ? sms : tiles), dim3(RS_THREADS), smem, stream, A,
                        lda, W, ldw, C, ldc, M, N, K, width);
}

template <int R, int CPL>
static int launch_rows(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N, int K,
                       cudaStream_t stream) {
    // Tiles of all columns that a block can take, or, where they would leave a fifth of the SMs' turns empty, of fewer: as many for
    // every SM, alike in width.  One row / 6 / 12 rows, us, whole tiles (at the second of 16 columns) / these: N = 2,560, K = 9,728 28.5, 36.4,
    // 49.5 / 25.4, 32.2, 42.7; N = 6,144, K = 1,024 8.1, 10.4, 12.8 / 6.5, 8.8, 10.4; N = 1,024, K = 3,072 6.2, 7.5, 11.7 / 5.3, 7.5, 10.9.
    // At fuller turns the columns that a warp leaves unused cost what the SMs gain (N = 4,096, K = 2,048 7.3, 8.5, 11.5 / 7.2, 8.6,
    // 12.1), and the form that knows its width at compile time is 2 to 7 % faster.
    const int sms = acorn_sms();
    const int64_t full = ((int64_t)N + 16 * CPL - 1) / (16 * CPL), turns = (full + sms - 1) / sms;
    const int even = (int)((N + turns * sms - 1) / (turns * sms));
    if (5 * full < 4 * turns * sms)
        return launch_rows_of<R, CPL, true>(A, lda, W, ldw, C, ldc, M, N, K, even < 4 ? 4 : even, stream);
    return launch_rows_of<R, CPL, false>(A, lda, W, ldw, C, ldc, M, N, K, 16 * CPL, stream);
}

template <bool SPLIT>
static int launch_tile(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N, int K,
                       cudaStream_t stream) {
    static AcornPerDevice configured;
    if (!configured.seen()) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_tile_kernel<SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, TL_SMEM);
        if (e != cudaSuccess) return (int)e;
        configured.mark();
    }
    const int tn = (N + TL_BN - 1) / TL_BN, tm = (M + TL_BM - 1) / TL_BM;
    if ((int64_t)tn * K_RANGES > 0x7fffffff) return ACORN_ERR_UNSUPPORTED;
    if (!SPLIT)
        return acorn_launch(gemm_f32_tile_kernel<SPLIT>, dim3(tn, tm), dim3(TL_THREADS), TL_SMEM, stream, A, lda, W, ldw,
                            C, ldc, M, N, K);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tn * K_RANGES, tm);
    cfg.blockDim = dim3(TL_THREADS);
    cfg.dynamicSmemBytes = TL_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = K_RANGES;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = acorn_pdl_enabled() ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_f32_tile_kernel<SPLIT>, A, lda, W, ldw, C, ldc, M, N, K);
    return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

extern "C" int acorn_gemm_f32(const float* A, int64_t lda, const float* W, int64_t ldw, float* C,
                              int64_t ldc, int M, int N, int K, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    constexpr int most = 65535 * TL_BM;          // rows a launch's grid covers (the plain kernel's tiles have as many)
    if (M > most) {
        const int rc = acorn_gemm_f32(A, lda, W, ldw, C, ldc, most, N, K, stream);
        return rc ? rc : acorn_gemm_f32(A + (int64_t)most * lda, lda, W, ldw, C + (int64_t)most * ldc, ldc, M - most, N, K, stream);
    }
    // the faster kernels move 16 bytes at a time along K
    const bool aligned = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
    if (aligned && M <= 16) {
        // Blocks of 32 columns read a row of A half as often for each weight: taken where blocks of 16 would give some SMs two or more
        // (more than 2,368 columns of 148 SMs).  N = 4,096, K = 2,048, blocks of 16 / 32: one row 8.0 / 7.2 us, 6 rows 9.9 / 8.5, 16
        // rows 18.0 / 13.4.
        const bool wide = N > 16 * acorn_sms();
        // As few rows a lane as hold them, since the reads of A set the pace.  (Two rows: one row a lane was slower, N = 6,144,
        // K = 1,024 8.5 us instead of 7.9, since both halves of a warp then read as much of W as of A.)
        switch (M == 2 ? 2 : (M + 1) / 2) {
#define ROWS(R) case R: return wide ? launch_rows<R, 2>(A, lda, W, ldw, C, ldc, M, N, K, stream) \
                                    : launch_rows<R, 1>(A, lda, W, ldw, C, ldc, M, N, K, stream)
            ROWS(1); ROWS(2); ROWS(3); ROWS(4); ROWS(5); ROWS(6); ROWS(7); ROWS(8);
#undef ROWS
        }
    }
    if (aligned && M <= 32 && (N <= 4096 || N >= 8192)) {
        // The weights twice through the rows kernel, half of the rows each: 32 rows, N = 2,048, K = 6,144: 54 us, in tiles 88 us;
        // N = 4,096, K = 1,024: 15 and 24 us; N = 12,288, K = 2,048: 77 and 93 us; between (N = 6,144, K = 1,024: 27 and 25 us) the
        // tiles fill the device.
        const int half = (M + 1) / 2;
        const int rc = acorn_gemm_f32(A, lda, W, ldw, C, ldc, half, N, K, stream);
        return rc ? rc : acorn_gemm_f32(A + half * lda, lda, W, ldw, C + half * ldc, ldc, M - half, N, K, stream);
    }
    if (aligned) {
        // A cluster to a tile where whole tiles would leave an SM fewer than two of them (777 rows, N = 1,024, K = 2,048, 104 tiles:
        // 131 us whole, 97 us split; 2,048 rows of the same, 256 tiles: 316 and 216 us; 777 rows, N = 4,096, K = 1,024, 416
        // tiles: 164 whole, 181 split), and a range of K is worth its share of the exchange.
        const int64_t tiles = (int64_t)((N + TL_BN - 1) / TL_BN) * ((M + TL_BM - 1) / TL_BM);
        if (tiles < 2 * acorn_sms() && K >= 256) return launch_tile<true>(A, lda, W, ldw, C, ldc, M, N, K, stream);
        return launch_tile<false>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    }
    dim3 grid((N + PL_BN - 1) / PL_BN, (M + PL_BM - 1) / PL_BM);
    gemm_f32_kernel<<<grid, 256, 0, stream>>>(A, lda, W, ldw, C, ldc, M, N, K);
    return acorn_launch_status();
}
