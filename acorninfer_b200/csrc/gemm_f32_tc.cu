// C[M, N] = A[M, K] * W[N, K]^T in float32 on the 5th-generation tensor cores, for prompts, many columns and long
// sums (acorninfer_b200/kernels/ops.py, gemm_f32_step): every operand, times 2^16, is the exact sum of three bfloat16 numbers,
// a = a0 + a1 + a2 (8 bits of mantissa each; rounding to nearest, so |a1| <= 2^-9 |a|, |a2| <= 2^-18 |a|), and a product is
// a0 b0 + (a0 b1 + a1 b0) + (a0 b2 + a1 b1 + a2 b0); what is left out (a1 b2 + a2 b1 + a2 b2) is at most 2^-26 |a b|, a quarter of a
// rounding of float32.  The scale takes float32's least number, 2^-149, to bfloat16's, 2^-133, so that no bit falls below: without it the
// parts of an operand of 2^-117 lost 4e-6 of it, of 2^-126 2e-3.  Operands from 2^112 and sums from 2^96 on overflow and go to f3_chain.
//
// The tensor cores round their sums towards zero, so no sum stays there for long.  K is cut into eight ranges of ceil(K / 512) * 64
// and a range into chunks of 64.  A chunk's sums are made in tensor memory: a0 b0 for every 16 of K apart, a single instruction each
// (added up there, the cut-off bits of sums of one sign had one sign, too: -6.6e-8 of the sum on average, now -1.3e-8), the lower
// products by their order of magnitude.  From there float32 adds, rounded to nearest, take them, the smaller ones apart: T += G over a
// range's chunks, and T0 + T1 + ... + T7 from the left.  That order does not depend on M, on the other rows or on who takes which
// range, so a row's bits do not either.
// Distance from 64 bits (relative 2-norm, K = 512 / 1,024 / 2,048 / 6,144), normally distributed operands: 7.5e-8, 8.0e-8, 8.6e-8,
// 1.0e-7 (the multiply-adds of gemm_f32.cu 1.6e-7, 2.1e-7, 2.9e-7, 5.0e-7); uniform in [0, 1): 5.0e-8, 5.2e-8, 5.0e-8, 5.2e-8 (6.1e-8,
// 7.3e-8, 9.0e-8, 1.5e-7).
//
// A CTA takes 128 rows of W (lanes of tensor memory) and 32 tokens.  Two groups of eight warps bring 64 floats of each row, split
// them and lay the parts out for the matrix instruction (K-major rows of 128 bytes, 128-byte swizzle; K permuted alike in both operands,
// so that a thread's 16 bytes of parts come from two coalesced loads); one warp multiplies: per 16 of K W0 x [b0], W0 x [b1 b2],
// W1 x [b0 b1] and W2 x [b0]; eight warps add up.  Only instructions of one shape on one accumulator are sure to run in the order they
// are issued in: columns that several add into belong to one shape (777 rows, N = 4,096, K = 1,024: 95 us with columns that shapes
// shared, 101 now).  A CTA holds all of tensor memory; its 197 KB of shared memory leave no room on the SM for a kernel
// that needs some, so that nobody waits for columns there.  Stages and accumulators are handed over by mbarriers; every wait is bounded.
//
// What bounds it: the loading warps, a load's latency and their arithmetic in turn (a chunk of 128 x 32 takes 1.0 us, of which shared
// memory's bytes take 0.55).  One group instead of two: 1.75 us; wider tiles of 48 and 64 tokens need registers that 25 warps do not
// have (spills: 1.7 and 2.0 us).  The products of a prompt of 777 rows (us, multiply-adds / this): N = 4,096, K = 1,024 164 / 101;
// N = 6,144 263 / 149; N = 1,024, K = 3,072 141 / 93; N = 12,288, K = 2,048 900 / 518 (75 TFLOP/s).
#include <cooperative_groups.h>

#include "tcgen05_helpers.cuh"

namespace cg = cooperative_groups;

#define F3_BM 128            // rows of W a tile
#define F3_NT 32             // tokens a tile
#define F3_BK 64             // floats of K a chunk
#define F3_RANGES 8
#define F3_SCALE 65536.f     // operands are split at this scale
#define F3_GROUP 8           // warps that load and split a chunk
#define F3_GROUPS 2          // such groups: they take turns
#define F3_LOADERS (F3_GROUP * F3_GROUPS)
#define F3_ADDERS 8          // warps that add up
#define F3_STAGES 3
#define F3_THREADS (32 * (F3_LOADERS + F3_ADDERS + 1))
#define F3_STAGE_BYTES (3 * (F3_BM + F3_NT) * 128)
#define F3_TOTAL_BYTES (F3_NT * F3_BM * 4)
#define F3_SMEM (F3_STAGES * F3_STAGE_BYTES + F3_TOTAL_BYTES + 1024 + 128)
#define F3_SUMS (7 * F3_NT)   // columns of a chunk's sums: W0 x b0 for every 16 of K, W0 x [b1 b2] + W1 x [b0 b1], W2 x b0
#define F3_TMEM_COLS 512     // two chunks' sums, a power of two

__device__ int g_gemm_f32_tc_error = 0;

struct F3Params {
    const float* a;
    const float* w;
    float* c;
    int64_t lda, ldw, ldc;
    int M, N, K;
    int range;               // floats of K a range
    int vec;                 // rows of both operands are made of aligned float4
    int tiles_m, tiles_n;
};

// Eight columns of 32 bits of this thread's lane from seven places F3_NT columns apart, one wait.
__device__ __forceinline__ void tmem_ld8x7(uint32_t at, float (&v)[7][8]) {
    uint32_t r[7][8];
#pragma unroll
    for (int q = 0; q < 7; ++q)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                     : "=r"(r[q][0]), "=r"(r[q][1]), "=r"(r[q][2]), "=r"(r[q][3]), "=r"(r[q][4]), "=r"(r[q][5]), "=r"(r[q][6]), "=r"(r[q][7])
                     : "r"(at + q * F3_NT));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < 7; ++q)
#pragma unroll
        for (int i = 0; i < 8; ++i) v[q][i] = __uint_as_float(r[q][i]);
}

// What float32 gives where a scaled sum is no number: chains of fused multiply-adds over ranges of K, as in gemm_f32.cu.  An operand that
// is infinite, NaN or, scaled, beyond bfloat16's largest number (2^112) makes every product of its row NaN above, and a sum from 2^96 on is
// infinite; such sums are made again here, up to the first NaN, which stays one
// (777 rows of nothing else, N = 4,096, K = 1,024: 13.8 ms to the end of K, 0.35 so; the multiply-adds 0.19).
static __device__ __noinline__ float f3_chain(const float* a, const float* w, int K) {
    const int range = (K + 127) / 128 * 16;
    float total = 0.f;
    for (int k0 = 0; k0 < K; k0 += range) {
        float acc = 0.f;
        const int end = min(K, k0 + range);
        for (int k1 = k0; k1 < end; k1 += 16) {
            for (int k = k1; k < min(end, k1 + 16); ++k) acc = fmaf(a[k], w[k], acc);
            if (acc != acc) return acc;
        }
        total = k0 == 0 ? acc : total + acc;
    }
    return total;
}

__device__ __forceinline__ void f3_store(const F3Params& p, int m, int n, float v) {
    const bool fine = fabsf(v) <= 3.0e38f;
    p.c[(int64_t)m * p.ldc + n] = fine ? v * (1.f / (F3_SCALE * F3_SCALE)) : f3_chain(p.a + (int64_t)m * p.lda, p.w + (int64_t)n * p.ldw, p.K);
}

__device__ __forceinline__ uint32_t f3_pack(float lo, float hi) {        // two bfloat16, rounded to nearest
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// Pairs of floats in the packed instructions of sm_100: a + b and F3_SCALE a, rounded as the single ones.
__device__ __forceinline__ float2 f3_add2(float2 a, float2 b) {
    unsigned long long r, x = *reinterpret_cast<unsigned long long*>(&a), y = *reinterpret_cast<unsigned long long*>(&b);
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return *reinterpret_cast<float2*>(&r);
}
__device__ __forceinline__ float2 f3_scale2(float2 a) {
    const float2 b = make_float2(F3_SCALE, F3_SCALE);
    unsigned long long r, x = *reinterpret_cast<unsigned long long*>(&a), y = *reinterpret_cast<const unsigned long long*>(&b);
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return *reinterpret_cast<float2*>(&r);
}

// What two floats leave beyond the bfloat16 numbers in p (exact): fused multiply-adds of mixed precision, p times -1 (0xbf80) on the floats.
// Unpacking p for a subtraction in float32 takes twice the instructions (777 rows, N = 12,288, K = 2,048: 512 us, unpacked 604).
__device__ __forceinline__ float2 f3_rest(float2 v, uint32_t p) {
    float2 r;
    asm("{\n .reg .b16 lo, hi, minus;\n mov.b32 {lo, hi}, %4;\n mov.b16 minus, 0xbf80;\n"
        " fma.rn.f32.bf16 %0, lo, minus, %2;\n fma.rn.f32.bf16 %1, hi, minus, %3;\n}\n"
        : "=f"(r.x), "=f"(r.y) : "f"(v.x), "f"(v.y), "r"(p));
    return r;
}

// The three parts of eight floats times F3_SCALE, 16 bytes each.
__device__ __forceinline__ void f3_split(const float (&x)[8], uint4 (&part)[3]) {
    uint32_t p[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 v = f3_scale2(make_float2(x[2 * i], x[2 * i + 1]));
        p[0][i] = f3_pack(v.x, v.y);
        v = f3_rest(v, p[0][i]);
        p[1][i] = f3_pack(v.x, v.y);
        v = f3_rest(v, p[1][i]);
        p[2][i] = f3_pack(v.x, v.y);             // exact
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) part[q] = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
}

// SPLIT: a cluster of eight CTAs shares a tile, a range of K each; else a CTA walks tiles, the next one's loads under way while
// the last sums of one are added.
template <bool SPLIT>
__global__ void __launch_bounds__(F3_THREADS, 1) gemm_f32_tc_kernel(const F3Params p) {
    constexpr int NT = F3_NT, STAGES = F3_STAGES, STAGE = F3_STAGE_BYTES, ADDERS = F3_ADDERS;
    constexpr int PART_W = F3_BM * 128, PART_A = NT * 128, COLS = F3_TMEM_COLS;
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(F3_BM >> 4) << 24);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (tc_smem(smem_raw) & 1023u)) & 1023u);
    float* totals = reinterpret_cast<float*>(smem + STAGES * STAGE);             // the ranges' sum so far, [token][row of W]
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE + F3_TOTAL_BYTES);   // full[S], empty[S], sum_full[2], sum_empty[2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    const uint32_t full0 = tc_smem(bars), empty0 = tc_smem(bars + STAGES), sfull0 = tc_smem(bars + 2 * STAGES),
                   sempty0 = tc_smem(bars + 2 * STAGES + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int part = SPLIT ? (int)(blockIdx.x % F3_RANGES) : 0;
    const int first = SPLIT ? (int)(blockIdx.x / F3_RANGES) : (int)blockIdx.x;
    const int step = SPLIT ? 0x40000000 : (int)gridDim.x;
    const int tiles = p.tiles_m * p.tiles_n;
    const int kbeg = SPLIT ? min(p.K, part * p.range) : 0, kend = SPLIT ? min(p.K, kbeg + p.range) : p.K;
    const int chunks = (kend - kbeg + F3_BK - 1) / F3_BK;

    // the first weights on their way to L2 while the kernel before this one ends (W may be its result: not read yet)
    if (warp < F3_GROUP && chunks > 0) {
        const int n = min(first / p.tiles_m * F3_BM + (int)(threadIdx.x >> 1), p.N - 1), k = kbeg + (threadIdx.x & 1) * 32;
        if (k < kend) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.w + (int64_t)n * p.ldw + k));
        if (k + F3_BK < kend) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.w + (int64_t)n * p.ldw + k + F3_BK));
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8 * s, F3_GROUP); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(sfull0 + 8 * b, 1); mbar_init(sempty0 + 8 * b, ADDERS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == F3_LOADERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(tc_smem(tmem_slot)), "r"((uint32_t)COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    pdl_trigger();

    if (warp < F3_LOADERS) {
        // ---- load and split.  A unit: 8 floats of a row, k = 4 j .. and 32 + 4 j .. of the chunk; a thread has units of four
        // of the tile's W rows and of one token.  It asks for its group's next chunk as it stores this one's; the
        // fence behind the stores waits for those loads too, so two groups take turns: one waits, one splits.
        constexpr int WU = F3_BM / 32, UNITS = WU + 1;
        const int group = warp / F3_GROUP, row0 = (threadIdx.x >> 3) & 31, j = threadIdx.x & 7;
        float x[UNITS][8];
        int off[UNITS];                            // of the units' rows in W and A (the host sees that 32 bits hold them)
        auto place = [&](int tile) {
            const int tn = tile / p.tiles_m, tm = tile - tn * p.tiles_m;
#pragma unroll
            for (int u = 0; u < UNITS; ++u)        // rows beyond the matrix: another row's values, never written
                off[u] = u < WU ? min(tn * F3_BM + 32 * u + row0, p.N - 1) * (int)p.ldw : min(tm * NT + row0, p.M - 1) * (int)p.lda;
        };
        auto fetch = [&](int u, int k, bool inner, float (&v)[8]) {
            const float* src = (u < WU ? p.w : p.a) + off[u];
            if (inner) {
                const float4 lo = *reinterpret_cast<const float4*>(src + k), hi = *reinterpret_cast<const float4*>(src + k + 32);
                v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
            } else {                               // the last chunk of a range that 64 does not divide, or unaligned rows
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int kk = k + (e & 3) + 32 * (e >> 2);
                    v[e] = kk < kend ? src[kk] : 0.f;
                }
            }
        };
        auto inside = [&](int chunk) { return p.vec && kbeg + (chunk + 1) * F3_BK <= kend; };
        int tile = first, chunk = 0;
        auto advance = [&](int by) {                           // `by` chunks on, into the next tiles
            chunk += by;
            while (tile < tiles && chunk >= chunks) {
                chunk -= chunks;
                tile += step;
            }
        };
        if (chunks > 0) advance(group);
        else tile = tiles;
        if (tile < tiles) {
            place(tile);
#pragma unroll
            for (int u = 0; u < UNITS; ++u) fetch(u, kbeg + chunk * F3_BK + 4 * j, inside(chunk), x[u]);
        }
        for (int it = group; tile < tiles; it += F3_GROUPS) {
            const int s = it % STAGES;
            bool ok = mbar_wait(empty0 + 8 * s, ((it / STAGES) & 1) ^ 1);
            if (!ok && lane == 0) tc_fail(&g_gemm_f32_tc_error, 1, ACORN_KERNEL_GEMM_F32_TC);
            if (!__all_sync(0xffffffffu, ok)) break;
            const int was = tile;
            advance(F3_GROUPS);
            const bool more = tile < tiles, inner = inside(chunk);
            const int k = kbeg + chunk * F3_BK + 4 * j;
            if (more && tile != was) place(tile);
            uint8_t* base = smem + s * STAGE + (row0 >> 3) * 1024 + (row0 & 7) * 128 + ((j ^ (row0 & 7)) << 4);
#pragma unroll
            for (int u = 0; u < UNITS; ++u) {
                uint4 parts[3];
                f3_split(x[u], parts);
                if (more) fetch(u, k, inner, x[u]);
                uint8_t* dst = base + (u < WU ? 4096 * u : 3 * PART_W);
#pragma unroll
                for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(dst + q * (u < WU ? PART_W : PART_A)) = parts[q];
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(full0 + 8 * s);
        }
    } else if (warp == F3_LOADERS) {
        // ---- multiply (the warp stays converged, an elected lane issues)
        const uint32_t w0 = umma_lo(tc_smem(smem)), a0 = umma_lo(tc_smem(smem) + 3 * PART_W);
        constexpr uint32_t I1 = IDESC | ((uint32_t)(NT >> 3) << 17), I2 = IDESC | ((uint32_t)(2 * NT >> 3) << 17);
        int it = 0;
        bool ok = true;
        for (int tile = first; ok && tile < tiles; tile += step) {
            for (int chunk = 0; chunk < chunks; ++chunk, ++it) {
                const int s = it % STAGES, b = it & 1;
                ok = mbar_wait(sempty0 + 8 * b, ((it >> 1) & 1) ^ 1);
                if (ok) ok = mbar_wait(full0 + 8 * s, (it / STAGES) & 1);
                if (!ok && lane == 0) tc_fail(&g_gemm_f32_tc_error, 2, ACORN_KERNEL_GEMM_F32_TC);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tmem + b * F3_SUMS;
                const uint32_t w = w0 + s * (STAGE >> 4), a = a0 + s * (STAGE >> 4);
#pragma unroll
                for (int k = 0; k < F3_BK / 16; ++k) {
                    umma_bf16_elect(d + k * NT, w + 2 * k, a + 2 * k, I1, 0u);
                    umma_bf16_elect(d + 4 * NT, w + 2 * k, a + 2 * k + (PART_A >> 4), I2, k > 0 ? 1u : 0u);
                    umma_bf16_elect(d + 4 * NT, w + 2 * k + (PART_W >> 4), a + 2 * k, I2, 1u);
                    umma_bf16_elect(d + 6 * NT, w + 2 * k + 2 * (PART_W >> 4), a + 2 * k, I1, k > 0 ? 1u : 0u);
                }
                umma_commit_elect(empty0 + 8 * s);
                umma_commit_elect(sfull0 + 8 * b);
            }
        }
    } else {
        // ---- add up: warp w reads lanes 32 (w % 4) .. of tensor memory, its share of the tokens
        constexpr int MINE = 4 * NT / ADDERS;                  // tokens a warp
        const int aw = warp - F3_LOADERS - 1, quarter = warp & 3, t0 = (aw >> 2) * MINE;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        const int range_chunks = p.range / F3_BK;
        int it = 0;
        bool ok = true;
        for (int tile = first; ok && tile < tiles; tile += step) {
            float2 sum[MINE / 2];
#pragma unroll
            for (int i = 0; i < MINE / 2; ++i) sum[i] = make_float2(0.f, 0.f);
            float* mine = totals + t0 * F3_BM + quarter * 32 + lane;
            bool folded = false;
            int in_range = 0;
            for (int chunk = 0; chunk < chunks; ++chunk, ++it) {
                if (!SPLIT && in_range == range_chunks) {
                    in_range = 0;
#pragma unroll
                    for (int i = 0; i < MINE / 2; ++i) {
                        float* at = mine + 2 * i * F3_BM;
                        at[0] = folded ? at[0] + sum[i].x : sum[i].x;
                        at[F3_BM] = folded ? at[F3_BM] + sum[i].y : sum[i].y;
                        sum[i] = make_float2(0.f, 0.f);
                    }
                    folded = true;
                }
                ++in_range;
                const int b = it & 1;
                ok = mbar_wait(sfull0 + 8 * b, (it >> 1) & 1);
                if (!ok && lane == 0) tc_fail(&g_gemm_f32_tc_error, 3, ACORN_KERNEL_GEMM_F32_TC);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const uint32_t at = tmem + lanes + b * F3_SUMS + t0;
#pragma unroll
                for (int c = 0; c < MINE; c += 8) {
                    float g[7][8];                             // W0 b0 four times; W0 b1 + W1 b0, W0 b2 + W1 b1; W2 b0
                    tmem_ld8x7(at + c, g);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        auto two = [&](int q) { return make_float2(g[q][2 * i], g[q][2 * i + 1]); };
                        const float2 lower = f3_add2(two(4), f3_add2(two(5), two(6)));
                        const float2 first = f3_add2(f3_add2(two(0), two(1)), f3_add2(two(2), two(3)));
                        sum[c / 2 + i] = f3_add2(sum[c / 2 + i], f3_add2(first, lower));
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(sempty0 + 8 * b);
            }
            if (!ok) break;
            if (SPLIT) {
#pragma unroll
                for (int i = 0; i < MINE; ++i) mine[i * F3_BM] = i & 1 ? sum[i / 2].y : sum[i / 2].x;
            } else {
                const int tn = tile / p.tiles_m, tm = tile - tn * p.tiles_m;
                const int n = tn * F3_BM + quarter * 32 + lane, m = tm * NT + t0;
                if (n < p.N) {
#pragma unroll
                    for (int i = 0; i < MINE; ++i) {
                        const float v = i & 1 ? sum[i / 2].y : sum[i / 2].x;
                        if (m + i < p.M) f3_store(p, m + i, n, folded ? mine[i * F3_BM] + v : v);
                    }
                }
            }
        }
    }
    if (SPLIT) {
        __syncwarp();
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        const int tn = first / p.tiles_m, tm = first - tn * p.tiles_m;
        constexpr int SHARE = NT * F3_BM / F3_RANGES;
        for (int o = threadIdx.x; o < SHARE; o += F3_THREADS) {
            const int at = part * SHARE + o, m = tm * NT + at / F3_BM, n = tn * F3_BM + at % F3_BM;
            float v[F3_RANGES];
#pragma unroll
            for (int q = 0; q < F3_RANGES; ++q) v[q] = cluster.map_shared_rank(totals, q)[at];
#pragma unroll
            for (int q = 1; q < F3_RANGES; ++q) v[0] += v[q];
            if (m < p.M && n < p.N) f3_store(p, m, n, v[0]);
        }
        cluster.sync();                          // a CTA's shared memory stays until all have read it
    }
    tc_fence_before();
    __syncthreads();
    if (warp == F3_LOADERS)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"((uint32_t)COLS) : "memory");
}

// ------------------------------------------------------------------ host side

template <bool SPLIT>
static int f3_launch(const F3Params& p, int grid, cudaStream_t stream) {
    static AcornPerDevice configured;
    if (!configured.seen()) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, F3_SMEM);
        if (e != cudaSuccess) return (int)e;
        configured.mark();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(F3_THREADS);
    cfg.dynamicSmemBytes = F3_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = F3_RANGES;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = acorn_pdl_enabled() ? attr : attr + 1;
    cfg.numAttrs = (acorn_pdl_enabled() ? 1 : 0) + (SPLIT ? 1 : 0);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_f32_tc_kernel<SPLIT>, p);
    return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// Offsets of both operands' elements fit 32 bits.
static bool f3_takes(int64_t M, int64_t N, int64_t lda, int64_t ldw) { return M * lda <= 0x7fffffff && N * ldw <= 0x7fffffff; }

// split 1: a cluster of eight CTAs to a tile, 0: whole tiles, -1: chosen here.  Any alignment.
extern "C" int acorn_gemm_f32_tc(const float* A, int64_t lda, const float* W, int64_t ldw, float* C, int64_t ldc, int M, int N, int K,
                                 int split, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || !f3_takes(M, N, lda, ldw)) return ACORN_ERR_UNSUPPORTED;
    F3Params p = {};
    p.a = A; p.w = W; p.c = C; p.lda = lda; p.ldw = ldw; p.ldc = ldc; p.M = M; p.N = N; p.K = K;
    p.range = (K + F3_BK * F3_RANGES - 1) / (F3_BK * F3_RANGES) * F3_BK;
    p.vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
    p.tiles_m = (M + F3_NT - 1) / F3_NT;
    p.tiles_n = (N + F3_BM - 1) / F3_BM;
    const int64_t tiles = (int64_t)p.tiles_m * p.tiles_n, sms = acorn_sms();
    if (tiles * F3_RANGES > 0x3fffffff) return ACORN_ERR_UNSUPPORTED;
    if (split < 0) {
        // Clusters where few tiles leave SMs idle: a chunk takes 1.0 us, a cluster's start, exchange and end 7 us beside its
        // chunks (128 rows, N = 1,024, K = 2,048, 32 tiles: 32 us whole, 23 in clusters; 256 rows: 32 and 39).
        const int64_t chunks = (K + F3_BK - 1) / F3_BK, part = p.range / F3_BK;
        split = K >= 4 * F3_BK && (tiles * F3_RANGES + sms - 1) / sms * (part + 7) < (tiles + sms - 1) / sms * chunks;
    }
    return split ? f3_launch<true>(p, (int)tiles * F3_RANGES, stream) : f3_launch<false>(p, (int)(tiles < sms ? tiles : sms), stream);
}

// Reads and clears the flag that a bounded wait sets when it gives up (0 = no error).
extern "C" int acorn_gemm_f32_tc_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_gemm_f32_tc_error, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_gemm_f32_tc_error, &zero, sizeof(int));
    return v;
}

ACORN_ERROR_WORD_SETTER(acorn_gemm_f32_tc_set_error_word)
