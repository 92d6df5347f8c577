// What the two decode attention kernels that take K and V by TMA share: the layout of a stage (64 keys of 128 dims, K then V, each
// in two swizzled halves) and the work of one warp on its 16 keys of it.
#pragma once

#include "mma_helpers.cuh"
#include "tcgen05_helpers.cuh"

#define DT_D 128
#define DT_CHUNK 64
#define DT_STAGES 3
#define DT_THREADS 160                      // 4 compute warps + 1 producer warp
#define DT_HALF_BYTES (DT_CHUNK * 128)      // [64 keys][64 dims] bf16
#define DT_STAGE_BYTES (4 * DT_HALF_BYTES)  // K half 0, K half 1, V half 0, V half 1

// byte offset of the 16-byte segment `seg` (0..15 over the 128 head dims) of key row `key` inside a
// K or V stage region (two swizzled halves of [64][128 bytes])
__device__ __forceinline__ uint32_t dt_swz(int key, int seg) {
    return (uint32_t)((seg >> 3) * DT_HALF_BYTES + key * 128 + (((seg & 7) ^ (key & 7)) << 4));
}

// The queries of a kv group's heads (rows of the mma's A operand, zeros from `rep` on).
__device__ __forceinline__ void dt_load_q(uint32_t (&qa)[DT_D / 16][4], const bf16* qrow, int rep, int lane) {
    const int g = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int ks = 0; ks < DT_D / 16; ++ks)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = g + (i & 1) * 8, col = ks * 16 + 2 * tq + (i >> 1) * 8;
            qa[ks][i] = row < rep ? *reinterpret_cast<const uint32_t*>(qrow + row * DT_D + col) : 0u;
        }
}

// One warp's 16 keys (the first is wkey0) of the stage at `kb`: scores, online softmax, values.  Keys outside [lo, hi) count nothing;
// at least one lies inside.
__device__ __forceinline__ void dt_chunk(float (&o)[DT_D / 8][4], float (&m_run)[2], float (&l_run)[2], const uint32_t (&qa)[DT_D / 16][4],
                                         uint32_t kb, int warp, int lane, int wkey0, int lo, int hi, float scale_log2) {
    const uint32_t vb = kb + 2 * DT_HALF_BYTES;
    const int mat = lane >> 3, rr = lane & 7, tq = lane & 3;
    float sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int ks = 0; ks < DT_D / 16; ++ks) {
        uint32_t b[4];
        ldmatrix_x4(b, kb + dt_swz(warp * 16 + (mat >> 1) * 8 + rr, ks * 2 + (mat & 1)));
        mma_bf16_16816(sc[0], qa[ks], b[0], b[1]);
        mma_bf16_16816(sc[1], qa[ks], b[2], b[3]);
    }
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int key = wkey0 + j * 8 + 2 * tq + (e & 1);
            sc[j][e] = (key < hi && key >= lo) ? sc[j][e] * scale_log2 : -INFINITY;
            mx[e >> 1] = fmaxf(mx[e >> 1], sc[j][e]);
        }
    float corr[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float mn = fmaxf(m_run[h], quad_max(mx[h]));  // finite: the group holds a valid key
        corr[h] = exp2f(m_run[h] - mn);
        m_run[h] = mn;
    }
    float psum[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            sc[j][e] = exp2f(sc[j][e] - m_run[e >> 1]);
            psum[e >> 1] += sc[j][e];
        }
    l_run[0] = l_run[0] * corr[0] + psum[0];
    l_run[1] = l_run[1] * corr[1] + psum[1];
    const uint32_t pa[4] = {pack_bf16(sc[0][0], sc[0][1]), pack_bf16(sc[0][2], sc[0][3]),
                            pack_bf16(sc[1][0], sc[1][1]), pack_bf16(sc[1][2], sc[1][3])};
#pragma unroll
    for (int n2 = 0; n2 < DT_D / 16; ++n2) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, vb + dt_swz(warp * 16 + (mat & 1) * 8 + rr, n2 * 2 + (mat >> 1)));
#pragma unroll
        for (int e = 0; e < 4; ++e) { o[2 * n2][e] *= corr[e >> 1]; o[2 * n2 + 1][e] *= corr[e >> 1]; }
        mma_bf16_16816(o[2 * n2], pa, b[0], b[1]);
        mma_bf16_16816(o[2 * n2 + 1], pa, b[2], b[3]);
    }
}
