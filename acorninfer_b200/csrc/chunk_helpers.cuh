// Recurrences over chunks of 64 tokens: which tokens a chunk holds, and how its rows come to shared memory.
//
// A row's chunks are counted from its first token of the step; chunk c of row r is number row_start[r] / 64 + r + c of the
// step (distinct for all chunks; some numbers stay unused).
#pragma once

#include "common.cuh"

#include <cfloat>

#define DC 64                       // tokens a chunk
#define DC_PAD 4                    // floats between rows in shared memory (16-byte reads of neighbouring rows hit distinct banks)

// Where only rows of min_row > 0 tokens or more run over chunks (another kernel takes the others), theirs alone are counted,
// without gaps: a step of many decoded rows and one prompt launches the prompt's blocks and no others.

// Among the rows of min_row tokens or more, the one that holds chunk number `id` (CHUNKS) or that is number `id`; id0: the
// number of its first chunk.  By all lanes of a warp, four rows each at a time.
template <bool CHUNKS>
__device__ __forceinline__ bool find_row(int id, const int* __restrict__ row_start, int rows, int min_row, int& r, int& id0) {
    const int lane = threadIdx.x & 31;
    int chunks = 0;                                     // of the rows before this pass
    for (int base = 0; base < rows; base += 128) {
        const int at = base + 4 * lane;
        int start[5], c[4], own = 0, all = 0;
#pragma unroll
        for (int q = 0; q < 5; ++q) start[q] = row_start[min(at + q, rows)];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int len = start[q + 1] - start[q];    // 0 beyond the last row
            c[q] = len >= min_row ? (len + DC - 1) / DC : 0;
            own += CHUNKS ? c[q] : c[q] > 0;
            all += c[q];
        }
        int upto = own, chunks_upto = all;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, upto, o), y = __shfl_up_sync(0xffffffffu, chunks_upto, o);
            if (lane >= o) { upto += x; chunks_upto += y; }
        }
        const unsigned int past = __ballot_sync(0xffffffffu, upto > id);
        if (past) {
            int left = id - (upto - own), row = at, first = chunks + chunks_upto - all;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int n = CHUNKS ? c[q] : c[q] > 0;
                if (row == at + q && left >= n) { left -= n; first += c[q]; ++row; }
            }
            r = __shfl_sync(0xffffffffu, row, __ffs(past) - 1);
            id0 = __shfl_sync(0xffffffffu, first, __ffs(past) - 1);
            return true;
        }
        id -= __shfl_sync(0xffffffffu, upto, 31);
        chunks += __shfl_sync(0xffffffffu, chunks_upto, 31);
    }
    return false;
}

// The row and chunk of a chunk number, or false for an unused one.  By all threads of a warp.
__device__ __forceinline__ bool chunk_of(int id, const int* __restrict__ row_start, int rows, int min_row, int& r, int& first, int& n) {
    int lo = 0, hi = rows - 1, id0;
    if (min_row > 0) {
        if (!find_row<true>(id, row_start, rows, min_row, lo, id0)) return false;
    } else {
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (row_start[mid] / DC + mid <= id) lo = mid;
            else hi = mid - 1;
        }
        id0 = row_start[lo] / DC + lo;
    }
    r = lo;
    first = row_start[lo] + (id - id0) * DC;
    n = min(DC, row_start[lo + 1] - first);
    return n > 0;
}

// The row of a block that walks along a row's chunks, and the number of its first one.  By all threads of a warp.
__device__ __forceinline__ bool row_of_block(int z, const int* __restrict__ row_start, int rows, int min_row, int& r, int& id0) {
    if (min_row > 0) return find_row<false>(z, row_start, rows, min_row, r, id0);
    r = z;
    id0 = row_start[z] / DC + z;
    return true;
}

// Rows of min_row tokens or more that a step can hold, and their chunks.
static inline int chunk_rows(int tokens, int rows, int min_row) { return min_row > 0 && tokens / min_row < rows ? tokens / min_row : rows; }
static inline int chunk_ids(int tokens, int rows, int min_row) { return tokens / DC + chunk_rows(tokens, rows, min_row); }

__device__ __forceinline__ void dc_cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}

// n rows of `width` floats (a multiple of 4), ld apart, into DC rows of DP + DC_PAD; the rest zeros
template <int DP> __device__ __forceinline__ void load_rows(float* dst, const float* src, int64_t ld, int n, int width) {
    for (int e = threadIdx.x; e < DC * (DP / 4); e += blockDim.x) {
        const int i = e / (DP / 4), c = (e % (DP / 4)) * 4;
        float* d = dst + i * (DP + DC_PAD) + c;
        if (i < n && c < width) dc_cp16(d, src + (int64_t)i * ld + c);
        else *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

__device__ __forceinline__ float dot4(const float4& a, const float4& b, float acc) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}

__device__ __forceinline__ bool not_finite(const float4& v) {
    return !(fabsf(v.x) <= FLT_MAX && fabsf(v.y) <= FLT_MAX && fabsf(v.z) <= FLT_MAX && fabsf(v.w) <= FLT_MAX);
}

__device__ __forceinline__ float4 add4(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
