// Recurrences over chunks of 64 tokens: which tokens a chunk holds, and how its rows come to shared memory.
//
// A row's chunks are counted from its first token of the step; chunk c of row r is number row_start[r] / 64 + r + c of the
// step (distinct for all chunks; some numbers stay unused).
#pragma once

#include "common.cuh"

#include <cfloat>

#define DC 64                       // tokens a chunk
#define DC_PAD 4                    // floats between rows in shared memory (16-byte reads of neighbouring rows hit distinct banks)

// The row and chunk of a chunk number, or false for an unused one.
__device__ __forceinline__ bool chunk_of(int id, const int* __restrict__ row_start, int rows, int& r, int& first, int& n) {
    int lo = 0, hi = rows - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (row_start[mid] / DC + mid <= id) lo = mid;
        else hi = mid - 1;
    }
    r = lo;
    const int start = row_start[lo], c = id - (start / DC + lo);
    first = start + c * DC;
    n = min(DC, row_start[lo + 1] - first);
    return n > 0;
}

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
