// Paged causal attention in float32 for head sizes 64 and 128: the float32 engine's kernels where the plain one
// (attention_plain.cu) leaves most of the device waiting.  Same meaning as there, for a causal mask with or without a
// window: the query at position p of a row reads keys lo..p of the row's pages, query head h reads kv head
// h / (nq / nkv), scores (q . k) * scale, softmax and the weighted sum in float32.
//
//   prefill   rows of two tokens or more: a block takes 64 queries of one head and walks the keys 64 at a time;
//             both products are register tiles of packed pairs of multiply-adds fed from shared memory;
//   decode    rows of one token: a block takes 128 keys of one kv head for all of its query heads, a second kernel
//             puts a row's blocks together.
//
// Key blocks and the runs of 512 (128) keys that a block takes start at multiples of their size, and a key that a query does
// not read adds exact zeros (nothing at all where its values are not finite), so a query's bits do not depend on the other
// queries of its tile, on the step's other rows or on padding.
//
// What bounded the plain kernel: a block a token read every key row again from L2 and made one chain of adds per thread.
// Measured (B200, launched alone): 777 tokens, 16 heads of 128: 1,402 -> 141 us; 6 rows of 1,500 keys, 8 kv heads:
// 109 -> 14 us (74 MB, which L2 holds).
//
// What bounds the prefill kernel: shared memory, whose reads into registers (8 of 16 bytes a lane for 32 packed multiply-adds of the
// scores, 3 for 16 of the sum) take 1.75 times the multiply-adds' time; 8,000 tokens run at half the multiply-adds' rate.  Eight
// queries a thread, which need a quarter fewer reads on half the warps, were no faster: 141 -> 148 us at 777 tokens, 31 -> 38 at 130.
// Short steps end with their longest blocks, so those of all heads come first (heads along the grid's first axis): 151 -> 141 us at 777
// tokens, 198 -> 161 at 1,000, 564 -> 529 at 2,000, 31 at 130 and 7,150 at 8,000 either way.
#include "mma_helpers.cuh"

#include <cfloat>

typedef unsigned long long f32x2_t;

__device__ __forceinline__ f32x2_t pair_of(float lo, float hi) {
    f32x2_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpair(f32x2_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ void fma_pair(f32x2_t& acc, f32x2_t a, f32x2_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ void mul_pair(f32x2_t& acc, f32x2_t a) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(a)); }

// ------------------------------------------------------------------ prefill

#define FP_Q 64
#define FP_K 64
#define FP_CHUNK 512            // keys a block walks at most: a tile late in a long prompt is several blocks' work
#define FP_THREADS 256

// Q and V rows are read whole by half warps (no padding); K rows by sixteen lanes at once (a pad of 16 bytes keeps them
// in different banks).  At head size 128 two blocks exactly fill an SM's shared memory.
template <int D> constexpr int fp_smem() { return (FP_Q * D + FP_K * (D + 4) + FP_K * D + FP_Q * FP_K) * (int)sizeof(float); }

// The partial results of a query in `n` slots from `slot` on: dimension d of their sum.
template <int D>
__device__ __forceinline__ void merge_parts(const float* __restrict__ part_o, const float* __restrict__ part_ml, float* __restrict__ out,
                                            int64_t slot, int n, int d) {
    float top = -INFINITY;
    for (int c = 0; c < n; ++c) top = fmaxf(top, part_ml[(slot + c) * 2]);
    float sum = 0.f, acc = 0.f;
#pragma unroll 4
    for (int c = 0; c < n; ++c) {
        const float w = expf(part_ml[(slot + c) * 2] - top);
        sum += w * part_ml[(slot + c) * 2 + 1];
        acc += w * part_o[(slot + c) * D + d];
    }
    out[d] = acc / sum;
}

template <int D>
__global__ void __launch_bounds__(FP_THREADS, 2) attention_f32_prefill_kernel(
    const float* __restrict__ q, int64_t q_stride, float* __restrict__ out, const float* __restrict__ k_pages,
    const float* __restrict__ v_pages, const int* __restrict__ block_table, const int* __restrict__ page_base, int table_stride,
    const int* __restrict__ row_start, const int* __restrict__ row_pos, const int* __restrict__ tiles, int n_tiles, int nq,
    int nkv, int P, float scale, int window, int chunks, float* __restrict__ part_o, float* __restrict__ part_ml) {
    extern __shared__ __align__(16) float fp_buf[];
    float* Qs = fp_buf;                             // [64][D], scaled
    float* Ks = Qs + FP_Q * D;                      // [64][D + 4]
    float* Vs = Ks + FP_K * (D + 4);                // [64][D]
    float* Ps = Vs + FP_K * D;                      // [64][64]
    constexpr int DC = D / 64;                      // runs of 64 dimensions; a thread holds four of each
    pdl_wait();
    pdl_trigger();
    const int tile = n_tiles - 1 - blockIdx.y;      // later tiles of a row read more keys: of all heads they start first
    const int r = tiles[2 * tile], q0 = tiles[2 * tile + 1];
    const int h = blockIdx.x, kvh = h / (nq / nkv);
    const int t0 = row_start[r] + q0, n = min(FP_Q, row_start[r + 1] - t0), p0 = row_pos[r] + q0;
    const int* table = block_table + (int64_t)r * table_stride - page_base[r];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // this block's share of the tile's keys: those of one run of FP_CHUNK positions
    const int lo0 = window > 0 ? max(0, p0 - window + 1) : 0, chunk0 = lo0 / FP_CHUNK, c = blockIdx.z;
    const int first = max(lo0, (chunk0 + c) * FP_CHUNK), last = min(p0 + n - 1, (chunk0 + c + 1) * FP_CHUNK - 1);
    if (first > p0 + n - 1) return;
    const int shift = __ffs(P) - 1;

    constexpr int CHUNKS = D / 4;                   // 16-byte pieces of a row
    auto load = [&](float* dst, int ld, const float* pages, int kb) {
#pragma unroll
        for (int e = 0; e < FP_K * CHUNKS / FP_THREADS; ++e) {
            const int c = e * FP_THREADS + threadIdx.x, key = c / CHUNKS, seg = (c % CHUNKS) * 4, j = kb + key;
            const bool valid = j >= first && j <= last;
            const int64_t at = valid ? ((int64_t)table[j >> shift] * nkv + kvh) * P + (j & (P - 1)) : 0;
            cp_async_16(smem_addr(dst + key * ld + seg), pages + at * D + seg, valid);
        }
        cp_async_commit();
    };

    const int kb0 = first & ~(FP_K - 1);
    load(Ks, D + 4, k_pages, kb0);
    load(Vs, D, v_pages, kb0);
    for (int c = threadIdx.x; c < FP_Q * CHUNKS; c += FP_THREADS) {
        const int row = c / CHUNKS, seg = (c % CHUNKS) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < n) {
            const float* src = q + (int64_t)(t0 + row) * q_stride + (int64_t)h * D + seg;
            v = make_float4(src[0] * scale, src[1] * scale, src[2] * scale, src[3] * scale);
        }
        *reinterpret_cast<float4*>(Qs + row * D + seg) = v;
    }

    f32x2_t acc[4][2 * DC];                         // rows ty * 4 + i, dimensions run * 64 + tx * 4 .. + 3
    float m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 2 * DC; ++j) acc[i][j] = 0ull;
    }
    for (int kb = kb0; kb <= last; kb += FP_K) {
        cp_async_wait<1>();                         // the keys have landed (the values may still be on their way)
        __syncthreads();
        // scores of rows ty * 4 + i and keys tx + 16 j: even and odd dimensions summed side by side
        f32x2_t s2[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s2[i][j] = 0ull;
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
            ulonglong2 b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(Ks + (tx + 16 * j) * (D + 4) + d);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(Qs + (ty * 4 + i) * D + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    fma_pair(s2[i][j], a.x, b[j].x);
                    fma_pair(s2[i][j], a.y, b[j].y);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = p0 + ty * 4 + i, lo = window > 0 ? pos - window + 1 : 0;
            float s[4], top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float even, odd;
                unpair(s2[i][j], even, odd);
                const int key = kb + tx + 16 * j;
                s[j] = key <= min(pos, last) && key >= max(lo, first) ? even + odd : -INFINITY;
                top = fmaxf(top, s[j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float m_new = fmaxf(m[i], top);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float p = s[j] == -INFINITY ? 0.f : expf(s[j] - m_new);
                Ps[(ty * 4 + i) * FP_K + tx + 16 * j] = p;
                sum += p;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            const float corr = m_new == -INFINITY ? 1.f : expf(m[i] - m_new);     // m = -inf: 0
            l[i] = l[i] * corr + sum;
            m[i] = m_new;
            const f32x2_t c2 = pair_of(corr, corr);
#pragma unroll
            for (int j = 0; j < 2 * DC; ++j) mul_pair(acc[i][j], c2);
        }
        cp_async_wait<0>();                         // the values
        // a block that some queries see in part: in a sum over all of it 0 times a value that is no number would reach them
        bool odd = false;
        if (kb + FP_K - 1 > p0 || (window > 0 && kb < p0 + n - window)) {
#pragma unroll
            for (int e = 0; e < FP_K * CHUNKS / FP_THREADS; ++e) {
                const int c = e * FP_THREADS + threadIdx.x;             // what this thread has brought
                const float4 v = *reinterpret_cast<const float4*>(Vs + c * 4);
                odd |= !(fabsf(v.x) <= FLT_MAX && fabsf(v.y) <= FLT_MAX && fabsf(v.z) <= FLT_MAX && fabsf(v.w) <= FLT_MAX);
            }
        }
        odd = __syncthreads_or(odd);                // and the probabilities; the keys' room is free
        if (kb + FP_K <= last) load(Ks, D + 4, k_pages, kb + FP_K);
        if (odd) {
            for (int k = 0; k < FP_K; ++k) {
                f32x2_t v[2 * DC];
#pragma unroll
                for (int c = 0; c < DC; ++c) {
                    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(Vs + k * D + c * 64 + tx * 4);
                    v[2 * c] = w.x;
                    v[2 * c + 1] = w.y;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int pos = p0 + ty * 4 + i, key = kb + k;
                    const float pv = Ps[(ty * 4 + i) * FP_K + k];
                    const f32x2_t pp = pair_of(pv, pv);
                    if (key <= pos && (window <= 0 || key > pos - window))
#pragma unroll
                        for (int j = 0; j < 2 * DC; ++j) fma_pair(acc[i][j], pp, v[j]);
                }
            }
        } else {
#pragma unroll 2
            for (int k = 0; k < FP_K; k += 4) {
                float4 p[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(Ps + (ty * 4 + i) * FP_K + k);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    f32x2_t v[2 * DC];
#pragma unroll
                    for (int c = 0; c < DC; ++c) {
                        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(Vs + (k + u) * D + c * 64 + tx * 4);
                        v[2 * c] = w.x;
                        v[2 * c + 1] = w.y;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float pv = u == 0 ? p[i].x : u == 1 ? p[i].y : u == 2 ? p[i].z : p[i].w;
                        const f32x2_t pp = pair_of(pv, pv);
#pragma unroll
                        for (int j = 0; j < 2 * DC; ++j) fma_pair(acc[i][j], pp, v[j]);
                    }
                }
            }
        }
        __syncthreads();                            // the values' room is free
        if (kb + FP_K <= last) load(Vs, D, v_pages, kb + FP_K);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = ty * 4 + i, pos = p0 + row;
        if (row >= n || pos < first) continue;
        // a query all of whose keys lie in one run is done here; the others' runs are put together by the merge kernel
        const int lo = window > 0 ? max(0, pos - window + 1) : 0, own0 = lo / FP_CHUNK;
        if (first > pos || chunk0 + c < own0) continue;
        const bool whole = pos / FP_CHUNK == own0;
        const int64_t slot = (((int64_t)tile * FP_Q + row) * nq + h) * chunks + (chunk0 + c - own0);
        float* dst = whole ? out + ((int64_t)(t0 + row) * nq + h) * D : part_o + slot * D;
        const float f = whole ? l[i] : 1.f;
        if (!whole && tx == 0) {
            part_ml[2 * slot] = m[i];
            part_ml[2 * slot + 1] = l[i];
        }
#pragma unroll
        for (int q4 = 0; q4 < DC; ++q4) {
            float4 o;
            unpair(acc[i][2 * q4], o.x, o.y);
            unpair(acc[i][2 * q4 + 1], o.z, o.w);
            *reinterpret_cast<float4*>(dst + q4 * 64 + tx * 4) = make_float4(o.x / f, o.y / f, o.z / f, o.w / f);
        }
    }
}

// A query whose keys lie in several runs: its runs put together.
template <int D>
__global__ void __launch_bounds__(D) attention_f32_prefill_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                                                        float* __restrict__ out, const int* __restrict__ row_start,
                                                                        const int* __restrict__ row_pos, const int* __restrict__ tiles,
                                                                        int nq, int window, int chunks) {
    pdl_wait();
    pdl_trigger();
    const int tile = blockIdx.x / FP_Q, row = blockIdx.x % FP_Q, h = blockIdx.y, d = threadIdx.x;
    const int r = tiles[2 * tile], q0 = tiles[2 * tile + 1] + row, t = row_start[r] + q0;
    if (t >= row_start[r + 1]) return;
    const int pos = row_pos[r] + q0, lo = window > 0 ? max(0, pos - window + 1) : 0, n = pos / FP_CHUNK - lo / FP_CHUNK + 1;
    if (n == 1) return;
    merge_parts<D>(part_o, part_ml, out + ((int64_t)t * nq + h) * D, ((int64_t)blockIdx.x * nq + h) * chunks, n, d);
}

// ------------------------------------------------------------------ decode

#define FD_KEYS 128             // keys a block takes
#define FD_THREADS 128

// A block takes keys 128 c .. of one (row, kv head) for G of its query heads.  Eight lanes share a key row in the scores
// (each 16 bytes of every 128), a warp a value row in the sum.
template <int D, int G>
__global__ void __launch_bounds__(FD_THREADS) attention_f32_decode_kernel(
    const float* __restrict__ q, int64_t q_stride, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
    const int* __restrict__ block_table, const int* __restrict__ page_base, int table_stride, const int* __restrict__ token_row,
    const int* __restrict__ positions, const int* __restrict__ token_list, int nq, int nkv, int P, float scale, int window,
    int chunks, float* __restrict__ part_o, float* __restrict__ part_ml) {
    constexpr int C = D / 32;                       // 16-byte pieces of a key row a lane takes
    constexpr int VL = D / 4, VK = 32 / VL;         // lanes a value row takes, value rows a warp reads at once
    __shared__ __align__(16) float qs[G * D];
    __shared__ float sc[G][FD_KEYS];
    __shared__ int64_t row_at[FD_KEYS];
    __shared__ float sums[4][VK][G][D];
    pdl_wait();
    pdl_trigger();
    const int t = token_list ? token_list[blockIdx.x] : blockIdx.x;
    const int parts = nq / nkv / G, kvh = blockIdx.y / parts, h0 = kvh * (nq / nkv) + (blockIdx.y % parts) * G;
    const int r = token_row[t], pos = positions[t];
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;
    const int kb = (lo / FD_KEYS + blockIdx.z) * FD_KEYS;
    if (kb > pos) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int* table = block_table + (int64_t)r * table_stride - page_base[r];
    for (int i = tid; i < G * D; i += FD_THREADS) qs[i] = q[(int64_t)t * q_stride + (int64_t)h0 * D + i] * scale;
    {
        const int j = min(max(kb + tid, lo), pos);  // a key that the row does not read: one that it does, with no weight
        row_at[tid] = (((int64_t)table[j / P] * nkv + kvh) * P + j % P) * D;
    }
    __syncthreads();
    const int sub = lane & 7;
#pragma unroll 4
    for (int e = 0; e < 8; ++e) {
        const int key = warp * 32 + e * 4 + (lane >> 3);
        const int64_t at = row_at[key];
        float dot[G];
#pragma unroll
        for (int g = 0; g < G; ++g) dot[g] = 0.f;
        float4 k[C];
#pragma unroll
        for (int c = 0; c < C; ++c) k[c] = *reinterpret_cast<const float4*>(k_pages + at + c * 32 + sub * 4);
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float4 w = *reinterpret_cast<const float4*>(qs + g * D + c * 32 + sub * 4);
                dot[g] = fmaf(w.x, k[c].x, dot[g]);
                dot[g] = fmaf(w.y, k[c].y, dot[g]);
                dot[g] = fmaf(w.z, k[c].z, dot[g]);
                dot[g] = fmaf(w.w, k[c].w, dot[g]);
            }
#pragma unroll
        for (int g = 0; g < G; ++g) {
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) dot[g] += __shfl_xor_sync(0xffffffffu, dot[g], o);
            if (sub == 0) sc[g][key] = kb + key >= lo && kb + key <= pos ? dot[g] : -INFINITY;
        }
    }
    __syncthreads();
    const int64_t slot = ((int64_t)blockIdx.x * nq + h0) * chunks + blockIdx.z;
    if (warp < G) {
        float s[4], top = -INFINITY, sum = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            s[i] = sc[warp][lane + 32 * i];
            top = fmaxf(top, s[i]);
        }
        top = warp_max(top);                        // the block holds a key of the row: finite unless a score is not
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float p = s[i] == -INFINITY ? 0.f : expf(s[i] - top);
            sc[warp][lane + 32 * i] = p;
            sum += p;
        }
        sum = warp_sum(sum);
        if (lane == 0) {
            part_ml[(slot + (int64_t)warp * chunks) * 2] = top;
            part_ml[(slot + (int64_t)warp * chunks) * 2 + 1] = sum;
        }
    }
    __syncthreads();
    float4 acc[G];
#pragma unroll
    for (int g = 0; g < G; ++g) acc[g] = make_float4(0.f, 0.f, 0.f, 0.f);
    const int vk = lane / VL, vd = (lane % VL) * 4;
#pragma unroll 8
    for (int e = 0; e < 32 / VK; ++e) {
        const int key = warp * 32 + e * VK + vk;
        const int64_t at = row_at[key];
        const float4 v = *reinterpret_cast<const float4*>(v_pages + at + vd);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float p = sc[g][key];
            acc[g].x = fmaf(p, v.x, acc[g].x);
            acc[g].y = fmaf(p, v.y, acc[g].y);
            acc[g].z = fmaf(p, v.z, acc[g].z);
            acc[g].w = fmaf(p, v.w, acc[g].w);
        }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) *reinterpret_cast<float4*>(&sums[warp][vk][g][vd]) = acc[g];
    __syncthreads();
    for (int i = tid; i < G * D; i += FD_THREADS) {
        const int g = i / D, d = i % D;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w)
#pragma unroll
            for (int k = 0; k < VK; ++k) v += sums[w][k][g][d];
        part_o[(slot + (int64_t)g * chunks) * D + d] = v;
    }
}

template <int D>
__global__ void __launch_bounds__(D) attention_f32_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                                                float* __restrict__ out, const int* __restrict__ positions,
                                                                const int* __restrict__ token_list, int nq, int window, int chunks) {
    pdl_wait();
    pdl_trigger();
    const int t = token_list ? token_list[blockIdx.x] : blockIdx.x, h = blockIdx.y, d = threadIdx.x;
    const int pos = positions[t], lo = window > 0 ? max(0, pos - window + 1) : 0;
    const int n = pos / FD_KEYS - lo / FD_KEYS + 1;
    merge_parts<D>(part_o, part_ml, out + ((int64_t)t * nq + h) * D, ((int64_t)blockIdx.x * nq + h) * chunks, n, d);
}

// ------------------------------------------------------------------ host side

extern "C" int acorn_attention_f32_supported(int nq, int nkv, int d) {
    return (d == 64 || d == 128) && nkv >= 1 && nq % nkv == 0 && nq <= 65535;
}

template <int D>
static int launch_prefill(const float* q, int64_t q_stride, float* out, const float* k_pages, const float* v_pages,
                          const int* block_table, const int* page_base, int table_stride, const int* row_start, const int* row_pos,
                          const int* tiles, int n_tiles, int nq, int nkv, int P, float scale, int window, int chunks, float* part_o,
                          float* part_ml, cudaStream_t stream) {
    static AcornPerDevice configured;
    if (!configured.seen()) {
        cudaError_t e = cudaFuncSetAttribute(attention_f32_prefill_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, fp_smem<D>());
        if (e != cudaSuccess) return (int)e;
        configured.mark();
    }
    int code = 0;                                   // 65,535 tiles a launch: what the grid's second axis takes
    for (int at = 0; at < n_tiles && code == 0; at += 65535) {
        const int n = min(n_tiles - at, 65535);
        const int64_t slots = (int64_t)at * FP_Q * nq * chunks;
        code = acorn_launch(attention_f32_prefill_kernel<D>, dim3(nq, n, chunks), dim3(FP_THREADS), fp_smem<D>(), stream, q, q_stride, out,
                            k_pages, v_pages, block_table, page_base, table_stride, row_start, row_pos, tiles + 2 * at, n, nq, nkv, P,
                            scale, window, chunks, chunks > 1 ? part_o + slots * D : part_o, chunks > 1 ? part_ml + slots * 2 : part_ml);
    }
    if (code != 0 || chunks == 1) return code;
    return acorn_launch(attention_f32_prefill_merge_kernel<D>, dim3(n_tiles * FP_Q, nq), dim3(D), 0, stream, part_o, part_ml, out, row_start,
                        row_pos, tiles, nq, window, chunks);
}

// `chunks`: runs of FP_CHUNK positions that a tile's keys can touch, at most; part_o [tiles, 64, nq, chunks, d], part_ml
// [tiles, 64, nq, chunks, 2] (unused for one run).
extern "C" int acorn_attention_f32_prefill(const float* q, int64_t q_stride, float* out, const float* k_pages, const float* v_pages,
                                           const int* block_table, const int* page_base, int table_stride, const int* row_start,
                                           const int* row_pos, const int* tiles, int n_tiles, int nq, int nkv, int d, int P,
                                           float scale, int window, int chunks, float* part_o, float* part_ml, cudaStream_t stream) {
    if (n_tiles <= 0) return 0;
    if (!acorn_attention_f32_supported(nq, nkv, d) || chunks < 1 || chunks > 65535) return ACORN_ERR_UNSUPPORTED;
    auto* run = d == 128 ? launch_prefill<128> : launch_prefill<64>;
    return run(q, q_stride, out, k_pages, v_pages, block_table, page_base, table_stride, row_start, row_pos, tiles, n_tiles, nq, nkv, P,
               scale, window, chunks, part_o, part_ml, stream);
}

template <int D, int G>
static int launch_decode(const float* q, int64_t q_stride, float* out, const float* k_pages, const float* v_pages,
                         const int* block_table, const int* page_base, int table_stride, const int* token_row, const int* positions,
                         const int* token_list, int n, int nq, int nkv, int P, float scale, int window, int chunks, float* part_o,
                         float* part_ml, cudaStream_t stream) {
    const int code = acorn_launch(attention_f32_decode_kernel<D, G>, dim3(n, nq / G, chunks), dim3(FD_THREADS), 0, stream, q, q_stride,
                                  k_pages, v_pages, block_table, page_base, table_stride, token_row, positions, token_list, nq, nkv, P,
                                  scale, window, chunks, part_o, part_ml);
    if (code != 0) return code;
    return acorn_launch(attention_f32_merge_kernel<D>, dim3(n, nq), dim3(D), 0, stream, part_o, part_ml, out, positions, token_list, nq,
                        window, chunks);
}

// `chunks`: blocks of 128 positions that a row's keys can touch, at most; part_o [n, nq, chunks, d], part_ml [n, nq, chunks, 2].
extern "C" int acorn_attention_f32_decode(const float* q, int64_t q_stride, float* out, const float* k_pages, const float* v_pages,
                                          const int* block_table, const int* page_base, int table_stride, const int* token_row,
                                          const int* positions, const int* token_list, int n, int nq, int nkv, int d, int P,
                                          float scale, int window, int chunks, float* part_o, float* part_ml, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (!acorn_attention_f32_supported(nq, nkv, d) || chunks < 1 || chunks > 65535) return ACORN_ERR_UNSUPPORTED;
    const int rep = nq / nkv, g = rep % 4 == 0 ? 4 : rep % 2 == 0 ? 2 : 1;
    auto* run = d == 128 ? (g == 4 ? launch_decode<128, 4> : g == 2 ? launch_decode<128, 2> : launch_decode<128, 1>)
                         : (g == 4 ? launch_decode<64, 4> : g == 2 ? launch_decode<64, 2> : launch_decode<64, 1>);
    return run(q, q_stride, out, k_pages, v_pages, block_table, page_base, table_stride, token_row, positions, token_list, n, nq, nkv, P,
               scale, window, chunks, part_o, part_ml, stream);
}
