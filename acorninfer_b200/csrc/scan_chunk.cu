// The linear recurrence of linear_recurrence.cu over chunks of 64 tokens (float32 throughout; long sums in parts of 16 or 32
// terms, which are then added: one chain over keys of 128 left c . b twice as far from 64 bits as the walk is):
//     S_i = a_i S_(i-1) + b_i (w_i x_i)^T,   y_i = S_i^T c_i + skip x_i,   a number a_i per token and head.
// With L_i the sum of log |a| up to i within the chunk (in double: differences of sums lose nothing that float32 would show),
// and the product of the decays' signs up to i beside it,
//     y = diag(exp(L)) C S_0 + P X + skip X,   P_ij = exp(L_i - L_j) w_j (c_i . b_j) for j <= i
//     S_end = exp(L_n) S_0 + sum_j exp(L_n - L_j) w_j b_j x_j^T
// (the block form of state space duality: Dao, Gu, "Transformers are SSMs").  Three kernels:
//   scan_chunk_sum    all chunks, heads and tiles of 64 columns side by side: what a chunk adds to the state
//   scan_chunk_fold   per state entry along a row's chunks: the state every chunk starts from, the end state into the slot
//   scan_chunk_out    all chunks and groups side by side: C B^T once for the heads that share the keys, then y head by head
//
// What bounds it: multiply-adds fed from shared memory (register tiles of 4 x 4 by 4 and of 8 x 4).  The walk over tokens it
// replaces for long rows is bound by the issue of dependent instructions, twice over in its two passes.  Measured (2,048
// tokens, B200): 64 heads of 64 columns, keys of 128, 8 groups: 492 -> 216 us; 16 heads of 128 columns, keys of 128:
// 277 -> 138 us.
#include "chunk_helpers.cuh"

#define SCO_VT 64                   // columns a block
#define SCO_LV (SCO_VT + DC_PAD)

struct ScanChunkParams {
    const float* b;  int64_t ldb;       // as ScanParams of linear_recurrence.cu
    const float* c;  int64_t ldc;
    const float* x;  int64_t ldx;
    const float* decay; int64_t lda;
    const float* w;  int64_t ldw;
    const float* skip;
    float* state; int64_t slot_stride;  // [H, V, N] of the row's slot
    float* y;                           // [T, H * V]
    const int* row_start;
    const int* row_slot;
    float* s0;                          // [chunk numbers, H, N, V]: the chunk's own sum, then the state it starts from
    float* dec;                         // [chunk numbers, H]: exp(L_n)
    int rows, H, G, N, V;
    int min_row;                        // rows of fewer tokens are left alone
};

// Sums of the logarithms of a chunk's decays, the products of their signs (1 or -1), and its step sizes times those, by one
// warp (two tokens a lane).  A decay of zero counts as exp(-1000): its products vanish as well.  What is no number stays none
// from its token on, and the tokens before do without it.
__device__ __forceinline__ void chunk_decays(const ScanChunkParams& p, int h, int first, int n, double* L, float* sign, float* w) {
    const int lane = threadIdx.x & 31;
    double v[2];
    bool neg[2];
    float step[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int i = 2 * lane + q;
        const int64_t t = first + i;
        const float a = i < n ? (p.lda ? p.decay[t * p.lda + h] : p.decay[h]) : 1.f;
        const double lg = log(fabs((double)a));
        v[q] = lg < -1000.0 ? -1000.0 : lg;
        neg[q] = a < 0.f;
        step[q] = i < n ? (p.w ? p.w[t * p.ldw + h] : 1.f) : 0.f;
    }
    double run = v[0] + v[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double before = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += before;
    }
    const double before = __shfl_up_sync(0xffffffffu, run, 1);
    L[2 * lane] = lane ? before + v[0] : v[0];
    L[2 * lane + 1] = run;
    const unsigned int below = (1u << lane) - 1, even = __ballot_sync(0xffffffffu, neg[0]), odd = __ballot_sync(0xffffffffu, neg[1]);
    const int count = __popc(even & below) + __popc(odd & below) + (neg[0] ? 1 : 0);
    const float s0 = count & 1 ? -1.f : 1.f, s1 = neg[1] ? -s0 : s0;
    sign[2 * lane] = s0;
    sign[2 * lane + 1] = s1;
    w[2 * lane] = step[0] * s0;
    w[2 * lane + 1] = step[1] * s1;
}

__device__ __forceinline__ void axpy4(float a, const float4& x, float4& y) {
    y.x = fmaf(a, x.x, y.x); y.y = fmaf(a, x.y, y.y); y.z = fmaf(a, x.z, y.z); y.w = fmaf(a, x.w, y.w);
}

template <int NP>
__global__ void __launch_bounds__(256) scan_chunk_sum_kernel(const ScanChunkParams p) {
    constexpr int LN = NP + DC_PAD, ND = NP / 64;
    extern __shared__ __align__(16) float sm[];
    float* sB = sm;                                     // [DC][LN]
    float* sX = sB + DC * LN;                           // [DC][SCO_LV], times exp(L_n - L_j) w_j
    __shared__ double L[DC];
    __shared__ float sign[DC], w[DC];
    pdl_wait();
    pdl_trigger();
    const int h = blockIdx.y, g = h / (p.H / p.G), v0 = blockIdx.z * SCO_VT, tid = threadIdx.x;
    int r, first, n;
    if (!chunk_of(blockIdx.x, p.row_start, p.rows, p.min_row, r, first, n)) return;
    load_rows<NP>(sB, p.b + (int64_t)first * p.ldb + (int64_t)g * p.N, p.ldb, n, p.N);
    asm volatile("cp.async.commit_group;\n" ::);
    if (tid < 32) chunk_decays(p, h, first, n, L, sign, w);
    __syncthreads();
    const double Ln = L[DC - 1];
    const float sign_n = sign[DC - 1];
    for (int e = tid; e < DC * (SCO_VT / 4); e += 256) {
        const int j = e / (SCO_VT / 4), c = (e % (SCO_VT / 4)) * 4;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < n && v0 + c < p.V) {
            x = *reinterpret_cast<const float4*>(p.x + (int64_t)(first + j) * p.ldx + (int64_t)h * p.V + v0 + c);
            const float f = expf((float)(Ln - L[j])) * (w[j] * sign_n);
            x = make_float4(x.x * f, x.y * f, x.z * f, x.w * f);
        }
        *reinterpret_cast<float4*>(sX + j * SCO_LV + c) = x;
    }
    if (tid == 0 && blockIdx.z == 0) p.dec[(int64_t)blockIdx.x * p.H + h] = expf((float)Ln) * sign_n;
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    const int tx = tid & 15, ty = tid >> 4;
    float4 acc[ND][4];
#pragma unroll
    for (int m = 0; m < ND; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[m][q] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int j = 0; j < DC; ++j) {
        const float4 x = *reinterpret_cast<const float4*>(sX + j * SCO_LV + 4 * tx);
#pragma unroll
        for (int m = 0; m < ND; ++m) {
            const float4 k = *reinterpret_cast<const float4*>(sB + j * LN + 4 * ty + 64 * m);
            axpy4(k.x, x, acc[m][0]); axpy4(k.y, x, acc[m][1]); axpy4(k.z, x, acc[m][2]); axpy4(k.w, x, acc[m][3]);
        }
    }
    float* E = p.s0 + ((int64_t)blockIdx.x * p.H + h) * p.N * p.V;
#pragma unroll
    for (int m = 0; m < ND; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int d = 4 * ty + 64 * m + q;
            if (d < p.N && v0 + 4 * tx < p.V) *reinterpret_cast<float4*>(E + (int64_t)d * p.V + v0 + 4 * tx) = acc[m][q];
        }
}

// A thread four columns of a key entry's state, along a row's chunks; the chunks' sums are fetched a few ahead.
__global__ void scan_chunk_fold_kernel(const ScanChunkParams p) {
    pdl_wait();
    pdl_trigger();
    const int h = blockIdx.y, V4 = p.V / 4;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    int r, id0;
    if (!row_of_block(blockIdx.z, p.row_start, p.rows, p.min_row, r, id0) || e >= p.N * V4) return;
    const int d = e / V4, v = (e % V4) * 4;
    const int chunks = (p.row_start[r + 1] - p.row_start[r] + DC - 1) / DC;
    float* slot = p.state + (int64_t)p.row_slot[r] * p.slot_stride + ((int64_t)h * p.V + v) * p.N + d;
    float4* E = reinterpret_cast<float4*>(p.s0 + ((int64_t)id0 * p.H + h) * p.N * p.V) + e;
    const float* a = p.dec + (int64_t)id0 * p.H + h;
    const int64_t step = (int64_t)p.H * p.N * V4;
    float4 cur = make_float4(slot[0], slot[p.N], slot[2 * p.N], slot[3 * p.N]);
    constexpr int AHEAD = 8;
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
        float4 x[AHEAD];
        float f[AHEAD];
#pragma unroll
        for (int q = 0; q < AHEAD; ++q) {
            const int c = min(c0 + q, chunks - 1);
            x[q] = E[c * step];
            f[q] = a[(int64_t)c * p.H];
        }
#pragma unroll
        for (int q = 0; q < AHEAD; ++q) {
            if (c0 + q >= chunks) break;
            E[(c0 + q) * step] = cur;
            cur = make_float4(fmaf(f[q], cur.x, x[q].x), fmaf(f[q], cur.y, x[q].y), fmaf(f[q], cur.z, x[q].z), fmaf(f[q], cur.w, x[q].w));
        }
    }
    slot[0] = cur.x; slot[p.N] = cur.y; slot[2 * p.N] = cur.z; slot[3 * p.N] = cur.w;
}

#define SCO_HEADS 8                 // heads a block of scan_chunk_out takes at most

// blockIdx.z: (share of the group's heads, tile of columns)
template <int NP>
__global__ void __launch_bounds__(256, 2) scan_chunk_out_kernel(const ScanChunkParams p, int per_block) {
    constexpr int LN = NP + DC_PAD;
    constexpr int BS = DC * LN > NP * SCO_LV ? DC * LN : NP * SCO_LV;
    extern __shared__ __align__(16) float sm[];
    float* sC = sm;                                     // [DC][LN]
    float* sB = sC + DC * LN;                           // [DC][LN], later a head's S_0 [NP][SCO_LV]
    float* sX = sB + BS;                                // [DC][SCO_LV]
    float* sP = sX + DC * SCO_LV;                       // [DC][DC + DC_PAD]
    constexpr int LP = DC + DC_PAD;
    __shared__ double L[SCO_HEADS][DC];
    __shared__ float sign[SCO_HEADS][DC], w[SCO_HEADS][DC];
    pdl_wait();
    pdl_trigger();
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int tiles = (p.V + SCO_VT - 1) / SCO_VT, rep = p.H / p.G;
    const int g = blockIdx.y, v0 = (blockIdx.z % tiles) * SCO_VT;
    const int h0 = g * rep + (blockIdx.z / tiles) * per_block, heads = min(per_block, (g + 1) * rep - h0);
    int r, first, n;
    if (!chunk_of(blockIdx.x, p.row_start, p.rows, p.min_row, r, first, n)) return;
    load_rows<NP>(sC, p.c + (int64_t)first * p.ldc + (int64_t)g * p.N, p.ldc, n, p.N);
    load_rows<NP>(sB, p.b + (int64_t)first * p.ldb + (int64_t)g * p.N, p.ldb, n, p.N);
    asm volatile("cp.async.commit_group;\n" ::);
    for (int q = tid >> 5; q < heads; q += 8) chunk_decays(p, h0 + q, first, n, L[q], sign[q], w[q]);
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    float M[4][4];                                      // c . b of rows ty + 16 ii and columns tx + 16 jj, jj <= ii
#pragma unroll
    for (int ii = 0; ii < 4; ++ii)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) M[ii][jj] = 0.f;
#pragma unroll 1
    for (int d0 = 0; d0 < NP; d0 += 16) {
        float part[4][4] = {};
#pragma unroll
        for (int d = d0; d < d0 + 16; d += 4) {
            float4 kj[4];
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) kj[jj] = *reinterpret_cast<const float4*>(sB + (tx + 16 * jj) * LN + d);
#pragma unroll
            for (int ii = 0; ii < 4; ++ii) {
                const float4 ci = *reinterpret_cast<const float4*>(sC + (ty + 16 * ii) * LN + d);
#pragma unroll
                for (int jj = 0; jj <= ii; ++jj) part[ii][jj] = dot4(ci, kj[jj], part[ii][jj]);
            }
        }
#pragma unroll
        for (int ii = 0; ii < 4; ++ii)
#pragma unroll
            for (int jj = 0; jj <= ii; ++jj) M[ii][jj] += part[ii][jj];
    }
    for (int q = 0; q < heads; ++q) {
        const int h = h0 + q;
        __syncthreads();                                // the head before is done with S_0, X and P (the first: with B)
        const float* S = p.s0 + ((int64_t)blockIdx.x * p.H + h) * p.N * p.V + v0;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int e = tid; e < DC * (SCO_VT / 4); e += 256) {
            const int j = e / (SCO_VT / 4), c = (e % (SCO_VT / 4)) * 4;
            if (j < n && v0 + c < p.V) dc_cp16(sX + j * SCO_LV + c, p.x + (int64_t)(first + j) * p.ldx + (int64_t)h * p.V + v0 + c);
            else *reinterpret_cast<float4*>(sX + j * SCO_LV + c) = zero;
        }
        for (int e = tid; e < NP * (SCO_VT / 4); e += 256) {
            const int d = e / (SCO_VT / 4), c = (e % (SCO_VT / 4)) * 4;
            if (d < p.N && v0 + c < p.V) dc_cp16(sB + d * SCO_LV + c, S + (int64_t)d * p.V + c);
            else *reinterpret_cast<float4*>(sB + d * SCO_LV + c) = zero;
        }
        asm volatile("cp.async.commit_group;\n" ::);
#pragma unroll
        for (int ii = 0; ii < 4; ++ii) {
            const int i = ty + 16 * ii;
            const double Li = L[q][i];
            const float sign_i = sign[q][i];
#pragma unroll
            for (int jj = 0; jj <= ii; ++jj) {
                const int j = tx + 16 * jj;
                sP[i * LP + j] = j <= i ? expf((float)(Li - L[q][j])) * (w[q][j] * sign_i) * M[ii][jj] : 0.f;
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::);
        bool odd = false;                               // an input that is no number: 0 times it would reach the tokens before
        for (int e = tid; e < DC * (SCO_VT / 4); e += 256)      // what this thread has brought
            odd |= not_finite(*reinterpret_cast<const float4*>(sX + (e / (SCO_VT / 4)) * SCO_LV + (e % (SCO_VT / 4)) * 4));
        odd = __syncthreads_or(odd);
        float4 acc[4];
#pragma unroll
        for (int ii = 0; ii < 4; ++ii) acc[ii] = zero;
#pragma unroll 1
        for (int d0 = 0; d0 < NP; d0 += 32) {
            float4 part[4] = {zero, zero, zero, zero};
#pragma unroll 2
            for (int d = d0; d < d0 + 32; d += 4) {
                float4 s[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) s[u] = *reinterpret_cast<const float4*>(sB + (d + u) * SCO_LV + 4 * tx);
#pragma unroll
                for (int ii = 0; ii < 4; ++ii) {
                    const float4 c4 = *reinterpret_cast<const float4*>(sC + (ty + 16 * ii) * LN + d);
                    axpy4(c4.x, s[0], part[ii]); axpy4(c4.y, s[1], part[ii]); axpy4(c4.z, s[2], part[ii]); axpy4(c4.w, s[3], part[ii]);
                }
            }
#pragma unroll
            for (int ii = 0; ii < 4; ++ii) acc[ii] = add4(acc[ii], part[ii]);
        }
#pragma unroll
        for (int ii = 0; ii < 4; ++ii) {
            const float e = expf((float)L[q][ty + 16 * ii]) * sign[q][ty + 16 * ii];
            acc[ii] = make_float4(acc[ii].x * e, acc[ii].y * e, acc[ii].z * e, acc[ii].w * e);
        }
        if (odd) {
            for (int j = 0; j < DC; ++j) {
                const float4 x = *reinterpret_cast<const float4*>(sX + j * SCO_LV + 4 * tx);
#pragma unroll
                for (int ii = 0; ii < 4; ++ii)
                    if (j <= ty + 16 * ii) axpy4(sP[(ty + 16 * ii) * LP + j], x, acc[ii]);
            }
        }
#pragma unroll
        for (int jb = 0; jb < 4; ++jb) {                // blocks of 16 tokens; rows before the block see none of it
            if (odd) break;
#pragma unroll
            for (int j = 16 * jb; j < 16 * jb + 16; j += 4) {
                float4 x[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) x[u] = *reinterpret_cast<const float4*>(sX + (j + u) * SCO_LV + 4 * tx);
#pragma unroll
                for (int ii = jb; ii < 4; ++ii) {
                    const float4 p4 = *reinterpret_cast<const float4*>(sP + (ty + 16 * ii) * LP + j);
                    axpy4(p4.x, x[0], acc[ii]); axpy4(p4.y, x[1], acc[ii]); axpy4(p4.z, x[2], acc[ii]); axpy4(p4.w, x[3], acc[ii]);
                }
            }
        }
        const float skip = p.skip ? p.skip[h] : 0.f;
#pragma unroll
        for (int ii = 0; ii < 4; ++ii) {
            const int i = ty + 16 * ii;
            if (i < n && v0 + 4 * tx < p.V) {
                axpy4(skip, *reinterpret_cast<const float4*>(sX + i * SCO_LV + 4 * tx), acc[ii]);
                *reinterpret_cast<float4*>(p.y + ((int64_t)(first + i) * p.H + h) * p.V + v0 + 4 * tx) = acc[ii];
            }
        }
    }
}

template <int NP> static int launch_scan_chunk(const ScanChunkParams& p, int ids, int walks, cudaStream_t stream) {
    constexpr int LN = NP + DC_PAD;
    constexpr int BS = DC * LN > NP * SCO_LV ? DC * LN : NP * SCO_LV;
    const size_t sum = (size_t)(DC * LN + DC * SCO_LV) * sizeof(float);
    const size_t out = (size_t)(DC * LN + BS + DC * SCO_LV + DC * (DC + DC_PAD)) * sizeof(float);
    static AcornPerDevice configured;
    if (!configured.seen()) {
        cudaError_t e = cudaFuncSetAttribute(scan_chunk_sum_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sum);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(scan_chunk_out_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out);
        if (e != cudaSuccess) return (int)e;
        configured.mark();
    }
    const int tiles = (p.V + SCO_VT - 1) / SCO_VT, rep = p.H / p.G;
    int rc = acorn_launch(scan_chunk_sum_kernel<NP>, dim3(ids, p.H, tiles), dim3(256), sum, stream, p);
    if (rc) return rc;
    rc = acorn_launch(scan_chunk_fold_kernel, dim3((p.N * (p.V / 4) + 255) / 256, p.H, walks), dim3(256), 0, stream, p);
    if (rc) return rc;
    // The heads of a group share C B^T, about 0.4 of a head's own work, so a block wants many of them, and the blocks that run
    // at a time (two to an SM) want to be filled: the share with the least estimated time.
    const int64_t at_once = 2 * acorn_sms();
    int best = 1;
    double best_cost = 1e30;
    for (int per = 1; per <= SCO_HEADS && per <= rep; ++per) {
        const int64_t blocks = (int64_t)ids * p.G * tiles * ((rep + per - 1) / per);
        const double cost = (double)((blocks + at_once - 1) / at_once) * (per + 0.4);
        if (cost < best_cost - 1e-9) { best_cost = cost; best = per; }
    }
    return acorn_launch(scan_chunk_out_kernel<NP>, dim3(ids, p.G, tiles * ((rep + best - 1) / best)), dim3(256), out, stream, p, best);
}

extern "C" int acorn_scan_chunk_supported(int N, int V) { return N >= 4 && N <= 128 && N % 4 == 0 && V >= 4 && V % 4 == 0; }

// Arguments as acorn_linear_scan (state at the first float of S in slot 0), for the rows of min_row tokens or more; s0 holds
// chunk_ids(tokens, rows, min_row) chunks of [H, N, V] floats, dec as many of [H].
extern "C" int acorn_scan_chunk(const float* b, int64_t ldb, const float* c, int64_t ldc, const float* x, int64_t ldx,
                                const float* decay, int64_t lda, const float* w, int64_t ldw, const float* skip, float* state,
                                int64_t slot_stride, float* y, const int* row_start, const int* row_slot, int tokens, int rows,
                                int H, int G, int N, int V, int min_row, float* s0, float* dec, cudaStream_t stream) {
    if (tokens <= 0 || rows <= 0) return 0;
    const uintptr_t all = (uintptr_t)b | (uintptr_t)c | (uintptr_t)x | (uintptr_t)y | (uintptr_t)s0;
    if (!acorn_scan_chunk_supported(N, V) || G < 1 || H < 1 || H % G || H > 65535 || rows > 65535 || (all & 15) || ldb % 4 ||
        ldc % 4 || ldx % 4)
        return ACORN_ERR_UNSUPPORTED;
    const int ids = chunk_ids(tokens, rows, min_row), walks = chunk_rows(tokens, rows, min_row);
    if (walks == 0) return 0;
    if ((int64_t)((V + SCO_VT - 1) / SCO_VT) * (H / G) > 65535) return ACORN_ERR_UNSUPPORTED;
    const ScanChunkParams p = {b, ldb, c, ldc, x, ldx, decay, lda, w, ldw, skip, state, slot_stride, y, row_start, row_slot, s0, dec,
                               rows, H, G, N, V, min_row};
    return N <= 64 ? launch_scan_chunk<64>(p, ids, walks, stream) : launch_scan_chunk<128>(p, ids, walks, stream);
}
