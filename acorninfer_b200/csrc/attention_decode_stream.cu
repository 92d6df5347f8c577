// Decode attention of many rows (bfloat16, head size 128): the chunks of 64 keys of all rows and kv heads in one line, cut into
// equal shares.
//
// The work on a chunk is that of attention_decode_tma.cu.  What differs is who takes it.  There a CTA takes one split of one
// (token, kv head), so rows of unequal lengths give CTAs of unequal work, a count of pairs just above what runs at once
// leaves a last wave nearly empty, and every CTA pays for its own start (lookups, the first tiles' latency) and end (the warps'
// merge) with its ring empty.  Here two CTAs an SM stay for the whole kernel and take
// one stretch each of the line [row][kv head][chunk]: the producer warp runs ahead across the borders of rows, so the ring stays full
// while a row's warps are merged.  A (row, kv head) that lies within a stretch is written at once; one that a border cuts leaves
// parts (at most two a CTA: one that began before, one that goes on after), which a second kernel merges.
// Bound by the memory and by the second kernel (3 to 4 us).  41 rows of 8 kv heads, 32 heads, 900 keys: 35.7 us (4.2 TB/s; a CTA
// a pair 43.7, in three splits 50.7); rows of 35 to 100 % of that 27.5 (28.5, 41.3).
#include "attention_decode_tile.cuh"

#define DS_MAX_ROWS 1024
#define DS_SMEM_MAX 115712               // half of an SM's 228 KB, less the 1 KB each CTA costs beside
#define DS_MAX_REP 8                        // query heads a kv head: two CTAs' rings and merge buffers fit an SM

__device__ int g_attn_dec_stream_error = 0;

struct DecodeStreamParams {
    const bf16* q;
    int64_t q_stride;
    bf16* out;
    const int* block_table;
    const int* page_base;
    const int* token_row;
    const int* positions;
    const int* token_list;
    float* part_o;           // [2 CTAs][rep][128]
    float* part_lse;         // [2 CTAs][rep]
    int n, ctas, table_stride, nq, nkv, logP, window;
    float scale_log2;
};

struct DsRow {
    int t, lo, hi, base_key, chunks;
};

__device__ __forceinline__ DsRow ds_row(const DecodeStreamParams& p, int ti) {
    DsRow r;
    r.t = p.token_list ? p.token_list[ti] : ti;
    const int pos = p.positions[r.t];
    r.lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
    r.hi = pos + 1;
    r.base_key = r.lo & ~(DT_CHUNK - 1);                            // chunks start at multiples of 64 keys
    r.chunks = (r.hi - r.base_key + DT_CHUNK - 1) / DT_CHUNK;
    return r;
}

// chunks a CTA's stretch holds
__device__ __forceinline__ int ds_share(int total, int ctas) { return max((total + ctas - 1) / ctas, 1); }

// `before[ti]`: chunks of all kv heads of the rows before ti; `before[n]`: of all rows.  Called by all threads.
__device__ __forceinline__ void ds_prefix(const DecodeStreamParams& p, int* before, int threads) {
    for (int ti = threadIdx.x; ti < p.n; ti += threads) before[ti + 1] = ds_row(p, ti).chunks * p.nkv;
    __syncthreads();
    if (threadIdx.x < 32) {
        int run = 0;
        for (int i = 0; i < p.n; i += 32) {
            int v = i + (int)threadIdx.x < p.n ? before[i + threadIdx.x + 1] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, v, o);
                if ((int)threadIdx.x >= o) v += up;
            }
            v += run;
            if (i + (int)threadIdx.x < p.n) before[i + threadIdx.x + 1] = v;
            run = __shfl_sync(0xffffffffu, v, 31);
        }
        if (threadIdx.x == 0) before[0] = 0;
    }
    __syncthreads();
}

// the row that holds chunk x of the line
__device__ __forceinline__ int ds_find(const int* before, int n, int x) {
    int lo = 0, hi = n;                                              // before[lo] <= x < before[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (before[mid] <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(DT_THREADS) attention_decode_stream_kernel(const __grid_constant__ CUtensorMap map_k,
                                                                            const __grid_constant__ CUtensorMap map_v,
                                                                            const DecodeStreamParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + DT_STAGES * DT_STAGE_BYTES);
    const uint32_t full0 = tc_smem(bars), empty0 = tc_smem(bars + DT_STAGES);
    const int rep = p.nq / p.nkv;
    float* sm_m = reinterpret_cast<float*>(bars + 2 * DT_STAGES + 2);   // [4][8]
    float* sm_l = sm_m + 4 * DS_MAX_REP;                                // [4][8]
    float* sm_o = sm_l + 4 * DS_MAX_REP;                                // [4][rep][128]
    int* before = reinterpret_cast<int*>(sm_o + 4 * rep * DT_D);        // [n + 1]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (tc_smem(smem) & 1023u) {
        if (threadIdx.x == 0) tc_fail(&g_attn_dec_stream_error, 9, ACORN_KERNEL_ATTN_DECODE_STREAM);
        return;
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < DT_STAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // Everything up to pdl_wait() reads only the step's own arrays (written by the host before the step).
    ds_prefix(p, before, DT_THREADS);
    const int total = before[p.n], share = ds_share(total, p.ctas);
    const int b = min(total, (int)blockIdx.x * share), e = min(total, b + share);

    if (warp == 4) {
        // ---- producer: lane l looks up the cache rows of the l-th TMA box (one page or 64 keys) of a batch of 32 boxes, a
        // batch ahead of the loads; an elected lane issues them
        const int P = 1 << p.logP;
        const int rows_per_op = P < DT_CHUNK ? P : DT_CHUNK;
        const int log_ops = 6 - (p.logP < 6 ? p.logP : 6);             // boxes a chunk: 64 / rows_per_op
        const int n_ops = (e - b) << log_ops;
        auto row_of = [&](int idx) -> int {                              // box idx of this CTA's stretch
            if (idx >= n_ops) return 0;
            const int x = b + (idx >> log_ops), ti = ds_find(before, p.n, x);
            const DsRow row = ds_row(p, ti);
            const int at = x - before[ti], kvh = at / row.chunks, c = at - kvh * row.chunks;
            const int r = p.token_row[row.t], first_page = p.page_base[r];
            int key = row.base_key + c * DT_CHUNK + (idx & ((1 << log_ops) - 1)) * rows_per_op;
            if (key >= row.hi) key = row.hi - 1 - ((row.hi - 1) & (rows_per_op - 1));  // masked later: any rows that exist
            key = max(key, first_page << p.logP);
            const int page = p.block_table[(int64_t)r * p.table_stride + (key >> p.logP) - first_page];
            return ((page * p.nkv + kvh) << p.logP) + (key & (P - 1));
        };
        int rows_next = row_of(lane);
        pdl_wait();
        pdl_trigger();
        bool good = true;
        for (int b0 = 0; b0 < n_ops && good; b0 += 32) {
            const int rows_cur = rows_next;
            if (b0 + 32 < n_ops) rows_next = row_of(b0 + 32 + lane);
            const int n_here = min(32, n_ops - b0);
            for (int l = 0; l < n_here; ++l) {
                const int idx = b0 + l, i = idx >> log_ops, k = idx & ((1 << log_ops) - 1), s = i % DT_STAGES;
                if (k == 0) {                                            // first box of a chunk: its stage must be free
                    bool got = mbar_wait(empty0 + 8 * s, ((i / DT_STAGES) & 1) ^ 1);
                    if (!got && lane == 0) tc_fail(&g_attn_dec_stream_error, 1, ACORN_KERNEL_ATTN_DECODE_STREAM);
                    good = __all_sync(0xffffffffu, got);
                    if (!good) break;
                    if (elect_one()) mbar_expect_tx(full0 + 8 * s, DT_STAGE_BYTES);
                }
                const int row = __shfl_sync(0xffffffffu, rows_cur, l);
                if (elect_one()) {
                    const uint32_t dst = tc_smem(smem + s * DT_STAGE_BYTES) + (uint32_t)(k * rows_per_op) * 128;
                    tma_load_2d(dst, &map_k, full0 + 8 * s, 0, row);
                    tma_load_2d(dst + DT_HALF_BYTES, &map_k, full0 + 8 * s, 64, row);
                    tma_load_2d(dst + 2 * DT_HALF_BYTES, &map_v, full0 + 8 * s, 0, row);
                    tma_load_2d(dst + 3 * DT_HALF_BYTES, &map_v, full0 + 8 * s, 64, row);
                }
            }
        }
        return;
    }
    // ---- compute warps
    pdl_wait();
    pdl_trigger();
    const int g = lane >> 2, tq = lane & 3;
    int i = 0;                                                           // chunks taken so far
    bool good = true;
    for (int x = b; x < e;) {
        const int ti = ds_find(before, p.n, x);
        const DsRow row = ds_row(p, ti);
        const int at = x - before[ti], kvh = at / row.chunks, c0 = at - kvh * row.chunks, c1 = min(row.chunks, c0 + e - x);
        uint32_t qa[DT_D / 16][4];
        dt_load_q(qa, p.q + (int64_t)row.t * p.q_stride + (int64_t)kvh * rep * DT_D, rep, lane);
        float o[DT_D / 8][4];
        float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
#pragma unroll
        for (int n = 0; n < DT_D / 8; ++n) { o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f; }
        for (int c = c0; c < c1 && good; ++c, ++i) {
            const int s = i % DT_STAGES;
            if (!mbar_wait(full0 + 8 * s, (i / DT_STAGES) & 1)) { tc_fail(&g_attn_dec_stream_error, 2, ACORN_KERNEL_ATTN_DECODE_STREAM); good = false; }
            good = __all_sync(0xffffffffu, good);
            if (!good) break;
            const int wkey0 = row.base_key + c * DT_CHUNK + warp * 16;  // first key of this warp's 16
            if (wkey0 < row.hi && wkey0 + 15 >= row.lo)
                dt_chunk(o, m_run, l_run, qa, tc_smem(smem + s * DT_STAGE_BYTES), warp, lane, wkey0, row.lo, row.hi, p.scale_log2);
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + 8 * s);
        }
        // the four warps' parts of this row's heads
        l_run[0] = quad_sum(l_run[0]);
        l_run[1] = quad_sum(l_run[1]);
        if (g < rep) {                                                   // rep <= 8: rows 8 .. of the tile hold nothing
            if (tq == 0) {
                sm_m[warp * DS_MAX_REP + g] = m_run[0];
                sm_l[warp * DS_MAX_REP + g] = l_run[0];
            }
#pragma unroll
            for (int n = 0; n < DT_D / 8; ++n)
                *reinterpret_cast<float2*>(sm_o + (warp * rep + g) * DT_D + n * 8 + 2 * tq) = make_float2(o[n][0], o[n][1]);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const bool whole = c0 == 0 && c1 == row.chunks;
        const int64_t slot = 2 * (int64_t)blockIdx.x + (c0 > 0 ? 0 : 1);
        for (int h = 0; h < rep; ++h) {
            const int d = threadIdx.x;
            float mstar = -INFINITY, L = 0.f, acc = 0.f;
#pragma unroll
            for (int w = 0; w < 4; ++w) mstar = fmaxf(mstar, sm_m[w * DS_MAX_REP + h]);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const float f = exp2f(sm_m[w * DS_MAX_REP + h] - mstar);
                L += sm_l[w * DS_MAX_REP + h] * f;
                acc += sm_o[(w * rep + h) * DT_D + d] * f;
            }
            if (whole) {
                p.out[((int64_t)row.t * p.nq + kvh * rep + h) * DT_D + d] = __float2bfloat16_rn(acc / L);
            } else {
                p.part_o[(slot * rep + h) * DT_D + d] = acc / L;
                if (d == 0) p.part_lse[slot * rep + h] = mstar + log2f(L);
            }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");                   // read before the next row's parts come
        x += c1 - c0;
    }
}

// Merges the parts of the (row, kv head)s that a border of the shares cuts; the others are written already.  A warp a head.
__global__ void __launch_bounds__(32 * DS_MAX_REP) attention_decode_stream_merge_kernel(const DecodeStreamParams p) {
    __shared__ int sums[2][DS_MAX_REP];
    const int ti = blockIdx.x, kvh = blockIdx.y, rep = p.nq / p.nkv, h = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const DsRow row = ds_row(p, ti);
    int mine = 0, all = 0;                                               // chunks of the rows before this one, of all rows
    for (int q = threadIdx.x; q < p.n; q += 32 * rep) {
        const int c = ds_row(p, q).chunks * p.nkv;
        all += c;
        if (q < ti) mine += c;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mine += __shfl_xor_sync(0xffffffffu, mine, o);
        all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    if (lane == 0) { sums[0][h] = mine; sums[1][h] = all; }
    __syncthreads();
    mine = all = 0;
    for (int w = 0; w < rep; ++w) { mine += sums[0][w]; all += sums[1][w]; }
    const int share = ds_share(all, p.ctas), first = mine + kvh * row.chunks;
    const int q0 = first / share, parts = (first + row.chunks - 1) / share - q0 + 1;
    pdl_wait();
    pdl_trigger();
    if (parts == 1) return;
    auto slot = [&](int q) { return (2 * (int64_t)(q0 + q) + (q == 0 ? 1 : 0)) * rep + h; };     // the first began at the row's first chunk
    float top = -INFINITY;
    for (int q = lane; q < parts; q += 32) top = fmaxf(top, p.part_lse[slot(q)]);
    top = warp_max(top);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float L = 0.f;
    for (int b = 0; b < parts; b += 32) {
        const float f = b + lane < parts ? exp2f(p.part_lse[slot(b + lane)] - top) : 0.f;
        L += f;
        const int here = min(32, parts - b);
#pragma unroll 4
        for (int q = 0; q < here; ++q) {
            const float g = __shfl_sync(0xffffffffu, f, q);
            const float4 o = reinterpret_cast<const float4*>(p.part_o + slot(b + q) * DT_D)[lane];
            acc.x += g * o.x; acc.y += g * o.y; acc.z += g * o.z; acc.w += g * o.w;
        }
    }
    L = warp_sum(L);
    Vec4<bf16>::store(p.out + ((int64_t)row.t * p.nq + kvh * rep + h) * DT_D + 4 * lane, make_float4(acc.x / L, acc.y / L, acc.z / L, acc.w / L));
}

// ------------------------------------------------------------------ host side

static size_t ds_smem(int rep, int n) {
    return (size_t)DT_STAGES * DT_STAGE_BYTES + (2 * DT_STAGES + 2) * 8 + (8 * DS_MAX_REP + 4 * rep * DT_D + n + 1) * 4;
}

// Whether rows of these sizes can be taken: two CTAs with their rings, merge buffers and the rows' prefix sums to an SM.
extern "C" int acorn_attention_decode_stream_supported(int nq, int nkv, int d, int P, int n) {
    return nkv > 0 && nq % nkv == 0 && nq / nkv <= DS_MAX_REP && d == DT_D && P >= 8 && (P & (P - 1)) == 0 && n > 0 &&
           n <= DS_MAX_ROWS && ds_smem(nq / nkv, n) <= DS_SMEM_MAX;
}

// part_o: 2 * ctas * (nq / nkv) rows of 128, part_lse: as many numbers.
extern "C" int acorn_attention_decode_stream(const void* q, int64_t q_stride, void* out, const void* k_pages, const void* v_pages,
                                             int64_t num_pages, const int* block_table, const int* page_base, int table_stride,
                                             const int* token_row, const int* positions, const int* token_list, int n, int nq, int nkv,
                                             int d, int P, float scale, int window, int ctas, float* part_o, float* part_lse,
                                             cudaStream_t stream) {
    if (n <= 0) return 0;
    if (!acorn_attention_decode_stream_supported(nq, nkv, d, P, n) || ctas < 1 || part_o == nullptr || part_lse == nullptr)
        return ACORN_ERR_UNSUPPORTED;
    DecodeStreamParams p;
    p.q = (const bf16*)q; p.q_stride = q_stride; p.out = (bf16*)out; p.block_table = block_table;
    p.page_base = page_base; p.token_row = token_row; p.positions = positions; p.token_list = token_list;
    p.part_o = part_o; p.part_lse = part_lse; p.n = n; p.ctas = ctas; p.table_stride = table_stride; p.nq = nq; p.nkv = nkv;
    p.logP = acorn_log2_exact_tc(P); p.window = window;
    p.scale_log2 = scale * 1.4426950408889634f;
    CUtensorMap mk, mv;
    const int box_rows = P < DT_CHUNK ? P : DT_CHUNK;
    int rc = make_map(&mk, k_pages, num_pages * nkv * P, d, d, 64, box_rows);
    if (rc) return rc;
    rc = make_map(&mv, v_pages, num_pages * nkv * P, d, d, 64, box_rows);
    if (rc) return rc;
    static AcornPerDevice configured;
    if (!configured.seen()) {
        cudaError_t e = cudaFuncSetAttribute(attention_decode_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DS_SMEM_MAX);
        if (e != cudaSuccess) return (int)e;
        configured.mark();
    }
    rc = acorn_launch(attention_decode_stream_kernel, dim3(ctas), dim3(DT_THREADS), ds_smem(nq / nkv, n), stream, mk, mv, p);
    if (rc) return rc;
    return acorn_launch(attention_decode_stream_merge_kernel, dim3(n, nkv), dim3(32 * (nq / nkv)), 0, stream, p);
}

extern "C" int acorn_attention_decode_stream_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_attn_dec_stream_error, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_attn_dec_stream_error, &zero, sizeof(int));
    return v;
}

ACORN_ERROR_WORD_SETTER(acorn_attention_decode_stream_set_error_word)
