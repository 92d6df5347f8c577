// Latent attention of long rows on the 5th-generation tensor cores (tcgen05), bfloat16: every head of a token reads the
// same cached row of d entries, whose first dv are the values too (the general kernel, for short rows and other sizes:
// latent_attention.cu).  d and dv multiples of 64, d <= 448, dv <= 384.
//
// One CTA per tile of 128 (token, head) rows, which lie one after another in q [tokens * H, d], against the keys its
// tokens see, in blocks of 64: S = Q K^T and O += P K[:, :dv], accumulators in tensor memory.  The queries stay in shared
// memory (7 x 16 KB at d = 448) beside two blocks of keys (56 KB each), so a block's columns come and go in groups of 128:
// a group of the block after next is brought as soon as the value product has read the group it takes the place of.
//   warps 0-3  softmax: thread r owns row r (= TMEM lane r): reads its 64 scores, masks, exponentiates in float32 base 2
//              against a reference maximum, writes P over them, as two bfloat16 numbers each (the nearest, and what that
//              lacks); O is rescaled only when a row's maximum outgrew its reference by 2^8.  At the end: O divided by the row's sum (and the sink's term), written out.
//   warps 4, 6, 7  producers: TMA loads of the queries (once) and, through the block table, of the keys, a third of a block's
//              boxes each (a block is 28 boxes of a page of 16 keys by 64 entries, and one warp issues a box in about 90 ns:
//              alone it set the pace, 3.1 us a block).
//   warp 5     MMA issuer (converged, one elected lane), blocks in pairs: P V of two blocks, then Q K of the next two.  (Q K
//              of block j + 1 ahead of P V of block j takes the same time.)
// Tensor memory (512 columns): S / P of even and odd blocks at 0 and 64, O at 128 ..
// P as one bfloat16 number was 11 % further from 64 bits than the general kernel in rows that a few keys decide (1.92e-3 and
// 1.74e-3 of the result, scores of standard deviation 3): there a row's largest weight is a power of two and not rounded, which
// here it is not unless O is rescaled with every new maximum.
//
// A block costs the tensor pipe 28 steps of N = 64 (48 clocks each, the reads of shared memory bound them) and 24 of
// N = 128 (64 clocks): 1.5 us at d = 448, dv = 384.  Measured 3.0 us, 1.95 us at d = 192, dv = 128 (56 rows of 4,000 keys; with
// P as one number 2.65 and 1.7 us): a block's own chain, its keys' way from L2, scores, softmax, values, is what bounds it, not
// the rates.
// Measured (B200, launched alone, rows of 448 with 384 values, 16 heads), the general kernel and this: 2,000 tokens under a
// window of 1,024 358 -> 97 us, 3 x 601 tokens 162 -> 54 us, 2,000 tokens behind 4,000 2,164 -> 428 us.
// A tile in which a value row that only some of its queries read holds an infinity or no number is computed again at the end,
// a row at a time: in a product, 0 times such a value would reach the queries that do not read it.
// Every mbarrier wait is bounded; a wait that gives up records g_latent_tc_error and the CTA drains.
#include "tcgen05_helpers.cuh"

#define LT_M 128
#define LT_KB 64
#define LT_THREADS 256
#define LT_PRODUCERS 3                   // warps 4, 6, 7
#define LT_RESCALE_LOG2 8.0f
#define LT_Q_PIECE (LT_M * 128)          // bytes: 64 entries of every row
#define LT_K_PIECE (LT_KB * 128)
#define LT_GROUPS 4                      // groups of 128 columns a block's keys come in, at most
#define LT_MAX_PIECES 7                  // queries and two blocks of keys within 227 KB
#define LT_BARS (1 + 2 * 2 * LT_GROUPS + 2 + 2 + 2)

__device__ int g_latent_tc_error = 0;

struct LatentTcParams {
    bf16* out;               // [tokens * H, dv]
    const bf16* q;           // [tokens * H, d]
    const bf16* pages;       // [pages, P, d]
    const int* block_table;
    const int* page_base;
    const int* row_start;
    const int* row_pos;
    const float* sink;       // [H] or null
    int table_stride, num_rows, H, d, dv, logP, window;
    float scale_log2;
};

__device__ __forceinline__ float lt_max(const float (&s)[64]) {
    float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int c = 0; c < 64; c += 4) {
        m[0] = fmaxf(m[0], s[c]); m[1] = fmaxf(m[1], s[c + 1]);
        m[2] = fmaxf(m[2], s[c + 2]); m[3] = fmaxf(m[3], s[c + 3]);
    }
    return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
}

// Whether one of eight bfloat16 entries is infinite or no number.
__device__ __forceinline__ bool lt_not_finite(const uint4& v) {
    auto full = [](uint32_t w) { return ((w & 0x7f807f80u) + 0x00800080u) & 0x80008000u; };       // an exponent of all ones
    return (full(v.x) | full(v.y) | full(v.z) | full(v.w)) != 0;
}

// One (token, head) row by one warp, key by key, float32 throughout.
__device__ __noinline__ void latent_row_alone(const LatentTcParams& p, const int* table, int64_t row, int head, int qpos) {
    const int lane = threadIdx.x & 31, P = 1 << p.logP;
    float q[2 * LT_MAX_PIECES], o[2 * LT_MAX_PIECES], m = -INFINITY, l = 0.f;
#pragma unroll
    for (int i = 0; i < 2 * LT_MAX_PIECES; ++i) {
        const int e = lane + 32 * i;
        q[i] = e < p.d ? to_float(p.q[row * p.d + e]) : 0.f;
        o[i] = 0.f;
    }
    for (int key = p.window > 0 ? max(0, qpos - p.window + 1) : 0; key <= qpos; ++key) {
        const bf16* k = p.pages + (((int64_t)table[key >> p.logP] << p.logP) + (key & (P - 1))) * p.d;
        float kv[2 * LT_MAX_PIECES], s = 0.f;
#pragma unroll
        for (int i = 0; i < 2 * LT_MAX_PIECES; ++i) {
            const int e = lane + 32 * i;
            kv[i] = e < p.d ? to_float(k[e]) : 0.f;
            s = fmaf(q[i], kv[i], s);
        }
        s = warp_sum(s) * p.scale_log2;
        const float top = fmaxf(m, s), corr = m == -INFINITY ? 0.f : exp2f(m - top), w = s == -INFINITY ? 0.f : exp2f(s - top);
        m = top;
        l = l * corr + w;
#pragma unroll
        for (int i = 0; i < 2 * LT_MAX_PIECES; ++i) o[i] = o[i] * corr + w * kv[i];
    }
    if (p.sink) l += exp2f(p.sink[head] * 1.4426950408889634f - m);
#pragma unroll
    for (int i = 0; i < 2 * LT_MAX_PIECES; ++i)
        if (lane + 32 * i < p.dv) p.out[row * p.dv + lane + 32 * i] = from_float<bf16>(o[i] / l);
}

__global__ void __launch_bounds__(LT_THREADS, 1) latent_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                          const __grid_constant__ CUtensorMap map_k,
                                                                          const LatentTcParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int pieces = p.d / 64, vpieces = p.dv / 64;
    const int groups = (pieces + 1) / 2, vgroups = (vpieces + 1) / 2;     // two pieces to a group, the last may have one
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + pieces * LT_Q_PIECE;
    const int slot_bytes = pieces * LT_K_PIECE;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sK + 2 * slot_bytes);
    const uint32_t q_full = tc_smem(bars);
    const uint32_t full0 = q_full + 8, empty0 = full0 + 8 * 2 * LT_GROUPS;     // [slot][group]
    const uint32_t s_full0 = empty0 + 8 * 2 * LT_GROUPS, p_full0 = s_full0 + 16, o_done = p_full0 + 16, o_last = o_done + 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + LT_BARS);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (tc_smem(smem) & 1023u) {            // the swizzled tiles need a 1024-byte aligned base
        if (threadIdx.x == 0) tc_fail(&g_latent_tc_error, 9, ACORN_KERNEL_LATENT_PREFILL_TC);
        return;
    }
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < 2 * LT_GROUPS; ++s) { mbar_init(full0 + 8 * s, LT_PRODUCERS); mbar_init(empty0 + 8 * s, 1); }
        for (int u = 0; u < 2; ++u) { mbar_init(s_full0 + 8 * u, 1); mbar_init(p_full0 + 8 * u, 4); }
        mbar_init(o_done, 1);
        mbar_init(o_last, 1);
        tmem_slot[1] = 0;                   // whether the rows are computed one by one at the end
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(tc_smem(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_s = *tmem_slot, tmem_o = tmem_s + 128;

    pdl_wait();
    pdl_trigger();
    // the tile: the rows' tiles in order, counted from the last one, so that a long row's later tokens, which see more keys,
    // come before its first ones
    const int TQ = LT_M / p.H;
    int r = -1, q0 = 0;
    for (int r0 = 0, left = (int)(gridDim.x - 1 - blockIdx.x); r0 < p.num_rows; r0 += 32) {
        const int n = r0 + lane < p.num_rows ? (p.row_start[r0 + lane + 1] - p.row_start[r0 + lane] + TQ - 1) / TQ : 0;
        int upto = n;
#pragma unroll
        for (int o = 1; o < 32; o *= 2) {
            const int below = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += below;
        }
        const uint32_t past = __ballot_sync(0xffffffffu, upto > left);
        if (past) {
            const int l = __ffs(past) - 1;
            r = r0 + l;
            q0 = (left - __shfl_sync(0xffffffffu, upto - n, l)) * TQ;
            break;
        }
        left -= __shfl_sync(0xffffffffu, upto, 31);
    }
    const bool live = r >= 0;               // not so only if the grid is larger than the rows' tiles
    r = max(r, 0);
    const int first = p.row_start[r], row_tokens = p.row_start[r + 1] - first;
    const int ntok = min(TQ, row_tokens - q0), rows_valid = ntok * p.H;
    const int64_t qrow0 = (int64_t)(first + q0) * p.H;
    const int pos0 = p.row_pos[r] + q0;
    const int hi = pos0 + ntok;                                          // keys < hi are read by the tile
    const int kept = p.row_pos[r] + row_tokens;                          // keys < kept are in the cache
    const int seen = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;      // keys >= seen are read by the tile
    const int lo = seen & ~(LT_KB - 1);
    const int nb = (hi - lo + LT_KB - 1) / LT_KB;

    if (!live) {
    } else if (warp == 4 || warp > 5) {
        // ---------------------------------------------------------------- producer
        // lane l looks up the cache rows of the l-th TMA box of a block (one page or 64 keys), a block ahead
        const int me = warp == 4 ? 0 : warp - 5;
        if (me == 0 && lane == 0) {
            mbar_expect_tx(q_full, pieces * LT_Q_PIECE);
            for (int c = 0; c < pieces; ++c) tma_load_2d(tc_smem(sQ) + c * LT_Q_PIECE, &map_q, q_full, 64 * c, (int)qrow0);
        }
        const int* table = p.block_table + (int64_t)r * p.table_stride - p.page_base[r];
        const int P = 1 << p.logP;
        const int box = P < LT_KB ? P : LT_KB, n_ops = LT_KB / box;      // <= 8 (pages of 8 keys or more)
        const int first_key = p.page_base[r] << p.logP;
        auto row_of = [&](int j) -> int {
            int key = lo + j * LT_KB + (lane < n_ops ? lane : 0) * box;
            // boxes no query of the tile may see (beyond the last key, or in pages a windowed request has given back)
            // are masked later: bring any that exist instead
            if (key >= kept) key = (kept - 1) & ~(box - 1);
            if (key < first_key) key = first_key;
            return (table[key >> p.logP] << p.logP) + (key & (P - 1));
        };
        int row_next = row_of(0);
        bool good = true;
        for (int j = 0; j < nb && good; ++j) {
            const int row_cur = row_next, slot = j & 1;
            if (j + 1 < nb) row_next = row_of(j + 1);
            for (int i = 0; i < groups && good; ++i) {                   // in the order the scores' product takes them
                const int g = i == 0 ? groups - 1 : i - 1;
                const int n = min(2, pieces - 2 * g);
                const uint32_t bar = full0 + 8 * (slot * LT_GROUPS + g);
                const bool got = mbar_wait(empty0 + 8 * (slot * LT_GROUPS + g), ((j >> 1) & 1) ^ 1);
                if (!got && lane == 0) tc_fail(&g_latent_tc_error, 1, ACORN_KERNEL_LATENT_PREFILL_TC);
                good = __all_sync(0xffffffffu, got);
                if (!good) break;
                if (elect_one()) mbar_expect_tx(bar, (n_ops - me + LT_PRODUCERS - 1) / LT_PRODUCERS * n * box * 128);
                const uint32_t base = tc_smem(sK) + slot * slot_bytes + 2 * g * LT_K_PIECE;
                for (int l = me; l < n_ops; l += LT_PRODUCERS) {
                    const int row = __shfl_sync(0xffffffffu, row_cur, l);
                    if (elect_one()) {
                        for (int c = 0; c < n; ++c)
                            tma_load_2d(base + c * LT_K_PIECE + l * box * 128, &map_k, bar, 64 * (2 * g + c), row);
                    }
                }
            }
        }
    } else if (warp == 5) {
        // ---------------------------------------------------------------- MMA issuer
        constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LT_M >> 4) << 24);
        constexpr uint32_t IDESC_QK = IDESC | ((uint32_t)(LT_KB >> 3) << 17);
        constexpr uint32_t IDESC_PV = IDESC | (1u << 16);                // values: head entries contiguous
        auto wait_all = [&](uint32_t bar, uint32_t parity, int code) -> bool {
            const bool ok = mbar_wait(bar, parity);
            if (!ok && lane == 0) tc_fail(&g_latent_tc_error, code, ACORN_KERNEL_LATENT_PREFILL_TC);
            return __all_sync(0xffffffffu, ok);
        };
        const uint32_t qlo = umma_lo(tc_smem(sQ)), klo0 = umma_lo(tc_smem(sK)), vlo0 = umma_lo_mn(tc_smem(sK), LT_K_PIECE);
        bool odd = false;
        auto scores = [&](int j) -> bool {                               // S[j & 1] = Q K_j^T
            // rows of the block that no query of the tile reads: in front of the first one's window (where pages were given back
            // others stand in for them), and from the last one's key on (where a page may hold no request's tokens)
            const int slot = j & 1, key0 = lo + j * LT_KB, front = min(LT_KB, seen - key0), tail = min(LT_KB, hi - key0);
            const int part_front = p.window > 0 ? min(tail, hi - p.window - key0) : 0, part_tail = max(max(part_front, 0), pos0 + 1 - key0);
            for (int i = 0; i < groups; ++i) {
                const int g = i == 0 ? groups - 1 : i - 1;
                const int n = min(2, pieces - 2 * g);
                if (!wait_all(full0 + 8 * (slot * LT_GROUPS + g), (j >> 1) & 1, 3)) return false;
                if (front > 0 || tail < LT_KB) {                         // values of zero there: their weights are, and 0 times no number is none
                    for (int c = 2 * g; c < min(2 * g + n, vpieces); ++c) {
                        uint8_t* piece = sK + slot * slot_bytes + c * LT_K_PIECE;
                        for (int at = lane * 16; at < front * 128; at += 32 * 16) *reinterpret_cast<uint4*>(piece + at) = make_uint4(0, 0, 0, 0);
                        for (int at = tail * 128 + lane * 16; at < LT_K_PIECE; at += 32 * 16) *reinterpret_cast<uint4*>(piece + at) = make_uint4(0, 0, 0, 0);
                    }
                    fence_proxy_async();
                    __syncwarp();
                }
                // rows that some queries of the tile read and some do not: a value that is no number would reach all of them
                for (int c = 2 * g; c < min(2 * g + n, vpieces); ++c) {
                    const uint8_t* piece = sK + slot * slot_bytes + c * LT_K_PIECE;
                    for (int at = max(0, front) * 128 + lane * 16; at < part_front * 128; at += 32 * 16)
                        odd |= lt_not_finite(*reinterpret_cast<const uint4*>(piece + at));
                    for (int at = part_tail * 128 + lane * 16; at < tail * 128; at += 32 * 16)
                        odd |= lt_not_finite(*reinterpret_cast<const uint4*>(piece + at));
                }
                for (int c = 2 * g; c < 2 * g + n; ++c)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16_elect(tmem_s + slot * 64, qlo + ((c * LT_Q_PIECE) >> 4) + 2 * k,
                                        klo0 + ((slot * slot_bytes + c * LT_K_PIECE) >> 4) + 2 * k, IDESC_QK, i > 0 || c > 2 * g || k > 0 ? 1u : 0u);
                if (g >= vgroups) umma_commit_elect(empty0 + 8 * (slot * LT_GROUPS + g));     // no values in these columns
            }
            umma_commit_elect(s_full0 + 8 * slot);
            return true;
        };
        auto values = [&](int j) -> bool {                               // O += P[j & 1] K_j[:, :dv]
            const int slot = j & 1;
            if (!wait_all(p_full0 + 8 * slot, (j >> 1) & 1, 4)) return false;
            tc_fence_after();
            for (int g = 0; g < vgroups; ++g) {
                const int n = min(2, vpieces - 2 * g);
                const uint32_t idesc = IDESC_PV | ((uint32_t)(n * 64 >> 3) << 17);
                // 16 keys a step: P advances 8 columns, the values 16 rows of 128 bytes; then the same keys with what P lacks
#pragma unroll
                for (int k = 0; k < 2 * LT_KB / 16; ++k)
                    umma_bf16_ts_elect(tmem_o + g * 128, tmem_s + slot * 64 + 8 * k,
                                       vlo0 + ((slot * slot_bytes + 2 * g * LT_K_PIECE + k % (LT_KB / 16) * 16 * 128) >> 4), idesc,
                                       j > 0 || k > 0 ? 1u : 0u);
                umma_commit_elect(empty0 + 8 * (slot * LT_GROUPS + g));
            }
            umma_commit_elect(o_done);
            if (j == nb - 1) umma_commit_elect(o_last);
            return true;
        };
        bool good = wait_all(q_full, 0, 2) && scores(0) && (nb < 2 || scores(1));
        for (int j = 0; j < nb && good; j += 2)
            good = values(j) && (j + 1 >= nb || values(j + 1)) && (j + 2 >= nb || scores(j + 2)) && (j + 3 >= nb || scores(j + 3));
        if (good && __any_sync(0xffffffffu, odd) && lane == 0) tmem_slot[1] = 1;
    } else {
        // ---------------------------------------------------------------- softmax and output
        const int row = warp * 32 + lane;                                // TMEM lane
        const bool row_ok = row < rows_valid;
        const int head = row % p.H, qpos = pos0 + row / p.H;
        const int first_seen = p.window > 0 ? qpos - p.window + 1 : 0;
        const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
        const uint32_t my_o = tmem_o + lane_addr;
        float m_ref = -INFINITY, l_run = 0.f;
        bool good = true;
        for (int j = 0; j < nb; ++j) {
            const uint32_t my_s = tmem_s + lane_addr + (j & 1) * 64;
            if (good && !mbar_wait(s_full0 + 8 * (j & 1), (j >> 1) & 1)) { tc_fail(&g_latent_tc_error, 6, ACORN_KERNEL_LATENT_PREFILL_TC); good = false; }
            good = __all_sync(0xffffffffu, good);
            if (!good) break;
            tc_fence_after();
            const int key0 = lo + j * LT_KB;
            // a block every query of the tile sees whole needs no mask
            const bool masked = key0 + LT_KB - 1 > pos0 || (p.window > 0 && key0 < hi - p.window) || rows_valid < LT_M;
            float s[64];
            tmem_ld64(my_s, s);
            if (masked) {
#pragma unroll
                for (int c = 0; c < 64; ++c) {
                    const int key = key0 + c;
                    s[c] = row_ok && key <= qpos && key >= first_seen ? s[c] : -INFINITY;
                }
            }
            const float mx = lt_max(s) * p.scale_log2;                   // the scale is positive
            if (__any_sync(0xffffffffu, mx > m_ref + LT_RESCALE_LOG2)) { // always so in a row's first block
                float corr = 1.f;
                if (mx > m_ref + LT_RESCALE_LOG2) {
                    corr = fast_exp2(m_ref - mx);                        // m_ref = -inf: 0
                    l_run *= corr;
                    m_ref = mx;
                }
                if (j > 0) {
                    // O holds the blocks before this one when the last of their products is done.  o_done completes a phase a
                    // block, and a wait by parity tells phase j - 1 from phase j - 2 only if j - 2 is over: the scores of block j
                    // have come, and they are issued behind the values of block j - 1 (j even) or j - 2 (j odd)
                    if (!mbar_wait(o_done, (j - 1) & 1)) { tc_fail(&g_latent_tc_error, 7, ACORN_KERNEL_LATENT_PREFILL_TC); good = false; }
                    good = __all_sync(0xffffffffu, good);
                    if (!good) break;
                    tc_fence_after();
                    for (int c = 0; c < p.dv; c += 32) {
                        float part[32];
                        tmem_ld32(my_o + c, part);
#pragma unroll
                        for (int i = 0; i < 32; ++i) part[i] *= corr;
                        tmem_st32(my_o + c, part);
                    }
                }
            }
            const float neg_ref = m_ref == -INFINITY ? 0.f : -m_ref;
            uint32_t w[32], rest[32];
            float ps[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 64; c += 2) {
                const float a = fast_exp2(fmaf(s[c], p.scale_log2, neg_ref)), b = fast_exp2(fmaf(s[c + 1], p.scale_log2, neg_ref));
                ps[(c >> 1) & 3] += a + b;
                __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
                w[c >> 1] = *reinterpret_cast<uint32_t*>(&v);
                v = __floats2bfloat162_rn(a - __uint_as_float(w[c >> 1] << 16), b - __uint_as_float(w[c >> 1] & 0xffff0000u));
                rest[c >> 1] = *reinterpret_cast<uint32_t*>(&v);
            }
            l_run += (ps[0] + ps[1]) + (ps[2] + ps[3]);
            tmem_st32_raw(my_s, w);                                      // column c holds keys 2 c and 2 c + 1
            tmem_st32_raw(my_s + 32, rest);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full0 + 8 * (j & 1));
        }
        if (good) {
            // a barrier of its own, of one phase: of the last two blocks' values neither need be done here (their scores are
            // issued together), and o_done's parity could not tell its state two phases ago from its last
            if (!mbar_wait(o_last, 0)) { tc_fail(&g_latent_tc_error, 8, ACORN_KERNEL_LATENT_PREFILL_TC); good = false; }
            good = __all_sync(0xffffffffu, good);
        }
        if (good) {
            tc_fence_after();
            if (p.sink && row_ok) l_run += exp2f(p.sink[head] * 1.4426950408889634f - m_ref);
            const float inv = row_ok ? 1.f / l_run : 0.f;
            bf16* orow = p.out + (qrow0 + row) * p.dv;
            for (int c = 0; c < p.dv; c += 32) {
                float part[32];
                tmem_ld32(my_o + c, part);
                if (row_ok) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint32_t ww[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            __nv_bfloat162 v = __floats2bfloat162_rn(part[i + 2 * q] * inv, part[i + 2 * q + 1] * inv);
                            ww[q] = *reinterpret_cast<uint32_t*>(&v);
                        }
                        *reinterpret_cast<uint4*>(orow + c + i) = make_uint4(ww[0], ww[1], ww[2], ww[3]);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (live && tmem_slot[1] != 0)          // (after the barrier: in the place of what the products gave)
        for (int row = warp; row < rows_valid; row += LT_THREADS / 32)
            latent_row_alone(p, p.block_table + (int64_t)r * p.table_stride - p.page_base[r], qrow0 + row, row % p.H, pos0 + row / p.H);
    if (warp == 5)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_s), "r"(512u) : "memory");
}

static size_t latent_prefill_smem(int d) {
    return (size_t)(d / 64) * (LT_Q_PIECE + 2 * LT_K_PIECE) + LT_BARS * 8 + 16;
}

extern "C" int acorn_latent_prefill_tc_supported(int H, int d, int dv, int P) {
    return H >= 1 && H <= LT_M && d % 64 == 0 && dv % 64 == 0 && dv >= 64 && dv <= d && dv <= 384 && d <= 64 * LT_MAX_PIECES &&
           P >= 8 && acorn_log2_exact_tc(P) >= 0;
}

// q: [tokens, H, d]; pages: [num_pages, 1, P, d]; num_tiles: the rows' tiles of 128 / H tokens, all together.
extern "C" int acorn_latent_prefill_tc(const void* q, int tokens, void* out, const void* pages, int64_t num_pages,
                                       const int* block_table, const int* page_base, int table_stride, const int* row_start,
                                       const int* row_pos, int num_rows, int num_tiles, const float* sink, float scale, int window,
                                       int H, int d, int dv, int P, cudaStream_t stream) {
    if (num_tiles <= 0) return 0;
    if (!acorn_latent_prefill_tc_supported(H, d, dv, P) || !(scale > 0.f) || ((uintptr_t)q & 15) || ((uintptr_t)pages & 15) ||
        ((uintptr_t)out & 15) || (int64_t)tokens * H > 0x7fffffff || num_pages * P > 0x7fffffff)
        return ACORN_ERR_UNSUPPORTED;
    LatentTcParams p;
    p.out = (bf16*)out; p.q = (const bf16*)q; p.pages = (const bf16*)pages; p.block_table = block_table; p.page_base = page_base;
    p.row_start = row_start; p.row_pos = row_pos; p.num_rows = num_rows; p.sink = sink; p.table_stride = table_stride;
    p.H = H; p.d = d; p.dv = dv; p.logP = acorn_log2_exact_tc(P); p.window = window; p.scale_log2 = scale * 1.4426950408889634f;
    CUtensorMap mq, mk;
    int rc = make_map(&mq, q, (int64_t)tokens * H, d, d, 64, LT_M);
    if (rc) return rc;
    rc = make_map(&mk, pages, num_pages * P, d, d, 64, P < LT_KB ? P : LT_KB);
    if (rc) return rc;
    static AcornPerDevice configured;
    if (!configured.seen()) {
        cudaError_t e = cudaFuncSetAttribute(latent_prefill_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)latent_prefill_smem(64 * LT_MAX_PIECES));
        if (e != cudaSuccess) return (int)e;
        configured.mark();
    }
    return acorn_launch(latent_prefill_tc_kernel, dim3((unsigned)num_tiles), dim3(LT_THREADS), latent_prefill_smem(d), stream, mq, mk, p);
}

extern "C" int acorn_latent_prefill_tc_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_latent_tc_error, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_latent_tc_error, &zero, sizeof(int));
    return v;
}

ACORN_ERROR_WORD_SETTER(acorn_latent_prefill_tc_set_error_word)
