// Token choice from float32 logits: argmax, and temperature / top-k / top-p sampling
// with a counter-based random number per (seed, counter), one block per row.
//
// Order of processing as in the reference (acorninfer/sampler.py:38-67): divide by the
// temperature; top-k keeps every logit >= the k-th largest; top-p removes, in ascending
// order, the tokens whose cumulative probability stays <= 1 - top_p (the largest token
// always stays); softmax over what is left; draw.  The draw is by inverse CDF in token
// order with u = uniform(seed, counter): the first token whose running sum exceeds
// u * total.  Rows do not interact, so the result does not depend on the batch.
// temperature == 0 selects argmax (lowest index among equal maxima).
// A row with a NaN or an infinite logit yields token -1 (the host raises).
//
// Two kernels.  `sample_cluster_kernel` takes vocabularies that fit the shared memory of a cluster of eight CTAs,
// `sample_kernel` walks the row in global memory.  The caller chooses (acorninfer_b200/kernels/ops.py, sample_in_clusters).
#include "common.cuh"

#include <cooperative_groups.h>
#include <cstring>
namespace cg = cooperative_groups;

#define SAMPLE_THREADS 1024

__device__ __forceinline__ unsigned int float_key(float x) {   // order-preserving map to uint
    unsigned int b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__host__ __device__ __forceinline__ unsigned long long splitmix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// uniform in [0, 1) with 24 bits, from (seed, counter)
__host__ __device__ __forceinline__ float uniform_from(unsigned long long seed, unsigned long long counter) {
    const unsigned long long z = splitmix64(splitmix64(seed) ^ (counter * 0xD1342543DE82EF95ull));
    return (float)(z >> 40) * (1.0f / 16777216.0f);
}

// A row's parameters: arrays in device memory, or the values themselves among the launch's arguments, which spares a step the
// copy of a block that the host has just made.
struct SampleArrays {
    const float* temperature;
    const int* top_k;
    const float* top_p;
    const unsigned long long* seed;
    const unsigned long long* counter;
};

#define SAMPLE_INLINE_ROWS 128

struct SampleInline {
    unsigned long long seed[SAMPLE_INLINE_ROWS], counter[SAMPLE_INLINE_ROWS];
    float temperature[SAMPLE_INLINE_ROWS], top_p[SAMPLE_INLINE_ROWS];
    int top_k[SAMPLE_INLINE_ROWS];
};

__device__ __forceinline__ unsigned int block_sum_u32(unsigned int v, unsigned int* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    unsigned int t = (lane < (int)(blockDim.x >> 5)) ? scratch[lane] : 0u;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

template <typename Rows>
__global__ void __launch_bounds__(SAMPLE_THREADS) sample_kernel(
    const float* __restrict__ logits, int64_t ld, int V, const __grid_constant__ Rows rows, int* __restrict__ token_out,
    float* __restrict__ logprob_out) {
    __shared__ float fscratch[32];
    __shared__ unsigned int uscratch[32];
    __shared__ float seg_prefix[SAMPLE_THREADS / 32];
    __shared__ int s_found;
    pdl_wait();
    pdl_trigger();
    const int r = blockIdx.x, tid = threadIdx.x;
    const float* x = logits + (int64_t)r * ld;
    const float temp = rows.temperature[r];

    // pass 1: max (first index among equals) and finiteness
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    unsigned int bad = 0;
    for (int i = tid; i < V; i += SAMPLE_THREADS) {
        const float v = x[i];
        if (!(fabsf(v) <= 3.0e38f)) bad = 1;
        if (v > best) { best = v; best_i = i; }
    }
    bad = block_sum_u32(bad, uscratch);
    const float gmax = block_max(best, fscratch);
    unsigned int cand = (best == gmax) ? (unsigned int)best_i : 0x7fffffffu;
    for (int o = 16; o > 0; o >>= 1) cand = min(cand, __shfl_xor_sync(0xffffffffu, cand, o));
    __syncthreads();
    if ((tid & 31) == 0) uscratch[tid >> 5] = cand;
    __syncthreads();
    cand = (tid & 31) < (SAMPLE_THREADS >> 5) ? uscratch[tid & 31] : 0x7fffffffu;
    for (int o = 16; o > 0; o >>= 1) cand = min(cand, __shfl_xor_sync(0xffffffffu, cand, o));
    const int arg = (int)cand;
    if (bad) {
        if (tid == 0) { token_out[r] = -1; if (logprob_out) logprob_out[r] = 0.f; }
        return;
    }
    if (!(temp > 0.f)) {
        if (tid == 0) { token_out[r] = arg; if (logprob_out) logprob_out[r] = 0.f; }
        return;
    }
    const float inv_t = 1.f / temp;
    // keys of the kept set: key >= lo_key
    unsigned int lo_key = 0u;
    int k = rows.top_k[r];
    if (k > 0 && k < V) {
        // largest K with count(key >= K) >= k  ==  key of the k-th largest logit
        unsigned int lo = 0u, hi = 0xffffffffu;
        while (lo < hi) {
            const unsigned int mid = lo + (unsigned int)(((unsigned long long)hi - lo + 1ull) >> 1);
            unsigned int c = 0;
            for (int i = tid; i < V; i += SAMPLE_THREADS) c += (float_key(x[i]) >= mid);
            c = block_sum_u32(c, uscratch);
            if (c >= (unsigned int)k) lo = mid; else hi = mid - 1u;
        }
        lo_key = lo;
    }
    const float p_keep = rows.top_p[r];
    if (p_keep < 1.f) {
        float z = 0.f;
        for (int i = tid; i < V; i += SAMPLE_THREADS)
            if (float_key(x[i]) >= lo_key) z += expf((x[i] - gmax) * inv_t);
        z = block_sum(z, fscratch);
        const float limit = (1.f - p_keep) * z;
        // smallest K with mass(lo_key <= key <= K) > limit
        unsigned int lo = lo_key, hi = float_key(gmax);
        while (lo < hi) {
            const unsigned int mid = lo + ((hi - lo) >> 1);
            float mass = 0.f;
            for (int i = tid; i < V; i += SAMPLE_THREADS) {
                const unsigned int key = float_key(x[i]);
                if (key >= lo_key && key <= mid) mass += expf((x[i] - gmax) * inv_t);
            }
            mass = block_sum(mass, fscratch);
            if (mass > limit) hi = mid; else lo = mid + 1u;
        }
        lo_key = lo;
    }
    // inverse CDF in token order over the kept set; thread tid owns a contiguous segment
    const int seg = (V + SAMPLE_THREADS - 1) / SAMPLE_THREADS;
    const int i0 = min(V, tid * seg), i1 = min(V, i0 + seg);
    float mine = 0.f;
    for (int i = i0; i < i1; ++i)
        if (float_key(x[i]) >= lo_key) mine += expf((x[i] - gmax) * inv_t);
    // exclusive scan of the 1024 segment sums: inside warps, then over warp totals
    float incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, incl, o);
        if ((tid & 31) >= o) incl += up;
    }
    if (tid == 0) s_found = -1;
    if ((tid & 31) == 31) seg_prefix[tid >> 5] = incl;
    __syncthreads();
    if (tid < 32) {
        const float wt = seg_prefix[tid];
        float winc = wt;
        for (int o = 1; o < 32; o <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, winc, o);
            if (tid >= o) winc += up;
        }
        seg_prefix[tid] = winc - wt;          // exclusive prefix of warp totals
        if (tid == 31) fscratch[0] = winc;    // total
    }
    __syncthreads();
    const float total = fscratch[0];
    const float excl = seg_prefix[tid >> 5] + (incl - mine);
    const float target = uniform_from(rows.seed[r], rows.counter[r]) * total;
    if (mine > 0.f && target >= excl && target < excl + mine) {
        float run = excl;
        int pick = -1, last_kept = -1;
        for (int i = i0; i < i1; ++i) {
            if (float_key(x[i]) >= lo_key) {
                run += expf((x[i] - gmax) * inv_t);
                last_kept = i;
                if (run > target) { pick = i; break; }
            }
        }
        if (pick < 0) pick = last_kept;
        atomicMax(&s_found, pick);
    }
    __syncthreads();
    if (tid == 0) {
        int pick = s_found;
        if (pick < 0) pick = arg;      // rounding left the target beyond the last segment
        token_out[r] = pick;
        if (logprob_out) logprob_out[r] = (x[pick] - gmax) * inv_t - logf(total);
    }
}

// ------------------------------------------------------------------ a cluster a row, the row in shared memory
//
// What bounds the walk above is one SM reading its row again for each of up to 64 bisection steps (64 rows of 151,936
// with top-k and top-p: 701 us).  Here the CTAs of a cluster hold the row in shared memory, read from HBM once.
//   top-k up to the number of warps (128): the k-th largest of the warps' maxima bounds the k-th largest key from below and
//     leaves few more than k candidates; the first CTA gathers them and ends alone (`sc_finish`), every pair compared.
//   top-p alone: one histogram of the probabilities in equal steps of the scaled logit, summed over the cluster through
//     distributed shared memory; the keys of the one bin that holds the bound are gathered by every CTA, which compares an eighth.
//   anything else, and rows whose candidates do not fit the lists (many equal logits): the bounds digit by digit (11 + 11 + 10
//     bits of the ordered key), a histogram a level (`sc_select`).
// All three ask the same: the smallest key K with weight(keys <= K) > limit, where a key weighs 1 and limit is the number of
// keys less k (the k-th largest), or weighs its probability and limit is (1 - top_p) of the total.  Probabilities are summed
// as integers of 2^-44 of the largest one (a sum's error is below that of float32 sums, and its order does not matter), so the
// three answers are the same.
// What bounds it: 64 clusters of 8 on 148 SMs are two waves (two CTAs an SM: shared memory), each a read of its slices and a
// chain of short steps with cluster barriers between them; rows with top-p alone, whose probabilities are all made twice, take
// longest.  64 rows of 151,936, parameters mixed: 63 us a call.  (Slices left in L2, so that all 64 run at once: 77 us.)
#define SC_THREADS 512
#define SC_WARPS (SC_THREADS / 32)
#define SC_BINS 2048
#define SC_CLUSTER 8
#define SC_MAXIMA (SC_CLUSTER * SC_WARPS)
#define SC_CAND 256                 // candidates a CTA can note
#define SC_LIST 1024                // candidates of a row that are compared in pairs
#define SC_STEPS 128.f              // bins of the first histogram by probability to a factor of e
#define SC_GROUPS 16                // parts of a warp's share whose sums it keeps for the draw
#define SC_MAX_SLICE 45056          // floats of a row a CTA can hold beside the histogram
typedef unsigned long long u64;

struct alignas(16) ScShared {
    u64 sums[SC_BINS / SC_CLUSTER]; // this CTA's share of a level's bins, summed over the cluster
    union {
        unsigned int hist[3][SC_BINS];  // a level's weights: 16-bit pieces, so that 32-bit atomics cannot overflow
        struct {
            u64 list[SC_LIST];          // gathered candidates: (key, index)
            u64 w[SC_LIST];             // their weights
        };
    };
    u64 cand[SC_CAND];              // candidates of this CTA's slice
    unsigned int tops[SC_WARPS];    // its warps' maxima (keys)
    unsigned int maxima[SC_MAXIMA]; // those of the whole row
    unsigned int first;             // least index of a largest logit in its slice
    unsigned int ncand;             // candidates met (more than SC_CAND: not all are noted)
    unsigned int lowest;            // a bound of the k-th largest key, or the least key found
    u64 total;                      // of `sums`
    u64 kept;                       // this CTA's part of the kept set
    u64 z;                          // probability of its slice
    unsigned int bad;
    u64 warp_a[SC_WARPS];
    u64 left;                       // answer of a level: the limit less the weight below the bin, the bin (SC_BINS: limit not exceeded)
    unsigned int found_bin;
};

// e^((x - gmax) / t) in units of 2^-44, cut off below; by shifts of the mantissa (a conversion to 64 bits runs at a sixteenth
// of their rate).  NaN, which 0 * inf gives, counts as 0.
__device__ __forceinline__ u64 prob_fixed(float x, float gmax, float inv_t) {
    const unsigned int b = __float_as_uint(expf((x - gmax) * inv_t));
    const int shift = (int)(b >> 23) - 106;                     // 2^(exponent - 150 + 44) a unit of the mantissa; at most 21
    const u64 m = (b & 0x7fffffu) | 0x800000u;
    return shift > 21 || shift < -24 ? 0ull : shift >= 0 ? m << shift : m >> -shift;
}

__device__ __forceinline__ u64 warp_sum_u64(u64 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ u64 block_sum_u64(u64 v, u64* scratch) {
    v = warp_sum_u64(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    return warp_sum_u64((threadIdx.x & 31) < SC_WARPS ? scratch[threadIdx.x & 31] : 0ull);
}

__device__ __forceinline__ float key_float(unsigned int key) {
    return __uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key);
}

// Adds a probability to a bin, in pieces of 16 bits.
__device__ __forceinline__ void sc_add_mass(ScShared& sh, int bin, u64 w) {
    atomicAdd(&sh.hist[0][bin], (unsigned int)w & 0xffffu);
    if (w >> 16) atomicAdd(&sh.hist[1][bin], (unsigned int)(w >> 16) & 0xffffu);
    if (w >> 32) atomicAdd(&sh.hist[2][bin], (unsigned int)(w >> 32));
}

// Notes element i of this CTA's slice, whose logit has this key, as a candidate (index i0 + i of the row).
__device__ __forceinline__ void sc_note(ScShared& sh, unsigned int key, int at) {
    const unsigned int slot = atomicAdd(&sh.ncand, 1u);
    if (slot < SC_CAND) sh.cand[slot] = ((u64)key << 32) | (unsigned int)at;
}

// The cluster has noted its candidates: brings them all into `sh.list` (of the CTAs that `take` them) and returns their number,
// or -1 where they do not fit, the same in every CTA.  The caller's cluster barrier ends the reads of other CTAs' notes.
__device__ int sc_gather(ScShared& sh, bool take) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    int first[SC_CLUSTER + 1];
    bool fits = true;
    first[0] = 0;
#pragma unroll
    for (int q = 0; q < SC_CLUSTER; ++q) {
        const unsigned int c = *cluster.map_shared_rank(&sh.ncand, q);
        fits = fits && c <= SC_CAND;
        first[q + 1] = first[q] + (int)min(c, (unsigned int)SC_CAND);
    }
    if (!fits || first[SC_CLUSTER] > SC_LIST) return -1;
    if (take) {
        const int warp = threadIdx.x >> 5;       // two warps bring a CTA's notes
        const int q = warp / (SC_WARPS / SC_CLUSTER);
        int at = 0, c = 0;
#pragma unroll
        for (int i = 0; i < SC_CLUSTER; ++i)
            if (i == q) { at = first[i]; c = first[i + 1] - first[i]; }
        const u64* notes = cluster.map_shared_rank(&sh.cand[0], q);
        for (int i = threadIdx.x % (SC_THREADS / SC_CLUSTER); i < c; i += SC_THREADS / SC_CLUSTER) sh.list[at + i] = notes[i];
    }
    __syncthreads();
    return first[SC_CLUSTER];
}

// top-k, top-p and the draw among `n` gathered candidates that hold the row's k largest keys: one CTA, every pair compared.
__device__ void sc_finish(ScShared& sh, int n, int k, float p_keep, unsigned int gkey, float gmax, float inv_t, u64 m, int* token,
                          float* logprob) {
    const int tid = threadIdx.x;
    u64 z = 0;
    for (int t = tid; t < n; t += SC_THREADS) {
        const unsigned int key = (unsigned int)(sh.list[t] >> 32);
        int greater = 0;
        for (int j = 0; j < n; ++j) greater += (unsigned int)(sh.list[j] >> 32) > key;
        const u64 w = greater < k ? prob_fixed(key_float(key), gmax, inv_t) : 0ull;       // kept: no less than the k-th largest
        sh.w[t] = w;
        z += w;
    }
    z = block_sum_u64(z, sh.warp_a);
    __syncthreads();
    if (p_keep < 1.f) {
        const u64 bound = (u64)((double)(1.f - p_keep) * (double)z);
        u64 own[SC_LIST / SC_THREADS] = {};
        z = 0;
#pragma unroll
        for (int e = 0; e < SC_LIST / SC_THREADS; ++e) {
            const int t = tid + e * SC_THREADS;
            if (t >= n) break;
            const unsigned int key = (unsigned int)(sh.list[t] >> 32);
            u64 upto = 0;
            for (int j = 0; j < n; ++j) upto += (unsigned int)(sh.list[j] >> 32) <= key ? sh.w[j] : 0ull;
            own[e] = upto > bound || key >= gkey ? sh.w[t] : 0ull;                        // the largest always stays
            z += own[e];
        }
        z = block_sum_u64(z, sh.warp_a);
        __syncthreads();
#pragma unroll
        for (int e = 0; e < SC_LIST / SC_THREADS; ++e)
            if (tid + e * SC_THREADS < n) sh.w[tid + e * SC_THREADS] = own[e];
        __syncthreads();
    }
    // u = m / 2^24: the first token whose running sum exceeds floor(m z / 2^24)
    const u64 target = (__umul64hi(m, z) << 40) | ((m * z) >> 24);
    for (int t = tid; t < n; t += SC_THREADS) {
        const unsigned int at = (unsigned int)sh.list[t];
        u64 before = 0;
        for (int j = 0; j < n; ++j) before += (unsigned int)sh.list[j] < at ? sh.w[j] : 0ull;
        if (target >= before && target < before + sh.w[t]) {
            *token = (int)at;
            if (logprob) *logprob = (key_float((unsigned int)(sh.list[t] >> 32)) - gmax) * inv_t - logf((float)((double)z * 5.684341886080802e-14));
        }
    }
    if (z == 0 && tid == 0) {                    // the first of the largest (-0 and 0 are equal), all of which are candidates
        unsigned int first = 0xffffffffu;
        for (int j = 0; j < n; ++j)
            if (key_float((unsigned int)(sh.list[j] >> 32)) == gmax) first = min(first, (unsigned int)sh.list[j]);
        *token = (int)first;
        if (logprob) *logprob = 0.f;
    }
}

// The row's first index among its largest logits (in every thread).  Called by all threads of the cluster.
__device__ int sc_first(ScShared& sh, const float* row, int n, int i0, float gmax) {
    cg::cluster_group cluster = cg::this_cluster();
    if (threadIdx.x == 0) sh.first = 0x7fffffffu;
    __syncthreads();
    unsigned int first = 0x7fffffffu;
    for (int i = threadIdx.x; i < n; i += SC_THREADS)
        if (row[i] == gmax) first = min(first, (unsigned int)(i0 + i));
    if (first != 0x7fffffffu) atomicMin(&sh.first, first);
    cluster.sync();
#pragma unroll
    for (int q = 0; q < SC_CLUSTER; ++q) first = min(first, *cluster.map_shared_rank(&sh.first, q));
    return (int)first;
}

// Sums this level's bins over the cluster and finds the first at which the weight so far exceeds the limit, which `limit_of`
// gives from the sum of all: `sh.found_bin` (SC_BINS: none) and `sh.left`, the limit less the weight before that bin.
// Called by all threads of the cluster after they have added to `sh.hist`.
template <bool MASS, typename LimitOf>
__device__ void sc_find_bin(ScShared& sh, int bins, LimitOf limit_of) {
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31;
    constexpr int PIECES = MASS ? 3 : 1;
    cluster.sync();
    // this CTA sums its share of the bins over the cluster (all remote reads of a bin in flight at once)
    const int share = bins / SC_CLUSTER, first = (int)cluster.block_rank() * share;
    u64 mine = 0;
    for (int i = tid; i < share; i += SC_THREADS) {
        unsigned int h[SC_CLUSTER][PIECES];
#pragma unroll
        for (int r = 0; r < SC_CLUSTER; ++r)
#pragma unroll
            for (int q = 0; q < PIECES; ++q) h[r][q] = cluster.map_shared_rank(&sh.hist[q][0], r)[first + i];
        u64 s = 0;
#pragma unroll
        for (int r = 0; r < SC_CLUSTER; ++r) {
            s += h[r][0];
            if (MASS) s += ((u64)h[r][PIECES / 2] << 16) + ((u64)h[r][PIECES - 1] << 32);
        }
        sh.sums[i] = s;
        mine += s;
    }
    mine = block_sum_u64(mine, sh.warp_a);
    if (tid == 0) sh.total = mine;
    cluster.sync();
    // one warp finds the bin: first the CTA whose share holds it, then the bin in that share
    if (tid < 32) {
        const u64 t = lane < SC_CLUSTER ? *cluster.map_shared_rank(&sh.total, lane) : 0ull;
        u64 incl = t;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const u64 up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        const u64 all = __shfl_sync(0xffffffffu, incl, SC_CLUSTER - 1);
        const u64 limit = limit_of(all);
        const unsigned int over = __ballot_sync(0xffffffffu, lane < SC_CLUSTER && incl > limit);
        if (over == 0) {
            if (lane == 0) sh.found_bin = SC_BINS;
        } else {
            const int owner = __ffs(over) - 1;
            u64 run = __shfl_sync(0xffffffffu, incl - t, owner);
            const u64* sums = cluster.map_shared_rank(&sh.sums[0], owner);
            constexpr int PER = SC_BINS / SC_CLUSTER / 32;                // a lane's bins (the last level has half as many)
            const int per = share / 32;
            u64 own[PER], part = 0;
#pragma unroll
            for (int i = 0; i < PER; ++i) own[i] = i < per ? sums[lane * per + i] : 0ull;
#pragma unroll
            for (int i = 0; i < PER; ++i) part += own[i];
            u64 pin = part;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u64 up = __shfl_up_sync(0xffffffffu, pin, o);
                if (lane >= o) pin += up;
            }
            const int who = __ffs(__ballot_sync(0xffffffffu, run + pin > limit)) - 1;
            if (lane == who) {
                run += pin - part;
                int i = 0;
                bool on = true;
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    on = on && run + own[k] <= limit;
                    if (on) { run += own[k]; ++i; }
                }
                sh.found_bin = owner * share + lane * per + i;
                sh.left = limit - run;
            }
        }
    }
    __syncthreads();
}

// The smallest key K of the row from `cut` on with weight(keys <= K) > limit; 0xffffffff if there is none.  MASS: keys from
// lo_key on weigh their probability, the total is z, the limit (1 - top_p) z; else keys weigh 1 and the limit leaves k above
// it.  No key below `cut` is K.  Called by all threads of the cluster with the same arguments.
template <bool MASS>
__device__ unsigned int sc_select(ScShared& sh, const float* row, int n, unsigned int cut, float gmax, float inv_t, u64 z, u64 bound) {
    const int tid = threadIdx.x;
    constexpr int PIECES = MASS ? 3 : 1;
    unsigned int prefix = 0;        // the digits found so far
#pragma unroll 1
    for (int level = 0; level < 3; ++level) {
        const int shift = level == 0 ? 21 : level == 1 ? 10 : 0;
        const int bins = level == 2 ? 1024 : 2048, above = level == 0 ? 32 : level == 1 ? 21 : 10;
        for (int i = tid; i < PIECES * SC_BINS; i += SC_THREADS) (&sh.hist[0][0])[i] = 0;
        __syncthreads();
        for (int i = tid; i < n; i += SC_THREADS) {
            const float v = row[i];
            const unsigned int key = float_key(v);
            if (key < cut || (level > 0 && (key >> above) != prefix)) continue;
            const int bin = (key >> shift) & (bins - 1);
            if (MASS) {
                const u64 w = prob_fixed(v, gmax, inv_t);
                if (w != 0) sc_add_mass(sh, bin, w);
            } else {
                atomicAdd(&sh.hist[0][bin], 1u);
            }
        }
        // counted from the cut on: less what lies below it
        sc_find_bin<MASS>(sh, bins, [&](u64 all) { return level > 0 ? sh.left : MASS ? bound - (z - all) : all - bound; });
        if (sh.found_bin == SC_BINS) return 0xffffffffu;
        prefix = (prefix << (level == 0 ? 11 : level == 1 ? 11 : 10)) | sh.found_bin;
    }
    return prefix;
}

template <typename Rows>
__global__ void __launch_bounds__(SC_THREADS, 2) sample_cluster_kernel(
    const float* __restrict__ logits, int64_t ld, int V, int slice, const __grid_constant__ Rows rows, int* __restrict__ token_out,
    float* __restrict__ logprob_out) {
    extern __shared__ __align__(16) unsigned char sc_smem[];
    ScShared& sh = *reinterpret_cast<ScShared*>(sc_smem);
    float* row = reinterpret_cast<float*>(sc_smem + sizeof(ScShared));
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int r = blockIdx.x / SC_CLUSTER, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_wait();
    pdl_trigger();
    const int i0 = min(V, rank * slice), n = min(V, i0 + slice) - i0;
    const float* x = logits + (int64_t)r * ld + i0;
    const float temp = rows.temperature[r];

    // the slice into shared memory; its largest logit, and finiteness: NaN and infinities make a NaN of their product with 0
    float top = -INFINITY, size = 0.f, zero = 0.f;
    auto take = [&](float v) {
        top = fmaxf(top, v);
        size = fmaxf(size, fabsf(v));
        zero = fmaf(v, 0.f, zero);
    };
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        const int n4 = n >> 2;
#pragma unroll 8
        for (int i = tid; i < n4; i += SC_THREADS) {
            const float4 v = reinterpret_cast<const float4*>(x)[i];
            take(v.x); take(v.y); take(v.z); take(v.w);
            reinterpret_cast<float4*>(row)[i] = v;
        }
        for (int i = 4 * n4 + tid; i < n; i += SC_THREADS) { take(x[i]); row[i] = x[i]; }
    } else {
#pragma unroll 8
        for (int i = tid; i < n; i += SC_THREADS) { const float v = x[i]; take(v); row[i] = v; }
    }
    unsigned int bad = !(size <= 3.0e38f) || zero != 0.f;
    top = warp_max(top);
    if (tid == 0) { sh.bad = 0; sh.ncand = 0; }
    if (lane == 0) sh.tops[warp] = float_key(top == 0.f ? 0.f : top);        // -0 and 0 are equal
    __syncthreads();
    if (bad) sh.bad = 1;
    const int k = rows.top_k[r];
    const float p_keep = rows.top_p[r];
    const u64 m = (u64)(uniform_from(rows.seed[r], rows.counter[r]) * 16777216.f);       // u = m / 2^24
    cluster.sync();
    if (tid < SC_MAXIMA) sh.maxima[tid] = cluster.map_shared_rank(&sh.tops[0], tid / SC_WARPS)[tid % SC_WARPS];
    bad = 0;
#pragma unroll
    for (int q = 0; q < SC_CLUSTER; ++q) bad |= *cluster.map_shared_rank(&sh.bad, q);
    __syncthreads();
    unsigned int gkey = 0;
#pragma unroll
    for (int q = 0; q < SC_MAXIMA / 32; ++q) gkey = max(gkey, sh.maxima[lane + 32 * q]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gkey = max(gkey, __shfl_xor_sync(0xffffffffu, gkey, o));
    const float gmax = key_float(gkey);
    if (bad || !(temp > 0.f)) {
        const int arg = bad ? -1 : sc_first(sh, row, n, i0, gmax);
        if (rank == 0 && tid == 0) {
            token_out[r] = arg;
            if (logprob_out) logprob_out[r] = 0.f;
        }
        cluster.sync();              // a CTA's shared memory stays until all have read it
        return;
    }
    const float inv_t = 1.f / temp;
    unsigned int lo_key = 0u;
    const bool by_k = k > 0 && k < V;
    if (by_k) {
        unsigned int low = 0u;
        if (k <= SC_MAXIMA) {
            // The k-th largest of the warps' maxima: k warps hold a key from it on, so the k-th largest key is one (a maximum of
            // -0 counts as 0 there).  Its rank by comparison, equal ones (warps without an element) in their order.
            if (tid < SC_MAXIMA) {
                const unsigned int own = sh.maxima[tid];
                int before = 0;
                for (int j = 0; j < SC_MAXIMA; ++j) before += sh.maxima[j] > own || (sh.maxima[j] == own && j < tid);
                if (before == k - 1) sh.lowest = own;
            }
            __syncthreads();
            low = sh.lowest;
            if (low == float_key(0.f)) low = float_key(-0.f);
            // as keys and as numbers the same: low is not the key of 0
            const float least = key_float(low);
            const int n4 = n >> 2;
            for (int i = tid; i < n4; i += SC_THREADS) {
                const float4 v = reinterpret_cast<const float4*>(row)[i];
                if (fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)) >= least) {
                    if (v.x >= least) sc_note(sh, float_key(v.x), i0 + 4 * i);
                    if (v.y >= least) sc_note(sh, float_key(v.y), i0 + 4 * i + 1);
                    if (v.z >= least) sc_note(sh, float_key(v.z), i0 + 4 * i + 2);
                    if (v.w >= least) sc_note(sh, float_key(v.w), i0 + 4 * i + 3);
                }
            }
            for (int i = 4 * n4 + tid; i < n; i += SC_THREADS)
                if (row[i] >= least) sc_note(sh, float_key(row[i]), i0 + i);
            const int found = sc_gather(sh, rank == 0);
            if (found >= 0) {
                cluster.sync();      // the others' notes have been read
                if (rank == 0)
                    sc_finish(sh, found, k, p_keep, gkey, gmax, inv_t, m, token_out + r, logprob_out ? logprob_out + r : nullptr);
                return;
            }
        }
        lo_key = sc_select<false>(sh, row, n, low, 0.f, 0.f, 0ull, (u64)k);
    }
    if (p_keep < 1.f) {
        // (1 - top_p) of all that is kept so far
        auto limit_of = [&](u64 all) { return (u64)((double)(1.f - p_keep) * (double)all); };
        int found = -1;
        if (!by_k) {
            // the bins ascend with the key: SC_STEPS a factor of e in probability, what is further down in the first
            auto bin_of = [&](float v) { return SC_BINS - 1 - (int)fminf((gmax - v) * inv_t * SC_STEPS, (float)(SC_BINS - 1)); };
            for (int i = tid; i < 3 * SC_BINS; i += SC_THREADS) (&sh.hist[0][0])[i] = 0;
            __syncthreads();
            for (int i = tid; i < n; i += SC_THREADS) {
                const u64 w = prob_fixed(row[i], gmax, inv_t);
                if (w != 0) sc_add_mass(sh, bin_of(row[i]), w);
            }
            sc_find_bin<true>(sh, SC_BINS, limit_of);
            const int bin = (int)sh.found_bin;
            lo_key = gkey;           // the largest always stays
            if (bin == SC_BINS) {
                found = 0;
            } else {
                for (int i = tid; i < n; i += SC_THREADS) {
                    const float v = row[i];
                    if (bin_of(v) == bin && prob_fixed(v, gmax, inv_t) != 0) sc_note(sh, float_key(v), i0 + i);
                }
                if (tid == 0) sh.lowest = gkey;
                found = sc_gather(sh, true);
                for (int t = tid; t < found; t += SC_THREADS) sh.w[t] = prob_fixed(key_float((unsigned int)(sh.list[t] >> 32)), gmax, inv_t);
                __syncthreads();
                // an eighth of the candidates to each CTA; the least key at which the sum exceeds the limit is told to all
                for (int t = rank + SC_CLUSTER * tid; t < found; t += SC_CLUSTER * SC_THREADS) {
                    const unsigned int key = (unsigned int)(sh.list[t] >> 32);
                    u64 upto = 0;
                    for (int j = 0; j < found; ++j) upto += (unsigned int)(sh.list[j] >> 32) <= key ? sh.w[j] : 0ull;
                    if (upto > sh.left && key < gkey)
                        for (int q = 0; q < SC_CLUSTER; ++q) atomicMin(cluster.map_shared_rank(&sh.lowest, q), key);
                }
                cluster.sync();
                if (found >= 0) lo_key = sh.lowest;
                else lo_key = 0u;
            }
        }
        if (found < 0) {
            u64 part = 0;
            for (int i = tid; i < n; i += SC_THREADS)
                if (float_key(row[i]) >= lo_key) part += prob_fixed(row[i], gmax, inv_t);
            part = block_sum_u64(part, sh.warp_a);
            if (tid == 0) sh.z = part;
            cluster.sync();
            u64 z = 0;
#pragma unroll
            for (int q = 0; q < SC_CLUSTER; ++q) z += *cluster.map_shared_rank(&sh.z, q);
            const u64 bound = limit_of(z);
            // V keys of half of bound / V each stay within the bound
            const float least = 0.5f * (float)((double)bound / V * 5.684341886080802e-14);
            const unsigned int cut = least > 1e-12f ? float_key(gmax + temp * logf(least)) : 0u;
            const unsigned int key = sc_select<true>(sh, row, n, max(cut, lo_key), gmax, inv_t, z, bound);
            lo_key = key < gkey ? key : gkey;            // the largest always stays
        }
    }
    // inverse CDF in token order over the kept set: a warp owns a run of the slice, in SC_GROUPS groups; lane g keeps the sum of
    // group g
    const int group = (n + SC_WARPS * SC_GROUPS - 1) / (SC_WARPS * SC_GROUPS);
    const int run0 = warp * SC_GROUPS * group;
    auto weigh = [&](int i) -> u64 { return float_key(row[i]) >= lo_key ? prob_fixed(row[i], gmax, inv_t) : 0ull; };
    u64 mine = 0;
    for (int g = 0; g < SC_GROUPS; ++g) {
        const int a = min(n, run0 + g * group), b = min(n, a + group);
        u64 part = 0;
        for (int i = a + lane; i < b; i += 32) part += weigh(i);
        part = warp_sum_u64(part);
        if (lane == g) mine = part;
    }
    u64 incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    __syncthreads();
    if (lane == 31) sh.warp_a[warp] = incl;
    __syncthreads();
    u64 before = 0, here = 0;                    // of the row up to this warp's run
    for (int w = 0; w < SC_WARPS; ++w) {
        if (w < warp) before += sh.warp_a[w];
        here += sh.warp_a[w];
    }
    const u64 own = sh.warp_a[warp];
    if (tid == 0) sh.kept = here;
    cluster.sync();
    u64 total = 0;
#pragma unroll
    for (int q = 0; q < SC_CLUSTER; ++q) {
        const u64 t = *cluster.map_shared_rank(&sh.kept, q);
        if (q < rank) before += t;
        total += t;
    }
    // the first token whose running sum exceeds floor(m total / 2^24)
    const u64 target = (__umul64hi(m, total) << 40) | ((m * total) >> 24);
    if (target >= before && target < before + own) {         // one warp of the cluster
        const int g = __ffs(__ballot_sync(0xffffffffu, before + incl > target)) - 1;
        before += __shfl_sync(0xffffffffu, incl - mine, g);
        const int a = min(n, run0 + g * group), b = min(n, a + group);
        for (int at = a; at < b; at += 32) {
            const int i = at + lane;
            const u64 w = i < b ? weigh(i) : 0ull;
            u64 upto = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u64 up = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += up;
            }
            const unsigned int over = __ballot_sync(0xffffffffu, before + upto > target);
            if (over != 0) {
                if (lane == __ffs(over) - 1) {
                    token_out[r] = i0 + i;
                    if (logprob_out) logprob_out[r] = (row[i] - gmax) * inv_t - logf((float)((double)total * 5.684341886080802e-14));
                }
                break;
            }
            before += __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    if (total == 0) {
        const int arg = sc_first(sh, row, n, i0, gmax);
        if (rank == 0 && tid == 0) {
            token_out[r] = arg;
            if (logprob_out) logprob_out[r] = 0.f;
        }
    }
    cluster.sync();
}

template <typename Rows>
static int launch_sample(const float* logits, int64_t ld, int n, int V, const Rows& rows, int* token_out, float* logprob_out, int clusters,
                         cudaStream_t stream) {
    // slices are multiples of four logits, so that they start on 16 bytes where the row does
    const int slice = ((V + SC_CLUSTER - 1) / SC_CLUSTER + 3) & ~3;
    if (!clusters || slice > SC_MAX_SLICE || n > 0x7fffffff / SC_CLUSTER)
        return acorn_launch(sample_kernel<Rows>, dim3(n), dim3(SAMPLE_THREADS), 0, stream, logits, ld, V, rows, token_out, logprob_out);
    static AcornPerDevice configured;
    if (!configured.seen()) {
        const int most = (int)(sizeof(ScShared) + SC_MAX_SLICE * sizeof(float));
        cudaError_t e = cudaFuncSetAttribute(sample_cluster_kernel<Rows>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e != cudaSuccess) return (int)e;
        configured.mark();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n * SC_CLUSTER));
    cfg.blockDim = dim3(SC_THREADS);
    cfg.dynamicSmemBytes = sizeof(ScShared) + (size_t)slice * sizeof(float);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = SC_CLUSTER;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = acorn_pdl_enabled() ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, sample_cluster_kernel<Rows>, logits, ld, V, slice, rows, token_out, logprob_out);
    return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

extern "C" int acorn_sample(const float* logits, int64_t ld, int rows, int V, const float* temperature,
                            const int* top_k, const float* top_p, const unsigned long long* seed,
                            const unsigned long long* counter, int* token_out, float* logprob_out, int clusters,
                            cudaStream_t stream) {
    if (rows <= 0) return 0;
    const SampleArrays r = {temperature, top_k, top_p, seed, counter};
    return launch_sample(logits, ld, rows, V, r, token_out, logprob_out, clusters, stream);
}

// The same with the parameters in host memory: one after the other `rows` seeds, counters (64 bits each), temperatures, top_p
// (float32) and top_k (int32).  At most SAMPLE_INLINE_ROWS rows; `block` is free again when this returns.
extern "C" int acorn_sample_inline(const float* logits, int64_t ld, int rows, int V, const void* block, int* token_out, float* logprob_out,
                                   int clusters, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (rows > SAMPLE_INLINE_ROWS || block == nullptr) return ACORN_ERR_UNSUPPORTED;
    SampleInline r = {};
    const unsigned char* at = (const unsigned char*)block;
    auto part = [&](void* to, size_t bytes) {
        memcpy(to, at, bytes);
        at += bytes;
    };
    part(r.seed, 8 * (size_t)rows);
    part(r.counter, 8 * (size_t)rows);
    part(r.temperature, 4 * (size_t)rows);
    part(r.top_p, 4 * (size_t)rows);
    part(r.top_k, 4 * (size_t)rows);
    return launch_sample(logits, ld, rows, V, r, token_out, logprob_out, clusters, stream);
}

// Host copy of the generator, for callers that need the same uniforms off the device.
extern "C" float acorn_uniform(unsigned long long seed, unsigned long long counter) {
    return uniform_from(seed, counter);
}
