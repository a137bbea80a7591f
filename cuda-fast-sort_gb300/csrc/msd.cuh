// msd.cuh — keys-only sorts of 4-, 8- and 16-byte keys above the short range,
// most significant bits first (sm_103a).
//
// A least-significant-digit sort makes one stable pass over the data per key
// byte, each bound by its rank.  Keys only, equal twiddled keys are equal
// bytes, so the order among equal keys cannot show and no step needs a stable
// order.  This path instead reads a key's leading bits as a group number
// (8 + b2 bits, so that groups average a third to 0.72 of a local sort):
//   sample:       4096 keys say which of their bits vary (keys of a small
//                 range leave the leading ones alone: the group number starts
//                 at the first that varies) and how many group bits to take;
//                 it also clears the path's counters;
//   count:        one read of the keys counts every group (65536 16-bit
//                 counters fit a CTA's shared memory);
//   scan:         group offsets, and the decision: a group that does not fit a
//                 CTA's local sort is left out of them (MSD_RANGES), and with
//                 more than a quarter of the keys in such groups MSD_OFF;
//   top split:    every tile counts its keys per top digit with shared
//                 atomics, claims its places in the digit's exact range with
//                 one global atomic per digit, stages the tile by digit and
//                 writes each digit's run — no tile waits for another (input
//                 -> alternate buffer, twiddled);
//   second split: the same inside every top bucket, by the group's b2 bits
//                 (alternate buffer -> caller's buffer);
//   local sorts:  each CTA sorts whole groups in place in shared memory: a
//                 counting pass on the next 11-12 bits moves every key into
//                 its sub-bucket (about one key each), then a few rounds of
//                 an odd-even transposition network in registers, as many as
//                 the largest sub-bucket holds keys, put the keys in order;
//                 a group with a sub-bucket of more keys than that can take
//                 is sorted another way (group_sort_crowded).
// The groups left out are sorted by themselves by the launch that follows
// (multi.cuh).  With MSD_OFF the least-significant-digit passes, launched after these
// kernels, sort from the caller's buffer, which then holds the input's keys
// in some order (untouched, or as the local sorts left them); otherwise they
// exit at once.
// Every key is read four times and written three times, whatever its width.
// 4-byte floats take it too, by a group number from the sample's distribution
// (MsdEvenCode; 2^27 keys of N(0, 1) 1.50 ms, four digit passes 2.03; the
// table's reads cost the count and the splits about a half: 6 * 10^7 keys
// 80 + 160 + 185 us, unsigned keys 49 + 110 + 138).
#pragma once

#include <cooperative_groups.h>

#include "fused_short.cuh"

namespace gbsort {

struct MsdParams {
    const void* keys_in;   // the input: the caller's keys or the input-preserving source
    void* keys_a;          // the caller's buffer (second split's output, sorted in place)
    void* keys_b;          // the alternate buffer (top split's output)
    uint64_t n;            // < 2^32
    int kind, desc;
    int b2_max;            // most group bits below the top digit (0 .. 8) that the counters have room for
    uint32_t* state;       // MSD_OFF: the digit passes sort; zeroed with the control block
    uint32_t* window;      // [2] leading bits that do not vary, group bits below the top digit (b2)
    uint32_t* zero;        // the counters below, cleared by the first kernel
    uint32_t zero_words;
    uint32_t* top_counts;  // [256] keys per top digit
    uint32_t* cursor1;     // [256] next place of every top digit
    uint32_t* joint;       // [256 << b2_max] keys per group
    uint32_t* cursor2;     // [256 << b2_max] next place of every group; its end after the second split
    uint32_t group_cap;    // largest group a local sort takes
    RangeList left;        // groups above group_cap, sorted by a later launch
    uint2* table;          // floats: the code of every leading 12 bits (MsdEvenCode), then a sampled key of each
    uint32_t* giants;      // floats: count, then group and key of every group of equal keys above group_cap
    uint32_t* err;         // workspace error word
};

// The leading 64 bits of a twiddled key (all of a 4-byte key's, left-aligned).
__device__ __forceinline__ uint64_t msd_top64(uint32_t k) { return uint64_t(k) << 32; }
__device__ __forceinline__ uint64_t msd_top64(uint64_t k) { return k; }
__device__ __forceinline__ uint64_t msd_top64(u128 k) { return uint64_t(k >> 64); }

// A key's code: the 32 bits of it after the `skip` leading ones that all keys
// share (zeros where they run past its leading 64).
struct MsdCode {
    uint32_t skip, b2;
    __device__ __forceinline__ explicit MsdCode(const MsdParams& p)
        : skip(ld_relaxed(p.window)), b2(ld_relaxed(p.window + 1)) {}
    __device__ __forceinline__ MsdCode(uint32_t left_out, uint32_t bits) : skip(left_out), b2(bits) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t k) const { return k << skip; }
    __device__ __forceinline__ uint32_t operator()(uint64_t k) const {
        const uint32_t hi = uint32_t(k >> 32), lo = uint32_t(k);
        const bool low = skip >= 32u;
        return __funnelshift_l(low ? 0u : lo, low ? lo : hi, skip);  // (the shift wraps at 32)
    }
    __device__ __forceinline__ uint32_t operator()(u128 k) const { return (*this)(uint64_t(k >> 64)); }
};

// The code of a float.  Floats crowd into few leading bits (the exponent), so
// their codes are the sample's distribution function instead: the leading 12
// bits (sign, exponent, 3 bits of mantissa) name a stretch of the codes as wide
// as the share of the sample there, {start, width}, and the 20 bits below
// divide it evenly (both after the `skip` bits that the sample's keys share; keys
// outside their range, few if any, count as its nearest end).
// Monotone; two keys may share a code.
struct MsdEvenCode {
    static constexpr uint32_t BINS = 4096;
    const uint2* table;
    uint32_t skip, b2, low, high;  // low, high: the range
    __device__ __forceinline__ MsdEvenCode(const MsdParams& p, const uint2* t)
        : table(t), skip(ld_relaxed(p.window)), b2(ld_relaxed(p.window + 1)), low(p.table[BINS + BINS / 2].x),
          high(low | 0xffffffffu >> skip) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t k) const {
        const uint32_t c = min(max(k, low), high) << skip;
        const uint2 e = table[c >> 20];
        return e.x + __umulhi(c << 12, e.y);
    }
    // copies the table to shared memory (the caller's barrier follows)
    __device__ __forceinline__ static void fetch(const MsdParams& p, uint2* to) {
        const uint4* from = reinterpret_cast<const uint4*>(p.table);
        for (uint32_t i = threadIdx.x; i < BINS / 2; i += blockDim.x) reinterpret_cast<uint4*>(to)[i] = from[i];
    }
};
template <bool EVEN>
__device__ __forceinline__ auto msd_code(const MsdParams& p, const uint2* table) {
    if constexpr (EVEN) return MsdEvenCode(p, table);
    else return MsdCode(p);
}

// The window of the codes, from a sample; the other CTAs clear the counters.
constexpr int MSD_SAMPLE_THREADS = 1024;
template <int KB>
__global__ void __launch_bounds__(MSD_SAMPLE_THREADS) msd_sample_kernel(MsdParams p) {
    using U = typename KeyBits<KB>::U;
    grid_launch_dependents();
    grid_dependency_wait();
    const int tid = threadIdx.x;
    if (blockIdx.x != 0) {
        const uint32_t stride = (gridDim.x - 1) * MSD_SAMPLE_THREADS;
        for (uint32_t i = (blockIdx.x - 1) * MSD_SAMPLE_THREADS + tid; i < p.zero_words; i += stride) p.zero[i] = 0u;
        return;
    }
    constexpr uint32_t SLOTS = 8192, NONE = 0xffffffffu;
    __shared__ uint32_t vary[2], top, again, fresh, neighbours, bins[256], seen[SLOTS], met[2][SLOTS / 32];
    if (tid < 2) vary[tid] = 0u;
    if (tid == 0) top = again = fresh = neighbours = 0u;
    for (uint32_t i = tid; i < SLOTS; i += MSD_SAMPLE_THREADS) seen[i] = NONE;
    if (tid < 256) bins[tid] = met[0][tid] = met[1][tid] = 0u;
    static_assert(SLOTS / 32 == 256, "two bits a slot");
    __syncthreads();
    const KeyMap<U> map(p.kind, p.desc);
    const U* keys = static_cast<const U*>(p.keys_in);
    constexpr int PER = 4;
    const uint32_t step = uint32_t(p.n / (MSD_SAMPLE_THREADS * PER));
    uint64_t x[PER], y;  // y: four keys after the first of them
    {
        const uint64_t j = uint64_t(tid) * step + (uint32_t(tid) * 2654435761u) % step;
        y = msd_top64(map.in(keys[j + 4u]));
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const uint32_t at = uint32_t(i * MSD_SAMPLE_THREADS + tid);
        x[i] = msd_top64(map.in(keys[uint64_t(at) * step + (at * 2654435761u) % step]));
    }
    const uint64_t first = msd_top64(map.in(keys[0]));
    uint64_t d = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) d |= x[i] ^ first;
    const uint32_t dh = __reduce_or_sync(0xffffffffu, uint32_t(d >> 32));
    const uint32_t dl = __reduce_or_sync(0xffffffffu, uint32_t(d));
    if ((tid & 31) == 0) {
        atomicOr(&vary[0], dh);
        atomicOr(&vary[1], dl);
    }
    __syncthreads();
    const uint32_t skip = vary[0] ? __clz(vary[0]) : vary[1] ? 32u + __clz(vary[1]) : 0u;
    // keys in order send whole tiles to one digit: shared atomics on one
    // address, slower than four digit passes (10^7 4-byte keys 290 and 207 us),
    // though not than eight or sixteen (5 x 10^7 8-byte keys 1.16 and 2.13 ms,
    // 2^24 16-byte ones 0.62 and 2.41)
    const uint32_t close = __popc(__ballot_sync(0xffffffffu, ((x[0] ^ y) << skip) >> 56 == 0u));
    if ((tid & 31) == 0) atomicAdd(&neighbours, close);
    uint32_t most = 0, twice = 0, distinct = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const uint32_t c = uint32_t((x[i] << skip) >> 32);
        most = max(most, c);
        // Codes met before in the sample (open addressing, half full at most):
        // those met twice, not oftener, are counted, and none counts again in its
        // digit: a few very frequent keys are no matter, their groups are sorted
        // apart.
        uint32_t h = (c * 2654435761u) >> 19;
        bool first_met = true;
        for (int probe = 0; probe < 64 && c != NONE; ++probe) {
            uint32_t v = seen[h];
            if (v == NONE) v = atomicCAS(&seen[h], NONE, c);
            if (v == NONE) break;
            if (v == c) {
                first_met = false;
                const uint32_t bit = 1u << (h & 31u);
                if (!(atomicOr(&met[0][h >> 5], bit) & bit)) ++twice;
                else if (!(atomicOr(&met[1][h >> 5], bit) & bit)) --twice;
                break;
            }
            h = (h + 1u) & (SLOTS - 1u);
        }
        if (first_met) atomicAdd(&bins[c >> 24], 1u);
        distinct += first_met;
    }
    twice = __reduce_add_sync(0xffffffffu, twice);
    distinct = __reduce_add_sync(0xffffffffu, distinct);
    if ((tid & 31) == 0 && twice) atomicAdd(&again, twice);
    if ((tid & 31) == 0) atomicAdd(&fresh, distinct);
    most = __reduce_max_sync(0xffffffffu, most);
    if ((tid & 31) == 0) atomicMax(&top, most);
    __syncthreads();
    // a top digit with five times its share has groups that do not fit, as have
    // very frequent keys of more than a quarter of the array, and codes that
    // repeat more than 64 times (S keys of D distinct codes meet S * S / 2 D of
    // them again) crowd the local sorts' sub-buckets
    const bool uneven = __syncthreads_or(tid < 256 && bins[tid] > MSD_SAMPLE_THREADS * PER / 256 * 5);
    if (tid == 0) {
        // the codes reach `top`: groups beyond it stay empty
        const float used = (float(top) + 1.f) * 0x1p-24f, n = float(p.n), cap = float(p.group_cap) * used;
        uint32_t b2 = 0;
        while (b2 < uint32_t(p.b2_max) && n > 0.72f * cap * float(1u << b2)) ++b2;
        constexpr float S = MSD_SAMPLE_THREADS * PER;
        const bool crowded = again >= 16u && 2.f * float(again) * n > 64.f * S * S;
        if (uneven || crowded || 4u * fresh < 3u * uint32_t(S) || (KB == 4 && 2u * neighbours > uint32_t(MSD_SAMPLE_THREADS)) || n > cap * float(1u << b2)) *p.state = MSD_OFF;
        p.window[0] = skip;
        p.window[1] = b2;
    }
}

// Exclusive scan over the CTA with one barrier: every warp scans the warp
// totals for itself (warp_tmp is written again only after another barrier).
template <int THREADS>
__device__ __forceinline__ uint32_t block_exclusive_scan_1b(uint32_t x, uint32_t* warp_tmp) {
    constexpr int WARPS = THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t v = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) warp_tmp[warp] = v;
    __syncthreads();
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp && lane < WARPS ? warp_tmp[lane] : 0u);
    return before + v - x;
}

// The codes of 4-byte floats, from 65536 keys in vectors of four spread over
// the array: a cluster of eight CTAs samples and counts the leading 12 bits
// (one SM alone would wait eight times as long for its gathers), its first CTA
// lays the codes out; the other clusters clear the counters.
// A bin with k keys of the sample gets a stretch of k + 4 sqrt(k) + 8, so that
// neither the sample's error nor the slope of the density inside the bin makes
// its groups too large, and in the ratio of the bin's range to the part of it
// that the keys take; an empty one gets 1, beside another bin 4.  A bin whose sampled keys, two at least, are all equal
// (zeros, infinities, NaNs) has a group of its own: equal keys need no sort, however
// many they are.
constexpr int MSD_EVEN_CLUSTER = 8;
constexpr size_t MSD_EVEN_SMEM = 6 * MsdEvenCode::BINS * 4;
constexpr uint32_t MSD_GIANTS = 31;
template <int KB>
__global__ void __cluster_dims__(MSD_EVEN_CLUSTER, 1, 1) __launch_bounds__(MSD_SAMPLE_THREADS)
    msd_even_sample_kernel(MsdParams p) {
    static_assert(KB == 4, "codes of 4-byte floats");
    namespace cg = cooperative_groups;
    constexpr uint32_t BINS = MsdEvenCode::BINS, NONE = 0xffffffffu, SLOTS = 8192;
    constexpr int VECS = 2, PER = MSD_SAMPLE_THREADS * MSD_EVEN_CLUSTER;
    constexpr float S = float(PER * VECS * 4);
    extern __shared__ __align__(16) uint32_t smem_even[];
    uint32_t* cnt = smem_even;  // keys per bin, their least and their largest
    uint32_t* low = cnt + BINS;
    uint32_t* high = low + BINS;
    uint32_t* all = high + BINS;  // (first CTA) the same of the cluster
    __shared__ uint32_t vary, again, neighbours, equal, dense, scan[2][32], total[2];
    grid_launch_dependents();
    grid_dependency_wait();
    const uint32_t tid = threadIdx.x;
    if (blockIdx.x >= MSD_EVEN_CLUSTER) {
        const uint32_t stride = (gridDim.x - MSD_EVEN_CLUSTER) * MSD_SAMPLE_THREADS;
        for (uint32_t i = (blockIdx.x - MSD_EVEN_CLUSTER) * MSD_SAMPLE_THREADS + tid; i < p.zero_words; i += stride)
            p.zero[i] = 0u;
        return;
    }
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = blockIdx.x;
    const KeyMap<uint32_t> map(p.kind, p.desc);
    const uint32_t* keys = static_cast<const uint32_t*>(p.keys_in);
    const uint32_t head = ((16u - (reinterpret_cast<uintptr_t>(keys) & 15u)) & 15u) / 4u;
    const uint32_t nvec = uint32_t((p.n - head) / 4u);
    const uint32_t step = nvec / uint32_t(PER * VECS);  // (the path's arrays are 32 times as long at least)
    uint32_t x[VECS * 4];
#pragma unroll
    for (int i = 0; i < VECS; ++i) {
        const uint32_t at = (uint32_t(i) * MSD_SAMPLE_THREADS + tid) * MSD_EVEN_CLUSTER + rank;
        const uint4 v = __ldcs(reinterpret_cast<const uint4*>(keys + head) + (at * step + (at * 2654435761u) % step));
        x[i * 4] = map.in(v.x);
        x[i * 4 + 1] = map.in(v.y);
        x[i * 4 + 2] = map.in(v.z);
        x[i * 4 + 3] = map.in(v.w);
    }
    const uint32_t first = map.in(keys[0]);
    for (uint32_t i = tid; i < BINS; i += MSD_SAMPLE_THREADS) {
        cnt[i] = high[i] = 0u;
        low[i] = NONE;
    }
    if (tid == 0) vary = again = neighbours = equal = dense = 0u;
    __syncthreads();
    uint32_t d = 0;
#pragma unroll
    for (int i = 0; i < VECS * 4; ++i) d |= x[i] ^ first;
    d = __reduce_or_sync(0xffffffffu, d);
    if ((tid & 31u) == 0u) atomicOr(&vary, d);
    cluster.sync();
    d = 0;
    for (uint32_t r = 0; r < MSD_EVEN_CLUSTER; ++r) d |= *cluster.map_shared_rank(&vary, r);
    const uint32_t skip = d ? __clz(d) : 0u;
#pragma unroll
    for (int i = 0; i < VECS * 4; ++i) {
        const uint32_t c = x[i] << skip, b = c >> 20;
        atomicAdd(&cnt[b], 1u);
        atomicMin(&low[b], c);
        atomicMax(&high[b], c);
    }
    cluster.sync();
    {  // every CTA merges its share of the bins into the first one's arrays
        uint32_t* to = cluster.map_shared_rank(all, 0);
        const uint32_t b = rank * (BINS / MSD_EVEN_CLUSTER) + tid;
        if (tid < BINS / MSD_EVEN_CLUSTER) {
            uint32_t k = 0, lo = NONE, hi = 0;
#pragma unroll
            for (uint32_t r = 0; r < MSD_EVEN_CLUSTER; ++r) {
                k += *cluster.map_shared_rank(cnt + b, r);
                lo = min(lo, *cluster.map_shared_rank(low + b, r));
                hi = max(hi, *cluster.map_shared_rank(high + b, r));
            }
            to[b] = k;
            to[BINS + b] = lo;
            to[2 * BINS + b] = hi;
        }
    }
    // Keys that repeat more than a dozen times would crowd the local sorts'
    // sub-buckets (those of a bin of equal keys do not matter): pairs of equal
    // keys among half of every CTA's sample.
    uint32_t count_in = 0;
#pragma unroll
    for (int i = 0; i < VECS * 4; ++i) {
        const uint32_t b = (x[i] << skip) >> 20;
        count_in |= uint32_t((i & 3) < 2 && low[b] != high[b] && x[i] != NONE) << i;
    }
    cluster.sync();  // (nobody reads the others' counts after this)
    for (uint32_t i = tid; i < SLOTS; i += MSD_SAMPLE_THREADS) cnt[i] = NONE;
    __syncthreads();
    uint32_t twice = 0, runs = 0;
#pragma unroll
    for (int i = 0; i < VECS * 4; ++i) {
        const uint32_t k = x[i];
        if (i % 4 == 0) runs += ((k ^ x[i + 1]) | (k ^ x[i + 2]) | (k ^ x[i + 3])) << skip < 1u << 24;
        if (!(count_in >> i & 1u)) continue;
        uint32_t h = (k * 2654435761u) >> 19;
        for (int probe = 0; probe < 64; ++probe) {
            uint32_t v = cnt[h];
            if (v == NONE) v = atomicCAS(&cnt[h], NONE, k);
            if (v == NONE) break;
            if (v == k) {
                ++twice;
                break;
            }
            h = (h + 1u) & (SLOTS - 1u);
        }
    }
    if (twice) atomicAdd(cluster.map_shared_rank(&again, 0), twice);
    if (runs) atomicAdd(cluster.map_shared_rank(&neighbours, 0), runs);
    cluster.sync();
    if (rank != 0) return;
    // the layout: four bins a thread
    uint32_t w[4], alone = 0, sum = 0, same = 0;
    float most = 0.f;  // keys of the sample per unit of stretch, where they lie densest
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t b = tid * 4 + i;
        const float k = float(all[b]);
        const uint32_t range = all[2 * BINS + b] - all[BINS + b];
        if (k == 0.f) w[i] = (b != 0u && all[b - 1]) || (b + 1 != BINS && all[b + 1]) ? 4u : 1u;
        else if (range == 0u && k >= 2.f) w[i] = 0u;  // a group of its own
        else {
            // (the least and the largest of k even ones lie (k - 1) / (k + 1) of their range apart)
            const float part =
                k < 2.f ? 1.f
                        : fminf(1.f, fmaxf((float(range) + 1.f) * 0x1p-20f * (k + 1.f) / (k - 1.f), k < 32.f ? 0.25f : 0.f));
            const float f = k + 4.f * sqrtf(k) + 8.f;
            w[i] = uint32_t(fminf(f / part, 8.f * S));
            most = fmaxf(most, k / f);
        }
        sum += w[i];
        alone += w[i] == 0u;
        same += w[i] == 0u ? uint32_t(k) : 0u;
    }
    if (same) atomicAdd(&equal, same);
    atomicMax(&dense, __float_as_uint(most));
    uint32_t at = block_exclusive_scan_1b<MSD_SAMPLE_THREADS>(sum, scan[0]);
    uint32_t alones = block_exclusive_scan_1b<MSD_SAMPLE_THREADS>(alone, scan[1]);
    if (tid == MSD_SAMPLE_THREADS - 1) {
        total[0] = at + sum;
        total[1] = alones + alone;
    }
    __syncthreads();
    const uint32_t W = total[0], P = total[1];
    const float n = float(p.n), units = float(W) * __uint_as_float(dense);
    uint32_t b2 = 0;  // groups of 0.6 of the largest at most where keys lie densest
    auto fits = [&] {
        const uint32_t groups = 256u << b2;
        return groups >= 4u * P && n * units <= 0.6f * S * float(p.group_cap) * float(groups - 2u * P);
    };
    while (b2 < uint32_t(p.b2_max) && !fits()) ++b2;
    const uint32_t shared = skip ? first >> (32u - skip) << (32u - skip) : 0u;
    const uint32_t group = 1u << (24u - b2);
    const uint64_t scale = ((uint64_t(1) << 32) - 2ull * P * group) / W;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t b = tid * 4 + i;
        const uint64_t r = at * scale + 2ull * alones * group;
        p.table[b] = w[i] == 0u ? make_uint2(uint32_t((r + group - 1u) & ~uint64_t(group - 1u)), group)
                                : make_uint2(uint32_t(r), uint32_t(w[i] * scale));
        // a bin of equal keys: the key
        reinterpret_cast<uint32_t*>(p.table + BINS)[b] = shared | all[BINS + b] >> skip;
        at += w[i];
        alones += w[i] == 0u;
    }
    if (tid == 0) {
        constexpr float R = MSD_SAMPLE_THREADS * VECS * 2;  // of CLUSTER * R * R / 2 pairs
        const bool crowded = again >= 6u && float(again) * n > 12.f * 0.5f * MSD_EVEN_CLUSTER * R * R;
        // Keys in order send whole tiles to one digit, and so do many equal
        // ones: shared atomics on one address, slower than the digit passes
        // (10^7 keys in order 294 and 207 us, with 60% zeros 267 and 250).
        // d == 0: equal keys, which no digit pass moves.
        const bool runs_of_keys = 2u * neighbours > uint32_t(PER * VECS) || float(equal) > 0.4f * S;
        if (crowded || runs_of_keys || d == 0u || !fits()) *p.state = MSD_OFF;
        p.table[BINS + BINS / 2].x = shared;
        p.window[0] = skip;
        p.window[1] = b2;
    }
}

// Keys per group, one read of the input.  16-bit counters, two to a word.
// Rounds of at most 2^14 keys a CTA: a counter that a key of the round found
// at 2^15 or above makes the CTA move those halves to the global counts after
// the round's barrier, so none ever passes 2^15 + 2^14.
constexpr int MSD_COUNT_THREADS = 1024;
constexpr int MSD_COUNT_SMEM = 32768 * 4 + 256 * 4;
template <int KB, bool EVEN>
__global__ void __launch_bounds__(MSD_COUNT_THREADS, 1) msd_count_kernel(MsdParams p) {
    using U = typename KeyBits<KB>::U;
    extern __shared__ __align__(128) uint8_t smem[];
    uint32_t* cnt = reinterpret_cast<uint32_t*>(smem);
    uint32_t* rows = cnt + 32768;
    const int tid = threadIdx.x;
    for (uint32_t i = tid; i < (128u << p.b2_max); i += MSD_COUNT_THREADS) cnt[i] = 0u;
    if (tid < 256) rows[tid] = 0u;
    grid_launch_dependents();
    grid_dependency_wait();
    if (ld_relaxed(p.state) & MSD_OFF) return;
    uint2* table = reinterpret_cast<uint2*>(smem + MSD_COUNT_SMEM);
    if constexpr (EVEN) MsdEvenCode::fetch(p, table);
    __syncthreads();
    const auto code_of = msd_code<EVEN>(p, table);
    const uint32_t b2 = code_of.b2, words = 128u << b2, shift = 24u - b2;
    const KeyMap<U> map(p.kind, p.desc);
    const U* keys = static_cast<const U*>(p.keys_in);
    const uint64_t n = p.n;
    uint64_t head = ((16u - (reinterpret_cast<uintptr_t>(keys) & 15u)) & 15u) / KB;
    if (head > n) head = n;
    const uint64_t nvec = (n - head) * KB / 16;
    constexpr int PER_VEC = 16 / KB, UNROLL = 4;
    static_assert(MSD_COUNT_THREADS * PER_VEC * UNROLL <= 16384, "keys a round");
    const uint64_t gthreads = uint64_t(gridDim.x) * MSD_COUNT_THREADS;
    const uint64_t gtid = uint64_t(blockIdx.x) * MSD_COUNT_THREADS + tid;
    const uint4* vec = reinterpret_cast<const uint4*>(keys + head);
    unsigned long long* joint = reinterpret_cast<unsigned long long*>(p.joint);
    const U first = map.in(keys[0]);
    U outside = U(0);  // a bit set: some key differs from the first one there
    auto sweep = [&](auto floats) {
        uint32_t seen = 0;
        auto count = [&](U k) {
            const U t = decltype(floats)::value ? map.in(k) : U(k ^ map.m);
            outside |= t ^ first;
            const uint32_t g = code_of(t) >> shift;
            seen |= atomicAdd(&cnt[g >> 1], __funnelshift_l(1u, 1u, g * 16u));
        };
        auto settle = [&] {
            if (__syncthreads_or(seen & 0x80008000u)) {
                for (uint32_t i = tid; i < words; i += MSD_COUNT_THREADS) {
                    const uint32_t w = cnt[i], lo = w & 0x8000u, hi = (w >> 16) & 0x8000u;
                    if (lo | hi) {
                        cnt[i] = w & 0x7fff7fffu;
                        atomicAdd(joint + i, (unsigned long long)(lo) | (unsigned long long)(hi) << 32);
                        if (lo) atomicAdd(p.top_counts + ((2 * i) >> b2), lo);
                        if (hi) atomicAdd(p.top_counts + ((2 * i + 1) >> b2), hi);
                    }
                }
                seen = 0;
                __syncthreads();
            }
        };
        if (gtid < head) count(keys[gtid]);
        // the same number of rounds for every thread (the barrier in them)
        uint64_t i0 = 0;
        for (; i0 + UNROLL * gthreads <= nvec; i0 += UNROLL * gthreads) {
            uint4 v[UNROLL];
#pragma unroll
            for (int r = 0; r < UNROLL; ++r) v[r] = __ldcs(vec + i0 + r * gthreads + gtid);
#pragma unroll
            for (int r = 0; r < UNROLL; ++r) {
                union { uint4 q; U k[PER_VEC]; } w;
                w.q = v[r];
#pragma unroll
                for (int e = 0; e < PER_VEC; ++e) count(w.k[e]);
            }
            settle();
        }
        for (uint64_t i = i0 + gtid; i < nvec; i += gthreads) {
            union { uint4 q; U k[PER_VEC]; } w;
            w.q = __ldcs(vec + i);
#pragma unroll
            for (int e = 0; e < PER_VEC; ++e) count(w.k[e]);
        }
        for (uint64_t j = head + nvec * PER_VEC + gtid; j < n; j += gthreads) count(keys[j]);
    };
    if (EVEN || p.kind == KIND_FLOAT) sweep(BoolTag<true>{});
    else sweep(BoolTag<false>{});
    if constexpr (EVEN) __syncthreads();  // (else the barrier of the next test)
    // a key that differs in the bits left out of the codes: the digit passes sort
    const uint64_t o64 = msd_top64(outside);
    if (!EVEN && __syncthreads_or(code_of.skip != 0u && (o64 >> (64u - code_of.skip)) != 0u)) {
        if (tid == 0) atomicOr(p.state, MSD_OFF);
        return;
    }
    // the CTA's counts to the global ones, two groups per 64-bit add (a
    // group's count stays below 2^32, so the halves never carry); CTAs start
    // at different words
    const uint32_t rot = uint32_t((uint64_t(words) * blockIdx.x / gridDim.x) & ~31u);
    for (uint32_t i0 = tid; i0 < words; i0 += MSD_COUNT_THREADS) {
        uint32_t i = i0 + rot;
        if (i >= words) i -= words;
        const uint32_t w = cnt[i];
        const uint32_t lo = w & 0xffffu, hi = w >> 16;
        if (w) atomicAdd(joint + i, (unsigned long long)(lo) | (unsigned long long)(hi) << 32);
        if (b2 >= 6) {  // a warp's 32 words lie in one row
            const uint32_t s = __reduce_add_sync(0xffffffffu, lo + hi);
            if ((tid & 31) == 0 && s) atomicAdd(&rows[(i * 2) >> b2], s);
        } else if (b2 >= 1) {
            if (w) atomicAdd(&rows[(i * 2) >> b2], lo + hi);
        } else {
            if (lo) atomicAdd(&rows[i * 2], lo);
            if (hi) atomicAdd(&rows[i * 2 + 1], hi);
        }
    }
    __syncthreads();
    if (tid < 256 && rows[tid]) atomicAdd(p.top_counts + tid, rows[tid]);
}

// Group offsets, one CTA per top digit, and the decision.
template <bool EVEN>
__global__ void __launch_bounds__(256) msd_scan_kernel(MsdParams p) {
    __shared__ uint32_t scan[32], base;
    grid_launch_dependents();
    grid_dependency_wait();
    if (ld_relaxed(p.state) & MSD_OFF) return;
    const int tid = threadIdx.x;
    const uint32_t b = blockIdx.x, b2 = ld_relaxed(p.window + 1);
    const uint32_t ex = block_exclusive_scan_256<uint32_t>(p.top_counts[tid], scan, nullptr);
    if (uint32_t(tid) == b) {
        base = ex;
        p.cursor1[b] = ex;
    }
    __syncthreads();
    const bool mine = tid < (1 << b2);
    const uint32_t c = mine ? p.joint[(b << b2) + tid] : 0u;
    const uint32_t e2 = block_exclusive_scan_256<uint32_t>(c, scan, nullptr);
    if (mine) p.cursor2[(b << b2) + tid] = base + e2;
    bool fits = c <= p.group_cap;
    if constexpr (EVEN) {
        if (!fits) {  // the group of a bin whose sampled keys were equal?
            const uint32_t width = 1u << (24u - b2), code = ((b << b2) + tid) * width;
            uint32_t lo = 0, hi = MsdEvenCode::BINS;  // the last bin that starts at or below it
            while (hi - lo > 1u) {
                const uint32_t mid = (lo + hi) / 2u;
                if (p.table[mid].x <= code) lo = mid;
                else hi = mid;
            }
            if (p.table[lo].x == code && p.table[lo].y == width) {
                const uint32_t i = atomicAdd(p.giants, 1u);
                if (i < MSD_GIANTS) {
                    fits = true;
                    p.giants[1 + 2 * i] = (b << b2) + tid;
                    p.giants[2 + 2 * i] = reinterpret_cast<const uint32_t*>(p.table + MsdEvenCode::BINS)[lo];
                }
            }
        }
    }
    if constexpr (!EVEN) {
        if (!fits) {  // left to be sorted by itself, while such groups are a quarter of the array at most
            const uint32_t i = atomicAdd(p.left.count, 1u), all = atomicAdd(p.left.count + 1, c) + c;
            if (i < p.left.most && all <= uint32_t(p.n / 4)) {
                p.left.ranges[2 * i] = base + e2;
                p.left.ranges[2 * i + 1] = c;
                atomicOr(p.state, MSD_RANGES);
                fits = true;
            }
        }
    }
    if (__syncthreads_or(!fits) && tid == 0) atomicOr(p.state, MSD_OFF);
}

// Shared memory of a split: the stage, in which every digit has CAP places of
// its own for a digit of 8 bits (more for a narrower one), then u32 bins[256],
// claims[256], counts[256], tstart, tcnt, tfirst[257], scan[32].
// CAP is odd, so that the digits' places start on different banks, and about
// five standard deviations above the mean of THREADS * IPT / 256 keys.
template <int KB, int THREADS, int IPT, int CAP>
struct MsdSplitGeom {
    static constexpr int TILE = THREADS * IPT;
    static constexpr int STAGE = CAP ? 256 * CAP : TILE;
    static_assert(STAGE >= TILE && (CAP % 2 == 1 || CAP == 0), "the stage also holds a dense tile");
    static_assert(IPT % (16 / KB) == 0, "16-byte loads");
    static constexpr size_t WORDS_OFF = size_t(STAGE) * KB;
    static constexpr int SPILL = CAP ? 512 : 0;  // keys beyond their digit's places
    static constexpr size_t SPILL_OFF = (WORDS_OFF + (256 * 6 + 1 + 32 + 4) * 4 + 15) & ~size_t(15);
    static constexpr size_t SMEM_BYTES = SPILL_OFF + SPILL * KB;
    // floats: then the table of the codes
    static constexpr size_t TABLE_OFF = (SMEM_BYTES + 15) & ~size_t(15);
    static constexpr size_t EVEN_BYTES = TABLE_OFF + MsdEvenCode::BINS * 8;
};

// Keys [lo, hi) from the 16-byte aligned src into registers, by 16-byte loads:
// key VEC * i + e of a thread is key (i * THREADS + tid) * VEC + e.  The whole
// vectors load without branches, so that nothing waits for them here.
template <int THREADS, class U, int N>
__device__ __forceinline__ void load_vectors(const U* src, uint32_t lo, uint32_t hi, U (&keys)[N]) {
    constexpr int VEC = 16 / int(sizeof(U));
#pragma unroll
    for (int i = 0; i < N / VEC; ++i) {
        const uint32_t j = uint32_t(i * THREADS + threadIdx.x) * VEC;
        union { uint4 q; U k[VEC]; } w;
        w.q = make_uint4(0u, 0u, 0u, 0u);
        if (j >= lo && j + VEC <= hi) w.q = __ldcs(reinterpret_cast<const uint4*>(src + j));
#pragma unroll
        for (int e = 0; e < VEC; ++e) keys[i * VEC + e] = w.k[e];
    }
    if (VEC > 1 && ((lo | hi) & uint32_t(VEC - 1))) {  // the ragged ends
#pragma unroll
        for (int i = 0; i < N / VEC; ++i) {
            const uint32_t j = uint32_t(i * THREADS + threadIdx.x) * VEC;
            if (j + VEC > lo && j < hi && (j < lo || j + VEC > hi)) {
#pragma unroll
                for (int e = 0; e < VEC; ++e)
                    if (j + e >= lo && j + e < hi) keys[i * VEC + e] = src[j + e];
            }
        }
    }
}

// The tile's keys [lo, hi) of THREADS * IPT from a 16-byte aligned address:
// key VEC * i + e of a thread is key (i * THREADS + tid) * VEC + e.
template <int KB, int THREADS, int IPT>
__device__ __forceinline__ void msd_load_tile(const typename KeyBits<KB>::U* src, uint32_t lo, uint32_t hi,
                                              typename KeyBits<KB>::U (&keys)[IPT]) {
    using U = typename KeyBits<KB>::U;
    load_vectors<THREADS>(src, lo, hi, keys);
}

// One tile (msd_load_tile's keys, mapped by in()) split by one digit (code >>
// shift, nb values, a power of two): its keys go to dst at the places that
// the tile claims from claim[d], one atomic per digit.  No order among a
// digit's keys.  bins: nb zeros on entry, left so.  refill() runs when the
// keys' registers are free.
// Every key takes its digit's next place with one shared atomic and goes
// there at once; a warp then writes whole digits.  Keys beyond their digit's
// places (uneven digits: a float's zeros) go to a list; more than the list
// holds send the tile through a dense stage, whose places need the tile's
// counts first (N(0, 1) floats with 1% zeros, 2^27: top split 606 -> 350 us
// with the list; 2 * 10^7 row identifiers, whole sort 240 -> 225).
// What bounds it: shared-memory wavefronts, 3.5 for a warp's access to random
// banks; this makes two such accesses a key, the dense stage three (2^28
// 4-byte keys: 0.43 against 0.58 ms).
template <int KB, int THREADS, int IPT, int CAP, class Code, class In, class Reload, class Refill>
__device__ __forceinline__ void msd_split_tile(typename KeyBits<KB>::U (&keys)[IPT], uint32_t lo, uint32_t hi,
                                               const Code& code_of, uint32_t shift, uint32_t nb, uint32_t* claim,
                                               typename KeyBits<KB>::U* dst, uint32_t n, uint32_t* err, uint8_t* smem,
                                               In in, Reload reload, Refill refill) {
    using U = typename KeyBits<KB>::U;
    using G = MsdSplitGeom<KB, THREADS, IPT, CAP>;
    constexpr int VEC = 16 / KB;
    U* stage = reinterpret_cast<U*>(smem);
    uint32_t* bins = reinterpret_cast<uint32_t*>(smem + G::WORDS_OFF);
    uint32_t* runs = bins + 256;  // u32 pairs: a digit's first place and its keys; dense: [256] twice
    uint32_t* scan = bins + 256 * 5 + 257;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool full = lo == 0u && hi == uint32_t(G::TILE);
    const uint32_t cap = nb == 256u ? uint32_t(CAP) : (uint32_t(G::STAGE) / nb - 1u) | 1u;
    auto digit = [&](U k) { return (code_of(k) >> shift) & (nb - 1u); };
    auto each = [&](auto f) {
        if (full) {
#pragma unroll
            for (int u = 0; u < IPT; ++u) f(u);
        } else {
#pragma unroll
            for (int u = 0; u < IPT; ++u) {
                const uint32_t j = uint32_t(u / VEC * THREADS + tid) * VEC + uint32_t(u % VEC);
                if (j >= lo && j < hi) f(u);
            }
        }
    };
    if constexpr (CAP == 0) {
        // dense stage: slots first, places once the tile's counts are scanned
        static_assert(IPT % 2 == 0 && G::TILE < 65536, "two slots to a register");
        uint32_t slot[IPT / 2];
#pragma unroll
        for (int u = 0; u < IPT / 2; ++u) slot[u] = 0u;
#pragma unroll
        for (int u = 0; u < IPT; ++u) keys[u] = in(keys[u]);
        each([&](int u) {
            slot[u / 2] = __byte_perm(slot[u / 2], atomicAdd(&bins[digit(keys[u])], 1u), (u & 1) ? 0x5410 : 0x3254);
        });
        __syncthreads();
        uint32_t c = 0, g = 0;
        if (uint32_t(tid) < nb) {
            c = bins[tid];
            if (c) g = atomicAdd(claim + tid, c);
        }
        const uint32_t ex = block_exclusive_scan_256<uint32_t>(c, scan, nullptr);
        if (uint32_t(tid) < nb) runs[tid] = ex;
        __syncthreads();
        each([&](int u) {
            stage[runs[digit(keys[u])] + __byte_perm(slot[u / 2], 0u, (u & 1) ? 0x4432 : 0x4410)] = keys[u];
        });
        if (uint32_t(tid) < nb) {
            runs[256 + tid] = g - ex;  // the claim's answer: only the write-out needs it
            bins[tid] = 0u;
        }
        refill();
        __syncthreads();
        bool bad = false;
        const uint32_t cnt = hi - lo;
#pragma unroll
        for (int u = 0; u < IPT; ++u) {  // coalesced runs, one per digit
            const uint32_t j = uint32_t(u * THREADS + tid);
            if (full || j < cnt) {
                const U k = stage[j];
                const uint32_t pos = runs[256 + digit(k)] + j;
                if (pos < n) dst[pos] = k;
                else bad = true;
            }
        }
        if (bad) atomicOr(err, ERRBIT_BOUNDS);
        __syncthreads();
        return;
    }
    U* spill = reinterpret_cast<U*>(smem + G::SPILL_OFF);
    uint32_t* spilled = scan + 32;
    each([&](int u) {
        const U k = in(keys[u]);
        const uint32_t d = digit(k);
        const uint32_t slot = atomicAdd(&bins[d], 1u);
        if (slot < cap) stage[d * cap + slot] = k;
        else {
            const uint32_t i = atomicAdd(spilled, 1u);
            if (i < uint32_t(G::SPILL)) spill[i] = k;
        }
    });
    __syncthreads();
    const uint32_t extra = *spilled;
    const bool over = extra > uint32_t(G::SPILL);
    uint32_t c = 0, g = 0;
    if (uint32_t(tid) < nb) {
        c = bins[tid];
        if (c) g = atomicAdd(claim + tid, c);
        bins[tid] = 0u;
    }
    bool bad = false;
    if (!over) {
        refill();
        if (uint32_t(tid) < nb) {
            if (uint64_t(g) + c > n) {
                bad = true;
                c = 0;
            }
            reinterpret_cast<uint2*>(runs)[tid] = make_uint2(g, min(c, cap));
        }
        __syncthreads();
        if (extra) {  // after their digit's staged keys
            for (uint32_t i = tid; i < extra; i += THREADS) {
                const U k = spill[i];
                const uint32_t d = digit(k), pos = reinterpret_cast<const uint2*>(runs)[d].x + cap + atomicAdd(&bins[d], 1u);
                if (pos < n) dst[pos] = k;
                else bad = true;
            }
            __syncthreads();
            if (uint32_t(tid) < nb) bins[tid] = 0u;
            if (tid == 0) *spilled = 0u;
        }
        // A warp writes a digit's keys 32 at a time, four digits in flight.
        // The digit's words reach the lanes by a broadcast read: shuffles
        // take the same pipe, and two would be needed.
        constexpr uint32_t WARPS = THREADS / 32, AHEAD = 4;
        if (nb == 256u) {
            constexpr int ROWS = (THREADS * IPT / 256 + 31) / 32;  // rows of a digit of average size
            const U* from = stage + warp * CAP + lane;
            const uint2* run = reinterpret_cast<const uint2*>(runs) + warp;
#pragma unroll 1
            for (uint32_t d0 = warp; d0 < 256u; d0 += AHEAD * WARPS) {
                U k[AHEAD][ROWS];
                uint2 w[AHEAD];
                uint32_t most = 0;
#pragma unroll
                for (uint32_t e = 0; e < AHEAD; ++e) {
                    w[e] = run[e * WARPS];
                    most = max(most, w[e].y);
#pragma unroll
                    for (int h = 0; h < ROWS; ++h)
                        if (lane + 32 * h < int(w[e].y)) k[e][h] = from[e * WARPS * CAP + 32 * h];
                }
#pragma unroll
                for (uint32_t e = 0; e < AHEAD; ++e) {
                    U* to = dst + (w[e].x + lane);
#pragma unroll
                    for (int h = 0; h < ROWS; ++h)
                        if (lane + 32 * h < int(w[e].y)) to[32 * h] = k[e][h];
                }
                if (most > 32u * ROWS) {
                    for (uint32_t e = 0; e < AHEAD; ++e) {
                        const uint2 v = run[e * WARPS];
                        for (uint32_t q = 32 * ROWS + lane; q < v.y; q += 32)
                            dst[v.x + q] = from[e * WARPS * CAP + q - lane];
                    }
                }
                from += AHEAD * WARPS * CAP;
                run += AHEAD * WARPS;
            }
        } else {  // fewer digits: cut into parts, 256 in all
            const uint32_t pl = 8u - (31u - __clz(nb));
            for (uint32_t item = warp; item < 256u; item += WARPS) {
                const uint32_t d = item >> pl, part = item & ((1u << pl) - 1u);
                const uint2 w = reinterpret_cast<const uint2*>(runs)[d];
                const U* from = stage + d * cap;
#pragma unroll 2
                for (uint32_t q = part * 32u + lane; q < w.y; q += 32u << pl) dst[w.x + q] = from[q];
            }
        }
    } else {
        __syncthreads();  // every zero of the bins is written
        const uint32_t ex = block_exclusive_scan_256<uint32_t>(c, scan, nullptr);
        if (uint32_t(tid) < nb) {
            runs[tid] = ex;
            runs[256 + tid] = g - ex;
        }
        reload();
        __syncthreads();
        each([&](int u) {
            const U k = in(keys[u]);
            const uint32_t d = digit(k);
            stage[runs[d] + atomicAdd(&bins[d], 1u)] = k;
        });
        refill();
        __syncthreads();
        if (uint32_t(tid) < nb) bins[tid] = 0u;
        if (tid == 0) *spilled = 0u;
        const uint32_t cnt = hi - lo;
        for (uint32_t j = tid; j < cnt; j += THREADS) {  // coalesced runs, one per digit
            const U k = stage[j];
            const uint32_t pos = runs[256 + digit(k)] + j;
            if (pos < n) dst[pos] = k;
            else bad = true;
        }
    }
    if (bad) atomicOr(err, ERRBIT_BOUNDS);
    __syncthreads();  // the stage and the digit words are free for the next tile
}

// Top split (8 bits), input -> alternate buffer.  Tiles start at 16-byte
// boundaries; each CTA's next tile loads while it writes one out.
template <int KB, int THREADS, int IPT, int MIN_CTAS, int CAP, bool EVEN>
__global__ void __launch_bounds__(THREADS, MIN_CTAS) msd_top_kernel(MsdParams p) {
    using U = typename KeyBits<KB>::U;
    using G = MsdSplitGeom<KB, THREADS, IPT, CAP>;
    extern __shared__ __align__(128) uint8_t smem[];
    uint32_t* bins = reinterpret_cast<uint32_t*>(smem + G::WORDS_OFF);
    const int tid = threadIdx.x;
    for (int i = tid; i < 256; i += THREADS) bins[i] = 0u;
    if (tid == 0) bins[256 * 5 + 257 + 32] = 0u;  // (the list's length)
    grid_launch_dependents();
    grid_dependency_wait();
    if (ld_relaxed(p.state) & MSD_OFF) return;
    const KeyMap<U> map(p.kind, p.desc);
    uint2* table = reinterpret_cast<uint2*>(smem + G::TABLE_OFF);
    if constexpr (EVEN) MsdEvenCode::fetch(p, table);  // (the barrier below)
    const auto code_of = msd_code<EVEN>(p, table);
    const U* keys_in = static_cast<const U*>(p.keys_in);
    const uint32_t skew = uint32_t(reinterpret_cast<uintptr_t>(keys_in) & 15u) / uint32_t(KB);
    const U* in = keys_in - skew;  // keys [skew, skew + n)
    const uint32_t n = uint32_t(p.n), end = n + skew;
    const uint32_t T = (end + G::TILE - 1) / G::TILE;
    U keys[IPT];
    auto load = [&](uint32_t t) {
        if (t >= T) return;
        const uint32_t b = t * uint32_t(G::TILE);
        msd_load_tile<KB, THREADS, IPT>(in + b, b == 0u ? skew : 0u, min(end - b, uint32_t(G::TILE)), keys);
    };
    uint32_t t = blockIdx.x;
    load(t);
    __syncthreads();
    for (; t < T; t += gridDim.x) {
        const uint32_t b = t * uint32_t(G::TILE);
        msd_split_tile<KB, THREADS, IPT, CAP>(
            keys, b == 0u ? skew : 0u, min(end - b, uint32_t(G::TILE)), code_of, 24u, 256u, p.cursor1, static_cast<U*>(p.keys_b),
            n, p.err, smem, [&](U k) { return map.in(k); }, [&] { load(t); }, [&] { load(t + gridDim.x); });
    }
}

// The tiles of the second level: every top bucket's keys from the 16-byte
// boundary at or below its first one, so that no tile crosses a bucket;
// tfirst[256] = the number of tiles.
__device__ __forceinline__ void msd_top_table(const uint32_t* top_counts, uint32_t tile, uint32_t vec, uint32_t skew,
                                              uint32_t* tstart, uint32_t* tcnt, uint32_t* tfirst, uint32_t* scan) {
    const int tid = threadIdx.x;
    const uint32_t c = (tid < 256) ? top_counts[tid] : 0u;
    const uint32_t ex = block_exclusive_scan_256<uint32_t>(c, scan, nullptr);
    __syncthreads();  // the scan words are read by every thread before the next scan writes them
    uint32_t tiles = 0;
    const uint32_t lead = (ex + skew) & (vec - 1u);
    const uint32_t tex =
        block_exclusive_scan_256<uint32_t>(c ? (lead + c + tile - 1) / tile : 0u, scan, &tiles);
    if (tid < 256) {
        tstart[tid] = ex;
        tcnt[tid] = c;
        tfirst[tid] = tex;
    }
    if (tid == 0) tfirst[256] = tiles;
    __syncthreads();
}

// The top bucket of second-level tile t: the last b with tfirst[b] <= t.
__device__ __forceinline__ uint32_t msd_bucket_of(const uint32_t* tfirst, uint32_t t) {
    uint32_t lo = 0, hi = 256;  // tfirst[lo] <= t < tfirst[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (tfirst[mid] <= t) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Second split: within every top bucket, into the groups' ranges (alternate
// buffer -> caller's buffer).
template <int KB, int THREADS, int IPT, int MIN_CTAS, int CAP, bool EVEN>
__global__ void __launch_bounds__(THREADS, MIN_CTAS) msd_second_kernel(MsdParams p) {
    using U = typename KeyBits<KB>::U;
    using G = MsdSplitGeom<KB, THREADS, IPT, CAP>;
    constexpr uint32_t VEC = 16 / KB;
    extern __shared__ __align__(128) uint8_t smem[];
    uint32_t* bins = reinterpret_cast<uint32_t*>(smem + G::WORDS_OFF);
    uint32_t* tstart = bins + 256 * 3;
    uint32_t* tcnt = tstart + 256;
    uint32_t* tfirst = tcnt + 256;
    uint32_t* scan = tfirst + 257;
    const int tid = threadIdx.x;
    for (int i = tid; i < 256; i += THREADS) bins[i] = 0u;
    if (tid == 0) bins[256 * 5 + 257 + 32] = 0u;  // (the list's length)
    grid_launch_dependents();
    grid_dependency_wait();
    if (ld_relaxed(p.state) & MSD_OFF) return;
    uint2* table = reinterpret_cast<uint2*>(smem + G::TABLE_OFF);
    if constexpr (EVEN) MsdEvenCode::fetch(p, table);  // (msd_top_table's barriers)
    const auto code_of = msd_code<EVEN>(p, table);
    const uint32_t b2 = code_of.b2;
    const U* in = static_cast<const U*>(p.keys_b);
    const uint32_t skew = uint32_t(reinterpret_cast<uintptr_t>(in) & 15u) / uint32_t(KB);
    msd_top_table(p.top_counts, G::TILE, VEC, skew, tstart, tcnt, tfirst, scan);
    const uint32_t T = tfirst[256];
    struct Tile {
        uint32_t b, lo, hi;
        const U* at;
    };
    auto tile = [&](uint32_t t) {
        Tile r;
        r.b = msd_bucket_of(tfirst, t);
        const uint32_t lead = (tstart[r.b] + skew) & (VEC - 1u);
        const uint32_t from = (t - tfirst[r.b]) * uint32_t(G::TILE);  // from the aligned start
        r.at = in + tstart[r.b] - lead + from;
        r.lo = from == 0u ? lead : 0u;
        r.hi = min(lead + tcnt[r.b] - from, uint32_t(G::TILE));
        return r;
    };
    U keys[IPT];
    uint32_t t = blockIdx.x;
    if (t >= T) return;
    Tile cur = tile(t);
    msd_load_tile<KB, THREADS, IPT>(cur.at, cur.lo, cur.hi, keys);
    for (; t < T; t += gridDim.x) {
        Tile next = cur;
        msd_split_tile<KB, THREADS, IPT, CAP>(
            keys, cur.lo, cur.hi, code_of, 24u - b2, 1u << b2, p.cursor2 + (cur.b << b2), static_cast<U*>(p.keys_a),
            uint32_t(p.n), p.err, smem, [](U k) { return k; },
            [&] { msd_load_tile<KB, THREADS, IPT>(cur.at, cur.lo, cur.hi, keys); },
            [&] {
                if (t + gridDim.x < T) {
                    next = tile(t + gridDim.x);
                    msd_load_tile<KB, THREADS, IPT>(next.at, next.lo, next.hi, keys);
                }
            });
        cur = next;
    }
}

// ---- local sorts ----------------------------------------------------------
// Largest sub-bucket ranked by comparison where the network's margin is too
// narrow (below); a larger one sends the whole sort to the digit passes.
constexpr uint32_t MSD_RANK_MAX = 32;

// Shared memory of a local sort by BINS = 16 * THREADS sub-buckets.  Keys lie
// in chunks of 64 bytes (LIPT keys, a lane's share), 80 bytes apart: sixteen
// bytes of padding put the chunks of eight lanes on all 32 banks.
// HALO lanes at either end of a warp hold its neighbours' keys: after m
// rounds of the network a key has met every key at most m places away, so a
// warp's inner lanes end up right when m <= HALO * LIPT.
template <int KB, int THREADS, int HALO>
struct GroupSortGeom {
    static constexpr int LIPT = 64 / KB;
    static constexpr int WARPS = THREADS / 32;
    static constexpr int BINS = 16 * THREADS;
    static constexpr int OUT = (32 - 2 * HALO) * LIPT;  // keys a warp puts in order
    static constexpr int PLACES = WARPS * OUT;
    static constexpr int ALIGN = 32 / KB;               // places keep the keys' position in their 32-byte sector
    static constexpr int CAP = PLACES - ALIGN;
    static_assert(PLACES < 65536, "16-bit places");
    static constexpr size_t KEYS_BYTES = size_t(PLACES / LIPT) * 80;
    static constexpr size_t CTR_OFF = (KEYS_BYTES + 127) & ~size_t(127);  // u8 [BINS]
    static constexpr size_t START_OFF = CTR_OFF + BINS;                   // u16 [BINS]
    static constexpr size_t SCAN_OFF = START_OFF + size_t(BINS) * 2;      // u32 [32]
    static constexpr size_t MISC_OFF = SCAN_OFF + 128;                    // u32 [4]
    static constexpr size_t SMEM_BYTES = MISC_OFF + 16;
    // byte address of a place
    __device__ __forceinline__ static uint32_t at(uint32_t place) {
        return place * uint32_t(KB) + (place & ~uint32_t(LIPT - 1)) * uint32_t(16 / LIPT);
    }
};

__device__ __forceinline__ void order_pair(uint32_t& a, uint32_t& b) {
    const uint32_t lo = min(a, b), hi = max(a, b);
    a = lo;
    b = hi;
}
template <class U>
__device__ __forceinline__ void order_pair(U& a, U& b) {
    const bool sw = b < a;
    const U lo = sw ? b : a, hi = sw ? a : b;
    a = lo;
    b = hi;
}
template <class U>
__device__ __forceinline__ U shfl_up1(U v) {
    if constexpr (sizeof(U) <= 8) return __shfl_up_sync(0xffffffffu, v, 1);
    else {
        const uint64_t lo = __shfl_up_sync(0xffffffffu, uint64_t(v), 1);
        const uint64_t hi = __shfl_up_sync(0xffffffffu, uint64_t(v >> 64), 1);
        return (U(hi) << 64) | U(lo);
    }
}
template <class U>
__device__ __forceinline__ U shfl_down1(U v) {
    if constexpr (sizeof(U) <= 8) return __shfl_down_sync(0xffffffffu, v, 1);
    else {
        const uint64_t lo = __shfl_down_sync(0xffffffffu, uint64_t(v), 1);
        const uint64_t hi = __shfl_down_sync(0xffffffffu, uint64_t(v >> 64), 1);
        return (U(hi) << 64) | U(lo);
    }
}

// The ascending network over places 0 .. m - 1, any m, by `threads` threads:
// order(a, b) puts the pair of places a < b in order, sync() orders one step's
// accesses before the next's.  Every step's first half meets its second half
// mirrored, so that all comparisons point up and places from m on, which
// would hold greatest keys, never take part.
template <class Order, class Sync>
__device__ __forceinline__ void ascending_network(uint32_t m, uint32_t thread, uint32_t threads, Order order, Sync sync) {
    uint32_t half = 1;
    while (2u * half < m) half *= 2u;
    if (m < 2u) return;
    for (uint32_t size = 2; size <= 2u * half; size *= 2u) {
        for (uint32_t i = thread; i < half; i += threads) {
            const uint32_t in = i & (size / 2u - 1u), first = 2u * (i - in);
            if (first + size - 1u - in < m) order(first + in, first + size - 1u - in);
        }
        sync();
        for (uint32_t gap = size / 4u; gap != 0u; gap /= 2u) {
            for (uint32_t i = thread; i < half; i += threads) {
                const uint32_t a = 2u * i - (i & (gap - 1u));
                if (a + gap < m) order(a, a + gap);
            }
            sync();
        }
    }
}

// `rounds` rounds of odd-even transposition over the warp's 32 * LIPT keys,
// LIPT consecutive ones per lane.
template <class U, int LIPT>
__device__ __forceinline__ void transposition_rounds(U (&k)[LIPT], uint32_t rounds, int lane) {
    for (uint32_t r = 0; r < rounds; r += 2) {
#pragma unroll
        for (int i = 0; i + 1 < LIPT; i += 2) order_pair(k[i], k[i + 1]);
        if (r + 1 < rounds) {
            const U before = shfl_up1(k[LIPT - 1]), after = shfl_down1(k[0]);
#pragma unroll
            for (int i = 1; i + 1 < LIPT; i += 2) order_pair(k[i], k[i + 1]);
            if (lane > 0 && before > k[0]) k[0] = before;
            if (lane < 31 && after < k[LIPT - 1]) k[LIPT - 1] = after;
        }
    }
}

// Sorts the CTA's `cnt` keys, all of one group: key VEC * i + e of a thread
// (VEC = 16 bytes' worth) is the group's key (i * THREADS + tid) * VEC + e -
// skew when that is below cnt, else nothing.  bin(key) names its sub-bucket (monotone in the key, 0 ..
// BINS-1).  Place p of the sorted group (p < cnt) is reported as pad + p, pad
// < ALIGN: chunk(c0, k) hands out the LIPT keys of places c0 .. (those of
// [pad, pad + cnt) count), one(place, key) a single key.  refill() runs when
// the keys' registers are free.  Returns false, having called none of these,
// when a sub-bucket is too big.
// The counters of the sub-buckets are bytes, four to a word: one 16-byte read
// per thread scans sixteen; a count that passes 255 loses at least 255 keys
// from the total, which shows.  They are zero on entry and left so.
// What bounds it: a random shared-memory access costs about 2.5 SM clocks a
// warp; a key needs three (the counter's atomic, whose answer is its slot,
// its sub-bucket's start, its place), and one conflict-free read.
template <class U, int THREADS, int HALO, class Bin, class Refill, class Chunk, class One>
__device__ __forceinline__ bool group_sort(const U (&keys)[64 / sizeof(U)], uint32_t cnt, uint32_t skew,
                                           uint32_t pad, uint8_t* smem, Bin bin, Refill refill, Chunk chunk, One one) {
    using G = GroupSortGeom<int(sizeof(U)), THREADS, HALO>;
    constexpr int LIPT = G::LIPT;
    constexpr int VEC = 16 / int(sizeof(U));
    auto sk = [&](uint32_t place) -> U& { return *reinterpret_cast<U*>(smem + G::at(place)); };
    uint32_t* ctr = reinterpret_cast<uint32_t*>(smem + G::CTR_OFF);
    uint16_t* start = reinterpret_cast<uint16_t*>(smem + G::START_OFF);
    uint32_t* scan = reinterpret_cast<uint32_t*>(smem + G::SCAN_OFF);
    uint32_t* misc = reinterpret_cast<uint32_t*>(smem + G::MISC_OFF);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t slot[(LIPT + 3) / 4];
#pragma unroll
    for (int u = 0; u < (LIPT + 3) / 4; ++u) slot[u] = 0u;
    // rows of VEC keys; a warp whose row lies past the group skips it
    auto rows = [&](auto f) {
#pragma unroll
        for (int i = 0; i < LIPT / VEC; ++i) {
            if (uint32_t(i * THREADS + warp * 32) * VEC >= skew + cnt) break;
            if (i != 0 || skew == 0u || warp != 0)  // (a warp of whole vectors: no test per key)
                if (uint32_t(i * THREADS + warp * 32 + 32) * VEC <= skew + cnt) {
#pragma unroll
                    for (int e = 0; e < VEC; ++e) f(i * VEC + e);
                    continue;
                }
            const uint32_t j = uint32_t(i * THREADS + tid) * VEC - skew;
#pragma unroll
            for (int e = 0; e < VEC; ++e)
                if (j + e < cnt) f(i * VEC + e);
        }
    };
    rows([&](int u) {
        const uint32_t b = bin(keys[u]);
        const uint32_t old = atomicAdd(reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(ctr) + (b & ~3u)),
                                       __funnelshift_l(1u, 1u, b * 8u));
        // byte (b & 3) of old into byte (u & 3) of the slots
        const uint32_t x = __funnelshift_r(old, old, b * 8u);
        slot[u >> 2] = __byte_perm(slot[u >> 2], x, (u & 3) == 0 ? 0x3214 : (u & 3) == 1 ? 0x3240 : (u & 3) == 2 ? 0x3410 : 0x4210);
    });
    __syncthreads();
    // scan: sixteen consecutive counters a thread
    {
        const uint4 c = reinterpret_cast<const uint4*>(ctr)[tid];
        uint32_t big = __vmaxu4(__vmaxu4(c.x, c.y), __vmaxu4(c.z, c.w));
        big = max(max(big & 0xffu, (big >> 8) & 0xffu), max((big >> 16) & 0xffu, big >> 24));
        const uint32_t sum = __dp4a(c.x, 0x01010101u, __dp4a(c.y, 0x01010101u, __dp4a(c.z, 0x01010101u, __dp4a(c.w, 0x01010101u, 0u))));
        big = __reduce_max_sync(0xffffffffu, big);
        if (lane == 0 && big > 1u) atomicMax(&misc[0], big);
        uint32_t run = block_exclusive_scan_1b<THREADS>(sum, scan);
        if (tid == THREADS - 1 && run + sum != cnt) atomicMax(&misc[0], 256u);
        run += pad;
        auto pack = [&](uint32_t w, uint32_t& lo, uint32_t& hi) {
            const uint32_t b = run + (w & 0xffu), d = b + ((w >> 8) & 0xffu), e = d + ((w >> 16) & 0xffu);
            lo = run | b << 16;
            hi = d | e << 16;
            run = e + (w >> 24);
        };
        uint4 v0, v1;
        pack(c.x, v0.x, v0.y);
        pack(c.y, v0.z, v0.w);
        pack(c.z, v1.x, v1.y);
        pack(c.w, v1.z, v1.w);
        reinterpret_cast<uint4*>(start)[tid * 2] = v0;
        reinterpret_cast<uint4*>(start)[tid * 2 + 1] = v1;
        reinterpret_cast<uint4*>(ctr)[tid] = make_uint4(0u, 0u, 0u, 0u);
    }
    __syncthreads();
    const uint32_t most = misc[0];
    if (most > MSD_RANK_MAX) {
        __syncthreads();
        if (tid == 0) misc[0] = 0u;
        return false;
    }
    rows([&](int u) { sk(start[bin(keys[u])] + __byte_perm(slot[u >> 2], 0u, 0x4440u | (u & 3))) = keys[u]; });
    __syncthreads();
    if (tid == 0) misc[0] = 0u;  // read by every thread before the barrier
    refill();
    const uint32_t end = pad + cnt;
    if (most <= uint32_t(HALO * LIPT)) {
        // chunks [warp * (32 - 2 HALO), ...) and the neighbours' beyond both ends
        const int ch = warp * (32 - 2 * HALO) + lane - HALO;
        const int c0 = ch * LIPT;
        if (warp * G::OUT < int(end)) {
            U k[LIPT];
            const bool inside = c0 >= int(pad) && uint32_t(c0 + LIPT) <= end;
            if (c0 + LIPT <= int(pad) || c0 >= int(end)) {
#pragma unroll
                for (int i = 0; i < LIPT; ++i) k[i] = c0 < int(pad) ? U(0) : U(~U(0));
            } else {
                const uint4* q = reinterpret_cast<const uint4*>(smem + uint32_t(ch) * 80u);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    union { uint4 v; U k[16 / sizeof(U)]; } w;
                    w.v = q[i];
#pragma unroll
                    for (int e = 0; e < int(16 / sizeof(U)); ++e) k[i * (16 / sizeof(U)) + e] = w.k[e];
                }
                if (!inside) {
#pragma unroll
                    for (int i = 0; i < LIPT; ++i) {
                        if (c0 + i < int(pad)) k[i] = U(0);
                        if (c0 + i >= int(end)) k[i] = U(~U(0));
                    }
                }
            }
            if (most > 1u) transposition_rounds<U, LIPT>(k, most, lane);
            if (lane >= HALO && lane < 32 - HALO && c0 < int(end)) chunk(uint32_t(c0), inside, k);
        }
    } else {
        // a key's place is its sub-bucket's start plus the sub-bucket's other
        // keys below it
        for (uint32_t i = pad + tid; i < end; i += THREADS) {
            const U k = sk(i);
            const uint32_t b = bin(k);
            const uint32_t s = start[b], e = b + 1 < uint32_t(G::BINS) ? uint32_t(start[b + 1]) : end;
            uint32_t below = 0;
            for (uint32_t q = s; q < e; ++q) {
                const U o = sk(q);
                below += uint32_t(o < k || (o == k && q < i));
            }
            one(s + below, k);
        }
    }
    return true;
}

// Sub-bucket of a key in its group: the 32 bits of its code after the `shift`
// that the group's keys share, evenly over the bins.
template <class Code>
struct SubBucket {
    Code code;
    uint32_t shift, bins;
    template <class U>
    __device__ __forceinline__ uint32_t operator()(U x) const { return __umulhi(code(x) << shift, bins); }
};

// A group that group_sort refuses (keys that repeat, or that share the
// sub-bucket's bits), from global memory, sorted in place and mapped back.  The
// same counting pass with 16-bit counters, then only sub-buckets whose keys
// differ are put in order: small ones by comparison, larger ones by a network
// of one warp, the largest by the CTA; equal keys, the usual crowd, need
// nothing.  Counters and misc[0] are zero on entry and left so.
template <class U, int THREADS, int HALO, class Bin>
__device__ __noinline__ void group_sort_crowded(U* group, uint32_t cnt, uint8_t* smem, Bin bin, KeyMap<U> map) {
    using G = GroupSortGeom<int(sizeof(U)), THREADS, HALO>;
    constexpr uint32_t BY_THREAD = 16, BY_WARP = 512;
    uint32_t* flags = reinterpret_cast<uint32_t*>(smem + G::CTR_OFF);  // a byte a sub-bucket whose keys differ: 1 large, 2 small
    uint32_t* place = reinterpret_cast<uint32_t*>(smem + G::START_OFF);
    const uint16_t* ends = reinterpret_cast<const uint16_t*>(place);
    uint32_t* scan = reinterpret_cast<uint32_t*>(smem + G::SCAN_OFF);
    uint32_t* misc = reinterpret_cast<uint32_t*>(smem + G::MISC_OFF);  // [1] sub-buckets left to the CTA
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto sk = [&](uint32_t i) -> U& { return *reinterpret_cast<U*>(smem + G::at(i)); };
    auto first_of = [&](uint32_t b) { return b ? uint32_t(ends[b - 1]) : 0u; };
    auto order = [&](uint32_t a, uint32_t b) {
        const U x = sk(a), y = sk(b);
        if (y < x) {
            sk(a) = y;
            sk(b) = x;
        }
    };
    __syncthreads();
    for (uint32_t i = tid; i < uint32_t(G::BINS) / 2; i += THREADS) place[i] = 0u;
    if (tid == 0) misc[1] = 0u;
    __syncthreads();
    for (uint32_t i = tid; i < cnt; i += THREADS) {
        const uint32_t b = bin(group[i]);
        atomicAdd(&place[b >> 1], 1u << 16 * (b & 1u));
    }
    __syncthreads();
    {
        uint4 w[2] = {reinterpret_cast<uint4*>(place)[2 * tid], reinterpret_cast<uint4*>(place)[2 * tid + 1]};
        uint32_t* c = reinterpret_cast<uint32_t*>(w);
        uint32_t sum = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) sum += (c[i] & 0xffffu) + (c[i] >> 16);
        uint32_t run = block_exclusive_scan_1b<THREADS>(sum, scan);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t next = run + (c[i] & 0xffffu), after = next + (c[i] >> 16);
            c[i] = run | next << 16;
            run = after;
        }
        reinterpret_cast<uint4*>(place)[2 * tid] = w[0];
        reinterpret_cast<uint4*>(place)[2 * tid + 1] = w[1];
    }
    __syncthreads();
    for (uint32_t i = tid; i < cnt; i += THREADS) {
        const U k = group[i];
        const uint32_t b = bin(k);
        sk((atomicAdd(&place[b >> 1], 1u << 16 * (b & 1u)) >> 16 * (b & 1u)) & 0xffffu) = k;
    }
    __syncthreads();  // now a sub-bucket's word is its end
    for (uint32_t i = tid; i < cnt; i += THREADS) {
        const U k = sk(i);
        const uint32_t b = bin(k), first = first_of(b);
        if (i > first && sk(i - 1) != k)
            atomicOr(&flags[b >> 2], (ends[b] - first > BY_THREAD ? 1u : 2u) << 8 * (b & 3u));
    }
    __syncthreads();
    for (uint32_t w0 = warp * 32; w0 < uint32_t(G::BINS) / 4; w0 += THREADS) {
        const uint32_t mine = flags[w0 + lane];
        for (uint32_t some = __ballot_sync(0xffffffffu, (mine & 0x01010101u) != 0u); some; some &= some - 1u) {
            const int l = __ffs(some) - 1;
            const uint32_t word = __shfl_sync(0xffffffffu, mine, l);
            for (uint32_t q = 0; q < 4; ++q) {
                if (!(word >> 8 * q & 1u)) continue;
                const uint32_t b = (w0 + l) * 4 + q, first = first_of(b), m = ends[b] - first;
                if (m > BY_WARP) {
                    if (lane == 0) scan[atomicAdd(&misc[1], 1u)] = b;
                } else {
                    ascending_network(
                        m, lane, 32u, [&](uint32_t x, uint32_t y) { order(first + x, first + y); }, [] { __syncwarp(); });
                }
            }
        }
    }
    static_assert(G::PLACES / BY_WARP <= 32, "the list of sub-buckets");
    __syncthreads();
    const uint32_t left = misc[1];
    for (uint32_t g = 0; g < left; ++g) {
        const uint32_t first = first_of(scan[g]), m = ends[scan[g]] - first;
        ascending_network(
            m, tid, THREADS, [&](uint32_t x, uint32_t y) { order(first + x, first + y); }, [] { __syncthreads(); });
    }
    for (uint32_t i = tid; i < cnt; i += THREADS) {
        const U k = sk(i);
        const uint32_t b = bin(k), first = first_of(b), m = ends[b] - first;
        uint32_t at = i;
        if (flags[b >> 2] >> 8 * (b & 3u) & 2u) {
            at = first;
            for (uint32_t q = first; q < first + m; ++q) {
                const U o = sk(q);
                at += uint32_t(o < k || (o == k && q < i));
            }
        }
        group[at] = map.out(k);
    }
    __syncthreads();
    for (uint32_t i = tid; i < uint32_t(G::BINS) / 4; i += THREADS) flags[i] = 0u;
    __syncthreads();
}

// 32 bytes to a 32-byte aligned address.
__device__ __forceinline__ void store_32b(void* dst, const uint4& a, const uint4& b) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(a.x), "r"(a.y), "r"(a.z),
                 "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

// Local sorts: groups blockIdx.x, + gridDim.x, ... sorted in place.  The next
// group's keys load while the network runs, and the one after it is pulled
// into L2.
template <int KB, int THREADS, int MIN_CTAS, int HALO, bool EVEN>
__global__ void __launch_bounds__(THREADS, MIN_CTAS) msd_local_kernel(MsdParams p) {
    using U = typename KeyBits<KB>::U;
    using G = GroupSortGeom<KB, THREADS, HALO>;
    constexpr int LIPT = G::LIPT, VEC = 16 / KB;
    extern __shared__ __align__(128) uint8_t smem[];
    grid_launch_dependents();
    const int tid = threadIdx.x;
    for (int i = tid; i < G::BINS / 4; i += THREADS) reinterpret_cast<uint32_t*>(smem + G::CTR_OFF)[i] = 0u;
    if (tid == 0) *reinterpret_cast<uint32_t*>(smem + G::MISC_OFF) = 0u;
    grid_dependency_wait();
    if (ld_relaxed(p.state) & MSD_OFF) return;
    __syncthreads();
    U* keys = static_cast<U*>(p.keys_a);
    // (floats: a group's keys share few bins, so the table's reads are broadcasts)
    auto code_of = msd_code<EVEN>(p, p.table);
    using Code = decltype(code_of);
    auto groups = [&] { return 256u << code_of.b2; };
    // The CTA's groups in turn: g, + gridDim.x, ...  Floats: two neighbours are
    // sorted as one where they fit, since their groups, as many as the densest
    // stretch needs, are small (6 * 10^7 keys of N(0, 1): 336 -> 243 us).
    struct Group {
        uint32_t off, word;  // word: its keys, below 2^16, and the leading bits that their codes share; 0: none left
        __device__ __forceinline__ uint32_t cnt() const { return word & 0xffffu; }
    };
    uint32_t ahead = blockIdx.x, half = 0u;  // the next one
    auto next_group = [&] {
        Group r{0u, 0u};
        if constexpr (EVEN) {
            if (ahead * 2u < groups()) {
                const uint32_t a = ahead ? p.cursor2[ahead * 2u - 1u] : 0u, b = p.cursor2[ahead * 2u], c = p.cursor2[ahead * 2u + 1u];
                const bool both = c - a <= p.group_cap;
                r.off = half ? b : a;
                uint32_t cnt = (both || half ? c : b) - r.off;
                if (cnt > p.group_cap) cnt = 0u;  // equal keys, below
                r.word = cnt | (8u + code_of.b2 - uint32_t(both)) << 16;
                half = both ? 0u : half ^ 1u;
                if (half) return r;
            }
        } else if (ahead < groups()) {
            r.off = ahead ? p.cursor2[ahead - 1u] : 0u;
            // (above the largest: one of the ranges left)
            r.word = min(p.cursor2[ahead] - r.off, 0xffffu) | (8u + code_of.b2) << 16;
        }
        ahead += gridDim.x;
        return r;
    };
    // Key VEC * i + e of a thread is the group's key
    // (i * THREADS + tid) * VEC + e - shift: 16-byte loads from the address
    // at or below the group's start (which keys a thread has does not matter)
    KeyMap<U> map(p.kind, p.desc);
    Group cur = next_group(), next = next_group();
    U k[LIPT];
    auto skew_of = [&](uint32_t o, uint32_t bytes) {
        return uint32_t(reinterpret_cast<uintptr_t>(keys + o) & (bytes - 1u)) / uint32_t(KB);
    };
    auto index = [&](uint32_t skew, int u) { return (uint32_t(u / VEC) * THREADS + tid) * VEC + uint32_t(u % VEC) - skew; };
    auto load = [&](const Group& f) {
        const uint32_t skew = skew_of(f.off, 16);
        load_vectors<THREADS>(const_cast<const U*>(keys) + f.off - skew, skew, skew + f.cnt(), k);
    };
    // A group that has to go another way (crowded) leaves the loop, and what the
    // loop knows goes through shared memory: nothing of it lives across the
    // call, which would otherwise spill in the usual path (5 x 10^7 u64 keys, the
    // whole sort 859 us with a call in the loop, 809 this way).  Wide keys keep
    // the two groups ahead too, 4-byte keys find them again: each as it spills less.
    constexpr bool KEEP = KB > 4;
    __shared__ uint32_t left_at[8];
    load(cur);
    for (;;) {
        while (cur.word != 0u) {
            const Group later = next_group();
            const uint32_t off = cur.off, cnt = cur.cnt();
            const bool some = cnt - 1u < p.group_cap;
            {
                const uintptr_t a = reinterpret_cast<uintptr_t>(keys + later.off) & ~uintptr_t(127);
                const uintptr_t e = reinterpret_cast<uintptr_t>(keys + later.off + later.cnt());
                for (uintptr_t q = a + uintptr_t(tid) * 128; q < e; q += uintptr_t(THREADS) * 128)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(q));
            }
            const uint32_t skew = skew_of(off, 16), pad = skew_of(off, 32);
            U* dst = keys + off - pad;  // place q goes to dst[q]
            bool sorted = true;
            if (some)
                sorted = group_sort<U, THREADS, HALO>(
                    k, cnt, skew, pad, smem,
                    SubBucket<Code>{code_of, cur.word >> 16, uint32_t(G::BINS)},
                    [&] { load(next); },
                    [&](uint32_t c0, bool inside, const U(&x)[LIPT]) {
                        union { uint4 q[4]; U k[LIPT]; } w;
#pragma unroll
                        for (int i = 0; i < LIPT; ++i) w.k[i] = map.out(x[i]);
                        if (inside) {
                            store_32b(dst + c0, w.q[0], w.q[1]);
                            store_32b(dst + c0 + LIPT / 2, w.q[2], w.q[3]);
                        } else {
#pragma unroll
                            for (int i = 0; i < LIPT; ++i)
                                if (c0 + i >= pad && c0 + i < pad + cnt) dst[c0 + i] = w.k[i];
                        }
                    },
                    [&](uint32_t place, U x) { dst[place] = map.out(x); });
            if (!sorted) {
                if constexpr (!EVEN) {
                    if (tid == 0) {
                        left_at[0] = cur.off;
                        left_at[1] = cur.word;
                        left_at[2] = KEEP ? ahead : ahead - 2u * gridDim.x;  // (the group after this one)
                        if constexpr (KEEP) {
                            left_at[3] = next.off;
                            left_at[4] = next.word;
                            left_at[5] = later.off;
                            left_at[6] = later.word;
                        }
                    }
                    break;
                }
                if constexpr (EVEN) {
                    // equal keys are in order, and values that the sample has
                    // missed take a bitonic network over the group, 91 steps at
                    // most, where a sort that gave up would be lost
                    U* sk = reinterpret_cast<U*>(smem);
#pragma unroll
                    for (int u = 0; u < LIPT; ++u)
                        if (index(skew, u) < cnt) sk[index(skew, u)] = k[u];
                    __syncthreads();
                    bool differ = false;
                    for (uint32_t i = tid; i < cnt; i += THREADS) differ |= sk[i] != sk[0];
                    differ = __syncthreads_or(differ) != 0;
                    uint32_t size = 1024u;
                    static_assert(KB != 4 || 8192 * KB <= int(G::SCAN_OFF), "the group padded to a power of two");
                    while (size < cnt) size *= 2u;
                    for (uint32_t i = cnt + tid; i < size; i += THREADS) sk[i] = U(~U(0));
                    for (uint32_t run = 2; differ && run <= size; run *= 2u)
                        for (uint32_t gap = run / 2u; gap != 0u; gap /= 2u) {
                            __syncthreads();
                            for (uint32_t i = tid; i < size / 2u; i += THREADS) {
                                const uint32_t a = 2u * i - (i & (gap - 1u)), b = a + gap;
                                U x = sk[a], y = sk[b];
                                if ((x > y) == ((a & run) == 0u)) {
                                    sk[a] = y;
                                    sk[b] = x;
                                }
                            }
                        }
                    __syncthreads();
                    for (uint32_t i = tid; i < cnt; i += THREADS) keys[off + i] = map.out(sk[i]);
                    __syncthreads();
                    for (int i = tid; i < G::BINS / 4; i += THREADS) reinterpret_cast<uint32_t*>(smem + G::CTR_OFF)[i] = 0u;
                    __syncthreads();
                }
            }
            if (!sorted || !some) load(next);
            cur = next;
            next = later;
        }
        if (EVEN || cur.word == 0u) break;
        if constexpr (!EVEN) {
            __syncthreads();
            const volatile uint32_t* at = left_at;
            group_sort_crowded<U, THREADS, HALO>(keys + at[0], at[1] & 0xffffu, smem,
                                                 SubBucket<Code>{code_of, at[1] >> 16, uint32_t(G::BINS)}, map);
            code_of = Code(p);
            map = KeyMap<U>(p.kind, p.desc);
            ahead = at[2];
            cur = KEEP ? Group{at[3], at[4]} : next_group();
            next = KEEP ? Group{at[5], at[6]} : next_group();
            load(cur);
        }
    }
    if constexpr (EVEN) {
        // groups of equal keys above the largest: every CTA takes a slice and
        // looks whether they are
        const uint32_t giants = min(p.giants[0], MSD_GIANTS);
        for (uint32_t i = 0; i < giants; ++i) {
            const uint32_t gi = p.giants[1 + 2 * i], value = p.giants[2 + 2 * i];
            const uint32_t from = gi != 0u ? p.cursor2[gi - 1] : 0u, to = p.cursor2[gi];
            bool d = false;
            for (uint64_t j = uint64_t(from) + blockIdx.x * THREADS + tid; j < to; j += uint64_t(gridDim.x) * THREADS) {
                const U x = keys[j];
                d |= x != value;
                keys[j] = map.out(x);
            }
            if (__syncthreads_or(d) && tid == 0) atomicOr(p.state, MSD_GAVE_UP);
        }
    }
}

// The groups above the largest, mapped back unsorted: only where the launch that
// sorts them is refused, and the digit passes sort everything instead.
template <int KB>
__global__ void __launch_bounds__(256) msd_map_ranges_kernel(MsdParams p) {
    using U = typename KeyBits<KB>::U;
    if (ld_relaxed(p.state) & MSD_OFF) return;
    const KeyMap<U> map(p.kind, p.desc);
    const uint32_t ranges = min(ld_relaxed(p.left.count), p.left.most);
    for (uint32_t i = 0; i < ranges; ++i) {
        U* keys = static_cast<U*>(p.keys_a) + p.left.ranges[2 * i];
        for (uint32_t j = blockIdx.x * 256 + threadIdx.x; j < p.left.ranges[2 * i + 1]; j += gridDim.x * 256)
            keys[j] = map.out(keys[j]);
    }
}

}  // namespace gbsort
