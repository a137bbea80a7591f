// short_pairs.cuh — key-value sort of a short array in one cooperative launch
// (sm_103a): keys of 4 and 8 bytes that are not floats, values of 4 and 8.
//
// A short array is bound by latency: a digit pass per key byte is a chain of
// dependent round trips each.  Here every pair becomes one word, its twiddled
// key above its index; words are unique, so an unstable sort of them is the
// stable sort of the pairs, and it goes most significant bits first:
//   partition: every CTA spreads its keys over 256 to 912 regions of the
//              workspace by their leading bits that vary (a sample of the keys
//              says which, and how far they reach), with one global atomic per
//              region and tile; in place, it also copies the values aside;
//   one grid barrier;
//   buckets:   each CTA sorts whole regions in shared memory (group_sort) and
//              writes the keys and, fetched by index, the values.  Where many
//              keys are equal a sub-bucket outgrows group_sort, and the region
//              is sorted by a bitonic network over its words instead.
// A region that overflows, or a key outside the sampled bits, raises a flag
// before the barrier; every CTA then counts the digits, and the digit passes,
// launched after this kernel, sort from the untouched input.
#pragma once

#include "msd.cuh"

namespace gbsort {

struct ShortPairsParams {
    HistParams hist;        // the digit counts and status clear for the digit passes
    const void* keys_in;
    const void* vals_in;
    void* vals_aside;       // in place: the values' copy; nullptr: vals_in is not written
    void* keys_out;
    void* vals_out;
    uint32_t n;
    int kind, desc;
    uint32_t nb;            // regions (<= 1024)
    void* regions;          // [nb][cap] words
    uint32_t cap;
    uint32_t* fill;         // [nb] words in each region, zeroed
    uint32_t* state;        // MSD_OFF: the digit passes sort; zeroed
    uint32_t* barrier;
    uint32_t* barrier_gen;
    uint64_t wait_limit_ns;
    uint32_t* err;
};

// Region of a key, and its place in the region's range as a 32-bit fraction:
// codes 0 .. top (a little above the sample's largest) over the regions.
struct RegionOf {
    uint32_t nb, mult;
    __device__ __forceinline__ RegionOf(uint32_t regions, uint32_t top) : nb(regions) {
        const uint64_t reach = uint64_t(top) + (top >> 9) + 1u;
        const uint64_t m = ((uint64_t(regions) << 32) - 1u) / reach;
        mult = m > 0xffffffffull ? 0xffffffffu : uint32_t(m);
    }
    __device__ __forceinline__ void operator()(uint32_t code, uint32_t& region, uint32_t& frac) const {
        const uint64_t x = uint64_t(code) * mult;
        region = uint32_t(x >> 32);
        frac = uint32_t(x);
        if (region >= nb) {
            region = nb - 1u;
            frac = 0xffffffffu;
        }
    }
};

template <int KB> struct PairWord;
template <> struct PairWord<4> { using W = uint64_t; };
template <> struct PairWord<8> { using W = u128; };

template <int KB, int THREADS, int HALO>
struct ShortPairsGeom {
    using G = GroupSortGeom<2 * KB, THREADS, HALO>;
    static constexpr int CAP = (G::PLACES - 8) & ~3;  // words a region may hold (places keep a 32-byte alignment)
    static constexpr int PADDED = KB == 4 ? 4096 : 2048;
    static_assert(CAP <= PADDED && size_t(PADDED) * 2 * KB <= G::SCAN_OFF, "the bitonic sort's words");
    static constexpr size_t BINS_OFF = (G::SMEM_BYTES + 15) & ~size_t(15);  // u32 [1024] tile counts, then first places
    static constexpr size_t CLAIM_OFF = BINS_OFF + 4096;                    // u32 [1024] claims, then sizes
    static constexpr size_t SMEM_BYTES = CLAIM_OFF + 4096;
};

template <int KB, int VB, int THREADS, int MIN_CTAS, int HALO>
__global__ void __launch_bounds__(THREADS, MIN_CTAS) short_pairs_kernel(ShortPairsParams p) {
    using U = typename KeyBits<KB>::U;
    using V = typename ValBits<VB>::V;
    using W = typename PairWord<KB>::W;
    using S = ShortPairsGeom<KB, THREADS, HALO>;
    using G = typename S::G;
    constexpr int LIPT = G::LIPT, VEC = 16 / int(sizeof(W)), IPT = 8;
    extern __shared__ __align__(128) uint8_t smem[];
    uint32_t* bins = reinterpret_cast<uint32_t*>(smem + S::BINS_OFF);
    uint32_t* claims = reinterpret_cast<uint32_t*>(smem + S::CLAIM_OFF);
    uint32_t* scan = reinterpret_cast<uint32_t*>(smem + G::SCAN_OFF);
    uint32_t* misc = reinterpret_cast<uint32_t*>(smem + G::MISC_OFF);  // [1] bits that vary, [2], [3] largest code
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t n = p.n, nb = p.nb;
    const U* keys = static_cast<const U*>(p.keys_in);
    const V* vals = static_cast<const V*>(p.vals_in);
    W* regions = static_cast<W*>(p.regions);
    const KeyMap<U> map(p.kind, p.desc);
    // ---- the sample, the same in every CTA
    constexpr int PER = 4;
    U x[PER];
    const uint32_t step = max(1u, n / uint32_t(THREADS * PER));
    const U first = map.in(keys[0]);
    U d = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        x[i] = map.in(keys[min(n - 1u, uint32_t(i * THREADS + tid) * step)]);
        d |= x[i] ^ first;
    }
    for (int i = tid; i < G::BINS / 4; i += THREADS) reinterpret_cast<uint32_t*>(smem + G::CTR_OFF)[i] = 0u;
    for (uint32_t i = tid; i < nb; i += THREADS) bins[i] = 0u;
    if (tid < 4) misc[tid] = 0u;
    __syncthreads();
    const uint64_t d64 = msd_top64(d);
    const uint32_t dh = __reduce_or_sync(0xffffffffu, uint32_t(d64 >> 32));
    const uint32_t dl = __reduce_or_sync(0xffffffffu, uint32_t(d64));
    if (lane == 0) {
        atomicOr(&misc[1], dh);
        atomicOr(&misc[2], dl);
    }
    __syncthreads();
    // one leading bit more than the sample's vary: a key a little above them
    // all goes to the last region
    const uint32_t same = misc[1] ? __clz(misc[1]) : misc[2] ? 32u + __clz(misc[2]) : 0u;
    const MsdCode code_of(same ? same - 1u : 0u, 0u);
    uint32_t most = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) most = max(most, code_of(x[i]));
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) atomicMax(&misc[3], most);
    __syncthreads();
    const RegionOf region_of(nb, misc[3]);
    // S keys in regions of g: S * S * g / 2n pairs of them meet in one
    bool off = false;
    {
        uint32_t pairs = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            uint32_t r, frac;
            region_of(code_of(x[i]), r, frac);
            pairs += atomicAdd(&bins[r], 1u);
        }
        pairs = __reduce_add_sync(0xffffffffu, pairs);
        if (lane == 0) atomicAdd(&misc[0], pairs);
        __syncthreads();
        constexpr float SS = float(THREADS * PER) * float(THREADS * PER);
        off = float(misc[0]) * 2.f * float(n) > 1.3f * float(p.cap) * SS;
        __syncthreads();
        for (uint32_t i = tid; i < nb; i += THREADS) bins[i] = 0u;
        if (tid == 0) misc[0] = 0u;
        __syncthreads();
    }
    // ---- partition: equal shares of the array, tiles of at most IPT keys a
    // thread
    const uint32_t share = ((n + gridDim.x - 1) / gridDim.x + 31u) & ~31u;
    const uint32_t from = min(n, blockIdx.x * share), to = off ? from : min(n, from + share);
    for (uint32_t t = from; t < to; t += THREADS * IPT) {
        U k[IPT];
        uint32_t at[IPT];  // region | slot << 16
#pragma unroll
        for (int u = 0; u < IPT; ++u) {
            const uint32_t j = t + u * THREADS + tid;
            k[u] = j < to ? map.in(keys[j]) : U(0);
            if (p.vals_aside && j < to) static_cast<V*>(p.vals_aside)[j] = vals[j];
        }
#pragma unroll
        for (int u = 0; u < IPT; ++u) {
            if (t + u * THREADS + tid < to) {
                uint32_t r, frac;
                region_of(code_of(k[u]), r, frac);
                at[u] = r | atomicAdd(&bins[r], 1u) << 16;
                off |= code_of.skip != 0u && (msd_top64(U(k[u] ^ first)) >> (64u - code_of.skip)) != 0u;
            }
        }
        __syncthreads();
        for (uint32_t r = tid; r < nb; r += THREADS) {
            const uint32_t c = bins[r];
            if (c) {
                const uint32_t g = atomicAdd(p.fill + r, c);
                off |= g + c > p.cap;
                claims[r] = g;
                bins[r] = 0u;
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < IPT; ++u) {
            const uint32_t j = t + u * THREADS + tid;
            if (j < to) {
                const uint32_t r = at[u] & 0xffffu, place = claims[r] + (at[u] >> 16);
                if (place < p.cap) regions[size_t(r) * p.cap + place] = W(k[u]) << (8 * KB) | W(j);
            }
        }
        __syncthreads();
    }
    if (off) atomicOr(p.state, MSD_OFF);
    if (!grid_barrier(p.barrier, p.barrier_gen, 1u, p.wait_limit_ns, p.err)) return;
    if (ld_relaxed(p.state) & MSD_OFF) {
        fused_counts<KB, THREADS>(p.hist, smem, G::SCAN_OFF);
        return;
    }
    // ---- every region's size and first place in the result
    {
        const uint32_t per = (nb + THREADS - 1) / THREADS;  // regions a thread
        constexpr int MOST = (1024 + THREADS - 1) / THREADS;
        uint32_t c[MOST], sum = 0;
#pragma unroll
        for (int i = 0; i < MOST; ++i) {
            c[i] = uint32_t(i) < per && tid * per + i < nb ? ld_relaxed(p.fill + tid * per + i) : 0u;
            sum += c[i];
        }
        uint32_t run = block_exclusive_scan_all<THREADS>(sum, scan);
#pragma unroll
        for (int i = 0; i < MOST; ++i) {
            if (uint32_t(i) < per && tid * per + i < nb) {
                bins[tid * per + i] = run;
                claims[tid * per + i] = c[i];
                run += c[i];
            }
        }
        __syncthreads();
        if (tid < 4) misc[tid] = 0u;
        __syncthreads();
    }
    if (p.vals_aside) vals = static_cast<const V*>(p.vals_aside);
    U* okeys = static_cast<U*>(p.keys_out);
    V* ovals = static_cast<V*>(p.vals_out);
    for (uint32_t b = blockIdx.x; b < nb; b += gridDim.x) {
        const uint32_t cnt = claims[b], off0 = bins[b];
        if (cnt == 0u) continue;
        const W* words = regions + size_t(b) * p.cap;
        W k[LIPT];
        load_vectors<THREADS>(words, 0u, cnt, k);
        const uint32_t pad = uint32_t(reinterpret_cast<uintptr_t>(okeys + off0) & 31u) / uint32_t(KB);
        U* ok = okeys + off0 - pad;
        V* ov = ovals + off0 - pad;
        auto put = [&](uint32_t place, W w) {
            const uint32_t j = uint32_t(w);
            ok[place] = map.out(U(w >> (8 * KB)));
            ov[place] = vals[j < n ? j : 0u];
        };
        const bool sorted = group_sort<W, THREADS, HALO>(
            k, cnt, 0u, pad, smem,
            [&](W w) {
                uint32_t r, frac;
                region_of(code_of(U(w >> (8 * KB))), r, frac);
                return __umulhi(frac, uint32_t(G::BINS));
            },
            [] {},
            [&](uint32_t c0, bool inside, const W(&w)[LIPT]) {
                if (inside) {
                    V v[LIPT];
#pragma unroll
                    for (int i = 0; i < LIPT; ++i) {
                        const uint32_t j = uint32_t(w[i]);
                        v[i] = vals[j < n ? j : 0u];
                    }
                    union { uint4 q[2]; U k[32 / KB]; } y;
                    static_assert(LIPT * KB == 32, "a sector of keys a lane");
#pragma unroll
                    for (int i = 0; i < LIPT; ++i) y.k[i] = map.out(U(w[i] >> (8 * KB)));
                    store_32b(ok + c0, y.q[0], y.q[1]);
#pragma unroll
                    for (int i = 0; i < LIPT; ++i) ov[c0 + i] = v[i];
                } else {
#pragma unroll
                    for (int i = 0; i < LIPT; ++i)
                        if (c0 + i >= pad && c0 + i < pad + cnt) put(c0 + i, w[i]);
                }
            },
            [&](uint32_t place, W w) { put(place, w); });
        if (!sorted) {
            // many equal keys: a bitonic network over the words, padded with
            // the largest one
            W* sw = reinterpret_cast<W*>(smem);
            uint32_t m = 32;
            while (m < cnt) m *= 2;
            __syncthreads();
            for (uint32_t i = tid; i < m; i += THREADS) sw[i] = i < cnt ? words[i] : ~W(0);
            __syncthreads();
            for (uint32_t size = 2; size <= m; size *= 2) {
                for (uint32_t stride = size / 2; stride; stride /= 2) {
                    for (uint32_t i = tid; i < m / 2; i += THREADS) {
                        const uint32_t lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                        const W a = sw[lo], z = sw[hi];
                        if ((z < a) == ((lo & size) == 0u)) {
                            sw[lo] = z;
                            sw[hi] = a;
                        }
                    }
                    __syncthreads();
                }
            }
            for (uint32_t i = tid; i < cnt; i += THREADS) put(pad + i, sw[i]);
            __syncthreads();
            for (int i = tid; i < G::BINS / 4; i += THREADS) reinterpret_cast<uint32_t*>(smem + G::CTR_OFF)[i] = 0u;
            __syncthreads();
        }
        __syncthreads();
    }
}

}  // namespace gbsort
