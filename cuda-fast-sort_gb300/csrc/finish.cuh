// finish.cuh — sorts by the keys' leading digits only (sm_103a): key-value
// arrays of 8- and 16-byte keys, and 8-byte floats alone, whose leading bits
// are too uneven for the splits of msd.cuh.
//
// A stable least-significant-digit sort makes a pass over keys and values per
// key byte.  Where the leading D bytes already cut the array into groups of a
// few thousand pairs, the passes over the other bytes can be one local sort:
//   sample:  4096 to 16384 keys say how many leading bytes that takes (or that
//            nothing is gained, MSD_OFF: every digit pass runs as before);
//   passes:  the digit passes of those bytes only (onesweep.cuh);
//   edges:   the array, now in stable order of its leading bytes, is cut near
//            every `chunk` pairs at the next group's start, so that windows of
//            whole groups fit a CTA;
//   finish:  each CTA sorts whole windows in shared memory, stable, and
//            writes them untwiddled to the caller's buffers.
// A window's keys keep their order by group; inside a group of m keys a key
// goes to one of m sub-buckets by its remaining bits (about one key each), and
// a few rounds of an odd-even transposition network over (key, place before)
// put it in its stable place.  A group whose keys are all equal keeps its
// order as it is, however large: an edge may cut through such a group.
// What bounds the finish: latency (two CTAs of 384 threads an SM, 80 registers;
// a window of 2300 pairs of 8-byte keys takes its CTA 7.7 us, of which the
// network's instructions are a fifth); 2 x 10^7 u64 + u32 0.22 ms.
// A window whose sub-buckets are too full (keys that repeat inside groups of
// different keys) is put in order by a network over all of it.
// A group of different keys that does not fit a window leaves its windows as
// they were, untwiddled, and their range is sorted by all digits afterwards
// (sort_ranges; pairs in an order that a stable sort completes).
// Where the leading digits do not vary, or those ranges are most of the array,
// every digit pass runs, from the caller's buffers.
#pragma once

#include "msd.cuh"

namespace gbsort {

struct FinishParams {
    const void* keys_in;   // the input (sample only)
    void* keys_a;          // the caller's buffers: the result
    void* vals_a;
    void* keys_b;          // the alternate buffers
    void* vals_b;
    uint64_t n;            // < 2^32
    int kind, desc;
    int copy;              // input-preserving: the passes end in the caller's buffers
    uint32_t* state;       // MSD_OFF, MSD_GAVE_UP: every digit pass sorts; MSD_RANGES: the list is not empty
    uint32_t* window;      // [2] lowest digit that the passes sort by, pairs per chunk
    const uint32_t* executed;  // passes run (bit 31 set; 0: none)
    uint32_t* ticket;      // the sample's CTAs, zeroed with the control block
    uint32_t* sampled;     // [FINISH_LEVELS + 2] their counts, and the keys met twice
    uint32_t* edges;       // [chunks + 1] first pair of every window (bit 31: the edge cuts a group)
    uint32_t* seen;        // [chunks + 1] bit 1: the cut edge has different keys on its sides; bit 0: listed
    uint32_t max_chunks;   // room in edges and seen
    RangeList left;        // ranges that the finish leaves to sort
    uint32_t places;       // pairs a window may hold
    uint32_t* err;
};

// ---- sample -----------------------------------------------------------------
// CTA l counts the pairs of sampled keys that share their l + 1 leading bytes
// (the last CTA: that are equal, which no digit tells apart), exactly, in a
// table of 2^15 slots at most half full: 17 more bits of a prefix's hash above
// its count.  (Counters without them met S * S / 2^16 pairs by chance, and
// their noise hid keys that repeat a hundred times.)  S keys in groups of g
// make S * S * g / 2n pairs.  The places are random: at even distances, keys in
// order came one to a group and groups of any size looked like none (2 x 10^7
// sorted u64 + u32 1.68 ms, by random places 0.60).  The CTA that finishes last
// decides.
constexpr int FINISH_SAMPLE_THREADS = 1024;
constexpr int FINISH_LEVELS = 6;  // leading bytes tried
constexpr int FINISH_SAMPLE_SMEM = 32768 * 4;
template <int KB>
constexpr int finish_levels() { return KB - 1 < FINISH_LEVELS ? KB - 1 : FINISH_LEVELS; }
// Copies of a key from which on its groups have to be of one key (below).
constexpr float FINISH_REPEATS = 12.f;

template <int KB>
__global__ void __launch_bounds__(FINISH_SAMPLE_THREADS, 1) finish_sample_kernel(FinishParams p) {
    using U = typename KeyBits<KB>::U;
    constexpr int LEVELS = finish_levels<KB>();
    extern __shared__ __align__(16) uint32_t cnt[];
    __shared__ uint32_t shared_pairs, vary, ticket, repeats, heavy;
    grid_launch_dependents();
    grid_dependency_wait();
    const int tid = threadIdx.x, level = blockIdx.x;
    // more of them where a group is a smaller part of the array
    constexpr int MOST = KB == 16 ? 8 : 16;
    const int per = p.n >= (uint64_t(1) << 26) ? MOST : p.n >= (uint64_t(1) << 23) ? 8 : 4;
    const float S = float(FINISH_SAMPLE_THREADS * per);
    const KeyMap<U> map(p.kind, p.desc);
    const U* keys = static_cast<const U*>(p.keys_in);
    U x[MOST];
#pragma unroll
    for (int i = 0; i < MOST; ++i) {
        if (i >= per) break;
        uint32_t h = uint32_t(i * FINISH_SAMPLE_THREADS + tid) * 0x9E3779B9u + 0x7F4A7C15u;
        h = (h ^ (h >> 16)) * 0x85EBCA6Bu;  // (murmur3's finalizer)
        h = (h ^ (h >> 13)) * 0xC2B2AE35u;
        h ^= h >> 16;
        x[i] = map.in(keys[(uint64_t(h) * p.n) >> 32]);
    }
    const U first = map.in(keys[0]);
    for (int i = tid; i < 8192; i += FINISH_SAMPLE_THREADS) reinterpret_cast<uint4*>(cnt)[i] = make_uint4(0, 0, 0, 0);
    if (tid == 0) shared_pairs = vary = repeats = heavy = 0u;
    __syncthreads();
    U d = 0;
    uint32_t pairs = 0, again = 0, more = 0;  // again, more: prefixes met for the second time, or oftener
    uint32_t at[MOST];
#pragma unroll
    for (int i = 0; i < MOST; ++i) {
        if (i >= per) break;
        d |= x[i] ^ first;
        const U v = level == LEVELS ? x[i] : x[i] >> (8 * (KB - 1 - level));
        uint64_t h = uint64_t(v);
        if constexpr (KB == 16) h ^= uint64_t(v >> 64) * 0x9E3779B97F4A7C15ull;
        // (splitmix64's finalizer: few distinct prefixes must not spread evenly)
        h = (h ^ (h >> 30)) * 0xBF58476D1CE4E5B9ull;
        h = (h ^ (h >> 27)) * 0x94D049BB133111EBull;
        h ^= h >> 31;
        at[i] = (uint32_t(h >> 32) & 0xffff8000u) | (uint32_t(h) & 32767u);  // tag | slot
    }
    auto meet = [&](uint32_t key, uint32_t w) {  // w: what its slot held at the first look
        const uint32_t tag = key & 0xffff8000u;
        uint32_t slot = key & 32767u;
        for (int probe = 0; probe < 128; ++probe) {
            if (w == 0u) w = atomicCAS(&cnt[slot], 0u, tag | 1u);
            if (w == 0u) break;
            if ((w & 0xffff8000u) == tag) {
                const uint32_t before = atomicAdd(&cnt[slot], 1u) & 32767u;  // the keys there before this one
                pairs += before;
                again += before == 1u;
                more += before > 1u;
                break;
            }
            slot = (slot + 1u) & 32767u;
            w = cnt[slot];
        }
    };
    // (a key a thread first: a prefix that many share then takes one atomic a
    // key; then every other key's first look at once)
    meet(at[0], cnt[at[0] & 32767u]);
    __syncthreads();
    uint32_t there[MOST];
#pragma unroll
    for (int i = 1; i < MOST; ++i) there[i] = i < per ? cnt[at[i] & 32767u] : 0u;
#pragma unroll
    for (int i = 1; i < MOST; ++i) {
        if (i >= per) break;
        meet(at[i], there[i]);
    }
    uint32_t bytes = 0;  // bit q: byte q differs somewhere
#pragma unroll
    for (int q = 0; q < KB; ++q) bytes |= uint32_t(((d >> (8 * q)) & U(0xff)) != U(0)) << q;
    bytes = __reduce_or_sync(0xffffffffu, bytes);
    pairs = __reduce_add_sync(0xffffffffu, pairs);
    again = __reduce_add_sync(0xffffffffu, again);
    more = __reduce_add_sync(0xffffffffu, more);
    if ((tid & 31) == 0) {
        atomicOr(&vary, bytes);
        atomicAdd(&shared_pairs, pairs);
        if (again) atomicAdd(&repeats, again);
        if (more) atomicAdd(&heavy, more);
    }
    __syncthreads();
    if (tid == 0) {
        p.sampled[level] = shared_pairs;
        if (level == LEVELS) p.sampled[LEVELS + 1] = repeats | heavy << 16;
        __threadfence();
        ticket = atomicAdd(p.ticket, 1u);
    }
    if (tid != 0 || ticket != uint32_t(LEVELS)) return;
    __threadfence();
    const float n = float(p.n), places = float(p.places), scale = 2.f * n / (S * S);
    uint32_t sampled[LEVELS + 2];  // (loaded at once: one by one they took half of the kernel)
#pragma unroll
    for (int l = 0; l < LEVELS + 2; ++l) sampled[l] = ld_relaxed(p.sampled + l);
    const float equal = float(sampled[LEVELS]);
    const uint32_t again_more = sampled[LEVELS + 1];
    // Others equal to a key, on average over the keys, every key that repeats
    // counted once (1% of zeros would make an average of thousands).
    const float copies = float(again_more & 0xffffu) * scale;
    const bool repeating = copies >= FINISH_REPEATS;
    // the keys unlike a key in its group by l + 1 leading bytes, on average over
    // the keys that are not of a few very frequent ones, and a little more than
    // half a deviation of the estimate
    const float rest = scale / max(0.05f, 1.f - float(again_more >> 16) / S);
    float group_of[LEVELS];
#pragma unroll
    for (int l = 0; l < LEVELS; ++l) {
        const float pairs = max(0.f, float(sampled[l]) - equal);
        group_of[l] = (pairs + 0.6f * sqrtf(pairs + 2.f)) * rest;
    }
    // The fewest leading bytes whose groups fit, and whose next byte spreads a
    // group's keys over its sub-buckets.  Groups of floats are uneven (the
    // largest of N(0, 1) hold twice the average): they have to be smaller.
    // Where keys repeat, one sub-bucket takes all copies of a key: groups that
    // are one key's keep their order instead, so that few may be of more (2 x
    // 10^7 u64 + u32 in 40 copies 0.90 ms; two bytes fit, but leave every window
    // crowded).
    // 16-byte keys' windows hold half as many: a pass more is cheaper than windows
    // half full (2^25 u128 + u32: three bytes 2.03 ms, two, groups of 512, 2.07).
    const float fits = (p.kind == KIND_FLOAT ? 0.4f : KB == 16 ? 0.36f : 0.84f) * places;
    int lo = 0;
    float group = 0.f, unlike = 0.f;  // unlike: its pairs of different keys
    bool chosen = false;
#pragma unroll
    for (int l = 0; l < LEVELS; ++l) {
        const float g = group_of[l];
        const bool spreads = l + 1 == LEVELS || group_of[l + 1 < LEVELS ? l + 1 : l] <= g * (1.f / 16.f) + 3.f * rest + 4.f;
        if (chosen || g > fits || !spreads) continue;
        group = g;
        unlike = max(0.f, float(sampled[l]) - equal);
        lo = KB - 1 - l;
        // (in less than half of the windows, which hold places / copies such groups)
        chosen = !repeating || unlike * rest * 2.f * places <= copies * copies;
    }
    // worth it when it replaces two passes or more
    const uint32_t low = vary & ((1u << lo) - 1u);
    uint32_t chunk = 0;
    if (lo == 0 || __popc(low) < 2) {
        *p.state = MSD_OFF;
    } else {
        // the larger the groups, the more of a window is left for the one
        // that starts last in it (and seven deviations of a random group's
        // size; where keys repeat and groups are of more than one, two keys' copies)
        const float lumps = repeating && unlike > 0.f ? min(2.2f * copies, 0.25f * places) : 0.f;
        const float c = 0.98f * places - (p.kind == KIND_FLOAT ? 2.f : 1.1f) * group - 7.f * sqrtf(group) - lumps;
        chunk = uint32_t(min(max(c, 0.1f * places), 0.93f * places)) & ~31u;
        chunk = max(chunk, (uint32_t(p.n / (p.max_chunks - 1u)) + 32u) & ~31u);
        if (float(chunk) > 0.95f * places) *p.state = MSD_OFF;
    }
    p.window[0] = uint32_t(lo);
    p.window[1] = chunk;
}

// Where the passes left the pairs: the alternate buffers after an odd count
// in place, else the caller's.
__device__ __forceinline__ bool finish_in_b(const FinishParams& p) {
    const uint32_t w = ld_relaxed(p.executed);
    return !p.copy && (w & 1u) != 0u;
}

// ---- edges ------------------------------------------------------------------
// Edge c: the first group start at or after pair c * chunk, found by a warp in
// three rounds of 32 reads; none within places - chunk pairs: the edge stays
// there and cuts the group, which should consist of equal keys.
template <int KB>
__global__ void __launch_bounds__(256) finish_edges_kernel(FinishParams p) {
    using U = typename KeyBits<KB>::U;
    grid_launch_dependents();
    grid_dependency_wait();
    if (ld_relaxed(p.state) & MSD_OFF) return;
    if (!(ld_relaxed(p.executed) >> 31)) {  // the leading digits do not vary: no pass has run
        if (threadIdx.x == 0 && blockIdx.x == 0) atomicOr(p.state, MSD_GAVE_UP);
        return;
    }
    const U* keys = static_cast<const U*>(finish_in_b(p) ? p.keys_b : p.keys_a);
    const uint32_t n = uint32_t(p.n), lo = ld_relaxed(p.window), chunk = ld_relaxed(p.window + 1);
    const uint32_t chunks = (n + chunk - 1) / chunk;
    const int lane = threadIdx.x & 31;
    const uint32_t shift = 8u * lo;
    for (uint32_t c = (blockIdx.x * 256 + threadIdx.x) >> 5; c <= chunks; c += gridDim.x * 8) {
        if (c == 0 || c == chunks) {
            if (lane == 0) {
                p.edges[c] = c ? n : 0u;
                p.seen[c] = 0u;
            }
            continue;
        }
        const uint32_t at = c * chunk;
        const U before = keys[at - 1];
        const U group = before >> shift;
        // first j in [from, from + 32 * step) with another group than `before`, by steps
        uint32_t from = at, limit = min(at + (p.places - chunk), n - 1u);  // heads looked for in [at, limit]
        uint32_t head = 0xffffffffu;
        if ((keys[at] >> shift) != group) {
            head = at;
        } else {
            // keys[from] is in the group; the answer, if any, is in (from, limit]
            uint32_t span = limit - from;
            while (span) {
                const uint32_t step = (span + 31) / 32;
                const uint32_t j = min(from + (lane + 1) * step, limit);
                const uint32_t past = __ballot_sync(0xffffffffu, (keys[j] >> shift) != group);
                if (!past) break;  // only in the first round: later ones hold the answer
                const int l = __ffs(past) - 1;
                const uint32_t hi = min(from + (l + 1) * step, limit);
                const uint32_t low = from + l * step;  // in the group
                if (hi - low <= 1u) {
                    head = hi;
                    break;
                }
                from = low;
                limit = hi;
                span = hi - low;
            }
        }
        if (lane == 0) {
            bool differ = false;
            if (head != 0xffffffffu) {
                p.edges[c] = head;
            } else if (at + (p.places - chunk) >= n) {
                p.edges[c] = n;  // the last group reaches the end of the array
            } else {
                p.edges[c] = at | 0x80000000u;
                differ = keys[at] != before;
            }
            p.seen[c] = differ ? 2u : 0u;
        }
    }
}

// ---- finish -----------------------------------------------------------------
// Shared memory of a window of up to CAP pairs, LIPT consecutive places (a
// chunk) a lane, HALO lanes of margin at a warp's ends.  Chunks lie 16 bytes
// apart from a multiple of their size, so that eight lanes' 16-byte accesses
// meet all banks.  A pair is put in order by its key and its place before, a
// 16-bit place apart from the key.
// (64-bit words of the sub-bucket, 35 bits below it and the place, with the
// keys fetched at the end: 2 x 10^7 8-byte keys 0.31 against 0.23 ms.)
template <int KB, int VB, int THREADS, int LIPT_, int HALO>
struct FinishGeom {
    static constexpr int LIPT = LIPT_;
    static constexpr int WARPS = THREADS / 32;
    static constexpr int OUT = (32 - 2 * HALO) * LIPT;  // places a warp puts in order
    static constexpr int PLACES = WARPS * OUT;
    static constexpr int ALIGN = 32 / KB;  // places keep the result's position in its 32-byte sector
    static constexpr int CAP = PLACES - ALIGN;
    static_assert(PLACES < 65536, "16-bit places");
    static_assert(LIPT * KB % 32 == 0 && LIPT % 2 == 0 && LIPT <= 16, "whole sectors a lane");
    // sub-buckets, one per place; byte counters scanned by a thread
    static constexpr int PER = (PLACES + THREADS * 4 - 1) / (THREADS * 4) * 4;
    static constexpr int BINS = PER * THREADS;
    static constexpr int STRIDE = LIPT * KB + 16;
    static constexpr size_t POS_OFF = (size_t(PLACES / LIPT) * STRIDE + 127) & ~size_t(127);  // u16
    static constexpr size_t VALS_OFF = (POS_OFF + size_t(PLACES) * 2 + 127) & ~size_t(127);
    static constexpr size_t CTR_OFF = (VALS_OFF + size_t(PLACES) * VB + 127) & ~size_t(127);  // u8 [BINS]
    static constexpr size_t START_OFF = CTR_OFF + BINS;                                       // u16 [BINS]
    static constexpr size_t SCAN_OFF = START_OFF + size_t(BINS) * 2;                          // u32 [32]
    static constexpr size_t MISC_OFF = SCAN_OFF + 128;                                        // u32 [4]
    static constexpr size_t HEADS_OFF = MISC_OFF + 16;                                        // u32 [2][WARPS]
    static constexpr size_t SMEM_BYTES = HEADS_OFF + size_t(WARPS) * 8;
    static_assert(size_t(PLACES) <= POS_OFF, "the groups' marks lie where the keys go later");
    __device__ __forceinline__ static uint32_t at(uint32_t place) {
        return place * uint32_t(KB) + (place / LIPT) * 16u;
    }
};

// A key and its place in the window before (unique, so the order is total).
template <class U>
struct Placed {
    U k;
    uint32_t j;
    __device__ __forceinline__ static Placed make(U key, uint32_t place) { return Placed{key, place}; }
    __device__ __forceinline__ U key() const { return k; }
    __device__ __forceinline__ uint32_t place() const { return j; }
};
// b comes before a: one borrow chain over the words.
__device__ __forceinline__ bool after(const Placed<uint64_t>& a, const Placed<uint64_t>& b) {
    uint32_t r;
    asm("{\n\t.reg .u32 t;\n\tsub.cc.u32 t, %1, %2;\n\tsubc.cc.u32 t, %3, %4;\n\tsubc.cc.u32 t, %5, %6;\n\t"
        "subc.u32 %0, 0, 0;\n\t}"
        : "=r"(r)
        : "r"(b.j), "r"(a.j), "r"(uint32_t(b.k)), "r"(uint32_t(a.k)), "r"(uint32_t(b.k >> 32)),
          "r"(uint32_t(a.k >> 32)));
    return r != 0u;
}
__device__ __forceinline__ bool after(const Placed<u128>& a, const Placed<u128>& b) {
    return b.k < a.k || (b.k == a.k && b.j < a.j);
}
template <class U>
__device__ __forceinline__ void order_pair(Placed<U>& a, Placed<U>& b) {
    const bool sw = after(a, b);
    const Placed<U> lo = sw ? b : a, hi = sw ? a : b;
    a = lo;
    b = hi;
}
template <class U>
__device__ __forceinline__ Placed<U> placed_up1(const Placed<U>& p) {
    return Placed<U>::make(shfl_up1(p.key()), __shfl_up_sync(0xffffffffu, p.place(), 1));
}
template <class U>
__device__ __forceinline__ Placed<U> placed_down1(const Placed<U>& p) {
    return Placed<U>::make(shfl_down1(p.key()), __shfl_down_sync(0xffffffffu, p.place(), 1));
}

template <class U, int LIPT>
__device__ __forceinline__ void placed_rounds(Placed<U> (&k)[LIPT], uint32_t rounds, int lane) {
    for (uint32_t r = 0; r < rounds; r += 2) {
#pragma unroll
        for (int i = 0; i + 1 < LIPT; i += 2) order_pair(k[i], k[i + 1]);
        if (r + 1 < rounds) {
            const Placed<U> before = placed_up1(k[LIPT - 1]), next = placed_down1(k[0]);
#pragma unroll
            for (int i = 1; i + 1 < LIPT; i += 2) order_pair(k[i], k[i + 1]);
            if (lane > 0 && after(before, k[0])) k[0] = before;
            if (lane < 31 && after(k[LIPT - 1], next)) k[LIPT - 1] = next;
        }
    }
}

// Global to shared memory without registers in between (4, 8 or 16 bytes,
// aligned to their size); waited for by the thread that issued it.
template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src) {
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Exclusive places of the sub-buckets from their byte counters (zeroed), the
// first at `base`; misc[0] takes the largest count, or 256 when one passed 255
// (the counts then do not add up to cnt).
template <class F, int THREADS>
__device__ __forceinline__ void scan_bins(uint8_t* smem, uint32_t cnt, uint32_t base) {
    constexpr int WORDS = F::PER / 4;
    static_assert(WORDS == 1 || WORDS == 2 || WORDS == 4, "whole vectors");
    uint32_t* ctr = reinterpret_cast<uint32_t*>(smem + F::CTR_OFF) + threadIdx.x * WORDS;
    uint32_t* misc = reinterpret_cast<uint32_t*>(smem + F::MISC_OFF);
    uint32_t c[WORDS], big = 0, sum = 0;
    if constexpr (WORDS == 4) {
        const uint4 q = *reinterpret_cast<const uint4*>(ctr);
        c[0] = q.x, c[1] = q.y, c[2] = q.z, c[3] = q.w;
        *reinterpret_cast<uint4*>(ctr) = make_uint4(0u, 0u, 0u, 0u);
    } else if constexpr (WORDS == 2) {
        const uint2 q = *reinterpret_cast<const uint2*>(ctr);
        c[0] = q.x, c[1] = q.y;
        *reinterpret_cast<uint2*>(ctr) = make_uint2(0u, 0u);
    } else {
        c[0] = *ctr;
        *ctr = 0u;
    }
#pragma unroll
    for (int i = 0; i < WORDS; ++i) {
        big = __vmaxu4(big, c[i]);
        sum = __dp4a(c[i], 0x01010101u, sum);
    }
    big = max(max(big & 0xffu, (big >> 8) & 0xffu), max((big >> 16) & 0xffu, big >> 24));
    big = __reduce_max_sync(0xffffffffu, big);
    if ((threadIdx.x & 31) == 0 && big > 1u) atomicMax(&misc[0], big);
    uint32_t run = block_exclusive_scan_1b<THREADS>(sum, reinterpret_cast<uint32_t*>(smem + F::SCAN_OFF));
    if (threadIdx.x == THREADS - 1 && run + sum != cnt) atomicMax(&misc[0], 256u);
    run += base;
    uint32_t v[2 * WORDS];
#pragma unroll
    for (int i = 0; i < WORDS; ++i) {
        const uint32_t b = run + (c[i] & 0xffu), d = b + ((c[i] >> 8) & 0xffu), e = d + ((c[i] >> 16) & 0xffu);
        v[2 * i] = run | b << 16;
        v[2 * i + 1] = d | e << 16;
        run = e + (c[i] >> 24);
    }
    uint32_t* start = reinterpret_cast<uint32_t*>(smem + F::START_OFF) + threadIdx.x * 2 * WORDS;
    if constexpr (WORDS == 1) {
        *reinterpret_cast<uint2*>(start) = make_uint2(v[0], v[1]);
    } else {
#pragma unroll
        for (int i = 0; i < WORDS / 2; ++i)
            reinterpret_cast<uint4*>(start)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
}

// Lists the windows that consecutive cut edges join, edge c one of them, once
// (a warp; more than FINISH_FAR windows: the whole sort gives up).
constexpr uint32_t FINISH_FAR = 16384;
template <int KB>  // (one instance per key width's translation unit)
__device__ __noinline__ void finish_list(const FinishParams& p, uint32_t c) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t first = c, last = c, steps = 0;
    for (bool found = false; !found && steps < FINISH_FAR / 32; ++steps) {  // (edge 0 is whole)
        const bool whole = lane < first && !(p.edges[first - 1u - lane] >> 31);
        const uint32_t b = __ballot_sync(0xffffffffu, whole || lane >= first);
        found = b != 0u;
        first -= found ? uint32_t(__ffs(b)) : 32u;
    }
    for (bool found = false; !found && steps < 2 * (FINISH_FAR / 32); ++steps) {  // (so is the last one)
        const bool whole = !(p.edges[last + 1u + lane] >> 31);
        const uint32_t b = __ballot_sync(0xffffffffu, whole);
        found = b != 0u;
        last += found ? uint32_t(__ffs(b)) : 32u;
    }
    if (lane != 0) return;
    const uint32_t begin = p.edges[first], end = p.edges[last];
    if ((begin | end) >> 31) {  // not found so near
        atomicOr(p.state, MSD_GAVE_UP);
        return;
    }
    if (atomicOr(p.seen + first, 1u) & 1u) return;
    const uint32_t i = atomicAdd(p.left.count, 1u);
    if (i < p.left.most) {
        p.left.ranges[2 * i] = begin;
        p.left.ranges[2 * i + 1] = end - begin;
    }
    atomicOr(p.state, i < p.left.most ? MSD_RANGES : MSD_GAVE_UP);
}

// A window whose keys and places are in shared memory as they came, places
// [pad, end), put in order by key and place: group by group (they are in order
// already), a warp each, groups beyond FINISH_BY_WARP by the whole CTA.  Out of
// line: it keeps the usual window's registers.
constexpr uint32_t FINISH_BY_WARP = 256;
template <int KB, int VB, int THREADS, int LIPT, int HALO>
__device__ __noinline__ void finish_crowded(uint8_t* smem, uint32_t pad, uint32_t end, uint32_t gshift,
                                            typename KeyBits<KB>::U* okeys, typename ValBits<VB>::V* ovals, int kind,
                                            int desc) {
    using U = typename KeyBits<KB>::U;
    using V = typename ValBits<VB>::V;
    using F = FinishGeom<KB, VB, THREADS, LIPT, HALO>;
    constexpr uint32_t WARPS = THREADS / 32, BIG = F::PLACES / FINISH_BY_WARP + 1;
    uint16_t* sp = reinterpret_cast<uint16_t*>(smem + F::POS_OFF);
    uint32_t* misc = reinterpret_cast<uint32_t*>(smem + F::MISC_OFF);    // [1] groups left to the CTA
    uint32_t* big = reinterpret_cast<uint32_t*>(smem + F::HEADS_OFF);    // their first places and ends
    static_assert(BIG <= 2 * WARPS, "the list of groups");
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto key = [&](uint32_t place) -> U& { return *reinterpret_cast<U*>(smem + F::at(place)); };
    auto group = [&](uint32_t place) { return key(place) >> gshift; };
    auto order = [&](uint32_t a, uint32_t b) {
        U& ka = key(a);
        U& kb = key(b);
        const U x = ka, y = kb;
        const uint16_t i = sp[a], j = sp[b];
        if (y < x || (y == x && j < i)) {
            ka = y;
            kb = x;
            sp[a] = j;
            sp[b] = i;
        }
    };
    if (threadIdx.x == 0) misc[1] = 0u;
    __syncthreads();
    const uint32_t share = (end - pad + WARPS - 1) / WARPS;
    const uint32_t from = pad + warp * share, to = min(from + share, end);
    for (uint32_t i0 = from; i0 < to; i0 += 32) {
        const uint32_t i = i0 + lane;
        uint32_t heads = __ballot_sync(0xffffffffu, i < to && (i == pad || group(i) != group(i - 1)));
        while (heads) {
            const uint32_t first = i0 + __ffs(heads) - 1;
            heads &= heads - 1u;
            // its end, and whether it is in order as it came
            uint32_t last = first + 1;
            bool ordered = true;
            for (;; last += 32) {
                const uint32_t q = last + lane;
                const bool in = q < end && group(q) == group(first);
                const uint32_t out = __ballot_sync(0xffffffffu, !in);
                ordered = __all_sync(0xffffffffu, !in || key(q) >= key(q - 1)) && ordered;
                if (out) {
                    last += __ffs(out) - 1;
                    break;
                }
            }
            if (ordered) continue;
            if (last - first > FINISH_BY_WARP) {
                if (lane == 0) big[atomicAdd(&misc[1], 1u)] = first | last << 16;
            } else {
                ascending_network(
                    last - first, lane, 32u, [&](uint32_t a, uint32_t b) { order(first + a, first + b); },
                    [] { __syncwarp(); });
            }
        }
    }
    __syncthreads();
    const uint32_t left = misc[1];
    for (uint32_t g = 0; g < left; ++g) {
        const uint32_t first = big[g] & 0xffffu, last = big[g] >> 16;
        ascending_network(
            last - first, threadIdx.x, THREADS, [&](uint32_t a, uint32_t b) { order(first + a, first + b); },
            [] { __syncthreads(); });
    }
    const KeyMap<U> map(kind, desc);
    const V* sv = reinterpret_cast<const V*>(smem + F::VALS_OFF);
    for (uint32_t i = pad + threadIdx.x; i < end; i += THREADS) {
        okeys[i] = map.out(key(i));
        if constexpr (VB > 0) ovals[i] = sv[sp[i]];
    }
}

template <int KB, int VB, int THREADS, int MIN_CTAS, int LIPT, int HALO>
__global__ void __launch_bounds__(THREADS, MIN_CTAS) finish_kernel(FinishParams p) {
    using U = typename KeyBits<KB>::U;
    using V = typename ValBits<VB>::V;
    using F = FinishGeom<KB, VB, THREADS, LIPT, HALO>;
    using E = Placed<U>;
    constexpr int WARPS = THREADS / 32, VEC = 16 / KB;
    extern __shared__ __align__(128) uint8_t smem[];
    uint32_t* ctr = reinterpret_cast<uint32_t*>(smem + F::CTR_OFF);
    uint16_t* start = reinterpret_cast<uint16_t*>(smem + F::START_OFF);
    uint32_t* misc = reinterpret_cast<uint32_t*>(smem + F::MISC_OFF);  // [0] largest sub-bucket
    uint32_t* heads_last = reinterpret_cast<uint32_t*>(smem + F::HEADS_OFF);
    uint32_t* heads_first = heads_last + WARPS;
    V* sv = reinterpret_cast<V*>(smem + F::VALS_OFF);
    uint8_t* uneven = smem;  // by a group's first place: its keys differ (before the keys are placed)
    uint16_t* sp = reinterpret_cast<uint16_t*>(smem + F::POS_OFF);
    auto put = [&](uint32_t place, U key, uint32_t before) {
        *reinterpret_cast<U*>(smem + F::at(place)) = key;
        sp[place] = uint16_t(before);
    };
    auto get = [&](uint32_t place) { return E::make(*reinterpret_cast<const U*>(smem + F::at(place)), sp[place]); };
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt = lanemask_lt();
    grid_launch_dependents();
    for (int i = tid; i < F::BINS / 4; i += THREADS) ctr[i] = 0u;
    if (tid == 0) misc[0] = 0u;
    grid_dependency_wait();
    if ((ld_relaxed(p.state) & MSD_OFF) || !(ld_relaxed(p.executed) >> 31)) return;
    const bool in_b = finish_in_b(p);
    const U* keys = static_cast<const U*>(in_b ? p.keys_b : p.keys_a);
    const V* vals = static_cast<const V*>(in_b ? p.vals_b : p.vals_a);
    U* okeys = static_cast<U*>(p.keys_a);
    V* ovals = static_cast<V*>(p.vals_a);
    const uint32_t n = uint32_t(p.n), lo = ld_relaxed(p.window), chunk = ld_relaxed(p.window + 1);
    const uint32_t chunks = (n + chunk - 1) / chunk, gshift = 8u * lo;
    const KeyMap<U> map(p.kind, p.desc);
    const U group_bits = U(~U(0)) << gshift;

    // The CTA's windows are blockIdx.x, + gridDim.x, ...; lane l holds the
    // edges of the l-th of the next 32, and those that are not empty (where
    // groups are larger than a chunk many are) come one by one.
    uint32_t batch = blockIdx.x, b0 = 0, b1 = 0, left = 0;
    uint32_t e0 = 0, e1 = 0;
    auto advance = [&] {  // the next window; false: none left
        while (left == 0u) {
            if (batch >= chunks) return false;
            const uint64_t c = uint64_t(batch) + uint64_t(lane) * gridDim.x;
            b0 = c < chunks ? p.edges[c] : 0u;
            b1 = c < chunks ? p.edges[c + 1] : 0u;
            left = __ballot_sync(0xffffffffu, ((b0 ^ b1) & 0x7fffffffu) != 0u);
            batch = uint64_t(batch) + 32ull * gridDim.x < chunks ? batch + 32u * gridDim.x : chunks;
        }
        const int l = __ffs(left) - 1;
        left &= left - 1u;
        e0 = __shfl_sync(0xffffffffu, b0, l);
        e1 = __shfl_sync(0xffffffffu, b1, l);
        return true;
    };
    // place q of a window: the pair at s - pad + q; pad puts the lanes' chunks
    // on 32-byte boundaries of the result
    const uint32_t c0 = uint32_t(tid) * LIPT;
    U k[LIPT];
    auto pad_of = [&](uint32_t at) { return uint32_t(reinterpret_cast<uintptr_t>(okeys + at) & 31u) / uint32_t(KB); };
    auto load = [&] {  // the window's keys, a chunk a thread
        const uint32_t at = e0 & 0x7fffffffu, pad = pad_of(at), end = pad + (e1 & 0x7fffffffu) - at;
        const U* kp = keys + at - pad + c0;
        if (c0 >= pad && c0 + LIPT <= end && (reinterpret_cast<uintptr_t>(kp) & 15u) == 0u) {
#pragma unroll
            for (int i = 0; i < LIPT / VEC; ++i) {
                union { uint4 q; U x[VEC]; } w;
                w.q = reinterpret_cast<const uint4*>(kp)[i];
#pragma unroll
                for (int e = 0; e < VEC; ++e) k[i * VEC + e] = w.x[e];
            }
        } else {
#pragma unroll
            for (int i = 0; i < LIPT; ++i) k[i] = (c0 + i >= pad && c0 + i < end) ? kp[i] : U(0);
        }
    };
    bool more = advance();
    if (more) load();
    __syncthreads();
    while (more) {
        const uint32_t w0 = e0, w1 = e1;
        const uint32_t s = w0 & 0x7fffffffu, cnt = (w1 & 0x7fffffffu) - s;
        if (cnt > uint32_t(F::CAP)) {  // (the edges keep cnt <= CAP)
            if (tid == 0) atomicOr(p.err, ERRBIT_BOUNDS);
            more = advance();
            if (more) load();
            continue;
        }
        const uint32_t pad = pad_of(s), end = pad + cnt;
        const U* kp = keys + s - pad;
        const bool some = c0 < end && c0 + LIPT > pad;
        const uint32_t i0 = some && c0 < pad ? pad - c0 : 0u, i1 = some ? min(end - c0, uint32_t(LIPT)) : 0u;
        // ---- group heads: the last one at or before, the first one after
        U prev = shfl_up1(k[LIPT - 1]);
        if (lane == 0 && some && c0 > pad) prev = kp[c0 - 1];
        const bool whole = i0 == 0u && i1 == uint32_t(LIPT) && c0 != pad;  // every key has one before it
        const bool all_whole = __all_sync(0xffffffffu, whole);
        const bool busy = warp * 32 * LIPT < int(end);  // the warp has keys of the window
        uint32_t heads = 0;  // bit i: key i starts a group
        if (busy)
#pragma unroll
        for (int i = 0; i < LIPT; ++i)
            if (((k[i] ^ (i ? k[i ? i - 1 : 0] : prev)) & group_bits) != U(0)) heads |= 1u << i;
        const uint32_t valid = (1u << i1) - (1u << i0);  // bit i: key i is one of the window
        if (!all_whole) {
            heads &= valid;
            if (some && c0 <= pad) heads |= 1u << (pad - c0);
        }
        const uint32_t last = heads ? c0 + 31u - __clz(heads) : 0u;
        const uint32_t firsth = heads ? c0 + __ffs(heads) - 1u : end;
        const uint32_t with = __ballot_sync(0xffffffffu, heads != 0u);  // lanes with a head
        const uint32_t under = with & lt, over = with & ~lt & ~(1u << lane);
        uint32_t gs = __shfl_sync(0xffffffffu, last, under ? 31 - __clz(under) : 0);
        uint32_t next = __shfl_sync(0xffffffffu, firsth, over ? __ffs(over) - 1 : 0);
        if (lane == (with ? 31 - __clz(with) : 0)) heads_last[warp] = last;
        if (lane == (with ? __ffs(with) - 1 : 0)) heads_first[warp] = firsth;
        __syncthreads();
        // the values arrive while the keys are sorted
        if constexpr (VB == 0) {
        } else if ((reinterpret_cast<uintptr_t>(vals + s - pad) & 15u) == 0u) {
            constexpr uint32_t VVEC = 16 / (VB ? VB : 1);
            for (uint32_t j = tid * VVEC; j < end; j += THREADS * VVEC) {
                if (j >= pad && j + VVEC <= end) copy_async<16>(sv + j, vals + s - pad + j);
                else
                    for (uint32_t e = j; e < j + VVEC; ++e)
                        if (e >= pad && e < end) copy_async<(VB ? VB : 4)>(sv + e, vals + s - pad + e);
            }
        } else {
            for (uint32_t j = pad + tid; j < end; j += THREADS) copy_async<(VB ? VB : 4)>(sv + j, vals + s - pad + j);
        }
        {
            const uint32_t l = __reduce_max_sync(0xffffffffu, lane < warp ? heads_last[lane] : 0u);
            const uint32_t f = __reduce_min_sync(0xffffffffu, lane > warp && lane < WARPS ? heads_first[lane] : end);
            gs = under ? gs : l;
            next = over ? next : f;
        }
        // ---- count: sub-bucket and slot of every key.  First without looking
        // whether groups consist of equal keys; when a sub-bucket then holds
        // too many (or an edge cuts a group), again with that known: such a
        // group's keys keep their places.
        uint32_t where[LIPT];  // sub-bucket | slot << 16
        // a key's bits below its group's, left-aligned in 32
        auto below = [&](U x) { return uint32_t((x << (8u * KB - gshift)) >> (8 * KB - 32)); };
        auto take = [&](int i, uint32_t b) {
            const uint32_t old = atomicAdd(reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(ctr) + (b & ~3u)),
                                           __funnelshift_l(1u, 1u, b * 8u));
            where[i] = __byte_perm(b, __funnelshift_r(old, old, b * 8u), 0x5410) & 0xffffffu;
        };
        bool marked = ((w0 | w1) >> 31) != 0u, cut = false;
        uint32_t most;
        const bool all_few = __all_sync(0xffffffffu, (heads & (heads - 1u)) == 0u);  // a lane's keys: two groups at most
        for (;;) {
            if (marked) {
                for (int i = tid; i < F::PLACES / 4; i += THREADS) reinterpret_cast<uint32_t*>(uneven)[i] = 0u;
                __syncthreads();
                uint32_t g = gs;
#pragma unroll
                for (int i = 0; i < LIPT; ++i) {
                    if ((heads >> i) & 1u) g = c0 + i;
                    else if (((valid >> i) & 1u) && k[i] != (i ? k[i ? i - 1 : 0] : prev)) uneven[g] = 1;
                }
                __syncthreads();
                // an edge through a group of different keys: nothing this window can do
                if ((w0 >> 31) && (uneven[pad] || (ld_relaxed(p.seen + s / chunk) & 2u))) cut = true;
                if (w1 >> 31) {  // the window's last group
                    uint32_t last_group = 0;
#pragma unroll
                    for (int q = 0; q < WARPS; ++q) last_group = max(last_group, heads_last[q]);
                    if (uneven[last_group]) cut = true;
                }
            }
            if (all_whole && all_few && !marked) {
                const int h = heads ? __ffs(heads) - 1 : LIPT;
                const uint32_t g1 = c0 + h, m0 = (heads ? g1 : next) - gs, m1 = next - g1;
#pragma unroll
                for (int i = 0; i < LIPT; ++i) take(i, (i < h ? gs : g1) + __umulhi(below(k[i]), i < h ? m0 : m1));
            } else if (busy) {
                uint32_t g = gs;
#pragma unroll
                for (int i = 0; i < LIPT; ++i) {
                    if ((heads >> i) & 1u) g = c0 + i;
                    const uint32_t rest = heads & ~((2u << i) - 1u);  // the heads after this key
                    const uint32_t m = (rest ? c0 + __ffs(rest) - 1u : next) - g;
                    if ((valid >> i) & 1u) take(i, marked && !uneven[g] ? c0 + i : g + __umulhi(below(k[i]), m));
                }
            }
            __syncthreads();
            scan_bins<F, THREADS>(smem, cnt, pad);
            __syncthreads();
            most = misc[0];
            if (marked || most <= uint32_t(HALO * LIPT)) break;
            marked = true;
            __syncthreads();
            if (tid == 0) misc[0] = 0u;
        }
        if (cut) {
            // as it was, untwiddled (keys are in registers, values in shared memory)
#pragma unroll
            for (int i = 0; i < LIPT; ++i)
                if ((valid >> i) & 1u) okeys[s - pad + c0 + i] = map.out(k[i]);
            if constexpr (VB > 0) {
                copy_async_wait();
                __syncthreads();
                for (uint32_t j = tid; j < cnt; j += THREADS) ovals[s + j] = sv[pad + j];
            }
            __syncthreads();
            if (tid == 0) misc[0] = 0u;
            if (warp == 0) finish_list<KB>(p, (w0 >> 31 ? w0 & 0x7fffffffu : w1 & 0x7fffffffu) / chunk);  // (cut edges lie at c * chunk)
            more = advance();
            if (more) load();
            __syncthreads();
            continue;
        }
        auto move = [&](int i) { put(uint32_t(start[where[i] & 0xffffu]) + (where[i] >> 16), k[i], c0 + i); };
        if (most > MSD_RANK_MAX) {  // (the slots of a count beyond 255 mean nothing)
#pragma unroll
            for (int i = 0; i < LIPT; ++i)
                if ((valid >> i) & 1u) put(c0 + i, k[i], c0 + i);
        } else if (all_whole) {
#pragma unroll
            for (int i = 0; i < LIPT; ++i) move(i);
        } else if (busy) {
#pragma unroll
            for (int i = 0; i < LIPT; ++i)
                if ((valid >> i) & 1u) move(i);
        }
        if constexpr (VB > 0) copy_async_wait();
        __syncthreads();
        if (tid == 0) misc[0] = 0u;
        if (most > MSD_RANK_MAX)
            finish_crowded<KB, VB, THREADS, LIPT, HALO>(smem, pad, end, gshift, okeys + s - pad, ovals + s - pad, p.kind,
                                                        p.desc);
        more = advance();
        if (more) load();  // the next window's keys, while this one's are put in order
        if (most <= uint32_t(HALO * LIPT)) {
            // chunks [warp * (32 - 2 HALO), ...) and the neighbours' beyond both ends
            const int ch = warp * (32 - 2 * HALO) + lane - HALO;
            const int d0 = ch * LIPT;
            if (warp * F::OUT < int(end)) {
                E x[LIPT];
                const bool inside = d0 >= int(pad) && uint32_t(d0 + LIPT) <= end;
                const E least = E::make(U(0), 0u), greatest = E::make(U(~U(0)), 0xffffu);
                if (d0 + LIPT <= int(pad) || d0 >= int(end)) {
#pragma unroll
                    for (int i = 0; i < LIPT; ++i) x[i] = d0 < int(pad) ? least : greatest;
                } else {
                    const uint4* q = reinterpret_cast<const uint4*>(smem + uint32_t(ch) * F::STRIDE);
                    const uint32_t* pj = reinterpret_cast<const uint32_t*>(sp + d0);
#pragma unroll
                    for (int i = 0; i < LIPT / VEC; ++i) {
                        union { uint4 v; U k[VEC]; } w;
                        w.v = q[i];
#pragma unroll
                        for (int e = 0; e < VEC; ++e) {
                            const int u = i * VEC + e;
                            const uint32_t jj = pj[u / 2];
                            x[u] = E::make(w.k[e], u & 1 ? jj >> 16 : jj & 0xffffu);
                        }
                    }
                    if (!inside) {
#pragma unroll
                        for (int i = 0; i < LIPT; ++i) {
                            if (d0 + i < int(pad)) x[i] = least;
                            if (d0 + i >= int(end)) x[i] = greatest;
                        }
                    }
                }
                if (most > 1u) placed_rounds<U, LIPT>(x, most, lane);
                if (lane >= HALO && lane < 32 - HALO && d0 < int(end)) {
                    U* ok = okeys + s - pad + d0;
                    V* ov = ovals + s - pad + d0;
                    if (inside) {
#pragma unroll
                        for (int i = 0; i < LIPT * KB / 32; ++i) {
                            union { uint4 q[2]; U k[32 / KB]; } y;
#pragma unroll
                            for (int e = 0; e < 32 / KB; ++e) y.k[e] = map.out(x[i * (32 / KB) + e].key());
                            store_32b(ok + i * (32 / KB), y.q[0], y.q[1]);
                        }
                        constexpr int VV = 16 / (VB ? VB : 16);
                        if constexpr (VB == 0) {
                        } else if ((reinterpret_cast<uintptr_t>(ov) & 15u) == 0u) {
#pragma unroll
                            for (int i = 0; i < LIPT / VV; ++i) {
                                union { uint4 q; V v[VV]; } y;
#pragma unroll
                                for (int e = 0; e < VV; ++e) y.v[e] = sv[x[i * VV + e].place()];
                                reinterpret_cast<uint4*>(ov)[i] = y.q;
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < LIPT; ++i) ov[i] = sv[x[i].place()];
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < LIPT; ++i) {
                            if (d0 + i >= int(pad) && d0 + i < int(end)) {
                                ok[i] = map.out(x[i].key());
                                if constexpr (VB > 0) ov[i] = sv[x[i].place()];
                            }
                        }
                    }
                }
            }
        } else if (most <= MSD_RANK_MAX) {
            // a pair's place is its sub-bucket's start plus the sub-bucket's
            // other pairs before it; the sub-bucket of a place: the last one
            // that starts at or before it and is not empty
            for (uint32_t i = pad + tid; i < end; i += THREADS) {
                uint32_t a = 0, z = F::BINS;
                while (z - a > 1u) {
                    const uint32_t mid = (a + z) / 2;
                    if (start[mid] <= i) a = mid;
                    else z = mid;
                }
                const uint32_t q0 = start[a], q1 = a + 1 < uint32_t(F::BINS) ? uint32_t(start[a + 1]) : end;
                const E me = get(i);
                uint32_t before = 0;
                for (uint32_t q = q0; q < q1; ++q) before += after(me, get(q));
                okeys[s - pad + q0 + before] = map.out(me.key());
                if constexpr (VB > 0) ovals[s - pad + q0 + before] = sv[me.place()];
            }
        }
    }
}

}  // namespace gbsort
