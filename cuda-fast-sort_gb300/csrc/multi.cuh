// multi.cuh — every digit pass in one launch (sm_103a), for paths that seldom
// need them all, and what such a path leaves over.
//
// A key that repeats very often makes its group too large for a window or a
// local sort, and any other key in the group keeps it from being done already.
// The ranges of such groups, usually a small part, are gathered, sorted by all
// their digits like an array of their own, and go back: they are in order
// among themselves, so the sorted whole is the ranges' sorted keys one after
// another.
#pragma once

#include "onesweep.cuh"

namespace gbsort {

// Sorts the listed ranges of the result (by the whole grid).  Returns the grid
// barriers used when they are more than half of the array, for which there is
// no room, else -1.  Out of line: it keeps the passes' registers.
template <int KB, int VB, class W, int THREADS, int IPT, int LBW>
__device__ __noinline__ int sort_ranges(const PassParams& p, uint8_t* smem) {
    using U = typename KeyBits<KB>::U;
    using V = typename ValBits<VB>::V;
    using G = PassGeom<KB, VB, THREADS, IPT>;
    constexpr uint32_t MOST = RANGES_MOST, FAR = 0xffffffffu;
    constexpr size_t HIST_OFF = size_t(MOST) * 16;  // before the passes: the list, its sorted form, digit counts
    static_assert(HIST_OFF + size_t(KB) * 1024 <= G::SMEM_BYTES, "the list and the counts");
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const RangeList& left = p.left;
    __shared__ PassView view;
    __shared__ uint32_t runs, barriers, moved;  // passes to run, barriers so far; pairs in the ranges
    __shared__ int done, total;
    // ---- the ranges in order, each with the place of its first pair among the gathered
    uint32_t* raw = reinterpret_cast<uint32_t*>(smem);
    uint32_t* begin = raw + 2 * MOST;  // sorted; FAR beyond the last
    uint32_t* place = begin + MOST;
    const uint32_t count = ld_relaxed(left.count);
    auto order_ranges = [&] {
        for (uint32_t i = tid; i < MOST; i += THREADS) {
            raw[2 * i] = i < count ? ld_relaxed(left.ranges + 2 * i) : FAR;
            raw[2 * i + 1] = i < count ? ld_relaxed(left.ranges + 2 * i + 1) : 0u;
            begin[i] = FAR;
            place[i] = FAR;
        }
        if (tid == 0) moved = 0u;
        __syncthreads();
        for (uint32_t i = tid; i < count; i += THREADS) {
            uint32_t rank = 0, before = 0;
            for (uint32_t j = 0; j < count; ++j) {
                const bool b = raw[2 * j] < raw[2 * i];
                rank += b;
                before += b ? raw[2 * j + 1] : 0u;
            }
            begin[rank] = raw[2 * i];
            place[rank] = before;
            if (rank + 1 == count) moved = before + raw[2 * i + 1];
        }
        __syncthreads();
    };
    if (tid == 0) {
        barriers = 0u;
        done = 0;
    }
    auto barrier = [&] {  // (thread 0 counts it)
        if (tid == 0) ++barriers;
        __syncthreads();
        return grid_barrier(p.barrier, p.barrier_gen, barriers, p.wait_limit_ns, p.err);
    };
    order_ranges();
    if (!barrier()) return -1;  // (every CTA has read the list, which the caller may clear)
    const uint32_t m = moved, second = (m + 31u) & ~31u;  // of the alternate buffers: halves
    if (2ull * second > p.n) return 1;
    if (tid == 0) {
        view.n = m;
        view.tiles = uint32_t((view.n + G::TILE - 1) / G::TILE);
    }
    __syncthreads();
    const uint64_t stride = uint64_t(gridDim.x) * THREADS, start = uint64_t(blockIdx.x) * THREADS + tid;
    U* const ka = static_cast<U*>(p.keys_a);
    V* const va = static_cast<V*>(p.vals_a);
    U* const kb = static_cast<U*>(p.keys_b);
    V* const vb = static_cast<V*>(p.vals_b);
    // pair q of the gathered ones lies at begin[i] + q - place[i]
    auto range_of = [&](uint32_t q) {
        uint32_t a = 0, z = count;
        while (z - a > 1u) {
            const uint32_t mid = (a + z) / 2;
            if (place[mid] <= q) a = mid;
            else z = mid;
        }
        return a;
    };
    {  // status words hold an earlier run's; the counts are the whole array's
        const uint64_t words = (uint64_t(view.tiles) * 256 * sizeof(W) + 15) / 16;
        uint4* st = static_cast<uint4*>(p.status);
        for (uint64_t i = start; i < words; i += stride) st[i] = make_uint4(0, 0, 0, 0);
        unsigned long long* gp = const_cast<unsigned long long*>(p.gp_all);
        for (uint64_t i = start; i < uint64_t(p.passes) * 256; i += stride) gp[i] = 0ull;
        if (!barrier()) return -1;
    }
    {  // gather, and count the digits
        uint32_t* counts = reinterpret_cast<uint32_t*>(smem + HIST_OFF);
        for (uint32_t i = tid; i < uint32_t(KB) * 256; i += THREADS) counts[i] = 0u;
        __syncthreads();
        for (uint64_t q0 = start - lane; q0 < m; q0 += stride) {  // (whole warps)
            const uint32_t q = uint32_t(q0) + lane;
            const bool in = q < m;
            const uint32_t r = in ? range_of(q) : 0u, at = in ? begin[r] + (q - place[r]) : 0u;
            U k = U(0);
            if (in) {
                const U x = ka[at];
                kb[q] = x;
                if constexpr (VB > 0) vb[q] = va[at];
                k = left.twiddled ? x : twiddle_in<U>(x, p.kind, p.desc);
            }
            const uint32_t active = __ballot_sync(0xffffffffu, in);
            if (!in) continue;
#pragma unroll 1
            for (int d = 0; d < KB; ++d) {  // equal digits, the usual case, with one addition
                const uint32_t b = digit_of(k, d);
                if (__reduce_min_sync(active, b) == __reduce_max_sync(active, b)) {
                    if (lane == uint32_t(__ffs(active) - 1)) atomicAdd(&counts[d * 256 + b], uint32_t(__popc(active)));
                } else {
                    atomicAdd(&counts[d * 256 + b], 1u);
                }
            }
        }
        __syncthreads();
        unsigned long long* gp = const_cast<unsigned long long*>(p.gp_all);
        for (uint32_t i = tid; i < uint32_t(KB) * 256; i += THREADS)
            if (counts[i]) atomicAdd(gp + i, static_cast<unsigned long long>(counts[i]));
        fence_proxy_async_all();  // (the passes' bulk copies read what was gathered)
        if (!barrier()) return -1;
        fence_proxy_async_all();
    }
    // ---- the digit passes
    if constexpr (!G::HALF && rank_uses_or(IPT)) {
        uint32_t* match_scratch = reinterpret_cast<uint32_t*>(smem + G::MATCH_OFF);
        for (int i = tid; i < G::WARPS * 256; i += THREADS) match_scratch[i] = 0u;
    }
    const uint32_t masked = pass_mask(p, view.n, reinterpret_cast<uint32_t*>(smem + G::SKIP_OFF));
    if (tid == 0) {
        runs = ~masked & ((1u << p.passes) - 1u);
        total = __popc(runs);
    }
    auto next_view = [&] {  // (thread 0) the buffers of the next pass
        const bool odd = (done & 1) != 0;
        view.keys_in = odd ? kb + second : kb;
        view.vals_in = odd ? vb + second : vb;
        view.keys_out = odd ? kb : kb + second;
        view.vals_out = odd ? vb : vb + second;
        view.twiddle_load = done == 0 && !left.twiddled;
        view.twiddle_store = done + 1 == total;
    };
    auto offsets = [&](int pass) {  // the pass's digit offsets
        const unsigned long long c = (tid < 256) ? p.gp_all[size_t(pass) * 256 + tid] : 0ull;
        const unsigned long long ex = block_exclusive_scan_256<unsigned long long>(
            c, reinterpret_cast<unsigned long long*>(smem + G::SCAN64_OFF), nullptr);
        if (tid < 256) reinterpret_cast<unsigned long long*>(smem + G::GEXCL_OFF)[tid] = ex;
    };
    if (tid == 0) next_view();
    __syncthreads();
    if (runs) offsets(__ffs(runs) - 1);
    while (runs) {
        if (!onesweep_pass_body<KB, VB, W, THREADS, IPT, false, LBW, true, true>(p, smem, __ffs(runs) - 1, 0u, true, &view))
            return -1;
        __syncthreads();
        if (tid < 3) mbar_inval(reinterpret_cast<uint64_t*>(smem + G::MBAR_OFF) + tid);
        if (tid == 0) {
            runs &= runs - 1u;
            ++done;
            next_view();
        }
        __syncthreads();
        if (runs) offsets(__ffs(runs) - 1);
        fence_proxy_async_all();  // (the next pass's bulk copies read what the CTAs stored)
        if (!barrier()) return -1;
        fence_proxy_async_all();
    }
    if (total == 0 && !left.twiddled) return -1;  // all equal
    order_ranges();  // back to their ranges
    const U* ks = (total & 1) ? kb + second : kb;
    const V* vs = (total & 1) ? vb + second : vb;
    for (uint64_t q = start; q < m; q += stride) {
        const uint32_t r = range_of(uint32_t(q)), at = begin[r] + (uint32_t(q) - place[r]);
        ka[at] = total == 0 ? twiddle_out<U>(ks[q], p.kind, p.desc) : ks[q];
        if constexpr (VB > 0) va[at] = vs[q];
    }
    return -1;
}

// Digits p.pass .. p.passes - 1 in one cooperative launch, a grid barrier
// between the passes that run, then the parity fix-up.  Used where most passes
// do not run (a launch that exits costs about 2.2 us, a barrier with the next
// pass's start about 2 us more than a launch that overlaps its predecessor's
// end: eight passes of 65537 8-byte keys with three that run 44 against 47 us,
// four that all run 55 against 47).
// LEFT: after a path that may have left ranges to sort.  (Apart from the others:
// the call costs their passes registers, 2 x 10^7 u64 identifiers + u32, whose
// sort is leading passes, 651 against 629 us.)
template <int KB, int VB, class W, int THREADS, int IPT, int MIN_CTAS, int LBW, bool LEFT>
__global__ void __launch_bounds__(THREADS, MIN_CTAS) onesweep_multi_kernel(const __grid_constant__ PassParams p) {
    using G = PassGeom<KB, VB, THREADS, IPT>;
    extern __shared__ __align__(128) uint8_t smem[];
    if constexpr (!G::HALF && rank_uses_or(IPT)) {
        uint32_t* match_scratch = reinterpret_cast<uint32_t*>(smem + G::MATCH_OFF);
        for (int i = threadIdx.x; i < G::WARPS * 256; i += THREADS) match_scratch[i] = 0u;
    }
    grid_launch_dependents();
    grid_dependency_wait();
    uint32_t barriers = 0;
    if (p.msd_state) {
        const uint32_t state = ld_relaxed(p.msd_state) & p.state_mask;
        if (state == 0u) return;  // sorted already
        if constexpr (LEFT) {
            if (state == MSD_RANGES) {
                const int used = sort_ranges<KB, VB, W, THREADS, IPT, LBW>(p, smem);
                if (used < 0) return;
                barriers = uint32_t(used);
                if constexpr (!G::HALF && rank_uses_or(IPT)) {  // (the list lay there)
                    uint32_t* match_scratch = reinterpret_cast<uint32_t*>(smem + G::MATCH_OFF);
                    for (int i = threadIdx.x; i < G::WARPS * 256; i += THREADS) match_scratch[i] = 0u;
                }
            }
        }
    }
    uint32_t left_out = 0;  // digits below the leading ones
    if (p.leading && !(ld_relaxed(p.leading) & MSD_OFF)) left_out = (1u << ld_relaxed(p.leading + 1)) - 1u;
    const uint32_t uniform = left_out | pass_mask(p, p.n, reinterpret_cast<uint32_t*>(smem + G::SKIP_OFF));
    const uint32_t all = (p.passes >= 32) ? 0xffffffffu : ((1u << p.passes) - 1u);
    const int total = __popc(~uniform & all);
    const bool to_b = !p.copy_keys_in && (total & 1) != 0;  // where the last pass leaves the result
    const bool move = left_out == 0u && (p.copy_keys_in ? total == 0 : (total & 1) != p.want_odd);
    auto offsets = [&](int pass) {  // the pass's digit offsets
        const int tid = threadIdx.x;
        const unsigned long long c = (tid < 256) ? p.gp_all[size_t(pass) * 256 + tid] : 0ull;
        const unsigned long long ex = block_exclusive_scan_256<unsigned long long>(
            c, reinterpret_cast<unsigned long long*>(smem + G::SCAN64_OFF), nullptr);
        if (tid < 256) reinterpret_cast<unsigned long long*>(smem + G::GEXCL_OFF)[tid] = ex;
    };
    if (p.clear_bytes) {
        uint4* st = static_cast<uint4*>(p.status);
        for (uint64_t i = uint64_t(blockIdx.x) * THREADS + threadIdx.x; i < p.clear_bytes / 16;
             i += uint64_t(gridDim.x) * THREADS)
            st[i] = make_uint4(0, 0, 0, 0);
        if (!grid_barrier(p.barrier, p.barrier_gen, ++barriers, p.wait_limit_ns, p.err)) return;
    }
    uint32_t runs = ~uniform & all;
    if (runs) offsets(__ffs(runs) - 1);
    while (runs) {
        const int pass = __ffs(runs) - 1;
        runs &= runs - 1u;
        if (!onesweep_pass_body<KB, VB, W, THREADS, IPT, false, LBW, true>(p, smem, pass, uniform, left_out == 0u))
            return;
        if (runs || move) {  // another pass, or the fix-up
            __syncthreads();
            if (threadIdx.x < 3) mbar_inval(reinterpret_cast<uint64_t*>(smem + G::MBAR_OFF) + threadIdx.x);
            if (runs) offsets(__ffs(runs) - 1);
            // the next pass's bulk copies read what the CTAs stored
            fence_proxy_async_all();
            if (!grid_barrier(p.barrier, p.barrier_gen, ++barriers, p.wait_limit_ns, p.err)) return;
            fence_proxy_async_all();
        }
    }
    if (move) {
        const bool copied = p.copy_keys_in != nullptr;
        const void* ks = copied ? p.copy_keys_in : to_b ? p.keys_b : p.keys_a;
        const void* vs = copied ? p.copy_vals_in : to_b ? p.vals_b : p.vals_a;
        const bool to_a = to_b || copied;
        grid_copy_bytes(to_a ? p.keys_a : p.keys_b, ks, p.n * uint64_t(KB));
        if constexpr (VB > 0) grid_copy_bytes(to_a ? p.vals_a : p.vals_b, vs, p.n * uint64_t(VB));
    }
}

}  // namespace gbsort
