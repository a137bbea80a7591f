// repair.cuh — what a sort by leading digits (finish.cuh) leaves over (sm_103a).
//
// A key that fills more than a window makes its group impossible to finish
// when the group holds another key too.  The pairs of such groups' windows,
// usually a small part, are gathered, sorted by all their digits like an array
// of their own, and go back: the ranges are in order among themselves, so the
// sorted whole is the ranges' sorted pairs one after another.  One cooperative
// launch; when the ranges are more than half of the array, every digit pass runs
// over all of it instead.
#pragma once

#include "finish.cuh"
#include "onesweep.cuh"

namespace gbsort {

template <int KB, int VB, class W, int THREADS, int IPT, int MIN_CTAS, int LBW>
__global__ void __launch_bounds__(THREADS, MIN_CTAS) finish_repair_kernel(PassParams p, RangeList left) {
    using U = typename KeyBits<KB>::U;
    using V = typename ValBits<VB>::V;
    using G = PassGeom<KB, VB, THREADS, IPT>;
    constexpr uint32_t MOST = RANGES_MOST, FAR = 0xffffffffu;
    constexpr size_t HIST_OFF = size_t(MOST) * 16;  // before the passes: the list, its sorted form, digit counts
    static_assert(HIST_OFF + size_t(KB) * 1024 <= G::SMEM_BYTES, "the list and the counts");
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    grid_launch_dependents();
    grid_dependency_wait();
    const uint32_t state = ld_relaxed(p.msd_state);
    if ((state & MSD_OFF) || !(state & (MSD_GAVE_UP | MSD_RANGES))) return;  // sorted already
    __shared__ PassView view;
    __shared__ uint32_t runs, barriers, moved;  // passes to run, barriers so far; pairs in the ranges
    __shared__ int done, total, move;
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
    const bool listed = !(state & MSD_GAVE_UP) && count <= left.most;
    if (listed) {
        order_ranges();
        if (!barrier()) return;  // (every CTA has read the list, which may be cleared below)
    }
    const uint32_t m = listed ? moved : 0u, second = (m + 31u) & ~31u;  // of the alternate buffers: halves
    const bool some = listed && 2ull * second <= p.n;
    if (tid == 0) {
        view.n = some ? m : p.n;
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
        const uint64_t words = some ? (uint64_t(view.tiles) * 256 * sizeof(W) + 15) / 16 : p.clear_bytes / 16;
        uint4* st = static_cast<uint4*>(p.status);
        for (uint64_t i = start; i < words; i += stride) st[i] = make_uint4(0, 0, 0, 0);
        unsigned long long* gp = const_cast<unsigned long long*>(p.gp_all);
        if (some)
            for (uint64_t i = start; i < uint64_t(p.passes) * 256; i += stride) gp[i] = 0ull;
        if (!barrier()) return;
    }
    if (some) {  // gather, and count the digits
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
                k = twiddle_in<U>(x, p.kind, p.desc);
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
        if (!barrier()) return;
        fence_proxy_async_all();
    }
    // ---- the digit passes
    if constexpr (!G::HALF && rank_uses_or(IPT)) {
        uint32_t* match_scratch = reinterpret_cast<uint32_t*>(smem + G::MATCH_OFF);
        for (int i = tid; i < G::WARPS * 256; i += THREADS) match_scratch[i] = 0u;
    }
    const uint32_t masked = pass_mask(p, view.n, reinterpret_cast<uint32_t*>(smem + G::SKIP_OFF));
    const bool copied = !some && p.copy_keys_in != nullptr;
    if (tid == 0) {
        runs = ~masked & ((1u << p.passes) - 1u);
        total = __popc(runs);
        move = some ? total != 0 : copied ? total == 0 : (total & 1) != p.want_odd;
    }
    auto next_view = [&] {  // (thread 0) the buffers of the next pass
        // ranges: between the alternate buffers' halves; all: as every sort
        const bool out_b = copied ? ((total - 1 - done) & 1) != 0 : (done & 1) == 0, in_b = !out_b;
        U* const k0 = some ? kb : ka;
        U* const k1 = some ? kb + second : kb;
        V* const v0 = some ? vb : va;
        V* const v1 = some ? vb + second : vb;
        view.keys_in = copied && done == 0 ? p.copy_keys_in : in_b ? k1 : k0;
        view.vals_in = copied && done == 0 ? p.copy_vals_in : in_b ? v1 : v0;
        view.keys_out = out_b ? k1 : k0;
        view.vals_out = out_b ? v1 : v0;
        view.twiddle_load = done == 0;
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
            return;
        __syncthreads();
        if (tid < 3) mbar_inval(reinterpret_cast<uint64_t*>(smem + G::MBAR_OFF) + tid);
        if (tid == 0) {
            runs &= runs - 1u;
            ++done;
            next_view();
        }
        __syncthreads();
        if (!runs && !move) return;
        if (runs) offsets(__ffs(runs) - 1);
        fence_proxy_async_all();  // (the next pass's bulk copies read what the CTAs stored)
        if (!barrier()) return;
        fence_proxy_async_all();
    }
    if (!move) return;
    if (some) {  // back to their ranges
        order_ranges();
        const U* ks = (total & 1) ? kb + second : kb;
        const V* vs = (total & 1) ? vb + second : vb;
        for (uint64_t q = start; q < m; q += stride) {
            const uint32_t r = range_of(uint32_t(q)), at = begin[r] + (uint32_t(q) - place[r]);
            ka[at] = ks[q];
            if constexpr (VB > 0) va[at] = vs[q];
        }
    } else {
        const bool in_b = !copied && (total & 1) != 0;  // where the last pass left the result
        const bool to_a = in_b || copied;
        grid_copy_bytes(to_a ? p.keys_a : p.keys_b, copied ? p.copy_keys_in : in_b ? p.keys_b : p.keys_a,
                        p.n * uint64_t(KB));
        if constexpr (VB > 0)
            grid_copy_bytes(to_a ? p.vals_a : p.vals_b, copied ? p.copy_vals_in : in_b ? p.vals_b : p.vals_a,
                            p.n * uint64_t(VB));
    }
}

}  // namespace gbsort
