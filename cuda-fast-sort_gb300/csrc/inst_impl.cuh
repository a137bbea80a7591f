// inst_impl.cuh — explicit kernel instantiations for one key width.  Each
// inst_k*.cu includes this with one width, so the five widths compile as
// parallel translation units.
#pragma once

#include "finish.cuh"
#include "fused_short.cuh"
#include "msd.cuh"
#include "multi.cuh"
#include "onesweep.cuh"
#include "segmented.cuh"
#include "shapes.h"
#include "short_pairs.cuh"

namespace gbsort {

template <int KB, int VB, class W, bool SEG, class S = PassShape<KB, VB>>
KernelEntry make_pass_entry() {
    using G = PassGeom<KB, VB, S::THREADS, S::IPT>;
    return KernelEntry{
        reinterpret_cast<const void*>(
            &onesweep_pass_kernel<KB, VB, W, S::THREADS, S::IPT, SEG, S::MIN_CTAS, S::LOOKBACK_WINDOW>),
        S::THREADS, S::IPT, G::TILE, static_cast<unsigned long>(G::SMEM_BYTES)};
}

// Several passes in one cooperative launch: [0: 32-bit status, 1: 64-bit
// status, 2: small-n shape], then those that follow a path which may leave
// ranges to sort.
template <int KB, int VB, class W, class S = PassShape<KB, VB>, bool LEFT = false>
KernelEntry make_multi_entry() {
    using G = PassGeom<KB, VB, S::THREADS, S::IPT>;
    return KernelEntry{reinterpret_cast<const void*>(&onesweep_multi_kernel<KB, VB, W, S::THREADS, S::IPT, S::MIN_CTAS,
                                                                            S::LOOKBACK_WINDOW, LEFT>),
                       S::THREADS, S::IPT, G::TILE, static_cast<unsigned long>(G::SMEM_BYTES)};
}
template <int KB, int VB>
const KernelEntry* multi_entries_of() {
    using S = PassShape<KB, VB>;
    using T = PassShapeSmall<KB, VB>;
    static const KernelEntry e[6] = {
        make_multi_entry<KB, VB, uint32_t>(), make_multi_entry<KB, VB, uint64_t>(),
        make_multi_entry<KB, VB, uint32_t, T>(),
        make_multi_entry<KB, VB, uint32_t, S, true>(), make_multi_entry<KB, VB, uint64_t, S, true>(),
        make_multi_entry<KB, VB, uint32_t, T, true>()};
    return e;
}

// [value size][0: 32-bit status, 1: 64-bit status, 2: small-n shape (32-bit)]
template <int KB, int VB>
struct PassRow {
    KernelEntry e[3];
    PassRow()
        : e{make_pass_entry<KB, VB, uint32_t, false>(), make_pass_entry<KB, VB, uint64_t, false>(),
            make_pass_entry<KB, VB, uint32_t, false, PassShapeSmall<KB, VB>>()} {}
};

template <int KB>
const KernelEntry* pass_entries_for() {
    static const PassRow<KB, 0> r0;
    static const PassRow<KB, 1> r1;
    static const PassRow<KB, 2> r2;
    static const PassRow<KB, 4> r4;
    static const PassRow<KB, 8> r8;
    static const PassRow<KB, 16> r16;
    static const KernelEntry e[6][3] = {
        {r0.e[0], r0.e[1], r0.e[2]},    {r1.e[0], r1.e[1], r1.e[2]},    {r2.e[0], r2.e[1], r2.e[2]},
        {r4.e[0], r4.e[1], r4.e[2]},    {r8.e[0], r8.e[1], r8.e[2]},    {r16.e[0], r16.e[1], r16.e[2]},
    };
    return &e[0][0];
}

// The one-launch sort of short keys-only arrays, in the short-array pass shape.
template <int KB>
const KernelEntry* fused_entry_for() {
    using S = FusedShape<KB>;
    using G = ShortGeom<KB, S::THREADS, S::IPT, S::LIPT>;
    static_assert(G::TILE == PassShapeSmall<KB, 0>::THREADS * PassShapeSmall<KB, 0>::IPT, "same tiles as the short shape");
    static const KernelEntry e = {
        reinterpret_cast<const void*>(&fused_short_kernel<KB, S::THREADS, S::IPT, S::LIPT, S::MIN_CTAS>), S::THREADS,
        S::IPT, G::TILE, static_cast<unsigned long>(G::SMEM_BYTES)};
    return &e;
}

// Keys-only sorts above the short range, most significant bits first: sample,
// count, scan, top split, second split, local sorts (two sizes).
template <int KB, int L, bool EVEN = false>
KernelEntry make_msd_local_entry() {
    using S = MsdShape<KB>;
    using GL = GroupSortGeom<KB, S::C_THREADS[L], S::C_HALO>;
    static_assert(GL::CAP == int(msd_group_cap_of<KB>(L)), "the plan's capacity");
    return KernelEntry{
        reinterpret_cast<const void*>(&msd_local_kernel<KB, S::C_THREADS[L], S::C_MIN_CTAS[L], S::C_HALO, EVEN>),
        S::C_THREADS[L], GL::LIPT, GL::CAP, static_cast<unsigned long>(GL::SMEM_BYTES)};
}

template <int KB>
const KernelEntry* msd_entries_for() {
    using S = MsdShape<KB>;
    using GS = MsdSplitGeom<KB, S::THREADS, S::IPT, S::CAP>;
    static const KernelEntry e[8] = {
        {reinterpret_cast<const void*>(&msd_sample_kernel<KB>), MSD_SAMPLE_THREADS, 0, 0, 0ul},
        {reinterpret_cast<const void*>(&msd_count_kernel<KB, false>), MSD_COUNT_THREADS, 0, 0,
         static_cast<unsigned long>(MSD_COUNT_SMEM)},
        {reinterpret_cast<const void*>(&msd_scan_kernel<false>), 256, 0, 0, 0ul},
        {reinterpret_cast<const void*>(&msd_top_kernel<KB, S::THREADS, S::IPT, S::MIN_CTAS, S::CAP, false>), S::THREADS,
         S::IPT, GS::TILE, static_cast<unsigned long>(GS::SMEM_BYTES)},
        {reinterpret_cast<const void*>(&msd_second_kernel<KB, S::THREADS, S::IPT, S::MIN_CTAS, S::CAP, false>), S::THREADS, S::IPT,
         GS::TILE, static_cast<unsigned long>(GS::SMEM_BYTES)},
        make_msd_local_entry<KB, 0>(),
        make_msd_local_entry<KB, 1>(),
        {reinterpret_cast<const void*>(&msd_map_ranges_kernel<KB>), 256, 0, 0, 0ul},
    };
    return e;
}

// The same for 4-byte floats.
template <int KB>
const KernelEntry* msd_even_entries_for() {
    using S = MsdShape<KB>;
    using GS = MsdSplitGeom<KB, S::THREADS, S::IPT, S::CAP>;
    static const KernelEntry e[6] = {
        {reinterpret_cast<const void*>(&msd_even_sample_kernel<KB>), MSD_SAMPLE_THREADS, 0, 0,
         static_cast<unsigned long>(MSD_EVEN_SMEM)},
        {reinterpret_cast<const void*>(&msd_count_kernel<KB, true>), MSD_COUNT_THREADS, 0, 0,
         static_cast<unsigned long>(MSD_COUNT_SMEM + MsdEvenCode::BINS * 8)},
        {reinterpret_cast<const void*>(&msd_scan_kernel<true>), 256, 0, 0, 0ul},
        {reinterpret_cast<const void*>(&msd_top_kernel<KB, S::THREADS, S::IPT, S::MIN_CTAS, S::CAP, true>), S::THREADS,
         S::IPT, GS::TILE, static_cast<unsigned long>(GS::EVEN_BYTES)},
        {reinterpret_cast<const void*>(&msd_second_kernel<KB, S::THREADS, S::IPT, S::MIN_CTAS, S::CAP, true>), S::THREADS,
         S::IPT, GS::TILE, static_cast<unsigned long>(GS::EVEN_BYTES)},
        make_msd_local_entry<KB, 0, true>(),
    };
    return e;
}

// Sorts by leading digits: sample, edges, finish (4- and 8-byte values; 8-byte
// keys without values too).
template <int KB, int VB>
KernelEntry make_finish_entry() {
    using S = FinishShape<KB>;
    using F = FinishGeom<KB, VB, S::THREADS, S::LIPT, S::HALO>;
    return KernelEntry{reinterpret_cast<const void*>(&finish_kernel<KB, VB, S::THREADS, S::MIN_CTAS, S::LIPT, S::HALO>),
                       S::THREADS, F::LIPT, F::CAP, static_cast<unsigned long>(F::SMEM_BYTES)};
}
template <int KB>
const KernelEntry* finish_entries_for() {
    static const KernelEntry e[5] = {
        {reinterpret_cast<const void*>(&finish_sample_kernel<KB>), FINISH_SAMPLE_THREADS, 0, finish_levels<KB>() + 1,
         static_cast<unsigned long>(FINISH_SAMPLE_SMEM)},
        {reinterpret_cast<const void*>(&finish_edges_kernel<KB>), 256, 0, 0, 0ul},
        make_finish_entry<KB, 4>(),
        make_finish_entry<KB, 8>(),
        [] {
            if constexpr (KB == 8) return make_finish_entry<KB, 0>();
            else return KernelEntry{};
        }(),
    };
    return e;
}

// Short key-value arrays in one launch: [4- or 8-byte values][that kernel, the
// digit passes in one launch].
template <int KB, int VB>
KernelEntry make_short_pairs_entry() {
    using S = ShortPairsShape;
    using G = ShortPairsGeom<KB, S::THREADS, S::halo(KB)>;
    static_assert(uint32_t(G::CAP) == short_pairs_cap(KB), "the plan's capacity");
    return KernelEntry{reinterpret_cast<const void*>(&short_pairs_kernel<KB, VB, S::THREADS, S::MIN_CTAS, S::halo(KB)>),
                       S::THREADS, 0, G::CAP, static_cast<unsigned long>(G::SMEM_BYTES)};
}
template <int KB>
const KernelEntry* short_pairs_entries_for() {
    static const KernelEntry e[4] = {
        make_short_pairs_entry<KB, 4>(), make_multi_entry<KB, 4, uint32_t, PassShapeSmall<KB, 4>>(),
        make_short_pairs_entry<KB, 8>(), make_multi_entry<KB, 8, uint32_t, PassShapeSmall<KB, 8>>()};
    return e;
}

template <int KB>
const KernelEntry* upsweep_entry_for() {
    static const KernelEntry e = {reinterpret_cast<const void*>(&upsweep_kernel<KB>), HIST_THREADS, 0, 0,
                                  static_cast<unsigned long>(HistGeom<KB>::SMEM_BYTES)};
    return &e;
}

// ---- batched mode ---------------------------------------------------------
// Small-segment CTA sorts: "S" = 256 threads x 8 items (8- or 4-bit digits),
// "L" = 512 threads x as many items as keep the two shared buffers within
// 128 KB (8-bit digits).
template <int KB, int VB>
struct CtaShapes {
    static constexpr int S_THREADS = 256, S_IPT = 8;
    static constexpr int L_THREADS = 512;
    static constexpr int L_ITEMS_RAW = 65536 / (KB + VB);
    static constexpr int L_IPT = L_ITEMS_RAW / L_THREADS > 32 ? 32 : (L_ITEMS_RAW / L_THREADS < 4 ? 4 : L_ITEMS_RAW / L_THREADS);
};

template <int KB, int VB, int THREADS, int IPT, int RBITS>
KernelEntry make_cta_entry() {
    using GC = CtaSortGeom<KB, VB, THREADS, IPT, RBITS>;
    return KernelEntry{reinterpret_cast<const void*>(&cta_sort_kernel<KB, VB, THREADS, IPT, RBITS>), THREADS, IPT,
                       GC::TILE, static_cast<unsigned long>(GC::SMEM_BYTES)};
}

template <int KB, int VB>
void make_seg_entries(KernelEntry* out /* [4]: pass, cta S, cta L, cta S 4-bit */) {
    using C = CtaShapes<KB, VB>;
    out[0] = make_pass_entry<KB, VB, uint32_t, true>();
    out[1] = make_cta_entry<KB, VB, C::S_THREADS, C::S_IPT, 8>();
    out[2] = make_cta_entry<KB, VB, C::L_THREADS, C::L_IPT, 8>();
    out[3] = make_cta_entry<KB, VB, C::S_THREADS, C::S_IPT, 4>();
}

template <int KB>
const KernelEntry* seg_entries_for() {
    static KernelEntry e[6][4];
    static const bool init = [] {
        make_seg_entries<KB, 0>(e[0]);
        make_seg_entries<KB, 1>(e[1]);
        make_seg_entries<KB, 2>(e[2]);
        make_seg_entries<KB, 4>(e[3]);
        make_seg_entries<KB, 8>(e[4]);
        make_seg_entries<KB, 16>(e[5]);
        return true;
    }();
    (void)init;
    return &e[0][0];
}

template <int KB>
const KernelEntry* seg_upsweep_entry_for() {
    static const KernelEntry e = {reinterpret_cast<const void*>(&seg_upsweep_kernel<KB>), SEG_UP_THREADS, 0, 0,
                                  static_cast<unsigned long>(SegHistGeom<KB>::SMEM_BYTES)};
    return &e;
}

}  // namespace gbsort
