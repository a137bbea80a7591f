// shapes.h — CTA geometry of the onesweep pass per (key bytes, value bytes).
//
// Chosen for GB300: items per thread sized so two CTAs fit in an SM's 228 KB
// of shared memory where possible (two double-buffered key tiles, one value
// tile, per-warp counters and match words per CTA) and the register file
// holds keys, values and ranks without spilling.
#pragma once

#include <cmath>

#include <cstdint>

namespace gbsort {

// Threads of the upsweep (global histogram) kernel.
constexpr int HIST_THREADS = 1024;

// Measured on a GB300 (pass kernel, bench.py configurations):
//   4-byte keys only, 2^28:      384 x 24, 2 CTAs/SM  (67 Gkeys/s)
//   f32 keys + u32 values, 2^28: 256 x 26, 2 CTAs/SM  (49 Gkeys/s)
//   u64 keys + u64 values, 2^27: 256 x 14, 2 CTAs/SM  (15.0 Gkeys/s)
//   u128 keys only, 2^26:        384 x 16, 1 CTA/SM   (7.45 Gkeys/s)
// Tile bytes per key are 2K + V (only keys are double-buffered), so with
// values the tile grows with 2(K + V) / (2K + V) over a layout that double
// buffers both; other widths follow by bytes per item in the same budget.
struct ShapeRow {
    int threads, ipt, min_ctas;
};
constexpr ShapeRow pass_shape_row(int kb, int vb) {
    if (kb <= 4) {
        if (vb == 0) return {384, 24, 2};
        if (vb <= 4) return {256, 26, 2};
        if (vb == 8) return {256, 22, 2};
        return {256, 13, 2};
    }
    if (kb == 8) {
        if (vb == 0) return {256, 22, 2};
        if (vb <= 4) return {256, 17, 2};
        if (vb == 8) return {256, 14, 2};
        return {256, 10, 2};
    }
    if (vb == 0) return {384, 16, 1};
    if (vb <= 8) return {256, 8, 2};
    return {256, 6, 2};
}

// Small inputs (n <= 2^22, the reference's "short" range): tiles of about half
// the size at 256 threads and two CTAs per SM, so a short array still spreads
// over the SMs (2^20 u32 keys: 114 tiles of 9216 keys leave SMs idle; 256 of
// 4096 keys took 12.8 -> 14.2 Gkeys/s on GB300).
constexpr ShapeRow pass_shape_small_row(int kb, int vb) {
    if (kb <= 4) return {256, vb == 0 ? 16 : vb <= 4 ? 13 : vb == 8 ? 11 : 7, 2};
    if (kb == 8) return {256, vb == 0 ? 11 : vb <= 4 ? 9 : vb == 8 ? 7 : 5, 2};
    return {256, vb == 0 ? 8 : vb <= 8 ? 4 : 3, 2};
}
constexpr uint64_t SMALL_N_MAX = uint64_t(1) << 22;

// Arrays sorted in one launch when keys-only (fused_short.cuh): up to 2^21
// keys (2^20 for 16-byte keys, whose buckets outgrow a CTA sooner and whose
// 16 passes then run slower inside one launch: 2^21 u128 610 vs 567 us).
// With every digit taking a pass inside the launch, u32 measured (CUDA
// events) 2^16 40.8 vs 59.0 us, 2^20 56-58 vs 76.6, 2^22 164.8 vs 157.4;
// with the MSD partition + bucket sorts, 2^17 28.6 vs 62.5, 2^20 36.6 vs
// 76.6, 2^21 98 vs 111.
constexpr uint64_t FUSED_N_MAX = uint64_t(1) << 21;
constexpr uint64_t fused_n_max(int kb) { return kb == 16 ? FUSED_N_MAX / 2 : FUSED_N_MAX; }

// The one-launch short sort: the short shape's tile, ranked by 512 threads
// where it divides (half the columns per warp: a shorter dependent chain in
// the rank, which bounds a short sort's passes).
template <int KB>
struct FusedShape {
    static constexpr int TILE = pass_shape_small_row(KB, 0).threads * pass_shape_small_row(KB, 0).ipt;
    static constexpr int THREADS = TILE % 512 == 0 ? 512 : pass_shape_small_row(KB, 0).threads;
    static constexpr int IPT = TILE / THREADS;
    static constexpr int MIN_CTAS = pass_shape_small_row(KB, 0).min_ctas;
    // keys per thread of the bucket sort after the MSD partition: buckets of
    // up to THREADS * LIPT keys (2 and 4-byte keys 8192, 8-byte 7168, 16-byte
    // 3072), sized so that two CTAs still fit an SM
    static constexpr int LIPT = KB == 1 ? IPT : KB <= 4 ? 2 * IPT : KB == 8 ? 28 : 6;
};

// Keys per bucket the one-launch sort's CTA sorts in shared memory.
constexpr int fused_local_tile(int kb) {
    return kb == 1    ? FusedShape<1>::THREADS * FusedShape<1>::LIPT
           : kb == 2  ? FusedShape<2>::THREADS * FusedShape<2>::LIPT
           : kb == 4  ? FusedShape<4>::THREADS * FusedShape<4>::LIPT
           : kb == 8  ? FusedShape<8>::THREADS * FusedShape<8>::LIPT
                      : FusedShape<16>::THREADS * FusedShape<16>::LIPT;
}

// Keys-only sorts above the short range, most significant bits first
// (msd.cuh).
// The two splits: THREADS x IPT keys a tile; CAP places per digit in the stage
// (0: a dense stage).  Measured, top + second split: 4-byte keys 2^28 512 x 20
// with 69 places 0.47 + 0.50 ms (512 x 24, 79 places 0.48 + 0.51; 256 x 24
// dense 0.61 + 0.58: the dense stage's second random read bounds it); 8-byte
// keys 5 x 10^7 256 x 16 dense, 4 CTAs an SM, 0.166 + 0.163 ms (512 x 12
// with 43 places 0.177 + 0.195); 16-byte keys 2^26 512 x 6 dense 0.368 + 0.380
// (256 x 12 0.372 + 0.383).
// The local sorts: CTAs of C_THREADS, 64 bytes of keys a lane, C_HALO lanes of
// margin at a warp's ends, in two sizes: L = 1 for the upper half of the range
// of 8- and 16-byte keys, whose groups are twice as large.  Three CTAs an SM
// keep their registers (2^28 4-byte keys: 0.88 ms, four CTAs 1.11 with spills).
template <int KB>
struct MsdShape {
    static constexpr int THREADS = KB == 8 ? 256 : 512;
    static constexpr int IPT = KB == 16 ? 6 : KB == 8 ? 16 : 20;
    static constexpr int MIN_CTAS = KB == 8 ? 4 : 2;
    static constexpr int CAP = KB == 4 ? 69 : 0;
    static constexpr int C_THREADS[2] = {384, KB == 4 ? 384 : 768};
    static constexpr int C_HALO = KB == 16 ? 2 : 1;
    static constexpr int C_MIN_CTAS[2] = {3, KB == 4 ? 3 : 1};
};
constexpr uint64_t msd_n_max(int kb) {
    return kb == 16 ? uint64_t(1) << 27 : kb == 8 ? uint64_t(1) << 28 : uint64_t(5) << 26;
}
// Sizes whose size query has always held a block of its own for this path
// (8- and 16-byte keys; elsewhere the path's counters lie in the lookback
// status words, which it does not use, and the stage count is not reported).
constexpr uint64_t msd_block_n_min(int kb) {
    return kb == 16 ? uint64_t(3) << 19 : kb == 8 ? uint64_t(3) << 23 : ~uint64_t(0);
}
// 4-byte floats: from here on (N(0, 1), against four digit passes: 5 * 10^6 128
// and 127 us, 10^7 183 and 207, 6 * 10^7 745 and 945; values of one exponent
// 10^7 177 and 220, 6 * 10^7, where they are sent back, 1087 and 1020), and as long as 65536 groups hold them (MsdEvenCode's stretches
// take about a quarter more of the codes than even keys do).
constexpr uint64_t MSD_EVEN_N_MIN = uint64_t(1) << 23;
constexpr uint64_t MSD_EVEN_N_MAX = uint64_t(9) << 24;
constexpr int msd_local_shape(int kb, uint64_t n) { return kb == 4 || n <= (msd_n_max(kb) >> 1) ? 0 : 1; }
template <int KB>
constexpr uint32_t msd_group_cap_of(int shape) {
    using S = MsdShape<KB>;
    return uint32_t(S::C_THREADS[shape] / 32 * (32 - 2 * S::C_HALO) * (64 / KB) - 32 / KB);
}
constexpr uint32_t msd_group_cap(int kb, int shape) {
    return kb == 16 ? msd_group_cap_of<16>(shape) : kb == 8 ? msd_group_cap_of<8>(shape) : msd_group_cap_of<4>(shape);
}
// Most group bits below the top digit (the sample chooses how many): groups
// average at most 0.72 of the largest a local sort takes, so that uniform keys
// (a few standard deviations of sqrt(average)) and mildly uneven ones fit, and
// one bit more for keys that use only part of the codes' range.
constexpr int msd_b2_max(uint64_t n, uint32_t cap) {
    int b2 = 1;
    while (b2 < 8 && double(n) > 0.36 * double(cap) * double(256u << b2)) ++b2;
    return b2;
}

// Key-value sorts by their leading digits (finish.cuh): the finishing CTAs.
// 8- and 16-byte keys with 4- or 8-byte values.  4-byte keys keep their four
// digit passes: two of them and a finish took longer (2^26 u32 + u32 1.51
// against 1.42 ms, with a kernel for 4-byte keys that this library does not
// hold).
template <int KB>
struct FinishShape {
    static constexpr int THREADS = 384;
    static constexpr int LIPT = KB == 8 ? 8 : 4;
    static constexpr int HALO = KB == 16 ? 2 : 1;
    static constexpr int MIN_CTAS = 2;
};
constexpr bool finish_pairs(int kb, int vb) { return kb >= 8 && (vb == 4 || vb == 8); }
// 8-byte floats without values too, from here on (N(0, 1): 140001 keys 58 us,
// the one-launch sort, whose regions overflow, 81; 1.6 x 10^7 564, eight digit
// passes 770).
constexpr uint64_t FINISH_KEYS_N_MIN = uint64_t(1) << 14;
constexpr uint64_t FINISH_N_MIN = 2048;  // (u64 + u32, uniform: 16385 pairs 45 us, the digit passes 78)
// Short key-value arrays in one launch (short_pairs.cuh): regions of up to
// `cap` words (key and index) a CTA of THREADS sorts.
struct ShortPairsShape {
    static constexpr int THREADS = 384;
    static constexpr int MIN_CTAS = 3;
    static constexpr int halo(int kb) { return kb == 8 ? 2 : 1; }
};
constexpr uint32_t short_pairs_cap(int kb) {
    return (uint32_t(ShortPairsShape::THREADS / 32 * (32 - 2 * ShortPairsShape::halo(kb)) * (32 / kb)) - 8u) & ~3u;
}
// Regions: 256, or one or two per resident CTA of a GB300 (a region more than
// that waits for a whole round: 10^6 pairs in 512 regions 48 us, in 456 42;
// more regions than needed cost a global atomic each per tile: 600001 pairs in
// 456 36 us, in 256 31), the first of these whose mean region of uniform keys
// and six of its standard deviations fit the cap; 0: none do.
inline uint32_t short_pairs_need(uint64_t n, int regions) {  // words a region has to take
    const double mean = double(n) / double(regions);
    return (uint32_t(mean * 1.01 + 6.0 * std::sqrt(mean) + 8.0) + 4u) & ~3u;
}
inline int short_pairs_regions(int kb, uint64_t n) {
    for (int regions : {256, 456, 912})
        if (short_pairs_need(n, regions) <= short_pairs_cap(kb)) return regions;
    return 0;
}
// Words that the size query holds for a region: six times the mean, where the
// cap is not nearer, so that keys whose leading bits take few values (2^16 keys
// with 256 upper halves: six to a region somewhere) still sort here.  A
// DoubleBuffer workspace, whose point is its size, holds what uniform keys need.
inline uint32_t short_pairs_room(int kb, uint64_t n, int regions) {
    const uint64_t six = (6 * n / uint64_t(regions) + 64) & ~uint64_t(3);
    const uint32_t need = short_pairs_need(n, regions);
    return six > short_pairs_cap(kb) ? short_pairs_cap(kb) : six < need ? need : uint32_t(six);
}
constexpr uint64_t SHORT_PAIRS_N_MIN = 2048;

constexpr uint64_t FINISH_N_MAX = (uint64_t(1) << 31) - 1;  // edges keep a flag in bit 31

// Keys per MSD region of the one-launch sort (one region per top digit):
// the mean bucket n/256 plus four of its standard deviations plus 64,
// rounded up to 32 (uniform top digits overflow a region about once in
// 10^4 sorts at 2^20 keys, and then the sort takes the per-digit passes);
// 0 where that exceeds a CTA's local sort.
inline uint32_t msd_region_cap(int kb, uint64_t n) {
    const double mean = double((n + 255) / 256);
    const uint64_t cap = (uint64_t(mean + 4.0 * std::sqrt(mean) + 64.0) + 31) & ~uint64_t(31);
    return cap <= uint64_t(fused_local_tile(kb)) ? uint32_t(cap) : 0u;
}

// Predecessor tiles per lookback round trip for short arrays: all their tiles
// are in flight at once, so the known-prefix frontier moves a window per L2
// round trip (2^20 u32: 4 -> 8 took 14.0 -> 14.35 Gkeys/s; 16 and 32 slower).
#ifndef GBSORT_SMALL_WINDOW
#define GBSORT_SMALL_WINDOW 8
#endif

template <int KB, int VB>
struct PassShapeSmall {
    static constexpr int THREADS = pass_shape_small_row(KB, VB).threads;
    static constexpr int IPT = pass_shape_small_row(KB, VB).ipt;
    static constexpr int MIN_CTAS = pass_shape_small_row(KB, VB).min_ctas;
    static constexpr int LOOKBACK_WINDOW = GBSORT_SMALL_WINDOW;
};

template <int KB, int VB>
struct PassShape {
    static constexpr int THREADS = pass_shape_row(KB, VB).threads;
    static constexpr int IPT = pass_shape_row(KB, VB).ipt;
    // Resident CTAs per SM the register allocation must allow.
    static constexpr int MIN_CTAS = pass_shape_row(KB, VB).min_ctas;
    // Predecessor tiles read per lookback round trip.
    static constexpr int LOOKBACK_WINDOW = 4;
};

// Build-time override of one (key bytes, value bytes) shape, for tuning
// sweeps: -DGBSORT_SHAPE_KB=.. -DGBSORT_SHAPE_VB=.. -DGBSORT_SHAPE_THREADS=..
// -DGBSORT_SHAPE_IPT=.. -DGBSORT_SHAPE_MIN_CTAS=..
#if defined(GBSORT_SHAPE_KB)
#ifndef GBSORT_SHAPE_WINDOW
#define GBSORT_SHAPE_WINDOW 4
#endif
template <>
struct PassShape<GBSORT_SHAPE_KB, GBSORT_SHAPE_VB> {
    static constexpr int THREADS = GBSORT_SHAPE_THREADS;
    static constexpr int IPT = GBSORT_SHAPE_IPT;
    static constexpr int MIN_CTAS = GBSORT_SHAPE_MIN_CTAS;
    static constexpr int LOOKBACK_WINDOW = GBSORT_SHAPE_WINDOW;
};
#endif

// Older form of the override for the 4-byte keys-only shape.
#if defined(GBSORT_SHAPE_K4V0_THREADS)
template <>
struct PassShape<4, 0> {
    static constexpr int THREADS = GBSORT_SHAPE_K4V0_THREADS;
    static constexpr int IPT = GBSORT_SHAPE_K4V0_IPT;
    static constexpr int MIN_CTAS = GBSORT_SHAPE_K4V0_MIN_CTAS;
    static constexpr int LOOKBACK_WINDOW = GBSORT_SHAPE_K4V0_WINDOW;
};
#endif

// Value-size index used by the dispatch tables: 0,1,2,4,8,16 bytes -> 0..5.
inline int value_index(int vb) {
    switch (vb) {
        case 0: return 0;
        case 1: return 1;
        case 2: return 2;
        case 4: return 3;
        case 8: return 4;
        case 16: return 5;
        default: return -1;
    }
}

struct KernelEntry {
    const void* fn;
    int threads;
    int ipt;
    int tile;
    unsigned long smem;
};

// Defined in inst_k{1,2,4,8,16}.cu: entries[value_index][wide_status].
const KernelEntry* pass_entries(int kb);
const KernelEntry* upsweep_entry(int kb);

}  // namespace gbsort
