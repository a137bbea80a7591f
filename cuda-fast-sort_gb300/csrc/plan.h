// plan.h — host-side planning of one sort: geometry, workspace layout and
// launch sizes.  Shared by the plain sort (sort_api.cu) and the batched path.
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "shapes.h"
#include "sort_params.h"

namespace gbsort {

constexpr size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Control block at the start of the workspace's control region:
//   [gp_counts: passes*256 u64][tile_counters: 16 u32][err: u32][executed: u32][barrier: u32][pad]
//   [barrier generation: u32, own 128-byte line][pad]
// executed: written by the pass kernels that run (bit 31 | passes executed)
// when uniform passes are skipped; 0 when none ran.
struct CtlLayout {
    size_t gp_off = 0;
    size_t counters_off = 0;
    size_t err_off = 0;
    size_t exec_off = 0;
    size_t barrier_off = 0;      // grid barrier counter of the one-launch short sort
    size_t barrier_gen_off = 0;  // its generation word (another 128-byte line)
    size_t fill_off = 0;         // [256] fill counts of its MSD regions
    size_t overflow_off = 0;     // its region overflow flag
    size_t msd_state_off = 0;    // outcome of the most-significant-first path, its code window [2]
    // Sorts by leading digits use the fill counts' words, which only the
    // one-launch sort needs: a second set of tile counters [16] and a second grid
    // barrier [2], for the digit passes after them, the sample's ticket and
    // [FINISH_LEVELS + 2] counts, and the number and the total of the ranges left
    // to sort (keys-only sorts above the short range, too).
    size_t counters2_off = 0;
    size_t sampled_off = 0;
    size_t ranges_off = 0;
    size_t bytes = 0;
    static constexpr CtlLayout make(int passes) {
        CtlLayout c;
        c.gp_off = 0;
        c.counters_off = size_t(passes) * 256 * 8;
        c.err_off = c.counters_off + 16 * 4;
        c.exec_off = c.err_off + 4;
        c.barrier_off = c.exec_off + 4;
        c.barrier_gen_off = align_up(c.barrier_off + 4, 128);
        c.fill_off = align_up(c.barrier_gen_off + 4, 128);
        c.overflow_off = c.fill_off + 256 * 4;
        c.msd_state_off = c.overflow_off + 4;
        c.counters2_off = c.fill_off;
        c.sampled_off = c.counters2_off + 18 * 4;
        c.ranges_off = c.sampled_off + 9 * 4;
        c.bytes = align_up(c.msd_state_off + 12, 256);
        return c;
    }
};

// The counters of the most-significant-first path (offsets from
// Plan::msd_off; msd.cuh): keys per top digit, their cursors, then keys per
// group and their cursors.  BYTES is what the size query has always held for
// it where it has a block of its own.
struct MsdLayout {
    static constexpr size_t TOP = 0;
    static constexpr size_t CURSOR1 = 256 * 4;
    static constexpr size_t JOINT = 512 * 4;
    static constexpr size_t bytes(int b2) { return JOINT + 2 * (size_t(256) << b2) * 4; }
    static constexpr size_t BYTES = 256 + 256 * 4 + 3 * 65536 * 4;
    static_assert(JOINT + 2 * 65536 * 4 <= BYTES, "the counters fit their block");
    // 4-byte floats: then the large groups of equal keys, cleared with the
    // counters, and the codes' table, a sampled key of every
    // bin, and the range of the codes
    static constexpr size_t GIANTS_BYTES = 256;
    static constexpr size_t even_bytes(int b2) { return bytes(b2) + GIANTS_BYTES + 4096 * 12 + 16; }
};

struct Plan {
    int key_type = 0;
    int kb = 0;            // key bytes
    int vb = 0;            // value bytes (0: keys only)
    int kind = 0;          // KeyKind
    int passes = 0;
    bool wide_status = false;
    KernelEntry pass{};
    KernelEntry upsweep{};
    // One-launch path (short keys-only arrays): upsweep, passes and fix-up in
    // one cooperative kernel of pass's shape.  fused.fn == nullptr: not used.
    KernelEntry fused{};
    uint64_t n = 0;
    uint32_t num_tiles = 0;
    // workspace layout (offsets from the workspace base)
    size_t alt_keys_off = 0;
    size_t alt_vals_off = 0;
    size_t ctl_off = 0;
    size_t status_off = 0;
    size_t status_bytes = 0;
    // the one-launch sort's MSD regions: 256 x msd_cap keys (msd_cap 0: none)
    size_t regions_off = 0;
    uint32_t msd_cap = 0;
    // keys-only sorts above the short range, most significant bits first
    // (msd.cuh): kernels (sample, count, scan, top split, second split, local
    // sorts), group capacity, most group bits below the top digit, and the place
    // of the counters: a block of their own (msd_block), else the lookback
    // status words, which only the digit passes use
    bool msd = false;
    bool msd_block = false;
    bool msd_even = false;  // 4-byte floats: codes by the sample's distribution
    KernelEntry msd_k[6]{};
    uint32_t msd_group_cap = 0;
    int msd_b2 = 0;
    size_t msd_off = 0;
    // the digit passes in one launch, after (or, by leading digits, in) a path
    // that seldom needs all of them
    KernelEntry multi{};
    KernelEntry after{};  // the same after a path that may have left ranges to sort
    // sorts by leading digits (finish.cuh): sample, edges,
    // finish; the edges lie in the status words
    bool finish = false;
    KernelEntry finish_k[3]{};
    // short key-value arrays in one launch (short_pairs.cuh): that kernel, the
    // digit passes after it, its regions, the words in each, and their place, at
    // the end of the workspace (their fill counts lie in the status words, which
    // only the digit passes use)
    bool short_pairs = false;
    KernelEntry short_k[2]{};
    int short_regions = 0;
    uint32_t short_cap = 0;
    size_t short_off = 0;
    size_t min_bytes = 0;    // workspace below which a sort is refused (without regions)
    size_t total_bytes = 0;  // what the size query asks for
    CtlLayout ctl{};
    // the process-wide switches as this plan found them, each read once: the
    // kernels, their parameters and the graph's key have to agree while another
    // thread changes them
    bool skip = false;       // uniform-digit pass skipping
    bool short_msd = false;  // most significant digit first inside the one-launch sort

    uint32_t ranges_most() const {  // room in the list of ranges left to sort
        const size_t most = status_bytes / 64;
        return num_tiles < 4 ? 0u : uint32_t(most < RANGES_MOST ? most : RANGES_MOST);
    }
};

// Fills *plan; returns a gbsort_status code.
int make_plan(int key_type, size_t value_bytes, uint64_t n, Plan* plan);

// DoubleBuffer form: the caller's second key (and value) buffer replaces
// the workspace's alternate buffers, and the workspace holds only the
// control block and the lookback status (double_buffer_bytes).  The result
// lands in the second buffer when the pass count is odd, else in the first.
struct AltBuffers {
    void* keys_b;
    void* vals_b;
};
size_t double_buffer_bytes(const Plan& plan);

// Makes the plan fit a workspace of `bytes` (of a DoubleBuffer sort: `alt`):
// regions as large as there is room for, or none.  False: too small for any sort.
bool fit_workspace(Plan* plan, size_t bytes, bool alt);

// Enqueues one sort on `stream`.  `ms` (optional) receives per-kernel event
// times after a stream sync: [upsweep, pass 0 .. pass P-1].
// keys_src != nullptr: input-preserving sort, reads keys_src (and vals_src)
// and leaves the result in d_keys (and d_values).
int enqueue_sort(const Plan& plan, int descending, void* d_keys, void* d_values, void* d_workspace,
                 cudaStream_t stream, float* ms, int ms_cap, int* n_ms, const void* keys_src = nullptr,
                 const void* vals_src = nullptr, const AltBuffers* alt = nullptr);

// Device facts (cached per device).
int device_sm_count();
int device_is_sm103();
int resident_ctas(const KernelEntry& e);  // per SM, after opting in to the smem
int prepare_kernel(const KernelEntry& e); // cudaFuncSetAttribute once per device
uint32_t upsweep_ctas(uint64_t n, int kb);  // grid of the plain upsweep

uint64_t wait_limit_ns();
int status_from_error_word(uint32_t err);  // workspace error word -> gbsort_status
void set_last_error(const char* what, cudaError_t err);
void set_last_error_text(const char* text);

}  // namespace gbsort
