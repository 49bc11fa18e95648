// Internal helpers shared by the engine, the kernels and the clause sharer.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <string>

#include "gpusharesat.h"

namespace gss {

// Longest clause the engine accepts. The reference stops at 100
// (MAX_CL_SIZE, gpuShareLib/BaseTypes.cuh:28); the sharer keeps that limit
// by default, the engine itself takes clauses up to this length.
constexpr int kMaxClauseLen = 4096;
// Most 32-slot words of a pass.
constexpr int kMaxWords = 4096;

// Tiles of the tiled check kernel: consecutive length-sorted clauses with at
// most kTileLits literals (a longer clause gets a tile of its own and is read
// from global memory). kBufLits leaves room for rounding a tile's literal
// range out to 16-byte boundaries for the bulk copy.
constexpr int kTileLits = 512;
constexpr int kBufLits = kTileLits + 8;

// Zero literals after the last clause: kernels that read a few literals ahead
// stay inside the buffer.
constexpr int kClausePad = 8;

// Database order by variable ranges of 2^shift variables: the key of a
// clause is (its most frequent range, its second range, its length);
// `reordered` (optional, len entries) receives its literals with those of
// the most frequent range first, then the second range's, and so on.
uint64_t range_order_key(const int32_t *lits, int64_t len, int shift, int32_t *reordered);
// The range shift for a database whose largest variable is max_var
// (range_log2: -1 automatic = 17, 0 = no ranges); 0 when one range would do.
int range_shift_for(int64_t max_var, int range_log2);

// Sets the calling thread's error message and returns `code`.
int set_error(int code, const char *fmt, ...);

// Checks a CUDA call; on failure records the message and returns GSS_ERR_CUDA.
#define GSS_CUDA_TRY(call)                                                        \
    do {                                                                          \
        cudaError_t _e = (call);                                                  \
        if (_e != cudaSuccess) {                                                  \
            return ::gss::set_error(GSS_ERR_CUDA, "%s failed: %s (%s:%d)", #call, \
                                    cudaGetErrorString(_e), __FILE__, __LINE__);  \
        }                                                                         \
    } while (0)

#define GSS_TRY(expr)          \
    do {                       \
        int _rc = (expr);      \
        if (_rc != GSS_OK) {   \
            return _rc;        \
        }                      \
    } while (0)

// A device buffer that grows by doubling and never shrinks.
struct DevBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
    int reserve(size_t need);  // keeps nothing of the old contents
    int grow_keep(size_t need, cudaStream_t stream, size_t keep_bytes);
    void release();
    ~DevBuf() { release(); }
};

struct PinnedBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
    int reserve(size_t need);
    void release();
    ~PinnedBuf() { release(); }
};

// Arguments of one check pass over the length-sorted CSR clause database.
struct CheckArgs {
    const int32_t *lits;        // device, CSR literals, clauses sorted by length
    const int64_t *offsets;     // device, n_clauses + 1
    const uint32_t *orig;       // device, original index of each sorted clause
    uint32_t n_clauses;
    const uint2 *state;         // device, [n_blocks][n_vars][lpc] {isDef, isTrue}
    uint32_t n_vars;
    uint32_t n_blocks;          // slot blocks of lpc words
    const uint32_t *start;      // device, [n_blocks * lpc], zero past the last word
    const int32_t *solver_of_word;  // device, [n_blocks * lpc]
    gss_report *out;            // device, n_parts * cap_per_part records
    uint32_t *counts;           // device, n_parts counters (zeroed by the caller)
    uint32_t count_stride;      // words from one counter to the next
    uint32_t n_parts;
    uint32_t cap_per_part;
    int lpc;                    // lanes (32-slot words) per clause
    int g;                      // state loads in flight per lane (direct) / clause slots (tiled)
    int cache_hints;            // L1/L2 eviction hints on the loads
    // tiled kernel only
    const uint32_t *tile_clause;  // device, n_tiles + 1: first sorted clause of each tile
    const uint32_t *tile_lit;     // device, n_tiles + 1: first literal of each tile
    uint32_t n_tiles;
    uint32_t *err;                // device flag, set to nonzero when a bounded wait gives up
    const uint32_t *alive;        // device, 1 bit per clause (NULL: every clause is live)
    uint32_t alive_by_id;         // alive is indexed by orig[c] rather than by c
    // Scan order: this launch checks the clauses at scan positions
    // [scan_begin, scan_end); position i is clause perm[i] when perm is set
    // and i < perm_end, clause i otherwise.
    const uint32_t *perm;
    uint32_t scan_begin, scan_end;
    uint32_t perm_end;
    // filtered kernel only: the word-level table [n_blocks][2 * n_vars] of the
    // state, and the counter of (clause, block) pairs it kept
    const uint2 *agg;
    uint32_t *kept;
};

__host__ __device__ __forceinline__ uint32_t scan_count(const CheckArgs &a) {
    return a.scan_end > a.scan_begin ? a.scan_end - a.scan_begin : 0u;
}
// Clause at offset i of this launch's scan range (i < scan_count).
__device__ __forceinline__ uint32_t scan_clause(const CheckArgs &a, uint32_t i) {
    const uint32_t p = a.scan_begin + i;
    return (a.perm && p < a.perm_end) ? __ldg(a.perm + p) : p;
}

// Whether clause c of the database takes part in the pass.
__device__ __forceinline__ bool clause_live(const CheckArgs &a, uint32_t c) {
    if (a.alive == nullptr) return true;
    const uint32_t i = a.alive_by_id ? __ldg(a.orig + c) : c;
    return (__ldg(a.alive + (i >> 5)) >> (i & 31)) & 1u;
}

// A per-range lane-layout plan for the bucketed kernel (device memory):
// range k covers scan positions [range_begin[k], range_end[k]) and is checked
// with lane layout layout[k] (GSS_LAYOUT_*); group_base[k] is the index of
// its first clause group over all ranges, group_base[n_ranges] their total.
constexpr uint32_t kMaxRanges = 8192;
struct BucketPlan {
    uint32_t n_ranges;
    uint32_t range_begin[kMaxRanges];
    uint32_t range_end[kMaxRanges];
    int32_t layout[kMaxRanges];
    uint32_t group_base[kMaxRanges + 1];
};
int layout_lanes(int layout);  // lanes per clause of a layout, 0 if unknown
int launch_check_bucketed(const CheckArgs *d_args, const BucketPlan *d_plan, uint32_t *work, cudaStream_t stream,
                          int sm_count);

// Order-preserving device compaction of a CSR clause database: keeps the
// clauses whose id (ids[c]) has its bit set in `alive`.
struct CompactArgs {
    const int32_t *lits;
    const int64_t *offsets;  // n_clauses + 1
    const uint32_t *ids;
    uint32_t n_clauses;
    const uint32_t *alive;   // bit per id
    int32_t *new_lits;       // room for the live literals + kClausePad
    int64_t *new_offsets;    // room for n_clauses + 1
    uint32_t *new_ids;       // room for n_clauses
    void *scratch;           // compact_scratch_bytes(n_clauses), 256-byte aligned
};
size_t compact_scratch_bytes(uint32_t n_clauses);
// Rebuilds a CSR clause database in a new order on the device: new clause c
// is old clause src[c], placed at new_offsets[c] (device arrays, n_new + 1
// offsets); new_ids[c] = c; kClausePad zero literals after the last one.
struct GatherArgs {
    const int32_t *lits;
    const int64_t *offsets;
    const uint32_t *src;
    const int64_t *new_offsets;
    uint32_t n_new;
    int64_t n_new_lits;
    int32_t *new_lits;     // room for n_new_lits + kClausePad
    uint32_t *new_ids;     // room for n_new
};
int gather_clauses(const GatherArgs &a, cudaStream_t stream, int sm_count);
// Packs report partitions (n_parts x cap records, counts[p] valid in
// partition p, device) into contiguous 12-byte {clause, word, mask} records,
// or, with cell_words > 0, 8-byte {clause * cell_words + word, mask} records.
int launch_pack_reports(const gss_report *parts, const uint32_t *counts, uint32_t n_parts, uint32_t cap,
                        uint32_t cell_words, uint32_t *packed, cudaStream_t stream, int sm_count);
// A pass's counters buffer: the n_parts report counters, the kernel's error
// flag and the filter's counter of kept clauses, and the work counters of the
// persistent kernels. One memset clears them all. An address takes an atomic
// every 1.5 ns or so, and neighbours in a line share that rate, so every
// counter has 256 bytes to itself (500k clauses x 96 words of fair-coin slots,
// eight reports a clause: 311 us, 559 with all counters side by side), and
// the tasks come from kWorkCounters (62500 tasks from one counter took 100 us
// whatever they did).
constexpr uint32_t kCountStride = 64;
constexpr uint32_t kExtraCounters = 2;
constexpr uint32_t kWorkCounters = 16;
constexpr size_t kWorkBytes = sizeof(uint32_t) * kWorkCounters * kCountStride;
__host__ __device__ __forceinline__ uint32_t *err_counter(uint32_t *counts, uint32_t n_parts) {
    return counts + n_parts * kCountStride;
}
__host__ __device__ __forceinline__ uint32_t *kept_counter(uint32_t *counts, uint32_t n_parts) {
    return counts + n_parts * kCountStride + 1;
}
__host__ __device__ __forceinline__ uint32_t *work_counter(uint32_t *counts, uint32_t n_parts) {
    return counts + (n_parts + 1) * kCountStride;
}
// Bytes of the buffer with `sets` sets of work counters: the head and the tail
// of an ordered pass have one each.
constexpr uint32_t kWorkSets = 2;
inline size_t counter_bytes(uint32_t n_parts, uint32_t sets = kWorkSets) {
    return sizeof(uint32_t) * (n_parts + 1) * kCountStride + sets * kWorkBytes;
}
// Hands a pass's outcome to the host: writes the report counters, the error
// flag and the filter's count, side by side, to `host` (pinned), and, when the pass has at most max_inline
// records and no partition overflowed, the records too, partition after
// partition from byte kInlineOffset on. With d_args the queues are those of
// the arguments in device memory (a captured graph outlives a queue's growth).
// clear: the counters are zero again when it is done (the last use of them in
// the pass; it takes the place of the next pass's memset).
constexpr size_t kInlineOffset = 256;
int launch_deliver(const CheckArgs *d_args, const gss_report *parts, uint32_t *counts, uint32_t n_parts,
                   uint32_t cap, void *host, uint32_t max_inline, bool clear, cudaStream_t stream);
// Synchronizes `stream`; returns the live clause and literal counts.
int compact_by_id(const CompactArgs &a, cudaStream_t stream, int sm_count, uint32_t *n_out, int64_t *lits_out);

// The automatic variant for a pass of n_words words: kind, lanes per clause,
// loads in flight. Up to four words a lane takes the whole clause (narrow
// kernel). From five on, four words a lane with 256-bit loads, and the
// narrowest row that holds all words (32 at most): one scan of the database
// where two blocks of half the width read every clause twice. Measured, one
// wide block against the narrower kind or two blocks (600k clauses, lengths
// 2-100), on fair-coin slots: 6 words 51 against 79 us, 11 words 73 against
// 84, 24 words 120 against 129, 17 words 114 against 110; on trails, behind
// the filter: 6 words 25 against 61, 11 and 17 words 28 against 37.
inline void auto_layout(int n_words, int &kind, int &lpc, int &depth) {
    kind = n_words > 4 ? GSS_KERNEL_WIDE4 : GSS_KERNEL_DIRECT;
    if (n_words > 4)
        lpc = n_words > 16 ? 8 : n_words > 8 ? 4 : 2;
    else
        lpc = n_words > 2 ? 4 : n_words > 1 ? 2 : 1;
    depth = lpc == 1 ? 1 : 2;
}

// Resident blocks of 256 threads per multiprocessor of a kernel; `known` is a
// static of its launcher (asked of the runtime once, not at every launch; an
// error is the call's, and the next one asks again).
template <typename K>
int resident_blocks(K kernel, std::atomic<int> &known, int &n) {
    n = known.load(std::memory_order_relaxed);
    if (n > 0) return GSS_OK;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 256, 0);
    if (e != cudaSuccess) {
        cudaGetLastError();  // said here; not to be met again after the next launch
        return set_error(GSS_ERR_CUDA, "cudaOccupancyMaxActiveBlocksPerMultiprocessor failed: %s",
                         cudaGetErrorString(e));
    }
    if (n < 1) n = 1;
    known.store(n, std::memory_order_relaxed);
    return GSS_OK;
}

// Launches the check kernel on `stream` (the counters must already be zero).
// Returns a GSS status.
int launch_check(const CheckArgs &a, cudaStream_t stream, int sm_count);
bool valid_variant(int lpc, int g);
int launch_check_tiled(const CheckArgs &a, cudaStream_t stream, int sm_count);
int launch_check_wide(const CheckArgs &a, int wpl, int occ, cudaStream_t stream, int sm_count);
// Pipelined wide kernel (occ: 4 blocks per SM register cap).
int launch_check_wide_pf(const CheckArgs &a, int wpl, int occ, cudaStream_t stream, int sm_count);
bool valid_wide_pf_variant(int wpl, int lpc, int g);
// Persistent wide kernel: arguments read from device memory (d_args, so that
// a captured graph serves every pass) or, when d_args is NULL, passed by
// value (h_args); tasks from the device counter `work` (zero it before each
// launch).
int launch_check_wide_persist(const CheckArgs *d_args, const CheckArgs &h_args, int wpl, int lpc, int g, uint32_t *work,
                              cudaStream_t stream, int sm_count);
bool valid_wide_persist_variant(int wpl, int lpc, int g);
bool valid_wide_variant(int wpl, int lpc, int g, int occ);
bool valid_tiled_variant(int lpc, int k);

// A pass of one slot block of 1, 2 or 4 words (a.lpc), a lane per clause;
// tasks from the counters at `work`.
int launch_check_narrow(const CheckArgs &a, uint32_t *work, cudaStream_t stream, int sm_count);
bool valid_narrow_variant(int words);
// The persistent wide kernel behind the word-level filter (h_args.agg, or
// that of d_args).
int launch_check_filtered(const CheckArgs *d_args, const CheckArgs &h_args, int wpl, int lpc, uint32_t *work,
                          cudaStream_t stream, int sm_count);
bool valid_filtered_variant(int wpl, int lpc);
// The share of its (clause, block) pairs that a filtered pass may keep: past it
// the pass costs more than the plain one, and the passes after it run without
// before the next try. The plain scan of a narrow block is cheap, so the line
// lies lower there. Break-even measured over states of rising mixture, clauses
// of 3, 2 to 30, 2 to 100, 20 to 60 and Zipf lengths, 5e5 and 1e6 of them, 2^13 /
// 2^16 / 2^18 / 2^20 variables: 8 words 0.20, 0.20, 0.05, 0.20; 16 words 0.30,
// 0.30, 0.25, 0.33; 32 words 0.6, 0.6, 0.33, 0.5; two blocks of 32 over 2^18
// 0.38. Under these lines no measured pass of 16 or 32 words lost to the plain
// one (32 words: 0.96 of it at most), six of 136 of 8 words lost 5 to 14%, and
// three of 90 of 14 words 6 to 19%; with 1/3 for all, 8 words had lost up to 48%.
inline double filter_keep_most(int bw) { return bw <= 8 ? 0.10 : bw <= 16 ? 0.20 : 1.0 / 3; }
inline bool filter_keeps_too_much(uint32_t kept, int64_t n_clauses, int64_t n_blocks, int bw) {
    return (double) kept > filter_keep_most(bw) * (double) n_clauses * (double) n_blocks;
}
// How long: a state that comes and goes should not cost the ones after it the
// filter, and one that stays should not be tried often. The pause doubles
// with every try that fails, from 4 passes to 64 (a state that stays costs
// five tries in its first 64 passes, one in 65 from then on), and starts
// again where a try succeeds or the database or the layout is another.
struct FilterPause {
    static constexpr int kLeast = 4, kMost = 64;
    int left = 0;  // passes to run without
    int next = kLeast;
    void note(bool kept_too_much) {  // of a pass that ran behind the filter
        if (left > 0) return;        // (launched before the pause began)
        if (kept_too_much) {
            left = next;
            next = next < kMost ? 2 * next : kMost;
        } else {
            next = kLeast;
        }
    }
    void end() { left = 0, next = kLeast; }
};
// What a pass saves behind a table that pays, in us: for the decision to fill
// it or to keep it up. Measured on model and trail states, 2 to 100 literals a
// clause, pass behind the table against plain, 5e3 / 2e5 / 4e5 clauses over
// 2^18 variables: 8 words 21/23, 27/30, 32/37 us; 13 words 21/25, 27/31, 32/42;
// 32 words 21/29, 27/42, 31/60; 64 words 21/28, 31/65, 39/96.
inline double filter_gain(int64_t n_clauses, int n_words) {
    return 0.25 * (n_words < 32 ? n_words : 32) + 2.0e-6 * (double) n_clauses * n_words;
}
// Its tasks are counted in 32 bits (with room for what the warps take past the end).
constexpr uint64_t kMaxFilterTasks = 1ull << 31;
inline uint64_t filter_tasks(const CheckArgs &a) { return ((uint64_t) scan_count(a) + 31) / 32 * a.n_blocks; }
// [n_vars][n_words] -> [n_blocks][n_vars][bw], zero-padded words (in_place:
// src is laid out already), and the filter's table `agg` (NULL: none), 16
// bytes a variable and block.
int launch_load_state(const uint2 *src, uint2 *dst, uint2 *agg, uint32_t n_vars, uint32_t n_words, uint32_t bw,
                      uint32_t n_blocks, bool in_place, cudaStream_t stream, int sm_count);
// A word of a variable's state that a pass changes.
struct StateUpdate {
    uint32_t var;
    uint32_t word;
    uint32_t is_def;
    uint32_t is_true;
};
// The table's entries of the rows that n updates changed, from the state.
int launch_refresh_agg(const StateUpdate *u, uint32_t n, const uint2 *state, uint2 *agg, uint32_t n_vars,
                       uint32_t n_words, uint32_t bw, cudaStream_t stream, int sm_count);
// start and solver_of_word of a pass from device memory, padded with zeros to
// `padded` words; solver_of_word NULL: the word's own number. With `state`,
// n_pairs (variable, word) pairs in any order, also counts the "false" bits
// that density_samples(n_pairs) of them give the filter's table, over both
// literals, into *n_false (pinned). start NULL: the masks are there already.
int launch_load_masks(const uint32_t *start, const int32_t *solver_of_word, uint32_t n_words, uint32_t padded,
                      uint32_t *start_out, int32_t *sow_out, const uint2 *state, uint64_t n_pairs, uint32_t *n_false,
                      cudaStream_t stream);
constexpr uint64_t kDensitySamples = 1 << 12;
inline uint64_t density_samples(uint64_t n_pairs) { return n_pairs < kDensitySamples ? n_pairs : kDensitySamples; }

}  // namespace gss
