// The check behind a word-level filter, and the kernels that keep the filter's
// tables.
//
// A slot word's 32 slots are the assignments of one solver. For a literal and
// a word, two bits say whether the literal is false, and whether it is
// undefined, in any of the word's slots. The check rule is monotone in its
// inputs, so running it once on these bits (a "slot" now being a whole word)
// keeps every word in which some slot reports: what it drops needs no look at
// the slots. The table is 8 bytes a literal and block of 32 words, a sixteenth
// of the state, and usually fits L2 whole (16 MB at 2^20 variables).
//
// What it saves depends on the slots. A solver's assignments differ by a few
// variables, and solvers of one formula agree on much, so on trails a clause
// is dropped after 4 to 6 literals of 8 bytes, where the exact scan gathers 7
// rows of 256 bytes. Independent fair-coin slots make every bit 1 and drop
// nothing; a sample of the state tells (use_filter), and such states keep
// the plain kernel and get no table.
//
// (The reference tests a clause first against an aggregate over all solvers,
// gpuShareLib/GpuRunner.cu:152-170; its aggregate is one bit per solver too,
// kept by atomics as variables change, gpuShareLib/Assigs.cu:100-141.)
#include <algorithm>

#include "check_rows.cuh"

namespace gss {
namespace {

// The filter's table of a literal: words with a slot where it is false (x)
// and where it is undefined (y).
__device__ __forceinline__ uint2 ld_agg(const uint2 *p) {
    uint2 v;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;"
        : "=r"(v.x), "=r"(v.y)
        : "l"(p), "l"(policy_keep()));
    return v;
}

constexpr int kPair = 2;        // table entries a lane reads at a time
// The warp turns to the clauses left one by one when they are this few and
// have more than these many chunks to go (1, 2, 4 and 8 lanes measured 67,
// 65, 69 and 71 us; short remainders are faster lane by lane).
constexpr int kFewLanes = 2;
constexpr uint32_t kFewChunks = 3;
constexpr int kFewWords = 4;    // words left for which a survivor is checked literal-parallel
constexpr int kFewSurvivors = 16;
// Literals a lane has in flight in both: a long clause that reports is the
// last thing a pass waits for (400k Zipf clauses x 11 words: 26 us with one,
// 24 with two; four spill, 59 against 57 us on 2e6 clauses x 1024 slots).
constexpr int kLong = 2;
constexpr int kFilterStage = 64;  // staged records per warp: few are found

// The rest of the filter for the clauses of the lanes in `open`, one by one
// with 32 * kLong literals a step; returns the lane's words left.
__device__ __forceinline__ uint32_t finish_clauses(const int32_t *__restrict__ lits, const uint2 *__restrict__ agg,
                                                unsigned open, uint32_t pos, uint32_t end, uint32_t all,
                                                uint32_t live) {
    const int lane = lane_id();
    while (open) {
        const int src = __ffs(open) - 1;
        open &= open - 1;
        uint32_t p = __shfl_sync(kFull, pos, src), fa = __shfl_sync(kFull, all, src),
                 fl = __shfl_sync(kFull, live, src);
        const uint32_t e = __shfl_sync(kFull, end, src);
        for (; p < e && fl; p += 32 * kLong) {
            uint32_t lit[kLong], f = ~0u, o = 0u;
#pragma unroll
            for (int k = 0; k < kLong; k++) {
                const uint32_t at = p + 32 * k + lane;
                lit[k] = at < e ? (uint32_t) __ldg(lits + at) : 0u;
            }
#pragma unroll
            for (int k = 0; k < kLong; k++) {
                const uint2 v = p + 32 * k + lane < e ? ld_agg(agg + lit[k]) : make_uint2(~0u, 0u);
                merge_runs(f, o, v.x, v.y);
            }
            warp_runs(f, o);
            fl = (fa & o) | (fl & f);
            fa &= f;
        }
        if (lane == src) live = fl;
    }
    return live;
}

// The exact check of the clauses (c of each lane) that the filter kept, on
// the words `live` it left; records go to the warp's stage, whose new fill is
// returned. Few survivors with few words each (reports, and clauses that the
// word-level bits could not tell from them) are checked literal-parallel;
// otherwise groups of LPC lanes scan them as the plain wide kernel does.
template <int WPL, int LPC, int G>
__device__ __forceinline__ uint32_t check_survivors(const CheckArgs &a, StagedReport *stage, uint32_t nstaged, uint32_t blk,
                                                 uint32_t c, uint32_t live) {
    constexpr int CPW = 32 / LPC;
    constexpr int BW = WPL * LPC;
    const int lane = lane_id(), sub = lane % LPC, grp = lane / LPC, gbase = grp * LPC;
    const uint32_t *start = a.start + blk * BW;
    const uint2 *rows = a.state + (size_t) blk * a.n_vars * BW;
    unsigned left = __ballot_sync(kFull, live != 0u);
    if (__popc(left) <= kFewSurvivors) {
        unsigned by_literal = __ballot_sync(kFull, live != 0u && __popc(live) <= kFewWords);
        left &= ~by_literal;
        // up to four (clause, word) pairs at a time, eight lanes each; a pair
        // on its own gets the whole warp
        uint32_t words = 0;
        int src = 0;
        while (by_literal || words) {
            int n_pairs = 0, my_src = 0, my_word = 0;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (!words && by_literal) {
                    src = __ffs(by_literal) - 1;
                    by_literal &= by_literal - 1;
                    words = __shfl_sync(kFull, live, src);
                }
                if (words) {
                    if (lane / 8 == q || q == 0) my_src = src, my_word = __ffs(words) - 1;
                    words &= words - 1;
                    n_pairs++;
                }
            }
            const bool alone = n_pairs == 1;
            const uint32_t cc = __shfl_sync(kFull, c, my_src);
            const bool on = alone || lane / 8 < n_pairs;
            const uint32_t step = alone ? 32u : 8u;
            uint32_t fa = 0, fl = 0, p = 0, e = 0;
            if (on) {
                p = (uint32_t) __ldg(a.offsets + cc) + (alone ? lane : lane % 8);
                e = (uint32_t) __ldg(a.offsets + cc + 1);
                fa = fl = __ldg(start + my_word);
            }
            while (__any_sync(kFull, p < e && fl)) {
                uint32_t lit[kLong], f = ~0u, o = 0u;
                Row<1> v[kLong];
#pragma unroll
                for (int k = 0; k < kLong; k++)
                    lit[k] = p + k * step < e && fl ? (uint32_t) __ldg(a.lits + p + k * step) : 0u;
#pragma unroll
                for (int k = 0; k < kLong; k++)
                    if (p + k * step < e && fl) ld_row<1>(rows + (size_t) (lit[k] >> 1) * BW + my_word, v[k]);
#pragma unroll
                for (int k = 0; k < kLong; k++)
                    if (p + k * step < e && fl)
                        merge_runs(f, o, (v[k].v[1] ^ ((lit[k] & 1u) - 1u)) & v[k].v[0], ~v[k].v[0]);
#pragma unroll
                for (int d = 1; d < 32; d *= 2) {
                    if (d >= 8 && !alone) break;
                    const uint32_t f2 = __shfl_xor_sync(kFull, f, d), o2 = __shfl_xor_sync(kFull, o, d);
                    merge_runs(f, o, f2, o2);
                }
                fl = (fa & o) | (fl & f);
                fa &= f;
                p += kLong * step;
            }
            const bool writes = alone ? lane == 0 : lane % 8 == 0;
            const unsigned bal = __ballot_sync(kFull, writes && fl != 0u);
            if (bal) {
                if (nstaged + 4 > (uint32_t) kFilterStage) {
                    flush_mapped(a, stage, nstaged);
                    nstaged = 0;
                }
                if (writes && fl) stage_record(stage + nstaged + __popc(bal & lanemask_lt()), cc, blk * BW + my_word, fl);
                nstaged += __popc(bal);
            }
        }
    }
    while (left) {  // CPW survivors at a time, a group of lanes each
        unsigned m = left;
        for (int q = 0; q < grp; q++) m &= m - 1;
        const int src = m ? __ffs(m) - 1 : 0;
        const uint32_t cc = __shfl_sync(kFull, c, src);
        uint32_t words = __shfl_sync(kFull, live, src);
        uint32_t p = 0, e = 0;
        if (m) {
            p = (uint32_t) __ldg(a.offsets + cc);
            e = (uint32_t) __ldg(a.offsets + cc + 1);
        } else {
            words = 0u;
        }
        uint32_t al[WPL], lv[WPL];
        Row<WPL> st[G];
#pragma unroll
        for (int k = 0; k < G; k++)
#pragma unroll
            for (int q = 0; q < 2 * WPL; q++) st[k].v[q] = 0u;
#pragma unroll
        for (int j = 0; j < WPL; j++)
            al[j] = lv[j] = (words >> (sub * WPL + j)) & 1u ? __ldg(start + sub * WPL + j) : 0u;
        scan_rows<WPL, LPC, G>(a, rows + sub * WPL, p, e, sub, gbase, al, lv, st);
#pragma unroll
        for (int j = 0; j < WPL; j++) {
            const unsigned bal = __ballot_sync(kFull, lv[j] != 0u);
            if (bal) {
                if (nstaged + 32 > (uint32_t) kFilterStage) {
                    flush_mapped(a, stage, nstaged);
                    nstaged = 0;
                }
                if (lv[j])
                    stage_record(stage + nstaged + __popc(bal & lanemask_lt()), cc, blk * BW + sub * WPL + j, lv[j]);
                nstaged += __popc(bal);
            }
        }
        for (int q = 0; q < CPW; q++) left &= left - 1;
    }
    return nstaged;
}

// A persistent warp takes 32 clauses of one slot block at a time, a lane per
// clause: the lane walks its literals, read 16 bytes at a time one chunk
// ahead, kPair table entries at a time. When few of the 32 are left with much
// to read, the whole warp takes them one by one (a 256-literal clause that
// reports would otherwise be 64 dependent steps); then the survivors get the
// exact check.
//
// Bound by the L2's rate of random requests, a table entry each (ncu on 2e6
// clauses x 1024 slots: 11.2M requests in 59 us, 189 G/s; the plain kernel
// takes 245 us there). Hence: table entries keep their place in L2
// (L1::no_allocate alone marks them evict-first there: half of them missed,
// 86 us), nothing scattered is allocated in L1 (its 128-byte lines bound the
// misses in flight: 65 against 59 us), two entries at a time rather than four
// (what a dropped clause had in flight is waste), and tasks from several
// counters (one counter's atomics alone took 100 us for 62500 tasks). More
// warps with fewer registers are no faster (65 us at 6 blocks a
// multiprocessor, 59 at 4: their spills cost the requests they add).
template <int WPL, int LPC, int G, int MINB>
__global__ void __launch_bounds__(kWarps * 32, MINB) check_filtered_kernel(const CheckArgs *__restrict__ pa,
                                                                            const CheckArgs av,
                                                                            uint32_t *__restrict__ work) {
    constexpr int BW = WPL * LPC;
    __shared__ CheckArgs sa;
    __shared__ StagedReport stage_all[kWarps][kFilterStage];
    __shared__ uint32_t survivors;
    if (threadIdx.x == 0) {
        sa = pa ? *pa : av;
        survivors = 0;
    }
    __syncthreads();
    const CheckArgs &a = sa;
    const int lane = threadIdx.x & 31;
    StagedReport *stage = stage_all[threadIdx.x >> 5];
    uint32_t nstaged = 0, kept = 0;

    const uint32_t n_scan = scan_count(a);
    const uint32_t n_groups = (n_scan + 31) / 32;
    const uint32_t n_tasks = n_groups * a.n_blocks;  // below 2^32 (launch_check_filtered)
    // A task's clauses and their offsets are loaded during the task before it,
    // its number two tasks before.
    const TaskCounter counter(work);
    auto clause_at = [&](uint32_t task) -> uint32_t {
        if (task >= n_tasks) return 0xFFFFFFFFu;
        const uint32_t i = task % n_groups * 32 + lane;
        return i < n_scan ? scan_clause(a, i) : 0xFFFFFFFFu;
    };
    uint32_t task = counter.first();
    uint32_t next = __shfl_sync(kFull, counter.take(lane), 0);
    uint32_t c = clause_at(task), pos = 0, end = 0;
    if (c < a.n_clauses) {
        pos = (uint32_t) __ldg(a.offsets + c);
        end = (uint32_t) __ldg(a.offsets + c + 1);
    }
    uint4 chunk = make_uint4(0u, 0u, 0u, 0u);  // the literals around pos
    if (pos < end) chunk = ld_chunk(a.lits, pos);
    while (task < n_tasks) {
        const uint32_t after = counter.take(lane);
        const uint32_t c1 = clause_at(next);
        uint32_t pos1 = 0, end1 = 0;
        if (c1 < a.n_clauses) {
            pos1 = (uint32_t) __ldg(a.offsets + c1);
            end1 = (uint32_t) __ldg(a.offsets + c1 + 1);
        }
        const uint32_t blk = task / n_groups;
        const bool valid = c < a.n_clauses && clause_live(a, c);
        const uint32_t *start = a.start + blk * BW;
        const uint2 *agg = a.agg + (size_t) blk * a.n_vars * 2;
        // words with a started slot
        const uint32_t started = __ballot_sync(kFull, lane < BW && __ldg(start + lane % BW) != 0u);
        bool fetch = true;
        uint4 ahead = make_uint4(0u, 0u, 0u, 0u);  // the next task's first chunk
        uint32_t all = valid ? started : 0u, live = all;
        unsigned open;  // lanes with a word and a literal left
        while ((open = __ballot_sync(kFull, live != 0u && pos < end)) != 0u) {
            // few clauses left, with much to read: the whole warp takes each
            if (__popc(open) <= kFewLanes &&
                __ballot_sync(kFull, live != 0u && pos + kFewChunks * 4 < end) == open)
                break;
            if (live == 0u) end = pos;  // nothing left to read
            const uint32_t b = pos & ~3u;
            uint4 after4 = chunk;
            if (b + 4 < end) after4 = ld_chunk(a.lits, b + 4);
            const uint32_t lit[4] = {chunk.x, chunk.y, chunk.z, chunk.w};
#pragma unroll
            for (int h = 0; h < 4; h += kPair) {
                uint2 r[kPair];
#pragma unroll
                for (int k = 0; k < kPair; k++)
                    r[k] = live != 0u && b + h + k >= pos && b + h + k < end ? ld_agg(agg + lit[h + k])
                                                                           : make_uint2(~0u, 0u);
                if (h == 0 && fetch) {  // while the table is read, the next task's first literals
                    if (pos1 < end1) ahead = ld_chunk(a.lits, pos1);
                    fetch = false;
                }
#pragma unroll
                for (int k = 0; k < kPair; k++) {
                    live = (all & r[k].y) | (live & r[k].x);
                    all &= r[k].x;
                }
            }
            pos = b + 4;
            chunk = after4;
        }
        if (fetch && pos1 < end1) ahead = ld_chunk(a.lits, pos1);
        if (open) live = finish_clauses(a.lits, agg, open, pos, end, all, live);
        const unsigned left = __ballot_sync(kFull, live != 0u);
        kept += __popc(left);
        if (left) nstaged = check_survivors<WPL, LPC, G>(a, stage, nstaged, blk, c, live);
        task = next;
        next = __shfl_sync(kFull, after, 0);
        c = c1;
        chunk = ahead;
        pos = pos1;
        end = end1;
    }
    if (nstaged) flush_mapped(a, stage, nstaged);
    // how many (clause, block) pairs the filter kept: tells whether it pays
    if (lane == 0 && kept) atomicAdd(&survivors, kept);
    __syncthreads();
    if (threadIdx.x == 0 && survivors) atomicAdd(a.kept, survivors);
}

// One row of the state (BW words of one variable, a lane each) to its table
// entries. Lane `w` holds word w of its row; the rows of a warp lie side by
// side, 32 / BW of them.
template <int BW>
__device__ __forceinline__ void row_entries(uint2 v, uint32_t real_words, int lane, uint2 &pos, uint2 &neg) {
    const int shift = lane / BW * BW;
    constexpr uint32_t mask = BW == 32 ? ~0u : (1u << (BW % 32)) - 1u;
    const bool real = (uint32_t) (lane % BW) < real_words;
    const uint32_t f = (__ballot_sync(kFull, real && (v.x & ~v.y) != 0u) >> shift) & mask;  // a slot where it is false
    const uint32_t t = (__ballot_sync(kFull, real && (v.x & v.y) != 0u) >> shift) & mask;   // ... true
    const uint32_t u = (__ballot_sync(kFull, real && v.x != ~0u) >> shift) & mask;          // ... undefined
    pos = make_uint2(f, u);  // the positive literal
    neg = make_uint2(t, u);
}

// Copies a state from the host-facing layout [n_vars][n_words] to slot blocks
// [n_blocks][n_vars][BW] (zero past the last word) and fills the filter's
// table on the way; src == dst leaves the state in place (it is laid out
// already). HBM-bound: a warp moves 256 bytes a step, kUnroll steps in
// flight, with a 32-bit division a row at most, and streaming stores (402 MB
// in three blocks, a whole gss_state_set: 201 us with plain stores, 193 so; a
// plain copy of it alone 123).
template <int BW>
__global__ void __launch_bounds__(256) load_state_kernel(const uint2 *__restrict__ src, uint2 *__restrict__ dst,
                                                         uint2 *__restrict__ agg, uint32_t n_vars, uint32_t n_words,
                                                         uint32_t n_blocks, bool in_place) {
    constexpr int RPW = 32 / BW;  // rows per warp step
    constexpr int kUnroll = 4;
    const int lane = threadIdx.x & 31;
    const uint32_t w = lane % BW;
    const uint64_t n_rows = (uint64_t) n_vars * n_blocks;  // row r: variable r / n_blocks, block r % n_blocks
    const uint64_t warps = (uint64_t) gridDim.x * (blockDim.x >> 5);
    for (uint64_t s = (uint64_t) blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); s * kUnroll * RPW < n_rows;
         s += warps) {
        uint2 v[kUnroll];
        size_t to[kUnroll];
        uint32_t real[kUnroll];
#pragma unroll
        for (int q = 0; q < kUnroll; q++) {
            const uint64_t r = (s * kUnroll + q) * RPW + lane / BW;
            uint32_t var = (uint32_t) r, blk = 0u;
            if (n_blocks != 1) {
                var = n_rows <= 0xFFFFFFFFull ? (uint32_t) r / n_blocks : (uint32_t) (r / n_blocks);
                blk = (uint32_t) (r - (uint64_t) var * n_blocks);
            }
            const uint32_t word = blk * BW + w;
            const bool in = r < n_rows;
            to[q] = in ? ((size_t) blk * n_vars + var) : ~(size_t) 0;
            real[q] = in ? min((uint32_t) BW, n_words - blk * BW) : 0u;
            v[q] = make_uint2(0u, 0u);
            if (in && word < n_words) v[q] = in_place ? src[to[q] * BW + w] : src[(uint64_t) var * n_words + word];
        }
#pragma unroll
        for (int q = 0; q < kUnroll; q++) {
            const bool in = to[q] != ~(size_t) 0;
            if (in && !in_place) __stcs(dst + to[q] * BW + w, v[q]);  // read rarely behind the filter
            if (agg) {
                uint2 p, n;
                row_entries<BW>(v[q], real[q], lane, p, n);
                if (in && w == 0) reinterpret_cast<uint4 *>(agg)[to[q]] = make_uint4(p.x, p.y, n.x, n.y);
            }
        }
    }
}

// The table entries of the rows that a list of updates touched (after all of
// them are in the state): a warp per update, 32 / BW at a time.
template <int BW>
__global__ void __launch_bounds__(256) refresh_agg_kernel(const StateUpdate *__restrict__ u, uint32_t n,
                                                          const uint2 *__restrict__ state, uint2 *__restrict__ agg,
                                                          uint32_t n_vars, uint32_t n_words) {
    constexpr int RPW = 32 / BW;
    const int lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); s * RPW < n; s += warps) {
        const uint32_t i = s * RPW + lane / BW;
        const bool in = i < n;
        const StateUpdate x = u[in ? i : n - 1];
        const uint32_t blk = x.word / BW;
        const size_t row = (size_t) blk * n_vars + x.var;
        uint2 p, q;
        row_entries<BW>(state[row * BW + lane % BW], min((uint32_t) BW, n_words - blk * BW), lane, p, q);
        if (in && lane % BW == 0) reinterpret_cast<uint4 *>(agg)[row] = make_uint4(p.x, p.y, q.x, q.y);
    }
}

// Block 0 copies the masks; block 1 samples the state for the density of its
// table, straight to the host: pairs spread over the state by a multiplicative
// hash, 4 for a thread. 2^12 pairs tell the share of a bit to within 0.8%
// (one standard deviation) in 2 us (2^14: 10), before a table is filled that
// may not be wanted. (The kernel that fills the table had counted all its
// bits, with a fill and a copy of their own: a whole gss_state_set of 8 words
// and 2^18 variables 32 us; so 25 with the table and 22 without.)
constexpr int kSampleThreads = 1024;
__global__ void __launch_bounds__(kSampleThreads)
    load_masks_kernel(const uint32_t *__restrict__ start, const int32_t *__restrict__ sow, uint32_t n_words,
                      uint32_t padded, uint32_t *__restrict__ start_out, int32_t *__restrict__ sow_out,
                      const uint2 *__restrict__ state, uint64_t n_pairs, uint32_t samples,
                      uint32_t *__restrict__ n_false) {
    if (blockIdx.x == 1) {
        __shared__ uint32_t sum;
        if (threadIdx.x == 0) sum = 0;
        __syncthreads();
        uint32_t n = 0;
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < samples; i += kSampleThreads) {
            const uint64_t at = samples == n_pairs ? i : __umul64hi(((uint64_t) i + 1) * 0x9E3779B97F4A7C15ull, n_pairs);
            const uint2 v = state[at];
            n += ((v.x & ~v.y) != 0u) + ((v.x & v.y) != 0u);
        }
        n = __reduce_add_sync(kFull, n);
        if ((threadIdx.x & 31) == 0) atomicAdd(&sum, n);
        __syncthreads();
        if (threadIdx.x == 0) *n_false = sum;
        return;
    }
    if (start == nullptr) return;
    for (uint32_t w = threadIdx.x; w < padded; w += blockDim.x) {
        start_out[w] = w < n_words ? start[w] : 0u;
        sow_out[w] = w < n_words ? (sow ? sow[w] : (int32_t) w) : 0;
    }
}

template <int WPL, int LPC, int G>
int launch_filtered_variant(const CheckArgs *d_args, const CheckArgs &h_args, uint32_t *work, cudaStream_t stream,
                            int sm_count) {
    constexpr int MINB = 4;
    static std::atomic<int> known{0};
    int per_sm = 0;
    GSS_TRY((resident_blocks(check_filtered_kernel<WPL, LPC, G, MINB>, known, per_sm)));
    // a captured graph serves databases of other sizes too: the full grid
    uint64_t blocks = (uint64_t) sm_count * per_sm;
    if (!d_args) {
        const uint64_t n_tasks = (uint64_t) ((scan_count(h_args) + 31) / 32) * h_args.n_blocks;
        blocks = std::min<uint64_t>(blocks, std::max<uint64_t>((n_tasks + kWarps - 1) / kWarps, 1));
    }
    check_filtered_kernel<WPL, LPC, G, MINB><<<(unsigned) blocks, kWarps * 32, 0, stream>>>(d_args, h_args, work);
    GSS_CUDA_TRY(cudaGetLastError());
    return GSS_OK;
}

}  // namespace

bool valid_filtered_variant(int wpl, int lpc) { return wpl == 4 && (lpc == 8 || lpc == 4 || lpc == 2); }

int launch_check_filtered(const CheckArgs *d_args, const CheckArgs &h_args, int wpl, int lpc, uint32_t *work,
                          cudaStream_t stream, int sm_count) {
    if (wpl == 4 && lpc == 8) return launch_filtered_variant<4, 8, 2>(d_args, h_args, work, stream, sm_count);
    if (wpl == 4 && lpc == 4) return launch_filtered_variant<4, 4, 2>(d_args, h_args, work, stream, sm_count);
    if (wpl == 4 && lpc == 2) return launch_filtered_variant<4, 2, 2>(d_args, h_args, work, stream, sm_count);
    return set_error(GSS_ERR_INVALID, "no filtered kernel for %d words per lane, %d lanes", wpl, lpc);
}

int launch_load_state(const uint2 *src, uint2 *dst, uint2 *agg, uint32_t n_vars, uint32_t n_words, uint32_t bw,
                      uint32_t n_blocks, bool in_place, cudaStream_t stream, int sm_count) {
    const uint64_t rows = (uint64_t) n_vars * n_blocks;
    if (rows == 0 || (in_place && !agg)) return GSS_OK;
    const uint64_t steps = (rows * bw + 127) / 128;  // 128 words a warp step
    const unsigned blocks = (unsigned) std::min<uint64_t>((steps + 7) / 8, (uint64_t) sm_count * 8);
#define GSS_LOAD(B)                                                                                                  \
    if (bw == B) {                                                                                                   \
        load_state_kernel<B><<<blocks, 256, 0, stream>>>(src, dst, agg, n_vars, n_words, n_blocks, in_place);         \
        GSS_CUDA_TRY(cudaGetLastError());                                                                            \
        return GSS_OK;                                                                                               \
    }
    GSS_LOAD(1) GSS_LOAD(2) GSS_LOAD(4) GSS_LOAD(8) GSS_LOAD(16) GSS_LOAD(32)
#undef GSS_LOAD
    return set_error(GSS_ERR_INVALID, "no state layout with %u words per block", bw);
}

int launch_load_masks(const uint32_t *start, const int32_t *solver_of_word, uint32_t n_words, uint32_t padded,
                      uint32_t *start_out, int32_t *sow_out, const uint2 *state, uint64_t n_pairs, uint32_t *n_false,
                      cudaStream_t stream) {
    if ((start == nullptr || padded == 0) && state == nullptr) return GSS_OK;
    load_masks_kernel<<<state ? 2 : 1, kSampleThreads, 0, stream>>>(start, solver_of_word, n_words, padded, start_out,
                                                                     sow_out, state, n_pairs,
                                                                     (uint32_t) density_samples(n_pairs), n_false);
    GSS_CUDA_TRY(cudaGetLastError());
    return GSS_OK;
}

int launch_refresh_agg(const StateUpdate *u, uint32_t n, const uint2 *state, uint2 *agg, uint32_t n_vars,
                       uint32_t n_words, uint32_t bw, cudaStream_t stream, int sm_count) {
    if (n == 0) return GSS_OK;
    const uint64_t warps = ((uint64_t) n * bw + 31) / 32;
    const unsigned blocks = (unsigned) std::min<uint64_t>((warps + 7) / 8, (uint64_t) sm_count * 8);
#define GSS_REFRESH(B)                                                                                 \
    if (bw == B) {                                                                                     \
        refresh_agg_kernel<B><<<blocks, 256, 0, stream>>>(u, n, state, agg, n_vars, n_words);          \
        GSS_CUDA_TRY(cudaGetLastError());                                                              \
        return GSS_OK;                                                                                 \
    }
    GSS_REFRESH(8) GSS_REFRESH(16) GSS_REFRESH(32)
#undef GSS_REFRESH
    return set_error(GSS_ERR_INVALID, "no filter table with %u words per block", bw);
}

}  // namespace gss
