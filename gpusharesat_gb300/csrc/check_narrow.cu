// The check for narrow passes: up to four 32-slot words, a few solvers or one.
//
// A literal's row is then 8, 16 or 32 bytes, one sector, and one lane takes a
// whole clause with all its words: 32 clauses a warp, with no lane idle on a
// word that does not exist and no shuffle to hand a literal around. The
// literals come 16 bytes at a time, one chunk ahead, kPair rows in flight; the
// next task's clauses, offsets and first chunk are loaded during the current
// one. Bound by the latency of that chain and the rate of random sectors. The
// direct kernel walked literal -> row one at a time: 600k clauses x 1 word
// 48 us cold, 38 us back to back; here 18 us.
#include <algorithm>

#include "check_rows.cuh"

namespace gss {
namespace {

constexpr int kPair = 2;
constexpr int kFewLanes = 2;  // as in the filtered kernel
constexpr uint32_t kFewChunks = 3;

template <int NW>
__device__ __forceinline__ void ld_narrow(const uint2 *p, Row<NW> &r);
template <>
__device__ __forceinline__ void ld_narrow<1>(const uint2 *p, Row<1> &r) {
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;"
        : "=r"(r.v[0]), "=r"(r.v[1])
        : "l"(p), "l"(policy_keep()));
}
template <>
__device__ __forceinline__ void ld_narrow<2>(const uint2 *p, Row<2> &r) {
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3])
        : "l"(p), "l"(policy_keep()));
}
template <>
__device__ __forceinline__ void ld_narrow<4>(const uint2 *p, Row<4> &r) {
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8], %9;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7])
        : "l"(p), "l"(policy_keep()));
}

template <int NW, int MINB>
__global__ void __launch_bounds__(kWarps * 32, MINB) check_narrow_kernel(const CheckArgs a,
                                                                          uint32_t *__restrict__ work) {
    __shared__ StagedReport stage_all[kWarps][kStage];
    const int lane = threadIdx.x & 31;
    StagedReport *stage = stage_all[threadIdx.x >> 5];
    uint32_t nstaged = 0;
    const uint32_t n_scan = scan_count(a);
    const uint32_t n_tasks = (n_scan + 31) / 32;
    uint32_t start[NW];
#pragma unroll
    for (int j = 0; j < NW; j++) start[j] = __ldg(a.start + j);
    const TaskCounter counter(work);
    auto clause_at = [&](uint32_t task) -> uint32_t {
        const uint64_t i = (uint64_t) task * 32 + lane;
        return i < n_scan ? scan_clause(a, (uint32_t) i) : 0xFFFFFFFFu;
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
        const bool valid = c < a.n_clauses && clause_live(a, c);
        bool fetch = true;
        uint4 ahead = make_uint4(0u, 0u, 0u, 0u);  // the next task's first chunk
        uint32_t all[NW], live[NW];
#pragma unroll
        for (int j = 0; j < NW; j++) all[j] = live[j] = valid ? start[j] : 0u;
        auto some = [&]() -> bool {
            uint32_t s = live[0];
#pragma unroll
            for (int j = 1; j < NW; j++) s |= live[j];
            return s != 0u;
        };
        unsigned open;  // lanes with a slot and a literal left
        while ((open = __ballot_sync(kFull, some() && pos < end)) != 0u) {
            // few clauses left, with much to read: the whole warp takes each
            if (__popc(open) <= kFewLanes && __ballot_sync(kFull, some() && pos + kFewChunks * 4 < end) == open) break;
            if (!some()) end = pos;  // nothing left to read
            const uint32_t b = pos & ~3u;
            uint4 after4 = chunk;
            if (b + 4 < end) after4 = ld_chunk(a.lits, b + 4);
            const uint32_t lit[4] = {chunk.x, chunk.y, chunk.z, chunk.w};
#pragma unroll
            for (int h = 0; h < 4; h += kPair) {
                Row<NW> r[kPair];
                bool on[kPair];
#pragma unroll
                for (int k = 0; k < kPair; k++) {
                    on[k] = b + h + k >= pos && b + h + k < end;
                    if (on[k] && some()) ld_narrow<NW>(a.state + (size_t) (lit[h + k] >> 1) * NW, r[k]);
                }
                if (h == 0 && fetch) {  // while the rows are read, the next task's first literals
                    if (pos1 < end1) ahead = ld_chunk(a.lits, pos1);
                    fetch = false;
                }
#pragma unroll
                for (int k = 0; k < kPair; k++) {
                    if (on[k]) {
                        const uint32_t neg = (lit[h + k] & 1u) - 1u;
#pragma unroll
                        for (int j = 0; j < NW; j++) apply_literal(r[k].v[2 * j], r[k].v[2 * j + 1], neg, all[j], live[j]);
                    }
                }
            }
            pos = b + 4;
            chunk = after4;
        }
        if (fetch && pos1 < end1) ahead = ld_chunk(a.lits, pos1);
        while (open) {  // the clauses left, one by one, 32 literals a step
            const int src = __ffs(open) - 1;
            open &= open - 1;
            const uint32_t e = __shfl_sync(kFull, end, src);
            uint32_t fa[NW], fl[NW], left = 0;
#pragma unroll
            for (int j = 0; j < NW; j++) {
                fa[j] = __shfl_sync(kFull, all[j], src);
                fl[j] = __shfl_sync(kFull, live[j], src);
                left |= fl[j];
            }
            for (uint32_t p = __shfl_sync(kFull, pos, src); p < e && left; p += 32) {
                Row<NW> r;
                uint32_t neg = 0;
                const bool on = p + lane < e;
                if (on) {
                    const uint32_t lit = (uint32_t) __ldg(a.lits + p + lane);
                    neg = (lit & 1u) - 1u;
                    ld_narrow<NW>(a.state + (size_t) (lit >> 1) * NW, r);
                }
                left = 0;
#pragma unroll
                for (int j = 0; j < NW; j++) {
                    uint32_t f = on ? (r.v[2 * j + 1] ^ neg) & r.v[2 * j] : ~0u, o = on ? ~r.v[2 * j] : 0u;
                    warp_runs(f, o);
                    fl[j] = (fa[j] & o) | (fl[j] & f);
                    fa[j] &= f;
                    left |= fl[j];
                }
            }
#pragma unroll
            for (int j = 0; j < NW; j++)
                if (lane == src) live[j] = fl[j];
        }
#pragma unroll
        for (int j = 0; j < NW; j++) {
            const unsigned bal = __ballot_sync(kFull, live[j] != 0u);
            if (bal) {
                if (nstaged + 32 > (uint32_t) kStage) {
                    flush_block_part(a, stage, nstaged);
                    nstaged = 0;
                }
                if (live[j]) {
                    gss_report rep;
                    rep.clause = __ldg(a.orig + c);
                    rep.word = j;
                    rep.mask = live[j];
                    rep.solver = (uint32_t) __ldg(a.solver_of_word + j);
                    stage[nstaged + __popc(bal & lanemask_lt())] = StagedReport{rep};
                }
                nstaged += __popc(bal);
            }
        }
        task = next;
        next = __shfl_sync(kFull, after, 0);
        c = c1;
        chunk = ahead;
        pos = pos1;
        end = end1;
    }
    if (nstaged) flush_block_part(a, stage, nstaged);
}

template <int NW, int MINB>
int launch_narrow_variant(const CheckArgs &a, uint32_t *work, cudaStream_t stream, int sm_count) {
    static std::atomic<int> known{0};
    int per_sm = 0;
    GSS_TRY((resident_blocks(check_narrow_kernel<NW, MINB>, known, per_sm)));
    const uint64_t n_tasks = ((uint64_t) scan_count(a) + 31) / 32;
    const uint64_t blocks = std::min<uint64_t>((uint64_t) sm_count * per_sm, (n_tasks + kWarps - 1) / kWarps);
    check_narrow_kernel<NW, MINB><<<(unsigned) blocks, kWarps * 32, 0, stream>>>(a, work);
    GSS_CUDA_TRY(cudaGetLastError());
    return GSS_OK;
}

}  // namespace

bool valid_narrow_variant(int words) { return words == 1 || words == 2 || words == 4; }

int launch_check_narrow(const CheckArgs &a, uint32_t *work, cudaStream_t stream, int sm_count) {
    if (a.n_clauses == 0 || a.n_blocks == 0 || scan_count(a) == 0) return GSS_OK;
    if (a.n_blocks == 1 && a.lpc == 1) return launch_narrow_variant<1, 4>(a, work, stream, sm_count);
    if (a.n_blocks == 1 && a.lpc == 2) return launch_narrow_variant<2, 4>(a, work, stream, sm_count);
    if (a.n_blocks == 1 && a.lpc == 4) return launch_narrow_variant<4, 4>(a, work, stream, sm_count);
    return set_error(GSS_ERR_INVALID, "no narrow kernel for %u blocks of %d words", a.n_blocks, a.lpc);
}

}  // namespace gss
