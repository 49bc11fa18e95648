// Device code shared by the kernels that check a clause against 32-slot words
// laid out in rows (a group of lanes per clause, WPL consecutive words per
// lane): the row loads, the rule, and the staged report records.
#pragma once

#include "common.h"

namespace gss {

constexpr int kWarps = 8;     // warps per block
constexpr int kStage = 128;   // staged records per warp
constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// A report record in a warp's stage in shared memory: read and written 16
// bytes at a time, so the type says where it lies (gss_report itself has the
// alignment of its words).
struct alignas(16) StagedReport : gss_report {};
static_assert(sizeof(StagedReport) == sizeof(gss_report) && sizeof(gss_report) == sizeof(uint4), "a record is 16 bytes");

// Writes a warp's staged records: one atomic reservation, then the records.
// streaming = cache-streaming stores (the records are read back by the host,
// not by the kernel: they need not displace state rows from L2).
__device__ __forceinline__ void flush_stage(const StagedReport *stage, uint32_t n, gss_report *out, uint32_t *counter,
                                            uint32_t cap, int lane, bool streaming = false) {
    __syncwarp();
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(counter, n);
    base = __shfl_sync(kFull, base, 0);
    for (uint32_t i = lane; i < n; i += 32) {
        uint32_t idx = base + i;
        if (idx < cap) {
            if (streaming)
                __stcs(reinterpret_cast<int4 *>(out + idx), *reinterpret_cast<const int4 *>(stage + i));
            else
                out[idx] = stage[i];
        }
    }
    __syncwarp();
}

__device__ __forceinline__ int lane_id() {
    int l;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));
    return l;
}

// Flushes a warp's stage into its block's partition.
__device__ __forceinline__ void flush_block_part(const CheckArgs &a, const StagedReport *stage, uint32_t n) {
    const uint32_t part = blockIdx.x % a.n_parts;
    flush_stage(stage, n, a.out + (size_t) part * a.cap_per_part, a.counts + (size_t) part * a.count_stride,
                a.cap_per_part, lane_id());
}

// A record as the kernels stage it: the clause's position; flush_mapped turns
// it into the clause's id (or leaves it, without an id map) and adds the
// solver, 32 records at a time. WIDE: the queues lie on 16 bytes, as the
// engine's do, and a record is one store; else it is four.
__device__ __forceinline__ void stage_record(StagedReport *to, uint32_t c, uint32_t word, uint32_t mask) {
    *reinterpret_cast<uint4 *>(to) = make_uint4(c, word, mask, 0u);
}
template <bool WIDE = true>
__device__ __forceinline__ void flush_mapped(const CheckArgs &a, const StagedReport *stage, uint32_t n) {
    const int lane = lane_id();
    const uint32_t part = blockIdx.x % a.n_parts;
    __syncwarp();
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(a.counts + (size_t) part * a.count_stride, n);
    base = __shfl_sync(kFull, base, 0);
    gss_report *out = a.out + (size_t) part * a.cap_per_part;
    for (uint32_t i = lane; i < n; i += 32) {
        uint4 r = reinterpret_cast<const uint4 *>(stage)[i];  // {clause, word, mask, solver}
        if (a.orig) r.x = __ldg(a.orig + r.x);
        r.w = (uint32_t) __ldg(a.solver_of_word + r.y);
        if (base + i >= a.cap_per_part) continue;
        if (WIDE)
            reinterpret_cast<uint4 *>(out)[base + i] = r;
        else
            out[base + i] = gss_report{r.x, r.y, r.z, r.w};
    }
    __syncwarp();
}

// L2 policy of small tables that every warp gathers from: they keep their
// place. (L1::no_allocate without a policy marks a load evict-first in L2.)
__device__ __forceinline__ uint64_t policy_keep() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// The 16-byte chunk of literals that holds position `pos` (kClausePad literals
// after the last clause keep it inside the buffer).
__device__ __forceinline__ uint4 ld_chunk(const int32_t *lits, uint32_t pos) {
    uint4 v;
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(lits + (pos & ~3u)));
    return v;
}

// Combines two runs of literals: f = every literal false, o = one undefined
// and the rest false; the order does not matter.
__device__ __forceinline__ void merge_runs(uint32_t &f, uint32_t &o, uint32_t f2, uint32_t o2) {
    o = (f & o2) | (o & f2);
    f &= f2;
}

// A run of up to 32 literals, one per lane, over the whole warp; every lane
// gets the result.
__device__ __forceinline__ void warp_runs(uint32_t &f, uint32_t &o) {
#pragma unroll
    for (int d = 16; d; d >>= 1) {
        const uint32_t f2 = __shfl_xor_sync(kFull, f, d), o2 = __shfl_xor_sync(kFull, o, d);
        merge_runs(f, o, f2, o2);
    }
}

// A persistent kernel's next task, from its block's counter: kWorkCounters
// of them share the tasks in turn, so that warps side by side in time stay
// side by side in the database. (The block number is read where it is needed:
// kept from the start it would cost a register.)
__device__ __forceinline__ uint32_t task_from(uint32_t *work) {
    uint32_t b;
    asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(b));
    const uint32_t n = min(gridDim.x, kWorkCounters), mine = b % n;
    return n * atomicAdd(work + mine * kCountStride, 1u) + mine;
}

// Tasks of a persistent kernel: every warp starts with the task of its own
// number; the rest come from its block's counter, of kWorkCounters that share
// the tasks in turn, so that warps side by side in time stay side by side in
// the database.
struct TaskCounter {
    uint32_t *counter;
    uint32_t base, step;
    __device__ __forceinline__ explicit TaskCounter(uint32_t *work) {
        step = gridDim.x < 4 * kWorkCounters ? 1u : kWorkCounters;
        const uint32_t mine = blockIdx.x % step;
        counter = work + mine * kCountStride;
        base = gridDim.x * kWarps + mine;
    }
    __device__ __forceinline__ uint32_t first() const { return blockIdx.x * kWarps + (threadIdx.x >> 5); }
    // lane 0 gets a task's number (to be broadcast), the others 0
    __device__ __forceinline__ uint32_t take(int lane) const {
        return lane == 0 ? base + step * atomicAdd(counter, 1u) : 0u;
    }
};

// {isDef, isTrue} of WPL consecutive words
template <int WPL>
struct Row {
    uint32_t v[2 * WPL];
};

template <int WPL>
__device__ __forceinline__ void ld_row(const uint2 *p, Row<WPL> &r);
template <>
__device__ __forceinline__ void ld_row<1>(const uint2 *p, Row<1> &r) {
    asm("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(r.v[0]), "=r"(r.v[1]) : "l"(p));
}
template <>
__device__ __forceinline__ void ld_row<2>(const uint2 *p, Row<2> &r) {
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]) : "l"(p));
}
template <>
__device__ __forceinline__ void ld_row<4>(const uint2 *p, Row<4> &r) {
    asm("ld.global.nc.L1::no_allocate.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7])
        : "l"(p));
}

// The rule on one word, with the slots that can still report (`live`) and
// those of them with every literal false so far (`all`): a literal that is
// false keeps both, an undefined one leaves in `live` the slots that had all
// false, a true one drops the slot. neg = 0 for a negative literal, ~0 for a
// positive one. Three three-input logic operations a word (all is a subset
// of live).
__device__ __forceinline__ void apply_literal(uint32_t d, uint32_t t, uint32_t neg, uint32_t &all, uint32_t &live) {
    const uint32_t x = live & (t ^ neg);
    live = (d & x) | (~d & all);
    all = all & d & x;
}

// Scans the literals [pos, end) of each group's clause against its rows:
// LPC lanes per clause, WPL words per lane, G literals' rows in flight, until
// no group has a slot left. `st` may hold anything a lane read before (a lane
// that is done loads nothing, and its zero masks ignore the rows).
template <int WPL, int LPC, int G>
__device__ __forceinline__ void scan_rows(const CheckArgs &a, const uint2 *__restrict__ rows, uint32_t pos,
                                          uint32_t end, int sub, int gbase, uint32_t (&all)[WPL],
                                          uint32_t (&live)[WPL], Row<WPL> (&st)[G]) {
    constexpr int BW = WPL * LPC;
    while (true) {
        uint32_t some = live[0];
#pragma unroll
        for (int j = 1; j < WPL; j++) some |= live[j];
        if (!__any_sync(kFull, some != 0u && pos < end)) break;
        const int32_t chunk = (pos + sub < end) ? __ldg(a.lits + pos + sub) : 0;
        const int navail = (int) min((uint32_t) LPC, end > pos ? end - pos : 0u);
#pragma unroll 1
        for (int k0 = 0; k0 < LPC; k0 += G) {
            some = live[0];
#pragma unroll
            for (int j = 1; j < WPL; j++) some |= live[j];
            if (!__any_sync(kFull, some != 0u && k0 < navail)) break;
            uint32_t lit[G];
#pragma unroll
            for (int i = 0; i < G; i++) lit[i] = (uint32_t) __shfl_sync(kFull, chunk, gbase + k0 + i);
#pragma unroll
            for (int i = 0; i < G; i++) {
                if (some != 0u && k0 + i < navail) ld_row<WPL>(rows + (size_t) (lit[i] >> 1) * BW, st[i]);
            }
#pragma unroll
            for (int i = 0; i < G; i++) {
                if (k0 + i < navail) {
                    const uint32_t neg = (lit[i] & 1u) - 1u;
#pragma unroll
                    for (int j = 0; j < WPL; j++)
                        apply_literal(st[i].v[2 * j], st[i].v[2 * j + 1], neg, all[j], live[j]);
                }
            }
        }
        pos += LPC;
    }
}

}  // namespace gss
