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

// Writes a warp's staged records: one atomic reservation, then the records.
// streaming = cache-streaming stores (the records are read back by the host,
// not by the kernel: they need not displace state rows from L2).
__device__ __forceinline__ void flush_stage(gss_report *stage, uint32_t n, gss_report *out, uint32_t *counter,
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
__device__ __forceinline__ void scan_rows(const int32_t *__restrict__ lits, const uint2 *__restrict__ rows, uint32_t pos,
                                          uint32_t end, int sub, int gbase, uint32_t (&all)[WPL],
                                          uint32_t (&live)[WPL], Row<WPL> (&st)[G]) {
    constexpr int BW = WPL * LPC;
    while (true) {
        uint32_t some = live[0];
#pragma unroll
        for (int j = 1; j < WPL; j++) some |= live[j];
        if (!__any_sync(kFull, some != 0u && pos < end)) break;
        const int32_t chunk = (pos + sub < end) ? __ldg(lits + pos + sub) : 0;
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
