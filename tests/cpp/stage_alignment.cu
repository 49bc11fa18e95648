// Compiles where the records that the kernels stage in shared memory lie on 16
// bytes by their type, as the 16-byte accesses of stage_record, flush_mapped
// and flush_stage need.
#include "check_rows.cuh"

template <typename A>
constexpr size_t second_alignment(void (*)(const gss::CheckArgs &, const A *, uint32_t)) {
    return alignof(A);
}
template <typename R, typename A, typename... B>
constexpr size_t target_alignment(R (*)(A *, B...)) {
    return alignof(A);
}

static_assert(target_alignment(gss::stage_record) >= 16, "stage_record");
static_assert(target_alignment(gss::flush_stage) >= 16, "flush_stage");
static_assert(second_alignment(gss::flush_mapped<true>) >= 16, "flush_mapped");
static_assert(second_alignment(gss::flush_mapped<false>) >= 16, "flush_mapped");
