// The chain kernel (beamform_tc.cuh) that splits its phasor images itself, for small
// blocks, and the rate-2 chain with direct voltage loads.
#include "beamform_tc.cuh"

namespace bb {
namespace {

template <int R, int MODE>
const void* pick(uint32_t logi) {
    switch (logi) {
        case 0: return reinterpret_cast<const void*>(bf_tc_kernel<R, 0, 4, MODE>);
        case 1: return reinterpret_cast<const void*>(bf_tc_kernel<R, 1, 4, MODE>);
        case 2: return reinterpret_cast<const void*>(bf_tc_kernel<R, 2, 4, MODE>);
        case 3: return reinterpret_cast<const void*>(bf_tc_kernel<R, 3, 4, MODE>);
        case 4: return reinterpret_cast<const void*>(bf_tc_kernel<R, 4, 4, MODE>);
        default: return reinterpret_cast<const void*>(bf_tc_kernel<R, 5, 4, MODE>);
    }
}

}  // namespace

const void* tc_self_kernel(uint64_t rate, uint64_t integration) {
    const uint32_t logi = tc_log2(integration);
    return rate == 1 ? pick<1, TC_SELF>(logi) : rate == 2 ? pick<2, TC_SELF>(logi) : pick<4, TC_SELF>(logi);
}

const void* tc_direct2_kernel(uint64_t integration) { return pick<2, TC_DIRECT2>(tc_log2(integration)); }

int tc_self_status_take(uint32_t* status) { return tc_status_take_here(status); }

}  // namespace bb
