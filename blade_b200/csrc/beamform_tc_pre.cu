// The chain kernel (beamform_tc.cuh) for ModeB's order: channelizer before the beamformer.
#include "beamform_tc.cuh"

namespace bb {
namespace {

template <int R>
const void* pick(uint32_t logi) {
    switch (logi) {
        case 0: return reinterpret_cast<const void*>(bf_tc_kernel<R, 0, 4, TC_PRE>);
        case 1: return reinterpret_cast<const void*>(bf_tc_kernel<R, 1, 4, TC_PRE>);
        case 2: return reinterpret_cast<const void*>(bf_tc_kernel<R, 2, 4, TC_PRE>);
        case 3: return reinterpret_cast<const void*>(bf_tc_kernel<R, 3, 4, TC_PRE>);
        case 4: return reinterpret_cast<const void*>(bf_tc_kernel<R, 4, 4, TC_PRE>);
        default: return reinterpret_cast<const void*>(bf_tc_kernel<R, 5, 4, TC_PRE>);
    }
}

}  // namespace

const void* tc_pre_kernel(uint64_t rate, uint64_t integration) {
    return rate == 4 ? pick<4>(tc_log2(integration)) : pick<2>(tc_log2(integration));
}

int tc_pre_status_take(uint32_t* status) { return tc_status_take_here(status); }

}  // namespace bb
