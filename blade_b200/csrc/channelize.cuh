// Entry of the register-blocked power-of-two channelizer (fft_pow2.cu).
#pragma once

#include "common.cuh"

namespace bb {

// Whether channelize_pow2 runs this rate: a power of two from 32 to 4096.
inline bool channelize_pow2_applies(uint64_t rate) { return rate >= 32 && rate <= 4096 && (rate & (rate - 1)) == 0; }

// [A, F, T, P] CF32 (or CI8, P = 2) -> [A, F rate, T / rate, P] CF32, fftshifted;
// circular != 0 (P = 2): (X, Y) -> (X + iY, X - iY) on the way out.  The caller has
// checked the arguments; 16-byte aligned buffers (4 bytes for CI8 input).
int channelize_pow2(const void* in, bool ci8, float2* out, uint64_t A, uint64_t F, uint64_t T, uint64_t P,
                    uint64_t rate, int circular, cudaStream_t s);

}  // namespace bb
