// Split of the time axis of the tensor-core adjoint into chunks, one CTA each.  Host code
// without CUDA types, so that the rule can be checked on its own.
#pragma once

#include <stdint.h>

namespace bb {

// Cost of F x chunks CTAs of `per` tiles: one CTA per SM (all of tensor memory), so the time
// is the number of waves times a chunk's tiles plus about one and a half tiles of start-up
// and final reduction, in half tiles.
inline uint64_t adjoint_chunk_cost(uint64_t F, uint64_t chunks, uint64_t per, uint64_t sms) {
    return (F * chunks + sms - 1) / sms * (2 * per + 3);
}

// Chunks per channel and tiles per chunk of least cost, the fewest chunks among equals.  Up to
// 64 chunks are tried (more change the last wave by less than a tile's share), and as many as
// give a block of one or two channels every SM: 32 antennas, 8 beams, one channel of 2^20
// samples 227 us in 147 chunks, 460 in 64.
inline void adjoint_chunks(uint64_t F, uint64_t ntiles, uint64_t sms, uint64_t& nch, uint64_t& tpc) {
    const uint64_t most = sms / F > 64 ? sms / F : 64;
    uint64_t best = ~0ull;
    for (uint64_t n = 1; n <= ntiles && n <= most; n++) {
        const uint64_t per = (ntiles + n - 1) / n, chunks = (ntiles + per - 1) / per;
        const uint64_t cost = adjoint_chunk_cost(F, chunks, per, sms);
        if (cost < best) {
            best = cost;
            nch = chunks;
            tpc = per;
        }
    }
}

}  // namespace bb
