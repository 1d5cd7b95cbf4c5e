// Streaming FP32 beamformer: the voltages stream through a private ring in shared
// memory, once per tile of NB beams.
//
//   y[b, f, t, p] = sum_a x[a, f, t, p] w[b, a, f, 0, p]
// (reference src/modules/beamformer/beamformer.cu:13-79), with the incoherent beam
// sum_a |x w[0]|^2 from the same loads (beamformer.cu:64-78), stored as beam
// voltages or, for Stokes-I and full-Stokes detection (detector.cu:7-51), as window
// sums that never leave the registers as voltages.
//
// A warp owns 32 NS consecutive samples of one channel (lane l: samples l + 32 s)
// and NB beams; a CTA's four warps take consecutive tiles, which may lie in up to
// four channels when the channels are short.  Each lane copies its own samples of the
// next kDepth - 1 antennas into shared memory (cp.async, read back by the same lane, so
// no barrier is involved) and reads each antenna's NB weights as broadcasts, which its
// NS samples share.
//
// Bound by the voltage read plus the FP32 pipe: 20 antennas x 192 channels x 8192
// samples, 8 beams: 122 us for 705 MB (5.8 TB/s); 130 when each copy computed its
// address from the antenna and tested its sample again.  Staging voltages and weights behind
// a barrier every two antennas took 288 us, two rounds of register loads 162 (128
// registers, 15 warps per SM waiting on memory).  Packed FP32x2 arithmetic is no
// faster; one sample per lane, four, a ring of four or of eight are 2 to 12 % slower, and
// so are several tiles per warp (spills) and a loop unrolled to the ring (128).  With
// detection (20 antennas x 6144 channels x 128 samples, 8 beams and the incoherent one,
// four products) 88 us against 470 us for the tiled kernel, the incoherent kernel and
// the detector.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace bb {

// Phasor element strides (float2 units) of beam, antenna, channel and
// polarisation: [B, A, F, 1, P] for ATA, (A, 1, 0, 0) for MeerKAT's [B, A] weights
// shared by every channel and polarisation.
struct PhLayout {
    uint64_t sb, sa, sf, sp;
};

struct StreamArgs {
    const void* in;
    const float2* ph;
    void* out;
    uint32_t B, A, F, T;
    uint32_t log_integ;  // detected outputs: window = 2^log_integ samples, at most 32
    uint32_t inc;        // 0 none, 1 sum of powers, 2 its square root
    uint32_t nbt;        // beam tiles, innermost in the grid (they read the same voltages)
    uint32_t ntt;        // time tiles per channel
    uint64_t tiles;      // F * ntt
    PhLayout lay;
};

struct StreamChunkArgs : StreamArgs {
    uint32_t chunk;  // antennas whose weights are in shared memory at a time
};

constexpr int kStreamWarps = 4;

enum { STREAM_CF32 = 0, STREAM_CI8 = 1 };

constexpr int kStreamDepth = 6;  // antennas in the ring

// Bytes of one sample (P polarisations) and its values.
template <int P, int IN>
struct StreamSample {
    static constexpr int kBytes = IN == STREAM_CI8 ? 4 : 8 * P;
    static_assert(IN == STREAM_CF32 || P == 2, "CI8 input is dual-polarisation");

    static __device__ __forceinline__ void copy(uint32_t dst, const void* in, uint64_t i) {
        const char* src = static_cast<const char*>(in) + i * kBytes;
        if constexpr (kBytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(kBytes) : "memory");
    }
    static __device__ __forceinline__ void read(const unsigned char* p, float2 (&v)[P]) {
        if constexpr (kBytes == 8) {
            v[0] = *reinterpret_cast<const float2*>(p);
        } else {
            const float4 q = kBytes == 16 ? *reinterpret_cast<const float4*>(p)
                                          : ci8_f4(*reinterpret_cast<const uint32_t*>(p));
            v[0] = make_float2(q.x, q.y);
            v[P - 1] = make_float2(q.z, q.w);
        }
    }
};

// OP = 0: beam voltages CF32 [B (+ 1), F, T, P]; OP = 1 or 4: detected products F32
// [B (+ 1), F, T / I, OP] (P = 2).
// CHUNKED: the antennas' weights do not fit beside enough CTAs per SM and pass through
// shared memory g.chunk antennas at a time (a barrier on either side of each gather); the
// plain kernel holds them all, and the loop over chunks would cost it registers (36 bytes
// of spills at eight beams and two samples).
template <int P, int NB, int NS, int IN, int OP, bool CHUNKED>
__global__ void __launch_bounds__(kStreamWarps * 32, NB == 8 && NS == 2 ? (CHUNKED ? 4 : 5) : 1)
    bf_stream_kernel(const std::conditional_t<CHUNKED, StreamChunkArgs, StreamArgs> g) {
    using Sample = StreamSample<P, IN>;
    constexpr uint32_t kThreads = kStreamWarps * 32, kSlot = kThreads * Sample::kBytes;
    extern __shared__ __align__(16) unsigned char stream_smem_raw[];  // ring [kStreamDepth][NS][thread], weights
    float2* ws = reinterpret_cast<float2*>(stream_smem_raw + kStreamDepth * NS * kSlot);  // [channel][chunk][NB][P]
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t blk = blockIdx.x / g.nbt, b0 = (blockIdx.x - blk * g.nbt) * NB;
    const uint64_t first = (uint64_t)blk * kStreamWarps;
    const uint64_t last = min(first + kStreamWarps, g.tiles) - 1;
    const uint32_t f0 = (uint32_t)(first / g.ntt), nch = (uint32_t)(last / g.ntt) - f0 + 1;
    const uint64_t tile = first + warp;
    const bool active = tile <= last;
    const uint32_t f = active ? (uint32_t)(tile / g.ntt) : f0;
    const uint32_t t0 = (uint32_t)(tile - (uint64_t)f * g.ntt) * (32 * NS) + lane;
    const uint64_t astride = (uint64_t)g.F * g.T, x0 = (uint64_t)f * g.T + t0;
    unsigned char* mine = stream_smem_raw + tid * Sample::kBytes;
    const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(mine));
    // antenna a, at src, into the ring position at `dst` (an empty group past the last
    // antenna keeps the count)
    bool in_row[NS];
#pragma unroll
    for (int s = 0; s < NS; s++) in_row[s] = active && t0 + 32 * s < g.T;
    const char* src = static_cast<const char*>(g.in) + x0 * Sample::kBytes;
    auto fetch = [&](uint32_t a, uint32_t dst) {
#pragma unroll
        for (int s = 0; s < NS; s++)
            if (in_row[s] && a < g.A) Sample::copy(dst + s * kSlot, src, 32 * s);
        src += astride * Sample::kBytes;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (uint32_t a = 0; a < kStreamDepth - 1; a++)  // on their way while the weights are gathered
        fetch(a, ring + a * NS * kSlot);
    // weight r of this CTA's channels and of the antennas held from a0 on, padded beams zero
    uint32_t held = g.A;
    if constexpr (CHUNKED) held = g.chunk;
    auto gather = [&](uint32_t r, uint32_t a0) {
        const uint32_t a = r / NB, j = r - a * NB;
        const bool ok = b0 + j < g.B;
        const float2* wsrc = g.ph + (b0 + j) * g.lay.sb + (a0 + a) * g.lay.sa + (uint64_t)f0 * g.lay.sf;
        for (uint32_t c = 0; c < nch; c++)
#pragma unroll
            for (int p = 0; p < P; p++)
                ws[((c * held + a) * NB + j) * P + p] = ok ? __ldg(wsrc + c * g.lay.sf + p * g.lay.sp) : make_float2(0.f, 0.f);
    };
    if constexpr (!CHUNKED) {
        for (uint32_t r = tid; r < NB * g.A; r += kThreads) gather(r, 0);
        __syncthreads();
        if (!active) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            return;
        }
    }
    const float2* wa = ws + (size_t)(f - f0) * held * NB * P;
    const bool inc = g.inc != 0 && b0 == 0;

    float2 acc[NB][NS][P];
    float pw[NS][P];
#pragma unroll
    for (int s = 0; s < NS; s++)
#pragma unroll
        for (int p = 0; p < P; p++) {
            pw[s][p] = 0.f;
#pragma unroll
            for (int j = 0; j < NB; j++) acc[j][s][p] = make_float2(0.f, 0.f);
        }
    uint32_t at = 0, to = (kStreamDepth - 1) * NS * kSlot;
    auto antenna = [&](uint32_t a) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStreamDepth - 2) : "memory");
        float2 x[NS][P];
#pragma unroll
        for (int s = 0; s < NS; s++) Sample::read(mine + at + s * kSlot, x[s]);
        fetch(a + kStreamDepth - 1, ring + to);
        to = at;
        at += NS * kSlot;
        if (at == kStreamDepth * NS * kSlot) at = 0;
#pragma unroll
        for (int j = 0; j < NB; j++) {
            float2 w[P];
            if constexpr (P == 2) {
                const float4 q = *reinterpret_cast<const float4*>(wa + j * P);
                w[0] = make_float2(q.x, q.y);
                w[1] = make_float2(q.z, q.w);
            } else {
                w[0] = wa[j];
            }
#pragma unroll
            for (int s = 0; s < NS; s++)
#pragma unroll
                for (int p = 0; p < P; p++) {
                    const float2 xv = x[s][p];
                    acc[j][s][p].x = fmaf(xv.x, w[p].x, fmaf(-xv.y, w[p].y, acc[j][s][p].x));
                    acc[j][s][p].y = fmaf(xv.x, w[p].y, fmaf(xv.y, w[p].x, acc[j][s][p].y));
                    if (j == 0 && inc) {
                        const float re = xv.x * w[p].x - xv.y * w[p].y, im = xv.x * w[p].y + xv.y * w[p].x;
                        pw[s][p] += re * re + im * im;
                    }
                }
        }
        wa += NB * P;
    };
    if constexpr (!CHUNKED) {
#pragma unroll 1
        for (uint32_t a = 0; a < g.A; a++) antenna(a);
    } else {
#pragma unroll 1
        for (uint32_t a0 = 0; a0 < g.A; a0 += held) {
            const uint32_t a1 = min(a0 + held, g.A);
            if (a0) __syncthreads();  // every warp has read the chunk before
            for (uint32_t r = tid; r < NB * (a1 - a0); r += kThreads) gather(r, a0);
            __syncthreads();
            if (!active) continue;
            wa = ws + (size_t)(f - f0) * held * NB * P;
#pragma unroll 1
            for (uint32_t a = a0; a < a1; a++) antenna(a);
        }
        if (!active) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            return;
        }
    }

    if constexpr (OP == 0) {
        float2* out = static_cast<float2*>(g.out);
#pragma unroll
        for (int s = 0; s < NS; s++) {
            if (t0 + 32 * s >= g.T) continue;
#pragma unroll
            for (int j = 0; j < NB; j++) {
                if (b0 + j >= g.B) continue;
                float2* o = out + ((b0 + j) * astride + x0 + 32 * s) * P;
                if constexpr (P == 2) stg_f4(o, make_float4(acc[j][s][0].x, acc[j][s][0].y, acc[j][s][1].x, acc[j][s][1].y));
                else o[0] = acc[j][s][0];
            }
            if (inc) {
                float2* o = out + (g.B * astride + x0 + 32 * s) * P;
#pragma unroll
                for (int p = 0; p < P; p++) o[p] = make_float2(g.inc == 2 ? sqrtf(pw[s][p]) : pw[s][p], 0.f);
            }
        }
    } else if constexpr (P == 2) {
        float* out = static_cast<float*>(g.out);
        const uint32_t I = 1u << g.log_integ, U = g.T >> g.log_integ;
        auto emit = [&](uint32_t row, int s, float2 x, float2 y) {
            float v[OP];
            if constexpr (OP == 1) {
                v[0] = x.x * x.x + x.y * x.y + (y.x * y.x + y.y * y.y);
            } else {
                v[0] = x.x * x.x + x.y * x.y;
                v[1] = y.x * y.x + y.y * y.y;
                v[2] = x.x * y.x + x.y * y.y;  // Re x conj(y)
                v[3] = x.y * y.x - x.x * y.y;  // Im x conj(y)
            }
            const bool stored = t0 + 32 * s < g.T;
            float* d = out + (((uint64_t)row * g.F + f) * U + ((t0 + 32 * s) >> g.log_integ)) * OP;
            if constexpr (OP == 4) {
                // windows of four and more: two halving exchanges leave one product per lane
                if (I >= 4) {
                    const bool hi = lane & 1u, up = lane & 2u;
                    const float s0 = hi ? v[0] : v[2], s1 = hi ? v[1] : v[3];
                    float k0 = hi ? v[2] : v[0], k1 = hi ? v[3] : v[1];
                    k0 += __shfl_xor_sync(0xffffffffu, s0, 1);
                    k1 += __shfl_xor_sync(0xffffffffu, s1, 1);
                    float k = (up ? k1 : k0) + __shfl_xor_sync(0xffffffffu, up ? k0 : k1, 2);
                    for (uint32_t o = 4; o < I; o <<= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
                    if (stored && (lane & (I - 1u)) < 4) d[2 * (lane & 1u) + ((lane >> 1) & 1u)] = k;
                    return;
                }
            }
            for (uint32_t o = 1; o < I; o <<= 1)
#pragma unroll
                for (int q = 0; q < OP; q++) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
            if ((lane & (I - 1u)) == 0 && stored) {
                if constexpr (OP == 4) stg_f4(d, make_float4(v[0], v[1], v[2], v[3]));
                else d[0] = v[0];
            }
        };
#pragma unroll
        for (int s = 0; s < NS; s++) {
#pragma unroll
            for (int j = 0; j < NB; j++)
                if (b0 + j < g.B) emit(b0 + j, s, acc[j][s][0], acc[j][s][1]);
            if (inc) emit(g.B, s, make_float2(g.inc == 2 ? sqrtf(pw[s][0]) : pw[s][0], 0.f),
                          make_float2(g.inc == 2 ? sqrtf(pw[s][1]) : pw[s][1], 0.f));
        }
    }
}

// Channels that a CTA's consecutive tiles (from a multiple of kStreamWarps on) can touch.
inline uint64_t stream_channels(uint64_t ntt, uint64_t F) {
    const uint64_t nch = ntt == 1 ? kStreamWarps : ntt % kStreamWarps == 0 ? 1 : 2;
    return nch < F ? nch : F;
}

// Beams and samples per thread.  Eight beams share each voltage load and two samples
// each weight read as long as every SM still gets eight warps; below that, fewer, so
// that a small block spreads over the SMs (20 antennas x 96 channels x 256 samples,
// 8 beams with the incoherent beam: 8.5 us against 17.3 us for one thread per
// output).  False: more CTAs than a grid holds.
inline bool stream_shape(uint64_t B, uint64_t F, uint64_t T, uint32_t& nb, uint32_t& ns) {
    nb = B > 4 ? 8 : B > 2 ? 4 : (uint32_t)B;
    ns = 2;
    const uint64_t want = 8ull * sm_count();
    if (F * ceil_div(T, 64) * ceil_div(B, nb) < want) ns = 1;
    while (nb > 2 && F * ceil_div(T, 32 * ns) * ceil_div(B, nb) < want) nb /= 2;
    return ceil_div(F * ceil_div(T, 32 * ns), kStreamWarps) * ceil_div(B, nb) < (1ull << 31);
}

template <int P, int NB, int NS, int IN, int OP>
int launch_stream(StreamArgs g, cudaStream_t s) {
    g.ntt = (uint32_t)ceil_div(g.T, 32 * NS);
    g.tiles = (uint64_t)g.F * g.ntt;
    g.nbt = (uint32_t)ceil_div(g.B, NB);
    const uint64_t ctas = ceil_div(g.tiles, kStreamWarps) * g.nbt, per_sm = ceil_div(ctas, (uint64_t)sm_count());
    const size_t ring = kStreamDepth * NS * kStreamWarps * 32 * StreamSample<P, IN>::kBytes;
    const size_t antenna = stream_channels(g.ntt, g.F) * NB * P * sizeof(float2);
    // Weights beside the ring so that the CTAs an SM gets, four at most, are resident at once:
    // held in whole they left two CTAs at 512 antennas and one from 768 on (eight beams, two
    // polarisations).  768 antennas x 170 channels x 1024 samples, 16 beams: 2010 us held in
    // whole, 957 in chunks (1357 for 4 x 4 register tiles staged behind a barrier); 2048 antennas,
    // 64 channels, 64 beams: 7920, 3430 (and 4057).
    const size_t room = 224 * 1024 / (per_sm < 4 ? per_sm : 4) - ring;
    const unsigned grid = (unsigned)ctas, block = kStreamWarps * 32;
    if (g.A * antenna <= room) {
        const auto fn = bf_stream_kernel<P, NB, NS, IN, OP, false>;
        const size_t smem = ring + g.A * antenna;
        if (int rc = ensure_smem(reinterpret_cast<const void*>(fn), smem)) return rc;
        fn<<<grid, block, smem, s>>>(g);
        return BLADE_SUCCESS;
    }
    StreamChunkArgs h;
    static_cast<StreamArgs&>(h) = g;
    h.chunk = (uint32_t)(room / antenna);
    const auto fn = bf_stream_kernel<P, NB, NS, IN, OP, true>;
    const size_t smem = ring + h.chunk * antenna;
    if (int rc = ensure_smem(reinterpret_cast<const void*>(fn), smem)) return rc;
    fn<<<grid, block, smem, s>>>(h);
    return BLADE_SUCCESS;
}

}  // namespace bb
