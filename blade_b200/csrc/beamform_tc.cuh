// Tensor-core (tcgen05 / TMEM) beamform + channelize + detect chain for sm_100a.
//
// Computes, for CI8 voltages x[A, F, T, 2] and phasors w[B, A, F, 1, 2],
//   y[b, f, t, p]            = sum_a x[a, f, t, p] w[b, a, f, 0, p]
//   Y[b, f*R + k, s, p]      = fftshift(FFT_R(y[b, f, sR:(s+1)R, p]))[k],  R in {1, 2, 4}
//   out[b, f*R + k, u, 0]    = sum_{s in window u of I spectra} sum_p |Y[b, f*R + k, s, p]|^2
// i.e. the reference chain Cast -> Beamformer::ATA -> Channelizer -> Detector
// (src/modules/cast/cast.cu, src/modules/beamformer/beamformer.cu:13-62,
// src/modules/channelizer/base.cc + channelizer.cu, src/modules/detector/detector.cu:34-51),
// fused so that only the Stokes-I output reaches HBM.
//
// Numerics.  CI8 values are exact in FP16.  The rate-R DFT with the (-1)^t
// fftshift pre-multiply has coefficients in {+-1, +-i}, so it is applied to the
// integer voltages while the MMA operand is built (values <= 4 * 128, still
// exact in FP16): Y = X_R . w with X_R exact.  Each phasor component is split into
// FP16 hi = rn(w) and lo = rn(w - hi) (about 22 significant bits); both products
// accumulate in FP32 in tensor memory.
//
// GEMM mapping per (channel f, polarisation p): D[m, n] = sum_k A[m, k] B[n, k]
// with m = one of 128 rows of a tile (R consecutive samples per spectrum,
// row = k * (128/R) + spectrum), k = [Xr of KA antennas | Xi of KA antennas]
// (KA = 32 or 64, antennas zero-padded), and the complex product embedded in reals
// (NB = beams of a 64-beam chunk padded to 16):
//   Re y = Xr Wr - Xi Wi,   Im y = Xr Wi + Xi Wr
// Three phasor-image layouts, all K-major with the 128-byte swizzle:
//   NB <= 32 ("stacked"): rows [hi Re | hi Im | lo Re | lo Im] x NB, K = 2 KA, so
//            one MMA per k-step with N = 4 NB gives both hi and lo products;
//   KA = 64: blocks [-Wi | Wr | Wi] per (p, hi/lo); the Xr k-steps read the window
//            [Wr | Wi], the Xi k-steps [-Wi | Wr] (N = 2 NB);
//   KA = 32: one embedded block of 2 NB rows per (p, hi/lo), K = 2 KA.
// Each 64-element K block of an operand is 128 rows x 128 bytes (16 KB).
//
// CTA organisation (persistent, one CTA per SM, 15 warps):
//   warp 0      TMEM allocation; lane 0 issues tcgen05.mma and commits (MMA
//               issuer 0; warp 14 is issuer 1 when two issuers apply)
//   warp 1      loader: the per-channel phasor image (one bulk copy) and the raw
//               CI8 tiles (one 3-D TMA tensor load per tile: 128 samples x 1
//               channel x A antennas) into a ring of raw stages
//   warps 2-5   epilogue: tcgen05.ld of the accumulators, |.|^2 over both
//               polarisations, window sums with lane shuffles, Stokes-I stores
//   warps 6-13  operand build from the raw ring: DFT, exact int8 -> FP16
//               conversion, swizzled stores; both polarisations of a tile in one
//               pass when the operand ring holds at least two tiles
// Pipelines (full/empty mbarrier pairs): raw stages, operand stages (one per tile
// and polarisation), up to four TMEM accumulator buffers, the phasor image.  Every
// wait is bounded (clock budget plus a shared abort flag) and sleeps on the
// mbarrier rather than spinning; on expiry the kernel records a status word,
// drains its own MMAs and copies, frees TMEM and returns.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>

#include <string.h>

#include <mutex>

#include "autotune.cuh"
#include "common.cuh"
#include "tc_ptx.cuh"

namespace bb {

namespace {

// Non-zero after a bounded wait expired in this source file's tensor-core kernels (read
// and cleared by blade_device_status()).
__device__ unsigned int g_tc_status = 0;

// Reads and clears it.
inline int tc_status_take_here(uint32_t* status) {
    unsigned int v = 0, zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(v));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(zero));
    if (e != cudaSuccess) return check_cuda(e, "blade_device_status");
    *status = v;
    return BLADE_SUCCESS;
}

// What an instantiation of the chain kernel adds to the plain one: each is a kernel of
// its own (and the added ones are built in source files of their own), because code
// that a shape never runs still moves the schedule of the code it does: 4 to 30 % on
// the 28-antenna rate-2 block.
enum { TC_BASE = 0, TC_PRE = 1, TC_SELF = 2, TC_DIRECT2 = 3 };

using namespace tc;

constexpr int kM = 128;  // tile rows
constexpr int kConvWarps = 8;
constexpr int kEpiWarps = 4;  // one or two per TMEM lane quarter
constexpr int kEpiGroups = kEpiWarps / 4;  // warps per lane quarter, each a share of the beams
constexpr int kWarps = 3 + kEpiWarps + kConvWarps;  // + MMA issuer 0, loader, MMA issuer 1
constexpr int kThreads = kWarps * 32;               // 480
constexpr int kMaxNB = 64;
constexpr int kMaxKA = 64;
constexpr int kMaxAcc = 4;   // TMEM accumulator buffers
constexpr int kMaxStages = 8;  // operand stages and raw stages, each
constexpr long long kWaitBudget = 4000000000ll;  // cycles (~2 s) before a wait gives up

struct TcArgs {
    const uint8_t* in;    // CI8 [A, F, T, 2]
    const uint8_t* plan;  // phasor images, one per channel, img_bytes each
    float* out;           // [beams, F*R, U]
    uint32_t A, F, T, beams, U;
    uint32_t NB, KA, a_stages, r_stages, stacked;
    uint32_t img_bytes, raw_bytes, tiles_per_ch;
    uint32_t raw_tiles, raw_row;  // tiles per raw stage (1, 2 or 4) and its antenna row stride (raw_tiles * 512)
    uint64_t total_tiles;
    uint32_t pdl;  // launched as a programmatic dependent of the phasor split: wait for it before the image
    uint32_t direct;  // CI8 at R = 1 or 2 without a raw ring: converter threads load the voltages themselves
    uint32_t transposed;  // outputs along TMEM lanes, samples along columns (64-beam chunks, rate 1, I = 8 or 16)
    const float2* ph;      // SELF: the chunk's phasors [beams][A][F][2]
    uint8_t* plan_out;     // SELF: where the images go besides
    uint32_t segs, seg_tiles;  // SELF: CTAs per channel, tiles per CTA
    uint32_t circ;  // PRE: (X, Y) -> (X + iY, X - iY) while the operand is built
};

__device__ __forceinline__ uint32_t cvt_pair(uint32_t v) {
    // bytes 0 and 2 of v hold two int8 values; returns them as an exact half2.
    uint32_t x = (v & 0x00FF00FFu) ^ 0x64806480u;  // 1024 + (b + 128) in each half
    half2 h = *reinterpret_cast<half2*>(&x);
    const half2 bias = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));  // 1152
    h = __hsub2(h, bias);
    return *reinterpret_cast<uint32_t*>(&h);
}

// One sample word [p0 re, p0 im, p1 re, p1 im] -> half2 (re, im) of polarisation p.
__device__ __forceinline__ half2 sample_h2(uint32_t w, int p) {
    uint32_t v = __byte_perm(w, 0, p == 0 ? 0x0100 : 0x0302);
    uint32_t r = cvt_pair(v);
    return *reinterpret_cast<half2*>(&r);
}

__device__ __forceinline__ uint32_t h2u(half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ half2 u2h(uint32_t u) { return *reinterpret_cast<half2*>(&u); }

// Address of K element k_total (a multiple of 4) of row `row` in one
// polarisation's operand: Xr occupies k_total in [0, KA), Xi [KA, 2 KA); every
// 64 K elements form one 128-row x 128-byte swizzled block of 16 KB.
__device__ __forceinline__ uint32_t op_off(uint32_t row, uint32_t k_total) {
    return (k_total >> 6) * 16384u + sw128_off(row, (k_total >> 3) & 7u) + ((k_total & 4u) << 1);
}

__device__ __forceinline__ void record_abort(volatile int* abort, unsigned code) {
    *abort = 1;
    atomicCAS(&g_tc_status, 0u, code);
}

// rate-4 spectrum of one antenna and polarisation from its 4 sample words:
// Z[k] = sum_j (-1)^j x_j e^{-2 pi i j k / 4}, exact in FP16 (|Z| <= 512).
__device__ __forceinline__ void dft4_h2(uint4 v, int p, half2 (&Z)[4]) {
    const half2 x0 = sample_h2(v.x, p), x1 = sample_h2(v.y, p), x2 = sample_h2(v.z, p), x3 = sample_h2(v.w, p);
    const half2 e02 = __hadd2(x0, x2), d02 = __hsub2(x0, x2);
    const half2 e13 = __hadd2(x1, x3), d13 = __hsub2(x1, x3);
    const half2 id13 = __hmul2(__lowhigh2highlow(d13), __halves2half2(__float2half(-1.f), __float2half(1.f)));
    Z[0] = __hsub2(e02, e13);  // x0 - x1 + x2 - x3
    Z[1] = __hadd2(d02, id13); // x0 + i x1 - x2 - i x3
    Z[2] = __hadd2(e02, e13);  // x0 + x1 + x2 + x3
    Z[3] = __hsub2(d02, id13); // x0 - i x1 - x2 + i x3
}

// R = 1 operand chunk: 8 antennas of one sample -> (re, im) chunks of polarisation p.
__device__ __forceinline__ void r1_chunks(const uint32_t (&w)[8], int p, uint4& vr, uint4& vi) {
    const uint32_t sre = p ? 0x0602u : 0x0400u, sim = p ? 0x0703u : 0x0501u;
    vr.x = cvt_pair(__byte_perm(w[0], w[1], sre));
    vr.y = cvt_pair(__byte_perm(w[2], w[3], sre));
    vr.z = cvt_pair(__byte_perm(w[4], w[5], sre));
    vr.w = cvt_pair(__byte_perm(w[6], w[7], sre));
    vi.x = cvt_pair(__byte_perm(w[0], w[1], sim));
    vi.y = cvt_pair(__byte_perm(w[2], w[3], sim));
    vi.z = cvt_pair(__byte_perm(w[4], w[5], sim));
    vi.w = cvt_pair(__byte_perm(w[6], w[7], sim));
}

// Builds the operand rows of polarisation p for one tile from the raw stage in
// shared memory (antenna-major rows of rrow bytes; `raw` points at this tile's
// 128 samples x 4 bytes in the first row).
// Row = k * (128 / R) + spectrum.  Consecutive lanes take consecutive rows, so
// every 16-byte store of a warp lands in a distinct bank group of the swizzle.
template <int R>
__device__ __forceinline__ void build_operand(const uint8_t* raw, uint32_t rrow, uint8_t* op, uint32_t A, uint32_t KA,
                                              int p, uint32_t ct) {
    constexpr uint32_t kStride = kConvWarps * 32;
    if constexpr (R == 1) {
        const uint32_t ntasks = kM * (KA / 8);
        // Two tasks per pass: both tasks' shared-memory loads are in flight together.
        for (uint32_t t0 = ct; t0 < ntasks; t0 += 2 * kStride) {
            const uint32_t t1 = t0 + kStride;
            const bool has1 = t1 < ntasks;
            const uint32_t s0 = t0 % kM, g0 = t0 / kM, s1 = t1 % kM, g1 = t1 / kM;
            uint32_t w0[8], w1[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t a0 = g0 * 8 + i, a1 = g1 * 8 + i;
                w0[i] = a0 < A ? *reinterpret_cast<const uint32_t*>(raw + a0 * rrow + s0 * 4) : 0u;
                w1[i] = (has1 && a1 < A) ? *reinterpret_cast<const uint32_t*>(raw + a1 * rrow + s1 * 4) : 0u;
            }
            uint4 vr, vi;
            r1_chunks(w0, p, vr, vi);
            *reinterpret_cast<uint4*>(op + op_off(s0, g0 * 8)) = vr;
            *reinterpret_cast<uint4*>(op + op_off(s0, KA + g0 * 8)) = vi;
            if (has1) {
                r1_chunks(w1, p, vr, vi);
                *reinterpret_cast<uint4*>(op + op_off(s1, g1 * 8)) = vr;
                *reinterpret_cast<uint4*>(op + op_off(s1, KA + g1 * 8)) = vi;
            }
        }
    } else if constexpr (R == 2) {
        const uint32_t ntasks = (kM / 2) * (KA / 8);
        for (uint32_t task = ct; task < ntasks; task += kStride) {
            const uint32_t s = task % (kM / 2), grp = task / (kM / 2);
            uint2 v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t a = grp * 8 + i;
                v[i] = a < A ? *reinterpret_cast<const uint2*>(raw + a * rrow + s * 8) : make_uint2(0u, 0u);
            }
            half2 Z0[8], Z1[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const half2 x0 = sample_h2(v[i].x, p), x1 = sample_h2(v[i].y, p);
                Z0[i] = __hsub2(x0, x1);  // k = 0: x0 - x1
                Z1[i] = __hadd2(x0, x1);  // k = 1: x0 + x1
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const half2* Z = k ? Z1 : Z0;
                uint4 vr, vi;
                vr.x = __byte_perm(h2u(Z[0]), h2u(Z[1]), 0x5410);
                vr.y = __byte_perm(h2u(Z[2]), h2u(Z[3]), 0x5410);
                vr.z = __byte_perm(h2u(Z[4]), h2u(Z[5]), 0x5410);
                vr.w = __byte_perm(h2u(Z[6]), h2u(Z[7]), 0x5410);
                vi.x = __byte_perm(h2u(Z[0]), h2u(Z[1]), 0x7632);
                vi.y = __byte_perm(h2u(Z[2]), h2u(Z[3]), 0x7632);
                vi.z = __byte_perm(h2u(Z[4]), h2u(Z[5]), 0x7632);
                vi.w = __byte_perm(h2u(Z[6]), h2u(Z[7]), 0x7632);
                const uint32_t row = k * (kM / 2) + s;
                *reinterpret_cast<uint4*>(op + op_off(row, grp * 8)) = vr;
                *reinterpret_cast<uint4*>(op + op_off(row, KA + grp * 8)) = vi;
            }
        }
    } else {
        // R == 4: a task is one spectrum of 4 antennas (half a K chunk, 8-byte stores).
        const uint32_t ntasks = (kM / 4) * (KA / 4);
        for (uint32_t task = ct; task < ntasks; task += kStride) {
            const uint32_t s = task % (kM / 4), g4 = task / (kM / 4);
            uint4 v[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t a = g4 * 4 + i;
                v[i] = a < A ? *reinterpret_cast<const uint4*>(raw + a * rrow + s * 16) : make_uint4(0u, 0u, 0u, 0u);
            }
            half2 Z[4][4];
#pragma unroll
            for (int i = 0; i < 4; i++) dft4_h2(v[i], p, Z[i]);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                uint2 vr, vi;
                vr.x = __byte_perm(h2u(Z[0][k]), h2u(Z[1][k]), 0x5410);
                vr.y = __byte_perm(h2u(Z[2][k]), h2u(Z[3][k]), 0x5410);
                vi.x = __byte_perm(h2u(Z[0][k]), h2u(Z[1][k]), 0x7632);
                vi.y = __byte_perm(h2u(Z[2][k]), h2u(Z[3][k]), 0x7632);
                const uint32_t row = k * (kM / 4) + s;
                *reinterpret_cast<uint2*>(op + op_off(row, g4 * 4)) = vr;
                *reinterpret_cast<uint2*>(op + op_off(row, KA + g4 * 4)) = vi;
            }
        }
    }
}

// R = 4, both polarisations in one pass.  Each sample word is split into two
// half2 words with the polarisations in the two halves, RE = (p0 re, p1 re) and
// IM = (p0 im, p1 im), read exactly as 1024 + (x + 128) = 1152 + x through the
// 0x64 exponent byte (one XOR of the sign bits, two byte permutes).  The DFT then
// runs in FP16 on the FMA pipe (the integer pipe issues at half rate): every
// intermediate is an integer of magnitude < 2048, so all of it is exact, and the
// 1152 biases cancel in differences or are removed together (x0 + x2 =
// ((1024 + u0) - 2304) + (1024 + u2) with both steps exact).  A warp covers 16
// spectra x 8 antennas (two 4-antenna groups): lanes 0-7 and 8-15 write the two
// 8-byte halves of one 16-byte chunk for 8 rows with distinct swizzle slots, lanes
// 16-31 the next 8 rows, so each 8-byte store is two conflict-free wavefronts.
// Row k * 32 + s of an operand sits 4096 * k bytes after row s (the swizzle phase
// depends on s only), so a task's addresses are fixed offsets computed once.
struct R4Task {
    uint32_t raw_off;  // a0 * rrow + s * 16 in the raw stage
    uint32_t o_r, o_i; // operand offsets of (row s, K = a0) and (row s, K = KA + a0)
    uint32_t nvalid;   // antennas a0 .. a0 + nvalid - 1 exist (0..4)
};

__device__ __forceinline__ R4Task r4_task(uint32_t wt, uint32_t lane, uint32_t A, uint32_t KA, uint32_t rrow) {
    const uint32_t c = wt >> 1;
    const uint32_t s = (wt & 1u) * 16u + (lane & 7u) + ((lane >> 4) << 3);
    const uint32_t a0 = (2u * c + ((lane >> 3) & 1u)) * 4u;
    R4Task t;
    t.raw_off = a0 * rrow + s * 16u;
    t.o_r = op_off(s, a0);
    t.o_i = op_off(s, KA + a0);
    t.nvalid = a0 < A ? min(4u, A - a0) : 0u;
    return t;
}

// Circular basis of one value of both polarisations, halves = (pol 0, pol 1):
// (X + iY, X - iY), integers of magnitude <= 1024 here, exact in FP16.
__device__ __forceinline__ void circular_h2(half2& re, half2& im) {
    const half2 mp = __halves2half2(__float2half(-1.f), __float2half(1.f));
    const half2 pm = __halves2half2(__float2half(1.f), __float2half(-1.f));
    const half2 xr = __low2half2(re), yr = __high2half2(re), xi = __low2half2(im), yi = __high2half2(im);
    re = __hfma2(yi, mp, xr);
    im = __hfma2(yr, pm, xi);
}

// PRE = true: with g.circ the polarisations are rotated after the transform.
template <bool PRE>
__device__ __forceinline__ void r4_pair_task(const uint8_t* raw, uint32_t rrow, uint8_t* op0, uint8_t* op1,
                                             const R4Task& t, uint32_t circ) {
    const half2 h2304 = __halves2half2(__ushort_as_half(0x6880), __ushort_as_half(0x6880));  // 2304
    uint2 out_r[2][4], out_i[2][4];  // [pol][k]
    if (t.nvalid) {
        half2 zr[4][4], zi[4][4];  // [antenna][k], halves = (pol 0, pol 1)
        const uint8_t* src = raw + t.raw_off;
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            const uint4 v = i < t.nvalid ? *reinterpret_cast<const uint4*>(src + i * rrow) : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t w[4] = {v.x ^ 0x80808080u, v.y ^ 0x80808080u, v.z ^ 0x80808080u, v.w ^ 0x80808080u};
            half2 re[4], im[4];  // 1152 + x
#pragma unroll
            for (int j = 0; j < 4; j++) {
                re[j] = u2h(__byte_perm(w[j], 0x64646464u, 0x4240));
                im[j] = u2h(__byte_perm(w[j], 0x64646464u, 0x4341));
            }
            const half2 aR = __hadd2(__hsub2(re[0], h2304), re[2]);  // x0 + x2
            const half2 bR = __hadd2(__hsub2(re[1], h2304), re[3]);  // x1 + x3
            const half2 cR = __hsub2(re[0], re[2]), dR = __hsub2(re[1], re[3]);
            const half2 aI = __hadd2(__hsub2(im[0], h2304), im[2]);
            const half2 bI = __hadd2(__hsub2(im[1], h2304), im[3]);
            const half2 cI = __hsub2(im[0], im[2]), dI = __hsub2(im[1], im[3]);
            zr[i][0] = __hsub2(aR, bR);  // x0 - x1 + x2 - x3
            zi[i][0] = __hsub2(aI, bI);
            zr[i][1] = __hsub2(cR, dI);  // x0 + i x1 - x2 - i x3
            zi[i][1] = __hadd2(cI, dR);
            zr[i][2] = __hadd2(aR, bR);  // x0 + x1 + x2 + x3
            zi[i][2] = __hadd2(aI, bI);
            zr[i][3] = __hadd2(cR, dI);  // x0 - i x1 - x2 + i x3
            zi[i][3] = __hsub2(cI, dR);
            if (PRE && circ) {
#pragma unroll
                for (int k = 0; k < 4; k++) circular_h2(zr[i][k], zi[i][k]);
            }
        }
#pragma unroll
        for (int p = 0; p < 2; p++) {
            const uint32_t sel = p ? 0x7632u : 0x5410u;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                out_r[p][k].x = __byte_perm(h2u(zr[0][k]), h2u(zr[1][k]), sel);
                out_r[p][k].y = __byte_perm(h2u(zr[2][k]), h2u(zr[3][k]), sel);
                out_i[p][k].x = __byte_perm(h2u(zi[0][k]), h2u(zi[1][k]), sel);
                out_i[p][k].y = __byte_perm(h2u(zi[2][k]), h2u(zi[3][k]), sel);
            }
        }
    } else {
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int k = 0; k < 4; k++) out_r[p][k] = out_i[p][k] = make_uint2(0u, 0u);
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) {
        *reinterpret_cast<uint2*>(op0 + t.o_r + k * 4096u) = out_r[0][k];
        *reinterpret_cast<uint2*>(op0 + t.o_i + k * 4096u) = out_i[0][k];
        *reinterpret_cast<uint2*>(op1 + t.o_r + k * 4096u) = out_r[1][k];
        *reinterpret_cast<uint2*>(op1 + t.o_i + k * 4096u) = out_i[1][k];
    }
}

// R = 2, both polarisations in one pass, arranged as the R = 4 tasks above: a warp
// covers 16 of the tile's 64 spectra x 8 antennas, row k * 64 + s sits 8192 * k bytes
// after row s, and the DFT runs on (p0, p1) halves (x0 - x1: the 1152 biases cancel;
// x0 + x1: removed together).
__device__ __forceinline__ R4Task r2_task(uint32_t wt, uint32_t lane, uint32_t A, uint32_t KA, uint32_t rrow) {
    const uint32_t s = (wt & 3u) * 16u + (lane & 7u) + ((lane >> 4) << 3);
    const uint32_t a0 = (2u * (wt >> 2) + ((lane >> 3) & 1u)) * 4u;
    R4Task t;
    t.raw_off = a0 * rrow + s * 8u;
    t.o_r = op_off(s, a0);
    t.o_i = op_off(s, KA + a0);
    t.nvalid = a0 < A ? min(4u, A - a0) : 0u;
    return t;
}

template <bool PRE>
__device__ __forceinline__ void r2_pair_words(const uint2 (&vs)[4], uint8_t* op0, uint8_t* op1, const R4Task& t,
                                              uint32_t circ) {
    const half2 h2304 = __halves2half2(__ushort_as_half(0x6880), __ushort_as_half(0x6880));  // 2304
    half2 zr[4][2], zi[4][2];  // [antenna][k], halves = (pol 0, pol 1)
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) {
        if (i < t.nvalid) {
            const uint2 v = vs[i];
            const uint32_t w[2] = {v.x ^ 0x80808080u, v.y ^ 0x80808080u};
            half2 re[2], im[2];  // 1152 + x
#pragma unroll
            for (int j = 0; j < 2; j++) {
                re[j] = u2h(__byte_perm(w[j], 0x64646464u, 0x4240));
                im[j] = u2h(__byte_perm(w[j], 0x64646464u, 0x4341));
            }
            zr[i][0] = __hsub2(re[0], re[1]);
            zi[i][0] = __hsub2(im[0], im[1]);
            zr[i][1] = __hadd2(__hsub2(re[0], h2304), re[1]);
            zi[i][1] = __hadd2(__hsub2(im[0], h2304), im[1]);
            if (PRE && circ) {
#pragma unroll
                for (int k = 0; k < 2; k++) circular_h2(zr[i][k], zi[i][k]);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 2; k++) zr[i][k] = zi[i][k] = u2h(0u);
        }
    }
#pragma unroll
    for (int p = 0; p < 2; p++) {
        const uint32_t sel = p ? 0x7632u : 0x5410u;
        uint8_t* op = p ? op1 : op0;
#pragma unroll
        for (uint32_t k = 0; k < 2; k++) {
            *reinterpret_cast<uint2*>(op + t.o_r + k * 8192u) =
                make_uint2(__byte_perm(h2u(zr[0][k]), h2u(zr[1][k]), sel), __byte_perm(h2u(zr[2][k]), h2u(zr[3][k]), sel));
            *reinterpret_cast<uint2*>(op + t.o_i + k * 8192u) =
                make_uint2(__byte_perm(h2u(zi[0][k]), h2u(zi[1][k]), sel), __byte_perm(h2u(zi[2][k]), h2u(zi[3][k]), sel));
        }
    }
}

template <bool PRE>
__device__ __forceinline__ void r2_pair_task(const uint8_t* raw, uint32_t rrow, uint8_t* op0, uint8_t* op1,
                                             const R4Task& t, uint32_t circ) {
    uint2 v[4];
#pragma unroll
    for (uint32_t i = 0; i < 4; i++)
        v[i] = i < t.nvalid ? *reinterpret_cast<const uint2*>(raw + t.raw_off + i * rrow) : make_uint2(0u, 0u);
    r2_pair_words<PRE>(v, op0, op1, t, circ);
}

// Direct mode at R = 2 (no raw ring, as at R = 1 below): the spectra of a warp-task
// straight from global memory, one 8-byte load per antenna (16 consecutive spectra of
// each antenna per warp load, 128 contiguous bytes).
struct Direct2 {
    uint32_t t_off, a0;  // first sample of the task's spectrum in the tile, first antenna
};

__device__ __forceinline__ Direct2 direct2_task(uint32_t wt, uint32_t lane) {
    const uint32_t s = (wt & 3u) * 16u + (lane & 7u) + ((lane >> 4) << 3);
    return {2u * s, (2u * (wt >> 2) + ((lane >> 3) & 1u)) * 4u};
}

__device__ __forceinline__ void direct2_load(const uint32_t* in, uint32_t F, uint32_t T, uint32_t f, uint32_t t0,
                                             const Direct2& d, uint32_t nvalid, uint2 (&v)[4]) {
    const uint32_t* row = in + ((uint64_t)d.a0 * F + f) * T + t0 + d.t_off;
#pragma unroll
    for (uint32_t i = 0; i < 4; i++)
        v[i] = i < nvalid ? __ldg(reinterpret_cast<const uint2*>(row + (uint64_t)i * F * T)) : make_uint2(0u, 0u);
}

// Rate 1 from CF16 voltages (the ModeB path: channelized and polarized on the
// way in, exact in FP16): raw rows of 128 samples x 8 bytes [p0 (re, im) | p1 (re,
// im)] per antenna.  A task is one sample of 8 antennas -> the (re, im) chunks of
// polarisation p; consecutive lanes take consecutive samples (rows).
__device__ __forceinline__ void build_operand_h16(const uint8_t* raw, uint32_t rrow, uint8_t* op, uint32_t A,
                                                  uint32_t KA, int p, uint32_t ct) {
    constexpr uint32_t kStride = kConvWarps * 32;
    const uint32_t ntasks = kM * (KA / 8);
    for (uint32_t t = ct; t < ntasks; t += kStride) {
        const uint32_t s = t % kM, g = t / kM;
        uint32_t h[8];  // half2 (re, im) of polarisation p, antennas g*8 .. g*8+7
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t a = g * 8 + i;
            h[i] = a < A ? *reinterpret_cast<const uint32_t*>(raw + a * rrow + s * 8 + p * 4) : 0u;
        }
        uint4 vr, vi;
        vr.x = __byte_perm(h[0], h[1], 0x5410);
        vr.y = __byte_perm(h[2], h[3], 0x5410);
        vr.z = __byte_perm(h[4], h[5], 0x5410);
        vr.w = __byte_perm(h[6], h[7], 0x5410);
        vi.x = __byte_perm(h[0], h[1], 0x7632);
        vi.y = __byte_perm(h[2], h[3], 0x7632);
        vi.z = __byte_perm(h[4], h[5], 0x7632);
        vi.w = __byte_perm(h[6], h[7], 0x7632);
        *reinterpret_cast<uint4*>(op + op_off(s, g * 8)) = vr;
        *reinterpret_cast<uint4*>(op + op_off(s, KA + g * 8)) = vi;
    }
}

// Both polarisations of one CF16 tile in one pass: one 8-byte load per (antenna,
// sample) feeds both operands (consecutive lanes read consecutive 8-byte samples,
// so a warp's loads are conflict-free).
__device__ __forceinline__ void build_operand_h16_pair(const uint8_t* raw, uint32_t rrow, uint8_t* op0, uint8_t* op1,
                                                       uint32_t A, uint32_t KA, uint32_t ct) {
    constexpr uint32_t kStride = kConvWarps * 32;
    const uint32_t ntasks = kM * (KA / 8);
    for (uint32_t t = ct; t < ntasks; t += kStride) {
        const uint32_t s = t % kM, g = t / kM;
        uint2 v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t a = g * 8 + i;
            v[i] = a < A ? *reinterpret_cast<const uint2*>(raw + a * rrow + s * 8) : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int p = 0; p < 2; p++) {
            uint32_t h[8];
#pragma unroll
            for (int i = 0; i < 8; i++) h[i] = p ? v[i].y : v[i].x;
            uint4 vr, vi;
            vr.x = __byte_perm(h[0], h[1], 0x5410);
            vr.y = __byte_perm(h[2], h[3], 0x5410);
            vr.z = __byte_perm(h[4], h[5], 0x5410);
            vr.w = __byte_perm(h[6], h[7], 0x5410);
            vi.x = __byte_perm(h[0], h[1], 0x7632);
            vi.y = __byte_perm(h[2], h[3], 0x7632);
            vi.z = __byte_perm(h[4], h[5], 0x7632);
            vi.w = __byte_perm(h[6], h[7], 0x7632);
            uint8_t* op = p ? op1 : op0;
            *reinterpret_cast<uint4*>(op + op_off(s, g * 8)) = vr;
            *reinterpret_cast<uint4*>(op + op_off(s, KA + g * 8)) = vi;
        }
    }
}

// R = 1 CI8, both polarisations of a tile in one pass.  Thread (converter warp w,
// lane l) owns samples 4l .. 4l + 3 (rows of the operand) and one group g of 8
// antennas, fixed for the whole kernel:
//   KA = 64: g = (l + w) & 7,         warps 0-7;
//   KA = 32: g = ((l >> 1) + w) & 3,  warps 0-3 (warps 4-7 only keep the handshakes).
// Loads: one 16-byte load per antenna (4 samples x [p0 re, p0 im, p1 re, p1 im]);
// the 8 lanes of a quarter-warp read 8 consecutive 16-byte slots of a row, so each
// is one wavefront.  Stores: a 16-byte chunk of row 4l + j holds 8 antennas of one
// component; its bank group is g ^ (row & 7) = g ^ 4 (l & 1) ^ j, which the
// mappings above make distinct over every quarter-warp.  Conversion: byte permutes
// gather one component of two antennas ([a p0, b p0, a p1, b p1]), the XOR with
// 0x80 per byte and a second permute with the 0x64 exponent byte give the half2
// (1024 + x + 128) per polarisation, and one subtraction of 1152 makes it exact x.
struct R1Task {
    uint32_t raw_off;        // 8 g * rrow + 16 l in the raw tile
    uint32_t o_r[4], o_i[4];  // operand offsets of (row 4l + j, K = 8 g) and (row 4l + j, K = KA + 8 g)
    uint32_t nvalid;         // antennas 8 g .. 8 g + nvalid - 1 exist (0..8)
    uint32_t active;
};

__device__ __forceinline__ R1Task r1_task(uint32_t w, uint32_t l, uint32_t A, uint32_t KA, uint32_t rrow) {
    R1Task t;
    const uint32_t ng = KA / 8;
    const uint32_t g = ng == 8 ? ((l + w) & 7u) : (((l >> 1) + w) & 3u);
    t.active = w < ng;
    t.raw_off = 8u * g * rrow + 16u * l;
    const uint32_t a0 = 8u * g;
    t.nvalid = (t.active && a0 < A) ? min(8u, A - a0) : 0u;
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
        t.o_r[j] = op_off(4u * l + j, a0);
        t.o_i[j] = op_off(4u * l + j, KA + a0);
    }
    return t;
}

// One sample of 8 antennas -> the (re, im) chunks of both polarisations (exact
// int8 -> FP16; see the R1Task comment).
__device__ __forceinline__ void r1_convert_store(const uint32_t (&wv)[8], uint8_t* op0, uint8_t* op1, uint32_t o_r,
                                                 uint32_t o_i) {
    const half2 h1152 = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));
    uint32_t r0[4], i0[4], r1[4], i1[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint32_t tr = __byte_perm(wv[2 * q], wv[2 * q + 1], 0x6240) ^ 0x80808080u;
        const uint32_t ti = __byte_perm(wv[2 * q], wv[2 * q + 1], 0x7351) ^ 0x80808080u;
        r0[q] = h2u(__hsub2(u2h(__byte_perm(tr, 0x64646464u, 0x4140)), h1152));
        r1[q] = h2u(__hsub2(u2h(__byte_perm(tr, 0x64646464u, 0x4342)), h1152));
        i0[q] = h2u(__hsub2(u2h(__byte_perm(ti, 0x64646464u, 0x4140)), h1152));
        i1[q] = h2u(__hsub2(u2h(__byte_perm(ti, 0x64646464u, 0x4342)), h1152));
    }
    *reinterpret_cast<uint4*>(op0 + o_r) = make_uint4(r0[0], r0[1], r0[2], r0[3]);
    *reinterpret_cast<uint4*>(op0 + o_i) = make_uint4(i0[0], i0[1], i0[2], i0[3]);
    *reinterpret_cast<uint4*>(op1 + o_r) = make_uint4(r1[0], r1[1], r1[2], r1[3]);
    *reinterpret_cast<uint4*>(op1 + o_i) = make_uint4(i1[0], i1[1], i1[2], i1[3]);
}

__device__ __forceinline__ void r1_pair_task(const uint8_t* raw, uint32_t rrow, uint8_t* op0, uint8_t* op1,
                                             const R1Task& t) {
    if (!t.active) return;
    const uint8_t* src = raw + t.raw_off;
    uint4 v[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; i++)
        v[i] = i < t.nvalid ? *reinterpret_cast<const uint4*>(src + i * rrow) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        uint32_t wv[8];
#pragma unroll
        for (int i = 0; i < 8; i++) wv[i] = j == 0 ? v[i].x : j == 1 ? v[i].y : j == 2 ? v[i].z : v[i].w;
        r1_convert_store(wv, op0, op1, t.o_r[j], t.o_i[j]);
    }
}

// R = 1 CI8 "direct" mode (no raw ring in shared memory, which leaves room for
// four operand stages beside a large phasor image): each converter thread loads
// its voltage words from global memory itself, one tile ahead of the one it
// builds.  Thread (converter warp w, lane l) owns antenna group g of 8 and the
// rows l + 32 j (j in its set of sample quarters), fixed for the kernel:
//   KA = 64: g = w, j = 0..3;   KA = 32: g = w & 3, j = 2 (w >> 2) and 2 (w >> 2) + 1.
// Loads: 4-byte words, consecutive lanes at consecutive samples of one antenna
// (128 contiguous bytes per warp load).  Stores: the 16-byte chunk (row l + 32 j,
// group g) has bank group g ^ (l & 7), distinct over a quarter-warp.
constexpr uint32_t kDirectMaxJ = 4;

struct DirectTask {
    uint32_t a0, nvalid, j0, nj;
    uint32_t o_r[kDirectMaxJ], o_i[kDirectMaxJ];  // offsets of (row l + 32 (j0 + j), K = a0) and (..., K = KA + a0)
};

__device__ __forceinline__ DirectTask direct_task(uint32_t w, uint32_t l, uint32_t A, uint32_t KA) {
    DirectTask t;
    const bool wide = KA == 64;
    const uint32_t g = wide ? w : (w & 3u);
    t.j0 = wide ? 0u : 2u * (w >> 2);
    t.nj = wide ? 4u : 2u;
    t.a0 = 8u * g;
    t.nvalid = t.a0 < A ? min(8u, A - t.a0) : 0u;
#pragma unroll
    for (uint32_t j = 0; j < kDirectMaxJ; j++) {
        const uint32_t row = l + 32u * (t.j0 + (j < t.nj ? j : 0u));
        t.o_r[j] = op_off(row, t.a0);
        t.o_i[j] = op_off(row, KA + t.a0);
    }
    return t;
}

// The words [j][i] = sample (t0 + l + 32 (j0 + j)) of antenna a0 + i in channel f.
__device__ __forceinline__ void direct_load(const uint32_t* in, uint32_t F, uint32_t T, uint32_t f, uint32_t t0,
                                            uint32_t l, const DirectTask& t, uint32_t (&v)[kDirectMaxJ][8]) {
#pragma unroll
    for (uint32_t i = 0; i < 8; i++) {
        const uint32_t* row = in + ((uint64_t)(t.a0 + i) * F + f) * T + t0 + l + 32u * t.j0;
#pragma unroll
        for (uint32_t j = 0; j < kDirectMaxJ; j++)
            v[j][i] = (i < t.nvalid && j < t.nj) ? __ldg(row + 32u * j) : 0u;
    }
}

__device__ __forceinline__ void direct_build(const uint32_t (&v)[kDirectMaxJ][8], uint8_t* op0, uint8_t* op1,
                                             const DirectTask& t) {
#pragma unroll
    for (uint32_t j = 0; j < kDirectMaxJ; j++)
        if (j < t.nj) r1_convert_store(v[j], op0, op1, t.o_r[j], t.o_i[j]);
}

// Both polarisations of one tile for R = 1 and 2: two single-polarisation passes.
template <int R>
__device__ __forceinline__ void build_operand_pair(const uint8_t* raw, uint32_t rrow, uint8_t* op0, uint8_t* op1, uint32_t A,
                                                   uint32_t KA, uint32_t ct) {
    build_operand<R>(raw, rrow, op0, A, KA, 0, ct);
    build_operand<R>(raw, rrow, op1, A, KA, 1, ct);
}

// Window sum of NV per-beam values over I = 2^LOGI adjacent lanes by a butterfly
// reduce-scatter: after min(LOGI, log2 NV) halving rounds each lane holds the
// window sums of NV >> min(LOGI, log2 NV) consecutive beams starting at *first; the
// remaining rounds (I > NV) are a plain exchange.  Returns the number of values
// this lane stores (0 for the lanes that hold duplicates when I > NV).
template <int NV, int LOGI>
__device__ __forceinline__ int window_reduce(float (&v)[NV], uint32_t lane, uint32_t* first) {
    constexpr int LOGNV = NV == 16 ? 4 : NV == 8 ? 3 : NV == 4 ? 2 : NV == 2 ? 1 : 0;
    constexpr int RS = LOGI < LOGNV ? LOGI : LOGNV;
    uint32_t off = 0;
#pragma unroll
    for (int s = 0; s < RS; s++) {
        const int half = NV >> (s + 1);
        const bool upper = (lane >> s) & 1u;
#pragma unroll
        for (int j = 0; j < half; j++) {
            const float send = upper ? v[j] : v[half + j];
            const float recv = __shfl_xor_sync(0xffffffffu, send, 1 << s);
            v[j] = (upper ? v[half + j] : v[j]) + recv;
        }
        if (upper) off += half;
    }
#pragma unroll
    for (int s = RS; s < LOGI; s++) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1 << s);
    *first = off;
    if (LOGI > LOGNV && ((lane >> LOGNV) & ((1u << (LOGI > LOGNV ? LOGI - LOGNV : 0)) - 1u))) return 0;
    return NV >> RS;
}

// ---- MMA issue ----------------------------------------------------------------
// Descriptors are built once per stage and stepped by adding 16-byte units to the
// start-address field, so each tcgen05.mma costs a handful of integer adds.
// A operand k-step j: column block j / 4 (16 KB each), 32 bytes per step in a row.
__device__ __forceinline__ uint64_t a_step(uint64_t ad, int j) {
    return ad + (uint64_t)((((j >> 2) * 16384) + (j & 3) * 32) >> 4);
}

// hi and lo stacked along N (4 NB rows per column block of the image): one MMA per k-step.
template <int KSTEPS>
__device__ __forceinline__ void issue_stacked(uint32_t d, uint64_t ad, uint64_t wd, uint32_t wblk16, uint32_t idesc) {
#pragma unroll
    for (int j = 0; j < KSTEPS; j++)
        mma_f16(d, a_step(ad, j), wd + (uint64_t)((j >> 2) * wblk16 + (j & 3) * 2), idesc, j > 0 ? 1u : 0u);
}

// KA = 64, hi and lo as separate MMAs: the Xr steps read blocks [Wr | Wi], the Xi
// steps [-Wi | Wr] of the [-Wi | Wr | Wi] image (nb16 = one block, 16-byte units).
__device__ __forceinline__ void issue_ka64(uint32_t d, uint64_t ad, uint64_t wd, uint32_t nb16, uint32_t idesc) {
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int j = 0; j < 8; j++)
            mma_f16(d, a_step(ad, j), wd + (uint64_t)(h * 3 * nb16 + (j < 4 ? nb16 : 0) + (j & 3) * 2), idesc,
                    (h | j) ? 1u : 0u);
}

// KA = 32, hi and lo as separate MMAs over one block of 2 NB rows per (p, h).
__device__ __forceinline__ void issue_ka32(uint32_t d, uint64_t ad, uint64_t wd, uint32_t nb16, uint32_t idesc) {
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            mma_f16(d, a_step(ad, j), wd + (uint64_t)(h * 2 * nb16 + j * 2), idesc, (h | j) ? 1u : 0u);
}

// The same products with the roles of the operands swapped: the image blocks are
// the A operand (M = 128 rows: Re outputs of the 64 beams, then Im outputs) and the
// tile's samples the B operand (N = 128), so the accumulator holds one output row
// per TMEM lane and the tile's samples along its columns.
__device__ __forceinline__ void issue_ka64_t(uint32_t d, uint64_t ad, uint64_t wd, uint32_t nb16, uint32_t idesc) {
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int j = 0; j < 8; j++)
            mma_f16(d, wd + (uint64_t)(h * 3 * nb16 + (j < 4 ? nb16 : 0) + (j & 3) * 2), a_step(ad, j), idesc,
                    (h | j) ? 1u : 0u);
}

__device__ __forceinline__ void issue_ka32_t(uint32_t d, uint64_t ad, uint64_t wd, uint32_t nb16, uint32_t idesc) {
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            mma_f16(d, wd + (uint64_t)(h * 2 * nb16 + j * 2), a_step(ad, j), idesc, (h | j) ? 1u : 0u);
}

// Epilogue of the transposed accumulator (rate 1 CI8, windows of I = 8 or 16
// samples, one 64-beam chunk): TMEM lane m holds output row m (Re of beam m for
// m < 64, Im of beam m - 64 after) and column c sample c of the tile, so a thread
// adds the squares of its row over each window of I consecutive columns (two
// columns per packed FP32x2 FMA) without any lane exchange.  Warps 0 and 1 of the
// lane quarters (the Re rows) store their window sums of both polarisations to
// the output; warps 2 and 3 (the Im rows) keep theirs in registers and add them to
// the stored partial sums one tile later, once pr_full says those are there.  The
// Re half signals a tile's partial sums after reading the next tile from TMEM, so
// neither half waits on the round trip through memory.
//
// Phases of pr_full: an mbarrier wait tests only the parity of its phase, so the Re
// half must never complete a barrier's next phase before the Im half has waited
// for the current one.  Inside the range, the Re half's signal for tile m needs the
// accumulator of tile m + 1, which needs the Im half's release of tile m + 1 - nacc,
// which it gives only after its wait for tile m - nacc, the previous phase of the
// same barrier.  The signal for the range's last tile comes after the loop with no
// accumulator to gate it, so the Re half first waits for the release of tile
// n - nacc (that wait of the Im half precedes it).
//
// At rate 1 a channel holds tpc tiles of NW outputs and U = tpc NW, so tile L of
// the chunk's F tpc tiles writes outputs L NW .. L NW + NW - 1 of each beam row.
template <int LOGI>
__device__ __forceinline__ void epilogue_transposed(const TcArgs& g, uint32_t tmem, uint32_t d_cols, uint32_t nacc,
                                                    uint64_t* d_full, uint64_t* d_empty, uint64_t* pr_full,
                                                    volatile int* abort, uint64_t L0, uint64_t L1, uint32_t q,
                                                    uint32_t lane) {
    constexpr uint32_t I = 1u << LOGI;
    constexpr int NW = kM / I;                      // windows per tile: 16 or 8
    constexpr int kCols = LOGI == 3 ? 32 : 16;      // TMEM columns read per wait
    const bool re_half = q < 2;
    const uint32_t b = 32u * (q & 1u) + lane;
    const bool valid = b < g.beams;
    float* row = g.out + (uint64_t)b * g.F * g.U + L0 * NW;  // this beam's outputs of tile L0
    const uint32_t n = (uint32_t)(L1 - L0);
    uint32_t db = 0, dph = 0;
    float pend[NW];  // Im half: the previous tile's own window sums
    uint32_t i = 0;
    for (; i < n; i++) {
        if (!mbar_wait(&d_full[db], dph, abort, kWaitBudget)) { record_abort(abort, 7); break; }
        tc_fence_after();
        const uint32_t lane_addr = tmem + ((32 * q) << 16) + db * (2 * d_cols);
        float2 acc[NW];
#pragma unroll
        for (int w = 0; w < NW; w++) acc[w] = make_float2(0.f, 0.f);
#pragma unroll
        for (uint32_t p = 0; p < 2; p++) {
#pragma unroll
            for (int c0 = 0; c0 < kM; c0 += kCols) {
                uint32_t r[kCols / 16][16];
#pragma unroll
                for (int k = 0; k < kCols / 16; k++) tmem_ld16(lane_addr + p * d_cols + c0 + 16 * k, r[k]);
                tmem_ld_wait();
#pragma unroll
                for (int k = 0; k < kCols / 16; k++)
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const int w = (c0 + 16 * k + 2 * j) / I;
                        const float2 v = make_float2(__uint_as_float(r[k][2 * j]), __uint_as_float(r[k][2 * j + 1]));
                        acc[w] = __ffma2_rn(v, v, acc[w]);
                    }
            }
        }
        tc_fence_before();
        __syncwarp();
        // the previous tile's accumulator slot and phase
        const uint32_t pdb = db ? db - 1 : nacc - 1, pph = db ? dph : dph ^ 1u;
        float* o = row + (uint64_t)i * NW;
        if (re_half) {
            if (lane == 0) {
                mbar_arrive(&d_empty[db]);
                if (i) mbar_arrive(&pr_full[pdb]);  // stored a tile ago
            }
            if (valid) {
#pragma unroll
                for (int w = 0; w < NW; w += 4)
                    *reinterpret_cast<float4*>(o + w) = make_float4(acc[w].x + acc[w].y, acc[w + 1].x + acc[w + 1].y,
                                                                    acc[w + 2].x + acc[w + 2].y, acc[w + 3].x + acc[w + 3].y);
            }
            __threadfence_block();  // ordered before lane 0's next arrive on pr_full
            __syncwarp();
        } else {
            if (i && !mbar_wait(&pr_full[pdb], pph, abort, kWaitBudget)) { record_abort(abort, 12); break; }
            __syncwarp();
            if (lane == 0) mbar_arrive(&d_empty[db]);
            if (i && valid) {
#pragma unroll
                for (int w = 0; w < NW; w += 4) {
                    const float4 r = *reinterpret_cast<const float4*>(o - NW + w);
                    *reinterpret_cast<float4*>(o - NW + w) =
                        make_float4(r.x + pend[w], r.y + pend[w + 1], r.z + pend[w + 2], r.w + pend[w + 3]);
                }
            }
#pragma unroll
            for (int w = 0; w < NW; w++) pend[w] = acc[w].x + acc[w].y;
        }
        if (++db == nacc) { db = 0; dph ^= 1; }
    }
    if (i == n && n) {
        // the last tile's exchange (db, dph now name tile n's slot and phase)
        const uint32_t pdb = db ? db - 1 : nacc - 1, pph = db ? dph : dph ^ 1u;
        float* o = row + (uint64_t)(n - 1) * NW;
        if (re_half) {
            // tile n - nacc used this slot in the phase before: wait for its release
            if (n >= nacc && !mbar_wait(&d_empty[db], dph ^ 1u, abort, kWaitBudget)) record_abort(abort, 13);
            else if (lane == 0) mbar_arrive(&pr_full[pdb]);
        } else if (mbar_wait(&pr_full[pdb], pph, abort, kWaitBudget)) {
            __syncwarp();
            if (valid) {
#pragma unroll
                for (int w = 0; w < NW; w += 4) {
                    const float4 r = *reinterpret_cast<const float4*>(o + w);
                    *reinterpret_cast<float4*>(o + w) =
                        make_float4(r.x + pend[w], r.y + pend[w + 1], r.z + pend[w + 2], r.w + pend[w + 3]);
                }
            }
        } else {
            record_abort(abort, 12);
        }
    }
}

// ---- phasor image ------------------------------------------------------------
// plan[chunk][f][p] in the 128-byte-swizzled K-major layout (K = 2 KA: Xr part
// then Xi part), h 0 = hi = rn(w), h 1 = lo = rn(w - hi):
//   stacked (NB <= 32): per p, (2 KA / 64) column blocks of 4 NB rows
//            [hi: b -> (Wr | -Wi), NB + b -> (Wi | Wr) ; lo: the same],
//   KA = 64, NB > 32: per (p, h) three blocks of NB rows x 64 K: [-Wi | Wr | Wi],
//   KA = 32, NB > 32: per (p, h) one block of 2 NB rows: b -> [Wr | -Wi], NB + b -> [Wi | Wr].
// One thread writes the 16-byte chunks of one (chunk c, channel f, polarisation p,
// beam row nb, 8-antenna group j) for hi and lo: 8 phasors in, 8 or 12 chunk
// stores out.  Consecutive threads take consecutive channels, so the phasor loads
// of a warp are 16 bytes apart.
__device__ __forceinline__ uint4 pack8(const __half (&v)[8]) {
    uint4 u;
    u.x = (uint32_t)__half_as_ushort(v[0]) | ((uint32_t)__half_as_ushort(v[1]) << 16);
    u.y = (uint32_t)__half_as_ushort(v[2]) | ((uint32_t)__half_as_ushort(v[3]) << 16);
    u.z = (uint32_t)__half_as_ushort(v[4]) | ((uint32_t)__half_as_ushort(v[5]) << 16);
    u.w = (uint32_t)__half_as_ushort(v[6]) | ((uint32_t)__half_as_ushort(v[7]) << 16);
    return u;
}

// 16-byte chunk holding K elements [k_total, k_total + 8) of `row` in a stack of
// 64-wide column blocks of `rows` rows each.
__device__ __forceinline__ void put_chunk(uint8_t* base, uint32_t rows, uint32_t row, uint32_t k_total, uint4 v) {
    *reinterpret_cast<uint4*>(base + (k_total >> 6) * rows * 128u + sw128_off(row, (k_total >> 3) & 7u)) = v;
}

// The split of 8 antennas' phasors of one beam, channel and polarisation.
struct SplitChunk {
    uint4 re[2], im[2], nim[2];  // [hi, lo]: Wr, Wi, -Wi
};

// 8 antennas from a0 of the beam row `w` (phasor (antenna a, this channel and
// polarisation) at w[a * astride]); hi = rn(w), lo = rn(w - hi) per component, antennas
// from A on are 0, all of them when !beam.
__device__ __forceinline__ void split_chunk(const float2* __restrict__ w, uint64_t astride, uint32_t a0, uint32_t A,
                                            bool beam, SplitChunk& c) {
    __half rh[8], ih[8], rl[8], il[8], nih[8], nil[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const uint32_t a = a0 + e;
        float wr = 0.f, wi = 0.f;
        if (a < A && beam) {
            const float2 v = w[a * astride];
            wr = v.x;
            wi = v.y;
        }
        rh[e] = __float2half_rn(wr);
        ih[e] = __float2half_rn(wi);
        rl[e] = __float2half_rn(wr - __half2float(rh[e]));
        il[e] = __float2half_rn(wi - __half2float(ih[e]));
        nih[e] = __hneg(ih[e]);
        nil[e] = __hneg(il[e]);
    }
    c.re[0] = pack8(rh);
    c.re[1] = pack8(rl);
    c.im[0] = pack8(ih);
    c.im[1] = pack8(il);
    c.nim[0] = pack8(nih);
    c.nim[1] = pack8(nil);
}

// put(offset, chunk) for every 16-byte chunk that beam row nb and the antennas from k0
// have in one polarisation's image (offsets from that polarisation's base); a stacked
// image of `fold` channels has its rows of channel fk behind those of the ones before.
template <class Put>
__device__ __forceinline__ void put_image(Put put, const SplitChunk& c, uint32_t NB, uint32_t KA, uint32_t nb,
                                          uint32_t k0, uint32_t stacked, uint32_t fold, uint32_t fk) {
    auto at = [&](uint32_t rows, uint32_t row, uint32_t k, uint4 v) {
        put((k >> 6) * rows * 128u + sw128_off(row, (k >> 3) & 7u), v);
    };
    if (stacked) {
        // (2 KA / 64) column blocks of 4 NB rows: hi: row nb -> [Wr | -Wi], row NB + nb -> [Wi | Wr];
        // lo: the same at rows + 2 NB
        const uint32_t r0 = fk * 4 * NB + nb, rows = fold * 4 * NB;
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            at(rows, r0 + 2 * h * NB, k0, c.re[h]);
            at(rows, r0 + 2 * h * NB, KA + k0, c.nim[h]);
            at(rows, r0 + (2 * h + 1) * NB, k0, c.im[h]);
            at(rows, r0 + (2 * h + 1) * NB, KA + k0, c.re[h]);
        }
        return;
    }
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
        if (KA == 64) {
            // three blocks of NB rows x 64 K: [-Wi | Wr | Wi]
            const uint32_t blk = h * 3u * NB * 128u;
            put(blk + sw128_off(nb, (k0 >> 3) & 7u), c.nim[h]);
            put(blk + NB * 128u + sw128_off(nb, (k0 >> 3) & 7u), c.re[h]);
            put(blk + 2u * NB * 128u + sw128_off(nb, (k0 >> 3) & 7u), c.im[h]);
        } else {
            // one block of 2 NB rows x 64 K: row nb -> [Wr | -Wi], row NB + nb -> [Wi | Wr]
            const uint32_t blk = h * 2u * NB * 128u;
            put(blk + sw128_off(nb, (k0 >> 3) & 7u), c.re[h]);
            put(blk + sw128_off(nb, ((32u + k0) >> 3) & 7u), c.nim[h]);
            put(blk + sw128_off(NB + nb, (k0 >> 3) & 7u), c.im[h]);
            put(blk + sw128_off(NB + nb, ((32u + k0) >> 3) & 7u), c.re[h]);
        }
    }
}

// ES = bytes per dual-polarisation input sample: 4 (CI8) or 8 (CF16, rate 1 only).
//
// PRE (ModeB's order, R = 2 or 4): the channelizer runs before the beamformer, so every
// fine channel has its own phasors.  The operand is the same (row = k * 128 / R +
// spectrum holds fine channel k), and the R fine channels' stacked images lie side
// by side along N: one MMA of N = 4 R NB columns per k-step gives every row the
// products of all R images, of which the epilogue reads the columns of the row's own
// fine channel.  The tensor pipe does R times the useful work and is still not what
// bounds the tile (1024 of about 1900 cycles at R = 4, NB = 16), and the fine-channel
// voltages never reach memory (28 antennas x 192 channels x 8192 samples, 16 beams,
// R = 4, I = 4: 96 us with the split, where CF16 fine channels through memory took 88
// to write and 104 to beamform).  An accumulator is one polarisation (2 x 256 columns
// fill tensor memory), and each MMA issuer owns one.
//
// SELF: every CTA's tiles lie in one channel, whose phasor image all warps split
// straight into shared memory before their roles begin (and store to the plan, once per
// channel), so small blocks need no split launch before the chain.
template <int R, int LOGI, int ES = 4, int MODE = TC_BASE>
__global__ void __launch_bounds__(kThreads, 1) bf_tc_kernel(const TcArgs g, const __grid_constant__ CUtensorMap tmap) {
    constexpr bool PRE = MODE == TC_PRE, SELF = MODE == TC_SELF;
    // direct loads at R = 2 (at R = 1 every instantiation has them)
    constexpr bool DIRECT2 = R == 2 && ES == 4 && (MODE == TC_SELF || MODE == TC_DIRECT2);
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // Swizzled operands need 1024-byte aligned atoms: align the working base.
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t NB = g.NB, KA = g.KA, AS = g.a_stages, RS = g.r_stages;
    const uint32_t op_bytes = (2 * KA / 64) * 16384u;  // one polarisation's operand
    uint8_t* w_smem = smem;                              // phasor image
    uint8_t* a_smem = w_smem + g.img_bytes;              // AS operand stages
    uint8_t* r_smem = a_smem + (size_t)AS * op_bytes;    // RS raw tiles
    uint64_t* bars = reinterpret_cast<uint64_t*>(r_smem + (size_t)RS * g.raw_bytes);
    uint64_t* a_full = bars;
    uint64_t* a_empty = a_full + AS;
    uint64_t* r_full = a_empty + AS;
    uint64_t* r_empty = r_full + RS;
    uint64_t* d_full = r_empty + RS;
    uint64_t* d_empty = d_full + kMaxAcc;
    uint64_t* w_full = d_empty + kMaxAcc;
    uint64_t* w_empty = w_full + 1;
    uint64_t* fin = w_empty + 1;  // one per MMA issuer
    uint64_t* pr_full = fin + 2;  // transposed epilogue: the Re half's partial sums are stored
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pr_full + kMaxAcc);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int never = 0;  // abort flag that is never raised (drain waits)
    // Accumulator columns per polarisation: [re | im] (2 NB), or with hi/lo stacked
    // along N [hi re | hi im | lo re | lo im] (4 NB).
    const uint32_t d_cols = (PRE ? 4u * R : g.stacked ? 4u : 2u) * NB;
    // Accumulator buffers (tiles in flight between MMA and epilogue): as many as
    // fit the 512 TMEM columns, at most kMaxAcc.
    // PRE: one accumulator per polarisation.
    const uint32_t nacc = PRE ? 2u : min((uint32_t)kMaxAcc, 512u / (2u * d_cols));
    const uint32_t need_cols = (PRE ? 2u : nacc * 2u) * d_cols;
    const uint32_t tmem_cols = need_cols <= 32 ? 32 : need_cols <= 64 ? 64 : need_cols <= 128 ? 128 : need_cols <= 256 ? 256 : 512;
    // Pair mode: the converter builds both polarisations of a tile in one pass and
    // signals them together on the second stage of the pair.
    const bool pair = AS >= 4 && (AS & 1u) == 0;

    // Two MMA issuers (warp 0 and the last warp, lane 0 each) take alternate tiles
    // when the operand ring holds an even number of tile pairs and the accumulator
    // count is even, so that every barrier is only ever used by one issuer.  An
    // issue of tcgen05.mma holds its thread for about the MMA's duration, so one
    // issuer's waits and commits overlap the other's MMAs.
    const uint32_t nis = PRE || (pair && ((AS / 2) & 1u) == 0 && (nacc & 1u) == 0) ? 2u : 1u;
    // Split operand build (R = 4, two issuers, two-tile raw stages): converter warps
    // 0-3 build the even tiles of the CTA's range (the first tile of each raw stage,
    // issuer 0's) and warps 4-7 the odd ones, so the two halves run independently
    // and each operand pair has four producers.
    const bool split = R == 4 && nis == 2 && g.raw_tiles == 2;  // PRE: nis is always 2

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < AS; i++) {
            mbar_init(&a_full[i], split ? kConvWarps / 2 : kConvWarps);
            mbar_init(&a_empty[i], PRE ? 2 : 1);  // PRE: both issuers read the tile's pair
        }
        for (uint32_t i = 0; i < RS; i++) {
            mbar_init(&r_full[i], 1);
            mbar_init(&r_empty[i], kConvWarps);
        }
        for (uint32_t i = 0; i < nacc; i++) {
            mbar_init(&d_full[i], 1);
            mbar_init(&d_empty[i], kEpiWarps);
            mbar_init(&pr_full[i], kEpiWarps / 2);
        }
        mbar_init(w_full, 1);
        mbar_init(w_empty, nis);
        mbar_init(&fin[0], 1);
        mbar_init(&fin[1], 1);
        *abort = 0;
        fence_mbar_init();
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, tmem_cols);
        tmem_relinquish();
    }
    if constexpr (SELF) {
        const uint32_t f = blockIdx.x / g.segs, groups = KA / 8;
        const bool keep = blockIdx.x - f * g.segs == 0;
        uint8_t* out = g.plan_out + (uint64_t)f * g.img_bytes;
        const uint32_t pol = g.img_bytes / 2;
        for (uint32_t i = threadIdx.x; i < 2u * NB * groups; i += kThreads) {
            const uint32_t p = i & 1u, j = (i >> 1) % groups, nb = (i >> 1) / groups;
            SplitChunk w;
            split_chunk(g.ph + ((uint64_t)nb * g.A * g.F + f) * 2 + p, 2ull * g.F, j * 8, g.A, nb < g.beams, w);
            put_image([&](uint32_t off, uint4 v) {
                          *reinterpret_cast<uint4*>(w_smem + p * pol + off) = v;
                          if (keep) *reinterpret_cast<uint4*>(out + p * pol + off) = v;
                      }, w, NB, KA, nb, j * 8, g.stacked, 1, 0);
        }
        fence_proxy_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // This CTA's contiguous range of (channel, time-tile) tiles, a whole number of
    // raw stages (tiles per channel is a multiple of raw_tiles).
    const uint64_t per = ((g.total_tiles + gridDim.x - 1) / gridDim.x + g.raw_tiles - 1) / g.raw_tiles * g.raw_tiles;
    const uint32_t sf = SELF ? blockIdx.x / g.segs : 0u, st0 = SELF ? (blockIdx.x - sf * g.segs) * g.seg_tiles : 0u;
    const uint64_t L0 = SELF ? (uint64_t)sf * g.tiles_per_ch + st0 : (uint64_t)blockIdx.x * per;
    const uint64_t L1 = SELF ? (uint64_t)sf * g.tiles_per_ch + min(g.tiles_per_ch, st0 + g.seg_tiles)
                             : min(g.total_tiles, L0 + per);
    const uint32_t tpc = g.tiles_per_ch;
    const int issuer = warp == 0 ? 0 : (warp == kWarps - 1 ? 1 : -1);

    if (issuer >= 0) {
        // ---------------- MMA issuers ----------------
        const uint32_t j = (uint32_t)issuer;
        // The whole warp runs the loop and the waits (a lone active lane beside lanes
        // parked at the final barrier progressed slowly); lane 0 issues the MMAs and
        // the commits, which track that thread's MMAs.
        auto wait_all = [&](uint64_t* bar, uint32_t parity, unsigned code) -> bool {
            const bool w = __all_sync(0xffffffffu, mbar_wait(bar, parity, abort, kWaitBudget));
            if (!w && lane == 0) record_abort(abort, code);
            return w;
        };
        if (L0 < L1 && j < nis) {
            const uint32_t idesc = idesc_f16(kM, d_cols);
            const uint64_t w_desc = smem_desc_sw128(smem_u32(w_smem));
            const uint64_t a_desc = smem_desc_sw128(smem_u32(a_smem));
            const uint32_t op16 = op_bytes >> 4;   // operand stage stride, 16-byte units
            const uint32_t nb16 = NB * 8;          // NB rows x 128 bytes, 16-byte units
            // Phasor image stride per polarisation, 16-byte units:
            //   stacked: (2 KA / 64) column blocks of 4 NB rows;
            //   KA = 64: two (hi, lo) x three NB-row blocks; KA = 32: two x one 2 NB-row block.
            const uint32_t wpol16 = g.stacked ? (2 * KA / 64) * 4 * nb16 : (KA == 64 ? 6 * nb16 : 4 * nb16);
            // This issuer's first tile is local tile j: operand stage 2 j (pair mode)
            // or 0, accumulator j; both advance by nis tiles per own tile.
            uint32_t as = pair && !PRE ? 2 * j : 0, aph = 0, db = j, dph = 0, wph = 0;
            uint32_t tt = (uint32_t)(L0 % tpc);  // time tile within the channel, stepped below
            bool ok = true;
            uint32_t i = 0;
            for (uint64_t L = L0; L < L1 && ok; L++, i++) {
                if (!SELF && (L == L0 || tt == 0)) {
                    if (!wait_all(w_full, wph, 1)) { ok = false; break; }
                }
                if constexpr (PRE) {
                    // issuer j: polarisation j of every tile into accumulator j
                    if (!wait_all(&d_empty[j], dph ^ 1, 3) || !wait_all(&a_full[as + 1], aph, 2)) { ok = false; break; }
                    tc_fence_after();
                    if (lane == 0) {
                        const uint64_t ad = a_desc + (uint64_t)((as + j) * op16), wd = w_desc + (uint64_t)(j * R * wpol16);
                        issue_stacked<4>(tmem + j * d_cols, ad, wd, 4 * R * nb16, idesc);  // KA = 32
                        mma_commit(&a_empty[as + 1]);
                        mma_commit(&d_full[j]);
                    }
                    __syncwarp();
                    dph ^= 1;
                    as += 2;
                    if (as == AS) { as = 0; aph ^= 1; }
                } else if ((i % nis) == j) {
                    if (!wait_all(&d_empty[db], dph ^ 1, 3)) { ok = false; break; }
                    const uint32_t np = pair ? 1u : 2u;  // operand handshakes per tile
                    for (uint32_t h = 0; h < np; h++) {
                        // pair mode: the converter signals both polarisation stages on as + 1
                        const uint32_t sig = pair ? as + 1 : as;
                        if (!wait_all(&a_full[sig], aph, 2)) { ok = false; break; }
                        tc_fence_after();
                        if (lane == 0) {
                            for (uint32_t p = pair ? 0u : h; p < (pair ? 2u : h + 1); p++) {
                                const uint64_t ad = a_desc + (uint64_t)((as + (pair ? p : 0u)) * op16);
                                const uint64_t wd = w_desc + (uint64_t)(p * wpol16);
                                const uint32_t d = tmem + db * (2 * d_cols) + p * d_cols;
                                if (g.stacked) {
                                    if (KA == 64) issue_stacked<8>(d, ad, wd, 4 * nb16, idesc);
                                    else issue_stacked<4>(d, ad, wd, 4 * nb16, idesc);
                                } else if (g.transposed) {
                                    if (KA == 64) issue_ka64_t(d, ad, wd, nb16, idesc);
                                    else issue_ka32_t(d, ad, wd, nb16, idesc);
                                } else if (KA == 64) {
                                    issue_ka64(d, ad, wd, nb16, idesc);
                                } else {
                                    issue_ka32(d, ad, wd, nb16, idesc);
                                }
                            }
                            mma_commit(&a_empty[sig]);
                        }
                        __syncwarp();
                        as += pair ? 2u * nis : 1u;
                        if (as >= AS) { as -= AS; aph ^= 1; }
                    }
                    if (!ok) break;
                    if (lane == 0) mma_commit(&d_full[db]);
                    __syncwarp();
                    db += nis;
                    if (db >= nacc) { db -= nacc; dph ^= 1; }
                }
                // Every issuer releases the phasor image at the end of each channel
                // segment (the barrier counts one arrival per issuer).
                if (tt == tpc - 1 || L + 1 == L1) {
                    if (lane == 0) mma_commit(w_empty);
                    __syncwarp();
                    wph ^= 1;
                }
                if (++tt == tpc) tt = 0;
            }
            // Drain every MMA issued by this thread before TMEM is released
            // (bounded, but not cut short by the abort flag).
            if (lane == 0) {
                mma_commit(&fin[j]);
                if (!mbar_wait(&fin[j], 0, &never, kWaitBudget)) record_abort(abort, 4);
            }
            __syncwarp();
        }
    } else if (warp == 1) {
        // ---------------- loader: phasor image + raw CI8 tiles (bulk copies) ----------------
        if (SELF && g.direct) {
            // neither images nor raw tiles to load
        } else if (L0 < L1 && g.direct) {
            // direct mode: the converter threads load the voltages; only the images here
            uint32_t wph = 0;
            bool w_issued = false;
            uint32_t f = (uint32_t)(L0 / tpc);
            for (uint64_t L = L0; L < L1; L = (uint64_t)(++f) * tpc) {
                int ok = 1;
                if (lane == 0) {
                    if (g.pdl && L == L0) asm volatile("griddepcontrol.wait;" ::: "memory");
                    ok = mbar_wait(w_empty, wph ^ 1, abort, kWaitBudget);
                    if (ok) {
                        mbar_arrive_expect_tx(w_full, g.img_bytes);
                        bulk_g2s(w_smem, g.plan + (uint64_t)f * g.img_bytes, g.img_bytes, w_full);
                    } else {
                        record_abort(abort, 5);
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) break;
                w_issued = true;
                wph ^= 1;
            }
            if (lane == 0 && w_issued && !mbar_wait(w_full, wph ^ 1, &never, kWaitBudget)) record_abort(abort, 6);
            __syncwarp();
        } else if (L0 < L1) {
            uint32_t rs = 0, rph = 0, wph = 0;
            bool w_issued = false;
            uint32_t issued_mask = 0, issued_par = 0;  // per raw stage: issued?, parity of last issue
            // One raw stage = raw_tiles consecutive tiles of one channel, loaded as one or
            // two TMA boxes of up to 256 samples x 1 channel x A antennas (rows of
            // raw_row bytes per antenna: 512-byte rows per tile leave DRAM bandwidth
            // unused, 1-2 KB rows do not).
            const uint32_t RT = g.raw_tiles, box = g.raw_row / ES, nbox = RT * kM / box;
            uint32_t f = (uint32_t)(L0 / tpc), tt = (uint32_t)(L0 % tpc);  // stepped below
            for (uint64_t L = L0; L < L1; L += RT) {
                int ok = 1;
                if (!SELF && (L == L0 || tt == 0)) {
                    if (lane == 0) {
                        // the phasor image is the preceding grid's output: with a programmatic
                        // launch, everything above overlapped that grid, and here it must be done
                        if (g.pdl && L == L0) asm volatile("griddepcontrol.wait;" ::: "memory");
                        ok = mbar_wait(w_empty, wph ^ 1, abort, kWaitBudget);
                        if (ok) {
                            mbar_arrive_expect_tx(w_full, g.img_bytes);
                            bulk_g2s(w_smem, g.plan + (uint64_t)f * g.img_bytes, g.img_bytes, w_full);
                        } else {
                            record_abort(abort, 5);
                        }
                    }
                    ok = __shfl_sync(0xffffffffu, ok, 0);
                    if (!ok) break;
                    w_issued = true;
                    wph ^= 1;
                }
                if (lane == 0) {
                    ok = mbar_wait(&r_empty[rs], rph ^ 1, abort, kWaitBudget);
                    if (ok) {
                        mbar_arrive_expect_tx(&r_full[rs], g.A * (uint32_t)(kM * ES) * RT);
                        uint8_t* dst = r_smem + (size_t)rs * g.raw_bytes;
                        for (uint32_t b = 0; b < nbox; b++)
                            tma_load_3d(dst + (size_t)b * g.A * g.raw_row, &tmap, (int)(tt * kM + b * box), (int)f, 0,
                                        &r_full[rs]);
                    } else {
                        record_abort(abort, 9);
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) break;
                issued_mask |= 1u << rs;
                issued_par = (issued_par & ~(1u << rs)) | (rph << rs);
                if (++rs == RS) { rs = 0; rph ^= 1; }
                tt += RT;
                if (tt == tpc) { tt = 0; f++; }
            }
            // Every bulk copy this warp issued must land before the CTA exits.
            if (lane == 0) {
                if (w_issued && !mbar_wait(w_full, wph ^ 1, &never, kWaitBudget)) record_abort(abort, 6);
                for (uint32_t s = 0; s < RS; s++)
                    if ((issued_mask >> s) & 1u)
                        if (!mbar_wait(&r_full[s], (issued_par >> s) & 1u, &never, kWaitBudget)) record_abort(abort, 10);
            }
            __syncwarp();
        }
    } else if (warp < 2 + kEpiWarps) {
        bool done = false;
        if constexpr (R == 1 && (LOGI == 3 || LOGI == 4) && ES == 4 && kEpiWarps == 4) {
            if (g.transposed) {
                epilogue_transposed<LOGI>(g, tmem, d_cols, nacc, d_full, d_empty, pr_full, abort, L0, L1,
                                          (uint32_t)(warp & 3), (uint32_t)lane);
                done = true;
            }
        }
        if constexpr (PRE) {
            // ---------------- epilogue, one polarisation at a time ----------------
            static_assert(kEpiGroups == 1, "one warp per lane quarter");
            constexpr uint32_t I = 1u << LOGI, rows_per_k = kM / R;
            constexpr int kB16 = R == 4 ? 1 : 2;  // 16-beam chunks at most (4 R NB <= 256 columns)
            const uint32_t q = warp & 3, row = 32 * q + lane, k = row / rows_per_k, s_local = row - k * rows_per_k;
            const uint64_t bstride = (uint64_t)g.F * R * g.U;
            uint32_t dph = 0, f = (uint32_t)(L0 / tpc), tt = (uint32_t)(L0 % tpc);
            bool ok = true;
            for (uint64_t L = L0; L < L1 && ok; L++) {
                float2 pw2[kB16][8];
#pragma unroll
                for (int c = 0; c < kB16; c++)
#pragma unroll
                    for (int j = 0; j < 8; j++) pw2[c][j] = make_float2(0.f, 0.f);
                for (uint32_t p = 0; p < 2; p++) {
                    if (!mbar_wait(&d_full[p], dph, abort, kWaitBudget)) { record_abort(abort, 7); ok = false; break; }
                    tc_fence_after();
                    const uint32_t pa = tmem + ((32 * q) << 16) + p * d_cols + k * 4 * NB;
#pragma unroll
                    for (int c = 0; c < kB16; c++) {
                        if (16u * c >= NB) break;
                        uint32_t hr[16], hi[16], lr[16], li[16];
                        tmem_ld(pa + 16 * c, hr);
                        tmem_ld(pa + NB + 16 * c, hi);
                        tmem_ld(pa + 2 * NB + 16 * c, lr);
                        tmem_ld(pa + 3 * NB + 16 * c, li);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const float2 a = __fadd2_rn(make_float2(__uint_as_float(hr[2 * j]), __uint_as_float(hr[2 * j + 1])),
                                                        make_float2(__uint_as_float(lr[2 * j]), __uint_as_float(lr[2 * j + 1])));
                            const float2 b = __fadd2_rn(make_float2(__uint_as_float(hi[2 * j]), __uint_as_float(hi[2 * j + 1])),
                                                        make_float2(__uint_as_float(li[2 * j]), __uint_as_float(li[2 * j + 1])));
                            pw2[c][j] = __ffma2_rn(a, a, __ffma2_rn(b, b, pw2[c][j]));
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&d_empty[p]);
                }
                if (!ok) break;
                float* obase = g.out + ((uint64_t)f * R + k) * g.U + (tt * rows_per_k + s_local) / I;
#pragma unroll
                for (int c = 0; c < kB16; c++) {
                    if (16u * c >= NB) break;
                    uint32_t first;
                    float(&pw)[16] = *reinterpret_cast<float(*)[16]>(pw2[c]);
                    const int cnt = window_reduce<16, LOGI>(pw, lane, &first);
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        const uint32_t b = 16 * c + first + j;
                        if (j < cnt && b < g.beams) obase[b * bstride] = pw[j];
                    }
                }
                dph ^= 1;
                if (++tt == tpc) { tt = 0; f++; }
            }
            done = true;
        }
        if (!done) {
            // ---------------- epilogue ----------------
            constexpr uint32_t I = 1u << LOGI;
            const uint32_t q = warp & 3;               // TMEM lane quarter this warp may access
            const uint32_t hw = (warp - 2) >> 2;       // which share of the beams
            const uint32_t nbh = NB / kEpiGroups;      // beams per warp, a multiple of 8
            constexpr uint32_t rows_per_k = kM / R;
            const uint32_t row = 32 * q + lane;
            const uint32_t k = row / rows_per_k;
            const uint32_t s_local = row - k * rows_per_k;
            const uint64_t bstride = (uint64_t)g.F * R * g.U;
            uint32_t db = 0, dph = 0;
            uint32_t f = (uint32_t)(L0 / tpc), tt = (uint32_t)(L0 % tpc);  // stepped below
            for (uint64_t L = L0; L < L1; L++) {
                if (!mbar_wait(&d_full[db], dph, abort, kWaitBudget)) { record_abort(abort, 7); break; }
                tc_fence_after();
                const uint32_t u = (tt * rows_per_k + s_local) / I;
                const uint32_t lane_addr = tmem + ((32 * q) << 16) + db * (2 * d_cols);
                float* obase = g.out + ((uint64_t)f * R + k) * g.U + u;
                constexpr int CH = 16 / kEpiGroups;  // beams per TMEM load (16 or 8)
                for (uint32_t bc = hw * nbh; bc < (hw + 1) * nbh; bc += CH) {
                    // Two beams per packed FP32x2 instruction (each lane of the pair rounds
                    // exactly as the scalar add / multiply / FMA would).
                    float2 pw2[CH / 2];
                    float(&pw)[CH] = *reinterpret_cast<float(*)[CH]>(pw2);
                    if (g.stacked) {
                        // per polarisation: (hi + lo) re, (hi + lo) im
    #pragma unroll
                        for (int j = 0; j < CH; j++) pw[j] = 0.f;
    #pragma unroll
                        for (uint32_t p = 0; p < 2; p++) {
                            uint32_t hr[CH], hi[CH], lr[CH], li[CH];
                            const uint32_t pa = lane_addr + p * d_cols + bc;
                            tmem_ld(pa, hr);
                            tmem_ld(pa + NB, hi);
                            tmem_ld(pa + 2 * NB, lr);
                            tmem_ld(pa + 3 * NB, li);
                            tmem_ld_wait();
    #pragma unroll
                            for (int j = 0; j < CH / 2; j++) {
                                const float2 a = __fadd2_rn(make_float2(__uint_as_float(hr[2 * j]), __uint_as_float(hr[2 * j + 1])),
                                                            make_float2(__uint_as_float(lr[2 * j]), __uint_as_float(lr[2 * j + 1])));
                                const float2 b = __fadd2_rn(make_float2(__uint_as_float(hi[2 * j]), __uint_as_float(hi[2 * j + 1])),
                                                            make_float2(__uint_as_float(li[2 * j]), __uint_as_float(li[2 * j + 1])));
                                pw2[j] = __ffma2_rn(a, a, __ffma2_rn(b, b, pw2[j]));
                            }
                        }
                    } else {
                        uint32_t r0[CH], i0[CH], r1[CH], i1[CH];
                        tmem_ld(lane_addr + bc, r0);
                        tmem_ld(lane_addr + NB + bc, i0);
                        tmem_ld(lane_addr + 2 * NB + bc, r1);
                        tmem_ld(lane_addr + 3 * NB + bc, i1);
                        tmem_ld_wait();
    #pragma unroll
                        for (int j = 0; j < CH / 2; j++) {
                            const float2 a0 = make_float2(__uint_as_float(r0[2 * j]), __uint_as_float(r0[2 * j + 1]));
                            const float2 b0 = make_float2(__uint_as_float(i0[2 * j]), __uint_as_float(i0[2 * j + 1]));
                            const float2 a1 = make_float2(__uint_as_float(r1[2 * j]), __uint_as_float(r1[2 * j + 1]));
                            const float2 b1 = make_float2(__uint_as_float(i1[2 * j]), __uint_as_float(i1[2 * j + 1]));
                            pw2[j] = __ffma2_rn(a0, a0, __ffma2_rn(b0, b0, __ffma2_rn(a1, a1, __fmul2_rn(b1, b1))));
                        }
                    }
                    uint32_t first;
                    const int cnt = window_reduce<CH, LOGI>(pw, lane, &first);
    #pragma unroll
                    for (int j = 0; j < CH; j++) {
                        if (j < cnt) {
                            const uint32_t b = bc + first + j;
                            if (b < g.beams) obase[b * bstride] = pw[j];
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&d_empty[db]);
                if (++db == nacc) { db = 0; dph ^= 1; }
                if (++tt == tpc) { tt = 0; f++; }
            }
        }
    } else if (warp < 2 + kEpiWarps + kConvWarps) {
        // ---------------- operand build ----------------
        const uint32_t ct = threadIdx.x - (2 + kEpiWarps) * 32;  // 0 .. 32 kConvWarps - 1
        if constexpr (R == 4) {
            if (split) {
                // Group grp takes local tiles grp, grp + 2, ...: tile `grp` of every raw
                // stage (512 bytes into each 1 KB antenna row) and operand pair 2 grp,
                // 2 grp + 4, ... (the pairs issuer grp consumes).  The CTA's range is a
                // whole number of two-tile stages, so both groups see every stage once.
                constexpr uint32_t kGroup = kConvWarps / 2;
                constexpr uint32_t kMaxTk = kMaxKA / 4 / kGroup;
                const uint32_t cw = ct >> 5, grp = cw / kGroup, gw = cw % kGroup;
                const uint32_t ntk = KA / 4 / kGroup;
                R4Task tk[kMaxTk];
#pragma unroll
                for (uint32_t i = 0; i < kMaxTk; i++) tk[i] = r4_task(gw + i * kGroup, lane, g.A, KA, g.raw_row);
                uint32_t rs = 0, rph = 0, as = 2 * grp, aph = 0;
                for (uint64_t L = L0 + grp; L < L1; L += 2) {
                    if (!mbar_wait(&r_full[rs], rph, abort, kWaitBudget)) { record_abort(abort, 11); break; }
                    if (!mbar_wait(&a_empty[as + 1], aph ^ 1, abort, kWaitBudget)) { record_abort(abort, 8); break; }
                    const uint8_t* raw = r_smem + (size_t)rs * g.raw_bytes + grp * (kM * 4u);
                    uint8_t* op0 = a_smem + (size_t)as * op_bytes;
                    uint8_t* op1 = op0 + op_bytes;
#pragma unroll
                    for (uint32_t i = 0; i < kMaxTk; i++)
                        if (i < ntk) r4_pair_task<PRE>(raw, g.raw_row, op0, op1, tk[i], g.circ);
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&a_full[as + 1]);
                        mbar_arrive(&r_empty[rs]);
                    }
                    as += 4;
                    if (as >= AS) { as -= AS; aph ^= 1; }
                    if (++rs == RS) { rs = 0; rph ^= 1; }
                }
            }
        }
        if constexpr (R == 1 && ES == 4) {
            if (g.direct) {
                // Pair mode without a raw ring: registers hold this tile's words, loaded
                // while the previous tile was built; the next tile's loads go out first.
                const DirectTask dt = direct_task(ct >> 5, lane, g.A, KA);
                const uint32_t* in32 = reinterpret_cast<const uint32_t*>(g.in);
                uint32_t va[kDirectMaxJ][8], vb[kDirectMaxJ][8];
                uint32_t f = (uint32_t)(L0 / tpc), tt = (uint32_t)(L0 % tpc);
                if (L0 < L1) direct_load(in32, g.F, g.T, f, tt * kM, lane, dt, va);
                uint32_t as = 0, aph = 0;
                for (uint64_t L = L0; L < L1; L += 2) {
                    // tile L from va (tile L + 1 into vb first), then tile L + 1 from vb
                    // (tile L + 2 into va first)
#pragma unroll
                    for (int half = 0; half < 2; half++) {
                        if (half == 1 && L + 1 >= L1) break;
                        uint32_t nf = f, ntt = tt + 1;
                        if (ntt == tpc) { ntt = 0; nf++; }
                        if (L + half + 1 < L1) direct_load(in32, g.F, g.T, nf, ntt * kM, lane, dt, half ? va : vb);
                        if (lane < dt.nvalid && L + half + 2 < L1) {
                            // the tile after next into L2: lanes 0-7 prefetch this thread group's rows
                            uint32_t pf = nf, pt = ntt + 1;
                            if (pt == tpc) { pt = 0; pf++; }
                            prefetch_l2_bulk(in32 + ((uint64_t)(dt.a0 + lane) * g.F + pf) * g.T + pt * kM + 32u * dt.j0,
                                             dt.nj * 128u);
                        }
                        if (!mbar_wait(&a_empty[as + 1], aph ^ 1, abort, kWaitBudget)) {
                            record_abort(abort, 8);
                            L = L1;
                            break;
                        }
                        uint8_t* op0 = a_smem + (size_t)as * op_bytes;
                        direct_build(half ? vb : va, op0, op0 + op_bytes, dt);
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&a_full[as + 1]);
                        as += 2;
                        if (as == AS) { as = 0; aph ^= 1; }
                        f = nf;
                        tt = ntt;
                    }
                }
            }
        }
        if constexpr (DIRECT2) {
            if (g.direct) {
                // Pair mode without a raw ring: registers hold the next tile's words, asked for as
                // soon as this tile's are converted; the tile after that is asked into L2.
                constexpr uint32_t kMaxTk = kMaxKA / 2 / kConvWarps;
                const uint32_t ntk = KA / 2 / kConvWarps;
                const uint32_t* in32 = reinterpret_cast<const uint32_t*>(g.in);
                R4Task tk[kMaxTk];
                Direct2 dt[kMaxTk];
                uint2 v[kMaxTk][4];
                uint32_t f = (uint32_t)(L0 / tpc), tt = (uint32_t)(L0 % tpc);
#pragma unroll
                for (uint32_t i = 0; i < kMaxTk; i++) {
                    const uint32_t wt = (ct >> 5) + i * kConvWarps;
                    tk[i] = r2_task(wt, lane, g.A, KA, 0);
                    dt[i] = direct2_task(wt, lane);
                    if (i >= ntk) tk[i].nvalid = 0;
                    if (L0 < L1) direct2_load(in32, g.F, g.T, f, tt * kM, dt[i], tk[i].nvalid, v[i]);
                }
                uint32_t as = 0, aph = 0;
                for (uint64_t L = L0; L < L1; L++) {
                    if (++tt == tpc) { tt = 0; f++; }
                    if (!mbar_wait(&a_empty[as + 1], aph ^ 1, abort, kWaitBudget)) { record_abort(abort, 8); break; }
                    uint8_t* op0 = a_smem + (size_t)as * op_bytes;
#pragma unroll
                    for (uint32_t i = 0; i < kMaxTk; i++) {
                        if (i < ntk) r2_pair_words<false>(v[i], op0, op0 + op_bytes, tk[i], 0);
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&a_full[as + 1]);
                    if (L + 1 < L1) {
#pragma unroll
                        for (uint32_t i = 0; i < kMaxTk; i++)
                            direct2_load(in32, g.F, g.T, f, tt * kM, dt[i], tk[i].nvalid, v[i]);
                    }
                    // antenna ct of the tile after next (512 bytes)
                    if (ct < g.A && L + 2 < L1) {
                        uint32_t pf = f, pt = tt + 1;
                        if (pt == tpc) { pt = 0; pf++; }
                        prefetch_l2_bulk(in32 + ((uint64_t)ct * g.F + pf) * g.T + pt * kM, kM * 4);
                    }
                    as += 2;
                    if (as == AS) { as = 0; aph ^= 1; }
                }
            }
        }
        if (!(R == 4 && split) && !g.direct) {
        // R = 4 pair mode: this warp's warp-tasks (KA / 4 of them over kConvWarps warps),
        // addresses fixed for the kernel
        constexpr uint32_t kMaxT4 = kMaxKA / 4 / kConvWarps;
        const uint32_t nt4 = KA / 4 / kConvWarps;
        R4Task t4[kMaxT4];
        if constexpr (R == 4) {
#pragma unroll
            for (uint32_t i = 0; i < kMaxT4; i++) t4[i] = r4_task((ct >> 5) + i * kConvWarps, lane, g.A, KA, g.raw_row);
        }
        // R = 2 pair mode: KA / 2 warp-tasks
        constexpr uint32_t kMaxT2 = kMaxKA / 2 / kConvWarps;
        const uint32_t nt2 = KA / 2 / kConvWarps;
        R4Task t2[kMaxT2];
        if constexpr (R == 2 && !SELF) {
#pragma unroll
            for (uint32_t i = 0; i < kMaxT2; i++) t2[i] = r2_task((ct >> 5) + i * kConvWarps, lane, g.A, KA, g.raw_row);
        }
        R1Task t1;
        if constexpr (R == 1 && ES == 4) t1 = r1_task(ct >> 5, lane, g.A, KA, g.raw_row);
        uint32_t rs = 0, rph = 0, as = 0, aph = 0;
        uint32_t sub = 0;  // tile within the raw stage (CTA ranges are stage-aligned)
        bool ok = true;
        for (uint64_t L = L0; L < L1 && ok; L++) {
            if (sub == 0) {
                if (!mbar_wait(&r_full[rs], rph, abort, kWaitBudget)) { record_abort(abort, 11); break; }
            }
            // this tile inside the stage: box (sub * 128 / box), column (sub * 128 % box)
            const uint32_t sb = sub * kM, box = g.raw_row / ES;
            const uint8_t* raw = r_smem + (size_t)rs * g.raw_bytes + (sb / box) * g.A * g.raw_row + (sb % box) * ES;
            if (pair) {
                // Both polarisations in one pass into stages as, as + 1 (AS is even).
                if (!mbar_wait(&a_empty[as + 1], aph ^ 1, abort, kWaitBudget)) {
                    record_abort(abort, 8);
                    break;
                }
                uint8_t* op0 = a_smem + (size_t)as * op_bytes;
                uint8_t* op1 = op0 + op_bytes;
                if constexpr (R == 4) {
#pragma unroll
                    for (uint32_t i = 0; i < kMaxT4; i++)
                        if (i < nt4) r4_pair_task<PRE>(raw, g.raw_row, op0, op1, t4[i], g.circ);
                } else if constexpr (ES == 8) {
                    build_operand_h16_pair(raw, g.raw_row, op0, op1, g.A, KA, ct);
                } else if constexpr (R == 1) {
                    r1_pair_task(raw, g.raw_row, op0, op1, t1);
                } else if constexpr (R == 2 && !SELF) {
                    // one pass: 6144 tiles of 8 to 32 antennas, 16 beams, 51.4-53.4 -> 45.5-53.4 us,
                    // 40 antennas 78.4 -> 72.2; inside SELF the two passes stay ahead (2048 tiles of
                    // 28 antennas: 24.7 us, 28.8 in one pass)
#pragma unroll
                    for (uint32_t i = 0; i < kMaxT2; i++)
                        if (i < nt2) r2_pair_task<PRE>(raw, g.raw_row, op0, op1, t2[i], g.circ);
                } else {
                    build_operand_pair<R>(raw, g.raw_row, op0, op1, g.A, KA, ct);
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[as + 1]);
                as += 2;
                if (as == AS) { as = 0; aph ^= 1; }
            } else {
                for (int p = 0; p < 2; p++) {
                    if (!mbar_wait(&a_empty[as], aph ^ 1, abort, kWaitBudget)) { record_abort(abort, 8); ok = false; break; }
                    if constexpr (ES == 8) build_operand_h16(raw, g.raw_row, a_smem + (size_t)as * op_bytes, g.A, KA, p, ct);
                    else build_operand<R>(raw, g.raw_row, a_smem + (size_t)as * op_bytes, g.A, KA, p, ct);
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&a_full[as]);
                    if (++as == AS) { as = 0; aph ^= 1; }
                }
                if (!ok) break;
            }
            if (++sub == g.raw_tiles) {
                sub = 0;
                __syncwarp();
                if (lane == 0) mbar_arrive(&r_empty[rs]);
                if (++rs == RS) { rs = 0; rph ^= 1; }
            }
        }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, tmem_cols);
    }
}

using TcKernel = void (*)(const TcArgs, const CUtensorMap);

}  // namespace

// The instantiations of the other source files, and their status words.
const void* tc_pre_kernel(uint64_t rate, uint64_t integration);           // beamform_tc_pre.cu
int tc_pre_status_take(uint32_t* status);
const void* tc_self_kernel(uint64_t rate, uint64_t integration);          // beamform_tc_self.cu
const void* tc_direct2_kernel(uint64_t integration);
int tc_self_status_take(uint32_t* status);

inline uint32_t tc_log2(uint64_t integration) {
    uint32_t logi = 0;
    while ((1ull << logi) < integration) logi++;
    return logi;
}

}  // namespace bb
