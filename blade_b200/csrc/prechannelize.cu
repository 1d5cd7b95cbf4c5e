// Pre-beamformer stages of the ATA ModeB bundle on CI8 voltages, exact in FP16:
// Cast<CI8,CF32> -> Channelizer(rate R <= 4) -> [Polarizer XY -> LR]
// (include/blade/bundles/ata/mode_b.hh:99-139; src/modules/channelizer/
// base.cc:59-138 + channelizer.cu:5-19, src/modules/polarizer/polarizer.cu:17-23):
//   out[a, f*R + k, s, p] = sum_j (-1)^j x[a, f, s*R + j, p] e^{-2 pi i j k / R}
// (the fftshifted R-point DFT), then (X, Y) -> (X + iY, X - iY) when circular.
// CI8 components are integers in [-128, 127], so every output component is an
// integer of magnitude <= 1024: the FP16 output holds the same values the FP32
// module chain computes, and the tensor-core beamformer reads them exactly.
#include "common.cuh"

namespace bb {
namespace {

// One thread per (a, f, spectrum s): R sample words in, R dual-polarisation
// CF16 samples out (8 bytes each, consecutive threads write consecutive s).  Each
// thread keeps the loads of kSpt spectra in flight before it computes any of them.
constexpr int kSpt = 4;

template <int R>
__device__ __forceinline__ void load_spectrum(const uint32_t* src, uint32_t (&ws)[R]) {
    if constexpr (R == 4) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(src));
        ws[0] = v.x;
        ws[1 % R] = v.y;
        ws[2 % R] = v.z;
        ws[3 % R] = v.w;
    } else if constexpr (R == 2) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(src));
        ws[0] = v.x;
        ws[1 % R] = v.y;
    } else {
        ws[0] = __ldg(src);
    }
}

template <int R, bool CIRC>
__device__ __forceinline__ void spectrum_out(const uint32_t (&ws)[R], uint2* __restrict__ out, uint64_t af,
                                             uint32_t S, uint32_t s) {
    float xr[2][R], xi[2][R];
#pragma unroll
    for (int j = 0; j < R; j++) {
        const uint32_t w = ws[j];
        const float sg = (R > 1 && (j & 1)) ? -1.f : 1.f;  // fftshift pre-multiply (even R)
        xr[0][j] = sg * (float)(int8_t)(w & 0xFFu);
        xi[0][j] = sg * (float)(int8_t)((w >> 8) & 0xFFu);
        xr[1][j] = sg * (float)(int8_t)((w >> 16) & 0xFFu);
        xi[1][j] = sg * (float)(int8_t)(w >> 24);
    }
#pragma unroll
    for (int k = 0; k < R; k++) {
        float zr[2], zi[2];
#pragma unroll
        for (int p = 0; p < 2; p++) {
            zr[p] = 0.f;
            zi[p] = 0.f;
#pragma unroll
            for (int j = 0; j < R; j++) {
                // e^{-2 pi i j k / R} for R <= 4 is one of 1, -i, -1, i
                const int q = (j * k * (4 / R)) & 3;
                const float re = xr[p][j], im = xi[p][j];
                zr[p] += q == 0 ? re : q == 1 ? im : q == 2 ? -re : -im;
                zi[p] += q == 0 ? im : q == 1 ? -re : q == 2 ? -im : re;
            }
        }
        if (CIRC) {
            const float lr = zr[0] - zi[1], li = zi[0] + zr[1];  // X + iY
            const float rr = zr[0] + zi[1], ri = zi[0] - zr[1];  // X - iY
            zr[0] = lr;
            zi[0] = li;
            zr[1] = rr;
            zi[1] = ri;
        }
        const __half2 h0 = __floats2half2_rn(zr[0], zi[0]), h1 = __floats2half2_rn(zr[1], zi[1]);
        uint2 o;
        o.x = *reinterpret_cast<const uint32_t*>(&h0);
        o.y = *reinterpret_cast<const uint32_t*>(&h1);
        out[(af * R + k) * (uint64_t)S + s] = o;
    }
}

template <int R, bool CIRC>
__global__ void __launch_bounds__(256) prechannelize_kernel(const uint32_t* __restrict__ in,
                                                            uint2* __restrict__ out, uint64_t AF, uint32_t S) {
    const uint64_t n = AF * S;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; base < n; base += kSpt * stride) {
        uint32_t ws[kSpt][R];
#pragma unroll
        for (int q = 0; q < kSpt; q++) {
            const uint64_t i = base + q * stride;
            if (i < n) load_spectrum<R>(in + i * R, ws[q]);  // spectrum i = af * S + s starts at word i * R
        }
#pragma unroll
        for (int q = 0; q < kSpt; q++) {
            const uint64_t i = base + q * stride;
            if (i < n) {
                const uint64_t af = i / S;
                spectrum_out<R, CIRC>(ws[q], out, af, S, (uint32_t)(i - af * S));
            }
        }
    }
}

template <int R>
void launch_pre(const uint32_t* in, uint2* out, uint64_t AF, uint32_t S, bool circ, cudaStream_t st) {
    const unsigned grid = grid_for(AF * S, 256);
    if (circ) prechannelize_kernel<R, true><<<grid, 256, 0, st>>>(in, out, AF, S);
    else prechannelize_kernel<R, false><<<grid, 256, 0, st>>>(in, out, AF, S);
}

}  // namespace
}  // namespace bb

extern "C" int blade_prechannelize_cf16(const void* in, void* out, uint64_t A, uint64_t F, uint64_t T, uint64_t P,
                                        uint64_t rate, int circular, blade_stream_t stream) {
    using namespace bb;
    if (P != 2) return set_error(BLADE_ERROR, "blade_prechannelize_cf16: P must be 2");
    if (rate != 1 && rate != 2 && rate != 4)
        return set_error(BLADE_ERROR, "blade_prechannelize_cf16: rate must be 1, 2 or 4 (got %llu)",
                         (unsigned long long)rate);
    if (T % rate != 0)
        return set_error(BLADE_ERROR, "blade_prechannelize_cf16: the number of time samples (%llu) should be "
                         "divisible by the rate (%llu)", (unsigned long long)T, (unsigned long long)rate);
    if (T / rate > 0xFFFFFFFFull) return set_error(BLADE_ERROR, "blade_prechannelize_cf16: T too large");
    if (A * F * T == 0) return BLADE_SUCCESS;
    if (!in || !out) return set_error(BLADE_ERROR, "blade_prechannelize_cf16: null buffer");
    if ((reinterpret_cast<uintptr_t>(in) & (4 * rate - 1)) || (reinterpret_cast<uintptr_t>(out) & 7))
        return set_error(BLADE_ERROR, "blade_prechannelize_cf16: input must be (4 x rate)-byte and output 8-byte "
                         "aligned");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const uint32_t* x = static_cast<const uint32_t*>(in);
    uint2* y = static_cast<uint2*>(out);
    const uint32_t S = (uint32_t)(T / rate);
    if (rate == 1) launch_pre<1>(x, y, A * F, S, circular != 0, st);
    else if (rate == 2) launch_pre<2>(x, y, A * F, S, circular != 0, st);
    else launch_pre<4>(x, y, A * F, S, circular != 0, st);
    return check_launch("blade_prechannelize_cf16");
}

// ---- incoherent beam of ModeB with the detector, on the CF16 fine channels ----
// Beamformer::ATA's incoherent beam (src/modules/beamformer/beamformer.cu:64-78:
// sum_a |x * w[0]|^2 per polarisation, square-rooted when the detector follows,
// mode_b.hh:146-147) followed by the Stokes-I detector (detector.cu:34-51), which
// squares the root back: out[f, u] = sum_{t in window u} sum_p sum_a
// |x[a,f,t,p]|^2 |w[0,a,f,0,p]|^2.  One thread per sample (coalesced 8-byte
// loads), the window closed with lane shuffles; I is a power of two <= 32.
namespace bb {
namespace {

__global__ void __launch_bounds__(256) incoherent_detect_cf16_kernel(const uint2* __restrict__ x,
                                                                     const float2* __restrict__ w0, float* out,
                                                                     uint32_t A, uint32_t F, uint32_t T, uint32_t I) {
    extern __shared__ float g2[];  // |w[0, a, f, 0, p]|^2, [a][p]
    const uint32_t f = blockIdx.y;
    for (uint32_t i = threadIdx.x; i < 2 * A; i += blockDim.x) {
        const float2 w = w0[((uint64_t)(i >> 1) * F + f) * 2 + (i & 1)];
        g2[i] = w.x * w.x + w.y * w.y;
    }
    __syncthreads();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    float acc = 0.f;
    if (t < T) {
        for (uint32_t a = 0; a < A; a++) {
            const uint2 v = __ldg(x + ((uint64_t)a * F + f) * T + t);
            const float2 p0 = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
            const float2 p1 = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
            acc = fmaf(p0.x * p0.x + p0.y * p0.y, g2[2 * a], acc);
            acc = fmaf(p1.x * p1.x + p1.y * p1.y, g2[2 * a + 1], acc);
        }
    }
    for (uint32_t off = 1; off < I; off <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (t < T && (t % I) == 0) out[(uint64_t)f * (T / I) + t / I] = acc;
}

}  // namespace
}  // namespace bb

extern "C" int blade_incoherent_detect_cf16(const void* in, const void* phasors, void* out, uint64_t A, uint64_t F,
                                            uint64_t T, uint64_t P, uint64_t integration, blade_stream_t stream) {
    using namespace bb;
    if (P != 2) return set_error(BLADE_ERROR, "blade_incoherent_detect_cf16: P must be 2");
    if (integration == 0 || integration > 32 || (integration & (integration - 1)) != 0 || T % integration != 0)
        return set_error(BLADE_ERROR, "blade_incoherent_detect_cf16: integration must be a power of two <= 32 "
                         "dividing T");
    if (A * F * T == 0) return BLADE_SUCCESS;
    if (F > 65535 || T >= (1ull << 31)) return set_error(BLADE_ERROR, "blade_incoherent_detect_cf16: too large");
    if (!in || !phasors || !out) return set_error(BLADE_ERROR, "blade_incoherent_detect_cf16: null buffer");
    if ((reinterpret_cast<uintptr_t>(in) & 7) || (reinterpret_cast<uintptr_t>(out) & 3))
        return set_error(BLADE_ERROR, "blade_incoherent_detect_cf16: misaligned buffer");
    const size_t smem = 2 * A * sizeof(float);
    if (int rc = ensure_smem(reinterpret_cast<const void*>(incoherent_detect_cf16_kernel), smem)) return rc;
    const dim3 grid((unsigned)((T + 255) / 256), (unsigned)F);
    incoherent_detect_cf16_kernel<<<grid, 256, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint2*>(in), static_cast<const float2*>(phasors), static_cast<float*>(out), (uint32_t)A,
        (uint32_t)F, (uint32_t)T, (uint32_t)integration);
    return check_launch("blade_incoherent_detect_cf16");
}

// ---- the same beam straight from the CI8 block ---------------------------------
// For a chain that never stores the fine channels: one thread per spectrum (a warp
// reads 32 x 4 R consecutive bytes of an antenna, four antennas in flight), the
// rate-R fftshifted transform and the circular basis in registers (exact integers),
// |x|^2 |w[0]|^2 summed over antennas and polarisations, windows closed with lane
// shuffles.  A 28-antenna block of 176 MB at R = 4: 45 us (bound by the FP32
// pipe: transforms, conversions and squares), where the kernel above reads 352 MB of fine
// channels in 57; 48 with CTAs of 256 threads, which close their last wave later, and 51
// when each load also computed its address from the antenna; transforming in FP32
// instead of FP16 pairs was 4 % slower.
namespace bb {
namespace {

// A complex value of both polarisations, halves = (pol 0, pol 1).
struct H2 {
    __half2 re, im;
};

__device__ __forceinline__ __half2 half2_of(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }

// R sample words -> the R fine channels, exact: 1152 + x through the 0x64 exponent
// byte; the biases cancel in differences, and x + y = ((1152 + x) - 2304) + (1152 + y).
template <int R>
__device__ __forceinline__ void fine_channels(const uint32_t (&w)[R], H2 (&z)[R]) {
    const __half2 h2304 = half2_of(0x68806880u);
    __half2 re[R], im[R];
#pragma unroll
    for (int j = 0; j < R; j++) {
        const uint32_t x = w[j] ^ 0x80808080u;
        re[j] = half2_of(__byte_perm(x, 0x64646464u, 0x4240));
        im[j] = half2_of(__byte_perm(x, 0x64646464u, 0x4341));
    }
    if constexpr (R == 2) {
        z[0] = {__hsub2(re[0], re[1]), __hsub2(im[0], im[1])};
        z[1] = {__hadd2(__hsub2(re[0], h2304), re[1]), __hadd2(__hsub2(im[0], h2304), im[1])};
    } else {
        const __half2 aR = __hadd2(__hsub2(re[0], h2304), re[2]), bR = __hadd2(__hsub2(re[1], h2304), re[3]);
        const __half2 aI = __hadd2(__hsub2(im[0], h2304), im[2]), bI = __hadd2(__hsub2(im[1], h2304), im[3]);
        const __half2 cR = __hsub2(re[0], re[2]), dR = __hsub2(re[1], re[3]);
        const __half2 cI = __hsub2(im[0], im[2]), dI = __hsub2(im[1], im[3]);
        z[0] = {__hsub2(aR, bR), __hsub2(aI, bI)};  // x0 - x1 + x2 - x3
        z[1] = {__hsub2(cR, dI), __hadd2(cI, dR)};  // x0 + i x1 - x2 - i x3
        z[2] = {__hadd2(aR, bR), __hadd2(aI, bI)};
        z[3] = {__hadd2(cR, dI), __hsub2(cI, dR)};
    }
}

constexpr uint32_t kIncThreads = 128;

template <int R, bool CIRC>
__global__ void __launch_bounds__(kIncThreads) incoherent_detect_ci8_kernel(const uint32_t* __restrict__ x,
                                                                    const float2* __restrict__ w0,
                                                                    float* __restrict__ out, uint32_t A, uint32_t F,
                                                                    uint32_t S, uint32_t I) {
    extern __shared__ float2 gw[];  // (|w[0, a, f R + k, 0, 0]|^2, |w[0, a, f R + k, 0, 1]|^2), [a][k]
    constexpr uint32_t kAhead = 4;
    const uint32_t f = blockIdx.y;
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t* src = x + ((uint64_t)f * S + (s < S ? s : 0u)) * R;
    const uint64_t astride = (uint64_t)F * S * R;
    // the next antennas' samples are on their way while these are summed
    uint32_t wa[kAhead][R], wb[kAhead][R];
    auto load = [&](uint32_t a0, uint32_t (&w)[kAhead][R]) {
#pragma unroll
        for (uint32_t u = 0; u < kAhead; u++)
            if (a0 + u < A) load_spectrum<R>(src + u * astride, w[u]);
        src += kAhead * astride;
    };
    load(0, wa);
    for (uint32_t i = threadIdx.x; i < A * R; i += blockDim.x) {
        const uint32_t a = i / R, k = i % R;
        const float2* w = w0 + (((uint64_t)a * F + f) * R + k) * 2;
        const float2 u = w[0], v = w[1];
        gw[i] = make_float2(u.x * u.x + u.y * u.y, v.x * v.x + v.y * v.y);
    }
    __syncthreads();
    float2 acc[R];
#pragma unroll
    for (int k = 0; k < R; k++) acc[k] = make_float2(0.f, 0.f);
    const float2* g = gw;
    auto sum = [&](uint32_t a0, const uint32_t (&w)[kAhead][R]) {
#pragma unroll
        for (uint32_t u = 0; u < kAhead; u++) {
            if (a0 + u >= A) break;
            H2 z[R];
            fine_channels<R>(w[u], z);
#pragma unroll
            for (int k = 0; k < R; k++) {
                float2 re = __half22float2(z[k].re), im = __half22float2(z[k].im);
                if constexpr (CIRC) {
                    const float2 r = re, i = im;
                    re = make_float2(r.x - i.y, r.x + i.y);
                    im = make_float2(i.x + r.y, i.x - r.y);
                }
                acc[k] = __ffma2_rn(__ffma2_rn(re, re, __fmul2_rn(im, im)), g[u * R + k], acc[k]);
            }
        }
        g += kAhead * R;
    };
    for (uint32_t a0 = 0; a0 < A; a0 += 2 * kAhead) {
        load(a0 + kAhead, wb);
        sum(a0, wa);
        load(a0 + 2 * kAhead, wa);
        sum(a0 + kAhead, wb);
    }
#pragma unroll
    for (int k = 0; k < R; k++) {
        float v = acc[k].x + acc[k].y;
        for (uint32_t off = 1; off < I; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (s < S && (s % I) == 0) out[((uint64_t)f * R + k) * (S / I) + s / I] = v;
    }
}

}  // namespace
}  // namespace bb

extern "C" int blade_incoherent_detect_ci8(const void* in, const void* phasors, void* out, uint64_t A, uint64_t F,
                                           uint64_t T, uint64_t P, uint64_t rate, uint64_t integration, int circular,
                                           blade_stream_t stream) {
    using namespace bb;
    const char* who = "blade_incoherent_detect_ci8";
    if (P != 2) return set_error(BLADE_ERROR, "%s: P must be 2", who);
    if (rate != 2 && rate != 4) return set_error(BLADE_ERROR, "%s: rate must be 2 or 4", who);
    if (integration == 0 || integration > 32 || (integration & (integration - 1)) != 0 || T % (rate * integration) != 0)
        return set_error(BLADE_ERROR, "%s: integration must be a power of two <= 32, rate x integration dividing T", who);
    if (A * F * T == 0) return BLADE_SUCCESS;
    if (F > 65535 || T >= (1ull << 31) || A * rate * sizeof(float2) > 160 * 1024)
        return set_error(BLADE_ERROR, "%s: too large", who);
    if (!in || !phasors || !out) return set_error(BLADE_ERROR, "%s: null buffer", who);
    if ((reinterpret_cast<uintptr_t>(in) & (4 * rate - 1)) || (reinterpret_cast<uintptr_t>(out) & 3))
        return set_error(BLADE_ERROR, "%s: misaligned buffer", who);
    const size_t smem = A * rate * sizeof(float2);
    const uint32_t S = (uint32_t)(T / rate);
    const dim3 grid((unsigned)ceil_div(S, kIncThreads), (unsigned)F);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const auto fn = rate == 4 ? (circular ? incoherent_detect_ci8_kernel<4, true> : incoherent_detect_ci8_kernel<4, false>)
                              : (circular ? incoherent_detect_ci8_kernel<2, true> : incoherent_detect_ci8_kernel<2, false>);
    if (int rc = ensure_smem(reinterpret_cast<const void*>(fn), smem)) return rc;
    fn<<<grid, kIncThreads, smem, st>>>(static_cast<const uint32_t*>(in), static_cast<const float2*>(phasors),
                                static_cast<float*>(out), (uint32_t)A, (uint32_t)F, S, (uint32_t)integration);
    return check_launch(who);
}
