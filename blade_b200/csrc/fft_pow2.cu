// Channelizer for power-of-two rates 32 .. 4096, registers between one or two
// shared-memory exchanges (reference: src/modules/channelizer/base.cc:9-146 and
// channelizer.cu:5-19 + cuFFT; layout of tests/modules/channelizer/advanced.py:49-65).
//
// N = R1 R2 (R3), n = t + (N / R1) m, t = R3 u + v, k = k1 + R1 k2 + R1 R2 k3:
//   Y[k1][t]     = w_N^(t k1)       DFT_R1 over m of x
//   Z[k1][k2][v] = w_(R2 R3)^(v k2) DFT_R2 over u of Y
//   X[k]         = DFT_R3 over v of Z             (two factors: X = DFT_R2 of Y)
// A unit is a pair of transforms (fft_regs.cuh): the two polarisations of one
// spectrum, or two consecutive spectra of a single-polarisation block, 16 bytes per
// element either way.  A CTA holds G units of one (a, f): stage 1 loads R1 samples
// per task straight into registers (consecutive tasks, consecutive samples), the
// last stage stores straight from registers with the units of a bin side by side
// (16 G contiguous bytes per bin of the [k][s][p] output).  The middle stage reads
// and writes the same shared-memory words, so the stages need one barrier each.
//
// Shared-memory rows: k1 rows of LD1 elements per unit, LD1 = N / R1 + (G mod 8),
// units LDs = R1 LD1 + 1 apart.  Consecutive tasks of stage 1 write consecutive
// words; eight consecutive tasks of the last stage read eight distinct 16-byte bank
// groups whether they cover eight units or fewer units and several k1 rows.
//
// Bound by HBM: 8 antennas x 192 channels x 8192 samples, two polarisations (403 MB
// in and out): 70 us at rates 32, 64 and 256 (5.7 TB/s), 73 at 128, 78 at 1024, 89 at
// 512, 112 at 4096 (one unit per CTA there: 16-byte runs), against 263 to 470 us for
// passes of radix 8 and 4 through shared memory on one transform at a time.  The radix-16
// stages carry their constants to twice FP32's precision (0 to 2 % of that, 4 to 6 on blocks
// that stay in L2): rounded, two of them put 5.3e-8 on the mean power at rate 256 and three
// 7.7e-8 at 4096, where passes of radix 8 and 4 gave 4.0e-8 and 5.7e-8; now 0.7e-8 and 0.9e-8.
#include "channelize.cuh"
#include "fft_regs.cuh"

namespace bb {
namespace {

using namespace fft;

constexpr uint32_t kPowThreads = 256;

template <int R1, int R2, int R3>
struct Geometry {
    static constexpr uint32_t N = R1 * R2 * R3, M1 = R2 * R3;
    // units per CTA at most: one task of 8 values per thread for the small rates,
    // two thirds of an SM's shared memory at most for the large ones
    static constexpr uint32_t kPoints = N <= 64 ? 2048 : 4096;
    static constexpr uint32_t kTwiddles = (R1 - 1) * M1 + (R3 > 1 ? (R2 - 1) * R3 : 0);
    static constexpr uint32_t kMaxG = kPoints / N;
    static __host__ __device__ constexpr uint32_t ld1(uint32_t G) { return M1 + (G < 8 ? G : 0); }
    static __host__ __device__ constexpr uint32_t lds(uint32_t G) { return R1 * ld1(G) + 1; }
};

template <int R1, int R2, int R3, int P, bool CI8>
__global__ void __launch_bounds__(kPowThreads, R1 == 16 ? 2 : 3)
    fft_pow2_kernel(const void* __restrict__ vin, float2* __restrict__ out, uint64_t rows, uint32_t S, uint32_t log_g,
                    int circular) {
    using Geo = Geometry<R1, R2, R3>;
    constexpr uint32_t N = Geo::N, M1 = Geo::M1;
    extern __shared__ __align__(16) float4 sm[];
    const uint32_t G = 1u << log_g, LD1 = Geo::ld1(G), LDs = Geo::lds(G);
    const uint32_t Su = P == 2 ? S : (S + 1) / 2;  // units per row
    const uint32_t ngr = (Su + G - 1) >> log_g;
    auto put = [&](uint32_t i, const c2& v) { sm[i] = make_float4(v.re.x, v.re.y, v.im.x, v.im.y); };
    auto get = [&](uint32_t i) {
        const float4 q = sm[i];
        return c2{make_float2(q.x, q.y), make_float2(q.z, q.w)};
    };
    // w_N^(t k1) at tw1[(k1 - 1) M1 + t], w_M1^(v k2) at tw2[(k2 - 1) R3 + v]
    float2* tw1 = reinterpret_cast<float2*>(sm + G * LDs);
    float2* tw2 = tw1 + (R1 - 1) * M1;
    for (uint32_t i = threadIdx.x; i < (R1 - 1) * M1; i += kPowThreads) tw1[i] = root((i / M1 + 1) * (i % M1), N);
    if constexpr (R3 > 1)
        for (uint32_t i = threadIdx.x; i < (R2 - 1) * R3; i += kPowThreads) tw2[i] = root((i / R3 + 1) * (i % R3), M1);
    __syncthreads();
    for (uint64_t grp = blockIdx.x; grp < rows * ngr; grp += gridDim.x) {
        const uint64_t af = grp / ngr;
        const uint32_t u0 = (uint32_t)(grp - af * ngr) << log_g, gn = min(G, Su - u0);
        for (uint32_t task = threadIdx.x; task < gn * M1; task += kPowThreads) {
            const uint32_t t = task % M1, u = task / M1;
            c2 v[R1];
            if constexpr (P == 2) {
                const uint64_t base = (af * S + u0 + u) * N + t;
#pragma unroll
                for (int m = 0; m < R1; m++)
                    v[m] = CI8 ? pair_ci8(__ldg(static_cast<const uint32_t*>(vin) + base + m * M1))
                               : pair(ldg_nc_f4(static_cast<const float4*>(vin) + base + m * M1));
            } else {
                const uint32_t s = 2 * (u0 + u);
                const float2* src = static_cast<const float2*>(vin) + (af * S + s) * N + t;
                const bool two = s + 1 < S;
#pragma unroll
                for (int m = 0; m < R1; m++) {
                    const float2 a = __ldg(src + m * M1), b = two ? __ldg(src + N + m * M1) : make_float2(0.f, 0.f);
                    v[m] = c2{make_float2(a.x, b.x), make_float2(a.y, b.y)};
                }
            }
            dft<R1, true>(v);
            twiddle_column<R1>(v, tw1 + t, M1);
#pragma unroll
            for (int k1 = 0; k1 < R1; k1++) put(u * LDs + k1 * LD1 + t, v[k1]);
        }
        __syncthreads();
        if constexpr (R3 > 1) {
            for (uint32_t task = threadIdx.x; task < gn * (R1 * R3); task += kPowThreads) {
                const uint32_t x = task % R3, k1 = (task / R3) % R1, u = task / (R1 * R3);
                const uint32_t base = u * LDs + k1 * LD1 + x;
                c2 v[R2];
#pragma unroll
                for (int i = 0; i < R2; i++) v[i] = get(base + i * R3);
                dft<R2, true>(v);
                twiddle_column<R2>(v, tw2 + x, R3);
#pragma unroll
                for (int k2 = 0; k2 < R2; k2++) put(base + k2 * R3, v[k2]);
            }
            __syncthreads();
        }
        constexpr int RL = R3 > 1 ? R3 : R2;  // radix of the last stage
        for (uint32_t task = threadIdx.x; task < (N / RL) << log_g; task += kPowThreads) {
            const uint32_t u = task & (G - 1), q = task >> log_g;
            if (u >= gn) continue;
            const uint32_t k1 = q % R1, k2 = q / R1;  // k2 = 0 with two factors
            const uint32_t base = u * LDs + k1 * LD1 + k2 * RL;
            c2 v[RL];
#pragma unroll
            for (int i = 0; i < RL; i++) v[i] = get(base + i);
            dft<RL, true>(v);
#pragma unroll
            for (int k3 = 0; k3 < RL; k3++) {
                const uint32_t kout = (q + (N / RL) * k3 + N / 2) & (N - 1);  // fftshift; q = k1 + R1 k2
                if constexpr (P == 2) {
                    stg_f4(out + ((af * N + kout) * S + u0 + u) * 2, unpair(v[k3], circular));
                } else {
                    const uint32_t s = 2 * (u0 + u);
                    float2* dst = out + (af * N + kout) * S + s;
                    if ((S & 1u) == 0) {
                        stg_f4(dst, unpair(v[k3], 0));
                    } else {
                        dst[0] = make_float2(v[k3].re.x, v[k3].im.x);
                        if (s + 1 < S) dst[1] = make_float2(v[k3].re.y, v[k3].im.y);
                    }
                }
            }
        }
        __syncthreads();
    }
}

template <int R1, int R2, int R3, int P, bool CI8>
int launch_pow2(const void* in, float2* out, uint64_t rows, uint32_t S, int circular, cudaStream_t s) {
    using Geo = Geometry<R1, R2, R3>;
    const uint32_t Su = P == 2 ? S : (S + 1) / 2;
    uint32_t log_g = 0;
    while ((2u << log_g) <= Geo::kMaxG && (1u << log_g) < Su) log_g++;
    const uint32_t G = 1u << log_g;
    const size_t smem = (size_t)G * Geo::lds(G) * sizeof(float4) + Geo::kTwiddles * sizeof(float2);
    const auto fn = fft_pow2_kernel<R1, R2, R3, P, CI8>;
    if (int rc = ensure_smem(reinterpret_cast<const void*>(fn), smem)) return rc;
    const uint64_t groups = rows * ceil_div(Su, G), cap = (uint64_t)sm_count() * (R1 == 16 ? 2 : 3);
    fn<<<(unsigned)(groups < cap ? groups : cap), kPowThreads, smem, s>>>(in, out, rows, S, log_g, circular);
    return BLADE_SUCCESS;
}

template <int P, bool CI8>
int dispatch_pow2(uint64_t rate, const void* in, float2* out, uint64_t rows, uint32_t S, int circular, cudaStream_t s) {
    switch (rate) {
        case 32: return launch_pow2<8, 4, 1, P, CI8>(in, out, rows, S, circular, s);
        case 64: return launch_pow2<8, 8, 1, P, CI8>(in, out, rows, S, circular, s);
        case 128: return launch_pow2<16, 8, 1, P, CI8>(in, out, rows, S, circular, s);
        case 256: return launch_pow2<16, 16, 1, P, CI8>(in, out, rows, S, circular, s);
        case 512: return launch_pow2<8, 8, 8, P, CI8>(in, out, rows, S, circular, s);
        case 1024: return launch_pow2<16, 8, 8, P, CI8>(in, out, rows, S, circular, s);
        case 2048: return launch_pow2<16, 16, 8, P, CI8>(in, out, rows, S, circular, s);
        default: return launch_pow2<16, 16, 16, P, CI8>(in, out, rows, S, circular, s);
    }
}

}  // namespace

int channelize_pow2(const void* in, bool ci8, float2* out, uint64_t A, uint64_t F, uint64_t T, uint64_t P,
                    uint64_t rate, int circular, cudaStream_t s) {
    const uint64_t rows = A * F;
    const uint32_t S = (uint32_t)(T / rate);
    int rc;
    if (P == 2) rc = ci8 ? dispatch_pow2<2, true>(rate, in, out, rows, S, circular, s)
                         : dispatch_pow2<2, false>(rate, in, out, rows, S, circular, s);
    else rc = dispatch_pow2<1, false>(rate, in, out, rows, S, 0, s);
    return rc ? rc : check_launch("blade_channelize");
}

}  // namespace bb
