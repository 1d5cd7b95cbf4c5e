// Host side of the tensor-core chain (beamform_tc.cuh): phasor images, launch layouts,
// the C entries and the plain instantiations of the kernel.
#include "beamform_tc.cuh"

namespace bb {
namespace {

__global__ void __launch_bounds__(256) tc_prepare_kernel(const float2* __restrict__ ph, uint8_t* __restrict__ plan,
                                                         uint32_t B, uint32_t A, uint32_t F, uint32_t NB,
                                                         uint32_t KA, uint32_t nchunks, uint32_t img_bytes,
                                                         uint32_t stacked, uint32_t fold) {
    // a chain kernel launched as this grid's programmatic dependent may start its
    // prologue now; it waits for this grid to finish before it reads the image
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t groups = KA / 8;
    const uint32_t n = nchunks * F * 2u * NB * groups;
    const uint32_t ph_bytes = (KA == 64 ? 3u : 2u) * NB * 128u;
    const uint32_t pol_stacked = (2 * KA / 64) * 4 * NB * 128u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t r = i;
        const uint32_t f = r % F;
        r /= F;
        const uint32_t p = r & 1u;
        r >>= 1;
        const uint32_t nb = r % NB;
        r /= NB;
        const uint32_t j = r % groups;
        const uint32_t c = r / groups;
        const uint32_t b = c * kMaxNB + nb, fk = f % fold;
        SplitChunk w;
        split_chunk(ph + ((uint64_t)b * A * F + f) * 2 + p, 2ull * F, j * 8, A, b < B, w);
        // fold > 1: the images of fold consecutive channels as one
        uint8_t* base = plan + ((uint64_t)c * F + (f - fk)) * img_bytes +
                        (uint64_t)p * (stacked ? fold * pol_stacked : 2 * ph_bytes);
        put_image([&](uint32_t off, uint4 v) { *reinterpret_cast<uint4*>(base + off) = v; }, w, NB, KA, nb, j * 8,
                  stacked, fold, fk);
    }
}

// The same split for KA = 64 images without stacking (more than 32 beams per
// chunk), through shared memory: a CTA takes 8 beams x 2 channels x both
// polarisations of one chunk (20 KB of shared memory; the dense block's 1024
// CTAs are resident at once).  It reads each (beam, antenna) row's 2 x 2 phasors
// as one 32-byte run, and each warp then writes 4 whole 128-byte image rows per
// block (lanes: 8 antenna groups x 4 beams), where the one-thread-per-chunk form
// writes 32 chunks into 32 different channels' images.  Same arithmetic per
// element, so the image is bit-identical.
constexpr uint32_t kPrepBeams = 8, kPrepChans = 2, kPrepPad = 10;  // float2 per 8-antenna group (8 + 2 pad)
__global__ void __launch_bounds__(256) tc_prepare_wide_kernel(const float2* __restrict__ ph, uint8_t* __restrict__ plan,
                                                              uint32_t B, uint32_t A, uint32_t F, uint32_t NB,
                                                              uint32_t img_bytes) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // [beam][channel][pol][antenna group][8 antennas + pad]: a task's 8 phasors are
    // contiguous, and the 80-byte group pitch keeps a quarter-warp's 16-byte reads
    // (8 groups) on distinct banks
    __shared__ __align__(16) float2 sp[kPrepBeams][kPrepChans][2][8][kPrepPad];
    const uint32_t f0 = blockIdx.x * kPrepChans, nb0 = blockIdx.y * kPrepBeams, c = blockIdx.z;
    // load: element q = (bl, a, col), col = 2 fl + p fastest (the phasors' own order)
    constexpr uint32_t kCol = 2 * kPrepChans;
#pragma unroll 4
    for (uint32_t q = threadIdx.x; q < kPrepBeams * 64 * kCol; q += blockDim.x) {
        const uint32_t col = q % kCol, a = (q / kCol) % 64u, bl = q / (64u * kCol);
        const uint32_t fl = col >> 1, pp = col & 1u;
        const uint32_t b = c * kMaxNB + nb0 + bl;
        float2 w = make_float2(0.f, 0.f);
        if (b < B && a < A && f0 + fl < F) w = ph[((uint64_t)(b * (uint64_t)A + a) * F + f0 + fl) * 2 + pp];
        sp[bl][fl][pp][a >> 3][a & 7u] = w;
    }
    __syncthreads();
    const uint32_t ph_bytes = 3u * NB * 128u;
    // tasks t = (j, bl, p, fl), j fastest: a warp covers 8 groups x 4 beams
    for (uint32_t t = threadIdx.x; t < kPrepBeams * 8 * 2 * kPrepChans; t += blockDim.x) {
        const uint32_t j = t & 7u, bl = (t / 8u) % kPrepBeams, pp = (t / (8u * kPrepBeams)) & 1u,
                       fl = t / (16u * kPrepBeams);
        const uint32_t f = f0 + fl;
        if (f >= F) continue;
        __half rh[8], ih[8], rl[8], il[8], nih[8], nil[8];
        const float4* src = reinterpret_cast<const float4*>(&sp[bl][fl][pp][j][0]);
#pragma unroll
        for (int e2 = 0; e2 < 4; e2++) {
            const float4 v = src[e2];
            const float wr[2] = {v.x, v.z}, wi[2] = {v.y, v.w};
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int e = 2 * e2 + u;
                rh[e] = __float2half_rn(wr[u]);
                ih[e] = __float2half_rn(wi[u]);
                rl[e] = __float2half_rn(wr[u] - __half2float(rh[e]));
                il[e] = __float2half_rn(wi[u] - __half2float(ih[e]));
                nih[e] = __hneg(ih[e]);
                nil[e] = __hneg(il[e]);
            }
        }
        const uint32_t nb = nb0 + bl, k0 = j * 8;
        uint8_t* base = plan + ((uint64_t)c * F + f) * img_bytes + (uint64_t)pp * 2 * ph_bytes;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint8_t* blk = base + h * ph_bytes;
            // three blocks of NB rows x 64 K: [-Wi | Wr | Wi]
            put_chunk(blk, NB, nb, k0, pack8(h ? nil : nih));
            put_chunk(blk + NB * 128u, NB, nb, k0, pack8(h ? rl : rh));
            put_chunk(blk + 2u * NB * 128u, NB, nb, k0, pack8(h ? il : ih));
        }
    }
}

struct TcShape {
    uint32_t NB, KA, nchunks, img_bytes, raw_bytes, a_stages, r_stages, stacked;
    uint32_t raw_tiles, raw_row, direct;
    size_t smem;
};

// T = 0 sizes only the phasor image (the ring layout needs the tiles per channel).
bool tc_shape(uint64_t B, uint64_t A, TcShape& s, uint64_t T = 0, uint32_t es = 4, uint64_t rate = 0) {
    s.direct = 0;
    if (A == 0 || A > kMaxKA || B == 0) return false;
    const uint64_t bc = B < (uint64_t)kMaxNB ? B : (uint64_t)kMaxNB;
    s.NB = (uint32_t)((bc + 15) / 16 * 16);
    s.KA = A <= 32 ? 32u : 64u;
    s.nchunks = (uint32_t)((B + kMaxNB - 1) / kMaxNB);
    // hi/lo stacked along N (one MMA per k-step, N = 4 NB <= 128) whenever the
    // doubled accumulators still fit twice in tensor memory.
    s.stacked = s.NB <= 32 ? 1u : 0u;
    s.img_bytes = s.stacked ? (2 * s.KA / 64) * 1024u * s.NB : (s.KA == 64 ? 1536u : 1024u) * s.NB;
    s.raw_bytes = (uint32_t)A * kM * es;
    const size_t op = (2ull * s.KA / 64) * 16384;   // one polarisation's operand
    // barriers (2 x 8 operand + 2 x 8 raw + 3 x 4 accumulator + 4, 8 bytes each),
    // TMEM slot and abort flag, alignment slack
    const size_t fixed = s.img_bytes + 512 + 1024;
    const size_t limit = 227 * 1024;
    // Two-tile raw stages (1 KB per antenna row) when the channel's tile count is even
    // and one of these rings fits: four operand tile pairs and two raw stages (the
    // operand build runs up to four tiles ahead of the MMAs), else two pairs and
    // four or three raw stages.
    const uint64_t tpc = T / kM;
    if (T && es == 8) {
        // CF16 input: single-tile raw stages of 1 KB rows; four operand pairs and two
        // raw stages (two issuers), else two pairs and four or three raw stages.
        const uint32_t cand[][2] = {{8, 2}, {4, 4}, {4, 3}};
        for (const auto& c : cand) {
            if (fixed + c[0] * op + c[1] * (size_t)s.raw_bytes <= limit) {
                s.raw_tiles = 1;
                s.raw_row = kM * es;
                s.a_stages = c[0];
                s.r_stages = c[1];
                s.smem = fixed + c[0] * op + c[1] * (size_t)s.raw_bytes;
                return true;
            }
        }
    }
    if (T && es == 4 && tpc % 2 == 0) {
        const size_t raw2 = (size_t)A * 1024u;
        const uint32_t cand[][2] = {{8, 2}, {4, 4}, {4, 3}};
        for (const auto& c : cand) {
            if (fixed + c[0] * op + c[1] * raw2 <= limit) {
                s.raw_tiles = 2;
                s.raw_row = 1024;
                s.raw_bytes = (uint32_t)raw2;
                s.a_stages = c[0];
                s.r_stages = c[1];
                s.smem = fixed + c[0] * op + c[1] * raw2;
                return true;
            }
        }
    }
    s.raw_tiles = 1;
    s.raw_row = kM * es;
    // Deepest rings that fit: operand stages in pairs (one per polarisation) down to
    // four, raw stages down to three, then both down to the minimum.
    uint32_t as = kMaxStages, rs = 6;
    while (fixed + as * op + rs * (size_t)s.raw_bytes > limit) {
        if (rs > 3 && (rs > as / 2 || as <= 4)) rs--;
        else if (as > 4) as -= 2;
        else if (rs > 2) rs--;
        else if (as > 2) as--;
        else if (rs > 1) rs--;
        else return false;
    }
    s.a_stages = as;
    s.r_stages = rs;
    s.smem = fixed + as * op + rs * (size_t)s.raw_bytes;
    if (T && es == 4 && (rate == 1 || (rate == 2 && !s.stacked)) && as < 4) {
        // A phasor image this large leaves no room for a raw ring and a build-ahead
        // operand ring together: at rate 1, and at rate 2 beyond 32 beams, the converter
        // threads load the voltages themselves and the shared memory holds operand tile pairs only (two pairs
        // at least, so that the build runs a tile ahead and two issuers alternate).
        // 42 antennas x 50 channels x 1920 samples, 37 beams, rate 2: 28.0 us with three
        // operand and two raw stages, 23.9 with direct loads; with a stacked image the ring
        // stays ahead (40 x 64 x 4096, 20 beams, rate 2: 38.1 us against 40.0).
        for (uint32_t c : {8u, 4u}) {
            if (fixed + c * op <= limit) {
                s.direct = 1;
                s.a_stages = c;
                s.r_stages = 0;
                s.raw_bytes = 0;
                s.smem = fixed + c * op;
                return true;
            }
        }
    }
    return true;
}

// A launch choice of the chain: mode 0 = raw ring of TMA tiles, 1 = converter
// threads load the voltages (CI8, rates 1 and 2), with the operand ring depth, the raw
// ring depth and the tiles per raw stage.
struct TcChoice {
    uint32_t mode, a_stages, r_stages, raw_tiles;
};

TcChoice tc_choice_of(const TcShape& s) {
    return TcChoice{s.direct ? 1u : 0u, s.a_stages, s.r_stages, s.raw_tiles};
}

// Lays out shape s (image part from tc_shape) for choice c; false when c does not
// apply to the shape or does not fit in shared memory.  Every choice computes the
// same arithmetic in the same order within a kernel (the ring depths only change
// scheduling), so modes 0 and 1 give bit-identical outputs.
bool tc_apply(TcShape& s, uint64_t A, uint64_t T, uint32_t es, uint64_t rate, const TcChoice& c) {
    const size_t op = (2ull * s.KA / 64) * 16384;
    const size_t limit = 227 * 1024;
    if (c.a_stages < 1 || c.a_stages > (uint32_t)kMaxStages) return false;
    s.direct = 0;
    s.a_stages = c.a_stages;
    if (c.mode == 1) {
        // direct loads run in pair mode: an even operand ring of at least four stages
        if (es != 4 || (rate != 1 && rate != 2) || (c.a_stages & 1u) || c.a_stages < 4u) return false;
        s.direct = 1;
        s.raw_tiles = 1;
        s.raw_row = kM * es;
        s.raw_bytes = 0;
        s.r_stages = 0;
        s.smem = s.img_bytes + 1536 + c.a_stages * op;
        return s.smem <= limit;
    }
    if (c.mode != 0 || c.r_stages < 1 || c.r_stages > (uint32_t)kMaxStages) return false;
    if (c.raw_tiles == 2) {
        if (es != 4 || (T / kM) % 2) return false;
        s.raw_row = 1024;
        s.raw_bytes = (uint32_t)A * 1024u;
    } else if (c.raw_tiles == 1) {
        s.raw_row = kM * es;
        s.raw_bytes = (uint32_t)A * kM * es;
    } else {
        return false;
    }
    s.raw_tiles = c.raw_tiles;
    s.r_stages = c.r_stages;
    s.smem = s.img_bytes + 1536 + c.a_stages * op + c.r_stages * (size_t)s.raw_bytes;
    return s.smem <= limit;
}

// Last word of the tuning key of a launch that splits its phasors itself; the plain
// chain's is the sample size.
constexpr uint64_t kTuneSelf = 5;

// The launch layout of a chain call: the tuned choice for this shape on this device
// when blade_beamform_detect_tc_autotune stored one, else the heuristic default.
bool tc_layout(uint64_t B, uint64_t A, uint64_t F, uint64_t T, uint64_t rate, uint64_t integration, uint32_t es,
               TcShape& s, bool* tuned = nullptr, TuneEntry* entry = nullptr) {
    if (!tc_shape(B, A, s, T, es, rate)) return false;
    if (tuned) *tuned = false;
    const uint64_t key[8] = {B, A, F, T, 2, rate, integration, es};
    TuneEntry e;
    if (tune_lookup(BLADE_TUNE_TC, key, &e)) {
        TcShape t = s;
        if (tc_apply(t, A, T, es, rate, TcChoice{e.params[0], e.params[1], e.params[2], e.params[3]})) {
            s = t;
            if (tuned) *tuned = true;
            if (entry) *entry = e;
        }
    }
    return true;
}

// Tensor map of the voltages seen as samples [A][F][T] of es bytes (CI8: one
// 4-byte word, CF16: one 8-byte word = both polarisations of one sample);
// box = `box` samples x 1 channel x A.
int encode_voltage_map(CUtensorMap* tm, const void* in, uint64_t A, uint64_t F, uint64_t T, uint32_t box_t,
                       uint32_t es = 4) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    static std::mutex mu;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!encode) {
            cudaDriverEntryPointQueryResult q;
            void* fn = nullptr;
            if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
                    cudaSuccess ||
                q != cudaDriverEntryPointSuccess || !fn)
                return set_error(BLADE_CUDA_ERROR, "blade_beamform_detect_tc: cuTensorMapEncodeTiled unavailable");
            encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
        }
    }
    const cuuint64_t dims[3] = {T, F, A};
    const cuuint64_t strides[2] = {T * es, F * T * es};
    const cuuint32_t box[3] = {box_t, 1, (cuuint32_t)A};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = encode(tm, es == 8 ? CU_TENSOR_MAP_DATA_TYPE_UINT64 : CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<void*>(in), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(BLADE_CUDA_ERROR, "blade_beamform_detect_tc: tensor map encode (%d)", (int)r);
    return BLADE_SUCCESS;
}

template <int R>
const void* pick_logi(uint32_t logi) {
    switch (logi) {
        case 0: return reinterpret_cast<const void*>(bf_tc_kernel<R, 0>);
        case 1: return reinterpret_cast<const void*>(bf_tc_kernel<R, 1>);
        case 2: return reinterpret_cast<const void*>(bf_tc_kernel<R, 2>);
        case 3: return reinterpret_cast<const void*>(bf_tc_kernel<R, 3>);
        case 4: return reinterpret_cast<const void*>(bf_tc_kernel<R, 4>);
        default: return reinterpret_cast<const void*>(bf_tc_kernel<R, 5>);
    }
}

const void* pick_kernel(uint64_t rate, uint64_t integration, const TcShape& s) {
    const uint32_t logi = tc_log2(integration);
    if (rate == 1) return pick_logi<1>(logi);
    if (rate == 2) return s.direct ? tc_direct2_kernel(integration) : pick_logi<2>(logi);
    return pick_logi<4>(logi);
}

// CTAs per channel and tiles per CTA when every CTA stays inside a channel and splits
// its image itself: in one wave, with at most one tile (or raw stage) more per CTA than
// an even spread of all tiles would give.  The split launch it saves is 1 to 3 us (20
// antennas x 96 channels x 256 samples, 8 beams: 8.2 us per call instead of 10.2), so the
// rule ends where a larger share of the tiles is worth more than that:
//   images up to 32 KB (64 antennas, 32 beams, 64 KB, 148 channels: 51.2 us against 47.3
//   at 16 tiles per CTA; beyond 32 beams 15.2 against 12.4 at one),
//   16 tiles per CTA, 8 at rate 2 (20 antennas, 16 beams: 14.0 us against 16.3 at 5 tiles,
//   16.5 at 8 on both, 24.6 against 23.0 at 14).
bool self_shape(const TcShape& s, uint64_t F, uint64_t T, uint64_t rate, uint32_t& segs, uint32_t& seg_tiles) {
    const uint64_t sms = (uint64_t)sm_count(), tpc = T / kM, rt = s.raw_tiles;
    if (!s.stacked || s.img_bytes > 32 * 1024 || F > sms || tpc * F > (rate == 2 ? 8 : 16) * sms) return false;
    uint64_t per = ceil_div(ceil_div(tpc, sms / F), rt) * rt;
    const uint64_t even = ceil_div(ceil_div(F * tpc, sms), rt) * rt;
    if (per > even + rt) return false;
    segs = (uint32_t)ceil_div(tpc, per);
    seg_tiles = (uint32_t)per;
    return true;
}

// The launch layout of a call that splits its phasors inside the chain kernel: the choice
// tuned for that launch (its operand build and grid are not the plain chain's, so neither's
// times hold for the other) or the default; false when the default layout is not such a launch.
bool tc_self_layout(uint64_t B, uint64_t A, uint64_t F, uint64_t T, uint64_t rate, uint64_t integration, TcShape& s,
                    uint32_t& segs, uint32_t& seg_tiles, bool* tuned = nullptr, TuneEntry* entry = nullptr) {
    if (tuned) *tuned = false;
    if (!tc_shape(B, A, s, T, 4, rate) || !self_shape(s, F, T, rate, segs, seg_tiles)) return false;
    const uint64_t key[8] = {B, A, F, T, 2, rate, integration, kTuneSelf};
    TuneEntry e;
    TcShape t = s;
    uint32_t g, gt;
    if (tune_lookup(BLADE_TUNE_TC, key, &e) &&
        tc_apply(t, A, T, 4, rate, TcChoice{e.params[0], e.params[1], e.params[2], e.params[3]}) &&
        self_shape(t, F, T, rate, g, gt)) {
        s = t;
        segs = g;
        seg_tiles = gt;
        if (tuned) *tuned = true;
        if (entry) *entry = e;
    }
    return true;
}

}  // namespace
}  // namespace bb

using namespace bb;

extern "C" uint64_t blade_beamform_tc_plan_size(uint64_t B, uint64_t A, uint64_t F, uint64_t P) {
    TcShape s;
    if (P != 2 || !tc_shape(B, A, s)) return 0;
    return (uint64_t)s.nchunks * F * s.img_bytes;
}

extern "C" int blade_beamform_tc_prepare(const void* phasors, void* plan, uint64_t B, uint64_t A, uint64_t F,
                                         uint64_t P, blade_stream_t stream) {
    TcShape s;
    if (P != 2) return set_error(BLADE_ERROR, "blade_beamform_tc_prepare: P must be 2");
    if (!tc_shape(B, A, s))
        return set_error(BLADE_ERROR, "blade_beamform_tc_prepare: unsupported shape (A=%llu must be 1..64)",
                         (unsigned long long)A);
    if (F == 0) return BLADE_SUCCESS;
    if (!phasors || !plan) return set_error(BLADE_ERROR, "blade_beamform_tc_prepare: null buffer");
    if (!aligned16(plan)) return set_error(BLADE_ERROR, "blade_beamform_tc_prepare: plan must be 16-byte aligned");
    const uint64_t n = (uint64_t)s.nchunks * F * 2 * s.NB * (s.KA / 8);
    if (n > 0xFFFFFFFFull) return set_error(BLADE_ERROR, "blade_beamform_tc_prepare: too many channels");
    if (!s.stacked && s.KA == 64) {
        const dim3 grid((unsigned)((F + kPrepChans - 1) / kPrepChans), s.NB / kPrepBeams, s.nchunks);
        tc_prepare_wide_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
            static_cast<const float2*>(phasors), static_cast<uint8_t*>(plan), (uint32_t)B, (uint32_t)A, (uint32_t)F,
            s.NB, s.img_bytes);
    } else {
        tc_prepare_kernel<<<grid_for(n, 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
            static_cast<const float2*>(phasors), static_cast<uint8_t*>(plan), (uint32_t)B, (uint32_t)A, (uint32_t)F,
            s.NB, s.KA, s.nchunks, s.img_bytes, s.stacked, 1u);
    }
    return check_launch("blade_beamform_tc_prepare");
}

extern "C" int blade_beamform_detect_tc_supported(uint64_t B, uint64_t A, uint64_t F, uint64_t T, uint64_t P,
                                                  uint64_t rate, uint64_t integration) {
    TcShape s;
    if (P != 2 || !tc_shape(B, A, s)) return 0;
    if (rate != 1 && rate != 2 && rate != 4) return 0;
    if (integration == 0 || integration > 32 || (integration & (integration - 1)) != 0) return 0;
    if (T == 0 || T % kM != 0 || F == 0) return 0;
    if (F > 0xffffffffull / (T / kM) || T >= (1ull << 31) || (uint64_t)A * F * T >= (1ull << 40)) return 0;
    return 1;
}

namespace bb {
namespace {

// Launches the chain over the 64-beam chunks once the arguments are checked.
int tc_run(const char* who, const void* in, const void* plan, void* out, uint64_t B, uint64_t A, uint64_t F,
           uint64_t T, uint64_t rate, uint64_t integration, uint32_t es, const void* fn, blade_stream_t stream,
           bool pdl = false, const TcShape* force = nullptr, const float2* self = nullptr, uint32_t segs = 0,
           uint32_t seg_tiles = 0) {
    TcShape s;
    if (force) {
        s = *force;
    } else {
        tc_layout(B, A, F, T, rate, integration, es, s);
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (!fn) fn = pick_kernel(rate, integration, s);
    if (int rc = ensure_smem(fn, s.smem)) return rc;
    const uint32_t U = (uint32_t)(T / (rate * integration));
    CUtensorMap tmap;
    if (int rc = encode_voltage_map(&tmap, in, A, F, T, s.raw_row / es, es)) return rc;
    for (uint32_t c = 0; c < s.nchunks; c++) {
        TcArgs g;
        g.in = static_cast<const uint8_t*>(in);
        g.plan = static_cast<const uint8_t*>(plan) + (uint64_t)c * F * s.img_bytes;
        g.out = static_cast<float*>(out) + (uint64_t)c * kMaxNB * F * rate * U;
        g.A = (uint32_t)A;
        g.F = (uint32_t)F;
        g.T = (uint32_t)T;
        const uint64_t rem = B - (uint64_t)c * kMaxNB;
        g.beams = (uint32_t)(rem < (uint64_t)kMaxNB ? rem : kMaxNB);
        g.U = U;
        g.NB = s.NB;
        g.KA = s.KA;
        g.a_stages = s.a_stages;
        g.r_stages = s.r_stages;
        g.img_bytes = s.img_bytes;
        g.raw_bytes = s.raw_bytes;
        g.raw_tiles = s.raw_tiles;
        g.raw_row = s.raw_row;
        g.stacked = s.stacked;
        g.tiles_per_ch = (uint32_t)(T / kM);
        g.total_tiles = (uint64_t)F * (T / kM);
        g.pdl = (pdl && c == 0) ? 1u : 0u;
        g.direct = s.direct;
        g.circ = 0;
        // outputs along TMEM lanes: full 64-beam chunks (separate hi/lo products),
        // rate 1 CI8, windows of 8 or 16 samples, 16-byte aligned output rows
        g.transposed = (!s.stacked && s.NB == 64 && rate == 1 && es == 4 && (integration == 8 || integration == 16) &&
                        U % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) ? 1u : 0u;
        // Whole raw stages per CTA (the kernel rounds its share up to raw_tiles); no
        // CTA is left without tiles.
        const uint64_t sms = (uint64_t)sm_count();
        const uint64_t per = ((g.total_tiles + sms - 1) / sms + s.raw_tiles - 1) / s.raw_tiles * s.raw_tiles;
        uint64_t grid = (g.total_tiles + per - 1) / per;
        g.ph = self ? self + (uint64_t)c * kMaxNB * A * F * 2 : nullptr;
        g.plan_out = const_cast<uint8_t*>(g.plan);
        g.segs = segs;
        g.seg_tiles = seg_tiles;
        if (self) grid = F * segs;
        void* args[2] = {&g, &tmap};
        if (g.pdl) {
            // programmatic dependent of the phasor split launched just before on this
            // stream: prologue and raw loads overlap it (the kernel waits before the image)
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)grid, 1, 1);
            cfg.blockDim = dim3(kThreads, 1, 1);
            cfg.dynamicSmemBytes = s.smem;
            cfg.stream = st;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
            if (e != cudaSuccess) return check_cuda(e, who);
        } else {
            const cudaError_t e = cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(kThreads), args, s.smem, st);
            if (e != cudaSuccess) return check_cuda(e, who);
        }
        if (int rc = check_launch(who)) return rc;
    }
    return BLADE_SUCCESS;
}

const void* pick_cf16(uint64_t integration) {
    switch (tc_log2(integration)) {
        case 0: return reinterpret_cast<const void*>(bf_tc_kernel<1, 0, 8>);
        case 1: return reinterpret_cast<const void*>(bf_tc_kernel<1, 1, 8>);
        case 2: return reinterpret_cast<const void*>(bf_tc_kernel<1, 2, 8>);
        case 3: return reinterpret_cast<const void*>(bf_tc_kernel<1, 3, 8>);
        case 4: return reinterpret_cast<const void*>(bf_tc_kernel<1, 4, 8>);
        default: return reinterpret_cast<const void*>(bf_tc_kernel<1, 5, 8>);
    }
}

}  // namespace
}  // namespace bb

extern "C" int blade_beamform_detect_tc(const void* in, const void* plan, void* out, uint64_t B, uint64_t A,
                                        uint64_t F, uint64_t T, uint64_t P, uint64_t rate, uint64_t integration,
                                        blade_stream_t stream) {
    if (!blade_beamform_detect_tc_supported(B, A, F, T, P, rate, integration))
        return set_error(BLADE_ERROR,
                         "blade_beamform_detect_tc: unsupported configuration (B=%llu A=%llu T=%llu P=%llu rate=%llu "
                         "I=%llu): needs P=2, 1<=A<=64, T%%128==0, rate in {1,2,4}, I a power of two <= 32",
                         (unsigned long long)B, (unsigned long long)A, (unsigned long long)T, (unsigned long long)P,
                         (unsigned long long)rate, (unsigned long long)integration);
    if (!in || !plan || !out) return set_error(BLADE_ERROR, "blade_beamform_detect_tc: null buffer");
    if (!aligned16(in) || !aligned16(plan) || (reinterpret_cast<uintptr_t>(out) & 3))
        return set_error(BLADE_ERROR, "blade_beamform_detect_tc: input and plan must be 16-byte aligned");
    return tc_run("blade_beamform_detect_tc", in, plan, out, B, A, F, T, rate, integration, 4,
                  nullptr, stream);
}

extern "C" int blade_beamform_prepare_detect_tc(const void* phasors, void* plan, const void* in, void* out,
                                                uint64_t B, uint64_t A, uint64_t F, uint64_t T, uint64_t P,
                                                uint64_t rate, uint64_t integration, blade_stream_t stream) {
    if (!blade_beamform_detect_tc_supported(B, A, F, T, P, rate, integration))
        return set_error(BLADE_ERROR,
                         "blade_beamform_prepare_detect_tc: unsupported configuration (B=%llu A=%llu T=%llu P=%llu "
                         "rate=%llu I=%llu): needs P=2, 1<=A<=64, T%%128==0, rate in {1,2,4}, I a power of two <= 32",
                         (unsigned long long)B, (unsigned long long)A, (unsigned long long)T, (unsigned long long)P,
                         (unsigned long long)rate, (unsigned long long)integration);
    if (!in || !plan || !out || !phasors) return set_error(BLADE_ERROR, "blade_beamform_prepare_detect_tc: null buffer");
    if (!aligned16(in) || !aligned16(plan) || (reinterpret_cast<uintptr_t>(out) & 3))
        return set_error(BLADE_ERROR, "blade_beamform_prepare_detect_tc: input and plan must be 16-byte aligned");
    if (F == 0) return BLADE_SUCCESS;  // no split launched: nothing may follow it programmatically
    TcShape s;
    uint32_t segs, seg_tiles;
    if (tc_self_layout(B, A, F, T, rate, integration, s, segs, seg_tiles))
        return tc_run("blade_beamform_prepare_detect_tc", in, plan, out, B, A, F, T, rate, integration, 4,
                      tc_self_kernel(rate, integration), stream, false, &s, static_cast<const float2*>(phasors), segs,
                      seg_tiles);
    if (int rc = blade_beamform_tc_prepare(phasors, plan, B, A, F, P, stream)) return rc;
    return tc_run("blade_beamform_prepare_detect_tc", in, plan, out, B, A, F, T, rate, integration, 4,
                  nullptr, stream, true);
}

extern "C" int blade_beamform_detect_tc_cf16(const void* in, const void* plan, void* out, uint64_t B, uint64_t A,
                                             uint64_t F, uint64_t T, uint64_t P, uint64_t integration,
                                             blade_stream_t stream) {
    if (!blade_beamform_detect_tc_supported(B, A, F, T, P, 1, integration))
        return set_error(BLADE_ERROR,
                         "blade_beamform_detect_tc_cf16: unsupported configuration (B=%llu A=%llu T=%llu P=%llu "
                         "I=%llu): needs P=2, 1<=A<=64, T%%128==0, I a power of two <= 32",
                         (unsigned long long)B, (unsigned long long)A, (unsigned long long)T, (unsigned long long)P,
                         (unsigned long long)integration);
    if (!in || !plan || !out) return set_error(BLADE_ERROR, "blade_beamform_detect_tc_cf16: null buffer");
    if (!aligned16(in) || !aligned16(plan) || (reinterpret_cast<uintptr_t>(out) & 3))
        return set_error(BLADE_ERROR, "blade_beamform_detect_tc_cf16: input and plan must be 16-byte aligned");
    return tc_run("blade_beamform_detect_tc_cf16", in, plan, out, B, A, F, T, 1, integration, 8,
                  pick_cf16(integration), stream);
}

extern "C" int blade_beamform_prepare_detect_tc_cf16(const void* phasors, void* plan, const void* in, void* out,
                                                     uint64_t B, uint64_t A, uint64_t F, uint64_t T, uint64_t P,
                                                     uint64_t integration, blade_stream_t stream) {
    if (!blade_beamform_detect_tc_supported(B, A, F, T, P, 1, integration))
        return set_error(BLADE_ERROR,
                         "blade_beamform_prepare_detect_tc_cf16: unsupported configuration (B=%llu A=%llu T=%llu "
                         "P=%llu I=%llu): needs P=2, 1<=A<=64, T%%128==0, I a power of two <= 32",
                         (unsigned long long)B, (unsigned long long)A, (unsigned long long)T, (unsigned long long)P,
                         (unsigned long long)integration);
    if (!in || !plan || !out || !phasors)
        return set_error(BLADE_ERROR, "blade_beamform_prepare_detect_tc_cf16: null buffer");
    if (!aligned16(in) || !aligned16(plan) || (reinterpret_cast<uintptr_t>(out) & 3))
        return set_error(BLADE_ERROR, "blade_beamform_prepare_detect_tc_cf16: input and plan must be 16-byte aligned");
    if (F == 0) return BLADE_SUCCESS;
    if (int rc = blade_beamform_tc_prepare(phasors, plan, B, A, F, P, stream)) return rc;
    return tc_run("blade_beamform_prepare_detect_tc_cf16", in, plan, out, B, A, F, T, 1, integration, 8,
                  pick_cf16(integration), stream, true);
}

namespace bb {
namespace {

// Layout of the PRE chain: up to 32 antennas, one chunk of beams whose R stacked images
// fit an MMA's 256 columns; three operand tile pairs and two two-tile raw stages (one
// KB rows) beside the 64 KB of images, or as many one-tile stages as fit when a
// channel's tiles are odd.
bool pre_shape(uint64_t B, uint64_t A, uint64_t T, uint64_t rate, TcShape& s) {
    if (rate != 2 && rate != 4) return false;
    if (!tc_shape(B, A, s) || s.KA != 32 || s.nchunks != 1 || !s.stacked || 4 * rate * s.NB > 256) return false;
    const size_t op = (2ull * s.KA / 64) * 16384, limit = 227 * 1024;
    s.direct = 0;
    s.a_stages = 6;
    s.raw_tiles = (T / kM) % 2 == 0 ? 2u : 1u;
    s.raw_row = s.raw_tiles * kM * 4;
    s.raw_bytes = (uint32_t)A * s.raw_row;
    const size_t fixed = rate * (size_t)s.img_bytes + 1536 + s.a_stages * op;
    s.r_stages = 2;
    while (s.r_stages < 4 && fixed + (s.r_stages + 1) * (size_t)s.raw_bytes <= limit) s.r_stages++;
    s.smem = fixed + s.r_stages * (size_t)s.raw_bytes;
    return s.smem <= limit;
}

}  // namespace
}  // namespace bb

extern "C" int blade_modeb_detect_tc_supported(uint64_t B, uint64_t A, uint64_t F, uint64_t T, uint64_t P,
                                               uint64_t rate, uint64_t integration) {
    TcShape s;
    if (rate == 1 || !blade_beamform_detect_tc_supported(B, A, F, T, P, rate, integration)) return 0;
    // windows of rate x integration samples must tile a channel, and close inside a tile's rows
    if (T % (rate * integration) != 0 || integration > kM / rate) return 0;
    const uint64_t split = F * rate * 2 * 64 * 4;  // threads of the split at most
    return split <= 0xFFFFFFFFull && pre_shape(B, A, T, rate, s) ? 1 : 0;
}

extern "C" int blade_modeb_detect_tc(const void* phasors, void* plan, const void* in, void* out, uint64_t B,
                                     uint64_t A, uint64_t F, uint64_t T, uint64_t P, uint64_t rate,
                                     uint64_t integration, int circular, blade_stream_t stream) {
    const char* who = "blade_modeb_detect_tc";
    if (!blade_modeb_detect_tc_supported(B, A, F, T, P, rate, integration))
        return set_error(BLADE_ERROR,
                         "%s: unsupported configuration (B=%llu A=%llu T=%llu P=%llu rate=%llu I=%llu): needs P=2, "
                         "1<=A<=32, rate 4 with B<=16 or 2 with B<=32, T%%128==0, I a power of two <= 32", who,
                         (unsigned long long)B, (unsigned long long)A, (unsigned long long)T, (unsigned long long)P,
                         (unsigned long long)rate, (unsigned long long)integration);
    if (!in || !plan || !out || !phasors) return set_error(BLADE_ERROR, "%s: null buffer", who);
    if (!aligned16(in) || !aligned16(plan) || (reinterpret_cast<uintptr_t>(out) & 3))
        return set_error(BLADE_ERROR, "%s: input and plan must be 16-byte aligned", who);
    TcShape s;
    pre_shape(B, A, T, rate, s);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const uint32_t FR = (uint32_t)(F * rate);
    const uint64_t n = (uint64_t)FR * 2 * s.NB * (s.KA / 8);
    tc_prepare_kernel<<<grid_for(n, 256), 256, 0, st>>>(static_cast<const float2*>(phasors),
                                                      static_cast<uint8_t*>(plan), (uint32_t)B, (uint32_t)A, FR, s.NB,
                                                      s.KA, 1u, s.img_bytes, 1u, (uint32_t)rate);
    if (int rc = check_launch(who)) return rc;
    const void* fn = tc_pre_kernel(rate, integration);
    if (int rc = ensure_smem(fn, s.smem)) return rc;
    CUtensorMap tmap;
    if (int rc = encode_voltage_map(&tmap, in, A, F, T, s.raw_row / 4, 4)) return rc;
    TcArgs g = {};
    g.in = static_cast<const uint8_t*>(in);
    g.plan = static_cast<const uint8_t*>(plan);
    g.out = static_cast<float*>(out);
    g.A = (uint32_t)A;
    g.F = (uint32_t)F;
    g.T = (uint32_t)T;
    g.beams = (uint32_t)B;
    g.U = (uint32_t)(T / (rate * integration));
    g.NB = s.NB;
    g.KA = s.KA;
    g.a_stages = s.a_stages;
    g.r_stages = s.r_stages;
    g.stacked = 1;
    g.img_bytes = (uint32_t)rate * s.img_bytes;
    g.raw_bytes = s.raw_bytes;
    g.raw_tiles = s.raw_tiles;
    g.raw_row = s.raw_row;
    g.tiles_per_ch = (uint32_t)(T / kM);
    g.total_tiles = (uint64_t)F * g.tiles_per_ch;
    g.pdl = 1;
    g.circ = circular ? 1u : 0u;
    const uint64_t sms = (uint64_t)sm_count();
    const uint64_t per = ((g.total_tiles + sms - 1) / sms + s.raw_tiles - 1) / s.raw_tiles * s.raw_tiles;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((g.total_tiles + per - 1) / per), 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = s.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[2] = {&g, &tmap};
    const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
    return e != cudaSuccess ? check_cuda(e, who) : check_launch(who);
}

namespace bb {
int adjoint_status_take(uint32_t* v);
}

extern "C" int blade_device_status(uint32_t* status) {
    uint32_t v = 0;
    if (int rc = bb::tc_status_take_here(&v)) return rc;
    uint32_t w = 0;
    if (int rc = bb::tc_pre_status_take(&w)) return rc;
    if (!v) v = w;
    if (int rc = bb::tc_self_status_take(&w)) return rc;
    if (!v) v = w;
    // the tensor-core adjoint's word: codes 0x100 | 1 (a phase wait expired), 0x100 | 2 (the drain did)
    uint32_t adj = 0;
    if (int rc = bb::adjoint_status_take(&adj)) return rc;
    if (!v && adj) v = 0x100u | adj;
    if (status) *status = v;
    return BLADE_SUCCESS;
}

// ---- bounded-wait self-test ---------------------------------------------------
// One thread waits on an mbarrier that nothing ever completes, through the same
// bounded wait as the pipelined kernels; when the budget runs out it records
// kSelftestCode in the status word and the kernel returns normally, so the
// expiry path is exercised without a fault and the context stays usable.
namespace bb {
namespace {
constexpr unsigned kSelftestCode = 0x20u;

__global__ void wait_selftest_kernel(long long budget) {
    __shared__ __align__(8) uint64_t bar;
    volatile int never = 0;
    if (threadIdx.x == 0) {
        tc::mbar_init(&bar, 1);  // one arrival completes phase 0; none is ever made
        tc::fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0 && !tc::mbar_wait(&bar, 0, &never, budget)) atomicCAS(&g_tc_status, 0u, kSelftestCode);
}
}  // namespace
}  // namespace bb

extern "C" int blade_wait_selftest(uint64_t budget_cycles, blade_stream_t stream) {
    using namespace bb;
    if (budget_cycles == 0 || budget_cycles > 10000000000ull)
        return set_error(BLADE_ERROR, "blade_wait_selftest: budget must be 1 .. 1e10 cycles (got %llu)",
                         (unsigned long long)budget_cycles);
    wait_selftest_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>((long long)budget_cycles);
    return check_launch("blade_wait_selftest");
}

// ---- allocation-free variant ---------------------------------------------------
// For callers that must not allocate device memory while they stream: an online
// beamformer that sizes its whole GPU budget once at start-up and then runs a
// fixed-cadence loop cannot call cudaMalloc / cudaFree per block, because those
// calls synchronise the device and take unbounded time, which the loop's
// real-time deadline cannot absorb.  This entry point keeps the phasor image in a
// fixed device array that every GPU loading the library holds until exit.

// Scratch for the phasor image: 8 MiB per device.
static __device__ __align__(256) uint8_t g_tc_noalloc_plan[8u << 20];

namespace {

constexpr uint64_t kNoAllocPlanBytes = 8ull << 20;

template <typename Fn>
int driver_entry(const char* name, unsigned version, Fn* fn) {
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    if (cudaGetDriverEntryPointByVersion(name, &p, version, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !p)
        return set_error(BLADE_CUDA_ERROR, "blade_beamform_detect_tc_noalloc: %s unavailable", name);
    *fn = reinterpret_cast<Fn>(p);
    return BLADE_SUCCESS;
}

// Device address of g_tc_noalloc_plan, looked up with the device current (the
// host-side name is only a stand-in for the device array) once per device and
// context: the cache is keyed on the current context's unique id as well, so
// after a cudaDeviceReset, which destroys the primary context and this module's
// copy of the array with it, the next call looks the address up again.
int noalloc_plan_address(void** out) {
    static std::mutex mu;
    static void* addr[64] = {nullptr};
    static unsigned long long ctx_of[64] = {0};
    static PFN_cuCtxGetCurrent_v4000 get_current = nullptr;
    static PFN_cuCtxGetId_v12000 get_id = nullptr;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return check_cuda(e, "blade_beamform_detect_tc_noalloc");
    if (dev < 0 || dev >= 64) return set_error(BLADE_ERROR, "blade_beamform_detect_tc_noalloc: device %d", dev);
    // makes the device's primary context current, creating it if a reset destroyed it
    e = cudaSetDevice(dev);
    if (e != cudaSuccess) return check_cuda(e, "blade_beamform_detect_tc_noalloc: cudaSetDevice");
    std::lock_guard<std::mutex> lock(mu);
    if (!get_current) {
        if (int rc = driver_entry("cuCtxGetCurrent", 4000, &get_current)) return rc;
        if (int rc = driver_entry("cuCtxGetId", 12000, &get_id)) return rc;
    }
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS)
        return set_error(BLADE_CUDA_ERROR, "blade_beamform_detect_tc_noalloc: no current CUDA context");
    if (!addr[dev] || ctx_of[dev] != id) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_tc_noalloc_plan);
        if (e != cudaSuccess) return check_cuda(e, "blade_beamform_detect_tc_noalloc: cudaGetSymbolAddress");
        addr[dev] = p;
        ctx_of[dev] = id;
    }
    *out = addr[dev];
    return BLADE_SUCCESS;
}

}  // namespace

extern "C" int blade_beamform_detect_tc_noalloc(const void* in, const void* phasors, void* out, uint64_t B,
                                                uint64_t A, uint64_t F, uint64_t T, uint64_t P, uint64_t rate,
                                                uint64_t integration, blade_stream_t stream) {
    if (!blade_beamform_detect_tc_supported(B, A, F, T, P, rate, integration))
        return set_error(BLADE_ERROR,
                         "blade_beamform_detect_tc_noalloc: unsupported configuration (needs P=2, 1<=A<=64, "
                         "T%%128==0, rate in {1,2,4}, I a power of two <= 32)");
    const uint64_t need = blade_beamform_tc_plan_size(B, A, F, P);
    if (need > kNoAllocPlanBytes)
        return set_error(BLADE_ERROR,
                         "blade_beamform_detect_tc_noalloc: the phasor image for B=%llu A=%llu F=%llu needs %llu "
                         "bytes, above the %llu-byte static workspace; use blade_beamform_tc_prepare + "
                         "blade_beamform_detect_tc with a caller-allocated image",
                         (unsigned long long)B, (unsigned long long)A, (unsigned long long)F,
                         (unsigned long long)need, (unsigned long long)kNoAllocPlanBytes);
    void* plan = nullptr;
    if (int rc = noalloc_plan_address(&plan)) return rc;
    return blade_beamform_prepare_detect_tc(phasors, plan, in, out, B, A, F, T, P, rate, integration, stream);
}

// ---- autotuner ------------------------------------------------------------------

namespace bb {
namespace {

// Device buffers of one tuning run, freed on every return path.
struct DevBufs {
    std::vector<void*> p;
    ~DevBufs() {
        for (void* q : p) cudaFree(q);
    }
    void* get(size_t bytes) {
        void* q = nullptr;
        if (cudaMalloc(&q, bytes < 16 ? 16 : bytes) != cudaSuccess) return nullptr;
        p.push_back(q);
        return q;
    }
};

}  // namespace

// Output bytes a and b (device) are identical; false on a copy failure too.
bool tune_same(const void* a, const void* b, size_t bytes) {
    std::vector<uint8_t> ha(bytes), hb(bytes);
    if (cudaMemcpy(ha.data(), a, bytes, cudaMemcpyDeviceToHost) != cudaSuccess) return false;
    if (cudaMemcpy(hb.data(), b, bytes, cudaMemcpyDeviceToHost) != cudaSuccess) return false;
    return memcmp(ha.data(), hb.data(), bytes) == 0;
}

int tc_query(const uint64_t (&shape)[8], uint32_t* params, float* us, int* tuned) {
    TcShape s;
    bool t = false;
    TuneEntry e;
    const uint32_t es = shape[7] ? (uint32_t)shape[7] : 4u;
    uint32_t segs, seg_tiles;
    const bool ok = shape[7] == kTuneSelf
                        ? blade_beamform_detect_tc_supported(shape[0], shape[1], shape[2], shape[3], 2, shape[5], shape[6]) &&
                              tc_self_layout(shape[0], shape[1], shape[2], shape[3], shape[5], shape[6], s, segs, seg_tiles, &t, &e)
                        : tc_layout(shape[0], shape[1], shape[2], shape[3], shape[5], shape[6], es, s, &t, &e);
    if (shape[4] != 2 || !ok) return set_error(BLADE_ERROR, "blade_autotune_query: unsupported tensor-core shape");
    const TcChoice c = tc_choice_of(s);
    for (int i = 0; i < kTuneParams; i++) params[i] = t ? e.params[i] : 0u;
    params[0] = c.mode;
    params[1] = c.a_stages;
    params[2] = c.r_stages;
    params[3] = c.raw_tiles;
    *us = t ? e.us : 0.f;
    *tuned = t ? 1 : 0;
    return BLADE_SUCCESS;
}

}  // namespace bb

extern "C" int blade_beamform_detect_tc_autotune(uint64_t B, uint64_t A, uint64_t F, uint64_t T, uint64_t P,
                                                 uint64_t rate, uint64_t integration, blade_stream_t stream) {
    using namespace bb;
    const char* who = "blade_beamform_detect_tc_autotune";
    if (!blade_beamform_detect_tc_supported(B, A, F, T, P, rate, integration))
        return set_error(BLADE_ERROR, "%s: unsupported configuration", who);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const uint64_t U = T / (rate * integration);
    const size_t in_bytes = (size_t)A * F * T * 4, ph_count = (size_t)B * A * F * 2;
    const size_t plan_bytes = blade_beamform_tc_plan_size(B, A, F, P);
    const size_t out_bytes = (size_t)B * F * rate * U * sizeof(float);
    DevBufs bufs;
    void* in = bufs.get(in_bytes);
    void* ph = bufs.get(ph_count * sizeof(float2));
    void* plan = bufs.get(plan_bytes);
    void* ref = bufs.get(out_bytes);
    void* out = bufs.get(out_bytes);
    if (!in || !ph || !plan || !ref || !out) return set_error(BLADE_CUDA_ERROR, "%s: allocation failed", who);
    if (int rc = tune_fill_ci8(in, in_bytes, st)) return rc;
    if (int rc = tune_fill_phasors(ph, ph_count, st)) return rc;
    if (int rc = blade_beamform_tc_prepare(ph, plan, B, A, F, P, stream)) return rc;
    TcShape base;
    tc_shape(B, A, base, T, 4, rate);
    // candidates: the default first, then every ring layout that fits
    std::vector<TcChoice> cands{tc_choice_of(base)};
    auto add = [&](TcChoice c) {
        for (const auto& d : cands)
            if (d.mode == c.mode && d.a_stages == c.a_stages && d.r_stages == c.r_stages && d.raw_tiles == c.raw_tiles)
                return;
        TcShape t = base;
        if (tc_apply(t, A, T, 4, rate, c)) cands.push_back(c);
    };
    const uint32_t rings[][2] = {{8, 2}, {8, 3}, {6, 2}, {4, 4}, {4, 3}, {4, 2}, {2, 4}, {2, 2}};
    for (uint32_t rt : {2u, 1u})
        for (const auto& r : rings) add(TcChoice{0, r[0], r[1], rt});
    for (uint32_t a : {8u, 6u, 4u}) add(TcChoice{1, a, 0, 1});
    // The plain chain, then, for a block whose prepared call splits its phasors inside the
    // chain kernel, that launch.
    uint32_t segs, seg_tiles;
    const bool small = self_shape(base, F, T, rate, segs, seg_tiles);
    for (int self = 0; self <= (small ? 1 : 0); self++) {
        int best = -1;
        float best_us = 0.f;
        uint32_t ndiff = 0, ntimed = 0;
        for (size_t i = 0; i < cands.size(); i++) {
            TcShape t = base;
            tc_apply(t, A, T, 4, rate, cands[i]);
            if (self && !self_shape(t, F, T, rate, segs, seg_tiles)) continue;
            void* dst = i == 0 ? ref : out;
            const float us = tune_time(
                [&]() {
                    return self ? tc_run(who, in, plan, dst, B, A, F, T, rate, integration, 4,
                                         tc_self_kernel(rate, integration), stream, false, &t,
                                         static_cast<const float2*>(ph), segs, seg_tiles)
                                : tc_run(who, in, plan, dst, B, A, F, T, rate, integration, 4, nullptr, stream, false, &t);
                },
                st);
            if (us < 0.f) return set_error(BLADE_CUDA_ERROR, "%s: candidate %zu failed: %s", who, i, blade_last_error());
            uint32_t status = 0;
            if (int rc = blade_device_status(&status)) return rc;
            if (status != 0) return set_error(BLADE_CUDA_ERROR, "%s: candidate %zu: device status %u", who, i, status);
            ntimed++;
            if (i > 0 && !tune_same(ref, out, out_bytes)) {
                ndiff++;
                continue;
            }
            if (best < 0 || us < best_us) {
                best = (int)i;
                best_us = us;
            }
        }
        TuneEntry e = {};
        e.params[0] = cands[best].mode;
        e.params[1] = cands[best].a_stages;
        e.params[2] = cands[best].r_stages;
        e.params[3] = cands[best].raw_tiles;
        e.params[4] = ntimed;
        e.params[5] = ndiff;
        e.us = best_us;
        const uint64_t key[8] = {B, A, F, T, P, rate, integration, self ? kTuneSelf : 4};
        tune_store(BLADE_TUNE_TC, key, e);
    }
    return BLADE_SUCCESS;
}
