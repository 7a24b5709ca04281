// demod.cu — quadrature demodulation + decimating FIR (reference
// demodulate.cpp:36-121).
//
// Layout: RF [trace][n_in] float -> IQ [trace][n_out] complex, trace =
// event*n_channels + channel.
//
// demod_slide_kernel<NT, R> (no decimation, NT taps; the default 33-tap filter):
// a warp filters a segment of 32 R output samples of up to four traces in
// turn; the block's eight warps share the segment's rotator. The 32 R + NT - 1
// input samples go to the warp's own row of shared memory already mixed to
// baseband (a lane's samples are lane + 32 m: no index arithmetic, and the next
// trace's are fetched behind the filter). Lane l then produces outputs R l ..
// R l + R - 1 from one descending pass over its R + NT - 1 window samples, each
// sample read from shared memory once and multiplied into every output it
// reaches (the taps are compile-time constant-bank operands); R is odd, so that
// lanes reading R-sample strides hit distinct banks. Every output still sums its
// taps in ascending order, as the reference does. The outputs go back through
// the warp's own shared-memory row so the IQ stores are coalesced. Samples
// outside the trace are staged as zeros: an output whose tap range the
// reference clips (j_lo > 0 or j_hi < NT-1) then adds exact zeros outside
// that range, which leaves its sum unchanged.
// 75 x 128 traces x 2,073 samples: 55 us (239 MB at 4.3 TB/s), where staging by
// the whole block with a division per sample and eight outputs per lane took 82;
// bound by issue (the 33 packed FMAs per output alone are 35 us of FP32 pipe).
// Three blocks per SM 57.8 us, five (51 registers) 63.7, taps stored twice as
// packed operands the same.
//
// demod_kernel (any decimation or tap count): a block owns 8 traces x 128
// outputs, one output per thread per trace, taps read from the parameter
// block in a runtime loop, the eight traces' sums side by side in it (one
// trace after the other was a single chain of dependent FMAs): 75 x 128 traces
// x 2,073 samples, 47 taps 304 -> 213 us; 33 taps, decimation 4 255 -> 154 us.
// Bound by shared memory, one 8-byte read per tap.
//
// Arithmetic follows the reference term by term (mix, then tap product and
// accumulation in ascending tap order, then x2); the tap product and the
// accumulation are one FMA (~1e-7 relative from the reference's separate
// multiply and add); the mixing phase -2*pi*f*t(n) is evaluated on the device
// with sincosf.
#include <algorithm>
#include <vector>

#include "usx_internal.cuh"

namespace usxcu {
namespace {

constexpr int kMaxTaps = 255;
constexpr int kTraces = 8;
constexpr int kOut = 128;

struct DemodParams {
  const float* rf;
  float2* iq;
  long n_traces;
  int n_in, n_out, dec, n_taps, gd;
  float neg_two_pi_f;   // -2*pi*fdem, float-rounded as the reference folds it
  float t0, fs;
  int per_warp;         // traces a warp filters in turn (demod_slide_kernel)
  float h[kMaxTaps];
};

template <int kT>   // traces of a block
__global__ void __launch_bounds__(kOut) demod_kernel(const DemodParams p) {
  extern __shared__ float4 smem_raw[];
  const int span = kOut * p.dec + p.n_taps - 1;
  float2* rot = reinterpret_cast<float2*>(smem_raw);          // [span]
  float2* mixed = rot + span;                                 // [kT][span]

  const int k0 = blockIdx.y * kOut;
  const long tr0 = static_cast<long>(blockIdx.x) * kT;
  // Input index of mixed[0]: centre(k0) - (n_taps - 1).
  const int n_base = k0 * p.dec + p.gd - (p.n_taps - 1);

  for (int s = threadIdx.x; s < span; s += blockDim.x) {
    const int n = n_base + s;
    float2 r = make_float2(0.f, 0.f);
    if (n >= 0 && n < p.n_in) {
      const float t = p.t0 + static_cast<float>(n) / p.fs;
      const float ph = p.neg_two_pi_f * t;
      float sv, cv;
      sincosf(ph, &sv, &cv);
      r = make_float2(cv, sv);
    }
    rot[s] = r;
  }
  for (int s = threadIdx.x; s < span; s += kOut) {
    const int n = n_base + s;
    const bool in = n >= 0 && n < p.n_in;
    const float2 r = rot[s];   // this thread's own
    float x[kT];
#pragma unroll
    for (int t = 0; t < kT; ++t)
      x[t] = in && tr0 + t < p.n_traces ? __ldg(p.rf + (tr0 + t) * p.n_in + n) : 0.f;
#pragma unroll
    for (int t = 0; t < kT; ++t) mixed[t * span + s] = make_float2(r.x * x[t], r.y * x[t]);
  }
  __syncthreads();

  const int k = k0 + threadIdx.x;
  if (k >= p.n_out) return;
  const int centre = k * p.dec + p.gd;
  const int j_lo = max(0, centre - p.n_in + 1);
  const int j_hi = min(p.n_taps - 1, centre);
  // mixed index of input sample (centre - j) is centre - j - n_base.
  const float2* m = mixed + (centre - n_base);
  float2 acc[kT];
#pragma unroll
  for (int t = 0; t < kT; ++t) acc[t] = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int j = j_lo; j <= j_hi; ++j) {
    const float2 h = make_float2(p.h[j], p.h[j]);
#pragma unroll
    for (int t = 0; t < kT; ++t) acc[t] = __ffma2_rn(m[t * span - j], h, acc[t]);
  }
#pragma unroll
  for (int t = 0; t < kT; ++t)
    if (tr0 + t < p.n_traces) p.iq[(tr0 + t) * p.n_out + k] = make_float2(acc[t].x * 2.0f, acc[t].y * 2.0f);
}

constexpr int kSlideWarps = 8;                   // traces of a block in flight

template <int NT, int R>
__global__ void __launch_bounds__(32 * kSlideWarps, 4) demod_slide_kernel(const __grid_constant__ DemodParams p) {
  constexpr int W = 32 * R + NT - 1;             // window samples per trace
  constexpr int kPer = (W + 31) / 32;
  __shared__ float2 rot[kPer * 32];
  __shared__ float2 mixed[kSlideWarps][kPer * 32];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k0 = blockIdx.y * 32 * R;
  const int n_base = k0 + p.gd - (NT - 1);       // input index of window sample 0
  const long tr_end = min(p.n_traces, (blockIdx.x + 1L) * kSlideWarps * p.per_warp);
  long tr = blockIdx.x * static_cast<long>(kSlideWarps) * p.per_warp + warp;

  // A lane's samples are lane + 32 m of every trace.
  unsigned in = 0;
#pragma unroll
  for (int m = 0; m < kPer; ++m) {
    const int n = n_base + lane + 32 * m;
    if (n >= 0 && n < p.n_in) in |= 1u << m;
  }
  float x[kPer];
  auto fetch = [&](long t) {
    const float* src = p.rf + t * p.n_in + n_base + lane;
#pragma unroll
    for (int m = 0; m < kPer; ++m) x[m] = (in >> m & 1u) ? __ldg(src + 32 * m) : 0.f;
  };
  if (tr < tr_end) fetch(tr);
  for (int s = threadIdx.x; s < kPer * 32; s += 32 * kSlideWarps) {
    const int n = n_base + s;
    float2 r = make_float2(0.f, 0.f);
    if (n >= 0 && n < p.n_in) {
      const float t = p.t0 + static_cast<float>(n) / p.fs;
      const float ph = p.neg_two_pi_f * t;
      float sv, cv;
      sincosf(ph, &sv, &cv);
      r = make_float2(cv, sv);
    }
    rot[s] = r;
  }
  __syncthreads();

  float2* row = mixed[warp];
  for (; tr < tr_end; tr += kSlideWarps) {
#pragma unroll
    for (int m = 0; m < kPer; ++m) {
      const float2 r = rot[lane + 32 * m];
      row[lane + 32 * m] = make_float2(r.x * x[m], r.y * x[m]);
    }
    __syncwarp();
    if (tr + kSlideWarps < tr_end) fetch(tr + kSlideWarps);   // the next trace's, behind the filter
    // (re, im) of each output accumulate as one packed pair (two FP32 FMAs per
    // instruction, each rounded as fmaf).
    float2 acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = make_float2(0.f, 0.f);
    // Window sample i of this lane is s = R * lane + i; output r uses tap
    // j = r + NT - 1 - i, so descending i visits each output's taps in ascending j.
#pragma unroll
    for (int i = R + NT - 2; i >= 0; --i) {
      const float2 v = row[R * lane + i];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int j = r + NT - 1 - i;
        if (j >= 0 && j < NT) acc[r] = __ffma2_rn(v, make_float2(p.h[j], p.h[j]), acc[r]);
      }
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; ++r) row[R * lane + r] = make_float2(acc[r].x * 2.0f, acc[r].y * 2.0f);
    __syncwarp();
    float2* dst = p.iq + tr * p.n_out + k0 + lane;
    const int n_here = p.n_out - k0 - lane;
#pragma unroll
    for (int q = 0; q < R; ++q)
      if (32 * q < n_here) dst[32 * q] = row[lane + 32 * q];
    __syncwarp();
  }
}

constexpr int kMaxSegments = 65535;   // gridDim.y

template <int NT, int R>
int launch_slide(usx_ctx* ctx, DemodParams& p) {
  const int gy = ceil_div(p.n_out, 32 * R);
  // Up to four traces per warp while eight blocks per SM (two waves) remain.
  p.per_warp = static_cast<int>(std::max(1L, std::min(4L, p.n_traces * gy / (kSlideWarps * 8L * ctx->sm_count))));
  const long per_block = static_cast<long>(kSlideWarps) * p.per_warp;
  const long gx = (p.n_traces + per_block - 1) / per_block;
  if (gx > 0x7fffffffL || gy > kMaxSegments)
    return fail(USX_ERR_UNSUPPORTED, "usx_cu_demodulate: acquisition too large");
  prof_begin(ctx, "demod_slide_kernel");
  demod_slide_kernel<NT, R>
      <<<dim3(static_cast<unsigned>(gx), static_cast<unsigned>(gy)), 32 * kSlideWarps, 0, ctx->stream>>>(p);
  prof_end(ctx);
  USX_CHECK_LAUNCH("demod_slide_kernel");
  return USX_OK;
}

// Outputs per lane: the time follows the outputs with their padding (segments x
// R), so the R with the fewest; the larger on a tie, which reads less of the
// window twice. 75 x 128 traces, 33 taps, R = 7 / 9 / 11 / 13: 2,073 samples
// (70 / 72 / 66 / 65 x 32 outputs) 60.1 / 63.4 / 57.6 / 55.6 us; 1,034 samples
// (35 / 36 / 33 / 39) 33.5 / 34.9 / 32.9 / 37.0. While the blocks of R = 7 are not
// four per SM a warp's own chain counts, and the shortest is R = 7 (32 traces
// of 660 samples 4.3 us, with R = 11 6.1).
template <int NT>
int launch_slide_r(usx_ctx* ctx, DemodParams& p) {
  auto cost = [&](int r) { return ceil_div(p.n_out, 32 * r) * r; };
  const long blocks = (p.n_traces + kSlideWarps - 1) / kSlideWarps * ceil_div(p.n_out, 32 * 7);
  // Segments are the grid's second dimension: past its limit with R = 7 (traces
  // of 14,679,840 samples), the longest segment.
  if (ceil_div(p.n_out, 32 * 7) > kMaxSegments) return launch_slide<NT, 13>(ctx, p);
  if (blocks > 4L * ctx->sm_count) {
    if (cost(13) <= cost(11) && cost(13) <= cost(7)) return launch_slide<NT, 13>(ctx, p);
    if (cost(11) <= cost(7)) return launch_slide<NT, 11>(ctx, p);
  }
  return launch_slide<NT, 7>(ctx, p);
}

}  // namespace
}  // namespace usxcu

using namespace usxcu;

extern "C" int usx_cu_demodulate(usx_ctx* ctx, const usx_channel_desc* cd,
                                 const usx_demod_config* cfg, const float* rf, float* iq,
                                 float* out_fdem) {
  if (!ctx || !cd || !cfg || !rf || !iq) return fail(USX_ERR_INVALID, "usx_cu_demodulate: null argument");
  if (cd->is_iq) return fail(USX_ERR_INVALID, "usx_cu_demodulate: input already holds IQ");
  if (int rc = validate_channel(*cd)) return rc;
  const float fdem = cfg->demodulation_frequency > 0.0f ? cfg->demodulation_frequency
                                                        : cd->probe.center_frequency;
  const int dec = std::max(1, cfg->decimation);
  const float fs = cd->acq.sampling_frequency;
  DemodParams p;
  int n_taps = 0;
  usx_cu_design_lowpass(cfg->filter_taps, cfg->cutoff_fraction * fdem / fs, nullptr, 0, &n_taps);
  if (n_taps > kMaxTaps) return fail(USX_ERR_UNSUPPORTED, "usx_cu_demodulate: more than 255 filter taps");
  if (dec > 32) return fail(USX_ERR_UNSUPPORTED, "usx_cu_demodulate: decimation above 32");
  usx_cu_design_lowpass(cfg->filter_taps, cfg->cutoff_fraction * fdem / fs, p.h, kMaxTaps, &n_taps);
  p.rf = rf;
  p.iq = reinterpret_cast<float2*>(iq);
  p.n_traces = static_cast<long>(cd->n_events) * cd->probe.n_elements;
  p.n_in = cd->acq.n_samples;
  p.n_out = (p.n_in + dec - 1) / dec;
  p.dec = dec;
  p.n_taps = n_taps;
  p.gd = n_taps / 2;
  p.neg_two_pi_f = -2.0f * kPi * fdem;
  p.t0 = cd->acq.t0;
  p.fs = fs;
  if (out_fdem) *out_fdem = fdem;
  if (dec == 1 && (n_taps == 33 || n_taps == 21)) {
    return n_taps == 33 ? launch_slide_r<33>(ctx, p) : launch_slide_r<21>(ctx, p);
  }
  const int span = kOut * dec + n_taps - 1;
  const size_t smem = sizeof(float2) * static_cast<size_t>(span) * (1 + kTraces);
  // Blocks of as many traces as there are: sums of absent ones cost as much (one
  // trace of 8,192 samples, 33 taps, decimation 4: 10.3 us as one of eight, 5.7
  // alone). From five on, one of eight is as fast (127 taps, decimation 16: 73).
  void (*const kernel)(DemodParams) = p.n_traces == 1  ? demod_kernel<1>
                                      : p.n_traces == 2 ? demod_kernel<2>
                                      : p.n_traces <= 4 ? demod_kernel<4>
                                                        : demod_kernel<kTraces>;
  if (smem > 48 * 1024)
    if (int rc_ = smem_limit(reinterpret_cast<const void*>(kernel), smem)) return rc_;
  const long gx = (p.n_traces + kTraces - 1) / kTraces;
  const int gy = ceil_div(p.n_out, kOut);
  if (gx > 0x7fffffffL || gy > 65535) return fail(USX_ERR_UNSUPPORTED, "usx_cu_demodulate: acquisition too large");
  dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy));
  prof_begin(ctx, "demod_kernel");
  kernel<<<grid, kOut, smem, ctx->stream>>>(p);
  prof_end(ctx);
  USX_CHECK_LAUNCH("demod_kernel");
  return USX_OK;
}
