// doppler.cu — polynomial-regression wall filter, colour flow (Kasai/Loupas
// autocorrelation with coherence and power gates), power Doppler, two-stage
// axial displacement tracking and least-squares strain (reference
// doppler.cpp:15-305).
//
// Ensembles are [frame][pixel] complex. The (I - P) clutter projector depends
// only on the ensemble length and is built on the host with the reference's
// float Gram-Schmidt (bit-identical), then applied per pixel on the device.
// Every per-pixel sum runs in the reference's loop order (lateral offset,
// axial offset, frame), so the maps match the reference to the last ulp of
// the device's atan2f/hypotf.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <vector>

#include "usx_internal.cuh"

namespace usxcu {
namespace {

constexpr int kMaxEns = 64;

// doppler.cpp:15-47, host float arithmetic.
std::vector<float> reject_matrix(int n, int order) {
  order = std::min(std::max(order, 0), n - 1);
  const int p = order + 1;
  std::vector<std::vector<float>> basis;
  for (int d = 0; d < p; ++d) {
    std::vector<float> v(static_cast<size_t>(n));
    for (int k = 0; k < n; ++k) {
      const float x = (n == 1) ? 0.0f : 2.0f * static_cast<float>(k) / static_cast<float>(n - 1) - 1.0f;
      v[static_cast<size_t>(k)] = static_cast<float>(std::pow(static_cast<double>(x), static_cast<double>(d)));
    }
    for (const auto& b : basis) {
      float dot = 0;
      for (int k = 0; k < n; ++k) dot += v[static_cast<size_t>(k)] * b[static_cast<size_t>(k)];
      for (int k = 0; k < n; ++k) v[static_cast<size_t>(k)] -= dot * b[static_cast<size_t>(k)];
    }
    float norm = 0;
    for (float x : v) norm += x * x;
    norm = std::sqrt(norm);
    if (norm < 1e-8f) continue;
    for (float& x : v) x /= norm;
    basis.push_back(v);
  }
  std::vector<float> M(static_cast<size_t>(n) * n, 0.0f);
  for (int i = 0; i < n; ++i) M[static_cast<size_t>(i) * n + i] = 1.0f;
  for (const auto& b : basis)
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j)
        M[static_cast<size_t>(i) * n + j] -= b[static_cast<size_t>(i)] * b[static_cast<size_t>(j)];
  return M;
}

struct WallArgs {
  const float2* ens;
  float2* out;          // filtered ensemble, or nullptr
  float* power;         // power Doppler sum, or nullptr
  long n_pix;
  int n;
  int identity;         // WallFilter::None: copy through
  float M[kMaxEns * kMaxEns];
};

// The wall filter: a pixel per thread, its ensemble z[n][kWallThreads] in shared
// memory, filtered frame i of src[j * n_pix] through the n x n projector M to
// store(i, value), ascending i. Eight rows at a time (four, two and one of what is
// left) share each read of z; M is read where the kernel's arguments lie; every row
// sums over j in ascending order, products and sums rounded separately. (in: the
// pixel exists. src may be the frames that store writes: a thread reads its pixel
// whole before it writes, and by ordinary loads.)
// What bounds it: latency at the occupancy that 1 KB per frame and block leaves.
// Polynomial filter of order 2, 131,072 pixels, us, a row at a time / this: 8
// frames 10 / 11, 16 18.8 / 16.9, 32 43 / 39, 48 90 / 79, 56 120 / 127, 64 181 /
// 134. M transposed in shared memory, for 16-byte reads of it, leaves fewer blocks
// beside one another: 17.9, 44, 149, 238 and 220 from 16 frames on; only from
// 262,144 pixels on, at 14 to 24 frames, is it the faster one (524,288 pixels, 16
// frames, 39 against 46).
constexpr int kWallThreads = 128;
__host__ __device__ constexpr size_t wall_smem(int n) { return sizeof(float2) * n * kWallThreads; }

template <typename Store>
__device__ __forceinline__ void wall_pixel(float4* smem, const float2* src, long n_pix, int n, const float* M,
                                           bool identity, bool in, Store store) {
  if (!in) return;
  float2* z = reinterpret_cast<float2*>(smem) + threadIdx.x;
#pragma unroll 8
  for (int j = 0; j < n; ++j) z[j * kWallThreads] = src[j * n_pix];
  if (identity) {
    for (int i = 0; i < n; ++i) store(i, z[i * kWallThreads]);
    return;
  }
  int i = 0;
  auto rows = [&](auto count) {   // the next count rows
    constexpr int R = decltype(count)::value;
    float2 acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = make_float2(0.f, 0.f);
#pragma unroll 2
    for (int j = 0; j < n; ++j) {
      const float2 v = z[j * kWallThreads];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float m = M[(i + r) * n + j];
        acc[r].x += v.x * m;
        acc[r].y += v.y * m;
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) store(i + r, acc[r]);
    i += R;
  };
  while (i + 8 <= n) rows(std::integral_constant<int, 8>{});
  if (i + 4 <= n) rows(std::integral_constant<int, 4>{});
  if (i + 2 <= n) rows(std::integral_constant<int, 2>{});
  if (i < n) rows(std::integral_constant<int, 1>{});
}

__global__ void __launch_bounds__(kWallThreads) wall_kernel(const WallArgs a) {
  extern __shared__ float4 wall_s[];
  const long k = blockIdx.x * static_cast<long>(kWallThreads) + threadIdx.x;
  float p = 0.0f;
  wall_pixel(wall_s, a.ens + k, a.n_pix, a.n, a.M, a.identity, k < a.n_pix, [&](int i, float2 v) {
    if (a.out) a.out[i * a.n_pix + k] = v;
    p += cnorm(mk(v.x, v.y));
  });
  if (a.power && k < a.n_pix) a.power[k] = p;
}

struct FlowArgs {
  const float2* filt;   // [n][n0*n1]
  int n, n0, n1, ka, kl, loupas;
  float dz, fdem, prf, c, coh_thr;
  float* velocity;
  float* power;
  float* variance;
  uint8_t* valid;
  unsigned* pmax_bits;
};

// Velocity, power, variance and the coherence gate of one pixel from its sums.
__device__ __forceinline__ void flow_finish(const FlowArgs& a, long k, float R00, cplx R01, cplx R10) {
  float vel = 0.0f, var = 0.0f;
  uint8_t ok = 0;
  if (R00 > 0.0f) {
    const float coherence = cabsf_(R01) / R00;
    var = fclamp(2.0f * (1.0f - coherence), 0.0f, 1.0f);
    if (!(coherence < a.coh_thr)) {
      const float phase_slow = atan2f(R01.im, R01.re);
      float f_centre = a.fdem;
      if (a.loupas) {
        const float phase_fast = atan2f(R10.im, R10.re);
        const float f_est = phase_fast * a.c / (4.0f * kPi * a.dz);
        if (f_est > 0.25f * a.fdem && f_est < 2.0f * a.fdem) f_centre = f_est;
      }
      if (f_centre > 0.0f) {
        vel = -phase_slow * a.c * a.prf / (4.0f * kPi * f_centre);
        ok = 1;
      }
    }
  }
  a.velocity[k] = vel;
  a.power[k] = R00;
  a.variance[k] = var;
  a.valid[k] = ok;
}

// The warp's largest power into the frame's maximum (every lane calls it;
// power is non-negative, so its bit pattern orders like its value).
__device__ __forceinline__ void flow_peak(const FlowArgs& a, float power) {
  const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(power, 0.0f)));
  if ((threadIdx.x & 31) == 0) atomicMax(a.pmax_bits, m);
}

__device__ __forceinline__ void flow_pixel(const FlowArgs& a) {
  const long k0 = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  const long n_pix = static_cast<long>(a.n0) * a.n1;
  // Out-of-range lanes evaluate the last pixel but do not store, so that the
  // whole warp reaches the max reduction below.
  const bool in_range = k0 < n_pix;
  const long k = in_range ? k0 : n_pix - 1;
  const int i = static_cast<int>(k / a.n1), j = static_cast<int>(k - static_cast<long>(i) * a.n1);
  cplx R01 = mk(0.f, 0.f), R10 = mk(0.f, 0.f);
  float R00 = 0.0f;
  for (int di = -a.kl; di <= a.kl; ++di) {
    const int ii = i + di;
    if (ii < 0 || ii >= a.n0) continue;
    for (int dj = -a.ka; dj <= a.ka; ++dj) {
      const int jj = j + dj;
      if (jj < 0 || jj >= a.n1) continue;
      const long kk = static_cast<long>(ii) * a.n1 + jj;
      for (int e = 0; e < a.n; ++e) {
        const float2 zf = a.filt[e * n_pix + kk];
        const cplx z = mk(zf.x, zf.y);
        R00 += cnorm(z);
        if (e + 1 < a.n) {
          const float2 w = a.filt[(e + 1) * n_pix + kk];
          R01 = cadd(R01, cmul(cconj(z), mk(w.x, w.y)));
        }
        if (jj + 1 < a.n1) {
          const float2 w = a.filt[e * n_pix + kk + 1];
          R10 = cadd(R10, cmul(cconj(z), mk(w.x, w.y)));
        }
      }
    }
  }
  if (in_range) flow_finish(a, k, R00, R01, R10);
  flow_peak(a, R00);
}

constexpr int kFlowCols = 128;   // depths per block of the line kernels

// The same sums for kFlowLines lateral lines per thread, a block of kFlowCols
// depths. An output's sums run over its window in (line, depth, frame) order,
// so a product z_e^* z_e+1 formed once for (line, depth, frame) can be added to
// each of the thread's outputs (up to 2 kKL + 1) whose window holds that line,
// and every output still adds its terms in that order: the maps equal
// flow_pixel's bit for bit. The block's lines pass through shared memory one
// at a time, all frames of each ([frame][depth], halo included, zeros outside
// the grid), because the frames are the innermost loop: read through L1, the
// frames of a line are evicted before the next depth of the window reads them
// again (413 us).
// What bounds it: dependent issue at 24 warps per SM (35 KB of shared memory
// per block at 32 frames). 8 ensembles of 8 to 32 frames, 256 x 512, 9 x 3
// windows: 333 us, flow_kernel's pixel per thread 469; 13 x 5 windows: 590
// against 1,080. Eight lines: 306 and 550, but half the threads (one ensemble
// of 32 frames 142 us against 108). The open outputs in a rolling set of
// registers, any number of lines: 394 to 556. A branch without the last
// depth's selects doubles the unrolled code: 358.
constexpr int kFlowLines = 4;
template <int kKL>
__device__ __forceinline__ void flow_lines(const FlowArgs& a) {
  extern __shared__ float2 fl_s[];   // [n][kFlowCols + 2 ka + 1]
  const long n_pix = static_cast<long>(a.n0) * a.n1;
  const int width = kFlowCols + 2 * a.ka + 1;
  const int i0 = blockIdx.y * kFlowLines, j0 = blockIdx.x * kFlowCols;
  const int j = j0 + threadIdx.x;
  float2 R01[kFlowLines], R10[kFlowLines];
  float R00[kFlowLines];
#pragma unroll
  for (int r = 0; r < kFlowLines; ++r) {
    R01[r] = R10[r] = make_float2(0.f, 0.f);
    R00[r] = 0.0f;
  }
#pragma unroll
  for (int q = 0; q < kFlowLines + 2 * kKL; ++q) {   // line i0 - kKL + q
    const int ii = i0 - kKL + q;
    if (ii < 0 || ii >= a.n0) continue;
    __syncthreads();   // the previous line is no longer read
    const float2* line = a.filt + static_cast<long>(ii) * a.n1;
    for (int c = threadIdx.x; c < width; c += kFlowCols) {
      const int jj = j0 - a.ka + c;
      const bool in = jj >= 0 && jj < a.n1;
#pragma unroll 8
      for (int e = 0; e < a.n; ++e) fl_s[e * width + c] = in ? __ldg(line + e * n_pix + jj) : make_float2(0.f, 0.f);
    }
    __syncthreads();
    for (int d = 0; d <= 2 * a.ka; ++d) {
      // z is zero outside the grid; the last depth has no next one.
      const int jj = j - a.ka + d;
      const bool next = jj >= 0 && jj + 1 < a.n1;
      const float2* p = fl_s + threadIdx.x + d;
      float2 z = *p;
      auto add = [&](float2 zc, float2 zn, float2 w, bool last) {
        const float zz = zc.x * zc.x + zc.y * zc.y;
        const float2 zr = next ? zc : make_float2(0.f, 0.f);
        const float2 wr = next ? w : make_float2(0.f, 0.f);
        const float2 fast = make_float2(zr.x * wr.x + zr.y * wr.y, zr.x * wr.y - zr.y * wr.x);
        float2 slow = make_float2(0.f, 0.f);
        if (!last) slow = make_float2(zc.x * zn.x + zc.y * zn.y, zc.x * zn.y - zc.y * zn.x);
#pragma unroll
        for (int r = 0; r < kFlowLines; ++r) {
          if (q < r || q > r + 2 * kKL) continue;   // the line is outside output r's window
          R00[r] += zz;
          if (!last) R01[r] = __fadd2_rn(R01[r], slow);
          R10[r] = __fadd2_rn(R10[r], fast);
        }
      };
#pragma unroll 4
      for (int e = 0; e + 1 < a.n; ++e) {
        const float2 zn = p[(e + 1) * width];
        add(z, zn, p[e * width + 1], false);
        z = zn;
      }
      add(z, z, p[(a.n - 1) * width + 1], true);
    }
  }
  float peak = 0.0f;
#pragma unroll
  for (int r = 0; r < kFlowLines; ++r) {
    const int i = i0 + r;
    if (i >= a.n0 || j >= a.n1) continue;
    flow_finish(a, static_cast<long>(i) * a.n1 + j, R00[r], mk(R01[r].x, R01[r].y), mk(R10[r].x, R10[r].y));
    peak = fmaxf(peak, R00[r]);
  }
  flow_peak(a, peak);
}

__global__ void flow_kernel(const FlowArgs a) { flow_pixel(a); }
template <int kKL>
__global__ void __launch_bounds__(kFlowCols) flow_lines_kernel(const FlowArgs a) {
  flow_lines<kKL>(a);
}

__global__ void power_gate_kernel(const float* power, uint8_t* valid, long n, float ratio,
                                  const unsigned* pmax_bits) {
  const long k = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (k >= n) return;
  const float pmax = __uint_as_float(*pmax_bits);
  if (pmax > 0.0f) {
    const float thr = pmax * ratio;
    if (power[k] < thr) valid[k] = 0;
  }
}

// Batched colour flow (usx_cu_color_flow_batch): all ensembles of one call
// in one wall-filter launch, one flow launch and one gate launch. blockIdx.y
// is the ensemble within a chunk; the per-ensemble lengths and offsets, and
// the clutter projector of every distinct length (they depend only on the
// length), ride in the kernel parameters. Per pixel the arithmetic is that
// of wall_kernel / flow_kernel / power_gate_kernel, so every map equals the
// one-ensemble path bit for bit.
constexpr int kBatchEns = 64;      // ensembles per launch
constexpr int kBatchPool = 6144;   // floats of projectors per launch (24 KB)

struct WallBatchArgs {
  const float2* ens;       // input frames, where the caller packed them
  float2* out;             // filtered frames, packed back to back
  long n_pix;
  int identity;
  int n[kBatchEns];
  int m_off[kBatchEns];    // projector offset in M
  long in_off[kBatchEns];  // first input frame of the ensemble
  long out_off[kBatchEns]; // first filtered frame of the ensemble
  float M[kBatchPool];
};

__global__ void __launch_bounds__(kWallThreads) wall_batch_kernel(const WallBatchArgs a) {
  extern __shared__ float4 wall_s[];
  const int e = blockIdx.y;
  const long k = blockIdx.x * static_cast<long>(kWallThreads) + threadIdx.x;
  const float2* src = a.ens + a.in_off[e] * a.n_pix;
  float2* dst = a.out + a.out_off[e] * a.n_pix;
  wall_pixel(wall_s, src + k, a.n_pix, a.n[e], a.M + a.m_off[e], a.identity, k < a.n_pix,
             [&](int i, float2 v) { dst[i * a.n_pix + k] = v; });
}

struct FlowBatchArgs {
  FlowArgs base;         // filt = packed filtered frames; maps = [ensemble][pixel]
  int n[kBatchEns];
  int ens[kBatchEns];    // ensemble index of this chunk's entry (map row)
  long f_off[kBatchEns];
};

// Entry e of the chunk as one ensemble's arguments.
__device__ __forceinline__ FlowArgs flow_entry(const FlowBatchArgs& b, int e) {
  FlowArgs a = b.base;
  const long n_pix = static_cast<long>(a.n0) * a.n1;
  const long row = b.ens[e];
  a.n = b.n[e];
  a.filt = b.base.filt + b.f_off[e] * n_pix;
  a.velocity += row * n_pix;
  a.power += row * n_pix;
  a.variance += row * n_pix;
  a.valid += row * n_pix;
  a.pmax_bits += row;
  return a;
}
__global__ void flow_batch_kernel(const FlowBatchArgs b) { flow_pixel(flow_entry(b, blockIdx.y)); }
template <int kKL>
__global__ void __launch_bounds__(kFlowCols) flow_lines_batch_kernel(const FlowBatchArgs b) {
  flow_lines<kKL>(flow_entry(b, blockIdx.z));
}

__global__ void power_gate_batch_kernel(const float* power, uint8_t* valid, long n, float ratio,
                                        const unsigned* pmax_bits) {
  const long row = blockIdx.y;
  const long k = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (k >= n) return;
  const float pmax = __uint_as_float(pmax_bits[row]);
  if (pmax > 0.0f) {
    const float thr = pmax * ratio;
    if (power[row * n + k] < thr) valid[row * n + k] = 0;
  }
}

struct DispArgs {
  const float2* a;
  const float2* b;
  int n0, n1, ka, kl, lag_max;
  float dz, fdem, c;
  float* axial;
  float* corr;
};

// The centre frequency of a pixel's phase slope along depth (the window's
// axial autocorrelation), the demodulation frequency where it is implausible.
__device__ __forceinline__ float disp_centre(const DispArgs& p, cplx R10) {
  const float f_est = atan2f(R10.im, R10.re) * p.c / (4.0f * kPi * p.dz);
  return (f_est > 0.25f * p.fdem && f_est < 2.0f * p.fdem) ? f_est : p.fdem;
}

// Correlation and displacement of a pixel from its best lag.
__device__ __forceinline__ void disp_store(const DispArgs& p, long k, float corr, cplx R, int lag, float f_centre) {
  p.corr[k] = fclamp(corr, 0.0f, 1.0f);
  const float residual = -atan2f(R.im, R.re) * p.c / (4.0f * kPi * f_centre);
  p.axial[k] = static_cast<float>(lag) * p.dz + residual;
}

// One pixel, any window and lag range, clipped to the grid.
__device__ void disp_pixel(const DispArgs& p, int i, int j) {
  const long k = static_cast<long>(i) * p.n1 + j;
  p.axial[k] = 0.0f;
  p.corr[k] = 0.0f;
  cplx R10 = mk(0.f, 0.f);
  for (int di = -p.kl; di <= p.kl; ++di) {
    const int ii = i + di;
    if (ii < 0 || ii >= p.n0) continue;
    for (int dj = -p.ka; dj <= p.ka; ++dj) {
      const int jj = j + dj;
      if (jj < 0 || jj + 1 >= p.n1) continue;
      const long kk = static_cast<long>(ii) * p.n1 + jj;
      const float2 u = p.a[kk], v = p.a[kk + 1];
      R10 = cadd(R10, cmul(cconj(mk(u.x, u.y)), mk(v.x, v.y)));
    }
  }
  const float f_centre = disp_centre(p, R10);
  if (f_centre <= 0.0f) return;
  cplx best_R = mk(0.f, 0.f);
  float best_corr = -1.0f;
  int best_lag = 0;
  for (int lag = -p.lag_max; lag <= p.lag_max; ++lag) {
    cplx R = mk(0.f, 0.f);
    float ea = 0.0f, eb = 0.0f;
    for (int di = -p.kl; di <= p.kl; ++di) {
      const int ii = i + di;
      if (ii < 0 || ii >= p.n0) continue;
      for (int dj = -p.ka; dj <= p.ka; ++dj) {
        const int jj = j + dj;
        const int jl = jj + lag;
        if (jj < 0 || jj >= p.n1 || jl < 0 || jl >= p.n1) continue;
        const float2 u = p.a[static_cast<long>(ii) * p.n1 + jj];
        const float2 v = p.b[static_cast<long>(ii) * p.n1 + jl];
        const cplx A = mk(u.x, u.y), B = mk(v.x, v.y);
        R = cadd(R, cmul(cconj(A), B));
        ea += cnorm(A);
        eb += cnorm(B);
      }
    }
    if (ea <= 0.0f || eb <= 0.0f) continue;
    const float cr = cabsf_(R) / sqrtf(ea * eb);
    if (cr > best_corr) {
      best_corr = cr;
      best_R = R;
      best_lag = lag;
    }
  }
  if (best_corr < 0.0f) return;
  disp_store(p, k, best_corr, best_R, best_lag, f_centre);
}

__global__ void displacement_kernel(const DispArgs p) {
  const long k = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (k >= static_cast<long>(p.n0) * p.n1) return;
  const int i = static_cast<int>(k / p.n1);
  disp_pixel(p, i, static_cast<int>(k - static_cast<long>(i) * p.n1));
}

// The same for kDispLines lateral lines per thread over the interior columns
// [col_lo, col_hi), where no window of any lag is clipped in depth. There
//   * the energy of `before` is one sum for all lags, and that of `after` at a
//     lag is the unshifted window's at the shifted column, so both are formed
//     once per pixel (the block's columns of `after` in shared memory);
//   * a product a^* b at (line, depth) goes to every output of the thread whose
//     window holds the line (up to 2 kKL + 1), and four lags share each load.
// Every sum adds the same terms in the same (line, depth) order as disp_pixel,
// so the maps are equal bit for bit. The first n_edge blocks take the other
// columns, a pixel per thread, beside the interior blocks.
// What bounds it: FP32 issue (the window sums' ordered additions). 256 x 1024,
// 17 x 5 windows, 17 lags: 156 us; 501 us with a pixel per thread, which forms
// its products and both energies anew for every lag.
constexpr int kDispCols = 128, kDispLines = 4, kDispLags = 4;
constexpr int kDispMaxLag = 1024;   // shared memory: 4 (128 + 2 lag_max) floats
struct DispLines {
  DispArgs p;
  int col_lo, col_hi, col_blocks, n_edge;
};
template <int kKL>
__global__ void __launch_bounds__(kDispCols) displacement_lines_kernel(const DispLines q) {
  extern __shared__ float eb_s[];   // [kDispLines][kDispCols + 2 lag_max]
  const DispArgs& p = q.p;
  const int n1 = p.n1, ka = p.ka;
  if (static_cast<int>(blockIdx.x) < q.n_edge) {
    const int n_cols = n1 - (q.col_hi - q.col_lo);
    const long m = static_cast<long>(blockIdx.x) * kDispCols + threadIdx.x;
    if (m >= static_cast<long>(p.n0) * n_cols) return;
    const int i = static_cast<int>(m / n_cols), c = static_cast<int>(m - static_cast<long>(i) * n_cols);
    disp_pixel(p, i, c < q.col_lo ? c : c - q.col_lo + q.col_hi);
    return;
  }
  const int blk = static_cast<int>(blockIdx.x) - q.n_edge;
  const int i0 = blk / q.col_blocks * kDispLines, j0 = q.col_lo + blk % q.col_blocks * kDispCols;
  const int j = j0 + threadIdx.x, width = kDispCols + 2 * p.lag_max;
  // Term t(line, depth) into the sums of the lines whose windows hold it.
  for (int c = threadIdx.x; c < width; c += kDispCols) {
    const int col = j0 - p.lag_max + c;
    float e[kDispLines] = {};
    if (col + ka < n1) {   // (col - ka >= 0 for every interior column and lag)
#pragma unroll
      for (int l = 0; l < kDispLines + 2 * kKL; ++l) {
        const int ii = i0 - kKL + l;
        if (ii < 0 || ii >= p.n0) continue;
        const float2* b = p.b + static_cast<long>(ii) * n1 + col - ka;
        for (int d = 0; d <= 2 * ka; ++d) {
          const float2 v = b[d];
          const float m = v.x * v.x + v.y * v.y;
#pragma unroll
          for (int r = 0; r < kDispLines; ++r)
            if (l >= r && l <= r + 2 * kKL) e[r] += m;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kDispLines; ++r) eb_s[r * width + c] = e[r];
  }
  __syncthreads();
  if (j >= q.col_hi) return;

  float ea[kDispLines] = {}, f_centre[kDispLines], best[kDispLines];
  float2 R10[kDispLines] = {}, best_R[kDispLines] = {};
  int best_lag[kDispLines] = {};
#pragma unroll
  for (int l = 0; l < kDispLines + 2 * kKL; ++l) {
    const int ii = i0 - kKL + l;
    if (ii < 0 || ii >= p.n0) continue;
    const float2* a = p.a + static_cast<long>(ii) * n1 + j - ka;
    float2 u = a[0];
    for (int d = 0; d <= 2 * ka; ++d) {
      const float2 v = a[d + 1];
      const float m = u.x * u.x + u.y * u.y;
      const float2 t = make_float2(u.x * v.x + u.y * v.y, u.x * v.y - u.y * v.x);
#pragma unroll
      for (int r = 0; r < kDispLines; ++r)
        if (l >= r && l <= r + 2 * kKL) {
          ea[r] += m;
          R10[r] = __fadd2_rn(R10[r], t);
        }
      u = v;
    }
  }
#pragma unroll
  for (int r = 0; r < kDispLines; ++r) {
    f_centre[r] = disp_centre(p, mk(R10[r].x, R10[r].y));
    best[r] = -1.0f;
  }
  for (int l0 = -p.lag_max; l0 <= p.lag_max; l0 += kDispLags) {
    float2 R[kDispLines][kDispLags] = {};
#pragma unroll
    for (int l = 0; l < kDispLines + 2 * kKL; ++l) {
      const int ii = i0 - kKL + l;
      if (ii < 0 || ii >= p.n0) continue;
      const float2* a = p.a + static_cast<long>(ii) * n1 + j - ka;
      const float2* b = p.b + static_cast<long>(ii) * n1;
      const int c0 = j - ka + l0;   // column of the first depth at the first lag
      float2 w[kDispLags];
#pragma unroll
      for (int x = 0; x < kDispLags; ++x) w[x] = b[min(c0 + x, n1 - 1)];
#pragma unroll 4
      for (int d = 0; d <= 2 * ka; ++d) {
        const float2 u = a[d];
#pragma unroll
        for (int x = 0; x < kDispLags; ++x) {
          const float2 t = make_float2(u.x * w[x].x + u.y * w[x].y, u.x * w[x].y - u.y * w[x].x);
#pragma unroll
          for (int r = 0; r < kDispLines; ++r)
            if (l >= r && l <= r + 2 * kKL) R[r][x] = __fadd2_rn(R[r][x], t);
        }
#pragma unroll
        for (int x = 0; x + 1 < kDispLags; ++x) w[x] = w[x + 1];
        w[kDispLags - 1] = b[min(c0 + d + kDispLags, n1 - 1)];
      }
    }
#pragma unroll
    for (int x = 0; x < kDispLags; ++x) {
      const int lag = l0 + x;
      if (lag > p.lag_max) break;
#pragma unroll
      for (int r = 0; r < kDispLines; ++r) {
        const float eb = eb_s[r * width + static_cast<int>(threadIdx.x) + p.lag_max + lag];
        if (ea[r] <= 0.0f || eb <= 0.0f) continue;
        const float cr = cabsf_(mk(R[r][x].x, R[r][x].y)) / sqrtf(ea[r] * eb);
        if (cr > best[r]) {
          best[r] = cr;
          best_R[r] = R[r][x];
          best_lag[r] = lag;
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kDispLines; ++r) {
    if (i0 + r >= p.n0) continue;
    const long k = static_cast<long>(i0 + r) * n1 + j;
    p.axial[k] = 0.0f;
    p.corr[k] = 0.0f;
    if (!(f_centre[r] <= 0.0f) && !(best[r] < 0.0f))
      disp_store(p, k, best[r], mk(best_R[r].x, best_R[r].y), best_lag[r], f_centre[r]);
  }
}

__global__ void strain_kernel(const float* axial, int n0, int n1, float dz, int half, float* strain) {
  const long k = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (k >= static_cast<long>(n0) * n1) return;
  const int i = static_cast<int>(k / n1), j = static_cast<int>(k - static_cast<long>(i) * n1);
  float sx = 0, sy = 0, sxx = 0, sxy = 0;
  int n = 0;
  for (int d = -half; d <= half; ++d) {
    const int jj = j + d;
    if (jj < 0 || jj >= n1) continue;
    const float x = static_cast<float>(d) * dz;
    const float y = axial[static_cast<long>(i) * n1 + jj];
    sx += x;
    sy += y;
    sxx += x * x;
    sxy += x * y;
    ++n;
  }
  float out = 0.0f;
  if (n >= 2) {
    const float denom = static_cast<float>(n) * sxx - sx * sx;
    if (!(fabsf(denom) < 1e-20f)) out = (static_cast<float>(n) * sxy - sx * sy) / denom;
  }
  strain[k] = out;
}

// Whether the four-line kernel pays over the `interior` columns of n0 lines. Its
// blocks are kDispCols columns x kDispLines lines and form kDispLags lags at a
// time, so what counts is the window terms x lags (terms) over the interior
// pixels, times the shares of the blocks' columns and lines and of the lags that
// are wanted; from two blocks per SM on, less of it. (Time with four lines over
// that with a pixel per thread, this kernel alone: 256 x 1024, 85 terms x 17 lags
// 0.31; 256 x 300, 45 x 9 0.46; 64 x 256, 27 x 9 0.93; 20,000 x 12, 15 x 5, eight
// interior columns 2.9; 5,000 x 30, 9 x 17 1.7; 2,000 x 50, 5 x 25 1.5.) Without
// lines to share (kl = 0, or a single line) a lag of a short window costs its
// set-up: 128 x 512, 3 x 61 1.5, 9 x 25 1.07, 17 x 17 0.8; 256 x 1024, 5 x 17 0.73;
// 1 x 100,000, 5 x 25 1.24, 17 x 17 0.70. Of 3,105 such shapes the rule takes
// 948, fourteen of them at a loss of more than 3% (at most 1.10).
bool disp_lines_pay(const DispArgs& p, int interior) {
  if (p.kl > 2 || p.lag_max > kDispMaxLag || interior <= 0) return false;
  const int kl = p.n0 == 1 ? 0 : p.kl;
  const double blocks = static_cast<double>(ceil_div(p.n0, kDispLines)) * ceil_div(interior, kDispCols);
  const bool many = blocks >= 300;
  if (kl == 0 && ((p.ka < 4 && (!many || p.n0 == 1)) || (p.n0 == 1 && p.lag_max < 4))) return false;
  const double fill = interior / (static_cast<double>(kDispCols) * ceil_div(interior, kDispCols));
  const double lines = p.n0 == 1 ? 1.0 : p.n0 * static_cast<double>(p.n0) / (kDispLines * ceil_div(p.n0, kDispLines));
  const double lags = 2.0 * p.lag_max + 1, passes = kDispLags * std::ceil(lags / kDispLags);
  const double terms = (2.0 * p.ka + 1) * (2.0 * kl + 1) * lags * (lags / passes);
  return fill >= 0.25 && terms * lines * interior * fill >= (kl == 0 ? 1e7 : many ? 3e6 : 5e6);
}

float axial_step(const float* axis1, int n1) {
  float dz = 1e-4f;
  if (n1 > 1 && axis1) dz = std::abs(axis1[1] - axis1[0]);
  return dz;
}

int launch_wall(usx_ctx* ctx, const float* ens, int n, long n_pix, int type, int order, float* out,
                float* power) {
  if (n > kMaxEns) return fail(USX_ERR_UNSUPPORTED, "ensembles longer than 64 frames are not supported");
  WallArgs a;
  a.ens = reinterpret_cast<const float2*>(ens);
  a.out = reinterpret_cast<float2*>(out);
  a.power = power;
  a.n_pix = n_pix;
  a.n = n;
  a.identity = type == USX_WALL_NONE;
  if (!a.identity) {
    const std::vector<float> M = reject_matrix(n, type == USX_WALL_MEAN ? 0 : order);
    std::copy(M.begin(), M.end(), a.M);
  }
  const int threads = kWallThreads;
  const size_t smem = wall_smem(n);
  if (smem > 48 * 1024)
    if (int rc_ = smem_limit(reinterpret_cast<const void*>(wall_kernel), static_cast<size_t>(static_cast<int>(smem)))) return rc_;
  prof_begin(ctx, "wall_kernel");
  wall_kernel<<<ceil_div(n_pix, threads), threads, smem, ctx->stream>>>(a);
  prof_end(ctx);
  USX_CHECK_LAUNCH("wall_kernel");
  return USX_OK;
}

// The flow sums of `count` ensembles of at most max_n frames: four lines per
// thread where the windows span lines (kl of 1 or 2) and the blocks are full of
// work: kFlowCols depths each, so that the depths must fill most of them (fill;
// 130 of 256: 1.0 to 1.6 times the time of a pixel per thread at 9 depths a
// window; 200 of 256: equal), enough of them for the SMs, and enough window terms to
// pay for the staging, which a short window does not. Time with four lines over
// that with a pixel per thread (this kernel alone):
//   kl = 1: 256 x 512, 8 to 64 frames, 3 depths a window 1.07 to 1.37, 7 depths
//     0.87 to 1.05, 9 depths 0.79 to 0.96, 13 depths 0.74 to 0.88; 180 x 380 (135
//     blocks), 13 depths 0.76 to 1.22; 640 x 200, 9 depths 1.00 to 1.12;
//   kl = 2: 256 x 512, 5 depths 0.73 to 0.96; 60 x 700 (90 blocks), 9 depths, 8 /
//     32 / 64 frames 1.07 / 0.84 / 0.67; 128 x 330, 32 frames, 9 depths 0.83;
//     400 x 128 (one block in depth), 24 / 32 / 64 frames 1.06 / 0.96 / 0.68.
// Of 3,984 such shapes, 3 to 25 depths, the rule takes a thousand, sixteen of them
// at a loss of more than 3% (at most 1.19).
bool flow_lines_pay(const FlowArgs& a, int max_n, int count, size_t smem) {
  if ((a.kl != 1 && a.kl != 2) || a.ka < 1 || max_n < 8 || a.n0 < 2 || smem > 200 * 1024 ||
      ceil_div(a.n0, kFlowLines) > 65535 || (a.n1 <= kFlowCols && (a.kl == 1 || max_n < 32)))
    return false;
  const double cols = ceil_div(a.n1, kFlowCols), fill = a.n1 / (cols * kFlowCols);
  const double blocks = cols * ceil_div(a.n0, kFlowLines) * count;
  const double work = static_cast<double>(a.n0) * a.n1 * count * fill * fill * (2.0 * a.ka + 1);
  return fill >= 0.65 &&
         (a.kl == 1 ? blocks >= 152 && work >= 9e5 : blocks >= 88 && work * std::sqrt(max_n / 16.0) >= 4e5);
}
// ctx: for the profiler, which gets the name of the kernel that runs (null: none).
template <typename Args, typename Pixel, typename Lines>
int launch_flow_sums(usx_ctx* ctx, cudaStream_t st, const FlowArgs& a, const Args& args, int max_n, int count,
                     Pixel pixel, Lines lines1, Lines lines2, const char* pixel_name, const char* lines_name) {
  const size_t smem = sizeof(float2) * static_cast<size_t>(max_n) * (kFlowCols + 2 * static_cast<size_t>(a.ka) + 1);
  const bool lines = flow_lines_pay(a, max_n, count, smem);
  const char* name = lines ? lines_name : pixel_name;
  Lines kern = a.kl == 1 ? lines1 : lines2;
  if (lines && smem > 48 * 1024)
    if (int rc_ = smem_limit(reinterpret_cast<const void*>(kern), smem)) return rc_;
  if (ctx) prof_begin(ctx, name);
  if (lines)
    kern<<<dim3(ceil_div(a.n1, kFlowCols), ceil_div(a.n0, kFlowLines), count), kFlowCols, smem, st>>>(args);
  else
    pixel<<<dim3(ceil_div(static_cast<long>(a.n0) * a.n1, 128), count), 128, 0, st>>>(args);
  if (ctx) prof_end(ctx);
  USX_CHECK_LAUNCH(name);
  return USX_OK;
}
int launch_flow_sums(usx_ctx* ctx, cudaStream_t st, const FlowArgs& a) {
  return launch_flow_sums(ctx, st, a, a, a.n, 1, flow_kernel, flow_lines_kernel<1>, flow_lines_kernel<2>, "flow_kernel",
                          "flow_lines_kernel");
}
int launch_flow_sums(usx_ctx* ctx, const FlowBatchArgs& b, int max_n, int count) {
  return launch_flow_sums(ctx, ctx->stream, b.base, b, max_n, count, flow_batch_kernel, flow_lines_batch_kernel<1>,
                          flow_lines_batch_kernel<2>, "flow_batch_kernel", "flow_lines_batch_kernel");
}

int launch_flow(usx_ctx* ctx, const float* filt, int n, int n0, int n1, float dz, float fdem,
                float prf, float c, const usx_doppler_config& cfg, float* velocity, float* power,
                float* variance, uint8_t* valid, unsigned* pmax_bits) {
  FlowArgs a;
  a.filt = reinterpret_cast<const float2*>(filt);
  a.n = n;
  a.n0 = n0;
  a.n1 = n1;
  a.ka = std::max(0, cfg.kernel_axial);
  a.kl = std::max(0, cfg.kernel_lateral);
  a.loupas = cfg.loupas;
  a.dz = dz;
  a.fdem = fdem;
  a.prf = prf;
  a.c = c;
  a.coh_thr = cfg.coherence_threshold;
  a.velocity = velocity;
  a.power = power;
  a.variance = variance;
  a.valid = valid;
  a.pmax_bits = pmax_bits;
  const long n_pix = static_cast<long>(n0) * n1;
  USX_CUDA(cudaMemsetAsync(pmax_bits, 0, sizeof(unsigned), ctx->stream));
  if (int rc = launch_flow_sums(ctx, ctx->stream, a)) return rc;
  const float ratio = std::pow(10.0f, cfg.power_threshold_db / 10.0f);
  prof_begin(ctx, "power_gate_kernel");
  power_gate_kernel<<<ceil_div(n_pix, 256), 256, 0, ctx->stream>>>(power, valid, n_pix, ratio, pmax_bits);
  prof_end(ctx);
  USX_CHECK_LAUNCH("power_gate_kernel");
  return USX_OK;
}

}  // namespace

// ------------------------------------------------------------------------
// Colour flow without allocation (usx_cu_color_flow_noalloc).
//
// For callers that must not allocate device memory once they are running: a
// scanner's real-time loop with a fixed memory budget, or code that hands this
// library a stream but owns the device's allocator. Its working
// memory, the wall-filtered ensemble and the frame's maximum power, is this
// fixed array, reserved on every device that loads the library for as long
// as the process lives: kNoAllocSamples complex samples (8 MiB) plus one
// word. Host code must not pass the array's name to a kernel: on the host it
// only stands in for the symbol, so its device address is looked up once per
// device with cudaGetSymbolAddress.
namespace {

constexpr long kNoAllocSamples = 1L << 20;
static __device__ __align__(256) float2 g_noalloc_scratch[kNoAllocSamples + 32];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
float2* g_noalloc_addr[kNoAllocMaxDevices] = {};

// Device address of the scratch on the current device, looked up on the
// first call for that device.
int noalloc_scratch(float2** out) {
  int dev = 0;
  USX_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices)
    return fail(USX_ERR_UNSUPPORTED, "usx_cu_color_flow_noalloc: device index above 63");
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
    g_noalloc_addr[dev] = static_cast<float2*>(p);
  }
  *out = g_noalloc_addr[dev];
  return USX_OK;
}

}  // namespace
}  // namespace usxcu

using namespace usxcu;

extern "C" {

int usx_cu_wall_filter(usx_ctx* ctx, const float* ens, int n_frames, int64_t n_pix, int type,
                       int order, float* out) {
  if (!ctx || !ens || !out) return fail(USX_ERR_INVALID, "usx_cu_wall_filter: null argument");
  if (n_frames <= 0 || n_pix <= 0) return USX_OK;
  return launch_wall(ctx, ens, n_frames, n_pix, type, order, out, nullptr);
}

int usx_cu_power_doppler(usx_ctx* ctx, const float* ens, int n_frames, int64_t n_pix, int type,
                         int order, float* power) {
  if (!ctx || !ens || !power) return fail(USX_ERR_INVALID, "usx_cu_power_doppler: null argument");
  if (n_frames <= 0 || n_pix <= 0) return USX_OK;
  return launch_wall(ctx, ens, n_frames, n_pix, type, order, nullptr, power);
}

int usx_cu_color_flow(usx_ctx* ctx, const float* ens, int n_frames, int n0, int n1,
                      const float* axis1_host, float fdem, float prf, float speed_of_sound,
                      const usx_doppler_config* cfg, float* velocity, float* power,
                      float* variance, uint8_t* valid, float* nyquist) {
  if (!ctx || !ens || !cfg || !velocity || !power || !variance || !valid)
    return fail(USX_ERR_INVALID, "usx_cu_color_flow: null argument");
  if (n_frames < 2) return fail(USX_ERR_INVALID, "color_flow: need at least 2 frames in the ensemble");
  if (n0 <= 0 || n1 <= 0) return fail(USX_ERR_INVALID, "color_flow: empty grid");
  const long n_pix = static_cast<long>(n0) * n1;
  void* ws = nullptr;
  if (int rc = scratch(ctx, sizeof(float2) * n_pix * n_frames, &ws)) return rc;
  float* filt = static_cast<float*>(ws);
  if (int rc = launch_wall(ctx, ens, n_frames, n_pix, cfg->wall_filter, cfg->polynomial_order, filt, nullptr))
    return rc;
  if (nyquist) *nyquist = (fdem > 0.0f) ? speed_of_sound * prf / (4.0f * fdem) : 0.0f;
  return launch_flow(ctx, filt, n_frames, n0, n1, axial_step(axis1_host, n1), fdem, prf,
                     speed_of_sound, *cfg, velocity, power, variance, valid,
                     reinterpret_cast<unsigned*>(ctx->d_status + 10));
}

int usx_cu_color_flow_batch(usx_ctx* ctx, const float* ens, int n_ens, const int* n_frames_host,
                            const int64_t* frame_offset_host, int n0, int n1,
                            const float* axis1_host, float fdem, float prf,
                            float speed_of_sound, const usx_doppler_config* cfg, float* velocity,
                            float* power, float* variance, uint8_t* valid) {
  if (!ctx || !ens || !n_frames_host || !frame_offset_host || !cfg)
    return fail(USX_ERR_INVALID, "usx_cu_color_flow_batch: null argument");
  if (n_ens <= 0) return USX_OK;
  if (n_ens > 65535) return fail(USX_ERR_UNSUPPORTED, "usx_cu_color_flow_batch: more than 65535 ensembles");
  if (!velocity || !power || !variance || !valid)
    return fail(USX_ERR_INVALID, "usx_cu_color_flow_batch: null argument");
  if (n0 <= 0 || n1 <= 0) return fail(USX_ERR_INVALID, "color_flow: empty grid");
  const long n_pix = static_cast<long>(n0) * n1;
  int max_frames = 0;
  long total_frames = 0;
  for (int e = 0; e < n_ens; ++e) {
    if (n_frames_host[e] < 2) return fail(USX_ERR_INVALID, "color_flow: need at least 2 frames in the ensemble");
    if (frame_offset_host[e] < 0) return fail(USX_ERR_INVALID, "usx_cu_color_flow_batch: negative frame offset");
    max_frames = std::max(max_frames, n_frames_host[e]);
    total_frames += n_frames_host[e];
  }
  if (max_frames > kMaxEns) return fail(USX_ERR_UNSUPPORTED, "ensembles longer than 64 frames are not supported");
  // Filtered ensembles packed back to back, then one power maximum per ensemble.
  const size_t filt_bytes = sizeof(float2) * static_cast<size_t>(n_pix) * static_cast<size_t>(total_frames);
  void* ws = nullptr;
  if (int rc = scratch(ctx, filt_bytes + sizeof(unsigned) * n_ens + 256, &ws)) return rc;
  float2* filt = static_cast<float2*>(ws);
  unsigned* pmax = reinterpret_cast<unsigned*>(static_cast<char*>(ws) + filt_bytes);
  USX_CUDA(cudaMemsetAsync(pmax, 0, sizeof(unsigned) * n_ens, ctx->stream));

  const int type = cfg->wall_filter;
  const int order = type == USX_WALL_MEAN ? 0 : cfg->polynomial_order;
  const int threads = kWallThreads;
  FlowBatchArgs fb;
  FlowArgs& f = fb.base;
  f.filt = filt;
  f.n0 = n0;
  f.n1 = n1;
  f.ka = std::max(0, cfg->kernel_axial);
  f.kl = std::max(0, cfg->kernel_lateral);
  f.loupas = cfg->loupas;
  f.dz = axial_step(axis1_host, n1);
  f.fdem = fdem;
  f.prf = prf;
  f.c = speed_of_sound;
  f.coh_thr = cfg->coherence_threshold;
  f.velocity = velocity;
  f.power = power;
  f.variance = variance;
  f.valid = valid;
  f.pmax_bits = pmax;

  // Chunks of at most kBatchEns ensembles whose distinct projectors fit the pool.
  long packed = 0;  // first filtered frame of the next ensemble
  int e0 = 0;
  while (e0 < n_ens) {
    WallBatchArgs w;
    w.ens = reinterpret_cast<const float2*>(ens);
    w.out = filt;
    w.n_pix = n_pix;
    w.identity = type == USX_WALL_NONE;
    int pool = 0, count = 0, chunk_max = 0, n_have = 0;
    int have_n[kBatchEns], have_off[kBatchEns];
    for (int e = e0; e < n_ens && count < kBatchEns; ++e) {
      const int n = n_frames_host[e];
      int off = 0;
      if (!w.identity) {
        off = -1;
        for (int q = 0; q < n_have; ++q)
          if (have_n[q] == n) off = have_off[q];
        if (off < 0) {
          if (pool + n * n > kBatchPool) break;  // 64 x 64 alone always fits
          const std::vector<float> M = reject_matrix(n, order);
          std::copy(M.begin(), M.end(), w.M + pool);
          off = pool;
          have_n[n_have] = n;
          have_off[n_have++] = pool;
          pool += n * n;
        }
      }
      w.n[count] = n;
      w.m_off[count] = off;
      w.in_off[count] = frame_offset_host[e];
      w.out_off[count] = packed;
      fb.n[count] = n;
      fb.ens[count] = e;
      fb.f_off[count] = packed;
      packed += n;
      chunk_max = std::max(chunk_max, n);
      ++count;
    }
    const size_t smem = wall_smem(chunk_max);
    if (smem > 48 * 1024)
      if (int rc_ = smem_limit(reinterpret_cast<const void*>(wall_batch_kernel), smem)) return rc_;
    prof_begin(ctx, "wall_batch_kernel");
    wall_batch_kernel<<<dim3(ceil_div(n_pix, threads), count), threads, smem, ctx->stream>>>(w);
    prof_end(ctx);
    USX_CHECK_LAUNCH("wall_batch_kernel");
    if (int rc = launch_flow_sums(ctx, fb, chunk_max, count)) return rc;
    e0 += count;
  }
  const float ratio = std::pow(10.0f, cfg->power_threshold_db / 10.0f);
  prof_begin(ctx, "power_gate_batch_kernel");
  power_gate_batch_kernel<<<dim3(ceil_div(n_pix, 256), n_ens), 256, 0, ctx->stream>>>(power, valid, n_pix, ratio,
                                                                                       pmax);
  prof_end(ctx);
  USX_CHECK_LAUNCH("power_gate_batch_kernel");
  return USX_OK;
}

int usx_cu_color_flow_noalloc(void* stream, const float* ens, int n_frames, int n0, int n1,
                              const float* axis1_host, float fdem, float prf, float speed_of_sound,
                              const usx_doppler_config* cfg, float* velocity, float* power,
                              float* variance, uint8_t* valid, float* nyquist) {
  if (!ens || !cfg || !velocity || !power || !variance || !valid)
    return fail(USX_ERR_INVALID, "usx_cu_color_flow_noalloc: null argument");
  if (n_frames < 2) return fail(USX_ERR_INVALID, "color_flow: need at least 2 frames in the ensemble");
  if (n0 <= 0 || n1 <= 0) return fail(USX_ERR_INVALID, "color_flow: empty grid");
  if (n_frames > kMaxEns) return fail(USX_ERR_UNSUPPORTED, "ensembles longer than 64 frames are not supported");
  const long n_pix = static_cast<long>(n0) * n1;
  if (n_pix * n_frames > kNoAllocSamples)
    return fail(USX_ERR_INVALID,
                "usx_cu_color_flow_noalloc: n_frames * n0 * n1 exceeds the 1048576 complex samples of its "
                "static scratch; use usx_cu_color_flow");
  float2* scratch = nullptr;
  if (int rc = noalloc_scratch(&scratch)) return rc;
  float2* filt = scratch;
  unsigned* pmax_bits = reinterpret_cast<unsigned*>(scratch + kNoAllocSamples);
  cudaStream_t st = static_cast<cudaStream_t>(stream);

  WallArgs w;
  w.ens = reinterpret_cast<const float2*>(ens);
  w.out = filt;
  w.power = nullptr;
  w.n_pix = n_pix;
  w.n = n_frames;
  w.identity = cfg->wall_filter == USX_WALL_NONE;
  if (!w.identity) {
    const std::vector<float> M = reject_matrix(n_frames, cfg->wall_filter == USX_WALL_MEAN ? 0 : cfg->polynomial_order);
    std::copy(M.begin(), M.end(), w.M);
  }
  const int threads = kWallThreads;
  const size_t smem = wall_smem(n_frames);
  if (smem > 48 * 1024)
    if (int rc_ = smem_limit(reinterpret_cast<const void*>(wall_kernel), static_cast<size_t>(static_cast<int>(smem)))) return rc_;
  wall_kernel<<<ceil_div(n_pix, threads), threads, smem, st>>>(w);
  USX_CHECK_LAUNCH("wall_kernel");

  FlowArgs f;
  f.filt = filt;
  f.n = n_frames;
  f.n0 = n0;
  f.n1 = n1;
  f.ka = std::max(0, cfg->kernel_axial);
  f.kl = std::max(0, cfg->kernel_lateral);
  f.loupas = cfg->loupas;
  f.dz = axial_step(axis1_host, n1);
  f.fdem = fdem;
  f.prf = prf;
  f.c = speed_of_sound;
  f.coh_thr = cfg->coherence_threshold;
  f.velocity = velocity;
  f.power = power;
  f.variance = variance;
  f.valid = valid;
  f.pmax_bits = pmax_bits;
  // The scratch keeps the previous call's contents: the running maximum must start at zero.
  USX_CUDA(cudaMemsetAsync(pmax_bits, 0, sizeof(unsigned), st));
  if (int rc = launch_flow_sums(nullptr, st, f)) return rc;
  const float ratio = std::pow(10.0f, cfg->power_threshold_db / 10.0f);
  power_gate_kernel<<<ceil_div(n_pix, 256), 256, 0, st>>>(power, valid, n_pix, ratio, pmax_bits);
  USX_CHECK_LAUNCH("power_gate_kernel");
  if (nyquist) *nyquist = (fdem > 0.0f) ? speed_of_sound * prf / (4.0f * fdem) : 0.0f;
  return USX_OK;
}

int usx_cu_axial_displacement(usx_ctx* ctx, const float* before, const float* after, int n0,
                              int n1, const float* axis1_host, float fdem, float speed_of_sound,
                              int kernel_axial, int kernel_lateral, int max_lag, float* axial,
                              float* correlation) {
  if (!ctx || !before || !after || !axial || !correlation)
    return fail(USX_ERR_INVALID, "usx_cu_axial_displacement: null argument");
  const long n = static_cast<long>(n0) * n1;
  if (n <= 0) return USX_OK;
  DispArgs p;
  p.a = reinterpret_cast<const float2*>(before);
  p.b = reinterpret_cast<const float2*>(after);
  p.n0 = n0;
  p.n1 = n1;
  p.ka = std::max(1, kernel_axial);
  p.kl = std::max(0, kernel_lateral);
  p.lag_max = std::max(0, max_lag);
  p.dz = axial_step(axis1_host, n1);
  p.fdem = fdem;
  p.c = speed_of_sound;
  p.axial = axial;
  p.corr = correlation;
  // Columns whose windows no lag clips in depth (nor the phase slope's next
  // sample) go kDispLines lines to a thread.
  DispLines q;
  q.p = p;
  const long reach = static_cast<long>(p.ka) + std::max(1, p.lag_max);
  q.col_lo = static_cast<int>(std::min<long>(reach, n1));
  q.col_hi = static_cast<int>(std::max<long>(q.col_lo, n1 - reach));
  const bool lines = disp_lines_pay(p, q.col_hi - q.col_lo);
  const char* name = lines ? "displacement_lines_kernel" : "displacement_kernel";
  prof_begin(ctx, name);
  if (lines) {
    q.col_blocks = ceil_div(q.col_hi - q.col_lo, kDispCols);
    q.n_edge = ceil_div(static_cast<long>(n0) * (n1 - (q.col_hi - q.col_lo)), kDispCols);
    const unsigned grid = static_cast<unsigned>(q.n_edge + static_cast<long>(q.col_blocks) * ceil_div(n0, kDispLines));
    const size_t smem = sizeof(float) * kDispLines * (kDispCols + 2 * p.lag_max);
    auto kern = p.kl == 0 ? displacement_lines_kernel<0> : p.kl == 1 ? displacement_lines_kernel<1> : displacement_lines_kernel<2>;
    kern<<<grid, kDispCols, smem, ctx->stream>>>(q);
  } else {
    displacement_kernel<<<ceil_div(n, 128), 128, 0, ctx->stream>>>(p);
  }
  prof_end(ctx);
  USX_CHECK_LAUNCH(name);
  return USX_OK;
}

int usx_cu_axial_strain(usx_ctx* ctx, const float* axial, int n0, int n1,
                        const float* axis1_host, int fit_length, float* strain) {
  if (!ctx || !axial || !strain) return fail(USX_ERR_INVALID, "usx_cu_axial_strain: null argument");
  const long n = static_cast<long>(n0) * n1;
  if (n <= 0) return USX_OK;
  prof_begin(ctx, "strain_kernel");
  strain_kernel<<<ceil_div(n, 256), 256, 0, ctx->stream>>>(axial, n0, n1, axial_step(axis1_host, n1),
                                                           std::max(1, fit_length / 2), strain);
  prof_end(ctx);
  USX_CHECK_LAUNCH("strain_kernel");
  return USX_OK;
}

}  // extern "C"
