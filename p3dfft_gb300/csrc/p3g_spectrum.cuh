// Shell-spectrum row processing shared by k_spectrum (p3g_spectrum.cu) and
// the batch kernel (p3g_batch.cu).  See p3g_spectrum.cu for the method.
#pragma once

#include "p3g_kernels.cuh"
#include "../../include/p3dfft_gb300.h"

struct p3g_plan_s;

namespace p3g {

struct SpecParams {
  const void* in;
  double* E;           // nv * (kmax + 1) bins
  long long field;     // element spacing between fields
  int rows, len;       // rows of the fast axis and their length
  int nyc;             // rows decode as (outer, y) with y fastest
  int nx, ny, nz;
  int stride1;         // fast axis is z (1) or x (0)
  int kmax;
  int flags;
  double s2;           // scale^2
};

// ik = floor(sqrt(k2) + 0.5) exactly: the largest m with k2 > m (m - 1).  The
// approximate root is within one of it (sides stay below 32768, so m < 2^16
// and the products fit 32 bits); one step either way corrects it.
P3G_D int shell_index(uint32_t k2) {
  float root;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(root) : "f"(__uint2float_rn(k2)));
  uint32_t m = (uint32_t)(root + 0.5f);
  if (m > 0 && m * (m - 1) >= k2) --m;
  else if (m * (m + 1) < k2) ++m;
  return (int)m;
}

// |frequency| of 0-based index i of an axis of n points (driver_spec.F90:294-298)
P3G_D int fold(int i, int n) { return i + 1 > n / 2 ? n - i : i; }

P3G_D df sq(df a) {
  df r;
  r.hi = fmul_rn(a.hi, a.hi);
  float e = ffma(a.hi, a.hi, -r.hi);
  r.lo = ffma(2.0f * a.hi, a.lo, e);
  return r;
}

template <bool CG>
P3G_D void load_mode(const double2* p, df& re, df& im) {
  const double2 v = gload<CG>(p);
  re = d2df(v.x);
  im = d2df(v.y);
}
template <bool CG>
P3G_D void load_mode(const float2* p, df& re, df& im) {
  const float2 v = gload<CG>(p);
  re = df{v.x, 0.0f};
  im = df{v.y, 0.0f};
}

// Adds the lanes' last sums to their bins.  Where the other wavenumbers are much
// larger than the fast axis's, nearly all lanes end in the same bin and their
// additions to it would follow one another, so neighbours of one bin add up
// theirs first (z rows of 64 modes of 600 x 64 x 64 STRIDE1: 30.8 us without, 20.6
// with).  Out of line: inlined, it slowed the loop over the modes (200 x 180 x
// 150 binary32 41 against 34.6 us).
static __device__ __noinline__ void flush_lanes(double* hist, int kmax, int bin, df acc) {
  const int lane = threadIdx.x & 31;
  const uint32_t le_mask = 0xFFFFFFFFu >> (31 - lane);
  const int prev = __shfl_up_sync(0xFFFFFFFFu, bin, 1);
  const uint32_t heads = __ballot_sync(0xFFFFFFFFu, lane == 0 || prev != bin);
  if (heads != 0xFFFFFFFFu) {
    const int seg = __popc(heads & le_mask);
#pragma unroll 1
    for (int d = 1; d < 32; d <<= 1) {
      const float oh = __shfl_down_sync(0xFFFFFFFFu, acc.hi, d);
      const float ol = __shfl_down_sync(0xFFFFFFFFu, acc.lo, d);
      const int os = __shfl_down_sync(0xFFFFFFFFu, seg, d);
      const bool same = lane + d < 32 && os == seg;
      if (same) acc = dadd(acc, df{oh, ol});
      if (!__any_sync(0xFFFFFFFFu, same)) break;
    }
    if (!((heads >> lane) & 1u)) bin = -1;
  }
  if (bin >= 0 && bin <= kmax) atomicAdd(hist + bin, df2d_any(acc.hi, acc.lo));
}

// Rows r_first, r_first + r_step, ... below r_end of field `field`, one warp
// per row; hist_all holds one histogram of kmax + 1 bins per warp (zeroed by
// the caller).  Each lane takes a run of consecutive modes, whose bins change
// by at most one from mode to mode, adds them up in double-float and adds the
// sum to its warp's histogram when the bin changes; the last sums of all lanes
// go through flush_lanes.  (A segmented reduction over 32 adjacent modes took
// five rounds of three shuffles and a double-float add per mode and as many
// histogram additions, each with two conversions on the binary64 pipe: 256^3
// STRIDE1 spectrum 118 us, 70 us now; with the conversions alone it is 118 again.)
constexpr int kSpecRun = 8;
template <class P, bool CG>
P3G_D void spectrum_rows(const SpecParams& prm, double* hist_all, int r_first, int r_end, int r_step, int field) {
  using UC = typename P::UC;
  const int nbins = prm.kmax + 1;
  const int lane = threadIdx.x & 31;
  double* hist = hist_all + (size_t)(threadIdx.x >> 5) * nbins;
  const UC* in = static_cast<const UC*>(prm.in) + (long long)field * prm.field;
  const bool k2w = (prm.flags & P3G_SPEC_K2) != 0;
  const bool herm = (prm.flags & P3G_SPEC_HERMITIAN) != 0;
  const int sweeps = (prm.len + 32 * kSpecRun - 1) / (32 * kSpecRun);
  const int run = (prm.len + 32 * sweeps - 1) / (32 * sweeps);  // modes per lane and sweep, at most kSpecRun
  for (int r = r_first; r < r_end; r += r_step) {
    const int y = r % prm.nyc;
    const int outer = r / prm.nyc;
    const int ky = fold(y, prm.ny);
    const UC* row = in + (long long)r * prm.len;
    for (int s = 0; s < sweeps; ++s) {
      const int i0 = (s * 32 + lane) * run, i1 = min(i0 + run, prm.len);
      int bin = -1;
      df acc{0.0f, 0.0f};
      auto flush = [&] {
        // modes beyond kmax are dropped (the sample would write past E); the sum
        // is widened with integer instructions, which leaves one binary64 add
        if (bin >= 0 && bin <= prm.kmax) atomicAdd(hist + bin, df2d_any(acc.hi, acc.lo));
      };
#pragma unroll 4
      for (int i = i0; i < i1; ++i) {
        const int kx = prm.stride1 ? outer : i;
        const int kz = fold(prm.stride1 ? i : outer, prm.nz);
        const uint32_t k2 = (uint32_t)kx * kx + (uint32_t)ky * ky + (uint32_t)kz * kz;
        df re, im;
        load_mode<CG>(row + i, re, im);
        df w = dadd(sq(re), sq(im));
        if (k2w) {
          const float khi = __uint2float_rn(k2);
          const float klo = (float)((long long)k2 - (long long)khi);
          w = dmulc(w, khi, klo);
        }
        if (herm && kx > 0 && 2 * kx != prm.nx) w = dscale2(w, 2.0f);
        const int m = shell_index(k2);
        if (m != bin) {
          flush();
          bin = m;
          acc = w;
        } else {
          acc = dadd(acc, w);
        }
      }
      flush_lanes(hist, prm.kmax, bin, acc);
    }
  }
}

// Sums the CTA's per-warp histograms into E (binary64 atomics, scaled by
// scale^2).  Call after a barrier; nwarps = histograms in hist_all.
P3G_D void spectrum_flush(const SpecParams& prm, const double* hist_all, int nwarps, int field) {
  const int nbins = prm.kmax + 1;
  double* E = prm.E + (long long)field * nbins;
  for (int b = threadIdx.x; b < nbins; b += blockDim.x) {
    double s = 0.0;
    for (int k = 0; k < nwarps; ++k) s += hist_all[(size_t)k * nbins + b];
    if (s != 0.0) atomicAdd(E + b, s * prm.s2);
  }
}

constexpr size_t kSpecMaxSmem = 200 * 1024;

// Validates a spectrum request against the plan and fills prm (kmax <= 0
// selects the sample's default).  Defined in p3g_spectrum.cu.
int make_spectrum_params(p3g_plan_s* p, const void* in, double* E, int kmax, double scale, int flags,
                         long long dim_in, SpecParams& prm);

}  // namespace p3g
