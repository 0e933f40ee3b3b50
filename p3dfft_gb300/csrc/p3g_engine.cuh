// CTA-level mixed-radix Stockham FFT over a tile of M lines in shared memory.
//
// A tile holds M independent lines of N complex points.  Element (line, j)
// lives at sm[line * LS + j * JS]; the X passes use line-major tiles
// (LS = N, JS = 1), the strided Y/Z passes point-major tiles (LS = 1, JS = M)
// so that consecutive threads touch consecutive x columns.
//
// Each stage of radix R runs the Stockham autosort step (Govindaraju et al.,
// SC'08): butterfly j of a line reads points j + q N/R (q < R), multiplies them
// by w_{Ns R}^{q (j mod Ns)}, runs a register DFT of size R and writes points
// (j / Ns) Ns R + (j mod Ns) + q Ns.  All reads of a stage finish before any
// write (one barrier), so a stage works in place: every thread keeps all of its
// butterflies of the stage in registers (at most stage_butterflies, for which
// the launch has enough threads).
//
// Radices 2 to 10, 12, 15, 16 and 32 are register codelets.  Any other prime p runs a
// generic direct-DFT stage through a second shared-memory buffer (O(N p) work).
#pragma once

#include <type_traits>

#include "p3g_codelets.cuh"

namespace p3g {

constexpr int kMaxStages = 20;
constexpr int kElemsPerThread = 16;  // E

// The register codelets in the order their stages run: powers of two first,
// so that the sub-transform length before any of them is a power of two.
constexpr int kFamilies[] = {32, 16, 8, 4, 2, 12, 10, 15, 9, 6, 3, 5, 7};
constexpr int kNumFamilies = sizeof(kFamilies) / sizeof(kFamilies[0]);
P3G_HD int family_count(unsigned long long fam, int i) { return (int)(fam >> (4 * i)) & 15; }
// Plans with a 6- or 7-point stage.  The binary32 CTA-wide kernels are compiled
// with and without these codelets: their registers and code cost every other
// plan (24 transforms of powers of two in one launch 1.59 against 1.55 ms, 220^3
// round trips, 20 x 11 points, 1.6 %), and generic 7-point stages are four times
// slower than the codelet.
P3G_HD bool has_c67(unsigned long long fam) { return family_count(fam, 9) + family_count(fam, 12) > 0; }

// Most butterflies of radix r that a thread of E elements runs per stage: as
// many as cover E elements or, where the launch can have the threads for it
// (the grouped kernels), as many as E elements hold.  Two butterflies of 9
// points may take 18 elements of 16, and eleven of 3 points 33 of 32, so that a
// 3 beside powers of two does not ask for more threads (384 x 768 x 384 binary32
// round trip 2.14 -> 1.83 ms; the same for the other radices cost 432-, 540- and
// 375-point lines 5-30 %).
P3G_HD constexpr int stage_butterflies(int E, int r, bool hold) {
  const int h = (E == 16 && r == 9 ? 18 : (E == 32 && r == 3 ? 33 : E)) / r;
  return hold ? (h > 1 ? h : 1) : (E + r - 1) / r;
}

struct StagePlan {
  int n;                   // transform length (1 allowed: no stages)
  int nstages;
  int has_generic;         // a stage with a radix outside kFamilies
  unsigned long long fam;  // stages of each radix family, 4 bits each in the order of kFamilies, then generic
  int radix[kMaxStages];
  int ns[kMaxStages];      // sub-transform length before the stage
  int tw_off[kMaxStages];  // float4 offset of this stage's twiddles [k < ns][q-1 < radix-1]
  int root_off[kMaxStages];  // generic stages: float4 offset of the radix-th roots of unity
};

// Twiddles are stored for the forward sign (exp(-2 pi i ...)) as double-float
// complex float4 (re.hi, im.hi, re.lo, im.lo); the backward direction
// multiplies by the conjugate.
P3G_D cdf load_tw(const float4* __restrict__ tw, int idx) {
  const float4 v = tw[idx];  // shared memory (pipelined passes) or global
  return cdf{pk2(v.x, v.y), pk2(v.z, v.w)};
}

// Division by a runtime divisor d <= 2^15 for dividends x < 2^15 with one
// multiply-high: q = floor(2x * ceil(2^31/d) / 2^32).  Exact because the
// magic's excess over 2^31/d is below 1/d and x < 2^15 (the error term stays
// under 1/d).  Tiles hold at most 2^14 elements, so every index fits.
// Powers of two use a shift (m == 0).
struct FastDiv {
  uint32_t d, m, sh;
  P3G_D explicit FastDiv(uint32_t dd) : d(dd), m(0), sh(0) {
    if ((dd & (dd - 1)) == 0) sh = (uint32_t)(__ffs((int)dd) - 1);
    else m = 0x7FFFFFFFu / dd + 1;  // ceil(2^31 / d)
  }
  P3G_D uint32_t div(uint32_t x) const { return m ? __umulhi(x << 1, m) : (x >> sh); }
  P3G_D void divmod(uint32_t x, uint32_t& q, uint32_t& r) const {
    q = div(x);
    r = x - q * d;
  }
};

// Shared-memory element access through 32-bit shared addresses (ld/st.shared)
// rather than generic pointers.
P3G_D float4 lds(uint32_t a, float4*) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
P3G_D float2 lds(uint32_t a, float2*) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
P3G_D double lds1(uint32_t a, double*) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];\n" : "=d"(v) : "r"(a));
  return v;
}
P3G_D float lds1(uint32_t a, float*) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(v) : "r"(a));
  return v;
}
P3G_D void sts(uint32_t a, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}
P3G_D void sts(uint32_t a, float2 v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};\n" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}

// Line-major tiles may be padded by one element every 2^ps elements (0 = no
// padding) so that the first stage's stride-R writes hit different banks.
// 2^ps divides the plan's first radix and every stage's N/R (and with the
// first radix every later stage's sub-length), so each stage's R inputs and
// the R outputs of every stage but the first stay equally spaced in the padded
// layout; output q of the first stage lies q + (q >> ps) further on.
P3G_D int pad_index(int j, int ps) { return ps ? j + (j >> ps) : j; }

// Hardware barrier with a compile-time id.  Each radix uses its own id: with a
// plain __syncthreads() the compiler merges the identical barriers of all
// switch cases in cta_fft, which keeps every case's registers live at once.
template <int ID>
P3G_D void cta_barrier() {
  asm volatile("bar.sync %0;" ::"n"(ID) : "memory");
}

// The threads that work on one tile: the whole CTA, or one group of a CTA
// whose groups work on tiles of their own (t = index in the group, n = its
// threads, id = its named barrier).
struct CtaThreads {
  static constexpr bool kHold = false;  // stage_butterflies
  P3G_D int tid() const { return (int)threadIdx.x; }
  P3G_D int count() const { return (int)blockDim.x; }
  P3G_D void sync() const { __syncthreads(); }
  template <int ID>
  P3G_D void stage_sync() const {
    cta_barrier<ID>();
  }
};
struct GroupThreads {
  static constexpr bool kHold = true;
  int t = 0, n = 0, id = 0;
  P3G_D int tid() const { return t; }
  P3G_D int count() const { return n; }
  P3G_D void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
  template <int ID>
  P3G_D void stage_sync() const {
    sync();
  }
  // barrier, true if p holds for any thread of the group (not the aligned
  // form: the threads come from wait loops of their own lengths)
  P3G_D bool sync_or(bool p) const {
    uint32_t r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.red.or.pred q, %2, %3, p;\n selp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"((uint32_t)p), "r"(id), "r"(n)
        : "memory");
    return r != 0;
  }
};

template <class P, class TH = CtaThreads>
struct Tile {
  typename P::W* sm;       // M lines x N points
  typename P::W* scratch;  // same size, generic stages only
  int M, log2m, LS, JS;    // point-major tiles (LS = 1) always have JS = M
  int ps = 0;              // line-major padding shift (0: none)
  // kRawR2C first stage only: the binary64 exponent bias of the conversion
  // and the thread's running largest |high word| (null: not tracked)
  int ebias = 0;
  uint32_t* amax = nullptr;
  TH th{};
  unsigned* amax_out = nullptr;  // grouped X tiles: where the first stage leaves each warp's largest
  P3G_D int addr(int line, int j) const { return line * LS + (LS == 1 ? j * JS : pad_index(j, ps)); }
  P3G_D uint32_t saddr(int line, int j) const {
    return (uint32_t)__cvta_generic_to_shared(sm) + (uint32_t)((line * LS + j * JS) * (int)sizeof(typename P::W));
  }
  // butterfly b -> (line, j) over M lines x (N / R) butterflies per line
  P3G_D void decode(int b, int per_line, int& line, int& j) const {
    if (LS == 1) {  // point-major: line fastest
      line = b & (M - 1);
      j = b >> log2m;
    } else {
      line = b / per_line;
      j = b - line * per_line;
    }
  }
  P3G_D void decode(int b, const FastDiv& per_line, int& line, int& j) const {
    if (LS == 1) {
      line = b & (M - 1);
      j = b >> log2m;
    } else {
      uint32_t q, r;
      per_line.divmod((uint32_t)b, q, r);
      line = (int)q;
      j = (int)r;
    }
  }
};

// Tile layouts a kernel can fix at compile time: the strided passes use
// point-major tiles (LS = 1, JS = M), the X passes line-major ones (LS =
// padded N, JS = 1); kAnyLayout reads the layout from the tile.
enum { kAnyLayout = -1, kLineMajor = 0, kPointMajor = 1 };

// One stage of radix R.  FULL: every thread owns exactly MAXB butterflies
// (M N / R == MAXB x threads), so no butterfly needs a guard or a placeholder
// value.  With a known layout the butterfly -> point mapping needs no runtime layout test: point-major, butterfly b reads
// element b (line b mod M, position b / M); line-major, b / (N / R) is the
// line.  In the power-of-two families ns is a power of two (they run first),
// so the twiddle index is a mask.
//
// RAW (first stage of a line-major X tile only) reads the tile's raw line
// pairs instead of the packed complex line, so no separate pass precedes the
// FFT:
//   kRawR2C: real lines 2*line, 2*line+1 ([line][x], one user real each);
//            z[p] = x1[p] + i x2[p].
//   kRawC2R: the pair's half spectra (lines 2*line, 2*line+1 at a stride of
//            rs working-format complexes, nh = N/2+1 modes each); the
//            Hermitian extension z[p] = X1[p] + i X2[p] with
//            X[p] = conj X[N-p] above N/2 and the imaginary parts of the
//            p = 0 and p = N/2 modes ignored (as c2r does).
enum { kRawNone = 0, kRawR2C = 1, kRawC2R = 2 };

template <class P, int DIR, int R, int E, int LAY, bool FULL, int RAW = kRawNone, class TH = CtaThreads>
__device__ __forceinline__ void stage_reg(const Tile<P, TH>& t, int N, int ns, const float4* __restrict__ tw) {
  using C = typename P::C;
  using W = typename P::W;
  constexpr int MAXB = stage_butterflies(E, R, TH::kHold);
  constexpr bool kPow2 = (R & (R - 1)) == 0;
  constexpr uint32_t kW = (uint32_t)sizeof(W);
  const int per_line = N / R;
  const int T = t.th.count();
  const bool pm = LAY == kPointMajor || (LAY == kAnyLayout && t.LS == 1);
  const FastDiv fd_line((uint32_t)(pm ? 1 : per_line)), fd_ns((uint32_t)(kPow2 ? 1 : ns));
  const int nb = t.M * per_line;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(t.sm);
  const int ps = pm ? 0 : t.ps;
  // bytes between inputs q, q+1 and between outputs q, q+1
  const uint32_t jstride = pm ? ((uint32_t)per_line << t.log2m) * kW
                              : (uint32_t)(t.JS * (int)kW) * (uint32_t)pad_index(per_line, ps);
  const uint32_t ostride =
      pm ? ((uint32_t)ns << t.log2m) * kW : (uint32_t)(t.JS * (int)kW) * (uint32_t)pad_index(ns, ps);
  // Non-full stages.  Grouped kernels: a thread past the last butterfly
  // computes that one again and stores nothing (no branches, every element
  // defined).  CTA-wide kernels skip it, with the arrays explicitly
  // initialised: they are written and read under correlated guards the
  // compiler cannot prove, and inside a persistent tile loop an uninitialised
  // element would otherwise be kept live around the loop.  (The batch kernel
  // spills 16 bytes with the guards and 220 without; the strided one the
  // reverse.)
  C v[MAXB][R];
  uint32_t oaddr[MAXB];
  if constexpr (!FULL && !TH::kHold) {
#pragma unroll
    for (int i = 0; i < MAXB; ++i) {
      oaddr[i] = 0;
#pragma unroll
      for (int q = 0; q < R; ++q) v[i][q] = P::zero();
    }
  }
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    const int bi = t.th.tid() + i * T;
    const int b = FULL || !TH::kHold ? bi : min(bi, nb - 1);
    if (FULL || TH::kHold || bi < nb) {
      int line, j;
      uint32_t ia;
      if (pm) {
        line = b & (t.M - 1);
        j = b >> t.log2m;
        ia = sbase + (uint32_t)b * kW;
      } else {
        uint32_t q, r;
        fd_line.divmod((uint32_t)b, q, r);
        line = (int)q;
        j = (int)r;
        ia = sbase + (uint32_t)(t.addr(line, j) * (int)kW);
      }
      if constexpr (RAW == kRawR2C) {
        using UR = typename P::UR;
        constexpr uint32_t kU = (uint32_t)sizeof(UR);
        const uint32_t ra = sbase + (uint32_t)((2 * line * N + j) * (int)kU);
        const uint32_t rstep = (uint32_t)per_line * kU, lstep = (uint32_t)N * kU;
        // one branch per butterfly for the values (or bias) that need the long
        // conversion, out of line: with one per value the inlined long route
        // made the stage's code several times larger
        // the fast route keeps the largest |high word| less that of 2^-74, as an
        // unsigned number: one value outside the route's window makes it too
        // large, and without one it gives the tracked maximum
        uint32_t off = 0;
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const UR x1 = lds1(ra + q * rstep, (UR*)nullptr), x2 = lds1(ra + lstep + q * rstep, (UR*)nullptr);
          v[i][q] = P::make_mid(x1, x2, off);
        }
        if constexpr (P::kF64) {
          uint32_t am = off + kD2dfMidLow;
          if (off >= kD2dfMidSpan || t.ebias != 0) {
            am = 0;
#pragma unroll
            for (int q = 0; q < R; ++q) {
              const UR x1 = lds1(ra + q * rstep, (UR*)nullptr), x2 = lds1(ra + lstep + q * rstep, (UR*)nullptr);
              P::track(am, x1);
              P::track(am, x2);
              v[i][q] = P::from_w(P::make_slow(x1, x2, t.ebias));
            }
          }
          if (t.amax) *t.amax = max(*t.amax, am);
        }
      } else if constexpr (RAW == kRawC2R) {
        const int nh = N / 2 + 1;
        const int rs = sizeof(W) == 8 ? (nh + 1) & ~1 : nh;  // raw line stride (xc2r_raw_stride)
        const uint32_t ra = sbase + (uint32_t)(line * 2 * rs * (int)kW);
        if constexpr (R % 2 == 0) {
          // points j + q N/R lie below N/2 for q < R/2 and mirror above it, at
          // addresses equally spaced in q; only j = 0 meets p = 0 (q = 0) and
          // p = N/2 (q = R/2)
          const uint32_t step = (uint32_t)(per_line * (int)kW), ro = (uint32_t)(rs * (int)kW);
          const uint32_t up = ra + (uint32_t)(j * (int)kW), down = ra + (uint32_t)((N - j) * (int)kW);
#pragma unroll
          for (int q = 0; q < R; ++q) {
            const uint32_t pa = q < R / 2 ? up + q * step : down - q * step;
            C x1 = P::from_w(lds(pa, (W*)nullptr));
            C x2 = P::from_w(lds(pa + ro, (W*)nullptr));
            if ((q == 0 || q == R / 2) && j == 0) {
              x1 = P::make(P::re(x1), P::re(P::zero()));
              x2 = P::make(P::re(x2), P::re(P::zero()));
            }
            if (q >= R / 2) {
              x1 = cconj(x1);
              x2 = cconj(x2);
            }
            v[i][q] = x1 + rot<1>(x2);
          }
        } else {
#pragma unroll
          for (int q = 0; q < R; ++q) {
            const int pt = j + q * per_line;
            const bool mir = 2 * pt > N;
            const int pm = mir ? N - pt : pt;
            C x1 = P::from_w(lds(ra + (uint32_t)(pm * (int)kW), (W*)nullptr));
            C x2 = P::from_w(lds(ra + (uint32_t)((rs + pm) * (int)kW), (W*)nullptr));
            if (pm == 0 || 2 * pm == N) {
              x1 = P::make(P::re(x1), P::re(P::zero()));
              x2 = P::make(P::re(x2), P::re(P::zero()));
            }
            if (mir) {
              x1 = cconj(x1);
              x2 = cconj(x2);
            }
            v[i][q] = x1 + rot<1>(x2);
          }
        }
      } else {
#pragma unroll
        for (int q = 0; q < R; ++q) v[i][q] = P::from_w(lds(ia + q * jstride, (W*)nullptr));
      }
      const int k = kPow2 ? (j & (ns - 1)) : (int)(j - fd_ns.div((uint32_t)j) * (uint32_t)ns);
      if (ns > 1) {
        const float4* twp = tw + k * (R - 1) - 1;
#pragma unroll
        for (int q = 1; q < R; ++q) v[i][q] = cmul<(DIR > 0)>(v[i][q], load_tw(twp, q));
      }
      dft<R, DIR>(v[i]);
      const int jo = (j - k) * R + k;
      oaddr[i] = sbase + (pm ? (uint32_t)(line + (jo << t.log2m)) * kW : (uint32_t)(t.addr(line, jo) * (int)kW));
    }
  }
  if constexpr (RAW == kRawR2C && TH::kHold && P::kF64) {
    const uint32_t w = __reduce_max_sync(0xFFFFFFFFu, *t.amax);
    if ((t.th.tid() & 31) == 0) atomicMax(t.amax_out, w);
  }
  t.th.template stage_sync<(R == 16 ? 1 : (R == 32 ? 6 : R))>();
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    if (FULL || t.th.tid() + i * T < nb) {
      if (LAY != kPointMajor && ns == 1 && ps > 0 && (1 << ps) < R) {
#pragma unroll
        for (int q = 0; q < R; ++q) sts(oaddr[i] + (uint32_t)((q + (q >> ps)) * t.JS) * kW, P::to_w(v[i][q]));
      } else {
#pragma unroll
        for (int q = 0; q < R; ++q) sts(oaddr[i] + q * ostride, P::to_w(v[i][q]));
      }
    }
  }
  t.th.template stage_sync<(R == 16 ? 1 : (R == 32 ? 6 : R))>();
}

// Generic prime radix p: twiddle the inputs into scratch, then each output is
// a direct p-term sum with the p-th roots of unity.
template <class P, int DIR>
__device__ __noinline__ void stage_generic(const Tile<P>& t, int N, int p, int ns, const float4* __restrict__ tw,
                                           const float4* __restrict__ roots) {
  using C = typename P::C;
  const int per_line = N / p;
  const int total = t.M * N;
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    int line, idx;
    t.decode(e, N, line, idx);
    const int q = idx / per_line;
    const int j = idx - q * per_line;
    C v = P::from_w(t.sm[t.addr(line, idx)]);
    const int k = j % ns;
    if (q > 0 && ns > 1) v = cmul<(DIR > 0)>(v, load_tw(tw, k * (p - 1) + q - 1));
    t.scratch[t.addr(line, idx)] = P::to_w(v);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    int line, idx;
    t.decode(e, N, line, idx);
    const int kout = idx / per_line;  // output index within the butterfly
    const int j = idx - kout * per_line;
    C acc = P::from_w(t.scratch[t.addr(line, j)]);
    int m = 0;
    for (int q = 1; q < p; ++q) {
      m += kout;
      if (m >= p) m -= p;
      const C x = P::from_w(t.scratch[t.addr(line, j + q * per_line)]);
      acc = acc + (m == 0 ? x : cmul<(DIR > 0)>(x, load_tw(roots, m)));
    }
    const int k = j % ns;
    t.sm[t.addr(line, (j - k) * p + k + kout * ns)] = P::to_w(acc);
  }
  __syncthreads();
}

// Stage s of radix R reads its twiddles at tw_off(s) and has sub-transform
// length ns(s) = product of the radices before it; both follow from the
// family counts, so they are carried in registers instead of being loaded
// per stage (stage 0 owns one placeholder twiddle, see build_stages).
template <class P, int DIR, int R, int E, int LAY, bool FULL, int RAW, class TH>
__device__ __forceinline__ void run_family(const Tile<P, TH>& t, const float4* __restrict__ tw, int N, int cnt, int& ns,
                                           int& off) {
  // the CTA-wide kernels run plans of every kind and take the unguarded form
  // stage by stage; the grouped kernels are compiled for one of them
  const bool full = FULL || (!TH::kHold && t.M * (N / R) == stage_butterflies(E, R, TH::kHold) * t.th.count());
#pragma unroll 1
  for (int c = 0; c < cnt; ++c) {
    if (RAW != kRawNone && ns == 1) {  // the plan's first stage reads the raw line pairs
      if (full) stage_reg<P, DIR, R, E, LAY, true, RAW>(t, N, ns, tw + off);
      else stage_reg<P, DIR, R, E, LAY, false, RAW>(t, N, ns, tw + off);
    } else if (full) {
      stage_reg<P, DIR, R, E, LAY, true>(t, N, ns, tw + off);
    } else {
      stage_reg<P, DIR, R, E, LAY, false>(t, N, ns, tw + off);
    }
    off += ns > 1 ? ns * (R - 1) : 1;
    ns *= R;
  }
}

// Runs all stages of the plan on the tile (sm must be filled and
// synchronised).  MAXR is the largest radix compiled in (the large codelets
// need many registers, so only kernels that may use them carry them; the
// plans they run never exceed MAXR).  Each family runs in its own loop: a
// single loop with a switch over the radix makes the register allocator keep
// the live ranges of every codelet at once and spill.  FULL: a plan of
// power-of-two radices whose stages all fill every thread; only those
// families are compiled, without guards.
// C67: the 6- and 7-point codelets are compiled in.
// The first stage's twiddles start at tw[off].  E = elements each thread holds
// per stage.  LAY: the tile layout when the caller knows it (kPointMajor, kLineMajor).  RAW: the
// tile still holds the raw line pairs of an X r2c or c2r tile (kRawR2C,
// kRawC2R; plans without generic stages only), read by the first stage.
template <class P, int DIR, int E, int LAY, int RAW, int MAXR, bool FULL, bool C67, class TH>
__device__ __forceinline__ void run_families(const Tile<P, TH>& t, const float4* __restrict__ tw, int N,
                                             unsigned long long fam, int off) {
  int ns = 1;
  if constexpr (MAXR >= 32) run_family<P, DIR, 32, E, LAY, FULL, RAW>(t, tw, N, family_count(fam, 0), ns, off);
  if constexpr (MAXR >= 16) run_family<P, DIR, 16, E, LAY, FULL, RAW>(t, tw, N, family_count(fam, 1), ns, off);
  run_family<P, DIR, 8, E, LAY, FULL, RAW>(t, tw, N, family_count(fam, 2), ns, off);
  run_family<P, DIR, 4, E, LAY, FULL, RAW>(t, tw, N, family_count(fam, 3), ns, off);
  run_family<P, DIR, 2, E, LAY, FULL, RAW>(t, tw, N, family_count(fam, 4), ns, off);
  if constexpr (!FULL) {
    if constexpr (MAXR >= 16 && TH::kHold) {
      run_family<P, DIR, 12, E, LAY, false, RAW>(t, tw, N, family_count(fam, 5), ns, off);
      run_family<P, DIR, 10, E, LAY, false, RAW>(t, tw, N, family_count(fam, 6), ns, off);
      run_family<P, DIR, 15, E, LAY, false, RAW>(t, tw, N, family_count(fam, 7), ns, off);
      run_family<P, DIR, 9, E, LAY, false, RAW>(t, tw, N, family_count(fam, 8), ns, off);
    }
    if constexpr (C67) run_family<P, DIR, 6, E, LAY, false, RAW>(t, tw, N, family_count(fam, 9), ns, off);
    run_family<P, DIR, 3, E, LAY, false, RAW>(t, tw, N, family_count(fam, 10), ns, off);
    run_family<P, DIR, 5, E, LAY, false, RAW>(t, tw, N, family_count(fam, 11), ns, off);
    if constexpr (C67) run_family<P, DIR, 7, E, LAY, false, RAW>(t, tw, N, family_count(fam, 12), ns, off);
  }
}

// The CTA-wide form reads the plan from global memory and runs generic primes.
template <class P, bool C67, int DIR, int E = kElemsPerThread, int LAY = kAnyLayout, int RAW = kRawNone,
          int MAXR = P::kF64 ? 8 : 16>
__device__ __forceinline__ void cta_fft(const Tile<P>& t, const StagePlan* __restrict__ sp,
                                        const float4* __restrict__ tw) {
  const int N = __ldg(&sp->n);
  const unsigned long long fam = __ldg(&sp->fam);
  run_families<P, DIR, E, LAY, RAW, MAXR, false, C67>(t, tw, N, fam, __ldg(&sp->tw_off[0]));
  if (__ldg(&sp->has_generic)) {
    int sg = 0;
    for (int i = 0; i < kNumFamilies; ++i) sg += family_count(fam, i);
    const int nst = __ldg(&sp->nstages);
#pragma unroll 1
    for (int s = sg; s < nst; ++s)
      stage_generic<P, DIR>(t, N, __ldg(&sp->radix[s]), __ldg(&sp->ns[s]), tw + __ldg(&sp->tw_off[s]),
                            tw + __ldg(&sp->root_off[s]));
  }
}

}  // namespace p3g
