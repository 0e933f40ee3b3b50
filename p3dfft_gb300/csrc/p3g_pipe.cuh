// Pipelined (persistent, multi-buffered) pass kernels.
//
// One CTA per SM walks a strided list of tiles.  Its threads form groups that
// each transform tiles of their own; the tiles go round a ring of more buffers
// than groups, and the copies into the free ones are in flight (TMA tensor
// tiles, bulk copies or cp.async) while the groups work, so HBM traffic
// overlaps the butterflies.  Each strided tile goes through: a fix-up step in shared
// memory (format conversion of user data, DCT-I/DST-I extension), the
// Stockham stages of p3g_engine.cuh with the pass's twiddles held in shared
// memory for the life of the CTA, and a store step with the pruning map and
// output format conversion fused in, or, for rows stored one to one, TMA
// tensor stores issued by one thread (a buffer is reloaded only after its
// store has read it).
#pragma once

#include <type_traits>

#include "p3g_async.cuh"
#include "p3g_kernels.cuh"

namespace p3g {

// ------------------------------------------------------------ parameters
struct PipeCommon {
  int ntiles;               // tiles over all fields
  int tiles_per_field;
  int tw_base, tw_count;    // this pass's slice of the twiddle table (float4)
  unsigned long long fam;   // the plan's stages (StagePlan::fam), read from the kernel's parameters
  int buf_elems;            // elements (W) per buffer
  int nbuf;                 // tile buffers
  int groups, gthreads;     // thread groups per CTA and threads of each
  int* err;                 // device error flag
};

struct SPipeParams {
  SParams s;
  PipeCommon c;
  int use_tma;              // 1: TMA tensor tiles, 0: cp.async
  int brows, nbox;          // TMA: rows per box, boxes per tile
  int box_bytes;
  int tx_extra;             // test hook: bytes the barrier expects beyond the boxes (0)
  // 1: the transformed tile leaves by TMA stores (one thread, asynchronous)
  // in onbox boxes of obrows rows
  int tma_store;
  int obrows, onbox;
};

struct XPipeParams {
  XParams x;
  PipeCommon c;
  int chunk;                // r2c: cp.async bytes per copy (4, 8 or 16)
  // 1: a group's first thread loads its tile with 1-D bulk copies on the
  // buffer's mbarrier (r2c: the tile's contiguous real lines in one copy;
  // c2r: one copy per line), else every thread issues cp.async
  int bulk;
};

P3G_D unsigned char* align1k(unsigned char* p) {
  return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}

// Strided passes: one CTA per SM, of up to 512 threads (128 registers each).
// A thread holds E elements per stage: 16 on F64 (one 16-point butterfly),
// 32 on F32 (one 32-point butterfly).  FULL kernels run the power-of-two
// lengths whose stages fill every thread (cta_fft): without the guarded
// stages of the other radices they fit their registers without spilling,
// which the others do not quite.
template <class P>
struct TileElems {
  static constexpr int value = P::kF64 ? 16 : 32;
};
constexpr int kMaxGroups = 8;        // named barriers 1..8
constexpr int kMaxTileBuffers = 16;  // ring of tile buffers

// ------------------------------------------------------------ strided Y/Z
template <class P>
struct RingSmem {
  typename P::W* buf0;
  float4* tw;
  uint64_t* mbar;  // one per buffer: its load has landed
  int* issued;     // loads issued into each buffer so far
  int* cta;        // [0] failure flag, [1] exponent bias, [2] largest |high word| seen
};
// Start of a pass kernel: lets the next pass's CTAs launch (they fit beside
// this one's on grids that leave SMs or shared memory free) and, after the
// part that only reads the plan's own tables, waits for the kernel before this
// one in the stream to complete (launch_pass; 32^3 FP64 forward 24.6 us per
// call without, 21.4 us with; 128^3 round trip 120 and 108 us).
P3G_D void pass_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
P3G_D void pass_begin() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class P>
P3G_D RingSmem<P> ring_smem(const PipeCommon& pc) {
  extern __shared__ unsigned char p3g_pipe_smem[];
  RingSmem<P> r;
  r.buf0 = reinterpret_cast<typename P::W*>(align1k(p3g_pipe_smem));
  r.tw = reinterpret_cast<float4*>(r.buf0 + pc.nbuf * pc.buf_elems);
  r.mbar = reinterpret_cast<uint64_t*>(r.tw + pc.tw_count);
  r.issued = reinterpret_cast<int*>(r.mbar + pc.nbuf);
  r.cta = r.issued + pc.nbuf;
  return r;
}

P3G_D void strided_decode(const SPipeParams& q, int tile, int& xt, int& o1, int& o2) {
  o2 = tile / q.c.tiles_per_field;
  const int r = tile - o2 * q.c.tiles_per_field;
  o1 = r / q.s.xtiles;
  xt = r - o1 * q.s.xtiles;
}

// cp.async copies of one strided tile (columns xt*M.., row block o1, field
// o2) into dst, without a commit; the DCT-I/DST-I extension rows are extra
// copies of the same elements (the DST-I negation happens in the fix-up
// step).
template <class P, bool WALK = false, class TH = CtaThreads>
P3G_D void strided_copy(const SParams& s, typename P::W* dst, int xt, int o1, int o2, const TH& th = TH()) {
  using W = typename P::W;
  const int M = s.M, L = s.L;
  const int ph = strided_phase(s, o1, o2);
  const int x0 = xt * M + ph;
  const long long ib0 = (long long)o1 * s.in_o1 + (long long)o2 * s.in_o2;
  const long long ib = ib0 + (long long)x0 * s.in_xs;
  const char* in = static_cast<const char*>(s.in);
  constexpr int esz = (int)sizeof(W);
  auto one = [&](int m, int j) {
    const int src = j >= s.lmap_a1 ? j - s.lmap_d : (j < s.lmap_a0 ? j : -1);
    const int c = x0 + m;
    const bool ok = src >= 0 && c < s.X + ph;
    const int cw = c < s.X ? c : c - s.X;  // the phase-shifted row's last tile wraps to column 0
    const char* g = ok ? in + (ib0 + (long long)cw * s.in_xs + (long long)src * s.in_axis) * esz : in;
    const uint32_t nb = ok ? (uint32_t)esz : 0u;
    int r0 = j, r1 = -1;
    if (s.pre == 2) {
      r0 = j + 1;
      r1 = 2 * (L + 1) - (j + 1);
    } else if (s.pre == 1 && j >= 1 && j <= L - 2) {
      r1 = 2 * (L - 1) - j;
    }
    if constexpr (esz == 16) {
      cp_async16(dst + r0 * M + m, g, nb);
      if (r1 >= 0) cp_async16(dst + r1 * M + m, g, nb);
      if (s.pre == 2 && j == 0) {  // rows 0 and L+1 of the odd extension are zero
        cp_async16(dst + m, in, 0);
        cp_async16(dst + (L + 1) * M + m, in, 0);
      }
    } else {
      cp_async8(dst + r0 * M + m, g, nb);
      if (r1 >= 0) cp_async8(dst + r1 * M + m, g, nb);
      if (s.pre == 2 && j == 0) {
        cp_async8(dst + m, in, 0);
        cp_async8(dst + (L + 1) * M + m, in, 0);
      }
    }
  };
  const int T = th.count(), tid = th.tid();
  if constexpr (esz == 8) {
    // 8-byte elements with adjacent columns: two columns per 16-byte copy when
    // the tile's first column and the row stride keep the pair 16-byte aligned
    // (a tile whose pair would cross the last valid column copies singly)
    const bool pairs = s.in_xs == 1 && M >= 2 && ((ib | s.in_axis) & 1) == 0 &&
                       (reinterpret_cast<uintptr_t>(in) & 15) == 0 && x0 + M <= s.X;
    if (pairs) {
      const int MP = M >> 1, lmp = s.log2m - 1;
      const bool identity =
          s.pre == 0 && ((s.lmap_a0 >= L && s.lmap_a1 >= L) || (s.lmap_d == 0 && s.lmap_a0 >= s.lmap_a1));
      if (WALK && identity && (T & (MP - 1)) == 0) {
        // rows one to one: each thread keeps one column pair and walks its
        // rows with addresses advanced by constant steps (faster inside the
        // batch kernel; slower for the long lines of the pass kernels, whose
        // loads are measured ~10 % slower with it)
        const int m = 2 * (tid & (MP - 1));
        const int j0 = tid >> lmp, js = T >> lmp;
        const char* g = in + (ib + m + (long long)j0 * s.in_axis) * esz;
        const long long gstep = (long long)js * s.in_axis * esz;
        W* d = dst + j0 * M + m;
#pragma unroll 4
        for (int j = j0; j < L; j += js, g += gstep, d += js * M) cp_async16(d, g, 16u);
        return;
      }
      for (int e = tid; e < MP * L; e += T) {
        const int m = 2 * (e & (MP - 1));
        const int j = e >> lmp;
        const int src = j >= s.lmap_a1 ? j - s.lmap_d : (j < s.lmap_a0 ? j : -1);
        const bool ok = src >= 0;
        const char* g = ok ? in + (ib + m + (long long)src * s.in_axis) * esz : in;
        const uint32_t nb = ok ? 16u : 0u;
        int r0 = j, r1 = -1;
        if (s.pre == 2) {
          r0 = j + 1;
          r1 = 2 * (L + 1) - (j + 1);
        } else if (s.pre == 1 && j >= 1 && j <= L - 2) {
          r1 = 2 * (L - 1) - j;
        }
        cp_async16(dst + r0 * M + m, g, nb);
        if (r1 >= 0) cp_async16(dst + r1 * M + m, g, nb);
        if (s.pre == 2 && j == 0) {
          cp_async16(dst + m, in, 0);
          cp_async16(dst + (L + 1) * M + m, in, 0);
        }
      }
      return;
    }
  }
  if (s.in_xs != 1) {  // rows adjacent in memory (STRIDE1 user layout): rows fastest
    const FastDiv div_l(L);
    for (int e = tid; e < M * L; e += T) {
      const int m = (int)div_l.div(e);
      one(m, e - m * L);
    }
  } else if ((T & (M - 1)) == 0) {  // each thread keeps one column m: rows strided by T/M
    const int m = tid & (M - 1);
    for (int j = tid >> s.log2m; j < L; j += T >> s.log2m) one(m, j);
  } else {
    for (int e = tid; e < M * L; e += T) one(e & (M - 1), e >> s.log2m);
  }
}

// A buffer's loads are counted when they are issued.  The wait for use `use`
// of a buffer first waits (bounded) until that load has been issued: groups
// drift, and a group that asked for a parity two phases ahead of the barrier
// would take the phase before last for its own.  Load `use` is issued only
// after tile use - 1 of the buffer was consumed, so from then on the parity
// is unambiguous.
P3G_D void ring_mark_issued(int* issued) {
  __threadfence_block();
  *reinterpret_cast<volatile int*>(issued) = *issued + 1;
}
P3G_D bool ring_wait(uint64_t* bar, const int* issued, int use, int* err) {
  const volatile int* n = issued;
  if (*n <= use) {
    const uint64_t t0 = global_ns();
    uint32_t i = 0;
    while (*n <= use) {
      if (++i >= kMbarSpinLimit || ((i & 15) == 15 && global_ns() - t0 > kMbarWaitNs)) {
        if (err) atomicExch(err, kErrMbarTimeout);
        return false;
      }
      if (i > 16) __nanosleep(32);
    }
  }
  __threadfence_block();
  return mbar_wait_bounded(bar, use & 1, err);
}

// Copies of one tile into buffer b by one group.  TMA: its first thread arms
// the buffer's barrier and issues the boxes.  cp.async: every thread of the
// group copies its share and arrives on the barrier when it has landed.
template <class P>
P3G_D void strided_issue(const SPipeParams& q, const CUtensorMap* tin, int tile, int b, const GroupThreads& th) {
  using W = typename P::W;
  const RingSmem<P> sm = ring_smem<P>(q.c);
  W* dst = sm.buf0 + b * q.c.buf_elems;
  int xt, o1, o2;
  strided_decode(q, tile, xt, o1, o2);
  if (q.use_tma) {
    if (th.t == 0) {
      constexpr int kWords = sizeof(W) / 4;
      ring_mark_issued(&sm.issued[b]);
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&sm.mbar[b], (uint32_t)(q.nbox * q.box_bytes + q.tx_extra));
      for (int i = 0; i < q.nbox; ++i)
        tma_load_4d(dst + i * q.brows * q.s.M, tin, &sm.mbar[b], xt * q.s.M * kWords, i * q.brows, o1, o2);
    }
    return;
  }
  if (th.t == 0) ring_mark_issued(&sm.issued[b]);
  strided_copy<P>(q.s, dst, xt, o1, o2, th);
  cp_async_mbar_arrive(&sm.mbar[b]);
}

// Fix-up of a loaded strided tile, element-wise in place: user format ->
// working format, DST-I negation, DCT-I mirror after a TMA load (tma).
// Ends with a barrier when it changed anything.
template <class P, class TH = CtaThreads>
P3G_D void strided_fix(const SParams& s, bool tma, typename P::W* sm, int k, uint32_t& amax, const TH& th = TH()) {
  using W = typename P::W;
  using C = typename P::C;
  const bool raw_user = s.in_user != 0 && P::kF64;  // binary32 user data is the working format
  if (raw_user || s.pre == 2 || (tma && s.pre == 1)) {
    const int M = s.M, L = s.L;
    const int rows = tma ? L : s.N;
    for (int e = th.tid(); e < M * rows; e += th.count()) {
      const int m = e & (M - 1);
      const int j = e >> s.log2m;
      C v;
      if (raw_user) {
        const typename P::UC u = reinterpret_cast<const typename P::UC*>(sm)[j * M + m];
        P::track(amax, u);
        v = P::from_uc(u, k);
      } else {
        v = P::from_w(sm[j * M + m]);
      }
      if (s.pre == 2 && j >= L + 2) v = cneg(v);
      const W w = P::to_w(v);
      sm[j * M + m] = w;
      if (tma && s.pre == 1 && j >= 1 && j <= L - 2) sm[(2 * (L - 1) - j) * M + m] = w;
    }
    th.sync();
  }
}

// Store of a transformed strided tile with the pruning map and the output
// format (DST-I output rows k+1 times i).
template <class P, class TH = CtaThreads>
P3G_D void strided_store(const SParams& s, const typename P::W* sm, int xt, int o1, int o2, int kb,
                         const TH& th = TH()) {
  using C = typename P::C;
  const int M = s.M;
  const int ph = strided_phase(s, o1, o2);  // the tile's columns as loaded by strided_copy
  const int x0 = xt * M + ph;
  const int xend = s.X + ph;
  const long long obase = (long long)o1 * s.out_o1 + (long long)o2 * s.out_o2;
  auto one = [&](int m, int jo) {
    const int k = jo < s.smap_s0 ? jo : jo + s.smap_d;
    const int c = x0 + m < s.X ? x0 + m : x0 + m - s.X;
    C v;
    if (s.post == 1) v = rot<1>(P::from_w(sm[(k + 1) * M + m]));
    else v = P::from_w(sm[k * M + m]);
    store_elem<P>(s.out, s.out_user, obase + strided_col_out(s, c) + (long long)jo * s.out_axis, v, kb);
  };
  const int T = th.count(), tid = th.tid();
  if (s.tw4) {
    // four-step twiddle w_N^(o1 jo) on every stored element (rows one to one)
    const unsigned long long n4 = (unsigned long long)s.tw4_n;
    for (int e = tid; e < M * s.Lout; e += T) {
      const int m = e & (M - 1), jo = e >> s.log2m;
      if (x0 + m >= xend) continue;
      const int c = x0 + m < s.X ? x0 + m : x0 + m - s.X;
      C v = P::from_w(sm[jo * M + m]);
      const cdf w = load_tw(s.tw4, (int)(((unsigned long long)o1 * (unsigned long long)jo) % n4));
      v = s.tw4_conj ? cmul<true>(v, w) : cmul<false>(v, w);
      store_elem<P>(s.out, s.out_user, obase + strided_col_out(s, c) + (long long)jo * s.out_axis, v, kb);
    }
    return;
  }
  if (s.out_xs == 1 && s.post == 0 && (s.smap_s0 >= s.Lout || s.smap_d == 0) && (T & (M - 1)) == 0) {
    // rows stored one to one (no pruning gap, no DST shift): each thread keeps
    // one column and walks its rows with a shared-memory address and an
    // output pointer advanced by constant steps
    const int m = tid & (M - 1);
    if (x0 + m >= xend) return;
    const int c = x0 + m < s.X ? x0 + m : x0 + m - s.X;
    const int j0 = tid >> s.log2m, js = T >> s.log2m;
    using W = typename P::W;
    uint32_t a = (uint32_t)__cvta_generic_to_shared(sm) + (uint32_t)((j0 * M + m) * (int)sizeof(W));
    const uint32_t astep = (uint32_t)(T * (int)sizeof(W));
    const long long o = obase + strided_col_out(s, c) + (long long)j0 * s.out_axis;
    const long long ostep = (long long)js * s.out_axis;
    if (s.out_user) {
      typename P::UC* d = static_cast<typename P::UC*>(s.out) + o;
#pragma unroll 4
      for (int jo = j0; jo < s.Lout; jo += js, a += astep, d += ostep) *d = P::to_uc(P::from_w(lds(a, (W*)nullptr)), kb);
    } else {
      W* d = static_cast<W*>(s.out) + o;
#pragma unroll 4
      for (int jo = j0; jo < s.Lout; jo += js, a += astep, d += ostep) *d = lds(a, (W*)nullptr);
    }
    return;
  }
  if (s.out_xs != 1) {  // rows adjacent in memory (STRIDE1 user layout): rows fastest
    const FastDiv div_lo(s.Lout);
    for (int e = tid; e < M * s.Lout; e += T) {
      const int m = (int)div_lo.div(e);
      if (x0 + m < xend) one(m, e - m * s.Lout);
    }
  } else if ((T & (M - 1)) == 0) {
    const int m = tid & (M - 1);
    if (x0 + m < xend)
      for (int jo = tid >> s.log2m; jo < s.Lout; jo += T >> s.log2m) one(m, jo);
  } else {
    for (int e = tid; e < M * s.Lout; e += T) {
      const int m = e & (M - 1);
      if (x0 + m < xend) one(m, e >> s.log2m);
    }
  }
}

// The CTA's threads form `groups` groups that each transform whole tiles with
// barriers of their own; the tiles go round the groups, and round a ring of
// nbuf > groups buffers.  While the groups work, the loads of the next tiles
// are in flight in the other buffers: a group that has finished a tile hands
// its buffer back by loading the tile nbuf places further on into it, for
// whichever group's turn that will be.  With one group of all threads every
// warp is in the same phase of a tile, and the FMA pipes idle through its
// shared-memory exchanges and barriers; two or more groups drift apart and
// fill each other's gaps.
template <class P, int DIR, int MODE>
__global__ void __launch_bounds__(tile_max_threads(MODE, P::kF64, false), 1)
    k_strided_pipe(const __grid_constant__ CUtensorMap tin, const __grid_constant__ CUtensorMap tout,
                   const __grid_constant__ SPipeParams pp, const float4* __restrict__ tw_g) {
  pass_launch_next();
  const int nb = pp.c.nbuf, G = pp.c.groups;
  const int step = (int)gridDim.x;
  {
    const RingSmem<P> sm = ring_smem<P>(pp.c);
    for (int i = threadIdx.x; i < pp.c.tw_count; i += blockDim.x) sm.tw[i] = __ldg(tw_g + pp.c.tw_base + i);
    if (threadIdx.x == 0) {
      for (int i = 0; i < nb; ++i) {
        mbar_init(&sm.mbar[i], pp.use_tma ? 1 : pp.c.gthreads);
        sm.issued[i] = 0;
      }
      sm.cta[0] = 0;
      mbar_fence_init();
    }
  }
  pass_begin();
  if (threadIdx.x == 0) {  // held in shared memory, not in registers across the stages
    ring_smem<P>(pp.c).cta[1] = range_k(pp.s.range);
    ring_smem<P>(pp.c).cta[2] = 0;
  }
  __syncthreads();
  const int g = (int)threadIdx.x / pp.c.gthreads;
  const GroupThreads th{(int)threadIdx.x - g * pp.c.gthreads, pp.c.gthreads, 1 + g};
  // one group alone (nb >= 3) loads one tile ahead, into the buffer whose store
  // was issued two tiles ago: its first thread never waits for a store that
  // has just begun
  const bool lag = G == 1 && nb >= 3 && pp.tma_store;
  const int first = lag ? 1 : nb;
  // the first tile of every buffer
  for (int j = 0, tile = blockIdx.x; j < first && tile < pp.c.ntiles; ++j, tile += step)
    if (pp.use_tma ? g == 0 : j % G == g) strided_issue<P>(pp, &tin, tile, j, th);
  int b = g, use = 0;  // this tile's buffer and how often it was used before
  int rtile = -1, rbuf = 0;  // a load to issue once the TMA store has read the buffer
#pragma unroll 1
  for (int tile = blockIdx.x + g * step; tile < pp.c.ntiles; tile += G * step) {
    if (lag && tile + step < pp.c.ntiles && th.t == 0) {
      bulk_wait_read<1>();
      strided_issue<P>(pp, &tin, tile + step, b + 1 == nb ? 0 : b + 1, th);
    }
    const bool ok = ring_wait(&ring_smem<P>(pp.c).mbar[b], &ring_smem<P>(pp.c).issued[b], use, pp.c.err);
    if (th.sync_or(!ok)) {
      if (th.t == 0) ring_smem<P>(pp.c).cta[0] = 1;
      break;
    }
    if (rtile >= 0 && th.t == 0) {
      bulk_wait_read<0>();
      strided_issue<P>(pp, &tin, rtile, rbuf, th);
    }
    {
      const RingSmem<P> sm = ring_smem<P>(pp.c);
      uint32_t amax = 0;
      strided_fix<P>(pp.s, pp.use_tma != 0, sm.buf0 + b * pp.c.buf_elems, sm.cta[1], amax, th);
      if (P::kF64 && pp.s.in_user) {
        amax = __reduce_max_sync(0xFFFFFFFFu, amax);
        if ((th.t & 31) == 0) atomicMax(reinterpret_cast<unsigned*>(&sm.cta[2]), amax);
      }
    }
    {
      const RingSmem<P> sm = ring_smem<P>(pp.c);
      Tile<P, GroupThreads> t{sm.buf0 + b * pp.c.buf_elems, nullptr, pp.s.M, pp.s.log2m, 1, pp.s.M, 0, 0, nullptr, th};
      constexpr int E = MODE == kTileSmall ? TileElems<P>::value / 2 : TileElems<P>::value;
      constexpr bool kFull = MODE == kTileFull || MODE == kTileFullWide;
      run_families<P, DIR, E, kPointMajor, kRawNone, E, kFull, true>(t, sm.tw, pp.s.N, pp.c.fam, 0);
    }
    {
      int xt, o1, o2;
      strided_decode(pp, tile, xt, o1, o2);
      typename P::W* tb = ring_smem<P>(pp.c).buf0 + b * pp.c.buf_elems;
      const int k = ring_smem<P>(pp.c).cta[1];
      rtile = !lag && tile + nb * step < pp.c.ntiles ? tile + nb * step : -1;
      rbuf = b;
      if (pp.tma_store) {
        if constexpr (P::kF64) {
          if (pp.s.out_user) {  // binary64 user format, converted in place (16 bytes each)
            const int ne = pp.s.Lout * pp.s.M;
            for (int e = th.t; e < ne; e += th.n)
              reinterpret_cast<typename P::UC*>(tb)[e] = P::to_uc(P::from_w(tb[e]), k);
          }
        }
        fence_proxy_async_smem();  // this thread's tile writes, before the async-proxy reads
        th.sync();
        if (th.t == 0) {
          constexpr int kWords = sizeof(typename P::W) / 4;
          for (int i = 0; i < pp.onbox; ++i)
            tma_store_4d(&tout, tb + i * pp.obrows * pp.s.M, xt * pp.s.M * kWords, i * pp.obrows, o1, o2);
          bulk_commit_group();
        }
        // A ring without a spare buffer: the next load is this group's own.  The
        // sizing always leaves one (nbuf > groups); without these lines the
        // compiler orders the loop so that 128^3 FP64 round trips take 110 us
        // instead of 104 and 1024^3 FP32 forward 6.36 ms instead of 6.29
        if (nb == G && rtile >= 0) {
          if (th.t == 0) bulk_wait_read<0>();
          th.sync();
          strided_issue<P>(pp, &tin, rtile, rbuf, th);
          rtile = -1;
        }
      } else {
        strided_store<P>(pp.s, tb, xt, o1, o2, k, th);
        th.sync();
        if (rtile >= 0) strided_issue<P>(pp, &tin, rtile, rbuf, th);
        rtile = -1;
      }
    }
    b += G;
    if (b >= nb) {
      b -= nb;
      ++use;
    }
  }
  if (!pp.use_tma) cp_async_wait_all();
  // the tile stores must have completed before the CTA's shared memory goes
  if (pp.tma_store && th.t == 0) bulk_wait_all();
  __syncthreads();
  // a wait timed out: loads may be in flight that no group waits for
  if (threadIdx.x == 0 && pp.use_tma) {
    const RingSmem<P> sm = ring_smem<P>(pp.c);
    if (sm.cta[0]) mbar_drain_bounded(sm.mbar, sm.issued, nb);
  }
  if (P::kF64 && pp.s.in_user && threadIdx.x < 32)
    range_flush(pp.s.range, threadIdx.x == 0 ? (uint32_t)ring_smem<P>(pp.c).cta[2] : 0u);
}

// ---------------------------------------------------------------- X passes
// cp.async of CH bytes (16, 8 or 4)
template <int CH>
P3G_D void cp_async_n(void* d, const void* g, uint32_t nb) {
  if constexpr (CH == 16) cp_async16(d, g, nb);
  else if constexpr (CH == 8) cp_async8(d, g, nb);
  else cp_async4(d, g, nb);
}

// Line by line: each thread copies every blockDim.x-th chunk of each line, with
// the line's addresses formed once (lines at least blockDim.x chunks long).
template <class P, int CH, class TH>
P3G_D void xr2c_copy_lines(const XParams& x, const char* in, char* dst, int p0, const TH& th) {
  using UR = typename P::UR;
  const int lbytes = x.nx * (int)sizeof(UR);
  const int step = th.count() * CH;
  for (int lt = 0; lt < 2 * x.M; ++lt) {
    const int line = 2 * p0 + lt;
    const bool ok = line < x.nlines;
    const char* g = in + (ok ? (long long)line * x.in_line * (long long)sizeof(UR) : 0LL);
    char* d = dst + lt * lbytes;
    const uint32_t nb = ok ? (uint32_t)CH : 0u;
    for (int c = th.tid() * CH; c < lbytes; c += step) cp_async_n<CH>(d + c, g + c, nb);
  }
}

// r2c: real lines 2p, 2p+1 of the tile (first pair p0 of field `field`)
// copied raw ([line][x]) into dst, `chunk` bytes per copy, without a commit.
template <class P, class TH = CtaThreads>
P3G_D void xr2c_copy(const XParams& x, int chunk, typename P::W* dst_w, int p0, int field, const TH& th = TH()) {
  using UR = typename P::UR;
  const int M = x.M, N = x.nx;
  const char* in = reinterpret_cast<const char*>(static_cast<const UR*>(x.in) + field * x.in_field);
  char* dst = reinterpret_cast<char*>(dst_w);
  const int cpl = N * (int)sizeof(UR) / chunk;  // copies per line
  if (cpl >= th.count()) {
    if (chunk == 16) xr2c_copy_lines<P, 16>(x, in, dst, p0, th);
    else if (chunk == 8) xr2c_copy_lines<P, 8>(x, in, dst, p0, th);
    else xr2c_copy_lines<P, 4>(x, in, dst, p0, th);
    return;
  }
  const FastDiv fcpl((uint32_t)cpl);
  for (int e = th.tid(); e < 2 * M * cpl; e += th.count()) {
    const int lt = (int)fcpl.div((uint32_t)e);
    const int c = e - lt * cpl;
    const int line = 2 * p0 + lt;
    const bool ok = line < x.nlines;
    const char* g = ok ? in + (long long)line * x.in_line * (long long)sizeof(UR) + (long long)c * chunk : in;
    char* d = dst + ((long long)lt * N * (long long)sizeof(UR) + (long long)c * chunk);
    const uint32_t nb = ok ? (uint32_t)chunk : 0u;
    if (chunk == 16) cp_async16(d, g, nb);
    else if (chunk == 8) cp_async8(d, g, nb);
    else cp_async4(d, g, nb);
  }
}

// Copies of one r2c tile into buffer b by one group (strided_issue's rules).
template <class P>
P3G_D void xr2c_issue(const XPipeParams& q, int tile, int b, const GroupThreads& th) {
  using UR = typename P::UR;
  const RingSmem<P> sm = ring_smem<P>(q.c);
  typename P::W* dst = sm.buf0 + b * q.c.buf_elems;
  const int field = tile / q.c.tiles_per_field;
  const int p0 = (tile - field * q.c.tiles_per_field) * q.x.M;
  if (q.bulk) {
    if (th.t == 0) {
      const int nl = min(2 * q.x.M, q.x.nlines - 2 * p0);
      const uint32_t bytes = (uint32_t)(nl * q.x.nx) * (uint32_t)sizeof(UR);
      ring_mark_issued(&sm.issued[b]);
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&sm.mbar[b], bytes);
      bulk_load(dst, static_cast<const UR*>(q.x.in) + field * q.x.in_field + (long long)2 * p0 * q.x.nx, bytes,
                &sm.mbar[b]);
    }
    return;
  }
  if (th.t == 0) ring_mark_issued(&sm.issued[b]);
  xr2c_copy<P>(q.x, q.chunk, dst, p0, field, th);
  cp_async_mbar_arrive(&sm.mbar[b]);
}

// X1[k] = (Z[k] + conj Z[N-k]) / 2, X2[k] = -i (Z[k] - conj Z[N-k]) / 2,
// modes k < nkeep stored to the working layout (USER: the user complex
// format, for the X-only transform).
template <class P, bool USER, class TH>
P3G_D void xr2c_store_t(const XParams& x, const typename P::W* sm, int p0, int field, int kb, const TH& th) {
  using C = typename P::C;
  using O = typename std::conditional<USER, typename P::UC, typename P::W>::type;
  const int N = x.nx, nk = x.nkeep;
  O* out = static_cast<O*>(x.out) + field * x.out_field;
  const FastDiv fnk((uint32_t)nk);
  for (int e = th.tid(); e < x.M * nk; e += th.count()) {
    const int pr = (int)fnk.div((uint32_t)e);
    const int k = e - pr * nk;
    const int line = 2 * (p0 + pr);
    if (line >= x.nlines) continue;
    const C a = P::from_w(sm[pr * x.LS + pad_index(k, x.ps)]);
    const C bb = cconj(P::from_w(sm[pr * x.LS + pad_index(k == 0 ? 0 : N - k, x.ps)]));
    const C r1 = cscale2(a + bb, 0.5f), r2 = cscale2(rot<-1>(a - bb), 0.5f);
    if constexpr (USER) {
      out[(long long)line * x.out_line + k] = P::to_uc(r1, kb);
      if (line + 1 < x.nlines) out[(long long)(line + 1) * x.out_line + k] = P::to_uc(r2, kb);
    } else {
      out[(long long)line * x.out_line + k] = P::to_w(r1);
      if (line + 1 < x.nlines) out[(long long)(line + 1) * x.out_line + k] = P::to_w(r2);
    }
  }
}
// kb: the exponent bias of the user-format output (X-only transform)
template <class P, class TH = CtaThreads>
P3G_D void xr2c_store(const XParams& x, const typename P::W* sm, int p0, int field, int kb, const TH& th = TH()) {
  if (x.out_user) xr2c_store_t<P, true>(x, sm, p0, field, kb, th);
  else xr2c_store_t<P, false>(x, sm, p0, field, kb, th);
}

// c2r: complex lines 2p, 2p+1 of nh = N/2+1 modes copied raw (pair stride
// 2 nh) into dst, modes beyond nkeep as zeros, without a commit.
template <class P, class TH = CtaThreads>
P3G_D void xc2r_copy(const XParams& x, typename P::W* dst, int p0, int field, const TH& th = TH()) {
  const int tid = th.tid(), nthr = th.count();
  using W = typename P::W;
  const int M = x.M, nh = x.nx / 2 + 1;
  const W* in = static_cast<const W*>(x.in) + field * x.in_field;
  if constexpr (sizeof(W) == 8) {
    // two complexes per 16-byte copy: raw stride rs even, line pitch even
    const int rs = xc2r_raw_stride(nh, 8), hp = rs >> 1;
    if ((x.in_line & 1) == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0) {
      if (hp >= nthr) {  // line by line, addresses formed once per line
        for (int lt = 0; lt < 2 * M; ++lt) {
          const int line = 2 * p0 + lt;
          const int keep = line < x.nlines ? x.nkeep : 0;
          const W* g = in + (line < x.nlines ? (long long)line * x.in_line : 0LL);
          W* d = dst + lt * rs;
          for (int k = 2 * tid; k < rs; k += 2 * nthr) {
            const int nv = min(max(keep - k, 0), 2);
            cp_async16(d + k, nv ? g + k : in, (uint32_t)(8 * nv));
          }
        }
        return;
      }
      const FastDiv fhp((uint32_t)hp);
      for (int e = tid; e < 2 * M * hp; e += nthr) {
        const int lt = (int)fhp.div((uint32_t)e);
        const int k = 2 * (e - lt * hp);
        const int line = 2 * p0 + lt;
        const int nv = line < x.nlines ? min(max(x.nkeep - k, 0), 2) : 0;  // valid elements of the pair
        const W* g = nv ? in + (long long)line * x.in_line + k : in;
        cp_async16(dst + lt * rs + k, g, (uint32_t)(8 * nv));
      }
      return;
    }
    const FastDiv fnh((uint32_t)nh);
    for (int e = tid; e < 2 * M * nh; e += nthr) {
      const int lt = (int)fnh.div((uint32_t)e);
      const int k = e - lt * nh;
      const int line = 2 * p0 + lt;
      const bool ok = line < x.nlines && k < x.nkeep;
      const W* g = ok ? in + (long long)line * x.in_line + k : in;
      cp_async8(dst + lt * rs + k, g, ok ? 8u : 0u);
    }
    return;
  }
  if (nh >= nthr) {  // line by line, addresses formed once per line
    for (int lt = 0; lt < 2 * M; ++lt) {
      const int line = 2 * p0 + lt;
      const int keep = line < x.nlines ? x.nkeep : 0;
      const W* g = in + (line < x.nlines ? (long long)line * x.in_line : 0LL);
      W* d = dst + lt * nh;
      for (int k = tid; k < nh; k += nthr) {
        const bool ok = k < keep;
        if constexpr (sizeof(W) == 16) cp_async16(d + k, ok ? g + k : in, ok ? 16u : 0u);
        else cp_async8(d + k, ok ? g + k : in, ok ? 8u : 0u);
      }
    }
    return;
  }
  const FastDiv fnh((uint32_t)nh);
  for (int e = tid; e < 2 * M * nh; e += nthr) {
    const int lt = (int)fnh.div((uint32_t)e);
    const int k = e - lt * nh;
    const int line = 2 * p0 + lt;
    const bool ok = line < x.nlines && k < x.nkeep;
    const W* g = ok ? in + (long long)line * x.in_line + k : in;
    if constexpr (sizeof(W) == 16) cp_async16(dst + lt * nh + k, g, ok ? 16u : 0u);
    else cp_async8(dst + lt * nh + k, g, ok ? 8u : 0u);
  }
}

// Copies of one c2r tile into buffer b by one group: one bulk copy per line
// (the nkeep modes rounded up to 16 bytes; the kernel zeroes the modes beyond),
// or cp.async.
template <class P>
P3G_D void xc2r_issue(const XPipeParams& q, int tile, int b, const GroupThreads& th) {
  using W = typename P::W;
  const RingSmem<P> sm = ring_smem<P>(q.c);
  W* dst = sm.buf0 + b * q.c.buf_elems;
  const int field = tile / q.c.tiles_per_field;
  const int p0 = (tile - field * q.c.tiles_per_field) * q.x.M;
  if (q.bulk) {
    if (th.t == 0) {
      const int rs = xc2r_raw_stride(q.x.nx / 2 + 1, (int)sizeof(W));
      const uint32_t lbytes = ((uint32_t)q.x.nkeep * (uint32_t)sizeof(W) + 15u) & ~15u;
      const int nl = min(2 * q.x.M, q.x.nlines - 2 * p0);
      const W* in = static_cast<const W*>(q.x.in) + field * q.x.in_field;
      ring_mark_issued(&sm.issued[b]);
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&sm.mbar[b], lbytes * (uint32_t)nl);
      for (int lt = 0; lt < nl; ++lt)
        bulk_load(dst + lt * rs, in + (long long)(2 * p0 + lt) * q.x.in_line, lbytes, &sm.mbar[b]);
    }
    return;
  }
  if (th.t == 0) ring_mark_issued(&sm.issued[b]);
  xc2r_copy<P>(q.x, dst, p0, field, th);
  cp_async_mbar_arrive(&sm.mbar[b]);
}

// x1 = Re z, x2 = Im z to the user's real lines (format conversion fused).
// Even N: each thread takes positions n, n+1 of a line pair, reads the two
// complex values once and writes two-element vectors to both lines.
template <class P, class TH = CtaThreads>
P3G_D void xc2r_store(const XParams& x, const typename P::W* sm, int p0, int field, int k, const TH& th = TH()) {
  using W = typename P::W;
  using UR = typename P::UR;
  const int M = x.M, N = x.nx, LS = x.LS, ps = x.ps;
  UR* out = static_cast<UR*>(x.out) + field * x.out_field;
  const bool vec = (N & 1) == 0 && (x.out_line & 1) == 0 &&
                   (reinterpret_cast<uintptr_t>(out) & (2 * sizeof(UR) - 1)) == 0;
  if (vec) {
    const int NH = N >> 1;
    const FastDiv fNH((uint32_t)NH);
    for (int e = th.tid(); e < M * NH; e += th.count()) {
      const int pr = (int)fNH.div((uint32_t)e);
      const int n = 2 * (e - pr * NH);
      const int line = 2 * (p0 + pr);
      if (line >= x.nlines) continue;
      const W a = sm[pr * LS + pad_index(n, ps)];  // n even: n and n+1 never straddle a pad
      const W b = sm[pr * LS + pad_index(n, ps) + 1];
      UR* o = out + (long long)line * x.out_line + n;
      if constexpr (P::kF64) {
        *reinterpret_cast<double2*>(o) = make_double2(P::to_ur(df{a.x, a.z}, k), P::to_ur(df{b.x, b.z}, k));
        if (line + 1 < x.nlines)
          *reinterpret_cast<double2*>(o + x.out_line) =
              make_double2(P::to_ur(df{a.y, a.w}, k), P::to_ur(df{b.y, b.w}, k));
      } else {
        *reinterpret_cast<float2*>(o) = make_float2(a.x, b.x);
        if (line + 1 < x.nlines) *reinterpret_cast<float2*>(o + x.out_line) = make_float2(a.y, b.y);
      }
    }
    return;
  }
  const float* smf = reinterpret_cast<const float*>(sm);
  constexpr int kW = sizeof(W) / sizeof(float);
  const FastDiv fN((uint32_t)N);
  for (int e = th.tid(); e < 2 * M * N; e += th.count()) {
    const int lt = (int)fN.div((uint32_t)e);
    const int n = e - lt * N;
    const int line = 2 * p0 + lt;
    if (line >= x.nlines) continue;
    const int c = lt & 1;
    const float* f = smf + ((lt >> 1) * LS + pad_index(n, ps)) * kW;
    if constexpr (P::kF64) out[(long long)line * x.out_line + n] = P::to_ur(df{f[c], f[2 + c]}, k);
    else out[(long long)line * x.out_line + n] = f[c];
  }
}

// X passes in groups over a ring of buffers, as k_strided_pipe; a tile is M
// line pairs.  Lines are contiguous in memory, so the tiles can be as small as
// two warps' work and eight groups keep the SM's FMA pipes, shared memory and
// stores busy at once.  The first FFT stage reads the raw line pairs (packing
// or Hermitian merge and format conversion fused into it).
template <class P, bool R2C, int MODE>
__global__ void __launch_bounds__(tile_max_threads(MODE, P::kF64, true), 1)
    k_x_pipe(const __grid_constant__ XPipeParams pp, const float4* __restrict__ tw_g) {
  pass_launch_next();
  const int nb = pp.c.nbuf, G = pp.c.groups;
  const int step = (int)gridDim.x;
  {
    const RingSmem<P> sm = ring_smem<P>(pp.c);
    for (int i = threadIdx.x; i < pp.c.tw_count; i += blockDim.x) sm.tw[i] = __ldg(tw_g + pp.c.tw_base + i);
    if (threadIdx.x == 0) {
      for (int i = 0; i < nb; ++i) {
        mbar_init(&sm.mbar[i], pp.bulk ? 1 : pp.c.gthreads);
        sm.issued[i] = 0;
      }
      sm.cta[0] = 0;
      sm.cta[2] = 0;
      mbar_fence_init();
    }
  }
  pass_begin();
  if (threadIdx.x == 0) ring_smem<P>(pp.c).cta[1] = range_k(pp.x.range);
  __syncthreads();
  // the exponent bias and the largest input seen live in shared memory: no
  // register of theirs is held across the stages
  const int g = (int)threadIdx.x / pp.c.gthreads;
  const GroupThreads th{(int)threadIdx.x - g * pp.c.gthreads, pp.c.gthreads, 1 + g};
  auto issue = [&](int tile, int b) {
    if constexpr (R2C) xr2c_issue<P>(pp, tile, b, th);
    else xc2r_issue<P>(pp, tile, b, th);
  };
  for (int j = 0, tile = blockIdx.x; j < nb && tile < pp.c.ntiles; ++j, tile += step)
    if (pp.bulk ? g == 0 : j % G == g) issue(tile, j);
  int b = g, use = 0;  // this tile's buffer and how often it was used before
#pragma unroll 1
  for (int tile = blockIdx.x + g * step; tile < pp.c.ntiles; tile += G * step) {
    const bool ok = ring_wait(&ring_smem<P>(pp.c).mbar[b], &ring_smem<P>(pp.c).issued[b], use, pp.c.err);
    if (th.sync_or(!ok)) {
      if (th.t == 0) ring_smem<P>(pp.c).cta[0] = 1;
      break;
    }
    const RingSmem<P> sm = ring_smem<P>(pp.c);
    typename P::W* tb = sm.buf0 + b * pp.c.buf_elems;
    auto place = [&](int& field, int& p0) {
      field = tile / pp.c.tiles_per_field;
      p0 = (tile - field * pp.c.tiles_per_field) * pp.x.M;
    };
    int field, p0;
    place(field, p0);
    if (pp.bulk && 2 * (p0 + pp.x.M) > pp.x.nlines) {  // the field's last tile: zeros for the lines it lacks
      const int from = pp.x.nlines - 2 * p0, lines = 2 * pp.x.M - from;
      const int words = (R2C ? pp.x.nx * (int)sizeof(typename P::UR)
                             : xc2r_raw_stride(pp.x.nx / 2 + 1, (int)sizeof(typename P::W)) * (int)sizeof(typename P::W)) / 4;
      float* z = reinterpret_cast<float*>(tb) + (long long)from * words;
      for (int e = th.t; e < lines * words; e += th.n) z[e] = 0.0f;
      th.sync();
    }
    if constexpr (!R2C) {
      const int nh = pp.x.nx / 2 + 1, drop = nh - pp.x.nkeep;
      if (pp.bulk && drop > 0) {  // the x modes the pruned spectrum lacks
        const int rs = xc2r_raw_stride(nh, (int)sizeof(typename P::W));
        const FastDiv fd((uint32_t)drop);
        for (int e = th.t; e < 2 * pp.x.M * drop; e += th.n) {
          const int lt = (int)fd.div((uint32_t)e);
          tb[lt * rs + pp.x.nkeep + e - lt * drop] = P::to_w(P::zero());
        }
        th.sync();
      }
    }
    {
      constexpr int E = MODE == kTileSmall ? TileElems<P>::value / 2 : TileElems<P>::value;
      constexpr bool kFull = MODE == kTileFull || MODE == kTileFullWide;
      uint32_t amax = 0;
      Tile<P, GroupThreads> t{tb, nullptr, pp.x.M, pp.x.log2m, pp.x.LS, 1, pp.x.ps, R2C ? sm.cta[1] : 0,
                              R2C ? &amax : nullptr, th, R2C ? reinterpret_cast<unsigned*>(&sm.cta[2]) : nullptr};
      run_families<P, R2C ? -1 : 1, E, kLineMajor, R2C ? kRawR2C : kRawC2R, E, kFull, true>(t, sm.tw, pp.x.nx, pp.c.fam, 0);
    }
    asm volatile("" : "+r"(tile));  // the tile's place again, rather than held across the stages
    place(field, p0);
    const int k = ring_smem<P>(pp.c).cta[1];
    if constexpr (R2C) xr2c_store<P>(pp.x, tb, p0, field, k, th);
    else xc2r_store<P>(pp.x, tb, p0, field, k, th);
    th.sync();
    if (tile + nb * step < pp.c.ntiles) issue(tile + nb * step, b);
    b += G;
    if (b >= nb) {
      b -= nb;
      ++use;
    }
  }
  if (!pp.bulk) cp_async_wait_all();
  __syncthreads();
  // a wait timed out: loads may be in flight that no group waits for
  if (threadIdx.x == 0 && pp.bulk) {
    const RingSmem<P> sm = ring_smem<P>(pp.c);
    if (sm.cta[0]) mbar_drain_bounded(sm.mbar, sm.issued, nb);
  }
  if constexpr (R2C) {
    if (threadIdx.x < 32) range_flush(pp.x.range, threadIdx.x == 0 ? (uint32_t)ring_smem<P>(pp.c).cta[2] : 0u);
  }
}

}  // namespace p3g
