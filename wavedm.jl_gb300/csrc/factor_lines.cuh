// Line passes (y and z axis) on the two-factor transforms of fft_factor.cuh: a
// TMA-fed persistent kernel, and one register tile per CTA.
#pragma once
#include "chain.cuh"
#include "fft_factor.cuh"
#include "passes.cuh"

namespace wdm {
namespace fx {

template <int N>
__host__ __device__ constexpr int line_threads() { return Plan<N>::T * LINES; }

// Registers per thread the line passes are compiled for, by the larger factor
// (the points a thread holds at a time), and the CTAs per SM they leave room for.
template <int N>
__host__ __device__ constexpr int line_ctas() {
  constexpr int R = Plan<N>::RA > Plan<N>::RB ? Plan<N>::RA : Plan<N>::RB;
  constexpr int regs = R > 24 ? 128 : R > 16 ? 104 : R > 12 ? 80 : 64;
  constexpr int m = 65536 / (regs * line_threads<N>());
  return m < 1 ? 1 : m > 16 ? 16 : m;
}

// ----------------------------------------------------------------------------
// k-space operators between the forward and inverse transforms of a fused pass:
// what a line's points share (Line), a table along the line (Entry), and the
// product at one mode.  FORMS: a runtime form is tested once per butterfly.
// ----------------------------------------------------------------------------
struct Drift {
  DriftOp o;
  static constexpr bool FORMS = true;
  struct Line {
    float4 wxy;
    float k2;
  };
  using Entry = float4;  // cz, or kz^2 in the plain form
  __device__ __forceinline__ Line line(int mx, int my) const {
    return o.precise ? Line{o.cxy[(long long)my * o.nxy + mx], 0.f}
                     : Line{make_float4(0.f, 0.f, 0.f, 0.f), o.kx2[mx] + o.ky2[my]};
  }
  __device__ __forceinline__ float4 entry(int pos) const {
    return o.precise ? o.cz[pos] : make_float4(o.kz2[pos], 0.f, 0.f, 0.f);
  }
  // ROT: cz may hold flagged entries (rot != 0)
  template <bool PRECISE, bool ROT>
  __device__ __forceinline__ float2 at(float2 v, const Line& ln, float4 wz) const {
    if constexpr (PRECISE) {
      const bool conj = o.sign < 0.f;
      return twiddle_mul<false>(twiddle_mul<ROT>(v, wz, conj), ln.wxy, conj);
    }
    const float2 sc = sincos_plain(o.sign * (ln.k2 + wz.x) * o.half_dt);
    return cmul(v, make_float2(sc.y * o.scale, -sc.x * o.scale));
  }
};

struct Poisson {
  PoissonOp o;
  static constexpr bool FORMS = false;
  struct Line {
    float k2;
  };
  using Entry = float;  // kz^2
  __device__ __forceinline__ Line line(int mx, int my) const { return Line{o.kx2[mx] + o.ky2[my]}; }
  __device__ __forceinline__ float entry(int pos) const { return o.kz2[pos]; }
  template <bool, bool>
  __device__ __forceinline__ float2 at(float2 v, const Line& ln, float kz) const {
    return o.scaled(v, ln.k2 + kz);
  }
};

struct None {
  static constexpr bool FORMS = false;
  struct Line {};
  using Entry = float;
  __device__ __forceinline__ Line line(int, int) const { return Line{}; }
  __device__ __forceinline__ float entry(int) const { return 0.f; }
  template <bool, bool>
  __device__ __forceinline__ float2 at(float2 v, const Line&, float) const {
    return v;
  }
};

// The operator on the frequencies k1 + RA k2 of one line (v[k2]), the entries
// of its table from tab (staged) or from global memory.
template <int N, bool TAB, class Op>
__device__ __forceinline__ void op_points(const Op& op, float2* v, const typename Op::Line& ln, int k1,
                                          const typename Op::Entry* tab) {
  using P = Plan<N>;
  auto all = [&](auto form) {
    constexpr bool A = decltype(form)::first, B = decltype(form)::second;
#pragma unroll
    for (int k2 = 0; k2 < P::RB; ++k2) {
      const int pos = k1 + P::RA * k2;
      v[k2] = op.template at<A, B>(v[k2], ln, TAB ? tab[pos] : op.entry(pos));
    }
  };
  if constexpr (Op::FORMS) {
    if (!op.o.precise) all(BoolPair<false, false>{});
    else if (op.o.rot) all(BoolPair<true, true>{});
    else all(BoolPair<true, false>{});
  } else {
    all(BoolPair<false, false>{});
  }
}

// MODE: 0 forward, 1 inverse, 2 forward / op / inverse (fused k-space step).
//
// A forward transform runs stage A, then stage B; an inverse runs stage B's
// transform on the frequencies k1 + RA k2 of each k1, then stage A's on the
// elements (k1, n2) of each n2.  The first stage takes its points from load(p)
// and leaves its elements in s (point p at s[p * LINES]; a half-warp touches 16
// neighbouring lines at one point, 128 contiguous bytes: free of bank
// conflicts).  In MODE 1 element (k1, n2) stays where frequency k1 + RA n2 was, so
// that both stages work in place.
template <int N, int MODE, class Load>
__device__ __forceinline__ void line_begin(Load load, float2* s, const float4* tw, int t) {
  using P = Plan<N>;
  if constexpr (MODE == 1) {
#pragma unroll 1
    for (int i = 0; i < P::RA / P::T; ++i) {
      const int k1 = t + P::T * i;
      float2 v[P::RB];
#pragma unroll
      for (int k2 = 0; k2 < P::RB; ++k2) v[k2] = load(k1 + P::RA * k2);
      dftR<P::RB, true>(v);
      factor_twiddle<N, true>(v, tw, k1);
#pragma unroll
      for (int n2 = 0; n2 < P::RB; ++n2) s[(k1 + P::RA * n2) * LINES] = v[n2];
    }
  } else {
    factor_a<N, false>(load, [&](int p, float2 v) { s[p * LINES] = v; }, t);
  }
}

// The rest of the transform after a barrier: from s to base[p * ps] (when ok).
// freed: called once the thread no longer needs s.
template <int N, int MODE, bool TAB, class Op, class Hook>
__device__ __forceinline__ void line_finish(float2* s, float2* base, long long ps, bool ok, const float4* tw,
                                            const Op& op, const typename Op::Line& ln, const typename Op::Entry* tab,
                                            int t, const Hook& freed) {
  using P = Plan<N>;
  auto load = [&](int p) { return s[p * LINES]; };
  auto put = [&](int p, float2 v) {
    if (ok) base[(long long)p * ps] = v;
  };
  if constexpr (MODE == 2) {
    factor_b<N, false>(
        load, tw,
        [&](int k1, float2* v) {
          op_points<N, TAB>(op, v, ln, k1, tab);
          dftR<P::RB, true>(v);
          factor_twiddle<N, true>(v, tw, k1);
#pragma unroll
          for (int n2 = 0; n2 < P::RB; ++n2) s[(P::RB * k1 + n2) * LINES] = v[n2];
        },
        t);
    __syncthreads();
    factor_a<N, true>(load, put, t);
  } else if constexpr (MODE == 1) {
#pragma unroll 1
    for (int i = 0; i < P::RB / P::T; ++i) {
      const int n2 = t + P::T * i;
      float2 v[P::RA];
#pragma unroll
      for (int k1 = 0; k1 < P::RA; ++k1) v[k1] = load(k1 + P::RA * n2);
      dftR<P::RA, true>(v);
#pragma unroll
      for (int n1 = 0; n1 < P::RA; ++n1) put(P::RB * n1 + n2, v[n1]);
    }
  } else {
    factor_b<N, false>(
        load, tw,
        [&](int k1, float2* v) {
#pragma unroll
          for (int k2 = 0; k2 < P::RB; ++k2) put(k1 + P::RA * k2, v[k2]);
        },
        t);
  }
  freed();
}

// One tile of LINES lines loaded straight into registers: lines line0 .. line0 +
// LINES - 1 of batch item b, by threads tid = 0 .. line_threads<N>() - 1 (all of
// which, and any other threads of the CTA, reach the same barriers), with the
// twiddle table already in shared memory at tw and the exchange buffer s (N
// LINES entries).
template <int N, int MODE, class Op>
__device__ __forceinline__ void line_tile(float2* data, const LineGeom& g, const float4* tw, const Op& op,
                                          int line0, int b, float2* s, int tid) {
  const int l = tid % LINES, t = tid / LINES;
  const int line = line0 + l;
  const bool ok = line < g.nlines;
  float2* base = data + b * g.bstride + (ok ? line_base(g, line) : 0);
  const int lc = ok ? line : 0;
  const typename Op::Line ln = op.line(g.x0 + lc % g.nxa, lc / g.nxa);
  line_begin<N, MODE>([&](int p) { return ok ? base[(long long)p * g.pstride] : make_float2(0.f, 0.f); }, s + l, tw, t);
  __syncthreads();
  line_finish<N, MODE, false>(s + l, base, g.pstride, ok, tw, op, ln, nullptr, t, NoHook{});
}

// One tile of LINES lines per CTA (line_tile); the hardware overlaps one
// resident CTA's loads with another's arithmetic.  This is the line pass where
// the array has no tensor-map view, or the autotuner prefers it.
template <int N, int MODE, class Op>
__global__ void __launch_bounds__(line_threads<N>(), line_ctas<N>())
k_line_tile(float2* data, LineGeom g, const float4* __restrict__ twg, Op op) {
  extern __shared__ float2 smem[];
  float4* tw = reinterpret_cast<float4*>(smem);
  load_twiddles(tw, twg, N);
  if (MODE == 1) __syncthreads();  // else visible after the tile's first barrier
  chain_wait<CHAIN_SMALL>();
  line_tile<N, MODE, Op>(data, g, tw, op, blockIdx.x * LINES, blockIdx.y, smem + 2 * N, threadIdx.x);
}

template <int N>
__host__ __device__ constexpr size_t line_tile_smem() {
  return sizeof(float2) * (size_t)(2 * N + N * LINES);
}

// TMA-fed persistent line pass.  A tile is LINES lines that are neighbours
// along x (one row of the box per point), so the box lands in shared memory as
// a dense [N][LINES] array.  With two tile slots per CTA the bulk
// tensor copy of its next tile is in flight while the current one is
// transformed in place in its own slot and stored from registers.
// One thread issues the copies; every wait on a slot's mbarrier is bounded,
// and a CTA that gives up records WDM_DEVERR_TMA_WAIT, drains its copies
// (bounded again) and exits.
//
// Shared memory of a CTA: the tile slots, the twiddle table, two mbarriers and
// (MODE 2) the operator's table along the lines.  CTAs per SM follow from it
// and from the registers; a CTA has two tile slots where that costs no CTA,
// else one (384^3: four CTAs of one slot, z pass 234 us; three CTAs, 243 us).  The
// plain passes of 384 and 512 points have two slots at half the CTAs all the same:
// bound by memory, they gain more from a copy that is always under way (psi y and H y
// passes, forward and inverse, 384^3: 160, 159, 97, 89 -> 158, 156, 93, 86 us; 512 x
// 512 x 256: 179, 188, 111, 115 -> 177, 184, 106, 104; 256^3: 51, 44, 31, 26 either way).
// The drift's table of four words per point is staged where that costs at
// most one CTA in seven (384: one in four, z pass 234 us without it, 243 us with
// it; 24 halos of 96^3: two in fifteen, 90 us without it, 81 us with it).
template <int N>
__host__ __device__ constexpr size_t line_tma_smem_of(int slots, size_t entry) {
  return slots * (size_t)TmaTile<N>::BYTES + sizeof(float4) * N + 2 * sizeof(uint64_t) + entry * N;
}
template <int N>
__host__ __device__ constexpr int line_tma_ctas_of(int slots, size_t entry) {
  const int s = (int)((228u * 1024u) / (line_tma_smem_of<N>(slots, entry) + 1024u));
  return s < 1 ? 1 : s < line_ctas<N>() ? s : line_ctas<N>();
}
template <int N, int MODE>
__host__ __device__ constexpr int line_tma_slots() {
  if (MODE != 2 && N >= 384) return 2;
  return line_tma_ctas_of<N>(2, sizeof(float)) == line_tma_ctas_of<N>(1, sizeof(float)) ? 2 : 1;
}
template <int N, int MODE, class Op>
__host__ __device__ constexpr bool line_tma_staged() {
  return MODE == 2 && (sizeof(typename Op::Entry) == sizeof(float) ||
                       7 * line_tma_ctas_of<N>(line_tma_slots<N, MODE>(), sizeof(typename Op::Entry)) >=
                           6 * line_tma_ctas_of<N>(line_tma_slots<N, MODE>(), sizeof(float)));
}
template <int N, int MODE, class Op>
__host__ __device__ constexpr size_t line_tma_smem() {
  return line_tma_smem_of<N>(line_tma_slots<N, MODE>(), line_tma_staged<N, MODE, Op>() ? sizeof(typename Op::Entry) : 0);
}

// Ask L2 for a full tile's boxes (ltma_issue's coordinates; edge tiles are small).
template <int N>
__device__ __forceinline__ void line_tma_prefetch(const CUtensorMap* map, const LineGeom& g, long long tile, int tx) {
  using TT = TmaTile<N>;
  const long long per_item = (long long)g.rows * tx + g.edge;
  const int b = (int)(tile / per_item);
  const int rem = (int)(tile - (long long)b * per_item);
  if (rem >= g.rows * tx) return;
  const int row = rem / tx, x0 = (rem - row * tx) * LINES;
#pragma unroll
  for (int q = 0; q < TT::NBOX; ++q) {
    if (g.axis == 1) tma_prefetch_4d(map, x0, q * TT::BOXP, row, b);
    else tma_prefetch_4d(map, x0, row, q * TT::BOXP, b);
  }
}

template <int N, int MODE, class Op, bool LATE>
__global__ void __launch_bounds__(line_threads<N>(), (line_tma_ctas_of<N>(line_tma_slots<N, MODE>(), sizeof(float))))
k_line_tma(float2* data, const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap emap,
           LineGeom g, const float4* __restrict__ twg, Op op, int batch) {
  using TT = TmaTile<N>;
  constexpr int SLOTS = line_tma_slots<N, MODE>();
  constexpr bool STAGED = line_tma_staged<N, MODE, Op>();
  extern __shared__ __align__(1024) unsigned char lsm[];
  float2* slots = reinterpret_cast<float2*>(lsm);
  float4* tw = reinterpret_cast<float4*>(lsm + SLOTS * TT::BYTES);
  uint64_t* bar = reinterpret_cast<uint64_t*>(lsm + SLOTS * TT::BYTES + sizeof(float4) * N);
  auto* optab = reinterpret_cast<typename Op::Entry*>(bar + 2);  // N entries (MODE 2)
  const int tid = threadIdx.x;
  const int l = tid % LINES, t = tid / LINES;
  // When the copy of the next tile goes out (LATE, chosen by the launcher).
  // Early: before the wait for the current tile, so that two copies are in
  // flight during the wait, and a barrier closes every tile so that the copy
  // after next may overwrite its slot.  Late: after the current tile's first
  // barrier, by which every thread has finished the other slot's tile, which
  // saves the closing barrier.
  // tiles of 16 columns; when 16 does not divide nxa the last tile of a row
  // reaches past the tensor (zero-filled by the copy, not stored), unless the
  // last column goes to edge tiles
  const int tx = g.edge ? g.nxa / LINES : (g.nxa + LINES - 1) / LINES;
  const long long per_item = (long long)g.rows * tx + g.edge;
  const long long total = per_item * batch;
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_fence_init();
  }
  load_twiddles(tw, twg, N);
  chain_wait<0>();
  if constexpr (STAGED)
    for (int i = tid; i < N; i += blockDim.x) optab[i] = op.entry(i);
  __syncthreads();
  long long tile = blockIdx.x;
  if (tid == 0 && tile < total) ltma_issue<N>(&map, &emap, slots, &bar[0], g, tile, tx);
  unsigned pending = tile < total ? 1u : 0u;  // bit s: slot s has a copy in flight
  for (int it = 0; tile < total; tile += gridDim.x, ++it) {
    const int cur = SLOTS == 2 ? it & 1 : 0;
    const unsigned par = (unsigned)(SLOTS == 2 ? it >> 1 : it) & 1u;  // slot cur's k-th use completes phase k
    const long long nxt = tile + gridDim.x;
    // one slot and few CTAs: the next tile's copy can go out only once this
    // one is done, so a fused pass asks its lines into L2 now (z pass at 512^3
    // 601 -> 558 us; with four CTAs, 384^3, and in the y passes it costs more
    // than it gives: 232 -> 235 us, 160 -> 181 us)
    if (MODE == 2 && SLOTS == 1 && line_tma_ctas_of<N>(1, sizeof(float)) <= 2 && tid == 0 && nxt < total)
      line_tma_prefetch<N>(&map, g, nxt, tx);
    if (SLOTS == 2 && !LATE && nxt < total) {
      if (tid == 0) ltma_issue<N>(&map, &emap, slots + (cur ^ 1) * N * LINES, &bar[cur ^ 1], g, nxt, tx);
      pending |= 1u << (cur ^ 1);
    }
    const int b = (int)(tile / per_item);
    const int rem = (int)(tile - (long long)b * per_item);
    const bool edge = rem >= g.rows * tx;
    const int row = edge ? (LINES / 2) * (rem - g.rows * tx) + (l >> 1) : rem / tx;
    const int x = edge ? g.nxa - 1 + (l & 1) : (rem - row * tx) * LINES + l;
    const bool ok = x < g.nxa;
    const int mx = ok ? x : 0;
    float2* base = data + b * g.bstride + (long long)row * g.outer + mx;
    // what the operator needs of the line is read ahead of the wait for the tile
    const typename Op::Line ln = op.line(g.x0 + mx, row);
    const bool landed = mbar_wait_bounded(&bar[cur], par);
    if constexpr (SLOTS == 2 && LATE) fence_proxy_async_smem();  // this thread is done with the other slot's last tile
    if (!__syncthreads_and(landed)) {
      if (tid == 0 && g.err) atomicOr(g.err, WDM_DEVERR_TMA_WAIT);
      // drain: the slot that timed out and the look-ahead copy, each bounded
      const bool d0 = mbar_wait_bounded(&bar[cur], par);
      const bool d1 = SLOTS == 1 || !((pending >> (cur ^ 1)) & 1u) || mbar_wait_bounded(&bar[cur ^ 1], (unsigned)((it + 1) >> 1) & 1u);
      if (tid == 0 && g.err && !(d0 && d1)) atomicOr(g.err, WDM_DEVERR_TMA_DRAIN);
      return;
    }
    pending &= ~(1u << cur);
    if (SLOTS == 2 && LATE && nxt < total) {
      if (tid == 0) ltma_issue<N>(&map, &emap, slots + (cur ^ 1) * N * LINES, &bar[cur ^ 1], g, nxt, tx);
      pending |= 1u << (cur ^ 1);
    }
    float2* s = slots + cur * N * LINES;
    // one slot: the next tile's copy goes out as soon as every thread has
    // read the tile for the last time
    auto refill = [&]() {
      if constexpr (SLOTS == 1) {
        fence_proxy_async_smem();
        __syncthreads();
        if (nxt < total) {
          if (tid == 0) ltma_issue<N>(&map, &emap, slots, &bar[0], g, nxt, tx);
          pending = 1u;
        }
      }
    };
    float2* sl = s + l;
    line_begin<N, MODE>([&](int p) { return sl[p * LINES]; }, sl, tw, t);
    __syncthreads();
    line_finish<N, MODE, STAGED>(sl, base, g.pstride, ok, tw, op, ln, optab, t, refill);
    if constexpr (SLOTS == 2 && !LATE) {
      // the slot's generic reads and writes are done before the copy of
      // tile + 2 gridDim overwrites it
      fence_proxy_async_smem();
      __syncthreads();
    }
  }
}

}  // namespace fx
}  // namespace wdm
