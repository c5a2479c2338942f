// Row passes (x axis) on the two-factor transforms of fft_factor.cuh: the kick,
// the density pass, the plain transform and the real transforms.
//
// A warp owns PW = 32 / RB row pairs (A, B) = (2p, 2p + 1) and two buffers of PW
// rows each, E(0) for the pairs' A rows or their packed lines A + iB, E(1) for the
// B rows, with element (k1, n2) of row j at E[j RP + k1 KP + n2].  A pass is up to
// three phases with a warp barrier between:
//   B items   one butterfly (row, k1) per lane and round: the RB elements of the
//             row's stage B, read from or written to global memory at the
//             frequencies k1 + RA k2 (runs of RA neighbours);
//   A lanes   lane (pair, n2) runs stage A of its pair's rows at n2, the points
//             RB n1 + n2 in registers, where all pointwise work happens: the
//             lanes of a pair touch RB neighbours;
//   B items   again, for the transform back.
// Stage A is where the packed potential line leaves its values and where the
// kicked rows' transforms begin, so a potential never leaves its lane, and a row
// goes through shared memory once per transform.  Rows are loaded from global
// memory straight into registers: enough loads are in flight per lane (up to 48)
// and enough warps per SM that nothing is staged ahead.
//
// Bound by the FMA pipe, shared memory and DRAM at about half of each (the
// Stockham row passes: by shared-memory wavefronts, 70-78% of the data pipe).
#pragma once
#include "chain.cuh"
#include "fft_factor.cuh"
#include "xpass_warp.cuh"

namespace wdm {
namespace fx {

// Row pitch RP and k1 pitch KP of a warp's buffers, from a search over pitches
// with the bank count of the three access patterns; most are free of conflicts.
// WARPS: warps per CTA at full size (the launcher takes fewer for small grids);
// KICK and RHO: CTAs per SM the kick and the other passes are compiled for.
// More warps against more registers per lane, measured (kick / density, us):
// 384^3 12 warps of 168 registers 232 / 223, 16 of 128 279 / 318; 256^3 16 of 128
// 68 / 68, 20 of 96 83 / 94; 512^3 8 of 255 603 / 518, 12 of 168 625 / 571; 96
// halos of 64^3 20 of 96 102 / 104, 32 of 64 95 / 113; 24 of 96^3 16 of 128 101 /
// 93, 20 of 96 94 / 90.  65536 rows: of 192 points 12 of 168 64 / 62, 8 of 255 69 / 70,
// 16 of 128 75 / 72; of 128 16 of 128 37 / 31, 12 of 168 41 / 35, 20 of 96 43 / 36; of
// 48 20 of 96 20.5 / 19.1, 28 of 72 20.6 / 20.4; of 32 32 of 64 14.4 / 14.3, 20 of 96
// 15.1 / 14.4, 36 of 56 15.1 / 15.9; of 24 12.9 / 12.3, 20 14.4 / 14.1, 48 14.4 / 16.4;
// of 16, 12 and 8 32 and 20 warps within 3%, more warps slower.
template <int N>
struct Rows;
#define WDM_ROWS(N_, KP_, RP_, WARPS_, KICK_, RHO_)                                      \
  template <>                                                                            \
  struct Rows<N_> {                                                                      \
    static constexpr int N = N_, KP = KP_, RP = RP_, WARPS = WARPS_;                     \
    static constexpr int KICK = KICK_, RHO = RHO_;                                       \
    static constexpr int RA = Plan<N_>::RA, RB = Plan<N_>::RB, PW = 32 / RB;             \
    static constexpr int WORDS = 2 * PW * RP; /* float2 words of a warp's two buffers */ \
    __host__ __device__ static constexpr size_t smem(int warps) {                        \
      return sizeof(float4) * N + sizeof(float2) * (size_t)WORDS * warps;                \
    }                                                                                    \
    static_assert((sizeof(float4) * N_ + 16 * (size_t)(32 / RB) * RP_ * WARPS_ + 1024) * \
                          (KICK_ > RHO_ ? KICK_ : RHO_) <= 228 * 1024, "shared memory"); \
  };
WDM_ROWS(8, 3, 14, 4, 8, 8)
WDM_ROWS(12, 3, 18, 4, 8, 8)
WDM_ROWS(16, 5, 20, 4, 8, 8)
WDM_ROWS(24, 5, 30, 4, 8, 8)
WDM_ROWS(32, 5, 44, 4, 8, 8)
WDM_ROWS(48, 5, 60, 4, 5, 5)
WDM_ROWS(64, 9, 72, 4, 8, 5)
WDM_ROWS(96, 9, 120, 4, 5, 5)
WDM_ROWS(128, 9, 152, 4, 4, 4)
WDM_ROWS(192, 9, 216, 12, 1, 1)
WDM_ROWS(256, 17, 280, 4, 4, 4)
WDM_ROWS(384, 17, 408, 12, 1, 1)
WDM_ROWS(512, 17, 543, 8, 1, 1)
#undef WDM_ROWS

// A warp's place in a pass.
template <int N>
struct Warp {
  using R = Rows<N>;
  const float4* tw;   // twiddle table (shared memory)
  float2* e;          // the warp's buffers
  unsigned pairs;     // row pairs of all batch items
  unsigned ppi;       // row pairs per batch item
  unsigned u, ustride, units;
  int lane;
  int pr, n2;         // A lanes: the lane's pair and its n2

  __device__ __forceinline__ Warp(float2* smem, const float4* __restrict__ twg, const XWork& w) {
    float4* t = reinterpret_cast<float4*>(smem);
    load_twiddles(t, twg, N);
    __syncthreads();
    chain_wait<CHAIN_SMALL_ROWS>();
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5;
    set(t, smem + 2 * N + (size_t)warp * R::WORDS, w, blockIdx.x * warps + warp, gridDim.x * warps);
  }
  __device__ __forceinline__ Warp() {}
  __device__ __forceinline__ void set(const float4* t, float2* buf, const XWork& w, unsigned u0, unsigned stride) {
    tw = t;
    e = buf;
    ppi = (unsigned)w.pairs_per_item;
    pairs = ppi * (unsigned)w.batch;
    u = u0;
    ustride = stride;
    units = (pairs + R::PW - 1) / R::PW;
    lane = threadIdx.x & 31;
    pr = lane / R::RB;
    n2 = lane % R::RB;
  }
  // pair j of the unit: its batch item and first row; false: past the last pair
  __device__ __forceinline__ bool pair(int j, int* b, int* ra) const {
    const unsigned pp = u * R::PW + j;
    const bool ok = pp < pairs;
    const unsigned q = ok ? pp : 0u;
    const unsigned item = q < ppi ? 0u : q / ppi;
    *b = (int)item;
    *ra = 2 * (int)(q - item * ppi);
    return ok;
  }
  // the A lane's element (k1, n2) of its pair's row `half`
  __device__ __forceinline__ float2* at(int half, int k1) const { return e + (half * R::PW + pr) * R::RP + k1 * R::KP + n2; }
  // elements (k1, 0 ..) of row j of 2 PW (the A rows first)
  __device__ __forceinline__ float2* row(int j, int k1) const { return e + j * R::RP + k1 * R::KP; }
};

// B items over ROWS rows of the unit: item(j, k1) for every row j and k1.
template <int N, int ROWS, class Item>
__device__ __forceinline__ void b_items(const Warp<N>& w, Item item) {
  constexpr int RA = Rows<N>::RA, ITEMS = ROWS * RA;
#pragma unroll 1
  for (int i = 0; i < (ITEMS + 31) / 32; ++i) {
    const int q = w.lane + 32 * i;
    if (ITEMS % 32 == 0 || q < ITEMS) item(q / RA, q % RA);
  }
}

// Stage B's transform of a row's frequencies k1 + RA k2 (in v) into its elements
// (k1, n2) at d: the first half of an inverse.
template <int N>
__device__ __forceinline__ void b_inverse(const float4* tw, float2* v, float2* d, int k1) {
  constexpr int RB = Rows<N>::RB;
  dftR<RB, true>(v);
  factor_twiddle<N, true>(v, tw, k1);
#pragma unroll
  for (int n2 = 0; n2 < RB; ++n2) d[n2] = v[n2];
}

// Stage B of a transform: a row's elements (k1, n2) at s into its frequencies
// k1 + RA k2 (in v).
template <int N, bool INV>
__device__ __forceinline__ void b_forward(const float4* tw, float2* v, const float2* s, int k1) {
  constexpr int RB = Rows<N>::RB;
#pragma unroll
  for (int n2 = 0; n2 < RB; ++n2) v[n2] = s[n2];
  factor_twiddle<N, INV>(v, tw, k1);
  dftR<RB, INV>(v);
}

// The frequencies k1 + RA k2 of a packed line A + iB from the half spectra of its
// rows: Z[p] = A[p] + iB[p], Z[N - p] = conj A[p] + i conj B[p].
template <int N>
__device__ __forceinline__ void pack_half(float2* v, const float2* ha, const float2* hb, bool ok, int k1) {
  constexpr int RA = Rows<N>::RA, RB = Rows<N>::RB;
#pragma unroll
  for (int k2 = 0; k2 < RB; ++k2) {
    // the frequency lies below N/2 for k2 < RB/2, above for k2 > RB/2
    const int k = k1 + RA * k2;
    const bool low = k2 < RB / 2 || (k2 == RB / 2 && k1 == 0);
    const int q = low ? k : N - k;
    float2 a = make_float2(0.f, 0.f), c = make_float2(0.f, 0.f);
    if (ok) {
      a = ha[q];
      c = hb[q];
    }
    v[k2] = low ? fma2(swapped(c), make_float2(-1.f, 1.f), a) : fma2(a, make_float2(1.f, -1.f), swapped(c));
  }
}

// The half spectra of a pair's rows at the frequencies of the packed line's
// butterflies k1 (va) and its partner (vb: RA - k1, or RA/2 for k1 = 0, which is
// its own partner as RA/2 is): between them they hold the frequencies k and N -
// k.  put(k, a, b): rows A and B at frequency k.
template <int N, class Put>
__device__ __forceinline__ void split_half(const float2* va, const float2* vb, int k1, Put put) {
  constexpr int RA = Rows<N>::RA, RB = Rows<N>::RB;
  const bool self = k1 == 0;
  const int kb = self ? RA / 2 : RA - k1;
  auto out = [&](int k, float2 z, float2 zn) {  // zn: the packed line at N - k
    put(k, cscale(fma2(zn, make_float2(1.f, -1.f), z), 0.5f),
        cscale(fma2(swapped(z), make_float2(1.f, -1.f), swapped(zn)), 0.5f));
  };
#pragma unroll
  for (int k2 = 0; k2 < RB / 2; ++k2) {
    out(k1 + RA * k2, va[k2], self ? va[(RB - k2) % RB] : vb[RB - 1 - k2]);
    out(kb + RA * k2, vb[k2], self ? vb[RB - 1 - k2] : va[RB - 1 - k2]);
  }
  if (self) out(N / 2, va[RB / 2], va[RB / 2]);
}

// The pairs' packed lines from their half spectra, through stage B into E(0).
template <int N>
__device__ __forceinline__ void packed_in(const Warp<N>& w, const float2* H, long long hpitch,
                                          long long hbstride) {
  using R = Rows<N>;
  b_items<N, R::PW>(w, [&](int j, int k1) {
    int b, ra;
    const bool ok = w.pair(j, &b, &ra);
    const float2* ha = H + b * hbstride + ra * hpitch;
    float2 v[R::RB];
    pack_half<N>(v, ha, ha + hpitch, ok, k1);
    b_inverse<N>(w.tw, v, w.row(j, k1), k1);
  });
}

// The half spectra of the pairs' rows from their packed lines in E(0).
template <int N>
__device__ __forceinline__ void packed_out(const Warp<N>& w, float2* H, long long hpitch,
                                           long long hbstride) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB, ITEMS = R::PW * RA / 2;
#pragma unroll 1
  for (int i = 0; i < (ITEMS + 31) / 32; ++i) {
    const int q = w.lane + 32 * i;
    if (ITEMS % 32 != 0 && q >= ITEMS) break;
    const int j = q / (RA / 2), k1 = q % (RA / 2), kb = k1 ? RA - k1 : RA / 2;
    float2 va[RB], vb[RB];
    b_forward<N, false>(w.tw, va, w.row(j, k1), k1);
    b_forward<N, false>(w.tw, vb, w.row(j, kb), kb);
    int b, ra;
    if (!w.pair(j, &b, &ra)) continue;
    float2* ha = H + b * hbstride + ra * hpitch;
    split_half<N>(va, vb, k1, [&](int k, float2 x, float2 y) {
      ha[k] = x;
      ha[hpitch + k] = y;
    });
  }
}

// ----------------------------------------------------------------------------
// kick: Phi rows from H, psi <- psi exp(-i dt pot), forward x transform (FWD) or not
// ----------------------------------------------------------------------------
// exp(-i dt pot) - 1 of two potentials in the precise form (kick_factor_t): the
// real parts in *ex, the imaginary parts in *ey.
__device__ __forceinline__ void kick_factor_pair(float2 pot, const KickArgs& a, float2* ex, float2* ey) {
  const float2 th = mul2(pot, both(a.dt_hi));
  const float2 te = fma2(pot, both(a.dt_lo), fma2(pot, both(a.dt_hi), make_float2(-th.x, -th.y)));
  const float2 u = mul2(th, both(0.15915494309189535f));
  const float2 n = make_float2(rintf(u.x), rintf(u.y));
  const float2 r = add2(fma2(n, both(-6.28318548202514648f), th), fma2(n, both(1.7484555e-07f), te));
  // the series of sincos_half on both halves
  const float2 h = mul2(r, both(0.5f)), x2 = mul2(h, h);
  float2 ps = fma2(x2, both(1.6059043836821614599e-10f), both(-2.5052108385441718775e-8f));
  ps = fma2(x2, ps, both(2.7557319223985890653e-6f));
  ps = fma2(x2, ps, both(-1.9841269841269841270e-4f));
  ps = fma2(x2, ps, both(8.3333333333333333333e-3f));
  ps = fma2(x2, ps, both(-1.6666666666666666667e-1f));
  const float2 s = fma2(mul2(h, x2), ps, h);
  float2 pc = fma2(x2, both(2.0876756987868098979e-9f), both(-2.7557319223985890653e-7f));
  pc = fma2(x2, pc, both(2.4801587301587301587e-5f));
  pc = fma2(x2, pc, both(-1.3888888888888888889e-3f));
  pc = fma2(x2, pc, both(4.1666666666666666667e-2f));
  pc = fma2(x2, pc, both(-0.5f));
  const float2 c = fma2(x2, pc, both(1.f));
  const float2 m = mul2(s, both(-2.f));
  *ex = mul2(m, s);
  *ey = mul2(m, c);
}

__device__ __forceinline__ float2 kick_precise(float2 v, float ex, float ey) {
  return add2(v, fma2(v, both(ex), mul2(swapped(v), make_float2(-ey, ey))));
}

// The kick of M points x of a row: phi their potentials, pos(m) their positions.
template <int M, class Pos>
__device__ __forceinline__ void kick_row_points(float2* x, float* phi, const float* T6, const KickArgs& a, int y, int z,
                                                const float* vrow, Pos pos) {
  if (a.tidal) {
    // 1/2 x^T T x about the tide's frame (T6[6..8]: cell 0's coordinates, T6[9]: constant)
    const float fy = T6[7] + a.dy * y, fz = T6[8] + a.dz * z;
    const float cyz = 0.5f * T6[1] * fy * fy + T6[5] * fy * fz + 0.5f * T6[2] * fz * fz + T6[9];
    const float lin = T6[3] * fy + T6[4] * fz;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const float fx = T6[6] + a.dx * pos(m);
      phi[m] += fmaf(fx, fmaf(0.5f * T6[0], fx, lin), cyz);
    }
  }
  if (a.kerr != 0.f) {
#pragma unroll
    for (int m = 0; m < M; ++m) phi[m] = fmaf(a.kerr, fmaf(x[m].x, x[m].x, x[m].y * x[m].y), phi[m]);
  }
  if (vrow) {
#pragma unroll
    for (int m = 0; m < M; ++m) phi[m] += vrow[pos(m)];
  }
  if (a.precise) {
#pragma unroll
    for (int m = 0; m < M; m += 2) {
      float2 ex, ey;
      kick_factor_pair(make_float2(phi[m], phi[m + 1]), a, &ex, &ey);
      x[m] = kick_precise(x[m], ex.x, ey.x);
      x[m + 1] = kick_precise(x[m + 1], ex.y, ey.y);
    }
  } else {
#pragma unroll
    for (int m = 0; m < M; ++m) x[m] = kick_by_t<false>(x[m], kick_factor_t<false>(phi[m], a));
  }
}

// The points RB n1 + n2 of a row (row: its point n2).
template <int N>
__device__ __forceinline__ void load_points(float2* x, const float2* row, bool ok) {
#pragma unroll
  for (int n1 = 0; n1 < Rows<N>::RA; ++n1) x[n1] = ok ? row[Rows<N>::RB * n1] : make_float2(0.f, 0.f);
}

// The kick of one pair by an A lane: the packed potential line's elements (k1,
// n2) at (0, k1), x: row A's points of psi.  FWD: the kicked rows' elements to
// at(half, k1); else the kicked rows to psi.  base: the offset of row A's point
// n2 in psi_in and psi.
template <int N, bool FWD, class At>
__device__ __forceinline__ void kick_lane(At at, float2* x, const float2* psi_in, float2* psi, long long base,
                                          const RowGeom& rg, int b, int ra, bool ok, int n2, const float* T6,
                                          const KickArgs& a) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB;
  float2 z[RA];  // (Phi of row A, Phi of row B)
#pragma unroll
  for (int k1 = 0; k1 < RA; ++k1) z[k1] = *at(0, k1);
  dftR<RA, true>(z);
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    const int r = ra + half;
    float phi[RA];
#pragma unroll
    for (int n1 = 0; n1 < RA; ++n1) phi[n1] = half ? z[n1].y : z[n1].x;
    const float* vrow = a.V && ok ? a.V + b * a.v_bstride + (long long)r * rg.pitch : nullptr;
    kick_row_points<RA>(x, phi, T6, a, r % rg.ny, r / rg.ny, vrow, [&](int n1) { return RB * n1 + n2; });
    if constexpr (FWD) {
      dftR<RA, false>(x);
#pragma unroll
      for (int k1 = 0; k1 < RA; ++k1) *at(half, k1) = x[k1];
    } else {
      if (ok)
#pragma unroll
        for (int n1 = 0; n1 < RA; ++n1) psi[base + half * rg.pitch + RB * n1] = x[n1];
    }
    if (half == 0) load_points<N>(x, psi_in + base + rg.pitch, ok);
  }
}

template <int N, bool FWD>
__device__ __forceinline__ void kick_units(Warp<N>& w, const float2* psi_in, float2* psi, const float2* H,
                                           const RowGeom& rg, long long hpitch, long long hbstride, const KickArgs& a) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB;
  for (; w.u < w.units; w.u += w.ustride) {
    packed_in<N>(w, H, hpitch, hbstride);
    int b, ra;
    const bool ok = w.pair(w.pr, &b, &ra);
    const long long base = b * rg.bstride + (long long)ra * rg.pitch + w.n2;
    float2 x[RA];
    load_points<N>(x, psi_in + base, ok);
    float T6[10];
    kick_tidal<N>(T6, a, rg, b);
    __syncwarp();
    kick_lane<N, FWD>([&](int half, int k1) { return w.at(half, k1); }, x, psi_in, psi, base, rg, b, ra, ok, w.n2, T6, a);
    __syncwarp();
    if constexpr (FWD) {
      b_items<N, 2 * R::PW>(w, [&](int j, int k1) {
        float2 v[RB];
        b_forward<N, false>(w.tw, v, w.row(j, k1), k1);
        int ib, ir;
        if (!w.pair(j % R::PW, &ib, &ir)) return;
        float2* row = psi + ib * rg.bstride + (long long)(ir + j / R::PW) * rg.pitch + k1;
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) row[RA * k2] = v[k2];
      });
      __syncwarp();
    }
  }
}

template <int N, bool FWD>
__global__ void __launch_bounds__(32 * Rows<N>::WARPS, Rows<N>::KICK)
k_rows_kick(const float2* psi_in, float2* psi, const float2* H, RowGeom rg, long long hpitch,
            long long hbstride, const float4* __restrict__ twg, KickArgs a, XWork work) {
  extern __shared__ __align__(16) float2 smem[];
  Warp<N> w(smem, twg, work);
  kick_units<N, FWD>(w, psi_in, psi, H, rg, hpitch, hbstride, a);
}

// ----------------------------------------------------------------------------
// density: psi x-inverse (+ mask), rho = |psi|^2 (+ rho_b) - shift, packed R2C -> H
// ----------------------------------------------------------------------------
// The pair is done: reduce its RB lanes' CentreAcc and add it to the pair's
// CentreSum (on its first lane).
template <int N>
__device__ __forceinline__ void rows_centre_done(const RhoArgs& a, const RowGeom& rg, const CentreAcc& ca,
                                                 CentreSum& cs, int b, int ra, bool ok, int n2) {
  constexpr int RB = Rows<N>::RB;
  float best = ca.best, s0a = ca.s0[0], s0b = ca.s0[1], si = ca.si;
  unsigned cell = ca.cell;
#pragma unroll
  for (int off = RB / 2; off > 0; off >>= 1) {
    const float ob = __shfl_xor_sync(0xffffffffu, best, off, RB);
    const unsigned oc = __shfl_xor_sync(0xffffffffu, cell, off, RB);
    if (ob > best || (ob == best && oc < cell)) {
      best = ob;
      cell = oc;
    }
    s0a += __shfl_xor_sync(0xffffffffu, s0a, off, RB);
    s0b += __shfl_xor_sync(0xffffffffu, s0b, off, RB);
    si += __shfl_xor_sync(0xffffffffu, si, off, RB);
  }
  if (__any_sync(0xffffffffu, n2 == 0 && ok && cs.item >= 0 && cs.item != b)) {
    centre_gather(cs, RB, a.centre);
    if ((threadIdx.x & 31) == 0) cs.flush(a.centre);
    cs.reset(-1);
  }
  if (n2 != 0 || !ok) return;
  if (cs.item < 0) cs.reset(b);
  const int ja = ra % rg.ny, ka = ra / rg.ny, jb = (ra + 1) % rg.ny, kb = (ra + 1) / rg.ny;
  cs.s0 += (double)s0a + (double)s0b;
  cs.si += (double)si;
  cs.sj += (double)s0a * ja + (double)s0b * jb;
  cs.sk += (double)s0a * ka + (double)s0b * kb;
  if (best >= 0.f) {
    const unsigned long long key =
        ((unsigned long long)__float_as_uint(best) << 32) | (unsigned long long)(0xffffffffu - cell);
    if (key > cs.key) cs.key = key;
  }
}

// The density of one pair by an A lane: psi from the elements at(half, k1)
// (write_psi: inverted, masked and stored at base) or from base; the packed
// (rho_A, rho_B) line's elements to at(0, k1).  base: row A's point n2 in psi.
template <int N, bool CEN, class At>
__device__ __forceinline__ void rho_lane(At at, float2* base, const RowGeom& rg, int b, int ra, bool ok, int n2,
                                         float shift, const RhoArgs& a, CentreAcc& ca) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB;
  float d0[RA];   // the density of row A
  float2 z[RA];   // (rho_A, rho_B)
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    const int r = ra + half;
    float2* row = base + half * rg.pitch;
    float2 v[RA];
    if (a.write_psi) {
#pragma unroll
      for (int k1 = 0; k1 < RA; ++k1) v[k1] = *at(half, k1);
      dftR<RA, true>(v);
      if (a.mx) {
        const float myz = ok ? a.my[r % rg.ny] * a.mz[r / rg.ny] : 0.f;
#pragma unroll
        for (int n1 = 0; n1 < RA; ++n1) v[n1] = cscale(v[n1], myz * a.mx[RB * n1 + n2]);
      }
      if (ok)
#pragma unroll
        for (int n1 = 0; n1 < RA; ++n1) row[RB * n1] = v[n1];
    } else {
      load_points<N>(v, row, ok);
    }
    // each optional step is tested once for the row's points
    float d[RA];
#pragma unroll
    for (int n1 = 0; n1 < RA; ++n1) d[n1] = fmaf(v[n1].x, v[n1].x, v[n1].y * v[n1].y);
    if (ok && a.nonfinite) {
      bool bad = false;
#pragma unroll
      for (int n1 = 0; n1 < RA; ++n1) bad |= !isfinite(d[n1]);
      if (bad) *a.nonfinite = 1;
    }
    if constexpr (CEN) {
#pragma unroll
      for (int n1 = 0; n1 < RA; ++n1) {
        const int x = RB * n1 + n2;
        ca.add(d[n1], (unsigned)r * (unsigned)N + (unsigned)x, x, half);
      }
    }
    // rows without baryon mass are zero and not read
    if (ok && a.rho_b && (!a.rb_rows || a.rb_rows[r])) {
      const float* rb = a.rho_b + b * a.rb_bstride + (long long)r * rg.pitch + n2;
#pragma unroll
      for (int n1 = 0; n1 < RA; ++n1) d[n1] += rb[RB * n1];
    }
#pragma unroll
    for (int n1 = 0; n1 < RA; ++n1) {
      if (half == 0) d0[n1] = d[n1] - shift;
      else z[n1] = make_float2(d0[n1], d[n1] - shift);
    }
  }
  dftR<RA, false>(z);
#pragma unroll
  for (int k1 = 0; k1 < RA; ++k1) *at(0, k1) = z[k1];
}

template <int N, bool CEN>
__device__ __forceinline__ void rho_units(Warp<N>& w, float2* psi, float2* H,
                                          const RowGeom& rg, long long hpitch, long long hbstride, const RhoArgs& a) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB;
  CentreSum cs;
  cs.reset(-1);
  for (; w.u < w.units; w.u += w.ustride) {
    if (a.write_psi) {
      b_items<N, 2 * R::PW>(w, [&](int j, int k1) {
        int ib, ir;
        const bool iok = w.pair(j % R::PW, &ib, &ir);
        const float2* row = psi + ib * rg.bstride + (long long)(ir + j / R::PW) * rg.pitch + k1;
        float2 v[RB];
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) v[k2] = iok ? row[RA * k2] : make_float2(0.f, 0.f);
        b_inverse<N>(w.tw, v, w.row(j, k1), k1);
      });
      __syncwarp();
    }
    int b, ra;
    const bool ok = w.pair(w.pr, &b, &ra);
    const float shift = a.shift ? a.shift[b] : 0.f;
    CentreAcc ca;
    ca.reset();
    rho_lane<N, CEN>([&](int half, int k1) { return w.at(half, k1); },
                     psi + b * rg.bstride + (long long)ra * rg.pitch + w.n2, rg, b, ra, ok, w.n2, shift, a, ca);
    if constexpr (CEN) rows_centre_done<N>(a, rg, ca, cs, b, ra, ok, w.n2);
    __syncwarp();
    packed_out<N>(w, H, hpitch, hbstride);
    __syncwarp();
  }
  if constexpr (CEN) centre_flush(cs, RB, a.centre);
}

// CEN: also accumulate the density maximum and moments for the tide's frame
template <int N, bool CEN>
__global__ void __launch_bounds__(32 * Rows<N>::WARPS, Rows<N>::RHO)
k_rows_rho(float2* psi, float2* H, RowGeom rg, long long hpitch, long long hbstride,
           const float4* __restrict__ twg, RhoArgs a, XWork work) {
  extern __shared__ __align__(16) float2 smem[];
  Warp<N> w(smem, twg, work);
  rho_units<N, CEN>(w, psi, H, rg, hpitch, hbstride, a);
}

// ----------------------------------------------------------------------------
// plain transforms
// ----------------------------------------------------------------------------
// C2C of every row, in place, scaled.
template <int N, bool INV>
__global__ void __launch_bounds__(32 * Rows<N>::WARPS, Rows<N>::RHO)
k_rows_fft(float2* data, RowGeom rg, const float4* __restrict__ twg, float scale, XWork work) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB;
  extern __shared__ __align__(16) float2 smem[];
  Warp<N> w(smem, twg, work);
  for (; w.u < w.units; w.u += w.ustride) {
    int b, ra;
    const bool ok = w.pair(w.pr, &b, &ra);
    const float2* base = data + b * rg.bstride + (long long)ra * rg.pitch + w.n2;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      float2 v[RA];
#pragma unroll
      for (int n1 = 0; n1 < RA; ++n1) v[n1] = ok ? base[half * rg.pitch + RB * n1] : make_float2(0.f, 0.f);
      dftR<RA, INV>(v);
#pragma unroll
      for (int k1 = 0; k1 < RA; ++k1) *w.at(half, k1) = v[k1];
    }
    __syncwarp();
    b_items<N, 2 * R::PW>(w, [&](int j, int k1) {
      float2 v[RB];
      b_forward<N, INV>(w.tw, v, w.row(j, k1), k1);
      int ib, ir;
      if (!w.pair(j % R::PW, &ib, &ir)) return;
      float2* row = data + ib * rg.bstride + (long long)(ir + j / R::PW) * rg.pitch + k1;
#pragma unroll
      for (int k2 = 0; k2 < RB; ++k2) row[RA * k2] = cscale(v[k2], scale);
    });
    __syncwarp();
  }
}

// Phi rows (real) from H.
template <int N>
__global__ void __launch_bounds__(32 * Rows<N>::WARPS, Rows<N>::RHO)
k_rows_c2r(const float2* H, float* out, RowGeom rg, long long hpitch, long long hbstride,
           const float4* __restrict__ twg, XWork work) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB;
  extern __shared__ __align__(16) float2 smem[];
  Warp<N> w(smem, twg, work);
  for (; w.u < w.units; w.u += w.ustride) {
    packed_in<N>(w, H, hpitch, hbstride);
    __syncwarp();
    int b, ra;
    const bool ok = w.pair(w.pr, &b, &ra);
    float2 z[RA];
#pragma unroll
    for (int k1 = 0; k1 < RA; ++k1) z[k1] = *w.at(0, k1);
    dftR<RA, true>(z);
    float* oa = out + b * rg.bstride + (long long)ra * rg.pitch + w.n2;
    if (ok)
#pragma unroll
      for (int n1 = 0; n1 < RA; ++n1) {
        oa[RB * n1] = z[n1].x;
        oa[rg.pitch + RB * n1] = z[n1].y;
      }
    __syncwarp();
  }
}

// Real rows, minus a per-item shift, to half spectra.
template <int N>
__global__ void __launch_bounds__(32 * Rows<N>::WARPS, Rows<N>::RHO)
k_rows_r2c(const float* in, float2* H, RowGeom rg, long long hpitch, long long hbstride,
           const float4* __restrict__ twg, const float* shift_b, XWork work) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB;
  extern __shared__ __align__(16) float2 smem[];
  Warp<N> w(smem, twg, work);
  for (; w.u < w.units; w.u += w.ustride) {
    int b, ra;
    const bool ok = w.pair(w.pr, &b, &ra);
    const float shift = shift_b ? shift_b[b] : 0.f;
    const float* ia = in + b * rg.bstride + (long long)ra * rg.pitch + w.n2;
    float2 z[RA];
#pragma unroll
    for (int n1 = 0; n1 < RA; ++n1)
      z[n1] = ok ? sub2(make_float2(ia[RB * n1], ia[rg.pitch + RB * n1]), both(shift)) : make_float2(0.f, 0.f);
    dftR<RA, false>(z);
#pragma unroll
    for (int k1 = 0; k1 < RA; ++k1) *w.at(0, k1) = z[k1];
    __syncwarp();
    packed_out<N>(w, H, hpitch, hbstride);
    __syncwarp();
  }
}

}  // namespace fx
}  // namespace wdm
