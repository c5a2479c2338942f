// Plane passes: the y and x transforms around the kick, or around the density,
// of one z plane in one CTA.
//
//   kick     H plane: y inverse; each row pair: C2R, kick, forward x; psi plane: y
//            forward (P8, P1 and P2 of the step in one launch)
//   density  psi plane: y inverse; each row pair: x inverse (+ mask), density, R2C;
//            H plane: y forward (P4, P5 and P6)
//
// With them a step is four launches instead of eight and moves 64 instead of 112
// bytes per cell.  H then stays y-spectral between the density pass and the kick.
// Measured, us per step on separate passes / on plane passes: 96 halos of 64^3
// 555 / 465, 24 of 96^3 494 / 452, 8 of 128^3 389 / 359, one 128^3 76 / 62, one
// 64^3 42 / 32, four of 32^3 43 / 26.  A plane that leaves room for one CTA per SM
// gains no more than that of 128^2, and one with longer rows loses (192 x 96 x 48
// 62 / 66, replayed 43 / 56; 256 x 96 x 256 158 / 169; 64 x 256 x 64 replayed 44 /
// 48): its three phases run one after another in too few warps.  So rows up to
// 128 and planes up to PLANE_BYTES (128^2 and its tables) take this path, where there
// are enough of them and not too many (plane_rule).
//
// The plane is ny rows of RP words.  While it is H, frequency h of row y is at
// word h; while it is psi, x element (k1, n2), and frequency k1 + RA k2 in its
// place, is at word k1 KP + n2 (or k2) as in the row passes, whose buffers E(0) and
// E(1) are the pair's own two rows here.  Everything works in place: the y
// transforms down the columns (an inverse takes its first stage, a forward its
// last, straight from and to global memory), the row phases within a warp's rows.
#pragma once
#include "factor_rows.cuh"

namespace wdm {
namespace fx {

// k1 pitch and row pitch of a plane, from a search with the bank count of the
// row phases and of the y stages.  0: no plane passes for this nx.
template <int N>
struct Plane {
  static constexpr int KP = 0, RP = 0;
};
#define WDM_PLANE(N_, KP_, RP_)                       \
  template <>                                         \
  struct Plane<N_> {                                  \
    static constexpr int KP = KP_, RP = RP_;          \
    static_assert((Plan<N_>::RA - 1) * KP_ + Plan<N_>::RB <= RP_ && N_ / 2 + 1 <= RP_, "row pitch"); \
  };
WDM_PLANE(8, 4, 15)
WDM_PLANE(12, 2, 13)
WDM_PLANE(16, 4, 17)
WDM_PLANE(24, 5, 30)
WDM_PLANE(32, 6, 46)
WDM_PLANE(48, 5, 60)
WDM_PLANE(64, 10, 79)
WDM_PLANE(96, 9, 108)
WDM_PLANE(128, 9, 148)
#undef WDM_PLANE

constexpr size_t PLANE_BYTES = 156 * 1024;
constexpr int PLANE_WARPS = 16;  // most warps per CTA (128 registers per thread)

// CTAs per SM that a plane's shared memory leaves room for.
__host__ __device__ constexpr int plane_fit(size_t smem) {
  const int fit = (int)(228 * 1024 / (smem + 1024));
  return fit > 1 ? fit : 1;
}

// Warps of a plane's CTA: 16 per SM (all that 128 registers a thread allow) over the
// CTAs that an SM holds at a time, of which there are no more than its share of the
// planes (by the room alone 256 planes of 48 x 64 got 3 warps each, two CTAs an SM:
// replayed 52 us a step, now 38, on the separate passes 41).
__host__ __device__ constexpr int plane_warps(size_t smem, int planes, int sms) {
  const int fit = plane_fit(smem), share = (planes + sms - 1) / sms;
  const int ctas = fit < share ? fit : share;
  return ctas < 8 ? (PLANE_WARPS + ctas - 1) / ctas : 2;
}

// Whether `planes` planes of `cells` cells are worth a CTA each, against the separate
// passes (the results are the same bits).  Replayed steps on plane passes / on
// separate ones, us:
// - Room for one CTA per SM: only where one wave of them fills the SMs, or there are
//   so many that the last wave does not count.  Of 128^2: 8 planes 39 / 26, 64 46 /
//   39, 128 54 / 58, 192 91 / 75, 512 224 / 201, 1024 359 / 389.
// - For two: not for a few.  96 x 128: 8 planes 34 / 25, 32 36 / 33, 64 41 / 40, 128
//   56 / 62.
// - Planes of a few hundred cells: not for thousands, whose CTAs are all overhead.
//   8^2: 2048 planes 36 / 34, 8192 73 / 42; 24 x 16: 8192 107 / 91; 12 x 64: 92 / 100.
__host__ __device__ constexpr bool plane_rule(size_t smem, int cells, int planes, int sms) {
  if (smem > PLANE_BYTES) return false;
  if (cells <= 512 && planes > 16 * sms) return false;
  const int fit = plane_fit(smem);
  if (fit == 1) return (4 * planes >= 3 * sms && planes <= sms) || planes >= 6 * sms;
  return fit > 2 || 5 * planes >= 2 * sms;
}

// Rows of the buffer (whole warp units of row pairs) and its bytes with the two
// twiddle tables.
template <int N>
__host__ __device__ constexpr int plane_rows(int ny) {
  constexpr int U = 2 * Rows<N>::PW;
  return (ny + U - 1) / U * U;
}
template <int N>
__host__ __device__ constexpr size_t plane_smem(int ny) {
  return sizeof(float4) * (size_t)(N + ny) + sizeof(float2) * (size_t)plane_rows<N>(ny) * Plane<N>::RP;
}

// The columns of a plane: column c of the global rows sits at word
// (c % ra) kp + c / ra of a plane row (ra = 0: at word c).
struct Columns {
  int n;         // columns
  int ra, kp, rp;
  __device__ __forceinline__ int word(int c) const { return ra ? (c % ra) * kp + c / ra : c; }
};

// y inverse of a plane from global memory (g: its row 0, rows `pitch` apart) into
// s, natural rows.
template <int NY>
__device__ __noinline__ void plane_y_in(const float2* g, long long pitch, float2* s, const Columns c, const float4* tw) {
  using P = Plan<NY>;
  for (int q = threadIdx.x; q < c.n * P::RA; q += blockDim.x) {
    const int k1 = q / c.n, x = q - k1 * c.n;
    float2 v[P::RB];
#pragma unroll
    for (int k2 = 0; k2 < P::RB; ++k2) v[k2] = g[(long long)(k1 + P::RA * k2) * pitch + x];
    dftR<P::RB, true>(v);
    factor_twiddle<NY, true>(v, tw, k1);
    float2* d = s + P::RB * k1 * c.rp + c.word(x);
#pragma unroll
    for (int n2 = 0; n2 < P::RB; ++n2) d[n2 * c.rp] = v[n2];
  }
  __syncthreads();
  for (int q = threadIdx.x; q < c.n * P::RB; q += blockDim.x) {
    const int n2 = q / c.n, x = q - n2 * c.n;
    float2* d = s + n2 * c.rp + c.word(x);
    float2 v[P::RA];
#pragma unroll
    for (int k1 = 0; k1 < P::RA; ++k1) v[k1] = d[P::RB * k1 * c.rp];
    dftR<P::RA, true>(v);
#pragma unroll
    for (int n1 = 0; n1 < P::RA; ++n1) d[P::RB * n1 * c.rp] = v[n1];
  }
  __syncthreads();
}

// y forward of the plane in s (natural rows) to global memory.
template <int NY>
__device__ __noinline__ void plane_y_out(float2* g, long long pitch, float2* s, const Columns c, const float4* tw) {
  using P = Plan<NY>;
  __syncthreads();
  for (int q = threadIdx.x; q < c.n * P::RB; q += blockDim.x) {
    const int n2 = q / c.n, x = q - n2 * c.n;
    float2* d = s + n2 * c.rp + c.word(x);
    float2 v[P::RA];
#pragma unroll
    for (int n1 = 0; n1 < P::RA; ++n1) v[n1] = d[P::RB * n1 * c.rp];
    dftR<P::RA, false>(v);
#pragma unroll
    for (int k1 = 0; k1 < P::RA; ++k1) d[P::RB * k1 * c.rp] = v[k1];
  }
  __syncthreads();
  for (int q = threadIdx.x; q < c.n * P::RA; q += blockDim.x) {
    const int k1 = q / c.n, x = q - k1 * c.n;
    const float2* d = s + P::RB * k1 * c.rp + c.word(x);
    float2 v[P::RB];
#pragma unroll
    for (int n2 = 0; n2 < P::RB; ++n2) v[n2] = d[n2 * c.rp];
    factor_twiddle<NY, false>(v, tw, k1);
    dftR<P::RB, false>(v);
#pragma unroll
    for (int k2 = 0; k2 < P::RB; ++k2) g[(long long)(k1 + P::RA * k2) * pitch + x] = v[k2];
  }
}

// ny a plane pass is built for
#define WDM_PLANE_NY(X) X(8) X(12) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256)

__device__ __forceinline__ void y_in(int ny, const float2* g, long long pitch, float2* s, const Columns& c,
                                     const float4* tw) {
  switch (ny) {
#define WDM_CASE(N_) \
  case N_: plane_y_in<N_>(g, pitch, s, c, tw); break;
    WDM_PLANE_NY(WDM_CASE)
#undef WDM_CASE
  }
}
__device__ __forceinline__ void y_out(int ny, float2* g, long long pitch, float2* s, const Columns& c, const float4* tw) {
  switch (ny) {
#define WDM_CASE(N_) \
  case N_: plane_y_out<N_>(g, pitch, s, c, tw); break;
    WDM_PLANE_NY(WDM_CASE)
#undef WDM_CASE
  }
}
inline bool plane_ny(int ny) {
  switch (ny) {
#define WDM_CASE(N_) case N_:
    WDM_PLANE_NY(WDM_CASE)
#undef WDM_CASE
    return true;
  }
  return false;
}

// What a CTA of a plane pass works on.
struct PlaneArgs {
  const float2* psi_in;   // kick: psi before it (psi: in place)
  float2* psi;
  float2* H;
  RowGeom rg;             // nrows = ny nz
  long long hpitch, hbstride;
  const float4 *twx, *twy;
};

template <int N>
struct PlaneCta {
  using R = Rows<N>;
  static constexpr int KP = Plane<N>::KP, RP = Plane<N>::RP;
  const float4 *twx, *twy;
  float2* s;
  int ny, b, z, warp, lane, pr, n2;
  long long psi0, h0;  // offsets of the plane in psi and H
  Columns hc, pc;      // its columns as H and as psi

  __device__ __forceinline__ PlaneCta(float2* smem, const PlaneArgs& p) {
    float4* t = reinterpret_cast<float4*>(smem);
    ny = p.rg.ny;
    load_twiddles(t, p.twx, N);
    load_twiddles(t + N, p.twy, ny);
    twx = t;
    twy = t + N;
    s = smem + 2 * (N + ny);
    const int nz = p.rg.nrows / ny;
    b = blockIdx.x / nz;
    z = blockIdx.x - b * nz;
    psi0 = b * p.rg.bstride + (long long)z * ny * p.rg.pitch;
    h0 = b * p.hbstride + (long long)z * ny * p.hpitch;
    warp = threadIdx.x >> 5;
    lane = threadIdx.x & 31;
    pr = lane / R::RB;
    n2 = lane % R::RB;
    hc = Columns{N / 2 + 1, 0, 0, RP};
    pc = Columns{N, R::RA, KP, RP};
    __syncthreads();
    chain_wait<CHAIN_SMALL>();
  }
  __device__ __forceinline__ int units() const { return (ny / 2 + R::PW - 1) / R::PW; }
  __device__ __forceinline__ float2* row(int y) const { return s + y * RP; }
};

// The packed lines of unit u replace the half spectra they come from, once all of the
// unit's are in registers.
template <int N>
__device__ __forceinline__ void plane_packed_in(const PlaneCta<N>& c, int u) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB, PW = R::PW, KP = Plane<N>::KP, ROUNDS = (PW * RA + 31) / 32;
  float2 v[ROUNDS][RB];
#pragma unroll
  for (int i = 0; i < ROUNDS; ++i) {
    const int q = c.lane + 32 * i, y = 2 * (u * PW + q / RA);
    pack_half<N>(v[i], c.row(y), c.row(y + 1), q < PW * RA, q % RA);
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < ROUNDS; ++i) {
    const int q = c.lane + 32 * i;
    if (q < PW * RA) b_inverse<N>(c.twx, v[i], c.row(2 * (u * PW + q / RA)) + (q % RA) * KP, q % RA);
  }
}

// Phi in real space (rows of `out` as those of psi) from a y-spectral H, which stays.
template <int N>
__global__ void __launch_bounds__(32 * PLANE_WARPS, 1) k_plane_c2r(PlaneArgs p, float* out) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB, PW = R::PW, KP = Plane<N>::KP;
  extern __shared__ __align__(16) float2 smem[];
  PlaneCta<N> c(smem, p);
  y_in(c.ny, p.H + c.h0, p.hpitch, c.s, c.hc, c.twy);
  for (int u = c.warp; u < c.units(); u += blockDim.x >> 5) {
    plane_packed_in(c, u);
    __syncwarp();
    const int y = 2 * (u * PW + c.pr);
    float2 z[RA];
#pragma unroll
    for (int k1 = 0; k1 < RA; ++k1) z[k1] = c.row(y)[k1 * KP + c.n2];
    dftR<RA, true>(z);
    float* oa = out + c.psi0 + (long long)y * p.rg.pitch + c.n2;
    if (y < c.ny)
#pragma unroll
      for (int n1 = 0; n1 < RA; ++n1) {
        oa[RB * n1] = z[n1].x;
        oa[p.rg.pitch + RB * n1] = z[n1].y;
      }
  }
}

template <int N, bool FWD>
__global__ void __launch_bounds__(32 * PLANE_WARPS, 1) k_plane_kick(PlaneArgs p, KickArgs a) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB, PW = R::PW, KP = Plane<N>::KP;
  extern __shared__ __align__(16) float2 smem[];
  PlaneCta<N> c(smem, p);
  y_in(c.ny, p.H + c.h0, p.hpitch, c.s, c.hc, c.twy);
  float T6[10];
  kick_tidal<N>(T6, a, p.rg, c.b);
  for (int u = c.warp; u < c.units(); u += blockDim.x >> 5) {
    plane_packed_in(c, u);
    const int y = 2 * (u * PW + c.pr);
    const bool ok = y < c.ny;
    const int ra = c.z * c.ny + (ok ? y : 0);
    const long long base = c.b * p.rg.bstride + (long long)ra * p.rg.pitch + c.n2;
    float2 x[RA];
    load_points<N>(x, p.psi_in + base, ok);
    __syncwarp();
    kick_lane<N, FWD>([&](int half, int k1) { return c.row(y + half) + k1 * KP + c.n2; }, x, p.psi_in, p.psi, base, p.rg,
                      c.b, ra, ok, c.n2, T6, a);
    if constexpr (FWD) {
      __syncwarp();
#pragma unroll 1
      for (int q = c.lane; q < 2 * PW * RA; q += 32) {
        const int k1 = q % RA;
        float2* d = c.row(2 * u * PW + q / RA) + k1 * KP;
        float2 v[RB];
        b_forward<N, false>(c.twx, v, d, k1);
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) d[k2] = v[k2];
      }
    }
  }
  if constexpr (FWD) y_out(c.ny, p.psi + c.psi0, p.rg.pitch, c.s, c.pc, c.twy);
}

template <int N, bool CEN>
__global__ void __launch_bounds__(32 * PLANE_WARPS, 1) k_plane_rho(PlaneArgs p, RhoArgs a) {
  using R = Rows<N>;
  constexpr int RA = R::RA, RB = R::RB, PW = R::PW, KP = Plane<N>::KP;
  constexpr int ITEMS = PW * RA / 2, ROUNDS = (ITEMS + 31) / 32;
  extern __shared__ __align__(16) float2 smem[];
  PlaneCta<N> c(smem, p);
  if (a.write_psi) y_in(c.ny, p.psi + c.psi0, p.rg.pitch, c.s, c.pc, c.twy);
  const float shift = a.shift ? a.shift[c.b] : 0.f;
  CentreSum cs;
  cs.reset(-1);
  for (int u = c.warp; u < c.units(); u += blockDim.x >> 5) {
    if (a.write_psi) {
#pragma unroll 1
      for (int q = c.lane; q < 2 * PW * RA; q += 32) {
        const int k1 = q % RA;
        float2* d = c.row(2 * u * PW + q / RA) + k1 * KP;
        float2 v[RB];
#pragma unroll
        for (int k2 = 0; k2 < RB; ++k2) v[k2] = d[k2];
        b_inverse<N>(c.twx, v, d, k1);
      }
      __syncwarp();
    }
    const int y = 2 * (u * PW + c.pr);
    const bool ok = y < c.ny;
    const int ra = c.z * c.ny + (ok ? y : 0);
    CentreAcc ca;
    ca.reset();
    rho_lane<N, CEN>([&](int half, int k1) { return c.row(y + half) + k1 * KP + c.n2; },
                     p.psi + c.b * p.rg.bstride + (long long)ra * p.rg.pitch + c.n2, p.rg, c.b, ra, ok, c.n2, shift, a, ca);
    if constexpr (CEN) rows_centre_done<N>(a, p.rg, ca, cs, c.b, ra, ok, c.n2);
    __syncwarp();
    // the half spectra replace the packed lines, once all of the unit's are in registers
    float2 va[ROUNDS][RB], vb[ROUNDS][RB];
#pragma unroll
    for (int i = 0; i < ROUNDS; ++i) {
      const int q = c.lane + 32 * i, k1 = q % (RA / 2), kb = k1 ? RA - k1 : RA / 2;
      if (q >= ITEMS) continue;
      const float2* e = c.row(2 * (u * PW + q / (RA / 2)));
      b_forward<N, false>(c.twx, va[i], e + k1 * KP, k1);
      b_forward<N, false>(c.twx, vb[i], e + kb * KP, kb);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < ROUNDS; ++i) {
      const int q = c.lane + 32 * i;
      if (q >= ITEMS) continue;
      float2* h = c.row(2 * (u * PW + q / (RA / 2)));
      split_half<N>(va[i], vb[i], q % (RA / 2), [&](int k, float2 xa, float2 xb) {
        h[k] = xa;
        h[Plane<N>::RP + k] = xb;
      });
    }
  }
  if constexpr (CEN) centre_flush(cs, RB, a.centre);
  y_out(c.ny, p.H + c.h0, p.hpitch, c.s, c.hc, c.twy);
}

}  // namespace fx
}  // namespace wdm
