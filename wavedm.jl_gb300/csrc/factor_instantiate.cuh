// Launchers of the two-factor passes for one axis length N (included by
// factor_*.cu).
#pragma once
#include "factor_lines.cuh"
#include "factor_planes.cuh"
#include "factor_rows.cuh"
#include "factor_set.h"
#include "launch_util.cuh"

namespace wdm {
namespace fx {

template <int N>
struct Launch {
  static constexpr int NT = line_threads<N>();

  template <int MODE, bool LATE, class Op>
  static cudaError_t tma(float2* data, const CUtensorMap& map, const CUtensorMap& emap, const LineGeom& ge,
                         const float4* tw, const Op& op, int batch, cudaStream_t st) {
    constexpr size_t SMEM = line_tma_smem<N, MODE, Op>();
    constexpr auto K = k_line_tma<N, MODE, Op, LATE>;
    cudaError_t e;
    if ((e = prep_once<K>(SMEM)) != cudaSuccess) return e;
    const int tx = ge.edge ? ge.nxa / LINES : (ge.nxa + LINES - 1) / LINES;
    const long long tiles = ((long long)ge.rows * tx + ge.edge) * batch;
    const long long cap = (long long)resident_ctas<K>(NT, SMEM) * sm_count();
    return launch_chained<K>(dim3((unsigned)(tiles < cap ? tiles : cap)), NT, SMEM, st, data, map, emap, ge, tw, op, batch);
  }

  // The line pass as the context's tuner chose it: the TMA pass where the
  // array has a tensor-map view, else one register tile per CTA (lines may
  // straddle rows).
  template <int MODE, class Op>
  static cudaError_t lines(float2* data, const LineGeom& g, const float4* tw, const Op& op, int batch,
                           cudaStream_t st) {
    if (g.nlines <= 0 || batch <= 0) return cudaSuccess;
    CUtensorMap map, emap;
    if (g.impl == LINE_IMPL_TMA && LineMaps<N>::line_map(&map, data, g, batch)) {
      LineGeom ge = g;
      ge.edge = LineMaps<N>::edge_map(&emap, data, g, batch) ? g.rows / 8 : 0;
      if (!ge.edge) emap = map;  // not read
      // With two slots the next tile's copy goes out late (k_line_tma) in the
      // fused z passes and in the y passes of a half spectrum (the ones with
      // edge tiles), early in the y passes of psi, which are bound by memory.
      if constexpr (MODE == 2) {
        return tma<MODE, true>(data, map, emap, ge, tw, op, batch, st);
      } else {
        if (ge.edge) return tma<MODE, true>(data, map, emap, ge, tw, op, batch, st);
        return tma<MODE, false>(data, map, emap, ge, tw, op, batch, st);
      }
    }
    constexpr size_t SMEM = line_tile_smem<N>();
    constexpr auto K = k_line_tile<N, MODE, Op>;
    cudaError_t e;
    if ((e = prep_once<K>(SMEM)) != cudaSuccess) return e;
    return launch_chained<K>(dim3((g.nlines + LINES - 1) / LINES, batch), NT, SMEM, st, data, g, tw, op);
  }
  static cudaError_t line(float2* data, const LineGeom& g, const float4* tw, bool inv, int batch, cudaStream_t st) {
    return inv ? lines<1>(data, g, tw, None{}, batch, st) : lines<0>(data, g, tw, None{}, batch, st);
  }
  static cudaError_t line_drift(float2* data, const LineGeom& g, const float4* tw, const DriftOp& op, int batch,
                                cudaStream_t st) {
    return lines<2>(data, g, tw, Drift{op}, batch, st);
  }
  static cudaError_t line_poisson(float2* data, const LineGeom& g, const float4* tw, const PoissonOp& op, int batch,
                                  cudaStream_t st) {
    return lines<2>(data, g, tw, Poisson{op}, batch, st);
  }

  // Row passes: one resident wave of warps over the units of PW row pairs; a
  // grid with fewer units than warps takes smaller CTAs, so that the units
  // spread over the SMs.
  using R = Rows<N>;
  template <auto K, int CTAS, class... Args>
  static cudaError_t rows(const RowGeom& rg, int batch, cudaStream_t st, const Args&... args) {
    XWork w;
    w.pairs_per_item = rg.nrows / 2;
    w.batch = batch;
    const long long units = ((long long)w.pairs_per_item * batch + R::PW - 1) / R::PW;
    if (units <= 0) return cudaSuccess;
    cudaError_t e;
    if ((e = prep_once<K>(R::smem(R::WARPS))) != cudaSuccess) return e;
    const int sms = sm_count();
    const long long per_sm = (units + sms - 1) / sms;
    const int warps = (int)(per_sm < R::WARPS ? per_sm : R::WARPS);
    const long long ctas = (units + warps - 1) / warps, cap = (long long)CTAS * sms;
    return launch_chained<K>(dim3((unsigned)(ctas < cap ? ctas : cap)), 32 * warps, R::smem(warps), st, args..., w);
  }
  static cudaError_t fft(float2* data, const RowGeom& rg, const float4* tw, bool inv, float scale, int batch,
                         cudaStream_t st) {
    return inv ? rows<k_rows_fft<N, true>, R::RHO>(rg, batch, st, data, rg, tw, scale)
               : rows<k_rows_fft<N, false>, R::RHO>(rg, batch, st, data, rg, tw, scale);
  }
  static cudaError_t rho(float2* psi, float2* H, const RowGeom& rg, long long hpitch, long long hbstride,
                         const float4* tw, const RhoArgs& a, int batch, cudaStream_t st) {
    return a.centre ? rows<k_rows_rho<N, true>, R::RHO>(rg, batch, st, psi, H, rg, hpitch, hbstride, tw, a)
                    : rows<k_rows_rho<N, false>, R::RHO>(rg, batch, st, psi, H, rg, hpitch, hbstride, tw, a);
  }
  static cudaError_t kick(const float2* psi_in, float2* psi, const float2* H, const RowGeom& rg, long long hpitch,
                          long long hbstride, const float4* tw, const KickArgs& a, bool fwd, int batch,
                          cudaStream_t st) {
    return fwd ? rows<k_rows_kick<N, true>, R::KICK>(rg, batch, st, psi_in, psi, H, rg, hpitch, hbstride, tw, a)
               : rows<k_rows_kick<N, false>, R::KICK>(rg, batch, st, psi_in, psi, H, rg, hpitch, hbstride, tw, a);
  }
  static cudaError_t c2r(const float2* H, float* out, const RowGeom& rg, long long hpitch, long long hbstride,
                         const float4* tw, int batch, cudaStream_t st) {
    return rows<k_rows_c2r<N>, R::RHO>(rg, batch, st, H, out, rg, hpitch, hbstride, tw);
  }
  static cudaError_t r2c(const float* in, float2* H, const RowGeom& rg, long long hpitch, long long hbstride,
                         const float4* tw, const float* shift, int batch, cudaStream_t st) {
    return rows<k_rows_r2c<N>, R::RHO>(rg, batch, st, in, H, rg, hpitch, hbstride, tw, shift);
  }
  // Plane passes: one CTA per plane.
  static bool plane_ok(int ny, int planes) {
    if constexpr (Plane<N>::KP == 0) return false;
    else return plane_ny(ny) && plane_rule(plane_smem<N>(ny), N * ny, planes, sm_count());
  }
  template <auto K, class Args>
  static cudaError_t plane(const PlaneArgs& p, const Args& a, int batch, cudaStream_t st) {
    cudaError_t e;
    if ((e = prep_once<K>(PLANE_BYTES)) != cudaSuccess) return e;
    const size_t smem = plane_smem<N>(p.rg.ny);
    const int planes = p.rg.nrows / p.rg.ny * batch;
    return launch_chained<K>(dim3(planes), 32 * plane_warps(smem, planes, sm_count()), smem, st, p, a);
  }
  static cudaError_t plane_kick(const float2* psi_in, float2* psi, const float2* H, const RowGeom& rg,
                                long long hpitch, long long hbstride, const float4* twx, const float4* twy,
                                const KickArgs& a, bool fwd, int batch, cudaStream_t st) {
    if constexpr (Plane<N>::KP == 0) {
      return cudaErrorInvalidValue;
    } else {
      const PlaneArgs p{psi_in, psi, const_cast<float2*>(H), rg, hpitch, hbstride, twx, twy};
      return fwd ? plane<k_plane_kick<N, true>>(p, a, batch, st) : plane<k_plane_kick<N, false>>(p, a, batch, st);
    }
  }
  static cudaError_t plane_rho(float2* psi, float2* H, const RowGeom& rg, long long hpitch, long long hbstride,
                               const float4* twx, const float4* twy, const RhoArgs& a, int batch, cudaStream_t st) {
    if constexpr (Plane<N>::KP == 0) {
      return cudaErrorInvalidValue;
    } else {
      const PlaneArgs p{psi, psi, H, rg, hpitch, hbstride, twx, twy};
      return a.centre ? plane<k_plane_rho<N, true>>(p, a, batch, st) : plane<k_plane_rho<N, false>>(p, a, batch, st);
    }
  }
  static cudaError_t plane_c2r(const float2* H, float* out, const RowGeom& rg, long long hpitch, long long hbstride,
                               const float4* twx, const float4* twy, int batch, cudaStream_t st) {
    if constexpr (Plane<N>::KP == 0) {
      return cudaErrorInvalidValue;
    } else {
      const PlaneArgs p{nullptr, nullptr, const_cast<float2*>(H), rg, hpitch, hbstride, twx, twy};
      return plane<k_plane_c2r<N>>(p, out, batch, st);
    }
  }
  static void fill_twiddles(float4* out) {
    fill_factor_twiddles<N>(out, [](long long m) {
      const double a = -2.0 * 3.14159265358979323846 * (double)m / (double)N;
      return pack_twiddle(std::cos(a), std::sin(a));
    });
  }
  static const FactorSet* set() {
    static const FactorSet fs = {N,    &line, &line_drift, &line_poisson, &fft,       &rho,          &kick,
                                 &c2r, &r2c,  &plane_ok,   &plane_kick,   &plane_rho, &plane_c2r,    &fill_twiddles};
    return &fs;
  }
};

}  // namespace fx
}  // namespace wdm

#define WDM_FACTORS(N) \
  namespace wdm {      \
  const FactorSet* fs_##N() { return fx::Launch<N>::set(); } \
  }
