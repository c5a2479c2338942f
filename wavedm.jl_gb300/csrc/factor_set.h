// Per-axis-length table of the two-factor pass launchers (factor_lines.cuh,
// factor_rows.cuh).  Each supported length is compiled in one of the
// factor_*.cu translation units.
#pragma once
#include <cuda_runtime.h>
#include "kernel_set.h"

namespace wdm {

struct FactorSet {
  int n;
  // strided lines (y or z axis), C2C in place
  cudaError_t (*line)(float2* data, const LineGeom& g, const float4* tw, bool inv, int batch, cudaStream_t st);
  cudaError_t (*line_drift)(float2* data, const LineGeom& g, const float4* tw, const DriftOp& op, int batch,
                            cudaStream_t st);
  cudaError_t (*line_poisson)(float2* data, const LineGeom& g, const float4* tw, const PoissonOp& op, int batch,
                              cudaStream_t st);
  // contiguous rows (x axis)
  cudaError_t (*fft)(float2* data, const RowGeom& rg, const float4* tw, bool inv, float scale, int batch,
                     cudaStream_t st);
  cudaError_t (*rho)(float2* psi, float2* H, const RowGeom& rg, long long hpitch, long long hbstride, const float4* tw,
                     const RhoArgs& a, int batch, cudaStream_t st);
  cudaError_t (*kick)(const float2* psi_in, float2* psi, const float2* H, const RowGeom& rg, long long hpitch,
                      long long hbstride, const float4* tw, const KickArgs& a, bool fwd, int batch, cudaStream_t st);
  cudaError_t (*c2r)(const float2* H, float* out, const RowGeom& rg, long long hpitch, long long hbstride,
                     const float4* tw, int batch, cudaStream_t st);
  cudaError_t (*r2c)(const float* in, float2* H, const RowGeom& rg, long long hpitch, long long hbstride,
                     const float4* tw, const float* shift, int batch, cudaStream_t st);
  // plane passes of rows of this length in planes of ny rows (factor_planes.cuh):
  // whether so many of them are worth it (plane_rule), and the launches (kick: H y-spectral ->
  // psi x- and y-spectral, or kicked in real space when !fwd; rho: psi x- and
  // y-spectral, or real when !a.write_psi -> H y-spectral)
  bool (*plane_ok)(int ny, int planes);
  cudaError_t (*plane_kick)(const float2* psi_in, float2* psi, const float2* H, const RowGeom& rg, long long hpitch,
                            long long hbstride, const float4* twx, const float4* twy, const KickArgs& a, bool fwd,
                            int batch, cudaStream_t st);
  cudaError_t (*plane_rho)(float2* psi, float2* H, const RowGeom& rg, long long hpitch, long long hbstride,
                           const float4* twx, const float4* twy, const RhoArgs& a, int batch, cudaStream_t st);
  // H y-spectral -> Phi in real space (H stays)
  cudaError_t (*plane_c2r)(const float2* H, float* out, const RowGeom& rg, long long hpitch, long long hbstride,
                           const float4* twx, const float4* twy, int batch, cudaStream_t st);
  // host: fill the n-entry twiddle table of this axis length
  void (*fill_twiddles)(float4* out);
};

const FactorSet* factors_for(int n);

}  // namespace wdm
