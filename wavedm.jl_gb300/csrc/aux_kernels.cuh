// Auxiliary kernels: density output, FP64 diagnostics reductions, CIC.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace wdm {

// CIC particle: base cell (wrapped into the grid) and fractional offsets in
// [0, 1) along each axis, built in FP64 on the host; m = mass / dV.
struct CicParticle {
  int i[3];
  float f[3];
  float m;
};

enum {
  RED_MASS = 0,  // sum rho
  RED_MAX,       // max rho
  RED_ARG,       // flat index of the max
  RED_MX,        // sum rho x
  RED_MY,
  RED_MZ,
  RED_W,         // sum rho Phi over interior cells
  RED_K,         // sum (rho v)^2 / rho over interior cells
  RED_Q,         // sum |grad sqrt rho|^2 over interior cells
  RED_PX,        // sum rho v (= Im(conj(psi) grad psi)) over interior cells
  RED_PY,
  RED_PZ,
  RED_PHIMAX,    // max |Phi|
  RED_SW,        // z-slice zmid: sum rho, sum rho r, sum rho r^2 (r from the coordinate origin)
  RED_SWR,
  RED_SWR2,
  RED_FIELDS
};
struct RedGeom {
  int nx, ny, nz;
  double dx, dy, dz, x0, y0, z0;
  int zmid;  // z index of the slice the RED_SW* sums cover
};

// The plane of psi that step z of a march over the cells z .. z1 - 1 asks L2 for:
// the one above the cell of step z + RED_AHEAD, which that step loads (k_reduce); -1
// where no step loads it or the grid of nz planes ends below it.
constexpr int RED_AHEAD = 3;  // steps between a plane's L2 prefetch and its loads
__host__ __device__ constexpr int red_ahead_plane(int z, int z1, int nz) {
  return z + RED_AHEAD < z1 && z + RED_AHEAD + 1 < nz ? z + RED_AHEAD + 1 : -1;
}

// Lagrangian radii about the density maximum (RED_ARG of `fields`): per squared
// cell distance key = di^2 + dj^2 + dk^2 the FP64 sum of rho over the cells at
// that distance (wsum, nkeys words), and what the nine quantiles read of it.
// bsum and blast: radii_blocks(nkeys) words.
constexpr int RADII_QUANTILES = 9;
__host__ __device__ constexpr double radii_p(int q) {
  constexpr double p[RADII_QUANTILES] = {0.1, 0.2, 0.3, 0.4, 0.5, 0.6, 0.7, 0.8, 0.9};
  return p[q];
}
struct RadiiOut {
  double total;                    // sum of all weights
  double w1;                       // the weight at distance 0
  double before[RADII_QUANTILES];  // cumulative weight before the quantile's group
  unsigned long long wmin[RADII_QUANTILES];  // bits of the group's smallest weight
  int key[RADII_QUANTILES];        // the group's key (-1: past the last one)
  int prev[RADII_QUANTILES];       // the key with weight before it (-1: none)
  int last;                        // the last key with weight (-1: none)
};
int radii_blocks(long long nkeys);
cudaError_t launch_radii(const float2* psi, int nx, int ny, int nz, const double* fields, double* wsum, long long nkeys,
                         double* bsum, int* blast, RadiiOut* out, cudaStream_t st);

cudaError_t launch_abs2(const float2* psi, float* out, long long n, cudaStream_t st);
// Adjoint seed of L = sum (|psi|^2 - rho_t)^2 dV: lam = 4 (|psi|^2 - rho_t) psi dV,
// loss[b] += sum (|psi|^2 - rho_t)^2 dV (FP64), per batch item of n cells.
cudaError_t launch_adj_seed(const float2* psi, const float* rho_t, float2* lam, long long n, int batch, double dV,
                            double* loss, cudaStream_t st);
// bounded mbarrier wait that runs out (self-test): out[0] error bits, out[1] ns waited
cudaError_t launch_bounded_wait_probe(unsigned long long limit_ns, unsigned long long* out, cudaStream_t st);
// out[2i], out[2i+1] = series sin, cos of h[i] (wdm_math.cuh), for self-tests
cudaError_t launch_sincos_half(const float* h, float* out, long long n, cudaStream_t st);
// shift[b] = mean over item b of |data|^2 (complex_in) or of data (float), + add
cudaError_t launch_mean_shift(const void* data, bool complex_in, long long n, int batch, double* sums, float* shift,
                              double add, cudaStream_t st, float2* copy = nullptr);
// fields[b]: the RED_FIELDS of batch item b (partials: nblocks x RED_FIELDS per item)
cudaError_t launch_reduce(const float2* psi, const float* phi, const RedGeom& g, double* partials, int nblocks,
                          int batch, double* fields, cudaStream_t st);
// CIC deposit of the particles into rho, which must be zero; rows (ny * nz
// ints, may be null) flags the x rows that hold deposited mass.  The deposit
// of static particles is kept: every density pass reads its flagged rows, and
// it is cleared only when the particles change.
cudaError_t launch_cic_deposit(float* rho, const CicParticle* p, long long n, int nx, int ny, int nz, int* rows,
                               cudaStream_t st);
cudaError_t launch_cic_interp(const float* field, const CicParticle* p, long long n, int nx, int ny, int nz,
                              double* out, cudaStream_t st);

}  // namespace wdm
