// Auxiliary kernels: density output, FP64 diagnostics reductions, CIC.
#include "aux_kernels.cuh"
#include "fft_factor.cuh"
#include "tma.cuh"
#include "wdm_math.cuh"

#include <type_traits>

namespace wdm {

__global__ void k_sincos_half(const float* __restrict__ h, float* __restrict__ out, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float s, c;
    sincos_half(h[i], &s, &c);
    out[2 * i] = s;
    out[2 * i + 1] = c;
  }
}

__global__ void k_adj_seed(const float2* __restrict__ psi, const float* __restrict__ rho_t, float2* __restrict__ lam,
                           long long n, double dV, double* __restrict__ loss) {
  const long long off = blockIdx.y * n;
  double acc = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float2 p = psi[off + i];
    const float d = p.x * p.x + p.y * p.y - rho_t[off + i];
    const float s = (float)(4.0 * dV) * d;
    lam[off + i] = make_float2(s * p.x, s * p.y);
    acc += (double)d * d;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  __shared__ double sh[32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
    atomicAdd(loss + blockIdx.y, s * dV);
  }
}

cudaError_t launch_adj_seed(const float2* psi, const float* rho_t, float2* lam, long long n, int batch, double dV,
                            double* loss, cudaStream_t st) {
  long long blocks = (n + 255) / 256;
  if (blocks > 608) blocks = 608;
  k_adj_seed<<<dim3((unsigned)blocks, batch), 256, 0, st>>>(psi, rho_t, lam, n, dV, loss);
  return cudaGetLastError();
}

// One CTA waits on an mbarrier phase that nothing completes (no arrival, no
// copy), through the same bounded wait the TMA line passes use; it records
// WDM_DEVERR_TMA_WAIT in out[0] and the nanoseconds it waited in out[1].
__global__ void k_bounded_wait_probe(unsigned long long limit_ns, unsigned long long* out) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  const unsigned long long t0 = globaltimer_ns();
  const bool landed = mbar_wait_bounded(&bar, 0u, limit_ns);
  const bool all = __syncthreads_and(landed);
  if (threadIdx.x == 0) {
    out[0] = all ? 0ull : (unsigned long long)WDM_DEVERR_TMA_WAIT;
    out[1] = globaltimer_ns() - t0;
  }
}

cudaError_t launch_bounded_wait_probe(unsigned long long limit_ns, unsigned long long* out, cudaStream_t st) {
  k_bounded_wait_probe<<<1, 128, 0, st>>>(limit_ns, out);
  return cudaGetLastError();
}

cudaError_t launch_sincos_half(const float* h, float* out, long long n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const long long b = (n + 255) / 256;
  k_sincos_half<<<(unsigned)(b < 4096 ? b : 4096), 256, 0, st>>>(h, out, n);
  return cudaGetLastError();
}

__global__ void k_abs2(const float2* __restrict__ psi, float* __restrict__ out, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float2 v = psi[i];
    out[i] = v.x * v.x + v.y * v.y;
  }
}

cudaError_t launch_abs2(const float2* psi, float* out, long long n, cudaStream_t st) {
  const int blocks = (int)((n + 255) / 256 < 152 * 16 ? (n + 255) / 256 : 152 * 16);
  k_abs2<<<blocks, 256, 0, st>>>(psi, out, n);
  return cudaGetLastError();
}

// Diagnostics sums.  The sums restate src/visualization/runtime.jl:210-238
// (interior cells, second-order central differences) and
// src/simulation_main.jl:652 (total mass).
//
// A warp takes 32 neighbouring x of one row y and marches along z with the cell
// below and the cell above it in registers: a cell's psi and |psi| are loaded and
// formed once as the cell above, its x neighbours come from the neighbouring
// lanes (the outer lanes load theirs), its y neighbours from memory (L1: the next
// warps' rows).  A step's loads are issued one step ahead, behind an L2 prefetch.
// That is four square roots per cell instead of seven.  Bound by instruction issue
// (300 a cell, 63% of the slots: the per-cell terms, four IEEE roots, a division,
// eleven compensated sums); 256^3 350 -> 210 us, with the per-cell terms and the
// precision of the sums unchanged.
constexpr int RED_THREADS = 128;
constexpr int RED_CTAS = 5;   // resident blocks an SM
// Cells along z of one march: long marches read the planes beside them less often,
// short ones give every warp of the grid some work.
static int red_depth(const RedGeom& g, int nblocks) {
  int depth = 32;
  auto tasks = [&] { return (long long)((g.nx + 31) / 32) * g.ny * ((g.nz + depth - 1) / depth); };
  while (depth > 4 && tasks() < (long long)nblocks * (RED_THREADS / 32)) depth /= 2;
  return depth;
}

// Two running sums side by side as unevaluated float pairs hi + lo (Knuth's
// two-sum moves every rounding error of hi into lo).  What is lost are the roundings of
// lo itself: with the n of 1,400 terms that a thread adds at most (512^3 over 760 blocks
// of 128) about 2^-50 n / 2 = 2^-40 of its sum as roundings fall, n^2 / 3 2^-48 = 2^-28
// at the worst, and less of the total of all threads.  FP64 arithmetic per cell runs at
// a small fraction of the FP32 rate on this GPU.
struct FAcc2 {
  float2 hi = {0.f, 0.f}, lo = {0.f, 0.f};
  __device__ __forceinline__ void add(float u, float v) {
    const float2 t = make_float2(u, v);
    const float2 s = fx::add2(hi, t);
    const float2 bb = fx::sub2(s, hi);
    lo = fx::add2(lo, fx::add2(fx::sub2(hi, fx::sub2(s, bb)), fx::sub2(t, bb)));
    hi = s;
  }
  __device__ __forceinline__ double x() const { return (double)hi.x + (double)lo.x; }
  __device__ __forceinline__ double y() const { return (double)hi.y + (double)lo.y; }
};

// One field's running value: sums, the largest |Phi|, the density maximum with the
// first cell that holds it.
struct RedTake {
  int q;
  double v, arg;
  __device__ RedTake(int field, double v0, double arg0) : q(field), v(v0), arg(arg0) {}
  __device__ __forceinline__ void take(double u, double ua) {
    if (q == RED_MAX) {
      if (u > v || (u == v && ua < arg)) {
        v = u;
        arg = ua;
      }
    } else if (q == RED_PHIMAX) {
      v = fmax(v, u);
    } else if (q != RED_ARG) {
      v += u;
    }
  }
  __device__ __forceinline__ void store(double* fields) const {
    if (q == RED_ARG) return;  // comes with RED_MAX
    fields[q] = v;
    if (q == RED_MAX) fields[RED_ARG] = arg;
  }
};

// One block partial per (block, batch item): RED_FIELDS doubles.
__global__ void __launch_bounds__(RED_THREADS, RED_CTAS)
k_reduce(const float2* __restrict__ psi_all, const float* __restrict__ phi_all, RedGeom g, int depth,
         double* __restrict__ partials) {
  const int nxy = g.nx * g.ny;  // an item has at most 512^3 cells
  const long long n = (long long)nxy * g.nz;
  const float2* psi = psi_all + blockIdx.y * n;
  const float* phi = phi_all + blockIdx.y * n;
  FAcc2 m_w, mxy, mz_k, q_pz, pxy;  // (mass, W), (x, y), (z, K), (Q, pz), (px, py)
  float best_hi = -1.f, best_lo = 0.f, phimax = 0.f;
  int best_i = 0;
  const float fi2dx = (float)(0.5 / g.dx), fi2dy = (float)(0.5 / g.dy), fi2dz = (float)(0.5 / g.dz);
  const float fx0 = (float)g.x0, fy0 = (float)g.y0, fz0 = (float)g.z0;
  const float fdx = (float)g.dx, fdy = (float)g.dy, fdz = (float)g.dz;
  auto mag = [](float2 v) { return sqrtf(fmaf(v.x, v.x, v.y * v.y)); };
  const int lane = threadIdx.x & 31;
  const int tiles = (g.nx + 31) / 32, depths = (g.nz + depth - 1) / depth;
  const int tasks = tiles * g.ny * depths;  // neighbouring warps: neighbouring rows
  for (int task = blockIdx.x * (RED_THREADS / 32) + (threadIdx.x >> 5); task < tasks; task += gridDim.x * (RED_THREADS / 32)) {
    const int y = task % g.ny, td = task / g.ny, tx = td % tiles, z0 = (td / tiles) * depth;
    const int z1 = z0 + depth < g.nz ? z0 + depth : g.nz;
    const int x = tx * 32 + lane;
    const bool in = x < g.nx;
    const bool xy_inner = in && x > 0 && x < g.nx - 1 && y > 0 && y < g.ny - 1;
    // the outer lanes' missing x neighbour
    const bool edge = (lane == 0 && x > 0) || (lane == 31 && x < g.nx - 1);
    const int i0 = z0 * nxy + y * g.nx + (in ? x : 0);
    const float rx = fmaf(fdx, (float)x, fx0), ry = fmaf(fdy, (float)y, fy0);
    const float2 zero = make_float2(0.f, 0.f);
    const float2* ps = psi + i0;
    const float* fs = phi + i0;
    // a step's loads are issued one step ahead of their use
    float2 n_zp = zero, n_e = zero, n_yp = zero, n_ym = zero;
    float n_ph = 0.f;
    auto load = [&](int z) {  // what step z reads; ps and fs point at its cell
      n_zp = z + 1 < g.nz && in ? ps[nxy] : zero;
      n_ph = in ? *fs : 0.f;
      n_e = edge ? ps[lane == 0 ? -1 : 1] : zero;
      n_yp = xy_inner ? ps[g.nx] : zero;
      n_ym = xy_inner ? ps[-g.nx] : zero;
    };
    float2 zm = z0 > 0 && in ? ps[-nxy] : zero, p = in ? *ps : zero;
    load(z0);
    float mzm = mag(zm), mp = mag(p);
    for (int z = z0; z < z1; ++z) {
      const float2 zp = n_zp, e = n_e, yp = n_yp, ym = n_ym;
      const float ph = n_ph;
      ps += nxy;
      fs += nxy;
      if (z + 1 < z1) load(z + 1);
      // ps and fs are at step z + 1 by now
      const int ahead = red_ahead_plane(z, z1, g.nz);
      if (in && ahead >= 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(ps + (ahead - (z + 1)) * nxy));
      if (in && z + RED_AHEAD < z1) asm volatile("prefetch.global.L2 [%0];" ::"l"(fs + (RED_AHEAD - 1) * nxy));
      const float mzp = mag(zp);
      const bool inner = xy_inner && z > 0 && z < g.nz - 1;
      const float me = mag(e);
      float2 xp, xm;
      xp.x = __shfl_down_sync(0xffffffffu, p.x, 1);
      xp.y = __shfl_down_sync(0xffffffffu, p.y, 1);
      xm.x = __shfl_up_sync(0xffffffffu, p.x, 1);
      xm.y = __shfl_up_sync(0xffffffffu, p.y, 1);
      float mxp = __shfl_down_sync(0xffffffffu, mp, 1), mxm = __shfl_up_sync(0xffffffffu, mp, 1);
      if (lane == 31) {
        xp = e;
        mxp = me;
      }
      if (lane == 0) {
        xm = e;
        mxm = me;
      }
      // rho = p.x^2 + p.y^2 as (rs, rt) to 2^-47: two-product of each square, two-sum of
      // the pair, normalised for the comparison.  __fmul_rn: a product that the compiler
      // fuses into one of the additions would no longer be the one whose rounding is ea.
      const float a = __fmul_rn(p.x, p.x), b = __fmul_rn(p.y, p.y);
      const float ea = fmaf(p.x, p.x, -a), eb = fmaf(p.y, p.y, -b);
      const float r0 = a + b;
      const float bb = r0 - a;
      const float r1 = ((a - (r0 - bb)) + (b - bb)) + (ea + eb);
      // beyond FP32 the errors are differences of infinities: rho = r0 alone
      const bool over = r0 == INFINITY;
      const float rs = over ? r0 : r0 + r1, rt = over ? 0.f : r1 - (rs - r0);
      if (in && rs >= best_hi) {
        const int i = i0 + (z - z0) * nxy;
        if (rs > best_hi || rt > best_lo || (rt == best_lo && i < best_i)) {
          best_hi = rs;
          best_lo = rt;
          best_i = i;
        }
      }
      phimax = fmaxf(phimax, fabsf(ph));
      // per-cell terms in FP32 (the reference forms them from its FP32 psi too)
      float jx = 0.f, jy = 0.f, jz = 0.f, k = 0.f, q = 0.f;
      if (inner) {
        // rho v = Im(conj(psi) grad psi)
        const float gxr = (xp.x - xm.x) * fi2dx, gxi = (xp.y - xm.y) * fi2dx;
        const float gyr = (yp.x - ym.x) * fi2dy, gyi = (yp.y - ym.y) * fi2dy;
        const float gzr = (zp.x - zm.x) * fi2dz, gzi = (zp.y - zm.y) * fi2dz;
        jx = fmaf(p.x, gxi, -p.y * gxr);
        jy = fmaf(p.x, gyi, -p.y * gyr);
        jz = fmaf(p.x, gzi, -p.y * gzr);
        if (rs > 0.f) k = fmaf(jx, jx, fmaf(jy, jy, jz * jz)) / rs;
        const float ax = (mxp - mxm) * fi2dx;
        const float ay = (mag(yp) - mag(ym)) * fi2dy;
        const float az = (mzp - mzm) * fi2dz;
        q = fmaf(ax, ax, fmaf(ay, ay, az * az));
      }
      m_w.add(rs, inner ? rs * ph : 0.f);
      m_w.lo.x += rt;
      mxy.add(rs * rx, rs * ry);
      mz_k.add(rs * fmaf(fdz, (float)z, fz0), k);
      q_pz.add(q, jz);
      pxy.add(jx, jy);
      zm = p;
      mzm = mp;
      p = zp;
      mp = mzp;
    }
  }
  // one z-slice only: FP64 is cheap there
  double sw = 0.0, swr = 0.0, swr2 = 0.0;
  for (int c = blockIdx.x * RED_THREADS + threadIdx.x; c < nxy; c += gridDim.x * RED_THREADS) {
    const int y = c / g.nx, x = c - y * g.nx;
    const float2 p = psi[g.zmid * nxy + c];
    const double rho = fma((double)p.x, (double)p.x, (double)p.y * p.y);
    const double fx = g.x0 + g.dx * x, fy = g.y0 + g.dy * y, fz = g.z0 + g.dz * g.zmid;
    const double r2 = fx * fx + fy * fy + fz * fz;
    sw += rho;
    swr += rho * sqrt(r2);
    swr2 += rho * r2;
  }
  // The block's sums: eight threads a field, 16 values each (a shuffle tree over
  // every field costs five times the FP64 additions, 22 us of the kernel)
  static_assert(RED_FIELDS * 8 == RED_THREADS, "eight threads a field");
  __shared__ double sh[RED_FIELDS][RED_THREADS + 2];
  const int t = threadIdx.x;
  sh[RED_MASS][t] = m_w.x();
  sh[RED_MAX][t] = best_hi < 0.f ? -1.0 : (double)best_hi + (double)best_lo;
  sh[RED_ARG][t] = (double)best_i;
  sh[RED_MX][t] = mxy.x();
  sh[RED_MY][t] = mxy.y();
  sh[RED_MZ][t] = mz_k.x();
  sh[RED_W][t] = m_w.y();
  sh[RED_K][t] = mz_k.y();
  sh[RED_Q][t] = q_pz.x();
  sh[RED_PX][t] = pxy.x();
  sh[RED_PY][t] = pxy.y();
  sh[RED_PZ][t] = q_pz.y();
  sh[RED_PHIMAX][t] = (double)phimax;
  sh[RED_SW][t] = sw;
  sh[RED_SWR][t] = swr;
  sh[RED_SWR2][t] = swr2;
  __syncthreads();
  const int q = t >> 3, part = t & 7;
  RedTake r(q, sh[q][part], sh[RED_ARG][part]);
  for (int k = part + 8; k < RED_THREADS; k += 8) r.take(sh[q][k], sh[RED_ARG][k]);
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) {
    const double u = __shfl_down_sync(0xffffffffu, r.v, off, 8), ua = __shfl_down_sync(0xffffffffu, r.arg, off, 8);
    r.take(u, ua);
  }
  if (part == 0) r.store(partials + ((long long)blockIdx.y * gridDim.x + blockIdx.x) * RED_FIELDS);
}

// The items' fields from their block partials: one warp, in a block of its own, per
// field and item (FP64 runs at one a cycle and SM: 18 us with all fields on one SM).
__global__ void __launch_bounds__(32)
k_reduce_final(const double* __restrict__ partials, int nblocks, double* __restrict__ fields) {
  const int lane = threadIdx.x, q = blockIdx.x;
  if (q == RED_ARG) return;  // comes with RED_MAX
  const double* o = partials + (long long)blockIdx.y * nblocks * RED_FIELDS;
  RedTake r(q, q == RED_MAX ? -1.0 : 0.0, 0.0);
  constexpr int U = 8;
  for (int k0 = lane; k0 < nblocks; k0 += 32 * U) {
    double u[U], ua[U];  // loads first: their latency is what the kernel takes
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int k = k0 + 32 * j;
      u[j] = k < nblocks ? o[k * RED_FIELDS + q] : q == RED_MAX ? -1.0 : 0.0;
      ua[j] = k < nblocks ? o[k * RED_FIELDS + RED_ARG] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < U; ++j)
      if (k0 + 32 * j < nblocks) r.take(u[j], ua[j]);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double u = __shfl_down_sync(0xffffffffu, r.v, off), ua = __shfl_down_sync(0xffffffffu, r.arg, off);
    r.take(u, ua);
  }
  if (lane == 0) r.store(fields + blockIdx.y * RED_FIELDS);
}

cudaError_t launch_reduce(const float2* psi, const float* phi, const RedGeom& g, double* partials, int nblocks,
                          int batch, double* fields, cudaStream_t st) {
  k_reduce<<<dim3(nblocks, batch), RED_THREADS, 0, st>>>(psi, phi, g, red_depth(g, nblocks), partials);
  k_reduce_final<<<dim3(RED_FIELDS, batch), 32, 0, st>>>(partials, nblocks, fields);
  return cudaGetLastError();
}

// ----------------------------------------------------------------------------
// Lagrangian radii: the weighted quantiles of src/simulation_main.jl:641-650 of
// the distance from the density maximum, on the device from the histogram to the
// few numbers the quantiles need (RadiiOut): fetching the histogram and summing it
// on the host took 0.3 ms of a 256^3 snapshot, beside 0.27 ms of kernels (now 0.1).
// ----------------------------------------------------------------------------
struct Centre {
  int x, y, z;
  __device__ Centre(const double* fields, int nx, int ny) {
    const long long arg = (long long)fields[RED_ARG];
    z = (int)(arg / ((long long)nx * ny));
    const int rem = (int)(arg - (long long)z * nx * ny);
    y = rem / nx;
    x = rem - y * nx;
  }
};

// Weights of the distances from the density maximum, keyed by the squared
// distance in cells.  A thread takes one offset (a, b, c) >= 0 and sums the up to
// eight cells at (cx +- a, cy +- b, cz +- c) inside the grid, which share the key
// a^2 + b^2 + c^2, so a centred halo needs one atomic add per eight cells.
//
// FP64 runs at one operation a cycle and SM, so two FP64 FMAs per cell took 145 us
// at 256^3 (now 56).  The eight cells are summed in three FP32 words instead: squares as
// exact pairs, every rounding of the leading sums kept by two-sums, roundings of
// the third word alone lost (2^-70 of the sum), one rounding into FP64 at the end.
// The squares' low words are exact for components from 2^-50 to 2^60 (and zero);
// threads that meet another one sum in FP64.
struct Sum3 {
  float h = 0.f, m = 0.f, l = 0.f;
  static __device__ __forceinline__ float two_sum(float& a, float b) {  // a += b, returns the rounding
    const float s = a + b, t = s - a;
    const float e = (a - (s - t)) + (b - t);
    a = s;
    return e;
  }
  __device__ __forceinline__ void add(float2 p) {
    float s = __fmul_rn(p.x, p.x), e = fmaf(p.x, p.x, -s);
    const float b = __fmul_rn(p.y, p.y), eb = fmaf(p.y, p.y, -b);
    const float e1 = two_sum(s, b), e2 = two_sum(e, eb);
    const float e3 = two_sum(h, s);
    l += ((two_sum(m, e3) + two_sum(m, e1)) + two_sum(m, e)) + e2;
  }
  __device__ __forceinline__ double value() const { return (double)h + ((double)m + (double)l); }
};

__global__ void __launch_bounds__(256)
k_radii_hist(const float2* __restrict__ psi, int nx, int ny, int nz, const double* __restrict__ fields,
             double* __restrict__ wsum) {
  const Centre o(fields, nx, ny);
  const unsigned da = max(o.x, nx - 1 - o.x) + 1, db = max(o.y, ny - 1 - o.y) + 1, dc = max(o.z, nz - 1 - o.z) + 1;
  const unsigned total = da * db * dc;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    const unsigned bc = t / da;
    const int a = (int)(t - bc * da), c = (int)(bc / db), b = (int)(bc - c * db);
    float2 p[8];
    bool exact = true;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int zz = k & 4 ? o.z - c : o.z + c, yy = k & 2 ? o.y - b : o.y + b, xx = k & 1 ? o.x - a : o.x + a;
      const bool in = zz >= 0 && zz < nz && !(k & 4 && !c) && yy >= 0 && yy < ny && !(k & 2 && !b) && xx >= 0 &&
                      xx < nx && !(k & 1 && !a);
      p[k] = in ? psi[((long long)zz * ny + yy) * nx + xx] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float u = fabsf(p[k].x), v = fabsf(p[k].y);
      exact = exact && (u == 0.f || (u >= 0x1p-50f && u < 0x1p60f)) && (v == 0.f || (v >= 0x1p-50f && v < 0x1p60f));
    }
    double s = 0.0;
    if (exact) {
      Sum3 w;
#pragma unroll
      for (int k = 0; k < 8; ++k) w.add(p[k]);
      if (w.h > 0.f) s = w.value();
    } else {
      for (int k = 0; k < 8; ++k) s = fma((double)p[k].x, (double)p[k].x, fma((double)p[k].y, (double)p[k].y, s));
    }
    if (s > 0.0) atomicAdd(&wsum[a * a + b * b + c * c], s);
  }
}

// Per block of RADII_BLOCK keys: the sum of their weights and the last key with
// weight (-1: none).
constexpr int RADII_BLOCK = 1024;
__global__ void __launch_bounds__(256)
k_radii_blocks(const double* __restrict__ wsum, int nkeys, double* __restrict__ bsum, int* __restrict__ blast) {
  const int base = blockIdx.x * RADII_BLOCK;
  double s = 0.0;
  int last = -1;
#pragma unroll
  for (int k = 0; k < RADII_BLOCK / 256; ++k) {
    const int key = base + k * 256 + threadIdx.x;
    const double w = key < nkeys ? wsum[key] : 0.0;
    s += w;
    if (w > 0.0) last = key;
  }
  __shared__ double ss[8];
  __shared__ int sl[8];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, off);
    last = max(last, __shfl_down_sync(0xffffffffu, last, off));
  }
  if ((threadIdx.x & 31) == 0) {
    ss[threadIdx.x >> 5] = s;
    sl[threadIdx.x >> 5] = last;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; ++k) {
      s += ss[k];
      last = max(last, sl[k]);
    }
    bsum[blockIdx.x] = s;
    blast[blockIdx.x] = last;
  }
}

// Inclusive sums over a block of RADII_BLOCK = 32 x 32 threads: one warp adds 32
// values a lane (a scan by shuffles in every warp does 5 FP64 additions a value,
// at one a cycle: 15 us for the kernel).  `sh`: 33 x 32 + 32 words.
__device__ double radii_scan(double v, double* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double* off = sh + 33 * 32;
  __syncthreads();  // sh may still be read from the scan before
  sh[33 * w + lane] = v;
  __syncthreads();
  if (w == 0) {
    double s = 0.0;
#pragma unroll 8
    for (int k = 0; k < 32; ++k) sh[33 * lane + k] = s += sh[33 * lane + k];
    double t = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const double u = __shfl_up_sync(0xffffffffu, t, d);
      if (lane >= d) t += u;
    }
    off[lane] = t;
  }
  __syncthreads();
  return w ? sh[33 * w + lane] + off[w - 1] : sh[lane];
}

// The groups the quantiles fall in, one block a quantile: h = p (S - w_1) + w_1
// (w_1: the weight at distance 0), the first key whose cumulative weight exceeds h,
// the cumulative weight and the key with weight before it.
__global__ void __launch_bounds__(RADII_BLOCK)
k_radii_find(const double* __restrict__ wsum, int nkeys, const double* __restrict__ bsum,
             const int* __restrict__ blast, int nblocks, RadiiOut* __restrict__ out) {
  __shared__ double scan[33 * 32 + 32], before;
  __shared__ int last[RADII_BLOCK], block, first, prev;
  const int t = threadIdx.x, q = blockIdx.x;
  const double w1 = wsum[0];
  const double own = t < nblocks ? bsum[t] : 0.0;
  last[t] = t < nblocks ? blast[t] : -1;
  if (t == 0) {
    block = nblocks;
    first = RADII_BLOCK;
    prev = -1;
  }
  const double incl = radii_scan(own, scan);
  const double total = scan[33 * 32 + 31];
  const double h = radii_p(q) * (total - w1) + w1;
  if (own > 0.0 && incl > h) atomicMin(&block, t);
  __syncthreads();
  const int blk = block;
  if (t == 0) {
    out->wmin[q] = ~0ull;
    if (q == 0) {
      int k = nblocks - 1;
      while (k >= 0 && last[k] < 0) --k;
      out->last = k >= 0 ? last[k] : -1;
      out->total = total;
      out->w1 = w1;
    }
    if (blk == nblocks) out->key[q] = -1;
  }
  if (blk == nblocks) return;
  if (t == blk) before = incl - own;
  const int key = blk * RADII_BLOCK + t;
  const double w = key < nkeys ? wsum[key] : 0.0;
  const double in_block = radii_scan(w, scan);
  const double cum = before + in_block;
  // the block's sum and the cumulative sum round differently: with no key past h its last one is meant
  if (w > 0.0 && (cum > h || key == last[blk])) atomicMin(&first, t);
  __syncthreads();
  if (w > 0.0 && t < first) atomicMax(&prev, t);
  __syncthreads();
  if (t == first) {
    int k = blk - 1;
    while (k >= 0 && last[k] < 0) --k;
    out->key[q] = key;
    out->prev[q] = prev >= 0 ? blk * RADII_BLOCK + prev : k >= 0 ? last[k] : -1;
    out->before[q] = cum - w;
  }
}

// Smallest nonzero weight (bits of a positive double) among the cells of each
// group the quantiles fall in: a row (y, z) holds at most the two cells cx +- r of
// a key, r^2 = key - dy^2 - dz^2.
__global__ void __launch_bounds__(256)
k_radii_min(const float2* __restrict__ psi, int nx, int ny, int nz, const double* __restrict__ fields,
            RadiiOut* __restrict__ out) {
  const Centre o(fields, nx, ny);
  const int nrows = ny * nz;
  int key[RADII_QUANTILES];
#pragma unroll
  for (int q = 0; q < RADII_QUANTILES; ++q) key[q] = out->key[q];
  for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < nrows; row += gridDim.x * blockDim.x) {
    const int z = row / ny, y = row - z * ny;
    const int d = (y - o.y) * (y - o.y) + (z - o.z) * (z - o.z);
#pragma unroll
    for (int q = 0; q < RADII_QUANTILES; ++q) {
      const int rem = key[q] - d;
      if (rem < 0) continue;
      int r = (int)sqrtf((float)rem);
      while (r * r > rem) --r;
      while ((r + 1) * (r + 1) <= rem) ++r;
      if (r * r != rem) continue;
      for (int side = 0; side < (r ? 2 : 1); ++side) {
        const int x = side ? o.x - r : o.x + r;
        if (x < 0 || x >= nx) continue;
        const float2 p = psi[(long long)row * nx + x];
        const double rho = (double)p.x * p.x + (double)p.y * p.y;
        if (rho > 0.0) atomicMin(&out->wmin[q], (unsigned long long)__double_as_longlong(rho));
      }
    }
  }
}

int radii_blocks(long long nkeys) { return (int)((nkeys + RADII_BLOCK - 1) / RADII_BLOCK); }

cudaError_t launch_radii(const float2* psi, int nx, int ny, int nz, const double* fields, double* wsum, long long nkeys,
                         double* bsum, int* blast, RadiiOut* out, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(wsum, 0, sizeof(double) * nkeys, st);
  if (e != cudaSuccess) return e;
  const long long cells = (long long)nx * ny * nz;
  const long long want = (cells + 255) / 256;  // the centre is known on the device only
  k_radii_hist<<<(unsigned)(want < 152 * 8 ? want : 152 * 8), 256, 0, st>>>(psi, nx, ny, nz, fields, wsum);
  const int nb = radii_blocks(nkeys);
  k_radii_blocks<<<nb, 256, 0, st>>>(wsum, (int)nkeys, bsum, blast);
  k_radii_find<<<RADII_QUANTILES, RADII_BLOCK, 0, st>>>(wsum, (int)nkeys, bsum, blast, nb, out);
  const int rows = (ny * nz + 255) / 256;
  k_radii_min<<<rows < 152 * 4 ? rows : 152 * 4, 256, 0, st>>>(psi, nx, ny, nz, fields, out);
  return cudaGetLastError();
}

__device__ __forceinline__ long long cic_cell(int ix, int iy, int iz, int nx, int ny, int nz) {
  ix = ix >= nx ? ix - nx : ix;
  iy = iy >= ny ? iy - ny : iy;
  iz = iz >= nz ? iz - nz : iz;
  return ((long long)iz * ny + iy) * nx + ix;
}

// rows (ny * nz flags, may be null): set to 1 for every x row a particle touches
__global__ void k_cic_deposit(float* __restrict__ rho, const CicParticle* __restrict__ p, long long n, int nx, int ny,
                              int nz, int* __restrict__ rows) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= n) return;
  const CicParticle a = p[q];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int ox = c & 1, oy = (c >> 1) & 1, oz = c >> 2;
    const float w = (ox ? a.f[0] : 1.f - a.f[0]) * (oy ? a.f[1] : 1.f - a.f[1]) * (oz ? a.f[2] : 1.f - a.f[2]);
    const long long cell = cic_cell(a.i[0] + ox, a.i[1] + oy, a.i[2] + oz, nx, ny, nz);
    atomicAdd(rho + cell, a.m * w);
    if (rows && c % 2 == 0) rows[cell / nx] = 1;
  }
}

__global__ void k_cic_interp(const float* __restrict__ f, const CicParticle* __restrict__ p, long long n, int nx,
                             int ny, int nz, double* __restrict__ out) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= n) return;
  const CicParticle a = p[q];
  double s = 0.0;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int ox = c & 1, oy = (c >> 1) & 1, oz = c >> 2;
    const double w = (double)(ox ? a.f[0] : 1.f - a.f[0]) * (oy ? a.f[1] : 1.f - a.f[1]) * (oz ? a.f[2] : 1.f - a.f[2]);
    s += w * f[cic_cell(a.i[0] + ox, a.i[1] + oy, a.i[2] + oz, nx, ny, nz)];
  }
  out[q] = s;
}

cudaError_t launch_cic_deposit(float* rho, const CicParticle* p, long long n, int nx, int ny, int nz, int* rows,
                               cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_cic_deposit<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(rho, p, n, nx, ny, nz, rows);
  return cudaGetLastError();
}

cudaError_t launch_cic_interp(const float* field, const CicParticle* p, long long n, int nx, int ny, int nz,
                              double* out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_cic_interp<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(field, p, n, nx, ny, nz, out);
  return cudaGetLastError();
}

}  // namespace wdm

namespace wdm {

// Mean of |psi|^2 (complex input) or of a float field, per batch item, as a
// float shift: FP64 block partial sums, FP64 atomics into sums[b] (zeroed by
// the launcher), then shift[b] = sums[b] / n + add.
// COPY: the values also go to `copy` (a new psi is stored and summed in one pass:
// set_psi of 256^3 91 -> 67 us).
template <bool COMPLEX, bool COPY>
__global__ void k_block_sum(const void* data, long long n, double* __restrict__ sums, float2* copy) {
  // per-thread FP32 partial sums (the shift only needs to be near the mean:
  // any value is exact), FP64 from the warp reduction on
  // eight loads in flight per thread (one at a time left DRAM at half its rate:
  // 256^3 38 us), added in the order of a plain loop
  using T = std::conditional_t<COMPLEX, float2, float>;
  constexpr int U = 8;
  const T* p = static_cast<const T*>(data) + blockIdx.y * n;
  const long long step = (long long)gridDim.x * blockDim.x;
  float accf = 0.f;
  auto add = [&](T v) {
    if constexpr (COMPLEX) accf = fmaf(v.x, v.x, fmaf(v.y, v.y, accf));
    else accf += v;
  };
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += U * step) {
    T v[U];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (i + k * step < n) v[k] = p[i + k * step];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (i + k * step < n) {
        add(v[k]);
        if constexpr (COPY) copy[blockIdx.y * n + i + k * step] = v[k];
      }
  }
  double acc = accf;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  __shared__ double sh[32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
    atomicAdd(sums + blockIdx.y, s);
  }
}

__global__ void k_finalize_shift(const double* __restrict__ sums, float* __restrict__ shift, int batch, double inv_n,
                                 double add) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < batch) shift[b] = (float)(sums[b] * inv_n + add);
}

cudaError_t launch_mean_shift(const void* data, bool complex_in, long long n, int batch, double* sums, float* shift,
                              double add, cudaStream_t st, float2* copy) {
  cudaError_t e = cudaMemsetAsync(sums, 0, sizeof(double) * batch, st);
  if (e != cudaSuccess) return e;
  long long blocks = (n + 255) / 256;
  if (blocks > 304) blocks = 304;
  const dim3 grid((unsigned)blocks, batch);
  if (copy) k_block_sum<true, true><<<grid, 256, 0, st>>>(data, n, sums, copy);
  else if (complex_in) k_block_sum<true, false><<<grid, 256, 0, st>>>(data, n, sums, nullptr);
  else k_block_sum<false, false><<<grid, 256, 0, st>>>(data, n, sums, nullptr);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  k_finalize_shift<<<(batch + 127) / 128, 128, 0, st>>>(sums, shift, batch, 1.0 / (double)n, add);
  return cudaGetLastError();
}

}  // namespace wdm
