// The z stage of the all-periodic Poisson solve as cyclic tridiagonal line
// solves (big_periodic_3D.f90:526-548 solves the whole problem with a 3D r2c
// FFT; this stage replaces its z FFT, 1/lambda and z IFFT).
//
// After the x and y transforms every spectrum line along z, mode (kx, ky), is
// the periodic system
//   p[j-1] - c p[j] + p[j+1] = rs R[j],  c = 2 + sigma, sigma = -h_z^2 (lambda_x + lambda_y),
// indices mod nz, rs = h_z^2 * scale * nz (the z FFT pair it replaces was
// unnormalised).  With rho the root below 1 of rho + 1/rho = c the operator is
// -(1 - rho S)(1 - rho S^-1) / rho, S the shift by one, so the solution is two
// first-order cyclic recursions,
//   y[j] = -rho rs R[j] + rho y[j-1],  p[j] = y[j] + rho p[j+1],
// with constants of the mode: rho = exp(-theta), theta = 2 asinh(sqrt(sigma) / 2).
// (theta keeps the digits of a small sigma that c = 2 + sigma rounds away.)
//
// A line is cut into segments of 16 unknowns (8 on small boxes), one thread
// each, held in registers: a segment's recursion from zero gives its end value, the end
// values e of the segments give the value that enters each,
//   sum_{m>=1} q^(m-1) e[s-m] / (1 - q^T),  q = rho^16 (rho^8), T segments,
// and the recursion runs again from it.  One read and one write of the
// spectrum, 10 FP64 instructions a complex unknown (the Thomas walk over
// tabulated factors that it replaces: the same, one thread a line, 24 bytes of
// tables an unknown).  A step's solve takes 10 us at 32^3 (the walk 23), 12 at
// 64^3 (42), 33 at 128^3 (79) and 182 at 256^3 (187), with the FP64 unit
// 82% busy at 128^3.
//
// The mode (0, 0) is singular (rho = 1): the FFT solve drops its mean
// (lambda(0) = +Inf), i.e. gives the zero-mean solution of the system with
// the right-hand side's mean removed.  Here the two recursions are prefix
// sums, with the mean of their input removed before each and the result's
// after, by a warp of its own.
#include "ns_internal.cuh"
#include "ns_kernels.cuh"

namespace ns {

namespace {

__global__ void __launch_bounds__(128) cyc_table_kernel(FftPlan P, double2* __restrict__ tab,
                                                        double* __restrict__ half) {
  const int S = P.nxh * P.ny, t = blockIdx.x * 128 + threadIdx.x;
  if (t >= S) return;
  cyc_mode(-P.cyc_h2 * (P.eig_x[t % P.nxh] + P.eig_o[t / P.nxh]), P.nz, P.cyc_rs, tab[2 * t], tab[2 * t + 1], half[t]);
}

// Lines per CTA: 128 threads, 256 for the long lines.
template <int N, int CYC_L>
constexpr int cyc_lines() { return (N / CYC_L >= 16 ? 256 : 128) * CYC_L / N; }

// The singular line by a warp, lane l the unknowns [l E, l E + E): the mean of
// the right-hand side removed, a prefix sum, its mean removed, a suffix sum,
// its mean removed.
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int N>
__device__ __forceinline__ void cyc_singular(double2* __restrict__ spec, int S, double sc, int lane) {
  constexpr int E = N >= 32 ? N / 32 : 1;
  const bool in = lane * E < N;
  double* g = reinterpret_cast<double*>(spec + (long long)(lane * E) * S);
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    double r[E];
#pragma unroll
    for (int j = 0; j < E; ++j) r[j] = in ? sc * g[2LL * j * S + part] : 0.0;
    auto remove_mean = [&]() {
      double m = 0.0;
#pragma unroll
      for (int j = 0; j < E; ++j) m += r[j];
      m = warp_sum(m) / N;
      if (in)
#pragma unroll
        for (int j = 0; j < E; ++j) r[j] -= m;
    };
    remove_mean();
#pragma unroll
    for (int j = 1; j < E; ++j) r[j] += r[j - 1];
    double run = r[E - 1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double q = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += q;
    }
    double before = __shfl_up_sync(0xffffffffu, run, 1);
    if (lane == 0) before = 0.0;
    if (in)
#pragma unroll
      for (int j = 0; j < E; ++j) r[j] += before;
    remove_mean();
#pragma unroll
    for (int j = E - 2; j >= 0; --j) r[j] += r[j + 1];
    run = r[0];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double q = __shfl_down_sync(0xffffffffu, run, o);
      if (lane + o < 32) run += q;
    }
    before = __shfl_down_sync(0xffffffffu, run, 1);
    if (lane == 31) before = 0.0;
    if (in)
#pragma unroll
      for (int j = 0; j < E; ++j) r[j] += before;
    remove_mean();
    if (in)
#pragma unroll
      for (int j = 0; j < E; ++j) g[2LL * j * S + part] = r[j];
  }
}

template <int N, int CYC_L>
__global__ void __launch_bounds__(cyc_lines<N, CYC_L>() * N / CYC_L) cyc_solve_kernel(FftPlan P, double2* __restrict__ spec,
                                                                                      FOne one) {
  constexpr int T = N / CYC_L, LPC = cyc_lines<N, CYC_L>();
  __shared__ double2 end[T][LPC];
  const int S = P.nxh * P.ny, l = threadIdx.x, s = threadIdx.y;
  const int t = blockIdx.x * LPC + l;
  if (blockIdx.x == gridDim.x - 1) {  // one more CTA for the singular line
    if (s * LPC + l < 32) cyc_singular<N>(spec, S, -P.cyc_rs, s * LPC + l);
    return;
  }
  const bool valid = t < S && t > 0;
  double2* g = spec + t + (long long)(s * CYC_L) * S;
  const double2 ca = valid ? __ldg(P.cyc_t + 2 * t) : make_double2(0.0, 0.0);      // rho, q
  const double2 cb = valid ? __ldg(P.cyc_t + 2 * t + 1) : make_double2(0.0, 0.0);  // 1 / (1 - q^T), -rho rs
  const double rho = ca.x, inv = cb.x, qs = CYC_L == 16 ? ca.y : __ldg(P.cyc_h + (valid ? t : 0));
  double2 r[CYC_L];
#pragma unroll
  for (int j = 0; j < CYC_L; ++j) r[j] = valid ? g[(long long)j * S] : make_double2(0.0, 0.0);
#pragma unroll
  for (int j = 0; j < CYC_L; ++j) {
    r[j].x = fmul(one, r[j].x, cb.y);
    r[j].y = fmul(one, r[j].y, cb.y);
  }
  // The value that enters this segment from the side dir (-1: from below), from the end values of all.
  auto enter = [&](int dir) -> double2 {
    double2 c = make_double2(0.0, 0.0);
    double pw = inv;
    for (int m = 1; m <= T; ++m) {
      const double2 e = end[(s + dir * m + T) & (T - 1)][l];
      c.x = fma(pw, e.x, c.x);
      c.y = fma(pw, e.y, c.y);
      pw *= qs;
      if (!__any_sync(0xffffffffu, pw > 0x1p-66)) break;
    }
    return c;
  };
  double2 y = make_double2(0.0, 0.0);
#pragma unroll
  for (int j = 0; j < CYC_L; ++j) y = make_double2(fma(rho, y.x, r[j].x), fma(rho, y.y, r[j].y));
  end[s][l] = y;
  __syncthreads();
  y = enter(-1);
#pragma unroll
  for (int j = 0; j < CYC_L; ++j) {
    y = make_double2(fma(rho, y.x, r[j].x), fma(rho, y.y, r[j].y));
    r[j] = y;
  }
  y = make_double2(0.0, 0.0);
#pragma unroll
  for (int j = CYC_L - 1; j >= 0; --j) y = make_double2(fma(rho, y.x, r[j].x), fma(rho, y.y, r[j].y));
  __syncthreads();
  end[s][l] = y;
  __syncthreads();
  y = enter(1);
#pragma unroll
  for (int j = CYC_L - 1; j >= 0; --j) {
    y = make_double2(fma(rho, y.x, r[j].x), fma(rho, y.y, r[j].y));
    r[j] = y;
  }
  if (valid) {
#pragma unroll
    for (int j = 0; j < CYC_L; ++j) g[(long long)j * S] = r[j];
  }
}

}  // namespace

size_t cyc_table_doubles(const FftPlan& P) { return 5 * (size_t)P.nxh * P.ny; }

cudaError_t launch_cyc_table(FftPlan& P, double* buf, cudaStream_t st) {
  const int S = P.nxh * P.ny;
  P.cyc_t = reinterpret_cast<double2*>(buf);
  P.cyc_h = buf + 4 * (size_t)S;
  cyc_table_kernel<<<(S + 127) / 128, 128, 0, st>>>(P, reinterpret_cast<double2*>(buf), buf + 4 * (size_t)S);
  return cudaGetLastError();
}

cudaError_t launch_cyc_z_solve(const FftPlan& P, double2* spec, cudaStream_t st) {
  const int S = P.nxh * P.ny;
  // segments of 8 where segments of 16 would leave less than two warps per SM partition (at 32^3
  // the solve takes 10 us against 14, at 128^3 the longer segments take 33 against 39)
  const bool half = (long long)S * P.nz / 16 < 2 * 608 * 32;
#define NS_CYC_RUN(N, L)                                                                                \
  cyc_solve_kernel<N, L><<<(S + cyc_lines<N, L>() - 1) / cyc_lines<N, L>() + 1, dim3(cyc_lines<N, L>(), N / L), 0, st>>>( \
      P, spec, FOne{1.0, -0.0})
#define NS_CYC_CASE(N)             \
  case N:                          \
    if (half) NS_CYC_RUN(N, 8);    \
    else NS_CYC_RUN(N, 16);        \
    break;
  switch (P.nz) {
    NS_CYC_CASE(16) NS_CYC_CASE(32) NS_CYC_CASE(64) NS_CYC_CASE(128) NS_CYC_CASE(256) NS_CYC_CASE(512)
    default: return cudaErrorInvalidValue;
  }
#undef NS_CYC_CASE
#undef NS_CYC_RUN
  return cudaGetLastError();
}

}  // namespace ns
