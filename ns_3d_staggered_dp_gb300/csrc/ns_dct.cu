// Wall-bounded pressure Poisson solve: the per-axis trigonometric transforms
// of DCT_poisson_solver (NS_functions.f90:1505-1630) and their mix with the
// periodic FFT axes.
//
// A non-periodic axis of N cells is transformed with an exact N x N matrix
// pair (forward F, inverse G = F^-1), built on the host from the MKL
// trigonometric-transform definitions the reference uses:
//   pbc 3 (Neumann on the wall)    : F = DCT-II  (MKL backward staggered cosine)
//   pbc 2 (Dirichlet on the wall)  : flip the sign of every other input,
//                                    DCT-II, reverse the output (= DST-II)
//   pbc 4 (Dirichlet on the ghost) : F = DST-I of N points
// and applied to a line held in shared memory, on fixed-point integers.
// Any N works (the subdomain edges 24 and 48 included).
//
// Data flow: with x periodic the x pass is the r2c FFT of ns_fft.cu and the
// y/z passes act on the complex half spectrum (real and imaginary parts
// transform alike).  With every axis non-periodic the x pass applies F_x to
// the real divergence line and packs modes (2q, 2q+1) into one complex value,
// so the y/z passes again act on complex lines.  The wall axis that is
// transformed last is not transformed at all: its lines are solved as
// tridiagonal systems (tri_solve_kernel), which gives the same solution as
// transform, eigenvalue divide and inverse transform along that axis; with
// packed x modes the real and imaginary parts are two systems.
// The divergence kernels add the pressure-BC terms of
// pr_bc_staggered_modify_rhs (NS_functions.f90:1345-1400) on the first and
// last cells of every non-periodic axis.
#include <cmath>
#include <cstring>
#include <vector>

#include "ns_fft_core.cuh"
#include "ns_internal.cuh"
#include "ns_kernels.cuh"

namespace ns {

namespace {

// Divergence of u*, v*, w* over dt at cell (i, j, k), plus the pressure-BC
// terms of the boundary cells; a given right-hand side is taken as it is
// (already BC-modified).
__device__ __forceinline__ double rhs_cell(const DivArgs& d, const SpecPlan& S, const FOne& c, int i, int j, int k) {
  const Layout& L = d.L;
  const long long g = L.at(i, j, k);
  if (d.rhs) return d.rhs[g];
  double r = fmul(c, fsub(c, d.us[g + 1], d.us[g]), d.cdx);
  r = fma(fsub(c, d.vs[g + L.sy], d.vs[g]), d.cdy, r);
  r = fma(fsub(c, d.ws[g + L.sz], d.ws[g]), d.cdz, r);
  return r + S.bc_term(i, j, k);
}

}  // namespace

// ---------------------------------------------------------------------------
// Dense transforms on block fixed-point integers (ns_fixed.cuh): a line
// becomes integers of one exponent, a matrix entry an integer in units of
// 2^-54 (times 2^-gexp for the inverse), both split at bit 27, so that a
// product and sum is three 32-bit multiply-adds into two 64-bit sums: 14
// integer issue clocks against the 64 of an FP64 FMA.  The entries' low parts
// are signed, so the dropped products of the low parts have mean 0.
// For codes 2, 3 and 4 and any N, F[k][N-1-n] = (-1)^k F[k][n] and
// G[N-1-n][k] = (-1)^k G[n][k], so each pass sums half the products: forward,
// an even mode takes s[n] = x[n] + x[N-1-n], an odd one d[n] = x[n] - x[N-1-n]
// (s kept at n, the middle sample of an odd N with it, d at N-1-n); inverse,
// the even and odd modes' sums E and O give E + O at n and E - O at N-1-n.
// ---------------------------------------------------------------------------
constexpr int DX_SEG = 128;  // terms per 64-bit partial sum

struct DxSum {
  long long hi = 0, mid = 0;
  __device__ __forceinline__ void add(int vh, int vl, int2 w) {
    hi = fx_wide(vh, w.x, hi);
    mid = fx_wide(vl, w.x, fx_wide(vh, w.y, mid));
  }
  __device__ __forceinline__ void fold() {
    hi += (mid + (1ll << 26)) >> 27;
    mid = 0;
  }
};
// A line whose largest biased exponent is E and whose magnitudes sum to less
// than 2^lb of its unit 2^(E+1): the exponent to convert at, so that a value
// takes at most `most` bits and any sum of products at most 62, the unit's
// exponent eb, and the power of two that brings extreme lines into range
// first (scaled).  (The sum of the magnitudes, not their number times the
// largest: a line with few large values keeps more bits.)
struct DxExp {
  int ec, eb;
  bool scaled, up;
};
__device__ __forceinline__ DxExp dx_exp(int E, int lb, int most) {
  DxExp x;
  x.scaled = E < 128 || E > 1900;
  x.up = E < 128;
  const int adj = x.scaled ? (x.up ? 512 : -512) : 0;
  x.ec = max(E + adj + (E == 0 ? 1 : 0), 64) + (58 - min(most, 62 - lb));
  x.eb = E == 0x7ff ? kFxNonfinite : x.ec - 1022 - 58 - adj;
  return x;
}
// A value's share of the sum, in units of 2^(E+1-20), rounded up; its lb.
__device__ __forceinline__ unsigned dx_share(int E, unsigned hi2) {
  return ((1u << 20) >> min(E - (int)(hi2 >> 21), 31)) + 1u;
}
__device__ __forceinline__ int dx_sum_bits(unsigned sum) { return 32 - __clz((int)sum) - 20; }
__device__ __forceinline__ long long dx_from(double d, const DxExp& x) {
  if (x.scaled) d *= x.up ? 0x1p512 : 0x1p-512;
  return fx_round<58>(d, x.ec);
}
__device__ __forceinline__ int2 dx_split(long long v) { return make_int2((int)(v >> 27), (int)v & ((1 << 27) - 1)); }
__device__ __forceinline__ int dx_biased(unsigned hi2) { return (int)(hi2 >> 21); }  // of 2 |high word|

// x pass for a non-periodic x axis: real line -> F_x -> packed modes.  A
// group of G lanes takes a line (128/G lines per CTA, several short lines
// share a warp); lane q computes the modes 2q and 2q+1.
__device__ __forceinline__ void dense_x_fwd_body(const SpecPlan& S, const DivArgs& d, double2* __restrict__ spec,
                                                 double* xs, int bx) {
  const int G = dense_x_group(S.nx);
  const int grp = threadIdx.x / G, gl = threadIdx.x % G;
  const int line = bx * (128 / G) + grp;
  const int nx = S.nx, ny = S.ny, nz = S.nz, H = nx / 2;
  const bool valid = line < ny * nz;
  const int j = valid ? 1 + line % ny : 1, k = valid ? 1 + line / ny : 1;
  double* r = xs + grp * nx;
  int2* v = reinterpret_cast<int2*>(r);
  const FOne c{d.one, d.mzero};
  unsigned m = 0;
  for (int i = gl; i < nx; i += G) {
    const double x = valid ? rhs_cell(d, S, c, i + 1, j, k) : 0.0;
    m = max(m, (unsigned)__double2hiint(x) << 1);
    r[i] = x;
  }
  for (int o = G / 2; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  const int E = dx_biased(m);
  unsigned sum = 0;
  for (int i = gl; i < nx; i += G) sum += dx_share(E, (unsigned)__double2hiint(r[i]) << 1);
  for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const DxExp e = dx_exp(E, dx_sum_bits(sum), 57);  // a bit for the fold
  __syncwarp();
  for (int n = gl; n < H; n += G) {
    const long long a = dx_from(r[n], e), b = dx_from(r[nx - 1 - n], e);
    v[n] = dx_split(a + b);
    v[nx - 1 - n] = dx_split(a - b);
  }
  __syncwarp();
  if (!valid) return;
  const int2* __restrict__ FT = S.fwd[0];  // F^T: FT[n * N + kk] = F[kk][n]
  double2* out = spec + (long long)S.nxs * ((j - 1) + (long long)ny * (k - 1));
  const FxOut fo = fx_out(e.eb);
  for (int q = gl; q < H; q += G) {
    DxSum a, b;
    for (int n0 = 0; n0 < H; n0 += DX_SEG) {
      const int n1 = min(H, n0 + DX_SEG);
#pragma unroll 4
      for (int n = n0; n < n1; ++n) {
        const int4 f = __ldg(reinterpret_cast<const int4*>(FT + (long long)n * nx + 2 * q));
        const int2 s = v[n], t = v[nx - 1 - n];
        a.add(s.x, s.y, make_int2(f.x, f.y));
        b.add(t.x, t.y, make_int2(f.z, f.w));
      }
      a.fold();
      b.fold();
    }
    double2 y = fx_to(i2{a.hi, b.hi}, fo, c);
    if (fo.odd) fx_rescale(y, fo);
    out[q] = y;
  }
}

// x inverse for a non-periodic x axis: packed modes -> G_x -> dp slots 1..nx.
__device__ __forceinline__ void dense_x_inv_body(const SpecPlan& S, const double2* __restrict__ spec, double* dp,
                                                 const Layout& L, double* xs, int bx, const FOne& c) {
  const int G = dense_x_group(S.nx);
  const int grp = threadIdx.x / G, gl = threadIdx.x % G;
  const int line = bx * (128 / G) + grp;
  const int nx = S.nx, ny = S.ny, nz = S.nz, H = nx / 2;
  const bool valid = line < ny * nz;
  const int j = valid ? 1 + line % ny : 1, k = valid ? 1 + line / ny : 1;
  double2* raw = reinterpret_cast<double2*>(xs + grp * nx);
  int4* v = reinterpret_cast<int4*>(raw);  // modes 2q, 2q+1
  const double2* in = spec + (long long)S.nxs * ((j - 1) + (long long)ny * (k - 1));
  unsigned m = 0;
  for (int q = gl; q < H; q += G) {
    const double2 x = valid ? in[q] : make_double2(0.0, 0.0);
    m = max(m, max((unsigned)__double2hiint(x.x) << 1, (unsigned)__double2hiint(x.y) << 1));
    raw[q] = x;
  }
  for (int o = G / 2; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  const int E = dx_biased(m);
  unsigned sum = 0;
  for (int q = gl; q < H; q += G)
    sum += dx_share(E, (unsigned)__double2hiint(raw[q].x) << 1) + dx_share(E, (unsigned)__double2hiint(raw[q].y) << 1);
  for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const DxExp e = dx_exp(E, dx_sum_bits(sum), 58);
  for (int q = gl; q < H; q += G) {  // each lane its own entries
    const int2 a = dx_split(dx_from(raw[q].x, e)), b = dx_split(dx_from(raw[q].y, e));
    v[q] = make_int4(a.x, a.y, b.x, b.y);
  }
  __syncwarp();
  if (!valid) return;
  const int2* __restrict__ GT = S.inv[0];  // G^T: GT[kk * N + n] = G[n][kk] (x = G X)
  double* o = dp + L.at(1, j, k);
  const FxOut fo = fx_out(e.eb >= kFxNonfinite / 2 ? e.eb : e.eb - S.gexp[0]);
  for (int n = gl; n < H; n += G) {
    DxSum ev, od;
    for (int q0 = 0; q0 < H; q0 += DX_SEG) {
      const int q1 = min(H, q0 + DX_SEG);
#pragma unroll 4
      for (int q = q0; q < q1; ++q) {
        const int4 x = v[q];
        ev.add(x.x, x.y, __ldg(GT + (long long)(2 * q) * nx + n));
        od.add(x.z, x.w, __ldg(GT + (long long)(2 * q + 1) * nx + n));
      }
      ev.fold();
      od.fold();
    }
    double2 y = fx_to(i2{ev.hi + od.hi, ev.hi - od.hi}, fo, c);
    if (fo.odd) fx_rescale(y, fo);
    o[n] = y.x;
    o[nx - 1 - n] = y.y;
  }
}

// Dense transform of complex lines along y (AXIS 1) or z (AXIS 2).  Lines are
// numbered t = col + nxs * o (o: z for y-lines, y for z-lines) and a CTA takes
// DX_LPC consecutive ones, so narrow spectra fill it too; neighbouring lanes
// read neighbouring columns (coalesced).  DX_T threads a line.
constexpr int DX_LPC = 8, DX_T = 16;
__host__ __device__ constexpr size_t dense_yz_smem(int n) {
  return (size_t)n * DX_LPC * sizeof(int4) + DX_LPC * DX_T * sizeof(unsigned);
}
template <int AXIS, bool FWD>
__device__ __forceinline__ void dense_yz_body(const SpecPlan& S, double2* __restrict__ spec, double2* ls, int bx,
                                              const FOne& c) {
  constexpr int LPC = DX_LPC, T = DX_T;
  const int l = threadIdx.x % LPC, t = threadIdx.x / LPC;
  const int N = (AXIS == 1) ? S.ny : S.nz;
  const int n_other = (AXIS == 1) ? S.nz : S.ny;
  const int tl = bx * LPC + l;
  const bool valid = tl < S.nxs * n_other;
  const int col = valid ? tl % S.nxs : 0;
  const int o = valid ? tl / S.nxs : 0;
  const long long st = (AXIS == 1) ? (long long)S.nxs : (long long)S.nxs * S.ny;
  const long long base = (AXIS == 1) ? col + (long long)S.nxs * S.ny * o : col + (long long)S.nxs * o;
  double2* raw = ls + l;  // element n at raw[n * LPC], then its integers at v[n * LPC]
  int4* v = reinterpret_cast<int4*>(ls) + l;
  unsigned* mx = reinterpret_cast<unsigned*>(ls + (long long)N * LPC);
  double2* g = spec + base;
  const int H = N / 2, He = (N + 1) / 2;  // pairs; terms of an even mode, rows of an inverse
  unsigned m = 0;
  for (int n = t; n < He; n += T) {  // both samples of a pair by one thread
    const double2 a = valid ? g[(long long)n * st] : make_double2(0.0, 0.0);
    const double2 b = valid ? g[(long long)(N - 1 - n) * st] : make_double2(0.0, 0.0);
    m = max(max(m, (unsigned)__double2hiint(a.x) << 1), (unsigned)__double2hiint(a.y) << 1);
    m = max(max(m, (unsigned)__double2hiint(b.x) << 1), (unsigned)__double2hiint(b.y) << 1);
    raw[n * LPC] = a;
    raw[(N - 1 - n) * LPC] = b;
  }
  mx[t * LPC + l] = m;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < T; ++q) m = max(m, mx[q * LPC + l]);
  const int E = dx_biased(m);
  unsigned sum = 0;
  for (int n = t; n < He; n += T) {  // of the larger component of each sample
    const double2 a = raw[n * LPC], b = raw[(N - 1 - n) * LPC];
    sum += dx_share(E, max((unsigned)__double2hiint(a.x) << 1, (unsigned)__double2hiint(a.y) << 1));
    if (n < H) sum += dx_share(E, max((unsigned)__double2hiint(b.x) << 1, (unsigned)__double2hiint(b.y) << 1));
  }
  __syncthreads();
  mx[t * LPC + l] = sum;
  __syncthreads();
  sum = 0;
#pragma unroll
  for (int q = 0; q < T; ++q) sum += mx[q * LPC + l];
  const DxExp e = dx_exp(E, dx_sum_bits(sum), FWD ? 57 : 58);  // a bit for the fold
  for (int n = t; n < He; n += T) {
    const double2 a = raw[n * LPC], b = raw[(N - 1 - n) * LPC];
    i2 p{dx_from(a.x, e), dx_from(a.y, e)}, q{dx_from(b.x, e), dx_from(b.y, e)};
    if (FWD && n < H) {
      const i2 s = p + q;
      q = p - q;
      p = s;
    }
    const int2 px = dx_split(p.x), py = dx_split(p.y), qx = dx_split(q.x), qy = dx_split(q.y);
    if (n < H) v[(N - 1 - n) * LPC] = make_int4(qx.x, qx.y, qy.x, qy.y);
    v[n * LPC] = make_int4(px.x, px.y, py.x, py.y);
  }
  __syncthreads();
  if (!valid) return;
  const int2* __restrict__ M = FWD ? S.fwd[AXIS] : S.inv[AXIS];  // row = output index
  if (FWD) {
    const FxOut fo = fx_out(e.eb);
    // two modes of one parity at a time: kk and kk + T
    for (int kk = t; kk < N; kk += 2 * T) {
      const bool odd = kk & 1, two = kk + T < N;
      const int4* src = odd ? v + (long long)(N - 1) * LPC : v;
      const int step = odd ? -LPC : LPC, terms = odd ? H : He;
      const int2* __restrict__ r0 = M + (long long)kk * N;
      const int2* __restrict__ r1 = M + (long long)(two ? kk + T : kk) * N;
      DxSum a, b, p, q;
      for (int n0 = 0; n0 < terms; n0 += DX_SEG) {
        const int n1 = min(terms, n0 + DX_SEG);
#pragma unroll 4
        for (int n = n0; n < n1; ++n) {
          const int4 x = src[n * step];
          const int2 w0 = __ldg(r0 + n), w1 = __ldg(r1 + n);
          a.add(x.x, x.y, w0);
          b.add(x.z, x.w, w0);
          p.add(x.x, x.y, w1);
          q.add(x.z, x.w, w1);
        }
        a.fold();
        b.fold();
        p.fold();
        q.fold();
      }
      double2 y = fx_to(i2{a.hi, b.hi}, fo, c);
      if (fo.odd) fx_rescale(y, fo);
      g[(long long)kk * st] = y;
      if (two) {
        y = fx_to(i2{p.hi, q.hi}, fo, c);
        if (fo.odd) fx_rescale(y, fo);
        g[(long long)(kk + T) * st] = y;
      }
    }
  } else {
    const FxOut fo = fx_out(e.eb >= kFxNonfinite / 2 ? e.eb : e.eb - S.gexp[AXIS]);
    for (int n = t; n < He; n += T) {
      const int2* __restrict__ row = M + (long long)n * N;
      DxSum ex, ey, ox, oy;
      for (int q0 = 0; q0 < N; q0 += DX_SEG) {
        const int q1 = min(N, q0 + DX_SEG);  // q0 is even
#pragma unroll 2
        for (int q = q0; q + 1 < q1; q += 2) {
          const int4 x = v[q * LPC], z = v[(q + 1) * LPC];
          const int2 w0 = __ldg(row + q), w1 = __ldg(row + q + 1);
          ex.add(x.x, x.y, w0);
          ey.add(x.z, x.w, w0);
          ox.add(z.x, z.y, w1);
          oy.add(z.z, z.w, w1);
        }
        if ((q1 - q0) & 1) {  // the last mode of an odd N
          const int4 x = v[(q1 - 1) * LPC];
          const int2 w0 = __ldg(row + q1 - 1);
          ex.add(x.x, x.y, w0);
          ey.add(x.z, x.w, w0);
        }
        ex.fold();
        ey.fold();
        ox.fold();
        oy.fold();
      }
      double2 y = fx_to(i2{ex.hi + ox.hi, ey.hi + oy.hi}, fo, c);
      if (fo.odd) fx_rescale(y, fo);
      g[(long long)n * st] = y;
      if (n < H) {
        y = fx_to(i2{ex.hi - ox.hi, ey.hi - oy.hi}, fo, c);
        if (fo.odd) fx_rescale(y, fo);
        g[(long long)(N - 1 - n) * st] = y;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Tridiagonal solve along the wall axis s.  After the transforms of the other
// two axes every spectrum line along s is an independent system
//   p[j-1] - (2 - e_j - sigma h^2) p[j] + p[j+1] = h^2 scale rhs[j],
// sigma = lambda_x + lambda_other, e_j the pressure-BC change of the end rows.
// Its solution is that of the per-axis transform, eigenvalue divide and
// inverse transform of DCT_poisson_solver (NS_functions.f90:1505-1630) along s.
// The solve used for lines of 8 rows and more is the twisted factorisation
// from a table of multipliers (tri_twist_body, below); this one-thread
// Thomas solve (no pivoting: the rows are diagonally dominant) computes its
// multipliers into shared memory and serves shorter lines.  The one singular
// line (Neumann/periodic everywhere, both modes 0) drops its rhs mean, pins
// its last entry and takes the mean value (NS_functions.f90:1576-1577).
// ---------------------------------------------------------------------------
constexpr int TRI_T = 32;  // lines per CTA (one warp)

// One real component of a line, general path (the singular line).
__device__ void tri_real(double* x, long long sx, int N, double sig_h2, double elo, double ehi, double rs, double* cm,
                         bool sing, double target) {
  double mean_r = 0.0;
  if (sing) {
    for (int j = 0; j < N; ++j) mean_r += x[j * sx];
    mean_r /= N;
  }
  const int last = sing ? N - 2 : N - 1;
  double m = 0.0, d = 0.0;
  for (int j = 0; j <= last; ++j) {
    double b = -2.0 + sig_h2;
    if (j == 0) b += elo;
    if (j == N - 1) b += ehi;
    m = 1.0 / (b - m);
    d = fma(x[j * sx] - mean_r, rs, -d) * m;
    x[j * sx] = d;
    cm[j * TRI_T] = m;
  }
  double p = 0.0;
  if (sing) x[(long long)(N - 1) * sx] = 0.0;
  else p = d;
  for (int j = N - 2; j >= 0; --j) {
    p = fma(-cm[j * TRI_T], p, x[j * sx]);
    x[j * sx] = p;
  }
  if (sing) {
    double mp = 0.0;
    for (int j = 0; j < N; ++j) mp += x[j * sx];
    const double shift = target - mp / N;
    for (int j = 0; j < N; ++j) x[j * sx] += shift;
  }
}

// The singular line by a whole warp.  Its system is the Neumann one along
// the axis (end rows -x_0 + x_1, x_{N-2} - x_{N-1}; sigma = 0), whose
// solution with the rhs mean dropped and the mean set to target (the
// reference pins the last entry and shifts, NS_functions.f90:1576-1577) is
// the flux F_j = x_{j+1} - x_j = sum_{i<=j} R_i, R = rs (r - mean r), then
// x_j = sum_{i<j} F_i shifted to the target mean: two prefix sums over the
// warp, lane l holding the rows [l seg, l seg + seg), seg = ceil(N/32).  r is
// read from src (stride 1, re-read by each pass), the solution written to x
// (stride sx doubles).
__device__ __noinline__ void sing_line_warp(const double* src, double* x, long long sx, int N, double rs,
                                            double target) {
  const int lane = threadIdx.x & 31;
  const int seg = (N + 31) / 32, j0 = min(lane * seg, N), j1 = min(j0 + seg, N);
  auto warp_sum = [](double v) {
#pragma unroll
    for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
  };
  auto warp_excl = [&](double tot) {  // exclusive scan of the lanes' totals
    double incl = tot;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += y;
    }
    return incl - tot;
  };
  double s = 0.0;
  for (int j = j0; j < j1; ++j) s += src[j];
  const double mean_r = warp_sum(s) / N;
  s = 0.0;
  for (int j = j0; j < j1; ++j) s += (src[j] - mean_r) * rs;
  const double f0 = warp_excl(s);  // F before this lane's rows
  // x_j = x_{j0} + sum_{j0<=i<j} F_i: the lane's sum of F over its rows
  double fs = 0.0, f = f0;
  for (int j = j0; j < j1; ++j) {
    f += (src[j] - mean_r) * rs;
    fs += f;
  }
  const double xb = warp_excl(fs);  // x at this lane's first row (x_0 = 0)
  double xv = xb, ms = 0.0;
  f = f0;
  for (int j = j0; j < j1; ++j) {
    x[(long long)j * sx] = xv;
    ms += xv;
    f += (src[j] - mean_r) * rs;
    xv += f;
  }
  const double shift = target - warp_sum(ms) / N;
  __syncwarp();
  for (int j = j0; j < j1; ++j) x[(long long)j * sx] += shift;
}


template <int AXIS, bool PACKED>
__device__ __forceinline__ void tri_solve_body(const SpecPlan& S, double2* __restrict__ spec, double* cm, int bx,
                                               int by) {
  // cm: [N][TRI_T] multipliers (x2 when PACKED)
  const int l = threadIdx.x;
  const int N = AXIS == 1 ? S.ny : S.nz;
  const int n_other = AXIS == 1 ? S.nz : S.ny;
  // Columns: with a periodic x the Nyquist column is handled by the last
  // block column, lanes over the other index (no idle lanes).
  const int nreg = PACKED ? S.nxs : S.nxs - 1;
  const int nblk = (nreg + TRI_T - 1) / TRI_T;
  int col, o;
  bool valid;
  if (bx < nblk) {
    col = bx * TRI_T + l;
    o = by;
    valid = col < nreg;
  } else {
    if (by * TRI_T >= n_other) return;
    col = S.nxs - 1;
    o = by * TRI_T + l;
    valid = o < n_other;
  }
  if (!valid) return;
  const long long st = AXIS == 1 ? (long long)S.nxs : (long long)S.nxs * S.ny;
  double2* g = spec + (AXIS == 1 ? col + (long long)S.nxs * S.ny * o : col + (long long)S.nxs * o);
  const double lo = __ldg(S.eig_o + o);
  const double sr = (__ldg(S.eig_x + (PACKED ? 2 * col : col)) + lo) * S.tri_h2;
  const double si = PACKED ? (__ldg(S.eig_x + 2 * col + 1) + lo) * S.tri_h2 : sr;
  const double rs = S.tri_rs, elo = S.tri_elo, ehi = S.tri_ehi;
  double* cmr = cm + l;
  double* cmi = PACKED ? cm + (long long)N * TRI_T + l : cmr;
  if (S.has_mean && col == 0 && o == 0) {  // the singular line
    double* x = reinterpret_cast<double*>(g);
    tri_real(x, 2 * st, N, sr, elo, ehi, rs, cmr, true, S.mean_dev ? S.mean_val * *S.mean_dev : S.mean_val);
    tri_real(x + 1, 2 * st, N, si, elo, ehi, rs, cmi, !PACKED, 0.0);
    return;
  }
  double mr = 0.0, mi = 0.0;
  double2 d = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int j = 0; j < N; ++j) {
    double br = -2.0 + sr, bi = -2.0 + si;
    if (j == 0) { br += elo; bi += elo; }
    if (j == N - 1) { br += ehi; bi += ehi; }
    mr = 1.0 / (br - mr);
    if (PACKED) mi = 1.0 / (bi - mi);
    else mi = mr;
    const double2 r = g[(long long)j * st];
    d.x = fma(r.x, rs, -d.x) * mr;
    d.y = fma(r.y, rs, -d.y) * mi;
    g[(long long)j * st] = d;
    cmr[j * TRI_T] = mr;
    if (PACKED) cmi[j * TRI_T] = mi;
  }
  double2 p = d;
#pragma unroll 4
  for (int j = N - 2; j >= 0; --j) {
    const double2 x = g[(long long)j * st];
    p.x = fma(-cmr[j * TRI_T], p.x, x.x);
    p.y = fma(-cmi[j * TRI_T], p.y, x.y);
    g[(long long)j * st] = p;
  }
}

__global__ void __launch_bounds__(128) dense_x_fwd_kernel(SpecPlan S, DivArgs d, double2* __restrict__ spec) {
  extern __shared__ __align__(16) double xs_fwd[];
  dense_x_fwd_body(S, d, spec, xs_fwd, blockIdx.x);
}
__global__ void __launch_bounds__(128) dense_x_inv_kernel(SpecPlan S, const double2* __restrict__ spec, double* dp,
                                                          Layout L, FOne c) {
  extern __shared__ __align__(16) double xs_inv[];
  dense_x_inv_body(S, spec, dp, L, xs_inv, blockIdx.x, c);
}
template <int AXIS, bool FWD>
__global__ void __launch_bounds__(128) dense_yz_kernel(SpecPlan S, double2* __restrict__ spec, FOne c) {
  extern __shared__ __align__(16) double2 ls_yz[];
  dense_yz_body<AXIS, FWD>(S, spec, ls_yz, blockIdx.x, c);
}

template <int AXIS, bool PACKED>
__global__ void __launch_bounds__(TRI_T) tri_solve_kernel(SpecPlan S, double2* __restrict__ spec) {
  extern __shared__ __align__(16) double cm_tri[];
  tri_solve_body<AXIS, PACKED>(S, spec, cm_tri, blockIdx.x, blockIdx.y);
}


// ---------------------------------------------------------------------------
// Twisted, table-driven line solve (the session's wall axis, 1 or 2, and
// the batch's z axis).  Line
// t = col + nxs o (o: z for y lines, y for z lines) of N rows; k = N/2.  Its
// table holds m_j = 1/(b_j - m_{j-1}) for j < k (top-down, as tri_solve_body),
// n_j = 1/(b_j - n_{j+1}) for j > k (bottom-up) and the middle pivot
// 1/(b_k - m_{k-1} - n_{k+1}).  Lanes l and l + 16 of a warp take line l:
// the top lane forms d_j = (rs r_j - d_{j-1}) m_j downwards, the bottom lane
// e_j = (rs r_j - e_{j+1}) n_j upwards; the middle row gives
// x_k = (rs r_k - d_{k-1} - e_{k+1}) piv, and the lanes substitute outwards,
// x_j = d_j - m_j x_{j+1} above and x_j = e_j - n_j x_{j-1} below.  No
// division in the solve, twice the lines' lanes in flight and half the
// recurrence length of the one-lane Thomas solve; the sums round
// differently.  The singular line takes the general path on its top lane.
// ---------------------------------------------------------------------------
struct TwLine {
  long long base, st;
  int col, o;
  bool valid;
};
template <int AXIS>
__device__ __forceinline__ TwLine tw_line(const SpecPlan& S, int t) {
  TwLine L;
  L.valid = t < S.nxs * (AXIS == 1 ? S.nz : S.ny);
  if (!L.valid) t = 0;
  L.col = t % S.nxs;
  L.o = t / S.nxs;
  if (AXIS == 1) { L.base = L.col + (long long)S.nxs * S.ny * L.o; L.st = S.nxs; }
  else { L.base = t; L.st = (long long)S.nxs * S.ny; }
  return L;
}

template <int AXIS, bool PACKED>
__global__ void __launch_bounds__(128) tri_twist_table_kernel(SpecPlan S, double2* __restrict__ tab) {
  const TwLine ln = tw_line<AXIS>(S, blockIdx.x * 128 + threadIdx.x);
  if (!ln.valid) return;
  const int N = AXIS == 1 ? S.ny : S.nz, k = N / 2;
  const double lo = __ldg(S.eig_o + ln.o);
  const double sr = (__ldg(S.eig_x + (PACKED ? 2 * ln.col : ln.col)) + lo) * S.tri_h2;
  const double si = PACKED ? (__ldg(S.eig_x + 2 * ln.col + 1) + lo) * S.tri_h2 : sr;
  const double elo = S.tri_elo, ehi = S.tri_ehi;
  auto bj = [&](int j, double s) {
    double b = -2.0 + s;
    if (j == 0) b += elo;
    if (j == N - 1) b += ehi;
    return b;
  };
  double2* g = tab + ln.base;
  double mr = 0.0, mi = 0.0;
  for (int j = 0; j < k; ++j) {
    mr = 1.0 / (bj(j, sr) - mr);
    mi = PACKED ? 1.0 / (bj(j, si) - mi) : mr;
    g[(long long)j * ln.st] = make_double2(mr, mi);
  }
  double nr = 0.0, ni = 0.0;
  for (int j = N - 1; j > k; --j) {
    nr = 1.0 / (bj(j, sr) - nr);
    ni = PACKED ? 1.0 / (bj(j, si) - ni) : nr;
    g[(long long)j * ln.st] = make_double2(nr, ni);
  }
  const double pr = 1.0 / (bj(k, sr) - mr - nr);
  const double pi = PACKED ? 1.0 / (bj(k, si) - mi - ni) : pr;
  g[(long long)k * ln.st] = make_double2(pr, pi);
}

// One 128-thread block bx of the twisted solve (64 lines); scr: scratch of
// 2 N TRI_T doubles for the singular line.
template <int AXIS, bool PACKED>
__device__ __forceinline__ void tri_twist_body(const SpecPlan& S, double2* __restrict__ spec, double* scr, int bx) {
  constexpr int TP = 4;  // rows and multipliers loaded ahead
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = lane >> 4;
  const int t0 = (bx * 4 + warp) * 16;
  if (t0 >= S.nxs * (AXIS == 1 ? S.nz : S.ny)) return;  // the whole warp
  const TwLine ln = tw_line<AXIS>(S, t0 + (lane & 15));
  const int N = AXIS == 1 ? S.ny : S.nz, k = N / 2;
  // The singular line (col 0, o 0: lane 0 of the first warp) of a Neumann
  // axis goes to the whole warp after the other lines (sing_line_warp); its
  // rhs is set aside in the scratch first, since the twisted lanes also run
  // over it (a packed box's second mode of that slot is a regular line).
  // Otherwise it takes the one-lane general path on its top lane.
  const bool warp_sing = t0 == 0 && S.has_mean && S.tri_elo == 1.0 && S.tri_ehi == 1.0 && N <= 512;
  const bool sing = ln.valid && S.has_mean && ln.col == 0 && ln.o == 0;
  const bool work = ln.valid && (!sing || warp_sing);
  if (warp_sing) {
    const double2* g0 = spec;  // line (0, 0)
    for (int j = lane; j < N; j += 32) {
      const double2 r = g0[(long long)j * (AXIS == 1 ? (long long)S.nxs : (long long)S.nxs * S.ny)];
      scr[j] = r.x;
      if (!PACKED) scr[N + j] = r.y;
    }
    __syncwarp();
  }
  double2* g = spec + ln.base;
  const double2* __restrict__ tm = S.tri_m + ln.base;
  const long long st = ln.st;
  const double rs = S.tri_rs;
  const int cnt = h ? N - 1 - k : k;
  auto row = [&](int q) { return h ? N - 1 - q : q; };
  const double2 z2 = make_double2(0.0, 0.0);
  // elimination towards the middle row
  double2 d = z2;
  if (work) {
    double2 rv[TP], mv[TP];
#pragma unroll
    for (int q = 0; q < TP; ++q) {
      const bool in = q < cnt;
      rv[q] = in ? g[(long long)row(q) * st] : z2;
      mv[q] = in ? __ldg(tm + (long long)row(q) * st) : z2;
    }
    for (int q0 = 0; q0 < cnt; q0 += TP) {
      double2 rn[TP], mn[TP];
#pragma unroll
      for (int q = 0; q < TP; ++q) {
        const int qq = q0 + TP + q;
        const bool in = qq < cnt;
        rn[q] = in ? g[(long long)row(qq) * st] : z2;
        mn[q] = in ? __ldg(tm + (long long)row(qq) * st) : z2;
      }
#pragma unroll
      for (int q = 0; q < TP; ++q)
        if (q0 + q < cnt) {
          d.x = fma(rv[q].x, rs, -d.x) * mv[q].x;
          d.y = fma(rv[q].y, rs, -d.y) * mv[q].y;
          g[(long long)row(q0 + q) * st] = d;
        }
#pragma unroll
      for (int q = 0; q < TP; ++q) {
        rv[q] = rn[q];
        mv[q] = mn[q];
      }
    }
  }
  // the middle row, on the top lane, with the bottom lane's e_{k+1}
  const double ex = __shfl_xor_sync(0xffffffffu, d.x, 16), ey = __shfl_xor_sync(0xffffffffu, d.y, 16);
  double2 xk = z2;
  if (work && h == 0) {
    const double2 r = g[(long long)k * st];
    const double2 pv = __ldg(tm + (long long)k * st);
    xk.x = (fma(r.x, rs, -d.x) - ex) * pv.x;
    xk.y = (fma(r.y, rs, -d.y) - ey) * pv.y;
    g[(long long)k * st] = xk;
  }
  xk.x = __shfl_sync(0xffffffffu, xk.x, lane & 15);
  xk.y = __shfl_sync(0xffffffffu, xk.y, lane & 15);
  // substitution away from the middle row (row index cnt - 1 - q)
  if (work) {
    double2 p = xk;
    double2 rv[TP], mv[TP];
#pragma unroll
    for (int q = 0; q < TP; ++q) {
      const int qq = cnt - 1 - q;
      const bool in = qq >= 0;
      rv[q] = in ? g[(long long)row(qq) * st] : z2;
      mv[q] = in ? __ldg(tm + (long long)row(qq) * st) : z2;
    }
    for (int q0 = 0; q0 < cnt; q0 += TP) {
      double2 rn[TP], mn[TP];
#pragma unroll
      for (int q = 0; q < TP; ++q) {
        const int qq = cnt - 1 - (q0 + TP + q);
        const bool in = qq >= 0;
        rn[q] = in ? g[(long long)row(qq) * st] : z2;
        mn[q] = in ? __ldg(tm + (long long)row(qq) * st) : z2;
      }
#pragma unroll
      for (int q = 0; q < TP; ++q) {
        const int qq = cnt - 1 - (q0 + q);
        if (qq >= 0) {
          p.x = fma(-mv[q].x, p.x, rv[q].x);
          p.y = fma(-mv[q].y, p.y, rv[q].y);
          g[(long long)row(qq) * st] = p;
        }
      }
#pragma unroll
      for (int q = 0; q < TP; ++q) {
        rv[q] = rn[q];
        mv[q] = mn[q];
      }
    }
  }
  const double target = S.mean_dev ? S.mean_val * *S.mean_dev : S.mean_val;
  if (warp_sing) {
    __syncwarp();
    const long long st0 = AXIS == 1 ? (long long)S.nxs : (long long)S.nxs * S.ny;
    double* x0 = reinterpret_cast<double*>(spec);
    sing_line_warp(scr, x0, 2 * st0, N, rs, target);
    if (!PACKED) sing_line_warp(scr + N, x0 + 1, 2 * st0, N, rs, 0.0);
  } else if (sing && h == 0) {
    const double lo = __ldg(S.eig_o);
    const double sr = (__ldg(S.eig_x) + lo) * S.tri_h2;
    const double si = PACKED ? (__ldg(S.eig_x + 1) + lo) * S.tri_h2 : sr;
    double* x = reinterpret_cast<double*>(g);
    tri_real(x, 2 * st, N, sr, S.tri_elo, S.tri_ehi, rs, scr, true, target);
    tri_real(x + 1, 2 * st, N, si, S.tri_elo, S.tri_ehi, rs, scr + (long long)N * TRI_T, !PACKED, 0.0);
  }
}

template <int AXIS, bool PACKED>
__global__ void __launch_bounds__(128) tri_twist_solve_kernel(SpecPlan S, double2* __restrict__ spec) {
  tri_twist_body<AXIS, PACKED>(S, spec, S.sing_cm, blockIdx.x);
}

// ---------------------------------------------------------------------------
// Batched passes: persistent CTAs walk (subdomain, block) work items; the
// subdomain's arguments are staged in shared memory once per item.
// PASS: 0 x forward, 1 x inverse, 2 y forward, 3 y inverse, 4 tridiagonal z (packed x,
// the twisted solve from the subdomain's table).
// A subdomain whose plan sets dct_x / dct_y (an axis of 24, 32, 48 or 64
// points, pressure code 2 or 3) takes the FFT-based line bodies of
// ns_fft_core.cuh there, with 128 / R1 lines per item so that all 128
// threads work; the others take the dense products.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int batch_dct_lpc(int n) {
  return 128 / (n == 64 ? Split<64>::R1 : n == 48 ? Split<48>::R1 : n == 32 ? Split<32>::R1 : Split<24>::R1);
}

template <int N, int PB>
__device__ __forceinline__ void batch_dct(int pass, const BatchSpecArgs& a, double2* sb, int bx) {
  constexpr int LPC = batch_dct_lpc(N);
  const FOne c{a.d.one, a.d.mzero};
  const int l = threadIdx.x % LPC, t = threadIdx.x / LPC;
  if (pass == 0) dct_x_fwd_body<N, PB, LPC>(a.S, a.spec, sb, bx, l, t, c);
  else if (pass == 1) dct_x_inv_body<N, PB, LPC>(a.S, a.spec, a.dp, a.L, sb, bx, l, t, c);
  else if (pass == 2) dct_y_body<N, true, PB, LPC>(a.S, a.spec, sb, bx, l, t, c);
  else dct_y_body<N, false, PB, LPC>(a.S, a.spec, sb, bx, l, t, c);
}

template <int PASS>
__device__ __forceinline__ void batch_dct_dispatch(const BatchSpecArgs& a, double2* sb, int bx) {
  const int n = PASS < 2 ? a.S.nx : a.S.ny;
  const int pb = PASS < 2 ? a.S.dct_x : a.S.dct_y;
  if (n == 64) {
    if (pb == 2) batch_dct<64, 2>(PASS, a, sb, bx);
    else batch_dct<64, 3>(PASS, a, sb, bx);
  } else if (n == 48) {
    if (pb == 2) batch_dct<48, 2>(PASS, a, sb, bx);
    else batch_dct<48, 3>(PASS, a, sb, bx);
  } else if (n == 32) {
    if (pb == 2) batch_dct<32, 2>(PASS, a, sb, bx);
    else batch_dct<32, 3>(PASS, a, sb, bx);
  } else {
    if (pb == 2) batch_dct<24, 2>(PASS, a, sb, bx);
    else batch_dct<24, 3>(PASS, a, sb, bx);
  }
}

template <int PASS>
__global__ void __launch_bounds__(128) spec_batch_kernel(const BatchSpecArgs* __restrict__ tab,
                                                         const BatchItem* __restrict__ items, int n_items) {
  extern __shared__ __align__(16) double sm_b[];
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const BatchItem w = items[it];
    // the subdomain's arguments from the read-only table (a copy in shared
    // memory would be reloaded after every barrier of the passes)
    const BatchSpecArgs& a = tab[w.sub];
    if (PASS == 0) dense_x_fwd_body(a.S, a.d, a.spec, sm_b, w.bx);
    const FOne c{a.d.one, a.d.mzero};
    if (PASS == 1) dense_x_inv_body(a.S, a.spec, a.dp, a.L, sm_b, w.bx, c);
    if (PASS == 2) dense_yz_body<1, true>(a.S, a.spec, reinterpret_cast<double2*>(sm_b), w.bx, c);
    if (PASS == 3) dense_yz_body<1, false>(a.S, a.spec, reinterpret_cast<double2*>(sm_b), w.bx, c);
    if (PASS == 4) tri_twist_body<2, true>(a.S, a.spec, sm_b, w.bx);
    __syncthreads();
  }
}

template <int PASS>
__global__ void __launch_bounds__(128) spec_batch_dct_kernel(const BatchSpecArgs* __restrict__ tab,
                                                             const BatchItem* __restrict__ items, int n_items) {
  extern __shared__ __align__(16) double2 sm_d[];
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const BatchItem w = items[it];
    batch_dct_dispatch<PASS>(tab[w.sub], sm_d, w.bx);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kDivChunk) spec_batch_div_kernel(const BatchSpecArgs* __restrict__ tab,
                                                                   const BatchItem* __restrict__ items, int n_items) {
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const BatchItem w = items[it];
    const BatchSpecArgs& a = tab[w.sub];
    const unsigned N = (unsigned)a.S.nx;
    const unsigned e = (unsigned)w.bx * kDivChunk + threadIdx.x;  // a subdomain box holds < 2^31 cells
    if (e < N * (unsigned)a.S.ny * (unsigned)a.S.nz) {
      const int row = (int)(e / N), i = (int)(e - (unsigned)row * N);
      const FOne c{a.d.one, a.d.mzero};
      const DivArgs& d = a.d;
      double v;
      if (d.rhs) {
        v = d.rhs[d.L.at(i + 1, 1 + row % a.S.ny, 1 + row / a.S.ny)];
      } else {  // the divergence; the boundary cells' terms follow in spec_batch_bc_kernel
        const long long g = d.L.at(i + 1, 1 + row % a.S.ny, 1 + row / a.S.ny);
        v = fmul(c, fsub(c, d.us[g + 1], d.us[g]), d.cdx);
        v = fma(fsub(c, d.vs[g + d.L.sy], d.vs[g]), d.cdy, v);
        v = fma(fsub(c, d.ws[g + d.L.sz], d.ws[g]), d.cdz, v);
        v = v + 0.0;
      }
      reinterpret_cast<double*>(a.spec)[e] = v;
    }
  }
}

// The pressure-BC terms of those subdomains' boundary cells, added to their
// divergence rows (item (sub, q): boundary cells [kDivChunk q, kDivChunk (q+1))
// in the order of SpecPlan::bc_cell).
__global__ void __launch_bounds__(kDivChunk) spec_batch_bc_kernel(const BatchSpecArgs* __restrict__ tab,
                                                                  const BatchItem* __restrict__ items, int n_items) {
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const BatchItem w = items[it];
    const BatchSpecArgs& a = tab[w.sub];
    const long long q = (long long)w.bx * kDivChunk + threadIdx.x;
    if (q < a.S.bc_cells()) {
      int i, j, k;
      a.S.bc_cell(q, i, j, k);
      double* out = reinterpret_cast<double*>(a.spec);
      const long long e = (long long)a.S.nx * ((j - 1) + (long long)a.S.ny * (k - 1)) + (i - 1);
      out[e] = out[e] + a.S.bc_term_edge(i, j, k);
    }
  }
}

cudaError_t launch_spec_batch_bc(const BatchSpecArgs* tab, const BatchItem* items, int n_items, int grid,
                                 cudaStream_t st) {
  if (n_items <= 0) return cudaSuccess;
  if (grid <= 0) grid = 8 * 152;
  if (grid > n_items) grid = n_items;
  spec_batch_bc_kernel<<<grid, kDivChunk, 0, st>>>(tab, items, n_items);
  return cudaGetLastError();
}

cudaError_t launch_spec_batch_div(const BatchSpecArgs* tab, const BatchItem* items, int n_items, int grid,
                                  cudaStream_t st) {
  if (n_items <= 0) return cudaSuccess;
  if (grid <= 0) {
    int per_sm = 0, dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, spec_batch_div_kernel, kDivChunk, 0);
    grid = (per_sm > 0 ? per_sm : 1) * nsm;
  }
  if (grid > n_items) grid = n_items;
  spec_batch_div_kernel<<<grid, kDivChunk, 0, st>>>(tab, items, n_items);
  return cudaGetLastError();
}

bool spec_pass_dct(int pass, const SpecPlan& S) {
  return ((pass == 0 || pass == 1) && S.dct_x) || ((pass == 2 || pass == 3) && S.dct_y);
}

// Work-item grid of one pass for one subdomain.
void spec_pass_grid(int pass, const SpecPlan& S, int& gx, int& gy) {
  gy = 1;
  if ((pass == 0 || pass == 1) && S.dct_x) gx = (S.ny * S.nz + 2 * batch_dct_lpc(S.nx) - 1) / (2 * batch_dct_lpc(S.nx));
  else if ((pass == 2 || pass == 3) && S.dct_y) gx = (S.nxs * S.nz + batch_dct_lpc(S.ny) - 1) / batch_dct_lpc(S.ny);
  else if (pass == 0 || pass == 1) {
    const int per = 128 / dense_x_group(S.nx);
    gx = (S.ny * S.nz + per - 1) / per;
  }
  else if (pass == 2 || pass == 3) gx = (S.nxs * S.nz + DX_LPC - 1) / DX_LPC;
  else gx = (S.nxs * S.ny + 63) / 64;  // tri_twist_body: 64 lines per item
}

size_t spec_pass_smem(int pass, const SpecPlan& S) {
  if ((pass == 0 || pass == 1) && S.dct_x) {
    const size_t L = batch_dct_lpc(S.nx);
    return (size_t)S.nx * L * sizeof(i2) + L * (S.nx + 1) * sizeof(double2) + 128 * sizeof(FxExp);
  }
  if ((pass == 2 || pass == 3) && S.dct_y) return (size_t)S.ny * batch_dct_lpc(S.ny) * sizeof(i2) + 128 * sizeof(FxExp);
  if (pass == 0 || pass == 1) return (size_t)(128 / dense_x_group(S.nx)) * S.nx * sizeof(double);
  if (pass == 2 || pass == 3) return dense_yz_smem(S.ny);
  return (size_t)S.nz * TRI_T * sizeof(double) * 2;
}

cudaError_t launch_spec_batch(int pass, bool dct, const BatchSpecArgs* tab, const BatchItem* items, int n_items,
                              size_t smem, int grid, cudaStream_t st) {
  if (n_items <= 0) return cudaSuccess;
  if (dct && (pass < 0 || pass > 3)) return cudaErrorInvalidValue;
  auto kern = dct ? (pass == 0 ? spec_batch_dct_kernel<0>
                   : pass == 1 ? spec_batch_dct_kernel<1>
                   : pass == 2 ? spec_batch_dct_kernel<2>
                               : spec_batch_dct_kernel<3>)
            : pass == 0 ? spec_batch_kernel<0>
            : pass == 1 ? spec_batch_kernel<1>
            : pass == 2 ? spec_batch_kernel<2>
            : pass == 3 ? spec_batch_kernel<3>
                        : spec_batch_kernel<4>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  if (grid <= 0) {
    int per_sm = 0, dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 128, smem);
    grid = (per_sm > 0 ? per_sm : 1) * nsm;
  }
  if (grid > n_items) grid = n_items;
  kern<<<grid, 128, smem, st>>>(tab, items, n_items);
  return cudaGetLastError();
}

cudaError_t launch_dense_x(bool fwd, const SpecPlan& S, const DivArgs& d, double2* spec, double* dp, const Layout& L,
                           cudaStream_t st) {
  const int lines = S.ny * S.nz, per = 128 / dense_x_group(S.nx);
  const size_t sm = (size_t)per * S.nx * sizeof(double);
  if (fwd) dense_x_fwd_kernel<<<(lines + per - 1) / per, 128, sm, st>>>(S, d, spec);
  else dense_x_inv_kernel<<<(lines + per - 1) / per, 128, sm, st>>>(S, spec, dp, L, FOne{1.0, -0.0});
  return cudaGetLastError();
}

int q54_table(std::vector<double>& M) {
  double m = 0.0;
  for (double x : M) m = std::fmax(m, std::fabs(x));
  int e = 0;
  if (m > 0.0) (void)std::frexp(m, &e);  // m in [2^(e-1), 2^e)
  if (m == std::ldexp(1.0, e - 1)) --e;  // an exact power of two is 1 in its own units
  for (double& x : M) {
    const long long q = std::llrint(std::ldexp(x, 54 - e));
    const int h = (int)((q + (1ll << 26)) >> 27);
    const int2 w = make_int2(h, (int)(q - ((long long)h << 27)));
    std::memcpy(&x, &w, sizeof(w));
  }
  return -e;
}

cudaError_t launch_dense_yz(int axis, bool fwd, const SpecPlan& S, double2* spec, cudaStream_t st) {
  const int N = axis == 1 ? S.ny : S.nz;
  if (N > 512) return cudaErrorInvalidValue;
  // DX_LPC lines of N complex values staged in shared memory: 64 KB at N = 512 (past the 48 KB
  // default: opt in)
  const size_t sm = dense_yz_smem(N);
  dim3 grid((S.nxs * (axis == 1 ? S.nz : S.ny) + DX_LPC - 1) / DX_LPC);
  auto kern = (axis == 1) ? (fwd ? dense_yz_kernel<1, true> : dense_yz_kernel<1, false>)
                          : (fwd ? dense_yz_kernel<2, true> : dense_yz_kernel<2, false>);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  kern<<<grid, DX_LPC * DX_T, sm, st>>>(S, spec, FOne{1.0, -0.0});
  return cudaGetLastError();
}



cudaError_t launch_tri_twist_table(int axis, const SpecPlan& S, double2* tab, cudaStream_t st) {
  const bool packed = S.kind[0] != 0;
  const int nlines = S.nxs * (axis == 1 ? S.nz : S.ny);
  const int grid = (nlines + 127) / 128;
  if (axis == 1) {
    if (packed) tri_twist_table_kernel<1, true><<<grid, 128, 0, st>>>(S, tab);
    else tri_twist_table_kernel<1, false><<<grid, 128, 0, st>>>(S, tab);
  } else {
    if (packed) tri_twist_table_kernel<2, true><<<grid, 128, 0, st>>>(S, tab);
    else tri_twist_table_kernel<2, false><<<grid, 128, 0, st>>>(S, tab);
  }
  return cudaGetLastError();
}

cudaError_t launch_tri_solve(int axis, const SpecPlan& S, double2* spec, cudaStream_t st) {
  const int N = axis == 1 ? S.ny : S.nz;
  const int n_other = axis == 1 ? S.nz : S.ny;
  const bool packed = S.kind[0] != 0;
  if (S.tri_tw && S.tri_m && S.sing_cm) {
    const int grid = (S.nxs * n_other + 63) / 64;
    if (axis == 1) {
      if (packed) tri_twist_solve_kernel<1, true><<<grid, 128, 0, st>>>(S, spec);
      else tri_twist_solve_kernel<1, false><<<grid, 128, 0, st>>>(S, spec);
    } else {
      if (packed) tri_twist_solve_kernel<2, true><<<grid, 128, 0, st>>>(S, spec);
      else tri_twist_solve_kernel<2, false><<<grid, 128, 0, st>>>(S, spec);
    }
    return cudaGetLastError();
  }
  const size_t sm = (size_t)N * TRI_T * sizeof(double) * (packed ? 2 : 1);
  if (sm > 200 * 1024) return cudaErrorInvalidValue;
  const int nreg = packed ? S.nxs : S.nxs - 1;
  const int nblk = (nreg + TRI_T - 1) / TRI_T;
  dim3 grid(nblk + (packed ? 0 : 1), n_other);
  auto kern = axis == 1 ? (packed ? tri_solve_kernel<1, true> : tri_solve_kernel<1, false>)
                        : (packed ? tri_solve_kernel<2, true> : tri_solve_kernel<2, false>);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  kern<<<grid, TRI_T, sm, st>>>(S, spec);
  return cudaGetLastError();
}

}  // namespace ns
