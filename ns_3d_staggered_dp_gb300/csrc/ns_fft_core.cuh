// The four-step line engine and the FFT-based (Makhoul) DCT-II/III line
// bodies, shared by the session passes (ns_fft.cu) and the batched spectral
// passes (ns_dct.cu).  Lines are doubles in memory; the transforms run on
// block fixed-point integers (ns_fixed.cuh).  Everything here is a template
// or an inline device function with internal linkage in each translation unit.
#pragma once

#include "ns_fixed.cuh"
#include "ns_internal.cuh"
#include "ns_kernels.cuh"

namespace ns {
namespace {

// Four-step split N = R1 * R2 (R1 <= R2), T = R1 threads per line.
template <int N> struct Split;
template <> struct Split<8> { static constexpr int R1 = 2, R2 = 4; };
template <> struct Split<24> { static constexpr int R1 = 2, R2 = 12; };
template <> struct Split<48> { static constexpr int R1 = 4, R2 = 12; };
template <> struct Split<16> { static constexpr int R1 = 4, R2 = 4; };
template <> struct Split<32> { static constexpr int R1 = 4, R2 = 8; };
template <> struct Split<64> { static constexpr int R1 = 8, R2 = 8; };
template <> struct Split<128> { static constexpr int R1 = 8, R2 = 16; };
template <> struct Split<256> { static constexpr int R1 = 16, R2 = 16; };
template <> struct Split<512> { static constexpr int R1 = 16, R2 = 32; };

// ---------------------------------------------------------------------------
// Line engine: LPC lines per CTA (lanes over lines, coalesced when the lines
// are neighbouring columns), T = R1 threads per line.
// Shared buffer index for line l: (r * R2 + q) * LPC + l; the exponents of
// thread t's block: t * LPC + l.
// ---------------------------------------------------------------------------
// Lines per CTA of the session kernels: 8 for the long lines (register-heavy
// 16-point DFTs), else 16.
template <int N>
constexpr int lpc() { return N >= 256 ? 8 : 16; }

template <int N, int LPC_ = lpc<N>()>
struct YZ {
  static constexpr int R1 = Split<N>::R1, R2 = Split<N>::R2, T = R1, KQ = R2 / T;
  static constexpr int LPC = LPC_;
  static constexpr int B1 = 60 - log2up(R1), B2 = 60 - log2up(R2);
  static constexpr size_t kSmem = (size_t)N * LPC * sizeof(i2) + (size_t)T * LPC * sizeof(FxExp);
  __device__ static __forceinline__ int sidx(int r, int q, int l) { return (r * R2 + q) * LPC + l; }

  // Forward step A: thread n1 = t holds x[n1 + R1 n2], R2-point DFT, twiddle, to smem (n1, k2).
  __device__ static __forceinline__ void fwdA(const double2 (&d)[R2], i2* sb, FxExp* se, const int4* __restrict__ tw,
                                              int l, int t) {
    i2 x[R2];
    const int eb = fx_block2<B2>(d, x);
    dft<R2, -1>(x);
    unsigned acc = 0;
    fx_bits(acc, x[0]);
    sb[sidx(t, 0, l)] = x[0];
#pragma unroll
    for (int k2 = 1; k2 < R2; ++k2) {
      const i2 y = fx_cmul(x[k2], fx_ldg(tw + ((t * k2) % N)));
      fx_bits(acc, y);
      sb[sidx(t, k2, l)] = y;
    }
    se[t * LPC + l] = fx_publish<B1>(eb, acc);
  }
  // Forward step B: for k2 = t + T*q: R1-point DFT over n1 -> X[k2 + R2 k1] in xk[q][k1]; returns
  // the line's exponent.
  __device__ static __forceinline__ int fwdB(i2 (&xk)[KQ][R1], const i2* sb, const FxExp* se, int l, int t) {
    int eb[R1], ec = -kFxNonfinite;
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) {
      const FxExp e = se[n1 * LPC + l];
      eb[n1] = e.eb;
      ec = max(ec, e.p);
    }
#pragma unroll
    for (int q = 0; q < KQ; ++q) {
      const int k2 = t + T * q;
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) xk[q][n1] = fx_align(sb[sidx(n1, k2, l)], eb[n1], ec);
      dft<R1, -1>(xk[q]);
    }
    return ec;
  }
  // Inverse step A: from X[k2 + R2 k1] held in xk (exponent eb, B1 bits), R1-point inverse DFT,
  // twiddle, to smem (k2, alpha).
  __device__ static __forceinline__ void invA(i2 (&xk)[KQ][R1], int eb, i2* sb, FxExp* se,
                                              const int4* __restrict__ tw, int l, int t) {
    unsigned acc = 0;
#pragma unroll
    for (int q = 0; q < KQ; ++q) {
      const int k2 = t + T * q;
      dft<R1, 1>(xk[q]);
      fx_bits(acc, xk[q][0]);
      sb[sidx(0, k2, l)] = xk[q][0];
#pragma unroll
      for (int a = 1; a < R1; ++a) {
        const i2 y = fx_cmulc(xk[q][a], fx_ldg(tw + ((a * k2) % N)));
        fx_bits(acc, y);
        sb[sidx(a, k2, l)] = y;
      }
    }
    se[t * LPC + l] = fx_publish<B2>(eb, acc);
  }
  // The thread's X[k2 + R2 k1] as a block for invA.
  __device__ static __forceinline__ int block(const double2 (&d)[KQ][R1], i2 (&xk)[KQ][R1]) {
    double2 f[R2];
    i2 v[R2];
#pragma unroll
    for (int i = 0; i < R2; ++i) f[i] = d[i / R1][i % R1];
    const int eb = fx_block2<B1>(f, v);
#pragma unroll
    for (int i = 0; i < R2; ++i) xk[i / R1][i % R1] = v[i];
    return eb;
  }
  // Inverse step B: thread alpha = t, R2-point inverse DFT over k2: x[beta] is point alpha + R1 beta;
  // returns the line's exponent.
  __device__ static __forceinline__ int invB(i2 (&x)[R2], const i2* sb, const FxExp* se, int l, int t) {
    int eb[T], ec = -kFxNonfinite;
#pragma unroll
    for (int q = 0; q < T; ++q) {
      const FxExp e = se[q * LPC + l];
      eb[q] = e.eb;
      ec = max(ec, e.p);
    }
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) x[k2] = fx_align(sb[sidx(t, k2, l)], eb[k2 % T], ec);
    dft<R2, 1>(x);
    return ec;
  }
};

// The y transform of a packed-x box (two real lines, .x and .y, per complex
// slot) through an FFT (Makhoul).  DCT-II of a real line x of N points
// (dense_pair's pbc-3 matrix F[k][s] = cos(pi k (2s+1) / (2N))) is
//   X_k = Re(exp(-i pi k / (2N)) V_k),  V = DFT_N(v),  v_m = x_{2m}, v_{N-1-m} = x_{2m+1}.
// The two real lines of a slot share one complex FFT and are separated in the
// post-twiddle: with U_k = exp(-i pi k / (2N)) V_k / 2 (and V_N = V_0),
//   X_k = (Re U_k - Im U_{N-k}) + i (Im U_k + Re U_{N-k}).
// pbc 2's matrix is the same transform of the line with its even (0-based)
// samples negated, modes reversed (k -> N-1-k).  The inverse is the exact
// inverse (DCT-III with its 1/N): V_k = exp(i pi k / (2N)) (X_k - i X_{N-k}) / N
// (X_N = 0), v = the unnormalised inverse DFT of V, x_{2m} = v_m,
// x_{2m+1} = v_{N-1-m}.  The pre-twiddle table holds exp(i pi k / (2N)) 2^f / N
// with f = floor(log2 N), the 2^-f goes into the block's exponent.  Lines are numbered
// tl = col + nxs kz; block blk of a pass takes lines blk LPC .. blk LPC + LPC-1.
template <int N, bool FWD, int PB, int LPC_ = lpc<N>()>
__device__ __forceinline__ void dct_y_body(const FftPlan& P, double2* __restrict__ spec, double2* smem, int blk, int l,
                                           int t, const FOne& c) {
  using F = YZ<N, LPC_>;
  constexpr int LPC = F::LPC, R1 = F::R1, R2 = F::R2, T = F::T, KQ = F::KQ;
  i2* sb = reinterpret_cast<i2*>(smem);
  FxExp* se = reinterpret_cast<FxExp*>(sb + N * LPC);
  const int tl = blk * LPC + l;
  const bool valid = tl < P.nxs * P.nz;
  const int col = valid ? tl % P.nxs : 0, o = valid ? tl / P.nxs : 0;
  const long long st = P.nxs;
  double2* g = spec + col + (long long)P.nxs * P.ny * o;
  auto src_of = [](int n) { return n < N / 2 ? 2 * n : 2 * (N - 1 - n) + 1; };  // the sample v_n holds
  auto mode_of = [](int k) { return PB == 2 ? N - 1 - k : k; };
  auto neg = [](double2 v) { return make_double2(-v.x, -v.y); };
  if (FWD) {
    double2 d[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) {
      const int s = src_of(t + R1 * n2);
      double2 v = valid ? g[(long long)s * st] : make_double2(0.0, 0.0);
      if (PB == 2 && (s & 1) == 0) v = neg(v);
      d[n2] = v;
    }
    F::fwdA(d, sb, se, P.dct_tw, l, t);
    __syncthreads();
    i2 xk[KQ][R1];
    const int ec = F::fwdB(xk, sb, se, l, t);  // xk[q][k1] = V[k2 + R2 k1], k2 = t + T q
    __syncthreads();
#pragma unroll
    for (int q = 0; q < KQ; ++q)
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) sb[(t + T * q + R2 * k1) * LPC + l] = xk[q][k1];
    __syncthreads();
    const FxOut fo = fx_out(ec);
    if (valid) {
      for (int k = t; k <= N / 2; k += R1) {
        const i2 Uk = fx_cmul(sb[k * LPC + l], fx_ldg(P.dct_wf + k));
        const i2 Um = fx_cmul(sb[((N - k) % N) * LPC + l], fx_ldg(P.dct_wf + (N - k)));
        g[(long long)mode_of(k) * st] = fx_to(i2{Uk.x - Um.y, Uk.y + Um.x}, fo, c);
        if (k != 0 && k != N / 2)
          g[(long long)mode_of(N - k) * st] = fx_to(i2{Um.x - Uk.y, Um.y + Uk.x}, fo, c);
      }
      if (fo.odd)
        for (int k = t; k <= N / 2; k += R1) {
          fx_rescale(g[(long long)mode_of(k) * st], fo);
          if (k != 0 && k != N / 2) fx_rescale(g[(long long)mode_of(N - k) * st], fo);
        }
    }
  } else {
    double2 d[KQ][R1];
#pragma unroll
    for (int q = 0; q < KQ; ++q)
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) {
        const int k = t + T * q + R2 * k1;
        const double2 X = valid ? g[(long long)mode_of(k) * st] : make_double2(0.0, 0.0);
        const double2 Xm = (valid && k != 0) ? g[(long long)mode_of(N - k) * st] : make_double2(0.0, 0.0);
        d[q][k1] = make_double2(fadd(c, X.x, Xm.y), fsub(c, X.y, Xm.x));  // X_k - i X_{N-k}
      }
    i2 xk[KQ][R1];
    const int eb = F::block(d, xk) - ilog2c(N);
#pragma unroll
    for (int q = 0; q < KQ; ++q)
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) xk[q][k1] = fx_cmul(xk[q][k1], fx_ldg(P.dct_wi + (t + T * q + R2 * k1)));
    F::invA(xk, eb, sb, se, P.dct_tw, l, t);
    __syncthreads();
    i2 x[R2];
    const FxOut fo = fx_out(F::invB(x, sb, se, l, t));
#pragma unroll
    for (int b = 0; b < R2; ++b) {
      const int s = src_of(t + R1 * b);
      double2 v = fx_to(x[b], fo, c);
      if (PB == 2 && (s & 1) == 0) v = neg(v);
      if (valid) g[(long long)s * st] = v;
    }
    if (fo.odd && valid)
#pragma unroll 1
      for (int b = 0; b < R2; ++b) fx_rescale(g[(long long)src_of(t + R1 * b) * st], fo);
  }
}

// The x transform of a wall x axis through the same FFT-based DCT: two real
// x lines (rows 2l and 2l+1 of a CTA's 2 LPC rows, row = (j-1) + ny (k-1))
// are the real and imaginary parts of one complex line.  Both passes stage
// the rows in shared memory as pairs, pr[l (N+1) + n] = (row 2l, row 2l+1) at
// sample or mode n (stride N+1 keeps the per-pair reads conflict-free), so
// the global side moves whole rows with coalesced accesses.  A packed
// spectrum row read as doubles is the modes in order.
// Forward, in place: the real rows in spec (block blk takes rows 2 LPC blk ..)
// become their packed modes.
template <int N, int LPC_ = lpc<N>()>
constexpr size_t dct_x_smem() { return YZ<N, LPC_>::kSmem + (size_t)LPC_ * (N + 1) * sizeof(double2); }

template <int N, int PB, int LPC_ = lpc<N>()>
__device__ __forceinline__ void dct_x_fwd_body(const FftPlan& P, double2* spec, double2* smem, int blk, int l, int t,
                                               const FOne& c) {
  using F = YZ<N, LPC_>;
  constexpr int LPC = F::LPC, R1 = F::R1, R2 = F::R2, T = F::T, KQ = F::KQ, PS = N + 1;
  i2* sb = reinterpret_cast<i2*>(smem);
  double2* pr = smem + N * LPC;
  FxExp* se = reinterpret_cast<FxExp*>(pr + LPC * PS);
  double* prd = reinterpret_cast<double*>(pr);
  const int nrows = P.ny * P.nz;
  const int row0 = blk * 2 * LPC;
  const int tid = t * LPC + l, nth = LPC * R1;
  double* out = reinterpret_cast<double*>(spec);
  for (int e = tid; e < 2 * LPC * N; e += nth) {
    const int rr = e / N, i = e % N, row = row0 + rr;
    prd[2 * PS * (rr >> 1) + 2 * i + (rr & 1)] = row < nrows ? out[(long long)N * row + i] : 0.0;
  }
  __syncthreads();
  auto src_of = [](int n) { return n < N / 2 ? 2 * n : 2 * (N - 1 - n) + 1; };
  auto mode_of = [](int k) { return PB == 2 ? N - 1 - k : k; };
  {
    double2 d[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) {
      const int s = src_of(t + R1 * n2);
      double2 v = pr[l * PS + s];
      if (PB == 2 && (s & 1) == 0) v = make_double2(-v.x, -v.y);
      d[n2] = v;
    }
    F::fwdA(d, sb, se, P.dctx_tw, l, t);
  }
  __syncthreads();
  i2 xk[KQ][R1];
  const int ec = F::fwdB(xk, sb, se, l, t);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < KQ; ++q)
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) sb[(t + T * q + R2 * k1) * LPC + l] = xk[q][k1];
  __syncthreads();
  const FxOut fo = fx_out(ec);
  for (int k = t; k <= N / 2; k += R1) {
    const i2 Uk = fx_cmul(sb[k * LPC + l], fx_ldg(P.dctx_wf + k));
    const i2 Um = fx_cmul(sb[((N - k) % N) * LPC + l], fx_ldg(P.dctx_wf + (N - k)));
    pr[l * PS + mode_of(k)] = fx_to(i2{Uk.x - Um.y, Uk.y + Um.x}, fo, c);
    if (k != 0 && k != N / 2) pr[l * PS + mode_of(N - k)] = fx_to(i2{Um.x - Uk.y, Um.y + Uk.x}, fo, c);
  }
  if (fo.odd)
    for (int k = t; k <= N / 2; k += R1) {
      fx_rescale(pr[l * PS + mode_of(k)], fo);
      if (k != 0 && k != N / 2) fx_rescale(pr[l * PS + mode_of(N - k)], fo);
    }
  __syncthreads();
  for (int e = tid; e < 2 * LPC * N; e += nth) {
    const int rr = e / N, i = e % N, row = row0 + rr;
    if (row < nrows) out[(long long)N * row + i] = prd[2 * PS * (rr >> 1) + 2 * i + (rr & 1)];
  }
}

// Inverse: packed modes of the rows of block blk -> dp slots 1..nx.
template <int N, int PB, int LPC_ = lpc<N>()>
__device__ __forceinline__ void dct_x_inv_body(const FftPlan& P, const double2* __restrict__ spec, double* dp,
                                               const Layout& L, double2* smem, int blk, int l, int t, const FOne& c) {
  using F = YZ<N, LPC_>;
  constexpr int LPC = F::LPC, R1 = F::R1, R2 = F::R2, T = F::T, KQ = F::KQ, PS = N + 1;
  i2* sb = reinterpret_cast<i2*>(smem);
  double2* pr = smem + N * LPC;
  FxExp* se = reinterpret_cast<FxExp*>(pr + LPC * PS);
  double* prd = reinterpret_cast<double*>(pr);
  const int nrows = P.ny * P.nz;
  const int row0 = blk * 2 * LPC;
  const int tid = t * LPC + l, nth = LPC * R1;
  const double* in = reinterpret_cast<const double*>(spec);
  for (int e = tid; e < 2 * LPC * N; e += nth) {
    const int rr = e / N, i = e % N, row = row0 + rr;
    prd[2 * PS * (rr >> 1) + 2 * i + (rr & 1)] = row < nrows ? in[(long long)N * row + i] : 0.0;
  }
  __syncthreads();
  auto src_of = [](int n) { return n < N / 2 ? 2 * n : 2 * (N - 1 - n) + 1; };
  auto mode_of = [](int k) { return PB == 2 ? N - 1 - k : k; };
  {
    double2 d[KQ][R1];
#pragma unroll
    for (int q = 0; q < KQ; ++q)
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) {
        const int k = t + T * q + R2 * k1;
        const double2 X = pr[l * PS + mode_of(k)];
        const double2 Xm = k ? pr[l * PS + mode_of(N - k)] : make_double2(0.0, 0.0);
        d[q][k1] = make_double2(fadd(c, X.x, Xm.y), fsub(c, X.y, Xm.x));  // X_k - i X_{N-k}
      }
    i2 xk[KQ][R1];
    const int eb = F::block(d, xk) - ilog2c(N);
#pragma unroll
    for (int q = 0; q < KQ; ++q)
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) xk[q][k1] = fx_cmul(xk[q][k1], fx_ldg(P.dctx_wi + (t + T * q + R2 * k1)));
    F::invA(xk, eb, sb, se, P.dctx_tw, l, t);
  }
  __syncthreads();
  {
    i2 x[R2];
    const FxOut fo = fx_out(F::invB(x, sb, se, l, t));
#pragma unroll
    for (int b = 0; b < R2; ++b) {
      const int s = src_of(t + R1 * b);
      double2 v = fx_to(x[b], fo, c);
      if (PB == 2 && (s & 1) == 0) v = make_double2(-v.x, -v.y);
      pr[l * PS + s] = v;
    }
    if (fo.odd)
#pragma unroll 1
      for (int b = 0; b < R2; ++b) fx_rescale(pr[l * PS + src_of(t + R1 * b)], fo);
  }
  __syncthreads();
  for (int e = tid; e < 2 * LPC * N; e += nth) {
    const int rr = e / N, i = e % N, row = row0 + rr;
    if (row < nrows) dp[L.at(i + 1, 1 + row % P.ny, 1 + row / P.ny)] = prd[2 * PS * (rr >> 1) + 2 * i + (rr & 1)];
  }
}

}  // namespace
}  // namespace ns
