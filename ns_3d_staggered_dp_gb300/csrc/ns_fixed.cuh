// Block fixed-point arithmetic on the integer pipes.
//
// This part issues one FP64 warp instruction per 64 clocks and SM partition;
// a 64-bit integer add takes 3, a 60-bit fixed-point product 20, a double ->
// fixed conversion 26 (measured, one SM, 16 warps).  A chain of FP64 adds and
// multiplies over values of one block therefore runs several times faster as
// 64-bit integers that share one exponent, and the conversion back (two FP64
// instructions) runs beside it on the otherwise idle FP64 pipe.
//
// A block is what one thread holds of a line: its values are written as
// v * 2^eb, with eb taken from the largest exponent of the block so that the
// largest magnitude uses B bits (B up to 60, against the 53 of a double).
// Threads that exchange values publish (eb, p), where p is the smallest
// exponent at which the block's actual values fit the reader's B bits; the
// reader shifts everything to the largest p.  Sums are exact, each product
// is rounded once at the 2^-60 level of the block.  Against 128-bit sums the
// relative L2 error of a transform of 16 to 512 points is 0.5e-16 to 1.5e-16,
// 0.2 to 0.7 of that of the FP64 transform it replaces, for noise, smooth,
// localised, one-signed and steeply decaying lines.
#pragma once

#include "ns_internal.cuh"

namespace ns {
namespace {

struct i2 {
  long long x, y;
};

// A constant |c| <= 1 in units of 2^-60, split at bit 30: c = h 2^30 + l, 0 <= l < 2^30.
struct FxW {
  int h, l;
};
__host__ __device__ constexpr FxW fxw(long long q60) {
  return FxW{(int)(q60 >> 30), (int)(q60 & ((1ll << 30) - 1))};
}
// One entry of a twiddle table: (re.h, re.l, im.h, im.l).
struct FxC {
  FxW re, im;
};
__device__ __forceinline__ FxC fx_ldg(const int4* t) {
  const int4 q = __ldg(t);
  return FxC{{q.x, q.y}, {q.z, q.w}};
}

__device__ __forceinline__ int fx_hi(long long a) { return (int)(a >> 30); }
__device__ __forceinline__ int fx_lo(long long a) { return (int)a & ((1 << 30) - 1); }
__device__ __forceinline__ long long fx_wide(int a, int b, long long c) { return (long long)a * b + c; }

// The middle sums start at half a unit, so that their shift rounds: a
// truncated product is biased, and a bias adds up along a line where
// rounding errors do not.  (The product of the two low parts, a quarter of
// a unit on average, is dropped.)
// a * w for |a| < 2^61.
__device__ __forceinline__ long long fx_mul(long long a, FxW w) {
  const int h = fx_hi(a), l = fx_lo(a);
  const long long t = fx_wide(l, w.h, fx_wide(h, w.l, 1ll << 29));
  return fx_wide(h, w.h, t >> 30);
}
// (a b) >> 60 of two variables below 2^61, rounded (the mean of the dropped
// product of the low parts included).
__device__ __forceinline__ long long fx_mulv(long long a, long long b) {
  const int ah = fx_hi(a), al = fx_lo(a), bh = fx_hi(b), bl = fx_lo(b);
  const long long t = fx_wide(al, bh, fx_wide(ah, bl, (1ll << 29) + (1ll << 28)));
  return fx_wide(ah, bh, t >> 30);
}
__device__ __forceinline__ long long fx_sqr(long long a) {
  const int ah = fx_hi(a), al = fx_lo(a);
  return fx_wide(ah, ah, fx_wide(ah, 2 * al, (1ll << 29) + (1ll << 28)) >> 30);
}
// a * w for |a| < 2^62 and |w| <= 1/2: the constant split at bit 29, its low part times 4.
__host__ __device__ constexpr FxW fxw62(long long q60) {
  return FxW{(int)(q60 >> 29), (int)((q60 & ((1ll << 29) - 1)) << 2)};
}
__device__ __forceinline__ long long fx_mul62(long long a, FxW w) {
  const int h = (int)(a >> 31), l = (int)a & 0x7fffffff;
  const long long t = fx_wide(l, w.h, fx_wide(h, w.l, 1ll << 30));
  return fx_wide(h, w.h, t >> 31);
}
// a * w and a * conj(w), complex, |a| < 2^61.
__device__ __forceinline__ i2 fx_cmul(i2 a, FxC w) {
  const int rh = fx_hi(a.x), rl = fx_lo(a.x), ih = fx_hi(a.y), il = fx_lo(a.y);
  const int nh = -ih, nl = -il;
  const long long t = fx_wide(nl, w.im.h, fx_wide(nh, w.im.l, fx_wide(rl, w.re.h, fx_wide(rh, w.re.l, 1ll << 29))));
  const long long s = fx_wide(il, w.re.h, fx_wide(ih, w.re.l, fx_wide(rl, w.im.h, fx_wide(rh, w.im.l, 1ll << 29))));
  return i2{fx_wide(nh, w.im.h, fx_wide(rh, w.re.h, t >> 30)), fx_wide(ih, w.re.h, fx_wide(rh, w.im.h, s >> 30))};
}
__device__ __forceinline__ i2 fx_cmulc(i2 a, FxC w) {
  const int rh = fx_hi(a.x), rl = fx_lo(a.x), ih = fx_hi(a.y), il = fx_lo(a.y);
  const int nh = -rh, nl = -rl;
  const long long t = fx_wide(il, w.im.h, fx_wide(ih, w.im.l, fx_wide(rl, w.re.h, fx_wide(rh, w.re.l, 1ll << 29))));
  const long long s = fx_wide(il, w.re.h, fx_wide(ih, w.re.l, fx_wide(nl, w.im.h, fx_wide(nh, w.im.l, 1ll << 29))));
  return i2{fx_wide(ih, w.im.h, fx_wide(rh, w.re.h, t >> 30)), fx_wide(ih, w.re.h, fx_wide(nh, w.im.h, s >> 30))};
}

// ---------------------------------------------------------------------------
// Blocks
// ---------------------------------------------------------------------------
// Exponents of a thread's block: its values are v 2^eb, and at exponent p
// they fit the next reader's bits.
struct FxExp {
  int eb, p;
};
constexpr int kFxNonfinite = 1 << 28;  // eb and p of a block that holds an Inf or a NaN

// Biased exponent of the largest magnitude (zeros and subnormals: 0).
template <int N>
__device__ __forceinline__ int fx_max_exp(const double (&d)[N]) {
  unsigned m = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) m = max(m, (unsigned)__double2hiint(d[i]) << 1);
  return (int)(m >> 21);
}
// d as an integer of B bits for biased exponent E, truncated; 0 or -1 when d's own exponent is larger.
template <int B>
__device__ __forceinline__ long long fx_from(double d, int E) {
  const int hi = __double2hiint(d);
  const unsigned long long m = ((unsigned long long)(unsigned)((hi & 0xfffff) | 0x100000) << 32) |
                               (unsigned)__double2loint(d);
  const unsigned s = min((unsigned)(E - ((hi >> 20) & 0x7ff)), 63u);
  const long long v = (long long)((m << (B - 53)) >> s), sg = (long long)(hi >> 31);
  return (v ^ sg) - sg;
}
// The same, rounded (half away from zero).
template <int B>
__device__ __forceinline__ long long fx_round(double d, int E) {
  const int hi = __double2hiint(d);
  const unsigned long long m = ((unsigned long long)(unsigned)((hi & 0xfffff) | 0x100000) << 32) |
                               (unsigned)__double2loint(d);
  const unsigned s = min((unsigned)(E - ((hi >> 20) & 0x7ff)), 63u);
  const long long v = (long long)(((m << (B - 53)) + ((1ull << s) >> 1)) >> s), sg = (long long)(hi >> 31);
  return (v ^ sg) - sg;
}
// The block's integers and its eb.  Blocks of very large or very small
// values (where the exponents of the way back could leave a double's range)
// are scaled by a power of two first; values below 2^-64 of the block's
// largest, its zeros among them, become 0.
template <int B, int N>
__device__ __forceinline__ int fx_block(double (&d)[N], long long (&v)[N]) {
  int E = fx_max_exp(d), adj = 0;
  if (E < 128 || E > 1900) {
    adj = E < 128 ? 512 : -512;
    const double s = E < 128 ? 0x1p512 : 0x1p-512;
    if (E != 0x7ff) {
#pragma unroll
      for (int i = 0; i < N; ++i) d[i] *= s;
      E = fx_max_exp(d);
    }
  }
  const int Ec = max(E, 64);
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = fx_round<B>(d[i], Ec);
  return E == 0x7ff ? kFxNonfinite : Ec - 1022 - B - adj;
}
// The same for complex values.
template <int B, int R>
__device__ __forceinline__ int fx_block2(const double2 (&d)[R], i2 (&v)[R]) {
  double a[2 * R];
  long long w[2 * R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    a[2 * r] = d[r].x;
    a[2 * r + 1] = d[r].y;
  }
  const int eb = fx_block<B>(a, w);
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = i2{w[2 * r], w[2 * r + 1]};
  return eb;
}

// Bits in use: the OR of all magnitudes, 32 high bits each.
__device__ __forceinline__ void fx_bits(unsigned& acc, i2 v) {
  const int a = (int)(v.x >> 32), b = (int)(v.y >> 32);
  acc |= (unsigned)(a ^ (a >> 31));
  acc |= (unsigned)(b ^ (b >> 31));
}
// What a block publishes for readers that take BR bits.
template <int BR>
__device__ __forceinline__ FxExp fx_publish(int eb, unsigned acc) {
  return FxExp{eb, eb >= kFxNonfinite / 2 ? eb : eb + max(64 - __clz((int)acc) - BR, 0)};
}
// A value of a block with exponent eb at the common exponent ec >= eb, rounded.
__device__ __forceinline__ i2 fx_align(i2 v, int eb, int ec) {
  const int s = min(ec - eb, 62);
  const long long half = (1ll << s) >> 1;
  return i2{(v.x + half) >> s, (v.y + half) >> s};
}

// ---------------------------------------------------------------------------
// Back to double: v 2^ec, rounded to nearest even.  The two 32-bit halves are
// placed in the mantissas of two doubles whose exponents carry ec; removing
// the two offsets and adding the halves takes two FP64 instructions, the
// first one exact.
// ---------------------------------------------------------------------------
struct FxOut {
  int ha, hb;     // high words of the two halves
  double noff;    // minus the offset (NaN for a line with an Inf or a NaN)
  bool odd;       // an extreme exponent: the stored results still take fx_rescale
  bool up;        // by 2^512 (else 2^-512)
};
__device__ __forceinline__ FxOut fx_out(int ec) {
  FxOut o;
  const bool bad = ec >= kFxNonfinite / 2;
  int e = bad ? 0 : ec;
  o.odd = e < -1000 || e > 850;
  o.up = e > 0;
  if (o.odd) e = max(min(e + (o.up ? -512 : 512), 850), -1000);
  o.ha = (1107 + e) << 20;
  o.hb = (1075 + e) << 20;
  o.noff = bad ? __hiloint2double(0x7ff80000, 0) : -__hiloint2double(o.ha, (int)0x80100000u);
  return o;
}
__device__ __forceinline__ double fx_to(long long v, const FxOut& o, const FOne& c) {
  const double a = __hiloint2double(o.ha, (int)(v >> 32) ^ (int)0x80000000u);
  const double b = __hiloint2double(o.hb, (int)v);
  return fadd(c, fadd(c, a, o.noff), b);
}
__device__ __forceinline__ double2 fx_to(i2 v, const FxOut& o, const FOne& c) {
  return make_double2(fx_to(v.x, o, c), fx_to(v.y, o, c));
}
// A second pass over stored results (a branch of its own: a predicated-off
// FP64 instruction would take its issue slot at every result).
__device__ __forceinline__ void fx_rescale(double2& r, const FxOut& o) {
  const double s = o.up ? 0x1p512 : 0x1p-512;
  r = make_double2(r.x * s, r.y * s);
}

// The same on the integer pipes, for kernels whose FP64 pipe is the busier
// one: |v| < 2^63, rounded half up, 33 clocks (the leading bit comes from the
// exponent of the 32-bit integer -> float conversion, which runs 4 times
// faster than the leading-zero count).  The result must be a normal number.
__device__ __forceinline__ double fx_to_int(long long v, int ec) {
  const int sg = (int)(v >> 32) >> 31;
  const long long sg64 = (long long)sg;
  const unsigned long long m = (unsigned long long)((v ^ sg64) - sg64);
  const unsigned mh = (unsigned)(m >> 32), ml = (unsigned)m;
  const unsigned w = mh ? mh : ml;
  const int up = (mh ? 157 : 189) - (__float_as_int(__uint2float_rz(w)) >> 23);  // leading bit to bit 62
  const unsigned long long q = ((m << (up & 63)) + 0x200) >> 10;
  const int hi = (int)(q >> 32) + ((ec + 1084 - up) << 20);  // the leading bit adds the missing 1
  return __hiloint2double(w ? hi | (sg & (int)0x80000000) : 0, (int)q);
}

// ---------------------------------------------------------------------------
// Register DFTs on integers
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int ilog2c(int n) { return n <= 1 ? 0 : 1 + ilog2c(n >> 1); }
__host__ __device__ constexpr int log2up(int n) { return n <= 1 ? 0 : 1 + log2up((n + 1) >> 1); }
__host__ __device__ constexpr int brevc(int i, int bits) {
  return bits == 0 ? 0 : (((i & 1) << (bits - 1)) | brevc(i >> 1, bits - 1));
}

__device__ __forceinline__ i2 operator+(i2 a, i2 b) { return i2{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ i2 operator-(i2 a, i2 b) { return i2{a.x - b.x, a.y - b.y}; }

// cos(k pi / 16) in units of 2^-60, k = 0..8
__host__ __device__ constexpr long long cos32_q60(int k) {
  return k == 0 ? 1152921504606846976ll : k == 1 ? 1130768441178740757ll : k == 2 ? 1065160580698383124ll
         : k == 3 ? 958619196450722178ll : k == 4 ? 815238614083298888ll : k == 5 ? 640528868967736374ll
         : k == 6 ? 441203958630471860ll : k == 7 ? 224923827593068887ll : 0ll;
}
// exp(-2 pi i q / 32), q in [0, 16)
__host__ __device__ constexpr FxC w32(int q) {
  return FxC{fxw(q <= 8 ? cos32_q60(q) : -cos32_q60(16 - q)), fxw(-(q <= 8 ? cos32_q60(8 - q) : cos32_q60(q - 8)))};
}

// DIT butterfly a' = a + W b, b' = a - W b with W = W32^Q (DIR = -1) or its
// conjugate (DIR = +1).
template <int Q, int DIR>
__device__ __forceinline__ void fx_bfly(i2& a, i2& b) {
  i2 y;
  if constexpr (Q == 0) {
    y = b;
  } else if constexpr (Q == 8) {  // -i forward, +i inverse
    y = DIR < 0 ? i2{b.y, -b.x} : i2{-b.y, b.x};
  } else if constexpr (Q == 4 || Q == 12) {  // sqrt(1/2) (+-1 -+ i)
    constexpr FxW sq = fxw(cos32_q60(4));
    const long long s = b.x + b.y, d = b.x - b.y;
    if constexpr (Q == 4) y = DIR < 0 ? i2{fx_mul(s, sq), -fx_mul(d, sq)} : i2{fx_mul(d, sq), fx_mul(s, sq)};
    else y = DIR < 0 ? i2{-fx_mul(d, sq), -fx_mul(s, sq)} : i2{-fx_mul(s, sq), fx_mul(d, sq)};
  } else {
    constexpr FxC w = w32(Q);
    y = DIR < 0 ? fx_cmul(b, w) : fx_cmulc(b, w);
  }
  const i2 a0 = a;
  a = a0 + y;
  b = a0 - y;
}

// Radix-2 in-place R-point DFT (R a power of two, R <= 32), natural order in and out.
// Every index is a template constant, so the array stays in registers.
template <int R, int I>
struct BitRev {
  static __device__ __forceinline__ void run(i2 (&x)[R]) {
    constexpr int J = brevc(I, ilog2c(R));
    if constexpr (J > I) {
      const i2 t = x[I];
      x[I] = x[J];
      x[J] = t;
    }
    BitRev<R, I + 1>::run(x);
  }
};
template <int R>
struct BitRev<R, R> {
  static __device__ __forceinline__ void run(i2 (&)[R]) {}
};
template <int R, int LEN, int S, int K, int DIR>
struct Bfly {  // butterfly K of group S of stage LEN, then the next one
  static __device__ __forceinline__ void run(i2 (&x)[R]) {
    fx_bfly<K*(32 / LEN), DIR>(x[S + K], x[S + K + LEN / 2]);
    if constexpr (K + 1 < LEN / 2) Bfly<R, LEN, S, K + 1, DIR>::run(x);
    else if constexpr (S + LEN < R) Bfly<R, LEN, S + LEN, 0, DIR>::run(x);
  }
};
template <int R, int LEN, int DIR>
struct Stage {
  static __device__ __forceinline__ void run(i2 (&x)[R]) {
    Bfly<R, LEN, 0, 0, DIR>::run(x);
    if constexpr (LEN < R) Stage<R, 2 * LEN, DIR>::run(x);
  }
};
template <int R, int DIR>
__device__ __forceinline__ void dft_pow2(i2 (&x)[R]) {
  BitRev<R, 0>::run(x);
  Stage<R, 2, DIR>::run(x);
}

// 3-point DFT: with s = a1 + a2, d = a1 - a2 and t = a0 - s/2,
// X0 = a0 + s, X1 = t - i (sqrt(3)/2) d, X2 = t + i (sqrt(3)/2) d (forward;
// the inverse takes the conjugate roots).
template <int DIR>
__device__ __forceinline__ void dft3(i2& a0, i2& a1, i2& a2) {
  constexpr FxW h3 = fxw(998459311558907194ll);  // sqrt(3)/2
  const i2 s = a1 + a2, d = a1 - a2;
  const i2 t{a0.x - (s.x >> 1), a0.y - (s.y >> 1)};
  const i2 g{fx_mul(d.y, h3), -fx_mul(d.x, h3)};  // -i h3 d
  a0 = a0 + s;
  a1 = DIR < 0 ? t + g : t - g;
  a2 = DIR < 0 ? t - g : t + g;
}

// 12-point DFT by the prime-factor (Good-Thomas) split 12 = 3 x 4, which
// needs no twiddles: 3-point DFTs over n1 of x[(4 n1 + 3 n2) mod 12] for each
// n2, then 4-point DFTs over n2, whose output k2 of row k1 is
// X[(4 k1 + 9 k2) mod 12] (9 = 3 x (3^-1 mod 4), 4 = 4 x (4^-1 mod 3)).
template <int DIR>
__device__ __forceinline__ void dft12(i2 (&x)[12]) {
  i2 y[4][3];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    i2 a0 = x[(3 * n2) % 12], a1 = x[(4 + 3 * n2) % 12], a2 = x[(8 + 3 * n2) % 12];
    dft3<DIR>(a0, a1, a2);
    y[n2][0] = a0;
    y[n2][1] = a1;
    y[n2][2] = a2;
  }
#pragma unroll
  for (int k1 = 0; k1 < 3; ++k1) {
    i2 z[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
    dft_pow2<4, DIR>(z);
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) x[(4 * k1 + 9 * k2) % 12] = z[k2];
  }
}

// In-place R-point DFT, natural order in and out: R a power of two up to 32,
// or 12.  The complex magnitude grows by at most R; the operands of its
// products stay below 2^61 when the inputs' components fit 60 - log2up(R) bits.
template <int R, int DIR>
__device__ __forceinline__ void dft(i2 (&x)[R]) {
  if constexpr (R == 12) dft12<DIR>(x);
  else dft_pow2<R, DIR>(x);
}

}  // namespace
}  // namespace ns
