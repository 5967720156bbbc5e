// Fused predictor: convection (cal_conv, NS_functions.f90:53-158), diffusion
// (cal_diff, NS_functions.f90:161-210), pressure gradient, Euler/AB2/AB2-CN
// predictor and AB2 history update (big_periodic_3D.f90:340-423,
// re_simulation_sub_tstep_interBC_combine.f90:543-654), in one pass over HBM.
//
// The divergence-form convection is rebuilt from shared products.  With the
// factor 1/2 of every two-point mean folded into the constants:
//   SX[c]  = u[c] + u[c+1]                 (x-mean of u at cell c, times 2)
//   QXY    = (u[f,J-1] + u[f,J]) * (v[f-1,J] + v[f,J])   at x-face f, y-face J
//   conv_x = (SX[f]^2 - SX[f-1]^2)/(4dx) + (QXY[J+1]-QXY[J])/(4dy) + (QXZ[K+1]-QXZ[K])/(4dz)
// which is cal_conv's avg/product/diff sequence with the products shared
// between conv_x, conv_y and conv_z (uy*vx serves both conv_x and conv_y).
//
// Tiling: a CTA owns 32 x-cells by TY y-rows and marches along z through a
// chunk of planes.  Warp w (0..TY) is y-row j0-1+w; warp 0 only computes
// products: those of the low y-halo row and, in one extra pass with lane r
// on row r, the low x-halo position of every row.  Products are owned
// one-sided (cell a owns SX[a], and the face products at faces a+1), so an
// output cell needs products of its own and its lower neighbours only.
//
// The predictor itself (MODE 0) runs on block fixed-point integers
// (predict_fx_planes); the convection and the diffusion alone (the routine
// tier) and planes out of the fixed-point range run in FP64, every operation
// in FMA form (see ns_internal.cuh).
//
// What bounds it: the FP64 stencils issue 62.7 FP64 instructions a cell, one
// per 64 clocks and SM partition: 2.09 ms at 256^3, 83% of that pipe.  The
// integer stencils take about 950 integer issue clocks a warp of cells beside
// 12 FP64 instructions: 0.81 ms with the block exponents, half of the issue
// slots busy.  TY = 8 at three CTAs per SM (72 registers) leaves room to hold
// the next plane's and the history's loads in flight; TY = 16 at two CTAs (56
// registers) waited for them at 1.9 ms.  Exponents of whole x-y planes, from a
// pass of their own, without the test for cells far below them took 0.77 ms
// (128^3 0.123 against 0.135 now, 128^3 with walls 0.130 against 0.158, FP64
// 0.309) and lost the quiet cells' digits.
#include <algorithm>
#include <cstddef>
#include <cmath>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "ns_fixed.cuh"
#include "ns_internal.cuh"
#include "ns_kernels.cuh"

namespace ns {

namespace {

constexpr int TX = 32;
constexpr int TY = 8;
constexpr int KC = 16;       // planes per CTA of the FP64 launches, at most of the others
constexpr int SXW = TX + 8;  // smem row width: column c is x = i0-2+c; columns 1..34 (x in
                             // [i0-1, i0+32]) are read, 0..35 loaded (a 320-byte row)
constexpr int SYH = TY + 2;  // smem rows: y in [j0-1, j0+TY]
constexpr int PXW = TX + 1;  // product row width: x in [i0-1, i0+31]
constexpr int PYH = TY + 1;  // product rows: y in [j0-1, j0+TY-1]

constexpr int RING = 4;       // planes k-1, k, k+1 in use, k+2 in flight

__device__ __forceinline__ int clampi(int a, int lo, int hi) { return a < lo ? lo : (a > hi ? hi : a); }

struct PredSmem {
  double u[RING][SYH][SXW];
  double v[RING][SYH][SXW];
  double w[RING][SYH][SXW];
  double sx2[PYH][PXW];
  double sy2[PYH][PXW];
  double sz2[2][PYH][PXW];
  double qxy[PYH][PXW];
  double qxz[2][PYH][PXW];
  double qyz[2][PYH][PXW];
};

// The fixed-point stencils' planes: the same ring and products as integers.
constexpr int GRP = 16;      // cell planes of one block exponent
constexpr int NWARP = TY + 1;
struct FxPredSmem {
  long long f[3][RING][SYH][SXW];
  long long sx2[PYH][PXW];
  long long sy2[PYH][PXW];
  long long sz2[2][PYH][PXW];
  long long qxy[PYH][PXW];
  long long qxz[2][PYH][PXW];
  long long qyz[2][PYH][PXW];
};
struct FxTail {  // behind the planes
  unsigned part[3][NWARP];       // largest magnitude of each field, per warp
  unsigned quiet[TY][GRP][3];    // cells left to the FP64 stencils: lanes of row, plane and component
  unsigned short list[TY][64];   // those a row's warp works on
  unsigned long long bar[2];     // the tile loader's barriers
};
struct FxRaw {  // tile loader: two planes of doubles, each field's box on a 128-byte boundary
  double f[2][3][SYH][SXW];
};
static_assert(sizeof(double) * SYH * SXW % 128 == 0, "boxes of the tile loader stay 128-byte aligned");
static_assert(sizeof(FxPredSmem) == sizeof(PredSmem), "one shared-memory area serves both stencils");
static_assert(offsetof(FxTail, bar) % 8 == 0, "the barriers are 8-byte aligned");

// ---- tile loader (TMA): one thread fills a staging slot with three 40 x 10 x 1
// boxes (u, v, w) and arms the slot's mbarrier with their byte count ----
constexpr unsigned kTileBytes = 3u * SYH * SXW * sizeof(double);
constexpr int kWaitLimit = 1 << 20;                   // try_wait polls before a wait gives up
constexpr unsigned long long kWaitNs = 200000000ull;  // or 0.2 s of global time, whichever comes first

__device__ __forceinline__ unsigned sm_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sm_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(sm_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// Wait for the phase `parity` of a barrier; false once max_polls polls or
// max_ns of global time found it incomplete (the caller records the error).
__device__ __forceinline__ bool mbar_wait_for(unsigned long long* bar, unsigned parity, int max_polls,
                                              unsigned long long max_ns) {
  // the common case (the plane has landed) reads no timer: a %globaltimer
  // read is a long-latency special-register access on every plane's path
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (int it = 0; it < max_polls; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 63) == 63 && global_ns() - t0 > max_ns) break;
  }
  return false;
}
// The tile loader's wait: kWaitLimit polls or kWaitNs.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
  return mbar_wait_for(bar, parity, kWaitLimit, kWaitNs);
}

// Self-test of the bounded wait: one thread arms a barrier for 8 bytes that
// no copy will deliver and waits with the loader's wait code and a time limit
// of limit_ns.  When the wait gives up (the expected outcome) the thread
// delivers the 8 bytes itself (complete_tx), so the barrier's phase completes
// before the CTA exits; nothing is in flight at any time.
__global__ void wait_selftest_kernel(unsigned long long limit_ns, int* __restrict__ gave_up,
                                     unsigned long long* __restrict__ waited_ns) {
  __shared__ unsigned long long bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar);
  const unsigned b = sm_addr(&bar);
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(8u) : "memory");
  const unsigned long long t0 = global_ns();
  const bool ok = mbar_wait_for(&bar, 0, 1 << 22, limit_ns);
  *waited_ns = global_ns() - t0;
  if (!ok) asm volatile("mbarrier.complete_tx.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(8u) : "memory");
  *gave_up = ok ? 0 : 1;
}
// Fill staging slot s with plane k (clamped into the box) of u, v, w: x from slot
// i0-2 (tensor x = slot + 7: 8 (32 bx + 6) bytes, 16-byte aligned), y from
// row j0-1.  Positions past the field read zeros or row padding; only inactive
// positions use them.
__device__ __forceinline__ void tma_plane(FxRaw& S, FxTail& T, const CUtensorMap* mu, const CUtensorMap* mv,
                                          const CUtensorMap* mw, int nz, int i0, int j0, int k, int s) {
  const int kk = clampi(k, 0, nz + 1);
  const int x = i0 - 2 + 7, y = j0 - 1;
  const unsigned b = sm_addr(&T.bar[s]);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the slot's last readers are done (barrier)
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(kTileBytes) : "memory");
  const CUtensorMap* maps[3] = {mu, mv, mw};
  double* dst[3] = {&S.f[s][0][0][0], &S.f[s][1][0][0], &S.f[s][2][0][0]};
#pragma unroll
  for (int f = 0; f < 3; ++f)
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(sm_addr(dst[f])), "l"(reinterpret_cast<unsigned long long>(maps[f])), "r"(x), "r"(y), "r"(kk), "r"(b)
        : "memory");
}


// Start copying plane k (clamped into the box) of u, v, w into ring slot s
// (cp.async; the caller commits the group).  Each smem row is 18 16-byte
// copies of slots i0-2 .. i0+33: index 7 + i0 - 2 = 32 bx + 6 (plus whole
// rows and planes of 8-double multiples) keeps every source 16-byte aligned.
// Rows and planes are clamped into the box; past x = nx + 1 the copies read
// row padding (or the next row, or the field's tail padding), which only
// positions without an output use.
__device__ __forceinline__ void issue_plane(PredSmem& S, const Layout& L, const double* __restrict__ u,
                                            const double* __restrict__ v, const double* __restrict__ w, int i0,
                                            int j0, int k, int s) {
  constexpr int NV = (TX + 4) / 2;
  const int kk = clampi(k, 0, L.nz + 1);
  const int nthr = blockDim.x * blockDim.y;
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;
  for (int e = tid; e < NV * SYH; e += nthr) {
    const int xv = e % NV, yy = e / NV;
    const int gj = clampi(j0 - 1 + yy, 0, L.ny + 1);
    const long long g = L.at(i0 - 2 + 2 * xv, gj, kk);
    cp_async16(&S.u[s][yy][2 * xv], u + g);
    cp_async16(&S.v[s][yy][2 * xv], v + g);
    cp_async16(&S.w[s][yy][2 * xv], w + g);
  }
}

// Products owned by position (a, b) = smem (x = xa, y = yb) at plane k, using
// ring slots s0 (plane k) and s1 (plane k+1).  Results go to product index
// (py, px) = (yb, xa) where xa/yb are smem coordinates of the position.
__device__ __forceinline__ void products(PredSmem& S, const FOne& c, int xa, int yb, int s0, int s1, int pb) {
  // SX[a] = u[a] + u[a+1]  (plane k, row b)
  const double sx = fadd(c, S.u[s0][yb][xa + 1], S.u[s0][yb][xa + 1 + 1]);
  // SY[b] = v[b] + v[b+1]
  const double sy = fadd(c, S.v[s0][yb][xa + 1], S.v[s0][yb + 1][xa + 1]);
  // SZ[k] = w[k] + w[k+1]
  const double sz = fadd(c, S.w[s0][yb][xa + 1], S.w[s1][yb][xa + 1]);
  // QXY at (x-face a+1, y-face b+1): (u[a+1,b] + u[a+1,b+1]) * (v[a,b+1] + v[a+1,b+1])
  const double q1 = fmul(c, fadd(c, S.u[s0][yb][xa + 1 + 1], S.u[s0][yb + 1][xa + 1 + 1]),
                         fadd(c, S.v[s0][yb + 1][xa + 1], S.v[s0][yb + 1][xa + 1 + 1]));
  // QXZ at (x-face a+1, cell b, z-face k+1): (u[a+1] at k, k+1) * (w[a], w[a+1] at k+1)
  const double q2 = fmul(c, fadd(c, S.u[s0][yb][xa + 1 + 1], S.u[s1][yb][xa + 1 + 1]),
                         fadd(c, S.w[s1][yb][xa + 1], S.w[s1][yb][xa + 1 + 1]));
  // QYZ at (cell a, y-face b+1, z-face k+1): (v[a,b+1] at k, k+1) * (w[a,b], w[a,b+1] at k+1)
  const double q3 = fmul(c, fadd(c, S.v[s0][yb + 1][xa + 1], S.v[s1][yb + 1][xa + 1]),
                         fadd(c, S.w[s1][yb][xa + 1], S.w[s1][yb + 1][xa + 1]));
  S.sx2[yb][xa] = fmul(c, sx, sx);
  S.sy2[yb][xa] = fmul(c, sy, sy);
  S.sz2[pb][yb][xa] = fmul(c, sz, sz);
  S.qxy[yb][xa] = q1;
  S.qxz[pb][yb][xa] = q2;
  S.qyz[pb][yb][xa] = q3;
}

// Products for z-face k only (the warm-up plane): SZ at cell k-1 (planes
// k-1, k) and QXZ/QYZ at z-face k.  s0 = plane k-1, s1 = plane k.
__device__ __forceinline__ void products_zface(PredSmem& S, const FOne& c, int xa, int yb, int s0, int s1, int pb) {
  const double sz = fadd(c, S.w[s0][yb][xa + 1], S.w[s1][yb][xa + 1]);
  const double q2 = fmul(c, fadd(c, S.u[s0][yb][xa + 1 + 1], S.u[s1][yb][xa + 1 + 1]),
                         fadd(c, S.w[s1][yb][xa + 1], S.w[s1][yb][xa + 1 + 1]));
  const double q3 = fmul(c, fadd(c, S.v[s0][yb + 1][xa + 1], S.v[s1][yb + 1][xa + 1]),
                         fadd(c, S.w[s1][yb][xa + 1], S.w[s1][yb + 1][xa + 1]));
  S.sz2[pb][yb][xa] = fmul(c, sz, sz);
  S.qxz[pb][yb][xa] = q2;
  S.qyz[pb][yb][xa] = q3;
}

}  // namespace

// MODE: 0 predictor, 1 conv only (writes conv into us/vs/ws), 2 diffusion only.
// One tile (bx, by) of TX x TY faces marching over the z-chunk bz.
template <int SCHEME, bool FIRST, bool DPF, int MODE>
__device__ __forceinline__ void predict_body(const PredictArgs& a, PredSmem& S, int bx, int by, int k0, int k1) {
  const Layout L = a.L;
  const FOne c{a.one, a.mzero};
  const int lane = threadIdx.x;
  const int wy = threadIdx.y;  // 0..TY
  const int i0 = 1 + TX * bx;
  const int j0 = 1 + TY * by;
  // smem coordinates of this thread's position: x = i0-1+lane+1 -> xa = lane+1; y = j0-1+wy -> yb = wy
  const int xa = lane + 1;
  const int yb = wy;

  // Warm-up: planes k0-1 and k0 (one copy group) and k0+1 (a second one);
  // products at z-face k0 once the first group has landed.
  issue_plane(S, L, a.u, a.v, a.w, i0, j0, k0 - 1, (k0 - 1) & 3);
  issue_plane(S, L, a.u, a.v, a.w, i0, j0, k0, k0 & 3);
  cp_async_commit();
  issue_plane(S, L, a.u, a.v, a.w, i0, j0, k0 + 1, (k0 + 1) & 3);
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();
  if (MODE != 2) {
    products_zface(S, c, xa, yb, (k0 - 1) & 3, k0 & 3, (k0 - 1) & 1);
    // low x-halo position of every row, by warp 0 (one partially active pass)
    if (wy == 0 && lane <= TY) products_zface(S, c, 0, lane, (k0 - 1) & 3, k0 & 3, (k0 - 1) & 1);
  }

  const int i = i0 + lane;
  const int j = j0 - 1 + wy;
  const int nx = L.nx, ny = L.ny;
  const bool in_xy = (wy >= 1) && (i <= nx) && (j <= ny);
  const bool act_u = in_xy && (i >= a.ulo);
  const bool act_v = in_xy && (j >= a.vlo);

  for (int k = k0; k < k1; ++k) {
    const int s0 = k & 3, s1 = (k + 1) & 3, sm = (k + 3) & 3;  // planes k, k+1, k-1
    const int pb = k & 1, pbm = (k - 1) & 1;
    // plane k+1 has landed and every thread is done with plane k-2, whose
    // slot receives plane k+2 while this plane is computed
    cp_async_wait<0>();
    __syncthreads();
    if (k + 2 <= k1) issue_plane(S, L, a.u, a.v, a.w, i0, j0, k + 2, (k + 2) & 3);
    cp_async_commit();
    if (MODE != 2) {
      products(S, c, xa, yb, s0, s1, pb);
      if (wy == 0 && lane <= TY) products(S, c, 0, lane, s0, s1, pb);
    }
    __syncthreads();
    const bool act_w = (k >= a.wlo);
    if (in_xy) {
      const long long g = L.at(i, j, k);
      // ---- x-component at x-face i ----
      if (act_u) {
        const double uc = S.u[s0][yb][xa + 1];
        const double sWE = fadd(c, S.u[s0][yb][xa - 1 + 1], S.u[s0][yb][xa + 1 + 1]);
        const double sSN = fadd(c, S.u[s0][yb - 1][xa + 1], S.u[s0][yb + 1][xa + 1]);
        const double sBT = fadd(c, S.u[sm][yb][xa + 1], S.u[s1][yb][xa + 1]);
        double C = 0.0;
        if (MODE != 2) {
          const double dX = fsub(c, S.sx2[yb][xa], S.sx2[yb][xa - 1]);
          const double dY = fsub(c, S.qxy[yb][xa - 1], S.qxy[yb - 1][xa - 1]);
          const double dZ = fsub(c, S.qxz[pb][yb][xa - 1], S.qxz[pbm][yb][xa - 1]);
          C = fmul(c, dX, a.cx);
          C = fma(dY, a.cy, C);
          C = fma(dZ, a.cz, C);  // C = -conv_x
        }
        double out;
        if (MODE == 1) {
          out = -C;
        } else if (MODE == 2) {
          out = fma(a.ix2, sWE, fma(a.iy2, sSN, fma(a.iz2, sBT, fmul(c, a.lap0, uc))));
        } else {
          out = predictor_combine<SCHEME, FIRST>(a, c, uc, sWE, sSN, sBT, C, a.hx[g], a.hx, g);
          if (DPF) out = fma(a.gpx, fsub(c, __ldg(a.p + g), __ldg(a.p + g - 1)), out);
        }
        a.us[g] = out;
      }
      // ---- y-component at y-face j ----
      if (act_v) {
        const double vc = S.v[s0][yb][xa + 1];
        const double sWE = fadd(c, S.v[s0][yb][xa - 1 + 1], S.v[s0][yb][xa + 1 + 1]);
        const double sSN = fadd(c, S.v[s0][yb - 1][xa + 1], S.v[s0][yb + 1][xa + 1]);
        const double sBT = fadd(c, S.v[sm][yb][xa + 1], S.v[s1][yb][xa + 1]);
        double C = 0.0;
        if (MODE != 2) {
          const double dX = fsub(c, S.qxy[yb - 1][xa], S.qxy[yb - 1][xa - 1]);
          const double dY = fsub(c, S.sy2[yb][xa], S.sy2[yb - 1][xa]);
          const double dZ = fsub(c, S.qyz[pb][yb - 1][xa], S.qyz[pbm][yb - 1][xa]);
          C = fmul(c, dX, a.cx);
          C = fma(dY, a.cy, C);
          C = fma(dZ, a.cz, C);
        }
        double out;
        if (MODE == 1) {
          out = -C;
        } else if (MODE == 2) {
          out = fma(a.ix2, sWE, fma(a.iy2, sSN, fma(a.iz2, sBT, fmul(c, a.lap0, vc))));
        } else {
          out = predictor_combine<SCHEME, FIRST>(a, c, vc, sWE, sSN, sBT, C, a.hy[g], a.hy, g);
          if (DPF) out = fma(a.gpy, fsub(c, __ldg(a.p + g), __ldg(a.p + g - L.sy)), out);
        }
        a.vs[g] = out;
      }
      // ---- z-component at z-face k ----
      if (act_w) {
        const double wc = S.w[s0][yb][xa + 1];
        const double sWE = fadd(c, S.w[s0][yb][xa - 1 + 1], S.w[s0][yb][xa + 1 + 1]);
        const double sSN = fadd(c, S.w[s0][yb - 1][xa + 1], S.w[s0][yb + 1][xa + 1]);
        const double sBT = fadd(c, S.w[sm][yb][xa + 1], S.w[s1][yb][xa + 1]);
        double C = 0.0;
        if (MODE != 2) {
          const double dX = fsub(c, S.qxz[pbm][yb][xa], S.qxz[pbm][yb][xa - 1]);
          const double dY = fsub(c, S.qyz[pbm][yb][xa], S.qyz[pbm][yb - 1][xa]);
          const double dZ = fsub(c, S.sz2[pb][yb][xa], S.sz2[pbm][yb][xa]);
          C = fmul(c, dX, a.cx);
          C = fma(dY, a.cy, C);
          C = fma(dZ, a.cz, C);
        }
        double out;
        if (MODE == 1) {
          out = -C;
        } else if (MODE == 2) {
          out = fma(a.ix2, sWE, fma(a.iy2, sSN, fma(a.iz2, sBT, fmul(c, a.lap0, wc))));
        } else {
          out = predictor_combine<SCHEME, FIRST>(a, c, wc, sWE, sSN, sBT, C, a.hz[g], a.hz, g);
          if (DPF) out = fma(a.gpz, fsub(c, __ldg(a.p + g), __ldg(a.p + g - L.sz)), out);
        }
        a.ws[g] = out;
      }
    }
  }
  cp_async_wait<0>();  // nothing left in flight when the tile is done
}

// ---------------------------------------------------------------------------
// The predictor on block fixed-point integers (MODE 0)
// ---------------------------------------------------------------------------
// The cell planes 16 g + 1 .. 16 g + 16 of a tile form a block; the exponents
// of the largest magnitudes that its stencils read (planes 16 g .. 16 g + 17,
// one row and column around the tile), one per field, are its block exponents
// (tile_exponents).  They depend on the fields alone, so the results do not
// depend on how the box is cut into launches or chunks.  (Exponents of each
// plane's own three planes changed every few planes of a turbulent field, and
// every change is a new warm-up: 3.0 ms at 256^3.)  A velocity is rounded to
// 59 bits (exact down to 2^-6 of the largest), a two-point sum takes 60, a
// product 60 (its unit is 2^-60 of four times the largest velocity squared,
// rounded).  Per component the convection C and the viscous increment L are
// formed as integers (the axis coefficients in units of 2^-60), brought back
// to doubles, and combined with u itself and the AB2 history in FP64.
//
// What an integer lacks is a double's relative accuracy far below the block's
// largest value.  So a cell whose component is below 2^-6 of it in all of the
// 7 points of its stencil, or whose component times the largest velocity
// beside it is below 2^-9 of the block's, gets the FP64 stencils instead
// (cell_fp64): they are marked here and worked off behind the block's planes,
// 32 marked cells of a row at a time.  What is left has a rounding error, in
// units of the local velocity (product, for C), of 0.3 to 1 times that of the
// FP64 stencils in the mean over turbulent and Taylor-Green fields and jets
// beside quiet fluid, and of 4e-15 at most (theirs: 1e-15).  Of a turbulent
// field no cell in ten thousand is marked, of a Taylor-Green vortex one in
// fifty (the surroundings of its axes), of a quiet region beside a jet those
// in the jet's own tiles; a field that is zero in a whole block marks none.
//
// A block that reads an Inf, a NaN or a velocity beyond 2^250, or whose
// largest one is below 2^-250, takes the FP64 stencils altogether.
constexpr int kFxB = 59;                    // bits of a velocity
constexpr int kFxLo = 773, kFxHi = 1273;    // biased exponents of the fixed-point stencils
constexpr unsigned kQuietOwn = 1u << (kFxB - 32 - 6 - 1);            // of high words below 2^(kFxB - 32)
constexpr unsigned kQuietProduct = 1u << (2 * (kFxB - 32) - 32 - 9 - 2);  // of the product's high word
struct FxPlane {
  int e[3];      // biased block exponents of u, v, w
  unsigned least[3], least_product[3];  // high words (of products) below these: FP64 stencils
};

// Whether the stencils of an output read slot (i, j, k) of field f.  The other
// slots (most edges of the box; the extra slot of a wall axis) hold whatever
// the caller's arrays hold there, and must not set a block exponent.  With a
// the field's own axis and b another one: its ghosts along b are read beside
// the field's own faces [lo, n], the low ones also beside every face in
// [1, n + 1] when b's lowest face has an output.
__device__ __forceinline__ bool slot_read(const PredictArgs& a, int f, int i, int j, int k) {
  const int pos[3] = {i, j, k}, n[3] = {a.L.nx, a.L.ny, a.L.nz}, lo[3] = {a.ulo, a.vlo, a.wlo};
  const int p = f == 0 ? i : f == 1 ? j : k, np = f == 0 ? n[0] : f == 1 ? n[1] : n[2];
  const int lp = f == 0 ? lo[0] : f == 1 ? lo[1] : lo[2];
  int ghosts = 0, first = lp - 1, last = np + 1;
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    if (b == f) continue;
    const bool low = pos[b] == 0, high = pos[b] > n[b];
    ghosts += low || high;
    if (high || (low && lo[b] > 1)) {
      first = lp;
      last = np;
    } else if (low) {
      first = 1;
    }
  }
  return ghosts < 2 && p >= first && p <= last;
}

// This thread's two column pairs of a plane (of 3 fields x 10 rows x 18 pairs).
constexpr int NV = (TX + 4) / 2, NPAIR = 3 * NV * SYH, NTHR = TX * NWARP;
static_assert(NPAIR <= 2 * NTHR, "two pairs per thread cover a plane");
struct FxPairs {
  const double* src[2];
  int f[2], yy[2], xv[2];
  bool two;  // the second one is a pair of its own
};
__device__ __forceinline__ FxPairs tile_pairs(const PredictArgs& a, int i0, int j0) {
  FxPairs p;
  const int tid = threadIdx.x + TX * threadIdx.y;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int e = min(tid + q * NTHR, NPAIR - 1);
    p.f[q] = e / (NV * SYH);
    p.yy[q] = e / NV % SYH;
    p.xv[q] = e % NV;
    p.src[q] = (p.f[q] == 0 ? a.u : p.f[q] == 1 ? a.v : a.w) +
               a.L.at(i0 - 2 + 2 * p.xv[q], clampi(j0 - 1 + p.yy[q], 0, a.L.ny + 1), 0);
  }
  p.two = tid + NTHR < NPAIR;
  return p;
}

// The largest magnitudes (high word; 0 for zeros alone) of the tile's group g
// of planes, per field.  A pass of its own over planes that the stencils are
// about to read (they come from L2 then): six planes of a thread in flight.
__device__ __forceinline__ void tile_exponents(const PredictArgs& a, FxTail& T, int i0, int j0, int g,
                                               unsigned (&top)[3]) {
  const Layout& L = a.L;
  const FxPairs pr = tile_pairs(a, i0, j0);
  const int kg = GRP * g, np = min(GRP + 2, L.nz + 2 - kg);
  unsigned m[2] = {0u, 0u};
  // whether a pair's two slots are read: a bit for plane 0, plane 1, the other inner ones, nz + 1
  // (plane 1 apart for w, whose own axis this is)
  unsigned rd[2][2];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int i = i0 - 2 + 2 * pr.xv[q] + x, j = j0 - 1 + pr.yy[q];
      rd[q][x] = 0u;
      if (i < i0 - 1 || i > min(i0 + TX, L.nx + 1) || j > L.ny + 1) continue;
      rd[q][x] = (slot_read(a, pr.f[q], i, j, 0) ? 1u : 0u) | (slot_read(a, pr.f[q], i, j, 1) ? 2u : 0u) |
                 (slot_read(a, pr.f[q], i, j, 2) ? 4u : 0u) | (slot_read(a, pr.f[q], i, j, L.nz + 1) ? 8u : 0u);
    }
#pragma unroll 1
  for (int p0 = 0; p0 < np; p0 += 6) {
    double2 d[6][2];
#pragma unroll
    for (int p = 0; p < 6; ++p) {
      const long long o = L.sz * (long long)(kg + min(p0 + p, np - 1));
#pragma unroll
      for (int q = 0; q < 2; ++q) d[p][q] = *reinterpret_cast<const double2*>(pr.src[q] + o);
    }
#pragma unroll
    for (int p = 0; p < 6; ++p) {
      const int k = kg + min(p0 + p, np - 1);
      const unsigned plane = k == 0 ? 1u : k > L.nz ? 8u : k == 1 ? 2u : 4u;
      auto mag = [](double v) {
        return ((unsigned)__double2hiint(v) & 0x7fffffffu) | (__double2loint(v) != 0 ? 1u : 0u);
      };
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (rd[q][0] & plane) m[q] = max(m[q], mag(d[p][q].x));
        if (rd[q][1] & plane) m[q] = max(m[q], mag(d[p][q].y));
      }
    }
  }
#pragma unroll
  for (int f = 0; f < 3; ++f) {
    const unsigned r = __reduce_max_sync(0xffffffffu, max(pr.f[0] == f ? m[0] : 0u, pr.f[1] == f ? m[1] : 0u));
    if (threadIdx.x == 0) T.part[f][threadIdx.y] = r;
  }
  __syncthreads();
#pragma unroll
  for (int f = 0; f < 3; ++f) {
    top[f] = 0u;
#pragma unroll
    for (int w = 0; w < NWARP; ++w) top[f] = max(top[f], T.part[f][w]);
  }
}

// C (minus the convection) and the viscous increment of one component at one
// cell in FP64: f the component at its face, g and h the two others at the
// same slot; strides and coefficients in the order own axis, g's, h's.
struct CellFp {
  double C, Lv;
};
__device__ __noinline__ CellFp cell_fp64(const double* __restrict__ f, const double* __restrict__ g,
                                         const double* __restrict__ h, long long s0, long long s1, long long s2,
                                         double c0, double c1, double c2, double v0, double v1, double v2) {
  const double x = f[0], a0 = f[-s0], b0 = f[s0], a1 = f[-s1], b1 = f[s1], a2 = f[-s2], b2 = f[s2];
  CellFp r;
  r.C = ((x + b0) * (x + b0) - (a0 + x) * (a0 + x)) * c0;
  r.C = fma((x + b1) * (g[s1 - s0] + g[s1]) - (a1 + x) * (g[-s0] + g[0]), c1, r.C);
  r.C = fma((x + b2) * (h[s2 - s0] + h[s2]) - (a2 + x) * (h[-s0] + h[0]), c2, r.C);
  r.Lv = fma(v0, fma(-2.0, x, a0 + b0), fma(v1, fma(-2.0, x, a1 + b1), v2 * fma(-2.0, x, a2 + b2)));
  return r;
}

// Bits in use of a velocity's high word.
__device__ __forceinline__ unsigned hi_bits(long long v) { return (unsigned)abs((int)(v >> 32)); }

__device__ __forceinline__ void products_fx(FxPredSmem& S, int xa, int yb, int s0, int s1, int pb, bool zonly) {
  const long long (*U0)[SXW] = S.f[0][s0], (*U1)[SXW] = S.f[0][s1];
  const long long (*V0)[SXW] = S.f[1][s0], (*V1)[SXW] = S.f[1][s1];
  const long long (*W0)[SXW] = S.f[2][s0], (*W1)[SXW] = S.f[2][s1];
  const long long ue = U0[yb][xa + 2], vn = V0[yb + 1][xa + 1], wt = W1[yb][xa + 1];
  S.sz2[pb][yb][xa] = fx_sqr(W0[yb][xa + 1] + wt);
  S.qxz[pb][yb][xa] = fx_mulv(ue + U1[yb][xa + 2], wt + W1[yb][xa + 2]);
  S.qyz[pb][yb][xa] = fx_mulv(vn + V1[yb + 1][xa + 1], wt + W1[yb + 1][xa + 1]);
  if (zonly) return;
  S.sx2[yb][xa] = fx_sqr(U0[yb][xa + 1] + ue);
  S.sy2[yb][xa] = fx_sqr(V0[yb][xa + 1] + vn);
  S.qxy[yb][xa] = fx_mulv(ue + U0[yb + 1][xa + 2], vn + V0[yb + 1][xa + 2]);
}

// The cell planes [k0, k1) of one tile, all with the block exponents P.
template <int SCHEME, bool FIRST, bool DPF, bool ISO, bool TMA>
__device__ __forceinline__ void predict_fx_planes(const PredictArgs& a, FxPredSmem& S, FxTail& T, FxRaw* raw,
                                                  const FxPlane& P, int bx, int by, int k0, int k1, unsigned& phase,
                                                  bool& ok, const CUtensorMap* mu, const CUtensorMap* mv,
                                                  const CUtensorMap* mw) {
  const Layout& L = a.L;
  const FOne c{a.one, a.mzero};
  const int lane = threadIdx.x, wy = threadIdx.y;
  const int i0 = 1 + TX * bx, j0 = 1 + TY * by;
  const int xa = lane + 1, yb = wy;
  const int tid = lane + TX * wy;
  const bool producer = tid == 0;
  const FxPairs pr = tile_pairs(a, i0, j0);
  int dst[2], ee[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    dst[q] = (pr.f[q] * RING * SYH + pr.yy[q]) * SXW + 2 * pr.xv[q];
    ee[q] = pr.f[q] == 0 ? P.e[0] : pr.f[q] == 1 ? P.e[1] : P.e[2];
  }
  const bool two = pr.two;
  double2 r[2];
  auto fetch = [&](int k) {  // plane k on its way: into registers, or (tile loader) into its staging slot
    if (TMA) {
      if (producer) tma_plane(*raw, T, mu, mv, mw, L.nz, i0, j0, k, k & 1);
    } else {
      const long long o = L.sz * (long long)clampi(k, 0, L.nz + 1);
      r[0] = *reinterpret_cast<const double2*>(pr.src[0] + o);
      if (two) r[1] = *reinterpret_cast<const double2*>(pr.src[1] + o);
    }
  };
  auto convert = [&](int k) {  // and into the ring
    if (TMA) {
      ok = mbar_wait(&T.bar[k & 1], (phase >> (k & 1)) & 1u) && ok;
      phase ^= 1u << (k & 1);
    }
    long long* ring = &S.f[0][k & 3][0][0];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (q == 1 && !two) break;
      double2 d = r[q];
      if (TMA) {
        const int e = tid + q * NTHR;
        d = *reinterpret_cast<const double2*>(&raw->f[k & 1][e / (NV * SYH)][e / NV % SYH][2 * (e % NV)]);
      }
      *reinterpret_cast<longlong2*>(ring + dst[q]) = make_longlong2(fx_round<kFxB>(d.x, ee[q]), fx_round<kFxB>(d.y, ee[q]));
    }
  };
  // units: a velocity of field f is v 2^(e[f] - 1022 - kFxB), a product of fields f, g the product's
  // 2^60 more.  The terms of C along the axes differ by the advecting field, so fields of about the
  // same magnitude are summed as integers (at the largest one's unit); otherwise every term is
  // brought back by itself, so that a small term keeps its digits where the large one vanishes
  // (a shear layer u(y): du/dx = 0).  Likewise where the axes' coefficients differ by more than 4
  // (far): summed as integers, the term along an axis 16 times coarser is off by 1e-15 of itself, 1000
  // times coarser by 5e-11.
  const int em = max(P.e[0], max(P.e[1], P.e[2]));
  const bool far = !ISO && a.far;
  const bool apart = far || em - min(P.e[0], min(P.e[1], P.e[2])) > 1;
  FxW qw[3], vw[3];
  if (ISO) {
    vw[0] = fxw62(a.v60[0]);
  } else {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      qw[q] = fxw(a.q60[q] >> (apart ? 0 : em - P.e[q]));
      vw[q] = fxw(a.v60[q]);
    }
  }
  const int kP = 60 - 2 * (1022 + kFxB), kL = a.kv + (ISO ? 1 : 0) - 1022 - kFxB;
  // C of the differences of the products along x, y, z, and L of a component
  auto conv = [&](long long dx, long long dy, long long dz, int e) -> double {
    if (apart) {
      double t = fmul(c, fx_to_int(dx, e + P.e[0] + kP), a.cx);
      t = fma(fx_to_int(dy, e + P.e[1] + kP), a.cy, t);
      return fma(fx_to_int(dz, e + P.e[2] + kP), a.cz, t);
    }
    if (ISO) {
      auto at = [&](long long d, int n) { return n ? (d + 1) >> 1 : d; };
      return fmul(c, fx_to_int(at(dx, em - P.e[0]) + at(dy, em - P.e[1]) + at(dz, em - P.e[2]), e + em + kP), a.cx);
    }
    return fx_to_int(fx_mul(dx, qw[0]) + fx_mul(dy, qw[1]) + fx_mul(dz, qw[2]), e + em + kP + a.kq);
  };
  auto visc = [&](long long uc, long long we, long long sn, long long bt, int e) -> double {
    if (far) {  // the coarse axis' coefficient would have few digits beside the fine one's
      const int k = e - 1022 - kFxB;
      double t = fmul(c, fx_to_int(we - 2 * uc, k), SCHEME == 2 ? a.ca : a.kx);
      t = fma(fx_to_int(sn - 2 * uc, k), SCHEME == 2 ? a.cb : a.ky, t);
      return fma(fx_to_int(bt - 2 * uc, k), SCHEME == 2 ? a.cc : a.kz, t);
    }
    long long s;
    if (ISO) s = fx_mul62((we + sn + bt - 6 * uc + 1) >> 1, vw[0]);
    else s = fx_mul(we - 2 * uc, vw[0]) + fx_mul(sn - 2 * uc, vw[1]) + fx_mul(bt - 2 * uc, vw[2]);
    return fx_to_int(s, e + kL);
  };
  // (u* but for the pressure gradient, the new history)
  auto combine = [&](double uc, double Lv, double C, double prev) -> double2 {
    if (SCHEME == 2) {  // AB2-CN explicit half (big_periodic_3D.f90:398-423)
      double t = fma(FIRST ? a.dt : a.cC, C, fma(a.cu, uc, Lv));  // Euler start: nu/2 diff - conv (:400-408)
      if (!FIRST) t = fma(a.cP, prev, t);
      return make_double2(t, C);  // rhs_?_previous = -conv
    }
    const double rhs = fadd(c, Lv, C);  // nu*diff - conv
    const double h = SCHEME == 0 ? 0.0 : rhs;
    if (SCHEME == 1 && !FIRST) return make_double2(fma(a.e1, rhs, fma(a.e2, prev, uc)), h);  // AB2 (:369-396)
    return make_double2(fma(a.dt, rhs, uc), h);  // Euler, or the Euler start of AB2
  };

  // Warm-up: planes k0-1, k0, k0+1 in the ring, k0+2 on its way; products at z-face k0.
  fetch(k0 - 1);
  convert(k0 - 1);
  fetch(k0);
  convert(k0);
  if (TMA) __syncthreads();  // both staging slots are read
  fetch(k0 + 1);
  convert(k0 + 1);
  if (k0 + 2 <= k1) fetch(k0 + 2);
  __syncthreads();
  products_fx(S, xa, yb, (k0 - 1) & 3, k0 & 3, (k0 - 1) & 1, true);
  // low x-halo position of every row, by warp 0 (one partially active pass)
  if (wy == 0 && lane <= TY) products_fx(S, 0, lane, (k0 - 1) & 3, k0 & 3, (k0 - 1) & 1, true);

  const int i = i0 + lane, j = j0 - 1 + wy;
  const bool in_xy = (wy >= 1) && (i <= L.nx) && (j <= L.ny);
  const bool act_u = in_xy && (i >= a.ulo), act_v = in_xy && (j >= a.vlo);
  unsigned marked = 0;  // planes (from k0 on) with cells left to the FP64 stencils
  for (int k = k0; k < k1; ++k) {
    const int s0 = k & 3, s1 = (k + 1) & 3, sm = (k + 3) & 3;  // planes k, k+1, k-1
    const int pb = k & 1, pbm = (k - 1) & 1;
    const long long g = L.at(i, j, k);
    double uc = 0.0, vc = 0.0, wc = 0.0, hu = 0.0, hv = 0.0, hw = 0.0;  // this cell's, ahead of the products
    if (in_xy) {
      uc = __ldg(a.u + g);
      vc = __ldg(a.v + g);
      wc = __ldg(a.w + g);
      if (SCHEME != 0 && !FIRST) {
        hu = a.hx[g];
        hv = a.hy[g];
        hw = a.hz[g];
      }
    }
    __syncthreads();  // plane k+1 is in the ring and every thread is done with plane k-2, whose slot takes plane k+2
    if (TMA && k + 3 <= k1) fetch(k + 3);  // its staging slot held plane k+1
    if (k + 2 <= k1) convert(k + 2);
    if (!TMA && k + 3 <= k1) fetch(k + 3);
    products_fx(S, xa, yb, s0, s1, pb, false);
    if (wy == 0 && lane <= TY) products_fx(S, 0, lane, s0, s1, pb, false);
    __syncthreads();
    unsigned mark = 0;  // components left to the FP64 stencils
    if (in_xy) {
      unsigned bits[3];  // of the 7 points of a component's stencil
      double2 res[3];
      auto component = [&](int f, double own, double prev, auto convection) {
        const long long (*F)[SXW] = S.f[f][s0];
        const long long x = F[yb][xa + 1], xw = F[yb][xa], xe = F[yb][xa + 2], xs = F[yb - 1][xa + 1],
                        xn = F[yb + 1][xa + 1], xb = S.f[f][sm][yb][xa + 1], xt = S.f[f][s1][yb][xa + 1];
        bits[f] = hi_bits(x) | hi_bits(xw) | hi_bits(xe) | hi_bits(xs) | hi_bits(xn) | hi_bits(xb) | hi_bits(xt);
        const double Lv = visc(x, xw + xe, xs + xn, xb + xt, P.e[f]);
        res[f] = combine(own, Lv, convection(), prev);
      };
      component(0, uc, hu, [&]() {  // at x-face i
        return conv(S.sx2[yb][xa] - S.sx2[yb][xa - 1], S.qxy[yb][xa - 1] - S.qxy[yb - 1][xa - 1],
                    S.qxz[pb][yb][xa - 1] - S.qxz[pbm][yb][xa - 1], P.e[0]);
      });
      component(1, vc, hv, [&]() {  // at y-face j
        return conv(S.qxy[yb - 1][xa] - S.qxy[yb - 1][xa - 1], S.sy2[yb][xa] - S.sy2[yb - 1][xa],
                    S.qyz[pb][yb - 1][xa] - S.qyz[pbm][yb - 1][xa], P.e[1]);
      });
      component(2, wc, hw, [&]() {  // at z-face k
        return conv(S.qxz[pbm][yb][xa] - S.qxz[pbm][yb][xa - 1], S.qyz[pbm][yb][xa] - S.qyz[pbm][yb - 1][xa],
                    S.sz2[pb][yb][xa] - S.sz2[pbm][yb][xa], P.e[2]);
      });
      unsigned near = 0;  // the largest velocity, at the largest block exponent
#pragma unroll
      for (int f = 0; f < 3; ++f) near |= bits[f] >> min(em - P.e[f], 31);
      auto put = [&](int f, double* __restrict__ hist, double* __restrict__ star, long long sp, double gp) {
        if (bits[f] < P.least[f] || __umulhi(bits[f], near) < P.least_product[f]) {
          mark |= 1u << f;
          return;
        }
        hist[g] = res[f].y;
        star[g] = DPF ? fma(gp, fsub(c, __ldg(a.p + g), __ldg(a.p + g - sp)), res[f].x) : res[f].x;
      };
      if (act_u) put(0, a.hx, a.us, 1, a.gpx);
      if (act_v) put(1, a.hy, a.vs, L.sy, a.gpy);
      if (k >= a.wlo) put(2, a.hz, a.ws, L.sz, a.gpz);
    }
    if (__any_sync(0xffffffffu, mark)) {  // (never in warp 0)
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        const unsigned w = __ballot_sync(0xffffffffu, (mark >> f) & 1u);
        if (lane == 0) T.quiet[wy - 1][k - k0][f] = w;
      }
      marked |= 1u << (k - k0);
    }
  }
  // The marked cells of this warp's row, 32 at a time.
  __syncwarp();
  int n = 0, f = 3, plane = 0;
  while (marked || f < 3 || n > 0) {
    while (n < 32 && (marked || f < 3)) {
      if (f == 3) {
        plane = __ffs((int)marked) - 1;
        marked &= marked - 1;
        f = 0;
      }
      const unsigned w = T.quiet[wy - 1][plane][f];
      if ((w >> lane) & 1u)
        T.list[wy - 1][n + __popc(w & ((1u << lane) - 1u))] = (unsigned short)(lane | f << 5 | plane << 7);
      n += __popc(w);
      ++f;
    }
    __syncwarp();
    if (lane < n) {
      const int code = T.list[wy - 1][lane], q = (code >> 5) & 3;
      const long long g = L.at(i0 + (code & 31), j, k0 + (code >> 7));
      const double *fu = a.u + g, *fv = a.v + g, *fw = a.w + g;
      const double vx = SCHEME == 2 ? a.ca : a.kx, vy = SCHEME == 2 ? a.cb : a.ky, vz = SCHEME == 2 ? a.cc : a.kz;
      double* hist = q == 0 ? a.hx : q == 1 ? a.hy : a.hz;
      const double own = q == 0 ? *fu : q == 1 ? *fv : *fw;
      const double prev = SCHEME != 0 && !FIRST ? hist[g] : 0.0;
      const CellFp r = cell_fp64(q == 0 ? fu : q == 1 ? fv : fw, q == 0 ? fv : fu, q == 2 ? fv : fw,
                                 q == 0 ? 1 : q == 1 ? L.sy : L.sz, q == 0 ? L.sy : 1, q == 2 ? L.sy : L.sz,
                                 q == 0 ? a.cx : q == 1 ? a.cy : a.cz, q == 0 ? a.cy : a.cx, q == 2 ? a.cy : a.cz,
                                 q == 0 ? vx : q == 1 ? vy : vz, q == 0 ? vy : vx, q == 2 ? vy : vz);
      double2 out = combine(own, r.Lv, r.C, prev);
      if (DPF)
        out.x = fma(q == 0 ? a.gpx : q == 1 ? a.gpy : a.gpz,
                    fsub(c, __ldg(a.p + g), __ldg(a.p + g - (q == 0 ? 1 : q == 1 ? L.sy : L.sz))), out.x);
      hist[g] = out.y;
      (q == 0 ? a.us : q == 1 ? a.vs : a.ws)[g] = out.x;
    }
    __syncwarp();
    const unsigned short rest = T.list[wy == 0 ? 0 : wy - 1][32 + lane];
    __syncwarp();
    if (n > 32) T.list[wy - 1][lane] = rest;
    n = max(n - 32, 0);
    __syncwarp();
  }
}

// One tile (bx, by) over the cell planes [k0, k1), group by group.
template <int SCHEME, bool FIRST, bool DPF, bool ISO, bool TMA>
__device__ __forceinline__ void predict_fx_body(const PredictArgs& a, unsigned char* smem, int bx, int by, int k0,
                                                int k1, const CUtensorMap* mu = nullptr,
                                                const CUtensorMap* mv = nullptr, const CUtensorMap* mw = nullptr) {
  FxRaw* raw = reinterpret_cast<FxRaw*>(smem);
  FxPredSmem& S = *reinterpret_cast<FxPredSmem*>(smem + (TMA ? sizeof(FxRaw) : 0));
  FxTail& T = *reinterpret_cast<FxTail*>(reinterpret_cast<unsigned char*>(&S) + sizeof(FxPredSmem));
  const int tid = threadIdx.x + TX * threadIdx.y;
  const int g0 = (k0 - 1) / GRP, ng = (k1 - 2) / GRP - g0 + 1;
  unsigned phase = 0;  // tile loader: bit s is the parity of slot s's next phase
  bool ok = true;      // false once a wait gave up (recorded in a.err); every issued plane
                       // is still waited for (bounded), so none is in flight at exit
  if (TMA) {
    if (tid == 0) {
      mbar_init(&T.bar[0]);
      mbar_init(&T.bar[1]);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  __syncthreads();
  for (int gi = 0; gi < ng; ++gi) {
    const int ks = max(k0, GRP * (g0 + gi) + 1), ke = min(k1, GRP * (g0 + gi + 1) + 1);
    FxPlane P{};
    bool bad = !a.fixed;  // coefficients outside the fixed-point range: FP64 stencils everywhere
    if (a.fixed) {
      unsigned top[3];
      tile_exponents(a, T, 1 + TX * bx, 1 + TY * by, g0 + gi, top);
      int em = kFxLo;
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        P.e[f] = (int)(top[f] >> 20);
        P.least[f] = top[f] ? kQuietOwn : 0u;
        P.least_product[f] = top[f] ? kQuietProduct : 0u;
        bad = bad || P.e[f] > kFxHi || (P.e[f] < kFxLo && top[f] != 0u);
        em = max(em, P.e[f]);
      }
#pragma unroll
      for (int f = 0; f < 3; ++f)
        if (top[f] == 0u) P.e[f] = em;
    }
    if (bad) predict_body<SCHEME, FIRST, DPF, 0>(a, reinterpret_cast<PredSmem&>(S), bx, by, ks, ke);
    else predict_fx_planes<SCHEME, FIRST, DPF, ISO, TMA>(a, S, T, raw, P, bx, by, ks, ke, phase, ok, mu, mv, mw);
    __syncthreads();
  }
  if (TMA && !ok && a.err) atomicExch(a.err, 1);
}

// The planes of chunk bz.
__device__ __forceinline__ void chunk_planes(const PredictArgs& a, int bz, int& k0, int& k1) {
  const int kc = a.kc > 0 ? a.kc : KC;
  k0 = 1 + a.koff + kc * bz;
  k1 = min(k0 + kc, a.kend > 0 ? a.kend : a.L.nz + 1);
}

template <int SCHEME, bool FIRST, bool DPF, int MODE>
__global__ void __launch_bounds__(TX*(TY + 1)) predict_kernel(PredictArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int k0, k1;
  chunk_planes(a, blockIdx.z, k0, k1);
  predict_body<SCHEME, FIRST, DPF, MODE>(a, *reinterpret_cast<PredSmem*>(smem_raw), blockIdx.x, blockIdx.y, k0, k1);
}

template <int SCHEME, bool FIRST, bool DPF, bool ISO>
__global__ void __launch_bounds__(TX*(TY + 1), 3) predict_fx_kernel(PredictArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int k0, k1;
  chunk_planes(a, blockIdx.z, k0, k1);
  predict_fx_body<SCHEME, FIRST, DPF, ISO, false>(a, smem_raw, blockIdx.x, blockIdx.y, k0, k1);
}

// The same with the tile loader: the maps of a.u, a.v, a.w as kernel
// parameters, the staging slots 128-byte aligned in dynamic shared memory.
template <int SCHEME, bool FIRST, bool DPF, bool ISO>
__global__ void __launch_bounds__(TX*(TY + 1)) predict_tma_kernel(PredictArgs a, const __grid_constant__ CUtensorMap mu,
                                                                  const __grid_constant__ CUtensorMap mv,
                                                                  const __grid_constant__ CUtensorMap mw) {
  extern __shared__ __align__(16) unsigned char smem_tma[];  // base rounded up to 128 B below
  int k0, k1;
  chunk_planes(a, blockIdx.z, k0, k1);
  predict_fx_body<SCHEME, FIRST, DPF, ISO, true>(a, smem_tma + ((128u - (sm_addr(smem_tma) & 127u)) & 127u), blockIdx.x,
                                                 blockIdx.y, k0, k1, &mu, &mv, &mw);
}

// Batched: persistent CTAs walk the work items (subdomain, tile) of a batch.
template <int SCHEME, bool FIRST, bool DPF, bool ISO>
__global__ void __launch_bounds__(TX*(TY + 1), 3) predict_batch_kernel(const PredictArgs* __restrict__ tab,
                                                                       const BatchItem* __restrict__ items,
                                                                       int n_items) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const BatchItem w = items[it];
    // the subdomain's arguments in registers: a reference into shared memory
    // would be reloaded after every barrier of the plane loop
    const PredictArgs a = tab[w.sub];
    int k0, k1;
    chunk_planes(a, w.bz, k0, k1);
    predict_fx_body<SCHEME, FIRST, DPF, ISO, false>(a, smem_raw, w.bx, w.by, k0, k1);
    __syncthreads();
  }
}

constexpr size_t kFxSmem = sizeof(FxPredSmem) + sizeof(FxTail);
size_t predict_smem_bytes() { return kFxSmem; }

// The tile loader serves a launch whose u, v, w are the mapped fields.
static bool tma_serves(const PredTma* t, const PredictArgs& a) {
  return t && t->ready && a.u == t->pu && a.v == t->pv && a.w == t->pw;
}

void set_predict_fixed(PredictArgs& a, int scheme) {
  const double c[3] = {a.cx, a.cy, a.cz};
  const double v[3] = {scheme == 2 ? a.ca : a.kx, scheme == 2 ? a.cb : a.ky, scheme == 2 ? a.cc : a.kz};
  auto scale = [](const double (&x)[3], long long (&q)[3], int& k, int below) {  // largest in [2^-below-1, 2^-below)
    const double m = std::max(std::fabs(x[0]), std::max(std::fabs(x[1]), std::fabs(x[2])));
    k = 0;
    for (int i = 0; i < 3; ++i) q[i] = 0;
    if (!(m > 0.0)) return m == 0.0;
    if (!std::isfinite(x[0]) || !std::isfinite(x[1]) || !std::isfinite(x[2])) return false;
    k = std::ilogb(m) + 1 + below;
    for (int i = 0; i < 3; ++i) q[i] = std::llrint(std::ldexp(x[i], 60 - k));
    return std::abs(k) <= 200;
  };
  const bool okc = scale(c, a.q60, a.kq, 0), okv = scale(v, a.v60, a.kv, 1);
  a.fixed = okc && okv;
  auto spread = [](const double (&x)[3]) {
    const double lo = std::min(std::fabs(x[0]), std::min(std::fabs(x[1]), std::fabs(x[2])));
    return 4.0 * lo < std::max(std::fabs(x[0]), std::max(std::fabs(x[1]), std::fabs(x[2])));
  };
  a.far = spread(c) || spread(v);
  a.iso = c[0] == c[1] && c[0] == c[2] && v[0] == v[1] && v[0] == v[2];
}

// Planes per CTA: a chunk's cost is its planes plus about two (its first
// planes and the products of its first face), and three CTAs share an SM, so
// the depth with the fewest waves x (depth + 2) is taken, of those that
// divide a group.  At 256^3 that is 16 (4096 CTAs), at 64^3 4 (256 CTAs), at
// 32^3 1 (128 CTAs).  With 16 planes a CTA at every size the 64^3 predictor
// took 0.180 ms (now 0.034), the 32^3 one 0.165 (0.017).
int predict_chunk(const std::vector<std::pair<long long, int>>& boxes) {
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return KC;
  const long long slots = 3LL * std::max(1, nsm);
  int best = KC;
  long long cost = -1;
  for (int kc = 1; kc <= GRP; kc *= 2) {
    long long ctas = 0;
    for (const auto& b : boxes) ctas += b.first * ((b.second + kc - 1) / kc);
    const long long t = (ctas + slots - 1) / slots * (kc + 2);
    if (cost < 0 || t <= cost) {
      cost = t;
      best = kc;
    }
  }
  return best;
}

template <typename K, typename... A>
static cudaError_t launch_smem(K kern, dim3 grid, size_t sm, cudaStream_t st, const A&... args) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  kern<<<grid, dim3(TX, TY + 1), sm, st>>>(args...);
  return cudaGetLastError();
}

template <int SCHEME, bool FIRST, bool DPF>
static cudaError_t launch_grid(const PredictArgs& b, dim3 grid, cudaStream_t st, const PredTma* tma) {
  if (tma_serves(tma, b)) {
    const size_t sm = kFxSmem + sizeof(FxRaw) + 128;
    if (b.iso) return launch_smem(predict_tma_kernel<SCHEME, FIRST, DPF, true>, grid, sm, st, b, tma->u, tma->v, tma->w);
    return launch_smem(predict_tma_kernel<SCHEME, FIRST, DPF, false>, grid, sm, st, b, tma->u, tma->v, tma->w);
  }
  if (b.iso) return launch_smem(predict_fx_kernel<SCHEME, FIRST, DPF, true>, grid, kFxSmem, st, b);
  return launch_smem(predict_fx_kernel<SCHEME, FIRST, DPF, false>, grid, kFxSmem, st, b);
}

static dim3 tile_grid(const Layout& L, int planes, int kc) {
  return dim3((L.nx + TX - 1) / TX, (L.ny + TY - 1) / TY, (planes + kc - 1) / kc);
}

template <int SCHEME, bool FIRST, bool DPF>
static cudaError_t launch_t(const PredictArgs& a, cudaStream_t st, const PredTma* tma) {
  PredictArgs b = a;
  const dim3 t = tile_grid(a.L, a.L.nz, 1);
  b.kc = predict_chunk({{(long long)t.x * t.y, a.L.nz}});
  b.koff = b.kend = 0;
  return launch_grid<SCHEME, FIRST, DPF>(b, tile_grid(a.L, a.L.nz, b.kc), st, tma);
}

// Convection (mode 1) or diffusion (mode 2) alone, in FP64, in chunks as the predictor's: with 16
// planes a CTA the 128^3 convection, 512 CTAs on 456 places, took 204 us (192 in the former 16-row tiles), now 179; 32^3 62 and 8.
template <int MODE>
static cudaError_t launch_mode(const PredictArgs& a, cudaStream_t st) {
  PredictArgs b = a;
  const dim3 t = tile_grid(a.L, a.L.nz, 1);
  b.kc = predict_chunk({{(long long)t.x * t.y, a.L.nz}});
  b.koff = b.kend = 0;
  return launch_smem(predict_kernel<0, false, false, MODE>, tile_grid(a.L, a.L.nz, b.kc), sizeof(PredSmem), st, b);
}

int predict_chunk_planes() { return KC; }

cudaError_t launch_wait_selftest(unsigned long long limit_ns, int* gave_up, unsigned long long* waited_ns,
                                 cudaStream_t st) {
  wait_selftest_kernel<<<1, 32, 0, st>>>(limit_ns, gave_up, waited_ns);
  return cudaGetLastError();
}

template <int SCHEME, bool FIRST, bool DPF>
static cudaError_t launch_planes_t(PredictArgs b, cudaStream_t st, int p0, int p1, int kc, const PredTma* tma) {
  b.kc = kc;
  b.koff = p0 - 1;
  b.kend = p1;
  return launch_grid<SCHEME, FIRST, DPF>(b, tile_grid(b.L, p1 - p0, kc), st, tma);
}

cudaError_t launch_predict_planes(PredictArgs a, int scheme, bool first, bool dpf, int p0, int p1, int kc,
                                  cudaStream_t st, const PredTma* tma) {
  if (p0 < 1 || p1 > a.L.nz + 1 || p0 > p1 || kc < 1 || kc > 2 * GRP) return cudaErrorInvalidValue;
  if (p0 == p1) return cudaSuccess;
#define NS_PRED_PCASE(S, F, D) \
  if (scheme == S && first == F && dpf == D) return launch_planes_t<S, F, D>(a, st, p0, p1, kc, tma);
  NS_PRED_PCASE(0, false, false) NS_PRED_PCASE(0, false, true) NS_PRED_PCASE(0, true, false) NS_PRED_PCASE(0, true, true)
  NS_PRED_PCASE(1, false, false) NS_PRED_PCASE(1, false, true) NS_PRED_PCASE(1, true, false) NS_PRED_PCASE(1, true, true)
  NS_PRED_PCASE(2, false, false) NS_PRED_PCASE(2, false, true) NS_PRED_PCASE(2, true, false) NS_PRED_PCASE(2, true, true)
#undef NS_PRED_PCASE
  return cudaErrorInvalidValue;
}

cudaError_t launch_predict(const PredictArgs& a, int scheme, bool first, bool dpf, int mode, cudaStream_t st,
                           const PredTma* tma) {
  if (mode == 1) return launch_mode<1>(a, st);
  if (mode == 2) return launch_mode<2>(a, st);
#define NS_PRED_CASE(S, F, D) \
  if (scheme == S && first == F && dpf == D) return launch_t<S, F, D>(a, st, tma);
  NS_PRED_CASE(0, false, false) NS_PRED_CASE(0, false, true) NS_PRED_CASE(0, true, false) NS_PRED_CASE(0, true, true)
  NS_PRED_CASE(1, false, false) NS_PRED_CASE(1, false, true) NS_PRED_CASE(1, true, false) NS_PRED_CASE(1, true, true)
  NS_PRED_CASE(2, false, false) NS_PRED_CASE(2, false, true) NS_PRED_CASE(2, true, false) NS_PRED_CASE(2, true, true)
#undef NS_PRED_CASE
  return cudaErrorInvalidValue;
}

bool make_pred_tma(PredTma& t, const Layout& L, const double* u, const double* v, const double* w) {
  t = PredTma{};
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q{};
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !fn)
    return false;
  auto encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  // element (x, y, z) of the tensor is slot (x - 7, y, z): index 7 + slot + sy*y + sz*z
  const cuuint64_t dims[3] = {(cuuint64_t)L.px, (cuuint64_t)(L.ny + 2), (cuuint64_t)(L.nz + 2)};
  const cuuint64_t strides[2] = {(cuuint64_t)L.sy * sizeof(double), (cuuint64_t)L.sz * sizeof(double)};
  const cuuint32_t box[3] = {(cuuint32_t)SXW, (cuuint32_t)SYH, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const double* f[3] = {u, v, w};
  CUtensorMap* m[3] = {&t.u, &t.v, &t.w};
  for (int i = 0; i < 3; ++i)
    if (encode(m[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double*>(f[i]), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return false;
  t.pu = u;
  t.pv = v;
  t.pw = w;
  t.ready = 1;
  return true;
}

void predict_tiles(const Layout& L, int kc, int& gx, int& gy, int& gz) {
  const dim3 g = tile_grid(L, L.nz, kc);
  gx = (int)g.x;
  gy = (int)g.y;
  gz = (int)g.z;
}

template <int SCHEME, bool FIRST, bool DPF, bool ISO>
static cudaError_t launch_bt(const PredictArgs* tab, const BatchItem* items, int n_items, int grid, cudaStream_t st) {
  auto kern = predict_batch_kernel<SCHEME, FIRST, DPF, ISO>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFxSmem);
  if (e != cudaSuccess) return e;
  if (grid <= 0) {
    int per_sm = 0, dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TX * (TY + 1), kFxSmem);
    grid = std::max(1, per_sm) * nsm;
  }
  grid = std::min(grid, n_items);
  if (grid <= 0) return cudaSuccess;
  kern<<<grid, dim3(TX, TY + 1), kFxSmem, st>>>(tab, items, n_items);
  return cudaGetLastError();
}

cudaError_t launch_predict_batch(const PredictArgs* tab, const BatchItem* items, int n_items, bool iso, int scheme,
                                 bool first, bool dpf, int grid, cudaStream_t st) {
#define NS_PRED_CASE(S, F, D)                                                         \
  if (scheme == S && first == F && dpf == D)                                          \
    return iso ? launch_bt<S, F, D, true>(tab, items, n_items, grid, st)              \
               : launch_bt<S, F, D, false>(tab, items, n_items, grid, st);
  NS_PRED_CASE(0, false, false) NS_PRED_CASE(0, false, true) NS_PRED_CASE(0, true, false) NS_PRED_CASE(0, true, true)
  NS_PRED_CASE(1, false, false) NS_PRED_CASE(1, false, true) NS_PRED_CASE(1, true, false) NS_PRED_CASE(1, true, true)
  NS_PRED_CASE(2, false, false) NS_PRED_CASE(2, false, true) NS_PRED_CASE(2, true, false) NS_PRED_CASE(2, true, true)
#undef NS_PRED_CASE
  return cudaErrorInvalidValue;
}

}  // namespace ns
