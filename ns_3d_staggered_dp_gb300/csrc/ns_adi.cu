// Crank-Nicolson ADI line solves (big_periodic_3D.f90:425-489 with getrs on
// mat_CN; re_simulation_sub_tstep_interBC_combine.f90:656-701 with dttrsb on
// mat_CN_tridiagonal).
//
// All lines of a sweep share one matrix, so its LU factors (no pivoting) are
// precomputed on the host (ns_api.cu) and read as broadcast loads.  A sweep
// reads the lines from one buffer and writes them to another (fixed ping-pong
// roles, see ns_api.cu).
//
// A step's sweeps solve a line in chunks ("Chunked sweeps" below).  The whole
// lines that follow, one thread each, one FMA forward and one multiply + one
// FMA backward an unknown, serve the sweeps whose unscaled result is handed
// out (ns_adi, keep_sweeps), large viscous numbers, and the batch.
//
// y and z sweeps: a persistent kernel, lanes over consecutive x so every
// access of the forward and backward walks is coalesced, right-hand sides
// prefetched 8 unknowns ahead in registers.
// x sweep: the lines are contiguous, so a warp owns 32 lines and walks them
// in 32 x 32 blocks staged through shared memory (padded stride 33): every
// global access is a coalesced 256-byte row segment, each thread runs its
// recurrence from shared memory.
//
// Walls (bc 2, 4): the full line including the BC rows is solved; the BC
// rows' right-hand side is the sweep's face value (vel_bc_staggered_CN2,
// NS_functions.f90:313-410).
// Periodic (bc 1): the ghost rows of mat_CN only tie the ghosts to interior
// values, so the solve is reduced to the n interior unknowns, a tridiagonal
// system T plus corner entries, solved by Sherman-Morrison,
// x = y - (s0*y[0] + s1*y[n-1]) * z, with z = T^-1 u precomputed; z decays
// geometrically away from the ends, so the correction is applied only where
// |z| > 1e-18 max|z| (zA, zB).  The periodic copies (slot 0 <- slot n,
// slot n+1 <- slot 1) are then written, which is what the ghost rows of
// mat_CN produce.
#include <algorithm>

#include "ns_internal.cuh"
#include "ns_kernels.cuh"

namespace ns {

namespace {

template <int AXIS>
__device__ __forceinline__ void line_of(const Layout& L, int s1, int s2, long long& base, long long& st) {
  if (AXIS == 0) { base = L.at(0, s1, s2); st = 1; }
  else if (AXIS == 1) { base = L.at(s1, 0, s2); st = L.sy; }
  else { base = L.at(s1, s2, 0); st = L.sz; }
}

__device__ __forceinline__ int axis_n(const Layout& L, int axis) { return axis == 0 ? L.nx : (axis == 1 ? L.ny : L.nz); }

// Periodic correction on the end regions and the slot copies, or the carried
// slots of a wall line; x points at slot 0 of the destination line.
__device__ __forceinline__ void finish_line(const LineSys& S, const double* __restrict__ src, double* __restrict__ x,
                                            long long st, int nax, double x_first, double x_last) {
  const int m = S.hi - S.lo + 1;
  double* xl = x + (long long)S.lo * st;
  if (S.periodic) {
    const double g = fma(S.s0, x_first, S.s1 * x_last);
    for (int e = 0; e < S.zA; ++e) xl[(long long)e * st] = fma(-g, __ldg(S.z + e), xl[(long long)e * st]);
    for (int e = (S.zB > S.zA ? S.zB : S.zA); e < m; ++e)
      xl[(long long)e * st] = fma(-g, __ldg(S.z + e), xl[(long long)e * st]);
    x[0] = xl[(long long)(m - 1) * st];         // slot 0 <- slot n
    x[(long long)(nax + 1) * st] = xl[0];       // slot n+1 <- slot 1
  } else {
    for (int s = 0; s < S.lo; ++s) x[(long long)s * st] = src[(long long)s * st];
    for (int s = S.hi + 1; s <= nax + 1; ++s) x[(long long)s * st] = src[(long long)s * st];
  }
}

}  // namespace

// x sweep: a warp owns 32 consecutive lines (line t = j + (ny+2)(k - z0),
// across plane boundaries, so every warp is full) and walks them in blocks
// of 32 unknowns through shared memory.  Row l of a block is line t0 + l,
// whose 32-bit slot offset lane l holds and hands out by shuffle.
namespace {
constexpr int XW = 4;           // warps per CTA
constexpr int XB = 32;          // unknowns per block
constexpr int XS = 33;          // padded stride
}  // namespace

__global__ void __launch_bounds__(32 * XW) adi_x_kernel(AdiArgs a) {
  __shared__ double sh[XW][XB * XS];
  const int fld = blockIdx.z;
  const LineSys& S = a.sys[fld];
  const Layout L = a.L;
  const int n1 = L.ny + 2;
  const int nplanes = a.z1 > 0 ? a.z1 - a.z0 : L.nz + 2;
  const int nlines = n1 * nplanes;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int t0 = (blockIdx.x * XW + warp) * 32;
  if (t0 >= nlines) return;
  const int nl = min(32, nlines - t0);
  const int t = t0 + min(lane, nl - 1);  // lanes past the end repeat the last line (never stored)
  const int j = t % n1, k = a.z0 + t / n1;
  const int my_off = (int)L.at(S.lo, j, k);  // unknown 0 of this lane's line
  double* sb = sh[warp];
  const double* lf = S.l + S.pad;
  const double* di = S.dinv + S.pad;
  const double* cu = S.cu + S.pad;
  const int m = S.hi - S.lo + 1;
  const int nb = (m + XB - 1) / XB;
  const double* src = a.src[fld];
  double* dst = a.dst[fld];
  const bool act = lane < nl;
  const bool walls = !S.periodic;
  double face_lo = 0.0, face_hi = 0.0;
  if (walls && act) {
    const int plane = j + n1 * k;
    if (a.face_lo[fld]) face_lo = __ldg(a.face_lo[fld] + plane);
    if (a.face_hi[fld]) face_hi = __ldg(a.face_hi[fld] + plane);
  }
  // forward elimination, block by block; y' goes to dst
  double yp = 0.0;
  for (int b = 0; b < nb; ++b) {
    const int e0 = b * XB;
    const int ne = min(XB, m - e0);
#pragma unroll 8
    for (int l = 0; l < XB; ++l) {
      const int off = __shfl_sync(0xffffffffu, my_off, l);
      if (l < nl && lane < ne) sb[lane * XS + l] = __ldg(src + off + e0 + lane);
    }
    __syncwarp();
    if (walls) {  // the BC rows take the sweep's face values
      if (e0 == 0) sb[lane] = face_lo;
      if (m - 1 - e0 < XB) sb[(m - 1 - e0) * XS + lane] = face_hi;
    }
    if (act) {
      for (int q = 0; q < ne; ++q) {
        yp = fma(-__ldg(lf + e0 + q), yp, sb[q * XS + lane]);
        sb[q * XS + lane] = yp;
      }
    }
    __syncwarp();
#pragma unroll 8
    for (int l = 0; l < XB; ++l) {
      const int off = __shfl_sync(0xffffffffu, my_off, l);
      if (l < nl && lane < ne) dst[off + e0 + lane] = sb[lane * XS + l];
    }
    __syncwarp();
  }
  // back substitution, blocks in reverse (cu[m-1] = 0 starts the walk)
  double xn = 0.0, x_last = 0.0;
  for (int b = nb - 1; b >= 0; --b) {
    const int e0 = b * XB;
    const int ne = min(XB, m - e0);
#pragma unroll 8
    for (int l = 0; l < XB; ++l) {
      const int off = __shfl_sync(0xffffffffu, my_off, l);
      if (l < nl && lane < ne) sb[lane * XS + l] = dst[off + e0 + lane];
    }
    __syncwarp();
    if (act) {
      for (int q = ne - 1; q >= 0; --q) {
        xn = fma(-__ldg(cu + e0 + q), xn, sb[q * XS + lane] * __ldg(di + e0 + q));
        sb[q * XS + lane] = xn;
      }
      if (b == nb - 1) x_last = sb[(ne - 1) * XS + lane];
    }
    __syncwarp();
#pragma unroll 8
    for (int l = 0; l < XB; ++l) {
      const int off = __shfl_sync(0xffffffffu, my_off, l);
      if (l < nl && lane < ne) dst[off + e0 + lane] = sb[lane * XS + l];
    }
    __syncwarp();
  }
  if (act) {
    const long long base = L.at(0, j, k);
    finish_line(S, src + base, dst + base, 1, L.nx, xn, x_last);
  }
}

// Persistent line solver for every sweep axis: one thread per line, a grid
// of a few CTAs per SM walking all lines of the three fields.  The right-hand
// sides are prefetched PD unknowns ahead in registers (the recurrence itself
// only waits on its own FMA), and the forward intermediate y' is written to
// the destination line and read back by the backward walk; with only
// grid x 128 lines in flight that round trip stays in L2.
template <int AXIS, int PD>
__global__ void __launch_bounds__(128) adi_line_kernel(AdiArgs a) {
  const Layout L = a.L;
  const int n1 = (AXIS == 0) ? L.ny + 2 : L.nx + 2;
  // the y sweep may be limited to the lines of z slots [z0, z1)
  const int zlo = (AXIS == 1 && a.z1 > 0) ? a.z0 : 0;
  const int n2 = (AXIS == 2) ? L.ny + 2 : ((AXIS == 1 && a.z1 > 0) ? a.z1 - a.z0 : L.nz + 2);
  const int per_field = n1 * n2;
  const int total = 3 * per_field;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    const int fld = t / per_field;
    const int tl = t - fld * per_field;
    const LineSys& S = a.sys[fld];
    long long base, st;
    line_of<AXIS>(L, tl % n1, zlo + tl / n1, base, st);
    const double* __restrict__ src = a.src[fld] + base;
    double* __restrict__ dst = a.dst[fld] + base;
    const double* lf = S.l + S.pad;
    const double* di = S.dinv + S.pad;
    const double* cu = S.cu + S.pad;
    const int m = S.hi - S.lo + 1;
    const double* sl = src + (long long)S.lo * st;
    double* xl = dst + (long long)S.lo * st;
    double r_lo, r_hi;
    if (S.periodic) {
      r_lo = 0.0; r_hi = 0.0;
    } else {
      const int pl = tl + zlo * n1;  // index in the full face plane
      r_lo = a.face_lo[fld] ? __ldg(a.face_lo[fld] + pl) : 0.0;
      r_hi = a.face_hi[fld] ? __ldg(a.face_hi[fld] + pl) : 0.0;
    }
    const bool per = S.periodic != 0;
    auto rhs = [&](int e) -> double {
      if (e < 0 || e >= m) return 0.0;
      if (!per && e == 0) return r_lo;
      if (!per && e == m - 1) return r_hi;
      return sl[(long long)e * st];
    };
    // forward: y[0] = r[0], y[e] = r[e] - l[e] y[e-1]  (l[0] = 0)
    double rb[PD];
#pragma unroll
    for (int q = 0; q < PD; ++q) rb[q] = rhs(q);
    double yp = 0.0;
    for (int g = 0; g < m; g += PD) {
      double nb[PD];
#pragma unroll
      for (int q = 0; q < PD; ++q) nb[q] = rhs(g + PD + q);
#pragma unroll
      for (int q = 0; q < PD; ++q) {
        const int e = g + q;
        if (e < m) {
          yp = fma(-__ldg(lf + e), yp, rb[q]);
          xl[(long long)e * st] = yp;
        }
      }
#pragma unroll
      for (int q = 0; q < PD; ++q) rb[q] = nb[q];
    }
    // backward: x[m-1] = y dinv, x[e] = y[e] dinv[e] - cu[e] x[e+1]  (cu[m-1] = 0)
    auto yv = [&](int e) -> double { return e >= 0 ? xl[(long long)e * st] : 0.0; };
#pragma unroll
    for (int q = 0; q < PD; ++q) rb[q] = yv(m - 1 - q);
    double xn = 0.0, x_last = 0.0;
    for (int g = m - 1; g >= 0; g -= PD) {
      double nb[PD];
#pragma unroll
      for (int q = 0; q < PD; ++q) nb[q] = yv(g - PD - q);
#pragma unroll
      for (int q = 0; q < PD; ++q) {
        const int e = g - q;
        if (e >= 0) {
          xn = fma(-__ldg(cu + e), xn, rb[q] * __ldg(di + e));
          xl[(long long)e * st] = xn;
          if (e == m - 1) x_last = xn;
        }
      }
#pragma unroll
      for (int q = 0; q < PD; ++q) rb[q] = nb[q];
    }
    finish_line(S, src, dst, st, axis_n(L, AXIS), xn, x_last);
  }
}

// Batched sweeps of the re-simulated sub-blocks (AB2-CN, all-wall boxes,
// re_simulation_sub_tstep_interBC_combine.f90:656-701 with dttrsb): one
// persistent kernel per sweep axis over (subdomain, field, 128-line chunk)
// items, one thread per line, solved in place (a line is read before it is
// written, and the carried slots outside the BC rows stay as they are).  The
// arithmetic is the line kernel's, FMA for FMA.
template <int AXIS>
__global__ void __launch_bounds__(kAdiBatchLines) adi_batch_kernel(const BatchAdiArgs* __restrict__ tab,
                                                                   const BatchItem* __restrict__ items, int n_items) {
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const BatchItem w = items[it];
    const BatchAdiArgs& A = tab[w.sub];
    const Layout L = A.L;
    const int fld = w.by;
    const int n1 = AXIS == 0 ? L.ny + 2 : L.nx + 2;
    const int n2 = AXIS == 2 ? L.ny + 2 : L.nz + 2;
    const int tl = w.bx * kAdiBatchLines + threadIdx.x;
    if (tl >= n1 * n2) continue;
    const LineSys& S = A.sys[AXIS][fld];
    long long base, st;
    line_of<AXIS>(L, tl % n1, tl / n1, base, st);
    double* xl = A.f[fld] + base + (long long)S.lo * st;
    const double* lf = S.l + S.pad;
    const double* di = S.dinv + S.pad;
    const double* cu = S.cu + S.pad;
    const int m = S.hi - S.lo + 1;
    const double r_lo = A.face_lo[AXIS][fld] ? __ldg(A.face_lo[AXIS][fld] + tl) : 0.0;
    const double r_hi = A.face_hi[AXIS][fld] ? __ldg(A.face_hi[AXIS][fld] + tl) : 0.0;
    // the right-hand sides PD unknowns ahead in registers, so no load waits
    // behind the store to the same line (same operations, same bits)
    constexpr int PD = 8;
    auto rhs = [&](int e) -> double {
      if (e < 0 || e >= m) return 0.0;
      if (e == 0) return r_lo;
      if (e == m - 1) return r_hi;
      return xl[(long long)e * st];
    };
    double rb[PD];
#pragma unroll
    for (int q = 0; q < PD; ++q) rb[q] = rhs(q);
    double yp = 0.0;
    for (int g = 0; g < m; g += PD) {
      double nb[PD];
#pragma unroll
      for (int q = 0; q < PD; ++q) nb[q] = rhs(g + PD + q);
#pragma unroll
      for (int q = 0; q < PD; ++q) {
        const int e = g + q;
        if (e < m) {
          yp = fma(-__ldg(lf + e), yp, rb[q]);
          xl[(long long)e * st] = yp;
        }
      }
#pragma unroll
      for (int q = 0; q < PD; ++q) rb[q] = nb[q];
    }
    auto yv = [&](int e) -> double { return e >= 0 ? xl[(long long)e * st] : 0.0; };
#pragma unroll
    for (int q = 0; q < PD; ++q) rb[q] = yv(m - 1 - q);
    double xn = 0.0;
    for (int g = m - 1; g >= 0; g -= PD) {
      double nb[PD];
#pragma unroll
      for (int q = 0; q < PD; ++q) nb[q] = yv(g - PD - q);
#pragma unroll
      for (int q = 0; q < PD; ++q) {
        const int e = g - q;
        if (e >= 0) {
          xn = fma(-__ldg(cu + e), xn, rb[q] * __ldg(di + e));
          xl[(long long)e * st] = xn;
        }
      }
#pragma unroll
      for (int q = 0; q < PD; ++q) rb[q] = nb[q];
    }
  }
}

// The batched x sweep with the session x sweep's staging: each warp of an
// item takes 32 of its 128 lines and walks them in blocks of 32 unknowns
// through shared memory, so every global access is a coalesced row segment
// (the lines are contiguous, the lanes of the one-thread-per-line kernel
// would stride across rows).  Same operations as adi_batch_kernel.
__global__ void __launch_bounds__(kAdiBatchLines) adi_batch_x_kernel(const BatchAdiArgs* __restrict__ tab,
                                                                     const BatchItem* __restrict__ items, int n_items) {
  constexpr int NW = kAdiBatchLines / 32;
  __shared__ double sh[NW][XB * XS];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  double* sb = sh[warp];
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const BatchItem w = items[it];
    const BatchAdiArgs& A = tab[w.sub];
    const Layout L = A.L;
    const int fld = w.by;
    const LineSys& S = A.sys[0][fld];
    const int n1 = L.ny + 2;
    const int nlines = n1 * (L.nz + 2);
    const int t0 = w.bx * kAdiBatchLines + warp * 32;
    if (t0 >= nlines) continue;  // warp-uniform
    const int nl = min(32, nlines - t0);
    const int t = t0 + min(lane, nl - 1);  // lanes past the end repeat the last line (never stored)
    const int j = t % n1, k = t / n1;
    const int my_off = (int)L.at(S.lo, j, k);
    double* f = A.f[fld];
    const double* lf = S.l + S.pad;
    const double* di = S.dinv + S.pad;
    const double* cu = S.cu + S.pad;
    const int m = S.hi - S.lo + 1;
    const int nb = (m + XB - 1) / XB;
    const bool act = lane < nl;
    const double face_lo = (act && A.face_lo[0][fld]) ? __ldg(A.face_lo[0][fld] + t) : 0.0;
    const double face_hi = (act && A.face_hi[0][fld]) ? __ldg(A.face_hi[0][fld] + t) : 0.0;
    double yp = 0.0;
    for (int b = 0; b < nb; ++b) {
      const int e0 = b * XB;
      const int ne = min(XB, m - e0);
#pragma unroll 8
      for (int l = 0; l < XB; ++l) {
        const int off = __shfl_sync(0xffffffffu, my_off, l);
        if (l < nl && lane < ne) sb[lane * XS + l] = f[off + e0 + lane];
      }
      __syncwarp();
      if (e0 == 0) sb[lane] = face_lo;  // the BC rows take the sweep's face values
      if (m - 1 - e0 < XB) sb[(m - 1 - e0) * XS + lane] = face_hi;
      if (act)
        for (int q = 0; q < ne; ++q) {
          yp = fma(-__ldg(lf + e0 + q), yp, sb[q * XS + lane]);
          sb[q * XS + lane] = yp;
        }
      __syncwarp();
#pragma unroll 8
      for (int l = 0; l < XB; ++l) {
        const int off = __shfl_sync(0xffffffffu, my_off, l);
        if (l < nl && lane < ne) f[off + e0 + lane] = sb[lane * XS + l];
      }
      __syncwarp();
    }
    double xn = 0.0;
    for (int b = nb - 1; b >= 0; --b) {
      const int e0 = b * XB;
      const int ne = min(XB, m - e0);
#pragma unroll 8
      for (int l = 0; l < XB; ++l) {
        const int off = __shfl_sync(0xffffffffu, my_off, l);
        if (l < nl && lane < ne) sb[lane * XS + l] = f[off + e0 + lane];
      }
      __syncwarp();
      if (act)
        for (int q = ne - 1; q >= 0; --q) {
          xn = fma(-__ldg(cu + e0 + q), xn, sb[q * XS + lane] * __ldg(di + e0 + q));
          sb[q * XS + lane] = xn;
        }
      __syncwarp();
#pragma unroll 8
      for (int l = 0; l < XB; ++l) {
        const int off = __shfl_sync(0xffffffffu, my_off, l);
        if (l < nl && lane < ne) f[off + e0 + lane] = sb[lane * XS + l];
      }
      __syncwarp();
    }
  }
}

cudaError_t launch_adi_batch(int axis, const BatchAdiArgs* tab, const BatchItem* items, int n_items, int grid,
                             cudaStream_t st) {
  if (n_items <= 0) return cudaSuccess;
  grid = std::max(1, std::min(grid, n_items));
  if (axis == 0) adi_batch_x_kernel<<<grid, kAdiBatchLines, 0, st>>>(tab, items, n_items);
  else if (axis == 1) adi_batch_kernel<1><<<grid, kAdiBatchLines, 0, st>>>(tab, items, n_items);
  else adi_batch_kernel<2><<<grid, kAdiBatchLines, 0, st>>>(tab, items, n_items);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Chunked sweeps
// ---------------------------------------------------------------------------
// With a small viscous number every factor of the LU is small (nu dt / 2 h^2 =
// 0.002: 0.002), so what rows W = 8 to 16 away weigh in a row is below 2^-57.
// A line's chunks of CH unknowns are solved in one CTA (32 lines, a thread a
// chunk) in registers: what enters a chunk is worked out by its neighbour from
// its W outermost unknowns and handed over through shared memory.  One read
// and one write of the fields, no intermediate in memory, CH-fold parallelism
// along the line, and a right-hand side takes part in 2 (CH + W) / CH FMAs:
// they come scaled by the pivots (ChunkSys), one FMA each way.
//
// 2^-57 of a value W + 1 rows away is not always rounding: where the W rows
// between are far below that value, it is what enters.  So a chunk compares
// what it handed on with what it then ends on itself, and where they differ by
// more than roundings (off) the neighbour adds the difference's part
// (chunk_fwd_add, chunk_bwd_add): what is still left out lies below 2^-114.
//
// Bound by the FP64 unit, 75 to 80% busy.  Sweeps x, y, z in us (one thread a
// line): 256^3 291, 257, 260 (512, 385, 369), 128^3 55, 46, 49, with walls 64,
// 55, 55, 32^3 13, 8, 9; without the comparison 280, 265, 267 at 256^3.
// The same in 58-bit integers with the exponent of the line takes 319, 296,
// 292 at 256^3: the chain of a product waits longer there than for an FMA.
// The batch keeps the whole-line kernels: 185, 108, 107 us for 64 blocks of 16
// to 64 cells, in chunks of 18 172, 176, 155.
// Chunks of a line in one CTA, at most: 10 of 26 unknowns (258: a wall line of
// 256 cells), 8 of 16, and 8 of 32 at three CTAs an SM or 17 (a wall line of
// 512 cells) at one.
constexpr int line_chunks_max(int ch) { return ch == 26 ? 10 : (ch == 16 ? 8 : 17); }
// Rows of a line's first end that may differ from the converged ones.
__host__ __device__ constexpr int line_low(int W) { return W + 2; }
// The system has its special rows where the kernels look for them: a few at
// the first end, the last one of a line that does not go on; and chunks divide a cyclic line.
inline bool line_chunk_ok(const ChunkSys& S, int ch, int W) {
  return S.c0 <= std::min(line_low(W), ch) && S.c1 >= (S.wrap_hi ? S.m : S.m - 1) &&
         S.m <= line_chunks_max(ch) * ch && !(S.periodic && S.m % ch);
}
// The recurrences over the unknowns [Q0, Q1) of a chunk, forward and backward,
// from the value that enters.  Rows below T1 take their factors from the
// tables; END: row ql is the line's last, with its own factor (selects, which
// cost nothing beside an FMA; its pivot is in the right-hand side, last_pivot).
// STORE: in place, else only the value that leaves.
template <int CH, int Q0, int Q1, int T1, bool END, bool STORE>
__device__ __forceinline__ double chunk_fwd(double (&r)[CH], const ChunkSys& S, int e0, int ql, double y) {
  const double* l = S.l + kAdiExt + e0;
  const double nl = -S.lc, ll = END ? -__ldg(l + ql) * __ldg(S.dm + kAdiExt + e0 + ql) : 0.0;
#pragma unroll
  for (int q = Q0; q < Q1; ++q) {
    const double f = q < T1 ? -__ldg(l + q) : (END ? (q < ql ? nl : (q == ql ? ll : 0.0)) : nl);
    y = fma(f, y, r[q]);
    if (STORE) r[q] = y;
  }
  return y;
}
template <int CH, int Q0, int Q1, int T1, bool STORE>
__device__ __forceinline__ double chunk_bwd(double (&r)[CH], const ChunkSys& S, int e0, double x) {
  const double* dm = S.dm + kAdiExt + e0;
  const double* cu = S.cu + kAdiExt + e0;
  const double nc = -S.cc;
#pragma unroll
  for (int q = Q1 - 1; q >= Q0; --q) {
    x = q < T1 ? fma(-__ldg(cu + q), x, r[q] * __ldg(dm + q)) : fma(nc, x, r[q]);
    if (STORE) r[q] = x;
  }
  return x;
}

// Two roundings of one number differ by a few units, no more.
__device__ __forceinline__ bool off(double a, double b) {
  return (unsigned long long)(__double_as_longlong(a) - __double_as_longlong(b) + 4) > 8;
}
// d more or less of a row's value y is no more than another rounding of it (and then of the rows behind,
// which hear of it through y).  In noise a value that happens to be small is off in one CTA of a hundred;
// the part run through all rows made the last CTA late (64 x 128 x 128: 30 us to 48, now 32).
__device__ __forceinline__ bool small(double d, double y) { return fabs(d) <= 0x1p-56 * fabs(y); }
// The rare part, on a copy of the chunk in local memory (unrolled over the registers it made the kernels
// too long for the instruction cache: the 128^3 box's step 10% slower, with no chunk taking it).
// Forward: y that enters is d more than was taken; returns what the chunk then hands on backward.
// low: rows before it are of the tables; ql: the line's last row, with its own factor.
__device__ __noinline__ double chunk_fwd_add(double* r, const ChunkSys& S, int e0, int ch, int w, int low, int ql,
                                             double d) {
  const double* l = S.l + kAdiExt + e0;
  const double* dm = S.dm + kAdiExt + e0;
  const double* cu = S.cu + kAdiExt + e0;
#pragma unroll 1
  for (int q = 0; q < ch && q <= ql; ++q) {
    d *= q == ql && q >= low ? -l[q] * dm[q] : -l[q];
    if (small(d, r[q])) break;
    r[q] += d;
  }
  double x = 0.0;
#pragma unroll 1
  for (int q = w - 1; q >= 0; --q) x = fma(-cu[q], x, q < low ? r[q] * dm[q] : r[q]);
  return x;
}
__device__ __noinline__ void chunk_bwd_add(double* r, const ChunkSys& S, int e0, int ch, double d) {
  const double* cu = S.cu + kAdiExt + e0;
#pragma unroll 1
  for (int q = ch - 1; q >= 0; --q) {
    d *= -cu[q];
    if (small(d, r[q])) break;
    r[q] += d;
  }
}

// r: the right-hand sides of chunk s of T (zero past the line's end), replaced by the solution.
// sh: 16 bytes a thread.
template <int CH, int W>
__device__ __forceinline__ void chunk_line_solve(double (&r)[CH], const ChunkSys& S, int s, int T, int l, double* sh) {
  constexpr int LOW = line_low(W) < CH ? line_low(W) : CH;
  double* ys = sh + l;
  double* xs = sh + 32 * T + l;
  const int e0 = s * CH, ql = S.m - 1 - e0;
  const bool low = s == 0 && S.c0 > 0, end = e0 + CH > S.c1;
  const int before = s > 0 ? s - 1 : (S.wrap_lo ? T - 1 : -1), after = s + 1 < T ? s + 1 : (S.wrap_hi ? 0 : -1);
  const bool feeds_up = s + 1 < T || S.wrap_lo, feeds_down = s > 0 || S.wrap_hi;  // a chunk takes its y, its x
  const double y = chunk_fwd<CH, CH - W, CH, CH - W < LOW ? LOW : 0, false, false>(r, S, e0, 0, 0.0);
  ys[32 * s] = y;
  __syncthreads();
  const double yi = before >= 0 ? ys[32 * before] : 0.0;
  double x;
  if (!low && !end) {
    chunk_fwd<CH, 0, CH, 0, false, true>(r, S, e0, 0, yi);
    x = chunk_bwd<CH, 0, W, 0, false>(r, S, e0, 0.0);
  } else if (!end) {
    chunk_fwd<CH, 0, CH, LOW, false, true>(r, S, e0, 0, yi);
    x = chunk_bwd<CH, 0, W, LOW, false>(r, S, e0, 0.0);
  } else if (!low) {
    if (ql >= 0) chunk_fwd<CH, 0, CH, 0, true, true>(r, S, e0, ql, yi);  // below: no row of the line
    x = chunk_bwd<CH, 0, W, 0, false>(r, S, e0, 0.0);
  } else {
    chunk_fwd<CH, 0, CH, LOW, true, true>(r, S, e0, ql, yi);
    x = 0.0;
  }
  xs[32 * s] = x;
  const bool far_y = feeds_up && off(r[CH - 1], y);
  if (__syncthreads_or(far_y)) {
    ys[32 * s] = far_y ? r[CH - 1] - y : 0.0;
    __syncthreads();
    const double d = before >= 0 ? ys[32 * before] : 0.0;
    if (d != 0.0 && !small(d * __ldg(S.l + kAdiExt + e0), r[0])) {  // (noise: a small value beside others)
      double t[CH];
#pragma unroll
      for (int q = 0; q < CH; ++q) t[q] = r[q];
      x = chunk_fwd_add(t, S, e0, CH, W, low ? LOW : 0, end ? ql : CH, d);
      xs[32 * s] = x;
#pragma unroll
      for (int q = 0; q < CH; ++q) r[q] = t[q];
    }
    __syncthreads();
  }
  const double xi = after >= 0 ? xs[32 * after] : 0.0;
  if (low) chunk_bwd<CH, 0, CH, LOW, true>(r, S, e0, xi);
  else chunk_bwd<CH, 0, CH, 0, true>(r, S, e0, xi);
  const bool far_x = feeds_down && off(r[0], x);
  if (__syncthreads_or(far_x)) {
    ys[32 * s] = far_x ? r[0] - x : 0.0;
    __syncthreads();
    const double d = after >= 0 ? ys[32 * after] : 0.0;
    if (d != 0.0 && !small(d * __ldg(S.cu + kAdiExt + e0 + CH - 1), r[CH - 1])) {
      double t[CH];
#pragma unroll
      for (int q = 0; q < CH; ++q) t[q] = r[q];
      chunk_bwd_add(t, S, e0, CH, d);
#pragma unroll
      for (int q = 0; q < CH; ++q) r[q] = t[q];
    }
  }
}

// Pivot ratio by which the last row's right-hand side of a wall line is given
// (one of the table rows scales it itself).
template <int CH, int W>
__device__ __forceinline__ double last_pivot(const ChunkSys& S) {
  return S.m > (line_low(W) < CH ? line_low(W) : CH) ? __ldg(S.dm + kAdiExt + S.m - 1) : 1.0;
}
// One sweep's lines of one field: n1 lines a row, nl lines from z slot zlo on,
// source, destination, BC-row planes.
struct LineJob {
  int n1, zlo, nl;
  const double* src;
  double* dst;
  const double* face_lo;
  const double* face_hi;
  double face_scale;
};

// y and z sweeps: blockDim (32 lines, T chunks), lanes over x; lines [t0, t0 + 32).
template <int AXIS, int CH, int W>
__device__ __forceinline__ void line_chunks(const Layout& L, const ChunkSys& S, const LineJob& J, int t0, double* sh) {
  const int l = threadIdx.x, s = threadIdx.y, T = blockDim.y, n1 = J.n1;
  const bool valid = t0 + l < J.nl;
  const int tl = min(t0 + l, J.nl - 1);  // lanes past the end repeat the last line (never stored)
  long long base, st;
  line_of<AXIS>(L, tl % n1, J.zlo + tl / n1, base, st);
  const double* src = J.src + base;
  double* dst = J.dst + base;
  const int e0 = s * CH, m = S.m;
  const double* sl = src + (S.lo + e0) * st;
  double r[CH];
#pragma unroll
  for (int q = 0; q < CH; ++q, sl += st) r[q] = e0 + q < m ? *sl : 0.0;
  const int nax = axis_n(L, AXIS);
  if (!S.periodic) {
    if (e0 == 0) r[0] = J.face_lo ? J.face_scale * __ldg(J.face_lo + tl + J.zlo * n1) : 0.0;
    if (e0 < m && e0 + CH >= m) {  // the BC rows take the sweep's face values
      const double hi = J.face_hi ? last_pivot<CH, W>(S) * J.face_scale * __ldg(J.face_hi + tl + J.zlo * n1) : 0.0;
#pragma unroll
      for (int q = 0; q < CH; ++q)
        if (e0 + q == m - 1) r[q] = hi;
    }
    if (valid && s == 0) {  // the carried slots
      for (int i = 0; i < S.lo; ++i) dst[i * st] = src[i * st];
      for (int i = S.lo + m; i <= nax + 1; ++i) dst[i * st] = src[i * st];
    }
  }
  chunk_line_solve<CH, W>(r, S, s, T, l, sh);
  if (!valid) return;
  double* xl = dst + (S.lo + e0) * st;
#pragma unroll
  for (int q = 0; q < CH; ++q, xl += st)
    if (e0 + q < m) *xl = r[q];
  if (S.periodic) {  // chunks divide m
    if (s == 0) dst[(nax + 1) * st] = r[0];       // slot n+1 <- slot 1
    if (s == T - 1) dst[0] = r[CH - 1];           // slot 0 <- slot n
  }
}

// x sweep: the CTA's 32 lines pass through shared memory in 16-byte units,
// unit u of line l at place u ^ (l & 7), so that rows are whole on the global
// side and 8 lanes read 8 different banks' worth on the other.
__host__ __device__ constexpr int line_pitch(int ch, int T) { return (ch / 2 * T + 7) & ~7; }  // units a line
template <int CH, int W>
__device__ __forceinline__ void line_chunks_x(const Layout& L, const ChunkSys& S, const LineJob& J, int t0, double* sh) {
  const int l = threadIdx.x, s = threadIdx.y, T = blockDim.y;
  const int pitch = line_pitch(CH, T), m = S.m, e0 = s * CH;
  double2* sb = reinterpret_cast<double2*>(sh);
  double* ex = sh + 64LL * pitch;
  const int nl = min(32, J.nl - t0);
  const int t = t0 + min(l, nl - 1);  // lanes past the end repeat the last line (never stored)
  const int j = t % J.n1, k = J.zlo + t / J.n1;
  const int my_off = (int)L.at(S.lo, j, k);  // unknown 0 of this lane's line
  // slot 1 is 16-byte aligned: whole units where it is unknown 0
  const int nu = S.lo == 1 ? m / 2 : 0;
  for (int q = s; q < 32; q += T) {
    const double* g = J.src + __shfl_sync(0xffffffffu, my_off, q);
    double2* row = sb + q * pitch;
    for (int u = l; u < nu; u += 32) cp_async16(row + (u ^ (q & 7)), g + 2 * u);
    for (int e = 2 * nu + l; e < CH * T; e += 32) {
      double* at = reinterpret_cast<double*>(row + ((e >> 1) ^ (q & 7))) + (e & 1);
      if (e < m) cp_async8(at, g + e);
      else *at = 0.0;
    }
  }
  cp_async_commit();
  const bool walls = !S.periodic;
  double lo = 0.0, hi = 0.0;
  if (walls) {
    if (J.face_lo) lo = J.face_scale * __ldg(J.face_lo + j + J.n1 * k);
    if (J.face_hi) hi = last_pivot<CH, W>(S) * J.face_scale * __ldg(J.face_hi + j + J.n1 * k);
  }
  cp_async_wait<0>();
  __syncthreads();
  double2* row = sb + l * pitch;
  double r[CH];
#pragma unroll
  for (int q = 0; q < CH; q += 2) {
    const double2 d = row[((e0 + q) >> 1) ^ (l & 7)];
    r[q] = d.x;
    r[q + 1] = d.y;
  }
  if (walls) {  // the BC rows take the sweep's face values
    if (e0 == 0) r[0] = lo;
    if (e0 < m && e0 + CH >= m) {
#pragma unroll
      for (int q = 0; q < CH; ++q)
        if (e0 + q == m - 1) r[q] = hi;
    }
  }
  chunk_line_solve<CH, W>(r, S, s, T, l, ex);
#pragma unroll
  for (int q = 0; q < CH; q += 2) row[((e0 + q) >> 1) ^ (l & 7)] = make_double2(r[q], r[q + 1]);
  __syncthreads();
  for (int q = s; q < nl; q += T) {
    double* g = J.dst + __shfl_sync(0xffffffffu, my_off, q);
    const double2* rq = sb + q * pitch;
    for (int u = l; u < nu; u += 32) *reinterpret_cast<double2*>(g + 2 * u) = rq[u ^ (q & 7)];
    for (int e = 2 * nu + l; e < m; e += 32)
      g[e] = reinterpret_cast<const double*>(rq + ((e >> 1) ^ (q & 7)))[e & 1];
  }
  if (l < nl) {
    const double* xs = J.src + L.at(0, j, k);
    double* xd = J.dst + L.at(0, j, k);
    if (walls) {  // the carried slots
      if (s == 0) {
        for (int i = 0; i < S.lo; ++i) xd[i] = xs[i];
        for (int i = S.lo + m; i <= L.nx + 1; ++i) xd[i] = xs[i];
      }
    } else {  // chunks divide m
      if (s == 0) xd[L.nx + 1] = r[0];    // slot n+1 <- slot 1
      if (s == T - 1) xd[0] = r[CH - 1];  // slot 0 <- slot n
    }
  }
}
size_t line_smem(int axis, int ch, int T) {
  return (size_t)T * 32 * 16 + (axis == 0 ? (size_t)32 * line_pitch(ch, T) * sizeof(double2) : 0);
}

template <int AXIS, int CH, int W, int TMAX>
__global__ void __launch_bounds__(32 * TMAX, TMAX == 17 ? 1 : (CH == 16 ? 4 : (CH == 26 ? 2 : 3)))
    adi_line_chunk_kernel(const __grid_constant__ AdiArgs a) {
  extern __shared__ __align__(16) double sh_line[];
  const int fld = blockIdx.y;
  const bool part = AXIS != 2 && a.z1 > 0;  // only the lines of z slots [z0, z1)
  const int n1 = AXIS == 0 ? a.L.ny + 2 : a.L.nx + 2;
  const int n2 = AXIS == 2 ? a.L.ny + 2 : (part ? a.z1 - a.z0 : a.L.nz + 2);
  const LineJob J{n1,        part ? a.z0 : 0, n1 * n2,          a.src[fld], a.dst[fld], a.face_lo[fld],
                  a.face_hi[fld], a.face_scale};
  if (AXIS == 0) line_chunks_x<CH, W>(a.L, a.ch[fld], J, blockIdx.x * 32, sh_line);
  else line_chunks<AXIS, CH, W>(a.L, a.ch[fld], J, blockIdx.x * 32, sh_line);
}

template <int AXIS, int CH, int W, int TMAX>
cudaError_t launch_adi_line_chunk(const AdiArgs& a, int T, cudaStream_t st) {
  const int n1 = AXIS == 0 ? a.L.ny + 2 : a.L.nx + 2;
  const int n2 = AXIS == 2 ? a.L.ny + 2 : (a.z1 > 0 ? a.z1 - a.z0 : a.L.nz + 2);
  if (n2 <= 0) return cudaSuccess;
  const size_t sm = line_smem(AXIS, CH, T);
  auto kern = adi_line_chunk_kernel<AXIS, CH, W, TMAX>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  kern<<<dim3((unsigned)((n1 * n2 + 31) / 32), 3), dim3(32, T), sm, st>>>(a);
  return cudaGetLastError();
}

// Unknowns per chunk: 32 or 26, whichever computes fewer (130, the unknowns of
// a wall line of 128 cells: 5 x 26), and 16 on boxes whose 32-unknown chunks
// leave SMs idle (a 32^3 sweep: 8 to 12 us against 20 a whole line).
int adi_chunk(const Layout& L, const ChunkSys (&S)[3], int W) {
  const int m = std::max(S[0].m, std::max(S[1].m, S[2].m));
  const long long cells = 3LL * (L.nx + 2) * (L.ny + 2) * (L.nz + 2);
  auto fits = [&](int ch) {
    for (const ChunkSys& s : S)
      if (!line_chunk_ok(s, ch, W)) return false;
    return true;
  };
  if (cells / 32 < 40000 && fits(16)) return 16;
  auto work = [&](int ch) { return fits(ch) ? (m + ch - 1) / ch * (ch + W) : 1 << 30; };
  const int ch = work(26) < work(32) ? 26 : 32;
  return fits(ch) ? ch : (fits(16) ? 16 : 0);  // 16: cyclic lines of 16 cells in a large box
}

cudaError_t launch_adi_chunks(int axis, const AdiArgs& a, cudaStream_t st) {
  const int m = std::max(a.ch[0].m, std::max(a.ch[1].m, a.ch[2].m));
  const int ch = adi_chunk(a.L, a.ch, a.halo);
  if (!ch) return cudaErrorInvalidValue;
  const int T = (m + ch - 1) / ch, tmax = ch == 26 ? 10 : (T <= 8 ? 8 : 17);
#define NS_ADI_LINE(A, C, H, M) \
  if (axis == A && ch == C && a.halo == H && tmax == M) return launch_adi_line_chunk<A, C, H, M>(a, T, st);
#define NS_ADI_LINES(C, H, M) NS_ADI_LINE(0, C, H, M) NS_ADI_LINE(1, C, H, M) NS_ADI_LINE(2, C, H, M)
  NS_ADI_LINES(16, 8, 8) NS_ADI_LINES(16, 10, 8) NS_ADI_LINES(16, 12, 8) NS_ADI_LINES(16, 16, 8)
  NS_ADI_LINES(32, 8, 8) NS_ADI_LINES(32, 10, 8) NS_ADI_LINES(32, 12, 8) NS_ADI_LINES(32, 16, 8)
  NS_ADI_LINES(26, 8, 10) NS_ADI_LINES(26, 10, 10) NS_ADI_LINES(26, 12, 10) NS_ADI_LINES(26, 16, 10)
  NS_ADI_LINES(32, 8, 17) NS_ADI_LINES(32, 10, 17) NS_ADI_LINES(32, 12, 17) NS_ADI_LINES(32, 16, 17)
#undef NS_ADI_LINES
#undef NS_ADI_LINE
  return cudaErrorInvalidValue;
}

// y and z sweeps: the persistent line kernel, 8 CTAs of 128 threads per SM
// (measured at 256^3: 0.38 / 0.37 ms against 0.44 / 0.41 ms for one thread
// per line without prefetch); the x sweep keeps the shared-memory blocked
// kernel, whose row loads are coalesced.
cudaError_t launch_adi(int axis, const AdiArgs& a, cudaStream_t st) {
  if (a.halo) return launch_adi_chunks(axis, a, st);
  if (axis != 0) {
    int dev = 0, nsm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const int n1 = a.L.nx + 2;
    const int n2 = (axis == 2) ? a.L.ny + 2 : (a.z1 > 0 ? a.z1 - a.z0 : a.L.nz + 2);
    if (n2 <= 0) return cudaSuccess;
    const int need = (3 * n1 * n2 + 127) / 128;
    const int grid = std::min(need, 8 * std::max(1, nsm));
    if (axis == 1) adi_line_kernel<1, 8><<<grid, 128, 0, st>>>(a);
    else adi_line_kernel<2, 8><<<grid, 128, 0, st>>>(a);
    return cudaGetLastError();
  }
  const int n2 = a.z1 > 0 ? a.z1 - a.z0 : a.L.nz + 2;
  if (n2 <= 0) return cudaSuccess;
  const long long lines = (long long)(a.L.ny + 2) * n2;
  dim3 grid((unsigned)((lines + 32 * XW - 1) / (32 * XW)), 1, 3);
  adi_x_kernel<<<grid, 32 * XW, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace ns
