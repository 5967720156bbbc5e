// Ghost/face fills.  Each fill runs one pass per axis in the reference's
// order (x, then y, then z), each pass over the full extent of the two other
// axes including their ghosts, so edge and corner values come out as in
// vel_bc_staggered (NS_functions.f90:213-310) and pr_bc_staggered
// (NS_functions.f90:1403-1464).
//
// The whole-box fills do the three passes in one launch: a thread works out
// one filled value as the passes would, the z rule of the y rule of the x rule
// of a slot that no pass writes, with the face values that each pass takes at
// its own line.  Three launches of about 5 us each for planes that take 1 us
// were 12 to 24% of the step of a 32^3 or 64^3 box.
#include <algorithm>

#include "ns_internal.cuh"
#include "ns_kernels.cuh"

namespace ns {

namespace {

struct AxisGeo {
  long long base, st;  // slot 0 of the line, stride along the axis
  int n;               // cells along the axis
  int plane;           // index into the face planes
  bool ok;
};

template <int AXIS>
__device__ __forceinline__ AxisGeo axis_geo(const Layout& L, int t) {
  const int n1 = (AXIS == 0) ? L.ny + 2 : L.nx + 2;
  const int n2 = (AXIS == 2) ? L.ny + 2 : L.nz + 2;
  AxisGeo g;
  g.ok = t < n1 * n2;
  const int s1 = t % n1, s2 = t / n1;
  g.plane = t;
  if (AXIS == 0) { g.base = L.at(0, s1, s2); g.st = 1; g.n = L.nx; }
  else if (AXIS == 1) { g.base = L.at(s1, 0, s2); g.st = L.sy; g.n = L.ny; }
  else { g.base = L.at(s1, s2, 0); g.st = L.sz; g.n = L.nz; }
  return g;
}

__device__ __forceinline__ double facev(const double* f, int i) { return f ? f[i] : 0.0; }

// The rule of one side of an axis: the filled value from the source value v
// (unused where the face value alone is taken) and the face value f.
// Velocity: normal, the field is staggered along the axis (slots 1 and n+1 of
// a wall, 0 and n+1 of a periodic axis); else its ghost slots 0 and n+1.
__device__ __forceinline__ double vel_rule(int bc, bool normal, double v, double f) {
  if (bc == 1) return v;
  if (normal || bc == 4) return f;
  return fma(2.0, f, -v);
}
__device__ __forceinline__ double pr_rule(int pbc, bool high, double h, double v, double f) {
  if (pbc == 1) return v;
  if (pbc == 2) return fma(2.0, f, -v);
  if (pbc == 3) return fma(high ? h : -h, f, v);
  return f;
}

// Field fld (0..2 u, v, w; 3 dp) of a box: which slots an axis pass fills.
template <bool PR>
struct Fill {
  const Layout& L;
  double* x;
  const FaceSet& F;
  const int* code;
  const double* h;
  int fld;
  __device__ __forceinline__ int n(int a) const { return a == 0 ? L.nx : a == 1 ? L.ny : L.nz; }
  __device__ __forceinline__ bool normal(int a) const { return !PR && a == fld; }
  __device__ __forceinline__ int low(int a) const { return normal(a) && code[a] != 1 ? 1 : 0; }  // lower filled slot
  __device__ __forceinline__ bool filled(int a, int i) const { return i == low(a) || i == n(a) + 1; }
  // the source slot of a filled one
  __device__ __forceinline__ int source(int a, int i) const {
    return code[a] == 1 ? (i == 0 ? n(a) : 1) : (i > 0 ? n(a) : 1);
  }
  __device__ __forceinline__ double rule(int a, int i, double v, int plane) const {
    const bool high = i == n(a) + 1;
    const double* f = F.ax[a].f[fld][high ? 1 : 0];
    const double fv = facev(f, plane);
    return PR ? pr_rule(code[a], high, h[a], v, fv) : vel_rule(code[a], normal(a), v, fv);
  }
  // Filled slots of the box: two z planes, then two y planes and two x planes
  // without what the later passes fill.
  __device__ __forceinline__ long long count() const {
    return 2LL * (L.nx + 2) * (L.ny + 2) + 2LL * (L.nx + 2) * L.nz + 2LL * L.ny * L.nz;
  }
  __device__ __forceinline__ int open(int a, int q) const { return low(a) == 0 ? q + 1 : (q == 0 ? 0 : q + 1); }
  __device__ __forceinline__ void fill(long long t) const {
    int i, j, k;
    const long long nz2 = 2LL * (L.nx + 2) * (L.ny + 2), ny2 = 2LL * (L.nx + 2) * L.nz;
    if (t < nz2) {
      const int q = (int)t, pl = (L.nx + 2) * (L.ny + 2), r = q % pl;
      k = q < pl ? low(2) : L.nz + 1;
      i = r % (L.nx + 2);
      j = r / (L.nx + 2);
    } else if (t - nz2 < ny2) {
      const int q = (int)(t - nz2), pl = (L.nx + 2) * L.nz, r = q % pl;
      j = q < pl ? low(1) : L.ny + 1;
      i = r % (L.nx + 2);
      k = open(2, r / (L.nx + 2));
    } else {
      const int q = (int)(t - nz2 - ny2), r = q >> 1;
      i = q & 1 ? L.nx + 1 : low(0);
      j = open(1, r % L.ny);
      k = open(2, r / L.ny);
    }
    const bool fz = filled(2, k), fy = filled(1, j), fx = filled(0, i);
    const int ks = fz ? source(2, k) : k, js = fy ? source(1, j) : j, is = fx ? source(0, i) : i;
    double v = x[L.at(is, js, ks)];
    if (fx) v = rule(0, i, v, js + (L.ny + 2) * ks);
    if (fy) v = rule(1, j, v, i + (L.nx + 2) * ks);
    if (fz) v = rule(2, k, v, i + (L.nx + 2) * j);
    x[L.at(i, j, k)] = v;
  }
};

// Velocity fills: a thread per filled slot of the three fields.
struct VelFillArgs {
  Layout L;
  double* f[3];
  FaceSet F;
  int bc[3];
};
__global__ void __launch_bounds__(256) vel_fill_kernel(const __grid_constant__ VelFillArgs a) {
  const Fill<false> g{a.L, a.f[blockIdx.y], a.F, a.bc, nullptr, (int)blockIdx.y};
  const long long t = blockIdx.x * 256LL + threadIdx.x;
  if (t < g.count()) g.fill(t);
}
struct PrFillArgs {
  Layout L;
  double* dp;
  FaceSet F;
  int pbc[3];
  double h[3];
};
__global__ void __launch_bounds__(256) pr_fill_kernel(const __grid_constant__ PrFillArgs a) {
  const Fill<true> g{a.L, a.dp, a.F, a.pbc, a.h, 3};
  const long long t = blockIdx.x * 256LL + threadIdx.x;
  if (t < g.count()) g.fill(t);
}

template <int AXIS>
__device__ __forceinline__ void pr_bc_body(const Layout& L, double* dp, const FacePlanes& F, int pbc, double h, int t) {
  const AxisGeo g = axis_geo<AXIS>(L, t);
  if (!g.ok) return;
  double* x = dp + g.base;
  const long long st = g.st;
  const int n = g.n;
  double* hi = x + (long long)(n + 1) * st;
  const double* flo = F.f[3][0];
  const double* fhi = F.f[3][1];
  if (pbc == 1) {
    x[0] = x[(long long)n * st];
    *hi = x[st];
  } else if (pbc == 2) {
    x[0] = fma(2.0, facev(flo, g.plane), -x[st]);
    *hi = fma(2.0, facev(fhi, g.plane), -x[(long long)n * st]);
  } else if (pbc == 3) {
    x[0] = fma(-h, facev(flo, g.plane), x[st]);
    *hi = fma(h, facev(fhi, g.plane), x[(long long)n * st]);
  } else if (pbc == 4) {
    x[0] = facev(flo, g.plane);
    *hi = facev(fhi, g.plane);
  }
}

// Lines t in [t0, t1) of the pass along AXIS.
template <int AXIS>
__global__ void pr_bc_kernel(Layout L, double* dp, FacePlanes F, int pbc, double h, int t0, int t1) {
  const int t = t0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (t < t1) pr_bc_body<AXIS>(L, dp, F, pbc, h, t);
}

// Batched: velocity (PR false; by: the field) or pressure fills, 256 filled slots per work item.
template <bool PR>
__global__ void __launch_bounds__(256) bc_batch_kernel(const BatchBcArgs* __restrict__ tab,
                                                       const BatchItem* __restrict__ items, int n_items) {
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const BatchItem w = items[it];
    const BatchBcArgs& a = tab[w.sub];
    const Fill<PR> g{a.L, PR ? a.dp : w.by == 0 ? a.us : w.by == 1 ? a.vs : a.ws, a.F, PR ? a.pbc : a.bc, a.h,
                     PR ? 3 : w.by};
    const long long t = w.bx * 256LL + threadIdx.x;
    if (t < g.count()) g.fill(t);
  }
}

// Extra face slot 0 of a periodic axis (face 0 = face n) for the face field of that axis.
__global__ void extra_slot_kernel(Layout L, double* f, int axis) {
  const int n1 = (axis == 0) ? L.ny + 2 : L.nx + 2;
  const int n2 = (axis == 2) ? L.ny + 2 : L.nz + 2;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n1 * n2) return;
  const int s1 = t % n1, s2 = t / n1;
  if (axis == 0) f[L.at(0, s1, s2)] = f[L.at(L.nx, s1, s2)];
  else if (axis == 1) f[L.at(s1, 0, s2)] = f[L.at(s1, L.ny, s2)];
  else f[L.at(s1, s2, 0)] = f[L.at(s1, s2, L.nz)];
}

}  // namespace

int plane_count(const Layout& L, int axis) {
  const int n1 = (axis == 0) ? L.ny + 2 : L.nx + 2;
  const int n2 = (axis == 2) ? L.ny + 2 : L.nz + 2;
  return n1 * n2;
}

long long fill_count(const Layout& L) {
  return 2LL * (L.nx + 2) * (L.ny + 2) + 2LL * (L.nx + 2) * L.nz + 2LL * L.ny * L.nz;
}

cudaError_t launch_bc_batch(bool pr, const BatchBcArgs* tab, const BatchItem* items, int n_items, int grid,
                            cudaStream_t st) {
  if (n_items <= 0) return cudaSuccess;
  grid = std::min(grid > 0 ? grid : 8 * 152, n_items);
  if (pr) bc_batch_kernel<true><<<grid, 256, 0, st>>>(tab, items, n_items);
  else bc_batch_kernel<false><<<grid, 256, 0, st>>>(tab, items, n_items);
  return cudaGetLastError();
}

cudaError_t launch_extra_slots(const Layout& L, double* u, double* v, double* w, const int bc[3], cudaStream_t st) {
  double* f[3] = {u, v, w};
  for (int a = 0; a < 3; ++a) {
    if (bc[a] != 1) continue;
    const int n = plane_count(L, a);
    extra_slot_kernel<<<(n + 255) / 256, 256, 0, st>>>(L, f[a], a);
  }
  return cudaGetLastError();
}

cudaError_t launch_vel_bc(const Layout& L, double* us, double* vs, double* ws, const FaceSet& F, const int bc[3],
                          cudaStream_t st) {
  VelFillArgs a{L, {us, vs, ws}, F, {bc[0], bc[1], bc[2]}};
  vel_fill_kernel<<<dim3((unsigned)((fill_count(L) + 255) / 256), 3), 256, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_pr_bc(const Layout& L, double* dp, const FaceSet& F, const int pbc[3], double dx, double dy,
                         double dz, cudaStream_t st) {
  PrFillArgs a{L, dp, F, {pbc[0], pbc[1], pbc[2]}, {dx, dy, dz}};
  pr_fill_kernel<<<(unsigned)((fill_count(L) + 255) / 256), 256, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_pr_bc_planes(const Layout& L, double* dp, const FaceSet& F, const int pbc[3], double dx,
                                double dy, int k0, int k1, cudaStream_t st) {
  if (k0 < 0 || k1 > L.nz + 2 || k0 > k1) return cudaErrorInvalidValue;
  if (k0 == k1) return cudaSuccess;
  // a line of the x pass is (j, k) with t = j + (ny+2) k, of the y pass (i, k) with t = i + (nx+2) k
  const int px = L.ny + 2, py = L.nx + 2;
  pr_bc_kernel<0><<<(px * (k1 - k0) + 255) / 256, 256, 0, st>>>(L, dp, F.ax[0], pbc[0], dx, px * k0, px * k1);
  pr_bc_kernel<1><<<(py * (k1 - k0) + 255) / 256, 256, 0, st>>>(L, dp, F.ax[1], pbc[1], dy, py * k0, py * k1);
  return cudaGetLastError();
}

cudaError_t launch_pr_bc_z(const Layout& L, double* dp, const FaceSet& F, int pbc_z, double dz, cudaStream_t st) {
  const int n = plane_count(L, 2);
  pr_bc_kernel<2><<<(n + 255) / 256, 256, 0, st>>>(L, dp, F.ax[2], pbc_z, dz, 0, n);
  return cudaGetLastError();
}

}  // namespace ns
