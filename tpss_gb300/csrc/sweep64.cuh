// sweep64.cuh -- additive vertex-patch Schwarz smoother on a Cartesian level, FP64, direction by direction.
//
// Same sum as the per-color kernels (preconditioner/schwarz_preconditioner.templates.h:585-688):
// dst = omega sum_v R_v^T S_v Lambda_v^-1 S_v^T R_v src over the interior vertices v = (vx, vy, vz).
// On a tensor-product level the 1-D problem of direction d depends on v_d alone, so the transforms
// of neighbouring patches share work: S_x^T along a line of DoFs is the same for all patches with
// this vx whatever their vy and vz, and by linearity the results of patches that differ only in
// vz can be added before S_y and S_x are applied. Per patch and DoF that leaves 1/4 of the x, 1/2
// of the y and all of the z contractions (3D; 2D: 1/2 and all) instead of two full ones per
// direction, no color needs its own pass over the vectors, and dst is written once:
//
//   sweep_x_forward    src -> T1[gz][gy][vx, a]                         a: mode of direction x
//   line, forward      T1 -> T2[gz][vy, b][vx, a]                       (3D) b: mode of y
//   line, solve        T2 -> U2[gz][vy, b][vx, a]                       S^T, 1 / eigenvalue sums, S and
//                                                                      the sum over vz along z
//   line, backward     U2 -> U1[gz][gy][vx, a]                          (3D) S and the sum over vy
//   sweep_x_backward   U1 -> dst                                       S, the sum over vx, omega
//
// (2D: forward x, solve along y, backward x.) The innermost index runs over (vx, a), so that all but
// the x transforms read and write coalesced with one thread per line; a thread marches along its
// line, so that the sum over neighbouring patches is a carry in registers. Long lines are cut into
// segments that recompute one patch at their ends, as many as it takes to fill the chip.
//
// 3D DGQ4 40^3 0.99 ms against 1.69 ms for the per-color kernel with the same arithmetic (x 0.10 +
// 0.15, y 0.12 + 0.14, z 0.48 ms: the wide-multiply pipe 50 to 62 % busy, HBM 17 to 40 %); 2D DGQ3
// 16^2 40 against 62 us. The intermediate arrays take 10 values per DoF (2D: 4).
// The contractions run on the integer pipe with one exponent per pencil (fixed64.cuh); pencils the
// integers do not cover (infinities, NaN, magnitudes outside 2^(+-300)) use FP64.
#pragma once

#include "fd_fixed.cuh"

namespace tpss
{
namespace sweep
{
using fd::cpow;
using fd::Entry;
using fd::EoEntry;

constexpr int kLineThreads = 128;
constexpr int kMaxGridY = 65535;  // a grid's second dimension (a longer line gets longer segments)

struct SweepTab
{
  const int2 *fix, *fix_eo;    // integer tables, dense and even/odd (FdTables::fix64*)
  const int2 *fexp, *fexp_eo;  // their scales: x for S^T, y for S
  const double *fd, *fd_eo;    // FP64 tables
  const int32_t *sym;          // entry has the even/odd form (or nullptr)
  int es, es_eo;               // words per entry
  bool fp64_only;              // all pencils on the FP64 path
};

template<int N>
struct Slot
{
  static constexpr int SIZE = Entry<double, N>::size > EoEntry<double, N>::size ? Entry<double, N>::size : EoEntry<double, N>::size;
};

// table of entry e into a slot; the threads of the CTA share the copy
template<int N>
__device__ __forceinline__ void load_slot(const SweepTab &t, int e, bool sy, int2 *slot, int tid, int nthr)
{
  const int nc = sy ? EoEntry<double, N>::LAM : Entry<double, N>::LAM;
  const int nt = sy ? EoEntry<double, N>::size : Entry<double, N>::size;
  const int2 *c2 = sy ? t.fix_eo + (size_t)e * t.es_eo : t.fix + (size_t)e * t.es;
  const double *cd = sy ? t.fd_eo + (size_t)e * t.es_eo : t.fd + (size_t)e * t.es;
  for(int o = tid; o < nt; o += nthr)
    slot[o] = o < nc ? c2[o] : make_int2(__double2loint(cd[o]), __double2hiint(cd[o]));
}

// exponent of a pencil: the largest biased exponent (1023 for all zeros), and whether it needs FP64
template<int N>
__device__ __forceinline__ int pencil_exponent(const double (&v)[N], bool fp64_only, bool &slow)
{
  unsigned hm = 0, lo = 0;
#pragma unroll
  for(int m = 0; m < N; ++m)
  {
    hm = max(hm, (unsigned)__double2hiint(v[m]) & 0x7fffffffu);
    lo |= (unsigned)__double2loint(v[m]);
  }
  const int emax = (int)(hm >> 20);
  const bool zero = hm == 0 && lo == 0;
  slow = fp64_only || (!zero && (emax < 1023 - 300 || emax > 1023 + 300));
  return zero ? 1023 : emax;
}

// S^T or S of one pencil v (FP64 values) into the thread's column col[m STRIDE] as FP64 values
template<int N, bool FWD, int STRIDE>
__device__ __forceinline__ void transform(const double (&v)[N], int64_t *col, const SweepTab &t, const int2 *slot, int e,
                                          bool sy, int F)
{
  bool slow;
  const int emax = pencil_exponent<N>(v, t.fp64_only, slow);
  double *out = reinterpret_cast<double *>(col);
  if(slow)
  {
#pragma unroll
    for(int m = 0; m < N; ++m) out[m * STRIDE] = v[m];
    fd::slow_pass<N, FWD>(out, STRIDE, sy ? t.fd_eo + (size_t)e * t.es_eo : t.fd + (size_t)e * t.es, sy, 1.0);
    return;
  }
  fd::fix_pass<N, FWD, STRIDE>(col, slot, sy, [&](int m) { return fx::from_double(v[m], emax); });
  const int ex = emax - 1023 - 58 + 64 - F;
#pragma unroll
  for(int m = 0; m < N; ++m) out[m * STRIDE] = fx::to_double(col[m * STRIDE], ex);
}

enum LineMode
{
  LINE_FORWARD,
  LINE_SOLVE,
  LINE_BACKWARD
};

struct LineArgs
{
  const double *in;
  double *out;
  int64_t ncol;               // lines: column c at (c / inner) * outer + c % inner
  int64_t inner, in_outer, out_outer, stride;
  const int32_t *vfd;         // table entry of vertex v of the line's direction
  int nc;                     // cells along the line
  int seg;                    // cells (forward: vertices) per segment
  SweepTab t;
  // solve: eigenvalues and table entries of the other directions' vertices
  const double *lam0, *lam1;  // per mode index of x and (3D) y
  const int32_t *vfd0, *vfd1;
  int64_t modes0;             // modes of x per row of the plane (vertices * n)
  const double *rcp;          // reciprocal eigenvalue sums per entry combination, or nullptr
  int E;
};

template<int DIM, int K1, int MODE>
__global__ void __launch_bounds__(kLineThreads, K1 <= 5 ? 6 : 4) line_kernel(LineArgs a)
{
  constexpr int N = 2 * K1, BT = kLineThreads, NLOC = cpow(N, DIM);
  __shared__ __align__(16) int2 s_tab[Slot<N>::SIZE];
  extern __shared__ __align__(16) int64_t s_col[];
  const int tid = threadIdx.x;
  const int64_t c = (int64_t)blockIdx.x * BT + tid;
  const bool active = c < a.ncol;
  const int64_t cc = active ? c : 0, co = cc / a.inner, ci = cc - co * a.inner;
  const double *in = a.in + co * a.in_outer + ci;
  double *out = a.out + co * a.out_outer + ci;
  int64_t *col = s_col + tid;
  double *cold = reinterpret_cast<double *>(col);
  // solve: the line's modes of the other directions
  double lxy = 0.0;
  const double *rt = nullptr;
  int combo = 0;
  if constexpr(MODE == LINE_SOLVE)
  {
    const int64_t m1 = DIM == 3 ? cc / a.modes0 : 0, m0 = cc - m1 * a.modes0;
    if(a.rcp)
    {
      combo = a.vfd0[m0 / N + 1];
      rt = a.rcp + m0 % N;
      if constexpr(DIM == 3)
      {
        combo += a.E * a.vfd1[m1 / N + 1];
        rt += N * (m1 % N);
      }
    }
    else
    {
      lxy = a.lam0[m0];
      if constexpr(DIM == 3) lxy += a.lam1[m1];
    }
  }
  double carry[K1];
#pragma unroll
  for(int k = 0; k < K1; ++k) carry[k] = 0.0;
  // cells [c0, c1) of the segment, patches around the vertices v0 .. v1 (forward: vertices only)
  const int c0 = blockIdx.y * a.seg, c1 = min(a.nc, c0 + a.seg);
  const int v0 = MODE == LINE_FORWARD ? c0 + 1 : max(1, c0), v1 = MODE == LINE_FORWARD ? min(a.nc - 1, c0 + a.seg) : min(a.nc - 1, c1);
  int e_now = -1;
  bool sy = false;
  int2 F = make_int2(0, 0);
  for(int v = v0; v <= v1; ++v)
  {
    const int e = a.vfd[v];
    if(e != e_now)
    {
      e_now = e;
      sy = a.t.sym && a.t.sym[e];
      F = sy ? a.t.fexp_eo[e] : a.t.fexp[e];
      __syncthreads();
      load_slot<N>(a.t, e, sy, s_tab, tid, BT);
      __syncthreads();
    }
    if(!active) continue;
    double x[N];
    const int64_t p = (int64_t)(v - 1) * (MODE == LINE_BACKWARD ? N : K1);
#pragma unroll
    for(int m = 0; m < N; ++m) x[m] = in[(p + m) * a.stride];
    if constexpr(MODE == LINE_FORWARD)
    {
      transform<N, true, BT>(x, col, a.t, s_tab, e, sy, F.x);
#pragma unroll
      for(int m = 0; m < N; ++m) out[((int64_t)(v - 1) * N + m) * a.stride] = cold[m * BT];
    }
    else
    {
      if constexpr(MODE == LINE_BACKWARD)
        transform<N, false, BT>(x, col, a.t, s_tab, e, sy, F.y);
      else
      {
        const double *r_tab = rt ? rt + (size_t)(DIM == 3 ? a.E * a.E * e + combo : a.E * e + combo) * NLOC : nullptr;
        constexpr int RS = NLOC / N;
        const double *lam = reinterpret_cast<const double *>(s_tab) + (sy ? EoEntry<double, N>::LAM : Entry<double, N>::LAM);
        bool slow;
        const int emax = pencil_exponent<N>(x, a.t.fp64_only, slow);
        if(slow)
        {
          const double *ent = sy ? a.t.fd_eo + (size_t)e * a.t.es_eo : a.t.fd + (size_t)e * a.t.es;
#pragma unroll
          for(int m = 0; m < N; ++m) cold[m * BT] = x[m];
          fd::slow_pass<N, true>(cold, BT, ent, sy, 1.0);
#pragma unroll 1
          for(int i = 0; i < N; ++i)
            cold[i * BT] = r_tab ? cold[i * BT] * __ldg(r_tab + i * RS) : cold[i * BT] / (lxy + lam[i]);
          fd::slow_pass<N, false>(cold, BT, ent, sy, 1.0);
        }
        else
        {
          fd::fix_pass<N, true, BT>(col, s_tab, sy, [&](int m) { return fx::from_double(x[m], emax); });
          int ex = emax - 1023 - 58 + 64 - F.x;
          ex += 61 + fd::scale_by_reciprocals<N, BT>(col, [&](int i, int &mh, int &ml, int &q) {
            // (levels without the table are rare; fx::reciprocal here cost the others 1.7 %)
            fx::split_positive(r_tab ? __ldg(r_tab + i * RS) : 1.0 / (lxy + lam[i]), mh, ml, q);
          });
          fd::fix_pass<N, false, BT>(col, s_tab, sy, [&](int m) { return col[m * BT]; });
          ex += 64 - F.y;
#pragma unroll
          for(int m = 0; m < N; ++m) cold[m * BT] = fx::to_double(col[m * BT], ex);
        }
      }
      if(v > c0)  // cell v - 1 is complete
#pragma unroll
        for(int k = 0; k < K1; ++k) out[((int64_t)(v - 1) * K1 + k) * a.stride] = carry[k] + cold[k * BT];
#pragma unroll
      for(int k = 0; k < K1; ++k) carry[k] = cold[(K1 + k) * BT];
      if(v == v1 && v1 < c1)  // the line's last cell
#pragma unroll
        for(int k = 0; k < K1; ++k) out[((int64_t)v * K1 + k) * a.stride] = carry[k];
    }
  }
}

// ---- transforms along x between the cell blocks of the vectors and the line arrays
struct XArgs
{
  const double *in;
  double *out;
  const int64_t *cell_start;  // nullptr: lexicographic cells
  const int32_t *vfd;
  int nx, ny, nz;             // cells
  int64_t modes;              // (nx - 1) N: row length of the line arrays
  SweepTab t;
  double omega;
  int ras;                    // divide by the cell's patch multiplicity
};

// A CTA takes XV vertices along x and XG cell rows (cy, cz); a thread one pencil, i.e. one row of
// DoFs of a cell row through the two cells of a vertex.
template<int DIM, int K1>
struct XCfg
{
  static constexpr int N = 2 * K1, R = cpow(K1, DIM - 1), CD = K1 * R;
  static constexpr int XV = R >= 32 ? 4 : 8;
  static constexpr int XG = R * XV >= 128 ? 1 : (128 + R * XV - 1) / (R * XV);
  static constexpr int PENCILS = XV * R * XG;
  static constexpr int THREADS = (PENCILS + 31) / 32 * 32;
  static constexpr int CS = PENCILS + 1;  // column stride: both access directions conflict free
  static constexpr int ES = (Slot<N>::SIZE + 1) / 2 * 2;
  static constexpr int ROWS = XG * R;     // rows of the line arrays per tile
  static constexpr size_t smem() { return ((size_t)XV * ES + (size_t)N * CS + ROWS) * 8; }
};

template<int DIM, int K1>
__device__ __forceinline__ int64_t cell_first(const XArgs &a, int cx, int g)
{
  const int64_t cell = cx + (int64_t)a.nx * g;
  return a.cell_start ? a.cell_start[cell] : cell * XCfg<DIM, K1>::CD;
}

// row of the line arrays that holds row r of cell row g
template<int DIM, int K1>
__device__ __forceinline__ int64_t line_row(const XArgs &a, int g, int r)
{
  if constexpr(DIM == 2) return (int64_t)g * K1 + r;
  const int cy = g % a.ny, cz = g / a.ny;
  return ((int64_t)cz * K1 + r / K1) * ((int64_t)a.ny * K1) + cy * K1 + r % K1;
}

template<int DIM, int K1, bool FWD>
__global__ void __launch_bounds__(XCfg<DIM, K1>::THREADS) sweep_x_kernel(XArgs a)
{
  using C = XCfg<DIM, K1>;
  constexpr int N = C::N, R = C::R, XV = C::XV, XG = C::XG, CS = C::CS, ES = C::ES, CD = C::CD, P = C::PENCILS;
  extern __shared__ __align__(16) int64_t sx[];
  int2 *s_tab = reinterpret_cast<int2 *>(sx);
  int64_t *s_col = sx + XV * ES;
  double *s_cold = reinterpret_cast<double *>(s_col);
  int64_t *s_row = s_col + N * CS;  // first value of each row, -1 beyond the last cell row
  const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32, ng = a.ny * a.nz, g0 = blockIdx.x * XG;
  // forward: vertices 1 + XV t ..; backward: the cells [x0, x0 + XV - 1) and the vertices around them
  const int x0 = (blockIdx.y + blockIdx.z * kMaxGridY) * (FWD ? XV : XV - 1);
  if(x0 >= (FWD ? a.nx - 1 : a.nx)) return;  // (all threads: the last multiple of the second dimension is not full)
  const int vfirst = FWD ? x0 + 1 : x0;
  for(int s = 0; s < XV; ++s)
  {
    const int v = vfirst + s;
    if(v < 1 || v > a.nx - 1) continue;
    const int e = a.vfd[v];
    load_slot<N>(a.t, e, a.t.sym && a.t.sym[e], s_tab + s * ES, tid, C::THREADS);
  }
  const int64_t base = (int64_t)(vfirst - 1) * N;  // first mode of the tile in a row (backward tile 0: -N)
  for(int i = tid; i < C::ROWS; i += C::THREADS)
  {
    const int g = g0 + i / R;
    s_row[i] = g < ng ? line_row<DIM, K1>(a, g, i % R) * a.modes + base : -1;
  }
  // modes of the tile within a row: [m0, m1)
  const int m0 = base < 0 ? N : 0, m1 = (int)(a.modes - base < XV * N ? a.modes - base : XV * N);
  if constexpr(!FWD)
  {
    __syncthreads();
    // a warp reads a row of the tile: lanes along the modes
    for(int i = warp; i < C::ROWS; i += C::THREADS / 32)
    {
      if(g0 + i / R >= ng) continue;
      const double *row = a.in + s_row[i];
      double *c = s_cold + (i / R) * XV * R + i % R;
#pragma unroll
      for(int mm = 0; mm < XV * N; mm += 32)
      {
        const int m = mm + lane;
        if(m >= m0 && m < m1) c[(m % N) * CS + (m / N) * R] = row[m];
      }
    }
  }
  __syncthreads();
  const int r = tid % R, s = (tid / R) % XV, gl = tid / (R * XV), v = vfirst + s;
  if(tid < P && g0 + gl < ng && v >= 1 && v <= a.nx - 1)
  {
    const int e = a.vfd[v];
    const bool sy = a.t.sym && a.t.sym[e];
    const int2 F = sy ? a.t.fexp_eo[e] : a.t.fexp[e];
    double x[N];
    if constexpr(FWD)
    {
      const double *lo = a.in + cell_first<DIM, K1>(a, v - 1, g0 + gl) + K1 * r;
      const double *hi = a.in + cell_first<DIM, K1>(a, v, g0 + gl) + K1 * r;
#pragma unroll
      for(int i = 0; i < K1; ++i)
      {
        x[i] = lo[i];
        x[K1 + i] = hi[i];
      }
    }
    else
#pragma unroll
      for(int m = 0; m < N; ++m) x[m] = s_cold[m * CS + tid];
    transform<N, FWD, CS>(x, s_col + tid, a.t, s_tab + s * ES, e, sy, FWD ? F.x : F.y);
  }
  __syncthreads();
  if constexpr(FWD)
  {
    for(int i = warp; i < C::ROWS; i += C::THREADS / 32)
    {
      if(g0 + i / R >= ng) continue;
      double *row = a.out + s_row[i];
      const double *c = s_cold + (i / R) * XV * R + i % R;
#pragma unroll
      for(int mm = 0; mm < XV * N; mm += 32)
      {
        const int m = mm + lane;
        if(m < m1) row[m] = c[(m % N) * CS + (m / N) * R];
      }
    }
  }
  else
  {
    // cells of the tile, a warp each: the sum of the patches around their two vertices along x
    for(int i = warp; i < XG * (XV - 1); i += C::THREADS / 32)
    {
      const int cl = i % (XV - 1), gg = i / (XV - 1), g = g0 + gg, cx = x0 + cl;
      if(g >= ng || cx >= a.nx) continue;
      double f = a.omega;
      if(a.ras)
      {
        const int cy = g % a.ny, cz = g / a.ny;
        int mult = (cx >= 1) + (cx + 1 <= a.nx - 1);
        mult *= (cy >= 1) + (cy + 1 <= a.ny - 1);
        if(DIM == 3) mult *= (cz >= 1) + (cz + 1 <= a.nz - 1);
        f *= 1.0 / mult;  // a power of two
      }
      const bool lo = cx >= 1, hi = cx + 1 <= a.nx - 1;
      double *out = a.out + cell_first<DIM, K1>(a, cx, g);
      const double *c = s_cold + (gg * XV + cl) * R;
      for(int d = lane; d < CD; d += 32)
      {
        const int k = d % K1, p = d / K1;
        double o = lo ? c[(K1 + k) * CS + p] : 0.0;  // vertex cx: the patch's upper cell
        if(hi) o += c[k * CS + p + R];                // vertex cx + 1: its lower cell
        out[d] = o * f;
      }
    }
  }
}
}  // namespace sweep
}  // namespace tpss
