// sweep64.cu -- launches of the direction-by-direction FP64 smoother (sweep64.cuh). Compiled in parts
// (SWEEP_PART) that hold the degrees k with k % 3 == SWEEP_PART.
#include "sweep64.cuh"
#include "internal.h"

#ifndef SWEEP_PART
#error "SWEEP_PART must be defined (0, 1 or 2)"
#endif
#define SWEEP_CAT2(a, b) a##b
#define SWEEP_CAT(a, b) SWEEP_CAT2(a, b)

namespace tpss
{
namespace
{
using namespace sweep;

template<int DIM, int K1, bool FWD>
void launch_x(const XArgs &a, cudaStream_t s)
{
  using C = XCfg<DIM, K1>;
  if constexpr(C::smem() > 48 * 1024)  // per device; a cheap host call
    TPSS_CUDA(cudaFuncSetAttribute(sweep_x_kernel<DIM, K1, FWD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)C::smem()));
  const int per = FWD ? C::XV : C::XV - 1, count = FWD ? a.nx - 1 : a.nx;
  // a long level has more tiles along x than a grid's second dimension holds: the third counts its multiples
  const int tiles = (count + per - 1) / per;
  const dim3 grid((a.ny * a.nz + C::XG - 1) / C::XG, tiles < kMaxGridY ? tiles : kMaxGridY, (tiles + kMaxGridY - 1) / kMaxGridY);
  sweep_x_kernel<DIM, K1, FWD><<<grid, C::THREADS, C::smem(), s>>>(a);
  TPSS_CUDA(cudaGetLastError());
}

// Segments of a line pass: enough threads to fill the chip a few times over, since a thread marches
// along its whole segment; a backward or solve segment recomputes one patch, so not more than that.
template<int DIM, int K1, int MODE>
void launch_line(LineArgs a, cudaStream_t s)
{
  constexpr int N = 2 * K1;
  const int len = MODE == LINE_FORWARD ? a.nc - 1 : a.nc;  // vertices or cells
  const int64_t want = (int64_t)num_sms() * 2048;
  int64_t segs = (want + a.ncol - 1) / a.ncol;
  if(segs > len) segs = len;
  if(segs > kMaxGridY) segs = kMaxGridY;
  if(segs < 1) segs = 1;
  a.seg = (int)((len + segs - 1) / segs);
  const dim3 grid((unsigned)((a.ncol + kLineThreads - 1) / kLineThreads), (unsigned)((len + a.seg - 1) / a.seg));
  line_kernel<DIM, K1, MODE><<<grid, kLineThreads, (size_t)N * kLineThreads * 8, s>>>(a);
  TPSS_CUDA(cudaGetLastError());
}

template<int DIM, int K1>
void run(const SweepLaunch &l, cudaStream_t s)
{
  constexpr int N = 2 * K1;
  const tpss_layout &L = *l.layout;
  const FdTables &T = *l.tables;
  const int nx = L.nc[0], ny = L.nc[1], nz = DIM == 3 ? L.nc[2] : 1;
  SweepTab t;
  t.fix = T.fix64;
  t.fix_eo = T.fix64_eo;
  t.fexp = T.fexp;
  t.fexp_eo = T.fexp_eo;
  t.fd = T.fd64.ptr;
  t.fd_eo = T.fd64_eo.ptr;
  t.sym = T.has_eo ? T.sym.ptr : nullptr;
  t.es = (2 * L.n + 1) * T.npad64;
  t.es_eo = 4 * (L.n / 2) * T.hpad64 + T.npad64;
  t.fp64_only = !T.fix_ok;
  XArgs x;
  x.cell_start = L.lexicographic ? nullptr : L.d_cell_start.ptr;
  x.vfd = L.d_vertex_fd[0].ptr;
  x.nx = nx;
  x.ny = ny;
  x.nz = nz;
  x.modes = (int64_t)(nx - 1) * N;
  x.t = t;
  x.omega = l.omega;
  x.ras = l.ras;
  const int64_t mx = x.modes, my = (int64_t)(ny - 1) * N, gy = (int64_t)ny * K1, gz = (int64_t)nz * K1;
  x.in = l.src;
  x.out = l.a;
  launch_x<DIM, K1, true>(x, s);
  LineArgs a{};
  a.t = t;
  a.stride = mx;
  if constexpr(DIM == 3)
  {
    a.in = l.a;
    a.out = l.b;
    a.ncol = mx * gz;
    a.inner = mx;
    a.in_outer = gy * mx;
    a.out_outer = my * mx;
    a.vfd = L.d_vertex_fd[1].ptr;
    a.nc = ny;
    launch_line<DIM, K1, LINE_FORWARD>(a, s);
  }
  // the last direction
  {
    LineArgs z = a;
    z.in = DIM == 3 ? l.b : l.a;
    z.out = DIM == 3 ? l.c : l.b;
    z.ncol = DIM == 3 ? mx * my : mx;
    z.inner = z.ncol;
    z.in_outer = z.out_outer = 0;
    z.stride = z.ncol;
    z.vfd = L.d_vertex_fd[DIM - 1].ptr;
    z.nc = L.nc[DIM - 1];
    z.lam0 = T.lam_modes[0].ptr;
    z.lam1 = T.lam_modes[1].ptr;
    z.vfd0 = L.d_vertex_fd[0].ptr;
    z.vfd1 = L.d_vertex_fd[1].ptr;
    z.modes0 = mx;
    z.rcp = T.rcp_E > 0 ? T.rcp64.ptr : nullptr;
    z.E = T.rcp_E;
    launch_line<DIM, K1, LINE_SOLVE>(z, s);
  }
  if constexpr(DIM == 3)
  {
    a.in = l.c;
    a.out = l.a;
    a.in_outer = my * mx;
    a.out_outer = gy * mx;
    launch_line<DIM, K1, LINE_BACKWARD>(a, s);
  }
  x.in = DIM == 3 ? l.a : l.b;
  x.out = l.dst;
  launch_x<DIM, K1, false>(x, s);
}
}  // namespace

bool SWEEP_CAT(launch_sweep_, SWEEP_PART)(const SweepLaunch &l, cudaStream_t s)
{
#define SWEEP_CASE(K)                                    \
  if constexpr((K) % 3 == SWEEP_PART)                    \
    if(l.layout->k == (K))                               \
    {                                                    \
      if(l.layout->dim == 2) run<2, (K) + 1>(l, s);      \
      else run<3, (K) + 1>(l, s);                        \
      return true;                                       \
    }
  SWEEP_CASE(1)
  SWEEP_CASE(2)
  SWEEP_CASE(3)
  SWEEP_CASE(4)
  SWEEP_CASE(5)
  SWEEP_CASE(6)
  SWEEP_CASE(7)
#undef SWEEP_CASE
  return false;
}
}  // namespace tpss
