// sipg_lines.cu -- tables and launches of the line-by-line FP64 SIPG operator (sipg_lines.cuh).
#include <cmath>
#include <cstring>
#include <map>
#include <type_traits>

#include "element_ext.h"
#include "internal.h"
#include "sipg_lines.cuh"

namespace tpss
{
using namespace lines;

namespace
{
// Table of one cell width h (layout OpTab<N>)
template<int N>
void fill_table(const ext::Element<N> &s, double h, long double sigma, std::vector<long double> &t)
{
  using T = OpTab<N>;
  constexpr int H = T::H, HE = T::HE;
  t.assign(T::SIZE, 0.0L);
  // own block: stiffness and the cell's own terms of two interior faces with penalty sigma (the basis is
  // 1 at its own face node and 0 at the others); trace towards the upper neighbour
  long double M[N][N], C[N][N], b[N], g[N];
  for(int j = 0; j < N; ++j)
  {
    g[j] = s.g[j] / h;
    b[j] = 0.5L * g[j] - (j == N - 1 ? sigma : 0.0L);
  }
  for(int i = 0; i < N; ++i)
    for(int j = 0; j < N; ++j)
    {
      M[i][j] = s.mass[i][j] * h;
      C[i][j] = s.stiff[i][j] / h;
      // outward derivatives: g at the upper face, mirrored at the lower one
      const long double v1 = i == N - 1, u1 = j == N - 1, v0 = i == 0, u0 = j == 0;
      C[i][j] += sigma * (v1 * u1 + v0 * u0) - 0.5L * (g[j] * v1 + g[i] * u1 + g[N - 1 - j] * v0 + g[N - 1 - i] * u0);
    }
  auto even = [&](auto at, int i, int j) { return 2 * j == N - 1 ? at(i, j) : 0.5L * (at(i, j) + at(i, N - 1 - j)); };
  auto odd = [&](auto at, int i, int j) { return 0.5L * (at(i, j) - at(i, N - 1 - j)); };
  auto m = [&](int i, int j) { return M[i][j]; };
  auto c = [&](int i, int j) { return C[i][j]; };
  auto tr = [&](int, int j) { return b[j]; };
  for(int i = 0; i < HE; ++i)
  {
    for(int j = 0; j < HE; ++j)
    {
      t[T::ME + i * T::LME + j] = even(m, i, j);
      t[T::CE + i * T::LCE + j] = even(c, i, j);
    }
    t[T::CE + i * T::LCE + HE] = 0.25L * (g[i] + g[N - 1 - i]);
    if(i >= H) continue;
    for(int j = 0; j < H; ++j)
    {
      t[T::MO + i * T::LMO + j] = odd(m, i, j);
      t[T::CO + i * T::LCO + j] = odd(c, i, j);
    }
    t[T::CO + i * T::LCO + H] = 0.25L * (g[i] - g[N - 1 - i]);
  }
  for(int j = 0; j < HE; ++j) t[T::TE + j] = even(tr, 0, j);
  for(int j = 0; j < H; ++j) t[T::TO + j] = odd(tr, 0, j);
}

// F with sum_j |c_j| 2^F <= 2^62 in every row of [b, e) with row length len (rows of two lengths)
int scale_of(const std::vector<long double> &t, int b, int rows, int len, int b2, int rows2, int len2)
{
  double mx = 0.0;
  for(int i = 0; i < rows + rows2; ++i)
  {
    double s = 0.0;
    for(int j = 0; j < (i < rows ? len : len2); ++j)
      s += (double)std::fabs(t[i < rows ? b + i * len + j : b2 + (i - rows) * len2 + j]);
    mx = std::max(mx, s * (1.0 + 1e-14));
  }
  int e = 0;
  std::frexp(mx, &e);
  return 62 - e;
}

// false: the matrices' magnitudes leave no room for the vectors'
template<int N>
bool build(tpss_operator &op, const tpss_layout &L, Penalty pen)
{
  using T = OpTab<N>;
  static const ext::Element<N> s(make_shape_1d(N - 1));  // (0.1 ms and more in the 113 bits of an Arm host)
  const double gamma = double(L.k) * (L.k + 1);
  OpLines &O = op.lines;
  // of all directions' distinct widths: [integer tables][FP64 tables][exponents: 3 per width]; per direction:
  // [sigma: 3 per cell][width per cell]
  std::vector<int64_t> buf, ti;
  std::map<double, int> id;
  std::vector<double> t64;
  std::vector<int> exps;
  auto put = [&](const void *p, size_t words) {
    const size_t at = buf.size();
    buf.resize(at + words);
    std::memcpy(buf.data() + at, p, words * 8);
    return at;
  };
  for(int d = 0; d < L.dim; ++d)
  {
    const int n = L.nc[d];
    const double *h = L.h[d].data();
    std::vector<int32_t> width(n + n % 2, 0);
    for(int c = 0; c < n; ++c)
    {
      auto it = id.find(h[c]);
      if(it == id.end())
      {
        it = id.emplace(h[c], (int)id.size()).first;
        std::vector<long double> t;
        fill_table<N>(s, h[c], (long double)pen.in * gamma / h[c], t);
        const int F[3] = {scale_of(t, T::ME, T::HE, T::LME, T::MO, T::H, T::LMO),
                          scale_of(t, T::CE, T::HE, T::LCE, T::CO, T::H, T::LCO),
                          scale_of(t, T::TE, 1, T::LME, T::TO, 1, T::LMO)};
        for(int f : F)
          if(std::abs(f - 62) > fx::kTableRange) return false;
        for(int i = 0; i < T::SIZE; ++i)
        {
          const int f = i < T::CE ? F[0] : i < T::TE ? F[1] : F[2];
          ti.push_back(ext::limbs(t[i], f));
        }
        t64.insert(t64.end(), t.begin(), t.end());
        exps.insert(exps.end(), F, F + 3);
      }
      width[c] = it->second;
    }
    std::vector<double> sig(3 * (size_t)n);
    for(int c = 0; c < n; ++c)
    {
      sig[3 * c] = c == 0 ? pen.bd * 2.0 * gamma / h[c] : pen.in * 0.5 * gamma * (1.0 / h[c - 1] + 1.0 / h[c]);
      sig[3 * c + 1] = c == n - 1 ? pen.bd * 2.0 * gamma / h[c] : pen.in * 0.5 * gamma * (1.0 / h[c] + 1.0 / h[c + 1]);
      sig[3 * c + 2] = pen.in * gamma / h[c];
      if(c == 0 || c == n - 1 || h[c - 1] != h[c] || h[c + 1] != h[c]) width[c] |= kSpecial;
    }
    O.off_sig[d] = put(sig.data(), sig.size());
    O.off_width[d] = put(width.data(), width.size() / 2);
  }
  if(exps.size() % 2) exps.push_back(0);
  O.off_exps = put(exps.data(), exps.size() / 2);
  O.off_tab64 = put(t64.data(), t64.size());
  if(buf.size() % 2) buf.push_back(0);  // table rows are read as 16-byte pairs
  O.off_tab = put(ti.data(), ti.size());
  O.tables.upload(buf.data(), buf.size());
  return true;
}

template<int DIM, int N>
void run(const tpss_operator &op, double *buf, double *dst, const double *src, cudaStream_t s, const double *rhs)
{
  const tpss_layout &L = *op.layout;
  const OpLines &O = op.lines;
  const int64_t nd = L.n_dofs, gx = (int64_t)L.nc[0] * N, gy = (int64_t)L.nc[1] * N;
  auto args = [&](int d) {
    OpLineArgs a{};
    const int64_t *b = O.tables.ptr;
    a.tab = reinterpret_cast<const int2 *>(b + O.off_tab);
    a.tab64 = reinterpret_cast<const double *>(b + O.off_tab64);
    a.sig = reinterpret_cast<const double *>(b + O.off_sig[d]);
    a.exps = reinterpret_cast<const int *>(b + O.off_exps);
    a.width = reinterpret_cast<const int32_t *>(b + O.off_width[d]);
    a.cell_start = L.lexicographic ? nullptr : L.d_cell_start.ptr;
    for(int e = 0; e < 3; ++e) a.nc[e] = L.nc[e];
    return a;
  };
  {
    using C = OpXCfg<DIM, N>;
    OpLineArgs a = args(0);
    a.q = src;
    a.r = buf;
    a.m = buf + nd;
    if constexpr(C::smem() > 48 * 1024)  // per device; a cheap host call
      TPSS_CUDA(cudaFuncSetAttribute(op_x_kernel<DIM, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem()));
    const int ng = L.nc[1] * (DIM == 3 ? L.nc[2] : 1);
    // a long level has more tiles along x than a grid's second dimension holds: the third counts its multiples
    const int tiles = (L.nc[0] + C::XC - 1) / C::XC;
    const dim3 grid((ng + C::XG - 1) / C::XG, std::min(tiles, kMaxGridY), (tiles + kMaxGridY - 1) / kMaxGridY);
    op_x_kernel<DIM, N><<<grid, C::THREADS, C::smem(), s>>>(a);
    TPSS_CUDA(cudaGetLastError());
  }
  auto line_launch = [&](auto mode, OpLineArgs a, int d) {
    // segments as for the smoother's lines (sweep64.cu): enough threads to fill the chip
    const int len = L.nc[d];
    int64_t segs = ((int64_t)num_sms() * 2048 + a.ncol - 1) / a.ncol;
    segs = std::min<int64_t>(std::max<int64_t>(segs, 1), std::min(len, kMaxGridY));
    a.seg = (int)((len + segs - 1) / segs);
    const dim3 grid((unsigned)((a.ncol + kOpThreads - 1) / kOpThreads), (unsigned)((len + a.seg - 1) / a.seg));
    op_line_kernel<DIM, N, decltype(mode)::value><<<grid, kOpThreads, 0, s>>>(a);
    TPSS_CUDA(cudaGetLastError());
  };
  if constexpr(DIM == 3)
  {
    OpLineArgs a = args(1);
    a.p = buf;
    a.q = buf + nd;
    a.r = buf + 2 * nd;
    a.m = buf + 3 * nd;
    a.ncol = gx * L.nc[2] * N;
    a.inner = gx;
    a.outer = gx * gy;
    a.stride = gx;
    line_launch(std::integral_constant<int, OP_INNER>{}, a, 1);
  }
  OpLineArgs a = args(DIM - 1);
  a.p = DIM == 3 ? buf + 2 * nd : buf;
  a.q = DIM == 3 ? buf + 3 * nd : buf + nd;
  a.r = dst;
  a.rhs = rhs;
  a.ncol = DIM == 3 ? gx * gy : gx;
  a.inner = a.ncol;
  a.outer = 0;
  a.stride = a.ncol;
  if(rhs) line_launch(std::integral_constant<int, OP_RESIDUAL>{}, a, DIM - 1);
  else line_launch(std::integral_constant<int, OP_LAST>{}, a, DIM - 1);
}
}  // namespace

namespace
{
template<typename F>
void for_size(int np, const F &f)
{
  switch(np)
  {
  case 2: f(std::integral_constant<int, 2>{}); break;
  case 3: f(std::integral_constant<int, 3>{}); break;
  case 4: f(std::integral_constant<int, 4>{}); break;
  case 5: f(std::integral_constant<int, 5>{}); break;
  case 6: f(std::integral_constant<int, 6>{}); break;
  case 7: f(std::integral_constant<int, 7>{}); break;
  case 8: f(std::integral_constant<int, 8>{}); break;
  default: break;
  }
}
}  // namespace

// Whether the passes are faster than the cell-wise kernel. On small levels both are latency: replayed in a graph the
// passes take 8 to 11 us in 2D and 13 to 20 us in 3D, the cell-wise kernel 6 to 10, 8 to 12 and 10 to 15 us for k = 1, 2, 3 in 2D
// and 9, 12, 14, 17 and 20 us for k = 1 .. 5 in 3D; beyond that its multiply-adds cost 1.7 us per million
// (2 per clock and SM), the passes' about 0.28 of that. The lines below are where the two meet. Measured, cell-wise and
// passes: 2D k = 1 160^2 cells 12.1 and 12.4 us; 3D k = 1 24^3 15.2 and 17.3, 28^3 23.1 and 20.6; k = 2 16^3 16.2 and 16.4, 20^3
// 25.2 and 20.5; k = 3 10^3 14.8 and 15.6, 12^3 19.2 and 16.2; k = 4 5^3 17.0 and 16.5
static bool lines_pay(const tpss_layout &L)
{
  static const double from[2][8] = {{0, 4.6, 1.4, 0, 0, 0, 0, 0}, {0, 11.3, 7.8, 5.5, 0.8, 0, 0, 0}};
  const double n = L.np, cells = (double)L.nc[0] * L.nc[1] * (L.dim == 3 ? L.nc[2] : 1);
  const double fma = L.dim == 2 ? n * (4 * n * n + 4 * (2 * n + 2)) : n * n * (8 * n * n + 6 * (2 * n + 2));
  return cells * fma * 1.7e-6 >= from[L.dim - 2][L.k];
}

// Tables and intermediate vectors, allocated with the operator: a first product costs what the others do, and one
// inside a stream capture takes the same route. Whether there is room is decided here once.
void build_op_lines(tpss_operator &op, const tpss_layout &L, Penalty pen)
{
  if(!lines_pay(L)) return;
  OpLines &O = op.lines;
  if(!O.buf.try_resize((size_t)L.n_dofs * (L.dim == 3 ? 4 : 2))) return;
  O.order.create();
  for_size(L.np, [&](auto n) {
    if(!build<decltype(n)::value>(op, L, pen)) O.buf.release();
  });
}

bool op_lines_apply(tpss_operator &op, double *dst, const double *src, cudaStream_t s, const double *rhs)
{
  const tpss_layout &L = *op.layout;
  OpLines &O = op.lines;
  if(O.buf.n == 0) return false;
  const ScratchUse use(O.order, s);
  for_size(L.np, [&](auto n) {
    if(L.dim == 2) run<2, decltype(n)::value>(op, O.buf.ptr, dst, src, s, rhs);
    else run<3, decltype(n)::value>(op, O.buf.ptr, dst, src, s, rhs);
  });
  return true;
}
}  // namespace tpss
