// transfer64.cu -- tables and launches of the FP64 level transfer (transfer64.cuh).
#include <cmath>
#include <cstring>

#include "element_ext.h"
#include "internal.h"
#include "transfer64.cuh"

namespace tpss
{
using namespace tr64;

namespace
{
template<int N>
void append_tables(std::vector<double> &buf)
{
  using T = TrTab<N>;
  const ext::Element<N> el(make_shape_1d(N - 1));
  // first child's rows; the second child's mirror them
  ext::Real E[N][N], d[N];
  for(int i = 0; i < N; ++i) el.lagrange(el.x[i] / 2, E[i], d);
  auto at = [&](int r, int m) { return r < N ? E[r][m] : E[2 * N - 1 - r][N - 1 - m]; };
  auto exponent = [](ext::Real s) {
    int e = 0;
    std::frexp(s * (1 + 1e-14L), &e);
    return 62 - e;
  };
  // rows of nodes that are coarse ones have a single entry and are left out (transfer64.cuh)
  constexpr int ROWS = T::ROWS;
  ext::Real row = 0, col = 0;
  for(int r = 1; r <= ROWS; ++r)
  {
    ext::Real s = 0;
    for(int m = 0; m < N; ++m) s += std::fabs(at(r, m));
    row = std::max(row, s);
  }
  for(int m = 0; m < N; ++m)
  {
    ext::Real s = 0;
    for(int r = 1; r <= ROWS; ++r) s += std::fabs(at(r, m)) + std::fabs(at(2 * N - 1 - r, m));
    col = std::max(col, s);
  }
  const int32_t F[2] = {exponent(row), exponent(col)};
  std::vector<int64_t> t(T::SIZE + 1, 0);
  for(int i = 0; i < ROWS; ++i)
    for(int j = 0; j < T::HE; ++j)
    {
      const ext::Real *e = E[1 + i];
      const bool mid = 2 * j == N - 1;
      t[T::PE + i * T::LPE + j] = ext::limbs(mid ? e[j] : (e[j] + e[N - 1 - j]) / 2, F[0]);
      if(!mid) t[T::PO + i * T::LPO + j] = ext::limbs((e[j] - e[N - 1 - j]) / 2, F[0]);
    }
  for(int i = 0; i < T::HE; ++i)
    for(int j = 0; j < ROWS; ++j)
    {
      // for the middle node both children's values have the same coefficient
      const ext::Real a = at(1 + j, i), b = at(2 * N - 2 - j, i);
      t[T::RE + i * T::LR + j] = ext::limbs((a + b) / 2, F[1]);
      if(i < T::H) t[T::RO + i * T::LR + j] = ext::limbs((a - b) / 2, F[1]);
    }
  std::memcpy(&t[T::SIZE], F, 8);
  const size_t n = buf.size();
  buf.resize(n + t.size());
  std::memcpy(buf.data() + n, t.data(), t.size() * 8);
}

template<int DIM, int N>
void launch(const TrArgs64 &a, bool restrict_mode, cudaStream_t s)
{
  using C = TrCfg<DIM, N>;
  const unsigned grid = (unsigned)((a.n_coarse + C::CPB - 1) / C::CPB);
  if(restrict_mode) transfer64_kernel<DIM, N, true><<<grid, C::THREADS, 0, s>>>(a);
  else transfer64_kernel<DIM, N, false><<<grid, C::THREADS, 0, s>>>(a);
  TPSS_CUDA(cudaGetLastError());
}

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
  default: fail(TPSS_ERR_NOT_IMPLEMENTED, "unsupported (dim, degree)");
  }
}
}  // namespace

void append_transfer_tables(int np, std::vector<double> &buf)
{
  for_size(np, [&](auto n) { append_tables<decltype(n)::value>(buf); });
}

void transfer_apply64(int dim, int k, const int *ncc, const double *E_dev, bool restrict_mode, double *coarse, double *fine,
                      cudaStream_t s)
{
  TrArgs64 a{coarse, fine, E_dev, {1, 1, 1}, 1};
  for(int d = 0; d < dim; ++d)
  {
    a.ncc[d] = ncc[d];
    a.n_coarse *= ncc[d];
  }
  for_size(k + 1, [&](auto n) {
    if(dim == 2) launch<2, decltype(n)::value>(a, restrict_mode, s);
    else launch<3, decltype(n)::value>(a, restrict_mode, s);
  });
}
}  // namespace tpss
