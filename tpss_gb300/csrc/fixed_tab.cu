// fixed_tab.cu -- integer forms of the FP64 fast-diagonalization tables (fixed64.cuh).
//
// Coefficients become c 2^F, rounded to the nearest integer, with one F per entry for the rows of
// S^T and one for the rows of S: the largest power of two with sum_j |c_ij| 2^F <= 2^62 in every
// row (even/odd forms: in every row of the two half matrices).
#include "internal.h"

namespace tpss
{
namespace
{
// One CTA per entry; an entry holds two matrices (S^T, S) of `rows` rows of npad coefficients each
// (stride npad, the padding zero), `size` words per entry.
__global__ void __launch_bounds__(64) fixed_table_kernel(const double *__restrict__ tab, int rows, int npad, int size,
                                                         int2 *__restrict__ out, int2 *__restrict__ fexp)
{
  __shared__ unsigned long long s_max[2];
  const double *E = tab + (size_t)blockIdx.x * size;
  int2 *O = out + (size_t)blockIdx.x * size;
  if(threadIdx.x < 2) s_max[threadIdx.x] = 0;
  __syncthreads();
  for(int i = threadIdx.x; i < 2 * rows; i += blockDim.x)
  {
    double s = 0.0;
    for(int j = 0; j < npad; ++j) s += fabs(E[i * npad + j]);
    // non-negative doubles compare like their bits
    atomicMax(&s_max[i / rows], (unsigned long long)__double_as_longlong(s * (1.0 + 1e-14)));
  }
  __syncthreads();
  int F[2];
  for(int m = 0; m < 2; ++m)
  {
    const double s = __longlong_as_double((long long)s_max[m]);
    int e = 0;
    if(s > 0.0 && s < 1e300) frexp(s, &e);  // s < 2^e
    F[m] = 62 - e;
  }
  for(int i = threadIdx.x; i < size; i += blockDim.x)
  {
    int2 v = make_int2(0, 0);
    if(i < 2 * rows * npad)
    {
      const double c = E[i];
      const long long x = fabs(c) < 1e300 ? llrint(scalbn(c, F[i / (rows * npad)])) : 0;
      v.x = (int)x;
      v.y = (int)((x - v.x) >> 32);
    }
    O[i] = v;
  }
  if(threadIdx.x == 0) fexp[blockIdx.x] = make_int2(F[0], F[1]);
}
}  // namespace

void build_fixed_tables(FdTables &T)
{
  static std::mutex mu;  // tables are shared by shallow copies
  std::lock_guard<std::mutex> lock(mu);
  if(T.n_entries == 0 || T.fix64) return;
  const int n = T.n, h = n / 2;
  const size_t E = T.n_entries, es = (2 * n + 1) * T.npad64, es_eo = T.has_eo ? 4 * h * T.hpad64 + T.npad64 : 0;
  T.fix_buf.resize(E * (es + es_eo + 2));
  int2 *fix = T.fix_buf.ptr, *eo = fix + E * es, *fe = eo + E * es_eo;
  fixed_table_kernel<<<T.n_entries, 64>>>(T.fd64.ptr, n, T.npad64, (int)es, fix, fe);
  if(T.has_eo) fixed_table_kernel<<<T.n_entries, 64>>>(T.fd64_eo.ptr, 2 * h, T.hpad64, (int)es_eo, eo, fe + E);
  TPSS_CUDA(cudaGetLastError());
  TPSS_CUDA(cudaStreamSynchronize(nullptr));  // the tables are read on any stream
  T.fix64 = fix;
  T.fix64_eo = eo;
  T.fexp = fe;
  T.fexp_eo = fe + E;
}
}  // namespace tpss
