// c0ip_band.cuh -- the two passes of the C0IP operator (c0ip.cu: bands along x, then along y) with their
// contractions on the integer pipe (fixed64.cuh).
//
// A thread takes the K nodes of one cell (its first vertex and the K - 1 inside, K the degree): they share a
// window of 4K + 1 values, which is turned into integers with one exponent once. Only the entries that the
// discretization couples are contracted: the vertex with the two cells on either side (B) or its own two
// (M, L), the other nodes with their cell and its neighbours, or their cell. On a uniform grid all cells but
// those next to the boundary have the same rows: a few classes of rows, held in shared memory, where the
// lanes of a warp read one address.
// Measured, 256^2 cells, K = 3 (767^2 values): x pass 48 -> 14 us, y pass 75 -> 16 us against a thread per
// node with FP64 bands (the x pass waited on its coefficients, 104 bytes apart from lane to lane, the y
// pass on the FP64 pipe: 41 instructions of 64 clocks).
#pragma once

#include "fixed64.cuh"

namespace tpss
{
namespace band
{
constexpr int kMaxClasses = 8;  // distinct sets of rows a launch can hold

// rows of one class, in 8-byte words: the vertex' rows of B, M and L, then those of the other nodes
template<int K>
struct Tab
{
  static constexpr int pad2(int x) { return (x + 1) / 2 * 2; }
  static constexpr int WB = 4 * K + 1, WM = 2 * K + 1;  // window of B; of M and L (its middle)
  static constexpr int NB = 3 * K + 1, NM = K + 1;      // entries of the other nodes, from K on in the windows
  static constexpr int M0 = pad2(WB), L0 = M0 + pad2(WM), R = L0 + pad2(WM);
  static constexpr int RM = pad2(NB), RL = RM + pad2(NM), RS = RL + pad2(NM);
  static constexpr int SIZE = R + (K - 1) * RS;
};

struct BandArgs
{
  const double *a, *b, *c;   // x pass: u; y pass: tm, tl, tb
  double *ra, *rb, *rc;      // x pass: tm, tl, tb; y pass: dst
  const double *M, *L, *B;   // FP64 bands (rows of 4 K + 1), for values the integers do not cover
  const int2 *tab;           // integer rows per class
  const int32_t *cls;        // class of every cell
  int n_cls, n, nc;
  int FM, FL, FB;            // exponents of the integer rows
  double mixed;
};

template<int LEN>
__device__ __forceinline__ int64_t dot(const int2 *__restrict__ row, const int *xh, const int *xl)
{
  fx::Acc M, S;
  const int4 *row4 = reinterpret_cast<const int4 *>(row);
#pragma unroll
  for(int j2 = 0; j2 < (LEN + 1) / 2; ++j2)
  {
    const int4 c = row4[j2];
    if(j2 == 0) M.start(c.y, xl[0]);
    else M.add(c.y, xl[2 * j2]);
    M.add(c.x, xh[2 * j2]);
    if(j2 == 0) S.start(c.y, xh[0]);
    else S.add(c.y, xh[2 * j2]);
    if(2 * j2 + 1 < LEN)
    {
      const int j = 2 * j2 + 1 < LEN ? 2 * j2 + 1 : 0;
      M.add(c.w, xl[j]);
      M.add(c.z, xh[j]);
      S.add(c.w, xh[j]);
    }
  }
  return S.value() + (M.hi + (int)(M.lo >> 31));
}

// a window in limbs: |x| < 2^58, so that up to 4 * 7 + 1 terms stay within the accumulators. Returns its
// exponent (unit 2^(e - 1023 - 57)), or -1 for values the integers do not cover
template<int W>
__device__ __forceinline__ int to_limbs(const double (&v)[W], int (&h)[W], int (&l)[W])
{
  unsigned hi = 0, lo = 0;
#pragma unroll
  for(int i = 0; i < W; ++i)
  {
    hi = max(hi, (unsigned)__double2hiint(v[i]) & 0x7fffffffu);
    lo |= (unsigned)__double2loint(v[i]);
  }
  const int e = (int)(hi >> 20);
  if((e < 1023 - 300 || e > 1023 + 300) && (hi | lo) != 0) return -1;
  const int emax = hi == 0 ? 1023 : e;
#pragma unroll
  for(int i = 0; i < W; ++i) fx::split(fx::from_double(v[i], emax + 1), h[i], l[i]);
  return emax;
}

// out[r] = row r of M or L (RO, RR: words of the vertex' and of the other nodes' rows) times the window of
// 2 K + 1 values
template<int K, int RO, int RR>
__device__ __forceinline__ void contract_m(const int2 *tab, const int *h, const int *l, int ex, double (&out)[K])
{
  using T = Tab<K>;
  out[0] = fx::to_double(dot<T::WM>(tab + RO, h, l), ex);
#pragma unroll
  for(int r = 1; r < K; ++r) out[r] = fx::to_double(dot<T::NM>(tab + T::R + (r - 1) * T::RS + RR, h + K, l + K), ex);
}
template<int K>
__device__ __forceinline__ void contract_b(const int2 *tab, const int *h, const int *l, int ex, double (&out)[K])
{
  using T = Tab<K>;
  out[0] = fx::to_double(dot<T::WB>(tab, h, l), ex);
#pragma unroll
  for(int r = 1; r < K; ++r) out[r] = fx::to_double(dot<T::NB>(tab + T::R + (r - 1) * T::RS, h + K, l + K), ex);
}

// FP64 band rows of the nodes of cell c (node numbers c K + r - 1, rolled): half width hw of 2 K
template<int K>
__device__ __forceinline__ void contract_fp64(const double *A, const double *v, int64_t stride, int n, int c, int hw,
                                              double *out)
{
#pragma unroll 1
  for(int r = 0; r < K; ++r)
  {
    const int i = c * K + r - 1;
    double s = 0.0;
#pragma unroll 1
    for(int j = max(0, i - hw); i >= 0 && j <= min(n - 1, i + hw); ++j)
      s = fma(A[(int64_t)i * (4 * K + 1) + j - i + 2 * K], v[j * stride], s);
    out[r] = s;
  }
}

template<int K, int W>
__device__ __forceinline__ void load_window(const double *v, int64_t stride, int n, int first, double (&w)[W])
{
#pragma unroll
  for(int j = 0; j < W; ++j)
  {
    const int i = first + j;
    w[j] = i >= 0 && i < n ? v[i * stride] : 0.0;
  }
}

template<int K>
__device__ __forceinline__ void load_tables(const BandArgs &a, int2 *s_tab)
{
  for(int i = threadIdx.x; i < a.n_cls * Tab<K>::SIZE; i += blockDim.x) s_tab[i] = a.tab[i];
  __syncthreads();
}

// ra = M_x u, rb = L_x u, rc = B_x u; consecutive threads take consecutive cells of a row
template<int K>
__global__ void __launch_bounds__(128) band_x_kernel(BandArgs a)
{
  using T = Tab<K>;
  extern __shared__ __align__(16) int2 s_tab[];
  load_tables<K>(a, s_tab);
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if(t >= (int64_t)a.nc * a.n) return;
  const int c = (int)(t % a.nc);
  const int64_t row = t / a.nc * a.n;
  double w[T::WB], om[K], ol[K], ob[K];
  load_window<K>(a.a + row, 1, a.n, c * K - 2 * K - 1, w);
  int h[T::WB], l[T::WB];
  const int e = to_limbs(w, h, l);
  if(e >= 0)
  {
    const int2 *tab = s_tab + a.cls[c] * T::SIZE;
    const int ex = e - 1023 - 57 + 64;
    contract_m<K, T::M0, T::RM>(tab, h + K, l + K, ex - a.FM, om);
    contract_m<K, T::L0, T::RL>(tab, h + K, l + K, ex - a.FL, ol);
    contract_b<K>(tab, h, l, ex - a.FB, ob);
  }
  else
  {
    double s[K];
    auto slow = [&](const double *A, int hw, double (&out)[K]) {
      contract_fp64<K>(A, a.a + row, 1, a.n, c, hw, s);
#pragma unroll
      for(int r = 0; r < K; ++r) out[r] = s[r];
    };
    slow(a.M, K, om);
    slow(a.L, K, ol);
    slow(a.B, 2 * K, ob);
  }
#pragma unroll
  for(int r = 0; r < K; ++r)
  {
    const int i = c * K + r - 1;
    if(i < 0) continue;
    a.ra[row + i] = om[r];
    a.rb[row + i] = ol[r];
    a.rc[row + i] = ob[r];
  }
}

// ra = M_y tb + mixed L_y tl + B_y tm; consecutive threads take consecutive columns
template<int K>
__global__ void __launch_bounds__(128) band_y_kernel(BandArgs a)
{
  using T = Tab<K>;
  extern __shared__ __align__(16) int2 s_tab[];
  load_tables<K>(a, s_tab);
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if(t >= (int64_t)a.nc * a.n) return;
  const int x = (int)(t % a.n), c = (int)(t / a.n);
  const int2 *tab = s_tab + a.cls[c] * T::SIZE;
  double s[K], o[K];
  auto slow = [&](const double *A, const double *v, int hw) {
    double q[K];
    contract_fp64<K>(A, v + x, a.n, a.n, c, hw, q);
#pragma unroll
    for(int r = 0; r < K; ++r) o[r] = q[r];
  };
  {
    double w[T::WB];
    int h[T::WB], l[T::WB];
    load_window<K>(a.a + x, a.n, a.n, c * K - 2 * K - 1, w);
    const int e = to_limbs(w, h, l);
    if(e >= 0) contract_b<K>(tab, h, l, e - 1023 - 57 + 64 - a.FB, o);
    else slow(a.B, a.a, 2 * K);
#pragma unroll
    for(int r = 0; r < K; ++r) s[r] = o[r];
  }
  double w[T::WM];
  int h[T::WM], l[T::WM];
  load_window<K>(a.c + x, a.n, a.n, c * K - K - 1, w);
  int e = to_limbs(w, h, l);
  if(e >= 0) contract_m<K, T::M0, T::RM>(tab, h, l, e - 1023 - 57 + 64 - a.FM, o);
  else slow(a.M, a.c, K);
#pragma unroll
  for(int r = 0; r < K; ++r) s[r] += o[r];
  load_window<K>(a.b + x, a.n, a.n, c * K - K - 1, w);
  e = to_limbs(w, h, l);
  if(e >= 0) contract_m<K, T::L0, T::RL>(tab, h, l, e - 1023 - 57 + 64 - a.FL, o);
  else slow(a.L, a.b, K);
#pragma unroll
  for(int r = 0; r < K; ++r)
  {
    const int i = c * K + r - 1;
    if(i >= 0) a.ra[(int64_t)i * a.n + x] = fma(a.mixed, o[r], s[r]);
  }
}
}  // namespace band
}  // namespace tpss
