// c0ip_band.cuh -- the two passes of the C0IP operator (c0ip.cu: bands along x, then along y) with their
// contractions on the integer pipe (fixed64.cuh).
//
// A thread takes the K nodes of one cell (its first vertex and the K - 1 inside, K the degree): they share a
// window of 4K + 1 values, which is turned into integers with one exponent, or with several where the part of
// it that a row contracts is much smaller than the rest (narrow_to). Only the entries that the
// discretization couples are contracted: the vertex with the two cells on either side (B) or its own two
// (M, L), the other nodes with their cell and its neighbours, or their cell. On a uniform grid all cells but
// those next to the boundary have the same rows: a few classes of rows, held in shared memory, where the
// lanes of a warp read one address.
// Measured, 256^2 cells, K = 3 (767^2 values): x pass 48 -> 12.6 us, y pass 75 -> 17.0 us against a thread per
// node with FP64 bands (the x pass waited on its coefficients, 104 bytes apart from lane to lane, the y
// pass on the FP64 pipe: 41 instructions of 64 clocks). With one unit for the whole window and
// without the low products 11.1 and 14.0 us.
#pragma once

#include <type_traits>

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

// with the products of the low limbs: the bilaplacian's entries differ by a factor of 1e2 to 1e5, and its small
// ones would lose them (k = 5, slowly varying vector: 1.03e-15 off without, 0.98e-15 with, as the FP64 bands)
template<int LEN>
__device__ __forceinline__ int64_t dot(const int2 *__restrict__ row, const int *xh, const int *xl)
{
  int h[LEN], l[LEN];
#pragma unroll
  for(int i = 0; i < LEN; ++i)
  {
    h[i] = xh[i];
    l[i] = xl[i];
  }
  return fx::row_dot<LEN, true>(row, h, l);
}

// A window of W values in limbs: |x| < 2^58, so that up to 4 * 7 + 1 terms stay within the accumulators, with
// unit 2^(e - 1023 - 57); e = -1: the integers do not cover the largest value
template<int W>
struct Window
{
  int h[W], l[W];
  int e;
};

// largest high word and OR of the low words of part of a window
struct Mag
{
  unsigned hi = 0, lo = 0;
  __device__ __forceinline__ void operator|=(const Mag &o)
  {
    hi = max(hi, o.hi);
    lo |= o.lo;
  }
  __device__ __forceinline__ bool zero() const { return (hi | lo) == 0; }
  // the integers' exponent, or -1
  __device__ __forceinline__ int exponent() const
  {
    const int e = (int)(hi >> 20);
    return e < 1023 - fx::kRange || e > 1023 + fx::kRange ? -1 : e;
  }
};

template<int FIRST, int LEN, int W>
__device__ __forceinline__ Mag magnitude(const double (&v)[W])
{
  Mag m;
#pragma unroll
  for(int i = FIRST; i < FIRST + LEN; ++i)
  {
    m.hi = max(m.hi, (unsigned)__double2hiint(v[i]) & 0x7fffffffu);
    m.lo |= (unsigned)__double2loint(v[i]);
  }
  return m;
}

template<int W>
__device__ __forceinline__ void to_limbs(const double (&v)[W], const Mag &all, Window<W> &w)
{
  w.e = all.zero() ? 1023 : all.exponent();
#pragma unroll
  for(int i = 0; i < W; ++i) fx::split(fx::from_double(v[i], w.e + 1), w.h[i], w.l[i]);
}

// Rows contract a part of the window only, and what they leave out must not set their unit: a value 1e8 times
// larger two cells away would cost an inside node 26 of its bits. The window is used from its widest part to its
// narrowest; where the next part's largest value (m) lies more than kSlack binades below the present unit's, its
// values at(i) are read once more and get a unit of their own. One binade is left as it is: it costs one of the
// bits beyond FP64's 53, and with values of one magnitude some thread of most warps would come here for it.
// Returns the unit's exponent, or -1 (the part is summed in FP64).
constexpr int kSlack = 1;
template<int FIRST, int LEN, int W, typename At>
__device__ __forceinline__ int narrow_to(Window<W> &w, const Mag &m, const At &at)
{
  if(w.e < 0 || m.zero()) return w.e;
  const int e = m.exponent();
  if(e >= 0 && w.e - e > kSlack)
  {
    w.e = e;
#pragma unroll
    for(int i = FIRST; i < FIRST + LEN; ++i) fx::split(fx::from_double(at(i), e + 1), w.h[i], w.l[i]);
  }
  return e < 0 ? -1 : w.e;
}

// FP64 band rows [r0, r1) of the nodes of cell c (node numbers c K + r - 1, rolled): half width hw of 2 K
template<int K>
__device__ __forceinline__ void contract_fp64(const double *A, const double *v, int64_t stride, int n, int c, int hw,
                                              int r0, int r1, double (&out)[K])
{
  double o[K];
#pragma unroll 1
  for(int r = r0; r < r1; ++r)
  {
    const int i = c * K + r - 1;
    double s = 0.0;
#pragma unroll 1
    for(int j = max(0, i - hw); i >= 0 && j <= min(n - 1, i + hw); ++j)
      s = fma(A[(int64_t)i * (4 * K + 1) + j - i + 2 * K], v[j * stride], s);
    o[r] = s;
  }
#pragma unroll
  for(int r = 0; r < K; ++r)
    if(r >= r0 && r < r1) out[r] = o[r];
}

// One direction's products with the K nodes of cell c of a line v (n values, stride apart): B v from a
// window of 4 K + 1 values, M v and L v from one of 2 K + 1; vertex: the vertex' row, else the
// others'; e: the exponent of the part they contract (-1: FP64)
template<int K>
struct Line
{
  const BandArgs &a;
  const int2 *tab;
  const double *v;
  int64_t stride;
  int c;

  // value i of a window that begins at node c K - FIRST
  template<int FIRST>
  __device__ __forceinline__ double at(int i) const
  {
    const int j = c * K - FIRST + i;
    return j >= 0 && j < a.n ? v[j * stride] : 0.0;
  }
  template<int RO, int RR, int F, int W>
  __device__ __forceinline__ void mass_like(const Window<W> &w, bool vertex, int e, const double *A, int fe,
                                            double (&out)[K]) const
  {
    // F: first value of the 2 K + 1 in the window
    using T = Tab<K>;
    if(e < 0)
    {
      contract_fp64<K>(A, v, stride, a.n, c, K, vertex ? 0 : 1, vertex ? 1 : K, out);
      return;
    }
    const int ex = e - 1023 - 57 + 64 - fe;
    if(vertex) out[0] = fx::to_double(dot<T::WM>(tab + RO, w.h + F, w.l + F), ex);
    else
#pragma unroll
      for(int r = 1; r < K; ++r)
        out[r] = fx::to_double(dot<T::NM>(tab + T::R + (r - 1) * T::RS + RR, w.h + F + K, w.l + F + K), ex);
  }
  template<int W>
  __device__ __forceinline__ void bilaplacian(const Window<W> &w, bool vertex, int e, double (&out)[K]) const
  {
    using T = Tab<K>;
    if(e < 0)
    {
      contract_fp64<K>(a.B, v, stride, a.n, c, 2 * K, vertex ? 0 : 1, vertex ? 1 : K, out);
      return;
    }
    const int ex = e - 1023 - 57 + 64 - a.FB;
    if(vertex) out[0] = fx::to_double(dot<T::WB>(tab, w.h, w.l), ex);
    else
#pragma unroll
      for(int r = 1; r < K; ++r)
        out[r] = fx::to_double(dot<T::NB>(tab + T::R + (r - 1) * T::RS, w.h + K, w.l + K), ex);
  }
};

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
  const Line<K> ln{a, s_tab + a.cls[c] * T::SIZE, a.a + row, 1, c};
  auto at = [&](int i) { return ln.template at<2 * K + 1>(i); };
  double v[T::WB], om[K], ol[K], ob[K];
#pragma unroll
  for(int i = 0; i < T::WB; ++i) v[i] = at(i);
  // parts of the window: the cell with its vertices, with the cell below (the vertex' rows of M and L), with
  // the cell above as well (the other nodes' rows of B), and all (the vertex' row of B)
  const Mag own = magnitude<2 * K, K + 1>(v);
  Mag mid = magnitude<K, K>(v);
  mid |= own;
  Mag three = magnitude<3 * K + 1, K>(v);
  three |= mid;
  Mag all = magnitude<0, K>(v);
  all |= three;
  Window<T::WB> w;
  to_limbs(v, all, w);
  ln.bilaplacian(w, true, w.e, ob);
  ln.bilaplacian(w, false, narrow_to<K, 3 * K + 1>(w, three, at), ob);
  int e = narrow_to<K, 2 * K + 1>(w, mid, at);
  ln.template mass_like<T::M0, T::RM, K>(w, true, e, a.M, a.FM, om);
  ln.template mass_like<T::L0, T::RL, K>(w, true, e, a.L, a.FL, ol);
  e = narrow_to<2 * K, K + 1>(w, own, at);
  ln.template mass_like<T::M0, T::RM, K>(w, false, e, a.M, a.FM, om);
  ln.template mass_like<T::L0, T::RL, K>(w, false, e, a.L, a.FL, ol);
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
  {
    const Line<K> ln{a, tab, a.a + x, a.n, c};
    auto at = [&](int i) { return ln.template at<2 * K + 1>(i); };
    double v[T::WB];
#pragma unroll
    for(int i = 0; i < T::WB; ++i) v[i] = at(i);
    const Mag three = magnitude<K, 3 * K + 1>(v);
    Mag all = magnitude<0, K>(v);
    all |= three;
    Window<T::WB> w;
    to_limbs(v, all, w);
    ln.bilaplacian(w, true, w.e, s);
    ln.bilaplacian(w, false, narrow_to<K, 3 * K + 1>(w, three, at), s);
  }
  auto add = [&](const double *q, auto row0, auto row, const double *A, int fe) {
    const Line<K> ln{a, tab, q + x, a.n, c};
    auto at = [&](int i) { return ln.template at<K + 1>(i); };
    double v[T::WM];
#pragma unroll
    for(int i = 0; i < T::WM; ++i) v[i] = at(i);
    const Mag own = magnitude<K, K + 1>(v);
    Mag mid = magnitude<0, K>(v);
    mid |= own;
    Window<T::WM> w;
    to_limbs(v, mid, w);
    ln.template mass_like<decltype(row0)::value, decltype(row)::value, 0>(w, true, w.e, A, fe, o);
    ln.template mass_like<decltype(row0)::value, decltype(row)::value, 0>(w, false, narrow_to<K, K + 1>(w, own, at), A,
                                                                          fe, o);
  };
  add(a.c, std::integral_constant<int, T::M0>{}, std::integral_constant<int, T::RM>{}, a.M, a.FM);
#pragma unroll
  for(int r = 0; r < K; ++r) s[r] += o[r];
  add(a.b, std::integral_constant<int, T::L0>{}, std::integral_constant<int, T::RL>{}, a.L, a.FL);
#pragma unroll
  for(int r = 0; r < K; ++r)
  {
    const int i = c * K + r - 1;
    if(i >= 0) a.ra[(int64_t)i * a.n + x] = fma(a.mixed, o[r], s[r]);
  }
}
}  // namespace band
}  // namespace tpss
