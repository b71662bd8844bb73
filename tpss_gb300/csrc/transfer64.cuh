// transfer64.cuh -- FP64 transfer between a coarse cell and its 2^dim children on the integer pipe.
//
// Embedding into both children along a direction is one mirror-symmetric 2N x N matrix, so a pencil takes
// N^2 products in even/odd form for all 2N results (and back). Prolongation widens the coarse cell
// along x, y and z in turn (N^(d-1), 2 N^(d-1), 4 N^(d-1) pencils), restriction goes the other way. The
// fine vector is read and written by the threads of the z (2D: y) pass, which hold a pencil of both children
// each; their order runs through a child's layer, so that they read and write whole rows. Between
// the passes the cell lives in shared memory as 64-bit integers with one exponent (fixed64.cuh):
// every pass is scaled by 4, the room its coefficients' row sums leave, so its rounding is 2^-58 of the
// cell's largest value.
// Values the integers do not cover (infinities, NaN, magnitudes outside 2^(+-300)) take FP64 passes on the
// same shared memory, cell by cell.
//
// Measured, 16^3 coarse cells, k = 4 (4.1M fine values): prolongation 24.9 us, restriction 24.5 us, where the tree
// of FP64 passes per child took 90 and 92 us (FP64 pipe). The fine values move in 10 and 5 us at the copy
// rate; the rest is the serial chain of three passes, hidden behind the other CTAs of the SM only in
// part. 2^3 coarse cells take 6 and 5 us instead of 25 and 27. Fetching the fine values that the prolongation adds to
// before the passes instead of at the addition: 31.8 -> 24.9 us.
#pragma once

#include "fixed64.cuh"

namespace tpss
{
namespace tr64
{
// integer tables of a degree, in 8-byte words, behind the FP64 embeddings [2][N N]
template<int N>
struct TrTab
{
  static constexpr int pad2(int x) { return (x + 1) / 2 * 2; }
  static constexpr int H = N / 2, HE = (N + 1) / 2;
  static constexpr int LPE = pad2(HE), LPO = pad2(H), LR = pad2(N);
  static constexpr int PE = 0;              // prolongation: N even rows (the first child's nodes)
  static constexpr int PO = PE + N * LPE;   // N odd rows
  static constexpr int RE = PO + N * LPO;   // restriction: HE even rows (the last one the middle node's)
  static constexpr int RO = RE + HE * LR;   // H odd rows
  static constexpr int SIZE = RO + H * LR;
  static constexpr int FEXP = 2 * N * N + SIZE;  // word with the two exponents F (int2)
  static constexpr int WORDS = FEXP + 1;
};

struct TrArgs64
{
  double *coarse, *fine;
  const double *E;  // tables of the degree
  int ncc[3];
  int64_t n_coarse;
};

template<int DIM, int N>
struct TrCfg
{
  static constexpr int ND = DIM == 2 ? N * N : N * N * N;
  static constexpr int PX = DIM == 2 ? N : N * N;           // pencils of the coarse cell along x
  static constexpr int PL = DIM == 2 ? 2 * N : 4 * N * N;   // threads per cell: pencils of the last pass
  static constexpr int SA = (2 * N) | 1;                    // row length of the first array
  static constexpr int A = PX * SA, B = DIM == 3 ? 4 * N * N * N : 0;
  // cells per CTA: of those with up to 256 threads the ones that fill their warps best
  static constexpr int best()
  {
    int b = 1, fill = 0;
    for(int c = 1; c * PL <= 256; ++c)
    {
      const int w = (c * PL + 31) / 32, f = w < 4 ? 10 * w : c * PL * 1000 / (w * 32);
      if(f > fill)
      {
        b = c;
        fill = f;
      }
    }
    return b;
  }
  static constexpr int CPB = best(), THREADS = (CPB * PL + 31) / 32 * 32;
};

// 4 sum_j c_j x_j / 2^64 of a row of L coefficients (read as pairs), |sum| <= 2^57. The products of the low
// limbs, a quarter of the last bit each before the scaling by 4, are kept (without their low three bits, so
// that 16 of them fit): without them the restriction's error is 4.9e-16 of its results' mean square for
// k = 4 in 3D, FP64's own 3.6e-16
template<int L>
__device__ __forceinline__ int64_t dot4(const int2 *__restrict__ row, const int *xh, const int *xl)
{
  fx::Acc M(1u << 29), S, Q;
  const int4 *row4 = reinterpret_cast<const int4 *>(row);
#pragma unroll
  for(int j2 = 0; j2 < (L + 1) / 2; ++j2)
  {
    const int4 c = row4[j2];
    M.add(c.y, xl[2 * j2]);
    M.add(c.x, xh[2 * j2]);
    if(j2 == 0) S.start(c.y, xh[0]);
    else S.add(c.y, xh[2 * j2]);
    if(j2 == 0) Q.start(c.x, xl[0] >> 3);
    else Q.add(c.x, xl[2 * j2] >> 3);
    if(2 * j2 + 1 < L)
    {
      const int j = 2 * j2 + 1 < L ? 2 * j2 + 1 : 0;
      Q.add(c.z, xl[j] >> 3);
      M.add(c.w, xl[j]);
      M.add(c.z, xh[j]);
      S.add(c.w, xh[j]);
    }
  }
  return (S.value() << 2) + ((M.value() + (Q.value() >> 29)) >> 30);
}

// 2N results of both children from the N values get(m)
template<int N, typename Get, typename Put>
__device__ __forceinline__ void widen(const int2 *tab, const Get &get, const Put &put)
{
  using T = TrTab<N>;
  constexpr int H = T::H, HE = T::HE;
  int eh[HE], el[HE], oh[HE], ol[HE];
#pragma unroll
  for(int j = 0; j < H; ++j)
  {
    const int64_t a = get(j), b = get(N - 1 - j);
    fx::split(a + b, eh[j], el[j]);
    fx::split(a - b, oh[j], ol[j]);
  }
  if constexpr(N % 2 == 1) fx::split(get(H), eh[H], el[H]);
#pragma unroll
  for(int i = 0; i < N; ++i)
  {
    const int64_t e = dot4<HE>(tab + T::PE + i * T::LPE, eh, el), o = dot4<H>(tab + T::PO + i * T::LPO, oh, ol);
    put(i, e + o);
    put(2 * N - 1 - i, e - o);
  }
}

// N results from the 2N values get(m) of both children
template<int N, typename Get, typename Put>
__device__ __forceinline__ void narrow(const int2 *tab, const Get &get, const Put &put)
{
  using T = TrTab<N>;
  constexpr int H = T::H;
  int eh[N], el[N], oh[N], ol[N];
#pragma unroll
  for(int j = 0; j < N; ++j)
  {
    const int64_t a = get(j), b = get(2 * N - 1 - j);
    fx::split(a + b, eh[j], el[j]);
    fx::split(a - b, oh[j], ol[j]);
  }
#pragma unroll(N <= 5 ? H : 1)
  for(int i = 0; i < H; ++i)
  {
    const int64_t e = dot4<N>(tab + T::RE + i * T::LR, eh, el), o = dot4<N>(tab + T::RO + i * T::LR, oh, ol);
    put(i, e + o);
    put(N - 1 - i, e - o);
  }
  if constexpr(N % 2 == 1) put(H, dot4<N>(tab + T::RE + H * T::LR, eh, el));
}

// the same in FP64, rolled
template<int N, typename Get, typename Put>
__device__ __forceinline__ void widen_fp64(const double *E, const Get &get, const Put &put)
{
#pragma unroll 1
  for(int r = 0; r < 2 * N; ++r)
  {
    double v = 0.0;
#pragma unroll 1
    for(int m = 0; m < N; ++m) v = fma(E[r * N + m], get(m), v);
    put(r, v);
  }
}
template<int N, typename Get, typename Put>
__device__ __forceinline__ void narrow_fp64(const double *E, const Get &get, const Put &put)
{
#pragma unroll 1
  for(int i = 0; i < N; ++i)
  {
    double v = 0.0;
#pragma unroll 1
    for(int r = 0; r < 2 * N; ++r) v = fma(E[r * N + i], get(r), v);
    put(i, v);
  }
}

template<int DIM, int N, bool RESTRICT>
__global__ void __launch_bounds__(TrCfg<DIM, N>::THREADS) transfer64_kernel(TrArgs64 a)
{
  using C = TrCfg<DIM, N>;
  using T = TrTab<N>;
  constexpr int ND = C::ND, PL = C::PL, PX = C::PX, SA = C::SA, F2 = 2 * N, L2 = N * N;
  __shared__ __align__(16) int2 s_tab[T::SIZE];
  __shared__ int64_t s_a[C::CPB * C::A], s_b[C::CPB * C::B + 1];
  __shared__ unsigned s_hi[C::CPB], s_lo[C::CPB];
  const int tid = threadIdx.x, slot = tid / PL, p = tid % PL;
  const int64_t cell = (int64_t)blockIdx.x * C::CPB + slot;
  const bool active = slot < C::CPB && cell < a.n_coarse;
  const int2 *src_tab = reinterpret_cast<const int2 *>(a.E + 2 * N * N);
  const int2 fexp = src_tab[T::SIZE];
  for(int i = tid; i < T::SIZE; i += C::THREADS) s_tab[i] = src_tab[i];
  if(tid < C::CPB) s_hi[tid] = s_lo[tid] = 0;
  // this thread's pencil of the last direction: node (X, Y) of the widened layer, in child (bx, by)
  const int bxy = p / (DIM == 2 ? N : L2), x = p % N, y = DIM == 2 ? 0 : p / N % N;
  const int bx = bxy % 2, by = bxy / 2, X = bx * N + x, Y = by * N + y;
  const int cx = (int)(cell % a.ncc[0]), cy = (int)(cell / a.ncc[0] % a.ncc[1]);
  const int64_t cz = cell / ((int64_t)a.ncc[0] * a.ncc[1]), nf0 = 2 * (int64_t)a.ncc[0], nf1 = 2 * (int64_t)a.ncc[1];
  const int64_t child = DIM == 2 ? 2 * cx + bx + nf0 * (2 * cy) : 2 * cx + bx + nf0 * (2 * cy + by + nf1 * (2 * cz));
  double *fine = a.fine + child * ND + (DIM == 2 ? x : x + N * y);
  const int64_t above = (DIM == 2 ? nf0 : nf0 * nf1) * ND;  // the upper child
  double *coarse = a.coarse + cell * ND;
  int64_t *A = s_a + (slot < C::CPB ? slot : 0) * C::A, *B = s_b + (slot < C::CPB ? slot : 0) * C::B;
  double *Ad = reinterpret_cast<double *>(A), *Bd = reinterpret_cast<double *>(B);
  auto fine_at = [&](int r) -> double & { return fine[(r >= N ? above : 0) + (r >= N ? r - N : r) * (DIM == 2 ? N : L2)]; };
  __syncthreads();
  // the values of this thread's first pass and the cell's largest exponent
  constexpr int NV = RESTRICT ? 2 * N : N;
  const bool first = active && (RESTRICT || p < PX);
  double v[NV], f[RESTRICT ? 1 : 2 * N];  // f: what the prolongation adds to, on its way during the passes
  unsigned hi = 0, lo = 0;
  if constexpr(!RESTRICT)
    if(active)
    {
#pragma unroll
      for(int r = 0; r < 2 * N; ++r) f[r] = fine_at(r);
    }
  if(first)
  {
#pragma unroll
    for(int i = 0; i < NV; ++i)
    {
      v[i] = RESTRICT ? fine_at(i) : coarse[p * N + i];
      hi = max(hi, (unsigned)__double2hiint(v[i]) & 0x7fffffffu);
      lo |= (unsigned)__double2loint(v[i]);
    }
    atomicMax(s_hi + slot, hi);
    if(lo) atomicOr(s_lo + slot, lo);
  }
  __syncthreads();
  if(active)
  {
    hi = s_hi[slot];
    lo = s_lo[slot];
  }
  const int ex = (int)(hi >> 20);
  const bool slow = active && (ex < 1023 - 300 || ex > 1023 + 300) && (hi | lo) != 0;
  const int emax = hi == 0 ? 1023 : ex;
  auto value = [&](int i) { return fx::from_double(v[i], emax); };
  const int unit = emax - 1023 - 58 + DIM * (62 - (RESTRICT ? fexp.y : fexp.x));  // exponent of the results
  // pencil q along y (3D: of the arrays between the x and the z pass)
  auto ay = [&](int q, int j) { return (q / F2 * N + j) * SA + q % F2; };
  auto by_ = [&](int q, int j) { return (q / F2 * F2 + j) * F2 + q % F2; };
  if constexpr(!RESTRICT)
  {
    if(first)
    {
      if(!slow) widen<N>(s_tab, value, [&](int r, int64_t w) { A[p * SA + r] = w; });
      else widen_fp64<N>(a.E, [&](int i) { return coarse[p * N + i]; }, [&](int r, double w) { Ad[p * SA + r] = w; });
    }
    __syncthreads();
    if constexpr(DIM == 3)
    {
      if(active && p < F2 * N)
      {
        if(!slow) widen<N>(s_tab, [&](int j) { return A[ay(p, j)]; }, [&](int r, int64_t w) { B[by_(p, r)] = w; });
        else widen_fp64<N>(a.E, [&](int j) { return Ad[ay(p, j)]; }, [&](int r, double w) { Bd[by_(p, r)] = w; });
      }
      __syncthreads();
    }
    if(active)
    {
      // pencil along the last direction
      auto in = [&](int j) { return DIM == 2 ? j * SA + X : (j * F2 + Y) * F2 + X; };
      if(!slow)
        widen<N>(s_tab, [&](int j) { return (DIM == 2 ? A : B)[in(j)]; },
                 [&](int r, int64_t w) { fine_at(r) = f[r] + fx::to_double_alu(w, unit); });
      else
        widen_fp64<N>(a.E, [&](int j) { return (DIM == 2 ? Ad : Bd)[in(j)]; }, [&](int r, double w) { fine_at(r) += w; });
    }
  }
  else
  {
    if(active)
    {
      auto out = [&](int j) { return DIM == 2 ? j * SA + X : (j * F2 + Y) * F2 + X; };
      if(!slow) narrow<N>(s_tab, value, [&](int j, int64_t w) { (DIM == 2 ? A : B)[out(j)] = w; });
      else
        narrow_fp64<N>(a.E, [&](int r) { return fine_at(r); }, [&](int j, double w) { (DIM == 2 ? Ad : Bd)[out(j)] = w; });
    }
    __syncthreads();
    if constexpr(DIM == 3)
    {
      if(active && p < F2 * N)
      {
        if(!slow) narrow<N>(s_tab, [&](int r) { return B[by_(p, r)]; }, [&](int j, int64_t w) { A[ay(p, j)] = w; });
        else narrow_fp64<N>(a.E, [&](int r) { return Bd[by_(p, r)]; }, [&](int j, double w) { Ad[ay(p, j)] = w; });
      }
      __syncthreads();
    }
    if(active && p < PX)
    {
      if(!slow)
        narrow<N>(s_tab, [&](int r) { return A[p * SA + r]; },
                  [&](int i, int64_t w) { coarse[p * N + i] += fx::to_double(w, unit); });
      else
        narrow_fp64<N>(a.E, [&](int r) { return Ad[p * SA + r]; }, [&](int i, double w) { coarse[p * N + i] += w; });
    }
  }
}
}  // namespace tr64
}  // namespace tpss
