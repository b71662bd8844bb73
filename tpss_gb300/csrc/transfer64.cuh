// transfer64.cuh -- FP64 transfer between a coarse cell and its 2^dim children on the integer pipe.
//
// Embedding into both children along a direction is one mirror-symmetric 2N x N matrix, so a pencil takes
// N^2 products in even/odd form for all 2N results (and back). Prolongation widens the coarse cell
// along x, y and z in turn (N^(d-1), 2 N^(d-1), 4 N^(d-1) pencils), restriction goes the other way. The
// fine vector is read and written by the threads of the z (2D: y) pass, which hold a pencil of both children
// each; their order runs through a child's layer, so that they read and write whole rows.
//
// Every pencil has a unit of its own, and between the passes the cell lives in shared memory in FP64. A fine
// node that is a coarse one (the ends, and the middle for odd N) takes its value as it is in FP64, in both
// directions: its row of the matrix has a single entry, and the others do not see it. The
// remaining rows have no zeros, so that what sets a pencil's unit enters all of its results: one pass's rounding
// is 2^-58 of the pencil's largest value, and small values next to large ones keep their digits.
// Values the integers do not cover (infinities, NaN, magnitudes outside 2^(+-800)) take FP64 passes, pencil by
// pencil.
//
// Measured, 16^3 coarse cells, k = 4 (4.1M fine values): prolongation 25 us, restriction 25.5 us, where the tree
// of FP64 passes per child took 90 and 92 us (FP64 pipe). The fine values move in 10 and 5 us at the copy
// rate; the rest is the serial chain of three passes, hidden behind the other CTAs of the SM only in
// part. 2^3 coarse cells take 5 us each way instead of 25 and 27. (One unit per cell, with the cell in
// integers between the passes, took 25 and 26.5 us and lost a small value's digits next to a large one anywhere in
// the cell.) Fetching the fine values that the prolongation adds to
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
  static constexpr int H = N / 2, HE = (N + 1) / 2, ODD = N % 2;
  static constexpr int ROWS = N - 1 - ODD;         // the first child's nodes 1 .. ROWS that are no coarse nodes
  static constexpr int LPE = pad2(HE), LPO = pad2(H), LR = pad2(ROWS);
  static constexpr int PE = 0;                     // prolongation: ROWS even rows
  static constexpr int PO = PE + ROWS * LPE;       // ROWS odd rows
  static constexpr int RE = PO + ROWS * LPO;       // restriction: HE even rows (the last one the middle node's)
  static constexpr int RO = RE + HE * LR;          // H odd rows
  static constexpr int SIZE = RO + H * LR;
  static constexpr int FEXP = 2 * N * N + SIZE;    // word with the two exponents F (int2)
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

// exponent of a pencil (1023: all zeros), -1: the integers do not cover it
__device__ __forceinline__ int exponent(unsigned hi, unsigned lo)
{
  const int e = (int)(hi >> 20);
  return (hi | lo) == 0 ? 1023 : e < 1023 - fx::kRange || e > 1023 + fx::kRange ? -1 : e;
}
__device__ __forceinline__ void magnitude(double v, unsigned &hi, unsigned &lo)
{
  hi = max(hi, (unsigned)__double2hiint(v) & 0x7fffffffu);
  lo |= (unsigned)__double2loint(v);
}

// 2N results of both children, put(r, value), from a pencil's N values; E: FP64 rows. put_at is put for an r
// that is not a constant
template<int N, typename Put, typename PutAt>
__device__ __forceinline__ void widen(const int2 *tab, const double *E, int F, const double (&v)[N], const Put &put,
                                      const PutAt &put_at)
{
  using T = TrTab<N>;
  constexpr int H = T::H, HE = T::HE, ROWS = T::ROWS;
  put(0, v[0]);
  put(2 * N - 1, v[N - 1]);
  if constexpr(T::ODD)
  {
    put(N - 1, v[H]);
    put(N, v[H]);
  }
  if constexpr(N == 2)
  {
    // one value at the middle of both: exactly rounded in FP64, and no more work
    const double s = fma(0.5, v[1], 0.5 * v[0]);
    put(1, s);
    put(2, s);
    return;
  }
  unsigned hi = 0, lo = 0;
#pragma unroll
  for(int i = 0; i < N; ++i) magnitude(v[i], hi, lo);
  const int e = exponent(hi, lo);
  if(e < 0)
  {
    double w[N];  // (a copy, so that v stays in registers)
#pragma unroll
    for(int i = 0; i < N; ++i) w[i] = v[i];
#pragma unroll 1
    for(int r = 1; r < 2 * N - 1; ++r)
    {
      if(T::ODD && (r == N - 1 || r == N)) continue;
      double s = 0.0;
#pragma unroll 1
      for(int m = 0; m < N; ++m) s = fma(E[r * N + m], w[m], s);
      put_at(r, s);
    }
    return;
  }
  int eh[HE], el[HE], oh[HE], ol[HE];
#pragma unroll
  for(int j = 0; j < H; ++j)
  {
    const int64_t a = fx::from_double(v[j], e), b = fx::from_double(v[N - 1 - j], e);
    fx::split(a + b, eh[j], el[j]);
    fx::split(a - b, oh[j], ol[j]);
  }
  if constexpr(T::ODD) fx::split(fx::from_double(v[H], e), eh[H], el[H]);
  const int unit = e - 1023 - 58 + 62 - F;
#pragma unroll
  for(int i = 0; i < ROWS; ++i)
  {
    const int64_t s = dot4<HE>(tab + T::PE + i * T::LPE, eh, el), o = dot4<H>(tab + T::PO + i * T::LPO, oh, ol);
    put(1 + i, fx::to_double_alu(s + o, unit));
    put(2 * N - 2 - i, fx::to_double_alu(s - o, unit));
  }
}

// N results, put(m, value), from the 2N values of both children
template<int N, typename Put>
__device__ __forceinline__ void narrow(const int2 *tab, const double *E, int F, const double (&v)[2 * N], const Put &put)
{
  using T = TrTab<N>;
  constexpr int H = T::H, ROWS = T::ROWS;
  if constexpr(N == 2)
  {
    const double s = fma(0.5, v[2], 0.5 * v[1]);
    put(0, v[0] + s);
    put(1, v[3] + s);
    return;
  }
  unsigned hi = 0, lo = 0;
#pragma unroll
  for(int j = 1; j <= ROWS; ++j)
  {
    magnitude(v[j], hi, lo);
    magnitude(v[2 * N - 1 - j], hi, lo);
  }
  const int e = exponent(hi, lo);
  if(e < 0)
  {
    double w[2 * N];
#pragma unroll
    for(int r = 0; r < 2 * N; ++r) w[r] = v[r];
#pragma unroll 1
    for(int i = 0; i < N; ++i)
    {
      double s = 0.0;
#pragma unroll 1
      for(int r = 0; r < 2 * N; ++r) s = fma(E[r * N + i], w[r], s);
      put(i, s);
    }
    return;
  }
  int eh[ROWS + 1], el[ROWS + 1], oh[ROWS + 1], ol[ROWS + 1];
#pragma unroll
  for(int j = 0; j < ROWS; ++j)
  {
    const int64_t a = fx::from_double(v[1 + j], e), b = fx::from_double(v[2 * N - 2 - j], e);
    fx::split(a + b, eh[j], el[j]);
    fx::split(a - b, oh[j], ol[j]);
  }
  const int unit = e - 1023 - 58 + 62 - F;
#pragma unroll
  for(int i = 0; i < H; ++i)
  {
    const int64_t s = dot4<ROWS>(tab + T::RE + i * T::LR, eh, el), o = dot4<ROWS>(tab + T::RO + i * T::LR, oh, ol);
    const double lower = fx::to_double_alu(s + o, unit), upper = fx::to_double_alu(s - o, unit);
    put(i, i == 0 ? v[0] + lower : lower);
    put(N - 1 - i, i == 0 ? v[2 * N - 1] + upper : upper);
  }
  if constexpr(T::ODD)
    put(H, v[N - 1] + v[N] + fx::to_double_alu(dot4<ROWS>(tab + T::RE + H * T::LR, eh, el), unit));
}

template<int DIM, int N, bool RESTRICT>
__global__ void __launch_bounds__(TrCfg<DIM, N>::THREADS) transfer64_kernel(TrArgs64 a)
{
  using C = TrCfg<DIM, N>;
  using T = TrTab<N>;
  constexpr int ND = C::ND, PL = C::PL, PX = C::PX, SA = C::SA, F2 = 2 * N, L2 = N * N;
  __shared__ __align__(16) int2 s_tab[T::SIZE];
  __shared__ double s_a[C::CPB * C::A], s_b[C::CPB * C::B + 1];
  const int tid = threadIdx.x, slot = tid / PL, p = tid % PL;
  const int64_t cell = (int64_t)blockIdx.x * C::CPB + slot;
  const bool active = slot < C::CPB && cell < a.n_coarse;
  const int2 *src_tab = reinterpret_cast<const int2 *>(a.E + 2 * N * N);
  const int2 fexp = src_tab[T::SIZE];
  const int F = RESTRICT ? fexp.y : fexp.x;
  for(int i = tid; i < T::SIZE; i += C::THREADS) s_tab[i] = src_tab[i];
  // this thread's pencil of the last direction: node (X, Y) of the widened layer, in child (bx, by)
  const int bxy = p / (DIM == 2 ? N : L2), x = p % N, y = DIM == 2 ? 0 : p / N % N;
  const int bx = bxy % 2, by = bxy / 2, X = bx * N + x, Y = by * N + y;
  const int cx = (int)(cell % a.ncc[0]), cy = (int)(cell / a.ncc[0] % a.ncc[1]);
  const int64_t cz = cell / ((int64_t)a.ncc[0] * a.ncc[1]), nf0 = 2 * (int64_t)a.ncc[0], nf1 = 2 * (int64_t)a.ncc[1];
  const int64_t child = DIM == 2 ? 2 * cx + bx + nf0 * (2 * cy) : 2 * cx + bx + nf0 * (2 * cy + by + nf1 * (2 * cz));
  double *fine = a.fine + child * ND + (DIM == 2 ? x : x + N * y);
  const int64_t above = (DIM == 2 ? nf0 : nf0 * nf1) * ND;  // the upper child
  double *coarse = a.coarse + cell * ND;
  double *A = s_a + (slot < C::CPB ? slot : 0) * C::A, *B = s_b + (slot < C::CPB ? slot : 0) * C::B;
  auto fine_at = [&](int r) -> double & { return fine[(r >= N ? above : 0) + (r >= N ? r - N : r) * (DIM == 2 ? N : L2)]; };
  // pencil q along y (3D: of the arrays between the x and the z pass)
  auto ay = [&](int q, int j) { return (q / F2 * N + j) * SA + q % F2; };
  auto by_ = [&](int q, int j) { return (q / F2 * F2 + j) * F2 + q % F2; };
  // pencil along the last direction
  auto last = [&](int j) { return DIM == 2 ? j * SA + X : (j * F2 + Y) * F2 + X; };
  __syncthreads();
  if constexpr(!RESTRICT)
  {
    double f[2 * N], v[N];  // f: what the prolongation adds to, on its way during the passes
    if(active)
    {
#pragma unroll
      for(int r = 0; r < 2 * N; ++r) f[r] = fine_at(r);
    }
    if(active && p < PX)
    {
#pragma unroll
      for(int i = 0; i < N; ++i) v[i] = coarse[p * N + i];
      auto put = [&](int r, double w) { A[p * SA + r] = w; };
      widen<N>(s_tab, a.E, F, v, put, put);
    }
    __syncthreads();
    if constexpr(DIM == 3)
    {
      if(active && p < F2 * N)
      {
#pragma unroll
        for(int j = 0; j < N; ++j) v[j] = A[ay(p, j)];
        auto put = [&](int r, double w) { B[by_(p, r)] = w; };
        widen<N>(s_tab, a.E, F, v, put, put);
      }
      __syncthreads();
    }
    if(active)
    {
#pragma unroll
      for(int j = 0; j < N; ++j) v[j] = (DIM == 2 ? A : B)[last(j)];
      widen<N>(s_tab, a.E, F, v, [&](int r, double w) { fine_at(r) = f[r] + w; },
               [&](int r, double w) { fine_at(r) += w; });
    }
  }
  else
  {
    double v[2 * N];
    if(active)
    {
#pragma unroll
      for(int r = 0; r < 2 * N; ++r) v[r] = fine_at(r);
      narrow<N>(s_tab, a.E, F, v, [&](int j, double w) { (DIM == 2 ? A : B)[last(j)] = w; });
    }
    __syncthreads();
    if constexpr(DIM == 3)
    {
      if(active && p < F2 * N)
      {
#pragma unroll
        for(int r = 0; r < 2 * N; ++r) v[r] = B[by_(p, r)];
        narrow<N>(s_tab, a.E, F, v, [&](int j, double w) { A[ay(p, j)] = w; });
      }
      __syncthreads();
    }
    if(active && p < PX)
    {
#pragma unroll
      for(int r = 0; r < 2 * N; ++r) v[r] = A[p * SA + r];
      narrow<N>(s_tab, a.E, F, v, [&](int i, double w) { coarse[p * N + i] += w; });
    }
  }
}
}  // namespace tr64
}  // namespace tpss
