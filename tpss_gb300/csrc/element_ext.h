// element_ext.h -- 1-D reference element in extended precision, for the kernels that contract with
// integers (fixed64.cuh): their tables hold 62 bits, and the rounding of the FP64 basis (some 1e-15 of an
// entry for high degrees) would be their largest error.
#pragma once

#include <cmath>

#include "internal.h"

namespace tpss
{
namespace ext
{
using Real = long double;

// P_m and its derivative at z in (-1, 1)
inline void legendre(int m, Real z, Real &p, Real &dp)
{
  Real p0 = 1, p1 = z;
  for(int j = 2; j <= m; ++j)
  {
    const Real p2 = ((2 * j - 1) * z * p1 - (j - 1) * p0) / j;
    p0 = p1;
    p1 = p2;
  }
  p = p1;
  dp = m * (z * p1 - p0) / (z * z - 1);
}

template<int N>
struct Element
{
  Real x[N];                     // support points
  Real mass[N][N], stiff[N][N];  // on [0, 1]
  Real g[N];                     // derivatives at the upper end (those at the lower end mirror them)

  // basis and derivatives at a point
  void lagrange(Real at, Real (&v)[N], Real (&d)[N]) const
  {
    for(int i = 0; i < N; ++i)
    {
      v[i] = 1;
      d[i] = 0;
      for(int j = 0; j < N; ++j)
      {
        if(j == i) continue;
        d[i] = (d[i] * (at - x[j]) + v[i]) / (x[i] - x[j]);
        v[i] *= (at - x[j]) / (x[i] - x[j]);
      }
    }
  }

  // the FP64 points, one Newton step each (quadratic: twice as many digits)
  explicit Element(const Shape1D &s)
  {
    Real qx[N], qw[N];
    x[0] = 0;
    x[N - 1] = 1;
    for(int i = 0; i < N; ++i)
    {
      Real z = 2 * (Real)s.qx[i] - 1, p, dp;
      legendre(N, z, p, dp);
      z -= p / dp;
      legendre(N, z, p, dp);
      qx[i] = (1 + z) / 2;
      qw[i] = 1 / ((1 - z * z) * dp * dp);
      if(i == 0 || i == N - 1) continue;
      z = 2 * (Real)s.nodes[i] - 1;
      legendre(N - 1, z, p, dp);
      z -= dp * (1 - z * z) / (2 * z * dp - (Real)(N - 1) * N * p);
      x[i] = (1 + z) / 2;
    }
    Real v[N], d[N];
    for(int i = 0; i < N; ++i)
      for(int j = 0; j < N; ++j) mass[i][j] = stiff[i][j] = 0;
    for(int q = 0; q < N; ++q)
    {
      lagrange(qx[q], v, d);
      for(int i = 0; i < N; ++i)
        for(int j = 0; j < N; ++j)
        {
          mass[i][j] += v[i] * v[j] * qw[q];
          stiff[i][j] += d[i] * d[j] * qw[q];
        }
    }
    lagrange(1, v, g);
  }
};

// c 2^f as limbs of the integer kernels' rows (low word first)
inline int64_t limbs(Real c, int f)
{
  const int64_t v = std::llrint(std::ldexp(c, f));
  const int32_t lo = (int32_t)(uint32_t)(uint64_t)v;
  const int32_t hi = (int32_t)((v - lo) >> 32);
  return (int64_t)((uint64_t)(uint32_t)hi << 32 | (uint32_t)lo);
}
}  // namespace ext
}  // namespace tpss
