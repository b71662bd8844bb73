// sipg_lines.cuh -- FP64 SIPG operator on a Cartesian level, line by line on the integer pipe.
//
// The same Kronecker sum as sipg_kernel (operator.cu), A = sum_d M x .. x A_d x .. x M, as one pass per
// direction over the whole level:
//   x:        t0 = A_x u,            t1 = M_x u
//   y (3D):   s  = M_y t0 + A_y t1,  m  = M_y t1
//   last:     dst = M s + A m        (2D: M_y t0 + A_y t1), or rhs minus that
// with t0, t1, s, m on the level's lexicographic node grid (x fastest), so that the passes along y and
// z read and write coalesced with one thread per line, which marches along it cell by cell.
//
// The 1-D SIPG matrix of a cell splits into a block that is mirror symmetric (its own stiffness and face
// terms with the penalty of a face between two cells of this width) and couplings to its two
// neighbours that need of a neighbour its face value u+ and one trace t+ = b . u+:
//   y = C u + De (uR + uL) +- Do (uR - uL) at the mirrored pairs of nodes, y[0] += tL, y[n-1] += tR.
// Every cell's traces serve both neighbours. Boundary faces are neighbours with u+ = -u and
// t+ = (sigma_b - 2 sigma) u - t; unequal widths shift t+ by the difference of the penalties.
// All contractions run in even/odd form with integers, one exponent per pencil (fixed64.cuh).
//
// Measured, 64^3 cells, k = 4 (32.8M DoFs): 940 us (x 382, y 303, last 252) against sipg_kernel's
// 3,168 us, whose FP64 pipe is busy throughout. The vectors in between cost 2.4 GB of traffic in all
// (0.36 ms at the copy rate), which the cell-wise kernel does not have; issue slots (56 % busy) and the
// 32-bit multiplier (46 to 55 %) bound the passes. Of the conversions back to FP64 the results' use the
// FP64 pipe's instruction and M q's and the traces' integer ones: all on the FP64 pipe takes 993 us.
#pragma once

#include "fixed64.cuh"

namespace tpss
{
namespace lines
{
// Table of one cell width, in 8-byte words: rows padded to an even length
template<int N>
struct OpTab
{
  static constexpr int H = N / 2, ODD = N % 2, HE = H + ODD;  // even parts: pairs and the middle node
  static constexpr int pad2(int x) { return (x + 1) / 2 * 2; }
  static constexpr int LME = pad2(HE), LMO = pad2(H), LCE = pad2(HE + 1), LCO = pad2(H + 1);
  static constexpr int ME = 0;                 // mass: HE even rows (the last one the middle node's)
  static constexpr int MO = ME + HE * LME;     // H odd rows
  static constexpr int CE = MO + H * LMO;      // own block, then De
  static constexpr int CO = CE + HE * LCE;     // own block, then Do
  static constexpr int TE = CO + H * LCO;      // trace: even and odd part
  static constexpr int TO = TE + LME;
  static constexpr int SIZE = TO + LMO;
};

struct OpLineArgs
{
  const double *p, *q;        // first and second input (x pass: q in cell blocks)
  double *r, *m;              // results M p + A q and M q (or nullptr)
  const double *rhs;          // last pass: dst = rhs - result
  const int64_t *cell_start;  // nullptr: lexicographic cells
  const int2 *tab;            // integer tables, one per distinct width
  const double *tab64;        // the same in FP64
  const int *exps;            // per width: F of M, C and the trace
  const int32_t *width;       // per cell of this direction: index of its width's tables, and kSpecial
  const double *sig;          // per cell: sigma of its lower face, of its upper face, its own (block)
  int nc[3];                  // cells per direction
  int64_t ncol, inner, outer, stride;  // line c starts at (c / inner) * outer + c % inner
  int seg;                    // cells per segment
};

// marks a cell with a face at the boundary or to a cell of another width: only these need the
// penalties in FP64. Kept behind one branch, since the compiler otherwise predicates the corrections and
// runs them for every cell (27 FP64 instructions per pencil instead of 7; the y pass of the level above
// took 376 us so, and 289 without)
constexpr int32_t kSpecial = 1 << 30;

__device__ __forceinline__ double negated(double v)
{
  return __hiloint2double(__double2hiint(v) ^ (int)0x80000000u, __double2loint(v));
}

__device__ __forceinline__ bool out_of_range(unsigned hm, unsigned lo)
{
  const int e = (int)(hm >> 20);
  return (e < 1023 - fx::kRange || e > 1023 + fx::kRange) && (hm | lo) != 0;
}

template<int CNT>
__device__ __forceinline__ void magnitude(const double (&v)[CNT], unsigned &hm, unsigned &lo)
{
#pragma unroll
  for(int i = 0; i < CNT; ++i)
  {
    hm = max(hm, (unsigned)__double2hiint(v[i]) & 0x7fffffffu);
    lo |= (unsigned)__double2loint(v[i]);
  }
}

// even and odd parts of a pencil in limbs: eh/el[0 .. HE) (pair sums, then the middle node), oh/ol
template<int N, int LE, int LO>
__device__ __forceinline__ void split_parts(const double (&u)[N], int emax, int (&eh)[LE], int (&el)[LE], int (&oh)[LO],
                                            int (&ol)[LO])
{
  constexpr int H = N / 2;
#pragma unroll
  for(int j = 0; j < H; ++j)
  {
    const int64_t a = fx::from_double(u[j], emax), b = fx::from_double(u[N - 1 - j], emax);
    fx::split(a + b, eh[j], el[j]);
    fx::split(a - b, oh[j], ol[j]);
  }
  if constexpr(N % 2 == 1) fx::split(fx::from_double(u[H], emax), eh[H], el[H]);
}

// One pencil of a cell. In: q (and p) of the cell, the neighbours' face values uL, uR. Out: r without
// the neighbours' traces, m, and the cell's traces towards its lower (tl) and upper (tu) neighbour.
// PARTS: 0 traces only, 1 everything.
// The unit of q's integers is that of q alone: a larger value in a neighbour neither costs the traces and m,
// which do not depend on it, any bits, nor makes them differ between a cell and its copy at the end of a tile
// or segment. A face value more than two binades above q enters r in FP64 instead; it is rare and read once more
// there (again: sets uL, uR), since the registers that would keep it cost 15 % of the passes' time (64^3 cells, k = 4:
// 1,106 us; 940 so; 903 with one unit for q and the face values).
template<int N, bool HAS_P, bool WANT_M, int PARTS, typename Again>
__device__ __forceinline__ void cell_pencil(const int2 *__restrict__ tab, const double *__restrict__ tab64, int FM, int FC,
                                            int FT, const double (&p)[N], const double (&q)[N], double uL, double uR,
                                            double (&r)[N], double (&m)[N], double &tl, double &tu, const Again &again)
{
  using T = OpTab<N>;
  constexpr int H = T::H, HE = T::HE;
  unsigned hq = 0, lq = 0, hn = 0, ln = 0, hp = 0, lp = 0;
  magnitude<N>(q, hq, lq);
  if constexpr(PARTS)
  {
    const double nb[2] = {uL, uR};
    magnitude<2>(nb, hn, ln);
    if constexpr(HAS_P) magnitude<N>(p, hp, lp);
  }
  if(out_of_range(hq, lq) || (PARTS && (out_of_range(hn, ln) || (HAS_P && out_of_range(hp, lp)))))
  {
    // FP64, rolled (on copies, so that the values above stay in registers)
    double u[N], v[N], rr[N], mm[N];
#pragma unroll
    for(int i = 0; i < N; ++i)
    {
      u[i] = q[i];
      v[i] = HAS_P ? p[i] : 0.0;
      rr[i] = mm[i] = 0.0;
    }
    double t0 = 0.0, t1 = 0.0;
#pragma unroll 1
    for(int i = 0; i < HE; ++i)
    {
      // pair (i, N - 1 - i), or the middle node
      const bool mid = 2 * i == N - 1;
      const double *ce = tab64 + T::CE + i * T::LCE, *me = tab64 + T::ME + i * T::LME;
      const double *cd = tab64 + T::CO + i * T::LCO, *md = tab64 + T::MO + i * T::LMO;
      double re = PARTS ? ce[HE] * (uR + uL) : 0.0, xe = 0.0, ro = PARTS && !mid ? cd[H] * (uR - uL) : 0.0, xo = 0.0;
#pragma unroll 1
      for(int j = 0; j < HE; ++j)
      {
        const bool mj = 2 * j == N - 1;
        const double e = mj ? u[j] : u[j] + u[N - 1 - j], o = mj ? 0.0 : u[j] - u[N - 1 - j];
        const double f = mj ? v[j] : v[j] + v[N - 1 - j], h = mj ? 0.0 : v[j] - v[N - 1 - j];
        if(i == 0)
        {
          t0 = fma(tab64[T::TE + j], e, t0);
          if(!mj) t1 = fma(tab64[T::TO + j], o, t1);
        }
        re = fma(ce[j], e, re);
        xe = fma(me[j], e, xe);
        if(HAS_P) re = fma(me[j], f, re);
        if(!mid && !mj)
        {
          ro = fma(cd[j], o, ro);
          xo = fma(md[j], o, xo);
          if(HAS_P) ro = fma(md[j], h, ro);
        }
      }
      rr[i] = re + ro;
      mm[i] = xe + xo;
      if(!mid)
      {
        rr[N - 1 - i] = re - ro;
        mm[N - 1 - i] = xe - xo;
      }
    }
    tu = t0 + t1;
    tl = t0 - t1;
#pragma unroll
    for(int i = 0; i < N; ++i)
    {
      r[i] = rr[i];
      m[i] = mm[i];
    }
    return;
  }
  // (a zero pencil takes the unit of its neighbours)
  const int en = (int)(hn >> 20), eq = hq != 0 ? (int)(hq >> 20) : hn != 0 ? en : 1023, ep = hp == 0 ? 1023 : (int)(hp >> 20);
  // limbs of the even parts and s, and of the odd parts and d
  int eh[HE + 1], el[HE + 1], oh[H + 1], ol[H + 1];
  split_parts<N>(q, eq, eh, el, oh, ol);
  const int uq = eq - 1023 - 58 + 64;
  {
    const int64_t te = fx::row_dot<HE>(tab + T::TE, eh, el), to = fx::row_dot<H>(tab + T::TO, oh, ol);
    tu = fx::to_double_alu(te + to, uq - FT);
    tl = fx::to_double_alu(te - to, uq - FT);
  }
  if constexpr(PARTS)
  {
    // up to two binades above q the one product that a row has with them stays within the accumulators
    const bool far = en > eq + 2;
    {
      const int64_t lo = far ? 0 : fx::from_double(uL, eq + 2) << 2, hi = far ? 0 : fx::from_double(uR, eq + 2) << 2;
      fx::split(hi + lo, eh[HE], el[HE]);
      fx::split(hi - lo, oh[H], ol[H]);
    }
    int ph[HE + 1], pl[HE + 1], sh[H + 1], sl[H + 1];
    if constexpr(HAS_P) split_parts<N>(p, ep, ph, pl, sh, sl);
    // the two contributions to r come to the coarser of their units (a zero one has none)
    const int u2 = ep - 1023 - 58 + 64 - FM, u1 = HAS_P && (hq | hn) == 0 ? u2 : uq - FC;
    const int U = HAS_P && hp != 0 ? max(u1, u2) : u1;
    auto even = [&](int i) {
      const int64_t a = fx::row_dot<HE + 1>(tab + T::CE + i * T::LCE, eh, el);
      if constexpr(HAS_P)
        return fx::shr_s(a, U - u1) + fx::shr_s(fx::row_dot<HE>(tab + T::ME + i * T::LME, ph, pl), max(U - u2, 0));
      else
        return a;
    };
    auto odd = [&](int i) {
      const int64_t a = fx::row_dot<H + 1>(tab + T::CO + i * T::LCO, oh, ol);
      if constexpr(HAS_P)
        return fx::shr_s(a, U - u1) + fx::shr_s(fx::row_dot<H>(tab + T::MO + i * T::LMO, sh, sl), max(U - u2, 0));
      else
        return a;
    };
#pragma unroll
    for(int i = 0; i < H; ++i)
    {
      const int64_t e = even(i), o = odd(i);
      r[i] = fx::to_double(e + o, U);
      r[N - 1 - i] = fx::to_double(e - o, U);
    }
    if constexpr(N % 2 == 1) r[H] = fx::to_double(even(H), U);
    if(far)
    {
      again(uL, uR);
      const double s = uR + uL, d = uR - uL;
#pragma unroll
      for(int i = 0; i < HE; ++i)
      {
        const double e = tab64[T::CE + i * T::LCE + HE] * s, o = i < H ? tab64[T::CO + i * T::LCO + H] * d : 0.0;
        r[i] += e + o;
        if(i < H) r[N - 1 - i] += e - o;
      }
    }
    if constexpr(WANT_M)
    {
#pragma unroll
      for(int i = 0; i < HE; ++i)
      {
        const int64_t e = fx::row_dot<HE>(tab + T::ME + i * T::LME, eh, el);
        const int64_t o = i < H ? fx::row_dot<H>(tab + T::MO + i * T::LMO, oh, ol) : 0;
        m[i] = fx::to_double_alu(e + o, uq - FM);
        if(i < H) m[N - 1 - i] = fx::to_double_alu(e - o, uq - FM);
      }
    }
  }
}

// Boundary faces and faces to a cell of another width: the cell's results and traces carry the penalty
// sg[2] of a face between two cells of its width; the lower face has sg[0], the upper one sg[1]
template<int N>
__device__ __forceinline__ void special_faces(const double *sg, bool below, bool above, bool own, double u0, double u1,
                                              double &r0, double &r1, double &tl, double &tu)
{
  const double s_lo = sg[0], s_hi = sg[1], s_own = sg[2];
  if(own)
  {
    r0 += below ? (s_lo - s_own) * u0 : fma(s_lo - 2.0 * s_own, u0, -tl);
    r1 += above ? (s_hi - s_own) * u1 : fma(s_hi - 2.0 * s_own, u1, -tu);
  }
  if(below) tl = fma(s_own - s_lo, u0, tl);
  if(above) tu = fma(s_own - s_hi, u1, tu);
}

// ---- y and last pass: one thread per line and segment
constexpr int kOpThreads = 128;
constexpr int kMaxGridY = 65535;  // a grid's second dimension (a longer line gets longer segments)

enum OpLineMode
{
  OP_INNER,     // y pass: r and m on the node grid
  OP_LAST,      // last pass: dst in cell blocks
  OP_RESIDUAL,  // the same, dst = rhs - result
};

// registers per thread: what the passes need without the rare branch of cell_pencil (the compiler, left alone, takes up to 20
// more for it, and an SM holds a block or two fewer)
constexpr int line_regs(int n, bool last)
{
  constexpr int to[9] = {0, 0, 56, 72, 64, 80, 88, 104, 112}, in[9] = {0, 0, 64, 72, 64, 96, 112, 128, 128};
  return last ? to[n] : in[n];
}

template<int DIM, int N, int MODE>
__global__ void __maxnreg__((line_regs(N, MODE != OP_INNER))) op_line_kernel(OpLineArgs a)
{
  using T = OpTab<N>;
  constexpr bool LAST = MODE != OP_INNER;
  constexpr int D = LAST ? DIM - 1 : 1, CD = DIM == 2 ? N * N : N * N * N;
  __shared__ __align__(16) int2 s_tab[T::SIZE];
  const int tid = threadIdx.x;
  const int64_t c = (int64_t)blockIdx.x * kOpThreads + tid;
  const bool active = c < a.ncol;
  const int64_t cc = active ? c : 0, co = cc / a.inner, ci = cc - co * a.inner;
  const double *p = a.p + co * a.outer + ci, *q = a.q + co * a.outer + ci;
  double *ro = a.r + co * a.outer + ci, *mo = LAST ? nullptr : a.m + co * a.outer + ci;
  // last pass: the line's cell column and DoF within the cells' layers
  int64_t cell0 = 0;
  int dof0 = 0;
  if constexpr(LAST)
  {
    const int64_t gx_n = (int64_t)a.nc[0] * N;
    const int gy = DIM == 3 ? (int)(cc / gx_n) : 0, gx = (int)(cc - gy * gx_n);
    cell0 = gx / N + (int64_t)a.nc[0] * (gy / N);
    dof0 = gx % N + N * (gy % N);
  }
  const int n = a.nc[D], c0 = blockIdx.y * a.seg, c1 = min(n, c0 + a.seg);
  int w_now = -1, FM = 0, FC = 0, FT = 0;
  double face = 0.0, trace = 0.0;  // of the cell below: value and trace at the shared face
  double held = 0.0;               // last result of the cell below, waiting for this cell's trace
  for(int x = c0 > 0 ? c0 - 1 : c0; x <= (c1 < n ? c1 : n - 1); ++x)
  {
    const int wf = a.width[x], w = wf & ~kSpecial;
    if(w != w_now)
    {
      w_now = w;
      __syncthreads();
      for(int o = tid; o < T::SIZE; o += kOpThreads) s_tab[o] = a.tab[(size_t)w * T::SIZE + o];
      FM = a.exps[3 * w];
      FC = a.exps[3 * w + 1];
      FT = a.exps[3 * w + 2];
      __syncthreads();
    }
    if(!active) continue;
    const double *t64 = a.tab64 + (size_t)w * T::SIZE;
    double pv[N] = {}, qv[N], r[N], m[N], tl, tu;
    const int64_t at = (int64_t)x * N;
#pragma unroll
    for(int i = 0; i < N; ++i) qv[i] = q[(at + i) * a.stride];
    const bool own = x >= c0 && x < c1;
    if(own)
    {
#pragma unroll
      for(int i = 0; i < N; ++i) pv[i] = p[(at + i) * a.stride];
      const double uL = x > 0 ? face : negated(qv[0]), uR = x + 1 < n ? q[(at + N) * a.stride] : negated(qv[N - 1]);
      cell_pencil<N, true, !LAST, 1>(s_tab, t64, FM, FC, FT, pv, qv, uL, uR, r, m, tl, tu, [&](double &lo, double &hi) {
        const double *f = q + at * a.stride;
        lo = x > 0 ? f[-a.stride] : negated(f[0]);
        hi = x + 1 < n ? f[N * a.stride] : negated(f[(N - 1) * a.stride]);
      });
      if(x > 0) r[0] += trace;
    }
    else
      cell_pencil<N, true, !LAST, 0>(s_tab, t64, FM, FC, FT, pv, qv, 0.0, 0.0, r, m, tl, tu, [](double &, double &) {});
    if(wf & kSpecial) special_faces<N>(a.sig + 3 * x, x > 0, x + 1 < n, own, qv[0], qv[N - 1], r[0], r[N - 1], tl, tu);
    auto store = [&](int64_t cell, int i, double v) {
      if constexpr(LAST)
      {
        const int64_t id = cell0 + cell * (DIM == 2 ? (int64_t)a.nc[0] : (int64_t)a.nc[0] * a.nc[1]);
        const int64_t g = (a.cell_start ? a.cell_start[id] : id * CD) + dof0 + (int64_t)i * (DIM == 2 ? N : N * N);
        a.r[g] = MODE == OP_RESIDUAL ? a.rhs[g] - v : v;
      }
      else
        ro[(cell * N + i) * a.stride] = v;
    };
    if(x > c0) store(x - 1, N - 1, held + tl);  // the cell below is complete
    if(own)
    {
#pragma unroll
      for(int i = 0; i < N - 1; ++i) store(x, i, r[i]);
      if(x + 1 < n) held = r[N - 1];
      else store(x, N - 1, r[N - 1]);
      if constexpr(!LAST)
#pragma unroll
        for(int i = 0; i < N; ++i) mo[(at + i) * a.stride] = m[i];
    }
    face = qv[N - 1];
    trace = tu;
  }
}

// ---- x pass: a CTA takes XC cells and one halo cell at either side along x, XG cell rows
template<int DIM, int N>
struct OpXCfg
{
  static constexpr int R = DIM == 2 ? N : N * N, CD = N * R;
  // 40 nodes per row: 60 take 385 us at the size above (barriers over larger CTAs), 80 take 431
  static constexpr int XC = 40 / N, XT = XC + 2, CH = (XC * N + 31) / 32;  // rows of CH warps of results
  static constexpr int XG = R * XT >= 160 ? 1 : (160 + R * XT - 1) / (R * XT);
  static constexpr int PENCILS = XT * R * XG, THREADS = (PENCILS + 31) / 32 * 32 > 1024 ? 1024 : (PENCILS + 31) / 32 * 32;
  static constexpr int CS = PENCILS + 1;
  static constexpr int ROWS = XG * R;
  // tables of up to XT widths, traces (2 per pencil), result columns (r and m), row offsets
  static constexpr int TS = (OpTab<N>::SIZE + 1) / 2 * 2;
  static constexpr size_t smem() { return ((size_t)XT * TS + 2 * PENCILS + 2 * (size_t)N * CS + ROWS) * 8; }
};

constexpr int x_regs(int n)
{
  constexpr int r[9] = {0, 0, 40, 56, 56, 64, 72, 72, 72};
  return r[n];
}

template<int DIM, int N>
__global__ void __maxnreg__((x_regs(N))) op_x_kernel(OpLineArgs a)
{
  using C = OpXCfg<DIM, N>;
  using T = OpTab<N>;
  constexpr int R = C::R, XC = C::XC, XT = C::XT, CS = C::CS, P = C::PENCILS;
  extern __shared__ __align__(16) int64_t sx[];
  int2 *s_tab = reinterpret_cast<int2 *>(sx);
  double *s_tr = reinterpret_cast<double *>(sx + XT * C::TS);  // [0]: towards below, [1]: towards above
  double *s_r = s_tr + 2 * P, *s_m = s_r + N * CS;
  int64_t *s_row = reinterpret_cast<int64_t *>(s_m + N * CS);
  const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32, nx = a.nc[0];
  const int ng = a.nc[1] * (DIM == 3 ? a.nc[2] : 1), g0 = blockIdx.x * C::XG, x0 = (blockIdx.y + blockIdx.z * kMaxGridY) * XC;
  if(x0 >= nx) return;  // (all threads: the last multiple of the second dimension is not full)
  const int64_t gx_n = (int64_t)nx * N;
  const int w0 = a.width[x0] & ~kSpecial;
  // one table serves the tile when its cells have the same width
  bool same = true;
  for(int s = 0; s < XT; ++s)
  {
    const int x = x0 - 1 + s;
    if(x >= 0 && x < nx) same = same && (a.width[x] & ~kSpecial) == w0;
  }
  for(int s = 0; s < (same ? 1 : XT); ++s)
  {
    const int x = same ? x0 : x0 - 1 + s;
    if(x < 0 || x >= nx) continue;
    for(int o = tid; o < T::SIZE; o += C::THREADS) s_tab[s * C::TS + o] = a.tab[(size_t)(a.width[x] & ~kSpecial) * T::SIZE + o];
  }
  for(int i = tid; i < C::ROWS; i += C::THREADS)
  {
    const int g = g0 + i / R, r = i % R;
    int64_t row = (int64_t)g * N + r;
    if(DIM == 3)
    {
      const int cy = g % a.nc[1], cz = g / a.nc[1];
      row = ((int64_t)cz * N + r / N) * ((int64_t)a.nc[1] * N) + cy * N + r % N;
    }
    s_row[i] = g < ng ? row * gx_n + (int64_t)x0 * N : -1;
  }
  __syncthreads();
  auto first = [&](int x, int g) {
    const int64_t id = x + (int64_t)nx * g;
    return a.cell_start ? a.cell_start[id] : id * C::CD;
  };
  for(int t = tid; t < P; t += C::THREADS)
  {
    const int rr = t % R, s = (t / R) % XT, g = g0 + t / (R * XT), x = x0 - 1 + s;
    if(g >= ng || x < 0 || x >= nx) continue;
    const int wf = a.width[x], w = wf & ~kSpecial;
    const double *u = a.q + first(x, g) + N * rr;
    double q[N], r[N], m[N], tl, tu;
#pragma unroll
    for(int i = 0; i < N; ++i) q[i] = u[i];
    const bool own = s >= 1 && s <= XC;
    const int2 *tab = s_tab + (same ? 0 : s) * C::TS;
    const double *t64 = a.tab64 + (size_t)w * T::SIZE;
    const int FM = a.exps[3 * w], FC = a.exps[3 * w + 1], FT = a.exps[3 * w + 2];
    if(own)
    {
      auto faces = [&](double &lo, double &hi) {
        lo = x > 0 ? a.q[first(x - 1, g) + N * rr + N - 1] : negated(u[0]);
        hi = x + 1 < nx ? a.q[first(x + 1, g) + N * rr] : negated(u[N - 1]);
      };
      double uL, uR;
      faces(uL, uR);
      cell_pencil<N, false, true, 1>(tab, t64, FM, FC, FT, q, q, uL, uR, r, m, tl, tu, faces);
    }
    else
      cell_pencil<N, false, true, 0>(tab, t64, FM, FC, FT, q, q, 0.0, 0.0, r, m, tl, tu, [](double &, double &) {});
    if(wf & kSpecial) special_faces<N>(a.sig + 3 * x, x > 0, x + 1 < nx, own, q[0], q[N - 1], r[0], r[N - 1], tl, tu);
    if(own)
#pragma unroll
      for(int i = 0; i < N; ++i)
      {
        s_r[i * CS + t] = r[i];
        s_m[i * CS + t] = m[i];
      }
    s_tr[t] = tl;
    s_tr[P + t] = tu;
  }
  __syncthreads();
  for(int t = tid; t < P; t += C::THREADS)
  {
    // the neighbours' traces
    const int s = (t / R) % XT, x = x0 - 1 + s;
    if(g0 + t / (R * XT) >= ng || s < 1 || s > XC || x >= nx) continue;
    if(x > 0) s_r[t] += s_tr[P + t - R];
    if(x + 1 < nx) s_r[(N - 1) * CS + t] += s_tr[t + R];
  }
  __syncthreads();
  // rows of the tile, a warp each
  const int cnt = (int)(gx_n - (int64_t)x0 * N < XC * N ? gx_n - (int64_t)x0 * N : XC * N);
  int at[C::CH];
#pragma unroll
  for(int h = 0; h < C::CH; ++h)
  {
    const int e = lane + 32 * h;
    at[h] = (e % N) * CS + (e / N) * R;
  }
  for(int i = warp; i < C::ROWS; i += C::THREADS / 32)
  {
    if(g0 + i / R >= ng) continue;
    const int t0 = ((i / R) * XT + 1) * R + i % R;
    double *r = a.r + s_row[i], *m = a.m + s_row[i];
#pragma unroll
    for(int h = 0; h < C::CH; ++h)
    {
      const int e = lane + 32 * h;
      if(e >= cnt) continue;
      r[e] = s_r[t0 + at[h]];
      m[e] = s_m[t0 + at[h]];
    }
  }
}
}  // namespace lines
}  // namespace tpss
