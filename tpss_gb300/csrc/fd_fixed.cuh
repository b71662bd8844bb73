// fd_fixed.cuh -- the per-color Schwarz kernel of fd_kernels.cuh for FP64 vectors and FP64 accuracy,
// with its contractions on the integer pipe (fixed64.cuh).
//
// Per patch: gather (the largest exponent of its values becomes the block exponent), S^T along
// x[, y], S^T along the last direction, the reciprocal eigenvalue sums and S along it in registers,
// S along [y,] x, damped scatter-add.  A thread owns one pencil.  Between passes the block lives in
// shared memory as 64-bit integers; every pass ORs the magnitudes of its results, and the next one
// shifts the values up by the headroom left.  The products with the reciprocal eigenvalue sums,
// which span several orders of magnitude, are floating point per value: they are aligned to a
// common exponent only after the largest one of the patch is known.
// Measured (all colors of one application): 3D DGQ4 40^3 5.14 ms with FP64 contractions (FP64 pipe 91 %
// busy), 1.69 ms with integers (the wide-multiply pipe 55 %, the rest waits on shared memory and
// barriers between passes); 2D DGQ3 16^2 106 -> 62 us, where FP64's latency (64 clocks per warp
// instruction) was the time. The FP64 form is kept for nothing else than the values below.
// What the integers do not cover -- infinities, NaN and magnitudes outside 2^(+-300) -- runs the
// FP64 passes of fd_kernels.cuh on the same shared memory, patch by patch.
#pragma once

#include <type_traits>

#include "fd_kernels.cuh"
#include "fixed64.cuh"

namespace tpss
{
namespace fd
{
// padded patch layout x + SX y + SXY z (8-byte values): pencils of consecutive threads fall into
// distinct banks in all three directions where the size allows it (searched over SX < N + 8)
template<int DIM, int N>
struct FixPad
{
  static constexpr int SX = DIM == 2 ? (N <= 4 ? N : N | 1)
                                     : N == 6 ? 9 : N == 8 ? 9 : N == 12 ? 13 : N == 14 ? 17 : N == 16 ? 17 : N;
  static constexpr int SXY = DIM == 2 ? 0
                                      : N == 2 ? 4 : N == 3 ? 12 : N == 4 ? 19 : N == 10 ? 101 : SX * N;
  static constexpr int SIZE = DIM == 2 ? SX * N : SXY * N;
};

template<int DIM, int NCP, int K1>
struct FixCfg
{
  using B = Cfg<double, DIM, NCP, K1>;
  static constexpr int N = B::N, NLOC = B::NLOC, NPENCIL = B::NPENCIL, NCELL = B::NCELL, CELLDOFS = B::CELLDOFS;
  static constexpr int ES = B::ESIZE;  // 8-byte words per table slot
  static constexpr int PS = FixPad<DIM, N>::SIZE;
  static constexpr int CTL = 8;        // control words per patch
  static constexpr int TPP = NPENCIL;  // threads per patch: one per pencil
  static constexpr int MAX_THREADS = 512, MAX_SMEM = 200 * 1024, MAX_VARIANTS = 3;
  // registers per thread (24 to 32 warps per SM; a pencil of up to 16 values takes 2 per value in limbs)
  static constexpr int REGS = N >= 8 ? 80 : 64;
  static constexpr int SLOT_BYTES = PS * 8 + DIM * ES * 8 + NCELL * 12 + CTL * 4;
  static constexpr int PPC_MEM = (96 * 1024) / SLOT_BYTES > 0 ? (96 * 1024) / SLOT_BYTES : 1;
  // patches per CTA: of those with 128 to 256 threads the ones that fill their warps best
  static constexpr int best_ppc()
  {
    int best = 1, best_fill = 0;
    for(int p = 1; p <= PPC_MEM && p * TPP <= 256; ++p)
    {
      const int warps = (p * TPP + 31) / 32, fill = warps < 4 ? 10 * warps : p * TPP * 1000 / (warps * 32);
      if(fill > best_fill)
      {
        best = p;
        best_fill = fill;
      }
    }
    return best;
  }
  static constexpr int PPC = best_ppc();
  static constexpr int ppc(int v) { return PPC << v; }
  static constexpr int threads(int ppc_) { return ((ppc_ * TPP + 31) / 32) * 32; }
  static constexpr size_t al16(size_t x) { return (x + 15) / 16 * 16; }
  struct Lay
  {
    size_t fd, exps, first, w, code, fresh, combo, cls, ctl, map, data, bytes;
  };
  static constexpr Lay lay(int ppc_)
  {
    Lay l{};
    l.fd = 0;
    l.exps = al16(l.fd + (size_t)ppc_ * DIM * ES * 8);
    l.first = al16(l.exps + (size_t)ppc_ * DIM * 8);
    l.w = al16(l.first + (size_t)ppc_ * NCELL * 8);
    l.code = al16(l.w + (size_t)ppc_ * NCELL * 4);
    l.fresh = al16(l.code + (size_t)ppc_ * DIM * 4);
    l.combo = al16(l.fresh + (size_t)ppc_ * DIM * 4);
    l.cls = al16(l.combo + (size_t)ppc_ * 4);
    l.ctl = al16(l.cls + (size_t)ppc_ * 4);
    l.map = al16(l.ctl + (size_t)ppc_ * CTL * 4);
    l.data = al16(l.map + (size_t)NLOC * 4);
    l.bytes = al16(l.data + (size_t)ppc_ * PS * 8);
    return l;
  }
  static constexpr bool variant_ok(int v)
  {
    return v >= 0 && v < MAX_VARIANTS && threads(ppc(v)) <= MAX_THREADS && lay(ppc(v)).bytes <= (size_t)MAX_SMEM;
  }
  static constexpr int n_variants() { return variant_ok(2) ? 3 : variant_ok(1) ? 2 : 1; }
};

// control words of a patch
enum FixCtl
{
  CTL_EMAX,   // largest high word of |value| of the gathered patch
  CTL_LO,     // OR of the low words
  CTL_X,      // exponent of the largest product with a reciprocal eigenvalue sum (biased, unsigned)
  CTL_OR0     // magnitudes after each pass: +0 x forward, +1 y forward, +2 last, +3 y backward
};
constexpr int kFixUnroll = 2;      // rows of a pass per loop iteration
constexpr int kExpBias = 1 << 20;  // CTL_X holds exponent + kExpBias, 0: all products are zero

// one control word per patch from the words of its threads: OR or maximum. All threads of the
// CTA call it; uniform: the warp's active threads belong to one patch.
template<int TPP, bool MAX>
__device__ __forceinline__ void slot_reduce(unsigned *dst, unsigned v, bool active, bool uniform)
{
  constexpr unsigned FULL = 0xffffffffu;
  if(!active) v = 0;
  if constexpr(TPP < 32 && (TPP & (TPP - 1)) == 0)
  {
#pragma unroll
    for(int o = 1; o < TPP; o *= 2)
    {
      const unsigned w = __shfl_xor_sync(FULL, v, o);
      v = MAX ? max(v, w) : (v | w);
    }
    if(active && threadIdx.x % TPP == 0) *dst = v;
  }
  else if(uniform)
  {
    v = MAX ? __reduce_max_sync(FULL, v) : __reduce_or_sync(FULL, v);
    if(active && threadIdx.x % 32 == 0)
    {
      if(MAX) atomicMax(dst, v);
      else atomicOr(dst, v);
    }
  }
  else if(active)
  {
    if(MAX) atomicMax(dst, v);
    else atomicOr(dst, v);
  }
}

// A pencil along a direction, data[m STRIDE], m < N: its values (get(m), |.| < 2^59)
// are replaced by S^T x (FWD) or S x, |.| <= 2^58; ent: the slot's table, dense [S^T][S] or even/odd
// [Se^T][So^T][Se][So]. Returns the OR of the results' magnitudes. The values are held as limbs in
// registers and every result goes straight to shared memory, so that the rows can be a loop: an
// unrolled kernel misses the instruction cache.
template<int N, bool FWD, int STRIDE, typename Get>
__device__ __forceinline__ unsigned fix_pass(int64_t *data, const int2 *__restrict__ ent, bool sym, const Get &get)
{
  unsigned mag = 0;
  if constexpr(N % 2 == 0)
  {
    if(sym)
    {
      using X = EoEntry<double, N>;
      constexpr int H = X::H, HP = X::HPAD;
      int eh[H], el[H], oh[H], ol[H];
#pragma unroll
      for(int i = 0; i < H; ++i)
      {
        // forward: sums and differences of mirrored values; backward: even and odd modes
        const int64_t a = get(i), b = get(FWD ? N - 1 - i : H + i);
        fx::split(FWD ? a + b : a, eh[i], el[i]);
        fx::split(FWD ? a - b : b, oh[i], ol[i]);
      }
      const int2 *re = ent + (FWD ? 0 : X::SE), *ro = ent + (FWD ? X::SOT : X::SO);
#pragma unroll kFixUnroll
      for(int k = 0; k < H; ++k)
      {
        const int64_t e = fx::row_dot<H>(re + k * HP, eh, el), o = fx::row_dot<H>(ro + k * HP, oh, ol);
        const int64_t y0 = FWD ? e : e + o, y1 = FWD ? o : e - o;
        data[k * STRIDE] = y0;
        data[(FWD ? H + k : N - 1 - k) * STRIDE] = y1;
        mag |= fx::mag_hi(y0) | fx::mag_hi(y1);
      }
      return mag;
    }
  }
  constexpr int NP = Entry<double, N>::NPAD;
  const int2 *row = ent + (FWD ? Entry<double, N>::ST : Entry<double, N>::S);
  int h[N], l[N];
#pragma unroll
  for(int i = 0; i < N; ++i) fx::split(get(i), h[i], l[i]);
#pragma unroll kFixUnroll
  for(int i = 0; i < N; ++i)
  {
    const int64_t y = fx::row_dot<N>(row + i * NP, h, l);
    data[i * STRIDE] = y;
    mag |= fx::mag_hi(y);
  }
  return mag;
}

// A pencil's values v[i STRIDE] times positive factors r(i) = m 2^q (in limbs), which may span many orders of magnitude:
// the products are floating point per value first and then share one exponent, with which the
// largest has 59 bits. Returns that exponent less 61 (and whether any product is not zero).
template<int N, int STRIDE, typename R>
__device__ __forceinline__ int scale_by_reciprocals(int64_t *v, const R &r, bool &any)
{
  int64_t y[N];
  int qe[N];
  int e0 = -kExpBias;
#pragma unroll
  for(int i = 0; i < N; ++i)
  {
    int mh, ml;
    r(i, mh, ml, qe[i]);
    y[i] = fx::mul_m61(v[i * STRIDE], mh, ml);
    e0 = max(e0, qe[i]);
  }
  uint64_t mag = 0;
#pragma unroll
  for(int i = 0; i < N; ++i) mag |= fx::shr_u((uint64_t)(y[i] ^ (y[i] >> 63)), e0 - qe[i]);
  const int g = e0 + (64 - __clzll((long long)mag)) - 59;
  any = mag != 0;
#pragma unroll
  for(int i = 0; i < N; ++i) v[i * STRIDE] = fx::shift(y[i], qe[i] - g);
  return g;
}

// FP64 pass for a patch the integers do not cover: the operations of pass() in fd_kernels.cuh on one
// pencil of the padded layout, entries from global memory, rolled loops
template<int N, bool FWD>
__device__ __forceinline__ void slow_pass(double *data, int stride, const double *ent, bool sym, double scale)
{
  double o[N];
  if(N % 2 == 0 && sym)
  {
    using X = EoEntry<double, N>;
    constexpr int H = X::H;
#pragma unroll 1
    for(int k = 0; k < H; ++k)
    {
      double e = 0.0, d = 0.0;
#pragma unroll 1
      for(int i = 0; i < H; ++i)
      {
        const double a = data[i * stride], b = data[(FWD ? N - 1 - i : H + i) * stride];
        e = fma(ent[(FWD ? 0 : X::SE) + k * X::HPAD + i], FWD ? a + b : a, e);
        d = fma(ent[(FWD ? X::SOT : X::SO) + k * X::HPAD + i], FWD ? a - b : b, d);
      }
      o[k] = FWD ? e : e + d;
      o[FWD ? H + k : N - 1 - k] = FWD ? d : e - d;
    }
  }
  else
  {
#pragma unroll 1
    for(int i = 0; i < N; ++i)
    {
      double acc = 0.0;
#pragma unroll 1
      for(int m = 0; m < N; ++m)
        acc = fma(ent[(FWD ? Entry<double, N>::ST : Entry<double, N>::S) + i * Entry<double, N>::NPAD + m],
                  data[m * stride], acc);
      o[i] = acc;
    }
  }
#pragma unroll 1
  for(int i = 0; i < N; ++i) data[i * stride] = o[i] * scale;
}

template<int N, int STRIDE, typename R>
__device__ __forceinline__ int scale_by_reciprocals(int64_t *v, const R &r)
{
  bool any;
  return scale_by_reciprocals<N, STRIDE>(v, r, any);
}

struct FixArgs
{
  KernelArgs k;                       // k.fd, k.fd_eo: FP64 tables (eigenvalues, slow path)
  const int2 *__restrict__ fix;       // integer forms of k.fd and k.fd_eo (same strides)
  const int2 *__restrict__ fix_eo;
  const int2 *__restrict__ fexp;      // per entry: F of S^T (x) and S (y), dense form
  const int2 *__restrict__ fexp_eo;
};

template<int DIM, int NCP, int K1>
__global__ void __maxnreg__((FixCfg<DIM, NCP, K1>::REGS))
  schwarz_color_fixed_kernel(FixArgs fa)
{
  using C = FixCfg<DIM, NCP, K1>;
  using P = FixPad<DIM, C::N>;
  constexpr int N = C::N, NLOC = C::NLOC, NCELL = C::NCELL, CELLDOFS = C::CELLDOFS, ES = C::ES, NPENCIL = C::NPENCIL;
  constexpr int TPP = C::TPP;
  constexpr int SX = P::SX, SXY = P::SXY, PS = C::PS;
  const KernelArgs &a = fa.k;
  const int PPC = a.ppc, NTHR = blockDim.x;
  const typename C::Lay lay = C::lay(PPC);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int2 *s_fd = reinterpret_cast<int2 *>(smem_raw + lay.fd);             // PPC * DIM * ES
  int2 *s_exp = reinterpret_cast<int2 *>(smem_raw + lay.exps);          // PPC * DIM
  int64_t *s_first = reinterpret_cast<int64_t *>(smem_raw + lay.first);  // PPC * NCELL
  float *s_w = reinterpret_cast<float *>(smem_raw + lay.w);
  int *s_code = reinterpret_cast<int *>(smem_raw + lay.code);           // PPC * DIM: 2 entry + symmetric
  int *s_new = reinterpret_cast<int *>(smem_raw + lay.fresh);           // PPC * DIM: the slot's table changed
  int *s_combo = reinterpret_cast<int *>(smem_raw + lay.combo);
  int *s_cls = reinterpret_cast<int *>(smem_raw + lay.cls);
  unsigned *s_ctl = reinterpret_cast<unsigned *>(smem_raw + lay.ctl);
  unsigned *s_map = reinterpret_cast<unsigned *>(smem_raw + lay.map);   // cell-wise DoF -> patch offset, cell, DoF
  int64_t *s_data = reinterpret_cast<int64_t *>(smem_raw + lay.data);   // PPC * PS
  const double *rcp_tab = reinterpret_cast<const double *>(a.rcp);
  const double *fd = reinterpret_cast<const double *>(a.fd);
  const double *fd_eo = reinterpret_cast<const double *>(a.fd_eo);
  const int tid = threadIdx.x;
  const int slot = tid / TPP, q = tid % TPP;
  // the warp's threads work on one patch
  const int warp_last = min(tid | 31, PPC * TPP - 1);
  const bool uniform = (tid & ~31) / TPP == warp_last / TPP;
  for(int i = tid; i < NLOC; i += NTHR)
  {
    const int cn = i / CELLDOFS, e = i % CELLDOFS;
    int off = 0, c = cn, r = e;
    for(int d = 0; d < DIM; ++d)
    {
      off += ((NCP == 1 ? 0 : c % NCP) * K1 + r % K1) * (d == 0 ? 1 : d == 1 ? SX : SXY);
      c /= NCP;
      r /= K1;
    }
    s_map[i] = (unsigned)off | (unsigned)cn << 13 | (unsigned)e << 16;
  }
  // this thread's pencils: x along (y, z), y along (x, z), last direction
  const int pa = q % N, pb = q / N;
  const int bx = DIM == 2 ? SX * q : SX * pa + SXY * pb;
  const int by = DIM == 2 ? q : pa + SXY * pb;
  const int bz = pa + SX * pb;  // 3D
  for(int i = tid; i < PPC * DIM; i += NTHR) s_code[i] = -1;
  __syncthreads();

  for(int64_t p0 = (int64_t)blockIdx.x * PPC; p0 < a.n_patches; p0 += (int64_t)gridDim.x * PPC)
  {
    const int64_t left = a.n_patches - p0;
    const int nvalid = left < PPC ? (int)left : PPC;
    for(int i = tid; i < PPC * NCELL; i += NTHR)
      if(i / NCELL < nvalid)
      {
        s_first[i] = a.patch_first[p0 * NCELL + i];
        if(a.ras_w) s_w[i] = a.ras_w[p0 * NCELL + i];
      }
    for(int i = tid; i < PPC * C::CTL; i += NTHR) s_ctl[i] = 0;
    for(int i = tid; i < nvalid * DIM; i += NTHR)
    {
      // table of the slot: refilled below only when the 1-D problem differs from the previous patch's
      const int e = a.patch_fd[p0 * DIM + i];
      const bool sy = N % 2 == 0 && a.sym && a.sym[e];
      const int code = 2 * e + sy;
      s_new[i] = code != s_code[i];
      s_code[i] = code;
      s_exp[i] = sy ? fa.fexp_eo[e] : fa.fexp[e];
    }
    if(rcp_tab && tid < nvalid)
    {
      int c = 0;
      if(a.rcp_E < 0)
        c = int(p0 + tid);  // one table per patch
      else
#pragma unroll
        for(int d = DIM - 1; d >= 0; --d) c = c * a.rcp_E + a.patch_fd[(p0 + tid) * DIM + d];
      s_combo[tid] = c;
    }
    if(a.keep_mask && tid < nvalid) s_cls[tid] = a.keep_class[p0 + tid];
    __syncthreads();
    const bool active = slot < nvalid;
    const int sl = active ? slot : 0;
    int64_t *my = s_data + sl * PS;
    double *myd = reinterpret_cast<double *>(my);
    unsigned *ctl = s_ctl + sl * C::CTL;
    const int2 *ent = s_fd + sl * DIM * ES;
    const int2 *ex2 = s_exp + sl * DIM;
    const int *code = s_code + sl * DIM;
    // --- gather: whole cells, coalesced; the FP64 values go to shared memory as they are
    {
      unsigned hm = 0, lo = 0;
      if(active)
      {
        double v[N];
#pragma unroll
        for(int j = 0; j < N; ++j)
        {
          const unsigned m = s_map[q + j * TPP];
          v[j] = a.src[s_first[sl * NCELL + ((m >> 13) & 7)] + (m >> 16)];
        }
#pragma unroll
        for(int j = 0; j < N; ++j)
        {
          my[s_map[q + j * TPP] & 0x1fff] = __double_as_longlong(v[j]);
          hm = max(hm, (unsigned)__double2hiint(v[j]) & 0x7fffffffu);
          lo |= (unsigned)__double2loint(v[j]);
        }
      }
      slot_reduce<TPP, true>(ctl + CTL_EMAX, hm, active, uniform);
      slot_reduce<TPP, false>(ctl + CTL_LO, lo, active, uniform);
    }
    for(int sd = 0; sd < nvalid * DIM; ++sd)
    {
      if(!s_new[sd]) continue;
      // coefficients, then the eigenvalues as the FP64 table has them
      const int e = s_code[sd] >> 1, sy = s_code[sd] & 1;
      const int nc = sy ? EoEntry<double, N>::LAM : Entry<double, N>::LAM;
      const int nt = sy ? EoEntry<double, N>::size : Entry<double, N>::size;
      const int2 *c2 = sy ? fa.fix_eo + (size_t)e * a.eo_stride : fa.fix + (size_t)e * a.entry_stride;
      const double *cd = sy ? fd_eo + (size_t)e * a.eo_stride : fd + (size_t)e * a.entry_stride;
      for(int o = tid; o < nt; o += NTHR)
        s_fd[sd * ES + o] = o < nc ? c2[o] : make_int2(__double2loint(cd[o]), __double2hiint(cd[o]));
    }
    __syncthreads();
    int emax = (int)(ctl[CTL_EMAX] >> 20);
    const bool zero = ctl[CTL_EMAX] == 0 && ctl[CTL_LO] == 0;
    const bool slow = !zero && (emax < 1023 - 300 || emax > 1023 + 300);
    if(zero) emax = 1023;
    int ex = emax - 1023 - 58;  // exponent of the block's unit
    // --- S^T along x[, y] and the last direction
    auto forward = [&](auto dir) {
      constexpr int d = decltype(dir)::value, STRIDE = d == 0 ? 1 : d == 1 ? SX : SXY;
      int64_t *p = my + (d == 0 ? bx : d == 1 ? by : bz);
      const int s = d == 0 ? 0 : fx::headroom(ctl[CTL_OR0 + (d > 0 ? d - 1 : 0)]);
      const bool sy = code[d] & 1;
      unsigned mag = 0;
      if(active)
      {
        if(slow)
        {
          const int e = code[d] >> 1;
          slow_pass<N, true>(reinterpret_cast<double *>(p), STRIDE,
                             sy ? fd_eo + (size_t)e * a.eo_stride : fd + (size_t)e * a.entry_stride, sy, 1.0);
        }
        else
          mag = fix_pass<N, true, STRIDE>(p, ent + d * ES, sy, [&](int m) {
            if constexpr(d == 0) return fx::from_double(__longlong_as_double(p[m]), emax);
            else return fx::shl(p[m * STRIDE], s);
          });
      }
      ex += 64 - ex2[d].x - s;
      if constexpr(d < DIM - 1)
      {
        slot_reduce<TPP, false>(ctl + CTL_OR0 + d, mag, active, uniform);
        __syncthreads();
      }
    };
    forward(std::integral_constant<int, 0>{});
    forward(std::integral_constant<int, 1>{});
    if constexpr(DIM == 3) forward(std::integral_constant<int, 2>{});
    // --- times the reciprocal eigenvalue sums (the thread's own pencil of the last direction)
    constexpr int L = DIM - 1, LSTR = DIM == 2 ? SX : SXY;
    int g = 0;  // exponent of the pencil's products
    unsigned xb = 0;
    if(active)
    {
      const double *lamL = reinterpret_cast<const double *>(ent + L * ES) +
                           ((code[L] & 1) ? EoEntry<double, N>::LAM : Entry<double, N>::LAM);
      int64_t *v = my + (DIM == 2 ? by : bz);
      const double *rt = rcp_tab ? rcp_tab + (size_t)s_combo[sl] * NLOC + q : nullptr;
      double lsum = 0.0;
      if(!rt)
      {
        int rem = q;
#pragma unroll
        for(int d = 0; d < DIM - 1; ++d)
        {
          const int lam = (code[d] & 1) ? EoEntry<double, N>::LAM : Entry<double, N>::LAM;
          lsum += reinterpret_cast<const double *>(ent)[d * ES + lam + rem % N];
          rem /= N;
        }
      }
      if(slow)
      {
        double *o = reinterpret_cast<double *>(v);
#pragma unroll 1
        for(int i = 0; i < N; ++i)
        {
          if(rt) o[i * LSTR] *= __ldg(rt + i * NPENCIL);
          else o[i * LSTR] = o[i * LSTR] / (lsum + lamL[i]);
        }
      }
      else
      {
        bool any;
        g = scale_by_reciprocals<N, LSTR>(
          v,
          [&](int i, int &mh, int &ml, int &e) {
            if(rt) fx::split_positive(__ldg(rt + i * NPENCIL), mh, ml, e);
            else fx::reciprocal(lsum + lamL[i], mh, ml, e);
          },
          any);
        if(any) xb = (unsigned)(g + 59 + kExpBias);
      }
    }
    slot_reduce<TPP, true>(ctl + CTL_X, xb, active, uniform);
    __syncthreads();
    // --- S along the last direction[, y] and x
    const unsigned X = ctl[CTL_X];
    const int G = X ? (int)X - kExpBias - 59 : 0;  // exponent of the aligned block
    ex += 61 + G;
    auto backward = [&](auto dir) {
      constexpr int d = decltype(dir)::value, STRIDE = d == 0 ? 1 : d == 1 ? SX : SXY;
      int64_t *p = my + (d == 0 ? bx : d == 1 ? by : bz);
      const int s = d == L ? 0 : fx::headroom(ctl[CTL_OR0 + DIM - 2 + L - d]);
      const bool sy = code[d] & 1;
      unsigned mag = 0;
      if(active)
      {
        if(slow)
        {
          const int e = code[d] >> 1;
          slow_pass<N, false>(reinterpret_cast<double *>(p), STRIDE,
                              sy ? fd_eo + (size_t)e * a.eo_stride : fd + (size_t)e * a.entry_stride, sy,
                              d == 0 ? a.omega : 1.0);
        }
        else
          // the last direction's pencils come down to the block's exponent
          mag = fix_pass<N, false, STRIDE>(p, ent + d * ES, sy, [&](int m) {
            return d == L ? fx::shr_s(p[m * STRIDE], G - g) : fx::shl(p[m * STRIDE], s);
          });
      }
      ex += 64 - ex2[d].y - s;
      if constexpr(d > 0) slot_reduce<TPP, false>(ctl + CTL_OR0 + DIM - 1 + L - d, mag, active, uniform);
      __syncthreads();
    };
    if constexpr(DIM == 3) backward(std::integral_constant<int, 2>{});
    backward(std::integral_constant<int, 1>{});
    backward(std::integral_constant<int, 0>{});
    // --- scatter-add: whole cells, coalesced read-modify-write, a few values in flight per thread
    if(active)
    {
      // value = integer * omega 2^ex; beyond the exponent range of one factor in two steps
      const bool far = ex < -1000 || ex > 900;
      const bool plain = !slow && !far && !a.ras_w && !a.keep_mask;
      const double sc = slow ? 1.0 : far ? a.omega : a.omega * fx::pow2(ex);
      constexpr int CH = N % 5 == 0 ? 5 : N % 4 == 0 ? 4 : N % 7 == 0 ? 7 : N % 3 == 0 ? 3 : N;
#pragma unroll 1
      for(int j0 = 0; j0 < N; j0 += CH)
      {
        double old[CH];
        double *at[CH];
        unsigned m[CH];
#pragma unroll
        for(int j = 0; j < CH; ++j)
        {
          m[j] = s_map[q + (j0 + j) * TPP];
          at[j] = a.dst + s_first[sl * NCELL + ((m[j] >> 13) & 7)] + (m[j] >> 16);
          old[j] = *at[j];
        }
        if(plain)
        {
#pragma unroll
          for(int j = 0; j < CH; ++j) *at[j] = fma(__ll2double_rn(my[m[j] & 0x1fff]), sc, old[j]);
        }
        else
        {
#pragma unroll 1
          for(int j = 0; j < CH; ++j)
          {
            const unsigned mj = s_map[q + (j0 + j) * TPP];
            const int off = mj & 0x1fff, cn = (mj >> 13) & 7;
            if(a.keep_mask)
            {
              // RAS boolean weights (rscatter_add): only the patch that owns the DoF adds it
              const int pl = DIM == 2 ? off % SX + N * (off / SX)
                                      : (off % SXY) % SX + N * ((off % SXY) / SX) + N * N * (off / SXY);
              if(!a.keep_mask[s_cls[sl] * NLOC + pl]) continue;
            }
            double *d = a.dst + s_first[sl * NCELL + cn] + (mj >> 16);
            double v = slow ? myd[off] : __ll2double_rn(my[off]) * sc;
            if(far && !slow) v = scalbn(v, ex);
            *d += a.ras_w ? v * double(s_w[sl * NCELL + cn]) : v;
          }
        }
      }
    }
    __syncthreads();
  }
}

template<int DIM, int NCP, int K1>
bool launch_fixed(FixArgs fa, cudaStream_t s, int n_sms, int variant)
{
  using C = FixCfg<DIM, NCP, K1>;
  if(!C::variant_ok(variant)) variant = 0;
  if(fa.k.n_patches <= 0) return true;
  // few patches: smaller CTAs, so that every SM gets some of them
  int ppc = C::ppc(variant);
  while(ppc > 1 && (fa.k.n_patches + ppc - 1) / ppc < 2 * n_sms) ppc = (ppc + 1) / 2;
  fa.k.ppc = ppc;
  const int threads = C::threads(ppc);
  const size_t smem = C::lay(ppc).bytes;
  static int per_sm[C::ppc(C::n_variants() - 1) + 1] = {};  // occupancy per size, queried once
  if(per_sm[ppc] == 0)
  {
    const size_t smem_max = C::lay(C::ppc(C::n_variants() - 1)).bytes;
    if(cudaFuncSetAttribute(schwarz_color_fixed_kernel<DIM, NCP, K1>,
                            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max) != cudaSuccess)
      return false;
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, schwarz_color_fixed_kernel<DIM, NCP, K1>, threads, smem);
    per_sm[ppc] = occ < 1 ? 1 : occ;
  }
  const int64_t batches = (fa.k.n_patches + ppc - 1) / ppc;
  const int64_t cap = (int64_t)n_sms * per_sm[ppc];
  const int grid = (int)(batches < cap ? batches : cap);
  schwarz_color_fixed_kernel<DIM, NCP, K1><<<grid, threads, smem, s>>>(fa);
  return cudaGetLastError() == cudaSuccess;
}
}  // namespace fd
}  // namespace tpss
