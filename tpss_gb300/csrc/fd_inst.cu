// fd_inst.cu -- instantiations of the fused Schwarz color kernel for one arithmetic type and
// dimension.  Compiled once per (FD_T, FD_DIM) pair (float/double x 2/3), so the four
// translation units build in parallel.
#include <type_traits>

#include "fd_fixed.cuh"
#include "fd_kernels.cuh"
#include "internal.h"

#ifndef FD_T
#error "FD_T must be defined (float or double)"
#endif
#ifndef FD_DIM
#error "FD_DIM must be defined (2 or 3)"
#endif

#define TPSS_CAT2(a, b) a##b
#define TPSS_CAT(a, b) TPSS_CAT2(a, b)
#define TPSS_FD_FN TPSS_CAT(TPSS_CAT(launch_fd_, FD_T), TPSS_CAT(_, FD_DIM))

namespace tpss
{
namespace
{
// FP64: the contractions run on the integer pipe (fd_fixed.cuh); where the tables rule that out (indefinite local
// problems) the FP64 kernel does all patches: the integer one's own FP64 passes, which are there for single
// patches out of range, take 1.1 to 1.4 times as long (cell patches, 2D k = 7, 20^2: 34.9 against 47.6 us)
template<typename T, int DIM, int NCP, int K1>
bool launch_one(const fd::KernelArgs &a, const FdLaunch &l, cudaStream_t s, int sms)
{
  if constexpr(std::is_same_v<T, double>)
  {
    if(l.fp64_only) return fd::launch<T, DIM, NCP, K1>(a, s, sms, l.variant);
    fd::FixArgs f;
    f.k = a;
    f.fix = l.fix;
    f.fix_eo = l.fix_eo;
    f.fexp = l.fexp;
    f.fexp_eo = l.fexp_eo;
    return fd::launch_fixed<DIM, NCP, K1>(f, s, sms, l.variant);
  }
  else
    return fd::launch<T, DIM, NCP, K1>(a, s, sms, l.variant);
}

template<typename T, int DIM, int NCP, int K1>
constexpr int variants()
{
  if constexpr(std::is_same_v<T, double>)
    return fd::FixCfg<DIM, NCP, K1>::n_variants();
  else
    return fd::Cfg<T, DIM, NCP, K1>::n_variants();
}
}  // namespace

bool TPSS_FD_FN(int k, int ncp, const FdLaunch &l, cudaStream_t s)
{
  fd::KernelArgs a;
  a.src = l.src;
  a.dst = l.dst;
  a.patch_first = l.patch_first;
  a.patch_fd = l.patch_fd;
  a.fd = l.fd;
  a.ras_w = l.ras_w;
  a.n_patches = l.n_patches;
  a.omega = l.omega;
  a.entry_stride = l.entry_stride;
  a.fd_eo = l.fd_eo;
  a.sym = l.sym;
  a.eo_stride = l.eo_stride;
  a.rcp = l.rcp;
  a.rcp_E = l.rcp_E;
  a.keep_mask = l.keep_mask;
  a.keep_class = l.keep_class;
  const int sms = num_sms();
#define TPSS_FD_CASE(NCP, K1) \
  if(ncp == NCP && k + 1 == K1) return launch_one<FD_T, FD_DIM, NCP, K1>(a, l, s, sms);
  TPSS_FD_CASE(1, 2) TPSS_FD_CASE(1, 3) TPSS_FD_CASE(1, 4) TPSS_FD_CASE(1, 5)
  TPSS_FD_CASE(1, 6) TPSS_FD_CASE(1, 7) TPSS_FD_CASE(1, 8)
  TPSS_FD_CASE(2, 2) TPSS_FD_CASE(2, 3) TPSS_FD_CASE(2, 4) TPSS_FD_CASE(2, 5)
  TPSS_FD_CASE(2, 6) TPSS_FD_CASE(2, 7) TPSS_FD_CASE(2, 8)
#undef TPSS_FD_CASE
  return false;
}

// work decompositions (patches per CTA) the kernel of (k, ncp) offers to the autotuner
int TPSS_CAT(TPSS_CAT(fd_variants_, FD_T), TPSS_CAT(_, FD_DIM))(int k, int ncp)
{
#define TPSS_FD_CASE(NCP, K1) \
  if(ncp == NCP && k + 1 == K1) return variants<FD_T, FD_DIM, NCP, K1>();
  TPSS_FD_CASE(1, 2) TPSS_FD_CASE(1, 3) TPSS_FD_CASE(1, 4) TPSS_FD_CASE(1, 5)
  TPSS_FD_CASE(1, 6) TPSS_FD_CASE(1, 7) TPSS_FD_CASE(1, 8)
  TPSS_FD_CASE(2, 2) TPSS_FD_CASE(2, 3) TPSS_FD_CASE(2, 4) TPSS_FD_CASE(2, 5)
  TPSS_FD_CASE(2, 6) TPSS_FD_CASE(2, 7) TPSS_FD_CASE(2, 8)
#undef TPSS_FD_CASE
  return 1;
}
}  // namespace tpss
