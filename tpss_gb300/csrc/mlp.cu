// Small fully connected network for the learned local solver, trained on the GPU.
//
// Layers: n_in -> n_hidden (tanh) -> ... -> n_hidden (tanh) -> n_out (linear), FP32. The
// widths are small (tens of units), so every layer is a tiled CUDA-core product with a fixed
// summation order. A mini-batch's products are far too small for tensor-core tiles; those of a whole level's patches
// (tens of thousands of rows) are not, but FP32 results would take several tensor-core products each.
// Training minimizes the mean squared error over all outputs with Adam (Kingma & Ba 2015:
// beta1 0.9, beta2 0.999, eps 1e-8, bias-corrected moments), mini-batches in a seeded
// permutation per epoch.
// Parameter vector: for every layer l, W_l [out][in] row-major, then b_l [out].
#include "internal.h"

#include <cmath>
#include <numeric>

struct tpss_mlp
{
  int n_in = 0, n_hidden = 0, n_hidden_layers = 0, n_out = 0;
  std::vector<int> width;      // n_layers + 1 widths, width[0] = n_in
  std::vector<int64_t> w_off;  // offset of W_l in the parameter vector
  std::vector<int64_t> b_off;
  int64_t n_params = 0;
  tpss::DeviceBuffer<float> params, grads, adam_m, adam_v;
  int64_t adam_step = 0;
  // activations of the last forward pass (for backward): one buffer per layer output
  std::vector<tpss::DeviceBuffer<float>> act;
  tpss::DeviceBuffer<float> delta0, delta1, partial, xb, yb;
  tpss::DeviceBuffer<float> wpart;  // partial weight gradients of the row chunks
  int64_t act_rows = 0;
  int n_layers() const { return (int)width.size() - 1; }
};

namespace tpss
{
namespace
{
constexpr int kLossBlocks = 256;

// The layers' products as one tiled kernel, C (M x N) = op(A) op(B) over K in FP32:
//   FWD   y[r][o]  = act(b[o] + sum_i x[r][i] W[o][i])           M rows, N outputs, K inputs
//   DGRAD dx[r][i] = (sum_o delta[r][o] W[o][i]) (1 - a[r][i]^2)  M rows, N inputs, K outputs
//   WGRAD dW[o][i] = sum_r delta[r][o] x[r][i], i = n_in: db[o]   M outputs, N inputs + 1, K rows
// A CTA computes a BM x BN tile, a thread TM x TN results; A and B pass through shared memory
// BK deep. FWD and DGRAD add in ascending k. WGRAD's long sum over the rows is cut into chunks, one
// grid layer each, whose partial results wgrad_reduce_kernel adds in ascending order: both orders are
// fixed. For the local-solver network (29,791 rows, 87-64-64-64-108) one forward pass and one gradient
// took 12.7 ms with a thread per result (the weight gradient's threads walked all rows, the others
// read the weights uncoalesced); now 0.47 ms, 19 to 25 us per product (about 20 TFLOP/s, bound by
// shared-memory reads). Large tiles below num_sms() * 64 rows would leave SMs empty.
enum GemmOp
{
  GEMM_FWD,
  GEMM_DGRAD,
  GEMM_WGRAD
};

struct GemmArgs
{
  const float *A, *B;   // FWD: x, W; DGRAD: delta, W; WGRAD: delta, x
  float *C;
  const float *bias;    // FWD: b; DGRAD: tanh outputs a of the layer below
  float *db;            // WGRAD without chunks: bias gradient
  int64_t M, N, K;
  int64_t lda, ldb;     // row lengths
  int64_t chunk;        // WGRAD: rows per grid layer
  int tanh_act;
};

template<int OP, int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_kernel(const GemmArgs g)
{
  constexpr int NT = (BM / TM) * (BN / TN);
  __shared__ __align__(16) float sa[BK][BM + 4], sb[BK][BN + 4];
  const int tid = threadIdx.x, tn = tid % (BN / TN), tm = tid / (BN / TN);
  const int64_t m0 = (int64_t)blockIdx.x * BM, n0 = (int64_t)blockIdx.y * BN;
  const int64_t k_begin = OP == GEMM_WGRAD ? blockIdx.z * g.chunk : 0;
  const int64_t k_end = OP == GEMM_WGRAD && k_begin + g.chunk < g.K ? k_begin + g.chunk : g.K;
  float acc[TM][TN];
#pragma unroll
  for(int i = 0; i < TM; ++i)
#pragma unroll
    for(int j = 0; j < TN; ++j)
    {
      const int64_t n = n0 + tn * TN + j;
      acc[i][j] = OP == GEMM_FWD && n < g.N ? g.bias[n] : 0.f;
    }
  // the next step's values are on their way to registers while this one's are used
  constexpr int PA = BM * BK / NT, PB = BN * BK / NT;
  static_assert(PA * NT == BM * BK && PB * NT == BN * BK, "the threads share a step's values evenly");
  float ra[PA], rb[PB];
  auto fetch = [&](int64_t k0) {
    // A: rows of K values (FWD, DGRAD) or K rows of M values (WGRAD)
#pragma unroll
    for(int p = 0; p < PA; ++p)
    {
      const int i = tid + p * NT;
      const int kk = OP == GEMM_WGRAD ? i / BM : i % BK, mm = OP == GEMM_WGRAD ? i % BM : i / BK;
      const int64_t m = m0 + mm, k = k0 + kk;
      ra[p] = m < g.M && k < k_end ? (OP == GEMM_WGRAD ? g.A[k * g.lda + m] : g.A[m * g.lda + k]) : 0.f;
    }
    // B: rows of K values (FWD) or K rows of N values; WGRAD has ones behind its last input
#pragma unroll
    for(int p = 0; p < PB; ++p)
    {
      const int i = tid + p * NT;
      const int kk = OP == GEMM_FWD ? i % BK : i / BN, nn = OP == GEMM_FWD ? i / BK : i % BN;
      const int64_t n = n0 + nn, k = k0 + kk;
      rb[p] = 0.f;
      if(n < g.N && k < k_end)
        rb[p] = OP == GEMM_FWD ? g.B[n * g.ldb + k] : OP == GEMM_WGRAD && n == g.N - 1 ? 1.f : g.B[k * g.ldb + n];
    }
  };
  fetch(k_begin);
  for(int64_t k0 = k_begin; k0 < k_end; k0 += BK)
  {
#pragma unroll
    for(int p = 0; p < PA; ++p)
    {
      const int i = tid + p * NT;
      sa[OP == GEMM_WGRAD ? i / BM : i % BK][OP == GEMM_WGRAD ? i % BM : i / BK] = ra[p];
    }
#pragma unroll
    for(int p = 0; p < PB; ++p)
    {
      const int i = tid + p * NT;
      sb[OP == GEMM_FWD ? i % BK : i / BN][OP == GEMM_FWD ? i / BK : i % BN] = rb[p];
    }
    __syncthreads();
    if(k0 + BK < k_end) fetch(k0 + BK);
    const int kn = k_end - k0 < BK ? (int)(k_end - k0) : BK;
    auto step = [&](int k) {
      float a[TM], b[TN];
#pragma unroll
      for(int i = 0; i < TM; ++i) a[i] = sa[k][tm * TM + i];
#pragma unroll
      for(int j = 0; j < TN; ++j) b[j] = sb[k][tn * TN + j];
#pragma unroll
      for(int i = 0; i < TM; ++i)
#pragma unroll
        for(int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    };
    if(kn == BK)
    {
#pragma unroll
      for(int k = 0; k < BK; ++k) step(k);
    }
    else
      for(int k = 0; k < kn; ++k) step(k);  // (zeros in the padding would turn infinities into NaN)
    __syncthreads();
  }
  float *C = g.C;
  if(OP == GEMM_WGRAD && gridDim.z > 1) C += blockIdx.z * g.M * g.N;
#pragma unroll
  for(int i = 0; i < TM; ++i)
  {
    const int64_t m = m0 + tm * TM + i;
    if(m >= g.M) continue;
#pragma unroll
    for(int j = 0; j < TN; ++j)
    {
      const int64_t n = n0 + tn * TN + j;
      if(n >= g.N) continue;
      float v = acc[i][j];
      if constexpr(OP == GEMM_FWD)
        C[m * g.N + n] = g.tanh_act ? tanhf(v) : v;
      else if constexpr(OP == GEMM_DGRAD)
      {
        const float ai = g.bias[m * g.N + n];
        C[m * g.N + n] = v * (1.f - ai * ai);
      }
      else if(gridDim.z > 1)
        C[m * g.N + n] = v;
      else if(n < g.N - 1)
        C[m * (g.N - 1) + n] = v;
      else
        g.db[m] = v;
    }
  }
}

// dW, db = sum of the chunks' partial results (chunks x M x N, N = n_in + 1), ascending
__global__ void wgrad_reduce_kernel(const float *__restrict__ part, int chunks, int64_t M, int64_t N,
                                    float *__restrict__ dW, float *__restrict__ db)
{
  const int64_t total = M * N;
  for(int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x)
  {
    float s = 0.f;
#pragma unroll 8
    for(int c = 0; c < chunks; ++c) s += part[c * total + t];  // 8 loads in flight, added in order
    const int64_t m = t / N, n = t % N;
    if(n < N - 1) dW[m * (N - 1) + n] = s;
    else db[m] = s;
  }
}

// delta = 2 (y - target) / (rows * n_out); per-block partial sums of the squared error
__global__ void mse_kernel(const float *__restrict__ y, const float *__restrict__ target,
                           int64_t total, float scale, float *__restrict__ delta,
                           float *__restrict__ partial)
{
  __shared__ float red[256];
  float s = 0.f;
  for(int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
      t += (int64_t)gridDim.x * blockDim.x)
  {
    const float e = y[t] - target[t];
    s += e * e;
    if(delta) delta[t] = 2.f * scale * e;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for(int w = blockDim.x / 2; w > 0; w /= 2)
  {
    if(threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if(threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

__global__ void adam_kernel(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, int64_t n, float lr, float c1, float c2)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
      i += (int64_t)gridDim.x * blockDim.x)
  {
    const float gi = g[i];
    const float mi = 0.9f * m[i] + 0.1f * gi;
    const float vi = 0.999f * v[i] + 0.001f * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
  }
}

__global__ void gather_rows_kernel(const float *__restrict__ src, const int64_t *__restrict__ idx,
                                   int64_t rows, int width, float *__restrict__ dst)
{
  const int64_t total = rows * width;
  for(int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
      t += (int64_t)gridDim.x * blockDim.x)
  {
    const int64_t r = t / width;
    dst[t] = src[idx[r] * width + t % width];
  }
}

unsigned grid_of(int64_t n)
{
  const int64_t b = (n + 255) / 256, cap = (int64_t)num_sms() * 8;
  return (unsigned)(b < 1 ? 1 : (b < cap ? b : cap));
}

// splitmix64 (Steele, Lea, Flood 2014) for the seeded initialisation and shuffles
uint64_t splitmix(uint64_t &s)
{
  uint64_t z = (s += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
double uniform01(uint64_t &s) { return (splitmix(s) >> 11) * (1.0 / 9007199254740992.0); }
}  // namespace
}  // namespace tpss

namespace tpss
{
namespace
{
void ensure_rows(tpss_mlp &m, int64_t rows)
{
  if(rows <= m.act_rows) return;
  const int L = m.n_layers();
  m.act.resize(L);
  int wmax = 0;
  for(int w : m.width) wmax = std::max(wmax, w);
  for(int l = 0; l < L; ++l) m.act[l].resize((size_t)(rows * m.width[l + 1]));
  m.delta0.resize((size_t)(rows * wmax));
  m.delta1.resize((size_t)(rows * wmax));
  m.act_rows = rows;
}

// tiles of 64 x 64 results (4 x 4 per thread) where there are enough rows to fill the chip with them,
// else 16 x 32 (2 x 1): a mini-batch of 256 rows makes 16 CTAs or more of a layer
template<int OP>
void launch_gemm(const GemmArgs &g, cudaStream_t s)
{
  if(g.M >= 64 * (int64_t)num_sms())
    gemm_kernel<OP, 64, 64, 16, 4, 4><<<dim3((unsigned)((g.M + 63) / 64), (unsigned)((g.N + 63) / 64)), 256, 0, s>>>(g);
  else
    gemm_kernel<OP, 16, 32, 32, 2, 1><<<dim3((unsigned)((g.M + 15) / 16), (unsigned)((g.N + 31) / 32)), 256, 0, s>>>(g);
  TPSS_CUDA(cudaGetLastError());
}

// weight and bias gradient of one layer; the rows are cut into chunks until the tiles fill the chip's 152 SMs
// twice, but not below 64 rows. The count is fixed, so that the order of the sums depends on the sizes alone
constexpr int kWgradCtas = 304;

void launch_wgrad(tpss_mlp &m, const float *delta, const float *x, int64_t rows, int ni, int no, float *dW, float *db,
                  cudaStream_t s)
{
  GemmArgs g{};
  g.A = delta;
  g.B = x;
  g.M = no;
  g.N = ni + 1;
  g.K = rows;
  g.lda = no;
  g.ldb = ni;
  const bool large = rows >= 4096;
  const int T = large ? 64 : 32;
  const int64_t tiles = ((g.M + T - 1) / T) * ((g.N + T - 1) / T);
  int64_t chunks = std::min<int64_t>((kWgradCtas + tiles - 1) / tiles, (rows + 63) / 64);
  g.chunk = (rows + chunks - 1) / chunks;
  chunks = (rows + g.chunk - 1) / g.chunk;
  g.db = db;
  g.C = dW;
  if(chunks > 1)
  {
    const size_t need = (size_t)(chunks * g.M * g.N);
    if(m.wpart.n < need) m.wpart.resize(need);
    g.C = m.wpart.ptr;
  }
  const dim3 grid((unsigned)((g.M + T - 1) / T), (unsigned)((g.N + T - 1) / T), (unsigned)chunks);
  if(large) gemm_kernel<GEMM_WGRAD, 64, 64, 16, 4, 4><<<grid, 256, 0, s>>>(g);
  else gemm_kernel<GEMM_WGRAD, 32, 32, 32, 4, 2><<<grid, 128, 0, s>>>(g);
  if(chunks > 1)
    wgrad_reduce_kernel<<<grid_of(g.M * g.N), 256, 0, s>>>(m.wpart.ptr, (int)chunks, g.M, g.N, dW, db);
  TPSS_CUDA(cudaGetLastError());
}

// forward pass of `rows` inputs; the output is m.act[L-1], or y where given
void mlp_forward(tpss_mlp &m, const float *x, int64_t rows, cudaStream_t s, float *y = nullptr)
{
  ensure_rows(m, rows);
  const int L = m.n_layers();
  const float *in = x;
  for(int l = 0; l < L; ++l)
  {
    GemmArgs g{};
    g.A = in;
    g.B = m.params.ptr + m.w_off[l];
    g.bias = m.params.ptr + m.b_off[l];
    g.C = l + 1 == L && y ? y : m.act[l].ptr;
    g.M = rows;
    g.N = m.width[l + 1];
    g.K = g.lda = g.ldb = m.width[l];
    g.tanh_act = l + 1 < L;
    launch_gemm<GEMM_FWD>(g, s);
    in = m.act[l].ptr;
  }
}

// MSE loss of the last forward pass against `target` and its gradient in m.grads
void mlp_loss_backward(tpss_mlp &m, const float *x, const float *target, int64_t rows, cudaStream_t s,
                       bool want_loss, double *loss)
{
  const int L = m.n_layers();
  const int64_t total = rows * m.n_out;
  if(m.partial.n < (size_t)kLossBlocks) m.partial.resize(kLossBlocks);
  mse_kernel<<<kLossBlocks, 256, 0, s>>>(m.act[L - 1].ptr, target, total, 1.f / float(total),
                                         m.delta0.ptr, m.partial.ptr);
  TPSS_CUDA(cudaGetLastError());
  float *delta = m.delta0.ptr, *other = m.delta1.ptr;
  for(int l = L - 1; l >= 0; --l)
  {
    const int ni = m.width[l], no = m.width[l + 1];
    const float *in = l == 0 ? x : m.act[l - 1].ptr;
    launch_wgrad(m, delta, in, rows, ni, no, m.grads.ptr + m.w_off[l], m.grads.ptr + m.b_off[l], s);
    if(l > 0)
    {
      GemmArgs g{};
      g.A = delta;
      g.B = m.params.ptr + m.w_off[l];
      g.bias = m.act[l - 1].ptr;
      g.C = other;
      g.M = rows;
      g.N = g.ldb = ni;
      g.K = g.lda = no;
      launch_gemm<GEMM_DGRAD>(g, s);
      std::swap(delta, other);
    }
  }
  TPSS_CUDA(cudaGetLastError());
  if(want_loss)
  {
    std::vector<float> h(kLossBlocks);
    TPSS_CUDA(cudaMemcpyAsync(h.data(), m.partial.ptr, sizeof(float) * kLossBlocks, cudaMemcpyDeviceToHost, s));
    TPSS_CUDA(cudaStreamSynchronize(s));
    double t = 0.0;
    for(float v : h) t += v;
    *loss = t / double(total);
  }
}

double mlp_loss_only(tpss_mlp &m, const float *x, const float *target, int64_t rows, cudaStream_t s)
{
  mlp_forward(m, x, rows, s);
  const int64_t total = rows * m.n_out;
  if(m.partial.n < (size_t)kLossBlocks) m.partial.resize(kLossBlocks);
  mse_kernel<<<kLossBlocks, 256, 0, s>>>(m.act[m.n_layers() - 1].ptr, target, total, 1.f, nullptr, m.partial.ptr);
  TPSS_CUDA(cudaGetLastError());
  std::vector<float> h(kLossBlocks);
  TPSS_CUDA(cudaMemcpyAsync(h.data(), m.partial.ptr, sizeof(float) * kLossBlocks, cudaMemcpyDeviceToHost, s));
  TPSS_CUDA(cudaStreamSynchronize(s));
  double t = 0.0;
  for(float v : h) t += v;
  return t / double(total);
}
}  // namespace

void mlp_infer(const tpss_mlp &mc, const float *x_dev, int64_t rows, float *y_dev, cudaStream_t s)
{
  tpss_mlp &m = const_cast<tpss_mlp &>(mc);  // activation scratch only
  // y may be x: the last of several layers reads activations, a single one x itself
  const bool single = m.n_layers() == 1;
  mlp_forward(m, x_dev, rows, s, single ? nullptr : y_dev);
  if(single)
    TPSS_CUDA(cudaMemcpyAsync(y_dev, m.act[0].ptr, sizeof(float) * rows * m.n_out, cudaMemcpyDeviceToDevice, s));
}

int mlp_n_in(const tpss_mlp &m) { return m.n_in; }
int mlp_n_out(const tpss_mlp &m) { return m.n_out; }
}  // namespace tpss

using namespace tpss;

extern "C" int tpss_mlp_create(const tpss_mlp_desc *d, tpss_mlp **out)
{
  return guarded([&] {
    TPSS_REQUIRE(d && out, "null argument");
    *out = nullptr;
    TPSS_REQUIRE(d->n_in >= 1 && d->n_out >= 1 && d->n_hidden >= 1 && d->n_hidden_layers >= 0 &&
                   d->n_in <= 4096 && d->n_out <= 4096 && d->n_hidden <= 4096 && d->n_hidden_layers <= 16,
                 "invalid network sizes");
    auto m = std::make_unique<tpss_mlp>();
    m->n_in = d->n_in;
    m->n_hidden = d->n_hidden;
    m->n_hidden_layers = d->n_hidden_layers;
    m->n_out = d->n_out;
    m->width.push_back(d->n_in);
    for(int l = 0; l < d->n_hidden_layers; ++l) m->width.push_back(d->n_hidden);
    m->width.push_back(d->n_out);
    const int L = m->n_layers();
    int64_t off = 0;
    for(int l = 0; l < L; ++l)
    {
      m->w_off.push_back(off);
      off += (int64_t)m->width[l] * m->width[l + 1];
      m->b_off.push_back(off);
      off += m->width[l + 1];
    }
    m->n_params = off;
    // Glorot-uniform weights, zero biases
    std::vector<float> p(off, 0.f);
    uint64_t st = d->seed;
    for(int l = 0; l < L; ++l)
    {
      const double a = std::sqrt(6.0 / (m->width[l] + m->width[l + 1]));
      for(int64_t i = 0; i < (int64_t)m->width[l] * m->width[l + 1]; ++i)
        p[m->w_off[l] + i] = float(a * (2.0 * uniform01(st) - 1.0));
    }
    m->params.upload(p.data(), p.size());
    m->grads.resize(off);
    std::vector<float> z(off, 0.f);
    m->adam_m.upload(z.data(), z.size());
    m->adam_v.upload(z.data(), z.size());
    *out = m.release();
  });
}

extern "C" int tpss_mlp_n_params(const tpss_mlp *m, int64_t *n)
{
  return guarded([&] {
    TPSS_REQUIRE(m && n, "null argument");
    *n = m->n_params;
  });
}

extern "C" int tpss_mlp_get_params(const tpss_mlp *m, float *host)
{
  return guarded([&] {
    TPSS_REQUIRE(m && host, "null argument");
    TPSS_CUDA(cudaMemcpy(host, m->params.ptr, sizeof(float) * m->n_params, cudaMemcpyDeviceToHost));
  });
}

extern "C" int tpss_mlp_set_params(tpss_mlp *m, const float *host)
{
  return guarded([&] {
    TPSS_REQUIRE(m && host, "null argument");
    for(int64_t i = 0; i < m->n_params; ++i) TPSS_REQUIRE(std::isfinite(host[i]), "parameters must be finite");
    TPSS_CUDA(cudaMemcpy(m->params.ptr, host, sizeof(float) * m->n_params, cudaMemcpyHostToDevice));
    m->adam_step = 0;
    TPSS_CUDA(cudaMemset(m->adam_m.ptr, 0, sizeof(float) * m->n_params));
    TPSS_CUDA(cudaMemset(m->adam_v.ptr, 0, sizeof(float) * m->n_params));
  });
}

extern "C" int tpss_mlp_forward(tpss_mlp *m, const float *x, int64_t rows, float *y, void *stream)
{
  return guarded([&] {
    TPSS_REQUIRE(m && x && y && rows >= 0, "invalid argument");
    if(rows) mlp_infer(*m, x, rows, y, as_stream(stream));
  });
}

extern "C" int tpss_mlp_loss_grad(tpss_mlp *m, const float *x, const float *target, int64_t rows,
                                  double *loss, float *grad_host)
{
  return guarded([&] {
    TPSS_REQUIRE(m && x && target && loss && rows >= 1, "invalid argument");
    mlp_forward(*m, x, rows, nullptr);
    mlp_loss_backward(*m, x, target, rows, nullptr, true, loss);
    if(grad_host)
      TPSS_CUDA(cudaMemcpy(grad_host, m->grads.ptr, sizeof(float) * m->n_params, cudaMemcpyDeviceToHost));
  });
}

extern "C" int tpss_mlp_train(tpss_mlp *m, const float *x, const float *target, int64_t rows, int epochs,
                              int batch, double lr, uint64_t seed, double *loss_per_epoch, void *stream)
{
  return guarded([&] {
    TPSS_REQUIRE(m && x && target && rows >= 1 && epochs >= 0 && batch >= 1 && lr > 0.0,
                 "invalid argument");
    cudaStream_t s = as_stream(stream);
    const int64_t B = std::min<int64_t>(batch, rows);
    if(m->xb.n < (size_t)(B * m->n_in)) m->xb.resize((size_t)(B * m->n_in));
    if(m->yb.n < (size_t)(B * m->n_out)) m->yb.resize((size_t)(B * m->n_out));
    std::vector<int64_t> perm(rows);
    DeviceBuffer<int64_t> dperm(rows);
    uint64_t st = seed;
    for(int ep = 0; ep < epochs; ++ep)
    {
      std::iota(perm.begin(), perm.end(), int64_t(0));
      for(int64_t i = rows - 1; i > 0; --i)  // Fisher-Yates
        std::swap(perm[i], perm[(int64_t)(splitmix(st) % uint64_t(i + 1))]);
      TPSS_CUDA(cudaMemcpyAsync(dperm.ptr, perm.data(), sizeof(int64_t) * rows, cudaMemcpyHostToDevice, s));
      for(int64_t b0 = 0; b0 + B <= rows; b0 += B)
      {
        gather_rows_kernel<<<grid_of(B * m->n_in), 256, 0, s>>>(x, dperm.ptr + b0, B, m->n_in, m->xb.ptr);
        gather_rows_kernel<<<grid_of(B * m->n_out), 256, 0, s>>>(target, dperm.ptr + b0, B, m->n_out, m->yb.ptr);
        mlp_forward(*m, m->xb.ptr, B, s);
        mlp_loss_backward(*m, m->xb.ptr, m->yb.ptr, B, s, false, nullptr);
        ++m->adam_step;
        const float c1 = float(1.0 - std::pow(0.9, double(m->adam_step)));
        const float c2 = float(1.0 - std::pow(0.999, double(m->adam_step)));
        adam_kernel<<<grid_of(m->n_params), 256, 0, s>>>(m->params.ptr, m->grads.ptr, m->adam_m.ptr,
                                                          m->adam_v.ptr, m->n_params, float(lr), c1, c2);
        TPSS_CUDA(cudaGetLastError());
      }
      // perm (pageable host memory) is reshuffled next epoch: wait for its copy and the epoch
      TPSS_CUDA(cudaStreamSynchronize(s));
      if(loss_per_epoch) loss_per_epoch[ep] = mlp_loss_only(*m, x, target, rows, s);
    }
  });
}

extern "C" int tpss_mlp_eval_loss(tpss_mlp *m, const float *x, const float *target, int64_t rows,
                                  double *loss)
{
  return guarded([&] {
    TPSS_REQUIRE(m && x && target && loss && rows >= 1, "invalid argument");
    *loss = mlp_loss_only(*m, x, target, rows, nullptr);
  });
}

extern "C" int tpss_mlp_sizes(const tpss_mlp *m, int *n_in, int *n_out)
{
  return guarded([&] {
    TPSS_REQUIRE(m, "null argument");
    if(n_in) *n_in = m->n_in;
    if(n_out) *n_out = m->n_out;
  });
}

extern "C" void tpss_mlp_destroy(tpss_mlp *m) { delete m; }
