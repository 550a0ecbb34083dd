// mlp.cu -- the learned warm start's network: a dense MLP with GELU hidden layers,
// trained and evaluated by this library's own kernels in FP32.
//
// Layout: one parameter vector P = [W1 (H x I), b1 (H), W2 (H x H), b2 (H),
// W3 (O x H), b3 (O)], row-major weights, and gradient / Adam moments of the same shape.
// Activations are row-major [batch][width].  Every reduction (GEMM inner products,
// bias-gradient column sums, the loss) runs in a fixed order, so training is bitwise
// reproducible for a given seed.
//
// Kernels: one tiled FP32 GEMM with arbitrary operand strides serves the forward pass
// (bias + GELU fused into its epilogue, pre-activations kept for the backward pass; in the
// output layer also the loss and its delta), the weight gradients (A^T B shapes, bias
// gradients as row sums of A) and the back-propagated deltas (GELU' fused).  A layer's weight
// gradient and the delta below it depend on the same delta, so they share a launch: a
// training step is six launches, two gathers and Adam.  One elementwise kernel applies Adam.  GELU is the exact
// erf form, 0.5 x (1 + erf(x / sqrt 2)).
#include "mlp.h"

#include <algorithm>
#include <cmath>
#include <random>
#include <vector>

namespace fg
{
namespace
{

constexpr int kTileM = 16, kTileN = 32;  // output tile
constexpr int kGemmThreads = 512, kGemmWarps = kGemmThreads / 32;
constexpr int kWarpK = 16; // inner dimension per warp
// A CTA of R row tiles: its warps split into R groups, the inner dimension over the warps of a
// group.  Floats of a staged k (16-byte rows), inner dimension staged at a time, bytes.
template <int R> struct GemmShape {
  static constexpr int kRows = R * kTileM, kSplit = kGemmWarps / R, kSlab = kSplit * kWarpK;
  static constexpr int kPitchA = kRows + 4, kPitchB = kTileN + 4;
  static constexpr int kParts = kGemmWarps * (kTileM * kTileN + kTileM); // the warps' tiles and row sums
  static constexpr int kStaged = kSlab * (kPitchA + kPitchB);
  static constexpr size_t kSmem = sizeof(float) * (kStaged > kParts ? kStaged : kParts);
};
constexpr int kThreads = 256;

enum Epilogue : int { kStore = 0, kBiasGelu = 1, kBias = 2, kGeluGrad = 3, kBiasDelta = 4 };

__device__ __forceinline__ float Gelu(float x)
{
  return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
}
__device__ __forceinline__ float GeluGrad(float x)
{
  const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
  return cdf + x * pdf;
}

// C(m, n) = epilogue(sum_k A(m, k) B(k, n)), A(m, k) = A[m * am + k * ak],
// B(k, n) = B[k * bk + n * bn], C row-major with leading dimension ldc.
// kBiasGelu: pre = acc + bias[n] -> aux(m, n) = pre, C = GELU(pre);  kBias: C = acc + bias[n];
// kGeluGrad: C = acc * GELU'(aux(m, n));  kBiasDelta: C = y = acc + bias[n] and, for the
// target t, delta = (y - t) / M and the tile's sum of 0.5 (y - t)^2 in loss[tile].
// row_sum (optional): row_sum[m] = sum_k A(m, k).
struct GemmArgs {
  int M, N, K;
  const float *A;
  int am, ak;
  const float *B;
  int bk, bn;
  float *C;
  int ldc, epilogue;
  const float *bias;
  float *aux;
  const float *target;
  float *delta, *loss, *row_sum;
  int tiles_n, tiles; // set by the launch
};

// Stages X(r, k) = X[r * rs + k * ks], r0 <= r < r0 + ROWS, a slab from k0 on, as
// smem[k][r], zero outside; 16-byte loads along the contiguous direction where aligned.
template <int ROWS, int PITCH, int SLAB>
__device__ __forceinline__ void Stage(float *smem, const float *X, int rs, int ks, int r0, int rows, int k0, int K)
{
  const int slab = min(SLAB, (K - k0 + kWarpK - 1) / kWarpK * kWarpK);
  const bool aligned = (reinterpret_cast<size_t>(X) & 15) == 0;
  if (rs == 1 && ks % 4 == 0 && aligned) {
    for (int t = threadIdx.x; t < slab * (ROWS / 4); t += kGemmThreads) {
      const int k = t / (ROWS / 4), r = t % (ROWS / 4) * 4;
      const float *x = X + static_cast<size_t>(k0 + k) * ks + r0 + r;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k0 + k < K) {
        if (r0 + r + 3 < rows) {
          v = *reinterpret_cast<const float4 *>(x);
        } else {
          v.x = r0 + r < rows ? x[0] : 0.f;
          v.y = r0 + r + 1 < rows ? x[1] : 0.f;
          v.z = r0 + r + 2 < rows ? x[2] : 0.f;
        }
      }
      *reinterpret_cast<float4 *>(smem + k * PITCH + r) = v;
    }
  } else if (ks == 1 && rs % 4 == 0 && aligned) {
    for (int t = threadIdx.x; t < slab / 4 * ROWS; t += kGemmThreads) {
      const int k = t / ROWS * 4, r = t % ROWS;
      const float *x = X + static_cast<size_t>(r0 + r) * rs + k0 + k;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r0 + r < rows) {
        if (k0 + k + 3 < K) {
          v = *reinterpret_cast<const float4 *>(x);
        } else {
          v.x = k0 + k < K ? x[0] : 0.f;
          v.y = k0 + k + 1 < K ? x[1] : 0.f;
          v.z = k0 + k + 2 < K ? x[2] : 0.f;
        }
      }
      smem[k * PITCH + r] = v.x;
      smem[(k + 1) * PITCH + r] = v.y;
      smem[(k + 2) * PITCH + r] = v.z;
      smem[(k + 3) * PITCH + r] = v.w;
    }
  } else {
    for (int t = threadIdx.x; t < slab * ROWS; t += kGemmThreads) {
      const int k = t / ROWS, r = t % ROWS;
      smem[k * PITCH + r] = r0 + r < rows && k0 + k < K
                                ? X[static_cast<size_t>(r0 + r) * rs + static_cast<size_t>(k0 + k) * ks]
                                : 0.f;
    }
  }
}

// One or two independent products per launch: CTA b computes tile b of g, or tile
// b - g.tiles of h; with `loss`, one CTA more sums `count` loss partials.
//
// These products are small (256 x 256 x 256 is 34 MFLOP): latency bounds them -- of the
// launch, of L2 and of each thread's chain -- not FP32 rate.  16 x 32 tiles give a 256 x 256
// output 128 CTAs; a slab of the inner dimension up to 256 is staged at once, every one of 16
// warps multiplies its own 16th of it with 4 x 4 outputs per lane (16 FMAs from two 16-byte
// shared-memory reads), and the 16 partial tiles are added in warp order.  Measured (B200): loss
// and gradient of a 4-256-256-64 network at batch 256 through host buffers 319 -> 111 us, six
// launches of about 5 us and copies.
//
// A short inner dimension (the first layer, narrow networks) has no work for 16 warps: with R > 1
// they take R row tiles instead (RowTiles).  Where R is used, sums and their order are those of
// R = 1.
template <int R>
__global__ void __launch_bounds__(kGemmThreads)
    GemmKernel(GemmArgs g, GemmArgs h, const float *__restrict__ partials, int count, float scale,
               float *__restrict__ loss)
{
  using G = GemmShape<R>;
  extern __shared__ __align__(16) float gemm_smem[];
  __shared__ float red[kGemmWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // Sum over the CTA in a fixed order, valid in thread 0.
  auto block_sum = [&](float v) {
    for (int o = 16; o > 0; o >>= 1)
      v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0)
      red[warp] = v;
    __syncthreads();
    float s = 0.f;
    if (threadIdx.x == 0)
      for (int i = 0; i < kGemmWarps; ++i)
        s += red[i];
    return s;
  };
  int tile = blockIdx.x;
  if (tile >= g.tiles + h.tiles) {
    float s = 0.f;
    for (int i = threadIdx.x; i < count; i += kGemmThreads)
      s += partials[i];
    s = block_sum(s);
    if (threadIdx.x == 0)
      *loss = s * scale;
    return;
  }
  const bool second = tile >= g.tiles;
  if (second)
    tile -= g.tiles;
  const GemmArgs &p = second ? h : g;
  const int m0 = tile / p.tiles_n * G::kRows, n0 = tile % p.tiles_n * kTileN;
  const int part = warp % G::kSplit; // of the inner dimension; the warp's row tile: warp / kSplit
  float *const As = gemm_smem, *const Bs = gemm_smem + G::kSlab * G::kPitchA;
  const int mm = (lane >> 3) * 4, nn = (lane & 7) * 4;
  const bool sums = p.row_sum && n0 == 0;
  float acc[4][4] = {}, sum[4] = {};
  for (int k0 = 0; k0 < p.K; k0 += G::kSlab) {
    if (k0 > 0)
      __syncthreads();
    Stage<G::kRows, G::kPitchA, G::kSlab>(As, p.A, p.am, p.ak, m0, p.M, k0, p.K);
    Stage<kTileN, G::kPitchB, G::kSlab>(Bs, p.B, p.bn, p.bk, n0, p.N, k0, p.K);
    __syncthreads();
    if (k0 + part * kWarpK >= p.K)
      continue;
    const float *a = As + part * kWarpK * G::kPitchA + warp / G::kSplit * kTileM + mm;
    const float *b = Bs + part * kWarpK * G::kPitchB + nn;
#pragma unroll
    for (int k = 0; k < kWarpK; ++k) {
      const float4 av = *reinterpret_cast<const float4 *>(a + k * G::kPitchA);
      const float4 bv = *reinterpret_cast<const float4 *>(b + k * G::kPitchB);
      const float ar[4] = {av.x, av.y, av.z, av.w}, br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          acc[i][j] = fmaf(ar[i], br[j], acc[i][j]);
        sum[i] += ar[i];
      }
    }
  }
  // The warps' partial tiles (and row sums) through shared memory.
  constexpr int kPart = kTileM * kTileN;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4 *>(gemm_smem + warp * kPart + (mm + i) * kTileN + nn) =
        make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  float *const row = gemm_smem + kGemmWarps * kPart;
  if (sums && nn == 0)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      row[warp * kTileM + mm + i] = sum[i];
  __syncthreads();
  if (sums && threadIdx.x < G::kRows && m0 + threadIdx.x < p.M) {
    const float *w0 = row + threadIdx.x / kTileM * G::kSplit * kTileM + threadIdx.x % kTileM;
    float s = 0.f;
    for (int w = 0; w < G::kSplit; ++w)
      s += w0[w * kTileM];
    p.row_sum[m0 + threadIdx.x] = s;
  }
  float l = 0.f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < G::kSplit; ++w)
      v += gemm_smem[(r * G::kSplit + w) * kPart + threadIdx.x];
    const int m = m0 + r * kTileM + static_cast<int>(threadIdx.x) / kTileN;
    const int n = n0 + static_cast<int>(threadIdx.x) % kTileN;
    if (m < p.M && n < p.N) {
      const size_t o = static_cast<size_t>(m) * p.ldc + n;
      if (p.epilogue == kBiasGelu) {
        v += p.bias[n];
        p.aux[o] = v;
        v = Gelu(v);
      } else if (p.epilogue == kBias) {
        v += p.bias[n];
      } else if (p.epilogue == kGeluGrad) {
        v *= GeluGrad(p.aux[o]);
      } else if (p.epilogue == kBiasDelta) {
        v += p.bias[n];
        const float e = v - p.target[o];
        p.delta[o] = e / static_cast<float>(p.M);
        l += 0.5f * e * e;
      }
      p.C[o] = v;
    }
  }
  if (p.epilogue == kBiasDelta) {
    l = block_sum(l);
    if (threadIdx.x == 0)
      p.loss[tile] = l;
  }
}
static_assert(kTileM * kTileN == kGemmThreads, "one output per thread in the epilogue");

__global__ void GatherRowsKernel(int rows, int width, const int32_t *__restrict__ index,
                                 const float *__restrict__ src, float *__restrict__ dst)
{
  const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= static_cast<size_t>(rows) * width)
    return;
  const int r = static_cast<int>(t / width), c = static_cast<int>(t % width);
  dst[t] = src[static_cast<size_t>(index[r]) * width + c];
}

// Adam (Kingma & Ba 2015) with bias correction folded into the step size.
__global__ void AdamKernel(int64_t n, float *__restrict__ p, const float *__restrict__ g,
                           float *__restrict__ m, float *__restrict__ v, float lr_t, float beta1,
                           float beta2, float eps)
{
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const float gi = g[i];
  const float mi = beta1 * m[i] + (1.f - beta1) * gi;
  const float vi = beta2 * v[i] + (1.f - beta2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr_t * mi / (sqrtf(vi) + eps);
}

unsigned Grid(size_t threads, int block) { return static_cast<unsigned>((threads + block - 1) / block); }

GemmArgs Product(int M, int N, int K, const float *A, int am, int ak, const float *B, int bk, int bn, float *C,
                 int ldc, int epilogue, const float *bias = nullptr, float *aux = nullptr)
{
  GemmArgs g{M, N, K, A, am, ak, B, bk, bn, C, ldc, epilogue, bias, aux, nullptr, nullptr, nullptr, nullptr, 0, 0};
  g.tiles_n = (N + kTileN - 1) / kTileN;
  g.tiles = g.tiles_n * ((M + kTileM - 1) / kTileM);
  return g;
}

template <int R>
cudaError_t LaunchGemm(GemmArgs g, const GemmArgs &h, cudaStream_t st, const float *partials = nullptr, int count = 0,
                       float scale = 0.f, float *loss = nullptr)
{
  g.tiles = g.tiles_n * ((g.M + GemmShape<R>::kRows - 1) / GemmShape<R>::kRows);
  GemmKernel<R><<<g.tiles + h.tiles + (loss ? 1 : 0), kGemmThreads, GemmShape<R>::kSmem, st>>>(g, h, partials, count,
                                                                                              scale, loss);
  return cudaGetLastError();
}

// Row tiles per CTA of a single product whose epilogue writes no sums: the fewest that leave one
// wave (two CTAs per SM, by registers) and a part of the inner dimension to every warp.  A CTA per
// tile and two to seven waves of them were slower than 32 x 32 tiles of 256 threads at narrow
// widths.  Forward pass through host buffers, us: 32 x 32 tiles, a CTA per tile, by this rule:
//   4-32-32-4:     8,192 rows  57  68  59,   32,768 rows 132 172 132
//   4-48-48-8:     4,096 rows  52  63  53,   32,768 rows 189 250 182
//   4-128-128-16:  4,096 rows  96  88  75,   32,768 rows 455 447 320
int RowTiles(const GemmArgs &g)
{
  constexpr int kWave = 2 * 148;
  int tiles = 1;
  if (g.epilogue == kBiasGelu || g.epilogue == kBias)
    for (const int r : {2, 4, 16})
      if (g.K <= kGemmWarps / r * kWarpK && g.tiles > kWave * tiles)
        tiles = r;
  return tiles;
}

// g and optionally h (h.tiles = 0: none); with loss, also the sum of `count` partials.
cudaError_t Gemm(const GemmArgs &g, const GemmArgs &h, cudaStream_t st, const float *partials = nullptr,
                 int count = 0, float scale = 0.f, float *loss = nullptr)
{
  if (h.tiles == 0 && !loss)
    switch (RowTiles(g)) {
    case 16: return LaunchGemm<16>(g, h, st);
    case 4: return LaunchGemm<4>(g, h, st);
    case 2: return LaunchGemm<2>(g, h, st);
    }
  return LaunchGemm<1>(g, h, st, partials, count, scale, loss);
}

} // namespace

Status Mlp::Create(int inputs, int hidden, int outputs, uint64_t seed)
{
  if (inputs < 1 || hidden < 1 || outputs < 1 || inputs > 4096 || hidden > 4096 || outputs > 4096)
    return Status::kInvalidArgument;
  I_ = inputs;
  H_ = hidden;
  O_ = outputs;
  const int64_t n = ParameterCount();
  Status s;
  if ((s = p_.ensure(n)) != Status::kOk || (s = g_.ensure(n + 1)) != Status::kOk ||
      (s = m_.ensure(n)) != Status::kOk || (s = v_.ensure(n)) != Status::kOk)
    return s;
  if (cudaFuncSetAttribute(GemmKernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(GemmShape<1>::kSmem)) != cudaSuccess) {
    cudaGetLastError();
    return Status::kInternalError;
  }
  // Uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights and biases from a seeded generator.
  std::mt19937_64 rng(seed);
  std::vector<float> host(n);
  size_t o = 0;
  auto fill = [&](int rows, int fan_in) {
    std::uniform_real_distribution<float> u(-1.0f / std::sqrt(float(fan_in)), 1.0f / std::sqrt(float(fan_in)));
    for (int i = 0; i < rows * fan_in; ++i)
      host[o++] = u(rng);
    for (int i = 0; i < rows; ++i)
      host[o++] = u(rng);
  };
  fill(H_, I_);
  fill(H_, H_);
  fill(O_, H_);
  if ((s = p_.upload(host.data(), n)) != Status::kOk)
    return s;
  steps_ = 0;
  return cudaMemset(m_.get(), 0, n * sizeof(float)) == cudaSuccess &&
                 cudaMemset(v_.get(), 0, n * sizeof(float)) == cudaSuccess &&
                 cudaDeviceSynchronize() == cudaSuccess
             ? Status::kOk
             : Status::kInternalError;
}

int64_t Mlp::ParameterCount() const
{
  return static_cast<int64_t>(H_) * I_ + H_ + static_cast<int64_t>(H_) * H_ + H_ +
         static_cast<int64_t>(O_) * H_ + O_;
}

Status Mlp::EnsureBatch(int batch)
{
  if (batch <= batch_cap_)
    return Status::kOk;
  Status s;
  const size_t b = batch;
  if ((s = x_.ensure(b * I_)) != Status::kOk || (s = t_.ensure(b * O_)) != Status::kOk ||
      (s = h1_.ensure(b * H_)) != Status::kOk || (s = a1_.ensure(b * H_)) != Status::kOk ||
      (s = h2_.ensure(b * H_)) != Status::kOk || (s = a2_.ensure(b * H_)) != Status::kOk ||
      (s = y_.ensure(b * O_)) != Status::kOk || (s = dy_.ensure(b * O_)) != Status::kOk ||
      (s = d2_.ensure(b * H_)) != Status::kOk || (s = d1_.ensure(b * H_)) != Status::kOk ||
      (s = row_loss_.ensure(static_cast<size_t>((batch + kTileM - 1) / kTileM) * ((O_ + kTileN - 1) / kTileN))) !=
          Status::kOk)
    return s;
  batch_cap_ = batch;
  return Status::kOk;
}

// Pointers into the parameter-shaped vector q (P, G or a moment).
Mlp::Views Mlp::Split(float *q) const
{
  Views v;
  v.w1 = q;
  v.b1 = v.w1 + static_cast<size_t>(H_) * I_;
  v.w2 = v.b1 + H_;
  v.b2 = v.w2 + static_cast<size_t>(H_) * H_;
  v.w3 = v.b2 + H_;
  v.b3 = v.w3 + static_cast<size_t>(O_) * H_;
  return v;
}

// y = f(x) for `batch` rows of x (device), keeping pre-activations for Backward; with a
// target also dy_ and the partials of the loss.
Status Mlp::Forward(int batch, const float *x, float *y, cudaStream_t st, const float *target)
{
  const Views w = Split(p_.get());
  const GemmArgs none{};
  // h1 = GELU(x W1^T + b1): A = x [b][i], B(k=i, n=h) = W1[h][i].
  GemmArgs out = Product(batch, O_, H_, a2_.get(), H_, 1, w.w3, 1, H_, y, O_, target ? kBiasDelta : kBias, w.b3);
  out.target = target;
  out.delta = dy_.get();
  out.loss = row_loss_.get();
  if (Gemm(Product(batch, H_, I_, x, I_, 1, w.w1, 1, I_, a1_.get(), H_, kBiasGelu, w.b1, h1_.get()), none, st) !=
          cudaSuccess ||
      Gemm(Product(batch, H_, H_, a1_.get(), H_, 1, w.w2, 1, H_, a2_.get(), H_, kBiasGelu, w.b2, h2_.get()), none,
           st) != cudaSuccess ||
      Gemm(out, none, st) != cudaSuccess)
    return Status::kInternalError;
  loss_partials_ = out.tiles;
  launches_ += 3;
  return Status::kOk;
}

// Gradient of 0.5 / batch * sum (y - t)^2 into g_ and the loss behind it, after
// Forward(x, y_, t).
Status Mlp::Backward(int batch, const float *x, cudaStream_t st)
{
  const Views w = Split(p_.get());
  const Views g = Split(g_.get());
  // dW3 = dy^T a2 (O x H), db3 = colsum(dy) | d2 = (dy W3) * GELU'(h2); dW2 = d2^T a1, db2 |
  // d1 = (d2 W2) * GELU'(h1); dW1 = d1^T x, db1 | the loss.
  GemmArgs w3 = Product(O_, H_, batch, dy_.get(), 1, O_, a2_.get(), H_, 1, g.w3, H_, kStore);
  GemmArgs w2 = Product(H_, H_, batch, d2_.get(), 1, H_, a1_.get(), H_, 1, g.w2, H_, kStore);
  GemmArgs w1 = Product(H_, I_, batch, d1_.get(), 1, H_, x, I_, 1, g.w1, I_, kStore);
  w3.row_sum = g.b3;
  w2.row_sum = g.b2;
  w1.row_sum = g.b1;
  if (Gemm(Product(batch, H_, O_, dy_.get(), O_, 1, w.w3, H_, 1, d2_.get(), H_, kGeluGrad, nullptr, h2_.get()), w3,
           st) != cudaSuccess ||
      Gemm(Product(batch, H_, H_, d2_.get(), H_, 1, w.w2, H_, 1, d1_.get(), H_, kGeluGrad, nullptr, h1_.get()), w2,
           st) != cudaSuccess ||
      Gemm(w1, GemmArgs{}, st, row_loss_.get(), loss_partials_, 1.0f / batch, Loss()) != cudaSuccess)
    return Status::kInternalError;
  launches_ += 3;
  return Status::kOk;
}

Status Mlp::Predict(int batch, const float *x_host, float *y_host)
{
  if (batch < 1 || !x_host || !y_host)
    return Status::kInvalidArgument;
  Status s = EnsureBatch(batch);
  if (s != Status::kOk || (s = x_.upload(x_host, static_cast<size_t>(batch) * I_)) != Status::kOk ||
      (s = Forward(batch, x_.get(), y_.get(), nullptr)) != Status::kOk)
    return s;
  return cudaMemcpy(y_host, y_.get(), sizeof(float) * batch * O_, cudaMemcpyDeviceToHost) == cudaSuccess
             ? Status::kOk
             : Status::kInternalError;
}

Status Mlp::PredictDevice(int batch, const float *x_dev, float *y_dev, cudaStream_t st)
{
  Status s = EnsureBatch(batch);
  if (s != Status::kOk)
    return s;
  return Forward(batch, x_dev, y_dev, st);
}

Status Mlp::LossGradient(int batch, const float *x_host, const float *t_host, float *loss,
                         float *gradient_host)
{
  if (batch < 1 || !x_host || !t_host)
    return Status::kInvalidArgument;
  Status s = EnsureBatch(batch);
  if (s != Status::kOk || (s = x_.upload(x_host, static_cast<size_t>(batch) * I_)) != Status::kOk ||
      (s = t_.upload(t_host, static_cast<size_t>(batch) * O_)) != Status::kOk ||
      (s = Forward(batch, x_.get(), y_.get(), nullptr, t_.get())) != Status::kOk ||
      (s = Backward(batch, x_.get(), nullptr)) != Status::kOk)
    return s;
  // A caller that keeps the loss behind the gradient gets both in one copy.  (The copy waits
  // about 10 us; the loss through pinned memory saved one too, but pinning cost the first call of
  // every network 1 to 5 ms.)
  const size_t n = static_cast<size_t>(ParameterCount());
  if (loss && gradient_host && loss == gradient_host + n)
    return cudaMemcpy(gradient_host, g_.get(), sizeof(float) * (n + 1), cudaMemcpyDeviceToHost) == cudaSuccess
               ? Status::kOk
               : Status::kInternalError;
  if (loss && cudaMemcpy(loss, Loss(), sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess)
    return Status::kInternalError;
  if (gradient_host && cudaMemcpy(gradient_host, g_.get(), sizeof(float) * n, cudaMemcpyDeviceToHost) != cudaSuccess)
    return Status::kInternalError;
  return Status::kOk;
}

Status Mlp::Train(int samples, const float *x_host, const float *t_host, int epochs, int batch,
                  float learning_rate, uint64_t seed, float *final_loss)
{
  if (samples < 1 || epochs < 0 || batch < 1 || !x_host || !t_host || !(learning_rate > 0.f))
    return Status::kInvalidArgument;
  batch = std::min(batch, samples);
  Status s = EnsureBatch(std::max(batch, samples));
  DeviceArray<float> xs, ts;
  DeviceArray<int32_t> perm;
  if (s != Status::kOk || (s = xs.upload(x_host, static_cast<size_t>(samples) * I_)) != Status::kOk ||
      (s = ts.upload(t_host, static_cast<size_t>(samples) * O_)) != Status::kOk ||
      (s = perm.ensure(samples)) != Status::kOk)
    return s;
  std::mt19937_64 rng(seed);
  std::vector<int32_t> order(samples);
  constexpr float kBeta1 = 0.9f, kBeta2 = 0.999f, kEps = 1e-8f;
  const int64_t n = ParameterCount();
  for (int epoch = 0; epoch < epochs; ++epoch) {
    for (int i = 0; i < samples; ++i)
      order[i] = i;
    std::shuffle(order.begin(), order.end(), rng);
    if ((s = perm.upload(order.data(), samples)) != Status::kOk)
      return s;
    for (int first = 0; first + batch <= samples; first += batch) {
      GatherRowsKernel<<<Grid(static_cast<size_t>(batch) * I_, kThreads), kThreads>>>(
          batch, I_, perm.get() + first, xs.get(), x_.get());
      GatherRowsKernel<<<Grid(static_cast<size_t>(batch) * O_, kThreads), kThreads>>>(
          batch, O_, perm.get() + first, ts.get(), t_.get());
      if (cudaGetLastError() != cudaSuccess ||
          (s = Forward(batch, x_.get(), y_.get(), nullptr, t_.get())) != Status::kOk ||
          (s = Backward(batch, x_.get(), nullptr)) != Status::kOk)
        return s != Status::kOk ? s : Status::kInternalError;
      ++steps_;
      const double c1 = 1.0 - std::pow(double(kBeta1), double(steps_));
      const double c2 = 1.0 - std::pow(double(kBeta2), double(steps_));
      const float lr_t = static_cast<float>(learning_rate * std::sqrt(c2) / c1);
      AdamKernel<<<Grid(n, kThreads), kThreads>>>(n, p_.get(), g_.get(), m_.get(), v_.get(), lr_t,
                                                  kBeta1, kBeta2, kEps);
      if (cudaGetLastError() != cudaSuccess)
        return Status::kInternalError;
      launches_ += 3;
    }
  }
  // Loss over the whole training set with the final parameters.
  if ((s = Forward(samples, xs.get(), y_.get(), nullptr, ts.get())) != Status::kOk ||
      (s = Backward(samples, xs.get(), nullptr)) != Status::kOk)
    return s;
  if (cudaDeviceSynchronize() != cudaSuccess)
    return Status::kInternalError;
  if (final_loss && cudaMemcpy(final_loss, Loss(), sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess)
    return Status::kInternalError;
  return Status::kOk;
}

Status Mlp::GetParameters(float *host) const
{
  return cudaMemcpy(host, p_.get(), sizeof(float) * ParameterCount(), cudaMemcpyDeviceToHost) == cudaSuccess
             ? Status::kOk
             : Status::kInternalError;
}

Status Mlp::SetParameters(const float *host)
{
  Status s = p_.upload(host, ParameterCount());
  if (s != Status::kOk)
    return s;
  return cudaDeviceSynchronize() == cudaSuccess ? Status::kOk : Status::kInternalError;
}

} // namespace fg
