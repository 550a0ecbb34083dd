// postprocess_kernel.cu -- device form of the frozen postprocess in one launch: the
// weighted-stress force and torque of every item (force CTAs) and the smoothed radial air-gap
// B of every (item, probe) from the probe corners' recipes (probe CTAs).  Both write to
// pinned host memory.
//
// The probe arithmetic uses explicitly rounded operations (no fused multiply-add) in the
// host smoothing's order, so the samples equal the host form's bit for bit; the sharp-corner
// fallback's |B| uses the device hypot.
#include "postprocess.h"

namespace fg
{
namespace
{

constexpr int kThreads = 256;
constexpr int kSms = 148;
constexpr int kPerThread = 2; // elements per thread of a force CTA, at least
constexpr double kInvTwoMu0 = 1.0 / (2.0 * 4.0e-7 * 3.141592653589793238462643383279502884);

// Items a force CTA takes together: an element's geometry is read once for all of them.
__host__ __device__ constexpr int ItemsTogether(int items) { return items > 2 ? 4 : (items > 1 ? 2 : 1); }

// Nodal B of one probe corner, in the host smoothing's operation order.  Term indices are
// loaded ahead of the values they address (two dependent hops per batch of terms, not two per
// term); the accumulation order stays the host's.
__device__ void Corner(const PostprocessDevice &p, const CornerStencil &c, const double *a,
                       const double *b1, const double *b2, double *nbx, double *nby)
{
  constexpr int kBatch = 8;
  double x = 0.0, y = 0.0;
  if (c.kind == 0 || c.kind == 3) {
    double largest = 0.0;
    for (int t0 = c.first; t0 < c.first + c.count; t0 += kBatch) {
      int e[kBatch];
      double v1[kBatch], v2[kBatch];
#pragma unroll
      for (int j = 0; j < kBatch; ++j)
        e[j] = t0 + j < c.first + c.count ? p.term_elem[t0 + j] : -1;
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        v1[j] = e[j] >= 0 ? b1[e[j]] : 0.0;
        v2[j] = e[j] >= 0 ? b2[e[j]] : 0.0;
      }
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (e[j] < 0)
          break;
        if (c.kind == 0) {
          const double w = p.term_w[t0 + j];
          x = __dadd_rn(x, __dmul_rn(w, v1[j]));
          y = __dadd_rn(y, __dmul_rn(w, v2[j]));
        } else {
          largest = fmax(largest, hypot(v1[j], v2[j]));
        }
      }
    }
    if (c.kind == 0) {
      x = __ddiv_rn(x, c.wsum);
      y = __ddiv_rn(y, c.wsum);
    } else {
      const double o1 = b1[c.element], o2 = b2[c.element];
      const double own = hypot(o1, o2);
      x = own > 0.0 ? __ddiv_rn(__dmul_rn(largest, o1), own) : 0.0;
      y = own > 0.0 ? __ddiv_rn(__dmul_rn(largest, o2), own) : 0.0;
    }
  } else if (c.kind == 1) {
    const double an = a[c.node];
    for (int t = c.first; t < c.first + c.count; ++t) {
      const int e = p.term_elem[t];
      const double tx = p.term_tx[t], ty = p.term_ty[t], w = p.term_w[t];
      const double bt = __dadd_rn(__dmul_rn(b1[e], tx), __dmul_rn(b2[e], ty));
      const double bn = __ddiv_rn(__dsub_rn(a[p.term_node[t]], an), p.term_len[t]);
      x = __dadd_rn(x, __dmul_rn(w, __dadd_rn(__dmul_rn(tx, bt), __dmul_rn(ty, bn))));
      y = __dadd_rn(y, __dmul_rn(w, __dsub_rn(__dmul_rn(ty, bt), __dmul_rn(tx, bn))));
    }
    x = __ddiv_rn(x, c.wsum);
    y = __ddiv_rn(y, c.wsum);
  } else {
    x = b1[c.element];
    y = b2[c.element];
  }
  *nbx = x;
  *nby = y;
}

// Force and torque of IT items over a contiguous element range, per CTA; the last CTA of an
// item group to finish adds the CTAs' partials in order.
//
// Bound by reading B once (16 bytes per element and item).  One item per CTA read the 40
// bytes of geometry again for every item, two and a half times B's own bytes, through L2:
// 14.4 us for 80,000 elements and 32 items.  Weight and centroid are only needed where the
// mask has a gradient (some hundred elements); the products with B are taken everywhere, so
// that a field that is not finite still shows in the sums.  With four items together, force,
// probes and the results' way to the host in one launch: 19.5 us from cold caches, against 14.4 +
// 5.4 us and a copy; the whole call 57.6 -> 34.4 us (32 items), 36 -> 22 us (one).
template <int IT> __device__ void ForceCta(const PostprocessDevice &p, int cta, int group)
{
  __shared__ double scratch[kThreads / 32][3 * IT];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int item0 = group * IT, count = min(IT, p.items - item0);
  const int64_t chunk = (static_cast<int64_t>(p.E) + p.ctas - 1) / p.ctas;
  const int64_t first = chunk * cta, end = min(first + chunk, static_cast<int64_t>(p.E));
  double f[3][IT] = {};
  constexpr int G = 3; // elements whose loads are issued together
  for (int64_t base = first + threadIdx.x; base < end; base += G * kThreads) {
    double hx[G], hy[G], bx[G][IT], by[G][IT];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int64_t e = base + g * kThreads;
      const bool in = e < end;
      hx[g] = in ? __ldg(p.hx + e) : 0.0;
      hy[g] = in ? __ldg(p.hy + e) : 0.0;
#pragma unroll
      for (int i = 0; i < IT; ++i) {
        bx[g][i] = in && i < count ? __ldcs(p.b1 + static_cast<int64_t>(item0 + i) * p.E + e) : 0.0;
        by[g][i] = in && i < count ? __ldcs(p.b2 + static_cast<int64_t>(item0 + i) * p.E + e) : 0.0;
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int64_t e = base + g * kThreads;
      double w = 1.0, cx = 0.0, cy = 0.0;
      if (hx[g] != 0.0 || hy[g] != 0.0) {
        w = __ldg(p.weight + e);
        cx = __ldg(p.cx + e);
        cy = __ldg(p.cy + e);
      }
#pragma unroll
      for (int i = 0; i < IT; ++i) {
        const double x = bx[g][i], y = by[g][i];
        const double fxd = ((x * x - y * y) * hx[g] + 2.0 * x * y * hy[g]) * kInvTwoMu0;
        const double fyd = (2.0 * x * y * hx[g] + (y * y - x * x) * hy[g]) * kInvTwoMu0;
        f[0][i] += w * fxd;
        f[1][i] += w * fyd;
        f[2][i] += w * (cx * fyd - cy * fxd);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 3; ++q)
#pragma unroll
    for (int i = 0; i < IT; ++i) {
      for (int o = 16; o > 0; o >>= 1)
        f[q][i] += __shfl_xor_sync(0xffffffffu, f[q][i], o);
      if (lane == 0)
        scratch[warp][3 * i + q] = f[q][i];
    }
  __syncthreads();
  double *const part = p.partials + static_cast<int64_t>(group) * p.ctas * 3 * IT;
  if (threadIdx.x < 3 * IT) {
    double s = 0.0;
    for (int w = 0; w < kThreads / 32; ++w)
      s += scratch[w][threadIdx.x];
    part[static_cast<int64_t>(cta) * 3 * IT + threadIdx.x] = s;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned before = atomicAdd(p.arrived + group, 1u);
    last = before == static_cast<unsigned>(p.ctas) - 1u;
    if (last)
      p.arrived[group] = 0; // for the next launch
  }
  __syncthreads();
  if (!last)
    return;
  __threadfence();
  // A warp per quantity: lanes stride the CTAs' partials, then a fixed tree.
  for (int t = warp; t < 3 * count; t += kThreads / 32) {
    double s = 0.0;
    for (int c = lane; c < p.ctas; c += 32)
      s += __ldcg(part + static_cast<int64_t>(c) * 3 * IT + t);
    for (int o = 16; o > 0; o >>= 1)
      s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0)
      p.sums[3 * item0 + t] = s;
  }
}

// Air-gap samples: four lanes per (item, probe), lanes 0-2 one corner each; lane 0
// combines the corners in the host's order.
__device__ void ProbeCta(const PostprocessDevice &p, int cta)
{
  const int64_t t = static_cast<int64_t>(cta) * kThreads + threadIdx.x;
  const int64_t sample = t >> 2;
  const int l = static_cast<int>(t & 3);
  const bool live = sample < static_cast<int64_t>(p.probes) * p.items;
  double nbx = 0.0, nby = 0.0;
  int item = 0, k = 0;
  if (live) {
    item = static_cast<int>(sample / p.probes);
    k = static_cast<int>(sample % p.probes);
    if (l < 3)
      Corner(p, p.corners[3 * k + l], p.a + static_cast<int64_t>(item) * p.N,
             p.b1 + static_cast<int64_t>(item) * p.E, p.b2 + static_cast<int64_t>(item) * p.E, &nbx, &nby);
  }
  double cx[3], cy[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    cx[j] = __shfl_sync(0xffffffffu, nbx, (threadIdx.x & ~3) + j);
    cy[j] = __shfl_sync(0xffffffffu, nby, (threadIdx.x & ~3) + j);
  }
  if (!live || l != 0)
    return;
  const double *pr = p.probe + 5 * k;
  double bx = 0.0, by = 0.0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    bx = __dadd_rn(bx, __dmul_rn(pr[j], cx[j]));
    by = __dadd_rn(by, __dmul_rn(pr[j], cy[j]));
  }
  p.radial[sample] = __dadd_rn(__dmul_rn(bx, pr[3]), __dmul_rn(by, pr[4]));
}

template <int IT> __global__ void __launch_bounds__(kThreads, 2) PostprocessKernel(PostprocessDevice p)
{
  // The probe CTAs (chains of dependent gathers) first.
  const int probes = static_cast<int>((4 * static_cast<int64_t>(p.probes) * p.items + kThreads - 1) / kThreads);
  const int b = static_cast<int>(blockIdx.x) - probes;
  if (b < 0)
    ProbeCta(p, b + probes);
  else
    ForceCta<IT>(p, b % p.ctas, b / p.ctas);
}

} // namespace

int PostprocessGroups(int32_t items) { return (items + ItemsTogether(items) - 1) / ItemsTogether(items); }

size_t PostprocessPartials(int32_t E, int32_t items)
{
  return static_cast<size_t>(PostprocessGroups(items)) * PostprocessCtas(E, items) * 3 * ItemsTogether(items);
}

int PostprocessCtas(int32_t E, int32_t items)
{
  // One wave: two resident CTAs per SM over all (range, item group) CTAs, and at least
  // kPerThread elements per thread.
  const int64_t by_size = (static_cast<int64_t>(E) + kPerThread * kThreads - 1) / (kPerThread * kThreads);
  const int64_t by_wave = (2 * kSms - kSms / 4) / PostprocessGroups(items > 0 ? items : 1); // room for the probes
  const int64_t want = by_size > by_wave ? by_wave : by_size;
  return static_cast<int>(want < 1 ? 1 : want);
}

cudaError_t LaunchPostprocess(const PostprocessDevice &p, cudaStream_t stream)
{
  if (p.items < 1 || p.items > 65535)
    return cudaErrorInvalidValue;
  const int64_t lanes = 4 * static_cast<int64_t>(p.probes) * p.items;
  const unsigned ctas = static_cast<unsigned>(PostprocessGroups(p.items) * static_cast<int64_t>(p.ctas) +
                                              (lanes + kThreads - 1) / kThreads);
  switch (ItemsTogether(p.items)) {
  case 1: PostprocessKernel<1><<<ctas, kThreads, 0, stream>>>(p); break;
  case 2: PostprocessKernel<2><<<ctas, kThreads, 0, stream>>>(p); break;
  default: PostprocessKernel<4><<<ctas, kThreads, 0, stream>>>(p); break;
  }
  return cudaGetLastError();
}

} // namespace fg
