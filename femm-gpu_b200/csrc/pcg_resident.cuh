// pcg_resident.cuh -- the FP64 Jacobi PCG with a CTA's share of the problem kept on chip.
//
// The algorithm, the partition (rows -> row groups -> warps -> lanes), every operation and
// every summation order are PcgBody's (pcg_kernel.cuh), so the results are the same bits;
// what differs is where the data lives and how the CTAs agree.  For launches of at most one
// row group per SM: then a warp has at most one warp-step, so a lane owns one row (for IV
// items) in both phases of a CG iteration.
//
// * x, r, q, the row's own direction p and the inverse diagonal stay in registers; the
//   operator's values and columns in shared memory.
// * Beside each operator entry sits the direction p_j of the entry's column: every reader
//   evaluates p_j = z_j + beta p_j itself, so z is the only vector that crosses CTAs.
// * There is no grid barrier in the CG loop.  Partial sums, their results and z are
//   messages whose arrival is their validity: a slot holds kUnset until it is written.  A
//   message costs one trip through L2 (about 0.4 us with its poll); a barrier costs that
//   for the data to become visible, again for the counter and again for the partials.
// * Warp 0 does the talking.  Once the warps have left their sums in shared memory it sends
//   them, sums what others sent and takes the scalar decisions; meanwhile the other warps
//   already gather the z of the next iteration, whose messages left their owners before the
//   partial sums did.
//
// Small systems are bound by latency: a CG iteration of PcgBody is six dependent L2 round
// trips in phase A (row length, column, two chunks of values and gathers, own row) and three
// per reduction.  Measured on a B200, microseconds per CG iteration, PcgBody -> here:
//   rows      961: 1 item  9.1 -> 4.5, 8 items 11.7 -> 6.4, 32 items 16.9 -> 9.2
//   rows    3,969: 1 item  8.8 -> 4.2, 8 items 11.9 -> 8.3, 32 items 16.9 -> 8.7
//   rows   16,129: 1 item  8.8 -> 4.4, 8 items 12.4 -> 8.9
//   rows   62,001: 1 item  9.0 -> 6.0, 2 items 10.8 -> 8.0
// What is left is messages: two trips through L2 per reduction (one with few partials) and
// the decisions between them.
//
// Message slots are reused, so a slot has to be seen unset (kUnset) before it is written
// again.  All of an iteration i's resets are issued in its phase B, by the CTA that reads
// the slot (mailboxes) or owns it (z).  Once per iteration, while its sums of phase A travel,
// warp 0 executes one acquire-release fence: every message it sends later releases what its
// CTA had stored before, and everything it polled before is acquired.  So a reset in phase B
// of i is released by the CTA's messages from phase B of i + 1 on, acquired by an item's
// warp with the fence of i + 2, passed on with its result in phase B of i + 2 and acquired
// by every CTA with the fence of i + 3 (one step sooner without results): it is in force for
// the messages of phase B of i + 3 and later, and for the z gathered there for iteration
// i + 4.  Hence four z buffers and eight mailbox buffers.  (The fence costs 0.4 us; beside
// the travelling sums it is nearly free.)
#pragma once

#include "pcg_kernel.cuh"

namespace fg
{
namespace
{

constexpr int kMailboxes = 8; // mailbox buffers, by reduction index
constexpr int kDirect = 64;   // partials every CTA may sum itself

// An unwritten message: a NaN pattern that is never sent.
constexpr unsigned long long kUnset = 0xffffffffffffffffull;

// (Its upper half is enough: Sendable keeps it out of every message.)
__device__ __forceinline__ bool Unset(double v) { return __double2hiint(v) == -1; }
__device__ __forceinline__ double UnsetValue() { return __longlong_as_double(static_cast<long long>(kUnset)); }
__device__ __forceinline__ double Sendable(double v) { return Unset(v) ? static_cast<double>(NAN) : v; }
__device__ __forceinline__ void FenceAcqRel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// A lane's IV consecutive doubles of a message.
template <int IV> __device__ __forceinline__ void LoadMessage(const double *p, double (&o)[IV])
{
  if constexpr (IV == 2)
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(o[0]), "=d"(o[1]) : "l"(p) : "memory");
  else
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(o[0]) : "l"(p) : "memory");
}
template <int IV> __device__ __forceinline__ void StoreMessage(double *p, const double (&v)[IV])
{
  if constexpr (IV == 2)
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v[0]), "d"(v[1]) : "memory");
  else
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v[0]) : "memory");
}
template <int IV> __device__ __forceinline__ bool Missing(const double (&v)[IV]) { return Unset(v[0]) || Unset(v[IV - 1]); }

template <int ID> __device__ __forceinline__ void NamedArrive()
{
  asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(kPcgThreads) : "memory");
}
template <int ID> __device__ __forceinline__ void NamedSync()
{
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(kPcgThreads) : "memory");
}

// GV: row groups per CTA.
template <int KP, int GV> struct ResidentShared {
  double warp[kPcgWarps * GV][2 * KP]; // the warps' sums, row group by row group
  int err;    // GridBarrier's
  int failed; // a wait for a message ran out
  // What the CTA goes on with after a reduction: the active items, and kStop (a wait ran out)
  // or kThreshold (an item is at its threshold).
  uint2 state;
};
constexpr unsigned kStop = 1, kThreshold = 2;

// A poll of a bounded wait failed: false when the wait has run out or another CTA failed
// (looked for on every 16th poll).
template <class R>
__device__ __forceinline__ bool PollAgain(const PcgArgs &a, unsigned &spin, unsigned long long t0, R &sm)
{
  const bool other = (spin & 15u) == 15u && *reinterpret_cast<volatile int32_t *>(a.error) != 0;
  const bool expired = GlobalTimer() - t0 > static_cast<unsigned long long>(a.timeout_ns);
  ++spin;
  if (!other && !expired)
    return true;
  if (!other)
    atomicExch(a.error, 2);
  *const_cast<volatile int *>(&sm.failed) = 1;
  return false;
}

// A warp's part of Q per-item sums (or maxima); place: row group in the CTA x kPcgWarps + the
// group's warp whose rows they are.
template <int KP, int IV, int GV, int Q, bool kMax>
__device__ __forceinline__ void WarpPart(double (&v)[Q][IV], int place, ResidentShared<KP, GV> &sm)
{
  constexpr int LR = KP / IV;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int off = 16; off >= LR; off >>= 1)
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int j = 0; j < IV; ++j) {
        const double y = __shfl_xor_sync(0xffffffffu, v[q][j], off);
        v[q][j] = kMax ? fmax(v[q][j], y) : v[q][j] + y;
      }
  if (lane < LR)
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int j = 0; j < IV; ++j)
        sm.warp[place][q * KP + lane * IV + j] = v[q][j];
}

// The mailboxes behind a.partials: after the two buffers of the barrier-based reductions
// (set-up, verification), kMailboxes x (partials, results); a partial is two doubles per
// (item, row group).  The CTA that owns an item (CTA = item) sums its partials and sends the
// result to every CTA, in lines of its own: 148 CTAs polling one line would slow its writer
// down.  With at most kDirect slots (row groups rounded up to a power of two) there are no
// results: every CTA reads all partials.
template <int KP> struct Mailboxes {
  double *base;
  int G, ctas, padded; // row groups, CTAs, row groups rounded up to a power of two
  bool direct;
  unsigned results, stride; // doubles before a buffer's results, and of a whole buffer
  static constexpr int kLine = 2 * KP > 16 ? 2 * KP : 16;
  __device__ __forceinline__ void Init(const PcgArgs &a, int ctas_)
  {
    ctas = ctas_;
    base = a.partials + static_cast<size_t>(2) * 2 * KP * a.row_groups;
    G = a.row_groups;
    padded = 1;
    while (padded < G)
      padded <<= 1;
    direct = ctas == G && KP * padded <= kDirect;
    results = static_cast<unsigned>(KP * G * 2);
    stride = results + static_cast<unsigned>(ctas * kLine);
  }
  __device__ __forceinline__ double *Buffer(int r) const
  {
    return base + static_cast<size_t>(static_cast<unsigned>(r & (kMailboxes - 1)) * stride);
  }
  __device__ __forceinline__ double *Partial(int r, int it, int g) const { return Buffer(r) + (it * G + g) * 2; }
  __device__ __forceinline__ double *Result(int r, int c, int it) const { return Buffer(r) + results + c * kLine + 2 * it; }
  // CTA c's resets of reduction r's buffer: its own partials (direct), or the partials of its
  // items and its line of results.  Thread t of n.
  __device__ __forceinline__ void Reset(int r, int c, int t, int n) const
  {
    const double unset[2] = {UnsetValue(), UnsetValue()};
    if (direct) {
      for (int it = t; it < KP; it += n)
        StoreMessage<2>(Partial(r, it, c), unset);
    } else {
      for (int it = c; it < KP; it += ctas)
        for (int g = t; g < G; g += n)
          StoreMessage<2>(Partial(r, it, g), unset);
      for (int it = t; it < KP; it += n)
        StoreMessage<2>(Result(r, c, it), unset);
    }
  }
};

// Polls the Q doubles at base + step * u, u < count (at most N), until all of them are set.
template <int N, int Q, class R>
__device__ __forceinline__ void Poll(const PcgArgs &a, const double *base, int step, int count, double (&y)[N][Q], R &sm)
{
#pragma unroll
  for (int u = 0; u < N; ++u)
#pragma unroll
    for (int q = 0; q < Q; ++q)
      y[u][q] = 0.0;
  const unsigned long long t0 = GlobalTimer();
  unsigned spin = 0;
  for (;;) {
    bool missing = false;
#pragma unroll
    for (int u = 0; u < N; ++u)
      if (u < count)
        LoadMessage<Q>(base + step * u, y[u]);
#pragma unroll
    for (int u = 0; u < N; ++u)
      missing = missing || Unset(y[u][0]) || Unset(y[u][Q - 1]);
    if (!missing || !PollAgain(a, spin, t0, sm))
      return;
  }
}

// Warp 0's half of a CG loop reduction of Q per-item sums, in GridReduce's order: the lanes
// of a warp (WarpPart), the 16 warps of a row group, then the row groups lane-strided over
// one warp.  First it sends the CTA's partials ...
template <int KP, int GV, int Q>
__device__ __forceinline__ void SendPartials(int rank, const Mailboxes<KP> &mail, ResidentShared<KP, GV> &sm, int r)
{
  constexpr int QK = Q * KP;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int t0 = 0; t0 < QK * GV; t0 += 32) {
    const int gv = (t0 + lane) / QK, t = (t0 + lane) % QK;
    if (gv < GV && rank * GV + gv < mail.G) {
      double w[kPcgWarps];
#pragma unroll
      for (int i = 0; i < kPcgWarps; ++i)
        w[i] = sm.warp[gv * kPcgWarps + i][t];
      double s = w[0];
#pragma unroll
      for (int i = 1; i < kPcgWarps; ++i)
        s += w[i];
      const double m[1] = {Sendable(s)};
      StoreMessage<1>(mail.Partial(r, t % KP, rank * GV + gv) + t / KP, m);
    }
  }
}

// ... then it sums the items this CTA owns and sends their results to every CTA (or sums
// every item itself, direct).  Lane `item` leaves with the item's sums.  kFence: and with
// everything acquired that the CTAs had released with their partials.  N: partials a lane polls at once.
template <int KP, int GV, int Q, bool kFence = false, int N = 5>
__device__ __forceinline__ void Collect(const PcgArgs &a, int rank, const Mailboxes<KP> &mail,
                                        ResidentShared<KP, GV> &sm, int r, double (&sum)[Q])
{
  const int lane = threadIdx.x & 31, G = mail.G;
  if (mail.direct) {
    // Two slots per lane: slot = item x padded + row group.
    double s[2][Q];
    const int shift = 31 - __clz(mail.padded);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int it = (lane + 32 * u) >> shift, g = (lane + 32 * u) & (mail.padded - 1);
      double y[1][Q];
      Poll<1, Q>(a, mail.Partial(r, it, g), 0, it < KP && g < G ? 1 : 0, y, sm);
#pragma unroll
      for (int q = 0; q < Q; ++q)
        s[u][q] = y[0][q];
    }
    __syncwarp();
    if (shift > 5) // one item: lane g's sum takes row group g + 32 too
#pragma unroll
      for (int q = 0; q < Q; ++q)
        s[0][q] += s[1][q];
#pragma unroll
    for (int o = 4; o >= 0; --o)
      if (o < shift)
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int q = 0; q < Q; ++q)
            s[u][q] += __shfl_xor_sync(0xffffffffu, s[u][q], 1 << o);
    const int from = (lane < KP ? lane : 0) << shift; // slot of the lane's item
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const double lo = __shfl_sync(0xffffffffu, s[0][q], from & 31), hi = __shfl_sync(0xffffffffu, s[1][q], from & 31);
      sum[q] = from < 32 ? lo : hi;
    }
    return;
  }
  for (int it = rank; it < KP; it += mail.ctas) {
    double s[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q)
      s[q] = 0.0;
    for (int g0 = 0; g0 < G; g0 += 32 * N) {
      double y[N][Q];
      const int count = (G - g0 - lane + 31) >> 5;
      Poll<N, Q>(a, mail.Partial(r, it, g0 + lane), 64, count, y, sm);
#pragma unroll
      for (int u = 0; u < N; ++u)
        if (u < count)
#pragma unroll
          for (int q = 0; q < Q; ++q)
            s[q] += y[u][q];
      __syncwarp();
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
      for (int q = 0; q < Q; ++q)
        s[q] += __shfl_xor_sync(0xffffffffu, s[q], off);
    const double m[2] = {Sendable(s[0]), Sendable(s[Q - 1])};
    if constexpr (kFence)
      FenceAcqRel();
    for (int c = lane; c < mail.ctas; c += 32)
      StoreMessage<2>(mail.Result(r, c, it), m);
  }
  double y[1][2];
  Poll<1, 2>(a, mail.Result(r, rank, lane), 0, lane < KP ? 1 : 0, y, sm);
  __syncwarp();
  sum[Q - 1] = y[0][1];
  sum[0] = y[0][0];
  if constexpr (kFence)
    FenceAcqRel();
}

// The same sums in the rare phases (set-up, verification, the end of the budget), behind a
// full grid barrier: every CTA's stores before it are seen by every CTA after it.
template <int KP, int GV, int Q, bool kMax, class F>
__device__ __forceinline__ bool BarrierReduce(const PcgArgs &a, int rank, int ctas, int G, ResidentShared<KP, GV> &sm,
                                              unsigned &epoch, int &buf, F control)
{
  constexpr int QK = Q * KP;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double *part = a.partials + static_cast<size_t>(buf) * 2 * KP * G;
  __syncthreads();
  if (threadIdx.x < QK * GV) {
    const int gv = static_cast<int>(threadIdx.x) / QK, t = static_cast<int>(threadIdx.x) % QK;
    double s = sm.warp[gv * kPcgWarps][t];
    for (int i = 1; i < kPcgWarps; ++i)
      s = kMax ? fmax(s, sm.warp[gv * kPcgWarps + i][t]) : s + sm.warp[gv * kPcgWarps + i][t];
    if (rank * GV + gv < G)
      part[static_cast<size_t>(t) * G + rank * GV + gv] = s;
  }
  if (!GridBarrier(a, GridShape{ctas, rank}, epoch, sm))
    return false;
  for (int it = warp; it < KP; it += kPcgWarps) {
    double s[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const double *pt = part + static_cast<size_t>(q * KP + it) * G;
      s[q] = 0.0;
      for (int g = lane; g < G; g += 32) {
        const double y = __ldcg(pt + g);
        s[q] = kMax ? fmax(s[q], y) : s[q] + y;
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, s[q], off);
        s[q] = kMax ? fmax(s[q], y) : s[q] + y;
      }
    }
    if (lane == 0)
      control(it, s);
  }
  __syncthreads();
  buf ^= 1;
  return true;
}

// Dynamic shared memory: a block per operator entry of a warp-step (p_j, a_ij, and the
// column of each row as a double's index), then the entry offsets of the CTA's steps at
// PcgArgs::resident_offset.  Offsets inside a block and its bytes:
template <int KP, int IV, bool SHARED> struct ResidentLayout {
  static constexpr int kRows = 32 * IV / KP; // of a warp-step
  static constexpr int kSlot = 32 * IV * 8;  // a lane's IV items, 32 lanes
  static constexpr int kValue = kSlot, kColumn = kSlot + (SHARED ? kRows * 8 : kSlot);
  static constexpr int kEntry = kColumn + (kRows * 4 + 15) / 16 * 16;
};

// SHARED: one operator for all items (value_stride 1), else one per item.
template <int KP, int IV, bool SHARED>
__global__ void __launch_bounds__(kPcgThreads, 1) PcgResidentKernel(PcgArgs a)
{
  __shared__ ResidentShared<KP, 1> sm;
  __shared__ Control ctl;
  __shared__ Trace tr;
  __shared__ Mailboxes<KP> mail;
  extern __shared__ __align__(16) unsigned char resident_smem[];
  using L = ResidentLayout<KP, IV, SHARED>;
  constexpr int LR = KP / IV, S = 32 / LR;
  constexpr int U = 8; // entries of a row gathered ahead
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rank = static_cast<int>(blockIdx.x), G = static_cast<int>(gridDim.x);
  const int item0 = (lane % LR) * IV, rl = lane / LR;
  const int WS = a.n_pad / S;
  const int ws0 = static_cast<int>(static_cast<long long>(WS) * rank / G);
  const int steps = static_cast<int>(static_cast<long long>(WS) * (rank + 1) / G) - ws0; // <= 16
  const bool has = warp < steps; // this warp's step
  const int row = (ws0 + warp) * S + rl;
  const size_t ri = static_cast<size_t>(row) * KP + item0;
  unsigned epoch = 0;
  int buf = 0; // of the barrier-based reductions
  int32_t *off = reinterpret_cast<int32_t *>(resident_smem + a.resident_offset);
  if (warp == 0) {
    // A running sum over the slice widths of the steps.
    int sum = 0;
    if (lane < steps) {
      const int s = ((ws0 + lane) * S) >> 5;
      sum = (__ldg(a.slice_off + s + 1) - __ldg(a.slice_off + s)) >> 5;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o)
        sum += y;
    }
    if (lane < steps)
      off[lane + 1] = sum;
    if (lane == 0)
      off[0] = 0;
  }
  if (threadIdx.x < KP) {
    const int it = threadIdx.x;
    ctl.active[it] = (it < a.items && ((a.active_mask >> it) & 1u)) ? 1 : 0;
    ctl.status[it] = kInternal;
    ctl.iters[it] = 0;
    ctl.resid[it] = INFINITY;
    ctl.flag[it] = 0;
    ctl.beta[it] = 0.0;
    ctl.scale[it] = 1.0;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kPcgTraceSlots; ++s)
      tr.slot[s] = 0;
    tr.mark = GlobalTimer();
    sm.err = sm.failed = 0;
    mail.Init(a, G);
  }
  __syncthreads();
  // The mailboxes start unset; the set-up's barriers make that known.
  for (int r = 0; r < kMailboxes; ++r)
    mail.Reset(r, rank, threadIdx.x, kPcgThreads);

  const double *B = static_cast<const double *>(a.b);
  double *GX = static_cast<double *>(a.x);
  // z of iterations 0, 1, 2 and 3 (mod 4): vectors this form does not need otherwise.
  auto z_buffer = [&](int t) {
    return static_cast<double *>((t & 2) ? ((t & 1) ? a.p0 : a.r) : ((t & 1) ? a.q : a.z));
  };
  auto on = [&](int j) { return ctl.active[item0 + j] != 0; };
  // The lane's part of the warp's entries: direction, value, and the row's column.
  const int e0 = has ? off[warp] : 0, W = has ? off[warp + 1] - e0 : 0;
  unsigned char *const entry = resident_smem + e0 * L::kEntry;
  auto direction = [&](int w) { return reinterpret_cast<double *>(entry + w * L::kEntry + lane * IV * 8); };
  auto value = [&](int w, double (&vv)[IV]) {
    const unsigned char *e = entry + w * L::kEntry + L::kValue;
    if constexpr (SHARED) {
#pragma unroll
      for (int j = 0; j < IV; ++j)
        vv[j] = *reinterpret_cast<const double *>(e + rl * 8);
    } else {
      Load<double, IV>(reinterpret_cast<const double *>(e + lane * IV * 8), vv);
    }
  };
  auto column = [&](int w) -> int32_t & {
    return *reinterpret_cast<int32_t *>(entry + w * L::kEntry + L::kColumn + rl * 4);
  };
  // The lane's row: iterate, residual, A p, direction and 1/d (or d, to divide by).
  double x[IV] = {}, rv[IV] = {}, qv[IV] = {}, pv[IV] = {}, inv[IV] = {};
  auto precond = [&](double (&zv)[IV]) {
#pragma unroll
    for (int j = 0; j < IV; ++j)
      zv[j] = a.use_inverse ? rv[j] * inv[j] : rv[j] / inv[j];
  };
  auto send_z = [&](double *z, const double (&zv)[IV]) {
    double m[IV];
#pragma unroll
    for (int j = 0; j < IV; ++j)
      m[j] = Sendable(zv[j]);
    StoreMessage<IV>(z + ri, m);
  };
  auto reset_z = [&](double *z) {
    double m[IV];
#pragma unroll
    for (int j = 0; j < IV; ++j)
      m[j] = UnsetValue();
    StoreMessage<IV>(z + ri, m);
  };

  // Operator, inverse diagonal; validity (first invalid row decides) and RHS max-scaling.
  {
    double v[2][IV] = {};
    if (has) {
      const double *vals = static_cast<const double *>(a.values);
      const int len = __ldg(a.row_len + row);
      const size_t base = static_cast<size_t>(__ldg(a.slice_off + (row >> 5))) + (row & 31);
      for (int w = 0; w < W; ++w) {
        // Places past the row's end: the row's own column with the value 0.
        const size_t pos = base + 32 * static_cast<size_t>(w);
        double t[IV] = {};
        if (lane % LR == 0)
          column(w) = (w < len ? __ldg(a.sell_col + pos) : row) * KP;
        if constexpr (SHARED) {
          if (lane % LR == 0)
            *reinterpret_cast<double *>(entry + w * L::kEntry + L::kValue + rl * 8) = w < len ? __ldg(vals + pos) : 0.0;
        } else {
          double vv[IV] = {};
          if (w < len)
            LoadStream<double, IV>(vals + pos * KP + item0, vv);
          Store<double, IV>(reinterpret_cast<double *>(entry + w * L::kEntry + L::kValue + lane * IV * 8), vv);
        }
        Store<double, IV>(direction(w), t);
      }
      double dd[IV], bb[IV];
      LoadOperand<double, IV>(static_cast<const double *>(a.use_inverse ? a.invd : a.diag), static_cast<size_t>(row),
                              a.diag_stride, a.diag_item, item0, inv);
      Load<double, IV>(B + ri, bb);
      LoadOperand<double, IV>(static_cast<const double *>(a.diag), static_cast<size_t>(row), a.diag_stride,
                              a.diag_item, item0, dd);
#pragma unroll
      for (int j = 0; j < IV; ++j)
        if (on(j) && row < a.n) {
          const double bj = bb[j], dj = dd[j];
          const bool nonfinite = !isfinite(bj) || !isfinite(dj);
          if (nonfinite || !(dj > 0.0))
            v[0][j] = fmax(v[0][j], 2.0 * static_cast<double>(a.n - row) + (nonfinite ? 1.0 : 0.0));
          v[1][j] = fmax(v[1][j], fabs(bj));
        }
    }
    WarpPart<KP, IV, 1, 2, true>(v, warp, sm);
    if (!BarrierReduce<KP, 1, 2, true>(a, rank, G, G, sm, epoch, buf, [&](int it, const double (&sum)[2]) {
          if (!ctl.active[it])
            return;
          const double pr = sum[0];
          if (pr != 0.0) {
            const bool nonfinite = pr - 2.0 * floor(0.5 * pr) != 0.0;
            ctl.status[it] = nonfinite ? kNonfinite : kBreakdown;
            ctl.active[it] = 0;
          } else {
            ctl.scale[it] = sum[1];
            if (ctl.scale[it] == 0.0) {
              ctl.resid[it] = 0.0;
              ctl.status[it] = kOk;
              ctl.active[it] = 0;
            }
          }
        }))
      return;
  }

  // r = b / s, z = M^-1 r, rho = r.z
  {
    double v[2][IV] = {};
    if (has) {
      double bb[IV], zv[IV];
      Load<double, IV>(B + ri, bb);
#pragma unroll
      for (int j = 0; j < IV; ++j)
        rv[j] = bb[j] / (ctl.scale[item0 + j] != 0.0 ? ctl.scale[item0 + j] : 1.0);
      precond(zv);
      send_z(z_buffer(0), zv);
#pragma unroll
      for (int t = 1; t < 4; ++t)
        reset_z(z_buffer(t));
#pragma unroll
      for (int j = 0; j < IV; ++j)
        if (on(j)) {
          v[0][j] += rv[j] * rv[j];
          v[1][j] += rv[j] * zv[j];
        }
    }
    WarpPart<KP, IV, 1, 2, false>(v, warp, sm);
    if (!BarrierReduce<KP, 1, 2, false>(a, rank, G, G, sm, epoch, buf, [&](int it, const double (&sum)[2]) {
          if (!ctl.active[it])
            return;
          const double rr = sum[0], rho = sum[1];
          if (!isfinite(rr) || !isfinite(rho)) {
            ctl.status[it] = kNonfinite;
            ctl.active[it] = 0;
          } else {
            ctl.resid[it] = sqrt(rr);
            ctl.thr[it] = (a.item_tolerance ? a.item_tolerance[it] : a.tolerance) * sqrt(rr);
            ctl.rho[it] = rho;
          }
        }))
      return;
  }

  // True residual of the lane's row: b / s - A x from the global copy of x.
  auto true_residual = [&](double (&t)[IV]) {
    double acc[IV] = {}, bb[IV];
    Load<double, IV>(B + ri, bb);
    for (int w = 0; w < W; ++w) {
      double g[IV], vv[IV];
      Load<double, IV>(GX + column(w) + item0, g);
      value(w, vv);
#pragma unroll
      for (int j = 0; j < IV; ++j)
        acc[j] = Fma(vv[j], g[j], acc[j]);
    }
#pragma unroll
    for (int j = 0; j < IV; ++j)
      t[j] = bb[j] / ctl.scale[item0 + j] - acc[j];
  };
  // Phase trace of CTA 0, kept by warp 0.
  auto mark = [&](int phase) {
    if (a.trace && rank == 0 && threadIdx.x == 0) {
      const unsigned long long now = GlobalTimer();
      tr.slot[phase] += now - tr.mark;
      tr.mark = now;
    }
  };

  // The z of the row's first U columns, on their way.
  double g[U][IV];
  auto fetch = [&](const double *z) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < W)
        LoadMessage<IV>(z + column(u) + item0, g[u]);
  };
  // Waits until they have arrived: z was sent before its owner's partial sums, so they
  // nearly always have.
  auto arrive = [&](const double *z) {
    auto missing = [&] {
      bool m = false;
#pragma unroll
      for (int u = 0; u < U; ++u)
        m = m || (u < W && Missing<IV>(g[u]));
      return m;
    };
    if (missing()) {
      const unsigned long long t0 = GlobalTimer();
      unsigned spin = 0;
      do
        fetch(z);
      while (missing() && PollAgain(a, spin, t0, sm));
    }
  };
  // What the whole CTA goes on with after a reduction, left in sm.state by warp 0.
  auto decide = [&](unsigned threshold) {
    const unsigned active = __ballot_sync(0xffffffffu, lane < KP && ctl.active[lane < KP ? lane : 0]);
    if (lane == 0)
      sm.state = make_uint2(active, (*const_cast<volatile int *>(&sm.failed) ? kStop : 0u) | threshold);
  };
  unsigned active = __ballot_sync(0xffffffffu, lane < KP && ctl.active[lane < KP ? lane : 0]);
  const unsigned bits = (IV == 2 ? 3u : 1u) << item0; // of the lane's items
  if (has && (active & bits))
    fetch(z_buffer(0));
  int red = 0; // reductions so far
  if (warp == 0)
    mark(6);

#pragma unroll 1
  for (int iteration = 0; iteration < a.max_iterations && active; ++iteration) {
    double *const z = z_buffer(iteration), *const zn = z_buffer(iteration + 1);
    // Phase A: p = z + beta p of every entry's column and of the row, q = A p, p . q.  beta
    // is 0 and the directions finite (at first 0) where p restarts at z.
    {
      double v[1][IV] = {};
      if (has && (active & bits)) {
        double be[IV], acc[IV] = {};
#pragma unroll
        for (int j = 0; j < IV; ++j)
          be[j] = ctl.beta[item0 + j];
        arrive(z);
        // Four entries at a time: all loads before the stores they might alias.
        constexpr int F = 4;
#pragma unroll
        for (int u0 = 0; u0 < U; u0 += F) {
          double pj[F][IV], vv[F][IV];
#pragma unroll
          for (int u = 0; u < F; ++u)
            if (u0 + u < W) {
              Load<double, IV>(direction(u0 + u), pj[u]);
              value(u0 + u, vv[u]);
            }
#pragma unroll
          for (int u = 0; u < F; ++u)
            if (u0 + u < W) {
#pragma unroll
              for (int j = 0; j < IV; ++j) {
                pj[u][j] = Fma(be[j], pj[u][j], g[u0 + u][j]);
                acc[j] = Fma(vv[u][j], pj[u][j], acc[j]);
              }
              Store<double, IV>(direction(u0 + u), pj[u]);
            }
        }
#pragma unroll 1
        for (int w = U; w < W; ++w) { // wide rows
          double zj[IV], pj[IV], vv[IV];
          const unsigned long long t0 = GlobalTimer();
          unsigned spin = 0;
          do
            LoadMessage<IV>(z + column(w) + item0, zj);
          while (Missing<IV>(zj) && PollAgain(a, spin, t0, sm));
          Load<double, IV>(direction(w), pj);
          value(w, vv);
#pragma unroll
          for (int j = 0; j < IV; ++j) {
            pj[j] = Fma(be[j], pj[j], zj[j]);
            acc[j] = Fma(vv[j], pj[j], acc[j]);
          }
          Store<double, IV>(direction(w), pj);
        }
        // The row's own z = M^-1 r again: the very product its readers were sent.
        double zr[IV];
        precond(zr);
#pragma unroll
        for (int j = 0; j < IV; ++j) {
          pv[j] = Fma(be[j], pv[j], zr[j]);
          qv[j] = acc[j];
          v[0][j] = pv[j] * qv[j];
        }
      }
      WarpPart<KP, IV, 1, 1, false>(v, warp, sm);
    }
    if (warp == 0) {
      const int it = lane < KP ? lane : 0;
      const double rho = ctl.rho[it];
      NamedSync<1>();
      mark(0);
      SendPartials<KP, 1, 1>(rank, mail, sm, red);
      FenceAcqRel();
      double sum[1];
      Collect<KP, 1, 1>(a, rank, mail, sm, red, sum);
      if (lane < KP && ((active >> lane) & 1u)) {
        const double pq = sum[0];
        if (pq > 0.0 && rho > 0.0 && isfinite(pq) && isfinite(rho)) {
          ctl.alpha[it] = rho / pq;
        } else {
          ctl.status[it] = !isfinite(pq) || !isfinite(rho) ? kNonfinite : kBreakdown;
          ctl.active[it] = 0;
        }
      }
      decide(0u);
    } else {
      NamedArrive<1>();
    }
    NamedSync<2>();
    ++red;
    if (warp == 0)
      mark(1);
    uint2 state = sm.state;
    active = state.x;
    if (state.y & kStop)
      return;

    // Phase B: x += alpha p, r -= alpha q, z = M^-1 r, r.r and r.z
    const bool mine = has && (active & bits);
    {
      double v[2][IV] = {};
      if (mine) {
        double zv[IV];
#pragma unroll
        for (int j = 0; j < IV; ++j)
          if ((active >> (item0 + j)) & 1u) {
            const double al = ctl.alpha[item0 + j];
            x[j] = x[j] + al * pv[j];
            rv[j] = rv[j] - al * qv[j];
          }
        precond(zv);
        send_z(zn, zv);
#pragma unroll
        for (int j = 0; j < IV; ++j) {
          v[0][j] = rv[j] * rv[j];
          v[1][j] = rv[j] * zv[j];
        }
      }
      WarpPart<KP, IV, 1, 2, false>(v, warp, sm);
    }
    // While the sums travel: gather the z of the next phase A, reset the z of this iteration
    // (every CTA's phase A of it is over: the buffer serves iteration + 4) and the mailboxes
    // of reductions red + 5 (direct) or red + 7, and red + 6: last read at red - 3 or red - 1,
    // and red - 2, which all their readers have finished.
    if (warp == 0) {
      const int it = lane < KP ? lane : 0;
      const double rho = ctl.rho[it], thr = ctl.thr[it];
      NamedSync<1>();
      mark(2);
      SendPartials<KP, 1, 2>(rank, mail, sm, red);
      if (mine) {
        fetch(zn);
        reset_z(z);
      }
      double sum[2];
      Collect<KP, 1, 2>(a, rank, mail, sm, red, sum);
      bool at = false;
      if (lane < KP) {
        ctl.flag[it] = 0;
        if ((active >> lane) & 1u) {
          ctl.iters[it] = iteration + 1;
          const double rr = sum[0], rz = sum[1];
          if (!isfinite(rr)) {
            ctl.status[it] = kNonfinite;
            ctl.active[it] = 0;
          } else {
            // ||r||, taken when it is needed: here only near the threshold (within the
            // rounding of the squares).
            ctl.resid[it] = -rr;
            at = rr <= thr * thr * (1.0 + 1e-14) && sqrt(rr) <= thr;
            if (at) {
              ctl.flag[it] = a.skip_verification ? 2 : 1;
            } else if (isfinite(rz) && rz > 0.0) {
              ctl.beta[it] = rz / rho;
              ctl.rho[it] = rz;
            } else {
              ctl.status[it] = kBreakdown;
              ctl.active[it] = 0;
            }
          }
        }
      }
      decide(__any_sync(0xffffffffu, at) ? kThreshold : 0u);
    } else {
      NamedArrive<1>();
      if (mine) {
        fetch(zn);
        reset_z(z);
      }
      mail.Reset(red + (mail.direct ? 5 : 7), rank, threadIdx.x - 32, kPcgThreads - 32);
      mail.Reset(red + 6, rank, threadIdx.x - 32, kPcgThreads - 32);
    }
    NamedSync<2>();
    ++red;
    if (warp == 0) {
      mark(3);
      if (a.trace && rank == 0 && lane == 0)
        tr.slot[9] += 2;
    }
    state = sm.state;
    active = state.x;
    if (state.y & kStop)
      return;

    // Items at the threshold: verify the true residual, then accept (scale x back) or
    // restart from it.
    if (state.y & kThreshold) {
      if (threadIdx.x < KP && ctl.resid[threadIdx.x] < 0.0)
        ctl.resid[threadIdx.x] = sqrt(-ctl.resid[threadIdx.x]);
      if (!a.skip_verification) {
        if (has)
          Store<double, IV>(GX + ri, x);
        if (!GridBarrier(a, GridShape{G, rank}, epoch, sm))
          return;
        double v[1][IV] = {};
        if (has) {
          double t[IV];
          true_residual(t);
#pragma unroll
          for (int j = 0; j < IV; ++j)
            if (on(j) && ctl.flag[item0 + j] == 1) {
              rv[j] = t[j];
              v[0][j] = t[j] * t[j];
            }
        }
        WarpPart<KP, IV, 1, 1, false>(v, warp, sm);
        if (!BarrierReduce<KP, 1, 1, false>(a, rank, G, G, sm, epoch, buf, [&](int it, const double (&sum)[1]) {
              if (!ctl.active[it] || ctl.flag[it] != 1)
                return;
              const double trr = sum[0];
              if (!isfinite(trr)) {
                ctl.status[it] = kNonfinite;
                ctl.active[it] = 0;
              } else {
                ctl.resid[it] = sqrt(trr);
                ctl.flag[it] = ctl.resid[it] <= ctl.thr[it] ? 2 : 3;
              }
            }))
          return;
      }
      double v[2][IV] = {};
      if (has) {
        double zv[IV];
        precond(zv);
        bool restart = false;
#pragma unroll
        for (int j = 0; j < IV; ++j) {
          const int f = on(j) ? ctl.flag[item0 + j] : 0;
          if (f == 2) {
            x[j] = x[j] * ctl.scale[item0 + j];
            if (!isfinite(x[j]))
              v[1][j] = 1.0;
          }
          if (f == 3) {
            v[0][j] = rv[j] * zv[j];
            restart = true;
          }
        }
        if (restart) // items that go on keep r, so their z is the same product again
          send_z(zn, zv);
      }
      WarpPart<KP, IV, 1, 2, false>(v, warp, sm);
      if (!BarrierReduce<KP, 1, 2, false>(a, rank, G, G, sm, epoch, buf, [&](int it, const double (&sum)[2]) {
            if (!ctl.active[it])
              return;
            if (ctl.flag[it] == 2) {
              if (sum[1] != 0.0) {
                ctl.status[it] = kNonfinite;
              } else {
                ctl.resid[it] *= ctl.scale[it];
                ctl.status[it] = isfinite(ctl.resid[it]) ? kOk : kNonfinite;
              }
              ctl.active[it] = 0;
            } else if (ctl.flag[it] == 3) {
              const double rho = sum[0];
              if (!isfinite(rho) || !(rho > 0.0)) {
                ctl.status[it] = kBreakdown;
                ctl.active[it] = 0;
              } else {
                ctl.rho[it] = rho;
                ctl.beta[it] = 0.0;
              }
            }
          }))
        return;
      active = __ballot_sync(0xffffffffu, lane < KP && ctl.active[lane < KP ? lane : 0]);
      if (has && (active & bits))
        fetch(zn);
    }
  }

  // Iteration budget exhausted: report the true residual and scale the iterate back.
  if (active) {
    if (has)
      Store<double, IV>(GX + ri, x);
    if (!GridBarrier(a, GridShape{G, rank}, epoch, sm))
      return;
    {
      double v[1][IV] = {};
      if (has) {
        double t[IV];
        true_residual(t);
#pragma unroll
        for (int j = 0; j < IV; ++j)
          if (on(j))
            v[0][j] = t[j] * t[j];
      }
      WarpPart<KP, IV, 1, 1, false>(v, warp, sm);
      if (!BarrierReduce<KP, 1, 1, false>(a, rank, G, G, sm, epoch, buf, [&](int it, const double (&sum)[1]) {
            if (!ctl.active[it])
              return;
            const double trr = sum[0];
            if (!isfinite(trr)) {
              ctl.status[it] = kNonfinite;
              ctl.active[it] = 0;
            } else {
              ctl.rz[it] = trr;
            }
          }))
        return;
    }
    double v[1][IV] = {};
#pragma unroll
    for (int j = 0; j < IV; ++j)
      if (has && on(j)) {
        x[j] = x[j] * ctl.scale[item0 + j];
        if (!isfinite(x[j]))
          v[0][j] = 1.0;
      }
    WarpPart<KP, IV, 1, 1, false>(v, warp, sm);
    if (!BarrierReduce<KP, 1, 1, false>(a, rank, G, G, sm, epoch, buf, [&](int it, const double (&sum)[1]) {
          if (!ctl.active[it])
            return;
          if (sum[0] != 0.0) {
            ctl.status[it] = kNonfinite;
          } else {
            ctl.resid[it] = sqrt(ctl.rz[it]) * ctl.scale[it];
            ctl.status[it] = isfinite(ctl.resid[it]) ? kNotConverged : kNonfinite;
          }
          ctl.active[it] = 0;
        }))
      return;
  }
  if (has)
    Store<double, IV>(GX + ri, x);

  if (rank == 0 && threadIdx.x < a.items) {
    const int it = threadIdx.x;
    a.info[3 * it] = static_cast<double>(ctl.status[it]);
    a.info[3 * it + 1] = static_cast<double>(ctl.iters[it]);
    a.info[3 * it + 2] = ctl.resid[it] < 0.0 ? sqrt(-ctl.resid[it]) : ctl.resid[it];
  }
  if (a.trace && rank == 0 && threadIdx.x == 0)
    for (int s = 0; s < kPcgTraceSlots; ++s)
      a.trace[s] += tr.slot[s];
}

} // namespace
} // namespace fg
