// pcg_window.cuh -- the FP64 Jacobi PCG for large systems of limited bandwidth: the SpMV's
// operand in a sliding window in shared memory.
//
// Partition, operations and summation orders are PcgBody's (pcg_kernel.cuh): the same bits.
// PcgBody gathers z and p of every entry's column through L1 and L2 (16 bytes per entry and
// item beside the 8 of its value) and evaluates p_j = z_j + beta p_j for each entry; the
// gathers, not the DRAM, set the pace of its SpMV.  Here a CTA of 512 threads per SM takes two
// adjacent row groups and walks their rows in ascending order, 16 warp-steps (a tile of rows)
// per round.  The new search direction of all columns that the tile can reach -- the rows
// within the operator's bandwidth -- sits in a ring in shared memory; a round adds the tile of
// rows that the round after the next needs, a row's z and p being read once, coalesced, by the
// thread that evaluates its p.  What remains of the SpMV is a stream of values and columns, read
// a round ahead into registers, against shared memory.
//  * A round ahead, and all at once: the loads of a warp share six scoreboards, so a load issued
//    between the uses of earlier ones makes later uses wait for it (the round took 2.2 us with
//    each entry's load behind its use, 1.9 us and less so).
//  * The warps agree once per round through an mbarrier that they arrive at when they are done
//    and test a round later: a warp may be a round ahead of another, hence a window of
//    2 bandwidths + 4 tiles.
//  * q = A p stays in shared memory where it fits beside the ring.
//  * x is updated in every other iteration with both directions (the two FMAs of the two
//    iterations, so the same bits): four passes over memory instead of six.
//  * Sums travel as messages (pcg_resident.cuh).  z and p are read in phase A only, so one
//    release and acquire per iteration, with the sums of phase B, covers them.
//
// Measured on a B200, microseconds per CG iteration, PcgBody -> here:
//   rows  249,001: 2 items 20.3 -> 17.1, 4 items 34.9 -> 26.0, 8 items 68.3 -> 56.3, 16 items 147 -> 115
//   rows  124,609: 8 items 34.3 -> 26.8, 16 items 73.7 -> 58.3
//   rows   98,790: 8 items 28.4 -> 22.8, 32 items 110 -> 92.7
//   rows   40,000: 16 items 28.9 -> 23.5, 32 items 46.3 -> 37.5
// At 249,001 rows and 8 items phase A takes 31 us for 190 MB from DRAM (the operator, and what
// the vectors lose of L2 to it), phase B 10.5 us for six passes at L2's rate; the two sums,
// with the CTAs' unequal speed, 14 us.
#pragma once

#include "pcg_resident.cuh"

namespace fg
{
namespace
{

// Loads under a predicate, into registers that keep their values where it is false, at a
// constant distance (bytes) from a pointer.  (An if around a plain load becomes a branch with
// a move behind it that waits for the load: eight loads one after the other.)
template <int IV, int AT> __device__ __forceinline__ void LoadStreamIf(bool p, const double *from, double (&o)[IV])
{
  if constexpr (IV == 2)
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %3, 0; @q ld.global.cs.v2.f64 {%0, %1}, [%2+%4]; }"
                 : "+d"(o[0]), "+d"(o[1])
                 : "l"(from), "r"(static_cast<int>(p)), "n"(AT));
  else
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %2, 0; @q ld.global.cs.f64 %0, [%1+%3]; }"
                 : "+d"(o[0])
                 : "l"(from), "r"(static_cast<int>(p)), "n"(AT));
}
template <int IV> __device__ __forceinline__ void LoadIf(bool p, const double *from, double (&o)[IV])
{
  if constexpr (IV == 2)
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %3, 0; @q ld.global.v2.f64 {%0, %1}, [%2]; }"
                 : "+d"(o[0]), "+d"(o[1])
                 : "l"(from), "r"(static_cast<int>(p))
                 : "memory");
  else
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %2, 0; @q ld.global.f64 %0, [%1]; }"
                 : "+d"(o[0])
                 : "l"(from), "r"(static_cast<int>(p))
                 : "memory");
}
template <int AT> __device__ __forceinline__ void LoadIf(bool p, const int32_t *from, int &o)
{
  asm volatile("{ .reg .pred q; setp.ne.s32 q, %2, 0; @q ld.global.nc.s32 %0, [%1+%3]; }"
               : "+r"(o)
               : "l"(from), "r"(static_cast<int>(p)), "n"(AT));
}

// f(0) ... f(N - 1), the argument a constant.
template <int N, int U = 0, class F> __device__ __forceinline__ void Each(const F &f)
{
  if constexpr (U < N) {
    f(std::integral_constant<int, U>{});
    Each<N, U + 1>(f);
  }
}

// A barrier of the CTA's warps in two halves: a warp arrives when it is done with a round and
// waits, a round later, for the others.
__device__ __forceinline__ void RoundInit(unsigned long long *b)
{
  asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(b))), "r"(kPcgWarps)
               : "memory");
}
__device__ __forceinline__ void RoundArrive(unsigned long long *b)
{
  asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(b))) : "memory");
}
__device__ __forceinline__ bool RoundOver(unsigned long long *b, unsigned parity)
{
  unsigned over;
  asm volatile("{ .reg .pred q; mbarrier.try_wait.parity.shared.b64 q, [%1], %2; selp.u32 %0, 1, 0, q; }"
               : "=r"(over)
               : "r"(static_cast<unsigned>(__cvta_generic_to_shared(b))), "r"(parity)
               : "memory");
  return over != 0;
}

// QG: q in global memory.
template <int KP, int IV, bool QG>
__global__ void __launch_bounds__(kPcgThreads, 1) PcgWindowKernel(PcgArgs a)
{
  constexpr int GV = 2;
  __shared__ ResidentShared<KP, GV> sm;
  __shared__ Control ctl;
  __shared__ Trace tr;
  __shared__ Mailboxes<KP> mail;
  __shared__ double behind[KP]; // the alpha that x still lacks
  extern __shared__ __align__(16) unsigned char window_smem[];
  constexpr int LR = KP / IV, S = 32 / LR, TILE = kPcgWarps * S; // rows per warp-step, per round
  constexpr int U = 8; // entries of a row read a round ahead
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rank = static_cast<int>(blockIdx.x), ctas = static_cast<int>(gridDim.x), G = a.row_groups;
  const int item0 = (lane % LR) * IV, rl = lane / LR;
  const int WS = a.n_pad / S;
  auto first_step = [&](int g) { return static_cast<int>(static_cast<long long>(WS) * (g < G ? g : G) / G); };
  const int ws0 = first_step(rank * GV), mid = first_step(rank * GV + 1) - ws0;
  const int steps = first_step(rank * GV + GV) - ws0;
  const int rounds0 = (mid + kPcgWarps - 1) / kPcgWarps;
  const int rounds = rounds0 + (steps - mid + kPcgWarps - 1) / kPcgWarps;
  // First step of a round, and one past its group's last.
  auto round_step = [&](int t) { return t < rounds0 ? t * kPcgWarps : mid + (t - rounds0) * kPcgWarps; };
  auto round_end = [&](int t) { return t < rounds0 ? mid : steps; };
  __shared__ unsigned long long round_bar[2];
  unsigned tick = 0; // rounds so far
  unsigned epoch = 0;
  int buf = 0;
  if (threadIdx.x < KP) {
    const int it = threadIdx.x;
    ctl.active[it] = (it < a.items && ((a.active_mask >> it) & 1u)) ? 1 : 0;
    ctl.status[it] = kInternal;
    ctl.iters[it] = 0;
    ctl.resid[it] = INFINITY;
    ctl.flag[it] = 0;
    ctl.beta[it] = 0.0;
    ctl.restart[it] = 1;
    ctl.scale[it] = 1.0;
    behind[it] = 0.0;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kPcgTraceSlots; ++s)
      tr.slot[s] = 0;
    tr.mark = GlobalTimer();
    sm.err = sm.failed = 0;
    mail.Init(a, ctas);
    RoundInit(&round_bar[0]);
    RoundInit(&round_bar[1]);
  }
  __syncthreads();
  for (int r = 0; r < kMailboxes; ++r)
    mail.Reset(r, rank, threadIdx.x, kPcgThreads);

  double *const ring = reinterpret_cast<double *>(window_smem);
  const int RW = a.window_rows, BW = a.bandwidth; // ring size, rows: 2 BW + 4 TILE
  const double *B = static_cast<const double *>(a.b), *vals = static_cast<const double *>(a.values);
  const double *DG = static_cast<const double *>(a.diag);
  const double *IDG = static_cast<const double *>(a.use_inverse ? a.invd : a.diag);
  double *X = static_cast<double *>(a.x), *R = static_cast<double *>(a.r), *Z = static_cast<double *>(a.z);
  double *const Qs = QG ? static_cast<double *>(a.q) : ring + static_cast<size_t>(RW) * KP;
  auto on = [&](int j) { return ctl.active[item0 + j] != 0; };
  auto row_at = [&](int st) { return (ws0 + st) * S + rl; };
  auto item_at = [&](int st) { return static_cast<size_t>(row_at(st)) * KP + item0; };
  auto q_at = [&](int st) { return Qs + (QG ? item_at(st) : (static_cast<size_t>(st) * 32 + lane) * IV); };
  auto position = [&](int row) { return static_cast<size_t>(__ldg(a.slice_off + (row >> 5))) + (row & 31); };
  auto precond = [&](const double (&rv)[IV], const double (&d)[IV], double (&zv)[IV]) {
#pragma unroll
    for (int j = 0; j < IV; ++j)
      zv[j] = a.use_inverse ? rv[j] * d[j] : rv[j] / d[j];
  };
#define FG_GROUPS _Pragma("unroll 1") for (int gv = 0; gv < GV; ++gv)
#define FG_STEPS                                                                                   \
  _Pragma("unroll 1") for (int st = (gv ? mid : 0) + warp, end = gv ? steps : mid; st < end; st += kPcgWarps)

  // Validity (first invalid row decides the status) and RHS max-scaling.
  {
    FG_GROUPS
    {
      double v[2][IV] = {};
      FG_STEPS
      {
        const int row = row_at(st);
        const size_t ri = item_at(st);
        const double zero[IV] = {};
        double dd[IV], bb[IV];
        Load<double, IV>(B + ri, bb);
        Load<double, IV>(DG + ri, dd);
        Store<double, IV>(X + ri, zero);
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
      WarpPart<KP, IV, GV, 2, true>(v, gv * kPcgWarps + warp, sm);
    }
    if (!BarrierReduce<KP, GV, 2, true>(a, rank, ctas, G, sm, epoch, buf, [&](int it, const double (&sum)[2]) {
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
    FG_GROUPS
    {
      double v[2][IV] = {};
      FG_STEPS
      {
        const size_t ri = item_at(st);
        double bb[IV], d[IV], rv[IV], zv[IV];
        Load<double, IV>(B + ri, bb);
        Load<double, IV>(IDG + ri, d);
#pragma unroll
        for (int j = 0; j < IV; ++j)
          rv[j] = bb[j] / (ctl.scale[item0 + j] != 0.0 ? ctl.scale[item0 + j] : 1.0);
        precond(rv, d, zv);
        Store<double, IV>(R + ri, rv);
        Store<double, IV>(Z + ri, zv);
#pragma unroll
        for (int j = 0; j < IV; ++j)
          if (on(j)) {
            v[0][j] += rv[j] * rv[j];
            v[1][j] += rv[j] * zv[j];
          }
      }
      WarpPart<KP, IV, GV, 2, false>(v, gv * kPcgWarps + warp, sm);
    }
    if (!BarrierReduce<KP, GV, 2, false>(a, rank, ctas, G, sm, epoch, buf, [&](int it, const double (&sum)[2]) {
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

  // True residual of a step's row: b / s - A x.
  auto true_residual = [&](int st, double (&t)[IV]) {
    const int row = row_at(st), len = __ldg(a.row_len + row);
    const size_t pos = position(row);
    double acc[IV] = {}, bb[IV];
    Load<double, IV>(B + item_at(st), bb);
    for (int w = 0; w < len; ++w) {
      double g[IV], vv[IV];
      const size_t at = pos + 32 * static_cast<size_t>(w);
      Load<double, IV>(X + static_cast<size_t>(__ldg(a.sell_col + at)) * KP + item0, g);
      LoadStream<double, IV>(vals + at * KP + item0, vv);
#pragma unroll
      for (int j = 0; j < IV; ++j)
        acc[j] = Fma(vv[j], g[j], acc[j]);
    }
#pragma unroll
    for (int j = 0; j < IV; ++j)
      t[j] = bb[j] / ctl.scale[item0 + j] - acc[j];
  };
  auto mark = [&](int phase) {
    if (a.trace && rank == 0 && threadIdx.x == 0) {
      const unsigned long long now = GlobalTimer();
      tr.slot[phase] += now - tr.mark;
      tr.mark = now;
    }
  };
  auto decide = [&](unsigned threshold) {
    const unsigned act = __ballot_sync(0xffffffffu, lane < KP && ctl.active[lane < KP ? lane : 0]);
    if (lane == 0)
      sm.state = make_uint2(act, (*const_cast<volatile int *>(&sm.failed) ? kStop : 0u) | threshold);
  };
  unsigned active = __ballot_sync(0xffffffffu, lane < KP && ctl.active[lane < KP ? lane : 0]);
  const unsigned bits = (IV == 2 ? 3u : 1u) << item0;
  int red = 0;
  double *pc = static_cast<double *>(a.p0), *pn = static_cast<double *>(a.p1);
  // x of every row up to date: the iteration whose direction is p still lacks `behind`.
  auto catch_up = [&](const double *p) {
    FG_GROUPS
    FG_STEPS
    {
      const size_t ri = item_at(st);
      double xv[IV], pv[IV];
      Load<double, IV>(X + ri, xv);
      Load<double, IV>(p + ri, pv);
#pragma unroll
      for (int j = 0; j < IV; ++j)
        if (behind[item0 + j] != 0.0)
          xv[j] = xv[j] + behind[item0 + j] * pv[j];
      Store<double, IV>(X + ri, xv);
    }
    __syncthreads();
    if (threadIdx.x < KP)
      behind[threadIdx.x] = 0.0;
    __syncthreads();
  };
  if (warp == 0)
    mark(6);

#pragma unroll 1
  for (int iteration = 0; iteration < a.max_iterations && active; ++iteration) {
    // Phase A: p_new = z + beta p into the ring, q = A p_new, p_new . q
    {
      const bool mine = active & bits;
      double be[IV];
      bool fold[IV];
#pragma unroll
      for (int j = 0; j < IV; ++j) {
        be[j] = ctl.beta[item0 + j];
        fold[j] = !ctl.restart[item0 + j];
      }
      const int own0 = ws0 * S, own1 = (ws0 + steps) * S; // the CTA's rows
      const int t_row = static_cast<int>(threadIdx.x) / LR; // the thread's row of a tile, its items item0 ...
      // z and p of a row on their way, and its p_new into the ring.
      auto read = [&](int row, bool p, double (&zv)[IV], double (&pv)[IV]) {
        const size_t ri = static_cast<size_t>(p ? row : 0) * KP + item0;
        LoadIf<IV>(p, Z + ri, zv);
        LoadIf<IV>(p, pc + ri, pv);
      };
      auto enter = [&](int row, bool p, double *slot, const double (&zv)[IV], const double (&pv)[IV]) {
        if (p) {
          double m[IV];
#pragma unroll
          for (int j = 0; j < IV; ++j)
            m[j] = fold[j] ? Fma(be[j], pv[j], zv[j]) : zv[j];
          Store<double, IV>(slot, m);
          if (row >= own0 && row < own1)
            Store<double, IV>(pn + static_cast<size_t>(row) * KP + item0, m);
        }
      };
      double *const ring0 = ring + item0;
      // Entries of the warp's step of a round: values and columns, read a round ahead.
      double vv[U][IV] = {};
      int col[U] = {}, len = -1, pos = 0, next_len = -1, next_pos = 0;
      // Slice's offset and row's entries of the warp's step in round t, on their way (nothing
      // waits for them here); the row's first entry; no step: no entries (-1).
      auto place = [&](int t, int &off, int &ln) {
        const bool p = mine && t < rounds && round_step(t) + warp < round_end(t);
        const int row = row_at(p ? round_step(t) + warp : 0);
        off = 0;
        ln = -1;
        LoadIf<0>(p, a.slice_off + (row >> 5), off);
        LoadIf<0>(p, a.row_len + row, ln);
      };
      auto first_entry = [&](int t, int off) { return off + (row_at(t < rounds ? round_step(t) + warp : 0) & 31); };
      int after_pos, after_len;
      place(0, pos, len);
      place(1, next_pos, next_len);
      place(2, after_pos, after_len);
      pos = first_entry(0, pos);
      next_pos = first_entry(1, next_pos);
      Each<U>([&](auto u) {
        constexpr int kU = decltype(u)::value;
        LoadIf<kU * 128>(kU < len, a.sell_col + pos, col[kU]);
        LoadStreamIf<IV, kU * 256 * KP>(kU < len, vals + static_cast<size_t>(pos) * KP + item0, vv[kU]);
      });
      // Fill the window of the first two rounds: rows own0 - BW ... , slots from 0.
      constexpr int F = 2;
      const int fill = 2 * BW + TILE + (rounds > 1 ? round_step(1) * S : 0);
      for (int r0 = t_row; r0 < fill; r0 += F * TILE) {
        double zv[F][IV] = {}, pv[F][IV] = {};
#pragma unroll
        for (int f = 0; f < F; ++f) {
          const int i = r0 + f * TILE, row = own0 - BW + i;
          read(row, mine && i < fill && row >= 0 && row < a.n_pad, zv[f], pv[f]);
        }
#pragma unroll
        for (int f = 0; f < F; ++f) {
          const int i = r0 + f * TILE, row = own0 - BW + i;
          enter(row, mine && i < fill && row >= 0 && row < a.n_pad, ring0 + static_cast<unsigned>(i) * KP, zv[f], pv[f]);
        }
      }
      __syncthreads();
      double v[1][IV] = {};
      int lo = own0 - BW, row0 = own0; // row of slot 0 in this lap of the ring; first row of the round
      int row1 = rounds > 1 ? (ws0 + round_step(1)) * S : own1; // ... of the next round
      auto slot = [&](int row) { // a row of the window, at most two laps from lo
        const unsigned s = row - lo;
        return ring0 + min(s, s - static_cast<unsigned>(RW)) * KP;
      };
      // z and p of the thread's row of those that the round after the next adds to the window,
      // read a round before they enter.
      int in = row1 + TILE + BW + t_row, row2;
      double zv[IV] = {}, pv[IV] = {};
      bool enters;
      auto fetch = [&](int t) {
        row2 = t + 2 < rounds ? (ws0 + round_step(t + 2)) * S : row1;
        in = row1 + TILE + BW + t_row;
        enters = mine && t_row < row2 - row1 && in < a.n_pad;
        read(in, enters, zv, pv);
      };
      fetch(0);
#pragma unroll 1
      for (int t = 0; t < rounds; ++t, ++tick) {
        if (t >= 2 && !RoundOver(&round_bar[tick & 1], ((tick >> 1) & 1) ^ 1)) { // round t - 2
          const unsigned long long t0 = GlobalTimer();
          unsigned spin = 0;
          while (!RoundOver(&round_bar[tick & 1], ((tick >> 1) & 1) ^ 1) && PollAgain(a, spin, t0, sm)) {
          }
          __syncwarp();
        }
        double acc[IV] = {};
        const int32_t *next_col = a.sell_col + next_pos;
        const double *next_val = vals + static_cast<size_t>(next_pos) * KP + item0;
        Each<U>([&](auto u) {
          constexpr int kU = decltype(u)::value;
          if (kU < len) {
            double g[IV];
            Load<double, IV>(slot(col[kU]), g);
#pragma unroll
            for (int j = 0; j < IV; ++j)
              acc[j] = Fma(vv[kU][j], g[j], acc[j]);
          }
        });
#pragma unroll 1
        for (int w = U; w < len; ++w) { // wide rows
          double g[IV], x[IV];
          const size_t ps = static_cast<size_t>(pos) + 32 * w;
          LoadStream<double, IV>(vals + ps * KP + item0, x);
          Load<double, IV>(slot(__ldg(a.sell_col + ps)), g);
#pragma unroll
          for (int j = 0; j < IV; ++j)
            acc[j] = Fma(x[j], g[j], acc[j]);
        }
        // The next round's entries, all at once: a load issued between the uses of others can share
        // one of the warp's six scoreboards with them, and their uses would wait for it.
        Each<U>([&](auto u) {
          constexpr int kU = decltype(u)::value;
          LoadIf<kU * 128>(kU < next_len, next_col, col[kU]);
          LoadStreamIf<IV, kU * 256 * KP>(kU < next_len, next_val, vv[kU]);
        });
        if (len >= 0) {
          const int st = round_step(t) + warp;
          double own[IV];
          Load<double, IV>(slot(row0 + warp * S + rl), own);
          Store<double, IV>(q_at(st), acc);
#pragma unroll
          for (int j = 0; j < IV; ++j)
            v[0][j] += own[j] * acc[j];
        }
        enter(in, enters, slot(in), zv, pv);
        __syncwarp();
        if (lane == 0)
          RoundArrive(&round_bar[tick & 1]);
        if (t + 1 == rounds0 || t + 1 == rounds) { // a row group is done
          WarpPart<KP, IV, GV, 1, false>(v, (t < rounds0 ? 0 : kPcgWarps) + warp, sm);
#pragma unroll
          for (int j = 0; j < IV; ++j)
            v[0][j] = 0.0;
        }
        row0 = row1;
        row1 = row2;
        lo = row0 - BW >= lo + RW ? lo + RW : lo;
        pos = next_pos;
        len = next_len;
        next_pos = first_entry(t + 2, after_pos);
        next_len = after_len;
        place(t + 3, after_pos, after_len);
        fetch(t + 1);
      }
      if (rounds == rounds0) { // no second row group
        WarpPart<KP, IV, GV, 1, false>(v, kPcgWarps + warp, sm);
      }
    }
    if (warp == 0) {
      const int it = lane < KP ? lane : 0;
      const double rho = ctl.rho[it];
      NamedSync<1>();
      mark(0);
      SendPartials<KP, GV, 1>(rank, mail, sm, red);
      double sum[1];
      Collect<KP, GV, 1, false, 10>(a, rank, mail, sm, red, sum);
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

    // Phase B: r -= alpha q, z = M^-1 r, r.r and r.z; in every other iteration
    // x += alpha' p' + alpha p.  pc is the previous direction, pn this one.
    const bool both = iteration & 1;
    {
      double al[IV], was[IV];
      bool act[IV];
#pragma unroll
      for (int j = 0; j < IV; ++j) {
        act[j] = (active >> (item0 + j)) & 1u;
        al[j] = act[j] ? ctl.alpha[item0 + j] : 0.0;
        was[j] = behind[item0 + j];
      }
      FG_GROUPS
      {
        double v[2][IV] = {};
        const int end = gv ? steps : mid;
        bool moves = false, lacks = false;
#pragma unroll
        for (int j = 0; j < IV; ++j) {
          moves = moves || act[j];
          lacks = lacks || (both && (act[j] || was[j] != 0.0));
        }
        if (lacks) {
          constexpr int F = 2; // steps whose loads are issued together
#pragma unroll 1
          for (int s0 = (gv ? mid : 0) + warp; s0 < end; s0 += F * kPcgWarps) {
            double xv[F][IV], p0[F][IV], p1[F][IV];
#pragma unroll
            for (int f = 0; f < F; ++f)
              if (s0 + f * kPcgWarps < end) {
                const size_t ri = item_at(s0 + f * kPcgWarps);
                LoadStream<double, IV>(X + ri, xv[f]);
                Load<double, IV>(pc + ri, p0[f]);
                Load<double, IV>(pn + ri, p1[f]);
              }
#pragma unroll
            for (int f = 0; f < F; ++f)
              if (s0 + f * kPcgWarps < end) {
#pragma unroll
                for (int j = 0; j < IV; ++j) {
                  if (was[j] != 0.0)
                    xv[f][j] = xv[f][j] + was[j] * p0[f][j];
                  if (act[j])
                    xv[f][j] = xv[f][j] + al[j] * p1[f][j];
                }
                Store<double, IV>(X + item_at(s0 + f * kPcgWarps), xv[f]);
              }
          }
        }
        if (moves) {
          constexpr int F = 2;
#pragma unroll 1
          for (int s0 = (gv ? mid : 0) + warp; s0 < end; s0 += F * kPcgWarps) {
            double rv[F][IV], d[F][IV];
#pragma unroll
            for (int f = 0; f < F; ++f)
              if (s0 + f * kPcgWarps < end) {
                const size_t ri = item_at(s0 + f * kPcgWarps);
                Load<double, IV>(R + ri, rv[f]);
                LoadRO<double, IV>(IDG + ri, d[f]);
              }
#pragma unroll
            for (int f = 0; f < F; ++f)
              if (s0 + f * kPcgWarps < end) {
                const size_t ri = item_at(s0 + f * kPcgWarps);
                double qv[IV], zv[IV];
                Load<double, IV>(q_at(s0 + f * kPcgWarps), qv);
#pragma unroll
                for (int j = 0; j < IV; ++j)
                  if (act[j])
                    rv[f][j] = rv[f][j] - al[j] * qv[j];
                precond(rv[f], d[f], zv);
                Store<double, IV>(R + ri, rv[f]);
                Store<double, IV>(Z + ri, zv);
#pragma unroll
                for (int j = 0; j < IV; ++j)
                  if (act[j]) {
                    v[0][j] += rv[f][j] * rv[f][j];
                    v[1][j] += rv[f][j] * zv[j];
                  }
              }
          }
        }
        WarpPart<KP, IV, GV, 2, false>(v, gv * kPcgWarps + warp, sm);
      }
    }
    if (warp == 0) {
      const int it = lane < KP ? lane : 0;
      const double rho = ctl.rho[it], thr = ctl.thr[it];
      NamedSync<1>();
      mark(2);
      FenceAcqRel();
      SendPartials<KP, GV, 2>(rank, mail, sm, red);
      if (lane < KP) // what this iteration leaves x behind by
        behind[lane] = !both && ((active >> lane) & 1u) ? ctl.alpha[lane] : 0.0;
      double sum[2];
      Collect<KP, GV, 2, true, 10>(a, rank, mail, sm, red, sum);
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
            ctl.resid[it] = -rr;
            at = rr <= thr * thr * (1.0 + 1e-14) && sqrt(rr) <= thr;
            if (at) {
              ctl.flag[it] = a.skip_verification ? 2 : 1;
            } else if (isfinite(rz) && rz > 0.0) {
              ctl.beta[it] = rz / rho;
              ctl.rho[it] = rz;
              ctl.restart[it] = 0;
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
      mail.Reset(red + 7, rank, threadIdx.x - 32, kPcgThreads - 32);
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
    double *const swap = pc; // pc: this iteration's direction
    pc = pn;
    pn = swap;

    // Items at the threshold: verify the true residual, then accept (scale x back) or
    // restart from it.
    if (state.y & kThreshold) {
      if (threadIdx.x < KP && ctl.resid[threadIdx.x] < 0.0)
        ctl.resid[threadIdx.x] = sqrt(-ctl.resid[threadIdx.x]);
      catch_up(pc);
      if (!a.skip_verification) {
        if (!GridBarrier(a, GridShape{ctas, rank}, epoch, sm))
          return;
        FG_GROUPS
        {
          double v[1][IV] = {};
          FG_STEPS
          {
            double rv[IV], t[IV];
            true_residual(st, t);
            Load<double, IV>(R + item_at(st), rv);
#pragma unroll
            for (int j = 0; j < IV; ++j)
              if (on(j) && ctl.flag[item0 + j] == 1) {
                rv[j] = t[j];
                v[0][j] += t[j] * t[j];
              }
            Store<double, IV>(R + item_at(st), rv);
          }
          WarpPart<KP, IV, GV, 1, false>(v, gv * kPcgWarps + warp, sm);
        }
        if (!BarrierReduce<KP, GV, 1, false>(a, rank, ctas, G, sm, epoch, buf, [&](int it, const double (&sum)[1]) {
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
      FG_GROUPS
      {
        double v[2][IV] = {};
        FG_STEPS
        {
          const size_t ri = item_at(st);
          double xv[IV], rv[IV], d[IV], zv[IV];
          Load<double, IV>(X + ri, xv);
          Load<double, IV>(R + ri, rv);
          Load<double, IV>(IDG + ri, d);
          precond(rv, d, zv);
          bool restart = false;
#pragma unroll
          for (int j = 0; j < IV; ++j) {
            const int f = on(j) ? ctl.flag[item0 + j] : 0;
            if (f == 2) {
              xv[j] = xv[j] * ctl.scale[item0 + j];
              if (!isfinite(xv[j]))
                v[1][j] += 1.0;
            }
            if (f == 3) {
              v[0][j] += rv[j] * zv[j];
              restart = true;
            }
          }
          Store<double, IV>(X + ri, xv);
          if (restart) // items that go on keep r, so their z is the same product again
            Store<double, IV>(Z + ri, zv);
        }
        WarpPart<KP, IV, GV, 2, false>(v, gv * kPcgWarps + warp, sm);
      }
      if (!BarrierReduce<KP, GV, 2, false>(a, rank, ctas, G, sm, epoch, buf, [&](int it, const double (&sum)[2]) {
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
                ctl.restart[it] = 1;
              }
            }
          }))
        return;
      active = __ballot_sync(0xffffffffu, lane < KP && ctl.active[lane < KP ? lane : 0]);
    }
  }

  catch_up(pc);
  // Iteration budget exhausted: report the true residual and scale the iterate back.
  if (active) {
    if (!GridBarrier(a, GridShape{ctas, rank}, epoch, sm))
      return;
    FG_GROUPS
    {
      double v[1][IV] = {};
      FG_STEPS
      {
        double t[IV];
        true_residual(st, t);
#pragma unroll
        for (int j = 0; j < IV; ++j)
          if (on(j))
            v[0][j] += t[j] * t[j];
      }
      WarpPart<KP, IV, GV, 1, false>(v, gv * kPcgWarps + warp, sm);
    }
    if (!BarrierReduce<KP, GV, 1, false>(a, rank, ctas, G, sm, epoch, buf, [&](int it, const double (&sum)[1]) {
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
    FG_GROUPS
    {
      double v[1][IV] = {};
      FG_STEPS
      {
        double xv[IV];
        Load<double, IV>(X + item_at(st), xv);
#pragma unroll
        for (int j = 0; j < IV; ++j)
          if (on(j)) {
            xv[j] = xv[j] * ctl.scale[item0 + j];
            if (!isfinite(xv[j]))
              v[0][j] += 1.0;
          }
        Store<double, IV>(X + item_at(st), xv);
      }
      WarpPart<KP, IV, GV, 1, false>(v, gv * kPcgWarps + warp, sm);
    }
    if (!BarrierReduce<KP, GV, 1, false>(a, rank, ctas, G, sm, epoch, buf, [&](int it, const double (&sum)[1]) {
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
#undef FG_GROUPS
#undef FG_STEPS

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
