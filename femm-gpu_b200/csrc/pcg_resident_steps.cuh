// pcg_resident_steps.cuh -- the resident PCG (pcg_resident.cuh) for systems of more than one
// row group per SM, as far as their share fits in shared memory: a CTA of 512 threads per SM
// for two row groups, whose warps take their steps of one group after the other.  (Two CTAs
// per SM would leave 64 registers a thread: spilled registers are dear here, since every
// fence empties L1.)  The vectors of a step sit in shared memory instead of registers, and
// where the operator's values do not fit beside the directions they are read from L2
// (STREAM).
//
// Measured on a B200, microseconds per CG iteration, PcgBody -> here (row-items = rows x
// padded items; about 330,000 fit):
//   40,000 rows: 4 items 14.7 -> 11.8, 8 items (values in L2) 19.4 -> 14.3
//   10,000 rows: 16 items 17.1 -> 11.9, 32 items (values in L2) 23.5 -> 14.8
//   159,201 rows, 1 item 12.8 -> 10.4; 9,480 rows with 20-entry rows, 8 items 16.0 -> 12.0
// Bounded by the gathers' latency and the two messages of each reduction.
#pragma once

#include "pcg_resident.cuh"

namespace fg
{
namespace
{

// Dynamic shared memory: a block per warp-step (x, r, q, p and 1/d of its rows), a block per
// operator entry of a step (p_j, a_ij unless STREAM, and the column of each row as a double's
// index), then the entry offsets of the CTA's steps at PcgArgs::resident_offset (STREAM:
// and the starts of their slices).  Offsets
// inside the blocks and their bytes:
template <int KP, int IV, bool SHARED, bool STREAM> struct ResidentStepsLayout {
  static constexpr int kRows = 32 * IV / KP; // of a warp-step
  static constexpr int kSlot = 32 * IV * 8;  // a lane's IV items, 32 lanes
  static constexpr int kX = 0, kR = kSlot, kQ = 2 * kSlot, kP = 3 * kSlot, kInv = 4 * kSlot;
  static constexpr int kStep = kInv + (SHARED ? kRows * 8 : kSlot);
  static constexpr int kValue = kSlot, kColumn = kSlot + (STREAM ? 0 : (SHARED ? kRows * 8 : kSlot));
  static constexpr int kEntry = kColumn + (kRows * 4 + 15) / 16 * 16;
};

// SHARED: one operator for all items (value_stride 1), else one per item.  STREAM: the
// values are read from L2.  GV: row groups per CTA.
template <int KP, int IV, bool SHARED, bool STREAM, int GV>
__global__ void __launch_bounds__(kPcgThreads, 1) PcgResidentStepsKernel(PcgArgs a)
{
  __shared__ ResidentShared<KP, GV> sm;
  __shared__ Control ctl;
  __shared__ Trace tr;
  __shared__ Mailboxes<KP> mail;
  extern __shared__ __align__(16) unsigned char resident_smem[];
  using L = ResidentStepsLayout<KP, IV, SHARED, STREAM>;
  constexpr int LR = KP / IV, S = 32 / LR;
  constexpr int U = 8; // entries of a row gathered together
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rank = static_cast<int>(blockIdx.x), ctas = static_cast<int>(gridDim.x), G = a.row_groups;
  const int item0 = (lane % LR) * IV, rl = lane / LR;
  const int WS = a.n_pad / S;
  // The CTA's steps [0, steps); its row group gv owns [gv ? mid : 0, gv ? steps : mid).
  auto first_step = [&](int g) { return static_cast<int>(static_cast<long long>(WS) * (g < G ? g : G) / G); };
  const int ws0 = first_step(rank * GV), mid = first_step(rank * GV + 1) - ws0;
  const int steps = first_step(rank * GV + GV) - ws0;
  unsigned epoch = 0;
  int buf = 0; // of the barrier-based reductions
  int32_t *off = reinterpret_cast<int32_t *>(resident_smem + a.resident_offset);
  // STREAM: where the steps' slices start in the global operator.  (Read from slice_off behind
  // a fence, each cost a trip to L2 before its step's values: 14.3 -> 14.0 us per iteration at
  // 40,000 rows and 8 items.)
  int32_t *slice_at = off + steps + 1;
  if (warp == 0) {
    // A running sum over the slice widths of the steps.
    int base = 0;
    for (int i = 0; i < steps; i += 32) {
      int sum = 0;
      if (i + lane < steps) {
        const int s = ((ws0 + i + lane) * S) >> 5, at = __ldg(a.slice_off + s);
        sum = (__ldg(a.slice_off + s + 1) - at) >> 5;
        if constexpr (STREAM)
          slice_at[i + lane] = at;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o)
          sum += y;
      }
      if (i + lane < steps)
        off[i + lane + 1] = base + sum;
      base += __shfl_sync(0xffffffffu, sum, 31);
    }
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
    mail.Init(a, ctas);
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
  // The lane's part of a step's vectors, of an entry's direction and value, and its column.
  const int entry0 = steps * L::kStep;
  auto row_at = [&](int st) { return (ws0 + st) * S + rl; };
  auto item_at = [&](int st) { return static_cast<size_t>(row_at(st)) * KP + item0; };
  auto vec = [&](int st, int k) {
    return reinterpret_cast<double *>(resident_smem + st * L::kStep + k + (SHARED && k == L::kInv ? rl * 8 : lane * IV * 8));
  };
  auto direction = [&](int e) {
    return reinterpret_cast<double *>(resident_smem + entry0 + e * L::kEntry + lane * IV * 8);
  };
  auto stored = [&](int e) {
    return reinterpret_cast<double *>(resident_smem + entry0 + e * L::kEntry + L::kValue + (SHARED ? rl * 8 : lane * IV * 8));
  };
  auto column = [&](int e) -> int32_t & {
    return *reinterpret_cast<int32_t *>(resident_smem + entry0 + e * L::kEntry + L::kColumn + rl * 4);
  };
  const double *vals = static_cast<const double *>(a.values);
  auto position = [&](int st) { // of the row's first entry in the global operator
    const int row = row_at(st);
    return static_cast<size_t>(STREAM ? slice_at[st] : __ldg(a.slice_off + (row >> 5))) + (row & 31);
  };
  // Value of entry e = the row's w-th, whose first is at pos.
  auto value = [&](size_t pos, int w, int e, double (&vv)[IV]) {
    if constexpr (STREAM) {
      LoadOperand<double, IV>(vals, pos + 32 * static_cast<size_t>(w), a.value_stride, SHARED ? 0 : 1, item0, vv);
    } else if constexpr (SHARED) {
      const double t = *stored(e);
#pragma unroll
      for (int j = 0; j < IV; ++j)
        vv[j] = t;
    } else {
      Load<double, IV>(stored(e), vv);
    }
  };
  auto precond = [&](int st, const double (&rv)[IV], double (&zv)[IV]) {
    double d[IV];
    if constexpr (SHARED) {
      const double t = *vec(st, L::kInv);
#pragma unroll
      for (int j = 0; j < IV; ++j)
        d[j] = t;
    } else {
      Load<double, IV>(vec(st, L::kInv), d);
    }
#pragma unroll
    for (int j = 0; j < IV; ++j)
      zv[j] = a.use_inverse ? rv[j] * d[j] : rv[j] / d[j];
  };
  auto send_z = [&](double *z, int st, const double (&zv)[IV]) {
    double m[IV];
#pragma unroll
    for (int j = 0; j < IV; ++j)
      m[j] = Sendable(zv[j]);
    StoreMessage<IV>(z + item_at(st), m);
  };
  auto reset_z = [&](double *z, int st) {
    double m[IV];
#pragma unroll
    for (int j = 0; j < IV; ++j)
      m[j] = UnsetValue();
    StoreMessage<IV>(z + item_at(st), m);
  };
// The row groups, and the steps of a group's warp that this warp stands for: a group's spare
// steps go to its first warps, so the two groups' first warps are different ones here, and
// not warp 0, which has the talking to do.
#define FG_GROUPS _Pragma("unroll 1") for (int gv = 0; gv < GV; ++gv)
  auto group_warp = [&](int gv) { return (warp + (gv ? kPcgWarps / 2 - 1 : kPcgWarps - 1)) & (kPcgWarps - 1); };
#define FG_STEPS                                                                                   \
  _Pragma("unroll 1") for (int st = (gv ? mid : 0) + group_warp(gv), end = GV == 1 || gv ? steps : mid; st < end; \
                           st += kPcgWarps)

  // Operator, inverse diagonal; validity (first invalid row decides) and RHS max-scaling.
  {
    FG_GROUPS
    {
      double v[2][IV] = {};
      FG_STEPS
      {
        const int row = row_at(st), len = __ldg(a.row_len + row), e0 = off[st], W = off[st + 1] - e0;
        const size_t base = position(st), ri = item_at(st);
        const double zero[IV] = {};
        for (int w = 0; w < W; ++w) {
          // Places past the row's end: the row's own column with the value 0 (STREAM: -1).
          const size_t pos = base + 32 * static_cast<size_t>(w);
          if (lane % LR == 0)
            column(e0 + w) = w < len ? __ldg(a.sell_col + pos) * KP : (STREAM ? -1 : row * KP);
          if constexpr (!STREAM) {
            if constexpr (SHARED) {
              if (lane % LR == 0)
                *stored(e0 + w) = w < len ? __ldg(vals + pos) : 0.0;
            } else {
              double vv[IV] = {};
              if (w < len)
                LoadStream<double, IV>(vals + pos * KP + item0, vv);
              Store<double, IV>(stored(e0 + w), vv);
            }
          }
          Store<double, IV>(direction(e0 + w), zero);
        }
        const double *src = static_cast<const double *>(a.use_inverse ? a.invd : a.diag);
        if constexpr (SHARED) {
          if (lane % LR == 0)
            *vec(st, L::kInv) = __ldg(src + row);
        } else {
          double d[IV];
          LoadRO<double, IV>(src + ri, d);
          Store<double, IV>(vec(st, L::kInv), d);
        }
        Store<double, IV>(vec(st, L::kX), zero);
        Store<double, IV>(vec(st, L::kP), zero);
        double dd[IV], bb[IV];
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
      WarpPart<KP, IV, GV, 2, true>(v, gv * kPcgWarps + group_warp(gv), sm);
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
        double bb[IV], rv[IV], zv[IV];
        Load<double, IV>(B + item_at(st), bb);
#pragma unroll
        for (int j = 0; j < IV; ++j)
          rv[j] = bb[j] / (ctl.scale[item0 + j] != 0.0 ? ctl.scale[item0 + j] : 1.0);
        precond(st, rv, zv);
        Store<double, IV>(vec(st, L::kR), rv);
        send_z(z_buffer(0), st, zv);
#pragma unroll
        for (int t = 1; t < 4; ++t)
          reset_z(z_buffer(t), st);
#pragma unroll
        for (int j = 0; j < IV; ++j)
          if (on(j)) {
            v[0][j] += rv[j] * rv[j];
            v[1][j] += rv[j] * zv[j];
          }
      }
      WarpPart<KP, IV, GV, 2, false>(v, gv * kPcgWarps + group_warp(gv), sm);
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

  // x of every row to its global copy, and the true residual b / s - A x from there.
  auto publish_x = [&] {
    FG_GROUPS
    FG_STEPS
    {
      double xv[IV];
      Load<double, IV>(vec(st, L::kX), xv);
      Store<double, IV>(GX + item_at(st), xv);
    }
  };
  auto true_residual = [&](int st, double (&t)[IV]) {
    const int e0 = off[st], W = off[st + 1] - e0;
    const size_t pos = position(st);
    double acc[IV] = {}, bb[IV];
    Load<double, IV>(B + item_at(st), bb);
    for (int w = 0; w < W; ++w) {
      const int c = column(e0 + w);
      if (c >= 0) {
        double gv[IV], vv[IV];
        Load<double, IV>(GX + c + item0, gv);
        value(pos, w, e0 + w, vv);
#pragma unroll
        for (int j = 0; j < IV; ++j)
          acc[j] = Fma(vv[j], gv[j], acc[j]);
      }
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

  // What the whole CTA goes on with after a reduction, left in sm.state by warp 0.
  auto decide = [&](unsigned threshold) {
    const unsigned active = __ballot_sync(0xffffffffu, lane < KP && ctl.active[lane < KP ? lane : 0]);
    if (lane == 0)
      sm.state = make_uint2(active, (*const_cast<volatile int *>(&sm.failed) ? kStop : 0u) | threshold);
  };
  unsigned active = __ballot_sync(0xffffffffu, lane < KP && ctl.active[lane < KP ? lane : 0]);
  const unsigned bits = (IV == 2 ? 3u : 1u) << item0; // of the lane's items
  int red = 0; // reductions so far
  if (warp == 0)
    mark(6);

#pragma unroll 1
  for (int iteration = 0; iteration < a.max_iterations && active; ++iteration) {
    double *const z = z_buffer(iteration), *const zn = z_buffer(iteration + 1);
    // Phase A: p = z + beta p of every entry's column and of the row, q = A p, p . q.  beta
    // is 0 and the directions finite (at first 0) where p restarts at z.
    {
      double be[IV];
#pragma unroll
      for (int j = 0; j < IV; ++j)
        be[j] = ctl.beta[item0 + j];
      FG_GROUPS
      {
        double v[1][IV] = {};
        if (active & bits) {
          FG_STEPS
          {
            const int e0 = off[st], W = off[st + 1] - e0;
            const size_t pos = STREAM ? position(st) : 0;
            double acc[IV] = {};
#pragma unroll 1
            for (int w0 = 0; w0 < W; w0 += U) {
              double g[U][IV], vv[U][IV];
              int c[U];
              unsigned char *const en = resident_smem + entry0 + (e0 + w0) * L::kEntry;
#pragma unroll
              for (int u = 0; u < U; ++u) {
                c[u] = -1;
                if (w0 + u < W)
                  c[u] = *reinterpret_cast<const int32_t *>(en + u * L::kEntry + L::kColumn + rl * 4);
              }
              auto gather = [&] {
#pragma unroll
                for (int u = 0; u < U; ++u)
                  if (c[u] >= 0)
                    LoadMessage<IV>(z + c[u] + item0, g[u]);
              };
              gather();
#pragma unroll
              for (int u = 0; u < U; ++u)
                if (w0 + u < W)
                  value(pos, w0 + u, e0 + w0 + u, vv[u]);
              auto missing = [&] {
                bool m = false;
#pragma unroll
                for (int u = 0; u < U; ++u)
                  m = m || (c[u] >= 0 && Missing<IV>(g[u]));
                return m;
              };
              if (missing()) { // z was sent before its owner's partial sums: rare
                const unsigned long long t0 = GlobalTimer();
                unsigned spin = 0;
                do
                  gather();
                while (missing() && PollAgain(a, spin, t0, sm));
              }
#pragma unroll
              for (int u = 0; u < U; ++u)
                if (c[u] >= 0) {
                  double *const d = reinterpret_cast<double *>(en + u * L::kEntry + lane * IV * 8);
                  double pj[IV];
                  Load<double, IV>(d, pj);
#pragma unroll
                  for (int j = 0; j < IV; ++j) {
                    pj[j] = Fma(be[j], pj[j], g[u][j]);
                    acc[j] = Fma(vv[u][j], pj[j], acc[j]);
                  }
                  Store<double, IV>(d, pj);
                }
            }
            // The row's own z = M^-1 r again: the very product its readers were sent.
            double rv[IV], zr[IV], pv[IV];
            Load<double, IV>(vec(st, L::kR), rv);
            Load<double, IV>(vec(st, L::kP), pv);
            precond(st, rv, zr);
#pragma unroll
            for (int j = 0; j < IV; ++j)
              pv[j] = Fma(be[j], pv[j], zr[j]);
            Store<double, IV>(vec(st, L::kP), pv);
            Store<double, IV>(vec(st, L::kQ), acc);
#pragma unroll
            for (int j = 0; j < IV; ++j)
              v[0][j] += pv[j] * acc[j];
          }
        }
        WarpPart<KP, IV, GV, 1, false>(v, gv * kPcgWarps + group_warp(gv), sm);
      }
    }
    if (warp == 0) {
      const int it = lane < KP ? lane : 0;
      const double rho = ctl.rho[it];
      NamedSync<1>();
      mark(0);
      SendPartials<KP, GV, 1>(rank, mail, sm, red);
      FenceAcqRel();
      double sum[1];
      Collect<KP, GV, 1>(a, rank, mail, sm, red, sum);
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
    const bool mine = active & bits;
    {
      double al[IV];
      bool act[IV];
#pragma unroll
      for (int j = 0; j < IV; ++j) {
        al[j] = ctl.alpha[item0 + j];
        act[j] = (active >> (item0 + j)) & 1u;
      }
      FG_GROUPS
      {
        double v[2][IV] = {};
        if (mine)
          FG_STEPS
          {
            double xv[IV], rv[IV], qv[IV], pv[IV], zv[IV];
            Load<double, IV>(vec(st, L::kR), rv);
            Load<double, IV>(vec(st, L::kQ), qv);
            Load<double, IV>(vec(st, L::kX), xv);
            Load<double, IV>(vec(st, L::kP), pv);
#pragma unroll
            for (int j = 0; j < IV; ++j)
              if (act[j]) {
                rv[j] = rv[j] - al[j] * qv[j];
                xv[j] = xv[j] + al[j] * pv[j];
              }
            precond(st, rv, zv);
            send_z(zn, st, zv);
            Store<double, IV>(vec(st, L::kX), xv);
            Store<double, IV>(vec(st, L::kR), rv);
#pragma unroll
            for (int j = 0; j < IV; ++j) {
              v[0][j] += rv[j] * rv[j];
              v[1][j] += rv[j] * zv[j];
            }
          }
        WarpPart<KP, IV, GV, 2, false>(v, gv * kPcgWarps + group_warp(gv), sm);
      }
    }
    // While the sums travel: reset the z of this iteration
    // (every CTA's phase A of it is over: the buffer serves iteration + 4) and the mailboxes
    // of reductions red + 5 (direct) or red + 7, and red + 6: last read at red - 3 or red - 1,
    // and red - 2, which all their readers have finished.
    if (warp == 0) {
      const int it = lane < KP ? lane : 0;
      const double rho = ctl.rho[it], thr = ctl.thr[it];
      NamedSync<1>();
      mark(2);
      SendPartials<KP, GV, 2>(rank, mail, sm, red);
      if (mine)
        FG_GROUPS
        FG_STEPS
        reset_z(z, st);
      double sum[2];
      Collect<KP, GV, 2>(a, rank, mail, sm, red, sum);
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
      if (mine)
        FG_GROUPS
        FG_STEPS
        reset_z(z, st);
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
        publish_x();
        if (!GridBarrier(a, GridShape{ctas, rank}, epoch, sm))
          return;
        FG_GROUPS
        {
          double v[1][IV] = {};
          FG_STEPS
          {
            double rv[IV], t[IV];
            true_residual(st, t);
            Load<double, IV>(vec(st, L::kR), rv);
#pragma unroll
            for (int j = 0; j < IV; ++j)
              if (on(j) && ctl.flag[item0 + j] == 1) {
                rv[j] = t[j];
                v[0][j] += t[j] * t[j];
              }
            Store<double, IV>(vec(st, L::kR), rv);
          }
          WarpPart<KP, IV, GV, 1, false>(v, gv * kPcgWarps + group_warp(gv), sm);
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
          double xv[IV], rv[IV], zv[IV];
          Load<double, IV>(vec(st, L::kX), xv);
          Load<double, IV>(vec(st, L::kR), rv);
          precond(st, rv, zv);
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
          Store<double, IV>(vec(st, L::kX), xv);
          if (restart) // items that go on keep r, so their z is the same product again
            send_z(zn, st, zv);
        }
        WarpPart<KP, IV, GV, 2, false>(v, gv * kPcgWarps + group_warp(gv), sm);
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
                ctl.beta[it] = 0.0;
              }
            }
          }))
        return;
      active = __ballot_sync(0xffffffffu, lane < KP && ctl.active[lane < KP ? lane : 0]);
    }
  }

  // Iteration budget exhausted: report the true residual and scale the iterate back.
  if (active) {
    publish_x();
    if (!GridBarrier(a, GridShape{ctas, rank}, epoch, sm))
      return;
    {
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
        WarpPart<KP, IV, GV, 1, false>(v, gv * kPcgWarps + group_warp(gv), sm);
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
    }
    FG_GROUPS
    {
      double v[1][IV] = {};
      FG_STEPS
      {
        double xv[IV];
        Load<double, IV>(vec(st, L::kX), xv);
#pragma unroll
        for (int j = 0; j < IV; ++j)
          if (on(j)) {
            xv[j] = xv[j] * ctl.scale[item0 + j];
            if (!isfinite(xv[j]))
              v[0][j] += 1.0;
          }
        Store<double, IV>(vec(st, L::kX), xv);
      }
      WarpPart<KP, IV, GV, 1, false>(v, gv * kPcgWarps + group_warp(gv), sm);
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
  publish_x();
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
