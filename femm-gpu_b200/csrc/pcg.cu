// pcg.cu -- kernel selection and the cooperative launch of the batched PCG
// (kernel template in pcg_kernel.cuh; instantiations in pcg_f64*.cu / pcg_f32*.cu).
#include "kernels.cuh"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace fg
{

const void *PcgKernelF64(int kp);
const void *PcgKernelF32(int kp);
const void *PcgKernelF64Block(int kp, int bs);
const void *PcgKernelF32Block(int kp, int bs);
const void *MultiPcgKernelF64(int kp);
const void *PcgKernelF64OneReduction(int kp);
const void *PcgKernelF64Wide(int kp);
// The resident form; *entry receives the shared-memory bytes of an operator entry of one
// warp-step.
const void *PcgKernelF64Resident(int kp, bool shared, int *entry);
// The same for several warp-steps per warp: `groups` (1 or 2) row groups per CTA, stream:
// values read from L2 (always with one); *step receives the bytes of a warp-step besides its
// entries.
const void *PcgKernelF64ResidentSteps(int kp, bool shared, bool stream, int groups, int *step, int *entry);
// The window form; q_global: q in global memory.
const void *PcgKernelF64Window(int kp, bool q_global);

namespace
{

constexpr int kPcgThreads = 512;
constexpr int kPcgWarps = kPcgThreads / 32;

const void *SelectKernel(int kp, int precision, int bs, bool one_reduction = false)
{
  if (one_reduction)
    return precision == 0 && bs == 0 ? PcgKernelF64OneReduction(kp) : nullptr;
  if (bs == 0)
    return precision == 0 ? PcgKernelF64(kp) : PcgKernelF32(kp);
  return precision == 0 ? PcgKernelF64Block(kp, bs) : PcgKernelF32Block(kp, bs);
}

int ItemsPerThread(int kp, int precision)
{
  if (precision == 0)
    return kp >= 2 ? 2 : 1;
  return kp >= 4 ? 4 : (kp >= 2 ? 2 : 1);
}

// Dynamic shared memory of the block-Jacobi staging buffer: U rows x KP items per warp.
size_t StagingBytes(int kp, int precision, int bs)
{
  if (bs == 0)
    return 0;
  const int rows_per_warp = 32 * ItemsPerThread(kp, precision) / kp;
  const int u = bs > rows_per_warp ? bs : rows_per_warp;
  return static_cast<size_t>(kPcgWarps) * u * kp * (precision == 0 ? 8 : 4);
}

// The most dynamic shared memory a launch of `kernel` may ask for on `device`: what a CTA may
// opt in to, less the kernel's static part; 0 on failure.  The attribute that admits it belongs
// to the kernel, which every plan and thread of the process launches, so it is set once, to
// this limit: set to a launch's own size it could be lowered by another thread's smaller launch
// before this one's.
size_t DynamicLimit(const void *kernel, int device)
{
  struct Known {
    const void *kernel;
    int device;
    size_t limit;
  };
  static Known known[512]; // more than there are kernels, for several devices; then it is set again
  static int count = 0;
  static std::mutex mutex;
  std::lock_guard<std::mutex> lock(mutex);
  for (int i = 0; i < count; ++i)
    if (known[i].kernel == kernel && known[i].device == device)
      return known[i].limit;
  cudaFuncAttributes attr;
  int most = 0;
  if (cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess ||
      cudaFuncGetAttributes(&attr, kernel) != cudaSuccess || attr.sharedSizeBytes >= static_cast<size_t>(most))
    return 0;
  const size_t limit = static_cast<size_t>(most) - attr.sharedSizeBytes;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(limit)) != cudaSuccess)
    return 0;
  if (count < static_cast<int>(sizeof(known) / sizeof(known[0])))
    known[count++] = Known{kernel, device, limit};
  return limit;
}

// Co-resident CTAs of one kernel shape (at most `cap` per SM), 0 on failure.
int KernelGrid(const void *kernel, size_t smem, int threads = kPcgThreads, int cap = 2)
{
  int device = 0, sms = 0, per_sm = 0;
  if (!kernel || cudaGetDevice(&device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
    return 0;
  if (smem > 0 && smem > DynamicLimit(kernel, device))
    return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess)
    return 0;
  return sms * (per_sm < cap ? per_sm : cap);
}

// Dynamic shared memory a launch may use for staging plus the column cache: two CTAs of
// 512 threads per SM must stay resident (228 KB per SM, about 12 KB static per CTA).
constexpr size_t kColumnCacheBudget = 104 * 1024;

// FG_PCG_VALUE_RING=0 in the environment turns the cp.async value ring off (for A/B timing).
bool ValueRingEnabled()
{
  static const bool enabled = [] {
    const char *v = std::getenv("FG_PCG_VALUE_RING");
    return !(v && v[0] == '0');
  }();
  return enabled;
}

// The column cache is off unless FG_PCG_COL_CACHE=1: beside the value ring its shared
// memory shrinks L1 and costs the update phase more than the cached indices save
// (measured on the 251k-node batch of 8: 69.9 us per CG iteration without, 73.2 with).
bool ColumnCacheEnabled()
{
  static const bool enabled = [] {
    const char *v = std::getenv("FG_PCG_COL_CACHE");
    return v && v[0] == '1';
  }();
  return enabled;
}

// FG_PCG_BLOCK=1024 selects the 1024-thread CTAs where a plan's autotuner has not chosen
// (read at every launch).
bool WideBlocksEnabled()
{
  const char *v = std::getenv("FG_PCG_BLOCK");
  return v && std::strcmp(v, "1024") == 0;
}

} // namespace

namespace
{
std::atomic<long long> g_wait_limit_ns{kDefaultWaitLimitNs};
} // namespace

long long PcgWaitLimitNs() { return g_wait_limit_ns.load(std::memory_order_relaxed); }

long long SetPcgWaitLimitNs(long long ns)
{
  return g_wait_limit_ns.exchange(ns > 0 ? ns : kDefaultWaitLimitNs, std::memory_order_relaxed);
}

bool PcgSupported(int kp, int precision, int block_size)
{
  return SelectKernel(kp, precision, block_size) != nullptr;
}

// Grid of the Jacobi kernels for kp items (the same for both precisions, so FP64 and
// FP32 launches of one batch reduce over the same partition); block-Jacobi launches use
// at most this many CTAs.
int PcgMaxGrid(int kp)
{
  int grid = 0;
  for (int precision = 0; precision < 2; ++precision) {
    const int g = KernelGrid(SelectKernel(kp, precision, 0), 0);
    if (g <= 0)
      return 0;
    grid = precision == 0 ? g : (g < grid ? g : grid);
  }
  return grid;
}

size_t PcgPartialsDoubles(int kp, int grid)
{
  // Double-buffered sums of the barrier-based reductions, then eight mailbox buffers of two sums
  // per item and row group and a line of results per CTA (pcg_resident.cuh); or the streamed
  // kernels' buffers (at most three sums of 32 items).  A mailbox buffer is counted as 64 KB at
  // least, more than narrow launches use: with a tighter buffer a plan's arrays lie at other
  // addresses, and how far a polled line is from the SMs that poll it depends on its address
  // (4,225 rows, one item: 4.64 and 4.72 ms a solve).
  const size_t k = static_cast<size_t>(kp), g = static_cast<size_t>(grid);
  const size_t sums = std::max<size_t>(2 * k * g, 8192), line = std::max<size_t>(2 * k, 16);
  return std::max<size_t>(4 * k * g + 8 * (sums + g * line), 2 * 96 * g);
}

namespace
{

// Row groups of a launch: kPcgWarps warps each, one warp-step of rows per warp at least,
// at most the co-resident CTAs of 512 threads.
int RowGroups(const PcgArgs &args, int max_grid)
{
  const int rows_per_warp = 32 * ItemsPerThread(args.kp, args.precision) / args.kp;
  const int grid = (args.n_pad / rows_per_warp + kPcgWarps - 1) / kPcgWarps;
  return grid > max_grid ? max_grid : (grid < 1 ? 1 : grid);
}

struct ResidentShape {
  const void *kernel = nullptr;
  int ctas = 0, offset = 0;
  size_t smem = 0;
};

// The resident form's launch, if the CTAs' shares fit in shared memory.  With an SM for every
// row group no warp has more than one warp-step and the state sits in registers (if the
// entries fit; wide rows may not); else a CTA has two row groups and the state sits in shared
// memory, the operator's values beside it or, where they do not fit, in L2.
bool ChooseResident(const PcgArgs &args, int groups, ResidentShape *out)
{
  if (args.resident_request != 0 || args.precision != 0 || args.blocks || args.one_reduction ||
      !args.host_slice_off)
    return false;
  int device = 0, sms = 0;
  if (cudaGetDevice(&device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
    return false;
  const int s = 32 * ItemsPerThread(args.kp, 0) / args.kp; // rows per warp-step
  const long long ws = args.n_pad / s;
  const bool shared = args.value_item == 0;
  const int per_cta = groups <= sms ? 1 : 2, ctas = (groups + per_cta - 1) / per_cta;
  // Where a few CTAs own many items' sums, each sums its own one after the other.  32 items on 3
  // CTAs (81 rows), 11 each: 3.37 ms a solve, streamed 2.75.  On 4 CTAs (121 rows), 8 each: 3.30,
  // streamed 3.45.  (One or two CTAs add up all items' sums themselves: 0.93, streamed 2.26.)
  if (ctas > 2 && args.kp > 8 * ctas)
    return false;
  // The least a CTA can need with the state in shared memory, before looking at the rows.
  int step = 0, entry = 0;
  if (!PcgKernelF64ResidentSteps(args.kp, shared, true, per_cta, &step, &entry) ||
      (ws / ctas) * (step + entry) > 227 * 1024)
    return false;
  // The forms to try, in order, and the bytes of the largest share of a CTA in each.  (No heap:
  // fg_csr_pcg_noalloc comes here, and nothing may throw.)
  struct Form {
    const void *kernel;
    bool stream;
    long long step, entry, data;
  } forms[3];
  int count = 0;
  if (per_cta == 1 && ws <= static_cast<long long>(groups) * kPcgWarps) {
    const void *kernel = PcgKernelF64Resident(args.kp, shared, &entry);
    forms[count++] = Form{kernel, false, 0, entry, 0};
  }
  for (const bool stream : {false, true}) {
    if (!stream && per_cta == 1)
      continue;
    const void *kernel = PcgKernelF64ResidentSteps(args.kp, shared, stream, per_cta, &step, &entry);
    forms[count++] = Form{kernel, stream, step, entry, 0};
  }
  long long most = 0; // steps of a CTA
  for (int c = 0; c < ctas; ++c) {
    const long long w0 = ws * (c * per_cta) / groups, w1 = ws * std::min(groups, (c + 1) * per_cta) / groups;
    long long entries = 0;
    for (long long w = w0; w < w1;) { // whole slices at a time
      const long long slice = (w * s) >> 5, end = ((slice + 1) * 32) / s;
      const long long n = (end < w1 ? end : w1) - w;
      entries += n * ((args.host_slice_off[slice + 1] - args.host_slice_off[slice]) / 32);
      w += n;
    }
    most = std::max(most, w1 - w0);
    for (int f = 0; f < count; ++f)
      forms[f].data = std::max(forms[f].data, (w1 - w0) * forms[f].step + entries * forms[f].entry);
  }
  for (int f = 0; f < count; ++f) {
    const Form &form = forms[f];
    const long long total = form.data + (most + 1 + (form.stream ? most : 0)) * 4;
    if (!form.kernel || total > 227 * 1024 ||
        KernelGrid(form.kernel, static_cast<size_t>(total), kPcgThreads, 1) < ctas)
      continue;
    *out = ResidentShape{form.kernel, ctas, static_cast<int>(form.data), static_cast<size_t>(total)};
    return true;
  }
  return false;
}

// The window form's launch, if the window (all rows that the operator's bandwidth can reach from
// a round's tile, and the tiles of the rounds in flight) fits in shared memory, with q beside it
// if that fits too.  `out` receives kernel, CTAs and shared memory; returns the window's rows,
// 0 if none.  Not where a CTA's two neighbourhoods have more rows than twice its own: filling
// the window would be most of the work.  (Who asks for the form has timed it: a plan's tuner.)
int ChooseWindow(const PcgArgs &args, int groups, ResidentShape *out)
{
  if (args.resident_request == 2 || args.precision != 0 || args.blocks || args.one_reduction || args.reliable ||
      args.bandwidth <= 0 || !args.host_slice_off || !args.value_item || !args.diag_item)
    return 0;
  const int s = 32 * ItemsPerThread(args.kp, 0) / args.kp, tile = kPcgWarps * s;
  const long long ws = args.n_pad / s, ctas = (groups + 1) / 2;
  const long long rows = 2ll * args.bandwidth + 4 * tile;
  if (ws < groups || 2ll * args.bandwidth > 2 * (ws / ctas) * s)
    return 0;
  long long most = 0;
  for (int c = 0; c < ctas; ++c) {
    const long long w0 = ws * (2 * c) / groups, w1 = ws * std::min(groups, 2 * c + 2) / groups;
    most = std::max(most, w1 - w0);
  }
  const long long ring = rows * args.kp * 8, q = most * s * args.kp * 8;
  for (const bool q_global : {false, true}) {
    const void *kernel = PcgKernelF64Window(args.kp, q_global);
    const long long total = ring + (q_global ? 0 : q);
    if (!kernel || total > 227 * 1024 || KernelGrid(kernel, static_cast<size_t>(total), kPcgThreads, 1) < ctas)
      continue;
    *out = ResidentShape{kernel, static_cast<int>(ctas), 0, static_cast<size_t>(total)};
    return static_cast<int>(rows);
  }
  return 0;
}

} // namespace

bool PcgWindow(const PcgArgs &args)
{
  ResidentShape shape;
  const int max_grid = PcgMaxGrid(args.kp);
  return max_grid > 0 && ChooseWindow(args, RowGroups(args, max_grid), &shape) > 0;
}

bool PcgResident(const PcgArgs &args)
{
  ResidentShape shape;
  const int max_grid = PcgMaxGrid(args.kp);
  return max_grid > 0 && ChooseResident(args, RowGroups(args, max_grid), &shape);
}

cudaError_t LaunchPcg(PcgArgs args, int *grid_out, int *block_out, cudaStream_t stream)
{
  const int bs = args.blocks ? args.block_size : 0;
  args.block_size = bs;
  const void *kernel = SelectKernel(args.kp, args.precision, bs, args.one_reduction != 0);
  if (args.one_reduction && (!args.t0 || !args.t1))
    return cudaErrorInvalidValue;
  if (!kernel)
    return cudaErrorInvalidValue;
  size_t smem = StagingBytes(args.kp, args.precision, bs);
  int max_grid = PcgMaxGrid(args.kp);
  const int own = KernelGrid(kernel, smem);
  if (own < max_grid)
    max_grid = own;
  if (max_grid <= 0)
    return cudaErrorInvalidConfiguration;
  const int iv = ItemsPerThread(args.kp, args.precision);
  const int rows_per_warp = 32 * iv / args.kp;
  const int warp_slices = args.n_pad / rows_per_warp;
  const int grid = RowGroups(args, max_grid);
  ResidentShape resident;
  bool on_chip = ChooseResident(args, grid, &resident);
  if (!on_chip && args.window_request == 1) {
    args.window_rows = ChooseWindow(args, grid, &resident);
    on_chip = args.window_rows > 0;
  }
  if (on_chip) {
    args.row_groups = grid;
    args.resident_offset = resident.offset;
    cudaError_t e = cudaMemsetAsync(args.barrier, 0, sizeof(unsigned), stream);
    if (e == cudaSuccess)
      e = cudaMemsetAsync(args.error, 0, sizeof(int32_t), stream);
    if (e != cudaSuccess)
      return e;
    void *params[] = {&args};
    e = cudaLaunchCooperativeKernel(resident.kernel, dim3(resident.ctas), dim3(kPcgThreads), params,
                                    resident.smem, stream);
    if (grid_out)
      *grid_out = resident.ctas;
    if (block_out)
      *block_out = kPcgThreads;
    return e;
  }
  // Wide CTAs (FP64 Jacobi): the same row groups two to a CTA of 1024 threads, one CTA per
  // SM -- the same rows, order and partial sums, so the same bits.
  const bool want_wide = args.block_request == 0 ? WideBlocksEnabled() : args.block_request == 1;
  const void *wide_kernel = want_wide && args.precision == 0 && bs == 0 && !args.one_reduction && grid % 2 == 0
                                ? PcgKernelF64Wide(args.kp)
                                : nullptr;
  const bool wide = wide_kernel && KernelGrid(wide_kernel, 0, 2 * kPcgThreads, 1) >= grid / 2;
  const int threads = wide ? 2 * kPcgThreads : kPcgThreads, warps = threads / 32;
  const int ctas = wide ? grid / 2 : grid, cap = wide ? 1 : 2;
  const size_t budget = wide ? 200 * 1024 : kColumnCacheBudget;
  if (wide)
    kernel = wide_kernel;
  // Value ring (16-byte item vectors, per-item operators): 2 stages x kRingEntries entries x
  // 32 lanes x 16 bytes per warp, after the block-Jacobi staging buffer.
  args.value_ring = 0;
  args.value_ring_offset = 0;
  const bool want_ring = args.ring_request == 0 ? ValueRingEnabled() : args.ring_request == 1;
  const bool ring_shape = (args.precision == 0 ? 8 : 4) * iv == 16 && args.value_item && want_ring;
  if (ring_shape) {
    const size_t offset = (smem + 15) / 16 * 16;
    const size_t total = offset + static_cast<size_t>(warps) * 2 * kRingEntries * 32 * 16;
    if (total <= budget && KernelGrid(kernel, total, threads, cap) >= ctas) {
      args.value_ring = 1;
      args.value_ring_offset = static_cast<int32_t>(offset);
      smem = total;
    }
  }
  // Column-index cache: the largest slice range any CTA's rows touch, if it fits in the
  // shared memory that still leaves the grid co-resident.
  args.col_cache = 0;
  args.col_cache_offset = 0;
  const bool want_cache = args.col_cache_request == 0 ? ColumnCacheEnabled() : args.col_cache_request == 1;
  if (args.host_slice_off && want_cache) {
    size_t most = 0;
    for (int g = 0; g < ctas; ++g) {
      const long long w0 = static_cast<long long>(warp_slices) * g / ctas;
      const long long w1 = static_cast<long long>(warp_slices) * (g + 1) / ctas;
      if (w1 <= w0)
        continue;
      const long long s0 = (w0 * rows_per_warp) >> 5, s1 = (w1 * rows_per_warp - 1) >> 5;
      const size_t p = static_cast<size_t>(args.host_slice_off[s1 + 1] - args.host_slice_off[s0]);
      most = p > most ? p : most;
    }
    const size_t offset = (smem + 15) / 16 * 16;
    const size_t total = offset + most * sizeof(int32_t);
    if (total <= budget && KernelGrid(kernel, total, threads, cap) >= ctas) {
      args.col_cache = 1;
      args.col_cache_offset = static_cast<int32_t>(offset);
      smem = total;
    }
  }
  cudaError_t e = cudaMemsetAsync(args.barrier, 0, sizeof(unsigned), stream);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(args.error, 0, sizeof(int32_t), stream);
  if (e != cudaSuccess)
    return e;
  void *params[] = {&args};
  e = cudaLaunchCooperativeKernel(kernel, dim3(ctas), dim3(threads), params, smem, stream);
  if (grid_out)
    *grid_out = ctas;
  if (block_out)
    *block_out = threads;
  return e;
}

size_t MultiPcgRingBytes(int kp)
{
  // The value ring carries 16-byte item vectors: FP64 with two items per thread.
  const int iv = ItemsPerThread(kp, 0);
  if (8 * iv != 16 || !ValueRingEnabled())
    return 0;
  return static_cast<size_t>(kPcgWarps) * 2 * kRingEntries * 32 * 16;
}

int MultiPcgMaxGrid(int kp)
{
  const void *kernel = MultiPcgKernelF64(kp);
  return kernel ? KernelGrid(kernel, MultiPcgRingBytes(kp)) : 0;
}

cudaError_t LaunchMultiPcg(PcgGroups t, int kp, int ctas, cudaStream_t stream)
{
  const void *kernel = MultiPcgKernelF64(kp);
  const int max_grid = MultiPcgMaxGrid(kp);
  if (!kernel || ctas < 1 || ctas > max_grid)
    return cudaErrorInvalidConfiguration;
  void *params[] = {&t};
  return cudaLaunchCooperativeKernel(kernel, dim3(ctas), dim3(kPcgThreads), params, MultiPcgRingBytes(kp),
                                     stream);
}

} // namespace fg
