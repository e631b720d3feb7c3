// Launches of the spread solve (spread_solve.cuh): layouts made and uploaded at first use, one
// factor's solves, and the complex batch over many factors.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "capi_common.hpp"
#include "spread_launch.hpp"
#include "spread_solve.cuh"

namespace yb {

namespace {

// The largest condition (the norms of what a map inverts, for the Schur complement a bound, and of the
// map) with which the top is taken densely.
constexpr double kSpreadTopCondition = 1e9;
constexpr size_t kSpreadWorkBytes = size_t(2) << 30;  // the largest work array one run of launches fills
// FP32 takes two right-hand sides a lane from this many on (below, more warps are worth more than
// fewer instructions; 10,000-bus B': 127 against 147 us at 999, 375 against 400 us at 4,096).
constexpr int64_t kSpreadPairCount = 2048;

template <class V> struct DeviceValue {
  using type = double;
  static double from(double v) { return v; }
};
template <> struct DeviceValue<host::c128> {
  using type = cplx<double>;
  static cplx<double> from(const host::c128 &v) { return from_std<double>(v); }
};

template <class V> std::vector<typename DeviceValue<V>::type> device_values(const std::vector<V> &v) {
  std::vector<typename DeviceValue<V>::type> out(std::max<size_t>(v.size(), 1));
  for (size_t i = 0; i < v.size(); ++i) out[i] = DeviceValue<V>::from(v[i]);
  return out;
}
std::vector<int32_t> some(const std::vector<int32_t> &v) { return v.empty() ? std::vector<int32_t>{0} : v; }

template <class T, bool BATCH> void allow_smem(const yb_gpu *gpu);
template <class V>
std::unique_ptr<DeviceSpread> make_spread(const Plan<V> &plan, int kind, int value_bytes, int64_t groups, const yb_gpu *gpu,
                                          cudaStream_t s) {
  using M = typename DeviceValue<V>::type;
  // the blocks an SM holds by the kernel's registers; where a layout's slots let it hold fewer, the cut
  // is chosen again for those
  const int most = value_bytes == 16 ? spread_blocks<cplx<double>>() : value_bytes == 8 ? spread_blocks<double>() : spread_blocks<float>();
  SpreadLayout<V> lay = spread_layout(plan, value_bytes, groups, gpu->sm_count, most);
  const size_t smem = (value_bytes == 16 ? spread_smem<cplx<double>>(lay.slots, kSpreadWarps)
                       : value_bytes == 8 ? spread_smem<double>(lay.slots, kSpreadWarps)
                                          : spread_smem<float>(lay.slots, kSpreadWarps)) + 1024;
  const int fit = std::max<int>(1, (int)((size_t)gpu->smem_per_sm / smem));
  if (fit < most) lay = spread_layout(plan, value_bytes, groups, gpu->sm_count, fit);
  if constexpr (std::is_same_v<V, double>)
    value_bytes == 8 ? allow_smem<double, false>(gpu) : (allow_smem<float, false>(gpu), allow_smem<pair2<float>, false>(gpu));
  else
    value_bytes == 16 ? allow_smem<cplx<double>, true>(gpu) : allow_smem<cplx<float>, true>(gpu);
  auto d = std::make_unique<DeviceSpread>();
  d->n = lay.n, d->tasks = lay.tasks, d->top = lay.top, d->slots = lay.slots, d->partials = lay.partials;
  d->domains = lay.domains, d->blob_bytes = (int64_t)lay.blob.size();
  d->blob.upload(lay.blob, s);
  d->task_row.upload(lay.task_row, s);
  d->fwd_page.upload(lay.fwd_page, s), d->bwd_page.upload(lay.bwd_page, s);
  d->in_pos.upload(lay.in_pos, s), d->out_pos.upload(lay.out_pos, s);
  d->part_ptr.upload(lay.part_ptr, s);
  d->host_out_pos = lay.out_pos;
  const int32_t t = lay.top;
  if (t > 0) {
    const size_t blocks = (size_t)(t + kSpreadTopRows - 1) / kSpreadTopRows;
    const size_t m_values = blocks * t * kSpreadTopRows;
    DeviceArray<int32_t> lp, lc, up, uc;
    DeviceArray<M> lv, ld, uv, ud, scratch((size_t)((t + 31) / 32) * t * 32);
    DeviceArray<unsigned long long> norm(2);
    lp.upload(lay.l_ptr, s), lc.upload(some(lay.l_col), s), up.upload(lay.u_ptr, s), uc.upload(some(lay.u_col), s);
    lv.upload(device_values(lay.l_val), s), ld.upload(device_values(lay.l_dinv), s);
    uv.upload(device_values(lay.u_val), s), ud.upload(device_values(lay.u_dinv), s);
    cuda_check(cudaMemsetAsync(norm.get(), 0, 2 * sizeof(unsigned long long), s), "clear the norms");
    auto map = [&](auto kernel, DeviceArray<uint8_t> &to, int at) {
      to.resize(m_values * sizeof(M));
      M *m = reinterpret_cast<M *>(to.get());
      cuda_check(cudaMemsetAsync(m, 0, m_values * sizeof(M), s), "clear a map");
      kernel<<<(unsigned)((t + 31) / 32), 32, 0, s>>>(t, lp.get(), lc.get(), lv.get(), ld.get(), up.get(), uc.get(), uv.get(),
                                                      ud.get(), scratch.get(), m);
      cuda_check(cudaGetLastError(), "spread_map_kernel launch");
      spread_norm_kernel<M><<<(unsigned)((t + 255) / 256), 256, 0, s>>>(t, m, norm.get() + at);
      cuda_check(cudaGetLastError(), "spread_norm_kernel launch");
    };
    d->split = kind == YB_LU;
    if (d->split)
      map(spread_map_kernel<M, true, false>, d->m, 0), map(spread_map_kernel<M, false, true>, d->m2, 1);
    else
      map(spread_map_kernel<M, true, true>, d->m, 0);
    unsigned long long bits[2] = {};
    cuda_check(cudaMemcpyAsync(bits, norm.get(), sizeof bits, cudaMemcpyDeviceToHost, s), "download the norms");
    cuda_check(cudaStreamSynchronize(s), "the top's maps");
    double norms[2];
    std::memcpy(norms, bits, sizeof norms);
    d->top_condition = d->split ? std::max(norms[0] * lay.l_norm, norms[1] * lay.u_norm) : norms[0] * lay.s_norm;
    if (!(d->top_condition <= kSpreadTopCondition)) return nullptr;
  }
  cuda_check(cudaStreamSynchronize(s), "spread layout upload");
  return d;
}

SpreadNet net_of(const DeviceSpread *d, int64_t groups, int64_t count) {
  SpreadNet net{};
  net.n = d->n, net.tasks = d->tasks, net.top = d->top, net.partials = d->partials;
  net.blob = d->blob.get(), net.fwd_page = d->fwd_page.get(), net.bwd_page = d->bwd_page.get();
  net.task_row = d->task_row.get(), net.part_ptr = d->part_ptr.get();
  net.in_pos = d->in_pos.get(), net.out_pos = d->out_pos.get(), net.m = d->m.get(), net.m2 = d->m2.get();
  net.groups = groups, net.count = count;
  return net;
}

bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  cuda_check(cudaStreamIsCapturing(s, &status), "cudaStreamIsCapturing");
  return status != cudaStreamCaptureStatusNone;
}

// A launch that may start its blocks while the kernel before it in the stream finishes (`overlap`;
// every kernel of this file waits for it before it reads what another wrote).
template <class... P, class... A>
void launch(void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t s, bool overlap, const A &...args) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid), c.blockDim = dim3(threads), c.dynamicSmemBytes = smem, c.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &attr, c.numAttrs = overlap ? 1 : 0;
  cuda_check(cudaLaunchKernelEx(&c, kernel, args...), "spread launch");
}

// Lets the sweeps take as much shared memory as a block may have (once per layout, always the same).
template <class T, bool BATCH> void allow_smem(const yb_gpu *gpu) {
  for (auto kernel : {spread_sweep_kernel<T, false, BATCH>, spread_sweep_kernel<T, true, BATCH>}) {
    cudaFuncAttributes attr{};
    cuda_check(cudaFuncGetAttributes(&attr, kernel), "cudaFuncGetAttributes");
    cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(gpu->smem_optin - attr.sharedSizeBytes)),
               "cudaFuncSetAttribute");
    cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared),
               "cudaFuncSetAttribute");
  }
}

// The ways the top's product splits M's columns: one where tiles of 16 rows by 32 columns, eight warps a
// block, fill the SMs at least twice (tiles: over all groups), else as many as a block can.
template <class T> int split_top(int64_t tiles, const yb_gpu *gpu) {
  return tiles >= 2 * spread_top_warps<T, 1>() * (int64_t)gpu->sm_count ? 1 : spread_split<T>();
}
int64_t top_tiles(const DeviceSpread *d) { return (d->top + 15) / 16; }
template <class T> int64_t top_blocks(const DeviceSpread *d, int split) {
  const int rows = split > 1 ? 16 : 16 * spread_top_warps<T, 1>();
  return (d->top + rows - 1) / rows;
}

// The groups per block of the sweeps: kSpreadWarps, fewer with fewer groups or when the slots do not
// fit shared memory.
template <class T> int sweep_warps(int32_t slots, int64_t groups, const yb_gpu *gpu) {
  int warps = (int)std::min<int64_t>(kSpreadWarps, groups);
  while (warps > 1 && spread_smem<T>(slots, warps) > (size_t)gpu->smem_optin) --warps;
  return warps;
}

template <class T> void one_sweeps(const DeviceSpread *d, const SpreadArgs &a, const yb_gpu *gpu, cudaStream_t s) {
  const int64_t groups = a.one.groups;
  const int warps = sweep_warps<T>(a.slots, groups, gpu);
  const size_t smem = spread_smem<T>(a.slots, warps);
  const unsigned grid = (unsigned)(d->tasks * ((groups + warps - 1) / warps));
  launch(spread_sweep_kernel<T, false, false>, grid, warps * 32, smem, s, true, a);
  if (d->top > 0) {
    launch(spread_sum_kernel<T, false>, (unsigned)(groups * ((d->top + 7) / 8)), 256, 0, s, true, a);
    const int64_t columns = groups * SpreadLane<T>::N;
    const int split = split_top<T>(columns * top_tiles(d), gpu);
    const unsigned blocks = (unsigned)(columns * top_blocks<T>(d, split));
    auto top = [&](auto phase) {
      constexpr int PHASE = decltype(phase)::value;
      if (split > 1)
        launch(spread_top_kernel<T, false, spread_split<T>(), PHASE>, blocks, spread_top_warps<T, spread_split<T>()>() * 32, 0, s, true, a);
      else
        launch(spread_top_kernel<T, false, 1, PHASE>, blocks, spread_top_warps<T, 1>() * 32, 0, s, true, a);
    };
    if (d->split)
      top(std::integral_constant<int, 1>()), top(std::integral_constant<int, 2>());
    else
      top(std::integral_constant<int, 0>());
  }
  launch(spread_sweep_kernel<T, true, false>, grid, warps * 32, smem, s, true, a);
}

// The partial array of `groups` groups: the partials and the top's solutions in T, then the top's
// right-hand sides (and, with two maps, what is between them) in full precision (every part a multiple of 128 bytes); at least one line.
template <class T> size_t partial_bytes(const DeviceSpread *d, int64_t groups) {
  return (size_t)groups * 32 * ((size_t)(d->partials + d->top) * sizeof(T) + (size_t)d->top * (d->split ? 2 : 1) * sizeof(typename SpreadLane<T>::Math)) + 128;
}
template <class T> void set_partial(SpreadNet &net, uint8_t *p) {
  net.partial = p;
  uint8_t *r = p + (size_t)net.groups * 32 * (size_t)(net.partials + net.top) * sizeof(T);
  net.r = r, net.r2 = r + (size_t)net.groups * 32 * net.top * sizeof(typename SpreadLane<T>::Math);
}

}  // namespace

DeviceSpread *spread_for(yb_factor *f, int value_bytes, int64_t groups, cudaStream_t stream) {
  const std::lock_guard<std::mutex> lock(f->spread_mutex);
  int64_t most = groups;  // a layout for groups up to each number of three significant bits
  for (int64_t unit = 1; most > 8 * unit || most % unit; unit *= 2) most = (most + 2 * unit - 1) / (2 * unit) * (2 * unit);
  const auto key = std::make_pair(value_bytes, most);
  auto it = f->spreads.find(key);
  if (it != f->spreads.end()) return it->second.get();
  if (capturing(stream)) {  // nothing may be made now: the nearest layout there is, if any
    auto near = f->spreads.end();
    for (auto i = f->spreads.begin(); i != f->spreads.end(); ++i)
      if (i->first.first == value_bytes && i->second &&
          (near == f->spreads.end() || std::abs(i->first.second - most) < std::abs(near->first.second - most)))
        near = i;
    return near == f->spreads.end() ? nullptr : near->second.get();
  }
  std::unique_ptr<DeviceSpread> d;
  try {
    d = f->is_complex ? make_spread(f->cplan, f->kind, value_bytes, most, f->gpu, stream)
                      : make_spread(f->plan, f->kind, value_bytes, most, f->gpu, stream);
    const int32_t limit = f->is_complex ? kSpreadAutoSlotsComplex : kSpreadAutoSlots;
    if (d && d->slots > limit) d.reset();
  } catch (const host::Error &e) {
    if (e.status != host::kInvalidArgument && e.status != host::kTooLarge) throw;
    d.reset();
  }
  auto *out = d.get();
  f->spreads.emplace(key, std::move(d));
  return out;
}

template <class T>
void spread_sweeps(yb_factor *f, DeviceSpread *d, T *work, T *xout, int64_t groups, const uint8_t *group_active,
                   cudaStream_t stream) {
  f->lane_partial.reserve(partial_bytes<T>(d, groups));
  SpreadArgs a{};
  a.one = net_of(d, groups, groups * 32);
  a.one.work = work, a.one.xout = xout;
  set_partial<T>(a.one, f->lane_partial.get());
  a.one.group_active = group_active;
  a.slots = d->slots;
  one_sweeps<T>(d, a, f->gpu, stream);
}
template void spread_sweeps<float>(yb_factor *, DeviceSpread *, float *, float *, int64_t, const uint8_t *, cudaStream_t);

namespace {

// The workspace a solve on `stream` takes, with at least the bytes asked for; null under capture when
// the stream has none that large. The mutex is held.
SpreadWork *work_for(yb_factor *f, size_t work_bytes, size_t partial, cudaStream_t stream) {
  SpreadWork *w = nullptr;
  for (auto &i : f->spread_work)
    if (i->stream == stream) w = i.get();
  if (capturing(stream)) return w && w->work.size() >= work_bytes && w->partial.size() >= partial ? w : nullptr;
  if (!w)
    for (auto &i : f->spread_work)
      if (!w && cudaEventQuery(i->done) == cudaSuccess) w = i.get();
  cudaGetLastError();  // a workspace still in use is no error
  if (!w && f->spread_work.size() < SpreadWork::kMost) {
    f->spread_work.push_back(std::make_unique<SpreadWork>());
    w = f->spread_work.back().get();
    cuda_check(cudaEventCreateWithFlags(&w->done, cudaEventDisableTiming), "cudaEventCreate");
  }
  if (!w) w = std::min_element(f->spread_work.begin(), f->spread_work.end(), [](auto &a, auto &b) { return a->used < b->used; })->get();
  cuda_check(cudaStreamWaitEvent(stream, w->done, 0), "cudaStreamWaitEvent");
  w->stream = stream;
  w->used = ++f->spread_solves;
  w->work.reserve(work_bytes), w->partial.reserve(partial);  // a larger array: the device is idle past the old one's free
  return w;
}

template <class L>
bool solve_lanes(yb_factor *f, DeviceSpread *d, const double *b, int64_t ldb, double *x, int64_t ldx, int64_t count,
                 cudaStream_t stream) {
  constexpr int64_t COLS = 32 * SpreadLane<L>::N;  // columns of a group
  const int64_t n = f->n, groups_all = (count + COLS - 1) / COLS;
  const size_t group_bytes = (size_t)n * 32 * sizeof(L), pad_bytes = 2 * kSpreadPad * 32 * sizeof(L);
  const int64_t per_run = std::max<int64_t>(1, std::min<int64_t>(groups_all, (int64_t)(kSpreadWorkBytes / group_bytes)));
  // small solves keep room for 1,536 right-hand sides (64 on factors of large order), so that any of
  // them can be captured once one has run
  const int64_t room = std::max<int64_t>(per_run, ((n <= 12800 ? 1536 : 64) + COLS - 1) / COLS);
  const std::lock_guard<std::mutex> lock(f->spread_mutex);
  SpreadWork *w = work_for(f, (size_t)(capturing(stream) ? per_run : room) * group_bytes + pad_bytes,
                           partial_bytes<L>(d, capturing(stream) ? per_run : room), stream);
  if (!w) return false;
  L *work = reinterpret_cast<L *>(w->work.get()) + kSpreadPad * 32;
  for (int64_t g0 = 0; g0 < groups_all; g0 += per_run) {
    const int64_t groups = std::min(per_run, groups_all - g0);
    SpreadArgs a{};
    a.one = net_of(d, groups, std::min(count - g0 * COLS, groups * COLS));
    a.one.work = a.one.xout = work;
    set_partial<L>(a.one, w->partial.get());
    a.one.b = b + g0 * COLS * ldb, a.one.ldb = ldb, a.one.x = x + g0 * COLS * ldx, a.one.ldx = ldx;
    a.slots = d->slots;
    const unsigned io = (unsigned)((groups * ((n + 31) / 32) + kSpreadIoWarps - 1) / kSpreadIoWarps);
    cudaEvent_t *ev = lane_timing_slot(f);
    if (ev) cuda_check(cudaEventRecord(ev[0], stream), "cudaEventRecord");
    launch(spread_in_kernel<L, false>, io, kSpreadIoWarps * 32, 0, stream, true, a);
    if (ev) cuda_check(cudaEventRecord(ev[1], stream), "cudaEventRecord");
    one_sweeps<L>(d, a, f->gpu, stream);
    if (ev) cuda_check(cudaEventRecord(ev[2], stream), "cudaEventRecord");
    launch(spread_out_kernel<L, false, false>, io, kSpreadIoWarps * 32, 0, stream, true, a);
    if (ev) cuda_check(cudaEventRecord(ev[3], stream), "cudaEventRecord");
  }
  if (!capturing(stream)) cuda_check(cudaEventRecord(w->done, stream), "cudaEventRecord");
  return true;
}

}  // namespace

template <class T>
bool spread_solve(yb_factor *f, const double *b, int64_t ldb, double *x, int64_t ldx, int64_t count, cudaStream_t stream) {
  DeviceSpread *d = spread_for(f, (int)sizeof(T), (count + 31) / 32, stream);
  if (!d) return false;
  if (sizeof(T) == 4 && count >= kSpreadPairCount) return solve_lanes<pair2<float>>(f, d, b, ldb, x, ldx, count, stream);
  return solve_lanes<T>(f, d, b, ldb, x, ldx, count, stream);
}
template bool spread_solve<double>(yb_factor *, const double *, int64_t, double *, int64_t, int64_t, cudaStream_t);
template bool spread_solve<float>(yb_factor *, const double *, int64_t, double *, int64_t, int64_t, cudaStream_t);

template <class R>
void spread_batch(const std::vector<SpreadSystem> &systems, bool add, SpreadBatchWork &w, cudaStream_t stream) {
  using T = cplx<R>;
  const size_t k = systems.size();
  if (k == 0) return;
  const yb_gpu *gpu = systems[0].factor->gpu;
  std::vector<SpreadNet> nets(k);
  size_t work_values = 0, part_bytes = 0;
  int64_t top_total = 0;
  int32_t slots = 0;
  int64_t most_groups = 1;
  for (const SpreadSystem &sys : systems) {
    const int64_t groups = (sys.count + 31) / 32;
    work_values += (size_t)groups * sys.layout->n * 32 + 2 * kSpreadPad * 32;
    part_bytes += partial_bytes<T>(sys.layout, groups);
    top_total += groups * top_tiles(sys.layout);
    slots = std::max(slots, sys.layout->slots);
    most_groups = std::max(most_groups, groups);
  }
  w.work.reserve(work_values * sizeof(T)), w.partial.reserve(part_bytes);
  const int split = split_top<T>(top_total, gpu);
  const int warps = sweep_warps<T>(slots, most_groups, gpu);
  // the blocks' items: the gather's and scatter's, the sweeps' (each network's tasks are longest
  // first; the networks' tasks by rank, so every network's long tasks start early), the top's
  std::vector<SpreadItem> io, sweep, sum, top;
  T *work = reinterpret_cast<T *>(w.work.get());
  uint8_t *partial = w.partial.get();
  int32_t most_tasks = 0;
  for (size_t i = 0; i < k; ++i) {
    const SpreadSystem &sys = systems[i];
    const DeviceSpread *d = sys.layout;
    const int64_t groups = (sys.count + 31) / 32;
    SpreadNet &net = nets[i];
    net = net_of(d, groups, sys.count);
    net.work = net.xout = work + kSpreadPad * 32;
    set_partial<T>(net, partial);
    net.b = sys.b, net.ldb = d->n, net.x = sys.x, net.ldx = d->n;
    work += (size_t)groups * d->n * 32 + 2 * kSpreadPad * 32;
    partial += partial_bytes<T>(d, groups);
    most_tasks = std::max(most_tasks, d->tasks);
    const int32_t row_blocks = (int32_t)((d->n + 32 * kSpreadIoWarps - 1) / (32 * kSpreadIoWarps));
    for (int64_t g = 0; g < groups; ++g) {
      for (int32_t c = 0; c < row_blocks; ++c) io.push_back({(int32_t)i, c, (int32_t)g, 0});
      for (int32_t c = 0; c < (d->top + 7) / 8; ++c) sum.push_back({(int32_t)i, c, (int32_t)g, 0});
      for (int32_t c = 0; c < top_blocks<T>(d, split); ++c) top.push_back({(int32_t)i, c, (int32_t)g, 0});
    }
  }
  for (int32_t t = 0; t < most_tasks; ++t)
    for (size_t i = 0; i < k; ++i)
      if (t < systems[i].layout->tasks)
        for (int64_t g = 0; g < nets[i].groups; g += warps) sweep.push_back({(int32_t)i, t, (int32_t)g, 0});
  const size_t n_io = io.size(), n_sweep = sweep.size(), n_sum = sum.size(), n_top = top.size();
  if (n_io == 0) return;
  std::vector<uint8_t> all(sizeof(SpreadNet) * k + sizeof(SpreadItem) * (n_io + n_sweep + n_sum + n_top));
  const size_t net_bytes = sizeof(SpreadNet) * k;
  std::memcpy(all.data(), nets.data(), net_bytes);
  auto *items = reinterpret_cast<SpreadItem *>(all.data() + net_bytes);
  std::copy(io.begin(), io.end(), items);
  std::copy(sweep.begin(), sweep.end(), items + n_io);
  std::copy(sum.begin(), sum.end(), items + n_io + n_sweep);
  std::copy(top.begin(), top.end(), items + n_io + n_sweep + n_sum);
  w.args.reserve(all.size());
  cuda_check(cudaMemcpyAsync(w.args.get(), all.data(), all.size(), cudaMemcpyHostToDevice, stream), "upload the batch");
  const auto *d_items = reinterpret_cast<const SpreadItem *>(w.args.get() + net_bytes);
  SpreadArgs a{};
  a.nets = reinterpret_cast<const SpreadNet *>(w.args.get());
  a.slots = slots;
  const size_t smem = spread_smem<T>(slots, warps);
  a.items = d_items;
  launch(spread_in_kernel<T, true>, (unsigned)n_io, kSpreadIoWarps * 32, 0, stream, true, a);
  a.items = d_items + n_io;
  launch(spread_sweep_kernel<T, false, true>, (unsigned)n_sweep, warps * 32, smem, stream, true, a);
  if (n_top) {
    a.items = d_items + n_io + n_sweep;
    launch(spread_sum_kernel<T, true>, (unsigned)n_sum, 256, 0, stream, true, a);
    a.items = d_items + n_io + n_sweep + n_sum;
    auto phase = [&](auto one) {  // complex factors are LU factors: two maps
      constexpr int PHASE = decltype(one)::value;
      if (split > 1)
        launch(spread_top_kernel<T, true, spread_split<T>(), PHASE>, (unsigned)n_top, spread_top_warps<T, spread_split<T>()>() * 32, 0, stream, true, a);
      else
        launch(spread_top_kernel<T, true, 1, PHASE>, (unsigned)n_top, spread_top_warps<T, 1>() * 32, 0, stream, true, a);
    };
    phase(std::integral_constant<int, 1>()), phase(std::integral_constant<int, 2>());
  }
  a.items = d_items + n_io;
  launch(spread_sweep_kernel<T, true, true>, (unsigned)n_sweep, warps * 32, smem, stream, true, a);
  a.items = d_items;
  if (add)
    launch(spread_out_kernel<T, true, true>, (unsigned)n_io, kSpreadIoWarps * 32, 0, stream, true, a);
  else
    launch(spread_out_kernel<T, true, false>, (unsigned)n_io, kSpreadIoWarps * 32, 0, stream, true, a);
}
template void spread_batch<double>(const std::vector<SpreadSystem> &, bool, SpreadBatchWork &, cudaStream_t);
template void spread_batch<float>(const std::vector<SpreadSystem> &, bool, SpreadBatchWork &, cudaStream_t);

}  // namespace yb
