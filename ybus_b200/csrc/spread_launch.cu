// Launches of the spread solve (spread_solve.cuh): layouts made and uploaded at first use, one
// factor's solves, and the complex batch over many factors.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <functional>
#include <optional>
#include <set>
#include <system_error>
#include <thread>

#include "capi_common.hpp"
#include "spread_launch.hpp"
#include "spread_solve.cuh"

namespace yb {

namespace {

// The largest condition (a bound of the Schur complement's norm, times its map's) with which the top is
// taken densely: its correction then leaves 1e-7 of the map's rounding, and FP32 values round more than the map.
constexpr double kSpreadTopCondition = 1e9;
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

template <class T, bool BATCH> void allow_smem(const yb_gpu *gpu);

// The layout on the host: for the blocks an SM holds by the kernel's registers, and where its slots let
// an SM hold fewer, with the cut chosen again for those.
template <class V> SpreadLayout<V> host_spread(const Plan<V> &plan, int value_bytes, int64_t groups, const yb_gpu *gpu) {
  const int most = value_bytes == 16 ? spread_blocks<cplx<double>>() : value_bytes == 8 ? spread_blocks<double>() : spread_blocks<float>();
  return spread_layout<V>(plan, value_bytes, groups, gpu->sm_count, most, [&](int32_t slots) {
    const size_t smem = (value_bytes == 16 ? spread_smem<cplx<double>>(slots, kSpreadWarps)
                         : value_bytes == 8 ? spread_smem<double>(slots, kSpreadWarps)
                                            : spread_smem<float>(slots, kSpreadWarps)) + 1024;
    return (int32_t)std::max<size_t>(1, (size_t)gpu->smem_per_sm / smem);
  });
}

// Arrays put one after the other, 256-byte aligned, into one allocation, their places told when it is made.
struct Packer {
  std::vector<uint8_t> bytes;
  size_t size = 0;  // what is uploaded and what is only reserved
  std::vector<std::pair<size_t, std::function<void(uint8_t *)>>> places;
  template <class P> void place(size_t n, P *&to) {
    size = (size + 255) / 256 * 256;
    places.emplace_back(size, [&to](uint8_t *p) { to = reinterpret_cast<P *>(p); });
    size += std::max<size_t>(n, 1) * sizeof(P);
  }
  template <class P, class T> void put(const std::vector<T> &v, P *&to) {  // all puts before the first reserve
    place(v.size(), to);
    bytes.resize(size);
    if (!v.empty()) std::memcpy(bytes.data() + places.back().first, v.data(), v.size() * sizeof(T));
  }
  void upload(DeviceArray<uint8_t> &to, cudaStream_t s) {
    to.resize(size);
    if (!bytes.empty()) cuda_check(cudaMemcpyAsync(to.get(), bytes.data(), bytes.size(), cudaMemcpyHostToDevice, s), "spread layout upload");
    for (auto &[at, tell] : places) tell(to.get() + at);
  }
};

// Layouts on the device, with their tops' maps; null where a map's condition is too large (or no layout
// came). A layout is one allocation, all that making the maps needs another, and all maps are made by one
// launch: an allocation for every array, and a launch and a wait for every map, took 105 ms for the first
// pass over 16 complex networks.
template <class V>
std::vector<std::unique_ptr<DeviceSpread>> make_spreads(const std::vector<const SpreadLayout<V> *> &lays, int value_bytes,
                                                        const yb_gpu *gpu, cudaStream_t s) {
  using M = typename DeviceValue<V>::type;
  if constexpr (std::is_same_v<V, double>)
    value_bytes == 8 ? allow_smem<double, false>(gpu) : (allow_smem<float, false>(gpu), allow_smem<pair2<float>, false>(gpu));
  else
    value_bytes == 16 ? allow_smem<cplx<double>, true>(gpu) : allow_smem<cplx<float>, true>(gpu);
  static std::atomic<int64_t> serial{0};
  const size_t k = lays.size();
  std::vector<std::unique_ptr<DeviceSpread>> out(k);
  std::vector<Packer> kept(k);
  struct Top {
    const int32_t *lp, *lc, *up, *uc;
    const M *lv, *ld, *uv, *ud, *low = nullptr, *up_v = nullptr;
    M *scratch, *m, *m_up = nullptr, *m_low = nullptr;
  };
  std::vector<Top> tops(k);
  Packer temp;
  const SpreadMap<M> *d_maps = nullptr;
  unsigned long long *norms = nullptr;
  std::vector<SpreadMap<M>> maps(k);
  temp.put(maps, d_maps);
  temp.put(std::vector<unsigned long long>(k), norms);
  for (size_t i = 0; i < k; ++i) {
    if (!lays[i]) continue;
    const SpreadLayout<V> &lay = *lays[i];
    out[i] = std::make_unique<DeviceSpread>();
    DeviceSpread *d = out[i].get();
    Top &t = tops[i];
    d->serial = ++serial;
    d->n = lay.n, d->tasks = lay.tasks, d->top = lay.top, d->slots = lay.slots, d->partials = lay.partials, d->domains = lay.domains;
    d->blob_bytes = (int64_t)lay.blob.size();
    d->host_out_pos = lay.out_pos;
    Packer &p = kept[i];
    p.put(lay.task_row, d->task_row), p.put(lay.fwd_page, d->fwd_page), p.put(lay.bwd_page, d->bwd_page);
    p.put(lay.in_pos, d->in_pos), p.put(lay.out_pos, d->out_pos), p.put(lay.part_ptr, d->part_ptr);
    if (lay.top == 0) continue;
    Packer &q = lay.dense ? temp : p;
    if (!lay.low_ptr.empty()) {
      q.put(lay.low_ptr, d->low_ptr), q.put(lay.low_col, d->low_col), q.put(device_values(lay.low_val), t.low);
      q.put(lay.up_ptr, d->up_ptr), q.put(lay.up_col, d->up_col), q.put(device_values(lay.up_val), t.up_v);
    }
    temp.put(lay.l_ptr, t.lp), temp.put(lay.l_col, t.lc);
    temp.put(device_values(lay.l_val), t.lv), temp.put(device_values(lay.l_dinv), t.ld);
    std::vector<int32_t> u_ptr{0}, u_col;  // the rows from the last to the first
    std::vector<V> u_val, u_dinv(lay.u_dinv.rbegin(), lay.u_dinv.rend());
    u_col.reserve(lay.u_col.size()), u_val.reserve(lay.u_val.size());
    for (int32_t r = lay.top - 1; r >= 0; --r) {
      u_col.insert(u_col.end(), lay.u_col.begin() + lay.u_ptr[r], lay.u_col.begin() + lay.u_ptr[r + 1]);
      u_val.insert(u_val.end(), lay.u_val.begin() + lay.u_ptr[r], lay.u_val.begin() + lay.u_ptr[r + 1]);
      u_ptr.push_back((int32_t)u_col.size());
    }
    temp.put(u_ptr, t.up), temp.put(u_col, t.uc), temp.put(device_values(u_val), t.uv), temp.put(device_values(u_dinv), t.ud);
  }
  const auto blocks = [](int64_t rows, int64_t of) { return (rows + of - 1) / of; };
  int32_t most = 0;
  for (size_t i = 0; i < k; ++i) {
    DeviceSpread *d = out[i].get();
    if (!d) continue;
    const int64_t t = d->top;
    most = std::max(most, d->top);
    if (t > 0) {
      const size_t full = (size_t)(blocks(t, kSpreadTopRows) * t * kSpreadTopRows);
      kept[i].place(full, tops[i].m);
      if (lays[i]->dense) kept[i].place(full, tops[i].m_up), kept[i].place(full, tops[i].m_low);
      temp.place((size_t)(blocks(t, 32) * t * 32), tops[i].scratch);
    }
    kept[i].place(lays[i]->blob.size(), d->blob);
    kept[i].upload(d->store, s);
    cuda_check(cudaMemcpyAsync(const_cast<uint8_t *>(d->blob), lays[i]->blob.data(), lays[i]->blob.size(), cudaMemcpyHostToDevice, s),
               "spread packet upload");
    if (t == 0) continue;
    d->m = tops[i].m, d->m_up = tops[i].m_up, d->m_low = tops[i].m_low;  // with the rows past the last of a block of rows
    cuda_check(cudaMemsetAsync(d->m, 0, (size_t)(d->blob - (uint8_t *)d->m), s), "clear the maps");
  }
  if (most > 0) {
    DeviceArray<uint8_t> temporary;
    // the maps' descriptors need the addresses: made first, then uploaded
    temporary.resize(temp.size);
    for (auto &[at, tell] : temp.places) tell(temporary.get() + at);
    for (size_t i = 0; i < k; ++i) {
      const DeviceSpread *d = out[i].get();
      if (!d || d->top == 0) continue;
      const Top &t = tops[i];
      maps[i] = {d->top, (int32_t)blocks(d->top, 32), t.lp, t.lc, t.lv, t.ld, t.up, t.uc, t.uv, t.ud, t.scratch, t.m, norms + i};
    }
    std::memcpy(temp.bytes.data() + temp.places[0].first, maps.data(), maps.size() * sizeof maps[0]);
    cuda_check(cudaMemcpyAsync(temporary.get(), temp.bytes.data(), temp.bytes.size(), cudaMemcpyHostToDevice, s), "upload the tops");
    spread_map_kernel<M><<<dim3((unsigned)blocks(most, 32), (unsigned)k), 32, 0, s>>>(d_maps);
    cuda_check(cudaGetLastError(), "spread_map_kernel launch");
    spread_norm_kernel<M><<<dim3((unsigned)blocks(most, 256), (unsigned)k), 256, 0, s>>>(d_maps);
    cuda_check(cudaGetLastError(), "spread_norm_kernel launch");
    for (size_t i = 0; i < k; ++i) {
      DeviceSpread *d = out[i].get();
      if (!d || d->top == 0) continue;
      if (lays[i]->dense) {
        const unsigned grid = (unsigned)blocks(d->top, 128);
        spread_dense_kernel<M><<<grid, 128, 0, s>>>(d->top, d->up_ptr, d->up_col, tops[i].up_v, tops[i].m_up);
        spread_dense_kernel<M><<<grid, 128, 0, s>>>(d->top, d->low_ptr, d->low_col, tops[i].low, tops[i].m_low);
        cuda_check(cudaGetLastError(), "spread_dense_kernel launch");
        d->low_ptr = d->low_col = d->up_ptr = d->up_col = nullptr;  // in the temporary array
      } else {
        d->low_val = tops[i].low, d->up_val = tops[i].up_v;
      }
    }
    std::vector<unsigned long long> bits(k);
    cuda_check(cudaMemcpyAsync(bits.data(), norms, bits.size() * sizeof bits[0], cudaMemcpyDeviceToHost, s), "download the norms");
    cuda_check(cudaStreamSynchronize(s), "the tops' maps");
    for (size_t i = 0; i < k; ++i) {
      DeviceSpread *d = out[i].get();
      if (!d || d->top == 0) continue;
      double norm;
      std::memcpy(&norm, &bits[i], sizeof norm);
      d->top_condition = norm * lays[i]->s_norm;
      if (!(d->top_condition <= kSpreadTopCondition)) out[i] = nullptr;
    }
  }
  cuda_check(cudaStreamSynchronize(s), "spread layout upload");
  return out;
}

SpreadNet net_of(const DeviceSpread *d, int64_t groups, int64_t count) {
  SpreadNet net{};
  net.n = d->n, net.tasks = d->tasks, net.top = d->top, net.partials = d->partials;
  net.blob = d->blob, net.fwd_page = d->fwd_page, net.bwd_page = d->bwd_page;
  net.task_row = d->task_row, net.part_ptr = d->part_ptr;
  net.in_pos = d->in_pos, net.out_pos = d->out_pos, net.m = d->m;
  net.low_ptr = d->low_ptr, net.low_col = d->low_col, net.low_val = d->low_val;
  net.up_ptr = d->up_ptr, net.up_col = d->up_col, net.up_val = d->up_val;
  net.m_up = d->m_up, net.m_low = d->m_low;
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
  const bool below = d->top < d->n;  // rows below the top
  if (below) launch(spread_sweep_kernel<T, false, false>, grid, warps * 32, smem, s, true, a);
  if (d->top > 0) {
    const unsigned rows = (unsigned)(groups * ((d->top + 7) / 8));
    launch(spread_sum_kernel<T, false>, rows, 256, 0, s, true, a);
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
    if constexpr (SpreadLane<T>::kCorrect) {
      top(std::integral_constant<int, 1>());
      if (d->m_up) {
        top(std::integral_constant<int, 3>()), top(std::integral_constant<int, 4>());
      } else {
        launch(spread_correct_kernel<T, false, true>, rows, 256, 0, s, true, a);
        launch(spread_correct_kernel<T, false, false>, rows, 256, 0, s, true, a);
      }
      top(std::integral_constant<int, 2>());
    } else {
      top(std::integral_constant<int, 0>());
    }
  }
  if (below) launch(spread_sweep_kernel<T, true, false>, grid, warps * 32, smem, s, true, a);
}

// The partial array of `groups` groups: the partials and the top's solutions in T, then the top's
// right-hand sides (and, where it is corrected, the first product and U_TT times it) in full precision (every
// part a multiple of 128 bytes); at least one line.
template <class T> size_t partial_bytes_of(const DeviceSpread *d, int64_t groups) {
  return (size_t)groups * 32 * ((size_t)(d->partials + d->top) * sizeof(T) + (size_t)d->top * (SpreadLane<T>::kCorrect ? 3 : 1) * sizeof(typename SpreadLane<T>::Math)) + 128;
}
template <class T> void set_partial(SpreadNet &net, uint8_t *p) {
  net.partial = p;
  uint8_t *r = p + (size_t)net.groups * 32 * (size_t)(net.partials + net.top) * sizeof(T);
  const size_t full = (size_t)net.groups * 32 * net.top * sizeof(typename SpreadLane<T>::Math);
  net.r = r, net.r2 = r + full, net.r3 = r + 2 * full;
}

}  // namespace

template <class T> size_t spread_partial_bytes(const DeviceSpread *d, int64_t groups) { return partial_bytes_of<T>(d, groups); }
template size_t spread_partial_bytes<float>(const DeviceSpread *, int64_t);

namespace {

// A layout serves the groups up to a power of two; from 4,096 on cuts no longer differ by the load. So a
// factor keeps 13 at most of one value's bytes, the same one for a number of right-hand sides whatever ran before.
int64_t group_class(int64_t groups) {
  int64_t most = 1;
  while (most < groups && most < 4096) most *= 2;
  return most;
}
// In a batch, up to a number of three significant bits: the longest task of any network sets a sweep's time, so
// the networks' cuts have to agree (16 networks of 730 to 46,293 buses: 929 us, by powers of two 972).
// These layouts are made only when they have paid for themselves, and kSpreadMostBatchLayouts of them.
int64_t batch_class(int64_t groups) {
  int64_t most = groups;
  for (int64_t unit = 1; most > 8 * unit || most % unit; unit *= 2) most = (most + 2 * unit - 1) / (2 * unit) * (2 * unit);
  return most;
}

template <class V> const Plan<V> &plan_of(const yb_factor *f) {
  if constexpr (std::is_same_v<V, double>) return f->plan;
  else return f->cplan;
}

// A layout or, where the factor admits none, nothing.
template <class V> std::unique_ptr<SpreadLayout<V>> try_layout(const yb_factor *f, int value_bytes, int64_t groups) {
  try {
    auto lay = std::make_unique<SpreadLayout<V>>(host_spread(plan_of<V>(f), value_bytes, groups, f->gpu));
    if (!std::is_same_v<V, double> || value_bytes == 8) {  // not in real FP32
      lay->dense = std::is_same_v<V, double> && 8 * (lay->l_col.size() + lay->u_col.size()) > (size_t)lay->top * (size_t)lay->top;
      spread_correction(*lay);
    }
    const int32_t limit = f->is_complex ? kSpreadAutoSlotsComplex : kSpreadAutoSlots;
    return lay->slots <= limit ? std::move(lay) : nullptr;
  } catch (const host::Error &e) {
    if (e.status != host::kInvalidArgument && e.status != host::kTooLarge) throw;
    return nullptr;
  }
}

}  // namespace

DeviceSpread *spread_for(yb_factor *f, int value_bytes, int64_t groups, cudaStream_t stream, int64_t matrix) {
  const std::lock_guard<std::mutex> lock(f->spread_mutex);
  const auto key = std::make_pair(value_bytes, group_class(groups));
  auto it = f->spreads.find(key);
  const bool no_more = (it == f->spreads.end() || matrix >= 0) && capturing(stream);
  auto ready = [&](const DeviceSpread *d) { return !no_more || matrix < 0 || (d && d->res_matrix == matrix); };
  if (it != f->spreads.end() && ready(it->second.get())) return it->second.get();
  if (no_more) {  // nothing may be made now: the nearest layout there is, if any
    auto near = f->spreads.end();
    for (auto i = f->spreads.begin(); i != f->spreads.end(); ++i)
      if (i->first.first == value_bytes && i->second && ready(i->second.get()) &&
          (near == f->spreads.end() || std::abs(i->first.second - key.second) < std::abs(near->first.second - key.second)))
        near = i;
    return near == f->spreads.end() ? nullptr : near->second.get();
  }
  const auto lay = try_layout<double>(f, value_bytes, key.second);
  std::unique_ptr<DeviceSpread> d;
  try {
    d = std::move(make_spreads<double>({lay.get()}, value_bytes, f->gpu, stream)[0]);
  } catch (const OutOfMemory &) {
    return nullptr;  // this time
  }
  auto *out = d.get();
  f->spreads.emplace(key, std::move(d));
  return out;
}

// Each network's class in a batch: its share of the load in groups of its own, since the cut weighs the whole
// batch's load.
static std::vector<std::pair<int, int64_t>> batch_keys(const std::vector<yb_factor *> &factors, int value_bytes,
                                                       const std::vector<int64_t> &counts) {
  double load = 0;
  for (size_t i = 0; i < factors.size(); ++i) load += (double)factors[i]->n * (double)((counts[i] + 31) / 32);
  std::vector<std::pair<int, int64_t>> keys;
  for (const yb_factor *f : factors)
    keys.push_back({value_bytes, batch_class(std::max<int64_t>(1, (int64_t)std::ceil(load / (double)f->n)))});
  return keys;
}

void spread_for_batch(const std::vector<yb_factor *> &factors, int value_bytes, const std::vector<int64_t> &counts,
                      std::vector<DeviceSpread *> &out, cudaStream_t stream) {
  const size_t k = factors.size();
  std::vector<std::unique_ptr<SpreadLayout<host::c128>>> made(k);
  const auto keys = batch_keys(factors, value_bytes, counts);
  std::vector<size_t> missing;
  std::set<std::pair<yb_factor *, int64_t>> seen;
  for (size_t i = 0; i < k; ++i) {
    const std::lock_guard<std::mutex> lock(factors[i]->spread_mutex);
    const auto &there = factors[i]->spreads;
    if (counts[i] > 0 && !small_for_batch(factors[i]) && !there.count(keys[i]) && factors[i]->spread_passes[keys[i]] >= kSpreadBatchPasses &&
        std::count_if(there.begin(), there.end(), [&](const auto &e) { return e.first.first == value_bytes; }) < kSpreadMostBatchLayouts &&
        seen.insert({factors[i], keys[i].second}).second)
      missing.push_back(i);
  }
  // the layouts not made yet, on the host's threads, largest networks first
  std::sort(missing.begin(), missing.end(), [&](size_t a, size_t b) { return factors[a]->n > factors[b]->n; });
  std::atomic<size_t> next{0};
  std::vector<std::exception_ptr> errors(missing.size());
  auto work = [&] {
    for (size_t m = next++; m < missing.size(); m = next++)
      try {
        made[missing[m]] = try_layout<host::c128>(factors[missing[m]], value_bytes, keys[missing[m]].second);
      } catch (...) {
        errors[m] = std::current_exception();
      }
  };
  std::vector<std::thread> threads;
  const size_t most = std::min<size_t>(missing.size(), std::max(1u, std::thread::hardware_concurrency()));
  try {
    for (size_t t = 1; t < most; ++t) threads.emplace_back(work);
  } catch (const std::system_error &) {  // no more threads: those there are do
  }
  work();
  for (auto &t : threads) t.join();
  for (auto &e : errors)
    if (e) std::rethrow_exception(e);
  if (!missing.empty()) {
    std::vector<const SpreadLayout<host::c128> *> lays;
    for (size_t i : missing) lays.push_back(made[i].get());
    std::vector<std::unique_ptr<DeviceSpread>> d;
    try {
      d = make_spreads<host::c128>(lays, value_bytes, factors[0]->gpu, stream);
    } catch (const OutOfMemory &) {  // none this time
    }
    for (size_t m = 0; m < d.size(); ++m) {
      const std::lock_guard<std::mutex> lock(factors[missing[m]]->spread_mutex);
      factors[missing[m]]->spreads.emplace(keys[missing[m]], std::move(d[m]));
    }
  }
  out.assign(k, nullptr);
  for (size_t i = 0; i < k; ++i) {
    const yb_factor *f = factors[i];
    const std::lock_guard<std::mutex> lock(factors[i]->spread_mutex);
    const auto it = f->spreads.find(keys[i]);
    if (it != f->spreads.end()) {
      out[i] = it->second.get();
      continue;
    }
    int64_t distance = INT64_MAX;  // until its class has a layout: the nearest class's, if any
    for (const auto &[key, d] : f->spreads)
      if (d && key.first == value_bytes && std::abs(key.second - keys[i].second) < distance)
        out[i] = d.get(), distance = std::abs(key.second - keys[i].second);
  }
}

void spread_batch_solved(const std::vector<yb_factor *> &factors, int value_bytes, const std::vector<int64_t> &counts, int solves) {
  const auto keys = batch_keys(factors, value_bytes, counts);
  for (size_t i = 0; i < factors.size(); ++i) {
    const std::lock_guard<std::mutex> lock(factors[i]->spread_mutex);
    if (counts[i] > 0 && !factors[i]->spreads.count(keys[i])) factors[i]->spread_passes[keys[i]] += solves;
  }
}

template <class T>
void spread_sweeps(yb_factor *f, DeviceSpread *d, T *work, T *xout, uint8_t *partial, int64_t groups, const uint8_t *group_active,
                   cudaStream_t stream) {
  SpreadArgs a{};
  a.one = net_of(d, groups, groups * 32);
  a.one.work = work, a.one.xout = xout, a.one.top_out = xout != work;
  set_partial<T>(a.one, partial);
  a.one.group_active = group_active;
  a.slots = d->slots;
  one_sweeps<T>(d, a, f->gpu, stream);
}
template void spread_sweeps<float>(yb_factor *, DeviceSpread *, float *, float *, uint8_t *, int64_t, const uint8_t *, cudaStream_t);

namespace {

// Lets this thread allocate while a stream of it, or of another thread, is being captured: what it
// allocates here belongs to no graph's work.
struct CaptureAside {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  CaptureAside() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~CaptureAside() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// `released` becomes true when `graph`, its clones and its executables are destroyed.
void keep_while(cudaGraph_t graph, const std::shared_ptr<std::atomic<bool>> &released) {
  using Held = std::shared_ptr<std::atomic<bool>>;
  auto held = std::make_unique<Held>(released);
  cudaUserObject_t object = nullptr;
  cuda_check(cudaUserObjectCreate(&object, held.get(), [](void *p) {
    const std::unique_ptr<Held> last(static_cast<Held *>(p));
    (*last)->store(true);
  }, 1, cudaUserObjectNoDestructorSync), "cudaUserObjectCreate");
  held.release();  // the object's
  const cudaError_t e = cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove);
  if (e != cudaSuccess) cudaUserObjectRelease(object, 1);
  cuda_check(e, "cudaGraphRetainUserObject");
}

}  // namespace

WorkLease::WorkLease(yb_factor *f, const SpreadBytes &bytes, cudaStream_t stream) : lock_(f->spread_mutex), stream_(stream) {
  const CaptureAside aside;
  auto &all = f->spread_work;
  // a graph that is gone gives its workspace back (the free waits for what still runs)
  all.erase(std::remove_if(all.begin(), all.end(), [](const auto &i) { return i->capture && i->released->load(); }), all.end());
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  cuda_check(cudaStreamGetCaptureInfo(stream, &status, &id, &graph), "cudaStreamGetCaptureInfo");
  if (status != cudaStreamCaptureStatusNone) {
    for (auto &i : all)
      if (i->capture == id && i->stream == stream && i->holds(bytes)) w_ = i.get();
    if (w_) return;
    auto own = std::make_unique<SpreadWork>();
    own->grow(bytes);
    own->stream = stream, own->capture = id;
    own->released = std::make_shared<std::atomic<bool>>(false);
    keep_while(graph, own->released);
    all.push_back(std::move(own));
    w_ = all.back().get();
    return;
  }
  size_t eager = 0;
  for (auto &i : all) {
    if (i->capture) continue;
    ++eager;
    if (i->stream == stream) w_ = i.get();
  }
  if (!w_)
    for (auto &i : all)
      if (!w_ && !i->capture && cudaEventQuery(i->done) == cudaSuccess) w_ = i.get();
  cudaGetLastError();  // a workspace still in use is no error
  if (!w_ && eager < SpreadWork::kMost) {
    all.push_back(std::make_unique<SpreadWork>());
    w_ = all.back().get();
    cuda_check(cudaEventCreateWithFlags(&w_->done, cudaEventDisableTiming), "cudaEventCreate");
  }
  if (!w_)
    for (auto &i : all)
      if (!i->capture && (!w_ || i->used < w_->used)) w_ = i.get();
  cuda_check(cudaStreamWaitEvent(stream, w_->done, 0), "cudaStreamWaitEvent");
  w_->stream = stream;
  w_->used = ++f->spread_solves;
  w_->grow(bytes);  // a larger array: the device is idle past the old one's free
}

WorkLease::~WorkLease() {
  if (w_ && !w_->capture) cudaEventRecord(w_->done, stream_);
}

namespace {

template <class L>
bool solve_lanes(yb_factor *f, DeviceSpread *d, const double *b, int64_t ldb, double *x, int64_t ldx, int64_t count,
                 cudaStream_t stream, const SpreadFinish &finish = {}) {
  constexpr int64_t COLS = 32 * SpreadLane<L>::N;  // columns of a group
  const int64_t n = f->n, groups_all = (count + COLS - 1) / COLS;
  const size_t group_bytes = (size_t)n * 32 * sizeof(L), pad_bytes = 2 * kSpreadPad * 32 * sizeof(L);
  const int64_t per_run = std::min<int64_t>(groups_all, f->gpu->work_bytes / (int64_t)group_bytes);
  if (per_run < 1) return false;
  SpreadBytes bytes;
  bytes.work = (size_t)per_run * group_bytes + pad_bytes;
  bytes.partial = partial_bytes_of<L>(d, per_run);
  std::optional<WorkLease> lease;
  try {
    lease.emplace(f, bytes, stream);
  } catch (const OutOfMemory &) {
    return false;
  }
  const WorkLease &w = *lease;
  L *work = reinterpret_cast<L *>(w->work.get()) + kSpreadPad * 32;
  for (int64_t g0 = 0; g0 < groups_all; g0 += per_run) {
    const int64_t groups = std::min(per_run, groups_all - g0);
    SpreadArgs a{};
    a.one = net_of(d, groups, std::min(count - g0 * COLS, groups * COLS));
    a.one.work = a.one.xout = work;
    a.one.top_out = (bool)finish;
    set_partial<L>(a.one, w->partial.get());
    a.one.b = b + g0 * COLS * ldb, a.one.ldb = ldb, a.one.x = x ? x + g0 * COLS * ldx : nullptr, a.one.ldx = ldx;
    a.slots = d->slots;
    const unsigned io = (unsigned)((groups * ((n + 31) / 32) + kSpreadIoWarps - 1) / kSpreadIoWarps);
    cudaEvent_t *ev = lane_timing_slot(f);
    if (ev) cuda_check(cudaEventRecord(ev[0], stream), "cudaEventRecord");
    launch(spread_in_kernel<L, false>, io, kSpreadIoWarps * 32, 0, stream, true, a);
    if (ev) cuda_check(cudaEventRecord(ev[1], stream), "cudaEventRecord");
    one_sweeps<L>(d, a, f->gpu, stream);
    if (ev) cuda_check(cudaEventRecord(ev[2], stream), "cudaEventRecord");
    if (finish)
      finish(reinterpret_cast<const double *>(work), d->out_pos, g0 * COLS, a.one.count);
    else
      launch(spread_out_kernel<L, false, false>, io, kSpreadIoWarps * 32, 0, stream, true, a);
    if (ev) cuda_check(cudaEventRecord(ev[3], stream), "cudaEventRecord");
  }
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
bool spread_solve_lanes(yb_factor *f, const double *b, int64_t ldb, int64_t count, cudaStream_t stream, const SpreadFinish &finish) {
  DeviceSpread *d = spread_for(f, (int)sizeof(double), (count + 31) / 32, stream);
  return d && solve_lanes<double>(f, d, b, ldb, nullptr, 0, count, stream, finish);
}
template bool spread_solve<double>(yb_factor *, const double *, int64_t, double *, int64_t, int64_t, cudaStream_t);
template bool spread_solve<float>(yb_factor *, const double *, int64_t, double *, int64_t, int64_t, cudaStream_t);

namespace {

// One run of launches over what fits the batch's work arrays.
template <class R> void batch_run(const std::vector<SpreadSystem> &systems, bool add, SpreadBatchWork &w, cudaStream_t stream) {
  using T = cplx<R>;
  const size_t k = systems.size();
  const yb_gpu *gpu = systems[0].factor->gpu;
  std::vector<SpreadNet> nets(k);
  int64_t top_total = 0;
  int32_t slots = 0;
  int64_t most_groups = 1;
  for (const SpreadSystem &sys : systems) {
    const int64_t groups = (sys.count + 31) / 32;
    top_total += groups * top_tiles(sys.layout);
    slots = std::max(slots, sys.layout->slots);
    most_groups = std::max(most_groups, groups);
  }
  const int split = split_top<T>(top_total, gpu);
  const int warps = sweep_warps<T>(slots, most_groups, gpu);
  T *work = reinterpret_cast<T *>(w.work.get());
  uint8_t *partial = w.partial.get();
  std::vector<int64_t> key{(int64_t)sizeof(T), warps, split};
  for (size_t i = 0; i < k; ++i) {
    const SpreadSystem &sys = systems[i];
    const int64_t groups = (sys.count + 31) / 32;
    SpreadNet &net = nets[i];
    net = net_of(sys.layout, groups, sys.count);
    net.work = net.xout = work + kSpreadPad * 32;
    set_partial<T>(net, partial);
    net.b = sys.b, net.ldb = sys.layout->n, net.x = sys.x, net.ldx = sys.layout->n;
    work += (size_t)groups * sys.layout->n * 32 + 2 * kSpreadPad * 32;
    partial += partial_bytes_of<T>(sys.layout, groups);
    key.push_back(sys.layout->serial), key.push_back(groups);
  }
  w.nets.reserve(sizeof(SpreadNet) * k);
  cuda_check(cudaMemcpyAsync(w.nets.get(), nets.data(), sizeof(SpreadNet) * k, cudaMemcpyHostToDevice, stream), "upload the batch");
  if (key != w.key) {
    // the blocks' items: the gather's and scatter's, the sweeps' (each network's tasks are longest
    // first; the networks' tasks by rank, so every network's long tasks start early), the top's
    std::vector<SpreadItem> io, sweep, sum, top;
    int32_t most_tasks = 0;
    for (size_t i = 0; i < k; ++i) {
      const DeviceSpread *d = systems[i].layout;
      most_tasks = std::max(most_tasks, d->tasks);
      const int32_t row_blocks = (int32_t)((d->n + 32 * kSpreadIoWarps - 1) / (32 * kSpreadIoWarps));
      for (int64_t g = 0; g < nets[i].groups; ++g) {
        for (int32_t c = 0; c < row_blocks; ++c) io.push_back({(int32_t)i, c, (int32_t)g, 0});
        for (int32_t c = 0; c < (d->top + 7) / 8; ++c) sum.push_back({(int32_t)i, c, (int32_t)g, 0});
        for (int32_t c = 0; c < top_blocks<T>(d, split); ++c) top.push_back({(int32_t)i, c, (int32_t)g, 0});
      }
    }
    for (int32_t t = 0; t < most_tasks; ++t)
      for (size_t i = 0; i < k; ++i)
        if (t < systems[i].layout->tasks)
          for (int64_t g = 0; g < nets[i].groups; g += warps) sweep.push_back({(int32_t)i, t, (int32_t)g, 0});
    w.key.clear();
    w.n_io = io.size(), w.n_sweep = sweep.size(), w.n_sum = sum.size(), w.n_top = top.size();
    for (auto *more : {&sweep, &sum, &top}) io.insert(io.end(), more->begin(), more->end());
    w.items.reserve(sizeof(SpreadItem) * io.size());
    cuda_check(cudaMemcpyAsync(w.items.get(), io.data(), sizeof(SpreadItem) * io.size(), cudaMemcpyHostToDevice, stream),
               "upload the batch's blocks");
    w.key = std::move(key);
  }
  const size_t n_io = w.n_io, n_sweep = w.n_sweep, n_sum = w.n_sum, n_top = w.n_top;
  const auto *d_items = reinterpret_cast<const SpreadItem *>(w.items.get());
  SpreadArgs a{};
  a.nets = reinterpret_cast<const SpreadNet *>(w.nets.get());
  a.slots = slots;
  const size_t smem = spread_smem<T>(slots, warps);
  a.items = d_items;
  launch(spread_in_kernel<T, true>, (unsigned)n_io, kSpreadIoWarps * 32, 0, stream, true, a);
  a.items = d_items + n_io;
  launch(spread_sweep_kernel<T, false, true>, (unsigned)n_sweep, warps * 32, smem, stream, true, a);
  if (n_top) {
    a.items = d_items + n_io + n_sweep;
    launch(spread_sum_kernel<T, true>, (unsigned)n_sum, 256, 0, stream, true, a);
    auto phase = [&](auto one) {
      a.items = d_items + n_io + n_sweep + n_sum;
      constexpr int PHASE = decltype(one)::value;
      if (split > 1)
        launch(spread_top_kernel<T, true, spread_split<T>(), PHASE>, (unsigned)n_top, spread_top_warps<T, spread_split<T>()>() * 32, 0, stream, true, a);
      else
        launch(spread_top_kernel<T, true, 1, PHASE>, (unsigned)n_top, spread_top_warps<T, 1>() * 32, 0, stream, true, a);
    };
    phase(std::integral_constant<int, 1>());
    a.items = d_items + n_io + n_sweep;
    launch(spread_correct_kernel<T, true, true>, (unsigned)n_sum, 256, 0, stream, true, a);
    launch(spread_correct_kernel<T, true, false>, (unsigned)n_sum, 256, 0, stream, true, a);
    phase(std::integral_constant<int, 2>());
  }
  a.items = d_items + n_io;
  launch(spread_sweep_kernel<T, true, true>, (unsigned)n_sweep, warps * 32, smem, stream, true, a);
  a.items = d_items;
  if (add)
    launch(spread_out_kernel<T, true, true>, (unsigned)n_io, kSpreadIoWarps * 32, 0, stream, true, a);
  else
    launch(spread_out_kernel<T, true, false>, (unsigned)n_io, kSpreadIoWarps * 32, 0, stream, true, a);
}

template <class T> size_t batch_work_bytes(const DeviceSpread *d, int64_t groups) {
  return ((size_t)groups * d->n * 32 + 2 * kSpreadPad * 32) * sizeof(T);
}

}  // namespace

template <class R> bool spread_batch_fits(const SpreadSystem &sys) {
  return (int64_t)batch_work_bytes<cplx<R>>(sys.layout, 1) <= sys.factor->gpu->work_bytes;
}
template bool spread_batch_fits<double>(const SpreadSystem &);
template bool spread_batch_fits<float>(const SpreadSystem &);

template <class R>
void spread_batch(const std::vector<SpreadSystem> &systems, bool add, SpreadBatchWork &w, cudaStream_t stream) {
  using T = cplx<R>;
  if (systems.empty()) return;
  const size_t limit = (size_t)systems[0].factor->gpu->work_bytes;
  // runs of as many groups as the work array holds, a network after the other
  std::vector<std::vector<SpreadSystem>> runs(1);
  size_t used = 0, work_most = 0, part = 0, part_most = 0;
  for (const SpreadSystem &sys : systems) {
    const size_t pad = batch_work_bytes<T>(sys.layout, 0), group = batch_work_bytes<T>(sys.layout, 1) - pad;
    for (int64_t g = 0, groups = (sys.count + 31) / 32; g < groups;) {
      if (used + pad + group > limit && used > 0) runs.emplace_back(), used = part = 0;
      const int64_t some = std::min<int64_t>(groups - g, std::max<int64_t>(1, ((int64_t)limit - (int64_t)(used + pad)) / (int64_t)group));
      SpreadSystem piece = sys;
      piece.b += g * 32 * sys.layout->n, piece.x += g * 32 * sys.layout->n;
      piece.count = std::min<int64_t>(sys.count - g * 32, some * 32);
      runs.back().push_back(piece);
      used += pad + (size_t)some * group, part += partial_bytes_of<T>(sys.layout, some);
      work_most = std::max(work_most, used), part_most = std::max(part_most, part);
      g += some;
    }
  }
  w.work.grow(work_most), w.partial.grow(part_most);  // before the first launch: the tiles can still take its place
  for (const auto &run : runs) batch_run<R>(run, add, w, stream);
}
template void spread_batch<double>(const std::vector<SpreadSystem> &, bool, SpreadBatchWork &, cudaStream_t);
template void spread_batch<float>(const std::vector<SpreadSystem> &, bool, SpreadBatchWork &, cudaStream_t);

}  // namespace yb
