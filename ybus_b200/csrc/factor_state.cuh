// The state behind the C ABI's opaque handles `yb_gpu` and `yb_factor`.
#pragma once

#include <cuda_runtime.h>

#include <array>
#include <atomic>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <tuple>

#include "../../include/ybgpu.h"
#include "cplx.cuh"
#include "device.cuh"
#include "plan.hpp"

// The widest block `yb_factor` chooses by itself. ybus_cuda caps its default at 1,024 because each
// block is one cuSPARSE SpSM call (ybus_cuda/src/factor.rs:12); here a block is one persistent
// launch that needs at least one tile per SM to fill the GPU, so the cap is higher.
constexpr int64_t kMaxDefaultWidth = 65536;
// The largest chunk of right-hand sides the host-array solve moves through its copy pipeline
constexpr int64_t kPipelineChunk = 1024;
// The widest block a single-row factor uses (ybus_cuda/src/factor.rs:14-16): kept for API parity.
constexpr int64_t kSingleRowWidth = 64;

struct yb_gpu {
  int device = 0;
  cudaStream_t stream = nullptr;
  int sm_count = 0, major = 0, minor = 0;
  int64_t l2_bytes = 0;
  int64_t smem_optin = 0;       // largest dynamic shared memory a block may opt into
  int64_t smem_per_sm = 0;
  std::string name;
  std::atomic<int64_t> work_bytes{int64_t(2) << 30};  // the largest work array one run of the spread solve fills
  std::shared_ptr<void> zwork;  // the complex batch's device workspace (capi_complex.cu), kept between calls
  std::mutex zmutex;            // held by the call that uses it
};

namespace yb {

// Seconds spent in `yb_solve_many`'s stages (ybus_cuda/src/factor.rs:22-31).
struct Timings {
  double upload = 0, solve = 0, download = 0;
  int64_t blocks = 0;
};

// Per-launch times of the lane solve, when switched on: events before the gather and after the
// gather, the solve and the scatter of every launch, kept for up to kSlots launches between reads.
struct LaneTiming {
  static constexpr int kSlots = 4096;
  bool on = false;
  int device = -1;
  std::vector<std::array<cudaEvent_t, 4>> ev;
  size_t used = 0;
  LaneTiming() = default;
  LaneTiming(const LaneTiming &) = delete;
  LaneTiming &operator=(const LaneTiming &) = delete;
  ~LaneTiming() {
    for (auto &slot : ev)
      for (auto &e : slot)
        if (e) cudaEventDestroy(e);
  }
};

// The host-array solve's overlap: chunks of right-hand sides pass through an upload stream, the
// solve stream and a download stream, so the two copy engines and the SMs work on successive
// chunks at once. Each of kSlots slots holds one chunk's device buffers (and, for pageable host
// arrays, pinned staging) and the events that time its three stages.
struct CopyPipeline {
  static constexpr int kSlots = 4;
  enum { kInStart, kInDone, kSolveStart, kSolved, kOutStart, kOutDone, kEvents };
  int device = -1;
  cudaStream_t in = nullptr, out = nullptr;
  cudaEvent_t ev[kSlots][kEvents] = {};
  PinnedBuffer stage_in[kSlots], stage_out[kSlots];
  CopyPipeline() = default;
  CopyPipeline(const CopyPipeline &) = delete;
  CopyPipeline &operator=(const CopyPipeline &) = delete;
  ~CopyPipeline() {
    for (auto &slot : ev)
      for (auto &e : slot)
        if (e) cudaEventDestroy(e);
    if (in) cudaStreamDestroy(in);
    if (out) cudaStreamDestroy(out);
  }
  void ensure() {
    if (in) return;
    cuda_check(cudaStreamCreateWithFlags(&in, cudaStreamNonBlocking), "cudaStreamCreate");
    cuda_check(cudaStreamCreateWithFlags(&out, cudaStreamNonBlocking), "cudaStreamCreate");
    for (auto &slot : ev)
      for (auto &e : slot) cuda_check(cudaEventCreate(&e), "cudaEventCreate");
  }
};

// Which tile solve runs: the shared-memory one (the tile's working vector in shared memory) when
// it fits, or the one whose working vectors live in a global scratch buffer.
enum TileKind : int { kTileAuto = 0, kTileShared = 1, kTileGlobal = 2, kTileStream = 3, kTileDomain = 4, kTileLane = 5 };

// The launch shape of the tile solve for one precision.
struct TileConfig {
  int width = 8;          // right-hand sides per tile
  int threads = 512;      // threads per block
  int blocks_per_sm = 1;  // resident blocks per SM the grid is sized for
  int kind = kTileAuto;
  // a caller set a shape or a threshold of the solves below: the automatic choice is then among them,
  // as it is for a factor that admits no spread layout
  bool shaped = false;
  // the autotuner left the shapes below as it found them fastest, and the spread solve faster still
  bool spread_first = false;
  bool admits_spread() const { return spread_first || (kind == kTileAuto && !shaped); }
  void shape() { shaped = true, spread_first = false; }
  // the streamed solve's shape: warps per block, pages in flight per warp, page bytes, and the
  // row count under which a level goes to warp 0 (0: twice the rows of a slice)
  int stream_warps = 8, ring = 4, page_bytes = 2048, narrow_rows = 0;
  int tail_level = -1;  // forward level from which rows form the dense tail (0: none, -1: chosen)
  // the domain solve's shape: warps per block, pages in flight per warp, page bytes, and the cut
  // (first forward level of the top block; -1: chosen by the layout's cost model)
  int domain_warps = 16, domain_ring = 2, domain_page = 2048, domain_cut = -1;
  // the automatic choice takes the lane solve from this many right-hand sides on (one warp per 32:
  // fewer leave SMs idle, where the domain solve's tiles spread over all of them); -1: by the
  // factor's domain tiles (lane_threshold in capi_gpu.cu)
  int64_t lane_min_count = -1;
  int lane_warps = 8, lane_page = 0;  // the lane solve's warps per block (one group of 32 right-hand sides), page bytes
  int lane_rpl = 1;                   // right-hand sides per lane of the plain lane solve (1 or 2)
  // lane_warps not set by a caller or the autotuner: a solve of no more groups of 32 than SMs then
  // takes blocks of kLaneMaxWarps (one an SM, each warp's chain of rows shorter)
  bool lane_warps_auto = true;
  // without the spread solve the refined one takes the lane solve from this many right-hand sides on (its passes cost more
  // launches than the plain solve's, so its crossover with the fused domain refinement lies higher:
  // 2,048 on the 10,000-bus B′ with blocks of 16 warps up to one wave)
  int64_t refine_lane_min_count = 2048;
  bool refine_shaped = false;  // a caller set it: the refined solve chooses among the lane and domain solves
};

// The refined solve's copy of the attached A for a layout (LaneRefineArgs' res_*): natural rows in
// slices of 32, columns as work rows; built at its first use, for the matrix attached then.
struct ResidualMatrix {
  int64_t res_matrix = -1;  // the attach count it was built for
  DeviceArray<int32_t> res_ptr, res_len, res_col;
  DeviceArray<double> res_val;
};

// A lane layout on the device (LaneLayout in plan.hpp).
struct DeviceLane : ResidualMatrix {
  int32_t warps = 0, slots = 0, page_bytes = 0, domains = 0, top = 0, partials = 0, fwd_live = 0, bwd_live = 0;
  int32_t rpl = 1;  // right-hand sides per lane the layout's offsets count
  int64_t entries = 0, pages = 0;
  DeviceArray<uint8_t> blob;
  DeviceArray<int32_t> warp_page, in_pos, out_pos;
  std::vector<int32_t> host_out_pos;
};

// A spread layout on the device (SpreadLayout in plan.hpp), with the top's dense map.
struct DeviceSpread : ResidualMatrix {
  int32_t n = 0, tasks = 0, domains = 0, top = 0, slots = 0, partials = 0;
  int64_t blob_bytes = 0;
  int64_t serial = 0;  // no two layouts of a process share one
  double top_condition = 0;
  DeviceArray<uint8_t> store;  // what the pointers below point into
  const uint8_t *blob = nullptr;
  const int32_t *task_row = nullptr, *fwd_page = nullptr, *bwd_page = nullptr, *in_pos = nullptr, *out_pos = nullptr;
  const int32_t *part_ptr = nullptr, *low_ptr = nullptr, *low_col = nullptr, *up_ptr = nullptr, *up_col = nullptr;
  const void *low_val = nullptr, *up_val = nullptr;
  void *m = nullptr, *m_up = nullptr, *m_low = nullptr;
  std::vector<int32_t> host_out_pos;
};

// The bytes of a workspace's arrays: the work and the partial array, and the refined solves' FP32
// corrections, FP64 iterate (the domain solve's: its residuals) and per-column state.
struct SpreadBytes {
  size_t work = 0, partial = 0, corrections = 0, iterate = 0, state = 0;
};

// A workspace of the spread solve and of the refined solves, for one stream at a time: the event marks its
// last use, so a stream that takes it over (or one that got a destroyed stream's handle) waits for that. One
// that a capture took belongs to that graph until the graph and its executables are gone, which `released`
// tells: no other solve takes it and it never grows, since the graph holds its pointers.
struct SpreadWork {
  static constexpr size_t kMost = 4;  // workspaces a factor keeps; a further stream waits for the oldest
  cudaStream_t stream = nullptr;
  cudaEvent_t done = nullptr;
  uint64_t used = 0;               // the solve that used it last
  unsigned long long capture = 0;  // the capture that took it, or 0
  std::shared_ptr<std::atomic<bool>> released;
  DeviceArray<uint8_t> work, partial, corrections, iterate, state;
  bool holds(const SpreadBytes &b) const {
    return work.size() >= b.work && partial.size() >= b.partial && corrections.size() >= b.corrections &&
           iterate.size() >= b.iterate && state.size() >= b.state;
  }
  void grow(const SpreadBytes &b) {
    work.grow(b.work), partial.grow(b.partial), corrections.grow(b.corrections);
    iterate.grow(b.iterate), state.grow(b.state);
  }
  SpreadWork() = default;
  SpreadWork(const SpreadWork &) = delete;
  SpreadWork &operator=(const SpreadWork &) = delete;
  ~SpreadWork() {
    if (done) cudaEventDestroy(done);
  }
};

// The complex batch's workspace for the spread solve, and the lists of its launches' blocks, which
// depend on the layouts (by their serial numbers) and the counts alone.
struct SpreadBatchWork {
  DeviceArray<uint8_t> work, partial, nets, items;
  std::vector<int64_t> key;
  size_t n_io = 0, n_sweep = 0, n_sum = 0, n_top = 0;
};

// A domain layout on the device (DomainLayout in plan.hpp).
struct DeviceDomain {
  int32_t K = 0, tail = 0, stages = 0, warps = 0, page_bytes = 0;
  int64_t records = 0, bytes = 0, entries = 0, dense_entries = 0;
  double cost = 0;
  DeviceArray<uint8_t> blob;
  DeviceArray<int32_t> warp_page, tail_slot;
};

// A streamed layout on the device (StreamLayout in plan.hpp).
struct DeviceStream {
  int32_t stages = 0, G = 0;
  int64_t records = 0, bytes = 0;
  int32_t fwd_wide = 0, bwd_wide = 0, fwd_narrow_rows = 0, bwd_narrow_rows = 0;
  DeviceArray<uint8_t> blob;
  DeviceArray<int32_t> warp_page;
  DeviceArray<uint8_t> load_scale;
  int32_t tail = 0;
  DeviceArray<int32_t> tail_slot;
};

// A sliced sweep on the device (SliceSweep in plan.hpp), at value type T.
template <class T> struct DeviceSlices {
  int32_t levels = 0;
  int64_t slices = 0, entries = 0;
  DeviceArray<int32_t> level_slice, row, col;
  DeviceArray<int2> span;
  DeviceArray<T> dinv, val;
};

}  // namespace yb

struct yb_factor {
  yb_gpu *gpu = nullptr;
  int64_t n = 0;
  int kind = 0;
  yb::Plan<double> plan;
  yb::DeviceArray<int32_t> in_slot, out_slot;
  yb::DeviceSweep<double> fwd64, bwd64;
  yb::DeviceSweep<float> fwd32, bwd32;
  yb::TileConfig tile64{8, 512, 1}, tile32{8, 512, 1};
  // sliced sweeps per tile width (built on first use): [width] -> {forward, backward}
  std::map<int, std::unique_ptr<yb::DeviceSlices<double>[]>> slices64;
  std::map<int, std::unique_ptr<yb::DeviceSlices<float>[]>> slices32;
  // streamed layouts by shape (precision, width, warps, page bytes, narrow rows)
  std::map<std::tuple<int, int, int, int, int, int>, std::unique_ptr<yb::DeviceStream>> streams;
  // domain layouts by shape (value bytes, warps, page bytes, cut); a null entry: the factor admits none
  std::map<std::tuple<int, int, int, int>, std::unique_ptr<yb::DeviceDomain>> domains;
  // lane layouts by (value bytes, warps, page bytes); a null entry: the factor admits none
  std::map<std::tuple<int, int, int, int>, std::unique_ptr<yb::DeviceLane>> lanes;
  // spread layouts by (value bytes, groups up to; a null entry: the factor admits none) and the
  // workspaces, one per stream in use; the mutex guards both
  std::map<std::pair<int, int64_t>, std::unique_ptr<yb::DeviceSpread>> spreads;
  std::map<std::pair<int, int64_t>, int> spread_passes;  // a complex factor's solves without the layout of their class
  std::vector<std::unique_ptr<yb::SpreadWork>> spread_work;
  uint64_t spread_solves = 0;
  std::mutex spread_mutex;
  yb::DeviceArray<uint8_t> lane_work, lane_partial;  // the lane solve's work and partial arrays
  yb::LaneTiming lane_timing;
  yb::DeviceArray<int32_t> error;  // the device error word (a bounded wait that ran out)
  int32_t lane_withhold = -1;      // a test's page to withhold in the next plain lane solve, or -1
  long long *phase_clock = nullptr;  // diagnostics buffer of the caller's, or null
  yb::DeviceArray<double> scratch64;
  yb::DeviceArray<float> scratch32;
  yb::DeviceArray<double> dev_b, dev_x;
  // the matrix A the factor factors, for refinement: rows in natural order, columns mapped to
  // the solution slots, FP64
  int64_t a_rows = -1;
  yb::DeviceArray<int32_t> a_ptr, a_idx;
  yb::DeviceArray<int32_t> a_csr_ptr, a_csr_idx;  // A as attached (CSR, natural order)
  yb::DeviceArray<double> a_csr_val;
  yb::DeviceArray<double> a_val;
  std::vector<int64_t> a_host_ptr, a_host_idx;  // A as attached (CSR, natural order), on the host
  std::vector<double> a_host_val;
  int64_t a_attached = 0;                  // how many times a matrix was attached
  int64_t a_longest = 0;                   // entries of its longest row
  // a complex LU factor (yb_factor_from_lu_complex): its plan, its sweeps in complex128 and
  // complex64, and the complex matrix attached for refinement (CSR, natural order)
  bool is_complex = false;
  yb::Plan<yb::host::c128> cplan;
  yb::DeviceSweep<yb::cplx<double>> fwdz, bwdz;
  yb::DeviceSweep<yb::cplx<float>> fwdc, bwdc;
  int64_t za_rows = -1, za_longest = 0;  // (its rows, and the entries of its longest)
  yb::DeviceArray<int32_t> za_ptr, za_idx;
  yb::DeviceArray<yb::cplx<double>> za_val;
  yb::PinnedBuffer staging;
  yb::CopyPipeline pipe;
  // an LU factor's arrays as given (yb_factor_from_lu or _transposed), from which the transposed
  // solve makes the factor of the transposed matrix at its first use
  bool has_lu_arrays = false, lu_transposed = false;
  std::vector<int64_t> lu_l_ptr, lu_l_idx, lu_u_ptr, lu_u_idx, lu_p, lu_q;
  std::vector<double> lu_l_val, lu_u_val;
  std::unique_ptr<yb_factor> transposed;
  // the host-array refined solve's device arrays
  yb::DeviceArray<double> mixed_b, mixed_x, mixed_ratio;
  yb::DeviceArray<int32_t> mixed_steps;
  int64_t width = 1;
  yb::Timings timings;
  bool single = false;
  double single_lower = 1.0, single_upper = 1.0;
};

namespace yb {
// The automatic choice leaves factors whose elimination forest has few levels (stars, stars of stars, shallow
// trees, a few rows) to the domain solve, one launch whose time goes by levels, and to the lane solve: by the
// spread solve two rows took 11.7 against 9.3 us, a star of 200 22 to 55 against 21 to 39 us, one of 5,000 89 to
// 359 against 59 to 121, eight to a branch over nine levels 44 and 77 against 31 and 58 with 300 and 1,024
// right-hand sides, four to a branch over eleven 36 against 27 with 1,024; with 14 levels and more the domain solve
// took 1.2 times as long and more. In the refined solve, whose passes are many launches either way, up to seven.
constexpr int32_t kSpreadFewLevels = 11, kSpreadFewLevelsRefined = 7;
inline bool takes_spread(const yb_factor *f, const TileConfig &t, int32_t few = kSpreadFewLevels) {
  return t.spread_first || (t.admits_spread() && f->plan.fwd.levels > few);
}
// Of a few rows and thousands of right-hand sides the nine launches of an FP64 solve are more than the lane solve's
// three (100 rows with 2,500, 7,000 and 13,499 right-hand sides 30, 35 and 50 us against 29, 29 and 37; 200 rows 34, 46 and
// 63 against 35, 42 and 53; 300 rows 38, 48 and 87 against 41, 47 and 72 us).
inline bool lanes_for_few_rows(const yb_factor *f, const TileConfig &t, int64_t count) {
  return !t.spread_first && f->n <= 256 && count >= 2048;
}
// A refined solve also looks at the matrix: its residual takes a row by four lanes, so a hub's sets the time
// (2,000 buses, a hub of 300 branches 295 us a solve against 543 by the domain solve; 10,000, of 1,500 1,062 against 579).
inline bool has_hub(const yb_factor *f) {
  return f->a_longest > 512 && f->a_longest * f->n > 16 * (int64_t)f->a_host_idx.size();
}
void solve_pairs_device(yb_factor *f, int64_t count, const int32_t *plus, const int32_t *minus, const double *base,
                        const double *alpha, const double *inverse_weight, int32_t *singular, double *out, int64_t ldo,
                        cudaStream_t stream, bool captured = false);
// Plain FP64 solves by the spread solve where it is the automatic choice and the factor admits one; false,
// with nothing done, elsewhere. x may be b (with its leading dimension).
bool admits_spread_fp64(yb_factor *f, int64_t count, cudaStream_t stream);
bool auto_spread_fp64(yb_factor *f, const double *b, int64_t ldb, double *x, int64_t ldx, int64_t count, cudaStream_t stream);
cudaEvent_t *lane_timing_slot(yb_factor *f);  // the events of the next timed lane or spread solve, or null
void solve_single_row_device(yb_factor *f, const double *b, int64_t ldb, double *x, int64_t ldx, int64_t count,
                             cudaStream_t stream);
}
