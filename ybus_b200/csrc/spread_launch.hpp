// The spread solve's entry points for the C ABI's translation units (spread_launch.cu).
#pragma once

#include <cstdint>
#include <functional>
#include <mutex>
#include <vector>

#include "factor_state.cuh"

namespace yb {

// The automatic choice takes the spread solve up to this many live values per lane: with more, too
// few warps fit an SM to cover their shared-memory latency.
constexpr int32_t kSpreadAutoSlots = 64, kSpreadAutoSlotsComplex = 96;

// The spread layout for `groups` groups of 32 right-hand sides with values of `value_bytes`, made and
// uploaded at its first use; null if the factor admits none. Under stream capture the nearest layout there
// is, of those that hold the refined solve's copy of the matrix attached as number `matrix` (-1: of all).
DeviceSpread *spread_for(yb_factor *f, int value_bytes, int64_t groups, cudaStream_t stream, int64_t matrix = -1);

// Solves `count` right-hand sides (device arrays, column-major) in T (double or float), in runs of the GPU's
// work limit; false, with nothing done, where the factor admits no spread layout (or has none yet under
// stream capture), where the limit is below a group's work array, and where the memory is not there.
template <class T>
bool spread_solve(yb_factor *f, const double *b, int64_t ldb, double *x, int64_t ldx, int64_t count, cudaStream_t stream);

// What takes the solutions where they are, in place of the scatter: columns `first` to `first + count` in groups
// of 32 at `work` ([group][position][32], an unknown's position in `out_pos`), by launches on the solve's stream.
using SpreadFinish = std::function<void(const double *work, const int32_t *out_pos, int64_t first, int64_t count)>;

// As spread_solve in FP64, the solutions taken by `finish`.
bool spread_solve_lanes(yb_factor *f, const double *b, int64_t ldb, int64_t count, cudaStream_t stream, const SpreadFinish &finish);

// A workspace for a solve on `stream` with at least the bytes asked for, held until the solve is enqueued
// (also by a launch that failed: what was enqueued before it still runs). Eagerly one of the factor's,
// ordered by its event; under capture one of that capture's own (a capture's solves on one stream follow one
// another), which the graph keeps by a user object.
class WorkLease {
 public:
  WorkLease(yb_factor *f, const SpreadBytes &bytes, cudaStream_t stream);
  ~WorkLease();
  WorkLease(const WorkLease &) = delete;
  WorkLease &operator=(const WorkLease &) = delete;
  SpreadWork *operator->() const { return w_; }

 private:
  std::lock_guard<std::mutex> lock_;
  cudaStream_t stream_;
  SpreadWork *w_ = nullptr;
};

// The sweeps and the top of `groups` groups whose right-hand sides are in `work` (at positions, with
// kSpreadPad rows before and after), the solutions into `xout` (work itself, or another array of its layout);
// `partial` holds spread_partial_bytes; groups with a zero in `group_active` (null: none) are skipped.
template <class T> size_t spread_partial_bytes(const DeviceSpread *d, int64_t groups);
template <class T>
void spread_sweeps(yb_factor *f, DeviceSpread *d, T *work, T *xout, uint8_t *partial, int64_t groups, const uint8_t *group_active,
                   cudaStream_t stream);

// A complex factor's solves that go without a layout before one is made: making it costs about what four take
// (16 networks of 730 to 46,293 buses with 128 right-hand sides each: 31 ms, against 7.5 ms a solve by tiles and
// 0.93 ms with it), so a factor that is solved once or twice never pays for it, and one that is solved often
// twice what the better choice would have cost.
constexpr int kSpreadBatchPasses = 4;
// A few rows, or some hundred in few levels, are less than the launches: two rows 14 us by tiles and 19 to 27 so,
// 585 rows of eight to a branch (13 levels) in complex64 with refinement 128 to 147 and 135 to 180. (30 buses, 17
// levels, 160 and 120 us, and a star of 3,000, 480 and 124 us, are not.)
inline bool small_for_batch(const yb_factor *f) { return f->n < 16 || (f->n <= 1024 && f->cplan.fwd.levels <= 13); }
constexpr int kSpreadMostBatchLayouts = 8;  // a complex factor keeps of one precision; further classes take the nearest

// The spread layouts of a batch of complex factors with these counts of right-hand sides: of the class the batch
// asks for, made on several threads of the host once the factor's solves in that class have paid for it;
// until then another class's, or null.
void spread_for_batch(const std::vector<yb_factor *> &factors, int value_bytes, const std::vector<int64_t> &counts,
                      std::vector<DeviceSpread *> &out, cudaStream_t stream);
// Counts a batch's solves of each factor.
void spread_batch_solved(const std::vector<yb_factor *> &factors, int value_bytes, const std::vector<int64_t> &counts, int solves);

// One factor's part of a complex batch: right-hand sides and solutions complex128, column-major.
struct SpreadSystem {
  yb_factor *factor;
  DeviceSpread *layout;
  const cplx<double> *b;
  cplx<double> *x;
  int64_t count;
};

// Whether the GPU's work limit holds a group of a system's right-hand sides in complex values of R.
template <class R> bool spread_batch_fits(const SpreadSystem &system);

// Solves every system's right-hand sides in complex values of R (double or float), into x or (add) onto it,
// in as many runs of launches as the GPU's work limit asks for. Throws OutOfMemory, with nothing done, where
// the work arrays cannot be had.
template <class R> void spread_batch(const std::vector<SpreadSystem> &systems, bool add, SpreadBatchWork &work, cudaStream_t stream);

}  // namespace yb
