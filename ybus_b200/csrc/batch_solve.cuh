// The multi-network batched solve (no ybus counterpart: ybus_cuda solves one real factor at a
// time): many factors of uneven orders and right-hand-side counts in one persistent launch. A
// work list of (network, tile) items, largest networks first, is dealt round-robin to the blocks;
// a block solves its item's tile of W right-hand sides through both sweeps of that network's
// factor, level by level with a block barrier between levels, its working vector in the block's
// slice of an L2-resident scratch buffer sized for the largest network. Values are complex here
// (cplx<float> or cplx<double>), for admittance (Ybus) LU factors; right-hand sides and solutions
// are complex128, column-major, natural order, interleaved (re, im).
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <type_traits>

#include "cplx.cuh"
#include "device.cuh"

namespace yb {

template <class T> struct BatchNet {
  int32_t n;
  SweepView<T> fwd, bwd;
  const int32_t *__restrict__ in_slot;
  const int32_t *__restrict__ out_slot;
  const cplx<double> *b;  // right-hand sides (or residuals), ldb per column
  int64_t ldb;
  cplx<double> *x;        // solutions, ldx per column
  int64_t ldx;
  int64_t count;
};

struct BatchItem {
  int32_t net, tile;
};

// One sweep of a network's tile: lane groups of W lanes take the rows of a level, lane c the
// right-hand side c; a block barrier after each level.
template <class T, int W>
__device__ __forceinline__ void batch_sweep(const SweepView<T> &s, T *Y, int group, int groups, int c) {
  for (int l = 0; l < s.levels; ++l) {
    const int k1 = s.level_ptr[l + 1];
    for (int k = s.level_ptr[l] + group; k < k1; k += groups) {
      const int r = s.row[k];
      const int p1 = s.ptr[k + 1];
      T acc = Y[(size_t)r * W + c];
      for (int p = s.ptr[k]; p < p1; ++p) acc -= s.val[p] * Y[(size_t)s.col[p] * W + c];
      Y[(size_t)r * W + c] = acc * s.dinv[k];
    }
    __syncthreads();
  }
}

// ACCUMULATE: x += the solution (a refinement step's correction) instead of x = the solution.
template <class T, int W, bool ACCUMULATE>
__global__ void __launch_bounds__(512) batch_solve_kernel(const BatchNet<T> *__restrict__ nets,
                                                          const BatchItem *__restrict__ items, int64_t n_items,
                                                          T *scratch, int64_t slice) {
  static_assert(32 % W == 0, "W divides a warp");
  constexpr int G = 32 / W;
  const int lane = threadIdx.x & 31;
  const int c = lane % W;
  const int group = (threadIdx.x >> 5) * G + lane / W;
  const int groups = (blockDim.x >> 5) * G;
  T *Y = scratch + (size_t)blockIdx.x * slice;
  for (int64_t i = blockIdx.x; i < n_items; i += gridDim.x) {
    const BatchItem item = items[i];
    const BatchNet<T> &net = nets[item.net];
    const int n = net.n;
    const int64_t col0 = (int64_t)item.tile * W;
    for (int r = threadIdx.x; r < n; r += blockDim.x) {
      const int sl = net.in_slot[r];
#pragma unroll
      for (int cc = 0; cc < W; ++cc) {
        const int64_t col = col0 + cc;
        Y[(size_t)sl * W + cc] = col < net.count ? T(net.b[col * net.ldb + r]) : T(0);
      }
    }
    __syncthreads();
    batch_sweep<T, W>(net.fwd, Y, group, groups, c);
    batch_sweep<T, W>(net.bwd, Y, group, groups, c);
    for (int r = threadIdx.x; r < n; r += blockDim.x) {
      const int sl = net.out_slot[r];
#pragma unroll
      for (int cc = 0; cc < W; ++cc) {
        const int64_t col = col0 + cc;
        if (col < net.count) {
          const cplx<double> v(Y[(size_t)sl * W + cc]);
          cplx<double> *xp = net.x + col * net.ldx + r;
          if (ACCUMULATE)
            *xp = *xp + v;
          else
            *xp = v;
        }
      }
    }
    __syncthreads();
  }
}

// The residual r = b - A x of every column of every network (A CSR in natural order, complex128,
// each row's products summed in stored order) and each column's ||r||inf / ||b||inf
// (accuracy.rs:58-79: 0 for a zero residual, infinity for a zero b with a nonzero residual).
struct ResidualNet {
  int32_t n;
  const int32_t *__restrict__ a_ptr;
  const int32_t *__restrict__ a_idx;
  const cplx<double> *__restrict__ a_val;
  const cplx<double> *b;
  int64_t ldb;
  const cplx<double> *x;
  int64_t ldx;
  cplx<double> *r;
  int64_t ldr;
  unsigned long long *norms;  // ||r||inf and ||b||inf of each column, as bit patterns (of doubles >= 0 these order alike), from the first residual on
};
struct ResidualItem {
  int32_t net, row, column, columns;  // kResidualRows rows from `row`, `columns` columns (at most kResidualColumns)
};
constexpr int kResidualRows = 1024, kResidualColumns = 4;
// A row of more entries is a chain that four columns at once make longer, so such a network's pieces have one (a
// star of 3,000 buses, complex64 refined with 16 and 1,024 right-hand sides: 1.0 and 2.9 against 2.1 and 3.0 ms), and so
// have all where four would leave SMs without a block.
constexpr int64_t kResidualLongRow = 128;

// ||r||inf / ||b||inf, 0 for a zero residual and infinity for a zero b with another
__host__ __device__ inline double batch_ratio(double rn, double bn) { return bn > 0.0 ? rn / bn : (rn > 0.0 ? HUGE_VAL : 0.0); }

// One block per ResidualItem. A row is a chain of loads (its bounds, a column index, an entry of x), so a
// thread takes four columns' at once, and the blocks are pieces of rows, so large and small networks
// fill the SMs alike. 21 million complex rows (16 networks of 730 to 46,293 buses, 128
// columns each): 654 us; a block per column, its threads striding over all rows, took 1,121 us. The
// entries of x come from L2 in sectors half used, 32 bytes each.
__global__ void __launch_bounds__(256) batch_residual_kernel(const ResidualNet *__restrict__ nets, const ResidualItem *__restrict__ items,
                                                             int64_t norms_at) {
  constexpr int C = kResidualColumns;
  __shared__ double most[8][2 * C];
  const ResidualItem it = items[blockIdx.x];
  const ResidualNet &net = nets[it.net];
  const int64_t ldx = net.ldx, ldb = net.ldb, ldr = net.ldr;
  const cplx<double> *b = net.b + it.column * ldb, *x = net.x + it.column * ldx;
  cplx<double> *r = net.r + it.column * ldr;
  double norm[2 * C] = {};
  // |z| is computed only where |re| + |im| says that it may be the largest so far
  auto larger = [](double &most, const cplx<double> &z) {
    if (fabs(z.re) + fabs(z.im) > most) most = fmax(most, magnitude(z));
  };
  const int end = min(net.n, it.row + kResidualRows);
  auto rows = [&](auto most_columns, auto all) {
    constexpr int C = decltype(most_columns)::value;
    for (int i = it.row + (int)threadIdx.x; i < end; i += 256) {
      cplx<double> ax[C];
      const int p1 = net.a_ptr[i + 1];
      for (int p = net.a_ptr[i]; p < p1; ++p) {
        const cplx<double> v = net.a_val[p];
        const cplx<double> *xj = x + net.a_idx[p];
#pragma unroll
        for (int c = 0; c < C; ++c)
          if (all || c < it.columns) ax[c] += v * xj[c * ldx];
      }
#pragma unroll
      for (int c = 0; c < C; ++c)
        if (all || c < it.columns) {
          const cplx<double> bi = b[c * ldb + i], ri = bi - ax[c];
          r[c * ldr + i] = ri;
          larger(norm[2 * c], ri), larger(norm[2 * c + 1], bi);
        }
    }
  };
  if (it.columns == C)
    rows(std::integral_constant<int, C>(), std::true_type());
  else if (it.columns == 1)
    rows(std::integral_constant<int, 1>(), std::true_type());
  else
    rows(std::integral_constant<int, C>(), std::false_type());
#pragma unroll
  for (int c = 0; c < 2 * C; ++c) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) norm[c] = fmax(norm[c], __shfl_xor_sync(0xffffffffu, norm[c], off));
    if ((threadIdx.x & 31) == 0) most[threadIdx.x >> 5][c] = norm[c];
  }
  __syncthreads();
  if (threadIdx.x < 2 * C && (int)threadIdx.x < 2 * it.columns) {
    double m = 0;
    for (int w = 0; w < 8; ++w) m = fmax(m, most[w][threadIdx.x]);
    atomicMax(net.norms + norms_at + 2 * it.column + threadIdx.x, (unsigned long long)__double_as_longlong(m));
  }
}

__global__ void __launch_bounds__(256) batch_ratio_kernel(int64_t columns, const unsigned long long *__restrict__ norms, double *__restrict__ ratio) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= columns) return;
  ratio[c] = batch_ratio(__longlong_as_double((long long)norms[2 * c]), __longlong_as_double((long long)norms[2 * c + 1]));
}

}  // namespace yb
