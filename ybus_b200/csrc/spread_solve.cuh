// The spread solve: one right-hand side per lane, one warp per (task, group of 32 right-hand sides),
// no warp waiting for another. A task is a bundle of subtree domains of the elimination forest
// (SpreadLayout in plan.hpp); the sweeps below the top and the top itself are launches of their own:
//
//   spread_in     b into the work array [group][position][32 lanes]
//   spread_sweep  every task forward: z over b in the work array, updates of top rows into the
//                 partial array
//   spread_sum    the top's right-hand sides r_T: b_T plus the partials
//   spread_top    x_T as a dense product of r_T; but in real FP32 twice, and between them the residual, by
//                 spread_correct or, where the top's triangles are dense, by spread_top
//   spread_sweep  every task backward, from the top solutions
//   spread_out    the work array into x
//
// The rows are chains of dependent operations on values in shared memory (a few tens of live values
// per lane), so what bounds a sweep is the instructions per row and, with few right-hand sides, the
// longest chain. Hence: packets of four rows decoded together, their entries at fixed places (no
// dispatch per row); a task's rows consecutive in the work array, so addresses are one pointer's
// increments and the next rows are loaded while these are solved; and as many tasks as fill the SMs
// (a block's cooperation on one group, as in the lane solve, allows 16 warps at most).
//
// Measured on a B200, FP64 with device arrays, against the domain and lane solves that took these
// sizes before: 2,000-bus B' with one right-hand side 71 to 44 us; 10,000-bus B' with 64, 87 to 62 us,
// with 999, 329 to 175 us, with 13,499, 1,684 to 1,585 us (the gather 0.36 and the scatter 0.34 ms at
// 6.1 TB/s, the sweeps and the top 0.90 ms); the 10,000-bus Jacobian's LU with 4,096, 1,333 to 1,076 us; 16 complex
// networks of 730 to 46,293 buses with 128 each, complex128 7.5 to 0.93 ms, complex64 with refinement 21.0 to
// 4.4 ms. Of these the top's correction costs 15, 25, 34, 90, 40 and 20 us. What bounds it: for large
// blocks HBM in the gather and scatter and the shared-memory pipe (about 18 wavefronts a row and sweep) near HBM in
// the sweeps; for small ones the nine launches and the longest task's chain (about 290 cycles a row where a warp is
// alone).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "cplx.cuh"
#include "plan.hpp"

namespace yb {

constexpr int kSpreadWarps = 4;     // warps (groups) per block at most: they share a task's pages
constexpr int kSpreadIoWarps = 8;   // warps per block of the gather and the scatter
constexpr int kSpreadTopRows = 64;  // rows of a block of M: stored [block][column][row]

// One factor's layout and arrays, as the kernels read them.
struct SpreadNet {
  int32_t n, tasks, top, partials;
  const uint8_t *__restrict__ blob;
  const int32_t *__restrict__ fwd_page, *__restrict__ bwd_page, *__restrict__ task_row, *__restrict__ part_ptr;
  const int32_t *__restrict__ in_pos, *__restrict__ out_pos;
  const void *__restrict__ m;  // the top's map in blocks of kSpreadTopRows rows
  // what the product is corrected by, by rows: U_TT and then -L_TT; or these two dense, as m
  const int32_t *__restrict__ low_ptr, *__restrict__ low_col, *__restrict__ up_ptr, *__restrict__ up_col;
  const void *__restrict__ low_val, *__restrict__ up_val;
  const void *__restrict__ m_up, *__restrict__ m_low;
  int64_t groups, count;       // groups of a warp's columns (32, or 64 with two per lane), and columns
  void *work, *xout, *partial; // xout: where the backward sweep writes (work, or an array of its layout)
  void *r, *r2, *r3;           // the top's right-hand sides [group][top row][32 lanes], full precision; the first product; U_TT times it
  bool top_out;                // the top's solutions go to xout as well (the scatter takes them from the partial array)
  const uint8_t *group_active; // [groups] 0: skipped; null: all run
  const void *b;               // the caller's right-hand sides and solutions
  int64_t ldb;
  void *x;
  int64_t ldx;
};

// One network's arguments by value, or a batch's in device memory with the blocks' items.
struct SpreadItem {
  int32_t net, a, b, c;
};
struct SpreadArgs {
  SpreadNet one;
  const SpreadNet *nets;    // null: `one`
  const SpreadItem *items;  // per block
  int32_t slots;
};

// Two right-hand sides of a lane (adjacent columns of its group), for FP32 with many of them.
template <class R> struct pair2 {
  R a, b;
};

// What a lane holds, L: one right-hand side, or in FP32 two (each record then serves twice the
// arithmetic, in slots as wide as FP64's). S: the factor's values; Math: a lane's
// values in the top's product; MathS: the top's map; kCorrect: the product takes one correction (real FP32
// values round far more than it).
template <class L> struct SpreadLane;
template <> struct SpreadLane<double> {
  using S = double;
  using Math = double;
  using MathS = double;
  static constexpr int N = 1;
  static constexpr bool kComplex = false, kCorrect = true;
};
template <> struct SpreadLane<float> : SpreadLane<double> {
  using S = float;
  static constexpr bool kCorrect = false;
};
template <> struct SpreadLane<pair2<float>> {
  using S = float;
  using Math = pair2<double>;
  using MathS = double;
  static constexpr int N = 2;
  static constexpr bool kComplex = false, kCorrect = false;
};
template <> struct SpreadLane<cplx<double>> {
  using S = cplx<double>;
  using Math = cplx<double>;
  using MathS = cplx<double>;
  static constexpr int N = 1;
  static constexpr bool kComplex = true, kCorrect = true;
};
template <> struct SpreadLane<cplx<float>> : SpreadLane<cplx<double>> {
  using S = cplx<float>;
};

// acc - v x, x + y, x v, and conversions, for a factor's value v and lanes' values x, y
__device__ __forceinline__ double sp_fnma(double v, double x, double acc) { return fma(-v, x, acc); }
__device__ __forceinline__ float sp_fnma(float v, float x, float acc) { return fmaf(-v, x, acc); }
template <class R> __device__ __forceinline__ cplx<R> sp_fnma(cplx<R> v, cplx<R> x, cplx<R> acc) {
  return cplx<R>(fma(v.im, x.im, fma(-v.re, x.re, acc.re)), fma(-v.im, x.re, fma(-v.re, x.im, acc.im)));
}
template <class R> __device__ __forceinline__ pair2<R> sp_fnma(R v, pair2<R> x, pair2<R> acc) {
  return {sp_fnma(v, x.a, acc.a), sp_fnma(v, x.b, acc.b)};
}
__device__ __forceinline__ double sp_add(double x, double y) { return x + y; }
__device__ __forceinline__ float sp_add(float x, float y) { return x + y; }
template <class R> __device__ __forceinline__ cplx<R> sp_add(cplx<R> x, cplx<R> y) { return x + y; }
template <class R> __device__ __forceinline__ pair2<R> sp_add(pair2<R> x, pair2<R> y) { return {x.a + y.a, x.b + y.b}; }
__device__ __forceinline__ double sp_mul(double x, double v) { return x * v; }
__device__ __forceinline__ float sp_mul(float x, float v) { return x * v; }
template <class R> __device__ __forceinline__ cplx<R> sp_mul(cplx<R> x, cplx<R> v) { return x * v; }
template <class R> __device__ __forceinline__ pair2<R> sp_mul(pair2<R> x, R v) { return {x.a * v, x.b * v}; }
template <class To> struct SpreadAs;  // between a lane's values and the same in full precision
template <> struct SpreadAs<double> {
  static __device__ __forceinline__ double of(double x) { return x; }
};
template <> struct SpreadAs<float> {
  static __device__ __forceinline__ float of(double x) { return (float)x; }
};
template <class R> struct SpreadAs<cplx<R>> {
  template <class Q> static __device__ __forceinline__ cplx<R> of(const cplx<Q> &x) { return cplx<R>((R)x.re, (R)x.im); }
};
template <class R> struct SpreadAs<pair2<R>> {
  template <class Q> static __device__ __forceinline__ pair2<R> of(const pair2<Q> &x) { return {(R)x.a, (R)x.b}; }
};

// A lane's value as plain words of 4, 8 or 16 bytes, moved in one access.
template <int BYTES> struct SpreadWord;
template <> struct SpreadWord<4> {
  using type = float;
};
template <> struct SpreadWord<8> {
  using type = float2;
};
template <> struct SpreadWord<16> {
  using type = float4;
};
template <class L> __device__ __forceinline__ L sp_cast(typename SpreadWord<sizeof(L)>::type w) {
  union U {
    typename SpreadWord<sizeof(L)>::type w;
    L l;
    __device__ U() {}
  } u;
  u.w = w;
  return u.l;
}
template <class L> __device__ __forceinline__ typename SpreadWord<sizeof(L)>::type sp_uncast(const L &l) {
  union U {
    typename SpreadWord<sizeof(L)>::type w;
    L l;
    __device__ U() {}
  } u;
  u.l = l;
  return u.w;
}
// global memory, past L1 (each row is read once per sweep)
template <class L> __device__ __forceinline__ L sp_ldg(const L *p) {
  return sp_cast<L>(__ldcg(reinterpret_cast<const typename SpreadWord<sizeof(L)>::type *>(p)));
}
template <class L> __device__ __forceinline__ void sp_stg(L *p, const L &v) {
  *reinterpret_cast<typename SpreadWord<sizeof(L)>::type *>(p) = sp_uncast(v);
}

// Group g's solutions of the top rows in the partial array, past every group's partials (in values).
__device__ __forceinline__ size_t spread_top_row(const SpreadNet &net, int64_t g) {
  return ((size_t)net.groups * net.partials + (size_t)g * net.top) * 32;
}

extern __shared__ __align__(128) unsigned char spread_shared[];

template <class T> __device__ __forceinline__ T &sp_at(uint32_t off) { return *reinterpret_cast<T *>(spread_shared + off); }
template <class L> __device__ __forceinline__ L sp_lds(uint32_t o) { return sp_cast<L>(sp_at<typename SpreadWord<sizeof(L)>::type>(o)); }
template <class L> __device__ __forceinline__ void sp_sts(uint32_t o, const L &v) {
  sp_at<typename SpreadWord<sizeof(L)>::type>(o) = sp_uncast(v);
}

// A row's record and a further pair at shared offset o (SpreadLayout in plan.hpp).
template <class S> struct SpreadRecord;
template <> struct SpreadRecord<double> {
  static __device__ __forceinline__ void row(uint32_t o, double &v0, double &v1, double &d, uint32_t &slots, uint32_t &flags) {
    const double2 v = sp_at<double2>(o);
    const uint4 h = sp_at<uint4>(o + 16);
    v0 = v.x, v1 = v.y, d = __hiloint2double((int)h.y, (int)h.x), slots = h.z, flags = h.w;
  }
  static __device__ __forceinline__ void pair(uint32_t o, double &v0, double &v1, uint32_t &w) {
    const double2 v = sp_at<double2>(o);
    v0 = v.x, v1 = v.y, w = sp_at<uint32_t>(o + 16);
  }
};
template <> struct SpreadRecord<float> {
  static __device__ __forceinline__ void row(uint32_t o, float &v0, float &v1, float &d, uint32_t &slots, uint32_t &flags) {
    const float4 v = sp_at<float4>(o);
    v0 = v.x, v1 = v.y, d = v.z, slots = __float_as_uint(v.w), flags = sp_at<uint32_t>(o + 16);
  }
  static __device__ __forceinline__ void pair(uint32_t o, float &v0, float &v1, uint32_t &w) {
    const float4 v = sp_at<float4>(o);
    v0 = v.x, v1 = v.y, w = __float_as_uint(v.z);
  }
};
template <> struct SpreadRecord<cplx<float>> {
  using C = cplx<float>;
  static __device__ __forceinline__ void row(uint32_t o, C &v0, C &v1, C &d, uint32_t &slots, uint32_t &flags) {
    const float4 v = sp_at<float4>(o), h = sp_at<float4>(o + 16);
    v0 = C(v.x, v.y), v1 = C(v.z, v.w), d = C(h.x, h.y), slots = __float_as_uint(h.z), flags = __float_as_uint(h.w);
  }
  static __device__ __forceinline__ void pair(uint32_t o, C &v0, C &v1, uint32_t &w) {
    const float4 v = sp_at<float4>(o);
    v0 = C(v.x, v.y), v1 = C(v.z, v.w), w = sp_at<uint32_t>(o + 16);
  }
};
template <> struct SpreadRecord<cplx<double>> {
  using C = cplx<double>;
  static __device__ __forceinline__ void row(uint32_t o, C &v0, C &v1, C &d, uint32_t &slots, uint32_t &flags) {
    const double2 a = sp_at<double2>(o), b = sp_at<double2>(o + 16), c = sp_at<double2>(o + 32);
    const uint2 h = sp_at<uint2>(o + 48);
    v0 = C(a.x, a.y), v1 = C(b.x, b.y), d = C(c.x, c.y), slots = h.x, flags = h.y;
  }
  static __device__ __forceinline__ void pair(uint32_t o, C &v0, C &v1, uint32_t &w) {
    const double2 a = sp_at<double2>(o), b = sp_at<double2>(o + 16);
    v0 = C(a.x, a.y), v1 = C(b.x, b.y), w = sp_at<uint32_t>(o + 32);
  }
};

// The work array's rows on their way to a warp: a ring of chunks of four rows.
template <class L> __host__ __device__ constexpr int spread_chunk_bytes() { return 4 * 32 * (int)sizeof(L); }
template <class L> __host__ __device__ constexpr int spread_ring() { return sizeof(L) == 16 ? 2 : 4; }
// A block's dynamic shared memory: two pages, then each warp's ring and slots.
template <class L> __host__ __device__ inline size_t spread_smem(int32_t slots, int warps) {
  return 2 * (size_t)kSpreadPage + (size_t)warps * (spread_ring<L>() * spread_chunk_bytes<L>() + (size_t)slots * 32 * sizeof(L));
}
// The blocks of kSpreadWarps warps an SM's registers hold, which the kernel is bounded to.
template <class L> __host__ __device__ constexpr int spread_blocks() {
  return sizeof(L) == 16 ? 5 : sizeof(L) == 8 ? 6 : 8;
}

// The launches of a solve overlap by programmatic dependent launch: a kernel lets the next one start
// its blocks as its own finish, and touches nothing another kernel writes before sp_ready(), which
// every thread passes (so a kernel never completes before the ones it follows).
__device__ __forceinline__ void sp_ready() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ void sp_barrier() { asm volatile("barrier.sync 0;" ::: "memory"); }

// One sweep of every task below the top. Block: one task, up to kSpreadWarps groups, which run the
// same packets in near lockstep and share the pages (cp.async into the half the block has left, one
// block barrier per page). A row's record is loaded while the row before it is solved; its slots are
// read together (the layout keeps them apart), a slot's first update stores without reading, and what
// one row leaves to the next (its parent forward, its child backward, in a postorder nearly half of
// all rows) stays in a register. The work array's rows come through a ring of chunks of four by
// cp.async, a chunk a packet (in registers they came out later: a value in flight is waited for with
// all loads that share its scoreboard).
template <class L, bool BACK, bool BATCH>
__global__ void __launch_bounds__(kSpreadWarps * 32, spread_blocks<L>()) spread_sweep_kernel(const __grid_constant__ SpreadArgs a) {
  using S = typename SpreadLane<L>::S;
  using Rec = SpreadRecord<S>;
  constexpr uint32_t VB = sizeof(L), RB = spread_row_bytes(sizeof(S)), PB = spread_pair_bytes(sizeof(S));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  int32_t task;
  int64_t g;
  const SpreadNet *np = &a.one;
  if constexpr (BATCH) {
    const SpreadItem it = a.items[blockIdx.x];
    np = a.nets + it.net;
    task = it.a, g = (int64_t)it.b + warp;
  } else {
    const int64_t chunks = (a.one.groups + warps - 1) / warps;
    task = (int32_t)(blockIdx.x / chunks), g = (blockIdx.x - task * chunks) * warps + warp;
  }
  const SpreadNet &net = *np;
  const int32_t *pages = BACK ? net.bwd_page : net.fwd_page;
  const int p0 = __ldg(pages + 2 * task), count = __ldg(pages + 2 * task + 1);
  const uint8_t *src = net.blob + (size_t)p0 * kSpreadPage;
  auto fetch = [&](int k) {  // page k into its half, by the whole block
    for (int o = threadIdx.x * 16; o < kSpreadPage; o += (int)blockDim.x * 16)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(spread_shared + (k & 1) * kSpreadPage + o)),
                   "l"(src + (size_t)k * kSpreadPage + o)
                   : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int since = 0;  // chunks fetched since the last page was
  constexpr int RING = spread_ring<L>();
  auto turn = [&](int k) {  // to page k: it is there, and every warp has left page k - 1
    if (since >= RING)
      asm volatile("cp.async.wait_group %0;" ::"n"(RING) : "memory");
    else
      asm volatile("cp.async.wait_all;" ::: "memory");
    sp_barrier();
    if (k + 1 < count) fetch(k + 1);
    since = 0;
  };
  fetch(0);  // the layout's: no kernel writes it
  sp_ready();
  const bool act = g < net.groups && (!net.group_active || net.group_active[g]);
  if (!__syncthreads_or(act)) {  // the whole block
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  if (!act) {  // a warp without a group helps with the pages
    for (int k = 0; k < count; ++k) turn(k);
    return;
  }
  constexpr uint32_t CHUNK = spread_chunk_bytes<L>();
  const uint32_t rows = 2 * kSpreadPage + (uint32_t)warp * (RING * CHUNK + (uint32_t)a.slots * 32 * VB);  // the ring
  const uint32_t live = rows + RING * CHUNK + lane * VB;  // slot 0
  auto slot = [&](uint32_t i) { return live + i * (32 * VB); };
  const int r0 = __ldg(net.task_row + task), r1 = __ldg(net.task_row + task + 1);
  const size_t base = (size_t)g * net.n * 32;
  constexpr int STEP = BACK ? -32 : 32;
  // this lane's part of the next chunk (four rows in the work array's order, the first of them the
  // last to be solved backward), and where the next row's result goes
  const char *in = nullptr;
  L *out = static_cast<L *>(BACK ? net.xout : net.work) + base + (int64_t)(BACK ? r1 - 1 : r0) * 32 + lane;
  uint32_t put = 0, get = 0;  // ring offsets
  auto chunk = [&]() {  // fetches the next chunk; past the task's rows: unused, in other rows or the padding
#pragma unroll
    for (uint32_t o = 0; o < CHUNK; o += 512)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(spread_shared) + rows + put + o + lane * 16),
                   "l"(in + o)
                   : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    in += STEP * 4 * (int)VB;
    put = (put + CHUNK) & (RING * CHUNK - 1);
    ++since;
  };
  auto refill = [&](int64_t done) {  // the ring from the task's done-th row on
    in = reinterpret_cast<const char *>(static_cast<const L *>(net.work) + base + (BACK ? r1 - 4 - done : r0 + done) * 32) + lane * 16;
#pragma unroll
    for (int c = 0; c < RING; ++c) chunk();
  };
  refill(0);
  bool stale = false;  // the ring no longer holds the rows to come
  L z{};               // forward: the last row's result; backward: the sum a long row starts from
  L carry{};           // what the last row leaves to the next
  auto further = [&](uint32_t o) {  // a further pair of the last row's entries
    S v0, v1;
    uint32_t w;
    Rec::pair(o, v0, v1, w);
    const uint32_t t0 = slot(w & 0xff), t1 = slot((w >> 8) & 0xff);
    L x0{}, x1{};
    if (w & (kSpreadLoad0 << 16)) x0 = sp_lds<L>(t0);
    if (w & (kSpreadLoad1 << 16)) x1 = sp_lds<L>(t1);
    if constexpr (!BACK) {
      sp_sts(t0, sp_fnma(v0, z, x0));
      if (w & (kSpreadStore1 << 16)) sp_sts(t1, sp_fnma(v1, z, x1));
    } else {
      z = sp_fnma(v0, x0, z);
      if (w & (kSpreadLoad1 << 16)) z = sp_fnma(v1, x1, z);
    }
  };
  int page = 0;
  uint32_t at = 0;
  turn(0);
  // solves the N rows of the packet at `at`; v(q): row q's value
  auto solve = [&](auto rows_c, auto v) {
    constexpr int N = decltype(rows_c)::value;
    uint32_t more = at + 16 + N * RB;
    S d, v0, v1;
    uint32_t slots, flags;
    Rec::row(at + 16, v0, v1, d, slots, flags);
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const S dq = d, a0 = v0, a1 = v1;
      const uint32_t f = flags, s0 = slot(slots & 0xff), t0 = slot((slots >> 8) & 0xff), t1 = slot(slots >> 16);
      if (q + 1 < N) Rec::row(at + 16 + (q + 1) * RB, v0, v1, d, slots, flags);
      if constexpr (!BACK) {
        L x0{}, x1{};
        if (f & kSpreadSelf) carry = sp_lds<L>(s0);
        if (f & kSpreadLoad0) x0 = sp_lds<L>(t0);
        if (f & kSpreadLoad1) x1 = sp_lds<L>(t1);
        z = sp_mul(sp_add(v(q), carry), dq);
        sp_stg(out + q * STEP, z);
        carry = sp_fnma(a0, z, x0);
        x1 = sp_fnma(a1, z, x1);
        if (f & kSpreadStore0) sp_sts(t0, carry);
        if (f & kSpreadStore1) sp_sts(t1, x1);
        if (!(f & kSpreadCarry)) carry = L{};
      } else {
        L x0 = carry, x1{};
        if (f & kSpreadLoad0) x0 = sp_lds<L>(t0);
        if (f & kSpreadLoad1) x1 = sp_lds<L>(t1);
        z = N == 1 ? sp_add(v(q), z) : v(q);  // a long row starts from its packets' sum
        if (f & (kSpreadLoad0 | kSpreadCarry)) z = sp_fnma(a0, x0, z);
        if (f & kSpreadLoad1) z = sp_fnma(a1, x1, z);
      }
      for (uint32_t left = f >> 8; left > 0; --left, more += PB) further(more);
      if constexpr (BACK) {
        carry = sp_mul(z, dq);
        if (f & kSpreadSelf) sp_sts(s0, carry);
        sp_stg(out + q * STEP, carry);
      }
    }
    if constexpr (BACK) z = L{};
    out += N * STEP;
  };
  for (;;) {
    const uint4 h = sp_at<uint4>(at);
    if (h.x == kSpreadRows4) {
      if (stale) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        put = get = 0, stale = false;
        const int64_t row = (out - lane - static_cast<L *>(BACK ? net.xout : net.work) - (int64_t)base) / 32;
        refill(BACK ? r1 - 1 - row : row - r0);
      }
      asm volatile("cp.async.wait_group %0;" ::"n"(RING - 1) : "memory");
      __syncwarp();  // every lane's part of the chunk is there
      const uint32_t from = rows + get + lane * VB;
      solve(std::integral_constant<int, 4>(), [&](int q) { return sp_lds<L>(from + (BACK ? 3 - q : q) * 32 * VB); });
      get = (get + CHUNK) & (RING * CHUNK - 1);
      __syncwarp();  // every lane has read the chunk
      chunk();
    } else {
      if (h.x == kSpreadRows1) {
        const L v = sp_ldg(static_cast<const L *>(net.work) + (out - static_cast<const L *>(BACK ? net.xout : net.work)));
        solve(std::integral_constant<int, 1>(), [&](int) { return v; });
        stale = true;
      } else if (h.x == kSpreadMove) {
        if constexpr (!BACK) {
          L *part = static_cast<L *>(net.partial) + (size_t)g * net.partials * 32 + lane;
          for (uint32_t i = 0; i < h.z; ++i) {
            const uint2 m = sp_at<uint2>(at + 16 + 8 * i);
            sp_stg(part + (size_t)m.x * 32, sp_lds<L>(slot(m.y)));
          }
        } else {
          const L *top = static_cast<const L *>(net.partial) + spread_top_row(net, g) + lane;
          for (uint32_t i = 0; i < h.z; i += 4) {  // four loads in flight
            L x[4];
            uint32_t o[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint2 m = sp_at<uint2>(at + 16 + 8 * min(i + q, h.z - 1));
              x[q] = sp_ldg(top + (size_t)m.x * 32), o[q] = slot(m.y);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) sp_sts(o[q], x[q]);
          }
        }
      } else if (h.x == kSpreadMore) {
        for (uint32_t i = 0; i < h.z; ++i) further(at + 16 + i * PB);
      } else if (h.x == kSpreadPageEnd) {
        turn(++page);
        at = (uint32_t)(page & 1) * kSpreadPage;
        continue;
      } else {
        break;
      }
    }
    at += h.y;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");  // the chunks past the task's rows
}

// Partial rows q0 to q1 of a group added to s, in order, eight loads in flight.
template <class T, class M> __device__ __forceinline__ M spread_sum_rows(const T *part, int q0, int q1, M s) {
  for (int q = q0; q < q1; q += 8) {
    T p[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) p[i] = sp_ldg(part + (size_t)min(q + i, q1 - 1) * 32);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (q + i < q1) s = sp_add(s, SpreadAs<M>::of(p[i]));
  }
  return s;
}

// A row of a block of eight that the block's eight warps share, an eighth each, added up in order: a hub's,
// of more than 64 entries and most of all the block's, which would be one warp's chain (2,000 buses with a hub of
// 300 branches: 52 us of 77 with the hub's rows to a warp each).
__device__ __forceinline__ bool spread_long_row(int some, int of_block) { return some > 64 && 2 * some > of_block; }

// The top's right-hand sides r_T: each top row's b and its partials, in order, in the factor's full
// precision. A warp per row and group, long rows by all.
template <class T, bool BATCH> __global__ void __launch_bounds__(256) spread_sum_kernel(const __grid_constant__ SpreadArgs a) {
  using M = typename SpreadLane<T>::Math;
  __shared__ __align__(16) unsigned char shared[8 * 32 * sizeof(M)];
  M *eighth = reinterpret_cast<M *>(shared);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t g;
  int k0;
  const SpreadNet *np = &a.one;
  if constexpr (BATCH) {
    const SpreadItem it = a.items[blockIdx.x];
    np = a.nets + it.net;
    g = it.b, k0 = it.a * 8;
  } else {
    const int blocks = (a.one.top + 7) / 8;
    g = blockIdx.x / blocks, k0 = (int)(blockIdx.x % blocks) * 8;
  }
  const SpreadNet &net = *np;
  sp_ready();
  if (net.group_active && !net.group_active[g]) return;  // the whole block
  const T *part = static_cast<const T *>(net.partial) + (size_t)g * net.partials * 32 + lane;
  const T *b = static_cast<const T *>(net.work) + ((size_t)g * net.n + net.n - net.top) * 32 + lane;
  M *r = static_cast<M *>(net.r) + (size_t)g * net.top * 32 + lane;
  const int k = k0 + warp, of_block = __ldg(net.part_ptr + min(k0 + 8, net.top)) - __ldg(net.part_ptr + k0);
  if (k < net.top) {
    const int q0 = __ldg(net.part_ptr + k), q1 = __ldg(net.part_ptr + k + 1);
    if (!spread_long_row(q1 - q0, of_block)) sp_stg(r + (size_t)k * 32, spread_sum_rows(part, q0, q1, SpreadAs<M>::of(sp_ldg(b + (size_t)k * 32))));
  }
  if (of_block <= 64) return;
  for (int j = k0; j < min(k0 + 8, net.top); ++j) {  // alike in every warp
    const int q0 = __ldg(net.part_ptr + j), some = __ldg(net.part_ptr + j + 1) - q0;
    if (!spread_long_row(some, of_block)) continue;
    eighth[warp * 32 + lane] = spread_sum_rows(part, q0 + some * warp / 8, q0 + some * (warp + 1) / 8, M{});
    __syncthreads();
    if (warp == 0) {
      M s = SpreadAs<M>::of(sp_ldg(b + (size_t)j * 32));
      for (int w = 0; w < 8; ++w) s = sp_add(s, eighth[w * 32 + lane]);
      sp_stg(r + (size_t)j * 32, s);
    }
    __syncthreads();
  }
}

__device__ __forceinline__ double sp_shfl(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
__device__ __forceinline__ cplx<double> sp_shfl(const cplx<double> &v, int lane) {
  return cplx<double>(__shfl_sync(0xffffffffu, v.re, lane), __shfl_sync(0xffffffffu, v.im, lane));
}

// s less the entries q0 to q1 times their rows of x: 32 entries at a time, a lane each, the next ones on their
// way; their values of x eight in flight.
template <class MS, class M>
__device__ __forceinline__ M spread_row_product(const int32_t *col, const MS *val, const M *x, int q0, int q1, M s) {
  const int lane = threadIdx.x & 31;
  int c_next = 0;
  MS v_next{};
  auto fetch = [&](int at) {
    if (at < q1) c_next = __ldg(col + at), v_next = sp_ldg(val + at);
  };
  fetch(q0 + lane);
  for (int q = q0; q < q1; q += 32) {
    const int some = min(32, q1 - q), c = c_next;
    const MS v = v_next;
    fetch(q + 32 + lane);
    for (int j = 0; j < some; j += 8) {
      M xs[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) xs[i] = sp_ldg(x + (size_t)__shfl_sync(0xffffffffu, c, min(j + i, some - 1)) * 32);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const MS vi = sp_shfl(v, min(j + i, some - 1));
        if (j + i < some) s = sp_fnma(vi, xs[i], s);
      }
    }
  }
  return s;
}

// The residual of the first product, for its correction: r3 = -U_TT r2 (UPPER), then r_T += L_TT r3, each row in
// place. A warp per row and group, long rows by all.
template <class T, bool BATCH, bool UPPER>
__global__ void __launch_bounds__(256) spread_correct_kernel(const __grid_constant__ SpreadArgs a) {
  using M = typename SpreadLane<T>::Math;
  using MS = typename SpreadLane<T>::MathS;
  __shared__ __align__(16) unsigned char shared[8 * 32 * sizeof(M)];
  M *eighth = reinterpret_cast<M *>(shared);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t g;
  int k0;
  const SpreadNet *np = &a.one;
  if constexpr (BATCH) {
    const SpreadItem it = a.items[blockIdx.x];
    np = a.nets + it.net;
    g = it.b, k0 = it.a * 8;
  } else {
    const int blocks = (a.one.top + 7) / 8;
    g = blockIdx.x / blocks, k0 = (int)(blockIdx.x % blocks) * 8;
  }
  const SpreadNet &net = *np;
  sp_ready();
  if (net.group_active && !net.group_active[g]) return;  // the whole block
  const int32_t *ptr = UPPER ? net.up_ptr : net.low_ptr, *col = UPPER ? net.up_col : net.low_col;
  const MS *val = static_cast<const MS *>(UPPER ? net.up_val : net.low_val);
  const M *x = static_cast<const M *>(UPPER ? net.r2 : net.r3) + (size_t)g * net.top * 32 + lane;
  M *to = static_cast<M *>(UPPER ? net.r3 : net.r) + (size_t)g * net.top * 32 + lane;
  const int k = k0 + warp, of_block = __ldg(ptr + min(k0 + 8, net.top)) - __ldg(ptr + k0);
  if (k < net.top) {
    const int q0 = __ldg(ptr + k), q1 = __ldg(ptr + k + 1);
    if (!spread_long_row(q1 - q0, of_block)) sp_stg(to + (size_t)k * 32, spread_row_product(col, val, x, q0, q1, UPPER ? M{} : sp_ldg(to + (size_t)k * 32)));
  }
  if (of_block <= 64) return;
  for (int j = k0; j < min(k0 + 8, net.top); ++j) {  // alike in every warp
    const int q0 = __ldg(ptr + j), some = __ldg(ptr + j + 1) - q0;
    if (!spread_long_row(some, of_block)) continue;
    eighth[warp * 32 + lane] = spread_row_product(col, val, x, q0 + some * warp / 8, q0 + some * (warp + 1) / 8, M{});
    __syncthreads();
    if (warp == 0) {
      M s = UPPER ? M{} : sp_ldg(to + (size_t)j * 32);
      for (int w = 0; w < 8; ++w) s = sp_add(s, eighth[w * 32 + lane]);
      sp_stg(to + (size_t)j * 32, s);
    }
    __syncthreads();
  }
}

// D += A B on the FP64 tensor cores: A 8 x 4 (lane: row lane / 4, column lane % 4), B 4 x 8 (row lane % 4,
// column lane / 4), D 8 x 8 (row lane / 4, columns 2 (lane % 4) and the next).
__device__ __forceinline__ void sp_mma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}
__device__ __forceinline__ void sp_mma(cplx<double> (&d)[2], cplx<double> a, cplx<double> b) {
  double re[2] = {d[0].re, d[1].re}, im[2] = {d[0].im, d[1].im};
  sp_mma(re, a.re, b.re), sp_mma(im, a.re, b.im);
  sp_mma(re, -a.im, b.im), sp_mma(im, a.im, b.re);
  d[0] = cplx<double>(re[0], im[0]), d[1] = cplx<double>(re[1], im[1]);
}
// two adjacent values of a row in one access
__device__ __forceinline__ void sp_store2(double *p, double a, double b) { *reinterpret_cast<double2 *>(p) = make_double2(a, b); }
__device__ __forceinline__ void sp_store2(float *p, double a, double b) { *reinterpret_cast<float2 *>(p) = make_float2((float)a, (float)b); }
__device__ __forceinline__ void sp_store2(cplx<double> *p, cplx<double> a, cplx<double> b) { sp_stg(p, a), sp_stg(p + 1, b); }
__device__ __forceinline__ void sp_store2(cplx<float> *p, cplx<double> a, cplx<double> b) {
  *reinterpret_cast<float4 *>(p) = make_float4((float)a.re, (float)a.im, (float)b.re, (float)b.im);
}

__device__ __forceinline__ bool sp_finite(double v) { return isfinite(v); }
__device__ __forceinline__ bool sp_finite(const cplx<double> &v) { return isfinite(v.re) && isfinite(v.im); }
__device__ __forceinline__ bool sp_zero(double v) { return v == 0.0; }
__device__ __forceinline__ bool sp_zero(const cplx<double> &v) { return v.re == 0.0 && v.im == 0.0; }

// An entry of the top's product over the map's entries that are not zero: the tensor product's zeros times a
// right-hand side that is not finite would carry it to rows that do not depend on it (another island's).
template <class V> __device__ __forceinline__ V spread_top_entry(const V *m, const V *r, int t, int cols) {
  V s(0);
#pragma unroll 1
  for (int k = 0; k < t; ++k)
    if (!sp_zero(m[(size_t)k * kSpreadTopRows])) s = sp_fnma(m[(size_t)k * kSpreadTopRows], r[(size_t)k * cols], s);
  return V(0) - s;
}

// The top's product on the FP64 tensor cores, 16 rows by 32 columns a warp, fragments straight from L2
// (the map and a group's columns are read by many warps; four steps of loads in flight). PHASE 0: x_T =
// M r_T; 1: r2 = M r_T; 2, with r_T the residual: x_T = r2 + M r_T, each entry of the correction where it is
// finite (a right-hand side that is not leaves a residual that is NaN). The residual by dense triangles, their
// zeros passed over: 3: r3 = U_TT r2; 4: r_T -= L_TT r3. KS > 1: a block's KS
// warps split the map's columns and add up in order at the end: with few groups there are too few
// tiles to fill the SMs, and a tile's chain of steps sets the time. x_T goes to its own rows after the
// partials (the work array's top rows stay b_T) and to the separate output array if there is one.
template <class T> __host__ __device__ constexpr int spread_split() { return SpreadLane<T>::kComplex ? 4 : 8; }
template <class T, int KS> __host__ __device__ constexpr int spread_top_warps() { return KS > 1 ? KS : 8; }
template <class T, bool BATCH, int KS, int PHASE>
__global__ void __launch_bounds__(spread_top_warps<T, KS>() * 32) spread_top_kernel(const __grid_constant__ SpreadArgs a) {
  constexpr int WARPS = spread_top_warps<T, KS>();
  using V = typename SpreadLane<T>::MathS;  // a value of M or r
  using S = typename SpreadLane<T>::S;      // of x
  constexpr int TILES = SpreadLane<T>::N, COLS = 32 * TILES;  // column tiles and columns of a group
  __shared__ V red[KS > 1 ? WARPS : 1][KS > 1 ? 16 : 1][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t block, g;
  const SpreadNet *np = &a.one;
  if constexpr (BATCH) {
    const SpreadItem it = a.items[blockIdx.x];
    np = a.nets + it.net;
    block = it.a, g = it.b;
  } else {
    const int64_t all = a.one.groups * TILES;
    block = blockIdx.x / all, g = blockIdx.x % all;
  }
  const int tile = (int)(g % TILES);
  g /= TILES;
  const SpreadNet &net = *np;
  sp_ready();
  if (net.group_active && !net.group_active[g]) return;  // the whole block
  const int t = net.top, row0 = ((int)block * (WARPS / KS) + warp / KS) * 16;
  const void *from = PHASE == 3 ? net.r2 : PHASE == 4 ? net.r3 : net.r, *by = PHASE == 3 ? net.m_up : PHASE == 4 ? net.m_low : net.m;
  const V *r = static_cast<const V *>(from) + (size_t)g * t * COLS + tile * 32 + lane / 4;
  const V *m = static_cast<const V *>(by) + (size_t)(row0 / kSpreadTopRows) * t * kSpreadTopRows + row0 % kSpreadTopRows + lane / 4;
  V acc[2][4][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = V(0);
  // the steps of four columns that hold entries of these rows, and this warp's share of them
  const int first = PHASE == 3 ? row0 / 4 : 0, steps = ((PHASE == 4 ? min(t, row0 + 16) : t) + 3) / 4 - first;
  const int s0 = first + (int)((int64_t)steps * (warp % KS) / KS), s1 = first + (int)((int64_t)steps * (warp % KS + 1) / KS);
  if (row0 < t) {
#pragma unroll 4
    for (int s = s0; s < s1; ++s) {
      const int k = 4 * s + (lane & 3);
      V av[2], bv[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) av[i] = k < t ? sp_ldg(m + (size_t)k * kSpreadTopRows + 8 * i) : V(0);
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = k < t ? sp_ldg(r + (size_t)k * COLS + 8 * j) : V(0);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) sp_mma(acc[i][j], av[i], bv[j]);
    }
  }
  S *xt = reinterpret_cast<S *>(static_cast<T *>(net.partial) + spread_top_row(net, g)) + tile * 32;
  S *xo = net.top_out ? reinterpret_cast<S *>(static_cast<T *>(net.xout) + ((size_t)g * net.n + net.n - t) * 32) + tile * 32 : nullptr;
  V *r2 = static_cast<V *>(net.r2) + (size_t)g * t * COLS + tile * 32;
  auto store = [&](int row, int col, V v0, V v1) {
    if (row >= t) return;
    if (!sp_finite(v0) || !sp_finite(v1)) {
      const V *mr = static_cast<const V *>(by) + (size_t)(row / kSpreadTopRows) * t * kSpreadTopRows + row % kSpreadTopRows;
      const V *rc = static_cast<const V *>(from) + (size_t)g * t * COLS + tile * 32 + col;
      if (!sp_finite(v0)) v0 = spread_top_entry(mr, rc, t, COLS);
      if (!sp_finite(v1)) v1 = spread_top_entry(mr, rc + 1, t, COLS);
    }
    V *between = r2 + (size_t)row * COLS + col;
    if constexpr (PHASE == 3 || PHASE == 4) {
      V *to = static_cast<V *>(PHASE == 3 ? net.r3 : net.r) + (size_t)g * t * COLS + tile * 32 + (size_t)row * COLS + col;
      if constexpr (PHASE == 4) v0 = sp_add(to[0], v0), v1 = sp_add(to[1], v1);  // m_low is -L_TT
      sp_store2(to, v0, v1);
      return;
    }
    if constexpr (PHASE == 1) {
      sp_store2(between, v0, v1);
      return;
    }
    if constexpr (PHASE == 2) {
      v0 = sp_finite(v0) ? sp_add(between[0], v0) : between[0];
      v1 = sp_finite(v1) ? sp_add(between[1], v1) : between[1];
    }
    sp_store2(xt + (size_t)row * COLS + col, v0, v1);
    if (xo) sp_store2(xo + (size_t)row * COLS + col, v0, v1);
  };
  if constexpr (KS == 1) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) store(row0 + 8 * i + lane / 4, 8 * j + 2 * (lane & 3), acc[i][j][0], acc[i][j][1]);
  } else {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        red[warp][8 * i + lane / 4][8 * j + 2 * (lane & 3)] = acc[i][j][0];
        red[warp][8 * i + lane / 4][8 * j + 2 * (lane & 3) + 1] = acc[i][j][1];
      }
    __syncthreads();
    for (int i = threadIdx.x; i < 16 * 16; i += KS * 32) {
      const int row = i / 16, col = i % 16 * 2;
      V v0 = red[0][row][col], v1 = red[0][row][col + 1];
#pragma unroll
      for (int w = 1; w < KS; ++w) v0 = sp_add(v0, red[w][row][col]), v1 = sp_add(v1, red[w][row][col + 1]);
      store(row0 + row, col, v0, v1);
    }
  }
}

// A top's map to make: the substitutions with its triangles applied to the identity, in the factor's full
// precision. The upper triangle's rows (pointers, entries and
// diagonals) run from the last to the first, as they are solved. `scratch` holds [column chunk][row][32].
template <class M> struct SpreadMap {
  int32_t t, chunks;  // chunks of 32 columns
  const int32_t *l_ptr, *l_col;
  const M *l_val, *l_dinv;
  const int32_t *u_ptr, *u_col;
  const M *u_val, *u_dinv;
  M *scratch, *m;
  unsigned long long *norm;
};

// One warp makes 32 columns of map blockIdx.y; the maps of all of a batch's networks in one launch. A
// chain of rows, each of a few entries: what bounds it is the latency from one row's solution to the
// next row's loads of it, so the entries come 32 at a time through registers into shared memory, one
// chunk ahead, and the rows' bounds and diagonals one row ahead.
template <class M> __global__ void __launch_bounds__(32) spread_map_kernel(const SpreadMap<M> *__restrict__ maps) {
  const SpreadMap<M> map = maps[blockIdx.y];
  if ((int)blockIdx.x >= map.chunks) return;
  __shared__ M sv[32];
  __shared__ int32_t sc[32];
  const int t = map.t, lane = threadIdx.x, e = blockIdx.x * 32 + lane;
  M *z = map.scratch + (size_t)blockIdx.x * t * 32 + lane;
  M *m = map.m;
  auto out = [&](int p, M x) {
    if (e < t) m[((size_t)(p / kSpreadTopRows) * t + e) * kSpreadTopRows + p % kSpreadTopRows] = x;
  };
  // Row i of the arrays is row i of the map, or (upper triangle) row t - 1 - i.
  auto sweep = [&](auto upper, const int32_t *__restrict__ ptr, const int32_t *__restrict__ col,
                   const M *__restrict__ val, const M *__restrict__ dinv) {
    const int total = __ldg(ptr + t);
    M v_next(0);
    int c_next = 0;
    auto fetch = [&](int k) {
      if (k < total) v_next = val[k], c_next = __ldg(col + k);
    };
    fetch(lane);
    int k = 0, end = __ldg(ptr + 1);
    M d = dinv[0];
    for (int i = 0; i < t; ++i) {
      const int p = upper ? t - 1 - i : i, end_now = end;
      const M d_now = d;
      if (i + 1 < t) end = __ldg(ptr + i + 2), d = dinv[i + 1];
      M s = upper ? z[(size_t)p * 32] : M(p == e ? 1 : 0);
      while (k < end_now) {
        if (k % 32 == 0) {
          __syncwarp();
          sv[lane] = v_next, sc[lane] = c_next;
          __syncwarp();
          fetch(k + 32 + lane);
        }
        const int run = min(end_now, (k / 32 + 1) * 32) - k, at = k % 32;
        int q = 0;
        for (; q + 4 <= run; q += 4) {
          M x[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = z[(size_t)sc[at + q + j] * 32];
#pragma unroll
          for (int j = 0; j < 4; ++j) s = sp_fnma(sv[at + q + j], x[j], s);
        }
        for (; q < run; ++q) s = sp_fnma(sv[at + q], z[(size_t)sc[at + q] * 32], s);
        k += run;
      }
      s = s * d_now;
      z[(size_t)p * 32] = s;
      if (upper) out(p, s);
    }
  };
  sweep(std::false_type(), map.l_ptr, map.l_col, map.l_val, map.l_dinv);
  sweep(std::true_type(), map.u_ptr, map.u_col, map.u_val, map.u_dinv);
}

__device__ __forceinline__ double spread_abs(double v) { return fabs(v); }
__device__ __forceinline__ double spread_abs(const cplx<double> &v) { return hypot(v.re, v.im); }

// A triangle by rows into a dense array of the maps' layout, which is zero elsewhere; a thread a row.
template <class M>
__global__ void spread_dense_kernel(int t, const int32_t *__restrict__ ptr, const int32_t *__restrict__ col, const M *__restrict__ val, M *m) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= t) return;
  for (int q = ptr[i]; q < ptr[i + 1]; ++q) m[((size_t)(i / kSpreadTopRows) * t + col[q]) * kSpreadTopRows + i % kSpreadTopRows] = val[q];
}

// ||M||inf as a bit pattern (positive doubles order as theirs; a NaN lies above them all).
template <class M> __global__ void spread_norm_kernel(const SpreadMap<M> *__restrict__ maps) {
  const SpreadMap<M> map = maps[blockIdx.y];
  const int t = map.t;
  const M *m = map.m;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= t) return;
  double s = 0;
  for (int k = 0; k < t; ++k) s += spread_abs(m[((size_t)(i / kSpreadTopRows) * t + k) * kSpreadTopRows + i % kSpreadTopRows]);
  atomicMax(map.norm, (unsigned long long)__double_as_longlong(fabs(s)));
}

// A lane's row of the work array in 32-byte pieces: COLS columns from column c, as reals.
template <class T> struct SpreadPiece;
template <> struct SpreadPiece<double> {
  static constexpr int COLS = 4;
  static __device__ __forceinline__ void store(double *p, const double *v) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3]) : "memory");
  }
  static __device__ __forceinline__ void load(const double *p, double *v) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
  }
};
template <> struct SpreadPiece<float> {
  static constexpr int COLS = 8;
  static __device__ __forceinline__ void store(float *p, const double *v) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"((float)v[0]), "f"((float)v[1]),
                 "f"((float)v[2]), "f"((float)v[3]), "f"((float)v[4]), "f"((float)v[5]), "f"((float)v[6]), "f"((float)v[7])
                 : "memory");
  }
  static __device__ __forceinline__ void load(const float *p, double *v) {
    float f[8];
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7])
                 : "l"(p));
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = f[k];
  }
};

// The block's network and the warp's 32 natural rows and group, for the gather and the scatter.
template <bool BATCH> __device__ __forceinline__ const SpreadNet &spread_io(const SpreadArgs &a, int64_t &g, int &row) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if constexpr (BATCH) {
    const SpreadItem it = a.items[blockIdx.x];
    g = it.b, row = (it.a * kSpreadIoWarps + warp) * 32 + lane;
    return a.nets[it.net];
  } else {
    const int64_t chunks = (a.one.n + 31) / 32, w = (int64_t)blockIdx.x * kSpreadIoWarps + warp;
    g = w / chunks, row = (int)(w % chunks) * 32 + lane;
    if (g >= a.one.groups) row = a.one.n;
    return a.one;
  }
}

// b (natural rows, column-major) into the work array, columns past the count as zero: each lane takes
// one row, reads its columns with one coalesced access of the warp each, and writes its row of the
// work array in 32-byte pieces. No shared memory, no barrier; HBM bandwidth bounds it.
template <class L, bool BATCH>
__global__ void __launch_bounds__(kSpreadIoWarps * 32) spread_in_kernel(const __grid_constant__ SpreadArgs a) {
  constexpr bool C = SpreadLane<L>::kComplex;
  constexpr int R = sizeof(L) / sizeof(typename SpreadLane<L>::S) * (C ? 2 : 1);  // reals per lane
  using Real = std::conditional_t<(sizeof(L) / R == 8), double, float>;
  constexpr int ALL = 32 * SpreadLane<L>::N, ONCE = C ? 16 : 32, COLS = SpreadPiece<Real>::COLS;  // columns
  int64_t g;
  int i;
  const SpreadNet &net = spread_io<BATCH>(a, g, i);
  sp_ready();
  if (i >= net.n || (net.group_active && !net.group_active[g])) return;
  Real *row = static_cast<Real *>(net.work) + ((size_t)g * net.n + __ldg(net.in_pos + i)) * 32 * R;
#pragma unroll 1
  for (int c0 = 0; c0 < ALL; c0 += ONCE) {
    double v[32];
#pragma unroll
    for (int c = 0; c < ONCE; ++c) {
      const int64_t col = g * ALL + c0 + c;
      if constexpr (C) {
        const double2 b = col < net.count ? __ldcs(static_cast<const double2 *>(net.b) + col * net.ldb + i) : make_double2(0, 0);
        v[2 * c] = b.x, v[2 * c + 1] = b.y;
      } else {
        v[c] = col < net.count ? __ldcs(static_cast<const double *>(net.b) + col * net.ldb + i) : 0.0;
      }
    }
#pragma unroll
    for (int k = 0; k < 32; k += COLS) SpreadPiece<Real>::store(row + c0 * (C ? 2 : 1) + k, v + k);
  }
}

// The solutions into x (natural rows, column-major), or added to it (ADD): the gather's mirror, the
// top's rows from their own place.
template <class L, bool BATCH, bool ADD>
__global__ void __launch_bounds__(kSpreadIoWarps * 32) spread_out_kernel(const __grid_constant__ SpreadArgs a) {
  constexpr bool C = SpreadLane<L>::kComplex;
  constexpr int R = sizeof(L) / sizeof(typename SpreadLane<L>::S) * (C ? 2 : 1);
  using Real = std::conditional_t<(sizeof(L) / R == 8), double, float>;
  constexpr int ALL = 32 * SpreadLane<L>::N, ONCE = C ? 16 : 32, COLS = SpreadPiece<Real>::COLS;
  int64_t g;
  int i;
  const SpreadNet &net = spread_io<BATCH>(a, g, i);
  sp_ready();
  if (i >= net.n) return;
  const int pos = __ldg(net.out_pos + i), top0 = net.n - net.top;
  const Real *row = pos < top0 ? static_cast<const Real *>(net.xout) + ((size_t)g * net.n + pos) * 32 * R
                               : static_cast<const Real *>(net.partial) + (spread_top_row(net, g) + (size_t)(pos - top0) * 32) * R;
#pragma unroll 1
  for (int c0 = 0; c0 < ALL; c0 += ONCE) {
    double v[32];
#pragma unroll
    for (int k = 0; k < 32; k += COLS) SpreadPiece<Real>::load(row + c0 * (C ? 2 : 1) + k, v + k);
#pragma unroll
    for (int c = 0; c < ONCE; ++c) {
      const int64_t col = g * ALL + c0 + c;
      if (col >= net.count) break;
      if constexpr (C) {
        double2 *x = static_cast<double2 *>(net.x) + col * net.ldx + i;
        double2 s = make_double2(v[2 * c], v[2 * c + 1]);
        if (ADD) {
          const double2 was = *x;
          s.x = was.x + s.x, s.y = was.y + s.y;
        }
        __stcs(x, s);
      } else {
        double *x = static_cast<double *>(net.x) + col * net.ldx + i;
        __stcs(x, ADD ? *x + v[c] : v[c]);
      }
    }
  }
}

}  // namespace yb
