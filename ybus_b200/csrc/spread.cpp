// The spread solve's layout (spread_solve.cuh, SpreadLayout in plan.hpp): the rows in a postorder of
// the elimination forest, a cut into subtree domains under a dense top, the domains bundled into
// tasks, and each task's two sweeps as packets.
//
// Forest: Liu's algorithm over the entries of the forward triangle and of the backward one
// transposed, so every entry's larger index is an ancestor of its smaller and one postorder serves
// both sweeps, for Cholesky and for pivoted LU factors.
//
// Cut: the subtrees whose work is at most a cap are the domains; the rows above them are the top.
// A warp takes a task (a bundle of domains) for 32 right-hand sides with no one to wait for, so more
// and smaller tasks shorten the chains and fill the GPU when there are few right-hand sides, and
// cost a larger top, whose dense map grows with its square. The cap is the one whose estimate is
// least (cost_of below).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <complex>
#include <cstring>
#include <exception>
#include <functional>
#include <mutex>
#include <numeric>
#include <system_error>
#include <thread>
#include <vector>

#include "plan.hpp"

namespace yb {

namespace {

// Live values' slots: the lowest free one.
struct SpreadSlots {
  std::vector<uint8_t> used;
  int32_t peak = 0;
  int32_t take() {
    const auto it = std::find(used.begin(), used.end(), 0);
    const int32_t s = (int32_t)(it - used.begin());
    if (it == used.end()) used.push_back(0);
    if (s >= kSpreadMostSlots) throw host::Error(host::kTooLarge, "the spread solve would keep too many live values");
    used[s] = 1;
    peak = std::max(peak, s + 1);
    return s;
  }
  void give(int32_t s) { used[s] = 0; }
};

template <class V> struct Packed;
template <> struct Packed<double> {
  static void put(uint8_t *p, double v, bool full) {
    if (full) {
      std::memcpy(p, &v, 8);
    } else {
      const float f = (float)v;
      std::memcpy(p, &f, 4);
    }
  }
};
template <> struct Packed<std::complex<double>> {
  static void put(uint8_t *p, const std::complex<double> &v, bool full) {
    if (full) {
      const double d[2] = {v.real(), v.imag()};
      std::memcpy(p, d, 16);
    } else {
      const float f[2] = {(float)v.real(), (float)v.imag()};
      std::memcpy(p, f, 8);
    }
  }
};

template <class V> struct Entry {
  V val;
  uint8_t slot;
  bool load, store, carry;
};

// Writes one sweep of one task into pages: packets never straddle a page, every page ends with a
// kSpreadPageEnd, the stream with a kSpreadEnd. Moves wait for the packet of rows that is being
// filled: forward they follow the rows added before them, backward they precede those after.
template <class V> struct PacketWriter {
  struct Row {
    V dinv;
    int32_t self;  // the row's own slot, -1: none
    std::vector<Entry<V>> entries;
  };
  using Moves = std::vector<std::pair<uint32_t, uint32_t>>;  // {index, slot}
  std::vector<uint8_t> &blob;
  const bool full, backward;
  const uint32_t vb, rb, pb;
  int32_t pages = 0;
  size_t pos = 0;
  Row held[4];  // rows waiting to make a packet of four; their storage is used again
  int n_held = 0;
  Moves waiting;          // forward: moves that follow the held rows
  PacketWriter(std::vector<uint8_t> &b, int32_t value_bytes, bool back)
      : blob(b), full(value_bytes == (int32_t)sizeof(V)), backward(back), vb((uint32_t)value_bytes),
        rb(spread_row_bytes(value_bytes)), pb(spread_pair_bytes(value_bytes)) {
    open();
  }
  void open() {
    blob.resize(blob.size() + kSpreadPage, 0);
    pos = 0;
    ++pages;
  }
  uint8_t *at() { return blob.data() + blob.size() - kSpreadPage + pos; }
  // Starts a packet of `bytes` in all (a new page when it does not fit before a page's end packet).
  uint8_t *packet(uint32_t kind, uint32_t bytes, uint32_t count) {
    if (bytes + 16 > (uint32_t)kSpreadPage) throw host::Error(host::kInternal, "a packet larger than a page");
    if (pos + bytes + 16 > (size_t)kSpreadPage) {
      const uint32_t end[4] = {kSpreadPageEnd, 16, 0, 0};
      std::memcpy(at(), end, 16);
      open();
    }
    uint8_t *p = at();
    const uint32_t head[4] = {kind, bytes, count, 0};
    std::memcpy(p, head, 16);
    pos += bytes;
    return p;
  }
  static uint32_t pairs_of(size_t entries) { return entries <= 2 ? 0u : (uint32_t)((entries - 1) / 2); }
  uint32_t row_bytes(const Row &r) const { return rb + pb * pairs_of(r.entries.size()); }
  uint32_t most_pairs() const { return std::min<uint32_t>(255, ((uint32_t)kSpreadPage - 32 - rb) / pb); }
  uint32_t pair_flags(const Entry<V> &a, const Entry<V> *b) const {
    uint32_t f = (a.load ? kSpreadLoad0 : 0u) | (a.store ? kSpreadStore0 : 0u) | (a.carry ? kSpreadCarry : 0u);
    if (b) f |= (b->load ? kSpreadLoad1 : 0u) | (b->store ? kSpreadStore1 : 0u);
    return f;
  }
  void pair(uint8_t *p, const Entry<V> &a, const Entry<V> *b) {
    Packed<V>::put(p, a.val, full);
    if (b) Packed<V>::put(p + vb, b->val, full);
    const uint32_t w = a.slot | (b ? (uint32_t)b->slot << 8 : 0u) | pair_flags(a, b) << 16;
    std::memcpy(p + 2 * vb, &w, 4);
  }
  void rows(const Row *r, int count) {
    uint32_t bytes = 16;
    for (int k = 0; k < count; ++k) bytes += row_bytes(r[k]);
    uint8_t *p = packet(count == 4 ? kSpreadRows4 : kSpreadRows1, bytes, (uint32_t)count) + 16;
    uint8_t *more = p + (size_t)count * rb;
    for (int k = 0; k < count; ++k, p += rb) {
      const auto &e = r[k].entries;
      const uint32_t pairs = pairs_of(e.size());
      uint32_t slots = r[k].self >= 0 ? (uint32_t)r[k].self : 0u, flags = r[k].self >= 0 ? (uint32_t)kSpreadSelf : 0u;
      if (!e.empty()) {
        const Entry<V> *second = e.size() > 1 ? &e[1] : nullptr;
        Packed<V>::put(p, e[0].val, full);
        if (second) Packed<V>::put(p + vb, second->val, full);
        slots |= (uint32_t)e[0].slot << 8 | (second ? (uint32_t)second->slot << 16 : 0u);
        flags |= pair_flags(e[0], second);
      }
      Packed<V>::put(p + 2 * vb, r[k].dinv, full);
      const uint32_t w[2] = {slots, flags | pairs << 8};
      std::memcpy(p + 3 * vb, w, 8);
      for (uint32_t i = 0; i < pairs; ++i, more += pb) pair(more, e[2 + 2 * i], 3 + 2 * i < e.size() ? &e[3 + 2 * i] : nullptr);
    }
  }
  void more(const Entry<V> *e, size_t count) {  // `count` entries of a long row, a packet's worth
    const uint32_t pairs = (uint32_t)((count + 1) / 2);
    uint8_t *p = packet(kSpreadMore, 16 + pb * pairs, pairs) + 16;
    for (uint32_t i = 0; i < pairs; ++i, p += pb) pair(p, e[2 * i], 2 * i + 1 < count ? e + 2 * i + 1 : nullptr);
  }
  void flush_rows() {  // held rows that make no packet of four: one by one
    for (int k = 0; k < n_held; ++k) rows(&held[k], 1);
    n_held = 0;
    put_moves(waiting);
    waiting.clear();
  }
  void row(Row &r) {  // r's storage is taken, another's left
    const size_t most = 2 + 2 * (size_t)most_pairs();
    if (r.entries.size() > most) {  // a row longer than a packet: in runs of pairs (forward after it, backward before)
      flush_rows();
      std::vector<Entry<V>> rest(r.entries.begin() + (long)most, r.entries.end());
      r.entries.resize(most);
      const size_t run = 2 * (size_t)(((uint32_t)kSpreadPage - 32) / pb);
      auto runs = [&] {
        for (size_t i = 0; i < rest.size(); i += run) more(rest.data() + i, std::min(run, rest.size() - i));
      };
      if (backward) runs();
      rows(&r, 1);
      if (!backward) runs();
      return;
    }
    std::swap(held[n_held++], r);
    if (n_held == 4) {
      uint32_t bytes = 16;
      for (const Row &h : held) bytes += row_bytes(h);
      if (bytes + 16 <= (uint32_t)kSpreadPage) {
        rows(held, 4);
        n_held = 0;
      }
      flush_rows();
    }
  }
  // Forward: after the rows so far; backward: before the rows to come (and so, when rows are held,
  // before their packet: the moved slots are free until then).
  void moves(const Moves &m) {
    if (backward || n_held == 0)
      put_moves(m);
    else
      waiting.insert(waiting.end(), m.begin(), m.end());
  }
  void put_moves(const Moves &m) {
    const size_t run = ((size_t)kSpreadPage - 48) / 8;
    for (size_t i = 0; i < m.size(); i += run) {
      const size_t k = std::min(run, m.size() - i);
      uint8_t *p = packet(kSpreadMove, (uint32_t)((16 + 8 * k + 15) & ~(size_t)15), (uint32_t)k) + 16;
      for (size_t j = 0; j < k; ++j, p += 8) {
        const uint32_t w[2] = {m[i + j].first, m[i + j].second};
        std::memcpy(p, w, 8);
      }
    }
  }
  void end() {
    flush_rows();
    packet(kSpreadEnd, 16, 0);
  }
};

template <class V> double magnitude_of(const V &v) { return std::abs(v); }

// Runs `work` on this thread and `most` - 1 others, or on as many as there are.
template <class F> void on_threads(int32_t most, const F &work) {
  std::vector<std::thread> threads;
  try {
    for (int32_t i = 1; i < std::min<int32_t>(most, (int32_t)std::thread::hardware_concurrency()); ++i) threads.emplace_back(work);
  } catch (const std::system_error &) {  // no more threads: those there are do
  }
  work();
  for (auto &t : threads) t.join();
}

}  // namespace

template <class V>
SpreadLayout<V> spread_layout(const Plan<V> &plan, int32_t value_bytes, int64_t groups, int32_t sms, int32_t blocks,
                              const std::function<int32_t(int32_t)> &fit) {
  if (value_bytes != (int32_t)sizeof(V) && value_bytes * 2 != (int32_t)sizeof(V))
    throw host::Error(host::kInvalidArgument, "packet values are the plan's, or half as wide");
  const int32_t n = plan.n;
  // each row's entries in both sweeps
  std::vector<int32_t> fat(n), bat(n);  // the row's index in each sweep's order
  for (int32_t p = 0; p < n; ++p) fat[plan.fwd.row[p]] = p, bat[plan.bwd.row[p]] = p;
  auto f0 = [&](int32_t r) { return plan.fwd.ptr[fat[r]]; };
  auto f1 = [&](int32_t r) { return plan.fwd.ptr[fat[r] + 1]; };
  auto b0 = [&](int32_t r) { return plan.bwd.ptr[bat[r]]; };
  auto b1 = [&](int32_t r) { return plan.bwd.ptr[bat[r] + 1]; };
  // the elimination forest
  std::vector<int32_t> below_ptr(n + 1, 0), below;
  for (int32_t r = 0; r < n; ++r)
    for (int32_t q = b0(r); q < b1(r); ++q) {
      if (plan.bwd.col[q] <= r) throw host::Error(host::kInvalidArgument, "the backward sweep is not upper triangular");
      ++below_ptr[plan.bwd.col[q] + 1];
    }
  for (int32_t c = 0; c < n; ++c) below_ptr[c + 1] += below_ptr[c];
  below.resize(below_ptr[n]);
  {
    std::vector<int32_t> fill(below_ptr.begin(), below_ptr.end() - 1);
    for (int32_t r = 0; r < n; ++r)
      for (int32_t q = b0(r); q < b1(r); ++q) below[fill[plan.bwd.col[q]]++] = r;
  }
  std::vector<int32_t> parent(n, -1), ancestor(n, -1);
  for (int32_t i = 0; i < n; ++i) {
    auto join = [&](int32_t k) {
      while (ancestor[k] >= 0 && ancestor[k] != i) {
        const int32_t up = ancestor[k];
        ancestor[k] = i;
        k = up;
      }
      if (ancestor[k] < 0) ancestor[k] = i, parent[k] = i;
    };
    for (int32_t q = f0(i); q < f1(i); ++q) {
      if (plan.fwd.col[q] >= i) throw host::Error(host::kInvalidArgument, "the forward sweep is not lower triangular");
      join(plan.fwd.col[q]);
    }
    for (int32_t q = below_ptr[i]; q < below_ptr[i + 1]; ++q) join(below[q]);
  }
  // postorder, larger subtrees first (fewer live values)
  std::vector<int32_t> size(n, 1);
  for (int32_t c = 0; c < n; ++c)
    if (parent[c] >= 0) size[parent[c]] += size[c];
  std::vector<int32_t> child_ptr(n + 2, 0), child(n), order;
  for (int32_t c = 0; c < n; ++c) ++child_ptr[(parent[c] < 0 ? n : parent[c]) + 1];
  for (int32_t i = 0; i <= n; ++i) child_ptr[i + 1] += child_ptr[i];
  {
    std::vector<int32_t> fill(child_ptr.begin(), child_ptr.end() - 1);
    for (int32_t c = 0; c < n; ++c) child[fill[parent[c] < 0 ? n : parent[c]]++] = c;
  }
  for (int32_t v = 0; v <= n; ++v)
    if (child_ptr[v + 1] - child_ptr[v] > 1)
      std::sort(child.begin() + child_ptr[v], child.begin() + child_ptr[v + 1],
                [&](int32_t a, int32_t b) { return size[a] != size[b] ? size[a] > size[b] : a < b; });
  order.reserve(n);
  {
    std::vector<std::pair<int32_t, int32_t>> stack{{n, child_ptr[n]}};
    while (!stack.empty()) {
      auto &top = stack.back();
      const int32_t v = top.first;
      if (top.second < child_ptr[v + 1]) {
        const int32_t c = child[top.second++];
        stack.push_back({c, child_ptr[c]});
      } else {
        if (v < n) order.push_back(v);
        stack.pop_back();
      }
    }
  }
  std::vector<int32_t> pos(n);
  for (int32_t t = 0; t < n; ++t) pos[order[t]] = t;
  // forward columns: the rows each row updates
  std::vector<int32_t> col_ptr(n + 1, 0), col_row;
  std::vector<V> col_val;
  for (int32_t r = 0; r < n; ++r)
    for (int32_t q = f0(r); q < f1(r); ++q) ++col_ptr[plan.fwd.col[q] + 1];
  for (int32_t c = 0; c < n; ++c) col_ptr[c + 1] += col_ptr[c];
  col_row.resize(col_ptr[n]), col_val.resize(col_ptr[n]);
  {
    std::vector<int32_t> fill(col_ptr.begin(), col_ptr.end() - 1);
    for (int32_t r = 0; r < n; ++r)
      for (int32_t q = f0(r); q < f1(r); ++q) {
        const int32_t c = plan.fwd.col[q];
        col_row[fill[c]] = r;
        col_val[fill[c]++] = plan.fwd.val[q];
      }
  }
  // each row's work over both sweeps, in cycles of a scheduler with warps to choose from (measured:
  // about 80 for a row of two entries and sweep, 290 where a warp is alone), and each subtree's; and what
  // a task costs before its first row, both sweeps' blocks (their first page and rows)
  constexpr double kRow = 110, kEntry = 12, kAlone = 3.6, kStart = 900;
  std::vector<double> work(n), sub(n, 0.0);
  for (int32_t v = 0; v < n; ++v)
    work[v] = kRow + kEntry * (std::max(2, col_ptr[v + 1] - col_ptr[v]) + std::max(2, b1(v) - b0(v)));
  for (int32_t t = 0; t < n; ++t) {
    const int32_t v = order[t];
    sub[v] += work[v];
    if (parent[v] >= 0) sub[parent[v]] += sub[v];
  }
  const double total = std::accumulate(work.begin(), work.end(), 0.0);
  struct Cut {
    std::vector<int32_t> roots;
    int32_t top = 0, tasks = 1;
    double longest = 0, cost = 0, cap = 0;
  };
  // The estimate of a cut, in cycles: the sweeps' blocks (a task for four groups, `blocks` an SM) in full
  // waves and one of what is left, each as long as the longest task with that many warps on its
  // scheduler; the top's map: a tile's chain of steps, its values from L2, half the FP64 rate; and, with
  // a top, its launches.
  const double G = (double)std::max<int64_t>(1, groups);
  // A complex top is four products of reals for one, and a real FP64 one is applied twice. That a complex
  // one is too is not charged: with 8 in place of 4 a batch of 16 networks of 730 to 46,293 buses took
  // 1,531 us for 1,001, with 2 1,082, and four other batches were within 3 %.
  const double kTop = sizeof(V) == 16 ? 4 : value_bytes == 8 ? 2 : 1;
  const double kLaunches = value_bytes == (int32_t)sizeof(V) ? 14000 : 8000;  // five more, or two; without rows below the top two fewer
  // and a corrected top's rows: their sums and residual (3,000 buses with 7,000 and 13,499 right-hand sides 310 to 286
  // and 587 to 530 us, 8,000 with 7,000 708 to 691, 10,000 with 1 to 13,499 the same within 2 %; with 150 in place of
  // 80 one 10,000-bus grid's 13,499 took 1,657 us for 1,585)
  const double kRows = value_bytes == (int32_t)sizeof(V) && sizeof(V) == 8 ? 80 : 0;
  auto cost_of = [&](const Cut &c) {
    const double all = c.tasks * std::ceil(G / 4), wave = (double)blocks * sms, full = std::floor(all / wave);
    const double left = std::ceil((all - full * wave) / sms);
    const double sweeps = (c.longest + kStart) * (full * std::max<double>(kAlone, blocks) + (left > 0 ? std::max(kAlone, left) : 0.0));
    const double t = c.top;
    return sweeps + (c.top ? 20 * t + t * t / 100 + kTop * G * t * t / sms + kRows * G * t / sms + kLaunches - (c.top == n ? 6000 : 0) : 0);
  };
  constexpr int kCaps = 45;  // caps a quarter octave apart
  auto cap_of = [&](int k) { return total / std::pow(2.0, 1 + k / 4.0); };
  std::vector<int32_t> near;  // the rows that some cap has at its top or roots a domain at
  for (int32_t v = 0; v < n; ++v)
    if (parent[v] < 0 || sub[parent[v]] > cap_of(kCaps - 1)) near.push_back(v);
  auto cut_at = [&](double cap) {
    Cut c;
    c.cap = cap;
    double domain_work = 0, largest = 0;
    for (int32_t v : near) {
      if (sub[v] > cap)
        ++c.top;
      else if (parent[v] < 0 || sub[parent[v]] > cap)
        c.roots.push_back(v), domain_work += sub[v], largest = std::max(largest, sub[v]);
    }
    // as many tasks as keep the longest near the largest domain, no more than domains; or a half, a quarter
    // and so on of them where starting so many costs more
    int32_t tasks = 1;
    if (!c.roots.empty())
      tasks = (int32_t)std::max<double>(1, std::min<double>((double)c.roots.size(), std::ceil(domain_work / std::max(largest, 1.0))));
    c.cost = INFINITY;
    for (; tasks >= 1 && c.top <= kSpreadMostTop; tasks /= 2) {
      Cut t;
      t.top = c.top, t.tasks = tasks, t.longest = std::max(largest, domain_work / tasks);
      t.cost = cost_of(t);
      if (t.cost < c.cost) c.tasks = t.tasks, c.longest = t.longest, c.cost = t.cost;
    }
    return c;
  };
  auto choose = [&] {
    Cut best = cut_at(total + 1);  // one domain per tree, no top
    for (int k = 0; k < kCaps; ++k) {
      Cut c = cut_at(cap_of(k));
      if (c.cost < best.cost) best = std::move(c);
    }
    return best;
  };
  auto lay_out = [&](const Cut &best) {
    SpreadLayout<V> lay;
    lay.n = n;
    lay.cost = best.cost;
    lay.domains = (int32_t)best.roots.size();
    lay.tasks = best.tasks;
    // LPT: the domains to the tasks by work, each task's domains in postorder, the longest task first
    std::vector<std::vector<int32_t>> task_domains(lay.tasks);
    {
      std::vector<int32_t> by_work(best.roots);
      std::stable_sort(by_work.begin(), by_work.end(), [&](int32_t a, int32_t b) { return sub[a] > sub[b]; });
      std::vector<double> load(lay.tasks, 0.0);
      for (int32_t r : by_work) {
        const size_t w = (size_t)(std::min_element(load.begin(), load.end()) - load.begin());
        load[w] += sub[r];
        task_domains[w].push_back(r);
      }
      std::vector<size_t> by_load(lay.tasks);
      std::iota(by_load.begin(), by_load.end(), 0);
      std::stable_sort(by_load.begin(), by_load.end(), [&](size_t a, size_t b) { return load[a] > load[b]; });
      std::vector<std::vector<int32_t>> sorted;
      for (size_t w : by_load) sorted.push_back(std::move(task_domains[w]));
      task_domains = std::move(sorted);
      for (auto &d : task_domains) std::sort(d.begin(), d.end(), [&](int32_t a, int32_t b) { return pos[a] < pos[b]; });
    }
    // positions: task by task, each domain in postorder, then the top in postorder
    std::vector<int32_t> newpos(n, -1), at(n), domain_of(n, -1);
    std::vector<std::vector<std::pair<int32_t, int32_t>>> ranges(lay.tasks);  // each domain's positions, first and last
    int32_t next = 0, domain_count = 0;
    for (int32_t w = 0; w < lay.tasks; ++w) {
      lay.task_row.push_back(next);
      for (int32_t r : task_domains[w]) {
        const int32_t d0 = next;
        for (int32_t t = pos[r] - size[r] + 1; t <= pos[r]; ++t) newpos[order[t]] = next++, domain_of[order[t]] = domain_count;
        ranges[w].push_back({d0, next - 1});
        ++domain_count;
      }
    }
    lay.task_row.push_back(next);
    const int32_t top0 = next;
    for (int32_t t = 0; t < n; ++t)
      if (newpos[order[t]] < 0) newpos[order[t]] = next++;
    lay.top = n - top0;
    for (int32_t v = 0; v < n; ++v) at[newpos[v]] = v;
    // the top rows each domain updates, and those it reads, by position; the partial rows: one per
    // (domain, top row it updates), each top row's together, by domain
    std::vector<std::vector<int32_t>> updates(domain_count), reads(domain_count);
    for (int32_t p = 0; p < top0; ++p) {
      const int32_t d = domain_of[at[p]];
      for (int32_t q = col_ptr[at[p]]; q < col_ptr[at[p] + 1]; ++q)
        if (newpos[col_row[q]] >= top0) updates[d].push_back(newpos[col_row[q]]);
      for (int32_t q = b0(at[p]); q < b1(at[p]); ++q)
        if (newpos[plan.bwd.col[q]] >= top0) reads[d].push_back(newpos[plan.bwd.col[q]]);
    }
    std::vector<int32_t> part_next(lay.top + 1, 0);
    for (auto *sets : {&updates, &reads})
      for (auto &v : *sets) {
        std::sort(v.begin(), v.end());
        v.erase(std::unique(v.begin(), v.end()), v.end());
      }
    for (const auto &v : updates)
      for (int32_t p : v) ++part_next[p - top0 + 1];
    for (int32_t i = 0; i < lay.top; ++i) part_next[i + 1] += part_next[i];
    lay.part_ptr = part_next;
    lay.partials = part_next[lay.top];
    // the packets. A domain's last row leaves nothing to the next domain's first (their trees differ),
    // and the slots a domain's moves use are given back only after the packet they may wait for.
    // Tasks share nothing here, so threads write them, each with its own marks.
    std::vector<int32_t> task_domain(lay.tasks + 1, 0);  // each task's first domain
    for (int32_t w = 0; w < lay.tasks; ++w) task_domain[w + 1] = task_domain[w] + (int32_t)ranges[w].size();
    std::vector<std::vector<uint32_t>> part_of(domain_count);  // the partial rows of each domain's updates
    for (int32_t d = 0; d < domain_count; ++d)
      for (int32_t p : updates[d]) part_of[d].push_back((uint32_t)part_next[p - top0]++);
    lay.fwd_page.resize(2 * (size_t)lay.tasks), lay.bwd_page.resize(2 * (size_t)lay.tasks);
    std::vector<std::vector<uint8_t>> blobs(lay.tasks);
    std::exception_ptr error;
    std::mutex error_mutex;
    std::atomic<int32_t> next_task{0}, peak{0};
    auto write_task = [&](int32_t w, std::vector<int32_t> &slot, std::vector<int32_t> &readers) {
      std::vector<uint8_t> &blob = blobs[w];
      std::vector<std::pair<uint32_t, uint32_t>> moves;
      typename PacketWriter<V>::Row row;
      const int32_t first_domain = task_domain[w];
      int32_t d = first_domain;
      auto note = [&](int32_t slots) {
        for (int32_t was = peak; was < slots && !peak.compare_exchange_weak(was, slots);) {}
      };
      {
        PacketWriter<V> pw(blob, value_bytes, false);
        SpreadSlots slots;
        std::vector<int32_t> late;  // slots whose moves wait for the held rows
        auto settle = [&] {
          if (pw.n_held > 0) return;
          for (int32_t s : late) slots.give(s);
          late.clear();
        };
        for (auto [d0, d1] : ranges[w]) {
          for (int32_t p = d0; p <= d1; ++p) {
            const int32_t j = at[p], after = p < d1 ? at[p + 1] : -1;
            row.dinv = plan.fwd.dinv[fat[j]], row.self = -1, row.entries.clear();
            // the targets' slots before the row's own is given back: the kernel reads them together
            int32_t given = -1;
            for (int32_t q = col_ptr[j]; q < col_ptr[j + 1]; ++q) {
              const int32_t r = col_row[q];
              const bool load = slot[r] >= 0;
              if (r == after) {  // to the next row, which alone reads it
                const uint8_t was = load ? (uint8_t)slot[r] : 0;
                if (load) given = slot[r], slot[r] = -1;
                row.entries.insert(row.entries.begin(), {col_val[q], was, load, false, true});
              } else {
                if (!load) slot[r] = slots.take();
                row.entries.push_back({col_val[q], (uint8_t)slot[r], load, true, false});
              }
            }
            if (slot[j] >= 0) row.self = slot[j], slots.give(slot[j]), slot[j] = -1;
            if (given >= 0) slots.give(given);
            pw.row(row);
            settle();
          }
          moves.clear();
          for (size_t i = 0; i < updates[d].size(); ++i) {
            const int32_t r = at[updates[d][i]];
            moves.push_back({part_of[d][i], (uint32_t)slot[r]});
            late.push_back(slot[r]);
            slot[r] = -1;
          }
          pw.moves(moves);
          settle();
          ++d;
        }
        pw.end();
        lay.fwd_page[2 * w + 1] = pw.pages;
        note(slots.peak);
      }
      lay.bwd_page[2 * w] = (int32_t)(blob.size() / kSpreadPage);
      {
        PacketWriter<V> pw(blob, value_bytes, true);
        SpreadSlots slots;
        std::vector<int32_t> late;  // slots given up while rows are held: a move may run before them
        auto settle = [&] {
          if (pw.n_held > 0) return;
          for (int32_t s : late) slots.give(s);
          late.clear();
        };
        for (size_t i = ranges[w].size(); i-- > 0;) {
          const auto [p0, p1] = ranges[w][i];
          const int32_t dom = first_domain + (int32_t)i;
          for (int32_t p = p0; p <= p1; ++p)
            for (int32_t q = b0(at[p]); q < b1(at[p]); ++q) ++readers[plan.bwd.col[q]];
          moves.clear();
          for (int32_t p : reads[dom]) {
            slot[at[p]] = slots.take();
            moves.push_back({(uint32_t)(p - top0), (uint32_t)slot[at[p]]});
          }
          pw.moves(moves);
          for (int32_t p = p1; p >= p0; --p) {
            const int32_t j = at[p], before = p < p1 ? at[p + 1] : -1, after = p > p0 ? at[p - 1] : -1;
            row.dinv = plan.bwd.dinv[bat[j]], row.self = -1, row.entries.clear();
            for (int32_t q = b0(j); q < b1(j); ++q) {
              const int32_t c = plan.bwd.col[q];
              if (c == before) {  // the row just solved: its x is still in a register (readers does not count this)
                row.entries.insert(row.entries.begin(), {plan.bwd.val[q], 0, false, false, true});
                continue;
              }
              row.entries.push_back({plan.bwd.val[q], (uint8_t)slot[c], true, false, false});
            }
            for (int32_t q = b0(j); q < b1(j); ++q) {
              const int32_t c = plan.bwd.col[q];
              if (c != before && --readers[c] == 0) {
                // in the last rows of a domain a slot may be taken next by the moves of another
                if (newpos[c] >= top0 || p - p0 < 4) late.push_back(slot[c]);
                else slots.give(slot[c]);
                slot[c] = -1;
              }
            }
            if (after >= 0)
              for (int32_t q = b0(after); q < b1(after); ++q)
                if (plan.bwd.col[q] == j) --readers[j];
            if (readers[j] > 0) slot[j] = slots.take(), row.self = slot[j];
            pw.row(row);
            settle();
          }
        }
        pw.end();
        lay.bwd_page[2 * w + 1] = pw.pages;
        note(slots.peak);
      }
    };
    auto write_tasks = [&] {
      try {
        std::vector<int32_t> slot(n, -1), readers(n, 0);
        for (int32_t w = next_task++; w < lay.tasks; w = next_task++) write_task(w, slot, readers);
      } catch (...) {
        const std::lock_guard<std::mutex> lock(error_mutex);
        error = std::current_exception();
      }
    };
    // a thread for 4,096 rows, at most eight: 46,293 rows' packets took 28 ms with one
    on_threads(std::min<int32_t>({8, n / 4096, lay.tasks}), write_tasks);
    if (error) std::rethrow_exception(error);
    size_t blob_bytes = 0;
    for (int32_t w = 0; w < lay.tasks; ++w) {
      lay.fwd_page[2 * w] = (int32_t)(blob_bytes / kSpreadPage), lay.bwd_page[2 * w] += lay.fwd_page[2 * w];
      blob_bytes += blobs[w].size();
    }
    lay.blob.reserve(blob_bytes);
    for (const auto &b : blobs) lay.blob.insert(lay.blob.end(), b.begin(), b.end());
    lay.slots = std::max<int32_t>(peak, 1);
    // the top's triangles by rows
    lay.l_ptr.assign(1, 0), lay.u_ptr.assign(1, 0);
    for (int32_t i = 0; i < lay.top; ++i) {
      const int32_t j = at[top0 + i];
      for (int32_t q = f0(j); q < f1(j); ++q)
        if (newpos[plan.fwd.col[q]] >= top0) lay.l_col.push_back(newpos[plan.fwd.col[q]] - top0), lay.l_val.push_back(plan.fwd.val[q]);
      for (int32_t q = b0(j); q < b1(j); ++q) {  // a top row's backward entries are top rows: its ancestors
        if (newpos[plan.bwd.col[q]] < top0) throw host::Error(host::kInternal, "a top row reads a row below the top");
        lay.u_col.push_back(newpos[plan.bwd.col[q]] - top0), lay.u_val.push_back(plan.bwd.val[q]);
      }
      lay.l_ptr.push_back((int32_t)lay.l_col.size()), lay.u_ptr.push_back((int32_t)lay.u_col.size());
      lay.l_dinv.push_back(plan.fwd.dinv[fat[j]]), lay.u_dinv.push_back(plan.bwd.dinv[bat[j]]);
    }
    // || |L_TT| |U_TT| e ||inf bounds the Schur complement's norm
    {
      std::vector<double> u(lay.top);
      for (int32_t i = 0; i < lay.top; ++i) {
        u[i] = 1.0 / magnitude_of(lay.u_dinv[i]);
        for (int32_t q = lay.u_ptr[i]; q < lay.u_ptr[i + 1]; ++q) u[i] += magnitude_of(lay.u_val[q]);
      }
      for (int32_t i = 0; i < lay.top; ++i) {
        double s = u[i] / magnitude_of(lay.l_dinv[i]);
        for (int32_t q = lay.l_ptr[i]; q < lay.l_ptr[i + 1]; ++q) s += magnitude_of(lay.l_val[q]) * u[lay.l_col[q]];
        lay.s_norm = std::max(lay.s_norm, s);
      }
    }
    lay.in_pos.resize(n), lay.out_pos.resize(n);
    for (int32_t i = 0; i < n; ++i) lay.in_pos[i] = newpos[plan.in_slot[i]], lay.out_pos[i] = newpos[plan.out_slot[i]];
    return lay;
  };
  // A cut's live values decide how many blocks an SM holds, which the cut was chosen for: where they let it hold
  // fewer, the cut is chosen again for those, and of those laid out the one that costs least with what it
  // lets an SM hold is taken (the 10,000-bus Jacobian with 4,096 right-hand sides: 512 blocks, for 148 SMs of four,
  // of which its 39 values let them hold three, took 1.60 ms).
  const int32_t most = blocks;
  Cut cut = choose();
  SpreadLayout<V> best;
  best.cost = INFINITY;
  for (int tries = 0; tries < 4; ++tries) {
    SpreadLayout<V> lay = lay_out(cut);
    const int32_t held = fit ? std::min(most, fit(lay.slots)) : most;
    const bool as_chosen = held == blocks;
    blocks = held;
    lay.cost = cost_of(cut);
    if (lay.cost < best.cost) best = std::move(lay);
    if (as_chosen) break;
    Cut again = choose();
    if (again.cap == cut.cap && again.tasks == cut.tasks) break;
    cut = std::move(again);
  }
  return best;
}

template SpreadLayout<double> spread_layout(const Plan<double> &, int32_t, int64_t, int32_t, int32_t, const std::function<int32_t(int32_t)> &);
template SpreadLayout<host::c128> spread_layout(const Plan<host::c128> &, int32_t, int64_t, int32_t, int32_t, const std::function<int32_t(int32_t)> &);

template <class V> void spread_correction(SpreadLayout<V> &lay) {
  lay.low_ptr.assign(1, 0), lay.up_ptr.assign(1, 0);
  for (int32_t i = 0; i < lay.top; ++i) {
    for (int32_t q = lay.l_ptr[i]; q < lay.l_ptr[i + 1]; ++q) lay.low_col.push_back(lay.l_col[q]), lay.low_val.push_back(-lay.l_val[q]);
    lay.low_col.push_back(i), lay.low_val.push_back(-V(1) / lay.l_dinv[i]);
    lay.low_ptr.push_back((int32_t)lay.low_col.size());
    for (int32_t q = lay.u_ptr[i]; q < lay.u_ptr[i + 1]; ++q) lay.up_col.push_back(lay.u_col[q]), lay.up_val.push_back(lay.u_val[q]);
    lay.up_col.push_back(i), lay.up_val.push_back(V(1) / lay.u_dinv[i]);
    lay.up_ptr.push_back((int32_t)lay.up_col.size());
  }
}
template void spread_correction(SpreadLayout<double> &);
template void spread_correction(SpreadLayout<host::c128> &);

}  // namespace yb
