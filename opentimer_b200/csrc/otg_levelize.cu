// otg_levelize.cu -- timing-graph levelization (frontier Kahn) on B200.
//
// Replaces toposort_advance + toposort_compute_cuda (ot/cuda/toposort.cu:4-72)
// which launch one kernel per level and copy the frontier size back to the
// host after each one.  Here:
//   pack    every pin's fanins as one 16-byte record (the whole GPU);
//   levels  one launch for all levels: level 0 is the caller's seed (pins
//           without candidate fanout); expanding a level decrements the
//           fanout counter of each fanin of its pins, and a pin whose
//           counter reaches zero belongs to the next level;
//   sort    the pins by (level, pin index) -- every level after the seed
//           comes out in ascending pin order, deterministically -- and the
//           levels' ends.
// A level is a chain of round trips, so the chain is kept short.  The step
// that decrements a pin's counter loads its record too: a pin that becomes
// ready enters the next level's list, in its CTA's shared memory, with its
// fanins, and that level starts its decrements from there, four lanes an
// entry: no fanin range to look up, no scan and no search to spread edges
// over threads, nothing read back.  Order and level ends are not on the
// chain at all.  A barrier, the counter's atomic and the list append are
// what is left.
//
// Two forms of the levels kernel, with the same outputs:
//   cluster  graphs of up to 650k pins run in ONE thread-block cluster: the
//            counters lie in the CTAs' shared memory, and a level ends at
//            the hardware cluster barrier;
//   grid     larger graphs run on every SM, counters in global memory, one
//            grid barrier per level.  It is a sense-counting barrier whose
//            waits are bounded by %globaltimer: a wait that runs past the
//            limit raises an abort flag that every other wait also watches,
//            so the kernel always returns and the host sees OTG_ERR_TIMEOUT.
// Before, a level's pins were found in ready bitmaps, written out in order,
// and their fanins looked up, scanned and searched by thread, all on the
// chain: 2.53 ms on 5M pins / 200 levels (grid; now 1.5), 1.30 ms on a
// 60k-gate design's 163k pins / 374 levels (cluster; now 0.55).  What bounds
// it now is the chain still: per level one barrier, one counter round trip
// and the appends, 1.4 us in the cluster and 2.6 us on the grid where a
// level has few pins.  32-byte records of eight fanins were 15-20% slower
// (their copies into the lists).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <climits>
#include <cstdlib>

#include "../../include/otg.h"
#include "otg_internal.cuh"

namespace otg {
namespace {

namespace cg = cooperative_groups;
constexpr unsigned FULL = 0xffffffffu;

// A pin's fanins: up to four (-1: none), or {first index in fanin[], their
// number, 0, kWide}.  In the lists a wide pin takes several records: of a quad
// of lanes' worth of fanins, up to kWideLong; beyond (a driver's sinks, where
// the fanouts are levelized) of a warp's worth, or twice that and so on, at
// most kWideRecs.  In one record a warp went through such a pin by itself: a
// pin of 12,000 fanins in a graph of 24,000 pins took 397 us, now 118 (510
// and 91 on the grid), one of 100,000 3.4 ms and 0.77.
constexpr int kWide = -2, kWideMax = 4, kWideLong = 64, kWideRecs = 512, kWideStay = 32;
// log2 of a record's fanins
__device__ __forceinline__ int wide_shift(int deg) {
  return deg <= kWideLong ? 2 : max(5, 32 - __clz((deg - 1) / kWideRecs));
}

struct LvCtl {
  GridCtl grid;
  int levels;    // found by the levels kernel
  int tot[4];    // ready pins' list entries of a level, by level (grid form)
  int spill[4];  // pins in the level's spill list
};

struct LvArgs {
  int n;
  const int* fanin_start;
  const int* fanin;
  const int* out_deg;
  const int* frontier0;
  int first_size;
  int* order;
  int* level;
  int* level_ends;
  int* counts;
  LvCtl* ctl;
  int* cnt;      // fanout counters (unless they lie on chip)
  int4* packed;  // records by pin; behind the levels, the sort's scratch
  int* spill;    // two lists of n pins, by level parity: what no CTA's list held
};

__global__ void levelize_pack(LvArgs a, bool counters) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (i0 == 0) *a.ctl = LvCtl{};
  for (int v = i0; v < a.n; v += gridDim.x * blockDim.x) {
    const int e0 = a.fanin_start[v], deg = a.fanin_start[v + 1] - e0;
    int f[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int u = k < deg && deg <= 4 ? a.fanin[e0 + k] : -1;
      f[k] = (unsigned)u < (unsigned)a.n ? u : -1;
    }
    a.packed[v] = deg > 4 ? make_int4(e0, deg, 0, kWide) : make_int4(f[0], f[1], f[2], f[3]);
    a.level[v] = -1;
    if (counters) a.cnt[v] = a.out_deg[v];
  }
}

// ---- the lists.  A CTA holds two (by level parity) of `cap` records and
// their pins (-1 in a record that continues the one before).
struct LvLists {
  int4* rec0;  // the even levels' records, then the odd ones'
  int* pin0;   // likewise their pins
  int cap;
  __device__ int4* rec(int L) const { return rec0 + (L & 1) * cap; }
  __device__ int* pin(int L) const { return pin0 + (L & 1) * cap; }
};

// Puts pin v's record into list entries [at, at + recs) of a list; entries
// past the capacity are left out.  False if some were.
__device__ __forceinline__ bool put_records(int4* rec, int* pin, int cap, int at, int recs, int v,
                                            int4 pk) {
  const bool fits = at + recs <= cap;
  const int len = recs > 1 ? 1 << wide_shift(pk.y) : 0;
  for (int k = 0; k < recs; ++k) {
    if (at + k >= cap) break;
    int4 x = pk;
    if (recs > 1) x = make_int4(pk.x + len * k, min(len, pk.y - len * k), 0, kWide);
    rec[at + k] = fits ? x : make_int4(-1, -1, -1, -1);
    pin[at + k] = fits && k == 0 ? v : -1;
  }
  return fits;
}

__device__ __forceinline__ void spill_pin(const LvArgs& a, int v, int L) {
  a.spill[(size_t)(L & 1) * a.n + atomicAdd(&a.ctl->spill[L & 3], 1)] = v;
}

// One fanin edge per lane (target v, or none): decrement v's fanout counter;
// a pin whose counter reaches zero is of level L.  Every lane of the warp
// must call it.  A seed pin's counter starts at INT_MAX, so a seed is never
// emitted twice.  (Lanes with the same target do not combine: finding them
// takes match_any 380 cycles when the targets differ, 1100 with every warp
// at it, against 440 for the counter's round trip.)
// The group gives the counter's place, this CTA's list length for L, how
// long that may grow, and takes what it does not hold (hand_on).
template <class Gp>
__device__ __forceinline__ void decrement(const Gp& g, const LvArgs& a, const LvLists& ls, int v,
                                          int L) {
  const int lane = threadIdx.x & 31;
  bool ready = false;
  int4 pk = make_int4(-1, -1, -1, -1);
  if ((unsigned)v < (unsigned)a.n) {
    pk = __ldcg(a.packed + v);
    ready = atomicSub(g.counter(v), 1) == 1;
  }
  const unsigned set = __ballot_sync(FULL, ready);
  if (set == 0u) return;
  int recs = ready ? 1 : 0;
  if (ready && pk.w == kWide) {
    const int s = wide_shift(pk.y);
    recs = (int)((unsigned)(pk.y - 1) >> s) + 1;
  }
  int at = __popc(set & ((1u << lane) - 1u)), total = __popc(set);
  bool stay = false;
  if (__any_sync(FULL, recs > 1)) {
    if constexpr (Gp::kKeepLong) stay = __any_sync(FULL, recs > kWideStay);
    int upto = recs;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(FULL, upto, d);
      if (lane >= d) upto += y;
    }
    at = upto - recs;
    total = __shfl_sync(FULL, upto, 31);
  }
  int* len = g.length(L);
  int base = -1;
  if (lane == 0 && (*(volatile int*)len < g.most() || stay)) base = atomicAdd(len, total);
  base = __shfl_sync(FULL, base, 0);
  if (ready) {
    if (base < 0) g.hand_on(v, pk, recs, L);
    else if (!put_records(ls.rec(L), ls.pin(L), ls.cap, base + at, recs, v, pk))
      g.spill(v, L);
  }
}

// Decrements for the records get(0), get(1), ..., get(m - 1), a quad of
// lanes each (get(k, f): word f of record k), by `threads` threads of which
// this is number `at`; the pins made ready are of level L.
template <class Gp, class GetF>
__device__ __forceinline__ void expand(const Gp& g, const LvArgs& a, const LvLists& ls, int m,
                                       int at, int threads, int L, GetF get) {
  const int lane = threadIdx.x & 31;
  // unsigned: m and the threads' stride may add up to more than an int holds
  for (unsigned k0 = (unsigned)(at & ~31) / 4; k0 < (unsigned)m; k0 += (unsigned)threads / 4) {
    const unsigned k = k0 + (lane >> 2);
    int x = k < (unsigned)m ? get((int)k, lane & 3) : -1;
    if (__any_sync(FULL, x == kWide)) {  // only a record's last word is kWide
      const bool wide = __shfl_sync(FULL, x, lane | 3) == kWide;
      const int e0 = __shfl_sync(FULL, x, lane & ~3), deg = __shfl_sync(FULL, x, (lane & ~3) | 1);
      if (wide) x = deg <= kWideMax && (lane & 3) < deg ? a.fanin[e0 + (lane & 3)] : -1;
      unsigned todo = __ballot_sync(FULL, wide && deg > kWideMax && (lane & 3) == 0);
      while (todo) {  // a warp at a time
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const int e1 = __shfl_sync(FULL, e0, src), d1 = __shfl_sync(FULL, deg, src);
        for (int e = 0; e < d1; e += 32)
          decrement(g, a, ls, e + lane < d1 ? a.fanin[e1 + e + lane] : -1, L);
      }
    }
    decrement(g, a, ls, x, L);
  }
}

// The seed: order and level 0, their counters out of reach of decrements.
template <class Gp>
__device__ __forceinline__ void seed(const Gp& g, const LvArgs& a, int at, int threads) {
  for (int k = at; k < a.first_size; k += threads) {
    const int v = a.frontier0[k];
    a.order[k] = v;
    if ((unsigned)v < (unsigned)a.n) {
      a.level[v] = 0;
      *g.counter(v) = INT_MAX;
    } else {
      atomicCAS(&a.ctl->grid.status, 0, (int)OTG_ERR_INVALID);
    }
  }
}
__device__ __forceinline__ int seed_word(const LvArgs& a, int k, int f) {
  const int u = a.frontier0[k];
  return (unsigned)u < (unsigned)a.n ? ((const int*)a.packed)[4 * (size_t)u + f] : -1;
}
__device__ __forceinline__ int spill_word(const LvArgs& a, int L, int k, int f) {
  const int u = __ldcg(a.spill + (size_t)(L & 1) * a.n + k);
  return __ldcg((const int*)a.packed + 4 * (size_t)u + f);
}

// ---- the cluster form ----------------------------------------------------
//
// Pin v's counter lies in CTA v mod S (neighbouring pins are often of one
// level, so ranges would send a level's atomics to one CTA).  A CTA that
// readied more than kLocalMax entries of a level hands the rest to a CTA
// chosen by a hash of the pin (a buffer tree readies its levels from one
// place); what no list holds goes to the spill list in global memory.  Two
// warps write the pins' levels and fetch the CTAs' list lengths, and find
// the end one level late: 16 stores from each CTA into all others cost 600
// cycles of the barrier that waits for them, and a global store 400.
//
// No wait here polls memory: the cluster barrier is hardware, and every CTA
// takes the same number of barriers (the loop ends on lengths that every
// CTA reads alike).
constexpr int kLocalMax = 64;
constexpr int kNoteWarps = 2;

struct ClWords {
  int len[4];  // list lengths by level (may exceed the capacity); a level's is filled in the
               // level before, read in its own, cleared in the next
  int ovf[4];  // some pin of the level was spilled (set in every CTA)
  int done;    // an empty level was reached
};

struct ClGroup {
  const cg::cluster_group& cl;
  const LvArgs& a;
  const LvLists& ls;
  ClWords& sw;
  int* scnt;   // this CTA's counters, or null: the global ones
  int sshift;  // log2 of the cluster size
  __device__ int* counter(int v) const {
    return scnt ? cl.map_shared_rank(scnt + (v >> sshift), v & ((1 << sshift) - 1)) : a.cnt + v;
  }
  __device__ int* length(int L) const { return &sw.len[L & 3]; }
  __device__ int most() const { return kLocalMax; }
  static constexpr bool kKeepLong = false;  // another CTA's list is as good
  __device__ void spill(int v, int L) const {
    spill_pin(a, v, L);
    for (int i = 0; i < (1 << sshift); ++i) *cl.map_shared_rank(&sw.ovf[L & 3], i) = 1;
  }
  __device__ void hand_on(int v, int4 pk, int recs, int L) const {
    const int t = sshift ? (int)(((unsigned)v * 0x9E3779B1u) >> (32 - sshift)) : 0;
    const int at = atomicAdd(cl.map_shared_rank(&sw.len[L & 3], t), recs);
    if (!put_records(cl.map_shared_rank(ls.rec(L), t), cl.map_shared_rank(ls.pin(L), t), ls.cap,
                     at, recs, v, pk))
      spill(v, L);
  }
};

template <int CT>
__global__ void __launch_bounds__(CT, 1)
    levelize_cluster_kernel(LvArgs a, int lst_cap, int scnt_on) {
  extern __shared__ __align__(16) unsigned lv_sm[];
  __shared__ ClWords sw;
  const cg::cluster_group cl = cg::this_cluster();
  const int S = (int)cl.num_blocks(), r = (int)cl.block_rank(), tid = threadIdx.x;
  const int gtid = r * CT + tid, gstride = S * CT, lane = tid & 31;
  const LvLists ls{(int4*)lv_sm, (int*)((int4*)lv_sm + 2 * lst_cap), lst_cap};
  const ClGroup g{cl, a, ls, sw, scnt_on ? ls.pin0 + 2 * lst_cap : nullptr, 31 - __clz(S)};
  if (g.scnt)
    for (int v = r + tid * S; v < a.n; v += CT * S) g.scnt[v >> g.sshift] = a.out_deg[v];
  if (tid < (int)(sizeof(ClWords) / 4)) ((int*)&sw)[tid] = 0;
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the records, counters and levels' fill
  cl.sync();
  seed(g, a, gtid, gstride);
  cl.sync();
  expand(g, a, ls, a.first_size, gtid, gstride, 1, [&](int k, int f) { return seed_word(a, k, f); });
  constexpr int XT = CT - 32 * kNoteWarps;  // expanding threads
  int L = 1;
  for (;; ++L) {
    cl.sync();
    if (sw.done) break;
    const int p = L & 1, m = min(sw.len[L & 3], ls.cap);
    const bool over = sw.ovf[L & 3] != 0;
    if (tid < XT) {
      const int4* rec = ls.rec(L);
      expand(g, a, ls, m, tid, XT, L + 1, [&](int k, int f) { return ((const int*)(rec + k))[f]; });
      if (over) {
        const int ns = __ldcg(&a.ctl->spill[L & 3]);
        for (int k = r * XT + tid; k < ns; k += S * XT) a.level[__ldcg(a.spill + (size_t)p * a.n + k)] = L;
        expand(g, a, ls, ns, r * XT + tid, S * XT, L + 1,
               [&](int k, int f) { return spill_word(a, L, k, f); });
      }
    } else {
      const int x = lane < S ? *(volatile int*)cl.map_shared_rank(&sw.len[L & 3], lane) : 0;
      for (int k = tid - XT; k < m; k += 32 * kNoteWarps) {
        const int v = ls.pin(L)[k];
        if (v >= 0) a.level[v] = L;
      }
      if (!__any_sync(FULL, x != 0) && !over && lane == 0) sw.done = 1;
    }
    // the level before this one is behind every CTA
    if (tid == 0) {
      sw.len[(L - 1) & 3] = sw.ovf[(L - 1) & 3] = 0;
      if (r == 0) a.ctl->spill[(L - 1) & 3] = 0;
    }
  }
  if (gtid == 0) a.ctl->levels = L - 1;
  cl.sync();  // no CTA leaves while another may still read its list length
}

// ---- the grid form -------------------------------------------------------
//
// A CTA per SM.  A CTA that has readied a quarter more than its share of a
// level's entries, going by the level before, puts further pins on the
// spill list, which all CTAs share out: the CTAs with the most pins ready
// the most, so that lists left alone drift apart (68 to 558 entries on
// average over 5M pins' 200 levels).
constexpr int LT = 1024;
constexpr int kGridCap = 4096, kGridLeast = 64;
constexpr int kSpillWarps = 4;  // the warps that take the CTA's share of the spill list

// A grid barrier for many uses in one launch: arrivals only count up, so the
// last CTA's arrival is itself what the others wait for (a counter that is
// reset and a generation that is then raised, each behind a fence, took
// 4.5 us a level).  Waits are bounded as grid_barrier's.
struct GridWait {
  GridCtl* c;
  unsigned target = 0;
  __device__ bool wait() {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&c->count) : "memory");
      target += gridDim.x;
      int ok = 1;
      unsigned long long t0 = 0;
      for (int k = 0;; ++k) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&c->count) : "memory");
        if ((int)(v - target) >= 0) break;
        if ((k & 15) != 15) continue;
        const unsigned long long t = gtime();
        if (t0 == 0) t0 = t;
        if (t - t0 > kGridWaitNs) {
          atomicExch(&c->abort, 1);
          atomicCAS(&c->status, 0, (int)OTG_ERR_TIMEOUT);
        }
        if (*(volatile int*)&c->abort) {
          ok = 0;
          break;
        }
      }
      s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
  }
};

struct GridGroup {
  const LvArgs& a;
  int* len;         // by level parity
  const int* room;  // entries before a warp puts pins on the spill list
  __device__ int* counter(int v) const { return a.cnt + v; }
  __device__ int* length(int L) const { return len + (L & 1); }
  __device__ int most() const { return *room; }
  // the list spreads a very long pin (over kWideStay records) over the CTA's
  // warps, the spill list does not
  static constexpr bool kKeepLong = true;
  __device__ void spill(int v, int L) const { spill_pin(a, v, L); }
  __device__ void hand_on(int v, int4, int, int L) const { spill_pin(a, v, L); }
};

__global__ void __launch_bounds__(LT, 1) levelize_grid_kernel(LvArgs a) {
  extern __shared__ __align__(16) unsigned lv_sm[];
  __shared__ int s_len[2], s_room, s_done;
  const int G = gridDim.x, tid = threadIdx.x;
  const int gtid = blockIdx.x * LT + tid, gstride = G * LT;
  const LvLists ls{(int4*)lv_sm, (int*)((int4*)lv_sm + 2 * kGridCap), kGridCap};
  const GridGroup g{a, s_len, &s_room};
  GridWait barrier{&a.ctl->grid};
  if (tid < 2) s_len[tid] = 0;
  if (tid == 0) {
    s_room = max(kGridLeast, a.first_size / G);
    s_done = 0;
  }
  seed(g, a, gtid, gstride);
  if (!barrier.wait()) return;
  expand(g, a, ls, a.first_size, gtid, gstride, 1, [&](int k, int f) { return seed_word(a, k, f); });
  constexpr int XT = LT - 32 * kSpillWarps;  // the threads of the CTA's own list
  int L = 1;
  for (;; ++L) {
    const int p = L & 1;
    __syncthreads();
    if (tid == 0 && s_len[p]) atomicAdd(&a.ctl->tot[L & 3], s_len[p]);
    if (!barrier.wait()) return;
    if (s_done) break;  // the same in every CTA: all read the same totals
    const int m = min(s_len[p], ls.cap);
    if (tid < XT) {
      for (int k = tid; k < m; k += XT) {
        const int v = ls.pin(L)[k];
        if (v >= 0) a.level[v] = L;
      }
      const int4* rec = ls.rec(L);
      expand(g, a, ls, m, tid, XT, L + 1, [&](int k, int f) { return ((const int*)(rec + k))[f]; });
    } else {
      // the level's totals (nobody else waits for them: the end is found a
      // level late), and every G-th pin of the spill list
      const int tot = __ldcg(&a.ctl->tot[L & 3]), ns = __ldcg(&a.ctl->spill[L & 3]);
      if (tid == XT) {
        if (tot == 0 && ns == 0) s_done = 1;
        s_room = max(kGridLeast, min((int)((long long)(tot + ns) * 5 / 4 / G), kGridCap / 2));
      }
      const int b = blockIdx.x, share = max(0, (ns - b + G - 1) / G);
      for (int k = tid - XT; k < share; k += LT - XT)
        a.level[__ldcg(a.spill + (size_t)p * a.n + b + k * G)] = L;
      expand(g, a, ls, share, tid - XT, LT - XT, L + 1,
             [&](int k, int f) { return spill_word(a, L, b + k * G, f); });
    }
    __syncthreads();
    if (tid == 0) {
      s_len[p] = 0;  // level L + 2's
      if (blockIdx.x == 0) a.ctl->tot[(L - 1) & 3] = a.ctl->spill[(L - 1) & 3] = 0;
    }
  }
  if (gtid == 0) a.ctl->levels = L - 1;
}

// ---- the sort ------------------------------------------------------------
//
// Pins by level - 1 (level 0 is the seed, in the caller's order), stable in
// the pin index: digits of kDigitBits, each by a histogram per tile of
// consecutive items, a scan and a scatter.  A pass whose digit is 0 for every
// level is left out: its kernels return at once, and where the graph has too
// few pins for so many levels, they are not launched.
constexpr int kDigitBits = 10, kDigits = 1 << kDigitBits, kMinTiles = 6, kMaxTiles = 256,
              ST = 1024;

struct LvSort {
  int per;      // items per tile
  int tiles;
  int* hist;    // [kDigits][tiles]
  int* part;    // two lists of n pins: sorted by the digits so far, by pass
  int* num;     // their number
};

// Whether a pass has nothing to sort: the digit of the highest level - 1,
// and all above it, are 0.
__host__ __device__ __forceinline__ bool sort_skip(int levels, int pass) {
  return pass > 0 && ((long long)levels - 2) >> (kDigitBits * pass) <= 0;
}

// Item i of a pass and its digit (-1: not an item): the pins in index order
// (pass 0), or the pass before's output.
__device__ __forceinline__ int sort_item(const LvArgs& a, const LvSort& s, int pass, int i,
                                         int& v) {
  if (pass == 0) {
    v = i;
    const int l = i < a.n ? a.level[i] : 0;
    return l > 0 ? (l - 1) & (kDigits - 1) : -1;
  }
  if (i >= *s.num) return -1;
  v = s.part[(size_t)((pass - 1) & 1) * a.n + i];
  return ((a.level[v] - 1) >> (kDigitBits * pass)) & (kDigits - 1);
}

__global__ void __launch_bounds__(ST) levelize_hist(LvArgs a, LvSort s, int pass) {
  __shared__ int h[kDigits];
  asm volatile("griddepcontrol.launch_dependents;\n griddepcontrol.wait;" ::: "memory");
  if (sort_skip(a.ctl->levels, pass)) return;
  for (int d = threadIdx.x; d < kDigits; d += ST) h[d] = 0;
  __syncthreads();
  const int b = blockIdx.x * s.per;
  for (int i = threadIdx.x; i < s.per; i += ST) {
    int v;
    const int d = sort_item(a, s, pass, b + i, v);
    if (d >= 0) atomicAdd(&h[d], 1);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kDigits; d += ST) s.hist[d * s.tiles + blockIdx.x] = h[d];
}

// Exclusive scan over (digit, tile), a thread per digit; with one digit, the
// levels' ends and the counts too.
__global__ void __launch_bounds__(kDigits) levelize_scan(LvArgs a, LvSort s, int pass) {
  __shared__ int wsum[kDigits / 32];
  asm volatile("griddepcontrol.launch_dependents;\n griddepcontrol.wait;" ::: "memory");
  if (sort_skip(a.ctl->levels, pass)) return;
  const int d = threadIdx.x, lane = d & 31, w = d >> 5;
  int* row = s.hist + d * s.tiles;
  int sum = 0;
#pragma unroll 8
  for (int t = 0; t < s.tiles; ++t) sum += row[t];
  int x = sum;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    const int y = __shfl_up_sync(FULL, x, k);
    if (lane >= k) x += y;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  const int below = wsum[lane];
  int run = __reduce_add_sync(FULL, lane < w ? below : 0) + x - sum;
  const int total = __reduce_add_sync(FULL, below);
  const int levels = a.ctl->levels, end = a.first_size + run + sum;
#pragma unroll 8
  for (int t = 0; t < s.tiles; ++t) {
    const int c = row[t];
    row[t] = run;
    run += c;
  }
  if (pass == 0 && d + 1 < levels) a.level_ends[d + 2] = min(end, a.n);
  if (pass == 0 && d == 0) {
    *s.num = total;
    a.level_ends[0] = 0;
    if (levels > 0) a.level_ends[1] = a.first_size;
    // only with duplicate seeds are there more than n
    if (a.first_size + total > a.n) atomicCAS(&a.ctl->grid.status, 0, (int)OTG_ERR_INVALID);
    a.counts[0] = levels;
    a.counts[1] = min(a.first_size + total, a.n);
  }
}

// The lanes with the same digit (d < 0: none), bit by bit; see decrement on
// match_any.
__device__ __forceinline__ unsigned same_digit(int d) {
  unsigned peers = __ballot_sync(FULL, d >= 0);
#pragma unroll
  for (int k = 0; k < kDigitBits; ++k) {
    const unsigned on = __ballot_sync(FULL, (d >> k) & 1);
    peers &= (d >> k) & 1 ? on : ~on;
  }
  return peers;
}

__global__ void __launch_bounds__(ST) levelize_scatter(LvArgs a, LvSort s, int pass) {
  extern __shared__ __align__(16) unsigned lv_sm[];
  uint16_t* cnt = (uint16_t*)lv_sm;                  // [warp][digit], then the warps' bases
  int* base = (int*)(cnt + (ST / 32) * kDigits);     // [digit] the tile's base
  asm volatile("griddepcontrol.launch_dependents;\n griddepcontrol.wait;" ::: "memory");
  if (sort_skip(a.ctl->levels, pass)) return;
  const bool last = sort_skip(a.ctl->levels, pass + 1);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < (ST / 32) * kDigits / 2; i += ST) ((unsigned*)cnt)[i] = 0u;
  for (int d = threadIdx.x; d < kDigits; d += ST) base[d] = s.hist[d * s.tiles + blockIdx.x];
  __syncthreads();
  // each warp takes consecutive items, 32 at a time
  const int b = blockIdx.x * s.per + w * (s.per / (ST / 32));
  const int per = min(s.per / (ST / 32), (pass == 0 ? a.n : *s.num) - b);
  uint16_t* mine = cnt + w * kDigits;
  for (int i = 0; i < per; i += 32) {
    int v;
    const int d = sort_item(a, s, pass, b + i + lane, v);
    const unsigned peers = same_digit(d);
    if (d >= 0 && __ffs(peers) - 1 == lane) mine[d] += (uint16_t)__popc(peers);
    __syncwarp();
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kDigits; d += ST) {
    int run = 0;
#pragma unroll 8
    for (int k = 0; k < ST / 32; ++k) {
      const int c = cnt[k * kDigits + d];
      cnt[k * kDigits + d] = (uint16_t)run;
      run += c;
    }
  }
  __syncthreads();
  int* out = last ? a.order : s.part + (size_t)(pass & 1) * a.n;
  const int off = last ? a.first_size : 0;
  for (int i = 0; i < per; i += 32) {
    int v;
    const int d = sort_item(a, s, pass, b + i + lane, v);
    const unsigned peers = same_digit(d);
    int pos = 0;
    if (d >= 0) pos = off + base[d] + mine[d] + __popc(peers & ((1u << lane) - 1u));
    __syncwarp();
    if (d >= 0) {
      if (__ffs(peers) - 1 == lane) mine[d] += (uint16_t)__popc(peers);
      if (pos < a.n) out[pos] = v;
    }
    __syncwarp();
  }
}

// The levels' ends from the sorted pins, where the first digit did not give
// them.
__global__ void levelize_ends(LvArgs a, LvSort s) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (sort_skip(a.ctl->levels, 1)) return;
  const int end = min(a.first_size + *s.num, a.n);
  for (int p = a.first_size + blockIdx.x * blockDim.x + threadIdx.x; p < end;
       p += gridDim.x * blockDim.x) {
    const int l = a.level[a.order[p]];
    if (p == a.first_size || a.level[a.order[p - 1]] != l) a.level_ends[l] = p;
    if (p == end - 1) a.level_ends[l + 1] = end;
  }
}

// ---- host ------------------------------------------------------------------
constexpr size_t kClusterSmemMax = 200 * 1024;
constexpr int kLstMin = 1024;  // entries of a CTA's list at least
constexpr size_t kEntry = 2 * (sizeof(int4) + sizeof(int));
size_t scnt_bytes(int n, int S) { return 4 * (((size_t)n + S - 1) / S); }

constexpr int kWidths[4] = {128, 256, 512, 1024};
const void* cluster_fn(int wi) {
  switch (wi) {
    case 0: return (const void*)levelize_cluster_kernel<128>;
    case 1: return (const void*)levelize_cluster_kernel<256>;
    case 2: return (const void*)levelize_cluster_kernel<512>;
    default: return (const void*)levelize_cluster_kernel<1024>;
  }
}
constexpr size_t kGridSmem = kEntry * kGridCap;
constexpr size_t kScatterSmem = 2 * (ST / 32) * kDigits + 4 * kDigits;

struct LvDev {
  int sms = 0;
  bool init = false;
  int max_cluster[4] = {0, 0, 0, 0};  // per CTA width: largest cluster (power of two <= 16) placed
};
LvDev g_lv[64];

LvDev& lv_dev() {
  int d = 0;
  cudaGetDevice(&d);
  LvDev& x = g_lv[d & 63];
  if (!x.init) {
    cudaDeviceGetAttribute(&x.sms, cudaDevAttrMultiProcessorCount, d);
    cudaFuncSetAttribute(levelize_grid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kGridSmem);
    cudaFuncSetAttribute(levelize_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kScatterSmem);
    // the cluster path: allow its largest shared memory and 16-CTA clusters,
    // then keep, per CTA width, the largest cluster size the device places
    for (int wi = 0; wi < 4; ++wi) {
      const void* fn = cluster_fn(wi);
      if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kClusterSmemMax) != cudaSuccess ||
          cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
              cudaSuccess)
        continue;
      for (int s = 16; s >= 1 && !x.max_cluster[wi]; s >>= 1) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)s;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(s);
        cfg.blockDim = dim3(kWidths[wi]);
        cfg.dynamicSmemBytes = kClusterSmemMax;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int nc = 0;
        if (cudaOccupancyMaxActiveClusters(&nc, fn, &cfg) == cudaSuccess && nc >= 1)
          x.max_cluster[wi] = s;
      }
    }
    cudaGetLastError();  // a refused attribute or query leaves no sticky error
    x.init = true;
  }
  return x;
}

// The cluster form's shape for an n-pin graph: S CTAs of kWidths[wi]
// threads.  S = 0: the grid form.
struct ClPlan {
  int S = 0, wi = 0, cap = 0;
  bool scnt = false;  // the fanout counters in shared memory
};
// Default: the largest cluster the device places (16 CTAs on B200) of 512
// threads each, for graphs whose counters it holds (up to 650k pins); larger
// graphs take the grid form, which spreads a level over every SM.  Cluster
// against grid: 163k pins / 374 levels 551 and 1053 us, 400k / 200 levels 593
// and 687, 329k / 106 levels 400 and 403; with the counters in global memory
// 900k / 300 levels 1289 and 1137.  256 threads take 712, 861 and 539 us on
// the first three (fewer warps expand), 1024 602 on the first.
// OTG_LEVELIZE_CLUSTER=0 turns the cluster form off, =1|2|4|8|16 asks for
// that size; OTG_LEVELIZE_CT=128|256|512|1024 asks for that width (both only
// where the device places the cluster); OTG_LEVELIZE_SCNT=0 keeps the
// counters in global memory.
ClPlan lv_cluster_plan(int n, const LvDev& d) {
  ClPlan p;
  p.wi = 2;
  if (const char* e = std::getenv("OTG_LEVELIZE_CT")) {
    const int want = std::atoi(e);
    for (int wi = 0; wi < 4; ++wi)
      if (kWidths[wi] == want) p.wi = wi;
  }
  const int maxc = d.max_cluster[p.wi];
  if (maxc < 1) return ClPlan{};
  int s = maxc;
  if (const char* e = std::getenv("OTG_LEVELIZE_CLUSTER")) {
    const int want = std::atoi(e);
    if (want <= 0) return ClPlan{};
    s = 1;
    while (s < want && s < maxc) s <<= 1;
  } else if (scnt_bytes(n, s) + kEntry * kLstMin > kClusterSmemMax) {
    return ClPlan{};
  }
  p.S = s;
  p.scnt = scnt_bytes(n, s) + kEntry * kLstMin <= kClusterSmemMax;
  if (const char* e = std::getenv("OTG_LEVELIZE_SCNT"))
    if (std::atoi(e) == 0) p.scnt = false;
  p.cap = (int)((kClusterSmemMax - (p.scnt ? scnt_bytes(n, s) : 0)) / kEntry) & ~3;
  return p;
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Items per sort tile: a multiple of 32 per warp, and no more than the
// scatter's 16-bit counts hold.  About kMinTiles tiles while these are small
// (one CTA for all takes as long as 8,192 pins whatever their number: 200 pins
// / 3 levels 31 us, now 21; 8,000 45 and 39), then kMaxTiles at most (the scan
// reads them one after another: 60k gates 813 us with tiles of 1,024, 686).
LvSort lv_tiles(int n) {
  LvSort s{};
  s.per = ST;
  while (s.per < 8 * ST && (long long)s.per * kMinTiles < n) s.per += ST;
  while (s.per < 63 * ST && (long long)s.per * kMaxTiles < n) s.per += ST;
  s.tiles = std::max(1, (int)(((long long)n + s.per - 1) / s.per));
  return s;
}

struct LvWs {
  size_t ctl, cnt, packed, spill, hist, total;
};
LvWs lv_ws(int n) {
  LvWs l;
  const size_t N = (size_t)std::max(n, 1);
  size_t o = 0;
  l.ctl = o; o = align256(o + sizeof(LvCtl) + 4);  // and the sort's item count
  l.cnt = o; o = align256(o + 4 * N);
  l.packed = o; o = align256(o + sizeof(int4) * N);
  l.spill = o; o = align256(o + 8 * N);
  l.hist = o; o = align256(o + 4 * (size_t)kDigits * lv_tiles(n).tiles);
  l.total = o + 16;
  return l;
}

// The records are read and written as 16-byte vectors.
char* lv_base(void* ws) { return (char*)(((uintptr_t)ws + 15) & ~(uintptr_t)15); }

template <class... P, class... A>
cudaError_t lv_launch(void (*kern)(P...), int grid, int block, size_t smem, bool overlap,
                      cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = overlap ? 1 : 0;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

}  // namespace
}  // namespace otg

extern "C" {

otg_status otg_levelize_workspace_size(int32_t n, int32_t num_edges, size_t* bytes) {
  (void)num_edges;
  if (!bytes || n < 0) return OTG_ERR_INVALID;
  if (otg::lv_dev().sms <= 0) return OTG_ERR_CUDA;
  *bytes = otg::lv_ws(n).total;
  return OTG_OK;
}

otg_status otg_levelize(int32_t n, int32_t num_edges, const int32_t* fanin_start,
                        const int32_t* fanin, const int32_t* out_deg, const int32_t* frontier0,
                        int32_t first_size, int32_t* order, int32_t* level, int32_t* level_ends,
                        int32_t* counts, void* workspace, size_t workspace_bytes,
                        otg_stream_t stream) {
  if (n < 0 || num_edges < 0 || first_size < 0 || first_size > n || !workspace || !counts ||
      !level_ends)
    return OTG_ERR_INVALID;
  if (n > 0 && (!fanin_start || !out_deg || !order || !level || (first_size && !frontier0) ||
                (num_edges && !fanin)))
    return OTG_ERR_INVALID;
  otg::LvDev& d = otg::lv_dev();
  const otg::LvWs l = otg::lv_ws(n);
  if (workspace_bytes < l.total) return OTG_ERR_WORKSPACE;
  char* ws = otg::lv_base(workspace);
  cudaStream_t st = (cudaStream_t)stream;
  otg::LvArgs a{n,     fanin_start, fanin,      out_deg, frontier0,
                first_size, order,  level,      level_ends, counts,
                (otg::LvCtl*)(ws + l.ctl), (int*)(ws + l.cnt), (int4*)(ws + l.packed),
                (int*)(ws + l.spill)};
  const otg::ClPlan pl = otg::lv_cluster_plan(n, d);
  const bool on_chip = pl.S > 0 && pl.scnt;
  cudaError_t e = otg::lv_launch(otg::levelize_pack, std::max(1, std::min((n + 255) / 256, 8 * d.sms)),
                                 256, 0, false, st, a, !on_chip);
  if (e == cudaSuccess && first_size > 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    cfg.stream = st;
    cfg.attrs = at;
    if (pl.S > 0) {
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = (unsigned)pl.S;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      // its counters are filled while the records are packed
      at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.numAttrs = 2;
      cfg.gridDim = dim3(pl.S);
      cfg.blockDim = dim3(otg::kWidths[pl.wi]);
      cfg.dynamicSmemBytes = otg::kClusterSmemMax;
      int cap = pl.cap, scnt = on_chip ? 1 : 0;
      void* args[] = {&a, &cap, &scnt};
      e = cudaLaunchKernelExC(&cfg, otg::cluster_fn(pl.wi), args);
    } else {
      void* args[] = {&a};
      e = cudaLaunchCooperativeKernel((const void*)otg::levelize_grid_kernel, dim3(d.sms),
                                      dim3(otg::LT), args, otg::kGridSmem, st);
    }
    otg::count_launch();
  }
  otg::LvSort s = otg::lv_tiles(n);
  s.hist = (int*)(ws + l.hist);
  s.part = (int*)(ws + l.packed);  // the records have been read
  s.num = (int*)(ws + l.ctl + sizeof(otg::LvCtl));
  int pass = 0;
  for (; !otg::sort_skip(n, pass) && e == cudaSuccess; ++pass) {  // n: a level has at least one pin
    e = otg::lv_launch(otg::levelize_hist, s.tiles, otg::ST, 0, pass > 0, st, a, s, pass);
    if (e == cudaSuccess)
      e = otg::lv_launch(otg::levelize_scan, 1, otg::kDigits, 0, true, st, a, s, pass);
    if (e == cudaSuccess)
      e = otg::lv_launch(otg::levelize_scatter, s.tiles, otg::ST, otg::kScatterSmem, true, st, a, s,
                         pass);
  }
  if (e == cudaSuccess && pass > 1)
    e = otg::lv_launch(otg::levelize_ends, std::max(1, std::min((n + 255) / 256, 4 * d.sms)), 256,
                       0, true, st, a, s);
  if (e == cudaSuccess) return OTG_OK;
  cudaGetLastError();
  return OTG_ERR_CUDA;
}

otg_status otg_levelize_status(const void* workspace, otg_stream_t stream) {
  if (!workspace) return OTG_ERR_INVALID;
  otg::GridCtl h;
  if (cudaMemcpyAsync(&h, otg::lv_base((void*)workspace), sizeof(h), cudaMemcpyDeviceToHost, (cudaStream_t)stream) !=
          cudaSuccess ||
      cudaStreamSynchronize((cudaStream_t)stream) != cudaSuccess)
    return OTG_ERR_CUDA;
  return (otg_status)h.status;
}

}  // extern "C"
