// otg_prop.cu -- levelized timing propagation on the GPU, the consumer of
// the RC pass: slew, arc delay, arrival time and timing-test RAT forward,
// required time and slack backward, two splits x two transitions.
//
// Semantics follow the reference Timer's per-pin tasks: Timer::_fprop_slew,
// _fprop_delay, _fprop_at, _fprop_test, _bprop_rat (ot/timer/timer.cpp:733-
// 832), Arc::_fprop_slew/_fprop_delay/_fprop_at/_bprop_rat (arc.cpp:82-
// 205), Pin::_relax_slew/_relax_at/_relax_rat (pin.cpp:324-380), Test::
// _fprop_rat (test.cpp:88-135), Timing::delay/slew/constraint and
// is_transition_defined (ot/liberty/timing.cpp:198-230, 411-628), and the
// look-up interpolation Lut::operator() (ot/liberty/lut.cpp:166-245).  Net
// arcs read the RC pass's outputs: the driver's load at BFS slot 0, the
// Elmore delay and sign(si)*sqrt(si^2 + impulse) at the sink's slot
// (net.cpp:626-699, FlatRct accessors).  A value the reference keeps as an
// empty std::optional is NaN here.  Every add and multiply is an explicit
// rounding intrinsic, so no compiler fusion changes a bit.
//
// Schedule: one cooperative launch, a warp per pin, dataflow instead of
// level barriers.  Pins are numbered in level order (otg_levelize: every
// pin after all of its fanouts); the forward pass takes them last level
// first, warp w the items w, w+W, w+2W, ...  A pin waits (bounded) until
// the values it reads from its fanins are there, computes, and stores its
// own.  Because a pin depends only on lower-numbered items and each warp
// works through its items in order, the lowest unfinished item always has
// every input ready: the schedule cannot deadlock while all CTAs are
// resident, which the cooperative launch guarantees.  One grid barrier
// separates the forward pass from the backward pass, which runs the same
// way first level first.
//
// Readiness is carried by the values themselves: a fill kernel sets every
// arrival time and slew to kPending, a NaN payload that no stored value
// carries (an empty value is stored as the canonical NaN), and the forward
// pass does the same to each pin's required time before the barrier.  A
// reader polls exactly the words it needs with relaxed loads, each word is
// written once, so no fence or flag sits on the critical path.
//
// Inside a warp the lanes split a pin's (arc, split, from-transition,
// to-transition) combinations and reduce with shuffles; min/max reductions
// are order-free, so the lane split does not change a value.  Values that
// other warps wrote after the barrier are read with __ldcg (L2); the graph
// and the library are read-only for the launch and go through __ldg.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "../../include/otg.h"
#include "otg_internal.cuh"

namespace otg {
namespace {

constexpr int MIN_ = 0, MAX_ = 1, RISE_ = 0, FALL_ = 1;

__device__ __forceinline__ bool none(float x) { return isnan(x); }

// Lut::operator(): clamped segment search by lower_bound, then linear
// inter/extrapolation per axis (boundary values returned as they are).
__device__ float interpolate(float x, float x1, float x2, float y1, float y2) {
  if (x >= 3.402823466e+38f || x <= -3.402823466e+38f) return x;
  const float slope = __fdiv_rn(__fsub_rn(y2, y1), __fsub_rn(x2, x1));
  if (x < x1) return __fsub_rn(y1, __fmul_rn(__fsub_rn(x1, x), slope));
  if (x > x2) return __fadd_rn(y2, __fmul_rn(__fsub_rn(x, x2), slope));
  if (x == x1) return y1;
  if (x == x2) return y2;
  return __fadd_rn(y1, __fmul_rn(__fsub_rn(x, x1), slope));
}

// Table reads go through a generic pointer: shared memory when the
// library is staged on chip, else global memory (cached in L1).
__device__ int lower_bound(const float* a, int n, float v) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid] < v) lo = mid + 1; else hi = mid;
  }
  return lo;
}

struct G {
  otg_prop_graph g;
  otg_prop_rc rc;
};

constexpr unsigned FULL = 0xffffffffu;

// A table chosen before the query values are known: lut_meta's (n1, n2,
// offset, variable order), n1 = -1 for "no table".
struct Lut {
  int n1, n2, off, var;
};

__device__ __forceinline__ Lut no_lut() { return Lut{-1, 0, 0, 0}; }

// Lut::operator() on (v1, v2) in the table's own axis order.
__device__ float lut_eval(const Lut& m, const float* data, float v1, float v2) {
  const int n1 = m.n1, n2 = m.n2;
  const float* i1 = data + m.off;
  const float* i2 = i1 + n1;
  const float* tb = i2 + n2;
  if (n1 < 1 || n2 < 1) return nanf("");
  if (n1 == 1 && n2 == 1) return tb[0];
  const int a1 = max(1, min(lower_bound(i1, n1, v1), n1 - 1));
  const int a2 = max(1, min(lower_bound(i2, n2, v2), n2 - 1));
  if (n1 == 1) return interpolate(v2, i2[a2 - 1], i2[a2], tb[a2 - 1], tb[a2]);
  const float x1 = i1[a1 - 1], x2 = i1[a1];
  if (n2 == 1) return interpolate(v1, x1, x2, tb[(a1 - 1) * n2], tb[a1 * n2]);
  const float lo = interpolate(v1, x1, x2, tb[(a1 - 1) * n2 + a2 - 1], tb[a1 * n2 + a2 - 1]);
  const float hi = interpolate(v1, x1, x2, tb[(a1 - 1) * n2 + a2], tb[a1 * n2 + a2]);
  return interpolate(v2, i2[a2 - 1], i2[a2], lo, hi);
}

// timing record: [sense, edge, constraint, lut x6]
__device__ bool transition_defined(const int* tr, int irf, int orf) {
  const int edge = __ldg(tr + 1), sense = __ldg(tr);
  if (edge == 1 && irf != RISE_) return false;
  if (edge == 2 && irf != FALL_) return false;
  if (sense == 0 && irf != orf) return false;  // positive unate
  if (sense == 1 && irf == orf) return false;  // negative unate
  return true;
}

// The table a Timing::delay/slew/constraint query of record t reads:
// which = 0 delay, 1 slew, 2 constraint.
__device__ Lut timing_lut(const G& G_, int t, int which, int irf, int orf) {
  if (t < 0) return no_lut();
  const int* tr = G_.g.timing + 9 * t;
  if (!transition_defined(tr, irf, orf)) return no_lut();
  const int lut = __ldg(tr + 3 + 2 * which + orf);
  if (lut < 0) return no_lut();
  const int4 m = __ldg(reinterpret_cast<const int4*>(G_.g.lut_meta) + lut);
  return Lut{m.x, m.y, m.z, m.w};
}

// The query itself; (a, b) = (slew, load) for delay and slew, (related
// slew, constrained slew) for constraint.
// Where the tables are read: the staged copy (floats [0, n)) for a table
// that lies inside it, global memory otherwise.
struct LutSrc {
  const float* smem;
  int n;
  const float* gmem;
};

__device__ __noinline__ float timing_value(const LutSrc& src, const Lut& m, float a, float b) {
  if (m.n1 < 0) return nanf("");
  const bool staged = m.off >= 0 && m.off + m.n1 + m.n2 + m.n1 * m.n2 <= src.n;
  const float* lutd = staged ? src.smem : src.gmem;
  if (m.var < 0) {  // no template: a scalar only
    if (m.n1 == 1 && m.n2 == 1) return lutd[m.off + 2];
    return nanf("");
  }
  // var 0: (slew | related) first; var 1: (load | constrained) first
  return m.var == 0 ? lut_eval(m, lutd, a, b) : lut_eval(m, lutd, b, a);
}

// A cell arc's table at a load that is known before the slew: while the
// slew's pin is waited for, the load's segment is found and how far along it
// the load is; what is left for after the wait is the slew's segment (by
// counting, all axis entries in flight at once), four table entries and
// three fused multiply-adds.  In exact arithmetic the same bilinear form as
// lut_eval's, whichever axis comes first; both lines start at the nearer end
// of their segment.  Slew axes of up to kPrepAxis entries; others go through
// timing_value, and so do queries that have no finite answer this way (see
// fprop_warp).  After the wait an arc's two tables take about 250 cycles of
// every gate on a path; interpolating both axes there with lut_eval took 1700
// (six divisions, each with its own branch), and two calls of timing_value
// 3500.  Reducing the tables to the load before the wait leaves one entry
// pair less behind it, but costs 16 shared-memory stores a lane (240k gates
// 1624 us against 1457) and rounds at the full value once more: slews of
// 2k..30k gates 6.1e-8 off 64 bits, against 5.7e-8 here and 5.8e-8 with
// lut_eval.
constexpr int kPrepAxis = 8, kPropT = 256;
struct Prep {
  int n;       // entries of the slew axis; 0: not prepared
  int ax;      // the axis
  int at;      // the entry of the load segment's start, first slew
  int ds, dl;  // steps along slew and load (0: one load entry)
  float f;     // how far along its segment the load is
  bool end;    // measured from the segment's end
};

// Entry i of the library: staged in shared memory, or in global memory.
template <bool kStaged>
__device__ __forceinline__ float lut_at(const LutSrc& src, int i) {
  extern __shared__ float s_lut[];
  if constexpr (kStaged) return s_lut[i];
  else return __ldg(src.gmem + i);
}

template <bool kStaged>
__device__ __forceinline__ Prep prep_lut(const LutSrc& src, const Lut& m, float load) {
  Prep p{0, 0, 0, 0, 0, 0.0f, false};
  const int ns = m.var == 0 ? m.n1 : m.n2, nl = m.var == 0 ? m.n2 : m.n1;
  if (m.n1 < 1 || m.n2 < 1 || m.var < 0 || ns > kPrepAxis || !(fabsf(load) < 3.402823466e+38f))
    return p;
  if (kStaged && (m.off < 0 || m.off + m.n1 + m.n2 + m.n1 * m.n2 > src.n)) return p;
  const int lax = m.off + (m.var == 0 ? m.n1 : 0);
  p.ax = m.off + (m.var == 0 ? 0 : m.n1);
  p.at = m.off + m.n1 + m.n2;
  p.ds = m.var == 0 ? m.n2 : 1;
  p.n = ns;
  if (nl > 1) {
    const int below = lower_bound((kStaged ? src.smem : src.gmem) + lax, nl, load);
    const int a = max(1, min(below, nl - 1));
    const float x1 = lut_at<kStaged>(src, lax + a - 1), x2 = lut_at<kStaged>(src, lax + a);
    const float up = __fsub_rn(load, x1), down = __fsub_rn(load, x2);
    p.dl = m.var == 0 ? 1 : m.n2;
    p.at += (a - 1) * p.dl;
    p.end = up > -down;
    p.f = __fdiv_rn(p.end ? down : up, __fsub_rn(x2, x1));
  }
  return p;
}

// Whether two prepared tables have the same slew axis.
template <bool kStaged>
__device__ __forceinline__ bool same_axis(const LutSrc& src, const Prep& a, const Prep& b) {
  bool same = a.n == b.n;
#pragma unroll
  for (int i = 0; i < kPrepAxis; ++i) {
    const int k = min(i, max(min(a.n, b.n) - 1, 0));
    same = same & (lut_at<kStaged>(src, a.ax + k) == lut_at<kStaged>(src, b.ax + k));
  }
  return same;
}

// The slew's segment on an axis of n entries from ax (its start, 0-based) and
// how far along it the slew is, from the segment's end or start.  No branch
// depends on n, which is 0 without a table: half of a gate's lanes have none
// (the other split's, or the transitions the arc does not make), and branching
// around them cost 1000 cycles per gate.
struct Along {
  int seg;
  float t;
  bool end;
  bool line;  // the entries below the slew are the axis' first ones
};
template <bool kStaged>
__device__ __forceinline__ Along prep_segment(const LutSrc& src, int n, int ax, float slew) {
  if constexpr (!kStaged)
    if (n == 0) return Along{0, 0.0f, false, true};  // there may be no library to read
  const int last = max(n - 1, 0);
  int below = 0;
  bool all = true, gap = false;
#pragma unroll
  for (int i = 0; i < kPrepAxis; ++i) {
    const bool is = (i < n) & (lut_at<kStaged>(src, ax + min(i, last)) < slew);
    below += (int)is;
    gap = gap | (is & !all);
    all = is;
  }
  Along s;
  s.line = !gap;
  s.seg = max(0, min(below, last) - 1);
  const float x1 = lut_at<kStaged>(src, ax + s.seg);
  const float x2 = lut_at<kStaged>(src, ax + min(s.seg + 1, last));
  const float up = __fsub_rn(slew, x1), down = __fsub_rn(slew, x2);
  s.end = up > -down;
  s.t = __fdiv_rn(n > 1 ? (s.end ? down : up) : 0.0f, n > 1 ? __fsub_rn(x2, x1) : 1.0f);
  return s;
}

template <bool kStaged>
__device__ __forceinline__ float prep_value(const LutSrc& src, const Prep& p, const Along& s) {
  if constexpr (!kStaged)
    if (p.n == 0) return nanf("");
  const int i0 = p.at + s.seg * p.ds, i1 = i0 + (p.n > 1 ? p.ds : 0);
  const float a0 = lut_at<kStaged>(src, i0), b0 = lut_at<kStaged>(src, i0 + p.dl);
  const float a1 = lut_at<kStaged>(src, i1), b1 = lut_at<kStaged>(src, i1 + p.dl);
  // the table and its step along the load at either end of the slew's segment
  const float e0 = p.end ? b0 : a0, e1 = p.end ? b1 : a1;
  const float g0 = __fsub_rn(b0, a0), g1 = __fsub_rn(b1, a1);
  const float e = __fmaf_rn(s.t, __fsub_rn(e1, e0), s.end ? e1 : e0);
  const float g = __fmaf_rn(s.t, __fsub_rn(g1, g0), s.end ? g1 : g0);
  return p.n > 0 ? __fmaf_rn(p.f, g, e) : nanf("");
}

// RC node of a net arc's sink (arc_node: its local id in the net) as a
// global BFS slot (-1: none)
__device__ __forceinline__ int rc_slot(const G& G_, int arc) {
  const int node = __ldg(G_.g.arc_node + arc);
  if (node < 0) return -1;
  const int b = __ldg(G_.rc.nodes_start + __ldg(G_.g.arc_net + arc));
  return b + __ldg(G_.rc.node2bfs + b + node);
}

constexpr unsigned kPending = 0x7fbadbadu;  // "not yet computed"
constexpr unsigned kEmpty = 0x7fffffffu;    // the stored empty value

__device__ __forceinline__ float canon(float x) { return none(x) ? __uint_as_float(kEmpty) : x; }

__device__ __forceinline__ float ld_relaxed(const float* p) {
  float v;
  asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ float4 ld_relaxed4(const float* p) {
  float4 v;
  asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

__device__ __forceinline__ void st_relaxed(float* p, float v) {
  asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed4(float* p, float a, float b, float c, float d) {
  asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b),
               "f"(c), "f"(d)
               : "memory");
}

// Bounded wait of a whole warp: load() reads a lane's words again, pending()
// says whether one of them is still not computed.  False (in every lane)
// when this or another wait gave up.  The lanes wait together: lanes that
// went on alone as their values came in would run the code after the wait
// one group after another, the last to come behind all others.  Each poll
// is one L2 round trip: the abort flag and the clock are read on every 8th
// poll only, and no poll sleeps, since a sleeping warp sees a new value
// only after it wakes.
template <class LoadF, class PendF>
__device__ __forceinline__ bool wait_warp(LoadF load, PendF pending, GridCtl* c) {
  load();
  if (!__any_sync(FULL, pending())) return true;
  const unsigned long long t0 = gtime();
  for (int k = 0;; ++k) {
    if (pending()) load();
    if (!__any_sync(FULL, pending())) return true;
    if ((k & 7) != 7) continue;
    const bool late = gtime() - t0 > kGridWaitNs;
    if (late) {
      atomicExch(&c->abort, 1);
      atomicCAS(&c->status, 0, (int)OTG_ERR_TIMEOUT);
    }
    if (__any_sync(FULL, late || *(volatile int*)&c->abort)) return false;
  }
}

__device__ __forceinline__ bool is_pending(float x) { return __float_as_uint(x) == kPending; }

// Until *p and *q hold computed values in the lanes that are `on`.
__device__ __forceinline__ bool wait_values(bool on, const float* p, const float* q, float& x,
                                            float& y, GridCtl* c) {
  x = y = 0.0f;
  return wait_warp(
      [&] {
        if (!on) return;
        x = ld_relaxed(p);
        y = ld_relaxed(q);
      },
      [&] { return is_pending(x) || is_pending(y); }, c);
}
__device__ __forceinline__ bool wait_value(bool on, const float* p, float& x, GridCtl* c) {
  x = 0.0f;
  return wait_warp(
      [&] {
        if (on) x = ld_relaxed(p);
      },
      [&] { return is_pending(x); }, c);
}

// Order-free relax of Pin::_relax_slew/_relax_at (MIN keeps the smallest,
// MAX the largest) and Pin::_relax_rat (the other way round); NaN is the
// empty value and loses to any number.
__device__ __forceinline__ float relax_fwd(int el, float cur, float v) {
  return el == MIN_ ? fminf(cur, v) : fmaxf(cur, v);
}
__device__ __forceinline__ float relax_bwd(int el, float cur, float v) {
  return el == MIN_ ? fmaxf(cur, v) : fminf(cur, v);
}

// What a pin's forward visit reads of each fanin arc, packed by the fill so
// that a visit follows one load instead of a chain of nine (fanin, arc,
// input pin, its net arc, net, node, slot): x the pin to wait on, y the BFS
// slot of the sink whose Elmore values the arc or its input pin adds (-1:
// none), z the arc, w kNetRec for a net arc, else the load's row (-1: none).
//
// A cell arc out of a pin whose only fanin is a net arc (a gate's input
// pin, without assertions) reads through it: the visit waits on the net's
// driver and derives the input pin's slew and arrival time exactly as that
// pin's own visit does.  The input pin still stores its own values; this
// only shortens the chain of waits.  y is kOwnRec for the other cell arcs.
constexpr int kNetRec = -2, kOwnRec = -2;
constexpr int4 kNoRec = {0, -1, 0, kNetRec};

__device__ __forceinline__ bool empty4(const float* p) {
  const float x = __ldg(p), y = __ldg(p + 1), z = __ldg(p + 2), w = __ldg(p + 3);
  return none(x) & none(y) & none(z) & none(w);
}

__device__ int4 fanin_rec(const G& G_, int arc) {
  const otg_prop_graph& g = G_.g;
  int4 r{__ldg(g.arc_from + arc), kOwnRec, arc, kNetRec};
  if (__ldg(g.arc_kind + arc) == 0) {
    r.y = rc_slot(G_, arc);
    return r;
  }
  const int net = __ldg(g.arc_net + arc);
  r.w = net >= 0 ? __ldg(G_.rc.nodes_start + net) : -1;
  const int u = r.x, f = __ldg(g.fanin_start + u);
  if (__ldg(g.fanin_start + u + 1) - f == 1) {
    const int a0 = __ldg(g.fanin + f);
    if (__ldg(g.arc_kind + a0) == 0 && empty4(g.pi_slew + 4 * u) && empty4(g.pi_at + 4 * u)) {
      r.x = __ldg(g.arc_from + a0);
      r.y = rc_slot(G_, a0);
    }
  }
  return r;
}

// A pin a warp is about to visit: its fanin (forward) or fanout range, and
// this lane's record or arc of the first pass.  The warp loads them while
// it waits at the pins before.
struct Visit {
  int v, lo, hi;
  int4 rec;
};

// Forward at pin v (one warp): Timer::_fprop_slew, _fprop_delay, _fprop_at
// and _fprop_test.  Lane j of a pass takes fanin arc j/8 and the combination
// (el, frf, trf) = bits (2, 1, 0) of j; its slew and arrival candidates go to
// output corner (el, trf).  Returns false if a wait gave up.
template <bool kStaged, class AfterF>
__device__ __forceinline__ bool fprop_warp(const G& G_, const int4* rec, const LutSrc& lutd,
                                           const Visit& me, int lane, float* at, float* slew,
                                           float* rat, float* arc_delay, float* test_rat,
                                           GridCtl* ctl, AfterF after) {
  const otg_prop_graph& g = G_.g;
  const int v = me.v;
  const int el = (lane >> 2) & 1, frf = (lane >> 1) & 1, trf = lane & 1;
  const int c_out = 2 * el + trf;
  const int f0 = me.lo, nitems = 8 * (me.hi - f0);
  // a primary input's assertions (NaN: none) seed the lanes with frf 0 of
  // the first pass, one per output corner
  float sl = nanf(""), a = nanf("");
  int last_arc = -1;
  float last_d = 0.0f;
  if (lane < 8 && frf == 0) {
    sl = __ldg(g.pi_slew + 4 * v + c_out);
    a = __ldg(g.pi_at + 4 * v + c_out);
  }
  for (int j0 = 0; j0 < nitems; j0 += 32) {
    const int j = j0 + lane;
    const bool on = j < nitems;  // the last pass may leave lanes without an arc
    const int4 R = j0 == 0 ? me.rec : (on ? __ldg(rec + f0 + (j >> 3)) : kNoRec);
    const int arc = R.z;
    const bool cell = R.w != kNetRec, thru = cell && R.y != kOwnRec;
    float d = nanf(""), so = nanf(""), imp = nanf("");
    Lut ls = no_lut(), ld = no_lut();
    Prep ps{}, pd{};
    bool one_axis = true, slow = false;
    float load = 0.0f;
    // the sink whose Elmore delay and impulse the lane adds: a net arc's
    // (equal transitions only), or the read-through input pin's, at (el, frf)
    const int s = cell ? (thru ? R.y : -1) : (frf == trf ? R.y : -1);
    if (s >= 0) {
      const size_t row = 4 * (size_t)s + 2 * el + frf;
      imp = __ldg(G_.rc.impulse + row);
      d = __ldg(G_.rc.delay + row);
    }
    if (cell) {
      const int t = __ldg(g.arc_timing + 2 * arc + el);
      ls = timing_lut(G_, t, 1, frf, trf);
      ld = timing_lut(G_, t, 0, frf, trf);
      if (R.w >= 0 && t >= 0) load = __ldg(G_.rc.load + 4 * (size_t)R.w + c_out);
      ps = prep_lut<kStaged>(lutd, ls, load);
      pd = prep_lut<kStaged>(lutd, ld, load);
      one_axis = ps.n == 0 || pd.n == 0 || same_axis<kStaged>(lutd, ps, pd);
      slow = (ls.n1 >= 0 && ps.n == 0) || (ld.n1 >= 0 && pd.n == 0);
    }
    // what the code after the wait reads is loaded here (the compiler may
    // otherwise move a load of read-only data down to its use)
    asm volatile("" ::"f"(imp), "f"(d), "f"(sl), "f"(a));
    float si, fa;
    if (!wait_values(on, slew + 4 * R.x + 2 * el + frf, at + 4 * R.x + 2 * el + frf, si, fa, ctl))
      return false;
    // sign(si) * sqrt(si^2 + impulse) at the sink (FlatRct::slew)
    float at_sink = nanf(""), sink = nanf("");
    if (s >= 0 && !none(si)) {
      const float r = sqrtf(__fadd_rn(__fmul_rn(si, si), imp));
      sink = si < 0.0f ? -r : r;
    }
    if (!none(fa) && !none(d)) at_sink = __fadd_rn(d, fa);
    float arr = at_sink;  // what the arc brings to the pin
    if (thru) {
      si = sink;
      fa = at_sink;
    }
    if (!cell) {
      so = sink;
    } else {
      bool line = !slow && fabsf(si) < 3.402823466e+38f;
      if (line) {
        // on the slew table's axis, or the delay table's where there is no other
        Along x = prep_segment<kStaged>(lutd, ps.n ? ps.n : pd.n, ps.n ? ps.ax : pd.ax, si);
        line = x.line;
        so = prep_value<kStaged>(lutd, ps, x);
        if (!one_axis) {
          x = prep_segment<kStaged>(lutd, pd.n, pd.ax, si);
          line = line && x.line;
        }
        d = prep_value<kStaged>(lutd, pd, x);
        line = line && (ps.n == 0 || isfinite(so)) && (pd.n == 0 || isfinite(d));
      }
      // rare: not one straight line for all of the warp's arcs, an axis out of
      // order, or a look-up that met a segment of no length or an entry that is
      // not finite, where the rule's own cases count (a query on an entry)
      if (!line) {
        so = none(si) ? nanf("") : timing_value(lutd, ls, si, load);
        d = none(si) ? nanf("") : timing_value(lutd, ld, si, load);
      }
    }
    if (cell) arr = none(fa) || none(d) ? nanf("") : __fadd_rn(d, fa);
    if (on) {
      sl = relax_fwd(el, sl, so);
      a = relax_fwd(el, a, arr);
    }
    if (j0 + 32 < nitems) {
      if (on) arc_delay[8 * (size_t)arc + (j & 7)] = d;
    } else {  // the last pass's delays are stored behind the pin's values
      last_arc = on ? arc : -1;
      last_d = d;
    }
  }
  // lanes sharing (el, trf) differ in bits 1, 3 and 4
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int m = k == 0 ? 2 : (k == 1 ? 8 : 16);
    sl = relax_fwd(el, sl, __shfl_xor_sync(FULL, sl, m));
    a = relax_fwd(el, a, __shfl_xor_sync(FULL, a, m));
  }
  // corner c's result sits in lane 4 * (c >> 1) + (c & 1), which stores it:
  // that releases the pin's readers.  Then the last arc delays, and the
  // required time is marked pending for the backward pass (both, like the
  // test RATs, are read only after the grid barrier)
  sl = canon(sl);
  a = canon(a);
  if ((lane & ~5) == 0) {
    st_relaxed(slew + 4 * v + c_out, sl);
    st_relaxed(at + 4 * v + c_out, a);
    rat[4 * v + c_out] = __uint_as_float(kPending);
  }
  if (last_arc >= 0) arc_delay[8 * (size_t)last_arc + (lane & 7)] = last_d;
  after();
  // timing tests constrained at v (Test::_fprop_rat): lane j of a pass takes
  // test j/4 and output corner j%4
  const int t0 = __ldg(g.test_start + v), ntest = 4 * (__ldg(g.test_start + v + 1) - t0);
  if (ntest == 0) return true;
  float slc[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) slc[c] = __shfl_sync(FULL, sl, 4 * (c >> 1) + (c & 1));
  for (int j0 = 0; j0 < ntest; j0 += 32) {
    const int j = j0 + lane;
    const bool on = j < ntest;
    const int test = on ? __ldg(g.test_of_pin + t0 + (j >> 2)) : 0;
    const int arc = on ? __ldg(g.test_arc + test) : 0, u = on ? __ldg(g.arc_from + arc) : 0;
    const int tel = (j >> 1) & 1, rf = j & 1;
    const int t = on ? __ldg(g.arc_timing + 2 * arc + tel) : -1;
    float val = nanf("");
    const int edge = t >= 0 ? __ldg(g.timing + 9 * t + 1) : 0;
    const int fel = tel == MIN_ ? MAX_ : MIN_;
    const int rrf = edge == 1 ? RISE_ : FALL_;
    const float csl = slc[2 * tel + rf];
    const bool asks =
        t >= 0 && !none(g.period) && !(rrf == FALL_ && edge != 2) && !none(csl);
    const Lut lc = asks ? timing_lut(G_, t, 2, rrf, rf) : no_lut();
    float rat_at, rsl;
    if (!wait_values(asks, at + 4 * u + 2 * fel + rrf, slew + 4 * u + 2 * fel + rrf, rat_at, rsl,
                     ctl))
      return false;
    if (asks && !none(rat_at) && !none(rsl)) {
      const float related = tel == MIN_ ? rat_at : __fadd_rn(rat_at, g.period);
      const float cons = timing_value(lutd, lc, rsl, csl);
      if (!none(cons)) val = tel == MIN_ ? __fadd_rn(cons, related) : __fsub_rn(related, cons);
    }
    if (on) test_rat[4 * (size_t)test + (j & 3)] = val;
  }
  return true;
}

// MIN: arrival - required; MAX: required - arrival; empty if either is.
__device__ __forceinline__ float slack_of(int c, float at, float rat) {
  if (none(at) || none(rat)) return __uint_as_float(kEmpty);
  return c < 2 ? __fsub_rn(at, rat) : __fsub_rn(rat, at);
}

// The net arcs among a driver's many fanouts, kNetArcs to a lane at a time,
// all four corners of an arc at once (a net arc only relates equal
// transitions).  Eight lanes an arc, as below, hold four arcs in flight: a
// clock driver of 12,000 sinks then takes 3000 rounds of three dependent
// loads, 3.9 ms of a 4.9 ms propagation of 240,000 gates.  *cells: some
// other arc is among them.
constexpr int kNetArcs = 4;
__device__ __forceinline__ bool bprop_net_arcs(const otg_prop_graph& g, int o0, int num, int lane,
                                               const float* rat, const float* arc_delay,
                                               float (&r)[4], bool* cells, GridCtl* ctl) {
  *cells = false;
  for (int j0 = 0; j0 < num; j0 += 32 * kNetArcs) {
    int arc[kNetArcs], w[kNetArcs];
    float4 lo[kNetArcs], hi[kNetArcs], x[kNetArcs];
#pragma unroll
    for (int u = 0; u < kNetArcs; ++u) {
      const int j = j0 + 32 * u + lane;
      arc[u] = j < num ? __ldg(g.fanout + o0 + j) : -1;
    }
#pragma unroll
    for (int u = 0; u < kNetArcs; ++u) {
      w[u] = -1;
      x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (arc[u] < 0) continue;
      if (__ldg(g.arc_kind + arc[u]) == 0) w[u] = __ldg(g.arc_to + arc[u]);
      else *cells = true;
      const float4* d = reinterpret_cast<const float4*>(arc_delay) + 2 * (size_t)arc[u];
      lo[u] = __ldcg(d);
      hi[u] = __ldcg(d + 1);
    }
    auto pend = [](const float4& v) {
      return is_pending(v.x) || is_pending(v.y) || is_pending(v.z) || is_pending(v.w);
    };
    const bool there = wait_warp(
        [&] {
#pragma unroll
          for (int u = 0; u < kNetArcs; ++u)
            if (w[u] >= 0) x[u] = ld_relaxed4(rat + 4 * w[u]);
        },
        [&] {
          bool p = false;
#pragma unroll
          for (int u = 0; u < kNetArcs; ++u) p |= pend(x[u]);
          return p;
        },
        ctl);
    if (!there) return false;
#pragma unroll
    for (int u = 0; u < kNetArcs; ++u) {
      if (w[u] < 0) continue;
      const float wr[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
      const float dl[4] = {lo[u].x, lo[u].w, hi[u].x, hi[u].w};
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (!none(wr[c]) && !none(dl[c]))
          r[c] = relax_bwd(c >> 1, r[c], __fsub_rn(wr[c], dl[c]));
    }
  }
  *cells = __any_sync(FULL, *cells);
  return true;
}

// Backward at pin v (one warp): Timer::_bprop_rat and the slack.  Lanes
// first take the tests constrained at v (4 corners each), then the fanout
// arcs (8 combinations each); every candidate lands in a 4-corner register
// set reduced over the whole warp.  The net arcs of a pin with more fanouts
// than one pass takes go through bprop_net_arcs.
__device__ bool bprop_warp(const G& G_, int v, int lane, const float* at, float* rat, float* slack,
                           const float* arc_delay, const float* test_rat, GridCtl* ctl) {
  const otg_prop_graph& g = G_.g;
  float r[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) r[c] = nanf("");
  const float po = __ldg(g.po_rat + 4 * v + ((lane >> 1) & 3));  // of corner (bits 2, 1)
  const int t0 = __ldg(g.test_start + v), ntest = 4 * (__ldg(g.test_start + v + 1) - t0);
  const int o0 = __ldg(g.fanout_start + v), nout = __ldg(g.fanout_start + v + 1) - o0;
  int nitems = ntest + 8 * nout;
  const bool many = nout > 4;
  if (many) {
    bool cells;
    if (!bprop_net_arcs(g, o0, nout, lane, rat, arc_delay, r, &cells, ctl)) return false;
    if (!cells) nitems = ntest;
  }
  // a single pass of arcs that only propagate: the candidates of corner
  // (split, transition) sit in the lanes that agree in bits 2 and 1
  const bool single = ntest == 0 && nitems <= 32 && !many;
  for (int j0 = 0; j0 < nitems; j0 += 32) {
    const int j = j0 + lane;
    int tc = 0;  // target corner
    float cand = nanf("");
    int mode = 0;  // 0 none, 1 propagation, 2 MIN constraint, 3 MAX constraint
    int wc = 0, w = 0, el = 0, frf = 0, trf = 0;
    float dl = nanf(""), a = nanf(""), wa = nanf("");
    if (j < ntest) {
      tc = j & 3;
      cand = __ldcg(test_rat + 4 * (size_t)__ldg(g.test_of_pin + t0 + (j >> 2)) + tc);
    } else if (j < nitems) {
      const int jj = j - ntest;
      const int arc = __ldg(g.fanout + o0 + (jj >> 3));
      w = __ldg(g.arc_to + arc);
      el = (jj >> 2) & 1;
      frf = (jj >> 1) & 1;
      trf = jj & 1;
      if (__ldg(g.arc_kind + arc) == 0) {
        mode = frf == trf && !many ? 1 : 0;
      } else {
        const int t = __ldg(g.arc_timing + 2 * arc + el);
        if (t >= 0) {
          const int* tr = g.timing + 9 * t;
          if (!__ldg(tr + 2)) mode = 1;
          else if (transition_defined(tr, frf, trf)) mode = el == MIN_ ? 2 : 3;
        }
      }
      // the fanout's required time this combination reads; arc delays and
      // arrival times are final since the forward pass, so they are loaded
      // before the wait and arrive during it
      wc = mode == 1 ? 2 * el + trf : (mode == 2 ? trf : 2 + trf);
      if (mode == 1) {
        dl = __ldcg(arc_delay + 8 * (size_t)arc + 4 * el + 2 * frf + trf);
      } else if (mode != 0) {
        const int ael = mode == 2 ? MAX_ : MIN_, wel = mode == 2 ? MIN_ : MAX_;
        a = __ldcg(at + 4 * v + 2 * ael + frf);
        wa = __ldcg(at + 4 * w + 2 * wel + trf);
      }
    }
    asm volatile("" ::"f"(dl), "f"(a), "f"(wa), "f"(po));
    float wr;
    if (!wait_value(mode != 0, rat + 4 * w + wc, wr, ctl)) return false;
    if (mode == 1) {
      tc = 2 * el + frf;
      if (!none(wr) && !none(dl)) cand = __fsub_rn(wr, dl);
    } else if (mode == 2) {  // hold-like: w's MIN slack moves v's MAX rat
      tc = 2 * MAX_ + frf;
      if (!none(a) && !none(wa) && !none(wr)) cand = __fadd_rn(a, __fsub_rn(wa, wr));
    } else if (mode == 3) {  // setup-like: w's MAX slack moves v's MIN rat
      tc = 2 * MIN_ + frf;
      if (!none(a) && !none(wa) && !none(wr)) cand = __fsub_rn(a, __fsub_rn(wr, wa));
    }
    if (single && !__any_sync(FULL, mode > 1)) {
      const int sel = (lane >> 2) & 1, c = (lane >> 1) & 3;
      float x = cand;
#pragma unroll
      for (int m : {1, 8, 16}) x = relax_bwd(sel, x, __shfl_xor_sync(FULL, x, m));
      if (lane < 8 && (lane & 1) == 0) {
        x = canon(relax_bwd(sel, x, po));
        st_relaxed(rat + 4 * v + c, x);
        slack[4 * v + c] = slack_of(c, __ldcg(at + 4 * v + c), x);
      }
      return true;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (c == tc) r[c] = relax_bwd(c >> 1, r[c], cand);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) r[c] = relax_bwd(c >> 1, r[c], __shfl_xor_sync(FULL, r[c], m));
#pragma unroll
  for (int c = 0; c < 4; ++c) r[c] = relax_bwd(c >> 1, r[c], __shfl_sync(FULL, po, 2 * c));
  if (lane == 0) {
    st_relaxed4(rat + 4 * v, canon(r[0]), canon(r[1]), canon(r[2]), canon(r[3]));
    const float4 a4 = __ldcg(reinterpret_cast<const float4*>(at) + v);
    const float a[4] = {a4.x, a4.y, a4.z, a4.w};
    float sk[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) sk[c] = slack_of(c, a[c], r[c]);
    reinterpret_cast<float4*>(slack)[v] = make_float4(sk[0], sk[1], sk[2], sk[3]);
  }
  return true;
}

// Marks every arrival time and slew pending and clears the control block.
// (pin_group: only the pins whose group is active, see otg_propagate_groups.)
__device__ __forceinline__ bool pin_on(const int32_t* pin_group, const uint8_t* group_active,
                                       int v) {
  return !pin_group || group_active[__ldg(pin_group + v)];
}

// (items: only the listed pins, see otg_propagate_items; num_pins is then
// the list's length.)
__global__ void prop_init_kernel(float4* at, float4* slew, int num_pins, GridCtl* ctl,
                                 const int32_t* pin_group, const uint8_t* group_active,
                                 const int32_t* items, int all_pins, G G_, int4* rec) {
  const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
  const bool all = !items && !pin_group;
  if (all)
    for (int f = i0, n = min(__ldg(G_.g.fanin_start + all_pins), G_.g.num_arcs); f < n;
         f += gridDim.x * blockDim.x)
      rec[f] = fanin_rec(G_, __ldg(G_.g.fanin + f));
  if (i0 == 0 && !items) *ctl = GridCtl{0u, 0u, 0, 0};
  const float p = __uint_as_float(kPending);
  for (int k = i0; k < num_pins; k += gridDim.x * blockDim.x) {
    const int i = items ? __ldg(items + k) : k;
    if (items && (unsigned)i >= (unsigned)all_pins) {
      atomicCAS(&ctl->status, 0, (int)OTG_ERR_INVALID);  // reported; the passes skip it
      continue;
    }
    if (!pin_on(pin_group, group_active, i)) continue;
    at[i] = make_float4(p, p, p, p);
    slew[i] = make_float4(p, p, p, p);
    if (!all) {
      const int f1 = min(__ldg(G_.g.fanin_start + i + 1), G_.g.num_arcs);
      for (int f = __ldg(G_.g.fanin_start + i); f < f1; ++f)
        rec[f] = fanin_rec(G_, __ldg(G_.g.fanin + f));
    }
  }
}

// The whole propagation in one cooperative launch; warp w of W takes items
// w, w + W, ... of each pass.  kCtas CTAs per SM: where a warp has many
// pins, more warps count (four CTAs, 64 registers: 240k gates 1.34 ms
// against 1.86 with two), where it has few, the chain of waits does (two,
// 90 registers, no spills on it: 2k gates 194 us against 216).
template <int kCtas, bool kStaged>
__global__ void __launch_bounds__(kPropT, kCtas)
    prop_kernel(G G_, const int* order, const int* fwd_order, int num_pins, float* at, float* slew,
                float* rat, float* slack, float* arc_delay, float* test_rat, GridCtl* ctl,
                int lut_smem, const int32_t* pin_group, const uint8_t* group_active,
                const int4* rec) {
  // the library's tables, staged on chip when the caller gave their size
  // and they fit (lut_smem floats)
  extern __shared__ float s_lut[];
  for (int i = threadIdx.x; i < lut_smem; i += blockDim.x) s_lut[i] = __ldg(G_.g.lut_data + i);
  __syncthreads();
  const LutSrc lutd{s_lut, lut_smem, G_.g.lut_data};
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int W = (gridDim.x * blockDim.x) >> 5;
  bool ok = true;
  // the pin of item j (-1: none, a bad item (reported by the fill), or one
  // whose group is off)
  auto pin = [&](const int* list, bool down, int j) {
    if (j >= num_pins) return -1;
    const int v = __ldg(list + (down ? num_pins - 1 - j : j));
    return (unsigned)v < (unsigned)G_.g.num_pins && pin_on(pin_group, group_active, v) ? v : -1;
  };
  auto range = [&](const int* start, Visit& x) {
    x.lo = x.v >= 0 ? __ldg(start + x.v) : 0;
    x.hi = x.v >= 0 ? __ldg(start + x.v + 1) : 0;
  };
  {
    const int* list = fwd_order ? fwd_order : order;
    const bool down = !fwd_order;
    auto first = [&](Visit& x) {
      const int f = x.lo + (lane >> 3);
      x.rec = f < x.hi ? __ldg(rec + f) : kNoRec;
    };
    Visit me, next;
    me.v = pin(list, down, warp);
    range(G_.g.fanin_start, me);
    first(me);
    next.v = pin(list, down, warp + W);
    for (int j = warp; ok && j < num_pins; j += W) {
      const int v2 = pin(list, down, j + 2 * W);
      range(G_.g.fanin_start, next);
      if (me.v >= 0)
        ok = fprop_warp<kStaged>(G_, rec, lutd, me, lane, at, slew, rat, arc_delay, test_rat, ctl,
                                 [&] { first(next); });
      else
        first(next);
      me = next;
      next.v = v2;
    }
  }
  // the barrier also lets every CTA leave together when a wait gave up
  if (!grid_barrier(ctl) || !ok) return;
  for (int j = warp; ok && j < num_pins; j += W) {
    const int v = __ldg(order + j);
    if ((unsigned)v >= (unsigned)G_.g.num_pins) continue;
    if (!pin_on(pin_group, group_active, v)) continue;
    ok = bprop_warp(G_, v, lane, at, rat, slack, arc_delay, test_rat, ctl);
  }
}

size_t align256p(size_t x) { return (x + 255) & ~(size_t)255; }

// Tables up to this many floats are staged in shared memory (40 KB per
// CTA leaves room for the four 256-thread CTAs per SM that the registers
// allow; a library with three drive strengths of its combinational cells
// takes about 33 KB).
constexpr int kLutSmemFloats = 10240;

// Up to this many pins per warp at two CTAs per SM, those are launched
// (2k gates have 2, a 6k-gate block 8: 666 us against 718; 60k gates 69:
// 657 against 645).
constexpr int kFewPins = 32;

struct PropDev {
  int sms = 0;
  bool init = false;
  std::atomic<long long> occ[2];  // per variant, of its last launch: (lut_smem + 1) << 32 | CTAs per SM
};
PropDev g_pdev[64];

}  // namespace
}  // namespace otg

extern "C" {

otg_status otg_prop_workspace_size(int32_t num_pins, int32_t num_arcs, int32_t num_tests,
                                   size_t* bytes) {
  if (!bytes || num_pins < 0 || num_arcs < 0 || num_tests < 0) return OTG_ERR_INVALID;
  *bytes = 256 + otg::align256p(32 * (size_t)num_arcs) + otg::align256p(16 * (size_t)num_tests) +
           otg::align256p(sizeof(int4) * (size_t)num_arcs);
  return OTG_OK;
}

// items (with num_items): propagate only the listed pins, `order` and
// fwd_order unused (see otg_propagate_items).
static otg_status propagate_impl(const otg_prop_graph* g, const otg_prop_rc* rc,
                                 const int32_t* order, const int32_t* fwd_order,
                                 const int32_t* pin_group, const uint8_t* group_active, float* at,
                                 float* slew, float* rat, float* slack, void* workspace,
                                 size_t workspace_bytes, otg_stream_t stream,
                                 const int32_t* items = nullptr, int num_items = 0) {
  if (items) {
    if (num_items < 0) return OTG_ERR_INVALID;
    order = items;
    fwd_order = nullptr;
  }
  if (!g || !rc || !order || !at || !slew || !rat || !slack || !workspace || g->num_pins < 0)
    return OTG_ERR_INVALID;
  // lut_meta rows and the per-pin [4] rows are read and written as 16-byte vectors
  if ((((uintptr_t)g->lut_meta | (uintptr_t)at | (uintptr_t)slew | (uintptr_t)rat |
        (uintptr_t)slack) & 15) != 0 || ((uintptr_t)workspace & 255) != 0)
    return OTG_ERR_INVALID;
  size_t need = 0;
  otg_prop_workspace_size(g->num_pins, g->num_arcs, g->num_tests, &need);
  if (workspace_bytes < need) return OTG_ERR_WORKSPACE;
  const int P = items ? num_items : g->num_pins;  // the items the two passes take
  char* ws = (char*)workspace;
  otg::GridCtl* ctl = (otg::GridCtl*)ws;
  float* arc_delay = (float*)(ws + 256);
  float* test_rat = (float*)(ws + 256 + otg::align256p(32 * (size_t)g->num_arcs));
  cudaStream_t st = (cudaStream_t)stream;
  // with items, the fill may record a bad item, so the control block is
  // cleared before it (without items the fill clears it itself)
  if (items && cudaMemsetAsync(ctl, 0, sizeof(otg::GridCtl), st) != cudaSuccess) return OTG_ERR_CUDA;
  int4* rec = (int4*)((char*)test_rat + otg::align256p(16 * (size_t)g->num_tests));
  otg::G G_{*g, *rc};
  const int work = items || pin_group ? P : std::max(P, (int)g->num_arcs);
  otg::prop_init_kernel<<<std::max(1, std::min(1184, (work + 255) / 256)), 256, 0, st>>>(
      (float4*)at, (float4*)slew, P, ctl, pin_group, group_active, items, g->num_pins, G_, rec);
  otg::count_launch();
  if (cudaGetLastError() != cudaSuccess) return OTG_ERR_CUDA;
  if (P == 0) return OTG_OK;
  int dev = 0;
  cudaGetDevice(&dev);
  otg::PropDev& d = otg::g_pdev[dev & 63];
  if (!d.init) {
    cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
    for (auto k : {otg::prop_kernel<2, true>, otg::prop_kernel<4, true>})
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           4 * otg::kLutSmemFloats);
    d.init = true;
  }
  int lut_smem = g->num_lut_data > 0 && g->num_lut_data <= otg::kLutSmemFloats ? g->num_lut_data : 0;
  const size_t smem = 4 * (size_t)lut_smem;
  const bool few = P <= otg::kFewPins * 2 * d.sms * (otg::kPropT / 32);
  auto kern = lut_smem ? (few ? otg::prop_kernel<2, true> : otg::prop_kernel<4, true>)
                       : (few ? otg::prop_kernel<2, false> : otg::prop_kernel<4, false>);
  long long known = d.occ[few].load(std::memory_order_relaxed);
  if ((known >> 32) != lut_smem + 1) {
    int o = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, otg::kPropT, smem);
    known = ((long long)(lut_smem + 1) << 32) | std::min(o, few ? 2 : 4);
    d.occ[few].store(known, std::memory_order_relaxed);
  }
  const int occ = (int)(known & 0xFFFFFFFFll);
  // every CTA resident (the schedule and the barrier rely on it), no more
  // warps than pins
  const int grid = std::max(1, std::min(d.sms * std::max(occ, 1), (P + 7) / 8));
  int num_pins = P;
  void* args[] = {&G_,       (void*)&order, (void*)&fwd_order, &num_pins,
                  &at,       &slew,         &rat,              &slack,
                  &arc_delay, &test_rat,    &ctl,              &lut_smem,
                  (void*)&pin_group, (void*)&group_active, &rec};
  const cudaError_t e = cudaLaunchCooperativeKernel(
      (const void*)kern, dim3(grid), dim3(otg::kPropT), args, smem, st);
  otg::count_launch();
  if (e != cudaSuccess) {
    cudaGetLastError();
    return OTG_ERR_CUDA;
  }
  return OTG_OK;
}

otg_status otg_propagate(const otg_prop_graph* g, const otg_prop_rc* rc, const int32_t* order,
                         const int32_t* fwd_order, float* at, float* slew, float* rat,
                         float* slack, void* workspace, size_t workspace_bytes,
                         otg_stream_t stream) {
  return propagate_impl(g, rc, order, fwd_order, nullptr, nullptr, at, slew, rat, slack,
                        workspace, workspace_bytes, stream);
}

otg_status otg_propagate_groups(const otg_prop_graph* g, const otg_prop_rc* rc,
                                const int32_t* order, const int32_t* fwd_order,
                                const int32_t* pin_group, const uint8_t* group_active,
                                float* at, float* slew, float* rat, float* slack,
                                void* workspace, size_t workspace_bytes, otg_stream_t stream) {
  if (!pin_group || !group_active) return OTG_ERR_INVALID;
  return propagate_impl(g, rc, order, fwd_order, pin_group, group_active, at, slew, rat, slack,
                        workspace, workspace_bytes, stream);
}

otg_status otg_propagate_items(const otg_prop_graph* g, const otg_prop_rc* rc,
                               const int32_t* items, int32_t num_items, float* at, float* slew,
                               float* rat, float* slack, void* workspace, size_t workspace_bytes,
                               otg_stream_t stream) {
  if (!items && num_items > 0) return OTG_ERR_INVALID;
  if (num_items <= 0) {  // nothing to propagate; the status word still reads OK
    if (num_items < 0 || !workspace) return OTG_ERR_INVALID;
    return cudaMemsetAsync(workspace, 0, sizeof(otg::GridCtl), (cudaStream_t)stream) ==
                   cudaSuccess
               ? OTG_OK
               : OTG_ERR_CUDA;
  }
  return propagate_impl(g, rc, nullptr, nullptr, nullptr, nullptr, at, slew, rat, slack,
                        workspace, workspace_bytes, stream, items, num_items);
}

otg_status otg_prop_arc_delays(const void* workspace, size_t workspace_bytes, int32_t num_arcs,
                               const float** arc_delay) {
  if (!workspace || !arc_delay || num_arcs < 0) return OTG_ERR_INVALID;
  if (workspace_bytes < 256 + 32 * (size_t)num_arcs) return OTG_ERR_WORKSPACE;
  *arc_delay = (const float*)((const char*)workspace + 256);
  return OTG_OK;
}

otg_status otg_prop_status(const void* workspace, otg_stream_t stream) {
  if (!workspace) return OTG_ERR_INVALID;
  otg::GridCtl h;
  if (cudaMemcpyAsync(&h, workspace, sizeof(h), cudaMemcpyDeviceToHost, (cudaStream_t)stream) !=
          cudaSuccess ||
      cudaStreamSynchronize((cudaStream_t)stream) != cudaSuccess) {
    cudaGetLastError();
    return OTG_ERR_CUDA;
  }
  return (otg_status)h.status;
}

}  // extern "C"
