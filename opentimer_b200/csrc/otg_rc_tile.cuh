// otg_rc_tile.cuh -- the block path of the fused RC pass: one CTA per net,
// the whole net staged in shared memory with 16-bit indices.  Included by
// otg_rc.cu inside its anonymous namespace (it uses RcArgs, report(),
// block_radix_sort, the fixed-point helpers and the splitter hash there).
//
// Replaces, per net, compute_net_bfs + block_couting_sort
// (ot/cuda/rct.cu:120-245, ot/cuda/sort.cuh:63-142), prepare_res_cap
// (rct.cu:314-359) and compute_net_timing (rct.cu:11-59).
//
// Topology (T1-T7) works edge by edge and needs no adjacency list:
//   T1  edges in (validated), packed 16-bit degree counters by atomics;
//   T2  degree scan -> each node's arc range [off(v), off(v+1));
//   T3  one atomic per arc end places the arc in its node's range, and
//       since the twin's place is known in the same step, the Euler-tour
//       successor follows at once: after (x->y) comes y's next arc after
//       (y->x), cyclically; the arc before the root's first arc is cut;
//   T4  tour ranking: hashed splitter arcs cut the tour into short
//       sublists, one thread walks each, pointer jumping ranks them;
//   T5  per edge, the arc of lower rank is the down arc: parent, child,
//       the child's tour entry and exit; the directed edge goes out;
//   T6  a bitmap of down-arc positions and its popcount prefix give each
//       child's preorder number (down arcs up to its entry) and depth
//       (downs - ups up to it); subtree size is half the entry/exit span;
//   T7  BFS slots: stable radix sort by depth of the ids in descending
//       order, the reference's (distance asc, local id desc) rule
//       (sort.cuh:102-121); node2bfs, pid.
// Elmore, one corner pair at a time, with exact int64 fixed-point sums
// (fx_scale): load and ldelay are subtree sums, taken as differences of an
// exclusive prefix over the preorder; delay and beta are path sums, taken as
// the prefix over the preorder less the prefix over the postorder of the
// nodes left before (a node's term goes straight to its postorder place
// i - depth + size - 1).  That is two prefixes of n terms read in order,
// where a signed prefix over the Euler tour gathers 2(n-1) terms by index
// twice over (2049..4096 nodes: 6.25 -> 6.65 nodes/ns, 81 -> 77 warp
// instructions and 28.8 -> 26 shared-memory wavefronts per node).  What
// bounds the kernel is the load/store unit, 61% busy over all phases and
// barriers; HBM is at 12%.
// Every scan is one tile: thread t owns an odd number KE of consecutive
// items (odd, so strided 8- and 16-byte accesses spread over the banks),
// sums them, and the block-wide base comes from the warp totals after a
// single barrier; a second pass over its items emits the prefixes.

// ---- layout -------------------------------------------------------------
struct RcTileLayout {
  // persistent
  uint32_t pre, bpre, nd;
  // topology scratch (T1-T7)
  uint32_t E, PX, deg, off, succ, sidx, subrk, spos, sl, db, dbp, depth, par, slot, rbuf, hist;
  // Elmore (E1-E9), overlaying the topology scratch
  uint32_t X, Y, Ip;
  uint32_t total, ns_cap;
};

__host__ __device__ inline RcTileLayout rc_tile_layout(int n, int T) {
  RcTileLayout l;
  const uint32_t N = (uint32_t)n, M = n > 0 ? (uint32_t)(n - 1) : 0u, A = 2u * M;
  const uint32_t W = (uint32_t)T / 32u;
  l.ns_cap = 2u * (A / (uint32_t)kSplit) + 64u;
  uint32_t o = 0;
#define OTG_AL(x) (((x) + 15u) & ~15u)
#define OTG_TAKE(f, bytes)   \
  do {                       \
    l.f = o;                 \
    o = OTG_AL(o + (bytes)); \
  } while (0)
  OTG_TAKE(pre, 2u * N);
  OTG_TAKE(bpre, 2u * N);
  OTG_TAKE(nd, 8u * N);
  const uint32_t scratch = o;
  // topology
  OTG_TAKE(E, 4u * M);
  OTG_TAKE(PX, 4u * M);
  OTG_TAKE(deg, 4u * ((N + 1u) / 2u));
  OTG_TAKE(off, 2u * (N + 1u));
  OTG_TAKE(succ, 2u * A);  // then the tour rank of every arc
  const uint32_t r1 = o;
  OTG_TAKE(sidx, 2u * A);
  OTG_TAKE(subrk, 4u * A);
  OTG_TAKE(spos, 2u * l.ns_cap);
  OTG_TAKE(sl, 8u * l.ns_cap);
  const uint32_t end_rank = o;
  o = r1;  // after the ranking: bitmap, depth, parent, BFS sort
  OTG_TAKE(db, 4u * ((A + 31u) / 32u));
  OTG_TAKE(dbp, 4u * ((A + 31u) / 32u));
  OTG_TAKE(depth, 2u * N);
  OTG_TAKE(par, 2u * N);
  OTG_TAKE(slot, 2u * N);
  OTG_TAKE(rbuf, 2u * 2u * N);
  OTG_TAKE(hist, 4u * (1u << rc_radix_bits(T)) * W);
  const uint32_t end_topo = o > end_rank ? o : end_rank;
  // Elmore
  o = scratch;
  OTG_TAKE(X, 8u * N);
  OTG_TAKE(Y, 8u * N);
  OTG_TAKE(Ip, 16u * (N + 1u));
#undef OTG_TAKE
#undef OTG_AL
  l.total = end_topo > o ? end_topo : o;
  return l;
}

// ---- scans --------------------------------------------------------------

// Items per thread for a one-tile scan of C items: odd, so that consecutive
// threads' strided accesses of 8- and 16-byte elements fall in different
// banks.
__device__ __forceinline__ int tile_items(int C, int T) {
  const int k = (C + T - 1) / T;
  return k | 1;
}

// Block-wide exclusive scan of one int per thread with a single barrier:
// wt[] (T/32 ints) holds the warps' totals; the caller alternates between
// two wt buffers so that consecutive scans need no barrier in between.
template <int T>
__device__ __forceinline__ int tile_excl_i32(int v, int* wt, int* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int W = T / 32;
  int x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(FULL, x, d);
    if (lane >= d) x += y;
  }
  if (lane == 31) wt[w] = x;
  __syncthreads();
  const int t = lane < W ? wt[lane] : 0;
  const int before = __reduce_add_sync(FULL, lane < w ? t : 0);
  if (total) *total = __reduce_add_sync(FULL, t);
  return before + x - v;
}

// Sum over the warp's lanes (mod 2^64), as three 32-bit reductions of 22,
// 22 and 20 bits a lane.
__device__ __forceinline__ long long warp_sum_ll(long long v) {
  const unsigned long long x = (unsigned long long)v;
  const unsigned lo = __reduce_add_sync(FULL, (unsigned)x & 0x3FFFFFu);
  const unsigned mid = __reduce_add_sync(FULL, (unsigned)(x >> 22) & 0x3FFFFFu);
  const unsigned hi = __reduce_add_sync(FULL, (unsigned)(x >> 44));
  return (long long)(lo + ((unsigned long long)mid << 22) + ((unsigned long long)hi << 44));
}

// Exclusive block base of N int64 values per thread (in: the thread's sums,
// out: the sums of the threads before it), one barrier.  wt holds N*(T/32)
// int64; the caller has a barrier between two uses of it.
template <int T, int N>
__device__ __forceinline__ void tile_excl_i64(long long (&v)[N], long long* wt) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int W = T / 32;
  long long x[N];
#pragma unroll
  for (int j = 0; j < N; ++j) x[j] = v[j];
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    long long y[N];
#pragma unroll
    for (int j = 0; j < N; ++j) y[j] = __shfl_up_sync(FULL, x[j], d);
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] += lane >= d ? y[j] : 0;
  }
  if (lane == 31) {
#pragma unroll
    for (int j = 0; j < N; ++j) wt[N * w + j] = x[j];
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const long long before = lane < w && lane < W ? wt[N * lane + j] : 0;
    v[j] = warp_sum_ll(before) + x[j] - v[j];
  }
}

__device__ __forceinline__ unsigned u16_half(unsigned word, int hi) {
  return hi ? (word >> 16) : (word & 0xFFFFu);
}

// Per-warp max of |v| for non-negative float bit patterns, committed to
// a shared max word.
__device__ __forceinline__ void commit_max(float m, unsigned* dst) {
  const unsigned x = __reduce_max_sync(FULL, __float_as_uint(fabsf(m)));
  if ((threadIdx.x & 31) == 0 && x) atomicMax(dst, x);
}

__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// ---- the net --------------------------------------------------------------
template <int T>
__device__ void rc_net_tile(const RcArgs& a, int net, char* ws, int n, int* sh, long long* shl) {
  using Ix = uint16_t;
  constexpr unsigned NONE = 0xFFFFu;
  constexpr int W = T / 32;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int b = a.nodes_start[net];
  const int m = n - 1, A = 2 * m, eb = b - net;
  const RcTileLayout L = rc_tile_layout(n, T);
  Ix* pre = (Ix*)(ws + L.pre);
  Ix* bpre = (Ix*)(ws + L.bpre);
  uint2* nd = (uint2*)(ws + L.nd);  // by preorder: depth | subtree size << 16, parent resistance
  unsigned* E = (unsigned*)(ws + L.E);
  unsigned* PX = (unsigned*)(ws + L.PX);
  unsigned* deg = (unsigned*)(ws + L.deg);
  Ix* off = (Ix*)(ws + L.off);
  Ix* succ = (Ix*)(ws + L.succ);
  Ix* rank = succ;
  Ix* sidx = (Ix*)(ws + L.sidx);
  unsigned* subrk = (unsigned*)(ws + L.subrk);
  Ix* spos = (Ix*)(ws + L.spos);
  volatile unsigned long long* sl = (volatile unsigned long long*)(ws + L.sl);
  unsigned* db = (unsigned*)(ws + L.db);
  unsigned* dbp = (unsigned*)(ws + L.dbp);
  Ix* depth = (Ix*)(ws + L.depth);
  Ix* par = (Ix*)(ws + L.par);
  Ix* slot = (Ix*)(ws + L.slot);
  Ix* rbuf = (Ix*)(ws + L.rbuf);
  int* hist = (int*)(ws + L.hist);
  float2* X = (float2*)(ws + L.X);
  float2* Y = (float2*)(ws + L.Y);
  longlong2* Ip = (longlong2*)(ws + L.Ip);
  int* wt0 = sh;        // [32] warp totals, ping
  int* wt1 = sh + 32;   // [32] pong
  int* s_flag = sh + 64;
  int* s_ns = sh + 65;
  int* s_maxd = sh + 66;
  int* s_sel = sh + 67;
  unsigned* smx = (unsigned*)(sh + 72);  // [16] float maxima
  const int root = a.roots[net];
  // the forest's pointers in registers (a lives in shared memory)
  int2* __restrict__ g_edges = a.edges;
  const float* __restrict__ g_res = a.res;
  const float2* __restrict__ cap2 = (const float2*)a.cap;

  auto fail = [&]() -> bool {
    __syncthreads();
    const int f = *s_flag;
    if (f && tid == 0) report(a, f, net);
    return f != 0;
  };

  PHASE_BEGIN();
  // ---- T1: edges and degrees
  if (tid == 0) {
    *s_flag = ((unsigned)root >= (unsigned)n) ? OTG_ERR_INVALID : 0;
    *s_ns = 0;
    *s_maxd = 0;
    *s_sel = 0;
  }
  if (tid < 16) smx[tid] = 0u;
  const int NW = (n + 1) >> 1;
  for (int w = tid; w < NW; w += T) deg[w] = 0u;
  // The caps and resistances, read many phases later, into L2: with one or
  // two CTAs on the SM nothing else hides their latency (2049..4096 nodes:
  // 6.65 -> 6.8 nodes/ns; smaller nets: no gain).
  if constexpr (T >= 512) {
    for (int v = 8 * tid; v < n; v += 8 * T) prefetch_l2(a.cap + b + v);
    for (int e = 32 * tid; e < m; e += 32 * T) prefetch_l2(g_res + eb + e);
  }
  __syncthreads();
  for (int e = tid; e < m; e += T) {
    int2 ed = g_edges[eb + e];
    if ((unsigned)ed.x >= (unsigned)n || (unsigned)ed.y >= (unsigned)n) {
      *s_flag = OTG_ERR_INVALID;
      ed = make_int2(0, 0);
    }
    E[e] = (unsigned)ed.x | ((unsigned)ed.y << 16);
    atomicAdd(&deg[ed.x >> 1], 1u << ((ed.x & 1) << 4));
    atomicAdd(&deg[ed.y >> 1], 1u << ((ed.y & 1) << 4));
  }
  if (fail()) return;

  PHASE(0);
  // ---- T2: arc ranges; the counters become placement cursors
  {
    const int KW = tile_items(NW, T);
    const int w0 = tid * KW, w1 = min(w0 + KW, NW);
    int local = 0;
    bool zero = false;
    for (int w = w0; w < w1; ++w) {
      const unsigned d = deg[w];
      const int d0 = (int)(d & 0xFFFFu), d1 = 2 * w + 1 < n ? (int)(d >> 16) : 1;
      zero |= d0 == 0 || d1 == 0;
      local += d0 + (2 * w + 1 < n ? d1 : 0);
    }
    if (zero) *s_flag = OTG_ERR_NOT_TREE;  // a node without an edge
    int run = tile_excl_i32<T>(local, wt0, nullptr);
    for (int w = w0; w < w1; ++w) {
      const unsigned d = deg[w];
      const int o0 = run, o1 = run + (int)(d & 0xFFFFu);
      run = o1 + (2 * w + 1 < n ? (int)(d >> 16) : 0);
      off[2 * w] = (Ix)o0;
      if (2 * w + 1 < n) off[2 * w + 1] = (Ix)o1;
      deg[w] = (unsigned)o0 | ((unsigned)o1 << 16);
    }
    if (tid == 0) off[n] = (Ix)A;
  }
  if (fail()) return;

  PHASE(1);
  // ---- T3: place arcs, Euler-tour successors
  const int head = (int)off[root];
  for (int e = tid; e < m; e += T) {
    const unsigned xy = E[e];
    const int x = (int)(xy & 0xFFFFu), y = (int)(xy >> 16);
    const int px = (int)u16_half(atomicAdd(&deg[x >> 1], 1u << ((x & 1) << 4)), x & 1);
    const int py = (int)u16_half(atomicAdd(&deg[y >> 1], 1u << ((y & 1) << 4)), y & 1);
    int sy = py + 1;
    if (sy == (int)off[y + 1]) sy = (int)off[y];
    int sx = px + 1;
    if (sx == (int)off[x + 1]) sx = (int)off[x];
    succ[px] = (Ix)(sy == head ? (int)NONE : sy);  // after x->y: y's next arc
    succ[py] = (Ix)(sx == head ? (int)NONE : sx);
    PX[e] = (unsigned)px | ((unsigned)py << 16);
  }
  // ---- T4: tour ranking.  Number the splitters (warp-aggregated), walk
  // the sublists, rank the sublists by pointer jumping.
  int ns = 0, sel = 0;
  for (;;) {
    __syncthreads();
    for (int p0 = (tid & ~31); p0 < A; p0 += T) {
      const int p = p0 + lane;
      const bool s = p < A && is_splitter(p, sel, head);
      const unsigned bal = __ballot_sync(FULL, s);
      int base = 0;
      if (lane == 0 && bal) base = atomicAdd(s_ns, __popc(bal));
      base = __shfl_sync(FULL, base, 0);
      if (s) {
        const int id = base + __popc(bal & ((1u << lane) - 1u));
        if (id < (int)L.ns_cap) {
          sidx[p] = (Ix)id;
          spos[id] = (Ix)p;
        }
      }
    }
    __syncthreads();
    ns = *s_ns;
    if (ns <= (int)L.ns_cap) break;
    __syncthreads();
    if (tid == 0) *s_ns = 0;
    ++sel;  // uniform: every thread read the same count
  }
  PHASE(2);
  for (int s = tid; s < ns; s += T) {
    int cur = (int)spos[s];
    unsigned o = 0, next = 0xFFFFFFFFu;
    for (int step = 0; step < A; ++step) {
      subrk[cur] = (unsigned)s | (o << 16);
      ++o;
      const int nx = (int)succ[cur];
      if (nx == (int)NONE) break;
      if (is_splitter(nx, sel, head)) {
        next = (unsigned)sidx[nx];
        break;
      }
      cur = nx;
    }
    sl[s] = sl_pack(next, o);
  }
  __syncthreads();
  PHASE(3);
  {
    int rounds = 1;
    while ((1 << rounds) < ns) ++rounds;
    for (int r = 0; r <= rounds; ++r) {
      for (int s = tid; s < ns; s += T) {
        const unsigned long long p = sl[s];
        if (sl_next(p) != 0xFFFFFFFFu) {
          const unsigned long long q = sl[sl_next(p)];
          sl[s] = sl_pack(sl_next(q), sl_acc(p) + sl_acc(q));
        }
      }
      __syncthreads();
    }
  }
  PHASE(4);
  // the head's chain must be the whole tour (else: a cycle or a second
  // component, i.e. not a tree)
  if (tid == 0) {
    const unsigned long long h = sl[sidx[head]];
    if (sl_next(h) != 0xFFFFFFFFu || sl_acc(h) != (unsigned)A) *s_flag = OTG_ERR_NOT_TREE;
  }
  if (fail()) return;
  for (int p = tid; p < A; p += T) {
    const unsigned sr = subrk[p];
    rank[p] = (Ix)(A - (int)sl_acc(sl[sr & 0xFFFFu]) + (int)(sr >> 16));
  }
  const int NDW = (A + 31) >> 5;
  __syncthreads();
  for (int w = tid; w < NDW; w += T) db[w] = 0u;
  __syncthreads();

  PHASE(5);
  // ---- T5: per edge: down arc, parent/child, entry/exit; directed edge out
  for (int e = tid; e < m; e += T) {
    const unsigned pp = PX[e], xy = E[e];
    const int rx = (int)rank[pp & 0xFFFFu], ry = (int)rank[pp >> 16];
    const int x = (int)(xy & 0xFFFFu), y = (int)(xy >> 16);
    const bool xdown = rx < ry;  // x->y entered y first: x is the parent
    const int par_ = xdown ? x : y, ch = xdown ? y : x;
    const int en = xdown ? rx : ry, ex = xdown ? ry : rx;
    atomicOr(&db[en >> 5], 1u << (en & 31));
    PX[e] = (unsigned)en | ((unsigned)ex << 16);
    E[e] = (unsigned)par_ | ((unsigned)ch << 16);
    g_edges[eb + e] = make_int2(par_, ch);
  }
  __syncthreads();
  PHASE(6);
  // ---- T6: preorder and depth from the down-arc bitmap
  {
    const int KW = tile_items(NDW, T);
    const int w0 = tid * KW, w1 = min(w0 + KW, NDW);
    int local = 0;
    for (int w = w0; w < w1; ++w) local += __popc(db[w]);
    int run = tile_excl_i32<T>(local, wt1, nullptr);
    for (int w = w0; w < w1; ++w) {
      dbp[w] = (unsigned)run;
      run += __popc(db[w]);
    }
  }
  if (tid == 0) {
    pre[root] = 0;
    nd[0] = make_uint2((unsigned)n << 16, 0u);
    depth[root] = 0;
    par[root] = (Ix)root;
  }
  __syncthreads();
  {
    int dmax = 0;
    for (int e = tid; e < m; e += T) {
      const unsigned pp = PX[e], pc = E[e];
      const int en = (int)(pp & 0xFFFFu), ex = (int)(pp >> 16);
      const int ch = (int)(pc >> 16);
      const int downs = (int)dbp[en >> 5] + __popc(db[en >> 5] & (0xFFFFFFFFu >> (31 - (en & 31))));
      const int pv = downs;  // the root is preorder 0
      const int d = 2 * downs - en - 1;
      pre[ch] = (Ix)pv;
      depth[ch] = (Ix)d;
      par[ch] = (Ix)(pc & 0xFFFFu);
      nd[pv] = make_uint2((unsigned)d | (unsigned)((ex - en + 1) >> 1) << 16,
                          __float_as_uint(g_res[eb + e]));
      dmax = max(dmax, d);
    }
    dmax = __reduce_max_sync(FULL, dmax);
    if (lane == 0 && dmax) atomicMax(s_maxd, dmax);
  }
  __syncthreads();
  PHASE(7);
  // ---- T7: BFS slots, the rank under (depth asc, local id desc)
  {
    Ix* nas = bpre;  // BFS slot -> id, then BFS slot -> preorder
    const int maxd = *s_maxd;
    const int NWB = (n + 31) >> 5;  // bitmap words per depth
    const int words = (maxd + 1) * NWB;
    const int region = (int)(L.hist - L.rbuf) + 4 * (1 << rc_radix_bits(T)) * W;
    if (words * 6 <= region) {
      // shallow trees: one bitmap of ids per depth; a node's slot is the
      // number of set bits before it in (depth asc, word desc, bit desc)
      // order: a prefix count per word plus the bits above it in its word
      unsigned* bm = (unsigned*)rbuf;
      Ix* wp = (Ix*)(bm + words);
      for (int k = tid; k < words; k += T) bm[k] = 0u;
      __syncthreads();
      for (int v = tid; v < n; v += T)
        atomicOr(&bm[(int)depth[v] * NWB + (v >> 5)], 1u << (v & 31));
      __syncthreads();
      // flattened order f = d * NWB + (NWB - 1 - w)
      const int KW = tile_items(words, T);
      const int f0 = tid * KW, f1 = min(f0 + KW, words);
      auto word_of = [&](int f) { const int d = f / NWB; return d * NWB + (NWB - 1 - (f - d * NWB)); };
      int local = 0;
      for (int f = f0; f < f1; ++f) local += __popc(bm[word_of(f)]);
      int run = tile_excl_i32<T>(local, wt0, nullptr);
      for (int f = f0; f < f1; ++f) {
        const int k = word_of(f);
        wp[k] = (Ix)run;
        run += __popc(bm[k]);
      }
      __syncthreads();
      for (int v = tid; v < n; v += T) {
        const int k = (int)depth[v] * NWB + (v >> 5);
        const int r = (int)wp[k] + __popc(bm[k] >> (v & 31) >> 1);
        slot[v] = (Ix)r;
        nas[r] = (Ix)v;
      }
    } else {
      // deep trees: stable radix sort by depth of the ids in descending order
      // (the reference's (distance asc, local id desc) rule, sort.cuh:102-121)
      block_radix_sort<T>(
          n, 32 - __clz(max(maxd, 1)), [&](int j) { return (int)depth[n - 1 - j]; }, rbuf,
          rbuf + n, nas, hist, wt0);
      for (int r = tid; r < n; r += T) {
        const int v = n - 1 - (int)nas[r];
        nas[r] = (Ix)v;
        slot[v] = (Ix)r;
      }
    }
    __syncthreads();
    for (int v = tid; v < n; v += T) a.node2bfs[b + v] = (int)slot[v];
    for (int r = tid; r < n; r += T) {
      const int v = (int)nas[r];
      a.pid[b + r] = r == 0 ? 0 : r - (int)slot[par[v]];
      bpre[r] = pre[v];
    }
    __syncthreads();
  }

  PHASE(8);
  // ---- E: Elmore per corner pair
  const int KE = tile_items(n, T);
  const int i0 = tid * KE, i1 = min(i0 + KE, n);
  // f(i) over this thread's items.  One at a time: reading a few items ahead
  // takes 90 registers, and what counts is the number of resident warps.
  auto own = [&](auto f) {
    for (int i = i0; i < i1; ++i) f(i);
  };
  auto res_of = [](uint2 q) { return __uint_as_float(q.y); };
  for (int cp = 0; cp < 2; ++cp) {
    // out[slot] = Y[node]: the pair's half of an output, BFS order
    auto rows_out = [&](float4* rows) {
      float2* out = (float2*)rows;
      for (int r = tid; r < n; r += T) out[2 * (size_t)(b + r) + cp] = Y[bpre[r]];
    };
    if (tid < 6) smx[4 + tid] = 0u;  // the pair's sweep maxima (w, delay, w2)
    // E0: the pair's caps, read once in id order (coalesced), staged by
    // preorder in X, and their maxima
    {
      float m0 = 0.f, m1 = 0.f;
      for (int v = tid; v < n; v += T) {
        const float2 c = cap2[2 * (size_t)(b + v) + cp];
        X[pre[v]] = c;
        m0 = fmaxf(m0, fabsf(c.x));
        m1 = fmaxf(m1, fabsf(c.y));
      }
      commit_max(m0, smx + 2 * cp);
      commit_max(m1, smx + 2 * cp + 1);
    }
    __syncthreads();
    // Ip[i] = exclusive prefix over the preorder of fx(term(i)); Ip[n] = total
    auto pre_scan = [&](auto term, const float (&up)[2], auto after) {
      long long e[2] = {0, 0};
      own([&](int i) {
        const float2 t = term(i);
        e[0] += to_fx(t.x, up[0]);
        e[1] += to_fx(t.y, up[1]);
      });
      tile_excl_i64<T, 2>(e, shl);
      own([&](int i) {
        const float2 t = term(i);
        Ip[i] = make_longlong2(e[0], e[1]);
        e[0] += to_fx(t.x, up[0]);
        e[1] += to_fx(t.y, up[1]);
        if (i == n - 1) Ip[n] = make_longlong2(e[0], e[1]);
        after(i);
      });
      __syncthreads();
    };
    // Y[i] = subtree sum, the prefix's difference over the subtree's range;
    // mx: the maxima of |R * sum|
    auto subtree = [&](const float (&dn)[2], unsigned* mx) {
      float m0 = 0.f, m1 = 0.f;
      own([&](int i) {
        const uint2 q = nd[i];
        const longlong2 lo = Ip[i], hi = Ip[i + (int)(q.x >> 16)];
        const float2 v = make_float2(from_fx(hi.x - lo.x, dn[0]), from_fx(hi.y - lo.y, dn[1]));
        Y[i] = v;
        m0 = fmaxf(m0, fabsf(v.x * res_of(q)));
        m1 = fmaxf(m1, fabsf(v.y * res_of(q)));
      });
      commit_max(m0, mx);
      commit_max(m1, mx + 1);
      __syncthreads();
    };
    // emit(i, s0, s1): the path sum of fx(R * Y) from the root to node i, the
    // prefix over the preorder less that over the nodes left before i is
    // entered (postorder; i - depth of them).  Y goes out to rows on the way.
    auto path = [&](const float (&up)[2], float4* rows, auto emit) {
      auto term = [&](int i, uint2 q) {
        const float2 v = Y[i];
        const float r = res_of(q);
        return i == 0 ? make_longlong2(0, 0)
                      : make_longlong2(to_fx(v.x * r, up[0]), to_fx(v.y * r, up[1]));
      };
      long long e[4] = {0, 0, 0, 0};
      own([&](int i) {
        const uint2 q = nd[i];
        const longlong2 w = term(i, q);
        e[0] += w.x;
        e[1] += w.y;
        // the node's place in the postorder
        Ip[i - (int)(q.x & 0xFFFFu) + (int)(q.x >> 16) - 1] = w;
      });
      rows_out(rows);
      __syncthreads();
      own([&](int i) {
        const longlong2 w = Ip[i];
        e[2] += w.x;
        e[3] += w.y;
      });
      tile_excl_i64<T, 4>(e, shl);
      own([&](int i) {
        const longlong2 w = Ip[i];
        Ip[i] = make_longlong2(e[2], e[3]);
        e[2] += w.x;
        e[3] += w.y;
      });
      __syncthreads();
      own([&](int i) {
        const uint2 q = nd[i];
        const longlong2 left = Ip[i - (int)(q.x & 0xFFFFu)], w = term(i, q);
        e[0] += w.x;
        e[1] += w.y;
        emit(i, e[0] - left.x, e[1] - left.y);
      });
    };
    float up[2], dn[2];
    // load
    fx_scale(__uint_as_float(smx[2 * cp]), n, up[0], dn[0]);
    fx_scale(__uint_as_float(smx[2 * cp + 1]), n, up[1], dn[1]);
    pre_scan([&](int i) { return X[i]; }, up, [](int) {});
    PHASE(10);
    subtree(dn, smx + 4);
    PHASE(11);
    // delay
    fx_scale(__uint_as_float(smx[4]), n, up[0], dn[0]);
    fx_scale(__uint_as_float(smx[5]), n, up[1], dn[1]);
    {
      float m0 = 0.f, m1 = 0.f;
      path(up, a.load, [&](int i, long long s0, long long s1) {
        const float2 d = make_float2(from_fx(s0, dn[0]), from_fx(s1, dn[1]));
        Y[i] = d;
        m0 = fmaxf(m0, fabsf(d.x));
        m1 = fmaxf(m1, fabsf(d.y));
      });
      commit_max(m0, smx + 6);
      commit_max(m1, smx + 7);
    }
    __syncthreads();
    PHASE(13);
    // ldelay (scale from the bound max|cap| * max|delay|); the delay moves to
    // X behind the cap's last use
    fx_scale(__uint_as_float(smx[2 * cp]) * __uint_as_float(smx[6]), n, up[0], dn[0]);
    fx_scale(__uint_as_float(smx[2 * cp + 1]) * __uint_as_float(smx[7]), n, up[1], dn[1]);
    rows_out(a.delay);
    pre_scan([&](int i) { return make_float2(X[i].x * Y[i].x, X[i].y * Y[i].y); }, up,
             [&](int i) { X[i] = Y[i]; });
    PHASE(14);
    subtree(dn, smx + 8);
    PHASE(15);
    // beta -> impulse = 2 beta - delay^2
    fx_scale(__uint_as_float(smx[8]), n, up[0], dn[0]);
    fx_scale(__uint_as_float(smx[9]), n, up[1], dn[1]);
    path(up, a.ldelay, [&](int i, long long s0, long long s1) {
      const float2 d = X[i];
      Y[i] = make_float2(fmaf(-d.x, d.x, 2.0f * from_fx(s0, dn[0])),
                         fmaf(-d.y, d.y, 2.0f * from_fx(s1, dn[1])));
    });
    __syncthreads();
    PHASE(17);
    rows_out(a.impulse);
    if (a.sinks_start) {
      const int s0 = a.sinks_start[net], s1 = a.sinks_start[net + 1];
      const float2 si = ((const float2*)a.driver_slew)[2 * (size_t)net + cp];
      float2* so = (float2*)a.sink_slew;
      for (int k = s0 + tid; k < s1; k += T) {
        const int v = a.sink_nodes[k];
        if ((unsigned)v >= (unsigned)n) {
          report(a, OTG_ERR_INVALID, net);
          continue;
        }
        const float2 iv = Y[pre[v]];
        so[2 * (size_t)k + cp] = make_float2(sink_slew1(si.x, iv.x), sink_slew1(si.y, iv.y));
      }
    }
    PHASE(18);
  }
}
