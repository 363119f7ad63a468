// otg_rc_small.cuh -- nets of at most 32 nodes: four lanes per net.
// Included by otg_rc.cu inside its anonymous namespace.
//
// A warp takes eight nets of up to 16 nodes, or four of up to 32, and gives
// each a column of its shared-memory slice: row k, column c at cell
// k * C + c, so whatever rows the nets touch, they stay in their own banks.
// The four lanes of a net move four consecutive nodes or edges at a time
// between HBM and the slice, and take one corner each in the Elmore sweeps.
// BFS (the same in all four lanes): adjacency is one 32-bit mask per node,
// and the next node is the highest id left in the level's mask, which is
// the reference's order (distance asc, local id desc) without a sort; its
// parent is the one neighbour in the previous level's mask.  Elmore: load
// and ldelay add up along descending slots, delay and beta along ascending
// ones, all but ldelay in 64 bits (the path sums in 32 were 12% further off
// than sums over the ancestors in id order).  The sums run in slot order,
// so a net's results depend on that net alone.
//
// Why four lanes: a net of nine nodes keeps nine lanes of a warp busy when
// the warp takes one net, and its sweeps are O(n) shuffles each (337 us for
// 250,000 nets of 2..16 nodes with sinks; now 152 us).  One lane per net
// runs fewer instructions but leaves six warps per SM, too few to hide the
// serial sweeps (261 us).  What bounds it: the load/store unit (15 wavefronts
// per node, 12 of them in shared memory, 85% busy) and the sweeps' latency;
// HBM is at a fifth.
constexpr int kSmallMax = 32;     // largest net: one mask bit per node
constexpr int kSmallCells = 128;  // cells of a warp's slice
constexpr int kSmallCtas = 22;  // one-warp CTAs per SM that the slices allow

struct SmallSlice {
  double sum[kSmallCells][4];  // by slot: load, then delay, then beta
  float4 cap[kSmallCells];     // by local id: cap; then by slot: impulse
  float4 acc[kSmallCells];     // cap * delay by slot, then ldelay
  uint2 meta[kSmallCells];     // by slot: local id | parent id << 8, then acc's byte offset of
                               // the parent's row; resistance to the parent
  uint8_t slot[kSmallCells];   // by local id
  uint8_t sorted[32];          // a batch's lanes by net size
};
// what lies in sum's space before the sweeps
struct SmallTopo {
  int2 ends[kSmallCells];      // by edge
  float res[kSmallCells];      // by edge
  unsigned adj[kSmallCells];   // by local id
};
static_assert(sizeof(SmallTopo) <= sizeof(double) * 4 * kSmallCells, "fits sum");

template <int B>
__device__ __forceinline__ void cp_async(void* s, const void* g) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
  if constexpr (B == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(g) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(sa), "l"(g), "n"(B) : "memory");
}

// One net per lane quad (lanes c, c + 8, c + 16, c + 24 for column c): net
// `net` of a, its nodes [b, b + n), n <= kSmallCells / C; n = 0 for lanes
// without a net.  Every lane of the warp calls it.
template <int C>
__device__ __forceinline__ void rc_nets_small(const RcArgs& a, int net, int b, int n,
                                              SmallSlice& sm) {
  const int lane = threadIdx.x & 31, c = lane & 7, j = lane >> 3;
  const unsigned quad = 0x01010101u << c;
  SmallTopo& tp = *reinterpret_cast<SmallTopo*>(sm.sum);
  const int eb = b - net;
  for (int k = j; k < n; k += 4) {
    const int cell = k * C + c;
    if (k < n - 1) {
      cp_async<8>(&tp.ends[cell], a.edges + eb + k);
      cp_async<4>(&tp.res[cell], a.res + eb + k);
    }
    tp.adj[cell] = 0u;
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int k = j; k < n; k += 4) cp_async<16>(&sm.cap[k * C + c], a.cap + b + k);
  const int root = n > 0 ? a.roots[net] : 0;
  int s0 = 0, s1 = 0, sink = 0;  // the net's sinks; this lane's first
  float4 si = make_float4(0.f, 0.f, 0.f, 0.f);
  if (n > 0 && a.sinks_start) {
    s0 = a.sinks_start[net] + j;
    s1 = a.sinks_start[net + 1];
    si = a.driver_slew[net];
    if (s0 < s1) sink = a.sink_nodes[s0];
  }
  asm volatile("cp.async.commit_group;\n cp.async.wait_group 1;" ::: "memory");
  __syncwarp();
  bool bad = n > 0 && (unsigned)root >= (unsigned)n;
  for (int e = j; e < n - 1; e += 4) {
    const int2 ed = tp.ends[e * C + c];
    if ((unsigned)ed.x >= (unsigned)n || (unsigned)ed.y >= (unsigned)n) {
      bad = true;
      continue;
    }
    atomicOr(&tp.adj[ed.x * C + c], 1u << ed.y);
    atomicOr(&tp.adj[ed.y * C + c], 1u << ed.x);
  }
  if (__ballot_sync(FULL, bad) & quad) {
    if (j == 0) report(a, OTG_ERR_INVALID, net);
    n = 0;
  }
  __syncwarp();
  if (n > 0) {  // BFS
    unsigned vis = 1u << root, left = vis, prev = 0u, cur = vis, next = 0u;
    int k = 0;
    for (; k < n; ++k) {
      if (left == 0u) {
        if (next == 0u) break;
        prev = cur;
        cur = left = next;
        vis |= next;
        next = 0u;
      }
      const int v = 31 - __clz(left);
      left &= ~(1u << v);
      const unsigned ad = tp.adj[v * C + c];
      next |= ad & ~vis;
      const unsigned up = ad & prev;
      sm.meta[k * C + c].x = (unsigned)(v | ((up ? 31 - __clz(up) : v) << 8));
      sm.slot[v * C + c] = (uint8_t)k;
    }
    if (k < n) {  // n - 1 edges and a node out of reach
      if (j == 0) report(a, OTG_ERR_NOT_TREE, net);
      n = 0;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  for (int e = j; e < n - 1; e += 4) {
    const int2 ed = tp.ends[e * C + c];
    const int sx = sm.slot[ed.x * C + c], sy = sm.slot[ed.y * C + c];
    const bool down = sx < sy;  // the later slot is the child
    sm.meta[(down ? sy : sx) * C + c].y = __float_as_uint(tp.res[e * C + c]);
    a.edges[eb + e] = down ? ed : make_int2(ed.y, ed.x);
  }
  __syncwarp();
  for (int k = j; k < n; k += 4) {
    const int cell = k * C + c;
    const unsigned o = sm.meta[cell].x;
    const int v = (int)(o & 255u), ps = sm.slot[(o >> 8) * C + c];
    a.node2bfs[b + v] = k;
    a.pid[b + k] = k - ps;  // root: 0
    sm.meta[cell].x = (unsigned)(ps * C * 16);
    const float4 x = sm.cap[v * C + c];
    sm.acc[cell] = x;
    double2* d = reinterpret_cast<double2*>(sm.sum[cell]);
    d[0] = make_double2(x.x, x.y);
    d[1] = make_double2(x.z, x.w);
  }
  __syncwarp();
  // Elmore: lane j of the quad is corner j
  char* const cap = reinterpret_cast<char*>(sm.cap + c) + 4 * j;
  char* const acc = reinterpret_cast<char*>(sm.acc + c) + 4 * j;
  char* const sum = reinterpret_cast<char*>(&sm.sum[c][j]);
  auto f32 = [](char* col, unsigned off) -> float& { return *reinterpret_cast<float*>(col + off); };
  auto f64 = [](char* col, unsigned off) -> double& { return *reinterpret_cast<double*>(col + off); };
  constexpr unsigned R = 16 * C;  // bytes per row of acc and cap; sum has twice that
  {
    const uint2* mp = sm.meta + c + (n - 1) * C;
    unsigned o = (n - 1) * R;
    for (int k = n - 1; k > 0; --k, mp -= C, o -= R) {
      const unsigned p = 2 * mp->x;
      f64(sum, p) = __dadd_rn(f64(sum, p), f64(sum, 2 * o));
    }
  }
  auto rows = [&](float4* out) {  // sum's rows to HBM
    __syncwarp();
    for (int k = j; k < n; k += 4) {
      const double2* d = reinterpret_cast<const double2*>(sm.sum[k * C + c]);
      const double2 x = d[0], y = d[1];
      out[b + k] = make_float4((float)x.x, (float)x.y, (float)y.x, (float)y.y);
    }
    __syncwarp();
  };
  rows(a.load);
  if (n > 0) {
    f64(sum, 0) = 0.0;
    f32(acc, 0) = __fmul_rn(f32(acc, 0), 0.0f);  // cap * delay at the root; not 0 for every cap
  }
  {
    const uint2* mp = sm.meta + c + C;
    unsigned o = R;
    for (int k = 1; k < n; ++k, mp += C, o += R) {
      const uint2 mt = *mp;
      const double d = __fma_rn((double)__uint_as_float(mt.y), f64(sum, 2 * o),
                                f64(sum, 2 * mt.x));
      f32(acc, o) = (float)__dmul_rn((double)f32(acc, o), d);
      f64(sum, 2 * o) = d;
    }
  }
  rows(a.delay);
  {
    const uint2* mp = sm.meta + c + (n - 1) * C;
    unsigned o = (n - 1) * R;
    for (int k = n - 1; k > 0; --k, mp -= C, o -= R) {
      const unsigned p = mp->x;
      f32(acc, p) = __fadd_rn(f32(acc, p), f32(acc, o));
    }
  }
  if (n > 0) f32(cap, 0) = 0.0f;
  {
    const uint2* mp = sm.meta + c + C;
    unsigned o = R;
    for (int k = 1; k < n; ++k, mp += C, o += R) {
      const uint2 mt = *mp;
      const double beta = __fma_rn((double)__uint_as_float(mt.y), (double)f32(acc, o),
                                   f64(sum, 2 * mt.x));
      const float d = (float)f64(sum, 2 * o);
      f64(sum, 2 * o) = beta;
      f32(cap, o) = __fmaf_rn(-d, d, 2.0f * (float)beta);
    }
  }
  __syncwarp();
  for (int k = j; k < n; k += 4) {
    a.ldelay[b + k] = sm.acc[k * C + c];
    a.impulse[b + k] = sm.cap[k * C + c];
  }
  if (n > 0) {
    for (int k = s0; k < s1; k += 4) {
      const int v = k == s0 ? sink : a.sink_nodes[k];
      if ((unsigned)v >= (unsigned)n) {
        report(a, OTG_ERR_INVALID, net);
        continue;
      }
      const float4 iv = sm.cap[sm.slot[v * C + c] * C + c];
      a.sink_slew[k] = make_float4(sink_slew1(si.x, iv.x), sink_slew1(si.y, iv.y),
                                   sink_slew1(si.z, iv.z), sink_slew1(si.w, iv.w));
    }
  }
  __syncwarp();  // the slice takes the next nets
}

// The nets of the list (list, *count), or, with no list, every item of a
// job whose nets all have at most kSmallMax nodes.  One warp per CTA; each
// takes an equal run of the items, 32 at a time, eight by eight in order of
// net size (a warp's sweeps last as long as its largest net: sizes 2..16
// in order of the list leave 42% of the lanes idle).
__global__ void __launch_bounds__(32) rc_small_kernel(RcJob job, const int* list,
                                                      const int* count, int cap,
                                                      int max_net_nodes, int* status) {
  __shared__ SmallSlice sm;
  const int lane = threadIdx.x, c = lane & 7;
  const int cnt = list ? *count : min(job_count(job), cap);
  if (!list && blockIdx.x == 0 && lane == 0) check_job_count(job, cap, status);
  const int per = (cnt + gridDim.x - 1) / gridDim.x;
  const int end = min(cnt, (int)(blockIdx.x + 1) * per);
  for (int g = blockIdx.x * per; g < end; g += 32) {
    int f = 0, net = 0, b = 0, n = 0;
    if (g + lane < end) {
      const int i = list ? list[g + lane] : g + lane;
      job_item(job, i, f, net);
      const RcArgs& a = job_forest(job, f);
      n = max(0, list ? job_net_size(a, net) : checked_net_size(a, net, i, max_net_nodes, status));
      if (n > 0) b = a.nodes_start[net];
    }
    // rank by (size descending, lane): the lanes of a larger size, then the
    // lower lanes of the same one
    unsigned same = FULL;
    int rank = 0;
#pragma unroll
    for (int bit = 5; bit >= 0; --bit) {
      const unsigned on = __ballot_sync(FULL, (n >> bit) & 1);
      if ((n >> bit) & 1) {
        same &= on;
      } else {
        rank += __popc(same & on);
        same &= ~on;
      }
    }
    rank += __popc(same & ((1u << lane) - 1u));
    sm.sorted[rank] = (uint8_t)lane;
    __syncwarp();
    const int places = __popc(__ballot_sync(FULL, n > 0));
    int width;
    for (int at = 0; at < places; at += width) {
      // eight nets, or four when the largest left has more than 16 nodes
      const int src = sm.sorted[min(at + c, 31)];
      const int most = __shfl_sync(FULL, n, sm.sorted[at]);
      width = most <= kSmallCells / 8 ? 8 : 4;
      const int f1 = __shfl_sync(FULL, f, src), net1 = __shfl_sync(FULL, net, src);
      const int b1 = __shfl_sync(FULL, b, src), n1 = __shfl_sync(FULL, n, src);
      const int ns = c < width && at + c < places ? n1 : 0;
      if (width == 8) rc_nets_small<8>(job_forest(job, f1), net1, b1, ns, sm);
      else rc_nets_small<4>(job_forest(job, f1), net1, b1, ns, sm);
    }
    __syncwarp();  // sorted is written again
  }
  chain_end();
}
