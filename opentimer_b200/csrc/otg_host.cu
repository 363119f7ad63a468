// otg_host.cu -- host-buffer entry points of libotg: a per-device context
// with cached device buffers, the chunked end-to-end RC pipeline, the
// levelization host path, and the drop-in C++ symbols of OpenTimer's CUDA
// module (see include/otg_compat.hpp).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <functional>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include "../../include/otg.h"
#include "../../include/otg_compat.hpp"
#include "otg_internal.cuh"

namespace otg {

static std::atomic<uint64_t> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

namespace {

// Grow-only device buffer.
struct DBuf {
  void* p = nullptr;
  size_t bytes = 0;
  bool ensure(size_t need) {
    if (need <= bytes) return true;
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    size_t b = std::max<size_t>(need + need / 8, 256);
    if (cudaMalloc(&p, b) != cudaSuccess) { cudaGetLastError(); return false; }
    bytes = b;
    return true;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
  template <class T> T* as() const { return (T*)p; }
};

// Copies between pageable host memory and the device, through a ring of
// pinned slots.  Lane 0, the caller, moves slots over PCIe; the other lanes
// (parked threads) copy between the slots and the caller's buffers, a slice
// at a time.  One thread copying through the driver's own staging, and
// faulting in the caller's fresh pages, is what a pageable cudaMemcpyAsync
// costs: 60,000 nets of 2..16 nodes (15 MB in, 46 MB out) take 10..14 ms into
// fresh buffers and 3.7 ms into used ones that way, 4.2 and 2.4 ms with eight
// lanes on 16 cores.  Only lane 0 calls CUDA: with a stream per lane the calls
// wait for one another (3.5 ms into used buffers).  The ring is 16 MB per
// device, allocated on first use; otg_release_host_context() frees it and
// ends the threads.
constexpr int kLanes = 8, kSlots = 8;
constexpr size_t kSlot = (size_t)2 << 20, kSlice = (size_t)256 << 10;
// Pageable bytes from which threads pay: 10,000 nets (10 MB) take 1.0 ms
// against 3.5; 5,000 (4 MB out) 0.6 ms without the ring.  Smaller buffers than
// kStagedMin are not worth cutting up.
constexpr size_t kStageBytes = (size_t)4 << 20, kStagedMin = (size_t)256 << 10;

// The lanes' threads, parked between calls (starting seven takes as long as
// copying 15 MB); lane 0 is the caller.  One job at a time, under the
// context's lock.
class Team {
 public:
  // f(0) .. f(lanes - 1), fewer where no more threads can be had; false, and
  // nothing run, where none can
  bool run(int lanes, const std::function<void(int)>& f) {
    {
      std::lock_guard<std::mutex> g(m_);
      try {
        while ((int)threads_.size() < lanes - 1)
          threads_.emplace_back(&Team::loop, this, (int)threads_.size() + 1, job_);
      } catch (const std::exception&) {
      }
      lanes = std::min(lanes, (int)threads_.size() + 1);
      if (lanes < 2) return false;
      f_ = &f;
      lanes_ = lanes;
      busy_ = lanes - 1;
      ++job_;
    }
    cv_.notify_all();
    f(0);
    std::unique_lock<std::mutex> g(m_);
    done_.wait(g, [&] { return busy_ == 0; });
    return true;
  }
  void stop() {
    {
      std::lock_guard<std::mutex> g(m_);
      stop_ = true;
    }
    cv_.notify_all();
    for (std::thread& t : threads_) t.join();
    threads_.clear();
    stop_ = false;
  }

 private:
  void loop(int lane, unsigned seen) {
    std::unique_lock<std::mutex> g(m_);
    for (;;) {
      cv_.wait(g, [&] { return stop_ || job_ != seen; });
      if (stop_) return;
      seen = job_;
      if (lane >= lanes_) continue;
      const std::function<void(int)>& f = *f_;
      g.unlock();
      f(lane);
      g.lock();
      if (--busy_ == 0) done_.notify_one();
    }
  }
  std::mutex m_;
  std::condition_variable cv_, done_;
  std::vector<std::thread> threads_;
  const std::function<void(int)>* f_ = nullptr;
  int lanes_ = 0, busy_ = 0;
  unsigned job_ = 0;
  bool stop_ = false;
};

struct Copy {
  void* dst;
  const void* src;
  size_t bytes;
};

struct Stager {
  char* ring = nullptr;  // [kSlots][kSlot]
  Team* team = nullptr;  // never destroyed at exit, where its threads may be parked
  cudaEvent_t moved[kSlots] = {};
  bool ok = false;
  bool ensure() {
    if (ok) return true;
    bool good = true;
    for (cudaEvent_t& e : moved)
      good = good && (e || cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess);
    good = good && (ring || cudaMallocHost((void**)&ring, kSlots * kSlot) == cudaSuccess);
    good = good && (team || (team = new (std::nothrow) Team));
    if (!good) cudaGetLastError();  // the caller copies without the ring
    return ok = good;
  }
  void release() {
    for (cudaEvent_t e : moved)
      if (e) cudaEventSynchronize(e);  // a call that failed may have left copies
    if (team) team->stop();
    if (ring) cudaFreeHost(ring);
    ring = nullptr;
    ok = false;
  }
};

struct RcChunkBufs {
  DBuf ns, edges, roots, res, cap, n2b, pid, load, delay, ldelay, imp, ss, sn, dslew, sslew, ws,
      status;
};

struct Ctx {
  int device = -1;
  bool ok = false;
  cudaStream_t st[2] = {nullptr, nullptr};
  RcChunkBufs rc[2];
  Stager stage;
  DBuf lv_fs, lv_fi, lv_out, lv_f0, lv_order, lv_level, lv_ends, lv_counts, lv_ws;
  std::mutex mu;
};

Ctx g_ctx[64];

Ctx* ctx_get() {
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess) return nullptr;
  Ctx& c = g_ctx[d & 63];
  if (!c.ok) {
    c.device = d;
    if (cudaStreamCreateWithFlags(&c.st[0], cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&c.st[1], cudaStreamNonBlocking) != cudaSuccess)
      return nullptr;
    c.ok = true;
  }
  return &c;
}

__global__ void rebase_kernel(int* a, int count, int base) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) a[i] -= base;
}

#define CK(x)                                 \
  do {                                        \
    if ((x) != cudaSuccess) {                 \
      cudaGetLastError();                     \
      return OTG_ERR_CUDA;                    \
    }                                         \
  } while (0)

// Whether p is ordinary pageable memory (a pinned buffer is copied directly).
bool pageable(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// The copies, in order behind what stream s holds.  On return the caller's
// pageable buffers have been read, or hold what came; the rest is on s, staged
// copies to the device among it: up to kSlots of the ring's slots are still
// being read then, and the next call waits for them.
cudaError_t copy_all(Ctx* c, const std::vector<Copy>& copies, bool to_device, cudaStream_t s) {
  const cudaMemcpyKind kind = to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
  std::vector<const Copy*> staged;
  size_t bytes = 0;
  for (const Copy& k : copies)
    if (k.bytes >= kStagedMin && pageable(to_device ? k.src : k.dst)) {
      staged.push_back(&k);
      bytes += k.bytes;
    }
  if (bytes < kStageBytes || !c->stage.ensure()) staged.clear();
  for (const Copy& k : copies)
    if (k.bytes && std::find(staged.begin(), staged.end(), &k) == staged.end()) {
      const cudaError_t e = cudaMemcpyAsync(k.dst, k.src, k.bytes, kind, s);
      if (e != cudaSuccess) return e;
    }
  if (staged.empty()) return cudaSuccess;
  // parts of at most a slot; every part's slices are numbered in one sequence
  struct Part {
    Copy c;
    int first, slices;  // slice numbers [first, first + slices)
  };
  std::vector<Part> parts;
  int total = 0;
  for (const Copy* k : staged)
    for (size_t o = 0; o < k->bytes; o += kSlot) {
      const size_t n = std::min(kSlot, k->bytes - o);
      const int sl = (int)((n + kSlice - 1) / kSlice);
      parts.push_back({{(char*)k->dst + o, (const char*)k->src + o, n}, total, sl});
      total += sl;
    }
  const int P = (int)parts.size();
  Stager& g = c->stage;
  std::vector<std::atomic<int>> copied(P);  // slices done by the lanes
  std::atomic<int> next{0}, moved{0};       // next slice; parts that crossed PCIe
  std::atomic<int> failed{(int)cudaSuccess};
  auto slot = [&](int p) { return g.ring + (size_t)(p % kSlots) * kSlot; };
  auto until = [&](auto ready) {
    while (!ready() && failed.load() == (int)cudaSuccess) std::this_thread::yield();
    return failed.load() == (int)cudaSuccess;
  };
  // one slice, if it is there to be copied (wait: or as soon as it is)
  auto copy_slices = [&] {
    int p = 0;
    for (int i; (i = next.fetch_add(1)) < total;) {
      while (i >= parts[p].first + parts[p].slices) ++p;
      const Copy& k = parts[p].c;
      // from the device: the part has come; to it: the slot's last part has gone
      const int need = to_device ? p - kSlots + 1 : p + 1;
      if (!until([&] { return moved.load(std::memory_order_acquire) >= need; })) return;
      const size_t o = (size_t)(i - parts[p].first) * kSlice, n = std::min(kSlice, k.bytes - o);
      if (to_device) std::memcpy(slot(p) + o, (const char*)k.src + o, n);
      else std::memcpy((char*)k.dst + o, slot(p) + o, n);
      copied[p].fetch_add(1, std::memory_order_release);
    }
  };
  auto filled = [&](int p) { return copied[p].load(std::memory_order_acquire) == parts[p].slices; };
  auto mover = [&]() -> cudaError_t {
    int issued = 0, came = 0;
    while (came < P) {
      // issue what can be: a filled slot, or one whose last part was copied out
      while (issued < P && issued < came + kSlots &&
             (to_device ? filled(issued) : issued < kSlots || filled(issued - kSlots))) {
        const Copy& k = parts[issued].c;
        cudaError_t e = to_device ? cudaMemcpyAsync(k.dst, slot(issued), k.bytes, kind, s)
                                  : cudaMemcpyAsync(slot(issued), k.src, k.bytes, kind, s);
        if (e == cudaSuccess) e = cudaEventRecord(g.moved[issued % kSlots], s);
        if (e != cudaSuccess) return e;
        ++issued;
      }
      if (came < issued) {
        const cudaError_t e = cudaEventQuery(g.moved[came % kSlots]);
        if (e == cudaSuccess) moved.store(++came, std::memory_order_release);
        else if (e != cudaErrorNotReady) return e;
      }
      if (to_device && issued == P) return cudaSuccess;  // the rest is the stream's
    }
    return cudaSuccess;
  };
  auto lane = [&](int l) {
    if (l > 0) {
      copy_slices();
    } else {
      const cudaError_t e = mover();
      if (e != cudaSuccess) failed.store((int)e);
    }
  };
  for (cudaEvent_t e : g.moved) {  // what the last call left in flight, maybe on another stream
    const cudaError_t err = cudaEventSynchronize(e);
    if (err != cudaSuccess) return err;
  }
  const int hw = (int)std::max(2u, std::thread::hardware_concurrency());
  if (g.team->run(std::min(kLanes, hw), lane)) return (cudaError_t)failed.load();
  for (const Copy* k : staged) {  // no thread to be had
    const cudaError_t e = cudaMemcpyAsync(k->dst, k->src, k->bytes, kind, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Target nodes per chunk: large enough that launch overhead vanishes,
// small enough that two chunks in flight overlap their copies.
constexpr int64_t kChunkNodes = 1 << 25;

otg_status rc_host(const otg_rc_forest* h) {
  if (!h || h->num_nets < 0) return OTG_ERR_INVALID;
  if (h->num_nets == 0) return OTG_OK;
  if (!h->nodes_start || !h->edges || !h->roots || !h->edges_res || !h->nodes_cap ||
      !h->node2bfs || !h->pid || !h->load || !h->delay || !h->ldelay || !h->impulse)
    return OTG_ERR_INVALID;
  const bool sinks = h->sinks_start != nullptr;
  if (sinks && (!h->sink_nodes || !h->driver_slew || !h->sink_slew)) return OTG_ERR_INVALID;
  const int N = h->num_nets;
  const int* ns = h->nodes_start;
  int max_n = 1;
  for (int i = 0; i < N; ++i) {
    const int n = ns[i + 1] - ns[i];
    if (n < 1) return OTG_ERR_INVALID;
    max_n = std::max(max_n, n);
  }
  Ctx* c = ctx_get();
  if (!c) return OTG_ERR_CUDA;
  std::lock_guard<std::mutex> lock(c->mu);
  // chunk plan
  std::vector<int> cut{0};
  while (cut.back() < N) {
    int i = cut.back();
    const int64_t b0 = ns[i];
    while (i < N && (i == cut.back() || (int64_t)ns[i + 1] - b0 <= kChunkNodes)) ++i;
    cut.push_back(i);
  }
  int64_t cap_nodes = 0, cap_nets = 0, cap_sinks = 1;
  for (size_t k = 0; k + 1 < cut.size(); ++k) {
    cap_nodes = std::max<int64_t>(cap_nodes, ns[cut[k + 1]] - ns[cut[k]]);
    cap_nets = std::max<int64_t>(cap_nets, cut[k + 1] - cut[k]);
    if (sinks)
      cap_sinks = std::max<int64_t>(cap_sinks,
                                    h->sinks_start[cut[k + 1]] - h->sinks_start[cut[k]]);
  }
  size_t wsb = 0;
  if (otg_rc_workspace_size((int)cap_nets, max_n, &wsb) != OTG_OK) return OTG_ERR_CUDA;
  const int nbuf = cut.size() > 2 ? 2 : 1;
  for (int k = 0; k < nbuf; ++k) {
    RcChunkBufs& B = c->rc[k];
    const size_t V = (size_t)cap_nodes, M = (size_t)cap_nodes, Nn = (size_t)cap_nets;
    bool ok = B.ns.ensure(4 * (Nn + 1)) && B.edges.ensure(8 * M) && B.roots.ensure(4 * Nn) &&
              B.res.ensure(4 * M) && B.cap.ensure(16 * V) && B.n2b.ensure(4 * V) &&
              B.pid.ensure(4 * V) && B.load.ensure(16 * V) && B.delay.ensure(16 * V) &&
              B.ldelay.ensure(16 * V) && B.imp.ensure(16 * V) && B.ws.ensure(wsb) &&
              B.status.ensure(256);
    if (ok && sinks)
      ok = B.ss.ensure(4 * (Nn + 1)) && B.sn.ensure(4 * (size_t)cap_sinks) &&
           B.dslew.ensure(16 * Nn) && B.sslew.ensure(16 * (size_t)cap_sinks);
    if (!ok) return OTG_ERR_OOM;
  }
  std::vector<int> status((cut.size() - 1) * 2, 0);
  for (size_t k = 0; k + 1 < cut.size(); ++k) {
    RcChunkBufs& B = c->rc[k % nbuf];
    cudaStream_t s = c->st[k % nbuf];
    const int n0 = cut[k], n1 = cut[k + 1], nn = n1 - n0;
    const int v0 = ns[n0], vn = ns[n1] - v0;
    const int e0 = v0 - n0, en = vn - nn;
    int s0 = 0, sn = 0;
    std::vector<Copy> in{{B.ns.p, ns + n0, 4 * (size_t)(nn + 1)},
                         {B.edges.p, h->edges + e0, 8 * (size_t)en},
                         {B.roots.p, h->roots + n0, 4 * (size_t)nn},
                         {B.res.p, h->edges_res + e0, 4 * (size_t)en},
                         {B.cap.p, h->nodes_cap + 4 * (size_t)v0, 16 * (size_t)vn}};
    if (sinks) {
      s0 = h->sinks_start[n0];
      sn = h->sinks_start[n1] - s0;
      in.push_back({B.ss.p, h->sinks_start + n0, 4 * (size_t)(nn + 1)});
      in.push_back({B.sn.p, h->sink_nodes + s0, 4 * (size_t)sn});
      in.push_back({B.dslew.p, h->driver_slew + 4 * (size_t)n0, 16 * (size_t)nn});
    }
    CK(copy_all(c, in, true, s));
    rebase_kernel<<<(nn + 1 + 255) / 256, 256, 0, s>>>(B.ns.as<int>(), nn + 1, v0);
    count_launch();
    otg_rc_forest f{};
    f.num_nets = nn;
    f.total_nodes = vn;
    f.nodes_start = B.ns.as<int>();
    f.edges = B.edges.as<otg_rc_edge>();
    f.roots = B.roots.as<int>();
    f.edges_res = B.res.as<float>();
    f.nodes_cap = B.cap.as<float>();
    f.node2bfs = B.n2b.as<int>();
    f.pid = B.pid.as<int>();
    f.load = B.load.as<float>();
    f.delay = B.delay.as<float>();
    f.ldelay = B.ldelay.as<float>();
    f.impulse = B.imp.as<float>();
    if (sinks) {
      rebase_kernel<<<(nn + 1 + 255) / 256, 256, 0, s>>>(B.ss.as<int>(), nn + 1, s0);
      count_launch();
      f.sinks_start = B.ss.as<int>();
      f.sink_nodes = B.sn.as<int>();
      f.driver_slew = B.dslew.as<float>();
      f.sink_slew = B.sslew.as<float>();
    }
    otg_status st = otg_rc_timing(&f, max_n, B.ws.p, B.ws.bytes, (otg_stream_t)s);
    if (st != OTG_OK) return st;
    CK(cudaMemcpyAsync(&status[2 * k], B.ws.p, 8, cudaMemcpyDeviceToHost, s));
    std::vector<Copy> out{{h->edges + e0, B.edges.p, 8 * (size_t)en},
                          {h->node2bfs + v0, B.n2b.p, 4 * (size_t)vn},
                          {h->pid + v0, B.pid.p, 4 * (size_t)vn},
                          {h->load + 4 * (size_t)v0, B.load.p, 16 * (size_t)vn},
                          {h->delay + 4 * (size_t)v0, B.delay.p, 16 * (size_t)vn},
                          {h->ldelay + 4 * (size_t)v0, B.ldelay.p, 16 * (size_t)vn},
                          {h->impulse + 4 * (size_t)v0, B.imp.p, 16 * (size_t)vn}};
    if (sinks) out.push_back({h->sink_slew + 4 * (size_t)s0, B.sslew.p, 16 * (size_t)sn});
    CK(copy_all(c, out, false, s));
  }
  CK(cudaStreamSynchronize(c->st[0]));
  CK(cudaStreamSynchronize(c->st[1]));
  for (size_t k = 0; k + 1 < cut.size(); ++k)
    if (status[2 * k]) return (otg_status)status[2 * k];
  return OTG_OK;
}

otg_status lv_host(int n, int num_edges, const int* fanin_start, const int* fanin,
                   const int* out_deg, const int* frontier0, int first_size, int* order,
                   int* level, int* level_ends, int* counts) {
  if (n < 0 || num_edges < 0 || first_size < 0 || first_size > n || !counts || !level_ends)
    return OTG_ERR_INVALID;
  if (n > 0 && (!fanin_start || !out_deg || !order || !level || (first_size && !frontier0) ||
                (num_edges && !fanin)))
    return OTG_ERR_INVALID;
  Ctx* c = ctx_get();
  if (!c) return OTG_ERR_CUDA;
  std::lock_guard<std::mutex> lock(c->mu);
  size_t wsb = 0;
  otg_status st = otg_levelize_workspace_size(n, num_edges, &wsb);
  if (st != OTG_OK) return st;
  const size_t N = (size_t)std::max(n, 1);
  if (!(c->lv_fs.ensure(4 * (N + 1)) && c->lv_fi.ensure(4 * (size_t)std::max(num_edges, 1)) &&
        c->lv_out.ensure(4 * N) && c->lv_f0.ensure(4 * N) && c->lv_order.ensure(4 * N) &&
        c->lv_level.ensure(4 * N) && c->lv_ends.ensure(4 * (N + 2)) && c->lv_counts.ensure(64) &&
        c->lv_ws.ensure(wsb)))
    return OTG_ERR_OOM;
  cudaStream_t s = c->st[0];
  CK(cudaMemcpyAsync(c->lv_fs.p, fanin_start, 4 * (size_t)(n + 1), cudaMemcpyHostToDevice, s));
  if (num_edges)
    CK(cudaMemcpyAsync(c->lv_fi.p, fanin, 4 * (size_t)num_edges, cudaMemcpyHostToDevice, s));
  if (n) CK(cudaMemcpyAsync(c->lv_out.p, out_deg, 4 * (size_t)n, cudaMemcpyHostToDevice, s));
  if (first_size)
    CK(cudaMemcpyAsync(c->lv_f0.p, frontier0, 4 * (size_t)first_size, cudaMemcpyHostToDevice, s));
  st = otg_levelize(n, num_edges, c->lv_fs.as<int>(), c->lv_fi.as<int>(), c->lv_out.as<int>(),
                    c->lv_f0.as<int>(), first_size, c->lv_order.as<int>(), c->lv_level.as<int>(),
                    c->lv_ends.as<int>(), c->lv_counts.as<int>(), c->lv_ws.p, c->lv_ws.bytes,
                    (otg_stream_t)s);
  if (st != OTG_OK) return st;
  int hc[2] = {0, 0};
  CK(cudaMemcpyAsync(hc, c->lv_counts.p, 8, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  st = otg_levelize_status(c->lv_ws.p, (otg_stream_t)s);
  if (st != OTG_OK) return st;
  counts[0] = hc[0];
  counts[1] = hc[1];
  if (hc[1]) CK(cudaMemcpyAsync(order, c->lv_order.p, 4 * (size_t)hc[1], cudaMemcpyDeviceToHost, s));
  if (n) CK(cudaMemcpyAsync(level, c->lv_level.p, 4 * (size_t)n, cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(level_ends, c->lv_ends.p, 4 * (size_t)(hc[0] + 1), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  return OTG_OK;
}

}  // namespace
}  // namespace otg

extern "C" {

otg_status otg_rc_timing_host(const otg_rc_forest* host_forest) {
  try {
    return otg::rc_host(host_forest);
  } catch (const std::bad_alloc&) {
    return OTG_ERR_OOM;
  }
}

otg_status otg_levelize_host(int32_t n, int32_t num_edges, const int32_t* fanin_start,
                             const int32_t* fanin, const int32_t* out_deg,
                             const int32_t* frontier0, int32_t first_size, int32_t* order,
                             int32_t* level, int32_t* level_ends, int32_t* counts) {
  return otg::lv_host(n, num_edges, fanin_start, fanin, out_deg, frontier0, first_size, order,
                      level, level_ends, counts);
}

void otg_release_host_context(void) {
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess) return;
  otg::Ctx& c = otg::g_ctx[d & 63];
  std::lock_guard<std::mutex> lock(c.mu);
  for (auto& B : c.rc) {
    for (otg::DBuf* b : {&B.ns, &B.edges, &B.roots, &B.res, &B.cap, &B.n2b, &B.pid, &B.load,
                         &B.delay, &B.ldelay, &B.imp, &B.ss, &B.sn, &B.dslew, &B.sslew, &B.ws,
                         &B.status})
      b->release();
  }
  for (otg::DBuf* b : {&c.lv_fs, &c.lv_fi, &c.lv_out, &c.lv_f0, &c.lv_order, &c.lv_level,
                       &c.lv_ends, &c.lv_counts, &c.lv_ws})
    b->release();
  c.stage.release();
}

const char* otg_status_string(otg_status s) {
  switch (s) {
    case OTG_OK: return "ok";
    case OTG_ERR_INVALID: return "invalid argument or id out of range";
    case OTG_ERR_CUDA: return "CUDA runtime error";
    case OTG_ERR_OOM: return "out of memory";
    case OTG_ERR_NOT_TREE: return "RC net is not a spanning tree";
    case OTG_ERR_CYCLE: return "timing graph has a cycle";
    case OTG_ERR_TIMEOUT: return "bounded device wait timed out";
    case OTG_ERR_TOO_LARGE: return "net larger than the workspace was sized for";
    case OTG_ERR_WORKSPACE: return "workspace too small";
    case OTG_ERR_ADMISSION: return "request exceeds the device memory budget";
  }
  return "unknown status";
}

uint64_t otg_kernel_launches(void) { return otg::g_launches.load(); }

}  // extern "C"

// ------------------------------------------------- reference drop-in symbols

void rct_bfs_and_compute_cuda(RctEdgeArrayCUDA d) {
  otg_rc_forest f{};
  f.num_nets = d.num_nets;
  f.total_nodes = d.total_num_nodes;
  f.nodes_start = d.rct_nodes_start;
  f.edges = reinterpret_cast<otg_rc_edge*>(d.rct_edges);
  f.roots = d.rct_roots;
  f.edges_res = d.rct_edges_res;
  f.nodes_cap = d.rct_nodes_cap;
  f.node2bfs = d.rct_node2bfs_order;
  f.pid = d.rct_pid;
  f.load = d.load;
  f.delay = d.delay;
  f.ldelay = d.ldelay;
  f.impulse = d.impulse;
  const otg_status st = otg_rc_timing_host(&f);
  if (st != OTG_OK) std::fprintf(stderr, "rct_bfs_and_compute_cuda: %s\n", otg_status_string(st));
}

void rct_compute_cuda(RctCUDA d) {
  // The tree arrives BFS-ordered (parent of i is i - pid[i]); rebuild it as
  // an edge list with slot ids, run the fused path and map the results back
  // to the caller's order.
  const int N = d.num_nets, V = d.total_num_nodes;
  std::vector<otg_rc_edge> edges((size_t)std::max(V - N, 0));
  std::vector<float> res(edges.size());
  std::vector<int> roots((size_t)N, 0), n2b((size_t)V), pid((size_t)V);
  std::vector<float> out[4];
  for (auto& o : out) o.resize(4 * (size_t)V);
  for (int net = 0; net < N; ++net) {
    const int b = d.rct_nodes_start[net], e = d.rct_nodes_start[net + 1];
    for (int i = b + 1; i < e; ++i) {
      const size_t k = (size_t)(i - net - 1);
      edges[k] = otg_rc_edge{i - b - d.rct_pid[i], i - b};
      res[k] = d.pres[i];
    }
  }
  otg_rc_forest f{};
  f.num_nets = N;
  f.total_nodes = V;
  f.nodes_start = d.rct_nodes_start;
  f.edges = edges.data();
  f.roots = roots.data();
  f.edges_res = res.data();
  f.nodes_cap = d.cap;
  f.node2bfs = n2b.data();
  f.pid = pid.data();
  f.load = out[0].data();
  f.delay = out[1].data();
  f.ldelay = out[2].data();
  f.impulse = out[3].data();
  const otg_status st = otg_rc_timing_host(&f);
  if (st != OTG_OK) {
    std::fprintf(stderr, "rct_compute_cuda: %s\n", otg_status_string(st));
    return;
  }
  float* dst[4] = {d.load, d.delay, d.ldelay, d.impulse};
  for (int net = 0; net < N; ++net) {
    const int b = d.rct_nodes_start[net], e = d.rct_nodes_start[net + 1];
    for (int i = b; i < e; ++i)
      for (int q = 0; q < 4; ++q)
        std::memcpy(dst[q] + 4 * (size_t)i, out[q].data() + 4 * (size_t)(b + n2b[i]),
                    4 * sizeof(float));
  }
}

void toposort_compute_cuda(int n, int num_edges, int first_size, int* edgelist_start,
                           int* edgelist, int* out, int* frontiers,
                           std::vector<int>& frontiers_ends) {
  std::vector<int> order((size_t)std::max(n, 1)), level((size_t)std::max(n, 1)),
      ends((size_t)n + 2);
  int counts[2] = {0, 0};
  const otg_status st = otg_levelize_host(n, num_edges, edgelist_start, edgelist, out, frontiers,
                                          first_size, order.data(), level.data(), ends.data(),
                                          counts);
  if (st != OTG_OK) {
    std::fprintf(stderr, "toposort_compute_cuda: %s\n", otg_status_string(st));
    return;
  }
  std::memcpy(frontiers, order.data(), sizeof(int) * (size_t)counts[1]);
  for (int k = 2; k <= counts[0]; ++k) frontiers_ends.push_back(ends[k]);
}
