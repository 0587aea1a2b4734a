// vf_batch.cu -- the batched-ensemble entry points (vf_batch_*) of
// include/volumefluxes_sm103.h.
//
// A batch takes handles that are ready to step and runs the time loop of each
// on the device in k_ensemble (vf_ensemble.cuh): one thread-block cluster per
// simulation, clusters sized from the simulation's tile count, one launch per
// (precision, cluster size) group on its own stream so the groups overlap.
// Simulations are ordered largest estimated work first inside a launch, which
// the block scheduler then starts in that order (longest-processing-time
// first). Each cluster writes its result and a done flag into pinned, mapped
// host memory, so the host sees every simulation finish without synchronising
// the launch it belongs to.
//
// Mid-size Float64 simulations are stepped together by launches that span them all
// (packs below, vf_pack.cuh).
//
// Other simulations of at least wide_cells interior cells (default 8192 in Float64,
// 65536 in Float32; wide_cells_for) are "wide": a 16-CTA cluster would leave most
// of the GPU to them alone and make them the batch's tail, so they run the plain
// whole-grid step kernels on their handle's stream instead, as the device loop
// of vf_simulate, in chunks of kChunk steps captured once as a CUDA graph.
// kInFlight chunks are kept queued; after each, the step record is copied to pinned
// memory behind an event, and the host retires chunks and enqueues new ones
// whenever the batch is polled. Their kernels share the SMs with the cluster
// launches, and their results are those of vf_simulate.
//
// Nothing here allocates with cudaMalloc, cudaFree or cudaFreeHost, which may
// synchronise the whole device: launch descriptors come from the library's
// stream-ordered pool and result slots from a pinned slab kept for the life of
// the process.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstring>
#include <limits>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "vf_handle.h"

namespace {
// A wide member: the plain device loop on its handle's stream, fed in chunks.
struct Wide {
  int member = 0;
  long long enqueued = 0;      // steps enqueued so far
  long long max_steps = 0;     // the record's limit: the device stops there by itself
  double endtime = 0;
  int head = 0, inflight = 0;  // chunks head .. head+inflight-1 are in flight; chunk c uses ev/rec slot c % 3
  long long chunk_end[3] = {0, 0, 0};
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  bool done = false;
};
// Members stepped together (vf_pack.cuh).
struct Pack {
  std::vector<int> members;     // batch indices, in item order
  std::vector<char> done;
  int live = 0;
  cudaStream_t stream = nullptr;
  vf::PackItem<double>* items = nullptr;
  vf::StepRecord* recs = nullptr;
  vf::PackBlock* map = nullptr;
  int n_blocks = 0;
  int live_at_map = 0;          // members the map holds
  long long enqueued = 0;
  int head = 0, inflight = 0;   // chunks head .. head+inflight-1; chunk c uses ev/report slot c % 3
  long long chunk_end[3] = {0, 0, 0};
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
};
// A slot holds the result a cluster writes (res) and, for wide and packed members,
// the step-record copies of the chunks in flight. A batch keeps its slots' addresses:
// its feeder reads them while other batches take slots from the table.
struct Slot {
  vf::EnsResult res;
  vf::StepRecord rec[3];
};
struct SlotRef {
  Slot* host;
  Slot* dev;  // the same memory's device address
};
}  // namespace

struct vf_batch {
  int device = 0;
  int n = 0;
  std::vector<Wide> wide;
  Pack pack;
  long long max_steps = 0;         // LLONG_MAX: no limit
  std::vector<double> endtime;
  std::chrono::steady_clock::time_point start;
  double time_limit_s = 0;
  std::vector<vf_handle*> hs;
  std::vector<cudaStream_t> streams;
  std::vector<SlotRef> slots;      // result slot of simulation i
  std::vector<char> collected;
  void* items_d[2] = {nullptr, nullptr};  // EnsItem<double>[], EnsItem<float>[]
  int* order_d = nullptr;
  unsigned long long* epoch_d = nullptr;  // watchdog start of the batch
  cudaStream_t setup = nullptr;    // stream of the descriptor copies (streams[0])
  std::mutex mu;                   // wide, pack and the feeder's error
  std::thread feeder;
  int feed_rc = 0;                 // the error that ended the feeder
  std::string feed_err;
  std::atomic<bool> stop{false};   // ends the feeder
  std::string err;
};

namespace {

thread_local std::string g_batch_error;

thread_local bool g_feeding = false;  // this thread is a batch's feeder

int bfail(vf_batch* b, int code, const std::string& msg) {
  if (b) (g_feeding ? b->feed_err : b->err) = msg;
  else g_batch_error = msg;
  return code;
}

// ---- result slots: pinned, device-mapped, never freed ---------------------
constexpr int kSlab = 4096;
std::mutex g_slot_mu;
size_t g_slots = 0;                // in all slabs
std::vector<SlotRef> g_free_slots;  // room for every slot is reserved

int acquire_slots(int n, std::vector<SlotRef>& out, std::string& err) try {
  std::lock_guard<std::mutex> lk(g_slot_mu);
  while ((int)g_free_slots.size() < n) {
    g_free_slots.reserve(g_slots + kSlab);
    void* p = nullptr;
    if (cudaHostAlloc(&p, sizeof(Slot) * kSlab, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      err = "pinned result slab allocation failed";
      return VF_ENOMEM;
    }
    void* d = nullptr;
    if (cudaHostGetDevicePointer(&d, p, 0) != cudaSuccess) {
      cudaGetLastError();
      err = "mapped result slab has no device address";
      return VF_ECUDA;
    }
    g_slots += kSlab;
    for (int i = kSlab - 1; i >= 0; --i)
      g_free_slots.push_back(SlotRef{static_cast<Slot*>(p) + i, static_cast<Slot*>(d) + i});
  }
  out.assign(g_free_slots.end() - n, g_free_slots.end());
  g_free_slots.resize(g_free_slots.size() - n);
  return VF_OK;
} catch (const std::bad_alloc&) {
  err = "no host memory";  // short enough to need none
  return VF_ENOMEM;
}

void release_slots(const std::vector<SlotRef>& s) {
  std::lock_guard<std::mutex> lk(g_slot_mu);
  for (const SlotRef& v : s) g_free_slots.push_back(v);
}

vf::EnsResult* slot_host(const SlotRef& s) { return &s.host->res; }
vf::EnsResult* slot_dev(const SlotRef& s) { return &s.dev->res; }
vf::StepRecord* slot_rec(const SlotRef& s, int k) { return &s.host->rec[k]; }
vf::StepRecord* slot_rec_dev(const SlotRef& s, int k) { return &s.dev->rec[k]; }

int slot_done(const SlotRef& s) { return __atomic_load_n(&slot_host(s)->done, __ATOMIC_ACQUIRE); }

// ---- cluster sizing ---------------------------------------------------------
struct Opts {
  int tiles_per_cta;
  int max_cluster;
  double time_limit_s;
  int seg_rows;  // 0: heuristic
  long long wide_cells;
};

Opts resolve(const vf_batch_options* o) {
  Opts r{4, 16, 600.0, 0, 0};
  if (o) {
    if (o->wide_cells > 0) r.wide_cells = o->wide_cells;
    if (o->wide_cells < 0) r.wide_cells = LLONG_MAX;
    if (o->tiles_per_cta > 0) r.tiles_per_cta = o->tiles_per_cta;
    if (o->max_cluster > 0) r.max_cluster = std::min(16, o->max_cluster);
    if (o->time_limit_s > 0) r.time_limit_s = o->time_limit_s;
    if (o->seg_rows > 0) r.seg_rows = std::min(256, std::max(8, o->seg_rows));
  }
  return r;
}

// Interior cells from which a member runs the whole-grid kernels. It depends on
// the member and the options alone, never on the batch: a Float32 member's bits
// differ between the designs, and its result must not depend on the mix. The
// plain kernels cut a grid into as many blocks as the GPU has room for, where a
// cluster has 16 CTAs at most; clusters win only while members are small and
// many. Makespan in ms, all members whole-grid / this threshold / clusters:
//   Float64 (before packs, below): 20 members of 64-224^2, 8 steps: 2.15 / - /
//   4.0; 8 of 64-160^2: 0.85 / - / 1.75; 200 of 64-256^2, 20 steps: 52 / - / 65;
//   but 200 of 64-80^2, 40 steps: 52 / 42 / 42.
//   Float32, 16 members of 64-448^2, 60 steps: 4.0 / 4.7 / 10.5; 40: 8.6 / 9.5 /
//   11.3; 100, 24 steps: 9.9 / 6.6 / 6.7; 128 of 64-1024^2, 40 steps: 30.5 /
//   28.6 / 29.2 (131072 cells: 7.0, 8.2, -, 28.9).
long long wide_cells_for(const vf_handle* h, const Opts& o) {
  if (h->elem == 4 && !vf::plane_fits_u32(h->af.g)) return 1;  // the clusters' offsets are 32-bit
  if (o.wide_cells > 0) return o.wide_cells;
  return h->elem == 8 ? 8192 : 65536;
}

// Float64 RK2 members of kPackCells interior cells and more are stepped together as
// a pack (vf_pack.cuh) while they are below kAloneCells, where launches of their
// own, with TMA staging, are 4% faster (24 members of 200-500^2 cells, 24 steps:
// 29.6 ms packed up to 512^2, 28.4 ms alone). kPackCells is the smallest size that
// was measured, 64^2, and a pack still wins there: the size at which clusters take
// over is not known, it lies below. A pack takes about 0.1 ms to set up: below
// kPackMembers of them each goes alone. All designs give the same Float64 bits, so
// this may depend on the batch.
// Makespan in ms, pack / all alone / alone from 8192 cells on, clusters below (the
// best of a state's first calls: of the 8 steps the members take four on average):
//   20 members of 64-224^2, 8 steps: 1.84 / 2.21 / 4.15; 64: 4.97 / 6.27 / 8.14;
//   8: 1.12 / 1.09 / 2.17; 4: 0.70 / 0.66 / 1.81; 64 of 64-96^2: 2.53 / 3.75 /
//   3.79; 200 of 64-80^2, 40 steps: 27.8 / 55.7 / 40.6; 4 of those: 2.17 / 1.66 /
//   12.3.
// Forward-Euler and faithful members, and an explicit threshold, are as before.
constexpr long long kPackCells = 4096, kAloneCells = 65536;
constexpr int kPackMembers = 8;

bool packs(const vf_handle* h, const Opts& o) {
  const long long cells = (long long)h->cfg.nx * h->cfg.ny;
  return o.wide_cells == 0 && cells >= kPackCells && cells < kAloneCells && h->elem == 8 && h->ad.rk2 &&
         h->ad.variant == 1 && h->ad.arith == VF_ARITH_REFERENCE;
}

// Kernel design of a cluster member: column marching for Float32 members with wall BCs, linear
// reconstruction and constant sources (0 with RK2, 2 with forward Euler);
// tiles (1) for everything else.
int variant_of(const vf_handle* h) {
  if (h->elem == 4 && h->af.variant == 0 && !h->af.general) return h->af.rk2 ? 0 : 2;
  return 1;
}

// Largest launchable cluster size <= c on the current device.
std::mutex g_fit_mu;
int g_fit[64][2][3][17];  // [device][precision][variant][c]: 0 unknown, else 1 + launchable

int fit_cluster(int device, int real_bytes, int variant, int c) {
  const int pi = real_bytes == 8 ? 0 : 1;
  for (; c > 1; c /= 2) {
    int ok;
    {
      std::lock_guard<std::mutex> lk(g_fit_mu);
      ok = device < 64 ? g_fit[device][pi][variant][c] : 0;
    }
    if (!ok) {
      int nclusters = 0;
      cudaError_t e = real_bytes == 8 ? vf::ensemble_max_clusters_f64(c, variant, &nclusters)
                                      : vf::ensemble_max_clusters_f32(c, variant, &nclusters);
      if (e != cudaSuccess) cudaGetLastError();
      ok = (e == cudaSuccess && nclusters > 0) ? 2 : 1;
      std::lock_guard<std::mutex> lk(g_fit_mu);
      if (device < 64) g_fit[device][pi][variant][c] = ok;
    }
    if (ok == 2) return c;
  }
  return 1;
}

// Rows per strip segment of a marching member: 8 (16 rows measured 4.6 instead
// of 4.1 ms on 32 members of 64-448^2 cells, 8.0 instead of 6.9 on 100).
int seg_rows_for(int fixed) { return fixed > 0 ? fixed : 8; }

int cluster_for(const vf_handle* h, const Opts& o) {
  const long long tiles =
      (long long)((h->cfg.nx + vf::TX - 1) / vf::TX) * ((h->cfg.ny + vf::TY - 1) / vf::TY);
  int c = 1;
  while (c < o.max_cluster && (long long)c * o.tiles_per_cta < tiles) c *= 2;
  return std::min(c, o.max_cluster);
}

template <typename T>
vf::EnsItem<T> make_item(vf_handle* h, const vf::StepArgs<T>& a, double t0, double endtime, int match,
                         double max_ts, long long max_steps, vf::EnsResult* res, unsigned long long* epoch) {
  vf::EnsItem<T> it;
  std::memset(&it, 0, sizeof(it));
  it.g = a.g;
  it.p = a.p;
  it.B = a.B;
  it.U[0] = static_cast<T*>(h->U[0]);
  it.U[1] = static_cast<T*>(h->U[1]);
  it.L = a.L;
  it.S = a.S;
  it.t0 = t0;
  it.endtime = endtime;
  it.max_ts = max_ts;
  it.match_endtime = match ? 1 : 0;
  it.has_max_ts = max_ts >= 0 ? 1 : 0;
  it.rk2 = a.rk2;
  it.max_steps = max_steps > 0 ? max_steps : LLONG_MAX;
  it.res = res;
  it.epoch = epoch;
  return it;
}

// While any thread captures a graph in the global mode, event queries, waits and
// pool allocations of the other threads are refused and end that capture. The calls
// that feed a batch touch its own streams alone, so they opt out for their duration:
// the feeder runs beside whatever its caller does.
struct BesideCaptures {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

void destroy_batch(vf_batch* b) {
  if (!b) return;
  const BesideCaptures beside;
  b->stop = true;
  if (b->feeder.joinable()) b->feeder.join();
  // After an error clusters and chunks may still run: they read the descriptors and
  // write states, result slots and record copies, all handed on below.
  for (cudaStream_t s : b->streams) cudaStreamSynchronize(s);
  for (const Wide& w : b->wide)
    if (!w.done) cudaStreamSynchronize(b->hs[w.member]->stream);  // the handle of one that is done may be gone
  if (b->setup) {
    cudaFreeAsync(b->items_d[0], b->setup);
    cudaFreeAsync(b->items_d[1], b->setup);
    cudaFreeAsync(b->order_d, b->setup);
    cudaFreeAsync(b->epoch_d, b->setup);
  }
  Pack& k = b->pack;
  if (k.stream) {
    cudaStreamSynchronize(k.stream);
    if (k.items) cudaFreeAsync(k.items, k.stream);
    if (k.recs) cudaFreeAsync(k.recs, k.stream);
    if (k.map) cudaFreeAsync(k.map, k.stream);
    cudaStreamDestroy(k.stream);
  }
  for (cudaEvent_t e : k.ev)
    if (e) cudaEventDestroy(e);
  for (cudaStream_t s : b->streams) cudaStreamDestroy(s);
  for (Wide& w : b->wide)
    for (cudaEvent_t e : w.ev)
      if (e) cudaEventDestroy(e);
  release_slots(b->slots);
  delete b;
}

constexpr int kChunk = 16;    // steps per graph launch of a wide member
constexpr int kInFlight = 3;  // chunks kept queued per wide member (rides out host stalls)
constexpr int kPlainChunks = 4;  // chunks a handle runs kernel by kernel before its graph is captured

// How the device loop of a wide or packed member ended, from its record after step k.
int end_status(const vf::StepRecord& r, long long k, long long max_steps, double endtime) {
  if (r.stalled) return vf::kEnsStalled;
  return r.n_done >= max_steps && r.t[k & 1] < endtime ? vf::kEnsMaxSteps : vf::kEnsOk;
}

// Final result of a wide member from the record copy of its last retired chunk.
void wide_finish(vf_batch* b, Wide& w, const vf::StepRecord& r, long long k, int status) {
  vf_handle* h = b->hs[w.member];
  cudaStreamSynchronize(h->stream);  // no-op steps of a chunk still in flight
  vf::EnsResult* res = slot_host(b->slots[w.member]);
  res->t = r.t[k & 1];
  res->last_dt = r.last_dt;
  res->steps = r.n_done;
  res->status = status;
  w.done = true;
  __atomic_store_n(&res->done, 1, __ATOMIC_RELEASE);
}

// Wide marching members that take a wave of the GPU together, as a power of two so
// that chunk graphs are captured anew only when half of them have ended; segment
// lengths do not change a member's bits, so this may depend on the batch. Four at
// most: the launches of more do not run side by side often enough. ms at a cap of
// 1 / 2 / 4 / 8: 16 members of 256-512^2 cells, 60 steps, 6.33 / 5.46 / 5.28 / 6.40;
// 16 of 128-1024^2 9.11 / 8.77 / 8.93 / 9.10; 32 of 64-448^2, 24 steps, 2.50 / 2.47 /
// 2.46 / 2.49.
constexpr int kMarchShare = 4;
int march_share(const vf_batch* b, const vf_handle* h) {
  if (h->elem != 4 || h->af.variant != 0) return 0;
  int live = 0, share = 1;
  for (const Wide& w : b->wide) live += !w.done && b->hs[w.member]->elem == 4 ? 1 : 0;
  while (2 * share <= live && share < kMarchShare) share *= 2;
  return share;
}

int wide_enqueue(vf_batch* b, Wide& w) {
  vf_handle* h = b->hs[w.member];
  // A handle's first chunks are launched kernel by kernel: capturing and
  // instantiating the graph costs as much host time as a few of them. Graph
  // chunks are whole: steps past max_steps find their record inactive.
  const bool graph = (w.enqueued & 1) == 0 && (h->chunk_exec || h->plain_chunks >= kPlainChunks);
  const int n = graph ? kChunk : (int)std::min<long long>(kChunk, w.max_steps - w.enqueued);
  h->plain_chunks += graph ? 0 : 1;
  h->af.share = march_share(b, h);
  const int rc = graph ? vf::handle_enqueue_chunk(h, kChunk) : vf::handle_enqueue_steps(h, w.enqueued, n);
  h->af.share = 0;
  if (rc) return rc;
  w.enqueued += n;
  const int slot = (w.head + w.inflight) % kInFlight;
  cudaError_t e = cudaMemcpyAsync(slot_rec(b->slots[w.member], slot), h->rec, sizeof(vf::StepRecord),
                                  cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaEventRecord(w.ev[slot], h->stream);
  if (e != cudaSuccess) return VF_ECUDA;
  w.chunk_end[slot] = w.enqueued;
  w.inflight += 1;
  return VF_OK;
}

// ---- packs ------------------------------------------------------------------
constexpr int kPackChunk = 8;  // steps per chunk of a pack

// The block map of the pack's live members, uploaded in stream order.
int pack_map(vf_batch* b, Pack& k) try {
  std::vector<vf::PackBlock> map;
  for (size_t i = 0; i < k.members.size(); ++i) {
    if (k.done[i]) continue;
    const vf_config& c = b->hs[k.members[i]]->cfg;
    const int n = vf::pack_blocks(c.nx, c.ny);
    for (int j = 0; j < n; ++j) map.push_back(vf::PackBlock{(int)i, j});
  }
  cudaMemPool_t pool = vf::device_pool(b->device);
  if (k.map) cudaFreeAsync(k.map, k.stream);
  k.map = nullptr;
  k.n_blocks = (int)map.size();
  const size_t bytes = sizeof(vf::PackBlock) * map.size();
  if (!pool || cudaMallocFromPoolAsync(reinterpret_cast<void**>(&k.map), bytes, pool, k.stream) != cudaSuccess)
    return VF_ENOMEM;
  cudaError_t e = cudaMemcpyAsync(k.map, map.data(), bytes, cudaMemcpyHostToDevice, k.stream);
  // the copy reads a pageable host vector: finish it before the vector goes
  if (e == cudaSuccess) e = cudaStreamSynchronize(k.stream);
  k.live_at_map = k.live;
  return e == cudaSuccess ? VF_OK : VF_ECUDA;
} catch (const std::bad_alloc&) {
  return VF_ENOMEM;
}

int pack_enqueue(vf_batch* b, Pack& k) {
  const int n = (int)std::min<long long>(kPackChunk, b->max_steps - k.enqueued);
  const vf::PackMap map{k.map, k.n_blocks};
  const int slot = (k.head + k.inflight) % kInFlight;
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < n && e == cudaSuccess; ++i)
    e = vf::launch_pack_step(k.items, map, (int)((k.enqueued + i) & 1), k.stream);
  if (e == cudaSuccess) e = vf::launch_pack_report(k.items, (int)k.members.size(), slot, k.stream);
  if (e == cudaSuccess) e = cudaEventRecord(k.ev[slot], k.stream);
  if (e != cudaSuccess) return VF_ECUDA;
  for (size_t j = 0; j < k.members.size(); ++j)
    if (!k.done[j]) {  // a member that is done may be gone
      b->hs[k.members[j]]->launches += 2 * n + 1;
      break;
    }
  k.enqueued += n;
  k.chunk_end[slot] = k.enqueued;
  k.inflight += 1;
  return VF_OK;
}

int pack_start(vf_batch* b, Pack& k, const double* t0, int match, double max_ts) try {
  const size_t n = k.members.size();
  cudaMemPool_t pool = vf::device_pool(b->device);
  bool ok = pool && cudaStreamCreateWithFlags(&k.stream, cudaStreamNonBlocking) == cudaSuccess;
  for (cudaEvent_t& e : k.ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  ok = ok && cudaMallocFromPoolAsync(reinterpret_cast<void**>(&k.items), sizeof(vf::PackItem<double>) * n, pool,
                                     k.stream) == cudaSuccess;
  ok = ok && cudaMallocFromPoolAsync(reinterpret_cast<void**>(&k.recs), sizeof(vf::StepRecord) * n, pool, k.stream) ==
                 cudaSuccess;
  if (!ok) return VF_ENOMEM;
  std::vector<vf::StepRecord> recs(n);
  std::vector<vf::PackItem<double>> items(n);
  for (size_t j = 0; j < n; ++j) {
    const int i = k.members[j];
    vf_handle* h = b->hs[i];
    vf::StepRecord& r = recs[j];
    std::memset(&r, 0, sizeof(r));
    r.t[0] = t0[i];
    r.active[0] = t0[i] < b->endtime[i] ? 1 : 0;
    r.match_endtime = match ? 1 : 0;
    r.has_max_ts = max_ts >= 0 ? 1 : 0;
    r.max_ts = max_ts;
    r.endtime = b->endtime[i];
    r.stop_time = std::numeric_limits<double>::infinity();
    r.max_steps = b->max_steps == LLONG_MAX ? 0 : b->max_steps;
    r.stop_stalled = 1;
    vf::PackItem<double>& it = items[j];
    std::memset(&it, 0, sizeof(it));
    it.g = h->ad.g;
    it.p = h->ad.p;
    it.B = h->ad.B;
    it.U[0] = static_cast<double*>(h->U[0]);
    it.U[1] = static_cast<double*>(h->U[1]);
    it.L = h->ad.L;
    it.S = h->ad.S;
    it.rec = k.recs + j;
    for (int c = 0; c < kInFlight; ++c) it.report[c] = slot_rec_dev(b->slots[i], c);
  }
  k.done.assign(n, 0);
  k.live = (int)n;
  ok = cudaMemcpyAsync(k.items, items.data(), sizeof(vf::PackItem<double>) * n, cudaMemcpyHostToDevice, k.stream) ==
       cudaSuccess;
  ok = ok && cudaMemcpyAsync(k.recs, recs.data(), sizeof(vf::StepRecord) * n, cudaMemcpyHostToDevice, k.stream) ==
                 cudaSuccess;
  if (!ok) return VF_ECUDA;
  if (int rc = pack_map(b, k)) return rc;  // waits for the copies above too
  for (int c = 0; c < kInFlight && k.enqueued < b->max_steps; ++c)
    if (int rc = pack_enqueue(b, k)) return rc;
  return VF_OK;
} catch (const std::bad_alloc&) {
  return VF_ENOMEM;
}

void pack_finish(vf_batch* b, Pack& k, size_t j, const vf::StepRecord& r, long long end, int status) {
  vf::EnsResult* res = slot_host(b->slots[k.members[j]]);
  res->t = r.t[end & 1];
  res->last_dt = r.last_dt;
  res->steps = r.n_done;
  res->status = status;
  k.done[j] = 1;
  k.live -= 1;
  __atomic_store_n(&res->done, 1, __ATOMIC_RELEASE);
}

// Retires the pack's finished chunks and keeps kInFlight queued.
int pack_pump(vf_batch* b, Pack& k, bool late) {
  while (k.inflight > 0) {
    const int slot = k.head % kInFlight;
    const cudaError_t q = cudaEventQuery(k.ev[slot]);
    if (q == cudaErrorNotReady) break;
    if (q != cudaSuccess) return bfail(b, VF_ECUDA, std::string("pack: ") + cudaGetErrorString(q));
    const long long end = k.chunk_end[slot];
    k.head += 1;
    k.inflight -= 1;
    for (size_t j = 0; j < k.members.size(); ++j) {
      if (k.done[j]) continue;
      const int i = k.members[j];
      const vf::StepRecord& r = *slot_rec(b->slots[i], slot);
      if (!r.active[end & 1])
        pack_finish(b, k, j, r, end, end_status(r, end, b->max_steps, b->endtime[i]));
      else if (late && k.inflight == 0)
        pack_finish(b, k, j, r, end, vf::kEnsTimeout);
    }
  }
  if (k.live == 0 || late) return VF_OK;
  if (2 * k.live <= k.live_at_map)  // half of the members have ended: drop their blocks
    if (int rc = pack_map(b, k)) return bfail(b, rc, "pack map");
  while (k.inflight < kInFlight && k.enqueued < b->max_steps)
    if (int rc = pack_enqueue(b, k)) return bfail(b, rc, "pack launch failed");
  return VF_OK;
}

bool fed(const vf_batch* b) {  // nothing left to enqueue
  return b->pack.live == 0 && std::all_of(b->wide.begin(), b->wide.end(), [](const Wide& w) { return w.done; });
}

// Retire finished chunks of the pack and of every wide member, keep kInFlight queued.
int pump(vf_batch* b) {
  if (b->wide.empty() && b->pack.members.empty()) return VF_OK;
  const BesideCaptures beside;
  std::lock_guard<std::mutex> lk(b->mu);
  if (b->feed_rc) return bfail(b, b->feed_rc, b->feed_err);
  if (fed(b)) return VF_OK;
  if (cudaSetDevice(b->device) != cudaSuccess) return bfail(b, VF_ECUDA, "cudaSetDevice failed");
  const double elapsed =
      std::chrono::duration<double>(std::chrono::steady_clock::now() - b->start).count();
  const bool late = elapsed > b->time_limit_s;
  if (b->pack.live > 0)
    if (int rc = pack_pump(b, b->pack, late)) return rc;
  for (Wide& w : b->wide) {
    if (w.done) continue;
    while (w.inflight > 0) {
      const int slot = w.head % kInFlight;
      const cudaError_t q = cudaEventQuery(w.ev[slot]);
      if (q == cudaErrorNotReady) break;
      if (q != cudaSuccess) return bfail(b, VF_ECUDA, std::string("wide member: ") + cudaGetErrorString(q));
      const vf::StepRecord& r = *slot_rec(b->slots[w.member], slot);
      const long long k = w.chunk_end[slot];
      w.head += 1;
      w.inflight -= 1;
      if (r.wait_fault)
        return bfail(b, VF_ECUDA, "wide member: a bounded wait for a TMA tile copy gave up");
      if (!r.active[k & 1]) {
        wide_finish(b, w, r, k, end_status(r, k, w.max_steps, w.endtime));
        break;
      }
      if (late && w.inflight == 0) {
        wide_finish(b, w, r, k, vf::kEnsTimeout);
        break;
      }
    }
    if (!w.done && late && w.inflight == 0) {
      const int last = (w.head + kInFlight - 1) % kInFlight;
      wide_finish(b, w, *slot_rec(b->slots[w.member], last), w.chunk_end[last], vf::kEnsTimeout);
    }
    if (w.done || late) continue;
    while (w.inflight < kInFlight && w.enqueued < w.max_steps)
      if (int rc = wide_enqueue(b, w)) return bfail(b, rc, "wide member launch: " + b->hs[w.member]->err);
  }
  return VF_OK;
}

// Feeds the batch while the caller is elsewhere. With the default threshold members
// that would run to their end in a cluster by themselves depend on the host; a batch
// that is launched and left alone has to get on all the same. The chunks in flight
// last several times the interval. An error ends the feeder; the caller's next call
// returns it.
void feed(vf_batch* b) {
  g_feeding = true;
  if (cudaSetDevice(b->device) != cudaSuccess) return;
  while (!b->stop) {
    int rc = VF_ENOMEM;
    try {
      rc = pump(b);
    } catch (...) {  // no memory for an error's text
    }
    {
      std::lock_guard<std::mutex> lk(b->mu);
      b->feed_rc = rc;
      if (rc != VF_OK || fed(b)) return;
    }
    std::this_thread::sleep_for(std::chrono::microseconds(100));
  }
}

void start_feeder(vf_batch* b) {
  if (b->wide.empty() && b->pack.members.empty()) return;
  try {
    b->feeder = std::thread(feed, b);
  } catch (...) {  // no thread: the batch is fed when it is polled or waited on
  }
}

struct Group {
  int prec;   // 0 double, 1 float
  int variant;
  int csize;
  std::vector<int> members;  // indices into the batch
};

}  // namespace

extern "C" {

int vf_batch_launch(vf_handle* const* hs, int32_t n, const double* t0, const double* endtime, int32_t match_endtime,
                    double maximum_timestep, int64_t max_steps, const vf_batch_options* opt, vf_batch** out) {
  if (!out) return bfail(nullptr, VF_EINVAL, "out is NULL");
  *out = nullptr;
  if (!hs || !t0 || !endtime || n < 1) return bfail(nullptr, VF_EINVAL, "need n >= 1 handles, t0 and endtime");
  const Opts o = resolve(opt);
  const int device = hs[0] ? hs[0]->device : 0;
  for (int i = 0; i < n; ++i) {
    if (!hs[i]) return bfail(nullptr, VF_EINVAL, "NULL handle");
    if (hs[i]->device != device) return bfail(nullptr, VF_EINVAL, "handles live on different devices");
    for (int j = 0; j < i; ++j)
      if (hs[j] == hs[i]) return bfail(nullptr, VF_EINVAL, "a handle appears twice in the batch");
    if (int rc = vf::handle_ready(hs[i])) return bfail(nullptr, rc, std::string("handle not ready: ") + hs[i]->err);
  }
  if (cudaSetDevice(device) != cudaSuccess) return bfail(nullptr, VF_ECUDA, "cudaSetDevice failed");

  vf_batch* b = new (std::nothrow) vf_batch();
  if (!b) return bfail(nullptr, VF_ENOMEM, "host allocation failed");
  b->device = device;
  b->n = n;
  b->hs.assign(hs, hs + n);
  b->collected.assign(n, 0);
  std::string err;
  if (int rc = acquire_slots(n, b->slots, err)) {
    destroy_batch(b);
    return bfail(nullptr, rc, err);
  }
  for (int i = 0; i < n; ++i) std::memset(slot_host(b->slots[i]), 0, sizeof(vf::EnsResult));

  b->start = std::chrono::steady_clock::now();
  b->time_limit_s = o.time_limit_s;
  b->max_steps = max_steps > 0 ? max_steps : LLONG_MAX;
  b->endtime.assign(endtime, endtime + n);
  // Wide members apart; the rest in groups by precision, kernel design and
  // cluster size, largest work first inside a group.
  std::vector<Group> groups;
  std::vector<double> work(n);
  const bool pack = std::count_if(hs, hs + n, [&](const vf_handle* h) { return packs(h, o); }) >= kPackMembers;
  for (int i = 0; i < n; ++i) {
    const vf_handle* h = hs[i];
    const bool packable = packs(h, o);
    if (pack && packable) {
      b->pack.members.push_back(i);
      continue;
    }
    if (packable || (long long)h->cfg.nx * h->cfg.ny >= wide_cells_for(h, o)) {
      Wide w;
      w.member = i;
      w.max_steps = max_steps > 0 ? max_steps : LLONG_MAX;
      w.endtime = endtime[i];
      b->wide.push_back(w);
      continue;
    }
    const int prec = h->elem == 8 ? 0 : 1;
    const int var = variant_of(h);
    const int c = fit_cluster(device, (int)h->elem, var, cluster_for(h, o));
    const double dxy = std::min(h->ad.g.dx, h->ad.g.dy);
    work[i] = (double)h->cfg.nx * h->cfg.ny * std::max(0.0, endtime[i] - t0[i]) / dxy;
    auto it = std::find_if(groups.begin(), groups.end(),
                           [&](const Group& g) { return g.prec == prec && g.variant == var && g.csize == c; });
    if (it == groups.end()) {
      groups.push_back(Group{prec, var, c, {}});
      it = groups.end() - 1;
    }
    it->members.push_back(i);
  }
  for (Group& g : groups)
    std::stable_sort(g.members.begin(), g.members.end(), [&](int a, int c) { return work[a] > work[c]; });
  std::stable_sort(groups.begin(), groups.end(), [](const Group& a, const Group& c) { return a.csize > c.csize; });

  if (pack) {
    if (int rc = pack_start(b, b->pack, t0, match_endtime, maximum_timestep)) {
      cudaGetLastError();
      destroy_batch(b);
      return bfail(nullptr, rc, "pack start failed");
    }
  }

  // Wide members start first: their first two chunks go in before any cluster.
  for (Wide& w : b->wide) {
    vf_handle* h = hs[w.member];
    bool ok = true;
    for (cudaEvent_t& e : w.ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    int rc = ok ? vf::handle_begin_loop(h, t0[w.member], endtime[w.member], match_endtime, maximum_timestep,
                                           max_steps, true)
                : VF_ECUDA;
    for (int k = 0; rc == VF_OK && k < kInFlight && w.enqueued < w.max_steps; ++k) rc = wide_enqueue(b, w);
    if (rc) {
      cudaGetLastError();
      const std::string msg = std::string("wide member start: ") + h->err;
      destroy_batch(b);
      return bfail(nullptr, rc ? rc : VF_ECUDA, msg);
    }
  }
  if (groups.empty()) {
    if (o.wide_cells == 0) start_feeder(b);
    *out = b;
    return VF_OK;
  }

  for (size_t g = 0; g < groups.size(); ++g) {
    cudaStream_t s = nullptr;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) {
      cudaGetLastError();
      destroy_batch(b);
      return bfail(nullptr, VF_ECUDA, "stream creation failed");
    }
    b->streams.push_back(s);
  }
  b->setup = b->streams[0];
  cudaMemPool_t pool = vf::device_pool(device);
  cudaError_t e = pool ? cudaSuccess : cudaErrorMemoryAllocation;
  if (e == cudaSuccess)
    e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(&b->epoch_d), sizeof(unsigned long long), pool, b->setup);
  if (e == cudaSuccess) e = cudaMemsetAsync(b->epoch_d, 0, sizeof(unsigned long long), b->setup);
  if (e != cudaSuccess) {
    cudaGetLastError();
    destroy_batch(b);
    return bfail(nullptr, VF_ENOMEM, "batch scratch allocation failed");
  }

  // Descriptors: one array per precision, one order array over all groups.
  std::vector<vf::EnsItem<double>> itd;
  std::vector<vf::EnsItem<float>> itf;
  std::vector<int> order;
  std::vector<int> group_base;
  for (const Group& g : groups) {
    group_base.push_back((int)order.size());
    for (int i : g.members) {
      vf_handle* h = hs[i];
      vf::EnsResult* res = slot_dev(b->slots[i]);
      if (g.prec == 0) {
        order.push_back((int)itd.size());
        itd.push_back(make_item<double>(h, h->ad, t0[i], endtime[i], match_endtime, maximum_timestep, max_steps, res,
                                         b->epoch_d));
        itd.back().seg_rows = seg_rows_for(o.seg_rows);
      } else {
        order.push_back((int)itf.size());
        itf.push_back(make_item<float>(h, h->af, t0[i], endtime[i], match_endtime, maximum_timestep, max_steps, res,
                                        b->epoch_d));
        itf.back().seg_rows = seg_rows_for(o.seg_rows);
      }
    }
  }

  if (!itd.empty())
    e = cudaMallocFromPoolAsync(&b->items_d[0], sizeof(vf::EnsItem<double>) * itd.size(), pool, b->setup);
  if (e == cudaSuccess && !itf.empty())
    e = cudaMallocFromPoolAsync(&b->items_d[1], sizeof(vf::EnsItem<float>) * itf.size(), pool, b->setup);
  if (e == cudaSuccess) e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(&b->order_d), sizeof(int) * order.size(), pool, b->setup);
  if (e == cudaSuccess && !itd.empty())
    e = cudaMemcpyAsync(b->items_d[0], itd.data(), sizeof(vf::EnsItem<double>) * itd.size(), cudaMemcpyHostToDevice,
                        b->setup);
  if (e == cudaSuccess && !itf.empty())
    e = cudaMemcpyAsync(b->items_d[1], itf.data(), sizeof(vf::EnsItem<float>) * itf.size(), cudaMemcpyHostToDevice,
                        b->setup);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(b->order_d, order.data(), sizeof(int) * order.size(), cudaMemcpyHostToDevice, b->setup);
  // The copies read pageable host vectors: finish them before the vectors go.
  if (e == cudaSuccess) e = cudaStreamSynchronize(b->setup);
  if (e != cudaSuccess) {
    cudaGetLastError();
    destroy_batch(b);
    return bfail(nullptr, VF_ECUDA, std::string("batch descriptors: ") + cudaGetErrorString(e));
  }
  const unsigned long long limit_ns = (unsigned long long)(o.time_limit_s * 1e9);
  for (size_t g = 0; g < groups.size(); ++g) {
    const Group& gr = groups[g];
    const int* ord = b->order_d + group_base[g];
    const int cnt = (int)gr.members.size();
    e = gr.prec == 0 ? vf::launch_ensemble(static_cast<const vf::EnsItem<double>*>(b->items_d[0]), ord, cnt,
                                           gr.csize, gr.variant, limit_ns, b->streams[g])
                     : vf::launch_ensemble(static_cast<const vf::EnsItem<float>*>(b->items_d[1]), ord, cnt, gr.csize,
                                           gr.variant, limit_ns, b->streams[g]);
    if (e != cudaSuccess) {
      cudaGetLastError();
      destroy_batch(b);
      return bfail(nullptr, VF_ECUDA, std::string("ensemble launch: ") + cudaGetErrorString(e));
    }
    hs[gr.members.front()]->launches += 1;  // one launch for the whole group
  }
  if (o.wide_cells == 0) start_feeder(b);
  *out = b;
  return VF_OK;
}

int vf_batch_poll(vf_batch* b, int32_t* n_done) {
  if (!b || !n_done) return bfail(b, VF_EINVAL, "NULL argument");
  if (int rc = pump(b)) return rc;
  int c = 0;
  for (int i = 0; i < b->n; ++i) c += slot_done(b->slots[i]) ? 1 : 0;
  *n_done = c;
  return VF_OK;
}

int vf_batch_is_done(vf_batch* b, int32_t i) {
  if (!b || i < 0 || i >= b->n) return bfail(b, VF_EINVAL, "bad batch index");
  if (int rc = pump(b)) return rc;
  return slot_done(b->slots[i]) ? 1 : 0;
}

int vf_batch_collect(vf_batch* b, int32_t i, double* t_out, int64_t* steps_out, double* last_dt_out,
                     int32_t* status_out) {
  if (!b || i < 0 || i >= b->n) return bfail(b, VF_EINVAL, "bad batch index");
  if (!slot_done(b->slots[i])) return bfail(b, VF_ESTATE, "simulation has not finished");
  const vf::EnsResult* r = slot_host(b->slots[i]);
  if (!b->collected[i]) {
    if (r->steps & 1) std::swap(b->hs[i]->U[0], b->hs[i]->U[1]);
    b->collected[i] = 1;
  }
  if (t_out) *t_out = r->t;
  if (steps_out) *steps_out = r->steps;
  if (last_dt_out) *last_dt_out = r->last_dt;
  if (status_out) *status_out = r->status;
  return VF_OK;
}

int vf_batch_wait(vf_batch* b) {
  if (!b) return bfail(b, VF_EINVAL, "NULL batch");
  const BesideCaptures beside;
  if (cudaSetDevice(b->device) != cudaSuccess) return bfail(b, VF_ECUDA, "cudaSetDevice failed");
  for (;;) {  // wide members and packs need the host to feed them
    if (int rc = pump(b)) return rc;
    cudaEvent_t next = nullptr;  // the end of the next chunk
    {
      std::lock_guard<std::mutex> lk(b->mu);
      if (fed(b)) break;
      if (b->pack.live > 0 && b->pack.inflight > 0) next = b->pack.ev[b->pack.head % kInFlight];
      for (const Wide& w : b->wide)
        if (!next && !w.done && w.inflight > 0) next = w.ev[w.head % kInFlight];
    }
    if (next) cudaEventSynchronize(next);
  }
  for (cudaStream_t s : b->streams) {
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return bfail(b, VF_ECUDA, std::string("ensemble: ") + cudaGetErrorString(e));
  }
  for (int i = 0; i < b->n; ++i)
    if (!slot_done(b->slots[i])) return bfail(b, VF_ECUDA, "ensemble finished without a result");
  return VF_OK;
}

int vf_batch_free(vf_batch* b) {
  if (!b) return VF_OK;
  int rc = vf_batch_wait(b);
  if (rc == VF_OK)
    for (int i = 0; i < b->n; ++i) vf_batch_collect(b, i, nullptr, nullptr, nullptr, nullptr);
  if (rc != VF_OK) g_batch_error = b->err;
  destroy_batch(b);
  return rc;
}

int vf_batch_simulate(vf_handle* const* hs, int32_t n, const double* t0, const double* endtime, int32_t match_endtime,
                      double maximum_timestep, int64_t max_steps, const vf_batch_options* opt, double* t_out,
                      int64_t* steps_out, double* last_dt_out, int32_t* status_out) {
  vf_batch* b = nullptr;
  int rc = vf_batch_launch(hs, n, t0, endtime, match_endtime, maximum_timestep, max_steps, opt, &b);
  if (rc) return rc;
  rc = vf_batch_wait(b);
  if (rc) {
    g_batch_error = b->err;
    destroy_batch(b);
    return rc;
  }
  for (int i = 0; i < n; ++i) {
    double t = 0, ldt = 0;
    int64_t st = 0;
    int32_t s = 0;
    vf_batch_collect(b, i, &t, &st, &ldt, &s);
    if (t_out) t_out[i] = t;
    if (steps_out) steps_out[i] = st;
    if (last_dt_out) last_dt_out[i] = ldt;
    if (status_out) status_out[i] = s;
  }
  destroy_batch(b);
  return VF_OK;
}

int vf_batch_cluster_size(vf_handle* h, const vf_batch_options* opt, int32_t* csize_out) {
  if (!h || !csize_out) return bfail(nullptr, VF_EINVAL, "NULL argument");
  if (cudaSetDevice(h->device) != cudaSuccess) return bfail(nullptr, VF_ECUDA, "cudaSetDevice failed");
  *csize_out = fit_cluster(h->device, (int)h->elem, variant_of(h), cluster_for(h, resolve(opt)));
  return VF_OK;
}

const char* vf_batch_last_error(vf_batch* b) { return b ? b->err.c_str() : g_batch_error.c_str(); }

}  // extern "C"
