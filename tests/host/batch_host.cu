// The host side of the batches (csrc/vf_batch.cu) on the CUDA runtime of
// fake_cudart.h; a step advances the step record alone. One scenario per run,
// named by the first argument; exit code 0 when it holds.
#include <cuda_runtime.h>

#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "fake_cudart.h"
#include "vf_handle.h"

#define LOCK std::lock_guard<std::recursive_mutex> lock_(fake::mu)

static double g_dt = 0.5;  // of every step; written under the lock
// ---- the units beside vf_batch.cu ------------------------------------------------
namespace vf {
static void advance(StepRecord* r, int parity) {
  if (!r->active[parity]) {
    r->t[parity ^ 1] = r->t[parity];
    r->active[parity ^ 1] = 0;
    return;
  }
  r->last_dt = g_dt;
  r->t[parity ^ 1] = r->t[parity] + g_dt;
  r->n_done += 1;
  if (r->stop_stalled && r->t[parity ^ 1] == r->t[parity]) r->stalled = 1;
  r->active[parity ^ 1] =
      r->t[parity ^ 1] < r->endtime && !(r->max_steps > 0 && r->n_done >= r->max_steps) && !r->stalled ? 1 : 0;
}
int handle_ready(vf_handle*) { return VF_OK; }
int handle_begin_loop(vf_handle* h, double t0, double endtime, int, double, long long max_steps, bool stop_stalled) {
  StepRecord r{};
  r.t[0] = t0;
  r.active[0] = t0 < endtime;
  r.endtime = endtime;
  r.max_steps = max_steps > 0 ? max_steps : 0;
  r.stop_stalled = stop_stalled;
  fake::enqueue(h->stream, [h, r] { *h->rec = r; });
  return VF_OK;
}
int handle_enqueue_steps(vf_handle* h, long long first, int n) {
  fake::enqueue(h->stream, [h, first, n] {
    for (int i = 0; i < n; ++i) advance(h->rec, (int)((first + i) & 1));
  });
  return VF_OK;
}
int handle_enqueue_chunk(vf_handle* h, int k) { return handle_enqueue_steps(h, 0, k); }
cudaMemPool_t device_pool(int) { return reinterpret_cast<cudaMemPool_t>(1); }
int pack_blocks(int, int) { return 1; }
cudaError_t launch_pack_step(const PackItem<double>* items, const PackMap& m, int parity, cudaStream_t st) {
  fake::enqueue(st, [items, m, parity] {
    for (int i = 0; i < m.n; ++i) advance(items[m.blocks[i].member].rec, parity);
  });
  return cudaSuccess;
}
cudaError_t launch_pack_report(const PackItem<double>* items, int n, int slot, cudaStream_t st) {
  fake::enqueue(st, [items, n, slot] {
    for (int i = 0; i < n; ++i) *items[i].report[slot] = *items[i].rec;
  });
  return cudaSuccess;
}
template <typename T>
static cudaError_t clusters(const EnsItem<T>* items, const int* order, int n, cudaStream_t st) {
  fake::enqueue(st, [items, order, n] {
    for (int k = 0; k < n; ++k) {
      const EnsItem<T>& it = items[order[k]];
      it.res->t = it.endtime;
      it.res->steps = 2;
      it.res->last_dt = g_dt;
      it.res->status = kEnsOk;
      __atomic_store_n(&it.res->done, 1, __ATOMIC_RELEASE);
    }
  });
  return cudaSuccess;
}
cudaError_t launch_ensemble(const EnsItem<double>* items, const int* order, int n, int, int, unsigned long long,
                            cudaStream_t st) {
  return clusters(items, order, n, st);
}
cudaError_t launch_ensemble(const EnsItem<float>* items, const int* order, int n, int, int, unsigned long long,
                            cudaStream_t st) {
  return clusters(items, order, n, st);
}
cudaError_t ensemble_max_clusters_f64(int, int, int* out) { return *out = 1, cudaSuccess; }
cudaError_t ensemble_max_clusters_f32(int, int, int* out) { return *out = 1, cudaSuccess; }
}  // namespace vf

// ---- scenarios -------------------------------------------------------------------
#define CHECK(x)                                                        \
  do {                                                                  \
    if (!(x)) {                                                         \
      std::printf("%s:%d: %s\n", __FILE__, __LINE__, #x);               \
      std::exit(1);                                                     \
    }                                                                   \
  } while (0)

// A handle of n x n cells; Float64 RK2 tiles.
static vf_handle* make(int n) {
  vf_handle* h = new vf_handle();
  std::memset(&h->cfg, 0, sizeof(h->cfg));
  std::memset(&h->ad, 0, sizeof(h->ad));
  std::memset(&h->af, 0, sizeof(h->af));
  h->cfg.nx = h->cfg.ny = n;
  h->cfg.gc = 2;
  h->elem = 8;
  h->ad.rk2 = 1;
  h->ad.variant = 1;
  h->ad.g.dx = h->ad.g.dy = 1.0;
  h->rec = static_cast<vf::StepRecord*>(std::calloc(1, sizeof(vf::StepRecord)));
  h->U[0] = std::malloc(1);
  h->U[1] = std::malloc(1);
  cudaStreamCreateWithFlags(&h->stream, 0);
  return h;
}
static std::vector<vf_handle*> make(int count, int n) {
  std::vector<vf_handle*> v;
  for (int i = 0; i < count; ++i) v.push_back(make(n));
  return v;
}
static vf_batch* launch(const std::vector<vf_handle*>& hs, double t0, double end, long long max_steps = 0,
                        long long wide_cells = 0) {
  vf_batch_options o{};
  o.wide_cells = wide_cells;
  std::vector<double> t(hs.size(), t0), e(hs.size(), end);
  vf_batch* b = nullptr;
  if (vf_batch_launch(hs.data(), (int)hs.size(), t.data(), e.data(), 1, -1.0, max_steps, &o, &b)) {
    std::printf("launch: %s\n", vf_batch_last_error(nullptr));
    std::exit(1);
  }
  return b;
}
// Waits until every member is done, by vf_batch_collect alone (which does not feed).
static bool left_alone(vf_batch* b, int n) {
  const auto limit = std::chrono::steady_clock::now() + std::chrono::seconds(20);
  for (int i = 0; i < n;) {
    if (vf_batch_collect(b, i, nullptr, nullptr, nullptr, nullptr) == VF_OK) {
      ++i;
      continue;
    }
    if (std::chrono::steady_clock::now() > limit) return false;
    std::this_thread::sleep_for(std::chrono::milliseconds(1));
  }
  return true;
}

// A batch that ends in an error returns with nothing of it running: its kernels
// write result slots, records and states that the next batch may use.
static void error() {
  for (long long wide_cells : {0LL, 8192LL}) {
    fake::device_runs = false;
    std::vector<vf_handle*> hs = make(2, 32);  // clusters of two sizes
    hs.push_back(make(60));
    hs.push_back(make(128));  // launches of their own
    hs.push_back(make(160));
    vf_batch* b = launch(hs, 0, 8, 0, wide_cells);
    {
      LOCK;
      fake::fail_queries = 1 << 30;
    }
    int32_t done = 0;
    CHECK(vf_batch_poll(b, &done) == VF_ECUDA);
    CHECK(fake::busy() > 0);
    CHECK(vf_batch_free(b) == VF_ECUDA);
    fake::fail_queries = 0;
    CHECK(fake::frees_while_busy == 0);
    CHECK(fake::busy() == 0);
  }
}

// A member whose time stands still ends with the step that left it unchanged, as a
// cluster member does: on launches of its own (3 members) and in a pack (9).
static void stall() {
  g_dt = 0;
  for (int members : {3, 9})
    for (long long max_steps : {0LL, 19LL, 1LL}) {
      std::vector<vf_handle*> hs = make(members, 70);
      std::vector<void*> u0;
      for (vf_handle* h : hs) u0.push_back(h->U[0]);
      vf_batch* b = launch(hs, 0, 8, max_steps);
      CHECK(vf_batch_wait(b) == VF_OK);
      for (int i = 0; i < members; ++i) {
        int64_t steps = 0;
        int32_t status = 0;
        double t = 1, dt = 1;
        CHECK(vf_batch_collect(b, i, &t, &steps, &dt, &status) == VF_OK);
        CHECK(steps == 1 && t == 0 && dt == 0 && status == VF_BATCH_STALLED);
        CHECK(hs[i]->U[1] == u0[i]);
      }
      CHECK(vf_batch_free(b) == VF_OK);
    }
}

// Batches of thousands of members are launched while the feeder of another one
// reads its members' records (run under the thread sanitizer).
static void slots() {
  vf_batch* first = launch({make(128)}, 0, 1e9);
  std::vector<vf_batch*> more;
  for (int k = 0; k < 5; ++k) {
    more.push_back(launch(make(3000, 8), 0, 1));
    std::this_thread::sleep_for(std::chrono::milliseconds(5));
  }
  for (vf_batch* b : more) CHECK(vf_batch_free(b) == VF_OK);
  {
    LOCK;
    g_dt = 1e9;
  }
  CHECK(left_alone(first, 1));
  CHECK(vf_batch_free(first) == VF_OK);
}

// A batch left alone gets on while a thread of the caller captures in the global
// mode, and its calls do not end that capture.
static void capture() {
  fake::device_runs = false;
  std::vector<vf_handle*> hs = make(9, 70);  // a pack
  hs.push_back(make(300));                   // launches of their own
  hs.push_back(make(8));                     // a cluster
  vf_batch* b = launch(hs, 0, 40);
  {
    LOCK;
    fake::capturing = fake::device_runs = true;
  }
  int32_t done = 0;
  CHECK(vf_batch_poll(b, &done) == VF_OK);
  CHECK(left_alone(b, 10));
  CHECK(vf_batch_poll(b, &done) == VF_OK);
  CHECK(vf_batch_wait(b) == VF_OK);
  CHECK(fake::refused == 0);
  fake::capturing = false;
  CHECK(vf_batch_free(b) == VF_OK);
}

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "error") error();
  else if (what == "stall") stall();
  else if (what == "slots") slots();
  else if (what == "capture") capture();
  else return 2;
  return 0;
}
