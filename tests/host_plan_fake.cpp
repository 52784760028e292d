// opencnn_b200/csrc/host_plan.h against a runtime that is made here: streams are queues of operations that run only when somebody waits, in
// any order that the events allow, chosen by a seed.  Operations are real copies between host arrays and a stand-in for the operator, so
// a missing wait shows as wrong numbers; any call can be made to fail.  No GPU, no CUDA library.
#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <new>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "../include/opencnn_b200.h"

// ------------------------------------------------- the runtime -------------------------------------------------
struct Event { long recorded = 0, done = 0; };
struct Op {
  std::function<void()> run;
  std::function<bool()> ready;
  bool host = false;                // reads or writes the caller's memory
};
struct Stream { std::deque<Op> ops; bool alive = true; };

std::mutex g_m;
std::condition_variable g_cv;
std::vector<Stream *> g_streams;
unsigned g_seed = 1;
std::atomic<int> g_copies_2d{0};
int g_fail_in = -1, g_streams_alive = 0, g_stream_creations_to_fail = 0;
std::set<const void *> g_pageable;

unsigned pick(unsigned n) {
  g_seed = g_seed * 1664525u + 1013904223u;
  return (g_seed >> 8) % n;
}
bool fails() { return g_fail_in >= 0 && g_fail_in-- == 0; }
Stream *as_stream(cudaStream_t s) { return reinterpret_cast<Stream *>(s); }
Event *as_event(cudaEvent_t e) { return reinterpret_cast<Event *>(e); }
cudaError_t push(cudaStream_t s, Op op) {
  std::lock_guard<std::mutex> l(g_m);
  if (fails()) return cudaErrorUnknown;
  as_stream(s)->ops.push_back(std::move(op));
  g_cv.notify_all();
  return cudaSuccess;
}
bool run_one() {                    // g_m held
  std::vector<Stream *> able;
  for (Stream *s : g_streams)
    if (!s->ops.empty() && (!s->ops.front().ready || s->ops.front().ready())) able.push_back(s);
  if (able.empty()) return false;
  Stream *s = able[pick((unsigned)able.size())];
  if (s->ops.front().run) s->ops.front().run();
  s->ops.pop_front();
  return true;
}

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { *p = calloc(n, 1); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  std::lock_guard<std::mutex> l(g_m);
  if (g_stream_creations_to_fail > 0 && g_streams_alive > 0) {       // (a plan's own stream is the first)
    --g_stream_creations_to_fail;
    return cudaErrorMemoryAllocation;
  }
  Stream *n = new Stream;
  g_streams.push_back(n);
  ++g_streams_alive;
  *s = reinterpret_cast<cudaStream_t>(n);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::unique_lock<std::mutex> l(g_m);
  const auto until = std::chrono::steady_clock::now() + std::chrono::seconds(3);
  while (!as_stream(s)->ops.empty())
    if (!run_one() && g_cv.wait_until(l, until) == std::cv_status::timeout) return cudaErrorLaunchTimeout;
  g_cv.notify_all();
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::lock_guard<std::mutex> l(g_m);
  as_stream(s)->alive = false;
  --g_streams_alive;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(new Event); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  Event *ev = as_event(e);
  long n;
  {
    std::lock_guard<std::mutex> l(g_m);
    n = ev->recorded + 1;
  }
  const cudaError_t err = push(s, {[ev, n] { if (ev->done < n) ev->done = n; }, {}, false});
  std::lock_guard<std::mutex> l(g_m);
  if (err == cudaSuccess) ev->recorded = n;
  return err;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  Event *ev = as_event(e);
  long n;
  {
    std::lock_guard<std::mutex> l(g_m);
    n = ev->recorded;
  }
  return push(s, {{}, [ev, n] { return ev->done >= n; }, false});
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  return push(st, {[=] { memmove(d, s, n); }, {}, true});
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t st) {
  ++g_copies_2d;
  return push(st, {[=] { for (size_t i = 0; i < h; ++i) memmove((char *)d + i * dp, (const char *)s + i * sp, w); }, {}, true});
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  memset(a, 0, sizeof *a);
  a->type = g_pageable.count(p) ? cudaMemoryTypeUnregistered : cudaMemoryTypeHost;
  return cudaSuccess;
}
size_t opencnn_workspace_bytes(int c, int k) { return (size_t)c * 16 * k * 4; }
}

// ------------------------------------------------- the operator -------------------------------------------------
// Filter k of the stand-in reads channel k % C, three rows of it, and one number of the transformed filter.
namespace {
constexpr int kMaxDevices = 4;
struct TileRows { int first, count; };
struct ShapeRule { int n_multiple; };
ShapeRule shape_rule(int) { return {4}; }
cudaError_t check_shape(int N, int C, int H, int W, int K, ShapeRule r) {
  return N > 0 && C > 0 && H > 0 && W > 0 && K > 0 && N % r.n_multiple == 0 ? cudaSuccess : cudaErrorInvalidValue;
}
void stand_in(const float *x, const float *ws, float *y, int N, int C, int H, int W, int K, int h0, int h1) {
  const size_t row = (size_t)W * N;
  for (int k = 0; k < K; ++k)
    for (int h = h0; h < h1; ++h)
      for (size_t i = 0; i < row; ++i) {
        const float *c = x + ((size_t)(k % C) * H + h) * row + i;
        y[((size_t)k * H + h) * row + i] = ws[k] * (c[0] + (h > 0 ? 2 * *(c - row) : 0) + (h + 1 < H ? 4 * *(c + row) : 0));
      }
}
cudaError_t transform_filter(const float *f, float *ws, int, int K, int, cudaStream_t s) {
  return push(s, {[=] { for (int k = 0; k < K; ++k) ws[k] = 1 + f[k]; }, {}, false});
}
cudaError_t convolve_rows(const float *x, const float *ws, float *y, int N, int C, int H, int W, int K, int, cudaStream_t s, TileRows r) {
  return push(s, {[=] { stand_in(x, ws, y, N, C, H, W, K, 2 * r.first, std::min(H, 2 * (r.first + r.count))); }, {}, false});
}
cudaError_t forward(const float *x, const float *f, float *y, float *ws, int N, int C, int H, int W, int K, int p, cudaStream_t s, ShapeRule) {
  const cudaError_t e = transform_filter(f, ws, C, K, p, s);
  return e != cudaSuccess ? e : convolve_rows(x, ws, y, N, C, H, W, K, p, s, {0, (H + 1) / 2});
}
}  // namespace

#ifndef HOST_PLAN
#define HOST_PLAN "../opencnn_b200/csrc/host_plan.h"
#endif
#include HOST_PLAN

// ------------------------------------------------- the checks -------------------------------------------------
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); std::exit(1); } } while (0)

struct Problem {
  int N, C, H, W, K;
  std::vector<float> x, f, y, expect;
  Problem(int N_, int C_, int H_, int W_, int K_, float filter = 1) : N(N_), C(C_), H(H_), W(W_), K(K_) {
    x.resize((size_t)C * H * W * N);
    for (size_t i = 0; i < x.size(); ++i) x[i] = (float)((i * 2654435761u >> 7) % 1000);
    f.assign((size_t)C * 9 * K, filter);
    for (int k = 0; k < K; ++k) f[k] += k;
    y.assign((size_t)K * H * W * N, -1);
    expect = y;
    std::vector<float> ws(K);
    for (int k = 0; k < K; ++k) ws[k] = 1 + f[k];
    stand_in(x.data(), ws.data(), expect.data(), N, C, H, W, K, 0, H);
  }
  void *plan() const {
    void *p = nullptr;
    CHECK(opencnn_host_plan_create(&p, N, C, H, W, K, 0) == 0 && p);
    return p;
  }
  int run(void *p) { return opencnn_host_plan_run(p, x.data(), f.data(), y.data()); }
};
int pending_on_host() {
  std::lock_guard<std::mutex> l(g_m);
  int n = 0;
  for (Stream *s : g_streams)
    for (const Op &o : s->ops) n += o.host;
  return n;
}
void finish_all() {
  std::lock_guard<std::mutex> l(g_m);
  while (run_one()) {}
}

// The numbers of the operator whatever order the streams run in: page-locked memory (bands) and other memory (one piece), odd and even
// heights, behind a run that was not waited for.
void results() {
  for (int trial = 0; trial < 40; ++trial) {
    g_seed = 77 + trial;
    Problem a(32, 24, trial % 2 ? 41 : 40, 40, 28), b(32, 24, a.H, 40, 28, 5);
    void *p = a.plan();
    CHECK(static_cast<HostPlan *>(p)->bands > 1);
    g_pageable.clear();
    if (trial % 4 == 3) g_pageable.insert(trial % 8 == 3 ? (void *)b.x.data() : (void *)b.y.data());
    const int copies = g_copies_2d;
    CHECK(opencnn_host_plan_run_async(p, a.x.data(), a.f.data(), a.y.data()) == 0);
    CHECK(b.run(p) == 0);
    CHECK((g_copies_2d > copies) == g_pageable.empty());
    CHECK(a.y == a.expect && b.y == b.expect && pending_on_host() == 0);
    CHECK(opencnn_host_plan_destroy(p) == 0);
  }
}

// Whichever call of a run fails, the error comes back when nothing reads or writes the caller's memory any more, and the next run is right.
void errors() {
  Problem a(32, 24, 40, 40, 28);
  for (int pageable = 0; pageable < 2; ++pageable)
    for (int n = 0;; ++n) {
      g_pageable.clear();
      if (pageable) g_pageable.insert(a.y.data());
      void *p = a.plan();
      g_seed = 3 + n;
      g_fail_in = n;
      const int e = a.run(p);
      const bool failed = g_fail_in < 0;
      g_fail_in = -1;
      CHECK((e != 0) == failed);
      CHECK(pending_on_host() == 0);
      std::fill(a.y.begin(), a.y.end(), -1.f);
      CHECK(a.run(p) == 0 && a.y == a.expect);
      CHECK(opencnn_host_plan_destroy(p) == 0);
      if (!failed) {
        CHECK(n > (pageable ? 4 : 20));
        break;
      }
    }
}

// A run waits for nothing of another plan: one whose work does not come to an end (here: is held back) keeps no other from it.
void apart() {
  Problem a(32, 24, 40, 40, 28), b(32, 24, 41, 40, 28, 3);
  void *pa = a.plan(), *pb = b.plan();
  CHECK(static_cast<HostPlan *>(pa)->bands > 1 && static_cast<HostPlan *>(pb)->bands > 1);
  bool open = false;
  int ea = -1;
  CHECK(push(static_cast<HostPlan *>(pa)->stream, {{}, [&open] { return open; }, false}) == cudaSuccess);
  std::thread t([&] { ea = a.run(pa); });
  for (int n = 0; n < 1000; ++n) {                  // until all of it is enqueued: the join of the download waits on a's stream
    std::this_thread::sleep_for(std::chrono::milliseconds(1));
    std::lock_guard<std::mutex> l(g_m);
    if (as_stream(static_cast<HostPlan *>(pa)->stream)->ops.size() > 10) break;
  }
  std::this_thread::sleep_for(std::chrono::milliseconds(100));
  for (int n = 0; n < 3; ++n) {
    std::fill(b.y.begin(), b.y.end(), -1.f);
    CHECK(b.run(pb) == 0 && b.y == b.expect);
  }
  {
    std::lock_guard<std::mutex> l(g_m);
    open = true;
    g_cv.notify_all();
  }
  t.join();
  CHECK(ea == 0 && a.y == a.expect);
  CHECK(opencnn_host_plan_destroy(pa) == 0 && opencnn_host_plan_destroy(pb) == 0);
}

// Runs in many threads: right, and on one pair of copy streams.  A plan for which the pair can't be made runs in one piece - until it can.
void streams() {
  Problem a(32, 24, 40, 40, 28);
  std::vector<Problem> many(6, a);
  std::vector<void *> plans;
  for (Problem &q : many) plans.push_back(q.plan());
  std::vector<std::thread> ts;
  std::vector<int> bad(many.size(), 0);
  for (size_t i = 0; i < many.size(); ++i)
    ts.emplace_back([&, i] {
      for (int n = 0; n < 5; ++n) {
        std::fill(many[i].y.begin(), many[i].y.end(), -1.f);
        bad[i] += many[i].run(plans[i]) != 0 || many[i].y != many[i].expect;
      }
    });
  for (std::thread &t : ts) t.join();
  for (int n : bad) CHECK(n == 0);
  CHECK(g_copies_2d > 0 && g_streams_alive == 6 + 2);
  for (void *p : plans) CHECK(opencnn_host_plan_destroy(p) == 0);
  CHECK(g_streams_alive == 2);
}
void no_streams() {
  Problem a(32, 24, 40, 40, 28);
  g_stream_creations_to_fail = 3;                   // at the plan's creation, and at its first runs
  void *p = a.plan();
  for (int n = 0; n < 4; ++n) {
    std::fill(a.y.begin(), a.y.end(), -1.f);
    CHECK(a.run(p) == 0 && a.y == a.expect);
  }
  CHECK(g_stream_creations_to_fail == 0 && g_copies_2d > 0);
  CHECK(opencnn_host_plan_destroy(p) == 0);
}

// Input and output in one array: the input has been read where the output is written, wherever the two start.
void overlap() {
  Problem a(32, 24, 40, 40, 28);
  const size_t row = (size_t)a.W * a.N;
  for (long shift : {0l, (long)row, -(long)row, 5l * (long)row, -17l * (long)row, (long)a.x.size() / 2, -(long)a.y.size() / 2, (long)a.x.size()})
    for (int trial = 0; trial < 4; ++trial) {
      g_seed = 11 + trial;
      std::vector<float> both(a.x.size() + 2 * a.y.size(), -1.f);
      float *x = both.data() + a.y.size(), *y = x + shift;
      std::copy(a.x.begin(), a.x.end(), x);
      void *p = a.plan();
      const int copies = g_copies_2d;
      CHECK(opencnn_host_plan_run(p, x, a.f.data(), y) == 0);
      CHECK(std::equal(a.expect.begin(), a.expect.end(), y));
      CHECK((g_copies_2d > copies) == (shift == 0 || shift == (long)a.x.size()));
      CHECK(opencnn_host_plan_destroy(p) == 0);
    }
}

int main(int argc, char **argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  const std::map<std::string, void (*)()> checks = {{"results", results}, {"errors", errors}, {"apart", apart}, {"streams", streams}, {"no_streams", no_streams}, {"overlap", overlap}};
  if (what == "bands" && argc == 7) {               // bands N C H W K
    std::printf("%d\n", band_count(atoi(argv[2]), atoi(argv[3]), atoi(argv[4]), atoi(argv[5]), atoi(argv[6])));
    return 0;
  }
  const auto it = checks.find(what);
  if (it == checks.end()) return 2;
  it->second();
  std::printf("ok\n");
  return 0;
}
