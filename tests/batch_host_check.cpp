// The host side of hmn_batch.cu (work list, classes, graphs, launch order) on
// a made-up runtime: the CUDA runtime calls and the kernel launchers it uses are
// defined here, on host memory, so that it runs without a GPU and a launch can
// be made to fail.  A "kernel" does to the descriptors what the real one does to
// a simulation's clock; a captured graph is the list of its launches.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <string>
#include <vector>

size_t __cvta_generic_to_shared(const void*);  // named by device functions that nothing here calls
#include "../hormone_b200/csrc/hmn_batch.cu"

using Work = std::vector<std::function<void()>>;
static Work* capturing = nullptr;       // launches go here while a stream is captured
static std::string fail_next;           // launcher to fail once
static std::vector<std::string> trace;  // launches as they run
static int captures = 0;

static cudaError_t launch(const char* name, std::function<void()> f) {
  if (fail_next == name) {
    fail_next.clear();
    return cudaErrorLaunchFailure;
  }
  auto run = [name, f] {
    trace.push_back(name);
    f();
  };
  if (capturing)
    capturing->push_back(run);
  else
    run();
  return cudaSuccess;
}

extern "C" {
const char* CUDARTAPI cudaGetErrorString(cudaError_t) { return "made up"; }
cudaError_t CUDARTAPI cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t CUDARTAPI cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t CUDARTAPI cudaMalloc(void** p, size_t n) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t CUDARTAPI cudaMallocHost(void** p, size_t n) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t CUDARTAPI cudaFree(void* p) { return free(p), cudaSuccess; }
cudaError_t CUDARTAPI cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t CUDARTAPI cudaMemset(void* p, int v, size_t n) { return memset(p, v, n), cudaSuccess; }
cudaError_t CUDARTAPI cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return memset(p, v, n), cudaSuccess; }
cudaError_t CUDARTAPI cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return memcpy(d, s, n), cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  return *s = (cudaStream_t)calloc(1, 1), cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamDestroy(cudaStream_t s) { return free(s), cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  return *e = (cudaEvent_t)calloc(1, 1), cudaSuccess;
}
cudaError_t CUDARTAPI cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t CUDARTAPI cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  captures++;
  return capturing = new Work, cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = (cudaGraph_t)capturing;
  return capturing = nullptr, cudaSuccess;
}
cudaError_t CUDARTAPI cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  return *e = (cudaGraphExec_t) new Work(*(Work*)g), cudaSuccess;
}
cudaError_t CUDARTAPI cudaGraphDestroy(cudaGraph_t g) { return delete (Work*)g, cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphExecDestroy(cudaGraphExec_t e) { return delete (Work*)e, cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  for (auto& f : *(Work*)e) f();
  return cudaSuccess;
}
}

namespace hmn {
int batch_tile_kind(const int s[3]) { return s[0] ? (s[1] ? (s[2] ? 0 : 1) : 2) : -1; }
int batch_tile_variants(int kind, int* ids) {
  const int first[3] = {0, 2, 4}, count[3] = {2, 2, 1};
  for (int v = 0; v < count[kind]; v++) ids[v] = first[kind] + v;
  return count[kind];
}
void batch_tile_shape(int id, int t[3]) {
  const int shapes[8][3] = {{8, 8, 8}, {8, 8, 4}, {16, 16, 1}, {32, 8, 1}, {256, 1, 1}, {8, 4, 4}, {8, 8, 1}, {30, 1, 1}};
  for (int a = 0; a < 3; a++) t[a] = shapes[id][a];
}
int batch_few_tile(int kind, int nsm, int* most) { return *most = (1 << kind) * nsm, 5 + kind; }
int batch_stage_blocks_per_sm(int, bool, bool, int) { return 3; }
cudaError_t launch_prim_init(double*, size_t, bool, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_prim_from_u(const double*, double*, size_t, bool, bool, int, cudaStream_t) { return cudaSuccess; }

constexpr double kDt = 0.25;
static void reduce(SimDesc* sims, const int2* items, int n, bool fresh) {
  for (int i = 0; i < n; i++) {
    if (fresh && !sims[items[i].x].fresh) continue;
    const double dti = kDt;
    memcpy(&sims[items[i].x].sc.min_dti_bits, &dti, sizeof(dti));
  }
}
static void next_dt(SimDesc& S) {
  memcpy(&S.sc.dt, &S.sc.min_dti_bits, sizeof(double));  // infinite where nothing was reduced
  S.sc.min_dti_bits = 0x7ff0000000000000ULL;
}
cudaError_t launch_batch_cfl(SimDesc* sims, const int2* items, int n, int, bool, int after, int, cudaStream_t) {
  return launch(after ? "cfl" : "cfl0", [=] { reduce(sims, items, n, after == 0); });
}
cudaError_t launch_batch_finalize(SimDesc* sims, int n, cudaStream_t) {
  return launch("finalize", [=] {
    for (int s = 0; s < n; s++)
      if (sims[s].active && !sims[s].sc.done && !sims[s].held && sims[s].fresh) next_dt(sims[s]), sims[s].fresh = 0;
  });
}
cudaError_t launch_batch_stage(SimDesc* sims, const int2* items, int n, int tile, bool, bool, int stage, int rk, int, int,
                               int*, cudaStream_t) {
  if (n == 0) return cudaSuccess;
  return launch(tile >= 5 ? "few" : "stage", [=] {
    if (tile >= 5 && stage == rk) reduce(sims, items, n, false);
  });
}
cudaError_t launch_batch_advance(SimDesc* sims, int n, cudaStream_t) {
  return launch("advance", [=] {
    for (int s = 0; s < n; s++) {
      SimDesc& S = sims[s];
      if (!S.active || S.sc.done || S.held) continue;
      S.sc.time += S.sc.dt;
      S.sc.tn++;
      next_dt(S);
    }
  });
}
}  // namespace hmn

#define CHECK(x)                                                  \
  do {                                                            \
    if (!(x)) return printf("line %d: %s\n", __LINE__, #x), 1;    \
  } while (0)

static int add(hmn_batch* b, int n0, int n1, bool mag) {
  hmn_grid g;
  hmn_params p;
  memset(&g, 0, sizeof(g));
  memset(&p, 0, sizeof(p));
  g.n[0] = n0, g.n[1] = n1, g.n[2] = 1;
  std::vector<double> line(n0 + n1 + 8, 1.0);
  for (int a = 0; a < 3; a++) g.x[a] = g.xi[a] = g.dx[a] = g.idx[a] = g.dxi[a] = g.idxi[a] = line.data();
  p.mag_on = mag, p.gamma = 1.4, p.courant = 0.5, p.rktype = 3;
  std::vector<double> u(9 * (size_t)n0 * n1, 1.0);
  int sim = -1;
  return hmn_batch_add(b, &g, &p, u.data(), nullptr, 0.0, 1e30, &sim) == HMN_OK ? sim : -1;
}

static long ran(const char* name) {
  long n = 0;
  for (auto& t : trace) n += t == name;
  return n;
}

// every simulation has taken `steps` steps of the full dt
static bool at(hmn_batch* b, int sim, int steps) {
  double t[8];
  int tn[8];
  return hmn_batch_poll(b, t, tn, nullptr, nullptr) == HMN_OK && tn[sim] == steps && t[sim] == steps * hmn::kDt;
}

// a step whose first launches fail leaves nothing behind: the next call starts
// the simulations anew
static int check_failed_start() {
  for (const char* what : {"cfl0", "finalize"}) {
    hmn_batch* b = nullptr;
    CHECK(hmn_batch_create(1 << 24, 8, 0, 3, &b) == HMN_OK);
    const int s = add(b, 64, 40, true);
    CHECK(s >= 0);
    fail_next = what;
    CHECK(hmn_batch_step(b, 3) == HMN_ECUDA);
    CHECK(hmn_batch_step(b, 3) == HMN_OK);
    CHECK(at(b, s, 3));
    hmn_batch_destroy(b);
  }
  return 0;
}

// the reduction that starts a simulation runs once for it, and not for those
// that others join, leave or pass by
static int check_start_once() {
  hmn_batch* b = nullptr;
  CHECK(hmn_batch_create(1 << 26, 8, 0, 3, &b) == HMN_OK);
  trace.clear();
  const int s0 = add(b, 400, 300, true), s1 = add(b, 30, 1, true);  // one class of many items, one of few
  CHECK(hmn_batch_step(b, 2) == HMN_OK && ran("cfl0") == 2 && ran("finalize") == 1);
  int held[8] = {};
  held[s1] = 1;
  CHECK(hmn_batch_set_held(b, held) == HMN_OK && hmn_batch_step(b, 3) == HMN_OK);
  held[s1] = 0;
  CHECK(hmn_batch_set_held(b, held) == HMN_OK && hmn_batch_step(b, 1) == HMN_OK);
  CHECK(ran("cfl0") == 2 && ran("finalize") == 1);
  const int s2 = add(b, 60, 1, true);  // the class of few items starts its new simulation only
  CHECK(hmn_batch_step(b, 4) == HMN_OK && ran("cfl0") == 3 && ran("finalize") == 2);
  CHECK(at(b, s0, 10) && at(b, s1, 7) && at(b, s2, 4));
  CHECK(hmn_batch_remove(b, s0) == HMN_OK && hmn_batch_step(b, 1) == HMN_OK && ran("cfl0") == 3);
  CHECK(at(b, s1, 8) && at(b, s2, 5));
  hmn_batch_destroy(b);
  return 0;
}

// the same steps whether they are launched directly or replayed from graphs,
// and graphs only for a list that lasts
static int check_graphs() {
  hmn_batch* b = nullptr;
  CHECK(hmn_batch_create(1 << 26, 8, 0, 3, &b) == HMN_OK);
  const int s0 = add(b, 400, 300, true), s1 = add(b, 30, 1, true);
  captures = 0;
  trace.clear();
  int steps = 0;
  const auto step = [&](int n) {
    steps += n;
    return hmn_batch_step(b, n) == HMN_OK && ran("advance") == steps && ran("few") == 3 * steps &&
           ran("cfl") == steps;
  };
  CHECK(step(kGraphAfter - 1) && step(1) && captures == 0);
  CHECK(step(1) && captures == 1);
  CHECK(step(kManyAfter - kGraphAfter - 1) && captures == 1);
  CHECK(step(kManySteps - 1) && step(1) && captures == 1);
  CHECK(step(3 * kManySteps + 2) && captures == 2);
  CHECK(step(kManySteps) && step(2) && captures == 2);
  CHECK(hmn_batch_launch_count(b) == 2 + (long long)trace.size());  // two launches of the additions
  CHECK(at(b, s0, steps) && at(b, s1, steps));
  const int s2 = add(b, 20, 1, true);
  CHECK(step(kGraphAfter) && captures == 2);
  CHECK(step(kManyAfter + kManySteps - kGraphAfter) && captures == 4);
  CHECK(at(b, s0, steps) && at(b, s1, steps) && at(b, s2, kManyAfter + kManySteps));
  hmn_batch_destroy(b);
  return 0;
}

int main() { return check_failed_start() || check_start_once() || check_graphs(); }
