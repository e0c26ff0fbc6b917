// hmn_batch.cu -- many independent simulations of uneven sizes on one GPU.
//
// A batch owns one device memory pool; each admitted simulation gets its
// state, its primitive planes and its geometry from the pool (admission is
// by footprint: hmn_batch_add fails with HMN_ENOMEM when the pool has no
// room) and a descriptor in a device array.  A batch step runs, for all
// simulations at once, the step of src/main/hormone.f90:126-147 on each
// simulation's own clock.  The simulations of one tile kind and physics form a
// class; the classes run side by side, each with one launch per RK stage and
// one that reduces the CFL quantities of the new state (in the last stage where
// the class has few items).  One launch for all then advances the clocks and
// forms the next dt with its clamps, so that a step ends with what the next one
// starts from.  A list of simulations that lasts is stepped by CUDA graphs.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

#include "../../include/hormone_gpu.h"
#include "hmn_internal.h"

using namespace hmn;

namespace {

struct SlotInfo {
  bool used = false;
  size_t off = 0, bytes = 0;
  int kind = -1;
  bool mag = false, glm = false;
  int nvar = 0;
  int n[3] = {1, 1, 1};
  int ntiles = 0;
};

struct Klass {
  int kind;
  int tile;          // the schedule's tile of its kind, or that of a class of few items
  bool few;          // the latter: the last stage reduces the CFL quantities too
  bool mag, glm;
  int first, count;  // range in the item list
  int grid;          // persistent CTAs of the stage launches
  bool dynamic;      // stage launches take items from the shared counter
  int* queue;        // that counter: {next item, CTAs finished}
  bool fresh;        // holds simulations that have not stepped yet
};

// Steps captured in one graph: between two replays the GPU idles a few
// microseconds, a tenth of a step of small grids.
constexpr int kManySteps = 8;
// Graphs are made for lists that last.  Capturing, instantiating and dropping a
// graph of one step costs 0.2 to 0.5 ms, of kManySteps up to 1.6 ms (24 small
// requests, six classes), and a scheduler may change the list every few steps.
// Launched directly, a step keeps the GPU as busy as the graph of one does, at
// more of the host's time; a graph of several saves 4 to 10 us per step.  So
// the first kGraphAfter steps of a list are launched directly, and a graph of
// several is captured once kManyAfter steps have shown the list to last.
// Against graphs from the first step: 1 step after a change, 24 small requests
// 694 -> 191 us, in the mixed form 632 -> 148; 8 steps 2791 -> 1210 and 2393 ->
// 895; 64 steps 10.2 -> 9.4 ms and 7.7 -> 6.8; the served stream 0.698 -> 0.687 s.
constexpr int kGraphAfter = 8, kManyAfter = 64;

constexpr int kMaxClasses = 9;  // three tile kinds x (hydro, MHD, MHD with GLM)

constexpr size_t kAlign = 256;
size_t align_up(size_t x) { return (x + kAlign - 1) / kAlign * kAlign; }

}  // namespace

struct hmn_batch {
  int max_sims = 0;
  int precision = 0;
  int rktype = 3;
  char* pool = nullptr;
  size_t pool_bytes = 0;
  std::vector<std::pair<size_t, size_t>> free_list;  // (offset, size), sorted by offset
  SimDesc* d_sims = nullptr;
  std::vector<SimDesc> h_sims;
  std::vector<SlotInfo> slots;
  int2* d_items = nullptr;
  size_t items_cap = 0;
  std::vector<Klass> classes;
  int listed = 0;  // simulations in the work list
  bool dirty = true;
  cudaStream_t st = nullptr;
  int nsm = 148;
  int blocks_per_sm[3] = {0, 0, 0};  // per tile kind; 0: occupancy-derived persistent grid
  int tile_id[3] = {0, 2, 4};         // tile of each kind (batch_tile_variants)
  int sweep[3] = {HMN_SWEEP_STATIC, HMN_SWEEP_STATIC, HMN_SWEEP_STATIC};  // item order and split per kind
  int* d_queue = nullptr;             // one counter pair per class: classes run side by side
  cudaStream_t side[kMaxClasses] = {};  // branches of the captured step beside st (classes 1, 2, ...)
  cudaEvent_t fork = nullptr, join[kMaxClasses] = {};
  cudaGraphExec_t graph = nullptr, graph_many = nullptr;  // one step; kManySteps steps
  long long step_launches = 0;        // kernel launches of one step
  long long ran = 0;                  // steps issued since the work list was made
  long long launches = 0;
  double* stage_h = nullptr;
  size_t stage_h_bytes = 0;
};

static void drop_graphs(hmn_batch* b) {
  if (b->graph) cudaGraphExecDestroy(b->graph);
  if (b->graph_many) cudaGraphExecDestroy(b->graph_many);
  b->graph = b->graph_many = nullptr;
}

static int cuda_fail(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return HMN_OK;
  fprintf(stderr, "hormone_b200 batch: %s: %s\n", what, cudaGetErrorString(e));
  return e == cudaErrorMemoryAllocation ? HMN_ENOMEM : HMN_ECUDA;
}
#define BCK(call, what)                       \
  do {                                        \
    cudaError_t _e = (call);                  \
    if (_e != cudaSuccess) return cuda_fail(_e, what); \
  } while (0)

static size_t sim_bytes(const int n[3], int nvar) {
  const size_t plane = (size_t)n[0] * n[1] * n[2];
  size_t b = 0;
  b += 3 * align_up((size_t)nvar * plane * sizeof(double));  // U[0..2]
  b += 2 * align_up((size_t)10 * plane * sizeof(double));    // P[0..1]
  for (int a = 0; a < 3; a++) b += align_up((size_t)kGeoArrays * (n[a] + 4) * sizeof(double));
  return b;
}

static bool pool_alloc(hmn_batch* b, size_t bytes, size_t* off) {
  for (size_t i = 0; i < b->free_list.size(); i++) {
    auto& f = b->free_list[i];
    if (f.second >= bytes) {
      *off = f.first;
      f.first += bytes;
      f.second -= bytes;
      if (f.second == 0) b->free_list.erase(b->free_list.begin() + i);
      return true;
    }
  }
  return false;
}

static void pool_free(hmn_batch* b, size_t off, size_t bytes) {
  b->free_list.push_back({off, bytes});
  std::sort(b->free_list.begin(), b->free_list.end());
  std::vector<std::pair<size_t, size_t>> merged;
  for (auto& f : b->free_list) {
    if (!merged.empty() && merged.back().first + merged.back().second == f.first)
      merged.back().second += f.second;
    else
      merged.push_back(f);
  }
  b->free_list.swap(merged);
}

extern "C" size_t hmn_batch_footprint(const hmn_grid* grid, const hmn_params* par) {
  if (!grid || !par) return 0;
  int dim = 0;
  for (int a = 0; a < 3; a++) dim += grid->n[a] > 1;
  const bool glm = par->mag_on && dim > 1;
  const int nvar = 5 + (par->mag_on ? 3 : 0) + (glm ? 1 : 0);
  return sim_bytes(grid->n, nvar);
}

extern "C" int hmn_batch_create(size_t pool_bytes, int max_sims, int precision, int rktype, hmn_batch** out) {
  if (!out || max_sims < 1 || pool_bytes < kAlign || (precision != 0 && precision != 1) || rktype < 1 || rktype > 3)
    return HMN_EINVAL;
  *out = nullptr;
  hmn_batch* b = new (std::nothrow) hmn_batch();
  if (!b) return HMN_ENOMEM;
  b->max_sims = max_sims;
  b->precision = precision;
  b->rktype = rktype;
  b->pool_bytes = align_up(pool_bytes);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&b->nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc((void**)&b->pool, b->pool_bytes);
  if (e == cudaSuccess) e = cudaMalloc((void**)&b->d_sims, (size_t)max_sims * sizeof(SimDesc));
  if (e == cudaSuccess) e = cudaMemset(b->d_sims, 0, (size_t)max_sims * sizeof(SimDesc));
  if (e == cudaSuccess) e = cudaMalloc((void**)&b->d_queue, 2 * kMaxClasses * sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(b->d_queue, 0, 2 * kMaxClasses * sizeof(int));
  if (e != cudaSuccess) {
    int rc = cuda_fail(e, "batch create");
    hmn_batch_destroy(b);
    return rc;
  }
  b->h_sims.assign(max_sims, SimDesc());
  memset(b->h_sims.data(), 0, (size_t)max_sims * sizeof(SimDesc));
  b->slots.assign(max_sims, SlotInfo());
  b->free_list.push_back({0, b->pool_bytes});
  *out = b;
  return HMN_OK;
}

extern "C" int hmn_batch_destroy(hmn_batch* b) {
  if (!b) return HMN_EINVAL;
  if (b->st) cudaStreamSynchronize(b->st);
  drop_graphs(b);
  cudaFree(b->pool);
  cudaFree(b->d_sims);
  cudaFree(b->d_items);
  cudaFree(b->d_queue);
  if (b->stage_h) cudaFreeHost(b->stage_h);
  if (b->fork) cudaEventDestroy(b->fork);
  for (int c = 0; c < kMaxClasses; c++) {
    if (b->join[c]) cudaEventDestroy(b->join[c]);
    if (b->side[c]) cudaStreamDestroy(b->side[c]);
  }
  if (b->st) cudaStreamDestroy(b->st);
  delete b;
  return HMN_OK;
}

// geometry arrays of one axis exactly as hmn_create derives them
static void axis_geometry(const hmn_grid* grid, int a, double* base) {
  const int L = grid->n[a] + 4;
  const double *x = grid->x[a], *xi = grid->xi[a];
  for (int s = 0; s < kGeoArrays * L; s++) base[s] = 0.0;
  for (int s = 0; s < L; s++) {
    base[0 * L + s] = x[s];
    base[1 * L + s] = grid->dx[a][s];
    base[2 * L + s] = grid->idx[a][s];
    base[3 * L + s] = grid->dxi[a][s];
    base[4 * L + s] = grid->idxi[a][s];
  }
  for (int s = 1; s < L; s++) base[5 * L + s] = x[s] - xi[s - 1];
  for (int s = 0; s < L; s++) base[6 * L + s] = xi[s] - x[s];
  for (int s = 1; s + 1 < L; s++) {
    base[7 * L + s] = (x[s + 1] - x[s]) / (xi[s] - x[s]);
    base[8 * L + s] = (x[s] - x[s - 1]) / (x[s] - xi[s - 1]);
    base[9 * L + s] = x[s + 1] - x[s];
    base[10 * L + s] = x[s] - x[s - 1];
    base[11 * L + s] = grid->idx[a][s] + grid->idx[a][s + 1];
    base[12 * L + s] = 1.0 / base[9 * L + s];
    base[13 * L + s] = base[9 * L + s] / base[10 * L + s];
    base[14 * L + s] = 1.0 / base[11 * L + s];
  }
}

static int ensure_stage(hmn_batch* b, size_t bytes) {
  if (b->stage_h_bytes >= bytes) return HMN_OK;
  if (b->stage_h) cudaFreeHost(b->stage_h);
  b->stage_h = nullptr;
  b->stage_h_bytes = 0;
  BCK(cudaMallocHost((void**)&b->stage_h, bytes), "pinned staging");
  b->stage_h_bytes = bytes;
  return HMN_OK;
}

extern "C" int hmn_batch_add(hmn_batch* b, const hmn_grid* grid, const hmn_params* par, const double* u,
                             const double* const prim[9], double time, double t_end, int* sim) {
  if (!b || !grid || !par || !u || !sim) return HMN_EINVAL;
  if (grid->ghost != 0 || par->gravswitch != 0 || par->rktype != b->rktype || par->limiter < 0 ||
      par->limiter > 2 || par->nspc != 0)
    return HMN_EBADCFG;
  int solve[3], dim = 0;
  for (int a = 0; a < 3; a++) {
    if (grid->n[a] < 1) return HMN_EINVAL;
    solve[a] = grid->n[a] > 1;
    dim += solve[a];
    if (solve[a]) {
      if (grid->n[a] < 2) return HMN_EBADCFG;
      for (int io = 0; io < 2; io++)
        for (int sv = 0; sv < 2; sv++)
          if (grid->bc[a][io][sv] < 0 || grid->bc[a][io][sv] > 5) return HMN_EBADCFG;  // codes 0-5
    }
  }
  const int kind = batch_tile_kind(solve);
  if (kind < 0) return HMN_EBADCFG;
  int slot = -1;
  for (int s = 0; s < b->max_sims; s++)
    if (!b->slots[s].used) {
      slot = s;
      break;
    }
  if (slot < 0) return HMN_ENOMEM;
  const bool mag = par->mag_on != 0, glm = mag && dim > 1;
  const int nvar = 5 + (mag ? 3 : 0) + (glm ? 1 : 0);
  const size_t bytes = sim_bytes(grid->n, nvar);
  size_t off;
  if (!pool_alloc(b, bytes, &off)) return HMN_ENOMEM;  // admission by footprint
  SlotInfo& si = b->slots[slot];
  si.used = true;
  si.off = off;
  si.bytes = bytes;
  si.kind = kind;
  si.mag = mag;
  si.glm = glm;
  si.nvar = nvar;
  for (int a = 0; a < 3; a++) si.n[a] = grid->n[a];
  SimDesc& S = b->h_sims[slot];
  memset(&S, 0, sizeof(S));
  const size_t plane = (size_t)grid->n[0] * grid->n[1] * grid->n[2];
  char* p = b->pool + off;
  for (int q = 0; q < 3; q++) {
    S.U[q] = (double*)p;
    p += align_up((size_t)nvar * plane * sizeof(double));
  }
  for (int q = 0; q < 2; q++) {
    S.P[q] = (double*)p;
    p += align_up((size_t)10 * plane * sizeof(double));
  }
  // geometry
  size_t geo_total = 0;
  for (int a = 0; a < 3; a++) geo_total += (size_t)kGeoArrays * (grid->n[a] + 4);
  int rc = ensure_stage(b, std::max(geo_total, (size_t)10 * plane) * sizeof(double));
  if (rc) {
    pool_free(b, off, bytes);
    si.used = false;
    return rc;
  }
  BCK(cudaStreamSynchronize(b->st), "sync");
  {
    double* h = b->stage_h;
    for (int a = 0; a < 3; a++) {
      const int L = grid->n[a] + 4;
      axis_geometry(grid, a, h);
      double* dbase = (double*)p;
      BCK(cudaMemcpyAsync(dbase, h, (size_t)kGeoArrays * L * sizeof(double), cudaMemcpyHostToDevice, b->st), "geo");
      BCK(cudaStreamSynchronize(b->st), "sync");
      AxisGeo& g = S.G.g[a];
      g.x = dbase + 0 * L;
      g.dx = dbase + 1 * L;
      g.idx = dbase + 2 * L;
      g.dxi = dbase + 3 * L;
      g.idxi = dbase + 4 * L;
      g.hl = dbase + 5 * L;
      g.hr = dbase + 6 * L;
      g.mcf = dbase + 7 * L;
      g.mcb = dbase + 8 * L;
      g.ga = dbase + 9 * L;
      g.gb = dbase + 10 * L;
      g.isum = dbase + 11 * L;
      g.rga = dbase + 12 * L;
      g.gab = dbase + 13 * L;
      g.risum = dbase + 14 * L;
      p += align_up((size_t)kGeoArrays * L * sizeof(double));
    }
  }
  for (int a = 0; a < 3; a++) {
    S.G.n[a] = grid->n[a];
    S.G.solve[a] = solve[a];
  }
  memcpy(S.G.bc, grid->bc, sizeof(S.G.bc));
  int tile[3];
  batch_tile_shape(b->tile_id[kind], tile);
  for (int a = 0; a < 3; a++) S.tiles[a] = (grid->n[a] + tile[a] - 1) / tile[a];
  si.ntiles = S.tiles[0] * S.tiles[1] * S.tiles[2];
  S.plane = plane;
  S.pcur = 0;
  S.nvar = nvar;
  S.limiter = par->limiter;
  S.rktype = par->rktype;
  S.glm = glm;
  S.active = 1;
  S.fresh = 1;
  S.gamma = par->gamma;
  S.gm1 = par->gamma - 1.0;
  S.damp = std::exp(-par->alpha9wave * par->courant);
  S.phifac = 1.0;
  S.sc.min_dti_bits = 0x7ff0000000000000ULL;
  S.sc.cfmax_bits = 0ULL;
  S.sc.time = time;
  S.sc.t_out = t_end;
  S.sc.t_end = t_end;
  S.sc.courant = par->courant;
  S.sc.outstyle = 1;
  S.sc.endstyle = 1;
  // state: u and the primitives as the reference holds them after start-up
  BCK(cudaMemcpyAsync(S.U[0], u, (size_t)nvar * plane * sizeof(double), cudaMemcpyHostToDevice, b->st), "upload u");
  if (prim) {
    for (int q = 0; q < 9; q++) {
      if (prim[q])
        BCK(cudaMemcpyAsync(S.P[0] + q * plane, prim[q], plane * sizeof(double), cudaMemcpyHostToDevice, b->st),
            "upload prim");
      else
        BCK(cudaMemsetAsync(S.P[0] + q * plane, 0, plane * sizeof(double), b->st), "memset");
    }
    BCK(launch_prim_init(S.P[0], plane, mag, (int)std::min<size_t>((plane + 255) / 256, (size_t)b->nsm * 8), b->st),
        "prim init");
  } else {
    BCK(launch_prim_from_u(S.U[0], S.P[0], plane, mag, glm, (int)std::min<size_t>((plane + 255) / 256, (size_t)b->nsm * 8),
                           b->st),
        "prim");
  }
  b->launches += 1;
  BCK(cudaMemcpyAsync(b->d_sims + slot, &S, sizeof(SimDesc), cudaMemcpyHostToDevice, b->st), "descriptor");
  BCK(cudaStreamSynchronize(b->st), "sync");
  b->dirty = true;
  *sim = slot;
  return HMN_OK;
}

extern "C" int hmn_batch_remove(hmn_batch* b, int sim) {
  if (!b || sim < 0 || sim >= b->max_sims || !b->slots[sim].used) return HMN_EINVAL;
  BCK(cudaStreamSynchronize(b->st), "sync");
  SlotInfo& si = b->slots[sim];
  pool_free(b, si.off, si.bytes);
  si = SlotInfo();
  SimDesc& S = b->h_sims[sim];
  memset(&S, 0, sizeof(S));
  BCK(cudaMemcpyAsync(b->d_sims + sim, &S, sizeof(SimDesc), cudaMemcpyHostToDevice, b->st), "descriptor");
  BCK(cudaStreamSynchronize(b->st), "sync");
  b->dirty = true;
  return HMN_OK;
}

// pull every descriptor (clocks, done flags, errors) to the host mirror
static int pull(hmn_batch* b) {
  BCK(cudaMemcpyAsync(b->h_sims.data(), b->d_sims, (size_t)b->max_sims * sizeof(SimDesc), cudaMemcpyDeviceToHost,
                      b->st),
      "poll");
  BCK(cudaStreamSynchronize(b->st), "sync");
  return HMN_OK;
}

// Hold (held[s] = 1) or release simulations: a held simulation is left out
// of every step (its clock, state and CFL partials stay as they are) until
// it is released, so a scheduler can advance some simulations alone.
extern "C" int hmn_batch_set_held(hmn_batch* b, const int* held) {
  if (!b || !held) return HMN_EINVAL;
  int rc = pull(b);
  if (rc) return rc;
  bool changed = false;
  for (int s = 0; s < b->max_sims; s++) {
    const int h = b->slots[s].used && held[s] ? 1 : 0;
    if (b->h_sims[s].held != h) changed = true;
    b->h_sims[s].held = h;
  }
  if (!changed) return HMN_OK;
  BCK(cudaMemcpyAsync(b->d_sims, b->h_sims.data(), (size_t)b->max_sims * sizeof(SimDesc), cudaMemcpyHostToDevice,
                      b->st),
      "descriptor");
  BCK(cudaStreamSynchronize(b->st), "sync");
  b->dirty = true;
  return HMN_OK;
}

static int start_steps(hmn_batch* b);

static int tiles_of(const int n[3], const int t[3]) {
  return ((n[0] + t[0] - 1) / t[0]) * ((n[1] + t[1] - 1) / t[1]) * ((n[2] + t[2] - 1) / t[2]);
}

static int rebuild(hmn_batch* b) {
  // work list: active, unfinished simulations grouped by (tile kind, mag, glm)
  std::vector<int2> items;
  b->classes.clear();
  for (int kind = 0; kind < 3; kind++)  // the tile kinds of batch_tile_kind
    for (int m = 0; m < 3; m++) {
      const bool mag = m > 0, glm = m == 2;
      const int sweep = b->sweep[kind];
      Klass k{kind, b->tile_id[kind], false, mag, glm, (int)items.size(), 0, 0, sweep == HMN_SWEEP_DYNAMIC, nullptr, false};
      std::vector<int> sims;
      int most_tiles = 0;
      for (int s = 0; s < b->max_sims; s++) {
        const SlotInfo& si = b->slots[s];
        if (!si.used || si.kind != kind || si.mag != mag || si.glm != glm || b->h_sims[s].sc.done ||
            b->h_sims[s].held)
          continue;
        sims.push_back(s);
        k.fresh |= b->h_sims[s].fresh != 0;
        most_tiles = std::max(most_tiles, si.ntiles);
      }
      // items of each listed simulation: the schedule's tiles, or smaller ones
      // where those are few (FP64)
      std::vector<int> ntiles(b->max_sims, 0);
      for (int s : sims) ntiles[s] = b->slots[s].ntiles;
      if (b->precision == 0 && !sims.empty()) {
        int most, few[3];
        const int id = batch_few_tile(kind, b->nsm, &most);
        batch_tile_shape(id, few);
        long long count = 0;
        for (int s : sims) count += tiles_of(b->slots[s].n, few);
        if (count <= most) {
          k.few = true;
          k.tile = id;
          k.dynamic = false;
          most_tiles = 0;
          for (int s : sims) {
            ntiles[s] = tiles_of(b->slots[s].n, few);
            most_tiles = std::max(most_tiles, ntiles[s]);
          }
        }
      }
      if (sweep == HMN_SWEEP_INTERLEAVED) {  // tile t of every simulation, then tile t + 1
        for (int t = 0; t < most_tiles; t++)
          for (int s : sims)
            if (t < ntiles[s]) items.push_back(make_int2(s, t));
      } else {
        if (sweep == HMN_SWEEP_DYNAMIC)  // the largest simulations first
          std::stable_sort(sims.begin(), sims.end(),
                           [b](int x, int y) { return b->slots[x].ntiles > b->slots[y].ntiles; });
        for (int s : sims)
          for (int t = 0; t < ntiles[s]; t++) items.push_back(make_int2(s, t));
      }
      k.count = (int)items.size() - k.first;
      if (k.count) {
        // occupancy queries run here, outside any stream capture
        int per = b->blocks_per_sm[kind];
        if (k.few)
          BCK(launch_batch_stage(b->d_sims, nullptr, 0, k.tile, mag, glm, 1, b->rktype, 0, 0, nullptr, b->st), "stage");
        else if (per <= 0)
          per = batch_stage_blocks_per_sm(b->tile_id[kind], mag, glm, b->precision);
        k.grid = k.few ? k.count : (int)std::min<long long>((long long)per * b->nsm, k.count);
        k.queue = b->d_queue + 2 * b->classes.size();
        b->classes.push_back(k);
      }
    }
  if (items.size() > b->items_cap) {
    cudaFree(b->d_items);
    b->d_items = nullptr;
    b->items_cap = std::max(items.size(), (size_t)1024);
    BCK(cudaMalloc((void**)&b->d_items, b->items_cap * sizeof(int2)), "items");
  }
  if (!items.empty())
    BCK(cudaMemcpyAsync(b->d_items, items.data(), items.size() * sizeof(int2), cudaMemcpyHostToDevice, b->st),
        "items");
  BCK(cudaStreamSynchronize(b->st), "sync");
  drop_graphs(b);
  b->ran = 0;
  b->listed = 0;
  for (const Klass& k : b->classes)
    for (int i = 0; i < k.count; i++) b->listed += items[(size_t)k.first + i].y == 0;
  // the branches of the captured step, made outside any capture
  if (b->classes.size() > 1 && !b->fork)
    BCK(cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming), "fork event");
  for (size_t c = 1; c < b->classes.size(); c++) {
    if (!b->side[c]) BCK(cudaStreamCreateWithFlags(&b->side[c], cudaStreamNonBlocking), "side stream");
    if (!b->join[c]) BCK(cudaEventCreateWithFlags(&b->join[c], cudaEventDisableTiming), "join event");
  }
  // the list stands once its steps can start; until then the next step makes it anew
  const int rc = start_steps(b);
  b->dirty = rc != HMN_OK;
  return rc;
}

// Run f(class, stream) for every class: the first on the batch's stream, the
// others on branches that start here and end before what follows on it.
template <class F>
static int for_each_class(hmn_batch* b, F&& f) {
  const size_t n = b->classes.size();
  if (n > 1) BCK(cudaEventRecord(b->fork, b->st), "fork");
  int rc = HMN_OK;
  for (size_t c = 0; c < n; c++) {
    if (c > 0) BCK(cudaStreamWaitEvent(b->side[c], b->fork, 0), "fork");
    const int r = f(b->classes[c], c > 0 ? b->side[c] : b->st);
    if (r && !rc) rc = r;
    if (c > 0) BCK(cudaEventRecord(b->join[c], b->side[c]), "join");
  }
  for (size_t c = 1; c < n; c++) BCK(cudaStreamWaitEvent(b->st, b->join[c], 0), "join");
  return rc;
}

static int enqueue_cfl(hmn_batch* b, const Klass& k, int after, cudaStream_t st) {
  BCK(launch_batch_cfl(b->d_sims, b->d_items + k.first, k.count, k.tile, k.mag, after, std::min(k.count, b->nsm * 4),
                       st),
      "batch cfl");
  return HMN_OK;
}

// The first dt of the simulations that have not stepped yet; every step then
// ends with the next one's, which a simulation keeps while others join, leave
// or are held.
static int start_steps(hmn_batch* b) {
  int started = 0;
  for (const Klass& k : b->classes) {
    if (!k.fresh) continue;
    const int rc = enqueue_cfl(b, k, 0, b->st);
    if (rc) return rc;
    started++;
  }
  if (started == 0) return HMN_OK;
  BCK(launch_batch_finalize(b->d_sims, b->max_sims, b->st), "batch finalize");
  b->launches += started + 1;
  return HMN_OK;
}

// One step of every listed simulation: its RK stages, the CFL reduction of the
// new state, and the advance of the clocks with the next dt.  A simulation is
// in one class and the launches of a class touch nothing of another's
// simulations, so the classes run side by side, as branches of the captured
// graph: a served stream of small 1-D, 2-D and 3-D grids waits on latency, and
// its step is as long as the slowest class instead of their sum (24 requests
// 1.00 -> 0.89 s).  With the tiles of classes of few items, the reduction in
// their last stage, the clocks' two kernels in one and several steps per graph
// the same stream takes 0.67 s.
static int enqueue_step(hmn_batch* b, long long* nlaunch) {
  const int rc = for_each_class(b, [&](const Klass& k, cudaStream_t st) {
    for (int s = 1; s <= b->rktype; s++) {
      BCK(launch_batch_stage(b->d_sims, b->d_items + k.first, k.count, k.tile, k.mag, k.glm, s, b->rktype,
                             b->precision, k.grid, k.dynamic ? k.queue : nullptr, st),
          "batch stage");
      (*nlaunch)++;
    }
    if (k.few) return (int)HMN_OK;
    (*nlaunch)++;
    return enqueue_cfl(b, k, b->rktype, st);
  });
  if (rc) return rc;
  BCK(launch_batch_advance(b->d_sims, b->max_sims, b->st), "batch advance");
  (*nlaunch)++;
  return HMN_OK;
}

// `steps` steps as one graph; replaying it advances every simulation by that many
static int capture_steps(hmn_batch* b, int steps, cudaGraphExec_t* out) {
  cudaGraph_t g;
  BCK(cudaStreamBeginCapture(b->st, cudaStreamCaptureModeThreadLocal), "capture");
  int rc = HMN_OK;
  for (int s = 0; s < steps && rc == HMN_OK; s++) {
    b->step_launches = 0;
    rc = enqueue_step(b, &b->step_launches);
  }
  cudaError_t e = cudaStreamEndCapture(b->st, &g);
  if (rc) {
    if (e == cudaSuccess) cudaGraphDestroy(g);
    return rc;
  }
  BCK(e, "capture end");
  e = cudaGraphInstantiate(out, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) *out = nullptr;
  BCK(e, "graph instantiate");
  return HMN_OK;
}

extern "C" int hmn_batch_step(hmn_batch* b, int nsteps) {
  if (!b || nsteps < 0) return HMN_EINVAL;
  if (b->dirty) {
    int rc = pull(b);
    if (rc) return rc;
    rc = rebuild(b);
    if (rc) return rc;
  }
  if (b->classes.empty() || nsteps == 0) return HMN_OK;
  int left = nsteps;
  while (left > 0) {
    const bool many = left >= kManySteps && (b->graph_many || b->ran >= kManyAfter);
    const int n = many ? kManySteps : 1;
    if (!many && !b->graph && b->ran < kGraphAfter) {
      const int rc = enqueue_step(b, &b->launches);
      if (rc) return rc;
    } else {
      cudaGraphExec_t* g = many ? &b->graph_many : &b->graph;
      if (!*g) {
        const int rc = capture_steps(b, n, g);
        if (rc) return rc;
      }
      BCK(cudaGraphLaunch(*g, b->st), "graph launch");
      b->launches += b->step_launches * n;
    }
    b->ran += n;
    left -= n;
  }
  return HMN_OK;
}

extern "C" int hmn_batch_poll(hmn_batch* b, double* time, int* tn, int* done, int* err) {
  if (!b) return HMN_EINVAL;
  int rc = pull(b);
  if (rc) return rc;
  bool any_done = false;
  for (int s = 0; s < b->max_sims; s++) {
    const SimDesc& S = b->h_sims[s];
    if (time) time[s] = S.sc.time;
    if (tn) tn[s] = S.sc.tn;
    if (done) done[s] = b->slots[s].used ? S.sc.done : 0;
    if (err) err[s] = S.sc.err_code;
    if (b->slots[s].used && S.sc.done) any_done = true;
  }
  // drop finished simulations from the work list at the next step: the list
  // is rebuilt only when it lists another number of simulations than are used,
  // unfinished and not held, so a finished simulation left in its slot does not
  // force a rebuild and graph re-capture at every poll
  if (any_done) {
    int want = 0;
    for (int s = 0; s < b->max_sims; s++)
      if (b->slots[s].used && !b->h_sims[s].sc.done && !b->h_sims[s].held) want++;
    if (want != b->listed) b->dirty = true;
  }
  return HMN_OK;
}

extern "C" int hmn_batch_download(hmn_batch* b, int sim, double* u, double* const prim[9]) {
  if (!b || sim < 0 || sim >= b->max_sims || !b->slots[sim].used) return HMN_EINVAL;
  int rc = pull(b);
  if (rc) return rc;
  const SimDesc& S = b->h_sims[sim];
  const SlotInfo& si = b->slots[sim];
  if (u)
    BCK(cudaMemcpyAsync(u, S.U[0], (size_t)si.nvar * S.plane * sizeof(double), cudaMemcpyDeviceToHost, b->st),
        "download u");
  if (prim) {
    // primitives of the current state; phi carries the pending phidamp factor
    const double* Pc = S.P[S.pcur];
    for (int q = 0; q < 9; q++)
      if (prim[q])
        BCK(cudaMemcpyAsync(prim[q], Pc + q * S.plane, S.plane * sizeof(double), cudaMemcpyDeviceToHost, b->st),
            "download prim");
    BCK(cudaStreamSynchronize(b->st), "sync");
    if (prim[8] && S.phifac != 1.0)
      for (size_t c = 0; c < S.plane; c++) prim[8][c] = prim[8][c] * S.phifac;
  }
  BCK(cudaStreamSynchronize(b->st), "sync");
  return S.sc.err_code;
}

extern "C" int hmn_batch_set_schedule(hmn_batch* b, int kind, int tile_id, int blocks_per_sm) {
  if (!b || kind < 0 || kind > 2 || blocks_per_sm < 0) return HMN_EINVAL;
  int ids[4], nv = batch_tile_variants(kind, ids);
  bool ok = false;
  for (int v = 0; v < nv; v++) ok = ok || ids[v] == tile_id;
  if (!ok) return HMN_EINVAL;
  BCK(cudaStreamSynchronize(b->st), "sync");
  b->blocks_per_sm[kind] = blocks_per_sm;
  if (tile_id != b->tile_id[kind]) {
    b->tile_id[kind] = tile_id;
    int tile[3];
    batch_tile_shape(tile_id, tile);
    int rc = pull(b);
    if (rc) return rc;
    for (int s = 0; s < b->max_sims; s++) {
      SlotInfo& si = b->slots[s];
      if (!si.used || si.kind != kind) continue;
      SimDesc& S = b->h_sims[s];
      for (int a = 0; a < 3; a++) S.tiles[a] = (si.n[a] + tile[a] - 1) / tile[a];
      si.ntiles = S.tiles[0] * S.tiles[1] * S.tiles[2];
      BCK(cudaMemcpyAsync(&b->d_sims[s].tiles, S.tiles, sizeof(S.tiles), cudaMemcpyHostToDevice, b->st), "tiles");
    }
    BCK(cudaStreamSynchronize(b->st), "sync");
  }
  b->dirty = true;
  drop_graphs(b);
  return HMN_OK;
}

extern "C" int hmn_batch_set_sweep(hmn_batch* b, int kind, int sweep) {
  if (!b || kind < 0 || kind > 2 || sweep < HMN_SWEEP_STATIC || sweep > HMN_SWEEP_DYNAMIC) return HMN_EINVAL;
  BCK(cudaStreamSynchronize(b->st), "sync");
  if (sweep == b->sweep[kind]) return HMN_OK;
  b->sweep[kind] = sweep;
  b->dirty = true;  // the next step rebuilds the work list and its graph
  return HMN_OK;
}

extern "C" long long hmn_batch_launch_count(hmn_batch* b) { return b ? b->launches : -1; }

extern "C" int hmn_batch_sync(hmn_batch* b) {
  if (!b) return HMN_EINVAL;
  BCK(cudaStreamSynchronize(b->st), "sync");
  return HMN_OK;
}

extern "C" void* hmn_batch_stream(hmn_batch* b) { return b ? (void*)b->st : nullptr; }
