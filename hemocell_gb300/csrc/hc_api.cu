// C ABI of the GB300 HemoCell IB-LBM step: handle lifecycle, device memory,
// stage orchestration (HemoCell::iterate, core/hemoCell.cpp:299-376), CUDA
// graph replay for the batched form, readback and launch autotuning.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <filesystem>
#include <fstream>
#include <functional>
#include <map>
#include <mutex>
#include <numeric>
#include <sstream>
#include <string>
#include <vector>

#include "../../include/hemocell_gb300.h"
#include "hc_d3q19.cuh"
#include "hc_dev.h"
#include "hc_host.h"

using hcd::LbmView;
using hcd::MechView;
using hcd::TileGrid;
using hcd::TypeDev;
using hcd::VertexView;

namespace {
std::string g_create_error;

struct TypeSlot {
  std::string name;
  hcg::TypeConstants tc;
  hcg::ModelK k;
  void* blob = nullptr;  // device arrays of this type
  TypeDev dev;
  int every = 1;
  std::vector<int> cells;
  int* dcells = nullptr;
  int dcells_cap = 0;
  bool cluster16 = false;  // the device can hold this type's staged assembly on 16 CTAs a cell
};
}  // namespace

struct hc_handle {
  hc_params p;
  hcg::Units u;
  std::string err;
  cudaStream_t stream = nullptr;
  int nx = 0, ny = 0, nz = 0;
  long long N = 0;
  bool f64 = true;
  size_t ts = 8;  // sizeof(T)
  void* f[2] = {nullptr, nullptr};
  void* F[2] = {nullptr, nullptr};
  int cur = 0;
  uint32_t* nbmask = nullptr;
  uint8_t* flag = nullptr;
  uint8_t* corner = nullptr;
  uint32_t* ntag = nullptr;
  void* unode = nullptr;
  uint32_t* stamp = nullptr;
  void* bodyz = nullptr;
  std::vector<uint8_t> hflag;
  double uw[hcd::MAX_WALL_CLASSES][3];
  int body_mode = 0;
  double body[3] = {0, 0, 0};
  // cells
  std::vector<TypeSlot> types;
  TypeDev* dtypes = nullptr;
  long long Vcap = 0;
  int nvert = 0;
  double* x = nullptr;
  void* v = nullptr;
  void* fv = nullptr;
  int* vcell = nullptr;
  int* vnode = nullptr;
  int* vtile = nullptr;
  int cellcap = 0, ncells = 0;
  int* cell_type = nullptr;
  int* cell_voff = nullptr;
  int* alive = nullptr;
  int* dcells_all = nullptr;
  std::vector<int> h_cell_type, h_cell_voff;
  unsigned int* status = nullptr;
  // binning
  TileGrid tg;
  int ntiles = 0;
  int* bin_counts = nullptr;
  int* bin_cursor = nullptr;
  int* bin_offsets = nullptr;
  int* tile_vertices = nullptr;
  int* tile_cell_counts = nullptr;
  int* tile_cell_offsets = nullptr;
  int* tile_cells = nullptr;
  long long bin_vcap = 0;
  // stepping
  int iter = 0;
  int velocity_every = 1;
  // k1 bx (0: row-staged, blocks of whole x-rows), k1 by, spread bs, ibm bs, mech bs, mech grid,
  // mech variant (0 vertex gather, 1 face/edge scatter, 2 staged gather)
  int tune[8] = {64, 2, 128, 128, 384, 0, 0, 0};
  bool tuned = false;  // tune is the caller's (hc_set_tuning, hc_autotune), not the rules' (apply_rules)
  int sms = 1;         // SMs of the device
  int l2 = 0;          // bytes of its L2
  int staged_limit = 0;  // dynamic shared memory the staged force assembly may take
  // repulsion (setRepulsion / enableBoundaryParticles): constants, cutoffs in
  // lattice units, timescales (0 = off) and device state
  double rep_k = 0, rep_rc = 0, brep_k = 0, brep_rc = 0;
  int rep_every = 0, brep_every = 0;
  int2* rep_cnt = nullptr;
  int* rep_slot = nullptr;
  int* rep_vq = nullptr;
  void* rep_xr = nullptr;
  uint8_t* rep_bnode = nullptr;
  void* frep_cell = nullptr;
  void* frep_wall = nullptr;
  long long rep_vcap = 0;
  // fluid nodes in lattice order, packed (collide-stream and node velocity over them)
  uint32_t* fluid = nullptr;
  int nfluid = 0;
  long long fluid_cap = 0;
  // bulk-copy collide-stream plan for tune[7] (stages | CTAs per SM << 4)
  hcd::BulkPlan bulk{};
  int bulk_key = 0;
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  // one-step graphs (iterate(1)), per buffer parity, built on first use
  cudaGraphExec_t graph1[2] = {nullptr, nullptr};
  // with timescale separation: a graph of one whole cycle of cycle_len steps
  // (the least common multiple of 2 and every timescale), captured starting
  // at an iteration that is a multiple of it, per buffer parity there
  cudaGraphExec_t cycle_graph[2] = {nullptr, nullptr};
  int cycle_len = 0;
  bool graph_valid = false;
  long long device_bytes = 0;
  cudaMemPool_t pool = nullptr;  // this device's library pool (all allocations)
  double* scratch = nullptr;  // readback staging
  size_t scratch_bytes = 0;
  // the spread of the coming step was already done by the last mechanics
  // pass (fused spread); anything that changes forces, positions or the
  // force field between steps clears it
  bool spread_done = false;
  // the last force assembly interpolated and advanced the vertices itself and
  // tagged the stencil nodes with stamp + 1: the next collide-stream (or a
  // state change) advances the stamp
  bool stamp_ahead = false;
  // body-force profile staging: pinned, mapped host [profile 3 nz | change
  // 3 nz] of T (and its device address), the device copy of the change, and
  // the event of the last upload
  void* hbody_pin = nullptr;
  void* hbody_dev = nullptr;
  void* bodyd = nullptr;
  cudaEvent_t body_copied = nullptr;
  // asynchronous position readback (hc_read_positions_async): a copy stream,
  // two device staging buffers of [V][3] doubles and their events
  cudaStream_t copy_stream = nullptr;
  double* pos_stage[2] = {nullptr, nullptr};
  long long pos_stage_v = 0;
  cudaEvent_t pos_ready[2] = {nullptr, nullptr}, pos_copied[2] = {nullptr, nullptr};
  bool pos_inflight[2] = {false, false};
  // per-kernel profile of the step (hc_profile_kernels): while prof_step >= 0,
  // enq_step records prof_ev[prof_step * 6 + slot] around its kernels
  std::vector<cudaEvent_t> prof_ev;
  int prof_step = -1;
  // external vertex forces (HemoCellStretch)
  int next = 0, next_cap = 0;
  int* ext_ids = nullptr;
  double* ext_f = nullptr;
};

namespace {

#define HC_CUDA(h, call)                                                                        \
  do {                                                                                         \
    cudaError_t e_ = (call);                                                                   \
    if (e_ != cudaSuccess) {                                                                   \
      (h)->err = std::string(#call) + ": " + cudaGetErrorString(e_);                           \
      return HC_ERR_CUDA;                                                                      \
    }                                                                                          \
  } while (0)

// CUDA events owned by one call: destroyed on every return path, including
// the early returns of HC_CUDA.
template <int K>
struct ScopedEvents {
  cudaEvent_t e[K] = {};
  ScopedEvents() = default;
  ScopedEvents(const ScopedEvents&) = delete;
  ScopedEvents& operator=(const ScopedEvents&) = delete;
  ~ScopedEvents() {
    for (auto& x : e)
      if (x) cudaEventDestroy(x);
  }
  cudaError_t create() {
    for (auto& x : e) {
      cudaError_t r = cudaEventCreate(&x);
      if (r != cudaSuccess) return r;
    }
    return cudaSuccess;
  }
  cudaEvent_t& operator[](int k) { return e[k]; }
};

int fail(hc_handle* h, int code, const std::string& msg) {
  h->err = msg;
  return code;
}

// One stream-ordered memory pool per device holds the memory of every handle
// on it.  Memory a handle frees stays in the pool (release threshold: never)
// and is reused by the next handle without another cudaMalloc; the pool is
// trimmed back to the system when the last handle on the device is destroyed.
constexpr int kPoolDevices = 64;
std::mutex g_pool_mutex;
cudaMemPool_t g_pool[kPoolDevices] = {};
int g_live_handles[kPoolDevices] = {};

cudaError_t acquire_pool(int dev, cudaMemPool_t* out) {
  if (dev < 0 || dev >= kPoolDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  if (!g_pool[dev]) {
    cudaMemPoolProps props;
    std::memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    cudaError_t e = cudaMemPoolCreate(&pool, &props);
    if (e != cudaSuccess) return e;
    uint64_t keep = ~0ull;
    if ((e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return e;
    }
    g_pool[dev] = pool;
  }
  g_live_handles[dev]++;
  *out = g_pool[dev];
  return cudaSuccess;
}

// Called by a handle that held the pool, after its frees were enqueued.
void release_pool(int dev, cudaStream_t s) {
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  if (dev < 0 || dev >= kPoolDevices || g_live_handles[dev] <= 0) return;
  if (--g_live_handles[dev] == 0 && g_pool[dev]) {
    if (s) cudaStreamSynchronize(s);
    cudaMemPoolTrimTo(g_pool[dev], 0);
  }
}

cudaError_t dalloc(hc_handle* h, void** p, size_t bytes) {
  cudaError_t e = cudaMallocFromPoolAsync(p, bytes, h->pool, h->stream);
  if (e == cudaSuccess) h->device_bytes += (long long)bytes;
  return e;
}

// Returns memory to the pool in the order of the handle's stream: unlike
// cudaFree it does not wait for the other streams of the device.
void dfree(hc_handle* h, void* p) {
  if (p) cudaFreeAsync(p, h->stream);
}

void invalidate_graph(hc_handle* h) {
  for (int k = 0; k < 2; ++k) {
    if (h->graph1[k]) {
      cudaGraphExecDestroy(h->graph1[k]);
      h->graph1[k] = nullptr;
    }
    if (h->cycle_graph[k]) {
      cudaGraphExecDestroy(h->cycle_graph[k]);
      h->cycle_graph[k] = nullptr;
    }
  }
  for (int k = 0; k < 2; ++k)
    if (h->graph[k]) {
      cudaGraphExecDestroy(h->graph[k]);
      h->graph[k] = nullptr;
    }
  h->graph_valid = false;
}

// Whether the node-velocity form of a tuning reads the node tags: every form
// but the dense one (every fluid node in whole warps), which needs 32-bit
// indices.  Without tags the spreads skip their tag stores, eight scattered
// 4-byte stores per vertex.
bool tags_needed(const hc_handle* h, const int* tune) {
  return !((tune[7] & 0x300) == 0x300 && 19LL * h->N < (1LL << 31));
}

int used_types(const hc_handle* h) {
  int used = 0;
  for (const TypeSlot& ts : h->types) used += !ts.cells.empty();
  return used;
}

int undo_fused_spread(hc_handle* h);

// A new tuning whose node velocity reads tags, while the spread already fused
// into the next force field wrote none: undo it, so that the next step
// spreads (and tags) afresh.
int retag_if_needed(hc_handle* h, const int* old_tune) {
  if (tags_needed(h, h->tune) && !tags_needed(h, old_tune)) return undo_fused_spread(h);
  return HC_OK;
}

template <typename T>
LbmView<T> lbm_view(hc_handle* h, int src, int fcur) {
  LbmView<T> L;
  L.nx = h->nx;
  L.ny = h->ny;
  L.nz = h->nz;
  for (int a = 0; a < 3; ++a) L.per[a] = h->p.periodic[a];
  L.N = h->N;
  L.fsrc = (const T*)h->f[src];
  L.fdst = (T*)h->f[1 - src];
  L.Fcur = (const T*)h->F[fcur];
  L.Fnext = (T*)h->F[1 - fcur];
  L.nbmask = h->nbmask;
  L.flag = h->flag;
  L.corner = h->corner;
  L.bodyz = (const T*)h->bodyz;
  L.ntag = tags_needed(h, h->tune) ? h->ntag : nullptr;
  L.unode = (T*)h->unode;
  L.stamp = h->stamp;
  L.reverse = src;  // alternates with the buffer parity
  L.ck = hcd::collide_constants<T>((T)(1.0 / h->u.tau));
  L.relax = hcfix::relax_constants(1.0 / h->u.tau);
  for (int c = 0; c < hcd::MAX_WALL_CLASSES; ++c)
    for (int a = 0; a < 3; ++a) L.uw[c][a] = (T)h->uw[c][a];
  L.status = h->status;
  L.pdl = (h->tune[7] & 0x400) ? 1 : 0;
  L.bump_stamp = 0;
  L.k1var = (h->tune[7] >> 12) & 3;
  L.moving_walls = 0;
  for (int c = 0; c < hcd::MAX_WALL_CLASSES; ++c)
    for (int a = 0; a < 3; ++a)
      if (h->uw[c][a] != 0.0) L.moving_walls = 1;
  L.fluid = h->nfluid > 0 ? h->fluid : nullptr;
  L.nfluid = h->nfluid;
  L.fast = 19LL * h->N < (1LL << 31) ? 1 : 0;
  const long long nxy = (long long)h->nx * h->ny;
  for (int j = 0; j < 19; ++j)
    L.off[j] = L.fast ? (int)(j * h->N - (hcd::cxi(j) + hcd::cyi(j) * (long long)h->nx + hcd::czi(j) * nxy)) : 0;
  return L;
}

template <typename T>
VertexView<T> vertex_view(hc_handle* h) {
  VertexView<T> vv;
  vv.V = h->Vcap;
  vv.nvert = h->nvert;
  vv.x = h->x;
  vv.v = (T*)h->v;
  vv.f = (T*)h->fv;
  vv.vcell = h->vcell;
  vv.alive = h->alive;
  vv.vnode = h->vnode;
  vv.vtile = h->vtile;
  vv.status = h->status;
  vv.frep_cell = h->rep_every > 0 ? (const T*)h->frep_cell : nullptr;
  vv.frep_wall = h->brep_every > 0 ? (const T*)h->frep_wall : nullptr;
  return vv;
}

// The launch shapes of a handle whose caller chose none (hc_set_tuning,
// hc_autotune), from its lattice and cells.  Steps in microseconds, this choice
// against the other side of the line:
//   Collide-stream in FP64: over the fluid-node list, as a warp with one fluid
//   node costs the issue slots as much as a full one (pipe 64x64x256 84 against
//   111 for the kernel, 150^3 Couette box 342 against 391).
//   In FP32: (x, y)-blocks, or the list where rows rounded up to warps idle a
//   twentieth of their lanes (pipe, rows of 64: 84 against 89; of 97: 29 against
//   32; of 181: 65 against 67).  Evict-last population stores while both buffers
//   take at most half the device's L2 (61x59x131 pipe with repulsion 22.5 against
//   22.7 ms for 400 steps); beyond it they cost (pipe 83.5 against 82.2, the
//   181x117x93 channel 65.7 against 63.6, the 128^3 suspension the same 212).  The
//   handle decides for itself alone: eight small ones side by side, which together
//   mark more than the L2 holds, take 22.7 against 22.5 ms.
//   Node velocity in FP32: every fluid node from one vertex for 24 nodes on (96^3
//   with 80 RBCs 71 against 72; with 20 60 against 68 the other way), else the
//   tagged nodes packed into warps from half a million nodes on (128^3 with 6
//   RBCs 90 against 97; 64^3 with 8 the same 32).  In FP64 tagged fluid nodes
//   (50^3 box 56; every node 62, packed 58; pipe 289, 295, 287).
//   Programmatic launch always (FP64 50^3 box 56 against 67, FP32 32^3 box 25.6
//   against 25.7).
//   Force assembly: variant 2, or 0 for a handful of small FP32 cells (see
//   mech_plan).
bool few_small(const hc_handle* h) {
  if (h->ncells > 16) return false;
  for (const TypeSlot& ts : h->types)
    if (!ts.cells.empty() && ts.tc.nv > 256) return false;
  return true;
}
void apply_rules(hc_handle* h) {
  if (h->tuned) return;
  const int rule[8] = {64, 4, 128, 128, 384, 0, 2, 0x400};
  std::memcpy(h->tune, rule, sizeof(rule));
  const bool fast32 = 19LL * h->N < (1LL << 31);
  const int pad = (h->nx + 31) / 32 * 32 - h->nx;
  if (h->nfluid > 0 && (h->f64 || 20 * pad >= h->nx)) {
    h->tune[0] = 128;
    h->tune[1] = 1;
    h->tune[7] |= 1;
  }
  if (h->f64) {
    if (h->nfluid > 0) h->tune[7] |= 0x100;
    return;
  }
  if (few_small(h)) h->tune[6] = 0;
  if (!fast32) return;
  if (h->nfluid > 0 && 2 * 152LL * h->nfluid <= h->l2) h->tune[7] |= 0x2000;
  if (24LL * h->nvert >= h->N) h->tune[7] |= 0x300;
  else if (h->N >= 500000) h->tune[7] |= 0x200;
}

// ----- nbmask: per node, which directions bounce back and the wall class
void build_nbmask(hc_handle* h, std::vector<uint32_t>& mask) {
  static const int C[19][3] = {{0, 0, 0},  {-1, 0, 0}, {0, -1, 0}, {0, 0, -1}, {-1, -1, 0}, {-1, 1, 0}, {-1, 0, -1},
                               {-1, 0, 1}, {0, -1, -1}, {0, -1, 1}, {1, 0, 0}, {0, 1, 0},  {0, 0, 1},  {1, 1, 0},
                               {1, -1, 0}, {1, 0, 1},  {1, 0, -1}, {0, 1, 1}, {0, 1, -1}};
  const int nx = h->nx, ny = h->ny, nz = h->nz;
  mask.assign(h->N, 0);
  for (int Z = 0; Z < nz; ++Z)
    for (int Y = 0; Y < ny; ++Y)
      for (int X = 0; X < nx; ++X) {
        const long long n = X + (long long)nx * (Y + (long long)ny * Z);
        if (h->hflag[n] != 0) {
          mask[n] = hcd::NB_SOLID;
          continue;
        }
        uint32_t m = 0;
        int cls = -1;
        bool mixed = false;
        for (int i = 1; i < 19; ++i) {
          int q[3] = {X + C[i][0], Y + C[i][1], Z + C[i][2]};
          const int dims[3] = {nx, ny, nz};
          bool out = false;
          for (int a = 0; a < 3; ++a)
            if (q[a] < 0 || q[a] >= dims[a]) {
              if (h->p.periodic[a]) q[a] = (q[a] + dims[a]) % dims[a];
              else out = true;
            }
          int c = -1;
          if (out) c = 0;
          else {
            const uint8_t fl = h->hflag[q[0] + (long long)nx * (q[1] + (long long)ny * q[2])];
            if (fl != 0) c = fl;
          }
          if (c >= 0) {
            m |= 1u << (i - 1);
            if (cls < 0) cls = c;
            else if (cls != c) mixed = true;
          }
        }
        uint32_t cw = cls < 0 ? 0u : (uint32_t)cls;
        if (mixed || cw >= (uint32_t)hcd::MAX_WALL_CLASSES) cw = hcd::NB_CLASS_MIXED;
        // interior: every link pulls from the unwrapped neighbour
        const bool face = (h->p.periodic[0] && (X == 0 || X == nx - 1)) ||
                          (h->p.periodic[1] && (Y == 0 || Y == ny - 1)) ||
                          (h->p.periodic[2] && (Z == 0 || Z == nz - 1));
        if (m == 0 && !face) m |= hcd::NB_INTERIOR;
        mask[n] = m | (cw << hcd::NB_CLASS_SHIFT);
      }
}

int upload_flags(hc_handle* h) {
  std::vector<uint32_t> mask;
  build_nbmask(h, mask);
  HC_CUDA(h, cudaMemcpyAsync(h->flag, h->hflag.data(), h->N, cudaMemcpyHostToDevice, h->stream));
  HC_CUDA(h, hcd::launch_corner_flags(h->flag, h->corner, h->nx, h->ny, h->nz, h->stream));
  HC_CUDA(h, cudaMemcpyAsync(h->nbmask, mask.data(), 4 * h->N, cudaMemcpyHostToDevice, h->stream));
  // the fluid-node list, when coordinates pack into 10/10/12 bits and every
  // population index fits 32 bits
  std::vector<uint32_t> fl;
  if (h->nx <= 1024 && h->ny <= 1024 && h->nz <= 4096 && 19LL * h->N < (1LL << 31)) {
    fl.reserve(h->N);
    for (int Z = 0; Z < h->nz; ++Z)
      for (int Y = 0; Y < h->ny; ++Y)
        for (int X = 0; X < h->nx; ++X)
          if (h->hflag[X + (long long)h->nx * (Y + (long long)h->ny * Z)] == 0)
            fl.push_back((uint32_t)X | ((uint32_t)Y << 10) | ((uint32_t)Z << 20));
    if ((long long)fl.size() > h->fluid_cap) {
      dfree(h, h->fluid);
      h->fluid = nullptr;
      h->device_bytes -= 4 * h->fluid_cap;
      h->fluid_cap = 0;
      HC_CUDA(h, dalloc(h, (void**)&h->fluid, 4 * std::max<size_t>(fl.size(), 1)));
      h->fluid_cap = (long long)std::max<size_t>(fl.size(), 1);
    }
    if (!fl.empty()) HC_CUDA(h, cudaMemcpyAsync(h->fluid, fl.data(), 4 * fl.size(), cudaMemcpyHostToDevice, h->stream));
  }
  h->nfluid = (int)fl.size();
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  apply_rules(h);
  return HC_OK;
}

// The per-plane body-force profile of the current body force (3 x nz).
std::vector<double> body_profile(const hc_handle* h) {
  std::vector<double> bz(3 * h->nz, 0.0);
  for (int z = 0; z < h->nz; ++z) {
    if (h->body_mode == HC_BODY_UNIFORM) {
      for (int a = 0; a < 3; ++a) bz[a * h->nz + z] = h->body[a];
    } else if (h->body_mode == HC_BODY_KOLMOGOROV) {
      bz[z] = h->body[0] * std::sin(2.0 * M_PI * (double)z / (double)h->nz);
    }
  }
  return bz;
}

// Copies the profile (and, when given, its change) to the device from the
// handle's pinned staging buffer, in the order of the handle's stream.  A
// kernel reads the mapped buffer, so the upload does not queue on a copy
// engine behind an asynchronous position readback.
int upload_profile(hc_handle* h, const std::vector<double>& prof, const std::vector<double>* change) {
  const size_t n = 3 * (size_t)h->nz;
  if (!h->hbody_pin) {
    HC_CUDA(h, cudaHostAlloc(&h->hbody_pin, 2 * n * h->ts, cudaHostAllocMapped));
    HC_CUDA(h, cudaHostGetDevicePointer(&h->hbody_dev, h->hbody_pin, 0));
    HC_CUDA(h, cudaEventCreateWithFlags(&h->body_copied, cudaEventDisableTiming));
  } else {
    HC_CUDA(h, cudaEventSynchronize(h->body_copied));  // the last upload has left the buffer
  }
  for (size_t k = 0; k < n; ++k) {
    const double c = change ? (*change)[k] : 0.0;
    if (h->f64) {
      static_cast<double*>(h->hbody_pin)[k] = prof[k];
      static_cast<double*>(h->hbody_pin)[n + k] = c;
    } else {
      static_cast<float*>(h->hbody_pin)[k] = (float)prof[k];
      static_cast<float*>(h->hbody_pin)[n + k] = (float)c;
    }
  }
  HC_CUDA(h, hcd::launch_copy_words(h->bodyz, h->hbody_dev, n * h->ts, h->stream));
  if (change) {
    if (!h->bodyd) HC_CUDA(h, dalloc(h, &h->bodyd, n * h->ts));
    HC_CUDA(h, hcd::launch_copy_words(h->bodyd, static_cast<char*>(h->hbody_dev) + n * h->ts, n * h->ts, h->stream));
  }
  HC_CUDA(h, cudaEventRecord(h->body_copied, h->stream));
  return HC_OK;
}

// Uploads the body-force profile and refills the next step's force field with it.
int upload_body(hc_handle* h) {
  int rc;
  if ((rc = upload_profile(h, body_profile(h), nullptr)) != HC_OK) return rc;
  const long long plane = (long long)h->nx * h->ny;
  if (h->f64)
    HC_CUDA(h, hcd::launch_fill_body<double>((double*)h->F[h->cur], (const double*)h->bodyz, plane, h->nz, h->N,
                                             h->stream));
  else
    HC_CUDA(h, hcd::launch_fill_body<float>((float*)h->F[h->cur], (const float*)h->bodyz, plane, h->nz, h->N,
                                            h->stream));
  return HC_OK;
}

int ensure_scratch(hc_handle* h, size_t bytes) {
  if (h->scratch_bytes >= bytes) return HC_OK;
  if (h->scratch) {
    dfree(h, h->scratch);
    h->device_bytes -= (long long)h->scratch_bytes;
  }
  h->scratch = nullptr;
  h->scratch_bytes = 0;
  HC_CUDA(h, dalloc(h, (void**)&h->scratch, bytes));
  h->scratch_bytes = bytes;
  return HC_OK;
}

// Staging larger than the steady readbacks need (hc_read_fluid: 4 doubles per
// node) is only used by set-up and population transfers: give it back, so a
// resident handle holds no more than hc_estimate_device_bytes counts.
void shrink_scratch(hc_handle* h) {
  if (h->scratch && h->scratch_bytes > sizeof(double) * 4 * (size_t)h->N) {
    dfree(h, h->scratch);
    h->device_bytes -= (long long)h->scratch_bytes;
    h->scratch = nullptr;
    h->scratch_bytes = 0;
  }
}

// grow a [3][V] SoA array from capacity oldV to newV
int grow3(hc_handle* h, void** p, size_t es, long long oldV, long long newV, int nused) {
  void* np = nullptr;
  HC_CUDA(h, dalloc(h, &np, 3 * es * newV));
  HC_CUDA(h, cudaMemsetAsync(np, 0, 3 * es * newV, h->stream));
  if (*p && nused > 0)
    for (int a = 0; a < 3; ++a)
      HC_CUDA(h, cudaMemcpyAsync((char*)np + a * es * newV, (char*)*p + a * es * oldV, es * nused,
                                 cudaMemcpyDeviceToDevice, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  if (*p) {
    dfree(h, *p);
    h->device_bytes -= (long long)(3 * es * oldV);
  }
  *p = np;
  return HC_OK;
}

int grow1(hc_handle* h, void** p, size_t es, long long oldn, long long newn, long long nused) {
  void* np = nullptr;
  HC_CUDA(h, dalloc(h, &np, es * newn));
  HC_CUDA(h, cudaMemsetAsync(np, 0, es * newn, h->stream));
  if (*p && nused > 0) HC_CUDA(h, cudaMemcpyAsync(np, *p, es * nused, cudaMemcpyDeviceToDevice, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  if (*p) {
    dfree(h, *p);
    h->device_bytes -= (long long)(es * oldn);
  }
  *p = np;
  return HC_OK;
}

// Device state of the repulsion terms that are enabled, sized for the
// vertex capacity (the kept forces are carried over when it grows).
int ensure_repulsion(hc_handle* h) {
  int rc;
  const bool any = h->rep_every > 0 || h->brep_every > 0;
  if (!any) return HC_OK;
  if (h->rep_every > 0 && !h->rep_cnt) {
    HC_CUDA(h, dalloc(h, (void**)&h->rep_cnt, sizeof(int2) * h->N));
    HC_CUDA(h, dalloc(h, (void**)&h->rep_slot, sizeof(int) * hcd::REP_SLOTS * h->N));
  }
  const long long cap = std::max<long long>(h->Vcap, 1);
  if (h->rep_vcap < cap || !h->rep_vq) {
    if ((rc = grow1(h, (void**)&h->rep_vq, 4, h->rep_vcap, cap, 0)) != HC_OK) return rc;
    if ((rc = grow1(h, &h->rep_xr, 4 * h->ts, h->rep_vcap, cap, 0)) != HC_OK) return rc;
    const int kept = (int)std::min<long long>(h->nvert, h->rep_vcap);
    if ((rc = grow3(h, &h->frep_cell, h->ts, h->rep_vcap, cap, h->frep_cell ? kept : 0)) != HC_OK) return rc;
    if ((rc = grow3(h, &h->frep_wall, h->ts, h->rep_vcap, cap, h->frep_wall ? kept : 0)) != HC_OK) return rc;
    h->rep_vcap = cap;
  }
  return HC_OK;
}

int upload_types(hc_handle* h) {
  std::vector<TypeDev> tv(hcd::MAX_TYPES);
  for (size_t t = 0; t < h->types.size(); ++t) tv[t] = h->types[t].dev;
  HC_CUDA(h, cudaMemcpyAsync(h->dtypes, tv.data(), sizeof(TypeDev) * hcd::MAX_TYPES, cudaMemcpyHostToDevice,
                             h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return HC_OK;
}

// per-type cell lists and the batched list (largest type first)
int upload_cell_lists(hc_handle* h) {
  for (TypeSlot& ts : h->types) {
    if ((int)ts.cells.size() > ts.dcells_cap) {
      dfree(h, ts.dcells);
      ts.dcells_cap = std::max<int>((int)ts.cells.size(), 2 * ts.dcells_cap);
      HC_CUDA(h, dalloc(h, (void**)&ts.dcells, sizeof(int) * ts.dcells_cap));
    }
    if (!ts.cells.empty())
      HC_CUDA(h, cudaMemcpyAsync(ts.dcells, ts.cells.data(), sizeof(int) * ts.cells.size(), cudaMemcpyHostToDevice,
                                 h->stream));
  }
  std::vector<int> order(h->types.size());
  for (size_t t = 0; t < order.size(); ++t) order[t] = (int)t;
  std::stable_sort(order.begin(), order.end(),
                   [&](int a, int b) { return h->types[a].tc.nv > h->types[b].tc.nv; });
  std::vector<int> all;
  for (int t : order) all.insert(all.end(), h->types[t].cells.begin(), h->types[t].cells.end());
  if (!all.empty())
    HC_CUDA(h, cudaMemcpyAsync(h->dcells_all, all.data(), sizeof(int) * all.size(), cudaMemcpyHostToDevice, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return HC_OK;
}

// After a fused step the next force field holds body force + the next
// spread.  A change that makes that spread stale restores the field to the
// body force so the next step spreads afresh.
int undo_fused_spread(hc_handle* h) {
  if (h->stamp_ahead) {
    // catch the stamp up with the tags the fused spread wrote
    HC_CUDA(h, hcd::launch_bump_stamp(h->stamp, h->stream));
    h->stamp_ahead = false;
  }
  if (!h->spread_done) return HC_OK;
  const long long plane = (long long)h->nx * h->ny;
  if (h->f64)
    HC_CUDA(h, hcd::launch_fill_body<double>((double*)h->F[h->cur], (const double*)h->bodyz, plane, h->nz, h->N,
                                             h->stream));
  else
    HC_CUDA(h, hcd::launch_fill_body<float>((float*)h->F[h->cur], (const float*)h->bodyz, plane, h->nz, h->N,
                                            h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  h->spread_done = false;
  return HC_OK;
}

// ----- stage launchers (enqueue only) -------------------------------------
template <typename T>
int enq_spread(hc_handle* h) {
  if (h->next > 0)
    HC_CUDA(h, hcd::launch_add_vertex_forces<T>(vertex_view<T>(h), h->ext_ids, h->ext_f, h->next, h->stream));
  LbmView<T> L = lbm_view<T>(h, h->cur, h->cur);
  HC_CUDA(h, hcd::launch_spread<T>(L, vertex_view<T>(h), h->u.f_limit, h->tune[2], h->stream));
  return HC_OK;
}

template <typename T>
cudaError_t launch_k1(hc_handle* h, const LbmView<T>& L) {
  const int mode = h->tune[7] & 0xff;
  if (mode == 1 && L.fluid) return hcd::launch_collide_stream_fluid<T>(L, h->tune[0], h->stream);
  if (mode >= 2 && h->bulk_key == mode) return hcd::launch_collide_stream_bulk<T>(L, h->bulk, h->stream);
  return hcd::launch_collide_stream<T>(L, h->tune[0], h->tune[1], h->stream);
}

template <typename T>
cudaError_t launch_nv(hc_handle* h, const LbmView<T>& L) {
  if ((h->tune[7] & 0x300) == 0x300 && L.fast) return hcd::launch_node_velocity_dense<T>(L, h->stream);
  if ((h->tune[7] & 0x200) && L.fast) return hcd::launch_node_velocity_packed<T>(L, h->stream);
  if ((h->tune[7] & 0x100) && L.fluid) return hcd::launch_node_velocity_fluid<T>(L, h->stream);
  return hcd::launch_node_velocity<T>(L, h->stream);
}

template <typename T>
int enq_collide(hc_handle* h) {
  LbmView<T> L = lbm_view<T>(h, h->cur, h->cur);
  L.bump_stamp = h->stamp_ahead ? 1 : 0;
  h->stamp_ahead = false;
  HC_CUDA(h, launch_k1<T>(h, L));
  h->cur ^= 1;
  return HC_OK;
}

// Plan (and shared-memory attribute) of the bulk-copy collide-stream for
// tune[7]; runs outside any stream capture.  Returns false when the lattice
// does not allow that configuration.
template <typename T>
bool set_bulk_plan(hc_handle* h, int code) {
  code &= 0xff;
  if (code < 2) return true;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->p.device);
  hcd::BulkPlan P;
  if (!hcd::make_bulk_plan<T>(h->nx, h->ny, h->nz, code & 15, (code >> 4) * sms, &P)) return false;
  if (hcd::prepare_collide_bulk<T>(P) != cudaSuccess) return false;
  h->bulk = P;
  h->bulk_key = code;
  return true;
}

// post-stream view: populations f[cur], force of the last collision F[1-cur].
// The stencil nodes were tagged by this step's spread; a standalone
// interpolation stage tags them itself (mark = 1).
template <typename T>
int enq_interp_advance(hc_handle* h, int do_interp, int do_advance, int mark = 0) {
  LbmView<T> L = lbm_view<T>(h, h->cur, 1 - h->cur);
  // no vertex, no stencil node to evaluate (the scan alone is thousands of blocks)
  if (do_interp && h->nvert > 0) {
    if (mark) HC_CUDA(h, hcd::launch_mark_nodes<T>(L, vertex_view<T>(h), h->stream));
    HC_CUDA(h, launch_nv<T>(h, L));
  }
  HC_CUDA(h, hcd::launch_interp_advance<T>(L, vertex_view<T>(h), h->tg, do_interp, do_advance, h->tune[3],
                                           h->stream));
  return HC_OK;
}

// The next spread can be fused into this mechanics pass when the batched
// vertex-centric kernel handles every cell this step, every type is due
// every step and no external vertex force is added before the spread.
// The repulsion terms due at iteration `it` (core/hemoCell.cpp:307-312),
// from the current positions; force = 1 recomputes every enabled term.
template <typename T>
int enq_repulsion(hc_handle* h, int it, bool force = false) {
  const bool dc = h->rep_every > 0 && (force || it % h->rep_every == 0);
  const bool dw = h->brep_every > 0 && (force || it % h->brep_every == 0);
  if ((!dc && !dw) || h->nvert == 0) return HC_OK;
  if (dc) HC_CUDA(h, cudaMemsetAsync(h->rep_cnt, 0, sizeof(int2) * h->N, h->stream));
  hcd::RepView<T> R;
  R.node = dc ? h->rep_cnt : nullptr;
  R.slot = h->rep_slot;
  R.vq = h->rep_vq;
  R.rec = (hcd::RepRecord<T>*)h->rep_xr;
  R.bnode = h->rep_bnode;
  R.fcell = dc ? (T*)h->frep_cell : nullptr;
  R.fwall = dw ? (T*)h->frep_wall : nullptr;
  R.kc = (T)h->rep_k;
  R.rc = (T)h->rep_rc;
  R.kw = (T)h->brep_k;
  R.rw = (T)h->brep_rc;
  LbmView<T> L = lbm_view<T>(h, h->cur, h->cur);
  HC_CUDA(h, hcd::launch_repulsion<T>(L, vertex_view<T>(h), R, h->stream));
  return HC_OK;
}

bool fusable(hc_handle* h) {
  if (h->p.launch != HC_LAUNCH_BATCHED || h->tune[6] == 1 || h->next > 0 || h->ncells == 0) return false;
  if (h->velocity_every != 1) return false;
  for (TypeSlot& ts : h->types)
    if (ts.every != 1) return false;
  return true;
}

size_t gather_bytes(const hc_handle* h, const TypeSlot& ts, int cluster = 1) {
  return h->f64 ? hcd::mechanics_smem_bytes<double>(ts.tc.nv, cluster)
                : hcd::mechanics_smem_bytes<float>(ts.tc.nv, cluster);
}

// How the force assembly launches the cells of one type (variants 0 and 2).
// CTAs a cell, a power of two.  FP32: as many as leave every CTA an SM of its
// own, at most 8.  FP64, whose one pipe an SM bounds it, splits finer, so that
// the SMs' shares come out even and one CTA's loads fill another's gaps: 2 at
// least, 4 up to three CTAs an SM (two where other types' CTAs need room beside
// them: 110 RBCs with 11 platelets and a WBC took 162 us a step on 4 CTAs a
// cell, some of which then wait for a second wave), 8 up to two.  Either form takes 16 where 8
// would leave a CTA more than 96 vertices.  The kernel in microseconds, staged,
// with the advance and spread in it, n RBCs of 642 vertices on 1 / 2 / 4 / 8 CTAs
// a cell:
//   FP64  n = 30: 103 / 60 / 49 / 48    110: 105 / 96 / 87 / 128
//         n = 220: 182 / 143 / 161 / 214    280: 182 / 181 / 223 / 249
//   FP32  n = 30: 27 / 26 / 26 / 27     60: 27 / 27 / 31 / 36
//         n = 110: 28 / 35 / 41 / 65    280: 39 / 68 / 108 / 130
// Threads, staged: one per face of the CTA's share, 128 to 384 (256 from four
// CTAs a cell on); the 384 of a whole RBC are two CTAs an SM.
// An FP32 type whose terms, kept face by face and edge by edge as vectors, would
// take more than 110 KB in one CTA (above 960 vertices of a red or white cell, 730
// of a platelet) is assembled vertex by vertex.  That is the line of an earlier
// layout; at the one size in use beyond it, the 2562-vertex white cell, both
// kernels take the same time (128^3 suspension with two of them, 300 steps: 69.7 ms
// each).  So is a type whose terms do not fit at all, and, by the rules, a handful
// of small cells: red cells alone 22 us a step against 24 staged; with platelets,
// whose dihedral terms it computes once for each incident vertex, 34 against 26.
// Nothing orders either kernel's spread (two runs' velocities are 4e-8 apart), but
// for such a handful the vertex-centric one repeats positions to 1e-9 over 21
// steps, where the staged one's were 9e-9 apart.
struct MechPlan {
  bool staged;
  int cluster, bs;
  size_t smem;
};
MechPlan mech_plan(const hc_handle* h, const TypeSlot& ts) {
  const long long n = (long long)ts.cells.size();
  const int nv = ts.tc.nv, nf = ts.tc.nf, ne = ts.tc.ne, model = ts.tc.model;
  auto bytes = [&](int cs) { return hcd::mechanics_staged_bytes(model, nv, nf, ne, cs, h->f64); };
  if (h->tune[6] == 1) return {false, 1, h->tune[4], gather_bytes(h, ts)};
  int cs = 1;
  if (h->f64) cs = 8 * n <= 2 * h->sms ? 8 : (4 * n <= (used_types(h) > 1 ? 2 : 3) * h->sms ? 4 : 2);
  else
    while (cs < 8 && 2 * n * cs <= h->sms) cs *= 2;
  // with the advance and the spread in it, a cell that one round of a CTA's threads
  // holds stays whole (against clusters, us a step: FP64, 8 cells of 42 vertices 34
  // and 40, 16 of 162 the same 41, with platelets 42 and 43; FP32, 40 of 162
  // vertices 24.6 and 29.7)
  if (h->p.launch == HC_LAUNCH_BATCHED && nv <= 256) cs = 1;
  if (cs == 8 && nv > 8 * 96 && 16 * n <= h->sms && ts.cluster16) cs = 16;
  const size_t whole = 4 * (6 * (size_t)nv + 7 * (size_t)nf + 3 * (size_t)ne * (model == HC_MODEL_PLT_SIMPLE ? 2 : 1)) +
                       (size_t)nv + 272;
  if (h->tune[6] == 2 && (h->f64 || whole <= 110 * 1024)) {
    int c = cs;
    while (c < 8 && bytes(c) > (size_t)h->staged_limit) c *= 2;
    if (bytes(c) <= (size_t)h->staged_limit) {
      int bs = std::max(128, std::min(c < 4 ? 384 : 256, ((nf + c - 1) / c + 31) / 32 * 32));
      if (h->tuned && c == 1) bs = std::min(h->tune[4], 384);
      return {true, c, bs, bytes(c)};
    }
  }
  const int bs = cs == 1 ? h->tune[4] : std::max(128, std::min(h->tune[4], ((nf + cs - 1) / cs + 31) / 32 * 32));
  return {false, cs, bs, gather_bytes(h, ts, cs)};
}

inline void prof_mark(hc_handle* h, int slot) {
  if (h->prof_step >= 0) cudaEventRecord(h->prof_ev[h->prof_step * 6 + slot], h->stream);
}

// The force assembly of the due types.  Variant 2 with every type due (all_due)
// runs the types side by side, the one with the most vertices last: a
// suspension's few large cells would otherwise hold the step up before or behind
// the red ones (one 2562-vertex WBC took 1550 of the 1557 us of an FP64
// suspension's force assembly) or, in one launch, make every CTA take their
// shared memory.  Each launch lets the next start once its CTAs run (programmatic
// launch), and ends after the one before it; on forked streams the same launches
// took 300 us a step instead of 250 inside a graph, which puts the large clusters
// last.  A handful of small cells (few_small) takes one launch.  Otherwise one
// launch per type, one after another.
template <typename T>
int enq_types(hc_handle* h, hcd::MechView<T> M, bool forced, bool all_due) {
  struct Launch {
    MechPlan plan;
    const int* cells;
    long long n, vertices;
  };
  std::vector<Launch> launches;
  const bool together = (h->tune[6] == 2 || !h->tuned) && all_due;
  for (const TypeSlot& ts : h->types)
    if (!ts.cells.empty() && (forced || h->iter % ts.every == 0))
      launches.push_back({mech_plan(h, ts), ts.dcells, (long long)ts.cells.size(), (long long)ts.cells.size() * ts.tc.nv});
  if (launches.empty()) return HC_OK;
  if (together && h->p.launch == HC_LAUNCH_BATCHED && few_small(h)) {
    Launch one = launches[0];
    for (const Launch& l : launches) {
      one.plan.smem = std::max(one.plan.smem, l.plan.smem);
      one.plan.bs = std::max(one.plan.bs, l.plan.bs);
    }
    launches = {{one.plan, h->dcells_all, h->ncells, 0}};
  } else if (together) {
    std::stable_sort(launches.begin(), launches.end(),
                     [](const Launch& a, const Launch& b) { return a.vertices < b.vertices; });
  }
  const bool overlap = together && launches.size() > 1;
  const int pdl = M.L.pdl;
  for (size_t k = 0; k < launches.size(); ++k) {
    const Launch& l = launches[k];
    M.cells = l.cells;
    M.ncells = (int)l.n;
    M.dyn_smem = (int)l.plan.smem;
    M.after_prev = overlap && k > 0;
    M.before_next = overlap && k + 1 < launches.size();
    M.L.pdl = pdl || M.after_prev;
    // an SM configured for small CTAs takes no large one until they end: side by
    // side all launches run on the same split of the SM's memory (FP32 128^3
    // suspension 212 us a step against 224 without, 220 at 100 percent; FP64
    // 67x81x50 suspension 140.5, 140.5, 147)
    M.carveout = overlap ? 55 : 0;
    if (l.plan.staged) HC_CUDA(h, hcd::launch_mechanics_staged<T>(M, l.plan.cluster, l.plan.bs, h->stream));
    else HC_CUDA(h, hcd::launch_mechanics<T>(M, l.plan.cluster, l.plan.bs, 0, h->tune[6] == 1 ? 1 : 0, h->stream));
  }
  return HC_OK;
}

template <typename T>
int enq_mechanics(hc_handle* h, bool forced, bool fuse = false, bool fuse_adv = false) {
  bool all_due = true;
  for (TypeSlot& ts : h->types)
    if (!(forced || h->iter % ts.every == 0)) all_due = false;
  MechView<T> M;
  M.cell_type = h->cell_type;
  M.cell_voff = h->cell_voff;
  M.types = h->dtypes;
  M.vv = vertex_view<T>(h);
  M.fuse_spread = 0;
  M.fuse_advance = 0;
  M.after_prev = M.before_next = M.carveout = 0;
  M.tg = h->tg;
  // Fcur = the next step's force field; unode = this step's node velocities
  M.L = lbm_view<T>(h, h->cur, h->cur);
  M.f_limit = (T)h->u.f_limit;
  const bool batched = h->p.launch == HC_LAUNCH_BATCHED && all_due && h->ncells > 0;
  if (batched) {
    M.fuse_spread = fuse ? 1 : 0;
    M.fuse_advance = fuse && fuse_adv ? 1 : 0;
    if (M.fuse_advance) h->stamp_ahead = true;
  }
  if (batched && (h->tune[6] == 1 || (h->tune[6] == 0 && (used_types(h) > 1 || h->tune[5] > 0)))) {
    // one launch across the cell types, largest first
    size_t smem = 0;
    for (TypeSlot& ts : h->types)
      if (!ts.cells.empty()) smem = std::max(smem, gather_bytes(h, ts));
    M.cells = h->dcells_all;
    M.ncells = h->ncells;
    M.dyn_smem = (int)smem;
    HC_CUDA(h, hcd::launch_mechanics<T>(M, 1, h->tune[4], h->tune[5], h->tune[6], h->stream));
    return HC_OK;
  }
  return enq_types<T>(h, M, forced, all_due);
}

// one HemoCell::iterate(): spread, collide+stream (+force reset), interpolate
// (every velocity_every), advance, constitutive model (due types).
template <typename T>
int enq_step(hc_handle* h) {
  int rc;
  if (!h->spread_done) {
    if ((rc = enq_repulsion<T>(h, h->iter)) != HC_OK) return rc;
    if ((rc = enq_spread<T>(h)) != HC_OK) return rc;
  }
  prof_mark(h, 0);
  if ((rc = enq_collide<T>(h)) != HC_OK) return rc;
  prof_mark(h, 1);
  const bool fuse = fusable(h);
  // without repulsion (which needs every cell advanced first) the force
  // assembly also interpolates and advances its cell's vertices
  const bool fuse_adv = fuse && h->rep_every == 0 && h->brep_every == 0 && (h->tune[7] & 0x800) == 0;
  prof_mark(h, 2);
  if (fuse_adv) {
    LbmView<T> L = lbm_view<T>(h, h->cur, 1 - h->cur);
    HC_CUDA(h, launch_nv<T>(h, L));
  } else {
    if ((rc = enq_interp_advance<T>(h, h->iter % h->velocity_every == 0, 1)) != HC_OK) return rc;
    // the fused spread is the next step's: its repulsion uses the positions
    // just advanced, which are that step's positions
    if (fuse && (rc = enq_repulsion<T>(h, h->iter + 1)) != HC_OK) return rc;
  }
  prof_mark(h, 3);
  prof_mark(h, 4);
  if ((rc = enq_mechanics<T>(h, false, fuse, fuse_adv)) != HC_OK) return rc;
  prof_mark(h, 5);
  h->spread_done = fuse;
  h->iter++;
  return HC_OK;
}

bool graph_eligible(hc_handle* h) {
  if (h->p.launch != HC_LAUNCH_BATCHED) return false;
  if (h->velocity_every != 1 || h->rep_every > 1 || h->brep_every > 1) return false;
  for (TypeSlot& ts : h->types)
    if (ts.every != 1) return false;
  return true;
}

// Steps of one timescale cycle of the batched launch: the least common
// multiple of 2 (the buffer parity) and every timescale in use, or 0 when
// there is none to cycle (every timescale 1: the two-step graphs serve) or
// the cycle exceeds 64 steps.
int timescale_cycle(const hc_handle* h) {
  if (h->p.launch != HC_LAUNCH_BATCHED) return 0;
  long long L = 2;
  auto lcm = [](long long a, long long b) { return a / std::gcd(a, b) * b; };
  L = lcm(L, h->velocity_every);
  for (const TypeSlot& ts : h->types) L = lcm(L, ts.every);
  if (h->rep_every > 0) L = lcm(L, h->rep_every);
  if (h->brep_every > 0) L = lcm(L, h->brep_every);
  return (L > 2 && L <= 64) ? (int)L : 0;
}

// Captures `steps` steps starting on buffer parity `parity` into h->graph
// (two steps, the parity returns), h->graph1 (one step) or h->cycle_graph
// (a whole timescale cycle, starting at h->iter).
template <typename T>
int build_graph(hc_handle* h, int parity, int steps = 2) {
  const int save_cur = h->cur, save_iter = h->iter;
  const bool save_sd = h->spread_done, save_sa = h->stamp_ahead;
  h->cur = parity;
  cudaGraph_t g = nullptr;
  HC_CUDA(h, cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
  int rc = enq_step<T>(h);
  for (int k = 1; k < steps && rc == HC_OK; ++k) rc = enq_step<T>(h);
  cudaError_t e = cudaStreamEndCapture(h->stream, &g);
  h->cur = save_cur;
  h->iter = save_iter;
  h->spread_done = save_sd;
  h->stamp_ahead = save_sa;
  if (rc != HC_OK) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  if (e != cudaSuccess) return fail(h, HC_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e));
  e = cudaGraphInstantiate(steps == 2 ? &h->graph[parity] : (steps == 1 ? &h->graph1[parity] : &h->cycle_graph[parity]),
                           g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return fail(h, HC_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e));
  return HC_OK;
}

template <typename T>
int run_steps(hc_handle* h, int nsteps) {
  int rc;
  // timescale separation: eager steps up to the start of a cycle, then whole
  // cycles replayed from their graph
  const int L = timescale_cycle(h);
  if (L > 0 && nsteps >= 2 * L) {
    while (nsteps > 0 && (h->iter % L != 0 || (fusable(h) && !h->spread_done))) {
      if ((rc = enq_step<T>(h)) != HC_OK) return rc;
      nsteps--;
    }
    if (h->cycle_len != L) {
      invalidate_graph(h);
      h->cycle_len = L;
    }
    while (nsteps >= L) {
      if (!h->cycle_graph[h->cur] && (rc = build_graph<T>(h, h->cur, L)) != HC_OK) return rc;
      HC_CUDA(h, cudaGraphLaunch(h->cycle_graph[h->cur], h->stream));
      h->iter += L;
      nsteps -= L;
    }
  }
  if (graph_eligible(h) && nsteps >= 3 && fusable(h) && !h->spread_done) {
    if ((rc = enq_step<T>(h)) != HC_OK) return rc;  // leaves the next spread done
    nsteps--;
  }
  if (graph_eligible(h) && nsteps >= 2 && (!fusable(h) || h->spread_done)) {
    if (!h->graph_valid) {
      invalidate_graph(h);
      if ((rc = build_graph<T>(h, 0)) != HC_OK) return rc;
      if ((rc = build_graph<T>(h, 1)) != HC_OK) return rc;
      h->graph_valid = true;
    }
    while (nsteps >= 2) {
      HC_CUDA(h, cudaGraphLaunch(h->graph[h->cur], h->stream));
      h->iter += 2;
      nsteps -= 2;
    }
  }
  // a single step in the same state (iterate(1) in a loop) replays the
  // one-step graph of its parity; the step flips the buffers
  // (invalidate_graph, run on every state change, drops these graphs too)
  if (nsteps == 1 && graph_eligible(h) && (!fusable(h) || h->spread_done)) {
    if (!h->graph1[h->cur] && (rc = build_graph<T>(h, h->cur, 1)) != HC_OK) return rc;
    HC_CUDA(h, cudaGraphLaunch(h->graph1[h->cur], h->stream));
    h->iter += 1;
    h->cur ^= 1;
    return HC_OK;
  }
  for (int k = 0; k < nsteps; ++k)
    if ((rc = enq_step<T>(h)) != HC_OK) return rc;
  return HC_OK;
}

template <typename T>
int run_stage(hc_handle* h, int stage) {
  if (stage != HC_STAGE_BIN) {
    int rc0 = undo_fused_spread(h);
    if (rc0 != HC_OK) return rc0;
  }
  switch (stage) {
    case HC_STAGE_SPREAD:
      return enq_spread<T>(h);
    case HC_STAGE_COLLIDE_STREAM:
      return enq_collide<T>(h);
    case HC_STAGE_INTERPOLATE:
      return enq_interp_advance<T>(h, 1, 0, 1);
    case HC_STAGE_ADVANCE:
      return enq_interp_advance<T>(h, 0, 1);
    case HC_STAGE_MECHANICS:
      return enq_mechanics<T>(h, false);
    case HC_STAGE_MECHANICS_FORCED:
      return enq_mechanics<T>(h, true);
    case HC_STAGE_REPULSION:
      return enq_repulsion<T>(h, h->iter, true);
    case HC_STAGE_BIN: {
      LbmView<T> L = lbm_view<T>(h, h->cur, h->cur);
      HC_CUDA(h, hcd::launch_bin_vertices<T>(L, vertex_view<T>(h), h->tg, h->stream));
      if (h->bin_vcap < h->Vcap || !h->bin_counts) {
        dfree(h, h->tile_vertices);
        dfree(h, h->tile_cells);
        HC_CUDA(h, dalloc(h, (void**)&h->tile_vertices, sizeof(int) * std::max<long long>(1, h->Vcap)));
        HC_CUDA(h, dalloc(h, (void**)&h->tile_cells, sizeof(int) * std::max<long long>(1, h->Vcap)));
        h->bin_vcap = h->Vcap;
      }
      if (!h->bin_counts) {
        const int nt = h->ntiles;
        HC_CUDA(h, dalloc(h, (void**)&h->bin_counts, sizeof(int) * nt));
        HC_CUDA(h, dalloc(h, (void**)&h->bin_cursor, sizeof(int) * nt));
        HC_CUDA(h, dalloc(h, (void**)&h->bin_offsets, sizeof(int) * (nt + 1)));
        HC_CUDA(h, dalloc(h, (void**)&h->tile_cell_counts, sizeof(int) * nt));
        HC_CUDA(h, dalloc(h, (void**)&h->tile_cell_offsets, sizeof(int) * (nt + 1)));
      }
      HC_CUDA(h, hcd::launch_bin_csr(h->vtile, h->nvert, h->ntiles, h->bin_counts, h->bin_offsets, h->bin_cursor,
                                     h->tile_vertices, h->vcell, h->tile_cell_counts, h->stream));
      HC_CUDA(h, hcd::launch_tile_cells(h->bin_offsets, h->tile_vertices, h->vcell, h->ntiles, h->tile_cell_counts,
                                        h->tile_cell_offsets, h->tile_cells, (int)h->bin_vcap, h->stream));
      return HC_OK;
    }
    default:
      return fail(h, HC_ERR_INVALID, "unknown stage");
  }
}

int add_cells_positions(hc_handle* h, int type, int n, const std::vector<double>& xyz) {
  TypeSlot& ts = h->types[type];
  const int nv = ts.tc.nv;
  const long long need = (long long)h->nvert + (long long)n * nv;
  if (need > (long long)INT32_MAX / 4) return fail(h, HC_ERR_INVALID, "too many vertices");
  for (double q : xyz)
    if (!std::isfinite(q)) return fail(h, HC_ERR_NUMERIC, "non-finite vertex position");
  invalidate_graph(h);
  int rc;
  // new vertices need the spread to tag their stencils
  if ((rc = undo_fused_spread(h)) != HC_OK) return rc;
  if (need > h->Vcap) {
    long long nc = std::max<long long>(need, 2 * h->Vcap);
    nc = std::max<long long>(nc, 1024);
    if ((rc = grow3(h, (void**)&h->x, 8, h->Vcap, nc, h->nvert)) != HC_OK) return rc;
    if ((rc = grow3(h, &h->v, h->ts, h->Vcap, nc, h->nvert)) != HC_OK) return rc;
    if ((rc = grow3(h, &h->fv, h->ts, h->Vcap, nc, h->nvert)) != HC_OK) return rc;
    if ((rc = grow1(h, (void**)&h->vcell, 4, h->Vcap, nc, h->nvert)) != HC_OK) return rc;
    if ((rc = grow1(h, (void**)&h->vnode, 4, h->Vcap, nc, h->nvert)) != HC_OK) return rc;
    if ((rc = grow1(h, (void**)&h->vtile, 4, h->Vcap, nc, h->nvert)) != HC_OK) return rc;
    h->Vcap = nc;
  }
  const int needc = h->ncells + n;
  if (needc > h->cellcap) {
    int nc = std::max(needc, std::max(2 * h->cellcap, 64));
    if ((rc = grow1(h, (void**)&h->cell_type, 4, h->cellcap, nc, h->ncells)) != HC_OK) return rc;
    if ((rc = grow1(h, (void**)&h->cell_voff, 4, h->cellcap, nc, h->ncells)) != HC_OK) return rc;
    if ((rc = grow1(h, (void**)&h->alive, 4, h->cellcap, nc, h->ncells)) != HC_OK) return rc;
    if ((rc = grow1(h, (void**)&h->dcells_all, 4, h->cellcap, nc, h->ncells)) != HC_OK) return rc;
    h->cellcap = nc;
  }
  // positions: host layout [V][3] -> device [3][Vcap]
  const int first = h->ncells;
  std::vector<double> comp(n * (size_t)nv);
  for (int a = 0; a < 3; ++a) {
    for (size_t k = 0; k < comp.size(); ++k) comp[k] = xyz[3 * k + a];
    HC_CUDA(h, cudaMemcpyAsync(h->x + a * h->Vcap + h->nvert, comp.data(), 8 * comp.size(), cudaMemcpyHostToDevice,
                               h->stream));
    HC_CUDA(h, cudaStreamSynchronize(h->stream));
  }
  std::vector<int> vc(n * (size_t)nv), ct(n), co(n), al(n, 1);
  for (int c = 0; c < n; ++c) {
    ct[c] = type;
    co[c] = h->nvert + c * nv;
    for (int k = 0; k < nv; ++k) vc[(size_t)c * nv + k] = first + c;
    h->h_cell_type.push_back(type);
    h->h_cell_voff.push_back(co[c]);
    ts.cells.push_back(first + c);
  }
  HC_CUDA(h, cudaMemcpyAsync(h->vcell + h->nvert, vc.data(), 4 * vc.size(), cudaMemcpyHostToDevice, h->stream));
  HC_CUDA(h, cudaMemcpyAsync(h->cell_type + first, ct.data(), 4 * n, cudaMemcpyHostToDevice, h->stream));
  HC_CUDA(h, cudaMemcpyAsync(h->cell_voff + first, co.data(), 4 * n, cudaMemcpyHostToDevice, h->stream));
  HC_CUDA(h, cudaMemcpyAsync(h->alive + first, al.data(), 4 * n, cudaMemcpyHostToDevice, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  h->nvert += n * nv;
  h->ncells += n;
  apply_rules(h);
  if ((rc = ensure_repulsion(h)) != HC_OK) return rc;
  return upload_cell_lists(h);
}

// device [3][Vcap] (T) -> host [V][3] double: transpose on the device, then
// one D2H copy straight into the caller's buffer
template <typename T>
int read3(hc_handle* h, const void* src, double* out) {
  int rc;
  if ((rc = ensure_scratch(h, sizeof(double) * 3 * std::max<int>(1, h->nvert))) != HC_OK) return rc;
  HC_CUDA(h, hcd::launch_soa_to_aos<T>((const T*)src, h->scratch, h->Vcap, h->nvert, h->stream));
  HC_CUDA(h, cudaMemcpyAsync(out, h->scratch, 8 * 3 * (size_t)h->nvert, cudaMemcpyDeviceToHost, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return HC_OK;
}

int write3(hc_handle* h, void* dst, size_t es, const double* in) {
  const long long V = h->Vcap;
  std::vector<double> buf(3 * V, 0.0);
  for (int i = 0; i < h->nvert; ++i)
    for (int a = 0; a < 3; ++a) buf[a * V + i] = in[3 * i + a];
  if (es == 8) {
    HC_CUDA(h, cudaMemcpyAsync(dst, buf.data(), 8 * 3 * V, cudaMemcpyHostToDevice, h->stream));
  } else {
    int rc;
    if ((rc = ensure_scratch(h, sizeof(double) * 3 * V)) != HC_OK) return rc;
    HC_CUDA(h, cudaMemcpyAsync(h->scratch, buf.data(), 8 * 3 * V, cudaMemcpyHostToDevice, h->stream));
    HC_CUDA(h, hcd::launch_convert_in<float>(h->scratch, (float*)dst, 3 * V, h->stream));
  }
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return HC_OK;
}

// ----- autotuner: time candidate launch shapes on the live state --------
std::string tune_key(hc_handle* h) {
  std::ostringstream k;
  k << (h->f64 ? "f64" : "f32") << "_" << h->nx << "x" << h->ny << "x" << h->nz << "_V" << h->nvert << "_C"
    << h->ncells << "_L" << h->p.launch;
  return k.str();
}

template <typename T>
int autotune(hc_handle* h, const char* cache) {
  const std::string key = tune_key(h);
  if (cache && *cache) {
    std::ifstream in(cache);
    std::string k;
    int t[8];
    while (in >> k >> t[0] >> t[1] >> t[2] >> t[3] >> t[4] >> t[5] >> t[6] >> t[7])
      if (k == key) {
        int old_tune[8];
        std::memcpy(old_tune, h->tune, sizeof(old_tune));
        std::memcpy(h->tune, t, sizeof(t));
        h->tuned = true;
        if (!set_bulk_plan<T>(h, h->tune[7])) h->tune[7] = 0;
        invalidate_graph(h);
        return retag_if_needed(h, old_tune);
      }
  }
  // Every candidate runs real steps (no graph) from the same device snapshot
  // of the state, and the fastest whole step wins; the state is put back at
  // the end.  Timing a kernel alone on repeated inputs favours variants that
  // reuse L2 in a way the step does not.
  const size_t Fb = h->f64 ? hcd::field_bytes<double>(h->N) : hcd::field_bytes<float>(h->N);
  std::vector<std::pair<void*, size_t>> parts = {{h->f[h->cur], 19 * h->ts * (size_t)h->N}, {h->F[0], Fb}, {h->F[1], Fb}};
  if (h->Vcap > 0 && h->x) {
    parts.push_back({h->x, 3 * 8 * (size_t)h->Vcap});
    parts.push_back({h->v, 3 * h->ts * (size_t)h->Vcap});
    parts.push_back({h->fv, 3 * h->ts * (size_t)h->Vcap});
  }
  if (h->ncells > 0) parts.push_back({h->alive, 4 * (size_t)h->ncells});
  if (h->frep_cell) parts.push_back({h->frep_cell, 3 * h->ts * (size_t)h->rep_vcap});
  if (h->frep_wall) parts.push_back({h->frep_wall, 3 * h->ts * (size_t)h->rep_vcap});
  parts.push_back({h->status, sizeof(unsigned int)});
  parts.push_back({h->stamp, sizeof(uint32_t)});
  // the node tags: a spread already fused into the next force field has
  // tagged its stencil nodes, and the tagged node-velocity forms evaluate
  // only nodes whose tag equals the step stamp; the trial steps overwrite
  // tags with later stamps
  parts.push_back({h->ntag, sizeof(uint32_t) * (size_t)h->N});
  size_t total = 0;
  for (auto& pr : parts) total += (pr.second + 255) / 256 * 256;
  char* snap = nullptr;
  HC_CUDA(h, cudaMallocFromPoolAsync((void**)&snap, total, h->pool, h->stream));
  // the snapshot goes back to the pool on every return path
  struct SnapGuard {
    char*& p;
    cudaStream_t s;
    ~SnapGuard() {
      if (p) cudaFreeAsync(p, s);
    }
  } snap_guard{snap, h->stream};
  {
    size_t off = 0;
    for (auto& pr : parts) {
      HC_CUDA(h, cudaMemcpyAsync(snap + off, pr.first, pr.second, cudaMemcpyDeviceToDevice, h->stream));
      off += (pr.second + 255) / 256 * 256;
    }
  }
  const int cur0 = h->cur, iter0 = h->iter;
  const bool sd0 = h->spread_done, sa0 = h->stamp_ahead;
  int tune0[8];
  std::memcpy(tune0, h->tune, sizeof(tune0));
  auto restore = [&]() -> int {
    size_t off = 0;
    for (auto& pr : parts) {
      HC_CUDA(h, cudaMemcpyAsync(pr.first, snap + off, pr.second, cudaMemcpyDeviceToDevice, h->stream));
      off += (pr.second + 255) / 256 * 256;
    }
    h->cur = cur0;
    h->iter = iter0;
    h->spread_done = sd0;
    h->stamp_ahead = sa0;
    return HC_OK;
  };
  ScopedEvents<2> tev;
  HC_CUDA(h, tev.create());
  cudaEvent_t ea = tev[0], eb = tev[1];
  // the fastest of five timings of the same steps from the same state:
  // candidates often differ by a few percent, about the spread of one timing
  auto trial = [&]() -> float {
    float best_ms = 1e30f;
    for (int rep = 0; rep < 5; ++rep) {
      if (restore() != HC_OK) return 1e30f;
      for (int k = 0; k < 2; ++k)
        if (enq_step<T>(h) != HC_OK) return 1e30f;
      cudaEventRecord(ea, h->stream);
      const int K = 12;
      for (int k = 0; k < K; ++k)
        if (enq_step<T>(h) != HC_OK) return 1e30f;
      cudaEventRecord(eb, h->stream);
      if (cudaEventSynchronize(eb) != cudaSuccess) return 1e30f;
      float ms = 0;
      cudaEventElapsedTime(&ms, ea, eb);
      if (cudaGetLastError() != cudaSuccess) return 1e30f;
      best_ms = std::min(best_ms, ms / K);
    }
    return best_ms;
  };
  // A candidate replaces the one kept so far only when it is faster by more
  // than half a percent, about the spread of a timing: among candidates that
  // time alike, the earlier one in the fixed order below stays, so repeated
  // runs on the same workload settle on the same pick.
  auto faster = [](float t, float kept) { return t < kept * 0.995f; };
  invalidate_graph(h);
  // collide-stream: (x, y)-blocks, whole rows, one thread per fluid node, bulk copies
  // (x, y)-blocks of whole rows, and blocks whose warps are 8 x 4 or 16 x 2
  // tiles, for which most warps away from walls hold only interior nodes
  const int k1[][2] = {{0, 1},  {0, 2},  {0, 4},  {32, 4}, {64, 2}, {64, 4}, {128, 1}, {128, 2},
                       {256, 1}, {32, 8}, {8, 16}, {8, 32}, {16, 8}, {16, 16}};
  const int nvflags = h->tune[7] & 0x300;
  h->tuned = true;
  float best = 1e30f;
  int bx = h->tune[0], by = h->tune[1], b7 = h->tune[7] & 0xff;
  auto try_k1 = [&](int x0, int y0, int code) {
    h->tune[0] = x0;
    h->tune[1] = y0;
    h->tune[7] = code | nvflags;
    const float t = trial();
    if (faster(t, best)) {
      best = t;
      bx = x0;
      by = y0;
      b7 = code;
    }
  };
  const bool fast32 = 19LL * h->N < (1LL << 31);
  for (auto& c : k1) {
    if (c[0] > 2 * h->nx && c[0] > 32) continue;
    if (c[0] == 0 && h->nx * c[1] > 256) continue;
    try_k1(c[0], c[1], 0);
    // the interior pull (bit 12) of the direct kernel
    if (fast32 && !(c[0] == 0 && h->nx <= 256)) try_k1(c[0], c[1], 0x1000);
  }
  if (h->nfluid > 0)
    for (int bs : {128, 256})
      for (int var : {0, 0x1000}) try_k1(bs, 1, 1 | var);
  for (int ctas : {1, 2})
    for (int st : {3, 4}) {
      const int code = st | (ctas << 4);
      if (set_bulk_plan<T>(h, code)) try_k1(bx, by, code);
    }
  h->tune[0] = bx;
  h->tune[1] = by;
  h->tune[7] = b7 | nvflags;
  if ((b7 & 0xff) >= 2) set_bulk_plan<T>(h, b7);
  // interpolation + advance fused into the force assembly (bit 11 turns it off)
  {
    const int keep = h->tune[7];
    h->tune[7] = keep | 0x800;
    const float t = trial();
    if (faster(t, best)) {
      best = t;
      b7 |= 0x800;
    } else {
      h->tune[7] = keep;
    }
  }
  // evict-last population stores of the direct or fluid-list collide-stream (bit 13)
  const bool direct = (b7 & 0xff) == 0 && fast32 && !(h->tune[0] == 0 && h->nx <= 256);
  if (direct || (b7 & 0xff) == 1) {
    const int keep = h->tune[7];
    h->tune[7] = keep | 0x2000;
    const float t = trial();
    if (faster(t, best)) {
      best = t;
      b7 |= 0x2000;
    } else {
      h->tune[7] = keep;
    }
  }
  // programmatic dependent launch of the step's kernels (bit 10)
  {
    const int keep = h->tune[7];
    h->tune[7] = keep | 0x400;
    const float t = trial();
    if (faster(t, best)) {
      best = t;
      b7 |= 0x400;
    } else {
      h->tune[7] = keep;
    }
  }
  if (h->nvert > 0) {
    // node velocity variant and the IBM block size
    best = 1e30f;
    int bb = h->tune[3], nvf = nvflags;
    for (int fl : {0, 0x100, 0x200, 0x300})
      for (int bs : {64, 128, 256}) {
        if (fl == 0x100 && h->nfluid == 0) continue;
        if (fl >= 0x200 && 19LL * h->N >= (1LL << 31)) continue;
        h->tune[2] = h->tune[3] = bs;
        h->tune[7] = b7 | fl;
        const float t = trial();
        if (faster(t, best)) {
          best = t;
          bb = bs;
          nvf = fl;
        }
      }
    h->tune[2] = h->tune[3] = bb;
    h->tune[7] = b7 | nvf;
    // membrane forces: variant x block size x grid
    best = 1e30f;
    int mb = h->tune[4], mg = h->tune[5], mv = h->tune[6];
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->p.device);
    for (int var : {0, 1, 2})
      for (int bs : {128, 256, 384, 512, 768})
        for (int gr : {0, 2 * sms}) {
          if (bs > (h->f64 ? 384 : 768)) continue;
          if (var == 2 && (gr != 0 || bs > 384)) continue;  // a cluster per cell, at most 384 threads a CTA
          if (gr != 0 && h->p.launch != HC_LAUNCH_BATCHED) continue;
          h->tune[4] = bs;
          h->tune[5] = gr;
          h->tune[6] = var;
          const float t = trial();
          if (faster(t, best)) {
            best = t;
            mb = bs;
            mg = gr;
            mv = var;
          }
        }
    h->tune[4] = mb;
    h->tune[5] = mg;
    h->tune[6] = mv;
  }
  int rc = restore();
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  HC_CUDA(h, cudaFreeAsync(snap, h->stream));
  snap = nullptr;
  if (rc != HC_OK) return rc;
  invalidate_graph(h);
  if ((rc = retag_if_needed(h, tune0)) != HC_OK) return rc;
  if (cache && *cache) {
    std::ofstream out(cache, std::ios::app);
    out << key;
    for (int k = 0; k < 8; ++k) out << " " << h->tune[k];
    out << "\n";
  }
  return HC_OK;
}

template <typename T>
int profile_stages(hc_handle* h, int nsteps, double* out) {
  int rc0 = undo_fused_spread(h);  // every profiled step spreads on its own
  if (rc0 != HC_OK) return rc0;
  ScopedEvents<5> ev;
  HC_CUDA(h, ev.create());
  double acc[5] = {0, 0, 0, 0, 0};
  for (int k = 0; k < nsteps; ++k) {
    int rc;
    HC_CUDA(h, cudaEventRecord(ev[0], h->stream));
    if ((rc = enq_spread<T>(h)) != HC_OK) return rc;
    HC_CUDA(h, cudaEventRecord(ev[1], h->stream));
    if ((rc = enq_collide<T>(h)) != HC_OK) return rc;
    HC_CUDA(h, cudaEventRecord(ev[2], h->stream));
    if ((rc = enq_interp_advance<T>(h, h->iter % h->velocity_every == 0, 1)) != HC_OK) return rc;
    HC_CUDA(h, cudaEventRecord(ev[3], h->stream));
    if ((rc = enq_mechanics<T>(h, false)) != HC_OK) return rc;
    HC_CUDA(h, cudaEventRecord(ev[4], h->stream));
    h->iter++;
    HC_CUDA(h, cudaEventSynchronize(ev[4]));
    float t;
    for (int s = 0; s < 4; ++s) {
      HC_CUDA(h, cudaEventElapsedTime(&t, ev[s], ev[s + 1]));
      acc[s] += t;
    }
    HC_CUDA(h, cudaEventElapsedTime(&t, ev[0], ev[4]));
    acc[4] += t;
  }
  for (int s = 0; s < 5; ++s) out[s] = nsteps > 0 ? acc[s] / nsteps : 0.0;
  return HC_OK;
}

// Device time of each kernel group inside the step as hc_step runs it in
// the batched launch (the same kernels and fusions as the graph), launched
// one after another without a graph: three unprofiled steps are queued
// first and nothing synchronises in between, so the host stays ahead of the
// GPU and no launch gap falls between a kernel's two events.
// out[0] collide-stream, out[1] node velocity (or interpolation + advance
// when not fused), out[2] force assembly, out[3] whole step, in ms per step.
template <typename T>
int profile_kernels(hc_handle* h, int nsteps, double* out) {
  int rc;
  if (h->prof_ev.size() < (size_t)nsteps * 6) {
    for (auto e : h->prof_ev) cudaEventDestroy(e);
    h->prof_ev.assign((size_t)nsteps * 6, nullptr);
    for (auto& e : h->prof_ev) HC_CUDA(h, cudaEventCreate(&e));
  }
  for (int k = 0; k < 3; ++k)
    if ((rc = enq_step<T>(h)) != HC_OK) return rc;
  for (int k = 0; k < nsteps; ++k) {
    h->prof_step = k;
    rc = enq_step<T>(h);
    h->prof_step = -1;
    if (rc != HC_OK) return rc;
  }
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  double acc[4] = {0, 0, 0, 0};
  for (int k = 0; k < nsteps; ++k) {
    cudaEvent_t* e = &h->prof_ev[(size_t)k * 6];
    float t;
    for (int g = 0; g < 3; ++g) {
      HC_CUDA(h, cudaEventElapsedTime(&t, e[2 * g], e[2 * g + 1]));
      acc[g] += t;
    }
    if (k + 1 < nsteps) {
      HC_CUDA(h, cudaEventElapsedTime(&t, e[0], e[6]));
      acc[3] += t;
    }
  }
  for (int g = 0; g < 3; ++g) out[g] = nsteps > 0 ? acc[g] / nsteps : 0.0;
  out[3] = nsteps > 1 ? acc[3] / (nsteps - 1) : 0.0;
  return HC_OK;
}

// The stored state is post-collision; the walls decide how it is pulled.
// Changing them re-stores the current post-stream populations so that the
// fluid state itself is unchanged.
int restore_populations(hc_handle* h, const std::function<int()>& change) {
  int rc;
  if ((rc = ensure_scratch(h, sizeof(double) * 19 * h->N)) != HC_OK) return rc;
  if (h->f64) HC_CUDA(h, hcd::launch_stream_out<double>(lbm_view<double>(h, h->cur, h->cur), h->scratch, h->stream));
  else HC_CUDA(h, hcd::launch_stream_out<float>(lbm_view<float>(h, h->cur, h->cur), h->scratch, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  if ((rc = change()) != HC_OK) return rc;
  if (h->f64) HC_CUDA(h, hcd::launch_stream_in<double>(lbm_view<double>(h, 1 - h->cur, h->cur), h->scratch, 1.0, nullptr, h->stream));
  else HC_CUDA(h, hcd::launch_stream_in<float>(lbm_view<float>(h, 1 - h->cur, h->cur), h->scratch, 1.0, nullptr, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  shrink_scratch(h);
  return HC_OK;
}

}  // namespace

void hcd::set_handleless_error(const std::string& msg) { g_create_error = msg; }
cudaStream_t hcd::handle_stream(const hc_handle* h) { return h->stream; }
int hcd::handle_device(const hc_handle* h) { return h->p.device; }
long long hcd::handle_bytes(const hc_handle* h) { return h->device_bytes; }

// ===========================================================================
extern "C" {

hc_handle* hc_create(const hc_params* p) {
  g_create_error.clear();
  if (!p) {
    g_create_error = "null params";
    return nullptr;
  }
  if (p->nx <= 0 || p->ny <= 0 || p->nz <= 0) {
    g_create_error = "lattice dimensions must be positive";
    return nullptr;
  }
  if ((long long)p->nx * p->ny * p->nz * 19 >= (1LL << 31) * 4) {
    g_create_error = "lattice too large";
    return nullptr;
  }
  if (!(p->dx > 0) || !(p->dt > 0) || !(p->rho_p > 0)) {
    g_create_error = "dx, dt and rhoP must be positive";
    return nullptr;
  }
  if (p->form != HC_FORM_PLAIN_F64 && p->form != HC_FORM_MIXED_F32) {
    g_create_error = "unknown precision form";
    return nullptr;
  }
  if (p->launch != HC_LAUNCH_PER_STAGE && p->launch != HC_LAUNCH_BATCHED) {
    g_create_error = "unknown launch mode";
    return nullptr;
  }
  hcg::Units u = hcg::derive_units(p->dx, p->dt, p->nu_p, p->rho_p, p->kBT_p, p->tau);
  if (!(u.tau > 0.5)) {
    // core/hemoCell.cpp sanityCheck: tau must exceed 1/2 for a positive viscosity
    g_create_error = "tau must be > 0.5";
    return nullptr;
  }
  hc_handle* h = new hc_handle();
  h->p = *p;
  h->u = u;
  std::memset(h->uw, 0, sizeof(h->uw));
  h->nx = p->nx;
  h->ny = p->ny;
  h->nz = p->nz;
  h->N = (long long)p->nx * p->ny * p->nz;
  h->f64 = p->form == HC_FORM_PLAIN_F64;
  h->ts = h->f64 ? 8 : 4;
  h->tg.tx = p->tile[0] > 0 ? p->tile[0] : 8;
  h->tg.ty = p->tile[1] > 0 ? p->tile[1] : 8;
  h->tg.tz = p->tile[2] > 0 ? p->tile[2] : 8;
  h->tg.ntx = (h->nx + h->tg.tx - 1) / h->tg.tx;
  h->tg.nty = (h->ny + h->tg.ty - 1) / h->tg.ty;
  h->tg.ntz = (h->nz + h->tg.tz - 1) / h->tg.tz;
  h->ntiles = h->tg.ntx * h->tg.nty * h->tg.ntz;
  auto bail = [&](const std::string& m) {
    g_create_error = m;
    hc_destroy(h);
    return (hc_handle*)nullptr;
  };
  cudaError_t e = cudaSetDevice(p->device);
  if (e != cudaSuccess) return bail(std::string("cudaSetDevice: ") + cudaGetErrorString(e));
  if ((e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking)) != cudaSuccess)
    return bail(std::string("stream: ") + cudaGetErrorString(e));
  if ((e = acquire_pool(p->device, &h->pool)) != cudaSuccess)
    return bail(std::string("memory pool: ") + cudaGetErrorString(e));
  const size_t fb = 19 * h->ts * (size_t)h->N;
  const size_t Fb = h->f64 ? hcd::field_bytes<double>(h->N) : hcd::field_bytes<float>(h->N);
  for (int k = 0; k < 2; ++k) {
    if ((e = dalloc(h, &h->f[k], fb)) != cudaSuccess) return bail("out of device memory (populations)");
    if ((e = dalloc(h, &h->F[k], Fb)) != cudaSuccess) return bail("out of device memory (force field)");
    cudaMemsetAsync(h->f[k], 0, fb, h->stream);
    cudaMemsetAsync(h->F[k], 0, Fb, h->stream);
  }
  if (dalloc(h, (void**)&h->ntag, 4 * h->N) != cudaSuccess || dalloc(h, &h->unode, Fb) != cudaSuccess ||
      dalloc(h, (void**)&h->stamp, 4) != cudaSuccess)
    return bail("out of device memory (node tags)");
  cudaMemsetAsync(h->ntag, 0, 4 * h->N, h->stream);
  cudaMemsetAsync(h->unode, 0, Fb, h->stream);
  {
    const uint32_t one = 1;
    cudaMemcpyAsync(h->stamp, &one, 4, cudaMemcpyHostToDevice, h->stream);
  }
  if (dalloc(h, (void**)&h->nbmask, 4 * h->N) != cudaSuccess || dalloc(h, (void**)&h->flag, h->N) != cudaSuccess ||
      dalloc(h, (void**)&h->corner, h->N) != cudaSuccess ||
      dalloc(h, &h->bodyz, 3 * h->ts * h->nz) != cudaSuccess ||
      dalloc(h, (void**)&h->dtypes, sizeof(TypeDev) * hcd::MAX_TYPES) != cudaSuccess ||
      dalloc(h, (void**)&h->status, sizeof(unsigned int)) != cudaSuccess)
    return bail("out of device memory");
  cudaMemsetAsync(h->bodyz, 0, 3 * h->ts * h->nz, h->stream);
  cudaMemsetAsync(h->status, 0, sizeof(unsigned int), h->stream);
  h->hflag.assign(h->N, 0);
  cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, p->device);
  cudaDeviceGetAttribute(&h->l2, cudaDevAttrL2CacheSize, p->device);
  if (upload_flags(h) != HC_OK) return bail(h->err);
  if ((e = cudaStreamSynchronize(h->stream)) != cudaSuccess) return bail(cudaGetErrorString(e));
  return h;
}

int hc_destroy(hc_handle* h) {
  if (!h) return HC_OK;
  if (h->stream) cudaStreamSynchronize(h->stream);
  invalidate_graph(h);
  for (int k = 0; k < 2; ++k) {
    dfree(h, h->f[k]);
    dfree(h, h->F[k]);
  }
  for (TypeSlot& ts : h->types) {
    dfree(h, ts.blob);
    dfree(h, ts.dcells);
  }
  void* ptrs[] = {h->ntag, h->unode, h->stamp, h->nbmask, h->flag, h->corner, h->bodyz,     h->dtypes,     h->x,          h->v,
                  h->fv,     h->vcell, h->vnode,     h->vtile,      h->cell_type,  h->cell_voff,
                  h->alive,  h->dcells_all, h->status, h->bin_counts, h->bin_cursor, h->bin_offsets,
                  h->tile_vertices, h->tile_cell_counts, h->tile_cell_offsets, h->tile_cells, h->scratch,
                  h->ext_ids, h->ext_f, h->rep_cnt, h->rep_slot, h->rep_vq, h->rep_xr, h->rep_bnode,
                  h->frep_cell, h->frep_wall, h->fluid};
  for (void* q : ptrs) dfree(h, q);
  for (auto e : h->prof_ev) cudaEventDestroy(e);
  if (h->copy_stream) cudaStreamSynchronize(h->copy_stream);
  for (int k = 0; k < 2; ++k) {
    dfree(h, h->pos_stage[k]);
    if (h->pos_ready[k]) cudaEventDestroy(h->pos_ready[k]);
    if (h->pos_copied[k]) cudaEventDestroy(h->pos_copied[k]);
  }
  if (h->copy_stream) cudaStreamDestroy(h->copy_stream);
  dfree(h, h->bodyd);
  if (h->body_copied) {
    cudaEventSynchronize(h->body_copied);
    cudaEventDestroy(h->body_copied);
  }
  if (h->hbody_pin) cudaFreeHost(h->hbody_pin);
  if (h->pool) release_pool(h->p.device, h->stream);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
  return HC_OK;
}

const char* hc_last_error(const hc_handle* h) { return h ? h->err.c_str() : g_create_error.c_str(); }

int hc_derived_units(const hc_handle* h, double* out) {
  if (!h || !out) return HC_ERR_INVALID;
  out[0] = h->u.tau;
  out[1] = h->u.nu_lbm;
  out[2] = h->u.dm;
  out[3] = h->u.df;
  out[4] = h->u.kBT_lbm;
  out[5] = h->u.f_limit;
  return HC_OK;
}

int hc_set_flags(hc_handle* h, const uint8_t* flags) {
  if (!h || !flags) return HC_ERR_INVALID;
  if (int rc0 = undo_fused_spread(h)) return rc0;
  invalidate_graph(h);
  return restore_populations(h, [&]() {
    std::memcpy(h->hflag.data(), flags, h->N);
    return upload_flags(h);
  });
}

int hc_set_wall_velocity(hc_handle* h, int cls, const double* u3) {
  if (!h || !u3) return HC_ERR_INVALID;
  if (cls < 0 || cls >= hcd::MAX_WALL_CLASSES) return fail(h, HC_ERR_INVALID, "wall class out of range [0,16)");
  invalidate_graph(h);
  return restore_populations(h, [&]() {
    for (int a = 0; a < 3; ++a) h->uw[cls][a] = u3[a];
    return HC_OK;
  });
}

int hc_set_body_force(hc_handle* h, int mode, const double* p) {
  if (!h) return HC_ERR_INVALID;
  if (mode < HC_BODY_NONE || mode > HC_BODY_KOLMOGOROV) return fail(h, HC_ERR_INVALID, "unknown body-force mode");
  if (mode != HC_BODY_NONE && !p) return fail(h, HC_ERR_INVALID, "body-force parameters missing");
  // the driver's setExternalVector after every iterate(): the profile is
  // copied again, and the same force changes nothing else (the reset to it is
  // part of the collide-stream)
  if (mode == h->body_mode &&
      (mode == HC_BODY_NONE || (p[0] == h->body[0] && (mode == HC_BODY_KOLMOGOROV || (p[1] == h->body[1] && p[2] == h->body[2])))))
    return upload_profile(h, body_profile(h), nullptr);
  if (h->spread_done) {
    // the next step's force field holds the old body force and the spread
    // fused into it: add the change of the body force, keep the spread
    const std::vector<double> old = body_profile(h);
    h->body_mode = mode;
    for (int a = 0; a < 3; ++a) h->body[a] = (mode != HC_BODY_NONE) ? p[a] : 0.0;
    if (mode == HC_BODY_KOLMOGOROV) h->body[1] = h->body[2] = 0.0;
    const std::vector<double> prof = body_profile(h);
    std::vector<double> change(prof.size());
    for (size_t k = 0; k < prof.size(); ++k) change[k] = prof[k] - old[k];
    int rc;
    if ((rc = upload_profile(h, prof, &change)) != HC_OK) return rc;
    const long long plane = (long long)h->nx * h->ny;
    if (h->f64)
      HC_CUDA(h, hcd::launch_add_body<double>((double*)h->F[h->cur], (const double*)h->bodyd, plane, h->nz, h->N,
                                              h->stream));
    else
      HC_CUDA(h, hcd::launch_add_body<float>((float*)h->F[h->cur], (const float*)h->bodyd, plane, h->nz, h->N,
                                             h->stream));
    return HC_OK;
  }
  // the force field is refilled with the body force (the node-tag stamp
  // caught up with a fused advance first)
  int rc0 = undo_fused_spread(h);
  if (rc0 != HC_OK) return rc0;
  h->body_mode = mode;
  for (int a = 0; a < 3; ++a) h->body[a] = (mode != HC_BODY_NONE) ? p[a] : 0.0;
  if (mode == HC_BODY_KOLMOGOROV) h->body[1] = h->body[2] = 0.0;
  return upload_body(h);
}

int hc_init_equilibrium(hc_handle* h, double rho, const double* u3) {
  if (!h) return HC_ERR_INVALID;
  if (!(rho > 0)) return fail(h, HC_ERR_INVALID, "density must be positive");
  // post-collision values whose pull is the equilibrium of (rho, u)
  if (h->f64) HC_CUDA(h, hcd::launch_stream_in<double>(lbm_view<double>(h, 1 - h->cur, h->cur), nullptr, rho, u3, h->stream));
  else HC_CUDA(h, hcd::launch_stream_in<float>(lbm_view<float>(h, 1 - h->cur, h->cur), nullptr, rho, u3, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return HC_OK;
}

int hc_add_cell_type(hc_handle* h, const char* name, int model, const hc_material* m, const double* xyz, int nv,
                     const int* tris, int nf, const int* inner, int ni) {
  if (!h || !m || !xyz || !tris) return HC_ERR_INVALID;
  if ((int)h->types.size() >= hcd::MAX_TYPES) return fail(h, HC_ERR_INVALID, "more than 8 cell types");
  if (model < HC_MODEL_RBC_HIGH_ORDER || model > HC_MODEL_WBC_HIGH_ORDER)
    return fail(h, HC_ERR_INVALID, "unknown constitutive model");
  if (nv <= 0 || nf <= 0 || ni < 0 || (ni > 0 && !inner)) return fail(h, HC_ERR_INVALID, "bad mesh sizes");
  if (nv > 65535) return fail(h, HC_ERR_INVALID, "more vertices per cell than UINT16_MAX");
  TypeSlot ts;
  ts.name = name ? name : "";
  std::vector<hcg::Vec3> P(nv);
  for (int i = 0; i < nv; ++i) P[i] = {xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]};
  std::vector<std::array<int, 3>> T(nf);
  for (int k = 0; k < nf; ++k) T[k] = {tris[3 * k], tris[3 * k + 1], tris[3 * k + 2]};
  std::vector<std::array<int, 2>> I(ni);
  for (int k = 0; k < ni; ++k) I[k] = {inner[2 * k], inner[2 * k + 1]};
  std::string why = hcg::build_constants(ts.tc, model, P, T, I);
  if (!why.empty()) return fail(h, HC_ERR_INVALID, "cell type " + ts.name + ": " + why);
  const double mat[9] = {m->kLink, m->kBend, m->kVolume, m->kArea, m->eta_m,
                         m->kInnerRigid, m->kCytoskeleton, m->coreRadius, m->radius};
  ts.k = hcg::scale_material(model, nf, h->u, h->p.dx, h->p.dt, mat);
  const size_t smem = gather_bytes(h, ts);
  if (smem > 227 * 1024) return fail(h, HC_ERR_INVALID, "cell type too large for one CTA's shared memory");
  HC_CUDA(h, h->f64 ? hcd::prepare_mechanics<double>((int)smem, &h->staged_limit)
                    : hcd::prepare_mechanics<float>((int)smem, &h->staged_limit));
  {
    const size_t s16 = hcd::mechanics_staged_bytes(model, nv, nf, ts.tc.ne, 16, h->f64), g16 = gather_bytes(h, ts, 16);
    ts.cluster16 =
        s16 <= (size_t)h->staged_limit &&
        (h->f64 ? hcd::mechanics_cluster_fits<double>(true, 16, 384, (int)s16) &&
                      hcd::mechanics_cluster_fits<double>(false, 16, 384, (int)g16)
                : hcd::mechanics_cluster_fits<float>(true, 16, 384, (int)s16) &&
                      hcd::mechanics_cluster_fits<float>(false, 16, 384, (int)g16));
  }
  // one device blob: ints then doubles
  const hcg::TypeConstants& c = ts.tc;
  std::vector<int> iv;
  auto put_i = [&](const std::vector<int>& a) {
    size_t o = iv.size();
    iv.insert(iv.end(), a.begin(), a.end());
    return o;
  };
  const size_t o_tris = put_i(c.tris), o_edges = put_i(c.edges), o_bt = put_i(c.bend_tris),
               o_bo = put_i(c.bend_outer), o_ring = put_i(c.ring), o_rn = put_i(c.ring_n), o_in = put_i(c.inner),
               o_ve = put_i(c.vedge), o_vo = put_i(c.vopp), o_vio = put_i(c.vinner_off), o_vi = put_i(c.vinner);
  // the packed tables (TypeDev), each from a 16-byte boundary.  Their 16-bit
  // indices hold every type: with at most six edges a vertex, nf <= 2 nv and
  // ne <= 3 nv, and the shared memory above limits nv to 9,300.
  auto align16 = [&] {
    while (iv.size() % 4) iv.push_back(0);
    return iv.size();
  };
  auto put_six = [&](const std::vector<int>& a, bool ring) {
    const size_t o = align16();
    for (int i = 0; i < c.nv; ++i) {
      uint32_t lane[8] = {};
      for (int j = 0; j < c.ring_n[i]; ++j) {
        lane[j] = (uint32_t)a[6 * i + j];
        if (ring) lane[7] |= (uint32_t)c.slot_rot[6 * i + j] << (2 * j);
      }
      if (ring) lane[6] = (uint32_t)c.ring_n[i];
      for (int w = 0; w < 4; ++w) iv.push_back((int)(lane[2 * w] | lane[2 * w + 1] << 16));
    }
    return o;
  };
  const size_t o_r16 = put_six(c.ring, true), o_vf16 = put_six(c.vface, false), o_ve16 = put_six(c.vedge, false),
               o_vo16 = put_six(c.vopp, false), o_t16 = align16();
  for (int k = 0; k < c.nf; ++k) {
    iv.push_back(c.tris[3 * k] | (int)((uint32_t)c.tris[3 * k + 1] << 16));
    iv.push_back(c.tris[3 * k + 2]);
  }
  const size_t o_e16 = align16();
  for (int e = 0; e < c.ne; ++e) iv.push_back(c.edges[2 * e] | (int)((uint32_t)c.edges[2 * e + 1] << 16));
  align16();
  std::vector<double> dv;
  auto put_d = [&](const std::vector<double>& a) {
    size_t o = dv.size();
    dv.insert(dv.end(), a.begin(), a.end());
    return o;
  };
  const size_t o_a0 = put_d(c.tri_a0), o_l0 = put_d(c.edge_l0), o_ang = put_d(c.edge_angle0),
               o_pd = put_d(c.patch_d0), o_il = put_d(c.inner_l0);
  // the mixed form reads 32-bit copies, and its slots' rest values from one
  // table; the plain form also the reciprocals of the rest areas and lengths
  std::vector<float> fv;
  size_t o_sa = 0, o_sl = 0, o_ia = 0, o_iel = 0, o_sf = 0;
  if (h->f64) {
    o_sa = put_d(c.slot_a0);
    o_sl = put_d(c.slot_l0);
    auto reciprocals = [](std::vector<double> a) {
      for (double& x : a) x = 1.0 / x;
      return a;
    };
    o_ia = put_d(reciprocals(c.tri_a0));
    o_iel = put_d(reciprocals(c.edge_l0));
  } else {
    fv.assign(dv.begin(), dv.end());
    while (fv.size() % 4) fv.push_back(0.f);
    o_sf = fv.size();
    for (int i = 0; i < c.nv; ++i) {
      for (int j = 0; j < 6; ++j) fv.push_back((float)c.slot_a0[6 * i + j]);
      for (int j = 0; j < 6; ++j) fv.push_back((float)c.slot_l0[6 * i + j]);
    }
  }
  if (dv.size() % 2) dv.push_back(0.0);  // the floats from a 16-byte boundary too
  const size_t ib = 4 * iv.size(), db = 8 * std::max<size_t>(dv.size(), 1), fb = 4 * std::max<size_t>(fv.size(), 1);
  HC_CUDA(h, dalloc(h, &ts.blob, ib + db + fb));
  HC_CUDA(h, cudaMemcpyAsync(ts.blob, iv.data(), ib, cudaMemcpyHostToDevice, h->stream));
  if (!dv.empty())
    HC_CUDA(h, cudaMemcpyAsync((char*)ts.blob + ib, dv.data(), 8 * dv.size(), cudaMemcpyHostToDevice, h->stream));
  if (!fv.empty())
    HC_CUDA(h, cudaMemcpyAsync((char*)ts.blob + ib + db, fv.data(), 4 * fv.size(), cudaMemcpyHostToDevice, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  const int* ibase = (const int*)ts.blob;
  const double* dbase = (const double*)((char*)ts.blob + ib);
  const float* fbase = (const float*)((char*)ts.blob + ib + db);
  TypeDev& d = ts.dev;
  d.model = model;
  d.nv = c.nv;
  d.nf = c.nf;
  d.ne = c.ne;
  d.ni = c.ni;
  d.tris = ibase + o_tris;
  d.edges = ibase + o_edges;
  d.bend_tris = ibase + o_bt;
  d.bend_outer = ibase + o_bo;
  d.ring = ibase + o_ring;
  d.ring_n = ibase + o_rn;
  d.inner = ibase + o_in;
  d.vedge = ibase + o_ve;
  d.vopp = ibase + o_vo;
  d.vinner_off = ibase + o_vio;
  d.vinner = ibase + o_vi;
  d.slot_a0 = h->f64 ? dbase + o_sa : nullptr;
  d.slot_l0 = h->f64 ? dbase + o_sl : nullptr;
  d.ring16 = (const uint4*)(ibase + o_r16);
  d.vface16 = (const uint4*)(ibase + o_vf16);
  d.vedge16 = (const uint4*)(ibase + o_ve16);
  d.vopp16 = (const uint4*)(ibase + o_vo16);
  d.tris16 = (const uint2*)(ibase + o_t16);
  d.edges16 = (const uint32_t*)(ibase + o_e16);
  d.slot_f = h->f64 ? nullptr : (const float4*)(fbase + o_sf);
  d.tri_a0 = dbase + o_a0;
  d.edge_l0 = dbase + o_l0;
  d.tri_ia0 = h->f64 ? dbase + o_ia : nullptr;
  d.edge_il0 = h->f64 ? dbase + o_iel : nullptr;
  d.edge_angle0 = dbase + o_ang;
  d.patch_d0 = dbase + o_pd;
  d.inner_l0 = dbase + o_il;
  d.tri_a0f = fbase + o_a0;
  d.edge_l0f = fbase + o_l0;
  d.edge_angle0f = fbase + o_ang;
  d.patch_d0f = fbase + o_pd;
  d.inner_l0f = fbase + o_il;
  d.volume_eq = c.volume_eq;
  d.inv_volume_eq = 1.0 / c.volume_eq;
  d.area_mean_eq = c.area_mean_eq;
  d.inv_area_mean_eq = 1.0 / c.area_mean_eq;
  d.edge_mean_eq = c.edge_mean_eq;
  d.k_link = ts.k.k_link;
  d.k_bend = ts.k.k_bend;
  d.k_volume = ts.k.k_volume;
  d.k_area = ts.k.k_area;
  d.eta_m = ts.k.eta_m;
  d.k_inner_rigid = ts.k.k_inner_rigid;
  d.k_cyto = ts.k.k_cyto;
  d.core_radius = ts.k.core_radius;
  d.radius = ts.k.radius;
  h->types.push_back(std::move(ts));
  invalidate_graph(h);
  int rc = upload_types(h);
  if (rc != HC_OK) return rc;
  return (int)h->types.size() - 1;
}

int hc_add_cells(hc_handle* h, int type, int n, const double* centres, const double* angles) {
  if (!h || n < 0 || (n > 0 && (!centres || !angles))) return HC_ERR_INVALID;
  if (type < 0 || type >= (int)h->types.size()) return fail(h, HC_ERR_INVALID, "unknown cell type");
  std::vector<double> xyz;
  xyz.reserve(3 * (size_t)n * h->types[type].tc.nv);
  for (int c = 0; c < n; ++c) hcg::place_cell(h->types[type].tc.rest, centres + 3 * c, angles + 3 * c, xyz);
  const int first = h->ncells;
  int rc = add_cells_positions(h, type, n, xyz);
  return rc == HC_OK ? first : rc;
}

// loadParticles' admission of one placed cell (io/readPositionsBloodCells.cpp:120-170
// and the deleteIncompleteCells that follows it, :354): a vertex is added only
// when it lies in the lattice's box (-0.5, n - 0.5] on every axis
// (isContainedABS on the particle field's box; periodic axes are not
// wrapped at loading) and its node int(x + 0.5) is not a boundary node; a
// cell missing any vertex is deleted.  The deny layer of
// setInitialMinimumDistanceFromSolid is an unsigned number of micrometres in
// the reference (core/hemoCellField.h:64), so the 0.5 um its cases pass
// truncates to 0 and only the vertex's own node is checked.
bool cell_admitted(const hc_handle* h, const double* xyz, int nv) {
  const int dims[3] = {h->nx, h->ny, h->nz};
  for (int i = 0; i < nv; ++i) {
    long long q[3];
    for (int a = 0; a < 3; ++a) {
      const double x = xyz[3 * i + a];
      if (!(x > -0.5 && x <= dims[a] - 0.5)) return false;
      q[a] = (long long)(x + 0.5);
      if (q[a] >= dims[a]) return false;
    }
    if (h->hflag[(size_t)q[0] + (size_t)dims[0] * ((size_t)q[1] + (size_t)dims[1] * (size_t)q[2])]) return false;
  }
  return true;
}

int hc_load_cells(hc_handle* h, int type, int n, const double* centres, const double* angles, int* loaded) {
  if (!h || n < 0 || (n > 0 && (!centres || !angles))) return HC_ERR_INVALID;
  if (type < 0 || type >= (int)h->types.size()) return fail(h, HC_ERR_INVALID, "unknown cell type");
  const int nv = h->types[type].tc.nv;
  std::vector<double> keep, one;
  int kept = 0;
  for (int c = 0; c < n; ++c) {
    one.clear();
    hcg::place_cell(h->types[type].tc.rest, centres + 3 * c, angles + 3 * c, one);
    const bool ok = cell_admitted(h, one.data(), nv);
    if (loaded) loaded[c] = ok ? 1 : 0;
    if (!ok) continue;
    keep.insert(keep.end(), one.begin(), one.end());
    ++kept;
  }
  if (kept == 0) return 0;
  int rc = add_cells_positions(h, type, kept, keep);
  return rc == HC_OK ? kept : rc;
}

int hc_add_cells_xyz(hc_handle* h, int type, int n, const double* xyz) {
  if (!h || n < 0 || (n > 0 && !xyz)) return HC_ERR_INVALID;
  if (type < 0 || type >= (int)h->types.size()) return fail(h, HC_ERR_INVALID, "unknown cell type");
  std::vector<double> v(xyz, xyz + 3 * (size_t)n * h->types[type].tc.nv);
  const int first = h->ncells;
  int rc = add_cells_positions(h, type, n, v);
  return rc == HC_OK ? first : rc;
}

int hc_set_timescales(hc_handle* h, const int* every, int ntypes, int velocity_every) {
  if (!h) return HC_ERR_INVALID;
  if (velocity_every < 1) return fail(h, HC_ERR_INVALID, "velocity timescale must be >= 1");
  if (ntypes != (int)h->types.size() || (ntypes > 0 && !every))
    return fail(h, HC_ERR_INVALID, "one material timescale per cell type is required");
  for (int t = 0; t < ntypes; ++t) {
    if (every[t] < 1) return fail(h, HC_ERR_INVALID, "material timescale must be >= 1");
    // core/hemoCell.cpp:620-627
    if (every[t] % velocity_every != 0)
      return fail(h, HC_ERR_INVALID, "velocity timescale separation cannot divide all material timescale separations");
  }
  if (int rc0 = undo_fused_spread(h)) return rc0;
  for (int t = 0; t < ntypes; ++t) h->types[t].every = every[t];
  h->velocity_every = velocity_every;
  invalidate_graph(h);
  return HC_OK;
}

int hc_set_vertex_forces(hc_handle* h, int n, const int* ids, const double* forces) {
  if (!h || n < 0 || (n > 0 && (!ids || !forces))) return HC_ERR_INVALID;
  if (int rc0 = undo_fused_spread(h)) return rc0;
  for (int k = 0; k < n; ++k)
    if (ids[k] < 0 || ids[k] >= h->nvert) return fail(h, HC_ERR_INVALID, "vertex id out of range");
  if (n > h->next_cap) {
    dfree(h, h->ext_ids);
    dfree(h, h->ext_f);
    h->ext_ids = nullptr;
    h->ext_f = nullptr;
    HC_CUDA(h, dalloc(h, (void**)&h->ext_ids, sizeof(int) * n));
    HC_CUDA(h, dalloc(h, (void**)&h->ext_f, sizeof(double) * 3 * n));
    h->next_cap = n;
  }
  if (n > 0) {
    HC_CUDA(h, cudaMemcpyAsync(h->ext_ids, ids, sizeof(int) * n, cudaMemcpyHostToDevice, h->stream));
    HC_CUDA(h, cudaMemcpyAsync(h->ext_f, forces, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, h->stream));
    HC_CUDA(h, cudaStreamSynchronize(h->stream));
  }
  h->next = n;
  invalidate_graph(h);
  return HC_OK;
}

// HemoCell::setRepulsion (core/hemoCell.cpp:420-426); cutoff in lattice units
int hc_set_repulsion(hc_handle* h, double k, double cutoff, int every) {
  if (!h || !(cutoff >= 0)) return HC_ERR_INVALID;
  int rc;
  if ((rc = undo_fused_spread(h)) != HC_OK) return rc;
  h->rep_k = k;
  h->rep_rc = cutoff;
  h->rep_every = every > 0 ? every : 0;
  invalidate_graph(h);
  return ensure_repulsion(h);
}

// HemoCell::enableBoundaryParticles (core/hemoCell.cpp:428-436) with
// populateBoundaryParticles (core/hemoCellParticleField.cpp:865-889): wall
// nodes with a fluid node among their 26 neighbours (wrapped on periodic axes)
int hc_set_boundary_repulsion(hc_handle* h, double k, double cutoff, int every) {
  if (!h || !(cutoff >= 0)) return HC_ERR_INVALID;
  int rc;
  if ((rc = undo_fused_spread(h)) != HC_OK) return rc;
  h->brep_k = k;
  h->brep_rc = cutoff;
  h->brep_every = every > 0 ? every : 0;
  invalidate_graph(h);
  if (h->brep_every == 0) return HC_OK;
  std::vector<uint8_t> b(h->N, 0);
  const int dims[3] = {h->nx, h->ny, h->nz};
  for (int Z = 0; Z < h->nz; ++Z)
    for (int Y = 0; Y < h->ny; ++Y)
      for (int X = 0; X < h->nx; ++X) {
        const long long n = X + (long long)h->nx * (Y + (long long)h->ny * Z);
        if (h->hflag[n] == 0) continue;
        bool near_fluid = false;
        for (int dz = -1; dz <= 1 && !near_fluid; ++dz)
          for (int dy = -1; dy <= 1 && !near_fluid; ++dy)
            for (int dx = -1; dx <= 1 && !near_fluid; ++dx) {
              int q[3] = {X + dx, Y + dy, Z + dz};
              bool out = false;
              for (int a = 0; a < 3; ++a)
                if (q[a] < 0 || q[a] >= dims[a]) {
                  if (h->p.periodic[a]) q[a] = (q[a] + dims[a]) % dims[a];
                  else out = true;
                }
              if (!out && h->hflag[q[0] + (long long)h->nx * (q[1] + (long long)h->ny * q[2])] == 0) near_fluid = true;
            }
        b[n] = near_fluid ? 1 : 0;
      }
  // bit 1: the node or one of its 26 neighbours is a boundary node
  for (int Z = 0; Z < h->nz; ++Z)
    for (int Y = 0; Y < h->ny; ++Y)
      for (int X = 0; X < h->nx; ++X) {
        if (!(b[X + (long long)h->nx * (Y + (long long)h->ny * Z)] & 1)) continue;
        for (int dz = -1; dz <= 1; ++dz)
          for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) {
              int q[3] = {X + dx, Y + dy, Z + dz};
              bool out = false;
              for (int a = 0; a < 3; ++a)
                if (q[a] < 0 || q[a] >= dims[a]) {
                  if (h->p.periodic[a]) q[a] = (q[a] + dims[a]) % dims[a];
                  else out = true;
                }
              if (!out) b[q[0] + (long long)h->nx * (q[1] + (long long)h->ny * q[2])] |= 2;
            }
      }
  if (!h->rep_bnode) HC_CUDA(h, dalloc(h, (void**)&h->rep_bnode, h->N));
  HC_CUDA(h, cudaMemcpyAsync(h->rep_bnode, b.data(), h->N, cudaMemcpyHostToDevice, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return ensure_repulsion(h);
}

// force_repulsion of every vertex, [V][3] (both terms summed)
int hc_read_repulsion(hc_handle* h, double* f) {
  if (!h || !f) return HC_ERR_INVALID;
  const int V = h->nvert;
  std::vector<double> sum((size_t)3 * V, 0.0);
  int rc;
  for (void* src : {h->rep_every > 0 ? h->frep_cell : nullptr, h->brep_every > 0 ? h->frep_wall : nullptr}) {
    if (!src || V == 0) continue;
    if ((rc = ensure_scratch(h, sizeof(double) * 3 * V)) != HC_OK) return rc;
    if (h->f64) HC_CUDA(h, hcd::launch_soa_to_aos<double>((const double*)src, h->scratch, h->Vcap, V, h->stream));
    else HC_CUDA(h, hcd::launch_soa_to_aos<float>((const float*)src, h->scratch, h->Vcap, V, h->stream));
    std::vector<double> part((size_t)3 * V);
    HC_CUDA(h, cudaMemcpyAsync(part.data(), h->scratch, 8 * part.size(), cudaMemcpyDeviceToHost, h->stream));
    HC_CUDA(h, cudaStreamSynchronize(h->stream));
    for (size_t k = 0; k < part.size(); ++k) sum[k] += part[k];
  }
  std::memcpy(f, sum.data(), 8 * sum.size());
  return HC_OK;
}

int hc_step(hc_handle* h, int nsteps) {
  if (!h || nsteps < 0) return HC_ERR_INVALID;
  return h->f64 ? run_steps<double>(h, nsteps) : run_steps<float>(h, nsteps);
}

int hc_stage(hc_handle* h, int stage) {
  if (!h) return HC_ERR_INVALID;
  return h->f64 ? run_stage<double>(h, stage) : run_stage<float>(h, stage);
}

int hc_sync(hc_handle* h) {
  if (!h) return HC_ERR_INVALID;
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return HC_OK;
}

int hc_time_steps(hc_handle* h, int nsteps, double* ms) {
  if (!h || !ms || nsteps < 0) return HC_ERR_INVALID;
  ScopedEvents<2> ev;
  HC_CUDA(h, ev.create());
  HC_CUDA(h, cudaEventRecord(ev[0], h->stream));
  int rc = h->f64 ? run_steps<double>(h, nsteps) : run_steps<float>(h, nsteps);
  HC_CUDA(h, cudaEventRecord(ev[1], h->stream));
  HC_CUDA(h, cudaEventSynchronize(ev[1]));
  float t = 0;
  HC_CUDA(h, cudaEventElapsedTime(&t, ev[0], ev[1]));
  *ms = t;
  return rc;
}

int hc_profile_stages(hc_handle* h, int nsteps, double* ms5) {
  if (!h || !ms5 || nsteps < 0) return HC_ERR_INVALID;
  return h->f64 ? profile_stages<double>(h, nsteps, ms5) : profile_stages<float>(h, nsteps, ms5);
}

int hc_profile_kernels(hc_handle* h, int nsteps, double* ms4) {
  if (!h || !ms4 || nsteps < 1 || nsteps > 100000) return HC_ERR_INVALID;
  return h->f64 ? profile_kernels<double>(h, nsteps, ms4) : profile_kernels<float>(h, nsteps, ms4);
}

int hc_read_fluid(hc_handle* h, double* rho, double* u) {
  if (!h) return HC_ERR_INVALID;
  int rc;
  if ((rc = ensure_scratch(h, sizeof(double) * 4 * h->N)) != HC_OK) return rc;
  double* drho = h->scratch;
  double* du = h->scratch + h->N;
  if (h->f64) HC_CUDA(h, hcd::launch_moments<double>(lbm_view<double>(h, h->cur, 1 - h->cur), drho, du, h->stream));
  else HC_CUDA(h, hcd::launch_moments<float>(lbm_view<float>(h, h->cur, 1 - h->cur), drho, du, h->stream));
  if (rho) HC_CUDA(h, cudaMemcpyAsync(rho, drho, 8 * h->N, cudaMemcpyDeviceToHost, h->stream));
  if (u) HC_CUDA(h, cudaMemcpyAsync(u, du, 8 * 3 * h->N, cudaMemcpyDeviceToHost, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return HC_OK;
}

int hc_read_populations(hc_handle* h, double* f) {
  if (!h || !f) return HC_ERR_INVALID;
  int rc;
  if ((rc = ensure_scratch(h, sizeof(double) * 19 * h->N)) != HC_OK) return rc;
  if (h->f64) HC_CUDA(h, hcd::launch_stream_out<double>(lbm_view<double>(h, h->cur, h->cur), h->scratch, h->stream));
  else HC_CUDA(h, hcd::launch_stream_out<float>(lbm_view<float>(h, h->cur, h->cur), h->scratch, h->stream));
  HC_CUDA(h, cudaMemcpyAsync(f, h->scratch, 8 * 19 * h->N, cudaMemcpyDeviceToHost, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  shrink_scratch(h);
  return HC_OK;
}

int hc_write_populations(hc_handle* h, const double* f) {
  if (!h || !f) return HC_ERR_INVALID;
  int rc;
  if ((rc = ensure_scratch(h, sizeof(double) * 19 * h->N)) != HC_OK) return rc;
  HC_CUDA(h, cudaMemcpyAsync(h->scratch, f, 8 * 19 * h->N, cudaMemcpyHostToDevice, h->stream));
  if (h->f64) HC_CUDA(h, hcd::launch_stream_in<double>(lbm_view<double>(h, 1 - h->cur, h->cur), h->scratch, 1.0, nullptr, h->stream));
  else HC_CUDA(h, hcd::launch_stream_in<float>(lbm_view<float>(h, 1 - h->cur, h->cur), h->scratch, 1.0, nullptr, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  shrink_scratch(h);
  return HC_OK;
}

int hc_read_force_field(hc_handle* h, double* F, int which) {
  if (!h || !F) return HC_ERR_INVALID;
  int rc;
  if ((rc = ensure_scratch(h, sizeof(double) * 3 * h->N)) != HC_OK) return rc;
  const void* src = h->F[which ? 1 - h->cur : h->cur];
  if (h->f64) HC_CUDA(h, hcd::launch_field_out<double>((const double*)src, h->scratch, h->N, h->stream));
  else HC_CUDA(h, hcd::launch_field_out<float>((const float*)src, h->scratch, h->N, h->stream));
  HC_CUDA(h, cudaMemcpyAsync(F, h->scratch, 8 * 3 * h->N, cudaMemcpyDeviceToHost, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return HC_OK;
}

int hc_write_force_field(hc_handle* h, const double* F) {
  if (!h || !F) return HC_ERR_INVALID;
  int rc;
  // the field is overwritten and holds no spread afterwards
  if ((rc = undo_fused_spread(h)) != HC_OK) return rc;
  if ((rc = ensure_scratch(h, sizeof(double) * 3 * h->N)) != HC_OK) return rc;
  HC_CUDA(h, cudaMemcpyAsync(h->scratch, F, 8 * 3 * h->N, cudaMemcpyHostToDevice, h->stream));
  for (int k = 0; k < 2; ++k) {
    if (h->f64) HC_CUDA(h, hcd::launch_field_in<double>(h->scratch, (double*)h->F[k], h->N, h->stream));
    else HC_CUDA(h, hcd::launch_field_in<float>(h->scratch, (float*)h->F[k], h->N, h->stream));
  }
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return HC_OK;
}

int hc_read_vertices(hc_handle* h, double* x, double* v, double* f) {
  if (!h) return HC_ERR_INVALID;
  if (h->nvert == 0) return HC_OK;
  int rc;
  if (x && (rc = read3<double>(h, h->x, x)) != HC_OK) return rc;
  if (h->f64) {
    if (v && (rc = read3<double>(h, h->v, v)) != HC_OK) return rc;
    if (f && (rc = read3<double>(h, h->fv, f)) != HC_OK) return rc;
  } else {
    if (v && (rc = read3<float>(h, h->v, v)) != HC_OK) return rc;
    if (f && (rc = read3<float>(h, h->fv, f)) != HC_OK) return rc;
  }
  return HC_OK;
}

int hc_read_positions_async(hc_handle* h, double* x, int slot) {
  if (!h || !x || slot < 0 || slot > 1) return HC_ERR_INVALID;
  if (h->nvert == 0) return HC_OK;
  if (!h->copy_stream) {
    HC_CUDA(h, cudaStreamCreateWithFlags(&h->copy_stream, cudaStreamNonBlocking));
    for (int k = 0; k < 2; ++k) {
      HC_CUDA(h, cudaEventCreateWithFlags(&h->pos_ready[k], cudaEventDisableTiming));
      HC_CUDA(h, cudaEventCreateWithFlags(&h->pos_copied[k], cudaEventDisableTiming));
    }
  }
  if (h->pos_stage_v < h->nvert) {
    // new staging buffers once the copies out of the old ones are done
    HC_CUDA(h, cudaStreamSynchronize(h->copy_stream));
    for (int k = 0; k < 2; ++k) {
      dfree(h, h->pos_stage[k]);
      h->pos_stage[k] = nullptr;
      if (h->pos_stage_v > 0) h->device_bytes -= 24 * h->pos_stage_v;
    }
    h->pos_stage_v = 0;
    for (int k = 0; k < 2; ++k) HC_CUDA(h, dalloc(h, (void**)&h->pos_stage[k], 24 * (size_t)h->Vcap));
    h->pos_stage_v = h->Vcap;
    h->pos_inflight[0] = h->pos_inflight[1] = false;
  }
  // the staging buffer is rewritten only after its last copy left it
  if (h->pos_inflight[slot]) HC_CUDA(h, cudaStreamWaitEvent(h->stream, h->pos_copied[slot], 0));
  HC_CUDA(h, hcd::launch_soa_to_aos<double>(h->x, h->pos_stage[slot], h->Vcap, h->nvert, h->stream));
  HC_CUDA(h, cudaEventRecord(h->pos_ready[slot], h->stream));
  HC_CUDA(h, cudaStreamWaitEvent(h->copy_stream, h->pos_ready[slot], 0));
  HC_CUDA(h, cudaMemcpyAsync(x, h->pos_stage[slot], 24 * (size_t)h->nvert, cudaMemcpyDeviceToHost, h->copy_stream));
  HC_CUDA(h, cudaEventRecord(h->pos_copied[slot], h->copy_stream));
  h->pos_inflight[slot] = true;
  return HC_OK;
}

int hc_wait_positions(hc_handle* h, int slot) {
  if (!h || slot < 0 || slot > 1) return HC_ERR_INVALID;
  if (!h->pos_inflight[slot]) return HC_OK;
  h->pos_inflight[slot] = false;
  HC_CUDA(h, cudaEventSynchronize(h->pos_copied[slot]));
  return HC_OK;
}

int hc_write_vertices(hc_handle* h, const double* x, const double* v, const double* f) {
  if (!h) return HC_ERR_INVALID;
  if (int rc0 = undo_fused_spread(h)) return rc0;
  if (h->nvert == 0) return HC_OK;
  int rc;
  if (x && (rc = write3(h, h->x, 8, x)) != HC_OK) return rc;
  if (v && (rc = write3(h, h->v, h->ts, v)) != HC_OK) return rc;
  if (f && (rc = write3(h, h->fv, h->ts, f)) != HC_OK) return rc;
  return HC_OK;
}

int hc_read_cells(hc_handle* h, int* alive, double* volume) {
  if (!h) return HC_ERR_INVALID;
  if (h->ncells == 0) return HC_OK;
  std::vector<int> al(h->ncells);
  HC_CUDA(h, cudaMemcpyAsync(al.data(), h->alive, 4 * h->ncells, cudaMemcpyDeviceToHost, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  if (alive) std::memcpy(alive, al.data(), 4 * h->ncells);
  if (volume) {
    std::vector<double> x(3 * (size_t)h->nvert);
    int rc = hc_read_vertices(h, x.data(), nullptr, nullptr);
    if (rc != HC_OK) return rc;
    for (int c = 0; c < h->ncells; ++c) {
      const hcg::TypeConstants& tc = h->types[h->h_cell_type[c]].tc;
      const double* X = x.data() + 3 * (size_t)h->h_cell_voff[c];
      double vol = 0;
      for (int k = 0; k < tc.nf; ++k) {
        double v0[3], v1[3], v2[3];
        for (int a = 0; a < 3; ++a) {
          v0[a] = X[3 * tc.tris[3 * k] + a] - X[a];
          v1[a] = X[3 * tc.tris[3 * k + 1] + a] - X[a];
          v2[a] = X[3 * tc.tris[3 * k + 2] + a] - X[a];
        }
        vol += (-v2[0] * v1[1] * v0[2] + v1[0] * v2[1] * v0[2] + v2[0] * v0[1] * v1[2] - v0[0] * v2[1] * v1[2] -
                v1[0] * v0[1] * v2[2] + v0[0] * v1[1] * v2[2]);
      }
      volume[c] = vol / 6.0;
    }
  }
  return HC_OK;
}

int hc_read_bins(hc_handle* h, int* vertex_node, int* vertex_tile, int* tile_offsets, int* tile_vertices,
                 int* tile_cell_offsets, int* tile_cells, int max_tile_cells) {
  if (!h) return HC_ERR_INVALID;
  int rc = hc_stage(h, HC_STAGE_BIN);
  if (rc != HC_OK) return rc;
  const int nt = h->ntiles;
  std::vector<int> tco(nt + 1);
  HC_CUDA(h, cudaMemcpyAsync(tco.data(), h->tile_cell_offsets, 4 * (nt + 1), cudaMemcpyDeviceToHost, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  if (tco[nt] > max_tile_cells) return fail(h, HC_ERR_INVALID, "tile_cells buffer too small");
  if (vertex_node && h->nvert)
    HC_CUDA(h, cudaMemcpyAsync(vertex_node, h->vnode, 4 * h->nvert, cudaMemcpyDeviceToHost, h->stream));
  if (vertex_tile && h->nvert)
    HC_CUDA(h, cudaMemcpyAsync(vertex_tile, h->vtile, 4 * h->nvert, cudaMemcpyDeviceToHost, h->stream));
  if (tile_offsets) HC_CUDA(h, cudaMemcpyAsync(tile_offsets, h->bin_offsets, 4 * (nt + 1), cudaMemcpyDeviceToHost, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  if (tile_vertices && tile_offsets && tile_offsets[nt] > 0)
    HC_CUDA(h, cudaMemcpyAsync(tile_vertices, h->tile_vertices, 4 * (size_t)tile_offsets[nt], cudaMemcpyDeviceToHost,
                               h->stream));
  if (tile_cell_offsets) std::memcpy(tile_cell_offsets, tco.data(), 4 * (nt + 1));
  if (tile_cells && tco[nt] > 0)
    HC_CUDA(h, cudaMemcpyAsync(tile_cells, h->tile_cells, 4 * (size_t)tco[nt], cudaMemcpyDeviceToHost, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return nt;
}

int hc_read_neighbours(hc_handle* h, int* nb_offsets, int* nb_cells, int max_cells) {
  if (!h || !nb_offsets || max_cells < 0 || (max_cells > 0 && !nb_cells)) return HC_ERR_INVALID;
  int rc = hc_stage(h, HC_STAGE_BIN);
  if (rc != HC_OK) return rc;
  const int nt = h->ntiles;
  const int per[3] = {h->p.periodic[0] ? 1 : 0, h->p.periodic[1] ? 1 : 0, h->p.periodic[2] ? 1 : 0};
  // scratch: counts[nt], offsets[nt + 1], then the cells
  const size_t head = 4 * (2 * (size_t)nt + 1);
  if ((rc = ensure_scratch(h, head)) != HC_OK) return rc;
  int* counts = reinterpret_cast<int*>(h->scratch);
  int* offs = counts + nt;
  HC_CUDA(h, hcd::launch_tile_neighbours(h->tg, per, h->tile_cell_offsets, h->tile_cells, nt, counts, nullptr,
                                         nullptr, h->stream));
  HC_CUDA(h, hcd::launch_exclusive_scan(counts, nt, offs, h->stream));
  HC_CUDA(h, cudaMemcpyAsync(nb_offsets, offs, 4 * ((size_t)nt + 1), cudaMemcpyDeviceToHost, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  const int total = nb_offsets[nt];
  if (total > max_cells) {
    shrink_scratch(h);
    return fail(h, HC_ERR_INVALID, "nb_cells buffer too small");
  }
  if (total > 0) {
    if ((rc = ensure_scratch(h, head + 4 * (size_t)total)) != HC_OK) return rc;
    counts = reinterpret_cast<int*>(h->scratch);
    offs = counts + nt;
    int* cells = offs + nt + 1;
    HC_CUDA(h, cudaMemcpyAsync(offs, nb_offsets, 4 * ((size_t)nt + 1), cudaMemcpyHostToDevice, h->stream));
    HC_CUDA(h, hcd::launch_tile_neighbours(h->tg, per, h->tile_cell_offsets, h->tile_cells, nt, counts, offs, cells,
                                           h->stream));
    HC_CUDA(h, cudaMemcpyAsync(nb_cells, cells, 4 * (size_t)total, cudaMemcpyDeviceToHost, h->stream));
    HC_CUDA(h, cudaStreamSynchronize(h->stream));
  }
  shrink_scratch(h);
  return nt;
}

long long hc_estimate_device_bytes(const hc_params* p, int nvertices, int ncells) {
  if (!p || p->nx <= 0 || p->ny <= 0 || p->nz <= 0 || nvertices < 0 || ncells < 0) return HC_ERR_INVALID;
  const long long N = (long long)p->nx * p->ny * p->nz;
  const bool f64 = p->form == HC_FORM_PLAIN_F64;
  const long long ts = f64 ? 8 : 4;
  const long long fb = 19 * ts * N;
  const long long Fb = (long long)(f64 ? hcd::field_bytes<double>(N) : hcd::field_bytes<float>(N));
  // lattice arrays, as hc_create allocates them
  long long b = 2 * fb + 2 * Fb + 4 * N + Fb + 4 + 4 * N + 2 * N + 3 * ts * p->nz +
                (long long)sizeof(TypeDev) * hcd::MAX_TYPES + 4;
  b += 4 * N;  // the fluid-node list (at most every node)
  // vertex and cell arrays at the capacity growth can reach (twice the need)
  const long long vcap = std::max<long long>(2LL * nvertices, 1024);
  const long long ccap = std::max<long long>(2LL * ncells, 64);
  b += vcap * (3 * 8 + 6 * ts + 3 * 4) + ccap * 4 * 4;
  // per-type rest-state blobs (hc_add_cell_type) and cell lists.  A closed mesh
  // has 2 faces and 3 edges a vertex, at most one inner link for two vertices:
  // 69 ints, 9.5 doubles, and 17 doubles or 21.5 floats more; 16-byte alignment
  // of the tables within a blob
  b += (f64 ? 488LL : 438LL) * nvertices + 128LL * hcd::MAX_TYPES + 4LL * ncells;
  // tile lists (hc_read_bins) and readback staging (hc_read_fluid, hc_read_vertices)
  const int tx = p->tile[0] > 0 ? p->tile[0] : 8, ty = p->tile[1] > 0 ? p->tile[1] : 8,
            tz = p->tile[2] > 0 ? p->tile[2] : 8;
  const long long ntiles =
      (long long)((p->nx + tx - 1) / tx) * ((p->ny + ty - 1) / ty) * ((p->nz + tz - 1) / tz);
  b += 5 * 4 * (ntiles + 1) + 2 * 4 * vcap;
  b += std::max<long long>(4 * 8 * N, 3 * 8 * vcap);
  return b;
}

int hc_get_stats(hc_handle* h, hc_stats* out) {
  if (!h || !out) return HC_ERR_INVALID;
  out->nodes = h->N;
  out->vertices = h->nvert;
  out->cells = h->ncells;
  out->types = (int)h->types.size();
  out->iter = h->iter;
  out->tau = h->u.tau;
  out->omega = 1.0 / h->u.tau;
  out->device_bytes = h->device_bytes;
  int alive = 0;
  if (h->ncells) {
    std::vector<int> al(h->ncells);
    HC_CUDA(h, cudaMemcpyAsync(al.data(), h->alive, 4 * h->ncells, cudaMemcpyDeviceToHost, h->stream));
    HC_CUDA(h, cudaStreamSynchronize(h->stream));
    for (int a : al) alive += a != 0;
  }
  out->cells_alive = alive;
  return HC_OK;
}

int hc_vertex_count(const hc_handle* h) { return h ? h->nvert : HC_ERR_INVALID; }

int hc_device_status(hc_handle* h, unsigned int* status) {
  if (!h || !status) return HC_ERR_INVALID;
  HC_CUDA(h, cudaMemcpyAsync(status, h->status, sizeof(unsigned int), cudaMemcpyDeviceToHost, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  return HC_OK;
}

int hc_autotune(hc_handle* h, const char* cache_path) {
  if (!h) return HC_ERR_INVALID;
  return h->f64 ? autotune<double>(h, cache_path) : autotune<float>(h, cache_path);
}

int hc_get_tuning(hc_handle* h, int* out8) {
  if (!h || !out8) return HC_ERR_INVALID;
  std::memcpy(out8, h->tune, sizeof(h->tune));
  return HC_OK;
}

int hc_set_tuning(hc_handle* h, const int* in8) {
  if (!h || !in8) return HC_ERR_INVALID;
  // width 0 (whole rows), a multiple of 32, or 8 / 16 (warps as 8 x 4 or 16 x 2
  // tiles); whole warps, at most 256 threads
  const bool width_ok = in8[0] == 0 || in8[0] % 32 == 0 || in8[0] == 8 || in8[0] == 16;
  if (in8[0] < 0 || in8[1] <= 0 || in8[0] * in8[1] > 256 || !width_ok || (in8[0] > 0 && in8[0] * in8[1] % 32 != 0))
    return fail(h, HC_ERR_INVALID,
                "collide-stream block must be 0 (whole rows), 8, 16 or a multiple of 32 wide, whole warps, "
                "at most 256 threads");
  for (int k = 2; k <= 3; ++k)
    if (in8[k] <= 0 || in8[k] > 512 || in8[k] % 32 != 0) return fail(h, HC_ERR_INVALID, "bad block size");
  if (in8[4] <= 0 || in8[4] > (h->f64 ? 384 : 768) || in8[4] % 32 != 0)
    return fail(h, HC_ERR_INVALID, "bad mechanics block size");
  if (in8[6] < 0 || in8[6] > 2)
    return fail(h, HC_ERR_INVALID, "mechanics variant is 0 (gather), 1 (scatter) or 2 (staged gather)");
  {
    const int mode = in8[7] & 0xff;
    if ((in8[7] & ~0x3fff) != 0) return fail(h, HC_ERR_INVALID, "tune[7]: only bits 0-13 are defined");
    if ((in8[7] & 0x300) == 0x300 && 19LL * h->N >= (1LL << 31))
      return fail(h, HC_ERR_INVALID, "tune[7]: the dense node velocity needs 19 N < 2^31");
    if ((in8[7] & 0x200) && 19LL * h->N >= (1LL << 31))
      return fail(h, HC_ERR_INVALID, "packed node velocity needs 19 N < 2^31");
    if ((mode == 1 || (in8[7] & 0x300) == 0x100) && h->nfluid == 0)
      return fail(h, HC_ERR_INVALID, "no fluid-node list for this lattice");
    if (mode >= 2) {
      const int st = mode & 15, ctas = mode >> 4;
      if (st < 2 || st > 8 || ctas < 1 || ctas > 4)
        return fail(h, HC_ERR_INVALID, "bulk collide-stream code is stages (2-8) | CTAs per SM (1-4) << 4");
      const bool ok = h->f64 ? set_bulk_plan<double>(h, mode) : set_bulk_plan<float>(h, mode);
      if (!ok) return fail(h, HC_ERR_INVALID, "the lattice does not allow the bulk collide-stream (row bytes, rows, shared memory)");
    }
  }
  int old_tune[8];
  std::memcpy(old_tune, h->tune, sizeof(old_tune));
  if (std::memcmp(old_tune, in8, sizeof(old_tune)) == 0) return HC_OK;  // the rules', or the caller's already
  std::memcpy(h->tune, in8, sizeof(h->tune));
  h->tuned = true;
  invalidate_graph(h);
  return retag_if_needed(h, old_tune);
}

// ---- cell information and CSV output --------------------------------------
int hc_cell_info(hc_handle* h, double* out) {
  if (!h || !out) return HC_ERR_INVALID;
  const int C = h->ncells;
  if (C == 0) return HC_OK;
  int rc;
  if ((rc = ensure_scratch(h, sizeof(double) * 16 * (size_t)C)) != HC_OK) return rc;
  if (h->f64)
    HC_CUDA(h, hcd::launch_cell_info<double>(vertex_view<double>(h), h->cell_type, h->cell_voff, h->dtypes, C,
                                             h->scratch, h->stream));
  else
    HC_CUDA(h, hcd::launch_cell_info<float>(vertex_view<float>(h), h->cell_type, h->cell_voff, h->dtypes, C,
                                            h->scratch, h->stream));
  HC_CUDA(h, cudaMemcpyAsync(out, h->scratch, sizeof(double) * 16 * (size_t)C, cudaMemcpyDeviceToHost, h->stream));
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  // centroids are reported inside the lattice on periodic axes
  const int n[3] = {h->nx, h->ny, h->nz};
  for (int c = 0; c < C; ++c)
    for (int a = 0; a < 3; ++a)
      if (h->p.periodic[a]) out[16 * c + a] -= n[a] * std::floor(out[16 * c + a] / n[a]);
  return HC_OK;
}

int hc_write_cell_info_csv(hc_handle* h, const char* dir, int si) {
  if (!h || !dir) return HC_ERR_INVALID;
  std::vector<double> info(16 * (size_t)h->ncells);
  int rc;
  if ((rc = hc_cell_info(h, info.data())) != HC_OK) return rc;
  std::error_code ec;
  std::filesystem::create_directories(dir, ec);
  if (ec) return fail(h, HC_ERR_INVALID, "cannot create " + std::string(dir) + ": " + ec.message());
  char iter[32];
  std::snprintf(iter, sizeof iter, "%012d", h->iter);
  const double dx = h->p.dx, dt = h->p.dt;
  for (size_t ty = 0; ty < h->types.size(); ++ty) {
    const std::string path = std::string(dir) + "/" + h->types[ty].name + "." + iter + ".csv";
    std::ofstream out(path, std::ios::trunc);
    if (!out) return fail(h, HC_ERR_INVALID, "cannot write " + path);
    out << "X,Y,Z,area,volume,atomic_block,cellId,baseCellId,velocity_x,velocity_y,velocity_z\n";
    out.precision(17);
    for (int c = 0; c < h->ncells; ++c) {
      const double* r = info.data() + 16 * (size_t)c;
      if ((int)r[15] != (int)ty) continue;  // other type, or deleted
      const double lp = si ? dx : 1.0, la = si ? dx * dx : 1.0, lv = si ? dx * dx * dx : 1.0,
                   lu = si ? dx / dt : 1.0;
      out << r[0] * lp << "," << r[1] * lp << "," << r[2] * lp << "," << r[6] * la << "," << r[7] * lv << ",0,"
          << c << "," << c << "," << r[3] * lu << "," << r[4] * lu << "," << r[5] * lu << "\n";
    }
  }
  return HC_OK;
}

// ---- field output (content of io/FluidHdf5IO.hh and io/ParticleHdf5IO.cpp) ----
namespace {

bool write_raw(const std::string& path, const void* data, size_t bytes) {
  std::ofstream out(path, std::ios::binary | std::ios::trunc);
  out.write((const char*)data, (std::streamsize)bytes);
  return (bool)out;
}

std::string xdmf_item(const std::string& file, const std::string& dims, const char* type, int precision) {
  return "<DataItem Format=\"Binary\" Endian=\"Little\" NumberType=\"" + std::string(type) + "\" Precision=\"" +
         std::to_string(precision) + "\" Dimensions=\"" + dims + "\">" + file + "</DataItem>";
}

}  // namespace

int hc_write_output(hc_handle* h, const char* dir, int si) {
  if (!h || !dir) return HC_ERR_INVALID;
  std::error_code ec;
  std::filesystem::create_directories(std::string(dir) + "/hdf5", ec);
  if (ec) return fail(h, HC_ERR_INVALID, "cannot create " + std::string(dir) + ": " + ec.message());
  const std::string d = std::string(dir) + "/hdf5/";
  char it[32];
  std::snprintf(it, sizeof it, "%012d", h->iter);
  const double dx = h->p.dx, dt = h->p.dt;
  const double su = si ? dx / dt : 1.0, sr = si ? h->p.rho_p : 1.0, sf = si ? h->u.df : 1.0, sl = si ? dx : 1.0;
  int rc;
  // fluid: Velocity, Density, Force on the nodes (x fastest)
  {
    const long long N = h->N;
    std::vector<double> rho(N), u(3 * N), F(3 * N);
    if ((rc = hc_read_fluid(h, rho.data(), u.data())) != HC_OK) return rc;
    if ((rc = hc_read_force_field(h, F.data(), 1)) != HC_OK) return rc;
    std::vector<float> vel(3 * N), den(N), frc(3 * N);
    for (long long n = 0; n < N; ++n) {
      den[n] = (float)(rho[n] * sr);
      for (int a = 0; a < 3; ++a) {
        vel[3 * n + a] = (float)(u[a * N + n] * su);
        frc[3 * n + a] = (float)(F[a * N + n] * sf);
      }
    }
    const std::string base = std::string("Fluid.") + it;
    if (!write_raw(d + base + ".Velocity.bin", vel.data(), 4 * vel.size()) ||
        !write_raw(d + base + ".Density.bin", den.data(), 4 * den.size()) ||
        !write_raw(d + base + ".Force.bin", frc.data(), 4 * frc.size()))
      return fail(h, HC_ERR_INVALID, "cannot write the fluid fields to " + d);
    const std::string dims = std::to_string(h->nz) + " " + std::to_string(h->ny) + " " + std::to_string(h->nx);
    std::ofstream x(d + base + ".xmf", std::ios::trunc);
    x << "<?xml version=\"1.0\" ?>\n<Xdmf Version=\"2.0\">\n <Domain>\n  <Grid Name=\"Fluid\" GridType=\"Uniform\">\n"
      << "   <Time Value=\"" << h->iter * (si ? dt : 1.0) << "\"/>\n"
      << "   <Topology TopologyType=\"3DCoRectMesh\" Dimensions=\"" << dims << "\"/>\n"
      << "   <Geometry GeometryType=\"ORIGIN_DXDYDZ\">\n    <DataItem Format=\"XML\" Dimensions=\"3\">0 0 0</DataItem>\n"
      << "    <DataItem Format=\"XML\" Dimensions=\"3\">" << sl << " " << sl << " " << sl << "</DataItem>\n   </Geometry>\n"
      << "   <Attribute Name=\"Velocity\" AttributeType=\"Vector\" Center=\"Node\">"
      << xdmf_item(base + ".Velocity.bin", dims + " 3", "Float", 4) << "</Attribute>\n"
      << "   <Attribute Name=\"Density\" AttributeType=\"Scalar\" Center=\"Node\">"
      << xdmf_item(base + ".Density.bin", dims, "Float", 4) << "</Attribute>\n"
      << "   <Attribute Name=\"Force\" AttributeType=\"Vector\" Center=\"Node\">"
      << xdmf_item(base + ".Force.bin", dims + " 3", "Float", 4) << "</Attribute>\n"
      << "  </Grid>\n </Domain>\n</Xdmf>\n";
    if (!x) return fail(h, HC_ERR_INVALID, "cannot write " + d + base + ".xmf");
  }
  // particles per cell type: Position (geometry), Triangles (topology),
  // Velocity, Total force (membrane + repulsion), Cell Id, of the live cells
  const int V = h->nvert;
  std::vector<double> x(3 * (size_t)V), v(3 * (size_t)V), f(3 * (size_t)V), rep(3 * (size_t)V, 0.0);
  std::vector<int> alive(h->ncells);
  if (V > 0) {
    if ((rc = hc_read_vertices(h, x.data(), v.data(), f.data())) != HC_OK) return rc;
    if ((h->rep_every > 0 || h->brep_every > 0) && (rc = hc_read_repulsion(h, rep.data())) != HC_OK) return rc;
  }
  if (h->ncells > 0) {
    HC_CUDA(h, cudaMemcpyAsync(alive.data(), h->alive, 4 * (size_t)h->ncells, cudaMemcpyDeviceToHost, h->stream));
    HC_CUDA(h, cudaStreamSynchronize(h->stream));
  }
  for (size_t ty = 0; ty < h->types.size(); ++ty) {
    const hcg::TypeConstants& tc = h->types[ty].tc;
    std::vector<float> pos, vel, frc;
    std::vector<int> tri, cid;
    int nv_out = 0;
    for (int c = 0; c < h->ncells; ++c) {
      if (h->h_cell_type[c] != (int)ty || !alive[c]) continue;
      const int off = h->h_cell_voff[c];
      for (int k = 0; k < tc.nf; ++k)
        for (int q = 0; q < 3; ++q) tri.push_back(nv_out + tc.tris[3 * k + q]);
      for (int k = 0; k < tc.nv; ++k) {
        const size_t i = 3 * (size_t)(off + k);
        for (int a = 0; a < 3; ++a) {
          pos.push_back((float)(x[i + a] * sl));
          vel.push_back((float)(v[i + a] * su));
          frc.push_back((float)((f[i + a] + rep[i + a]) * sf));
        }
        cid.push_back(c);
      }
      nv_out += tc.nv;
    }
    const std::string base = h->types[ty].name + "." + it;
    if (!write_raw(d + base + ".Position.bin", pos.data(), 4 * pos.size()) ||
        !write_raw(d + base + ".Triangles.bin", tri.data(), 4 * tri.size()) ||
        !write_raw(d + base + ".Velocity.bin", vel.data(), 4 * vel.size()) ||
        !write_raw(d + base + ".TotalForce.bin", frc.data(), 4 * frc.size()) ||
        !write_raw(d + base + ".CellId.bin", cid.data(), 4 * cid.size()))
      return fail(h, HC_ERR_INVALID, "cannot write the particle fields to " + d);
    const std::string nvs = std::to_string(nv_out), nfs = std::to_string(tri.size() / 3);
    std::ofstream xf(d + base + ".xmf", std::ios::trunc);
    xf << "<?xml version=\"1.0\" ?>\n<Xdmf Version=\"2.0\">\n <Domain>\n  <Grid Name=\"" << h->types[ty].name
       << "\" GridType=\"Uniform\">\n   <Time Value=\"" << h->iter * (si ? dt : 1.0) << "\"/>\n"
       << "   <Topology TopologyType=\"Triangle\" NumberOfElements=\"" << nfs << "\">"
       << xdmf_item(base + ".Triangles.bin", nfs + " 3", "Int", 4) << "</Topology>\n"
       << "   <Geometry GeometryType=\"XYZ\">" << xdmf_item(base + ".Position.bin", nvs + " 3", "Float", 4)
       << "</Geometry>\n"
       << "   <Attribute Name=\"Velocity\" AttributeType=\"Vector\" Center=\"Node\">"
       << xdmf_item(base + ".Velocity.bin", nvs + " 3", "Float", 4) << "</Attribute>\n"
       << "   <Attribute Name=\"Total force\" AttributeType=\"Vector\" Center=\"Node\">"
       << xdmf_item(base + ".TotalForce.bin", nvs + " 3", "Float", 4) << "</Attribute>\n"
       << "   <Attribute Name=\"Cell Id\" AttributeType=\"Scalar\" Center=\"Node\">"
       << xdmf_item(base + ".CellId.bin", nvs, "Int", 4) << "</Attribute>\n"
       << "  </Grid>\n </Domain>\n</Xdmf>\n";
    if (!xf) return fail(h, HC_ERR_INVALID, "cannot write " + d + base + ".xmf");
  }
  return HC_OK;
}

// ---- checkpoints ------------------------------------------------------------
namespace {

struct LatticeHeader {
  char magic[8];
  int32_t version, nx, ny, nz, ts, cur, iter, body_mode;
  double body[3];
  double uw[hcd::MAX_WALL_CLASSES][3];
};

struct ParticleHeader {
  char magic[8];
  int32_t version, ts, ntypes, ncells, nvert, has_frep_cell, has_frep_wall;
  int32_t nv[hcd::MAX_TYPES];
};

const char kLatMagic[8] = {'H', 'C', 'G', 'B', 'L', 'A', 'T', '1'};
const char kParMagic[8] = {'H', 'C', 'G', 'B', 'P', 'A', 'R', '1'};

int put_device(hc_handle* h, std::ofstream& out, const void* d, size_t bytes) {
  std::vector<char> buf(std::min<size_t>(bytes, (size_t)64 << 20));
  for (size_t off = 0; off < bytes; off += buf.size()) {
    const size_t n = std::min(buf.size(), bytes - off);
    HC_CUDA(h, cudaMemcpyAsync(buf.data(), (const char*)d + off, n, cudaMemcpyDeviceToHost, h->stream));
    HC_CUDA(h, cudaStreamSynchronize(h->stream));
    out.write(buf.data(), (std::streamsize)n);
  }
  return out ? HC_OK : fail(h, HC_ERR_INVALID, "checkpoint write failed");
}

int get_device(hc_handle* h, std::ifstream& in, void* d, size_t bytes) {
  std::vector<char> buf(std::min<size_t>(bytes, (size_t)64 << 20));
  for (size_t off = 0; off < bytes; off += buf.size()) {
    const size_t n = std::min(buf.size(), bytes - off);
    in.read(buf.data(), (std::streamsize)n);
    if (!in) return fail(h, HC_ERR_INVALID, "checkpoint file is truncated");
    HC_CUDA(h, cudaMemcpyAsync((char*)d + off, buf.data(), n, cudaMemcpyHostToDevice, h->stream));
    HC_CUDA(h, cudaStreamSynchronize(h->stream));
  }
  return HC_OK;
}

// [3][Vcap] device array: the first nvert entries of each component
int put_soa(hc_handle* h, std::ofstream& out, const void* d, size_t es) {
  int rc;
  for (int a = 0; a < 3; ++a)
    if ((rc = put_device(h, out, (const char*)d + a * es * h->Vcap, es * h->nvert)) != HC_OK) return rc;
  return HC_OK;
}
int get_soa(hc_handle* h, std::ifstream& in, void* d, size_t es) {
  int rc;
  for (int a = 0; a < 3; ++a)
    if ((rc = get_device(h, in, (char*)d + a * es * h->Vcap, es * h->nvert)) != HC_OK) return rc;
  return HC_OK;
}

}  // namespace

int hc_save_checkpoint(hc_handle* h, const char* dir) {
  if (!h || !dir) return HC_ERR_INVALID;
  int rc;
  // a canonical state: the next step's force field holds the body force only
  if ((rc = undo_fused_spread(h)) != HC_OK) return rc;
  namespace fs = std::filesystem;
  std::error_code ec;
  fs::create_directories(dir, ec);
  if (ec) return fail(h, HC_ERR_INVALID, "cannot create " + std::string(dir) + ": " + ec.message());
  const std::string d = std::string(dir) + "/";
  for (const char* f : {"lattice.dat", "particleField.dat", "checkpoint.xml"})
    if (fs::exists(d + f)) fs::rename(d + f, d + f + ".old", ec);
  {
    std::ofstream out(d + "lattice.dat", std::ios::binary | std::ios::trunc);
    if (!out) return fail(h, HC_ERR_INVALID, "cannot write " + d + "lattice.dat");
    LatticeHeader hd;
    std::memset(&hd, 0, sizeof hd);
    std::memcpy(hd.magic, kLatMagic, 8);
    hd.version = 1;
    hd.nx = h->nx;
    hd.ny = h->ny;
    hd.nz = h->nz;
    hd.ts = h->ts;
    hd.cur = h->cur;
    hd.iter = h->iter;
    hd.body_mode = h->body_mode;
    for (int a = 0; a < 3; ++a) hd.body[a] = h->body[a];
    std::memcpy(hd.uw, h->uw, sizeof hd.uw);
    out.write((const char*)&hd, sizeof hd);
    out.write((const char*)h->hflag.data(), h->N);
    if ((rc = put_device(h, out, h->f[h->cur], 19 * h->ts * (size_t)h->N)) != HC_OK) return rc;
    const size_t Fb = h->f64 ? hcd::field_bytes<double>(h->N) : hcd::field_bytes<float>(h->N);
    for (int k = 0; k < 2; ++k)
      if ((rc = put_device(h, out, h->F[k], Fb)) != HC_OK) return rc;
  }
  {
    std::ofstream out(d + "particleField.dat", std::ios::binary | std::ios::trunc);
    if (!out) return fail(h, HC_ERR_INVALID, "cannot write " + d + "particleField.dat");
    ParticleHeader hd;
    std::memset(&hd, 0, sizeof hd);
    std::memcpy(hd.magic, kParMagic, 8);
    hd.version = 1;
    hd.ts = h->ts;
    hd.ntypes = (int)h->types.size();
    hd.ncells = h->ncells;
    hd.nvert = h->nvert;
    hd.has_frep_cell = h->rep_every > 0 && h->frep_cell ? 1 : 0;
    hd.has_frep_wall = h->brep_every > 0 && h->frep_wall ? 1 : 0;
    for (size_t t = 0; t < h->types.size(); ++t) hd.nv[t] = h->types[t].tc.nv;
    out.write((const char*)&hd, sizeof hd);
    out.write((const char*)h->h_cell_type.data(), 4 * (size_t)h->ncells);
    out.write((const char*)h->h_cell_voff.data(), 4 * (size_t)h->ncells);
    if (h->ncells > 0 && (rc = put_device(h, out, h->alive, 4 * (size_t)h->ncells)) != HC_OK) return rc;
    if (h->nvert > 0) {
      if ((rc = put_soa(h, out, h->x, 8)) != HC_OK) return rc;
      if ((rc = put_soa(h, out, h->v, h->ts)) != HC_OK) return rc;
      if ((rc = put_soa(h, out, h->fv, h->ts)) != HC_OK) return rc;
      if (hd.has_frep_cell && (rc = put_soa(h, out, h->frep_cell, h->ts)) != HC_OK) return rc;
      if (hd.has_frep_wall && (rc = put_soa(h, out, h->frep_wall, h->ts)) != HC_OK) return rc;
    }
  }
  std::ofstream xml(d + "checkpoint.xml", std::ios::trunc);
  xml << "<?xml version=\"1.0\" ?>\n<Checkpoint>\n  <General>\n    <Iteration> " << h->iter
      << " </Iteration>\n    <OutDirectory> " << dir << " </OutDirectory>\n  </General>\n  <Lattice> "
      << h->nx << " " << h->ny << " " << h->nz << " </Lattice>\n  <Form> " << (h->f64 ? "plain_f64" : "mixed_f32")
      << " </Form>\n  <Cells> " << h->ncells << " </Cells>\n</Checkpoint>\n";
  return xml ? HC_OK : fail(h, HC_ERR_INVALID, "cannot write checkpoint.xml");
}

int hc_load_checkpoint(hc_handle* h, const char* dir) {
  if (!h || !dir) return HC_ERR_INVALID;
  int rc;
  const std::string d = std::string(dir) + "/";
  std::ifstream lin(d + "lattice.dat", std::ios::binary);
  std::ifstream pin(d + "particleField.dat", std::ios::binary);
  if (!lin || !pin) return fail(h, HC_ERR_INVALID, "no checkpoint in " + std::string(dir));
  LatticeHeader lh;
  lin.read((char*)&lh, sizeof lh);
  if (!lin || std::memcmp(lh.magic, kLatMagic, 8) != 0 || lh.version != 1)
    return fail(h, HC_ERR_INVALID, "lattice.dat is not a checkpoint of this library");
  if (lh.nx != h->nx || lh.ny != h->ny || lh.nz != h->nz || lh.ts != h->ts)
    return fail(h, HC_ERR_INVALID, "checkpoint lattice size or precision form differs from this handle's");
  ParticleHeader ph;
  pin.read((char*)&ph, sizeof ph);
  if (!pin || std::memcmp(ph.magic, kParMagic, 8) != 0 || ph.version != 1 || ph.ts != h->ts)
    return fail(h, HC_ERR_INVALID, "particleField.dat is not a checkpoint of this library");
  if (ph.ntypes != (int)h->types.size()) return fail(h, HC_ERR_INVALID, "checkpoint cell types differ from this handle's");
  for (int t = 0; t < ph.ntypes; ++t)
    if (ph.nv[t] != h->types[t].tc.nv) return fail(h, HC_ERR_INVALID, "checkpoint cell type meshes differ");
  std::vector<int> ctype(ph.ncells), cvoff(ph.ncells), alive(ph.ncells);
  pin.read((char*)ctype.data(), 4 * (size_t)ph.ncells);
  pin.read((char*)cvoff.data(), 4 * (size_t)ph.ncells);
  pin.read((char*)alive.data(), 4 * (size_t)ph.ncells);
  if (!pin) return fail(h, HC_ERR_INVALID, "particleField.dat is truncated");
  if (h->ncells != 0 && (h->ncells != ph.ncells || h->h_cell_type != ctype))
    return fail(h, HC_ERR_INVALID, "this handle holds other cells than the checkpoint");
  if ((rc = undo_fused_spread(h)) != HC_OK) return rc;
  invalidate_graph(h);
  // lattice: flags, wall velocities, body force, populations and force fields
  lin.read((char*)h->hflag.data(), h->N);
  if (!lin) return fail(h, HC_ERR_INVALID, "lattice.dat is truncated");
  if ((rc = upload_flags(h)) != HC_OK) return rc;
  std::memcpy(h->uw, lh.uw, sizeof h->uw);
  h->body_mode = lh.body_mode;
  for (int a = 0; a < 3; ++a) h->body[a] = lh.body[a];
  if ((rc = upload_body(h)) != HC_OK) return rc;
  h->cur = lh.cur;
  h->iter = lh.iter;
  if ((rc = get_device(h, lin, h->f[h->cur], 19 * h->ts * (size_t)h->N)) != HC_OK) return rc;
  const size_t Fb = h->f64 ? hcd::field_bytes<double>(h->N) : hcd::field_bytes<float>(h->N);
  for (int k = 0; k < 2; ++k)
    if ((rc = get_device(h, lin, h->F[k], Fb)) != HC_OK) return rc;
  // cells: a handle without cells receives them in the checkpoint's order
  if (h->ncells == 0 && ph.ncells > 0) {
    std::vector<double> xs((size_t)3 * ph.nvert);
    for (int a = 0; a < 3; ++a) {
      std::vector<double> comp(ph.nvert);
      pin.read((char*)comp.data(), 8 * (size_t)ph.nvert);
      for (int i = 0; i < ph.nvert; ++i) xs[3 * (size_t)i + a] = comp[i];
    }
    if (!pin) return fail(h, HC_ERR_INVALID, "particleField.dat is truncated");
    int c = 0;
    while (c < ph.ncells) {
      int e = c;
      while (e < ph.ncells && ctype[e] == ctype[c]) ++e;
      const int nv = h->types[ctype[c]].tc.nv;
      std::vector<double> part(xs.begin() + 3 * (size_t)cvoff[c], xs.begin() + 3 * ((size_t)cvoff[c] + (size_t)(e - c) * nv));
      if ((rc = add_cells_positions(h, ctype[c], e - c, part)) != HC_OK) return rc;
      c = e;
    }
    if (h->h_cell_voff != cvoff) return fail(h, HC_ERR_INVALID, "checkpoint cell layout could not be rebuilt");
    pin.seekg((std::streamoff)(sizeof ph + 12 * (size_t)ph.ncells));
  }
  if (ph.nvert != h->nvert) return fail(h, HC_ERR_INVALID, "checkpoint vertex count differs");
  if (h->ncells > 0) HC_CUDA(h, cudaMemcpyAsync(h->alive, alive.data(), 4 * (size_t)h->ncells, cudaMemcpyHostToDevice, h->stream));
  if (h->nvert > 0) {
    if ((rc = get_soa(h, pin, h->x, 8)) != HC_OK) return rc;
    if ((rc = get_soa(h, pin, h->v, h->ts)) != HC_OK) return rc;
    if ((rc = get_soa(h, pin, h->fv, h->ts)) != HC_OK) return rc;
    if (ph.has_frep_cell) {
      if (!(h->rep_every > 0 && h->frep_cell))
        return fail(h, HC_ERR_INVALID, "the checkpoint holds repulsion forces: enable repulsion before loading it");
      if ((rc = get_soa(h, pin, h->frep_cell, h->ts)) != HC_OK) return rc;
    }
    if (ph.has_frep_wall) {
      if (!(h->brep_every > 0 && h->frep_wall))
        return fail(h, HC_ERR_INVALID, "the checkpoint holds wall repulsion forces: enable it before loading");
      if ((rc = get_soa(h, pin, h->frep_wall, h->ts)) != HC_OK) return rc;
    }
  }
  HC_CUDA(h, cudaStreamSynchronize(h->stream));
  h->spread_done = false;
  return HC_OK;
}

// ---- geometry ---------------------------------------------------------------
int hc_stl_voxelize(const char* path, int ref_dir, double ref_length, int margin, int open_ends, int* dims3,
                    uint8_t* flags, long long max_nodes) {
  if (!path || !dims3) return HC_ERR_INVALID;
  std::vector<std::array<hcg::Vec3, 3>> tris;
  std::string err = hcg::read_stl(path, tris);
  std::vector<uint8_t> fl;
  if (err.empty()) err = hcg::voxelize(tris, ref_dir, ref_length, margin, open_ends != 0, dims3, fl);
  if (!err.empty()) {
    hcd::set_handleless_error("hc_stl_voxelize: " + err);
    return HC_ERR_INVALID;
  }
  if (!flags) return HC_OK;
  if ((long long)fl.size() > max_nodes) {
    hcd::set_handleless_error("hc_stl_voxelize: flags buffer holds fewer nodes than the lattice");
    return HC_ERR_INVALID;
  }
  std::memcpy(flags, fl.data(), fl.size());
  return HC_OK;
}

// ---- mesh helpers ---------------------------------------------------------
static int copy_mesh(const hcg::Mesh& m, double* xyz, int max_nv, int* tris, int max_nf, int* nv, int* nf) {
  if (nv) *nv = (int)m.v.size();
  if (nf) *nf = (int)m.t.size();
  if ((int)m.v.size() > max_nv || (int)m.t.size() > max_nf) return HC_ERR_INVALID;
  for (size_t i = 0; i < m.v.size(); ++i) {
    xyz[3 * i] = m.v[i].x;
    xyz[3 * i + 1] = m.v[i].y;
    xyz[3 * i + 2] = m.v[i].z;
  }
  for (size_t k = 0; k < m.t.size(); ++k)
    for (int c = 0; c < 3; ++c) tris[3 * k + c] = m.t[k][c];
  return HC_OK;
}

int hc_mesh_icosphere(int min_triangles, double radius, double* xyz, int max_nv, int* tris, int max_nf, int* nv,
                      int* nf) {
  if (min_triangles < 8 || min_triangles > 400000 || !(radius > 0)) return HC_ERR_INVALID;
  return copy_mesh(hcg::icosphere(min_triangles, radius), xyz, max_nv, tris, max_nf, nv, nf);
}
int hc_mesh_rbc(int min_triangles, double radius, double* xyz, int max_nv, int* tris, int max_nf, int* nv, int* nf) {
  if (min_triangles < 8 || min_triangles > 400000 || !(radius > 0)) return HC_ERR_INVALID;
  return copy_mesh(hcg::rbc_from_sphere(min_triangles, radius), xyz, max_nv, tris, max_nf, nv, nf);
}
int hc_mesh_ellipsoid(int min_triangles, double radius, double aspect, double* xyz, int max_nv, int* tris, int max_nf,
                      int* nv, int* nf) {
  if (min_triangles < 8 || min_triangles > 400000 || !(radius > 0) || !(aspect > 0)) return HC_ERR_INVALID;
  return copy_mesh(hcg::ellipsoid_from_sphere(min_triangles, radius, aspect), xyz, max_nv, tris, max_nf, nv, nf);
}
int hc_mesh_antipodal_pairs(const double* xyz, int nv, int* pairs, int max_pairs) {
  if (!xyz || nv <= 0) return HC_ERR_INVALID;
  std::vector<hcg::Vec3> v(nv);
  for (int i = 0; i < nv; ++i) v[i] = {xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]};
  auto pr = hcg::antipodal_pairs(v);
  if ((int)pr.size() > max_pairs) return HC_ERR_INVALID;
  for (size_t k = 0; k < pr.size(); ++k) {
    pairs[2 * k] = pr[k][0];
    pairs[2 * k + 1] = pr[k][1];
  }
  return (int)pr.size();
}

int hc_place_cells(const double* txyz, int nv, int n, const double* centres, const double* angles, double* out) {
  if (!txyz || nv <= 0 || n < 0 || (n > 0 && (!centres || !angles || !out))) return HC_ERR_INVALID;
  std::vector<hcg::Vec3> rest(nv);
  for (int i = 0; i < nv; ++i) rest[i] = {txyz[3 * i], txyz[3 * i + 1], txyz[3 * i + 2]};
  std::vector<double> xyz;
  xyz.reserve(3 * (size_t)n * nv);
  for (int c = 0; c < n; ++c) hcg::place_cell(rest, centres + 3 * c, angles + 3 * c, xyz);
  std::memcpy(out, xyz.data(), sizeof(double) * xyz.size());
  return HC_OK;
}

int hc_pack_cells(int nx, int ny, int nz, const int* periodic, const uint8_t* solid, int ntypes,
                  const double* const* type_xyz, const int* type_nv, const int* const* type_tris, const int* type_nf,
                  const int* counts, double margin, unsigned long long seed, int max_attempts, double* centres,
                  double* angles, int* types) {
  if (nx <= 0 || ny <= 0 || nz <= 0 || !periodic || ntypes <= 0 || !type_xyz || !type_nv || !type_tris ||
      !type_nf || !counts || !centres || !angles || !types)
    return HC_ERR_INVALID;
  std::vector<hcg::Mesh> shapes(ntypes);
  for (int t = 0; t < ntypes; ++t) {
    for (int i = 0; i < type_nv[t]; ++i)
      shapes[t].v.push_back({type_xyz[t][3 * i], type_xyz[t][3 * i + 1], type_xyz[t][3 * i + 2]});
    for (int k = 0; k < type_nf[t]; ++k)
      shapes[t].t.push_back({type_tris[t][3 * k], type_tris[t][3 * k + 1], type_tris[t][3 * k + 2]});
  }
  return hcg::pack_cells(nx, ny, nz, periodic, solid, ntypes, shapes, counts, margin, seed, max_attempts, centres,
                         angles, types);
}

}  // extern "C"
