// C ABI of the batched rigid-body step (declared in include/cubez_gpu.h).
//
// A batch owns every device buffer it uses (allocated once in
// cz_batch_create), one non-blocking CUDA stream, and a cache of captured
// CUDA graphs for multi-step rollouts.  Calls on one batch are serialised by
// the caller (the reference is single-threaded, contact.go has no locking).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <numeric>
#include <string>
#include <thread>
#include <utility>
#include <vector>

#include "../../include/cubez_gpu.h"
#include "cz_forms.h"
#include "cz_layout.cuh"

// Worlds of more bodies than this are resolved by k_resolve_big (bodies and
// contacts in global memory, a CTA of four warps per world).
constexpr int kBigWorld = 64;

namespace {

thread_local std::string g_last_error;
std::atomic<long long> g_launches{0};

int fail(int status, const std::string& msg) {
  g_last_error = msg;
  return status;
}

#define CZ_CUDA(call)                                                                                   \
  do {                                                                                                  \
    cudaError_t e_ = (call);                                                                            \
    if (e_ != cudaSuccess)                                                                              \
      return fail(CZ_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));                    \
  } while (0)

long long round_up(long long x, long long m) { return (x + m - 1) / m * m; }

}  // namespace

int cz::set_error(int status, const char* what, cudaError_t e) {
  g_last_error = std::string(what) + (e != cudaSuccess ? std::string(": ") + cudaGetErrorString(e) : "");
  return status;
}

struct cz_batch {
  const cz::FormOps* ops = nullptr;
  int form = 0;
  int device = 0;
  int sm_count = 0;
  size_t smem_optin = 0;
  cudaStream_t stream = nullptr;

  int num_worlds = 0;
  long long nb = 0, nb_pad = 0, nc_total = 0;
  std::vector<int> counts, bstart, ccap, h2p;
  std::vector<long long> cstart;
  int max_n = 0, nbs = 4, max_cap = 1;
  // worlds of more than kBigWorld bodies are resolved by k_resolve_big; the
  // others by k_resolve with a shared-memory slot of rs_nbs bodies
  int rs_nbs = 4, nsmall = 0;
  std::vector<int> big_ids;
  // Rollouts run the batch in parts, each its own chain of launches (part_rule)
  struct Part {
    int w0, w1;           // worlds
    long long b0, b1;     // padded bodies
    int nsmall, big0, nbig;
  };
  std::vector<Part> parts;
  std::vector<cudaStream_t> part_streams;  // of parts 1.. (part 0: the batch's)
  int* d_order_part = nullptr;             // the parts' narrowphase queues, one after the other
  int* d_order_rs_part = nullptr;          // ... and their resolver queues
  int* d_big = nullptr;
  int* d_units = nullptr;  // cz_collide's unit list
  long long units_cap = 0;
  void* big_bw = nullptr;
  void* big_br = nullptr;
  uint8_t* big_aw = nullptr;
  int* big_adj = nullptr;
  void* big_key = nullptr;
  int big_csm = 0;       // contacts whose arrays k_resolve_big keeps in shared memory
  size_t big_smem = 0;   // its shared memory per world

  // device buffers
  void* body = nullptr;
  uint8_t* awake = nullptr;
  uint8_t* can_sleep = nullptr;
  int* shape = nullptr;
  int *d_bstart = nullptr, *d_bcount = nullptr, *d_ccap = nullptr, *d_ccount = nullptr;
  long long* d_cstart = nullptr;
  uint32_t* d_wstatus = nullptr;
  int *d_piters = nullptr, *d_viters = nullptr, *d_cost = nullptr;
  void* contact = nullptr;
  int* cbodies = nullptr;
  void* work = nullptr;
  int* wbodies = nullptr;
  void* kmat = nullptr;  // per contact: friction K and response row, 16 reals
  int* d_order = nullptr;
  int* d_order_rs = nullptr;
  unsigned* d_queue = nullptr;
  uint32_t* d_status = nullptr;
  unsigned long long* d_counters = nullptr;
  int* d_h2p = nullptr;
  double* d_stage = nullptr;
  uint8_t* d_stage_u8 = nullptr;
  int* d_stage_i32 = nullptr;
  double* d_cstage = nullptr;
  int* d_cstage_b = nullptr;
  double* d_pow = nullptr;
  // collider Offsets (allocated by the first upload that carries them)
  void* d_offset = nullptr;       // [12][nb_pad] rows in the form's real type
  double* d_off_stage = nullptr;  // [n][12]
  double* h_off_stage = nullptr;  // pinned [n][12]
  bool has_offset = false;        // the last upload carried Offsets
  // pinned host staging
  double* h_stage = nullptr;
  uint8_t* h_stage_u8 = nullptr;
  int* h_stage_i32 = nullptr;
  double* h_cstage = nullptr;
  int* h_cstage_b = nullptr;
  double* h_pow = nullptr;
  uint32_t* h_status = nullptr;

  std::vector<double> lin_damp, ang_damp;
  double pow_dt = std::nan("");
  double plane[4] = {0, 1, 0, 0};
  int iter_mult = 4;
  int max_iterations = -1;

  // tuning
  int np_threads = 128, np_grid = 1, rs_cs = 128, rs_grid = 1, rs_ctas_per_sm = 0;
  int int_threads = 0;  // integrate_threads as set (0: integrate_cta)
  int rs_lanes = 8;  // resolver_lanes as set
  // lanes per world in the resolver (32 / run_lanes() worlds per warp): an island takes eight
  int run_lanes() const { return std::max(rs_lanes, 8); }
  int big_lanes = 32; // large_world_lanes as set (both settings run a CTA of four warps per world)
  int wait_limit = 1 << 22;  // polls of the narrowphase's bounded wait
  int wait_extra_tx = 0;     // test hook: bytes that wait expects beyond its copies
  int grid_min_bodies = 128; // narrowphase grid for worlds of at least this many bodies (0: never)
  int fused = 0;             // one launch per frame (the fused frame) where the batch allows it
  size_t fr_smem = 0;        // the fused frame's shared memory per CTA (0: it does not fit)
  int fr_grid = 1;           // the fused frame's CTAs
  int mode = 0;      // resolver mode: 0 plain, 1 harvest, 2 learned warm start
  cz::MlpDev mlp{};  // device copy of the warm-start network
  void* mlp_mem = nullptr;
  float* hv_features = nullptr;
  float* hv_labels = nullptr;
  unsigned long long* hv_count = nullptr;
  long long hv_cap = 0;
  void* ws_imp = nullptr;
  void* ws_rows = nullptr;  // per-body warm-start / harvest scratch (allocated on first use)
  int* ws_int = nullptr;
  uint8_t* ws_world = nullptr;
  float* ws_feat = nullptr;  // harvest features, allocated by the first cz_harvest
  int wf_grid = 1;           // k_warm_features CTAs
  int warm_shift = 2;        // warm-start worlds whose last solve used <= max_it >> warm_shift
  size_t np_smem = 0, rs_smem = 0;  // per narrowphase CTA; per resolver warp
  int rs_wpc = 1;                    // warps per resolver CTA
  bool rs_cs_set = false;            // the caller chose rs_cs (tile_rule otherwise)
  size_t wide_smem = 0;              // k_resolve_wide's shared memory per world (0: not used)
  int wide_cs = 0, wide_per_sm = 0;  // its contact tile, worlds per SM (wide_rule)
  int wide_grid = 0;                 // its CTAs: a world's each, or what rs_ctas_per_sm allows

  // graph cache: (nsteps, dt) -> executable graph
  std::map<std::pair<int, double>, cudaGraphExec_t> graphs;
  // the same rollouts with marks between the phases (cz_step_timed): event-record
  // nodes in one chain, stamps (k_stamp) in parts
  struct Timed {
    cudaGraphExec_t exec = nullptr;
    std::vector<cudaEvent_t> ev;  // 3 * nsteps + 1
  };
  std::map<std::pair<int, double>, Timed> timed;
  unsigned long long* stamps = nullptr;  // [kTimedParts][1 + stamp_cap]: how many, then the times
  size_t stamp_cap = 0;
  cudaEvent_t roll_ev[2] = {};  // around a rollout in parts
  // on-device copy of the body state (cz_snapshot / cz_restore)
  void* snap_body = nullptr;
  uint8_t* snap_u8 = nullptr;  // awake, can_sleep
  double snap_pow_dt = std::nan("");

  cz::HostView view() const {
    cz::HostView v;
    v.body = body;
    v.awake = awake;
    v.can_sleep = can_sleep;
    v.shape = shape;
    v.offset = has_offset ? d_offset : nullptr;
    v.nb_pad = nb_pad;
    v.first_body = 0;
    v.nb_run = nb_pad;
    v.first_world = 0;
    v.num_worlds = num_worlds;
    v.max_bodies = max_n;
    v.body_start = d_bstart;
    v.body_count = d_bcount;
    v.contact_start = d_cstart;
    v.contact_cap = d_ccap;
    v.contact_count = d_ccount;
    v.world_status = d_wstatus;
    v.pos_iters = d_piters;
    v.vel_iters = d_viters;
    v.cost = d_cost;
    v.contact = contact;
    v.contact_bodies = cbodies;
    v.work = work;
    v.kmat = kmat;
    v.work_bodies = wbodies;
    v.nc_total = nc_total;
    v.order = d_order;
    v.order_rs = d_order_rs;
    v.queue = d_queue;
    v.status = d_status;
    v.counters = d_counters;
    for (int i = 0; i < 4; ++i) v.plane[i] = plane[i];
    v.iter_mult = iter_mult;
    v.max_iterations = max_iterations;
    v.contact_writeback = 0;
    v.uniform_material = 1;
    v.mode = mode;
    v.mlp = mlp;
    v.hv_features = hv_features;
    v.hv_labels = hv_labels;
    v.hv_count = hv_count;
    v.hv_cap = hv_cap;
    v.ws_rows = ws_rows;
    v.ws_imp = ws_imp;
    v.ws_int = ws_int;
    v.ws_world = ws_world;
    v.ws_feat = ws_feat;
    v.warm_shift = warm_shift;
    v.big_list = d_big;
    v.big_count = (int)big_ids.size();
    v.big_bw = big_bw;
    v.big_br = big_br;
    v.big_aw = big_aw;
    v.big_adj = big_adj;
    v.big_key = big_key;
    v.wait_limit = wait_limit;
    v.wait_extra_tx = wait_extra_tx;
    v.grid_min_bodies = grid_min_bodies;
    return v;
  }
  // the view of one part of the batch
  cz::HostView view(const Part& p, int index) const {
    cz::HostView v = view();
    v.first_body = p.b0;
    v.nb_run = p.b1 - p.b0;
    v.first_world = p.w0;
    v.num_worlds = p.w1 - p.w0;
    v.order = d_order_part + p.w0;
    v.order_rs = d_order_rs_part + p.w0;
    v.queue = d_queue + 4 * index;
    v.big_list = d_big + p.big0;
    return v;
  }
};

namespace {

// Resolver queue for the next frame: worlds in decreasing rounds of this
// frame's resolve (a counting sort in one CTA), so that the longest chains
// start first and the worlds sharing a warp in lockstep have similar work (the
// rounds of a world, not its iterations: its islands run side by side).  The
// order of independent worlds does not change any result.
constexpr int kReorderBuckets = 2048;
__global__ void __launch_bounds__(1024) k_reorder(const int* __restrict__ cost, int w0, int W,
                                                  int* __restrict__ order,
                                                  const uint8_t* __restrict__ plain_next = nullptr) {
  __shared__ int hist[kReorderBuckets];
  __shared__ int wsum[32];
  const int tid = threadIdx.x;
  for (int i = tid; i < kReorderBuckets; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  // with the warm start on, the worlds it will serve (plain_next[w] == 0)
  // go first: their solve is usually short, but one that falls back solves
  // twice, and late in the queue that would be the frame's tail
  auto key_of_world = [&](int w) {
    if (plain_next && !plain_next[w]) return kReorderBuckets - 1;
    return min(cost[w], kReorderBuckets - 1);  // kExhausted: the longest chains, first
  };
  for (int w = w0 + tid; w < w0 + W; w += blockDim.x) atomicAdd(&hist[kReorderBuckets - 1 - key_of_world(w)], 1);
  __syncthreads();
  // exclusive scan of 2048 buckets, two per thread
  const int a = hist[2 * tid], c = hist[2 * tid + 1];
  int x = a + c;
  const int lane = tid & 31, wid = tid >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= d) x += y;
  }
  if (lane == 31) wsum[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int t = wsum[lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, t, d);
      if (lane >= d) t += y;
    }
    wsum[lane] = t;
  }
  __syncthreads();
  const int excl = x - (a + c) + (wid > 0 ? wsum[wid - 1] : 0);
  __syncthreads();
  hist[2 * tid] = excl;
  hist[2 * tid + 1] = excl + a;
  __syncthreads();
  for (int w = w0 + tid; w < w0 + W; w += blockDim.x)
    order[atomicAdd(&hist[kReorderBuckets - 1 - key_of_world(w)], 1)] = w;
}

void free_batch(cz_batch* b) {
  if (!b) return;
  cudaSetDevice(b->device);
  for (auto& kv : b->graphs) cudaGraphExecDestroy(kv.second);
  for (auto& kv : b->timed) {
    cudaGraphExecDestroy(kv.second.exec);
    for (cudaEvent_t e : kv.second.ev) cudaEventDestroy(e);
  }
  for (cudaEvent_t e : b->roll_ev)
    if (e) cudaEventDestroy(e);
  void* dev[] = {
      b->d_offset,  b->d_off_stage, b->ws_feat,   b->d_units,     b->d_big,      b->big_bw,      b->big_br,
      b->big_aw,    b->big_adj,     b->big_key,   b->ws_imp,      b->ws_rows,    b->ws_int,
      b->ws_world,  b->mlp_mem,     b->hv_features, b->hv_labels, b->hv_count,   b->snap_body,   b->snap_u8,
      b->stamps,    b->body,      b->awake,       b->can_sleep, b->shape,       b->d_bstart,   b->d_bcount,    b->d_ccap,
      b->d_ccount,  b->d_cstart,    b->d_wstatus, b->d_piters,    b->d_viters,    b->d_cost,   b->contact,     b->cbodies,
      b->work,      b->wbodies,     b->kmat,      b->d_order,    b->d_order_rs,  b->d_order_part, b->d_order_rs_part, b->d_queue,
      b->d_status,  b->d_counters,  b->d_h2p,     b->d_stage,     b->d_stage_u8, b->d_stage_i32, b->d_cstage,
      b->d_cstage_b, b->d_pow};
  for (void* p : dev)
    if (p) cudaFree(p);
  void* host[] = {b->h_off_stage, b->h_stage,    b->h_stage_u8, b->h_stage_i32,
                  b->h_cstage,     b->h_cstage_b, b->h_pow,      b->h_status};
  for (void* p : host)
    if (p) cudaFreeHost(p);
  for (cudaStream_t s : b->part_streams) cudaStreamDestroy(s);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

// Synchronise the batch stream and turn the device status word into a cz_status.
int finish(cz_batch* b) {
  CZ_CUDA(cudaMemcpyAsync(b->h_status, b->d_status, sizeof(uint32_t), cudaMemcpyDeviceToHost, b->stream));
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  const uint32_t bits = *b->h_status;
  const int st = cz::status_from_bits(bits);
  if (st != CZ_OK) {
    char buf[96];
    std::snprintf(buf, sizeof buf, "device status bits 0x%x", bits);
    g_last_error = buf;
  }
  return st;
}

// Copies between the caller's arrays and the pinned staging, in equal shares
// of at least 1 MB on up to eight threads, which end with the call: one thread
// copied, and faulted in the pages of fresh arrays, at 12 to 20 GB/s (147k
// bodies up 2.42 -> 0.97 ms, down 2.88 -> 1.29; the state of 524k bodies down
// 5.85 -> 2.20, of which a part is that only the fields asked for leave the GPU).
struct HostCopy {
  void* dst;
  const void* src;
  size_t bytes;
};
struct HostCopies {
  HostCopy c[20];
  int n = 0;
  void add(void* dst, const void* src, size_t bytes) { c[n++] = {dst, src, bytes}; }
};
void copy_share(const HostCopies& list, size_t from, size_t to) {
  size_t at = 0;
  for (int i = 0; i < list.n; ++i) {
    const HostCopy& c = list.c[i];
    const size_t a = std::max(from, at), e = std::min(to, at + c.bytes);
    if (a < e) std::memcpy(static_cast<char*>(c.dst) + (a - at), static_cast<const char*>(c.src) + (a - at), e - a);
    at += c.bytes;
  }
}
void host_copy(const HostCopies& list) {
  size_t total = 0;
  for (int i = 0; i < list.n; ++i) total += list.c[i].bytes;
  size_t shares = std::min<size_t>(total >> 20, 8);
  if (shares > 1) shares = std::min<size_t>(shares, std::thread::hardware_concurrency());
  shares = std::max<size_t>(shares, 1);
  auto cut = [&](size_t q) { return total / 64 * q / shares * 64 + (q == shares ? total % 64 : 0); };
  std::thread t[8];
  size_t started = 1;  // share 0 is this thread's
  try {
    for (; started < shares; ++started)
      t[started] = std::thread(copy_share, std::cref(list), cut(started), cut(started + 1));
  } catch (...) {  // no more threads: the rest is this thread's too
  }
  copy_share(list, 0, cut(1));
  if (started < shares) copy_share(list, cut(started), total);
  for (size_t q = 1; q < started; ++q) t[q].join();
}

int reset_status(cz_batch* b) {
  CZ_CUDA(cudaMemsetAsync(b->d_status, 0, sizeof(uint32_t), b->stream));
  return CZ_OK;
}

// pow(LinearDamping, dt) and pow(AngularDamping, dt) per body, computed on the
// host (math.Pow in the reference, rigidbody.go:233-234).
int ensure_pows(cz_batch* b, double dt) {
  if (b->pow_dt == dt) return CZ_OK;
  const long long P = b->nb_pad;
  for (long long i = 0; i < 2 * P; ++i) b->h_pow[i] = 1.0;
  // a pow for each run of equal values (by bits: -0 and NaN keep theirs), which
  // is most of them: 2.78 -> 0.29 ms for 147k bodies
  double lin = 0.0, ang = 0.0, lin_pow = 0.0, ang_pow = 0.0;
  for (long long h = 0; h < b->nb; ++h) {
    const long long p = b->h2p[h];
    if (h == 0 || std::memcmp(&b->lin_damp[h], &lin, sizeof lin) != 0)
      lin_pow = std::pow(lin = b->lin_damp[h], dt);
    if (h == 0 || std::memcmp(&b->ang_damp[h], &ang, sizeof ang) != 0)
      ang_pow = std::pow(ang = b->ang_damp[h], dt);
    b->h_pow[p] = lin_pow;
    b->h_pow[P + p] = ang_pow;
  }
  CZ_CUDA(cudaMemcpyAsync(b->d_pow, b->h_pow, sizeof(double) * 2 * P, cudaMemcpyHostToDevice, b->stream));
  CZ_CUDA(b->ops->set_rows(b->view(), cz::B_LINPOW, 2, b->d_pow, b->stream));
  g_launches++;
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  b->pow_dt = dt;
  return CZ_OK;
}

// Whether stepping runs the fused frame: one world per warp, plain resolver,
// every world within the shared-memory slot.
bool uses_frame(const cz_batch* b) {
  return b->fused && b->fr_smem > 0 && b->big_ids.empty() && b->rs_lanes == 32 && b->mode == 0 && b->nsmall > 0;
}

// Whether the resolver launch is k_resolve_wide (wide_rule, the plain resolver).
bool uses_wide(const cz_batch* b, int mode) { return b->wide_smem > 0 && mode == 0; }

// Whether a rollout runs the batch in parts.
bool in_parts(const cz_batch* b) { return !uses_frame(b) && b->parts.size() > 1; }
// Frames in one graph where the batch runs in parts (longer rollouts launch it
// again: the parts meet that often, and the graph has 6144 launches at most: 32
// parts of six, with the sort, the warm start's features and large worlds).
constexpr int kPartFrames = 32;
// Parts whose phases cz_step_timed marks, evenly spaced.
constexpr int kTimedParts = 4;
// The re-queue by cost matters where a launch's worlds do not all start at once.
constexpr int kReorderWorlds = 256;

// One frame's launches over a view of the batch (the whole of it, or a part),
// on a stream.
struct Chain {
  cz::HostView v;
  int nsmall, nbig;
  bool requeue;  // sort the worlds by cost for the next frame
  cudaStream_t s;
};
bool requeues(const cz_batch* b, int nsmall) { return nsmall > 32 / b->run_lanes(); }
Chain whole(cz_batch* b) {
  return {b->view(), b->nsmall, (int)b->big_ids.size(), requeues(b, b->nsmall), b->stream};
}

// CTAs for a view's worlds, of a kernel that takes `per_cta` worlds at a time
// and fills the GPU with `most`.
int chain_grid(int worlds, int per_cta, int most) {
  return std::max(1, std::min((worlds + per_cta - 1) / per_cta, most));
}

int launches_of(const cz_batch* b, int nsmall, int nbig, bool requeue) {
  return 2 + (nsmall > 0 ? 1 + (requeue ? 1 : 0) + (b->mode != 0 ? 1 : 0) : 0) + (nbig > 0 ? 1 : 0);
}
int launches_per_step(const cz_batch* b) {
  if (uses_frame(b)) return 1 + (b->nsmall > 1 ? 1 : 0);
  if (b->parts.size() == 1)
    return launches_of(b, b->nsmall, (int)b->big_ids.size(), requeues(b, b->nsmall));
  int n = 0;
  for (const auto& p : b->parts) n += launches_of(b, p.nsmall, p.nbig, p.nsmall > kReorderWorlds);
  return n;
}

// Integrate's CTA size unless the caller sets one: a warp per CTA in batches of
// up to 32768 body rows, so that few warps have an SM each, and 256 threads
// above, where the launch covers the GPU anyway.  By the batch's rows, not the
// launch's: a rollout's parts are on the GPU together.  float64, 20 frames from
// the fall, with 256 and with 32: 500 worlds of 30 bodies 3.02 and 2.84 ms,
// 1000 of 32 3.41 and 3.31, 1300 of 32 3.89 and 3.86, 2000 of 24 4.38 and 4.49,
// 2000 of 32 5.26 and 5.46; one launch (with its call) over 20000 rows 36.7 and
// 28.2 us, over 32000 36.8 both.  float32: one launch over 15600 rows 24.5 and
// 16.3 us, from 25000 rows on and in rollouts the same.
int integrate_cta(const cz_batch* b) { return b->int_threads > 0 ? b->int_threads : (b->nb_pad <= 32768 ? 32 : 256); }

int launch_integrate(cz_batch* b, const Chain& c, double dt) {
  CZ_CUDA(b->ops->integrate(c.v, dt, std::pow(0.5, dt), integrate_cta(b), c.s));
  g_launches++;
  return CZ_OK;
}
// `reset`: zero the queue first (in a frame, the integrate launch has)
int launch_narrowphase(cz_batch* b, const Chain& c, bool reset) {
  if (reset) CZ_CUDA(cudaMemsetAsync(c.v.queue, 0, sizeof(unsigned), c.s));
  CZ_CUDA(b->ops->narrowphase(c.v, b->nbs, b->np_threads, chain_grid(c.v.num_worlds, 1, b->np_grid), b->np_smem, c.s));
  g_launches++;
  return CZ_OK;
}
// The resolver launches of one frame: k_resolve over the worlds that fit its
// slot (then the re-queue of those worlds by cost), k_resolve_big over the
// others.
int launch_resolve(cz_batch* b, const Chain& c, double dt, bool reset) {
  if (c.nsmall > 0) {
    const int worlds_per_warp = 32 / b->run_lanes();
    if (reset) CZ_CUDA(cudaMemsetAsync(c.v.queue + 1, 0, 2 * sizeof(unsigned), c.s));
    if (c.v.mode != 0) {  // features (and, warm-starting, predictions) ahead of the resolver
      CZ_CUDA(b->ops->warm_features(c.v, b->rs_nbs, chain_grid(c.v.num_worlds, 1, b->wf_grid), dt, c.s));
      g_launches++;
    }
    if (uses_wide(b, c.v.mode))
      CZ_CUDA(b->ops->resolve_wide(c.v, b->rs_nbs, b->wide_cs, b->wide_per_sm, chain_grid(c.nsmall, 1, b->wide_grid),
                                   b->wide_smem, dt, c.s));
    else
      CZ_CUDA(b->ops->resolve(c.v, b->rs_nbs, b->rs_cs, b->run_lanes(),
                              chain_grid(c.v.num_worlds, worlds_per_warp * b->rs_wpc, b->rs_grid), b->rs_wpc,
                              b->rs_smem, dt, c.s));
    g_launches++;
    if (c.requeue) {
      k_reorder<<<1, 1024, 0, c.s>>>(b->d_cost, c.v.first_world, c.v.num_worlds, const_cast<int*>(c.v.order_rs),
                                     c.v.mode == 2 ? c.v.ws_world : nullptr);
      CZ_CUDA(cudaGetLastError());
      g_launches++;
    }
  }
  if (c.nbig > 0) {
    CZ_CUDA(b->ops->resolve_big(c.v, c.nbig, b->big_csm, b->big_smem, dt, c.s));
    g_launches++;
  }
  return CZ_OK;
}
// The fused frame: integrate, narrowphase and resolve of every world in one
// launch (then the re-queue by cost).
int launch_frame(cz_batch* b, double dt) {
  CZ_CUDA(cudaMemsetAsync(b->d_queue + 1, 0, sizeof(unsigned), b->stream));
  CZ_CUDA(b->ops->frame(b->view(), b->rs_nbs, b->rs_cs, b->fr_grid, b->fr_smem, dt, std::pow(0.5, dt), b->stream));
  g_launches++;
  if (b->nsmall > 1) {
    k_reorder<<<1, 1024, 0, b->stream>>>(b->d_cost, 0, b->num_worlds, b->d_order_rs);
    CZ_CUDA(cudaGetLastError());
    g_launches++;
  }
  return CZ_OK;
}

// How many parts a rollout runs the batch in: parallel branches of its graph,
// each a chain of frames over its own worlds.  Worlds are independent, but a
// launch over all of them ends with its longest world, and a frame's next
// launch waited for that: half of a resolver launch was its tail (8192 worlds
// of 32 bodies, float32: 0.62 of 1.2 ms with the SMs busy).  With parts, one
// part's tail runs beside the others' work.  At least 64 worlds each, at most 32
// parts in float64 and 8 in float32, whose launches are short.  32 frames from
// the fall, from frame 120 and from 400, with 1, 8 and 32 parts, ms:
//   float64  1001 x 24       6.4  38.0  27.8    5.0  27.7  25.7    4.7  26.1  23.9 (15 parts)
//            2000 x 32      12.1  62.0  46.9    9.0  50.3  40.0    9.8  47.3  42.7
//            4096 x 8 to 64 20.3 142.5 114.3   16.0 119.7 114.7   18.3 128.7 129.2
//            8192 x 32      27.8 159.9 140.7   23.7 134.3 124.1   26.3 147.3 140.0
//   float32  1000 x 32       3.4  16.4  11.4    2.9  13.8  11.2    2.9  13.6  11.3
//            4096 x 8 to 64  7.5  48.0  43.0    6.3  41.0  40.4    7.6  36.8  40.4
//           16384 x 32      15.9  65.2  59.0   14.6  56.4  50.1   17.5  66.5  60.7
// (float64's 32 were the fastest of these while a resolver launch took twice as
// long; from some 2000 worlds on eight now are, and a settled mixed batch of
// 4096 is 13 % faster in one part than in 32.)
int part_rule(int form, int num_worlds) {
  return std::max(1, std::min(num_worlds / 64, form == CZ_FORM_FP64 ? 32 : 8));
}

// Contacts of the resolver's shared-memory tile: three a body, which a settled
// heap of cubes reaches (2.6 to 2.8), at least 96.  A world with more keeps all
// its records in global memory, and its iterations then load through what L1
// the tiles leave: 4096 worlds of 62 bodies x 10 frames, float32, took 29.4 ms
// with 96 and 22.6 with 192 although 9 worlds fit an SM then instead of 12; 48
// bodies 16.2 and 14.0 (160), 40 bodies 11.0 and 9.6 (128); 4096 worlds of 8 to
// 64 bodies x 30 45.1 and 39.1.  More than that only costs occupancy: 16384
// worlds of 32 bodies x 30 51.2 with 96, 52.9 with 128.  float64: 1024 x 62
// bodies 35.9 -> 31.6, 4096 x 8 to 64 125.5 -> 124.8.  Narrower groups have
// several worlds' tiles to a warp, and stay with 96.
int tile_rule(int nbs, int lanes) { return lanes < 32 ? 96 : std::max(96, (int)round_up(3 * nbs, 32)); }

// Worlds per SM that k_resolve_wide holds, four warps to each; 0: k_resolve
// takes the batch, one warp to a world.  Up to one world per SM that is where
// they have more than a dozen bodies: one world of 20 cubes, float64, 278 ->
// 215 us a frame; 61 worlds of 8 to 64 bodies, float32, 604 -> 494; 150 of 62
// bodies x 20 frames, float64, 28.1 -> 24.8 ms (150 of 8, float32, 2.18 ->
// 2.24: few islands, and one warp is as good).  Up to three worlds per SM where
// their tiles leave an SM few warps otherwise, x 10 frames: 450 of 62 bodies,
// float64 34.4 -> 26.5 ms, float32 13.4 -> 11.4; 450 of 8 to 64 33.4 -> 23.3 and
// 11.9 -> 9.4; but 300 freshly landed ones of 24 bodies x 3, float32, 0.47 ->
// 0.49.  Up to seven per SM (three at a time) where they are nearly the largest:
// 1000 of 62 settled bodies x 3, float64 12.8 -> 11.1 ms, float32 4.62 -> 4.27,
// of 8 to 64 float32 4.70 -> 3.73, fresh ones the same; 1000 of 40 gain 5 to 10 %
// settled and lose 4 fresh.  With many worlds one warp is better throughout
// (4096 of 62, float32, 11.8 -> 14.3).
// In float64, whose rate one warp reaches a quarter of, up to seven per SM from
// 24 slots on: 1001 worlds of 24 bodies with Offsets x 20 20.3 -> 19.4 ms, 600
// settled of 31 x 4 5.95 -> 5.21, 1000 settled of 32 x 5 7.55 -> 6.63, against
// fresh ones of 24 to 40 bodies, 0.97 to 1.04 times (300 of 24 x 3, 1.05 -> 1.08).
// Around the ends, 6 frames from frame 60 and from 240, one warp's time over
// four warps': float64, 24 bodies, 450 worlds 0.99 and 1.16, 1000 (7 per SM)
// 0.99 and 1.04, 1200 (8) 0.98 and 1.03, 1500 0.97 and 1.06, 2100 0.93 and 0.99;
// 62 bodies, 1000 1.06 and 1.11, 1500 1.04 and 1.22, 2100 1.01 and 1.14; 20
// bodies, 300 1.02 and 1.01, 1000 1.01 and 0.99; 16 bodies, 450 1.02 and 1.04,
// 1000 1.00 and 0.97, 1500 0.97 and 0.93.  float32, 62 bodies, 1000 1.10 and
// 1.12, 1500 1.04 and 1.09; 450 of 36 0.98 and 1.14, 450 of 32 0.97 and 1.08.
// So from eight per SM on small falling worlds lose what they gain at rest (the
// largest would still gain), and below 24 slots nothing is gained by seven.
int wide_rule(int form, int worlds, int nbs, int lanes, int sms) {
  if (lanes != 32 || worlds <= 0) return 0;
  const int per_sm = (worlds + sms - 1) / sms;
  if (per_sm == 1) return nbs >= 16 ? 1 : 0;
  const bool wide = form == CZ_FORM_FP64 ? nbs >= 24 : nbs >= (per_sm <= 3 ? 36 : 52);
  return wide && per_sm <= 7 ? std::min(per_sm, 3) : 0;
}

void drop_timed(cz_batch* b) {
  for (auto& kv : b->timed) {
    cudaGraphExecDestroy(kv.second.exec);
    for (cudaEvent_t e : kv.second.ev) cudaEventDestroy(e);
  }
  b->timed.clear();
}
// The captured graphs hold the kernels' parameters (the batch view); drop them
// whenever those change.
void drop_graphs(cz_batch* b) {
  for (auto& kv : b->graphs) cudaGraphExecDestroy(kv.second);
  b->graphs.clear();
  drop_timed(b);
}

int configure(cz_batch* b) {
  // resolver shared-memory tile: shrink the contact capacity until it fits
  if (!b->rs_cs_set) b->rs_cs = tile_rule(b->rs_nbs, b->run_lanes());
  int cs = std::min<long long>(b->rs_cs, round_up(b->max_cap, 32));
  cs = std::max(cs, 32);
  while (cs > 32 && b->ops->rs_smem(b->rs_nbs, cs, b->run_lanes()) > b->smem_optin) cs -= 32;
  b->rs_cs = cs;
  b->rs_smem = b->ops->rs_smem(b->rs_nbs, cs, b->run_lanes());
  b->np_smem = b->ops->np_smem(b->nbs);
  if (b->np_smem > b->smem_optin || b->rs_smem > b->smem_optin)
    return fail(CZ_ERR_BODY_LIMIT, "world too large for the shared-memory tiles");
  int npb = 0, rsb = 0;
  // Resolver warps are independent (each takes its own worlds), so a CTA holds
  // as many as make the most resident warps per SM (the SM keeps 1 KB of
  // shared memory per CTA), the fewest where several counts do; few worlds are
  // spread over the SMs.
  const int lanes = b->run_lanes();
  const long long groups = (std::max(b->nsmall, 1) + 32 / lanes - 1) / (32 / lanes);
  const int fit = (int)(b->smem_optin / b->rs_smem);
  const int most = (int)std::min<long long>(std::min(b->ops->rs_wpc(lanes), fit),
                                            (groups + b->sm_count - 1) / b->sm_count);
  CZ_CUDA(b->ops->prepare(b->np_smem, std::max(most, 1) * b->rs_smem, lanes));
  b->rs_wpc = 1;
  for (int wpc = 1; wpc <= std::max(most, 1); ++wpc) {
    int blocks = 0;
    CZ_CUDA(b->ops->rs_occupancy(&blocks, wpc, b->rs_smem, lanes, b->mode));
    if (wpc == 1 || blocks * wpc > rsb * b->rs_wpc) {
      rsb = blocks;
      b->rs_wpc = wpc;
    }
  }
  // Four warps to a world (wide_rule), in tiles of eight contacts a body with
  // their friction matrices, or what lets the SMs hold all the worlds at once.
  b->wide_smem = 0;
  const int per_sm = wide_rule(b->form, b->nsmall, b->rs_nbs, lanes, b->sm_count);
  if (per_sm > 0) {
    b->wide_cs = std::max(b->rs_cs, std::min((int)round_up(b->max_cap, 32), 8 * b->rs_nbs));
    while (b->wide_cs > b->rs_cs &&
           (b->ops->wide_smem(b->rs_nbs, b->wide_cs) + 1024) * per_sm > b->smem_optin + 1024)
      b->wide_cs -= 32;
    const size_t bytes = b->ops->wide_smem(b->rs_nbs, b->wide_cs);
    if (bytes <= b->smem_optin) {
      CZ_CUDA(b->ops->wide_prepare(per_sm, bytes));
      b->wide_per_sm = per_sm;
      b->wide_grid = b->nsmall;
      if (b->rs_ctas_per_sm > 0)
        b->wide_grid = (int)std::min<long long>(b->nsmall, (long long)b->rs_ctas_per_sm * b->sm_count);
      b->wide_smem = bytes;
    }
  }
  CZ_CUDA(b->ops->occupancy(&npb, b->np_threads, b->np_smem,
                            cz::np_mode(b->grid_min_bodies, b->max_n)));
  npb = std::max(npb, 1);
  rsb = std::max(rsb, 1);
  if (b->rs_ctas_per_sm > 0) rsb = std::min(rsb, b->rs_ctas_per_sm);
  b->np_grid = (int)std::min<long long>(b->num_worlds, (long long)npb * b->sm_count);
  b->rs_grid = (int)std::min<long long>((groups + b->rs_wpc - 1) / b->rs_wpc, (long long)rsb * b->sm_count);
  b->np_grid = std::max(b->np_grid, 1);
  b->rs_grid = std::max(b->rs_grid, 1);
  b->wf_grid = (int)std::min<long long>(std::max(b->nsmall, 1),
                                        (long long)b->ops->warm_features_blocks(b->rs_nbs) * b->sm_count);
  if (!b->big_ids.empty()) {
    // the large-world resolver's shared memory: half an SM's where several
    // worlds share an SM (1024 bodies with 6 contacts each fit that), else all
    int n = 0, cap = 0;
    for (int w : b->big_ids) {
      n = std::max(n, b->counts[w]);
      cap = std::max(cap, b->ccap[w]);
    }
    const size_t budget = (int)b->big_ids.size() > b->sm_count ? (size_t)112 * 1024 : b->smem_optin;
    CZ_CUDA(b->ops->big_smem(n, cap, budget, &b->big_csm, &b->big_smem));
  }
  // the fused frame's slot holds the resolver's tile and the narrowphase's
  b->fr_smem = b->ops->frame_smem(b->rs_nbs, b->rs_cs);
  if (b->fr_smem > b->smem_optin) {
    b->fr_smem = 0;
  } else {
    int frb = 0;
    CZ_CUDA(b->ops->frame_occupancy(&frb, b->fr_smem));
    frb = std::max(frb, 1);
    if (b->rs_ctas_per_sm > 0) frb = std::min(frb, b->rs_ctas_per_sm);
    b->fr_grid = (int)std::max<long long>(1, std::min<long long>(std::max(b->nsmall, 1), (long long)frb * b->sm_count));
  }
  drop_graphs(b);
  return CZ_OK;
}

}  // namespace

extern "C" {

const char* cz_status_string(int status) {
  switch (status) {
    case CZ_OK: return "ok";
    case CZ_ERR_BAD_ARG: return "bad argument";
    case CZ_ERR_CUDA: return "CUDA error";
    case CZ_ERR_NO_DEVICE: return "no CUDA device";
    case CZ_ERR_NONFINITE: return "non-finite box transform in the box-box test";
    case CZ_ERR_CAPACITY: return "contact capacity exceeded";
    case CZ_ERR_TIMEOUT: return "device wait timed out";
    case CZ_ERR_FRICTIONLESS: return "frictionless impulse on a single-body contact";
    case CZ_ERR_BODY_LIMIT: return "world too large for the kernel tiles";
    default: return "unknown status";
  }
}

const char* cz_last_error(void) { return g_last_error.c_str(); }

int64_t cz_kernel_launches(void) { return g_launches.load(); }

int cz_batch_create(const cz_batch_desc* d, cz_batch** out) {
  if (!d || !out || d->num_worlds <= 0 || !d->body_counts || (d->form != CZ_FORM_FP64 && d->form != CZ_FORM_FP32))
    return fail(CZ_ERR_BAD_ARG, "cz_batch_create: bad descriptor");
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) return fail(CZ_ERR_NO_DEVICE, "no CUDA device");
  if (d->device < 0 || d->device >= ndev) return fail(CZ_ERR_BAD_ARG, "cz_batch_create: bad device ordinal");
  for (int w = 0; w < d->num_worlds; ++w)
    if (d->body_counts[w] < 0 || d->body_counts[w] >= 65535)
      return fail(CZ_ERR_BAD_ARG, "cz_batch_create: body count out of range");
  cz_batch* b = new cz_batch();
  b->form = d->form;
  b->ops = d->form == CZ_FORM_FP64 ? &cz::kFormFP64 : &cz::kFormFP32;
  b->device = d->device;
  int st = CZ_OK;
  auto bail = [&](int s) {
    free_batch(b);
    return s;
  };
  if (cudaSetDevice(b->device) != cudaSuccess) return bail(fail(CZ_ERR_CUDA, "cudaSetDevice failed"));
  cudaDeviceGetAttribute(&b->sm_count, cudaDevAttrMultiProcessorCount, b->device);
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, b->device);
  b->smem_optin = (size_t)optin;
  b->num_worlds = d->num_worlds;
  b->counts.assign(d->body_counts, d->body_counts + d->num_worlds);
  for (int i = 0; i < 3; ++i) b->plane[i] = d->plane[i];
  b->plane[3] = d->plane[3];
  if (d->plane[0] == 0 && d->plane[1] == 0 && d->plane[2] == 0) {
    b->plane[0] = 0; b->plane[1] = 1; b->plane[2] = 0;
  }
  b->iter_mult = d->iteration_multiplier > 0 ? d->iteration_multiplier : 4;
  b->max_iterations = d->max_iterations > 0 ? d->max_iterations : -1;
  // layout
  long long nb = 0, np = 0, nc = 0;
  for (int w = 0; w < b->num_worlds; ++w) {
    const int n = b->counts[w];
    b->bstart.push_back((int)np);
    for (int i = 0; i < n; ++i) b->h2p.push_back((int)(np + i));
    np = round_up(np + n, 4);
    nb += n;
    b->max_n = std::max(b->max_n, n);
    const long long worst = 8LL * n + (long long)n * (n - 1);
    long long cap = std::min<long long>(worst, std::max<long long>(64LL * n, 4608));
    if (d->contact_capacity > 0) cap = std::min<long long>(worst, d->contact_capacity);
    cap = std::max<long long>(cap, 1);
    b->ccap.push_back((int)cap);
    b->cstart.push_back(nc);
    nc += round_up(cap, 4);
    b->max_cap = std::max<int>(b->max_cap, (int)cap);
  }
  b->nb = nb;
  b->nb_pad = std::max<long long>(np, 4);
  b->nc_total = std::max<long long>(nc, 4);
  b->nbs = (int)std::max<long long>(round_up(b->max_n, 4), 4);
  int max_small = 0;
  for (int w = 0; w < b->num_worlds; ++w) {
    if (b->counts[w] > kBigWorld)
      b->big_ids.push_back(w);
    else
      max_small = std::max(max_small, b->counts[w]);
  }
  b->nsmall = b->num_worlds - (int)b->big_ids.size();
  b->rs_nbs = (int)std::max<long long>(round_up(max_small, 4), 4);
  b->np_threads = b->max_n >= 256 ? 256 : 128;
  // a world per warp: its islands share the warp's instructions (the tuner may
  // change it)
  b->rs_lanes = 32;
  // world queue: decreasing body count (pair work grows as n^2)
  std::vector<int> order(b->num_worlds);
  std::iota(order.begin(), order.end(), 0);
  const auto larger = [&](int a, int c) { return b->counts[a] > b->counts[c]; };
  std::vector<int> order_part(order);
  std::stable_sort(order.begin(), order.end(), larger);
  // parts: consecutive worlds, about as many in each
  const int nparts = part_rule(b->form, b->num_worlds);
  for (int p = 0; p < nparts; ++p) {
    cz_batch::Part part{};
    part.w0 = (int)((long long)b->num_worlds * p / nparts);
    part.w1 = (int)((long long)b->num_worlds * (p + 1) / nparts);
    part.b0 = b->bstart[part.w0];
    part.b1 = part.w1 < b->num_worlds ? b->bstart[part.w1] : b->nb_pad;
    for (int w = part.w0; w < part.w1; ++w) part.nbig += b->counts[w] > kBigWorld;
    part.nsmall = part.w1 - part.w0 - part.nbig;
    part.big0 = (int)(std::lower_bound(b->big_ids.begin(), b->big_ids.end(), part.w0) - b->big_ids.begin());
    std::stable_sort(order_part.begin() + part.w0, order_part.begin() + part.w1, larger);
    b->parts.push_back(part);
  }

  const size_t R = b->ops->real_size;
  const long long P = b->nb_pad, C = b->nc_total, W = b->num_worlds;
  auto dmalloc = [&](void** p, size_t bytes) -> bool {
    if (cudaMalloc(p, std::max<size_t>(bytes, 16)) != cudaSuccess) return false;
    return true;
  };
  bool ok = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) == cudaSuccess;
  for (int p = 1; ok && p < nparts; ++p) {
    cudaStream_t s = nullptr;
    ok = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess;
    if (ok) b->part_streams.push_back(s);
  }
  ok = ok && dmalloc((void**)&b->d_order_part, sizeof(int) * W) && dmalloc((void**)&b->d_order_rs_part, sizeof(int) * W);
  ok = ok && dmalloc(&b->body, R * cz::B_NROWS * P);
  ok = ok && dmalloc((void**)&b->awake, P) && dmalloc((void**)&b->can_sleep, P) &&
       dmalloc((void**)&b->shape, sizeof(int) * P);
  ok = ok && dmalloc((void**)&b->d_bstart, sizeof(int) * W) && dmalloc((void**)&b->d_bcount, sizeof(int) * W) &&
       dmalloc((void**)&b->d_ccap, sizeof(int) * W) && dmalloc((void**)&b->d_ccount, sizeof(int) * W) &&
       dmalloc((void**)&b->d_cstart, sizeof(long long) * W) && dmalloc((void**)&b->d_wstatus, sizeof(uint32_t) * W) &&
       dmalloc((void**)&b->d_piters, sizeof(int) * W) && dmalloc((void**)&b->d_viters, sizeof(int) * W) &&
       dmalloc((void**)&b->d_cost, sizeof(int) * W) &&
       dmalloc((void**)&b->d_order, sizeof(int) * W) && dmalloc((void**)&b->d_order_rs, sizeof(int) * W);
  ok = ok && dmalloc(&b->contact, R * cz::C_NROWS * C) && dmalloc((void**)&b->cbodies, sizeof(int) * C);
  ok = ok && dmalloc(&b->work, R * cz::CREC * C) && dmalloc((void**)&b->wbodies, sizeof(int) * C);
  ok = ok && dmalloc(&b->kmat, R * cz::K_ROW * C);
  ok = ok && dmalloc((void**)&b->d_queue, 4 * sizeof(unsigned) * nparts) && dmalloc((void**)&b->d_status, sizeof(uint32_t)) &&
       dmalloc((void**)&b->d_counters, 8 * sizeof(unsigned long long));
  ok = ok && dmalloc((void**)&b->d_h2p, sizeof(int) * std::max<long long>(nb, 1));
  ok = ok && dmalloc((void**)&b->d_stage, sizeof(double) * cz::SG_NDOUBLES * std::max<long long>(nb, 1)) &&
       dmalloc((void**)&b->d_stage_u8, 2 * std::max<long long>(nb, 1)) &&
       dmalloc((void**)&b->d_stage_i32, sizeof(int) * std::max<long long>(nb, 1));
  ok = ok && dmalloc((void**)&b->d_cstage, sizeof(double) * cz::C_NROWS * b->max_cap) &&
       dmalloc((void**)&b->d_cstage_b, sizeof(int) * b->max_cap);
  ok = ok && dmalloc((void**)&b->d_pow, sizeof(double) * 2 * P);
  ok = ok && dmalloc(&b->snap_body, R * cz::B_NROWS * P) && dmalloc((void**)&b->snap_u8, 2 * P);
  if (!b->big_ids.empty()) {
    ok = ok && dmalloc((void**)&b->d_big, sizeof(int) * b->big_ids.size()) &&
         dmalloc(&b->big_bw, sizeof(double) * 7 * P) && dmalloc(&b->big_br, R * cz::BREC * P) &&
         dmalloc((void**)&b->big_aw, P) && dmalloc((void**)&b->big_adj, sizeof(int) * 2 * C) &&
         dmalloc(&b->big_key, R * C);
  }
  if (!ok) return bail(fail(CZ_ERR_CUDA, "device allocation failed"));
  ok = cudaMallocHost((void**)&b->h_stage, sizeof(double) * cz::SG_NDOUBLES * std::max<long long>(nb, 1)) ==
           cudaSuccess &&
       cudaMallocHost((void**)&b->h_stage_u8, 2 * std::max<long long>(nb, 1)) == cudaSuccess &&
       cudaMallocHost((void**)&b->h_stage_i32, sizeof(int) * std::max<long long>(nb, 1)) == cudaSuccess &&
       cudaMallocHost((void**)&b->h_cstage, sizeof(double) * cz::C_NROWS * b->max_cap) == cudaSuccess &&
       cudaMallocHost((void**)&b->h_cstage_b, sizeof(int) * b->max_cap) == cudaSuccess &&
       cudaMallocHost((void**)&b->h_pow, sizeof(double) * 2 * P) == cudaSuccess &&
       cudaMallocHost((void**)&b->h_status, sizeof(uint32_t)) == cudaSuccess;
  if (!ok) return bail(fail(CZ_ERR_CUDA, "pinned host allocation failed"));
  cudaStream_t s = b->stream;
  std::vector<int> bcount(b->counts);
  if (cudaMemsetAsync(b->body, 0, R * cz::B_NROWS * P, s) != cudaSuccess ||
      cudaMemsetAsync(b->awake, 0, P, s) != cudaSuccess || cudaMemsetAsync(b->can_sleep, 0, P, s) != cudaSuccess ||
      cudaMemsetAsync(b->shape, 0xFF, sizeof(int) * P, s) != cudaSuccess ||
      cudaMemsetAsync(b->d_ccount, 0, sizeof(int) * W, s) != cudaSuccess ||
      cudaMemsetAsync(b->d_wstatus, 0, sizeof(uint32_t) * W, s) != cudaSuccess ||
      cudaMemsetAsync(b->d_piters, 0, sizeof(int) * W, s) != cudaSuccess ||
      cudaMemsetAsync(b->d_viters, 0, sizeof(int) * W, s) != cudaSuccess ||
      cudaMemsetAsync(b->d_cost, 0, sizeof(int) * W, s) != cudaSuccess ||
      cudaMemsetAsync(b->d_queue, 0, 4 * sizeof(unsigned) * nparts, s) != cudaSuccess ||
      cudaMemsetAsync(b->d_status, 0, sizeof(uint32_t), s) != cudaSuccess ||
      cudaMemsetAsync(b->d_counters, 0, 8 * sizeof(unsigned long long), s) != cudaSuccess ||
      cudaMemsetAsync(b->cbodies, 0xFF, sizeof(int) * C, s) != cudaSuccess ||
      cudaMemcpyAsync(b->d_bstart, b->bstart.data(), sizeof(int) * W, cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(b->d_bcount, bcount.data(), sizeof(int) * W, cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(b->d_ccap, b->ccap.data(), sizeof(int) * W, cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(b->d_cstart, b->cstart.data(), sizeof(long long) * W, cudaMemcpyHostToDevice, s) !=
          cudaSuccess ||
      cudaMemcpyAsync(b->d_order, order.data(), sizeof(int) * W, cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(b->d_order_rs, order.data(), sizeof(int) * W, cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(b->d_order_part, order_part.data(), sizeof(int) * W, cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(b->d_order_rs_part, order_part.data(), sizeof(int) * W, cudaMemcpyHostToDevice, s) !=
          cudaSuccess ||
      (!b->big_ids.empty() && cudaMemcpyAsync(b->d_big, b->big_ids.data(), sizeof(int) * b->big_ids.size(),
                                              cudaMemcpyHostToDevice, s) != cudaSuccess) ||
      (nb > 0 &&
       cudaMemcpyAsync(b->d_h2p, b->h2p.data(), sizeof(int) * nb, cudaMemcpyHostToDevice, s) != cudaSuccess) ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return bail(fail(CZ_ERR_CUDA, "device initialisation failed"));
  b->lin_damp.assign(nb, 0.95);
  b->ang_damp.assign(nb, 0.95);
  st = configure(b);
  if (st != CZ_OK) return bail(st);
  *out = b;
  return CZ_OK;
}

int cz_batch_destroy(cz_batch* b) {
  if (!b) return fail(CZ_ERR_BAD_ARG, "cz_batch_destroy: null batch");
  free_batch(b);
  return CZ_OK;
}

int cz_set_tuning(cz_batch* b, const cz_tuning* t) {
  if (!b || !t) return fail(CZ_ERR_BAD_ARG, "cz_set_tuning: null argument");
  CZ_CUDA(cudaSetDevice(b->device));
  if (t->narrowphase_threads > 0) {
    if (t->narrowphase_threads % 32 != 0 || t->narrowphase_threads > 256)
      return fail(CZ_ERR_BAD_ARG, "narrowphase_threads must be a multiple of 32, at most 256");
    b->np_threads = t->narrowphase_threads;
  }
  if (t->resolver_contacts > 0) {
    b->rs_cs = (int)round_up(t->resolver_contacts, 32);
    b->rs_cs_set = true;
  }
  if (t->resolver_lanes > 0) {
    if (t->resolver_lanes != 4 && t->resolver_lanes != 8 && t->resolver_lanes != 16 && t->resolver_lanes != 32)
      return fail(CZ_ERR_BAD_ARG, "resolver_lanes must be 4, 8, 16 or 32");
    b->rs_lanes = t->resolver_lanes;
  }
  if (t->resolver_ctas_per_sm > 0) b->rs_ctas_per_sm = t->resolver_ctas_per_sm;
  if (t->integrate_threads > 0) {
    if (t->integrate_threads % 32 != 0 || t->integrate_threads > 256)
      return fail(CZ_ERR_BAD_ARG, "integrate_threads must be a multiple of 32, at most 256");
    b->int_threads = t->integrate_threads;
  }
  if (t->large_world_lanes > 0) {
    if (t->large_world_lanes != 16 && t->large_world_lanes != 32)
      return fail(CZ_ERR_BAD_ARG, "large_world_lanes must be 16 or 32");
    b->big_lanes = t->large_world_lanes;
  }
  if (t->warm_start_budget_shift > 0) {
    if (t->warm_start_budget_shift > 8) return fail(CZ_ERR_BAD_ARG, "warm_start_budget_shift must be 1 to 8");
    b->warm_shift = t->warm_start_budget_shift;
  }
  if (t->fused_frame != 0) b->fused = t->fused_frame > 0 ? 1 : 0;
  if (t->broadphase_min_bodies != 0) {
    if (t->broadphase_min_bodies < -1) return fail(CZ_ERR_BAD_ARG, "broadphase_min_bodies must be -1 or positive");
    b->grid_min_bodies = t->broadphase_min_bodies < 0 ? 0 : t->broadphase_min_bodies;
  }
  return configure(b);
}

int cz_set_wait_test(cz_batch* b, int32_t extra_bytes, int32_t wait_limit) {
  if (!b || extra_bytes < 0 || extra_bytes > 4096 || wait_limit < 0) return CZ_ERR_BAD_ARG;
  b->wait_extra_tx = extra_bytes;
  b->wait_limit = wait_limit > 0 ? wait_limit : (1 << 22);
  drop_graphs(b);
  return CZ_OK;
}

int cz_get_tuning(cz_batch* b, cz_tuning* t) {
  if (!b || !t) return fail(CZ_ERR_BAD_ARG, "cz_get_tuning: null argument");
  t->narrowphase_threads = b->np_threads;
  t->resolver_contacts = b->rs_cs;
  const int sms = std::max(b->sm_count, 1);
  t->resolver_ctas_per_sm = uses_wide(b, b->mode) ? (b->wide_grid + sms - 1) / sms : b->rs_grid / sms;
  t->integrate_threads = integrate_cta(b);
  t->resolver_lanes = b->rs_lanes;
  t->warm_start_budget_shift = b->warm_shift;
  t->broadphase_min_bodies = b->grid_min_bodies > 0 ? b->grid_min_bodies : -1;
  t->fused_frame = b->fused ? 1 : -1;
  t->large_world_lanes = b->big_lanes;
  return CZ_OK;
}

int cz_upload_bodies(cz_batch* b, const cz_bodies* in) {
  if (!b || !in) return fail(CZ_ERR_BAD_ARG, "cz_upload_bodies: null argument");
  if (!in->position || !in->orientation || !in->velocity || !in->rotation || !in->acceleration ||
      !in->inverse_inertia || !in->inverse_mass || !in->linear_damping || !in->angular_damping || !in->is_awake ||
      !in->can_sleep || !in->shape || !in->half_size || !in->radius)
    return fail(CZ_ERR_BAD_ARG, "cz_upload_bodies: missing body field");
  CZ_CUDA(cudaSetDevice(b->device));
  const long long n = b->nb;
  if (n == 0) return CZ_OK;
  for (long long h = 0; h < n; ++h)
    if (in->shape[h] != CZ_SHAPE_SPHERE && in->shape[h] != CZ_SHAPE_CUBE)
      return fail(CZ_ERR_BAD_ARG, "cz_upload_bodies: unknown shape");
  double* sg = b->h_stage;
  const int has_iw = in->inverse_inertia_world != nullptr;
  const int has_lfa = in->last_frame_acceleration != nullptr;
  HostCopies list;
  auto add = [&](int blk, const double* src, int width) {
    if (src) list.add(sg + (long long)blk * n, src, sizeof(double) * width * n);
  };
  add(cz::SG_POS, in->position, 3);
  add(cz::SG_Q, in->orientation, 4);
  add(cz::SG_VEL, in->velocity, 3);
  add(cz::SG_ROT, in->rotation, 3);
  add(cz::SG_ACC, in->acceleration, 3);
  add(cz::SG_IB, in->inverse_inertia, 9);
  add(cz::SG_INVM, in->inverse_mass, 1);
  add(cz::SG_MOTION, in->motion, 1);
  add(cz::SG_HALF, in->half_size, 3);
  add(cz::SG_RAD, in->radius, 1);
  add(cz::SG_IW, in->inverse_inertia_world, 9);
  add(cz::SG_LFA, in->last_frame_acceleration, 3);
  list.add(b->h_stage_u8, in->is_awake, (size_t)n);
  list.add(b->h_stage_u8 + n, in->can_sleep, (size_t)n);
  list.add(b->h_stage_i32, in->shape, sizeof(int) * n);
  const bool has_off = in->collider_offset != nullptr;
  if (has_off && !b->d_offset) {
    const size_t rows = b->ops->real_size * 12 * std::max<long long>(b->nb_pad, 1);
    void* rows_d = nullptr;
    double *stage_d = nullptr, *stage_h = nullptr;
    if (cudaMalloc(&rows_d, rows) != cudaSuccess ||
        cudaMalloc((void**)&stage_d, sizeof(double) * 12 * n) != cudaSuccess ||
        cudaMallocHost((void**)&stage_h, sizeof(double) * 12 * n) != cudaSuccess) {
      if (rows_d) cudaFree(rows_d);
      if (stage_d) cudaFree(stage_d);
      return fail(CZ_ERR_CUDA, "cz_upload_bodies: Offset allocation failed");
    }
    b->d_offset = rows_d;
    b->d_off_stage = stage_d;
    b->h_off_stage = stage_h;
    CZ_CUDA(cudaMemsetAsync(b->d_offset, 0, rows, b->stream));
  }
  if (has_off != b->has_offset) {
    drop_graphs(b);  // the narrowphase's view changes
    b->has_offset = has_off;
  }
  if (has_off) list.add(b->h_off_stage, in->collider_offset, sizeof(double) * 12 * n);
  host_copy(list);
  if (!in->motion)
    for (long long h = 0; h < n; ++h) sg[cz::SG_MOTION * n + h] = 0.3 * 2.0;
  if (has_off) {
    CZ_CUDA(cudaMemcpyAsync(b->d_off_stage, b->h_off_stage, sizeof(double) * 12 * n, cudaMemcpyHostToDevice,
                            b->stream));
  }
  b->lin_damp.assign(in->linear_damping, in->linear_damping + n);
  b->ang_damp.assign(in->angular_damping, in->angular_damping + n);
  b->pow_dt = std::nan("");
  // the blocks the caller gave: all up to SG_IW, and the last two
  auto send = [&](int blk, int width) {
    const long long at = (long long)blk * n;
    return cudaMemcpyAsync(b->d_stage + at, sg + at, sizeof(double) * width * n, cudaMemcpyHostToDevice, b->stream);
  };
  CZ_CUDA(send(0, cz::SG_IW));
  if (has_iw) CZ_CUDA(send(cz::SG_IW, 9));
  if (has_lfa) CZ_CUDA(send(cz::SG_LFA, 3));
  CZ_CUDA(cudaMemcpyAsync(b->d_stage_u8, b->h_stage_u8, 2 * n, cudaMemcpyHostToDevice, b->stream));
  CZ_CUDA(cudaMemcpyAsync(b->d_stage_i32, b->h_stage_i32, sizeof(int) * n, cudaMemcpyHostToDevice, b->stream));
  CZ_CUDA(b->ops->upload(b->view(), b->d_stage, b->d_stage_u8, b->d_stage_i32, b->d_h2p, (int)n, has_iw, has_lfa,
                         has_off ? b->d_off_stage : nullptr, b->stream));
  g_launches++;
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  return CZ_OK;
}

int cz_download_bodies(cz_batch* b, cz_bodies* out) {
  if (!b || !out) return fail(CZ_ERR_BAD_ARG, "cz_download_bodies: null argument");
  CZ_CUDA(cudaSetDevice(b->device));
  const long long n = b->nb;
  if (n == 0) return CZ_OK;
  const bool want_off = out->collider_offset && b->has_offset;
  CZ_CUDA(b->ops->download(b->view(), b->d_stage, b->d_stage_u8, b->d_stage_i32, b->d_h2p, (int)n,
                           want_off ? b->d_off_stage : nullptr, b->stream));
  g_launches++;
  if (want_off)
    CZ_CUDA(cudaMemcpyAsync(b->h_off_stage, b->d_off_stage, sizeof(double) * 12 * n, cudaMemcpyDeviceToHost,
                            b->stream));
  // only the blocks the caller wants, in one copy where what lies between is short
  const struct {
    int blk, width;
    double* dst;
  } fields[] = {{cz::SG_POS, 3, out->position},        {cz::SG_Q, 4, out->orientation},
                {cz::SG_VEL, 3, out->velocity},        {cz::SG_ROT, 3, out->rotation},
                {cz::SG_ACC, 3, out->acceleration},    {cz::SG_IB, 9, out->inverse_inertia},
                {cz::SG_INVM, 1, out->inverse_mass},   {cz::SG_MOTION, 1, out->motion},
                {cz::SG_HALF, 3, out->half_size},      {cz::SG_RAD, 1, out->radius},
                {cz::SG_IW, 9, out->inverse_inertia_world},
                {cz::SG_LFA, 3, out->last_frame_acceleration}};
  HostCopies list;
  int first = 0, next = 0;  // blocks [first, next) are still to be copied
  auto fetch = [&]() {
    const long long at = (long long)first * n;
    if (first == next) return cudaSuccess;
    return cudaMemcpyAsync(b->h_stage + at, b->d_stage + at, sizeof(double) * (next - first) * n,
                           cudaMemcpyDeviceToHost, b->stream);
  };
  for (const auto& f : fields) {
    if (!f.dst) continue;
    list.add(f.dst, b->h_stage + (long long)f.blk * n, sizeof(double) * f.width * n);
    if (sizeof(double) * (f.blk - next) * n > 32768) {
      CZ_CUDA(fetch());
      first = f.blk;
    }
    next = f.blk + f.width;
  }
  CZ_CUDA(fetch());
  if (out->is_awake || out->can_sleep)
    CZ_CUDA(cudaMemcpyAsync(b->h_stage_u8, b->d_stage_u8, 2 * n, cudaMemcpyDeviceToHost, b->stream));
  if (out->shape)
    CZ_CUDA(cudaMemcpyAsync(b->h_stage_i32, b->d_stage_i32, sizeof(int) * n, cudaMemcpyDeviceToHost, b->stream));
  if (out->linear_damping) list.add(out->linear_damping, b->lin_damp.data(), sizeof(double) * n);
  if (out->angular_damping) list.add(out->angular_damping, b->ang_damp.data(), sizeof(double) * n);
  if (out->is_awake) list.add(out->is_awake, b->h_stage_u8, (size_t)n);
  if (out->can_sleep) list.add(out->can_sleep, b->h_stage_u8 + n, (size_t)n);
  if (out->shape) list.add(out->shape, b->h_stage_i32, sizeof(int) * n);
  if (want_off) list.add(out->collider_offset, b->h_off_stage, sizeof(double) * 12 * n);
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  host_copy(list);
  if (out->collider_offset && !want_off) {
    static const double id[12] = {1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0};
    for (long long h = 0; h < n; ++h) std::memcpy(out->collider_offset + 12 * h, id, sizeof id);
  }
  return CZ_OK;
}

int cz_integrate(cz_batch* b, double dt) {
  if (!b) return fail(CZ_ERR_BAD_ARG, "cz_integrate: null batch");
  CZ_CUDA(cudaSetDevice(b->device));
  int st = ensure_pows(b, dt);
  if (st) return st;
  if ((st = reset_status(b))) return st;
  if ((st = launch_integrate(b, whole(b), dt))) return st;
  return finish(b);
}

int cz_narrowphase(cz_batch* b) {
  if (!b) return fail(CZ_ERR_BAD_ARG, "cz_narrowphase: null batch");
  CZ_CUDA(cudaSetDevice(b->device));
  int st = reset_status(b);
  if (st) return st;
  if ((st = launch_narrowphase(b, whole(b), true))) return st;
  return finish(b);
}

int cz_resolve(cz_batch* b, double dt) {
  if (!b) return fail(CZ_ERR_BAD_ARG, "cz_resolve: null batch");
  CZ_CUDA(cudaSetDevice(b->device));
  int st = reset_status(b);
  if (st) return st;
  if ((st = launch_resolve(b, whole(b), dt, true))) return st;
  return finish(b);
}

// The end of a phase in a part's chain of a timed rollout: the time, appended to
// the part's log.  With event nodes the branches of a graph did not run side by
// side: 4096 worlds of 32 bodies x 60 frames, float64, 137 ms by cz_step, 138.6
// timed so, 142 to 280 with events in 4 to 32 of the 32 parts; 4096 of 8 to 64
// bodies x 600 frames 2177, 2167 and 2620 and more.
__global__ void k_stamp(unsigned long long* log, size_t cap) {
  unsigned long long now;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
  const unsigned long long at = log[0];
  if (at < cap) log[1 + at] = now;
  log[0] = at + 1;
}

// What a timed rollout leaves between the phases of a chain (an untimed one:
// nothing).
struct Marks {
  const std::vector<cudaEvent_t>* ev = nullptr;
  unsigned long long* log = nullptr;
  size_t cap = 0, next = 0;
  int mark(cudaStream_t s) {
    if (ev) CZ_CUDA(cudaEventRecordWithFlags((*ev)[next++], s, cudaEventRecordExternal));
    if (log) {
      k_stamp<<<1, 1, 0, s>>>(log, cap);
      CZ_CUDA(cudaGetLastError());
    }
    return CZ_OK;
  }
};

// One frame of a chain.
static int launch_step(cz_batch* b, const Chain& c, double dt, Marks* m = nullptr) {
  Marks none;
  if (!m) m = &none;
  int st = launch_integrate(b, c, dt);
  if (!st) st = m->mark(c.s);
  if (!st) st = launch_narrowphase(b, c, false);
  if (!st) st = m->mark(c.s);
  if (!st) st = launch_resolve(b, c, dt, false);
  if (!st) st = m->mark(c.s);
  return st;
}
static int launch_chain(cz_batch* b, const Chain& c, int nsteps, double dt, Marks m) {
  int st = m.mark(c.s);
  for (int s = 0; s < nsteps && !st; ++s) st = launch_step(b, c, dt, &m);
  return st;
}

// The parts whose chains a timed rollout marks: every so many, the first kTimedParts of them.
static int timed_parts(const cz_batch* b) { return std::min((int)b->parts.size(), kTimedParts); }

// The batch's parts as parallel branches of the graph being captured on its
// stream, each its own chain of frames.
static int capture_parts(cz_batch* b, int nsteps, double dt, bool timed) {
  cudaEvent_t fork = nullptr;
  std::vector<cudaEvent_t> joins;
  auto run = [&]() -> int {
    CZ_CUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    CZ_CUDA(cudaEventRecord(fork, b->stream));
    for (size_t p = 0; p < b->parts.size(); ++p) {
      const cz_batch::Part& part = b->parts[p];
      const Chain c{b->view(part, (int)p), part.nsmall, part.nbig, part.nsmall > kReorderWorlds,
                    p == 0 ? b->stream : b->part_streams[p - 1]};
      if (p > 0) CZ_CUDA(cudaStreamWaitEvent(c.s, fork, 0));
      const size_t every = b->parts.size() / timed_parts(b), index = p / every;
      Marks m;
      if (timed && p % every == 0 && index < (size_t)timed_parts(b)) {
        m.log = b->stamps + index * (1 + b->stamp_cap);
        m.cap = b->stamp_cap;
      }
      if (int st = launch_chain(b, c, nsteps, dt, m)) return st;
      if (p > 0) {
        cudaEvent_t e = nullptr;
        CZ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        joins.push_back(e);
        CZ_CUDA(cudaEventRecord(e, c.s));
      }
    }
    for (cudaEvent_t e : joins) CZ_CUDA(cudaStreamWaitEvent(b->stream, e, 0));
    return CZ_OK;
  };
  const int st = run();
  if (fork) cudaEventDestroy(fork);
  for (cudaEvent_t e : joins) cudaEventDestroy(e);
  return st;
}

// Frames the next graph of a rollout with `left` frames to go holds.
static int graph_frames(const cz_batch* b, int left) { return in_parts(b) ? std::min(left, kPartFrames) : left; }

// A rollout's launches, on the batch's stream: the fused frames, the parts, or
// one chain over the whole batch.  With `t`, the marks between its phases (a
// fused frame, one launch, is its resolve phase).
static int launch_rollout(cz_batch* b, int nsteps, double dt, const cz_batch::Timed* t) {
  if (in_parts(b)) return capture_parts(b, nsteps, dt, t != nullptr);
  Marks m;
  if (t) m.ev = &t->ev;
  if (!uses_frame(b)) return launch_chain(b, whole(b), nsteps, dt, m);
  int st = m.mark(b->stream);
  for (int s = 0; s < nsteps && !st; ++s) {
    st = m.mark(b->stream);
    if (!st) st = m.mark(b->stream);
    if (!st) st = launch_frame(b, dt);
    if (!st) st = m.mark(b->stream);
  }
  return st;
}

static int capture_rollout(cz_batch* b, int nsteps, double dt, const cz_batch::Timed* t, cudaGraphExec_t* exec) {
  CZ_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
  const long long before = g_launches.load();
  const int cst = launch_rollout(b, nsteps, dt, t);
  g_launches.store(before);  // captured launches are counted when the graph runs
  cudaGraph_t graph = nullptr;
  cudaError_t e = cudaStreamEndCapture(b->stream, &graph);
  if (cst != CZ_OK || e != cudaSuccess) {
    if (graph) cudaGraphDestroy(graph);
    return cst != CZ_OK ? cst : fail(CZ_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e));
  }
  e = cudaGraphInstantiate(exec, graph, 0);
  cudaGraphDestroy(graph);
  if (e != cudaSuccess) return fail(CZ_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e));
  return CZ_OK;
}

// Capture (once per (nsteps, dt)) the plain rollout graph.
static int get_graph(cz_batch* b, int nsteps, double dt, cudaGraphExec_t* out) {
  auto key = std::make_pair(nsteps, dt);
  auto it = b->graphs.find(key);
  if (it != b->graphs.end()) {
    *out = it->second;
    return CZ_OK;
  }
  if (int st = capture_rollout(b, nsteps, dt, nullptr, out)) return st;
  b->graphs.emplace(key, *out);
  return CZ_OK;
}

// The same graph with marks around every phase.
static int get_timed(cz_batch* b, int nsteps, double dt, cz_batch::Timed** out) {
  auto key = std::make_pair(nsteps, dt);
  auto it = b->timed.find(key);
  if (it != b->timed.end()) {
    *out = &it->second;
    return CZ_OK;
  }
  cz_batch::Timed t;
  if (!in_parts(b)) t.ev.resize(3 * (size_t)nsteps + 1);
  cudaError_t e = cudaSuccess;
  for (size_t k = 0; k < t.ev.size() && e == cudaSuccess; ++k) e = cudaEventCreate(&t.ev[k]);
  int st = e == cudaSuccess ? capture_rollout(b, nsteps, dt, &t, &t.exec)
                            : fail(CZ_ERR_CUDA, std::string("event: ") + cudaGetErrorString(e));
  if (st) {
    for (cudaEvent_t ev : t.ev)
      if (ev) cudaEventDestroy(ev);
    return st;
  }
  *out = &b->timed.emplace(key, std::move(t)).first->second;
  return CZ_OK;
}

// Room in the log for the marks of a rollout of nsteps frames: three a frame, and
// one a graph.  The graphs hold its address, so those of a shorter one go.
static int ensure_stamps(cz_batch* b, int nsteps) {
  const size_t need = 3 * (size_t)nsteps + ((size_t)nsteps + kPartFrames - 1) / kPartFrames;
  if (!in_parts(b) || need <= b->stamp_cap) return CZ_OK;
  drop_timed(b);
  CZ_CUDA(cudaFree(b->stamps));
  b->stamps = nullptr;
  b->stamp_cap = 0;
  CZ_CUDA(cudaMalloc((void**)&b->stamps, sizeof(unsigned long long) * kTimedParts * (1 + need)));
  b->stamp_cap = need;
  return CZ_OK;
}

int cz_step(cz_batch* b, int32_t nsteps, double dt) {
  if (!b || nsteps < 0) return fail(CZ_ERR_BAD_ARG, "cz_step: bad argument");
  if (nsteps == 0) return CZ_OK;
  CZ_CUDA(cudaSetDevice(b->device));
  int st = ensure_pows(b, dt);
  if (st) return st;
  if ((st = reset_status(b))) return st;
  for (int left = nsteps; left > 0;) {
    const int n = graph_frames(b, left);
    cudaGraphExec_t exec = nullptr;
    if ((st = get_graph(b, n, dt, &exec))) return st;
    CZ_CUDA(cudaGraphLaunch(exec, b->stream));
    left -= n;
  }
  g_launches += (long long)launches_per_step(b) * nsteps;
  return finish(b);
}

int cz_prepare_rollout(cz_batch* b, int32_t nsteps, double dt) {
  if (!b || nsteps <= 0) return fail(CZ_ERR_BAD_ARG, "cz_prepare_rollout: bad argument");
  CZ_CUDA(cudaSetDevice(b->device));
  int st = ensure_pows(b, dt);
  if (st) return st;
  if ((st = ensure_stamps(b, nsteps))) return st;
  for (int n : {graph_frames(b, nsteps), nsteps % graph_frames(b, nsteps)}) {
    cudaGraphExec_t exec = nullptr;
    cz_batch::Timed* t = nullptr;
    if (n > 0 && ((st = get_graph(b, n, dt, &exec)) || (st = get_timed(b, n, dt, &t)))) return st;
  }
  return CZ_OK;
}

int cz_contact_counts(cz_batch* b, int32_t* counts) {
  if (!b || !counts) return fail(CZ_ERR_BAD_ARG, "cz_contact_counts: null argument");
  CZ_CUDA(cudaSetDevice(b->device));
  CZ_CUDA(cudaMemcpyAsync(counts, b->d_ccount, sizeof(int) * b->num_worlds, cudaMemcpyDeviceToHost, b->stream));
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  return CZ_OK;
}

int cz_download_contacts(cz_batch* b, int32_t world, cz_contact* out, int32_t capacity, int32_t* count) {
  if (!b || world < 0 || world >= b->num_worlds || (capacity > 0 && !out))
    return fail(CZ_ERR_BAD_ARG, "cz_download_contacts: bad argument");
  CZ_CUDA(cudaSetDevice(b->device));
  int n = 0;
  CZ_CUDA(cudaMemcpyAsync(&n, b->d_ccount + world, sizeof(int), cudaMemcpyDeviceToHost, b->stream));
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  if (count) *count = n;
  int m = std::min(n, b->ccap[world]);
  m = std::min(m, std::max(capacity, 0));
  if (m <= 0) return n > b->ccap[world] ? fail(CZ_ERR_CAPACITY, "world exceeded its contact capacity") : CZ_OK;
  CZ_CUDA(b->ops->contacts_out(b->view(), b->cstart[world], m, b->d_cstage, b->d_cstage_b, b->stream));
  g_launches++;
  CZ_CUDA(cudaMemcpyAsync(b->h_cstage, b->d_cstage, sizeof(double) * cz::C_NROWS * m, cudaMemcpyDeviceToHost,
                          b->stream));
  CZ_CUDA(cudaMemcpyAsync(b->h_cstage_b, b->d_cstage_b, sizeof(int) * m, cudaMemcpyDeviceToHost, b->stream));
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  for (int k = 0; k < m; ++k) {
    const double* c = b->h_cstage + (long long)k * cz::C_NROWS;
    cz_contact& o = out[k];
    o.body[0] = cz::body0_of(b->h_cstage_b[k]);
    o.body[1] = cz::body1_of(b->h_cstage_b[k]);
    o.point[0] = c[cz::C_PX]; o.point[1] = c[cz::C_PY]; o.point[2] = c[cz::C_PZ];
    o.normal[0] = c[cz::C_NX]; o.normal[1] = c[cz::C_NY]; o.normal[2] = c[cz::C_NZ];
    o.penetration = c[cz::C_PEN];
    o.friction = c[cz::C_FRIC];
    o.restitution = c[cz::C_REST];
  }
  if (n > b->ccap[world]) return fail(CZ_ERR_CAPACITY, "world exceeded its contact capacity");
  return CZ_OK;
}

int cz_world_stats(cz_batch* b, int32_t* pos_it, int32_t* vel_it, uint32_t* status) {
  if (!b) return fail(CZ_ERR_BAD_ARG, "cz_world_stats: null batch");
  CZ_CUDA(cudaSetDevice(b->device));
  const size_t W = b->num_worlds;
  if (pos_it) CZ_CUDA(cudaMemcpyAsync(pos_it, b->d_piters, sizeof(int) * W, cudaMemcpyDeviceToHost, b->stream));
  if (vel_it) CZ_CUDA(cudaMemcpyAsync(vel_it, b->d_viters, sizeof(int) * W, cudaMemcpyDeviceToHost, b->stream));
  if (status) CZ_CUDA(cudaMemcpyAsync(status, b->d_wstatus, sizeof(uint32_t) * W, cudaMemcpyDeviceToHost, b->stream));
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  return CZ_OK;
}

int cz_resolve_contacts(cz_batch* b, int32_t max_iterations, cz_contact* contacts, int32_t ncontacts,
                        double duration, cz_bodies* bodies) {
  if (!b || !bodies || ncontacts < 0 || (ncontacts > 0 && !contacts))
    return fail(CZ_ERR_BAD_ARG, "cz_resolve_contacts: bad argument");
  if (b->num_worlds != 1) return fail(CZ_ERR_BAD_ARG, "cz_resolve_contacts: the batch must hold one world");
  if (ncontacts > b->ccap[0]) return fail(CZ_ERR_CAPACITY, "cz_resolve_contacts: more contacts than capacity");
  // ResolveContacts' own guards (contact.go:210-212): nothing changes
  if (duration <= 0.0 || ncontacts == 0) return CZ_OK;
  const int n = b->counts[0];
  for (int k = 0; k < ncontacts; ++k) {
    const int b0 = contacts[k].body[0], b1 = contacts[k].body[1];
    if (b0 < -1 || b0 >= n || b1 < -1 || b1 >= n || (b0 < 0 && b1 < 0))
      return fail(CZ_ERR_BAD_ARG, "cz_resolve_contacts: contact body index out of range");
  }
  int st = cz_upload_bodies(b, bodies);
  if (st) return st;
  CZ_CUDA(cudaSetDevice(b->device));
  for (int k = 0; k < ncontacts; ++k) {
    double* c = b->h_cstage + (long long)k * cz::C_NROWS;
    const cz_contact& s = contacts[k];
    c[cz::C_PX] = s.point[0]; c[cz::C_PY] = s.point[1]; c[cz::C_PZ] = s.point[2];
    c[cz::C_NX] = s.normal[0]; c[cz::C_NY] = s.normal[1]; c[cz::C_NZ] = s.normal[2];
    c[cz::C_PEN] = s.penetration;
    c[cz::C_FRIC] = s.friction;
    c[cz::C_REST] = s.restitution;
    b->h_cstage_b[k] = cz::pack_bodies(s.body[0], s.body[1]);
  }
  CZ_CUDA(cudaMemcpyAsync(b->d_cstage, b->h_cstage, sizeof(double) * cz::C_NROWS * ncontacts, cudaMemcpyHostToDevice,
                          b->stream));
  CZ_CUDA(cudaMemcpyAsync(b->d_cstage_b, b->h_cstage_b, sizeof(int) * ncontacts, cudaMemcpyHostToDevice, b->stream));
  CZ_CUDA(b->ops->contacts_in(b->view(), b->cstart[0], ncontacts, b->d_cstage, b->d_cstage_b, b->stream));
  g_launches++;
  CZ_CUDA(cudaMemcpyAsync(b->d_ccount, &ncontacts, sizeof(int), cudaMemcpyHostToDevice, b->stream));
  if ((st = reset_status(b))) return st;
  Chain c = whole(b);
  c.v.max_iterations = std::max(max_iterations, 0);
  c.v.contact_writeback = 1;
  c.v.uniform_material = 0;
  if ((st = launch_resolve(b, c, duration, true))) return st;
  st = finish(b);
  if (st != CZ_OK && st != CZ_ERR_FRICTIONLESS) return st;
  const int st2 = cz_download_bodies(b, bodies);
  if (st2) return st2;
  // write the resolved contacts back (penetration, swapped bodies/normal)
  CZ_CUDA(b->ops->contacts_out(b->view(), b->cstart[0], ncontacts, b->d_cstage, b->d_cstage_b, b->stream));
  g_launches++;
  CZ_CUDA(cudaMemcpyAsync(b->h_cstage, b->d_cstage, sizeof(double) * cz::C_NROWS * ncontacts, cudaMemcpyDeviceToHost,
                          b->stream));
  CZ_CUDA(cudaMemcpyAsync(b->h_cstage_b, b->d_cstage_b, sizeof(int) * ncontacts, cudaMemcpyDeviceToHost, b->stream));
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  for (int k = 0; k < ncontacts; ++k) {
    const double* c = b->h_cstage + (long long)k * cz::C_NROWS;
    contacts[k].body[0] = cz::body0_of(b->h_cstage_b[k]);
    contacts[k].body[1] = cz::body1_of(b->h_cstage_b[k]);
    contacts[k].normal[0] = c[cz::C_NX];
    contacts[k].normal[1] = c[cz::C_NY];
    contacts[k].normal[2] = c[cz::C_NZ];
    contacts[k].penetration = c[cz::C_PEN];
  }
  return st;
}

int cz_snapshot(cz_batch* b) {
  if (!b) return fail(CZ_ERR_BAD_ARG, "cz_snapshot: null batch");
  CZ_CUDA(cudaSetDevice(b->device));
  const size_t bytes = b->ops->real_size * cz::B_NROWS * b->nb_pad;
  CZ_CUDA(cudaMemcpyAsync(b->snap_body, b->body, bytes, cudaMemcpyDeviceToDevice, b->stream));
  CZ_CUDA(cudaMemcpyAsync(b->snap_u8, b->awake, b->nb_pad, cudaMemcpyDeviceToDevice, b->stream));
  CZ_CUDA(cudaMemcpyAsync(b->snap_u8 + b->nb_pad, b->can_sleep, b->nb_pad, cudaMemcpyDeviceToDevice, b->stream));
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  b->snap_pow_dt = b->pow_dt;
  return CZ_OK;
}

int cz_restore(cz_batch* b) {
  if (!b) return fail(CZ_ERR_BAD_ARG, "cz_restore: null batch");
  CZ_CUDA(cudaSetDevice(b->device));
  const size_t bytes = b->ops->real_size * cz::B_NROWS * b->nb_pad;
  CZ_CUDA(cudaMemcpyAsync(b->body, b->snap_body, bytes, cudaMemcpyDeviceToDevice, b->stream));
  CZ_CUDA(cudaMemcpyAsync(b->awake, b->snap_u8, b->nb_pad, cudaMemcpyDeviceToDevice, b->stream));
  CZ_CUDA(cudaMemcpyAsync(b->can_sleep, b->snap_u8 + b->nb_pad, b->nb_pad, cudaMemcpyDeviceToDevice, b->stream));
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  b->pow_dt = b->snap_pow_dt;  // the snapshot holds the damping factors of its own dt
  return CZ_OK;
}

int cz_step_timed(cz_batch* b, int32_t nsteps, double dt, double* total_ms, double* phase_ms) {
  if (!b || nsteps <= 0) return fail(CZ_ERR_BAD_ARG, "cz_step_timed: bad argument");
  CZ_CUDA(cudaSetDevice(b->device));
  int st = ensure_pows(b, dt);
  if (st) return st;
  if ((st = reset_status(b))) return st;
  const bool fused = uses_frame(b), parts = in_parts(b);
  if ((st = ensure_stamps(b, nsteps))) return st;
  for (cudaEvent_t& e : b->roll_ev)
    if (parts && !e) CZ_CUDA(cudaEventCreate(&e));
  if (parts) {
    CZ_CUDA(cudaMemset2DAsync(b->stamps, sizeof(*b->stamps) * (1 + b->stamp_cap), 0, sizeof(*b->stamps), kTimedParts,
                              b->stream));
    CZ_CUDA(cudaEventRecord(b->roll_ev[0], b->stream));
  }
  cz_batch::Timed* t = nullptr;
  for (int left = nsteps; left > 0;) {
    const int n = graph_frames(b, left);
    if ((st = get_timed(b, n, dt, &t))) return st;
    CZ_CUDA(cudaGraphLaunch(t->exec, b->stream));
    left -= n;
  }
  if (parts) CZ_CUDA(cudaEventRecord(b->roll_ev[1], b->stream));
  g_launches += (long long)launches_per_step(b) * nsteps;
  st = finish(b);
  float ms = 0.f;
  double tot = 0, ph[3] = {0, 0, 0};
  if (parts) {
    CZ_CUDA(cudaEventElapsedTime(&ms, b->roll_ev[0], b->roll_ev[1]));
    tot = ms;
    // the parts overlap: their phases' times are shares of the rollout's
    const size_t row = 1 + b->stamp_cap;
    std::vector<unsigned long long> log(timed_parts(b) * row);
    CZ_CUDA(cudaMemcpy(log.data(), b->stamps, sizeof(log[0]) * log.size(), cudaMemcpyDeviceToHost));
    for (size_t p = 0; p < log.size(); p += row) {
      const unsigned long long* at = &log[p + 1];
      for (int left = nsteps; left > 0; ++at) {  // (a graph's first mark)
        const int n = graph_frames(b, left);
        for (int k = 0; k < 3 * n; ++k, ++at) ph[k % 3] += (double)(at[1] - at[0]);
        left -= n;
      }
    }
    const double sum = ph[0] + ph[1] + ph[2];
    for (double& x : ph) x = sum > 0 ? x * tot / sum : 0;
  } else {
    for (size_t k = 0; k + 1 < t->ev.size(); ++k) {
      CZ_CUDA(cudaEventElapsedTime(&ms, t->ev[k], t->ev[k + 1]));
      // a fused frame, with the gaps between its event nodes, is all resolve
      ph[fused ? 2 : k % 3] += ms;
    }
    CZ_CUDA(cudaEventElapsedTime(&ms, t->ev.front(), t->ev.back()));
    tot = ms;
  }
  if (total_ms) *total_ms = tot;
  if (phase_ms)
    for (int k = 0; k < 3; ++k) phase_ms[k] = ph[k];
  return st;
}

// The per-body scratch of the warm start and the harvest.
static int ensure_ws(cz_batch* b) {
  if (b->ws_rows) return CZ_OK;
  const size_t P = (size_t)b->nb_pad;
  CZ_CUDA(cudaMalloc(&b->ws_rows, b->ops->real_size * 6 * P));
  CZ_CUDA(cudaMalloc(&b->ws_imp, b->ops->real_size * 3 * (size_t)b->nc_total));
  CZ_CUDA(cudaMalloc((void**)&b->ws_int, sizeof(int) * cz::WS_NINT * P));
  CZ_CUDA(cudaMalloc((void**)&b->ws_world, (size_t)b->num_worlds));
  CZ_CUDA(cudaMemset(b->ws_world, 0, (size_t)b->num_worlds));
  return CZ_OK;
}

int cz_collide(cz_batch* b, int32_t world, const double* plane, const int32_t* units, int32_t nunits) {
  if (!b || world < 0 || world >= b->num_worlds || nunits < 0 || (nunits > 0 && !units))
    return fail(CZ_ERR_BAD_ARG, "cz_collide: bad argument");
  const int n = b->counts[world];
  for (int u = 0; u < nunits; ++u) {
    const int i = units[2 * u], j = units[2 * u + 1];
    if (i < 0 || i >= n || j < -1 || j >= n || j == i)
      return fail(CZ_ERR_BAD_ARG, "cz_collide: unit " + std::to_string(u) + " is not (body, other body or -1)");
  }
  CZ_CUDA(cudaSetDevice(b->device));
  if (nunits > b->units_cap) {
    cudaFree(b->d_units);
    b->d_units = nullptr;
    b->units_cap = 0;
    CZ_CUDA(cudaMalloc((void**)&b->d_units, sizeof(int) * 2 * (size_t)nunits));
    b->units_cap = nunits;
  }
  if (nunits > 0)
    CZ_CUDA(cudaMemcpyAsync(b->d_units, units, sizeof(int) * 2 * (size_t)nunits, cudaMemcpyHostToDevice, b->stream));
  int st = reset_status(b);
  if (st) return st;
  cz::HostView v = b->view();
  if (plane)
    for (int k = 0; k < 4; ++k) v.plane[k] = plane[k];
  CZ_CUDA(b->ops->collide(v, world, b->d_units, nunits, b->nbs, b->np_smem, b->stream));
  g_launches++;
  return finish(b);
}

int cz_set_warm_start(cz_batch* b, const float* blob) {
  if (!b) return fail(CZ_ERR_BAD_ARG, "cz_set_warm_start: null batch");
  CZ_CUDA(cudaSetDevice(b->device));
  if (!blob) {
    b->mode = 0;
    return configure(b);
  }
  if (int st = ensure_ws(b)) return st;
  const size_t blob_bytes = sizeof(float) * cz::MLP_BLOB;
  const size_t off = (blob_bytes + 255) & ~(size_t)255;
  if (!b->mlp_mem) CZ_CUDA(cudaMalloc(&b->mlp_mem, off + cz::mlp_packed_bytes()));
  unsigned char* mem = static_cast<unsigned char*>(b->mlp_mem);
  CZ_CUDA(cudaMemcpyAsync(mem, blob, blob_bytes, cudaMemcpyHostToDevice, b->stream));
  CZ_CUDA(cz::mlp_pack(reinterpret_cast<const float*>(mem), mem + off, b->stream));
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  b->mlp = cz::mlp_view(mem + off);
  b->mode = 2;
  return configure(b);
}

int cz_harvest(cz_batch* b, int32_t nsteps, double dt, int32_t every, float* features, float* labels,
               int64_t capacity, int64_t* count) {
  if (!b || nsteps < 0 || every <= 0 || capacity < 0 || (capacity > 0 && (!features || !labels)))
    return fail(CZ_ERR_BAD_ARG, "cz_harvest: bad argument");
  CZ_CUDA(cudaSetDevice(b->device));
  if (capacity > b->hv_cap) {
    cudaFree(b->hv_features);
    cudaFree(b->hv_labels);
    b->hv_features = b->hv_labels = nullptr;
    b->hv_cap = 0;
    CZ_CUDA(cudaMalloc((void**)&b->hv_features, sizeof(float) * cz::MLP_IN * std::max<int64_t>(capacity, 1)));
    CZ_CUDA(cudaMalloc((void**)&b->hv_labels, sizeof(float) * cz::MLP_OUT * std::max<int64_t>(capacity, 1)));
    b->hv_cap = capacity;
  }
  if (!b->hv_count) CZ_CUDA(cudaMalloc((void**)&b->hv_count, sizeof(unsigned long long)));
  if (int st0 = ensure_ws(b)) return st0;
  if (!b->ws_feat) CZ_CUDA(cudaMalloc((void**)&b->ws_feat, sizeof(float) * cz::MLP_IN * (size_t)b->nc_total));
  CZ_CUDA(cudaMemsetAsync(b->hv_count, 0, sizeof(unsigned long long), b->stream));
  int st = ensure_pows(b, dt);
  if (st) return st;
  if ((st = reset_status(b))) return st;
  // the plain resolver, writing features and applied impulses every `every` frames
  const int saved_mode = b->mode;
  for (int s = 0; s < nsteps && st == CZ_OK; ++s) {
    Chain c = whole(b);
    c.v.mode = (s % every) == every - 1 ? 1 : 0;
    c.v.hv_cap = b->hv_cap;
    st = launch_step(b, c, dt);
  }
  b->mode = saved_mode;
  if (st) return st;
  st = finish(b);
  unsigned long long n = 0;
  CZ_CUDA(cudaMemcpy(&n, b->hv_count, sizeof n, cudaMemcpyDeviceToHost));
  const int64_t m = std::min<int64_t>((int64_t)n, capacity);
  if (m > 0) {
    CZ_CUDA(cudaMemcpy(features, b->hv_features, sizeof(float) * cz::MLP_IN * m, cudaMemcpyDeviceToHost));
    CZ_CUDA(cudaMemcpy(labels, b->hv_labels, sizeof(float) * cz::MLP_OUT * m, cudaMemcpyDeviceToHost));
  }
  if (count) *count = m;
  return st;
}

int cz_counters(cz_batch* b, int64_t* out, int32_t reset) {
  if (!b) return fail(CZ_ERR_BAD_ARG, "cz_counters: null batch");
  CZ_CUDA(cudaSetDevice(b->device));
  unsigned long long c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  CZ_CUDA(cudaMemcpyAsync(c, b->d_counters, sizeof c, cudaMemcpyDeviceToHost, b->stream));
  if (reset) CZ_CUDA(cudaMemsetAsync(b->d_counters, 0, sizeof c, b->stream));
  CZ_CUDA(cudaStreamSynchronize(b->stream));
  if (out)
    for (int i = 0; i < 8; ++i) out[i] = (int64_t)c[i];
  return CZ_OK;
}

int cz_batch_info(cz_batch* b, int64_t* info) {
  if (!b || !info) return fail(CZ_ERR_BAD_ARG, "cz_batch_info: null argument");
  info[0] = b->nb;
  info[1] = b->nb_pad;
  info[2] = b->nc_total;
  info[3] = (int64_t)b->ops->real_size;
  info[4] = b->sm_count;
  info[5] = b->np_grid;
  const bool wide = uses_wide(b, b->mode);
  info[6] = wide ? b->wide_grid : b->rs_grid;
  info[7] = (int64_t)b->np_smem;
  info[8] = (int64_t)(wide ? b->wide_smem : b->rs_wpc * b->rs_smem);
  return CZ_OK;
}

}  // extern "C"
