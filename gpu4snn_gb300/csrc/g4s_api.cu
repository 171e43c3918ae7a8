// g4s_api.cu — the C ABI (include/gpu4snn.h): network handles, the chunked step loop, the
// reference's result files and its experiment sweep.
//
// A run is executed in chunks of at most `chunk_steps` steps; a chunk's spike ids go to a
// device raster buffer sized so that every neuron could fire at every step of the chunk
// (or of the run, if that is shorter), so it can never overflow.  After each chunk the per-step counts, raster offsets and
// globaltimer stamps come back to the host (and the raster, when it is recorded).
#include <cuda_runtime.h>
#include <sys/stat.h>

#include <algorithm>
#include <atomic>
#include <cerrno>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <cmath>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "../../include/gpu4snn.h"
#include "g4s_internal.h"

using namespace g4s;

// ---------------------------------------------------------------------------------------
// Errors.
// ---------------------------------------------------------------------------------------
static thread_local std::string g_last_error;

namespace g4s {
int set_error(int code, const std::string &msg) {
  g_last_error = msg;
  return code;
}
int cuda_error(cudaError_t e, const char *what) {
  return set_error(e == cudaErrorMemoryAllocation ? G4S_ERR_NOMEM : G4S_ERR_CUDA,
                   std::string(what) + ": " + cudaGetErrorString(e));
}
}  // namespace g4s

#define G4S_CUDA(call)                                  \
  do {                                                  \
    cudaError_t e_ = (call);                            \
    if (e_ != cudaSuccess) return cuda_error(e_, #call); \
  } while (0)

// Buffers of the launches of one handle, or of one thread's batches: what a round uploads
// (descriptors, the networks' places in the pack, queue slots and head: one copy) and
// the pack that it brings back, each side one allocation.
struct TeamLaunch {
  unsigned char *d_mem = nullptr, *h_mem = nullptr;
  size_t cap = 0;
  // the round's parts, at the same offsets on both sides
  size_t o_off = 0, o_slots = 0, o_head = 0, o_pack = 0;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  std::vector<int> order;  // networks of the round in flight (team_round_start .. finish)
  std::vector<g4s_net *> nets;
  std::vector<int> steps;
  std::vector<size_t> at;  // per network: its share of the pack
  TeamLaunch() = default;
  TeamLaunch(const TeamLaunch &) = delete;
  TeamLaunch &operator=(const TeamLaunch &) = delete;
  ~TeamLaunch() { release(); }  // (a thread's own launch buffers go when the thread ends)
  void release() {
    cudaFree(d_mem);
    cudaFreeHost(h_mem);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    d_mem = h_mem = nullptr;
    cap = 0;
    e0 = e1 = nullptr;
    order.clear();
  }
  int reserve(int items, int slots, size_t pack) {
    if (!e0 && (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess))
      return set_error(G4S_ERR_CUDA, "team launch events");
    o_off = sizeof(TeamItem) * (size_t)items;
    o_slots = o_off + sizeof(int64_t) * (size_t)items;
    o_head = o_slots + sizeof(int2) * (size_t)slots;
    o_pack = (o_head + 16 + 15) / 16 * 16;
    const size_t bytes = o_pack + pack;
    if (bytes <= cap) return G4S_OK;
    cudaFree(d_mem);
    cudaFreeHost(h_mem);
    d_mem = h_mem = nullptr;
    const size_t want = std::max({bytes, 2 * cap, (size_t)1 << 16});
    cap = 0;  // (until the new buffers exist)
    if (cudaMalloc((void **)&d_mem, want) != cudaSuccess || cudaMallocHost((void **)&h_mem, want) != cudaSuccess)
      return set_error(G4S_ERR_NOMEM, "team launch buffers");
    cap = want;
    return G4S_OK;
  }
  TeamItem *items(unsigned char *m) const { return reinterpret_cast<TeamItem *>(m); }
  int64_t *off(unsigned char *m) const { return reinterpret_cast<int64_t *>(m + o_off); }
  int2 *slots(unsigned char *m) const { return reinterpret_cast<int2 *>(m + o_slots); }
  int *head(unsigned char *m) const { return reinterpret_cast<int *>(m + o_head); }  // queue head
};
static_assert(sizeof(TeamItem) % 8 == 0, "the upload's parts follow one another");

// A scheme and, for SKL, a team size chosen by the autotuner (0 = the default team).
struct TuneChoice {
  int alg = kAlgSKL;
  int team = 0;
  int mode = kDeliverAuto;
  int nt = 0;  // threads per CTA of the team kernel (0: chosen from the step size)
};

constexpr unsigned long long kBarrierNs = 2000000000ull;  // default time limit of a grid barrier

// Spike ids of a handle's recorded chunks: a growing array that is not cleared when it grows
// (every id is written once, by the thread that files its step).
struct IdStore {
  int32_t *p = nullptr;
  size_t n = 0, cap = 0;
  IdStore() = default;
  IdStore(const IdStore &) = delete;
  IdStore &operator=(const IdStore &) = delete;
  ~IdStore() { free(p); }
  int32_t *extend(size_t more) {  // (null: no memory; the ids so far stay)
    if (n + more > cap) {
      const size_t want = std::max(n + more, cap + cap / 2);
      void *q = realloc(p, want * sizeof(int32_t));
      if (!q) return nullptr;
      p = static_cast<int32_t *>(q);
      cap = want;
    }
    n += more;
    return p + (n - more);
  }
};

// ---------------------------------------------------------------------------------------
// Handle.
// ---------------------------------------------------------------------------------------
struct g4s_net {
  g4s_net_desc desc{};
  NetView v{};
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, ek0 = nullptr, ek1 = nullptr;
  double last_kernel_ms = 0;
  int64_t last_launches = 0;
  GridSync *gs = nullptr;
  double *d_stats = nullptr;
  int64_t chunk_steps = 0;   // steps per chunk of the team kernel
  int64_t chunk_legacy = 0;  // steps per chunk of the other kernels (raster = spike list)
  int64_t t_abs = 0;
  uint32_t tag_next = 0;  // record tags of the team kernel: never repeated for this handle's lists
  unsigned long long barrier_ns = kBarrierNs;
  size_t device_bytes = 0;
  // per-step arrays of the last finished chunk, and the packs they came in from k_persistent
  std::vector<unsigned char> c_pack;
  std::vector<int> c_counts;
  std::vector<long long> c_base;
  std::vector<unsigned long long> c_stamps;
  // pinned staging, sized by need: a chunk's raster on its way to the host record, or blocks
  // of the neuron state (never both at once)
  unsigned char *h_stage = nullptr;
  size_t stage_bytes = 0;
  bool stage_pinned = false;
  int *h_raster = nullptr;  // the staged raster (in h_stage)
  void *arena = nullptr;    // device memory of the neuron state and the per-step arrays
  int64_t raster_full = 0;  // raster ids of a full chunk (the buffer holds v.raster_cap, by need)
  int *raster_step = nullptr;  // the first buffer: one step's ids, in the arena
  // host results since the last reset: the recorded ids, and for each recorded chunk its
  // first step, its steps' place in `counts` and its ids' place in `rid`
  std::vector<int32_t> counts;
  IdStore rid;
  struct Recorded {
    int64_t t0;
    size_t c0, off;
    int cs;
  };
  std::vector<Recorded> recorded;
  std::vector<float> upd_ms, step_ms;
  int64_t total_spikes = 0;
  double last_ms = 0, last_wall_ms = 0;
  int64_t last_spikes = 0;
  int last_alg = -1;
  int barrier_stall = 0;  // injected: the waits of the next SKL launch run out
  // SKL team kernel: team size and slice, per-step spike lists, per-row segment table,
  // requested team size (0 = auto), whether the tables satisfy the exactness bound of the
  // split accumulation, and the launch buffers of the handle's own runs
  int team_p = 0;
  int64_t team_rc = 0;
  bool team_ready = false;
  int team_batch = 0;       // geometry planned for a multi-network batch with this many CTAs (0: alone)
  bool team_ok = true;
  bool pair_ready = false;  // the packed rows match the tables
  bool pair_fits = false;   // every weight fits a packed word beside its target
  unsigned long long *list = nullptr;
  uint16_t *seg = nullptr;
  size_t seg_bytes = 0;
  // device memory from this stream-ordered pool (a server's, which keeps freed memory for
  // the next requests' networks), allocated and freed on the handle's stream; null: cudaMalloc
  cudaMemPool_t pool = nullptr;
  int want_p = 0;
  int deliver_mode = kDeliverAuto;
  int team_nt = 0;            // threads per CTA asked for: kTeamNT, kTeamNTSmall, 0 = automatic
  int team_nt_eff = kTeamNT;  // ... in use (set when the team is planned)
  bool tables_fit = false;
  TeamLaunch launch;
  // autotuner: this handle's measured choice
  bool tuned = false;
  TuneChoice tune;
  // raster streamed to a binary file (while set, the raster is not kept in host memory)
  RasterFile *rstream = nullptr;
};

static std::atomic<int> g_fail_next_alloc{0};

static cudaError_t net_malloc(g4s_net *n, void **p, size_t bytes) {
  if (n->pool) return cudaMallocFromPoolAsync(p, bytes, n->pool, n->stream);
  return cudaMalloc(p, bytes);
}
static void net_free(g4s_net *n, const void *p) {
  if (!p) return;
  if (n->pool)
    cudaFreeAsync(const_cast<void *>(p), n->stream);
  else
    cudaFree(const_cast<void *>(p));
}

static void free_stage(g4s_net *n) {
  if (n->stage_pinned)
    cudaFreeHost(n->h_stage);
  else
    free(n->h_stage);
  n->h_stage = nullptr;
  n->stage_bytes = 0;
}

static void free_net(g4s_net *n) {
  if (!n) return;
  NetView &v = n->v;
  if (n->rstream) {
    raster_close(n->rstream);
    n->rstream = nullptr;
  }
  n->launch.release();
  net_free(n, const_cast<unsigned long long *>(v.pair));
  net_free(n, n->arena);
  net_free(n, const_cast<int *>(v.idx));
  net_free(n, const_cast<float *>(v.w));
  if (v.raster != n->raster_step) net_free(n, v.raster);
  net_free(n, n->seg);
  net_free(n, n->list);
  free_stage(n);
  if (n->ev0) cudaEventDestroy(n->ev0);
  if (n->ev1) cudaEventDestroy(n->ev1);
  if (n->ek0) cudaEventDestroy(n->ek0);
  if (n->ek1) cudaEventDestroy(n->ek1);
  if (n->stream) cudaStreamDestroy(n->stream);
  delete n;
}

static int64_t row_stride(int32_t nsyn) { return ((int64_t)nsyn + 3) / 4 * 4; }

static int validate(const g4s_net_desc *d) {
  if (!d) return set_error(G4S_ERR_INVALID, "null descriptor");
  if (d->n < 2 || d->n > (int64_t)INT32_MAX) return set_error(G4S_ERR_INVALID, "n must be in [2, 2^31)");
  if (d->nsyn < 1) return set_error(G4S_ERR_INVALID, "nsyn must be >= 1");
  if (d->nsyn > kMaxSortedNsyn) return set_error(G4S_ERR_INVALID, "nsyn must be <= 16384");
  const int64_t maxsyn = d->self_loops ? d->n : d->n - 1;
  if (d->nsyn > maxsyn) return set_error(G4S_ERR_INVALID, "nsyn exceeds the number of possible targets");
  if (d->exc_permille < 0 || d->exc_permille > 1000) return set_error(G4S_ERR_INVALID, "exc_permille must be in [0, 1000]");
  if (d->conn_law != G4S_CONN_PHILOX && d->conn_law != G4S_CONN_GLIBC)
    return set_error(G4S_ERR_INVALID, "unknown connectivity law");
  if (d->conn_law == G4S_CONN_GLIBC && d->n > (int64_t)INT32_MAX / 2)
    return set_error(G4S_ERR_INVALID, "glibc law limited to n < 2^30");
  if (!(d->drive_scale >= 0.0f) || d->drive_scale > 1e6f) return set_error(G4S_ERR_INVALID, "bad drive_scale");
  return G4S_OK;
}

template <class T>
static int dalloc(g4s_net *n, T **p, size_t count, const char *what) {
  const size_t bytes = count * sizeof(T);
  cudaError_t e = g_fail_next_alloc.exchange(0) ? cudaErrorMemoryAllocation : net_malloc(n, (void **)p, bytes ? bytes : 16);
  if (e != cudaSuccess) {
    *p = nullptr;
    return set_error(G4S_ERR_NOMEM, std::string("cudaMalloc of ") + what + " (" + std::to_string(bytes) +
                                        " bytes): " + cudaGetErrorString(e));
  }
  n->device_bytes += bytes;
  return G4S_OK;
}

static void set_drive(g4s_net *n) {
  n->v.ge = 5.0f * n->desc.drive_scale;
  n->v.gi = 2.0f * n->desc.drive_scale;
}

static int alloc_net(const g4s_net_desc *d, g4s_net **out, cudaMemPool_t pool = nullptr) {
  int rc = validate(d);
  if (rc) return rc;
  g4s_net *n = new (std::nothrow) g4s_net;
  if (!n) return set_error(G4S_ERR_NOMEM, "host allocation");
  n->pool = pool;
  n->desc = *d;
  NetView &v = n->v;
  v.n = d->n;
  v.nexc = (d->n * (int64_t)d->exc_permille) / 1000;
  v.nsyn = d->nsyn;
  v.stride = (int32_t)row_stride(d->nsyn);
  v.pair_bits = pair_target_bits(d->n);
  v.seed = d->seed;
  set_drive(n);
  const size_t N = (size_t)d->n, S = (size_t)v.stride;
  // chunk: a raster buffer that holds every neuron firing at every step of the chunk (the
  // host-driven schemes and the fallback kernel use it as the spike list).  The team
  // kernel keeps its spike lists elsewhere, so when the raster is not recorded its chunk
  // is bounded only by the per-step arrays.
  const int64_t dflt = d->record_raster ? ((int64_t)1 << 30) : ((int64_t)64 << 20);
  int64_t budget = d->raster_budget_bytes > 0 ? d->raster_budget_bytes : dflt;
  int64_t cs = budget / (int64_t)(4 * N);
  if (cs < 1) cs = 1;
  if (cs > 100000) cs = 100000;
  n->chunk_legacy = cs;
  n->chunk_steps = d->record_raster ? cs : 16384;
  n->raster_full = cs * (int64_t)N;
  cs = std::max<int64_t>(cs, n->chunk_steps);
  size_t free_b = 0, total_b = 0;
  cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
  if (e != cudaSuccess) {
    free_net(n);
    return cuda_error(e, "cudaMemGetInfo");
  }
  if (pool) {  // memory the pool holds for reuse counts as free
    uint64_t reserved = 0, used = 0;
    if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) == cudaSuccess &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess && reserved > used)
      free_b += (size_t)(reserved - used);
    (void)cudaGetLastError();
    // (a pool allocates on the handle's stream)
    if ((e = cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking)) != cudaSuccess) {
      free_net(n);
      return cuda_error(e, "stream");
    }
  }
  const size_t need = N * S * 8 + N * (8 + 16 + 4 + 8 + 4 + 32) + (size_t)n->raster_full * 4 + (size_t)cs * 32;
  if (need + ((size_t)256 << 20) > free_b) {
    free_net(n);
    return set_error(G4S_ERR_NOMEM, "network needs " + std::to_string(need) + " bytes of device memory, " +
                                        std::to_string(free_b) + " free");
  }
  // The neuron state and the per-step arrays in one allocation (a cudaMalloc and its cudaFree
  // take 0.14 ms, a small network has little else to pay for), each on a 256-byte boundary.
  size_t bytes = 0;
  auto place = [&](size_t b) {
    const size_t at = bytes;
    bytes = (bytes + b + 255) / 256 * 256;
    return at;
  };
  const size_t o_vu = place(N * sizeof(float2)), o_abcd = place(N * sizeof(float4)), o_rpar = place(N * sizeof(float)),
               o_acc = place(N * sizeof(long long)), o_ilast = place(N * sizeof(float)),
               o_sstat = place(N * sizeof(SpikeStat)), o_counts = place((size_t)cs * sizeof(int)),
               o_base = place((size_t)cs * sizeof(long long)),
               o_stamps = place(((size_t)cs * 2 + 2) * sizeof(unsigned long long)), o_status = place(sizeof(int)),
               o_gs = place(sizeof(GridSync) * (1 + 2 * (size_t)kMaxTeam * kRecLines)), o_stats = place(2 * sizeof(double)),
               o_raster = place(pool ? 0 : N * sizeof(int));
  unsigned char *mem = nullptr;
  if ((rc = dalloc(n, &mem, bytes, "neuron state and per-step arrays"))) {
    free_net(n);
    return rc;
  }
  n->arena = mem;
  v.vu = reinterpret_cast<float2 *>(mem + o_vu);
  v.abcd = reinterpret_cast<float4 *>(mem + o_abcd);
  v.rpar = reinterpret_cast<float *>(mem + o_rpar);
  v.acc = reinterpret_cast<long long *>(mem + o_acc);
  v.ilast = reinterpret_cast<float *>(mem + o_ilast);
  v.sstat = reinterpret_cast<SpikeStat *>(mem + o_sstat);
  v.counts = reinterpret_cast<int *>(mem + o_counts);
  v.base = reinterpret_cast<long long *>(mem + o_base);
  v.stamps = reinterpret_cast<unsigned long long *>(mem + o_stamps);
  v.status = reinterpret_cast<int *>(mem + o_status);
  n->gs = reinterpret_cast<GridSync *>(mem + o_gs);
  n->d_stats = reinterpret_cast<double *>(mem + o_stats);
  if (!pool) n->raster_step = v.raster = reinterpret_cast<int *>(mem + o_raster);
  if ((rc = dalloc(n, const_cast<int **>(&v.idx), N * S, "targets")) ||
      (rc = dalloc(n, const_cast<float **>(&v.w), N * S, "weights")) ||
      // (a pool's network gets its whole raster now: a run may use another network's stream)
      (pool && (rc = dalloc(n, &v.raster, (size_t)n->raster_full, "raster")))) {
    free_net(n);
    return rc;
  }
  v.raster_cap = pool ? n->raster_full : d->n;
  if ((!n->stream && (e = cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking)) != cudaSuccess) ||
      (e = cudaEventCreate(&n->ev0)) != cudaSuccess || (e = cudaEventCreate(&n->ev1)) != cudaSuccess ||
      (e = cudaEventCreate(&n->ek0)) != cudaSuccess || (e = cudaEventCreate(&n->ek1)) != cudaSuccess) {
    free_net(n);
    return cuda_error(e, "stream/event");
  }
  if ((e = cudaMemsetAsync(v.status, 0, sizeof(int), n->stream)) != cudaSuccess ||
      (e = cudaMemsetAsync(n->gs, 0, sizeof(GridSync), n->stream)) != cudaSuccess) {
    free_net(n);
    return cuda_error(e, "clearing status words");
  }
  *out = n;
  return G4S_OK;
}

static int status_rc(int st, int bar, const char *what);

static int check_status(g4s_net *n, const char *what) {
  int st = 0, bar = 0;
  G4S_CUDA(cudaMemcpyAsync(&st, n->v.status, sizeof(int), cudaMemcpyDeviceToHost, n->stream));
  G4S_CUDA(cudaMemcpyAsync(&bar, &n->gs->error, sizeof(int), cudaMemcpyDeviceToHost, n->stream));
  G4S_CUDA(cudaStreamSynchronize(n->stream));
  return status_rc(st, bar, what);
}

// The device's status word and a team's error word as a G4S status.
static int status_rc(int st, int bar, const char *what) {
  if (bar == kErrTimeoutCode) return set_error(G4S_ERR_TIMEOUT, std::string(what) + ": grid barrier timed out");
  if (st == kErrOverflowCode) return set_error(G4S_ERR_OVERFLOW, std::string(what) + ": raster overflow");
  if (st == kErrConnCode) return set_error(G4S_ERR_INVALID, std::string(what) + ": connectivity draws exhausted");
  if (st != 0 || bar != 0) return set_error(G4S_ERR_CUDA, std::string(what) + ": device error " + std::to_string(st));
  return G4S_OK;
}

static int reset_net(g4s_net *n) {
  NetView &v = n->v;
  if (n->rstream) {  // the step numbering restarts: a streamed raster ends here
    RasterFile *f = n->rstream;
    n->rstream = nullptr;
    int rc = raster_close(f);
    if (rc) return rc;
  }
  set_drive(n);
  G4S_CUDA(cudaMemsetAsync(v.status, 0, sizeof(int), n->stream));
  G4S_CUDA(cudaMemsetAsync(n->gs, 0, sizeof(GridSync), n->stream));
  G4S_CUDA(launch_init(v, n->stream));
  G4S_CUDA(cudaStreamSynchronize(n->stream));
  n->t_abs = 0;
  n->rid.n = 0;
  n->recorded.clear();
  n->counts.clear();
  n->upd_ms.clear();
  n->step_ms.clear();
  n->total_spikes = 0;
  return G4S_OK;
}

static int prepare_rows(g4s_net *n);  // (defined with the team set-up below)

// ---------------------------------------------------------------------------------------
// Host generator of the reference's tables (glibc rand).  The k-th remaining target of a
// row is found by a binary search over the sorted list of targets already taken, which
// gives the reference's list-and-memmove result (gpu4snn.cu:880-898) in O(nsyn log nsyn)
// per synapse instead of O(n).
// ---------------------------------------------------------------------------------------
namespace g4s {
int conn_glibc_host(unsigned seed, int32_t n, int32_t nsyn, int32_t stride, int32_t *idx, float *w) {
  if (n < 1 || nsyn < 0 || nsyn > n || stride < nsyn) return set_error(G4S_ERR_INVALID, "bad glibc table request");
  const int32_t nexc = (int32_t)(((int64_t)n * 4) / 5);
  const float wscale = 1000.0f / (float)nsyn;
  std::vector<int32_t> taken;
  taken.reserve((size_t)nsyn);
  srand(seed);
  for (int32_t i = 0; i < n; ++i) {
    taken.clear();
    int32_t *ri = idx + (int64_t)i * stride;
    float *rw = w + (int64_t)i * stride;
    for (int32_t j = 0; j < nsyn; ++j) {
      const int32_t size = n - j;
      const int32_t k = (int32_t)((size_t)rand() % (size_t)size);
      float x = i < nexc ? wscale * 0.5f : wscale * -1.0f;
      x = x * (float)rand();
      x = x / (float)RAND_MAX;
      int32_t lo = k, hi = k + (int32_t)taken.size();
      while (lo < hi) {
        const int32_t mid = lo + (hi - lo) / 2;
        const int32_t le = (int32_t)(std::upper_bound(taken.begin(), taken.end(), mid) - taken.begin());
        if (mid + 1 - le >= k + 1)
          hi = mid;
        else
          lo = mid + 1;
      }
      taken.insert(std::upper_bound(taken.begin(), taken.end(), lo), lo);
      ri[j] = lo;
      rw[j] = x;
    }
    for (int32_t j = nsyn; j < stride; ++j) {
      ri[j] = -1;
      rw[j] = 0.0f;
    }
  }
  return G4S_OK;
}

int net_prepare_rows(g4s_net *n) { return n && n->tables_fit ? prepare_rows(n) : G4S_OK; }

double net_recent_step_ms(const g4s_net *n, int64_t k) {
  double sum = 0.0;
  int64_t used = 0;
  for (int64_t i = (int64_t)n->step_ms.size() - 1; i >= 0 && k > 0; --i, --k)
    if (n->step_ms[(size_t)i] > 0.0f) {  // (the last step of a launch has no successor stamp)
      sum += n->step_ms[(size_t)i];
      ++used;
    }
  return used ? sum / (double)used : 0.0;
}

const NetView &net_view(const g4s_net *n) { return n->v; }
cudaStream_t net_stream(const g4s_net *n) { return n->stream; }
int64_t net_steps_done(const g4s_net *n) { return n->t_abs; }
int net_team_size(const g4s_net *n) { return n->team_ready && n->team_ok && n->team_p > 0 ? n->team_p : 1; }

}  // namespace g4s

// ---------------------------------------------------------------------------------------
// Step loop.
// ---------------------------------------------------------------------------------------
// ---------------------------------------------------------------------------------------
// Autotuner.  Choices are cached process-wide by (log2 N, log2 Nsyn, log2 firing rate):
// a scheme and, for SKL, the team size.  g4s_net_autotune measures the candidates on the
// handle itself from a device snapshot of its state, restored afterwards, so tuning does
// not change the simulation.  ALG_AUTO uses the handle's own choice, else the cached one
// for its key (with the rate of its last run), else SKL with the default team.
// ---------------------------------------------------------------------------------------
static std::mutex g_tune_mu;
static std::map<std::tuple<int, int, int>, TuneChoice> g_tune_cache;

static int ilog2(double x) { return x < 1.0 ? 0 : (int)std::floor(std::log2(x)); }

static std::tuple<int, int, int> tune_key(const g4s_net *n, double rate_hz) {
  return std::make_tuple(ilog2((double)n->v.n), ilog2((double)n->v.nsyn), ilog2(rate_hz + 1.0));
}

static double recent_rate(const g4s_net *n) {
  const size_t k = std::min<size_t>(n->counts.size(), 200);
  if (!k) {
    // no history: the generated networks' rate at this drive (measured on 64 networks of 1,100
    // to 46,000 neurons, and the same within 10% at 10^6)
    static const double kDrive[] = {0.5, 0.6, 0.75, 1.0, 1.25, 1.5, 2.0}, kRate[] = {0.1, 0.4, 2.3, 7.5, 12.5, 16.9, 22.0};
    const double d = n->desc.drive_scale;
    for (int j = 0; j < 7; ++j)
      if (d <= kDrive[j])
        return j == 0 ? kRate[0]
                      : kRate[j - 1] + (kRate[j] - kRate[j - 1]) * (d - kDrive[j - 1]) / (kDrive[j] - kDrive[j - 1]);
    return kRate[6];
  }
  double s = 0;
  for (size_t i = n->counts.size() - k; i < n->counts.size(); ++i) s += n->counts[i];
  return s / (double)k / (double)n->v.n * 1000.0;
}

static int resolve_alg(g4s_net *n, int alg) {
  if (alg != kAlgAuto) return alg;
  TuneChoice c;
  if (n->tuned) {
    c = n->tune;
  } else {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tune_cache.find(tune_key(n, recent_rate(n)));
    if (it != g_tune_cache.end()) c = it->second;
  }
  if (c.alg == kAlgSKL && c.team != n->want_p && n->want_p == 0 && c.team > 0) {
    n->want_p = c.team;
    n->team_ready = false;
    n->team_ok = true;
  }
  if (c.alg == kAlgSKL) {
    n->deliver_mode = c.mode;
    if (n->team_nt != c.nt) {
      n->team_nt = c.nt;
      n->team_ready = false;
    }
  }
  return c.alg;
}

// ---------------------------------------------------------------------------------------
// CTAs of a network running alone: one up to kLoneNeurons, whose steps are then free of the
// exchange (us per step with one CTA, one per 128 neurons and 12 CTAs: N=256 x 50 2.10, 2.98,
// 2.70; 600 x 500 2.77, 3.75, 3.40, at drive 2 3.51, 3.90, 3.59; 800 x 500 at drive 2 4.26, 4.03,
// 3.68); above, one per 52 neurons, as steps are bound by the longest chain of a rank and not by
// its work (with one per 128 and per 52: N=1,000 x 500 3.89, 3.54; 2,500 x 1000 3.82, 3.66 and
// 4.24, 3.85 at drive 2; 5,000 x 1000 4.09, 3.82), not below the size from which every warp
// polls source ranks of its own (N=800 x 50 with 7 CTAs 3.57, 12 2.88), and as many as it takes,
// where that is possible, for segments short enough to be walked as runs (N=2,500 x 2000 with
// 77 CTAs 3.92, 88 3.72; 11,000 x 2000 5.15, 4.48).
// Slices of more than kTeamSlice neurons (beyond N=2,264,192 on 152 SMs; the largest that fit hold
// 15,445) take the global-atomic kernel: never more than 5% slower, and far faster where a rank
// reads many spikes for few synapses (team / global-atomic, N=2,340,000: x 10 at drive 1 35.0 /
// 33.8, at drive 2 67.3 / 35.6, at drive 8 695 / 61; x 400 39.9 / 37.7, 35.8 / 35.3, 973 / 470; the
// worst x 400 at drive 1.5 30.4 / 32.0).
constexpr int64_t kTeamSlice = 14896;
constexpr int64_t kLoneNeurons = 640, kLoneSlice = 52;
static int64_t lone_team(int64_t n, int64_t nsyn, int64_t pmax) {
  if (n <= kLoneNeurons) return 1;
  const int64_t p = std::max<int64_t>(kOwnSources, (n + kLoneSlice - 1) / kLoneSlice);
  const int64_t runs = nsyn / kGroupMinSegment + 1;
  return runs <= pmax ? std::max(p, runs) : p;
}

// Team geometry of one network for the SKL team kernel: p CTAs (at most the co-resident
// count, one per SM), by default lone_team's alone and the batch plan's in a batch,
// and the currents plus the spike buffer of a slice within the shared-memory limit.
// Returns false if the network does not fit or its tables break the exactness bound of
// the split accumulation (the global-atomic persistent kernel is used instead).
// ---------------------------------------------------------------------------------------
static bool plan_team(g4s_net *n, int want, int batch_p, int *p_out, int64_t *rc_out) {
  const NetView &v = n->v;
  if (!n->tables_fit) return false;
  int pmax = 0;
  // (both CTA sizes fit one CTA per SM: planned with the default)
  if (team_max_blocks(kTeamSmemLimit, &pmax) != cudaSuccess || pmax < 1) {
    (void)cudaGetLastError();
    return false;
  }
  pmax = std::min(pmax, kMaxTeam);
  int64_t p = want > 0 ? want : batch_p > 0 ? batch_p : lone_team(v.n, v.nsyn, pmax);
  if (p < 1) p = 1;
  if (p > pmax) p = pmax;
  int64_t rc = (v.n + p - 1) / p;
  if (team_smem(rc, (int)p) == 0) {
    rc = (v.n + pmax - 1) / pmax;
    p = (v.n + rc - 1) / rc;
    if (team_smem(rc, (int)p) == 0) return false;
  }
  if (want <= 0 && batch_p <= 0 && rc > kTeamSlice) return false;
  *p_out = (int)p;
  *rc_out = rc;
  return true;
}

// The team kernel's buffers that do not depend on the team: the packed rows of its reads
// (optional: without them, as when the device has no room left for them or a weight is too
// large to be packed beside its target, the kernel reads the separate arrays) and the tagged
// spike lists.  Both are ready on return (a batch may launch on another handle's stream).
static int prepare_rows(g4s_net *n) {
  if (!n->v.pair && n->pair_fits) {
    const size_t bytes = (size_t)n->v.n * (size_t)n->v.stride * sizeof(unsigned long long);
    if (!g_fail_next_alloc.exchange(0) && net_malloc(n, (void **)&n->v.pair, bytes) == cudaSuccess) {
      n->device_bytes += bytes;
      n->pair_ready = false;
    } else {
      (void)cudaGetLastError();
      n->v.pair = nullptr;
    }
  }
  if (n->v.pair && !n->pair_ready) {
    G4S_CUDA(launch_pairs(n->v, n->stream));
    G4S_CUDA(cudaStreamSynchronize(n->stream));
    n->pair_ready = true;
  }
  if (!n->list) {
    cudaError_t e = net_malloc(n, (void **)&n->list, (size_t)n->v.n * 2 * sizeof(unsigned long long));
    if (e != cudaSuccess) return cuda_error(e, "spike lists");
    G4S_CUDA(cudaMemsetAsync(n->list, 0, (size_t)n->v.n * 2 * sizeof(unsigned long long), n->stream));
    G4S_CUDA(cudaStreamSynchronize(n->stream));
    n->tag_next = 0;
    n->device_bytes += (size_t)n->v.n * 2 * sizeof(unsigned long long);
  }
  return G4S_OK;
}

// Team geometry (in a batch, of batch_p CTAs), the per-step spike lists and, for teams of more
// than one CTA, the per-row segment table.
static int prepare_team(g4s_net *n, int batch_p = 0) {
  if (n->team_ready && n->team_batch == batch_p) return G4S_OK;
  int p = 0;
  int64_t rc = 0;
  const bool batch = batch_p > 0;
  n->team_ready = false;  // (until everything below is in place)
  n->team_batch = batch_p;
  if (!plan_team(n, n->want_p, batch_p, &p, &rc)) {
    n->team_ok = false;
    return G4S_OK;
  }
  // CTA size: the one asked for; automatically 768 threads when a rank's expected share of
  // a step is small (fewer than 32768 synapses, from the recent firing rate), where the
  // spill-free kernel's shorter chain wins, else 1024 (more reads in flight); a batch takes
  // 1024, as its CTAs hold large shares of their networks (64 networks of 10^3 to 5 x 10^4
  // neurons in one launch 29.8 ms against 31.9, 256 of them 326 against 368)
  if (n->team_nt) {
    n->team_nt_eff = n->team_nt;
  } else {
    const double syn = (double)n->v.n * recent_rate(n) / 1000.0 * (double)n->v.nsyn / (double)p;
    n->team_nt_eff = !batch && syn < 32768.0 ? kTeamNTSmall : kTeamNT;
  }
  int rc0 = prepare_rows(n);
  if (rc0) return rc0;
  if (p > 1) {
    const size_t bytes = (size_t)n->v.n * (size_t)(p + 1) * sizeof(uint16_t);
    if (bytes > n->seg_bytes) {
      net_free(n, n->seg);
      n->seg = nullptr;
      n->device_bytes -= n->seg_bytes;
      n->seg_bytes = 0;
      cudaError_t e = g_fail_next_alloc.exchange(0) ? cudaErrorMemoryAllocation : net_malloc(n, (void **)&n->seg, bytes);
      if (e != cudaSuccess) {
        n->seg = nullptr;
        (void)cudaGetLastError();
        return cuda_error(e, "segment table");
      }
      n->seg_bytes = bytes;
      n->device_bytes += bytes;
    }
    G4S_CUDA(launch_segoff(n->v, p, rc, n->seg, n->stream));
    G4S_CUDA(cudaStreamSynchronize(n->stream));
  }
  n->team_p = p;
  n->team_rc = rc;
  n->team_ready = true;
  n->team_ok = true;
  return G4S_OK;
}

// Largest in-degree (h[0]) of the tables and, with with_mag, the largest sum(|q| >> 16) + 1
// over a neuron's inputs (h[1]), else the largest (|q| >> 16) + 1 of any synapse (h[2]); on
// the network's stream (stream-ordered scratch).
static int bound_pass(g4s_net *n, bool with_mag, unsigned long long h[3]) {
  cudaStream_t st = n->stream;
  unsigned *cnt = nullptr;
  unsigned long long *mag = nullptr, *out = nullptr;
  cudaError_t e = cudaMallocAsync((void **)&cnt, (size_t)n->v.n * 4, st);
  if (e == cudaSuccess && with_mag) e = cudaMallocAsync((void **)&mag, (size_t)n->v.n * 8, st);
  if (e == cudaSuccess) e = cudaMallocAsync((void **)&out, 24, st);
  if (e == cudaSuccess) e = launch_inbound(n->v, cnt, mag, out, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, out, 24, cudaMemcpyDeviceToHost, st);
  if (cnt) cudaFreeAsync(cnt, st);
  if (mag) cudaFreeAsync(mag, st);
  if (out) cudaFreeAsync(out, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return e == cudaSuccess ? G4S_OK : cuda_error(e, "table bound pass");
}

// Tables are kept with every row sorted by target (the pairs stay together); the
// segment table of the team kernel is rebuilt on the next SKL run.  The exactness bound
// of the split shared-memory accumulation is measured here: fewer than 65536 synapses
// into any neuron and sum(|q| >> 16) + 1 over them below 2^31 - 2^20.
static int finish_tables(g4s_net *n, bool may_be_sorted) {
  // (rows that arrive sorted, as tables read back from a network do, skip the sort)
  // Scratch is stream-ordered (cudaMallocAsync / cudaFreeAsync on the network's stream):
  // a plain cudaFree waits for the whole device, i.e. for whatever other networks are
  // running, where a server creates networks while its rounds run.
  cudaStream_t st = n->stream;
  int *flag = nullptr, h_unsorted = 1;
  cudaError_t ef = cudaSuccess;
  if (may_be_sorted)
    ef = g_fail_next_alloc.exchange(0) ? cudaErrorMemoryAllocation : cudaMallocAsync((void **)&flag, sizeof(int), st);
  if (ef == cudaSuccess && flag) ef = launch_rows_sorted(n->v, flag, st);
  if (ef == cudaSuccess && flag) ef = cudaMemcpyAsync(&h_unsorted, flag, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (flag) cudaFreeAsync(flag, st);
  if (ef == cudaSuccess && flag) ef = cudaStreamSynchronize(st);
  if (ef != cudaSuccess) return cuda_error(ef, "row order check");
  if (h_unsorted) G4S_CUDA(launch_sort_rows(n->v, !may_be_sorted, st));
  n->team_ready = false;
  n->pair_ready = false;
  // The bound.  One pass counts the in-degrees and finds the largest term (|q| >> 16) + 1
  // of any synapse: sum(|q| >> 16) + 1 over a neuron's inputs is at most its in-degree x
  // that term, which settles the bound unless some neuron has many large inputs (for the
  // generated law, an in-degree of about 32 x nsyn); only then are the sums formed exactly,
  // by a second pass with one more atomic per synapse.
  // Generated tables need no pass where the law itself settles it: a row's targets are
  // distinct, so that no in-degree exceeds n, and no weight exceeds 1000 / nsyn (below 32.7
  // neurons a synapse of the fan-out, up to N=65,535; creation of N=14,000 x 700 0.86 -> 0.44 ms).
  const unsigned long long limit = (1ull << 31) - (1ull << 20), pair_limit = 1ull << (47 - n->v.pair_bits);
  unsigned long long h[3] = {~0ull, ~0ull, ~0ull};
  int rc = G4S_OK;
  if (!may_be_sorted && n->v.nsyn > 0) {
    const float wscale = 1000.0f / (float)n->v.nsyn;
    h[0] = (unsigned long long)n->v.n;
    h[2] = ((unsigned long long)std::llrint((double)wscale * 4294967296.0) >> 16) + 1ull;
  }
  if (!(h[0] < 65536ull && h[0] * h[2] < limit && h[2] <= pair_limit) && (rc = bound_pass(n, false, h))) return rc;
  // Packed rows hold a weight in the bits that the target leaves, with its sign.
  n->pair_fits = h[2] <= pair_limit;
  if (!n->pair_fits && n->v.pair) {  // (no launch that reads them is in flight)
    net_free(n, n->v.pair);
    n->v.pair = nullptr;
    n->device_bytes -= (size_t)n->v.n * (size_t)n->v.stride * sizeof(unsigned long long);
  }
  if (h[0] < 65536ull && h[2] < limit && h[0] * h[2] < limit)
    h[1] = h[0] * h[2];  // (an upper bound of the sum)
  else if ((rc = bound_pass(n, true, h)))
    return rc;
  n->tables_fit = h[0] < 65536ull && h[1] < limit;
  return check_status(n, "row sort");
}

// The per-step arrays of `cs` steps out of their pack (round_pack_bytes, status words first), as
// the steps from `at` of the chunk.
static void chunk_unpack(g4s_net *n, const unsigned char *p, size_t cs, size_t at = 0) {
  const int *counts = reinterpret_cast<const int *>(p + 8);
  const long long *base = reinterpret_cast<const long long *>(p + 8 + ((cs * 4 + 7) & ~(size_t)7));
  const unsigned long long *stamps = reinterpret_cast<const unsigned long long *>(base + cs);
  n->c_counts.resize(at);
  n->c_base.resize(at);
  n->c_stamps.resize(2 * at);
  n->c_counts.insert(n->c_counts.end(), counts, counts + cs);
  n->c_base.insert(n->c_base.end(), base, base + cs);
  n->c_stamps.insert(n->c_stamps.end(), stamps, stamps + 2 * cs);
}

static int64_t chunk_total(const g4s_net *n, int cs) { return (int64_t)n->c_base[cs - 1] + n->c_counts[cs - 1]; }

// At least `bytes` of staging (its contents are not kept), pinned if that is to be had, else
// pageable; `pinned`: a failure instead.
static int need_stage(g4s_net *n, size_t bytes, bool pinned) {
  if (bytes <= n->stage_bytes && (n->stage_pinned || !pinned)) return G4S_OK;
  bytes = std::max(bytes, (size_t)1 << 18);
  free_stage(n);
  n->stage_pinned = !g_fail_next_alloc.exchange(0) && cudaMallocHost((void **)&n->h_stage, bytes) == cudaSuccess;
  if (!n->stage_pinned) {
    (void)cudaGetLastError();
    n->h_stage = pinned ? nullptr : static_cast<unsigned char *>(malloc(bytes));
    if (!n->h_stage) return set_error(G4S_ERR_NOMEM, "host staging buffer");
  }
  n->stage_bytes = bytes;
  return G4S_OK;
}

// The raster buffer for chunks of up to `steps` steps (every neuron firing at every step).  A
// full chunk's buffer is up to 1 GiB, of which a short run uses little: allocated by need, and
// where the device has no room for that much, by halves down to the one step's ids that the
// handle holds from its creation.  Chunks are then as long as the buffer allows.
static void need_raster(g4s_net *n, int64_t steps) {
  const int64_t want = std::min(n->raster_full, std::max<int64_t>(1, steps) * n->v.n);
  if (want <= n->v.raster_cap) return;
  if (n->v.raster != n->raster_step) {
    net_free(n, n->v.raster);
    n->device_bytes -= (size_t)n->v.raster_cap * 4;
  }
  n->v.raster = n->raster_step;
  n->v.raster_cap = n->v.n;
  for (int64_t ids = std::min(n->raster_full, std::max(want, (int64_t)1 << 20)); ids > n->v.n; ids /= 2) {
    int *p = nullptr;
    if (!g_fail_next_alloc.exchange(0) && net_malloc(n, (void **)&p, (size_t)ids * 4) == cudaSuccess) {
      n->v.raster = p;
      n->v.raster_cap = ids;
      n->device_bytes += (size_t)ids * 4;
      return;
    }
    (void)cudaGetLastError();
  }
}

// Steps of a chunk at most, where the raster buffer is written (recorded runs, and the schemes
// whose spike list it is).
static int64_t raster_steps(const g4s_net *n) { return std::max<int64_t>(1, n->v.raster_cap / n->v.n); }

static int chunk_copy_raster(g4s_net *n, int cs, cudaStream_t s) {
  const int64_t total = chunk_total(n, cs);
  if (n->desc.record_raster && total > 0) {
    const int rc = need_stage(n, (size_t)total * 4, false);
    if (rc) return rc;
    n->h_raster = reinterpret_cast<int *>(n->h_stage);
    G4S_CUDA(cudaMemcpyAsync(n->h_raster, n->v.raster, (size_t)total * 4, cudaMemcpyDeviceToHost, s));
  }
  return G4S_OK;
}

// Scratch of a thread that sorts ids (none: no memory, which only costs time).
struct SortScratch {
  int *p = nullptr;
  size_t cap = 0;
  SortScratch() = default;
  SortScratch(const SortScratch &) = delete;
  SortScratch &operator=(const SortScratch &) = delete;
  ~SortScratch() { free(p); }
  int *get(size_t n) {
    if (n > cap) {
      free(p);
      p = static_cast<int *>(malloc(n * sizeof(int)));
      cap = p ? n : 0;
    }
    return p;
  }
};

// One step's ids in ascending order: the team kernel writes them in order (but for a rank's
// bursts), the other schemes' blocks append as they come.  Large steps by digits of 11 bits, two
// or three passes, where a comparison sort takes 30 ns an id (200 steps of N=10^6 x 100, 312,000
// ids in the largest: 12.1 -> 2.6 ms; N=200,000 x 100 by scheme AB 4.9 -> 1.3 ms).
static void sort_step_ids(int *b, int cnt, SortScratch &tmp) {
  int back = 0, top = 0;
  for (int i = 1; i < cnt; ++i) back |= b[i - 1] > b[i];
  if (!back) return;
  int *from = b, *to = cnt >= 1024 ? tmp.get((size_t)cnt) : nullptr;
  if (!to) {
    std::sort(b, b + cnt);
    return;
  }
  constexpr int kBits = 11, kBins = 1 << kBits;
  for (int i = 0; i < cnt; ++i) top |= b[i];
  for (int sh = 0; sh < 31 && (top >> sh) != 0; sh += kBits) {
    int at[kBins] = {0}, sum = 0;
    for (int i = 0; i < cnt; ++i) ++at[(from[i] >> sh) & (kBins - 1)];
    for (int k = 0; k < kBins; ++k) {
      const int c = at[k];
      at[k] = sum;
      sum += c;
    }
    for (int i = 0; i < cnt; ++i) to[at[(from[i] >> sh) & (kBins - 1)]++] = from[i];
    std::swap(from, to);
  }
  if (from != b) memcpy(b, from, (size_t)cnt * sizeof(int));
}

// Steps [0, cs) of a chunk in runs of about equal ids, f(l0, l1) on each, on a host thread per
// 2^18 ids (a thread's start costs about what it saves on fewer; here, if none is to be had).
template <class F>
static void for_step_runs(int cs, const long long *base, int64_t total, F f) {
  const int64_t hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
  const int parts = (int)std::max<int64_t>(1, std::min({hw, (int64_t)cs, total >> 18}));
  std::vector<std::thread> pool;
  int l0 = 0;
  for (int p = 0; p < parts; ++p) {
    const int64_t goal = total * (p + 1) / parts;  // the steps up to the p+1-th share of the ids
    int l1 = l0;
    while (l1 < cs && (p == parts - 1 || (int64_t)base[l1] < goal)) ++l1;
    if (l1 > l0) {
      bool here = p == parts - 1;
      if (!here) try {
          pool.emplace_back(f, l0, l1);
        } catch (...) {
          here = true;
        }
      if (here) f(l0, l1);
    }
    l0 = l1;
  }
  for (auto &th : pool) th.join();
}

// The host side of a finished chunk that began at step t0, from its per-step arrays and the
// raster in the pinned staging buffer: the raster in order (kept or streamed to its file), the
// counts and the per-step times.
static int chunk_finish_from(g4s_net *n, int cs, int64_t t0, int64_t *spikes) {
  const int *counts = n->c_counts.data();
  const long long *base = n->c_base.data();
  const unsigned long long *stamps = n->c_stamps.data();
  const int64_t total = (int64_t)base[cs - 1] + counts[cs - 1];
  if (n->desc.record_raster && n->rstream) {
    SortScratch tmp;
    for (int lt = 0; lt < cs; ++lt) sort_step_ids(n->h_raster + base[lt], counts[lt], tmp);
    raster_push(n->rstream, counts, cs, n->h_raster, total);
  } else if (n->desc.record_raster && total > 0) {
    const size_t off = n->rid.n;
    int32_t *ids = n->rid.extend((size_t)total);
    if (!ids) return set_error(G4S_ERR_NOMEM, "host raster");
    n->recorded.push_back({t0, n->counts.size(), off, cs});
    for_step_runs(cs, base, total, [=](int l0, int l1) {
      SortScratch tmp;
      for (int lt = l0; lt < l1; ++lt) sort_step_ids(n->h_raster + base[lt], counts[lt], tmp);
      const size_t i0 = (size_t)base[l0], i1 = (size_t)base[l1 - 1] + (size_t)counts[l1 - 1];
      memcpy(ids + i0, n->h_raster + i0, (i1 - i0) * 4);
    });
  }
  for (int lt = 0; lt < cs; ++lt) {
    n->counts.push_back(counts[lt]);
    const unsigned long long s0 = stamps[2 * lt], s1 = stamps[2 * lt + 1];
    const unsigned long long s2 = lt + 1 < cs ? stamps[2 * lt + 2] : 0ull;
    n->upd_ms.push_back(s1 > s0 ? (float)((s1 - s0) * 1e-6) : 0.0f);
    n->step_ms.push_back(s2 > s0 ? (float)((s2 - s0) * 1e-6) : 0.0f);
  }
  *spikes = total;
  return G4S_OK;
}

static int chunk_finish(g4s_net *n, int cs, int64_t *spikes) {
  const int rc = chunk_finish_from(n, cs, n->t_abs, spikes);
  n->t_abs += cs;
  return rc;
}

// The recorded raster's first m spikes: the step of each (t) and its id.  Large rasters on
// several host threads (a fresh destination is mostly page faults).
static void raster_copy_out(const g4s_net *n, int32_t *t, int32_t *id, int64_t m) {
  for (const auto &r : n->recorded) {
    if ((int64_t)r.off >= m) break;
    std::vector<long long> base((size_t)r.cs);
    int64_t total = 0;
    for (int lt = 0; lt < r.cs; ++lt) {
      base[(size_t)lt] = total;
      total += n->counts[r.c0 + (size_t)lt];
    }
    for_step_runs(r.cs, base.data(), total, [&](int l0, int l1) {
      for (int lt = l0; lt < l1; ++lt) {
        const int64_t q0 = (int64_t)r.off + base[(size_t)lt], q1 = std::min(m, q0 + n->counts[r.c0 + (size_t)lt]);
        for (int64_t q = q0; q < q1; ++q) t[q] = (int32_t)(r.t0 + lt);
        if (q1 > q0) memcpy(id + q0, n->rid.p + q0, (size_t)(q1 - q0) * 4);
      }
    });
  }
}

// Delivery mapping of a network's multi-CTA team: the one set or tuned, else eight-lane
// groups when a rank's segment of a row holds kGroupMinSegment synapses or more on average.
static int deliver_mode_of(const g4s_net *n) {
  if (n->deliver_mode != kDeliverAuto) return n->deliver_mode;
  return n->team_p > 1 && (int64_t)n->v.nsyn >= (int64_t)kGroupMinSegment * n->team_p ? kDeliverGroup : kDeliverRun;
}

// ---------------------------------------------------------------------------------------
// One launch of the team kernel over several networks (a "round"): network i advances
// steps[i] steps (at most its chunk length).  Multi-CTA teams are queued first, then the
// one-CTA teams by decreasing work, so that long networks start early.
// ---------------------------------------------------------------------------------------
// A lone network's ranks keep their columns of the segment table in shared memory where they
// fit beside the slice in 186 KB (up to about 40,000 neurons: the next larger carve-out leaves
// the row reads 32 KB of L1 less, N=42,000 x 1000 5.11 -> 5.32), which takes a trip to L2 out of every
// step (us a step without and with: N=2,500 x 1000 3.36, 3.30; 8,000 x 500 3.59, 3.54; 33,333 x
// 777 at drive 1.5 5.32, 5.18), for launches of more than one step per kColumnRows rows: reading
// a column costs about 0.6 ns a row (14,000 rows 8 us).  The 768-thread kernel only, whose steps
// are short.
constexpr int64_t kColumnRows = 128;
constexpr size_t kColumnSmem = 186 * 1024;

// team_round_start enqueues the round on stream s and returns; team_round_finish waits for
// it and checks every network's status words.  Between the two, the host may work on the
// previous round's results, but must not touch the launch buffers (the round writes its pack
// at its end) nor the networks' device arrays.
static int team_round_start(g4s_net *const *nets, const int *steps, const bool *last, int count, TeamLaunch &L,
                            cudaStream_t s, unsigned long long limit_ns, int stall) {
  std::vector<int> order;
  L.order.clear();
  int nslots = 0, maxteam = 1;
  size_t smem = 16;
  for (int i = 0; i < count; ++i)
    if (steps[i] > 0) {
      order.push_back(i);
      nslots += nets[i]->team_p;
      maxteam = std::max(maxteam, nets[i]->team_p);
      smem = std::max(smem, team_smem(nets[i]->team_rc, nets[i]->team_p));
    }
  if (order.empty()) return G4S_OK;
  int64_t col = 0;
  if (order.size() == 1) {
    const g4s_net *n = nets[order[0]];
    const bool wants = n->team_p > 1 && n->team_nt_eff == kTeamNTSmall && steps[order[0]] > n->v.n / kColumnRows;
    const size_t with = wants ? team_smem(n->team_rc, n->team_p, n->v.n) : 0;
    if (with && with <= kColumnSmem) {
      smem = with;
      col = n->v.n;
    }
  }
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    const g4s_net *x = nets[a], *y = nets[b];
    if ((x->team_p > 1) != (y->team_p > 1)) return x->team_p > 1;
    if (x->team_p != y->team_p) return x->team_p > y->team_p;
    return (double)x->v.n * steps[a] * x->v.nsyn > (double)y->v.n * steps[b] * y->v.nsyn;
  });
  size_t pack = 0;
  L.at.assign((size_t)count, 0);
  for (int i : order) {
    L.at[(size_t)i] = pack;
    pack += round_pack_bytes(steps[i]);
  }
  int rc = L.reserve(count, nslots, pack);
  if (rc) return rc;
  bool pair = true;  // every network of the round has its packed rows
  for (int i : order) pair = pair && nets[i]->v.pair != nullptr;
  int nt = nets[order[0]]->team_nt_eff;  // threads per CTA: the networks' own when they agree
  // delivery mapping of the launch's multi-CTA teams: the one that most of their work asks for
  double group_work = 0.0, run_work = 0.0;
  bool solo = false;  // one-CTA teams in the round
  for (int i : order) {
    const g4s_net *n = nets[i];
    if (n->team_nt_eff != nt) nt = kTeamNT;
    solo = solo || n->team_p == 1;
    if (n->team_p > 1) (deliver_mode_of(n) == kDeliverGroup ? group_work : run_work) += (double)n->v.n * n->v.nsyn * steps[i];
  }
  const int mode = group_work > run_work ? kDeliverGroup : kDeliverRun;
  int gmax = 0;
  G4S_CUDA(team_max_blocks(smem, &gmax, nt));  // also raises the kernel's shared-memory ceiling
  if (gmax < maxteam) return set_error(G4S_ERR_CUDA, "team larger than the co-resident grid");
  const int grid = std::min(nslots, gmax);
  // this round's descriptors, in pinned host memory
  int k = 0;
  for (int i : order) {
    g4s_net *n = nets[i];
    TeamItem &it = L.items(L.h_mem)[i];
    it.v = n->v;
    if (!n->desc.record_raster) it.v.raster_cap = 0;  // (its raster is never read)
    it.seg = n->seg;
    it.list = n->list;
    it.rec = reinterpret_cast<unsigned long long *>(n->gs + 1);
    it.t_abs0 = n->t_abs;
    it.steps = steps[i];
    it.last = last[i] ? 1 : 0;
    it.team = n->team_p;
    it.rc = (int)n->team_rc;
    it.col = (int)col;
    it.sync = n->gs;
    if ((uint64_t)n->tag_next + (uint64_t)steps[i] + 2 >= 0xFFFFFFFFull) {  // tags would wrap: start over
      G4S_CUDA(cudaMemsetAsync(n->list, 0, (size_t)n->v.n * 2 * sizeof(unsigned long long), s));
      n->tag_next = 0;
    }
    it.tag0 = n->tag_next;
    n->tag_next += (uint32_t)steps[i];
    for (int r = 0; r < n->team_p; ++r) L.slots(L.h_mem)[k++] = make_int2(i, r);
    L.off(L.h_mem)[i] = (int64_t)L.at[(size_t)i];
  }
  for (int i = 0; i < count; ++i)
    if (steps[i] <= 0) L.items(L.h_mem)[i].steps = 0;
  *L.head(L.h_mem) = 0;
  L.nets.assign(nets, nets + count);
  L.steps.assign(steps, steps + count);
  // One copy up, one kernel clearing every network's words of the launch, the team kernel
  // between two events, one kernel packing every network's results, one copy down: sized by
  // the round's own steps and networks.  (As a CUDA graph, a lone network's round cleared and
  // copied arrays of its longest chunk: 0.18 ms beside the kernel for 2000 steps of N=2,500,
  // 0.04 so, and a new network had its graph to build first.)
  G4S_CUDA(cudaMemcpyAsync(L.d_mem, L.h_mem, L.o_pack, cudaMemcpyHostToDevice, s));
  G4S_CUDA(launch_round_clear(L.items(L.d_mem), count, s));
  G4S_CUDA(cudaEventRecord(L.e0, s));
  G4S_CUDA(launch_team(L.items(L.d_mem), L.slots(L.d_mem), nslots, L.head(L.d_mem), grid, smem, limit_ns,
                       stall, s, pair, mode, solo, nt));
  G4S_CUDA(cudaEventRecord(L.e1, s));
  G4S_CUDA(launch_round_gather(L.items(L.d_mem), L.off(L.d_mem), count, L.d_mem + L.o_pack, s));
  G4S_CUDA(cudaMemcpyAsync(L.h_mem + L.o_pack, L.d_mem + L.o_pack, pack, cudaMemcpyDeviceToHost, s));
  L.order = order;
  return G4S_OK;
}

static int team_round_finish(TeamLaunch &L, cudaStream_t s, double *kernel_ms, int64_t *launches) {
  if (L.order.empty()) return G4S_OK;  // nothing was launched
  G4S_CUDA(cudaStreamSynchronize(s));
  float ms = 0.0f;
  G4S_CUDA(cudaEventElapsedTime(&ms, L.e0, L.e1));
  *kernel_ms += ms;
  *launches += 1;
  for (int i : L.order) {
    // (each network's share of the pack)
    chunk_unpack(L.nets[(size_t)i], L.h_mem + L.o_pack + L.at[(size_t)i], (size_t)L.steps[(size_t)i]);
  }
  for (int i : L.order) {
    const int *status = reinterpret_cast<const int *>(L.h_mem + L.o_pack + L.at[(size_t)i]);
    const int rc = status_rc(status[0], status[1], "team step kernel");
    if (rc) return rc;
  }
  return G4S_OK;
}

static int team_round(g4s_net *const *nets, const int *steps, const bool *last, int count, TeamLaunch &L,
                      cudaStream_t s, unsigned long long limit_ns, int stall, double *kernel_ms, int64_t *launches) {
  const int rc = team_round_start(nets, steps, last, count, L, s, limit_ns, stall);
  return rc ? rc : team_round_finish(L, s, kernel_ms, launches);
}

// Steps that one pack holds in the memory of the spike records.
constexpr int kPackSteps = (int)((sizeof(GridSync) * 2 * kMaxTeam * kRecLines - 16) / 28);

// Why the waits of a handle's next SKL launch run out (0: they need not).
static int stall_of(const g4s_net *n) { return n->barrier_stall ? kStallFault : n->barrier_ns == 0 ? kStallLimit : 0; }

// One chunk of steps by a launch that works on the handle's global arrays.
static int run_chunk(g4s_net *n, int cs, bool last, bool skl, StepLaunch &launch, int64_t *spikes, double *kernel_ms) {
  NetView &v = n->v;
  G4S_CUDA(cudaMemsetAsync(v.counts, 0, (size_t)cs * sizeof(int), n->stream));
  G4S_CUDA(cudaMemsetAsync(v.stamps, 0, ((size_t)cs * 2 + 2) * 8, n->stream));
  G4S_CUDA(cudaMemsetAsync(n->gs, 0, sizeof(GridSync), n->stream));
  G4S_CUDA(cudaEventRecord(n->ek0, n->stream));
  G4S_CUDA(launch(v, n->t_abs, cs, last, n->gs, skl ? n->barrier_ns : kBarrierNs, skl ? stall_of(n) : 0, n->stream));
  if (skl) n->barrier_stall = 0;
  G4S_CUDA(cudaEventRecord(n->ek1, n->stream));
  // (packed on the device, where the team kernel has its records, and brought back by one copy for
  // some 3,200 steps: as five pageable ones, and two waits, a run of one step of N=2,500 took 75
  // us, 43 so)
  unsigned char *d_pack = reinterpret_cast<unsigned char *>(n->gs + 1);
  n->c_pack.resize((size_t)((cs - 1) / kPackSteps + 1) * round_pack_bytes(kPackSteps));
  auto piece = [&](int s0) { return n->c_pack.data() + (size_t)(s0 / kPackSteps) * round_pack_bytes(kPackSteps); };
  for (int s0 = 0; s0 < cs; s0 += kPackSteps) {
    const int k = std::min(kPackSteps, cs - s0);
    NetView part = v;
    part.counts += s0;
    part.base += s0;
    part.stamps += 2 * s0;
    G4S_CUDA(launch_chunk_gather(part, n->gs, k, d_pack, n->stream));
    G4S_CUDA(cudaMemcpyAsync(piece(s0), d_pack, round_pack_bytes(k), cudaMemcpyDeviceToHost, n->stream));
  }
  G4S_CUDA(cudaStreamSynchronize(n->stream));
  const int *status = reinterpret_cast<const int *>(piece(0));
  int rc = status_rc(status[0], status[1], "persistent step kernel");
  if (rc) return rc;
  float kms = 0.0f;
  G4S_CUDA(cudaEventElapsedTime(&kms, n->ek0, n->ek1));
  *kernel_ms += kms;
  for (int s0 = 0; s0 < cs; s0 += kPackSteps) chunk_unpack(n, piece(s0), (size_t)std::min(kPackSteps, cs - s0), (size_t)s0);
  if (n->desc.record_raster && chunk_total(n, cs) > 0) {
    if ((rc = chunk_copy_raster(n, cs, n->stream))) return rc;
    G4S_CUDA(cudaStreamSynchronize(n->stream));
  }
  return chunk_finish(n, cs, spikes);
}

namespace g4s {
int64_t net_chunk_steps(g4s_net *n, int64_t steps) {
  steps = std::min(steps, n->chunk_legacy);
  need_raster(n, steps);
  return std::min(steps, raster_steps(n));
}

int net_run_by(g4s_net *n, int steps, bool last, StepLaunch &launch) {
  int64_t spikes = 0;
  double ms = 0.0;
  const int rc = run_chunk(n, steps, last, true, launch, &spikes, &ms);
  if (rc) return rc;
  n->last_ms = n->last_wall_ms = n->last_kernel_ms = ms;
  n->last_launches = 1;
  n->last_spikes = spikes;
  n->total_spikes += spikes;
  n->last_alg = kAlgSKL;
  return G4S_OK;
}
}  // namespace g4s

static int run_net(g4s_net *n, int32_t steps, int32_t alg_in) {
  if (steps < 0) return set_error(G4S_ERR_INVALID, "steps must be >= 0");
  if (alg_in < 0 || alg_in > kAlgAuto) return set_error(G4S_ERR_INVALID, "unknown algorithm");
  if (n->t_abs + steps > (int64_t)INT32_MAX) return set_error(G4S_ERR_INVALID, "step counter limit");
  const int alg = resolve_alg(n, alg_in);
  NetView &v = n->v;
  if (alg == kAlgSKL) {
    int rc0 = prepare_team(n);
    if (rc0) return rc0;
  }
  const bool team = alg == kAlgSKL && n->team_ok && n->team_ready;
  // (the team kernel writes a raster only where it is recorded; the other schemes' spike lists
  // are the raster)
  int64_t longest = team ? n->chunk_steps : n->chunk_legacy;
  if (!team || n->desc.record_raster) {
    need_raster(n, std::min<int64_t>(steps, longest));
    longest = std::min(longest, raster_steps(n));
  }
  const auto w0 = std::chrono::steady_clock::now();
  G4S_CUDA(cudaEventRecord(n->ev0, n->stream));
  int64_t remaining = steps, spikes = 0, launches = 0;
  double kernel_ms = 0.0;
  if (team) {
    // Chunks as team rounds, pipelined: once a round has ended and its raster is copied
    // down, the next round is launched, and the host sorts and files the finished chunk
    // while the GPU runs the next one.
    int cs = 0;
    auto start = [&]() -> int {
      cs = (int)std::min<int64_t>(remaining, longest);
      const bool last_chunk = remaining == cs;
      g4s_net *one[1] = {n};
      const int rc = team_round_start(one, &cs, &last_chunk, 1, n->launch, n->stream, n->barrier_ns, stall_of(n));
      n->barrier_stall = 0;
      remaining -= cs;
      return rc;
    };
    int rc = remaining > 0 ? start() : G4S_OK;
    if (rc) return rc;
    while (cs > 0) {
      if ((rc = team_round_finish(n->launch, n->stream, &kernel_ms, &launches))) return rc;
      // (this chunk's raster out of the device buffer that the next round overwrites)
      if ((rc = chunk_copy_raster(n, cs, n->stream))) return rc;
      G4S_CUDA(cudaStreamSynchronize(n->stream));
      const int done = cs;
      const int64_t t0 = n->t_abs;
      n->t_abs += done;
      cs = 0;
      const int rs = remaining > 0 ? start() : G4S_OK;
      int64_t chunk_spikes = 0;  // (the finished chunk is filed even if the next launch failed)
      rc = chunk_finish_from(n, done, t0, &chunk_spikes);
      spikes += chunk_spikes;
      if (rs || rc) {
        if (!rs && cs > 0) team_round_finish(n->launch, n->stream, &kernel_ms, &launches);  // (the round in flight ends first)
        return rs ? rs : rc;
      }
    }
  }
  struct Schemes : StepLaunch {  // (the time limit and injected faults are the SKL scheme's)
    int alg;
    double synapses;
    int64_t *launches;
    cudaError_t operator()(const NetView &v, int64_t t_abs0, int cs, bool last, GridSync *gs, unsigned long long limit_ns,
                           int stall, cudaStream_t s) override {
      int made = 0;
      const cudaError_t e = launch_steps(v, t_abs0, cs, last, gs, limit_ns, alg, synapses, stall, s, &made);
      *launches += made;
      return e;
    }
  } schemes;
  schemes.alg = alg;
  schemes.launches = &launches;
  while (!team && remaining > 0) {
    const int cs = (int)std::min<int64_t>(remaining, longest);
    int64_t chunk_spikes = 0;
    schemes.synapses = (double)v.n * recent_rate(n) * 1e-3 * (double)v.nsyn;
    const int rc = run_chunk(n, cs, remaining == cs, alg == kAlgSKL, schemes, &chunk_spikes, &kernel_ms);
    if (rc) return rc;
    spikes += chunk_spikes;
    remaining -= cs;
  }
  G4S_CUDA(cudaEventRecord(n->ev1, n->stream));
  G4S_CUDA(cudaEventSynchronize(n->ev1));
  float ms = 0.0f;
  G4S_CUDA(cudaEventElapsedTime(&ms, n->ev0, n->ev1));
  n->last_ms = ms;
  n->last_wall_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - w0).count();
  n->last_spikes = spikes;
  n->total_spikes += spikes;
  n->last_alg = alg;
  n->last_kernel_ms = kernel_ms;
  n->last_launches = launches;
  return G4S_OK;
}

// Estimated device time in us of one step of a network on a team of p CTAs of 1024 threads: a chain
// of round trips, the update and drive of a CTA's neurons, and its share of the step's synapses.
// One CTA walks rows in pieces of 128 synapses.  A larger team's share depends on the length of
// its segments; where a step has few spikes the time is that of walking the longest one, eight
// lanes a spike.
static double team_step_us(const g4s_net *n, double syn, int p) {
  const double neurons = (double)n->v.n / p, seg = std::max(1.0, (double)n->v.nsyn / p);
  if (p == 1) return 2.0 + 1.35e-3 * neurons + 0.185e-3 * syn * (double)((n->v.nsyn + 127) / 128 * 128) / n->v.nsyn;
  return std::max(3.6 + 1.6e-3 * neurons + (0.19e-3 + 2.2e-3 / seg) * syn / p, 2.8 + 1.6e-3 * neurons + 5.8e-3 * seg);
}

// CTAs of each network of a batch.  At one CTA per kBatchSlice neurons the networks take about
// their share of a full GPU's time.  Where those teams would leave SMs idle the launch lasts
// as long as its slowest network, so the CTAs go where the estimated time is: the shortest
// time for which every network's smallest sufficient team fits one CTA per SM together (64
// networks of 10^3 to 5 x 10^4 neurons, 16-fold apart in work: 44.3 ms by equal slices, 32.3 so, both with 768 threads).
// Teams of an earlier plan are kept while they are within a fifth of that time (a new team has
// its segment table to build).
static void plan_batch(g4s_net *const *nets, const int32_t *steps, int count, std::vector<int> &teams) {
  teams.assign((size_t)count, 1);
  int gmax = 0;
  if (team_max_blocks(kTeamSmemLimit, &gmax) != cudaSuccess || gmax < 1) {
    (void)cudaGetLastError();
    gmax = 1;
  }
  const int pcap = std::min(gmax, kMaxTeam);
  std::vector<double> syn((size_t)count);
  int64_t least = 0, held = 0;
  double held_us = 0.0;
  bool planned = true;  // every network has a team of an earlier plan
  for (int i = 0; i < count; ++i) {
    const g4s_net *n = nets[i];
    teams[(size_t)i] = (int)std::min<int64_t>(pcap, (n->v.n + kBatchSlice - 1) / kBatchSlice);
    syn[(size_t)i] = (double)n->v.n * recent_rate(n) * 1e-3 * (double)n->v.nsyn;
    if (steps[i] <= 0) continue;
    least += teams[(size_t)i];
    planned = planned && n->team_ready && n->team_batch > 0;
    held += n->team_p;
    if (n->team_p > 0) held_us = std::max(held_us, steps[i] * team_step_us(n, syn[(size_t)i], n->team_p));
  }
  if (least >= gmax) return;
  // the CTAs that network i needs to finish in `us` (more than the GPU has: too many)
  auto need = [&](int i, double us) {
    const g4s_net *n = nets[i];
    const int most = (int)std::min<int64_t>(pcap, (n->v.n + kBatchMinSlice - 1) / kBatchMinSlice);
    int lo = teams[(size_t)i], hi = std::max(lo, most);
    while (lo < hi && steps[i] * team_step_us(n, syn[(size_t)i], lo) > us) ++lo;
    return lo;
  };
  auto total = [&](double us) {
    int64_t t = 0;
    for (int i = 0; i < count && t <= gmax; ++i)
      if (steps[i] > 0) t += need(i, us);
    return t;
  };
  double lo = 0.0, hi = 0.0;
  for (int i = 0; i < count; ++i) hi = std::max(hi, steps[i] * team_step_us(nets[i], syn[(size_t)i], teams[(size_t)i]));
  for (int k = 0; k < 24; ++k) {
    const double mid = 0.5 * (lo + hi);
    (total(mid) <= gmax ? hi : lo) = mid;
  }
  const bool keep = planned && held <= gmax && held_us <= 1.2 * hi;
  for (int i = 0; i < count; ++i)
    if (steps[i] > 0) teams[(size_t)i] = keep ? nets[i]->team_batch : need(i, hi);
}

// Several networks advanced together by the SKL team kernel: network i runs steps[i]
// further steps; each round advances every unfinished network by up to its chunk length
// in one persistent launch.
static int run_nets(g4s_net *const *nets, const int32_t *steps, int count, double *dev_ms, int64_t *launches) {
  if (count <= 0) return set_error(G4S_ERR_INVALID, "count must be > 0");
  for (int i = 0; i < count; ++i)
    if (!nets[i]) return set_error(G4S_ERR_INVALID, "null handle in batch");
  std::vector<int> teams;
  if (count > 1) plan_batch(nets, steps, count, teams);
  std::vector<int64_t> remaining(count), longest(count);
  for (int i = 0; i < count; ++i) {
    if (steps[i] < 0 || nets[i]->t_abs + steps[i] > (int64_t)INT32_MAX)
      return set_error(G4S_ERR_INVALID, "bad step count in batch");
    for (int j = 0; j < i; ++j)
      if (nets[j] == nets[i]) return set_error(G4S_ERR_INVALID, "a handle appears twice in the batch");
    int rc = prepare_team(nets[i], count > 1 ? teams[(size_t)i] : 0);
    if (rc) return rc;
    if (!nets[i]->team_ok)
      return set_error(G4S_ERR_INVALID, "a network of the batch does not fit the team kernel");
    longest[i] = nets[i]->chunk_steps;
    if (nets[i]->desc.record_raster) {
      need_raster(nets[i], std::min<int64_t>(steps[i], longest[i]));
      longest[i] = std::min(longest[i], raster_steps(nets[i]));
    }
    remaining[i] = steps[i];
    nets[i]->last_spikes = 0;
  }
  static thread_local TeamLaunch L;
  cudaStream_t s = nets[0]->stream;
  std::vector<int> cs(count);
  std::unique_ptr<bool[]> last(new bool[count]);
  double kms = 0.0;
  int64_t nl = 0;
  const auto w0 = std::chrono::steady_clock::now();
  for (;;) {
    bool any = false;
    for (int i = 0; i < count; ++i) {
      cs[i] = (int)std::min<int64_t>(remaining[i], longest[i]);
      last[i] = cs[i] > 0 && cs[i] == remaining[i];
      any = any || cs[i] > 0;
    }
    if (!any) break;
    int rc = team_round(nets, cs.data(), last.get(), count, L, s, nets[0]->barrier_ns, nets[0]->barrier_ns == 0 ? kStallLimit : 0, &kms, &nl);
    if (rc) return rc;
    for (int i = 0; i < count; ++i)
      if (cs[i] > 0 && (rc = chunk_copy_raster(nets[i], cs[i], s))) return rc;
    G4S_CUDA(cudaStreamSynchronize(s));
    for (int i = 0; i < count; ++i)
      if (cs[i] > 0) {
        int64_t sp = 0;
        if ((rc = chunk_finish(nets[i], cs[i], &sp))) return rc;
        nets[i]->last_spikes += sp;
        nets[i]->total_spikes += sp;
        remaining[i] -= cs[i];
      }
  }
  const double wall = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - w0).count();
  for (int i = 0; i < count; ++i) {
    nets[i]->last_alg = kAlgSKL;
    nets[i]->last_kernel_ms = kms;
    nets[i]->last_ms = wall;
    nets[i]->last_wall_ms = wall;
    nets[i]->last_launches = nl;
  }
  if (dev_ms) *dev_ms = kms;
  if (launches) *launches = nl;
  return G4S_OK;
}

// ---------------------------------------------------------------------------------------
// Autotuner measurement: a device snapshot of the mutable state and the host record,
// each candidate timed on `probe` steps from the snapshot, the snapshot restored.
// Candidates: SKL with the default team and with teams of 1, 2, 4, ... CTAs up to the
// co-resident grid (those that fit), AB and AP.
// ---------------------------------------------------------------------------------------
struct StateSnapshot {
  float2 *vu = nullptr;
  long long *acc = nullptr;
  SpikeStat *ss = nullptr;
  float *il = nullptr;
  int64_t t_abs = 0, total = 0;
  size_t nr = 0, nrec = 0, nc = 0;
  ~StateSnapshot() {
    cudaFree(vu);
    cudaFree(acc);
    cudaFree(ss);
    cudaFree(il);
  }
};

static int snapshot_take(g4s_net *n, StateSnapshot &s) {
  const size_t N = (size_t)n->v.n;
  G4S_CUDA(cudaMalloc((void **)&s.vu, N * sizeof(float2)));
  G4S_CUDA(cudaMalloc((void **)&s.acc, N * sizeof(long long)));
  G4S_CUDA(cudaMalloc((void **)&s.ss, N * sizeof(SpikeStat)));
  G4S_CUDA(cudaMalloc((void **)&s.il, N * sizeof(float)));
  G4S_CUDA(cudaMemcpyAsync(s.vu, n->v.vu, N * sizeof(float2), cudaMemcpyDeviceToDevice, n->stream));
  G4S_CUDA(cudaMemcpyAsync(s.acc, n->v.acc, N * sizeof(long long), cudaMemcpyDeviceToDevice, n->stream));
  G4S_CUDA(cudaMemcpyAsync(s.ss, n->v.sstat, N * sizeof(SpikeStat), cudaMemcpyDeviceToDevice, n->stream));
  G4S_CUDA(cudaMemcpyAsync(s.il, n->v.ilast, N * sizeof(float), cudaMemcpyDeviceToDevice, n->stream));
  G4S_CUDA(cudaStreamSynchronize(n->stream));
  s.t_abs = n->t_abs;
  s.total = n->total_spikes;
  s.nr = n->rid.n;
  s.nrec = n->recorded.size();
  s.nc = n->counts.size();
  return G4S_OK;
}

static int snapshot_restore(g4s_net *n, const StateSnapshot &s) {
  const size_t N = (size_t)n->v.n;
  G4S_CUDA(cudaMemcpyAsync(n->v.vu, s.vu, N * sizeof(float2), cudaMemcpyDeviceToDevice, n->stream));
  G4S_CUDA(cudaMemcpyAsync(n->v.acc, s.acc, N * sizeof(long long), cudaMemcpyDeviceToDevice, n->stream));
  G4S_CUDA(cudaMemcpyAsync(n->v.sstat, s.ss, N * sizeof(SpikeStat), cudaMemcpyDeviceToDevice, n->stream));
  G4S_CUDA(cudaMemcpyAsync(n->v.ilast, s.il, N * sizeof(float), cudaMemcpyDeviceToDevice, n->stream));
  G4S_CUDA(cudaStreamSynchronize(n->stream));
  n->t_abs = s.t_abs;
  n->total_spikes = s.total;
  n->rid.n = s.nr;
  n->recorded.resize(s.nrec);
  n->counts.resize(s.nc);
  n->upd_ms.resize(s.nc);
  n->step_ms.resize(s.nc);
  return G4S_OK;
}

static int autotune(g4s_net *n, int32_t probe, TuneChoice *best, double *best_us) {
  probe = std::max(8, std::min(probe, 4000));
  StateSnapshot snap;
  int rc = snapshot_take(n, snap);
  if (rc) return rc;
  const int keep_p = n->want_p;
  std::vector<TuneChoice> cand;
  int pmax = 0;
  if (team_max_blocks(team_smem(1, 1), &pmax) != cudaSuccess) pmax = 1;
  (void)cudaGetLastError();
  pmax = std::min(pmax, kMaxTeam);
  std::vector<int> teams = {0};
  for (int p = 1; p <= pmax; p *= 2) teams.push_back(p);
  if (pmax > 1) teams.push_back(pmax);
  // each team size with both CTA sizes of the team kernel, by segment runs and, where a
  // rank's segment of a row averages half the automatic threshold or more, by eight-lane
  // groups too
  for (int p : teams)
    for (int nt : {kTeamNT, kTeamNTSmall}) {
      cand.push_back(TuneChoice{kAlgSKL, p, kDeliverRun, nt});
      const int pe = p == 0 ? pmax : p;
      if (pe > 1 && 2 * (int64_t)n->v.nsyn >= (int64_t)kGroupMinSegment * pe)
        cand.push_back(TuneChoice{kAlgSKL, p, kDeliverGroup, nt});
    }
  cand.push_back(TuneChoice{kAlgAB, 0, kDeliverRun});
  cand.push_back(TuneChoice{kAlgAP, 0, kDeliverRun});
  const int keep_mode = n->deliver_mode, keep_nt = n->team_nt;
  double best_t = 1e300, rate = 0.0;
  TuneChoice pick = cand[0];
  for (const TuneChoice &c : cand) {
    if (c.alg == kAlgSKL) {
      n->want_p = c.team;
      n->deliver_mode = c.mode;
      n->team_nt = c.nt;
      n->team_ready = false;
      n->team_ok = true;
      if ((rc = prepare_team(n))) break;
      if (!n->team_ok || (c.team > 0 && n->team_p != c.team)) continue;  // does not fit
    }
    if ((rc = run_net(n, 8, c.alg)) || (rc = snapshot_restore(n, snap))) break;
    if ((rc = run_net(n, probe, c.alg))) break;
    const double t = n->last_kernel_ms * 1e3 / probe;
    rate = (double)n->last_spikes / ((double)n->v.n * probe) * 1000.0;
    if ((rc = snapshot_restore(n, snap))) break;
    if (t < best_t) {
      best_t = t;
      pick = c;
      if (c.alg == kAlgSKL && c.team == 0) pick.team = n->team_p;
    }
  }
  n->want_p = keep_p;
  n->deliver_mode = keep_mode;
  n->team_nt = keep_nt;
  n->team_ready = false;
  n->team_ok = true;
  if (rc) return rc;
  n->tune = pick;
  n->tuned = true;
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune_cache[tune_key(n, rate)] = pick;
  }
  *best = pick;
  *best_us = best_t;
  return G4S_OK;
}

// ---------------------------------------------------------------------------------------
// Result files in the reference's formats.
// ---------------------------------------------------------------------------------------
static int mkdirs(const std::string &path) {
  std::string cur;
  for (size_t i = 0; i <= path.size(); ++i) {
    if (i == path.size() || path[i] == '/') {
      if (!cur.empty() && mkdir(cur.c_str(), 0775) != 0 && errno != EEXIST)
        return set_error(G4S_ERR_IO, "mkdir " + cur + ": " + strerror(errno));
    }
    if (i < path.size()) cur.push_back(path[i]);
  }
  return G4S_OK;
}

static void write_record(std::ofstream &o, float a, float b, float c, float d, float v, float u, float I, int64_t id,
                         int nospks) {
  o << a << " " << b << " " << c << " " << d << " " << v << " " << u << " " << I << " " << id << " " << nospks
    << "\n";
}

static int write_results(g4s_net *n, const std::string &dir, double elapsed, double ewd) {
  int rc = mkdirs(dir);
  if (rc) return rc;
  const std::string p = dir.back() == '/' ? dir : dir + "/";
  const int64_t N = n->v.n;
  std::vector<float> v(N), u(N), I(N), a(N), b(N), c(N), d(N);
  std::vector<int32_t> nos(N);
  rc = g4s_net_state(n, v.data(), u.data(), I.data(), a.data(), b.data(), c.data(), d.data(), nos.data());
  if (rc) return rc;
  {
    std::ofstream o(p + "neuroninfo.csv");
    if (!o.is_open()) return set_error(G4S_ERR_IO, "cannot open " + p + "neuroninfo.csv");
    o << "a b c d v u I id nospks" << "\n";
    for (int64_t i = 0; i < N; ++i) write_record(o, a[i], b[i], c[i], d[i], -65.0f, b[i] * -65.0f, 0.0f, i, 0);
  }
  {
    std::ofstream o(p + "spiketimes.csv");
    if (!o.is_open()) return set_error(G4S_ERR_IO, "cannot open " + p + "spiketimes.csv");
    o << "SpkTime NeuronID" << "\n";
    for (const auto &r : n->recorded) {
      size_t q = r.off;
      for (int lt = 0; lt < r.cs; ++lt)
        for (int k = 0; k < n->counts[r.c0 + (size_t)lt]; ++k) o << r.t0 + lt << " " << n->rid.p[q++] << "\n";
    }
  }
  {
    std::ofstream o(p + "computetime.csv");
    if (!o.is_open()) return set_error(G4S_ERR_IO, "cannot open " + p + "computetime.csv");
    o << "TimeStep SpksPerStep TimeKernelUpdate TimeSpent" << "\n";
    for (size_t t = 0; t < n->counts.size(); ++t)
      o << t << " " << n->counts[t] << " " << (double)n->upd_ms[t] << " " << (double)n->step_ms[t] << "\n";
  }
  {
    std::ofstream o(p + "sim_overview.csv");
    if (!o.is_open()) return set_error(G4S_ERR_IO, "cannot open " + p + "sim_overview.csv");
    o << "N elapsed(ms) elapsedwithdata(ms) totalspkcount" << "\n";
    o << N << " " << elapsed << " " << ewd << " " << n->total_spikes;
  }
  {
    std::ofstream o(p + "neuroninfoafter.csv");
    if (!o.is_open()) return set_error(G4S_ERR_IO, "cannot open " + p + "neuroninfoafter.csv");
    o << "a b c d v u I id nospks" << "\n";
    for (int64_t i = 0; i < N; ++i) write_record(o, a[i], b[i], c[i], d[i], v[i], u[i], I[i], i, nos[i]);
  }
  return G4S_OK;
}

// ---------------------------------------------------------------------------------------
// Exported entry points.
// ---------------------------------------------------------------------------------------
// First entry of host tables that targets no neuron of a network (SIZE_MAX: none), on all
// host cores, block by block (the largest target of 4096, a loop the compiler vectorises; a
// block over the limit is searched for its first offending entry).
static size_t first_bad_host(const int32_t *idx, size_t cnt, int32_t nn) {
  const unsigned hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
  const size_t parts = cnt >= ((size_t)1 << 22) ? hw : 1, per = (cnt + parts - 1) / parts;
  std::vector<size_t> bad(parts, SIZE_MAX);
  auto scan = [&](size_t p) {
    const size_t end = std::min(cnt, (p + 1) * per);
    for (size_t k0 = p * per; k0 < end; k0 += 4096) {
      const size_t k1 = std::min(end, k0 + 4096);
      int32_t mx = INT32_MIN;
      for (size_t k = k0; k < k1; ++k) mx = std::max(mx, idx[k]);
      if (mx < nn) continue;
      for (size_t k = k0; k < k1; ++k)
        if (idx[k] >= nn) {
          bad[p] = k;
          return;
        }
    }
  };
  std::vector<std::thread> pool;
  for (size_t p = 1; p < parts; ++p) pool.emplace_back(scan, p);
  scan(0);
  for (auto &t : pool) t.join();
  return *std::min_element(bad.begin(), bad.end());
}

// Before the tables change: no plan, and no new one until finish_tables has passed the new ones
// (if it does not get there, runs take the global-atomic kernel, whose additions any table of
// checked targets keeps in range).
static void drop_plan(g4s_net *n) { n->team_ready = n->pair_ready = n->tables_fit = false; }

// The same on the device, on the targets' way to it: into memory that holds nothing needed
// (the packed rows, formed again from the tables; else stream-ordered scratch), checked there
// and only then moved to v.idx (*moved).  The 400 MB of targets of N=100,000 x 1000 take
// 0.06 ms so, and 0.13 ms to move, instead of 2 ms on 16 host cores before the copy begins.
// With no memory for it nothing is done.
constexpr size_t kHostCheckSlots = 65536;  // (fewer: 10 us on the host, as long as a wait for the device)
static int first_bad_device(g4s_net *n, const int32_t *idx, size_t *bad, bool *moved) {
  NetView &v = n->v;
  cudaStream_t s = n->stream;
  const size_t bytes = (size_t)v.n * (size_t)v.stride * 4;
  unsigned long long first = ~0ull, *d_first = nullptr;
  int *scratch = nullptr;
  if (cudaMallocAsync((void **)&d_first, 8, s) != cudaSuccess ||
      (!v.pair && cudaMallocAsync((void **)&scratch, bytes, s) != cudaSuccess)) {
    if (d_first) cudaFreeAsync(d_first, s);
    (void)cudaGetLastError();
    return G4S_OK;
  }
  int *stage = scratch ? scratch : reinterpret_cast<int *>(const_cast<unsigned long long *>(v.pair));
  // (the plan goes with its packed rows: a run after a failure below forms them again)
  const bool pair_was_ready = n->pair_ready, team_was_ready = n->team_ready;
  if (!scratch) n->pair_ready = n->team_ready = false;
  cudaError_t e = cudaMemcpyAsync(stage, idx, bytes, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = launch_first_bad(stage, v, d_first, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&first, d_first, 8, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess && first == ~0ull) {
    drop_plan(n);
    e = cudaMemcpyAsync(const_cast<int *>(v.idx), stage, bytes, cudaMemcpyDeviceToDevice, s);
    *moved = e == cudaSuccess;
  } else if (e == cudaSuccess && !scratch && pair_was_ready) {
    e = launch_pairs(v, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    n->pair_ready = e == cudaSuccess;
    n->team_ready = n->pair_ready && team_was_ready;
  }
  cudaFreeAsync(d_first, s);
  if (scratch) cudaFreeAsync(scratch, s);
  *bad = (size_t)first;
  return e == cudaSuccess ? G4S_OK : cuda_error(e, "table upload");
}

extern "C" {

int g4s_abi_version(void) { return G4S_ABI_VERSION; }

const char *g4s_last_error(void) { return g_last_error.c_str(); }

int g4s_set_device(int32_t device) {
  G4S_CUDA(cudaSetDevice(device));
  return G4S_OK;
}

static int create_net(const g4s_net_desc *desc, cudaMemPool_t pool, g4s_net **out) {
  if (!out) return set_error(G4S_ERR_INVALID, "null output handle");
  *out = nullptr;
  g4s_net *n = nullptr;
  int rc = alloc_net(desc, &n, pool);
  if (rc) return rc;
  if (desc->conn_law == G4S_CONN_GLIBC) {
    const size_t cnt = (size_t)n->v.n * (size_t)n->v.stride;
    std::vector<int32_t> idx;
    std::vector<float> w;
    try {
      idx.resize(cnt);
      w.resize(cnt);
    } catch (...) {
      free_net(n);
      return set_error(G4S_ERR_NOMEM, "host tables");
    }
    rc = conn_glibc_host((unsigned)desc->seed, (int32_t)n->v.n, n->v.nsyn, n->v.stride, idx.data(), w.data());
    if (!rc) rc = g4s_net_load_tables(n, idx.data(), w.data(), n->v.stride);
  } else {
    cudaError_t e = launch_conngen(n->v, desc->self_loops, n->stream);
    if (e != cudaSuccess) rc = cuda_error(e, "connectivity kernel");
    if (!rc) rc = check_status(n, "connectivity kernel");
    if (!rc) rc = finish_tables(n, false);  // (generated rows are in draw order)
  }
  if (!rc) rc = reset_net(n);
  if (rc) {
    free_net(n);
    return rc;
  }
  *out = n;
  return G4S_OK;
}

int g4s_net_create(const g4s_net_desc *desc, g4s_net **out) { return create_net(desc, nullptr, out); }

int g4s_net_create_from_tables(const g4s_net_desc *desc, const int32_t *idx, const float *w, int32_t stride,
                               g4s_net **out) {
  if (!out || !idx || !w) return set_error(G4S_ERR_INVALID, "null argument");
  *out = nullptr;
  g4s_net *n = nullptr;
  int rc = alloc_net(desc, &n);
  if (rc) return rc;
  rc = g4s_net_load_tables(n, idx, w, stride);
  if (!rc) rc = reset_net(n);
  if (rc) {
    free_net(n);
    return rc;
  }
  *out = n;
  return G4S_OK;
}

int g4s_net_load_tables(g4s_net *n, const int32_t *idx, const float *w, int32_t stride) {
  if (!n || !idx || !w) return set_error(G4S_ERR_INVALID, "null argument");
  NetView &v = n->v;
  if (stride != v.stride)
    return set_error(G4S_ERR_INVALID, "table stride must be " + std::to_string(v.stride));
  const size_t cnt = (size_t)v.n * (size_t)v.stride, bytes = cnt * 4;
  // every target must be a neuron of this network or negative (an unused slot), else the first
  // offending entry is reported and the network keeps its tables
  size_t bad = SIZE_MAX;
  bool moved = false;
  int rc = cnt < kHostCheckSlots ? G4S_OK : first_bad_device(n, idx, &bad, &moved);
  if (rc) return rc;
  if (!moved && bad == SIZE_MAX) bad = first_bad_host(idx, cnt, (int32_t)v.n);  // (n < 2^31)
  if (bad != SIZE_MAX)
    return set_error(G4S_ERR_INVALID, "table entry " + std::to_string(bad) + " targets neuron " +
                                          std::to_string(idx[bad]) + " >= n");
  drop_plan(n);
  if (!moved) G4S_CUDA(cudaMemcpyAsync(const_cast<int *>(v.idx), idx, bytes, cudaMemcpyHostToDevice, n->stream));
  G4S_CUDA(cudaMemcpyAsync(const_cast<float *>(v.w), w, bytes, cudaMemcpyHostToDevice, n->stream));
  return finish_tables(n, true);
}

int g4s_net_set_geometry(g4s_net *n, int32_t owner_blocks, int32_t delivery) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  if (owner_blocks < 0) return set_error(G4S_ERR_INVALID, "owner_blocks must be >= 0 (0 = automatic)");
  if (delivery != kDeliverAuto && delivery != kDeliverRun && delivery != kDeliverGroup)
    return set_error(G4S_ERR_INVALID,
                     "delivery must be -1 (automatic), 0 (segment runs) or 1 (eight lanes a spike)");
  n->want_p = owner_blocks;
  n->deliver_mode = delivery;
  n->team_ready = false;
  n->team_ok = true;
  return G4S_OK;
}

int g4s_net_set_block_threads(g4s_net *n, int32_t threads) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  if (threads != 0 && threads != kTeamNT && threads != kTeamNTSmall)
    return set_error(G4S_ERR_INVALID, "threads must be 1024, 768 or 0 (automatic)");
  n->team_nt = threads;
  n->team_ready = false;
  n->team_ok = true;
  return G4S_OK;
}

int g4s_net_get_block_threads(g4s_net *n, int32_t *threads) {
  if (!n || !threads) return set_error(G4S_ERR_INVALID, "null argument");
  const int rc = prepare_team(n);
  if (rc) return rc;
  *threads = n->team_nt_eff;
  return G4S_OK;
}

int g4s_net_get_geometry(g4s_net *n, int32_t *owner_blocks, int64_t *slice) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  int rc = prepare_team(n);
  if (rc) return rc;
  const bool ok = n->team_ok && n->team_ready;
  if (owner_blocks) *owner_blocks = ok ? n->team_p : 0;
  if (slice) *slice = ok ? n->team_rc : 0;
  return G4S_OK;
}

int g4s_net_get_delivery(g4s_net *n, int32_t *delivery) {
  if (!n || !delivery) return set_error(G4S_ERR_INVALID, "null argument");
  const int rc = prepare_team(n);
  if (rc) return rc;
  *delivery = n->team_ok && n->team_ready && n->team_p > 1 ? deliver_mode_of(n) : kDeliverAuto;
  return G4S_OK;
}

int g4s_net_autotune(g4s_net *n, int32_t probe_steps, int32_t *algorithm, int32_t *team, double *us_per_step) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  TuneChoice c;
  double us = 0.0;
  int rc = autotune(n, probe_steps, &c, &us);
  if (rc) return rc;
  if (algorithm) *algorithm = c.alg;
  if (team) *team = c.team;
  if (us_per_step) *us_per_step = us;
  return G4S_OK;
}

int g4s_nets_run(g4s_net **nets, const int32_t *steps, int32_t count, double *device_ms, int64_t *launches) {
  if (!nets || !steps) return set_error(G4S_ERR_INVALID, "null argument");
  return run_nets(nets, steps, count, device_ms, launches);
}

int g4s_net_reset(g4s_net *n) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  return reset_net(n);
}

int g4s_net_run(g4s_net *n, int32_t steps, int32_t algorithm) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  return run_net(n, steps, algorithm);
}

int g4s_net_get_info(g4s_net *n, g4s_net_info *info) {
  if (!n || !info) return set_error(G4S_ERR_INVALID, "null argument");
  info->n = n->v.n;
  info->nsyn = n->v.nsyn;
  info->stride = n->v.stride;
  info->steps_done = n->t_abs;
  info->total_spikes = n->total_spikes;
  info->raster_size = (int64_t)n->rid.n;
  info->last_run_ms = n->last_ms;
  info->last_run_wall_ms = n->last_wall_ms;
  info->last_run_spikes = n->last_spikes;
  info->last_algorithm = n->last_alg;
  info->persistent_blocks = persistent_blocks();
  info->device_bytes = (int64_t)n->device_bytes;
  info->last_run_kernel_ms = n->last_kernel_ms;
  info->last_run_launches = n->last_launches;
  return G4S_OK;
}

int g4s_pinned_alloc(uint64_t bytes, void **out) {
  if (!out) return set_error(G4S_ERR_INVALID, "null output pointer");
  *out = nullptr;
  G4S_CUDA(cudaMallocHost(out, bytes ? (size_t)bytes : 16));
  return G4S_OK;
}

int g4s_pinned_free(void *p) {
  if (p) G4S_CUDA(cudaFreeHost(p));
  return G4S_OK;
}

int g4s_net_raster(g4s_net *n, int32_t *t, int32_t *id, int64_t cap, int64_t *size) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  const int64_t s = (int64_t)n->rid.n;
  if (size) *size = s;
  const int64_t m = std::min(s, cap);
  if (m > 0) {
    if (!t || !id) return set_error(G4S_ERR_INVALID, "null raster buffer");
    raster_copy_out(n, t, id, m);
  }
  return G4S_OK;
}

int g4s_net_counts(g4s_net *n, int32_t *counts, int64_t cap, int64_t *size) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  const int64_t s = (int64_t)n->counts.size();
  if (size) *size = s;
  const int64_t m = std::min(s, cap);
  if (m > 0) {
    if (!counts) return set_error(G4S_ERR_INVALID, "null counts buffer");
    memcpy(counts, n->counts.data(), (size_t)m * 4);
  }
  return G4S_OK;
}

int g4s_net_step_times(g4s_net *n, float *upd, float *step, int64_t cap, int64_t *size) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  const int64_t s = (int64_t)n->upd_ms.size();
  if (size) *size = s;
  const int64_t m = std::min(s, cap);
  if (m > 0) {
    if (upd) memcpy(upd, n->upd_ms.data(), (size_t)m * 4);
    if (step) memcpy(step, n->step_ms.data(), (size_t)m * 4);
  }
  return G4S_OK;
}

int g4s_net_state(g4s_net *n, float *v, float *u, float *i_last, float *a, float *b, float *c, float *d,
                  int32_t *nospks) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  void *const dst[8] = {v, u, i_last, a, b, c, d, nospks};
  unsigned fields = 0;
  for (int k = 0; k < 8; ++k)
    if (dst[k]) fields |= 1u << k;
  if (!fields) return G4S_OK;
  // Blocks of kStateBlock neurons: the device packs a block field by field into the pinned
  // staging buffer (two blocks, one being packed while the other is copied out).  Large
  // networks are copied out by a thread per field: a fresh destination is mostly page faults
  // (N=10^6: 2.5 ms of them on one thread).
  const int64_t N = n->v.n;
  const int nb = (int)((N + kStateBlock - 1) / kStateBlock);
  const int64_t blk = std::min<int64_t>(N, kStateBlock);
  if (need_stage(n, (size_t)blk * 32 * (nb > 1 ? 2 : 1), true) != G4S_OK) {
    // (no pinned memory: field by field out of the device's records, slowly)
    const NetView &w = n->v;
    const struct {
      const void *at;
      size_t pitch;
    } src[8] = {{w.vu, 8},    {&w.vu->y, 8},    {w.ilast, 4},    {w.abcd, 16}, {&w.abcd->y, 16}, {&w.abcd->z, 16},
                {&w.abcd->w, 16}, {w.sstat, sizeof(SpikeStat)}};
    for (int k = 0; k < 8; ++k)
      if (dst[k])
        G4S_CUDA(cudaMemcpy2DAsync(dst[k], 4, src[k].at, src[k].pitch, 4, (size_t)N, cudaMemcpyDeviceToHost, n->stream));
    G4S_CUDA(cudaStreamSynchronize(n->stream));
    return G4S_OK;
  }
  float *const h_state = reinterpret_cast<float *>(n->h_stage);
  float *const half[2] = {h_state, h_state + (nb > 1 ? blk * 8 : 0)};
  auto count = [&](int b) { return (int)std::min<int64_t>(kStateBlock, N - (int64_t)b * kStateBlock); };
  auto copy = [&](int b, int slot, int k) {  // field k, the slot-th of those asked for, of block b
    const size_t cnt = (size_t)count(b);
    memcpy((char *)dst[k] + (size_t)b * kStateBlock * 4, half[b & 1] + (size_t)slot * cnt, cnt * 4);
  };
  std::atomic<int> ready{0}, out[2] = {{0}, {0}};  // blocks packed (-1: give up); fields copied out of each half
  std::vector<std::thread> pool;
  int nf = 0;
  for (int k = 0; k < 8; ++k) nf += dst[k] ? 1 : 0;
  bool threads = nb >= kStateThreadBlocks;
  if (threads) {
    try {
      for (int k = 0, slot = 0; k < 8; ++k)
        if (dst[k])
          pool.emplace_back([&, k, slot = slot++] {
            for (int b = 0; b < nb; ++b) {
              int r;
              while ((r = ready.load(std::memory_order_acquire)) <= b && r >= 0) std::this_thread::yield();
              if (r < 0) return;
              copy(b, slot, k);
              out[b & 1].fetch_add(1, std::memory_order_release);
            }
          });
    } catch (...) {  // (no thread to be had: this one copies)
      ready.store(-1, std::memory_order_release);
      for (auto &t : pool) t.join();
      pool.clear();
      threads = false;
    }
  }
  cudaError_t e = launch_state_pack(n->v, 0, count(0), fields, half[0], n->stream);
  for (int b = 0; b < nb && e == cudaSuccess; ++b) {
    e = cudaStreamSynchronize(n->stream);  // block b is packed
    if (e != cudaSuccess) break;
    if (b + 1 < nb) {
      // (the next block's half is free once block b - 1 has been copied out of it)
      if (threads)
        while (out[(b + 1) & 1].load(std::memory_order_acquire) < nf * ((b + 1) / 2)) std::this_thread::yield();
      e = launch_state_pack(n->v, (int64_t)(b + 1) * kStateBlock, count(b + 1), fields, half[(b + 1) & 1], n->stream);
      if (e != cudaSuccess) break;
    }
    if (threads) {
      ready.store(b + 1, std::memory_order_release);
    } else {
      for (int k = 0, slot = 0; k < 8; ++k)
        if (dst[k]) copy(b, slot++, k);
    }
  }
  if (e != cudaSuccess) ready.store(-1, std::memory_order_release);
  for (auto &t : pool) t.join();
  return e == cudaSuccess ? G4S_OK : cuda_error(e, "reading the neuron state");
}

int g4s_net_currents(g4s_net *n, int64_t *acc) {
  if (!n || !acc) return set_error(G4S_ERR_INVALID, "null argument");
  G4S_CUDA(cudaMemcpyAsync(acc, n->v.acc, (size_t)n->v.n * 8, cudaMemcpyDeviceToHost, n->stream));
  G4S_CUDA(cudaStreamSynchronize(n->stream));
  return G4S_OK;
}

int g4s_net_tables(g4s_net *n, int64_t row0, int64_t nrows, int32_t *idx, float *w) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  if (row0 < 0 || nrows < 0 || row0 + nrows > n->v.n) return set_error(G4S_ERR_INVALID, "row range");
  const size_t off = (size_t)row0 * (size_t)n->v.stride, cnt = (size_t)nrows * (size_t)n->v.stride;
  if (idx) G4S_CUDA(cudaMemcpyAsync(idx, n->v.idx + off, cnt * 4, cudaMemcpyDeviceToHost, n->stream));
  if (w) G4S_CUDA(cudaMemcpyAsync(w, n->v.w + off, cnt * 4, cudaMemcpyDeviceToHost, n->stream));
  G4S_CUDA(cudaStreamSynchronize(n->stream));
  return G4S_OK;
}

int g4s_net_stats(g4s_net *n, double *rate_hz, double *isi_cv, int64_t *total_spikes) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  double h[2] = {0, 0};
  G4S_CUDA(cudaMemsetAsync(n->d_stats, 0, 16, n->stream));
  G4S_CUDA(launch_stats(n->v, n->d_stats, n->stream));
  G4S_CUDA(cudaMemcpyAsync(h, n->d_stats, 16, cudaMemcpyDeviceToHost, n->stream));
  G4S_CUDA(cudaStreamSynchronize(n->stream));
  if (rate_hz) *rate_hz = n->t_abs ? (double)n->total_spikes * 1000.0 / ((double)n->v.n * (double)n->t_abs) : 0.0;
  if (isi_cv) *isi_cv = h[1] > 0 ? h[0] / h[1] : 0.0;
  if (total_spikes) *total_spikes = n->total_spikes;
  return G4S_OK;
}

int g4s_net_set_barrier_timeout(g4s_net *n, uint64_t ns) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  n->barrier_ns = ns;
  return G4S_OK;
}

int g4s_inject_fault(g4s_net *n, int32_t kind) {
  if (kind == G4S_FAULT_ALLOC) {
    g_fail_next_alloc.store(1);
    return G4S_OK;
  }
  if (kind == G4S_FAULT_BARRIER_STALL) {
    if (!n) return set_error(G4S_ERR_INVALID, "null handle");
    n->barrier_stall = 1;
    return G4S_OK;
  }
  return set_error(G4S_ERR_INVALID, "unknown fault kind");
}

int g4s_net_destroy(g4s_net *n) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  free_net(n);
  return G4S_OK;
}

int g4s_net_write_results(g4s_net *n, const char *dir, const float *init_state, double elapsed_ms,
                          double elapsed_with_data_ms) {
  (void)init_state;
  if (!n || !dir) return set_error(G4S_ERR_INVALID, "null argument");
  return write_results(n, dir, elapsed_ms, elapsed_with_data_ms);
}

int g4s_run_protocol(int32_t n, int32_t nsyn, int32_t iterations, int32_t algorithm, int32_t mode, uint64_t seed,
                     int32_t conn_law, const char *results_root) {
  if (!results_root) return set_error(G4S_ERR_INVALID, "null results root");
  if (iterations < 0) return set_error(G4S_ERR_INVALID, "iterations must be >= 0");
  if (algorithm < -1 || algorithm > kAlgAuto) return set_error(G4S_ERR_INVALID, "algorithm must be -1..5");
  if (mode < -1 || mode > 2) return set_error(G4S_ERR_INVALID, "mode must be -1..2");
  g4s_net_desc d{};
  d.n = n;
  d.nsyn = nsyn;
  d.exc_permille = 800;
  d.self_loops = conn_law == G4S_CONN_GLIBC ? 1 : 0;
  d.conn_law = conn_law;
  d.seed = seed;
  d.drive_scale = 1.0f;
  d.record_raster = 1;
  g4s_net *net = nullptr;
  int rc = g4s_net_create(&d, &net);
  if (rc) return rc;
  static const float kModeScale[3] = {0.5f, 1.0f, 1.5f};
  for (int m = 0; m < 3; ++m) {
    if (mode >= 0 && m != mode) continue;
    for (int a = 0; a < 5; ++a) {
      const int alg = algorithm < 0 ? a : algorithm;
      if (algorithm >= 0 && a > 0) break;
      net->desc.drive_scale = kModeScale[m];
      if ((rc = reset_net(net))) break;
      char sub[256];
      snprintf(sub, sizeof sub, "/Results/N%dNsyn%dRegime%dAlg%d/", n, nsyn, m, alg);
      const auto w0 = std::chrono::steady_clock::now();
      if ((rc = run_net(net, iterations, alg))) break;
      const double ewd = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - w0).count();
      if ((rc = write_results(net, std::string(results_root) + sub, net->last_ms, ewd))) break;
      printf("Regime %d Alg %d: %d steps, %lld spikes, %.3f ms device, %.3f ms with data\n", m, alg, iterations,
             (long long)net->total_spikes, net->last_ms, ewd);
    }
    if (rc) break;
  }
  g4s_net_destroy(net);
  return rc;
}

int g4s_conn_glibc(uint32_t seed, int32_t n, int32_t nsyn, int32_t stride, int32_t *idx, float *w) {
  if (!idx || !w) return set_error(G4S_ERR_INVALID, "null table buffer");
  return conn_glibc_host(seed, n, nsyn, stride, idx, w);
}

int g4s_net_stream_raster(g4s_net *n, const char *path) {
  if (!n) return set_error(G4S_ERR_INVALID, "null handle");
  if (n->rstream) {
    RasterFile *f = n->rstream;
    n->rstream = nullptr;
    int rc = raster_close(f);
    if (rc) return rc;
  }
  if (!path) return G4S_OK;
  if (!n->desc.record_raster) return set_error(G4S_ERR_STATE, "the raster is not recorded (record_raster = 0)");
  return raster_open(path, n->v.n, n->t_abs, &n->rstream);
}

int g4s_net_write_raster_file(g4s_net *n, const char *path) {
  if (!n || !path) return set_error(G4S_ERR_INVALID, "null argument");
  if (n->rid.n != (size_t)n->total_spikes || n->counts.size() != (size_t)n->t_abs)
    return set_error(G4S_ERR_STATE, "the host raster does not hold every step since the reset "
                                    "(not recorded, or streamed to a file)");
  return raster_write_all(path, n->v.n, 0, n->counts, n->rid.p, n->rid.n);
}

int g4s_net_save_tables(g4s_net *n, const char *path) {
  if (!n || !path) return set_error(G4S_ERR_INVALID, "null argument");
  const size_t cnt = (size_t)n->v.n * (size_t)n->v.stride;
  std::vector<int32_t> idx;
  std::vector<float> w;
  try {
    idx.resize(cnt);
    w.resize(cnt);
  } catch (...) {
    return set_error(G4S_ERR_NOMEM, "host tables");
  }
  int rc = g4s_net_tables(n, 0, n->v.n, idx.data(), w.data());
  if (rc) return rc;
  TableHeader h{};
  h.n = n->v.n;
  h.nsyn = n->v.nsyn;
  h.stride = n->v.stride;
  h.seed = n->desc.seed;
  h.conn_law = n->desc.conn_law;
  h.self_loops = n->desc.self_loops;
  h.exc_permille = n->desc.exc_permille;
  h.flags = 1;
  return tables_write(path, h, idx.data(), w.data());
}

int g4s_net_create_from_file(const g4s_net_desc *desc, const char *path, g4s_net **out) {
  if (!desc || !path || !out) return set_error(G4S_ERR_INVALID, "null argument");
  *out = nullptr;
  TableHeader h{};
  int rc = tables_read_header(path, &h);
  if (rc) return rc;
  if (h.n != desc->n || h.nsyn != desc->nsyn)
    return set_error(G4S_ERR_INVALID, std::string(path) + " holds a network of n=" + std::to_string(h.n) +
                                          ", nsyn=" + std::to_string(h.nsyn));
  const size_t cnt = (size_t)h.n * (size_t)h.stride;
  std::vector<int32_t> idx;
  std::vector<float> w;
  try {
    idx.resize(cnt);
    w.resize(cnt);
  } catch (...) {
    return set_error(G4S_ERR_NOMEM, "host tables");
  }
  if ((rc = tables_read(path, h, idx.data(), w.data()))) return rc;
  return g4s_net_create_from_tables(desc, idx.data(), w.data(), h.stride, out);
}

}  // extern "C"

namespace g4s {
int net_create_pooled(const g4s_net_desc *desc, cudaMemPool_t pool, g4s_net **out) {
  return create_net(desc, pool, out);
}
}  // namespace g4s
