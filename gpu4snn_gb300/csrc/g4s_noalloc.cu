// g4s_noalloc.cu — g4s_run_noalloc: the SKL team kernel on caller-owned device arrays,
// without any allocation.
//
// Some callers cannot call cudaMalloc while they step a network: real-time loops that
// must not pay the device-wide synchronisation an allocation or a free may imply, and
// hosts whose device memory is owned by a capped pool that this library cannot draw
// from.  For them this entry point uses only memory it already has: the caller passes the
// network's arrays and the output buffers, and the kernel's scratch (the team's per-step
// spike records and overflow ids, the per-row segment table of a multi-CTA team, the error
// word and the work-queue words) lives in one file-scope __device__ array of fixed size,
// which every GPU that loads the library holds until the process exits.  The call copies
// nothing from host memory: the launch descriptor reaches the device as a kernel argument.
//
// Limits: at most kNoAllocMaxNeurons neurons and kNoAllocMaxTeam CTAs, and at most 16384
// neurons per CTA (the shared-memory slice of the team kernel).  Every call shares the
// scratch array and leaves its contents behind; calls that overlap on the GPU (on
// different streams, or without ordering between them) race on it and must not be made.
// A multi-CTA call rebuilds the per-row segment table from the caller's tables (a search of
// every row, reading 32 targets and 32 per team boundary of a row of 1000),
// since it cannot know whether they changed since the last call.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>

#include "../../include/gpu4snn.h"
#include "g4s_internal.h"

using namespace g4s;

namespace {

constexpr int64_t kNoAllocMaxNeurons = 131072;
constexpr int kNoAllocMaxTeam = 8;
constexpr int64_t kNoAllocMaxSlice = 16384;

// Layout of the scratch array.
constexpr size_t kOffSync = 0;                                       // GridSync (128 B): error word
constexpr size_t kOffRec = 128;                                      // spike records: [2][team][2 x 16] u64
constexpr size_t kOffCtl = kOffRec + 2 * kNoAllocMaxTeam * kRecLines * 128;  // int[5]: -, queue head, status, -, next tag
constexpr size_t kOffSlots = kOffCtl + 128;                          // int2[kNoAllocMaxTeam]
constexpr size_t kOffItem = kOffSlots + 256;                         // TeamItem
constexpr size_t kOffList = 16384;                                   // u64[2][kNoAllocMaxNeurons]: spikes beyond a record
constexpr size_t kOffSeg = kOffList + 2 * kNoAllocMaxNeurons * 8;  // u16[kNoAllocMaxNeurons][kNoAllocMaxTeam + 1]
constexpr size_t kScratchBytes = kOffSeg + (size_t)kNoAllocMaxNeurons * (kNoAllocMaxTeam + 1) * 2;

static_assert(sizeof(GridSync) <= kOffRec - kOffSync, "error word");
static_assert(sizeof(int2) * kNoAllocMaxTeam <= kOffItem - kOffSlots, "slots");
static_assert(sizeof(TeamItem) <= kOffList - kOffItem, "item");
static_assert(kNoAllocMaxTeam <= 32, "one setup thread per slot");
// about 4.5 MB: the documented size of the array in gpu4snn.h
static_assert(kScratchBytes > 4400000 && kScratchBytes < 4600000, "scratch size as documented");

// Everything a call needs before the team kernel, in one launch: the work-queue words, the
// team's slots and the launch descriptor (which arrives by value as a kernel argument, so the
// call stages nothing through host memory), cleared counts, status and error words, and the
// team's segment table.  The records and id lists keep the words of earlier calls: their tags
// go on from call to call (a device word, so that a captured call replays), and no stale word
// carries a tag that is still to come; they are cleared when the tags would wrap.  (As three
// memsets, two kernels and a copy of the status word these took 20 us of a 34 us call of one
// step of N=2,500.)
//
// Segment table, a warp per row: 32 probes at a time narrow every boundary's range 32-fold, the
// first probes shared by all of them (rows of 1000: two dependent loads in place of ten).
constexpr int kSetupNT = 256;
__global__ void __launch_bounds__(kSetupNT) k_noalloc_setup(TeamItem item, int *ctl, int2 *slots, TeamItem *dst,
                                                            uint16_t *seg, int64_t scratch_words) {
  const int T = item.team;
  if (blockIdx.x == 0) {
    __shared__ unsigned s_tag;
    __shared__ int s_wrap;
    if (threadIdx.x == 0) {
      unsigned *next = reinterpret_cast<unsigned *>(ctl + 4);
      s_wrap = (unsigned long long)*next + (unsigned)item.steps + 2ull >= 0xFFFFFFFFull;
      s_tag = s_wrap ? 0u : *next;
      *next = s_tag + (unsigned)item.steps;
      ctl[1] = 0;  // queue head
      *item.v.status = 0;
      item.sync->error = 0;
      item.tag0 = s_tag;
      *dst = item;
    }
    if ((int)threadIdx.x < T) slots[threadIdx.x] = make_int2(0, (int)threadIdx.x);
    __syncthreads();
    if (s_wrap) {
      for (int k = threadIdx.x; k < 2 * kNoAllocMaxTeam * kRecLines * kRecWords; k += kSetupNT) item.rec[k] = 0ull;
      for (int64_t k = threadIdx.x; k < scratch_words; k += kSetupNT) item.list[k] = 0ull;
    }
  }
  for (int k = blockIdx.x * kSetupNT + threadIdx.x; k < item.steps; k += gridDim.x * kSetupNT) item.v.counts[k] = 0;
  if (T == 1) return;
  const int lane = threadIdx.x & 31, stride = item.v.stride;
  const int64_t nwarps = (int64_t)gridDim.x * (kSetupNT / 32);
  for (int64_t row = (int64_t)blockIdx.x * (kSetupNT / 32) + (threadIdx.x >> 5); row < item.v.n; row += nwarps) {
    const unsigned *ri = reinterpret_cast<const unsigned *>(item.v.idx) + row * stride;
    int lo[kNoAllocMaxTeam], len[kNoAllocMaxTeam];  // where boundary k + 1 lies
    const int step0 = (stride + 31) >> 5;
    const unsigned t0 = lane * step0 < stride ? ri[lane * step0] : 0xFFFFFFFFu;
    int most = 0;
#pragma unroll
    for (int k = 0; k < kNoAllocMaxTeam; ++k) {
      const int c = __popc(__ballot_sync(0xFFFFFFFFu, t0 < (unsigned)(k + 1) * (unsigned)item.rc));
      lo[k] = c ? (c - 1) * step0 + 1 : 0;
      len[k] = c && k < T ? min(stride, c * step0) - lo[k] : 0;
      most = max(most, len[k]);
    }
    while (most > 0) {
      most = 0;
      unsigned t[kNoAllocMaxTeam];
#pragma unroll
      for (int k = 0; k < kNoAllocMaxTeam; ++k) {
        const int at = lane * ((len[k] + 31) >> 5);
        t[k] = at < len[k] ? ri[lo[k] + at] : 0xFFFFFFFFu;
      }
#pragma unroll
      for (int k = 0; k < kNoAllocMaxTeam; ++k) {
        const int step = (len[k] + 31) >> 5;
        const int c = __popc(__ballot_sync(0xFFFFFFFFu, t[k] < (unsigned)(k + 1) * (unsigned)item.rc));
        const int end = c ? min(lo[k] + len[k], lo[k] + c * step) : lo[k];
        if (c) lo[k] += (c - 1) * step + 1;
        len[k] = end - lo[k];
        most = max(most, len[k]);
      }
    }
    uint16_t *so = seg + row * (T + 1);
    if (lane == 0) so[0] = 0;
#pragma unroll
    for (int k = 0; k < kNoAllocMaxTeam; ++k)
      if (lane == k && k < T) so[k + 1] = (uint16_t)lo[k];
  }
}

}  // namespace

// The scratch of g4s_run_noalloc (about 4.5 MB per GPU, held until exit).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

// In host code g_noalloc_scratch names a host-side stand-in, not device memory: its
// device address is looked up once per device, with that device current, and cached, and
// with it the device's SMs.
static std::mutex g_scratch_mu;
static void *g_scratch_dev[256];
static int g_scratch_sms[256];

static int scratch_address(unsigned char **out, int *sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
  if (dev < 0 || dev >= 256) return set_error(G4S_ERR_CUDA, "device index out of range");
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (!g_scratch_dev[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) return cuda_error(e, "cudaGetSymbolAddress of the no-alloc scratch");
    // once per device, outside any stream capture of the caller's launches
    if ((e = team_smem_ceiling()) != cudaSuccess) return cuda_error(e, "team kernel shared-memory ceiling");
    e = cudaDeviceGetAttribute(&g_scratch_sms[dev], cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return cuda_error(e, "cudaDeviceGetAttribute");
    g_scratch_dev[dev] = p;
  }
  *sms = g_scratch_sms[dev];
  *out = static_cast<unsigned char *>(g_scratch_dev[dev]);
  return G4S_OK;
}

extern "C" int g4s_run_noalloc(const g4s_dev_net *d, int64_t t_abs0, int32_t steps, int32_t team, int32_t last,
                               int32_t *d_counts, int64_t *d_base, int32_t *d_raster, int64_t raster_cap,
                               int32_t *d_status, void *stream) {
  if (!d) return set_error(G4S_ERR_INVALID, "null network");
  if (d->n < 2 || d->n > kNoAllocMaxNeurons)
    return set_error(G4S_ERR_INVALID, "g4s_run_noalloc: n must be in [2, " + std::to_string(kNoAllocMaxNeurons) +
                                          "], got " + std::to_string(d->n));
  if (team < 1 || team > kNoAllocMaxTeam)
    return set_error(G4S_ERR_INVALID, "g4s_run_noalloc: team must be in [1, " + std::to_string(kNoAllocMaxTeam) +
                                          "], got " + std::to_string(team));
  const int64_t rc = (d->n + team - 1) / team;
  if (rc > kNoAllocMaxSlice || team_smem(rc, team) == 0)
    return set_error(G4S_ERR_INVALID, "g4s_run_noalloc: more than " + std::to_string(kNoAllocMaxSlice) +
                                          " neurons per CTA; use a larger team");
  if (d->nsyn < 1 || d->stride < d->nsyn || d->stride % 4 != 0 || d->stride > kMaxSortedNsyn)
    return set_error(G4S_ERR_INVALID, "g4s_run_noalloc: need 1 <= nsyn <= stride <= 16384, stride % 4 == 0");
  if (d->nexc < 0 || d->nexc > d->n) return set_error(G4S_ERR_INVALID, "g4s_run_noalloc: bad nexc");
  if (steps < 0 || t_abs0 < 0 || t_abs0 + steps > (int64_t)INT32_MAX)
    return set_error(G4S_ERR_INVALID, "g4s_run_noalloc: bad step range");
  if (!d->vu || !d->abcd || !d->acc || !d->i_last || !d->spike_stat || !d->idx || !d->w)
    return set_error(G4S_ERR_INVALID, "g4s_run_noalloc: null network array");
  if (steps > 0 && (!d_counts || !d_base)) return set_error(G4S_ERR_INVALID, "g4s_run_noalloc: null counts/base");
  if (raster_cap < 0 || (raster_cap > 0 && !d_raster))
    return set_error(G4S_ERR_INVALID, "g4s_run_noalloc: bad raster buffer");
  if (steps == 0) return G4S_OK;

  unsigned char *scr = nullptr;
  int sms = 1;
  int rc0 = scratch_address(&scr, &sms);
  if (rc0) return rc0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  GridSync *sync = reinterpret_cast<GridSync *>(scr + kOffSync);
  int *ctl = reinterpret_cast<int *>(scr + kOffCtl);
  int2 *slots = reinterpret_cast<int2 *>(scr + kOffSlots);
  TeamItem *item = reinterpret_cast<TeamItem *>(scr + kOffItem);
  unsigned long long *list = reinterpret_cast<unsigned long long *>(scr + kOffList);
  uint16_t *seg = reinterpret_cast<uint16_t *>(scr + kOffSeg);

  TeamItem h{};
  NetView &v = h.v;
  v.n = d->n;
  v.nexc = d->nexc;
  v.nsyn = d->nsyn;
  v.stride = d->stride;
  v.seed = d->seed;
  v.ge = d->ge;
  v.gi = d->gi;
  v.vu = static_cast<float2 *>(d->vu);
  v.abcd = static_cast<float4 *>(d->abcd);
  v.acc = reinterpret_cast<long long *>(d->acc);
  v.ilast = d->i_last;
  v.sstat = static_cast<SpikeStat *>(d->spike_stat);
  v.idx = d->idx;
  v.w = d->w;
  v.raster = d_raster;
  v.raster_cap = raster_cap;
  v.counts = d_counts;
  v.base = reinterpret_cast<long long *>(d_base);
  v.stamps = nullptr;
  v.status = d_status ? d_status : ctl + 2;
  h.seg = seg;
  h.list = list;
  h.rec = reinterpret_cast<unsigned long long *>(scr + kOffRec);
  h.t_abs0 = t_abs0;
  h.steps = steps;
  h.last = last ? 1 : 0;
  h.team = team;
  h.rc = (int)rc;
  h.sync = sync;
  const int64_t rows = team > 1 ? (d->n + kSetupNT / 32 - 1) / (kSetupNT / 32) : 1;
  k_noalloc_setup<<<(unsigned)std::min<int64_t>(rows, 16 * sms), kSetupNT, 0, s>>>(h, ctl, slots, item, seg,
                                                                                    2 * kNoAllocMaxNeurons);
  cudaError_t e = cudaGetLastError();
  // (768 threads for slices whose state lives in shared memory, as for small steps elsewhere)
  if (e == cudaSuccess)
    e = launch_team(item, slots, team, ctl + 1, team, team_smem(rc, team), 2000000000ull, 0, s, false, kDeliverRun, team == 1,
                    rc <= kVuSlice ? kTeamNTSmall : kTeamNT);
  if (e != cudaSuccess) return cuda_error(e, "g4s_run_noalloc launch");
  return G4S_OK;
}
