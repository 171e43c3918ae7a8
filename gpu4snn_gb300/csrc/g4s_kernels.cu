// g4s_kernels.cu — sm_103a kernels of one network's simulation step, and their launchers.
//
//   k_init_state   neuron parameters and initial state        (initNeuron, gpu4snn.cu:286-320)
//   k_conngen      distinct-target tables, Philox law          (host generator, gpu4snn.cu:873-905)
//   k_persistent   the steps of a chunk of the N, S, AP and AB schemes (and of SKL where the team
//                  kernel does not fit): update (stateupdate, gpu4snn.cu:334-417) and delivery in
//                  one cooperative launch with timed grid barriers (k_update and k_deliver, two
//                  launches a step, for S where steps have many synapses):
//                    N  a warp per spiking neuron              (deliverspks1, gpu4snn.cu:420-443)
//                    S  flat over the step's synapses          (deliverspks2, gpu4snn.cu:446-467)
//                    AP thread group per spiking row           (propagatespikes, gpu4snn.cu:323-331)
//                    AB flat over the step's synapses          (AB_deliverspks, gpu4snn.cu:554-584)
//   k_state_pack   the neuron record for the host
//   k_stats        FP64 firing rate and ISI CV reductions
//
// Delivery reads the compacted spike list of the step (int32 ids), streams each spiking row
// with 128-bit evict-first loads (int32 targets, fp32 weights) and adds Q32.32 weights into
// the L2-resident current array with red.global.add.u64, so the result does not depend on
// the order of the additions.
#include <cuda_runtime.h>

#include <algorithm>

#include <cstdio>

#include "g4s_device.cuh"
#include "g4s_internal.h"

namespace g4s {

// ---------------------------------------------------------------------------------------
// Initial state.
// ---------------------------------------------------------------------------------------
__global__ void k_init_state(NetView v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < v.n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float r = izh_r(v.seed, i);
    const float4 p = izh_abcd(r, i < v.nexc);
    v.abcd[i] = p;
    if (v.rpar) v.rpar[i] = r;
    v.vu[i] = make_float2(-65.0f, __fmul_rn(p.y, -65.0f));
    v.acc[i] = 0;
    v.ilast[i] = 0.0f;
    SpikeStat s;
    s.nospks = 0;
    s.last = -1;
    s.nisi = 0;
    s.pad = 0;
    s.s1 = 0;
    s.s2 = 0;
    v.sstat[i] = s;
  }
}

// ---------------------------------------------------------------------------------------
// Connectivity.  One warp per row keeps the row's accepted targets in a shared-memory set:
// a bitmap of the n targets when that is the smaller (bits > 0 words), else an
// open-addressing hash of 2^log2h ints.  Draws are consumed in the order the oracle
// defines: block b, word r, lane l is draw 128b + 32r + l.  Within one word round, a draw
// is fresh iff its target is not in the set and no lower lane drew the same target
// (__match_any_sync: only the lowest such lane inserts); fresh draws are accepted in lane
// order until the row holds nsyn targets.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ bool set_insert(int *set, unsigned mask, int log2h, int t) {
  unsigned h = ((unsigned)t * 0x9E3779B1u) >> (32 - log2h);
  for (unsigned probe = 0; probe <= mask; ++probe) {
    const int old = atomicCAS(set + h, -1, t);
    if (old == -1) return true;
    if (old == t) return false;
    h = (h + 1) & mask;
  }
  return false;  // unreachable: the set is sized for twice the row plus one round
}

__device__ __forceinline__ bool bit_insert(int *bits, int t) {
  const unsigned b = 1u << (t & 31);
  return (atomicOr(reinterpret_cast<unsigned *>(bits) + (t >> 5), b) & b) == 0u;
}

__global__ void k_conngen(NetView v, int self_loops, int log2h, int bits, int64_t row0, int64_t nrows,
                          unsigned long long max_blocks) {
  extern __shared__ __align__(16) int s_set[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const unsigned hsize = 1u << log2h, mask = hsize - 1;
  const unsigned words = bits > 0 ? (unsigned)bits : hsize;  // (a multiple of 4)
  int *set = s_set + (size_t)wib * words;
  const int fill = bits > 0 ? 0 : -1;
  const uint64_t range = self_loops ? (uint64_t)v.n : (uint64_t)(v.n - 1);
  const float wscale = __fdiv_rn(1000.0f, (float)v.nsyn);
  for (int64_t rr = (int64_t)blockIdx.x * wpb + wib; rr < nrows; rr += (int64_t)gridDim.x * wpb) {
    const int64_t row = row0 + rr;
    int *ri = const_cast<int *>(v.idx) + row * v.stride;
    float *rw = const_cast<float *>(v.w) + row * v.stride;
    for (unsigned j = lane; j < words / 4; j += 32) reinterpret_cast<int4 *>(set)[j] = make_int4(fill, fill, fill, fill);
    __syncwarp();
    int accepted = 0;
    for (unsigned long long b = 0; accepted < v.nsyn; ++b) {
      if (b >= max_blocks) {
        if (lane == 0) atomicCAS(v.status, 0, kErrConnCode);
        break;
      }
      const U64x4 o = philox(v.seed, kStreamConn, (uint64_t)row, 32ull * b + lane, 0);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        uint64_t t = __umul64hi(o.x[r], range);
        if (!self_loops && t >= (uint64_t)row) t += 1;
        const int ti = (int)t;
        const unsigned same = __match_any_sync(0xFFFFFFFFu, ti);
        const bool leader = (__ffs(same) - 1) == lane;
        bool fresh = false;
        if (leader) fresh = bits > 0 ? bit_insert(set, ti) : set_insert(set, mask, log2h, ti);
        const unsigned fb = __ballot_sync(0xFFFFFFFFu, fresh);
        const int pos = accepted + __popc(fb & ((1u << lane) - 1u));
        if (fresh && pos < v.nsyn) ri[pos] = ti;
        accepted += __popc(fb);
        __syncwarp();
        if (accepted >= v.nsyn) break;
      }
    }
    const float sc = row < v.nexc ? __fmul_rn(wscale, 0.5f) : __fmul_rn(wscale, -1.0f);
    for (int j = lane * 4; j < v.nsyn; j += 128) {
      const U64x4 o = philox(v.seed, kStreamWeight, (uint64_t)row, (uint64_t)(j >> 2), 0);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (j + q < v.nsyn) rw[j + q] = __fmul_rn(sc, u24(o.x[q]));
    }
    for (int j = v.nsyn + lane; j < v.stride; j += 32) {
      ri[j] = -1;
      rw[j] = 0.0f;
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------
// The step loop of the schemes that add into global memory: every step of a chunk in one
// cooperative launch.  Per step: update and compaction of the spikes into the raster, grid
// barrier, delivery, grid barrier.  Bound by the two barriers and the chain of global round
// trips between them for small networks, by the L2's additions for large ones.  (Two
// launches a step instead took 8.5 us of host time, or 6.1 us a step as a captured graph,
// for N=2,500.)
//
// The drive of a thread's first neuron is drawn while it waits at the second barrier.
// ---------------------------------------------------------------------------------------
// The update of a block's neurons (tiles of NT, every gridDim.x-th), the next tile's state in
// flight while a tile's drive is drawn (1024 threads an SM so, 64 registers each: N=10^6 at
// drive 0.5 22.1 us a step against 23.9 with 1536 and nothing in flight); spikes are collected in
// shared memory and appended to the raster at base_t with one global atomic per kSpikeTiles
// tiles.  z0: the drive of the block's first tile (kDrawn; else it is drawn here).  Returns
// the block's spikes.
constexpr int kSpikeTiles = 8;
template <int NT, bool kDrawn>
__device__ __forceinline__ unsigned update_phase(const NetView &v, int lt, int64_t t_abs, long long base_t, bool last,
                                                 float z0, int *s_ids, int *s_n, long long *s_slot) {
  unsigned mine = 0;
  const int64_t tiles = (v.n + NT - 1) / NT;
  for (int64_t g = blockIdx.x; g < tiles; g += (int64_t)gridDim.x * kSpikeTiles) {
    const int64_t end = min(tiles, g + (int64_t)gridDim.x * kSpikeTiles);
    int64_t i = g * NT + threadIdx.x;
    float2 sn = make_float2(0.0f, 0.0f);
    float rn = 0.0f;
    long long an = 0;
    if (i < v.n) {
      sn = v.vu[i];
      rn = v.rpar[i];
      an = __ldcg(v.acc + i);
    }
    for (int64_t tile = g; tile < end; tile += gridDim.x, i += (int64_t)gridDim.x * NT) {
      if (i < v.n) {
        float2 s = sn;
        const float r = rn;
        const long long a = an;
        const int64_t in = i + (int64_t)gridDim.x * NT;
        if (in < v.n && tile + gridDim.x < end) {
          sn = v.vu[in];
          rn = v.rpar[in];
          an = __ldcg(v.acc + in);
        }
        const float z = kDrawn && tile == blockIdx.x ? z0 : normal(v.seed, (uint64_t)i, (uint64_t)t_abs);
        float I;
        const bool spk = izh_step(s.x, s.y, I, izh_abcd(r, i < v.nexc), i < v.nexc ? v.ge : v.gi, z, q32_current(a));
        v.vu[i] = s;
        if (a != 0) v.acc[i] = 0;  // (written back only when it was non-zero)
        if (last) v.ilast[i] = I;
        if (spk) {
          s_ids[atomicAdd(s_n, 1)] = (int)i;
          SpikeStat st = v.sstat[i];
          st.nospks += 1;
          if (st.last >= 0) {
            const long long isi = t_abs - st.last;
            st.nisi += 1;
            st.s1 += isi;
            st.s2 += isi * isi;
          }
          st.last = (int)t_abs;
          v.sstat[i] = st;
        }
      }
    }
    __syncthreads();
    const int total = *s_n;
    if (total) {  // (the same for the whole block)
      if (threadIdx.x == 0) *s_slot = base_t + atomicAdd(v.counts + lt, total);
      __syncthreads();
      for (int k = threadIdx.x; k < total; k += NT) {
        const long long pos = *s_slot + k;
        if (pos < v.raster_cap)
          v.raster[pos] = s_ids[k];
        else
          atomicCAS(v.status, 0, kErrOverflowCode);
      }
      mine += total;
      __syncthreads();
      if (threadIdx.x == 0) *s_n = 0;
    }
    __syncthreads();
  }
  return mine;
}

// Groups of `group` consecutive threads take whole spiking rows (N, AP), four vectors a thread
// in flight: a thread's share of a row is a chain of loads otherwise (us a step with one and
// with four: N=2,500 x 1000 N 7.3, 6.5, AP 6.1, 5.7; 20,000 x 1000 at drive 1.5 N 12.4, 9.7, AP
// 10.1, 8.7).
__device__ __forceinline__ void deliver_groups(const NetView &v, const int *list, int K, int group) {
  const uint32_t rv = (uint32_t)(v.stride >> 2);
  const int gpb = blockDim.x / group;
  const int lig = threadIdx.x % group;
  const int64_t ngroups = (int64_t)gridDim.x * gpb;
  // (consecutive rows to different blocks: a step's few rows spread over the SMs)
  for (int64_t q = (int64_t)(threadIdx.x / group) * gridDim.x + blockIdx.x; q < K; q += ngroups) {
    const int row = __ldcg(list + q);
    for (uint32_t j = lig; j < rv; j += 4 * group) {
      Vec4 x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = load_vec(v, row, j + u * group < rv ? j + u * group : j);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j + u * group < rv) deliver4(v.acc, x[u].t, x[u].w);
    }
  }
}

// The barrier's counter carries the chunk's spikes so far in its high half: past the step's
// first barrier every block knows the step's count.  group: threads per spiking row, 0 = flat.
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_persistent(NetView v, int64_t t_abs0, int nsteps, int last_chunk,
                                                      GridSync *gs, unsigned long long limit_ns, int group,
                                                      int stall) {
  __shared__ int s_ids[kSpikeTiles * NT];
  __shared__ int s_n;
  __shared__ long long s_slot;
  unsigned epoch = 0;
  long long base = 0;
  const unsigned nb = gridDim.x + (unsigned)stall;  // stall > 0 only under fault injection
  const int64_t first = (int64_t)blockIdx.x * NT + threadIdx.x;
  float z0 = first < v.n ? normal(v.seed, (uint64_t)first, (uint64_t)t_abs0) : 0.0f;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  for (int lt = 0; lt < nsteps; ++lt) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      v.base[lt] = base;
      v.stamps[2 * lt] = globaltimer();
    }
    const unsigned mine =
        update_phase<NT, true>(v, lt, t_abs0 + lt, base, last_chunk && lt == nsteps - 1, z0, s_ids, &s_n, &s_slot);
    grid_arrive(gs, epoch, mine);
    unsigned spikes;
    if (!grid_wait(gs, epoch, nb, limit_ns, spikes)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) v.stamps[2 * lt + 1] = globaltimer();
    const int K = (int)(spikes - (unsigned)base);
    const int *list = v.raster + base;
    if (group > 0)
      deliver_groups(v, list, K, group);
    else
      deliver_flat(v, list, K);
    grid_arrive(gs, epoch, 0u);
    if (first < v.n && lt + 1 < nsteps) z0 = normal(v.seed, (uint64_t)first, (uint64_t)(t_abs0 + lt + 1));
    if (!grid_wait(gs, epoch, nb, limit_ns, spikes)) return;
    base += K;
  }
}

// A step as two launches: the update, and a flat delivery with a grid sized for its work.
template <int NT>
__global__ void __launch_bounds__(NT) k_update(NetView v, int64_t t_abs0, int lt, int last) {
  __shared__ int s_ids[kSpikeTiles * NT];
  __shared__ int s_n;
  __shared__ long long s_slot;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  const long long base_t = lt == 0 ? 0ll : __ldcg(v.base + lt - 1) + __ldcg(v.counts + lt - 1);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    v.base[lt] = base_t;
    v.stamps[2 * lt] = globaltimer();
  }
  update_phase<NT, false>(v, lt, t_abs0 + lt, base_t, last != 0, 0.0f, s_ids, &s_n, &s_slot);
}

__global__ void k_deliver(NetView v, int lt) {
  if (blockIdx.x == 0 && threadIdx.x == 0) v.stamps[2 * lt + 1] = globaltimer();
  deliver_flat(v, v.raster + __ldcg(v.base + lt), __ldcg(v.counts + lt));
}

// ---------------------------------------------------------------------------------------
// FP64 statistics: sum of per-neuron ISI CVs and the number of neurons with >= 2 ISIs.
// ---------------------------------------------------------------------------------------
__global__ void k_stats(NetView v, double *out) {
  double cv = 0.0, cnt = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < v.n; i += (int64_t)gridDim.x * blockDim.x) {
    const SpikeStat s = v.sstat[i];
    if (s.nisi >= 2) {
      const double m = (double)s.nisi;
      const double mean = (double)s.s1 / m;
      const double var = (double)((long long)s.nisi * s.s2 - s.s1 * s.s1) / (m * m);
      cv += sqrt(var) / mean;
      cnt += 1.0;
    }
  }
  for (int o = 16; o; o >>= 1) {
    cv += __shfl_down_sync(0xFFFFFFFFu, cv, o);
    cnt += __shfl_down_sync(0xFFFFFFFFu, cnt, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(out, cv);
    atomicAdd(out + 1, cnt);
  }
}

// ---------------------------------------------------------------------------------------
// The neuron record for the host: neurons [i0, i0 + cnt) field by field (v, u, I, a, b, c, d,
// spike count, those of `fields` by bit, `cnt` values each, in that order), written straight
// to page-locked host memory.  Bound by the link to the host: 32 bytes a neuron instead of
// the 60 of the device's records, and nothing to take apart there (N=10^6: 8.6 ms for four
// copies into pageable buffers and a pass over them).
// ---------------------------------------------------------------------------------------
__global__ void k_state_pack(NetView v, int64_t i0, int cnt, unsigned fields, float *out) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < cnt; k += gridDim.x * blockDim.x) {
    const int64_t i = i0 + k;
    float *o = out + k;
    auto put = [&](unsigned bit, float x) {
      if (fields & bit) {
        *o = x;
        o += cnt;
      }
    };
    if (fields & 3u) {
      const float2 s = v.vu[i];
      put(1u, s.x);
      put(2u, s.y);
    }
    if (fields & 4u) put(4u, v.ilast[i]);
    if (fields & 0x78u) {
      const float4 p = v.abcd[i];
      put(8u, p.x);
      put(16u, p.y);
      put(32u, p.z);
      put(64u, p.w);
    }
    if (fields & 128u) put(128u, __int_as_float(v.sstat[i].nospks));
  }
}

// ---------------------------------------------------------------------------------------
// Launchers.
// ---------------------------------------------------------------------------------------
static int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 1;
  }
  return n;
}

static unsigned grid_for(int64_t work, int nt, int cap_per_sm) {
  int64_t g = (work + nt - 1) / nt;
  const int64_t cap = (int64_t)sm_count() * cap_per_sm;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (unsigned)g;
}

cudaError_t launch_init(const NetView &v, cudaStream_t s) {
  k_init_state<<<grid_for(v.n, 256, 32), 256, 0, s>>>(v);
  return cudaGetLastError();
}

cudaError_t launch_conngen(const NetView &v, int self_loops, cudaStream_t s) {
  int log2h = 5;
  while ((1 << log2h) < 2 * v.nsyn + 64) ++log2h;
  // the target bitmap (n bits, in 16-byte units) where it is smaller than the hash
  const int64_t bm_words = ((v.n + 127) / 128) * 4;
  const int bits = bm_words < ((int64_t)1 << log2h) ? (int)bm_words : 0;
  const size_t per_warp = bits > 0 ? (size_t)4 * bits : (size_t)4 << log2h;
  if (per_warp > 200 * 1024) return cudaErrorInvalidValue;
  // one ceiling for every network (concurrent host threads generating tables of different
  // fan-outs must not lower it under one another's launch)
  cudaError_t e = cudaFuncSetAttribute(k_conngen, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e != cudaSuccess) return e;
  // warps per CTA (at most 8): the most resident warps per SM
  int wpb = 1, best = 0, occ_best = 1;
  for (int w = 1; w <= 8 && per_warp * w <= 200 * 1024; ++w) {
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_conngen, w * 32, per_warp * w);
    if (occ * w > best) best = occ * w, wpb = w, occ_best = occ < 1 ? 1 : occ;
  }
  const size_t smem = per_warp * wpb;
  const uint64_t range = self_loops ? (uint64_t)v.n : (uint64_t)(v.n - 1);
  // generous cap on draw blocks (a full row needs about range * ln(range) draws)
  unsigned long long max_blocks = (64ull * (range + (uint64_t)v.nsyn) + 4096ull) / 128ull + 64ull;
  int64_t g = (v.n + wpb - 1) / wpb;
  const int64_t cap = (int64_t)sm_count() * occ_best * 8;
  if (g > cap) g = cap;
  k_conngen<<<(unsigned)g, wpb * 32, smem, s>>>(v, self_loops, log2h, bits, 0, v.n, max_blocks);
  return cudaGetLastError();
}

// CTA size of the persistent kernel by the neurons: 256 threads and one block per SM where
// that covers them (N=2,500 S 5.1 us a step against 5.9), else 512 (N=100,000 13.1 against
// 19.4), two blocks per SM if one does not cover them.
constexpr int kPerSmall = 256, kPerLarge = 512;

template <int NT>
static int persistent_occupancy() {
  int occ = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_persistent<NT>, NT, 0);
  return occ < 1 ? 1 : occ;
}

int persistent_blocks() { return persistent_occupancy<kPerLarge>() * sm_count(); }

// Threads per spiking row of a scheme: N a warp for each spiking neuron (one thread, the
// reference's choice, walks a row as a chain of loads: 88 us a step for N=2,500 x 1000 against
// 6.5), AP a group of 64, S and AB flat over all synapses of the step, as the SKL fallback.
static int deliver_group(int alg) { return alg == kAlgN ? 32 : alg == kAlgAP ? 64 : 0; }

template <int NT>
static cudaError_t persistent_nt(const NetView &v, int64_t t_abs0, int nsteps, bool last_chunk, GridSync *gs,
                                 unsigned long long limit_ns, int group, int stall, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  const int sms = sm_count();
  cfg.gridDim = dim3((unsigned)(v.n <= (int64_t)sms * NT ? sms : sms * persistent_occupancy<NT>()));
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_persistent<NT>, v, t_abs0, nsteps, last_chunk ? 1 : 0, gs, limit_ns, group, stall);
}

cudaError_t launch_steps(const NetView &v, int64_t t_abs0, int nsteps, bool last_chunk, GridSync *gs,
                         unsigned long long limit_ns, int alg, double synapses, int stall, cudaStream_t s, int *launches) {
  const int group = deliver_group(alg);
  *launches = 1;
  // S where steps are expected to have many synapses: two launches a step, the delivery's grid
  // oversubscribed, which costs 10 to 20 us a step and then delivers 7 to 12% faster (us a step
  // persistent / two, with the synapses: N=100,000 x 1000 15.2 / 24.2 at 1.7 million, 250,000 x 10,000
  // 33.0 / 42.9 at 4.3, 100,000 x 10,000 100 / 97 at 15.8, 300,000 x 1000 127 / 131 at 21, 100,000 x
  // 10,000 179 / 166 at 29, 10^6 x 3000 288 / 265 at 48, 250,000 x 10,000 435 / 388 at 73)
  constexpr double kTwoLaunches = 16e6;
  if (!(alg == kAlgS && synapses >= kTwoLaunches))
    return v.n <= (int64_t)sm_count() * kPerSmall
               ? persistent_nt<kPerSmall>(v, t_abs0, nsteps, last_chunk, gs, limit_ns, group, stall, s)
               : persistent_nt<kPerLarge>(v, t_abs0, nsteps, last_chunk, gs, limit_ns, group, stall, s);
  *launches = 2 * nsteps;
  // (a thread per vector for up to 5% of the neurons firing)
  const unsigned grid = grid_for(v.n / 20 * (v.stride >> 2), 256, 64);
  for (int lt = 0; lt < nsteps; ++lt) {
    k_update<256><<<grid_for(v.n, 256, 8), 256, 0, s>>>(v, t_abs0, lt, last_chunk && lt == nsteps - 1);
    k_deliver<<<grid, 256, 0, s>>>(v, lt);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_state_pack(const NetView &v, int64_t i0, int cnt, unsigned fields, float *out, cudaStream_t s) {
  k_state_pack<<<grid_for(cnt, 256, 4), 256, 0, s>>>(v, i0, cnt, fields, out);
  return cudaGetLastError();
}

cudaError_t launch_stats(const NetView &v, double *out, cudaStream_t s) {
  k_stats<<<grid_for(v.n, 256, 8), 256, 0, s>>>(v, out);
  return cudaGetLastError();
}

}  // namespace g4s
