// g4s_team.cu — the SKL step loop as an owner-computes team kernel (the GB300 design of
// SKL_deliverspks, gpu4snn.cu:669-716), for one network or many, plus the table
// preparation it needs.
//
// Teams.  A launch runs a list of networks (TeamItem); network i is simulated by a team
// of T_i CTAs.  The CTAs of the cooperative, persistent grid take (network, rank) slots
// from one ordered queue; multi-CTA teams come first in the queue, so a team's members
// start together.  A single network on the whole GPU is a one-item launch with a team of
// one CTA per SM; a batched ensemble is a many-item launch where most networks fit one
// CTA.
//
// Target ownership.  Team rank r owns the neurons [r Rc, (r+1) Rc) of its network and
// keeps their synaptic currents in shared memory for the whole launch, as two 32-bit
// words per neuron: the Q32.32 current q = A * 2^16 + B, with B the sum of the weights'
// low 16 bits and A the sum of their high 48 bits.  Shared-memory 32-bit atomics are
// about five times faster than 64-bit ones on this part, and the split is exact as long
// as no neuron has 65536 or more incoming synapses and the sum of |q_i| / 2^16 + 1 over
// its incoming synapses stays below 2^31; k_inbound checks both once per table (the
// host falls back to the global-atomic persistent kernel otherwise).  Small slices also
// keep v, u (and a, b, c, d) in shared memory for the launch.
//
// Per step, for each team:
//   update    every rank updates its own neurons (current read from and cleared in shared
//             memory; drive precomputed in shared memory during the previous step) and
//             collects its spikes in shared memory;
//   exchange  one-CTA team: nothing, the spike list stays in shared memory.  Larger team:
//             each rank publishes its spike count and ids as 64-bit words, each tagged
//             with a step number that never repeats for the network's buffers, so a
//             reader that sees the tag it expects needs no fence to trust the payload:
//             two 128-byte record lines (count and 31 ids), further ids in a per-rank
//             overflow list.  In teams of kOwnSources CTAs and more (kOwnSourcesLarge where
//             steps are large) every warp polls the
//             records of a few source ranks of its own (line 0, and line 1 of the ranks that
//             had more than kLine1After spikes in the previous step, with a time limit) and
//             goes on to deliver those ranks' spikes at once: no warp waits for another
//             one's sources, and the step has two block barriers (after the update, at its
//             end).  In smaller teams every warp reads every rank's count and takes its share
//             of the step's spikes.  Records are cleared before each launch.  Two record sets
//             (by step parity) suffice: a rank writes step t+2's words only after every rank
//             has published step t+1, i.e. finished reading step t.
//   delivery  one-CTA team: whole spiking rows.  Larger team: every rank reads, for every
//             spike, the segment of the spiking row whose targets fall in its slice (rows
//             are sorted by target and a per-row offset table gives the segment).  The rows
//             are read as packed words, the weight already in fixed point beside its target,
//             so that a segment of ~7 synapses is one contiguous run of sectors and needs no
//             float conversion.  Run mapping: a warp walks the concatenated segments of 32
//             spikes.  Group mapping (the team's choice for long segments): eight lanes walk
//             one spike's segment each.  Each weight goes into the rank's own shared memory.
//   tail      the raster and the spike statistics of this rank's spikes, and the next
//             step's drive, handed out in chunks of 32 neurons to warps as they finish
//             delivering.
//   What bounds a step: with few spikes the chain update -> publish -> poll -> bounds ->
//   rows, of whose 6,500 cycles (N=2,500) the four trips to L2 are half, the other half the
//   straight code between them, which all warps issue; with many, the LSU's shared-memory
//   pipe, by the additions and the row reads (ncu: busy 66% of N=10^6 x 1000, 75% at drive 2, 77%
//   and 82% of N=250,000 x 10,000; issue 56, 53, 43 and 42%).  us per step of this kernel and of the one before it (block-wide scan and
//   staging of the step's ids, a search per synapse, a conversion per synapse; all mappings in
//   one kernel): N=2,500 x 1000 3.30 / 4.55, 33,333 x 777 at drive 1.5 5.19 / 7.10, 100,000 x
//   1000 7.28 / 8.77, 10^6 x 1000 40.1 / 43.4 (drive 0.5 13.0 / 17.6, drive 2 106 / 112),
//   250,000 x 10,000 39.6 / 54.7; 64 networks in one launch 29.8 / 60.7 ms.
//   The raster records the spike ids of every step while its buffer has room.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <map>
#include <mutex>

#include "g4s_device.cuh"
#include "g4s_internal.h"

namespace g4s {

// ---------------------------------------------------------------------------------------
// Row sort: every row's (target, weight) pairs in ascending target order, unused slots
// (negative targets, i.e. huge as unsigned) last.  One CTA of NT threads per row, a bitonic
// network over p2 = E * NT 64-bit keys (target << 32 | weight bits); thread t holds the
// keys of elements t, t + NT, ..., in registers.  A compare-exchange over distance j takes
// place in registers when j >= NT (the partner is the same thread's), through shuffles
// when j < 32 (the partner is in the same warp), and through shared memory between warps
// otherwise, so that only those stages need block barriers.
// ---------------------------------------------------------------------------------------
template <int E>
__global__ void __launch_bounds__(1024) k_sort_rows(NetView v, int p2) {
  extern __shared__ unsigned long long s_key[];
  const int NT = blockDim.x, t = threadIdx.x;
  for (int64_t row = blockIdx.x; row < v.n; row += gridDim.x) {
    int *ri = const_cast<int *>(v.idx) + row * v.stride;
    float *rw = const_cast<float *>(v.w) + row * v.stride;
    unsigned long long key[E];
#pragma unroll
    for (int r = 0; r < E; ++r) {
      const int e = r * NT + t;
      key[r] = e < v.stride ? ((unsigned long long)(unsigned)ri[e] << 32) | __float_as_uint(rw[e])
                            : 0xFFFFFFFFFFFFFFFFull;
    }
    for (int k = 2; k <= p2; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        if (j >= NT) {
          const int rj = j / NT;
#pragma unroll
          for (int RJ = 1; RJ < E; RJ <<= 1)  // (each distance unrolled: registers, not memory)
            if (rj == RJ) {
#pragma unroll
              for (int r = 0; r < E; ++r)
                if ((r & RJ) == 0) {
                  const bool asc = ((r * NT + t) & k) == 0;
                  const unsigned long long a = key[r], b = key[r | RJ];
                  if ((a > b) == asc) {
                    key[r] = b;
                    key[r | RJ] = a;
                  }
                }
            }
        } else {
          if (j >= 32) {
            __syncthreads();  // (the previous stage's reads are done)
#pragma unroll
            for (int r = 0; r < E; ++r) s_key[r * NT + t] = key[r];
            __syncthreads();
          }
#pragma unroll
          for (int r = 0; r < E; ++r) {
            const int e = r * NT + t;
            const unsigned long long o = j >= 32 ? s_key[e ^ j] : __shfl_xor_sync(0xFFFFFFFFu, key[r], j);
            const bool keep_min = ((e & j) == 0) == ((e & k) == 0);
            key[r] = keep_min ? (o < key[r] ? o : key[r]) : (o > key[r] ? o : key[r]);
          }
        }
      }
#pragma unroll
    for (int r = 0; r < E; ++r) {
      const int e = r * NT + t;
      if (e < v.stride) {
        ri[e] = (int)(key[r] >> 32);
        rw[e] = __uint_as_float((unsigned)key[r]);
      }
    }
  }
}

// Generated rows (distinct targets, every unused slot (-1, 0.0f)) in the same order as
// k_sort_rows' by a bucket sort of narrower keys: 32-bit key target << pb | slot (n << pb
// | slot for an unused slot), 2^pb >= p2 and (n << pb) + p2 - 1 below 2^32 - 1, unique, so
// that every key names the slot its weight comes from.  Bucket of a key: its target >> sh
// (targets taken as n for unused slots; n >> sh < nb), monotone in the key, about two to
// four keys each as the targets are drawn uniformly.  Per row: the weights into shared
// memory; a histogram whose atomics also give each key its rank in its bucket; a block
// scan of the counts; each key stored at its bucket's start + its rank; one thread per
// bucket orders the bucket's keys by insertion; the row written back (target from the
// key, weight gathered from the shared copy).  E keys a thread, element r * NT + t.
template <int E>
__global__ void __launch_bounds__(1024) k_sort_gen(NetView v, int pb, int nb, int sh) {
  extern __shared__ __align__(16) unsigned s_gen[];
  const int NT = blockDim.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  unsigned *s_cnt = s_gen;                                  // nb counts, then bucket starts
  unsigned *s_part = s_cnt + nb;                            // 32 warp sums
  unsigned *s_key = s_part + 32;                            // stride keys, by bucket
  float *s_w = reinterpret_cast<float *>(s_key + v.stride);  // the row's weights
  const unsigned n = (unsigned)v.n, smask = (1u << pb) - 1u, lim = n << pb;
  const int per = nb / NT;  // buckets a thread scans (nb is a multiple of NT)
  for (int64_t row = blockIdx.x; row < v.n; row += gridDim.x) {
    int *ri = const_cast<int *>(v.idx) + row * v.stride;
    float *rw = const_cast<float *>(v.w) + row * v.stride;
    for (int b = t; b < nb; b += NT) s_cnt[b] = 0u;
    unsigned key[E];
#pragma unroll
    for (int r = 0; r < E; ++r) {
      const int e = r * NT + t;
      if (e < v.stride) {
        const unsigned ti = (unsigned)ri[e];
        key[r] = ((ti < n ? ti : n) << pb) | (unsigned)e;
        s_w[e] = rw[e];
      }
    }
    __syncthreads();
    unsigned rank[E];
#pragma unroll
    for (int r = 0; r < E; ++r)
      if (r * NT + t < v.stride) rank[r] = atomicAdd(s_cnt + ((key[r] >> pb) >> sh), 1u);
    __syncthreads();
    // exclusive scan of the counts: thread t's buckets t*per .. t*per+per-1, then warps
    unsigned mine = 0;
    for (int q = 0; q < per; ++q) mine += s_cnt[t * per + q];
    unsigned incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= d) incl += o;
    }
    if (lane == 31) s_part[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const int nw = NT >> 5;
      unsigned x = lane < nw ? s_part[lane] : 0u, xi = x;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned o = __shfl_up_sync(0xFFFFFFFFu, xi, d);
        if (lane >= d) xi += o;
      }
      if (lane < nw) s_part[lane] = xi - x;
    }
    __syncthreads();
    unsigned start = s_part[warp] + incl - mine;
    for (int q = 0; q < per; ++q) {
      const unsigned c = s_cnt[t * per + q];
      s_cnt[t * per + q] = start;
      start += c;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < E; ++r)
      if (r * NT + t < v.stride) s_key[s_cnt[(key[r] >> pb) >> sh] + rank[r]] = key[r];
    __syncthreads();
    for (int b = t; b < nb; b += NT) {
      const unsigned lo = s_cnt[b], hi = b + 1 < nb ? s_cnt[b + 1] : (unsigned)v.stride;
      for (unsigned i = lo + 1; i < hi; ++i) {
        const unsigned x = s_key[i];
        unsigned j = i;
        while (j > lo && s_key[j - 1] > x) {
          s_key[j] = s_key[j - 1];
          --j;
        }
        s_key[j] = x;
      }
    }
    __syncthreads();
    for (int e = t; e < v.stride; e += NT) {
      const unsigned k = s_key[e];
      ri[e] = k < lim ? (int)(k >> pb) : -1;
      rw[e] = s_w[k & smask];
    }
    __syncthreads();  // (before the next row overwrites the shared arrays)
  }
}

// Rows already in the sort's order (ascending 64-bit keys target << 32 | weight bits, the
// targets taken as unsigned so that unused slots come last)?  *unsorted = 1 if not.
// One warp per row, consecutive lanes on consecutive slots.
__global__ void k_rows_sorted(NetView v, int *unsorted) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  bool bad = false;
  for (int64_t row = warp; row < v.n; row += nwarps) {
    const int *ri = v.idx + row * v.stride;
    const float *rw = v.w + row * v.stride;
    for (int j = lane; j + 1 < v.stride; j += 32) {
      const unsigned long long a = ((unsigned long long)(unsigned)ri[j] << 32) | __float_as_uint(rw[j]);
      const unsigned long long b = ((unsigned long long)(unsigned)ri[j + 1] << 32) | __float_as_uint(rw[j + 1]);
      bad |= a > b;
    }
  }
  if (__any_sync(0xFFFFFFFFu, bad) && lane == 0) *unsorted = 1;
}

// First slot of `idx` (a table of v's shape) that targets neuron n or a later one, into
// *first (~0 at launch: none); four slots a thread, bound by memory.
__global__ void k_first_bad(const int4 *idx, NetView v, unsigned long long *first) {
  const int64_t quads = v.n * (int64_t)(v.stride >> 2);
  unsigned long long mine = ~0ull;
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < quads; g += (int64_t)gridDim.x * blockDim.x) {
    const int4 t = __ldcs(idx + g);
    const int bad = t.x >= v.n ? 0 : t.y >= v.n ? 1 : t.z >= v.n ? 2 : t.w >= v.n ? 3 : 4;
    if (bad < 4 && mine == ~0ull) mine = 4ull * (unsigned long long)g + (unsigned long long)bad;
  }
  if (mine != ~0ull) atomicMin(first, mine);
}

// Segment table: seg[row][k] = first slot of the sorted row whose target is >= k*Rc, for
// k = 0..T (unused slots compare as huge and lie beyond seg[row][T]).  One warp per row,
// one binary search per boundary.
__global__ void k_segoff(NetView v, int T, int64_t Rc, uint16_t *seg) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row = warp; row < v.n; row += nwarps) {
    const int *ri = v.idx + row * v.stride;
    for (int k = lane; k <= T; k += 32) {
      const int64_t bound = (int64_t)k * Rc;
      int lo = 0, hi = v.stride;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((int64_t)(unsigned)ri[mid] < bound)
          lo = mid + 1;
        else
          hi = mid;
      }
      seg[row * (T + 1) + k] = (uint16_t)lo;
    }
  }
}

// Packed rows for the team kernel: pair[g] = Q32.32 weight of slot g << pair_bits | its
// target; an unused slot is weight 0 into neuron 0, which adds nothing.  The conversion of
// every weight to fixed point happens here, once per table change, instead of at every
// delivery: F2I.S64 runs on the FP64 pipe, about 16 cycles a warp instruction per SM on this
// part (N=250,000 x 10,000: 4,200 of them a step and SM, 33 of the step's 55 us).
// Four slots a thread (rows are multiples of four slots): bound by memory, 16 bytes a slot.
__global__ void k_pairs(NetView v, ulonglong2 *pair) {
  const int64_t quads = v.n * (int64_t)(v.stride >> 2);
  const int4 *idx = reinterpret_cast<const int4 *>(v.idx);
  const float4 *w = reinterpret_cast<const float4 *>(v.w);
  const int bits = v.pair_bits;
  auto word = [&](int t, float x) {
    return t < 0 ? 0ull : ((unsigned long long)wfix(x) << bits) | (unsigned long long)(unsigned)t;
  };
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < quads; g += (int64_t)gridDim.x * blockDim.x) {
    const int4 t = __ldcs(idx + g);
    const float4 x = __ldcs(w + g);
    pair[2 * g] = make_ulonglong2(word(t.x, x.x), word(t.y, x.y));
    pair[2 * g + 1] = make_ulonglong2(word(t.z, x.z), word(t.w, x.w));
  }
}

// Exactness bound of the split accumulation: per target, the number of incoming synapses
// and the sum of (|q| >> 16) + 1 over them; out[0] = max count, out[1] = max sum.
// Per neuron the in-degree and, with mag, sum(|q| >> 16) + 1 over its inputs; without mag,
// the largest (|q| >> 16) + 1 of the table into *term instead.
__global__ void k_inbound(NetView v, unsigned *cnt, unsigned long long *mag, unsigned long long *term) {
  const int64_t total = v.n * (int64_t)v.stride;
  unsigned long long mx = 0;
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < total; g += (int64_t)gridDim.x * blockDim.x) {
    const int t = v.idx[g];
    if (t < 0) continue;
    atomicAdd(cnt + t, 1u);
    const long long q = wfix(v.w[g]);
    const unsigned long long a = ((unsigned long long)(q < 0 ? -q : q) >> 16) + 1ull;
    if (mag)
      atomicAdd(mag + t, a);
    else
      mx = max(mx, a);
  }
  if (!mag) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, d));
    if ((threadIdx.x & 31) == 0) atomicMax(term, mx);
  }
}

// The same counts and largest term with the counters in shared memory: CTA b counts the
// targets of part b % parts (kInboundPart neurons) over the rows of its group, so that the
// targets are read once per part and every synapse is one shared addition; the CTA's counts
// then go to cnt, and the weights are shared out between the parts.  Bound by its reads and
// the shared additions: N=100,000 x 1000 (two parts) 250 us, where k_inbound takes 626, its
// 10^8 global additions 6.3 ps each.
constexpr int kInboundPart = 51200;
__global__ void __launch_bounds__(1024, 1) k_inbound_shared(NetView v, int parts, unsigned *cnt,
                                                            unsigned long long *term) {
  extern __shared__ unsigned s_in[];
  const int part = (int)(blockIdx.x % (unsigned)parts), groups = (int)(gridDim.x / (unsigned)parts);
  const int group = (int)(blockIdx.x / (unsigned)parts);
  const int lo = part * kInboundPart;  // (parts * kInboundPart < 2^31)
  const unsigned len = (unsigned)min((int64_t)kInboundPart, v.n - lo);
  for (unsigned k = threadIdx.x; k < len; k += blockDim.x) s_in[k] = 0u;
  __syncthreads();
  const int64_t quads = v.n * (int64_t)(v.stride >> 2);  // (rows are multiples of four slots)
  const int4 *idx = reinterpret_cast<const int4 *>(v.idx);
  const float4 *w = reinterpret_cast<const float4 *>(v.w);
  unsigned long long mx = 0;
  auto count = [&](int t) {
    const unsigned k = (unsigned)t - (unsigned)lo;  // (an unused slot's target is negative: beyond len)
    if (k < len) atomicAdd(s_in + k, 1u);
  };
  auto size = [&](int t, float x) {
    const long long q = wfix(x);
    if (t >= 0) mx = max(mx, ((unsigned long long)(q < 0 ? -q : q) >> 16) + 1ull);
  };
  if (group < groups) {
    int64_t g = group * (int64_t)blockDim.x + threadIdx.x;
    const int64_t hop = (int64_t)groups * blockDim.x;
    for (int turn = 0; g < quads; g += hop) {
      const int4 t = idx[g];
      if (turn == part) {
        const float4 x = __ldcs(w + g);
        size(t.x, x.x);
        size(t.y, x.y);
        size(t.z, x.z);
        size(t.w, x.w);
      }
      count(t.x);
      count(t.y);
      count(t.z);
      count(t.w);
      if (++turn == parts) turn = 0;
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, d));
  if ((threadIdx.x & 31) == 0 && mx) atomicMax(term, mx);
  __syncthreads();
  for (unsigned k = threadIdx.x; k < len; k += blockDim.x)
    if (s_in[k]) atomicAdd(cnt + lo + k, s_in[k]);
}

// The largest count and sum (one atomic per block: one per thread took 200 us by itself,
// at any size).
__global__ void k_inbound_max(int64_t n, const unsigned *cnt, const unsigned long long *mag,
                              unsigned long long *out) {
  __shared__ unsigned long long s_mc, s_mm;
  if (threadIdx.x == 0) s_mc = s_mm = 0ull;
  __syncthreads();
  unsigned long long mc = 0, mm = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    mc = max(mc, (unsigned long long)cnt[i]);
    if (mag) mm = max(mm, mag[i]);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    mc = max(mc, __shfl_xor_sync(0xFFFFFFFFu, mc, d));
    mm = max(mm, __shfl_xor_sync(0xFFFFFFFFu, mm, d));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&s_mc, mc);
    atomicMax(&s_mm, mm);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_mc) atomicMax(out, s_mc);
    if (s_mm) atomicMax(out + 1, s_mm);
  }
}

// Split-accumulator add: A += q >> 16 (arithmetic), B += q & 0xFFFF.
__device__ __forceinline__ void acc_add(unsigned base_a, unsigned base_b, unsigned off, long long q) {
  asm volatile("red.shared.add.s32 [%0], %1;" ::"r"(base_a + off * 4u), "r"((int)(q >> 16)) : "memory");
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(base_b + off * 4u), "r"((unsigned)(q & 0xFFFF)) : "memory");
}

__device__ __forceinline__ void acc_add4(unsigned base_a, unsigned base_b, int lo, const int4 t, const float4 w) {
  if (t.x >= 0) acc_add(base_a, base_b, (unsigned)(t.x - lo), wfix(w.x));
  if (t.y >= 0) acc_add(base_a, base_b, (unsigned)(t.y - lo), wfix(w.y));
  if (t.z >= 0) acc_add(base_a, base_b, (unsigned)(t.z - lo), wfix(w.z));
  if (t.w >= 0) acc_add(base_a, base_b, (unsigned)(t.w - lo), wfix(w.w));
}

// A synapse as the delivery loads it: a packed word (kPair), or target and weight bits.
struct Syn {
  unsigned x, y;
};

// The synapse `at` slots after a place of the tables, where `rem` > `at`; `row` is the
// place: an address in the packed rows (kPair), or a slot of the separate arrays.
template <bool kPair>
__device__ __forceinline__ Syn load_syn(const NetView &v, long long row, int rem, int at) {
  Syn s;
  if constexpr (kPair) {
    asm("{.reg .pred p;\n\tsetp.gt.s32 p, %3, %4;\n\t@p ld.global.nc.v2.u32 {%0, %1}, [%2];}"
        : "=r"(s.x), "=r"(s.y)
        : "l"(row + at * 8), "r"(rem), "r"(at));
  } else {
    asm("{.reg .pred p;\n\tsetp.gt.s32 p, %4, %5;\n\t@p ld.global.nc.u32 %0, [%2];\n\t@p ld.global.nc.u32 %1, [%3];}"
        : "=r"(s.x), "=r"(s.y)
        : "l"(v.idx + row + at), "l"(v.w + row + at), "r"(rem), "r"(at));
  }
  return s;
}
template <bool kPair>
__device__ __forceinline__ long long syn_row(const NetView &v, long long slot) {
  return kPair ? (long long)reinterpret_cast<uintptr_t>(v.pair + slot) : slot;
}
template <bool kPair>
__device__ __forceinline__ long long syn_after(long long row, int slots) {
  return row + (kPair ? slots * 8 : slots);
}

// Adds a synapse to the split accumulators, where `rem` > `at` (red.shared of random words:
// 3.9 cycles a warp instruction per SM, 1.2 without bank conflicts); base_a and base_b are the
// shared addresses that neuron 0's words would have.  The packed word's high part shifted
// right is q >> 16.
template <bool kPair, bool kSink>
__device__ __forceinline__ void acc_syn(unsigned base_a, unsigned base_b, int bits, unsigned tmask, const Syn s,
                                        int rem, int at) {
  int a;
  unsigned b, t;
  if constexpr (kPair) {
    t = s.x & tmask;
    a = (int)s.y >> (bits - 16);
    b = __funnelshift_r(s.x, s.y, bits) & 0xFFFFu;
  } else {
    const long long q = wfix(__uint_as_float(s.y));
    t = s.x;
    a = (int)(q >> 16);
    b = (unsigned)(q & 0xFFFF);
  }
  const bool on = rem > at;
  if constexpr (kSink) {
    // lanes past the end add to a word of their own that is never read (whole rows: few such
    // lanes, and no divergence region per synapse, 70.4 against 79.0 us a step for a lone CTA)
    __shared__ int s_sink[32];
    const unsigned sink = (unsigned)__cvta_generic_to_shared(&s_sink[threadIdx.x & 31]);
    asm volatile("red.shared.add.s32 [%0], %1;" ::"r"(on ? base_a + t * 4u : sink), "r"(a));
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(on ? base_b + t * 4u : sink), "r"(b));
  } else if (on) {
    asm volatile("red.shared.add.s32 [%0], %1;" ::"r"(base_a + t * 4u), "r"(a));
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(base_b + t * 4u), "r"(b));
  }
}

// Scratch of one warp: the delivery's segment runs, then the drive's repeated draws.
struct WarpScratch {
  union {
    struct {
      long long row[32];  // place of every segment of a batch, less its position in the run
      unsigned head[8];   // segment heads of 256 synapses
    };
    int retry[64];  // neurons whose first draw was rejected
  };
};

__device__ __forceinline__ unsigned lanemask_le() { return 0xFFFFFFFFu >> (31u - (threadIdx.x & 31u)); }

// Scalars of one CTA shared by the phases of a step; the per-step counters come in pairs
// (by step parity) so that one is cleared while the other is in use.
struct TeamShared {
  int nown[2];    // spikes of this rank in the step
  int work[2];    // next chunk of the next step's drive (a warp adds at most two past the last one)
  int off[2];     // spikes of the ranks before this one in the step
  unsigned k[2];  // spikes of the team, plus kPolled for every warp that has added its source
                  // ranks' to off and to this
  long long base; // raster offset of the step
  int fail;       // the exchange gave up (time limit, or the team's error word was set)
  int slot;       // queue slot taken by this CTA
  int rank;       // rank and layout of the network's slice, read where they are needed (kept
  TeamLayout L;   // in registers they would spill the delivery's reads in flight)
  unsigned long long lim;  // time limit of the step's waits
};

// (a team holds fewer than 2^26 neurons: kMaxTeam slices within the shared memory)
constexpr unsigned kPolled = 1u << 26;

// Record words of a rank per step: word 0 = spike count, words 1.. = ids (kInline inline).
constexpr int kRankWords = kRecLines * kRecWords;
constexpr int kInline = kRankWords - 1;
constexpr int kLine1After = 7;  // line 1 of a rank is polled if it had more spikes in the previous step

// Gives up a wait: first error wins, every CTA of the team leaves at its next check.
__device__ __forceinline__ void give_up(const TeamItem &it, TeamShared &sh) {
  if (atomicCAS(&it.sync->error, 0, kErrTimeoutCode) == 0) *(volatile int *)it.v.status = kErrTimeoutCode;
  *(volatile int *)&sh.fail = 1;
}

// One tagged word of another rank, polled until it carries `tag` (or the time limit).
__device__ __forceinline__ int tagged_id(const unsigned long long *p, unsigned tag, const TeamItem &it, TeamShared &sh,
                                         unsigned long long lim) {
  unsigned long long w = ld_relaxed_u64(p);
  if ((unsigned)(w >> 32) == tag) return (int)(unsigned)w;
  const unsigned long long t0 = globaltimer();
  for (;;) {
    w = ld_relaxed_u64(p);
    if ((unsigned)(w >> 32) == tag) return (int)(unsigned)w;
    if (*(volatile int *)&sh.fail || ld_relaxed(&it.sync->error) != 0 || globaltimer() - t0 > lim) {
      give_up(it, sh);
      return 0;
    }
  }
}

// The checks of a poll by a warp whose words are not all there yet, every kPollCheck rounds
// (a round is one trip to L2; t0: the time of the first check, 0 before it): true when the
// wait is given up.
constexpr unsigned kPollCheck = 16;
__device__ __forceinline__ bool poll_check(const TeamItem &it, TeamShared &sh, unsigned iter, unsigned long long &t0,
                                           unsigned long long lim) {
  if (iter % kPollCheck != kPollCheck - 1) return false;
  int f = 0;
  if ((threadIdx.x & 31) == 0) {
    const unsigned long long now = globaltimer();
    if (t0 == 0) t0 = now;
    f = *(volatile int *)&sh.fail;
    if (!f && threadIdx.x == 0 && ld_relaxed(&it.sync->error) != 0) f = 1;
    if (!f && now - t0 > lim) {
      give_up(it, sh);
      f = 1;
    }
    if (f) *(volatile int *)&sh.fail = 1;
  }
  return __shfl_sync(0xFFFFFFFFu, f, 0) != 0;
}

// Warps that poll source ranks and deliver their spikes; the others go straight to the next
// step's drive, beside the first ones' waits.  Of the 768-thread CTA's 24 warps, 22 with
// segment runs (us per step with 24, 23 and 22: N=33,333 x 777 5.37, 5.30, 5.19, N=100,000
// 7.46, 7.33, 7.28; 20 were slower again); all of them for long segments and for 1024 threads, whose steps deliver
// most of the time (N=10^6 at drive 2: 107 with 32 warps, 116 with 28).
__host__ __device__ constexpr int source_warps(int nt, int mode) {
  return nt == kTeamNTSmall && mode == kDeliverRun ? 22 : nt / 32;
}

static_assert(kMaxTeam <= 8 * source_warps(kTeamNT, kDeliverRun) && kMaxTeam <= 8 * source_warps(kTeamNTSmall, kDeliverRun),
              "a warp polls two lines of at most eight source ranks, two slots of each line a lane");

// The spikes a warp delivers in a step: a concatenation of source ranks' id lists.  Lane k
// holds source k: its offset in the concatenation and how many of its ids are staged in
// shared memory.  The source's rank is k, or warp + k x warps where warps have sources of
// their own.
struct Source {
  int off;      // this lane's source: offset in the concatenation (large: no such source)
  int inl;      // ... ids staged
  int total;    // ids of the concatenation
  int q0, dq;   // the warp's batches of 32: positions q0, q0 + dq, ...
  int wi, wpb;  // ... and its share of each (share wi of wpb)
  int lt;       // step of the launch
};

static_assert(kOwnSources <= 17 && kOwnSourcesLarge <= 17, "fetch_spike searches sixteen sources");
// This lane's spike of the batch at position q0 (whole warps call it): its row and the
// bounds of this rank's segment in it; an empty segment past the end.
template <int NT, int kMode>
__device__ __forceinline__ void fetch_spike(const TeamItem &it, TeamShared &sh, const unsigned char *s_raw,
                                            const Source &c, int q0, uint64_t pkeep, int &s, int &b, int &e) {
  const int q = q0 + (threadIdx.x & 31);
  s = b = e = 0;
  if (q0 >= c.total) return;
  // the source holding position q: the last one that starts at or before it (at most sixteen
  // sources, or eight of the warp's own; its offset and count in one word, as the shuffles
  // share the shared-memory pipe that bounds large steps: N=10^6 41.1 -> 40.7 us)
  int k = 0;
#pragma unroll
  for (int step = 8; step; step >>= 1)
    if (__shfl_sync(0xFFFFFFFFu, c.off, k + step) <= q) k += step;
  const int oi = __shfl_sync(0xFFFFFFFFu, (int)((unsigned)c.off << 5) | c.inl, k), j = q - (oi >> 5), staged = oi & 31;
  if (q < c.total) {
    const bool col = NT == kTeamNTSmall && sh.L.col_sm;  // (read ahead of the id)
    const int r = sh.L.pay_sm ? (int)(threadIdx.x >> 5) + k * source_warps(NT, kMode) : k;
    if (j < staged) {
      s = reinterpret_cast<const int *>(s_raw + sh.L.pay)[r * kRankWords + 1 + j];
    } else {
      const int par = c.lt & 1;
      s = tagged_id(j < kInline ? it.rec + ((size_t)par * it.team + r) * kRankWords + 1 + j
                                : it.list + (size_t)par * it.v.n + (size_t)r * it.rc + j,
                    it.tag0 + (unsigned)c.lt + 1u, it, sh, sh.lim);
    }
    if (col) {
      const unsigned be = reinterpret_cast<const unsigned *>(s_raw + sh.L.col)[s];
      b = (int)(be & 0xFFFFu);
      e = (int)(be >> 16);
    } else {
      const uint16_t *so = it.seg + (size_t)s * (unsigned)(it.team + 1) + sh.rank;
      b = ld_keep_u16(so, pkeep);
      e = ld_keep_u16(so + 1, pkeep);
    }
  }
}

// Delivery of a one-CTA team: K whole spiking rows.
template <int NT, bool kPair>
__device__ __forceinline__ void deliver_solo(const TeamItem &it, const int *list, int K, unsigned base_a,
                                             unsigned base_b) {
  const NetView &v = it.v;
  if constexpr (kPair) {
    // warps take the rows in pieces of 128 packed words, two 16-byte vectors a lane in flight
    // (pieces of 256 words, four vectors, spill: 64 networks in one launch 52.6 ms against 45.5)
    constexpr int kWarps = NT / 32;
    const int lane = threadIdx.x & 31;
    const int rv = v.stride >> 1, np = (rv + 63) >> 6, total = K * np;
    const int dq = kWarps / np, dp = kWarps - dq * np;
    const int bits = v.pair_bits;
    const unsigned tmask = (1u << bits) - 1u;
    int task = threadIdx.x >> 5, q = task / np, pc = task - q * np;
    for (; task < total; task += kWarps) {
      const int rem = rv - pc * 64 - lane;
      const long long at = syn_row<true>(v, (long long)list[q] * v.stride) + (pc * 64 + lane) * 16;
      int4 p[2];
#pragma unroll
      for (int u = 0; u < 2; ++u)
        asm("{.reg .pred p;\n\tsetp.gt.s32 p, %5, %6;\n\t@p ld.global.nc.L1::no_allocate.v4.s32 {%0,%1,%2,%3}, [%4];}"
            : "=r"(p[u].x), "=r"(p[u].y), "=r"(p[u].z), "=r"(p[u].w)
            : "l"(at + u * 512), "r"(rem), "r"(u * 32));
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        acc_syn<true, true>(base_a, base_b, bits, tmask, Syn{(unsigned)p[u].x, (unsigned)p[u].y}, rem, u * 32);
        acc_syn<true, true>(base_a, base_b, bits, tmask, Syn{(unsigned)p[u].z, (unsigned)p[u].w}, rem, u * 32);
      }
      q += dq;
      pc += dp;
      if (pc >= np) {
        pc -= np;
        q += 1;
      }
    }
  } else {
    const uint64_t pol = policy_evict_first();
    const int rv = v.stride >> 2;
    const int total = K * rv;
    const int dq = NT / rv, dj = NT - dq * rv;
    int q = threadIdx.x / rv, j = threadIdx.x - q * rv;
    const int4 *ti = reinterpret_cast<const int4 *>(v.idx);
    const float4 *wi = reinterpret_cast<const float4 *>(v.w);
    for (int g = threadIdx.x; g < total; g += 2 * NT) {
      const size_t o0 = (size_t)list[q] * rv + j;
      int q1 = q + dq, j1 = j + dj;
      if (j1 >= rv) {
        j1 -= rv;
        q1 += 1;
      }
      const bool h1 = g + NT < total;
      const size_t o1 = h1 ? (size_t)list[q1] * rv + j1 : o0;
      const int4 t0 = ld_stream_i4(ti + o0, pol), t1 = ld_stream_i4(ti + o1, pol);
      const float4 w0 = ld_stream_f4(wi + o0, pol), w1 = ld_stream_f4(wi + o1, pol);
      acc_add4(base_a, base_b, 0, t0, w0);
      if (h1) acc_add4(base_a, base_b, 0, t1, w1);
      q = q1 + dq;
      j = j1 + dj;
      if (j >= rv) {
        j -= rv;
        q += 1;
      }
    }
  }
}

// Delivery of a larger team, eight lanes a spike (long segments): a batch of 32 spikes is
// walked in 8 rounds of 4, lane group g (lanes 8g .. 8g+7) reading spike 4r+g's segment in
// contiguous 64-synapse steps, eight reads a lane in flight; warps sharing a batch take its
// rounds in turn.  The next batch's ids and bounds are loaded while the current one is
// walked.  rel_a, rel_b: the shared addresses that neuron 0's accumulator words would have.
template <int NT, bool kPair>
__device__ __forceinline__ void deliver_group(const TeamItem &it, TeamShared &sh, const unsigned char *s_raw,
                                              const Source &c, unsigned rel_a, unsigned rel_b) {
  const NetView &v = it.v;
  const int lane = threadIdx.x & 31;
  const int bits = v.pair_bits;
  const unsigned tmask = (1u << (bits & 31)) - 1u;
  const uint64_t pkeep = policy_evict_last();
  const int sub = lane & 7, grp = lane >> 3;
  int s, b, e;
  fetch_spike<NT, kDeliverGroup>(it, sh, s_raw, c, c.q0, pkeep, s, b, e);
  for (int q0 = c.q0; q0 < c.total; q0 += c.dq) {
    const long long rowb = syn_row<kPair>(v, (long long)s * v.stride + b);  // segment start of this lane's spike
    const int len = e - b;
    fetch_spike<NT, kDeliverGroup>(it, sh, s_raw, c, q0 + c.dq, pkeep, s, b, e);  // next batch, in flight meanwhile
    for (int r = c.wi; r < 8; r += c.wpb) {
      long long at = syn_after<kPair>(__shfl_sync(0xFFFFFFFFu, rowb, r * 4 + grp), sub);
      for (int rem = __shfl_sync(0xFFFFFFFFu, len, r * 4 + grp) - sub; rem > 0; rem -= 64) {
        Syn x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = load_syn<kPair>(v, at, rem, u * 8);
#pragma unroll
        for (int u = 0; u < 8; ++u) acc_syn<kPair, false>(rel_a, rel_b, bits, tmask, x[u], rem, u * 8);
        at = syn_after<kPair>(at, 64);
      }
    }
  }
}

// Delivery of a larger team, segment runs: the segments of a batch of 32 spikes as one run,
// walked 256 synapses at a time with eight reads a lane in flight; warps sharing a batch
// take its 256-synapse pieces in turn.  A synapse finds its segment without a search: the
// heads of the batch's segments are set as bits in shared memory, and the segment's number
// is the count of heads up to the synapse (the binary search by shuffles that this replaces
// took about 25 of 93 instructions per 32 synapses; now 32 in all).
template <int NT, bool kPair>
__device__ __forceinline__ void deliver_run(const TeamItem &it, TeamShared &sh, const unsigned char *s_raw,
                                            const Source &c, unsigned rel_a, unsigned rel_b, WarpScratch &ws) {
  const NetView &v = it.v;
  const int lane = threadIdx.x & 31;
  const unsigned lane_le = lanemask_le();
  const int bits = v.pair_bits;
  const unsigned tmask = (1u << (bits & 31)) - 1u;
  const uint64_t pkeep = policy_evict_last();
  int s, b, e;
  fetch_spike<NT, kDeliverRun>(it, sh, s_raw, c, c.q0, pkeep, s, b, e);
  for (int q0 = c.q0; q0 < c.total; q0 += c.dq) {
    const int len = e - b;
    int excl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, excl, o);
      if (lane >= o) excl += y;
    }
    const int total = __shfl_sync(0xFFFFFFFFu, excl, 31);
    excl -= len;
    const bool has = len > 0;
    // the batch's segments that are not empty, in order: synapse f of the run that lies in
    // the k-th of them is f slots after row[k]
    const unsigned some = __ballot_sync(0xFFFFFFFFu, has);
    if (has) ws.row[__popc(some & (lane_le >> 1))] = syn_row<kPair>(v, (long long)s * v.stride + b - excl);
    fetch_spike<NT, kDeliverRun>(it, sh, s_raw, c, q0 + c.dq, pkeep, s, b, e);  // next batch, in flight meanwhile
    for (int f0 = c.wi * 256; f0 < total; f0 += c.wpb * 256) {
      const unsigned at = (unsigned)(excl - f0);
      int k = __popc(__ballot_sync(0xFFFFFFFFu, has && excl < f0)) - 1;
      if (lane < 8) ws.head[lane] = 0u;
      __syncwarp();
      if (has && at < 256u) atomicOr(&ws.head[at >> 5], 1u << (at & 31u));
      __syncwarp();
      const int rem = total - f0 - lane;
      Syn x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const unsigned h = ws.head[u];
        x[u] = load_syn<kPair>(v, syn_after<kPair>(ws.row[k + __popc(h & lane_le)], f0 + lane), rem, u * 32);
        k += __popc(h);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) acc_syn<kPair, false>(rel_a, rel_b, bits, tmask, x[u], rem, u * 32);
      __syncwarp();  // (the bits are read before they are cleared again)
    }
    __syncwarp();
  }
}

// The update of a rank's neurons (their arrays, at the slice's first neuron).
struct Update {
  float2 *vu;
  const float4 *abcd;
  const float *rpar;
  const float *z;  // the step's drive
  int *a;
  unsigned *b;
  float *ilast;  // input current, on the run's last step (else null)
  int *own;      // spikes: global ids ...
  int *nown;     // ... and their count
  int cnt, nexc; // neurons of the slice; the first nexc are excitatory
  int lo;        // first neuron
  float ge, gi;
};

// kUpd neurons a thread per round, the state loads of all of them first (a slice whose state
// lives in global memory takes one memory round trip per round), then each in turn; kFromR:
// a, b, c, d recomputed from the parameter r.  Two rather than four: the registers that
// leaves are worth more than the round trips (N=2,500 3.69 us a step against 3.84, N=10^6
// equal, 64 networks in one launch 52.9 ms against 58.3).
constexpr int kUpd = 2;
template <int NT, bool kFromR>
__device__ __forceinline__ void update_slice(const Update &w) {
  for (int i0 = threadIdx.x; i0 < w.cnt; i0 += kUpd * NT) {
    float2 sv[kUpd];
    float rr[kUpd];
#pragma unroll
    for (int u = 0; u < kUpd; ++u) {
      const int i = i0 + u * NT, j = i < w.cnt ? i : i0;
      sv[u] = w.vu[j];
      if (kFromR) rr[u] = w.rpar[j];
    }
    unsigned spk = 0;
#pragma unroll
    for (int u = 0; u < kUpd; ++u) {
      const int i = i0 + u * NT;
      if (i < w.cnt) {
        const float4 p = kFromR ? izh_abcd(rr[u], i < w.nexc) : w.abcd[i];
        const float isyn = split_current(w.a[i], w.b[i]);
        float I;
        const bool k = izh_step(sv[u].x, sv[u].y, I, p, i < w.nexc ? w.ge : w.gi, w.z[i], isyn);
        w.a[i] = 0;
        w.b[i] = 0;
        w.vu[i] = sv[u];
        if (w.ilast) w.ilast[i] = I;
        if (k) spk |= 1u << u;
      }
    }
    for (; spk; spk &= spk - 1) w.own[atomicAdd(w.nown, 1)] = w.lo + i0 + (__ffs(spk) - 1) * NT;
  }
}

// The drive of step `step` for the slice's neurons, in chunks of 32 handed to warps as they
// come.  Bound by instruction issue: the generator and the transform take 47 SM cycles per 32
// normals.  A neuron's first Philox call holds an accepted pair 95% of the time; in slices
// of more than kListDraws neurons the other draws are repeated in full warps (retried in
// place, four chunks out of five go through the generator again for one or two lanes: N=10^6
// at drive 0.5 14.5 us a step against 16.1).  Smaller slices, a chunk or two a warp, retry in
// place: a second pass by each warp costs them 0.1 us a step more.
constexpr int kListDraws = 1024;
__device__ __forceinline__ void drive_chunks(uint64_t seed, int lo, int cnt, int step, float *z, int *next,
                                             int *retry) {
  const int lane = threadIdx.x & 31;
  const unsigned below = lanemask_le() >> 1;
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  if (cnt <= kListDraws) {
    for (;;) {
      int c = 0;
      if (lane == 0) c = atomicAdd(next, 1);
      c = __shfl_sync(0xFFFFFFFFu, c, 0) * 32;
      if (c >= cnt) return;
      if (c + lane < cnt) z[c + lane] = normal(seed, (uint64_t)(lo + c + lane), (uint64_t)step);
    }
  }
  int pend = 0;  // neurons in `retry`
  auto again = [&](int from, int count) {
    __syncwarp();
    if (lane < count) {
      const int i = retry[from + lane];
      float x = 0.0f, s = 0.0f;
      bool ok = false;
      for (uint32_t attempt = 1; attempt < 16 && !ok; ++attempt)
        ok = normal_try(k0, k1, (uint32_t)(lo + i), (uint32_t)step, attempt, x, s);
      z[i] = ok ? normal_value(x, s) : 0.0f;
    }
    __syncwarp();
  };
  for (;;) {
    int c = 0;
    if (lane == 0) c = atomicAdd(next, 1);
    c = __shfl_sync(0xFFFFFFFFu, c, 0) * 32;
    if (c >= cnt) break;
    const int i = c + lane;
    float x = 0.0f, s = 0.0f;
    bool ok = false;
    ok = normal_try(k0, k1, (uint32_t)(lo + i), (uint32_t)step, 0, x, s);
    if (i < cnt && ok) z[i] = normal_value(x, s);
    const unsigned bad = __ballot_sync(0xFFFFFFFFu, !ok && i < cnt);
    if (bad) {
      if (bad >> lane & 1u) retry[pend + __popc(bad & below)] = i;
      pend += __popc(bad);
      if (pend >= 32) {
        pend -= 32;
        again(pend, 32);
      }
    }
  }
  if (pend) again(0, pend);
}

// Ids of a[0..n) below x.  A rank's spikes go to the raster in ascending order by it (ranks own
// ascending ranges, so the step's ids are then in order and the host has nothing to sort:
// 546,000 ids took it 3.5 ms), up to kOrderSpikes of them: a rank has some tens, four ids a
// load; a larger burst is left to the host rather than compared in n^2.
constexpr int kOrderSpikes = 512;
__device__ __forceinline__ int rank_of(const int *a, int n, int x) {
  int r = 0, k = 0;
  for (; k + 4 <= n; k += 4) {
    const int4 q = *reinterpret_cast<const int4 *>(a + k);
    r += (q.x < x) + (q.y < x) + (q.z < x) + (q.w < x);
  }
  for (; k < n; ++k) r += a[k] < x;
  return r;
}

// ---------------------------------------------------------------------------------------
// One team member's share of one network for the steps of this launch.
// ---------------------------------------------------------------------------------------

template <int NT, bool kPair, int kMode, bool kSolo>
__device__ void team_run(const TeamItem &it, int rank, unsigned char *s_raw, TeamShared &sh,
                         unsigned long long limit_ns, int stall) {
  const NetView &v = it.v;
  const int lo = (int)min((int64_t)rank * it.rc, v.n);
  const int cnt = (int)min((int64_t)it.rc, v.n - lo);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kWarps = NT / 32, kSrc = source_warps(NT, kMode);
  const bool solo = kSolo && it.team == 1;  // the whole network in this CTA: no exchange
  const bool lead = rank == 0 && threadIdx.x == 0;
  if (threadIdx.x == 0) {
    sh.L = team_layout(it.rc, it.team, it.col, own_sources(it.team, NT == kTeamNTSmall && kMode == kDeliverRun));
    sh.rank = rank;
    sh.nown[0] = sh.nown[1] = 0;
    sh.work[0] = sh.work[1] = 0;
    sh.k[0] = sh.k[1] = 0u;
    sh.off[0] = sh.off[1] = 0;
    sh.base = 0;
    sh.fail = 0;
  }
  __shared__ __align__(16) WarpScratch s_ws[kWarps];
  __syncthreads();
  const TeamLayout &L = sh.L;
  // arrays of the slice in shared memory, by their offsets
  auto s_abcd = [&] { return reinterpret_cast<float4 *>(s_raw + L.abcd); };
  auto s_vu = [&] { return reinterpret_cast<float2 *>(s_raw + L.vu); };
  auto s_a = [&] { return reinterpret_cast<int *>(s_raw + L.a); };
  auto s_b = [&] { return reinterpret_cast<unsigned *>(s_raw + L.b); };
  auto s_own = [&] { return reinterpret_cast<int *>(s_raw + L.own); };
  auto s_z = [&] { return reinterpret_cast<float *>(s_raw + L.z); };
  auto s_pay = [&] { return reinterpret_cast<unsigned *>(s_raw + L.pay); };

  for (int i = threadIdx.x; i < cnt; i += NT) {
    const long long q = __ldcg(v.acc + lo + i);
    s_a()[i] = (int)(q >> 16);
    s_b()[i] = (unsigned)(q & 0xFFFF);
    if (L.vu_sm) s_vu()[i] = v.vu[lo + i];
    if (L.abcd_sm) s_abcd()[i] = v.abcd[lo + i];
  }
  if (L.col_sm) {
    unsigned *col = reinterpret_cast<unsigned *>(s_raw + L.col);
    const uint16_t *so = it.seg + rank;
    const int64_t pitch = it.team + 1;
#pragma unroll 4
    for (int i = threadIdx.x; i < it.col; i += NT)
      col[i] = (unsigned)__ldg(so + i * pitch) | (unsigned)__ldg(so + i * pitch + 1) << 16;
  }
  if (L.pay_sm)  // the first step polls one record line per rank
    for (int r = threadIdx.x; r < it.team; r += NT) s_pay()[r * kRankWords] = 0;
  if (L.prez) drive_chunks(v.seed, lo, cnt, (int)it.t_abs0, s_z(), &sh.work[1], s_ws[warp].retry);
  __syncthreads();

  const int steps = it.steps;
  for (int lt = 0; lt < steps; ++lt) {
    const int t_abs = (int)it.t_abs0 + lt;
    const bool last = it.last && lt == steps - 1;
    const int par = lt & 1;
    if (threadIdx.x == NT - 32) {  // (a warp with less to do than the first ones)
      // the previous step's counters are final: its team count, then cleared for the next step
      const int k = (int)(sh.k[par ^ 1] & (kPolled - 1u));
      if (rank == 0 && lt > 0) v.counts[lt - 1] = k;
      sh.base += k;
      sh.lim = lt == 0 ? limit_ns * 16 : limit_ns;  // (members may start late)
      sh.nown[par ^ 1] = 0;
      sh.work[par ^ 1] = 0;
      sh.k[par ^ 1] = 0u;
      sh.off[par ^ 1] = 0;
      if (rank == 0) {
        v.base[lt] = sh.base;
        if (v.stamps) v.stamps[2 * lt] = globaltimer();
      }
    }
    // ---- update of the owned neurons, their state in shared memory for the launch when it
    // fits, else in global memory (a, b, c, d then recomputed from the parameter r)
    if (L.prez && warp * 32 < cnt) {
      const Update w{L.vu_sm ? s_vu() : v.vu + lo, L.abcd_sm ? s_abcd() : v.abcd + lo, v.rpar + lo, s_z(), s_a(), s_b(),
                     last ? v.ilast + lo : nullptr, s_own(), &sh.nown[par], cnt, (int)min(v.nexc - lo, (int64_t)cnt),
                     lo, v.ge, v.gi};
      if (L.abcd_sm || !v.rpar)
        update_slice<NT, false>(w);
      else
        update_slice<NT, true>(w);
    } else if (!L.prez) {
      // no room for the next step's drive: computed here, one neuron at a time with the next
      // one's state in flight
      float2 *vu = v.vu + lo;
      int *sa = s_a();
      unsigned *sb = s_b();
      float2 sn = threadIdx.x < cnt ? vu[threadIdx.x] : make_float2(0.0f, 0.0f);
      for (int i = threadIdx.x; i < cnt; i += NT) {
        float2 s = sn;
        if (i + NT < cnt) sn = vu[i + NT];
        const int nn = lo + i;
        const float4 p = v.rpar ? izh_abcd(v.rpar[nn], nn < v.nexc) : v.abcd[nn];
        const float z = normal(v.seed, (uint64_t)nn, (uint64_t)t_abs);
        const float isyn = split_current(sa[i], sb[i]);
        sa[i] = 0;
        sb[i] = 0;
        float I;
        const bool k = izh_step(s.x, s.y, I, p, nn < v.nexc ? v.ge : v.gi, z, isyn);
        vu[i] = s;
        if (last) v.ilast[nn] = I;
        if (k) s_own()[atomicAdd(&sh.nown[par], 1)] = nn;
      }
    }
    __syncthreads();
    const int nown = sh.nown[par];
    if (stall == kStallFault && solo) {
      // injected fault of a one-CTA team: wait for a member that does not exist
      if (threadIdx.x == 0) {
        const unsigned long long lim = sh.lim, t0 = globaltimer();
        while (ld_relaxed(&it.sync->error) == 0 && globaltimer() - t0 <= lim) {
        }
        give_up(it, sh);
      }
      __syncthreads();
      return;
    }
    const unsigned rel_a = (unsigned)__cvta_generic_to_shared(s_a()) - (unsigned)lo * 4u;
    const unsigned rel_b = (unsigned)__cvta_generic_to_shared(s_b()) - (unsigned)lo * 4u;
    if (solo) {
      if (threadIdx.x == 0) {
        sh.k[par] = (unsigned)nown;
        if (lead && v.stamps) v.stamps[2 * lt + 1] = globaltimer();
      }
      deliver_solo<NT, kPair>(it, s_own(), nown, rel_a, rel_b);
    } else {
      Source c;
      c.lt = lt;
      const bool own_sources = L.pay_sm;  // every warp polls source ranks of its own
      const unsigned tag = it.tag0 + (unsigned)lt + 1u;
      const unsigned long long *recs = it.rec + (size_t)par * it.team * kRankWords;
      // ---- publish: both record lines of this rank (count, ids, padding), ids beyond them
      // in the overflow list; every word tagged with the step, so no fence is needed
      {
        const unsigned long long tg = (unsigned long long)tag << 32;
        static_assert(kRankWords == 32, "one warp publishes");
        if (warp == 0) {
          const int j = lane;
          const unsigned pay = j == 0 ? (unsigned)nown : (j - 1 < nown ? (unsigned)s_own()[j - 1] : 0xFFFFFFFFu);
          st_relaxed_u64(it.rec + ((size_t)par * it.team + rank) * kRankWords + j, tg | pay);
        }
        if (nown > kInline) {
          unsigned long long *ovf = it.list + (size_t)par * v.n + lo;
          for (int j = kInline + threadIdx.x; j < nown; j += NT) st_relaxed_u64(ovf + j, tg | (unsigned)s_own()[j]);
        }
      }
      // ---- the other ranks' spikes, polled until the words carry the step's tag
      int n_src, cl = 0;  // sources of this warp; this lane's source's spikes
      unsigned long long t0 = 0;
      c.inl = 0;
      if (own_sources) {
        // every warp its own source ranks warp, warp + kSrc, ...: line 0 of each, and line 1
        // of those that had more than kLine1After spikes in the previous step, as 16-byte
        // slots, eight a line, up to two lines' slots per lane.  No warp waits for another
        // one's sources: it delivers as soon as its own have arrived.
        n_src = warp < min(kSrc, it.team) ? (it.team - 1 - warp) / kSrc + 1 : 0;
        if (n_src) {
          const int mine = lane < n_src ? (int)s_pay()[(warp + lane * kSrc) * kRankWords] : 0;
          const unsigned more = __ballot_sync(0xFFFFFFFFu, mine > kLine1After);
          c.inl = mine > kLine1After ? kInline : kRecWords - 1;
          const int src = lane >> 3;
          unsigned need = (src < n_src ? 1u : 0u) | (src + 4 < n_src ? 2u : 0u);
          need |= need << 2 & ((more >> src & 1u) << 2 | (more >> (src + 4) & 1u) << 3);
          const unsigned long long *p = recs + (warp + src * kSrc) * kRankWords + 2 * (lane & 7);
          unsigned *to = s_pay() + (warp + src * kSrc) * kRankWords + 2 * (lane & 7);
          for (unsigned iter = 0;; ++iter) {
            ulonglong2 a[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (need & (1u << k))
                a[k] = ld_relaxed_u64x2(p + (k & 1) * 4 * kSrc * kRankWords + (k >> 1) * kRecWords);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if ((need & (1u << k)) && (unsigned)(a[k].x >> 32) == tag && (unsigned)(a[k].y >> 32) == tag) {
                *reinterpret_cast<uint2 *>(to + (k & 1) * 4 * kSrc * kRankWords + (k >> 1) * kRecWords) =
                    make_uint2((unsigned)a[k].x, (unsigned)a[k].y);
                need &= ~(1u << k);
              }
            if (__all_sync(0xFFFFFFFFu, need == 0) && stall == 0) break;
            if (NT == kTeamNT && kMode == kDeliverRun && !kSolo && L.prez && lt + 1 < steps) {
              // large steps, whose ranks finish some thousand cycles apart: a chunk of the next
              // step's drive instead of waiting (N=10^6 40.7 -> 40.1 us a step; smaller steps wait
              // for about one trip to L2, and lose by it).  Taken only while there is one: a warp
              // goes past the last chunk once, not in every round of a wait of any length.
              int ch = cnt;
              if (lane == 0 && *(volatile int *)&sh.work[par] * 32 < cnt) ch = atomicAdd(&sh.work[par], 1) * 32;
              ch = __shfl_sync(0xFFFFFFFFu, ch, 0) + lane;
              if (ch < cnt) s_z()[ch] = normal(v.seed, (uint64_t)(lo + ch), (uint64_t)(t_abs + 1));
              __syncwarp();
            }
            if (poll_check(it, sh, iter, t0, sh.lim)) {
              n_src = 0;  // (the words read may be old)
              break;
            }
          }
          __syncwarp();
          if (lane < n_src) cl = (int)s_pay()[(warp + lane * kSrc) * kRankWords];
        }
      } else {
        // few ranks: every warp reads every rank's count and takes its share of the batches
        n_src = it.team;
        for (unsigned iter = 0;; ++iter) {
          unsigned long long w = 0;
          if (lane < n_src) w = ld_relaxed_u64(recs + lane * kRankWords);
          if (__all_sync(0xFFFFFFFFu, lane >= n_src || (unsigned)(w >> 32) == tag) && stall == 0) {
            cl = lane < n_src ? (int)(unsigned)w : 0;
            break;
          }
          if (poll_check(it, sh, iter, t0, sh.lim)) break;
        }
      }
      {
        int incl = cl;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {  // (at most sixteen sources)
          const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
          if (lane >= o) incl += y;
        }
        c.total = __shfl_sync(0xFFFFFFFFu, incl, 15);
        c.off = lane < n_src ? incl - cl : INT_MAX;
      }
      if (c.total) {
        const int below = __reduce_add_sync(0xFFFFFFFFu, (own_sources ? warp + lane * kSrc : lane) < rank ? cl : 0);
        if (lane == 0 && below && (own_sources || warp == 0)) atomicAdd(&sh.off[par], below);
      }
      if (lane == 0 && (own_sources || warp == 0)) {
        // the step's team count and this rank's raster offset, for the tail
        __threadfence_block();
        atomicAdd(&sh.k[par], kPolled + (unsigned)c.total);
      }
      if (lead && v.stamps) v.stamps[2 * lt + 1] = globaltimer();
      c.q0 = 0;
      c.dq = 32;
      c.wi = 0;
      c.wpb = 1;
      if (!own_sources) {
        const int nbatch = (c.total + 31) >> 5;
        int wpb = nbatch >= kWarps ? 1 : kWarps / max(nbatch, 1);
        if (kMode == kDeliverGroup) wpb = min(8, wpb);
        const int groups = kWarps / wpb;
        c.q0 = warp / wpb < groups ? warp / wpb * 32 : c.total;
        c.dq = groups * 32;
        c.wi = warp % wpb;
        c.wpb = wpb;
      }
      if constexpr (kMode == kDeliverGroup)
        deliver_group<NT, kPair>(it, sh, s_raw, c, rel_a, rel_b);
      else
        deliver_run<NT, kPair>(it, sh, s_raw, c, rel_a, rel_b, s_ws[warp]);
    }
    // ---- tail, by warps as they finish delivering: the raster and the statistics of this
    // rank's spikes (from the highest thread down), then the next step's drive in chunks of
    // 32 neurons
    if (NT - 32 - warp * 32 < nown) {
      if (!solo) {  // (every warp's sources are counted, unless the exchange gave up)
        const int all = L.pay_sm ? kWarps : 1;
        while ((int)(*(volatile unsigned *)&sh.k[par] / kPolled) < all && !*(volatile int *)&sh.fail) {
        }
        __threadfence_block();
      }
      const long long pos0 = sh.base + *(volatile int *)&sh.off[par];
      for (int j = NT - 1 - threadIdx.x; j < nown; j += NT) {
        const int n = s_own()[j];
        if (v.raster_cap > 0) {
          const long long pos = pos0 + (nown <= kOrderSpikes ? rank_of(s_own(), nown, n) : j);
          if (pos < v.raster_cap) v.raster[pos] = n;
        }
        SpikeStat st = v.sstat[n];
        st.nospks += 1;
        if (st.last >= 0) {
          const long long isi = t_abs - st.last;
          st.nisi += 1;
          st.s1 += isi;
          st.s2 += isi * isi;
        }
        st.last = t_abs;
        v.sstat[n] = st;
      }
    }
    if (L.prez && lt + 1 < steps && __any_sync(0xFFFFFFFFu, *(volatile int *)&sh.work[par] * 32 < cnt))
      drive_chunks(v.seed, lo, cnt, t_abs + 1, s_z(), &sh.work[par], s_ws[warp].retry);
    __syncthreads();
    if (!solo && sh.fail) return;
  }
  if (lead) v.counts[steps - 1] = (int)(sh.k[(steps - 1) & 1] & (kPolled - 1u));
  // pending currents (from the last delivery) and the state back to global memory
  for (int i = threadIdx.x; i < cnt; i += NT) {
    v.acc[lo + i] = (long long)s_a()[i] * 65536 + s_b()[i];
    if (L.vu_sm) v.vu[lo + i] = s_vu()[i];
  }
  __syncthreads();
}

// The persistent grid: CTA b takes (network, rank) slot b, then the next ones of the queue
// until it is empty (a launch whose slots all fit the grid makes no trip to the queue head).
template <int NT, bool kPair, int kMode, bool kSolo>
__global__ void __launch_bounds__(NT, 1) k_team(const TeamItem *__restrict__ items, const int2 *__restrict__ slots,
                                                int nslots, int *slot_head, unsigned long long limit_ns, int stall) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ TeamShared sh;
  // the network's descriptor in shared memory: read on every step's dependent chains
  __shared__ TeamItem s_it;
  for (int sl = blockIdx.x; sl < nslots;) {
    const int2 x = slots[sl];
    for (unsigned k = threadIdx.x; k < sizeof(TeamItem) / 8; k += NT)
      reinterpret_cast<unsigned long long *>(&s_it)[k] = reinterpret_cast<const unsigned long long *>(items + x.x)[k];
    __syncthreads();
    if (s_it.steps > 0) team_run<NT, kPair, kMode, kSolo>(s_it, x.y, s_raw, sh, limit_ns, stall);
    if (nslots <= (int)gridDim.x) break;
    if (threadIdx.x == 0) sh.slot = (int)gridDim.x + atomicAdd(slot_head, 1);
    __syncthreads();
    sl = sh.slot;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------
// Launchers.
// ---------------------------------------------------------------------------------------

size_t team_smem(int64_t rc, int team, int64_t col) {
  if (rc < 1 || team < 1 || team > kMaxTeam) return 0;
  const size_t bytes = team_layout(rc, team, col, own_sources(team, true)).bytes;  // (the kernel that takes most)
  return bytes > kTeamSmemLimit ? 0 : (bytes < 16 ? 16 : bytes);
}

// The instantiation of the team kernel for a CTA size, table layout and delivery mapping.
using TeamKernel = void (*)(const TeamItem *, const int2 *, int, int *, unsigned long long, int);
template <int NT, bool kPair, int kMode>
static TeamKernel team_kernel_of(bool solo) {
  return solo ? k_team<NT, kPair, kMode, true> : k_team<NT, kPair, kMode, false>;
}
template <int NT>
static TeamKernel team_kernel_nt(bool pair, int mode, bool solo) {
  if (mode == kDeliverGroup)
    return pair ? team_kernel_of<NT, true, kDeliverGroup>(solo) : team_kernel_of<NT, false, kDeliverGroup>(solo);
  return pair ? team_kernel_of<NT, true, kDeliverRun>(solo) : team_kernel_of<NT, false, kDeliverRun>(solo);
}
static TeamKernel team_kernel(int nt, bool pair, int mode, bool solo) {
  return nt == kTeamNTSmall ? team_kernel_nt<kTeamNTSmall>(pair, mode, solo) : team_kernel_nt<kTeamNT>(pair, mode, solo);
}
constexpr int kTeamVariants = 8;  // of one CTA size
static TeamKernel team_variant(int nt, int k) {
  return team_kernel(nt, k & 1, k & 2 ? kDeliverGroup : kDeliverRun, k & 4);
}

// The kernel's shared-memory ceiling is always the largest layout's (every team layout
// stays under it), so host threads that launch teams of different sizes never lower it
// under one another, and a captured launch needs no attribute call.
cudaError_t team_smem_ceiling() {
  cudaError_t e = cudaSuccess;
  for (int nt : {kTeamNT, kTeamNTSmall})
    for (int k = 0; k < kTeamVariants && e == cudaSuccess; ++k)
      e = cudaFuncSetAttribute(team_variant(nt, k), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTeamSmemLimit);
  return e;
}

cudaError_t team_max_blocks(size_t smem, int *out, int nt) {
  if (smem > kTeamSmemLimit || (nt != kTeamNT && nt != kTeamNTSmall)) return cudaErrorInvalidValue;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  // Constants of the device (a CTA's registers leave room for one per SM, whatever its shared
  // memory): asked for once, a batch plans with them once per network.
  static std::mutex mu;
  static std::map<std::pair<int, int>, int> known;
  std::lock_guard<std::mutex> lk(mu);
  auto it = known.find({dev, nt});
  if (it == known.end()) {
    if ((e = team_smem_ceiling()) != cudaSuccess) return e;
    int least = INT_MAX, sms = 1;  // (of the instantiations, which need nearly the same resources)
    for (int k = 0; k < kTeamVariants; ++k) {
      int occ = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, team_variant(nt, k), nt, kTeamSmemLimit);
      if (e != cudaSuccess) return e;
      least = std::min(least, occ);
    }
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    it = known.emplace(std::make_pair(dev, nt), least * sms).first;
  }
  *out = it->second;
  return cudaSuccess;
}

cudaError_t launch_team(const TeamItem *items, const int2 *slots, int nslots, int *slot_head, int grid,
                        size_t smem, unsigned long long limit_ns, int stall, cudaStream_t s, bool pair, int mode,
                        bool solo, int nt) {
  if (smem > kTeamSmemLimit || (nt != kTeamNT && nt != kTeamNTSmall)) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, team_kernel(nt, pair, mode, solo), items, slots, nslots, slot_head, limit_ns, stall);
}

cudaError_t launch_rows_sorted(const NetView &v, int *unsorted, cudaStream_t s) {
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e = cudaMemsetAsync(unsorted, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  k_rows_sorted<<<(unsigned)(sms * 8), 512, 0, s>>>(v, unsorted);
  return cudaGetLastError();
}

cudaError_t launch_first_bad(const int *idx, const NetView &v, unsigned long long *first, cudaStream_t s) {
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e = cudaMemsetAsync(first, 0xFF, 8, s);
  if (e != cudaSuccess) return e;
  k_first_bad<<<(unsigned)(sms * 4), 512, 0, s>>>(reinterpret_cast<const int4 *>(idx), v, first);
  return cudaGetLastError();
}

// One CTA per row, as many resident as fit (at most one per row).  The shared-memory
// ceiling is the same for every network, so that host threads sorting rows of different
// lengths never lower it under one another's launch.
template <typename Kernel>
static cudaError_t row_grid(Kernel kern, int nt, size_t smem, int64_t rows, unsigned *grid) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e != cudaSuccess) return e;
  int occ = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, nt, smem);
  if (occ < 1) occ = 1;
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int64_t g = (int64_t)sms * occ;
  *grid = (unsigned)(g > rows ? rows : g);
  return cudaSuccess;
}

template <int E>
static cudaError_t sort_rows_e(const NetView &v, int p2, int nt, cudaStream_t s) {
  const size_t smem = nt > 32 ? (size_t)p2 * 8 : 0;  // (one warp needs no shared memory)
  unsigned g = 0;
  cudaError_t e = row_grid(k_sort_rows<E>, nt, smem, v.n, &g);
  if (e != cudaSuccess) return e;
  k_sort_rows<E><<<g, nt, smem, s>>>(v, p2);
  return cudaGetLastError();
}

template <int E>
static cudaError_t sort_gen_e(const NetView &v, int p2, int pb, cudaStream_t s) {
  const int nt = p2 / E, nb = std::max(nt, p2 / 2);
  int sh = 0;
  while ((v.n >> sh) >= nb) ++sh;
  const size_t smem = ((size_t)nb + 32 + 2 * (size_t)v.stride) * 4;
  unsigned g = 0;
  cudaError_t e = row_grid(k_sort_gen<E>, nt, smem, v.n, &g);
  if (e != cudaSuccess) return e;
  k_sort_gen<E><<<g, nt, smem, s>>>(v, pb, nb, sh);
  return cudaGetLastError();
}

cudaError_t launch_sort_rows(const NetView &v, bool generated, cudaStream_t s) {
  int p2 = 32, pb = 5;
  while (p2 < v.stride) p2 <<= 1, ++pb;
  if ((size_t)p2 * 8 > 200 * 1024) return cudaErrorInvalidValue;
  if (generated && ((uint64_t)v.n << pb) + (uint64_t)p2 - 1 < 0xFFFFFFFFull) {
    // E keys a thread: 8 (16 for rows longer than 8192), fewer for rows shorter than 256
    const int E = p2 / 32 < 8 ? p2 / 32 : (p2 / 8 > 1024 ? 16 : 8);
    switch (E) {
      case 1: return sort_gen_e<1>(v, p2, pb, s);
      case 2: return sort_gen_e<2>(v, p2, pb, s);
      case 4: return sort_gen_e<4>(v, p2, pb, s);
      case 8: return sort_gen_e<8>(v, p2, pb, s);
      case 16: return sort_gen_e<16>(v, p2, pb, s);
      default: return cudaErrorInvalidValue;
    }
  }
  const int nt = std::min(1024, std::max(32, p2 / 4));  // four keys a thread (up to 16 for long rows)
  switch (p2 / nt) {
    case 1: return sort_rows_e<1>(v, p2, nt, s);
    case 2: return sort_rows_e<2>(v, p2, nt, s);
    case 4: return sort_rows_e<4>(v, p2, nt, s);
    case 8: return sort_rows_e<8>(v, p2, nt, s);
    case 16: return sort_rows_e<16>(v, p2, nt, s);
    default: return cudaErrorInvalidValue;
  }
}

// ---------------------------------------------------------------------------------------
// Set-up and read-back of a launch over many networks, one CTA per network.  k_round_clear
// zeroes each network's per-step counts and stamps of the launch, its status word and its
// team's error word and spike records; k_round_gather packs its status words, counts,
// raster offsets and stamps at its offset in one buffer (round_pack_bytes each), which one
// copy brings to the host.  Networks with no steps in the launch are skipped.
// ---------------------------------------------------------------------------------------
__global__ void k_round_clear(const TeamItem *items) {
  const TeamItem &it = items[blockIdx.x];
  const int s = it.steps;
  if (s <= 0) return;
  for (int i = threadIdx.x; i < s; i += blockDim.x) it.v.counts[i] = 0;
  for (int i = threadIdx.x; i < 2 * s + 2; i += blockDim.x) it.v.stamps[i] = 0ull;
  if (threadIdx.x == 0) *it.v.status = 0;
  unsigned long long *g = reinterpret_cast<unsigned long long *>(it.sync);
  const int64_t words = (int64_t)(1 + 2 * it.team * kRecLines) * (int64_t)(sizeof(GridSync) / 8);
  for (int64_t i = threadIdx.x; i < words; i += blockDim.x) g[i] = 0ull;
}

__device__ __forceinline__ void gather_steps(const NetView &v, const GridSync *gs, int s, unsigned char *p) {
  if (threadIdx.x == 0) {
    reinterpret_cast<int *>(p)[0] = *v.status;
    reinterpret_cast<int *>(p)[1] = gs->error;
  }
  int *c = reinterpret_cast<int *>(p + 8);
  long long *b = reinterpret_cast<long long *>(p + 8 + (((size_t)s * 4 + 7) & ~(size_t)7));
  unsigned long long *t = reinterpret_cast<unsigned long long *>(b + s);
  for (int i = threadIdx.x; i < s; i += blockDim.x) {
    c[i] = v.counts[i];
    b[i] = v.base[i];
  }
  for (int i = threadIdx.x; i < 2 * s; i += blockDim.x) t[i] = v.stamps[i];
}

__global__ void k_round_gather(const TeamItem *items, const int64_t *off, unsigned char *pack) {
  const TeamItem &it = items[blockIdx.x];
  if (it.steps > 0) gather_steps(it.v, it.sync, it.steps, pack + off[blockIdx.x]);
}

// The same for one network's chunk by another kernel.
__global__ void k_chunk_gather(NetView v, const GridSync *gs, int steps, unsigned char *pack) {
  gather_steps(v, gs, steps, pack);
}

cudaError_t launch_round_clear(const TeamItem *items, int count, cudaStream_t s) {
  k_round_clear<<<(unsigned)count, 512, 0, s>>>(items);
  return cudaGetLastError();
}

cudaError_t launch_round_gather(const TeamItem *items, const int64_t *off, int count, unsigned char *pack,
                                cudaStream_t s) {
  k_round_gather<<<(unsigned)count, 512, 0, s>>>(items, off, pack);
  return cudaGetLastError();
}

cudaError_t launch_chunk_gather(const NetView &v, const GridSync *gs, int steps, unsigned char *pack, cudaStream_t s) {
  k_chunk_gather<<<1, 512, 0, s>>>(v, gs, steps, pack);
  return cudaGetLastError();
}

cudaError_t launch_segoff(const NetView &v, int team, int64_t rc, uint16_t *seg, cudaStream_t s) {
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int64_t blocks = (v.n + 7) / 8;
  if (blocks > (int64_t)sms * 16) blocks = (int64_t)sms * 16;
  k_segoff<<<(unsigned)blocks, 256, 0, s>>>(v, team, rc, seg);
  return cudaGetLastError();
}

// Counters in shared memory up to this many parts, as each part reads every target again:
// with six parts (N=300,000) 4.5 ps a synapse, with eight 5.4, against k_inbound's 6.3.
constexpr int kInboundMaxParts = 8;

cudaError_t launch_inbound(const NetView &v, unsigned *cnt, unsigned long long *mag, unsigned long long *out,
                           cudaStream_t s) {
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e = cudaMemsetAsync(cnt, 0, (size_t)v.n * 4, s);
  if (e == cudaSuccess && mag) e = cudaMemsetAsync(mag, 0, (size_t)v.n * 8, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(out, 0, 24, s);
  if (e != cudaSuccess) return e;
  const int64_t parts = (v.n + kInboundPart - 1) / kInboundPart;
  if (!mag && parts <= kInboundMaxParts && parts <= sms) {
    const size_t smem = (size_t)std::min<int64_t>(v.n, kInboundPart) * 4;
    e = cudaFuncSetAttribute(k_inbound_shared, cudaFuncAttributeMaxDynamicSharedMemorySize, kInboundPart * 4);
    if (e != cudaSuccess) return e;
    k_inbound_shared<<<(unsigned)sms, 1024, smem, s>>>(v, (int)parts, cnt, out + 2);
  } else {
    k_inbound<<<(unsigned)(sms * 8), 512, 0, s>>>(v, cnt, mag, out + 2);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  k_inbound_max<<<(unsigned)std::min<int64_t>(sms, (v.n + 511) / 512), 512, 0, s>>>(v.n, cnt, mag, out);
  return cudaGetLastError();
}

cudaError_t launch_pairs(const NetView &v, cudaStream_t s) {
  if (!v.pair) return cudaErrorInvalidValue;
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  k_pairs<<<(unsigned)(sms * 4), 512, 0, s>>>(
      v, reinterpret_cast<ulonglong2 *>(const_cast<unsigned long long *>(v.pair)));
  return cudaGetLastError();
}

}  // namespace g4s
