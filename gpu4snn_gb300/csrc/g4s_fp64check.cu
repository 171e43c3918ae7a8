// g4s_fp64check.cu — on-device FP64 check of a network's FP32 trajectory.
//
// The library computes the reference's update in FP32 (gpu4snn.cu:376-405) with exact
// Q32.32 currents.  This check steps the network together with an FP64 twin, a chunk of
// steps in one cooperative launch, the FP32 side with the library's own step arithmetic (in
// the global-memory form, whose results are those of every scheme), on the same random
// draws: the float normal of each (neuron, step) and the float parameters promoted to
// double; v and u in double, every operation an explicit round-to-nearest double
// intrinsic in the C order of the reference's expressions (no fused multiply-add); the
// synaptic currents as exact Q64.64 sums of the weights — a 128-bit two's-complement
// integer per neuron, added with two 64-bit atomics and a carry — converted to double,
// correctly rounded, when the neuron consumes them.  Exact sums make the twin independent
// of the delivery order, so it equals the CPU oracle's FP64 mode bit for bit.  After every
// step it reports the maximum, 99th percentile and median of |v32 - v64| over all neurons
// (nearest-rank percentiles) and whether the two steps' spike sets agree.  The differences
// of a chunk's steps are kept, and a CTA per step selects their percentiles afterwards.
// Per step of N=20,000 x 1000: a one-step launch, three kernels, n doubles to the host and a
// selection there took 340 us.
//
// FP64 arithmetic on the GPU is used only here and in the statistics reductions.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/gpu4snn.h"
#include "g4s_device.cuh"
#include "g4s_internal.h"

using namespace g4s;

namespace {

struct alignas(16) Q128 {
  unsigned long long lo, hi;  // two's complement, value = (hi:lo) x 2^-64
};

// Q64.64 value of a float weight: exact for |w| >= 2^-41 (24 significant bits land on or
// above the 2^-64 bit), rounded to nearest even below.  Weights of magnitude 2^40 or more,
// infinities and NaNs do not fit: they raise *bad and count as 0.
__device__ __forceinline__ Q128 wq64(float w, int *bad) {
  const uint32_t b = __float_as_uint(w);
  const int e = (int)((b >> 23) & 0xFFu);
  Q128 q{0ull, 0ull};
  if (e == 0) return q;  // zero or subnormal (< 2^-126): rounds to 0 at 2^-64
  if (e >= 127 + 40) {
    atomicOr(bad, 1);
    return q;
  }
  const unsigned long long m = (unsigned long long)((b & 0x7FFFFFu) | 0x800000u);  // w = m 2^(e-150)
  const int sh = e - 86;                                                           // w 2^64 = m 2^sh < 2^104
  unsigned __int128 mag;
  if (sh >= 0) {
    mag = (unsigned __int128)m << sh;
  } else {
    const int r = -sh;
    if (r > 25) return q;  // m 2^-r < 2^-1: rounds to 0
    unsigned long long t = m >> r;
    const unsigned long long rem = m & ((1ull << r) - 1ull), half = 1ull << (r - 1);
    if (rem > half || (rem == half && (t & 1ull))) ++t;
    mag = t;
  }
  if (b >> 31) mag = (unsigned __int128)0 - mag;
  q.lo = (unsigned long long)mag;
  q.hi = (unsigned long long)(mag >> 64);
  return q;
}

__device__ __forceinline__ void q128_add(Q128 *a, Q128 x) {
  const unsigned long long old = atomicAdd(&a->lo, x.lo);
  const unsigned long long carry = (old + x.lo < old) ? 1ull : 0ull;  // unsigned wrap of the low word
  const unsigned long long hi = x.hi + carry;
  if (hi) atomicAdd(&a->hi, hi);
}

// (hi:lo) x 2^-64 to the nearest double (ties to even): the top 53 significant bits of the
// magnitude, rounded on the bits below them, scaled by exact powers of two.
__device__ __forceinline__ double q128_to_double(Q128 q) {
  unsigned __int128 x = ((unsigned __int128)q.hi << 64) | q.lo;
  const bool neg = (q.hi >> 63) != 0;
  if (neg) x = (unsigned __int128)0 - x;
  if (x == 0) return 0.0;
  const unsigned long long xh = (unsigned long long)(x >> 64), xl = (unsigned long long)x;
  const int bits = xh ? 128 - __clzll((long long)xh) : 64 - __clzll((long long)xl);
  unsigned long long top;
  int sh = 0;
  if (bits <= 53) {
    top = xl;
  } else {
    sh = bits - 53;
    top = (unsigned long long)(x >> sh);
    const unsigned __int128 rem = x & (((unsigned __int128)1 << sh) - 1);
    const unsigned __int128 half = (unsigned __int128)1 << (sh - 1);
    if (rem > half || (rem == half && (top & 1ull))) ++top;
    if (top == (1ull << 53)) {
      top >>= 1;
      ++sh;
    }
  }
  // 2^(sh - 64) as a double: sh - 64 lies in [-64, 11], a normal exponent
  const double scale = __longlong_as_double((long long)(1023 + sh - 64) << 52);
  const double d = __dmul_rn(__ull2double_rn(top), scale);
  return neg ? -d : d;
}

__global__ void k64_init(NetView v, double2 *vu64, Q128 *acc) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < v.n; i += (int64_t)gridDim.x * blockDim.x) {
    const double v0 = (double)v.vu[i].x;
    vu64[i] = make_double2(v0, __dmul_rn((double)v.abcd[i].y, v0));
    acc[i] = Q128{0ull, 0ull};
  }
}

// One step of the network and its twin, the phases of the library's persistent kernel
// (g4s_kernels.cu) for both: update of every neuron in FP32 and in FP64, |v32 - v64| of each to
// dv, the spiking ids to the raster and to the twin's list; grid barrier; both sides' spiking
// rows into their currents; grid barrier.  The drive of a thread's first neuron is drawn while
// it waits.  Bound by the barriers and round trips for small networks, by the FP64 pipe (two
// lanes a cycle and SM; some 25 operations a neuron) for large ones.
struct Twin {
  double2 *vu;
  Q128 *acc;
  int *list;     // the step's spiking ids
  int *count;    // [steps] ... and their number
  double *dv;    // [steps][n]
  int *first;    // first step whose spike sets differ
  int *bad;      // a weight that Q64.64 does not hold
};

constexpr int kTwinNT = 256;

__global__ void __launch_bounds__(kTwinNT, 2) k64_lockstep(NetView v, Twin w, int64_t t_abs0, int nsteps, int last_chunk,
                                                           GridSync *gs, unsigned long long limit_ns, int stall) {
  constexpr int NT = kTwinNT;
  __shared__ int s_ids[2][NT], s_n[2];
  __shared__ long long s_at[2];
  unsigned epoch = 0;
  long long base = 0;
  const unsigned nb = gridDim.x + (unsigned)stall;  // stall > 0 only under fault injection
  const int64_t first = (int64_t)blockIdx.x * NT + threadIdx.x;
  float z0 = first < v.n ? normal(v.seed, (uint64_t)first, (uint64_t)t_abs0) : 0.0f;
  for (int lt = 0; lt < nsteps; ++lt) {
    const int64_t t_abs = t_abs0 + lt;
    const bool last = last_chunk && lt == nsteps - 1;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      v.base[lt] = base;
      v.stamps[2 * lt] = globaltimer();
    }
    unsigned mine = 0;
    for (int64_t i0 = (int64_t)blockIdx.x * NT; i0 < v.n; i0 += (int64_t)gridDim.x * NT) {
      if (threadIdx.x < 2) s_n[threadIdx.x] = 0;
      __syncthreads();
      const int64_t i = i0 + threadIdx.x;
      if (i < v.n) {
        const float4 p = v.abcd[i];
        const float z = i == first ? z0 : normal(v.seed, (uint64_t)i, (uint64_t)t_abs);
        const float g = i < v.nexc ? v.ge : v.gi;
        float2 s = v.vu[i];
        const long long a = __ldcg(v.acc + i);
        float I32;
        const bool spk = izh_step(s.x, s.y, I32, p, g, z, q32_current(a));
        v.vu[i] = s;
        v.acc[i] = 0;
        if (last) v.ilast[i] = I32;
        if (spk) {
          s_ids[0][atomicAdd(&s_n[0], 1)] = (int)i;
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
        // the FP64 step (stateupdate, gpu4snn.cu:356-405, in double)
        const Q128 q{__ldcg(&w.acc[i].lo), __ldcg(&w.acc[i].hi)};
        w.acc[i] = Q128{0ull, 0ull};
        const double I = __dadd_rn(__dmul_rn((double)g, (double)z), q128_to_double(q));
        double vv = w.vu[i].x, uu = w.vu[i].y;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          double t1 = __dmul_rn(__dmul_rn(0.04, vv), vv);
          t1 = __dadd_rn(t1, __dmul_rn(5.0, vv));
          t1 = __dadd_rn(t1, 140.0);
          t1 = __dsub_rn(t1, uu);
          t1 = __dadd_rn(t1, I);
          vv = __dadd_rn(vv, __dmul_rn(0.5, t1));
        }
        uu = __dadd_rn(uu, __dmul_rn((double)p.x, __dsub_rn(__dmul_rn((double)p.y, vv), uu)));
        const bool spk64 = (vv >= 30.0) || !isfinite(vv);
        if (spk64) {
          vv = (double)p.z;
          uu = __dadd_rn(uu, (double)p.w);
          s_ids[1][atomicAdd(&s_n[1], 1)] = (int)i;
        }
        w.vu[i] = make_double2(vv, uu);
        w.dv[(size_t)lt * (size_t)v.n + (size_t)i] = fabs(__dsub_rn((double)s.x, vv));
        if (spk != spk64) atomicMin(w.first, (int)t_abs);
      }
      __syncthreads();
      const int n32 = s_n[0], n64 = s_n[1];
      if (threadIdx.x == 0 && n32) s_at[0] = base + atomicAdd(v.counts + lt, n32);
      if (threadIdx.x == 1 && n64) s_at[1] = atomicAdd(w.count + lt, n64);
      __syncthreads();
      if ((int)threadIdx.x < n32) {
        const long long pos = s_at[0] + threadIdx.x;
        if (pos < v.raster_cap)
          v.raster[pos] = s_ids[0][threadIdx.x];
        else
          atomicCAS(v.status, 0, kErrOverflowCode);
      }
      if ((int)threadIdx.x < n64) w.list[s_at[1] + threadIdx.x] = s_ids[1][threadIdx.x];
      mine += (unsigned)n32;
      __syncthreads();
    }
    grid_arrive(gs, epoch, mine);
    unsigned sum;
    if (!grid_wait(gs, epoch, nb, limit_ns, sum)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) v.stamps[2 * lt + 1] = globaltimer();
    const int K = (int)(sum - (unsigned)base), K64 = __ldcg(w.count + lt);
    deliver_flat(v, v.raster + base, K);
    // the twin's rows, flat over all synapses
    const uint64_t total = (uint64_t)K64 * (uint64_t)v.stride;
    for (uint64_t g = (uint64_t)blockIdx.x * NT + threadIdx.x; g < total; g += (uint64_t)gridDim.x * NT) {
      const uint64_t r = g / (uint32_t)v.stride, j = g - r * (uint32_t)v.stride;
      const size_t off = (size_t)__ldcg(w.list + r) * (size_t)v.stride + j;
      const int tg = v.idx[off];
      if (tg >= 0) q128_add(w.acc + tg, wq64(v.w[off], w.bad));
    }
    grid_arrive(gs, epoch, 0u);
    if (first < v.n && lt + 1 < nsteps) z0 = normal(v.seed, (uint64_t)first, (uint64_t)(t_abs + 1));
    if (!grid_wait(gs, epoch, nb, limit_ns, sum)) return;
    base += K;
  }
}

// Maximum and the values of ranks r99 and r50 of each row of dv (n non-negative doubles, which
// order as their bits), a CTA per row: radix selection from the top, 11 bits a pass, both
// ranks in each pass.  Six reads of a row, from L2 for the chunks that the host sizes.
constexpr int kSelBits = 11, kSelNT = 1024;
__global__ void __launch_bounds__(kSelNT) k64_select(const double *dv, int64_t n, int64_t r99, int64_t r50, double *out) {
  __shared__ unsigned s_hist[2][1 << kSelBits];
  __shared__ unsigned long long s_max, s_prefix[2];
  __shared__ long long s_rank[2];
  __shared__ unsigned s_part[32];
  const unsigned long long *x = reinterpret_cast<const unsigned long long *>(dv) + (size_t)blockIdx.x * (size_t)n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    s_max = 0ull;
    s_prefix[0] = s_prefix[1] = 0ull;
    s_rank[0] = r99;
    s_rank[1] = r50;
  }
  for (int shift = 64 - kSelBits; shift > -kSelBits; shift -= kSelBits) {
    const int sh = max(shift, 0);  // (the last pass takes the bits that are left)
    const int bits = shift < 0 ? kSelBits + shift : kSelBits;
    for (int k = threadIdx.x; k < 2 << kSelBits; k += kSelNT) (&s_hist[0][0])[k] = 0u;
    __syncthreads();
    const unsigned long long p0 = s_prefix[0], p1 = s_prefix[1];
    unsigned long long mx = 0ull;
    for (int64_t i = threadIdx.x; i < n; i += kSelNT) {
      const unsigned long long b = x[i];
      if (shift == 64 - kSelBits) mx = b > mx ? b : mx;
      const unsigned long long top = sh + bits < 64 ? b >> (sh + bits) : 0ull;
      const unsigned d = (unsigned)(b >> sh) & ((1u << bits) - 1u);
      if (top == p0) atomicAdd(&s_hist[0][d], 1u);
      if (top == p1) atomicAdd(&s_hist[1][d], 1u);
    }
    if (mx) atomicMax(&s_max, mx);
    __syncthreads();
    for (int h = 0; h < 2; ++h) {
      // the digit at whose bin the rank lies: thread t scans bins 2t, 2t + 1
      const unsigned c0 = s_hist[h][2 * threadIdx.x], c1 = s_hist[h][2 * threadIdx.x + 1];
      unsigned incl = c0 + c1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) s_part[warp] = incl;
      __syncthreads();
      unsigned before = 0;
      for (int k = 0; k < warp; ++k) before += s_part[k];
      const long long e = (long long)before + incl - c0 - c1, r = s_rank[h];
      const unsigned long long p = s_prefix[h];
      __syncthreads();
      if (r >= e && r < e + c0 + c1) {
        const bool second = r >= e + c0;
        s_rank[h] = r - e - (second ? (long long)c0 : 0ll);
        s_prefix[h] = (p << bits) | (unsigned long long)(2 * threadIdx.x + (second ? 1 : 0));
      }
      __syncthreads();
    }
  }
  if (threadIdx.x == 0) {
    out[3 * blockIdx.x] = __longlong_as_double((long long)s_max);
    out[3 * blockIdx.x + 1] = __longlong_as_double((long long)s_prefix[0]);
    out[3 * blockIdx.x + 2] = __longlong_as_double((long long)s_prefix[1]);
  }
}
static_assert(1 << kSelBits == 2 * kSelNT, "two bins a thread");

struct DevBuf {
  unsigned char *p = nullptr;
  ~DevBuf() {
    if (p) cudaFree(p);
  }
};

struct LockstepLaunch : StepLaunch {
  Twin w;
  cudaError_t operator()(const NetView &v, int64_t t_abs0, int steps, bool last, GridSync *gs, unsigned long long limit_ns,
                         int stall, cudaStream_t s) override {
    int dev = 0, sms = 1, occ = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k64_lockstep, kTwinNT, 0);
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(w.count, 0, (size_t)steps * sizeof(int), s)) != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(v.n <= (int64_t)sms * kTwinNT ? sms : sms * std::max(occ, 1)));
    cfg.blockDim = dim3(kTwinNT);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k64_lockstep, v, w, t_abs0, steps, last ? 1 : 0, gs, limit_ns, stall);
  }
};

}  // namespace

extern "C" int g4s_net_fp64_check(g4s_net *net, int32_t steps, double *dv_max, double *dv_p99, double *dv_median,
                                  int32_t *first_divergent, double *v64_out, double *u64_out) {
  if (!net) return set_error(G4S_ERR_INVALID, "null network");
  if (steps < 0) return set_error(G4S_ERR_INVALID, "g4s_net_fp64_check: negative step count");
  if (net_steps_done(net) != 0)
    return set_error(G4S_ERR_STATE, "g4s_net_fp64_check: the network must be at step 0 (after create or reset)");
  const NetView &v0 = net_view(net);
  const int64_t n = v0.n;
  cudaStream_t s = net_stream(net);
  // steps of a chunk: differences of up to kTwinBytes at a time (so that the selection reads
  // them from L2), the handle's own chunk, a few thousand steps
  constexpr int64_t kTwinBytes = (int64_t)64 << 20;
  int64_t chunk = net_chunk_steps(net, std::max<int64_t>(1, std::min({kTwinBytes / (n * 8), (int64_t)4096, (int64_t)steps})));
  size_t bytes, o_vu, o_acc, o_list, o_cnt, o_dv, o_out, o_words;
  auto place = [&](size_t b) {
    const size_t at = bytes;
    bytes = (bytes + b + 255) / 256 * 256;
    return at;
  };
  DevBuf buf;
  cudaError_t e;
  for (;; chunk /= 2) {  // (shorter chunks where the device has no room for the differences of these)
    bytes = 0;
    o_vu = place((size_t)n * sizeof(double2));
    o_acc = place((size_t)n * sizeof(Q128));
    o_list = place((size_t)n * sizeof(int));
    o_cnt = place((size_t)chunk * sizeof(int));
    o_dv = place((size_t)chunk * (size_t)n * sizeof(double));
    o_out = place((size_t)chunk * 3 * sizeof(double));
    o_words = place(2 * sizeof(int));
    if ((e = cudaMalloc((void **)&buf.p, bytes)) == cudaSuccess) break;
    (void)cudaGetLastError();
    buf.p = nullptr;
    if (chunk == 1) return cuda_error(e, "g4s_net_fp64_check: allocation");
  }
  LockstepLaunch run;
  run.w = Twin{reinterpret_cast<double2 *>(buf.p + o_vu), reinterpret_cast<Q128 *>(buf.p + o_acc),
               reinterpret_cast<int *>(buf.p + o_list),   reinterpret_cast<int *>(buf.p + o_cnt),
               reinterpret_cast<double *>(buf.p + o_dv),  reinterpret_cast<int *>(buf.p + o_words),
               reinterpret_cast<int *>(buf.p + o_words) + 1};
  double *out = reinterpret_cast<double *>(buf.p + o_out);
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)sms * 8));
  int words[2] = {INT32_MAX, 0};  // first step that differs, bad weight
  e = cudaMemcpyAsync(run.w.first, words, sizeof words, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return cuda_error(e, "g4s_net_fp64_check: init");
  k64_init<<<grid, 256, 0, s>>>(v0, run.w.vu, run.w.acc);
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_error(e, "g4s_net_fp64_check: init");
  // nearest-rank percentiles: the ceil(p n)-th smallest value
  const int64_t r99 = (int64_t)std::ceil(0.99 * (double)n) - 1, r50 = (int64_t)std::ceil(0.5 * (double)n) - 1;
  std::vector<double> h_out((size_t)chunk * 3);
  for (int32_t t = 0; t < steps;) {
    const int cs = (int)std::min<int64_t>(chunk, steps - t);
    const int rc = net_run_by(net, cs, t + cs == steps, run);
    if (rc) return rc;
    k64_select<<<(unsigned)cs, kSelNT, 0, s>>>(run.w.dv, n, r99, r50, out);
    if ((e = cudaGetLastError()) == cudaSuccess)
      e = cudaMemcpyAsync(h_out.data(), out, (size_t)cs * 3 * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(words, run.w.first, sizeof words, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_error(e, "g4s_net_fp64_check: step");
    if (words[1]) return set_error(G4S_ERR_INVALID, "g4s_net_fp64_check: a weight of magnitude >= 2^40 or not finite");
    for (int k = 0; k < cs; ++k, ++t) {
      if (dv_max) dv_max[t] = h_out[(size_t)k * 3];
      if (dv_p99) dv_p99[t] = h_out[(size_t)k * 3 + 1];
      if (dv_median) dv_median[t] = h_out[(size_t)k * 3 + 2];
    }
  }
  if (first_divergent) *first_divergent = words[0] == INT32_MAX ? -1 : words[0];
  if (v64_out || u64_out) {
    std::vector<double2> h((size_t)n);
    e = cudaMemcpyAsync(h.data(), run.w.vu, (size_t)n * sizeof(double2), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_error(e, "g4s_net_fp64_check: state");
    for (int64_t i = 0; i < n; ++i) {
      if (v64_out) v64_out[i] = h[(size_t)i].x;
      if (u64_out) u64_out[i] = h[(size_t)i].y;
    }
  }
  return G4S_OK;
}
