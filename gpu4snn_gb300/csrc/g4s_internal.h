// g4s_internal.h — declarations shared by the host library's translation units.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "g4s_types.h"

struct g4s_net;  // the handle of the C ABI
struct g4s_net_desc;

namespace g4s {

// Propagation schemes, numbered as the reference's `dynamic` (gpu4snn.cu:1083).
constexpr int kAlgAP = 0;
constexpr int kAlgN = 1;
constexpr int kAlgS = 2;
constexpr int kAlgAB = 3;
constexpr int kAlgSKL = 4;
constexpr int kAlgAuto = 5;

cudaError_t launch_init(const NetView &v, cudaStream_t s);
cudaError_t launch_conngen(const NetView &v, int self_loops, cudaStream_t s);
// nsteps steps of a scheme (kAlgSKL: the fallback of the team kernel) with the currents in
// global memory; synapses: those expected of a step; *launches: kernel launches made
cudaError_t launch_steps(const NetView &v, int64_t t_abs0, int nsteps, bool last_chunk, GridSync *gs,
                         unsigned long long limit_ns, int alg, double synapses, int stall, cudaStream_t s, int *launches);
cudaError_t launch_stats(const NetView &v, double *out, cudaStream_t s);
// fields of neurons [i0, i0 + cnt) as separate arrays: bits 0..7 of `fields` are v, u, I, a, b,
// c, d and the spike count; `out` is device-accessible, cnt values per field asked for
cudaError_t launch_state_pack(const NetView &v, int64_t i0, int cnt, unsigned fields, float *out, cudaStream_t s);
int persistent_blocks();

// SKL team kernel (g4s_team.cu).
constexpr int kMaxSortedNsyn = 16384;          // rows are sorted in shared memory
constexpr size_t kTeamSmemLimit = 200 * 1024;  // shared memory per CTA for currents + spikes
constexpr int64_t kPrezSlice = 12288;          // slices up to this size precompute the next drive
constexpr int64_t kVuSlice = 2048;             // ... keep v, u in shared memory for the whole launch
constexpr int64_t kAbcdSlice = 2048;           // ... keep a, b, c, d in shared memory (larger slices
                                               // keep them in global memory: the L1 left by a larger
                                               // shared-memory carve-out holds fewer table loads in flight)
constexpr int64_t kBatchMinSlice = 128;        // a network in a batch takes at most one CTA per this
                                               // many neurons
constexpr int64_t kBatchSlice = 8192;          // neurons per CTA of a network in a batch that fills the
                                               // GPU (256 networks, 3.2e9 synapses: 326 ms)
constexpr int kStateBlock = 65536;             // neurons of the state read back at a time
constexpr int kStateThreadBlocks = 3;          // ... in this many blocks or more, a thread per field
constexpr int kMaxTeam = 176;                  // CTAs of one team (eight source ranks a warp, 22 such warps)
// Spike records of a multi-CTA team: per rank and step parity kRecLines lines of 16
// tagged 64-bit words (count, then up to 16 kRecLines - 1 ids); readers fetch the second
// line of a rank only if it had enough spikes in the previous step (g4s_team.cu).
constexpr int kRecLines = 2;
constexpr int kRecWords = 16;

// Ranks of a team from which every warp polls source ranks of its own; in smaller teams, where
// that would leave most warps idle, every warp reads every rank's count and takes its share
// of the step's spikes.  Small steps (768 threads, segment runs) gain by it from 12 ranks on,
// as each warp waits for less (us a step: N=800 x 50 with 12 CTAs 2.88, with 7 and shares 3.57;
// N=5,000 x 1000 with 11 and shares 5.42, with 12 4.84).  Large steps, and those of the group
// mapping, are bound by the delivery, for which idle warps count: shares up to the sixteen
// ranks that fetch_spike's search takes (shares / own sources with 12 and with 16 CTAs of 1024
// threads: groups N=50,000 x 1000 18.7 / 28.7, 15.7 / 20.3, N=40,000 x 4000 35.6 / 62.5, 28.1 / 40.4;
// runs N=50,000 x 1000 19.8 / 28.9, 16.3 / 20.2, but N=5,000 x 1000 5.8 / 5.7, 5.6 / 5.1).
constexpr int kOwnSources = 12;
constexpr int kOwnSourcesLarge = 17;
__host__ __device__ constexpr bool own_sources(int team, bool small_steps) {
  return team >= (small_steps ? kOwnSources : kOwnSourcesLarge);
}

// Shared-memory layout of one team rank (byte offsets; the optional arrays are present
// when their flag is set).
struct TeamLayout {
  unsigned abcd, vu, a, b, own, z, pay, col, bytes;
  bool abcd_sm, vu_sm, prez, pay_sm, col_sm;
};
// (col: rows of the rank's column of the segment table, 0 if it stays in global memory; own:
// every warp polls source ranks of its own)
__host__ __device__ inline unsigned team_align16(size_t x) { return (unsigned)((x + 15) & ~(size_t)15); }
__host__ __device__ inline TeamLayout team_layout(int64_t rc, int team, int64_t col, bool own) {
  TeamLayout L{};
  L.abcd_sm = rc <= kAbcdSlice;
  L.vu_sm = rc <= kVuSlice;
  L.prez = rc <= kPrezSlice;
  L.pay_sm = own;
  size_t o = 0;
  L.abcd = (unsigned)o;
  if (L.abcd_sm) o += (size_t)rc * 16;
  L.vu = (unsigned)o;
  if (L.vu_sm) o = team_align16(o + (size_t)rc * 8);
  L.a = (unsigned)o;
  o = team_align16(o + (size_t)rc * 4);
  L.b = (unsigned)o;
  o = team_align16(o + (size_t)rc * 4);
  L.own = (unsigned)o;
  o = team_align16(o + (size_t)rc * 4);
  L.z = (unsigned)o;
  if (L.prez) o = team_align16(o + (size_t)rc * 4);
  L.pay = (unsigned)o;  // payloads of the record lines
  if (L.pay_sm) o = team_align16(o + (size_t)team * kRecLines * kRecWords * 4);
  L.col_sm = col > 0;
  L.col = (unsigned)o;
  o = team_align16(o + (size_t)col * 4);
  L.bytes = o < 0xFFFFFFFFull ? (unsigned)o : 0xFFFFFFFFu;
  return L;
}
// Rows sorted by target (unsigned, so unused slots last), equal targets by weight bits;
// generated = rows as the connectivity kernel writes them (distinct targets, unused slots
// (-1, 0.0f)), which a narrower key sorts into the same order.
cudaError_t launch_sort_rows(const NetView &v, bool generated, cudaStream_t s);
// *unsorted <- 1 if some row is not in launch_sort_rows' order, else 0
cudaError_t launch_first_bad(const int *idx, const NetView &v, unsigned long long *first, cudaStream_t s);
cudaError_t launch_rows_sorted(const NetView &v, int *unsorted, cudaStream_t s);
// A launch over many networks: clear (before it) and pack (after it) every network's
// per-launch words; network i's share of the pack is round_pack_bytes(steps_i) bytes at
// off[i]: status word, team error word, counts, raster offsets, stamps.
inline size_t round_pack_bytes(int steps) { return 8 + (((size_t)steps * 4 + 7) & ~(size_t)7) + (size_t)steps * 24; }
cudaError_t launch_round_clear(const TeamItem *items, int count, cudaStream_t s);
cudaError_t launch_round_gather(const TeamItem *items, const int64_t *off, int count, unsigned char *pack,
                                cudaStream_t s);
cudaError_t launch_chunk_gather(const NetView &v, const GridSync *gs, int steps, unsigned char *pack, cudaStream_t s);
cudaError_t launch_segoff(const NetView &v, int team, int64_t rc, uint16_t *seg, cudaStream_t s);
// out (3 words): the largest in-degree, the largest sum(|q| >> 16) + 1 over a neuron's
// inputs (with mag, n words of scratch; else 0), the largest (|q| >> 16) + 1 (without mag)
cudaError_t launch_inbound(const NetView &v, unsigned *cnt, unsigned long long *mag, unsigned long long *out,
                           cudaStream_t s);
// team_max_blocks also raises the kernel's shared-memory ceiling: call it once before the
// first launch_team (which may then be captured in a CUDA graph)
// Threads per CTA of the team kernel: 1024 (the default; the most reads in flight) or 768
// (80 registers a thread instead of 64: no spills, or 48 bytes in launches with one-CTA teams;
// faster when a step's work is small).
constexpr int kTeamNT = 1024;
constexpr int kTeamNTSmall = 768;
// pair: the tables are read from v.pair (packed words) instead of v.idx and v.w;
// mode: delivery mapping of the launch's multi-CTA teams (kDeliverRun or kDeliverGroup);
// solo: the launch has one-CTA teams; nt: kTeamNT or kTeamNTSmall threads per CTA
// slot_head: device word, 0 at launch (the queue's slots beyond the grid)
cudaError_t launch_team(const TeamItem *items, const int2 *slots, int nslots, int *slot_head, int grid,
                        size_t smem, unsigned long long limit_ns, int stall, cudaStream_t s, bool pair, int mode,
                        bool solo, int nt = kTeamNT);
// v.pair <- the rows of v.idx and v.w as packed words (after every change of the tables)
cudaError_t launch_pairs(const NetView &v, cudaStream_t s);
// Bits of a packed word's target field: what n needs, at least 16 (so that the decoding
// shifts stay within a word).
inline int pair_target_bits(int64_t n) {
  int b = 16;
  while (b < 31 && ((int64_t)1 << b) < n) ++b;
  return b;
}
cudaError_t team_max_blocks(size_t smem, int *out, int nt = kTeamNT);
// mean duration in ms of the last k simulated steps of a handle with a step time (0: none)
double net_recent_step_ms(const g4s_net *n, int64_t k);
// the team kernel's team-independent buffers of a handle (its packed rows and spike
// lists), made ready ahead of its first team run; nothing for tables the kernel cannot run
int net_prepare_rows(g4s_net *n);
// g4s_net_create with the handle's device memory from a stream-ordered pool (a server's)
int net_create_pooled(const g4s_net_desc *desc, cudaMemPool_t pool, g4s_net **out);
cudaError_t team_smem_ceiling();  // the part of team_max_blocks that launch_team needs
// shared memory of one rank of a team of `team` CTAs with `rc` neurons each (0: does not fit)
size_t team_smem(int64_t rc, int team, int64_t col = 0);

// A handle's arrays, stream and absolute step, for the library's other translation units
// (the on-device FP64 check, g4s_fp64check.cu).
const NetView &net_view(const g4s_net *n);
// `steps` further steps of the handle (at most net_chunk_steps' last answer) by a launch of the caller's:
// it does what the library's own step kernels do with the handle's arrays, and the handle's
// record takes the results.  `stall`: blocks too many for its grid barrier to wait for, so that
// it runs out.
struct StepLaunch {
  virtual cudaError_t operator()(const NetView &v, int64_t t_abs0, int steps, bool last, GridSync *gs,
                                 unsigned long long limit_ns, int stall, cudaStream_t s) = 0;
};
int net_run_by(g4s_net *n, int steps, bool last, StepLaunch &launch);
// steps that one such launch may take, of the `steps` asked for (by the raster buffer to be had)
int64_t net_chunk_steps(g4s_net *n, int64_t steps);
cudaStream_t net_stream(const g4s_net *n);
int64_t net_steps_done(const g4s_net *n);
// CTAs of the team the handle's last planned geometry uses (solo or batched), without
// planning anything (1 when no team geometry is planned)
int net_team_size(const g4s_net *n);

// Binary files (g4s_formats.cu): the raster, streamed by a writer thread, and the tables.
struct RasterFile;
int raster_open(const char *path, int64_t n, int64_t t0, RasterFile **out);
void raster_push(RasterFile *f, const int32_t *counts, int cs, const int32_t *ids, int64_t nids);
int raster_close(RasterFile *f);
int raster_write_all(const char *path, int64_t n, int64_t t0, const std::vector<int32_t> &counts,
                     const int32_t *ids, size_t nids);
struct TableHeader {
  int64_t n;
  int32_t nsyn, stride;
  uint64_t seed;
  int32_t conn_law, self_loops, exc_permille, flags;  // flags: 1 = rows sorted by target
  int32_t pad[2];
};
int tables_write(const char *path, const TableHeader &h, const int32_t *idx, const float *w);
int tables_read_header(const char *path, TableHeader *h);
int tables_read(const char *path, const TableHeader &h, int32_t *idx, float *w);

// Error reporting (thread-local message behind g4s_last_error()).
int set_error(int code, const std::string &msg);
int cuda_error(cudaError_t e, const char *what);

// Host generator of the reference's glibc-rand tables (gpu4snn.cu:873-898).
int conn_glibc_host(unsigned seed, int32_t n, int32_t nsyn, int32_t stride, int32_t *idx, float *w);

}  // namespace g4s
