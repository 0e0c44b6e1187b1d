// Pieces shared by the persistent tensor-core decode-attention kernels: the
// scratch handed to a launch, the record a producer publishes per tile, the
// merge of a segment's partial results, and the host-side scratch layout.
#pragma once

#include <limits.h>
#include <math.h>

#include <atomic>

#include "attention_common.cuh"

namespace jpt {

constexpr int kThreads = 128;
constexpr int kD = 128;
constexpr int kMaxRows = 16;
constexpr int kPieceCost = 1;  // overhead slots charged per segment, in tiles
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// Scratch handed to the kernel (all inside the caller's workspace).
struct MmaScratch {
  unsigned* counters;  // [B * Hkv] wrapping arrival counters, zero between launches
  int32_t* seqinfo;    // [B][4] (first, n, use_add, -) for additive masks
  unsigned* ticket;    // the next item of the work list; wraps to zero by the end of the launch
  float* part_o;       // [num_ctas][2][16][128] unnormalised partial outputs
  float* part_m;       // [num_ctas][2][16] reference maximum (log2 domain)
  float* part_l;       // [num_ctas][2][16] sum of exp2(x - reference)
  float* part_t;       // [num_ctas][2][16] true maximum (log2 domain)
  int num_ctas;
  int early;           // launched under the kernel before it (programmatic launch)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int sz = valid ? 16 : 0;  // src-size 0: the 16 bytes are zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(sz));
}
// L2 policy of the cache rows: read once per step, they leave first and do not push out what the launches share (their
// instructions, page tables, lengths, the weights of the layers around them).
__device__ __forceinline__ uint64_t evict_first_policy() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid, uint64_t policy) {
  const int sz = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;\n" ::"r"(dst), "l"(src), "r"(sz), "l"(policy));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}
__device__ __forceinline__ float fast_exp2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(x));
  return r;
}


// What the producer publishes about the tile it put into a stage.
struct TileMeta {
  int b, h;        // sequence, KV head
  int t, T;        // tile inside the segment (-1: no tile, the CTA's share is exhausted), tiles of the segment
  int n, first;    // valid tokens of the sequence and position of its first one
  int use_add;     // additive mask values must be applied
  int first_cta;   // CTA that holds tile 0 of the segment
  int parts;       // number of CTAs the segment is spread over
  int pad[3];
};

// Where a segment's partial results lie: the first in slot `first`, piece p > 0 in slot first + 1 + (p - 1) * stride.
struct PartSlots {
  int first, stride;
  __device__ __forceinline__ int of(int piece) const { return piece == 0 ? first : first + 1 + (piece - 1) * stride; }
};

// Valid range of a sequence for every mask mode (additive masks have been
// reduced to ranges by mask_ranges_kernel).
template <bool kL2 = false>
__device__ __forceinline__ SeqRange seq_range_x(const AttnArgs& a, const MmaScratch& x, int b, int* use_add) {
  *use_add = 0;
  if (a.mask_mode == JPT_MASK_ADD) {
    SeqRange r;
    if (kL2) {
      const int4 info = __ldcg(reinterpret_cast<const int4*>(x.seqinfo) + b);
      r.first = min(max(info.x, 0), a.S - 1);  // (scratch that no launch may have written yet)
      r.n = min(max(info.y, 0), a.S);
      return r;
    }
    r.first = x.seqinfo[4 * b];
    r.n = x.seqinfo[4 * b + 1];
    *use_add = x.seqinfo[4 * b + 2];
    return r;
  }
  return seq_range<kL2>(a, b);
}

// Combine the `parts` partials of one segment and write its R final rows.  Called by 128 threads
// (threadIdx.x 0..127): thread t owns head-dim index t of every row and the rows' statistics travel by
// warp shuffles, so there is no staging in shared memory and no barrier; `kStep` pieces are combined per
// step with all of their loads in flight at once (four of up to 8 rows: one L2 round trip for nearly
// every segment).
template <int kR, int kStep>
static __device__ __forceinline__ void merge_rows(const AttnArgs& a, const MmaScratch& x, PartSlots at, int parts, int64_t row_base) {
  const int tid = threadIdx.x, lane = tid & 31, R = a.R;
  // Lane r of every warp keeps row r's statistics (reference maximum, denominator relative to
  // it, true maximum) and hands the weights to the other lanes by shuffles.
  const bool mine = lane < R;
  float Mr = -INFINITY, Lr = 0.f, Tr = -INFINITY;
  float acc[kR];
#pragma unroll
  for (int r = 0; r < kR; ++r) acc[r] = 0.f;
  for (int pi = 0; pi < parts; pi += kStep) {
    float m[kStep], l[kStep], t[kStep], v[kStep][kR];
#pragma unroll
    for (int z = 0; z < kStep; ++z) {
      const bool there = pi + z < parts;
      const int64_t i0 = (int64_t)at.of(there ? pi + z : pi) * kMaxRows;
      m[z] = (mine && there) ? __ldcg(x.part_m + i0 + lane) : -INFINITY;
      l[z] = (mine && there) ? __ldcg(x.part_l + i0 + lane) : 0.f;
      t[z] = (mine && there) ? __ldcg(x.part_t + i0 + lane) : -INFINITY;
#pragma unroll
      for (int r = 0; r < kR; ++r) v[z][r] = (there && r < R) ? __ldcg(x.part_o + (i0 + r) * kD + tid) : 0.f;
    }
    float mn = Mr;
#pragma unroll
    for (int z = 0; z < kStep; ++z) {
      mn = fmaxf(mn, m[z]);
      Tr = fmaxf(Tr, t[z]);
    }
    const float s = Mr == -INFINITY ? 0.f : fast_exp2(Mr - mn);
    Lr *= s;
    Mr = mn;
#pragma unroll
    for (int r = 0; r < kR; ++r) acc[r] *= __shfl_sync(0xffffffffu, s, r);
#pragma unroll
    for (int z = 0; z < kStep; ++z) {
      const float w = m[z] == -INFINITY ? 0.f : fast_exp2(m[z] - mn);
      Lr = fmaf(w, l[z], Lr);
#pragma unroll
      for (int r = 0; r < kR; ++r) acc[r] = fmaf(__shfl_sync(0xffffffffu, w, r), v[z][r], acc[r]);
    }
  }
  // the denominator and the output relative to the true maximum, which is what gets reported
  const float c = Lr > 0.f ? fast_exp2(Mr - Tr) : 0.f;
  Lr *= c;
  Mr = Tr;
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const float L = __shfl_sync(0xffffffffu, Lr, r);
    const float o = acc[r] * __shfl_sync(0xffffffffu, c, r);
    if (r < R) store_o(a, (row_base + r) * kD + tid, L > 0.f ? o / L : 0.f);
  }
  if (tid < R) {
    if (a.m) a.m[row_base + tid] = Mr * kLn2;
    if (a.l) a.l[row_base + tid] = Lr;
  }
}

static __device__ void merge_segment(const AttnArgs& a, const MmaScratch& x, PartSlots at, int parts, int64_t row_base) {
  if (a.R <= 8) {
    merge_rows<8, 4>(a, x, at, parts, row_base);
  } else {
    merge_rows<kMaxRows, 2>(a, x, at, parts, row_base);
  }
}

// ------------------------------------------------------------------ the work list
// The (sequence, KV head) segments of a launch as a list of items, longest first: a whole segment, or one of `parts`
// equal runs of its tiles.  CTA i starts with item i and takes further ones as it finishes (one ticket counter), so
// long segments start first and the short ones fill up the end of the launch.  Against equal contiguous shares of one
// tile list (which cut nearly every CTA's first and last segment) far fewer segments are cut: every cut costs a
// partial result, an arrival and a merge.
// Sequences are sorted by their number of tiles ("bins"): a counting sort, since comparing all pairs took 3 us with the
// 12 warps of an SM at it.
constexpr int kPlanSeqs = 2 * kThreads;  // more sequences than this, or longer ones: equal shares
constexpr int kPlanBins = kThreads;      // tiles of a sequence: 1 .. kPlanBins - 2
struct __align__(16) WorkList {
  uint16_t prefix[kPlanBins];  // items in front of the bin's first one (0xffff: the bin is empty)
  uint8_t seq0[kPlanBins];     // the bin's first entry of `order`
  uint8_t parts[kPlanBins];
  uint8_t order[kPlanSeqs];    // sequences, bin by bin
};
struct __align__(16) PlanScratch {  // while planning only
  uint32_t count[2][kPlanBins];     // sequences of the bin: one byte per warp, [128 of the sequences]
  uint2 bin[kPlanBins];             // x: sort key, y: items << 16 | sequences
};

// Before the first plan_items of a launch, by all threads, with a barrier behind it.
static __device__ __forceinline__ void plan_clear(PlanScratch& ps) {
  ps.count[0][threadIdx.x] = 0u;
  ps.count[1][threadIdx.x] = 0u;
}
__device__ __forceinline__ int ceil_div_by(int t, float inv) { return (int)(((float)t - 0.5f) * inv) + 1; }  // t >= 1, both below 2^15

// All 128 threads; `tiles(b)` = tiles of sequence b, `T` takes those of this thread's sequences.  Returns the number of items of the
// list left in `wl`, or -1 when equal shares are expected to be faster (or the list is too long to sort).  `red`: 8 ints of shared
// memory.  The estimate is in tiles: a piece costs kPiece more, an end that is cut kCut more than that.  Among the longest pieces c
// (32 candidates from the mean load of a CTA up to whole segments) the cheapest is taken: with at most one item per CTA
// the longest piece, else the mean load plus one for the uneven end.  The caller's barrier publishes `wl`.
template <typename Tiles>
static __device__ __forceinline__ int plan_items(int B, int Hkv, int n, const Tiles& tiles, int (&T)[2], PlanScratch& ps,
                                                 int* red, WorkList& wl, float kPiece, float kCut) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (B > kPlanSeqs) return -1;
  const int groups = B > kThreads ? 2 : 1;
  int nth[2] = {0, 0};  // which of its warp's sequences in the bin
  T[0] = T[1] = 0;
  for (int z = 0; z < groups; ++z) {
    const int b = tid + kThreads * z;
    T[z] = b < B ? min(tiles(b), kPlanBins - 1) : 0;
    const unsigned same = __match_any_sync(0xffffffffu, T[z]);
    nth[z] = __popc(same & ((1u << lane) - 1u));
    if (nth[z] == 0) reinterpret_cast<uint8_t*>(&ps.count[z][T[z]])[warp] = (uint8_t)__popc(same);
  }
  if (tid < 8) red[tid] = 0;
  __syncthreads();
  auto in_bin = [&](int t) {
    unsigned v = __dp4a(ps.count[0][t], 0x01010101u, 0u);
    if (groups > 1) v = __dp4a(ps.count[1][t], 0x01010101u, v);
    return (int)v;
  };
  int W = 0, segs = 0, longest = 0;
#pragma unroll
  for (int z = 0; z < kPlanBins / 32; ++z) {
    const int t = lane + 32 * z, h = t > 0 ? in_bin(t) : 0;
    W += t * h;
    segs += h;
    if (h > 0) longest = t;
  }
  W = Hkv * __reduce_add_sync(0xffffffffu, W);
  segs = Hkv * __reduce_add_sync(0xffffffffu, segs);
  longest = __reduce_max_sync(0xffffffffu, longest);
  if (W == 0) return 0;
  if (longest == kPlanBins - 1) return -1;
  const float inv_n = 1.f / (float)n;
  int c;
  float cost;
  {
    const int c0 = min(longest, (W + n - 1) / n), step = (longest - c0) / 31 + 1;
    const int mine = min(longest, c0 + lane * step);
    const float rc = 1.f / (float)mine;
    int N = 0, cut = 0;
#pragma unroll 4
    for (int t = 1; t <= longest; ++t) {
      const int parts = ceil_div_by(t, rc), items = parts * in_bin(t);
      N += items;
      cut += parts > 1 ? items : 0;
    }
    N *= Hkv;
    cut *= Hkv;
    float e = (float)mine + kPiece + (cut ? kCut : 0.f);
    if (N > n) {
      e = fmaxf(e, ((float)W + kPiece * (float)N + kCut * (float)cut) * inv_n + 1.f);
      if (cut && N > 2 * n) e = 1.0e6f;  // partial results have two slots per CTA
    }
    const unsigned best = __reduce_min_sync(0xffffffffu, ((unsigned)(e * 16.f) << 5) | (unsigned)lane);
    c = min(longest, c0 + (int)(best & 31u) * step);
    cost = (float)(best >> 5) * (1.f / 16.f);
  }
  // thread t: bin t; longer pieces first, then the longer sequences
  const int h = tid > 0 ? in_bin(tid) : 0;
  const int parts = h > 0 ? ceil_div_by(tid, 1.f / (float)c) : 0, size = h > 0 ? (tid + parts - 1) / parts : 0;
  const uint32_t key = (uint32_t)(size << 8 | tid);
  ps.bin[tid] = make_uint2(key, (uint32_t)(h * parts) << 16 | (uint32_t)h);
  __syncthreads();
  uint32_t before = 0u;  // sums of both halves: items < 2^16 (at most two a CTA, or one a sequence), sequences <= 256
#pragma unroll 4
  for (int t = 1; t <= longest; ++t) {
    const uint2 o = ps.bin[t];
    before += o.x > key ? o.y : 0u;
  }
  const int lo = (int)(before >> 16) * Hkv, hi = lo + h * parts * Hkv;
  if (h > 0) {
    // lengths of the items that share a CTA when the n longest are one to each: n - 1 and n, 2 n, 3 n
    if (lo <= n - 1 && n - 1 < hi) red[0] = size;
#pragma unroll
    for (int m = 1; m < 4; ++m)
      if (lo <= m * n && m * n < hi) red[m] = size;
    atomicMax(&red[4], hi);
  }
  wl.prefix[tid] = (uint16_t)(h > 0 ? lo : 0xffff);
  wl.seq0[tid] = (uint8_t)(before & 0xffu);  // (256 only behind the last sequence)
  wl.parts[tid] = (uint8_t)parts;
  __syncthreads();
  for (int z = 0; z < groups; ++z) {
    const int b = tid + kThreads * z;
    if (b < B && T[z] > 0) {
      // in the order of the sequences: those of the first group, then of the warps before, then of this warp
      int at = wl.seq0[T[z]] + nth[z] + (int)__dp4a(ps.count[z][T[z]] & ((1u << (8 * warp)) - 1u), 0x01010101u, 0u);
      if (z > 0) at += (int)__dp4a(ps.count[0][T[z]], 0x01010101u, 0u);
      wl.order[at] = (uint8_t)b;
    }
  }
  // n + 1 items of about one length take two rounds, whatever the mean says
  cost = fmaxf(cost, red[1] > 0 ? (float)(red[0] + red[1]) + 2.f * kPiece : 0.f);
  cost = fmaxf(cost, fmaxf(red[2] > 0 ? 3.f * ((float)red[2] + kPiece) : 0.f, red[3] > 0 ? 4.f * ((float)red[3] + kPiece) : 0.f));
  const float shares = ((float)W + kPiece * (float)segs) * inv_n + kPiece + 2.f * kCut;
  return cost <= shares ? red[4] : -1;
}

// Item k of the list, by a whole warp: sequence, head and part.
struct WorkItem {
  int b, h, part, parts;
};
static __device__ __forceinline__ WorkItem find_item(const WorkList& wl, int Hkv, int k) {
  const int lane = threadIdx.x & 31;
  const uint2 p = *reinterpret_cast<const uint2*>(&wl.prefix[4 * lane]);
  const int v[4] = {(int)(p.x & 0xffffu), (int)(p.x >> 16), (int)(p.y & 0xffffu), (int)(p.y >> 16)};
  int best = -1;  // the last bin that starts at or in front of item k
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (v[e] <= k) best = max(best, v[e] << 8 | (4 * lane + e));
  best = __reduce_max_sync(0xffffffffu, best);
  const int t = best & 255, j = k - (best >> 8);
  WorkItem it;
  it.parts = wl.parts[t];
  const int per_seq = it.parts * Hkv, s = j / per_seq, r = j - s * per_seq;
  it.b = wl.order[wl.seq0[t] + s];
  it.h = r / it.parts;
  it.part = r - it.h * it.parts;
  return it;
}

// Per-device facts are kept per device ordinal: a process may drive several GPUs.
constexpr int kMaxDevices = 64;

inline int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) dev = 0;
  return dev;
}

inline int sm_count() {
  static std::atomic<int> n[kMaxDevices];
  const int dev = current_device();
  int v = n[dev].load(std::memory_order_relaxed);
  if (v == 0) {
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    n[dev].store(v, std::memory_order_relaxed);
  }
  return v;
}

// Runs `configure` (which returns a cudaError_t) once per device, with that
// device current; cudaFuncSetAttribute applies to the current device only.
// Returns 0 or the positive CUDA error of a failed configuration (not cached,
// so the next call tries again).
template <typename F>
inline int configure_once_per_device(std::atomic<bool> (&done)[kMaxDevices], const char* what, F configure) {
  const int dev = current_device();
  if (done[dev].load(std::memory_order_acquire)) return 0;
  const cudaError_t e = configure();
  if (e != cudaSuccess) return fail((int)e, "%s: configuring the kernel on device %d: %s", what, dev, cudaGetErrorString(e));
  done[dev].store(true, std::memory_order_release);
  return 0;
}

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct ScratchLayout {
  size_t counters, seqinfo, part_m, part_l, part_t, part_o, total;
  int num_ctas;
};

// Exchange area of one rank for the per-token amax of a decode step: 64 bytes of
// state {launches done, CTAs done, gave up}, then slots[parity][writer rank][2 B]
// of 64-bit words (the buffers of a jpt_peer_exchange).
constexpr size_t kExchangeStateBytes = 64;
inline size_t exchange_bytes(int B, int world) {
  return kExchangeStateBytes + (size_t)2 * world * 2 * B * sizeof(unsigned long long);
}

// Layout of the scratch of a persistent launch of `num_ctas` CTAs.
inline ScratchLayout scratch_layout(const jpt_attn_params& p, int num_ctas) {
  ScratchLayout s;
  s.num_ctas = num_ctas;
  size_t off = 0;
  s.counters = off;  // fixed-size header shared by every shape that uses the workspace
  off = kWorkspaceCounterBytes;
  s.seqinfo = off;
  off = align_up(off + sizeof(int32_t) * 4 * p.B, 256);
  s.part_m = off;
  off = align_up(off + sizeof(float) * s.num_ctas * 2 * kMaxRows, 256);
  s.part_l = off;
  off = align_up(off + sizeof(float) * s.num_ctas * 2 * kMaxRows, 256);
  s.part_t = off;
  off = align_up(off + sizeof(float) * s.num_ctas * 2 * kMaxRows, 256);
  s.part_o = off;
  off = align_up(off + sizeof(float) * s.num_ctas * 2 * kMaxRows * kD, 256);
  s.total = off;
  return s;
}

// Additive masks -> valid ranges in x.seqinfo (one CTA per sequence).
int launch_mask_ranges(const AttnArgs& a, const MmaScratch& x, cudaStream_t st);

}  // namespace jpt
