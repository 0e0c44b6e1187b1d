// Weight-only int8 linear layer for decode batches: y[m, n] = (sum_k x[m, k] W[n, k]) * scale[n]
// with x bf16 [M <= 128, K], W int8 [N, K] (one scale per output channel), y bf16 [M, N]
// (WeightOnlyPerChannelQuantizedLinear.forward, symmetric weights, no activation quantisation:
// jetstream_pt/layers.py:141-166).
//
// A decode step streams every weight byte once, so the kernel is bound by the HBM read of W.  The
// int8 weights go from HBM to shared memory by the copy engine and from there straight into the
// tensor core: the contraction runs as tcgen05 integer MMAs with the weights as the M = 128 operand
// and the activations as the N operand.  The bf16 activations become 8-bit without losing their
// precision by the same two-level split the attention kernel uses for its queries: a row x of the
// batch is s (h + l / 254) with s = amax|x| / 127 and h, l signed bytes (error 2^-16 of the row's
// amax), so the N operand holds 2 M rows (all h rows, then all l rows) and
//   y[m, n] = scale[n] * s_m * (S_h[n, m] + S_l[n, m] / 254)
// with exact int32 sums S_h, S_l in tensor memory.  Nothing is converted in registers.
//
// Launches: (1) split of the activations into levels (one CTA per row of x), (2) the GEMM: pairs of CTAs
// (cta_group::2) with up to 256 output channels per CTA; the CTAs of a pair's K splits form a thread-block
// cluster.  One thread requests the tiles of a ring of 128-byte-swizzled weight and activation tiles, one
// warp of the pair's first CTA issues the MMAs, two per K step of 32 bytes, one for each half of the channels, and
// frees the stages through tcgen05.commit.  Epilogue: eight warps read the accumulators out of tensor memory; without a
// split they finish the result there.  With one, the rows of the batch are dealt out to the splits in groups of eight, every
// CTA stores its partial sums of a group into the shared memory of the group's owner (the ring is
// free by then), and the owner adds the partials in the order of the splits, rounds to bf16,
// multiplies by the channel's scale and rounds again, as the reference's two bf16 operations do.
// No partial result goes through global memory.  Every wait on data is bounded; a CTA that gives up
// raises the status word, still meets its cluster at the cluster barriers, and returns.
//
// Also here, because they write the same level matrix: RMSNorm and the feed-forward gate (SiLU-mul) as
// kernels that can leave the level split of their result behind, so that the layers after them start
// at their GEMM; and the row-parallel form of the layer over the GPUs of one box, in which the owner
// of a group of rows adds the partial sums of all ranks (fetched over NVLink) before it rounds.
#include <cuda.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>

#include "common.cuh"

namespace jpt {
namespace {

constexpr int kTileN = 256;      // output channels per CTA at most: two accumulators of 128 TMEM lanes
constexpr int kTileK = 128;      // int8 elements per stage and row: one 128-byte swizzle atom
constexpr int kStages = 3;
constexpr int kMaxM = 128;       // rows of x: the N operand holds 2 * M rows (<= 256)
constexpr int kTmemColsL = 512;  // two accumulators [128 lanes x 2 M columns]
constexpr int kThreadsL = 256;
constexpr long long kWaitCyclesL = 1000000000ll;

struct LinearMaps {
  CUtensorMap w, x;
};

// Row-parallel layer over the GPUs of one box (the input features are sharded: every rank holds x[:, K_r] and
// W[:, K_r], the result is the sum over the ranks).  buffers[r] is rank r's receive buffer (own or an IPC
// mapping): a status word and the launch counter, launch numbers [2 (launch parity)][8 (source rank)][1024 (tile)]
// [8 (K split)] u32, then the rank's OWN fp32 partial sums [2][128][N].  A rank writes its sums into its own buffer,
// tells the others with the launch number (one small peer store per CTA and rank, behind a system-scope fence) and
// reads theirs with 16-byte peer loads, twelve of a thread in flight at a time: loads cross NVLink at about
// twice the rate of narrow peer stores.  world = 1: a layer of one GPU.
struct TpArgs {
  int world, rank;
  // number of this launch (the same on every rank): counted on the device by the level kernel in front of the GEMM,
  // so that a captured graph can be replayed
  unsigned* launch_counter;
  long long wait_cycles;
  char* buffers[8];
  int* status;  // in the rank's own buffer: raised when a wait for a peer ran out
};
constexpr int kTpMaxTiles = 1024;
constexpr size_t kTpFlagOffset = 256;
constexpr size_t kTpFlagBytes = (size_t)2 * 8 * kTpMaxTiles * 8 * sizeof(unsigned);
constexpr size_t kTpDataOffset = kTpFlagOffset + kTpFlagBytes;
__device__ __forceinline__ void st_sys_u32(unsigned* p, unsigned v) {
  asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_sys_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// (no memory clobber: the loads of a batch must be free to go out together; the flag's wait, fence and barrier
// stand before them)
__device__ __forceinline__ float4 ld_sys_f32x4(const float* p) {
  float4 v;
  asm volatile("ld.relaxed.sys.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for the phase with the given parity; false when it gave up.
__device__ __noinline__ bool mbar_wait_l(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 16; ++i) {
      if (mbar_try(bar, parity)) return true;
    }
    if (clock64() - t0 > kWaitCyclesL) return false;
  }
}
__device__ __forceinline__ uint64_t desc_k_major_128b(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);  // start address
  d |= (uint64_t)(1024 >> 4) << 16;       // leading byte offset (one swizzle atom)
  d |= (uint64_t)(1024 >> 4) << 32;       // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                 // descriptor version of sm_100
  d |= (uint64_t)2 << 61;                 // SWIZZLE_128B
  return d;
}
// The box: a number of 128-byte steps of K from step `z` on, each a swizzled tile of rows from `y` on.  (A CTA of a pair: the bytes
// land in this CTA, the barrier `bar`, a shared::cluster address, may be the other one's.)
// `policy`: how long its lines stay in L2.  Weights of more than half of L2 leave first: even a program that calls one layer over and over
// finds little of them there, and the activation levels that all CTAs read stay (hint on and off in turn: block 8192 / 28672 with 96
// rows 169.2 -> 164.8 us, 5120 / 13824 with 1 row 58.3 -> 55.8).  Smaller ones keep the usual policy.
__device__ __forceinline__ uint64_t l2_policy(bool once) {
  uint64_t first, normal;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(first));
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(normal));
  return once ? first : normal;
}
template <bool kPair>
__device__ __forceinline__ void tma_load_steps(uint32_t dst, const CUtensorMap* map, int y, int z, uint32_t bar, uint64_t policy) {
  if constexpr (kPair)
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(y), "r"(z), "r"(bar), "l"(policy)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(y), "r"(z), "r"(bar), "l"(policy)
        : "memory");
}
// The same box into L2 only.
__device__ __forceinline__ void tma_prefetch_steps(const CUtensorMap* map, int y, int z, uint64_t policy) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile.L2::cache_hint [%0, {%1, %2, %3}], %4;" ::"l"(reinterpret_cast<uint64_t>(map)),
               "r"(0), "r"(y), "r"(z), "l"(policy)
               : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// Thread-block cluster: barrier over all its threads (with release / acquire of shared-memory stores),
// the address of a shared-memory location in the CTA of another rank, a store there.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t remote_smem(uint32_t local_addr, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  // (no memory clobber: the cluster barriers order these stores, and the loads around them must stay free to move)
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v));
}

__device__ __forceinline__ bool elect_sync() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(r));
  return r != 0;
}
__device__ __forceinline__ void tmem_ld_16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                 "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(addr));
}
__device__ __forceinline__ void tmem_ld_8(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(addr));
}

// ---------------------------------------------------------------- (1) activation levels
// x [M, K] bf16 -> levels [2 Mp, K] int8 (rows 0 .. M-1: h, rows Mp .. Mp+M-1: l, the others zero)
// and xs[m] = s_m / 254.  More than 128 rows: one such matrix per block of Mp rows, one after the other.
__global__ void __launch_bounds__(256) x_levels_kernel(const __nv_bfloat16* x, int8_t* lev, float* xs, int* status, int M,
                                                       int Mp, int K, int clear_status, unsigned* launch_counter) {
  __shared__ float red[33];
  const int m = blockIdx.x, tid = threadIdx.x;  // one CTA per row of the padded batch
  // In this order: a GEMM that starts under this kernel takes its first weight tiles at once (GemmArgs::own_levels), and what wrote
  // the weights is complete then.  (Triggered before the wait, the GEMM also took its SMs earlier than it could use them: 8192 x 10240
  // with 84 rows 30.4 us, 27.4 in this order.)
  grid_dependency_wait();
  grid_dependency_trigger();
  if (m == 0 && tid == 0 && clear_status) *status = 0;
  if (m == 0 && tid == 0 && launch_counter) *launch_counter += 1u;  // (one thread, launches in stream order)
  uint2* hrow = reinterpret_cast<uint2*>(lev + (int64_t)(m + m / Mp * Mp) * K);
  uint2* lrow = reinterpret_cast<uint2*>(lev + (int64_t)(m + m / Mp * Mp + Mp) * K);
  const int nvec = K / 8;  // eight elements per step: 16 bytes in, 8 + 8 bytes out
  if (m >= M) {  // padding rows of the level matrix
    for (int v = tid; v < nvec; v += 256) hrow[v] = lrow[v] = make_uint2(0u, 0u);
    return;
  }
  const uint4* row = reinterpret_cast<const uint4*>(x + (int64_t)m * K);
  constexpr int kHeld = 8;  // steps of a thread kept in registers between the two passes (rows of up to 16384 elements)
  uint4 held[kHeld];
  __nv_bfloat162 mx = __float2bfloat162_rn(0.f);
  auto fold = [&](const uint4& r) {
    const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
    for (int j = 0; j < 4; ++j) mx = __hmax2(mx, __habs2(h2[j]));
  };
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    const int v = tid + 256 * i;
    held[i] = v < nvec ? __ldg(row + v) : make_uint4(0u, 0u, 0u, 0u);
  }
#pragma unroll
  for (int i = 0; i < kHeld; ++i) fold(held[i]);
  for (int v = tid + 256 * kHeld; v < nvec; v += 256) fold(__ldg(row + v));
  const float amax = block_max(fmaxf(__low2float(mx), __high2float(mx)), red);
  const float inv = amax > 0.f ? 127.f / amax : 0.f;
  auto split_levels = [&](const uint4& r, int v) {
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&r);
    uint32_t hb[2] = {0u, 0u}, lb[2] = {0u, 0u};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float t = __bfloat162float(e[j]) * inv;
      const float h = rintf(t);
      const float l = rintf((t - h) * 254.f);
      hb[j >> 2] |= ((uint32_t)(int)h & 0xffu) << (8 * (j & 3));
      lb[j >> 2] |= ((uint32_t)(int)l & 0xffu) << (8 * (j & 3));
    }
    hrow[v] = make_uint2(hb[0], hb[1]);
    lrow[v] = make_uint2(lb[0], lb[1]);
  };
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    const int v = tid + 256 * i;
    if (v < nvec) split_levels(held[i], v);
  }
  for (int v = tid + 256 * kHeld; v < nvec; v += 256) split_levels(__ldg(row + v), v);
  if (tid == 0) xs[m] = amax * (1.f / 127.f) * (1.f / 254.f);
}

// ---------------------------------------------------------------- producers of the activations that split on the way
// Eight bf16 values of a row -> their two level bytes each, stored at step v of the row's h and l rows.
__device__ __forceinline__ void split_levels8(const __nv_bfloat16 (&e)[8], float inv, uint2* hrow, uint2* lrow, int v) {
  uint32_t hb[2] = {0u, 0u}, lb[2] = {0u, 0u};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float t = __bfloat162float(e[j]) * inv;
    const float h = rintf(t);
    const float l = rintf((t - h) * 254.f);
    hb[j >> 2] |= ((uint32_t)(int)h & 0xffu) << (8 * (j & 3));
    lb[j >> 2] |= ((uint32_t)(int)l & 0xffu) << (8 * (j & 3));
  }
  hrow[v] = make_uint2(hb[0], hb[1]);
  lrow[v] = make_uint2(lb[0], lb[1]);
}
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) v += __shfl_xor_sync(0xffffffffu, v, sh);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float x = lane < (int)((blockDim.x + 31) >> 5) ? red[lane] : 0.f;
#pragma unroll
    for (int sh = 16; sh > 0; sh >>= 1) x += __shfl_xor_sync(0xffffffffu, x, sh);
    if (lane == 0) red[32] = x;
  }
  __syncthreads();
  return red[32];
}

constexpr int kRowThreads = 1024;  // threads of a CTA of the element-wise producers
// The CTAs of a cluster (gridDim.x of them, rank blockIdx.x) share a row: a value of every CTA combined in the
// order of the ranks.  Every CTA stores its value into slot `rank` of every CTA's `slots`; one cluster barrier later
// all slots are there.  (`slots` must not be reused for another reduction: a fast CTA could overwrite a slot
// that a slow one has not read yet.)
template <typename Op>
__device__ __forceinline__ float cluster_combine(float v, float* slots, Op op) {
  const int csize = (int)gridDim.x, rank = (int)blockIdx.x;
  if (csize == 1) return v;
  if ((int)threadIdx.x < csize) st_cluster_f32(remote_smem(smem_addr(&slots[rank]), (int)threadIdx.x), v);
  cluster_sync();
  float r = slots[0];
  for (int c = 1; c < csize; ++c) r = op(r, slots[c]);
  return r;
}

// A row of results, eight at a time from `compute(step, out)`: written to `dst`, and with `levels` split into the
// row's level bytes once the row's amax is known.  The first steps of a thread stay in registers between the two
// passes (1024 threads x 4 steps x 8: rows of up to 32768 elements); longer rows compute their tail twice.
template <typename Compute>
__device__ __forceinline__ void write_row_and_levels(Compute& compute, uint4* dst, int v_lo, int nvec, bool levels, uint2* hrow,
                                                     uint2* lrow, float* xs, int m, float* red, float* slots) {
  constexpr int kHeldOut = 4;
  const int tid = threadIdx.x + v_lo;  // (this CTA's steps are v_lo .. nvec - 1)
  uint4 held[kHeldOut];
  float amax = 0.f;
  auto fold = [&](const __nv_bfloat16 (&o)[8]) {
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(__bfloat162float(o[j])));
  };
#pragma unroll
  for (int i = 0; i < kHeldOut; ++i) {
    const int v = tid + kRowThreads * i;
    if (v < nvec) {
      __nv_bfloat16 o[8];
      compute(v, o);
      fold(o);
      held[i] = *reinterpret_cast<const uint4*>(o);
      dst[v] = held[i];
    }
  }
  for (int v = tid + kRowThreads * kHeldOut; v < nvec; v += kRowThreads) {
    __nv_bfloat16 o[8];
    compute(v, o);
    fold(o);
    dst[v] = *reinterpret_cast<const uint4*>(o);
  }
  if (!levels) return;
  amax = cluster_combine(block_max(amax, red), slots, [](float p, float q) { return fmaxf(p, q); });
  const float inv = amax > 0.f ? 127.f / amax : 0.f;
#pragma unroll
  for (int i = 0; i < kHeldOut; ++i) {
    const int v = tid + kRowThreads * i;
    if (v < nvec) split_levels8(*reinterpret_cast<const __nv_bfloat16(*)[8]>(&held[i]), inv, hrow, lrow, v);
  }
  for (int v = tid + kRowThreads * kHeldOut; v < nvec; v += kRowThreads) {
    __nv_bfloat16 o[8];
    compute(v, o);
    split_levels8(o, inv, hrow, lrow, v);
  }
  if (threadIdx.x == 0 && blockIdx.x == 0) xs[m] = amax * (1.f / 127.f) * (1.f / 254.f);
}

// RMSNorm (jetstream_pt/layers.py:337-350 with a bf16 weight): n = bf16(x * rsqrt(mean(x^2) + eps)) in fp32,
// y = bf16(n * weight).  With `lev` the row's levels are written too (the rows M .. Mp-1 of the level matrix as zeros),
// so that the linear layers that read y start at their GEMM.  One CTA per row.
__global__ void __launch_bounds__(kRowThreads) rmsnorm_levels_kernel(const __nv_bfloat16* x, const __nv_bfloat16* weight, float eps,
                                                             __nv_bfloat16* y, int8_t* lev, float* xs, int* status, int M, int Mp,
                                                             int K) {
  __shared__ float red[33], slots_ss[8], slots_amax[8];
  // row m = blockIdx.y; the CTAs of the row's cluster (blockIdx.x) take equal parts of its steps of eight elements
  const int m = blockIdx.y, tid = threadIdx.x, per = K / 8 / (int)gridDim.x;
  const int v_lo = (int)blockIdx.x * per, nvec = v_lo + per;
  grid_dependency_wait();
  grid_dependency_trigger();
  if (m == 0 && blockIdx.x == 0 && tid == 0 && status) *status = 0;
  uint2* hrow = lev ? reinterpret_cast<uint2*>(lev + (int64_t)m * K) : nullptr;
  uint2* lrow = lev ? reinterpret_cast<uint2*>(lev + (int64_t)(Mp + m) * K) : nullptr;
  if (m >= M) {  // (a padding row: the whole cluster is here, nobody waits for it)
    for (int v = v_lo + tid; v < nvec; v += kRowThreads) hrow[v] = lrow[v] = make_uint2(0u, 0u);
    return;
  }
  const uint4* row = reinterpret_cast<const uint4*>(x + (int64_t)m * K);
  const uint4* wrow = reinterpret_cast<const uint4*>(weight);
  float ss = 0.f;
  for (int v = v_lo + tid; v < nvec; v += kRowThreads) {
    const uint4 r = __ldg(row + v);
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&r);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float f = __bfloat162float(e[j]);
      ss = fmaf(f, f, ss);
    }
  }
  ss = cluster_combine(block_sum(ss, red), slots_ss, [](float p, float q) { return p + q; });
  const float rs = 1.f / sqrtf(ss / (float)K + eps);
  auto normed = [&](int v, __nv_bfloat16 (&o)[8]) {
    const uint4 r = __ldg(row + v), wv = __ldg(wrow + v);
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&r);
    const __nv_bfloat16* we = reinterpret_cast<const __nv_bfloat16*>(&wv);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float n = __bfloat162float(__float2bfloat16_rn(__bfloat162float(e[j]) * rs));
      o[j] = __float2bfloat16_rn(n * __bfloat162float(we[j]));
    }
  };
  write_row_and_levels(normed, reinterpret_cast<uint4*>(y + (int64_t)m * K), v_lo, nvec, lev != nullptr, hrow, lrow, xs, m, red,
                       slots_amax);
  if (gridDim.x > 1) cluster_sync();  // (no CTA leaves while a peer may still store into its slots)
}

// RMSNorm without levels for many rows (a prompt): one warp per row, the row held in its registers (K = 256 kVec elements),
// so that it is read once and nothing waits at a barrier.  A CTA of 1024 threads per row took 18.6 us for [1024, 4096] (16.8 MB).
template <int kVec>
__global__ void __launch_bounds__(128) rmsnorm_rows_kernel(const __nv_bfloat16* x, const __nv_bfloat16* weight, float eps,
                                                           __nv_bfloat16* y, int M, int K) {
  const int m = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  grid_dependency_wait();
  grid_dependency_trigger();
  if (m >= M) return;
  const uint4* row = reinterpret_cast<const uint4*>(x + (int64_t)m * K);
  const uint4* wrow = reinterpret_cast<const uint4*>(weight);
  uint4* out = reinterpret_cast<uint4*>(y + (int64_t)m * K);
  const int nvec = K / 8;
  uint4 held[kVec];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < kVec; ++i) held[i] = lane + 32 * i < nvec ? __ldg(row + lane + 32 * i) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&held[i]);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float f = __bfloat162float(e[j]);
      ss = fmaf(f, f, ss);
    }
  }
  const float rs = 1.f / sqrtf(warp_sum(ss) / (float)K + eps);
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    if (lane + 32 * i < nvec) {
      const uint4 wv = __ldg(wrow + lane + 32 * i);
      const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&held[i]);
      const __nv_bfloat16* we = reinterpret_cast<const __nv_bfloat16*>(&wv);
      uint4 o;
      __nv_bfloat16* oe = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float n = __bfloat162float(__float2bfloat16_rn(__bfloat162float(e[j]) * rs));
        oe[j] = __float2bfloat16_rn(n * __bfloat162float(we[j]));
      }
      out[lane + 32 * i] = o;
    }
  }
}

// One value of the gate: bf16(bf16(silu(a)) * b).  (Fast exponential and division: the quotient is rounded to bf16, and the
// exact forms are subroutines.)
__device__ __forceinline__ __nv_bfloat16 gate_value(__nv_bfloat16 a, __nv_bfloat16 b) {
  const float f = __bfloat162float(a);
  const float s = __bfloat162float(__float2bfloat16_rn(__fdividef(f, 1.f + __expf(-f))));
  return __float2bfloat16_rn(s * __bfloat162float(b));
}

// The feed-forward block's gate (third_party/llama/model_exportable.py:84-86): h = bf16(bf16(silu(a)) * b), and with
// `lev` the levels of h for the down projection.
__global__ void __launch_bounds__(kRowThreads) silu_mul_levels_kernel(const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* h,
                                                              int8_t* lev, float* xs, int* status, int M, int Mp, int K) {
  __shared__ float red[33], slots_amax[8];
  const int m = blockIdx.y, tid = threadIdx.x, per = K / 8 / (int)gridDim.x;
  const int v_lo = (int)blockIdx.x * per, nvec = v_lo + per;
  grid_dependency_wait();
  grid_dependency_trigger();
  if (m == 0 && blockIdx.x == 0 && tid == 0 && status) *status = 0;
  uint2* hrow = lev ? reinterpret_cast<uint2*>(lev + (int64_t)m * K) : nullptr;
  uint2* lrow = lev ? reinterpret_cast<uint2*>(lev + (int64_t)(Mp + m) * K) : nullptr;
  if (m >= M) {
    for (int v = v_lo + tid; v < nvec; v += kRowThreads) hrow[v] = lrow[v] = make_uint2(0u, 0u);
    return;
  }
  const uint4* arow = reinterpret_cast<const uint4*>(a + (int64_t)m * K);
  const uint4* brow = reinterpret_cast<const uint4*>(b + (int64_t)m * K);
  auto gated = [&](int v, __nv_bfloat16 (&o)[8]) {
    const uint4 ra = __ldg(arow + v), rb = __ldg(brow + v);
    const __nv_bfloat16* ea = reinterpret_cast<const __nv_bfloat16*>(&ra);
    const __nv_bfloat16* eb = reinterpret_cast<const __nv_bfloat16*>(&rb);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o[j] = gate_value(ea[j], eb[j]);
    }
  };
  write_row_and_levels(gated, reinterpret_cast<uint4*>(h + (int64_t)m * K), v_lo, nvec, lev != nullptr, hrow, lrow, xs, m, red,
                       slots_amax);
  if (gridDim.x > 1) cluster_sync();  // (no CTA leaves while a peer may still store into its slots)
}

// ---------------------------------------------------------------- (2) the GEMM
// Two CTAs of a TPC work as a pair (cta_group::2): each holds the weights of its own channels, the activation tile is shared
// between them (the even CTA loads the h rows, the odd one the l rows, and the tensor cores of both read both halves).  What
// bounds the K loop besides the HBM read is the L2: at 96 rows a CTA of its own reads 24 KB of activations per 32 KB of
// weights, a pair half of that.
// grid (tiles, splits), clusters of (2, splits): blockIdx.x is the channel tile, blockIdx.y the K split.  A tile is as wide as
// it takes to give every SM one (plan_gemm): the tensor core works on 128 rows whatever the tile's width; the rows behind
// the tile's, whatever lies there, only feed accumulator lanes that nobody reads.  (Fixed tiles of 256 channels left 36 of
// 148 SMs idle at 28672 channels.)  A stage holds `kb` steps of 128 bytes of K: the hand-over of a stage between the copy
// engine, the issuing warp and back costs 0.44 us whatever it holds (64 steps of 32 to 104 channels took 34 us).
struct GemmArgs {
  const float* xs;
  const __nv_bfloat16* scale;
  __nv_bfloat16* y;
  int* status;
  int M, Mp, N, k_steps;  // k_steps: stages' worth of K (the last one may reach beyond K, where the copy engine fills zeros)
  int tile;               // channels of a CTA
  int kb, stages, stage_bytes, tail;  // tail: where the ring (and the landing area that takes its place) ends
  int weights_once;       // the weights are more than L2 would keep until the next call: they leave it first
  int own_levels;         // the launch in front is this call's level kernel, which waits before it lets this one start
};
constexpr int kMaxStages = 12;
struct GemmTail {  // behind the ring
  uint64_t full[kMaxStages], empty[kMaxStages], done;
  alignas(16) float xs[kMaxM];  // s_m / 254 of the rows of x (read four at a time)
  uint32_t tmem_base;
};
constexpr int kRingBytes = 208 * 1024;
constexpr int kTailBytes = 16 * 1024;  // (the tail, and what the 128 rows of the ring's last operand reach beyond it)
static_assert(sizeof(GemmTail) <= kTailBytes && kRingBytes + kTailBytes <= 227 * 1024, "shared memory of a CTA");

template <bool kPair, int kHalves>
__global__ void __launch_bounds__(kThreadsL, 1)
    w8a16_gemm_kernel(const __grid_constant__ LinearMaps maps, const __grid_constant__ GemmArgs a, const __grid_constant__ TpArgs tp) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  GemmTail& sm = *reinterpret_cast<GemmTail*>(smem_raw + a.tail);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((smem_addr(smem_raw) & 1023u) != 0u) {  // (the same in every CTA)
    grid_dependency_wait();  // (the launch before this one clears the status word)
    if (tid == 0) atomicExch(a.status, 2);
    return;
  }
  const int M = a.M, Mp = a.Mp, N = a.N;
  constexpr int halves = kHalves;  // of the tile, of up to 128 tensor memory lanes each
  constexpr int kCtas = kPair ? 2 : 1;  // CTAs that an MMA instruction runs on
  const int pair_rank = kPair ? (int)(blockIdx.x & 1u) : 0, split = (int)blockIdx.y, nsplit = (int)gridDim.y;
  const int width = a.tile / halves;  // channels of a half
  const int n0 = (int)blockIdx.x * a.tile;
  // stages of this split: the k_steps dealt out as evenly as whole ones allow (the first splits one more)
  const int k_lo = split * (a.k_steps / nsplit) + min(split, a.k_steps % nsplit);
  const int iters = a.k_steps / nsplit + (split < a.k_steps % nsplit ? 1 : 0);
  const int n_mma = 2 * Mp;  // columns of an accumulator (a multiple of 32)
  uint32_t tmem_cols = 32;
  while ((int)tmem_cols < halves * n_mma) tmem_cols *= 2;
  // Every CTA of a split reads the same activation tiles: each pair starts at another K step (the sums are exact integers,
  // their order is free), so that the pairs do not ask the same L2 lines at the same time.
  const int rot = (int)(blockIdx.x / kCtas % (unsigned)iters);
  const uint32_t w_bytes = (uint32_t)(a.kb * a.tile * kTileK), x_bytes = (uint32_t)(a.kb * (n_mma / kCtas) * kTileK);
  const uint32_t leader = (uint32_t)(kCtas * split);  // rank of the pair's even CTA in the cluster: it owns the `full` barriers
  uint8_t* const ring = smem_raw;
  const int x_off = (int)w_bytes;

  if (tid == 0) {
    for (int s = 0; s < a.stages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.full[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.empty[s])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.done)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.w)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.x)) : "memory");
  }
  if (warp == 1) {
    if constexpr (kPair) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sm.tmem_base)), "r"(tmem_cols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sm.tmem_base)), "r"(tmem_cols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  if constexpr (kPair) {
    __syncthreads();
    cluster_sync();  // the barriers of the pair's leader are there
  }
  auto full_bar = [&](int s) {
    const uint32_t bar = smem_addr(&sm.full[s]);
    return kPair ? remote_smem(bar, (int)leader) : bar;
  };
  const uint64_t w_policy = l2_policy(a.weights_once != 0), x_policy = l2_policy(false);
  if (tid == 0) {
    // The weight tiles of the first stages, before the wait on the launch in front.  Behind this call's own level kernel whatever wrote
    // the weights is complete, and they are requested: their bytes are announced to the stage's barrier without an arrival; the
    // arrival comes with the activation tile's request.  Behind any other launch (levels that the caller kept) that launch may be
    // the one that writes them, and may still run: the tiles are requested into L2 only, where a later write replaces them, and
    // loaded behind the wait (1 row: 3584 x 8192 10.9 us loaded here, 11.7 from L2; block 5120 / 13824, whose GEMMs follow one
    // another, 55.7 and 51.9).
    for (int it = 0; it < a.stages && it < iters; ++it) {
      const int z = (k_lo + (it + rot < iters ? it + rot : it + rot - iters)) * a.kb;
      if (a.own_levels) {
        if (pair_rank == 0)
          asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&sm.full[it])), "r"(kCtas * w_bytes) : "memory");
        tma_load_steps<kPair>(smem_addr(ring + it * a.stage_bytes), &maps.w, n0, z, full_bar(it), w_policy);
      } else {
        tma_prefetch_steps(&maps.w, n0, z, w_policy);
      }
    }
  }
  grid_dependency_wait();
  grid_dependency_trigger();
  const unsigned tp_epoch = tp.world > 1 ? *reinterpret_cast<volatile unsigned*>(tp.launch_counter) : 0u;
  if (tid < kMaxM) sm.xs[tid] = tid < M ? a.xs[tid] : 0.f;
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sm.tmem_base;
  bool dead = false;

  if (warp == 0) {
    // ---- producer (both CTAs of a pair): tiles of stage s are requested when the MMAs that read its previous contents are
    // done.  The warp stays together and one lane issues, here and in the MMA warp: addresses and descriptors then live in
    // uniform registers (issued by a thread of its own, a stage of one step took 0.44 us whatever it held).
    const bool elected = elect_sync();
    int s = 0, kt = rot;
    uint32_t parity = 1;  // of the stage's previous use
    for (int it = 0; it < iters; ++it) {
      const bool early = a.own_levels && it < a.stages;  // (the weight tiles of the first stages are on their way already)
      if (it >= a.stages && !__all_sync(0xffffffffu, mbar_wait_l(smem_addr(&sm.empty[s]), parity))) {
        dead = true;
        break;
      }
      if (elected) {
        if (pair_rank == 0)
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&sm.full[s])),
                       "r"(kCtas * (x_bytes + (early ? 0u : w_bytes)))
                       : "memory");
        if (!early) tma_load_steps<kPair>(smem_addr(ring + s * a.stage_bytes), &maps.w, n0, (k_lo + kt) * a.kb, full_bar(s), w_policy);
        tma_load_steps<kPair>(smem_addr(ring + s * a.stage_bytes + x_off), &maps.x, pair_rank * Mp, (k_lo + kt) * a.kb, full_bar(s), x_policy);
      }
      if (++kt == iters) kt = 0;
      if (++s == a.stages) s = 0, parity ^= 1u;
    }
    if constexpr (kPair) {  // the last hand-overs, which come from the other CTA, arrive before this one may leave
      for (int it = iters; it < iters + a.stages && !dead; ++it) {
        if (it >= a.stages) dead = !__all_sync(0xffffffffu, mbar_wait_l(smem_addr(&sm.empty[s]), parity));
        if (++s == a.stages) s = 0, parity ^= 1u;
      }
    }
  } else if (warp == 1 && pair_rank == 0) {
    // ---- MMA issue (for the pair): D_half[128 kCtas n x 2 Mp] += W_tile[half] . Xl_tile^T, four K steps of 32 bytes per tile
    const bool elected = elect_sync();
    const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)n_mma >> 3) << 17) | ((128u * kCtas >> 4) << 24);
    const uint16_t both = (uint16_t)(3u << leader);
    auto commit = [&](uint64_t* bar) {  // arrives at this barrier, in both CTAs of a pair
      if constexpr (kPair)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_addr(bar)),
                     "h"(both)
                     : "memory");
      else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
    };
    const uint64_t w_step = (uint64_t)((a.tile * kTileK) >> 4), x_step = (uint64_t)(((n_mma / kCtas) * kTileK) >> 4);
    const uint64_t w_half = (uint64_t)((width * kTileK) >> 4);
    int s = 0;
    uint32_t parity = 0, acc = 0;
    for (int it = 0; it < iters; ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait_l(smem_addr(&sm.full[s]), parity))) {
        dead = true;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint64_t wd = desc_k_major_128b(smem_addr(ring + s * a.stage_bytes)), xd = desc_k_major_128b(smem_addr(ring + s * a.stage_bytes + x_off));
      for (int kt = 0; kt < a.kb; ++kt) {
        if (elected) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
            for (int half = 0; half < halves; ++half) {
              const uint32_t d = tmem + (uint32_t)(half * n_mma);
              const uint64_t wk = wd + (half ? w_half : 0u) + (uint64_t)(2 * ks), xk = xd + (uint64_t)(2 * ks);
              if constexpr (kPair)
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
                    "l"(wk), "l"(xk), "r"(idesc), "r"(ks ? 1u : acc)
                    : "memory");
              else
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
                    "l"(wk), "l"(xk), "r"(idesc), "r"(ks ? 1u : acc)
                    : "memory");
            }
          }
        }
        acc = 1;
        wd += w_step, xd += x_step;
      }
      if (elected) commit(&sm.empty[s]);  // the stage is free again when these MMAs have read it
      if (++s == a.stages) s = 0, parity ^= 1u;
    }
    if (elected) commit(&sm.done);
  }
  __syncwarp();
  // ---- epilogue: thread (half, j) of the 256 owns lane j of accumulator `half`, i.e. channel n0 + half * width + j, and with
  // one half only every second part of that lane's rows
  const int groups = Mp / 8;  // groups of eight rows of the batch; group j belongs to split j % nsplit
  const int owned = (groups + nsplit - 1) / nsplit;
  const int half = halves == 2 ? warp >> 2 : 0, j = (warp & 3) * 32 + lane;
  const int c_first = halves == 2 ? 0 : warp >> 2, c_step = halves == 2 ? 1 : 2;  // (sixteen rows at a time)
  const int n = n0 + half * width + j;
  const bool live = j < width && n < N;
  const float sc = live ? __bfloat162float(a.scale[n]) : 0.f;
  // landing area in the ring: [source split][owned group][half][row of the group][lane] fp32
  float* land = reinterpret_cast<float*>(smem_raw);
  const bool ok = mbar_wait_l(smem_addr(&sm.done), 0u);
  const bool bad = __syncthreads_or(dead || !ok) != 0;
  if (bad && tid == 0) atomicExch(a.status, 1);  // (only if the copy engine or the tensor core stopped answering)
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const bool exchange = nsplit > 1 || tp.world > 1;
  if (exchange) cluster_sync();  // every ring of the cluster has been read to the end: the landing areas are free
  auto store = [&](int m, float dot32) {
    const float dot = __bfloat162float(__float2bfloat16_rn(dot32));                  // F.linear's bf16 result
    if (live && m < M) a.y[(int64_t)m * N + n] = __float2bfloat16_rn(dot * sc);      // * weight_scaler
  };
  if (!bad) {
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(half * n_mma);
    uint32_t v[2][2][16];  // [parity][h, l][row]: the next sixteen rows leave tensor memory while these are worked on
    auto fetch = [&](int c, uint32_t (&d)[2][16]) {
      tmem_ld_16(lanes + (uint32_t)(16 * c), d[0]);
      tmem_ld_16(lanes + (uint32_t)(Mp + 16 * c), d[1]);
    };
    auto finish = [&](int c, const uint32_t (&d)[2][16]) {
      float sum[16];
#pragma unroll
      for (int r = 0; r < 16; r += 4) {
        const float4 x4 = *reinterpret_cast<const float4*>(&sm.xs[16 * c + r]);
        const float xr[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[r + e] = fmaf((float)(int)d[0][r + e], 254.f, (float)(int)d[1][r + e]) * xr[e];
      }
      if (!exchange) {
#pragma unroll
        for (int r = 0; r < 16; ++r) store(16 * c + r, sum[r]);
        return;
      }
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        const int g = 2 * c + part, q = g / nsplit, owner = kCtas * (g - q * nsplit) + pair_rank;
        const uint32_t base = remote_smem(smem_addr(land + ((split * owned + q) * halves + half) * 8 * 128 + j), owner);
#pragma unroll
        for (int r = 0; r < 8; ++r) st_cluster_f32(base + (uint32_t)(r * 128 * 4), sum[8 * part + r]);
      }
    };
    const int chunks = Mp / 16;
    if (c_first < chunks) fetch(c_first, v[0]);
    for (int c = c_first; c < chunks; c += 2 * c_step) {
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (c + c_step < chunks) fetch(c + c_step, v[1]);
      finish(c, v[0]);
      if (c + c_step < chunks) {
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c + 2 * c_step < chunks) fetch(c + 2 * c_step, v[0]);
        finish(c + c_step, v[1]);
      }
    }
  }
  if (exchange) {
    cluster_sync();  // all partial sums have landed
    if (!bad) {
      auto reduce = [&](auto cs_tag) {
        constexpr int kCs = decltype(cs_tag)::value;
        // (the landing area is written with a lane per channel: with one half the two groups of warps take turns here too)
        for (int q = c_first; q < owned; q += c_step) {
          const int g = q * kCs + split;
          if (g >= groups) break;
          float acc[8];  // (eight independent chains; all loads before the stores)
#pragma unroll
          for (int r = 0; r < 8; ++r) acc[r] = land[(((0 * owned + q) * halves + half) * 8 + r) * 128 + j];
#pragma unroll
          for (int src = 1; src < kCs; ++src) {
#pragma unroll
            for (int r = 0; r < 8; ++r) acc[r] += land[(((src * owned + q) * halves + half) * 8 + r) * 128 + j];
          }
          if (tp.world > 1) {
            // this rank's sums of the group go into its own buffer, where the other ranks read them; the roundings
            // follow below, on the sum over the ranks
            float* dst = reinterpret_cast<float*>(tp.buffers[tp.rank] + kTpDataOffset) + (int64_t)(tp_epoch & 1u) * kMaxM * N;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              const int m = 8 * g + r;
              if (m < M && live) __stcg(&dst[(int64_t)m * N + n], acc[r]);
            }
            continue;
          }
#pragma unroll
          for (int r = 0; r < 8; ++r) store(8 * g + r, acc[r]);
        }
      };
      switch (nsplit) {
        case 1: reduce(std::integral_constant<int, 1>{}); break;
        case 2: reduce(std::integral_constant<int, 2>{}); break;
        case 3: reduce(std::integral_constant<int, 3>{}); break;
        case 4: reduce(std::integral_constant<int, 4>{}); break;
        case 5: reduce(std::integral_constant<int, 5>{}); break;
        case 6: reduce(std::integral_constant<int, 6>{}); break;
        case 7: reduce(std::integral_constant<int, 7>{}); break;
        default: reduce(std::integral_constant<int, 8>{}); break;
      }
      if (tp.world > 1 && split < groups) {  // (a CTA without a group of rows has nothing to send or to wait for)
        // ---- sum over the ranks: tell every rank that this CTA's groups are in this rank's buffer, wait (bounded) for
        // the same CTA of every rank, read their sums and add them in the order of the ranks
        const int par = (int)(tp_epoch & 1u);
        auto flag_of = [&](int buffer_of, int src) {  // the sums of rank `src` are ready, as told to rank `buffer_of`
          return reinterpret_cast<unsigned*>(tp.buffers[buffer_of] + kTpFlagOffset) +
                 (((size_t)par * 8 + src) * kTpMaxTiles + blockIdx.x) * 8 + split;
        };
        __syncthreads();  // every thread's stores are issued ...
        if (tid < tp.world && tid != tp.rank) {
          __threadfence_system();  // ... and ordered before the launch number that announces them
          st_sys_u32(flag_of(tid, tp.rank), tp_epoch);
          const long long t0c = clock64();
          while (ld_sys_u32(flag_of(tp.rank, tid)) != tp_epoch) {
            if (clock64() - t0c > tp.wait_cycles) {  // a rank never came: report, go on with what is there
              atomicExch(tp.status, 1);
              break;
            }
          }
          __threadfence_system();
        }
        __syncthreads();
        asm volatile("" ::: "memory");  // (the peer loads below carry no memory clobber of their own)
        const size_t part_off = kTpDataOffset + (size_t)par * kMaxM * N * sizeof(float);
        // A group is eight rows x `tile` channels, in pieces of four channels (16 bytes; a tile is a multiple of eight
        // channels).  A thread has twelve pieces (twelve loads per rank) in flight at a time.
        constexpr int kBatch = 12;
        const int my_groups = (groups - split + nsplit - 1) / nsplit, per_row = a.tile / 4, pieces = my_groups * 8 * per_row;
        for (int base = tid; base < pieces; base += kBatch * kThreadsL) {
          float4 sum[kBatch];
          int64_t at[kBatch];  // element offset of the piece, -1: none
#pragma unroll
          for (int b = 0; b < kBatch; ++b) {
            const int idx = base + b * kThreadsL, row = idx / per_row;
            const int m = 8 * ((row >> 3) * nsplit + split) + (row & 7), c = n0 + 4 * (idx % per_row);
            at[b] = (idx < pieces && m < M && c < N) ? (int64_t)m * N + c : -1;
            sum[b] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
          for (int src = 0; src < tp.world; ++src) {
            const float* part = reinterpret_cast<const float*>(tp.buffers[src] + part_off);
            float4 v[kBatch];
#pragma unroll
            for (int b = 0; b < kBatch; ++b) {
              v[b] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (at[b] >= 0) v[b] = src == tp.rank ? __ldcg(reinterpret_cast<const float4*>(part + at[b])) : ld_sys_f32x4(part + at[b]);
            }
#pragma unroll
            for (int b = 0; b < kBatch; ++b) sum[b].x += v[b].x, sum[b].y += v[b].y, sum[b].z += v[b].z, sum[b].w += v[b].w;
          }
#pragma unroll
          for (int b = 0; b < kBatch; ++b) {
            if (at[b] < 0) continue;
            const int c = (int)(at[b] % N);
            const uint2 sraw = __ldg(reinterpret_cast<const uint2*>(a.scale + c));
            const __nv_bfloat16* sb = reinterpret_cast<const __nv_bfloat16*>(&sraw);
            const float a4[4] = {sum[b].x, sum[b].y, sum[b].z, sum[b].w};
            uint2 o;
            __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              ob[e] = __float2bfloat16_rn(__bfloat162float(__float2bfloat16_rn(a4[e])) * __bfloat162float(sb[e]));
            *reinterpret_cast<uint2*>(a.y + at[b]) = o;
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if constexpr (kPair) cluster_sync();  // (tensor memory is given back by both CTAs of a pair, when neither reads it any more)
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if constexpr (kPair)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
  }
}

// ---------------------------------------------------------------- more than 128 rows (prefill)
// Bound: the integer MMAs (two levels: 4 M N K operations) where a tile has many steps of K (tensor pipe 0.88 of the active cycles with
// 112), and the epilogue between the tiles where it has few (0.62 with the gate's 32).  Weights as the M = 128 operand twice (256 channels), a block of up
// to 128 rows as the N operand (h rows, then l rows), accumulators in all of tensor memory; persistent CTAs, one per SM,
// walk the tiles with the row blocks fastest, so that the CTAs of a moment share weight tiles in L2.  A tile step (128 bytes
// of K) reads 64 KB for 1024 cycles of MMA.  The ring keeps filling under the epilogue; the accumulators do not double, but where
// the CTA has a further tile they are given back as soon as their sums are held as bf16 in registers: the gate's exponentials and the stores
// run under the next tile's MMAs (feed-forward block 4096 / 14336 with 1024 rows, seven rounds of tiles: 325.0 us stored as it goes, 280.6 held).  A CTA's last
// tile has nothing to wait for and stores as it goes (4096 x 6144 with 146 rows, one round: 19.9 us held, 18.7).
// The 128-row blocks through the decode kernel that this replaces streamed the weights again for every block and paid its
// set-up and cluster reduction each time: 27 us per block of 4096 x 14336, where this takes 15.
//   warp 0 requests tiles, warp 1 issues MMAs, warps 2-9 run the epilogue (a warp owns 32 TMEM lanes = channels and half
//   of the block's rows).
// Two forms: a layer (256 channels of one weight matrix), and the feed-forward block's gate (128 channels of w1 and the same 128
// of w3: the thread that has both writes bf16(silu(a)) * b, so that neither projection goes through memory).
constexpr int kThreadsT = 320;
struct __align__(1024) SmemT {
  uint8_t w[kStages][kTileN * kTileK];
  uint8_t x[kStages][2 * kMaxM * kTileK];
  uint64_t full[kStages], empty[kStages], acc_full, acc_empty;
  uint32_t tmem_base;
  volatile int dead;
};
struct TileMaps {
  CUtensorMap w0, w1, x;  // w1: the second matrix of the gate form
};
struct TileArgs {
  const float* xs;               // [blocks * Rb]
  const __nv_bfloat16 *s0, *s1;  // channel scales
  __nv_bfloat16* y;
  int M, N, Rb, blocks, k_tiles, tiles;
};

template <bool kGate>
__global__ void __launch_bounds__(kThreadsT, 1)
    w8a16_tiles_kernel(const __grid_constant__ TileMaps maps, const __grid_constant__ TileArgs a, int* status) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  SmemT& sm = *reinterpret_cast<SmemT*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((smem_addr(smem_raw) & 1023u) != 0u) {
    grid_dependency_wait();
    if (tid == 0) atomicExch(status, 2);
    return;
  }
  const int n_mma = 2 * a.Rb;
  constexpr int kChannels = kGate ? 128 : 256;  // output channels of a tile
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.full[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.empty[s])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.acc_full)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 256;" ::"r"(smem_addr(&sm.acc_empty)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sm.dead = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sm.tmem_base)),
                 "r"((uint32_t)kTmemColsL)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  grid_dependency_wait();
  grid_dependency_trigger();
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sm.tmem_base;
  // a wait that gives up ends the roles of its CTA one after the other (the others see `dead`)
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    const uint32_t b = smem_addr(bar);
    if (mbar_try(b, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
      for (int i = 0; i < 16; ++i)
        if (mbar_try(b, parity)) return true;
      if (sm.dead || clock64() - t0 > kWaitCyclesL) {
        sm.dead = 1;
        return false;
      }
    }
  };

  if (warp == 0) {
    if (elect_sync()) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < a.tiles && ok; t += gridDim.x) {
        const int rb = t % a.blocks, c0 = t / a.blocks * kChannels;
        for (int k = 0; k < a.k_tiles && ok; ++k, ++it) {
          const uint32_t s = it % kStages;
          if (it >= kStages) ok = wait(&sm.empty[s], (it / kStages - 1) & 1u);
          if (!ok) break;
          const uint32_t bar = smem_addr(&sm.full[s]);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                       "r"((uint32_t)(kTileN * kTileK + n_mma * kTileK))
                       : "memory");
          tma_load_2d(smem_addr(&sm.w[s][0]), &maps.w0, k * kTileK, c0, bar);
          if constexpr (kGate) tma_load_2d(smem_addr(&sm.w[s][128 * kTileK]), &maps.w1, k * kTileK, c0, bar);
          tma_load_2d(smem_addr(&sm.x[s][0]), &maps.x, k * kTileK, rb * n_mma, bar);
        }
      }
      if (!ok) {  // (requests in flight get their time before the CTA leaves)
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {
        }
      }
    }
  } else if (warp == 1) {
    const bool elected = elect_sync();
    const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)n_mma >> 3) << 17) | ((128u >> 4) << 24);
    uint32_t it = 0, done = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < a.tiles && ok; t += gridDim.x, ++done) {
      if (done > 0) ok = __all_sync(0xffffffffu, wait(&sm.acc_empty, (done - 1) & 1u));
      for (int k = 0; k < a.k_tiles && ok; ++k, ++it) {
        const uint32_t s = it % kStages;
        ok = __all_sync(0xffffffffu, wait(&sm.full[s], (it / kStages) & 1u));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elected) {
          const uint64_t wd = desc_k_major_128b(smem_addr(&sm.w[s][0])), xd = desc_k_major_128b(smem_addr(&sm.x[s][0]));
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const uint32_t acc = (k > 0 || ks > 0) ? 1u : 0u;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              asm volatile(
                  "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                  "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem + (uint32_t)(half * n_mma)),
                  "l"(wd + (uint64_t)((half * (128 * kTileK) + 32 * ks) >> 4)), "l"(xd + (uint64_t)((32 * ks) >> 4)), "r"(idesc), "r"(acc)
                  : "memory");
            }
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(&sm.empty[s]))
                       : "memory");
        }
      }
      if (elected)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(&sm.acc_full))
                     : "memory");
    }
  } else {
    // ---- epilogue: warp w owns TMEM lanes 32 (w % 4) .. and rows [r_lo, r_hi) of the block
    const int part = (warp - 2) >> 2, quad = warp & 3;
    const int chunks = a.Rb / 8, r_lo = (part ? (chunks + 1) / 2 : 0) * 8, r_hi = (part ? chunks : (chunks + 1) / 2) * 8;
    const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
    uint32_t done = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < a.tiles && ok; t += gridDim.x, ++done) {
      const int rb = t % a.blocks, c0 = t / a.blocks * kChannels, ch = c0 + quad * 32 + lane;
      const int ch1 = kGate ? ch : ch + 128;
      const float sc0 = ch < a.N ? __bfloat162float(a.s0[ch]) : 0.f;
      const float sc1 = ch1 < a.N ? __bfloat162float((kGate ? a.s1 : a.s0)[ch1]) : 0.f;
      // the row scales of this warp's up to 64 rows, a lane each (fetched ahead: read one by one in the loop below they
      // cost it an L2 round trip per chunk)
      const int m_lo = rb * a.Rb + r_lo;
      const float xs_a = r_lo + lane < r_hi ? __ldg(a.xs + m_lo + lane) : 0.f;
      const float xs_b = r_lo + 32 + lane < r_hi ? __ldg(a.xs + m_lo + 32 + lane) : 0.f;
      ok = wait(&sm.acc_full, done & 1u);
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      __nv_bfloat16* row0 = a.y + (int64_t)m_lo * a.N;
      const int live = a.M - m_lo;  // rows of this warp that exist
      uint32_t v[2][4][8];          // [chunk parity][h0, l0, h1, l1][row]
      auto fetch = [&](int r, uint32_t (&d)[4][8]) {
        tmem_ld_8(lanes + (uint32_t)(r_lo + r), d[0]);
        tmem_ld_8(lanes + (uint32_t)(a.Rb + r_lo + r), d[1]);
        tmem_ld_8(lanes + (uint32_t)(n_mma + r_lo + r), d[2]);
        tmem_ld_8(lanes + (uint32_t)(n_mma + a.Rb + r_lo + r), d[3]);
      };
      const bool more = t + (int)gridDim.x < a.tiles;  // a further tile's MMAs wait for tensor memory
      auto store = [&](int r, __nv_bfloat162 y) {
        if (r >= live) return;
        __nv_bfloat16* row = row0 + (int64_t)r * a.N;
        if constexpr (kGate) {
          if (ch < a.N) row[ch] = gate_value(y.x, y.y);
        } else {
          if (ch < a.N) row[ch] = y.x;
          if (ch1 < a.N) row[ch1] = y.y;
        }
      };
      // F.linear's bf16 result, then the channel's scale: two bf16 operations
      auto value = [&](int r, int j, const uint32_t (&d)[4][8]) {
        const float xr = __shfl_sync(0xffffffffu, r < 32 ? xs_a : xs_b, (r & 31) + j);
        const float d0 = __bfloat162float(__float2bfloat16_rn(fmaf((float)(int)d[0][j], 254.f, (float)(int)d[1][j]) * xr));
        const float d1 = __bfloat162float(__float2bfloat16_rn(fmaf((float)(int)d[2][j], 254.f, (float)(int)d[3][j]) * xr));
        return __floats2bfloat162_rn(d0 * sc0, d1 * sc1);
      };
      // the next chunk leaves tensor memory while this one is worked on
      const int nr = r_hi - r_lo;
      if (nr > 0) fetch(0, v[0]);
      auto chunks_of_16 = [&](int r, auto take) {
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (r + 8 < nr) fetch(r + 8, v[1]);
#pragma unroll
        for (int j = 0; j < 8; ++j) take(r + j, value(r, j, v[0]));
        if (r + 8 < nr) {
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (r + 16 < nr) fetch(r + 16, v[0]);
#pragma unroll
          for (int j = 0; j < 8; ++j) take(r + 8 + j, value(r + 8, j, v[1]));
        }
      };
      auto give_back = [&]() {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&sm.acc_empty)) : "memory");
      };
      if (more) {
        // The projections' bf16 results of both channels, packed, for all rows of the thread: tensor memory is free for the
        // next tile's MMAs when the last of them has left it, before the gate's exponentials and divisions and before the stores.
        uint32_t held[kMaxM / 2];
#pragma unroll
        for (int r = 0; r < kMaxM / 2; r += 16)
          if (r < nr) chunks_of_16(r, [&](int i, __nv_bfloat162 y) { held[i] = *reinterpret_cast<const uint32_t*>(&y); });
        give_back();
#pragma unroll
        for (int r = 0; r < kMaxM / 2; ++r)
          if (r < nr) store(r, *reinterpret_cast<const __nv_bfloat162*>(&held[r]));
      } else {
#pragma unroll 1
        for (int r = 0; r < nr; r += 16) chunks_of_16(r, store);
        give_back();
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && sm.dead) atomicExch(status, 1);
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kTmemColsL) : "memory");
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}
// rows x K bytes, row-major, seen as K / 128 steps of [rows x 128 bytes]; boxes of kb steps of box_rows rows, 128-byte swizzle
bool encode_steps(CUtensorMap* map, const void* base, int64_t rows, int64_t K, int box_rows, int kb) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)kTileK, (cuuint64_t)rows, (cuuint64_t)(K / kTileK)};
  const cuuint64_t str[2] = {(cuuint64_t)K, (cuuint64_t)kTileK};
  const cuuint32_t box[3] = {(cuuint32_t)kTileK, (cuuint32_t)box_rows, (cuuint32_t)kb};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, str, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// rows x K bytes, row-major; boxes of box_rows x 128 bytes with the 128-byte swizzle
bool encode_2d(CUtensorMap* map, const void* base, int64_t rows, int64_t K, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t str[1] = {(cuuint64_t)K};
  const cuuint32_t box[2] = {(cuuint32_t)kTileK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, str, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int sm_count_l() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  return sms;
}

// How more than 128 rows are cut into blocks: equal blocks of Rb rows (a multiple of 8), so that no block is mostly padding,
// and so many of them that the tiles fill whole rounds of the SMs.  Cost of a round in cycles: the tile's steps (MMA 8 Rb, or
// the step's bytes at about 55 per cycle and SM where the block is narrow) and the epilogue that the next tile's MMAs wait for.
struct RowBlocks {
  int Rb, blocks;
};
RowBlocks row_blocks(int M, int N, int K, int channels) {
  static const int sms = sm_count_l();
  const int ctiles = (N + channels - 1) / channels, k_tiles = K / kTileK;
  RowBlocks best{0, 0};
  double best_cost = 0;
  for (int nb = (M + kMaxM - 1) / kMaxM; nb <= (M + 15) / 16; ++nb) {
    const int rb = ((M + nb - 1) / nb + 7) / 8 * 8, blocks = (M + rb - 1) / rb;
    const double step = std::max(8.0 * rb, (32768.0 + 256.0 * rb) / 55.0);
    const int64_t rounds = ((int64_t)ctiles * blocks + sms - 1) / sms;
    const double cost = (double)rounds * (k_tiles * step + 2500.0 + 25.0 * rb);
    if (best.Rb == 0 || cost < best_cost) best_cost = cost, best = RowBlocks{rb, blocks};
  }
  return best;
}

// How the channels and the K steps are dealt out over the SMs.  Clusters of `split` CTAs or pairs; `slots` of them fit the GPU at
// once (a cluster lies within a group of SMs, so that larger ones leave some SMs over: the driver says how many).  For
// every form the tile is the narrowest that covers the channels in whole waves of clusters; the plan with the shortest
// estimated run is taken.  A stage costs its hand-over and its MMAs or bytes (the weights at a share of the memory rate, the
// activations from L2); a wave costs set-up, first fetch and epilogue.  The constants (us, bytes per us) are fitted to the
// measured times of up to nine forms each of 9 shapes (1280 to 28672 channels, K of 4096 to 28672) with 7 and 96 rows, the estimate
// mostly within 10 %.  Against every form timed for 10 such shapes with 1, 7, 16, 32, 48, 64, 80, 96 and 128 rows the form taken is
// within 5 % of the fastest in 87 of the 90 and within 9 % in all (3584 -> 8192 with 32 rows: 10.9 against 10.0 for pairs in two
// splits).  Measured, us, 96 rows / 7 rows: pairs on
// 8192 -> 28672 49.0 / 40.7 (single CTAs 52.1 / 42.4), pairs in two splits on 28672 -> 8192 46.4 / 37.8 (single CTAs in four 51.0 /
// 42.0), single CTAs in four splits on 14336 -> 4096 17.1 / 12.7 (one pair per tile 31.8 / 18.2).
struct GemmPlan {
  int pair, split, tile, halves, tiles, kb;
};
constexpr int kMaxCluster = 8;  // CTAs of a cluster: the portable limit
// Clusters of single CTAs [0] and of pairs [1] by their number of splits that fit the GPU at once.
struct ClusterSlots {
  int n[2][kMaxCluster + 1];
};
// The row-parallel form (`tp`) exchanges its sums by tile and split, so every rank has to come to the same plan: it is made for
// these counts (what the driver said of one B200 with 148 SMs), whatever the rank's own GPU holds.  How many clusters fit differs from GPU to GPU with
// the SMs that each of them has switched off; a GPU that holds fewer runs the same plan in one more wave.
constexpr ClusterSlots kTpSlots = {{{0, 148, 74, 45, 33, 26, 22, 15, 15}, {0, 74, 33, 22, 15, 0, 0, 0, 0}}};
GemmPlan plan_gemm(int M, int N, int K, bool tp, const ClusterSlots& own_slots) {
  const ClusterSlots& all_slots = tp ? kTpSlots : own_slots;
  const int k_tiles = K / kTileK, Mp = (M + 15) / 16 * 16;
  GemmPlan best{};
  float best_cost = 0.f;
  for (int ctas = 1; ctas <= 2; ++ctas) {
    const int x_rows = 2 * Mp / ctas;
    for (int c = 1; c * ctas <= kMaxCluster && c <= k_tiles; ++c) {
      const int slots = all_slots.n[ctas - 1][c];
      const int waves = (N + ctas * kTileN * slots - 1) / (ctas * kTileN * slots);
      int tile = (N + ctas * slots * waves - 1) / (ctas * slots * waves);
      tile = tile <= 128 ? std::max(32, (tile + 7) / 8 * 8) : (tile + 15) / 16 * 16;
      if (tp && (N + tile - 1) / tile >= kTpMaxTiles) tile = kTileN;  // (the exchange between the ranks counts its tiles)
      const int halves = tile <= 128 ? 1 : 2;
      // Stages of about 32 KB: four to six of them are in flight, and none is so short that its hand-over is what it costs.
      int kb = 1;
      while (kb < 8 && 2 * kb * c <= k_tiles && 2 * kb * (tile + x_rows) * kTileK <= 40 * 1024) kb *= 2;
      const int groups = (N + ctas * tile - 1) / (ctas * tile), rounds = (groups + slots - 1) / slots;
      const int steps = ((k_tiles + kb - 1) / kb + c - 1) / c;
      const int active = std::min(groups, slots) * c * ctas;
      const float mma = (float)halves * std::max(0.11f, 0.0021f * (float)Mp);
      const float bytes = (float)(tile * kTileK) * (float)active / 8.6e6f + (float)(x_rows * kTileK) / 288e3f + 0.045f * (float)(halves - 1);
      const float step = 0.063f + (float)kb * std::max(mma, bytes);
      const float cost = (float)rounds * (4.35f + 0.024f * (float)(Mp * halves) + (ctas == 2 ? 0.7f : 0.f) + (c > 1 ? 0.33f : 0.f) + (float)steps * step);
      if (best.tiles == 0 || cost < best_cost) best_cost = cost, best = GemmPlan{ctas == 2, c, tile, halves, ctas * groups, kb};
    }
  }
  return best;
}

}  // namespace
}  // namespace jpt

using namespace jpt;

static size_t blocks_workspace_bytes(const RowBlocks& rb, int K) {
  const size_t rows = (size_t)rb.blocks * rb.Rb;
  return 256 + (2 * rows * K + 255) / 256 * 256 + (rows * sizeof(float) + 255) / 256 * 256;
}

extern "C" size_t jpt_w8a16_linear_workspace_bytes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M > kMaxM) return blocks_workspace_bytes(row_blocks(M, N, K, kTileN), K);
  const int Mp = (M + 15) / 16 * 16;
  const size_t levels = ((size_t)2 * Mp * K + 255) / 256 * 256;
  const size_t xs = 1024;
  return 256 + levels + xs;
}

extern "C" size_t jpt_w8a16_gate_workspace_bytes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  return blocks_workspace_bytes(row_blocks(M, N, K, 128), K);
}

namespace jpt {
namespace {
// The workspace of up to 128 rows: status word, level matrix [2 Mp, K], row scales.
struct LevelsView {
  int* status;  // 0, or the code of a CTA that gave up
  int8_t* lev;
  float* xs;
  int Mp;
};
LevelsView levels_view(void* workspace, int M, int K) {
  LevelsView v;
  v.Mp = (M + 15) / 16 * 16;
  char* ws = static_cast<char*>(workspace);
  v.status = reinterpret_cast<int*>(ws);
  v.lev = reinterpret_cast<int8_t*>(ws + 256);
  const size_t levels = ((size_t)2 * v.Mp * K + 255) / 256 * 256;
  v.xs = reinterpret_cast<float*>(ws + 256 + levels);
  return v;
}

// Clusters that the current device holds at once; the kernels' attributes are set on the way.
constexpr size_t kGemmSmem = kRingBytes + kTailBytes;
using GemmKernel = void (*)(const LinearMaps, const GemmArgs, const TpArgs);
GemmKernel gemm_kernel(bool pair, int halves) {
  if (pair) return halves == 2 ? w8a16_gemm_kernel<true, 2> : w8a16_gemm_kernel<true, 1>;
  return halves == 2 ? w8a16_gemm_kernel<false, 2> : w8a16_gemm_kernel<false, 1>;
}
cudaLaunchConfig_t gemm_config(dim3 grid, size_t smem, cudaStream_t st, cudaLaunchAttribute (&attr)[2], bool pair, int split) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kThreadsL);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = pair ? 2 : 1;
  attr[0].val.clusterDim.y = split;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}
// (filled on first use per device; a query that failed is made again at the next call, and the launch reports what is wrong)
const ClusterSlots& device_slots() {
  static std::mutex mu;
  static ClusterSlots known[64];
  static thread_local ClusterSlots guess;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  ClusterSlots& slots = known[dev & 63];
  bool all = true;
  for (int pair = 0; pair < 2; ++pair) {
    for (int split = 1; split * (pair + 1) <= kMaxCluster; ++split) {
      int& n = slots.n[pair][split];
      if (n == 0) {
        cudaLaunchAttribute attr[2];
        const cudaLaunchConfig_t cfg = gemm_config(dim3(pair ? 2 : 1, split), kGemmSmem, nullptr, attr, pair, split);
        bool ok = true;
        for (int halves = 1; halves <= 2; ++halves)
          ok = ok && cudaFuncSetAttribute(gemm_kernel(pair, halves), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem) == cudaSuccess;
        if (!ok || cudaOccupancyMaxActiveClusters(&n, gemm_kernel(pair, 2), &cfg) != cudaSuccess || n <= 0) {
          cudaGetLastError();
          n = 0;
          all = false;
        }
      }
      guess.n[pair][split] = n > 0 ? n : std::max(1, sm_count_l() / ((pair ? 2 : 1) * split));
    }
  }
  return all ? slots : guess;
}

// The GEMM on levels that a launch before this one in the stream wrote (`own_levels`: the launch directly in front, by this call).  The
// launch may start while the one in front drains (it asks for its first weight tiles at once) and waits for its results on
// the device.
int launch_gemm(const LevelsView& lv, const void* w, const void* w_scale, void* y, int M, int N, int K, cudaStream_t st, bool own_levels,
                const TpArgs* tp_in = nullptr) {
  const GemmPlan plan = plan_gemm(M, N, K, tp_in != nullptr, device_slots());
  const int x_rows = plan.pair ? lv.Mp : 2 * lv.Mp;  // rows of levels that a CTA loads
  TpArgs tp;
  memset(&tp, 0, sizeof(tp));
  tp.world = 1;
  if (tp_in) tp = *tp_in;
  LinearMaps maps;
  memset(&maps, 0, sizeof(maps));
  JPT_REQUIRE(encode_steps(&maps.w, w, N, K, plan.tile, plan.kb) && encode_steps(&maps.x, lv.lev, 2 * lv.Mp, K, x_rows, plan.kb), JPT_EINVAL,
              "w8a16_linear: the tensors cannot be described by a tensor map");
  GemmArgs a;
  memset(&a, 0, sizeof(a));
  a.xs = lv.xs;
  a.scale = static_cast<const __nv_bfloat16*>(w_scale);
  a.y = static_cast<__nv_bfloat16*>(y);
  a.status = lv.status;
  a.M = M, a.Mp = lv.Mp, a.N = N, a.k_steps = (K / kTileK + plan.kb - 1) / plan.kb;
  a.tile = plan.tile, a.kb = plan.kb;
  a.weights_once = (int64_t)N * K > (64ll << 20);  // (half of L2)
  a.own_levels = own_levels;
  a.stage_bytes = plan.kb * (plan.tile + x_rows) * kTileK;
  a.stages = std::min(kMaxStages, kRingBytes / a.stage_bytes);
  // the landing area of the partial sums: [split][groups a split owns][half][8 rows][128 lanes] fp32, at most 23 groups = 184 KB
  const int landing = plan.split * ((lv.Mp / 8 + plan.split - 1) / plan.split) * plan.halves * 8 * 128 * (int)sizeof(float);
  a.tail = std::max(a.stages * a.stage_bytes, landing);
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = gemm_config(dim3(plan.tiles, plan.split), (size_t)a.tail + kTailBytes, st, attr, plan.pair, plan.split);
  cfg.numAttrs = pdl_enabled() ? 2 : 1;  // (also inside a graph capture: the weight tiles stream in under the level kernel)
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_kernel(plan.pair, plan.halves), maps, a, tp);
  if (e != cudaSuccess) return fail((int)e, "w8a16_gemm_kernel: %s", cudaGetErrorString(e));
  return 0;
}

// (the level kernel also clears the status word and the padding rows of the level matrix)
int launch_levels(const void* x, const LevelsView& lv, int M, int K, cudaStream_t st, bool clear_status,
                  unsigned* launch_counter = nullptr) {
  // Started under the launch in front, the CTAs crowd on the SMs that it leaves free, eight on one; this much shared memory keeps them to two
  // (8192 x 1280 with 128 rows 15.4 us, 13.9 with it; 8192 x 8192 with 84 22.4 and 21.2).  Few CTAs start earlier without (3584 x 8192
  // with 33 rows 13.2 us, 13.8 with it).
  size_t apart = 0;
  if (lv.Mp > 64) {
    apart = 100 * 1024;
    static bool configured[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
      const cudaError_t e = cudaFuncSetAttribute(x_levels_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)apart);
      if (e != cudaSuccess) return fail((int)e, "x_levels_kernel: configuring the kernel: %s", cudaGetErrorString(e));
      if (dev >= 0 && dev < 64) configured[dev] = true;
    }
  }
  launch_after_previous(x_levels_kernel, dim3(lv.Mp), dim3(256), apart, st, static_cast<const __nv_bfloat16*>(x), lv.lev, lv.xs, lv.status, M,
                        lv.Mp, K, clear_status ? 1 : 0, launch_counter);
  return check_launch("x_levels_kernel");
}

// More than 128 rows: the level kernel over all of them, then the tiles.
template <bool kGate>
int launch_tiles(const void* x, const void* w0, const void* s0, const void* w1, const void* s1, void* y, int M, int N, int K,
                 void* workspace, int* status, cudaStream_t st) {
  const RowBlocks rb = row_blocks(M, N, K, kGate ? 128 : kTileN);
  const int rows = rb.blocks * rb.Rb;
  char* ws = static_cast<char*>(workspace);
  LevelsView lv;
  lv.status = status ? status : reinterpret_cast<int*>(ws);
  lv.lev = reinterpret_cast<int8_t*>(ws + 256);
  lv.xs = reinterpret_cast<float*>(ws + 256 + ((size_t)2 * rows * K + 255) / 256 * 256);
  lv.Mp = rb.Rb;
  launch_after_previous(x_levels_kernel, dim3(rows), dim3(256), 0, st, static_cast<const __nv_bfloat16*>(x), lv.lev, lv.xs, lv.status, M, rb.Rb,
                        K, 1, static_cast<unsigned*>(nullptr));
  if (int rc = check_launch("x_levels_kernel")) return rc;
  TileMaps maps;
  memset(&maps, 0, sizeof(maps));
  JPT_REQUIRE(encode_2d(&maps.w0, w0, N, K, kGate ? 128 : kTileN) && (!kGate || encode_2d(&maps.w1, w1, N, K, 128)) &&
                  encode_2d(&maps.x, lv.lev, 2 * (int64_t)rows, K, 2 * rb.Rb),
              JPT_EINVAL, "w8a16_linear: the tensors cannot be described by a tensor map");
  static bool configured[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(w8a16_tiles_kernel<kGate>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemT));
    if (e != cudaSuccess) return fail((int)e, "w8a16_linear: configuring the kernel: %s", cudaGetErrorString(e));
    configured[dev] = true;
  }
  TileArgs a;
  memset(&a, 0, sizeof(a));
  a.xs = lv.xs;
  a.s0 = static_cast<const __nv_bfloat16*>(s0), a.s1 = static_cast<const __nv_bfloat16*>(s1);
  a.y = static_cast<__nv_bfloat16*>(y);
  a.M = M, a.N = N, a.Rb = rb.Rb, a.blocks = rb.blocks, a.k_tiles = K / kTileK;
  constexpr int kChannels = kGate ? 128 : kTileN;
  const int64_t tiles = (int64_t)((N + kChannels - 1) / kChannels) * rb.blocks;
  JPT_REQUIRE(tiles < (1ll << 31), JPT_ERANGE, "w8a16_linear: too many rows");
  a.tiles = (int)tiles;
  static const int sms = sm_count_l();
  launch_after_previous(w8a16_tiles_kernel<kGate>, dim3((unsigned)std::min<int64_t>(tiles, sms)), dim3(kThreadsT), sizeof(SmemT), st, maps, a,
                        lv.status);
  return check_launch("w8a16_tiles_kernel");
}

// CTAs per row of the element-wise producers (a cluster along x): enough of them to fill the GPU
int row_parts(int rows, int K) {
  const int steps = K / 8;
  int c = 1;
  // (one CTA of 1024 threads per row measured faster than a row split over a cluster: 3.7 against 9.8 us for
  // RMSNorm of [96, 8192]; the split stays available for single rows of long vectors)
  while (c < 8 && rows * c < 8 && steps % (c * 2) == 0 && steps / (c * 2) >= kRowThreads) c *= 2;
  return c;
}
template <typename... KArgs, typename... Args>
int launch_rows(const char* name, void (*kernel)(KArgs...), int rows, int parts, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(parts, rows);
  cfg.blockDim = dim3(kRowThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = parts;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
  if (e != cudaSuccess) return fail((int)e, "%s: %s", name, cudaGetErrorString(e));
  return 0;
}

int check_levels_args(const char* who, int M, int K, const void* workspace, size_t workspace_bytes) {
  JPT_REQUIRE(M >= 1 && M <= kMaxM, JPT_EINVAL, "%s: M = %d rows, activation levels are kept for 1 .. %d rows", who, M, kMaxM);
  JPT_REQUIRE(K >= kTileK && K % kTileK == 0, JPT_EINVAL, "%s: K = %d must be a multiple of %d", who, K, kTileK);
  const size_t need = jpt_w8a16_linear_workspace_bytes(M, 1, K);
  JPT_REQUIRE(workspace && workspace_bytes >= need, JPT_EWORKSPACE, "%s: workspace of %zu bytes needed, %zu given", who, need,
              workspace_bytes);
  JPT_REQUIRE(aligned(workspace, 256), JPT_EALIGN, "%s: workspace must be 256-byte aligned", who);
  return 0;
}
}  // namespace
}  // namespace jpt

extern "C" int jpt_w8a16_linear(const void* x, const void* w, const void* w_scale, void* y, int M, int N, int K,
                                void* workspace, size_t workspace_bytes, void* stream) {
  return jpt_w8a16_linear_reporting(x, w, w_scale, y, M, N, K, workspace, workspace_bytes, nullptr, stream);
}

extern "C" int jpt_w8a16_linear_reporting(const void* x, const void* w, const void* w_scale, void* y, int M, int N, int K,
                                          void* workspace, size_t workspace_bytes, int32_t* status, void* stream) {
  JPT_REQUIRE(x && w && w_scale && y, JPT_EINVAL, "w8a16_linear: null tensor");
  JPT_REQUIRE(M >= 1, JPT_EINVAL, "w8a16_linear: M = %d rows", M);
  JPT_REQUIRE(N >= 1 && K >= kTileK && K % kTileK == 0, JPT_EINVAL, "w8a16_linear: K = %d must be a multiple of %d", K, kTileK);
  JPT_REQUIRE(aligned(x, 16) && aligned(w, 16) && aligned(y, 2), JPT_EALIGN, "w8a16_linear: x and w must be 16-byte aligned");
  const size_t need = jpt_w8a16_linear_workspace_bytes(M, N, K);
  JPT_REQUIRE(workspace && workspace_bytes >= need, JPT_EWORKSPACE, "w8a16_linear: workspace of %zu bytes needed, %zu given", need,
              workspace_bytes);
  JPT_REQUIRE(aligned(workspace, 256), JPT_EALIGN, "w8a16_linear: workspace must be 256-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (M > kMaxM) return launch_tiles<false>(x, w, w_scale, nullptr, nullptr, y, M, N, K, workspace, status, st);
  LevelsView lv = levels_view(workspace, M, K);
  if (status) lv.status = status;
  if (int rc = launch_levels(x, lv, M, K, st, true)) return rc;
  return launch_gemm(lv, w, w_scale, y, M, N, K, st, true);
}

extern "C" int jpt_w8a16_gate(const void* x, const void* w1, const void* w1_scale, const void* w3, const void* w3_scale, void* h, int M,
                              int N, int K, void* workspace, size_t workspace_bytes, void* stream) {
  return jpt_w8a16_gate_reporting(x, w1, w1_scale, w3, w3_scale, h, M, N, K, workspace, workspace_bytes, nullptr, stream);
}

extern "C" int jpt_w8a16_gate_reporting(const void* x, const void* w1, const void* w1_scale, const void* w3, const void* w3_scale, void* h,
                                        int M, int N, int K, void* workspace, size_t workspace_bytes, int32_t* status, void* stream) {
  JPT_REQUIRE(x && w1 && w1_scale && w3 && w3_scale && h, JPT_EINVAL, "w8a16_gate: null tensor");
  JPT_REQUIRE(M >= 1 && N >= 1 && K >= kTileK && K % kTileK == 0, JPT_EINVAL, "w8a16_gate: M = %d, K = %d (a multiple of %d)", M, K, kTileK);
  JPT_REQUIRE(aligned(x, 16) && aligned(w1, 16) && aligned(w3, 16), JPT_EALIGN, "w8a16_gate: x and the weights must be 16-byte aligned");
  const size_t need = jpt_w8a16_gate_workspace_bytes(M, N, K);
  JPT_REQUIRE(workspace && workspace_bytes >= need, JPT_EWORKSPACE, "w8a16_gate: workspace of %zu bytes needed, %zu given", need,
              workspace_bytes);
  JPT_REQUIRE(aligned(workspace, 256), JPT_EALIGN, "w8a16_gate: workspace must be 256-byte aligned");
  return launch_tiles<true>(x, w1, w1_scale, w3, w3_scale, h, M, N, K, workspace, status, static_cast<cudaStream_t>(stream));
}

extern "C" int jpt_w8a16_split_levels(const void* x, int M, int K, void* workspace, size_t workspace_bytes, void* stream) {
  JPT_REQUIRE(x && aligned(x, 16), JPT_EALIGN, "w8a16_split_levels: x must be 16-byte aligned");
  if (int rc = check_levels_args("w8a16_split_levels", M, K, workspace, workspace_bytes)) return rc;
  return launch_levels(x, levels_view(workspace, M, K), M, K, static_cast<cudaStream_t>(stream), true);
}

extern "C" int jpt_w8a16_linear_from_levels(void* workspace, size_t workspace_bytes, const void* w, const void* w_scale, void* y,
                                            int M, int N, int K, void* stream) {
  JPT_REQUIRE(w && w_scale && y && N >= 1, JPT_EINVAL, "w8a16_linear_from_levels: null tensor");
  JPT_REQUIRE(aligned(w, 16), JPT_EALIGN, "w8a16_linear_from_levels: w must be 16-byte aligned");
  if (int rc = check_levels_args("w8a16_linear_from_levels", M, K, workspace, workspace_bytes)) return rc;
  return launch_gemm(levels_view(workspace, M, K), w, w_scale, y, M, N, K, static_cast<cudaStream_t>(stream), false);
}

extern "C" int jpt_rmsnorm(const void* x, const void* weight, float eps, void* y, int M, int K, void* levels_workspace,
                           size_t workspace_bytes, void* stream) {
  JPT_REQUIRE(x && weight && y && M >= 1 && K >= 8 && K % 8 == 0, JPT_EINVAL, "rmsnorm: M = %d, K = %d (K must be a multiple of 8)", M, K);
  JPT_REQUIRE(aligned(x, 16) && aligned(weight, 16) && aligned(y, 16), JPT_EALIGN, "rmsnorm: tensors must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
  const __nv_bfloat16* wp = static_cast<const __nv_bfloat16*>(weight);
  if (!levels_workspace) {
    // (from two rows per SM on, rows of up to 8192 elements: below that a CTA per row has the shorter chain)
    if (M >= 296 && K <= 8192) {
      const dim3 grid((M + 3) / 4), block(128);
      if (K <= 4096)
        launch_after_previous(rmsnorm_rows_kernel<16>, grid, block, 0, st, xp, wp, eps, static_cast<__nv_bfloat16*>(y), M, K);
      else
        launch_after_previous(rmsnorm_rows_kernel<32>, grid, block, 0, st, xp, wp, eps, static_cast<__nv_bfloat16*>(y), M, K);
      return check_launch("rmsnorm_rows_kernel");
    }
    return launch_rows("rmsnorm_levels_kernel", rmsnorm_levels_kernel, M, row_parts(M, K), st, xp, wp, eps, static_cast<__nv_bfloat16*>(y),
                       nullptr, nullptr, nullptr, M, M, K);
  }
  if (int rc = check_levels_args("rmsnorm", M, K, levels_workspace, workspace_bytes)) return rc;
  const LevelsView lv = levels_view(levels_workspace, M, K);
  return launch_rows("rmsnorm_levels_kernel", rmsnorm_levels_kernel, lv.Mp, row_parts(lv.Mp, K), st, xp, wp, eps,
                     static_cast<__nv_bfloat16*>(y), lv.lev, lv.xs, lv.status, M, lv.Mp, K);
}

extern "C" int jpt_silu_mul(const void* a, const void* b, void* h, int M, int K, void* levels_workspace, size_t workspace_bytes,
                            void* stream) {
  JPT_REQUIRE(a && b && h && M >= 1 && K >= 8 && K % 8 == 0, JPT_EINVAL, "silu_mul: M = %d, K = %d (K must be a multiple of 8)", M, K);
  JPT_REQUIRE(aligned(a, 16) && aligned(b, 16) && aligned(h, 16), JPT_EALIGN, "silu_mul: tensors must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16* ap = static_cast<const __nv_bfloat16*>(a);
  const __nv_bfloat16* bp = static_cast<const __nv_bfloat16*>(b);
  if (!levels_workspace) {
    return launch_rows("silu_mul_levels_kernel", silu_mul_levels_kernel, M, row_parts(M, K), st, ap, bp, static_cast<__nv_bfloat16*>(h),
                       nullptr, nullptr, nullptr, M, M, K);
  }
  if (int rc = check_levels_args("silu_mul", M, K, levels_workspace, workspace_bytes)) return rc;
  const LevelsView lv = levels_view(levels_workspace, M, K);
  return launch_rows("silu_mul_levels_kernel", silu_mul_levels_kernel, lv.Mp, row_parts(lv.Mp, K), st, ap, bp,
                     static_cast<__nv_bfloat16*>(h), lv.lev, lv.xs, lv.status, M, lv.Mp, K);
}

extern "C" int jpt_w8a16_plan(int M, int N, int K, int row_parallel, const int* slots, int* plan) {
  JPT_REQUIRE(M >= 1 && M <= kMaxM && N >= 1 && K >= kTileK && K % kTileK == 0 && plan, JPT_EINVAL, "w8a16_plan: bad arguments");
  ClusterSlots given;
  if (slots) memcpy(&given, slots, sizeof(given));
  const GemmPlan p = plan_gemm(M, N, K, row_parallel != 0, slots ? given : device_slots());
  plan[0] = p.pair, plan[1] = p.split, plan[2] = p.tile, plan[3] = p.tiles, plan[4] = p.kb;
  return 0;
}

extern "C" size_t jpt_w8a16_tp_buffer_bytes(int N, int world) {
  if (N < 4 || N % 4 || world < 1 || world > 8 || (N + kTileN - 1) / kTileN > kTpMaxTiles) return 0;
  return kTpDataOffset + (size_t)2 * kMaxM * N * sizeof(float);
}

extern "C" int jpt_w8a16_linear_tp(const void* x, const void* w, const void* w_scale, void* y, int M, int N, int K, void* workspace,
                                   size_t workspace_bytes, const jpt_tp_sum* tp, void* stream) {
  JPT_REQUIRE(x && w && w_scale && y && tp, JPT_EINVAL, "w8a16_linear_tp: null argument");
  JPT_REQUIRE(N >= 4 && N % 4 == 0, JPT_EINVAL, "w8a16_linear_tp: N = %d must be a multiple of 4", N);
  JPT_REQUIRE(aligned(x, 16) && aligned(w, 16) && aligned(y, 8) && aligned(w_scale, 8), JPT_EALIGN,
              "w8a16_linear_tp: x and w must be 16-byte aligned, y and the scales 8-byte aligned");
  JPT_REQUIRE(tp->world >= 1 && tp->world <= 8 && tp->rank >= 0 && tp->rank < tp->world, JPT_EINVAL,
              "w8a16_linear_tp: rank %d of %d", tp->rank, tp->world);
  JPT_REQUIRE(tp->buffer_bytes >= jpt_w8a16_tp_buffer_bytes(N, tp->world) && jpt_w8a16_tp_buffer_bytes(N, tp->world) > 0, JPT_EWORKSPACE,
              "w8a16_linear_tp: receive buffers of %zu bytes are too small for N = %d on %d ranks", tp->buffer_bytes, N, tp->world);
  if (int rc = check_levels_args("w8a16_linear_tp", M, K, workspace, workspace_bytes)) return rc;
  TpArgs t;
  memset(&t, 0, sizeof(t));
  t.world = tp->world;
  t.rank = tp->rank;
  t.wait_cycles = tp->wait_cycles > 0 ? tp->wait_cycles : kWaitCyclesL;
  for (int r = 0; r < tp->world; ++r) {
    JPT_REQUIRE(tp->buffers[r], JPT_EINVAL, "w8a16_linear_tp: no buffer for rank %d", r);
    t.buffers[r] = static_cast<char*>(tp->buffers[r]);
  }
  t.status = reinterpret_cast<int*>(t.buffers[t.rank]);
  t.launch_counter = reinterpret_cast<unsigned*>(t.buffers[t.rank] + 8);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const LevelsView lv = levels_view(workspace, M, K);
  if (int rc = launch_levels(x, lv, M, K, st, true, t.launch_counter)) return rc;
  return launch_gemm(lv, w, w_scale, y, M, N, K, st, true, &t);
}

extern "C" int jpt_w8a16_tp_status(const jpt_tp_sum* tp, void* stream) {
  JPT_REQUIRE(tp && tp->buffers[tp->rank], JPT_EINVAL, "w8a16_tp_status: null buffer");
  int v = 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(&v, static_cast<const char*>(tp->buffers[tp->rank]), sizeof(v), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail((int)e, "w8a16_tp_status: %s", cudaGetErrorString(e));
  return v;
}
