// Prefill attention (many query rows per KV head, head_dim 128, bf16 q / K / V, an additive mask or none): tcgen05
// with both contractions out of tensor memory and TMA.  Covers dense_attention and flash_attention
// (jetstream_pt/attention_kernel.py:605-710) on the shapes of a prompt.
//
// Bound: compute (4 Hq D per score; the exponentials of the softmax cost about as much as the MMAs).
//
// Work item of a CTA: two tiles of 128 query rows of one KV head ("a" and "b": two grouped query heads at the same
// token block where the model groups heads, two consecutive token blocks otherwise), so that a K/V tile read from L2
// serves 256 rows and the tensor core works on one tile while the other one's 256 threads do their softmax (grids of one wave: see
// row_tile).  Tiles are
// made per query head through a tensor map with the caller's strides: a transposed view of the projection needs no copy.
// Items with the most K/V tiles under a causal mask start first.
//
//   warps 0-7, 8-15 softmax of tile a / b: thread = query row (TMEM lane) and half of the 128 keys; the two halves
//                   of a row exchange their maxima through shared memory, one barrier per K/V tile.  (One thread per
//                   whole row left two warps per scheduler and the chain from S to P was the time: 38.6 us for
//                   1024 tokens of 32 heads.)
//   warp 16         thread 0 requests Q once and K, V tiles through two rings of two 32 KB slots
//   warp 17         thread 0 issues the MMAs: S_t = Q_t K^T (shared x shared), O_t += P_t V (TMEM x shared)
//
// P lies over S in tensor memory (S: 128 fp32 columns; P: 64 columns of bf16 pairs for the leading part and 64 for
// the rest, so that the probabilities keep 17 bits; two MMAs per step).  Measured against fp64 over 24 causal prompts of
// 24 to 1024 tokens, relative error in the 2-norm and signed: 1.562775e-3 and -2.4e-6, the scalar kernel with fp32
// probabilities 1.562775e-3 and -2.2e-6 (both parts cut instead of rounded: 1.562789e-3 and -6.8e-6).  With the logits
// rounded to bf16 1.5635e-3 against 1.5621e-3: the fp32 sums of the tensor core (1.2e-7 of the rms) put a few more logits
// on the other side of a rounding boundary than those of the scalar kernel (5e-8).  S of the next K tile is issued
// behind the PV product that reads P: the tensor core takes them in order.
// The row maximum is raised lazily (when a tile's maximum is more than 2^8 above the reference in exp2 units): O
// is rescaled in tensor memory only then, and m, l that go out are those of the true maximum.
//
// An additive mask is classified beforehand, one byte per [128 x 128] tile: all zero (no mask work), all -inf (tile
// skipped), mixed (added value by value).  With up to kSmallK tiles per row every tile counts as mixed and that launch
// (2 us and more) is saved.  The values of masked keys may hold anything, NaN and infinities too (plain_rows).  Every wait is
// bounded; a CTA that gives up raises the workspace's status word.
#include <cuda.h>
#include <string.h>

#include <atomic>
#include <cmath>

#include "attention_tiles.cuh"

namespace jpt {
namespace {

constexpr int kDp = 128, kRowsP = 128, kKeysP = 128;
constexpr int kThreadsP = 576, kGroup = 256;  // threads in all, threads of a row tile
constexpr int kProducerP = 512, kIssuerP = 544;  // the threads that request tiles and issue MMAs
constexpr int kMaxKTiles = 512;  // K/V tiles of a row (65 536 tokens)
constexpr int kSmallK = 3;
constexpr uint32_t kTileBytes = 128 * 128 * 2;  // one bf16 tile: two halves of 64 dims, [128 x 128 B] each, swizzled
constexpr long long kWaitCyclesP = 400000000ll;  // about a fifth of a second
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLazy = 8.f;  // P may reach 2^8 before O is rescaled

enum : uint8_t { kClsZero = 0, kClsMixed = 1, kClsSkip = 2 };

struct __align__(1024) SmemP {
  uint8_t q[2][kTileBytes];
  uint8_t k[2][kTileBytes];
  uint8_t v[2][kTileBytes];
  uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_ready[2], o_done;
  uint32_t tmem_base;
  int n_tiles;
  volatile int dead;
  float vs[2][2][kKeysP];          // scales of the K/V tile, per row tile and parity of the K/V tile
  float ks[2][2][kKeysP];
  float half_max[2][2][2][kRowsP]; // [row tile][parity][half][row]
  uint16_t list[kMaxKTiles];       // K/V tiles with work for a or b, in order
  uint8_t cls[2][kMaxKTiles];      // class of the list's entry for tile a and b
};

struct PrefillMaps {
  CUtensorMap q, k, v, o;
};
struct PrefillGeom {
  const uint8_t* cls;  // null: every tile is mixed (additive mask) or zero (no mask)
  int n_rows_t;        // row blocks of 128 per query head
  int n_k;             // K/V tiles
  int pairs;           // items per KV head
  int fold;            // how row tiles make items: see row_tile
  int cls_rows, cls_heads, cls_batch;  // extents of the class table (1 where the mask broadcasts)
  int mask_vec, mask_pairs;  // mask rows can be read 16, 4 bytes at a time
  int64_t q_b, q_h, q_t;     // strides of the queries
};

// Row tile t (0: a, 1: b) of item `item` of a KV head: token block index / rep, grouped query head index % rep.  Under a causal mask a
// tile has as many K/V tiles as blocks up to its own.
// Folded: the longest with the shortest, the second longest with the second shortest, ..., so that every item has about
// as much work; for grids of one wave, whose time is that of the longest item (1024 tokens, 32 / 8 heads: 37.5 -> 35.1 us;
// a step of one tile alone takes nearly as long as one of two, so two blocks of tokens gain nothing).  Else neighbours, the longest
// items first, which fill up the end of several waves: items of one length would take whole waves.
template <bool kFold>
__device__ __forceinline__ int row_tile(const PrefillGeom& g, int rep, int item, int t, bool* have) {
  const int tiles = g.n_rows_t * rep;
  if constexpr (kFold) {
    *have = t == 0 || item < tiles - 1 - item;
    return t == 0 ? tiles - 1 - item : item;
  } else {
    const int idx = 2 * (g.pairs - 1 - item) + t;
    *have = idx < tiles;
    return idx;
  }
}

__device__ __forceinline__ uint32_t smem_u32p(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init_p(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32p(bar)), "r"(count));
}
__device__ __forceinline__ bool mbar_probe_p(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.b32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(20000u)  // (may sleep for up to 20 us)
      : "memory");
  return ok != 0;
}
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, volatile int* dead) {
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 16; ++i) {
      if (mbar_probe_p(bar, parity)) return true;
    }
    if (*dead || clock64() - t0 > kWaitCyclesP) {
      *dead = 1;
      return false;
    }
  }
}
// Bounded wait for the phase with the given parity; false when it (or another warp of the CTA) gave up.
__device__ __forceinline__ bool mbar_wait_p(uint64_t* b, uint32_t parity, SmemP& sm) {
  const uint32_t bar = smem_u32p(b);
  return mbar_probe_p(bar, parity) || mbar_wait_slow(bar, parity, &sm.dead);
}
__device__ __forceinline__ void mbar_arrive_p(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32p(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_p(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32p(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void commit_p(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32p(bar)) : "memory");
}
// one bf16 tile (two boxes of 64 dims x 128 rows)
__device__ __forceinline__ void tma_tile(const void* dst, const CUtensorMap* map, int row, int h, int b, uint64_t* bar) {
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
            smem_u32p(dst) + half * (kTileBytes / 2)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(half * 64), "r"(row), "r"(h), "r"(b), "r"(smem_u32p(bar))
        : "memory");
  }
}
// Shared-memory descriptors: the low word carries the start address (16-byte units) and the leading byte offset, the
// high word the stride of 1024 bytes between 8-row groups, the version and the 128-byte swizzle.  K-major operands (Q, K)
// do not use the leading offset; V as [token][dim] is MN-major, its 64-dim halves lie half a tile apart.
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr) {
  return ((addr >> 4) & 0x3FFF) | (uint32_t)((kTileBytes / 2) >> 4) << 16;
}
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(r));
  return r != 0;
}
// D fp32, A and B bf16, M = 128, N = 128
constexpr uint32_t kIdescQk = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t kIdescPv = kIdescQk | (1u << 16);  // B is MN-major

__device__ __forceinline__ void mma_ss(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}\n" ::"r"(d),
      "r"(a_lo), "r"(b_lo), "r"(kDescHi), "r"(kIdescQk), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}\n" ::"r"(d),
      "r"(a), "r"(b_lo), "r"(kDescHi), "r"(kIdescPv), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr));
}
__device__ __forceinline__ void tmem_st32(uint32_t addr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};\n" ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
        "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
        "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]),
        "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};\n" ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
        "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before_p() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_p() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ float ex2p(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float lo_f32(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float hi_f32(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
__device__ __forceinline__ uint32_t mul2(uint32_t x, uint32_t y) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(y));
  return r;
}
__device__ __forceinline__ uint32_t add2(uint32_t x, uint32_t y) {
  uint32_t r;
  asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(y));
  return r;
}
__device__ __forceinline__ uint32_t max2(uint32_t x, uint32_t y) {
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(y));
  return r;
}
// two fp32 values in one 64-bit register, and the packed arithmetic on them
__device__ __forceinline__ uint64_t pack_f32(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32(uint64_t x, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x));
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t x, uint64_t y) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t x, uint64_t y) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  return r;
}
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 256;" ::"r"(1 + group) : "memory"); }
// barrier of the group's 256 threads; whether `pred` holds in all of them
__device__ __forceinline__ bool group_all(int group, bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %2, 0;\n\tbarrier.cta.red.and.pred q, %1, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"(1 + group), "r"((uint32_t)pred)
      : "memory");
  return r != 0;
}

// ---------------------------------------------------------------- mask classes
// One CTA per [128 rows x 128 keys] tile of the mask: all zero, all -inf, or mixed.  Reads the mask once (the bound).
__global__ void __launch_bounds__(256) mask_class_kernel(AttnArgs a, uint8_t* cls, int rows_per_head, int cls_heads, int vec) {
  grid_dependency_wait();
  grid_dependency_trigger();
  const int j = blockIdx.x, tb = blockIdx.y, r = blockIdx.z % cls_heads, b = blockIdx.z / cls_heads;
  const int t0 = tb * kRowsP, s0 = j * kKeysP;
  const int nr = min(kRowsP, rows_per_head - t0), nc = min(kKeysP, a.S - s0);
  const uint16_t* m = static_cast<const uint16_t*>(a.mask) + (int64_t)b * a.mk_b + ((int64_t)r * rows_per_head + t0) * a.mk_r + s0;
  bool zero = true, inf = true;
  if (vec && nc == kKeysP) {
    for (int i = threadIdx.x; i < nr * 16; i += 256) {
      const uint4 w = __ldg(reinterpret_cast<const uint4*>(m + (int64_t)(i >> 4) * a.mk_r) + (i & 15));
      const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        zero = zero && (x[e] & 0x7fff7fffu) == 0u;
        inf = inf && x[e] == 0xff80ff80u;
      }
    }
  } else {
    for (int i = threadIdx.x; i < nr * kKeysP; i += 256) {
      const int c = i & (kKeysP - 1);
      if (c < nc) {
        const uint32_t x = m[(int64_t)(i >> 7) * a.mk_r + c];
        zero = zero && (x & 0x7fffu) == 0u;
        inf = inf && x == 0xff80u;
      }
    }
  }
  zero = __syncthreads_and(zero);
  inf = __syncthreads_and(inf);
  if (threadIdx.x == 0)
    cls[(((int64_t)b * cls_heads + r) * gridDim.y + tb) * gridDim.x + j] = zero ? kClsZero : inf ? kClsSkip : kClsMixed;
}

// The products of one row (TMEM lane) with 64 keys turned into final logits in place, as fp32: scaled, rounded where the
// reference rounds, the mask row added; keys from `valid` on get -inf.  ks: the tile's K scales, read when `scaled`.
template <bool kRound, bool kScale>
__device__ __noinline__ void final_logits(uint32_t tl, const AttnArgs& a, const float* ks, bool scaled, const uint16_t* mask,
                                          int valid, bool mask_vec) {
  const float mul = a.sm_scale;
#pragma unroll 1
  for (int q = 0; q < 2; ++q) {
    uint32_t v[32], mk[16];
    tmem_ld32(tl + 32 * q, v);
    if (mask && mask_vec && valid >= kKeysP / 2) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(mask + 32 * q) + e);
        mk[4 * e] = w.x, mk[4 * e + 1] = w.y, mk[4 * e + 2] = w.z, mk[4 * e + 3] = w.w;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int p = 32 * q + 2 * e;
        const uint32_t x0 = p >= valid ? 0xff80u : mask ? (uint32_t)__ldg(mask + p) : 0u;
        const uint32_t x1 = p + 1 >= valid ? 0xff80u : mask ? (uint32_t)__ldg(mask + p + 1) : 0u;
        mk[e] = x0 | (x1 << 16);
      }
    }
    tmem_wait_ld();
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const float k0 = kScale && scaled ? ks[32 * q + 2 * e] : 1.f, k1 = kScale && scaled ? ks[32 * q + 2 * e + 1] : 1.f;
      if constexpr (kRound) {
        uint32_t x = pack_bf16(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
        x = pack_bf16(lo_f32(x) * mul, hi_f32(x) * mul);
        if (kScale) x = pack_bf16(lo_f32(x) * k0, hi_f32(x) * k1);
        x = add2(x, mk[e]);
        v[2 * e] = __float_as_uint(lo_f32(x)), v[2 * e + 1] = __float_as_uint(hi_f32(x));
      } else {
        v[2 * e] = __float_as_uint(fmaf(__uint_as_float(v[2 * e]) * mul, k0, lo_f32(mk[e])));
        v[2 * e + 1] = __float_as_uint(fmaf(__uint_as_float(v[2 * e + 1]) * mul, k1, hi_f32(mk[e])));
      }
    }
    tmem_st32(tl + 32 * q, v);
  }
  tmem_wait_st();
}

// Bits of the keys a row must not see among its 64: lane r of the warp gets row r's (lo: keys 2 e at bit e, hi: keys
// 2 e + 1).  The warp reads one row after the other, 128 bytes at a time.  `warp_mask`: the warp's first row at the
// thread half's first key, null without a mask; rows and keys beyond `rows`, `valid` are not read.  False when the mask
// holds anything but 0 and -inf.
// The result: {lo, hi, 1 if so, 0}.
__device__ __noinline__ uint4 masked_bits(const uint16_t* warp_mask, int64_t mk_r, int rows, int valid, bool pairs) {
  const int lane = threadIdx.x & 31;
  const bool in0 = 2 * lane < valid, in1 = 2 * lane + 1 < valid;
  const uint32_t out_lo = __ballot_sync(0xffffffffu, !in0), out_hi = __ballot_sync(0xffffffffu, !in1);
  uint32_t lo = out_lo, hi = out_hi;
  bool odd = false;
  auto fold = [&](uint32_t x, int r) {
    const bool inf0 = (x & 0xffffu) == 0xff80u, inf1 = (x >> 16) == 0xff80u;
    odd = odd || !(inf0 || (x & 0x7fffu) == 0u) || !(inf1 || (x & 0x7fff0000u) == 0u);
    const uint32_t b0 = __ballot_sync(0xffffffffu, inf0), b1 = __ballot_sync(0xffffffffu, inf1);
    if (lane == r) lo = out_lo | b0, hi = out_hi | b1;
  };
  if (warp_mask && pairs && valid >= kKeysP / 2 && rows >= 32) {
    // (eight rows in flight, in a short loop: this code runs once per item, and fetching its instructions is most of
    // its time; one row after the other cost 17 000 cycles a tile)
#pragma unroll 1
    for (int r0 = 0; r0 < 32; r0 += 8) {
      uint32_t x[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) x[r] = __ldg(reinterpret_cast<const uint32_t*>(warp_mask + (int64_t)(r0 + r) * mk_r) + lane);
#pragma unroll
      for (int r = 0; r < 8; ++r) fold(x[r], r0 + r);
    }
  } else if (warp_mask) {
#pragma unroll 1
    for (int r0 = 0; r0 < 32 && r0 < rows; r0 += 8) {
      uint32_t x[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const uint16_t* p = warp_mask + (int64_t)(r0 + r) * mk_r + 2 * lane;
        const bool row = r0 + r < rows;
        const uint32_t x0 = row && in0 ? (uint32_t)__ldg(p) : 0u, x1 = row && in1 ? (uint32_t)__ldg(p + 1) : 0u;
        x[r] = x0 | (x1 << 16);
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) fold(x[r], r0 + r);
    }
  }
  return make_uint4(lo, hi, __any_sync(0xffffffffu, odd) ? 0u : 1u, 0u);
}

// Rows whose accumulator is not finite, once more with plain arithmetic: the calling warp's half (64 dims) of the rows `rows`
// (bits), a lane each, 32 dims at a time.  The tensor core multiplies every V row of a tile, with a probability of zero where
// the key is masked and in two parts elsewhere, so that one infinite or NaN value of V turns rows into NaN that must not see
// it, and an infinite one that they do see as well.  Here a masked key is left out and the others are multiplied by the whole
// probability, as in the scalar kernel.  When every row needs it, a causal prompt of 1024 tokens and 32 / 8 heads takes 3.9 ms
// (the scalar kernel 6.4 ms), one of 128 tokens 0.48 ms (0.13 ms).  Everything but the rows follows from the indexes again: kept
// for this call, the values cost the main path registers (1 us of 38).
template <bool kRound, bool kScale>
__device__ __noinline__ void plain_rows(const AttnArgs& a, const PrefillGeom& g, unsigned rows) {
  extern __shared__ __align__(1024) uint8_t smem_raw_p[];
  SmemP& sm = *reinterpret_cast<SmemP*>(smem_raw_p);
  constexpr int kKeys = 4, kDims = 32;  // at a time
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = warp >> 3, half = (warp >> 2) & 1;
  const int rep = a.Hq / a.Hkv, heads = a.B * a.Hkv, bh = (int)blockIdx.x % heads, b = bh / a.Hkv, hkv = bh % a.Hkv;
  bool have;
  const int item = (int)blockIdx.x / heads;
  const int idx = g.fold ? row_tile<true>(g, rep, item, t, &have) : row_tile<false>(g, rep, item, t, &have), hq = hkv * rep + idx % rep;
  const int token = min(idx / rep * kRowsP + (warp & 3) * 32 + lane, a.Tq - 1);
  // (all tiles of the item are done: the rings are free.  The query rows read once a key from global memory, a line per lane,
  // were most of the time.)
  uint8_t *q_rows = (half ? sm.v[t] : sm.k[t]) + (warp & 3) * 32 * 256, *out = sm.q[t] + half * (kTileBytes / 2) + (warp & 3) * 32 * 128;
  const uint4* q = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.q) + b * g.q_b + hq * g.q_h + token * g.q_t);
  const int64_t head = (int64_t)b * a.kv_b + (int64_t)hkv * a.kv_h;
  const __nv_bfloat16 *k = static_cast<const __nv_bfloat16*>(a.k) + head, *v = static_cast<const __nv_bfloat16*>(a.v) + head + 64 * half;
  const __nv_bfloat16* mask = nullptr;
  if (a.mask_mode == JPT_MASK_ADD)
    mask = static_cast<const __nv_bfloat16*>(a.mask) + b * a.mk_b + ((int64_t)(hq % rep) * a.Tq + token) * a.mk_r;
#pragma unroll
  for (int c = 0; c < kDp / 8; ++c) *reinterpret_cast<uint4*>(q_rows + lane * 256 + ((c ^ (lane & 15)) * 16)) = __ldg(q + c);
#pragma unroll 1
  for (int dim0 = 0; dim0 < 64; dim0 += kDims, v += kDims) {
    float m = -INFINITY, l = 0.f, acc[kDims];
#pragma unroll
    for (int d = 0; d < kDims; ++d) acc[d] = 0.f;
#pragma unroll 1
    for (int p0 = 0; p0 < a.S; p0 += kKeys) {
      float s[kKeys];
#pragma unroll
      for (int j = 0; j < kKeys; ++j) s[j] = 0.f;
#pragma unroll 4
      for (int c = 0; c < kDp / 8; ++c) {
        const uint4 x = *reinterpret_cast<const uint4*>(q_rows + lane * 256 + ((c ^ (lane & 15)) * 16));
        const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int j = 0; j < kKeys; ++j) {
          const uint4 y = __ldg(reinterpret_cast<const uint4*>(k + (int64_t)min(p0 + j, a.S - 1) * a.kv_s) + c);
          const uint32_t yw[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) s[j] = fmaf(hi_f32(xw[e]), hi_f32(yw[e]), fmaf(lo_f32(xw[e]), lo_f32(yw[e]), s[j]));
        }
      }
      float top = m;
#pragma unroll
      for (int j = 0; j < kKeys; ++j) {
        const int p = min(p0 + j, a.S - 1);
        const float ks = kScale ? load_scale(a.k_scale, (int64_t)b * a.sc_b + (int64_t)p * a.sc_s, a.scale_is_f32) : 1.f;
        const float add = mask ? __bfloat162float(mask[p]) : 0.f;
        s[j] = kRound ? rounded_logit(s[j], __frcp_rn(a.sm_scale), ks, kScale, add) : s[j] * a.sm_scale * ks + add;
        if (p0 + j >= a.S) s[j] = -INFINITY;
        top = fmaxf(top, s[j]);
      }
      if (top > m) {
        const float f = expf(m - top);
        m = top, l *= f;
#pragma unroll
        for (int d = 0; d < kDims; ++d) acc[d] *= f;
      }
#pragma unroll 1
      for (int j = 0; j < kKeys; ++j) {
        float sj = s[0];
#pragma unroll
        for (int i = 1; i < kKeys; ++i) sj = i == j ? s[i] : sj;
        if (sj == -INFINITY) continue;
        float pr = expf(sj - m);
        l += pr;
        if (kScale) pr *= load_scale(a.v_scale, (int64_t)b * a.sc_b + (int64_t)(p0 + j) * a.sc_s, a.scale_is_f32);
        const uint4* row = reinterpret_cast<const uint4*>(v + (int64_t)(p0 + j) * a.kv_s);
#pragma unroll
        for (int c = 0; c < kDims / 8; ++c) {
          const uint4 y = __ldg(row + c);
          const uint32_t yw[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            acc[8 * c + 2 * e] = fmaf(pr, lo_f32(yw[e]), acc[8 * c + 2 * e]);
            acc[8 * c + 2 * e + 1] = fmaf(pr, hi_f32(yw[e]), acc[8 * c + 2 * e + 1]);
          }
        }
      }
    }
    if ((rows >> lane) & 1u) {
#pragma unroll
      for (int c = 0; c < kDims / 8; ++c) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = l > 0.f ? pack_bf16(acc[8 * c + 2 * e] / l, acc[8 * c + 2 * e + 1] / l) : 0u;
        *reinterpret_cast<uint4*>(out + lane * 128 + (((dim0 / 8 + c) ^ lane) & 7) * 16) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
}

// ---------------------------------------------------------------- the kernel
// kRound: dense_attention's logit chain with a bf16 rounding after every step; kScale: per-token K and V scales; kFold: see row_tile (in
// the geometry alone the choice cost short prompts 3 to 5 %: the main path's registers are all in use).
template <bool kRound, bool kScale, bool kFold>
__global__ void __launch_bounds__(kThreadsP, 1)
    prefill_attention_kernel(const __grid_constant__ PrefillMaps maps, const __grid_constant__ AttnArgs a,
                             const __grid_constant__ PrefillGeom g, int* status) {
  extern __shared__ __align__(1024) uint8_t smem_raw_p[];
  SmemP& sm = *reinterpret_cast<SmemP*>(smem_raw_p);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((smem_u32p(smem_raw_p) & 1023u) != 0u) {  // (the swizzled tiles need it; the launch has no static shared memory)
    if (tid == 0) atomicExch(status, 2);
    return;
  }
  const int rep = a.Hq / a.Hkv;
  const int heads = a.B * a.Hkv;
  const int bh = (int)blockIdx.x % heads, b = bh / a.Hkv, hkv = bh % a.Hkv;
  // the item's row tiles: query head and token block of a and b
  int hq[2], tb[2];
  bool have[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int idx = row_tile<kFold>(g, rep, (int)blockIdx.x / heads, t, &have[t]);
    tb[t] = idx / rep;
    hq[t] = hkv * rep + idx % rep;
  }

  if (tid == kProducerP) {
    mbar_init_p(&sm.q_full, 1);
    mbar_init_p(&sm.o_done, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init_p(&sm.k_full[i], 1);
      mbar_init_p(&sm.k_empty[i], 1);
      mbar_init_p(&sm.v_full[i], 1);
      mbar_init_p(&sm.v_empty[i], 1);
      mbar_init_p(&sm.s_full[i], 1);
      mbar_init_p(&sm.p_ready[i], kGroup);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sm.dead = 0;
  }
  if (warp == kIssuerP / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32p(&sm.tmem_base)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    fence_before_p();
  }
  grid_dependency_wait();
  grid_dependency_trigger();
  // ---- the K/V tiles with work, in order (one warp)
  if (warp == 0) {
    int count = 0;
    const uint8_t* row[2] = {nullptr, nullptr};
    if (g.cls) {
#pragma unroll
      for (int t = 0; t < 2; ++t)
        row[t] = g.cls + (((int64_t)(g.cls_batch > 1 ? b : 0) * g.cls_heads + (g.cls_heads > 1 ? hq[t] % rep : 0)) * g.cls_rows +
                          (g.cls_rows > 1 ? tb[t] : 0)) * g.n_k;
    }
    for (int j0 = 0; j0 < g.n_k; j0 += 32) {
      const int j = j0 + lane;
      uint8_t c[2] = {kClsSkip, kClsSkip};
      if (j < g.n_k) {
#pragma unroll
        for (int t = 0; t < 2; ++t)
          if (have[t]) c[t] = g.cls ? row[t][j] : (a.mask_mode == JPT_MASK_ADD ? (uint8_t)kClsMixed : (uint8_t)kClsZero);
      }
      const bool use = c[0] != kClsSkip || c[1] != kClsSkip;
      const unsigned votes = __ballot_sync(0xffffffffu, use);
      if (use) {
        const int at = count + __popc(votes & ((1u << lane) - 1u));
        sm.list[at] = (uint16_t)j;
        sm.cls[0][at] = c[0];
        sm.cls[1][at] = c[1];
      }
      count += __popc(votes);
    }
    if (lane == 0) sm.n_tiles = count;
  }
  __syncthreads();
  fence_after_p();
  const uint32_t tmem = sm.tmem_base;
  const int n = sm.n_tiles;

  if (tid == kProducerP && n > 0) {
    // ---- producer
    mbar_expect_p(&sm.q_full, have[1] ? 2 * kTileBytes : kTileBytes);
#pragma unroll
    for (int t = 0; t < 2; ++t)
      if (have[t]) tma_tile(sm.q[t], &maps.q, tb[t] * kRowsP, hq[t], b, &sm.q_full);
    for (int i = 0; i < n; ++i) {
      const int s = i & 1;
      const uint32_t par = (uint32_t)((i >> 1) - 1) & 1u;
      if (i >= 2 && !mbar_wait_p(&sm.k_empty[s], par, sm)) break;
      mbar_expect_p(&sm.k_full[s], kTileBytes);
      tma_tile(sm.k[s], &maps.k, sm.list[i] * kKeysP, hkv, b, &sm.k_full[s]);
      if (i >= 2 && !mbar_wait_p(&sm.v_empty[s], par, sm)) break;
      mbar_expect_p(&sm.v_full[s], kTileBytes);
      tma_tile(sm.v[s], &maps.v, sm.list[i] * kKeysP, hkv, b, &sm.v_full[s]);
    }
    if (sm.dead) {  // (gave up: requests in flight get their time before the CTA leaves)
      const long long t0 = clock64();
      while (clock64() - t0 < 2000000) {
      }
    }
  } else if (warp == kIssuerP / 32 && n > 0) {
    // ---- MMA issue: the whole warp walks the list, one elected thread issues (a branch on the thread index makes the
    // compiler treat descriptors as per-thread values and move each into uniform registers)
    const bool elected = elect_one();
    bool ok = mbar_wait_p(&sm.q_full, 0, sm);
    uint32_t cnt[2] = {0, 0};  // products P V issued so far per tile
    const uint32_t q_lo = desc_lo(smem_u32p(sm.q[0])), k_lo = desc_lo(smem_u32p(sm.k[0])), v_lo = desc_lo(smem_u32p(sm.v[0]));
    auto qk = [&](int t, int i) {
      if (elected) {
        const uint32_t qa = q_lo + (uint32_t)t * (kTileBytes >> 4), ka = k_lo + (uint32_t)(i & 1) * (kTileBytes >> 4);
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          const uint32_t off = ((uint32_t)((s >> 2) * (kTileBytes / 2) + (s & 3) * 32)) >> 4;
          mma_ss(tmem + (uint32_t)(t * 256), qa + off, ka + off, s > 0);
        }
        commit_p(&sm.s_full[t]);
      }
    };
    ok = ok && mbar_wait_p(&sm.k_full[0], 0, sm);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      fence_after_p();
#pragma unroll
      for (int t = 0; t < 2; ++t)
        if (sm.cls[t][0] != kClsSkip) qk(t, 0);
      if (elected) commit_p(&sm.k_empty[0]);
    }
    for (int i = 0; i < n && ok; ++i) {
      ok = mbar_wait_p(&sm.v_full[i & 1], (uint32_t)(i >> 1) & 1u, sm);
      if (ok && i + 1 < n) ok = mbar_wait_p(&sm.k_full[(i + 1) & 1], (uint32_t)((i + 1) >> 1) & 1u, sm);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      fence_after_p();
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (ok && sm.cls[t][i] != kClsSkip) {
          ok = __all_sync(0xffffffffu, mbar_wait_p(&sm.p_ready[t], cnt[t] & 1u, sm));
          fence_after_p();
          if (ok) {
            if (elected) {
              const uint32_t p = tmem + (uint32_t)(t * 256), o = p + 128, va = v_lo + (uint32_t)(i & 1) * (kTileBytes >> 4);
#pragma unroll
              for (int s = 0; s < 16; ++s)  // (the leading parts, then the rests)
                mma_ts(o, p + (uint32_t)(8 * s), va + (uint32_t)((s & 7) * (2048 >> 4)), (s > 0 || cnt[t] > 0) ? 1u : 0u);
            }
            ++cnt[t];
          }
        }
        // S of the next tile goes over the P just read: the tensor core takes the two in order
        if (ok && i + 1 < n && sm.cls[t][i + 1] != kClsSkip) qk(t, i + 1);
      }
      if (!ok) break;
      if (elected) {
        if (i + 1 < n) commit_p(&sm.k_empty[(i + 1) & 1]);
        commit_p(&sm.v_empty[i & 1]);
      }
    }
    if (elected) commit_p(&sm.o_done);
  } else if (warp < 16) {
    // ---- softmax of tile t: one query row and 64 keys per thread
    const int t = warp >> 3, half = (warp >> 2) & 1, row_in = tid & 127;
    const uint32_t tl = tmem + (uint32_t)(t * 256) + ((uint32_t)((warp & 3) * 32) << 16);  // S, P and behind them O
    const uint32_t sl = tl + (uint32_t)(64 * half);                                         // this thread's keys
    const int trow = (t ? tb[1] : tb[0]) * kRowsP + row_in;  // token of the row
    const int my_hq = t ? hq[1] : hq[0];
    // this row's mask at this thread's half of the keys, and the warp's first row
    const uint16_t *mrow = nullptr, *mwarp = nullptr;
    const int wrow = (t ? tb[1] : tb[0]) * kRowsP + (warp & 3) * 32;
    if (a.mask_mode == JPT_MASK_ADD) {
      const uint16_t* base = static_cast<const uint16_t*>(a.mask) + (int64_t)b * a.mk_b + (int64_t)(my_hq % rep) * a.Tq * a.mk_r + 64 * half;
      mrow = base + (int64_t)min(trow, a.Tq - 1) * a.mk_r;
      mwarp = base + (int64_t)min(wrow, a.Tq - 1) * a.mk_r;
    }
    float m_ref = -INFINITY, m_true = -INFINITY, l = 0.f;
    uint32_t cnt = 0;
    bool ok = true, scaled = false;
    // a scale of list entry i (lower half of the threads: K, upper half: V)
    auto scale_of = [&](int i) {
      const int p = sm.list[i] * kKeysP + row_in;
      return p < a.S ? load_scale(half ? a.v_scale : a.k_scale, (int64_t)b * a.sc_b + (int64_t)p * a.sc_s, a.scale_is_f32) : 1.f;
    };
    auto keep_scale = [&](float x, uint32_t par) { (half ? sm.vs : sm.ks)[t][par][row_in] = x; };
    auto next_of = [&](int i) {
      while (i < n && sm.cls[t][i] == kClsSkip) ++i;
      return i;
    };
    int i = next_of(0);
    if constexpr (kScale) {
      if (i < n) {
        const float x = scale_of(i);
        keep_scale(x, 0);
        scaled = !group_all(t, x == 1.f);  // (an unquantised prefill has unit scales)
      }
    }
    while (i < n) {
      const uint8_t c = sm.cls[t][i];
      const int s0 = sm.list[i] * kKeysP, nxt = next_of(i + 1);
      const uint32_t par = cnt & 1u;
      float next_scale = 1.f;
      if constexpr (kScale) {
        if (nxt < n) next_scale = scale_of(nxt);
      }
      // (after a wait that gave up the later ones return at once: the loop runs to its end, so that the group's
      // barriers are met by all of its threads)
      ok = mbar_wait_p(&sm.s_full[t], par, sm) && ok;
      __syncwarp();
      fence_after_p();
      // Keys that the row must not see (0 / -inf masks, keys behind the last one) are struck out of the logits below.  A
      // tile with other mask values or with scales to multiply by first turns its products into final logits in tensor
      // memory, in a function of its own: spelled out inside the main path these cases cost every tile their
      // predicated instructions (54 instead of 39 us for 1024 tokens of 32 heads).
      const int valid = a.S - s0 - 64 * half;
      float mul = a.sm_scale;
      uint32_t out_lo = 0u, out_hi = 0u;
      bool strike = false;
      if (c == kClsMixed || valid < kKeysP / 2 || (kScale && scaled)) {
        const uint16_t* mw = c == kClsMixed ? mwarp + s0 : nullptr;
        const uint4 bits = masked_bits(mw, a.mk_r, a.Tq - wrow, valid, g.mask_pairs != 0);
        out_lo = bits.x, out_hi = bits.y, strike = bits.z != 0u;
        if (!strike || (kScale && scaled)) {
          final_logits<kRound, kScale>(sl, a, sm.ks[t][par] + 64 * half, kScale && scaled, c == kClsMixed ? mrow + s0 : nullptr,
                                       valid, g.mask_vec != 0);
          mul = 1.f;
          strike = false;
        }
      }
      // logits of the row: packed pairs of bf16 (kRound) or fp32
      uint32_t lg[kRound ? 32 : 64];
      float mt;
      {
        const uint64_t mul2x = pack_f32(mul, mul);
        uint32_t mx = 0xff80ff80u;
        float mxf = -INFINITY;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint32_t v[32];  // (both halves at once would not fit the 96 registers of a thread)
          tmem_ld32(sl + 32 * q, v);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float d0 = __uint_as_float(v[2 * e]), d1 = __uint_as_float(v[2 * e + 1]);
            float f0, f1;
            if constexpr (kRound) {
              uint32_t x = pack_bf16(d0, d1);  // bf16(q . k)
              unpack_f32(mul_f32x2(pack_f32(lo_f32(x), hi_f32(x)), mul2x), f0, f1);
              x = pack_bf16(f0, f1);  // bf16(. / sqrt(D))
              mx = max2(mx, x);
              lg[16 * q + e] = x;
            } else {
              unpack_f32(mul_f32x2(pack_f32(d0, d1), mul2x), f0, f1);
              mxf = fmaxf(mxf, fmaxf(f0, f1));
              lg[(32 * q + 2 * e) & (kRound ? 31 : 63)] = __float_as_uint(f0);
              lg[(32 * q + 2 * e + 1) & (kRound ? 31 : 63)] = __float_as_uint(f1);
            }
          }
        }
        if (strike) {
          mx = 0xff80ff80u;
          mxf = -INFINITY;
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            if constexpr (kRound) {
              uint32_t x = lg[e];
              if ((out_lo >> e) & 1u) x = (x & 0xffff0000u) | 0xff80u;
              if ((out_hi >> e) & 1u) x = (x & 0xffffu) | 0xff800000u;
              lg[e] = x;
              mx = max2(mx, x);
            } else {
              if ((out_lo >> e) & 1u) lg[(2 * e) & (kRound ? 31 : 63)] = 0xff800000u;
              if ((out_hi >> e) & 1u) lg[(2 * e + 1) & (kRound ? 31 : 63)] = 0xff800000u;
              mxf = fmaxf(mxf, fmaxf(__uint_as_float(lg[(2 * e) & (kRound ? 31 : 63)]),
                                     __uint_as_float(lg[(2 * e + 1) & (kRound ? 31 : 63)])));
            }
          }
        }
        mt = kRound ? fmaxf(lo_f32(mx), hi_f32(mx)) : mxf;
      }
      // the row's maximum; every thread of the tile has also read its part of S behind this barrier: P may go over it
      sm.half_max[t][par][half][row_in] = mt;
      // (S of this tile is there, so every thread has handed over its P of the last tile and is done with its scales)
      if constexpr (kScale) keep_scale(next_scale, par ^ 1u);
      fence_before_p();
      const bool next_ones = group_all(t, next_scale == 1.f);
      fence_after_p();
      const bool scaled_now = scaled;
      scaled = !next_ones;
      mt = fmaxf(mt, sm.half_max[t][par][half ^ 1][row_in]);
      m_true = fmaxf(m_true, mt);
      // raise the reference maximum: on the first tile, later only where P would leave its range
      float m_new = m_ref;
      if (m_ref == -INFINITY || (mt - m_ref) * kLog2e > kLazy) m_new = fmaxf(m_ref, mt);
      const bool raise = m_new > m_ref && cnt > 0;
      if (__any_sync(0xffffffffu, raise)) {
        // (S of this tile is there, so the products issued before it are complete: O is at rest)
        const float f = raise ? ex2p((m_ref - m_new) * kLog2e) : 1.f;
        l *= f;
#pragma unroll 1
        for (int q = 0; q < 2; ++q) {
          uint32_t v[32];
          tmem_ld32(tl + 128 + 64 * half + 32 * q, v);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * f);
          tmem_st32(tl + 128 + 64 * half + 32 * q, v);
        }
      }
      m_ref = m_new;
      // The reference maximum is subtracted before the product with log2 e: one fused step x log2 e - (m_ref log2 e) carries the
      // rounding of the second product, which for finite masks of large magnitude (-1e10, the lowest bf16) exceeds the range
      // of the exponential.
      const float off = m_ref == -INFINITY ? 0.f : m_ref;
      const uint64_t l2e = pack_f32(kLog2e, kLog2e), noff = pack_f32(-off, -off);
      uint64_t lsum = pack_f32(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t hi[16], rest[16];
        float f[32];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          uint64_t x;
          if constexpr (kRound) {
            x = pack_f32(lo_f32(lg[16 * q + e]), hi_f32(lg[16 * q + e]));
          } else {
            x = pack_f32(__uint_as_float(lg[(32 * q + 2 * e) & (kRound ? 31 : 63)]),
                         __uint_as_float(lg[(32 * q + 2 * e + 1) & (kRound ? 31 : 63)]));
          }
          unpack_f32(mul_f32x2(add_f32x2(x, noff), l2e), f[2 * e], f[2 * e + 1]);
          f[2 * e] = ex2p(f[2 * e]), f[2 * e + 1] = ex2p(f[2 * e + 1]);
          lsum = add_f32x2(lsum, pack_f32(f[2 * e], f[2 * e + 1]));
        }
        if (kScale && scaled_now) {
#pragma unroll
          for (int e = 0; e < 32; ++e) f[e] *= sm.vs[t][par][64 * half + 32 * q + e];
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          // p rounded to bf16 and the remainder rounded to bf16 again: both to the nearest, so that what is left out (below 2^-17
          // of p) has no side
          hi[e] = pack_bf16(f[2 * e], f[2 * e + 1]);
          rest[e] = pack_bf16(f[2 * e] - lo_f32(hi[e]), f[2 * e + 1] - hi_f32(hi[e]));
        }
        tmem_st16(tl + 32 * half + 16 * q, hi);
        tmem_st16(tl + 64 + 32 * half + 16 * q, rest);
      }
      {
        float l0, l1;
        unpack_f32(lsum, l0, l1);
        l += l0 + l1;
      }
      tmem_wait_st();
      fence_before_p();
      mbar_arrive_p(&sm.p_ready[t]);
      ++cnt;
      i = nxt;
    }
    // ---- output rows: the row's sum over both halves, 64 dims per thread
    // (the buffer of the parity before the last: everybody is done with it)
    sm.half_max[t][cnt & 1u][half][row_in] = l;
    group_sync(t);
    l = sm.half_max[t][cnt & 1u][0][row_in] + sm.half_max[t][cnt & 1u][1][row_in];
    if (n > 0) ok = mbar_wait_p(&sm.o_done, 0, sm) && ok;
    __syncwarp();
    fence_after_p();
    const float inv = l > 0.f && ok ? 1.f / l : 0.f;
    const bool any = cnt > 0;
    float finite[4] = {0.f, 0.f, 0.f, 0.f};  // (stay 0 while the values are finite)
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {
      uint32_t v[32];
      if (any) {
        tmem_ld32(tl + 128 + 64 * half + 32 * q, v);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; ++e) finite[e & 3] = fmaf(__uint_as_float(v[e]), 0.f, finite[e & 3]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint32_t w[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int d = 8 * e + 2 * x;
          w[x] = inv > 0.f && any ? pack_bf16(__uint_as_float(v[d]) * inv, __uint_as_float(v[d + 1]) * inv) : 0u;
        }
        const int chunk = q * 4 + e;  // 16-byte piece of the row's 128-byte half
        *reinterpret_cast<uint4*>(sm.q[t] + half * (kTileBytes / 2) + row_in * 128 + ((chunk ^ (row_in & 7)) * 16)) =
            make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    const bool mine = t ? have[1] : have[0];
    const unsigned again = __ballot_sync(0xffffffffu, mine && any && inv > 0.f && trow < a.Tq && !((finite[0] + finite[1]) + (finite[2] + finite[3]) == 0.f));
    if (mine && half == 0 && trow < a.Tq && (a.m || a.l)) {
      const int64_t at = ((int64_t)b * a.Hq + my_hq) * a.Tq + trow;
      if (a.m) a.m[at] = m_true;
      if (a.l) a.l[at] = l > 0.f ? l * ex2p((m_ref - m_true) * kLog2e) : 0.f;
    }
    if (again) plain_rows<kRound, kScale>(a, g, again);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    group_sync(t);
    if (row_in == 0 && half == 0 && mine) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(
                         reinterpret_cast<uint64_t>(&maps.o)),
                     "r"(h * 64), "r"(t ? tb[1] * kRowsP : tb[0] * kRowsP), "r"(my_hq), "r"(b),
                     "r"(smem_u32p(sm.q[t]) + h * (kTileBytes / 2))
                     : "memory");
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    fence_before_p();
  }
  __syncwarp();
  __syncthreads();
  if (tid == 0 && sm.dead) atomicExch(status, 1);
  if (warp == kIssuerP / 32) {
    fence_after_p();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// bf16 [batch][head][row][128] with strides in elements; boxes of 64 dims x 128 rows
bool encode_heads(CUtensorMap* map, const void* base, int64_t rows, int64_t heads, int64_t batch, int64_t s_row, int64_t s_head,
                  int64_t s_batch) {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  if (!fn) return false;
  // (the stride of an axis of one entry is never used, but has to be a legal one)
  if (rows == 1) s_row = kDp;
  if (heads == 1) s_head = s_row * rows;
  if (batch == 1) s_batch = s_head * heads;
  const cuuint64_t dims[4] = {(cuuint64_t)kDp, (cuuint64_t)rows, (cuuint64_t)heads, (cuuint64_t)batch};
  const cuuint64_t str[3] = {(cuuint64_t)s_row * 2, (cuuint64_t)s_head * 2, (cuuint64_t)s_batch * 2};
  const cuuint32_t box[4] = {64, (cuuint32_t)kRowsP, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, str, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Whether the product with sm_scale rounds to the same bf16 values as the division by its reciprocal (the reference
// divides by sqrt(D)): the quotient of a bf16 number depends on its 128 mantissas only.
bool product_rounds_like_quotient(float sm_scale) {
  static std::atomic<uint32_t> known_good{0};
  uint32_t bits;
  memcpy(&bits, &sm_scale, 4);
  if (!(sm_scale > 0.f) || !std::isfinite(sm_scale)) return false;
  if (known_good.load(std::memory_order_relaxed) == bits) return true;
  auto bf16 = [](float x) {
    uint32_t u;
    memcpy(&u, &x, 4);
    u += 0x7fffu + ((u >> 16) & 1u);
    return u >> 16;
  };
  const float root = 1.f / sm_scale;
  for (int m = 0; m < 128; ++m) {
    const float x = 1.f + (float)m / 128.f;
    const volatile float prod = x * sm_scale, quot = x / root;
    if (bf16(prod) != bf16(quot)) return false;
  }
  known_good.store(bits, std::memory_order_relaxed);
  return true;
}

struct ClassTable {
  int rows, heads, batch, n_k;
  size_t bytes() const { return (size_t)rows * heads * batch * n_k; }
};
ClassTable class_table(const jpt_attn_params& p) {
  ClassTable t;
  t.n_k = (p.S + kKeysP - 1) / kKeysP;
  t.rows = p.mk_r ? (p.Tq + kRowsP - 1) / kRowsP : 1;
  t.heads = p.mk_r ? p.Hq / p.Hkv : 1;
  t.batch = p.mk_b ? p.B : 1;
  return t;
}
bool wants_classes(const jpt_attn_params& p) { return p.mask_mode == JPT_MASK_ADD && (p.S + kKeysP - 1) / kKeysP > kSmallK; }

}  // namespace

bool attention_prefill_eligible(const jpt_attn_params& p, int64_t q_b, int64_t q_h, int64_t q_t) {
  if (p.D != kDp || p.q_dtype != JPT_BF16 || p.kv_dtype != JPT_BF16 || p.paged) return false;
  if (p.mask_mode != JPT_MASK_NONE && p.mask_mode != JPT_MASK_ADD) return false;
  if (p.S > kMaxKTiles * kKeysP) return false;
  if (!aligned(p.q, 16) || !aligned(p.k, 16) || !aligned(p.v, 16) || !aligned(p.o, 16)) return false;
  // (tensor maps take positive strides of a multiple of 16 bytes)
  auto legal = [](int64_t stride, int extent) { return extent == 1 || (stride > 0 && stride % 8 == 0 && stride < (1ll << 38)); };
  if (!legal(p.kv_b, p.B) || !legal(p.kv_h, p.Hkv) || !legal(p.kv_s, p.S)) return false;
  if (!legal(q_b, p.B) || !legal(q_h, p.Hq) || !legal(q_t, p.Tq)) return false;
  if (p.logit_rounding != 0 && !product_rounds_like_quotient(p.sm_scale)) return false;
  const double items = (double)p.B * p.Hkv * (((double)(p.Tq + kRowsP - 1) / kRowsP) * (p.Hq / p.Hkv) + 1);
  return items < 1.0e9 && (double)p.B * (p.Hq / p.Hkv) < 65536 && p.Tq <= 65535 * kRowsP;
}

size_t attention_prefill_workspace_bytes(const jpt_attn_params& p) {
  return kWorkspaceCounterBytes + (wants_classes(p) ? (class_table(p).bytes() + 255) / 256 * 256 : 0);
}

int launch_attention_prefill(const jpt_attn_params& p, const AttnArgs& a, int64_t q_b, int64_t q_h, int64_t q_t, cudaStream_t st) {
  const size_t need = attention_prefill_workspace_bytes(p);
  JPT_REQUIRE(p.workspace && p.workspace_bytes >= need, JPT_EWORKSPACE, "flash_decode: workspace of %zu bytes needed, %zu given",
              need, p.workspace_bytes);
  JPT_REQUIRE(aligned(p.workspace, 256), JPT_EALIGN, "flash_decode: workspace must be 256-byte aligned");
  char* ws = static_cast<char*>(p.workspace);
  int* status = reinterpret_cast<int*>(ws + kWorkspaceStatusOffset);
  static std::atomic<bool> configured[kMaxDevices];
  if (int rc = configure_once_per_device(configured, "prefill_attention_kernel", [] {
        cudaError_t e = cudaSuccess;
        auto set = [&e](auto kernel) {
          if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemP));
        };
        set(prefill_attention_kernel<true, true, false>);
        set(prefill_attention_kernel<true, true, true>);
        set(prefill_attention_kernel<true, false, false>);
        set(prefill_attention_kernel<true, false, true>);
        set(prefill_attention_kernel<false, true, false>);
        set(prefill_attention_kernel<false, true, true>);
        set(prefill_attention_kernel<false, false, false>);
        set(prefill_attention_kernel<false, false, true>);
        return e;
      }))
    return rc;
  PrefillMaps maps;
  const int64_t o_h = (int64_t)p.Tq * kDp;
  JPT_REQUIRE(encode_heads(&maps.q, p.q, p.Tq, p.Hq, p.B, q_t, q_h, q_b) &&
                  encode_heads(&maps.k, p.k, p.S, p.Hkv, p.B, p.kv_s, p.kv_h, p.kv_b) &&
                  encode_heads(&maps.v, p.v, p.S, p.Hkv, p.B, p.kv_s, p.kv_h, p.kv_b) &&
                  encode_heads(&maps.o, p.o, p.Tq, p.Hq, p.B, kDp, o_h, o_h * p.Hq),
              JPT_EINVAL, "flash_decode: the tensors cannot be described by a tensor map");
  PrefillGeom g;
  memset(&g, 0, sizeof(g));
  const ClassTable t = class_table(p);
  g.n_rows_t = (p.Tq + kRowsP - 1) / kRowsP;
  g.n_k = t.n_k;
  g.pairs = (g.n_rows_t * (p.Hq / p.Hkv) + 1) / 2;
  // (an odd number of blocks without grouped heads: the longest tile is alone in its item either way; 600 tokens, 32 heads 35.5 us, 34.8)
  g.fold = g.pairs * p.B * p.Hkv <= sm_count() && g.n_rows_t > 2 && (p.Hq > p.Hkv || g.n_rows_t % 2 == 0);
  g.q_b = q_b, g.q_h = q_h, g.q_t = q_t;
  g.mask_vec = p.mask_mode == JPT_MASK_ADD && aligned(p.mask, 16) && p.mk_b % 8 == 0 && p.mk_r % 8 == 0;
  g.mask_pairs = p.mask_mode == JPT_MASK_ADD && aligned(p.mask, 4) && p.mk_b % 2 == 0 && p.mk_r % 2 == 0 && p.Tq * p.mk_r % 2 == 0;
  if (wants_classes(p)) {
    uint8_t* cls = reinterpret_cast<uint8_t*>(ws + kWorkspaceCounterBytes);
    g.cls = cls;
    g.cls_rows = t.rows, g.cls_heads = t.heads, g.cls_batch = t.batch;
    const dim3 tiles(t.n_k, t.rows, t.heads * t.batch), threads(256);
    const int mask_rows = p.mk_r ? p.Tq : 1;
    // Read 16 bytes at a time the classes take a few microseconds, and the launch starts under the one in front; its CTAs crowd on
    // the SMs that that one leaves free, and this much shared memory keeps them to four each (1024 tokens, 32 / 8 heads 35.2 us started behind
    // it, 34.8 under it, 34.0 kept apart).  Element by element they take several times that, and few SMs cost more than the start
    // gains (700 tokens: 32 / 8 heads 36.4 us under it, 35.1 behind it; 64 / 8 48.5 and 41.7).
    if (g.mask_vec)
      launch_after_previous(mask_class_kernel, tiles, threads, 48 * 1024, st, a, cls, mask_rows, (int)t.heads, 1);
    else
      mask_class_kernel<<<tiles, threads, 0, st>>>(a, cls, mask_rows, t.heads, 0);
    if (int rc = check_launch("mask_class_kernel")) return rc;
  }
  const dim3 grid(g.pairs * p.B * p.Hkv), block(kThreadsP);
  const size_t smem = sizeof(SmemP);
  const bool scale = p.k_scale != nullptr;
  auto launch = [&](auto kernel) { launch_after_previous(kernel, grid, block, smem, st, maps, a, g, status); };
  auto pick = [&](auto plain, auto folded) { g.fold ? launch(folded) : launch(plain); };
  if (a.round_logits) {
    if (scale) pick(prefill_attention_kernel<true, true, false>, prefill_attention_kernel<true, true, true>);
    else pick(prefill_attention_kernel<true, false, false>, prefill_attention_kernel<true, false, true>);
  } else {
    if (scale) pick(prefill_attention_kernel<false, true, false>, prefill_attention_kernel<false, true, true>);
    else pick(prefill_attention_kernel<false, false, false>, prefill_attention_kernel<false, false, true>);
  }
  return check_launch("prefill_attention_kernel");
}

}  // namespace jpt
