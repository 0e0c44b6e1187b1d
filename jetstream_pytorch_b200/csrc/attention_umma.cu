// Ragged flash-decode attention for int8 caches, head_dim 128 and up to 8
// grouped query rows on the 5th-generation tensor cores (tcgen05, sm_100a).
//
// The int8 codes never pass through registers: both contractions run as
// integer MMAs that read K, V and the small second operands straight from
// shared memory and accumulate int32 in tensor memory (TMEM).
//
//   S^T[128 tok x 16] = K[128 tok x 128 d] . Ql^T       kind::i8, K-major A and B
//   O^T[128 d  x 16] = V^T[128 d x 128 tok] . Pl^T      kind::i8, MN-major A, K-major B
//
// "Levels" make the small operands 8-bit without losing the precision of the
// bf16 / fp32 values they stand for:
//   * a query row q (bf16) is split as q = u (256 h + l) with u a power of two and h, l
//     signed bytes: exact but for values below 1/127 of the row's largest, which are rounded to
//     u (2^-14 of it at most); rows 0..7 of Ql hold h, rows 8..15 hold l, so the two partial
//     dot products of a token arrive in the same TMEM lane and S = u (256 S_h + S_l).  (The
//     chain of rounded logits keeps q = s (h + l / 254), s = amax|q| / 127.)
//   * a probability p in [0, 1] (relative to the maximum of its round), times the
//     token's V scale relative to the largest V scale c of its tile, becomes a
//     16-bit fixed-point number whose two bytes are the unsigned levels of the
//     token's row of Pl; O = (O_0 + 2^8 O_1) c / (2^16 - 1), a sum of its own for each tile: an error of
//     2^-17 c per token and unit of its V code, far below the bf16 rounding of the result.
// Every int32 sum is exact (|sum| <= 128 * 128 * 65535), so the only roundings
// are the two splits above and the fp32 online-softmax arithmetic.
//
// A tile is 128 consecutive valid tokens of one (sequence, KV head) segment, a
// round two consecutive tiles of a piece (or its last one).  CTAs take whole
// segments, longest first, or equal runs of tiles of cut ones (plan_items), or, where
// that balances badly, contiguous shares of the list of all tiles; the last
// arriver merges the pieces of a cut segment.  K and V rows of a tile land
// in shared memory as 128-byte rows, 16-byte chunks XORed with (row & 7): that
// is the canonical 128-byte-swizzle layout of the tensor core for both operand
// roles (K-major for K, MN-major for V), so nothing is rearranged.  Where a tensor
// map describes the cache the rows are moved by the copy engine
// (cp.async.bulk.tensor, completion counted on an mbarrier per tile that only the
// MMA-issuing threads wait for), else by 16-byte cp.async of all threads.  In the
// softmax phase thread t owns tokens t of both tiles (TMEM lane t of their S^T); in
// the output phase thread t owns head-dim index t (TMEM lane t of O^T), which also
// removes the cross-warp merge of the accumulators.  The softmax phase is compiled
// for 8, 4 or 2 query rows.
//
// What bounds it: rows wait for no one (about 200 of 9000 cycles of a round with three
// CTAs on an SM, at 40 KB per us and SM); the time is instructions and their fetch
// (the stall reasons are "no instruction", barriers and fixed latencies) and the start of a
// launch, when all CTAs meet cold instructions behind a burst of row requests.  So work per
// thread went from one token a pass to two (774 -> 490 instructions per warp and tile),
// the levels of a token are one 16-byte store (16 byte stores before), page ids are looked up a
// round ahead (the scales' addresses waited 4000 cycles a round for them), a piece's rows leave
// with the next round's logits, and segments are not cut where they need not be.
// B200, 96 sequences of 8 KV heads, a step of two layers with these changes and the row's L2 policy: 1 .. 2047 tokens with the
// new token 130.2 -> 107.2 us; paged, 512 .. 2047 tokens, 131.8 -> 108.2.
//
// Fused decode update (jpt_decode_update_attend): the launch also takes the
// step's new K/V token, which becomes the last token of its segment: the
// schedule counts one token more per sequence, and the CTA that processes the
// segment's last tile writes the token's int8 codes into the row behind the
// existing tokens of that tile IN SHARED MEMORY (K tile before the S^T MMA, V
// tile before the O^T MMA), so the token is attended to like any other, with
// no separate softmax term.  On one GPU that CTA reduces the token's amax over all heads
// itself.  With the KV heads sharded CTA b mod grid computes it over
// this GPU's heads while its first rows are in flight and stores it into the
// exchange slots of every rank (NVLink peer stores); the CTA with the last tile
// reads the ranks' words (long there by then).  It quantises the token's row of its head
// with the decode quantiser and also writes cache row, scale and stash.  One launch per
// layer, the exchange's round trip hidden under the existing tokens.
//
// Every wait (mbarriers, exchange words) is bounded; a CTA that gives up raises
// the status word of the workspace, frees its tensor memory and returns.
#include <cuda.h>
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>

#include "attention_tiles.cuh"

namespace jpt {
namespace {

constexpr int kTileU = 128;     // tokens per tile = TMEM lanes = threads per CTA
constexpr int kTmemCols = 64;   // S^T of the two tiles of a round: columns 0..15 and 16..31, their O^T: columns 32..47 and 48..63
constexpr int kColO = 32;
constexpr int kCtasPerSm = 3;
#ifndef JPT_PIECE_COST_U
#define JPT_PIECE_COST_U 2
#endif
#ifndef JPT_PIECE_COST_FUSED
#define JPT_PIECE_COST_FUSED 2
#endif
constexpr float kPieceTiles = 1.5f, kCutTiles = 1.3f;  // what a piece and its cut end cost, in tiles: see plan_items
constexpr int kPieceCostU = JPT_PIECE_COST_U;  // overhead slots charged per segment, in 128-token tiles
constexpr long long kWaitCycles = 1000000000ll;  // about half a second: far beyond any wait of a healthy run

// What the walker of the tile list publishes about a round: two consecutive tiles of a piece, or its last one.
struct RoundRec {
  int info;                 // kRound... bits, valid rows of the two tiles << 8 and << 16 (0: no second tile)
  int b, h;                 // sequence, KV head
  int pos[2];               // position of each tile's first row (paged: token index)
  int parts;                // pieces of the segment; their partial results (unless there is just one):
  int slot, first, stride;  // this piece's slot, and PartSlots of the segment
  int pad[3];               // (three 16-byte stores)
};
constexpr int kRoundValid = 1;                   // without it the CTA is done
constexpr int kRoundStarts = 2, kRoundEnds = 4;  // first / last round of a piece
constexpr int kRoundNew = 8;                     // the last row of its last tile is the step's new token
constexpr int kRoundParB = 16;                   // parity of the second tile's barriers
constexpr int kRoundAdd = 32;                    // additive mask values must be applied
__device__ __forceinline__ int rows_a(int info) { return (info >> 8) & 255; }
__device__ __forceinline__ int rows_b(int info) { return info >> 16; }

struct __align__(1024) SmemU {
  uint8_t k[2][kTileU * kD];             // K rows of the round's tiles: [tile][token][128 bytes], swizzled
  uint8_t v[2][kTileU * kD];             // V rows
  uint8_t qlev[16 * kD];                 // query levels: rows 0..7 high bytes, 8..15 low bytes
  uint8_t plev[2][16 * kTileU];          // probability levels of each tile: 16 bytes per token, byte 8 l + r
  alignas(16) uint8_t qraw[8 * kD * 2];  // bf16 query rows of the piece that starts with the next round
  alignas(16) uint8_t ntkv[2][kD * 4];   // new token: its K and V rows of this head (bf16 or fp32)
  uint8_t ntv[kD];                       // ... and its V codes between the K tile's turn and the V tile's
  float ntsc[2];                         // ... and its K and V scales
  unsigned long long ntw[2][8];          // ... the ranks' amax words (K, V) as they were when the round was prepared
                                         //     (one GPU: floats, the K and V maxima of the warps)
  int ntpos;                             // ... and where the token is written
  alignas(16) float xch[4][12];          // per warp: row maxima of the round [8], largest V scale of each tile [2]
  float red[4][8];                       // per warp: denominators at the end of a piece
  alignas(16) float qsc[8];              // u_r * sm_scale * log2(e)
  float qsr[8];                          // s_r / 254 (the chain of rounded logits starts from the plain dot product)
  float ntx[4];                          // new token: K amax, V amax
  uint64_t bar[2];                       // MMA completion: S^T, O^T
  uint64_t bar_k[2], bar_v[2];           // rows landed (copy-engine path), per tile of the round
  uint32_t tmem_base;
  int start[3];
  int flag;
  alignas(16) RoundRec meta[4];          // records of the rounds in flight (by number mod 4)
  int pages[2][16];                      // paged caches: the pages of their tiles (8 at most of each), by number mod 2
  WorkList work;
};

// 16-byte copy with compile-time offsets on both addresses (one pair of base registers per tensor)
template <int kOff>
__device__ __forceinline__ void cp_async16_at(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0 + %2], [%1 + %2], 16;\n" ::"r"(dst), "l"(src), "n"(kOff));
}
template <int kI>
__device__ __forceinline__ void cp_async_tile_rows(uint32_t dst, const void* src) {
  if constexpr (kI < 8) {  // 8 passes of 16 rows
    cp_async16_at<2048 * kI>(dst, src);
    cp_async_tile_rows<kI + 1>(dst, src);
  }
}
// Pairs of floats in one 64-bit register: one instruction for both.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// dst = the 2 or 4 bytes at p where `yes` (else as it was): no branch, and nothing that waits for the load.
template <int kBytes>
__device__ __forceinline__ void load_if(uint32_t& dst, const void* p, bool yes) {
  if constexpr (kBytes == 2) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p ld.global.u16 %0, [%1];\n\t}" : "+r"(dst) : "l"(p), "r"((int)yes));
  } else {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p ld.global.u32 %0, [%1];\n\t}" : "+r"(dst) : "l"(p), "r"((int)yes));
  }
}
constexpr float kNoMax = -1.0e30f;  // "no logit seen yet": finite, far below any logit
__device__ __forceinline__ float ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(x));
  return r;
}
// The level bytes of one token from the fixed-point numbers of its rows: byte r the low, byte 8 + r the high byte of row r.
template <int kR, int kOff>
__device__ __forceinline__ void store_levels(uint32_t addr, const uint32_t (&y)[8]) {
  // low bytes of a pair, then its high bytes
  const uint32_t a01 = __byte_perm(y[0], y[1], 0x5140), a23 = kR > 2 ? __byte_perm(y[2], y[3], 0x5140) : 0u;
  const uint32_t a45 = kR > 4 ? __byte_perm(y[4], y[5], 0x5140) : 0u, a67 = kR > 4 ? __byte_perm(y[6], y[7], 0x5140) : 0u;
  const uint32_t lo0 = __byte_perm(a01, a23, 0x5410), hi0 = __byte_perm(a01, a23, 0x7632);
  const uint32_t lo1 = kR > 4 ? __byte_perm(a45, a67, 0x5410) : 0u, hi1 = kR > 4 ? __byte_perm(a45, a67, 0x7632) : 0u;
  asm volatile("st.shared.v4.b32 [%0 + %5], {%1, %2, %3, %4};" ::"r"(addr), "r"(lo0), "r"(lo1), "r"(hi0), "r"(hi1), "n"(kOff) : "memory");
}
// The thread's two tokens: new running maxima, rescale factors, probabilities and denominator shares of its kR rows, and the levels.
// The probabilities are relative to the round's own maximum, so that every round has all 16 bits (relative to the running maximum, long
// pieces had 4.1e-5 of their rows' norm, not 4.0e-5): the sums so far are scaled by `alpha`, the round's by `beta`.
// Adding 2^23 rounds a probability's product to its fixed-point number and leaves that in the low bits of the float.
// m_run starts at kNoMax (finite), so exp2(old - new) and exp2(-inf - new) need no special case.
template <int kR>
__device__ __forceinline__ void softmax_rows(float (&m_run)[8], float (&l_run)[8], float (&alpha)[8], float (&beta)[8],
                                             const float (&tm)[8], const f32x2 (&x)[8], float ps0, float ps1, uint32_t p_addr) {
  const f32x2 ps = pack2(ps0, ps1), magic = pack2(8388608.f, 8388608.f);
  uint32_t y0[8], y1[8];
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const float top = fmaxf(tm[r], kNoMax);  // (every logit of the round masked: probabilities 0, beta 0 or 1)
    const float e = ex2(-fabsf(m_run[r] - top));
    const bool up = top > m_run[r];
    alpha[r] = up ? e : 1.f;
    beta[r] = up ? 1.f : e;
    m_run[r] = fmaxf(m_run[r], top);
    float d0, d1, f0, f1;
    unpack2(add2(x[r], pack2(-top, -top)), d0, d1);
    const float p0 = ex2(d0), p1 = ex2(d1);
    l_run[r] = fmaf(l_run[r], alpha[r], beta[r] * (p0 + p1));
    unpack2(fma2(pack2(p0, p1), ps, magic), f0, f1);
    y0[r] = __float_as_uint(f0);
    y1[r] = __float_as_uint(f1);
  }
  store_levels<kR, 0>(p_addr, y0);
  store_levels<kR, 16 * kTileU>(p_addr, y1);
}
// A segment's valid tokens form one run of consecutive rows, or two when the
// ring wraps: [first, first + nA) and [0, n - nA).  Tiles never straddle the
// wrap: run A is cut into tiles of 128 rows (the last one partial), then run B,
// so a tile is always one range of rows (one box for the copy engine).
__device__ __forceinline__ int run_a(const SeqRange& r, int S) { return min(r.n, S - r.first); }
__device__ __forceinline__ int tiles_run(int n) { return (n + kTileU - 1) / kTileU; }
__device__ __forceinline__ int tiles_u(const SeqRange& r, int S) {
  const int na = run_a(r, S);
  return tiles_run(na) + tiles_run(r.n - na);
}
__device__ __forceinline__ int slots_u(const SeqRange& r, int S, int cost) { return r.n > 0 ? tiles_u(r, S) + cost : 0; }
// Tile t of the segment: physical position of its first row and its number of valid rows.
__device__ __forceinline__ void tile_rows(const SeqRange& r, int S, int t, int* pos, int* cnt) {
  const int na = run_a(r, S), ta = tiles_run(na);
  if (t < ta) {
    *pos = r.first + t * kTileU;
    *cnt = min(kTileU, na - t * kTileU);
  } else {
    *pos = (t - ta) * kTileU;
    *cnt = min(kTileU, r.n - na - (t - ta) * kTileU);
  }
}

// Byte offset of (row, byte) in a tile of 128-byte rows with 128-byte swizzle.
__device__ __forceinline__ uint32_t swz(int row, int byte) {
  return (uint32_t)(row * 128 + ((((byte >> 4) ^ (row & 7))) << 4) + (byte & 15));
}

// Shared-memory matrix descriptor: 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);  // start address
  d |= (uint64_t)(1024 >> 4) << 16;       // leading byte offset (one swizzle atom; unused for these shapes)
  d |= (uint64_t)(1024 >> 4) << 32;       // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                 // descriptor version of sm_100
  d |= (uint64_t)2 << 61;                 // SWIZZLE_128B
  return d;
}
// The probability levels, MN-major without swizzle: core matrices of 8 tokens x 16 bytes, one behind the other.
__device__ __forceinline__ uint64_t umma_desc_levels(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)(128 >> 4) << 16;  // leading byte offset: to the next 8 tokens
  d |= (uint64_t)(128 >> 4) << 32;  // stride byte offset: to the next 16 columns (there are none)
  d |= (uint64_t)1 << 46;           // descriptor version of sm_100
  return d;                         // no swizzle
}
// Instruction descriptors: int32 accumulators, M = 128.
constexpr uint32_t kIdescS = (2u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);  // s8 x s8, N = 16
constexpr uint32_t kIdescO =
    (2u << 4) | (1u << 7) | (0u << 10) | (1u << 15) | (1u << 16) | ((16u >> 3) << 17) | ((128u >> 4) << 24);  // s8 x u8, both MN-major, N = 16

__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Bounded wait for the phase with the given parity; false when it gave up.
__device__ __forceinline__ bool mbar_probe(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 16; ++i) {
      uint32_t ok;
      asm volatile(
          "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}\n"
          : "=r"(ok)
          : "r"(bar), "r"(parity)
          : "memory");
      if (ok) return true;
    }
    if (clock64() - t0 > kWaitCycles) return false;
  }
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  return mbar_probe(bar, parity) || mbar_wait_slow(bar, parity);
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// One box of a 4-d tensor map (128 bytes x rows x 1 x 1) into swizzled shared memory of this CTA.  (evict_first_policy: with the default
// one the launches met their own code in DRAM again: two layers of 96 sequences, 8 KV heads, 116.3 -> 108.4 us, paged 112.4 -> 106.8.)
__device__ __forceinline__ void tma_load_rows(uint32_t dst, const CUtensorMap* map, int row, int c2, int c3, uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4, %5}], [%6], %7;" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(row), "r"(c2), "r"(c3), "r"(bar), "l"(policy)
      : "memory");
}
// The same box into L2 only.
__device__ __forceinline__ void tma_prefetch_rows(const CUtensorMap* map, int row, int c2, int c3) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(reinterpret_cast<uint64_t>(map)),
               "r"(0), "r"(row), "r"(c2), "r"(c3)
               : "memory");
}
// Tensor maps of the K and V tensors: dense [B, Hkv, S, 128 bytes] with the caller's strides
// (box: the 128 rows of a tile), or the page pool [Hkv, pages, page_size, 128 bytes] (box: a
// page, or 128 rows of a larger one).
struct TmaMaps {
  CUtensorMap k, v;
};
constexpr int kTmaNone = 0, kTmaDense = 1, kTmaPaged = 2;

// true in one lane of a converged warp, always the same one
__device__ __forceinline__ bool elect_sync() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(r));
  return r != 0;
}

// maximum over the 32 lanes in one instruction
__device__ __forceinline__ float warp_max(float x) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
  return r;
}

#ifdef JPT_UMMA_SPANS
// Debug builds only: per CTA, nanosecond stamps of the phases of its life.
__device__ unsigned long long g_umma_spans[1024 * 8];
__device__ __forceinline__ unsigned long long gtimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
#define JPT_SPAN(k)                                                                    \
  do {                                                                                 \
    if (threadIdx.x == 0 && blockIdx.x < 1024) g_umma_spans[8 * blockIdx.x + (k)] = gtimer_ns(); \
  } while (0)
#else
#define JPT_SPAN(k) do {} while (0)
#endif


// kFused = the launch carries the decode step's new token, kRound = dense_attention's rounded
// logit chain, kTma = the copy engine moves the K/V rows (tensor maps) instead of the threads, kR = query
// rows the softmax phase works on (8; 4 for groups of up to four query heads; 2 for multi-head attention
// with its single row per KV head; the level rows of the others hold zeros, their results are never
// looked at).
template <bool kFused, bool kRound, bool kTma, int kR>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
    flash_decode_i8_umma_kernel(const __grid_constant__ AttnArgs a, const __grid_constant__ MmaScratch x, int* status,
                                const __grid_constant__ NewTokenArgs nt, const __grid_constant__ TmaMaps maps, int tma_mode,
                                int box_rows) {
  // The swizzled tiles need a 1024-byte aligned base.  The array is declared
  // with that alignment (and used in place, so that every access compiles to a
  // shared-memory instruction); a base that is not aligned after all is reported.
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  SmemU& sm = *reinterpret_cast<SmemU*>(smem_raw);
  if ((smem_u32(smem_raw) & 1023u) != 0u) {
    if (threadIdx.x == 0) atomicExch(status, 2);
    return;
  }

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // Instructions of the tensor core and the copy engine are issued by the elected lane of a warp: the compiler takes their operands
  // out of uniform registers, and under any other condition (tid == 0) wraps every one of them in a loop over the lanes. (B200,
  // 96 sequences of 8 KV heads and 1 to 2047 tokens: 62.3 -> 59.4 us with the new token; paged, 512 to 2047: 62.7 -> 59.3.)
  const bool elected = elect_sync();
  // slots charged per segment on top of its tiles (with the new token: one more for its quantisation)
  constexpr int kPieceCost = kFused ? JPT_PIECE_COST_FUSED : kPieceCostU;
  const int R = a.R;
  const bool quant = a.k_scale != nullptr;
  const int cta = blockIdx.x;
#ifdef JPT_UMMA_SPANS
  if (threadIdx.x == 0 && blockIdx.x < 1024)
    for (int z = 0; z < 8; ++z) g_umma_spans[8 * blockIdx.x + z] = 0;
#endif
  JPT_SPAN(2);  // entry

  // ------------------------------------------------------------------ barriers and tensor memory
  // (warp 1; warp 0 is busy with the scan below, the barriers of the schedule publish the result)
  if (tid == 32) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sm.bar[0])));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sm.bar[1])));
    if constexpr (kTma) {
      for (int z = 0; z < 2; ++z) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sm.bar_k[z])));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sm.bar_v[z])));
      }
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.k)) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.v)) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"((uint32_t)kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    tc_fence_before();
  }
  if constexpr (kTma) {
    plan_clear(*reinterpret_cast<PlanScratch*>(&sm.plev[0][0]));
    __syncthreads();
  }
  grid_dependency_trigger();  // the kernel after this one may set itself up (it waits for the whole of this one)
  // The list of items where the walker can be one warp (the copy engine moves the rows); else, or where the estimate
  // says so, equal contiguous shares of the tiles of all segments.
  // Under the kernel before this one (a programmatic launch) the list is made from the lengths as they are then, and the
  // first tiles' rows start to travel into L2; behind it the lengths are looked at again, and the list is made again in the
  // rare case that they changed.  Nothing else of global memory is touched before that kernel is complete.
  const int n_ctas = (int)gridDim.x;
  int items = -1;
  if constexpr (kTma) {
    PlanScratch& ps = *reinterpret_cast<PlanScratch*>(&sm.plev[0][0]);
    int T[2] = {0, 0};
    bool guessed = false;
#pragma unroll 1
    for (int pass = x.early && a.B <= kPlanSeqs ? 0 : 1; pass < 2; ++pass) {
      auto tiles = [&](int b) {
        int ua;
        SeqRange r = pass == 0 ? seq_range_x<true>(a, x, b, &ua) : seq_range_x(a, x, b, &ua);
        if (kFused && r.n < a.S) r.n += 1;
        return tiles_u(r, a.S);
      };
      if (pass == 1) {
        grid_dependency_wait();
        JPT_SPAN(0);  // the kernel before this one is complete
        if (guessed) {
          bool changed = false;
          for (int z = 0; z < 2; ++z) {
            const int b = tid + kThreads * z;
            changed |= b < a.B && min(tiles(b), kPlanBins - 1) != T[z];
          }
          if (!__syncthreads_or(changed)) break;
          plan_clear(ps);
          __syncthreads();
        }
      }
      items = plan_items(a.B, a.Hkv, n_ctas, tiles, T, ps, reinterpret_cast<int*>(&sm.xch[0][0]), sm.work, kPieceTiles, kCutTiles);
      __syncthreads();  // the list is visible; the scratch is free
      guessed = true;
      if (pass == 0 && cta < items && warp == 1) {
        const WorkItem it = find_item(sm.work, a.Hkv, cta);
        int ua;
        SeqRange r = seq_range_x<true>(a, x, it.b, &ua);
        if (kFused && r.n < a.S) r.n += 1;
        const int nt_tiles = tiles_u(r, a.S), t1 = (it.part + 1) * nt_tiles / it.parts;
        for (int t = it.part * nt_tiles / it.parts, z = 0; z < 2 && t < t1; ++z, ++t) {
          int pos, cnt;
          tile_rows(r, a.S, t, &pos, &cnt);
          if (elected) {
            if (tma_mode == kTmaDense) {
              tma_prefetch_rows(&maps.k, pos, it.h, it.b);
              tma_prefetch_rows(&maps.v, pos, it.h, it.b);
            } else {
              for (int row = 0; row < cnt; row += box_rows) {
                const int page = __ldcg(a.page_table + (int64_t)it.b * a.max_pages + (pos + row) / a.page_size);
                tma_prefetch_rows(&maps.k, (pos + row) % a.page_size, page, it.h);
                tma_prefetch_rows(&maps.v, (pos + row) % a.page_size, page, it.h);
              }
            }
          }
        }
      }
    }
  } else {
    grid_dependency_wait();
    JPT_SPAN(0);
  }

  // ------------------------------------------------------------------ new token: amax to every rank
  // One GPU: every CTA with a last tile reduces the token's row itself (2 Hkv x 128 values, out of L2; nothing to wait for).
  const bool peers = kFused && nt.px_world > 1;
  unsigned nt_epoch = 0;
  if constexpr (kFused) {
    if (peers) nt_epoch = *reinterpret_cast<volatile unsigned*>(&nt.px_state[0]) + 1u;
  }
  // Largest magnitude of token b's K (which = 0) or V row over this GPU's heads: this warp's share.
  auto token_amax = [&](int b, int which) {
    const int HD = a.Hkv * kD;
    // 16 bytes per load, the loads of a pass in flight together (rows are kD elements: 16-byte multiples)
    const int chunks = HD * (nt.in_f32 ? 4 : 2) / 16;
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(nt.x[which]) + (int64_t)b * HD * (nt.in_f32 ? 4 : 2));
    float v = 0.f;
    for (int c0 = 0; c0 < chunks; c0 += 4 * kThreads) {
      uint4 u[4];
#pragma unroll
      for (int z = 0; z < 4; ++z) {
        const int c = c0 + z * kThreads + tid;
        u[z] = c < chunks ? src[c] : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int z = 0; z < 4; ++z) {
        const uint32_t w[4] = {u[z].x, u[z].y, u[z].z, u[z].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (nt.in_f32) {
            v = fmaxf(v, fabsf(__uint_as_float(w[e])));
          } else {  // two bf16 values: their magnitudes as floats
            v = fmaxf(v, fmaxf(fabsf(__uint_as_float(w[e] << 16)), fabsf(__uint_as_float(w[e] & 0xffff0000u))));
          }
        }
      }
    }
    return warp_max(v);
  };
  // Called once by every CTA, after its first rows have been requested (the reduction runs under their latency).
  auto post_amax = [&]() {
    for (int b = cta; b < a.B; b += gridDim.x) {
      const float am[2] = {token_amax(b, 0), token_amax(b, 1)};
      __syncthreads();  // the scratch may still be read for the slot before
      if (lane == 0) {
        sm.xch[warp][0] = am[0];
        sm.xch[warp][1] = am[1];
      }
      __syncthreads();
      if (tid < 2) {
        const float m4 = fmaxf(fmaxf(sm.xch[0][tid], sm.xch[1][tid]), fmaxf(sm.xch[2][tid], sm.xch[3][tid]));
        const size_t row = (size_t)(nt_epoch & 1u) * nt.px_world + nt.px_rank;
        const unsigned long long word = ((unsigned long long)nt_epoch << 32) | __float_as_uint(m4);
        for (int r = 0; r < nt.px_world; ++r)
          asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(nt.px_slots[r] + row * (2 * a.B) + tid * a.B + b), "l"(word)
                       : "memory");
      }
    }
    __syncthreads();
  };
  // Counts this CTA as done with the exchange of this launch; the last one advances the launch number.
  auto exchange_done = [&]() {
    if constexpr (kFused) {
      if (peers && tid == 0) {
        __threadfence();
        const unsigned done = atomicAdd(&nt.px_state[1], 1u);
        if (done == gridDim.x - 1) {
          nt.px_state[1] = 0;
          __threadfence();
          atomicAdd(&nt.px_state[0], 1u);
        }
      }
    }
  };

  // Valid range of sequence b as the schedule sees it: with the fused update the step's new token
  // counts as the segment's last token (a full cache has no row for it: reported, the token is dropped).
  auto seg_range = [&](int b, int* use_add, bool* extended = nullptr) {
    SeqRange r = seq_range_x(a, x, b, use_add);
    if constexpr (kFused) {
      const bool room = r.n < a.S;
      if (room) {
        r.n += 1;
      } else {
        atomicExch(status, 3);
      }
      if (extended) *extended = room;
    }
    return r;
  };

  // ------------------------------------------------------------------ schedule
  // Slots per sequence (tiles + overhead) -> exclusive prefix over sequences;
  // each thread owns a slice of ceil(B/128) sequences.  The scan scratch
  // aliases the probability levels, which are not in use yet.
  const bool listed = kTma && items >= 0;
  int share_lo = 0, rem = 0, G0 = cta, G1 = listed ? items : 0;
  if (!listed) {
    int* scan = reinterpret_cast<int*>(&sm.plev[0][0]);  // 129 ints
    const int per = (a.B + kThreads - 1) / kThreads;
    const int b_lo = min(a.B, tid * per), b_hi = min(a.B, b_lo + per);
    int mine = 0;
    for (int b = b_lo; b < b_hi; ++b) {
      int ua;
      mine += slots_u(seg_range(b, &ua), a.S, kPieceCost);
    }
    scan[tid] = mine;
    __syncthreads();
    if (warp == 0) {
      int v4[4], s = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v4[i] = scan[4 * lane + i];
        s += v4[i];
      }
      int incl = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
      }
      int run = incl - s;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        scan[4 * lane + i] = run;
        run += v4[i];
      }
      if (lane == 31) scan[kThreads] = incl;
    }
    __syncthreads();
    const int total = scan[kThreads] * a.Hkv;  // the host checked that this fits in 31 bits
    // CTA c takes slots [G0, G1): the first `rem` CTAs one slot more than the others
    share_lo = total / n_ctas;
    rem = total - share_lo * n_ctas;
    G0 = cta * share_lo + min(cta, rem);
    G1 = G0 + share_lo + (cta < rem ? 1 : 0);
    {
      // the thread whose slice holds slot G0 walks it and publishes (b, h, slot in segment)
      const int lo = scan[tid] * a.Hkv, hi = scan[tid + 1] * a.Hkv;
      if (G0 < G1 && G0 >= lo && G0 < hi) {
        int run = lo;
        for (int b = b_lo; b < b_hi; ++b) {
          int ua;
          const int sl = slots_u(seg_range(b, &ua), a.S, kPieceCost);
          const int nxt = run + sl * a.Hkv;
          if (G0 < nxt) {
            const int into = G0 - run;
            sm.start[0] = b;
            sm.start[1] = into / sl;
            sm.start[2] = into % sl;
            break;
          }
          run = nxt;
        }
      }
    }
  }
  auto cta_of_slot = [&](int slot) {
    const int big = rem * (share_lo + 1);
    return slot < big ? slot / (share_lo + 1) : rem + (slot - big) / max(share_lo, 1);
  };
  __syncthreads();  // sm.start and the tensor-memory address visible; last reads of `scan` done
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  JPT_SPAN(1);

  const __nv_bfloat16* qbase = static_cast<const __nv_bfloat16*>(a.q);
  // The new token of segment (b, h), whose last round is the next one: the copies of its K and V
  // rows start an iteration before they are needed ...
  const int nt_row_bytes = nt.in_f32 ? kD * 4 : kD * 2;
  auto stage_new_token = [&](int b, int h) {
    const int64_t row = ((int64_t)b * a.Hkv + h) * nt_row_bytes;
    const int chunks = nt_row_bytes / 16;
    if (tid < 2 * chunks) {
      const int which = tid / chunks, ch = tid - which * chunks;
      cp_async16(smem_u32(&sm.ntkv[which][0]) + ch * 16, static_cast<const uint8_t*>(nt.x[which]) + row + ch * 16, true);
    }
    // the exchange words of this sequence (normally posted long ago; looked at again if not) and the position
    if (peers && tid >= 64 && tid < 64 + 2 * nt.px_world) {
      const int which = (tid - 64) / nt.px_world, r = (tid - 64) - which * nt.px_world;
      const unsigned long long* p =
          nt.px_slots[nt.px_rank] + ((size_t)(nt_epoch & 1u) * nt.px_world + r) * (2 * a.B) + which * a.B + b;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_u32(&sm.ntw[which][r])), "l"(p));
    }
    if (tid == 96) {
      if (nt.pos) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_u32(&sm.ntpos)),
                     "l"(nt.pos + (nt.pos_count == 1 ? 0 : b)));
      } else {
        sm.ntpos = nt.pos_host;
      }
    }
    if (!peers) {
      const float am[2] = {token_amax(b, 0), token_amax(b, 1)};
      if (lane < 2) reinterpret_cast<float*>(&sm.ntw[lane][0])[warp] = lane == 0 ? am[0] : am[1];
    }
  };
  // ... and once the tile's K rows are in shared memory, the whole CTA (thread tid: head-dim index tid)
  // turns the token into codes: amax over all heads -> scales -> codes of this head's row -> the K code into
  // row `row` of the K tile, the V code aside for the V tile's turn, cache row, scales and stash to
  // global memory.  The caller's barrier publishes the shared-memory writes.
  auto quantise_new_token = [&](int half, int b, int h, int row) {
    if (!peers) {
      if (tid < 2) {
        const float* w = reinterpret_cast<const float*>(&sm.ntw[tid][0]);
        sm.ntx[tid] = fmaxf(fmaxf(w[0], w[1]), fmaxf(w[2], w[3]));
      }
    } else if (tid < 2) {  // K amax, V amax: largest partial over the ranks
      const size_t xrow = (size_t)(nt_epoch & 1u) * nt.px_world;
      float m = 0.f;
      const long long t0 = clock64();
      for (int r = 0; r < nt.px_world; ++r) {
        const unsigned long long* p = nt.px_slots[nt.px_rank] + (xrow + r) * (2 * a.B) + tid * a.B + b;
        unsigned long long w = sm.ntw[tid][r];
        while ((unsigned)(w >> 32) != nt_epoch) {
          asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
          if ((unsigned)(w >> 32) == nt_epoch) break;
          if (clock64() - t0 > nt.px_wait_cycles) {  // a rank never came: report, go on with what is there
            atomicExch(&nt.px_state[2], 1u);
            w = 0;
            break;
          }
        }
        m = fmaxf(m, __uint_as_float((unsigned)w));
      }
      sm.ntx[tid] = m;
    }
    __syncthreads();
    const float amax_k = sm.ntx[0], amax_v = sm.ntx[1];
    const float sc_k = nt.in_f32 ? decode_scale<float>(amax_k) : decode_scale<__nv_bfloat16>(amax_k);
    const float sc_v = nt.in_f32 ? decode_scale<float>(amax_v) : decode_scale<__nv_bfloat16>(amax_v);
    const int64_t xi = ((int64_t)b * a.Hkv + h) * kD + tid;
    float xk, xv;
    if (nt.in_f32) {
      xk = reinterpret_cast<const float*>(&sm.ntkv[0][0])[tid];
      xv = reinterpret_cast<const float*>(&sm.ntkv[1][0])[tid];
    } else {
      xk = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(&sm.ntkv[0][0])[tid]);
      xv = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(&sm.ntkv[1][0])[tid]);
    }
    const int8_t ck = nt.in_f32 ? decode_code<float>(xk, sc_k) : decode_code<__nv_bfloat16>(xk, sc_k);
    const int8_t cv = nt.in_f32 ? decode_code<float>(xv, sc_v) : decode_code<__nv_bfloat16>(xv, sc_v);
    sm.k[half][swz(row, tid)] = (uint8_t)ck;
    sm.ntv[tid] = (uint8_t)cv;
    if (tid < 2) sm.ntsc[tid] = tid == 0 ? sc_k : sc_v;
    if (nt.quant[0]) nt.quant[0][xi] = ck;
    if (nt.quant[1]) nt.quant[1][xi] = cv;
    int pos = sm.ntpos;
    if (pos < 0) pos += a.S;
    const bool write = nt.write_cache && pos >= 0 && pos < a.S;
    if (write) {
      const int64_t off = (int64_t)b * a.kv_b + (int64_t)h * a.kv_h + (int64_t)pos * a.kv_s + tid;
      static_cast<int8_t*>(const_cast<void*>(a.k))[off] = ck;
      static_cast<int8_t*>(const_cast<void*>(a.v))[off] = cv;
    }
    if (tid < 2) {  // every head's CTA writes the same scale: harmless, and no CTA has to wait for another
      const float sc = tid == 0 ? sc_k : sc_v;
      void* out = nt.scale_out[tid];
      void* cache = const_cast<void*>(tid == 0 ? a.k_scale : a.v_scale);
      const int64_t sidx = (int64_t)b * a.sc_b + (int64_t)pos * a.sc_s;
      if (nt.in_f32) {
        if (out) static_cast<float*>(out)[b] = sc;
        if (write) static_cast<float*>(cache)[sidx] = sc;
      } else {
        if (out) static_cast<__nv_bfloat16*>(out)[b] = __float2bfloat16_rn(sc);
        if (write) static_cast<__nv_bfloat16*>(cache)[sidx] = __float2bfloat16_rn(sc);
      }
    }
  };
  // Rows of empty sequences are nobody's tile: sequence b is cleared by CTA b mod grid (at the end of
  // the CTA's life, off the path to its first tile).  (With the fused update no sequence is empty.)
  auto clear_empty_rows = [&]() {
    for (int b = cta; b < a.B; b += gridDim.x) {
      int ua;
      if (seg_range(b, &ua).n == 0) {
        const int64_t r0 = (int64_t)b * a.Hkv * R;
        for (int i = tid; i < a.Hkv * R * kD; i += kThreads) store_o(a, r0 * kD + i, 0.f);
        for (int i = tid; i < a.Hkv * R; i += kThreads) {
          if (a.m) a.m[r0 + i] = -INFINITY;
          if (a.l) a.l[r0 + i] = 0.f;
        }
      }
    }
  };
  if (G0 >= G1) {  // no tile for this CTA
    if constexpr (kFused) {
      if (peers) post_amax();
    }
    clear_empty_rows();
    exchange_done();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kTmemCols) : "memory");
    }
    return;
  }
  const uint32_t tmem_lane = tmem + ((uint32_t)(warp * 32) << 16);  // this warp's 32 lanes

  const int8_t* kbase = static_cast<const int8_t*>(a.k);
  const int8_t* vbase = static_cast<const int8_t*>(a.v);
  const __nv_bfloat16* mask = static_cast<const __nv_bfloat16*>(a.mask);

  // ------------------------------------------------------------------ producer
  // A round's K rows are free as soon as its S^T MMAs are complete, its V rows when the O^T MMAs are: the K rows of round
  // i + 1 are requested near the start of iteration i and have the softmax phase to land, its V rows at the end
  // of iteration i and have the S^T MMAs and the softmax phase of iteration i + 1.
  // The next round's first tile: (pb, ph, pt), in a piece that ends before tile pt_end.  Kept by every thread, or
  // by the walker warp alone (below).
  int pb = 0, ph = 0, pt = 0, pt_end = 0;
  int pslot = G0;  // equal shares: global slot index of tile pt
  int pT = 0, pn = 0, pfirst = 0, puse_add = 0;
  bool pext = false;    // the sequence's last token is the step's new one
  bool pfresh = true;   // the next round is the first one of its piece
  bool pmore = true;    // there is a next round
  unsigned puses_b = 0u;  // rounds with two tiles so far
  int pparts = 0, ppart_slot = 0;
  PartSlots pparts_at{0, 0};
  unsigned ticket = 0;  // lane 0: the item after this one, drawn ahead of its turn
  // ... and what follows from it for this thread: 16-byte column tid % 8 of
  // rows tid / 8 + 16 i of a tile.  The swizzled shared-memory offset of row
  // + 16 i is that of row plus 2048 i.
  const int prow = tid >> 3, pcol = tid & 7;
  const uint32_t pdst = (uint32_t)(prow * kD + ((pcol ^ (prow & 7)) << 4));
  // pages that hold whole 16-row copy passes: one table entry per pass
  const bool pass_pages = a.paged && (a.page_size % 16) == 0 &&
                          ((kTileU % a.page_size) == 0 || (a.page_size % kTileU) == 0);
  const int passes_per_page = pass_pages ? a.page_size / 16 : 1;
  const bool rows_packed = !a.paged && a.kv_s == kD;  // rows of a tile kD bytes apart
  const int kv_s32 = (int)a.kv_s, sc_s32 = (int)a.sc_s;
  const int page_shift = a.paged && (a.page_size & (a.page_size - 1)) == 0 ? 31 - __clz(a.page_size) : -1;

  auto load_seq = [&]() {
    const SeqRange r = seg_range(pb, &puse_add, &pext);
    pn = r.n;
    pfirst = r.first;
    pT = tiles_u(r, a.S);
  };
  // Items beyond the first of each CTA are handed out by a ticket: N - n of them, and one refusal for each CTA, so that the counter
  // has come round to zero when the launch is over.  Drawn when one round of the piece is left, a round's time before
  // the answer is needed: drawn a whole piece ahead, CTAs with long pieces drew as early as the others, and the lists of some grew
  // twice as long as those of others.
  auto draw_ticket = [&]() {
    if (items > n_ctas && lane == 0) ticket = atomicInc(x.ticket, (unsigned)items - 1u);
  };
  auto open_item = [&](int k) {  // the walker warp
    const WorkItem it = find_item(sm.work, a.Hkv, k);
    pb = it.b;
    ph = it.h;
    load_seq();
    pt = it.part * pT / it.parts;
    pt_end = (it.part + 1) * pT / it.parts;
    pparts = it.parts;
    ppart_slot = k;
    pparts_at = PartSlots{k - it.part, 1};
    if (pt + 2 >= pt_end) draw_ticket();
  };
  auto open_share_piece = [&]() {  // pt, pslot are set
    pt_end = min(pT, pt + (G1 - pslot));
    const int t0slot = pslot - pt;  // slot of tile 0 of this segment
    const int first_cta = cta_of_slot(t0slot);
    pparts = cta_of_slot(t0slot + pT - 1) - first_cta + 1;
    pparts_at = PartSlots{2 * first_cta + 1, 2};
    ppart_slot = 2 * cta + (pt > 0 ? 0 : 1);
  };
  auto advance = [&](int tiles) {
    pfresh = false;
    pslot += tiles;
    pt += tiles;
    if (pt < pt_end) {
      if (listed && pt + 2 >= pt_end) draw_ticket();
      return;
    }
    pfresh = true;
    if (listed) {
      int k = items;
      if (items > n_ctas) k = n_ctas + (int)__shfl_sync(0xffffffffu, ticket, 0);
      if (k < items) open_item(k);
      else pmore = false;
      return;
    }
    pt = 0;
    pslot += kPieceCost;  // the overhead slots of the next segment
    if (++ph == a.Hkv) {
      ph = 0;
      do {
        if (++pb >= a.B) {  // past the end of the list
          pmore = false;
          return;
        }
        load_seq();
      } while (pT == 0);
    }
    pmore = pslot < G1;
    if (pmore) open_share_piece();
  };
  if (!listed) {
    pb = sm.start[0];
    ph = sm.start[1];
    load_seq();
    const int v0 = sm.start[2];  // slot inside the segment: overhead slots come first
    if (v0 < kPieceCost) {
      pslot += kPieceCost - v0;
      pt = 0;
    } else {
      pt = v0 - kPieceCost;
    }
    pmore = pslot < G1;
    if (pmore) open_share_piece();
  }

  // Rows [pos, pos + cnt) of segment (b, h) of one tensor (a tile: cnt <= 128, no ring wrap inside)
  // into the 16 KB at `dst`, by all threads; paged caches: pos is the token index.
  auto copy_rows = [&](uint32_t dst, const int8_t* base, int b, int h, int pos, int cnt) {
    const int8_t* seg = base + (a.paged ? (int64_t)h * a.kv_h : (int64_t)b * a.kv_b + (int64_t)h * a.kv_h) + pcol * 16;
    dst += pdst;
    if (rows_packed && cnt == kTileU) {
      // whole tile valid, rows kD bytes apart: one address
      cp_async_tile_rows<0>(dst, seg + (int64_t)(pos + prow) * kD);
    } else if (pass_pages) {
      // pass i (rows 16 i ..) lies inside one page (tiles of paged caches start at multiples of 128)
      int pi = pos / a.page_size, within = (pos % a.page_size) / 16;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const bool valid = 16 * i + prow < cnt;
        const int page = 16 * i < cnt ? a.page_table[(int64_t)b * a.max_pages + pi] : 0;
        const int64_t off = (int64_t)page * a.kv_page + (int64_t)(within * 16 + prow) * kD;
        cp_async16(dst + 2048 * i, seg + off, valid);
        if (++within == passes_per_page) {
          within = 0;
          ++pi;
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = prow + 16 * i;
        const bool valid = r < cnt;
        const int tok = valid ? pos + r : pos;
        int64_t off;
        if (a.paged) {
          const int pg = a.page_table[(int64_t)b * a.max_pages + tok / a.page_size];
          off = (int64_t)pg * a.kv_page + (int64_t)(tok % a.page_size) * kD;
        } else {
          off = (int64_t)tok * kv_s32;
        }
        cp_async16(dst + 2048 * i, seg + off, valid);
      }
    }
  };
  // The same by the copy engine, requested by the calling thread alone: whole boxes (rows past cnt
  // hold other tokens or the zero fill of the tensor's edge; their logits are masked and their
  // probabilities zero), 16 KB in all, counted on `bar`.  `pages`: those of the tile.
  auto request_rows = [&](uint32_t dst, const CUtensorMap* map, uint32_t bar, int b, int h, int pos, const int* pages) {
    fence_async_smem();  // earlier accesses of the threads to this slot (the merge scratch) come first
    mbar_arrive_expect_tx(bar, (uint32_t)(kTileU * kD));
    const uint64_t policy = evict_first_policy();
    if (tma_mode == kTmaDense) {
      tma_load_rows(dst, map, pos, h, b, bar, policy);
    } else if (box_rows == kTileU) {  // pages of 128 rows or more: the tile lies inside one
      tma_load_rows(dst, map, page_shift >= 0 ? pos & (a.page_size - 1) : pos % a.page_size, pages[0], h, bar, policy);
    } else {  // one box per page
      for (int r = 0; r < kTileU; r += box_rows, ++pages) tma_load_rows(dst + r * kD, map, 0, *pages, h, bar, policy);
    }
  };

  // The per-round bookkeeping of the CTA is spread over its warps: warp 0 issues the S^T MMAs, warp 1 walks
  // the tile list, writes the records and requests the K rows, warp 2 requests the V rows, warp 3 issues the O^T MMAs
  // (44.1 us per launch on the bench workload against 45.2 with everything in thread 0).
  constexpr bool kSpread = kTma;
  constexpr int kWalkerWarp = kSpread ? 1 : 0, kVRequestWarp = kSpread ? 2 : 0, kPvWarp = kSpread ? 3 : 0;
  // The page ids of a round, looked up when its record is published and put beside it at the end of the iteration, before they are
  // needed: in the way of the scales' addresses the look-up's latency came on top of theirs in every round.
  const bool tile_in_page = a.page_size >= kTileU;
  int page_ids = 0;  // lane l: page l % 8 of tile l / 8
  auto first_page = [&](int pos) { return page_shift >= 0 ? pos >> page_shift : pos / a.page_size; };
  auto put_pages = [&](int seq) {
    if (kTma && a.paged && warp == kWalkerWarp) {
      asm volatile("" : "+r"(page_ids));
      if (lane < 16) sm.pages[seq & 1][lane] = page_ids;
    }
  };
  // The record of round `seq`; an empty one when the CTA has nothing left.
  auto publish = [&](int seq) {
    if (kSpread && warp != kWalkerWarp) return;
    if (pmore) {
      SeqRange rg;
      rg.n = pn;
      rg.first = pfirst;
      const int tiles = pt + 1 < pt_end ? 2 : 1;
      int pos[2] = {0, 0}, cnt[2] = {0, 0};
      tile_rows(rg, a.S, pt, &pos[0], &cnt[0]);
      if (tiles > 1) tile_rows(rg, a.S, pt + 1, &pos[1], &cnt[1]);
      const bool last = pt + tiles == pt_end;
      if (warp == kWalkerWarp && elected) {
        RoundRec mt;
        mt.info = kRoundValid | (pfresh ? kRoundStarts : 0) | (last ? kRoundEnds : 0) | (last && pext && pt_end == pT ? kRoundNew : 0) |
                  (puses_b & 1u ? kRoundParB : 0) | (puse_add ? kRoundAdd : 0) | cnt[0] << 8 | cnt[1] << 16;
        mt.b = pb; mt.h = ph;
        mt.pos[0] = pos[0]; mt.pos[1] = pos[1];
        mt.parts = pparts; mt.slot = ppart_slot;
        mt.first = pparts_at.first; mt.stride = pparts_at.stride;
        mt.pad[0] = mt.pad[1] = mt.pad[2] = 0;
        sm.meta[seq & 3] = mt;
      }
      if (kTma && a.paged) {
        const int rows = lane < 8 ? cnt[0] : lane < 16 ? cnt[1] : 0, e = lane & 7;
        page_ids = 0;
        if (tile_in_page ? e == 0 && rows > 0 : e * a.page_size < rows)
          page_ids = a.page_table[(int64_t)pb * a.max_pages + first_page(lane < 8 ? pos[0] : pos[1]) + e];
      }
      puses_b += tiles > 1 ? 1u : 0u;
      advance(tiles);
    } else if (warp == kWalkerWarp && elected) {
      sm.meta[seq & 3].info = 0;
    }
  };
  // A word of a record in every lane, known to be the same (branches on it need no reconvergence).
  auto info_of = [&](int seq) { return (int)__reduce_or_sync(0xffffffffu, (unsigned)sm.meta[seq & 3].info); };
  // The rows of a round of one tensor, by one warp (the copy engine) or by all threads.
  auto fetch_rows = [&](int seq, int info, uint8_t (&dst)[2][kTileU * kD], const int8_t* base, const CUtensorMap* map, uint64_t (&bar)[2]) {
    const RoundRec& m = sm.meta[seq & 3];
    if constexpr (kTma) {
      if (elected) {
        const int* pages = sm.pages[seq & 1];
        request_rows(smem_u32(&dst[0][0]), map, smem_u32(&bar[0]), m.b, m.h, m.pos[0], pages);
        if (rows_b(info) > 0) request_rows(smem_u32(&dst[1][0]), map, smem_u32(&bar[1]), m.b, m.h, m.pos[1], pages + 8);
      }
    } else {
      copy_rows(smem_u32(&dst[0][0]), base, m.b, m.h, m.pos[0], rows_a(info));
      if (rows_b(info) > 0) copy_rows(smem_u32(&dst[1][0]), base, m.b, m.h, m.pos[1], rows_b(info));
    }
  };
  // V rows of round `seq`.  Copy groups of the threads: those of K (with the query rows and the new token), then V.
  auto issue_v = [&](int seq, int info) {
    __syncwarp();
    if (!kTma || warp == kVRequestWarp) fetch_rows(seq, info, sm.v, vbase, &maps.v, sm.bar_v);
    cp_async_commit();
  };
  // Query rows of round `seq` when it starts a piece (converted at the end of this iteration), the new token when it is in it, the
  // scales of this thread's tokens, consumed by this same thread an iteration later: they stay raw bits until then, so that nothing
  // here waits for the loads; and the K rows.
  const bool sc_f32 = a.scale_is_f32 != 0;
  const uint32_t raw_one = sc_f32 ? 0x3f800000u : 0x3f80u;
  auto scale_of = [&](uint32_t raw) { return __uint_as_float(sc_f32 ? raw : raw << 16); };
  uint32_t nks[2] = {0u, 0u}, nvs[2] = {0u, 0u};
  auto issue_k = [&](int seq, int info) {
    const RoundRec& m = sm.meta[seq & 3];
    const int mb = m.b;
    if (info & kRoundStarts) {
      const __nv_bfloat16* q = qbase + ((int64_t)mb * a.Hkv + m.h) * R * kD;
      for (int ch = tid; ch < R * 16; ch += kThreads) cp_async16(smem_u32(&sm.qraw[0]) + ch * 16, q + ch * 8, true);
    }
    if (!kTma || warp == kWalkerWarp) fetch_rows(seq, info, sm.k, kbase, &maps.k, sm.bar_k);
    // (a tile that is not there: no rows.  Where there is no token the scales are zero: a stale row's product, or the second tile's columns
    // of tensor memory from before, could be infinite, and minus infinity added to that is no mask.)
    const bool in_a = tid < rows_a(info), in_b = tid < rows_b(info);
    nks[0] = nvs[0] = in_a ? raw_one : 0u;
    nks[1] = nvs[1] = in_b ? raw_one : 0u;
    if (quant) {
      int64_t at[2];
      if (a.paged) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int first = m.pos[half], tok = first + tid;
          int pg, in_page;
          if constexpr (kTma) {
            if (tile_in_page) {
              pg = sm.pages[seq & 1][8 * half];
              in_page = tok - first_page(first) * a.page_size;
            } else {  // (a divisor of 128)
              pg = sm.pages[seq & 1][8 * half + (tid >> page_shift)];
              in_page = tid & (a.page_size - 1);
            }
          } else {
            const int pi = first_page(tok);
            pg = (half ? in_b : in_a) ? a.page_table[(int64_t)mb * a.max_pages + pi] : 0;
            in_page = tok - pi * a.page_size;
          }
          at[half] = (int64_t)pg * a.page_size + in_page;
        }
      } else {
        at[0] = (int64_t)mb * a.sc_b + (int64_t)(m.pos[0] + tid) * sc_s32;
        at[1] = at[0] + (int64_t)(m.pos[1] - m.pos[0]) * sc_s32;
      }
      if (sc_f32) {
        load_if<4>(nks[0], static_cast<const uint32_t*>(a.k_scale) + at[0], in_a);
        load_if<4>(nvs[0], static_cast<const uint32_t*>(a.v_scale) + at[0], in_a);
        load_if<4>(nks[1], static_cast<const uint32_t*>(a.k_scale) + at[1], in_b);
        load_if<4>(nvs[1], static_cast<const uint32_t*>(a.v_scale) + at[1], in_b);
      } else {
        load_if<2>(nks[0], static_cast<const uint16_t*>(a.k_scale) + at[0], in_a);
        load_if<2>(nvs[0], static_cast<const uint16_t*>(a.v_scale) + at[0], in_a);
        load_if<2>(nks[1], static_cast<const uint16_t*>(a.k_scale) + at[1], in_b);
        load_if<2>(nvs[1], static_cast<const uint16_t*>(a.v_scale) + at[1], in_b);
      }
    }
    if constexpr (kFused) {
      if (info & kRoundNew) stage_new_token(mb, m.h);
    }
    cp_async_commit();
  };

  // ------------------------------------------------------------------ consumer state
  float m_run[8], l_run[8], o[8];  // l_run: this thread's tokens' share of the denominators; o: head-dim index tid
  bool dead = false;  // a wait ran out
  const float unit2 = a.sm_scale * kLog2e;
  const uint32_t bar_s = smem_u32(&sm.bar[0]), bar_o = smem_u32(&sm.bar[1]);
  const uint32_t q_desc_addr = smem_u32(&sm.qlev[0]), p_desc_addr = smem_u32(&sm.plev[0][0]);
  const uint32_t p_addr = smem_u32(&sm.plev[0][0]) + 16u * (uint32_t)tid;  // this thread's token of the first tile

  // Query levels of the piece that starts with round `seq` of this CTA (when it
  // starts one), then S^T of its tiles on the tensor core.  Called by the whole
  // CTA once the round's K rows have landed and a barrier has made them (and the
  // record) visible; the logits of the round before are out of tensor memory.
  auto prepare = [&](int seq, int info) {
    if (info & kRoundStarts) {
      // thread (row = tid / 16, chunk = tid % 16) converts 8 values of one query row
      const int row = tid >> 4, ch = tid & 15;
      float f[8];
      if (row < R) {
        const uint4 raw = *reinterpret_cast<const uint4*>(&sm.qraw[row * (kD * 2) + ch * 16]);
        const __nv_bfloat162* p2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 t = __bfloat1622float2(p2[e]);
          f[2 * e] = t.x;
          f[2 * e + 1] = t.y;
        }
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = 0.f;
      }
      float amax = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(f[e]));
#pragma unroll
      for (int sh = 1; sh <= 8; sh <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, sh));
      uint32_t hi[2] = {0u, 0u}, lo[2] = {0u, 0u};
      float unit;  // of the dot products
      if constexpr (kRound) {
        const float inv = amax > 0.f ? 127.f / amax : 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float t = f[e] * inv;
          const float h = rintf(t);
          const float l = rintf((t - h) * 254.f);
          hi[e >> 2] |= ((uint32_t)(int)h & 0xffu) << (8 * (e & 3));
          lo[e >> 2] |= ((uint32_t)(int)l & 0xffu) << (8 * (e & 3));
        }
        unit = amax * (1.f / 127.f) * (1.f / 254.f);
      } else {
        // 2^(E - 14) for an amax in [2^E, 2^(E + 1)), twice that for the amax of mantissa 255 (its 32640 units would be an h of 128); normal
        // numbers.  An infinite amax leaves levels of zero and an infinite unit: no logit of the row is a number.
        const int e2 = max((int)((__float_as_uint(amax) + 0x10000u) >> 23), 27);
        const bool finite = amax < INFINITY;
        unit = finite ? __uint_as_float((uint32_t)(e2 - 14) << 23) : INFINITY;
        const float inv = finite ? __uint_as_float((uint32_t)(268 - e2) << 23) : 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int t = __float2int_rn(f[e] * inv);  // (|t| < 32640)
          hi[e >> 2] |= ((uint32_t)((t + 128) >> 8) & 0xffu) << (8 * (e & 3));
          lo[e >> 2] |= ((uint32_t)t & 0xffu) << (8 * (e & 3));  // (t - 256 h is -128 .. 127)
        }
      }
      *reinterpret_cast<uint2*>(&sm.qlev[swz(row, 8 * ch)]) = make_uint2(hi[0], hi[1]);
      *reinterpret_cast<uint2*>(&sm.qlev[swz(8 + row, 8 * ch)]) = make_uint2(lo[0], lo[1]);
      if (ch == 0) {
        if constexpr (kRound) sm.qsr[row] = unit;
        else sm.qsc[row] = unit * unit2;
      }
      fence_async_smem();
      tc_fence_before();
      __syncthreads();
    }
    const uint32_t par_a = (uint32_t)seq & 1u, par_b = info & kRoundParB ? 1u : 0u;
    if constexpr (kFused) {
      if (info & kRoundNew) {  // the new token becomes the row behind the tile's existing tokens
        const int half = rows_b(info) > 0 ? 1 : 0;
        if constexpr (kTma) {
          if (!mbar_wait(smem_u32(&sm.bar_k[half]), half ? par_b : par_a)) dead = true;  // the rows must be there first
        }
        quantise_new_token(half, sm.meta[seq & 3].b, sm.meta[seq & 3].h, (half ? rows_b(info) : rows_a(info)) - 1);
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
      }
    }
    if (warp == 0) {
      if constexpr (kTma) {
        if (!mbar_wait(smem_u32(&sm.bar_k[0]), par_a)) dead = true;
        if (rows_b(info) > 0 && !mbar_wait(smem_u32(&sm.bar_k[1]), par_b)) dead = true;
      }
      __syncwarp();
      tc_fence_after();
      if (elected) {
        const uint64_t ka = umma_desc(smem_u32(&sm.k[0][0])), kb = umma_desc(smem_u32(&sm.k[1][0])), qd = umma_desc(q_desc_addr);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) umma_i8(tmem, ka + (uint64_t)(2 * ks), qd + (uint64_t)(2 * ks), kIdescS, ks > 0);
        if (rows_b(info) > 0) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) umma_i8(tmem + 16, kb + (uint64_t)(2 * ks), qd + (uint64_t)(2 * ks), kIdescS, ks > 0);
        }
        umma_commit(bar_s);
      }
      __syncwarp();
    }
  };
  // A piece has ended: its rows, or a partial result for the merge.  The denominators of the four warps are in shared memory.
  auto flush = [&](const RoundRec& m) {
    const bool is_final = m.parts == 1;
    const int64_t row_base = ((int64_t)m.b * a.Hkv + m.h) * R;
    float L = 0.f;  // lane r: row r
    if (lane < kR) L = (sm.red[0][lane] + sm.red[1][lane]) + (sm.red[2][lane] + sm.red[3][lane]);
    float M = m_run[0];
#pragma unroll
    for (int r = 1; r < kR; ++r) M = lane == r ? m_run[r] : M;
    if (!(M > 0.5f * kNoMax)) M = -INFINITY;  // every logit of the row was masked
    if (is_final) {
      // (times the reciprocal: 1e-7 of a row at most, beside 4e-5 from the levels; divisions, or a correction by the remainder, cost 1 % of a step)
      const float inv = L > 0.f ? __frcp_rn(L) : 0.f;
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        const float c = __shfl_sync(0xffffffffu, inv, r);
        if (r < R) store_o(a, (row_base + r) * kD + tid, c > 0.f ? o[r] * c : 0.f);
      }
      if (tid < R) {
        if (a.m) a.m[row_base + tid] = M * kLn2;
        if (a.l) a.l[row_base + tid] = L > 0.f ? L : 0.f;
      }
      return;
    }
    const int64_t p0 = (int64_t)m.slot * kMaxRows;
#pragma unroll
    for (int r = 0; r < kR; ++r)
      if (r < R) __stcg(&x.part_o[(p0 + r) * kD + tid], o[r]);
    if (tid < R) {
      __stcg(&x.part_m[p0 + tid], M);
      __stcg(&x.part_l[p0 + tid], L);
      __stcg(&x.part_t[p0 + tid], M);
    }
    // Whoever delivers the last piece of the segment combines all of them.
    // The counter wraps back to zero on that arrival, ready for the next launch.
    // (the barrier orders the CTA's stores before thread 0's fence, which publishes them with the arrival)
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      const unsigned old = atomicInc(&x.counters[m.b * a.Hkv + m.h], (unsigned)(m.parts - 1));
      sm.flag = old == (unsigned)(m.parts - 1);
    }
    __syncthreads();
    if (sm.flag) {
      __threadfence();
      merge_rows<kR, 4>(a, x, PartSlots{m.first, m.stride}, m.parts, row_base);
    }
  };

  // The tensor core works one step ahead of the threads: S^T of round i+1 is issued in iteration i, and O^T of round i is
  // collected in iteration i+1, in the same trip to tensor memory as the logits of round i+1 (a piece that ended with round i
  // leaves there), so neither MMA is waited for right after it was issued.
  // Two tiles a round: what a thread does per round and not per token (barriers, maxima across the warps, rescaling, the
  // output's way out of tensor memory) is paid for 256 tokens.
  // Iterations -2 and -1 only fill the pipeline: the code of a round exists once.  The first ones, which all CTAs of an SM work on
  // at the same time and behind a burst of row requests, do not fetch it twice.
  if (listed && warp == kWalkerWarp) open_item(cta);
  float alpha[8], beta[8], cmax[2] = {0.f, 0.f};  // (cmax: the largest V scale of each tile of the round)
#pragma unroll
  for (int r = 0; r < 8; ++r) m_run[r] = l_run[r] = o[r] = alpha[r] = beta[r] = 0.f;
  int info = 0;   // of the round at hand; what is needed less often is read from its record
  bool ended = false;  // the round before ended a piece
  int i = -2, info_next = 0;
#pragma unroll 1
  for (;; ++i) {
    const bool more = (info & kRoundValid) != 0, filled = i >= 0 && more;
    const bool pending = i > 0;  // O^T of the round before has not been added yet
    const RoundRec& mt = sm.meta[i & 3];
    const uint32_t par = (uint32_t)i & 1u;

    // ---------------- the output of the round before and the logits of this one leave tensor memory; the K rows of this
    // round are free after that
    uint32_t s0[16], s1[16];
    if (i >= 0) {
      if (filled && !mbar_wait(bar_s, par)) dead = true;
      if (pending && !mbar_wait(bar_o, par ^ 1u)) dead = true;
      tc_fence_after();
      uint32_t oa[16], ob[16];
      tmem_ld16(tmem_lane + kColO, oa);  // (in iteration 0 there is none yet: not looked at)
      tmem_ld16(tmem_lane + kColO + 16, ob);
      tmem_ld_wait();
      if (pending) {
        const float ca = cmax[0] * (1.f / 65535.f), cb = cmax[1] * (1.f / 65535.f);  // (0 for a tile that is not there: its columns hold an earlier sum)
#pragma unroll
        for (int r = 0; r < kR; r += 2) {  // the two levels combine exactly in int32 (|O_0 + 256 O_1| <= 128 * 128 * 65535 < 2^31)
          const f32x2 fa = pack2((float)((int)oa[r] + ((int)oa[8 + r] << 8)), (float)((int)oa[r + 1] + ((int)oa[9 + r] << 8)));
          const f32x2 fb = pack2((float)((int)ob[r] + ((int)ob[8 + r] << 8)), (float)((int)ob[r + 1] + ((int)ob[9 + r] << 8)));
          const f32x2 f = fma2(fb, pack2(cb, cb), mul2(fa, pack2(ca, ca)));
          unpack2(fma2(pack2(o[r], o[r + 1]), pack2(alpha[r], alpha[r + 1]), mul2(f, pack2(beta[r], beta[r + 1]))), o[r], o[r + 1]);
        }
      }
      if (ended) flush(sm.meta[(i - 1) & 3]);
      // (after it: a second load in the other branch would cost a move for each of its registers)
      tmem_ld16(tmem_lane, s0);
      tmem_ld16(tmem_lane + 16, s1);
      tmem_ld_wait();
      if (!more) break;
    }
    if (info & kRoundStarts) {
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        m_run[r] = kNoMax;
        l_run[r] = 0.f;
        o[r] = 0.f;
      }
    }
    // scales of this thread's tokens in round i, requested an iteration ago (pinned: converted earlier, they are waited for earlier)
    float cks[2], cvs[2];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      asm volatile("" : "+r"(nks[half]), "+r"(nvs[half]));
      cks[half] = scale_of(nks[half]);
      cvs[half] = scale_of(nvs[half]);
    }
    if constexpr (kFused) {
      if (info & kRoundNew) {  // the new token: its scales were just computed
        const float ks = sm.ntsc[0], vs = sm.ntsc[1];
        const bool in_b = rows_b(info) > 0, mine_a = !in_b && tid == rows_a(info) - 1, mine_b = in_b && tid == rows_b(info) - 1;
        cks[0] = mine_a ? ks : cks[0];
        cvs[0] = mine_a ? vs : cvs[0];
        cks[1] = mine_b ? ks : cks[1];
        cvs[1] = mine_b ? vs : cvs[1];
      }
    }
    f32x2 xv[8];  // logits of the two tokens (log2 units)
    if (!filled) {
#pragma unroll
      for (int r = 0; r < kR; ++r) xv[r] = 0ull;
    } else {
      // a row past the tile's tokens: product with a scale of 0, + (-inf)
      const bool in_a = tid < rows_a(info), in_b = tid < rows_b(info);
      float mk[2] = {in_a ? 0.f : -INFINITY, in_b ? 0.f : -INFINITY};
      if (info & kRoundAdd) {  // additive mask that is not a plain 0 / -inf range (rare)
        const __nv_bfloat16* mrow = mask + (int64_t)mt.b * a.mk_b + tid;
        if (in_a) mk[0] = __bfloat162float(mrow[mt.pos[0]]);
        if (in_b) mk[1] = __bfloat162float(mrow[mt.pos[1]]);
      }
      if constexpr (!kRound) {
        const f32x2 ks = pack2(cks[0], cks[1]), ml = pack2(mk[0] * kLog2e, mk[1] * kLog2e);
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          const float qc = sm.qsc[r];
          xv[r] = fma2(pack2((float)((int)s0[r] * 256 + (int)s0[8 + r]), (float)((int)s1[r] * 256 + (int)s1[8 + r])), mul2(pack2(qc, qc), ks), ml);
        }
      } else {
        // dense_attention on bf16 tensors: the reference rounds the logit to bf16 after every step
        const float sqrt_d = __frcp_rn(a.sm_scale), inv_sqrt_d = __frcp_rn(sqrt_d);
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          const float qr = sm.qsr[r];
          const float x0 = rounded_logit((float)((int)s0[r] * 254 + (int)s0[8 + r]) * qr, sqrt_d, inv_sqrt_d, cks[0], quant, mk[0]);
          const float x1 = rounded_logit((float)((int)s1[r] * 254 + (int)s1[8 + r]) * qr, sqrt_d, inv_sqrt_d, cks[1], quant, mk[1]);
          xv[r] = pack2(in_a ? kLog2e * x0 : -INFINITY, in_b ? kLog2e * x1 : -INFINITY);
        }
      }
    }
    info_next = i >= -1 ? info_of(i + 1) : 0;
    if (info_next & kRoundValid) issue_k(i + 1, info_next);
    else cp_async_commit();  // (an empty group: behind it the V rows of this round are never the youngest group, see below)
    publish(i + 2);
    if constexpr (kFused) {
      if (peers && i == -1) post_amax();
    }
    if (i >= -1) {  // (once without a round, while the first rows travel: the first round then finds its instructions at hand)
      // maxima per row across the 256 tokens, and the largest V scale of each tile
      {
        float wm[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          float lo, hi;
          unpack2(xv[r], lo, hi);
          wm[r] = warp_max(fmaxf(lo, hi));
        }
        const float ca = warp_max(cvs[0]), cb = warp_max(cvs[1]);
        if (lane == 0) {
          *reinterpret_cast<float4*>(&sm.xch[warp][0]) = make_float4(wm[0], wm[1], wm[2], wm[3]);
          if (kR > 4) *reinterpret_cast<float4*>(&sm.xch[warp][4]) = make_float4(wm[4], wm[5], wm[6], wm[7]);
          *reinterpret_cast<float2*>(&sm.xch[warp][8]) = make_float2(ca, cb);
        }
      }
      tc_fence_before();
      __syncthreads();

      {
        float2 c[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) c[w] = *reinterpret_cast<const float2*>(&sm.xch[w][8]);
        cmax[0] = fmaxf(fmaxf(c[0].x, c[1].x), fmaxf(c[2].x, c[3].x));
        cmax[1] = fmaxf(fmaxf(c[0].y, c[1].y), fmaxf(c[2].y, c[3].y));
        float tm[8];
#pragma unroll
        for (int g = 0; g < (kR > 4 ? 2 : 1); ++g) {
          float4 t[4];
#pragma unroll
          for (int w = 0; w < 4; ++w) t[w] = *reinterpret_cast<const float4*>(&sm.xch[w][4 * g]);
          tm[4 * g + 0] = fmaxf(fmaxf(t[0].x, t[1].x), fmaxf(t[2].x, t[3].x));
          tm[4 * g + 1] = fmaxf(fmaxf(t[0].y, t[1].y), fmaxf(t[2].y, t[3].y));
          tm[4 * g + 2] = fmaxf(fmaxf(t[0].z, t[1].z), fmaxf(t[2].z, t[3].z));
          tm[4 * g + 3] = fmaxf(fmaxf(t[0].w, t[1].w), fmaxf(t[2].w, t[3].w));
        }
        // p <= 1 and the product is held at 2^16 - 1 (the fast division may land one ulp above)
        const float ps0 = cmax[0] > 0.f ? fminf(cvs[0] * __fdividef(65535.f, cmax[0]), 65535.f) : 0.f;
        const float ps1 = cmax[1] > 0.f ? fminf(cvs[1] * __fdividef(65535.f, cmax[1]), 65535.f) : 0.f;
        softmax_rows<kR>(m_run, l_run, alpha, beta, tm, xv, ps0, ps1, p_addr);
      }
      if (info & kRoundEnds) {
        // denominators: the warp's sum of its threads' shares, rows dealt out to the lanes on the way (row = lane / (32 / kR))
        float v[kR];
#pragma unroll
        for (int r = 0; r < kR; ++r) v[r] = l_run[r];
        int sh = 16;
#pragma unroll
        for (int n = kR / 2; n > 0; n >>= 1, sh >>= 1) {
          const bool hi = (lane & sh) != 0;
#pragma unroll
          for (int r = 0; r < n; ++r) {
            const float away = hi ? v[r] : v[r + n], keep = hi ? v[r + n] : v[r];
            v[r] = keep + __shfl_xor_sync(0xffffffffu, away, sh);
          }
        }
#pragma unroll
        for (; sh > 0; sh >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], sh);
        if (lane % (32 / kR) == 0) sm.red[warp][lane / (32 / kR)] = v[0];
      }
      if constexpr (kFused) {
        if (info & kRoundNew) {  // the new token's V codes into the row behind the tile's existing tokens
          const int half = rows_b(info) > 0 ? 1 : 0;
          if constexpr (kTma) {
            if (!mbar_wait(smem_u32(&sm.bar_v[half]), half ? (info & kRoundParB ? 1u : 0u) : par)) dead = true;
          } else {
            cp_async_wait<1>();  // (the younger group: that of the next round's K rows)
            __syncthreads();     // every thread's copies into this tile have landed
          }
          sm.v[half][swz((half ? rows_b(info) : rows_a(info)) - 1, tid)] = sm.ntv[tid];
        }
      }
    }
    put_pages(i + 2);
    cp_async_wait<0>();  // the query rows and the new token of round i+1 (without the copy engine also its K rows and V of this one)
    fence_async_smem();
    tc_fence_before();
    if (__syncthreads_or(dead)) break;
    if (i < -1) continue;
    if (i == -1 && (info_next & kRoundValid)) issue_v(0, info_next);  // behind the first query and K rows

    // ---------------- O^T = V^T Pl^T on the tensor core
    if (filled && warp == kPvWarp) {
      if constexpr (kTma) {
        if (!mbar_wait(smem_u32(&sm.bar_v[0]), par)) dead = true;
        if (rows_b(info) > 0 && !mbar_wait(smem_u32(&sm.bar_v[1]), info & kRoundParB ? 1u : 0u)) dead = true;
      }
      __syncwarp();
      tc_fence_after();
      if (elected) {
        const uint64_t va = umma_desc(smem_u32(&sm.v[0][0])), vb = umma_desc(smem_u32(&sm.v[1][0]));
        const uint64_t pa = umma_desc_levels(p_desc_addr), pc = umma_desc_levels(p_desc_addr + 16 * kTileU);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) umma_i8(tmem + kColO, va + (uint64_t)(256 * ks), pa + (uint64_t)(32 * ks), kIdescO, ks > 0);
        if (rows_b(info) > 0) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) umma_i8(tmem + kColO + 16, vb + (uint64_t)(256 * ks), pc + (uint64_t)(32 * ks), kIdescO, ks > 0);
        }
        umma_commit(bar_o);
      }
      __syncwarp();
    }

    // ---------------- the next round: its K rows were requested near the start of this iteration
    if (info_next & kRoundValid) {
      prepare(i + 1, info_next);
      if (filled) {  // its V rows, as soon as those of this round have been read
        if (!kTma || warp == kVRequestWarp) {
          if (!mbar_wait(bar_o, par)) dead = true;
        }
        issue_v(i + 1, info_next);
      }
    }
    ended = (info & kRoundEnds) != 0;
    info = info_next;
    if (i == 0) JPT_SPAN(4);
#ifdef JPT_UMMA_SPANS
    if (threadIdx.x == 0 && blockIdx.x < 1024) {
      g_umma_spans[8 * blockIdx.x + 6] += 1;                                  // rounds
    }
#endif
    if (i < 0 && !(info & kRoundValid)) break;
  }
  JPT_SPAN(5);
  clear_empty_rows();
  exchange_done();
  cp_async_wait<0>();
  tc_fence_before();
  // A wait ran out, in front of a round's barrier or behind that of the last one (its V rows, its output): reported; the requests of the
  // copy engine that may still be in flight get their (bounded) time, the ticket comes round to zero all the same.
  if (__syncthreads_or(dead)) {
    if (tid == 0) {
      atomicExch(status, 1);
      if constexpr (kTma) {
        auto landed = [&](uint64_t (&bar)[2], int round, int bits) {
          if (!(bits & kRoundValid)) return;
          mbar_wait(smem_u32(&bar[0]), (uint32_t)round & 1u);
          if (rows_b(bits) > 0) mbar_wait(smem_u32(&bar[1]), bits & kRoundParB ? 1u : 0u);
        };
        const int round = (info & kRoundValid) ? i : i - 1;  // the last one whose V rows were requested
        landed(sm.bar_k, i + 1, info_next);
        landed(sm.bar_v, round, round >= 0 ? sm.meta[round & 3].info : 0);
      }
    }
    if (listed && items > n_ctas && warp == kWalkerWarp && lane == 0 && pmore) {
      if (pt + 2 < pt_end) ticket = atomicInc(x.ticket, (unsigned)items - 1u);
      for (int z = 0; z < items && n_ctas + (int)ticket < items; ++z) ticket = atomicInc(x.ticket, (unsigned)items - 1u);
    }
    __syncthreads();
  }
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kTmemCols) : "memory");
  }
  JPT_SPAN(7);  // end
}

int umma_num_ctas() { return sm_count() * kCtasPerSm; }

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn() {
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

// [dims[3]][dims[2]][dims[1]][128] bytes with byte strides str[0..2] between rows / dims[2] / dims[3].
bool encode_rows_map(CUtensorMap* map, const void* base, const cuuint64_t (&dims)[4], const cuuint64_t (&str)[3], int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return false;
  const cuuint32_t box[4] = {(cuuint32_t)kD, (cuuint32_t)box_rows, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(base), dims, str, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct MapKey {
  const void *k, *v;
  int64_t d1, d2, d3, s0, s1, s2;
  int mode, box_rows, device;
  bool operator==(const MapKey& o) const {
    return k == o.k && v == o.v && d1 == o.d1 && d2 == o.d2 && d3 == o.d3 && s0 == o.s0 && s1 == o.s1 && s2 == o.s2 &&
           mode == o.mode && box_rows == o.box_rows && device == o.device;
  }
};
struct MapEntry {
  MapKey key;
  TmaMaps maps;
};

// Tensor maps for this call (cached per tensor pair and geometry); kTmaNone when
// the layout cannot be described (the kernel then copies the rows with its threads).
// JPT_NO_TMA=1 in the environment forces that path.
int tensor_maps_for(const jpt_attn_params& p, TmaMaps* out, int* box_rows) {
  static const bool off = [] {
    const char* e = getenv("JPT_NO_TMA");
    return e && e[0] == '1';
  }();
  if (off) return kTmaNone;
  MapKey key{};
  key.k = p.k;
  key.v = p.v;
  key.device = current_device();
  if (p.paged) {
    if (p.page_size % 16 != 0 || p.kv_page != (int64_t)p.page_size * kD || p.kv_h <= 0 || p.kv_h % p.kv_page != 0) return kTmaNone;
    if ((kTileU % p.page_size) != 0 && (p.page_size % kTileU) != 0) return kTmaNone;
    key.mode = kTmaPaged;
    key.box_rows = p.page_size < kTileU ? p.page_size : kTileU;
    key.d1 = p.page_size; key.d2 = p.kv_h / p.kv_page; key.d3 = p.Hkv;
    key.s0 = kD; key.s1 = p.kv_page; key.s2 = p.kv_h;
  } else {
    key.mode = kTmaDense;
    key.box_rows = kTileU;
    key.d1 = p.S; key.d2 = p.Hkv; key.d3 = p.B;
    key.s0 = p.kv_s; key.s1 = p.kv_h; key.s2 = p.kv_b;
    if (p.Hkv == 1 && key.s1 <= 0) key.s1 = key.s0 * p.S;  // a single head: its stride is never used
    if (p.B == 1 && key.s2 <= 0) key.s2 = key.s1 * p.Hkv;
  }
  if (key.s0 % 16 || key.s1 % 16 || key.s2 % 16 || key.s0 < kD || key.s1 <= 0 || key.s2 <= 0) return kTmaNone;
  if (!aligned(p.k, 16) || !aligned(p.v, 16)) return kTmaNone;
  *box_rows = key.box_rows;
  static std::mutex mu;
  static std::vector<MapEntry> cache;
  std::lock_guard<std::mutex> lock(mu);
  for (const MapEntry& e : cache) {
    if (e.key == key) {
      *out = e.maps;
      return key.mode;
    }
  }
  const cuuint64_t dims[4] = {(cuuint64_t)kD, (cuuint64_t)key.d1, (cuuint64_t)key.d2, (cuuint64_t)key.d3};
  const cuuint64_t str[3] = {(cuuint64_t)key.s0, (cuuint64_t)key.s1, (cuuint64_t)key.s2};
  MapEntry e;
  e.key = key;
  if (!encode_rows_map(&e.maps.k, p.k, dims, str, key.box_rows) || !encode_rows_map(&e.maps.v, p.v, dims, str, key.box_rows))
    return kTmaNone;
  if (cache.size() >= 4096) cache.clear();
  cache.push_back(e);
  *out = e.maps;
  return key.mode;
}

}  // namespace

bool attention_umma_eligible(const jpt_attn_params& p) {
  const int R = (p.Hq / p.Hkv) * p.Tq;
  return attention_mma_eligible(p) && p.kv_dtype == JPT_INT8 && R <= 8;
}

int launch_attention_umma(const jpt_attn_params& p, const AttnArgs& a, cudaStream_t st, const NewTokenArgs* nt_in) {
  const ScratchLayout lay = scratch_layout(p, umma_num_ctas());
  JPT_REQUIRE(p.workspace && p.workspace_bytes >= lay.total, JPT_EWORKSPACE,
              "flash_decode: workspace of %zu bytes needed, %zu given", lay.total, p.workspace_bytes);
  JPT_REQUIRE(aligned(p.workspace, 256), JPT_EALIGN, "flash_decode: workspace must be 256-byte aligned");
  char* ws = static_cast<char*>(p.workspace);
  MmaScratch x;
  x.counters = reinterpret_cast<unsigned*>(ws + lay.counters);
  x.seqinfo = reinterpret_cast<int32_t*>(ws + lay.seqinfo);
  x.part_m = reinterpret_cast<float*>(ws + lay.part_m);
  x.part_l = reinterpret_cast<float*>(ws + lay.part_l);
  x.part_t = reinterpret_cast<float*>(ws + lay.part_t);
  x.part_o = reinterpret_cast<float*>(ws + lay.part_o);
  x.ticket = reinterpret_cast<unsigned*>(ws + kWorkspaceTicketOffset);
  x.early = starts_early(st) ? 1 : 0;
  // no more CTAs than the longest sequences could have tiles (a ring's two runs may add one)
  x.num_ctas = (int)std::min<int64_t>(lay.num_ctas, (int64_t)p.B * p.Hkv * ((p.S + kTileU - 1) / kTileU + 1));
  int* status = reinterpret_cast<int*>(ws + kWorkspaceStatusOffset);

  constexpr int smem_bytes = (int)sizeof(SmemU);
  static_assert(offsetof(SmemU, plev) % 1024 == 0 && offsetof(SmemU, qlev) % 1024 == 0, "operand tiles need a 1024-byte aligned base");
  static_assert(kCtasPerSm * (smem_bytes + 1024) <= 228 * 1024, "shared memory of the resident CTAs exceeds the SM");
  static std::atomic<bool> configured[kMaxDevices];
  if (int rc = configure_once_per_device(configured, "flash_decode_i8_umma_kernel", [] {
        cudaError_t e = cudaSuccess;
        auto set = [&e](auto kernel) {  // three CTAs of 73 KB per SM
          if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
          if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
        };
        set(flash_decode_i8_umma_kernel<false, false, false, 8>);
        set(flash_decode_i8_umma_kernel<false, false, true, 8>);
        set(flash_decode_i8_umma_kernel<false, true, false, 8>);
        set(flash_decode_i8_umma_kernel<false, true, true, 8>);
        set(flash_decode_i8_umma_kernel<true, false, false, 8>);
        set(flash_decode_i8_umma_kernel<true, false, true, 8>);
        set(flash_decode_i8_umma_kernel<true, true, false, 8>);
        set(flash_decode_i8_umma_kernel<true, true, true, 8>);
        set(flash_decode_i8_umma_kernel<false, false, false, 4>);
        set(flash_decode_i8_umma_kernel<false, false, true, 4>);
        set(flash_decode_i8_umma_kernel<false, true, false, 4>);
        set(flash_decode_i8_umma_kernel<false, true, true, 4>);
        set(flash_decode_i8_umma_kernel<true, false, false, 4>);
        set(flash_decode_i8_umma_kernel<true, false, true, 4>);
        set(flash_decode_i8_umma_kernel<true, true, false, 4>);
        set(flash_decode_i8_umma_kernel<true, true, true, 4>);
        set(flash_decode_i8_umma_kernel<false, false, false, 2>);
        set(flash_decode_i8_umma_kernel<false, false, true, 2>);
        set(flash_decode_i8_umma_kernel<false, true, false, 2>);
        set(flash_decode_i8_umma_kernel<false, true, true, 2>);
        set(flash_decode_i8_umma_kernel<true, false, false, 2>);
        set(flash_decode_i8_umma_kernel<true, false, true, 2>);
        set(flash_decode_i8_umma_kernel<true, true, false, 2>);
        set(flash_decode_i8_umma_kernel<true, true, true, 2>);
        return e;
      }))
    return rc;
  if (a.mask_mode == JPT_MASK_ADD) {
    if (int rc = launch_mask_ranges(a, x, st)) return rc;
  }
  NewTokenArgs nt;
  memset(&nt, 0, sizeof(nt));
  if (nt_in) {
    nt = *nt_in;
    if (nt.px_wait_cycles <= 0) nt.px_wait_cycles = kWaitCycles;
    nt.enabled = 1;
  }
  TmaMaps maps;
  memset(&maps, 0, sizeof(maps));
  int box_rows = kTileU;
  const int tma_mode = tensor_maps_for(p, &maps, &box_rows);
  const bool fused = nt.enabled != 0, round = a.round_logits != 0, tma = tma_mode != kTmaNone;
  const dim3 grid(x.num_ctas), block(kThreads);
#define JPT_UMMA_LAUNCH2(F, Rd, T)                                                                                       \
  do {                                                                                                                   \
    if (a.R <= 2)                                                                                                        \
      launch_after_previous(flash_decode_i8_umma_kernel<F, Rd, T, 2>, grid, block, smem_bytes, st, a, x, status, nt, maps, \
                            tma_mode, box_rows);                                                                         \
    else if (a.R <= 4)                                                                                                   \
      launch_after_previous(flash_decode_i8_umma_kernel<F, Rd, T, 4>, grid, block, smem_bytes, st, a, x, status, nt, maps, \
                            tma_mode, box_rows);                                                                         \
    else                                                                                                                 \
      launch_after_previous(flash_decode_i8_umma_kernel<F, Rd, T, 8>, grid, block, smem_bytes, st, a, x, status, nt, maps, \
                            tma_mode, box_rows);                                                                         \
  } while (0)
#define JPT_UMMA_LAUNCH(F, Rd, T) JPT_UMMA_LAUNCH2(F, Rd, T)
  if (fused) {
    if (round) { if (tma) JPT_UMMA_LAUNCH(true, true, true); else JPT_UMMA_LAUNCH(true, true, false); }
    else       { if (tma) JPT_UMMA_LAUNCH(true, false, true); else JPT_UMMA_LAUNCH(true, false, false); }
  } else {
    if (round) { if (tma) JPT_UMMA_LAUNCH(false, true, true); else JPT_UMMA_LAUNCH(false, true, false); }
    else       { if (tma) JPT_UMMA_LAUNCH(false, false, true); else JPT_UMMA_LAUNCH(false, false, false); }
  }
#undef JPT_UMMA_LAUNCH2
#undef JPT_UMMA_LAUNCH
  return check_launch("flash_decode_i8_umma_kernel");
}

}  // namespace jpt

#ifdef JPT_UMMA_SPANS
extern "C" int jpt_debug_umma_spans(unsigned long long* out_host, int n_ctas) {
  return (int)cudaMemcpyFromSymbol(out_host, jpt::g_umma_spans, sizeof(unsigned long long) * 8 * n_ctas);
}
#endif
