// The bookkeeping of a decode step and of an insert (jetstream_pt/engine.py:371-395, 506-524, 674-729, 774-848): a
// handful of values per slot, which as tensor operations were about 45 launches and 450 us of host time per step.
// One launch in front of the model (block tables, this step's mask entry) and one behind it (argmax, tokens, lengths,
// result rows); one launch for the rows of an inserted slot.
#include <math.h>

#include "common.cuh"

namespace jpt {
namespace {

struct MaskRef {
  void* p;  // [B, S], null: leave it alone
  int f32;
  int64_t stride;
};
__device__ __forceinline__ void mask_put(const MaskRef& m, int b, int s, float v) {
  if (m.f32)
    static_cast<float*>(m.p)[b * m.stride + s] = v;
  else
    static_cast<__nv_bfloat16*>(m.p)[b * m.stride + s] = __float2bfloat16_rn(v);
}
// This step's position opened in the mask: the shared one (ring buffer) or one per slot; negative counts from the end.
__device__ __forceinline__ void mask_open(const MaskRef& m, int b, int S, int ring, int pos, const int32_t* input_pos) {
  int p = ring ? pos : input_pos[b];
  if (p < 0) p += S;
  if (p >= 0 && p < S) mask_put(m, b, p, 0.f);
}

// Block tables: where the reference's kernel fetches next when block i of slot b lies outside [start, end).  Integer
// division truncates, as the reference's jax.lax.div does.
__global__ void engine_begin_kernel(const int32_t* start, const int32_t* input_pos, int B, int S, int bk, int nb, int32_t* next_b,
                                    int32_t* next_i, MaskRef mask, int ring, int pos) {
  grid_dependency_wait();
  grid_dependency_trigger();
  for (int at = blockIdx.x * blockDim.x + threadIdx.x; at < B * nb; at += gridDim.x * blockDim.x) {
    const int b = at / nb, i = at - b * nb;
    const int st = start[b];
    int end = (st + input_pos[b]) % S;
    if (end < 0) end += S;
    const bool last = b == B - 1;
    const int last_good = st < end ? (end - 1) / bk : (S - 1) / bk;
    const int nxt_b = last ? b : b + 1, nxt_i = last ? last_good : 0;
    const bool past_end = i * bk >= end, before = (i + 1) * bk <= st;
    int rb, ri;
    if (st < end) {
      rb = past_end ? nxt_b : b;
      ri = before ? st / bk : past_end ? nxt_i : i;
    } else if (st == end) {
      rb = nxt_b;
      ri = nxt_i;
    } else {
      rb = b;
      ri = past_end && before ? st / bk : i;
    }
    next_b[at] = rb;
    next_i[at] = ri;
  }
  if (mask.p) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < B; b += gridDim.x * blockDim.x) mask_open(mask, b, S, ring, pos, input_pos);
  }
}

// Order-preserving key of a logit: larger key = larger value, NaN above everything (torch.argmax), -0 equal to 0.
__device__ __forceinline__ unsigned long long key_of(float x, unsigned index) {
  unsigned u = __float_as_uint(x);
  if (x != x) u = 0xffffffffu;
  else if (x == 0.f) u = 0x80000000u;
  else u = u & 0x80000000u ? ~u : u | 0x80000000u;
  return ((unsigned long long)u << 32) | (0xffffffffu - index);  // (of equal values the first wins)
}

constexpr int kEndCtas = 8, kEndThreads = 256;
// One cluster of eight CTAs per slot reads the slot's logits (one CTA would take a whole vocabulary at the rate of one
// SM); the eight results meet in the first CTA's shared memory.
template <typename T>
__global__ void __launch_bounds__(kEndThreads) engine_end_kernel(const T* logits, int64_t row_stride, int V, int vec,
                                                                 const int32_t* tokens, const int32_t* lens, const int32_t* input_pos,
                                                                 int S, int ring, int pos, int32_t* next_token, int32_t* lens_out,
                                                                 int32_t* pos_out, int32_t* data, MaskRef mask) {
  __shared__ unsigned long long best_of[kEndThreads / 32], best_cta[kEndCtas];
  const int part = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // (met below: the first CTA runs before it is written to)
  grid_dependency_wait();
  grid_dependency_trigger();
  unsigned long long best = 0ull;
  const T* row = logits + (int64_t)b * row_stride;
  constexpr int kPer = 16 / (int)sizeof(T);
  const int nvec = vec ? V / kPer : 0;
  for (int i = part * kEndThreads + tid; i < nvec; i += kEndCtas * kEndThreads) {
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(row) + i);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int j = 0; j < kPer; ++j) best = max(best, key_of(to_f32<T>(e[j]), (unsigned)(i * kPer + j)));
  }
  for (int i = nvec * kPer + part * kEndThreads + tid; i < V; i += kEndCtas * kEndThreads) best = max(best, key_of(to_f32<T>(row[i]), (unsigned)i));
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, sh));
  if ((tid & 31) == 0) best_of[tid >> 5] = best;
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int w = 1; w < kEndThreads / 32; ++w) best = max(best, best_of[w]);
    uint32_t remote;
    const uint32_t local = (uint32_t)__cvta_generic_to_shared(&best_cta[part]);
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(local));
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote), "l"(best) : "memory");
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (part != 0 || tid != 0) return;
#pragma unroll
  for (int c = 0; c < kEndCtas; ++c) best = max(best, best_cta[c]);
  if (mask.p) mask_open(mask, b, S, ring, pos, input_pos);
  const int p = input_pos[b], l = lens[b];
  const int l_new = ring || l != 0 ? l + 1 : 0;
  next_token[b] = (int32_t)(0xffffffffu - (unsigned)best);
  lens_out[b] = l_new;
  pos_out[b] = ring || p != 0 ? p + 1 : 0;
  data[3 * b] = tokens[b];
  data[3 * b + 1] = 1;
  data[3 * b + 2] = l_new;
}

// The rows of one slot after an insert: mask (0 on the prefix's positions, -inf elsewhere), token, start, length, count.
__global__ void engine_slot_kernel(MaskRef mask, int S, int slot, int pos, int cur, int wrap, int start_value, int seq_len,
                                   int32_t* start, int32_t* input_pos, int32_t* lens, int32_t* tokens, const void* token, int token_bytes) {
  grid_dependency_wait();
  grid_dependency_trigger();
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < S && mask.p; s += gridDim.x * blockDim.x) {
    const bool in = !wrap ? s >= pos && s < cur : cur > pos ? s >= pos && s < cur : s >= pos || s < cur;
    mask_put(mask, slot, s, in ? 0.f : -INFINITY);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (start) start[slot] = start_value;
    if (input_pos) input_pos[slot] = seq_len;
    if (lens) lens[slot] = 1;
    if (tokens) tokens[slot] = token_bytes == 8 ? (int32_t)*static_cast<const int64_t*>(token) : *static_cast<const int32_t*>(token);
  }
}

}  // namespace
}  // namespace jpt

using namespace jpt;

extern "C" int jpt_engine_begin(const int32_t* start, const int32_t* input_pos, int B, int S, int block, int32_t* next_b,
                                int32_t* next_i, void* mask, int mask_dtype, int64_t mask_stride, int ring, int pos, void* stream) {
  JPT_REQUIRE(start && input_pos && B > 0 && S > 0 && block > 0, JPT_EINVAL, "engine_begin: bad arguments");
  JPT_REQUIRE(S < block || (next_b && next_i), JPT_EINVAL, "engine_begin: null block table");
  JPT_REQUIRE(!mask || mask_dtype == JPT_BF16 || mask_dtype == JPT_F32, JPT_EINVAL, "engine_begin: the mask must be bf16 or f32");
  const int nb = S / block;
  const int work = B * nb > B ? B * nb : B;
  int blocks = (work + 127) / 128;
  if (blocks > 148) blocks = 148;
  const MaskRef m{mask, mask_dtype == JPT_F32, mask_stride};
  launch_after_previous(engine_begin_kernel, dim3(blocks), dim3(128), 0, static_cast<cudaStream_t>(stream), start, input_pos, B, S, block,
                        nb, next_b, next_i, m, ring, pos);
  return check_launch("engine_begin_kernel");
}

extern "C" int jpt_engine_end(const void* logits, int dtype, int64_t row_stride, int V, const int32_t* tokens, const int32_t* lens,
                              const int32_t* input_pos, int B, int S, int ring, int pos, int32_t* next_token, int32_t* lens_out,
                              int32_t* pos_out, int32_t* data, void* mask, int mask_dtype, int64_t mask_stride, void* stream) {
  JPT_REQUIRE(logits && tokens && lens && input_pos && next_token && lens_out && pos_out && data, JPT_EINVAL, "engine_end: null tensor");
  JPT_REQUIRE(B > 0 && B <= 65535 && S > 0 && V > 0, JPT_EINVAL, "engine_end: bad shape");
  JPT_REQUIRE(dtype == JPT_BF16 || dtype == JPT_F32, JPT_EINVAL, "engine_end: logits must be bf16 or f32");
  JPT_REQUIRE(!mask || mask_dtype == JPT_BF16 || mask_dtype == JPT_F32, JPT_EINVAL, "engine_end: the mask must be bf16 or f32");
  const MaskRef m{mask, mask_dtype == JPT_F32, mask_stride};
  const int vec = aligned(logits, 16) && (row_stride * dtype_bytes(dtype)) % 16 == 0;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kEndCtas, B);
  cfg.blockDim = dim3(kEndThreads);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[2];
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kEndCtas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = starts_early(cfg.stream) ? 2 : 1;
  const cudaError_t e =
      dtype == JPT_F32
          ? cudaLaunchKernelEx(&cfg, engine_end_kernel<float>, static_cast<const float*>(logits), row_stride, V, vec, tokens, lens,
                               input_pos, S, ring, pos, next_token, lens_out, pos_out, data, m)
          : cudaLaunchKernelEx(&cfg, engine_end_kernel<__nv_bfloat16>, static_cast<const __nv_bfloat16*>(logits), row_stride, V, vec,
                               tokens, lens, input_pos, S, ring, pos, next_token, lens_out, pos_out, data, m);
  if (e != cudaSuccess) return fail((int)e, "engine_end_kernel: %s", cudaGetErrorString(e));
  return check_launch("engine_end_kernel");
}

extern "C" int jpt_engine_insert_slot(void* mask, int mask_dtype, int64_t mask_stride, int S, int slot, int pos, int cur, int wrap,
                                      int start_value, int seq_len, int32_t* start, int32_t* input_pos, int32_t* lens, int32_t* tokens,
                                      const void* token, int token_bytes, void* stream) {
  JPT_REQUIRE(S > 0 && slot >= 0, JPT_EINVAL, "engine_insert_slot: bad slot or cache length");
  JPT_REQUIRE(!mask || mask_dtype == JPT_BF16 || mask_dtype == JPT_F32, JPT_EINVAL, "engine_insert_slot: the mask must be bf16 or f32");
  JPT_REQUIRE(!tokens || (token && (token_bytes == 4 || token_bytes == 8)), JPT_EINVAL, "engine_insert_slot: the token must be int32 or int64");
  const MaskRef m{mask, mask_dtype == JPT_F32, mask_stride};
  const int blocks = mask ? (S + 255) / 256 : 1;
  launch_after_previous(engine_slot_kernel, dim3(blocks > 148 ? 148 : blocks), dim3(256), 0, static_cast<cudaStream_t>(stream), m, S, slot, pos,
                        cur, wrap, start_value, seq_len, start, input_pos, lens, tokens, token, token_bytes);
  return check_launch("engine_slot_kernel");
}
