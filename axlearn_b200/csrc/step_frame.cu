// The two ends of a decoding step, one launch each: token embeddings (with the lengths' bump) in front of the layers,
// and behind the output product the greedy pick with the step's bookkeeping.  All of it is a few KB to a few MB, so
// what counts is the number of launches and one round trip to memory in each.  As separate operators they were 6 to 11
// launches (argmax 11 us, a gather of 16 rows 12, increments and copies of 2 each, none of them chained); captured steps,
// before / now: 1B widths, batch 1 245 / 229 us; Sagisun batch 1 178 / 161; Zukitar batch 16 354 / 334.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "chain.cuh"
#include "sm100.cuh"

namespace axb {

constexpr int kMaxKept = 4;

struct StepEndArgs {
  const float* logits;  // [B, ld]
  float* logits_out;    // [B, V], null: leave the logits where they are
  int64_t* tokens;      // [B]
  int* lengths;         // [B] += active, null: not here
  const int* active;
  int* kept_dst[kMaxKept];  // [B] each
  const int* kept_src[kMaxKept];
  int64_t ld;
  int B, V, kept;
};

namespace {

// Torch's order of a maximum: NaN above everything, the first of equals.
__device__ __forceinline__ bool is_nan(float x) { return (__float_as_uint(x) & 0x7fffffffu) > 0x7f800000u; }
__device__ __forceinline__ bool beats(float a, int ia, float b, int ib) {
  const bool na = is_nan(a), nb = is_nan(b);
  if (na || nb) return na && (!nb || ia < ib);
  return a > b || (a == b && ia < ib);
}

constexpr int kEndThreads = 1024;

template <bool VEC>
__global__ void __launch_bounds__(kEndThreads) step_end_kernel(StepEndArgs a) {
  chain_link();
  const int b = blockIdx.x;
  const float* row = a.logits + b * a.ld;
  float* copy = a.logits_out != nullptr ? a.logits_out + static_cast<int64_t>(b) * a.V : nullptr;
  float best = -INFINITY;
  int at = 0x7fffffff;
  if (VEC) {
    constexpr int kFlight = 8;
    const int vecs = a.V / 4;
    for (int i0 = threadIdx.x; i0 < vecs; i0 += kEndThreads * kFlight) {
      float4 v[kFlight];
#pragma unroll
      for (int u = 0; u < kFlight; ++u)
        if (i0 + u * kEndThreads < vecs) v[u] = reinterpret_cast<const float4*>(row)[i0 + u * kEndThreads];
#pragma unroll
      for (int u = 0; u < kFlight; ++u) {
        const int i = i0 + u * kEndThreads;
        if (i >= vecs) break;
        if (copy != nullptr) reinterpret_cast<float4*>(copy)[i] = v[u];
        const float x[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (beats(x[j], 4 * i + j, best, at)) best = x[j], at = 4 * i + j;
      }
    }
  } else {
    for (int i = threadIdx.x; i < a.V; i += kEndThreads) {
      const float x = row[i];
      if (copy != nullptr) copy[i] = x;
      if (beats(x, i, best, at)) best = x, at = i;
    }
  }
  __shared__ float s_best[32];
  __shared__ int s_at[32];
  auto reduce = [&]() {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, off);
      const int oa = __shfl_xor_sync(0xffffffffu, at, off);
      if (beats(ob, oa, best, at)) best = ob, at = oa;
    }
  };
  reduce();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) s_best[warp] = best, s_at[warp] = at;
  __syncthreads();
  if (warp > 0) return;
  best = s_best[lane], at = s_at[lane];
  reduce();
  if (lane != 0) return;
  a.tokens[b] = at;
  if (a.lengths != nullptr) a.lengths[b] += a.active[b];
#pragma unroll
  for (int i = 0; i < kMaxKept; ++i)
    if (i < a.kept) a.kept_dst[i][b] = a.kept_src[i][b];
}

// One CTA per token, 16 bytes a thread and pass.  An id outside the table gives NaN and a mark in the status word.
__global__ void __launch_bounds__(256)
embed_rows_kernel(const uint4* __restrict__ table, const int64_t* ids, uint4* out, int* lengths, int max_len, int V,
                  int vecs, int64_t table_ld, int wrap, int* status) {
  chain_link();
  const int64_t b = blockIdx.x;
  int64_t id = ids[b];
  if (wrap && id < 0) id += V;
  const bool ok = id >= 0 && id < V;
  for (int i = threadIdx.x; i < vecs; i += blockDim.x)
    out[b * vecs + i] = ok ? __ldg(table + id * table_ld + i)
                           : make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
  if (threadIdx.x == 0) {
    if (!ok && status != nullptr) atomicCAS(status, 0, kStatusBadArgument);
    if (lengths != nullptr) lengths[b] = min(lengths[b] + 1, max_len);
  }
}

// out = counts + by.  A chained launch of its own only so that the chain does not end: the output product behind it starts its
// weights while the last layer still runs.
__global__ void __launch_bounds__(256) add_counts_kernel(const int* counts, const int* by, int* out, int n) {
  chain_link();
  for (int i = threadIdx.x; i < n; i += 256) out[i] = counts[i] + by[i];
}

// Tokens that a caller hands to a step, one CTA; ids outside [low, high) become 0, and `ok` tells whether there were none.
__global__ void __launch_bounds__(256)
take_tokens_kernel(const int64_t* ids, int64_t* tokens, int count, int64_t low, int64_t high, bool* ok) {
  int good = 1;
  for (int i = threadIdx.x; i < count; i += 256) {
    const int64_t id = ids[i];
    const bool inside = id >= low && id < high;
    tokens[i] = inside ? id : 0;
    good &= inside;
  }
  good = __syncthreads_and(good);
  if (threadIdx.x == 0) *ok = good != 0;
}

}  // namespace
}  // namespace axb

// tokens [count] = ids [count], see the kernel.
extern "C" int axb_take_tokens(const int64_t* ids, int64_t* tokens, int count, int64_t low, int64_t high, bool* ok,
                               cudaStream_t stream) {
  if (count <= 0) return 0;
  axb::take_tokens_kernel<<<1, 256, 0, stream>>>(ids, tokens, count, low, high, ok);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// out [n] = counts + by, a handful of numbers; chained like a step's other kernels.
extern "C" int axb_add_counts(const int* counts, const int* by, int* out, int n, cudaStream_t stream) {
  using namespace axb;
  if (n <= 0) return 0;
  launch_chained(add_counts_kernel, 1, 256, 0, stream, counts, by, out, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// Returns 0, -10 for unsupported sizes.
extern "C" int axb_step_end(const axb::StepEndArgs* args, cudaStream_t stream) {
  using namespace axb;
  const StepEndArgs& a = *args;
  if (a.B <= 0) return 0;
  if (a.V <= 0 || (a.B > 1 && a.ld < a.V) || a.kept < 0 || a.kept > kMaxKept ||
      (a.lengths != nullptr && a.active == nullptr))
    return -10;
  const uintptr_t align = reinterpret_cast<uintptr_t>(a.logits) | reinterpret_cast<uintptr_t>(a.logits_out);
  if (!(align & 15) && !((a.V | a.ld) & 3))
    launch_chained(step_end_kernel<true>, a.B, kEndThreads, 0, stream, a);
  else
    launch_chained(step_end_kernel<false>, a.B, kEndThreads, 0, stream, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// out [count, width] = table[ids] (bf16 rows, `table_ld` elements apart; width and pitch multiples of 8, pointers
// 16-byte aligned); `wrap`: negative ids count from the end.  With `lengths` [count] also lengths = min(lengths + 1, max_len).
extern "C" int axb_embed_rows(const void* table, const int64_t* ids, void* out, int* lengths, int max_len, int64_t count,
                              int V, int width, int64_t table_ld, int wrap, int* status, cudaStream_t stream) {
  using namespace axb;
  if (count <= 0) return 0;
  const uintptr_t align = reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(out);
  if (V <= 0 || width <= 0 || (width % 8) || (table_ld % 8) || table_ld < width || count > 0x7fffffff || (align & 15))
    return -10;
  const int vecs = width / 8, want = (vecs + 31) / 32 * 32;
  launch_chained(embed_rows_kernel, static_cast<unsigned>(count), want < 256 ? want : 256, 0, stream,
                 static_cast<const uint4*>(table), ids, static_cast<uint4*>(out), lengths, max_len, V, vecs, table_ld / 8,
                 wrap, status);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
