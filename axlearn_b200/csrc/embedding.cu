// Gradient of an embedding table: dw[v, :] = sum over the tokens with id v of dy[token, :], summed in 32 bits in token
// order and rounded once.  The bound is the table's own size (every row is written, most of them with zeros), so there is
// no pass that clears it and no sort of all tokens: ids are counted per row, the rows' lists are filled in any order, and
// put in order row by row -- up to kEmbList tokens by the warp that sums them, longer lists in a bitmap over the tokens.
// Rows with more tokens than a segment are summed by segment over many CTAs (partial sums of 32 bits, added in order):
// padding and the frequent words of a text would otherwise be thousands of rows for one CTA.
//
// 32768 x 4096, 8192 tokens, us (torch's operator -- fill, radix sort, partial sums -- in brackets): uniform ids 122 (765),
// frequency 1 / rank 177 (570), half of the tokens one id 182 (600), all of them 250 (446); without segments and bitmap
// 113, 585, 2499 and 5063.  Uniform: 76 for the rows (51 at the copy rate), 31 for the offsets, 2 or 3 for each other pass.
// A gradient's scaling by the loss's own gradient, 32768 x 4096: 95 us against 190.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mma_sync.cuh"

namespace axb {
namespace {

constexpr int kEmbThreads = 256, kEmbList = 32;

__global__ void emb_count_kernel(const int64_t* __restrict__ ids, int n, int V, int* __restrict__ counts) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t id = ids[i];
  if (id >= 0 && id < V) atomicAdd(counts + id, 1);
}

// offsets[v] = sum of counts[0 .. v); cursor = offsets.  One CTA: a table's counters are a few hundred KB at most.
__global__ void __launch_bounds__(1024) emb_scan_kernel(const int* __restrict__ counts, int V, int* __restrict__ offsets,
                                                        int* __restrict__ cursor) {
  __shared__ int s_warp[32];
  __shared__ int s_base;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_base = 0;
  __syncthreads();
  for (int v0 = 0; v0 < V; v0 += 4096) {
    int c[4], sum = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int v = v0 + tid * 4 + j;
      c[j] = v < V ? counts[v] : 0;
      sum += c[j];
    }
    int incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += o;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      int w = s_warp[lane];
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, w, off);
        if (lane >= off) w += o;
      }
      s_warp[lane] = w;
    }
    __syncthreads();
    int at = s_base + incl - sum + (warp > 0 ? s_warp[warp - 1] : 0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int v = v0 + tid * 4 + j;
      if (v < V) offsets[v] = at, cursor[v] = at;
      at += c[j];
    }
    __syncthreads();
    if (tid == 0) s_base += s_warp[31];
    __syncthreads();
  }
}

__global__ void emb_fill_kernel(const int64_t* __restrict__ ids, int n, int V, int* __restrict__ cursor,
                                int* __restrict__ list) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t id = ids[i];
  if (id >= 0 && id < V) list[atomicAdd(cursor + id, 1)] = i;
}

__device__ __forceinline__ void emb_add(float (&acc)[8], const uint4& u) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 f = unpack2(w[k]);
    acc[2 * k] += f.x, acc[2 * k + 1] += f.y;
  }
}

// The lists of rows with more than kEmbList tokens, in order: a list's tokens are marked in a bitmap over the tokens (a
// window of them at a time), and the marks read off in order.
constexpr int kEmbWindow = 1 << 18;  // tokens: 32 KB

__global__ void __launch_bounds__(kEmbThreads)
emb_order_kernel(const int* __restrict__ counts, const int* __restrict__ offsets, const int* __restrict__ list,
                 int* __restrict__ sorted, int n, int V) {
  __shared__ unsigned s_bits[kEmbWindow / 32];
  __shared__ int s_rows[kEmbThreads], s_found, s_warp[kEmbThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int64_t v0 = blockIdx.x; v0 < V; v0 += static_cast<int64_t>(gridDim.x) * kEmbThreads) {
    if (tid == 0) s_found = 0;
    __syncthreads();
    const int64_t v = v0 + static_cast<int64_t>(tid) * gridDim.x;
    if (v < V && counts[v] > kEmbList) s_rows[atomicAdd(&s_found, 1)] = static_cast<int>(v);
    __syncthreads();
    const int found = s_found;
    for (int r = 0; r < found; ++r) {
      const int row = s_rows[r], count = counts[row], first = offsets[row];
      int done = 0;
      for (int t0 = 0; t0 < n; t0 += kEmbWindow) {
        const int words = (min(kEmbWindow, n - t0) + 31) / 32;
        for (int i = tid; i < words; i += kEmbThreads) s_bits[i] = 0;
        __syncthreads();
        for (int i = tid; i < count; i += kEmbThreads) {
          const int t = list[first + i] - t0;
          if (t >= 0 && t < kEmbWindow) atomicOr(s_bits + (t >> 5), 1u << (t & 31));
        }
        __syncthreads();
        const int each = (words + kEmbThreads - 1) / kEmbThreads, w0 = min(words, tid * each), w1 = min(words, w0 + each);
        int sum = 0;
        for (int w = w0; w < w1; ++w) sum += __popc(s_bits[w]);
        int incl = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const int o = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += o;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        int at = first + done + incl - sum, total = 0;
#pragma unroll
        for (int w = 0; w < kEmbThreads / 32; ++w) {
          at += w < warp ? s_warp[w] : 0;
          total += s_warp[w];
        }
        for (int w = w0; w < w1; ++w)
          for (unsigned m = s_bits[w]; m != 0; m &= m - 1) sorted[at++] = t0 + w * 32 + __ffs(m) - 1;
        done += total;
        __syncthreads();
      }
    }
    __syncthreads();
  }
}

// acc += dy[tokens[lo .. hi), 8 columns c] in order; the whole CTA, which shares the tokens (`c` may lie beyond the row).
template <int kFlight>
__device__ __forceinline__ void emb_sum(float (&acc)[8], const uint4* dy, const int* tokens, int lo, int hi, int c,
                                        int vecs, int* s_tok) {
  for (int i0 = lo; i0 < hi; i0 += kEmbThreads) {
    const int some = min(kEmbThreads, hi - i0);
    __syncthreads();
    if (static_cast<int>(threadIdx.x) < some) s_tok[threadIdx.x] = tokens[i0 + threadIdx.x];
    __syncthreads();
    if (c < vecs) {
#pragma unroll kFlight
      for (int j = 0; j < some; ++j) emb_add(acc, __ldg(dy + static_cast<int64_t>(s_tok[j]) * vecs + c));
    }
  }
}

__device__ __forceinline__ uint4 emb_pack(const float (&acc)[8]) {
  return make_uint4(pack2(acc[0], acc[1]), pack2(acc[2], acc[3]), pack2(acc[4], acc[5]), pack2(acc[6], acc[7]));
}

// Rows with more tokens than a segment of the (concatenated, ordered) lists: a CTA sums what lies in its segment, in 32
// bits, for 2048 columns.  That is part of at most two such rows: one that began in an earlier segment (slot 2 g of
// `partial`) and one that begins in this one (slot 2 g + 1).
__global__ void __launch_bounds__(kEmbThreads)
emb_segments_kernel(const uint4* __restrict__ dy, const int64_t* __restrict__ ids, const int* __restrict__ counts,
                    const int* __restrict__ offsets, const int* __restrict__ list, const int* __restrict__ sorted,
                    float4* __restrict__ partial, int V, int vecs, int segment) {
  __shared__ int s_tok[kEmbThreads];
  const int g = blockIdx.x, lo = g * segment, hi = min(lo + segment, offsets[V - 1] + counts[V - 1]);
  if (lo >= hi) return;
  const int first = static_cast<int>(ids[list[lo]]), last = static_cast<int>(ids[list[hi - 1]]);
  const int c = blockIdx.y * kEmbThreads + threadIdx.x;
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    const int row = k == 0 ? first : last, begin = offsets[row], end = begin + counts[row];
    if (end - begin <= segment || (begin < lo) != (k == 0)) continue;
    float acc[8] = {};
    emb_sum<8>(acc, dy, sorted, max(lo, begin), min(hi, end), c, vecs, s_tok);
    if (c >= vecs) continue;
    float4* out = partial + (static_cast<int64_t>(2 * g + k) * vecs + c) * 2;
    out[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    out[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
  }
}

// A CTA takes every gridDim-th row of the table, its threads 8 columns each.  Eight CTAs fit an SM: most rows of a large table
// are written and nothing else (five CTAs: 13 us more for 128256 x 2048).
__global__ void __launch_bounds__(kEmbThreads, 8)
emb_rows_kernel(const uint4* __restrict__ dy, const int* __restrict__ counts, const int* __restrict__ offsets,
                const int* __restrict__ list, const int* __restrict__ sorted, const float4* __restrict__ partial,
                uint4* __restrict__ dw, int V, int vecs, int segment) {
  __shared__ int s_tok[kEmbThreads];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int v = blockIdx.x; v < V; v += gridDim.x) {
    uint4* out = dw + static_cast<int64_t>(v) * vecs;
    const int count = counts[v];
    if (count == 0) {
      for (int c = tid; c < vecs; c += kEmbThreads) out[c] = make_uint4(0, 0, 0, 0);
      continue;
    }
    if (count <= kEmbList) {
      if (warp == 0) {  // tokens are all different: a token's place is the number of smaller ones
        const int mine = lane < count ? list[offsets[v] + lane] : 0x7fffffff;
        int place = 0;
        for (int j = 0; j < count; ++j) place += __shfl_sync(0xffffffffu, mine, j) < mine;
        if (lane < count) s_tok[place] = mine;
      }
      __syncthreads();
      for (int c = tid; c < vecs; c += kEmbThreads) {
        float acc[8] = {};
#pragma unroll 4
        for (int j = 0; j < count; ++j) emb_add(acc, __ldg(dy + static_cast<int64_t>(s_tok[j]) * vecs + c));
        out[c] = emb_pack(acc);
      }
      __syncthreads();
      continue;
    }
    const int begin = offsets[v], end = begin + count;
    if (count <= segment) {
      for (int c0 = 0; c0 < vecs; c0 += kEmbThreads) {
        float acc[8] = {};
        emb_sum<4>(acc, dy, sorted, begin, end, c0 + tid, vecs, s_tok);
        if (c0 + tid < vecs) out[c0 + tid] = emb_pack(acc);
      }
      __syncthreads();
      continue;
    }
    const int g0 = begin / segment, g1 = (end - 1) / segment;
    for (int c = tid; c < vecs; c += kEmbThreads) {
      float acc[8] = {};
#pragma unroll 2
      for (int g = g0; g <= g1; ++g) {
        const float4* part = partial + (static_cast<int64_t>(2 * g + (g == g0 ? 1 : 0)) * vecs + c) * 2;
        const float4 x = __ldg(part), y = __ldg(part + 1);
        acc[0] += x.x, acc[1] += x.y, acc[2] += x.z, acc[3] += x.w;
        acc[4] += y.x, acc[5] += y.y, acc[6] += y.z, acc[7] += y.w;
      }
      out[c] = emb_pack(acc);
    }
  }
}

// Tokens of a segment: 64, more for many tokens, so that the segments' sums stay a few hundred rows of 32 bits.
inline int emb_segment(int n) {
  int s = 64;
  while (s < 512 && n / s > 256) s *= 2;
  return s;
}

// out = x * g with g rounded to bf16 first, as a product of bf16 tensors; g in device memory.
__global__ void __launch_bounds__(256)
scale_bf16_kernel(const uint4* __restrict__ x, const float* __restrict__ g, uint4* __restrict__ out, int64_t vecs) {
  const float s = __bfloat162float(__float2bfloat16(*g));
  constexpr int kFlight = 4;
  const int64_t step = static_cast<int64_t>(gridDim.x) * 256;
  for (int64_t i0 = blockIdx.x * 256ll + threadIdx.x; i0 < vecs; i0 += step * kFlight) {
    uint4 v[kFlight];
#pragma unroll
    for (int u = 0; u < kFlight; ++u)
      if (i0 + u * step < vecs) v[u] = __ldcs(x + i0 + u * step);
#pragma unroll
    for (int u = 0; u < kFlight; ++u) {
      if (i0 + u * step >= vecs) break;
      uint32_t* w = reinterpret_cast<uint32_t*>(&v[u]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = unpack2(w[k]);
        w[k] = pack2(f.x * s, f.y * s);
      }
      out[i0 + u * step] = v[u];
    }
  }
}

}  // namespace
}  // namespace axb

// Bytes of `work` for axb_embedding_bwd.
extern "C" int64_t axb_embedding_bwd_bytes(int n, int V, int D) {
  if (n < 0 || V <= 0 || D <= 0) return 0;
  const int segment = axb::emb_segment(n);
  const int64_t slots = n > segment ? 2 * ((static_cast<int64_t>(n) + segment - 1) / segment) : 0;
  return slots * D * 4 + (2 * static_cast<int64_t>(n) + 3 * static_cast<int64_t>(V)) * 4;
}

// dw [V, D] (bf16, every row written) from dy [n, D] and ids [n]; ids outside [0, V) are left out.  `work`:
// axb_embedding_bwd_bytes, 16-byte aligned.
extern "C" int axb_embedding_bwd(const void* dy, const int64_t* ids, void* dw, void* work, int n, int V, int D,
                                 cudaStream_t stream) {
  using namespace axb;
  if (V <= 0 || D <= 0 || (D % 8) || n < 0 ||
      ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dw) | reinterpret_cast<uintptr_t>(work)) & 15))
    return -10;
  const int vecs = D / 8, segment = emb_segment(n);
  const int segments = n > segment ? (n + segment - 1) / segment : 0;
  float4* partial = static_cast<float4*>(work);
  int* counts = reinterpret_cast<int*>(partial + static_cast<int64_t>(segments) * 2 * vecs * 2);
  int *offsets = counts + V, *cursor = offsets + V, *list = cursor + V, *sorted = list + n;
  if (cudaMemsetAsync(counts, 0, sizeof(int) * static_cast<size_t>(V), stream) != cudaSuccess) return -4;
  const uint4* g = static_cast<const uint4*>(dy);
  if (n > 0) {
    const int grid = (n + 255) / 256;
    emb_count_kernel<<<grid, 256, 0, stream>>>(ids, n, V, counts);
    emb_scan_kernel<<<1, 1024, 0, stream>>>(counts, V, offsets, cursor);
    emb_fill_kernel<<<grid, 256, 0, stream>>>(ids, n, V, cursor, list);
  }
  if (n > kEmbList)
    emb_order_kernel<<<V < 148 * 4 ? V : 148 * 4, kEmbThreads, 0, stream>>>(counts, offsets, list, sorted, n, V);
  if (segments > 0)
    emb_segments_kernel<<<dim3(segments, (vecs + kEmbThreads - 1) / kEmbThreads), kEmbThreads, 0, stream>>>(
        g, ids, counts, offsets, list, sorted, partial, V, vecs, segment);
  emb_rows_kernel<<<V < 148 * 8 ? V : 148 * 8, kEmbThreads, 0, stream>>>(g, counts, offsets, list, sorted, partial,
                                                                         static_cast<uint4*>(dw), V, vecs, segment);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// out = x * g[0], n bf16 values, n a multiple of 8, pointers 16-byte aligned.
extern "C" int axb_scale_bf16(const void* x, const float* g, void* out, int64_t n, cudaStream_t stream) {
  using namespace axb;
  if (n <= 0) return 0;
  if ((n % 8) || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15)) return -10;
  const int64_t want = (n / 8 + 1023) / 1024;
  scale_bf16_kernel<<<static_cast<unsigned>(want < 148 * 8 ? want : 148 * 8), 256, 0, stream>>>(
      static_cast<const uint4*>(x), g, static_cast<uint4*>(out), n / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
