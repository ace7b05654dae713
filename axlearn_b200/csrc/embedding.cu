// Gradient of an embedding table: dw[v, :] = sum over the tokens with id v of dy[token, :], summed in 32 bits in token
// order and rounded once.  The bound is the table's own size (every row is written, most of them with zeros), so there is
// no pass that clears it and no sort: ids are counted per row, the rows' lists are filled in any order, and whoever sums
// a row puts its short list in order first.  A row with more than kEmbList tokens finds them by walking the ids in order.
//
// 8192 tokens, 32768 x 4096: 76 us for the rows (51 at the copy rate), 31 for the offsets and about 10 for the two passes
// over the ids, against 780 for the operator (fill, radix sort, partial sums).  A gradient's scaling by the loss's own
// gradient, 32768 x 4096: 95 us against 190.
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

// A CTA takes every gridDim-th row of the table, its threads 8 columns each.
__global__ void __launch_bounds__(kEmbThreads)
emb_rows_kernel(const uint4* __restrict__ dy, const int64_t* __restrict__ ids, const int* __restrict__ counts,
                const int* __restrict__ offsets, const int* __restrict__ list, uint4* __restrict__ dw, int n, int V,
                int vecs) {
  __shared__ int s_tok[kEmbThreads];
  __shared__ int s_warp[kEmbThreads / 32];
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
        out[c] = make_uint4(pack2(acc[0], acc[1]), pack2(acc[2], acc[3]), pack2(acc[4], acc[5]), pack2(acc[6], acc[7]));
      }
      __syncthreads();
      continue;
    }
    // A frequent id: 256 ids at a time, those of this row in order into shared memory.
    for (int c0 = 0; c0 < vecs; c0 += kEmbThreads) {
      const int c = c0 + tid;
      float acc[8] = {};
      for (int i0 = 0; i0 < n; i0 += kEmbThreads) {
        const bool hit = i0 + tid < n && ids[i0 + tid] == v;
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) s_warp[warp] = __popc(m);
        __syncthreads();
        int before = 0, total = 0;
#pragma unroll
        for (int w = 0; w < kEmbThreads / 32; ++w) {
          before += w < warp ? s_warp[w] : 0;
          total += s_warp[w];
        }
        if (hit) s_tok[before + __popc(m & ((1u << lane) - 1))] = i0 + tid;
        __syncthreads();
        if (c < vecs) {
#pragma unroll 4
          for (int j = 0; j < total; ++j) emb_add(acc, __ldg(dy + static_cast<int64_t>(s_tok[j]) * vecs + c));
        }
        __syncthreads();
      }
      if (c < vecs)
        out[c] = make_uint4(pack2(acc[0], acc[1]), pack2(acc[2], acc[3]), pack2(acc[4], acc[5]), pack2(acc[6], acc[7]));
    }
  }
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

// dw [V, D] (bf16, every row written) from dy [n, D] and ids [n]; ids outside [0, V) are left out.  `work`: n + 3 V ints.
extern "C" int axb_embedding_bwd(const void* dy, const int64_t* ids, void* dw, int* work, int n, int V, int D,
                                 cudaStream_t stream) {
  using namespace axb;
  if (V <= 0 || D <= 0 || (D % 8) || n < 0 ||
      ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dw)) & 15))
    return -10;
  int *counts = work, *offsets = work + V, *cursor = offsets + V, *list = cursor + V;
  if (cudaMemsetAsync(counts, 0, sizeof(int) * static_cast<size_t>(V), stream) != cudaSuccess) return -4;
  if (n > 0) {
    const int grid = (n + 255) / 256;
    emb_count_kernel<<<grid, 256, 0, stream>>>(ids, n, V, counts);
    emb_scan_kernel<<<1, 1024, 0, stream>>>(counts, V, offsets, cursor);
    emb_fill_kernel<<<grid, 256, 0, stream>>>(ids, n, V, cursor, list);
  }
  const int grid = V < 148 * 8 ? V : 148 * 8;
  emb_rows_kernel<<<grid, kEmbThreads, 0, stream>>>(static_cast<const uint4*>(dy), ids, counts, offsets, list,
                                                    static_cast<uint4*>(dw), n, V, D / 8);
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
