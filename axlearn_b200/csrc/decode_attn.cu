// Decode-time attention over a paged KV cache, and the fused RoPE + cache append that feeds it.
//
// One new token per sequence attends to everything cached for that sequence; every cached K and V byte is used by the
// query heads of one KV head only, so the bound is the rate at which the cache comes out of HBM, and, for few or short
// sequences, the chain length -> page -> K -> softmax -> merge.
//
// One CTA of four warps takes one (KV split, KV head, up to eight of its query heads), so K and V are read once for a
// whole group of query heads.  A warp walks every fourth tile of 16 tokens of its split through a ring of two tiles
// (8 KB of K and V each) that `cp.async` fills ahead of the arithmetic; three CTAs fit an SM.
//   S = Q K^T: rows 0-7 of the m16n8k16 tile are the query heads, K is the B operand (a lane takes 8 neighbouring dims
//   of a key; Q uses the same order of dims).  Four chains of two products each, added in 32 bits.
//   O^T = V^T P^T: 16 dims are the rows, the heads the columns (the scores' accumulators are the B operand as they
//   lie); a lane packs two keys' V entries into one register of the A operand.  P enters as three bf16 terms that add
//   up to its 32 bits.  Up to four (two) heads leave room for two (four) copies of them in the tile: copy i takes term i
//   of P, so that two (one) products do for three.  A tile's products are added to the sums in 32 bits.
// Relative error against 64 bits before the output's rounding, the two CUDA-core kernels that this replaces / this (two
// bf16 terms and one chain: 1.4e-6 throughout): 8 x 16 heads on 16, up to 2000 tokens 2.5e-7 / 2.4e-7; 16 x 32 on 8, up to
// 2048 2.7e-7 / 2.5e-7; 1 x 32 on 8, up to 4000 3.3e-7 / 2.9e-7.  Time of two terms / three (us a launch, inputs beyond
// L2): 18.6 / 18.8, 21.4 / 22.4, 10.8 / 11.2; without the copies 20.0, 23.1 and 11.2.
// The warps meet in shared memory and the KV splits of up to a cluster (8) in distributed shared memory, so there is no
// second launch; more splits leave partials (max, sum, out) for `decode_combine_kernel`.
//
// Measured against the two CUDA-core kernels that this replaces (one query head per 8 lanes, or four query heads on
// four neighbouring KV heads; us a launch, weights of other layers in between, K and V bytes at 6.65 TB/s in brackets):
//   batch  1, 16 heads on 16,  300 tokens  14.3 ->  4.8 (0.4)   batch 16, 32 on  8, up to 2048  64.4 ->  27.1 (13)
//   batch  1, 32 heads on  8, 4000 tokens  20.2 -> 10.0 (2.5)   batch 64, 32 on  8, up to 1000 116.7 ->  42.0 (23)
//   batch  4, 32 heads on  8, 2000 tokens  31.6 -> 12.4 (4.9)   batch 64, 32 on 32, up to 2000 208.8 -> 187.4 (184)
//   batch  8, 16 heads on 16, up to 2000   36.9 -> 24.6 (13)    batch 64, 16 on 16, up to 500   46.1 ->  36.9 (23)
// Three tiles a ring and two CTAs an SM: as fast for few CTAs, 10 % slower for many; registers instead of shared memory
// for the tiles: 1.3 to 2 times as long.  What is left with ragged lengths is that the longest sequence's CTAs finish
// last: a split is a share of its own sequence.
//
// Cache layout: pool [num_pages, page_size, Nkv, H] for K and for V (H = 128), page table
// [B, max_pages] of pool page ids, `lengths[b]` = number of valid tokens (the new token
// included).  A dense cache is the same thing with an identity page table.
//
// `rope_append_kernel` takes the fused QKV projection of the new token(s), rotates q and k
// (interleaved pairs, position = lengths[b] - 1), writes the rotated q out and stores k / v
// into their page slot -- the cache append is not a separate pass.
//
// Reference behaviour being replaced: `PagedKVCache.extend_step` + reference attention over
// gathered pages (axlearn/common/kv_cache/paged_kv_cache.py:22-150) and the Pallas paged
// attention kernel the reference uses on GPU (axlearn/common/flash_attention/gpu_paged_attention.py).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "chain.cuh"
#include "cluster.cuh"
#include "mma_sync.cuh"

namespace axb {

constexpr int kHeadDim = 128;
constexpr int kDecodeThreads = 128;

struct DecodeParams {
  const __nv_bfloat16* q;     // [B, Nq, H]
  const __nv_bfloat16* k_pool;
  const __nv_bfloat16* v_pool;
  const int* page_table;      // [B, max_pages]
  const int* lengths;         // [B]
  float* part_out;            // [B, Nq, splits, H]
  float* part_ml;             // [B, Nq, splits, 2]
  __nv_bfloat16* out;         // [B, Nq, H]
  int num_q_heads, num_kv_heads, page_size, max_pages, splits;
  float scale_log2;           // softmax scale * log2(e)
  float log2_theta;           // kAppend: q is the packed projection [B, Nq + 2 Nkv, H] of the new token, not rotated
};

constexpr int kMmaRows = 8;       // query heads of a CTA
constexpr int kTileKeys = 16;
constexpr int kMaxClusterSplits = 8;

constexpr int kTileBytes = 2 * kTileKeys * kHeadDim * 2;  // K and V
constexpr int kStages = 2;
constexpr int attn_smem_bytes(int rows) {
  const int merge = (4 + 1) * rows * (kHeadDim + 2) * 4, tiles = 4 * kStages * kTileBytes;
  return merge > tiles ? merge : tiles;
}

// term[0] + term[1] + term[2] = (x, y) >= 0, exactly: a 24-bit mantissa is three of 8 bits, cut off from the top.  Every
// term of a positive number is positive (2^-126 stands in for nothing left, as in a fourth term), so that an infinite V
// gives an infinity as in one product, not 0 * infinity.
template <int N>
__device__ __forceinline__ void split_exact(float x, float y, uint32_t (&term)[N]) {
  const float tiny = 1.17549435e-38f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t ux = __float_as_uint(x), uy = __float_as_uint(y);
    term[i] = __byte_perm(ux, uy, 0x7632);
    const float dx = x - __uint_as_float(ux & 0xffff0000u), dy = y - __uint_as_float(uy & 0xffff0000u);
    x = x > 0.f ? fmaxf(dx, tiny) : dx;
    y = y > 0.f ? fmaxf(dy, tiny) : dy;
  }
}

// 16 bytes to shared memory, zeros when `ok` is false (`src` is not read then).
__device__ __forceinline__ void cp16_or_zero(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

// The pair (2i, 2i + 1) of a head turned by `pos * theta^(-2i / H)`.
__device__ __forceinline__ __nv_bfloat162 turned(__nv_bfloat162 x, int i, int pos, float log2_theta) {
  const float2 f = __bfloat1622float2(x);
  const float inv = exp2f(-log2_theta * (2.f * i) / kHeadDim);
  float sn, cs;
  sincosf(static_cast<float>(pos) * inv, &sn, &cs);
  return __floats2bfloat162_rn(f.x * cs - f.y * sn, f.y * cs + f.x * sn);
}

// kAppend: what rope_append_kernel does ahead of the attention happens here.  A warp turns its query heads in registers; the
// warp whose tile holds the new token turns its key, stores key and value into their page slot and puts them into the
// tile itself, so nobody reads the slot.  One launch and one hand-over less a layer; us, two launches / one, chained:
//   batch 1, 16 heads on 16, 308 tokens 5.6 / 4.9       batch  1, 32 heads on  8, 2000 tokens   8.1 /   7.3
//   batch 16, 32 on 8, 2056 tokens 28.3 / 27.4          batch 64, 32 heads on 32, 1000 tokens 156.5 / 154.0
template <bool kCluster, int kCopies, bool kAppend>
__global__ void __launch_bounds__(kDecodeThreads)
decode_attn_kernel(DecodeParams p) {
  chain_link();
  extern __shared__ __align__(16) float s_part[];  // the warps' tiles; then 4 warps and the CTA: [rows][kHeadDim] sums,
                                                   // [rows] maxima, [rows] weights
  const int split = blockIdx.x;
  const int group = p.num_q_heads / p.num_kv_heads;
  const int parts = (group + kMmaRows - 1) / kMmaRows;
  const int kvh = blockIdx.y / parts;
  const int first = blockIdx.y % parts * kMmaRows;
  const int rows = min(kMmaRows, group - first);
  const int qh0 = kvh * group + first;
  const int b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = lane >> 2, c = lane & 3;
  constexpr int kHeads = kMmaRows / kCopies, kPasses = (3 + kCopies - 1) / kCopies;
  const int head = r % kHeads, copy = r / kHeads;
  const int len = p.lengths[b];
  const int tiles = (len + kTileKeys - 1) / kTileKeys;
  const int per_split = (tiles + p.splits - 1) / p.splits;
  const int hi = min(tiles, (split + 1) * per_split);
  const int* table = p.page_table + static_cast<int64_t>(b) * p.max_pages;

  // Slot (token row of the pools) of key `lane & 15` of a tile, -1 beyond the sequence.
  auto slot_of = [&](int tile) {
    const int t = tile * kTileKeys + (lane & 15);
    if (tile >= hi || t >= (kAppend ? len - 1 : len)) return -1;
    return table[t / p.page_size] * p.page_size + t % p.page_size;
  };

  const int64_t row_stride = static_cast<int64_t>(p.num_kv_heads) * kHeadDim;
  const int head_off = kvh * kHeadDim + (lane & 15) * 8;
  uint8_t* ring = reinterpret_cast<uint8_t*>(s_part) + warp * kStages * kTileBytes;
  const uint32_t ring_addr = sptr(ring);
  // A row of a tile is 16 chunks of 16 bytes.  Chunks are swapped within their row so that the eight lanes of a
  // 128-byte phase hit all banks: they read two neighbouring rows of K, and every second row of V.
  auto k_chunk = [](int row, int chunk) { return row * 256 + ((chunk ^ ((row & 1) << 2)) << 4); };
  auto v_chunk = [](int row, int chunk) { return row * 256 + ((chunk ^ (row & 6)) << 4); };
  auto load_tile = [&](int stage, int slot) {  // half a warp per row: two rows of K or V an instruction
    const uint32_t dst = ring_addr + stage * kTileBytes;
#pragma unroll
    for (int i = 0; i < kTileKeys / 2; ++i) {
      const int row = 2 * i + (lane >> 4);
      const int at = __shfl_sync(0xffffffffu, slot, row);
      const int64_t off = (at < 0 ? 0 : at) * row_stride + head_off;
      cp16_or_zero(dst + k_chunk(row, lane & 15), p.k_pool + off, at >= 0);
      cp16_or_zero(dst + kTileBytes / 2 + v_chunk(row, lane & 15), p.v_pool + off, at >= 0);
    }
  };

  constexpr int kStep = kDecodeThreads / 32;
  int tile = split * per_split + warp;
  int slots[kStages];
#pragma unroll
  for (int i = 0; i < kStages; ++i) slots[i] = slot_of(tile + i * kStep);
#pragma unroll
  for (int i = 0; i < kStages; ++i) {
    if (tile + i * kStep < hi) load_tile(i, slots[i]);
    cp_commit();
  }
  int slot = slot_of(tile + kStages * kStep);
  const int q_heads = kAppend ? p.num_q_heads + 2 * p.num_kv_heads : p.num_q_heads;  // of a row of q
  // The new token's key and value: lane l has dims 4 l .. 4 l + 3.
  const int new_tile = (len - 1) / kTileKeys;
  const bool appends = kAppend && len > 0 && new_tile >= split * per_split && new_tile < hi &&
                       (new_tile - split * per_split) % kStep == warp;
  uint2 new_k = make_uint2(0, 0), new_v = make_uint2(0, 0);
  if (appends) {
    const __nv_bfloat16* src =
        p.q + (static_cast<int64_t>(b) * q_heads + p.num_q_heads + kvh) * kHeadDim + lane * 4;
    new_k = *reinterpret_cast<const uint2*>(src);
    new_v = *reinterpret_cast<const uint2*>(src + static_cast<int64_t>(p.num_kv_heads) * kHeadDim);
  }
  uint4 q[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int64_t row = static_cast<int64_t>(b) * q_heads + qh0 + head;
    q[j] = head < rows ? *reinterpret_cast<const uint4*>(p.q + row * kHeadDim + j * 32 + c * 8) : make_uint4(0, 0, 0, 0);
  }
  if constexpr (kAppend) {
    const int pos = len - 1;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&q[j]);
#pragma unroll
      for (int u = 0; u < 4; ++u) pairs[u] = turned(pairs[u], j * 16 + c * 4 + u, pos, p.log2_theta);
    }
    if (appends) {
      __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&new_k);
#pragma unroll
      for (int u = 0; u < 2; ++u) pairs[u] = turned(pairs[u], lane * 2 + u, pos, p.log2_theta);
      if (first == 0) {  // (the other parts of a large group have the same)
        const int64_t slot = static_cast<int64_t>(table[pos / p.page_size]) * p.page_size + pos % p.page_size;
        const int64_t at = slot * row_stride + kvh * kHeadDim + lane * 4;
        *reinterpret_cast<uint2*>(const_cast<__nv_bfloat16*>(p.k_pool) + at) = new_k;
        *reinterpret_cast<uint2*>(const_cast<__nv_bfloat16*>(p.v_pool) + at) = new_v;
      }
    }
  }
  float m = -INFINITY, l = 0.f;
  float acc[8][4];  // [16 dims][columns 2c, 2c + 1]
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;

  int stage = 0;
  for (; tile < hi; tile += kStep) {
    cp_wait_group<kStages - 1>();
    __syncwarp();
    const uint8_t* kt = ring + stage * kTileBytes;
    const uint8_t* vt = kt + kTileBytes / 2;
    if (appends && tile == new_tile) {
      const int row = (len - 1) % kTileKeys, half = (lane & 1) * 8;
      uint8_t* to = ring + stage * kTileBytes;
      *reinterpret_cast<uint2*>(to + k_chunk(row, lane >> 1) + half) = new_k;
      *reinterpret_cast<uint2*>(to + kTileBytes / 2 + v_chunk(row, lane >> 1) + half) = new_v;
      __syncwarp();
    }
    float s[4];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      float part[4][4] = {};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint4 k = *reinterpret_cast<const uint4*>(kt + k_chunk(n * 8 + r, j * 4 + c));
        const uint32_t a0[4] = {q[j].x, 0u, q[j].y, 0u}, a1[4] = {q[j].z, 0u, q[j].w, 0u};
        mma(part[(2 * j) % 4], a0, k.x, k.y);
        mma(part[(2 * j + 1) % 4], a1, k.z, k.w);
      }
      const int t = tile * kTileKeys + n * 8 + 2 * c;
      s[2 * n] = t < len ? ((part[0][0] + part[2][0]) + (part[1][0] + part[3][0])) * p.scale_log2 : -INFINITY;
      s[2 * n + 1] = t + 1 < len ? ((part[0][1] + part[2][1]) + (part[1][1] + part[3][1])) * p.scale_log2 : -INFINITY;
    }
    float top = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
    const float m_new = fmaxf(m, top);
    if (__any_sync(0xffffffffu, m_new != m)) {
      const float corr = m_new == -INFINITY ? 1.f : exp2f(m - m_new);
      l *= corr;
      const float c0 = __shfl_sync(0xffffffffu, corr, 8 * c), c1 = __shfl_sync(0xffffffffu, corr, 8 * c + 4);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        acc[i][0] *= c0;
        acc[i][1] *= c1;
        acc[i][2] *= c0;
        acc[i][3] *= c1;
      }
      m = m_new;
    }
    // exp2(-inf - -inf) would be NaN: a row that has seen no finite score keeps zeros.
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] = m == -INFINITY ? 0.f : exp2f(s[i] - m);
    l += (s[0] + s[1]) + (s[2] + s[3]);
    constexpr int kTerms = kPasses * kCopies;
    uint32_t t0[kTerms], t1[kTerms], p0[kPasses], p1[kPasses];  // all terms; those of this copy
    split_exact(s[0], s[1], t0);
    split_exact(s[2], s[3], t1);
#pragma unroll
    for (int i = 0; i < kPasses; ++i) {
      p0[i] = t0[i * kCopies], p1[i] = t1[i * kCopies];
#pragma unroll
      for (int u = 1; u < kCopies; ++u)
        if (copy == u) p0[i] = t0[i * kCopies + u], p1[i] = t1[i * kCopies + u];
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      uint32_t v[4][4];  // keys 2c, 2c + 1, 8 + 2c, 8 + 2c + 1: the columns of P that this lane holds
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<uint4*>(v[i]) =
            *reinterpret_cast<const uint4*>(vt + v_chunk((i >> 1) * 8 + 2 * c + (i & 1), j * 8 + r));
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t a[4] = {__byte_perm(v[0][e], v[1][e], 0x5410), __byte_perm(v[0][e], v[1][e], 0x7632),
                               __byte_perm(v[2][e], v[3][e], 0x5410), __byte_perm(v[2][e], v[3][e], 0x7632)};
        float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = kPasses - 1; i >= 0; --i) mma(o, a, p0[i], p1[i]);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j * 4 + e][i] += o[i];
      }
    }
    __syncwarp();  // the stage has been read
    if (tile + kStages * kStep < hi) load_tile(stage, slot);
    cp_commit();
    slot = slot_of(tile + (kStages + 1) * kStep);
    if (++stage == kStages) stage = 0;
  }
  cp_wait_all();
  __syncthreads();  // the merge buffers overlay the tiles
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);

  // The copies' terms of P meet.
#pragma unroll
  for (int off = 2; off >= 4 / kCopies; off /= 2) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][e] += __shfl_xor_sync(0xffffffffu, acc[i][e], off);
  }

  // Rows r and r + 8 of MMA tile (j, e) are dims 64 j + 8 r + 2 e and the next.
  const int per_warp = rows * kHeadDim;
  float* s_m = s_part + 5 * per_warp;
  float* s_l = s_m + 5 * rows;
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    if (2 * c + n >= rows) break;
    float* dst = s_part + warp * per_warp + (2 * c + n) * kHeadDim + r * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      *reinterpret_cast<float2*>(dst + (i >> 2) * 64 + (i & 3) * 2) = make_float2(acc[i][n], acc[i][2 + n]);
  }
  if (r < rows && c == 0) {
    s_m[warp * rows + r] = m;
    s_l[warp * rows + r] = l;
  }
  __syncthreads();
  // Thread d owns output dim d.
  const int d = threadIdx.x;
  for (int g = 0; g < rows; ++g) {
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) mm = fmaxf(mm, s_m[w * rows + g]);
    float ll = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float f = mm == -INFINITY ? 0.f : exp2f(s_m[w * rows + g] - mm);
      ll += s_l[w * rows + g] * f;
      o += s_part[w * per_warp + g * kHeadDim + d] * f;
    }
    const int64_t row = static_cast<int64_t>(b) * p.num_q_heads + qh0 + g;
    if (p.splits == 1) {
      p.out[row * kHeadDim + d] = __float2bfloat16(ll > 0.f ? o / ll : 0.f);
    } else if (kCluster) {
      s_part[4 * per_warp + g * kHeadDim + d] = o;
      if (d == 0) {
        s_m[4 * rows + g] = mm;
        s_l[4 * rows + g] = ll;
      }
    } else {
      p.part_out[(row * p.splits + split) * kHeadDim + d] = o;
      if (d == 0) {
        p.part_ml[(row * p.splits + split) * 2] = mm;
        p.part_ml[(row * p.splits + split) * 2 + 1] = ll;
      }
    }
  }
  if constexpr (kCluster) {
    cluster_sync_all();
    for (int g = split; g < rows; g += p.splits) {
      float mv[kMaxClusterSplits], lv[kMaxClusterSplits], ov[kMaxClusterSplits];
#pragma unroll
      for (int s = 0; s < kMaxClusterSplits; ++s) {
        const bool have = s < p.splits;
        mv[s] = have ? ld_cluster_f32(sptr(s_m + 4 * rows + g), s) : -INFINITY;
        lv[s] = have ? ld_cluster_f32(sptr(s_l + 4 * rows + g), s) : 0.f;
        ov[s] = have ? ld_cluster_f32(sptr(s_part + 4 * per_warp + g * kHeadDim + d), s) : 0.f;
      }
      float mm = -INFINITY;
#pragma unroll
      for (int s = 0; s < kMaxClusterSplits; ++s) mm = fmaxf(mm, mv[s]);
      float ll = 0.f, o = 0.f;
#pragma unroll
      for (int s = 0; s < kMaxClusterSplits; ++s) {
        const float f = mm == -INFINITY ? 0.f : exp2f(mv[s] - mm);
        ll += lv[s] * f;
        o += ov[s] * f;
      }
      p.out[(static_cast<int64_t>(b) * p.num_q_heads + qh0 + g) * kHeadDim + d] =
          __float2bfloat16(ll > 0.f ? o / ll : 0.f);
    }
    cluster_sync_all();  // a CTA's shared memory outlives its readers
  }
}

template <bool kCluster, int kCopies, bool kAppend>
static int launch_attn(const DecodeParams& p, dim3 grid, int rows, cudaStream_t stream) {
  constexpr auto kernel = decode_attn_kernel<kCluster, kCopies, kAppend>;
  static const cudaError_t configured = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                             attn_smem_bytes(kMmaRows));
  if (configured != cudaSuccess) return -3;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {grid.x, 1, 1};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kDecodeThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(attn_smem_bytes(rows));
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = static_cast<unsigned>(chain_attribute(attr, kCluster ? 1 : 0));
  return cudaLaunchKernelEx(&cfg, kernel, p) == cudaSuccess ? 0 : -4;
}

__global__ void __launch_bounds__(kHeadDim)
decode_combine_kernel(const float* part_out, const float* part_ml, __nv_bfloat16* out, int splits) {
  chain_link();
  const int64_t row = blockIdx.x;  // b * Nq + head
  const int d = threadIdx.x;
  float mm = -INFINITY;
  for (int s = 0; s < splits; ++s) mm = fmaxf(mm, part_ml[(row * splits + s) * 2]);
  float ll = 0.f, o = 0.f;
  for (int s = 0; s < splits; ++s) {
    const float ms = part_ml[(row * splits + s) * 2];
    const float c = (mm == -INFINITY) ? 0.f : exp2f(ms - mm);
    ll += part_ml[(row * splits + s) * 2 + 1] * c;
    o += part_out[(row * splits + s) * kHeadDim + d] * c;
  }
  out[row * kHeadDim + d] = __float2bfloat16(ll > 0.f ? o / ll : 0.f);
}

// qkv: [B, (Nq + 2 Nkv) * H] (q heads, then k heads, then v heads).  One CTA per (b, head);
// thread i rotates the pair (2i, 2i+1).
__global__ void __launch_bounds__(kHeadDim / 2)
rope_append_kernel(const __nv_bfloat16* qkv, __nv_bfloat16* q_out, __nv_bfloat16* k_pool, __nv_bfloat16* v_pool,
                   const int* page_table, const int* lengths, int num_q_heads, int num_kv_heads, int page_size,
                   int max_pages, float log2_theta, int apply_rope) {
  chain_link();
  const int b = blockIdx.y;
  const int head = blockIdx.x;  // 0..Nq+2Nkv-1
  const int i = threadIdx.x;
  const int total_heads = num_q_heads + 2 * num_kv_heads;
  const int pos = lengths[b] - 1;
  const __nv_bfloat162 x =
      reinterpret_cast<const __nv_bfloat162*>(qkv + (static_cast<int64_t>(b) * total_heads + head) * kHeadDim)[i];
  float2 f = __bfloat1622float2(x);
  const bool is_v = head >= num_q_heads + num_kv_heads;
  if (!is_v && apply_rope) {
    // inv_freq = theta^(-2i/H)
    const float inv = exp2f(-log2_theta * (2.f * i) / kHeadDim);
    float sn, cs;
    sincosf(static_cast<float>(pos) * inv, &sn, &cs);
    f = make_float2(f.x * cs - f.y * sn, f.y * cs + f.x * sn);
  }
  const __nv_bfloat162 y = __floats2bfloat162_rn(f.x, f.y);
  if (head < num_q_heads) {
    reinterpret_cast<__nv_bfloat162*>(q_out + (static_cast<int64_t>(b) * num_q_heads + head) * kHeadDim)[i] = y;
    return;
  }
  const int kvh = is_v ? head - num_q_heads - num_kv_heads : head - num_q_heads;
  const int page = page_table[static_cast<int64_t>(b) * max_pages + pos / page_size];
  const int64_t slot = static_cast<int64_t>(page) * page_size + pos % page_size;
  __nv_bfloat16* dst = (is_v ? v_pool : k_pool) + (slot * num_kv_heads + kvh) * kHeadDim;
  reinterpret_cast<__nv_bfloat162*>(dst)[i] = y;
}

}  // namespace axb

// Scratch needed by axb_decode_attn: floats.  Up to a cluster's splits meet without any.
extern "C" int64_t axb_decode_attn_scratch_floats(int B, int num_q_heads, int splits) {
  if (splits <= axb::kMaxClusterSplits) return 0;
  return static_cast<int64_t>(B) * num_q_heads * splits * (axb::kHeadDim + 2);
}

namespace axb {

template <bool kAppend>
static int decode_attn(const void* q, const void* k_pool, const void* v_pool, const int* page_table, const int* lengths,
                       void* out, float* scratch, int B, int num_q_heads, int num_kv_heads, int head_dim, int page_size,
                       int max_pages, int splits, float theta, float softmax_scale, cudaStream_t stream) {
  if (head_dim != kHeadDim || page_size % 4 || num_q_heads % num_kv_heads || splits < 1) return -10;
  if (B <= 0) return 0;
  const int g = num_q_heads / num_kv_heads;
  DecodeParams p;
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k_pool = static_cast<const __nv_bfloat16*>(k_pool);
  p.v_pool = static_cast<const __nv_bfloat16*>(v_pool);
  p.page_table = page_table;
  p.lengths = lengths;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.part_out = scratch;
  p.part_ml = scratch == nullptr ? nullptr
                                 : scratch + static_cast<int64_t>(B) * num_q_heads * splits * kHeadDim;
  if (splits > kMaxClusterSplits && scratch == nullptr) return -10;
  p.num_q_heads = num_q_heads;
  p.num_kv_heads = num_kv_heads;
  p.page_size = page_size;
  p.max_pages = max_pages;
  p.splits = splits;
  p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.log2_theta = log2f(theta);
  const bool cluster = splits > 1 && splits <= kMaxClusterSplits;
  const dim3 grid(splits, num_kv_heads * ((g + kMmaRows - 1) / kMmaRows), B);
  const int rows = g < kMmaRows ? g : kMmaRows;
  const auto launch = rows <= 2   ? (cluster ? launch_attn<true, 4, kAppend> : launch_attn<false, 4, kAppend>)
                      : rows <= 4 ? (cluster ? launch_attn<true, 2, kAppend> : launch_attn<false, 2, kAppend>)
                                  : (cluster ? launch_attn<true, 1, kAppend> : launch_attn<false, 1, kAppend>);
  const int rc = launch(p, grid, rows, stream);
  if (rc != 0) return rc;
  if (splits > kMaxClusterSplits)
    launch_chained(decode_combine_kernel, B * num_q_heads, kHeadDim, 0, stream, p.part_out, p.part_ml, p.out, splits);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace axb

// Returns 0 on success, -10 for unsupported shapes (H != 128, page_size % 4, group size).
extern "C" int axb_decode_attn(const void* q, const void* k_pool, const void* v_pool, const int* page_table,
                               const int* lengths, void* out, float* scratch, int B, int num_q_heads,
                               int num_kv_heads, int head_dim, int page_size, int max_pages, int splits,
                               float softmax_scale, cudaStream_t stream) {
  return axb::decode_attn<false>(q, k_pool, v_pool, page_table, lengths, out, scratch, B, num_q_heads, num_kv_heads, head_dim,
                                 page_size, max_pages, splits, 1.f, softmax_scale, stream);
}

// axb_rope_append_paged and axb_decode_attn in one launch: qkv [B, (Nq + 2 Nkv) * H] of the token at position lengths - 1.
extern "C" int axb_rope_decode_attn(const void* qkv, void* k_pool, void* v_pool, const int* page_table, const int* lengths,
                                    void* out, float* scratch, int B, int num_q_heads, int num_kv_heads, int head_dim,
                                    int page_size, int max_pages, int splits, float theta, float softmax_scale,
                                    cudaStream_t stream) {
  return axb::decode_attn<true>(qkv, k_pool, v_pool, page_table, lengths, out, scratch, B, num_q_heads, num_kv_heads, head_dim,
                                page_size, max_pages, splits, theta, softmax_scale, stream);
}

extern "C" int axb_rope_append_paged(const void* qkv, void* q_out, void* k_pool, void* v_pool,
                                     const int* page_table, const int* lengths, int B, int num_q_heads,
                                     int num_kv_heads, int head_dim, int page_size, int max_pages,
                                     float theta, int apply_rope, cudaStream_t stream) {
  using namespace axb;
  if (head_dim != kHeadDim) return -10;
  if (B <= 0) return 0;
  dim3 grid(num_q_heads + 2 * num_kv_heads, B);
  launch_chained(rope_append_kernel, grid, kHeadDim / 2, 0, stream, static_cast<const __nv_bfloat16*>(qkv),
                 static_cast<__nv_bfloat16*>(q_out), static_cast<__nv_bfloat16*>(k_pool),
                 static_cast<__nv_bfloat16*>(v_pool), page_table, lengths, num_q_heads, num_kv_heads, page_size,
                 max_pages, log2f(theta), apply_rope);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

namespace axb {

// Whole prompts: qkv [B * T, (Nq + 2 Nkv) * H] of one projection.  Rotates q in place and puts rotated k and plain v into
// the sequences' runs of the pools (sequence b at token row b * pool_rows), where attention reads them: one pass over
// the projection, which replaces copies of q, k and v out of it, two rotations and two copies into the pools
// (a layer's 16384 x 48 heads: 80 us against 445, of 61 at the copy rate; 333 x 24 heads: 3 us against 18).  A thread
// keeps its (sin, cos) pairs in registers and has four 16-byte loads in flight.
constexpr int kRopeThreads = 256;

__global__ void __launch_bounds__(kRopeThreads)
rope_append_prompt_kernel(uint4* __restrict__ qkv, uint4* __restrict__ k_pool, uint4* __restrict__ v_pool,
                          const float4* __restrict__ table, int64_t rows, int T, int64_t pool_rows, int num_q_heads,
                          int num_kv_heads) {
  constexpr int kVecs = kHeadDim / 8, kHeads = kRopeThreads / kVecs, kFlight = 4;
  const int pv = threadIdx.x % kVecs, h0 = threadIdx.x / kVecs;
  const int heads = num_q_heads + 2 * num_kv_heads;
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const int64_t b = row / T;
    const int t = static_cast<int>(row - b * T);
    const float4* tab = table + static_cast<int64_t>(t) * (kHeadDim / 4) + pv * 2;
    const float4 sc0 = __ldg(tab), sc1 = __ldg(tab + 1);  // (s0, c0, s1, c1), (s2, c2, s3, c3)
    const float sn[4] = {sc0.x, sc0.z, sc1.x, sc1.z}, cs[4] = {sc0.y, sc0.w, sc1.y, sc1.w};
    uint4* src = qkv + row * heads * kVecs + pv;
    const int64_t slot = (b * pool_rows + t) * num_kv_heads;
    for (int n0 = h0; n0 < heads; n0 += kHeads * kFlight) {
      uint4 v[kFlight];
#pragma unroll
      for (int u = 0; u < kFlight; ++u)
        if (n0 + u * kHeads < heads) v[u] = src[(n0 + u * kHeads) * kVecs];
#pragma unroll
      for (int u = 0; u < kFlight; ++u) {
        const int n = n0 + u * kHeads;
        if (n >= heads) break;
        if (n >= num_q_heads + num_kv_heads) {
          v_pool[(slot + n - num_q_heads - num_kv_heads) * kVecs + pv] = v[u];
          continue;
        }
        uint32_t* w = reinterpret_cast<uint32_t*>(&v[u]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 f = unpack2(w[q]);
          w[q] = pack2(f.x * cs[q] - f.y * sn[q], f.y * cs[q] + f.x * sn[q]);
        }
        if (n < num_q_heads)
          src[n * kVecs] = v[u];
        else
          k_pool[(slot + n - num_q_heads) * kVecs + pv] = v[u];
      }
    }
  }
}

__device__ __forceinline__ float silu_times(float g, float u) { return g / (1.f + __expf(-g)) * u; }

// out[r, c] = silu(gu[r, c]) * gu[r, F + c] for gu = [rows, 2F] (gate | up packed by one GEMM).
__global__ void swiglu_packed_kernel(const __nv_bfloat16* gu, __nv_bfloat16* out, int64_t rows, int F) {
  chain_link();
  const int64_t total = rows * (F / 2);
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / (F / 2);
    const int c = static_cast<int>(i % (F / 2)) * 2;
    const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(gu + r * 2 * F + c));
    const float2 u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(gu + r * 2 * F + F + c));
    *reinterpret_cast<__nv_bfloat162*>(out + r * F + c) = __floats2bfloat162_rn(silu_times(g.x, u.x), silu_times(g.y, u.y));
  }
}

// The same, 16 bytes a load, for F % 8 == 0 and 16-byte aligned operands: a block takes 256 vectors of one row, so no
// index is divided, and a thread has four loads in flight.  16384 x 14336: 474 -> 221 us (212 at the copy rate).
constexpr int kSwigluThreads = 256, kSwigluVecs = 2;

__global__ void __launch_bounds__(kSwigluThreads)
swiglu_packed_vec_kernel(const uint4* gu, uint4* out, int64_t rows, int vecs) {
  chain_link();
  const int c0 = blockIdx.x * (kSwigluThreads * kSwigluVecs) + threadIdx.x;
  for (int64_t row = blockIdx.y; row < rows; row += gridDim.y) {
    uint4 g[kSwigluVecs], u[kSwigluVecs];
#pragma unroll
    for (int i = 0; i < kSwigluVecs; ++i) {
      const int c = c0 + i * kSwigluThreads;
      if (c < vecs) {
        g[i] = gu[row * 2 * vecs + c];
        u[i] = gu[row * 2 * vecs + vecs + c];
      }
    }
#pragma unroll
    for (int i = 0; i < kSwigluVecs; ++i) {
      const int c = c0 + i * kSwigluThreads;
      if (c >= vecs) break;
      uint32_t* gw = reinterpret_cast<uint32_t*>(&g[i]);
      const uint32_t* uw = reinterpret_cast<const uint32_t*>(&u[i]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 a = unpack2(gw[k]), b = unpack2(uw[k]);
        gw[k] = pack2(silu_times(a.x, b.x), silu_times(a.y, b.y));
      }
      out[row * vecs + c] = g[i];
    }
  }
}

}  // namespace axb

// qkv [B * T, (Nq + 2 Nkv) * 128], pools at the first sequence's run, `pool_rows` token rows a sequence (>= T); `table` of
// axb_rope_table.  Pointers 16-byte aligned.
extern "C" int axb_rope_append_prompt(void* qkv, void* k_pool, void* v_pool, const float* table, int B, int T,
                                      int64_t pool_rows, int num_q_heads, int num_kv_heads, int head_dim,
                                      cudaStream_t stream) {
  using namespace axb;
  const uintptr_t align = reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(k_pool) |
                          reinterpret_cast<uintptr_t>(v_pool) | reinterpret_cast<uintptr_t>(table);
  if (head_dim != kHeadDim || pool_rows < T || num_q_heads <= 0 || num_kv_heads <= 0 || (align & 15)) return -10;
  const int64_t rows = static_cast<int64_t>(B) * T;
  if (rows <= 0) return 0;
  const int64_t grid = rows < 148 * 16 ? rows : 148 * 16;
  rope_append_prompt_kernel<<<static_cast<unsigned>(grid), kRopeThreads, 0, stream>>>(
      static_cast<uint4*>(qkv), static_cast<uint4*>(k_pool), static_cast<uint4*>(v_pool),
      reinterpret_cast<const float4*>(table), rows, T, pool_rows, num_q_heads, num_kv_heads);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int axb_swiglu_packed(const void* gu, void* out, int64_t rows, int F, cudaStream_t stream) {
  using namespace axb;
  if (F % 2) return -10;
  const int64_t total = rows * (F / 2);
  if (total <= 0) return 0;
  if (F % 8 == 0 && !((reinterpret_cast<uintptr_t>(gu) | reinterpret_cast<uintptr_t>(out)) & 15)) {
    const int vecs = F / 8;
    const dim3 grid((vecs + kSwigluThreads * kSwigluVecs - 1) / (kSwigluThreads * kSwigluVecs),
                    static_cast<unsigned>(rows < 65535 ? rows : 65535));
    launch_chained(swiglu_packed_vec_kernel, grid, kSwigluThreads, 0, stream, static_cast<const uint4*>(gu),
                   static_cast<uint4*>(out), rows, vecs);
    return cudaGetLastError() == cudaSuccess ? 0 : -4;
  }
  int64_t ctas = (total + 255) / 256;
  if (ctas > 148 * 8) ctas = 148 * 8;
  launch_chained(swiglu_packed_kernel, static_cast<unsigned>(ctas), 256, 0, stream, static_cast<const __nv_bfloat16*>(gu),
                 static_cast<__nv_bfloat16*>(out), rows, F);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
