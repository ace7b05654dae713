// Skinny bf16 GEMM for sm_100a: C[M, N] = X[M, K] * W[K, N] (+ C) with M <= 128 -- the products of a decoding
// step and of short prompts.  Every weight byte is used once, so the bound is the rate at which W comes
// out of HBM; the shape of the kernel follows from that:
//
//   * operands are swapped: 128 output FEATURES are the M side of the tcgen05 tile and the (16 .. 128) rows of X
//     its N side, so a pipeline stage is 16 KB of weights and 2 KB of X per 16 rows, not 16 KB of mostly
//     zero-filled X rows beside 8 KB of weights (the 128-row tile of gemm.cu);
//   * two CTAs fit one SM (<= 113 KB each), so about 190 KB of weights per SM are on their way at any time and the
//     prologue / epilogue of one CTA runs under the stream of the other;
//   * the K slices of a tile are the CTAs of one cluster: partial sums meet through distributed shared
//     memory (no fp32 workspace in global memory, no counters, no fence), each CTA finishing every
//     split-th row of X in a fixed order, so results are reproducible.
//
// Warp 0 streams tiles with TMA, one thread of warp 1 issues the MMAs, warps 2-5 read the accumulator (thread =
// feature, so a warp stores 32 neighbouring features of a row).  Either layout of W is read in place.
//
// In a chain of small products neither HBM nor the L2 is the bound (1 x 2048 x 2048 took 4.8 us with its weights in HBM
// and 4.6 with them in the L2) but what a launch does one after the other, so for up to 32 rows:
//   * a stage is two k-blocks (up to 16 rows): the thread that issues the MMAs spends 40 clocks on each and about 110
//     on a stage's wait and commit; a stage that is not filled again is not committed;
//   * partial sums are stored into the inbox of the CTA that finishes their row (behind the stages), which then reads
//     its own shared memory: one cluster barrier behind the products and no round trip between SMs, where fetching them
//     took both and a second barrier (2.0 -> 1.0 us);
//   * C is read while the products run, and no CTA looks at the status word in memory before it leaves (0.6 us).
//
// us, chained launches with weights from HBM, before these / now, the weights alone at 6.55 TB/s in brackets:
//   1 x 512 x 2048    4.5 /  3.4 (0.3)     1 x 2048 x 2048  4.8 /  3.6 (1.3)     1 x 2048 x 8192  9.0 / 7.7 (5.1)
//   1 x 16384 x 2048 12.7 / 11.3 (10.2)   16 x 4096 x 4096  9.4 /  7.9 (5.1)    16 x 4096 x 14336 22.8 / 19.9 (17.9)
// Separate launches, this file's first form (64-column tiles with a split-K workspace before it in brackets) and the
// library:
//  16 x 28672 x 4096 37.0 (38.8) / 37.1    64 x 4096 x 11008 21.1 (26.4) / 18.1   64 x 32768 x 4096 49.2 (49.4) / 46.8
// Half tiles (64 features, twice the CTAs) were no faster: an MMA costs its issuer the same 40 clocks.
#include <atomic>

#include "chain.cuh"
#include "cluster.cuh"
#include "host_utils.cuh"
#include "sm100.cuh"

namespace axb {

constexpr int kSkTile = 128;  // features of one MMA
constexpr int kSkK = 64;
constexpr int kSkThreads = 192;
constexpr int kSkMaxSplit = 8;  // portable cluster size

// BN rows of X; `LAYOUT`: how a CTA fills its SM.
//   kPair  one 128-feature tile, half an SM's shared memory: two CTAs per SM;
//   kDeep  one tile, the whole SM: twice the stages in flight, for grids of at most one CTA per SM;
//   kWide  two tiles side by side, the whole SM: 512 contiguous bytes per K row of an N-major W where one tile has 256.
enum SkinnyLayout { kPair, kDeep, kWide };

template <int BN, SkinnyLayout LAYOUT>
struct SkinnyCfg {
  static constexpr int kTiles = LAYOUT == kWide ? 2 : 1;
  static constexpr int kFeatures = kTiles * kSkTile;
  static constexpr int kWBytes = kFeatures * kSkK * 2;
  static constexpr int kXBytes = BN * kSkK * 2;
  static constexpr int kBlockBytes = kWBytes + kXBytes;
  static constexpr int kBlocks = (LAYOUT == kPair ? 110 * 1024 : 200 * 1024) / kBlockBytes;
  // A stage, the unit of waits and commits, is one or two k-blocks.
  static constexpr int kGroup = BN <= 16 ? 2 : 1;
  static constexpr int kStages = kBlocks / kGroup;
  // A split tile of few rows receives the other slices' partial sums behind the stages: [slice][own row][feature].
  static constexpr bool kPush = LAYOUT != kWide && BN <= 32;
  static constexpr int kInboxBytes = kPush ? (BN + kSkMaxSplit - 1) * kSkTile * 4 : 0;
  static constexpr int kSplitStages = kPush ? (kBlocks * kBlockBytes - kInboxBytes) / (kGroup * kBlockBytes) : kStages;
  static constexpr int kRingBytes = kBlocks * kBlockBytes;
  static constexpr int kSmem = kRingBytes + 512 + 1024;  // barriers, alignment slack
  static constexpr int kResident = LAYOUT == kPair ? 2 : 1;
  static constexpr int kTmemCols = kTiles * BN < 32 ? 32 : kTiles * BN;
  static_assert(kResident * (kSmem + 1024) <= 228 * 1024 && kSmem <= 227 * 1024, "resident CTAs per SM");
  static_assert(kSplitStages >= 2, "a ring");
  static_assert(LAYOUT == kWide || kPush || BN * kSkTile * 4 <= kRingBytes, "partial sums reuse the stages");
};

struct SkinnyGemmParams {
  int M, N, K;
  void* C;
  int64_t ldc;
  int* status;
  int accumulate;
  int split;
  int w_resident;  // in a chained launch: nothing that runs just before this kernel writes W
};

template <typename OutT>
__device__ __forceinline__ float skinny_read(const OutT* src) {
  if constexpr (sizeof(OutT) == 2) return __bfloat162float(*src);
  else return *src;
}

template <typename OutT>
__device__ __forceinline__ void skinny_write(OutT* dst, float v) {
  if constexpr (sizeof(OutT) == 2) *dst = __float2bfloat16(v);
  else *dst = v;
}

__device__ __forceinline__ float ld_shared_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

template <int BN, SkinnyLayout LAYOUT, bool X_MN, bool W_MN, typename OutT>
__global__ void __launch_bounds__(kSkThreads, LAYOUT == kPair ? 2 : 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                   SkinnyGemmParams p) {
  using S = SkinnyCfg<BN, LAYOUT>;
  constexpr int kGroup = S::kGroup;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem =
      reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::kRingBytes);
  uint64_t* empty_bar = full_bar + S::kStages;
  uint64_t* done_bar = empty_bar + S::kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = p.split;
  const bool splits = LAYOUT != kWide && split > 1;
  const int stages = splits ? S::kSplitStages : S::kStages;
  const int rank = splits ? static_cast<int>(cluster_rank()) : 0;
  const int n0 = static_cast<int>(blockIdx.x) / split * S::kFeatures;
  const int num_kb = (p.K + kSkK - 1) / kSkK;
  const int kb_lo = rank * num_kb / split, kb_hi = (rank + 1) * num_kb / split;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, S::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (S::kPush && splits) cluster_arrive();  // waited for ahead of the first store to another CTA: it runs by then
  const uint32_t tmem = *tmem_slot;
  chain_start_next();

  // TMEM lanes [32 * (warp & 3), +32) belong to an epilogue warp; a thread owns one feature.
  const int feature = (warp & 3) * 32 + lane;
  OutT* out = static_cast<OutT*>(p.C) + n0 + feature;
  // C of up to 16 rows is read while the products run: rows rank, rank + split, ...
  constexpr int kEarlyC = BN <= 16 && LAYOUT != kWide ? 16 : 1;
  float before[kEarlyC];

  bool ok = true;
  if (warp == 0) {
    if (elect_one()) {
      auto block_at = [&](int stage, int j) { return smem + (stage * kGroup + j) * S::kBlockBytes; };
      auto load_w = [&](int stage, int kb) {
        const int blocks = kb_hi - kb < kGroup ? kb_hi - kb : kGroup;
        mbar_arrive_expect_tx(&full_bar[stage], blocks * S::kBlockBytes);
#pragma unroll
        for (int j = 0; j < kGroup; ++j) {
          if (j >= blocks) break;
          uint8_t* sw = block_at(stage, j);
          const int k0 = (kb + j) * kSkK;
          if constexpr (!W_MN) {
#pragma unroll
            for (int t = 0; t < S::kTiles; ++t)
              tma_load_2d(sw + t * (kSkTile * kSkK * 2), &tmap_w, &full_bar[stage], k0, n0 + t * kSkTile);
          } else {
            // (A box that starts beyond the last feature reads the fill value like any other out-of-range column.)
#pragma unroll
            for (int i = 0; i < S::kFeatures / 64; ++i)
              tma_load_2d(sw + i * 8192, &tmap_w, &full_bar[stage], n0 + i * 64, k0);
          }
        }
      };
      // The stages are empty at the start: in a chained launch with resident weights they fill with weights while the
      // kernels before this one still run, and only X waits for them.
      const int early = p.w_resident ? min((kb_hi - kb_lo + kGroup - 1) / kGroup, stages) : 0;
      for (int i = 0; i < early; ++i) load_w(i, kb_lo + i * kGroup);
      chain_wait();
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb_lo; kb < kb_hi; kb += kGroup) {
        if (kb - kb_lo >= early * kGroup) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, p.status, kStatusWaitTimeoutProducer)) break;
          load_w(stage, kb);
        }
#pragma unroll
        for (int j = 0; j < kGroup; ++j) {
          if (kb + j >= kb_hi) break;
          uint8_t* sx = block_at(stage, j) + S::kWBytes;
          const int k0 = (kb + j) * kSkK;
          if constexpr (!X_MN) {
            tma_load_2d(sx, &tmap_x, &full_bar[stage], k0, 0);
          } else {
#pragma unroll
            for (int i = 0; i < BN / 64; ++i) tma_load_2d(sx + i * 8192, &tmap_x, &full_bar[stage], i * 64, k0);
          }
        }
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      chain_wait();
      constexpr uint32_t idesc = umma_idesc_f16(kSkTile, BN, 1, 1, W_MN ? 1 : 0, X_MN ? 1 : 0);
      int stage = 0;
      uint32_t phase = 0;
      bool fed = true;
      for (int kb = kb_lo; kb < kb_hi; kb += kGroup) {
        if (!mbar_wait(&full_bar[stage], phase, p.status, kStatusWaitTimeoutMma)) {
          fed = false;
          break;
        }
        tc_fence_after_sync();
#pragma unroll
        for (int j = 0; j < kGroup; ++j) {
          if (kb + j >= kb_hi) break;
          const uint32_t sw = smem_u32(smem + (stage * kGroup + j) * S::kBlockBytes);
          const uint32_t sx = sw + S::kWBytes;
#pragma unroll
          for (int k = 0; k < kSkK / 16; ++k) {
            const uint64_t dx =
                X_MN ? umma_smem_desc(sx + k * 2048, 8192, 1024) : umma_smem_desc(sx + k * 32, 16, 1024);
#pragma unroll
            for (int t = 0; t < S::kTiles; ++t) {
              const uint32_t st = sw + t * (kSkTile * kSkK * 2);
              const uint64_t dw =
                  W_MN ? umma_smem_desc(st + k * 2048, 8192, 1024) : umma_smem_desc(st + k * 32, 16, 1024);
              tc_mma_f16(tmem + t * BN, dw, dx, idesc, (kb + j > kb_lo || k > 0) ? 1u : 0u);
            }
          }
        }
        if (kb + stages * kGroup < kb_hi) tc_commit(&empty_bar[stage]);  // a stage that is filled again
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (fed) tc_commit(done_bar);
    }
  } else {
    chain_wait();  // ahead of the first read or write of C
    if (kEarlyC > 1 && p.accumulate && n0 + feature < p.N) {
#pragma unroll
      for (int i = 0; i < kEarlyC; ++i)
        if (rank + i * split < p.M) before[i] = skinny_read(out + static_cast<int64_t>(rank + i * split) * p.ldc);
    }
    ok = mbar_wait_warp(done_bar, 0, p.status, kStatusWaitTimeoutEpilogue);
  }
  __syncwarp();
  if (S::kPush && splits) cluster_wait();

  // All MMAs of this CTA have retired.  Partial sums of a split tile go to the CTA that finishes their row, or, where
  // they are too many for its inbox, to the own stages (which are free), to be fetched from there.
  const int own_rows = (p.M + split - 1) / split;
  float* part = reinterpret_cast<float*>(smem);
  const uint32_t inbox = smem_u32(smem + S::kRingBytes - S::kInboxBytes);
  if (warp >= 2 && ok) {
    tc_fence_after_sync();
#pragma unroll
    for (int t = 0; t < S::kTiles; ++t) {
      const uint32_t taddr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + t * BN;
      const bool stores = n0 + t * kSkTile + feature < p.N;
#pragma unroll 1
      for (int c = 0; c < BN; c += 16) {
        if (c >= p.M) break;
        uint32_t r[16];
        tmem_ld_32x16(taddr + c, r);
        tmem_ld_wait();
        if (splits && S::kPush) {
          int to = c % split, row = c / split;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (c + j >= p.M) break;
            st_cluster_f32(inbox + ((rank * own_rows + row) * kSkTile + feature) * 4, to, __uint_as_float(r[j]));
            if (++to == split) to = 0, ++row;
          }
        } else if (splits) {
#pragma unroll
          for (int j = 0; j < 16; ++j) part[(c + j) * kSkTile + feature] = __uint_as_float(r[j]);
        } else if (stores) {
          OutT* dst = out + t * kSkTile + static_cast<int64_t>(c) * p.ldc;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (c + j >= p.M) break;
            float v = __uint_as_float(r[j]);
            if (p.accumulate) v += kEarlyC > 1 ? before[j] : skinny_read(dst + j * p.ldc);
            skinny_write(dst + j * p.ldc, v);
          }
        }
      }
    }
  }
  if (splits) {
    cluster_sync_all();
    if (warp >= 2 && ok && n0 + feature < p.N) {
      auto finish = [&](int i, int row, float old) {
        float v[kSkMaxSplit];
#pragma unroll
        for (int s = 0; s < kSkMaxSplit; ++s) {
          if (s >= split) v[s] = 0.f;
          else if (S::kPush) v[s] = ld_shared_f32(inbox + ((s * own_rows + i) * kSkTile + feature) * 4);
          else v[s] = ld_cluster_f32(smem_u32(part) + (row * kSkTile + feature) * 4, s);
        }
        float sum = v[0];
#pragma unroll
        for (int s = 1; s < kSkMaxSplit; ++s) sum += v[s];
        skinny_write(out + static_cast<int64_t>(row) * p.ldc, p.accumulate ? sum + old : sum);
      };
      if constexpr (kEarlyC > 1) {
#pragma unroll
        for (int i = 0; i < kEarlyC / 2; ++i)
          if (rank + i * split < p.M) finish(i, rank + i * split, before[i]);
      } else {
#pragma unroll 4
        for (int row = rank, i = 0; row < p.M; row += split, ++i)
          finish(i, row, p.accumulate ? skinny_read(out + static_cast<int64_t>(row) * p.ldc) : 0.f);
      }
    }
    if (!S::kPush) cluster_sync_all();  // a CTA's shared memory outlives its readers
  }

  tc_fence_before_sync();
  const int gave_up = __syncthreads_or(!ok);
  if (warp == 1) {
    if (gave_up) {
      // A wait gave up (whichever it was, the epilogue's did, too): let copies that may still be in flight land before
      // the CTA exits.
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
    tc_fence_after_sync();
    tmem_dealloc(tmem, S::kTmemCols);
  }
}

// CTAs of clusters of `split` that the GPU holds at once (GPCs hold whole clusters only).
template <typename Kernel>
static int resident_ctas(Kernel kernel, int smem, int split, std::atomic<int>* cache) {
  int n = cache[split].load(std::memory_order_relaxed);
  if (n > 0) return n;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(split));
  cfg.blockDim = dim3(kSkThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {static_cast<unsigned>(split), 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    clusters = 1;
  }
  cache[split].store(clusters * split, std::memory_order_relaxed);
  return clusters * split;
}

template <int BN, SkinnyLayout LAYOUT, bool X_MN, bool W_MN, typename OutT>
struct SkinnyKernel {
  using S = SkinnyCfg<BN, LAYOUT>;
  static constexpr auto kernel = gemm_skinny_kernel<BN, LAYOUT, X_MN, W_MN, OutT>;

  static bool configure() {
    static const cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem);
    return e == cudaSuccess;
  }

  // Expected time in us of N features cut into `split` slices of `num_kb` k-blocks: what a k-block takes at the slowest
  // of an SM's port to the L2 (110 GB/s), the thread that issues its MMAs (0.21 us a tile, more for many rows) and the
  // memory that all CTAs share; every wave starts and drains, and a split pays for its hand-over, an uneven cluster a
  // little more.  Fitted to chained launches of every split and layout over N of 640 to 32768, K of 1024 to 14336 and 1
  // to 100 rows: the choice is 2 % behind the fastest on average (6 % with the constants of the kernel before this
  // one).
  static float cost(int N, int num_kb, int split) {
    static std::atomic<int> cache[kSkMaxSplit + 1];
    const int ctas = (N + S::kFeatures - 1) / S::kFeatures * split;
    const int resident = resident_ctas(kernel, S::kSmem, split, cache);
    const float sms = static_cast<float>(resident_ctas(kernel, S::kSmem, 1, cache)) / S::kResident;
    const int waves = (ctas + resident - 1) / resident;
    const int stages = ((num_kb + split - 1) / split + S::kGroup - 1) / S::kGroup;
    const float at_once = static_cast<float>(ctas < resident ? ctas : resident);
    const float port = S::kBlockBytes * fmaxf(1.f, at_once / sms) / 1.1e5f;
    const float memory = at_once * S::kWBytes / 7.1e6f;
    const float issue = (BN > 16 ? 0.23f : 0.21f) * S::kTiles;
    const float work = static_cast<float>(stages * S::kGroup) * fmaxf(fmaxf(port, memory), issue);
    const float rows = S::kPush ? 0.01f * BN : 0.13f * BN / split;
    const float meet = 1.5f + 0.15f * split + rows + ((split & (split - 1)) != 0 ? 0.15f : 0.f);
    return static_cast<float>(waves) * (work + 1.25f) + (split > 1 ? meet : 0.f);
  }

  static int launch(const CUtensorMap& tw, const CUtensorMap& tx, const SkinnyGemmParams& p, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>((p.N + S::kFeatures - 1) / S::kFeatures * p.split));
    cfg.blockDim = dim3(kSkThreads);
    cfg.dynamicSmemBytes = S::kSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {static_cast<unsigned>(p.split), 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = static_cast<unsigned>(chain_attribute(attr, p.split > 1 ? 1 : 0));
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tw, tx, p);
    if (e != cudaSuccess) {
      fprintf(stderr, "axb skinny gemm: launch failed: %s\n", cudaGetErrorString(e));
      return -4;
    }
    return 0;
  }
};

// The cheapest layout and split; `forced` split (0 = free).
template <int BN, bool X_MN, bool W_MN, typename OutT>
static bool skinny_plan(int N, int K, int forced, int* split, SkinnyLayout* layout) {
  using Pair = SkinnyKernel<BN, kPair, X_MN, W_MN, OutT>;
  using Deep = SkinnyKernel<BN, kDeep, X_MN, W_MN, OutT>;
  using Wide = SkinnyKernel<BN, kWide, X_MN, W_MN, OutT>;
  if (!Deep::configure() || !Pair::configure() || !Wide::configure()) return false;
  const int num_kb = (K + kSkK - 1) / kSkK;
  float best = 0.f;
  *split = 0;
  auto consider = [&](float cost, int s, SkinnyLayout l) {
    if (*split != 0 && cost >= best) return;
    best = cost;
    *split = s;
    *layout = l;
  };
  for (int s = 1; s <= kSkMaxSplit && s <= num_kb; ++s) {
    if (forced > 0 ? s != forced : (s > 1 && num_kb / s < 2)) continue;
    consider(Deep::cost(N, num_kb, s), s, kDeep);
    consider(Pair::cost(N, num_kb, s), s, kPair);
    if (s == 1) consider(Wide::cost(N, num_kb, 1), 1, kWide);
  }
  return *split > 0;
}

template <int BN, bool X_MN, bool W_MN, typename OutT>
static int launch_skinny(const void* X, const void* W, int64_t ldx, int64_t ldw, SkinnyGemmParams p,
                         cudaStream_t stream) {
  SkinnyLayout layout = kPair;
  if (!skinny_plan<BN, X_MN, W_MN, OutT>(p.N, p.K, p.split, &p.split, &layout)) return -15;
  CUtensorMap tw, tx;
  const uint64_t k = static_cast<uint64_t>(p.K), n = static_cast<uint64_t>(p.N), m = static_cast<uint64_t>(p.M);
  const uint64_t wdims[2] = {W_MN ? n : k, W_MN ? k : n};
  const uint64_t wstride[1] = {static_cast<uint64_t>(ldw) * 2};
  const uint32_t wbox[2] = {64, static_cast<uint32_t>(W_MN ? kSkK : kSkTile)};
  int rc = make_tensor_map(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, W, wdims, wstride, wbox,
                           CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != 0) return rc;
  static_assert(!X_MN || BN >= 64, "an M-major tile of X is at least one 128-byte row wide");
  const uint64_t xdims[2] = {X_MN ? m : k, X_MN ? k : m};
  const uint64_t xstride[1] = {static_cast<uint64_t>(ldx) * 2};
  const uint32_t xbox[2] = {64, X_MN ? static_cast<uint32_t>(kSkK) : static_cast<uint32_t>(BN)};
  rc = make_tensor_map(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, X, xdims, xstride, xbox, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != 0) return rc;
  switch (layout) {
    case kDeep: return SkinnyKernel<BN, kDeep, X_MN, W_MN, OutT>::launch(tw, tx, p, stream);
    case kWide: return SkinnyKernel<BN, kWide, X_MN, W_MN, OutT>::launch(tw, tx, p, stream);
    default: return SkinnyKernel<BN, kPair, X_MN, W_MN, OutT>::launch(tw, tx, p, stream);
  }
}

}  // namespace axb

// Chains the launches of the calling thread (chain.cuh) from here on; returns the previous setting.
extern "C" int axb_chain_launches(int on) {
  const int before = axb::chain_launches ? 1 : 0;
  axb::chain_launches = on != 0;
  return before;
}

// K slices that the kernel would choose for a problem with K-major X and N-major W (1 = no split).
extern "C" int axb_gemm_splitk_plan(int M, int N, int K) {
  using namespace axb;
  int split = 1;
  SkinnyLayout layout;
  bool ok;
  if (M <= 16) ok = skinny_plan<16, false, true, __nv_bfloat16>(N, K, 0, &split, &layout);
  else if (M <= 32) ok = skinny_plan<32, false, true, __nv_bfloat16>(N, K, 0, &split, &layout);
  else if (M <= 64) ok = skinny_plan<64, false, true, __nv_bfloat16>(N, K, 0, &split, &layout);
  else if (M <= 128) ok = skinny_plan<128, false, true, __nv_bfloat16>(N, K, 0, &split, &layout);
  else ok = false;
  return ok ? split : 1;
}

// C[M, N] (bf16 or fp32, row pitch ldc) = X * W (+ C when accumulate), M <= 128.
//   x_mn_major = 0: X is [M, K] row-major (pitch ldx);         1: X is stored [K, M] row-major.
//   w_mn_major = 0: W is stored [N, K] row-major (pitch ldw);  1: W is [K, N] row-major.
// `w_resident`: W is not written by what runs before it on the stream (weights); counts in chained launches only.
// `split`: K slices per tile, 0 = the kernel's own choice.  Alignment as for axb_gemm_bf16; -20 = not one of mine.
extern "C" int axb_gemm_skinny(const void* X, const void* W, void* C, int M, int N, int K, int64_t ldx, int64_t ldw,
                               int64_t ldc, int x_mn_major, int w_mn_major, int out_fp32, int accumulate, int split,
                               int w_resident, int* status, cudaStream_t stream) {
  using namespace axb;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  // One wave of two-tile CTAs at most: beyond it the persistent 256-column tiles of gemm.cu, which overlap a tile's
  // epilogue with the next tile's stream, are faster (64 x 128256 x 2048: 89 us, here 102; 32 x 40960 x 4096: 71 and
  // 79).  Above 64 rows X weighs as much as W in every stage, and they win as soon as they fill half the SMs
  // (128 x 12288 x 4096: 23.2 and 24.5; 128 x 4096 x 4096: 20.7 and 15.7).
  if (M > 128 || N > (M <= 64 ? 148 * 256 : 8192)) return -20;
  if ((ldx % 8) || (ldw % 8) || (reinterpret_cast<uintptr_t>(X) & 15) || (reinterpret_cast<uintptr_t>(W) & 15) ||
      (reinterpret_cast<uintptr_t>(C) & 15) || (ldc % (out_fp32 ? 4 : 8)))
    return -10;
  if (split < 0 || split > kSkMaxSplit || split > (K + kSkK - 1) / kSkK) return -15;
  const SkinnyGemmParams p{M, N, K, C, ldc, status, accumulate, split, w_resident && chain_launches ? 1 : 0};
#define AXB_SKINNY_BN(BN, XM, WM, T) return launch_skinny<BN, XM, WM, T>(X, W, ldx, ldw, p, stream)
#define AXB_SKINNY(WM, T)                                  \
  do {                                                     \
    if (x_mn_major && M <= 64) AXB_SKINNY_BN(64, true, WM, T); \
    if (x_mn_major) AXB_SKINNY_BN(128, true, WM, T);       \
    if (M <= 16) AXB_SKINNY_BN(16, false, WM, T);          \
    if (M <= 32) AXB_SKINNY_BN(32, false, WM, T);          \
    if (M <= 64) AXB_SKINNY_BN(64, false, WM, T);          \
    AXB_SKINNY_BN(128, false, WM, T);                      \
  } while (0)
  if (w_mn_major) {
    if (out_fp32) AXB_SKINNY(true, float);
    AXB_SKINNY(true, __nv_bfloat16);
  }
  if (out_fp32) AXB_SKINNY(false, float);
  AXB_SKINNY(false, __nv_bfloat16);
#undef AXB_SKINNY
#undef AXB_SKINNY_BN
}
