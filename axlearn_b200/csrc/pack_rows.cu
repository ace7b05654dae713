// Where the live tokens of right-padded prompts lie when they are packed one sequence after the other.
//
// One launch for what is a clamp, a sum, a scan and the two index lists; as separate operators these were 18 launches, 0.2 ms
// of a host that has just waited for the lengths and of a GPU that waits for the host.  A few hundred KB: the launch is all.
#include <cuda_runtime.h>
#include <stdint.h>

namespace axb {

constexpr int kPackThreads = 256;

// Block (tile of 256 positions, sequence).  first [B]: the packed row of a sequence's first token; live_out [B]: its live
// tokens, clamped to [0, T]; total [2]: of all, and whether a sequence has none.  rows_of: the padded row of each packed
// row; row_of: the packed row of each padded row, -1 for padding.
__global__ void __launch_bounds__(kPackThreads)
pack_rows_kernel(const int* __restrict__ live, int B, int T, int* __restrict__ first, int* __restrict__ live_out,
                 int* __restrict__ total, int* __restrict__ rows_of, int* __restrict__ row_of) {
  const int b = blockIdx.y, t = blockIdx.x * kPackThreads + threadIdx.x;
  __shared__ int partial[kPackThreads / 32];
  int sum = 0, none = 0;
  for (int i = threadIdx.x; i < b; i += kPackThreads) sum += min(max(live[i], 0), T), none += live[i] <= 0;
  sum = __reduce_add_sync(0xffffffffu, sum);
  none = __syncthreads_or(none != 0);
  if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = sum;
  __syncthreads();
  int begin = 0;
#pragma unroll
  for (int w = 0; w < kPackThreads / 32; ++w) begin += partial[w];
  const int n = min(max(live[b], 0), T);
  if (t == 0) {
    first[b] = begin;
    live_out[b] = n;
    if (b == B - 1) total[0] = begin + n, total[1] = none || n == 0;
  }
  if (t >= T) return;
  const int padded = b * T + t;
  row_of[padded] = t < n ? begin + t : -1;
  if (t < n) rows_of[begin + t] = padded;
}

// One CTA per padded row: its packed row, zeros for padding (what a kernel multiplies by the zero probabilities of padding
// must be finite, whatever the sequences hold).  Reads and writes bound it.  16 Zukitar prompts of up to 1000 tokens and 16
// steps, which unpack the latent layer's projection and the output: 9793 us with an index operator that fills padding with
// a row, 9768 with this.
template <typename V>
__global__ void __launch_bounds__(kPackThreads)
unpack_rows_kernel(const V* __restrict__ x, V* __restrict__ out, const int* __restrict__ row_of, int64_t width) {
  const int64_t row = blockIdx.x;
  const int from = row_of[row];
  for (int64_t i = threadIdx.x; i < width; i += kPackThreads) out[row * width + i] = from < 0 ? V{} : x[from * width + i];
}

}  // namespace axb

// rows_of and row_of have B T entries, of which the first `total` of rows_of are written.
extern "C" int axb_pack_rows(const int* live, int B, int T, int* first, int* live_out, int* total, int* rows_of, int* row_of,
                             cudaStream_t stream) {
  if (B <= 0 || T <= 0 || B > 65535 || static_cast<int64_t>(B) * T > 0x7fffffff) return -10;
  const dim3 grid(static_cast<unsigned>((T + axb::kPackThreads - 1) / axb::kPackThreads), static_cast<unsigned>(B));
  axb::pack_rows_kernel<<<grid, axb::kPackThreads, 0, stream>>>(live, B, T, first, live_out, total, rows_of, row_of);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// out [rows, row_bytes] = x[row_of], zeros where row_of is negative; row_bytes is even.
extern "C" int axb_unpack_rows(const void* x, void* out, const int* row_of, int64_t rows, int64_t row_bytes,
                               cudaStream_t stream) {
  using namespace axb;
  if (rows <= 0 || rows > 0x7fffffff || row_bytes <= 0 || row_bytes % 2) return -10;
  const unsigned grid = static_cast<unsigned>(rows);
  if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) | static_cast<uintptr_t>(row_bytes)) & 15) == 0)
    unpack_rows_kernel<<<grid, kPackThreads, 0, stream>>>(static_cast<const uint4*>(x), static_cast<uint4*>(out), row_of,
                                                          row_bytes / 16);
  else
    unpack_rows_kernel<<<grid, kPackThreads, 0, stream>>>(static_cast<const uint16_t*>(x), static_cast<uint16_t*>(out),
                                                          row_of, row_bytes / 2);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
