// Columns of several [n, k_i] buffers side by side in one [n, K] buffer: the
// attribute rows that the interpolation takes, and the gradient of splitting
// its packed result back into attributes (a concatenation, elementwise per
// row). Bound by HBM: 8 K bytes per row.
#include <string>

#include "common.cuh"
#include "internal.h"

namespace dr {
namespace {

constexpr int kRows = 128, kThreads = 256;

struct Columns {
  const float* src[DR_MAX_CHANNELS];  // null: zeros
  int64_t stride[DR_MAX_CHANNELS];    // floats from a row to the next
  int width[DR_MAX_CHANNELS], first[DR_MAX_CHANNELS];
  int count, K;
  int64_t n;
  float* out;
};

// A block takes 128 rows: every part's values go to shared memory in the
// order they lie in, then the rows leave as float4s (128 K floats are a
// multiple of 16 bytes), so that both sides are whole lines whatever the
// widths are.
__global__ void __launch_bounds__(kThreads) pack_columns_kernel(Columns a) {
  extern __shared__ __align__(16) float rows[];
  const int64_t r0 = int64_t(blockIdx.x) * kRows;
  const int n = int(min(int64_t(kRows), a.n - r0));
  for (int p = 0; p < a.count; ++p) {
    const int w = a.width[p];
    const float* src = a.src[p] ? a.src[p] + r0 * a.stride[p] : nullptr;
    const int dr = kThreads / w, dc = kThreads - dr * w;
    int r = threadIdx.x / w, c = threadIdx.x - r * w;
    while (r < n) {
      rows[r * a.K + a.first[p] + c] = src ? __ldg(src + r * a.stride[p] + c) : 0.0f;
      r += dr;
      c += dc;
      if (c >= w) {
        c -= w;
        ++r;
      }
    }
  }
  __syncthreads();
  float* out = a.out + r0 * a.K;
  const int total = n * a.K;
  if ((reinterpret_cast<uintptr_t>(a.out) & 15) == 0) {
    for (int i = threadIdx.x; i < total >> 2; i += kThreads)
      reinterpret_cast<float4*>(out)[i] = reinterpret_cast<const float4*>(rows)[i];
    for (int i = (total & ~3) + int(threadIdx.x); i < total; i += kThreads) out[i] = rows[i];
  } else {
    for (int i = threadIdx.x; i < total; i += kThreads) out[i] = rows[i];
  }
}

}  // namespace

int pack_columns_launch(const float* const* parts, const int32_t* widths, const int64_t* strides,
                        int count, int64_t n, float* out, cudaStream_t stream, std::string& err) {
  if (count < 1 || count > DR_MAX_CHANNELS || n < 0 || !parts || !widths || !strides) {
    err = "pack_columns takes 1 to 16 parts with their widths and strides";
    return DR_ERR_INVALID_ARGUMENT;
  }
  Columns a{};
  a.count = count;
  a.n = n;
  a.out = out;
  for (int p = 0; p < count; ++p) {
    if (widths[p] < 1 || widths[p] > DR_MAX_CHANNELS || strides[p] < 0) {
      err = "part widths must be in [1, 16] and strides >= 0";
      return DR_ERR_INVALID_ARGUMENT;
    }
    a.src[p] = parts[p];
    a.stride[p] = strides[p];
    a.width[p] = widths[p];
    a.first[p] = a.K;
    a.K += widths[p];
  }
  if (a.K > DR_MAX_CHANNELS) {
    err = "pack_columns takes at most 16 channels";
    return DR_ERR_INVALID_ARGUMENT;
  }
  if (n == 0) return DR_OK;
  if (!out) { err = "out must be non-null"; return DR_ERR_INVALID_ARGUMENT; }
  pack_columns_kernel<<<unsigned((n + kRows - 1) / kRows), kThreads, size_t(kRows) * a.K * 4,
                        stream>>>(a);
  return launch_status("pack columns", err);
}

}  // namespace dr
