// 3x3 / stride 2 / pad 1 max pooling on NHWC activations (the ResNet stem pool), forward and backward.
//
// Forward: one thread per (output pixel, 8 channels): nine 16-byte loads, a running maximum that keeps the
// FIRST maximum in scan order (rows, then columns), one 16-byte store of the result and 8 bytes of argmax
// codes (0..8).  Backward: one thread per (2 x 2 input pixels, 8 channels) gathers from the at most four windows
// that contain them the gradients whose argmax code points at each: no atomics, deterministic, and the
// input activation is not read again.
//
// The reference has no pooling (model math is TensorFlow's); this serves the ResNet-50 benchmark model.
#include <algorithm>

#include "kernels/common.cuh"
#include "kernels/tips_kernels.h"

namespace tipsk {
namespace {

// Two 16-bit floats in a register: minus infinity twice, and a mask of the halves in which a > b (NaN: not greater).
template <typename T>
__device__ __forceinline__ uint32_t NegInf2();
template <>
__device__ __forceinline__ uint32_t NegInf2<__nv_bfloat16>() { return 0xff80ff80u; }
template <>
__device__ __forceinline__ uint32_t NegInf2<__half>() { return 0xfc00fc00u; }
template <typename T>
__device__ __forceinline__ uint32_t Greater2(uint32_t a, uint32_t b);
template <>
__device__ __forceinline__ uint32_t Greater2<__nv_bfloat16>(uint32_t a, uint32_t b) {
  return __hgt2_mask(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
}
template <>
__device__ __forceinline__ uint32_t Greater2<__half>(uint32_t a, uint32_t b) {
  return __hgt2_mask(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
}

// Both directions are bound by HBM.  A block works on one row (of outputs, or of 2 x 2 input quads), or with kRows on several
// rows of few elements, so a thread needs a single 32-bit division to find its pixel, and all its loads are issued before
// the first comparison.  (The two forms are apart because the row's own division is uniform in the first: 33 us for 64
// images of 64 x 112 x 112, 41 with a row per thread.)
template <bool kRows>
__device__ __forceinline__ int64_t FirstRow() {
  return kRows ? static_cast<int64_t>(blockIdx.y) * blockDim.y + threadIdx.y : blockIdx.y;
}
template <bool kRows>
__device__ __forceinline__ int64_t RowStep() {
  return kRows ? static_cast<int64_t>(gridDim.y) * blockDim.y : gridDim.y;
}

template <typename T, bool kRows>
__global__ void __launch_bounds__(256, 4)
MaxPoolFwdKernel(const T* __restrict__ x, T* __restrict__ y, uint8_t* __restrict__ idx, int64_t rows, int h, int w, int c,
                 int ho, int wo) {
  constexpr int V = 8;
  const int cv = c / V;
  const int i  = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= wo * cv) return;
  const int ow = i / cv, cg = i - ow * cv;
  for (int64_t row = FirstRow<kRows>(); row < rows; row += RowStep<kRows>()) {  // row = image * ho + oh
    const int64_t in = row / ho;
    const int oh     = static_cast<int>(row - in * ho);
    const T* base    = x + in * h * w * c + cg * V;
    Vec16<T> v[9];
    bool have[9];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int ih = oh * 2 - 1 + r;
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        const int iw = ow * 2 - 1 + s;
        have[r * 3 + s] = ih >= 0 && ih < h && iw >= 0 && iw < w;
        if (have[r * 3 + s]) v[r * 3 + s] = LoadVec(base + (static_cast<int64_t>(ih) * w + iw) * c);
      }
    }
    // two channels per register: the comparison yields a mask that selects value and position of both
    uint32_t best[4], arg[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { best[i] = NegInf2<T>(); arg[i] = 0; }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      if (!have[k]) continue;
      const uint32_t* q = reinterpret_cast<const uint32_t*>(&v[k]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t gt = Greater2<T>(q[i], best[i]);
        best[i] = (q[i] & gt) | (best[i] & ~gt);
        arg[i]  = (k * 0x10001u & gt) | (arg[i] & ~gt);
      }
    }
    const int64_t at = (row * wo + ow) * c + cg * V;
    *reinterpret_cast<uint4*>(y + at) = make_uint4(best[0], best[1], best[2], best[3]);
    // bytes 0 and 2 of each: the positions of eight channels
    *reinterpret_cast<uint2*>(idx + at) = make_uint2(__byte_perm(arg[0], arg[1], 0x6420), __byte_perm(arg[2], arg[3], 0x6420));
  }
}

// One thread per 2 x 2 input quad (2a..2a+1, 2b..2b+1) and 8 channels: exactly the windows (a..a+1, b..b+1) reach the
// quad, so four gradients and four code words serve four outputs (a thread per pixel read nine of each).
template <typename T, bool kRows>
__global__ void __launch_bounds__(256)
MaxPoolBwdKernel(const T* __restrict__ dy, const uint8_t* __restrict__ idx, T* __restrict__ dx, int64_t rows, int h, int w,
                 int c, int ho, int wo) {
  constexpr int V = 8;
  const int cv = c / V;
  const int hq = (h + 1) / 2, wq = (w + 1) / 2;
  const int i  = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= wq * cv) return;
  const int b = i / cv, cg = i - b * cv;
  for (int64_t row = FirstRow<kRows>(); row < rows; row += RowStep<kRows>()) {  // row = image * hq + a
    const int64_t in = row / hq;
    const int a      = static_cast<int>(row - in * hq);
    Vec16<T> g[4];
    uint2 code[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int oh = a + (k >> 1), ow = b + (k & 1);
      if (oh < ho && ow < wo) {
        const int64_t at = ((in * ho + oh) * wo + ow) * c + cg * V;
        g[k]    = LoadVec(dy + at);
        code[k] = *reinterpret_cast<const uint2*>(idx + at);
      } else {
        code[k] = make_uint2(0xffffffffu, 0xffffffffu);  // matches no position
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int dh = q >> 1, dw = q & 1;
      const int ih = 2 * a + dh, iw = 2 * b + dw;
      if (ih >= h || iw >= w) continue;
      float acc[V];
#pragma unroll
      for (int j = 0; j < V; ++j) acc[j] = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        // window (a + kh, b + kw) covers input rows 2(a + kh) - 1 .. 2(a + kh) + 1
        const int r = dh + 1 - 2 * (k >> 1), s = dw + 1 - 2 * (k & 1);
        if (r < 0 || s < 0) continue;
        const uint32_t want = static_cast<uint32_t>(r * 3 + s);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          const uint32_t got = ((j < 4 ? code[k].x : code[k].y) >> ((j & 3) * 8)) & 0xffu;
          if (got == want) acc[j] += ToFloat(g[k].v[j]);
        }
      }
      Vec16<T> o;
#pragma unroll
      for (int j = 0; j < V; ++j) o.v[j] = FromFloat<T>(acc[j]);
      StoreVec(dx + ((in * h + ih) * w + iw) * c + cg * V, o);
    }
  }
}

// Block and grid of the pooling kernels: x covers the elements of a row, y the rows.  Rows of up to 128 elements share a block
// (17 x 17 outputs of 8 channels for 512 images: 17 threads of each block at work, 14.3 us, against 5 with 15 rows in it).
dim3 RowBlock(int64_t per_row) {
  const unsigned tx = static_cast<unsigned>(per_row <= 128 ? per_row : 256);
  return dim3(tx, 256 / tx);
}
dim3 RowGrid(int64_t per_row, int64_t rows, dim3 block) {
  return dim3(static_cast<unsigned>((per_row + block.x - 1) / block.x),
              static_cast<unsigned>(std::min<int64_t>((rows + block.y - 1) / block.y, 65535)));
}

// Global average pooling of an NHWC activation: y[n, c] = mean over the hw pixels; one thread per (image, 8
// channels), 16-byte loads down the pixel axis.  Backward spreads dy / hw over the pixels.
template <typename T>
__global__ void __launch_bounds__(256)
GlobalAvgPoolFwdKernel(const T* __restrict__ x, T* __restrict__ y, int n, int hw, int c) {
  constexpr int V = 16 / sizeof(T);
  const int cv = c / V;
  const int64_t total = static_cast<int64_t>(n) * cv;
  const float inv = 1.f / static_cast<float>(hw);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int cg = static_cast<int>(i % cv);
    const int in = static_cast<int>(i / cv);
    float acc[V];
#pragma unroll
    for (int j = 0; j < V; ++j) acc[j] = 0.f;
    const T* base = x + static_cast<int64_t>(in) * hw * c + cg * V;
    for (int p = 0; p < hw; ++p) {
      const Vec16<T> v = LoadVec(base + static_cast<int64_t>(p) * c);
#pragma unroll
      for (int j = 0; j < V; ++j) acc[j] += ToFloat(v.v[j]);
    }
    Vec16<T> o;
#pragma unroll
    for (int j = 0; j < V; ++j) o.v[j] = FromFloat<T>(acc[j] * inv);
    StoreVec(y + static_cast<int64_t>(in) * c + cg * V, o);
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
GlobalAvgPoolBwdKernel(const T* __restrict__ dy, T* __restrict__ dx, int n, int hw, int c) {
  constexpr int V = 16 / sizeof(T);
  const int cv = c / V;
  const int64_t total = static_cast<int64_t>(n) * hw * cv;
  const float inv = 1.f / static_cast<float>(hw);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int cg = static_cast<int>(i % cv);
    const int in = static_cast<int>(i / (static_cast<int64_t>(cv) * hw));
    const Vec16<T> g = LoadVec(dy + static_cast<int64_t>(in) * c + cg * V);
    Vec16<T> o;
#pragma unroll
    for (int j = 0; j < V; ++j) o.v[j] = FromFloat<T>(ToFloat(g.v[j]) * inv);
    StoreVec(dx + i * V, o);
  }
}

}  // namespace
}  // namespace tipsk

using namespace tipsk;

extern "C" {

/* y[n, ho, wo, c] = max over 3x3 windows (stride 2, pad 1) of x[n, h, w, c]; idx (uint8, same shape as y) receives
 * the position 0..8 of the maximum inside its window.  dtype: 6 bf16 or 7 fp16; c must be a multiple of 8. */
int tipsk_maxpool3x3s2_fwd(const void* x, void* y, void* idx, int n, int h, int w, int c, int dtype, void* stream) {
  TIPSK_REQUIRE(c % 8 == 0, "maxpool: channel count must be a multiple of 8");
  TIPSK_REQUIRE(dtype == kBF16 || dtype == kF16, "maxpool: bf16 or fp16 only");
  const int ho = (h + 2 - 3) / 2 + 1, wo = (w + 2 - 3) / 2 + 1;
  const int64_t per_row = static_cast<int64_t>(wo) * (c / 8), rows = static_cast<int64_t>(n) * ho;
  if (per_row <= 0 || rows <= 0) return 0;
  TIPSK_REQUIRE(per_row < (int64_t{1} << 30), "maxpool: a row has too many elements");
  const dim3 block = RowBlock(per_row), grid = RowGrid(per_row, rows, block);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == kBF16) {
    auto* kernel = block.y > 1 ? MaxPoolFwdKernel<__nv_bfloat16, true> : MaxPoolFwdKernel<__nv_bfloat16, false>;
    kernel<<<grid, block, 0, s>>>(static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y),
                                  static_cast<uint8_t*>(idx), rows, h, w, c, ho, wo);
  } else {
    auto* kernel = block.y > 1 ? MaxPoolFwdKernel<__half, true> : MaxPoolFwdKernel<__half, false>;
    kernel<<<grid, block, 0, s>>>(static_cast<const __half*>(x), static_cast<__half*>(y), static_cast<uint8_t*>(idx), rows,
                                  h, w, c, ho, wo);
  }
  TIPSK_LAUNCH_CHECK();
  return 0;
}

int tipsk_maxpool3x3s2_bwd(const void* dy, const void* idx, void* dx, int n, int h, int w, int c, int dtype,
                           void* stream) {
  TIPSK_REQUIRE(c % 8 == 0, "maxpool: channel count must be a multiple of 8");
  TIPSK_REQUIRE(dtype == kBF16 || dtype == kF16, "maxpool: bf16 or fp16 only");
  const int ho = (h + 2 - 3) / 2 + 1, wo = (w + 2 - 3) / 2 + 1;
  const int64_t per_row = static_cast<int64_t>((w + 1) / 2) * (c / 8), rows = static_cast<int64_t>(n) * ((h + 1) / 2);
  if (per_row <= 0 || rows <= 0) return 0;
  TIPSK_REQUIRE(per_row < (int64_t{1} << 30), "maxpool: a row has too many elements");
  const dim3 block = RowBlock(per_row), grid = RowGrid(per_row, rows, block);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == kBF16) {
    auto* kernel = block.y > 1 ? MaxPoolBwdKernel<__nv_bfloat16, true> : MaxPoolBwdKernel<__nv_bfloat16, false>;
    kernel<<<grid, block, 0, s>>>(static_cast<const __nv_bfloat16*>(dy), static_cast<const uint8_t*>(idx),
                                  static_cast<__nv_bfloat16*>(dx), rows, h, w, c, ho, wo);
  } else {
    auto* kernel = block.y > 1 ? MaxPoolBwdKernel<__half, true> : MaxPoolBwdKernel<__half, false>;
    kernel<<<grid, block, 0, s>>>(static_cast<const __half*>(dy), static_cast<const uint8_t*>(idx), static_cast<__half*>(dx),
                                  rows, h, w, c, ho, wo);
  }
  TIPSK_LAUNCH_CHECK();
  return 0;
}

/* Global average pooling on NHWC: x [n, hw, c] -> y [n, c]; c a multiple of 8 (16-bit types) / 4 (fp32). */
int tipsk_global_avgpool_fwd(const void* x, void* y, int n, int hw, int c, int dtype, void* stream) {
  if (n <= 0 || hw <= 0 || c <= 0) return 0;
  const int v = 16 / static_cast<int>(DTypeSize(dtype));
  TIPSK_REQUIRE(dtype == kBF16 || dtype == kF16 || dtype == kF32, "avgpool: bf16, fp16 or fp32");
  TIPSK_REQUIRE(c % v == 0, "avgpool: the channel count must be a multiple of 16 bytes");
  const int64_t total = static_cast<int64_t>(n) * (c / v);
  const int grid = static_cast<int>(std::min<int64_t>((total + 255) / 256, NumSMs() * 8));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == kBF16)
    GlobalAvgPoolFwdKernel<__nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(x),
                                                               static_cast<__nv_bfloat16*>(y), n, hw, c);
  else if (dtype == kF16)
    GlobalAvgPoolFwdKernel<__half><<<grid, 256, 0, s>>>(static_cast<const __half*>(x), static_cast<__half*>(y), n, hw, c);
  else
    GlobalAvgPoolFwdKernel<float><<<grid, 256, 0, s>>>(static_cast<const float*>(x), static_cast<float*>(y), n, hw, c);
  TIPSK_LAUNCH_CHECK();
  return 0;
}

int tipsk_global_avgpool_bwd(const void* dy, void* dx, int n, int hw, int c, int dtype, void* stream) {
  if (n <= 0 || hw <= 0 || c <= 0) return 0;
  const int v = 16 / static_cast<int>(DTypeSize(dtype));
  TIPSK_REQUIRE(dtype == kBF16 || dtype == kF16 || dtype == kF32, "avgpool: bf16, fp16 or fp32");
  TIPSK_REQUIRE(c % v == 0, "avgpool: the channel count must be a multiple of 16 bytes");
  const int64_t total = static_cast<int64_t>(n) * hw * (c / v);
  const int grid = static_cast<int>(std::min<int64_t>((total + 255) / 256, NumSMs() * 8));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == kBF16)
    GlobalAvgPoolBwdKernel<__nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(dy),
                                                               static_cast<__nv_bfloat16*>(dx), n, hw, c);
  else if (dtype == kF16)
    GlobalAvgPoolBwdKernel<__half><<<grid, 256, 0, s>>>(static_cast<const __half*>(dy), static_cast<__half*>(dx), n, hw, c);
  else
    GlobalAvgPoolBwdKernel<float><<<grid, 256, 0, s>>>(static_cast<const float*>(dy), static_cast<float*>(dx), n, hw, c);
  TIPSK_LAUNCH_CHECK();
  return 0;
}

}  // extern "C"
