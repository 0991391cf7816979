// tm_filter.cu -- imageproc's filter_clamped on the device (src/filter/mod.rs:
// 29-70, :202-212): the 2-D correlation of a u8 image (1, 3 or 4 interleaved
// channels) with a row-major kernel, padded by continuity (coordinates clamped
// to the image), accumulated per channel in the kernel's type and clamped to
// the output type by the reference's Clamp (src/definitions.rs:114-190).
//
// The reference's arithmetic is kept exactly: for each output pixel the sum
// runs k_y outer, k_x inner, acc = acc + (K)pixel * weight with one rounding
// per multiply and per add for f32 kernels (explicitly rounded intrinsics, no
// contraction) and wrapping two's-complement arithmetic for i32 kernels (a
// release build).
//
// Kernels up to 8 columns by 32 rows on images of more blocks than run at
// once: filter_rows_kernel. A row of the image
// is W * C elements, a tap k_x columns away is k_x * C elements away, so one
// kernel serves every channel count. A block stages its clamped input window
// once, converted to the kernel's type, in shared memory; a thread owns 4
// elements x 4 rows, reads each input row of its strip once as 16-byte words
// and adds it to the output rows it feeds, from the first tap row to the last
// (so each output's sum keeps the order above). The bound is the two f32
// operations per tap (no fused multiply-add): 4096 x 4096 u8, 5 x 5 f32 to u8,
// 23 us at the FP32 issue rate. Against one thread per pixel reading a byte and
// converting it per tap: 209 -> 56 us.
// Smaller images and larger kernels: filter_tile_kernel (to 64 x 64, a 32 x 8
// output tile and its input window as bytes) and filter_global_kernel.
#include <type_traits>

#include "tm_common.cuh"
#include "tm_filter_rule.h"
#include "tm_internal.h"

namespace ipb {
namespace {

__device__ __forceinline__ uint32_t align_up_dev(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }

constexpr int kTX = kFilterTileW, kTY = kFilterTileH;
constexpr uint32_t kMaxTileKernel = 64;  // kernels up to 64 x 64 use the shared-memory tile

// Clamp<K> for S (src/definitions.rs:119-190): values at or above the maximum
// (and NaN) give the maximum, values at or below the minimum the minimum,
// the rest convert (f32 -> integer truncates toward zero).
template <typename S, typename K>
__device__ __forceinline__ S clamp_to(K x) {
  if constexpr (std::is_same<S, K>::value) {
    return x;
  } else {
    constexpr K hi = std::is_same<S, uint8_t>::value ? (K)255 : std::is_same<S, uint16_t>::value ? (K)65535 : (K)32767;
    constexpr K lo = std::is_same<S, int16_t>::value ? (K)-32768 : (K)0;
    if (x < hi) return x > lo ? (S)x : (S)lo;
    return (S)hi;
  }
}

template <typename K>
__device__ __forceinline__ K mac(K acc, K pix, K w) {
  if constexpr (std::is_same<K, float>::value) {
    return __fadd_rn(acc, __fmul_rn(pix, w));
  } else {  // i32, wrapping
    return (int32_t)((uint32_t)acc + (uint32_t)pix * (uint32_t)w);
  }
}

template <typename S>
constexpr int elem_of() {
  return std::is_same<S, uint8_t>::value    ? IPB_ELEM_U8
         : std::is_same<S, uint16_t>::value ? IPB_ELEM_U16
         : std::is_same<S, int16_t>::value  ? IPB_ELEM_I16
         : std::is_same<S, int32_t>::value  ? IPB_ELEM_I32
                                            : IPB_ELEM_F32;
}

template <int C, typename K, typename S>
__global__ void __launch_bounds__(kTX* kTY) filter_tile_kernel(const uint8_t* __restrict__ img, uint32_t W, uint32_t H,
                                                              const K* __restrict__ kern, uint32_t kw, uint32_t kh,
                                                              S* __restrict__ out) {
  extern __shared__ __align__(16) uint8_t smem[];
  K* s_k = reinterpret_cast<K*>(smem);
  uint8_t* s_img = smem + align_up_dev(kw * kh * sizeof(K), 16);
  const uint32_t tw = kTX + kw - 1, th = kTY + kh - 1;
  const int x0 = (int)(blockIdx.x * kTX) - (int)(kw / 2), y0 = (int)(blockIdx.y * kTY) - (int)(kh / 2);
  const uint32_t tid = threadIdx.y * kTX + threadIdx.x;
  for (uint32_t i = tid; i < kw * kh; i += kTX * kTY) s_k[i] = kern[i];
  for (uint32_t i = tid; i < tw * th; i += kTX * kTY) {
    const int ty = (int)(i / tw), tx = (int)(i % tw);
    const int yy = min((int)H - 1, max(0, y0 + ty)), xx = min((int)W - 1, max(0, x0 + tx));
#pragma unroll
    for (int c = 0; c < C; ++c) s_img[i * C + c] = img[((size_t)yy * W + xx) * C + c];
  }
  __syncthreads();
  const uint32_t x = blockIdx.x * kTX + threadIdx.x, y = blockIdx.y * kTY + threadIdx.y;
  if (x >= W || y >= H) return;
  K acc[C];
#pragma unroll
  for (int c = 0; c < C; ++c) acc[c] = 0;
  for (uint32_t ky = 0; ky < kh; ++ky) {
    const uint8_t* row = s_img + ((threadIdx.y + ky) * tw + threadIdx.x) * C;
    const K* krow = s_k + ky * kw;
    for (uint32_t kx = 0; kx < kw; ++kx) {
      const K w = krow[kx];
#pragma unroll
      for (int c = 0; c < C; ++c) acc[c] = mac(acc[c], (K)row[kx * C + c], w);
    }
  }
#pragma unroll
  for (int c = 0; c < C; ++c) out[((size_t)y * W + x) * C + c] = clamp_to<S>(acc[c]);
}

// Kernels wider or taller than the tile path takes: the same loop with
// clamped coordinates read through the cache.
template <int C, typename K, typename S>
__global__ void __launch_bounds__(kTX* kTY) filter_global_kernel(const uint8_t* __restrict__ img, uint32_t W,
                                                                uint32_t H, const K* __restrict__ kern, uint32_t kw,
                                                                uint32_t kh, S* __restrict__ out) {
  const uint32_t x = blockIdx.x * kTX + threadIdx.x, y = blockIdx.y * kTY + threadIdx.y;
  if (x >= W || y >= H) return;
  K acc[C];
#pragma unroll
  for (int c = 0; c < C; ++c) acc[c] = 0;
  for (uint32_t ky = 0; ky < kh; ++ky) {
    const long long yy = min((long long)H - 1, max(0ll, (long long)y + ky - kh / 2));
    for (uint32_t kx = 0; kx < kw; ++kx) {
      const long long xx = min((long long)W - 1, max(0ll, (long long)x + kx - kw / 2));
      const K w = __ldg(kern + (size_t)ky * kw + kx);
#pragma unroll
      for (int c = 0; c < C; ++c) acc[c] = mac(acc[c], (K)__ldg(img + ((size_t)yy * W + xx) * C + c), w);
    }
  }
#pragma unroll
  for (int c = 0; c < C; ++c) out[((size_t)y * W + x) * C + c] = clamp_to<S>(acc[c]);
}

constexpr int kRowVec = 4, kRowRows = kFilterStripRows;  // elements and rows per thread
constexpr uint32_t kRowTile = kFilterStripW;              // elements per block row
constexpr uint32_t kRowMaxW = 8, kRowMaxH = 32;           // taps
static_assert(kRowTile == 32 * kRowVec, "a warp per strip row");

template <typename K>
__device__ __forceinline__ K from_byte(uint32_t word, int k) {
  const uint32_t b = (word >> (8 * k)) & 255u;
  if constexpr (std::is_same<K, float>::value)
    return __uint_as_float(0x4B000000u | b) - 8388608.0f;  // 2^23 + b, exact
  else
    return (int32_t)b;
}

template <typename S, typename K>
__device__ __forceinline__ void store_vec(void* out, size_t at, const K (&acc)[kRowVec], uint32_t n, bool aligned) {
  S* o = static_cast<S*>(out) + at;
  S v[kRowVec];
#pragma unroll
  for (int e = 0; e < kRowVec; ++e) v[e] = clamp_to<S>(acc[e]);
  if (aligned && n == kRowVec) {
    if constexpr (sizeof(S) == 1) *reinterpret_cast<uchar4*>(o) = *reinterpret_cast<uchar4*>(v);
    else if constexpr (sizeof(S) == 2) *reinterpret_cast<ushort4*>(o) = *reinterpret_cast<ushort4*>(v);
    else *reinterpret_cast<uint4*>(o) = *reinterpret_cast<uint4*>(v);
  } else {
#pragma unroll
    for (int e = 0; e < kRowVec; ++e)
      if ((uint32_t)e < n) o[e] = v[e];
  }
}

// in_aligned / out_aligned: every row starts on a 4-element boundary.
// (kPitch * C is a multiple of C above any distance to the left of a row.)
template <int C, int KW, typename K>
__global__ void __launch_bounds__(256) filter_rows_kernel(const uint8_t* __restrict__ img, uint32_t W, uint32_t H,
                                                         const K* __restrict__ kern, uint32_t kh, int otype,
                                                         bool in_aligned, bool out_aligned, void* __restrict__ out) {
  extern __shared__ __align__(16) uint8_t smem[];
  constexpr uint32_t kPad = filter_strip_pad(C, KW), kPitch = filter_strip_pitch(C, KW), kWords = kPitch / 4;
  constexpr uint32_t kFirst = kPad - (KW / 2) * C;           // the leftmost tap of element 0
  constexpr uint32_t kLast = kFirst + kRowVec + (KW - 1) * C;  // elements a thread reads per row
  constexpr uint32_t kVecs = (kLast + 3) / 4, kTaps = (KW + 3) & ~3;
  K* s_k = reinterpret_cast<K*>(smem);  // [kh][kTaps]
  K* s_in = s_k + kh * kTaps;
  const uint32_t rows = blockDim.y * kRowRows, nt = 32 * blockDim.y, tid = threadIdx.y * 32 + threadIdx.x;
  const long long n = (long long)W * C;  // elements per image row
  const long long x0 = (long long)blockIdx.x * kRowTile, y0 = (long long)blockIdx.y * rows;
  for (uint32_t i = tid; i < kh * kTaps; i += nt) {
    const uint32_t ky = i / kTaps, kx = i - ky * kTaps;
    s_k[i] = kx < KW ? kern[ky * KW + kx] : K(0);
  }
  for (uint32_t i = tid; i < (rows + kh - 1) * kWords; i += nt) {
    const uint32_t r = i / kWords, c = (i - r * kWords) * 4;
    const long long yy = min((long long)H - 1, max(0ll, y0 + r - kh / 2));
    const long long e = x0 - kPad + c;  // first of four elements
    const uint8_t* row = img + yy * n;
    uint32_t v = 0;
    if (e >= 0 && e + 4 <= n) {
      if (in_aligned) {
        v = __ldg(reinterpret_cast<const uint32_t*>(row + e));
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) v |= (uint32_t)__ldg(row + e + k) << (8 * k);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        // the same channel of the nearest pixel; past the ends by no more than
        // a staged row, so the remainders are of 32 bits
        long long x = e + k;
        if (x < 0) x = (int)(x + (long long)(kPitch * C)) % C;
        else if (x >= n) x = n - C + (int)(x - n) % C;
        v |= (uint32_t)__ldg(row + x) << (8 * k);
      }
    }
    K f[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) f[k] = from_byte<K>(v, k);
    *reinterpret_cast<uint4*>(s_in + r * kPitch + c) = *reinterpret_cast<uint4*>(f);
  }
  __syncthreads();
  const uint32_t ty = threadIdx.y * kRowRows;
  K acc[kRowRows][kRowVec];
#pragma unroll
  for (int r = 0; r < kRowRows; ++r)
#pragma unroll
    for (int e = 0; e < kRowVec; ++e) acc[r][e] = K(0);
  const K* in = s_in + ty * kPitch + threadIdx.x * kRowVec;
  for (uint32_t i = 0; i < kh + kRowRows - 1; ++i, in += kPitch) {
    K v[4 * kVecs];
#pragma unroll
    for (uint32_t q = 0; q < kVecs; ++q)
      *reinterpret_cast<uint4*>(v + 4 * q) = *reinterpret_cast<const uint4*>(in + 4 * q);
#pragma unroll
    for (int r = 0; r < kRowRows; ++r) {
      const uint32_t ky = i - r;  // wraps when the row lies above output row r's window
      if (ky < kh) {
        K w[kTaps];
#pragma unroll
        for (int q = 0; q < kTaps / 4; ++q)
          *reinterpret_cast<uint4*>(w + 4 * q) = *reinterpret_cast<const uint4*>(s_k + ky * kTaps + 4 * q);
#pragma unroll
        for (int kx = 0; kx < KW; ++kx)
#pragma unroll
          for (int e = 0; e < kRowVec; ++e) acc[r][e] = mac(acc[r][e], v[kFirst + e + kx * C], w[kx]);
      }
    }
  }
  const long long x = x0 + threadIdx.x * kRowVec;
  if (x >= n) return;
  const uint32_t left = (uint32_t)min((long long)kRowVec, n - x);
#pragma unroll
  for (int r = 0; r < kRowRows; ++r) {
    const long long y = y0 + ty + r;
    if (y >= H) return;
    const size_t at = (size_t)(y * n + x);
    if constexpr (std::is_same<K, float>::value) {
      if (otype == IPB_ELEM_U8) store_vec<uint8_t>(out, at, acc[r], left, out_aligned);
      else if (otype == IPB_ELEM_U16) store_vec<uint16_t>(out, at, acc[r], left, out_aligned);
      else store_vec<float>(out, at, acc[r], left, out_aligned);
    } else {
      if (otype == IPB_ELEM_U8) store_vec<uint8_t>(out, at, acc[r], left, out_aligned);
      else if (otype == IPB_ELEM_U16) store_vec<uint16_t>(out, at, acc[r], left, out_aligned);
      else if (otype == IPB_ELEM_I16) store_vec<int16_t>(out, at, acc[r], left, out_aligned);
      else store_vec<int32_t>(out, at, acc[r], left, out_aligned);
    }
  }
}

template <int C, int KW, typename K>
cudaError_t launch_filter_rows_k(const uint8_t* img, uint32_t W, uint32_t H, const K* kern, uint32_t kh, uint32_t by,
                                 int otype, size_t osize, void* out, cudaStream_t s) {
  const uint64_t n = (uint64_t)W * C;
  const uint32_t rows = by * kRowRows, gx = (uint32_t)((n + kRowTile - 1) / kRowTile), gy = (H + rows - 1) / rows;
  // at most 40 KB: 4 channels, 8 x 32 taps, 32 rows
  const size_t smem = sizeof(K) * ((size_t)kh * ((KW + 3) & ~3) + (size_t)(rows + kh - 1) * filter_strip_pitch(C, KW));
  const bool in_aligned = n % 4 == 0 && (reinterpret_cast<uintptr_t>(img) & 3u) == 0;
  const bool out_aligned = n % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & (4 * osize - 1)) == 0;
  filter_rows_kernel<C, KW, K><<<dim3(gx, gy), dim3(32, by), smem, s>>>(img, W, H, kern, kh, otype, in_aligned,
                                                                       out_aligned, out);
  count_launch(kKernelFilter);
  return cudaGetLastError();
}

template <int C, typename K>
cudaError_t launch_filter_rows(const uint8_t* img, uint32_t W, uint32_t H, const void* kern, uint32_t kw, uint32_t kh,
                               uint32_t by, int otype, size_t osize, void* out, cudaStream_t s) {
  const K* k = static_cast<const K*>(kern);
  switch (kw) {
    case 1: return launch_filter_rows_k<C, 1, K>(img, W, H, k, kh, by, otype, osize, out, s);
    case 2: return launch_filter_rows_k<C, 2, K>(img, W, H, k, kh, by, otype, osize, out, s);
    case 3: return launch_filter_rows_k<C, 3, K>(img, W, H, k, kh, by, otype, osize, out, s);
    case 4: return launch_filter_rows_k<C, 4, K>(img, W, H, k, kh, by, otype, osize, out, s);
    case 5: return launch_filter_rows_k<C, 5, K>(img, W, H, k, kh, by, otype, osize, out, s);
    case 6: return launch_filter_rows_k<C, 6, K>(img, W, H, k, kh, by, otype, osize, out, s);
    case 7: return launch_filter_rows_k<C, 7, K>(img, W, H, k, kh, by, otype, osize, out, s);
    default: return launch_filter_rows_k<C, 8, K>(img, W, H, k, kh, by, otype, osize, out, s);
  }
}

template <int C, typename K, typename S>
cudaError_t launch_filter_t(const uint8_t* img, uint32_t W, uint32_t H, const void* kern, uint32_t kw, uint32_t kh,
                            void* out, cudaStream_t s) {
  const dim3 grid((W + kTX - 1) / kTX, (H + kTY - 1) / kTY), block(kTX, kTY);
  if (grid.y > 65535u) return cudaErrorInvalidValue;
  if (kw <= kRowMaxW && kh <= kRowMaxH)
    if (const uint32_t by = filter_strip_warps(W, H, C, kw, kh, (uint32_t)device_sm_count()))
      return launch_filter_rows<C, K>(img, W, H, kern, kw, kh, by, elem_of<S>(), sizeof(S), out, s);
  const K* k = static_cast<const K*>(kern);
  S* o = static_cast<S*>(out);
  if (kw <= kMaxTileKernel && kh <= kMaxTileKernel) {
    const size_t smem = align_up((size_t)kw * kh * sizeof(K), 16) + (size_t)(kTX + kw - 1) * (kTY + kh - 1) * C;
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(filter_tile_kernel<C, K, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem);
      if (e != cudaSuccess) return e;
    }
    filter_tile_kernel<C, K, S><<<grid, block, smem, s>>>(img, W, H, k, kw, kh, o);
  } else {
    filter_global_kernel<C, K, S><<<grid, block, 0, s>>>(img, W, H, k, kw, kh, o);
  }
  count_launch(kKernelFilter);
  return cudaGetLastError();
}

template <int C>
cudaError_t launch_filter_c(const uint8_t* img, uint32_t W, uint32_t H, const void* kern, int ktype, uint32_t kw,
                            uint32_t kh, int otype, void* out, cudaStream_t s) {
  if (ktype == IPB_KERNEL_TYPE_F32) {
    switch (otype) {
      case IPB_ELEM_U8: return launch_filter_t<C, float, uint8_t>(img, W, H, kern, kw, kh, out, s);
      case IPB_ELEM_U16: return launch_filter_t<C, float, uint16_t>(img, W, H, kern, kw, kh, out, s);
      case IPB_ELEM_F32: return launch_filter_t<C, float, float>(img, W, H, kern, kw, kh, out, s);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (otype) {
    case IPB_ELEM_U8: return launch_filter_t<C, int32_t, uint8_t>(img, W, H, kern, kw, kh, out, s);
    case IPB_ELEM_U16: return launch_filter_t<C, int32_t, uint16_t>(img, W, H, kern, kw, kh, out, s);
    case IPB_ELEM_I16: return launch_filter_t<C, int32_t, int16_t>(img, W, H, kern, kw, kh, out, s);
    case IPB_ELEM_I32: return launch_filter_t<C, int32_t, int32_t>(img, W, H, kern, kw, kh, out, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

bool filter_types_supported(int ktype, int otype) {
  if (ktype == IPB_KERNEL_TYPE_F32) return otype == IPB_ELEM_U8 || otype == IPB_ELEM_U16 || otype == IPB_ELEM_F32;
  if (ktype == IPB_KERNEL_TYPE_I32)
    return otype == IPB_ELEM_U8 || otype == IPB_ELEM_U16 || otype == IPB_ELEM_I16 || otype == IPB_ELEM_I32;
  return false;
}

cudaError_t launch_filter(const uint8_t* img, uint32_t W, uint32_t H, uint32_t channels, const void* kern, int ktype,
                          uint32_t kw, uint32_t kh, int otype, void* out, cudaStream_t s) {
  if (W == 0 || H == 0) return cudaSuccess;
  switch (channels) {
    case 1: return launch_filter_c<1>(img, W, H, kern, ktype, kw, kh, otype, out, s);
    case 3: return launch_filter_c<3>(img, W, H, kern, ktype, kw, kh, otype, out, s);
    case 4: return launch_filter_c<4>(img, W, H, kern, ktype, kw, kh, otype, out, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace ipb
