// tm_sat.cu -- imageproc's integral_image / integral_squared_image on the
// device (src/integral_image.rs:50-153): a (W+1) x (H+1) table per channel,
// S[y][x][c] = sum of F(x', y')[c] (or its square) over x' < x, y' < y, with a
// zero top row and left column; channels (1 Luma, 3 Rgb, 4 Rgba) interleaved
// like the source pixels.
//
// Element types: u64 (exact for any image that fits in device memory) and
// u32, whose additions wrap modulo 2^32 like the reference's u32 sums in a
// release build; because addition modulo 2^32 is associative, the parallel
// scans below give the reference's sequential result bit for bit.
//
// One channel (sat_strip_sums, sat_strip_cols, sat_tiles): the table is
// written once. The image is cut into strips of 16 rows and tiles of 1024
// columns. The first pass reads the image and leaves in each strip's last
// table row the strip's column sums, prefix-summed along x, and in the tile's
// own part of each other row the row's sum ahead of the tile. The second
// sums the strips' last rows down the image (in place: they are final then).
// The third forms every other row of a tile from the final row above its
// strip, its rows' sums ahead of the tile and the tile's own two-dimensional
// prefix (16 rows at once: per-thread runs of four columns, one warp scan and
// one exchange between warps per row, staged in 32 bits so that warps store
// contiguous runs). Nothing but the table holds intermediates. The bound is
// the table's one write: 4096 x 4096 squared u64, 23 us for image and table
// at the copy rate; two passes over the table 117 us, this 60 us.
//
// Three and four channels: two passes over the table: a row scan (one block
// per row, tiles of 1024 pixels scanned block-wide and stored through shared
// memory in contiguous runs), then a column scan of the (W+1)*C interleaved
// columns in place (32 row segments per block: segment totals, then the
// rescan with offsets).
#include "tm_common.cuh"
#include "tm_internal.h"
#include "tm_strip.h"

namespace ipb {
namespace {

constexpr int kRowThreads = 256;
constexpr int kPix = 4;                          // pixels per thread per tile
constexpr int kTile = kRowThreads * kPix;        // pixels per tile

// Row pass: each block scans whole rows in tiles of kTile pixels -- a
// per-thread scan of kPix pixels, a block-wide exclusive scan of the thread
// totals per channel, the running carry of the row -- and stages the tile in
// shared memory so that warps store contiguous runs of the table.
template <typename T, bool kSquare, int C>
__global__ void __launch_bounds__(kRowThreads) sat_rows_kernel(const uint8_t* __restrict__ img, uint32_t W,
                                                               uint32_t H, T* __restrict__ sat) {
  __shared__ T s_tile[kTile * C];
  __shared__ T s_warp[C][kRowThreads / 32];
  const uint32_t pitch = (W + 1) * C;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t y = blockIdx.x; y < H; y += gridDim.x) {
    const uint8_t* row = img + (size_t)y * W * C;
    T* out = sat + (size_t)(y + 1) * pitch;
    if (threadIdx.x < C) out[threadIdx.x] = 0;
    T carry[C];
#pragma unroll
    for (int c = 0; c < C; ++c) carry[c] = 0;
    for (uint32_t tile = 0; tile < W; tile += kTile) {
      T pre[kPix][C], acc[C];
#pragma unroll
      for (int c = 0; c < C; ++c) acc[c] = 0;
#pragma unroll
      for (int j = 0; j < kPix; ++j) {
        const uint32_t x = tile + threadIdx.x * kPix + j;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const T v = x < W ? (T)row[(size_t)x * C + c] : (T)0;
          acc[c] += kSquare ? v * v : v;
          pre[j][c] = acc[c];
        }
      }
      T off[C], tot[C];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        T incl = acc[c];
        for (int o = 1; o < 32; o <<= 1) {
          const T n = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += n;
        }
        if (lane == 31) s_warp[c][warp] = incl;
        off[c] = incl - acc[c];
      }
      __syncthreads();
#pragma unroll
      for (int c = 0; c < C; ++c) {
        tot[c] = 0;
        for (int k = 0; k < kRowThreads / 32; ++k) {
          const T wsum = s_warp[c][k];
          if (k < warp) off[c] += wsum;
          tot[c] += wsum;
        }
      }
#pragma unroll
      for (int j = 0; j < kPix; ++j)
#pragma unroll
        for (int c = 0; c < C; ++c) s_tile[(threadIdx.x * kPix + j) * C + c] = carry[c] + off[c] + pre[j][c];
      __syncthreads();
      const uint32_t n = min((uint32_t)kTile, W - tile) * C;
      T* dst = out + (size_t)(tile + 1) * C;
      for (uint32_t e = threadIdx.x; e < n; e += kRowThreads) dst[e] = s_tile[e];
#pragma unroll
      for (int c = 0; c < C; ++c) carry[c] += tot[c];
      __syncthreads();  // s_tile and s_warp are rewritten by the next tile
    }
  }
}

// Column pass: 32 columns x 32 row segments per block; each warp sums its
// segment of 32 columns (coalesced rows), the block turns the segment totals
// into offsets, and each warp rescans its segment adding the offset.
constexpr int kSegs = 32;

template <typename T>
__global__ void __launch_bounds__(32 * kSegs) sat_cols_kernel(uint32_t cols, uint32_t H, T* __restrict__ sat) {
  __shared__ T s_tot[kSegs][33];
  const uint32_t col = blockIdx.x * 32 + (threadIdx.x & 31);
  const int segi = threadIdx.x >> 5;
  const uint32_t seg = (H + kSegs - 1) / kSegs;
  const uint32_t r0 = 1 + segi * seg;
  const uint32_t r1 = min(H + 1, r0 + seg);
  T tot = 0;
  if (col < cols) {
#pragma unroll 8
    for (uint32_t r = r0; r < r1; ++r) tot += sat[(size_t)r * cols + col];
  }
  s_tot[segi][threadIdx.x & 31] = tot;
  __syncthreads();
  T run = 0;
  for (int k = 0; k < segi; ++k) run += s_tot[k][threadIdx.x & 31];
  if (col < cols) {
    // eight rows loaded before any is stored, so the reads overlap instead of
    // waiting on each other through the stores
    uint32_t r = r0;
    for (; r + 8 <= r1; r += 8) {
      T v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = sat[(size_t)(r + k) * cols + col];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        run += v[k];
        sat[(size_t)(r + k) * cols + col] = run;
      }
    }
    for (; r < r1; ++r) {
      T* p = sat + (size_t)r * cols + col;
      run += *p;
      *p = run;
    }
  }
}

constexpr uint32_t kTileCols = 1024, kTileThreads = 256;

// A thread's four pixels at x of each of a strip's first n rows, zero past the
// image: one word per row where rows are word-aligned, else the two aligned
// words around them, without a branch between the rows' loads (with one, or
// byte by byte, the rows' latencies added up and odd widths were slower than
// by a pass per row and one per column); by bytes in the strips at the image's
// ends, where the words would leave it.
__device__ __forceinline__ void strip_pixels(const uint8_t* __restrict__ img, uint32_t W, uint32_t H, uint32_t y0,
                                             uint32_t n, uint32_t x, bool aligned, uint32_t (&v)[kStripRows]) {
  const uint8_t* p = img + (size_t)y0 * W + min(x, W - 1);
  const uint32_t in = x < W ? min(4u, W - x) : 0u, mask = in < 4 ? (1u << (8 * in)) - 1u : 0xFFFFFFFFu;
  if (aligned) {
#pragma unroll
    for (uint32_t r = 0; r < kStripRows; ++r)
      v[r] = r < n && in ? __ldg(reinterpret_cast<const uint32_t*>(p + (size_t)r * W)) : 0u;
  } else if (strip_words_inside(W, H, y0)) {
#pragma unroll
    for (uint32_t r = 0; r < kStripRows; ++r) {
      const uint8_t* g = p + (size_t)r * W;
      const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(g) & 3u);
      const uint32_t* w = reinterpret_cast<const uint32_t*>(g - off);
      v[r] = __byte_perm(__ldg(w), __ldg(w + 1), 0x3210u + off * 0x1111u) & mask;
    }
  } else {
#pragma unroll
    for (uint32_t r = 0; r < kStripRows; ++r) {
      v[r] = 0;
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k)
        if (r < n && k < in) v[r] |= (uint32_t)__ldg(p + (size_t)r * W + k) << (8 * k);
    }
  }
}
template <bool kSquare>
__device__ __forceinline__ uint32_t term(uint32_t v, int k) {
  const uint32_t b = (v >> (8 * k)) & 255u;
  return kSquare ? b * b : b;
}

// First pass: one block per strip. Sums of up to 16 rows x 1024 columns stay
// below 2^32 (65025 * 16384).
template <typename T, bool kSquare>
__global__ void __launch_bounds__(kTileThreads) sat_strip_sums_kernel(const uint8_t* __restrict__ img, uint32_t W,
                                                                     uint32_t H, bool aligned, T* __restrict__ sat) {
  __shared__ uint32_t s_row[kStripRows][kTileThreads / 32];
  __shared__ uint32_t s_col[kTileThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t pitch = (size_t)W + 1;
  for (uint32_t strip = blockIdx.x; strip * kStripRows < H; strip += gridDim.x) {
    const uint32_t y0 = strip * kStripRows, rows = min(kStripRows, H - y0);
    const bool whole = rows == kStripRows;  // the last row's sums are wanted
    if (threadIdx.x < rows) sat[(y0 + 1 + threadIdx.x) * pitch] = 0;  // left column
    T col_carry = 0, row_carry = 0;         // row_carry: thread r's row
    for (uint32_t tile = 0; tile < W; tile += kTileCols) {
      const uint32_t x = tile + 4 * threadIdx.x;
      uint32_t v[kStripRows], c[4] = {0u, 0u, 0u, 0u};
      strip_pixels(img, W, H, y0, rows, x, aligned, v);
#pragma unroll
      for (uint32_t r = 0; r < kStripRows; ++r) {
        uint32_t t;
        if constexpr (kSquare) t = __dp4a(v[r], v[r], 0u);
        else t = __dp4a(v[r], 0x01010101u, 0u);
        t = __reduce_add_sync(0xffffffffu, t);
        if (lane == 0) s_row[r][warp] = t;
#pragma unroll
        for (int k = 0; k < 4; ++k) c[k] += term<kSquare>(v[r], k);
      }
      const uint32_t own = c[0] + c[1] + c[2] + c[3];
      uint32_t incl = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
      }
      if (lane == 31) s_col[warp] = incl;
      __syncthreads();
      uint32_t off = incl - own, tot = 0;
#pragma unroll
      for (int k = 0; k < (int)kTileThreads / 32; ++k) {
        if (k < warp) off += s_col[k];
        tot += s_col[k];
      }
      if (whole) {
        T run = col_carry + off;
        T* dst = sat + (size_t)(y0 + kStripRows) * pitch + 1;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
          run += c[k];
          if (x + k < W) dst[x + k] = run;
        }
      }
      col_carry += tot;
      // rows whose table row is formed by the third pass
      if (threadIdx.x < (whole ? kStripRows - 1 : rows)) {
        sat[(size_t)(y0 + 1 + threadIdx.x) * pitch + 1 + tile] = row_carry;
#pragma unroll
        for (int k = 0; k < (int)kTileThreads / 32; ++k) row_carry += s_row[threadIdx.x][k];
      }
      __syncthreads();  // s_row and s_col are rewritten by the next tile
    }
  }
}

// Second pass: sums the strips' last table rows down the image, 32 columns x
// 32 segments of strips per block.
template <typename T>
__global__ void __launch_bounds__(1024) sat_strip_cols_kernel(uint32_t W, uint32_t strips, T* __restrict__ sat) {
  __shared__ T s_tot[32][33];
  const uint32_t col = blockIdx.x * 32 + (threadIdx.x & 31);
  const int segi = threadIdx.x >> 5;
  const uint32_t seg = (strips + 31) / 32;
  const uint32_t s0 = segi * seg, s1 = min(strips, s0 + seg);
  const size_t step = (size_t)kStripRows * (W + 1);
  T* p = sat + (size_t)kStripRows * (W + 1) + 1 + col;  // strip 0's last row
  T tot = 0;
  if (col < W) {
#pragma unroll 8
    for (uint32_t i = s0; i < s1; ++i) tot += p[i * step];
  }
  s_tot[segi][threadIdx.x & 31] = tot;
  __syncthreads();
  T run = 0;
  for (int k = 0; k < segi; ++k) run += s_tot[k][threadIdx.x & 31];
  if (col < W) {
    uint32_t i = s0;
    for (; i + 8 <= s1; i += 8) {  // eight rows loaded before any is stored
      T v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = p[(i + k) * step];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        run += v[k];
        p[(i + k) * step] = run;
      }
    }
    for (; i < s1; ++i) {
      run += p[i * step];
      p[i * step] = run;
    }
  }
}

// Third pass: one block per tile.
constexpr uint32_t kTileSmem = kStripRows * kTileCols * 4;

template <typename T, bool kSquare>
__global__ void __launch_bounds__(kTileThreads) sat_tiles_kernel(const uint8_t* __restrict__ img, uint32_t W,
                                                                uint32_t H, uint32_t tiles_x, bool aligned,
                                                                T* __restrict__ sat) {
  extern __shared__ __align__(16) uint32_t s_tile[];  // [kStripRows][kTileCols] prefix within the tile
  __shared__ uint32_t s_warp[kStripRows][kTileThreads / 32];
  __shared__ T s_ahead[kStripRows];  // sum of the strip's rows so far, ahead of the tile
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t pitch = (size_t)W + 1;
  const uint32_t strip = blockIdx.x / tiles_x, tile = (blockIdx.x - strip * tiles_x) * kTileCols;
  const uint32_t y0 = strip * kStripRows, rows = min(kStripRows, H - y0);
  const uint32_t form = rows == kStripRows ? kStripRows - 1 : rows;  // the whole strip's last row is final
  const uint32_t x = tile + 4 * threadIdx.x;
  uint32_t v[kStripRows];
  strip_pixels(img, W, H, y0, form, x, aligned, v);
  // the row above the strip, in the columns this thread stores
  T base[4];
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
    const uint32_t c = tile + threadIdx.x + k * kTileThreads;
    base[k] = strip && c < W ? sat[(size_t)y0 * pitch + 1 + c] : T(0);
  }
  if (warp == 0) {
    T ahead = lane < (int)form ? sat[(size_t)(y0 + 1 + lane) * pitch + 1 + tile] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T n = __shfl_up_sync(0xffffffffu, ahead, o);
      if (lane >= o) ahead += n;
    }
    if (lane < (int)kStripRows) s_ahead[lane] = ahead;
  }
  uint32_t c0 = 0, c1 = 0, c2 = 0, c3 = 0, own[kStripRows], excl[kStripRows];
#pragma unroll
  for (uint32_t r = 0; r < kStripRows; ++r) {
    c0 += term<kSquare>(v[r], 0);
    c1 += term<kSquare>(v[r], 1);
    c2 += term<kSquare>(v[r], 2);
    c3 += term<kSquare>(v[r], 3);
    own[r] = c0 + c1 + c2 + c3;
    excl[r] = own[r];
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
    for (uint32_t r = 0; r < kStripRows; ++r) {
      const uint32_t n = __shfl_up_sync(0xffffffffu, excl[r], o);
      if (lane >= o) excl[r] += n;
    }
  }
#pragma unroll
  for (uint32_t r = 0; r < kStripRows; ++r) {
    if (lane == 31) s_warp[r][warp] = excl[r];
    excl[r] -= own[r];
  }
  __syncthreads();  // also: every read of the table above is done before any store below
  c0 = c1 = c2 = c3 = 0;
#pragma unroll
  for (uint32_t r = 0; r < kStripRows; ++r) {
    uint32_t run = excl[r];
#pragma unroll
    for (int k = 0; k < (int)kTileThreads / 32; ++k)
      if (k < warp) run += s_warp[r][k];
    c0 += term<kSquare>(v[r], 0);
    c1 += term<kSquare>(v[r], 1);
    c2 += term<kSquare>(v[r], 2);
    c3 += term<kSquare>(v[r], 3);
    uint4 q;
    q.x = run + c0;
    q.y = q.x + c1;
    q.z = q.y + c2;
    q.w = q.z + c3;
    *reinterpret_cast<uint4*>(s_tile + r * kTileCols + 4 * threadIdx.x) = q;
  }
  __syncthreads();
#pragma unroll 4
  for (uint32_t r = 0; r < form; ++r) {
    const T ahead = s_ahead[r];
    T* dst = sat + (size_t)(y0 + 1 + r) * pitch + 1 + tile;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      const uint32_t c = threadIdx.x + k * kTileThreads;
      if (tile + c < W) dst[c] = base[k] + ahead + (T)s_tile[r * kTileCols + c];
    }
  }
}

template <typename T, bool kSquare>
cudaError_t launch_sat_one_channel(const uint8_t* img, uint32_t W, uint32_t H, T* sat, cudaStream_t s) {
  const uint32_t strips = (H + kStripRows - 1) / kStripRows, whole = H / kStripRows;
  const uint32_t tiles_x = (W + kTileCols - 1) / kTileCols;
  const bool aligned = W % 4 == 0 && (reinterpret_cast<uintptr_t>(img) & 3u) == 0;
  static PerDeviceOnce attr;
  cudaError_t e = attr.run([] {
    return cudaFuncSetAttribute(sat_tiles_kernel<T, kSquare>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kTileSmem);
  });
  if (e != cudaSuccess) return e;
  sat_strip_sums_kernel<T, kSquare><<<strips < 65535u ? strips : 65535u, kTileThreads, 0, s>>>(img, W, H, aligned,
                                                                                             sat);
  count_launch(kKernelIntegralRows);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (whole > 1) {
    sat_strip_cols_kernel<T><<<(W + 31) / 32, 1024, 0, s>>>(W, whole, sat);
    count_launch(kKernelIntegralCols);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  sat_tiles_kernel<T, kSquare><<<strips * tiles_x, kTileThreads, kTileSmem, s>>>(img, W, H, tiles_x, aligned, sat);
  count_launch(kKernelIntegralCols);
  return cudaGetLastError();
}

template <typename T, bool kSquare, int C>
cudaError_t launch_sat_typed(const uint8_t* img, uint32_t W, uint32_t H, T* sat, cudaStream_t s) {
  const uint32_t cols = (W + 1) * C;
  cudaError_t e = cudaMemsetAsync(sat, 0, sizeof(T) * cols, s);  // top row
  if (e != cudaSuccess || H == 0) return e;
  if (W == 0) return cudaMemsetAsync(sat, 0, sizeof(T) * (size_t)cols * (H + 1), s);
  if constexpr (C == 1) {
    // One block per strip sums it tile after tile, so with few strips the SMs
    // stand idle and the row pass, a block per row, is the faster one; rows
    // that are not word-aligned cost the strips two words per four pixels,
    // twice. u64 squares, row and column pass against this: 512 x 2048 16.8
    // and 21.2 us, 900 x 2048 24.8 and 21.1, 1024 x 4096 29.5 and 30.3, 1500
    // x 4096 42.5 and 34, 4096 x 4096 117 and 60; 1500 x 2047 29.6 and 32.6,
    // 2111 x 4095 50.7 and 50.3, 3333 x 4095 86 and 80. Tiles are counted in
    // 31 bits.
    const uint32_t strips = H / kStripRows, tiles_x = (W + kTileCols - 1) / kTileCols;
    const bool words = W % 4 == 0 && (reinterpret_cast<uintptr_t>(img) & 3u) == 0;
    if (strips >= (words ? 72 + 4 * tiles_x : 100 + 25 * tiles_x) &&
        (uint64_t)(strips + 1) * tiles_x < 0x7FFFFFFFull)
      return launch_sat_one_channel<T, kSquare>(img, W, H, sat, s);
  }
  sat_rows_kernel<T, kSquare, C><<<H < 65535u ? H : 65535u, kRowThreads, 0, s>>>(img, W, H, sat);
  count_launch(kKernelIntegralRows);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  sat_cols_kernel<T><<<(cols + 31) / 32, 32 * kSegs, 0, s>>>(cols, H, sat);
  count_launch(kKernelIntegralCols);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_sat_t(const uint8_t* img, uint32_t W, uint32_t H, uint32_t channels, bool squared, T* sat,
                         cudaStream_t s) {
  switch (channels * 2 + (squared ? 1 : 0)) {
    case 2: return launch_sat_typed<T, false, 1>(img, W, H, sat, s);
    case 3: return launch_sat_typed<T, true, 1>(img, W, H, sat, s);
    case 6: return launch_sat_typed<T, false, 3>(img, W, H, sat, s);
    case 7: return launch_sat_typed<T, true, 3>(img, W, H, sat, s);
    case 8: return launch_sat_typed<T, false, 4>(img, W, H, sat, s);
    case 9: return launch_sat_typed<T, true, 4>(img, W, H, sat, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_sat(const uint8_t* img, uint32_t W, uint32_t H, uint32_t channels, bool squared, int bits,
                       void* sat, cudaStream_t s) {
  if (bits == 32) return launch_sat_t<uint32_t>(img, W, H, channels, squared, static_cast<uint32_t*>(sat), s);
  return launch_sat_t<unsigned long long>(img, W, H, channels, squared, static_cast<unsigned long long*>(sat), s);
}

}  // namespace ipb
