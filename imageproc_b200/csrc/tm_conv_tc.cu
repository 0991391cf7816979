// tm_conv_tc.cu -- the proposal network's 3x3 32 -> 32 convolution on the
// 5th-generation tensor cores (tcgen05.mma kind::f16: bf16 operands from
// shared memory, fp32 accumulators in tensor memory).
//
// Formulation (implicit GEMM per output row segment): a tile is one output
// row y of one image and 128 consecutive pixels x0 .. x0 + 127 (M = 128 =
// tensor-memory lanes), all 32 output channels (N = 32), and K = 9 taps x 32
// input channels = 18 MMAs of K = 16. The A operand of tap (ky, kx) is input
// row y + ky - 1 at pixels x0 + kx - 1 .. : the staged row, in the canonical
// no-swizzle K-major layout (for each 8-channel chunk, pixels 16 bytes apart),
// started kx pixels (16 * kx bytes) later, so one staged row serves all three
// kx taps. B is the tap's weights [co][ci], resident for the CTA's life.
//
// Images narrower than half a tile share one: a tile is the same row of as many
// images as fit 128 lanes side by side, one zero pixel between them (the right
// padding of one is the left padding of the next), so 24-pixel training crops
// go five to a tile and 12-pixel templates nine.
//
// A CTA walks a band of output rows of one column segment (or group of
// images), so each input row is loaded once and used by three tiles: a ring of
// staged rows, filled by a loader warp with one bulk copy per 8-channel chunk
// and image (a chunk's pixels are contiguous; the slots' padding is zeroed
// once), an MMA warp whose elected lane issues a tile's 18 MMAs into one of two
// accumulators, and four epilogue warps (one per tensor-memory lane quadrant)
// that add the bias, apply the ReLU, round to bf16 and store the row-chunked
// activations. mbarriers hand rows and accumulators between the roles; every
// wait is bounded and a wait that runs out sets the error word.
// What bounded it: the loader's per-pixel copies with their index arithmetic,
// one row in flight. A 2048 x 2048 layer (82 us at the copy rate) went from 215
// to 154 us, a layer of 128 crops of 24 x 24 from 40 to 14 us.
#include <algorithm>

#include "imageproc_b200.h"
#include "tm_internal.h"
#include "tm_learned.cuh"
#include "tm_sm100.cuh"

namespace ipb {
namespace learned {
namespace {

using namespace sm100;

constexpr int kSeg = 128;                 // output pixels per tile (tensor-memory lanes)
constexpr int kRowPx = 136;               // staged pixels per row: kSeg + 2 halo, padded to 8
constexpr int kChunkBytes = kRowPx * 16;  // one 8-channel chunk of a staged row (2176 B)
constexpr int kRowBytes = kChunks * kChunkBytes;  // 8704 B
constexpr int kRing = 8;                  // staged input rows
constexpr int kWBytes = 9 * kChunks * kC * 16;    // 18432 B of weights
constexpr int kThreadsTc = 192;           // warp 0 MMA, warp 1 loader, warps 2..5 epilogue
constexpr uint32_t kTmemColsTc = 64;      // two accumulators of 32 columns

struct TcSmemLayout {
  static constexpr uint32_t w = 0;
  static constexpr uint32_t ring = kWBytes;
  static constexpr uint32_t bars = ring + kRing * kRowBytes;   // 21 mbarriers
  static constexpr uint32_t misc = bars + 24 * 8;              // tmem address, error flag
  static constexpr uint32_t bias = misc + 16;                  // 32 floats
  static constexpr uint32_t total = bias + kC * 4;
};

// instruction descriptor of kind::f16: bf16 A and B, fp32 D, both K-major, M x N
__host__ __device__ constexpr uint32_t idesc_bf16_f32(uint32_t M, uint32_t N) {
  return (1u << 4)            // D format: f32
         | (1u << 7)          // A format: bf16
         | (1u << 10)         // B format: bf16
         | ((N >> 3) << 17)   // N / 8
         | ((M >> 4) << 24);  // M / 16
}

__device__ __forceinline__ void mma_bf16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// two f32 rounded to bf16 (nearest even), lo in the low half
__device__ __forceinline__ uint32_t bf16x2_rn(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

struct TcArgs {
  const uint4* in;
  uint4* out;
  const uint16_t* wt;   // [tap][co][ci] bf16
  const float* bias;    // [32]
  int relu;
  uint32_t n, H, W, band;  // images, their size, rows per CTA
  uint32_t group;          // images per tile
  unsigned long long wait_ns;
  uint32_t stall;       // pipeline_stall() at launch
  unsigned int* err;    // error word or null
  unsigned int tag;
  const uint4* mask;    // or null: keeps an output bf16 only where this activation is > 0 (ReLU')
};

__global__ void __launch_bounds__(kThreadsTc) conv_tc_kernel(const TcArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* row_full = reinterpret_cast<uint64_t*>(smem + TcSmemLayout::bars);
  uint64_t* row_empty = row_full + kRing;
  uint64_t* acc_full = row_empty + kRing;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* drain = acc_empty + 2;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + TcSmemLayout::misc);
  volatile uint32_t* s_err = s_tmem + 1;
  float* s_bias = reinterpret_cast<float*>(smem + TcSmemLayout::bias);

  const uint32_t n0 = blockIdx.z * a.group, ni = min(a.group, a.n - n0);  // the tile's images
  const uint32_t x0 = blockIdx.x * kSeg;
  const uint32_t yb = blockIdx.y * a.band;
  const uint32_t ntiles = yb < a.H ? min(a.band, a.H - yb) : 0u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // weights: [tap][chunk][co] 16-byte units (K-major B per tap and chunk), all
  // of a thread's loads in flight at once
  {
    static_assert(9 * kC * kChunks % kThreadsTc == 0, "weight units per thread");
    constexpr int kPer = 9 * kC * kChunks / kThreadsTc;
    uint4 v[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) v[k] = reinterpret_cast<const uint4*>(a.wt)[threadIdx.x + k * kThreadsTc];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const uint32_t i = threadIdx.x + k * kThreadsTc, c = i & 3u, row = i >> 2, tap = row / kC, co = row % kC;
      reinterpret_cast<uint4*>(smem + TcSmemLayout::w)[(tap * kChunks + c) * kC + co] = v[k];
    }
  }
  for (uint32_t i = threadIdx.x; i < (uint32_t)(kRing * kRowBytes / 16); i += kThreadsTc)
    reinterpret_cast<uint4*>(smem + TcSmemLayout::ring)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (threadIdx.x < kC) s_bias[threadIdx.x] = a.bias ? a.bias[threadIdx.x] : 0.f;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kRing; ++s) {
      mbar_init(&row_full[s], 1);
      mbar_init(&row_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);
    }
    mbar_init(drain, 1);
    *s_err = 0;
    mbar_init_fence();
  }
  fence_proxy_async_smem();  // weights and padding are read by the tensor cores
  if (warp == 0) {
    tmem_alloc(s_tmem, kTmemColsTc);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  const unsigned long long deadline = global_ns() + a.wait_ns;
  const uint32_t ring0 = smem_u32(smem + TcSmemLayout::ring);
  const uint32_t w0 = smem_u32(smem + TcSmemLayout::w);

  if (warp == 1) {
    // loader: input rows yb - 1 .. yb + ntiles (index i = row - yb + 1). Copy
    // l = lane, lane + 32, ... takes chunk l % 4 of image l / 4: pixels x0 - 1
    // .. x0 + 128 inside the image, to staged pixel 0 (1 at the left edge) on,
    // images W + 1 pixels apart.
    const uint32_t nrows = ntiles ? ntiles + 2 : 0u;
    const uint32_t xa = x0 ? x0 - 1 : 0u, xb = min(a.W, x0 + (uint32_t)kSeg + 1), bytes = (xb - xa) * 16;
    const uint32_t px0 = x0 ? 0u : 1u;
    uint32_t i = 0;
    for (; i < nrows; ++i) {
      const uint32_t s = i % kRing, u = i / kRing;
      if (!__all_sync(0xffffffffu, u == 0 || mbar_wait_sleep(&row_empty[s], (u - 1) & 1u, deadline))) {
        *s_err = 1;
        break;
      }
      const int y = (int)yb - 1 + (int)i;
      const uint32_t dst0 = ring0 + s * kRowBytes;
      if (y >= 0 && y < (int)a.H) {
        if (lane == 0) mbar_arrive_expect_tx(&row_full[s], bytes * kChunks * ni);
        __syncwarp();
        for (uint32_t l = lane; l < kChunks * ni; l += 32) {
          const uint32_t c = l % kChunks, im = l / kChunks;
          bulk_g2s(dst0 + c * kChunkBytes + (px0 + im * (a.W + 1)) * 16,
                   a.in + ((((size_t)n0 + im) * a.H + y) * kChunks + c) * a.W + xa, bytes, &row_full[s]);
        }
      } else {
        // a row of padding (the slot may hold an earlier row)
        for (uint32_t l = lane; l < (uint32_t)(kRowBytes / 16); l += 32)
          reinterpret_cast<uint4*>(smem + TcSmemLayout::ring + s * kRowBytes)[l] = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&row_full[s]);
      }
    }
    // no copy is in flight when the CTA leaves, whatever the other roles did
    for (uint32_t j = i > (uint32_t)kRing ? i - kRing : 0u; j < i; ++j)
      mbar_wait(&row_full[j % kRing], (j / kRing) & 1u, global_ns() + kDefaultWaitNs);
  } else if (warp == 0) {
    // MMA issue: tile k reads staged rows k, k + 1, k + 2 (input rows y - 1 .. y + 1)
    constexpr uint32_t idesc = idesc_bf16_f32(kSeg, kC);
    const bool leader = elect_one();
    // test hook: a wait on the drain barrier, which nothing arrives at before the end
    if (a.stall && !__all_sync(0xffffffffu, mbar_wait(drain, 0, deadline))) *s_err = 1;
    for (uint32_t k = 0; k < ntiles && !*s_err; ++k) {
      bool ok = true;
      for (uint32_t j = 0; j < 3 && ok; ++j) ok = mbar_wait(&row_full[(k + j) % kRing], ((k + j) / kRing) & 1u, deadline);
      const uint32_t b = k & 1u, v = k >> 1;
      if (ok && v > 0) ok = mbar_wait(&acc_empty[b], (v - 1) & 1u, deadline);
      if (!__all_sync(0xffffffffu, ok)) {
        *s_err = 1;
        break;
      }
      tc_fence_after();
      if (leader) {
        const uint32_t d = tmem + b * kC;
#pragma unroll
        for (uint32_t tap = 0; tap < 9; ++tap) {
          const uint32_t ky = tap / 3, kx = tap % 3;
          const uint32_t arow = ring0 + ((k + ky) % kRing) * kRowBytes + kx * 16;
#pragma unroll
          for (uint32_t js = 0; js < 2; ++js) {
            const uint64_t ad = smem_desc_noswizzle(arow + 2 * js * kChunkBytes, kChunkBytes, 128);
            const uint64_t bd = smem_desc_noswizzle(w0 + (tap * kChunks + 2 * js) * kC * 16, kC * 16, 128);
            mma_bf16_ss(d, ad, bd, idesc, (tap | js) != 0);
          }
        }
        mma_commit(&acc_full[b]);
        mma_commit(&row_empty[k % kRing]);  // staged row k is not read again
      }
      __syncwarp();
    }
  } else {
    // epilogue: warp's lane quadrant q; lane m = 32 q + lane is pixel x0 + m, or
    // pixel m % (W + 1) of image m / (W + 1)
    const uint32_t q = warp & 3;
    const uint32_t m = 32 * q + lane, im = a.group > 1 ? m / (a.W + 1) : 0u;
    const uint32_t x = a.group > 1 ? m - im * (a.W + 1) : x0 + m;
    const bool inside = im < ni && x < a.W;
    const size_t first = (((size_t)n0 + im) * a.H * kChunks) * a.W + x;
    for (uint32_t k = 0; k < ntiles; ++k) {
      const uint32_t b = k & 1u, v = k >> 1;
      const size_t row = first + (size_t)(yb + k) * kChunks * a.W;
      // the mask's units are in flight while the tile's MMAs run
      uint4 mk[kChunks];
      if (a.mask && inside) {
#pragma unroll
        for (int c = 0; c < kChunks; ++c) mk[c] = a.mask[row + (size_t)c * a.W];
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[b], v & 1u, deadline))) {
        *s_err = 1;
        break;
      }
      tc_fence_after();
      uint32_t r[32];
      tmem_ld32(tmem_addr(tmem, 32 * q, b * kC), r);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[b]);
      if (inside) {
        uint4* dst = a.out + row;
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          uint32_t pk[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float lo = __uint_as_float(r[8 * c + 2 * e]) + s_bias[8 * c + 2 * e];
            float hi = __uint_as_float(r[8 * c + 2 * e + 1]) + s_bias[8 * c + 2 * e + 1];
            if (a.relu) {
              lo = lo > 0.f ? lo : 0.f;
              hi = hi > 0.f ? hi : 0.f;
            }
            pk[e] = bf16x2_rn(lo, hi);
          }
          if (a.mask) {
            // the data gradient: times ReLU'(Z) = [A > 0] of the layer's activation
            const uint32_t mw[4] = {mk[c].x, mk[c].y, mk[c].z, mk[c].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const bool plo = (int16_t)(mw[e] & 0xFFFFu) > 0, phi = (int16_t)(mw[e] >> 16) > 0;
              pk[e] &= (plo ? 0x0000FFFFu : 0u) | (phi ? 0xFFFF0000u : 0u);
            }
          }
          dst[(size_t)c * a.W] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
      }
    }
  }

  // every tensor-core operation of this CTA completes before its tensor
  // memory is freed (this wait keeps the full default budget)
  __syncthreads();
  if (warp == 0) {
    mma_commit_warp(drain);
    if (!mbar_wait(drain, 0, global_ns() + kDefaultWaitNs)) *s_err = 1;
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, kTmemColsTc);
  }
  if (threadIdx.x == 0 && *s_err && a.err) atomicMax(a.err, a.tag);
}

}  // namespace

cudaError_t launch_conv_tc(const uint4* in, uint32_t n, uint32_t H, uint32_t W, const uint16_t* wt,
                           const float* bias, int relu, uint4* out, unsigned int* err, unsigned int tag,
                           cudaStream_t s, const uint4* mask) {
  if (n == 0 || H == 0 || W == 0) return cudaSuccess;
  static PerDeviceOnce attr;
  cudaError_t e = attr.run([] {
    return cudaFuncSetAttribute(conv_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)TcSmemLayout::total);
  });
  if (e != cudaSuccess) return e;
  const uint32_t segs = (W + kSeg - 1) / kSeg;
  // images side by side: G W pixels and the G - 1 zeros between them in 128 lanes
  uint32_t group = std::min<uint32_t>(n, (kSeg + 1) / (W + 1));
  if (group < 1) group = 1;
  const uint32_t sets = (n + group - 1) / group;
  // about two CTAs per SM over the whole launch, at least 4 rows per band
  const uint64_t want = 2ull * (uint64_t)device_sm_count();
  uint64_t bands = want / ((uint64_t)segs * sets);
  if (bands < 1) bands = 1;
  uint32_t band = (uint32_t)((H + bands - 1) / bands);
  if (band < 4) band = 4;
  if (band > H) band = H;
  const dim3 grid(segs, (H + band - 1) / band, sets);
  TcArgs args{in, out, wt, bias, relu, n, H, W, band, group, pipeline_wait_ns(), pipeline_stall() ? 1u : 0u, err, tag,
              mask};
  conv_tc_kernel<<<grid, kThreadsTc, TcSmemLayout::total, s>>>(args);
  count_launch(kKernelLearned);
  return cudaGetLastError();
}

}  // namespace learned
}  // namespace ipb
