// tm_many.cu -- many templates of one size against one image on tcgen05.
//
// The reference scores one template per call (match_template,
// src/template_matching.rs:78-92). For a bank of templates the work becomes
// one GEMM per output column x:
//   D[m][t] = sum_{dy,dx} I[y0 + m + dy][x + dx] * T_t[dy][dx]
// over 128 consecutive output rows m, a block of templates t and
// K = the template's pixels in (dy, dx) order, 32 bytes per MMA step.
//
// Image operand: a "strip" of the image for column x -- for each 16-byte
// column chunk j, the rows y0 .. y0 + 127 + h - 1 of bytes [x + 16j,
// x + 16j + 16), stored 16 bytes per row in the canonical no-swizzle K-major
// layout. The operand for template row dy is the same strip started dy rows
// (16*dy bytes) later, so one strip (about 5 KB) serves all h template rows.
// Template operand: the template block, K-major, resident in shared memory
// for the CTA's lifetime.
//
// Two operand assignments:
//  * templates as M: A = up to 128 templates, B = the strip (N = 128
//    positions). Tensor-memory lanes are templates, so each epilogue store
//    instruction writes 32 consecutive templates of one position -- a full
//    128-byte line of the position-major output -- and every lane keeps its
//    template's extremes in registers. Used where the bank fits (see below).
//  * positions as M: A = the strip (M = 128 positions), B = NB templates
//    (a multiple of 16, at most 112), for larger templates.
//
// Roles (positions as M): all warps stage each image tile (cp.async) and
// compute the window sums Y = sum I^2 of its positions; then 2 builder warps
// build strips, one warp issues the MMAs (one flat loop, one elected lane) and
// 16 epilogue warps (four per tensor-memory lane quadrant) read the accumulator
// (double-buffered in tensor memory), apply the method, write the scores and
// fold them into per-template extremes. Scores are position-major:
// out[(y * Wo + x) * n_templates + t].
// Every wait is bounded (2 s) and reports through the error word.
#include <type_traits>

#include "tm_common.cuh"
#include "tm_internal.h"
#include "tm_sm100.cuh"

namespace ipb {
namespace {

using namespace sm100;

constexpr int kM = 128;           // output rows per tile
constexpr int kXT = 32;           // output columns per tile
constexpr int kVP = kXT + 1;      // pitch of the row sums: a thread per row, all rows on their own banks
constexpr int kBuildWarps = 2;
constexpr int kEpiWarps = 16;  // four per lane quadrant: the epilogue is the longest role
constexpr int kMmaWarp = kBuildWarps + kEpiWarps;
constexpr int kEpiPerQuad = kEpiWarps / 4;      // epilogue warps per tensor-memory lane quadrant
constexpr int kThreads = (kMmaWarp + 1) * 32;
constexpr int kStrips = 3;
constexpr uint32_t kTmemCols = 256;  // two accumulators of up to 128 columns
constexpr unsigned long long kWaitNs = kDefaultWaitNs;  // the final drain's budget

struct ManyParams {
  const uint8_t* img;
  uint32_t W, H;
  const uint8_t* tpl;  // n templates of w x h, contiguous
  uint32_t w, h, n;
  uint32_t kw;       // w rounded up to 32
  uint32_t NB;       // templates per block: 128 (templates as M) or a multiple of 16
  uint32_t nch, units, part, xt, img_bytes;  // templates as M: 16-byte chunks per row, units of K, units staged at
                                             // once, columns per tile, bytes of a staged image tile
  uint32_t nblocks;  // ceil(n / NB)
  uint32_t Wo, Ho, bands, xtiles, spatial;  // spatial tiles = bands * xtiles
  uint32_t rows;     // strip rows: 128 + h - 1
  uint32_t ip;       // staged image row pitch
  uint32_t b_off, tss_off, img_off, strip_off, y_off, v_off, ext_off, ry_off;
  int method, precision, vec4;  // vec4: 16-byte score stores (positions as M)
  int img16, img4;              // image rows 16-byte, 4-byte aligned: cp.async staging
  float* out;                 // may be null (extremes only)
  unsigned long long* ext;    // 2 keys per template or null
  unsigned int* err;
  unsigned int tag;
  unsigned long long wait_ns;  // budget of the bounded waits per tile (pipeline_wait_ns())
  uint32_t stall;              // pipeline_stall() at launch
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// n <= 16 bytes at g, zero past them, read as aligned words where those lie
// inside [p0, end).
__device__ __forceinline__ uint4 row_chunk(const uint8_t* g, uint32_t n, const uint8_t* p0, const uint8_t* end) {
  uint32_t v[4] = {0u, 0u, 0u, 0u};
  const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(g) & 3u);
  const uint8_t* a = g - off;
  if (a >= p0 && a + 20 <= end) {
    const uint32_t* a4 = reinterpret_cast<const uint32_t*>(a);
    uint32_t w[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) w[k] = __ldg(a4 + k);
    const uint32_t sel = 0x3210u + off * 0x1111u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = __byte_perm(w[k], w[k + 1], sel);
      if (n < 4u * k + 4u) v[k] = n <= 4u * k ? 0u : v[k] & ((1u << (8 * (n - 4 * k))) - 1u);
    }
  } else {
#pragma unroll
    for (uint32_t k = 0; k < 16; ++k)
      if (k < n) v[k >> 2] |= (uint32_t)__ldg(g + k) << (8 * (k & 3));
  }
  return make_uint4(v[0], v[1], v[2], v[3]);
}

// State of an epilogue warp for one tile.
struct EpiCtx {
  const ManyParams* p;
  uint32_t tmem;
  uint64_t* dfull;
  uint64_t* dempty;
  const uint32_t* s_y;
  const uint32_t* s_tss;
  unsigned long long* s_ext;
  uint32_t gx, nx, x0, y0, t0, nt;
  uint32_t e;  // epilogue warp index: lane quadrant (e + kBuildWarps) & 3, share e >> 2
  uint32_t lane;
  unsigned long long deadline;
};

// Drains the tile's accumulators with the method and precision fixed at
// compile time, so the 16 scores of a tensor-memory load are independent
// straight-line code. Returns false when a wait ran out.
template <int kMethod, int kPrec, bool kExt>
__device__ __forceinline__ bool epilogue(EpiCtx& c) {
  const ManyParams& p = *c.p;
  const uint32_t q = (c.e + kBuildWarps) & 3;  // = warp & 3, the lanes this warp may access
  // lanes are positions (rows); the quadrant's warps take the block's
  // 16-template chunks in turn
  const uint32_t m = q * 32 + c.lane, y = c.y0 + m;
  const bool row_ok = y < p.Ho;
  for (uint32_t xi = 0; xi < c.nx; ++xi) {
    const uint32_t g = c.gx + xi, d = g & 1u;
    if (!__all_sync(0xffffffffu, mbar_wait_sleep(&c.dfull[d], (g >> 1) & 1u, c.deadline))) return false;
    tc_fence_after();
    const uint32_t x = c.x0 + xi;
    const uint32_t Y = c.s_y[xi * kM + m];
    float* orow = p.out ? p.out + ((size_t)y * p.Wo + x) * p.n + c.t0 : nullptr;
    for (uint32_t cc = (c.e >> 2) * 16; cc < p.NB; cc += 16 * kEpiPerQuad) {
      uint32_t v[16];
      tmem_ld16(tmem_addr(c.tmem, q * 32, d * 128 + cc), v);
      tmem_wait_ld();
      float f[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) f[k] = finish_score32(kMethod, kPrec, v[k], Y, c.s_tss[cc + k]);
      if (orow && row_ok) {
        if (p.vec4 && cc + 16 <= c.nt) {
#pragma unroll
          for (int k = 0; k < 16; k += 4)
            *reinterpret_cast<float4*>(orow + cc + k) = make_float4(f[k], f[k + 1], f[k + 2], f[k + 3]);
        } else {
          for (int k = 0; k < 16; ++k)
            if (cc + k < c.nt) orow[cc + k] = f[k];
        }
      }
      if constexpr (kExt) {
        // per template: smallest / largest value over this warp's 32 rows,
        // the lowest row (= lowest linear index at this x) among ties;
        // lane k keeps template cc + k's result
        uint32_t my_mn = 0xFFFFFFFFu, my_ln = 0, my_mx = 0, my_lx = 0;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const uint32_t key = row_ok ? order_key(f[k]) : 0xFFFFFFFFu;
          const uint32_t kmn = __reduce_min_sync(0xffffffffu, key);
          const uint32_t ln = __ffs(__ballot_sync(0xffffffffu, key == kmn)) - 1;
          const uint32_t keyx = row_ok ? order_key(f[k]) : 0u;
          const uint32_t kmx = __reduce_max_sync(0xffffffffu, keyx);
          const uint32_t lx = __ffs(__ballot_sync(0xffffffffu, keyx == kmx)) - 1;
          if (c.lane == (uint32_t)k) {
            my_mn = kmn;
            my_ln = ln;
            my_mx = kmx;
            my_lx = lx;
          }
        }
        if (c.lane < 16 && cc + c.lane < c.nt) {
          const uint32_t ymn = c.y0 + q * 32 + my_ln, ymx = c.y0 + q * 32 + my_lx;
          if (ymn < p.Ho)
            atomicMin(&c.s_ext[2 * (cc + c.lane)], ((unsigned long long)my_mn << 32) | (ymn * p.Wo + x));
          if (ymx < p.Ho)
            atomicMax(&c.s_ext[2 * (cc + c.lane) + 1],
                      ((unsigned long long)my_mx << 32) | (0xFFFFFFFFu - (ymx * p.Wo + x)));
        }
      }
    }
    tc_fence_before();
    __syncwarp();
    if (c.lane == 0) mbar_arrive(&c.dempty[d]);
  }
  return true;
}

// One kernel per (method, precision, extremes): each gets its own register
// allocation for its epilogue. Precision only affects
// the normalised methods; the others use EXACT_FP64's instance.
template <int kMethod, int kPrec, bool kExt>
__global__ void __launch_bounds__(kThreads, 1) many_match_kernel(const __grid_constant__ ManyParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* sfull = reinterpret_cast<uint64_t*>(smem);   // [kStrips] strip built
  uint64_t* sempty = sfull + kStrips;                    // [kStrips] strip consumed by the MMAs
  uint64_t* dfull = sempty + kStrips;                    // [2] accumulator ready
  uint64_t* dempty = dfull + 2;                          // [2] accumulator drained
  uint64_t* drain = dempty + 2;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + 128);
  volatile int* s_err = reinterpret_cast<volatile int*>(smem + 132);
  uint8_t* bmat = smem + p.b_off;                        // templates, K-major chunks
  uint32_t* s_tss = reinterpret_cast<uint32_t*>(smem + p.tss_off);
  uint8_t* s_img = smem + p.img_off;
  uint8_t* s_strip = smem + p.strip_off;
  uint32_t* s_y = reinterpret_cast<uint32_t*>(smem + p.y_off);   // [kXT][kM]
  uint32_t* s_v = reinterpret_cast<uint32_t*>(smem + p.v_off);   // [rows][kXT]
  unsigned long long* s_ext = reinterpret_cast<unsigned long long*>(smem + p.ext_off);  // [NB][2]

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t nch = p.kw / 16;
  const uint32_t strip_bytes = nch * p.rows * 16;
  const uint32_t tb = blockIdx.x % p.nblocks;              // this CTA's template block
  const uint32_t t0 = tb * p.NB;
  const uint32_t nt = min(p.NB, p.n - t0);                 // templates in the block

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStrips; ++s) {
      mbar_init(&sfull[s], kBuildWarps);  // one arrive per builder warp
      mbar_init(&sempty[s], 1);
    }
    for (int d = 0; d < 2; ++d) {
      mbar_init(&dfull[d], 1);
      mbar_init(&dempty[d], kEpiWarps);   // one arrive per epilogue warp
    }
    mbar_init(drain, 1);
    *s_err = 0;
    mbar_init_fence();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(s_tmem, kTmemCols);
    tmem_relinquish();
  }
  // template block: chunk (dy, j) holds NB rows of 16 bytes (template t's
  // bytes [16j, 16j+16) of row dy; zero past w and for absent templates).
  // Eight templates and four chunks per warp: 64 neighbouring bytes of each
  // are read and 128 of each chunk written. (Byte by byte, a lane per
  // template, the block of 128 32 x 32 templates took 65 us longer.)
  {
    const uint32_t chunks = p.h * nch, c4 = (chunks + 3) / 4, items = c4 * (p.NB / 8);
    const uint8_t* end = p.tpl + (size_t)p.n * p.w * p.h;
    for (uint32_t i = warp; i < items; i += kThreads / 32) {
      const uint32_t c = 4 * (i % c4) + (lane >> 3), t = 8 * (i / c4) + (lane & 7);
      if (c >= chunks) continue;
      const uint32_t dy = c / nch, x = 16 * (c % nch);
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (t < nt && x < p.w) v = row_chunk(p.tpl + ((size_t)(t0 + t) * p.h + dy) * p.w + x, min(16u, p.w - x), p.tpl, end);
      *reinterpret_cast<uint4*>(bmat + (size_t)c * p.NB * 16 + t * 16) = v;
    }
  }
  for (uint32_t t = threadIdx.x; t < p.NB; t += kThreads) s_tss[t] = 0u;
  __syncthreads();
  // template constants TSS_t = sum T_t^2 (< 2^32 for templates up to 64 x 64)
  // from the block, its chunks shared out over four threads per template
  for (uint32_t i = threadIdx.x; i < 4 * p.NB; i += kThreads) {
    const uint32_t t = i % p.NB;
    uint32_t s = 0;
    for (uint32_t c = i / p.NB; c < p.h * nch; c += 4) {
      const uint4 v = *reinterpret_cast<const uint4*>(bmat + (size_t)c * p.NB * 16 + t * 16);
      s = __dp4a(v.x, v.x, __dp4a(v.y, v.y, __dp4a(v.z, v.z, __dp4a(v.w, v.w, s))));
    }
    atomicAdd(&s_tss[t], s);
  }
  for (uint32_t i = threadIdx.x; i < 2 * p.NB; i += kThreads) s_ext[i] = (i & 1) ? 0ull : ~0ull;
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  const uint32_t idesc = idesc_u8u8_s32(kM, p.NB);
  constexpr bool do_ext = kExt;

  uint32_t gx = 0;  // strips built / consumed so far (global x counter, same in all roles)
  bool ok = true;
  const uint32_t cta_in_block = blockIdx.x / p.nblocks;
  const uint32_t ctas_per_block = gridDim.x / p.nblocks;

  for (uint32_t sp = cta_in_block; sp < p.spatial; sp += ctas_per_block) {
    __syncthreads();
    if (*s_err) break;
    const uint32_t y0 = (sp / p.xtiles) * kM, x0 = (sp % p.xtiles) * kXT;
    const uint32_t nrows = min(p.rows, p.H - y0);
    const uint32_t nx = min((uint32_t)kXT, p.Wo - x0);
    // stage the tile's image rows (all threads), zero past the right edge
    {
      const uint32_t chunks = p.ip / 16;
      const uint8_t* src = p.img + (size_t)y0 * p.W;
      for (uint32_t idx = threadIdx.x; idx < nrows * chunks; idx += kThreads) {
        const uint32_t r = idx / chunks, c = (idx % chunks) * 16, gxx = x0 + c;
        uint8_t* dst = s_img + r * p.ip + c;
        if (p.img16 && gxx + 16 <= p.W) {
          cp_async16(smem_u32(dst), src + (size_t)r * p.W + gxx, 16);
        } else {
          uint32_t wd[4] = {0u, 0u, 0u, 0u};
          for (int k = 0; k < 16; ++k)
            if (gxx + k < p.W) wd[k >> 2] |= (uint32_t)__ldg(src + (size_t)r * p.W + gxx + k) << (8 * (k & 3));
          *reinterpret_cast<uint4*>(dst) = make_uint4(wd[0], wd[1], wd[2], wd[3]);
        }
      }
      cp_async_commit();
      cp_async_wait_all();
    }
    __syncthreads();
    // window sums of I^2 for the tile's positions: V = row sums over w, then Y over h
    for (uint32_t r = threadIdx.x; r < nrows; r += kThreads) {
      const uint8_t* row = s_img + r * p.ip;
      uint32_t s = 0;
      for (uint32_t dx = 0; dx < p.w; ++dx) s += (uint32_t)row[dx] * row[dx];
      for (uint32_t xi = 0; xi < (uint32_t)kXT; ++xi) {
        s_v[r * kVP + xi] = s;
        const uint32_t a = row[xi + p.w], b = row[xi];
        s += a * a - b * b;
      }
    }
    __syncthreads();
    for (uint32_t idx = threadIdx.x; idx < (uint32_t)kXT * (kM / 32); idx += kThreads) {
      const uint32_t xi = idx % kXT, m0 = (idx / kXT) * 32;
      uint32_t s = 0;
      for (uint32_t dy = 0; dy < p.h; ++dy) s += (m0 + dy < nrows) ? s_v[(m0 + dy) * kVP + xi] : 0u;
      for (uint32_t m = m0; m < m0 + 32; ++m) {
        s_y[xi * kM + m] = s;
        const uint32_t a = (m + p.h < nrows) ? s_v[(m + p.h) * kVP + xi] : 0u;
        const uint32_t b = (m < nrows) ? s_v[m * kVP + xi] : 0u;
        s += a - b;
      }
    }
    __syncthreads();
    const unsigned long long deadline = global_ns() + p.wait_ns;

    if (warp < kBuildWarps) {
      // strips: S_x[j][rho] = image row rho, bytes [xi + 16j, xi + 16j + 16)
      for (uint32_t xi = 0; xi < nx; ++xi) {
        const uint32_t g = gx + xi, s = g % kStrips;
        const bool got = g < kStrips || mbar_wait_sleep(&sempty[s], ((g / kStrips) + 1) & 1u, deadline);
        if (!__all_sync(0xffffffffu, got)) {  // warp-uniform: the warp arrives as one below
          ok = false;
          break;
        }
        uint8_t* strip = s_strip + s * strip_bytes;
        const uint32_t sel = 0x3210u + (xi & 3u) * 0x1111u;
        for (uint32_t idx = threadIdx.x; idx < nch * nrows; idx += kBuildWarps * 32) {
          const uint32_t j = idx / nrows, r = idx % nrows;
          const uint32_t* wp = reinterpret_cast<const uint32_t*>(s_img + r * p.ip) + (xi >> 2) + 4 * j;
          const uint32_t w0 = wp[0], w1 = wp[1], w2 = wp[2], w3 = wp[3], w4 = wp[4];
          *reinterpret_cast<uint4*>(strip + (j * p.rows + r) * 16) =
              make_uint4(__byte_perm(w0, w1, sel), __byte_perm(w1, w2, sel), __byte_perm(w2, w3, sel),
                         __byte_perm(w3, w4, sel));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sfull[s]);
      }
      if (!ok) {
        *s_err = 1;
        atomicMax(p.err, p.tag);
      }
    } else if (warp == kMmaWarp) {
      // warp-uniform issue loop: descriptors advance by adding to their
      // 16-byte-unit start-address field (shared addresses stay below 2^18)
      const uint32_t lbo_s = p.rows * 16, lbo_t = p.NB * 16;
      const uint32_t sstep = lbo_s >> 4, tstep = lbo_t >> 4;
      const uint64_t tdesc0 = smem_desc_noswizzle(smem_u32(bmat), lbo_t, 128);
      const uint32_t nk = p.kw / 32;
      // test hook: a wait on the drain barrier, which nothing arrives at before the end
      if (p.stall && !__all_sync(0xffffffffu, mbar_wait(drain, 0, deadline))) ok = false;
      for (uint32_t xi = 0; ok && xi < nx; ++xi) {
        const uint32_t g = gx + xi, s = g % kStrips, d = g & 1u;
        const bool got_s = mbar_wait(&sfull[s], (g / kStrips) & 1u, deadline);
        const bool got_d = got_s && (g < 2 || mbar_wait(&dempty[d], ((g >> 1) + 1) & 1u, deadline));
        if (!__all_sync(0xffffffffu, got_s && got_d)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t dt = tmem + d * 128;
        // one flat loop over template rows with running descriptors: the
        // strip advances one 16-byte row per template row, the template block
        // one row of nch chunks (a nested loop with computed descriptors
        // issued at under half the tensor pipe's rate)
        uint64_t sd = smem_desc_noswizzle(smem_u32(s_strip + s * strip_bytes), lbo_s, 128);
        uint64_t td = tdesc0;
        const uint64_t tdy = (uint64_t)(nch * tstep);
        auto mma = [&](uint64_t tdk, uint64_t sdk, uint32_t acc) { mma_i8_ss_warp(dt, sdk, tdk, idesc, acc); };
        if (nk == 1) {
          for (uint32_t dy = 0; dy < p.h; ++dy, sd += 1, td += tdy) mma(td, sd, dy != 0);
        } else {  // two 32-byte K steps per template row (w in 33..64)
          for (uint32_t dy = 0; dy < p.h; ++dy, sd += 1, td += tdy) {
            mma(td, sd, dy != 0);
            mma(td + 2 * tstep, sd + 2 * sstep, 1u);
          }
        }
        mma_commit_warp(&sempty[s]);
        mma_commit_warp(&dfull[d]);
      }
      if (!ok && lane == 0) {
        *s_err = 1;
        atomicMax(p.err, p.tag);
      }
    } else {
      EpiCtx c{&p, tmem, dfull, dempty, s_y, s_tss, s_ext, gx, nx, x0, y0, t0, nt,
               (uint32_t)(warp - kBuildWarps), (uint32_t)lane, deadline};
      ok = epilogue<kMethod, kPrec, kExt>(c);
      if (!ok) {
        *s_err = 1;
        atomicMax(p.err, p.tag);
      }
    }
    gx += nx;
  }

  __syncthreads();
  if (do_ext)
    for (uint32_t t = threadIdx.x; t < nt; t += kThreads) {
      atomicMin(&p.ext[2 * (t0 + t)], s_ext[2 * t]);
      atomicMax(&p.ext[2 * (t0 + t) + 1], s_ext[2 * t + 1]);
    }
  if (warp == kMmaWarp) {
    mma_commit_warp(drain);
    if (!mbar_wait(drain, 0, global_ns() + kWaitNs) && lane == 0) atomicMax(p.err, p.tag);
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// ---- templates as M -----------------------------------------------------------
//
// Up to 128 templates are the MMA's M side for every strip of the CTA, so the
// bank is laid out once: the K bytes of every template, 32 to a unit, the first
// 32 units in tensor memory (A operands of eight columns each, beside two
// accumulators of 128), the others in shared memory. A unit is two 16-byte
// chunks of template rows: neighbours in a row, or, of an odd number of chunks
// per row, the last ones of two rows (so 48 pixels are 48 bytes of K, not 64);
// the strip's descriptor takes their distance as its leading offset.
//
// Bounds (128 templates of 32 x 32 on 2048 x 2048, CrossCorrelationNormalized):
// the 2.1 GB of scores take 320 us at the copy rate and the MMAs, 32 of 64
// cycles per strip, 237 us. Double arithmetic and the MMAs hold each other up:
// a strip's 128 reciprocal roots take a builder warp 900 cycles with the
// tensor pipe idle and 3600 beside its MMAs, and each template row adds its
// MMAs' whole time to a normalised launch (8 us) where it adds a third of it
// to an unnormalised one of the same length. So a score takes two double
// operations and a conversion, and accumulators are emptied into registers at
// once, so that the next MMAs run beside the stores and folds, which use
// neither. Measured: 631 us, CrossCorrelation 440 (with A in shared memory, an
// epilogue in one pass per 16 positions and a CTA-wide phase per tile: 1020
// and 570).
//
// Roles (20 warps): three builder warps stage the next image tile while they
// build the strips of this one, a strip each, with the window sums of its
// positions and their reciprocal roots, into a ring of six; one warp issues
// the MMAs; sixteen epilogue warps (four per tensor-memory lane quadrant, 32
// positions each) score, store and fold extremes. Nothing waits for a whole
// tile. (24 epilogue warps of 16 positions: 840 against 780 us; the epilogue
// warps in two groups on alternate strips: 657 against 631.)
constexpr int kBankBuild = 3, kBankEpi = 16, kBankMma = kBankBuild + kBankEpi;
constexpr int kBankThreads = (kBankMma + 1) * 32;
constexpr int kBankStrips = 6;
static_assert(kBankStrips % kBankBuild == 0, "one builder waits for every use of a ring slot, in turn");
constexpr uint32_t kTmemUnits = 32, kUnitBytes = 4096;  // 128 templates x 32 bytes
constexpr int kYP = kM + 1;                             // pitch of the window sums: a lane per column, no conflicts
constexpr uint32_t kNormBytes = 12 * kM;                // a strip's reciprocal roots (f64) and window sums (u32)

struct BankShared {
  uint64_t sfull[kBankStrips], sempty[kBankStrips];  // strip built; read by the MMAs and its norms by the epilogue
  uint64_t dfull[2], dempty[2];                      // accumulator ready; drained
  uint64_t drain;
  uint32_t tmem;
  uint32_t zero[kBankStrips][4];  // whether any of a strip's 32 positions has a window of zeros
};

// The chunks (template row, 16-byte column) of unit u; `second` is false where
// the last row of an odd number has no partner.
struct UnitChunks {
  uint32_t dy0, j0, dy1, j1;
  bool second;
};
__host__ __device__ inline uint32_t unit_count(uint32_t nch, uint32_t h) {
  return (nch & 1u) ? (h / 2) * nch + (h & 1u) * ((nch + 1) / 2) : h * (nch / 2);
}
__device__ __forceinline__ UnitChunks unit_chunks(uint32_t u, uint32_t nch, uint32_t h) {
  if (!(nch & 1u)) {
    const uint32_t per = nch / 2, dy = u / per, j = 2 * (u % per);
    return {dy, j, dy, j + 1, true};
  }
  const uint32_t dy = 2 * (u / nch), k = u % nch, m = (nch - 1) / 2;
  const bool pair = dy + 1 < h;
  if (k < m) return {dy, 2 * k, dy, 2 * k + 1, true};
  if (pair && k < 2 * m) return {dy + 1, 2 * (k - m), dy + 1, 2 * (k - m) + 1, true};
  return {dy, nch - 1, dy + 1, nch - 1, pair};
}

// Units [ua, ub) of the block's templates to dst (per unit two halves of 128
// 16-byte rows), by all threads: eight templates and two units per warp.
__device__ __forceinline__ void stage_units(const ManyParams& p, uint32_t t0, uint32_t nt, uint32_t ua, uint32_t ub,
                                            uint8_t* dst, uint32_t warp, uint32_t lane) {
  const uint8_t* end = p.tpl + (size_t)p.n * p.w * p.h;
  const uint32_t items = ((ub - ua + 1) / 2) * 16;
  for (uint32_t i = warp; i < items; i += kBankThreads / 32) {
    const uint32_t u = ua + 2 * (i / 16) + (lane >> 4), half = (lane >> 3) & 1u, t = 8 * (i & 15u) + (lane & 7u);
    if (u >= ub) continue;
    const UnitChunks c = unit_chunks(u, p.nch, p.h);
    const uint32_t dy = half ? c.dy1 : c.dy0, x = 16 * (half ? c.j1 : c.j0);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (t < nt && x < p.w && (!half || c.second))
      v = row_chunk(p.tpl + ((size_t)(t0 + t) * p.h + dy) * p.w + x, min(16u, p.w - x), p.tpl, end);
    *reinterpret_cast<uint4*>(dst + (u - ua) * kUnitBytes + half * 2048 + t * 16) = v;
  }
}

// Adds the units' share of TSS_t = sum T_t^2 (< 2^32), four threads per template.
__device__ __forceinline__ void add_tss(const uint8_t* units, uint32_t n, uint32_t* s_tss) {
  for (uint32_t i = threadIdx.x; i < 4 * kM; i += kBankThreads) {
    const uint32_t t = i % kM;
    uint32_t s = 0;
    for (uint32_t c = i / kM; c < 2 * n; c += 4) {
      const uint4 v = *reinterpret_cast<const uint4*>(units + c * 2048 + t * 16);
      s = __dp4a(v.x, v.x, __dp4a(v.y, v.y, __dp4a(v.z, v.z, __dp4a(v.w, v.w, s))));
    }
    atomicAdd(&s_tss[t], s);
  }
}

// The image rows of the tile at (x0, y0), zero past the right edge, by the
// builder warps: asynchronously by 16 bytes where the addresses are multiples
// of 16 (a tile's left edge is one of xt only), by words where rows and edge
// are word-aligned, else through registers.
__device__ __forceinline__ void stage_image(const ManyParams& p, uint32_t x0, uint32_t y0, uint8_t* dst, uint32_t t) {
  const uint32_t nrows = min(p.rows, p.H - y0);
  const uint8_t *src = p.img + (size_t)y0 * p.W, *end = p.img + (size_t)p.W * p.H;
  if (p.img4 && ((x0 & 15u) || !p.img16)) {
    const uint32_t words = p.ip / 4;
    for (uint32_t i = t; i < nrows * words; i += kBankBuild * 32) {
      const uint32_t r = i / words, c = (i - r * words) * 4, gx = x0 + c;
      if (gx < p.W) cp_async4(smem_u32(dst + r * p.ip + c), src + (size_t)r * p.W + gx);
      else *reinterpret_cast<uint32_t*>(dst + r * p.ip + c) = 0u;
    }
  } else {
    const uint32_t chunks = p.ip / 16;
    for (uint32_t i = t; i < nrows * chunks; i += kBankBuild * 32) {
      const uint32_t r = i / chunks, c = (i - r * chunks) * 16, gx = x0 + c;
      uint8_t* d = dst + r * p.ip + c;
      const uint8_t* g = src + (size_t)r * p.W + gx;
      if (p.img16 && gx < p.W)  // W and gx are multiples of 16: the chunk is whole
        cp_async16(smem_u32(d), g, 16);
      else
        *reinterpret_cast<uint4*>(d) =
            gx < p.W ? row_chunk(g, min(16u, p.W - gx), p.img, end) : make_uint4(0u, 0u, 0u, 0u);
    }
  }
  cp_async_commit();
}

// Window sums Y = sum I^2 of the tile's 32 columns x 128 rows: sums over w
// along each row, then over h down each column, both slid.
__device__ __forceinline__ void row_sums(const ManyParams& p, const uint8_t* img, uint32_t nrows, uint32_t* s_v,
                                         uint32_t t) {
  const uint32_t w4 = p.w >> 2, sel = 0x3210u + (p.w & 3u) * 0x1111u;
  for (uint32_t r = t; r < nrows; r += kBankBuild * 32) {
    const uint32_t* row = reinterpret_cast<const uint32_t*>(img + r * p.ip);
    uint32_t s = 0, lead = row[w4];
    for (uint32_t i = 0; i < w4; ++i) s = __dp4a(row[i], row[i], s);
    const uint32_t rest = lead & ((1u << (8 * (p.w & 3u))) - 1u);
    s = __dp4a(rest, rest, s);
#pragma unroll
    for (uint32_t xq = 0; xq < kXT / 4; ++xq) {
      const uint32_t next = row[w4 + xq + 1], a = __byte_perm(lead, next, sel), b = row[xq];
      lead = next;
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        s_v[r * kVP + 4 * xq + k] = s;
        const uint32_t ak = (a >> (8 * k)) & 255u, bk = (b >> (8 * k)) & 255u;
        s += ak * ak - bk * bk;
      }
    }
  }
}
__device__ __forceinline__ void column_sums(const ManyParams& p, const uint32_t* s_v, uint32_t nrows, uint32_t* s_y,
                                            uint32_t t) {
  const uint32_t xi = t & 31u;
  const uint32_t* v = s_v + xi;
  for (uint32_t m0 = (t >> 5) * 32; m0 < (uint32_t)kM; m0 += 32 * kBankBuild) {
    uint32_t s = 0;
#pragma unroll 8
    for (uint32_t r = m0; r < min(m0 + p.h, nrows); ++r) s += v[r * kVP];
#pragma unroll 8
    for (uint32_t m = m0; m < m0 + 32; ++m) {
      s_y[xi * kYP + m] = s;
      s += (m + p.h < nrows ? v[(m + p.h) * kVP] : 0u) - (m < nrows ? v[m * kVP] : 0u);
    }
  }
}

// The strip of column xi: strip[j][r] = image row r, bytes [xi + 16j, xi + 16j
// + 16), by one warp. A lane reads whole 16-byte words of its row (rows an odd
// number of them apart: no bank conflicts; word by word, four lanes shared a
// bank and the builders were the slowest role) and picks its bytes from two.
template <uint32_t kWord>
__device__ __forceinline__ void build_rows(const ManyParams& p, const uint8_t* img, uint32_t sel, uint32_t nrows,
                                           uint8_t* strip, uint32_t lane) {
#pragma unroll 2
  for (uint32_t r = lane; r < nrows; r += 32) {
    const uint4* src = reinterpret_cast<const uint4*>(img + r * p.ip);
    uint4 a = src[0];
    for (uint32_t j = 0; j < p.nch; ++j) {
      const uint4 b = src[j + 1];
      const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      *reinterpret_cast<uint4*>(strip + (j * p.rows + r) * 16) =
          make_uint4(__byte_perm(w[kWord], w[kWord + 1], sel), __byte_perm(w[kWord + 1], w[kWord + 2], sel),
                     __byte_perm(w[kWord + 2], w[kWord + 3], sel), __byte_perm(w[kWord + 3], w[kWord + 4], sel));
      a = b;
    }
  }
}
__device__ __forceinline__ void build_strip(const ManyParams& p, const uint8_t* img, uint32_t xi, uint32_t nrows,
                                            uint8_t* strip, uint32_t lane) {
  const uint8_t* src = img + (xi & ~15u);
  const uint32_t sel = 0x3210u + (xi & 3u) * 0x1111u;
  switch ((xi >> 2) & 3u) {
    case 0: build_rows<0>(p, src, sel, nrows, strip, lane); break;
    case 1: build_rows<1>(p, src, sel, nrows, strip, lane); break;
    case 2: build_rows<2>(p, src, sel, nrows, strip, lane); break;
    default: build_rows<3>(p, src, sel, nrows, strip, lane); break;
  }
}

// An epilogue warp's lanes: templates t_first + lane. kmin, kmax: the lane's
// running extremes keys.
struct BankLane {
  uint32_t lane, tss, t_first;
  bool t_ok, general;  // a template of the bank; all zeros
  double rT, ncT;      // the template's reciprocal root, -2^52 times it
  unsigned long long kmin, kmax;
};

// The f32 bits of 32 positions' scores: sums at taddr, reciprocal roots and
// window sums at r_pos and y_pos.
//
// Normalised FP64: the quotient's estimate is a = RN(RN(s r_T) r_Y), the first
// product one fused multiply-add, fma(2^52 + s, r_T, -2^52 r_T): two
// roundings, as in norm_quotient_fp64_w's s w, so its bound (fewer than 2^5
// units of a's last place) and norm_bits_fp64_fast's window of 2^8 hold. a
// rounds to f32 on the conversion unit, which leaves the integer unit to the
// folds; `near` keeps the least distance of the dropped bits from 256 units
// below their midpoint: under 512 units some quotient is undecided.
template <int kMethod, int kPrec>
__device__ __forceinline__ void bank_scores(const BankLane& c, uint32_t taddr, const double* r_pos,
                                            const uint32_t* y_pos, bool zeros, uint32_t (&b)[32]) {
  constexpr bool kNormW = method_is_norm(kMethod) && kPrec == IPB_PRECISION_EXACT_FP64;
  constexpr bool kNeedY = kMethod != kCcorr && !(kNormW && !method_is_sse(kMethod));
  auto score_of = [&](uint32_t v, uint32_t yk) -> uint32_t {
    return method_is_sse(kMethod) ? (yk + c.tss - 2u * v) : v;
  };
  uint32_t near = 0xFFFFFFFFu;
  tmem_ld32(taddr, b);
  tmem_wait_ld();
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    uint32_t Y[4] = {0u, 0u, 0u, 0u};
    if constexpr (kNeedY) {
      const uint4 y4 = *reinterpret_cast<const uint4*>(y_pos + k);
      Y[0] = y4.x;
      Y[1] = y4.y;
      Y[2] = y4.z;
      Y[3] = y4.w;
    }
    if constexpr (kNormW) {
#pragma unroll
      for (int u = 0; u < 4; u += 2) {
        const double2 r = *reinterpret_cast<const double2*>(r_pos + k + u);
        const double a0 = __dmul_rn(
            __fma_rn(__hiloint2double(0x43300000, (int)score_of(b[k + u], Y[u])), c.rT, c.ncT), r.x);
        const double a1 = __dmul_rn(
            __fma_rn(__hiloint2double(0x43300000, (int)score_of(b[k + u + 1], Y[u + 1])), c.rT, c.ncT), r.y);
        near = min(near, min((uint32_t)__double2loint(a0) * 8u + 0x80000800u,
                             (uint32_t)__double2loint(a1) * 8u + 0x80000800u));
        b[k + u] = __float_as_uint(__double2float_rn(a0));
        b[k + u + 1] = __float_as_uint(__double2float_rn(a1));
      }
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        b[k + u] = __float_as_uint(finish_score32(kMethod, kPrec, b[k + u], Y[u], c.tss));
    }
  }
  // Rare and warp-uniform: with a flagged or zero-norm quotient (a window of
  // zeros, or a template all zeros) the sums are read again and the flagged
  // values go through the general quotient.
  if constexpr (kNormW) {
    const bool general = zeros || c.general;
    if (__any_sync(0xffffffffu, general || near < 0x1000u)) {
#pragma unroll
      for (int h = 0; h < 32; h += 8) {
        uint32_t v[8];
        tmem_ld8(taddr + h, v);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t yk = y_pos[h + k], sk = score_of(v[k], yk);
          const double w = __dmul_rn(r_pos[h + k], c.rT);
          bool u = general;
          if (!general) norm_bits_fp64_fast(sk, w, u);
          if (u) b[h + k] = __float_as_uint(norm_quotient_fp64_w(sk, w, yk, c.tss));
        }
      }
    }
  }
}

// Stores the first nv (at most 32) of the scores, rows y .. of column x, and
// folds them into the lane's extremes (scores are never negative, so their f32
// bits order like the values).
template <bool kExt, bool kFull>
__device__ __forceinline__ void bank_store(const ManyParams& p, BankLane& c, uint32_t x, uint32_t y, int nv,
                                           const uint32_t (&b)[32]) {
  if (p.out && c.t_ok) {
    const size_t rstride = (size_t)p.Wo * p.n;
    float* o = p.out + ((size_t)y * p.Wo + x) * p.n + c.t_first + c.lane;
#pragma unroll
    for (int k = 0; k < 32; ++k)
      if (kFull || k < nv) o[k * rstride] = __uint_as_float(b[k]);
  }
  if constexpr (kExt) {
    uint32_t mn = 0xFFFFFFFFu, mx = 0u;
#pragma unroll
    for (int k = 0; k < 32; k += 2)
      if (kFull || k + 1 < nv) {
        mn = min(mn, min(b[k], b[k + 1]));
        mx = max(mx, max(b[k], b[k + 1]));
      } else if (k < nv) {
        mn = min(mn, b[k]);
        mx = max(mx, b[k]);
      }
    // they reach the lane's running keys only when the key with the first
    // index does (the positions are rows of one column: the lowest k is the
    // lowest index); then the first occurrence is found in this lane alone
    const uint32_t idx0 = y * p.Wo + x;
    const unsigned long long lo = ((unsigned long long)(mn | 0x80000000u) << 32) | idx0;
    const unsigned long long hi = ((unsigned long long)(mx | 0x80000000u) << 32) | (0xFFFFFFFFu - idx0);
    if (c.t_ok && lo < c.kmin) {
      uint32_t j = 0;
#pragma unroll
      for (int k = 31; k >= 0; --k)
        if ((kFull || k < nv) && b[k] == mn) j = k;
      c.kmin = min(c.kmin, lo + j * p.Wo);
    }
    if (c.t_ok && hi > c.kmax) {
      uint32_t j = 0;
#pragma unroll
      for (int k = 31; k >= 0; --k)
        if ((kFull || k < nv) && b[k] == mx) j = k;
      c.kmax = max(c.kmax, hi - j * p.Wo);
    }
  }
}

template <int kMethod, int kPrec, bool kExt>
__global__ void __launch_bounds__(kBankThreads, 1) many_bank_kernel(const __grid_constant__ ManyParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  BankShared* sh = reinterpret_cast<BankShared*>(smem);
  uint32_t* s_unit = reinterpret_cast<uint32_t*>(smem + p.ext_off);  // per unit: strip offset, leading offset
  uint32_t* s_tss = reinterpret_cast<uint32_t*>(smem + p.tss_off);
  uint8_t* s_norm = smem + p.ry_off;   // [kBankStrips] reciprocal roots, window sums
  uint8_t* s_bank = smem + p.b_off;    // units past the first 32
  uint8_t* s_strip = smem + p.strip_off;
  uint8_t* s_img = smem + p.img_off;   // two tiles
  uint32_t* s_y = reinterpret_cast<uint32_t*>(smem + p.y_off);  // [kXT][kYP]
  uint32_t* s_v = reinterpret_cast<uint32_t*>(smem + p.v_off);  // [rows][kVP]
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t strip_bytes = p.nch * p.rows * 16;
  const uint32_t t0 = (blockIdx.x % p.nblocks) * kM, nt = min((uint32_t)kM, p.n - t0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kBankStrips; ++s) {
      mbar_init(&sh->sfull[s], 1);
      mbar_init(&sh->sempty[s], 1 + kBankEpi);
    }
    for (int d = 0; d < 2; ++d) {
      mbar_init(&sh->dfull[d], 1);
      mbar_init(&sh->dempty[d], kBankEpi);
    }
    mbar_init(&sh->drain, 1);
    mbar_init_fence();
  }
  if (warp == kBankMma) {
    tmem_alloc(&sh->tmem, 512);
    tmem_relinquish();
  }
  for (uint32_t t = threadIdx.x; t < (uint32_t)kM; t += kBankThreads) s_tss[t] = 0u;
  for (uint32_t u = threadIdx.x; u < ((p.units + 3u) & ~3u); u += kBankThreads) {
    const UnitChunks c = unit_chunks(min(u, p.units - 1), p.nch, p.h);
    const uint32_t at = c.j0 * p.rows + c.dy0;
    s_unit[u] = at | ((c.j1 * p.rows + c.dy1 - at) << 16);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem;

  // ---- the bank: shared-memory units in place, the others through the room
  // of the strips, images and sums, a part at a time
  const uint32_t in_tmem = min(p.units, kTmemUnits);
  if (p.units > in_tmem) stage_units(p, t0, nt, in_tmem, p.units, s_bank, warp, lane);
  for (uint32_t ua = 0; ua < in_tmem; ua += p.part) {
    const uint32_t ub = min(ua + p.part, in_tmem);
    stage_units(p, t0, nt, ua, ub, s_strip, warp, lane);
    __syncthreads();
    if (ua == 0 && p.units > in_tmem) add_tss(s_bank, p.units - in_tmem, s_tss);
    add_tss(s_strip, ub - ua, s_tss);
    if (warp >= kBankBuild && warp < kBankMma) {
      const uint32_t q = warp & 3u, t = q * 32 + lane;
      for (uint32_t u = ua + ((warp - kBankBuild) >> 2); u < ub; u += kBankEpi / 4) {
        const uint4 lo = *reinterpret_cast<const uint4*>(s_strip + (u - ua) * kUnitBytes + t * 16);
        const uint4 hi = *reinterpret_cast<const uint4*>(s_strip + (u - ua) * kUnitBytes + 2048 + t * 16);
        const uint32_t v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        tmem_st8(tmem_addr(tmem, q * 32, 256 + 8 * u), v);
      }
      tmem_wait_st();
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }

  const uint32_t first = blockIdx.x / p.nblocks, step = gridDim.x / p.nblocks;
  bool fail = false;
  if (warp < kBankBuild) {
    // ---- builders
    const uint32_t t = threadIdx.x;
    uint32_t g = 0;
    stage_image(p, (first % p.xtiles) * p.xt, (first / p.xtiles) * kM, s_img, t);
    for (uint32_t sp = first, k = 0; sp < p.spatial; sp += step, ++k) {
      const unsigned long long deadline = global_ns() + p.wait_ns;
      const uint32_t x0 = (sp % p.xtiles) * p.xt, y0 = (sp / p.xtiles) * kM;
      const uint32_t nrows = min(p.rows, p.H - y0), nx = min(p.xt, p.Wo - x0);
      const uint8_t* img = s_img + (k & 1u) * p.img_bytes;
      cp_async_wait_all();
      // this tile's image is staged and the last tile's is read
      if (bar_or<kBankBuild * 32>(1, fail)) {
        fail = true;
        break;
      }
      if (sp + step < p.spatial)
        stage_image(p, ((sp + step) % p.xtiles) * p.xt, ((sp + step) / p.xtiles) * kM,
                    s_img + ((k + 1) & 1u) * p.img_bytes, t);
      row_sums(p, img, nrows, s_v, t);
      bar_or<kBankBuild * 32>(1, false);
      column_sums(p, s_v, nrows, s_y, t);
      bar_or<kBankBuild * 32>(1, false);
      // the warps take the strips in turn
      for (uint32_t xi = (warp + kBankBuild - g % kBankBuild) % kBankBuild; xi < nx; xi += kBankBuild) {
        const uint32_t gs = g + xi, s = gs % kBankStrips;
        bool got = true;
        if (gs >= (uint32_t)kBankStrips)
          got = mbar_wait_sleep(&sh->sempty[s], (gs / kBankStrips + 1) & 1u, deadline);
        fail |= !__all_sync(0xffffffffu, got);  // the role ends at the next tile's barrier
        build_strip(p, img, xi, nrows, s_strip + s * strip_bytes, lane);
        if constexpr (kMethod != kCcorr) {
#pragma unroll
          for (uint32_t m0 = 0; m0 < (uint32_t)kM; m0 += 32) {
            const uint32_t m = m0 + lane, yv = y0 + m < p.Ho ? s_y[xi * kYP + m] : 1u;
            reinterpret_cast<uint32_t*>(s_norm + s * kNormBytes + 8 * kM)[m] = yv;
            if constexpr (method_is_norm(kMethod) && kPrec == IPB_PRECISION_EXACT_FP64) {
              reinterpret_cast<double*>(s_norm + s * kNormBytes)[m] = yv ? rsqrt_u32(yv) : 0.0;
              const bool any = __any_sync(0xffffffffu, yv == 0u);
              if (lane == 0) sh->zero[s][m0 >> 5] = any;
            }
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->sfull[s]);
      }
      g += nx;
    }
    cp_async_wait_all();
  } else if (warp == kBankMma) {
    // ---- MMA issue
    const bool leader = elect_one();
    const uint32_t idesc = idesc_u8u8_s32(kM, kM), hi = 8u | (1u << 14);  // 128 bytes between 8-row groups
    const uint32_t strips = smem_u32(s_strip) >> 4, bank = (smem_u32(s_bank) >> 4) | (128u << 16);
    uint32_t g = 0;
    // test hook: a wait on the drain barrier, which nothing arrives at before the end
    if (p.stall && !mbar_wait(&sh->drain, 0, global_ns() + p.wait_ns)) fail = true;
    fail = __any_sync(0xffffffffu, fail);
    for (uint32_t sp = first; sp < p.spatial && !fail; sp += step) {
      const unsigned long long deadline = global_ns() + p.wait_ns;
      const uint32_t nx = min(p.xt, p.Wo - (sp % p.xtiles) * p.xt);
      for (uint32_t xi = 0; xi < nx; ++xi, ++g) {
        const uint32_t s = g % kBankStrips, d = g & 1u;
        bool got = mbar_wait(&sh->sfull[s], (g / kBankStrips) & 1u, deadline);
        if (g >= 2) got = got && mbar_wait(&sh->dempty[d], ((g >> 1) + 1) & 1u, deadline);
        if (!__all_sync(0xffffffffu, got)) {
          fail = true;
          break;
        }
        tc_fence_after();
        if (leader) {
          const uint32_t dt = tmem + d * kM, base = strips + s * (strip_bytes >> 4);
          for (uint32_t u = 0; u < p.units; u += 4) {
            const uint4 off = *reinterpret_cast<const uint4*>(s_unit + u);
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
              const uint32_t v = u + k, lo = base + (k == 0 ? off.x : k == 1 ? off.y : k == 2 ? off.z : off.w);
              if (v < in_tmem)
                mma_i8_ts(dt, tmem + 256 + 8 * v, ((uint64_t)hi << 32) | lo, idesc, v != 0);
              else if (v < p.units)
                mma_i8_ss(dt, bank + (v - kTmemUnits) * (kUnitBytes >> 4), hi, lo, hi, idesc, 1u);
            }
          }
          mma_commit(&sh->sempty[s]);
          mma_commit(&sh->dfull[d]);
        }
        __syncwarp();
      }
    }
    // every MMA issued has completed before tensor memory is freed
    if (leader) mma_commit(&sh->drain);
    __syncwarp();
    if (!mbar_wait(&sh->drain, 0, global_ns() + kWaitNs) && lane == 0) atomicMax(p.err, p.tag);
  } else {
    // ---- epilogue
    const uint32_t q = warp & 3u, share = __shfl_sync(0xffffffffu, (warp - kBankBuild) >> 2, 0);
    BankLane c{};
    c.lane = lane;
    c.t_first = t0 + q * 32;
    c.t_ok = q * 32 + lane < nt;
    c.tss = s_tss[q * 32 + lane];
    c.general = c.t_ok && c.tss == 0u;
    c.rT = c.tss ? rsqrt_u32(c.tss) : c.t_ok ? 0.0 : 1.0;  // lanes past the bank write nothing
    c.ncT = -4503599627370496.0 * c.rT;
    c.kmin = ~0ull;
    c.kmax = 0ull;
    const bool idle = q * 32 >= nt;  // no template in these lanes
    uint32_t g = 0;
    for (uint32_t sp = first; sp < p.spatial && !fail; sp += step) {
      const unsigned long long deadline = global_ns() + p.wait_ns;
      const uint32_t x0 = (sp % p.xtiles) * p.xt, y0 = (sp / p.xtiles) * kM, nx = min(p.xt, p.Wo - x0);
      for (uint32_t xi = 0; xi < nx; ++xi, ++g) {
        const uint32_t s = g % kBankStrips, d = g & 1u;
        // the strip's norms were written before its barrier; its accumulator
        const bool got = mbar_wait(&sh->sfull[s], (g / kBankStrips) & 1u, deadline) &&
                         mbar_wait(&sh->dfull[d], (g >> 1) & 1u, deadline);
        if (!__all_sync(0xffffffffu, got)) {
          fail = true;
          break;
        }
        tc_fence_after();
        const uint32_t m = share * 32, y = y0 + m;
        const bool work = !idle && y < p.Ho;
        uint32_t b[32];
        if (work) {
          const uint8_t* norm = s_norm + s * kNormBytes;
          bank_scores<kMethod, kPrec>(c, tmem_addr(tmem, q * 32, d * kM + m), reinterpret_cast<const double*>(norm) + m,
                                      reinterpret_cast<const uint32_t*>(norm + 8 * kM) + m, sh->zero[s][share] != 0u,
                                      b);
        }
        // the accumulator and the norms are free: the MMAs two strips on run
        // beside the stores and folds
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&sh->dempty[d]);
          mbar_arrive(&sh->sempty[s]);
        }
        if (work) {
          const int nv = (int)(p.Ho - y);
          if (nv >= 32) bank_store<kExt, true>(p, c, x0 + xi, y, 32, b);
          else bank_store<kExt, false>(p, c, x0 + xi, y, nv, b);
        }
      }
    }
    if (kExt && c.t_ok && !fail) {
      atomicMin(&p.ext[2 * (c.t_first + lane)], c.kmin);
      atomicMax(&p.ext[2 * (c.t_first + lane) + 1], c.kmax);
    }
  }
  if (fail && lane == 0) atomicMax(p.err, p.tag);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == kBankMma) tmem_dealloc(tmem, 512);
}

int sm_count() { return device_sm_count(); }

__global__ void many_keys_init_kernel(unsigned long long* keys, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    keys[2 * i] = ~0ull;
    keys[2 * i + 1] = 0ull;
  }
}

// keys of template t -> ipb_extremes_f32 (locations in the Wo-wide score map)
__global__ void many_keys_finish_kernel(const unsigned long long* keys, uint32_t Wo, ipb_extremes_f32* out,
                                        uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned long long kmin = keys[2 * i], kmax = keys[2 * i + 1];
  auto value = [](uint32_t ok) { return __uint_as_float((ok & 0x80000000u) ? (ok & 0x7FFFFFFFu) : ~ok); };
  const uint32_t imin = (uint32_t)kmin, imax = 0xFFFFFFFFu - (uint32_t)kmax;
  ipb_extremes_f32 r;
  r.max_value = value((uint32_t)(kmax >> 32));
  r.min_value = value((uint32_t)(kmin >> 32));
  r.max_value_location_x = imax % Wo;
  r.max_value_location_y = imax / Wo;
  r.min_value_location_x = imin % Wo;
  r.min_value_location_y = imin / Wo;
  out[i] = r;
}

// Shared-memory carve for a template block of nb; returns the total bytes.
uint32_t many_carve(ManyParams& p, uint32_t nb) {
  uint32_t off = 1024;
  p.b_off = off;
  off += (uint32_t)align_up((size_t)p.h * p.kw * nb, 128);
  p.tss_off = off;
  off += (uint32_t)align_up(4 * nb, 128);
  p.ext_off = off;
  off += (uint32_t)align_up(16 * nb, 128);
  p.img_off = off;
  off += (uint32_t)align_up((size_t)p.rows * p.ip, 128);
  p.strip_off = off;
  off += (uint32_t)align_up((size_t)kStrips * (p.kw / 16) * p.rows * 16, 128);
  p.y_off = off;
  off += kXT * kM * 4;
  p.v_off = off;
  off += (uint32_t)align_up((size_t)p.rows * kVP * 4, 128);
  return off;
}

// The same for a bank of 128 templates as M.
uint32_t bank_carve(ManyParams& p) {
  uint32_t off = 1024;
  p.ext_off = off;  // unit table
  off += (uint32_t)align_up((size_t)4 * p.units + 12, 128);
  p.tss_off = off;
  off += 4 * kM;
  p.ry_off = off;
  off += kBankStrips * kNormBytes;
  p.b_off = off;
  off += (p.units > kTmemUnits ? p.units - kTmemUnits : 0u) * kUnitBytes;
  p.strip_off = off;
  off += kBankStrips * p.nch * p.rows * 16;
  p.img_off = off;
  p.img_bytes = (uint32_t)align_up((size_t)p.rows * p.ip, 128);
  off += 2 * p.img_bytes;
  p.y_off = off;
  off += (uint32_t)align_up((size_t)kXT * kYP * 4, 128);
  p.v_off = off;
  off += (uint32_t)align_up((size_t)p.rows * kVP * 4, 128);
  p.part = std::min(kTmemUnits, ((off - p.strip_off) / kUnitBytes) & ~1u);
  return off;
}

constexpr uint32_t kSmemLimit = 227u * 1024u;

// The bank kernel from three templates on, and with extremes always: its
// epilogue's time hardly depends on how many of a quadrant's lanes hold a
// template, and the other kernel finds extremes by reductions across its
// positions (2048 x 2048, 32 x 32, CrossCorrelationNormalized, bank against
// positions as M: one template 494 and 464 us, four 490 and 524, 64 515 and
// 922; with extremes 558 and 678, 564 and 753, 625 and 1242).
constexpr uint32_t kBankMin = 2;

using ManyKernel = void (*)(ManyParams);

template <bool kBank, int kMethod, int kPrec, bool kExt>
constexpr ManyKernel many_kernel_of() {
  if constexpr (kBank) return many_bank_kernel<kMethod, kPrec, kExt>;
  else return many_match_kernel<kMethod, kPrec, kExt>;
}

// Precision only affects the normalised methods; the others use EXACT_FP64's instance.
template <bool kBank, int kMethod>
ManyKernel many_kernel_m(bool fp64, bool ext) {
  if (!method_is_norm(kMethod) || fp64)
    return ext ? many_kernel_of<kBank, kMethod, IPB_PRECISION_EXACT_FP64, true>()
               : many_kernel_of<kBank, kMethod, IPB_PRECISION_EXACT_FP64, false>();
  return ext ? many_kernel_of<kBank, kMethod, IPB_PRECISION_EXACT_F32, true>()
             : many_kernel_of<kBank, kMethod, IPB_PRECISION_EXACT_F32, false>();
}

template <bool kBank>
ManyKernel many_kernel_a(int method, bool fp64, bool ext) {
  switch (method) {
    case kSse:
      return many_kernel_m<kBank, kSse>(fp64, ext);
    case kSseNorm:
      return many_kernel_m<kBank, kSseNorm>(fp64, ext);
    case kCcorr:
      return many_kernel_m<kBank, kCcorr>(fp64, ext);
    default:
      return many_kernel_m<kBank, kCcorrNorm>(fp64, ext);
  }
}

ManyKernel many_kernel_for(bool bank, int method, bool fp64, bool ext) {
  return bank ? many_kernel_a<true>(method, fp64, ext) : many_kernel_a<false>(method, fp64, ext);
}

}  // namespace

cudaError_t launch_many_keys_init(unsigned long long* keys, uint32_t n, cudaStream_t s) {
  many_keys_init_kernel<<<(n + 255) / 256, 256, 0, s>>>(keys, n);
  count_launch(kKernelExtremes);
  return cudaGetLastError();
}

cudaError_t launch_many_keys_finish(const unsigned long long* keys, uint32_t Wo, ipb_extremes_f32* out, uint32_t n,
                                    cudaStream_t s) {
  many_keys_finish_kernel<<<(n + 255) / 256, 256, 0, s>>>(keys, Wo, out, n);
  count_launch(kKernelExtremes);
  return cudaGetLastError();
}

bool many_supported(uint32_t w, uint32_t h, uint32_t n, int precision) {
  return precision != IPB_PRECISION_REFERENCE_F32 && w >= 16 && w <= 64 && h >= 1 && h <= 64 && n >= 1;
}

cudaError_t launch_many(const uint8_t* img, uint32_t W, uint32_t H, const uint8_t* tpl, uint32_t w, uint32_t h,
                        uint32_t n, int method, int precision, float* out, unsigned long long* ext_keys,
                        unsigned int* err, unsigned int tag, cudaStream_t stream, KernelTimer* timer) {
  ManyParams p{};
  p.img = img;
  p.W = W;
  p.H = H;
  p.tpl = tpl;
  p.w = w;
  p.h = h;
  p.n = n;
  p.kw = (w + 31) & ~31u;
  p.Wo = W - w + 1;
  p.Ho = H - h + 1;
  p.bands = (p.Ho + kM - 1) / kM;
  p.xtiles = (p.Wo + kXT - 1) / kXT;
  p.spatial = p.bands * p.xtiles;
  p.rows = kM + h - 1;
  p.ip = (uint32_t)align_up(kXT + p.kw + 16, 16);
  // templates as M where the bank fits; otherwise the largest positions-as-M
  // block (multiple of 16) that fits
  ManyParams q = p;
  q.nch = (w + 15) / 16;
  q.units = unit_count(q.nch, h);
  q.ip = 16 * ((3 + q.nch) | 1u);  // 32 columns + w - 1, a whole word more; an odd number of 16-byte words
  uint32_t smem = bank_carve(q);
  const bool bank = smem <= kSmemLimit && (n > kBankMin || ext_keys);
  uint32_t nb = kM;
  if (bank) {
    p = q;
  } else {
    for (nb = std::min(112u, (n + 15) & ~15u); nb >= 16; nb -= 16)
      if ((smem = many_carve(p, nb)) <= kSmemLimit) break;
    if (nb < 16) return cudaErrorNotSupported;
  }
  p.NB = nb;
  p.nblocks = (n + nb - 1) / nb;
  p.method = method;
  p.precision = precision;
  p.vec4 = ((n & 3u) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) ? 1 : 0;
  p.img16 = ((reinterpret_cast<uintptr_t>(img) & 15u) == 0 && (W & 15u) == 0) ? 1 : 0;
  p.img4 = ((reinterpret_cast<uintptr_t>(img) & 3u) == 0 && (W & 3u) == 0) ? 1 : 0;
  p.out = out;
  p.ext = ext_keys;
  p.err = err;
  p.tag = tag;
  p.wait_ns = pipeline_wait_ns();
  p.stall = pipeline_stall() ? 1u : 0u;
  static PerDeviceOnce attr;
  cudaError_t e = attr.run([] {
    cudaError_t r = cudaSuccess;
    for (int a = 0; a < 2 && r == cudaSuccess; ++a)
      for (int m = 0; m < 4 && r == cudaSuccess; ++m)
        for (int f = 0; f < 2 && r == cudaSuccess; ++f)
          for (int x = 0; x < 2 && r == cudaSuccess; ++x)
            r = cudaFuncSetAttribute(many_kernel_for(a != 0, m, f != 0, x != 0),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
    return r;
  });
  if (e != cudaSuccess) return e;
  // CTAs come in groups of nblocks (one per template block)
  uint32_t per = (uint32_t)sm_count() / p.nblocks;
  if (per < 1) per = 1;
  if (bank) {
    // the tile width (whole words of image) of the least last wave, a tile's
    // sums worth about three columns
    uint32_t best = 0;
    for (uint32_t xt = 8; xt <= (uint32_t)kXT; xt += 4) {
      const uint32_t tiles = p.bands * ((p.Wo + xt - 1) / xt), cost = (tiles + per - 1) / per * (xt + 3);
      if (best == 0 || cost <= best) {
        best = cost;
        p.xt = xt;
      }
    }
    p.xtiles = (p.Wo + p.xt - 1) / p.xt;
    p.spatial = p.bands * p.xtiles;
  }
  if (per > p.spatial) per = p.spatial;
  const uint32_t grid = per * p.nblocks;
  timer_begin(timer, kKernelMany, stream);
  many_kernel_for(bank, method, precision == IPB_PRECISION_EXACT_FP64, ext_keys != nullptr)
      <<<grid, bank ? kBankThreads : kThreads, smem, stream>>>(p);
  count_launch(kKernelMany);
  timer_end(timer, stream);
  return cudaGetLastError();
}

}  // namespace ipb
