// tm_window.cu -- exact template matching on the 5th-generation tensor cores
// with the staged image tile itself as the MMA's A operand (tcgen05.mma
// kind::i8, unsigned u8 x u8 -> s32, accumulators in tensor memory).
//
// Replaces the scalar walk of methods::*::score_at (src/template_matching.rs:
// 219-376) for unmasked and binary-masked matches with templates up to
// 128 x 128 pixels, for one problem or a batch of many (image, template)
// pairs in one persistent launch, with find_extremes (:479-511) optionally
// fused into the epilogue.
//
// Formulation. A tile is 128 output columns by 16 NJ output rows (NJ = 1, 2,
// 4 or 8). Tensor-memory lane m = 8 G + c (G = 0..15, c = 0..7) stands for
// the output columns x0 + 16 c + s (s = 0..15) of the output rows y0 + NJ G +
// j (j = 0..NJ-1); the accumulator column of (j, s) is 16 j + s. For every
// step rho = 0 .. NJ + h - 2 and K step kk (32 bytes):
//   A_rho[8 G + c][k] = I[y0 + NJ G + rho][x0 + 16 c + k]            k < K
//   B_rho[(j, s)][k]  = T[rho - j][k - s]  (0 <= k - s < w, 0 <= rho - j < h)
//   D[m][(j, s)] += sum_k A_rho[m][k] B_rho[(j, s)][k]
// with K = w + 15 rounded up to 32, so that D[m][(j, s)] is the correlation X
// at its output position. A needs no building: in the canonical no-swizzle
// K-major layout a core matrix is eight 16-byte rows, 16 bytes apart, and the
// tile of image rows staged with a pitch of P >= 127 + w bytes is read in
// place: lanes 16 bytes apart are the overlapping windows of one image row,
// 16 bytes between the two K halves (LBO), NJ P bytes between 8-lane groups
// (SBO), and step rho starts rho rows further down. The whole tile is resident,
// so no step waits for data. B is a window of one buffer: the template rows'
// 16-shift blocks (16 rows of K bytes each) in decreasing template row, so
// the blocks of the output rows that a step feeds are consecutive and the
// MMA's N is 16 times their number.
//
// Against the Hankel-row kernel (tm_umma.cu), which forms every image row's A
// operand with builder warps and hands stages of rows to the MMA warp, the
// tensor pipe runs a whole tile without a hand-off; it pays K / w in extra
// MACs (1.5 at w = 64) where that kernel pays its 16-row bands.
//
//   unmasked:     X from I and T; the window sums Y = sum I^2 are formed from
//                 the staged tile by the workers beside the MMAs (column
//                 sums slid down the rows, a prefix sum along each row).
//   binary mask:  X from I and T m; Y = sum I^2 m as two more correlations,
//                 I^2 = 256 hi + lo (both u8) with m, into accumulators of
//                 their own: Y = 256 Dhi + Dlo, exact below 2^31. Masked
//                 CrossCorrelation needs X alone and skips them.
//
// Problems on one image with one template size (and mask) form sets: a CTA
// takes a tile's members in turn, which share the staged image and the window
// sums.
//
// Roles (20 warps): sixteen workers, one MMA warp, three loader warps (image
// tile by one tensor copy; template blocks, built in chunks of template
// rows into two slots, so a template of any height streams through; a
// template that fits the slots stays for the following tiles of its problem).
// Before the roles part, all warps load the CTA's first tile and build its
// first blocks. The X accumulators are double-buffered, the image tile where
// shared memory allows. Every wait is bounded;
// one that runs out records the launch's tag in the error word and the CTA
// leaves its loops, drains its MMAs and frees its tensor memory.
#include <algorithm>
#include <tuple>
#include <vector>

#include "tm_common.cuh"
#include "tm_internal.h"
#include "tm_sm100.cuh"

namespace ipb {
namespace {

using namespace sm100;

constexpr uint32_t kTileW = 128;  // output columns per tile
constexpr uint32_t kWorkWarps = 16;  // four per tensor-memory lane quadrant
constexpr uint32_t kMmaWarp = kWorkWarps, kLoadWarp = kMmaWarp + 1, kLoadWarps = 3;
constexpr uint32_t kWarps = kLoadWarp + kLoadWarps, kThreads = kWarps * 32, kLoaders = kLoadWarps * 32;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kRing = 8;  // tile indices in flight: roles are at most four tiles apart
constexpr uint32_t kHeader = 1024;
// the zero operands of the clearing MMA: 128 rows 16 bytes apart, 32 bytes each
constexpr uint32_t kZeroBytes = 16 * 127 + 32;
constexpr uint32_t kZeroRegion = 2176;
constexpr uint32_t kFixed = kHeader + kZeroRegion;
constexpr uint32_t kSmemMax = 227 * 1024;
constexpr uint32_t kMinSmem = 120 * 1024;  // one CTA per SM: two never wait on each other's tensor memory
constexpr uint32_t kMaxSide = 128;         // template width and height

static_assert(kZeroBytes <= kZeroRegion, "zero operands");

__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// Barrier of kCount threads that also tells every one of them whether any
// passed `fail` (so a wait that ran out in one warp ends the role in all).
template <int kCount>
__device__ __forceinline__ bool bar_or(uint32_t id, bool fail) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.or.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)fail), "r"(id), "n"(kCount)
      : "memory");
  return r != 0;
}

struct Shared {
  uint64_t img_full[2], img_empty[2];  // image tile slots
  uint64_t b_full[2], b_empty[2];      // template-block slots
  uint64_t acc_full[2], acc_empty[2];  // X accumulator buffers
  uint64_t planes_full, yacc_empty;    // masked: the tile's planes of I^2; Y accumulators read
  uint64_t tile_full[kRing];           // tile indices, claimed by the first loader warp
  uint64_t drain;
  uint32_t tile[kRing];
  uint32_t tss[2 * kRing];  // sum of (T m)^2 of each member's template
  uint32_t tmem, flag;
};
static_assert(sizeof(Shared) <= kHeader, "kernel header");

// first problem of the set that owns a tile, advancing from the set at `pi`
__device__ __forceinline__ uint32_t find_problem(const WindowLaunch& L, const WindowProblem* P, uint32_t pi,
                                                 uint32_t tile) {
  for (;;) {
    const uint32_t nx = pi + P[pi].set_n;
    if (nx >= L.nprobs || tile < P[nx].tile_begin) return pi;
    pi = nx;
  }
}

// A role's walk over the CTA's tiles: `ti` counts tiles, `it` tiles times set
// members (the accumulator hand-overs).
struct Walk {
  uint32_t ti, it, pi, x0, y0, nrows, nset;
  bool ok;
};
__device__ __forceinline__ void set_tile(Walk& w, const WindowLaunch& L, const WindowProblem* P, uint32_t tile) {
  w.pi = find_problem(L, P, w.pi, tile);
  const WindowProblem& q = P[w.pi];
  const uint32_t lt = tile - q.tile_begin;
  w.x0 = (lt % q.tiles_x) * kTileW;
  w.y0 = (lt / q.tiles_x) * (16 * L.nj);
  w.nrows = min(16 * L.nj + q.h - 1, q.H - w.y0);
  w.nset = q.set_n;
}
// Waits for the walk's next claimed tile; false at the end (or, with w.ok
// false, when the wait ran out).
template <bool kSpin>
__device__ __forceinline__ bool next_tile(Walk& w, const WindowLaunch& L, const WindowProblem* P, Shared* sh,
                                          unsigned long long deadline) {
  const uint32_t s = w.ti % kRing, par = (w.ti / kRing) & 1u;
  const bool got = kSpin ? mbar_wait(&sh->tile_full[s], par, deadline)
                         : mbar_wait_sleep(&sh->tile_full[s], par, deadline);
  if (!got) {
    w.ok = false;
    return false;
  }
  const uint32_t tile = *reinterpret_cast<volatile uint32_t*>(&sh->tile[s]);
  if (tile >= L.tiles) return false;
  set_tile(w, L, P, tile);
  return true;
}

// The template side in the slots: which one, whether it stays, and the slot
// of its first chunk (tracked alike by the loader and the MMA warps).
struct BlockState {
  const uint8_t* tpl = nullptr;
  const uint8_t* mask = nullptr;
  uint32_t w = 0, h = 0, first = 0, nch = 0;
  bool with_mask = false;  // the mask's blocks lie beside the template's
  // moves on to q's template; true when all its blocks are still in the slots
  __device__ __forceinline__ bool enter(const WindowProblem& q, bool need_mask) {
    if (nch && nch <= 2 && tpl == q.tpl && mask == q.mask && w == q.w && h == q.h && (with_mask || !need_mask))
      return true;
    first = (first + nch) & 1u;
    nch = q.nch;
    tpl = q.tpl;
    mask = q.mask;
    w = q.w;
    h = q.h;
    with_mask = need_mask;
    return false;
  }
};

// Image rows [y0, y0 + nrows) x columns [x0, x0 + pitch) into the slot, zero
// past the right edge, by `nt` threads, for images whose rows do not all start
// on 16-byte boundaries (the others are one tensor copy): by words where the
// rows are word-aligned, else by 16-byte chunks read as aligned words and
// shifted (a chunk whose words would leave the image, by bytes).
__device__ __forceinline__ void load_image(const WindowProblem& q, const Walk& w, uint8_t* dst, uint32_t t,
                                           uint32_t nt) {
  const uint32_t chunks = q.pitch / 16, total = w.nrows * chunks;
  const uint8_t* src = q.img + (size_t)w.y0 * q.W;
  const uint8_t* end = q.img + (size_t)q.W * q.H;
  if (q.load_mode == 1) {
    for (uint32_t i = t; i < 4 * total; i += nt) {
      const uint32_t r = i / (4 * chunks), c = (i - r * 4 * chunks) * 4, gx = w.x0 + c;
      const uint32_t avail = gx < q.W ? min(4u, q.W - gx) : 0u;
      cp_async4(smem_u32(dst + r * q.pitch + c), src + (size_t)r * q.W + (avail ? gx : 0u), avail);
    }
  } else {
#pragma unroll 4
    for (uint32_t i = t; i < total; i += nt) {
      const uint32_t r = i / chunks, c = (i - r * chunks) * 16, gx = w.x0 + c;
      uint32_t v[4] = {0u, 0u, 0u, 0u};
      if (gx < q.W) {
        const uint8_t* g = src + (size_t)r * q.W + gx;
        const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(g) & 3u);
        const uint8_t* a = g - off;
        if (a >= q.img && a + 20 <= end) {  // bytes past the row's end belong to the next row: never scored
          const uint32_t* a4 = reinterpret_cast<const uint32_t*>(a);
          uint32_t wd[5];
#pragma unroll
          for (int k = 0; k < 5; ++k) wd[k] = __ldg(a4 + k);
          const uint32_t sel = 0x3210u + off * 0x1111u;
#pragma unroll
          for (int k = 0; k < 4; ++k) v[k] = __byte_perm(wd[k], wd[k + 1], sel);
        } else {
          const uint32_t avail = min(16u, q.W - gx);
#pragma unroll
          for (int k = 0; k < 16; ++k)
            if ((uint32_t)k < avail) v[k >> 2] |= (uint32_t)__ldg(g + k) << (8 * (k & 3));
        }
      }
      *reinterpret_cast<uint4*>(dst + r * q.pitch + c) = make_uint4(v[0], v[1], v[2], v[3]);
    }
  }
}

// The same as one tensor copy (rows and columns past the image are zeros),
// issued by one thread and counted on `bar`, its arrival included.
__device__ __forceinline__ void load_tensor(const CUtensorMap* map, const Walk& w, uint8_t* dst, uint32_t bytes,
                                            uint64_t* bar) {
  mbar_arrive_expect_tx(bar, bytes);
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(smem_u32(dst)),
      "l"(map), "r"(w.x0), "r"(w.y0), "r"(smem_u32(bar))
      : "memory");
}

// The template (plane 0: T or T m) and, masked, the mask (plane 1) as they lie
// in memory, by words, zero past the end.
template <bool MASKED>
__device__ __forceinline__ void load_template(const WindowProblem& q, uint8_t* raw, uint32_t raw_bytes, uint32_t t,
                                              uint32_t nt) {
  const uint32_t n = q.w * q.h, words = (n + 3) / 4;
  const bool aligned = ((reinterpret_cast<uintptr_t>(q.tpl) | (MASKED ? reinterpret_cast<uintptr_t>(q.mask) : 0)) & 3u) == 0;
  auto word = [&](const uint8_t* p, uint32_t i) {
    if (aligned && 4 * i + 4 <= n) return __ldg(reinterpret_cast<const uint32_t*>(p) + i);
    uint32_t v = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
      if (4 * i + k < n) v |= (uint32_t)__ldg(p + 4 * i + k) << (8 * k);
    return v;
  };
#pragma unroll 8
  for (uint32_t i = t; i < words; i += nt) {
    uint32_t v = word(q.tpl, i);
    if constexpr (MASKED) {
      const uint32_t m = word(q.mask, i);
      v &= m * 255u;  // bytes of m are 0 or 1
      reinterpret_cast<uint32_t*>(raw + raw_bytes)[i] = m;
    }
    reinterpret_cast<uint32_t*>(raw)[i] = v;
  }
}

// Adds sum T^2 of the words in shared memory (u32: at most 16384 template
// pixels) to *tss, by `nt` threads in whole warps.
__device__ __forceinline__ void add_tss(const uint8_t* raw, uint32_t pixels, uint32_t* tss, uint32_t t, uint32_t nt) {
  uint32_t t2 = 0;
  for (uint32_t i = t; i < (pixels + 3) / 4; i += nt) {
    const uint32_t v = reinterpret_cast<const uint32_t*>(raw)[i];
    t2 = __dp4a(v, v, t2);
  }
  t2 = __reduce_add_sync(0xffffffffu, t2);
  if ((t & 31u) == 0) atomicAdd(tss, t2);
}

// The 16-shift blocks of template rows [d0, d0 + n), in decreasing row: block
// b holds rows s = 0..15 of K bytes, byte k = T[d0 + n - 1 - b][k - s] (0
// outside the row), in the canonical no-swizzle K-major layout (s / 8) 8K +
// (k / 16) 128 + (s % 8) 16. A warp writes four core matrices (512 bytes) of a
// row at once; the K / 32 such groups of all rows are shared out over `nw`
// warps group by group, so that a lane mostly keeps its shift, its chunk and
// the bytes of it that lie in the row while it goes down the rows.
__device__ __forceinline__ void build_blocks(uint32_t K, uint32_t w, uint32_t d0, uint32_t n, const uint8_t* raw,
                                             uint8_t* dst, uint32_t iw, uint32_t nw, uint32_t lane) {
  const uint32_t cpr = K / 16, items = (K / 32) * n;
  uint32_t item = iw * items / nw;
  const uint32_t end = (iw + 1) * items / nw;
  while (item < end) {
    const uint32_t grp = item / n, b_end = min(n, end - grp * n);
    const uint32_t m = 4 * grp + (lane >> 3);
    const uint32_t hi = m >= cpr ? 1u : 0u, ch = m - hi * cpr, sft = 8 * hi + (lane & 7u);
    uint32_t mask[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      mask[i] = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (16 * ch + 4 * i + k - sft < w) mask[i] |= 0xFFu << (8 * k);  // wraps for the bytes ahead of the row
    }
    uint8_t* out = dst + m * 128 + (lane & 7u) * 16;
    const uint32_t first = 16 + 16 * ch - sft;  // sixteen bytes of slack lie ahead of the template
    // four rows' reads ahead of their stores
    for (uint32_t b0 = item - grp * n; b0 < b_end; b0 += 4) {
      uint32_t wd[4][5], sel[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t at = first + (d0 + n - 1 - min(b0 + i, n - 1)) * w;
        const uint32_t* a4 = reinterpret_cast<const uint32_t*>(raw - 16 + (at & ~3u));
        sel[i] = 0x3210u + (at & 3u) * 0x1111u;
#pragma unroll
        for (int k = 0; k < 5; ++k) wd[i][k] = a4[k];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (b0 + i < b_end)
          *reinterpret_cast<uint4*>(out + (b0 + i) * 16 * K) =
              make_uint4(__byte_perm(wd[i][0], wd[i][1], sel[i]) & mask[0],
                         __byte_perm(wd[i][1], wd[i][2], sel[i]) & mask[1],
                         __byte_perm(wd[i][2], wd[i][3], sel[i]) & mask[2],
                         __byte_perm(wd[i][3], wd[i][4], sel[i]) & mask[3]);
    }
    item = grp * n + b_end;
  }
}

// One chunk of the problem's template (and, masked, of the mask) into a slot.
template <bool MASKED>
__device__ __forceinline__ void build_chunk(const WindowProblem& q, uint32_t c, const uint8_t* raw,
                                            uint32_t raw_bytes, uint8_t* slot, bool with_mask, uint32_t iw,
                                            uint32_t nw, uint32_t lane) {
  const uint32_t d0 = c * q.crows, n = min(q.crows, q.h - d0);
  build_blocks(q.K, q.w, d0, n, raw, slot, iw, nw, lane);
  if (MASKED && with_mask)
    build_blocks(q.K, q.w, d0, n, raw + raw_bytes, slot + q.crows * 16 * q.K, iw, nw, lane);
}

__device__ __forceinline__ void add_squares(uint2 v, uint32_t (&a)[8]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t b = ((k < 4 ? v.x : v.y) >> (8 * (k & 3))) & 255u;
    a[k] += b * b;
  }
}
__device__ __forceinline__ void sub_squares(uint2 v, uint32_t (&a)[8]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t b = ((k < 4 ? v.x : v.y) >> (8 * (k & 3))) & 255u;
    a[k] -= b * b;
  }
}

// The squares of four rows: the 4 x 4 bytes of four columns are transposed so
// that each word holds one column's bytes, one dp4a per column.
__device__ __forceinline__ void add_squares4(uint2 r0, uint2 r1, uint2 r2, uint2 r3, uint32_t (&a)[8]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t w0 = h ? r0.y : r0.x, w1 = h ? r1.y : r1.x, w2 = h ? r2.y : r2.x, w3 = h ? r3.y : r3.x;
    const uint32_t a01 = __byte_perm(w0, w1, 0x5140), b01 = __byte_perm(w0, w1, 0x7362);
    const uint32_t a23 = __byte_perm(w2, w3, 0x5140), b23 = __byte_perm(w2, w3, 0x7362);
    const uint32_t c0 = __byte_perm(a01, a23, 0x5410), c1 = __byte_perm(a01, a23, 0x7632);
    const uint32_t c2 = __byte_perm(b01, b23, 0x5410), c3 = __byte_perm(b01, b23, 0x7632);
    a[4 * h] = __dp4a(c0, c0, a[4 * h]);
    a[4 * h + 1] = __dp4a(c1, c1, a[4 * h + 1]);
    a[4 * h + 2] = __dp4a(c2, c2, a[4 * h + 2]);
    a[4 * h + 3] = __dp4a(c3, c3, a[4 * h + 3]);
  }
}

// 16-byte chunk of a 128-word row, permuted so that lanes that own runs of 16
// words, lanes that own runs of 8 and lanes that own single words all reach
// different banks.
__device__ __forceinline__ uint32_t chunk_at(uint32_t cc) { return cc ^ ((cc >> 3) & 3u); }

// Window sums Y = sum I^2 of `nr` output rows from tile row `row0` (one warp):
// a lane owns eight image columns, keeps their sums over h rows (one row added
// and one taken off per output row) and the exclusive prefix of those sums
// along the row; Y is the difference of two prefixes w = 8 a + B columns
// apart, the further one fetched from its lane by shuffles. All arithmetic is
// modulo 2^32; every Y is below 2^31.
template <int B>
__device__ __forceinline__ void window_sums(const uint8_t* img, uint32_t pitch, uint32_t a, uint32_t h,
                                            uint32_t row0, uint32_t nr, uint32_t lane, uint32_t* ytile) {
  const bool in = 8 * lane < pitch;
  const uint2* col = reinterpret_cast<const uint2*>(img + (size_t)row0 * pitch + (in ? 8 * lane : 0u));
  const uint32_t st = pitch / 8;
  uint32_t vs[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  uint32_t dy = 0;
#pragma unroll 2
  for (; dy + 4 <= h; dy += 4)
    add_squares4(col[dy * st], col[(dy + 1) * st], col[(dy + 2) * st], col[(dy + 3) * st], vs);
  for (; dy < h; ++dy) add_squares(col[dy * st], vs);
  // two output rows at a time: their prefix sums are independent chains
  for (uint32_t i = 0; i < nr; i += 2) {
    uint32_t v2[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v2[k] = vs[k];
    const bool two = i + 1 < nr;  // a tile of one row per group has no second row
    if (two) {
      add_squares(col[(i + h) * st], v2);
      sub_squares(col[i * st], v2);
    }
    uint32_t q0[8], q1[8], r0 = 0, r1 = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      q0[k] = r0;
      q1[k] = r1;
      r0 += vs[k];
      r1 += v2[k];
    }
    if (!in) r0 = r1 = 0;
    uint32_t i0 = r0, i1 = r1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t n0 = __shfl_up_sync(0xffffffffu, i0, o), n1 = __shfl_up_sync(0xffffffffu, i1, o);
      if (lane >= (uint32_t)o) {
        i0 += n0;
        i1 += n1;
      }
    }
    i0 -= r0;
    i1 -= r1;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      q0[k] = (in ? q0[k] : 0u) + i0;
      q1[k] = (in ? q1[k] : 0u) + i1;
    }
    uint32_t y0[8], y1[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t from = (lane + a + ((k + B) >> 3)) & 31u;
      y0[k] = __shfl_sync(0xffffffffu, q0[(k + B) & 7], from) - q0[k];
      y1[k] = __shfl_sync(0xffffffffu, q1[(k + B) & 7], from) - q1[k];
    }
    if (lane < 16) {
      uint4* row = reinterpret_cast<uint4*>(ytile + (row0 + i) * kTileW);
      row[chunk_at(2 * lane)] = make_uint4(y0[0], y0[1], y0[2], y0[3]);
      row[chunk_at(2 * lane + 1)] = make_uint4(y0[4], y0[5], y0[6], y0[7]);
      if (two) {
        row += kTileW / 4;
        row[chunk_at(2 * lane)] = make_uint4(y1[0], y1[1], y1[2], y1[3]);
        row[chunk_at(2 * lane + 1)] = make_uint4(y1[4], y1[5], y1[6], y1[7]);
      }
    }
    if (i + 2 < nr) {
#pragma unroll
      for (int k = 0; k < 8; ++k) vs[k] = v2[k];
      add_squares(col[(i + 1 + h) * st], vs);
      sub_squares(col[(i + 1) * st], vs);
    }
  }
}

__device__ __forceinline__ void window_sums_dispatch(const uint8_t* img, uint32_t pitch, uint32_t w, uint32_t h,
                                                     uint32_t row0, uint32_t nr, uint32_t lane, uint32_t* yt) {
  const uint32_t a = w >> 3;
  switch (w & 7u) {
    case 0: window_sums<0>(img, pitch, a, h, row0, nr, lane, yt); break;
    case 1: window_sums<1>(img, pitch, a, h, row0, nr, lane, yt); break;
    case 2: window_sums<2>(img, pitch, a, h, row0, nr, lane, yt); break;
    case 3: window_sums<3>(img, pitch, a, h, row0, nr, lane, yt); break;
    case 4: window_sums<4>(img, pitch, a, h, row0, nr, lane, yt); break;
    case 5: window_sums<5>(img, pitch, a, h, row0, nr, lane, yt); break;
    case 6: window_sums<6>(img, pitch, a, h, row0, nr, lane, yt); break;
    default: window_sums<7>(img, pitch, a, h, row0, nr, lane, yt); break;
  }
}

// The low and high bytes of the squares of four pixels.
__device__ __forceinline__ void square_planes(uint32_t v, uint32_t& lo, uint32_t& hi) {
  uint32_t s[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t b = (v >> (8 * k)) & 255u;
    s[k] = b * b;
  }
  const uint32_t p01 = __byte_perm(s[0], s[1], 0x5140), p23 = __byte_perm(s[2], s[3], 0x5140);
  lo = __byte_perm(p01, p23, 0x5410);  // p: {lo0, lo1, hi0, hi1}
  hi = __byte_perm(p01, p23, 0x7632);
}

// One worker warp's share of a tile's epilogue: lane quadrant `quad` (lane
// groups 4 quad .. + 3), rows j0 .. j1 - 1 of each group.
struct Epi {
  const WindowProblem& q;
  const Walk& w;
  uint32_t nj, acc, accw;  // tensor-memory address (lane quadrant, buffer), columns per accumulator
  uint32_t quad, lane, j0, j1, tss;
  double td, tc;    // TSS and -2^52 TSS
  uint32_t* ytile;  // window sums; each row's place also stages its scores
  bool keep;        // the set's later members need the window sums
};

// Masked: the warp's window sums Y = 256 Dhi + Dlo from the accumulators at
// `acc` (then accw columns further) into the tile.
__device__ __forceinline__ void gather_sums(const Epi& e, uint32_t acc) {
  const uint32_t g = e.lane >> 3, c = e.lane & 7u;
  for (uint32_t j = e.j0; j < e.j1; ++j) {
    uint4* mine = reinterpret_cast<uint4*>(e.ytile + (e.nj * (4 * e.quad + g) + j) * kTileW);
    uint32_t lo[16], hi[16];
    tmem_ld16(acc + 16 * j, lo);
    tmem_ld16(acc + e.accw + 16 * j, hi);
    tmem_wait_ld();
#pragma unroll
    for (int k = 0; k < 16; ++k) lo[k] += 256u * hi[k];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      mine[chunk_at(4 * c + k)] = make_uint4(lo[4 * k], lo[4 * k + 1], lo[4 * k + 2], lo[4 * k + 3]);
  }
}

template <int kMethod, bool kFp64, bool kExt>
__device__ __forceinline__ void epilogue(const Epi& e) {
  constexpr bool kNeedY = kMethod != kCcorr;
  constexpr bool kFilter = method_is_norm(kMethod) && kFp64;
  const WindowProblem& q = e.q;
  const uint32_t g = e.lane >> 3, c = e.lane & 7u;
  const uint32_t xl = e.w.x0 + 16 * c;              // the lane's first column
  const uint32_t gy0 = e.w.y0 + e.nj * 4 * e.quad;  // the quadrant's first row
  unsigned long long kmin = ~0ull, kmax = 0ull;
  for (uint32_t j = e.j0; j < e.j1; ++j) {
    if (gy0 + j >= q.Ho) break;  // warp-uniform: the lowest group's row
    uint4* mine = reinterpret_cast<uint4*>(e.ytile + (e.nj * (4 * e.quad + g) + j) * kTileW);
    const uint32_t y = gy0 + e.nj * g + j;
    const uint32_t nv = y < q.Ho && xl < q.Wo ? min(16u, q.Wo - xl) : 0u;  // the lane's scores inside the map
    uint32_t mn = 0xFFFFFFFFu, jmn = 0, mx = 0u, jmx = 0;
    uint4 ys[4];
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      uint32_t x[8], yw[8];
      tmem_ld8(e.acc + 16 * j + 8 * hf, x);
      const uint32_t at0 = chunk_at(4 * c + 2 * hf), at1 = chunk_at(4 * c + 2 * hf + 1);
      if constexpr (kNeedY) {
        const uint4 v0 = mine[at0], v1 = mine[at1];
        ys[2 * hf] = v0;
        ys[2 * hf + 1] = v1;
        yw[0] = v0.x, yw[1] = v0.y, yw[2] = v0.z, yw[3] = v0.w;
        yw[4] = v1.x, yw[5] = v1.y, yw[6] = v1.z, yw[7] = v1.w;
      } else if (e.keep) {
        ys[2 * hf] = mine[at0];
        ys[2 * hf + 1] = mine[at1];
      }
      tmem_wait_ld();
      uint32_t b[8];
      if constexpr (kFilter) {
        // every score through the filter, as independent chains; if any is
        // undecided (rare), the lane's eight again, exactly
        bool again = e.tss == 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t score = method_is_sse(kMethod) ? yw[k] + e.tss - 2u * x[k] : x[k];
          b[k] = norm_bits_fp64_filter(score, yw[k], e.td, e.tc, again);
        }
        if (again) {
#pragma unroll
          for (int k = 0; k < 8; ++k)
            b[k] = __float_as_uint(finish_score32(kMethod, IPB_PRECISION_EXACT_FP64, x[k], yw[k], e.tss));
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          b[k] = __float_as_uint(finish_score32(kMethod, kFp64 ? IPB_PRECISION_EXACT_FP64 : IPB_PRECISION_EXACT_F32,
                                                x[k], kNeedY ? yw[k] : 0u, e.tss));
      }
      if constexpr (kExt) {
        // scores are never negative, so their f32 bits order like the values;
        // strict comparisons keep the first occurrence
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if ((uint32_t)(8 * hf + k) < nv) {
            if (b[k] < mn) {
              mn = b[k];
              jmn = 8 * hf + k;
            }
            if (b[k] > mx) {
              mx = b[k];
              jmx = 8 * hf + k;
            }
          }
      }
      if (q.out) {
        mine[at0] = make_uint4(b[0], b[1], b[2], b[3]);
        mine[at1] = make_uint4(b[4], b[5], b[6], b[7]);
      }
    }
    if constexpr (kExt) {
      if (nv) {
        const uint32_t lin = y * q.Wo + xl;
        kmin = min(kmin, ((unsigned long long)(mn | 0x80000000u) << 32) | (lin + jmn));
        kmax = max(kmax, ((unsigned long long)(mx | 0x80000000u) << 32) | (0xFFFFFFFFu - (lin + jmx)));
      }
    }
    if (q.out) {
      __syncwarp();
#pragma unroll
      for (uint32_t r = 0; r < 4; ++r) {
        const uint32_t yr = gy0 + e.nj * r + j;
        if (yr >= q.Ho) break;
        const uint32_t* row = e.ytile + (e.nj * (4 * e.quad + r) + j) * kTileW;
        float* orow = q.out + (size_t)yr * q.Wo + e.w.x0;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
          const uint32_t col = 32 * k + e.lane;
          if (e.w.x0 + col < q.Wo) orow[col] = __uint_as_float(row[4 * chunk_at(col >> 2) + (col & 3u)]);
        }
      }
      if (e.keep) {
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) mine[chunk_at(4 * c + k)] = ys[k];
      }
    }
  }
  if constexpr (kExt) {
    for (int o = 16; o > 0; o >>= 1) {
      kmin = min(kmin, __shfl_xor_sync(0xffffffffu, kmin, o));
      kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
    }
    if (e.lane == 0 && kmin != ~0ull) {
      atomicMin(q.ext, kmin);
      atomicMax(q.ext + 1, kmax);
    }
  }
}

template <int kMethod>
__device__ __forceinline__ void epilogue_m(const Epi& e, bool fp64, bool ext) {
  if constexpr (!method_is_norm(kMethod)) fp64 = true;  // precision only affects the normalisation
  if (fp64) {
    if (ext) epilogue<kMethod, true, true>(e);
    else epilogue<kMethod, true, false>(e);
  } else {
    if (ext) epilogue<kMethod, false, true>(e);
    else epilogue<kMethod, false, false>(e);
  }
}

// The MMAs of one chunk of template rows [d0, d0 + n) for one image plane and
// one block buffer, issued by one thread. Step t (rho = d0 + t) feeds the
// tile's rows j = jlo .. jhi from the blocks of template rows rho - j: the
// window of blocks grows with t until every row is fed, then moves through
// the buffer, then shrinks.
struct Chunk {
  uint32_t d, a_lo, a_hi, b_lo, b_hi, row16, K, nj, d0, n;
};

template <uint32_t KSTEPS>
__device__ __forceinline__ void issue_steps(const Chunk& c, uint32_t t0, uint32_t t1, uint32_t d, uint32_t dd,
                                            uint32_t b, uint32_t db, uint32_t id, uint32_t did) {
  uint32_t a = c.a_lo + (c.d0 + t0) * c.row16;
  for (uint32_t t = t0; t < t1; ++t) {
#pragma unroll
    for (uint32_t kk = 0; kk < KSTEPS; ++kk) mma_i8_ss(d, a + 2 * kk, c.a_hi, b + 16 * kk, c.b_hi, id, 1u);
    a += c.row16;
    d += dd;
    b -= db;
    id += did;
  }
}

template <uint32_t KSTEPS>
__device__ __forceinline__ void issue_chunk_k(const Chunk& c) {
  const uint32_t m = min(c.n, c.nj), last = c.n + c.nj - 1;
  const uint32_t one = idesc_u8u8_s32(128, 0) | (2u << 17), step = 2u << 17;  // N = 16, and 16 more
  const uint32_t top = c.b_lo + (c.n - 1) * c.K;                              // block of template row d0
  // growing: steps 0 .. m - 1 feed rows 0 .. t
  issue_steps<KSTEPS>(c, 0, m, c.d, 0, top, c.K, one, step);
  const uint32_t full = one + (m - 1) * step;
  if (c.n >= c.nj) {
    // all nj rows, blocks n - 1 - t down to 0
    issue_steps<KSTEPS>(c, m, c.n, c.d, 0, top - m * c.K, c.K, full, 0);
    issue_steps<KSTEPS>(c, c.n, last, c.d + 16, 16, c.b_lo, 0, full - step, 0u - step);
  } else {
    // fewer template rows than tile rows: n rows at a time, moving down the tile
    issue_steps<KSTEPS>(c, m, c.nj, c.d + 16, 16, c.b_lo, 0, full, 0);
    issue_steps<KSTEPS>(c, c.nj, last, c.d + 16 * (c.nj - m + 1), 16, c.b_lo, 0, full - step, 0u - step);
  }
}

__device__ __forceinline__ void issue_chunk(const Chunk& c) {
  switch (c.K / 32) {
    case 1: issue_chunk_k<1>(c); break;
    case 2: issue_chunk_k<2>(c); break;
    case 3: issue_chunk_k<3>(c); break;
    case 4: issue_chunk_k<4>(c); break;
    default: issue_chunk_k<5>(c); break;
  }
}

template <bool MASKED>
__global__ void __launch_bounds__(kThreads, 1) window_match_kernel(const __grid_constant__ WindowLaunch L) {
  extern __shared__ __align__(1024) uint8_t smem[];
  Shared* sh = reinterpret_cast<Shared*>(smem);
  uint8_t* zero = smem + kHeader;
  // window sums of the tile; masked, in the place of its planes of I^2 (low
  // bytes, high bytes), which no MMA reads any more by then
  uint32_t* ytile = reinterpret_cast<uint32_t*>(smem + kFixed);
  uint8_t* planes = smem + kFixed;
  uint8_t* img = smem + L.img_off;
  uint8_t* bslot = smem + L.b_off;
  uint8_t* raw = smem + L.raw_off + 16;  // the template as it lies in memory
  const bool inl = L.nprobs <= kInlineProblems;
  const WindowProblem* P = inl ? L.inl : L.probs;
  const CUtensorMap* maps = inl ? L.inl_maps : L.maps;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t nj = L.nj, accw = 16 * nj;  // tensor memory: two X accumulators, then (masked) Y low and high
  Walk w{0, 0, 0, 0, 0, 0, 0, true};
  bool fail = false;  // a wait of this warp ran out

  // ---- set-up and the first tile's image, template and first two chunks of
  // blocks, by all warps
  set_tile(w, L, P, blockIdx.x);
  if (tid == kLoadWarp * 32) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh->img_full[i], kLoadWarps);
      mbar_init(&sh->img_empty[i], 1 + kWorkWarps);
      mbar_init(&sh->b_full[i], kLoadWarps);
      mbar_init(&sh->b_empty[i], 1);
      mbar_init(&sh->acc_full[i], 1);
      mbar_init(&sh->acc_empty[i], kWorkWarps);
    }
    mbar_init(&sh->planes_full, kWorkWarps);
    mbar_init(&sh->yacc_empty, kWorkWarps);
    for (uint32_t i = 0; i < kRing; ++i) mbar_init(&sh->tile_full[i], 1);
    mbar_init(&sh->drain, 1);
    sh->flag = 0;
    sh->tss[0] = 0;
    mbar_init_fence();
    fence_proxy_async_smem();
    if (P[w.pi].load_mode == 2) load_tensor(maps + w.pi, w, img, P[w.pi].tile_bytes, &sh->img_full[0]);
  }
  if (P[w.pi].load_mode != 2) load_image(P[w.pi], w, img, tid, kThreads);
  load_template<MASKED>(P[w.pi], raw, L.raw_bytes, tid, kThreads);
  if (warp == kMmaWarp) {
    tmem_alloc(&sh->tmem, kTmemCols);
    tmem_relinquish();
  }
  for (uint32_t i = tid; i < kZeroRegion / 4; i += kThreads) reinterpret_cast<uint32_t*>(zero)[i] = 0u;
  __syncthreads();
  for (uint32_t c = 0; c < min(2u, P[w.pi].nch); ++c)
    build_chunk<MASKED>(P[w.pi], c, raw, L.raw_bytes, bslot + c * L.slot_bytes, P[w.pi].need_y, warp, kWarps, lane);
  add_tss(raw, P[w.pi].w * P[w.pi].h, &sh->tss[0], tid, kThreads);
  cp_async_wait_all();
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = sh->tmem;
  volatile uint32_t* flag = &sh->flag;

  if (warp >= kLoadWarp) {
    // ---- loaders
    const uint32_t lt = tid - kLoadWarp * 32, lw = warp - kLoadWarp;
    BlockState bs;
    uint32_t uses0 = 0, uses1 = 0;  // MMA uses of each block slot so far
    uint32_t claim = blockIdx.x;
    bool pending = true;                   // a tile's image is loading, this warp has not arrived for it
    bool tensor = P[w.pi].load_mode == 2;  // ... by a tensor copy
    uint32_t pslot = 0;
    int last0 = tensor ? 0 : -1, last1 = -1;  // phase of each slot's last load if by a tensor copy
    for (;; ++w.ti) {
      const unsigned long long deadline = global_ns() + L.wait_ns;
      if (lt == 0) {
        if (w.ti) claim = L.sched ? gridDim.x + atomicAdd(L.sched, 1u) : claim + gridDim.x;
        *reinterpret_cast<volatile uint32_t*>(&sh->tile[w.ti % kRing]) = *flag ? 0xFFFFFFFFu : claim;
        mbar_arrive(&sh->tile_full[w.ti % kRing]);
      }
      const bool more = next_tile<true>(w, L, P, sh, deadline);
      fail |= !w.ok;
      if (bar_or<kLoaders>(1, fail)) {
        fail = true;
        break;
      }
      if (!more) break;
      const uint32_t slot = L.nbuf == 2 ? (w.ti & 1u) : 0u;
      uint8_t* dst = img + slot * L.plane_bytes;
      const bool by_tensor = P[w.pi].load_mode == 2, need_y = P[w.pi].need_y;
      auto load = [&]() {
        const uint32_t use = w.ti / L.nbuf;  // earlier tiles in this slot
        pending = true;
        tensor = by_tensor;
        pslot = slot;
        if (by_tensor && lw) return;  // the first loader warp's
        bool got = true;
        if (use) got = mbar_wait_sleep(&sh->img_empty[slot], (use - 1) & 1u, deadline);
        if (!__all_sync(0xffffffffu, got)) {
          fail = true;
        } else if (by_tensor) {
          if (lane == 0) load_tensor(maps + w.pi, w, dst, P[w.pi].tile_bytes, &sh->img_full[slot]);
          __syncwarp();
          (slot ? last1 : last0) = (int)use;
        } else {
          load_image(P[w.pi], w, dst, lt, kLoaders);
          (slot ? last1 : last0) = -1;
        }
      };
      auto publish_image = [&]() {
        if (!by_tensor) {
          cp_async_wait_all();
          fence_proxy_async_smem();
          __syncwarp();
        }
        if (lane == 0 && !(by_tensor && lw == 0)) mbar_arrive(&sh->img_full[slot]);
        pending = false;
      };
      for (uint32_t m = 0; m < w.nset && !fail; ++m, ++w.it) {
        const WindowProblem q = P[w.pi + m];
        const bool resident = bs.enter(q, m == 0 && need_y), first = w.it == 0;
        uint32_t* tss = &sh->tss[w.it % (2 * kRing)];
        if (m == 0 && !first && (L.nbuf == 2 || resident)) load();
        if (!first && !resident) {
          if (lt == 0) *tss = 0;
          if (m && bar_or<kLoaders>(1, fail)) {  // the last member's blocks are built
            fail = true;
            break;
          }
          load_template<MASKED>(q, raw, L.raw_bytes, lt, kLoaders);
          if (bar_or<kLoaders>(1, fail)) {
            fail = true;
            break;
          }
          add_tss(raw, q.w * q.h, tss, lt, kLoaders);
        }
        if (resident) {
          if (lt == 0) *tss = sh->tss[(w.it - 1) % (2 * kRing)];
          if (m == 0) publish_image();
        }
        for (uint32_t c = 0; c < q.nch; ++c) {
          const uint32_t s = (bs.first + c) & 1u, uses = s ? uses1 : uses0;
          if (s) ++uses1;
          else ++uses0;
          if (resident) continue;  // the MMA warp uses the chunk's slot once more
          if (!(first && c < 2)) {
            if (uses && !mbar_wait_sleep(&sh->b_empty[s], (uses - 1) & 1u, deadline)) fail = true;
            if (bar_or<kLoaders>(1, fail)) {
              fail = true;
              break;
            }
            build_chunk<MASKED>(q, c, raw, L.raw_bytes, bslot + s * L.slot_bytes, m == 0 && need_y, lw, kLoadWarps,
                                lane);
            fence_proxy_async_smem();
            __syncwarp();
          }
          if (lane == 0) mbar_arrive(&sh->b_full[s]);
          if (c == 0 && m == 0) {
            if (!first && L.nbuf == 1) load();
            publish_image();
          }
        }
      }
      if (fail) break;
    }
    // no copy is in flight when the CTA leaves: a load cut short gets this
    // warp's arrival, and the first warp waits for the tensor copies it issued
    cp_async_wait_all();
    if (pending && tensor && lw && lane == 0) mbar_arrive(&sh->img_full[pslot]);
    if (lw == 0) {
      const unsigned long long deadline = global_ns() + kDefaultWaitNs;
      if (last0 >= 0) mbar_wait_sleep(&sh->img_full[0], last0 & 1, deadline);
      if (last1 >= 0) mbar_wait_sleep(&sh->img_full[1], last1 & 1, deadline);
    }
  } else if (warp == kMmaWarp) {
    // ---- MMA issue
    BlockState bs;
    uint32_t builds0 = 0, builds1 = 0, ytiles = 0;
    const bool leader = elect_one();
    const uint32_t z = smem_u32(zero) >> 4, imga = smem_u32(img) >> 4, pla = smem_u32(planes) >> 4,
                   ba = smem_u32(bslot) >> 4;
    auto clear = [&](uint32_t d) {
      const uint32_t id = idesc_u8u8_s32(128, 0) | ((accw >> 3) << 17);
      mma_i8_ss(d, z | (1u << 16), 8u | (1u << 14), z | (1u << 16), 8u | (1u << 14), id, 0u);
    };
    // test hook: a wait on the drain barrier, which nothing arrives at before the end
    if (L.stall && !mbar_wait(&sh->drain, 0, global_ns() + L.wait_ns)) fail = true;
    fail = __any_sync(0xffffffffu, fail);
    for (; !fail; ++w.ti) {
      const unsigned long long deadline = global_ns() + L.wait_ns;
      const bool more = next_tile<true>(w, L, P, sh, deadline);
      if (!__all_sync(0xffffffffu, w.ok)) fail = true;
      if (!more || fail) break;
      const uint32_t slot = L.nbuf == 2 ? (w.ti & 1u) : 0u;
      const bool set_y = MASKED && P[w.pi].need_y;
      if (!__all_sync(0xffffffffu, mbar_wait(&sh->img_full[slot], (w.ti / L.nbuf) & 1u, deadline))) {
        fail = true;
        break;
      }
      tc_fence_after();
      bool planes_ready = false;
      for (uint32_t m = 0; m < w.nset && !fail; ++m, ++w.it) {
        const WindowProblem q = P[w.pi + m];
        const bool with_y = set_y && m == 0;
        const uint32_t buf = w.it & 1u, use = w.it >> 1;
        bool got = true;
        if (use) got = mbar_wait(&sh->acc_empty[buf], (use - 1) & 1u, deadline);
        if (!__all_sync(0xffffffffu, got)) {
          fail = true;
          break;
        }
        tc_fence_after();
        const uint32_t d = tbase + buf * accw, dy = tbase + 2 * accw;
        const uint32_t row16 = q.pitch >> 4;
        const uint32_t a_lo = (imga + slot * (L.plane_bytes >> 4)) | (1u << 16), a_hi = (nj * row16) | (1u << 14);
        const uint32_t b_hi = (q.K >> 1) | (1u << 14);  // 8 K bytes between 8-row groups
        if (leader) clear(d);
        const bool resident = bs.enter(q, m == 0 && P[w.pi].need_y);
        for (uint32_t c = 0; c < q.nch && !fail; ++c) {
          const uint32_t s = (bs.first + c) & 1u;
          if (!resident) {
            const uint32_t builds = s ? builds1++ : builds0++;
            if (!__all_sync(0xffffffffu, mbar_wait(&sh->b_full[s], builds & 1u, deadline))) {
              fail = true;
              break;
            }
            tc_fence_after();
          }
          const uint32_t d0 = c * q.crows, n = min(q.crows, q.h - d0);
          const uint32_t b_lo = (ba + s * (L.slot_bytes >> 4)) | (8u << 16);
          if (leader) issue_chunk(Chunk{d, a_lo, a_hi, b_lo, b_hi, row16, q.K, nj, d0, n});
          __syncwarp();
          if constexpr (MASKED) {
            if (with_y) {
              if (!planes_ready) {
                got = mbar_wait(&sh->planes_full, w.ti & 1u, deadline);
                if (ytiles) got = got && mbar_wait(&sh->yacc_empty, (ytiles - 1) & 1u, deadline);
                if (!__all_sync(0xffffffffu, got)) {
                  fail = true;
                  break;
                }
                tc_fence_after();
                planes_ready = true;
                ++ytiles;
                if (leader) {
                  clear(dy);
                  clear(dy + accw);
                }
              }
              if (leader)
                for (uint32_t p = 0; p < 2; ++p)
                  issue_chunk(Chunk{dy + p * accw, (pla + p * (L.plane_bytes >> 4)) | (1u << 16), a_hi,
                                    b_lo + q.crows * q.K, b_hi, row16, q.K, nj, d0, n});
              __syncwarp();
            }
          }
          if (leader) mma_commit(&sh->b_empty[s]);
          __syncwarp();
        }
        if (fail) break;
        if constexpr (MASKED) {
          // every phase of planes_full is waited for, also by sets that need X
          // alone, so that its parity stays in step with the tiles
          if (m == 0 && !planes_ready &&
              !__all_sync(0xffffffffu, mbar_wait(&sh->planes_full, w.ti & 1u, deadline))) {
            fail = true;
            break;
          }
        }
        if (leader) {
          if (m + 1 == w.nset) mma_commit(&sh->img_empty[slot]);
          mma_commit(&sh->acc_full[buf]);
        }
        __syncwarp();
      }
    }
    // every MMA issued has completed before tensor memory is freed
    if (leader) mma_commit(&sh->drain);
    __syncwarp();
    if (!mbar_wait(&sh->drain, 0, global_ns() + kDefaultWaitNs) && lane == 0) atomicMax(L.err, L.tag);
  } else {
    // ---- workers: window sums (unmasked) or planes of I^2 (masked) of a tile
    // beside its MMAs, then the epilogue of each of its set's members. A
    // quadrant's four warps share the rows of its lane groups: each forms one
    // group's window sums, then scores a quarter of every group's rows.
    const uint32_t quad = warp & 3, sub = warp >> 2;
    const uint32_t j0 = sub * nj / 4, j1 = (sub + 1) * nj / 4;
    for (;; ++w.ti) {
      const unsigned long long deadline = global_ns() + L.wait_ns;
      const bool more = next_tile<false>(w, L, P, sh, deadline);
      fail = __any_sync(0xffffffffu, fail || !w.ok);
      if constexpr (MASKED) {
        // the planes replace the last tile's window sums
        if (bar_or<kWorkWarps * 32>(6, fail)) {
          fail = true;
          break;
        }
      }
      const uint32_t slot = L.nbuf == 2 ? (w.ti & 1u) : 0u;
      const bool need_y = P[w.pi].need_y;
      if (more && !fail) {
        if (need_y) {
          const bool got = mbar_wait_sleep(&sh->img_full[slot], (w.ti / L.nbuf) & 1u, deadline);
          if (!__all_sync(0xffffffffu, got)) fail = true;
          const WindowProblem& q = P[w.pi];
          const uint8_t* src = img + slot * L.plane_bytes;
          if constexpr (MASKED) {
            if (!fail)
              for (uint32_t i = tid; i < w.nrows * (q.pitch >> 4); i += kWorkWarps * 32) {
                const uint4 v = reinterpret_cast<const uint4*>(src)[i];
                uint4 lo, hi;
                square_planes(v.x, lo.x, hi.x);
                square_planes(v.y, lo.y, hi.y);
                square_planes(v.z, lo.z, hi.z);
                square_planes(v.w, lo.w, hi.w);
                reinterpret_cast<uint4*>(planes)[i] = lo;
                reinterpret_cast<uint4*>(planes + L.plane_bytes)[i] = hi;
              }
            fence_proxy_async_smem();
          } else if (!fail) {
            window_sums_dispatch(src, q.pitch, q.w, q.h, nj * (4 * quad + sub), nj, lane, ytile);
          }
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&sh->img_empty[slot]);
          if constexpr (MASKED) mbar_arrive(&sh->planes_full);
        }
      }
      if (bar_or<128>(2 + quad, fail)) {
        fail = true;
        break;
      }
      if (!more) break;
      for (uint32_t m = 0; m < w.nset && !fail; ++m, ++w.it) {
        const WindowProblem& q = P[w.pi + m];
        const uint32_t buf = w.it & 1u;
        const bool got = mbar_wait_sleep(&sh->acc_full[buf], (w.it >> 1) & 1u, deadline);
        if (!__all_sync(0xffffffffu, got)) {
          fail = true;
          break;
        }
        tc_fence_after();
        const uint32_t tss = *reinterpret_cast<volatile uint32_t*>(&sh->tss[w.it % (2 * kRing)]);
        const double td = u32_to_double(tss);
        const uint32_t acc = tmem_addr(tbase, 32 * quad, 0);
        const Epi e{q, w, nj, acc + buf * accw, accw, quad, lane, j0, j1, tss, td, -4503599627370496.0 * td, ytile,
                    need_y && m + 1 < w.nset};
        if constexpr (MASKED) {
          if (need_y && m == 0) {
            gather_sums(e, acc + 2 * accw);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->yacc_empty);
          }
        }
        const bool fp64 = q.precision == IPB_PRECISION_EXACT_FP64, ext = q.ext != nullptr;
        switch (q.method) {
          case kSse: epilogue_m<kSse>(e, fp64, ext); break;
          case kSseNorm: epilogue_m<kSseNorm>(e, fp64, ext); break;
          case kCcorr: epilogue_m<kCcorr>(e, fp64, ext); break;
          default: epilogue_m<kCcorrNorm>(e, fp64, ext); break;
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->acc_empty[buf]);
      }
      // the quadrant's rows hold the next tile's window sums from here on
      if (bar_or<128>(2 + quad, fail)) {
        fail = true;
        break;
      }
    }
  }
  if (fail && lane == 0) {
    *flag = 1u;
    atomicMax(L.err, L.tag);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (L.sched && tid == 0) {
    // every CTA has made its last claim before it counts itself out, so the
    // last one out re-arms the counter for the next launch that uses it
    __threadfence();
    if (atomicAdd(L.sched + 1, 1u) == gridDim.x - 1) {
      atomicExch(L.sched, 0u);
      atomicExch(L.sched + 1, 0u);
    }
  }
  if (warp == kMmaWarp) tmem_dealloc(tbase, kTmemCols);
}

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
  static const EncodeTiled fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &r) != cudaSuccess ||
        r != cudaDriverEntryPointSuccess) {
      (void)cudaGetLastError();
      p = nullptr;
    }
    return reinterpret_cast<EncodeTiled>(p);
  }();
  return fn;
}

uint32_t k_of(uint32_t w) { return (w + 15 + 31) & ~31u; }
// Staged image row: the columns a tile's outputs read. A row's last K windows
// run on into the next row, where B is zero.
uint32_t pitch_of(uint32_t w) { return (kTileW - 1 + w + 15) & ~15u; }

}  // namespace

bool window_supported(const MatchArgs& a) {
  if (a.precision == IPB_PRECISION_REFERENCE_F32 || (a.mask && !a.mask_binary)) return false;
  if (a.w < 1 || a.h < 1 || a.w > kMaxSide || a.h > kMaxSide || a.w > a.W || a.h > a.H) return false;
  // tile indices are 32-bit whatever the tile height
  return (uint64_t)((a.W - a.w) / kTileW + 1) * ((a.H - a.h) / 16 + 1) < 0xFFFF0000ull;
}

bool window_plan_for(uint32_t wmax, uint32_t hmax, bool masked, uint32_t nj, uint32_t nbuf, WindowPlan& pl) {
  const uint32_t K = k_of(wmax), rows = 16 * nj + hmax - 1;
  pl.masked = masked;
  pl.nj = nj;
  pl.nbuf = masked ? 1u : nbuf;
  // the last row's K windows end up to 16 bytes past it
  pl.plane_bytes = (uint32_t)align_up((size_t)rows * pitch_of(wmax) + 64, 128);
  const uint32_t yreg = 16 * nj * kTileW * 4;
  pl.img_off = kFixed + (masked ? std::max(yreg, 2u * pl.plane_bytes) : yreg);
  pl.b_off = pl.img_off + pl.nbuf * pl.plane_bytes;
  // the template (and mask) as it lies in memory, with slack on both sides
  // for the blocks' 20-byte reads
  pl.raw_bytes = (uint32_t)align_up((size_t)wmax * hmax + 96, 128);
  const uint32_t raw = pl.raw_bytes * (masked ? 2u : 1u);
  if (pl.b_off + raw >= kSmemMax) return false;
  pl.slot_bytes = (kSmemMax - pl.b_off - raw) / 2 & ~127u;
  const uint32_t block = 16 * K * (masked ? 2u : 1u);
  // a template needs no more than a slot of its own size
  pl.slot_bytes = std::min(pl.slot_bytes, (uint32_t)align_up((size_t)hmax * block, 128));
  if (pl.slot_bytes < 8 * block && pl.slot_bytes < hmax * block) return false;
  pl.raw_off = pl.b_off + 2 * pl.slot_bytes;
  pl.smem = std::max(kMinSmem, pl.raw_off + raw);
  return pl.smem <= kSmemMax;
}

// Two image tiles where the largest template still fits the block slots beside
// them (its blocks then stay from tile to tile), else one.
bool window_plan_best(uint32_t wmax, uint32_t hmax, bool masked, uint32_t nj, WindowPlan& pl) {
  if (!masked && window_plan_for(wmax, hmax, masked, nj, 2, pl) &&
      2 * (pl.slot_bytes / (16 * k_of(wmax))) >= hmax)
    return true;
  return window_plan_for(wmax, hmax, masked, nj, 1, pl);
}

WindowProblem window_problem(const MatchArgs& a, const WindowPlan& pl, unsigned long long* ext, CUtensorMap* map) {
  WindowProblem q{};
  q.img = a.img;
  q.tpl = a.tpl;
  q.mask = a.mask;
  q.out = a.out;
  q.ext = ext;
  q.W = a.W;
  q.H = a.H;
  q.w = a.w;
  q.h = a.h;
  q.Wo = a.W - a.w + 1;
  q.Ho = a.H - a.h + 1;
  q.tiles_x = (q.Wo + kTileW - 1) / kTileW;
  q.K = k_of(a.w);
  q.pitch = pitch_of(a.w);
  const uint32_t fit = pl.slot_bytes / (16 * q.K * (a.mask ? 2u : 1u));  // template rows per slot
  q.nch = (a.h + fit - 1) / fit;
  q.crows = (a.h + q.nch - 1) / q.nch;
  const uintptr_t ia = reinterpret_cast<uintptr_t>(a.img);
  q.load_mode = ((ia & 3u) == 0 && (a.W & 3u) == 0) ? 1 : 0;
  const uint32_t rows = 16 * pl.nj + a.h - 1;
  q.tile_bytes = q.pitch * rows;
  if ((ia & 15u) == 0 && (a.W & 15u) == 0 && encode_tiled()) {
    const cuuint64_t dims[2] = {a.W, a.H}, strides[1] = {a.W};
    const cuuint32_t box[2] = {q.pitch, rows}, step[2] = {1, 1};
    if (encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(a.img), dims, strides, box, step,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS)
      q.load_mode = 2;
  }
  q.method = a.method;
  q.precision = a.precision;
  q.set_n = 1;
  q.need_y = a.method != IPB_CROSS_CORRELATION;
  return q;
}

namespace {
// one image, one template size, one mask buffer: a tile of the class's
// problems shares its image rows and its window sums
auto set_class(const WindowProblem& q) { return std::make_tuple(q.img, q.W, q.H, q.w, q.h, q.mask); }
}  // namespace

uint32_t window_make_sets(std::vector<WindowProblem>& probs, std::vector<CUtensorMap>& maps, const WindowPlan& pl,
                          uint32_t most) {
  std::vector<uint32_t> order(probs.size());
  for (uint32_t i = 0; i < order.size(); ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
    // one template's problems follow each other: its blocks stay in shared memory
    return std::make_tuple(set_class(probs[a]), probs[a].tpl) < std::make_tuple(set_class(probs[b]), probs[b].tpl);
  });
  std::vector<WindowProblem> p;
  std::vector<CUtensorMap> mp;
  for (uint32_t i : order) {
    p.push_back(probs[i]);
    mp.push_back(maps[i]);
  }
  uint32_t tiles = 0;
  for (size_t i = 0, j; i < p.size(); i = j) {
    for (j = i + 1; j < p.size() && set_class(p[i]) == set_class(p[j]); ++j) {
    }
    // sets whose sizes differ by at most one
    const uint32_t cnt = (uint32_t)(j - i), nsets = (cnt + most - 1) / most;
    size_t k = i;
    for (uint32_t t = 0; t < nsets; ++t) {
      const uint32_t sz = cnt / nsets + (t < cnt % nsets ? 1u : 0u);
      uint32_t need_y = 0;
      for (uint32_t u = 0; u < sz; ++u) need_y |= p[k + u].need_y;
      for (uint32_t u = 0; u < sz; ++u) {
        p[k + u].set_n = u == 0 ? sz : 0u;
        p[k + u].need_y = need_y;
        p[k + u].tile_begin = tiles;
      }
      tiles += window_problem_tiles(p[k], pl);
      k += sz;
    }
  }
  probs.swap(p);
  maps.swap(mp);
  return tiles;
}

uint32_t window_problem_tiles(const WindowProblem& q, const WindowPlan& pl) {
  return q.tiles_x * ((q.Ho + 16 * pl.nj - 1) / (16 * pl.nj));
}

cudaError_t window_prepare_kernels() {
  static PerDeviceOnce attr;
  return attr.run([] {
    cudaError_t e = cudaFuncSetAttribute(window_match_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kSmemMax);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(window_match_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kSmemMax);
  });
}

cudaError_t launch_window_batch(const WindowPlan& pl, WindowLaunch& L, cudaStream_t stream, KernelTimer* timer) {
  L.nj = pl.nj;
  L.nbuf = pl.nbuf;
  L.plane_bytes = pl.plane_bytes;
  L.slot_bytes = pl.slot_bytes;
  L.img_off = pl.img_off;
  L.b_off = pl.b_off;
  L.raw_off = pl.raw_off;
  L.raw_bytes = pl.raw_bytes;
  if (L.tiles == 0) return cudaSuccess;
  cudaError_t e = window_prepare_kernels();
  if (e != cudaSuccess) return e;
  const uint32_t grid = std::min<uint32_t>(L.tiles, (uint32_t)device_sm_count());
  timer_begin(timer, kKernelUmma, stream);
  if (pl.masked) window_match_kernel<true><<<grid, kThreads, pl.smem, stream>>>(L);
  else window_match_kernel<false><<<grid, kThreads, pl.smem, stream>>>(L);
  count_launch(kKernelUmma);
  timer_end(timer, stream);
  return cudaGetLastError();
}

// Tile height of one launch of n problems of one size in sets of up to `set`:
// the smallest estimate of waves x (the set's MMAs and last epilogue) +
// set-up, in cycles. An SS MMA of 128 x N x 32 takes max(32 + N/4, N/2); the
// epilogue about 1000 per 16 output rows.
uint32_t window_tile_nj(const MatchArgs& a, uint32_t n, uint32_t set) {
  const uint32_t sms = (uint32_t)device_sm_count(), nsets = (n + set - 1) / set;
  const uint32_t Wo = a.W - a.w + 1, Ho = a.H - a.h + 1;
  double best = 0;
  uint32_t nj_best = 8;
  for (uint32_t nj : {8u, 4u, 2u, 1u}) {
    const uint64_t tiles = (uint64_t)((Wo + kTileW - 1) / kTileW) * ((Ho + 16 * nj - 1) / (16 * nj)) * nsets;
    const double full = std::max(32.0 + 4.0 * nj, 8.0 * nj), part = 32.0 + 2.0 * nj;
    const double steps = (a.h >= nj ? a.h - nj + 1 : 1) * full + 2.0 * (nj - 1) * part;
    const double corr = (double)((n + nsets - 1) / nsets) + (a.mask ? 2.0 : 0.0);
    const double unit = corr * (k_of(a.w) / 32) * steps + 1000.0 * nj;
    const double cost = (double)((tiles + sms - 1) / sms) * unit + 6000.0;
    if (best == 0 || cost < best) {
      best = cost;
      nj_best = nj;
    }
  }
  return nj_best;
}

// One launch of n <= kInlineProblems problems of one image, template size and
// mask. The image tile is double-buffered when a CTA has several of them and
// the template still fits the block slots.
cudaError_t launch_window_few(const MatchArgs* a, uint32_t n, unsigned long long* keys, unsigned int* err_word,
                              unsigned int tag, cudaStream_t stream, KernelTimer* timer) {
  if (n == 0) return cudaSuccess;
  if (n > kInlineProblems) return cudaErrorNotSupported;
  for (uint32_t i = 0; i < n; ++i)
    if (!window_supported(a[i])) return cudaErrorNotSupported;
  const uint32_t nsets = (n + kMaxSet - 1) / kMaxSet, set = (n + nsets - 1) / nsets;
  WindowPlan pl;
  bool have = false;
  for (uint32_t nj = window_tile_nj(a[0], n, set); nj >= 1 && !have; nj /= 2)
    have = window_plan_best(a[0].w, a[0].h, a[0].mask != nullptr, nj, pl);
  if (!have) return cudaErrorNotSupported;
  std::vector<WindowProblem> probs(n);
  std::vector<CUtensorMap> maps(n);
  for (uint32_t i = 0; i < n; ++i) probs[i] = window_problem(a[i], pl, keys ? keys + 2 * i : nullptr, &maps[i]);
  WindowLaunch L{};
  L.tiles = window_make_sets(probs, maps, pl, set);
  for (uint32_t i = 0; i < n; ++i) {
    L.inl[i] = probs[i];
    L.inl_maps[i] = maps[i];
  }
  L.nprobs = n;
  L.err = err_word;
  L.tag = tag;
  L.wait_ns = pipeline_wait_ns();
  L.stall = pipeline_stall() ? 1u : 0u;
  return launch_window_batch(pl, L, stream, timer);
}

cudaError_t launch_window(const MatchArgs& a, unsigned int* err_word, unsigned int tag) {
  return launch_window_few(&a, 1, nullptr, err_word, tag, a.stream, a.timer);
}

}  // namespace ipb
