// tm_window.cu -- exact template matching on the 5th-generation tensor cores
// with the staged image tile itself as an MMA operand (tcgen05.mma kind::i8,
// unsigned u8 x u8 -> s32, accumulators in tensor memory).
//
// Replaces the scalar walk of methods::*::score_at (src/template_matching.rs:
// 219-376) for unmasked and binary-masked matches with templates up to
// 128 x 128 pixels, for one problem or a batch of many (image, template)
// pairs in one persistent launch, with find_extremes (:479-511) optionally
// fused into the epilogue.
//
// Formulation. A tile is 128 output columns by 16 NJ output rows (NJ = 1, 2,
// 4 or 8). Tensor-memory lane m = 16 j + s (j = 0..7, s = 0..15) and
// accumulator column n = 8 G + c (G = 0..2NJ-1, c = 0..7) stand for the output
// at row y0 + 8 G + j, column x0 + 16 c + s. For every step rho = 0 .. h + 6
// and K step kk (32 bytes):
//   A_rho[(j, s)][k]  = T[rho - j][k - s]  (0 where outside the template)
//   B_rho[8 G + c][k] = I[y0 + 8 G + rho][x0 + 16 c + k]             k < K
//   D[m][n] += sum_k A_rho[m][k] B_rho[n][k]
// with K = w + 15 rounded up to 32, so that D[m][n] is the correlation X at
// its output position. B needs no building: in the canonical no-swizzle
// K-major layout a core matrix is eight 16-byte rows, and the tile of image
// rows staged with a pitch of P >= 127 + w bytes is read in place: rows n 16
// bytes apart are the overlapping windows of one image row, 16 bytes between
// the two K halves (LBO), 8 P bytes between 8-row groups (SBO), and step rho
// starts rho rows further down. The whole tile is resident, so no step waits
// for data. A is a window of one buffer: the template rows' 16-shift blocks
// (16 rows of K bytes each) in decreasing template row, with zero blocks on
// both sides; moving to the next step moves A's start back by one block.
//
// Against the Hankel-row kernel (tm_umma.cu), which forms every image row's A
// operand with builder warps and hands stages of rows to the MMA warp, the
// tensor pipe runs a whole tile without a hand-off; it pays K / w in extra
// MACs (1.5 at w = 64) where that kernel pays its 16-row bands. What is short
// then is shared memory: an MMA of 128 x 128 x 32 reads 8 KB of operands in 64
// cycles, all the bandwidth there is, so every other access delays the tile.
// Hence the lanes stand for (row, shift): sixteen lanes hold sixteen
// neighbouring columns, and scores go from registers to the map without
// staging (with lanes for 16-column groups, scores were transposed through
// shared memory: four unmasked 1080p maps with 64 x 64 templates 65 us, so
// 56 us).
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
// tile by one tensor copy where its rows allow one, else the workers load it;
// template blocks, built in chunks of template rows into two slots, so a
// template of any height streams through; a template that fits the slots stays
// for the following tiles of its problem).
// Before the roles part, all warps load the CTA's first tile and build its
// first blocks. The X accumulators are double-buffered, the image tile where
// shared memory allows. Every wait is bounded;
// one that runs out records the launch's tag in the error word and the CTA
// leaves its loops, drains its MMAs and frees its tensor memory.
#include <algorithm>
#include <cmath>
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
// Uses of a block slot that may be complete beyond the one a loader waits for.
// While a template stays in its slots the MMA warp needs nothing from the
// loaders but the next tile's image, which they load after they have waited
// for every use but a slot's last one: at most kMaxSet uses follow.
constexpr uint32_t kUses = 8;
static_assert(kUses > kMaxSet + 1, "a slot's uses in flight");
constexpr uint32_t kHeader = 1024;
constexpr uint32_t kFixed = kHeader;
constexpr uint32_t kSmemMax = 227 * 1024;
constexpr uint32_t kMinSmem = 120 * 1024;  // one CTA per SM: two never wait on each other's tensor memory
constexpr uint32_t kMaxSide = 128;         // template width and height

__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

struct Shared {
  uint64_t img_full[2], img_empty[2];  // image tile slots
  uint64_t b_full[2];                  // template-block slots: a chunk is built,
  uint64_t b_empty[2][kUses];          // ... use n of the slot's blocks is complete (n % kUses)
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
  bool mask_last = false;  // the mask's blocks followed the template's
  // moves on to q's template (with_y: and its mask); true when all its blocks
  // are still in the slots
  __device__ __forceinline__ bool enter(const WindowProblem& q, bool with_y) {
    if (nch && nch <= 2 && !mask_last && !with_y && tpl == q.tpl && mask == q.mask && w == q.w && h == q.h)
      return true;
    first = q.both ? 0u : (first + nch) & 1u;
    nch = (q.both ? 2u : q.nch) * (with_y ? 2u : 1u);  // a chunk over both slots uses each once
    tpl = q.tpl;
    mask = q.mask;
    w = q.w;
    h = q.h;
    mask_last = with_y;
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
// issued by one thread, which makes all of the phase's arrivals on `bar`: no
// arrival for a phase may precede the last phase's bytes. A map in global
// memory was written by the host: the fence orders its reads after that.
__device__ __forceinline__ void load_tensor(const CUtensorMap* map, bool global, const Walk& w, uint8_t* dst,
                                            uint32_t bytes, uint64_t* bar) {
  if (global) asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
  mbar_arrive_expect_tx(bar, bytes);
  for (uint32_t i = 1; i < kWorkWarps; ++i) mbar_arrive(bar);
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(smem_u32(dst)),
      "l"(map), "r"(w.x0), "r"(w.y0), "r"(smem_u32(bar))
      : "memory");
}

// Bytes [x, x + 4) of a w-byte row that starts at p, zero past its end, read
// as aligned words where those lie inside [p0, end).
__device__ __forceinline__ uint32_t row_word(const uint8_t* p, uint32_t x, uint32_t w, const uint8_t* p0,
                                             const uint8_t* end) {
  if (x >= w) return 0u;
  const uint8_t* g = p + x;
  const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(g) & 3u), n = min(4u, w - x);
  const uint8_t* a = g - off;
  if (a >= p0 && a + 8 <= end) {
    const uint32_t* a4 = reinterpret_cast<const uint32_t*>(a);
    const uint32_t v = __byte_perm(__ldg(a4), __ldg(a4 + 1), 0x3210u + off * 0x1111u);
    return n == 4 ? v : v & ((1u << (8 * n)) - 1u);
  }
  uint32_t v = 0;
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k)
    if (k < n) v |= (uint32_t)__ldg(g + k) << (8 * k);
  return v;
}

// The template (T or T m) and, masked, the mask behind it, as rows of K bytes,
// zero past the row's w (at least 15 zeros, which are also the zeros ahead of
// the next row; sixteen more lie ahead of the first).
template <bool MASKED>
__device__ __forceinline__ void load_template(const WindowProblem& q, uint8_t* raw, uint32_t raw_bytes, uint32_t t,
                                              uint32_t nt) {
  const uint32_t words = q.K / 4, n = q.h * words;
  const uint8_t *tend = q.tpl + q.w * q.h, *mend = MASKED ? q.mask + q.w * q.h : nullptr;
  if (t < 4) {
    reinterpret_cast<uint32_t*>(raw - 16)[t] = 0u;
    if constexpr (MASKED) reinterpret_cast<uint32_t*>(raw + raw_bytes - 16)[t] = 0u;
  }
#pragma unroll 4
  for (uint32_t i = t; i < n; i += nt) {
    const uint32_t r = i / words, x = (i - r * words) * 4;
    uint32_t v = row_word(q.tpl + r * q.w, x, q.w, q.tpl, tend);
    if constexpr (MASKED) {
      const uint32_t m = row_word(q.mask + r * q.w, x, q.w, q.mask, mend);
      v &= m * 255u;  // bytes of m are 0 or 1
      reinterpret_cast<uint32_t*>(raw + raw_bytes)[i] = m;
    }
    reinterpret_cast<uint32_t*>(raw)[i] = v;
  }
}

// Adds sum T^2 of the words in shared memory (u32: at most 16384 template
// pixels) to *tss, by `nt` threads in whole warps.
__device__ __forceinline__ void add_tss(const uint8_t* raw, uint32_t words, uint32_t* tss, uint32_t t, uint32_t nt) {
  uint32_t t2 = 0;
  for (uint32_t i = t; i < words; i += nt) {
    const uint32_t v = reinterpret_cast<const uint32_t*>(raw)[i];
    t2 = __dp4a(v, v, t2);
  }
  t2 = __reduce_add_sync(0xffffffffu, t2);
  if ((t & 31u) == 0) atomicAdd(tss, t2);
}

// The 16-shift blocks of n consecutive template rows in decreasing order from
// row `top` (rows outside the template are zero): block b holds rows s = 0..15
// of K bytes, byte k = T[top - b][k - s] (0 outside the row), in the no-swizzle
// K-major layout (s / 8) (8K + 16) + (k / 16) 128 + (s % 8) 16. A thread takes
// one 16-byte chunk and eight shifts of a row: a window of 24 bytes, from
// which every shift is a fixed byte selection. The 16 bytes of padding per
// eight rows spread the stores of four blocks and both halves over all banks.
// (A lane per shift read five words per 16-byte unit: 3000 cycles for the 64
// rows of a 64 x 64 template by 20 warps, this 700.)
__device__ __forceinline__ void build_blocks(uint32_t K, uint32_t h, uint32_t top, uint32_t n, const uint8_t* raw,
                                             uint8_t* dst, uint32_t t, uint32_t nt) {
  const uint32_t cpr = K / 16, items = 8 * cpr * ((n + 3) / 4);
  for (uint32_t i = t; i < items; i += nt) {
    const uint32_t hi = i & 1u, rest = i >> 3, quad = rest / cpr, ch = rest - quad * cpr;
    const uint32_t b = 4 * quad + ((i >> 1) & 3u), d = top - b;  // wraps below row 0
    if (b >= n) continue;
    uint32_t w[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    if (d < h) {
      const uint2* src = reinterpret_cast<const uint2*>(raw + (int)(d * K + 16 * ch) - 8 * (int)hi - 8);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const uint2 v = src[k];
        w[2 * k] = v.x;
        w[2 * k + 1] = v.y;
      }
    }
    uint4* out = reinterpret_cast<uint4*>(dst + b * (16 * K + 32) + hi * (8 * K + 16) + ch * 128);
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const int o = 8 - s, f = o >> 2;  // first byte of the shift's sixteen in the window, its word
      const uint32_t sel = 0x3210u + (uint32_t)(o & 3) * 0x1111u;
      if ((o & 3) == 0)
        out[s] = make_uint4(w[f], w[f + 1], w[f + 2], w[f + 3]);
      else
        out[s] = make_uint4(__byte_perm(w[f], w[f + 1], sel), __byte_perm(w[f + 1], w[f + 2], sel),
                            __byte_perm(w[f + 2], w[f + 3], sel), __byte_perm(w[f + 3], w[f + 4], sel));
    }
  }
}

// Chunk cc of a problem: the blocks of template rows r1 - 1 down to r0 - 7 for
// its steps [r0, r1); the template's chunks first, then (masked sets that need
// window sums) the mask's.
__device__ __forceinline__ void build_chunk(const WindowProblem& q, uint32_t cc, const uint8_t* raw,
                                            uint32_t raw_bytes, uint8_t* slot, uint32_t t, uint32_t nt) {
  const uint32_t c = cc < q.nch ? cc : cc - q.nch;
  const uint32_t r0 = c * q.csteps, r1 = min(r0 + q.csteps, q.h + 7);
  build_blocks(q.K, q.h, r1 - 1, r1 - r0 + 7, cc < q.nch ? raw : raw + raw_bytes, slot, t, nt);
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

// Word of the window sum at (row, x) of the tile: odd rows have the halves of
// each 32-word run swapped, so that the sixteen lanes that read one row and
// the sixteen that read the next reach different banks.
__device__ __forceinline__ uint32_t sum_at(uint32_t row, uint32_t x) {
  return row * kTileW + (x ^ ((row & 1u) << 4));
}

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
      uint4* row = reinterpret_cast<uint4*>(ytile + sum_at(row0 + i, 8 * lane));
      row[0] = make_uint4(y0[0], y0[1], y0[2], y0[3]);
      row[1] = make_uint4(y0[4], y0[5], y0[6], y0[7]);
      if (two) {
        row = reinterpret_cast<uint4*>(ytile + sum_at(row0 + i + 1, 8 * lane));
        row[0] = make_uint4(y1[0], y1[1], y1[2], y1[3]);
        row[1] = make_uint4(y1[4], y1[5], y1[6], y1[7]);
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

// One worker warp's share of a tile's epilogue: lane quadrant `quad` (rows j =
// 2 quad and 2 quad + 1 of every group), groups g0 .. g1 - 1 of eight rows.
struct Epi {
  const WindowProblem& q;
  const Walk& w;
  uint32_t acc;  // tensor-memory address (lane quadrant, buffer)
  uint32_t j, s, lane, g0, g1, tss;  // j, s: the lane's row of a group and shift
  double td, tc;                     // TSS and -2^52 TSS
  uint32_t* ytile;
};

// Masked: the warp's window sums Y = 256 Dhi + Dlo from the accumulators at
// `lo` and `hi` into the tile.
__device__ __forceinline__ void gather_sums(const Epi& e, uint32_t lo, uint32_t hi) {
  for (uint32_t g = e.g0; g < e.g1; ++g) {
    uint32_t a[8], b[8];
    tmem_ld8(lo + 8 * g, a);
    tmem_ld8(hi + 8 * g, b);
    tmem_wait_ld();
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) e.ytile[sum_at(8 * g + e.j, 16 * c + e.s)] = a[c] + 256u * b[c];
  }
}

template <int kMethod, bool kFp64, bool kExt>
__device__ __forceinline__ void epilogue(const Epi& e) {
  constexpr bool kNeedY = kMethod != kCcorr;
  constexpr bool kFilter = method_is_norm(kMethod) && kFp64;
  const WindowProblem& q = e.q;
  const uint32_t x0 = e.w.x0 + e.s;  // the lane's first column; the others 16 further each
  const uint32_t nv = x0 < q.Wo ? min(8u, (q.Wo - x0 + 15) / 16) : 0u;  // columns inside the map
  unsigned long long kmin = ~0ull, kmax = 0ull;
  for (uint32_t g = e.g0; g < e.g1; ++g) {
    if (e.w.y0 + 8 * g >= q.Ho) break;  // the group's first row
    uint32_t x[8], yw[8];
    tmem_ld8(e.acc + 8 * g, x);
    if constexpr (kNeedY) {
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c) yw[c] = e.ytile[sum_at(8 * g + e.j, 16 * c + e.s)];
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
    const uint32_t y = e.w.y0 + 8 * g + e.j;
    const bool row_in = y < q.Ho;
    if (q.out && row_in) {
      float* o = q.out + (size_t)y * q.Wo + x0;
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c)
        if (c < nv) o[16 * c] = __uint_as_float(b[c]);
    }
    if constexpr (kExt) {
      // scores are never negative, so their f32 bits order like the values;
      // strict comparisons keep the first occurrence
      uint32_t mn = 0xFFFFFFFFu, jmn = 0, mx = 0u, jmx = 0;
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c)
        if (c < nv) {
          if (b[c] < mn) {
            mn = b[c];
            jmn = 16 * c;
          }
          if (b[c] > mx) {
            mx = b[c];
            jmx = 16 * c;
          }
        }
      if (nv && row_in) {
        const uint32_t lin = y * q.Wo + x0;
        kmin = min(kmin, ((unsigned long long)(mn | 0x80000000u) << 32) | (lin + jmn));
        kmax = max(kmax, ((unsigned long long)(mx | 0x80000000u) << 32) | (0xFFFFFFFFu - (lin + jmx)));
      }
    }
    __syncwarp();
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

// The MMAs of one chunk of steps for one image plane and one block buffer,
// issued by one thread: from step to step A moves back by one block and B down
// by one image row.
struct Chunk {
  uint32_t d, a_lo, a_hi, b_lo, b_hi, row16, K, steps, id;
  bool clear;  // the accumulator's first chunk: its first MMA overwrites
};

template <uint32_t KSTEPS>
__device__ __forceinline__ void issue_steps(const Chunk& c) {
  const uint32_t blk = c.K + 2;  // 16 K + 32 bytes per block
  uint32_t a = c.a_lo + (c.steps - 1) * blk, b = c.b_lo, acc = c.clear ? 0u : 1u;
  for (uint32_t t = 0; t < c.steps; ++t) {
#pragma unroll
    for (uint32_t kk = 0; kk < KSTEPS; ++kk) {
      mma_i8_ss(c.d, a + 16 * kk, c.a_hi, b + 2 * kk, c.b_hi, c.id, acc);
      acc = 1u;
    }
    a -= blk;
    b += c.row16;
  }
}

__device__ __forceinline__ void issue_chunk(const Chunk& c) {
  switch (c.K / 32) {
    case 1: issue_steps<1>(c); break;
    case 2: issue_steps<2>(c); break;
    case 3: issue_steps<3>(c); break;
    case 4: issue_steps<4>(c); break;
    default: issue_steps<5>(c); break;
  }
}

template <bool MASKED>
__global__ void __launch_bounds__(kThreads, 1) window_match_kernel(const __grid_constant__ WindowLaunch L) {
  extern __shared__ __align__(1024) uint8_t smem[];
  Shared* sh = reinterpret_cast<Shared*>(smem);
  // window sums of the tile; masked, in the place of its planes of I^2 (low
  // bytes, high bytes), which no MMA reads any more by then
  uint32_t* ytile = reinterpret_cast<uint32_t*>(smem + kFixed);
  uint8_t* planes = smem + kFixed;
  uint8_t* img = smem + L.img_off;
  uint8_t* bslot = smem + L.b_off;
  uint8_t* raw = smem + L.raw_off + 16;  // the template's rows
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
      mbar_init(&sh->img_full[i], kWorkWarps);
      mbar_init(&sh->img_empty[i], 1 + kWorkWarps);
      mbar_init(&sh->b_full[i], kLoadWarps);
      for (uint32_t u = 0; u < kUses; ++u) mbar_init(&sh->b_empty[i][u], 1);
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
    if (P[w.pi].load_mode == 2) load_tensor(maps + w.pi, !inl, w, img, P[w.pi].tile_bytes, &sh->img_full[0]);
  }
  if (P[w.pi].load_mode != 2) load_image(P[w.pi], w, img, tid, kThreads);
  load_template<MASKED>(P[w.pi], raw, L.raw_bytes, tid, kThreads);
  if (warp == kMmaWarp) {
    tmem_alloc(&sh->tmem, kTmemCols);
    tmem_relinquish();
  }
  __syncthreads();
  // chunks of the first tile that the slots hold at once
  const uint32_t prebuilt =
      P[w.pi].both ? 1u : min(2u, P[w.pi].nch * (MASKED && P[w.pi].need_y ? 2u : 1u));
  for (uint32_t c = 0; c < prebuilt; ++c)
    build_chunk(P[w.pi], c, raw, L.raw_bytes, bslot + c * L.slot_bytes, tid, kThreads);
  add_tss(raw, P[w.pi].h * (P[w.pi].K / 4), &sh->tss[0], tid, kThreads);
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
    // phase of each slot's last load if by a tensor copy (the first warp's)
    int last0 = P[w.pi].load_mode == 2 ? 0 : -1, last1 = -1;
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
      // one tensor copy, where the rows allow it; the workers load other
      // images. The slot's last tile is waited for either way: every phase in
      // turn, so that the parity says which.
      auto load = [&]() {
        const uint32_t use = w.ti / L.nbuf;  // earlier tiles in this slot
        if (lw) return;
        bool got = true;
        if (use) got = mbar_wait_sleep(&sh->img_empty[slot], (use - 1) & 1u, deadline);
        if (!__all_sync(0xffffffffu, got)) {
          fail = true;
          return;
        }
        (slot ? last1 : last0) = by_tensor ? (int)use : -1;
        if (by_tensor && lane == 0)
          load_tensor(maps + w.pi, !inl, w, dst, P[w.pi].tile_bytes, &sh->img_full[slot]);
        __syncwarp();
      };
      auto wait_use = [&](uint32_t s, uint32_t n) {
        return mbar_wait_sleep(&sh->b_empty[s][n % kUses], (n / kUses) & 1u, deadline);
      };
      // a wait that ran out ends the role at the next barrier, in all three
      // warps at once
      bool stop = false;
      for (uint32_t m = 0; m < w.nset && !stop; ++m, ++w.it) {
        const WindowProblem q = P[w.pi + m];
        const bool with_y = MASKED && m == 0 && need_y;
        const bool resident = bs.enter(q, with_y), first = w.it == 0;
        uint32_t* tss = &sh->tss[w.it % (2 * kRing)];
        if (m == 0 && !first && (L.nbuf == 2 || resident)) load();
        if (!first && !resident) {
          if (lt == 0) *tss = 0;
          if (m && bar_or<kLoaders>(1, fail)) {  // the last member's blocks are built
            stop = true;
            break;
          }
          load_template<MASKED>(q, raw, L.raw_bytes, lt, kLoaders);
          if (bar_or<kLoaders>(1, fail)) {
            stop = true;
            break;
          }
          add_tss(raw, q.h * (q.K / 4), tss, lt, kLoaders);
        }
        for (uint32_t c = 0; c < q.nch * (with_y ? 2u : 1u); ++c) {
          const uint32_t s = q.both ? 0u : (bs.first + c) & 1u;
          // the slots' last uses first, also where the blocks stay: every use is
          // waited for in turn, so the barriers' parities say which
          const bool in0 = !s || q.both, in1 = s || q.both;
          if (in0 && uses0 && !wait_use(0, uses0 - 1)) fail = true;
          if (in1 && uses1 && !wait_use(1, uses1 - 1)) fail = true;
          uses0 += in0;
          uses1 += in1;
          if (resident) continue;
          if (!(first && c < prebuilt)) {
            if (bar_or<kLoaders>(1, fail)) {
              stop = true;
              break;
            }
            build_chunk(q, c, raw, L.raw_bytes, bslot + s * L.slot_bytes, lt, kLoaders);
            fence_proxy_async_smem();
            __syncwarp();
          }
          if (lane == 0) mbar_arrive(&sh->b_full[s]);
          if (c == 0 && m == 0 && !first && L.nbuf == 1) load();
        }
      }
      if (stop) {
        fail = true;
        break;
      }
    }
    // no copy is in flight when the CTA leaves
    if (lw == 0) {
      const unsigned long long deadline = global_ns() + kDefaultWaitNs;
      if (last0 >= 0) mbar_wait_sleep(&sh->img_full[0], last0 & 1, deadline);
      if (last1 >= 0) mbar_wait_sleep(&sh->img_full[1], last1 & 1, deadline);
    }
  } else if (warp == kMmaWarp) {
    // ---- MMA issue
    BlockState bs;
    uint32_t builds0 = 0, builds1 = 0, uses0 = 0, uses1 = 0, ytiles = 0;
    const bool leader = elect_one();
    const uint32_t imga = smem_u32(img) >> 4, pla = smem_u32(planes) >> 4, ba = smem_u32(bslot) >> 4;
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
        const uint32_t row16 = q.pitch >> 4, id = idesc_u8u8_s32(128, 0) | ((accw >> 3) << 17);
        const uint32_t a_hi = ((q.K >> 1) + 1u) | (1u << 14);  // 8 K + 16 bytes between 8-row groups
        const uint32_t b_lo = (imga + slot * (L.plane_bytes >> 4)) | (1u << 16), b_hi = (8 * row16) | (1u << 14);
        const bool resident = bs.enter(q, with_y);
        for (uint32_t cc = 0; cc < q.nch * (with_y ? 2u : 1u) && !fail; ++cc) {
          const uint32_t s = q.both ? 0u : (bs.first + cc) & 1u, c = cc < q.nch ? cc : cc - q.nch;
          if (!resident) {
            const uint32_t builds = s ? builds1++ : builds0++;
            if (!__all_sync(0xffffffffu, mbar_wait(&sh->b_full[s], builds & 1u, deadline))) {
              fail = true;
              break;
            }
            tc_fence_after();
          }
          const uint32_t r0 = c * q.csteps, steps = min(q.csteps, q.h + 7 - r0);
          const uint32_t a_lo = (ba + s * (L.slot_bytes >> 4)) | (8u << 16);
          if (!MASKED || cc < q.nch) {
            if (leader) issue_chunk(Chunk{d, a_lo, a_hi, b_lo + r0 * row16, b_hi, row16, q.K, steps, id, c == 0});
          } else {
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
            }
            if (leader)
              for (uint32_t p = 0; p < 2; ++p)
                issue_chunk(Chunk{dy + p * accw, a_lo, a_hi,
                                  ((pla + p * (L.plane_bytes >> 4)) | (1u << 16)) + r0 * row16, b_hi, row16, q.K, steps,
                                  id, c == 0});
          }
          __syncwarp();
          if (leader) {
            if (!s || q.both) mma_commit(&sh->b_empty[0][uses0 % kUses]);
            if (s || q.both) mma_commit(&sh->b_empty[1][uses1 % kUses]);
          }
          uses0 += !s || q.both;
          uses1 += s || q.both;
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
    // beside its MMAs, then the epilogue of each of its set's members. The four
    // warps of a quarter (one per tensor-memory lane quadrant) share a quarter
    // of the tile's rows: each forms the window sums of a quarter of those,
    // then scores two rows of every group of eight (of a 16-row tile, whose two
    // groups span quarters, all warps wait for one another).
    const uint32_t quad = warp & 3, sub = warp >> 2;
    const uint32_t g0 = sub * 2 * nj / 4, g1 = (sub + 1) * 2 * nj / 4;
    const bool together = MASKED || nj == 1;
    if (P[w.pi].load_mode != 2 && lane == 0) mbar_arrive(&sh->img_full[0]);  // the first tile, loaded by all
    uint32_t tss = 0, tss_of = 0xFFFFFFFFu;  // sum (T m)^2 and the problem it is of
    for (;; ++w.ti) {
      const unsigned long long deadline = global_ns() + L.wait_ns;
      const bool more = next_tile<false>(w, L, P, sh, deadline);
      fail = __any_sync(0xffffffffu, fail || !w.ok);
      const uint32_t slot = L.nbuf == 2 ? (w.ti & 1u) : 0u;
      const bool need_y = P[w.pi].need_y;
      if (more && !fail) {
        // waited for also where nothing is read, so that no warp arrives for a
        // tile while another still reads the last one
        const bool got = mbar_wait_sleep(&sh->img_full[slot], (w.ti / L.nbuf) & 1u, deadline);
        if (!__all_sync(0xffffffffu, got)) fail = true;
        if (need_y) {
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
            window_sums_dispatch(src, q.pitch, q.w, q.h, nj * (4 * sub + quad), nj, lane, ytile);
          }
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&sh->img_empty[slot]);
          if constexpr (MASKED) mbar_arrive(&sh->planes_full);
        }
      }
      if (together ? bar_or<kWorkWarps * 32>(6, fail) : bar_or<128>(2 + sub, fail)) {
        fail = true;
        break;
      }
      if (!more) break;
      // The next tile's image, where no tensor copy takes it: by all workers
      // (three loader warps took 2.5 us longer per tile, on which the MMAs
      // waited: 60 uneven maps, 57 of them with rows on odd addresses, 1365
      // us, so 1000), once the slot is free: with one slot when the last member's MMAs
      // are done, before its epilogue, which then runs beside the next MMAs.
      auto load_next = [&]() {
        Walk nx = w;
        ++nx.ti;
        const bool have = next_tile<false>(nx, L, P, sh, deadline);
        if (!__all_sync(0xffffffffu, nx.ok)) fail = true;
        if (fail || !have || P[nx.pi].load_mode == 2) return;
        const uint32_t ns = L.nbuf == 2 ? (nx.ti & 1u) : 0u, use = nx.ti / L.nbuf;
        bool free = true;
        if (use) free = mbar_wait_sleep(&sh->img_empty[ns], (use - 1) & 1u, deadline);
        if (!__all_sync(0xffffffffu, free)) {
          fail = true;
          return;
        }
        load_image(P[nx.pi], nx, img + ns * L.plane_bytes, tid, kWorkWarps * 32);
        cp_async_wait_all();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->img_full[ns]);
      };
      for (uint32_t m = 0; m < w.nset && !fail; ++m, ++w.it) {
        const WindowProblem& q = P[w.pi + m];
        const uint32_t buf = w.it & 1u;
        // not before the last member: the loaders claim the next tile when
        // they have built the last one's blocks
        if (L.nbuf == 2 && m + 1 == w.nset) load_next();
        const bool got = mbar_wait_sleep(&sh->acc_full[buf], (w.it >> 1) & 1u, deadline);
        if (!__all_sync(0xffffffffu, got && !fail)) {
          fail = true;
          break;
        }
        tc_fence_after();
        if (L.nbuf == 1 && m + 1 == w.nset) load_next();
        // a template that follows itself may have stayed in its slots; its sum
        // is then not handed over again
        if (tss_of == 0xFFFFFFFFu || P[tss_of].tpl != q.tpl || P[tss_of].mask != q.mask || P[tss_of].w != q.w ||
            P[tss_of].h != q.h)
          tss = *reinterpret_cast<volatile uint32_t*>(&sh->tss[w.it % (2 * kRing)]);
        tss_of = w.pi + m;
        const double td = u32_to_double(tss);
        const uint32_t acc = tmem_addr(tbase, 32 * quad, 0);
        const Epi e{q, w, acc + buf * accw, 2 * quad + ((uint32_t)lane >> 4), (uint32_t)lane & 15u, (uint32_t)lane, g0, g1,
                    tss, td, -4503599627370496.0 * td, ytile};
        if constexpr (MASKED) {
          if (need_y && m == 0) {
            gather_sums(e, acc + 2 * accw, acc + 3 * accw);
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
      // the quarter's rows hold the next tile's window sums from here on (all
      // rows, its planes of I^2)
      if (together ? bar_or<kWorkWarps * 32>(6, fail) : bar_or<128>(2 + sub, fail)) {
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

// Every template of up to 128 x 128, the smallest included: SumOfSquaredErrors
// with 1 x 1, 7 x 7 and 1 x 64 templates takes 12, 12 and 12 us where the
// CUDA-core kernel takes 50, 52 and 75 (512 x 512), and 46, 48 and 58 where
// that takes 472, 492 and 797 (4096 x 3000).
bool window_supported(const MatchArgs& a) {
  if (a.precision == IPB_PRECISION_REFERENCE_F32 || (a.mask && !a.mask_binary)) return false;
  if (a.w < 1 || a.h < 1 || a.w > kMaxSide || a.h > kMaxSide || a.w > a.W || a.h > a.H) return false;
  // tile indices are 32-bit whatever the tile height
  if ((uint64_t)((a.W - a.w) / kTileW + 1) * ((a.H - a.h) / 16 + 1) >= 0xFFFF0000ull) return false;
  // the largest masked templates leave too little shared memory beside the
  // image and its planes for tiles of 64 rows: the Hankel-row kernel's
  WindowPlan pl;
  return !a.mask || window_plan_for(a.w, a.h, true, 4, 1, pl);
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
  // the template's (and mask's) rows of K bytes, sixteen zeros ahead
  pl.raw_bytes = (uint32_t)align_up((size_t)K * hmax + 16, 128);
  const uint32_t raw = pl.raw_bytes * (masked ? 2u : 1u);
  if (pl.b_off + raw >= kSmemMax) return false;
  pl.slot_bytes = (kSmemMax - pl.b_off - raw) / 2 & ~127u;
  const uint32_t block = 16 * K + 32;
  // a template needs no more than a slot of its own size; chunks of fewer than
  // eight steps would build more than they use
  pl.slot_bytes = std::min(pl.slot_bytes, (uint32_t)align_up((size_t)(hmax + 14) * block, 128));
  if (pl.slot_bytes < 15 * block) return false;
  pl.raw_off = pl.b_off + 2 * pl.slot_bytes;
  pl.smem = std::max(kMinSmem, pl.raw_off + raw);
  return pl.smem <= kSmemMax;
}

// Two image tiles where the largest template still fits the block slots beside
// them (its blocks then stay from tile to tile), else one.
bool window_plan_best(uint32_t wmax, uint32_t hmax, bool masked, uint32_t nj, WindowPlan& pl) {
  if (!masked && window_plan_for(wmax, hmax, masked, nj, 2, pl) &&
      2 * pl.slot_bytes / (16 * k_of(wmax) + 32) >= hmax + 14)
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
  // steps 0 .. h + 6 in chunks of csteps, csteps + 7 blocks each: one chunk in
  // a slot, one over both slots (it then stays, but the next template's blocks
  // wait for its last MMA), or as many as it takes
  const uint32_t block = 16 * q.K + 32, fit = pl.slot_bytes / block, steps = a.h + 7;
  q.both = steps + 7 > fit && steps + 7 <= 2 * pl.slot_bytes / block;
  q.nch = q.both ? 1u : (steps + fit - 8) / (fit - 7);
  q.csteps = (steps + q.nch - 1) / q.nch;
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

// Estimated cycles of one launch of n problems in tiles of 16 nj rows and sets
// of up to `set`: waves of tiles x (what a tile costs whatever its height, a
// set's MMAs and its epilogues) + set-up. An SS MMA of 128 x N x 32 takes
// max(32 + N/4, N/2); a tile about 2000, its epilogue about 600 per 16 output
// rows. Those two were fitted to single maps timed at every height (59 images
// of 91 x 107 to 4100 x 3000 with 21 templates of 1 to 128 a side, masked or
// not): the height of the least estimate is 0.1 % slower than the fastest on
// average, at most 1.23 times. Without the tile's own cost, small templates on
// images of more tiles than SMs were cut into tiles of 16 rows (1280 x 957, 16
// x 16, CrossCorrelationNormalized: 27 us, 128 rows 19, the Hankel-row kernel
// 24).
double window_cost(const MatchArgs* const* a, uint32_t n, uint32_t nj, uint32_t set) {
  const double sms = (double)device_sm_count(), mma = std::max(32.0 + 4.0 * nj, 8.0 * nj);
  double tiles = 0, work = 0;
  for (uint32_t i = 0; i < n; ++i) {
    const MatchArgs& q = *a[i];
    const double t = (double)(((q.W - q.w) / kTileW + 1) * (uint64_t)((q.H - q.h) / (16 * nj) + 1));
    const double corr = 1.0 + (q.mask && q.method != IPB_CROSS_CORRELATION ? 2.0 / set : 0.0);
    tiles += t / set;
    work += t * (2000.0 / set + corr * (k_of(q.w) / 32) * (q.h + 7.0) * mma + 600.0 * nj);
  }
  return work / tiles * std::ceil(tiles / sms) + 6000.0;
}

namespace {
uint32_t window_tile_nj(const MatchArgs* a, uint32_t n, uint32_t set) {
  const MatchArgs* p[kInlineProblems];
  for (uint32_t i = 0; i < n; ++i) p[i] = a + i;
  uint32_t best = 8;
  for (uint32_t nj : {4u, 2u, 1u})
    if (window_cost(p, n, nj, set) < window_cost(p, n, best, set)) best = nj;
  return best;
}
}  // namespace

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
  for (uint32_t nj = window_tile_nj(a, n, set); nj >= 1 && !have; nj /= 2)
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
