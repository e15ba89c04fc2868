// gslice.cu -- the FP64 form's temporal-gauge loop stage (gram.cu's identities
// and slab layout) with the banded Gram product on the tensor cores, exactly:
// the lines are written as signed 8-bit digits and multiplied by tcgen05.mma
// of kind::i8 with 32-bit integer accumulation.
//
//     x = sum_p q_p 2^(-6-8p),  q_p in [-128, 127],  p < 7
//
// (x rounded to 2^-54; |x| < 1.99).  A line entry is bounded by the product of
// the operator norms it is made of, so that
//     (1 + c delta)^(R/2) / (1 - c dev) <= 1.98,  c = 1 + 2 sqrt 2
// (delta, dev: largest real or imaginary part of U^dag U - 1 over the stored
// levels and of g g^dag - 1 over the gauge field; c times it bounds the norm)
// admits a lattice.  Where spatial links are too far from
// unitary for it (spatial HYP leaves such links), a walk that stores nothing
// finds the largest entry and the least norm of a slice per extent and level, and
// the lines of each extent and level are scaled by 2^-e for the smallest e <= 3
// that holds them, unless their norm is so far below it that FP64 FMAs would be
// nearer (slice_scales; 32 x 20^3, msl 4, three levels of spatial HYP: 10.4 ms a
// measurement with the walk and the digits, 11.8 with the FMA kernel).  The FMA kernel of
// gram.cu measures the rest, and a NaN anywhere fails every comparison.  A dot
// product is then
//     sum_c a_c b_c = sum_m 2^(-12-8m) C_m,   C_m = sum_{i+j=m} q_a,i . q_b,j
// over the classes m < 7.  The classes that are left out and the rounding of x
// are absolute errors of 4.5e-17 a column (of lines scaled to the digits' range) that
// add up as random ones: of W, a mean over 9 N1 N2 N3, about 3.7e-17 / sqrt(N1 N2 N3)
// times the lines' 2^(e1 + e2), whatever W is (emulated: 4.5e-18 at 4^3, 3.8e-19 at 20^3).
// The integer sums are exact, so a result does not depend on how columns are
// split over blocks or in which order blocks add theirs.  FP64 FMAs of the same
// lines are 2.4e-18 .. 2.4e-17 off where W is small, more where it is not.  Against
// 64-bit loops of the same fields W is 1.3e-16 .. 4.9e-16 off (2-norm, lines included)
// where the FMA kernel's sums are 4.1e-16 .. 6.5e-16 off.
//
// The mixed form keeps FP32 FMAs (gpair.cu): its sums' rounding is part of its
// results.
//
// Work is cut into chunks of column units (a unit: one direction, one 32-site
// tile).  Per chunk k_slice_lines walks the lines of its units through all
// spatial extents R = 1..mwlr in registers and writes the digit planes of
// every R; k_slice_gram then forms all R's sums of the chunk.  The first
// lines and the recursion links are read from HBM once per measurement
// (per R before), and the chunk bounds the memory the planes take.
//
// Plane layout, one buffer for the A rows (start slice, level) and one for the
// B rows (unrolled slice, level), row = slice * L + level: per (R, unit, row)
// 4096 bytes that hold the 7 x 576 digits of one 32-site tile as 9 K blocks of
// 64 columns, planes 0 .. 5 in pairs so that an operand row is a whole 128-byte
// line (TMA moves about one row in 2.4 cycles, of 64 or of 128 bytes):
//     plane p < 6 of block b at  b * 384 + (p / 2) * 128 + (p % 2) * 64
//     plane 6 of block b at      3456 + b * 64
// Block b < 8 holds the first 16 components of lanes 4 b .. 4 b + 3 and block
// 8 the last two components of all lanes (the columns of a sum may come in any
// order): a lane writes 16 bytes and 2 bytes per plane at offsets the compiler
// knows, a warp one contiguous row.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <set>
#include <utility>

#include "internal.h"
#include "mbar.cuh"
#include "slab.cuh"
#include "tensormap.h"

namespace wlg {
namespace {

constexpr int kPlanes = 7;
constexpr int kKB = 64;       // bytes (columns) per K block
constexpr int kRow = 4096;    // bytes of one row of planes
constexpr int kSingle = 9 * 6 * kKB;  // where plane 6 starts in it
constexpr int kMaxStages = 8;
constexpr int kGramThreads = 192;  // producer warp, MMA warp, four epilogue warps

// ---------------------------------------------------------------------------
// digits
// ---------------------------------------------------------------------------
// Two roundings by magic addition: t1 = x + 1.5 2^22 rounds x to 2^-30, its low
// word is round(x 2^30); the remainder (at most 2^-31) plus 0.375, exact up to
// the one rounding to 2^-54, holds the rest in its low word.  The low part may
// round up to 2^23, its carry goes into the high part.  Bytes below the top one
// carry a bias of 128, taken off by the flip of their top bit.
struct Digits {
  unsigned hi, lo;
  __device__ explicit __forceinline__ Digits(double x) {
    constexpr double M1 = 6291456.0;  // 1.5 * 2^22: unit in the last place 2^-30
    const double t1 = x + M1;
    const double t2 = x - (t1 - (M1 + 0.375));  // unit in the last place 2^-54
    lo = (unsigned)__double2loint(t2) + 0x00808080u;
    hi = (unsigned)__double2loint(t1) + ((int)lo >> 24) + 0x00808080u;
  }
  static constexpr unsigned flip(int p) { return p == 0 ? 0u : 0x80808080u; }
};

// the digits of one complex number: planes 0|1, 2|3, 4|5 as the low and high
// halves of a word (two bytes: real, imaginary), plane 6 as a low half
__device__ __forceinline__ void digits_of(unsigned (&w)[4], double2 v) {
  const Digits a(v.x), b(v.y);
  w[0] = __byte_perm(a.hi, b.hi, 0x6273);
  w[1] = __byte_perm(a.hi, b.hi, 0x4051);
  w[2] = __byte_perm(a.lo, b.lo, 0x5162);
  w[3] = __byte_perm(a.lo, b.lo, 0x0040);
}

// where plane p starts in a lane's 16-byte (o6 for plane 6: o16) column
__device__ constexpr int plane_at(int p) { return (p >> 1) * 128 + (p & 1) * kKB; }

template <bool SCALED> __device__ __forceinline__ double2 scaled(double2 v, double s) {
  return SCALED ? make_double2(v.x * s, v.y * s) : v;  // s a power of two
}

// the digit planes of one matrix into its row (this lane's 16 + 2 bytes per
// plane)
template <bool SCALED>
__device__ __forceinline__ void store_digits(unsigned char* __restrict__ row, int lane,
                                             const M3<double>& m, double scale) {
  constexpr int P = kPlanes;
  uint4 q[P];
#pragma unroll
  for (int h = 0; h < 4; h++) {
    unsigned w0[4], w1[4];
    digits_of(w0, scaled<SCALED>(m.e[2 * h], scale));
    digits_of(w1, scaled<SCALED>(m.e[2 * h + 1], scale));
#pragma unroll
    for (int p = 0; p < P; p++) {
      const unsigned v =
          __byte_perm(w0[p >> 1], w1[p >> 1], p & 1 ? 0x7632 : 0x5410) ^ Digits::flip(p);
      if (h == 0) q[p].x = v;
      if (h == 1) q[p].y = v;
      if (h == 2) q[p].z = v;
      if (h == 3) q[p].w = v;
    }
  }
  unsigned w[4];
  digits_of(w, scaled<SCALED>(m.e[8], scale));
  unsigned char* o16 = row + (lane >> 2) * (6 * kKB) + (lane & 3) * 16;
  unsigned char* s16 = row + kSingle + lane * 16;
  unsigned char* o2 = row + 8 * 6 * kKB + lane * 2;
  unsigned char* s2 = row + kSingle + 8 * kKB + lane * 2;
#pragma unroll
  for (int p = 0; p < P; p++) {
    *reinterpret_cast<uint4*>(p < 6 ? o16 + plane_at(p) : s16) = q[p];
    const unsigned v = w[p >> 1] ^ (p < 2 ? 0x80800000u : 0x80808080u);
    *reinterpret_cast<unsigned short*>(p < 6 ? o2 + plane_at(p) : s2) =
        (unsigned short)(p & 1 ? v >> 16 : v);
  }
}

// tile of unit index v (0 <= v < ntile) for direction k: for k = 0 the tiles
// along the x1 line are consecutive, so that the shifted links a chunk reads
// are those of its own units (k = 1, 2: the lexicographic order has that)
__device__ __forceinline__ int unit_tile(const Geo& g, int ntile, int k, int v) {
  if (k != 0) return v;
  const int tp = max(1, min(ntile, (g.st[1] + 16) >> 5));  // tiles per x1 plane, rounded
  const int q = ntile / tp, rem = ntile - q * tp;
  // column m holds tiles m, m + tp, ...: q + 1 of them for m < rem, else q
  if (v < rem * (q + 1)) return v / (q + 1) + (v % (q + 1)) * tp;
  const int w = v - rem * (q + 1);
  return rem + w / q + (w % q) * tp;
}

struct LineArgs {
  Geo g;
  int Nu, ntile, msl, mwlr, u0, cur, nuc;
  size_t A;  // elements of one slab array
  const double *uh, *bl, *hinv;
  unsigned char *sa, *sb;
  const double* scale;        // [extent][level] (WALK_SCALED)
  unsigned long long* range;  // see slice_range_bytes (WALK_RANGE)
};
enum { WALK_PLAIN, WALK_SCALED, WALK_RANGE };

// this warp's share of one extent's range: the largest entry (its high word, for
// NaN and infinity above every finite one) and the sum of squares in units of
// 2^-30, as integers so that their order does not matter
__device__ __forceinline__ void add_range(unsigned long long* top, unsigned long long* sum,
                                          const M3<double>& m, bool live, int lane) {
  unsigned hi = 0;
  double sq = 0.0;
#pragma unroll
  for (int e = 0; e < 9; e++) {
    hi = max(hi, max((unsigned)__double2hiint(m.e[e].x) & 0x7fffffffu,
                     (unsigned)__double2hiint(m.e[e].y) & 0x7fffffffu));
    sq = fma(m.e[e].x, m.e[e].x, fma(m.e[e].y, m.e[e].y, sq));
  }
  hi = __reduce_max_sync(0xffffffffu, live ? hi : 0u);
  if (!live) sq = 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  if (lane == 0) {
    if (hi > *(volatile unsigned long long*)top) atomicMax(top, (unsigned long long)hi);
    // (at most 2^18 where every entry fits the largest exponent)
    atomicAdd(sum, (unsigned long long)(fmin(sq, 0x1p18) * 0x1p30));
  }
}

// B(x, R) and A(x, R) = H^-1(x) B(x, R) H^-1(x + R k) for R = 1..mwlr, as
// digit planes.  One warp per (y0, unit, level), levels in neighbouring warps
// (they share the H^-1 tiles), the walk over R in registers.
//
// Bound by the writes, 4 KB a matrix: 184 GB and 41-42 ms a measurement at
// 32^3 x 64 (4.4 TB/s, clocks and bandwidth shared with the Gram product under the
// power limit).  Neither fewer loads (H^-1(x) B kept in registers), prefetches,
// streaming stores nor 2 or 4 blocks per SM change it by more than 2 %; three
// roundings a real instead of four, and no selects, took 3 %.
template <int WALK>
__global__ void __launch_bounds__(128, 3) k_slice_lines(LineArgs a) {
  const int lane = threadIdx.x & 31;
  unsigned w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lev = (int)(w % a.msl);
  w /= a.msl;
  const int ul = (int)(w % a.cur);
  const int y0 = (int)(w / a.cur);
  if (y0 >= a.Nu) return;
  const Geo& g = a.g;
  const int u = a.u0 + ul, k = u / a.ntile;
  const int jt = unit_tile(g, a.ntile, k, u - k * a.ntile);
  const bool live = jt * 32 + lane < g.vs;
  const int j = live ? jt * 32 + lane : g.vs - 1;
  const bool start = y0 < g.n[0];
  // slices of this y0: the recursion links of (level, k), and H^-1
  const size_t slice = (size_t)y0 * a.ntile * kSlabTile;
  const double* uh = a.uh + (size_t)(lev * 3 + k) * a.A + slice;
  const double* hinv = a.hinv + slice;
  const int nk = k == 0 ? g.n[1] : (k == 1 ? g.n[2] : g.n[3]);
  const int st = k == 0 ? g.st[1] : (k == 1 ? g.st[2] : 1);
  int z = j, y = (j / st) % nk;  // x + (R - 1) k and its coordinate along k
  const size_t rows_a = (size_t)g.n[0] * a.msl, rows_b = (size_t)a.Nu * a.msl;
  const int row = y0 * a.msl + lev;
  unsigned char* ob = a.sb + (ul * rows_b + row) * kRow;
  unsigned char* oa = a.sa + (ul * rows_a + row) * kRow;
  const size_t step_b = a.nuc * rows_b * kRow, step_a = a.nuc * rows_a * kRow;
  M3<double> c, f, t;
  ld_slab_as(c, a.bl + (size_t)(lev * 3 + k) * a.A + slice, j >> 5, j & 31);
  if (!live) {  // zero digits in a tile's lanes without a site
#pragma unroll
    for (int e = 0; e < 9; e++) c.e[e] = make_double2(0.0, 0.0);
  }
#pragma unroll 1
  for (int R = 1; R <= a.mwlr; R++) {
    if (R > 1) {
      ld_slab_as(f, uh, z >> 5, z & 31);
      mul(t, c, f);
      c = t;
    }
    z += st;
    if (++y == nk) {
      y = 0;
      z -= nk * st;
    }
    const int el = (R - 1) * a.msl + lev;
    const double scale = WALK == WALK_SCALED ? __ldg(a.scale + el) : 1.0;
    unsigned long long* sums = a.range + (size_t)a.mwlr * a.msl + (size_t)el * 2 * a.Nu + y0;
    if constexpr (WALK == WALK_RANGE)
      add_range(a.range + el, sums, c, live, lane);
    else
      store_digits<WALK == WALK_SCALED>(ob, lane, c, scale);
    if (start) {
      ld_slab_as(f, hinv, z >> 5, z & 31);
      mul(t, c, f);
      ld_slab_as(f, hinv, j >> 5, j & 31);
      M3<double> s;
      mul(s, f, t);
      if constexpr (WALK == WALK_RANGE)
        add_range(a.range + el, sums + a.Nu, s, live, lane);
      else
        store_digits<WALK == WALK_SCALED>(oa, lane, s, scale);
    }
    ob += step_b;
    oa += step_a;
  }
}

// ---------------------------------------------------------------------------
// The banded Gram product of one chunk.  A work item is (R, column split,
// tile); a tile is 128 A rows against TN of the B rows their band reaches.
// One CTA per SM walks items; per 64-column block the producer thread fetches
// the digit rows of both operands with four TMA boxes, the MMA thread issues
// the digit pairs i + j < 7, one A plane with up to three B planes per MMA
// (their accumulators, the classes i + j, are neighbours in TMEM), and the
// epilogue warps read the classes, combine them as 64-bit integers and add the
// entries inside the band to the result with integer atomics.  At 32^3x64 the
// tensor pipe is 77 % busy (85 % with its set-up) at the 1.66 GHz the power
// limit leaves: 70 ms a measurement; 84 ms with one 64-byte row per plane and
// descriptors worked out by the issuing thread, 102 ms with a ring of single A
// planes (two more blocks in flight, but seven boxes a block).  Every wait is bounded: one that
// runs out sets *fail, and all roles leave.
// ---------------------------------------------------------------------------
struct GramTileArgs {
  int N0, Nu, L, mwlt, mwlr;
  int rows_a, rows_b, TN, nmt, ntiles;
  int kstride;  // K blocks of one R in the plane buffers
  int kcur;     // K blocks of one R in this chunk
  int kps, nsplit, stages;
  unsigned tmem_cols;
  long long nwl;
  unsigned long long* acc;  // [2][nwl]: 2^24 times the first plus the second
  int* fail;
};

struct TileAt {
  int r, kb0, nkb, m0, b0;
};

// B rows a 128-row A tile reaches: [first, last)
__host__ __device__ __forceinline__ void band_rows(int L, int mwlt, int rows_a, int rows_b, int m0,
                                                   int& first, int& last) {
  const int m1 = m0 + 127 < rows_a ? m0 + 127 : rows_a - 1;
  first = (m0 / L + 1) * L;
  last = (m1 / L + mwlt + 1) * L;
  if (last > rows_b) last = rows_b;
  if (first > last) first = last;
}

__device__ __forceinline__ TileAt tile_at(const GramTileArgs& a, long long it) {
  TileAt t;
  int tile = (int)(it % a.ntiles);
  it /= a.ntiles;
  const int sp = (int)(it % a.nsplit);
  t.r = (int)(it / a.nsplit);
  t.kb0 = t.r * a.kstride + sp * a.kps;
  t.nkb = min(a.kps, a.kcur - sp * a.kps);
  t.m0 = t.b0 = 0;
  for (int m = 0; m < a.nmt; m++) {
    int first, last;
    band_rows(a.L, a.mwlt, a.rows_a, a.rows_b, m * 128, first, last);
    const int n = (last - first + a.TN - 1) / a.TN;
    if (tile < n) {
      t.m0 = m * 128;
      t.b0 = first + tile * a.TN;
      break;
    }
    tile -= n;
  }
  return t;
}

__device__ __forceinline__ void tma_pairs(unsigned dst, const CUtensorMap* map, int row, int b,
                                          int u, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %2, %4, %5}], [%6];\n" ::"r"(dst),
      "l"(map), "r"(0), "r"(row), "r"(b), "r"(u), "r"(smem_addr(bar))
      : "memory");
}
__device__ __forceinline__ void tma_single(unsigned dst, const CUtensorMap* map, int row, int b,
                                           int u, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(dst),
      "l"(map), "r"(0), "r"(row), "r"(b), "r"(u), "r"(smem_addr(bar))
      : "memory");
}

// K-major shared-memory operands: 8-row groups of 1024 bytes with 128-byte
// swizzle (plane pairs), of 512 bytes with 64-byte swizzle (plane 6)
__device__ __forceinline__ uint64_t pair_desc(unsigned addr) {
  return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ uint64_t single_desc(unsigned addr) {
  return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
// TMEM column (in units of TN) of class m: the even classes, then the odd ones,
// so that the classes of one A plane and B planes j, j + 2, ... are neighbours
__host__ __device__ constexpr int class_col(int m) { return (m & 1) ? 4 + m / 2 : m / 2; }

__device__ __forceinline__ void mma_i8(unsigned d, uint64_t da, uint64_t db, unsigned idesc,
                                       bool accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(da), "l"(db), "r"(idesc), "r"((unsigned)accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                   smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_ld16(int (&v)[16], unsigned addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(addr));
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

template <int TN>
__global__ void __launch_bounds__(kGramThreads, 1)
    k_slice_gram(const __grid_constant__ CUtensorMap map_a2, const __grid_constant__ CUtensorMap map_a1,
                 const __grid_constant__ CUtensorMap map_b2, const __grid_constant__ CUtensorMap map_b1,
                 const GramTileArgs a) {
  constexpr int P = kPlanes;
  extern __shared__ unsigned char raw[];
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], acc_full, acc_empty, drain;
  __shared__ unsigned tmem_base;
  __shared__ int quit;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned base = (smem_addr(raw) + 1023u) & ~1023u;
  // a stage: A pairs, B pairs, A plane 6, B plane 6
  constexpr unsigned at_b2 = 3 * 128 * 128, at_a1 = at_b2 + 3 * TN * 128, at_b1 = at_a1 + 128 * kKB;
  constexpr unsigned stage_bytes = at_b1 + TN * kKB;
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; s++) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    mbar_init(&acc_full, 1);
    mbar_init(&acc_empty, 4);
    mbar_init(&drain, 1);
    mbar_init_fence();
    quit = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_addr(&tmem_base)),
                 "r"(a.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tmem_base;
  const long long items = (long long)a.mwlr * a.nsplit * a.ntiles;

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      unsigned ph = 0;
      long long issued = 0;
      bool ok = true;
      for (long long it = blockIdx.x; ok && it < items; it += gridDim.x) {
        const TileAt t = tile_at(a, it);
        for (int kb = 0; kb < t.nkb; kb++) {
          if (!(ok = wait_or_quit(empty + s, ph ^ 1, &quit))) break;
          const unsigned dst = base + s * stage_bytes;
          mbar_expect_tx(full + s, stage_bytes);
          const int un = (t.kb0 + kb) / 9, bl = t.kb0 + kb - un * 9;
          tma_pairs(dst, &map_a2, t.m0, bl, un, full + s);
          tma_pairs(dst + at_b2, &map_b2, t.b0, bl, un, full + s);
          tma_single(dst + at_a1, &map_a1, t.m0, bl, un, full + s);
          tma_single(dst + at_b1, &map_b1, t.b0, bl, un, full + s);
          issued++;
          if (++s == a.stages) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      if (!ok) {
        // the copies in flight, the last use of each stage
        for (long long b = issued > a.stages ? issued - a.stages : 0; b < issued; b++)
          mbar_wait_bounded(full + b % a.stages, (unsigned)((b / a.stages) & 1));
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int s = 0;
      unsigned ph = 0, aph = 0;
      bool ok = true;
      constexpr unsigned idesc0 =
          (2u << 4) | (1u << 7) | (1u << 10) | (8u << 24);  // S32, S8 x S8, M 128
      for (long long it = blockIdx.x; ok && it < items; it += gridDim.x) {
        const TileAt t = tile_at(a, it);
        if (t.nkb <= 0) continue;
        if (!(ok = wait_or_quit(&acc_empty, aph ^ 1, &quit))) break;
        tc_fence_after();
        for (int kb = 0; ok && kb < t.nkb; kb++) {
          if (!(ok = wait_or_quit(full + s, ph, &quit))) break;
          tc_fence_after();
          const unsigned sa = base + s * stage_bytes;
          const uint64_t a2 = pair_desc(sa), b2 = pair_desc(sa + at_b2);
          const uint64_t a1 = single_desc(sa + at_a1), b1 = single_desc(sa + at_b1);
          // everything but the base addresses is known here: one thread issues
          // all MMAs of the block.  A plane i against the B planes of one
          // parity, j + i < 7, which lie one below the other: one MMA of up to
          // 3 TN columns; plane 6 only meets plane 0.
#pragma unroll
          for (int ks = 0; ks < kKB / 32; ks++)
#pragma unroll
            for (int i = 0; i < P; i++) {
              const bool acc = kb > 0 || ks > 0 || i > 0;
              const uint64_t da = i < 6 ? a2 + (uint64_t)(((i >> 1) * 128 * 128 + (i & 1) * kKB + ks * 32) >> 4)
                                        : a1 + (uint64_t)(ks * 32 >> 4);
#pragma unroll
              for (int h = 0; h < 2; h++) {
                const int last = i == 0 ? 5 : 6 - i;
                const int n = last < h ? 0 : (last - h) / 2 + 1;
                if (n > 0)
                  mma_i8(tmem + (unsigned)(class_col(i + h) * TN), da,
                         b2 + (uint64_t)((h * kKB + ks * 32) >> 4),
                         idesc0 | ((unsigned)(n * TN >> 3) << 17), acc);
              }
              if (i == 0)
                mma_i8(tmem + (unsigned)(class_col(6) * TN), da, b1 + (uint64_t)(ks * 32 >> 4),
                       idesc0 | ((unsigned)(TN >> 3) << 17), acc);
            }
          mma_commit(empty + s);
          if (++s == a.stages) {
            s = 0;
            ph ^= 1;
          }
        }
        if (!ok) break;
        mma_commit(&acc_full);
        aph ^= 1;
      }
      if (!ok) {  // the MMAs in flight
        mma_commit(&drain);
        mbar_wait_bounded(&drain, 0);
      }
    }
  } else {
    const int quad = warp & 3;
    unsigned ph = 0;
    for (long long it = blockIdx.x; it < items; it += gridDim.x) {
      const TileAt t = tile_at(a, it);
      if (t.nkb <= 0) continue;
      if (!__all_sync(0xffffffffu, wait_or_quit(&acc_full, ph, &quit))) break;
      tc_fence_after();
      ph ^= 1;
      const int r0 = t.m0 + quad * 32;
      if (r0 < a.rows_a) {
        const int row = r0 + lane, x0 = row / a.L, s1 = row - x0 * a.L;
        // the columns any row of this warp needs
        const int lo = max(0, (r0 / a.L + 1) * a.L - t.b0);
        const int hi = min(min(TN, a.rows_b - t.b0),
                           (min(r0 + 31, a.rows_a - 1) / a.L + a.mwlt + 1) * a.L - t.b0);
        const bool live = row < a.rows_a;
        for (int c0 = lo & ~15; c0 < hi; c0 += 16) {
          int v[P][16];
#pragma unroll
          for (int m = 0; m < P; m++)
            tmem_ld16(v[m], tmem + ((unsigned)(quad * 32) << 16) + (unsigned)(class_col(m) * TN + c0));
          tmem_ld_wait();
          int e = (t.b0 + c0) / a.L, s2 = t.b0 + c0 - e * a.L;
#pragma unroll
          for (int c = 0; c < 16; c++) {
            const int T = e - x0;
            if (live && c0 + c < hi && T >= 1 && T <= a.mwlt) {
              const long long o =
                  s1 + (long long)a.L * (s2 + (long long)a.L *
                                                  ((T - 1) + (long long)a.mwlt *
                                                                 (t.r + (long long)a.mwlr * x0)));
              const long long zh = ((long long)v[0][c] << 24) + ((long long)v[1][c] << 16) +
                                   ((long long)v[2][c] << 8) + v[3][c];
              const long long zl = ((long long)v[4][c] << 16) + ((long long)v[5][c] << 8) + v[6][c];
              atomicAdd(a.acc + o, (unsigned long long)zh);
              atomicAdd(a.acc + a.nwl + o, (unsigned long long)zl);
            }
            if (++s2 == a.L) {
              s2 = 0;
              e++;
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && quit) atomicExch(a.fail, 1);
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem),
                 "r"(a.tmem_cols));
}

// wl = the integer sums scaled; loops through the last slice of open time are
// exact zeros
__global__ void __launch_bounds__(256) k_slice_finish(const long long* __restrict__ acc,
                                                      long long nwl, int N0, int mwlt, int mwlr,
                                                      int L, int open, double norm,
                                                      const double* __restrict__ scale,
                                                      double* __restrict__ wl) {
  for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < nwl;
       o += (long long)gridDim.x * blockDim.x) {
    const int s1 = (int)(o % L), s2 = (int)((o / L) % L), t = (int)((o / (L * L)) % mwlt);
    const int r = (int)((o / ((long long)L * L * mwlt)) % mwlr);
    const int x0 = (int)(o / ((long long)L * L * mwlt * mwlr));
    double v = 0.0;
    if (!open || x0 + t + 1 < N0) {
      const double both =
          scale ? 1.0 / (__ldg(scale + r * L + s1) * __ldg(scale + r * L + s2)) : 1.0;
      v = fma((double)acc[o], 0x1p-36 * both, (double)acc[nwl + o] * (0x1p-60 * both)) / norm;
    }
    wl[o] = v;
  }
}

// largest real or imaginary part of U^dag U - 1 over the stored levels, as the bits
// of a non-negative double (a NaN counts as the largest value)
__global__ void __launch_bounds__(256) k_levels_dev(const double2* __restrict__ lev,
                                                    size_t stride, int narr, int vol,
                                                    unsigned long long* __restrict__ dev) {
  double worst = 0.0;
  const long long n = (long long)narr * vol;
  for (long long w = blockIdx.x * (long long)blockDim.x + threadIdx.x; w < n;
       w += (long long)gridDim.x * blockDim.x) {
    const int q = (int)(w / vol), s = (int)(w - (long long)q * vol);
    M3<double> u;
    ld<double>(u, lev + q * stride, vol, s);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = i; j < 3; j++) {
        double re = i == j ? -1.0 : 0.0, im = 0.0;
#pragma unroll
        for (int m = 0; m < 3; m++) {
          const double2 a = u.e[3 * m + i], b = u.e[3 * m + j];
          re = fma(a.x, b.x, fma(a.y, b.y, re));
          im = fma(a.x, b.y, fma(-a.y, b.x, im));
        }
        re = fabs(re);
        im = fabs(im);
        if (re > worst || re != re) worst = re;  // a NaN sticks
        if (im > worst || im != im) worst = im;
      }
  }
  double d = worst != worst ? 1e300 : worst;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) d = fmax(d, __shfl_xor_sync(0xffffffffu, d, o));
  if ((threadIdx.x & 31) == 0) atomicMax(dev, (unsigned long long)__double_as_longlong(d));
}

constexpr size_t kSmemMax = 227 * 1024 - 1024;  // beside the barriers and the alignment slack
// K blocks one 32-bit accumulation takes: the last class adds P products of
// at most 2^14 a column, 64 columns a block
constexpr int kRunMax = (int)((1ll << 31) / ((long long)kPlanes * (1 << 14) * kKB)) - 1;

// plane pairs as a tensor of (128 bytes, rows, pairs, blocks, (R, unit)), plane 6
// as one of (64 bytes, rows, blocks, (R, unit)); a box is `box` rows of one block
bool plane_maps(CUtensorMap* pairs, CUtensorMap* single, unsigned char* base, int rows,
                long long units, int box) {
  TensorMapEncode fn = tensor_map_encode();
  if (!fn) return false;
  const cuuint64_t all = (cuuint64_t)kRow * rows;
  const cuuint32_t one[5] = {1, 1, 1, 1, 1};
  const cuuint64_t dim2[5] = {2 * kKB, (cuuint64_t)rows, 3, 9, (cuuint64_t)units};
  const cuuint64_t str2[4] = {kRow, 2 * kKB, 6 * kKB, all};
  const cuuint32_t box2[5] = {2 * kKB, (cuuint32_t)box, 3, 1, 1};
  const cuuint64_t dim1[4] = {kKB, (cuuint64_t)rows, 9, (cuuint64_t)units};
  const cuuint64_t str1[3] = {kRow, kKB, all};
  const cuuint32_t box1[4] = {kKB, (cuuint32_t)box, 1, 1};
  return fn(pairs, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, base, dim2, str2, box2, one,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS &&
         fn(single, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, base + kSingle, dim1, str1, box1, one,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

static void* slice_kernel(int TN) {
  switch (TN) {
    case 16: return (void*)k_slice_gram<16>;
    case 32: return (void*)k_slice_gram<32>;
    case 48: return (void*)k_slice_gram<48>;
    default: return (void*)k_slice_gram<64>;
  }
}

bool slice_plan(SlicePlan& p, const Geo& g, int bc, int msl, int mwlt, int mwlr,
                size_t budget) {
  p = SlicePlan();
  // the 64-bit sums hold 70 x 3 N1 N2 N3 products of 2^36
  if (msl < 1 || msl > 8 || mwlt < 1 || mwlr < 1 || g.vs > 600000) return false;
  p.L = msl;
  p.N0 = g.n[0];
  p.Nu = g.n[0] + (bc == 0 ? 0 : mwlt);
  p.mwlt = mwlt;
  p.mwlr = mwlr;
  p.ntile = (g.vs + 31) / 32;
  p.rows_a = p.N0 * msl;
  p.rows_b = p.Nu * msl;
  p.nmt = (p.rows_a + 127) / 128;
  // B rows per tile: the band of a 128-row tile in the fewest equal tiles
  // whose P classes fit the 512 TMEM columns
  constexpr int nmax = (512 / kPlanes) & ~15;
  int widest = 0;
  for (int m = 0; m < p.nmt; m++) {
    int first, last;
    band_rows(msl, mwlt, p.rows_a, p.rows_b, m * 128, first, last);
    widest = std::max(widest, last - first);
  }
  if (widest == 0) return false;
  const int parts = (widest + nmax - 1) / nmax;
  p.TN = (((widest + parts - 1) / parts) + 15) & ~15;
  for (int m = 0; m < p.nmt; m++) {
    int first, last;
    band_rows(msl, mwlt, p.rows_a, p.rows_b, m * 128, first, last);
    p.ntiles += (last - first + p.TN - 1) / p.TN;
  }
  const size_t stage = (size_t)kPlanes * kKB * (128 + p.TN);
  p.stages = (int)std::min<size_t>(kMaxStages, (kSmemMax - 1024) / stage);
  if (p.stages < 2) return false;
  // more than half of an SM's shared memory: one CTA, one TMEM owner per SM
  p.smem = std::max<size_t>(p.stages * stage + 1024, 116 * 1024);
  p.tmem_cols = 32;
  while (p.tmem_cols < kPlanes * p.TN) p.tmem_cols *= 2;
  // column units per chunk: as many as the budget holds, in equal chunks
  const int units = 3 * p.ntile;
  const size_t unit = (size_t)mwlr * kRow * (p.rows_a + p.rows_b);
  long long nuc = (long long)(budget / unit);
  if (nuc < 1) return false;
  if (nuc > units) nuc = units;
  p.nchunk = (int)((units + nuc - 1) / nuc);
  p.nuc = (units + p.nchunk - 1) / p.nchunk;
  p.nchunk = (units + p.nuc - 1) / p.nuc;
  p.bytes_a = (size_t)mwlr * p.nuc * p.rows_a * kRow;
  p.bytes_b = (size_t)mwlr * p.nuc * p.rows_b * kRow;
  p.nwl = (size_t)msl * msl * mwlt * mwlr * p.N0;
  p.acc_bytes = p.nwl * 2 * sizeof(unsigned long long);
  // column splits: enough for the 32-bit range, then the fewest waves of the
  // SMs, an item costing its K blocks and about 6 more for its epilogue
  const int kc = p.nuc * 9, lo = (kc + kRunMax - 1) / kRunMax;
  const long long per = (long long)mwlr * p.ntiles;
  double best = 1e300;
  for (int ns = lo; ns <= std::min(kc, std::max(lo, lo * 16 + 160)); ns++) {
    const int kps = (kc + ns - 1) / ns;
    const long long items = per * ((kc + kps - 1) / kps);
    const double cost = (double)((items + num_sms() - 1) / num_sms()) * (kps + 6);
    if (cost < best * 0.999) {
      best = cost;
      p.kps = kps;
      p.nsplit = (kc + kps - 1) / kps;
    }
  }
  return true;
}

// Lines whose digits' unit is 2^-54 c (c: 2^e over the lines' norm) make sums 9 c^2 /
// sqrt(run + runs) times as far off as FP64 FMAs of `run` columns each, `runs` of
// them added up: 0.04 to 0.33 at c = 1 for the plans of 32768 sites and more. The
// largest c^2 that keeps the digits ahead, and 1.1 for the lines of SU(3) links.
static double most_spread(int run, int runs) {
  return std::max(1.1, 0.08 * std::sqrt((double)run + runs));
}

bool slice_in_range(double dev, double delta, int mwlr, int run, int runs) {
  // a Hermitian matrix whose entries' real and imaginary parts are at most d has a
  // norm of at most its largest row sum, (1 + 2 sqrt 2) d
  constexpr double row = 3.8284271247461903;
  const double s = row * delta, h = row * dev;
  if (!(s < 1.0) || !(h < 1.0)) return false;
  const double least = std::pow(1.0 - s, 0.5 * mwlr) * (1.0 - h);  // norm of a line
  return std::pow(1.0 + s, 0.5 * mwlr) / (1.0 - h) <= 1.98 &&
         1.0 <= most_spread(run, runs) * least * least;
}

size_t slice_range_bytes(const SlicePlan& p) {
  return (size_t)p.mwlr * p.L * (1 + 2 * (size_t)p.Nu) * sizeof(unsigned long long);
}

bool slice_scales(const Geo& g, const SlicePlan& p, int run, int runs,
                  const unsigned long long* range, double* scale) {
  const double most = most_spread(run, runs);
  const unsigned long long* sums = range + (size_t)p.mwlr * p.L;
  for (int el = 0; el < p.mwlr * p.L; el++) {
    // above every entry with this high word
    const unsigned long long bits = (range[el] + 1) << 32;
    double top;
    memcpy(&top, &bits, sizeof(top));
    int e;
    if (range[el] >= 0x7ff00000ull || !(top <= std::ldexp(1.98, kSliceMaxExponent))) return false;
    std::frexp(top / 1.98, &e);  // top <= 1.98 2^e
    scale[el] = std::ldexp(1.0, -e);
    // the slice of least norm, against lines in SU(3) (three units a matrix)
    unsigned long long least = ~0ull;
    for (int y0 = 0; y0 < p.Nu; y0++) least = std::min(least, sums[(size_t)el * 2 * p.Nu + y0]);
    for (int y0 = 0; y0 < p.N0; y0++)
      least = std::min(least, sums[(size_t)(el * 2 + 1) * p.Nu + y0]);
    const double norm2 = std::ldexp((double)least, -30) / (9.0 * g.vs);
    if (!(std::ldexp(1.0, 2 * e) <= most * norm2)) return false;
  }
  return true;
}

int slice_prepare(const SlicePlan& p) {
  void* fn = slice_kernel(p.TN);
  static std::mutex mu;
  static std::set<std::pair<int, void*>> done;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  if (done.count({dev, fn})) return 0;
  if (!tensor_map_encode()) {
    set_error("slice gram: the driver has no cuTensorMapEncodeTiled");
    return -1;
  }
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax) !=
      cudaSuccess) {
    set_error("slice gram: %zu bytes of shared memory per block: %s", kSmemMax,
              cudaGetErrorString(cudaGetLastError()));
    return -1;
  }
  done.insert({dev, fn});
  return 0;
}

void levels_deviation(const Geo& g, int msl, const double2* levels,
                      unsigned long long* dev, cudaStream_t st) {
  cudaMemsetAsync(dev, 0, sizeof(unsigned long long), st);
  const long long n = (long long)3 * msl * g.vol;
  const long long grid = std::min<long long>((n + 255) / 256, num_sms() * 16);
  k_levels_dev<<<(int)grid, 256, 0, st>>>(levels, link_elems<double>(g.vol), 3 * msl, g.vol, dev);
  WLG_LAUNCH_CHECK("levels_dev");
}

static LineArgs line_args(const Geo& g, const SlicePlan& p, const double* uh, const double* blines,
                          const double* hinv) {
  LineArgs a = {};
  a.g = g;
  a.Nu = p.Nu;
  a.ntile = p.ntile;
  a.msl = p.L;
  a.mwlr = p.mwlr;
  a.nuc = p.nuc;
  a.A = (size_t)p.Nu * p.ntile * kSlabTile;
  a.uh = uh;
  a.bl = blines;
  a.hinv = hinv;
  return a;
}

void slice_ranges(const Geo& g, const SlicePlan& p, const double* uh, const double* blines,
                  const double* hinv, unsigned long long* range, cudaStream_t st) {
  LineArgs a = line_args(g, p, uh, blines, hinv);
  a.cur = 3 * p.ntile;
  a.range = range;
  cudaMemsetAsync(range, 0, slice_range_bytes(p), st);
  const long long warps = (long long)p.Nu * a.cur * p.L;
  k_slice_lines<WALK_RANGE><<<(unsigned)((warps + 3) / 4), 128, 0, st>>>(a);
  WLG_LAUNCH_CHECK("slice_ranges");
}

void slice_lines(const Geo& g, const SlicePlan& p, const double* scale, int chunk,
                 const double* uh, const double* blines, const double* hinv, unsigned char* sa,
                 unsigned char* sb, cudaStream_t st) {
  LineArgs a = line_args(g, p, uh, blines, hinv);
  a.u0 = chunk * p.nuc;
  a.cur = std::min(p.nuc, 3 * p.ntile - a.u0);
  a.sa = sa;
  a.sb = sb;
  a.scale = scale;
  const long long warps = (long long)p.Nu * a.cur * p.L;
  const unsigned grid = (unsigned)((warps + 3) / 4);
  if (scale)
    k_slice_lines<WALK_SCALED><<<grid, 128, 0, st>>>(a);
  else
    k_slice_lines<WALK_PLAIN><<<grid, 128, 0, st>>>(a);
  WLG_LAUNCH_CHECK("slice_lines");
}

void slice_gram(const SlicePlan& p, int chunk, unsigned char* sa, unsigned char* sb,
                unsigned long long* acc, int* fail, cudaStream_t st) {
  CUtensorMap ma2, ma1, mb2, mb1;
  const long long un = (long long)p.mwlr * p.nuc;
  if (!plane_maps(&ma2, &ma1, sa, p.rows_a, un, 128) ||
      !plane_maps(&mb2, &mb1, sb, p.rows_b, un, p.TN)) {
    set_error("kernel slice_gram: tensor map refused");
    return;
  }
  GramTileArgs a;
  a.N0 = p.N0;
  a.Nu = p.Nu;
  a.L = p.L;
  a.mwlt = p.mwlt;
  a.mwlr = p.mwlr;
  a.rows_a = p.rows_a;
  a.rows_b = p.rows_b;
  a.TN = p.TN;
  a.nmt = p.nmt;
  a.ntiles = p.ntiles;
  a.kstride = p.nuc * 9;
  a.kcur = std::min(p.nuc, 3 * p.ntile - chunk * p.nuc) * 9;
  a.kps = p.kps;
  a.nsplit = p.nsplit;
  a.stages = p.stages;
  a.tmem_cols = (unsigned)p.tmem_cols;
  a.nwl = (long long)p.nwl;
  a.acc = acc;
  a.fail = fail;
  const long long items = (long long)p.mwlr * p.nsplit * p.ntiles;
  const unsigned grid = (unsigned)std::min<long long>(items, num_sms());
  void* args[] = {&ma2, &ma1, &mb2, &mb1, &a};
  cudaLaunchKernel(slice_kernel(p.TN), dim3(grid), dim3(kGramThreads), args, p.smem, st);
  WLG_LAUNCH_CHECK("slice_gram");
}

void slice_finish(const Geo& g, const SlicePlan& p, const double* scale, int bc,
                  const unsigned long long* acc, double* wl, cudaStream_t st) {
  const double norm = 9.0 * g.n[1] * g.n[2] * g.n[3];  // wloop.c:535
  const unsigned grid =
      (unsigned)std::min<size_t>((p.nwl + 255) / 256, (size_t)num_sms() * 16);
  const long long* s = reinterpret_cast<const long long*>(acc);
  k_slice_finish<<<grid, 256, 0, st>>>(s, (long long)p.nwl, p.N0, p.mwlt, p.mwlr, p.L, bc == 0,
                                       norm, scale, wl);
  WLG_LAUNCH_CHECK("slice_finish");
}

}  // namespace wlg
