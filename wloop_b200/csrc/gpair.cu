// gpair.cu -- the mixed form's temporal-gauge loop stage (gram.cu's identities)
// with the lines of all spatial extents walked in registers, stored with two
// levels side by side, and the banded Gram product in packed two-lane FP32
// FMAs on tiles that TMA stages.
//
// Every sum is the one of gram.cu's k_gram: over the runs of column chunks of
// the same plan, each accumulated with FP32 FMAs in column order, the runs
// added in FP64 in order.  (fma.rn.f32x2 rounds each lane as fmaf does, and
// the line products are gram.cu's, so the results are the same bit for bit.)
//
// A pass covers a contiguous range of runs, whose columns lie in the column
// units [u0, u0 + nu) (a unit: one direction, one 32-site tile; 18 chunks of
// 32 columns).  k_pair_lines writes the pass's lines of every R,
//     float2 index ((((R - 1) * LP + lp) * rows + y0) * nuc + unit) * 576 + c * 32 + lane
// with {level 2 lp, level 2 lp + 1} (the second zero past the last level) in
// one float2, rows = N0 for the A lines and Nu for the B lines; k_pair_gram
// forms the sums of every (R, run); k_pair_reduce adds them to the result.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <set>
#include <utility>

#include "internal.h"
#include "mbar.cuh"
#include "slab.cuh"
#include "tensormap.h"

namespace wlg {
namespace {

struct PairLineArgs {
  Geo g;
  int Nu, ntile, msl, LP, mwlr, u0, nu, nuc;
  size_t A;  // elements of one slab array
  const float *uh, *bl, *hinv;
  float2 *pa, *pb;
};

__device__ __forceinline__ void st_pair(float2* __restrict__ o, const M3<float>& a,
                                        const M3<float>& b, bool live) {
#pragma unroll
  for (int e = 0; e < 9; e++) {
    o[(2 * e) * 32] = live ? make_float2(a.e[e].x, b.e[e].x) : make_float2(0.f, 0.f);
    o[(2 * e + 1) * 32] = live ? make_float2(a.e[e].y, b.e[e].y) : make_float2(0.f, 0.f);
  }
}

// One warp per (y0, unit, level pair): B(x, R) = B(x, R - 1) Uh(x + (R - 1) k)
// and A(x, R) = (H^-1(x) B(x, R)) H^-1(x + R k) for R = 1..mwlr.
__global__ void __launch_bounds__(128, 4) k_pair_lines(PairLineArgs a) {
  const int lane = threadIdx.x & 31;
  unsigned w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lp = (int)(w % a.LP);
  w /= a.LP;
  const int ul = (int)(w % a.nu);
  const int y0 = (int)(w / a.nu);
  if (y0 >= a.Nu) return;
  const Geo& g = a.g;
  const int u = a.u0 + ul, k = u / a.ntile, jt = u - k * a.ntile;
  const bool live = jt * 32 + lane < g.vs;
  const int j = live ? jt * 32 + lane : g.vs - 1;
  const bool start = y0 < g.n[0], two = 2 * lp + 1 < a.msl;
  const size_t slice = (size_t)y0 * a.ntile * kSlabTile;
  const size_t q0 = (size_t)(2 * lp * 3 + k) * a.A + slice, q1 = q0 + (two ? 3 * a.A : 0);
  const float* hinv = a.hinv + slice;
  const int nk = k == 0 ? g.n[1] : (k == 1 ? g.n[2] : g.n[3]);
  const int st = k == 0 ? g.st[1] : (k == 1 ? g.st[2] : 1);
  int z = j, y = (j / st) % nk;  // x + (R - 1) k and its coordinate along k
  const size_t row = (size_t)a.nuc * kSlabTile;
  float2* ob = a.pb + ((size_t)lp * a.Nu + y0) * row + (size_t)ul * kSlabTile + lane;
  float2* oa = a.pa + ((size_t)lp * g.n[0] + y0) * row + (size_t)ul * kSlabTile + lane;
  const size_t step_b = (size_t)a.LP * a.Nu * row, step_a = (size_t)a.LP * g.n[0] * row;
  M3<float> c0, c1, f, t;
  ld_slab_as(c0, a.bl + q0, j >> 5, j & 31);
  zero(c1);
  if (two) ld_slab_as(c1, a.bl + q1, j >> 5, j & 31);
#pragma unroll 1
  for (int R = 1; R <= a.mwlr; R++) {
    if (R > 1) {
      ld_slab_as(f, a.uh + q0, z >> 5, z & 31);
      mul(t, c0, f);
      c0 = t;
      if (two) {
        ld_slab_as(f, a.uh + q1, z >> 5, z & 31);
        mul(t, c1, f);
        c1 = t;
      }
    }
    z += st;
    if (++y == nk) {
      y = 0;
      z -= nk * st;
    }
    st_pair(ob, c0, c1, live);
    if (start) {
      M3<float> t0, t1, s0, s1;
      ld_slab_as(f, hinv, j >> 5, j & 31);
      mul(t0, f, c0);
      if (two) mul(t1, f, c1);
      ld_slab_as(f, hinv, z >> 5, z & 31);
      mul(s0, t0, f);
      if (two)
        mul(s1, t1, f);
      else
        zero(s1);
      st_pair(oa, s0, s1, live);
    }
    ob += step_b;
    oa += step_a;
  }
}

// ---------------------------------------------------------------------------
// The Gram product.  An item is (R, run, start-slice block); a CTA walks items,
// one CTA per SM (up to four where blocks are small).  Thread 0 stages 16 columns at a time, stages - 2 ahead: one TMA
// box of the block's BXp start slices and one of its NYBp partner slices, all
// level pairs, as 128-byte rows (128-byte swizzle; slice counts padded to 8, so
// a thread's swizzle is fixed).  Thread (i, gq) owns start slice
// blk BX + i and the extents T = gq + 1 + NG j, as in k_gram: per two columns
// it reads LP A vectors and per extent LP B vectors, each {level, level + 1}
// of both columns, and advances its TQ L^2 sums.  The sums of a level pair of
// B are one packed accumulator; with an odd level count the last B level's
// sums are packed over pairs of A levels instead, so that only one of its L
// sums is a scalar FMA.
// ---------------------------------------------------------------------------
constexpr int kCols = 16;           // columns per stage
constexpr int kPairMaxStages = 8;

struct PairGramArgs {
  int N0, Nu, mwlt, BX, BXp, NYBp, NG, nblk;
  int mwlr, run0, nruns, cpc, nchunks, c_base;  // runs [run0, run0 + nruns), chunk of unit u0
  int stages, block;
  float* partial;  // [mwlr][nruns][N0][mwlt][L][L]
  int* fail;
};

__device__ __forceinline__ void tma_rows(unsigned dst, const CUtensorMap* map, int x, int y0, int R,
                                         uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(dst),
      "l"(map), "r"(x), "r"(y0), "r"(0), "r"(R), "r"(smem_addr(bar))
      : "memory");
}

__device__ __forceinline__ float4 lds4(unsigned addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

template <int L, int TQ, int THREADS>
__global__ void __launch_bounds__(THREADS, 1)
    k_pair_gram(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const PairGramArgs p) {
  constexpr int LP = (L + 1) / 2, NP = L / 2;
  constexpr bool ODD = L & 1;
  extern __shared__ unsigned char raw[];
  __shared__ __align__(8) uint64_t full[kPairMaxStages], empty[kPairMaxStages];
  __shared__ int quit;
  const int lane = threadIdx.x & 31;
  const unsigned base = (smem_addr(raw) + 1023u) & ~1023u;
  const unsigned bytes_a = (unsigned)(LP * p.BXp * 128), bytes_b = (unsigned)(LP * p.NYBp * 128);
  const unsigned stage_bytes = bytes_a + bytes_b;
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; s++) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, p.block / 32);
    }
    mbar_init_fence();
    quit = 0;
  }
  __syncthreads();
  const int per_r = p.nruns * p.nblk;
  const int items = p.mwlr * per_r;

  // thread 0's producer: the next stage to fetch
  int pit = blockIdx.x, pt = 0, pn = 0, px = 0, ps = 0, py = 0, pR = 0;
  unsigned pph = 0;
  long long issued = 0;
  auto produce = [&]() {
    while (pt == pn) {  // next item
      if (pit >= items) return;
      const int rest = pit % per_r, c0 = (p.run0 + rest / p.nblk) * p.cpc;
      pR = pit / per_r;
      py = (rest % p.nblk) * p.BX;
      px = (c0 - p.c_base) * 64;  // floats: 32 columns x 2 levels a chunk
      pn = (min(p.nchunks, c0 + p.cpc) - c0) * (32 / kCols);
      pt = 0;
      pit += gridDim.x;
    }
    if (!wait_or_quit(empty + ps, pph ^ 1, &quit)) return;
    const unsigned dst = base + ps * stage_bytes;
    mbar_expect_tx(full + ps, stage_bytes);
    tma_rows(dst, &map_a, px + pt * 2 * kCols, py, pR, full + ps);
    tma_rows(dst + bytes_a, &map_b, px + pt * 2 * kCols, py + 1, pR, full + ps);
    issued++;
    pt++;
    if (++ps == p.stages) {
      ps = 0;
      pph ^= 1;
    }
  };
  if (threadIdx.x == 0)
    for (int s = 0; s < p.stages - 2; s++) produce();

  {
    int i = threadIdx.x / p.NG;
    const int gq = threadIdx.x - i * p.NG;
    const bool inside = i < p.BX;
    if (!inside) i = p.BX - 1;  // idle threads read in-range rows and store nothing
    const unsigned row_a = (unsigned)(i * 128), swz_a = (unsigned)(i & 7) << 4;
    unsigned row_b[TQ], swz_b[TQ];
#pragma unroll
    for (int j = 0; j < TQ; j++) {
      int T = gq + 1 + p.NG * j;
      if (T > p.mwlt) T = p.mwlt;
      row_b[j] = bytes_a + (unsigned)((i + T - 1) * 128);
      swz_b[j] = (unsigned)((i + T - 1) & 7) << 4;
    }
    const unsigned lp_a = (unsigned)(p.BXp * 128), lp_b = (unsigned)(p.NYBp * 128);
    int s = 0;
    unsigned ph = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
      const int R = it / per_r, rest = it - R * per_r, rr = rest / p.nblk, run = p.run0 + rr;
      const int blk = rest % p.nblk;
      const int c0 = run * p.cpc, nk = min(p.nchunks, c0 + p.cpc) - c0;
      float2 acc[TQ][L][NP > 0 ? NP : 1], tail[TQ][NP > 0 ? NP : 1];
      float last[TQ];
#pragma unroll
      for (int j = 0; j < TQ; j++) {
#pragma unroll
        for (int l = 0; l < NP; l++) {
          tail[j][l] = make_float2(0.f, 0.f);
#pragma unroll
          for (int s1 = 0; s1 < L; s1++) acc[j][s1][l] = make_float2(0.f, 0.f);
        }
        last[j] = 0.f;
      }
      bool ok = true;
      for (int t = 0; t < nk * (32 / kCols); t++) {
        if (threadIdx.x == 0) produce();
        ok = __all_sync(0xffffffffu, wait_or_quit(full + s, ph, &quit));
        if (!ok) break;
        const unsigned sb = base + s * stage_bytes;
#pragma unroll
        for (unsigned q = 0; q < 8 * 16; q += 16) {  // two columns
          float4 a[LP];
#pragma unroll
          for (int l = 0; l < LP; l++) a[l] = lds4(sb + row_a + l * lp_a + (q ^ swz_a));
#pragma unroll
          for (int j = 0; j < TQ; j++) {
            const unsigned rb = sb + row_b[j] + (q ^ swz_b[j]);
            float4 b[LP];
#pragma unroll
            for (int l = 0; l < LP; l++) b[l] = lds4(rb + l * lp_b);
#pragma unroll
            for (int c = 0; c < 2; c++) {
              // the A levels back and forth, so that neighbouring FMAs share
              // an operand (register reads bound packed FMAs)
#pragma unroll
              for (int l = 0; l < NP; l++) {
                const float2 bp = c ? make_float2(b[l].z, b[l].w) : make_float2(b[l].x, b[l].y);
#pragma unroll
                for (int ss = 0; ss < L; ss++) {
                  const int s1 = ((l + c * NP) & 1) ? L - 1 - ss : ss;
                  const float4 v = a[s1 >> 1];
                  const float x = (s1 & 1) ? (c ? v.w : v.y) : (c ? v.z : v.x);
                  acc[j][s1][l] = __ffma2_rn(make_float2(x, x), bp, acc[j][s1][l]);
                }
              }
              if constexpr (ODD) {
                const float x = c ? b[LP - 1].z : b[LP - 1].x;
#pragma unroll
                for (int l = 0; l < NP; l++) {
                  const float2 ap = c ? make_float2(a[l].z, a[l].w) : make_float2(a[l].x, a[l].y);
                  tail[j][l] = __ffma2_rn(ap, make_float2(x, x), tail[j][l]);
                }
                last[j] = fmaf(c ? a[LP - 1].z : a[LP - 1].x, x, last[j]);
              }
            }
          }
        }
        // The slot's next content comes through the async proxy: each lane's reads
        // are ordered before it by the lane's own proxy fence, then by the warp's
        // barrier and lane 0's arrive (a release) and thread 0's wait (an acquire).
        // Without any fence a warp freed slots before its last read.
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + s);
        if (++s == p.stages) {
          s = 0;
          ph ^= 1;
        }
      }
      if (!ok) break;
      const int x0 = blk * p.BX + i;
      if (inside && x0 < p.N0) {
        float* out = p.partial +
                     (((size_t)R * p.nruns + rr) * p.N0 + x0) * ((size_t)p.mwlt * L * L);
#pragma unroll
        for (int j = 0; j < TQ; j++) {
          const int T = gq + 1 + p.NG * j;
          if (T <= p.mwlt) {
            float* o = out + (size_t)(T - 1) * L * L;
#pragma unroll
            for (int l = 0; l < NP; l++)
#pragma unroll
              for (int s1 = 0; s1 < L; s1++) {
                o[(2 * l) * L + s1] = acc[j][s1][l].x;
                o[(2 * l + 1) * L + s1] = acc[j][s1][l].y;
              }
            if constexpr (ODD) {
#pragma unroll
              for (int l = 0; l < NP; l++) {
                o[(L - 1) * L + 2 * l] = tail[j][l].x;
                o[(L - 1) * L + 2 * l + 1] = tail[j][l].y;
              }
              o[(L - 1) * L + L - 1] = last[j];
            }
          }
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && quit) {
    // the copies in flight, the last use of each stage
    for (long long b = issued > p.stages ? issued - p.stages : 0; b < issued; b++)
      mbar_wait_bounded(full + b % p.stages, (unsigned)((b / p.stages) & 1));
    atomicExch(p.fail, 1);
  }
}

// adds the pass's runs in order to wl (FP64); the last pass divides by the norm
// and writes exact zeros for the loops through the last slice of open time
__global__ void __launch_bounds__(256) k_pair_reduce(const float* __restrict__ partial, int nruns,
                                                     int N0, int mwlt, int LL, int mwlr, int first,
                                                     int last, int open, double norm,
                                                     double* __restrict__ wl) {
  const int per = mwlt * LL, nout = N0 * per;
  const long long n = (long long)mwlr * nout;
  for (long long w = blockIdx.x * (long long)blockDim.x + threadIdx.x; w < n;
       w += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(w / nout), o = (int)(w - (long long)r * nout);
    const int x0 = o / per, in = o - x0 * per;
    double* out = wl + ((size_t)x0 * mwlr + r) * per + in;
    double v = first ? 0.0 : *out;
    const float* q = partial + (size_t)r * nruns * nout + o;
    for (int i = 0; i < nruns; i++) v += (double)__ldg(q + (size_t)i * nout);
    if (last) v = (!open || x0 + in / LL + 1 < N0) ? v / norm : 0.0;
    *out = v;
  }
}

__global__ void k_narrow(const double2* __restrict__ src, float2* __restrict__ dst, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const double2 v = __ldg(src + i);
    dst[i] = make_float2((float)v.x, (float)v.y);
  }
}

// kernels: levels, extents per thread, threads per block (256: 255 registers a
// thread, 384: 168)
#define WLG_PAIR_VARIANTS(X)                                                                   \
  X(2, 12, 256) X(2, 8, 384) X(3, 8, 256) X(3, 6, 384) X(4, 6, 256) X(4, 4, 384) X(5, 4, 256)  \
  X(5, 3, 384) X(6, 3, 256) X(6, 2, 384) X(7, 2, 256) X(8, 2, 256)

void* pair_kernel(int L, int TQ) {
#define WLG_PAIR_PICK(LL, TT, NN) \
  if (L == LL && TQ == TT) return (void*)k_pair_gram<LL, TT, NN>;
  WLG_PAIR_VARIANTS(WLG_PAIR_PICK)
#undef WLG_PAIR_PICK
  return nullptr;
}

constexpr size_t kPairSmem = 226 * 1024;

bool line_map(CUtensorMap* m, void* base, int nuc, int rows, int LP, int mwlr, int box) {
  TensorMapEncode fn = tensor_map_encode();
  if (!fn) return false;
  const cuuint64_t row = (cuuint64_t)nuc * kSlabTile * 8;
  const cuuint64_t dim[4] = {(cuuint64_t)nuc * kSlabTile * 2, (cuuint64_t)rows, (cuuint64_t)LP,
                             (cuuint64_t)mwlr};
  const cuuint64_t str[3] = {row, row * rows, row * rows * LP};
  const cuuint32_t bx[4] = {2 * kCols, (cuuint32_t)box, (cuuint32_t)LP, 1}, one[4] = {1, 1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, dim, str, bx, one,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

bool pair_plan(PairPlan& p, const GramPlan& gp, const Geo& g, int msl, int mwlt, int mwlr,
               size_t budget) {
  p = PairPlan();
  if (msl < 2 || msl > 8 || mwlr < 1 || gp.esize != 4 || gp.nsplit < 1) return false;
  p.L = msl;
  p.LP = (msl + 1) / 2;
  p.N0 = g.n[0];
  p.Nu = gp.Nu;
  p.ntile = gp.ntile;
  p.mwlt = mwlt;
  p.mwlr = mwlr;
  p.cpc = gp.cpc;
  p.nsplit = gp.nsplit;
  p.nchunks = gp.nchunks;
  // extents per thread: fewest idle ones (ties: most per thread)
  int bw = 1 << 30, cap = 0;
#define WLG_PAIR_WASTE(LL, TT, NN)                              \
  if (msl == LL) {                                              \
    const int ng = (mwlt + TT - 1) / TT, waste = ng * TT - mwlt; \
    if (ng <= NN && waste < bw) {                               \
      bw = waste;                                               \
      cap = NN;                                                 \
      p.TQ = TT;                                                \
      p.NG = ng;                                                \
    }                                                           \
  }
  WLG_PAIR_VARIANTS(WLG_PAIR_WASTE)
#undef WLG_PAIR_WASTE
  if (p.TQ == 0) return false;
  const int bxmax = std::min(cap / p.NG, p.N0);
  for (int nblk = (p.N0 + bxmax - 1) / bxmax; nblk <= p.N0; nblk++) {
    const int BX = (p.N0 + nblk - 1) / nblk;
    const int BXp = (BX + 7) & ~7, NYBp = (BX + mwlt - 1 + 7) & ~7;
    const size_t stage = (size_t)p.LP * (BXp + NYBp) * 128;
    if (BXp > 256 || NYBp > 256 || 3 * stage + 1024 > kPairSmem) continue;
    p.BX = BX;
    p.BXp = BXp;
    p.NYBp = NYBp;
    p.nblk = (p.N0 + BX - 1) / BX;
    p.block = ((p.BX * p.NG + 31) / 32) * 32;
    // small blocks: several CTAs per SM, as many as the registers allow
    p.ctas = std::max(1, std::min(cap / p.block, (int)(kPairSmem / (3 * stage + 2048))));
    p.stages = (int)std::min<size_t>(
        kPairMaxStages, (kPairSmem / p.ctas - (p.ctas > 1 ? 2048 : 1024)) / stage);
    p.smem = p.stages * stage + 1024;
    break;
  }
  if (p.BX == 0) return false;
  // passes: as many runs as the line buffers and partial sums of the budget
  // hold; the units of r runs are at most (r cpc + 34) / 18
  const size_t unit = (size_t)mwlr * p.LP * (p.N0 + p.Nu) * kSlabTile * 8;
  const size_t run = (size_t)mwlr * p.N0 * mwlt * msl * msl * sizeof(float);
  const int units = 3 * p.ntile;
  auto need = [&](long long r) {
    return (size_t)std::min<long long>(units, (r * p.cpc + 34) / 18) * unit + (size_t)r * run + 512;
  };
  if (need(1) > budget) return false;
  long long lo = 1, hi = p.nsplit;
  while (lo < hi) {
    const long long mid = (lo + hi + 1) / 2;
    if (need(mid) <= budget)
      lo = mid;
    else
      hi = mid - 1;
  }
  p.npass = (int)((p.nsplit + lo - 1) / lo);
  p.runs = (p.nsplit + p.npass - 1) / p.npass;
  p.npass = (p.nsplit + p.runs - 1) / p.runs;
  p.nuc = (int)std::min<long long>(units, ((long long)p.runs * p.cpc + 34) / 18);
  p.bytes_a = (size_t)mwlr * p.LP * p.N0 * p.nuc * kSlabTile * 8;
  p.bytes_b = (size_t)mwlr * p.LP * p.Nu * p.nuc * kSlabTile * 8;
  p.bytes_p = (size_t)p.runs * run;
  return true;
}

int pair_prepare(const PairPlan& p) {
  void* fn = pair_kernel(p.L, p.TQ);
  if (!fn || !tensor_map_encode()) {
    set_error("pair gram: no kernel for %d levels, or no tensor maps", p.L);
    return -1;
  }
  static std::mutex mu;
  static std::set<std::pair<int, void*>> done;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  if (done.count({dev, fn})) return 0;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmem) !=
      cudaSuccess) {
    set_error("pair gram: %zu bytes of shared memory per block: %s", kPairSmem,
              cudaGetErrorString(cudaGetLastError()));
    return -1;
  }
  done.insert({dev, fn});
  return 0;
}

void narrow(const double* src, float* dst, size_t n, cudaStream_t st) {
  const size_t grid = std::min<size_t>((n / 2 + 255) / 256, (size_t)num_sms() * 16);
  k_narrow<<<(unsigned)grid, 256, 0, st>>>((const double2*)src, (float2*)dst, n / 2);
  WLG_LAUNCH_CHECK("narrow");
}

// first unit and unit count of a pass
static void pass_units(const PairPlan& p, int pass, int& run0, int& nruns, int& u0, int& nu) {
  run0 = pass * p.runs;
  nruns = std::min(p.runs, p.nsplit - run0);
  const long long c0 = (long long)run0 * p.cpc;
  const long long c1 = std::min<long long>(p.nchunks, (long long)(run0 + nruns) * p.cpc);
  u0 = (int)(c0 / 18);
  nu = (int)((c1 + 17) / 18) - u0;
}

void pair_lines(const Geo& g, const PairPlan& p, int pass, const float* uh, const float* blines,
                const float* hinv, void* pa, void* pb, cudaStream_t st) {
  PairLineArgs a;
  int run0, nruns;
  pass_units(p, pass, run0, nruns, a.u0, a.nu);
  a.g = g;
  a.Nu = p.Nu;
  a.ntile = p.ntile;
  a.msl = p.L;
  a.LP = p.LP;
  a.mwlr = p.mwlr;
  a.nuc = p.nuc;
  a.A = (size_t)p.Nu * p.ntile * kSlabTile;
  a.uh = uh;
  a.bl = blines;
  a.hinv = hinv;
  a.pa = (float2*)pa;
  a.pb = (float2*)pb;
  const long long warps = (long long)p.Nu * a.nu * p.LP;
  k_pair_lines<<<(unsigned)((warps + 3) / 4), 128, 0, st>>>(a);
  WLG_LAUNCH_CHECK("pair_lines");
}

void pair_gram(const PairPlan& p, int pass, void* pa, void* pb, float* partial, int* fail,
               cudaStream_t st) {
  CUtensorMap ma, mb;
  if (!line_map(&ma, pa, p.nuc, p.N0, p.LP, p.mwlr, p.BXp) ||
      !line_map(&mb, pb, p.nuc, p.Nu, p.LP, p.mwlr, p.NYBp)) {
    set_error("kernel pair_gram: tensor map refused");
    return;
  }
  PairGramArgs a;
  int u0, nu;
  pass_units(p, pass, a.run0, a.nruns, u0, nu);
  a.c_base = u0 * 18;
  a.N0 = p.N0;
  a.Nu = p.Nu;
  a.mwlt = p.mwlt;
  a.BX = p.BX;
  a.BXp = p.BXp;
  a.NYBp = p.NYBp;
  a.NG = p.NG;
  a.nblk = p.nblk;
  a.mwlr = p.mwlr;
  a.cpc = p.cpc;
  a.nchunks = p.nchunks;
  a.stages = p.stages;
  a.block = p.block;
  a.partial = partial;
  a.fail = fail;
  const long long items = (long long)p.mwlr * a.nruns * p.nblk;
  const unsigned grid = (unsigned)std::min<long long>(items, (long long)num_sms() * p.ctas);
  void* args[] = {&ma, &mb, &a};
  cudaLaunchKernel(pair_kernel(p.L, p.TQ), dim3(grid), dim3(p.block), args, p.smem, st);
  WLG_LAUNCH_CHECK("pair_gram");
}

void pair_reduce(const Geo& g, const PairPlan& p, int pass, int bc, const float* partial, double* wl,
                 cudaStream_t st) {
  const double norm = 9.0 * g.n[1] * g.n[2] * g.n[3];  // wloop.c:535
  const int run0 = pass * p.runs, nruns = std::min(p.runs, p.nsplit - run0);
  const long long n = (long long)p.mwlr * p.N0 * p.mwlt * p.L * p.L;
  k_pair_reduce<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
      partial, nruns, p.N0, p.mwlt, p.L * p.L, p.mwlr, pass == 0, pass == p.npass - 1, bc == 0, norm,
      wl);
  WLG_LAUNCH_CHECK("pair_reduce");
}

}  // namespace wlg
