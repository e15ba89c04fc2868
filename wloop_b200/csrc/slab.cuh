// slab.cuh -- the temporal-gauge slab layout (gram.cu, gslice.cu, gpair.cu): component c
// (= 2 e + {0: re, 1: im} of entry e, row-major) of site (y0, j) of one array
// at ((y0 * ntile + j / 32) * 18 + c) * 32 + j % 32, ntile = ceil(vs / 32).
#pragma once
#include "common.cuh"

namespace wlg {

constexpr int kSlabTile = 576;  // elements per 32-site tile of one slab array

__host__ __device__ __forceinline__ size_t slab_tile(int y0, int ntile, int jt) {
  return (size_t)y0 * ntile + jt;
}

template <class E>
__device__ __forceinline__ void ld_slab(M3<double>& m, const E* __restrict__ base, size_t tile,
                                        int lane) {
  const E* p = base + tile * kSlabTile + lane;
#pragma unroll
  for (int e = 0; e < 9; e++) {
    m.e[e].x = (double)__ldg(p + (2 * e) * 32);
    m.e[e].y = (double)__ldg(p + (2 * e + 1) * 32);
  }
}

template <class E>
__device__ __forceinline__ void st_slab(E* __restrict__ base, size_t tile, int lane,
                                        const M3<double>& m) {
  E* p = base + tile * kSlabTile + lane;
#pragma unroll
  for (int e = 0; e < 9; e++) {
    p[(2 * e) * 32] = (E)m.e[e].x;
    p[(2 * e + 1) * 32] = (E)m.e[e].y;
  }
}

// the same in arithmetic type A (loads convert from the stored type S)
template <class A, class S>
__device__ __forceinline__ void ld_slab_as(M3<A>& m, const S* __restrict__ base, size_t tile,
                                           int lane) {
  const S* p = base + tile * kSlabTile + lane;
#pragma unroll
  for (int e = 0; e < 9; e++) {
    m.e[e].x = (A)__ldg(p + (2 * e) * 32);
    m.e[e].y = (A)__ldg(p + (2 * e + 1) * 32);
  }
}

template <class E, class A>
__device__ __forceinline__ void st_slab_from(E* __restrict__ base, size_t tile, int lane,
                                             const M3<A>& m) {
  E* p = base + tile * kSlabTile + lane;
#pragma unroll
  for (int e = 0; e < 9; e++) {
    p[(2 * e) * 32] = (E)m.e[e].x;
    p[(2 * e + 1) * 32] = (E)m.e[e].y;
  }
}

template <class E> __device__ __forceinline__ void zero_slab(E* __restrict__ base, size_t tile, int lane) {
  E* p = base + tile * kSlabTile + lane;
#pragma unroll
  for (int c = 0; c < 18; c++) p[c * 32] = E(0);
}

}  // namespace wlg
