// Transforms whose pencils are shared by two lanes of a warp.
//
// Lanes l and l ^ 16 (h = 0, 1) hold the two halves of one pencil, N/2 values
// each.  An N-point transform is one radix-2 step across the pair (register
// exchange by shuffles) around N/2-point register transforms:
//   DIT  in  x[2m + h],     out X[h N/2 + m]
//   DIF  in  x[h N/2 + m],  out X[2m + h]
// Sixteen consecutive lanes own sixteen consecutive pencils, so row accesses
// (padded pitch) stay free of bank conflicts and column, remote and global
// accesses move 16 contiguous elements per half-warp.  Two lanes per pencil
// halve the registers per thread, i.e. double the warps an SM can hold for
// the same shared memory.
#pragma once
#include "cluster_slab.cuh"
#include "fft_reg.cuh"

namespace dgfs {

template <typename T> __device__ __forceinline__ T pair_swap(T a) {
  T r;
  r.x = __shfl_xor_sync(0xffffffffu, a.x, 16);
  r.y = __shfl_xor_sync(0xffffffffu, a.y, 16);
  return r;
}

template <typename R, int N, int SIGN>
__device__ __forceinline__ void half_twiddle(c2_t<R>* v, int h) {
  if (h) {
#pragma unroll
    for (int k = 1; k < N / 2; ++k) v[k] = twiddle_mul<R, N, SIGN>(v[k], k);
  }
}

// v[k] <- recv + sgn v[k], sgn = +1 (h = 0), -1 (h = 1)
template <typename R, int H>
__device__ __forceinline__ void half_butterfly(c2_t<R>* v, R sgn) {
#pragma unroll
  for (int k = 0; k < H; ++k) {
    const c2_t<R> o = pair_swap(v[k]);
    v[k] = cfma(sgn, v[k], o);
  }
}

template <typename R, int N, int SIGN>
__device__ __forceinline__ void fft_half_dit(c2_t<R>* v, int h) {
  fft<R, N / 2, SIGN>(v);
  half_twiddle<R, N, SIGN>(v, h);
  half_butterfly<R, N / 2>(v, h ? R(-1) : R(1));
}

template <typename R, int N, int SIGN>
__device__ __forceinline__ void fft_half_dif(c2_t<R>* v, int h) {
  half_butterfly<R, N / 2>(v, h ? R(-1) : R(1));
  half_twiddle<R, N, SIGN>(v, h);
  fft<R, N / 2, SIGN>(v);
}

// Geometry of an N^3 cube over C CTAs with two lanes per pencil.
template <int N, int C> struct HalfGeo {
  static_assert(N % C == 0, "cluster size must divide N");
  static constexpr int P = N / C;            // planes per CTA
  static constexpr int ROW = N + 1;          // padded row (complex elements)
  static constexpr int PLANE = N * ROW;
  static constexpr int SLAB = P * PLANE;
  static constexpr int H = N / 2;            // values per lane
  static constexpr int NT = 2 * P * N;       // threads
  static constexpr int n = N * N * N;
  static_assert((P * N) % 16 == 0, "pencils per CTA must fill half-warps");
  // y values h H .. h H + H - 1 of a lane belong to H / P CTAs (P <= H), or
  // to one CTA
  static constexpr int GRP = P <= H ? H / P : 1;
  static_assert(P > H || H % P == 0, "a lane's values must fill whole CTAs");
};

// pencil index and half of thread t
__device__ __forceinline__ int half_pencil(int t) { return (t >> 5) * 16 + (t & 15); }
__device__ __forceinline__ int half_lane(int t) { return (t >> 4) & 1; }

}  // namespace dgfs
