// Change of activation layout: per batch element a [rows][cols] matrix becomes [cols][dst_cols], with
// zeros in columns rows .. dst_cols - 1.  rows = channels, cols = pixels turns the reference's NCHW into
// channels-last (optionally with padded channels); rows = pixels, cols = channels turns it back.
//
// Bound: HBM, one read and one write of the tensor.  64 x 64 tiles go through shared memory so that both
// sides move 16 bytes per lane along their own rows; a 64-channel bf16 tensor of 4 x 250 x 500 pixels takes
// 30 us = 4.3 TB/s where torch's strided copy takes 122 us.
#include "common.cuh"

namespace mc {

constexpr int LT = 64;  // tile edge

template <typename T>
__global__ void __launch_bounds__(256) transpose_kernel(const T* __restrict__ src, T* __restrict__ dst, long rows,
                                                        long cols, long dst_cols, long tiles_r, long tiles_c,
                                                        int vec_src, int vec_dst) {
  constexpr int V = 16 / sizeof(T);
  constexpr int PITCH = sizeof(T) == 2 ? LT + 2 : LT + 1;  // an odd number of words
  __shared__ __align__(16) T tile[LT * PITCH];
  const long per = tiles_r * tiles_c;
  const long b = blockIdx.x / per, t = blockIdx.x - b * per;
  const long r0 = (t / tiles_c) * LT, c0 = (t % tiles_c) * LT;
  const T* s = src + b * rows * cols;
  T* d = dst + b * cols * dst_cols;
  const int tid = threadIdx.x;
  if (vec_src) {
    // LT rows of LT / V vectors; a vector is wholly inside or outside (cols is a multiple of V)
#pragma unroll
    for (int i = tid; i < LT * (LT / V); i += 256) {
      const int r = i / (LT / V), cv = (i % (LT / V)) * V;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (r0 + r < rows && c0 + cv < cols) v = __ldg(reinterpret_cast<const uint4*>(s + (r0 + r) * cols + c0 + cv));
      uint32_t* w = reinterpret_cast<uint32_t*>(tile + r * PITCH + cv);
      w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    }
  } else {
    for (int i = tid; i < LT * LT; i += 256) {
      const int r = i / LT, c = i % LT;
      tile[r * PITCH + c] = r0 + r < rows && c0 + c < cols ? __ldg(s + (r0 + r) * cols + c0 + c) : T(0);
    }
  }
  __syncthreads();
  if (vec_dst) {
#pragma unroll
    for (int i = tid; i < LT * (LT / V); i += 256) {
      const int c = i / (LT / V), rv = (i % (LT / V)) * V;
      if (c0 + c >= cols || r0 + rv >= dst_cols) continue;
      __align__(16) T o[V];
#pragma unroll
      for (int j = 0; j < V; ++j) o[j] = tile[(rv + j) * PITCH + c];
      *reinterpret_cast<uint4*>(d + (c0 + c) * dst_cols + r0 + rv) = *reinterpret_cast<const uint4*>(o);
    }
  } else {
    for (int i = tid; i < LT * LT; i += 256) {
      const int c = i / LT, r = i % LT;
      if (c0 + c < cols && r0 + r < dst_cols) d[(c0 + c) * dst_cols + r0 + r] = tile[r * PITCH + c];
    }
  }
}

// Few rows or few columns (images of up to 16 channels): a tile would be mostly empty.  One thread per
// pixel; its channels are neighbours on one side, the pixels on the other.
constexpr int LT_FEW = 16;

template <typename T>
__global__ void __launch_bounds__(256) few_rows_kernel(const T* __restrict__ src, T* __restrict__ dst, int rows,
                                                       long cols, int dst_cols, long total) {
  for (long i = blockIdx.x * 256L + threadIdx.x; i < total; i += gridDim.x * 256L) {
    const long b = i / cols, c = i - b * cols;
    const T* s = src + b * rows * cols + c;
    T* d = dst + i * dst_cols;
    for (int r = 0; r < dst_cols; ++r) d[r] = r < rows ? __ldg(s + r * cols) : T(0);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) few_cols_kernel(const T* __restrict__ src, T* __restrict__ dst, long rows,
                                                       int cols, long total) {
  for (long i = blockIdx.x * 256L + threadIdx.x; i < total; i += gridDim.x * 256L) {
    const long b = i / rows, r = i - b * rows;
    const T* s = src + i * cols;
    T* d = dst + b * rows * cols + r;
    for (int c = 0; c < cols; ++c) d[c * rows] = __ldg(s + c);
  }
}

template <typename T>
static int transpose_launch(long B, long rows, long cols, const void* src, void* dst, long dst_cols, cudaStream_t st) {
  if (dst_cols <= LT_FEW) {
    few_rows_kernel<T><<<grid_for(B * cols, 256), 256, 0, st>>>((const T*)src, (T*)dst, (int)rows, cols, (int)dst_cols,
                                                              B * cols), MC_COUNT(1);
  } else if (cols <= LT_FEW && dst_cols == rows) {
    few_cols_kernel<T><<<grid_for(B * rows, 256), 256, 0, st>>>((const T*)src, (T*)dst, rows, (int)cols, B * rows),
        MC_COUNT(1);
  } else {
    constexpr int V = 16 / sizeof(T);
    const long tr = (dst_cols + LT - 1) / LT, tc = (cols + LT - 1) / LT, n = B * tr * tc;
    if (n >= (1L << 31)) return MC_ERR_TOO_LARGE;
    const int vs = cols % V == 0 && ((uintptr_t)src & 15) == 0, vd = dst_cols % V == 0 && ((uintptr_t)dst & 15) == 0;
    transpose_kernel<T><<<(unsigned)n, 256, 0, st>>>((const T*)src, (T*)dst, rows, cols, dst_cols, tr, tc, vs, vd),
        MC_COUNT(1);
  }
  MC_CHECK_LAUNCH();
  return MC_OK;
}

// float32 sums of a weight / bias gradient -> bf16 parameters' gradients, both in one launch.
__global__ void __launch_bounds__(256) round_pair_kernel(const float* __restrict__ a, bf16* __restrict__ da, long na,
                                                         const float* __restrict__ b, bf16* __restrict__ db, long n) {
  for (long i = blockIdx.x * 256L + threadIdx.x; i < n; i += gridDim.x * 256L) {
    if (i < na) da[i] = __float2bfloat16_rn(a[i]);
    else db[i - na] = __float2bfloat16_rn(b[i - na]);
  }
}

}  // namespace mc

extern "C" int mc_round_pair(const float* a, void* da, int64_t na, const float* b, void* db, int64_t nb, void* stream) {
  using namespace mc;
  if (na < 0 || nb < 0 || na + nb <= 0 || (na && (!a || !da)) || (nb && (!b || !db))) return MC_ERR_BAD_ARG;
  round_pair_kernel<<<grid_for(na + nb, 256), 256, 0, (cudaStream_t)stream>>>(a, (bf16*)da, na, b, (bf16*)db, na + nb),
      MC_COUNT(1);
  MC_CHECK_LAUNCH();
  return MC_OK;
}

extern "C" int mc_transpose(int32_t elem_bytes, int64_t B, int64_t rows, int64_t cols, const void* src, void* dst,
                            int64_t dst_cols, void* stream) {
  using namespace mc;
  if (!src || !dst || B <= 0 || rows <= 0 || cols <= 0 || dst_cols < rows) return MC_ERR_BAD_ARG;
  if (elem_bytes == 2) return transpose_launch<uint16_t>(B, rows, cols, src, dst, dst_cols, (cudaStream_t)stream);
  if (elem_bytes == 4) return transpose_launch<uint32_t>(B, rows, cols, src, dst, dst_cols, (cudaStream_t)stream);
  return MC_ERR_UNSUPPORTED;
}
