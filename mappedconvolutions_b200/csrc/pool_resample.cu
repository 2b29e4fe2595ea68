// Mapped max / avg pooling, their adjoints, and resample gather / scatter.
//
// One launch covers the whole batch (the reference launches once per batch element,
// src/nn/cuda/mapped_max_pooling_layer.cu:31-35).  Element order follows the memory layout so
// that consecutive threads write consecutive addresses.  Semantics per element:
//   max pool   include/nn/common/mapped_max_pool.h:14-58   (+weighted :80-130)
//   max unpool include/nn/common/mapped_max_pool.h:61-78   (+weighted :132-169)
//   avg pool   include/nn/common/mapped_avg_pool.h:14-70   (+weighted :72-143)
//   resample   include/nn/common/resample.h:11-103
#include "common.cuh"

namespace mc {

enum { OP_GATHER = 0, OP_AVG = 1, OP_MAX = 2 };

// pool_fast.cu: bandwidth-oriented kernels for unweighted nearest (K in {1,4,7,9}) and single-tap
// bilinear maps; returns false when the generic kernel below has to take the call.
bool sample_fwd_fast(const mc_desc* d, int op, const void* x, const void* map, void* y, int64_t* idx,
                     cudaStream_t st, int* rc);
bool weighted3_ok(const mc_desc* d);
int weighted3_gather_launch(const mc_desc* d, const float* x, const float* map, const float* iw, float* y,
                            cudaStream_t st);
int weighted3_scatter_launch(const mc_desc* d, const float* g, const float* map, const float* iw, float* out,
                             cudaStream_t st);

struct SampleArgs {
  const void* x;
  const void* map;
  const void* iw;
  void* y;
  int64_t* idx;
  int B, C, IH, IW, K, P, interp, layout;
  long npix_in, npix_out;
};

// Weighted sample of one tap: sum_i iw_i * interp(point i)   (include/core/resample.h:145-162)
template <typename T, typename CT, typename MT>
__device__ __forceinline__ CT sample_tap(const T* plane, long sp, const MT* m, const MT* wts, int P,
                                         int H, int W, int interp) {
  Tap<CT> t;
  if (P == 0) {
    decode_tap<MT, CT>(m[0], m[1], H, W, interp, t);
    return tap_gather<T, CT>(plane, sp, t);
  }
  CT acc = CT(0);
  for (int i = 0; i < P; ++i) {
    decode_tap<MT, CT>(m[2 * i], m[2 * i + 1], H, W, interp, t);
    acc = add_rn(acc, mul_rn((CT)wts[i], tap_gather<T, CT>(plane, sp, t)));
  }
  return acc;
}

template <typename T, int OP>
__global__ void __launch_bounds__(256) sample_fwd_kernel(SampleArgs a) {
  typedef typename Traits<T>::CT CT;
  typedef typename Traits<T>::MT MT;
  const T* x = (const T*)a.x;
  const MT* map = (const MT*)a.map;
  const MT* iw = (const MT*)a.iw;
  T* y = (T*)a.y;
  const Strides xs = make_strides(a.layout, a.C, a.npix_in);
  const Strides ys = make_strides(a.layout, a.C, a.npix_out);
  const long total = (long)a.B * a.C * a.npix_out;
  const int pp = a.P > 0 ? a.P : 1;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total;
       i += (long)gridDim.x * blockDim.x) {
    int b, c;
    long p;
    split_index(i, a.layout, a.C, a.npix_out, b, c, p);
    const T* plane = x + b * xs.b + c * xs.c;
    const long tap0 = p * a.K * pp;  // index of this location's first (tap, point)
    CT acc = OP == OP_MAX ? (CT)(-FLT_MAX) : CT(0);
    long best = -1;
    for (int k = 0; k < a.K; ++k) {
      const long e = tap0 + (long)k * pp;
      const CT v = sample_tap<T, CT, MT>(plane, xs.p, map + 2 * e, iw ? iw + e : nullptr, a.P,
                                         a.IH, a.IW, a.interp);
      if (OP == OP_MAX) {
        if (v > acc) { acc = v; best = 2 * e; }
      } else if (OP == OP_AVG) {
        acc = add_rn(acc, v);
      } else {
        acc = v;
      }
    }
    if (OP == OP_AVG) acc = div_rn(acc, (CT)a.K);
    const long o = b * ys.b + c * ys.c + p * ys.p;
    stv(y + o, acc);
    if (OP == OP_MAX) a.idx[o] = best;
  }
}

// ---- adjoints (scatter) ------------------------------------------------------------------

struct ScatterArgs {
  const void* g;       // values on the map grid (B, C, npix_grid)
  const int64_t* idx;  // max-unpool only
  const void* map;
  const void* iw;
  void* out;  // accumulation target in CT (B, C, npix_img), pre-zeroed
  int B, C, IH, IW, K, P, interp, layout;
  long npix_img, npix_grid;
};

template <typename CT, typename MT>
__device__ __forceinline__ void scatter_tap(CT* plane, long sp, const MT* m, const MT* wts, int P,
                                            int H, int W, int interp, CT value) {
  Tap<CT> t;
  if (P == 0) {
    decode_tap<MT, CT>(m[0], m[1], H, W, interp, t);
    tap_scatter<CT>(plane, sp, t, value);
    return;
  }
  for (int i = 0; i < P; ++i) {
    decode_tap<MT, CT>(m[2 * i], m[2 * i + 1], H, W, interp, t);
    tap_scatter<CT>(plane, sp, t, mul_rn((CT)wts[i], value));
  }
}

// Scatter of `units` whole planes (NCHW) or images (NHWC) from unit u0 on, into a.out.  OP_GATHER here means "adjoint of gather" (resample scatter, K = 1).
template <typename T, int OP>
__global__ void __launch_bounds__(256) sample_bwd_kernel(ScatterArgs a, long u0, long units) {
  typedef typename Traits<T>::CT CT;
  typedef typename Traits<T>::MT MT;
  const T* g = (const T*)a.g;
  const MT* map = (const MT*)a.map;
  const MT* iw = (const MT*)a.iw;
  const bool nhwc = a.layout == MC_NHWC;
  const long n = nhwc ? a.npix_grid * a.C : a.npix_grid;  // values per unit
  const long nimg = nhwc ? a.npix_img * a.C : a.npix_img;
  const long sp = nhwc ? a.C : 1;
  const int pp = a.P > 0 ? a.P : 1;
  const long nt = (long)gridDim.x * 256;
  const long t0 = blockIdx.x * 256L + threadIdx.x;
  for (long u = blockIdx.y; u < units; u += gridDim.y) {
    CT* img = (CT*)a.out + u * nimg;
    const long base = (u0 + u) * n;
    constexpr int U = OP == OP_MAX ? 4 : 1;  // values in flight per thread
    for (long i0 = t0; i0 < n; i0 += nt * U) {
      CT v[U];
      int off[U];  // the stored offset is read back as a 32-bit int (mapped_max_pool.h:72-73)
      MT mx[U], my[U];
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const long i = i0 + j * nt;
        off[j] = -1;
        v[j] = CT(0);
        if (i < n) {
          if (OP == OP_MAX) off[j] = (int)a.idx[base + i];
          v[j] = (CT)ldv(g + base + i);
        }
      }
      if (OP == OP_MAX && a.P == 0) {
#pragma unroll
        for (int j = 0; j < U; ++j) {
          mx[j] = off[j] >= 0 ? map[off[j]] : MT(0);
          my[j] = off[j] >= 0 ? map[(long)off[j] + 1] : MT(0);
        }
      }
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const long i = i0 + j * nt;
        if (i >= n) break;
        long p = i;
        int c = 0;
        if (nhwc) {
          if (n < (1L << 31)) {
            p = (unsigned)i / (unsigned)a.C;
            c = (int)((unsigned)i - (unsigned)p * (unsigned)a.C);
          } else {
            p = i / a.C;
            c = (int)(i - p * a.C);
          }
        }
        CT* plane = img + c;
        if (OP == OP_MAX) {
          if (off[j] < 0) continue;
          if (a.P == 0) {
            Tap<CT> t;
            decode_tap<MT, CT>(mx[j], my[j], a.IH, a.IW, a.interp, t);
            tap_scatter<CT>(plane, sp, t, v[j]);
          } else {
            scatter_tap<CT, MT>(plane, sp, map + off[j], iw ? iw + off[j] / 2 : nullptr, a.P, a.IH, a.IW, a.interp,
                                v[j]);
          }
        } else {
          const CT val = OP == OP_AVG ? div_rn(v[j], (CT)a.K) : v[j];
          const long tap0 = p * a.K * pp;
          for (int k = 0; k < a.K; ++k) {
            const long e = tap0 + (long)k * pp;
            scatter_tap<CT, MT>(plane, sp, map + 2 * e, iw ? iw + e : nullptr, a.P, a.IH, a.IW, a.interp, val);
          }
        }
      }
    }
  }
}

// dst = src rounded, src = 0 (ready for the next chunk)
template <typename T>
__global__ void take_from_f32_kernel(float* src, T* dst, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
       i += (long)gridDim.x * blockDim.x) {
    stv(dst + i, src[i]);
    src[i] = 0.f;
  }
}

static int check_desc(const mc_desc* d, bool need_k1) {
  if (!d) return MC_ERR_BAD_ARG;
  if (d->B <= 0 || d->C_in <= 0 || d->IH <= 0 || d->IW <= 0 || d->OH <= 0 || d->OW <= 0 ||
      d->K <= 0 || d->P < 0)
    return MC_ERR_BAD_ARG;
  if (d->dtype != MC_F32 && d->dtype != MC_F64 && d->dtype != MC_BF16) return MC_ERR_BAD_ARG;
  if (d->layout != MC_NCHW && d->layout != MC_NHWC) return MC_ERR_BAD_ARG;
  if ((long)d->IH * d->IW >= (1L << 31) || (long)d->OH * d->OW * d->K * (d->P ? d->P : 1) >= (1L << 30))
    return MC_ERR_TOO_LARGE;
  if (need_k1 && d->K != 1) return MC_ERR_BAD_ARG;
  return MC_OK;
}

template <int OP>
static int launch_fwd(const mc_desc* d, const void* x, const void* map, const void* iw, void* y,
                      int64_t* idx, cudaStream_t st) {
  SampleArgs a;
  a.x = x; a.map = map; a.iw = iw; a.y = y; a.idx = idx;
  a.B = d->B; a.C = d->C_in; a.IH = d->IH; a.IW = d->IW; a.K = d->K; a.P = d->P;
  a.interp = d->interp; a.layout = d->layout;
  a.npix_in = (long)d->IH * d->IW;
  a.npix_out = (long)d->OH * d->OW;
  if (OP == OP_GATHER && weighted3_ok(d))
    return weighted3_gather_launch(d, (const float*)x, (const float*)map, (const float*)iw, (float*)y, st);
  int frc = MC_OK;
  if (sample_fwd_fast(d, OP, x, map, y, idx, st, &frc)) return frc;  // decode-once kernels
  const long total = (long)a.B * a.C * a.npix_out;
  const int grid = grid_for(total, 256);
  if (d->dtype == MC_F32) sample_fwd_kernel<float, OP><<<grid, 256, 0, st>>>(a), MC_COUNT(1);
  else if (d->dtype == MC_F64) sample_fwd_kernel<double, OP><<<grid, 256, 0, st>>>(a), MC_COUNT(1);
  else sample_fwd_kernel<bf16, OP><<<grid, 256, 0, st>>>(a), MC_COUNT(1);
  MC_CHECK_LAUNCH();
  return MC_OK;
}

// float32 and float64: one memset and one scatter of everything.  (In chunks of whole planes that stay in L2, each
// launch clearing the next one's target, every size is slower - max unpooling, everything / chunks of 64 / 32 / 16 MB:
// 32 x 128 planes of 163 842 vertices 1539 / 1893 / 1972 / 2175 us, of 40 962 401 / 473 / 490 / 507 us, 8 x 64 planes
// of 512 x 1024 pixels 840 / 943 / 915 / 922 us.)
// bf16: the float32 sums of a chunk are rounded into the result before the next chunk reuses their buffer, so that they
// stay in L2, with a third of it for them.  Max unpooling of bf16 in chunks of 24 / 32 / 43 / 64 / 96 MB: channels-last
// 32 x 128 x 40 962 vertices 685 / 684 / 556 / 660 / 719 us, 32 x 256 x 10 242 364 / 318 / 290 / 335 / 364 us; planes, 32 x 64 x
// 163 842 1386 / 1259 / 1214 / 1393 / 1496 us, 8 x 64 x 512 x 1024 1174 / 1065 / 1092 / 1268 / 1364 us.
constexpr long SCATTER_CHUNK_BYTES = 42L << 20;

// units: planes (NCHW) or images (NHWC) of unit_bytes
static long scatter_units_per_chunk(long units, long unit_bytes) {
  const long per = SCATTER_CHUNK_BYTES / unit_bytes;
  return per < 1 ? 1 : per > units ? units : per;
}

template <typename T, int OP>
static int launch_bwd_units(ScatterArgs a, typename Traits<T>::CT* acc, bf16* rounded, cudaStream_t st) {
  typedef typename Traits<T>::CT CT;
  const bool nhwc = a.layout == MC_NHWC;
  const long nimg = nhwc ? a.npix_img * a.C : a.npix_img, n = nhwc ? a.npix_grid * a.C : a.npix_grid;
  const long units = nhwc ? a.B : (long)a.B * a.C;
  const long per = rounded ? scatter_units_per_chunk(units, nimg * (long)sizeof(CT)) : units;
  a.out = acc;
  if (cudaMemsetAsync(acc, 0, per * nimg * sizeof(CT), st) != cudaSuccess) return MC_ERR_LAUNCH;
  const long vals = 256L * (OP == OP_MAX ? 4 : 1);
  const unsigned gx = (unsigned)((n + vals - 1) / vals < 148 * 32 ? (n + vals - 1) / vals : 148 * 32);
  for (long u0 = 0; u0 < units; u0 += per) {
    const long m = units - u0 < per ? units - u0 : per;
    const dim3 grid(gx, (unsigned)(m < 65535 ? m : 65535));
    sample_bwd_kernel<T, OP><<<grid, 256, 0, st>>>(a, u0, m), MC_COUNT(1);
    MC_CHECK_LAUNCH();
    if (rounded) {
      take_from_f32_kernel<bf16><<<grid_for(m * nimg, 256), 256, 0, st>>>((float*)acc, rounded + u0 * nimg,
                                                                          m * nimg), MC_COUNT(1);
      MC_CHECK_LAUNCH();
    }
  }
  return MC_OK;
}

template <int OP>
static int launch_bwd(const mc_desc* d, const void* g, const int64_t* idx, const void* map,
                      const void* iw, void* out, void* ws, size_t ws_bytes, cudaStream_t st) {
  ScatterArgs a;
  a.g = g; a.idx = idx; a.map = map; a.iw = iw;
  a.B = d->B; a.C = d->C_in; a.IH = d->IH; a.IW = d->IW; a.K = d->K; a.P = d->P;
  a.interp = d->interp; a.layout = d->layout;
  a.npix_img = (long)d->IH * d->IW;
  a.npix_grid = (long)d->OH * d->OW;
  if (OP == OP_GATHER && weighted3_ok(d))
    return weighted3_scatter_launch(d, (const float*)g, (const float*)map, (const float*)iw, (float*)out, st);
  if (d->dtype == MC_F32) return launch_bwd_units<float, OP>(a, (float*)out, nullptr, st);
  if (d->dtype == MC_F64) return launch_bwd_units<double, OP>(a, (double*)out, nullptr, st);
  if (!ws || ws_bytes < mc_scatter_workspace_bytes(d)) return MC_ERR_WORKSPACE;
  return launch_bwd_units<bf16, OP>(a, (float*)ws, (bf16*)out, st);
}

}  // namespace mc

using namespace mc;

extern "C" {

size_t mc_scatter_workspace_bytes(const mc_desc* d) {
  if (!d || d->dtype != MC_BF16 || d->B <= 0 || d->C_in <= 0 || d->IH <= 0 || d->IW <= 0) return 0;
  const bool nhwc = d->layout == MC_NHWC;  // one chunk of float32 sums
  const long unit = (long)d->IH * d->IW * (nhwc ? d->C_in : 1) * (long)sizeof(float);
  return (size_t)(scatter_units_per_chunk(nhwc ? d->B : (long)d->B * d->C_in, unit) * unit);
}

int mc_pool_max_fwd(const mc_desc* d, const void* x, const void* map, const void* iw, void* y,
                    int64_t* idx, void* stream) {
  int rc = check_desc(d, false);
  if (rc) return rc;
  if (!x || !map || !y || !idx || (d->P > 0 && !iw)) return MC_ERR_BAD_ARG;
  return launch_fwd<OP_MAX>(d, x, map, d->P ? iw : nullptr, y, idx, (cudaStream_t)stream);
}

int mc_pool_avg_fwd(const mc_desc* d, const void* x, const void* map, const void* iw, void* y,
                    void* stream) {
  int rc = check_desc(d, false);
  if (rc) return rc;
  if (!x || !map || !y || (d->P > 0 && !iw)) return MC_ERR_BAD_ARG;
  return launch_fwd<OP_AVG>(d, x, map, d->P ? iw : nullptr, y, nullptr, (cudaStream_t)stream);
}

int mc_resample_gather(const mc_desc* d, const void* x, const void* map, const void* iw, void* y,
                       void* stream) {
  int rc = check_desc(d, true);
  if (rc) return rc;
  if (!x || !map || !y || (d->P > 0 && !iw)) return MC_ERR_BAD_ARG;
  return launch_fwd<OP_GATHER>(d, x, map, d->P ? iw : nullptr, y, nullptr, (cudaStream_t)stream);
}

int mc_pool_max_bwd(const mc_desc* d, const void* gy, const int64_t* idx, const void* map,
                    const void* iw, void* gx, void* ws, size_t ws_bytes, void* stream) {
  int rc = check_desc(d, false);
  if (rc) return rc;
  if (!gy || !idx || !map || !gx || (d->P > 0 && !iw)) return MC_ERR_BAD_ARG;
  return launch_bwd<OP_MAX>(d, gy, idx, map, d->P ? iw : nullptr, gx, ws, ws_bytes,
                            (cudaStream_t)stream);
}

int mc_pool_avg_bwd(const mc_desc* d, const void* gy, const void* map, const void* iw, void* gx,
                    void* ws, size_t ws_bytes, void* stream) {
  int rc = check_desc(d, false);
  if (rc) return rc;
  if (!gy || !map || !gx || (d->P > 0 && !iw)) return MC_ERR_BAD_ARG;
  return launch_bwd<OP_AVG>(d, gy, nullptr, map, d->P ? iw : nullptr, gx, ws, ws_bytes,
                            (cudaStream_t)stream);
}

int mc_resample_scatter(const mc_desc* d, const void* x, const void* map, const void* iw, void* y,
                        void* ws, size_t ws_bytes, void* stream) {
  int rc = check_desc(d, true);
  if (rc) return rc;
  if (!x || !map || !y || (d->P > 0 && !iw)) return MC_ERR_BAD_ARG;
  return launch_bwd<OP_GATHER>(d, x, nullptr, map, d->P ? iw : nullptr, y, ws, ws_bytes,
                               (cudaStream_t)stream);
}

}  // extern "C"
