// float32 mapped convolution on the CUDA cores: forward, input gradient, weight gradient.
//
//   forward  : src/nn/cuda/mapped_convolution_layer.cu:16-73   (im2col: include/nn/common/mapped_im2col.h:12-43)
//   dgrad    : src/nn/cuda/mapped_convolution_layer.cu:75-132  (col2im: mapped_im2col.h:45-78)
//   wgrad    : src/nn/cuda/mapped_convolution_layer.cu:134-193
//
// Takes every map whose tap reads at most four (source element, weight) pairs: plain nearest, bilinear
// and bispherical maps, and weighted maps of up to four nearest points.  Other maps, and float64, stay
// with the generic kernels, which decode one sample per im2col element.
//
// Bound: the contraction (fp32 FMA) and, close behind it, the L1 pipe that serves the gathers and the
// operand reads.  The im2col axis is therefore ordered (tap, channel): a thread decodes a tap of its pixel
// once and gathers eight channels with it (the generic order (channel, tap) decodes the map again for
// every element).  All three directions run the same register tile - 8 x 4 values a thread, packed
// fma.rn.f32x2, four 16-byte shared loads per 16 of them - on chunks of 16 steps of the contracted axis
// that are double buffered: the loads of the next chunk are issued before the current one is multiplied.
// The input gradient is staged in shared memory so that a warp adds 32 neighbouring pixels of one
// channel at a time; the right corner of one lane and the left corner of the next are usually the same
// source element and are added in registers first.
// 4 x 128 x 256 pixels, 32 -> 64 channels, 3 x 3 bilinear taps (4.8 GFLOP a direction), generic kernels -> these:
// forward 462 -> 227 us, input gradient 628 -> 343 us, weight gradient 600 -> 325 us; 64 x 128 pixels, 3 -> 16
// channels, forward 10.0 -> 6.6 us.
#include "common.cuh"

namespace mc {
namespace f32 {

constexpr int KK = 16;  // steps of the contracted axis per chunk

struct Args {
  const float* x;
  const float* gy;
  const float* map;
  const float* iw;
  const float* w;
  const float* bias;
  float* out;
  int B, Cin, Cout, IH, IW, K, P, interp, relu;
  long npix_img, npix_grid, total;  // total = B * npix_grid
  Strides xs, gs;                   // image side (x, gx) and grid side (y, gy)
  int CIP;       // channels per tap, padded: 4 where Cin <= 4, else a multiple of 8
  int rows;      // K * CIP: the padded im2col axis
  int n_tiles;   // tiles of the second output axis (fastest in the grid)
  int vec_out;   // 16-byte stores of the result are possible
  long pix_per_split;  // wgrad
};

struct Rec {
  int off[4];
  float w[4];
};

__device__ __forceinline__ Rec empty_rec() {
  Rec r;
#pragma unroll
  for (int i = 0; i < 4; ++i) { r.off[i] = -1; r.w[i] = 0.f; }
  return r;
}

// Up to four (source element, weight) pairs of tap k of grid element p.  For weighted nearest maps the
// sum of iw_i * value_i in the order of the points is the same rounded sequence as four corners.
__device__ __forceinline__ Rec load_rec(const Args& a, long p, int k) {
  Rec r = empty_rec();
  if (k >= a.K) return r;
  if (a.P == 0) {
    const long e = p * a.K + k;
    Tap<float> t;
    decode_tap<float, float>(__ldg(a.map + 2 * e), __ldg(a.map + 2 * e + 1), a.IH, a.IW, a.interp, t);
    r.off[0] = t.off[0];
    r.w[0] = t.w[0];
    if (t.n == 4) {
#pragma unroll
      for (int i = 1; i < 4; ++i) { r.off[i] = t.off[i]; r.w[i] = t.w[i]; }
    }
  } else {
    const long e = (p * a.K + k) * a.P;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i < a.P) {
        Tap<float> t;
        decode_tap<float, float>(__ldg(a.map + 2 * (e + i)), __ldg(a.map + 2 * (e + i) + 1), a.IH, a.IW, 0, t);
        r.off[i] = t.off[0];
        r.w[i] = __ldg(a.iw + e + i);
      }
    }
  }
  return r;
}

// raw[c][corner] of channels c0 .. c0 + N - 1 (zero beyond Cin and for inactive corners)
template <int VEC, int N, int R>
__device__ __forceinline__ void gather(const Args& a, const float* xb, const Rec& r, int c0, float (&raw)[R][4],
                                       int at) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float* src = xb + (long)r.off[i] * a.xs.p + c0 * a.xs.c;
    if (VEC) {  // channels-last, Cin % 4 == 0, 16-byte aligned rows
#pragma unroll
      for (int c = 0; c < N; c += 4) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r.off[i] >= 0 && c0 + c < a.Cin) v = __ldg(reinterpret_cast<const float4*>(src + c));
        raw[at + c][i] = v.x; raw[at + c + 1][i] = v.y; raw[at + c + 2][i] = v.z; raw[at + c + 3][i] = v.w;
      }
    } else {
#pragma unroll
      for (int c = 0; c < N; ++c)
        raw[at + c][i] = (r.off[i] >= 0 && c0 + c < a.Cin) ? __ldg(src + c * a.xs.c) : 0.f;
    }
  }
}

__device__ __forceinline__ float blend(const Rec& r, const float (&v)[4]) {
  float s = __fmul_rn(r.w[0], v[0]);
  s = __fadd_rn(s, __fmul_rn(r.w[1], v[1]));
  s = __fadd_rn(s, __fmul_rn(r.w[2], v[2]));
  return __fadd_rn(s, __fmul_rn(r.w[3], v[3]));
}

// Eight consecutive positions of the (tap, channel) axis at one pixel: one tap, or two where CIP == 4.
template <int VEC, bool C4>
struct ColLoader {
  Rec r0, r1;
  int k0 = -1;
  float raw[8][4];
  // row: a multiple of 8 (of 4 taps-worth where C4); p < 0: no pixel
  __device__ __forceinline__ void issue(const Args& a, const float* xb, long p, int row) {
    if (C4) {
      const int k = row >> 2;
      r0 = p >= 0 ? load_rec(a, p, k) : empty_rec();
      r1 = p >= 0 ? load_rec(a, p, k + 1) : empty_rec();
      gather<0, 4>(a, xb, r0, 0, raw, 0);
      gather<0, 4>(a, xb, r1, 0, raw, 4);
    } else {
      const int k = row / a.CIP;
      if (k != k0) {
        r0 = p >= 0 ? load_rec(a, p, k) : empty_rec();
        k0 = k;
      }
      gather<VEC, 8>(a, xb, r0, row - k * a.CIP, raw, 0);
    }
  }
  __device__ __forceinline__ float value(int j) const { return blend(C4 && j >= 4 ? r1 : r0, raw[j]); }
};

__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)),
        "l"(reinterpret_cast<const unsigned long long&>(c)));
  return d;
}

// A: KK rows of AW values (thread's eight: 4 tx .. and AW / 2 + 4 tx ..), row pitch AW + 4.
// B: KK rows of BW values, each stored twice; thread's CPT start at CPT ty.  Row pitch 2 BW + 4.
// Both pitches keep 16-byte alignment and spread a column over the banks.
template <int AW, int CPT>
struct Tile {
  static constexpr int BW = 16 * CPT;
  static constexpr int NT = 2 * AW;       // threads: AW / 8 along A, 16 along B
  static constexpr int AP = AW + 4, BP = 2 * BW + 4;
  float a[2][KK][AP];
  float b[2][KK][BP];
};

template <int AW, int CPT>
__device__ __forceinline__ void multiply(const float (&sa)[KK][Tile<AW, CPT>::AP],
                                         const float (&sb)[KK][Tile<AW, CPT>::BP], int tx, int ty,
                                         float2 (&acc)[4][CPT]) {
#pragma unroll
  for (int q = 0; q < KK; ++q) {
    const float4 u = *reinterpret_cast<const float4*>(&sa[q][4 * tx]);
    const float4 v = *reinterpret_cast<const float4*>(&sa[q][AW / 2 + 4 * tx]);
    float2 bb[CPT];
    if (CPT == 1) {
      bb[0] = *reinterpret_cast<const float2*>(&sb[q][2 * ty]);
    } else {
#pragma unroll
      for (int j = 0; j < CPT; j += 2) {
        const float4 t = *reinterpret_cast<const float4*>(&sb[q][2 * (ty * CPT + j)]);
        bb[j] = make_float2(t.x, t.y);
        if (j + 1 < CPT) bb[j + 1] = make_float2(t.z, t.w);
      }
    }
    const float2 aa[4] = {make_float2(u.x, u.y), make_float2(u.z, u.w), make_float2(v.x, v.y), make_float2(v.z, v.w)};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < CPT; ++j) acc[i][j] = ffma2(aa[i], bb[j], acc[i][j]);
  }
}

template <int CPT>
__device__ __forceinline__ void clear(float2 (&acc)[4][CPT]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < CPT; ++j) acc[i][j] = make_float2(0.f, 0.f);
}

__device__ __forceinline__ void put2(float* p, float v) { *reinterpret_cast<float2*>(p) = make_float2(v, v); }

// ---- forward: A = im2col values of AW pixels, B = weights of BW output channels --------------------------
template <int AW, int CPT, int VEC, bool C4>
__global__ void __launch_bounds__(2 * AW, 256 / AW) fwd_kernel(const Args a) {
  typedef Tile<AW, CPT> S;
  __shared__ __align__(16) S s;
  const int tid = threadIdx.x, tx = tid % (AW / 8), ty = tid / (AW / 8);
  const int px = tid % AW, h = tid / AW;  // gathering: this thread's pixel and half of the chunk's rows
  const long g0 = (long)(blockIdx.x / a.n_tiles) * AW;
  const int co0 = (int)(blockIdx.x % a.n_tiles) * S::BW;
  const long g = g0 + px;
  long p = -1;
  const float* xb = a.x;
  if (g < a.total) {
    const long b = g / a.npix_grid;
    p = g - b * a.npix_grid;
    xb = a.x + b * a.xs.b;
  }
  constexpr int NB = KK * S::BW / S::NT;  // weights a thread stages per chunk
  ColLoader<VEC, C4> col;
  float wr[NB];
  auto issue = [&](int row0) {
    col.issue(a, xb, p, row0 + 8 * h);
    const int row = row0 + (tid & 15);
    const int k = row / a.CIP, ci = row - k * a.CIP;
    const bool ok = k < a.K && ci < a.Cin;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const int co = co0 + (tid >> 4) + j * (S::NT / 16);
      wr[j] = ok && co < a.Cout ? __ldg(a.w + ((long)co * a.Cin + ci) * a.K + k) : 0.f;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int j = 0; j < 8; ++j) s.a[buf][8 * h + j][px] = col.value(j);
#pragma unroll
    for (int j = 0; j < NB; ++j) put2(&s.b[buf][tid & 15][2 * ((tid >> 4) + j * (S::NT / 16))], wr[j]);
  };
  float2 acc[4][CPT];
  clear(acc);
  issue(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int row0 = 0; row0 < a.rows; row0 += KK, buf ^= 1) {
    const bool more = row0 + KK < a.rows;
    if (more) issue(row0 + KK);
    multiply<AW, CPT>(s.a[buf], s.b[buf], tx, ty, acc);
    if (more) store(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const long gq = g0 + half * (AW / 2) + 4 * tx;
    if (gq >= a.total) continue;
    long b = gq / a.npix_grid;
    long q = gq - b * a.npix_grid;
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
      const int co = co0 + ty * CPT + j;
      if (co >= a.Cout) break;
      const float bv = a.bias ? __ldg(a.bias + co) : 0.f;
      const float2 lo = acc[2 * half][j], hi = acc[2 * half + 1][j];
      float v[4] = {lo.x + bv, lo.y + bv, hi.x + bv, hi.y + bv};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (a.relu && v[i] < 0.f) v[i] = 0.f;
      if (a.vec_out) {  // NCHW, npix_grid % 4 == 0: the four pixels are neighbours in one image
        *reinterpret_cast<float4*>(a.out + b * a.gs.b + co * a.gs.c + q) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
        long bi = b, qi = q;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (gq + i < a.total) a.out[bi * a.gs.b + co * a.gs.c + qi * a.gs.p] = v[i];
          if (++qi == a.npix_grid) { qi = 0; ++bi; }
        }
      }
    }
  }
}

// ---- dgrad: A = grad_output of AW pixels, B = weights of 64 (tap, channel) positions ---------------------
template <int AW, bool C4>
__global__ void __launch_bounds__(2 * AW, 256 / AW) dgrad_kernel(const Args a) {
  typedef Tile<AW, 4> S;
  __shared__ __align__(16) S s;
  const int tid = threadIdx.x, tx = tid % (AW / 8), ty = tid / (AW / 8);
  const int px = tid % AW, h = tid / AW;
  const long g0 = (long)(blockIdx.x / a.n_tiles) * AW;
  const int n0 = (int)(blockIdx.x % a.n_tiles) * 64;
  const long g = g0 + px;
  long b = -1, p = -1;
  if (g < a.total) {
    b = g / a.npix_grid;
    p = g - b * a.npix_grid;
  }
  const float* gyb = a.gy + (p >= 0 ? b * a.gs.b + p * a.gs.p : 0);
  constexpr int NB = KK * 64 / S::NT;
  const int n = n0 + (tid & 63), nk = n / a.CIP, nci = n - nk * a.CIP;
  const bool nok = nk < a.K && nci < a.Cin;
  const float* wn = a.w + (nok ? (long)nci * a.K + nk : 0);
  const long wstep = (long)a.Cin * a.K;
  float gr[8], wr[NB];
  auto issue = [&](int c0) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int co = c0 + 8 * h + j;
      gr[j] = p >= 0 && co < a.Cout ? __ldg(gyb + co * a.gs.c) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const int co = c0 + (tid >> 6) + j * (S::NT / 64);
      wr[j] = nok && co < a.Cout ? __ldg(wn + co * wstep) : 0.f;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int j = 0; j < 8; ++j) s.a[buf][8 * h + j][px] = gr[j];
#pragma unroll
    for (int j = 0; j < NB; ++j) put2(&s.b[buf][(tid >> 6) + j * (S::NT / 64)][2 * (tid & 63)], wr[j]);
  };
  float2 acc[4][4];
  clear(acc);
  issue(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int c0 = 0; c0 < a.Cout; c0 += KK, buf ^= 1) {
    const bool more = c0 + KK < a.Cout;
    if (more) issue(c0 + KK);
    multiply<AW, 4>(s.a[buf], s.b[buf], tx, ty, acc);
    if (more) store(buf ^ 1);
    __syncthreads();
  }
  // the tile [64][AW] over the operand buffers (the loop ended with a barrier)
  static_assert(64 * S::AP * sizeof(float) <= sizeof(S), "the staged tile fits the operand buffers");
  float (*z)[S::AP] = reinterpret_cast<float (*)[S::AP]>(&s);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 c0 = acc[0][j], c1 = acc[1][j], c2 = acc[2][j], c3 = acc[3][j];
    *reinterpret_cast<float4*>(&z[ty * 4 + j][4 * tx]) = make_float4(c0.x, c0.y, c1.x, c1.y);
    *reinterpret_cast<float4*>(&z[ty * 4 + j][AW / 2 + 4 * tx]) = make_float4(c2.x, c2.y, c3.x, c3.y);
  }
  __syncthreads();
  // Each warp: 32 neighbouring pixels, groups of NG positions that share a tap.
  constexpr int NG = C4 ? 4 : 8;
  const int lane = tid & 31;
  float* ob = a.out + (p >= 0 ? b * a.xs.b : 0);
  const int bi = (int)b;
  int klast = -1;
  Rec r = empty_rec();
  bool take[2] = {false, false}, give[2] = {false, false}, any = false;
  for (int q = h * NG; q < 64; q += 2 * NG) {
    const int k = (n0 + q) / a.CIP, ci0 = n0 + q - k * a.CIP;
    if (k >= a.K) break;
    if (k != klast) {
      klast = k;
      r = p >= 0 ? load_rec(a, p, k) : empty_rec();
      any = false;
#pragma unroll
      for (int e = 0; e < 2; ++e) {  // corner pairs (0, 1) and (2, 3): the two ends of a row
        const int left = __shfl_up_sync(0xffffffffu, r.off[2 * e + 1], 1);
        const int lb = __shfl_up_sync(0xffffffffu, bi, 1);
        take[e] = a.P == 0 && lane > 0 && lb == bi && r.off[2 * e] >= 0 && left == r.off[2 * e];
        const int right = __shfl_down_sync(0xffffffffu, (int)take[e], 1);
        give[e] = lane < 31 && right != 0;
        any |= take[e];
      }
      any = __any_sync(0xffffffffu, any);
    }
#pragma unroll
    for (int j = 0; j < NG; ++j) {
      if (ci0 + j >= a.Cin) break;
      const float zv = z[q + j][px];
      float c[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) c[i] = r.off[i] >= 0 ? __fmul_rn(r.w[i], zv) : 0.f;
      if (any) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float left = __shfl_up_sync(0xffffffffu, c[2 * e + 1], 1);
          if (take[e]) c[2 * e] += left;
          if (give[e]) c[2 * e + 1] = 0.f;
        }
      }
      float* o = ob + (ci0 + j) * a.xs.c;
      // (adding an exact zero changes nothing: the sums start from the bias or +0)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (c[i] != 0.f) atomicAdd(o + (long)r.off[i] * a.xs.p, c[i]);
    }
  }
}

// ---- wgrad: A = im2col values of AW (tap, channel) positions, B = grad_output of BW channels ---------------
template <int AW, int CPT, int VEC, bool C4>
__global__ void __launch_bounds__(2 * AW, 256 / AW) wgrad_kernel(const Args a) {
  typedef Tile<AW, CPT> S;
  __shared__ __align__(16) S s;
  const int tid = threadIdx.x, tx = tid % (AW / 8), ty = tid / (AW / 8);
  const int px = tid & 15, rg = tid >> 4;  // gathering: pixel of the chunk, group of eight positions
  const int n_rt = (a.rows + AW - 1) / AW;
  const int row0 = (int)(blockIdx.x % a.n_tiles) % n_rt * AW;
  const int co0 = (int)(blockIdx.x % a.n_tiles) / n_rt * S::BW;
  const long beg = (long)(blockIdx.x / a.n_tiles) * a.pix_per_split;
  long end = beg + a.pix_per_split;
  if (end > a.total) end = a.total;
  constexpr int NB = KK * S::BW / S::NT;
  ColLoader<VEC, C4> col;
  float gr[NB];
  auto issue = [&](long g1) {
    const long g = g1 + px;
    const bool ok = g < end;
    const long b = ok ? g / a.npix_grid : 0;
    const long p = ok ? g - b * a.npix_grid : -1;
    col.k0 = -1;
    col.issue(a, a.x + b * a.xs.b, p, row0 + 8 * rg);
    const float* gyb = a.gy + (ok ? b * a.gs.b + p * a.gs.p : 0);
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const int co = co0 + rg + j * (S::NT / 16);
      gr[j] = ok && co < a.Cout ? __ldg(gyb + co * a.gs.c) : 0.f;
    }
  };
  auto store = [&](int buf) {
    float* d = &s.a[buf][px][8 * rg];
    *reinterpret_cast<float4*>(d) = make_float4(col.value(0), col.value(1), col.value(2), col.value(3));
    *reinterpret_cast<float4*>(d + 4) = make_float4(col.value(4), col.value(5), col.value(6), col.value(7));
#pragma unroll
    for (int j = 0; j < NB; ++j) put2(&s.b[buf][px][2 * (rg + j * (S::NT / 16))], gr[j]);
  };
  float2 acc[4][CPT];
  clear(acc);
  issue(beg);
  store(0);
  __syncthreads();
  int buf = 0;
  for (long g1 = beg; g1 < end; g1 += KK, buf ^= 1) {
    const bool more = g1 + KK < end;
    if (more) issue(g1 + KK);
    multiply<AW, CPT>(s.a[buf], s.b[buf], tx, ty, acc);
    if (more) store(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int row = row0 + (i >> 1) * (AW / 2) + 4 * tx + 2 * (i & 1) + e;
      const int k = row / a.CIP, ci = row - k * a.CIP;
      if (k >= a.K || ci >= a.Cin) continue;
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        const int co = co0 + ty * CPT + j;
        if (co < a.Cout) atomicAdd(a.out + ((long)co * a.Cin + ci) * a.K + k, e ? acc[i][j].y : acc[i][j].x);
      }
    }
}

static Args make_args(const mc_desc* d) {
  Args a = {};
  a.B = d->B; a.Cin = d->C_in; a.Cout = d->C_out; a.IH = d->IH; a.IW = d->IW; a.K = d->K; a.P = d->P;
  a.interp = d->interp;
  a.relu = (d->flags & MC_FLAG_RELU) ? 1 : 0;
  a.npix_img = (long)d->IH * d->IW;
  a.npix_grid = (long)d->OH * d->OW;
  a.total = d->B * a.npix_grid;
  a.xs = make_strides(d->layout, d->C_in, a.npix_img);
  a.gs = make_strides(d->layout, d->C_out, a.npix_grid);
  a.CIP = d->C_in <= 4 ? 4 : (d->C_in + 7) / 8 * 8;
  a.rows = d->K * a.CIP;
  return a;
}

// 16-byte gathers: channels-last rows of whole float4s
static bool vec_ok(const mc_desc* d, const void* x) {
  return d->layout == MC_NHWC && d->C_in > 4 && d->C_in % 4 == 0 && ((uintptr_t)x & 15) == 0;
}

// Output channels a thread owns: the narrowest tile that holds C_out (up to 64 per block).
static int cpt_of(int cout) { return cout <= 16 ? 1 : cout <= 32 ? 2 : 4; }

// 64-pixel tiles where 128-pixel ones would leave SMs without a pair of blocks.
static bool small_tiles(long total, long n_tiles) { return (total + 127) / 128 * n_tiles < 2 * 148; }

template <int AW, int CPT>
static void launch_fwd(const Args& a, unsigned grid, bool vec, cudaStream_t st) {
  if (a.CIP == 4) fwd_kernel<AW, CPT, 0, true><<<grid, 2 * AW, 0, st>>>(a), MC_COUNT(1);
  else if (vec) fwd_kernel<AW, CPT, 1, false><<<grid, 2 * AW, 0, st>>>(a), MC_COUNT(1);
  else fwd_kernel<AW, CPT, 0, false><<<grid, 2 * AW, 0, st>>>(a), MC_COUNT(1);
}
template <int AW, int CPT>
static void launch_wgrad(const Args& a, unsigned grid, bool vec, cudaStream_t st) {
  if (a.CIP == 4) wgrad_kernel<AW, CPT, 0, true><<<grid, 2 * AW, 0, st>>>(a), MC_COUNT(1);
  else if (vec) wgrad_kernel<AW, CPT, 1, false><<<grid, 2 * AW, 0, st>>>(a), MC_COUNT(1);
  else wgrad_kernel<AW, CPT, 0, false><<<grid, 2 * AW, 0, st>>>(a), MC_COUNT(1);
}

}  // namespace f32

constexpr long F32_MAX_BLOCKS = (1L << 31) - 1;

// (the launch functions below return MC_ERR_UNSUPPORTED where a grid would not fit; nothing has run then)
bool conv_f32_supported(const mc_desc* d) {
  return d->dtype == MC_F32 && (d->P == 0 || (d->P <= 4 && d->interp != 1 && d->interp != 2));
}

int conv_fwd_f32_launch(const mc_desc* d, const void* x, const void* map, const void* iw, const void* w,
                        const void* bias, void* y, cudaStream_t st) {
  using namespace f32;
  Args a = make_args(d);
  a.x = (const float*)x; a.map = (const float*)map; a.iw = (const float*)iw; a.w = (const float*)w;
  a.bias = (const float*)bias; a.out = (float*)y;
  a.vec_out = d->layout == MC_NCHW && a.npix_grid % 4 == 0 && ((uintptr_t)y & 15) == 0;
  const int cpt = cpt_of(d->C_out);
  a.n_tiles = (d->C_out + 16 * cpt - 1) / (16 * cpt);
  const bool sm = small_tiles(a.total, a.n_tiles), vec = vec_ok(d, x);
  const long grid = (a.total + (sm ? 63 : 127)) / (sm ? 64 : 128) * a.n_tiles;
  if (grid > F32_MAX_BLOCKS) return MC_ERR_UNSUPPORTED;
  if (sm) {
    if (cpt == 1) launch_fwd<64, 1>(a, (unsigned)grid, vec, st);
    else if (cpt == 2) launch_fwd<64, 2>(a, (unsigned)grid, vec, st);
    else launch_fwd<64, 4>(a, (unsigned)grid, vec, st);
  } else {
    if (cpt == 1) launch_fwd<128, 1>(a, (unsigned)grid, vec, st);
    else if (cpt == 2) launch_fwd<128, 2>(a, (unsigned)grid, vec, st);
    else launch_fwd<128, 4>(a, (unsigned)grid, vec, st);
  }
  MC_CHECK_LAUNCH();
  return MC_OK;
}

// gx holds the start values (zero or bias)
int conv_dgrad_f32_launch(const mc_desc* d, const void* gy, const void* map, const void* iw, const void* w,
                          void* gx, cudaStream_t st) {
  using namespace f32;
  Args a = make_args(d);
  a.gy = (const float*)gy; a.map = (const float*)map; a.iw = (const float*)iw; a.w = (const float*)w;
  a.out = (float*)gx;
  a.n_tiles = (a.rows + 63) / 64;
  const bool sm = small_tiles(a.total, a.n_tiles);
  const long grid = (a.total + (sm ? 63 : 127)) / (sm ? 64 : 128) * a.n_tiles;
  if (grid > F32_MAX_BLOCKS) return MC_ERR_UNSUPPORTED;
  if (sm) {
    if (a.CIP == 4) dgrad_kernel<64, true><<<(unsigned)grid, 128, 0, st>>>(a), MC_COUNT(1);
    else dgrad_kernel<64, false><<<(unsigned)grid, 128, 0, st>>>(a), MC_COUNT(1);
  } else {
    if (a.CIP == 4) dgrad_kernel<128, true><<<(unsigned)grid, 256, 0, st>>>(a), MC_COUNT(1);
    else dgrad_kernel<128, false><<<(unsigned)grid, 256, 0, st>>>(a), MC_COUNT(1);
  }
  MC_CHECK_LAUNCH();
  return MC_OK;
}

// gw is zero
int conv_wgrad_f32_launch(const mc_desc* d, const void* gy, const void* x, const void* map, const void* iw,
                          void* gw, cudaStream_t st) {
  using namespace f32;
  Args a = make_args(d);
  a.gy = (const float*)gy; a.x = (const float*)x; a.map = (const float*)map; a.iw = (const float*)iw;
  a.out = (float*)gw;
  const int cpt = cpt_of(d->C_out);
  const long ct = (d->C_out + 16 * cpt - 1) / (16 * cpt);
  const long r64 = (a.rows + 63) / 64, r128 = (a.rows + 127) / 128;
  const bool narrow = 5 * r64 * 64 < 4 * r128 * 128;  // 128-wide tiles unless a fifth of them is padding
  const long tiles = ct * (narrow ? r64 : r128);
  // four 128-thread or two 256-thread blocks fit an SM; at least 64 pixels each
  long splits = (148L * (narrow ? 4 : 2)) / tiles;
  if (splits > (a.total + 63) / 64) splits = (a.total + 63) / 64;
  if (splits < 1) splits = 1;
  a.pix_per_split = ((a.total + splits - 1) / splits + KK - 1) / KK * KK;
  splits = (a.total + a.pix_per_split - 1) / a.pix_per_split;
  const long grid = tiles * splits;
  if (grid > F32_MAX_BLOCKS) return MC_ERR_UNSUPPORTED;
  a.n_tiles = (int)tiles;
  const bool vec = vec_ok(d, x);
  if (narrow) {
    if (cpt == 1) launch_wgrad<64, 1>(a, (unsigned)grid, vec, st);
    else if (cpt == 2) launch_wgrad<64, 2>(a, (unsigned)grid, vec, st);
    else launch_wgrad<64, 4>(a, (unsigned)grid, vec, st);
  } else {
    if (cpt == 1) launch_wgrad<128, 1>(a, (unsigned)grid, vec, st);
    else if (cpt == 2) launch_wgrad<128, 2>(a, (unsigned)grid, vec, st);
    else launch_wgrad<128, 4>(a, (unsigned)grid, vec, st);
  }
  MC_CHECK_LAUNCH();
  return MC_OK;
}

}  // namespace mc
