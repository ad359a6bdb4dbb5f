// Bandwidth-bound reductions over one or several axes: softmax, RMSNorm, LayerNorm, the fused
// RMSNorm + residual + softmax + cast chain, and sum / mean / max(+argmax).
//
// Four kernels:
//  * row_kernel  : the reduced axes are the trailing, contiguous dims, up to 16384 elements. A group of G
//                  threads owns a row, keeps it in registers (4 x 128-bit loads per thread, 16 single loads
//                  where the length or alignment is odd), reduces with warp shuffles (+ one shared-memory
//                  hop above 32 threads) and writes the result once: one read and one write of HBM per element.
//  * span_kernel : a line is one or two runs-of-runs whose elements are neighbours in memory (a channel over
//                  batch and image, a group of channels, a long row). A cluster of CTAs shares the line.
//  * column_kernel : the reduced axes are one stride apart and the kept elements are neighbours. A cluster of
//                  CTAs shares the rows of 32 columns.
//  * line_kernel : any axes, any strides. A "line" is the set of elements reduced together; its
//                  elements are walked as an odometer over the reduced dims in the order the caller
//                  listed them (the order the reference's argmax index refers to). Either one CTA
//                  per line, or one thread per line when neighbouring lines are contiguous in memory.
//
// Replaces yt::function::softmax / rmsNorm / layerNorm (reference src/function/activation.inl:130-409,
// src/function/normalization.inl:3-54,159-277) and YTensor::sum / mean / max
// (src/ytensor_math.inl:414-692).
#include <math_constants.h>

#include <atomic>
#include <mutex>

#include "ptx_sm100.cuh"
#include "ytc_common.cuh"

namespace ytk {

enum RowOp { OP_SOFTMAX = 0, OP_RMSNORM = 1, OP_LAYERNORM = 2, OP_CHAIN = 3, OP_SUM = 4, OP_MEAN = 5, OP_MAX = 6,
             OP_LPNORM = 7,
             OP_RMSPLANES = 8 };  // rmsNorm of fp32 rows into two bf16 planes (row_kernel only)

struct F4 {
  float v[4];
};

__device__ __forceinline__ F4 load4(const void* p, int64_t i, int dt) {
  F4 r;
  if (dt == YTC_F32) {
    const float4 t = *reinterpret_cast<const float4*>(static_cast<const float*>(p) + i);
    r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
  } else {
    const uint2 t = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(p) + i);
    const uint16_t h[4] = {static_cast<uint16_t>(t.x & 0xFFFF), static_cast<uint16_t>(t.x >> 16),
                           static_cast<uint16_t>(t.y & 0xFFFF), static_cast<uint16_t>(t.y >> 16)};
#pragma unroll
    for (int k = 0; k < 4; ++k) r.v[k] = (dt == YTC_BF16) ? bf16_bits_to_f32(h[k]) : f16_bits_to_f32_ref(h[k]);
  }
  return r;
}
__device__ __forceinline__ void store4(void* p, int64_t i, const F4& r, int dt) {
  if (dt == YTC_F32) {
    *reinterpret_cast<float4*>(static_cast<float*>(p) + i) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
  } else {
    uint16_t h[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = (dt == YTC_BF16) ? f32_to_bf16_bits_ref(r.v[k]) : f32_to_f16_bits_ref(r.v[k]);
    uint2 t;
    t.x = static_cast<uint32_t>(h[0]) | (static_cast<uint32_t>(h[1]) << 16);
    t.y = static_cast<uint32_t>(h[2]) | (static_cast<uint32_t>(h[3]) << 16);
    *reinterpret_cast<uint2*>(static_cast<uint16_t*>(p) + i) = t;
  }
}

struct MaxIdx {
  float v;
  int i;
};
// Keeps the first maximum: a later element wins only if it is strictly greater
// (reference src/ytensor_math.inl:591-617 compares with `>` walking upwards).
__device__ __forceinline__ MaxIdx max_combine(MaxIdx a, MaxIdx b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

template <int G>
__device__ __forceinline__ float group_sum(float v, float* red, int group, int t) {
#pragma unroll
  for (int o = (G < 32 ? G : 32) / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if constexpr (G > 32) {
    constexpr int W = G / 32;
    if ((t & 31) == 0) red[group * W + (t >> 5)] = v;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) s += red[group * W + w];
    __syncthreads();
    v = s;
  }
  return v;
}
template <int G>
__device__ __forceinline__ float group_max(float v, float* red, int group, int t) {
#pragma unroll
  for (int o = (G < 32 ? G : 32) / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if constexpr (G > 32) {
    constexpr int W = G / 32;
    if ((t & 31) == 0) red[group * W + (t >> 5)] = v;
    __syncthreads();
    float s = -CUDART_INF_F;
#pragma unroll
    for (int w = 0; w < W; ++w) s = fmaxf(s, red[group * W + w]);
    __syncthreads();
    v = s;
  }
  return v;
}
template <int G>
__device__ __forceinline__ MaxIdx group_maxidx(MaxIdx m, float* red, int* redi, int group, int t) {
#pragma unroll
  for (int o = (G < 32 ? G : 32) / 2; o > 0; o >>= 1) {
    MaxIdx b;
    b.v = __shfl_xor_sync(0xffffffffu, m.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, m.i, o);
    m = max_combine(m, b);
  }
  if constexpr (G > 32) {
    constexpr int W = G / 32;
    if ((t & 31) == 0) {
      red[group * W + (t >> 5)] = m.v;
      redi[group * W + (t >> 5)] = m.i;
    }
    __syncthreads();
    MaxIdx s = {red[group * W], redi[group * W]};
#pragma unroll
    for (int w = 1; w < W; ++w) s = max_combine(s, MaxIdx{red[group * W + w], redi[group * W + w]});
    __syncthreads();
    m = s;
  }
  return m;
}

struct RowParams {
  const void* x;
  void* y;
  const void* w;   // weight / gamma (per column), may be null
  const void* b;   // beta (layernorm) or residual r (chain), may be null
  int* idx;        // argmax output (OP_MAX), may be null
  int64_t rows;
  int L;           // row length
  int64_t x_rs, y_rs;  // row strides in elements
  int64_t r_rows;  // chain: residual row = row % r_rows
  float eps;
  int dt_in, dt_out, dt_w;
};

// VEC: elements per load, 4 (element e of load v of thread t is column (v G + t) 4 + e) or 1 (column (4 v + e) G + t).
template <int OP, int G, int VEC>
__global__ void __launch_bounds__(G < 256 ? 256 : G) row_kernel(const RowParams p) {
  dependent_wait();     // (under a programmatic dependent launch: the kernel before this one has finished)
  dependent_trigger();  // the kernel queued behind this one may be scheduled meanwhile
  constexpr int THREADS = G < 256 ? 256 : G;
  constexpr int RPC = THREADS / G;  // rows per CTA
  constexpr int VPT = 4;
  __shared__ float red[32];
  __shared__ int redi[32];
  const int group = threadIdx.x / G, t = threadIdx.x % G;
  const int64_t row_blocks = (p.rows + RPC - 1) / RPC;
  const float invL = 1.0f / static_cast<float>(p.L);

  // chain with a residual shared by `copies` batch items: walk the rows so that the `copies` rows that read the same
  // residual row are handled back to back (by neighbouring CTAs) - the residual row then comes from HBM once and
  // from L2 for the other uses, instead of being evicted between uses that lie a whole batch item apart.
  const int64_t copies = (OP == OP_CHAIN && p.r_rows < p.rows) ? p.rows / p.r_rows : 1;
  for (int64_t rb = blockIdx.x; rb < row_blocks; rb += gridDim.x) {
    int64_t row = rb * RPC + group;
    const bool row_ok = row < p.rows;
    if (OP == OP_CHAIN && copies > 1 && row_ok) row = (row % copies) * p.r_rows + row / copies;
    F4 x[VPT];
    auto at = [&](int v, int e) { return VEC == 4 ? (v * G + t) * 4 + e : (4 * v + e) * G + t; };
    // (a load that is off for its first element is off for all: its arithmetic is jumped over. Softmax of fp32 100000 x 100: 24 us,
    // 43 with a test per element alone)
    auto on = [&](int v, int e) { return row_ok && at(v, VEC == 4 ? 0 : e) < p.L; };
    auto load = [&](const void* src, int64_t row0, int v, int dt) {
      F4 r = {{0.f, 0.f, 0.f, 0.f}};
      if constexpr (VEC == 4) {
        if (on(v, 0)) r = load4(src, row0 + at(v, 0), dt);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (on(v, e)) r.v[e] = load_as_f32(src, row0 + at(v, e), dt);
      }
      return r;
    };
#pragma unroll
    for (int v = 0; v < VPT; ++v) x[v] = load(p.x, row * p.x_rs, v, p.dt_in);

    if constexpr (OP == OP_SUM || OP == OP_MEAN) {
      float s = 0.f;
#pragma unroll
      for (int v = 0; v < VPT; ++v) s += (x[v].v[0] + x[v].v[1]) + (x[v].v[2] + x[v].v[3]);
      s = group_sum<G>(s, red, group, t);
      if (row_ok && t == 0) store_from_f32(p.y, row, OP == OP_MEAN ? s * invL : s, p.dt_out);
      continue;
    }
    if constexpr (OP == OP_MAX) {
      MaxIdx m = {-CUDART_INF_F, 0x7fffffff};
#pragma unroll
      for (int v = 0; v < VPT; ++v)
        if (on(v, 0)) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (VEC == 4 || on(v, k)) m = max_combine(m, MaxIdx{x[v].v[k], at(v, k)});
        }
      m = group_maxidx<G>(m, red, redi, group, t);
      if (row_ok && t == 0) {
        if (m.i == 0x7fffffff) {  // every element failed `>` (all NaN): the reference keeps element 0
          m.v = load_as_f32(p.x, row * p.x_rs, p.dt_in);
          m.i = 0;
        }
        store_from_f32(p.y, row, m.v, p.dt_out);
        if (p.idx) p.idx[row] = m.i;
      }
      continue;
    }

    if constexpr (OP == OP_RMSNORM || OP == OP_CHAIN || OP == OP_RMSPLANES) {
      float ss = 0.f;
#pragma unroll
      for (int v = 0; v < VPT; ++v)
#pragma unroll
        for (int k = 0; k < 4; ++k) ss = fmaf(x[v].v[k], x[v].v[k], ss);
      // issue the residual / weight loads before the reduction so that they overlap it
      F4 rr[VPT], ww[VPT];
      if constexpr (OP == OP_CHAIN) {
        const int64_t r_off = (row_ok ? (p.r_rows == p.rows ? row : row % p.r_rows) : 0) * static_cast<int64_t>(p.L);
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
          rr[v] = load(p.b, r_off, v, YTC_F32);
          ww[v] = load(p.w, 0, v, YTC_F32);
        }
      }
      ss = group_sum<G>(ss, red, group, t);
      const float inv = 1.0f / sqrtf(ss * invL + p.eps);
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        if (!on(v, 0)) continue;
#pragma unroll
        for (int k = 0; k < 4; ++k) x[v].v[k] *= inv;
        if constexpr (OP == OP_CHAIN) {
#pragma unroll
          for (int k = 0; k < 4; ++k) x[v].v[k] = fmaf(x[v].v[k], ww[v].v[k], rr[v].v[k]);
        } else if (p.w) {
          const F4 w = load(p.w, 0, v, p.dt_w);
#pragma unroll
          for (int k = 0; k < 4; ++k) x[v].v[k] *= w.v[k];
        }
      }
    }
    if constexpr (OP == OP_LAYERNORM) {
      float s = 0.f;
#pragma unroll
      for (int v = 0; v < VPT; ++v) s += (x[v].v[0] + x[v].v[1]) + (x[v].v[2] + x[v].v[3]);
      const float mu = group_sum<G>(s, red, group, t) * invL;
      float ss = 0.f;
#pragma unroll
      for (int v = 0; v < VPT; ++v)
        if (on(v, 0)) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (VEC == 4 || on(v, k)) {
              x[v].v[k] -= mu;
              ss = fmaf(x[v].v[k], x[v].v[k], ss);
            }
        }
      ss = group_sum<G>(ss, red, group, t);
      const float inv = 1.0f / sqrtf(ss * invL + p.eps);
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        if (!on(v, 0)) continue;
#pragma unroll
        for (int k = 0; k < 4; ++k) x[v].v[k] *= inv;
        if (p.w) {
          const F4 w = load(p.w, 0, v, p.dt_w);
          const F4 bb = load(p.b, 0, v, p.dt_w);
#pragma unroll
          for (int k = 0; k < 4; ++k) x[v].v[k] = x[v].v[k] * w.v[k] + bb.v[k];
        }
      }
    }
    if constexpr (OP == OP_SOFTMAX || OP == OP_CHAIN) {
      float m = -CUDART_INF_F;
#pragma unroll
      for (int v = 0; v < VPT; ++v)
        if (on(v, 0)) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (VEC == 4 || on(v, k)) m = fmaxf(m, x[v].v[k]);
        }
      m = group_max<G>(m, red, group, t);
      float s = 0.f;
#pragma unroll
      for (int v = 0; v < VPT; ++v)
        if (on(v, 0)) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (VEC == 4 || on(v, k)) {
              x[v].v[k] = __expf(x[v].v[k] - m);
              s += x[v].v[k];
            }
        }
      s = group_sum<G>(s, red, group, t);
      const float inv = 1.0f / s;
#pragma unroll
      for (int v = 0; v < VPT; ++v)
#pragma unroll
        for (int k = 0; k < 4; ++k) x[v].v[k] *= inv;
    }
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      if constexpr (OP == OP_RMSPLANES) {  // x = hi + lo, both rounded to nearest: 16 mantissa bits
        if (on(v, 0)) {
          F4 lo;
          uint32_t h[2], l[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const __nv_bfloat162 hb = __floats2bfloat162_rn(x[v].v[2 * e], x[v].v[2 * e + 1]);
            lo.v[2 * e] = x[v].v[2 * e] - __low2float(hb);
            lo.v[2 * e + 1] = x[v].v[2 * e + 1] - __high2float(hb);
            const __nv_bfloat162 lb = __floats2bfloat162_rn(lo.v[2 * e], lo.v[2 * e + 1]);
            h[e] = *reinterpret_cast<const uint32_t*>(&hb);
            l[e] = *reinterpret_cast<const uint32_t*>(&lb);
          }
          uint16_t* hi = static_cast<uint16_t*>(p.y) + row * p.y_rs + at(v, 0);
          *reinterpret_cast<uint2*>(hi) = make_uint2(h[0], h[1]);
          *reinterpret_cast<uint2*>(hi + p.rows * p.y_rs) = make_uint2(l[0], l[1]);
        }
      } else if constexpr (VEC == 4) {
        if (on(v, 0)) store4(p.y, row * p.y_rs + at(v, 0), x[v], p.dt_out);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (on(v, e)) store_from_f32(p.y, row * p.y_rs + at(v, e), x[v].v[e], p.dt_out);
      }
    }
  }
}



// ------------------------------------------------------------------ fused chain, specialised
// fp32 in, bf16 out, contiguous rows of exactly 1024 * VPT columns, 256 threads per row: no predicates, no dtype
// switches, exp2 by ex2.approx with the log2(e) factor folded into one FMA, bf16 narrowing (the reference's rule:
// add half an ulp only when the kept LSB is 1, then truncate) in three integer operations plus one byte permute per
// pair. About a dozen instructions per element, 4 CTAs per SM.
__device__ __forceinline__ float ex2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t bf16_pair_ref(float lo, float hi) {
  uint32_t a = __float_as_uint(lo), b = __float_as_uint(hi);
  a += (a >> 1) & 0x8000u;
  b += (b >> 1) & 0x8000u;
  return __byte_perm(a, b, 0x7632);  // {a.byte2, a.byte3, b.byte2, b.byte3}: the two upper halves
}

template <int VPT>
__global__ void __launch_bounds__(256, 4) chain_fast_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                            const float* __restrict__ r, uint2* __restrict__ out,
                                                            int64_t rows, int64_t r_rows, float eps) {
  constexpr int L = 1024 * VPT;
  __shared__ float red[32];
  const int t = threadIdx.x;
  const int64_t copies = r_rows < rows ? rows / r_rows : 1;
  const float invL = 1.0f / static_cast<float>(L);
  float4 wv[VPT];
#pragma unroll
  for (int v = 0; v < VPT; ++v) wv[v] = *reinterpret_cast<const float4*>(w + (v * 256 + t) * 4);
  for (int64_t rb = blockIdx.x; rb < rows; rb += gridDim.x) {
    // rows that share a residual row are handled back to back (see row_kernel)
    const int64_t row = copies > 1 ? (rb % copies) * r_rows + rb / copies : rb;
    const int64_t rrow = copies > 1 ? rb / copies : (r_rows == rows ? rb : rb % r_rows);
    const float4* xp = reinterpret_cast<const float4*>(x + row * L);
    const float4* rp = reinterpret_cast<const float4*>(r + rrow * L);
    float4 xv[VPT], rv[VPT];
#pragma unroll
    for (int v = 0; v < VPT; ++v) xv[v] = xp[v * 256 + t];
#pragma unroll
    for (int v = 0; v < VPT; ++v) rv[v] = rp[v * 256 + t];
    float ss = 0.f;
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      ss = fmaf(xv[v].x, xv[v].x, ss);
      ss = fmaf(xv[v].y, xv[v].y, ss);
      ss = fmaf(xv[v].z, xv[v].z, ss);
      ss = fmaf(xv[v].w, xv[v].w, ss);
    }
    ss = group_sum<256>(ss, red, 0, t);
    const float inv = 1.0f / sqrtf(ss * invL + eps);
    float m = -CUDART_INF_F;
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      xv[v].x = fmaf(xv[v].x * inv, wv[v].x, rv[v].x);
      xv[v].y = fmaf(xv[v].y * inv, wv[v].y, rv[v].y);
      xv[v].z = fmaf(xv[v].z * inv, wv[v].z, rv[v].z);
      xv[v].w = fmaf(xv[v].w * inv, wv[v].w, rv[v].w);
      m = fmaxf(m, fmaxf(fmaxf(xv[v].x, xv[v].y), fmaxf(xv[v].z, xv[v].w)));
    }
    m = group_max<256>(m, red, 0, t);
    const float nm = -m * 1.4426950408889634f;
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      xv[v].x = ex2_ftz(fmaf(xv[v].x, 1.4426950408889634f, nm));
      xv[v].y = ex2_ftz(fmaf(xv[v].y, 1.4426950408889634f, nm));
      xv[v].z = ex2_ftz(fmaf(xv[v].z, 1.4426950408889634f, nm));
      xv[v].w = ex2_ftz(fmaf(xv[v].w, 1.4426950408889634f, nm));
      s0 += xv[v].x + xv[v].y;
      s1 += xv[v].z + xv[v].w;
    }
    const float isum = 1.0f / group_sum<256>(s0 + s1, red, 0, t);
    uint2* op = out + row * (L / 4);
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      uint2 o;
      o.x = bf16_pair_ref(xv[v].x * isum, xv[v].y * isum);
      o.y = bf16_pair_ref(xv[v].z * isum, xv[v].w * isum);
      op[v * 256 + t] = o;
    }
  }
}

// ------------------------------------------------------------------ generic lines
constexpr int MAXD = 8;

struct LineParams {
  const void* x;
  void* y;
  const void* w;
  const void* b;
  int* idx;
  int nk, nr;                       // kept / reduced dim counts
  int64_t kshape[MAXD], kxs[MAXD], kys[MAXD];   // kept dims: extent, x stride, y stride
  int64_t rshape[MAXD], rxs[MAXD], rys[MAXD];   // reduced dims in LISTED order: extent, x stride, y stride
  int64_t rws[MAXD];                // stride of each reduced dim inside the weight (ascending-axis order layout)
  int64_t lines, R;
  float eps;
  float lp;  // exponent of OP_LPNORM
  int dt_in, dt_out, dt_w;
};

struct LineCtx {
  int64_t xbase, ybase;
};

__device__ __forceinline__ void line_offsets(const LineParams& p, int64_t r, int64_t& xo, int64_t& yo, int64_t& wo) {
  xo = 0; yo = 0; wo = 0;
  for (int d = p.nr - 1; d >= 0; --d) {
    const int64_t c = r % p.rshape[d];
    r /= p.rshape[d];
    xo += c * p.rxs[d];
    yo += c * p.rys[d];
    wo += c * p.rws[d];
  }
}

// PER_THREAD: one thread walks a whole line; otherwise the CTA's threads stride over it.
template <int OP, bool PER_THREAD>
__global__ void __launch_bounds__(128) line_kernel(const LineParams p) {
  __shared__ float red[32];
  __shared__ int redi[32];
  const int tid = threadIdx.x;
  int64_t line = PER_THREAD ? (blockIdx.x * static_cast<int64_t>(blockDim.x) + tid) : blockIdx.x;
  const int64_t line_step = PER_THREAD ? static_cast<int64_t>(gridDim.x) * blockDim.x : gridDim.x;
  const int64_t r0 = PER_THREAD ? 0 : tid, rstep = PER_THREAD ? 1 : 128;
  const float invR = 1.0f / static_cast<float>(p.R);
  // PER_THREAD lines finish independently; CTA lines keep every thread in the loop (block reductions inside).
  for (; PER_THREAD ? (line < p.lines) : (line < p.lines); line += line_step) {
    int64_t xb = 0, yb = 0, rem = line;
    for (int d = p.nk - 1; d >= 0; --d) {
      const int64_t c = rem % p.kshape[d];
      rem /= p.kshape[d];
      xb += c * p.kxs[d];
      yb += c * p.kys[d];
    }
    auto bsum = [&](float v) -> float {
      if constexpr (PER_THREAD) return v;
      else return group_sum<128>(v, red, 0, tid);
    };
    auto bmax = [&](float v) -> float {
      if constexpr (PER_THREAD) return v;
      else return group_max<128>(v, red, 0, tid);
    };
    int64_t xo, yo, wo;
    if constexpr (OP == OP_SUM || OP == OP_MEAN) {
      float s = 0.f;
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        s += load_as_f32(p.x, xb + xo, p.dt_in);
      }
      s = bsum(s);
      if (PER_THREAD || tid == 0) store_from_f32(p.y, yb, OP == OP_MEAN ? s * invR : s, p.dt_out);
    } else if constexpr (OP == OP_MAX) {
      MaxIdx m = {-CUDART_INF_F, 0x7fffffff};
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        m = max_combine(m, MaxIdx{load_as_f32(p.x, xb + xo, p.dt_in), static_cast<int>(r)});
      }
      if constexpr (!PER_THREAD) m = group_maxidx<128>(m, red, redi, 0, tid);
      if (PER_THREAD || tid == 0) {
        if (m.i == 0x7fffffff) {
          m.v = load_as_f32(p.x, xb, p.dt_in);
          m.i = 0;
        }
        store_from_f32(p.y, yb, m.v, p.dt_out);
        if (p.idx) p.idx[line] = m.i;
      }
    } else if constexpr (OP == OP_SOFTMAX) {
      float m = -CUDART_INF_F;
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        m = fmaxf(m, load_as_f32(p.x, xb + xo, p.dt_in));
      }
      m = bmax(m);
      float s = 0.f;
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        s += __expf(load_as_f32(p.x, xb + xo, p.dt_in) - m);
      }
      s = bsum(s);
      const float inv = 1.0f / s;
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        store_from_f32(p.y, yb + yo, __expf(load_as_f32(p.x, xb + xo, p.dt_in) - m) * inv, p.dt_out);
      }
    } else if constexpr (OP == OP_RMSNORM) {
      float ss = 0.f;
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        const float v = load_as_f32(p.x, xb + xo, p.dt_in);
        ss = fmaf(v, v, ss);
      }
      ss = bsum(ss);
      const float inv = 1.0f / sqrtf(ss * invR + p.eps);
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        float v = load_as_f32(p.x, xb + xo, p.dt_in) * inv;
        if (p.w) v *= load_as_f32(p.w, wo, p.dt_w);
        store_from_f32(p.y, yb + yo, v, p.dt_out);
      }
    } else if constexpr (OP == OP_LPNORM) {
      // yt::function::normalize (reference src/function/normalization.inl:56-85): x / (sum |x|^p + eps)^(1/p)
      float s = 0.f;
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        s += powf(fabsf(load_as_f32(p.x, xb + xo, p.dt_in)), p.lp);
      }
      s = bsum(s);
      const float den = powf(s + p.eps, 1.0f / p.lp);
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        store_from_f32(p.y, yb + yo, load_as_f32(p.x, xb + xo, p.dt_in) / den, p.dt_out);
      }
    } else if constexpr (OP == OP_LAYERNORM) {
      float s = 0.f;
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        s += load_as_f32(p.x, xb + xo, p.dt_in);
      }
      const float mu = bsum(s) * invR;
      float ss = 0.f;
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        const float c = load_as_f32(p.x, xb + xo, p.dt_in) - mu;
        ss = fmaf(c, c, ss);
      }
      ss = bsum(ss);
      const float inv = 1.0f / sqrtf(ss * invR + p.eps);
      for (int64_t r = r0; r < p.R; r += rstep) {
        line_offsets(p, r, xo, yo, wo);
        float v = (load_as_f32(p.x, xb + xo, p.dt_in) - mu) * inv;
        if (p.w) v = v * load_as_f32(p.w, wo, p.dt_w) + load_as_f32(p.b, wo, p.dt_w);
        store_from_f32(p.y, yb + yo, v, p.dt_out);
      }
    }
  }
}

// ------------------------------------------------------------------ lines shared by a cluster of CTAs
// span_kernel: the reduced elements of a line are R1 runs of R2 neighbours. column_kernel: they lie one stride apart and the
// kept elements next to a line are its neighbours in memory. Both bring a line's elements into shared memory once, as fp32,
// a share per CTA of a cluster, and pass the partial results through distributed shared memory in the order of the ranks:
// one read and one write of HBM per element and one launch, where line_kernel walks an odometer with a 64-bit division per
// element and pass, on one CTA (or thread) per line. Shares above CACHE_FLOATS are read again instead.
// What bounds them: span_kernel the two trips to memory with the sums between them: fp32 shares come in and leave as bulk copies
// of whole runs (16 x 96 x 56 x 56 fp32 over all axes but the channel, gamma and bias included: 965 us with line_kernel and two
// elementwise passes, 20.9 with four 16-byte loads a thread in flight and a division a load, 12.2 here, 6 at the copy rate);
// column_kernel the latency of its 32-column rows (softmax of fp32 2048 x 4096 along the first axis: 2891 / 60 us).
constexpr int SHARE_UNROLL = 4, MAX_SHARES = 8;
constexpr uint32_t CACHE_FLOATS = 50u * 1024;

struct ShareParams {
  const void* x;
  void* y;
  const void* w;
  const void* b;
  int* idx;
  int nk;                                                // kept dims (without the columns of column_kernel)
  int64_t kshape[MAXD], kxs[MAXD], kys[MAXD], kws[MAXD];  // extent, strides in x, y and gamma / beta
  uint32_t R, R2;          // elements of a line, of a run (span_kernel)
  int64_t xs1, ys1, ws1;   // strides of the runs (span_kernel), of the line's elements (column_kernel)
  int64_t ws2;             // span_kernel: stride of a run's elements in gamma / beta
  int64_t cols, cws;       // column_kernel: columns, their stride in gamma / beta
  uint32_t share;          // elements per CTA
  int shares;
  int cached;
  int bulk;                // span_kernel<.., BULK>
  int* status;
  float eps, lp;
  int dt_in, dt_out, dt_w;
};

// The sum (or maximum, or first maximum) of `mine` over the CTAs of the cluster, in the order of their ranks; `slot` is a
// word (pair) of this CTA that nothing else uses until the cluster's last barrier.
struct ShareSum {
  __device__ __forceinline__ float operator()(float a, float b) const { return a + b; }
};
struct ShareMax {
  __device__ __forceinline__ float operator()(float a, float b) const { return fmaxf(a, b); }
};
__device__ __forceinline__ float ld_cluster_f32(const void* p, uint32_t rank) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(map_to_cta(smem_u32(p), rank)) : "memory");
  return v;
}
template <class F>
__device__ __forceinline__ float over_shares(float mine, float* slot, bool writes, int shares, F f) {
  if (shares == 1) return mine;
  if (writes) *slot = mine;
  cluster_sync_all();
  float v = ld_cluster_f32(slot, 0);
  for (int r = 1; r < shares; ++r) v = f(v, ld_cluster_f32(slot, r));
  return v;
}
__device__ __forceinline__ MaxIdx over_shares(MaxIdx mine, float* slot, int* islot, bool writes, int shares) {
  if (shares == 1) return mine;
  if (writes) {
    *slot = mine.v;
    *islot = mine.i;
  }
  cluster_sync_all();
  MaxIdx m = {-CUDART_INF_F, 0x7fffffff};
  for (int r = 0; r < shares; ++r) m = max_combine(m, MaxIdx{ld_cluster_f32(slot, r), __float_as_int(ld_cluster_f32(islot, r))});
  return m;
}

// The passes over a line: `sweep(first, f)` calls f(value, index, n) for this thread's elements of the share (n: how many),
// from global memory the first time and from the cache afterwards; bsum / bmax / bmaxidx reduce over the whole line.
// `emit(g)` writes y = g(value) * gamma + beta.
template <int OP, class Sweep, class BSum, class BMax, class BMaxIdx, class Emit, class Result>
__device__ __forceinline__ void line_passes(const ShareParams& p, Sweep&& sweep, BSum&& bsum, BMax&& bmax, BMaxIdx&& bmaxidx,
                                            Emit&& emit, Result&& result) {
  const float invR = 1.0f / static_cast<float>(p.R);
  if constexpr (OP == OP_MAX) {
    MaxIdx m = {-CUDART_INF_F, 0x7fffffff};
    sweep(true, [&](float v, uint32_t r) { m = max_combine(m, MaxIdx{v, static_cast<int>(r)}); });
    m = bmaxidx(m);
    result(m.v, m.i);
  } else if constexpr (OP == OP_SUM || OP == OP_MEAN) {
    float s = 0.f;
    sweep(true, [&](float v, uint32_t) { s += v; });
    s = bsum(s, 0);
    result(OP == OP_MEAN ? s * invR : s, 0);
  } else if constexpr (OP == OP_SOFTMAX) {
    float m = -CUDART_INF_F;
    sweep(true, [&](float v, uint32_t) { m = fmaxf(m, v); });
    m = bmax(m, 0);
    float s = 0.f;
    sweep(false, [&](float v, uint32_t) { s += __expf(v - m); });
    const float inv = 1.0f / bsum(s, 1);
    emit([&](float v) { return __expf(v - m) * inv; });
  } else if constexpr (OP == OP_RMSNORM) {
    float ss = 0.f;
    sweep(true, [&](float v, uint32_t) { ss = fmaf(v, v, ss); });
    const float inv = 1.0f / sqrtf(bsum(ss, 0) * invR + p.eps);
    emit([&](float v) { return v * inv; });
  } else if constexpr (OP == OP_LPNORM) {
    float s = 0.f;
    sweep(true, [&](float v, uint32_t) { s += powf(fabsf(v), p.lp); });
    const float den = powf(bsum(s, 0) + p.eps, 1.0f / p.lp);
    emit([&](float v) { return v / den; });
  } else {
    float s = 0.f;
    sweep(true, [&](float v, uint32_t) { s += v; });
    const float mu = bsum(s, 0) * invR;
    float ss = 0.f;
    sweep(false, [&](float v, uint32_t) { ss = fmaf(v - mu, v - mu, ss); });
    const float inv = 1.0f / sqrtf(bsum(ss, 1) * invR + p.eps);
    emit([&](float v) { return (v - mu) * inv; });
  }
}

__device__ __forceinline__ void share_copy_in(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src),
               "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void share_copy_out(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)), "r"(bytes) : "memory");
}

// BULK (fp32): whole runs come into the cache, and results leave it, as bulk copies.
template <int OP, int VEC, int THREADS, bool BULK>
__global__ void __launch_bounds__(THREADS) span_kernel(const ShareParams p) {
  static_assert(!BULK || VEC == 4, "whole runs start at 16 bytes");
  extern __shared__ __align__(16) float cache[];
  __shared__ float red[32], slot[2];
  __shared__ int redi[32], islot;
  const int tid = threadIdx.x;
  const int rank = blockIdx.x % p.shares;
  const int64_t line = blockIdx.x / p.shares;
  int64_t xb = 0, yb = 0, wb = 0, rem = line;
  for (int d = p.nk - 1; d >= 0; --d) {
    const int64_t c = rem % p.kshape[d];
    rem /= p.kshape[d];
    xb += c * p.kxs[d];
    yb += c * p.kys[d];
    wb += c * p.kws[d];
  }
  const uint32_t begin = rank * p.share, end = min(begin + p.share, p.R);
  // f(element of the share, its run, its place in the run, elements) for the parts of runs that the share holds, by one warp
  auto parts = [&](auto f) {
    const uint32_t first = begin < end ? begin / p.R2 : 0, n = begin < end ? (end - 1) / p.R2 - first + 1 : 0;
    for (uint32_t k = tid; k < n && tid < 32; k += 32) {
      const uint32_t run = first + k, lo = max(begin, run * p.R2), hi = min(end, (run + 1) * p.R2);
      f(lo - begin, run, lo - run * p.R2, hi - lo);
    }
  };
  if constexpr (BULK) {
    __shared__ __align__(8) uint64_t arrived;
    __shared__ int abort_word;
    if (tid == 0) {
      abort_word = 0;
      mbar_init(&arrived, 1);
      fence_mbar_init();
      mbar_expect_tx(&arrived, (begin < end ? end - begin : 0) * 4);
    }
    __syncthreads();
    parts([&](uint32_t at, uint32_t run, uint32_t off, uint32_t n) {
      share_copy_in(cache + at, static_cast<const float*>(p.x) + xb + run * p.xs1 + off, n * 4, &arrived);
    });
    if (!mbar_wait(&arrived, 0, &abort_word)) atomicExch(p.status, YTC_TIMEOUT);
  }
  auto load = [&](uint32_t r) {
    const uint32_t r1 = p.R2 == p.R ? 0u : r / p.R2;
    const int64_t o = xb + r1 * p.xs1 + (r - r1 * p.R2);
    if constexpr (VEC == 4) return load4(p.x, o, p.dt_in);
    else return F4{{load_as_f32(p.x, o, p.dt_in), 0.f, 0.f, 0.f}};
  };
  auto cached = [&](uint32_t r) {
    if (!BULK && !p.cached) return load(r);
    if constexpr (VEC == 4) {
      const float4 t = *reinterpret_cast<const float4*>(cache + (r - begin));
      return F4{{t.x, t.y, t.z, t.w}};
    } else {
      return F4{{cache[r - begin], 0.f, 0.f, 0.f}};
    }
  };
  auto weights = [&](const void* src, int64_t o) {
    F4 r;
    r.v[0] = load_as_f32(src, o, p.dt_w);
#pragma unroll
    for (int e = 1; e < VEC; ++e) r.v[e] = p.ws2 == 0 ? r.v[0] : load_as_f32(src, o + e * p.ws2, p.dt_w);
    return r;
  };
  auto sweep = [&](bool first, auto f) {
    constexpr uint32_t STEP = THREADS * VEC;
    for (uint32_t r0 = begin + tid * VEC; r0 < end; r0 += STEP * SHARE_UNROLL) {
      F4 x[SHARE_UNROLL];
#pragma unroll
      for (int u = 0; u < SHARE_UNROLL; ++u)
        if (r0 + u * STEP < end) x[u] = first && !BULK ? load(r0 + u * STEP) : cached(r0 + u * STEP);
#pragma unroll
      for (int u = 0; u < SHARE_UNROLL; ++u) {
        const uint32_t r = r0 + u * STEP;
        if (r >= end) break;
        if (first && !BULK && p.cached && OP != OP_SUM && OP != OP_MEAN && OP != OP_MAX) {
          if constexpr (VEC == 4) *reinterpret_cast<float4*>(cache + (r - begin)) = make_float4(x[u].v[0], x[u].v[1], x[u].v[2], x[u].v[3]);
          else cache[r - begin] = x[u].v[0];
        }
#pragma unroll
        for (int e = 0; e < VEC; ++e) f(x[u].v[e], r + e);
      }
    }
  };
  line_passes<OP>(
      p, sweep,
      [&](float v, int k) { return over_shares(group_sum<THREADS>(v, red, 0, tid), &slot[k], tid == 0, p.shares, ShareSum{}); },
      [&](float v, int k) { return over_shares(group_max<THREADS>(v, red, 0, tid), &slot[k], tid == 0, p.shares, ShareMax{}); },
      [&](MaxIdx m) { return over_shares(group_maxidx<THREADS>(m, red, redi, 0, tid), &slot[0], &islot, tid == 0, p.shares); },
      [&](auto g) {
        constexpr uint32_t STEP = THREADS * VEC;
        if constexpr (BULK) {  // results over the cache, then out (gamma and beta belong to the line)
          const float w = p.w ? load_as_f32(p.w, wb, p.dt_w) : 1.f, b = p.b ? load_as_f32(p.b, wb, p.dt_w) : 0.f;
#pragma unroll 2
          for (uint32_t r = begin + tid * VEC; r < end; r += STEP) {
            F4 v = cached(r);
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
              const float x = g(v.v[e]);
              v.v[e] = p.w && p.b ? fmaf(x, w, b) : p.w ? x * w : p.b ? x + b : x;
            }
            *reinterpret_cast<float4*>(cache + (r - begin)) = make_float4(v.v[0], v.v[1], v.v[2], v.v[3]);
          }
          fence_proxy_async_smem();
          __syncthreads();
          parts([&](uint32_t at, uint32_t run, uint32_t off, uint32_t n) {
            share_copy_out(static_cast<float*>(p.y) + yb + run * p.ys1 + off, cache + at, n * 4);
          });
          if (tid < 32) {
            tma_store_commit();
            tma_store_wait_all<0>();
          }
          return;
        }
        // (gamma and beta of several trips are asked for before the first result is stored: one trip to the L2 for all)
        for (uint32_t r0 = begin + tid * VEC; r0 < end; r0 += STEP * SHARE_UNROLL) {
          F4 v[SHARE_UNROLL], wv[SHARE_UNROLL], bv[SHARE_UNROLL];
#pragma unroll
          for (int u = 0; u < SHARE_UNROLL; ++u) {
            const uint32_t r = r0 + u * STEP;
            if (r >= end) break;
            const uint32_t r1 = p.R2 == p.R ? 0u : r / p.R2;
            const int64_t wo = wb + r1 * p.ws1 + (r - r1 * p.R2) * p.ws2;
            v[u] = cached(r);
            if (p.w) wv[u] = weights(p.w, wo);
            if (p.b) bv[u] = weights(p.b, wo);
          }
#pragma unroll
          for (int u = 0; u < SHARE_UNROLL; ++u) {
            const uint32_t r = r0 + u * STEP;
            if (r >= end) break;
            const uint32_t r1 = p.R2 == p.R ? 0u : r / p.R2;
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
              v[u].v[e] = g(v[u].v[e]);
              if (p.w) v[u].v[e] *= wv[u].v[e];
              if (p.b) v[u].v[e] += bv[u].v[e];
            }
            const int64_t o = yb + r1 * p.ys1 + (r - r1 * p.R2);
            if constexpr (VEC == 4) store4(p.y, o, v[u], p.dt_out);
            else store_from_f32(p.y, o, v[u].v[0], p.dt_out);
          }
        }
      },
      [&](float v, int i) {
        if (rank != 0 || tid != 0) return;
        if (OP == OP_MAX && i == 0x7fffffff) {  // every element failed `>` (all NaN): the reference keeps element 0
          v = load_as_f32(p.x, xb, p.dt_in);
          i = 0;
        }
        store_from_f32(p.y, yb, v, p.dt_out);
        if (OP == OP_MAX && p.idx) p.idx[line] = i;
      });
  if (p.shares > 1) cluster_sync_all();  // the others may still read this CTA's partial results
}

template <int OP, int THREADS>
__global__ void __launch_bounds__(THREADS) column_kernel(const ShareParams p) {
  constexpr int ROWS = THREADS / 32;
  extern __shared__ __align__(16) float cache[];  // [share][32]
  __shared__ float red[ROWS][32], slot[2][32];
  __shared__ int redi[ROWS][32], islot[32];
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  const int rank = blockIdx.x % p.shares;
  const int64_t tiles = (p.cols + 31) / 32, item = blockIdx.x / p.shares;
  const int64_t outer = item / tiles, col = (item - outer * tiles) * 32 + lane;
  int64_t xb = col, yb = col, wb = col * p.cws, rem = outer;
  for (int d = p.nk - 1; d >= 0; --d) {
    const int64_t c = rem % p.kshape[d];
    rem /= p.kshape[d];
    xb += c * p.kxs[d];
    yb += c * p.kys[d];
    wb += c * p.kws[d];
  }
  const bool on = col < p.cols;
  const uint32_t begin = rank * p.share, end = on ? min(begin + p.share, p.R) : 0u;
  auto sweep = [&](bool first, auto f) {
    constexpr int U = 2 * SHARE_UNROLL;
    for (uint32_t r0 = begin + q; r0 < end; r0 += ROWS * U) {
      float x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t r = r0 + u * ROWS;
        if (r < end) x[u] = !first && p.cached ? cache[(r - begin) * 32 + lane] : load_as_f32(p.x, xb + r * p.xs1, p.dt_in);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t r = r0 + u * ROWS;
        if (r >= end) break;
        if (first && p.cached && OP != OP_SUM && OP != OP_MEAN && OP != OP_MAX) cache[(r - begin) * 32 + lane] = x[u];
        f(x[u], r);
      }
    }
  };
  auto down = [&](float v, auto f) {  // over the eight threads of a column, in their order
    red[q][lane] = v;
    __syncthreads();
    v = red[0][lane];
#pragma unroll
    for (int i = 1; i < ROWS; ++i) v = f(v, red[i][lane]);
    __syncthreads();
    return v;
  };
  line_passes<OP>(
      p, sweep, [&](float v, int k) { return over_shares(down(v, ShareSum{}), &slot[k][lane], q == 0, p.shares, ShareSum{}); },
      [&](float v, int k) { return over_shares(down(v, ShareMax{}), &slot[k][lane], q == 0, p.shares, ShareMax{}); },
      [&](MaxIdx m) {
        red[q][lane] = m.v;
        redi[q][lane] = m.i;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ROWS; ++i) m = max_combine(m, MaxIdx{red[i][lane], redi[i][lane]});
        return over_shares(m, &slot[0][lane], &islot[lane], q == 0, p.shares);
      },
      [&](auto g) {
        for (uint32_t r0 = begin + q; r0 < end; r0 += ROWS * SHARE_UNROLL) {
          float v[SHARE_UNROLL], wv[SHARE_UNROLL], bv[SHARE_UNROLL];
#pragma unroll
          for (int u = 0; u < SHARE_UNROLL; ++u) {
            const uint32_t r = r0 + u * ROWS;
            if (r >= end) break;
            v[u] = p.cached ? cache[(r - begin) * 32 + lane] : load_as_f32(p.x, xb + r * p.xs1, p.dt_in);
            if (p.w) wv[u] = load_as_f32(p.w, wb + r * p.ws1, p.dt_w);
            if (p.b) bv[u] = load_as_f32(p.b, wb + r * p.ws1, p.dt_w);
          }
#pragma unroll
          for (int u = 0; u < SHARE_UNROLL; ++u) {
            const uint32_t r = r0 + u * ROWS;
            if (r >= end) break;
            v[u] = g(v[u]);
            if (p.w) v[u] *= wv[u];
            if (p.b) v[u] += bv[u];
            store_from_f32(p.y, yb + r * p.ys1, v[u], p.dt_out);
          }
        }
      },
      [&](float v, int i) {
        if (rank != 0 || q != 0 || !on) return;
        if (OP == OP_MAX && i == 0x7fffffff) {
          v = load_as_f32(p.x, xb, p.dt_in);
          i = 0;
        }
        store_from_f32(p.y, yb, v, p.dt_out);
        if (OP == OP_MAX && p.idx) p.idx[outer * p.cols + col] = i;
      });
  if (p.shares > 1) cluster_sync_all();
}

// ------------------------------------------------------------------ few lines, long reductions
// sum / mean / max over very many elements per output (e.g. a whole-tensor sum) would leave all but a
// few SMs idle with one CTA per line. The reduced range of every line is cut into `chunks` pieces, one
// CTA each; the partial results go to a scratch buffer in global memory and a second small kernel
// combines them. The scratch holds chunks * lines (value, index) pairs.
struct SplitParams {
  LineParams lp;
  int chunks;
  int64_t chunk_len;
  int contiguous;  // the reduced elements of a line are one contiguous run in x
  float* part_val;
  int* part_idx;
};

template <int OP>
__global__ void __launch_bounds__(256) split_partial_kernel(const SplitParams sp) {
  __shared__ float red[32];
  __shared__ int redi[32];
  const LineParams& p = sp.lp;
  const int tid = threadIdx.x;
  const int chunk = blockIdx.x;
  const int64_t line = blockIdx.y;
  int64_t xb = 0, rem = line;
  for (int d = p.nk - 1; d >= 0; --d) {
    const int64_t c = rem % p.kshape[d];
    rem /= p.kshape[d];
    xb += c * p.kxs[d];
  }
  const int64_t r_begin = chunk * sp.chunk_len;
  const int64_t r_end = (r_begin + sp.chunk_len < p.R) ? r_begin + sp.chunk_len : p.R;
  int64_t xo, yo, wo;
  if constexpr (OP == OP_MAX) {
    MaxIdx m = {-CUDART_INF_F, 0x7fffffff};
    for (int64_t r = r_begin + tid; r < r_end; r += 256) {
      if (sp.contiguous) xo = r; else line_offsets(p, r, xo, yo, wo);
      m = max_combine(m, MaxIdx{load_as_f32(p.x, xb + xo, p.dt_in), static_cast<int>(r)});
    }
    m = group_maxidx<256>(m, red, redi, 0, tid);
    if (tid == 0) {
      sp.part_val[line * sp.chunks + chunk] = m.v;
      sp.part_idx[line * sp.chunks + chunk] = m.i;
    }
  } else {
    float s = 0.f;
    for (int64_t r = r_begin + tid; r < r_end; r += 256) {
      if (sp.contiguous) xo = r; else line_offsets(p, r, xo, yo, wo);
      s += load_as_f32(p.x, xb + xo, p.dt_in);
    }
    s = group_sum<256>(s, red, 0, tid);
    if (tid == 0) sp.part_val[line * sp.chunks + chunk] = s;
  }
}

template <int OP>
__global__ void __launch_bounds__(32) split_finish_kernel(const SplitParams sp) {
  const LineParams& p = sp.lp;
  const int lane = threadIdx.x;
  const int64_t line = blockIdx.x;
  if constexpr (OP == OP_MAX) {
    MaxIdx m = {-CUDART_INF_F, 0x7fffffff};
    for (int c = lane; c < sp.chunks; c += 32)
      m = max_combine(m, MaxIdx{sp.part_val[line * sp.chunks + c], sp.part_idx[line * sp.chunks + c]});
    m = group_maxidx<32>(m, nullptr, nullptr, 0, lane);
    if (lane == 0) {
      int64_t xb = 0, rem = line;
      for (int d = p.nk - 1; d >= 0; --d) {
        const int64_t c = rem % p.kshape[d];
        rem /= p.kshape[d];
        xb += c * p.kxs[d];
      }
      if (m.i == 0x7fffffff) {
        m.v = load_as_f32(p.x, xb, p.dt_in);
        m.i = 0;
      }
      store_from_f32(p.y, line, m.v, p.dt_out);
      if (p.idx) p.idx[line] = m.i;
    }
  } else {
    float s = 0.f;
    for (int c = lane; c < sp.chunks; c += 32) s += sp.part_val[line * sp.chunks + c];
    s = group_sum<32>(s, nullptr, 0, lane);
    if (lane == 0) store_from_f32(p.y, line, OP == OP_MEAN ? s / static_cast<float>(p.R) : s, p.dt_out);
  }
}

// ------------------------------------------------------------------ host side
struct NdArgs {
  const int64_t* shape;
  const int64_t* xs;
  const int64_t* ys;
  int ndim;
  const int* axes;
  int naxes;
};

static int normalize_axes(const NdArgs& a, int* ax, bool* used, const char* who) {
  if (a.ndim < 1 || a.ndim > MAXD) {
    set_last_error("%s: ndim %d outside [1, %d]", who, a.ndim, MAXD);
    return YTC_INVALID_ARG;
  }
  if (a.naxes < 1 || a.naxes > a.ndim) {
    set_last_error("%s: %d axes for %d dims", who, a.naxes, a.ndim);
    return YTC_INVALID_ARG;
  }
  for (int d = 0; d < a.ndim; ++d) used[d] = false;
  for (int i = 0; i < a.naxes; ++i) {
    const int v = ((a.axes[i] % a.ndim) + a.ndim) % a.ndim;
    if (used[v]) {
      set_last_error("%s: axis %d listed twice", who, v);
      return YTC_INVALID_ARG;
    }
    used[v] = true;
    ax[i] = v;
  }
  for (int d = 0; d < a.ndim; ++d)
    if (a.shape[d] < 0) {
      set_last_error("%s: negative extent", who);
      return YTC_INVALID_ARG;
    }
  return YTC_OK;
}

template <int OP, int G, int VEC>
static void launch_row(const RowParams& p, cudaStream_t st) {
  constexpr int THREADS = G < 256 ? 256 : G;
  constexpr int RPC = THREADS / G;
  const int64_t row_blocks = (p.rows + RPC - 1) / RPC;
  const int64_t cap = static_cast<int64_t>(sm_count()) * (2048 / THREADS) * 2;
  const int grid = static_cast<int>(row_blocks < cap ? row_blocks : cap);
  (void)launch_overlapped(row_kernel<OP, G, VEC>, dim3(grid), dim3(THREADS), 0, st, p);
  count_launch();
}
template <int OP, int VEC>
static void launch_row_g(const RowParams& p, cudaStream_t st) {
  if (p.L <= 512) launch_row<OP, 32, VEC>(p, st);
  else if (p.L <= 2048) launch_row<OP, 128, VEC>(p, st);
  else if (p.L <= 4096) launch_row<OP, 256, VEC>(p, st);
  else if (p.L <= 8192) launch_row<OP, 512, VEC>(p, st);
  else launch_row<OP, 1024, VEC>(p, st);
}
template <int VEC>
static void launch_row_op(int op, const RowParams& p, cudaStream_t st) {
  switch (op) {
    case OP_SOFTMAX: launch_row_g<OP_SOFTMAX, VEC>(p, st); break;
    case OP_RMSNORM: launch_row_g<OP_RMSNORM, VEC>(p, st); break;
    case OP_LAYERNORM: launch_row_g<OP_LAYERNORM, VEC>(p, st); break;
    case OP_CHAIN:
      if constexpr (VEC == 4) launch_row_g<OP_CHAIN, VEC>(p, st);
      break;
    case OP_SUM: launch_row_g<OP_SUM, VEC>(p, st); break;
    case OP_MEAN: launch_row_g<OP_MEAN, VEC>(p, st); break;
    default: launch_row_g<OP_MAX, VEC>(p, st); break;
  }
}
template <int OP>
static void launch_line(const LineParams& p, bool per_thread, cudaStream_t st) {
  if (per_thread) {
    const int64_t blocks = (p.lines + 127) / 128;
    const int64_t cap = static_cast<int64_t>(sm_count()) * 32;
    line_kernel<OP, true><<<static_cast<int>(blocks < cap ? blocks : cap), 128, 0, st>>>(p);
  } else {
    const int64_t cap = static_cast<int64_t>(sm_count()) * 32;
    line_kernel<OP, false><<<static_cast<int>(p.lines < cap ? p.lines : cap), 128, 0, st>>>(p);
  }
  count_launch();
}
static void launch_line_op(int op, const LineParams& p, bool per_thread, cudaStream_t st) {
  switch (op) {
    case OP_SOFTMAX: launch_line<OP_SOFTMAX>(p, per_thread, st); break;
    case OP_RMSNORM: launch_line<OP_RMSNORM>(p, per_thread, st); break;
    case OP_LAYERNORM: launch_line<OP_LAYERNORM>(p, per_thread, st); break;
    case OP_LPNORM: launch_line<OP_LPNORM>(p, per_thread, st); break;
    case OP_SUM: launch_line<OP_SUM>(p, per_thread, st); break;
    case OP_MEAN: launch_line<OP_MEAN>(p, per_thread, st); break;
    default: launch_line<OP_MAX>(p, per_thread, st); break;
  }
}

// one thread per line when neighbouring lines sit next to each other in memory
static bool line_per_thread(const LineParams& p) {
  return p.nk > 0 && p.kxs[p.nk - 1] == 1 && p.kshape[p.nk - 1] >= 32 && p.lines >= 4096;
}
// Lines shorter than these stay with line_kernel. Measured, fp32, line_kernel / here: softmax over the first axis of 12 x 600000 81 /
// 84 us, 16 x 600000 108 / 92, 5 x 300000 22 / 35, 2 x 4000000 100 / 354; sum of 24 x 600000 48.6 / 47.7, 32 x 600000 65 / 43, 3 x
// 1000000 21 / 47; over the outer axes of 4 x 30000 x w, softmax: w = 48 127 / 160, 72 178 / 166, 512 1036 / 261.
constexpr int SHORT_COLUMNS = 14, SHORT_COLUMNS_REDUCED = 32, SHORT_SPANS = 256;

// Launches span_kernel or column_kernel where the dims allow it; YTC_UNSUPPORTED: nothing was launched. `ws`: strides of gamma
// and beta per dim, null: they are laid out like the reduced dims.
template <class K>
static int launch_share(K kernel, const ShareParams& p, int64_t blocks, int threads, size_t smem, cudaStream_t st) {
  if (p.shares == 1 && smem <= 32 * 1024) {  // the smallest calls: nothing to look up, an ordinary launch
    kernel<<<static_cast<unsigned>(blocks), threads, smem, st>>>(p);
    count_launch();
    YTC_CUDA(cudaGetLastError());
    return YTC_OK;
  }
  const int s = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), static_cast<int>(smem));
  if (s != YTC_OK) return s;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.shares;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  YTC_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
  count_launch();
  return YTC_OK;
}
template <int OP, int THREADS>
static int launch_share_op(int kind, const ShareParams& p, int64_t blocks, size_t smem, cudaStream_t st) {
  if (kind == 0) return launch_share(column_kernel<OP, THREADS>, p, blocks, THREADS, smem, st);
  if constexpr (OP != OP_SUM && OP != OP_MEAN && OP != OP_MAX)
    if (p.bulk) return launch_share(span_kernel<OP, 4, THREADS, true>, p, blocks, THREADS, smem, st);
  return kind == 4 ? launch_share(span_kernel<OP, 4, THREADS, false>, p, blocks, THREADS, smem, st)
                   : launch_share(span_kernel<OP, 1, THREADS, false>, p, blocks, THREADS, smem, st);
}
template <int OP>
static int launch_share_threads(int kind, const ShareParams& p, int64_t blocks, size_t smem, bool many, cudaStream_t st) {
  return many ? launch_share_op<OP, 1024>(kind, p, blocks, smem, st) : launch_share_op<OP, 256>(kind, p, blocks, smem, st);
}
static int launch_shared_line(int op, const LineParams& lp, const NdArgs& a, const int64_t* ws, bool reduce_out, cudaStream_t st) {
  if (lp.R < 2 || lp.R > 0x3fffffff) return YTC_UNSUPPORTED;
  ShareParams p{};
  p.x = lp.x; p.y = lp.y; p.w = lp.w; p.b = lp.b; p.idx = lp.idx;
  p.eps = lp.eps; p.lp = lp.lp; p.dt_in = lp.dt_in; p.dt_out = lp.dt_out; p.dt_w = lp.dt_w;
  p.R = static_cast<uint32_t>(lp.R);
  // the reduced dims in listed order, neighbours joined where x, y and the weights allow it
  int nr = 0;
  int64_t shape[MAXD], xs[MAXD], ys[MAXD], wst[MAXD];
  for (int i = 0; i < lp.nr; ++i) {
    if (lp.rshape[i] == 1) continue;
    const int ax = ((a.axes[i] % a.ndim) + a.ndim) % a.ndim;
    const int64_t wd = ws ? ws[ax] : lp.rws[i];
    if (nr > 0 && xs[nr - 1] == lp.rxs[i] * lp.rshape[i] && (reduce_out || ys[nr - 1] == lp.rys[i] * lp.rshape[i]) &&
        (!lp.w || wst[nr - 1] == wd * lp.rshape[i])) {
      shape[nr - 1] *= lp.rshape[i];
      xs[nr - 1] = lp.rxs[i];
      ys[nr - 1] = lp.rys[i];
      wst[nr - 1] = wd;
      continue;
    }
    shape[nr] = lp.rshape[i];
    xs[nr] = lp.rxs[i];
    ys[nr] = lp.rys[i];
    wst[nr++] = wd;
  }
  // the kept dims
  for (int d = 0, k = 0; d < a.ndim; ++d) {
    bool reduced = false;
    for (int i = 0; i < a.naxes; ++i) reduced = reduced || ((a.axes[i] % a.ndim) + a.ndim) % a.ndim == d;
    if (reduced) continue;
    if (lp.kshape[k] != 1) {
      p.kshape[p.nk] = lp.kshape[k];
      p.kxs[p.nk] = lp.kxs[k];
      p.kys[p.nk] = lp.kys[k];
      p.kws[p.nk++] = ws ? ws[d] : 0;
    }
    ++k;
  }
  const int sms = sm_count();
  int kind;
  int64_t lines;       // items of one cluster each
  uint32_t floats = 1;  // of the cache per element of a share
  if (nr <= 2 && xs[nr - 1] == 1 && (reduce_out || ys[nr - 1] == 1)) {
    p.R2 = static_cast<uint32_t>(shape[nr - 1]);
    p.ws2 = wst[nr - 1];
    if (nr == 2) {
      p.xs1 = xs[0];
      p.ys1 = ys[0];
      p.ws1 = wst[0];
    }
    const int ein = dtype_size(lp.dt_in), eout = dtype_size(lp.dt_out);
    bool quads = p.R2 % 4 == 0 && reinterpret_cast<uint64_t>(lp.x) % (4 * ein) == 0 && p.xs1 % 4 == 0 &&
                 (reduce_out || (reinterpret_cast<uint64_t>(lp.y) % (4 * eout) == 0 && p.ys1 % 4 == 0));
    for (int d = 0; d < p.nk; ++d) quads = quads && p.kxs[d] % 4 == 0 && (reduce_out || p.kys[d] % 4 == 0);
    kind = quads ? 4 : 1;
    lines = lp.lines;
  } else if (nr == 1 && p.nk > 0 && p.kxs[p.nk - 1] == 1 && p.kys[p.nk - 1] == 1 && p.kshape[p.nk - 1] >= 8) {
    --p.nk;
    p.cols = p.kshape[p.nk];
    p.cws = p.kws[p.nk];
    p.xs1 = xs[0];
    p.ys1 = ys[0];
    p.ws1 = wst[0];
    kind = 0;
    lines = lp.lines / p.cols * ((p.cols + 31) / 32);
    floats = 32;
  } else {
    return YTC_UNSUPPORTED;
  }
  // Short lines stay with line_kernel, whose CTAs are smaller and which takes a thread per line where lines lie side by side.
  // With gamma and beta (one launch here, three there) only where the lines are so many that the launches don't matter.
  const bool keeps = op != OP_SUM && op != OP_MEAN && op != OP_MAX;
  if (kind == 0 ? lp.R < (keeps ? SHORT_COLUMNS : SHORT_COLUMNS_REDUCED) && line_per_thread(lp) && (!ws || lp.lines > (1 << 20))
                : lp.R < SHORT_SPANS && (!ws || lp.lines > (1 << 15)))
    return YTC_UNSUPPORTED;
  // Shares: enough CTAs for two per SM while a share keeps 2048 elements, and shares of half an SM's shared memory.
  int shares = 1;
  auto share_of = [&](int n) { return ((p.R + n - 1) / n + 3) / 4 * 4; };
  while (shares < MAX_SHARES && ((lines * shares < 2 * sms && static_cast<uint64_t>(share_of(shares)) * floats >= 4096) ||
                                 static_cast<uint64_t>(share_of(shares)) * floats > CACHE_FLOATS / 2))
    shares *= 2;
  if (lines * shares > 0x7fffffff) return YTC_UNSUPPORTED;
  p.shares = shares;
  p.share = share_of(shares);
  p.cached = keeps && static_cast<uint64_t>(p.share) * floats <= CACHE_FLOATS;
  const size_t smem = p.cached ? static_cast<size_t>(p.share) * floats * 4 : 0;
  // Runs of 512 bytes and more, fp32, with one gamma and beta a line or none: copied whole, all of a share at once, instead of 64
  // bytes a thread and trip. Registers / copies, calls back to back: batchNorm of 16 x 96 x 56 x 56 20.9 / 12.2 us, 256 channels of 512
  // values 4.3 / 3.8. With gamma and beta inside the line (groupNorm) a second pass asks for them per element and the copies only wait
  // one for the other: 32 x 256 x 14 x 14 in 8 groups 16.8 / 20.3. 16-bit shares have no such form, and keep the code without it: the
  // two in one kernel cost them 5 to 9 %.
  p.bulk = kind == 4 && p.cached && (p.R2 == p.R || p.R2 >= 128) && lp.dt_in == YTC_F32 && lp.dt_out == YTC_F32 &&
           (!(lp.w || lp.b) || (p.ws1 == 0 && p.ws2 == 0));
  if (p.bulk && !(p.status = device_status_word())) p.bulk = 0;
  // A share of which only one fits an SM needs more threads to keep enough loads in flight (batchNorm, bf16, 32 x 256 x 112 x
  // 112: 1617 us with 256 threads, 605 with 1024); where more fit, 256 are faster (16 x 96 x 56 x 56 fp32: 25 us, 37).
  const bool many = smem > 110 * 1024;
  switch (op) {
    case OP_SOFTMAX: return launch_share_threads<OP_SOFTMAX>(kind, p, lines * shares, smem, many, st);
    case OP_RMSNORM: return launch_share_threads<OP_RMSNORM>(kind, p, lines * shares, smem, many, st);
    case OP_LAYERNORM: return launch_share_threads<OP_LAYERNORM>(kind, p, lines * shares, smem, many, st);
    case OP_LPNORM: return launch_share_threads<OP_LPNORM>(kind, p, lines * shares, smem, many, st);
    case OP_SUM: return launch_share_threads<OP_SUM>(kind, p, lines * shares, smem, many, st);
    case OP_MEAN: return launch_share_threads<OP_MEAN>(kind, p, lines * shares, smem, many, st);
    default: return launch_share_threads<OP_MAX>(kind, p, lines * shares, smem, many, st);
  }
}

// Shared driver of all N-d reductions. `reduce_out` = the output keeps size-1 dims on the reduced axes
// (sum / mean / max) instead of the input's shape (softmax / norms).
static int run_nd(int op, int dt_in, int dt_out, int dt_w, const void* x, void* y, const void* w, const void* b,
                  int* idx, const NdArgs& a, float eps, bool reduce_out, cudaStream_t st, const char* who,
                  void* scratch = nullptr, size_t scratch_bytes = 0, float lp = 2.f, const int64_t* ws = nullptr) {
  int ax[MAXD];
  bool used[MAXD];
  int s = normalize_axes(a, ax, used, who);
  if (s != YTC_OK) return s;
  YTC_REQUIRE(dt_in >= 0 && dt_in <= 2 && dt_out >= 0 && dt_out <= 2 && dt_w >= 0 && dt_w <= 2, "%s: bad dtype", who);
  int64_t total = 1, R = 1;
  for (int d = 0; d < a.ndim; ++d) total *= a.shape[d];
  for (int i = 0; i < a.naxes; ++i) R *= a.shape[ax[i]];
  if (total == 0) return YTC_OK;
  YTC_REQUIRE(x && y, "%s: null tensor", who);
  YTC_REQUIRE(R <= 0x7fffffffll, "%s: more than 2^31 elements per reduction", who);
  const int64_t lines = total / R;

  // Fast path: the reduced axes are the trailing dims in ascending listed order, contiguous in x (and in y
  // for the shape-preserving ops).
  bool trailing = true;
  for (int i = 0; i < a.naxes; ++i)
    if (ax[i] != a.ndim - a.naxes + i) trailing = false;
  if (trailing) {
    int64_t exp = 1;
    for (int d = a.ndim - 1; d >= a.ndim - a.naxes; --d) {
      if (a.shape[d] != 1 && (a.xs[d] != exp || (!reduce_out && a.ys[d] != exp))) trailing = false;
      exp *= a.shape[d];
    }
  }
  // kept dims must collapse into one row stride
  int64_t x_rs = R, y_rs = reduce_out ? 1 : R;
  if (trailing) {
    int64_t expx = -1, expy = -1;
    for (int d = a.ndim - a.naxes - 1; d >= 0; --d) {
      if (a.shape[d] == 1) continue;
      if (expx < 0) {
        expx = a.xs[d];
        expy = a.ys[d];
        x_rs = a.xs[d];
        y_rs = a.ys[d];
      } else if (a.xs[d] != expx || a.ys[d] != expy) {
        trailing = false;
        break;
      }
      expx *= a.shape[d];
      expy *= a.shape[d];
    }
    if (reduce_out && lines > 1 && y_rs != 1) trailing = false;
  }
  const int esz_in = dtype_size(dt_in), esz_out = dtype_size(dt_out);
  const bool spread = ws != nullptr;  // gamma / beta by strides of their own: the span kernel alone knows them
  // Rows that can't be read four at a time take single loads: 32 lanes still read neighbours. Measured, rmsNorm bf16
  // 4096 x 8191: 77 us, 323 with line_kernel; 8192 wide 4 at a time 39.
  const bool quads = R % 4 == 0 && (reinterpret_cast<uint64_t>(x) % (4 * esz_in)) == 0 && x_rs % 4 == 0 &&
                     (reduce_out || ((reinterpret_cast<uint64_t>(y) % (4 * esz_out)) == 0 && y_rs % 4 == 0)) &&
                     (!w || reinterpret_cast<uint64_t>(w) % (4 * dtype_size(dt_w)) == 0) &&
                     (!b || reinterpret_cast<uint64_t>(b) % (4 * dtype_size(dt_w)) == 0);
  // (lines of one element side by side: a thread each, line_kernel)
  const int last_kept = a.ndim - a.naxes - 1;
  const bool single = R == 1 && x_rs == 1 && lines >= 4096 && last_kept >= 0 && a.shape[last_kept] >= 32;
  if (op != OP_LPNORM && trailing && !spread && !single && R <= 16384 && x_rs >= 0 && y_rs >= 0) {
    RowParams p;
    p.x = x; p.y = y; p.w = w; p.b = b; p.idx = idx;
    p.rows = lines; p.L = static_cast<int>(R);
    p.x_rs = x_rs; p.y_rs = y_rs; p.r_rows = 1; p.eps = eps;
    p.dt_in = dt_in; p.dt_out = dt_out; p.dt_w = dt_w;
    if (quads) launch_row_op<4>(op, p, st);
    else launch_row_op<1>(op, p, st);
    YTC_CUDA(cudaGetLastError());
    return YTC_OK;
  }

  LineParams p;
  p.x = x; p.y = y; p.w = w; p.b = b; p.idx = idx;
  p.nk = 0; p.nr = a.naxes;
  p.eps = eps; p.lp = lp; p.dt_in = dt_in; p.dt_out = dt_out; p.dt_w = dt_w;
  p.lines = lines; p.R = R;
  for (int d = 0; d < a.ndim; ++d)
    if (!used[d]) {
      p.kshape[p.nk] = a.shape[d];
      p.kxs[p.nk] = a.xs[d];
      p.kys[p.nk] = a.ys[d];
      ++p.nk;
    }
  // weight layout: contiguous over the reduced dims in ASCENDING axis order (the reference views the
  // weight's memory with shape [1,..,size(axis),..,1], src/ytensor_function.inl:137-158)
  int64_t wstride[MAXD];
  {
    int64_t acc = 1;
    for (int d = a.ndim - 1; d >= 0; --d)
      if (used[d]) {
        wstride[d] = acc;
        acc *= a.shape[d];
      }
  }
  for (int i = 0; i < a.naxes; ++i) {
    p.rshape[i] = a.shape[ax[i]];
    p.rxs[i] = a.xs[ax[i]];
    p.rys[i] = reduce_out ? 0 : a.ys[ax[i]];
    p.rws[i] = wstride[ax[i]];
  }
  // few outputs, long reductions: split every line over several CTAs through a scratch buffer
  if (reduce_out && !spread && lines <= 2 * sm_count() && R >= 32768) {
    SplitParams sp;
    sp.lp = p;
    int64_t chunks = (4ll * sm_count() + lines - 1) / lines;
    const int64_t max_chunks = (R + 2047) / 2048;
    if (chunks > max_chunks) chunks = max_chunks;
    if (chunks > 4096) chunks = 4096;
    sp.chunks = static_cast<int>(chunks);
    sp.chunk_len = (R + chunks - 1) / chunks;
    bool contig = true;
    {
      int64_t exp = 1;
      for (int i = a.naxes - 1; i >= 0; --i) {
        if (p.rshape[i] != 1 && p.rxs[i] != exp) contig = false;
        exp *= p.rshape[i];
      }
    }
    sp.contiguous = contig ? 1 : 0;
    const size_t need = static_cast<size_t>(lines) * chunks;
    const WorkspaceScope workspace(st);
    void* ws = scratch ? scratch : device_workspace(need * 8, st);
    if (!ws) {
      set_last_error("%s: cannot allocate %zu bytes of scratch", who, need * 8);
      return YTC_CUDA_ERROR;
    }
    if (scratch && need * 8 > scratch_bytes) {
      set_last_error("%s: needs %zu bytes of scratch, the fixed buffer holds %zu", who, need * 8, scratch_bytes);
      return YTC_INVALID_ARG;
    }
    sp.part_val = static_cast<float*>(ws);
    sp.part_idx = reinterpret_cast<int*>(sp.part_val + need);
    dim3 grid(static_cast<unsigned>(chunks), static_cast<unsigned>(lines));
    if (op == OP_SUM) {
      split_partial_kernel<OP_SUM><<<grid, 256, 0, st>>>(sp);
      split_finish_kernel<OP_SUM><<<static_cast<unsigned>(lines), 32, 0, st>>>(sp);
    } else if (op == OP_MEAN) {
      split_partial_kernel<OP_MEAN><<<grid, 256, 0, st>>>(sp);
      split_finish_kernel<OP_MEAN><<<static_cast<unsigned>(lines), 32, 0, st>>>(sp);
    } else {
      split_partial_kernel<OP_MAX><<<grid, 256, 0, st>>>(sp);
      split_finish_kernel<OP_MAX><<<static_cast<unsigned>(lines), 32, 0, st>>>(sp);
    }
    count_launch(2);
    YTC_CUDA(cudaGetLastError());
    return YTC_OK;
  }
  const int shared = launch_shared_line(op, p, a, ws, reduce_out, st);
  if (shared != YTC_UNSUPPORTED) return shared;
  if (spread) {
    set_last_error("%s: these strides are not supported", who);
    return YTC_UNSUPPORTED;
  }
  launch_line_op(op, p, line_per_thread(p), st);
  YTC_CUDA(cudaGetLastError());
  return YTC_OK;
}

int rmsnorm_planes(const float* x, const float* w, uint16_t* planes, int64_t rows, int hidden, float eps, cudaStream_t st) {
  YTC_REQUIRE(hidden % 4 == 0 && hidden <= RMS_PLANES_MAX, "rmsnorm_planes: rows of %d", hidden);
  RowParams p{};
  p.x = x; p.y = planes; p.w = w;
  p.rows = rows; p.L = hidden; p.x_rs = p.y_rs = hidden; p.r_rows = 1; p.eps = eps;
  p.dt_in = p.dt_w = YTC_F32; p.dt_out = YTC_BF16;
  launch_row_g<OP_RMSPLANES, 4>(p, st);
  YTC_CUDA(cudaGetLastError());
  return YTC_OK;
}

// ------------------------------------------------------------------ fixed scratch for callers that cannot allocate
// Partial results of the split reduction for ytcuda_reduce_noalloc live here instead of in a cudaMalloc'ed
// workspace: 8192 (value, index) pairs. Every GPU that loads the library carries these 64 KiB until exit.
constexpr size_t NOALLOC_SCRATCH_BYTES = 64 * 1024;
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];
// Bytes of the array a call may use (ytcuda_reduce_noalloc_set_limit); never more than the array holds.
static std::atomic<size_t> g_noalloc_limit{NOALLOC_SCRATCH_BYTES};

// The array's name is only a host-side handle here: the device address has to be asked for, once per device,
// while that device is current.
static void* noalloc_scratch_address() {
  static void* addr[16] = {nullptr};
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) {
    set_last_error("ytcuda_reduce_noalloc: cannot identify the current device");
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      set_last_error("ytcuda_reduce_noalloc: cudaGetSymbolAddress failed with %d (%s)", static_cast<int>(e),
                     cudaGetErrorString(e));
      return nullptr;
    }
    addr[dev] = p;
  }
  return addr[dev];
}

}  // namespace ytk

using namespace ytk;

extern "C" {

int ytcuda_reduce_noalloc(int op, int dt_in, int dt_out, const void* x, void* y, int32_t* index, const int64_t* shape,
                          const int64_t* xstrides, int ndim, const int* axes, int naxes, void* stream) {
  YTC_REQUIRE(op >= 0 && op <= 2, "ytcuda_reduce_noalloc: op must be 0 (sum), 1 (mean) or 2 (max)");
  YTC_REQUIRE(shape && xstrides && axes, "ytcuda_reduce_noalloc: null shape/strides/axes");
  YTC_REQUIRE(ndim >= 1 && ndim <= MAXD, "ytcuda_reduce_noalloc: ndim %d outside [1, %d]", ndim, MAXD);
  void* scratch = noalloc_scratch_address();
  if (!scratch) return YTC_CUDA_ERROR;
  int64_t ys[MAXD];
  {
    bool red[MAXD] = {false};
    for (int i = 0; i < naxes && i < MAXD; ++i) red[((axes[i] % ndim) + ndim) % ndim] = true;
    int64_t acc = 1;
    for (int d = ndim - 1; d >= 0; --d) {
      ys[d] = red[d] ? 0 : acc;
      if (!red[d]) acc *= shape[d];
    }
  }
  NdArgs a{shape, xstrides, ys, ndim, axes, naxes};
  const int rop = op == 0 ? OP_SUM : op == 1 ? OP_MEAN : OP_MAX;
  return run_nd(rop, dt_in, dt_out, YTC_F32, x, y, nullptr, nullptr, index, a, 0.f, true,
                static_cast<cudaStream_t>(stream), "ytcuda_reduce_noalloc", scratch, g_noalloc_limit.load());
}

int ytcuda_reduce_noalloc_set_limit(uint64_t bytes) {
  YTC_REQUIRE(bytes <= NOALLOC_SCRATCH_BYTES, "ytcuda_reduce_noalloc_set_limit: %llu bytes asked for, the array holds %zu",
              static_cast<unsigned long long>(bytes), NOALLOC_SCRATCH_BYTES);
  g_noalloc_limit.store(bytes == 0 ? NOALLOC_SCRATCH_BYTES : static_cast<size_t>(bytes));
  return YTC_OK;
}

int ytcuda_softmax(int dt_in, int dt_out, const void* x, void* y, const int64_t* shape, const int64_t* xstrides,
                   const int64_t* ystrides, int ndim, const int* axes, int naxes, void* stream) {
  YTC_REQUIRE(shape && xstrides && ystrides && axes, "ytcuda_softmax: null shape/strides/axes");
  NdArgs a{shape, xstrides, ystrides, ndim, axes, naxes};
  return run_nd(OP_SOFTMAX, dt_in, dt_out, YTC_F32, x, y, nullptr, nullptr, nullptr, a, 0.f, false,
                static_cast<cudaStream_t>(stream), "ytcuda_softmax");
}

int ytcuda_normalize(int dt_in, int dt_out, const void* x, void* y, const int64_t* shape, const int64_t* xstrides,
                     const int64_t* ystrides, int ndim, const int* axes, int naxes, float p, float eps, void* stream) {
  YTC_REQUIRE(shape && xstrides && ystrides && axes, "ytcuda_normalize: null shape/strides/axes");
  YTC_REQUIRE(p > 0.f, "yt::function::normalize: p must be positive");
  NdArgs a{shape, xstrides, ystrides, ndim, axes, naxes};
  return run_nd(OP_LPNORM, dt_in, dt_out, YTC_F32, x, y, nullptr, nullptr, nullptr, a, eps, false,
                static_cast<cudaStream_t>(stream), "ytcuda_normalize", nullptr, 0, p);
}

int ytcuda_rmsnorm(int dt_in, int dt_out, int dt_w, const void* x, const void* weight, void* y, const int64_t* shape,
                   const int64_t* xstrides, const int64_t* ystrides, int ndim, const int* axes, int naxes, float eps,
                   void* stream) {
  YTC_REQUIRE(shape && xstrides && ystrides && axes, "ytcuda_rmsnorm: null shape/strides/axes");
  NdArgs a{shape, xstrides, ystrides, ndim, axes, naxes};
  return run_nd(OP_RMSNORM, dt_in, dt_out, dt_w, x, y, weight, nullptr, nullptr, a, eps, false,
                static_cast<cudaStream_t>(stream), "ytcuda_rmsnorm");
}

int ytcuda_layernorm(int dt_in, int dt_out, int dt_w, const void* x, const void* gamma, const void* beta, void* y,
                     const int64_t* shape, const int64_t* xstrides, const int64_t* ystrides, int ndim, const int* axes,
                     int naxes, float eps, void* stream) {
  YTC_REQUIRE(shape && xstrides && ystrides && axes, "ytcuda_layernorm: null shape/strides/axes");
  YTC_REQUIRE((gamma == nullptr) == (beta == nullptr), "ytcuda_layernorm: gamma and beta come together");
  NdArgs a{shape, xstrides, ystrides, ndim, axes, naxes};
  return run_nd(OP_LAYERNORM, dt_in, dt_out, dt_w, x, y, gamma, beta, nullptr, a, eps, false,
                static_cast<cudaStream_t>(stream), "ytcuda_layernorm");
}

int ytcuda_layernorm_strided(int dt_in, int dt_out, int dt_w, const void* x, const void* gamma, const void* beta, void* y,
                             const int64_t* shape, const int64_t* xstrides, const int64_t* ystrides, const int64_t* wstrides,
                             int ndim, const int* axes, int naxes, float eps, void* stream) {
  YTC_REQUIRE(shape && xstrides && ystrides && wstrides && axes, "ytcuda_layernorm_strided: null shape/strides/axes");
  YTC_REQUIRE(gamma && beta, "ytcuda_layernorm_strided: null gamma/beta");
  NdArgs a{shape, xstrides, ystrides, ndim, axes, naxes};
  return run_nd(OP_LAYERNORM, dt_in, dt_out, dt_w, x, y, gamma, beta, nullptr, a, eps, false,
                static_cast<cudaStream_t>(stream), "ytcuda_layernorm_strided", nullptr, 0, 2.f, wstrides);
}

int ytcuda_reduce(int op, int dt_in, int dt_out, const void* x, void* y, int32_t* index, const int64_t* shape,
                  const int64_t* xstrides, int ndim, const int* axes, int naxes, void* stream) {
  YTC_REQUIRE(op >= 0 && op <= 2, "ytcuda_reduce: op must be 0 (sum), 1 (mean) or 2 (max)");
  YTC_REQUIRE(shape && xstrides && axes, "ytcuda_reduce: null shape/strides/axes");
  YTC_REQUIRE(ndim >= 1 && ndim <= MAXD, "ytcuda_reduce: ndim %d outside [1, %d]", ndim, MAXD);
  // the output is contiguous with size-1 dims on the reduced axes
  int64_t ys[MAXD];
  {
    bool red[MAXD] = {false};
    for (int i = 0; i < naxes && i < MAXD; ++i) red[((axes[i] % ndim) + ndim) % ndim] = true;
    int64_t acc = 1;
    for (int d = ndim - 1; d >= 0; --d) {
      ys[d] = red[d] ? 0 : acc;
      if (!red[d]) acc *= shape[d];
    }
  }
  NdArgs a{shape, xstrides, ys, ndim, axes, naxes};
  const int rop = op == 0 ? OP_SUM : op == 1 ? OP_MEAN : OP_MAX;
  return run_nd(rop, dt_in, dt_out, YTC_F32, x, y, nullptr, nullptr, index, a, 0.f, true,
                static_cast<cudaStream_t>(stream), "ytcuda_reduce");
}

int ytcuda_rmsnorm_add_softmax_cast(int dt_out, const float* x, const float* weight, const float* residual, void* out,
                                    int64_t batch, int64_t rows, int hidden, int residual_batched, float eps,
                                    void* stream) {
  YTC_REQUIRE(dt_out >= 0 && dt_out <= 2, "ytcuda_rmsnorm_add_softmax_cast: bad dt_out");
  YTC_REQUIRE(batch >= 0 && rows >= 0 && hidden >= 0, "ytcuda_rmsnorm_add_softmax_cast: negative extent");
  if (batch == 0 || rows == 0 || hidden == 0) return YTC_OK;
  YTC_REQUIRE(x && weight && residual && out, "ytcuda_rmsnorm_add_softmax_cast: null tensor");
  if (hidden % 4 != 0 || hidden > 16384 || (reinterpret_cast<uint64_t>(x) & 15) || (reinterpret_cast<uint64_t>(weight) & 15) ||
      (reinterpret_cast<uint64_t>(residual) & 15) || (reinterpret_cast<uint64_t>(out) & 7)) {
    set_last_error("ytcuda_rmsnorm_add_softmax_cast: hidden must be a multiple of 4, at most 16384, tensors 16-byte aligned");
    return YTC_UNSUPPORTED;
  }
  RowParams p;
  p.x = x; p.y = out; p.w = weight; p.b = residual; p.idx = nullptr;
  p.rows = batch * rows; p.L = hidden;
  p.x_rs = hidden; p.y_rs = hidden;
  p.r_rows = residual_batched ? batch * rows : rows;
  p.eps = eps; p.dt_in = YTC_F32; p.dt_out = dt_out; p.dt_w = YTC_F32;
  if (dt_out == YTC_BF16 && (hidden == 1024 || hidden == 2048 || hidden == 4096)) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t cap = static_cast<int64_t>(sm_count()) * 4 * 4;
    const unsigned grid = static_cast<unsigned>(p.rows < cap ? p.rows : cap);
    uint2* o2 = static_cast<uint2*>(out);
    if (hidden == 4096) chain_fast_kernel<4><<<grid, 256, 0, st>>>(x, weight, residual, o2, p.rows, p.r_rows, eps);
    else if (hidden == 2048) chain_fast_kernel<2><<<grid, 256, 0, st>>>(x, weight, residual, o2, p.rows, p.r_rows, eps);
    else chain_fast_kernel<1><<<grid, 256, 0, st>>>(x, weight, residual, o2, p.rows, p.r_rows, eps);
    count_launch();
    YTC_CUDA(cudaGetLastError());
    return YTC_OK;
  }
  launch_row_op<4>(OP_CHAIN, p, static_cast<cudaStream_t>(stream));
  YTC_CUDA(cudaGetLastError());
  return YTC_OK;
}

}  // extern "C"
