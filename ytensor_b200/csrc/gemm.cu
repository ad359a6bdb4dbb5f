// GEMM for the YTensor device backend.
//
//  * gemm_tc_kernel   : bf16 / fp16 inputs, fp32 accumulation in tensor memory. Persistent,
//                       one CTA per SM, warp-specialised: warp 0 feeds a shared-memory
//                       ring with TMA, warp 1 issues tcgen05.mma (128 x BN x 16 per instruction),
//                       warps 4-11 drain the accumulator (tcgen05.ld) and write C (TMA stores) while
//                       the next tile's MMAs run into the second accumulator stage.
//  * gemm_simt_kernel : any strides, any of {f32, bf16, f16}, FFMA with fp32 accumulation.
//                       It is the fp32 path and the layout catch-all of the tensor-core path.
//
// Replaces yt::kernel::avx2::sgemm / matmul / hgemm (reference src/kernel/avx2/sgemm.inl:586-806,
// src/kernel/avx2/hgemm.inl:139-288) behind ytcuda_gemm.
#include <atomic>

#include "lm_ops.cuh"
#include "ptx_sm100.cuh"
#include "ytc_common.cuh"

namespace ytk {

// ------------------------------------------------------------------ tcgen05 path
constexpr int TC_BM = 128;
constexpr int TC_BK = 64;  // 64 x 16-bit = one 128-byte swizzle row
constexpr int TC_EPI_WARPS = 8;  // two per quarter of the accumulator's lanes
constexpr int TC_THREADS = 128 + 32 * TC_EPI_WARPS;

struct GemmTcParams {
  int M, N, K;
  int batch;
  int a_mn, b_mn;        // 1 = the operand's unit stride runs along M (A) / N (B), 0 = along K
  int a_bcast, b_bcast;  // 1 = operand shared by all batch items
  uint32_t idesc;
  float alpha, beta;
  void* C;
  int64_t rsc, csc, bsc;
  int out_dtype;
  int tiles_m, tiles_n, total_tiles, k_blocks;
  int a_prefetch;  // k-blocks by which an L2 prefetch of A runs ahead of the shared-memory loads (0 = off)
  int split_loads; // K-major tiles fetched as 64-row boxes
  // a product of planes (TcPlanes): `fold` blocks of k of one pair of planes after another; 0 = ordinary
  int fold, planes_a, planes_b;
  uint32_t pa, pb;         // plane of A / B per pair, two bits each
  // k cut into `splits` pieces of split_blocks blocks, one work item each; batch item split * batch + b of C gets a piece
  int splits, split_blocks;
  int* status;
  // masked product: tile_live[mb * tiles_n + nb] == 0 marks an output tile no element of which is asked for; every
  // role of the kernel passes over it (no loads, no MMAs, no stores). NULL = every tile is computed.
  const uint8_t* tile_live;
  // linear layers of the language models (LinearEpilogue, lm_ops.cuh)
  int epi;                 // EPI_NONE: the store rules above; otherwise tc_store_epilogue
  int cluster;             // pieces of k that the CTAs of a cluster share (gemm_split_kernel)
  int n_step, n_cta;       // CTA pairs: columns from one tile to the next, from the one CTA's share of B to the other's
  int tma_out;             // C through TMA stores: 0 no, 1 yes, 2 added to what C holds (fp32)
  int act_cols;            // EPI_SILU
  float limit, alpha_gate, shift;  // EPI_CLAMP_PAIRS
  // grouped product: every 128-row block of A belongs to one group (expert) or to none (-1, passed over); group g
  // multiplies rows g * group_rows .. of the stacked B operand. NULL = ordinary product.
  const int* tile_group;
  int group_rows;
};

constexpr int TC_OUT_BYTES = 32 * 128;  // an epilogue warp's 32 rows of 128 bytes on their way to C
template <int BN>
struct TcSmem {
  // 192 KB of operands on their way: with four slots of 128 columns a block of k took 0.43 us on an idle chip, twice its MMAs
  static constexpr int STAGES = BN == 128 ? 6 : 4;
  static constexpr int FREED = BN == 128 ? 2 : 1;  // slots freed together
  static constexpr int A_BYTES = TC_BM * TC_BK * 2;
  static constexpr int B_BYTES = BN * TC_BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int BAR_OFFSET = STAGES * STAGE_BYTES;
  // full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2], tmem base word, abort word
  static constexpr int TOTAL = BAR_OFFSET + (2 * STAGES + 4) * 8 + 16;
  static constexpr int DYN_BYTES = TOTAL + 1024;  // slack to align the ring to 1024 B
  static constexpr int OUT_OFFSET = (TOTAL + 1023) / 1024 * 1024;  // TMA stores: the epilogue warps' areas
  static constexpr int DYN_STAGED = OUT_OFFSET + TC_EPI_WARPS * TC_OUT_BYTES + 1024;
};

// Work item -> batch item of the operands, first and end k block; a product of planes counts its blocks pair by pair from 0
// and every pair starts at block `first` of k.
struct TcPiece {
  int b, kb0, kb1, first;
};
__device__ __forceinline__ TcPiece tc_piece(const GemmTcParams& p, int bf) {
  if (p.splits == 1) return {bf, 0, p.k_blocks, 0};
  const int split = bf / p.batch, b = bf - split * p.batch;
  if (p.fold > 0) return {b, 0, p.split_blocks, split * p.fold};
  return {b, split * p.split_blocks, min(p.k_blocks, (split + 1) * p.split_blocks), 0};
}
// Where a k block lies: block kk of plane (or batch item) za of A and zb of B; next() steps to the block behind it.
template <bool PIECES>
struct TcBlock {
  int kk, za, zb, end, pair;
  __device__ __forceinline__ void plane(const GemmTcParams& p, int ba, int bb, int first) {
    kk = first;
    end = first + p.fold;
    za = ba * p.planes_a + static_cast<int>((p.pa >> (2 * pair)) & 3);
    zb = bb * p.planes_b + static_cast<int>((p.pb >> (2 * pair)) & 3);
  }
  __device__ __forceinline__ TcBlock(const GemmTcParams& p, const TcPiece& w, int ba, int bb)
      : kk(w.kb0), za(ba), zb(bb), end(0x7fffffff), pair(0) {
    if (PIECES && p.fold > 0) plane(p, ba, bb, w.first);
  }
  __device__ __forceinline__ void next(const GemmTcParams& p, const TcPiece& w, int ba, int bb) {
    if (++kk == end && PIECES) {
      ++pair;
      plane(p, ba, bb, w.first);
    }
  }
};

template <int BN, int OUT_DT>
__device__ __forceinline__ void tc_store_chunk(const GemmTcParams& p, const uint32_t (&r)[32], int64_t row_off,
                                               int gn0, bool row_ok, bool vec_ok) {
  // One thread holds 32 consecutive columns of one row.
  if (!row_ok) return;
  char* cbase = static_cast<char*>(p.C);
  const float alpha = p.alpha, beta = p.beta;
  if (vec_ok && gn0 + 32 <= p.N) {
    if constexpr (OUT_DT == YTC_F32) {
      float4* dst = reinterpret_cast<float4*>(cbase + (row_off + gn0) * 4);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float4 v;
        v.x = alpha * __uint_as_float(r[4 * j + 0]);
        v.y = alpha * __uint_as_float(r[4 * j + 1]);
        v.z = alpha * __uint_as_float(r[4 * j + 2]);
        v.w = alpha * __uint_as_float(r[4 * j + 3]);
        if (beta != 0.f) {
          float4 o = dst[j];
          v.x += beta * o.x; v.y += beta * o.y; v.z += beta * o.z; v.w += beta * o.w;
        }
        dst[j] = v;
      }
    } else {
      uint4* dst = reinterpret_cast<uint4*>(cbase + (row_off + gn0) * 2);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float v[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) v[t] = alpha * __uint_as_float(r[8 * j + t]);
        if (beta != 0.f) {
          uint4 o = dst[j];
          const uint32_t ow[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const uint16_t lo = static_cast<uint16_t>(ow[t] & 0xFFFFu), hi = static_cast<uint16_t>(ow[t] >> 16);
            if constexpr (OUT_DT == YTC_BF16) {
              v[2 * t] += beta * bf16_bits_to_f32(lo);
              v[2 * t + 1] += beta * bf16_bits_to_f32(hi);
            } else {
              v[2 * t] += beta * f16_bits_to_f32_ref(lo);
              v[2 * t + 1] += beta * f16_bits_to_f32_ref(hi);
            }
          }
        }
        uint32_t w[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          uint16_t lo, hi;
          if constexpr (OUT_DT == YTC_BF16) {
            lo = f32_to_bf16_bits_ref(v[2 * t]);
            hi = f32_to_bf16_bits_ref(v[2 * t + 1]);
          } else {
            lo = f32_to_f16_bits_ref(v[2 * t]);
            hi = f32_to_f16_bits_ref(v[2 * t + 1]);
          }
          w[t] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
        }
        dst[j] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  } else {
#pragma unroll 4
    for (int j = 0; j < 32; ++j) {
      const int gn = gn0 + j;
      if (gn < p.N) {
        const int64_t idx = row_off + static_cast<int64_t>(gn) * p.csc;
        float v = alpha * __uint_as_float(r[j]);
        if (beta != 0.f) v += beta * DType<OUT_DT>::load(p.C, idx);
        DType<OUT_DT>::store(p.C, idx, v);
      }
    }
  }
}

__device__ __forceinline__ float tc_clamped_gate(const GemmTcParams& p, float gate, float up) {
  const float g = fminf(gate, p.limit), u = fminf(fmaxf(up, -p.limit), p.limit);
  return __fdividef(g, 1.f + __expf(-p.alpha_gate * g)) * (u + p.shift);
}
// The fused activation and round-to-nearest-even narrowing of 32 consecutive columns of one row (see LinearEpilogue): 16
// words of two bf16 each, 8 for the gated pairs. One loop per activation, so that its 32 results are independent work.
__device__ __forceinline__ void tc_activate(const GemmTcParams& p, const uint32_t (&r)[32], int gn0, uint32_t (&w)[16]) {
  auto at = [&](int i) { return __uint_as_float(r[i]); };
  if (p.epi == EPI_SWIGLU_PAIRS) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      w[j] = pack_bf16x2_rn(lm_silu_fast(at(4 * j)) * at(4 * j + 1), lm_silu_fast(at(4 * j + 2)) * at(4 * j + 3));
  } else if (p.epi == EPI_CLAMP_PAIRS) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      w[j] = pack_bf16x2_rn(tc_clamped_gate(p, at(4 * j), at(4 * j + 1)), tc_clamped_gate(p, at(4 * j + 2), at(4 * j + 3)));
  } else if (p.epi == EPI_GELU_ERF) {
#pragma unroll
    for (int j = 0; j < 16; ++j) w[j] = pack_bf16x2_rn(lm_gelu_erf(at(2 * j)), lm_gelu_erf(at(2 * j + 1)));
  } else if (p.epi == EPI_RELU2) {
#pragma unroll
    for (int j = 0; j < 16; ++j) w[j] = pack_bf16x2_rn(lm_relu2(at(2 * j)), lm_relu2(at(2 * j + 1)));
  } else if (p.epi == EPI_SILU && gn0 + 32 <= p.act_cols) {
#pragma unroll
    for (int j = 0; j < 16; ++j) w[j] = pack_bf16x2_rn(lm_silu_fast(at(2 * j)), lm_silu_fast(at(2 * j + 1)));
  } else if (p.epi != EPI_SILU || gn0 >= p.act_cols) {
#pragma unroll
    for (int j = 0; j < 16; ++j) w[j] = pack_bf16x2_rn(at(2 * j), at(2 * j + 1));
  } else {
    const int n = p.act_cols - gn0;  // (activated columns among these)
#pragma unroll
    for (int j = 0; j < 16; ++j)
      w[j] = pack_bf16x2_rn(2 * j < n ? lm_silu_fast(at(2 * j)) : at(2 * j),
                            2 * j + 1 < n ? lm_silu_fast(at(2 * j + 1)) : at(2 * j + 1));
  }
}
__device__ __forceinline__ bool tc_pairs(const GemmTcParams& p) { return p.epi == EPI_SWIGLU_PAIRS || p.epi == EPI_CLAMP_PAIRS; }

// Direct store: one thread holds 32 consecutive columns of one row; the gated pairs make 16 results of them.
__device__ __forceinline__ void tc_store_epilogue(const GemmTcParams& p, const uint32_t (&r)[32], int64_t row_off, int gn0,
                                                  bool row_ok) {
  if (!row_ok) return;
  uint32_t w[16];
  tc_activate(p, r, gn0, w);
  const bool pairs = tc_pairs(p);
  uint16_t* dst = static_cast<uint16_t*>(p.C) + row_off + (pairs ? gn0 >> 1 : gn0);
#pragma unroll
  for (int j = 0; j < 32; ++j)
    if (j < (pairs ? 16 : 32) && (pairs ? gn0 + 2 * j + 1 : gn0 + j) < p.N)
      dst[j] = static_cast<uint16_t>(w[j >> 1] >> ((j & 1) * 16));
}

// 32 columns of one row as ytcuda_gemm narrows them: 16 words of two 16-bit results.
template <int OUT_DT>
__device__ __forceinline__ void tc_narrow(const uint32_t (&r)[32], float alpha, uint32_t (&w)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float lo = alpha * __uint_as_float(r[2 * j]), hi = alpha * __uint_as_float(r[2 * j + 1]);
    if constexpr (OUT_DT == YTC_BF16) w[j] = f32_to_bf16_bits_ref(lo) | (static_cast<uint32_t>(f32_to_bf16_bits_ref(hi)) << 16);
    else w[j] = f32_to_f16_bits_ref(lo) | (static_cast<uint32_t>(f32_to_f16_bits_ref(hi)) << 16);
  }
}

// A warp's share of an accumulator to C: every other group of columns that make 128 bytes of a row of C (32 fp32, 64 16-bit, 128
// for gated pairs) is narrowed into the warp's 32 rows of 128 bytes, 16-byte pieces exchanged by row as the tensor map has them,
// and leaves as one TMA store, which clips what lies outside C. Bound by the instructions of four schedulers: with one warp
// on each, and 16-byte stores of its lanes, a 128 x 256 tile took 10.8 us (bf16; 6.2 with an activation that unrolled), more
// than its MMAs for k below 2500; now 3.3. 4096 x 4096 x 1024 with nearest-even stores 53.6 -> 33.2 us, x 64 43.3 -> 13.2.
// n0: C's column under the accumulator's first, m0: C's row under the warp's first, half: which of the groups.
struct TcNothing {
  __device__ __forceinline__ void operator()(uint32_t (&)[32], int) const {}
};
// more(r, c): what is added to columns c .. c + 31 of the accumulator first.
template <int BN, class More = TcNothing>
__device__ __forceinline__ void tc_drain(const GemmTcParams& p, const CUtensorMap* tmC, uint32_t t_row, uint8_t* buf, int n0, int m0,
                                         int b, int half, int lane, More more = More{}) {
  if (m0 >= p.M) return;
  const bool pairs = tc_pairs(p), wide = p.epi == EPI_NONE && p.out_dtype == YTC_F32;
  const int cols = wide ? 32 : pairs ? 128 : 64;
  uint8_t* mine = buf + lane * 128;
  auto put = [&](int piece, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    *reinterpret_cast<uint4*>(mine + ((piece ^ (lane & 7)) << 4)) = make_uint4(x, y, z, w);
  };
#pragma unroll 1
  for (int g = half * cols; g < BN && n0 + g < p.N; g += 2 * cols) {
    if (lane == 0) tma_store_wait_read<0>();  // the rows of the store before this one have been read
    __syncwarp();
    int piece = 0;
#pragma unroll 1
    for (int c = 0; c < cols; c += 32) {
      uint32_t r[32];
      tmem_ld_32x32b_x32(t_row + g + c, r);
      tmem_ld_wait();
      more(r, g + c);
      if (wide) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          put(j, __float_as_uint(p.alpha * __uint_as_float(r[4 * j])), __float_as_uint(p.alpha * __uint_as_float(r[4 * j + 1])),
              __float_as_uint(p.alpha * __uint_as_float(r[4 * j + 2])), __float_as_uint(p.alpha * __uint_as_float(r[4 * j + 3])));
        continue;
      }
      uint32_t w[16];
      if (p.epi != EPI_NONE) tc_activate(p, r, n0 + g + c, w);
      else if (p.out_dtype == YTC_BF16) tc_narrow<YTC_BF16>(r, p.alpha, w);
      else tc_narrow<YTC_F16>(r, p.alpha, w);
      put(piece, w[0], w[1], w[2], w[3]);
      put(piece + 1, w[4], w[5], w[6], w[7]);
      if (!pairs) {
        put(piece + 2, w[8], w[9], w[10], w[11]);
        put(piece + 3, w[12], w[13], w[14], w[15]);
      }
      piece += pairs ? 2 : 4;
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      const int col = pairs ? (n0 + g) >> 1 : n0 + g;
      if (p.tma_out == 2) tma_add_3d(tmC, buf, col, m0, b);
      else tma_store_3d(tmC, buf, col, m0, b);
      tma_store_commit();
    }
  }
}

// The same for EPI_SWIGLU_PLANES: accumulator columns 0 .. 127 are gates, 128 .. 255 the ups of the same 128 outputs; a warp forms 64
// of them, whose hi and lo planes leave one after the other.
__device__ __forceinline__ void tc_drain_swiglu(const GemmTcParams& p, const CUtensorMap* tmC, uint32_t t_row, uint8_t* buf, int n0,
                                                int m0, int half, int lane) {
  if (m0 >= p.M || n0 + half * 64 >= p.N) return;
  uint8_t* mine = buf + lane * 128;
  if (lane == 0) tma_store_wait_read<0>();
  __syncwarp();
  uint32_t lo[32];
#pragma unroll
  for (int c = 0; c < 64; c += 16) {
    uint32_t g[16], u[16], hi[8];
    tmem_ld_32x32b_x16(t_row + half * 64 + c, g);
    tmem_ld_32x32b_x16(t_row + 128 + half * 64 + c, u);
    tmem_ld_wait();
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float f[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float v = __uint_as_float(g[2 * e + x]), z = expf(-fabsf(v)), s = 1.0f / (1.0f + z);
        f[x] = v * (v >= 0.f ? s : z * s) * __uint_as_float(u[2 * e + x]);
      }
      const __nv_bfloat162 h = __floats2bfloat162_rn(f[0], f[1]);
      hi[e] = *reinterpret_cast<const uint32_t*>(&h);
      lo[c / 2 + e] = pack_bf16x2_rn(f[0] - __low2float(h), f[1] - __high2float(h));
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
      *reinterpret_cast<uint4*>(mine + (((c / 8 + i) ^ (lane & 7)) << 4)) = make_uint4(hi[4 * i], hi[4 * i + 1], hi[4 * i + 2], hi[4 * i + 3]);
  }
  auto store = [&](int plane) {
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_3d(tmC, buf, n0 + half * 64, m0, plane);
      tma_store_commit();
    }
  };
  store(0);
  if (lane == 0) tma_store_wait_read<0>();
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i)
    *reinterpret_cast<uint4*>(mine + ((i ^ (lane & 7)) << 4)) = make_uint4(lo[4 * i], lo[4 * i + 1], lo[4 * i + 2], lo[4 * i + 3]);
  store(1);
}

// PIECES: a product of planes, or k in pieces (the few instructions more cost an ordinary short product 0.2 us).
template <int BN, bool PIECES>
__global__ void __launch_bounds__(TC_THREADS, 1)
    gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ CUtensorMap tmC, const GemmTcParams p) {
  using S = TcSmem<BN>;
  constexpr int TC_STAGES = S::STAGES;
  extern __shared__ uint8_t smem_raw[];
  // The 128-byte swizzle pattern is a function of the shared address: keep the ring 1024-byte aligned.
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);

  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::BAR_OFFSET);
  uint64_t* empty_bar = full_bar + TC_STAGES;
  uint64_t* tfull_bar = empty_bar + TC_STAGES / S::FREED;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // (known to be the same for the whole warp)
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < TC_STAGES; ++s) mbar_init(&full_bar[s], 1);
    for (int s = 0; s < TC_STAGES / S::FREED; ++s) mbar_init(&empty_bar[s], 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull_bar[s], 1);
      mbar_init(&tempty_bar[s], TC_EPI_WARPS);
    }
    *abort_word = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if (p.tma_out) tma_prefetch_desc(&tmC);
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Everything above touched shared and tensor memory only: under a programmatic dependent launch it ran while the
  // kernel before this one was finishing. From here on global memory is read and written.
  dependent_wait();
  dependent_trigger();

  const int tiles_per_batch = p.tiles_m * p.tiles_n;

  if (warp == 0) {
    // ------------------------------------------------ TMA producer (converged, as the MMA issuer: a copy issued inside a
    // branch of one lane costs some hundred instructions; block by block they took 700 clk)
    const uint32_t lead = lane == 0 ? 1u : 0u;
    const uint32_t ring_at = smem_u32(smem), full_at = smem_u32(full_bar);
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    bool ok = true;
    // A is streamed from HBM once; an L2 prefetch a few k-blocks ahead of the shared-memory ring
    // takes the DRAM latency off the ring (B is small and stays L2-resident by reuse).
    auto prefetch_a = [&](int tile, int kb) {
      if (tile >= p.total_tiles) return;
      const int b = tile / tiles_per_batch;
      const int rem = tile - b * tiles_per_batch;
      const int mb = rem / p.tiles_n;
      const int ba = p.a_bcast ? 0 : b;
      if (!p.a_mn) {
        tma_prefetch_l2_3d_lead(&tmA, kb * TC_BK, mb * TC_BM, ba, lead);
      } else {
#pragma unroll
        for (int c = 0; c < TC_BM / 64; ++c) tma_prefetch_l2_3d_lead(&tmA, mb * TC_BM + c * 64, kb * TC_BK, ba, lead);
      }
    };
    int pf_tile = blockIdx.x, pf_kb = 0;
    auto prefetch_next = [&]() {
      prefetch_a(pf_tile, pf_kb);
      if (++pf_kb == p.k_blocks) {
        pf_kb = 0;
        pf_tile += gridDim.x;
      }
    };
#pragma unroll 1
    for (int i = 0; i < p.a_prefetch; ++i) prefetch_next();
    for (int tile = blockIdx.x; ok && tile < p.total_tiles; tile += gridDim.x) {
      const int bf = tile / tiles_per_batch;
      const int rem = tile - bf * tiles_per_batch;
      TcPiece piece{bf, 0, p.k_blocks, 0};
      if (PIECES) piece = tc_piece(p, bf);
      if (p.tile_live && !p.tile_live[rem]) continue;
      const int mb = rem / p.tiles_n;
      const int nb = rem - mb * p.tiles_n;
      const int group = p.tile_group ? __shfl_sync(0xffffffffu, p.tile_group[mb], 0) : 0;
      if (group < 0) continue;
      const int n_row0 = group * p.group_rows + nb * BN;
      const int ba = p.a_bcast ? 0 : piece.b;
      const int bb = p.b_bcast ? 0 : piece.b;
      TcBlock<PIECES> at(p, piece, ba, bb);
#pragma unroll 1
      for (int kb = piece.kb0; kb < piece.kb1; ++kb, at.next(p, piece, ba, bb)) {
        if (stage % S::FREED == 0 && !mbar_wait_warp(&empty_bar[stage / S::FREED], phase ^ 1u, abort_word)) {
          ok = false;
          break;
        }
        if (p.a_prefetch > 0) prefetch_next();
        const uint32_t bar = full_at + 8 * stage, sa = ring_at + stage * S::STAGE_BYTES, sb = sa + S::A_BYTES;
        mbar_expect_tx_lead(bar, S::STAGE_BYTES, lead);
        if (!p.a_mn && !p.split_loads) {
          tma_load_3d_lead(sa, &tmA, bar, at.kk * TC_BK, mb * TC_BM, at.za, lead);
        } else {
#pragma unroll 1
          for (int c = 0; c < TC_BM / 64; ++c) {
            const int mn = mb * TC_BM + c * 64, kk = at.kk * TC_BK;
            tma_load_3d_lead(sa + c * 8192, &tmA, bar, p.a_mn ? mn : kk, p.a_mn ? kk : mn, at.za, lead);
          }
        }
        if (!p.b_mn && !p.split_loads) {
          tma_load_3d_lead(sb, &tmB, bar, at.kk * TC_BK, n_row0, at.zb, lead);
        } else {
#pragma unroll 1
          for (int c = 0; c < BN / 64; ++c) {
            const int mn = n_row0 + c * 64, kk = at.kk * TC_BK;
            tma_load_3d_lead(sb + c * 8192, &tmB, bar, p.b_mn ? mn : kk, p.b_mn ? kk : mn, at.zb, lead);
          }
        }
        ++issued;
        if (++stage == TC_STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (!ok) {
      // Give the copies already in flight a bounded time to land before the CTA goes away.
      const int pending = issued < TC_STAGES ? issued : TC_STAGES;
      int s = stage;
      uint32_t ph = phase;
      for (int i = 0; i < pending; ++i) {
        if (--s < 0) {
          s = TC_STAGES - 1;
          ph ^= 1u;
        }
        const long long t0 = clock64();
        while (!mbar_try_wait(&full_bar[s], ph) && clock64() - t0 < 20000000ll) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    // The tensor pipe takes the next instruction only when it can start it, so whatever else the issuing warp does is time in
    // which no MMA runs. The warp stays converged (operands in uniform registers), looks at the next slot before it issues this
    // one's MMAs, and frees two slots with one commit: a block of k of 128 x 128 takes 290 clk to issue, of which 256 are MMAs;
    // with one lane that waits, issues and commits block by block it took 576. With the producer's copies (below): 500 x 1024 x
    // 4608 32.8 -> 22.9 us, 4096^3 105 -> 94, 8 x 2048 x 4096 x 4096 449 -> 409.
    const uint32_t lead = lane == 0 ? 1u : 0u;
    const uint32_t free_at = smem_u32(empty_bar), tfull_at = smem_u32(tfull_bar);
    const uint64_t a_desc = p.a_mn ? umma_smem_desc_sw128(smem_u32(smem), 8192, 1024) : umma_smem_desc_sw128(smem_u32(smem), 16, 1024);
    const uint64_t b_desc = (p.b_mn ? umma_smem_desc_sw128(smem_u32(smem), 8192, 1024) : umma_smem_desc_sw128(smem_u32(smem), 16, 1024)) + (S::A_BYTES >> 4);
    const uint32_t a_step = p.a_mn ? 2048 >> 4 : 32 >> 4, b_step = p.b_mn ? 2048 >> 4 : 32 >> 4;
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true, ready = false;
    for (int tile = blockIdx.x; ok && tile < p.total_tiles; tile += gridDim.x) {
      if (p.tile_live && !p.tile_live[tile % tiles_per_batch]) continue;
      if (p.tile_group && p.tile_group[(tile % tiles_per_batch) / p.tiles_n] < 0) continue;
      if (!mbar_wait_warp(&tempty_bar[acc], acc_phase ^ 1u, abort_word)) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
      TcPiece piece{0, 0, p.k_blocks, 0};
      if (PIECES) piece = tc_piece(p, tile / tiles_per_batch);
#pragma unroll 1
      for (int kb = piece.kb0; kb < piece.kb1; ++kb) {
        if (!ready && !mbar_wait_warp(&full_bar[stage], phase, abort_word)) {
          ok = false;
          break;
        }
        const int next = stage + 1 == TC_STAGES ? 0 : stage + 1;
        ready = __all_sync(0xffffffffu, mbar_test_wait(&full_bar[next], next ? phase : phase ^ 1u)) != 0;
        tc_fence_after();
        const uint64_t ad = a_desc + (stage * S::STAGE_BYTES >> 4), bd = b_desc + (stage * S::STAGE_BYTES >> 4);
#pragma unroll
        for (int k = 0; k < TC_BK / 16; ++k)
          tc_mma_f16_lead(d_tmem, ad + k * a_step, bd + k * b_step, p.idesc, kb != piece.kb0 || k != 0 ? 1u : 0u, lead);
        // frees the slots once their MMAs have read them
        if (stage % S::FREED == S::FREED - 1) tc_commit_lead(free_at + 8 * (stage / S::FREED), lead);
        stage = next;
        if (next == 0) phase ^= 1u;
      }
      if (!ok) break;
      tc_commit_lead(tfull_at + 8 * acc, lead);  // accumulator complete
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  } else if (warp >= 4) {
    // ------------------------------------------------ epilogue (TMEM -> registers -> global)
    const int q = warp & 3, half = (warp - 4) >> 2;  // a warp may only touch TMEM lanes 32q .. 32q+31
    const int row = q * 32 + lane;
    uint8_t* out_buf = smem + S::OUT_OFFSET + (warp - 4) * TC_OUT_BYTES;
    int acc = 0;
    uint32_t acc_phase = 0;
    const bool c_unit = (p.csc == 1);
    const int esz = (p.out_dtype == YTC_F32) ? 4 : 2;
    for (int tile = blockIdx.x; tile < p.total_tiles; tile += gridDim.x) {
      const int b = tile / tiles_per_batch;
      const int rem = tile - b * tiles_per_batch;
      if (p.tile_live && !p.tile_live[rem]) continue;
      const int mb = rem / p.tiles_n;
      const int nb = rem - mb * p.tiles_n;
      if (p.tile_group && p.tile_group[mb] < 0) continue;
      if (!mbar_wait(&tfull_bar[acc], acc_phase, abort_word)) break;
      tc_fence_after();
      const int gm = mb * TC_BM + row;
      const bool row_ok = gm < p.M;
      const int64_t row_off = static_cast<int64_t>(b) * p.bsc + static_cast<int64_t>(gm) * p.rsc;
      const bool vec_ok =
          c_unit && (((reinterpret_cast<uint64_t>(p.C) + static_cast<uint64_t>(row_off) * esz) & 15u) == 0) &&
          ((static_cast<int64_t>(nb) * BN * esz & 15) == 0);
      const uint32_t t_row = tmem_base + static_cast<uint32_t>(acc * BN) + (static_cast<uint32_t>(q * 32) << 16);
      if (p.tma_out) {
        tc_drain<BN>(p, &tmC, t_row, out_buf, nb * BN, mb * TC_BM + q * 32, b, half, lane);
      } else {
#pragma unroll 1
        for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 32) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(t_row + c0, r);
          tmem_ld_wait();
          const int gn0 = nb * BN + c0;
          if (gn0 < p.N) {
            if (p.epi != EPI_NONE) tc_store_epilogue(p, r, row_off, gn0, row_ok);
            else if (p.out_dtype == YTC_BF16) tc_store_chunk<BN, YTC_BF16>(p, r, row_off, gn0, row_ok, vec_ok);
            else if (p.out_dtype == YTC_F32) tc_store_chunk<BN, YTC_F32>(p, r, row_off, gn0, row_ok, vec_ok);
            else tc_store_chunk<BN, YTC_F16>(p, r, row_off, gn0, row_ok, vec_ok);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[acc]);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
    if (p.tma_out && lane == 0) tma_store_wait_all<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
  if (threadIdx.x == 0 && *abort_word) atomicExch(p.status, YTC_TIMEOUT);
}


// ------------------------------------------------------------------ tcgen05 path, CTA pairs
// Two CTAs (a cluster of 2 on neighbouring SMs) share one 256 x 256 output tile: each loads its own 128 rows of A
// and HALF of the B tile (128 columns), the leader CTA issues 256 x 256 x 16 MMAs (cta_group::2) that read both
// halves, and each CTA drains its own 128 x 256 accumulator. Per SM this halves the B bytes moved through shared
// memory and leaves room for a 6-stage ring. Barriers: TMA completion of both CTAs is counted on the leader's
// `full` barrier; the leader's commits free the stage in both CTAs and publish the accumulator to both.
constexpr int TC2_STAGES = 6;
constexpr int TC2_BN = 256;

struct Tc2Smem {
  static constexpr int A_BYTES = TC_BM * TC_BK * 2;         // 128 rows of A
  static constexpr int B_BYTES = (TC2_BN / 2) * TC_BK * 2;  // 128 columns of B
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int BAR_OFFSET = TC2_STAGES * STAGE_BYTES;
  static constexpr int TOTAL = BAR_OFFSET + (2 * TC2_STAGES + 4) * 8 + 16;
  static constexpr int DYN_BYTES = TOTAL + 1024;
  static constexpr int OUT_OFFSET = (TOTAL + 1023) / 1024 * 1024;
  static constexpr int DYN_STAGED = OUT_OFFSET + TC_EPI_WARPS * TC_OUT_BYTES + 1024;
};

template <bool PIECES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
    gemm_tc2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ CUtensorMap tmC, const GemmTcParams p) {
  using S = Tc2Smem;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::BAR_OFFSET);
  uint64_t* empty_bar = full_bar + TC2_STAGES;
  uint64_t* tfull_bar = empty_bar + TC2_STAGES / 2;  // (two slots are freed together)
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t cta = blockIdx.x & 1;  // rank in the cluster, 0 = leader
  const bool leader = cta == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < TC2_STAGES; ++s) mbar_init(&full_bar[s], 1);
    for (int s = 0; s < TC2_STAGES / 2; ++s) mbar_init(&empty_bar[s], 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull_bar[s], 1);
      mbar_init(&tempty_bar[s], 2 * TC_EPI_WARPS);  // the epilogue warps of both CTAs
    }
    *abort_word = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if (p.tma_out) tma_prefetch_desc(&tmC);
  }
  if (warp == 2) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // (set-up done in shared and tensor memory only; under a programmatic dependent launch global memory may be touched
  // from here on)
  dependent_wait();
  dependent_trigger();

  const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  const int tiles_per_batch = p.tiles_m * p.tiles_n;

  if (warp == 0) {
    // ------------------------------------------------ TMA producer (both CTAs)
    const uint32_t lead = lane == 0 ? 1u : 0u, first_cta = leader ? lead : 0u;
    const uint32_t ring_at = smem_u32(smem), full_at = smem_u32(full_bar), full_leader = map_to_cta(full_at, 0);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = cluster_id; ok && tile < p.total_tiles; tile += n_clusters) {
      const int b = tile / tiles_per_batch;
      const int rem = tile - b * tiles_per_batch;
      const int mb = rem / p.tiles_n;
      const int nb = rem - mb * p.tiles_n;
      const int ba = p.a_bcast ? 0 : b;
      const int bb = p.b_bcast ? 0 : b;
      const int m0 = mb * 256 + static_cast<int>(cta) * TC_BM;
      const int n0 = nb * p.n_step + static_cast<int>(cta) * p.n_cta;
      const TcPiece piece{b, 0, p.k_blocks, 0};
      TcBlock<PIECES> at(p, piece, ba, bb);
#pragma unroll 1
      for (int kb = 0; kb < p.k_blocks; ++kb, at.next(p, piece, ba, bb)) {
        if ((stage & 1) == 0 && !mbar_wait_warp(&empty_bar[stage >> 1], phase ^ 1u, abort_word)) {
          ok = false;
          break;
        }
        const uint32_t bar = full_leader + 8 * stage, sa = ring_at + stage * S::STAGE_BYTES, sb = sa + S::A_BYTES;
        mbar_expect_tx_lead(full_at + 8 * stage, 2 * S::STAGE_BYTES, first_cta);
        const int kk = at.kk * TC_BK;
        if (!p.a_mn) {
          tma_load_3d_pair_lead(sa, &tmA, bar, kk, m0, at.za, lead);
        } else {
#pragma unroll 1
          for (int c = 0; c < TC_BM / 64; ++c) tma_load_3d_pair_lead(sa + c * 8192, &tmA, bar, m0 + c * 64, kk, at.za, lead);
        }
        if (!p.b_mn) {
          tma_load_3d_pair_lead(sb, &tmB, bar, kk, n0, at.zb, lead);
        } else {
#pragma unroll 1
          for (int c = 0; c < TC2_BN / 128; ++c) tma_load_3d_pair_lead(sb + c * 8192, &tmB, bar, n0 + c * 64, kk, at.zb, lead);
        }
        if (++stage == TC2_STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer (leader CTA only; see gemm_tc_kernel)
    if (leader) {
      const uint32_t lead = lane == 0 ? 1u : 0u;
      const uint32_t free_at = smem_u32(empty_bar), tfull_at = smem_u32(tfull_bar);
      const uint64_t a_desc = p.a_mn ? umma_smem_desc_sw128(smem_u32(smem), 8192, 1024) : umma_smem_desc_sw128(smem_u32(smem), 16, 1024);
      const uint64_t b_desc = (p.b_mn ? umma_smem_desc_sw128(smem_u32(smem), 8192, 1024) : umma_smem_desc_sw128(smem_u32(smem), 16, 1024)) + (S::A_BYTES >> 4);
      const uint32_t a_step = p.a_mn ? 2048 >> 4 : 32 >> 4, b_step = p.b_mn ? 2048 >> 4 : 32 >> 4;
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true, ready = false;
      for (int tile = cluster_id; ok && tile < p.total_tiles; tile += n_clusters) {
        if (!mbar_wait_warp(&tempty_bar[acc], acc_phase ^ 1u, abort_word)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * TC2_BN);
#pragma unroll 1
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!ready && !mbar_wait_warp(&full_bar[stage], phase, abort_word)) {
            ok = false;
            break;
          }
          const int next = stage + 1 == TC2_STAGES ? 0 : stage + 1;
          ready = __all_sync(0xffffffffu, mbar_test_wait(&full_bar[next], next ? phase : phase ^ 1u)) != 0;
          tc_fence_after();
          const uint64_t ad = a_desc + (stage * S::STAGE_BYTES >> 4), bd = b_desc + (stage * S::STAGE_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < TC_BK / 16; ++k)
            tc_mma_f16_pair_lead(d_tmem, ad + k * a_step, bd + k * b_step, p.idesc, (kb | k) != 0 ? 1u : 0u, lead);
          // the slots are free in both CTAs once these MMAs have read them
          if (stage & 1) tc_commit_pair_lead(free_at + 8 * (stage >> 1), 3, lead);
          stage = next;
          if (next == 0) phase ^= 1u;
        }
        if (!ok) break;
        tc_commit_pair_lead(tfull_at + 8 * acc, 3, lead);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------ epilogue (both CTAs, own 128 rows x 256 columns)
    const int q = warp & 3, half = (warp - 4) >> 2;
    const int row = q * 32 + lane;
    uint8_t* out_buf = smem + S::OUT_OFFSET + (warp - 4) * TC_OUT_BYTES;
    int acc = 0;
    uint32_t acc_phase = 0;
    const bool c_unit = (p.csc == 1);
    const int esz = (p.out_dtype == YTC_F32) ? 4 : 2;
    for (int tile = cluster_id; tile < p.total_tiles; tile += n_clusters) {
      const int b = tile / tiles_per_batch;
      const int rem = tile - b * tiles_per_batch;
      const int mb = rem / p.tiles_n;
      const int nb = rem - mb * p.tiles_n;
      if (!mbar_wait(&tfull_bar[acc], acc_phase, abort_word)) break;
      tc_fence_after();
      const int gm = mb * 256 + static_cast<int>(cta) * TC_BM + row;
      const bool row_ok = gm < p.M;
      const int64_t row_off = static_cast<int64_t>(b) * p.bsc + static_cast<int64_t>(gm) * p.rsc;
      const bool vec_ok =
          c_unit && (((reinterpret_cast<uint64_t>(p.C) + static_cast<uint64_t>(row_off) * esz) & 15u) == 0);
      const uint32_t t_row = tmem_base + static_cast<uint32_t>(acc * TC2_BN) + (static_cast<uint32_t>(q * 32) << 16);
      if (PIECES && p.epi == EPI_SWIGLU_PLANES) {
        tc_drain_swiglu(p, &tmC, t_row, out_buf, nb * p.n_step, mb * 256 + static_cast<int>(cta) * TC_BM + q * 32, half, lane);
      } else if (p.tma_out) {
        tc_drain<TC2_BN>(p, &tmC, t_row, out_buf, nb * TC2_BN, mb * 256 + static_cast<int>(cta) * TC_BM + q * 32, b, half, lane);
      } else {
#pragma unroll 1
        for (int c0 = half * (TC2_BN / 2); c0 < (half + 1) * (TC2_BN / 2); c0 += 32) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(t_row + c0, r);
          tmem_ld_wait();
          const int gn0 = nb * TC2_BN + c0;
          if (gn0 < p.N) {
            if (p.epi != EPI_NONE) tc_store_epilogue(p, r, row_off, gn0, row_ok);
            else if (p.out_dtype == YTC_BF16) tc_store_chunk<TC2_BN, YTC_BF16>(p, r, row_off, gn0, row_ok, vec_ok);
            else if (p.out_dtype == YTC_F32) tc_store_chunk<TC2_BN, YTC_F32>(p, r, row_off, gn0, row_ok, vec_ok);
            else tc_store_chunk<TC2_BN, YTC_F16>(p, r, row_off, gn0, row_ok, vec_ok);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&tempty_bar[acc]), 0));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
    if (p.tma_out && lane == 0) tma_store_wait_all<0>();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves while the other may still read its shared or tensor memory
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
  if (threadIdx.x == 0 && *abort_word) atomicExch(p.status, YTC_TIMEOUT);
}

// ------------------------------------------------------------------ tcgen05 path, k shared by a cluster
// Products of less than half as many 128 x 128 tiles as the chip has SMs: the two or four CTAs of a cluster take a piece of k of one
// tile each (of every pair of planes), and the accumulators meet in the cluster: CTA j finishes the j-th share of the tile's rows,
// whose partial sums the others push into its shared memory, where its operands were (it says so first), and adds them to its
// own in a fixed order. No partial sums in memory, no second launch, and every store rule of the other kernels (tc_drain).
// What bounds it is the issue of one tile's blocks, now a half or a quarter of them, and 2 us for the exchange. Before / here: bf16
// 500 x 1024 x 4608 22.9 / 15.2 us, two planes 43.7 / 25.4; fp32 1024^3 (six products, two launches) 31.7 / 23.8.
__device__ __forceinline__ void tc_push4(uint32_t dst, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst), "r"(a),
               "r"(b), "r"(c), "r"(d), "r"(bar)
               : "memory");
}
__global__ void __launch_bounds__(TC_THREADS, 1)
    gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ CUtensorMap tmC, const GemmTcParams p) {
  using S = TcSmem<128>;
  constexpr int BN = 128, STAGES = S::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::BAR_OFFSET);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t *tfull_bar = empty_bar + STAGES / 2, *ready_bar = tfull_bar + 1, *recv_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull_bar + 4);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);
  static_assert(S::FREED == 2 && STAGES % 2 == 0 && (STAGES + STAGES / 2 + 4) * 8 + 8 <= (2 * STAGES + 4) * 8 + 16, "barriers");
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int pieces = p.cluster, piece = blockIdx.x % pieces, tile = blockIdx.x / pieces;
  const int tiles_per_batch = p.tiles_m * p.tiles_n;
  const int b = tile / tiles_per_batch, rem = tile - b * tiles_per_batch, mb = rem / p.tiles_n, nb = rem - mb * p.tiles_n;
  // blocks [f0, f1) of k of each pair of planes (an ordinary product is one pair)
  const int fold = p.fold > 0 ? p.fold : p.k_blocks, pairs = p.k_blocks / fold;
  const int f0 = fold * piece / pieces, f1 = fold * (piece + 1) / pieces;
  const int quads = 4 / pieces;  // quarters of the accumulator's lanes that a CTA finishes

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) mbar_init(&full_bar[s], 1);
    for (int s = 0; s < STAGES / 2; ++s) mbar_init(&empty_bar[s], 1);
    mbar_init(tfull_bar, 1);
    mbar_init(ready_bar, pieces - 1);
    mbar_init(recv_bar, 1);
    *abort_word = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    mbar_expect_tx(recv_bar, (pieces - 1) * quads * (BN / 4) * 512);
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if (p.tma_out) tma_prefetch_desc(&tmC);
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // everyone's barriers are there
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  dependent_wait();
  dependent_trigger();

  if (warp == 0) {
    // ------------------------------------------------ TMA producer
    const uint32_t lead = lane == 0 ? 1u : 0u;
    const uint32_t ring_at = smem_u32(smem), full_at = smem_u32(full_bar);
    const int ba = p.a_bcast ? 0 : b, bb = p.b_bcast ? 0 : b;
    const int m0 = mb * TC_BM, n0 = nb * BN;
    int stage = 0, issued = 0;
    uint32_t phase = 0;
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < pairs && ok; ++i) {
      const int za = p.fold > 0 ? ba * p.planes_a + static_cast<int>((p.pa >> (2 * i)) & 3) : ba;
      const int zb = p.fold > 0 ? bb * p.planes_b + static_cast<int>((p.pb >> (2 * i)) & 3) : bb;
#pragma unroll 1
      for (int f = f0; f < f1; ++f) {
        if ((stage & 1) == 0 && !mbar_wait_warp(&empty_bar[stage >> 1], phase ^ 1u, abort_word)) {
          ok = false;
          break;
        }
        const uint32_t bar = full_at + 8 * stage, sa = ring_at + stage * S::STAGE_BYTES, sb = sa + S::A_BYTES;
        mbar_expect_tx_lead(bar, S::STAGE_BYTES, lead);
        const int kk = f * TC_BK;
#pragma unroll 1
        for (int c = 0; c < (p.a_mn ? 2 : 1); ++c)
          tma_load_3d_lead(sa + c * 8192, &tmA, bar, p.a_mn ? m0 + c * 64 : kk, p.a_mn ? kk : m0, za, lead);
#pragma unroll 1
        for (int c = 0; c < (p.b_mn ? 2 : 1); ++c)
          tma_load_3d_lead(sb + c * 8192, &tmB, bar, p.b_mn ? n0 + c * 64 : kk, p.b_mn ? kk : n0, zb, lead);
        ++issued;
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (!ok) {  // copies in flight land before the CTA goes away
      const long long t0 = clock64();
      for (int i = issued > STAGES ? issued - STAGES : 0; i < issued; ++i)
        while (!mbar_try_wait(&full_bar[i % STAGES], (i / STAGES) & 1) && clock64() - t0 < 20000000ll) {
        }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer (see gemm_tc_kernel)
    const uint32_t lead = lane == 0 ? 1u : 0u;
    const uint32_t free_at = smem_u32(empty_bar);
    const uint64_t a_desc = p.a_mn ? umma_smem_desc_sw128(smem_u32(smem), 8192, 1024) : umma_smem_desc_sw128(smem_u32(smem), 16, 1024);
    const uint64_t b_desc = (p.b_mn ? umma_smem_desc_sw128(smem_u32(smem), 8192, 1024) : umma_smem_desc_sw128(smem_u32(smem), 16, 1024)) + (S::A_BYTES >> 4);
    const uint32_t a_step = p.a_mn ? 2048 >> 4 : 32 >> 4, b_step = p.b_mn ? 2048 >> 4 : 32 >> 4;
    const int blocks = pairs * (f1 - f0);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true, ready = false;
#pragma unroll 1
    for (int i = 0; i < blocks; ++i) {
      if (!ready && !mbar_wait_warp(&full_bar[stage], phase, abort_word)) {
        ok = false;
        break;
      }
      const int next = stage + 1 == STAGES ? 0 : stage + 1;
      ready = __all_sync(0xffffffffu, mbar_test_wait(&full_bar[next], next ? phase : phase ^ 1u)) != 0;
      tc_fence_after();
      const uint64_t ad = a_desc + (stage * S::STAGE_BYTES >> 4), bd = b_desc + (stage * S::STAGE_BYTES >> 4);
#pragma unroll
      for (int k = 0; k < TC_BK / 16; ++k)
        tc_mma_f16_lead(tmem, ad + k * a_step, bd + k * b_step, p.idesc, (i | k) != 0 ? 1u : 0u, lead);
      if (stage & 1) tc_commit_lead(free_at + 8 * (stage >> 1), lead);
      stage = next;
      if (next == 0) phase ^= 1u;
    }
    if (ok) tc_commit_lead(smem_u32(tfull_bar), lead);
    __syncwarp();
  } else if (warp >= 4) {
    // ------------------------------------------------ exchange, then the epilogue of this CTA's share of the rows
    const int q = warp & 3, half = (warp - 4) >> 2;
    const int dest = q / quads, ql = q - dest * quads;
    uint8_t* out_buf = smem + S::OUT_OFFSET + (warp - 4) * TC_OUT_BYTES;
    const uint32_t t_row = tmem + (static_cast<uint32_t>(q * 32) << 16);
    bool ok = mbar_wait_warp(tfull_bar, 0, abort_word);  // (the operands have been read: their place is free)
    tc_fence_after();
    if (ok && warp == 4 && lane < pieces && lane != piece) mbar_arrive_cluster(map_to_cta(smem_u32(ready_bar), lane));
    __syncwarp();
    if (ok && dest != piece) {
      ok = mbar_wait_warp(ready_bar, 0, abort_word);
      const uint32_t bar = map_to_cta(smem_u32(recv_bar), dest);
      const int slot = piece < dest ? piece : piece - 1;  // among the pieces other than dest
      const uint32_t dst = map_to_cta(smem_u32(smem), dest) + (slot * quads + ql) * (BN / 4) * 512 + lane * 16;
#pragma unroll 1
      for (int c = half * (BN / 2); ok && c < (half + 1) * (BN / 2); c += 32) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(t_row + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) tc_push4(dst + (c / 4 + j) * 512, bar, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
      }
    } else if (ok && mbar_wait_warp(recv_bar, 0, abort_word)) {
      auto more = [&](uint32_t (&r)[32], int c) {  // the others' parts, in the order of the pieces
#pragma unroll 1
        for (int i = 0; i < pieces - 1; ++i) {
          const uint8_t* from = smem + ((i * quads + ql) * (BN / 4) + c / 4) * 512 + lane * 16;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 v = *reinterpret_cast<const float4*>(from + j * 512);
            r[4 * j] = __float_as_uint(__uint_as_float(r[4 * j]) + v.x);
            r[4 * j + 1] = __float_as_uint(__uint_as_float(r[4 * j + 1]) + v.y);
            r[4 * j + 2] = __float_as_uint(__uint_as_float(r[4 * j + 2]) + v.z);
            r[4 * j + 3] = __float_as_uint(__uint_as_float(r[4 * j + 3]) + v.w);
          }
        }
      };
      const int m_first = mb * TC_BM + q * 32;
      if (p.tma_out) {
        tc_drain<BN>(p, &tmC, t_row, out_buf, nb * BN, m_first, b, half, lane, more);
        if (lane == 0) tma_store_wait_all<0>();
      } else {
        const int gm = m_first + lane;
        const bool row_ok = gm < p.M;
        const int esz = p.out_dtype == YTC_F32 ? 4 : 2;
        const int64_t row_off = static_cast<int64_t>(b) * p.bsc + static_cast<int64_t>(gm) * p.rsc;
        const bool vec_ok = p.csc == 1 && (((reinterpret_cast<uint64_t>(p.C) + static_cast<uint64_t>(row_off) * esz) & 15u) == 0);
#pragma unroll 1
        for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 32) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(t_row + c0, r);
          tmem_ld_wait();
          more(r, c0);
          const int gn0 = nb * BN + c0;
          if (gn0 >= p.N) continue;
          if (p.epi != EPI_NONE) tc_store_epilogue(p, r, row_off, gn0, row_ok);
          else if (p.out_dtype == YTC_BF16) tc_store_chunk<BN, YTC_BF16>(p, r, row_off, gn0, row_ok, vec_ok);
          else if (p.out_dtype == YTC_F32) tc_store_chunk<BN, YTC_F32>(p, r, row_off, gn0, row_ok, vec_ok);
          else tc_store_chunk<BN, YTC_F16>(p, r, row_off, gn0, row_ok, vec_ok);
        }
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (*abort_word && threadIdx.x < 32) {  // a give-up: what is on its way into this CTA's memory lands first
    const long long t0 = clock64();
    while (clock64() - t0 < 4000000ll) {
    }
  }
  __syncwarp();
  cluster_sync_all();  // nobody leaves while others may still write here
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem, BN);
  }
  if (threadIdx.x == 0 && *abort_word) atomicExch(p.status, YTC_TIMEOUT);
}

// ------------------------------------------------------------------ FFMA path
constexpr int SM_BM = 128, SM_BN = 128, SM_BK = 16, SM_THREADS = 256, SM_PAD = 4;

struct GemmSimtParams {
  const void* A;
  const void* B;
  void* C;
  int M, N, K;
  int64_t rsa, csa, rsb, csb, rsc, csc, bsa, bsb, bsc;
  float alpha, beta;
  int in_dtype, out_dtype;
  int tiles_m, tiles_n;
  const uint8_t* tile_live;  // masked product: 0 marks a 128 x 128 output tile nobody asks for (NULL: all computed)
  const int* gate;  // GATED: the kernel runs only if one of these `n_gate` words is set
  int n_gate;
  int scan;         // ... and for tiles of C (fp32) that hold a number that isn't finite
};

// GATED: behind a product of planes, for what that cannot form. (An instance of its own: one for both took 167 registers, and
// an SM one CTA. 8 x 500 x 700 x 100: 63 us, 84 with that.)
template <int IN_DT, bool GATED>
__global__ void __launch_bounds__(SM_THREADS, 2) gemm_simt_kernel(const GemmSimtParams p) {
  __shared__ __align__(16) float As[2][SM_BK][SM_BM + SM_PAD];
  __shared__ __align__(16) float Bs[2][SM_BK][SM_BN + SM_PAD];

  const int tid = threadIdx.x;
  const int tile = blockIdx.x;
  const int mb = tile / p.tiles_n, nb = tile - mb * p.tiles_n;
  const int m0 = mb * SM_BM, n0 = nb * SM_BN;
  if constexpr (GATED) {
    int any = 0;
    for (int i = tid; i < p.n_gate; i += SM_THREADS) any |= p.gate[i];
    if (!__syncthreads_or(any)) {
      if (!p.scan) return;
      // A product that overflows has plane products of either sign that overflow: NaN where the sum is an infinity.
      const float* c = static_cast<const float*>(p.C) + blockIdx.y * p.bsc;
      const int fast = tid % SM_BN, slow0 = tid / SM_BN;
      constexpr int AT_ONCE = 16, ROWS = SM_THREADS / SM_BN;
#pragma unroll 1
      for (int s0 = slow0; s0 < SM_BM; s0 += AT_ONCE * ROWS) {
        float v[AT_ONCE];
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) {
          const int slow = s0 + u * ROWS, r = m0 + (p.csc == 1 ? slow : fast), col = n0 + (p.csc == 1 ? fast : slow);
          v[u] = r < p.M && col < p.N ? c[r * p.rsc + col * p.csc] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) any |= !isfinite(v[u]);
      }
      if (!__syncthreads_or(any)) return;
    }
  }
  if (p.tile_live && !p.tile_live[tile]) return;
  const int b = blockIdx.y;
  const int64_t a_off = static_cast<int64_t>(b) * p.bsa;
  const int64_t b_off = static_cast<int64_t>(b) * p.bsb;

  // Loader mapping: consecutive threads walk the operand's unit-stride axis.
  const bool a_kfast = (p.csa == 1) || (p.rsa != 1);
  const bool b_nfast = (p.csb == 1) || (p.rsb != 1);

  float ra[8], rb[8];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int idx = tid + i * SM_THREADS;
      int m, kk;
      if (a_kfast) { kk = idx & (SM_BK - 1); m = idx >> 4; } else { m = idx & (SM_BM - 1); kk = idx >> 7; }
      const int gm = m0 + m, gk = k0 + kk;
      ra[i] = (gm < p.M && gk < p.K)
                  ? DType<IN_DT>::load(p.A, a_off + static_cast<int64_t>(gm) * p.rsa + static_cast<int64_t>(gk) * p.csa)
                  : 0.f;
      int n, kb;
      if (b_nfast) { n = idx & (SM_BN - 1); kb = idx >> 7; } else { kb = idx & (SM_BK - 1); n = idx >> 4; }
      const int gn = n0 + n, gk2 = k0 + kb;
      rb[i] = (gn < p.N && gk2 < p.K)
                  ? DType<IN_DT>::load(p.B, b_off + static_cast<int64_t>(gk2) * p.rsb + static_cast<int64_t>(gn) * p.csb)
                  : 0.f;
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int idx = tid + i * SM_THREADS;
      int m, kk;
      if (a_kfast) { kk = idx & (SM_BK - 1); m = idx >> 4; } else { m = idx & (SM_BM - 1); kk = idx >> 7; }
      As[buf][kk][m] = ra[i];
      int n, kb;
      if (b_nfast) { n = idx & (SM_BN - 1); kb = idx >> 7; } else { kb = idx & (SM_BK - 1); n = idx >> 4; }
      Bs[buf][kb][n] = rb[i];
    }
  };

  const int ty = tid >> 4, tx = tid & 15;
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;

  const int kt = (p.K + SM_BK - 1) / SM_BK;
  fetch(0);
  stash(0);
  __syncthreads();
  for (int t = 0; t < kt; ++t) {
    const int buf = t & 1;
    if (t + 1 < kt) fetch((t + 1) * SM_BK);
#pragma unroll
    for (int kk = 0; kk < SM_BK; ++kk) {
      const float4 a0 = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 4]);
      const float4 a1 = *reinterpret_cast<const float4*>(&As[buf][kk][64 + ty * 4]);
      const float4 b0 = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * 4]);
      const float4 b1 = *reinterpret_cast<const float4*>(&Bs[buf][kk][64 + tx * 4]);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    if (t + 1 < kt) {
      stash(buf ^ 1);
      __syncthreads();
    }
  }

  const int64_t c_off = static_cast<int64_t>(b) * p.bsc;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int gm = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4));
    if (gm >= p.M) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int gn = n0 + (j < 4 ? tx * 4 + j : 64 + tx * 4 + (j - 4));
      if (gn >= p.N) continue;
      const int64_t idx = c_off + static_cast<int64_t>(gm) * p.rsc + static_cast<int64_t>(gn) * p.csc;
      float v = p.alpha * acc[i][j];
      if (p.beta != 0.f) v += p.beta * load_as_f32(p.C, idx, p.out_dtype);
      store_from_f32(p.C, idx, v, p.out_dtype);
    }
  }
}

// beta-only update for k == 0 (C = beta * C), any strides.
__global__ void gemm_scale_c_kernel(void* C, int M, int N, int64_t rsc, int64_t csc, int64_t bsc, float beta,
                                    int out_dtype) {
  const int64_t total = static_cast<int64_t>(M) * N;
  const int64_t c_off = static_cast<int64_t>(blockIdx.y) * bsc;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t m = i / N, n = i - m * N;
    const int64_t idx = c_off + m * rsc + n * csc;
    const float v = (beta == 0.f) ? 0.f : beta * load_as_f32(C, idx, out_dtype);
    store_from_f32(C, idx, v, out_dtype);
  }
}

// ------------------------------------------------------------------ host dispatch
static bool tc_operand_ok(const void* ptr, int64_t rs, int64_t cs, int64_t bs, int64_t batch, int rows, int cols,
                          int* mn_major) {
  // rows x cols operand with the reduction axis K as `cols` for A (A[m,k]) and as `rows` for B (B[k,n]):
  // the caller passes (unit-stride axis along K ?) through which stride is 1.
  (void)rows;
  (void)cols;
  if ((reinterpret_cast<uint64_t>(ptr) & 15u) != 0) return false;
  int64_t lead;
  if (cs == 1) {
    *mn_major = 0;
    lead = rs;
  } else if (rs == 1) {
    *mn_major = 1;
    lead = cs;
  } else {
    return false;
  }
  if (lead <= 0 || (lead * 2) % 16 != 0) return false;
  if (batch > 1 && bs != 0 && (bs < 0 || (bs * 2) % 16 != 0)) return false;
  return true;
}

// L2 prefetch distance of the A operand in k-blocks (see GemmTcParams::a_prefetch).
static std::atomic<int> g_tc_a_prefetch{0};
// 1 = fetch K-major operand tiles as 64-row boxes instead of one tall box.
static std::atomic<int> g_tc_split_loads{0};
// CTA-pair kernel: 0 = automatic, 1 = whenever the layout allows, 2 = never.
static std::atomic<int> g_tc_pair{0};

// Masked products (YTensor::masked_matmul): what the entry point asked for, seen by the launchers below.
// kind 0: no mask; 1: bool matrix [m, n]; 2: the causal predicate j <= i + offset, evaluated on the device.
struct MaskCtx {
  int kind = 0;
  const uint8_t* mask = nullptr;
  int64_t row_stride = 0;
  int offset = 0;
};
static thread_local MaskCtx g_mask;

__device__ __forceinline__ bool mask_at(int kind, const uint8_t* mask, int64_t mrs, int offset, int i, int j) {
  return kind == 2 ? (j <= i + offset) : (mask[static_cast<int64_t>(i) * mrs + j] != 0);
}

// live[mb * tiles_n + nb] = 1 when some element of output tile (mb, nb) is asked for. The counterpart of the
// tileAllFalse test that lets the reference's sgemm_masked skip whole tiles (src/kernel/avx2/sgemm.inl:449-475).
__global__ void __launch_bounds__(256) gemm_tile_live_kernel(uint8_t* live, int kind, const uint8_t* mask, int64_t mrs,
                                                             int offset, int m, int n, int bm, int bn, int tiles_n) {
  const int mb = blockIdx.x / tiles_n, nb = blockIdx.x - mb * tiles_n;
  const int i0 = mb * bm, j0 = nb * bn;
  const int i1 = i0 + bm < m ? i0 + bm : m, j1 = j0 + bn < n ? j0 + bn : n;
  int any = 0;
  if (kind == 2) {
    any = j0 <= (i1 - 1) + offset;  // the tile's smallest column against its largest row
  } else {
    const int w = j1 - j0;
    for (int e = threadIdx.x; e < (i1 - i0) * w && !any; e += 256) {
      const int i = i0 + e / w, j = j0 + e % w;
      any = mask[static_cast<int64_t>(i) * mrs + j] != 0;
    }
  }
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) live[blockIdx.x] = any ? 1 : 0;
}

// Tile liveness for the current mask and a bm x bn tiling, in stream-ordered scratch (freed by the caller's launcher
// after its kernel has been queued). NULL without a mask.
static int make_tile_live(int m, int n, int bm, int bn, cudaStream_t st, uint8_t** out) {
  *out = nullptr;
  if (g_mask.kind == 0) return YTC_OK;
  const int tiles_m = (m + bm - 1) / bm, tiles_n = (n + bn - 1) / bn;
  uint8_t* live = nullptr;
  YTC_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&live), static_cast<size_t>(tiles_m) * tiles_n, st));
  gemm_tile_live_kernel<<<tiles_m * tiles_n, 256, 0, st>>>(live, g_mask.kind, g_mask.mask, g_mask.row_stride,
                                                          g_mask.offset, m, n, bm, bn, tiles_n);
  count_launch();
  *out = live;
  return YTC_OK;
}

// A product of planes: operand A is [batch][planes_a][rows][cols] with plane_a elements a plane (its batch stride is
// planes_a * plane_a), B likewise; the accumulator takes `pairs` plane products in the order of pa / pb (two bits a pair).
struct TcPlanes {
  int planes_a, planes_b, pairs;
  uint32_t pa, pb;
  int64_t plane_a, plane_b;
};

// Whether CTA pairs take this product (large problems; small ones keep one CTA per tile: more tiles to spread over the SMs).
static bool tc_takes_pairs(int m, int n, int64_t k, int64_t batch) {
  return g_mask.kind == 0 && g_tc_pair != 2 &&
         (g_tc_pair == 1 || (m >= 512 && n >= 256 && k >= 256 &&
                             static_cast<int64_t>((m + 255) / 256) * ((n + 255) / 256) * batch >= 74));
}
static int tc_tile_n(int m, int n, int64_t batch) {
  return (n <= 128 || static_cast<int64_t>((m + 127) / 128) * ((n + 255) / 256) * batch < sm_count() / 2) ? 128 : 256;
}
// Pieces of k for gemm_split_kernel (0: not its product): as many as keep every CTA resident (66 clusters of two fit any B200
// seen, 33 of four) and leave a piece eight blocks of k, the exchange costing about as much as seven (2 us). (256 x 256 tiles of two
// pairs of CTAs for products of 72 to 132 tiles of 128, half the operand bytes per result, lost: 2000 x 1024 x 2048 14.4 -> 17.4 us.)
static int tc_cluster(int m, int n, int64_t fold, int64_t pairs, int64_t batch) {
  if (g_mask.kind != 0 || g_tc_pair != 0 || g_tc_split_loads) return 0;
  const int64_t tiles = static_cast<int64_t>((m + 127) / 128) * ((n + 127) / 128) * batch, blocks = fold * pairs;
  if (tiles <= 33 && blocks >= 32 && fold >= 4) return 4;
  if (tiles <= 66 && blocks >= 16 && fold >= 2) return 2;
  return 0;
}
// Pieces of k that fill the SMs when the tiles alone leave more than half of them idle; a piece keeps 512 / pairs of k. Not for
// products of less than 6144 / pairs of k: they take a cluster's pieces, if any, need no scratch and no second launch, and stay below
// the 16 us that a call of api.matmul takes by itself. One call behind the other from C, bf16, without / with pieces: 16 x 1024 x k,
// k = 2048 10.4 / 8.0 us, 4096 12.4 / 7.9, 6144 14.4 / 8.7, 8192 16.5 / 8.5, 16384 22.6 / 11.1; 300 x 512 x 4096 12.4 / 9.9, x 6144
// 14.4 / 10.9; 128 x 4096 x 6144 16.1 / 16.9.
constexpr int SPLIT_MIN_BLOCKS = 96;
static int tc_splits(int m, int n, int k, int pairs, int64_t batch) {
  const int k_blocks = (k + TC_BK - 1) / TC_BK;
  if (g_mask.kind != 0 || g_tc_pair != 0 || tc_takes_pairs(m, n, static_cast<int64_t>(k) * pairs, batch)) return 1;
  const int bn = tc_tile_n(m, n, batch);
  const int64_t tiles = static_cast<int64_t>((m + 127) / 128) * ((n + bn - 1) / bn) * batch;
  if (tiles * 2 > sm_count()) return 1;
  if (static_cast<int64_t>(k_blocks) * pairs < SPLIT_MIN_BLOCKS) return 1;
  const int64_t most = static_cast<int64_t>(k_blocks) * pairs / 8;
  int64_t want = sm_count() / tiles < most ? sm_count() / tiles : most;
  if (want > k_blocks) want = k_blocks;
  if (want < 2) return 1;
  // (a cluster's pieces need no scratch and no second launch; more than four only where they are many more)
  if (want <= 6 && tc_cluster(m, n, k_blocks, pairs, batch)) return 1;
  const int64_t per = (k_blocks + want - 1) / want;
  return static_cast<int>((k_blocks + per - 1) / per);
}

static int launch_tc(int dtype_in, int dtype_out, const void* A, const void* B, void* C, int m, int n, int k,
                     float alpha, float beta, int a_mn, int64_t lda, int b_mn, int64_t ldb, int64_t rsc, int64_t csc,
                     int64_t batch, int64_t bsa, int64_t bsb, int64_t bsc, cudaStream_t st,
                     const LinearEpilogue* ex = nullptr, const TcPlanes* pl = nullptr, int splits = 1) {
  // A: unit axis = K (a_mn 0, dims {K, M}) or M (a_mn 1, dims {M, K}). B likewise with N.
  CUtensorMap tmA, tmB;
  const int a_bcast = (batch > 1 && bsa == 0) ? 1 : 0;
  const int b_bcast = (batch > 1 && bsb == 0) ? 1 : 0;
  // 256-wide tiles unless the problem is narrow or would leave most SMs without a tile
  const int BN = tc_tile_n(m, n, batch);
  // (a masked product keeps one CTA per tile: the tile-skipping form of the kernel)
  const bool grouped = ex && ex->tile_group;
  // (k pieces are work items of the one-CTA kernel; gemm_tc2_kernel knows whole products only)
  const bool pair = !grouped && splits == 1 && tc_takes_pairs(m, n, pl ? static_cast<int64_t>(k) * pl->pairs : k, batch);
  // Linear layers of the 16-bit models keep k in one accumulator: the last bit of a partial sum becomes a step of bf16 in what is
  // stored and the layers behind carry it on, so a token's logits would depend on how many tokens its prompt has. (500 tokens through
  // 12 Derupel layers: 0.11 ms more than with shared k, and the same bits in any company.)
  const bool one_sum = ex && !ex->add_in_memory;
  const int cluster = grouped || pair || splits > 1 || one_sum ? 0 : tc_cluster(m, n, (k + TC_BK - 1) / TC_BK, pl ? pl->pairs : 1, batch);
  if (splits > 1 && (ex || g_mask.kind != 0 || splits > (k + TC_BK - 1) / TC_BK)) {
    set_last_error("ytcuda_gemm: %d pieces of k = %d do not go with an epilogue or a mask", splits, k);
    return YTC_UNSUPPORTED;
  }
  {
    const uint64_t nb = (a_bcast || batch == 1) ? 1 : static_cast<uint64_t>(batch);
    uint64_t dims[3], strides[2];
    uint32_t box[3];
    if (!a_mn) { dims[0] = k; dims[1] = m; box[0] = TC_BK; box[1] = g_tc_split_loads ? 64 : TC_BM; }
    else       { dims[0] = m; dims[1] = k; box[0] = 64;    box[1] = TC_BK; }
    dims[2] = nb * (pl ? pl->planes_a : 1);
    box[2] = 1;
    strides[0] = static_cast<uint64_t>(lda) * 2;
    strides[1] = pl ? static_cast<uint64_t>(pl->plane_a) * 2 : (nb > 1) ? static_cast<uint64_t>(bsa) * 2 : strides[0] * dims[1];
    int s = encode_tensor_map(&tmA, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, A, dims, strides, box,
                              CU_TENSOR_MAP_SWIZZLE_128B);
    if (s != YTC_OK) return s;
  }
  {
    const uint64_t nb = (b_bcast || batch == 1) ? 1 : static_cast<uint64_t>(batch);
    uint64_t dims[3], strides[2];
    uint32_t box[3];
    const uint64_t b_rows = grouped ? static_cast<uint64_t>(n) * ex->groups : static_cast<uint64_t>(n);
    if (!b_mn) { dims[0] = k; dims[1] = b_rows; box[0] = TC_BK; box[1] = pair || cluster ? 128u : (g_tc_split_loads ? 64u : static_cast<uint32_t>(BN)); }
    else       { dims[0] = n; dims[1] = k; box[0] = 64;    box[1] = TC_BK; }
    dims[2] = nb * (pl ? pl->planes_b : 1);
    box[2] = 1;
    strides[0] = static_cast<uint64_t>(ldb) * 2;
    strides[1] = pl ? static_cast<uint64_t>(pl->plane_b) * 2 : (nb > 1) ? static_cast<uint64_t>(bsb) * 2 : strides[0] * dims[1];
    int s = encode_tensor_map(&tmB, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, B, dims, strides, box,
                              CU_TENSOR_MAP_SWIZZLE_128B);
    if (s != YTC_OK) return s;
  }
  GemmTcParams p;
  p.M = m; p.N = n; p.K = k;
  p.batch = static_cast<int>(batch);
  p.a_mn = a_mn; p.b_mn = b_mn;
  p.a_bcast = a_bcast || batch == 1; p.b_bcast = b_bcast || batch == 1;
  p.idesc = umma_idesc(dtype_in == YTC_BF16 ? 1u : 0u, a_mn, b_mn, TC_BM, BN);
  p.alpha = alpha; p.beta = beta;
  p.C = C; p.rsc = rsc; p.csc = csc; p.bsc = bsc;
  p.out_dtype = dtype_out;
  p.tiles_m = (m + TC_BM - 1) / TC_BM;
  p.tiles_n = (n + BN - 1) / BN;
  const int64_t total = static_cast<int64_t>(p.tiles_m) * p.tiles_n * batch * splits;
  if (total > 0x7FFFFFFFll) {
    set_last_error("ytcuda_gemm: too many tiles (%lld)", (long long)total);
    return YTC_UNSUPPORTED;
  }
  p.total_tiles = static_cast<int>(total);
  p.k_blocks = (k + TC_BK - 1) / TC_BK;
  p.fold = 0;
  p.splits = splits;
  p.split_blocks = (p.k_blocks + splits - 1) / splits;
  if (pl) {  // (every piece holds its share of k of all pairs)
    p.fold = p.split_blocks;
    p.split_blocks *= pl->pairs;
    p.k_blocks = p.split_blocks;
    p.planes_a = pl->planes_a; p.planes_b = pl->planes_b; p.pa = pl->pa; p.pb = pl->pb;
  }
  const bool pieces = pl || splits > 1;
  p.a_prefetch = pieces ? 0 : g_tc_a_prefetch.load();
  p.split_loads = g_tc_split_loads;
  p.n_step = TC2_BN;
  p.n_cta = TC2_BN / 2;
  p.tile_live = nullptr;
  const LinearEpilogue none, *e = ex ? ex : &none;
  p.epi = e->epi;
  // C through TMA stores: rows (and batch items, pieces of k) that start at 16 bytes. What C holds already is added there only
  // where the caller leaves that to the memory's adders (IEEE sums like an epilogue's, subnormal numbers kept: 1024 sums of such
  // operands the same bits as the host's; the epilogue's own reads of C cost a prompt of 2000 tokens 1.6 %).
  const int esz = dtype_size(dtype_out);
  const int64_t items = batch * splits;
  const bool rows16 = csc == 1 && rsc > 0 && (reinterpret_cast<uint64_t>(C) & 15u) == 0 && rsc * esz % 16 == 0 &&
                      rsc * esz < (int64_t{1} << 40) && (items == 1 || (bsc > 0 && bsc * esz % 16 == 0 && bsc * esz < (int64_t{1} << 40)));
  p.tma_out = !rows16 ? 0 : beta == 0.f ? 1 : e->add_in_memory && beta == 1.f && alpha == 1.f && dtype_out == YTC_F32 ? 2 : 0;
  CUtensorMap tmC{};
  if (p.tma_out) {
    const bool planes_out = e->epi == EPI_SWIGLU_PLANES;  // C is [2][m][n / 2]
    const uint64_t dims[3] = {static_cast<uint64_t>(epi_pairs(e->epi) || planes_out ? n / 2 : n), static_cast<uint64_t>(m),
                              static_cast<uint64_t>(planes_out ? 2 : items)};
    const uint64_t strides[2] = {static_cast<uint64_t>(rsc * esz), items > 1 ? static_cast<uint64_t>(bsc * esz) : static_cast<uint64_t>(rsc * esz) * m};
    const uint32_t box[3] = {static_cast<uint32_t>(128 / esz), 32, 1};
    if (strides[1] >= (uint64_t{1} << 40)) p.tma_out = 0;
    else {
      const int s = encode_tensor_map(&tmC, esz == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, C, dims, strides,
                                      box, CU_TENSOR_MAP_SWIZZLE_128B);
      if (s != YTC_OK) return s;
    }
  }
  p.act_cols = e->act_cols;
  p.limit = e->limit; p.alpha_gate = e->alpha; p.shift = e->shift;
  p.tile_group = grouped ? ex->tile_group : nullptr;
  p.group_rows = n;
  p.status = device_status_word();
  if (!p.status) {
    set_last_error("ytcuda_gemm: no device status word");
    return YTC_CUDA_ERROR;
  }
  if (cluster) {
    p.cluster = cluster;
    p.idesc = umma_idesc(dtype_in == YTC_BF16 ? 1u : 0u, a_mn, b_mn, TC_BM, 128);
    p.tiles_n = (n + 127) / 128;
    p.total_tiles = static_cast<int>(static_cast<int64_t>(p.tiles_m) * p.tiles_n * batch);
    const int s = ensure_dynamic_smem(reinterpret_cast<const void*>(gemm_split_kernel), TcSmem<128>::DYN_STAGED);
    if (s != YTC_OK) return s;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(p.total_tiles * cluster));
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = TcSmem<128>::DYN_STAGED;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap_scope() ? 2 : 1;
    YTC_CUDA(cudaLaunchKernelEx(&cfg, gemm_split_kernel, tmA, tmB, tmC, p));
    count_launch();
    YTC_CUDA(cudaGetLastError());
    return YTC_OK;
  }
  if (pair) {
    p.idesc = umma_idesc(dtype_in == YTC_BF16 ? 1u : 0u, a_mn, b_mn, 256, TC2_BN);
    p.tiles_m = (m + 255) / 256;
    p.tiles_n = (n + TC2_BN - 1) / TC2_BN;
    if (e->epi == EPI_SWIGLU_PLANES) {  // 128 gates and their 128 ups a tile
      p.N = n / 2;
      p.n_step = 128;
      p.n_cta = n / 2;
      p.tiles_n = (n / 2 + 127) / 128;
    }
    p.total_tiles = static_cast<int>(static_cast<int64_t>(p.tiles_m) * p.tiles_n * batch);
    const int smem = p.tma_out ? Tc2Smem::DYN_STAGED : Tc2Smem::DYN_BYTES;
    int clusters = sm_count() / 2;
    if (clusters > p.total_tiles) clusters = p.total_tiles;
    {
      const int s = ensure_dynamic_smem(reinterpret_cast<const void*>(pieces ? gemm_tc2_kernel<true> : gemm_tc2_kernel<false>), smem);
      if (s != YTC_OK) return s;
    }
    YTC_CUDA(launch_overlapped(pieces ? gemm_tc2_kernel<true> : gemm_tc2_kernel<false>, dim3(clusters * 2), dim3(TC_THREADS), smem, st, tmA, tmB, tmC, p));
    count_launch();
    YTC_CUDA(cudaGetLastError());
    return YTC_OK;
  }
  const int grid = p.total_tiles < sm_count() ? p.total_tiles : sm_count();
  uint8_t* live = nullptr;
  {
    const int s = make_tile_live(m, n, TC_BM, BN, st, &live);
    if (s != YTC_OK) return s;
    p.tile_live = live;
  }
  if (BN == 256) {
    const int smem = p.tma_out ? TcSmem<256>::DYN_STAGED : TcSmem<256>::DYN_BYTES;
    auto* fn = pieces ? gemm_tc_kernel<256, true> : gemm_tc_kernel<256, false>;
    const int s = ensure_dynamic_smem(reinterpret_cast<const void*>(fn), smem);
    if (s != YTC_OK) return s;
    YTC_CUDA(launch_overlapped(fn, dim3(grid), dim3(TC_THREADS), smem, st, tmA, tmB, tmC, p));
  } else {
    const int smem = p.tma_out ? TcSmem<128>::DYN_STAGED : TcSmem<128>::DYN_BYTES;
    auto* fn = pieces ? gemm_tc_kernel<128, true> : gemm_tc_kernel<128, false>;
    const int s = ensure_dynamic_smem(reinterpret_cast<const void*>(fn), smem);
    if (s != YTC_OK) return s;
    YTC_CUDA(launch_overlapped(fn, dim3(grid), dim3(TC_THREADS), smem, st, tmA, tmB, tmC, p));
  }
  count_launch();
  if (live) cudaFreeAsync(live, st);
  YTC_CUDA(cudaGetLastError());
  return YTC_OK;
}

// y[m, n] = epilogue(x[m, k] . W[n, k]^T) on the tensor cores (lm_ops.cuh).
int linear_tc(const void* x, int64_t ldx, const void* w, int64_t ldw, void* y, int64_t ldy, int out_dtype, int m, int n,
              int k, const LinearEpilogue& ex, cudaStream_t st) {
  if (m <= 0 || n <= 0) return YTC_OK;
  int unused;
  YTC_REQUIRE(tc_operand_ok(x, ldx, 1, 0, 1, m, k, &unused) && tc_operand_ok(w, ldw, 1, 0, 1, n, k, &unused),
              "linear_tc: operand rows must be 16-byte aligned");
  YTC_REQUIRE(ex.epi == EPI_NONE || out_dtype == YTC_BF16, "linear_tc: fused epilogues store bf16");
  YTC_REQUIRE(!epi_pairs(ex.epi) || n % 2 == 0, "linear_tc: an odd number of gate / up rows");
  YTC_REQUIRE(!ex.tile_group || m % TC_BM == 0, "linear_tc: grouped rows come in blocks of %d", TC_BM);
  return launch_tc(YTC_BF16, out_dtype, x, w, y, m, n, k, 1.f, 0.f, 0, ldx, 0, ldw, ldy, 1, 1, 0, 0, 0, st, &ex);
}

static int launch_simt(int dtype_in, int dtype_out, const void* A, const void* B, void* C, int m, int n, int k,
                       float alpha, float beta, int64_t rsa, int64_t csa, int64_t rsb, int64_t csb, int64_t rsc,
                       int64_t csc, int64_t batch, int64_t bsa, int64_t bsb, int64_t bsc, cudaStream_t st,
                       const int* gate = nullptr, int n_gate = 0, bool scan = false) {
  GemmSimtParams p;
  p.gate = gate; p.n_gate = n_gate; p.scan = scan;
  p.A = A; p.B = B; p.C = C;
  p.M = m; p.N = n; p.K = k;
  p.rsa = rsa; p.csa = csa; p.rsb = rsb; p.csb = csb; p.rsc = rsc; p.csc = csc;
  p.bsa = bsa; p.bsb = bsb; p.bsc = bsc;
  p.alpha = alpha; p.beta = beta;
  p.in_dtype = dtype_in; p.out_dtype = dtype_out;
  p.tiles_m = (m + SM_BM - 1) / SM_BM;
  p.tiles_n = (n + SM_BN - 1) / SM_BN;
  uint8_t* live = nullptr;
  {
    const int s = make_tile_live(m, n, SM_BM, SM_BN, st, &live);
    if (s != YTC_OK) return s;
    p.tile_live = live;
  }
  const int64_t tiles = static_cast<int64_t>(p.tiles_m) * p.tiles_n;
  if (tiles > 0x7FFFFFFFll || batch > 65535) {
    // gridDim.y is limited to 65535: split the batch.
    if (tiles > 0x7FFFFFFFll) {
      set_last_error("ytcuda_gemm: too many tiles");
      return YTC_UNSUPPORTED;
    }
  }
  for (int64_t b0 = 0; b0 < batch; b0 += 65535) {
    const int64_t nb = (batch - b0 < 65535) ? batch - b0 : 65535;
    GemmSimtParams q = p;
    q.A = static_cast<const char*>(A) + b0 * bsa * dtype_size(dtype_in);
    q.B = static_cast<const char*>(B) + b0 * bsb * dtype_size(dtype_in);
    q.C = static_cast<char*>(C) + b0 * bsc * dtype_size(dtype_out);
    dim3 grid(static_cast<unsigned>(tiles), static_cast<unsigned>(nb));
    if (gate) gemm_simt_kernel<YTC_F32, true><<<grid, SM_THREADS, 0, st>>>(q);
    else if (dtype_in == YTC_F32) gemm_simt_kernel<YTC_F32, false><<<grid, SM_THREADS, 0, st>>>(q);
    else if (dtype_in == YTC_BF16) gemm_simt_kernel<YTC_BF16, false><<<grid, SM_THREADS, 0, st>>>(q);
    else gemm_simt_kernel<YTC_F16, false><<<grid, SM_THREADS, 0, st>>>(q);
    count_launch();
  }
  if (live) cudaFreeAsync(live, st);
  YTC_CUDA(cudaGetLastError());
  return YTC_OK;
}

// Operands that the TMA cannot take as they lie, rewritten: fp32 as three bf16 planes, x = h + m + l with h = bf16(x),
// m = bf16(x - h), l = bf16(x - h - m), which together carry the 24 mantissa bits of x (the differences are exact in fp32);
// 16-bit operands of odd strides as they are. Rows of `cols` elements become rows of a multiple of 8, zeros behind the end.
// Of the nine plane products of an fp32 GEMM the six that matter, (l,h) (m,m) (h,l) (m,h) (h,m) (h,h), smallest first, form
// in one accumulator (TcPlanes). Non-finite values keep m = l = 0 (an infinite operand then meets zero planes of the other
// operand and the sum becomes NaN where the FFMA kernel gives the infinity), and below 2^-110 the last plane would lie under
// bf16's smallest number; `unfit`, a word per block, says whether there were any of either. fp16 numbers below the normal ones are doubled, which is how the reference's type and the FFMA kernel read them.
struct PlaneOp {
  const void* x;
  int64_t rs, cs, bs;
  int rows, cols, cols8;   // cols8: groups of 8 columns of an output row
  int64_t n8;              // groups over all rows and batch items
  uint16_t* out;
  int64_t plane;           // elements of a plane of one batch item
  int blocks;
  int wide;                // fp32: groups of 8 can be read 16 bytes at a time
};
// One launch for both operands: CTAs [0, a.blocks) take a, the rest b. Bound by memory: 4 bytes read, 6 written a value.
// `keep`: the words in `unfit` hold what an earlier launch saw of the same operands, and stay set.
template <int DT>
__global__ void __launch_bounds__(256) gemm_planes_kernel(const PlaneOp oa, const PlaneOp ob, int* unfit, int keep) {
  dependent_wait();     // (under a programmatic dependent launch: the kernel before this one has finished)
  dependent_trigger();  // the kernel queued behind this one may be scheduled and set itself up meanwhile
  constexpr int PLANES = DT == YTC_F32 ? 3 : 1;
  const bool second = static_cast<int>(blockIdx.x) >= oa.blocks;
  const PlaneOp& op = second ? ob : oa;
  const int64_t block = static_cast<int64_t>(blockIdx.x) - (second ? oa.blocks : 0);
  bool bad = false;
  for (int64_t t = block * 256 + threadIdx.x; t < op.n8; t += op.blocks * 256ll) {
    const int64_t row = t / op.cols8;  // (of all batch items)
    const int c = static_cast<int>(t - row * op.cols8) * 8;
    const int64_t b = row / op.rows, i = row - b * op.rows;
    const int64_t from = b * op.bs + i * op.rs + c * op.cs;
    uint16_t p[PLANES][8];
    if constexpr (DT == YTC_F32) {
      float v[8];
      if (op.wide && c + 8 <= op.cols) {
        const float4 v0 = *reinterpret_cast<const float4*>(static_cast<const float*>(op.x) + from);
        const float4 v1 = *reinterpret_cast<const float4*>(static_cast<const float*>(op.x) + from + 4);
        v[0] = v0.x; v[1] = v0.y; v[2] = v0.z; v[3] = v0.w; v[4] = v1.x; v[5] = v1.y; v[6] = v1.z; v[7] = v1.w;
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = c + e < op.cols ? static_cast<const float*>(op.x)[from + e * op.cs] : 0.f;
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        __nv_bfloat16 q = __float2bfloat16_rn(v[e]);
        float fh = __bfloat162float(q);
        if (!isfinite(fh) && isfinite(v[e])) {
          // a finite value so close to the largest float that rounding its top plane overflows: truncate instead, the
          // two lower planes still hold the remaining 16 mantissa bits exactly
          fh = __uint_as_float(__float_as_uint(v[e]) & 0xffff0000u);
          q = __float2bfloat16_rn(fh);
        }
        p[0][e] = *reinterpret_cast<const uint16_t*>(&q);
        p[1][e] = p[2][e] = 0;
        bad |= (__float_as_uint(v[e]) & 0x7FFFFFFFu) - 1u < 0x08800000u - 1u;  // (below 2^-110, but not zero)
        if (isfinite(fh)) {
          const float r1 = v[e] - fh;
          q = __float2bfloat16_rn(r1);
          p[1][e] = *reinterpret_cast<const uint16_t*>(&q);
          q = __float2bfloat16_rn(r1 - __bfloat162float(q));
          p[2][e] = *reinterpret_cast<const uint16_t*>(&q);
        } else {
          bad = true;
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        uint16_t h = c + e < op.cols ? static_cast<const uint16_t*>(op.x)[from + e * op.cs] : 0;
        if (DT == YTC_F16 && (h & 0x7C00u) == 0) h = static_cast<uint16_t>((h & 0x8000u) | ((h & 0x3FFu) << 1));
        p[0][e] = h;
      }
    }
    uint16_t* o = op.out + b * op.plane * PLANES + (i * op.cols8 * 8 + c);
#pragma unroll
    for (int i3 = 0; i3 < PLANES; ++i3) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = p[i3][2 * e] | (static_cast<uint32_t>(p[i3][2 * e + 1]) << 16);
      *reinterpret_cast<uint4*>(o + i3 * op.plane) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  const int any = __syncthreads_or(bad);
  if (unfit && threadIdx.x == 0) unfit[blockIdx.x] = any | (keep ? unfit[blockIdx.x] : 0);
}

// C = alpha * (the sum of the partial sums, in their order) + beta * C; part is [splits][batch][m][ldp], `stride` elements each.
// `unfit` (may be null) is set where a sum isn't finite.
__global__ void __launch_bounds__(256) gemm_sum_kernel(const float* part, int splits, int64_t stride, int64_t total, int m, int n,
                                                       int64_t ldp, void* C, int dt, int64_t rsc, int64_t csc, int64_t bsc,
                                                       float alpha, float beta, int* unfit) {
  dependent_wait();
  dependent_trigger();
  bool bad = false;
  for (int64_t t = blockIdx.x * 256ll + threadIdx.x; t < total; t += gridDim.x * 256ll) {
    // (64-bit divisions took most of the kernel: 2048 x 2500, four pieces, 81 us under the profiler)
    const int64_t row = total <= 0xffffffffll ? static_cast<uint32_t>(t) / static_cast<uint32_t>(n) : t / n, col = t - row * n;
    const float* from = part + row * ldp + col;
    float v = 0.f;
#pragma unroll 8
    for (int s = 0; s < splits; ++s) v += from[s * stride];
    const int64_t b = row < m ? 0 : total <= 0xffffffffll ? static_cast<uint32_t>(row) / static_cast<uint32_t>(m) : row / m;
    const int64_t at = b * bsc + (row - b * m) * rsc + col * csc;
    v *= alpha;
    if (beta != 0.f) v += beta * load_as_f32(C, at, dt);
    store_from_f32(C, at, v, dt);
    bad |= !isfinite(v);
  }
  if (unfit && bad) *unfit = 1;
}

// C[b][i][j] = masked_value wherever mask[i][j] == 0 (the mask is shared by every batch item); the second half of
// YTensor::masked_matmul (reference src/ytensor_math.inl:1053-1090 fills the output with maskedValue and lets
// sgemm_masked write the masked-in products only).
__global__ void __launch_bounds__(256) gemm_apply_mask_kernel(void* C, int dt, int m, int n, int64_t rsc, int64_t csc,
                                                              int64_t batch, int64_t bsc, const uint8_t* mask,
                                                              int64_t mask_rs, float masked_value, int causal,
                                                              int offset) {
  const int64_t per = static_cast<int64_t>(m) * n;
  const int64_t total = per * batch;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t b = t / per, r = t - b * per;
    const int i = static_cast<int>(r / n), j = static_cast<int>(r - static_cast<int64_t>(i) * n);
    const bool keep = causal ? (j <= i + offset) : (mask[static_cast<int64_t>(i) * mask_rs + j] != 0);
    if (!keep) store_from_f32(C, b * bsc + i * rsc + j * csc, masked_value, dt);
  }
}

// Which kernel ytcuda_gemm picks: 0 = automatic, 1 = force FFMA, 2 = require tcgen05.
static std::atomic<int> g_gemm_path{0};

// fp32 GEMM on the tensor cores (see gemm_planes_kernel): 0 = automatic (where it is faster), 1 = never,
// 2 = whenever the shapes allow.
static std::atomic<int> g_f32_split{0};

// What FFMA and the planes take, as estimates: FFMA 0.17 to 0.22 us (fp32; 16 bit 0.25 to 0.36) per element of k and wave of 128 x 128
// tiles, the less where the left operand has few rows to load; the planes 19 us of launches, 10 bytes of traffic a value, six products a
// sixth of the tensor rate, and 8 bytes per result and 256 of k for their partial sums. The callers ask for a ratio of 1.5, and the
// estimate of the planes is high by up to 10 us for small operands since the products behind them became shorter, so the line lies on
// FFMA's side: what is near it keeps FFMA's sums and needs no scratch. One call behind the other, FFMA / planes, us, * on FFMA's side:
// fp32 1 x 512 x 60 14.5 / 13.1 *, x 120 26.7 / 14.4 *, x 180 37.0 / 16.5, 60 x 1001 x 180
// 47.2 / 18.5, 16 x 4096 x 120 34.9 / 16.5 *, x 180 47.1 / 18.5, 2000 x 500 x 180 61.5 / 22.6 *, x 257 75.9 / 28.8, 777 x 1001 x 777
// 168 / 38; bf16 1 x 513 x 101 26.7 / 8.2 *, x 131 32.9 / 8.2, 60 x 1002 x 75 32.8 / 13.9 *, x 101 41.0 / 14.1, 777 x 1001 x 501 172 / 28.
static double simt_us(int m, int n, int k, int64_t batch, bool wide) {
  const int64_t tiles = static_cast<int64_t>((m + SM_BM - 1) / SM_BM) * ((n + SM_BN - 1) / SM_BN) * batch;
  const double each = wide ? (m < 16 ? 0.17 : 0.22) : (m < 16 ? 0.25 : 0.36);
  return each * k * static_cast<double>((tiles + sm_count() - 1) / sm_count());
}
static double planes_us(int m, int n, int k, int64_t batch, bool b_shared, bool wide) {
  const double values = static_cast<double>(m) * k * batch + static_cast<double>(k) * n * (b_shared ? 1 : batch);
  const double sums = wide ? static_cast<double>(m) * n * batch * ((k + 255) / 256) * 8 : 0.0;
  return 19.0 + (values * (wide ? 10 : 4) + sums) / 3e6 + 2.0 * m * n * k * batch * (wide ? 6 : 1) / 5e8;
}

// 0: FFMA, 1: planes, as for every large problem, 2: planes where FFMA is slower, with FFMA behind them for what has none
static int f32_planes_form(int m, int n, int k, float beta, int64_t rsc, int64_t csc, int64_t bsc, int64_t batch, int64_t bsb) {
  if (g_f32_split == 1) return 0;
  if (rsc < 0 || csc < 0 || bsc < 0) return 0;
  if (k % 8 == 0 && n % 8 == 0 && (g_f32_split == 2 ? n >= 8 && k >= 8 : m >= 256 && n >= 256 && k >= 256)) return 1;
  return g_mask.kind == 0 && beta == 0.f && simt_us(m, n, k, batch, true) > 1.5 * planes_us(m, n, k, batch, bsb == 0, true) ? 2 : 0;
}

static bool stream_captures(cudaStream_t st) {  // (scratch that grows inside a capture would belong to the graph)
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone;
}

// The product through rewritten operands (gemm_planes_kernel), k cut into pieces where the tiles are few. `check`: FFMA runs
// behind it if an operand held a number without planes (beta must be 0). NO_SCRATCH: nothing was queued.
constexpr int NO_SCRATCH = -1;
template <int DT>
static int launch_planes(const void* A, const void* B, void* C, int dtype_out, int m, int n, int k, float alpha, float beta,
                         int64_t rsa, int64_t csa, int64_t rsb, int64_t csb, int64_t rsc, int64_t csc, int64_t batch,
                         int64_t bsa, int64_t bsb, int64_t bsc, bool check, cudaStream_t st) {
  // the launches are one chain of dependent kernels: each is scheduled while the one before it still runs
  struct Scope {
    bool was = overlap_scope();
    Scope() { overlap_scope() = true; }
    ~Scope() { overlap_scope() = was; }
  } scope;
  const WorkspaceScope workspace(st);
  constexpr int PLANES = DT == YTC_F32 ? 3 : 1;
  const int esz = dtype_size(DT);
  const bool a_shared = batch > 1 && bsa == 0, b_shared = batch > 1 && bsb == 0;
  // rows along the operand's unit stride: A as [m][k] or [k][m], B as [k][n] or [n][k]
  const bool a_mn = csa != 1 && rsa == 1, b_kn = csb == 1 || rsb != 1;
  auto op_of = [&](const void* x, int64_t rs, int64_t cs, int64_t bs, int rows, int cols, int64_t items) {
    PlaneOp o{};
    o.x = x; o.rs = rs; o.cs = cs; o.bs = bs; o.rows = rows; o.cols = cols;
    o.cols8 = (cols + 7) / 8;
    o.n8 = items * rows * o.cols8;
    o.plane = static_cast<int64_t>(rows) * o.cols8 * 8;
    const int64_t want = (o.n8 + 511) / 512, most = static_cast<int64_t>(sm_count()) * 8;
    o.blocks = static_cast<int>(want < most ? want : most);
    o.wide = DT == YTC_F32 && cs == 1 && rs % 4 == 0 && bs % 4 == 0 && (reinterpret_cast<uint64_t>(x) & 15) == 0;
    return o;
  };
  auto a_op = [&](int64_t b0, int64_t items, int k0, int kc) {
    const char* x = static_cast<const char*>(A) + (b0 * bsa + k0 * csa) * esz;
    return a_mn ? op_of(x, csa, rsa, bsa, kc, m, items) : op_of(x, rsa, csa, bsa, m, kc, items);
  };
  auto b_op = [&](int64_t b0, int64_t items, int k0, int kc) {
    const char* x = static_cast<const char*>(B) + (b0 * bsb + k0 * rsb) * esz;
    return b_kn ? op_of(x, rsb, csb, bsb, kc, n, items) : op_of(x, csb, rsb, bsb, n, kc, items);
  };
  TcPlanes pl{PLANES, PLANES, 1, 0, 0, 0, 0};
  if (PLANES == 3) {  // (l,h) (m,m) (h,l) (m,h) (h,m) (h,h)
    pl.pairs = 6;
    pl.pa = 2u | (1u << 2) | (0u << 4) | (1u << 6) | (0u << 8) | (0u << 10);
    pl.pb = 0u | (1u << 2) | (2u << 4) | (0u << 6) | (1u << 8) | (0u << 10);
  }
  // An accumulator of the tensor cores drops a fraction of a unit at every step of 16; FFMA rounds. Products that FFMA took
  // before (`check`) keep 256 of k per accumulator and add the pieces in fp32. Error against 64 bits (2-norm), 16 x 4096 x 4096:
  // FFMA 1.2e-6, here 2.5e-7; one accumulator would be above 3e-6. Their scratch stays below the size that a stream keeps (256 MB;
  // larger buffers come and go with every call, which took from 0.6 to 6 ms at 130 x 8192 x 8192), however long k is: k goes by in
  // windows of some pieces, each rewritten and multiplied by a launch of its own, whose partial sums stay and are added to. Only
  // C itself may need more (partial sums of a C that is larger, or whose rows do not start at 16 bytes).
  // The other products take whole k, and as many batch items per pass as keep the planes below 2 GiB.
  constexpr int PIECE = 256;
  constexpr int64_t PLANE_ROOM = int64_t{112} << 20, PART_ROOM = int64_t{128} << 20;
  const int64_t ldp = check ? (n + 3) / 4 * 4 : n, mn = m * ldp;  // (rows of partial sums that are added to start at 16 bytes)
  const int64_t a_item = a_op(0, 1, 0, check && k > PIECE ? PIECE : k).plane * PLANES * 2;
  const int64_t b_item = b_op(0, 1, 0, check && k > PIECE ? PIECE : k).plane * PLANES * 2;
  const int64_t fixed = (a_shared ? a_item : 0) + (b_shared ? b_item : 0);
  const int64_t per_item = (a_shared ? 0 : a_item) + (b_shared ? 0 : b_item);
  int64_t chunk = batch;
  auto at_most = [&](int64_t room, int64_t each) {
    if (each > 0 && each * chunk > room) chunk = room / each > 1 ? room / each : 1;
  };
  at_most((check ? PLANE_ROOM : int64_t{2} << 30) - fixed, per_item);
  if (check) at_most(PART_ROOM, mn * 4);
  int splits = DT == YTC_F32 && g_f32_split != 0 ? 1 : tc_splits(m, n, k, pl.pairs, chunk), window = k;
  if (check) {
    const int64_t pieces = (k + PIECE - 1) / PIECE, room = PART_ROOM / (chunk * mn * 4), wide = PLANE_ROOM / (fixed + chunk * per_item);
    int64_t side = g_tc_pair == 1 ? 1 : pieces;  // pieces side by side
    if (side > room) side = room;
    if (side > wide) side = wide;
    splits = side < 1 ? 1 : static_cast<int>(side);
    if (splits < pieces) window = splits * PIECE;
  }
  // C itself takes the sums where its rows start at 16 bytes. Elsewhere its elements would be stored one by one (777 x 1001 x 200: 34.9 us,
  // 22.7 through partial sums; 60 x 1001 x 180 29.8, 18.5), which is left to a C that is larger than the room for them, and to products without FFMA behind them.
  const bool rows16 = csc == 1 && rsc % 4 == 0 && (batch == 1 || bsc % 4 == 0) && (reinterpret_cast<uint64_t>(C) & 15) == 0;
  const bool direct = splits == 1 && (rows16 || (window == k && !(check && chunk * mn * 4 <= PART_ROOM)));
  auto up = [](int64_t v) { return static_cast<size_t>((v + 255) / 256 * 256); };
  // CTAs (and words of the gate) of either operand: those of the first, largest rewriting
  const PlaneOp largest_a = a_op(0, a_shared ? 1 : chunk, 0, window), largest_b = b_op(0, b_shared ? 1 : chunk, 0, window);
  const int n_gate = largest_a.blocks + largest_b.blocks;
  const size_t gate_bytes = up(n_gate * 4), a_bytes = up(largest_a.plane * PLANES * 2 * (a_shared ? 1 : chunk));
  const size_t b_bytes = up(largest_b.plane * PLANES * 2 * (b_shared ? 1 : chunk));
  const size_t part_bytes = direct ? 0 : up(static_cast<int64_t>(splits) * chunk * mn * 4);
  char* ws = static_cast<char*>(device_workspace(gate_bytes + a_bytes + b_bytes + part_bytes, st));
  if (!ws) return NO_SCRATCH;
  int* gate = check ? reinterpret_cast<int*>(ws) : nullptr;
  uint16_t* a_out = reinterpret_cast<uint16_t*>(ws + gate_bytes);
  uint16_t* b_out = reinterpret_cast<uint16_t*>(ws + gate_bytes + a_bytes);
  float* part = reinterpret_cast<float*>(ws + gate_bytes + a_bytes + b_bytes);
  const int tc_dt = DT == YTC_F32 ? YTC_BF16 : DT;
  for (int64_t b0 = 0; b0 < batch; b0 += chunk) {
    const int64_t nb = batch - b0 < chunk ? batch - b0 : chunk;
    char* c = static_cast<char*>(C) + b0 * bsc * dtype_size(dtype_out);
    int s;
    for (int k0 = 0; k0 < k; k0 += window) {
      const int kc = k - k0 < window ? k - k0 : window;
      PlaneOp oa = a_op(a_shared ? 0 : b0, a_shared ? 1 : nb, k0, kc), ob = b_op(b_shared ? 0 : b0, b_shared ? 1 : nb, k0, kc);
      oa.out = a_out;
      ob.out = b_out;
      oa.blocks = largest_a.blocks;
      ob.blocks = largest_b.blocks;
      const int64_t lda = oa.cols8 * 8, ldb = ob.cols8 * 8;
      pl.plane_a = oa.plane;
      pl.plane_b = ob.plane;
      // an operand that all batch items share is rewritten once, if it is rewritten whole
      const bool again = b0 > 0 && window == k, do_a = !(a_shared && again), do_b = !(b_shared && again);
      const PlaneOp none{};
      auto planes = [&](const PlaneOp& x, const PlaneOp& y, int word) {  // (no blocks: nothing to do for that operand)
        const cudaError_t e = launch_overlapped(gemm_planes_kernel<DT>, dim3(static_cast<unsigned>(x.blocks + y.blocks)), dim3(256), 0,
                                                st, x, y, gate ? gate + word : nullptr, k0 > 0 ? 1 : 0);
        count_launch();
        return e;
      };
      if (do_a && do_b && (check || !b_shared)) {
        YTC_CUDA(planes(oa, ob, 0));
      } else {
        if (do_b) YTC_CUDA(planes(none, ob, oa.blocks));
        if (do_a) YTC_CUDA(planes(oa, none, 0));
      }
      const int64_t bsa_p = a_shared ? 0 : oa.plane * PLANES, bsb_p = b_shared ? 0 : ob.plane * PLANES;
      s = direct ? launch_tc(tc_dt, dtype_out, a_out, b_out, c, m, n, kc, alpha, k0 > 0 ? 1.f : beta, a_mn, lda, b_kn, ldb, rsc, csc,
                             nb, bsa_p, bsb_p, bsc, st, nullptr, &pl)
                 : launch_tc(tc_dt, YTC_F32, a_out, b_out, part, m, n, kc, 1.f, k0 > 0 ? 1.f : 0.f, a_mn, lda, b_kn, ldb, ldp, 1, nb,
                             bsa_p, bsb_p, mn, st, nullptr, &pl, check ? (kc + PIECE - 1) / PIECE : splits);
      if (s != YTC_OK) return s;
    }
    if (!direct) {
      const int64_t total = nb * m * n, blocks = (total + 255) / 256, cap = static_cast<int64_t>(sm_count()) * 8;
      YTC_CUDA(launch_overlapped(gemm_sum_kernel, dim3(static_cast<unsigned>(blocks < cap ? blocks : cap)), dim3(256), 0, st, part,
                                 splits, nb * mn, total, m, n, ldp, c, dtype_out, rsc, csc, bsc, alpha, beta, gate));
      count_launch();
    }
    if (check && (s = launch_simt(DT, dtype_out, static_cast<const char*>(A) + b0 * bsa * esz, static_cast<const char*>(B) + b0 * bsb * esz,
                                  c, m, n, k, alpha, beta, rsa, csa, rsb, csb, rsc, csc, nb, bsa, bsb, bsc, st, gate, n_gate, direct)) !=
                     YTC_OK)
      return s;
  }
  device_workspace_release(st);  // large operands do not stay resident
  return YTC_OK;
}

// The product with k in pieces, operands as they lie.
static int launch_tc_split(int dtype_in, int dtype_out, const void* A, const void* B, void* C, int m, int n, int k, float alpha,
                           float beta, int a_mn, int64_t lda, int b_mn, int64_t ldb, int64_t rsc, int64_t csc, int64_t batch,
                           int64_t bsa, int64_t bsb, int64_t bsc, int splits, float* part, cudaStream_t st) {
  struct Scope {
    bool was = overlap_scope();
    Scope() { overlap_scope() = true; }
    ~Scope() { overlap_scope() = was; }
  } scope;
  const int64_t mn = static_cast<int64_t>(m) * n, total = batch * mn;
  const int s = launch_tc(dtype_in, YTC_F32, A, B, part, m, n, k, 1.f, 0.f, a_mn, lda, b_mn, ldb, n, 1, batch, bsa, bsb, mn, st,
                          nullptr, nullptr, splits);
  if (s != YTC_OK) return s;
  const int64_t blocks = (total + 255) / 256, cap = static_cast<int64_t>(sm_count()) * 8;
  YTC_CUDA(launch_overlapped(gemm_sum_kernel, dim3(static_cast<unsigned>(blocks < cap ? blocks : cap)), dim3(256), 0, st, part, splits,
                             total, total, m, n, n, C, dtype_out, rsc, csc, bsc, alpha, beta, static_cast<int*>(nullptr)));
  count_launch();
  return YTC_OK;
}

// Prompts of the Qwen3-shape decoder: the activation in the product's epilogue instead of a launch that reads both halves of an
// fp32 result and writes the planes (2000 x 6144: 18.8 us, 74 MB).
int swiglu_two_planes(const void* planes, const void* w, void* out, int m, int inter, int k, cudaStream_t st) {
  int unused;
  if (inter % 8 != 0 || !tc_takes_pairs(m, 2 * inter, 2ll * k, 1) || (reinterpret_cast<uint64_t>(out) & 15u) != 0 ||
      !tc_operand_ok(planes, k, 1, 0, 1, m, k, &unused) || !tc_operand_ok(w, k, 1, 0, 1, 2 * inter, k, &unused) ||
      static_cast<int64_t>(m) * inter * 2 >= (int64_t{1} << 40))
    return YTC_UNSUPPORTED;
  const TcPlanes pl{2, 1, 2, 1u, 0u, static_cast<int64_t>(m) * k, static_cast<int64_t>(2) * inter * k};
  LinearEpilogue ex;
  ex.epi = EPI_SWIGLU_PLANES;
  return launch_tc(YTC_BF16, YTC_BF16, planes, w, out, m, 2 * inter, k, 1.f, 0.f, 0, k, 0, k, inter, 1, 1, 0, 0, 0, st, &ex, &pl);
}

// y[m, n] (+)= (hi + lo)[m, k] . W[n, k]^T: both bf16 planes ([2][m][k]) of the activations in one accumulator, lo first; rows
// that do not start at 16 bytes (of a rank's share of the FFN width, say) as two products.
int linear_two_planes(const void* planes, const void* w, float* y, int64_t ldy, int m, int n, int k, bool accumulate, cudaStream_t st) {
  int unused;
  if (!tc_operand_ok(planes, k, 1, 0, 1, m, k, &unused) || !tc_operand_ok(w, k, 1, 0, 1, n, k, &unused)) {
    const char* lo = static_cast<const char*>(planes) + static_cast<int64_t>(m) * k * 2;
    const int s = ytcuda_gemm(YTC_BF16, YTC_F32, planes, w, y, m, n, k, 1.f, accumulate ? 1.f : 0.f, k, 1, 1, k, ldy, 1, 1, 0, 0, 0, st);
    return s != YTC_OK ? s : ytcuda_gemm(YTC_BF16, YTC_F32, lo, w, y, m, n, k, 1.f, 1.f, k, 1, 1, k, ldy, 1, 1, 0, 0, 0, st);
  }
  const TcPlanes pl{2, 1, 2, 1u, 0u, static_cast<int64_t>(m) * k, static_cast<int64_t>(n) * k};
  LinearEpilogue ex;
  ex.add_in_memory = true;
  return launch_tc(YTC_BF16, YTC_F32, planes, w, y, m, n, k, 1.f, accumulate ? 1.f : 0.f, 0, k, 0, k, ldy, 1, 1, 0, 0, 0, st, &ex, &pl);
}

}  // namespace ytk

using namespace ytk;

extern "C" {

int ytcuda_gemm_set_pair_mode(int mode) {
  YTC_REQUIRE(mode >= 0 && mode <= 2, "ytcuda_gemm_set_pair_mode: mode must be 0 (auto), 1 (always) or 2 (never)");
  g_tc_pair = mode;
  return YTC_OK;
}

int ytcuda_gemm_set_tuning(int a_prefetch_kblocks, int split_loads) {
  YTC_REQUIRE(a_prefetch_kblocks >= 0 && a_prefetch_kblocks <= 64, "ytcuda_gemm_set_tuning: prefetch distance outside [0, 64]");
  g_tc_a_prefetch = a_prefetch_kblocks;
  g_tc_split_loads = split_loads ? 1 : 0;
  return YTC_OK;
}

int ytcuda_gemm_set_f32_mode(int mode) {
  YTC_REQUIRE(mode >= 0 && mode <= 2, "ytcuda_gemm_set_f32_mode: mode must be 0, 1 or 2");
  g_f32_split = mode;
  return YTC_OK;
}

int ytcuda_gemm_set_path(int path) {
  YTC_REQUIRE(path >= 0 && path <= 2, "ytcuda_gemm_set_path: path must be 0, 1 or 2");
  g_gemm_path = path;
  return YTC_OK;
}

}  // extern "C"

namespace ytk {

// scratch: whether the call may use this stream's workspace (a caller that writes into the workspace itself says no)
static int gemm_any(int dtype_in, int dtype_out, const void* A, const void* B, void* C, int m, int n, int k, float alpha,
                    float beta, int64_t rsa, int64_t csa, int64_t rsb, int64_t csb, int64_t rsc, int64_t csc,
                    int64_t batch, int64_t bsa, int64_t bsb, int64_t bsc, bool scratch, void* stream) {
  YTC_REQUIRE(dtype_in >= YTC_F32 && dtype_in <= YTC_F16, "ytcuda_gemm: bad dtype_in %d", dtype_in);
  YTC_REQUIRE(dtype_out >= YTC_F32 && dtype_out <= YTC_F16, "ytcuda_gemm: bad dtype_out %d", dtype_out);
  YTC_REQUIRE(m >= 0 && n >= 0 && k >= 0 && batch >= 0, "ytcuda_gemm: negative extent (m=%d n=%d k=%d batch=%lld)", m,
              n, k, (long long)batch);
  if (m == 0 || n == 0 || batch == 0) return YTC_OK;
  YTC_REQUIRE(C != nullptr, "ytcuda_gemm: C is null");
  YTC_REQUIRE(k == 0 || (A != nullptr && B != nullptr), "ytcuda_gemm: A or B is null");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (k == 0) {
    if (beta == 1.f) return YTC_OK;
    for (int64_t b0 = 0; b0 < batch; b0 += 65535) {
      const int64_t nb = (batch - b0 < 65535) ? batch - b0 : 65535;
      dim3 grid(static_cast<unsigned>(sm_count() * 4), static_cast<unsigned>(nb));
      gemm_scale_c_kernel<<<grid, 256, 0, st>>>(static_cast<char*>(C) + b0 * bsc * dtype_size(dtype_out), m, n, rsc,
                                                csc, bsc, beta, dtype_out);
      count_launch();
    }
    YTC_CUDA(cudaGetLastError());
    return YTC_OK;
  }
  if (dtype_in == YTC_F32 && dtype_out == YTC_F32 && g_gemm_path != 1) {
    const int form = f32_planes_form(m, n, k, beta, rsc, csc, bsc, batch, bsb);
    if (form == 1 || (form == 2 && scratch && !stream_captures(st))) {
      const int s = launch_planes<YTC_F32>(A, B, C, dtype_out, m, n, k, alpha, beta, rsa, csa, rsb, csb, rsc, csc, batch, bsa, bsb,
                                           bsc, form == 2, st);
      if (s != NO_SCRATCH) return s;  // (FFMA needs none)
    }
  }
  int a_mn = 0, b_mn = 0;
  bool tc = (dtype_in != YTC_F32) && g_gemm_path != 1;
  if (tc) {
    // A[m,k]: unit stride along k (csa == 1) or along m (rsa == 1).
    tc = tc_operand_ok(A, rsa, csa, bsa, batch, m, k, &a_mn);
    // B[k,n]: unit stride along n (csb == 1) means N-major; along k (rsb == 1) means K-major.
    int b_k_unit = 0;
    if (tc) {
      tc = tc_operand_ok(B, csb, rsb, bsb, batch, n, k, &b_k_unit);  // view B as [n,k]
      b_mn = b_k_unit;  // viewed as [n,k]: "cs == 1" is rsb == 1 (K-major, 0); "rs == 1" is csb == 1 (N-major, 1)
    }
    if (tc && (rsc < 0 || csc < 0 || bsc < 0)) tc = false;
  }
  if (!tc && g_gemm_path == 2) {
    set_last_error("ytcuda_gemm: tcgen05 path required but the operands do not qualify");
    return YTC_UNSUPPORTED;
  }
  if (tc) {
    const int64_t lda = a_mn ? csa : rsa;
    const int64_t ldb = b_mn ? rsb : csb;
    // A single k extent of 1 makes both strides of an axis "unit"; the leading stride must still be sane.
    const int splits = scratch ? tc_splits(m, n, k, 1, batch) : 1;
    if (splits > 1 && !stream_captures(st)) {
      const WorkspaceScope workspace(st);
      float* part = static_cast<float*>(device_workspace(static_cast<size_t>(splits) * batch * m * n * 4, st));
      if (part) {
        const int s = launch_tc_split(dtype_in, dtype_out, A, B, C, m, n, k, alpha, beta, a_mn, lda, b_mn, ldb, rsc, csc, batch,
                                      bsa, bsb, bsc, splits, part, st);
        device_workspace_release(st);
        return s;
      }
    }
    return launch_tc(dtype_in, dtype_out, A, B, C, m, n, k, alpha, beta, a_mn, lda, b_mn, ldb, rsc, csc, batch, bsa,
                     bsb, bsc, st);
  }
  // 16-bit operands that the TMA cannot take (odd sizes and strides): rewritten where that pays
  if (dtype_in != YTC_F32 && g_gemm_path != 1 && scratch && g_mask.kind == 0 && rsc >= 0 && csc >= 0 && bsc >= 0 &&
      dtype_out != YTC_F32 &&  // (an fp32 result would show the tensor cores' accumulation)
      simt_us(m, n, k, batch, false) > 1.5 * planes_us(m, n, k, batch, bsb == 0, false) && !stream_captures(st)) {
    const int s = dtype_in == YTC_BF16
                      ? launch_planes<YTC_BF16>(A, B, C, dtype_out, m, n, k, alpha, beta, rsa, csa, rsb, csb, rsc, csc, batch, bsa, bsb, bsc, false, st)
                      : launch_planes<YTC_F16>(A, B, C, dtype_out, m, n, k, alpha, beta, rsa, csa, rsb, csb, rsc, csc, batch, bsa, bsb, bsc, false, st);
    if (s != NO_SCRATCH) return s;
  }
  return launch_simt(dtype_in, dtype_out, A, B, C, m, n, k, alpha, beta, rsa, csa, rsb, csb, rsc, csc, batch, bsa,
                     bsb, bsc, st);
}

// ytcuda_gemm for callers whose C lies in this stream's workspace.
int gemm_into_workspace(int dtype_in, int dtype_out, const void* A, const void* B, void* C, int m, int n, int k, float alpha,
                        float beta, int64_t rsa, int64_t csa, int64_t rsb, int64_t csb, int64_t rsc, int64_t csc, int64_t batch,
                        int64_t bsa, int64_t bsb, int64_t bsc, cudaStream_t st) {
  return gemm_any(dtype_in, dtype_out, A, B, C, m, n, k, alpha, beta, rsa, csa, rsb, csb, rsc, csc, batch, bsa, bsb, bsc, false, st);
}

}  // namespace ytk

extern "C" {

int ytcuda_gemm(int dtype_in, int dtype_out, const void* A, const void* B, void* C, int m, int n, int k, float alpha,
                float beta, int64_t rsa, int64_t csa, int64_t rsb, int64_t csb, int64_t rsc, int64_t csc,
                int64_t batch, int64_t bsa, int64_t bsb, int64_t bsc, void* stream) {
  return gemm_any(dtype_in, dtype_out, A, B, C, m, n, k, alpha, beta, rsa, csa, rsb, csb, rsc, csc, batch, bsa, bsb, bsc, true, stream);
}

}  // extern "C"

// ------------------------------------------------------------------ host-buffer variant
namespace ytk {

struct HostGemmCtx {
  cudaStream_t s_in = nullptr, s_run = nullptr, s_out = nullptr;
  static constexpr int NBUF = 3;
  cudaEvent_t in_done[NBUF] = {}, run_done[NBUF] = {}, out_done[NBUF] = {}, b_done = nullptr;
  void* a_buf[NBUF] = {};
  void* c_buf[NBUF] = {};
  void* b_buf = nullptr;
  size_t b_cap = 0;
  bool ready = false;
};

static HostGemmCtx* host_ctx() {
  static HostGemmCtx ctx[16];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return nullptr;
  HostGemmCtx& c = ctx[dev];
  if (!c.ready) {
    if (cudaStreamCreateWithFlags(&c.s_in, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
    if (cudaStreamCreateWithFlags(&c.s_run, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
    if (cudaStreamCreateWithFlags(&c.s_out, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
    for (int i = 0; i < HostGemmCtx::NBUF; ++i) {
      if (cudaEventCreateWithFlags(&c.in_done[i], cudaEventDisableTiming) != cudaSuccess) return nullptr;
      if (cudaEventCreateWithFlags(&c.run_done[i], cudaEventDisableTiming) != cudaSuccess) return nullptr;
      if (cudaEventCreateWithFlags(&c.out_done[i], cudaEventDisableTiming) != cudaSuccess) return nullptr;
    }
    if (cudaEventCreateWithFlags(&c.b_done, cudaEventDisableTiming) != cudaSuccess) return nullptr;
    c.ready = true;
  }
  return &c;
}

static int grow(void** buf, size_t* cap, size_t need) {
  if (*cap >= need) return YTC_OK;
  if (*buf) YTC_CUDA(cudaFree(*buf));
  *buf = nullptr;
  *cap = 0;
  YTC_CUDA(cudaMalloc(buf, need));
  *cap = need;
  return YTC_OK;
}

// Elements spanned by an r x c view with non-negative strides.
static int64_t span_of(int64_t r, int64_t c, int64_t rs, int64_t cs) { return (r - 1) * rs + (c - 1) * cs + 1; }

}  // namespace ytk

// The product skips the output tiles the mask leaves nothing in (the launchers read g_mask), then one pass writes
// masked_value wherever the mask does not hold (dead tiles included).
static int gemm_masked_impl(int kind, int dtype_in, int dtype_out, const void* A, const void* B, void* C, int m, int n,
                            int k, int64_t rsa, int64_t csa, int64_t rsb, int64_t csb, int64_t rsc, int64_t csc,
                            int64_t batch, int64_t bsa, int64_t bsb, int64_t bsc, const void* mask,
                            int64_t mask_row_stride, int offset, float masked_value, void* stream) {
  ytk::g_mask.kind = kind;
  ytk::g_mask.mask = static_cast<const uint8_t*>(mask);
  ytk::g_mask.row_stride = mask_row_stride;
  ytk::g_mask.offset = offset;
  const int s = ytcuda_gemm(dtype_in, dtype_out, A, B, C, m, n, k, 1.0f, 0.0f, rsa, csa, rsb, csb, rsc, csc, batch, bsa,
                            bsb, bsc, stream);
  ytk::g_mask = ytk::MaskCtx{};
  if (s != YTC_OK) return s;
  const int64_t total = static_cast<int64_t>(m) * n * batch;
  const int64_t blocks = (total + 255) / 256;
  const int64_t cap = static_cast<int64_t>(sm_count()) * 16;
  gemm_apply_mask_kernel<<<static_cast<unsigned>(blocks < cap ? blocks : cap), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      C, dtype_out, m, n, rsc, csc, batch, bsc, static_cast<const uint8_t*>(mask), mask_row_stride, masked_value,
      kind == 2 ? 1 : 0, offset);
  count_launch();
  YTC_CUDA(cudaGetLastError());
  return YTC_OK;
}

int ytcuda_gemm_masked_causal(int dtype_in, int dtype_out, const void* A, const void* B, void* C, int m, int n, int k,
                              int64_t rsa, int64_t csa, int64_t rsb, int64_t csb, int64_t rsc, int64_t csc,
                              int64_t batch, int64_t bsa, int64_t bsb, int64_t bsc, int causal_offset,
                              float masked_value, void* stream) {
  YTC_REQUIRE(m >= 0 && n >= 0 && k >= 0 && batch >= 0, "ytcuda_gemm_masked_causal: negative extent");
  if (m == 0 || n == 0 || batch == 0) return YTC_OK;
  return gemm_masked_impl(2, dtype_in, dtype_out, A, B, C, m, n, k, rsa, csa, rsb, csb, rsc, csc, batch, bsa, bsb, bsc,
                          nullptr, 0, causal_offset, masked_value, stream);
}

int ytcuda_gemm_masked(int dtype_in, int dtype_out, const void* A, const void* B, void* C, int m, int n, int k,
                       int64_t rsa, int64_t csa, int64_t rsb, int64_t csb, int64_t rsc, int64_t csc, int64_t batch,
                       int64_t bsa, int64_t bsb, int64_t bsc, const void* mask, int64_t mask_row_stride,
                       float masked_value, void* stream) {
  YTC_REQUIRE(m >= 0 && n >= 0 && k >= 0 && batch >= 0, "ytcuda_gemm_masked: negative extent");
  if (m == 0 || n == 0 || batch == 0) return YTC_OK;
  YTC_REQUIRE(mask != nullptr, "ytcuda_gemm_masked: mask is null");
  YTC_REQUIRE(mask_row_stride >= n, "ytcuda_gemm_masked: mask row stride %lld shorter than n = %d",
              (long long)mask_row_stride, n);
  return gemm_masked_impl(1, dtype_in, dtype_out, A, B, C, m, n, k, rsa, csa, rsb, csb, rsc, csc, batch, bsa, bsb, bsc,
                          mask, mask_row_stride, 0, masked_value, stream);
}


extern "C" int ytcuda_gemm_host(int dtype_in, int dtype_out, const void* A, const void* B, void* C, int m, int n, int k,
                                float alpha, float beta, int64_t rsa, int64_t csa, int64_t rsb, int64_t csb,
                                int64_t rsc, int64_t csc, int64_t batch, int64_t bsa, int64_t bsb, int64_t bsc) {
  YTC_REQUIRE(dtype_in >= YTC_F32 && dtype_in <= YTC_F16, "ytcuda_gemm_host: bad dtype_in %d", dtype_in);
  YTC_REQUIRE(dtype_out >= YTC_F32 && dtype_out <= YTC_F16, "ytcuda_gemm_host: bad dtype_out %d", dtype_out);
  YTC_REQUIRE(m >= 0 && n >= 0 && k >= 0 && batch >= 0, "ytcuda_gemm_host: negative extent");
  if (m == 0 || n == 0 || batch == 0) return YTC_OK;
  YTC_REQUIRE(A && B && C, "ytcuda_gemm_host: null operand");
  YTC_REQUIRE(k > 0, "ytcuda_gemm_host: k must be positive");
  YTC_REQUIRE(rsa >= 0 && csa >= 0 && rsb >= 0 && csb >= 0 && bsa >= 0 && bsb >= 0,
              "ytcuda_gemm_host: negative input strides are not supported");
  const bool c_rows = (csc == 1 && rsc >= n), c_cols = (rsc == 1 && csc >= m);
  if (!(c_rows || c_cols) || bsc < 0) {
    set_last_error("ytcuda_gemm_host: C must have a unit stride along one axis and no overlap");
    return YTC_UNSUPPORTED;
  }
  HostGemmCtx* cx = host_ctx();
  if (!cx) {
    set_last_error("ytcuda_gemm_host: cannot create streams");
    return YTC_CUDA_ERROR;
  }
  const int64_t ein = dtype_size(dtype_in), eout = dtype_size(dtype_out);
  const int64_t a_span = span_of(m, k, rsa, csa), b_span = span_of(k, n, rsb, csb), c_span = span_of(m, n, rsc, csc);
  const bool b_shared = (batch == 1 || bsb == 0);
  const bool a_shared = (batch > 1 && bsa == 0);
  // Batch items per chunk: about 64 MiB of A + C traffic per chunk, at least one item.
  const int64_t per_item = a_span * ein + c_span * eout;
  int64_t g = (64ll << 20) / (per_item > 0 ? per_item : 1);
  if (g < 1) g = 1;
  if (g > batch) g = batch;
  const int64_t a_chunk = a_shared ? a_span : ((g - 1) * bsa + a_span);
  const int64_t c_chunk = (g - 1) * bsc + c_span;
  const int64_t b_all = b_shared ? b_span : ((batch - 1) * bsb + b_span);
  static size_t a_caps[16][HostGemmCtx::NBUF], c_caps[16][HostGemmCtx::NBUF];
  int dev = 0;
  YTC_CUDA(cudaGetDevice(&dev));
  for (int i = 0; i < HostGemmCtx::NBUF; ++i) {
    int s = grow(&cx->a_buf[i], &a_caps[dev][i], static_cast<size_t>(a_chunk * ein));
    if (s != YTC_OK) return s;
    s = grow(&cx->c_buf[i], &c_caps[dev][i], static_cast<size_t>(c_chunk * eout));
    if (s != YTC_OK) return s;
  }
  {
    int s = grow(&cx->b_buf, &cx->b_cap, static_cast<size_t>(b_all * ein));
    if (s != YTC_OK) return s;
  }
  YTC_CUDA(cudaMemcpyAsync(cx->b_buf, B, static_cast<size_t>(b_all * ein), cudaMemcpyHostToDevice, cx->s_in));
  YTC_CUDA(cudaEventRecord(cx->b_done, cx->s_in));
  YTC_CUDA(cudaStreamWaitEvent(cx->s_run, cx->b_done, 0));
  if (a_shared) {
    YTC_CUDA(cudaMemcpyAsync(cx->a_buf[0], A, static_cast<size_t>(a_span * ein), cudaMemcpyHostToDevice, cx->s_in));
    YTC_CUDA(cudaEventRecord(cx->b_done, cx->s_in));
    YTC_CUDA(cudaStreamWaitEvent(cx->s_run, cx->b_done, 0));
  }
  const bool c_dense = (c_span == static_cast<int64_t>(m) * n) && (batch == 1 || bsc == c_span);
  int64_t chunk_idx = 0;
  for (int64_t b0 = 0; b0 < batch; b0 += g, ++chunk_idx) {
    const int64_t nb = (batch - b0 < g) ? batch - b0 : g;
    const int buf = static_cast<int>(chunk_idx % HostGemmCtx::NBUF);
    const char* a_src = static_cast<const char*>(A) + b0 * bsa * ein;
    char* c_host = static_cast<char*>(C) + b0 * bsc * eout;
    void* a_dev = a_shared ? cx->a_buf[0] : cx->a_buf[buf];
    if (chunk_idx >= HostGemmCtx::NBUF) YTC_CUDA(cudaStreamWaitEvent(cx->s_in, cx->out_done[buf], 0));
    if (!a_shared)
      YTC_CUDA(cudaMemcpyAsync(a_dev, a_src, static_cast<size_t>(((nb - 1) * bsa + a_span) * ein),
                               cudaMemcpyHostToDevice, cx->s_in));
    if (beta != 0.f)
      YTC_CUDA(cudaMemcpyAsync(cx->c_buf[buf], c_host, static_cast<size_t>(((nb - 1) * bsc + c_span) * eout),
                               cudaMemcpyHostToDevice, cx->s_in));
    YTC_CUDA(cudaEventRecord(cx->in_done[buf], cx->s_in));
    YTC_CUDA(cudaStreamWaitEvent(cx->s_run, cx->in_done[buf], 0));
    const char* b_dev = static_cast<const char*>(cx->b_buf) + (b_shared ? 0 : b0 * bsb * ein);
    int s = ytcuda_gemm(dtype_in, dtype_out, a_dev, b_dev, cx->c_buf[buf], m, n, k, alpha, beta, rsa, csa, rsb, csb,
                        rsc, csc, nb, a_shared ? 0 : bsa, b_shared ? 0 : bsb, bsc, cx->s_run);
    if (s != YTC_OK) {
      cudaDeviceSynchronize();
      return s;
    }
    YTC_CUDA(cudaEventRecord(cx->run_done[buf], cx->s_run));
    YTC_CUDA(cudaStreamWaitEvent(cx->s_out, cx->run_done[buf], 0));
    if (c_dense) {
      YTC_CUDA(cudaMemcpyAsync(c_host, cx->c_buf[buf], static_cast<size_t>(nb * c_span * eout),
                               cudaMemcpyDeviceToHost, cx->s_out));
    } else {
      for (int64_t i = 0; i < nb; ++i) {
        const size_t off = static_cast<size_t>(i * bsc * eout);
        const size_t pitch = static_cast<size_t>((c_rows ? rsc : csc) * eout);
        const size_t width = static_cast<size_t>((c_rows ? n : m) * eout);
        const size_t height = static_cast<size_t>(c_rows ? m : n);
        YTC_CUDA(cudaMemcpy2DAsync(c_host + off, pitch, static_cast<char*>(cx->c_buf[buf]) + off, pitch, width, height,
                                   cudaMemcpyDeviceToHost, cx->s_out));
      }
    }
    YTC_CUDA(cudaEventRecord(cx->out_done[buf], cx->s_out));
  }
  YTC_CUDA(cudaStreamSynchronize(cx->s_out));
  YTC_CUDA(cudaStreamSynchronize(cx->s_run));
  YTC_CUDA(cudaStreamSynchronize(cx->s_in));
  return read_device_status(cx->s_run) == 0 ? YTC_OK : YTC_TIMEOUT;
}
