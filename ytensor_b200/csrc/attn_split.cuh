// Attention with fp32 products on the tensor cores: every operand is cut into bf16 planes that sum to it exactly (fp32:
// three planes of 8 mantissa bits, fp16: two, bf16: itself) and the plane products above 2^-24 of the result are added up
// in fp32, smallest first. P stays fp32 too: three truncated planes, also exact.
//
//  * attn_planes_kernel: K and V (any type, any strides of whole groups of four) -> planes
//    [plane][batch * kv head][key][64 or 128] in scratch memory, and a word per block that says whether it met a number
//    that has no planes (infinity, NaN, 2^127 and above).
//  * attn_split_kernel: 128 query rows x 128 keys per step, one persistent CTA per SM. The planes of Q sit in shared memory;
//    K and V come plane by plane, 32 KB each, by TMA through a ring of four, in the order in which the MMAs take them. Two
//    softmax warpgroups take the key tiles in turn, each with a running maximum, sum and O of its own in registers, so that
//    the chain S -> maximum -> P of one tile runs under the MMAs of the other; P V of a tile starts from zero in tensor
//    memory and is added to the registers in fp32 (a sum over thousands of keys inside the accumulator would collect a
//    truncation per step). At the end the warpgroups merge through tensor memory.
//
// What bounds it: the tensor pipe and the shared memory that feeds it (Q K^T reads 8 KB per MMA of 64 clocks, the copies add a
// quarter): 6 products of 128 x 128 x 128 for S and for P V, 96 MMAs a tile. Measured on a B200, causal, fp32, 16 query and 8
// key heads of 128, planes and check included, FFMA kernel / here: 1000 queries and keys 256 / 64 us, 2000: 761 / 146 (68 and 158
// while one lane of the service warps issued copies, MMAs and commits inside a branch); bf16,
// 8 heads of 80, 1024: 1345 / 58. (Q in tensor memory and tiles of 64 keys: 78, 185 and 59 us; an MMA of 64 columns takes as
// long there as one of 128.) Error against 64 bits (2-norm) at 1000 keys: 3.9e-7 / 2.1e-7.
#pragma once

namespace ytk {

constexpr int SA_BM = 128, SA_BN = 128, SA_THREADS = 384;  // a service warpgroup, two softmax warpgroups
constexpr int SA_BLOCK = SA_BN * 128;               // bytes of 128 rows x 64 columns of one plane
constexpr int SA_PLANE = 2 * SA_BLOCK;
constexpr int SA_SLOTS = 4;
constexpr int SA_Q_OFF = 0, SA_RING_OFF = 3 * SA_PLANE;
constexpr int SA_BAR_OFF = SA_RING_OFF + SA_SLOTS * SA_PLANE;
constexpr int SA_NBAR = 2 * SA_SLOTS + 6 + 4;
constexpr int SA_DYN_BYTES = SA_BAR_OFF + SA_NBAR * 8 + 32 + 1024;
// tensor-memory columns: two S / P buffers of 192 (S 128, three planes of P 64 each), one O
constexpr uint32_t SA_T_SP = 192, SA_T_O = 384;

struct SplitAttnParams {
  AttnSimtParams a;
  int planes;       // of Q, K and V
  int rows_unit;    // query rows of a unit: q_len of one head, or all groups * q_len of a K/V head
  int row_tiles;    // tiles of 128 rows per unit
  int n_units, n_items;
  int flat;         // a unit is a K/V head
  int o_vec;        // O is stored four values at a time
  uint32_t idesc_s, idesc_s_half, idesc_pv;  // (half: a last tile of at most 64 keys)
  float scale_log2;
  int* unfit;       // [CTAs] set where Q holds a number without planes
  int* status;
};

struct PlanesParams {
  const void* src[2];       // K, V
  int64_t sb[2], sh[2], sr[2];
  uint16_t* dst[2];
  int width[2], cols[2];    // columns of a row, and of its planes (a multiple of 64; the rest is zero)
  int64_t n4[2];            // groups of four columns
  int64_t plane[2];         // elements of a plane
  int kv_heads, len, dt, planes;
  int* unfit;               // [blocks]
};

// Infinities, NaN and 2^127 and above; and where a number takes more than one plane, those under 2^-110 (the last plane would
// lie below bf16's smallest number) but zero.
__device__ __forceinline__ bool has_no_planes(float x, int planes) {
  const uint32_t e = __float_as_uint(x) & 0x7FFFFFFFu;
  return e >= 0x7F000000u || (planes > 1 && e != 0u && e < 0x08800000u);
}

__device__ __forceinline__ void split_planes(float x, uint16_t (&pl)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    pl[i] = *reinterpret_cast<const uint16_t*>(&h);
    x -= __bfloat162float(h);
  }
}

// Bound by memory: 4 bytes read and 6 written per fp32 value.
__global__ void __launch_bounds__(256) attn_planes_kernel(const PlanesParams p) {
  dependent_wait();
  dependent_trigger();
  bool unfit = false;
  const int64_t total = p.n4[0] + p.n4[1];
  for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const int s = i >= p.n4[0];
    const uint32_t e = static_cast<uint32_t>(s ? i - p.n4[0] : i);  // (n4 is below 2^31)
    const uint32_t per_row = static_cast<uint32_t>(p.cols[s]) >> 2;
    const uint32_t rw = e / per_row, c = (e - rw * per_row) * 4;
    const uint32_t bh = rw / static_cast<uint32_t>(p.len), r = rw - bh * p.len;
    const uint32_t b = bh / static_cast<uint32_t>(p.kv_heads), h = bh - b * p.kv_heads;
    float x[4] = {0.f, 0.f, 0.f, 0.f};
    if (static_cast<int>(c) < p.width[s]) {
      const int64_t o = b * p.sb[s] + h * p.sh[s] + r * p.sr[s] + c;
      if (p.dt == YTC_F32) {
        const float4 v = *reinterpret_cast<const float4*>(static_cast<const float*>(p.src[s]) + o);
        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
      } else {
        const uint2 v = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(p.src[s]) + o);
        const uint16_t q[4] = {static_cast<uint16_t>(v.x), static_cast<uint16_t>(v.x >> 16), static_cast<uint16_t>(v.y),
                               static_cast<uint16_t>(v.y >> 16)};
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = p.dt == YTC_BF16 ? bf16_bits_to_f32(q[k]) : f16_bits_to_f32_ref(q[k]);
      }
    }
    uint16_t pl[4][3];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      unfit |= has_no_planes(x[k], p.planes);
      split_planes(x[k], pl[k]);
    }
    uint16_t* d = p.dst[s] + static_cast<int64_t>(e) * 4;
#pragma unroll
    for (int i3 = 0; i3 < 3; ++i3)
      if (i3 < p.planes)
        *reinterpret_cast<uint2*>(d + i3 * p.plane[s]) =
            make_uint2(pl[0][i3] | (static_cast<uint32_t>(pl[1][i3]) << 16), pl[2][i3] | (static_cast<uint32_t>(pl[3][i3]) << 16));
  }
  const int any = __syncthreads_or(unfit);
  if (threadIdx.x == 0) p.unfit[blockIdx.x] = any;
}

struct SplitItem {
  int r0, unit, n;  // first query row within the unit, unit, key tiles
  bool half;        // no row sees more than 64 keys of the last tile
};
__device__ __forceinline__ SplitItem split_item(const SplitAttnParams& p, int w) {
  SplitItem it;
  it.unit = w % p.n_units;
  it.r0 = (p.row_tiles - 1 - w / p.n_units) * SA_BM;  // the longest causal rows first
  int last = p.a.kv_len - 1;
  if (p.a.causal) {
    const int r1 = min(it.r0 + SA_BM, p.rows_unit) - 1;
    const int q0 = it.r0 / p.a.q_len, q1 = r1 / p.a.q_len;
    last = min(last, (q0 == q1 ? r1 - q1 * p.a.q_len : p.a.q_len - 1) + p.a.causal_off);
  }
  it.n = last < 0 ? 0 : last / SA_BN + 1;
  it.half = last % SA_BN < 64;
  return it;
}

__global__ void __launch_bounds__(SA_THREADS, 1)
    attn_split_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const SplitAttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SA_BAR_OFF);
  uint64_t *full = bars, *empty = bars + SA_SLOTS, *s_full = empty + SA_SLOTS, *p_full = s_full + 2, *o_full = p_full + 2;
  uint64_t *o_free = o_full + 2, *q_ready = o_free + 1, *merge_in = o_free + 2, *merge_out = o_free + 3;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + SA_NBAR);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* unfit_word = reinterpret_cast<int*>(tmem_slot + 2);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // (known to be the same for the warp)
  const int bkv = p.a.batch * p.a.kv_heads;

  if (threadIdx.x == 0) {
    for (int s = 0; s < SA_SLOTS; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&o_full[s], 1);
      mbar_init(&p_full[s], 4);  // one arrival per warp of a warpgroup
    }
    mbar_init(o_free, 4);
    mbar_init(q_ready, 8);
    mbar_init(merge_in, 8);
    mbar_init(merge_out, 8);
    *abort_word = 0;
    *unfit_word = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = 0;  // (all 512 columns are this CTA's)
  dependent_wait();
  dependent_trigger();

  // `g` counts the key tiles of all items so far: S / P buffer and warpgroup g & 1, phase (g >> 1) & 1. `n_pl` counts the
  // planes of K and V, loaded and multiplied in one order: K of tiles 0 and 1, then V of tile j and K of tile j + 2; of a tile
  // the last plane first. Items without a visible key touch no barrier.
  if (warp < 4) {
    // (168 registers a thread at launch, 72 + 2 * 216 afterwards, the same sum: the softmax keeps 128 columns of O)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 0) {
      // ------------------------------------------------------------ TMA producer
      // (converged like the issuer: inside a branch of one lane the twelve copies of a tile took as long as its MMAs)
      const uint32_t lead = lane == 0 ? 1u : 0u;
      const uint32_t ring_at = smem_u32(smem + SA_RING_OFF), full_at = smem_u32(full);
      const int kblocks = (p.a.d + 63) / 64, vblocks = (p.a.dv + 63) / 64;
      int n_pl = 0;
      auto load = [&](const CUtensorMap* tm, int blocks, int tile, int bh) {
#pragma unroll 1
        for (int i = p.planes - 1; i >= 0; --i, ++n_pl) {
          const int s = n_pl % SA_SLOTS;
          if (!mbar_wait_warp(&empty[s], ((n_pl / SA_SLOTS) & 1) ^ 1, abort_word)) return false;
          mbar_expect_tx_lead(full_at + 8 * s, static_cast<uint32_t>(blocks * SA_BLOCK), lead);
#pragma unroll 1
          for (int c = 0; c < blocks; ++c)
            tma_load_3d_lead(ring_at + s * SA_PLANE + c * SA_BLOCK, tm, full_at + 8 * s, c * 64, tile * SA_BN, i * bkv + bh, lead);
        }
        return true;
      };
      bool ok = true;
      for (int w = blockIdx.x; ok && w < p.n_items; w += gridDim.x) {
        const SplitItem it = split_item(p, w);
        const int bh = p.flat ? it.unit : it.unit / p.a.groups;
        for (int j = 0; ok && j < 2 && j < it.n; ++j) ok = load(&tmK, kblocks, j, bh);
        for (int j = 0; ok && j < it.n; ++j) {
          ok = load(&tmV, vblocks, j, bh);
          if (ok && j + 2 < it.n) ok = load(&tmK, kblocks, j + 2, bh);
        }
      }
      // a give-up elsewhere: bounded drain of the last copies
      const long long t0 = clock64();
      for (int k = n_pl - SA_SLOTS > 0 ? n_pl - SA_SLOTS : 0; k < n_pl; ++k)
        while (!mbar_try_wait(&full[k % SA_SLOTS], (k / SA_SLOTS) & 1) && clock64() - t0 < 20000000ll) {
        }
      __syncwarp();
    } else if (warp == 1) {
      // ------------------------------------------------------------ MMA issuer
      // The whole warp runs this code and lane 0 issues: straight code, constant offsets, operands in uniform registers
      // (a loop that forms descriptors in a one-lane branch costs 190 clocks per MMA, the tensor pipe needs 64).
      const uint32_t lead = lane == 0 ? 1u : 0u;
      const uint64_t qd = umma_smem_desc_sw128(smem_u32(smem + SA_Q_OFF), 16, 1024);
      const uint64_t kd = umma_smem_desc_sw128(smem_u32(smem + SA_RING_OFF), 16, 1024);
      const uint64_t vd = umma_smem_desc_sw128(smem_u32(smem + SA_RING_OFF), SA_BLOCK, 1024);
      constexpr uint32_t PLANE = SA_PLANE / 16, BLOCK = SA_BLOCK / 16;  // (descriptors count 16 bytes)
      const int ksteps = (p.a.d + 15) / 16;
      // (every lane waits: a give-up is agreed on before the next step)
      auto wait = [&](uint64_t* bar, uint32_t ph) { return mbar_wait_warp(bar, ph, abort_word); };
      auto commit = [&](uint64_t* bar) { tc_commit_lead(smem_u32(bar), lead); };
      int n_pl = 0;
      // The products of plane J of K (or V) with planes I of Q (or P), I + J <= 2, the smallest first
      auto k_plane = [&](auto plane, uint32_t ds, uint32_t idesc) {
        constexpr int J = decltype(plane)::value;
        if (J >= p.planes) return true;
        const int s = n_pl % SA_SLOTS;
        if (!wait(&full[s], (n_pl / SA_SLOTS) & 1)) return false;
        tc_fence_after();
        const uint64_t kb = kd + s * PLANE;
        auto steps = [&](int k0, int k1, int i, bool add) {
#pragma unroll
          for (int k = k0; k < k1; ++k)
            tc_mma_f16_lead(ds, qd + (i * PLANE + (k >> 2) * BLOCK + (k & 3) * 2), kb + ((k >> 2) * BLOCK + (k & 3) * 2), idesc,
                            add || k > 0, lead);
        };
#pragma unroll
        for (int i = 2 - J; i >= 0; --i) {
          if (i >= p.planes) continue;
          const bool add = !(J == p.planes - 1 && i == (2 - J < p.planes - 1 ? 2 - J : p.planes - 1));
          steps(0, 4, i, add);  // (zeros behind column d, to 64, 96 or 128)
          if (ksteps > 4) steps(4, 6, i, true);
          if (ksteps > 6) steps(6, 8, i, true);
        }
        commit(&empty[s]);
        ++n_pl;
        return true;
      };
      auto v_plane = [&](auto plane, uint32_t as, bool half) {  // P: see the softmax for where its planes lie
        constexpr int J = decltype(plane)::value;
        if (J >= p.planes) return true;
        const int s = n_pl % SA_SLOTS;
        if (!wait(&full[s], (n_pl / SA_SLOTS) & 1)) return false;
        tc_fence_after();
        const uint64_t vb = vd + s * PLANE;
        auto steps = [&](int k0, int k1, int i, bool add) {
#pragma unroll
          for (int k = k0; k < k1; ++k)
            tc_mma_f16_ts_lead(SA_T_O, as + (i == 0 ? 128 + k * 8 : (k >> 1) * 32 + (i - 1) * 16 + (k & 1) * 8), vb + k * 128,
                               p.idesc_pv, add || k > 0, lead);
        };
#pragma unroll
        for (int i = 2 - J; i >= 0; --i) {
          steps(0, 4, i, !(J == p.planes - 1 && i == 2 - J));
          if (!half) steps(4, 8, i, true);
        }
        commit(&empty[s]);
        ++n_pl;
        return true;
      };
      using P0 = std::integral_constant<int, 0>;
      using P1 = std::integral_constant<int, 1>;
      using P2 = std::integral_constant<int, 2>;
      auto issue_s = [&](int b, bool half) {
        const uint32_t ds = b * SA_T_SP, idesc = half ? p.idesc_s_half : p.idesc_s;
        if (!k_plane(P2{}, ds, idesc) || !k_plane(P1{}, ds, idesc) || !k_plane(P0{}, ds, idesc)) return false;
        commit(&s_full[b]);
        return true;
      };
      auto issue_pv = [&](int b, bool half) {
        const uint32_t as = b * SA_T_SP;
        if (!v_plane(P2{}, as, half) || !v_plane(P1{}, as, half) || !v_plane(P0{}, as, half)) return false;
        commit(&o_full[b]);
        return true;
      };
      int g = 0, n_item = 0;
      bool ok = true;
      for (int w = blockIdx.x; ok && w < p.n_items; w += gridDim.x) {
        const SplitItem it = split_item(p, w);
        if (it.n == 0) continue;
        if (!wait(q_ready, n_item & 1)) break;
        tc_fence_after();
        for (int j = 0; ok && j < 2 && j < it.n; ++j) ok = issue_s((g + j) & 1, it.half && j == it.n - 1);
        for (int j = 0; ok && j < it.n; ++j, ++g) {
          const int b = g & 1;
          ok = wait(&p_full[b], (g >> 1) & 1) && (g == 0 || wait(o_free, (g - 1) & 1));
          if (!ok) break;
          tc_fence_after();
          ok = issue_pv(b, it.half && j == it.n - 1);
          // (S of tile j + 2 runs behind the P V that reads this buffer: MMAs of one thread keep their order)
          if (ok && j + 2 < it.n) ok = issue_s(b, it.half && j + 2 == it.n - 1);
        }
        ++n_item;
      }
    }
  } else {
    // ------------------------------------------------------------ softmax warpgroups
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    const int wg = (warp - 4) >> 2, quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t tl = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t ts = tl + wg * SA_T_SP, to = tl + SA_T_O;
    const bool general = p.a.mask != nullptr || p.a.bias != nullptr;
    // Scores are kept in log2 units, under a bias in its own: the lowest float, the usual mask, would become -infinity, and a
    // row that holds nothing else would weigh none of its keys instead of all alike. `unit`: one score in log2 units.
    const bool biased = p.a.bias != nullptr;
    const float unit = biased ? FA_LOG2E : 1.f;
    const int esz = p.a.dt == YTC_F32 ? 4 : 2;
    int g = 0, n_item = 0;
    bool ok = true, unfit = false;
    for (int w = blockIdx.x; ok && w < p.n_items; w += gridDim.x) {
      const SplitItem it = split_item(p, w);
      const int ru = it.r0 + row;
      const bool valid = ru < p.rows_unit;
      const int grp = p.flat ? ru / p.a.q_len : 0;
      const int qi = ru - grp * p.a.q_len;
      const int heads = p.a.kv_heads * p.a.groups;
      const int b = p.flat ? it.unit / p.a.kv_heads : it.unit / heads;
      const int h = p.flat ? (it.unit - b * p.a.kv_heads) * p.a.groups + grp : it.unit - b * heads;
      const int limit = !valid ? -1 : p.a.causal ? min(p.a.kv_len - 1, qi + p.a.causal_off) : p.a.kv_len - 1;
      char* orow = static_cast<char*>(p.a.O) + (b * p.a.o_sb + h * p.a.o_sh + qi * p.a.o_sr) * esz;
      auto store4 = [&](int c, float x0, float x1, float x2, float x3) {  // columns c .. c + 3 (dv is a multiple of 4)
        if (p.o_vec && p.a.dt == YTC_F32) {
          *reinterpret_cast<float4*>(orow + c * 4) = make_float4(x0, x1, x2, x3);
        } else if (p.o_vec) {
          const float x[4] = {x0, x1, x2, x3};
          uint32_t u[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) u[k] = p.a.dt == YTC_BF16 ? f32_to_bf16_bits_ref(x[k]) : f32_to_f16_bits_ref(x[k]);
          *reinterpret_cast<uint2*>(orow + c * 2) = make_uint2(u[0] | (u[1] << 16), u[2] | (u[3] << 16));
        } else {
          store_from_f32(orow, c, x0, p.a.dt);
          store_from_f32(orow, c + 1, x1, p.a.dt);
          store_from_f32(orow, c + 2, x2, p.a.dt);
          store_from_f32(orow, c + 3, x3, p.a.dt);
        }
      };
      if (it.n == 0) {
        if (valid)
          for (int c = wg * 64; c < min(p.a.dv, wg * 64 + 64); c += 4) store4(c, 0.f, 0.f, 0.f, 0.f);
        continue;
      }
      {  // columns 64 wg .. 64 wg + 63 of this thread's query row, three planes, swizzled as the TMA would
        if (n_item > 0 && !mbar_wait(merge_out, (n_item - 1) & 1, abort_word)) break;
        const char* qrow = static_cast<const char*>(p.a.Q) + (b * p.a.q_sb + h * p.a.q_sh + qi * p.a.q_sr) * esz;
        uint8_t* qs = smem + SA_Q_OFF + wg * SA_BLOCK + row * 128;
#pragma unroll 1
        for (int c0 = wg * 64; c0 < (wg == 0 ? 64 : p.a.d); c0 += 8) {  // (zeros behind the last column)
          float x[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = 0.f;
#pragma unroll
          for (int c = 0; c < 8; c += 4)
            if (valid && c0 + c < p.a.d) {
              if (p.a.dt == YTC_F32) {
                const float4 v = *reinterpret_cast<const float4*>(qrow + (c0 + c) * 4);
                x[c] = v.x; x[c + 1] = v.y; x[c + 2] = v.z; x[c + 3] = v.w;
              } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) x[c + k] = load_as_f32(qrow, c0 + c + k, p.a.dt);
              }
            }
          uint16_t pl[8][3];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            unfit |= has_no_planes(x[e], p.planes);
            split_planes(x[e], pl[e]);
          }
          uint8_t* dst = qs + ((((c0 & 63) >> 3) ^ (row & 7)) << 4);
#pragma unroll
          for (int i = 0; i < 3; ++i)
            if (i < p.planes) {
              uint32_t u[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) u[e] = pl[2 * e][i] | (static_cast<uint32_t>(pl[2 * e + 1][i]) << 16);
              *reinterpret_cast<uint4*>(dst + i * SA_PLANE) = make_uint4(u[0], u[1], u[2], u[3]);
            }
        }
        // columns of the 16-column steps that the products of a d above 64 take with the last ones
        if (wg == 1 && p.a.d > 64)
          for (int c0 = (p.a.d + 7) / 8 * 8; c0 < (p.a.d + 31) / 32 * 32; c0 += 8)
            for (int i = 0; i < p.planes; ++i)
              *reinterpret_cast<uint4*>(qs + i * SA_PLANE + ((((c0 & 63) >> 3) ^ (row & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(q_ready);
      }
      float m_run = -CUDART_INF_F, l_run = 0.f;
      float acc[128];
#pragma unroll
      for (int c = 0; c < 128; ++c) acc[c] = 0.f;
      for (int j = (wg + g) & 1; j < it.n; j += 2) {
        const int gg = g + j;
        ok = mbar_wait(&s_full[wg], (gg >> 1) & 1, abort_word);
        if (!ok) break;
        tc_fence_after();
        const int key0 = j * SA_BN, cl = limit - key0;  // columns 0 .. cl are visible to this row
        const int cols = it.half && j == it.n - 1 ? 64 : SA_BN;
        const bool full = !general && __all_sync(0xffffffffu, cl >= cols - 1);
        // Pass 1: the maximum. Tiles with hidden keys, a mask or a bias get their scores (-inf where hidden)
        // written back over S, so that pass 2 is one piece of code: the instructions a softmax warp cycles through stay few.
        float mx = -CUDART_INF_F;
#pragma unroll 1
        for (int c0 = 0; c0 < cols; c0 += 32) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(ts + c0, r);
          tmem_ld_wait();
          if (full) {
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
              float t0, t1;
              f2_unpack(f2_mul(f2_pack(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), f2_pack(p.scale_log2, p.scale_log2)), t0, t1);
              mx = fmax3(mx, t0, t1);
            }
            continue;
          }
          if (!general) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              r[e] = __float_as_uint(c0 + e <= cl ? __uint_as_float(r[e]) * p.scale_log2 : -CUDART_INF_F);
          } else {
            masked_scores(r, p.a.mask ? p.a.mask + qi * p.a.mask_rs + key0 + c0 : nullptr,
                          p.a.bias ? p.a.bias + qi * p.a.bias_rs + (key0 + c0) * p.a.bias_cs : nullptr, p.a.bias_cs, cl - c0 + 1,
                          biased ? p.a.scale : p.scale_log2, 1.f);
          }
#pragma unroll
          for (int e = 0; e < 32; e += 2) mx = fmax3(mx, __uint_as_float(r[e]), __uint_as_float(r[e + 1]));
          tmem_st_32x32b_x32(ts + c0, r);
        }
        if (!full) tmem_st_wait();
        const float m_new = fmaxf(m_run, mx);
        const float m_use = m_new == -CUDART_INF_F ? 0.f : m_new;
        const float alpha = m_run == -CUDART_INF_F ? 0.f : fast_exp2((m_run - m_use) * unit);
        m_run = m_new;
        // Pass 2: P of 32 keys at a time, the second and third plane over the 32 columns of S that have been read, the first
        // plane behind S.
        const float sl = full ? p.scale_log2 : 1.f, sub = biased ? 0.f : -m_use;
        uint64_t ps = f2_pack(0.f, 0.f);
#pragma unroll 1
        for (int c0 = 0; c0 < cols; c0 += 32) {
          uint32_t r[32], pk[16];
          tmem_ld_32x32b_x32(ts + c0, r);
          tmem_ld_wait();
          if (biased) {  // (the difference first: score and maximum may both be the lowest float)
#pragma unroll
            for (int e = 0; e < 32; ++e) r[e] = __float_as_uint((__uint_as_float(r[e]) - m_use) * FA_LOG2E);
          }
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            float t0, t1;
            f2_unpack(f2_fma(f2_pack(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), f2_pack(sl, sl), f2_pack(sub, sub)), t0, t1);
            t0 = fast_exp2(t0);
            t1 = fast_exp2(t1);
            ps = f2_add(ps, f2_pack(t0, t1));
            r[e] = __float_as_uint(t0);
            r[e + 1] = __float_as_uint(t1);
          }
#pragma unroll
          for (int i = 0; i < 3; ++i) {
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
              pk[e >> 1] = __byte_perm(r[e], r[e + 1], 0x7632);  // the upper halves: a plane by truncation
              if (i < 2) {
                r[e] = __float_as_uint(__uint_as_float(r[e]) - __uint_as_float(r[e] & 0xFFFF0000u));
                r[e + 1] = __float_as_uint(__uint_as_float(r[e + 1]) - __uint_as_float(r[e + 1] & 0xFFFF0000u));
              }
            }
            tmem_st_32x32b_x16(ts + (i == 0 ? 128 + c0 / 2 : c0 + (i - 1) * 16), pk);
          }
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[wg]);
        float ps0, ps1;
        f2_unpack(ps, ps0, ps1);
        l_run = l_run * alpha + (ps0 + ps1);
        ok = mbar_wait(&o_full[wg], (gg >> 1) & 1, abort_word);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int c0 = 0; c0 < 128; c0 += 32) {
          if (c0 < p.a.dv) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(to + c0, r);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) acc[c0 + e] = fmaf(acc[c0 + e], alpha, __uint_as_float(r[e]));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(o_free);
      }
      if (!ok) break;
      g += it.n;
      // Merge: each warpgroup hands the other 64 columns of its O, its maximum and its sum over in its own S / P buffer, whose
      // last P V it has waited for.
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        uint32_t r[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(wg == 0 ? acc[64 + c + e] : acc[c + e]);
        tmem_st_32x32b_x32(ts + c, r);
      }
      uint32_t ml[16];
#pragma unroll
      for (int e = 2; e < 16; ++e) ml[e] = 0u;
      ml[0] = __float_as_uint(m_run);
      ml[1] = __float_as_uint(l_run);
      tmem_st_32x32b_x16(ts + 64, ml);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(merge_in);
      if (!mbar_wait(merge_in, n_item & 1, abort_word)) break;
      tc_fence_after();
      const uint32_t tx = tl + (1 - wg) * SA_T_SP;
      tmem_ld_32x32b_x16(tx + 64, ml);
      tmem_ld_wait();
      const float m_o = __uint_as_float(ml[0]), l_o = __uint_as_float(ml[1]);
      const float m = fmaxf(m_run, m_o);
      const float f = m_run == -CUDART_INF_F ? 0.f : fast_exp2((m_run - m) * unit), f_o = m_o == -CUDART_INF_F ? 0.f : fast_exp2((m_o - m) * unit);
      const float l = l_run * f + l_o * f_o;
      const float inv = l > 0.f ? 1.0f / l : 0.f;
      // A score or a sum that overflows has plane products of either sign that overflow: NaN where FFMA has an infinity, of which
      // a negative one weighs nothing. Rows that are not finite, or weigh no key though they see some, are left to FFMA.
      if (valid && !general && limit >= 0) unfit |= !(l > 0.f);
      float zero = 0.f;
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(tx + c, r);
        tmem_ld_wait();
        float x[32];
#pragma unroll
        for (int e = 0; e < 32; ++e)
          x[e] = ((wg == 0 ? acc[c + e] : acc[64 + c + e]) * f + __uint_as_float(r[e]) * f_o) * inv;
        if (valid) {
#pragma unroll
          for (int e = 0; e < 32; e += 4)
            if (wg * 64 + c + e < p.a.dv) {
              store4(wg * 64 + c + e, x[e], x[e + 1], x[e + 2], x[e + 3]);
              zero = fmaf(x[e], 0.f, fmaf(x[e + 1], 0.f, fmaf(x[e + 2], 0.f, fmaf(x[e + 3], 0.f, zero))));
            }
        }
      }
      unfit |= !(zero == 0.f);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(merge_out);
      ++n_item;
    }
    if (unfit) *unfit_word = 1;
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(*tmem_slot, 512);
  }
  if (threadIdx.x == 0) {
    p.unfit[blockIdx.x] = *unfit_word;
    if (*abort_word) atomicExch(p.status, YTC_TIMEOUT);
  }
}

constexpr int64_t SA_SCRATCH = int64_t{240} << 20;
static int64_t split_attention_bytes(const AttnSimtParams& a) {  // (of the planes)
  const int planes = a.dt == YTC_F32 ? 3 : a.dt == YTC_F16 ? 2 : 1;
  return static_cast<int64_t>(a.batch) * a.kv_heads * a.kv_len * ((a.d + 63) / 64 + (a.dv + 63) / 64) * 64 * 2 * planes;
}

// Queues the planes and the attention; false: nothing was queued (a size, alignment or capture the path does not take, no
// scratch). On true the caller queues the fp32 kernel behind it with `gate`, which runs only where a number had no planes.
static bool split_attention(const AttnSimtParams& a, const int** gate, int* n_gate, cudaStream_t st) {
  const int esz = dtype_size(a.dt), heads = a.kv_heads * a.groups;
  auto quads = [&](const void* ptr, int64_t s0, int64_t s1, int64_t s2) {
    return (reinterpret_cast<uint64_t>(ptr) % (4 * esz)) == 0 && s0 % 4 == 0 && s1 % 4 == 0 && s2 % 4 == 0;
  };
  if (a.d > 128 || a.dv > 128 || a.d <= 0 || a.d % 4 || a.dv % 4 || a.kv_len <= 0 || !quads(a.Q, a.q_sb, a.q_sh, a.q_sr) ||
      !quads(a.K, a.k_sb, a.k_sh, a.k_sr) || !quads(a.V, a.v_sb, a.v_sh, a.v_sr))
    return false;
  const int64_t bkv = static_cast<int64_t>(a.batch) * a.kv_heads;
  const int kcols = (a.d + 63) / 64 * 64, vcols = (a.dv + 63) / 64 * 64;
  if (bkv * a.kv_len * 128 > 0x7fffffffll || bkv > 0x7fffff || static_cast<int64_t>(a.groups) * a.q_len > 0x3fffffff) return false;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;  // (scratch that grows inside a capture would belong to the graph)
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return false;

  SplitAttnParams p;
  p.a = a;
  p.planes = a.dt == YTC_F32 ? 3 : a.dt == YTC_F16 ? 2 : 1;
  // few queries per head: the heads of a group share tiles of 128 rows
  p.flat = a.q_len % SA_BM != 0 && a.groups > 1 &&
           (static_cast<int64_t>(a.groups) * a.q_len + SA_BM - 1) / SA_BM < static_cast<int64_t>(a.groups) * ((a.q_len + SA_BM - 1) / SA_BM);
  p.rows_unit = p.flat ? a.groups * a.q_len : a.q_len;
  p.row_tiles = (p.rows_unit + SA_BM - 1) / SA_BM;
  const int64_t units = p.flat ? bkv : static_cast<int64_t>(a.batch) * heads;
  if (units * p.row_tiles > 0x3fffffff) return false;
  p.n_units = static_cast<int>(units);
  p.n_items = static_cast<int>(units * p.row_tiles);
  p.o_vec = (reinterpret_cast<uint64_t>(a.O) % (4 * esz)) == 0 && a.o_sb % 4 == 0 && a.o_sh % 4 == 0 && a.o_sr % 4 == 0;
  p.idesc_s = umma_idesc(1u, 0, 0, SA_BM, SA_BN);
  p.idesc_s_half = umma_idesc(1u, 0, 0, SA_BM, 64);
  p.idesc_pv = umma_idesc(1u, 0, 1, SA_BM, static_cast<uint32_t>((a.dv + 15) / 16 * 16));
  p.scale_log2 = a.scale * FA_LOG2E;
  p.status = device_status_word();
  if (!p.status) return false;

  PlanesParams q;
  q.src[0] = a.K; q.src[1] = a.V;
  q.sb[0] = a.k_sb; q.sh[0] = a.k_sh; q.sr[0] = a.k_sr;
  q.sb[1] = a.v_sb; q.sh[1] = a.v_sh; q.sr[1] = a.v_sr;
  q.width[0] = a.d; q.width[1] = a.dv;
  q.cols[0] = kcols; q.cols[1] = vcols;
  q.kv_heads = a.kv_heads; q.len = a.kv_len; q.dt = a.dt; q.planes = p.planes;
  for (int s = 0; s < 2; ++s) {
    q.plane[s] = bkv * a.kv_len * q.cols[s];
    q.n4[s] = q.plane[s] / 4;
  }
  const int64_t want = (q.n4[0] + q.n4[1] + 511) / 512, most = static_cast<int64_t>(sm_count()) * 8;
  const int blocks = static_cast<int>(want < most ? want : most);
  const int ctas = p.n_items < sm_count() ? p.n_items : sm_count();
  const size_t gate_bytes = (static_cast<size_t>(blocks + ctas) * 4 + 255) / 256 * 256;
  const size_t k_bytes = (static_cast<size_t>(q.plane[0]) * 2 * p.planes + 255) / 256 * 256;
  const size_t v_bytes = static_cast<size_t>(q.plane[1]) * 2 * p.planes;
  char* ws = static_cast<char*>(device_workspace(gate_bytes + k_bytes + v_bytes, st));
  if (!ws) return false;
  q.unfit = reinterpret_cast<int*>(ws);
  p.unfit = q.unfit + blocks;
  q.dst[0] = reinterpret_cast<uint16_t*>(ws + gate_bytes);
  q.dst[1] = reinterpret_cast<uint16_t*>(ws + gate_bytes + k_bytes);
  CUtensorMap tm[2];
  for (int s = 0; s < 2; ++s) {
    const uint64_t dims[3] = {static_cast<uint64_t>(q.cols[s]), static_cast<uint64_t>(a.kv_len), static_cast<uint64_t>(bkv * p.planes)};
    const uint64_t strides[2] = {dims[0] * 2, dims[0] * 2 * dims[1]};
    const uint32_t box[3] = {64, SA_BN, 1};
    if (encode_tensor_map(&tm[s], CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, q.dst[s], dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B) != YTC_OK)
      return false;
  }
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(attn_split_kernel), SA_DYN_BYTES) != YTC_OK) return false;
  if (launch_overlapped(attn_planes_kernel, dim3(blocks), dim3(256), 0, st, q) != cudaSuccess ||
      launch_overlapped(attn_split_kernel, dim3(ctas), dim3(SA_THREADS), SA_DYN_BYTES, st, tm[0], tm[1], p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  count_launch(2);
  *gate = q.unfit;
  *n_gate = blocks + ctas;
  return true;
}

}  // namespace ytk
