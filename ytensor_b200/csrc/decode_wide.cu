// One decode step (one new token per sequence, up to 32 sequences) of the Qwen3-shape decoder as one persistent kernel
// (operator sequence: reference example/qwen3/src/qwen3.cpp:237-283, 365-457).
//
// What bounds it: hand-overs. A step of 32 sequences reads 0.88 GB of layer weights and the K/V rows (0.15 ms at the copy rate);
// as ten dependent launches per layer it took 1.9 ms (32 sequences, 70 keys), here it takes 0.92 ms, 33 us a layer: five phases,
// each of them about 1.4 us of stores becoming visible and of polling, 0.8 us until the activations are in shared memory,
// 0.8-2 us of MMAs (61 cycles each, however narrow), 1.4 us until the partial sums are added and stored. 128 CTAs stay resident.
// They form 32 clusters of 4 (more than 120 CTAs do not fit in clusters of 8). In every projection a cluster owns a range of
// output rows and CTA r of it the r-th quarter of k, so that a CTA needs only a quarter of the activations, and the four partial
// sums meet inside the cluster:
//   * weights are the 128-row operand of tcgen05.mma, read once by TMA into a ring that one warp keeps filled ahead of the
//     phases (they depend on nothing); old K / V rows go through the same ring in chunks of 32 keys;
//   * activations are the narrow operand: hi and lo bf16 planes (16 mantissa bits) of up to 32 sequences side by side, so
//     that one MMA of N = 64 does both planes. Whoever finishes an activation writes it to global memory as the planes lie in
//     shared memory, so that one bulk copy brings a quarter of k in (a CTA that split them itself took twice as long);
//   * every output row's partial sums are pushed with st.async into the CTA that finishes that row (a quarter of the
//     cluster's rows each), which adds the four in rank order: results do not depend on timing;
//   * the norm in front of a projection is applied behind it: the weight goes into the published activations, the factor
//     1 / rms, which needs the whole row, onto the finished sums. The residual stream stays in the registers of its owners.
// Phases are separated by arrival words, one line each (four lines for all of them took 4 us a phase): every CTA stores its phase
// number, and a warp polls the 128 words at once. Every wait is bounded: on give-up the device status word is raised and the
// CTAs leave together (a CTA whose shared memory peers may still write must not be gone).
// The code is kept short on purpose (loops rolled, no variants, copies and MMAs issued by converged warps whose operands stay in
// uniform registers): an SM fetches about 32 KB of instructions at full speed, and with 122 KB of them a layer took 115 k cycles
// instead of 64 k.
#include <math_constants.h>

#include <vector>

#include "decode_wide.cuh"
#include "ptx_sm100.cuh"

namespace ytk {

constexpr int WD_CTAS = 128;
constexpr int WD_CLUSTER = 4;
constexpr int WD_NC = WD_CTAS / WD_CLUSTER;
constexpr int WD_WARPS = 16;  // that stage, finish and attend; two more issue copies and MMAs
constexpr int WD_COMPUTE = WD_WARPS * 32;
constexpr int WD_THREADS = WD_COMPUTE + 96;
constexpr int WD_FLAG = 32;  // words from one arrival word to the next: a line each
constexpr int WD_PIECE_KB = 4, WD_MAX_PIECES = 8;  // activations arrive in pieces of 4 k blocks
constexpr int WD_SLOT = 32768;  // one ring slot: two blocks of 128 weight rows x 64 columns, or 32 keys and their values
constexpr int WD_MAX_SLOTS = 6;
constexpr int WD_VALUES = WD_SLOT / 2;  // the values' place in a slot
constexpr int WD_KEYS = 32;
constexpr int WD_D = 128;

struct WdLinear {
  int ks;       // columns of a CTA's quarter of k
  int kb;       // ... in blocks of 64
  int nt;       // tiles of the cluster's rows
  int rows;     // rows of a tile (gate_up: gate rows of a tile; as many up rows follow at up_off)
  int up_off;   // byte offset of the up rows in a block, 0: none
  int block;    // bytes from one k block to the next within a slot
  int kbps;     // k blocks per slot
  int out;      // rows that each CTA finishes (gate_up: pairs)
};

struct WdParams {
  WdShape s;
  WdStep t;
  const WdLayer* lw;
  const CUtensorMap* maps;  // [layers][4]
  unsigned int* flags;      // [WD_CTAS] phase numbers, a line each
  unsigned int* abort_at;   // epoch of the launch that gave up
  float* ss;                // [WD_CTAS][WD_MAX_B] sums of squares of the owned columns
  uint8_t *x_planes, *attn_planes, *act_planes;  // [k / 64][hi, lo][MB] rows of 128 swizzled bytes
  WdLinear lin[4];
  unsigned int epoch;
  int nslot, planes_bytes, recv_bytes;
  uint32_t wait_limit;  // units of 1024 cycles
  int* status;
};

__device__ __forceinline__ void wd_bar(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
// true for all when all pass true
__device__ __forceinline__ bool wd_bar_and(int id, int threads, bool v) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.s32 p, %3, 0;\n\t"
      "barrier.cta.red.and.pred q, %1, %2, p;\n\t"
      "selp.s32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(id), "r"(threads), "r"(v ? 1 : 0)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void wd_push4(uint32_t dst, uint32_t bar, float a, float b, float c, float d) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(__float_as_uint(d)), "r"(bar)
               : "memory");
}
// Issued by one lane (`lead`) of a warp that runs converged: their operands then stay in uniform registers, where these
// instructions want them; inside a branch of one lane each of them costs some hundred instructions.
__device__ __forceinline__ void wd_expect(uint32_t bar, uint32_t bytes, uint32_t lead) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar),
               "r"(bytes), "r"(lead)
               : "memory");
}
__device__ __forceinline__ void wd_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t}" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar), "r"(lead)
      : "memory");
}
__device__ __forceinline__ void wd_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
      "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar), "r"(lead)
      : "memory");
}
__device__ __forceinline__ void wd_commit(uint32_t bar, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar),
      "r"(lead)
      : "memory");
}
// x * sigmoid(x): one exponential of a number <= 0, as the two-sided stable form takes
__device__ __forceinline__ float wd_swish(float v) {
  const float z = expf(-fabsf(v));
  const float s = 1.0f / (1.0f + z);
  return v * (v >= 0.f ? s : z * s);
}
__device__ __forceinline__ float wd_inv_rms(float squares, float inv_n, float eps) { return 1.0f / sqrtf(squares * inv_n + eps); }
// an activation -> its place in both planes, as the bulk copies bring them in
template <int MB>
__device__ __forceinline__ void wd_put(uint8_t* dst, int b, int col, float v) {
  const __nv_bfloat16 h = __float2bfloat16_rn(v);
  const __nv_bfloat16 lo = __float2bfloat16_rn(v - __bfloat162float(h));
  const unsigned at = (col >> 6) * (2 * MB * 128) + b * 128 + (((col & 63) * 2) ^ ((b & 7) << 4));
  __stcg(reinterpret_cast<unsigned short*>(dst + at), __bfloat16_as_ushort(h));
  __stcg(reinterpret_cast<unsigned short*>(dst + at + MB * 128), __bfloat16_as_ushort(lo));  // (MB % 8 == 0: swizzled alike)
}
// A wait of at most `limit` units of 1024 cycles. Short code (32-bit addresses and times): see the head of the file.
__device__ __forceinline__ uint32_t wd_time() { return static_cast<uint32_t>(clock64() >> 10); }
__device__ __forceinline__ bool wd_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool wd_wait(uint64_t* barrier, uint32_t parity, volatile int* abort_word, uint32_t limit) {
  const uint32_t bar = smem_u32(barrier);
  if (wd_try(bar, parity)) return true;
  const uint32_t t0 = wd_time();
#pragma unroll 1
  do {
    if (wd_try(bar, parity)) return true;
  } while (!*abort_word && wd_time() - t0 <= limit);
  *abort_word = 1;
  return false;
}
// ... for a whole converged warp
__device__ __forceinline__ bool wd_wait_warp(uint64_t* barrier, uint32_t parity, volatile int* abort_word, uint32_t limit) {
  return __all_sync(0xffffffffu, wd_wait(barrier, parity, abort_word, limit)) != 0;
}
// a load that stays where it is written: ahead of a wait
__device__ __forceinline__ float wd_load_early(const float* p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

struct WdShared {
  uint64_t full[WD_MAX_SLOTS], free_mma[WD_MAX_SLOTS], free_att[WD_MAX_SLOTS];
  uint64_t seen, staged[WD_MAX_PIECES], recv, drain, done[8];
  uint32_t tmem;
  int abort_word;
  float inv[WD_MAX_B];
  float ssp[WD_WARPS][WD_MAX_B];
  float ssr[WD_COMPUTE];
};

// MB: sequences rounded up (columns of a plane)
template <int MB>
__global__ void __launch_bounds__(WD_THREADS, 1) decode_wide_kernel(const __grid_constant__ WdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr int N = 2 * MB;
  constexpr int PLANE_BLOCK = N * 128;  // 64 columns of both planes
  constexpr int RS = MB + 4;            // floats per row of a partial sum: rows 16 bytes apart in the banks
  uint8_t* ring = smem;
  uint8_t* planes = smem + p.nslot * WD_SLOT;
  float* recv = reinterpret_cast<float*>(planes + p.planes_bytes);
  WdShared& sh = *reinterpret_cast<WdShared*>(planes + p.planes_bytes + p.recv_bytes);
  volatile int* abort_word = &sh.abort_word;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (known to be the same for the whole warp, as are r and c)
  const int r = static_cast<int>(blockIdx.x) % WD_CLUSTER, c = static_cast<int>(blockIdx.x) / WD_CLUSTER;
  const int B = p.s.B, hidden = p.s.hidden, kvh_n = p.s.kv_heads, heads = p.s.heads;
  const int qkv_w = (heads + 2 * kvh_n) * WD_D, G = heads / kvh_n;

  if (tid == 0) {
    for (int i = 0; i < p.nslot; ++i) {
      mbar_init(&sh.full[i], 1);
      mbar_init(&sh.free_mma[i], 1);
      mbar_init(&sh.free_att[i], 8);
    }
    mbar_init(&sh.seen, 1);
    for (int i = 0; i < WD_MAX_PIECES; ++i) mbar_init(&sh.staged[i], 1);
    mbar_init(&sh.recv, 1);
    mbar_init(&sh.drain, 1);
    for (int i = 0; i < 8; ++i) mbar_init(&sh.done[i], 1);
    sh.abort_word = 0;
    fence_mbar_init();
  }
  if (warp == WD_WARPS + 1) {
    tmem_alloc(&sh.tmem, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  cluster_sync_all();
  const uint32_t tmem = sh.tmem;

  // the attention units (sequence, key head) of this CTA: neighbours share a key head
  const int units = B * kvh_n, upc = (units + WD_CTAS - 1) / WD_CTAS;
  const int u0 = (r * WD_NC + c) * upc;
  const int nu = units - u0 < upc ? (units - u0 > 0 ? units - u0 : 0) : upc;
  const bool shared_unit = upc == 1;  // one unit for all 16 warps, else one for each group of 8
  const int n_old = p.t.pos, nch = (n_old + WD_KEYS - 1) / WD_KEYS;
  const int kv_slots = nch * nu;
  const size_t cache_layer = static_cast<size_t>(B) * kvh_n * p.s.max_pos * WD_D;

  if (warp == WD_WARPS) {
    // ------------------------------------------------ weights, keys and values
    const uint32_t lead = lane == 0 ? 1u : 0u;
    const uint32_t ring_at = smem_u32(ring), full_at = smem_u32(sh.full);
    uint32_t used = 0, by_att = 0, par_mma = 0, par_att = 0;
    uint32_t issued_par = 0;  // parity of the fill in flight of every slot
    int slot = 0;
    bool ok = true;
    auto acquire = [&](bool att) {  // the slot is free for a use of the given kind
      const uint32_t bit = 1u << slot;
      if (used & bit) {
        const bool by = by_att & bit;
        ok = wd_wait_warp(by ? &sh.free_att[slot] : &sh.free_mma[slot], ((by ? par_att : par_mma) >> slot) & 1u, abort_word, p.wait_limit);
        if (by) par_att ^= bit;
        else par_mma ^= bit;
      }
      used |= bit;
      by_att = att ? by_att | bit : by_att & ~bit;
      return ok;
    };
    auto filled = [&]() {
      issued_par ^= 1u << slot;
      slot = slot + 1 == p.nslot ? 0 : slot + 1;
    };
#pragma unroll 1
    for (int l = 0; l < p.s.layers && ok; ++l) {
      const CUtensorMap* maps = p.maps + 4 * l;
#pragma unroll 1
      for (int q = 0; q < 4 && ok; ++q) {
        if (l + 1 < p.s.layers) tma_prefetch_desc(maps + 4 + q);
        const WdLinear& L = p.lin[q];
        int n0 = c * L.nt * L.rows;
#pragma unroll 1
        for (int t = 0; t < L.nt && ok; ++t, n0 += L.rows) {
#pragma unroll 1
          for (int kb0 = 0; kb0 < L.kb; kb0 += L.kbps) {
            if (!acquire(false)) break;
            const int nkb = L.kb - kb0 < L.kbps ? L.kb - kb0 : L.kbps;
            const uint32_t bar = full_at + 8 * slot;
            wd_expect(bar, nkb * L.rows * 128 * (L.up_off ? 2 : 1), lead);
            uint32_t dst = ring_at + slot * WD_SLOT;
            int k = r * L.ks + kb0 * 64;
#pragma unroll 1
            for (int i = 0; i < nkb; ++i, k += 64, dst += L.block) {
              wd_tile(dst, maps + q, bar, k, n0, lead);
              if (L.up_off) wd_tile(dst + L.up_off, maps + q, bar, k, p.s.inter + n0, lead);
            }
            filled();
          }
        }
        if (q) continue;
#pragma unroll 1
        for (int j = 0; j < nu && ok; j += 2)
#pragma unroll 1
          for (int ch = 0; ch < nch && ok; ++ch)
#pragma unroll 1
            for (int e = j; e < j + 2 && e < nu; ++e) {
              if (!acquire(true)) break;
              const int u = u0 + e, kvh = u / B, b = u - kvh * B;
              const size_t at = l * cache_layer + ((static_cast<size_t>(b) * kvh_n + kvh) * p.s.max_pos + ch * WD_KEYS) * WD_D;
              const int bytes = (n_old - ch * WD_KEYS < WD_KEYS ? n_old - ch * WD_KEYS : WD_KEYS) * WD_D * 4;
              const uint32_t bar = full_at + 8 * slot, dst = ring_at + slot * WD_SLOT;
              wd_expect(bar, 2 * bytes, lead);
              wd_copy(dst, p.t.k_cache + at, bytes, bar, lead);
              wd_copy(dst + WD_VALUES, p.t.v_cache + at, bytes, bar, lead);
              filled();
            }
      }
    }
    if (!ok) {  // copies in flight land before this memory goes away
      const uint32_t t0 = wd_time();
#pragma unroll 1
      for (int i = 0; i < p.nslot; ++i)
        if (used & (1u << i))
          while (!wd_try(full_at + 8 * i, ((issued_par >> i) & 1u) ^ 1u) && wd_time() - t0 < 8000u) {
          }
    }
    __syncwarp();
  } else if (warp == WD_WARPS + 1) {
    // ------------------------------------------------ MMAs (the warp stays converged, one lane issues)
    constexpr uint32_t idesc = umma_idesc(1u, 0, 0, 128, N);
    const uint32_t lead = lane == 0 ? 1u : 0u;
    int slot = 0;
    uint32_t fill = 0;  // parity of the next fill
    uint32_t piece_par = 0;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) { return wd_wait_warp(bar, parity, abort_word, p.wait_limit); };
    const uint32_t free_at = smem_u32(sh.free_mma), done_at = smem_u32(sh.done);
    const uint64_t w_desc = umma_smem_desc_sw128(smem_u32(ring), 16, 1024), x_desc = umma_smem_desc_sw128(smem_u32(planes), 16, 1024);
#pragma unroll 1
    for (int l = 0; l < p.s.layers && ok; ++l)
#pragma unroll 1
      for (int q = 0; q < 4 && ok; ++q) {
        const WdLinear& L = p.lin[q];
        int pieces_in = 0;  // pieces of the activations that have arrived
#pragma unroll 1
        for (int t = 0; t < L.nt && ok; ++t) {
#pragma unroll 1
          for (int kb0 = 0; kb0 < L.kb && ok; kb0 += L.kbps) {
            const int nkb = L.kb - kb0 < L.kbps ? L.kb - kb0 : L.kbps;
            ok = wait(&sh.full[slot], fill);
            while (ok && pieces_in * WD_PIECE_KB < kb0 + nkb) {
              ok = wait(&sh.staged[pieces_in], (piece_par >> pieces_in) & 1u);
              piece_par ^= 1u << pieces_in;
              ++pieces_in;
            }
            if (!ok) break;
            tc_fence_after();
            // (a tile of fewer than 128 rows leaves the rest of the operand to whatever lies behind it in the slot or the
            // next one: rows of the result that nobody reads)
            uint64_t wd = w_desc + (slot * WD_SLOT >> 4), xd = x_desc + (kb0 * PLANE_BLOCK >> 4);
#pragma unroll 1
            for (int i = 0; i < nkb; ++i) {
#pragma unroll
              for (int k = 0; k < 4; ++k) tc_mma_f16_lead(tmem + t * N, wd + 2 * k, xd + 2 * k, idesc, kb0 + i + k != 0 ? 1u : 0u, lead);
              wd += L.block >> 4;
              xd += PLANE_BLOCK >> 4;
            }
            wd_commit(free_at + 8 * slot, lead);
            if (++slot == p.nslot) {
              slot = 0;
              fill ^= 1u;
            }
          }
          if (ok) wd_commit(done_at + 8 * t, lead);
        }
        if (q == 0) {  // past the K / V chunks
          const unsigned to = slot + kv_slots, laps = to / static_cast<unsigned>(p.nslot);
          fill ^= laps & 1u;
          slot = to - laps * p.nslot;
        }
      }
    if (!ok) {  // MMAs in flight end before their operands go away
      wd_commit(smem_u32(&sh.drain), lead);
      const uint32_t t0 = wd_time();
      while (!wd_try(smem_u32(&sh.drain), 0) && wd_time() - t0 < 8000u) {
      }
    }
    __syncwarp();
  } else if (warp == WD_WARPS + 2) {
    // ------------------------------------------------ arrival words and activations
    unsigned int epoch = p.epoch;
    uint32_t used = 0, piece_par = 0;
    bool ok = true;
    auto wait_all = [&]() {  // every CTA has finished phase `epoch`
      const uint32_t t0 = wd_time();
#pragma unroll 1
      for (int spins = 0;; ++spins) {
        uint32_t f[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(f[i]) : "l"(p.flags + (lane + 32 * i) * WD_FLAG) : "memory");
        bool here = true;
#pragma unroll
        for (int i = 0; i < 4; ++i) here = here && static_cast<int>(f[i] - epoch) >= 0;
        if (__all_sync(0xffffffffu, here)) break;
        if ((spins & 63) == 63) {
          uint32_t gave_up;
          asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(gave_up) : "l"(p.abort_at) : "memory");
          const bool late = gave_up == p.epoch + 1u || *abort_word || wd_time() - t0 > p.wait_limit;
          if (__any_sync(0xffffffffu, late)) {
            *abort_word = 1;
            return false;
          }
        }
      }
      if (lane == 0) mbar_arrive(&sh.seen);
      return true;
    };
    const uint32_t lead = lane == 0 ? 1u : 0u;
    const uint32_t planes_at = smem_u32(planes), staged_at = smem_u32(sh.staged);
    auto fetch = [&](const uint8_t* src, const WdLinear& L) {
      asm volatile("fence.proxy.async;" ::: "memory");  // (written by ordinary stores, read by bulk copies)
      src += r * L.kb * PLANE_BLOCK;
      int left = L.kb * PLANE_BLOCK;
      uint32_t dst = planes_at;
#pragma unroll 1
      for (int i = 0; left > 0; ++i) {
        const int n = left < WD_PIECE_KB * PLANE_BLOCK ? left : WD_PIECE_KB * PLANE_BLOCK;
        wd_expect(staged_at + 8 * i, n, lead);
        wd_copy(dst, src, n, staged_at + 8 * i, lead);
        used |= 1u << i;
        piece_par ^= 1u << i;
        left -= n;
        dst += n;
        src += n;
      }
    };
#pragma unroll 1
    for (int i = 0; i < 5 * p.s.layers; ++i) {  // the five phases of a layer; phase 1 is the attention, which reads for itself
      const int ph = i % 5, q = ph ? ph - 1 : 0;
      ++epoch;
      if (!(ok = wait_all())) break;
      if (ph != 1) fetch(q == 1 ? p.attn_planes : q == 3 ? p.act_planes : p.x_planes, p.lin[q]);
    }
    if (!ok) {
      const uint32_t t0 = wd_time();
#pragma unroll 1
      for (int i = 0; i < WD_MAX_PIECES; ++i)
        if (used & (1u << i))
          while (!wd_try(staged_at + 8 * i, ((piece_par >> i) & 1u) ^ 1u) && wd_time() - t0 < 8000u) {
          }
    }
    __syncwarp();
  } else if (warp < WD_WARPS) {
    // ------------------------------------------------ sums, norms, attention
    unsigned int epoch = p.epoch;
    const int own = hidden / WD_CTAS;  // columns of the residual stream that this CTA keeps
    uint32_t lin_no = 0, seen_no = 0;  // projections and arrivals so far
    uint32_t done_par = 0;             // of the tiles this warp reads (bit t)
    int kv_slot = 0;                   // slot and parity of the next fill, as the other roles count them
    uint32_t kv_par = 0;
    bool ok = true;

    auto ring_skip = [&](int n) {
      const unsigned to = kv_slot + n, laps = to / static_cast<unsigned>(p.nslot);
      kv_par ^= laps & 1u;
      kv_slot = to - laps * p.nslot;
    };
    auto wait_seen = [&](bool read) {  // the phase before this one is complete everywhere
      if (read) ok = wd_wait(&sh.seen, seen_no & 1u, abort_word, p.wait_limit) && ok;
      ++seen_no;
    };
    // ends a phase: this CTA's writes are visible to whoever reads its arrival word. False: leave
    auto arrive_phase = [&](bool sums) {
      ++epoch;
      ok = wd_bar_and(1, WD_COMPUTE, ok && !*abort_word);
      if (warp == 0 && ok) {
        if (sums && lane < MB) {  // squares of the owned columns of x
          float s = 0.f;
#pragma unroll 4
          for (int i = 0; i < own; ++i) s += sh.ssr[i * MB + lane];
          __stcg(p.ss + blockIdx.x * WD_MAX_B + lane, s);
        }
        __syncwarp();
        if (lane == 0)
          asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p.flags + blockIdx.x * WD_FLAG), "r"(epoch) : "memory");
      }
      return ok;
    };
    // 1 / rms of every sequence's row of x, into sh.inv (a barrier follows before it is read)
    auto row_factors = [&]() {
      constexpr int PARTS = WD_COMPUTE / MB;
      const int b = tid % MB, part = tid / MB;
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < WD_CTAS / PARTS; ++i) s += __ldcg(p.ss + (part * (WD_CTAS / PARTS) + i) * WD_MAX_B + b);
#pragma unroll
      for (int o = MB; o < 32; o *= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane < MB) sh.ssp[warp][lane] = s;
      wd_bar(1, WD_COMPUTE);
      if (tid < MB) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < WD_WARPS; ++i) t += sh.ssp[i][tid];
        sh.inv[tid] = wd_inv_rms(t, 1.0f / static_cast<float>(hidden), p.t.eps);
      }
    };
    // this CTA's partial sums go to the CTAs that finish their rows; then all four parts of its own rows are here
    auto exchange = [&](const WdLinear& L) {
      const int cols_out = L.up_off ? 2 * L.out : L.out;  // rows of the result that a CTA finishes
      if (tid == 0) mbar_expect_tx(&sh.recv, WD_CLUSTER * cols_out * MB * 4);
      const int quad = warp & 3;
#pragma unroll 1
      for (int t = warp >> 2; t < L.nt; t += 4) {
        const int row = quad * 32 + lane, up0 = L.up_off / 128;
        int kind = 0, rr = row;
        if (L.up_off && row >= up0) {
          kind = 1;
          rr = row - up0;
        }
        const bool valid = rr < L.rows;
        const int at = t * L.rows + (valid ? rr : 0), dest = (at >= L.out) + (at >= 2 * L.out) + (at >= 3 * L.out), drow = at - dest * L.out + kind * L.out;
        const uint32_t dst = map_to_cta(smem_u32(recv + (r * cols_out + drow) * RS), dest);
        const uint32_t bar = map_to_cta(smem_u32(&sh.recv), dest);
        const uint32_t ta = tmem + t * N + (static_cast<uint32_t>(quad * 32) << 16);
        ok = wd_wait(&sh.done[t], (done_par >> t) & 1u, abort_word, p.wait_limit) && ok;
        done_par ^= 1u << t;
        __syncwarp();
        tc_fence_after();
        constexpr int W = MB < 16 ? MB : 16;
#pragma unroll 1
        for (int b0 = 0; b0 < MB; b0 += W) {  // (sixteen sequences at a time: registers)
          uint32_t h[16], lo[16];
          tmem_ld_32x32b_x16(ta + b0, h);
          if constexpr (MB >= 16) tmem_ld_32x32b_x16(ta + MB + b0, lo);
          tmem_ld_wait();
#pragma unroll
          for (int b = 0; b < W; b += 4) {
            float f[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) f[e] = __uint_as_float(h[b + e]) + __uint_as_float(MB >= 16 ? lo[b + e] : h[(8 + b + e) & 15]);
            if (valid) wd_push4(dst + (b0 + b) * 4, bar, f[0], f[1], f[2], f[3]);
          }
        }
        __syncwarp();
      }
      tc_fence_before();
      ok = wd_wait(&sh.recv, lin_no & 1u, abort_word, p.wait_limit) && ok;
      ++lin_no;
      ring_skip(((L.kb + L.kbps - 1) / L.kbps) * L.nt);
    };
    // the four parts of finished row `drow` of sequence b, in rank order
    auto finished = [&](int rows_here, int drow, int b) {
      const float* at = recv + drow * RS + b;
      float t = at[0];
#pragma unroll
      for (int k = 1; k < WD_CLUSTER; ++k) t += at[k * rows_here * RS];
      return t;
    };

    // ---- the residual stream: a thread keeps one column of one sequence
    const int xb = tid / own, xd = tid - xb * own, x_col = c * (hidden / WD_NC) + r * own + xd;
    const bool owner = xb < B;
    float xr = 0.f;

    const int grp = warp >> 3, wg = warp & 7;
    const int j8 = lane & 7, kq = lane >> 3, head = wg % G;
    // One unit for all warps, or one for each half of them: as numbers, not branches, so that the code is there once.
    const int tw = shared_unit ? warp : wg;         // this warp's place in its team
    const int team = shared_unit ? 0 : grp;         // whose scratch
    int teams = shared_unit ? 1 : 2;                // units at a time
    int ch0 = shared_unit ? grp : 0;                // this half's first chunk of keys
    asm volatile("" : "+r"(teams), "+r"(ch0));      // (the compiler would write the loops out for both cases)
    const int twarps = WD_WARPS / teams, bar_id = teams == 1 ? 1 : 2 + grp, bar_n = WD_COMPUTE / teams, ch_step = 3 - teams;
    // attention scratch, where the planes are between two projections
    float* att = reinterpret_cast<float*>(planes);
    float* a_m = att;                                            // [16 warps]
    float* a_l = a_m + WD_WARPS;                                 // [16 warps]
    float* a_o = a_l + WD_WARPS;                                 // [16 warps][128]
    float* vec = a_o + WD_WARPS * WD_D + team * (G + 2) * WD_D;  // [2 teams][q of G heads, k, v][128]
    float rot_c[2] = {0.f, 0.f}, rot_s[2] = {0.f, 0.f};
    if (tw <= G) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        rot_c[i] = __ldg(p.t.cos_t + static_cast<size_t>(p.t.pos) * WD_D + lane + 32 * i);
        rot_s[i] = __ldg(p.t.sin_t + static_cast<size_t>(p.t.pos) * WD_D + lane + 32 * i);
      }
    }
    float w_next = 0.f;  // weight of the norm that x goes through next
    if (owner) {
      int id = p.t.ids[xb];
      id = id < 0 ? 0 : (id >= p.s.vocab ? p.s.vocab - 1 : id);
      xr = bf16_bits_to_f32(p.t.embed[static_cast<size_t>(id) * hidden + x_col]);
      w_next = __ldg(p.lw[0].norm1 + x_col);
      wd_put<MB>(p.x_planes, xb, x_col, xr * w_next);
      sh.ssr[xd * MB + xb] = xr * xr;
    }
    bool go = arrive_phase(true);

#pragma unroll 1
    for (int l = 0; l < p.s.layers && go; ++l) {
      // (norm weights of this layer, requested before they are waited for)
      const WdLayer& W = p.lw[l];
      const bool last = l + 1 == p.s.layers;
      float n2 = 0.f, n1_next = 0.f, wn[4] = {0.f, 0.f, 0.f, 0.f};
      if (owner) {
        n2 = wd_load_early(W.norm2 + x_col);
        if (!last) n1_next = wd_load_early(p.lw[l + 1].norm1 + x_col);
      }
      if (tw <= G) {
        const float* src = tw < G ? W.q_norm : W.k_norm;
#pragma unroll
        for (int i = 0; i < 4; ++i) wn[i] = wd_load_early(src + lane + 32 * i);
      }
#pragma unroll 1
      for (int q = 0; q < 4 && go; ++q) {
        const WdLinear& L = p.lin[q];
        const bool normed = (q & 1) == 0;
        wait_seen(normed);
        if (normed) row_factors();
        exchange(L);
        if (!normed) {  // o, down: joins the residual stream, which goes on times the weight of the norm behind it
          if (owner) {
            xr += finished(own, xd, xb);
            sh.ssr[xd * MB + xb] = xr * xr;
            if (q == 3 && last) __stcg(p.t.x + static_cast<size_t>(xb) * hidden + x_col, xr);
            else wd_put<MB>(p.x_planes, xb, x_col, xr * (q == 1 ? n2 : n1_next));
          }
          go = arrive_phase(true);
          continue;
        }
        wd_bar(1, WD_COMPUTE);
        const int n0 = c * WD_CLUSTER * L.out + r * L.out;
#pragma unroll 1
        for (int i = tid; i < L.out * B; i += WD_COMPUTE) {
          const int b = static_cast<unsigned>(i) / static_cast<unsigned>(L.out), d = i - b * L.out;
          const float inv = sh.inv[b], f = finished(q ? 2 * L.out : L.out, d, b) * inv;
          if (q) wd_put<MB>(p.act_planes, b, n0 + d, wd_swish(f) * (finished(2 * L.out, L.out + d, b) * inv));
          else __stcg(p.t.qkv + static_cast<size_t>(b) * qkv_w + n0 + d, f);
        }
        go = arrive_phase(false);
        if (q || !go) continue;

      // ---- per-head norm, rotation, append, attention over the cache
      wait_seen(true);
#pragma unroll 1
      for (int j = 0; j < nu; j += teams) {
        const int here = nu - j < teams ? nu - j : teams;  // units in hand; a chunk of each lies in the ring in turn
        if (team < here) {
          const int u = u0 + j + team, kvh = u / B, b = u - kvh * B;
          if (tw < G + 2) {
            const int hh = tw < G ? kvh * G + tw : tw == G ? heads + kvh : heads + kvh_n + kvh;
            const float* src = p.t.qkv + static_cast<size_t>(b) * qkv_w + hh * WD_D;
            float x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = __ldcg(src + lane + 32 * i);
            if (tw <= G) {
              float s2 = x[0] * x[0];
              s2 = fmaf(x[1], x[1], s2);
              s2 = fmaf(x[2], x[2], s2);
              s2 = fmaf(x[3], x[3], s2);
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
              const float inv = wd_inv_rms(s2, 1.0f / WD_D, p.t.eps);
#pragma unroll
              for (int i = 0; i < 4; ++i) x[i] = x[i] * inv * wn[i];
#pragma unroll
              for (int i = 0; i < 2; ++i) {  // rotate-half pairs (i, i + 64)
                const float re = x[i], im = x[i + 2];
                x[i] = re * rot_c[i] - im * rot_s[i];
                x[i + 2] = im * rot_c[i] + re * rot_s[i];
              }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) vec[tw * WD_D + lane + 32 * i] = x[i];
            if (tw >= G) {
              float* dst = (tw == G ? p.t.k_cache : p.t.v_cache) + l * cache_layer +
                           ((static_cast<size_t>(b) * kvh_n + kvh) * p.s.max_pos + p.t.pos) * WD_D;
#pragma unroll
              for (int i = 0; i < 4; ++i) dst[lane + 32 * i] = x[i];
            }
          }
          wd_bar(bar_id, bar_n);
          // a warp has one head; 8 lanes share a key's dot product, a lane holds 4 dims of the values
          float4 q4[4], acc = make_float4(0.f, 0.f, 0.f, 0.f);
          float m_run = -CUDART_INF_F, l_run = 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) q4[i] = *reinterpret_cast<const float4*>(vec + head * WD_D + (j8 + 8 * i) * 4);
          // Chunk -1 is the new token's own key (first warp of each head); then this team's chunks of 32 keys, of which the
          // warps of a head take eight keys each at a time.
          int at = kv_slot + grp;
          uint32_t par = kv_par;
          if (at >= p.nslot) {
            at -= p.nslot;
            par ^= 1u;
          }
#pragma unroll 1
          for (int ch = tw < G ? -1 : ch0; ch < nch; ch = ch < 0 ? ch0 : ch + ch_step) {
            asm volatile("" : "+r"(ch));  // (or the first pass would be written out apart)
            const float *k4 = vec + G * WD_D, *v4 = vec + (G + 1) * WD_D;
            int n_here = 1, first = 0;
            if (ch >= 0) {
              ok = wd_wait(&sh.full[at], par, abort_word, p.wait_limit) && ok;
              k4 = reinterpret_cast<const float*>(ring + at * WD_SLOT);
              v4 = k4 + WD_VALUES / 4;
              n_here = n_old - ch * WD_KEYS < WD_KEYS ? n_old - ch * WD_KEYS : WD_KEYS;
              first = wg / G * 8;
            }
#pragma unroll 1
            for (int key = first; key < n_here; key += 64 / G) {
              float sc[2];
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int mine = key + 4 * h + kq;
                const float* row = k4 + (mine < n_here ? mine : key) * WD_D + j8 * 4;
                float d = 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const float4 kr = *reinterpret_cast<const float4*>(row + 32 * i);
                  d = fmaf(q4[i].x, kr.x, d);
                  d = fmaf(q4[i].y, kr.y, d);
                  d = fmaf(q4[i].z, kr.z, d);
                  d = fmaf(q4[i].w, kr.w, d);
                }
                d += __shfl_xor_sync(0xffffffffu, d, 1);
                d += __shfl_xor_sync(0xffffffffu, d, 2);
                d += __shfl_xor_sync(0xffffffffu, d, 4);
                sc[h] = mine < n_here ? d * p.t.scale : -CUDART_INF_F;
              }
              float mx = fmaxf(sc[0], sc[1]);
              mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
              mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
              const float m_new = fmaxf(m_run, mx);
              const float alpha = __expf(m_run - m_new);  // 0 the first time (m_run = -inf)
              m_run = m_new;
              sc[0] = __expf(sc[0] - m_new);
              sc[1] = __expf(sc[1] - m_new);
              l_run = l_run * alpha + (sc[0] + sc[1]);  // (of this lane's keys)
              acc.x *= alpha; acc.y *= alpha; acc.z *= alpha; acc.w *= alpha;
#pragma unroll
              for (int t = 0; t < 8; ++t) {
                const float pt = __shfl_sync(0xffffffffu, sc[t >> 2], (t & 3) * 8);  // 0 past the end: the first key's row stands in
                const float4 v = *reinterpret_cast<const float4*>(v4 + (key + t < n_here ? key + t : key) * WD_D + lane * 4);
                acc.x = fmaf(pt, v.x, acc.x);
                acc.y = fmaf(pt, v.y, acc.y);
                acc.z = fmaf(pt, v.z, acc.z);
                acc.w = fmaf(pt, v.w, acc.w);
              }
            }
            __syncwarp();
            if (ch >= 0) {
              if (lane == 0) mbar_arrive(&sh.free_att[at]);
              at += here * ch_step;
#pragma unroll 1
              while (at >= p.nslot) {
                at -= p.nslot;
                par ^= 1u;
              }
            }
          }
          l_run += __shfl_xor_sync(0xffffffffu, l_run, 8);
          l_run += __shfl_xor_sync(0xffffffffu, l_run, 16);
          const int sw = team * 8 + tw;  // this warp's place in the scratch
          if (lane == 0) {
            a_m[sw] = m_run;
            a_l[sw] = l_run;
          }
          *reinterpret_cast<float4*>(a_o + sw * WD_D + lane * 4) = acc;
          wd_bar(bar_id, bar_n);
#pragma unroll 1
          for (int i = tw; i < 4 * G; i += twarps) {  // a quarter of a head per warp; the head's warps are G apart
            const int g = i >> 2, d = (i & 3) * 32 + lane;
            const int n_w = twarps / G, w0 = team * 8 + g;  // lane e < n_w stands for the head's e-th warp
            const float mw = lane < n_w ? a_m[w0 + lane * G] : -CUDART_INF_F, lw = lane < n_w ? a_l[w0 + lane * G] : 0.f;
            float m = mw;
#pragma unroll
            for (int x = 8; x > 0; x >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));  // (finite: one has the new key)
            const float fw = __expf(mw - m);
            float ls = lw * fw, o = 0.f;
#pragma unroll
            for (int x = 8; x > 0; x >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, x);
#pragma unroll 2
            for (int e = 0; e < n_w; ++e) o = fmaf(a_o[(w0 + e * G) * WD_D + d], __shfl_sync(0xffffffffu, fw, e), o);
            wd_put<MB>(p.attn_planes, b, (kvh * G + g) * WD_D + d, o / __shfl_sync(0xffffffffu, ls, 0));
          }
          if (j + teams < nu) wd_bar(bar_id, bar_n);  // the scratch is written again
        }
        ring_skip(here * nch);
      }
        go = arrive_phase(false);
      }
    }
    if (!ok) {
      *abort_word = 1;
      atomicExch(p.status, YTC_TIMEOUT);
      atomicExch(p.abort_at, p.epoch + 1u);
      const long long t0 = clock64();  // pushes to peers land before anyone leaves
      while (clock64() - t0 < 100000) {
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  if (warp == WD_WARPS + 1) tmem_dealloc(tmem, 512);
  cluster_sync_all();
}

// ------------------------------------------------------------------ host
namespace {

struct WdPlan {
  WdLinear lin[4];
  int mb, nslot, planes_bytes, recv_bytes, smem;
};

bool wide_plan(const WdShape& s, WdPlan* out) {
  const int g = s.kv_heads > 0 ? s.heads / s.kv_heads : 0;
  if (s.B < 1 || s.B > WD_MAX_B || (g != 1 && g != 2 && g != 4) || s.heads != g * s.kv_heads) return false;
  WdPlan p{};
  p.mb = s.B <= 8 ? 8 : s.B <= 16 ? 16 : 32;
  const int n[4] = {(s.heads + 2 * s.kv_heads) * WD_D, s.hidden, s.inter, s.hidden};
  const int k[4] = {s.hidden, s.heads * WD_D, s.hidden, s.inter};
  int kb_max = 0, recv_rows = 0;
  for (int i = 0; i < 4; ++i) {
    WdLinear& L = p.lin[i];
    const bool pairs = i == 2;
    if (k[i] % (64 * WD_CLUSTER) || n[i] % (8 * WD_NC)) return false;
    L.ks = k[i] / WD_CLUSTER;
    L.kb = L.ks / 64;
    const int rows = n[i] / WD_NC, cap = pairs ? 64 : 128;
    L.nt = (rows + cap - 1) / cap;
    while (L.nt <= 8 && (rows % L.nt || (!pairs && (rows / L.nt) % 8))) ++L.nt;
    if (L.nt > 8 || L.kb > WD_PIECE_KB * WD_MAX_PIECES) return false;
    L.rows = rows / L.nt;
    const int padded = (L.rows + 7) / 8 * 8;
    L.up_off = pairs ? padded * 128 : 0;
    L.block = padded * 128 * (pairs ? 2 : 1);
    L.kbps = WD_SLOT / L.block;
    if (L.kbps > L.kb) L.kbps = L.kb;
    L.out = rows / WD_CLUSTER;
    if (L.kb > kb_max) kb_max = L.kb;
    const int rr = pairs ? 2 * L.out : L.out;
    if (rr > recv_rows) recv_rows = rr;
  }
  const int own = s.hidden / WD_CTAS;
  if (own * p.mb > WD_COMPUTE) return false;  // (a thread for every element of the residual stream)
  const int att = (2 * WD_WARPS + WD_WARPS * WD_D + 2 * (g + 2) * WD_D) * 4;
  p.planes_bytes = kb_max * 2 * p.mb * 128;
  if (p.planes_bytes < att) p.planes_bytes = att;
  p.planes_bytes = (p.planes_bytes + 1023) / 1024 * 1024;
  p.recv_bytes = (WD_CLUSTER * recv_rows * (p.mb + 4) * 4 + 127) / 128 * 128;
  if (p.planes_bytes < 16384) p.planes_bytes = 16384;  // (an MMA may read 16 KB past the start of any block in the ring)
  const int rest = 227 * 1024 - p.planes_bytes - p.recv_bytes - static_cast<int>(sizeof(WdShared));
  p.nslot = rest / WD_SLOT < WD_MAX_SLOTS ? rest / WD_SLOT : WD_MAX_SLOTS;
  if (rest < 0 || p.nslot < 3) return false;
  p.smem = p.nslot * WD_SLOT + p.planes_bytes + p.recv_bytes + static_cast<int>(sizeof(WdShared));
  *out = p;
  return true;
}

const void* wide_kernel(int mb) {
  return mb == 8    ? reinterpret_cast<const void*>(decode_wide_kernel<8>)
         : mb == 16 ? reinterpret_cast<const void*>(decode_wide_kernel<16>)
                    : reinterpret_cast<const void*>(decode_wide_kernel<32>);
}

cudaLaunchConfig_t wide_config(const WdPlan& p, cudaStream_t st, cudaLaunchAttribute (&attr)[2]) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(WD_CTAS);
  cfg.blockDim = dim3(WD_THREADS);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = WD_CLUSTER;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cfg;
}

// state: [layers] WdLayer, [layers][4] CUtensorMap, a line for every arrival word and the abort word, sums of squares, planes
constexpr size_t WD_FLAG_BYTES = (WD_CTAS + 1) * WD_FLAG * sizeof(unsigned int);
size_t wide_maps_off(const WdShape& s) { return (s.layers * sizeof(WdLayer) + 127) / 128 * 128; }
size_t wide_flags_off(const WdShape& s) { return wide_maps_off(s) + static_cast<size_t>(s.layers) * 4 * sizeof(CUtensorMap); }
size_t wide_ss_off(const WdShape& s) { return wide_flags_off(s) + WD_FLAG_BYTES; }
size_t wide_planes_off(const WdShape& s) { return wide_ss_off(s) + WD_CTAS * WD_MAX_B * sizeof(float); }
size_t plane_bytes(const WdPlan& p, int k) { return static_cast<size_t>(k) * 2 * p.mb * 2; }  // both planes of k columns

}  // namespace

bool wide_step_supported(const WdShape& s) {
  // One attention unit per CTA: the form of two or more in a row faulted on 32 sequences behind 513 keys, its cause is open;
  // one per CTA ran to 3500 keys. What does not fit takes one launch per operator.
  if (s.B * s.kv_heads > WD_CTAS) return false;
  WdPlan p;
  if (!wide_plan(s, &p)) return false;
  // All clusters have to be resident at once. How many fit depends on the GPU's layout of SMs: asked once per device and kernel.
  static std::mutex mutex;
  static int fits[16][3];  // 0: not asked, 1: yes, 2: no
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return false;
  std::lock_guard<std::mutex> lock(mutex);
  int& known = fits[dev][p.mb / 16];
  if (!known) {
    const void* fn = wide_kernel(p.mb);
    cudaLaunchAttribute attr[2];
    WdPlan most = p;
    most.smem = 227 * 1024;
    cudaLaunchConfig_t cfg = wide_config(most, nullptr, attr);
    cfg.numAttrs = 1;
    int n = 0;
    known = ensure_dynamic_smem(fn, most.smem) == YTC_OK && cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n >= WD_NC ? 1 : 2;
    (void)cudaGetLastError();
  }
  return known == 1;
}

size_t wide_state_bytes(const WdShape& s) {
  WdPlan p;
  return wide_plan(s, &p) ? wide_planes_off(s) + plane_bytes(p, s.hidden + s.heads * WD_D + s.inter) : 0;
}

int wide_step_launch(const WdShape& s, const WdStep& step, const WdLayer* layers, WdState& state, cudaStream_t st) {
  WdPlan plan;
  YTC_REQUIRE(wide_plan(s, &plan) && state.dev, "decode step: shape not supported");
  char* dev = static_cast<char*>(state.dev);
  const unsigned int phases = 1u + 5u * static_cast<unsigned int>(s.layers);
  if (state.stale) {
    std::vector<CUtensorMap> maps(static_cast<size_t>(s.layers) * 4);
    for (int l = 0; l < s.layers; ++l) {
      const uint16_t* w[4] = {layers[l].qkv, layers[l].o, layers[l].gate_up, layers[l].down};
      const int n[4] = {(s.heads + 2 * s.kv_heads) * WD_D, s.hidden, 2 * s.inter, s.hidden};
      const int k[4] = {s.hidden, s.heads * WD_D, s.hidden, s.inter};
      for (int i = 0; i < 4; ++i) {
        const uint64_t dims[2] = {static_cast<uint64_t>(k[i]), static_cast<uint64_t>(n[i])};
        const uint64_t strides[1] = {static_cast<uint64_t>(k[i]) * 2};
        const uint32_t box[2] = {64, static_cast<uint32_t>(plan.lin[i].rows)};
        const int e = encode_tensor_map(&maps[4 * l + i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w[i], dims, strides, box,
                                        CU_TENSOR_MAP_SWIZZLE_128B);
        if (e != YTC_OK) return e;
      }
    }
    YTC_CUDA(cudaMemcpyAsync(dev, layers, s.layers * sizeof(WdLayer), cudaMemcpyHostToDevice, st));
    YTC_CUDA(cudaMemcpyAsync(dev + wide_maps_off(s), maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice, st));
    YTC_CUDA(cudaMemsetAsync(dev + wide_flags_off(s), 0, WD_FLAG_BYTES, st));
    YTC_CUDA(cudaStreamSynchronize(st));  // (the host arrays leave scope)
    state.epoch = 0;
    state.stale = false;
  } else if (state.epoch > 0x70000000u) {  // long before the phase numbers wrap
    YTC_CUDA(cudaMemsetAsync(dev + wide_flags_off(s), 0, WD_FLAG_BYTES, st));
    state.epoch = 0;
  }
  WdParams p{};
  p.s = s;
  p.t = step;
  p.lw = reinterpret_cast<const WdLayer*>(dev);
  p.maps = reinterpret_cast<const CUtensorMap*>(dev + wide_maps_off(s));
  p.flags = reinterpret_cast<unsigned int*>(dev + wide_flags_off(s));
  p.abort_at = p.flags + WD_CTAS * WD_FLAG;
  p.ss = reinterpret_cast<float*>(dev + wide_ss_off(s));
  p.x_planes = reinterpret_cast<uint8_t*>(dev + wide_planes_off(s));
  p.attn_planes = p.x_planes + plane_bytes(plan, s.hidden);
  p.act_planes = p.attn_planes + plane_bytes(plan, s.heads * WD_D);
  for (int i = 0; i < 4; ++i) p.lin[i] = plan.lin[i];
  p.epoch = state.epoch;
  p.nslot = plan.nslot;
  p.planes_bytes = plan.planes_bytes;
  p.recv_bytes = plan.recv_bytes;
  p.wait_limit = static_cast<uint32_t>(wait_cycle_limit() >> 10) + 1u;
  p.status = device_status_word();
  const void* fn = wide_kernel(plan.mb);
  const int sa = ensure_dynamic_smem(fn, plan.smem);
  if (sa != YTC_OK) return sa;
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = wide_config(plan, st, attr);
  void* args[] = {&p};
  YTC_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
  count_launch();
  state.epoch += phases;
  return YTC_OK;
}

}  // namespace ytk
