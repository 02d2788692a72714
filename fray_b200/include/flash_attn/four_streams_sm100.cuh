#pragma once
// Attention forward for sm_100a at head dim 64 with four independent streams per CTA, as a persistent grid.
//
// One CTA of 20 warps per SM walks through its list of work items; an item is two 128-row query tiles of one (batch, head)
// slice against all of their keys, in steps of 64.
//   warps 0-15  softmax: query tile (warp >> 2) & 1, group warp >> 3, 32 rows of the tile each, thread = row
//   warps 16, 19  MMA issue for query tile 0 / 1 (warp-uniform code, one elected lane issues)
//   warp 17     TMA producer (Q tiles, K and V through a ring of stages of two steps)
//   warp 18     TMA stores of finished tiles
//
// Two softmax threads per row (fwd_duo_sm100.cuh) have to agree on every step's offset, and a tile's next scores wait for its last
// product.  At head dim 64 tensor memory has room to do without both: a tile's steps go to two groups in turn, each with a score
// buffer, an accumulator, an offset and a row sum of its own, so that no warp waits for another one inside an item, and while one
// group's product and next scores run the other three are in their exponentials.  At the item's end the two accumulators are
// weighted with what their offsets differ in and added.  What bounds it is the special-function unit (2048 cycles per 128 keys of
// two tiles at 16 results a clock; exponentials and nothing else 2400 with the items' ends) and, in long calls, the board's power:
// 2520 cycles per 128 keys at 4096 keys, 2627 with two threads per row.
//
//   * An issuing warp per query tile: one for both tiles' four streams was busy all the time (969 k cycles of a call of 1197 k with
//     nothing to wait for, two 645 k).  At head dim 128 two lose (12 to 15 %): there both tiles' products fill the pipe.
//   * Steps of 64 keys also leave less behind a sequence's end and above the diagonal.
//   * What an item's end costs was half of a short call: items are decoded once (CTA's list in shared memory; divisions in the
//     roles took 11 k cycles an item with the rest below), Q has two buffers, and each tile's last stage issues the next item's
//     first scores.
//   * One tensor-memory load of 64 columns instead of two of 32 (715 : 705 us at 8 x 16 x 4096).
//
// us, two threads per row -> four streams, each behind lasting load: 6 x 12 x 333 causal 8.9 -> 8.1, 3 x 16/4 x 1326 causal 27.8
// -> 26.2, 2 x 32/8 x 3000 causal 119.8 -> 115.5, 4 x 16 x 4096 causal 209.5 -> 203.4, 1 x 32 x 16384 causal 1490 -> 1452,
// 8 x 16 x 4096 725 -> 712, 16 x 16 x 900 with large logits 110.2 -> 105.0.
// Wide scores, whose offsets move often, two of them per row: 0.81 to 0.97 of the time of two threads per row over 34 drawn calls of
// up to 8413 keys (unit variance 0.82 to 0.98).  The compiler spills: 88 bytes of stores and 92 of loads at 96 registers.
// Tried and left out: 12 or 25 % of the exponentials on the FMA pipe (level, 2 to 5 % slower: the board is at its power limit),
// scores fetched again instead of kept (spills elsewhere, 3 % slower), the merge by the group that ends last while the other goes on
// (400 bytes of spills, 10 % slower), tile 1 started behind tile 0 (level), offsets moved from 2^12 on instead of 2^8 (level).
//
// Every barrier wait is bounded (see sm100_ptx.cuh).  A softmax warp goes through its items whether or not a wait ran out, so the
// named barriers always meet; producer, stores and issue stop at a step, a tile or an item of their own, the issuing warps as whole
// warps.

#include <type_traits>

#include "host_sm100.cuh"
#include "sm100_ptx.cuh"
#include "softmax_tile_sm100.cuh"

namespace fray {
namespace sm100 {

template <int D>
struct QuadCfg {
  static_assert(D == 64, "tensor memory holds four accumulators of 64 columns beside four score buffers");
  static constexpr int BM = 128, BN = 64;      // rows per query tile, keys per step
  static constexpr int kThreads = 640;
  static constexpr int STAGES = 3;             // ring stages: K and V of two steps (one TMA box each)
  static constexpr int kTileBytes = BM * 128;  // a query tile, or K or V of a stage: 128 rows of one 128-byte panel
  static constexpr int kStepBytes = BN * 128;
  static constexpr int kStageBytes = 2 * kTileBytes;
  static constexpr int kOffQ = 0;
  static constexpr int kOffKV = 4 * kTileBytes;  // Q tiles of two items
  static constexpr int kOffOut = kOffKV + STAGES * kStageBytes;  // a staging tile per query tile
  static constexpr int kOffBars = kOffOut + 2 * kTileBytes;
  static constexpr int kNumBars = 8 + 2 * STAGES + 3 * 4 + 2 + 4;
  static constexpr int kOffStats = kOffBars + ((kNumBars * 8 + 16 + 127) / 128) * 128;  // [2][2 tiles][2 groups][128] offset, row sum
  static constexpr int kOffItems = kOffStats + 2 * 2 * 2 * 128 * 8;
  static constexpr int kMaxItems = 256;  // of a CTA, with the end mark; a launch of more than 255 items per SM has more CTAs
  static constexpr int kUsedBytes = kOffItems + kMaxItems * 16;
  static constexpr int kSmemBytes = kUsedBytes + 1024;  // slack to bring the dynamic segment to a 1024-byte boundary
  static_assert(kSmemBytes <= 232448, "exceeds the 227 KB shared memory of one CTA");
  static constexpr int kTmemCols = 512;
  static constexpr uint32_t kColS = 0, kColO = 256;  // 64 columns per tile and group each
  // Register budgets after setmaxnreg: per scheduler four softmax warps and one other, 4 x 104 + 64 = 5 x 96.
  static constexpr int kRegsLaunch = 96, kRegsSoftmax = 104, kRegsOther = 64;
  static constexpr int kRegsTotal = 512 * kRegsSoftmax + 128 * kRegsOther;
  static_assert(kRegsTotal <= kThreads * kRegsLaunch, "register budgets exceed the CTA's allocation");
};

template <int D>
__global__ void __launch_bounds__(640, 1)
attn_fwd_quad_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o, int num_heads, int num_bh,
                     int seq_len, int causal, float scale_log2, int kv_group, float* lse, int seq_k, int heaviest_first, int matched,
                     int n_kv, int n_pairs, int total) {
  using Cfg = QuadCfg<D>;
  constexpr int BN = Cfg::BN, STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t align_off = ((raw_addr + 1023u) & ~1023u) - raw_addr;
  uint8_t* smem = smem_raw + align_off;
  uint8_t* q_smem = smem + Cfg::kOffQ;
  uint8_t* kv_smem = smem + Cfg::kOffKV;
  uint8_t* out_smem = smem + Cfg::kOffOut;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBars);
  uint64_t* q_full = bars;                 // [2][2]   producer -> MMA: Q of tile i, of every other item
  uint64_t* q_free = bars + 4;             // [2][2]   MMA -> producer  (the item's last scores of tile i have read Q_i)
  uint64_t* kv_full = bars + 8;            // [STAGES] producer -> MMA
  uint64_t* kv_empty = kv_full + STAGES;   // [STAGES] MMA of either tile -> producer
  uint64_t* s_full = kv_empty + STAGES;    // [2][2]   MMA -> softmax group g of tile i
  uint64_t* p_full = s_full + 4;           // [2][2]   softmax group g of tile i -> MMA
  uint64_t* o_full = p_full + 4;           // [2][2]   MMA -> softmax i (the item's last P.V of group g)
  uint64_t* o_free = o_full + 4;           // [2]      softmax i -> MMA (the item's accumulators are in registers)
  uint64_t* out_full = o_free + 2;         // [2]      softmax i -> store warp
  uint64_t* out_free = out_full + 2;       // [2]      store warp -> softmax i
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::kNumBars);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);
  float2* stats = reinterpret_cast<float2*>(smem + Cfg::kOffStats);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;

  const int stride = static_cast<int>(gridDim.x), unit = static_cast<int>(blockIdx.x);
  // Steps of the query tile whose first row is row0.
  auto steps = [&](int row0) {
    const int lim = (row0 + Cfg::BM) / BN;
    return row0 >= seq_len ? 0 : causal && lim < n_kv ? lim : n_kv;
  };

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(o_free + i, 8);
      mbar_init(out_full + i, 8);
      mbar_init(out_free + i, 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(q_full + i, 1);
      mbar_init(q_free + i, 1);
      mbar_init(s_full + i, 1);
      mbar_init(p_full + i, 4);
      mbar_init(o_full + i, 1);
    }
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(kv_full + s, 1);
      mbar_init(kv_empty + s, 2);
    }
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  // The CTA's items (first row, batch, head, K/V head; a first row of -1 ends them).  Items are numbered slice by slice (CTAs that run side by side share a
  // slice's K and V in L2) or, with a causal mask and by duo_heaviest_first, pair by pair, the heaviest of all slices first; dealt
  // round by round, causal rounds in alternating direction, or matched by twos (duo_matched).
  int4* items = reinterpret_cast<int4*>(smem + Cfg::kOffItems);
  for (int k = tid - 64; k >= 0 && k < Cfg::kMaxItems; k += Cfg::kThreads - 64) {
    int idx;
    if (matched) idx = matched_item(k, stride, unit, n_pairs, total);
    else idx = k * stride + ((causal && (k & 1)) ? stride - 1 - unit : unit);
    int4 item = make_int4(-1, 0, 0, 0);
    if (idx < total) {
      const int run = heaviest_first ? num_bh : n_pairs;
      const int hi = idx / run, lo = idx - hi * run;
      const int bh = heaviest_first ? lo : hi, u = heaviest_first ? hi : lo;
      item.x = (causal ? n_pairs - 1 - u : u) * (2 * Cfg::BM);
      item.y = bh / num_heads;
      item.z = bh - item.y * num_heads;
      item.w = item.z / kv_group;
    }
    items[k] = item;
  }
  grid_dependency_wait();
  if (tid == 32) *abort_flag = (*reinterpret_cast<volatile int*>(&fray_attn_status[0]) != 0) ? 2u : 0u;
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  grid_launch_dependents();
  const uint32_t tmem_base = *tmem_slot;
  if (*abort_flag == 2u) {  // an earlier launch left the device status raised
    if (warp == 0) tmem_dealloc(tmem_base, Cfg::kTmemCols);
    return;
  }
  if (warp < 16) {
    // =============================================================== softmax
    set_max_regs_inc<Cfg::kRegsSoftmax>();
    const int i = (warp >> 2) & 1;  // query tile
    const int g = warp >> 3;        // group: steps g, g + 2, ... of an item; which 32 columns of O
    const int w = warp & 3;
    const int r = tid & 127;        // row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>(w * 32) << 16;
    const uint32_t t_s = tmem_base + Cfg::kColS + (i * 2 + g) * 64 + lane_base;
    const uint32_t t_o = tmem_base + Cfg::kColO + i * 128 + lane_base;  // group 0's accumulator, 64 columns on group 1's
    const uint32_t s_bar = smem_u32(s_full + i * 2 + g);
    const uint32_t p_bar = smem_u32(p_full + i * 2 + g);
    float2* my_stat = stats + (i * 2 + g) * 128 + r;
    const int other_off = g ? -128 : 128;
    const int pair_bar = 1 + i * 4 + w;
    uint32_t phases = 0;  // parities: bit 0 s_full, bits 1, 2 o_full of group 0 / 1, bit 3 out_free, bit 4 slots
    float m_ref = -INFINITY, l_run = 0.f;

    // One step: 64 scores of a row.  lim (MASK): keys from lim on are past the end or above the diagonal.
    auto step = [&](auto mask_tag, int lim) __attribute__((always_inline)) {
      constexpr bool MASK = decltype(mask_tag)::value;
      mbar_wait(s_bar, phases & 1, abort_flag, 0x201 + i, lim);
      phases ^= 1u;
      tc_fence_after_sync();
      uint32_t sa[32], sb[32];
      tmem_ld_x64(t_s, sa, sb);
      tmem_wait_ld();
      if constexpr (MASK) {
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          if (c >= lim) sa[c] = __float_as_uint(-INFINITY);
          if (c + 32 >= lim) sb[c] = __float_as_uint(-INFINITY);
        }
      }
      const float mine = max_64(sa, sb);
      if (__any_sync(0xffffffffu, (mine - m_ref) * scale_log2 > kRescaleThreshold)) {
        float alpha = 1.f;
        if ((mine - m_ref) * scale_log2 > kRescaleThreshold) {
          // a row without any offset yet has nothing in O (its first product overwrites it)
          alpha = m_ref == -INFINITY ? 1.f : ex2_approx((m_ref - mine) * scale_log2);
          l_run *= alpha;
          m_ref = mine;
        }
        // These scores were issued behind the group's previous product: they are complete, so is it.
        if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
          for (int c = 0; c < D; c += 16) {
            uint32_t orr[16];
            tmem_ld_x16(t_o + g * 64 + c, orr);
            tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < 16; ++x) orr[x] = __float_as_uint(__uint_as_float(orr[x]) * alpha);
            tmem_st_x16(t_o + g * 64 + c, orr);
          }
          tmem_wait_st();
        }
      }
      const float neg_m = (m_ref == -INFINITY) ? 0.f : -m_ref * scale_log2;
      const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2), neg_m2 = pack_f32x2(neg_m, neg_m);
      uint64_t rsp0 = 0ull, rsp1 = 0ull;
      uint32_t pk[16], pk2[16];
      exp_32(sa, scale2, neg_m2, rsp0, rsp1, pk);
      tmem_st_x16(t_s, pk);
      exp_32(sb, scale2, neg_m2, rsp0, rsp1, pk2);
      tmem_st_x16(t_s + 16, pk2);
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) arrive_on(p_bar);
      float r0, r1, r2, r3;
      unpack_f32x2(rsp0, r0, r1);
      unpack_f32x2(rsp1, r2, r3);
      l_run += (r0 + r1) + (r2 + r3);
    };

    for (int k = 0;; ++k) {
      const int m0 = items[k].x;
      if (m0 < 0) break;
      const int row = m0 + i * Cfg::BM;
      const int n_i = steps(row);
      if (n_i == 0) continue;
      // the first steps see every key of their tile
      int n_full = seq_k / BN;
      if (causal) n_full = (row + 1) / BN < n_full ? (row + 1) / BN : n_full;
      if (n_full > n_i) n_full = n_i;
      const int lim = causal && row + r + 1 < seq_k ? row + r + 1 : seq_k;  // keys the row may see
      m_ref = -INFINITY;
      l_run = 0.f;
      int j = g;
      for (; j < n_full; j += 2) step(std::false_type{}, 0);
      for (; j < n_i; j += 2) step(std::true_type{}, lim - j * BN);
      // The groups' streams meet: weights of their accumulators, over the whole row sum.  The slots alternate from item to item: a group writes one again two items on, past a barrier behind the other's read.
      float2* slot = my_stat + ((phases >> 4) & 1) * 512;
      phases ^= 16u;
      *slot = make_float2(m_ref, l_run);
      named_barrier_sync(pair_bar, 64);
      const float2 other = slot[other_off];
      const float m_all = fmaxf(m_ref, other.x);
      const float m_safe = m_all == -INFINITY ? 0.f : m_all;
      const float w_mine = m_ref == -INFINITY ? 1.f : ex2_approx((m_ref - m_safe) * scale_log2);
      const float w_other = other.x == -INFINITY ? 1.f : ex2_approx((other.x - m_safe) * scale_log2);
      l_run = l_run * w_mine + other.y * w_other;
      const float inv_l = l_run > 0.f ? 1.f / l_run : 1.f;
      const float w0 = (g ? w_other : w_mine) * inv_l, w1 = (g ? w_mine : w_other) * inv_l;
      mbar_wait(out_free + i, (phases >> 3) & 1, abort_flag, 0x321 + i, k);
      mbar_wait(o_full + i * 2, (phases >> 1) & 1, abort_flag, 0x331 + i, k);
      phases ^= 8u | 2u;
      uint32_t oa[32], ob[32];
      if (n_i > 1) {
        mbar_wait(o_full + i * 2 + 1, (phases >> 2) & 1, abort_flag, 0x333 + i, k);
        phases ^= 4u;
        tc_fence_after_sync();
        tmem_ld_x32(t_o + g * 32, oa);
        tmem_ld_x32(t_o + 64 + g * 32, ob);
        tmem_wait_ld();
#pragma unroll
        for (int x = 0; x < 32; ++x) oa[x] = __float_as_uint(__uint_as_float(oa[x]) * w0 + __uint_as_float(ob[x]) * w1);
      } else {  // a single step: group 1 has left nothing
        tc_fence_after_sync();
        tmem_ld_x32(t_o + g * 32, oa);
        tmem_wait_ld();
#pragma unroll
        for (int x = 0; x < 32; ++x) oa[x] = __float_as_uint(__uint_as_float(oa[x]) * w0);
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(o_free + i);
      uint8_t* out_row = out_smem + i * Cfg::kTileBytes + r * 128;
#pragma unroll
      for (int x = 0; x < 32; x += 8) {
        uint4 v4;
        v4.x = pack_half2(__uint_as_float(oa[x + 0]), __uint_as_float(oa[x + 1]));
        v4.y = pack_half2(__uint_as_float(oa[x + 2]), __uint_as_float(oa[x + 3]));
        v4.z = pack_half2(__uint_as_float(oa[x + 4]), __uint_as_float(oa[x + 5]));
        v4.w = pack_half2(__uint_as_float(oa[x + 6]), __uint_as_float(oa[x + 7]));
        const int chunk = g * 4 + (x >> 3);  // 16-byte chunk inside the 128-byte row
        *reinterpret_cast<uint4*>(out_row + ((chunk ^ (r & 7)) << 4)) = v4;
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(out_full + i);
      if (lse != nullptr && g == 0) {
        const int4 item = items[k];
        const int row_r = item.x + i * Cfg::BM + r;
        if (row_r < seq_len)
          lse[(static_cast<size_t>(item.y) * num_heads + item.z) * seq_len + row_r] =
              l_run > 0.f ? (m_all * scale_log2 + log2f(l_run)) * 0.69314718055994531f : -INFINITY;
      }
    }
  } else {
    set_max_regs_dec<Cfg::kRegsOther>();
    if (warp == 18 && lane == 0) {
      // ============================================================= stores of finished tiles
      uint32_t stores = 0;  // parities of the two staging tiles
      mbar_arrive(out_free);
      mbar_arrive(out_free + 1);
      bool stop = false;
      for (int k = 0; !stop; ++k) {
        const int4 item = items[k];
        if (item.x < 0) break;
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          const int row = item.x + i * Cfg::BM;
          if (row >= seq_len) continue;
          mbar_wait(out_full + i, (stores >> i) & 1, abort_flag, 0x341 + i, k);
          stores ^= 1u << i;
          stop = *abort_flag != 0;
          if (stop) break;
          tma_store_4d(&tm_o, out_smem + i * Cfg::kTileBytes, 0, row, item.z, item.y);
          tma_store_commit();
          tma_store_wait_read();
          mbar_arrive(out_free + i);
        }
      }
    } else if (warp == 17 && lane == 0) {
      // ============================================================= TMA producer
      uint32_t t_run = 0;  // ring stages loaded so far
      uint32_t q_cnt = 0;  // items whose Q this CTA has loaded: tile 0's in the low half, tile 1's in the high half
      bool stop = false;
      for (int k = 0; !stop; ++k) {
        const int4 item = items[k];
        if (item.x < 0) break;
        const int n0 = steps(item.x), n1 = steps(item.x + Cfg::BM);
        auto load_q = [&](int i) __attribute__((always_inline)) {
          const uint32_t cnt = (q_cnt >> (16 * i)) & 0xffffu, buf = cnt & 1;
          mbar_wait(q_free + i * 2 + buf, ((cnt >> 1) & 1) ^ 1, abort_flag, 0x402 + i, k);
          mbar_expect_tx(q_full + i * 2 + buf, Cfg::kTileBytes);
          tma_load_4d(q_smem + (i * 2 + buf) * Cfg::kTileBytes, &tm_q, q_full + i * 2 + buf, 0, item.x + i * Cfg::BM, item.z, item.y);
          q_cnt += 1u << (16 * i);
        };
        load_q(0);
        const int stages = ((n0 > n1 ? n0 : n1) + 1) / 2;
        for (int t = 0; t < stages; ++t) {
          const int slot = t_run % STAGES;
          mbar_wait(kv_empty + slot, ((t_run / STAGES) & 1) ^ 1, abort_flag, 0x401, t);
          stop = *abort_flag != 0;
          if (stop) break;
          mbar_expect_tx(kv_full + slot, Cfg::kStageBytes);
          uint8_t* dst = kv_smem + slot * Cfg::kStageBytes;
          tma_load_4d(dst, &tm_k, kv_full + slot, 0, 2 * t * BN, item.w, item.y);
          tma_load_4d(dst + Cfg::kTileBytes, &tm_v, kv_full + slot, 0, 2 * t * BN, item.w, item.y);
          ++t_run;
          if (t == 0 && n1 > 0) load_q(1);
        }
      }
    } else if (warp == 16 || warp == 19) {
      // ============================================================= MMA issue of a query tile (whole warp, one elected lane issues)
      // tile; as tmem_cols below read from lane 0, so that the compiler knows it to be the same in all lanes
      const int i = __shfl_sync(0xffffffffu, warp, 0) == 16 ? 0 : 1;
      constexpr uint64_t kDescK = smem_desc_sw128(16, 1024);
      constexpr uint64_t kDescV = smem_desc_sw128(Cfg::kTileBytes, 1024);
      constexpr uint32_t kIdescQK = idesc_f16_f32(Cfg::BM, BN, false, false);
      constexpr uint32_t kIdescPV = idesc_f16_f32(Cfg::BM, D, false, true);
      const uint32_t q_addr = smem_u32(q_smem);
      const uint32_t kv_addr = smem_u32(kv_smem);
      const uint32_t tmem_cols = __shfl_sync(0xffffffffu, tmem_base, 0);

      uint32_t phases = 4;  // bits 0, 1 p_full of group g; bit 2 o_free
      uint32_t q_cnt = 0;    // items whose Q has been met
      uint32_t kv_seen = 0;  // ring stages met: in order, each once
      uint64_t* p_bar = p_full + i * 2;
      uint64_t* s_bar = s_full + i * 2;
      const uint32_t t_s0 = tmem_cols + Cfg::kColS + i * 128, t_o0 = tmem_cols + Cfg::kColO + i * 128;
      auto meet_kv = [&](uint32_t t) __attribute__((always_inline)) {
        for (; kv_seen <= t; ++kv_seen)
          mbar_wait(kv_full + kv_seen % STAGES, (kv_seen / STAGES) & 1, abort_flag, 0x501, kv_seen);
      };
      auto meet_p = [&](int g, int j) __attribute__((always_inline)) {
        mbar_wait(p_bar + g, (phases >> g) & 1, abort_flag, 0x503 + i, j);
        phases ^= 1u << g;
        tc_fence_after_sync();
      };
      // (one lane) accumulator of group g (+)= P . V of its step in ring stage t
      auto mma_pv = [&](int g, uint32_t t, uint32_t more) __attribute__((always_inline)) {
        const uint64_t v_d = smem_desc_at(kDescV, kv_addr + (t % STAGES) * Cfg::kStageBytes + Cfg::kTileBytes + g * Cfg::kStepBytes);
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk)
          mma_ts(t_o0 + g * 64, t_s0 + g * 64 + kk * 8, v_d + ((kk * 2048) >> 4), kIdescPV, more | (kk > 0));
      };
      // (one lane) scores of group g's step in ring stage t
      auto mma_qk = [&](int g, uint32_t t, uint32_t q_buf) __attribute__((always_inline)) {
        const uint64_t q_d = smem_desc_at(kDescK, q_addr + (i * 2 + q_buf) * Cfg::kTileBytes);
        const uint64_t k_d = smem_desc_at(kDescK, kv_addr + (t % STAGES) * Cfg::kStageBytes + g * Cfg::kStepBytes);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          mma_ss(t_s0 + g * 64, q_d + ((kk * 32) >> 4), k_d + ((kk * 32) >> 4), kIdescQK, kk > 0);
      };
      auto item_row = [&](int k) { return __shfl_sync(0xffffffffu, items[k].x, 0); };
      // Steps of the tile in the current and the next item (the first time round there is no current one), ring stages of the two
      // items, ring stage of their first steps.
      int n = 0, nn = 0, s_max = 0, s_nxt = 0;
      uint32_t t_base = 0, t_next = 0;
      int k = 0;
      int row = item_row(0);
      auto load_next = [&]() {
        nn = 0;
        s_nxt = 0;
        if (row >= 0) {
          const int a0 = steps(row), a1 = steps(row + Cfg::BM);
          nn = i ? a1 : a0;
          s_nxt = ((a0 > a1 ? a0 : a1) + 1) / 2;
        }
      };
      load_next();
      if (row >= 0) {
        while (true) {
          const int s_i = (n + 1) / 2;
          const int steady_end = (n - 3) >> 1;  // stages before it have both steps, and so has the next one, not the item's last
          // Group g's first scores of the next item: in the tile's last stage, or straight away if it has none.
          auto first_scores = [&](int g) __attribute__((always_inline)) {
            if (g < nn) {
              if (g == 0) {
                mbar_wait(q_full + i * 2 + (q_cnt & 1), (q_cnt >> 1) & 1, abort_flag, 0x511 + i);
                ++q_cnt;
                meet_kv(t_next);
              }
              tc_fence_after_sync();
              const uint32_t q_buf = (q_cnt - 1) & 1;
              if (elect_one()) {
                mma_qk(g, t_next, q_buf);
                mma_commit(s_bar + g);
                if (g + 1 == nn) mma_commit(q_free + i * 2 + q_buf);
              }
              __syncwarp();
            }
          };
          for (int st = 0; st < s_i; ++st) {
            const bool last = st + 1 == s_i;
            if (!last) meet_kv(t_base + st + 1);
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              const int j = 2 * st + g;
              const uint32_t t = t_base + st, q_buf = (q_cnt - 1) & 1;
              if (j < n) {
                if (j == 0) {
                  // the first products of an item overwrite O: the previous item's epilogue must have read both accumulators
                  mbar_wait(o_free + i, (phases >> 2) & 1, abort_flag, 0x507 + i);
                  phases ^= 4u;
                }
                meet_p(g, j);
                if (elect_one()) {
                  mma_pv(g, t, st > 0);
                  if (j + 2 >= n) mma_commit(o_full + i * 2 + g);
                  if (g == 1 || j + 1 == n) mma_commit(kv_empty + t % STAGES);
                  if (!last && j + 2 < n) {
                    mma_qk(g, t + 1, q_buf);
                    mma_commit(s_bar + g);
                    if (j + 3 == n) mma_commit(q_free + i * 2 + q_buf);
                  }
                }
                __syncwarp();
              }
              if (last) first_scores(g);
            }
            if (st == 0) {
              // the stages between, with nothing to decide
              for (; st + 1 < steady_end; ++st) {
                const uint32_t t = t_base + st + 1, q_buf = (q_cnt - 1) & 1;
                meet_kv(t + 1);
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                  meet_p(g, 2 * st + 2 + g);
                  if (elect_one()) {
                    mma_pv(g, t, 1);
                    if (g == 1) mma_commit(kv_empty + t % STAGES);
                    mma_qk(g, t + 1, q_buf);
                    mma_commit(s_bar + g);
                  }
                  __syncwarp();
                }
              }
            }
          }
          // Stages that only the other tile uses: handed back once they have landed, as an arrival must not come before the slot's
          // last phase is complete.
          for (int st = s_i; st < s_max; ++st) {
            meet_kv(t_base + st);
            if (elect_one()) mbar_arrive(kv_empty + (t_base + st) % STAGES);
            __syncwarp();
          }
          if (s_i == 0)
            for (int g = 0; g < 2; ++g) first_scores(g);
          if (row < 0) break;
          if (__any_sync(0xffffffffu, *abort_flag != 0)) break;  // by vote: item_row and the elections need every lane
          n = nn;
          s_max = s_nxt;
          t_base = t_next;
          t_next = t_base + s_nxt;
          row = item_row(++k);
          load_next();
        }
      }
    }
  }

  if (*abort_flag == 1u) settle_after_abort();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, Cfg::kTmemCols);
}

// Host launcher, with the tensor maps (boxes of 128 rows) and the deal that the row-pair kernel's launcher has worked out.  Returns an
// AttnReturnCode.
template <int D>
inline int launch_attn_fwd_quad(const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_v, const CUtensorMap& tm_o,
                                const AttnShape& shp, const AttnExtras& ex, bool causal, float scale_log2, bool heaviest_first,
                                bool matched, int n_pairs, int items, int sms, cudaStream_t stream) {
  using Cfg = QuadCfg<D>;
  auto kernel = attn_fwd_quad_kernel<D>;
  const int rc = ensure_dynamic_smem<Cfg>(kernel, Cfg::kSmemBytes, Cfg::kThreads, Cfg::kRegsTotal);
  if (rc != kAttnOk) return rc;
  const int fewest = (items + Cfg::kMaxItems - 2) / (Cfg::kMaxItems - 1);  // CTAs: their lists hold no more
  return launch_overlapped(kernel, dim3(items < sms ? items : sms > fewest ? sms : fewest), Cfg::kThreads, Cfg::kSmemBytes, stream, tm_q,
                           tm_k, tm_v, tm_o, shp.H, shp.B * shp.H, shp.S, causal ? 1 : 0, scale_log2, ex.kv_group, ex.lse, ex.seq_k,
                           heaviest_first ? 1 : 0, matched ? 1 : 0, pieces(ex.seq_k, Cfg::BN), n_pairs, items);
}

}  // namespace sm100
}  // namespace fray
