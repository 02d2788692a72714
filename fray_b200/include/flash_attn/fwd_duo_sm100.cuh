#pragma once
// Attention forward for sm_100a with two softmax threads per query row, as a persistent grid.
//
// One CTA of 20 warps per SM walks through the work items blockIdx.x, blockIdx.x + gridDim.x, ...; an item is two
// 128-row query tiles of one (batch, head) slice against all of their KV tiles.
//   warps 0-15  softmax: query tile (warp >> 2) & 1, keys 64 * (warp >> 3) .. + 63 of every step; warps w and w + 8 hold
//               the same 32 rows (a warp reaches the 32 tensor-memory lanes of warp & 3 only), thread = row
//   warp 16     MMA issue for both tiles (warp-uniform code, one elected lane issues)
//   warp 17     TMA producer (Q tiles, K_j, V_j through a ring of STAGES buffers)
//   warp 18     TMA stores of finished tiles
//   warp 19     idle (fills the warpgroup for setmaxnreg)
// At head dim 64 most calls go to four independent streams per CTA instead (duo_quad, four_streams_sm100.cuh).
// At head dim 128 long calls put a pair of CTAs to an item (duo_pair): two query tiles in each of the two, every product one
// cta_group::2 instruction that the leader's warp 16 issues for both, each CTA with half of K's rows and of V's columns.
//
// What bounds the kernel is the chain S(j) -> softmax -> P.V(j) -> S(j+1) of each query tile (P overwrites its S, tensor
// memory has no room for another buffer).  With one thread per row (fwd_ws_sm100.cuh) a tile's softmax is one in-order
// warp per scheduler: 2100 cycles per step, half of them latency, and 3250 for the chain.  Here each scheduler has two
// warps per tile, each with half of the exponentials, which cover each other's latencies.  Per step the halves of a row
// only have to agree on the exponent offset: one OR-reducing barrier of the two warps asks whether any row's maximum
// outgrew its offset by 2^8 (the lazy-rescale rule), and only then are maxima exchanged and O rescaled, by the softmax
// warps themselves (S(j) complete implies P.V(j-1) complete: the commit covers it).  There is no correction group.
//
//   * P of a half sits in the first 32 columns of that half's 64 score columns, so neither half overwrites scores the
//     other still needs; the first 32 keys are handed over while the second 32 are fetched from tensor memory again
//     (keeping them costs registers and lets the compiler move their exponentials in front of the hand-over: 3-5 %).
//   * Between items (as a CTA's exit and the next one's set-up cost 6-8 us): barriers, tensor memory and the ring live on,
//     the next item's Q, K and first scores come behind the current item's last steps, accumulators are handed back as
//     soon as they are in registers, and a warp of its own stores finished tiles from one staging tile that both query
//     tiles use in turn, which leaves room for four ring slots at head dim 128.
//   * Values a step does not need are worked out again per item instead of kept: 104 registers hold a half row and its
//     P with 4 to 24 bytes of spill stores, by form (10 % against the first version, which spilled 100).
//
// Measured against the faster of the two-tile and the one-tile kernel, each behind 150 ms of its own load (us, same run): 4 x
// 32 x 4096 x 128 981-1028 : 1051-1099, causal 569-572 : 648-656, 1 x 32 x 16384 causal 2070-2080 : 2180-2261, 2 x 16 x 2048 75 :
// 79, 16 x 16 x 1024 x 64 103 : 122, 16 x 16 x 1024 x 128 causal 105 : 127, 8 x 16 x 4096 x 64 721-726 : 801-807, 4 x 16 x 2048
// x 64 causal 59 : 83; 20 launches of the first from an idle board 853-890 : 909-956 (with products issued as they are now:
// 823-840, see the MMA warp).  2870 cycles per 128 keys of two tiles inside an item; an item costs 2 to 3 us beside its steps.
// Tried and left out (us or thousand cycles a CTA, 4 x 32 x 4096 behind lasting load unless noted): 6 to 25 % of the exponentials as
// a polynomial of degree 4 or 5 on the FMA pipe (cycles level to -2 %, but the board is at its power limit: +2 to +5 %), the first 32
// exponentials on trust, ahead of the halves' agreement (1326 -> 1366: those of the two tiles meet at the unit then), the MMA warp's
// waits for K and V once per step (level), an issuing warp per query tile (975 -> 1111: the tiles' products interleave in the pipe), the
// issuing role in one lane altogether (its operands are not known to be uniform then, 2 to 3 times as long), polling instead of
// suspending waits (level), the second fetch of scores ahead of the first exponentials (-2 %).  The softmax alone takes 2746 cycles of
// the step's 2960 with the items' ends and the products with their copies 2586, so what helps one of them alone does not show.
//
// Every barrier wait is bounded (see sm100_ptx.cuh), and what a warp does next never depends on whether a wait ran out, so
// the named barriers always meet: a protocol error ends as a status word and a wrong answer, never as a hung GPU.

#include <type_traits>

#include "four_streams_sm100.cuh"
#include "host_sm100.cuh"
#include "sm100_ptx.cuh"
#include "softmax_tile_sm100.cuh"

namespace fray {
namespace sm100 {

// CTAS == 2: a CTA pair works on one item, every product is one cta_group::2 instruction of 256 rows, and each CTA holds half of
// K's rows and of V's columns.
template <int D, int STAGES, int CTAS = 1>
struct DuoCfg {
  static_assert(D == 64 || D == 128, "head dim must be 64 or 128");
  static_assert(CTAS == 1 || D == 128, "a CTA of a pair holds 64 head dims of V, one 128-byte panel");
  static_assert(STAGES >= 3 && STAGES <= 8, "3..8 K/V buffers");
  static constexpr int BM = 128, BN = 128;     // rows per query tile, keys per step
  static constexpr int kThreads = 640;
  // A half hands its 64 keys to the MMA warp in two chunks of 32, so that half of P.V runs while the second chunk is
  // still in its exponentials (chunks of 48 + 16 keys: level to 2 % slower).
  static constexpr int kPChunks = 2;
  static constexpr int kPanels = D / 64;       // 64-element (128-byte) column panels
  static constexpr int kQPanelBytes = BM * 128;
  static constexpr int kQTileBytes = kPanels * kQPanelBytes;
  static constexpr int kKVPanelBytes = BN * 128;
  static constexpr int kKVTileBytes = kPanels * kKVPanelBytes;
  static constexpr int kKRows = BN / CTAS;
  static constexpr int kKPanelBytes = kKRows * 128;
  static constexpr int kVPanels = kPanels / CTAS;
  static constexpr int kSlotBytes = kKVTileBytes / CTAS;
  // A pair's slots are half as large: six of them leave room for a staging tile per query tile, so that tile 1's end does not
  // wait for tile 0's store to have been read (eight slots and one staging tile: 1.5 % more cycles on 4 x 32 x 4096).
  static constexpr int kRing = CTAS == 2 ? 6 : STAGES;
  static constexpr int kStageTiles = CTAS == 2 ? 2 : 1;
  static constexpr int kOffQ = 0;
  static constexpr int kOffKV = 2 * kQTileBytes;
  static constexpr int kOffStage = kOffKV + kRing * kSlotBytes;  // O staging tile behind the ring, for both query tiles (a pair: one each)
  static constexpr int kOffBars = kOffStage + kStageTiles * kQTileBytes;
  static constexpr int kNumBars = 2 * 2 + 2 * kRing + 2 * 3 + 2 * kPChunks + 4;
  static constexpr int kOffStats = kOffBars + ((kNumBars * 8 + 16 + 127) / 128) * 128;  // [2 tiles][2 halves][128]
  static constexpr int kOffDeal = kOffStats + 4 * 128 * 4;
  // kDuoMatched (head dim 128): a CTA's items and the end mark, as many as shared memory has room for with four slots: 189 items a
  // CTA, 28 000 on 148 SMs (4 x 32 x 4096 has 2048), and 139 a pair.  Causal problems of more items are dealt slice by slice, at head
  // dim 64, too, where four streams deal by lists of their own: matched is level there (us, 28 000 to 37 000 items, slice by slice :
  // matched: 80 x 80 x 1280 2471 : 2473, 50 x 80 x 2048 3459 : 3464, 60 x 80/40 x 1792 3223 : 3188, 40 x 50 x 4096 6061 : 6096).
  static constexpr int kMaxDeal = CTAS == 2 ? 140 : 190;
  static constexpr int kUsedBytes = kOffDeal + (D == 128 ? kMaxDeal * 4 : 0);
  // slack for the forms that bring the dynamic segment to a 1024-byte boundary themselves (its base is one already; checked)
  static constexpr int kSmemBytes = kUsedBytes + 1024 <= 232448 ? kUsedBytes + 1024 : 232448;
  static_assert(kUsedBytes <= 232448, "exceeds the 227 KB shared memory of one CTA");
  static constexpr int kPartStride = D + 4;  // SPLIT: floats from row to row of the partial results
  static constexpr int kOffPartMl = 2 * BM * kPartStride * 4;
  static_assert(kOffPartMl + 2 * BM * 8 <= kOffStage, "the partial results fit Q and the ring");
  static constexpr int kTmemCols = 512;
  static constexpr uint32_t kColS0 = 0, kColS1 = 128, kColO0 = 256, kColO1 = 384;
  // Register budgets after setmaxnreg: per scheduler four softmax warps and one other, 4 x 104 + 64 = 5 x 96.
  static constexpr int kRegsLaunch = 96, kRegsSoftmax = 104, kRegsOther = 64;
  static constexpr int kRegsTotal = 512 * kRegsSoftmax + 128 * kRegsOther;
  static_assert(kRegsTotal <= kThreads * kRegsLaunch, "register budgets exceed the CTA's allocation");
};

// Meets the barrier and returns whether any of its threads passed `p`.
__device__ __forceinline__ bool named_barrier_or(int id, int threads, bool p) {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 p, %3, 0;\n"
      "barrier.cta.red.or.aligned.pred q, %1, %2, p;\n"
      "selp.u32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(r)
      : "r"(id), "r"(threads), "r"(static_cast<uint32_t>(p))
      : "memory");
  return r != 0;
}

// One step of half a row: 64 scores at t_s, the P chunks of 32 keys overwrite their head.
// p_bar: the first chunk's barrier, by pointer or by its cluster-wide address (of a pair, the leader's).
// my_max: this thread's slot for the exchange of maxima, the other half's is other_off floats away; pair_bar: the named
// barrier of the two warps that share the rows; lim (MASK): keys from lim on are past the end or above the diagonal.
// MOVE_ALL: when a row's offset has to move, the warp's other rows move theirs to their maxima too, as O is read and written for all 32
// anyway: fewer steps then have a row whose offset has to move.
template <bool MASK, bool MOVE_ALL, class Bar, class Rescale>
__device__ __forceinline__ void softmax_half(uint32_t t_s, Bar p_bar, float* my_max, int other_off, int pair_bar,
                                             Rescale&& rescale_o, int lim, float scale_log2, int lane,
                                             float& m_ref, float& l_run) {
  constexpr int kBarStep = std::is_pointer<Bar>::value ? 1 : 8;  // from a barrier to the next
  uint32_t sa[32], sb[32];
  tmem_ld_x32(t_s, sa);
  tmem_ld_x32(t_s + 32, sb);
  tmem_wait_ld();
  if constexpr (MASK) {
#pragma unroll
    for (int c = 0; c < 32; ++c) {
      if (c >= lim) sa[c] = __float_as_uint(-INFINITY);
      if (c + 32 >= lim) sb[c] = __float_as_uint(-INFINITY);
    }
  }
  const float mine = max_64(sa, sb);
  if (named_barrier_or(pair_bar, 64, (mine - m_ref) * scale_log2 > kRescaleThreshold)) {
    *my_max = mine;
    named_barrier_sync(pair_bar, 64);
    const float m_new = max3(mine, my_max[other_off], m_ref);
    float alpha = 1.f;
    if (MOVE_ALL ? m_new > m_ref : (m_new - m_ref) * scale_log2 > kRescaleThreshold) {
      // a row without any offset yet has nothing in O (its first product overwrites it)
      alpha = m_ref == -INFINITY ? 1.f : ex2_approx((m_ref - m_new) * scale_log2);
      l_run *= alpha;
      m_ref = m_new;
    }
    if (__any_sync(0xffffffffu, alpha != 1.f)) rescale_o(alpha);
  }
  const float neg_m = (m_ref == -INFINITY) ? 0.f : -m_ref * scale_log2;
  uint64_t rsp0 = 0ull, rsp1 = 0ull;
  const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2), neg_m2 = pack_f32x2(neg_m, neg_m);
  auto hand_over = [&](int q) {
    tmem_wait_st();
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) arrive_on(p_bar + q * kBarStep);
  };
  uint32_t pk[16];
  exp_32(sa, scale2, neg_m2, rsp0, rsp1, pk);
  tmem_st_x16(t_s, pk);
  tmem_ld_x32(t_s + 32, sb);
  hand_over(0);
  tmem_wait_ld();
  if constexpr (MASK) {
#pragma unroll
    for (int c = 0; c < 32; ++c)
      if (c + 32 >= lim) sb[c] = __float_as_uint(-INFINITY);
  }
  uint32_t pk2[16];
  exp_32(sb, scale2, neg_m2, rsp0, rsp1, pk2);
  tmem_st_x16(t_s + 16, pk2);
  hand_over(1);
  float r0, r1, r2, r3;
  unpack_f32x2(rsp0, r0, r1);
  unpack_f32x2(rsp1, r2, r3);
  l_run += (r0 + r1) + (r2 + r3);
}

// How a CTA comes by its items: dealt round by round; a part of one (SPLIT below); matched by twos (causal): an item and the one
// that has as many steps less than the middle of the slice as it has more.
enum DuoMode : int { kDuoDealt = 0, kDuoSplit = 1, kDuoMatched = 2 };

// One work item: two query tiles of slice (b, h) from row m0 on and the number of KV tiles each of them consumes, from tile j0 on
// (SPLIT; 0 otherwise).  A tile is 128 rows; of a CTA pair 256 rows, 128 in each CTA, or the same 128 rows of two heads (h: this
// CTA's) that share a K/V head.
struct DuoItem {
  int m0, b, h, n0, n1, j0;
};

// SPLIT: where the results go (the merge writes them with plain stores).
struct DuoOut {
  operand_t* o;
  long long sb, sh, ss;
};

// SPLIT, for problems of few items: a cluster of `parts` CTAs (blockIdx.x = item * parts + part) shares the KV tiles of one
// item and merges the partial results (fp32, 512 bytes a row and part) through each other's shared memory: no workspace, no
// second launch, no order between clusters.  One CTA per item left most of the chip idle, and its chain of steps set the time
// (1.75 us a step).  The merge takes 3.7 us among two CTAs, 5 among four.  us, one CTA per item -> split: 72 items x 47 steps
// 81 -> 50, 24 x 32 57 -> 26, 4 x 24 39 -> 13, 64 x 16 32 -> 24, 64 causal items of up to 32 steps 56 -> 37; head dim 64 71 ->
// 44, 50 -> 21, 33 -> 11, 28 -> 20, 50 -> 33.  Tried and left out: equal stretches of all items' steps for any number of CTAs,
// partial results in global memory, merged by whoever finds the others' written (9 us for the merge, and the steps 5 to 15 %
// slower, as the items' arithmetic took registers from them).
template <int D, int STAGES, DuoMode MODE, int CTAS>
__global__ void __launch_bounds__(640, 1)
attn_fwd_duo_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
                    int num_heads, int num_bh, int seq_len, int causal, float scale_log2, int kv_group, float* lse, int seq_k,
                    int heaviest_first, int n_kv, int n_pairs, int total, int parts, int pair_heads, const DuoOut out) {
  using Cfg = DuoCfg<D, STAGES, CTAS>;
  constexpr int BN = Cfg::BN;
  constexpr int RING = Cfg::kRing;
  constexpr bool SPLIT = MODE == kDuoSplit;
  static_assert(CTAS == 1 || !SPLIT, "a split item's clusters are of single CTAs");
  static_assert(MODE != kDuoMatched || D == 128, "head dim 64 has no room for a deal: four streams match its items");
  uint8_t* smem;
  bool fits;
  // Aligned by declaration every address in it is a constant, which the long items of the matched form and of pairs gain 1 % by
  // (1 x 32 x 16384 causal 1930 -> 1912 us); short items lose (3 x 32 x 826 on 184 keys 21.8 : 23.6, 6 x 16 x 333 causal 16.8 :
  // 17.5, split: 2 slices of 264 rows on 1913 keys 15.2 : 15.5), so the other forms round it up here.  Why they lose is not known.
  if constexpr (SPLIT || (D == 128 && MODE == kDuoDealt && CTAS == 1)) {
    extern __shared__ uint8_t duo_raw[];
    const uint32_t raw_addr = smem_u32(duo_raw);
    const uint32_t align_off = ((raw_addr + 1023u) & ~1023u) - raw_addr;
    smem = duo_raw + align_off;
    fits = align_off + Cfg::kUsedBytes <= Cfg::kSmemBytes;
  } else {
    extern __shared__ __align__(1024) uint8_t duo_smem[];
    smem = duo_smem;
    fits = (opaque(smem_u32(smem)) & 1023u) == 0;
  }
  uint8_t* q_smem = smem + Cfg::kOffQ;
  uint8_t* kv_smem = smem + Cfg::kOffKV;
  uint8_t* stage_smem = smem + Cfg::kOffStage;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBars);
  // Of a pair, the barriers that both CTAs' threads or copies arrive on are the leader's (rank 0, whose warp 16 issues for both).
  uint64_t* q_full = bars;                      // [2]   producer -> MMA
  uint64_t* q_free = bars + 2;                  // [2]   MMA -> producer  (the item's last S of tile i has read Q_i)
  uint64_t* kv_full = bars + 4;                 // [RING] producer -> MMA
  uint64_t* kv_empty = kv_full + RING;          // [RING] MMA -> producer
  uint64_t* s_full = kv_empty + RING;           // [2]   MMA -> softmax i
  uint64_t* o_full = s_full + 2;                // [2]   MMA -> softmax i (the item's last P.V)
  uint64_t* o_free = o_full + 2;                // [2]   softmax i -> MMA (the item's O_i is in registers)
  uint64_t* p_full = o_free + 2;                // [2][kPChunks] softmax i -> MMA
  uint64_t* stage_full = p_full + 2 * Cfg::kPChunks;  // [kStageTiles] softmax -> store warp
  uint64_t* stage_free = stage_full + 2;        // [2]   store warp -> softmax i (the staging tile is tile i's turn)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::kNumBars);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);
  float* stats = reinterpret_cast<float*>(smem + Cfg::kOffStats);

  const uint32_t* deal = reinterpret_cast<const uint32_t*>(smem + Cfg::kOffDeal);
  float* part_o = reinterpret_cast<float*>(smem);  // SPLIT: partial results, in place of Q and the ring
  float2* part_ml = reinterpret_cast<float2*>(smem + Cfg::kOffPartMl);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;

  if (!fits) {  // never seen: the segment's base is 1024-byte aligned
    if (tid == 0) atomicCAS(&fray_attn_status[0], 0, 0x601);
    return;
  }

  const int rank = CTAS == 2 ? static_cast<int>(cluster_ctarank()) : 0;
  const int unit = static_cast<int>(blockIdx.x) / CTAS;
  const int stride = static_cast<int>(gridDim.x) / CTAS;
  // Rows from a query tile to the next, and from a tile's first row to this CTA's; heads that an item takes.
  const int tile_rows = CTAS == 2 && !pair_heads ? 2 * Cfg::BM : Cfg::BM;
  const int row_off = CTAS == 2 && !pair_heads ? rank * Cfg::BM : 0;
  const int item_heads = CTAS == 2 && pair_heads ? 2 : 1;
  const int part = SPLIT ? static_cast<int>(blockIdx.x) % parts : 0;
  // Items are numbered slice by slice (CTAs that run side by side share a slice's K and V in L2) or, with a causal mask and
  // by duo_heaviest_first, pair by pair, the heaviest of all slices first.  CTA (CTA pair) c takes the positions c, G + c, ...;
  // with a causal mask the direction alternates from round to round, which evens out most of what is left.
  auto pos = [&](int k) {
    const int c = unit;
    if constexpr (SPLIT) return c / parts;  // its only one
    if constexpr (MODE == kDuoMatched) return static_cast<int>(deal[k]);
    return k * stride + ((causal && (k & 1)) ? stride - 1 - c : c);  // >= total: the CTA is done; grows with k
  };
  auto decode = [&](int idx) {
    DuoItem it;
    const int run = heaviest_first ? num_bh / item_heads : n_pairs;
    const int hi = idx / run;
    const int lo = idx - hi * run;
    const int bh = heaviest_first ? lo : hi;
    const int pr = heaviest_first ? hi : lo;
    const int pair = causal ? (n_pairs - 1 - pr) : pr;
    it.m0 = pair * (2 * tile_rows);
    it.b = bh * item_heads / num_heads;
    it.h = bh * item_heads - it.b * num_heads + (item_heads > 1 ? rank : 0);
    int n[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row0 = it.m0 + i * tile_rows;
      n[i] = row0 < seq_len ? n_kv : 0;
      if (causal && n[i] > 0) {
        const int lim = (row0 + tile_rows + BN - 1) / BN;
        n[i] = lim < n[i] ? lim : n[i];
      }
    }
    it.n0 = n[0];
    it.n1 = n[1];
    it.j0 = 0;
    if constexpr (SPLIT) {  // the step that only a causal item's tile 1 has goes with tile 0's last one
      it.j0 = n[0] * part / parts;
      const int end = n[0] * (part + 1) / parts;
      it.n0 = end - it.j0;
      it.n1 = n[1] == 0 || it.n0 == 0 ? 0 : (end == n[0] ? n[1] : end) - it.j0;
    }
    return it;
  };

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(q_full + i, 1);
      mbar_init(q_free + i, 1);
      mbar_init(s_full + i, 1);
      for (int c = 0; c < Cfg::kPChunks; ++c) mbar_init(p_full + i * Cfg::kPChunks + c, 8 * CTAS);
      mbar_init(o_full + i, 1);
      mbar_init(o_free + i, 8 * CTAS);
    }
    for (int s = 0; s < RING; ++s) {
      mbar_init(kv_full + s, 1);
      mbar_init(kv_empty + s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(stage_full + i, 8);
      mbar_init(stage_free + i, 1);
    }
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols, CtaGroup<CTAS>{});
    tmem_relinquish(CtaGroup<CTAS>{});
  }
  if constexpr (MODE == kDuoMatched) {
    // worked out once, as in the roles it took registers from the KV loop
    for (int k = tid - 64; k >= 0 && k < Cfg::kMaxDeal; k += Cfg::kThreads - 64)
      reinterpret_cast<uint32_t*>(smem + Cfg::kOffDeal)[k] = matched_item(k, stride, unit, n_pairs, total);
  }
  grid_dependency_wait();
  if (tid == 32) *abort_flag = (*reinterpret_cast<volatile int*>(&fray_attn_status[0]) != 0) ? 2u : 0u;
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  grid_launch_dependents();
  const uint32_t tmem_base = *tmem_slot;
  // An earlier launch left the device status raised: nothing is computed (SPLIT: the cluster's barriers have to be met).
  bool dead = *abort_flag == 2u;
  if constexpr (CTAS == 2) {
    // The barriers of both CTAs exist before anything arrives on them, and both agree on whether to run.
    cluster_sync_all();
    dead |= ld_shared_cluster_u32(mapa_shared(smem_u32(const_cast<uint32_t*>(abort_flag)), rank ^ 1)) == 2u;
    cluster_sync_all();  // the peer has read this CTA's flag before anything may raise it
  }
  auto leader = [&](uint64_t* bar) { return CTAS == 2 ? mapa_shared(smem_u32(bar), 0) : smem_u32(bar); };
  if (!SPLIT && dead) {
    if (warp == 0) tmem_dealloc(tmem_base, Cfg::kTmemCols, CtaGroup<CTAS>{});
    return;
  }
  const int idx_end = SPLIT && dead ? 0 : total;

  if (warp < 16) {
    // =============================================================== softmax
    set_max_regs_inc<Cfg::kRegsSoftmax>();
    const int i = (warp >> 2) & 1;  // query tile
    const int hf = warp >> 3;       // which 64 keys of a step, which D / 2 columns of O
    const int r = tid & 127;        // row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t t_s = tmem_base + (i == 0 ? Cfg::kColS0 : Cfg::kColS1) + hf * 64 + lane_base;
    const uint32_t t_o = tmem_base + (i == 0 ? Cfg::kColO0 : Cfg::kColO1) + hf * (D / 2) + lane_base;
    // At head dim 128 the loop's barriers go by 32-bit addresses that are worked out once; by pointers, which are converted where
    // they are used, 1 to 3 % slower (us, behind lasting load: 4 x 32 x 4096 977 : 960, causal 548 : 534, 1 x 32 x 16384 causal
    // 1933 : 1904; as a pair 977 : 941).  At head dim 64 it is the other way round (8 x 16 x 4096 715 : 728, 16 x 16 x 1024 107.6 : 110).
    auto bar_ref = [&](uint64_t* bar) {
      if constexpr (D == 64 || SPLIT) return bar;
      else return leader(bar);
    };
    const auto p_bar = bar_ref(p_full + i * Cfg::kPChunks);
    const uint32_t s_bar = smem_u32(s_full + i);
    float* my_stat = stats + (i * 2 + hf) * 128 + r;
    const int other_off = hf ? -128 : 128;
    const int pair_bar = 1 + i * 4 + (warp & 3);
    // In a pair a row that moves its offset holds up 16 warps instead of 8: with wide scores, where one does in most steps, pairs with
    // the code of single CTAs lost 3 % by rows and 2 % by heads to single CTAs.  So all rows of the warp move at a time and O goes
    // through registers in two pieces; its stores are waited for with those of P (softmax_half).  us, single CTAs : pairs as they
    // were : now, wide scores, behind lasting load: 7 x 8 x 4046 on 6058 752 : 787 : 755, 9 x 12 x 5029 1421 : 1480 : 1431, causal by
    // heads 9 x 16/2 x 5161 1054 : 1083 : 1049; scores of unit variance level.
    auto rescale_o = [&](float alpha) {
      if constexpr (CTAS == 2) {
#pragma unroll 1
        for (int c = 0; c < D / 2; c += 32) {
          uint32_t orr[32];
          tmem_ld_x32(t_o + c, orr);
          tmem_wait_ld();
#pragma unroll
          for (int x = 0; x < 32; ++x) orr[x] = __float_as_uint(__uint_as_float(orr[x]) * alpha);
          tmem_st_x32(t_o + c, orr);
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < D / 2; c += 16) {
          uint32_t orr[16];
          tmem_ld_x16(t_o + c, orr);
          tmem_wait_ld();
#pragma unroll
          for (int x = 0; x < 16; ++x) orr[x] = __float_as_uint(__uint_as_float(orr[x]) * alpha);
          tmem_st_x16(t_o + c, orr);
        }
        tmem_wait_st();
      }
    };
    // phase parities, toggled: bit 0 s_full, bit 1 o_full, bit 2 stage_free
    uint32_t phases = 0;
    auto wait_scores = [&](int j) __attribute__((always_inline)) {
      if constexpr (D == 64 || SPLIT) mbar_wait(s_full + i, phases & 1, abort_flag, 0x201 + i, j);
      else mbar_wait(s_bar, phases & 1, abort_flag, 0x201 + i, j);
    };
    for (int k = 0, idx = pos(0); idx < idx_end; idx = SPLIT ? idx_end : pos(++k)) {
      int n_i, n_full, lim;
      {
        const DuoItem it = decode(idx);
        n_i = i ? it.n1 : it.n0;
        if (n_i == 0) continue;
        const int row = it.m0 + i * tile_rows + row_off;
        // the first steps see every key of their tile
        n_full = seq_k / BN;
        if (causal) n_full = (row + 1) / BN < n_full ? (row + 1) / BN : n_full;
        if constexpr (SPLIT) n_full = n_full > it.j0 ? n_full - it.j0 : 0;
        if (n_full > n_i) n_full = n_i;
        lim = (causal && row + r + 1 < seq_k ? row + r + 1 : seq_k) - hf * 64 - (it.j0 + n_full) * BN;  // keys the row may see from there
      }
      float m_ref = -INFINITY;
      float l_run = 0.f;
      for (int j = 0; j < n_full; ++j) {
        wait_scores(j);
        tc_fence_after_sync();
        softmax_half<false, CTAS == 2>(t_s, p_bar, my_stat, other_off, pair_bar, rescale_o, 0, scale_log2, lane, m_ref, l_run);
        phases ^= 1u;
      }
      for (int j = n_full; j < n_i; ++j, lim -= BN) {
        wait_scores(j);
        tc_fence_after_sync();
        softmax_half<true, CTAS == 2>(t_s, p_bar, my_stat, other_off, pair_bar, rescale_o, lim, scale_log2, lane, m_ref, l_run);
        phases ^= 1u;
      }
      // The slots carried maxima up to the last step, whose exchange ends with a read of the partner's: both warps have to
      // be past it before a row sum takes a maximum's place.
      named_barrier_sync(pair_bar, 64);
      *my_stat = l_run;
      named_barrier_sync(pair_bar, 64);
      l_run += my_stat[other_off];  // the next write to a slot comes behind the next step's OR barrier
      if constexpr (SPLIT) {
        // Q and the ring give way to the partial results once both tiles' products have read them.
        mbar_wait(o_full, 0, abort_flag, 0x331, idx);
        if (decode(idx).n1 > 0) mbar_wait(o_full + 1, 0, abort_flag, 0x332, idx);
        tc_fence_after_sync();
#pragma unroll
        for (int c = 0; c < D / 2; c += 32) {
          uint32_t orr[32];
          tmem_ld_x32(t_o + c, orr);
          tmem_wait_ld();
          float* to = part_o + (i * Cfg::BM + r) * Cfg::kPartStride + hf * (D / 2) + c;
#pragma unroll
          for (int x = 0; x < 32; x += 4) *reinterpret_cast<uint4*>(to + x) = make_uint4(orr[x], orr[x + 1], orr[x + 2], orr[x + 3]);
        }
        if (hf == 0) part_ml[i * Cfg::BM + r] = make_float2(m_ref, l_run);
        continue;
      }
      // The tile's turn at the staging buffer.  Each tile has a barrier of its own and meets every phase of it once: phase
      // j completes when the store in front of the tile's j-th one has been read, and phase j + 1 not before the tile's
      // j-th store, which needs all eight warps past this wait.  So the parity says whether phase j is complete whatever
      // the store warp's delay; on one barrier for both tiles a wait could look over an open phase or miss two.
      mbar_wait(stage_free + i, (phases >> 2) & 1, abort_flag, 0x321 + i, idx);
      phases ^= 4u;
      mbar_wait(o_full + i, (phases >> 1) & 1, abort_flag, 0x331 + i, idx);
      phases ^= 2u;
      tc_fence_after_sync();
      const float inv_l = l_run > 0.f ? 1.f / l_run : 1.f;
#pragma unroll
      for (int c = 0; c < D / 2; c += 32) {
        uint32_t orr[32];
        tmem_ld_x32(t_o + c, orr);
        tmem_wait_ld();
        if (c + 32 == D / 2) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) arrive_on(bar_ref(o_free + i));
        }
        const int col = hf * (D / 2) + c;  // first column of these 32
        uint8_t* panel_row = stage_smem + (Cfg::kStageTiles == 2 ? i * Cfg::kQTileBytes : 0) + (col >> 6) * Cfg::kQPanelBytes + r * 128;
#pragma unroll
        for (int x = 0; x < 32; x += 8) {
          uint4 v4;
          v4.x = pack_half2(__uint_as_float(orr[x + 0]) * inv_l, __uint_as_float(orr[x + 1]) * inv_l);
          v4.y = pack_half2(__uint_as_float(orr[x + 2]) * inv_l, __uint_as_float(orr[x + 3]) * inv_l);
          v4.z = pack_half2(__uint_as_float(orr[x + 4]) * inv_l, __uint_as_float(orr[x + 5]) * inv_l);
          v4.w = pack_half2(__uint_as_float(orr[x + 6]) * inv_l, __uint_as_float(orr[x + 7]) * inv_l);
          const int chunk = ((col & 63) + x) >> 3;  // 16-byte chunk inside the 128-byte row
          *reinterpret_cast<uint4*>(panel_row + ((chunk ^ (r & 7)) << 4)) = v4;
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(stage_full + (Cfg::kStageTiles == 2 ? i : 0));
      if (lse != nullptr && hf == 0) {
        int again = idx;
        asm volatile("" : "+r"(again));  // worked out again here instead of kept through the steps
        const DuoItem it = decode(again);
        const int row = it.m0 + i * tile_rows + row_off + r;
        if (row < seq_len)
          lse[(static_cast<size_t>(it.b) * num_heads + it.h) * seq_len + row] =
              l_run > 0.f ? (m_ref * scale_log2 + log2f(l_run)) * 0.69314718055994531f : -INFINITY;
      }
    }
    if constexpr (SPLIT) {
      // Merge: every CTA of the cluster adds up a share of the item's rows.  Here and not behind the roles, where the other
      // warps' smaller register budget would hold.
      __syncwarp();
      cluster_sync_all();
      if (!dead) {
        const DuoItem it = decode(static_cast<int>(blockIdx.x) / parts);
        const int diagonal = (it.m0 + Cfg::BM + BN - 1) / BN, units = causal && diagonal < n_kv ? diagonal : n_kv;
        const int rows = seq_len - it.m0 < 2 * Cfg::BM ? seq_len - it.m0 : 2 * Cfg::BM;
        const uint32_t o_addr = smem_u32(part_o), ml_addr = smem_u32(part_ml);
        // This CTA's rows: [row_lo, row_lo + mine).
        const int row_lo = rows * part / parts, mine = rows * (part + 1) / parts - row_lo;
        uint32_t has = 0;  // parts with any step: the others have left nothing (whatever their shared memory held)
        for (int p = 0; p < parts; ++p) has |= static_cast<uint32_t>(units * p / parts < units * (p + 1) / parts) << p;
        // One thread per row: the parts' weights, over the row sum.
        float* weights = stats;  // [parts][mine], parts * mine <= rows + parts, in place of the 512 slots for maxima and row sums
        if (tid < mine) {
          float m[kMaxClusterCtas], l[kMaxClusterCtas];
          float m_all = -INFINITY, l_all = 0.f;
#pragma unroll
          for (int p = 0; p < kMaxClusterCtas; ++p) {
            float2 ml = make_float2(-INFINITY, 0.f);
            if ((has >> p) & 1u) ml = ld_cluster_f2(mapa_shared(ml_addr, p) + (row_lo + tid) * 8);
            m[p] = ml.x;
            l[p] = ml.y;
          }
#pragma unroll
          for (int p = 0; p < kMaxClusterCtas; ++p) m_all = fmaxf(m_all, m[p]);
          const float m_safe = m_all == -INFINITY ? 0.f : m_all;  // no key at all: every weight is 0
#pragma unroll
          for (int p = 0; p < kMaxClusterCtas; ++p) {
            m[p] = ex2_approx((m[p] - m_safe) * scale_log2);
            l_all = fmaf(l[p], m[p], l_all);
          }
          const float inv_l = l_all > 0.f ? 1.f / l_all : 1.f;
#pragma unroll
          for (int p = 0; p < kMaxClusterCtas; ++p)
            if (p < parts) weights[p * mine + tid] = m[p] * inv_l;
          if (lse != nullptr)
            lse[(static_cast<size_t>(it.b) * num_heads + it.h) * seq_len + it.m0 + row_lo + tid] =
                l_all > 0.f ? (m_all * scale_log2 + log2f(l_all)) * 0.69314718055994531f : -INFINITY;
        }
        named_barrier_sync(9, 512);
        // A warp takes 4 rows at a time (head dim 64: half a warp to a row, 8), a lane 16 bytes of each, and fetches two parts of
        // them together: a load from another SM takes some hundred cycles.
        constexpr int kLanes = D / 4, kRowsPerLoad = 32 / kLanes, kRows = 4;
        const int c4 = lane % kLanes, sub = lane / kLanes;
        for (int r0 = warp * kRows * kRowsPerLoad; r0 < mine; r0 += 16 * kRows * kRowsPerLoad) {
          float4 acc[kRows];
          int at[kRows];
#pragma unroll
          for (int x = 0; x < kRows; ++x) {
            acc[x] = make_float4(0.f, 0.f, 0.f, 0.f);
            at[x] = min(r0 + x * kRowsPerLoad + sub, mine - 1);
          }
          for (int p0 = 0; p0 < parts; p0 += 2) {
            float4 v[2][kRows];
            float w[2][kRows];
#pragma unroll
            for (int a = 0; a < 2; ++a) {
              int p = part + (p0 + a < parts ? p0 + a : p0);  // each CTA begins with its own: not all of them at one SM's memory
              if (p >= parts) p -= parts;
              const bool counts = p0 + a < parts && ((has >> p) & 1u);
              const uint32_t from = mapa_shared(o_addr, p);
#pragma unroll
              for (int x = 0; x < kRows; ++x) {
                v[a][x] = counts ? ld_cluster_f4(from + ((row_lo + at[x]) * Cfg::kPartStride + c4 * 4) * 4)
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
                w[a][x] = weights[p * mine + at[x]];
              }
            }
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
              for (int x = 0; x < kRows; ++x) {
                acc[x].x = fmaf(v[a][x].x, w[a][x], acc[x].x);
                acc[x].y = fmaf(v[a][x].y, w[a][x], acc[x].y);
                acc[x].z = fmaf(v[a][x].z, w[a][x], acc[x].z);
                acc[x].w = fmaf(v[a][x].w, w[a][x], acc[x].w);
              }
          }
#pragma unroll
          for (int x = 0; x < kRows; ++x)
            if (r0 + x * kRowsPerLoad + sub < mine)
              *reinterpret_cast<uint2*>(out.o + it.b * out.sb + it.h * out.sh + (it.m0 + row_lo + at[x]) * out.ss + c4 * 4) =
                  make_uint2(pack_half2(acc[x].x, acc[x].y), pack_half2(acc[x].z, acc[x].w));
        }
      }
    }
  } else {
    set_max_regs_dec<Cfg::kRegsOther>();
    if (!SPLIT && warp == 18 && lane == 0) {
      // ============================================================= stores of finished tiles
      uint32_t stores = 0;      // parity of the stores from each staging tile
      mbar_arrive(stage_free);  // the first store is a tile 0's (every item has one)
      if (Cfg::kStageTiles == 2) mbar_arrive(stage_free + 1);
      for (int k = 0, idx = pos(0); idx < idx_end; idx = SPLIT ? idx_end : pos(++k)) {
        const DuoItem it = decode(idx);
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          if ((i ? it.n1 : it.n0) == 0) continue;
          const int tile = Cfg::kStageTiles == 2 ? i : 0;
          mbar_wait(stage_full + tile, (stores >> tile) & 1, abort_flag, 0x341 + i, idx);
          stores ^= 1u << tile;
          if (*abort_flag != 0) break;
          const int row0 = it.m0 + i * tile_rows + row_off;
          if (CTAS == 1 || row0 < seq_len) {  // of a pair's tile, the second CTA's rows may all be past the last query
#pragma unroll
            for (int p = 0; p < Cfg::kPanels; ++p)
              tma_store_4d(&tm_o, stage_smem + tile * Cfg::kQTileBytes + p * Cfg::kQPanelBytes, p * 64, row0, it.h, it.b);
            tma_store_commit();
            tma_store_wait_read();
          }
          // whose store comes next: with one staging tile, this item's tile 1 or an item's tile 0
          mbar_arrive(stage_free + (Cfg::kStageTiles == 2 ? i : (i == 0 && it.n1 > 0)));
        }
      }
    } else if (warp == 17 && lane == 0) {
      // ============================================================= TMA producer
      uint32_t t_run = 0;               // K/V tiles loaded so far: ring slot and phase
      uint32_t q_cnt0 = 0, q_cnt1 = 0;  // items whose Q_0 / Q_1 this CTA has loaded
      for (int k = 0, idx = pos(0); idx < idx_end; idx = SPLIT ? idx_end : pos(++k)) {
        const DuoItem it = decode(idx);
        const int h_kv = it.h / kv_group;
        const int n_max = it.n0 > it.n1 ? it.n0 : it.n1;
        auto load = [&](void* dst, const CUtensorMap* tm, uint64_t* bar, int c0, int c1, int c2, int c3) __attribute__((always_inline)) {
          if constexpr (CTAS == 2) tma_load_4d_pair(dst, tm, leader(bar), c0, c1, c2, c3);
          else tma_load_4d(dst, tm, bar, c0, c1, c2, c3);
        };
        auto load_q = [&](int i) __attribute__((always_inline)) {
          if ((i ? it.n1 : it.n0) > 0) {
            const uint32_t cnt = i ? q_cnt1 : q_cnt0;
            if (cnt > 0) mbar_wait(q_free + i, (cnt - 1) & 1, abort_flag, 0x402 + i, idx);
            if (rank == 0) mbar_expect_tx(q_full + i, CTAS * Cfg::kQTileBytes);
#pragma unroll
            for (int p = 0; p < Cfg::kPanels; ++p)
              load(q_smem + i * Cfg::kQTileBytes + p * Cfg::kQPanelBytes, &tm_q, q_full + i, p * 64,
                   it.m0 + i * tile_rows + row_off, it.h, it.b);
            if (i) ++q_cnt1; else ++q_cnt0;
          }
        };
        load_q(0);
        for (int t = 0; t < 2 * n_max; ++t) {
          const int slot = t_run % RING;
          const uint32_t ph = (t_run / RING) & 1;
          mbar_wait(kv_empty + slot, ph ^ 1, abort_flag, 0x401, t);
          if (*abort_flag != 0) break;
          if (rank == 0) mbar_expect_tx(kv_full + slot, Cfg::kKVTileBytes);
          uint8_t* dst = kv_smem + slot * Cfg::kSlotBytes;
          const int row = (it.j0 + (t >> 1)) * BN;
          if (t & 1) {
#pragma unroll
            for (int p = 0; p < Cfg::kVPanels; ++p)
              load(dst + p * Cfg::kKVPanelBytes, &tm_v, kv_full + slot, (rank * Cfg::kVPanels + p) * 64, row, h_kv, it.b);
          } else {
#pragma unroll
            for (int p = 0; p < Cfg::kPanels; ++p)
              load(dst + p * Cfg::kKPanelBytes, &tm_k, kv_full + slot, p * 64, row + rank * Cfg::kKRows, h_kv, it.b);
          }
          ++t_run;
          if (t == 0) load_q(1);
        }
        if (*abort_flag != 0) break;
      }
    } else if (warp == 16 && rank == 0) {
      // ============================================================= MMA issue (whole warp, one elected lane issues)
      constexpr uint64_t kDescK = smem_desc_sw128(16, 1024);
      constexpr uint64_t kDescV = smem_desc_sw128(Cfg::kKVPanelBytes, 1024);
      constexpr uint32_t kIdescQK = idesc_f16_f32(CTAS * Cfg::BM, BN, false, false);
      constexpr uint32_t kIdescPV = idesc_f16_f32(CTAS * Cfg::BM, D, false, true);
      const uint32_t q_addr = smem_u32(q_smem);
      const uint32_t kv_addr = smem_u32(kv_smem);
      // One copy of the issue code per query tile (constant descriptors and columns) or one for both.  One elected lane issues
      // a whole product; electing a lane for every instruction, with its operands through opaque registers, kept the warp
      // busy for 1600 cycles per product pair and tile, longer than the tensor pipe (1024) and than the chain through the
      // softmax needs: 3200 -> 2870 cycles per 128 keys of two tiles.  us, 20 launches from an idle board / behind 150 ms
      // of load: 4 x 32 x 4096 x 128 848 / 962 -> 823 / 935 with a copy each, 847 / 964 with one for both; causal 497 /
      // 564 -> 477 / 541; 8 x 16 x 4096 x 64 661 / 700 -> 657 / 705 with a copy each, 648 / 695 with one for both.
      constexpr int kIssueCopies = D == 128 ? 2 : 1;
      // phase parities of tile 0 / 1: bits 0, 1 p_full; bits 2, 3 q_full; bits 4, 5 o_free (parity 1 at first: the
      // accumulators are free)
      uint32_t phases = 0x30;

      // read from lane 0, so that the compiler knows it to be the same in all lanes
      const uint32_t tmem_cols = __shfl_sync(0xffffffffu, tmem_base, 0);
      auto wait_kv = [&](uint32_t t_abs, int j) __attribute__((always_inline)) {
        mbar_wait(kv_full + t_abs % RING, (t_abs / RING) & 1, abort_flag, 0x501, j);
      };
      // S_i(j) = Q_i . K_j^T of item `it` (ring index t_abs)
      auto issue_qk = [&](int i, const DuoItem& it, int j, uint32_t t_abs) __attribute__((always_inline)) {
        const int slot = t_abs % RING;
        tc_fence_after_sync();
        const uint64_t q_d = smem_desc_at(kDescK, q_addr + i * Cfg::kQTileBytes);
        const uint64_t k_d = smem_desc_at(kDescK, kv_addr + slot * Cfg::kSlotBytes);
        const uint32_t t_s = tmem_cols + (i == 0 ? Cfg::kColS0 : Cfg::kColS1);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t qoff = ((kk >> 2) * Cfg::kQPanelBytes + (kk & 3) * 32) >> 4;
            const uint32_t koff = ((kk >> 2) * Cfg::kKPanelBytes + (kk & 3) * 32) >> 4;
            mma_ss_g<CTAS>(t_s, q_d + qoff, k_d + koff, kIdescQK, kk > 0);
          }
          mma_commit_g<CTAS>(s_full + i);
          if ((i == 1) || !(j < it.n1)) mma_commit_g<CTAS>(kv_empty + slot);
          if (j + 1 == (i ? it.n1 : it.n0)) mma_commit_g<CTAS>(q_free + i);
        }
        __syncwarp();
      };
      auto issue_pv = [&](int i, const DuoItem& it, int j, uint32_t t_abs) __attribute__((always_inline)) {
        const int slot = t_abs % RING;
        const bool last = j + 1 == (i ? it.n1 : it.n0);
        wait_kv(t_abs, j);
        if (j == 0) {
          // the first product of an item overwrites O: the previous item's epilogue must have read it
          mbar_wait(o_free + i, (phases >> (4 + i)) & 1, abort_flag, 0x507 + i, j);
          phases ^= 0x10u << i;
        }
        if (!last) wait_kv(t_abs + 1, j);  // the next K tile: ahead of P, off the path to the next scores
        const uint64_t v_d = smem_desc_at(kDescV, kv_addr + slot * Cfg::kSlotBytes);
        const uint32_t t_p = tmem_cols + (i == 0 ? Cfg::kColS0 : Cfg::kColS1);
        const uint32_t t_o = tmem_cols + (i == 0 ? Cfg::kColO0 : Cfg::kColO1);
        const uint32_t ph = (phases >> i) & 1;
#pragma unroll
        for (int q = 0; q < Cfg::kPChunks; ++q) {
          mbar_wait(p_full + i * Cfg::kPChunks + q, ph, abort_flag, 0x503 + i, j);
          tc_fence_after_sync();
          if (elect_one()) {
#pragma unroll
            for (int s2 = 0; s2 < 4; ++s2) {
              // 16 keys per MMA: the chunk's 32 keys of either half; a half's P sits in columns [0,32) / [64,96)
              const int kk = (s2 >> 1) * 4 + q * 2 + (s2 & 1);
              mma_ts_g<CTAS>(t_o, t_p + (kk >> 2) * 64 + (kk & 3) * 8, v_d + ((kk * 2048) >> 4), kIdescPV, (j > 0 || q > 0 || s2 > 0));
            }
            if (q == Cfg::kPChunks - 1) {
              if (last) mma_commit_g<CTAS>(o_full + i);
              if ((i == 1) || !(j < it.n1)) mma_commit_g<CTAS>(kv_empty + slot);
            }
          }
          __syncwarp();
        }
        phases ^= 1u << i;
      };
      auto first_qk = [&](int i, const DuoItem& it, uint32_t t_abs) __attribute__((always_inline)) {
        mbar_wait(q_full + i, (phases >> (2 + i)) & 1, abort_flag, 0x511 + i);
        phases ^= 4u << i;
        wait_kv(t_abs, 0);
        issue_qk(i, it, 0, t_abs);
      };

      int k = 0;
      const int idx = pos(0);
      if (idx < idx_end && decode(idx).n0 > 0) {
        DuoItem cur = decode(idx);
        uint32_t t_base = 0;  // ring index of the current item's K_0
#pragma unroll 1
        for (int i = 0; i < 2; ++i)
          if ((i ? cur.n1 : cur.n0) > 0) first_qk(i, cur, t_base);
        while (true) {
          const int idx_next = SPLIT ? idx_end : pos(k + 1);
          const bool has_next = idx_next < idx_end;
          DuoItem nxt = cur;
          nxt.n0 = 0;
          nxt.n1 = 0;
          if (has_next) nxt = decode(idx_next);
          const int n_max = cur.n0 > cur.n1 ? cur.n0 : cur.n1;
          const uint32_t t_next = t_base + 2 * n_max;
          for (int j = 0; j < n_max; ++j) {
#pragma unroll kIssueCopies
            for (int i = 0; i < 2; ++i) {
              const int n_i = i ? cur.n1 : cur.n0;
              if (j < n_i) {
                issue_pv(i, cur, j, t_base + 2 * j + 1);
                if (j + 1 < n_i) {
                  issue_qk(i, cur, j + 1, t_base + 2 * (j + 1));
                } else if ((i ? nxt.n1 : nxt.n0) > 0 && (i == 1 || cur.n0 == cur.n1)) {
                  first_qk(i, nxt, t_next);  // the next item's first scores, right behind this item's last P.V
                }
              }
            }
            // A tile 0 that ends a step before tile 1: its next first scores go behind tile 1's product of this
            // step, which hands back the ring slot the next item's K_0 needs.
            if (cur.n0 != cur.n1 && j + 1 == cur.n0 && nxt.n0 > 0) first_qk(0, nxt, t_next);
          }
          // a tile that had nothing to do in this item (past the last query) but has in the next
#pragma unroll 1
          for (int i = 0; i < 2; ++i)
            if ((i ? cur.n1 : cur.n0) == 0 && (i ? nxt.n1 : nxt.n0) > 0) first_qk(i, nxt, t_next);
          if (!has_next) break;
          cur = nxt;
          t_base = t_next;
          ++k;
        }
      }
    }
    if constexpr (SPLIT) {
      __syncwarp();
      cluster_sync_all();
    }
  }

  if (*abort_flag == 1u) settle_after_abort();
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (CTAS == 2) cluster_sync_all();  // neither CTA leaves while the other may still signal it
  if (warp == 0) tmem_dealloc(tmem_base, Cfg::kTmemCols, CtaGroup<CTAS>{});
  if constexpr (SPLIT) {
    __syncwarp();
    cluster_sync_all();  // shared memory stays until every CTA has read it
  }
}

// Item order of a causal problem.  The deal is fixed, so slice by slice the busiest CTA has 6 to 60 % more than its share, and
// heaviest first evens that out; but it has all slices under way at once, and once their K and V outgrow L2 (126 MB) every item
// fetches them from HBM, at the price of clock under the board's power limit.  Heaviest first : slice by slice, us, each
// behind 120 ms of its own load (a first version of this comparison, the two in turn, had them share one clock and showed
// heaviest first ahead throughout): 1 x 32 heads on 8 x 3000 x 128 (12 MB) 88 : 109 (the one-tile kernel 100), 2 x 32 on 8 x
// 3000 163 : 175, 4 x 16 x 2048 (67 MB) 86 : 90, 1 x 16 x 8192 (67 MB) 274 : 350, 3 x 16 x 4096 (101 MB) 227 : 247, 64-wide
// heads 2 x 32 x 3000 (49 MB) 123 : 131; 1 % behind at worst.  From 134 MB on: 4 x 32 x 2048 177 : 170, 3 x 32 x 3000 (147
// MB) 278 : 259, 4 x 32 x 4096 (268 MB) 645 : 580, 8 x 32 on 8 x 4096 (134 MB) 1135 : 1095; with few long slices still ahead
// a little further: 1 x 16 x 16384 (134 MB) 1030 : 1110, 1 x 32 x 8192 (134 MB) 545 : 555, but 1 x 32 x 16384 (268 MB) 2117 :
// 2085.  Up to 1024 rows a slice's few items run side by side anyway: 2 % behind to 2 % ahead in most of 16 shapes.
inline bool duo_heaviest_first(bool causal, const AttnShape& shp, const AttnShape& shp_kv) {
  const long long kv_bytes = 2LL * shp_kv.B * shp_kv.H * shp_kv.S * shp_kv.D * 2;
  return causal && shp.S > 1024 && kv_bytes <= (shp.S >= 8192 ? kHeaviestFirstMaxKvBytes : 126LL * 1000 * 1000);
}

// Slice by slice the busiest CTA of a causal problem has 6 to 25 % more steps than its share.  Matched by twos every CTA has the
// same number of steps per round of two items, and what is left is the incomplete last round: taken where that is 13 % at
// most, for grouped heads 5 %.  The slices under way at a time are twice as many as slice by slice, but still few.
// us, behind lasting load, slice by slice -> matched: 4 x 32 x 4096 x 128 578 -> 558, 1 x 32 x 16384 2043 -> 1967.  58 shapes
// of 5 to 13 % (1420 to 11577 rows, K and V of 130 to 465 MB, both head dims) took 0.68 to 1.01 of the time, half of them less
// than 0.96: 2 x 16 x 10841 x 128 1200 -> 811, 8 x 32 x 3311 x 64 542 -> 533, 7 x 16 x 4653 x 64 472 -> 478; at 15 to 19 % 0.77
// to 1.04 (8 x 12 x 3935 x 128 420 -> 439), and two query heads per K/V head from 5 % on 0.91 to 1.08 (5 x 32 x 6605 x 128
// 1608 -> 1732).
inline bool duo_matched(bool causal, const AttnShape& shp, const AttnShape& shp_kv, long long items, int units, int max_deal) {
  if (!causal || shp.S <= 1024 || shp.S > 128LL * pieces(shp_kv.S, 128) || (items & 1) != 0 || items >= (1LL << 30) ||
      duo_heaviest_first(causal, shp, shp_kv))
    return false;
  const long long twos = items / 2, rounds = (twos + units - 1) / units;
  return twos >= units && 2 * rounds < max_deal &&
         100 * rounds * units <= (shp.H == shp_kv.H ? 113 : 105) * twos;
}

// CTAs per work item for a problem of few items: the cluster size whose rounds take the fewest KV steps, counting 3 steps for a
// CTA's start and end and 2 or 3 for the merge.  steps: of the longest item.  active[c]: clusters of c CTAs that run at the same
// time, which is not SMs / c, as a cluster lives in one GPC (37 items as 37 clusters of 4 took two rounds, 35 us against 23 as
// clusters of 2).  Causal items of a second round could only be short ones, which this does not look at: one round.
inline int duo_parts(int items, int steps, bool causal, int sms, const int (&active)[kMaxClusterCtas + 1]) {
  int best = 1;
  long long best_cost = static_cast<long long>((items + sms - 1) / sms) * steps + 3;
  for (int c = 2; c <= kMaxClusterCtas && c <= steps; ++c) {
    if (active[c] <= 0 || (causal && items > active[c])) continue;
    const long long rounds = (items + active[c] - 1) / active[c];
    const long long cost = rounds * ((steps + c - 1) / c + 3 + (c > 2 ? 3 : 2));
    if (cost < best_cost) {
      best_cost = cost;
      best = c;
    }
  }
  return best;
}

// Whether it can be more than one, as a test that asks the device nothing: two CTAs per item have to fit, and up to four steps even
// the best split costs what it saves (a step each and the merge: 7, against 4 + 3).  The smallest calls run at the host's pace, and
// what duo_parts needs from the device costs it 0.1 to 0.2 us a call (4 heads of 256 rows: 6.20 -> 6.00 us).
inline bool duo_may_split(int items, int steps, int sms) { return 2 * items <= sms && steps > 4; }

// Whether CTA pairs take the items, by rows (items of 512) or by heads (items of 256 rows of two heads of a K/V head's group).
//
// A pair's products read half as much of K and V from shared memory, and half as much of them is copied into it: products and copies
// alone take 2106 cycles per 128 keys of two tiles instead of 2586 (of 2048 at the tensor pipe's rate: shared memory is full in
// single CTAs, whose scores' operands alone ask for its 128 bytes a cycle).  The chain through the softmax, 2900 cycles, does not get
// shorter by it, but the board, which is at its power limit in long calls, runs 3 % faster.  So it pays in long calls; in short ones
// the pair's start, end and common pace cost more (behind 15 ms of load instead of 60, up to 120 us: 1.00 to 1.07 times as long).
// us, single CTAs -> pairs, behind lasting load: 4 x 32 x 4096 993 -> 973, 16 x 16 x 1024 148 -> 147, 2 x 32 x 2325 203 -> 198,
// causal, by heads: 2 x 32/8 x 3000 164 -> 161, 4 x 40/20 x 2895 411 -> 389, 9 x 40/20 x 1741 358 -> 345; of 71 drawn calls that
// the rule takes, with scores of unit variance, 0.946 to 0.992 times as long.  What it leaves:
//   * items of 512 rows that need more rounds (1 x 40 x 2610: 1.14, 5 x 40 x 1130: 1.08; by heads they never do);
//   * items that leave more than a quarter of the last rounds' places empty: the board is not at its limit then, and with wide scores
//     (see rescale_o) pairs lose 3 to 7 % (1 x 8 x 6031 195 -> 206 us, unit variance 169 -> 168).  With fewer places empty, of 84
//     drawn calls: unit variance 0.98 by rows and 0.99 by heads, wide scores 1.017 and 0.995 on average (1.00 to 1.03, 0.98 to 1.03);
//   * fewer than 48 steps of two tiles per SM, or items of fewer than 8 steps (16 x 40 x 3490 on 116 keys: 1.06);
//   * causal items by rows, whose second pair of tiles works alone for two steps instead of one (4 x 32 x 4096 534 -> 552).
enum DuoPair : int { kDuoSingle = 0, kDuoPairRows = 1, kDuoPairHeads = 2 };
// pairs: that run at the same time.
inline DuoPair duo_pair(bool causal, int slices, int group, int seq_len, int steps, int sms, int pairs) {
  const bool heads = group % 2 == 0;
  if ((causal && !heads) || steps < 8) return kDuoSingle;
  const long long items = static_cast<long long>(slices) * pieces(seq_len, 256);
  const long long pair_items = heads ? items / 2 : static_cast<long long>(slices) * pieces(seq_len, 512);
  if (pairs <= 0) return kDuoSingle;
  const long long rounds = (pair_items + pairs - 1) / pairs;
  if (rounds > (items + sms - 1) / sms || 3 * rounds * pairs > 4 * pair_items) return kDuoSingle;
  if (items * (causal ? (steps + 1) / 2 : steps) < 48LL * sms) return kDuoSingle;
  return heads ? kDuoPairHeads : kDuoPairRows;
}
inline DuoPair duo_pair(bool causal, int slices, int group, int seq_len, int steps, int sms) {
  return duo_pair(causal, slices, group, seq_len, steps, sms, sms / 2);
}

// Head dim 64: whether the items go to the kernel with four independent streams per CTA (four_streams_sm100.cuh) instead.  Of
// 105 drawn calls that the rule sends there (1 to 46 steps, 80 to 4800 items, with and without a causal mask) it took 0.84 to 1.01
// times as long, 0.92 on average; with wide scores 0.81 to 0.97, 0.92 in the middle (34 calls, up to 8413 keys).  What it loses are many short items that all end with whole steps, where its
// end of an item, which adds up two accumulators, weighs more than its finer steps gain: 16 x 16 x 1024 with large logits 113 : 110
// us, 32 x 16 x 512 62.9 : 61.9, 256 keys 39.1 : 38.3, 511 rows on 194 keys 23.7 : 22.7; 1280 keys 122.1 : 122.6.
inline bool duo_quad(bool causal, long long items, int seq_k, int sms) {
  const bool whole_steps = pieces(seq_k, 64) % 2 == 0;  // the last 128 keys are more than half there
  return causal || !whole_steps || seq_k > 1024 || 2 * items < 5LL * sms;
}

// How a problem is dealt to the CTAs; parts: CTAs per item (kDuoSplit); quad: four independent streams per CTA (head dim 64);
// units: CTAs, or CTA pairs, that run at the same time.
struct DuoPlan {
  DuoMode mode;
  DuoPair pair;
  bool quad;
  int parts, sms, units, items, n_pairs, n_kv;
};

// CTA pairs that run at the same time: half of the SMs, unless the device or its share of one places fewer; 0 on failure.
template <int D, int STAGES>
inline int duo_pairs_at_a_time(int sms, cudaStream_t stream) {
  using Cfg = DuoCfg<D, STAGES, 2>;
  auto kernel = attn_fwd_duo_kernel<D, STAGES, kDuoDealt, 2>;
  struct Tag {};
  if (ensure_dynamic_smem<Tag>(kernel, Cfg::kSmemBytes, Cfg::kThreads, Cfg::kRegsTotal) != kAttnOk) return 0;
  ClusterLaunch launch(1, Cfg::kThreads, Cfg::kSmemBytes, stream);
  const auto* active = active_cluster_counts<Tag>(kernel, launch);
  return active == nullptr ? 0 : (*active)[2] < sms / 2 ? (*active)[2] : sms / 2;
}

template <int D, int STAGES>
inline int duo_plan(const AttnShape& shp, const AttnShape& shp_kv, bool causal, cudaStream_t stream, DuoPlan& plan) {
  using Cfg = DuoCfg<D, STAGES>;
  plan = DuoPlan{kDuoDealt, kDuoSingle, false, 1, device_sm_count(), 0, 0, 0, 0};
  if (plan.sms <= 0) return kAttnLaunchFailed;
  plan.units = plan.sms;
  plan.n_pairs = pieces(shp.S, 2 * Cfg::BM);
  plan.n_kv = pieces(shp_kv.S, Cfg::BN);
  plan.items = plan.n_pairs * shp.B * shp.H;
  const int steps = causal && 2 * plan.n_pairs < plan.n_kv ? 2 * plan.n_pairs : plan.n_kv;
  if (duo_may_split(plan.items, steps, plan.sms)) {
    auto split = attn_fwd_duo_kernel<D, STAGES, kDuoSplit, 1>;
    struct Tag {};
    const int rc = ensure_dynamic_smem<Tag>(split, Cfg::kSmemBytes, Cfg::kThreads, Cfg::kRegsTotal);
    if (rc != kAttnOk) return rc;
    ClusterLaunch launch(plan.items, Cfg::kThreads, Cfg::kSmemBytes, stream);
    const auto* active = active_cluster_counts<Tag>(split, launch);
    if (active == nullptr) return kAttnLaunchFailed;
    plan.parts = duo_parts(plan.items, steps, causal, plan.sms, *active);
    if (plan.parts > 1) plan.mode = kDuoSplit;
  } else {
    int max_deal = Cfg::kMaxDeal;
    if constexpr (D == 64) {
      plan.quad = duo_quad(causal, plan.items, shp_kv.S, plan.sms);
    } else {
      plan.pair = duo_pair(causal, shp.B * shp.H, shp.H / shp_kv.H, shp.S, steps, plan.sms);
      if (plan.pair != kDuoSingle) {
        const int pairs = duo_pairs_at_a_time<D, STAGES>(plan.sms, stream);
        plan.pair = duo_pair(causal, shp.B * shp.H, shp.H / shp_kv.H, shp.S, steps, plan.sms, pairs);
        if (plan.pair != kDuoSingle) plan.units = pairs;
      }
      if (plan.pair != kDuoSingle) {
        if (plan.pair == kDuoPairRows) plan.n_pairs = pieces(shp.S, 4 * Cfg::BM);
        plan.items = plan.n_pairs * shp.B * shp.H / (plan.pair == kDuoPairHeads ? 2 : 1);
        max_deal = DuoCfg<D, STAGES, 2>::kMaxDeal;
      }
    }
    if (duo_matched(causal, shp, shp_kv, plan.items, plan.units, max_deal)) plan.mode = kDuoMatched;  // two items per SM and more
  }
  return kAttnOk;
}

template <int D, int STAGES, DuoMode MODE, int CTAS>
inline int launch_duo_dealt(const DuoPlan& plan, cudaStream_t stream, const CUtensorMap& tm_q, const CUtensorMap& tm_k,
                            const CUtensorMap& tm_v, const CUtensorMap& tm_o, const AttnShape& shp, const AttnExtras& ex, bool causal,
                            float scale_log2, bool heaviest_first) {
  using Cfg = DuoCfg<D, STAGES, CTAS>;
  auto kernel = attn_fwd_duo_kernel<D, STAGES, MODE, CTAS>;
  struct Tag {};
  const int rc = ensure_dynamic_smem<Tag>(kernel, Cfg::kSmemBytes, Cfg::kThreads, Cfg::kRegsTotal);
  if (rc != kAttnOk) return rc;
  const int clusters = plan.items < plan.units ? plan.items : plan.units;
  auto launch = [&](auto... args) {
    if constexpr (CTAS == 1) return launch_overlapped(kernel, dim3(clusters), Cfg::kThreads, Cfg::kSmemBytes, stream, args...);
    ClusterLaunch cluster(clusters, Cfg::kThreads, Cfg::kSmemBytes, stream);
    cluster.set_ctas(CTAS);
    return cluster(kernel, args...);
  };
  return launch(tm_q, tm_k, tm_v, tm_o, shp.H, shp.B * shp.H, shp.S, causal ? 1 : 0, scale_log2, ex.kv_group, ex.lse, ex.seq_k,
                heaviest_first ? 1 : 0, plan.n_kv, plan.n_pairs, plan.items, 1, plan.pair == kDuoPairHeads ? 1 : 0, DuoOut{});
}

// Host launcher for the kernel with two softmax threads per row. Returns an AttnReturnCode.
template <int D, int STAGES>
inline int launch_attn_fwd_duo(const operand_t* q, const operand_t* k, const operand_t* v, operand_t* o, const AttnShape& shp,
                               const AttnStrides (&st)[4], const AttnExtras& ex, bool causal, float scale,
                               cudaStream_t stream) {
  using Cfg = DuoCfg<D, STAGES>;
  const AttnShape shp_kv{shp.B, shp.H / ex.kv_group, ex.seq_k, shp.D};
  CUtensorMap tm_q, tm_k, tm_v, tm_o;
  int rc = cached_attn_tensor_map(&tm_q, q, shp, st[0], Cfg::BM);
  if (rc != kAttnOk) return rc;
  DuoPlan plan;
  rc = duo_plan<D, STAGES>(shp, shp_kv, causal, stream, plan);
  if (rc != kAttnOk) return rc;
  rc = cached_attn_tensor_map(&tm_k, k, shp_kv, st[1], plan.pair == kDuoSingle ? Cfg::BN : Cfg::BN / 2);
  if (rc != kAttnOk) return rc;
  rc = cached_attn_tensor_map(&tm_v, v, shp_kv, st[2], Cfg::BN);
  if (rc != kAttnOk) return rc;
  rc = cached_attn_tensor_map(&tm_o, o, shp, st[3], Cfg::BM);
  if (rc != kAttnOk) return rc;

  const float scale_log2 = scale * 1.44269504088896340736f;
  if (plan.mode == kDuoSplit) {
    ClusterLaunch launch(plan.items, Cfg::kThreads, Cfg::kSmemBytes, stream);
    launch.set_ctas(plan.parts);
    const DuoOut out{o, shp.B > 1 ? st[3].b : 0, shp.H > 1 ? st[3].h : 0, shp.S > 1 ? st[3].s : 0};
    return launch(attn_fwd_duo_kernel<D, STAGES, kDuoSplit, 1>, tm_q, tm_k, tm_v, tm_o, shp.H, shp.B * shp.H, shp.S, causal ? 1 : 0,
                  scale_log2, ex.kv_group, ex.lse, ex.seq_k, 1, plan.n_kv, plan.n_pairs, plan.items, plan.parts, 0, out);
  }
  const bool heaviest_first = duo_heaviest_first(causal, shp, shp_kv);
  if constexpr (D == 64) {
    if (plan.quad)
      return launch_attn_fwd_quad<D>(tm_q, tm_k, tm_v, tm_o, shp, ex, causal, scale_log2, heaviest_first, plan.mode == kDuoMatched,
                                     plan.n_pairs, plan.items, plan.sms, stream);
    return launch_duo_dealt<D, STAGES, kDuoDealt, 1>(plan, stream, tm_q, tm_k, tm_v, tm_o, shp, ex, causal, scale_log2, heaviest_first);
  } else {
    auto dealt = [&](auto mode, auto ctas) {
      return launch_duo_dealt<D, STAGES, decltype(mode)::value, decltype(ctas)::value>(plan, stream, tm_q, tm_k, tm_v, tm_o, shp, ex, causal,
                                                                                        scale_log2, heaviest_first);
    };
    using Dealt = std::integral_constant<DuoMode, kDuoDealt>;
    using Matched = std::integral_constant<DuoMode, kDuoMatched>;
    using One = std::integral_constant<int, 1>;
    using Two = std::integral_constant<int, 2>;
    if (plan.pair != kDuoSingle) return plan.mode == kDuoMatched ? dealt(Matched{}, Two{}) : dealt(Dealt{}, Two{});
    return plan.mode == kDuoMatched ? dealt(Matched{}, One{}) : dealt(Dealt{}, One{});
  }
}

}  // namespace sm100
}  // namespace fray
