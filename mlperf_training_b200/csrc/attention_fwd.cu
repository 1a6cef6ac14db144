// Flash-attention forward for sm_100a: S = Q K^T and O += P V on tcgen05 tensor cores with the
// accumulators in TMEM, Q/K/V tiles brought in by TMA, online softmax in registers.
//
//   causal / non-causal, GQA (Hq a multiple of Hkv), sliding window, learned per-head sink
//   logits (an extra softmax column without a value), head_dim 64 or 128, bf16 in / bf16 out,
//   fp32 log-sum-exp saved for the backward pass.
//
// Persistent CTAs, one per SM; a work item is a (batch, head, pair of 128-query tiles).  384 threads:
//   warp 8      TMA producer (both Q tiles of an item, K/V double buffered, shared by the two tiles)
//   warp 9      MMA issuer, ping-pong over the two query tiles:
//                 S0(0) S1(0) | PV0(n) S0(n+1) PV1(n) S1(n+1) | ...
//               so the tensor core works on one tile while the other tile's softmax runs; the next
//               item's Q, K and first S are fetched and computed under this item's epilogue
//   warps 0-3   softmax of tile 0 (one query row per thread), warps 4-7 softmax of tile 1
//   (warps 10, 11 only complete the third warpgroup, which hands its registers to the softmax warps)
// TMEM (512 columns): S0 | S1 | O0 | O1.  The bf16 probabilities P overwrite the first half of
// their own S columns (tcgen05.st) and feed the second GEMM straight from TMEM (A operand in
// TMEM), so P never touches shared memory.  O is rescaled lazily: only when the running row
// maximum grew by more than 2^8.  A quarter of the exponentials run as a polynomial on the FMA
// pipe to relieve the MUFU unit.
//
// What bounds it: a pair of 128 x 128 tiles costs 4 x 512 tensor-core cycles.  The MMA issuer was the limit before: one
// lane of a divergent warp that rebuilt its descriptors needed about 130 cycles per instruction of 64 (clock64 in the
// roles), so the two tiles took 4900 cycles.  Now the warp stays converged, one elected lane issues, and descriptors
// advance by an addition.  Beside that, whatever the MMAs do not wait for has left the path from S to P: they start on
// the first 96 keys of P while the last 32 are still being exponentiated, the row sum is taken after P has been handed
// over, and the softmax warps hold 200 registers (all 128 scores in flight, no spills).  Items are handed out longest
// first over all heads (head after head left 14 % of the SM cycles idle at the end of a causal launch), in snake order
// over the rounds so that no CTA gets the longest of each.
// Measured (causal unless noted), one CTA per item -> now: 8192 x 32 heads of 128 622 -> 507 us (1.08 PFLOP/s); 4 x 2048
// 218 -> 172; 3 x 1337 107 -> 87; 8192 x 64 heads of 64, window 128 200 -> 158; 2000 x 64 of 64 114 -> 84; 8 x 512 x 24, full
// 56 -> 45.
//
// Stands in for the attention kernels the reference selects by config: Primus-Turbo / AITER /
// CK flash attention (small_llm_pretraining/primus/conf/llama3.1_8B-pretrain-fp4.yaml:117,125)
// and the sink / sliding-window attention of the GPT-OSS config
// (small_llm_moe_pretraining/primus/conf/gpt_oss_20B-MXFP4-deosc-mlperf-pretrain.yaml:125-127).
#include "common.cuh"
#include "runtime.h"

namespace {

#ifndef B200_ATTN_FWD_POLY
#define B200_ATTN_FWD_POLY 3
#endif
constexpr int POLY = B200_ATTN_FWD_POLY;  // pairs with (i & POLY) == POLY take the FMA-pipe polynomial: 3 = a quarter, 1 = half
constexpr int BQ = 128;   // query rows per tile (two tiles per CTA)
constexpr int BKV = 128;  // keys per tile
constexpr int NTHREADS = 384;  // warps 0-3 / 4-7: softmax of tile 0 / 1; warp 8: TMA; warp 9: MMA
constexpr int PV_EARLY = 96;   // keys of P the second GEMM starts on
// 3 x 128 threads launch with 168 registers each (504 per triple): 104 + 2 x 200 (56 or 72 for the other warps spilled)
constexpr int REGS_SOFTMAX = 200, REGS_OTHER = 104;

struct FwdParams {
  int B, Hq, Hkv, Sq, Skv;
  int causal;       // 1: key position <= query position (+ Skv - Sq offset)
  int window;       // > 0: query attends to keys with q_pos - k_pos < window
  float scale_log2; // softmax scale * log2(e)
  const float* sink;  // [Hq] learned sink logits (natural-log domain, unscaled) or null
  float* lse;         // [B, Hq, Sq] natural-log log-sum-exp of the scaled scores
  int* status;
  int bh_group;       // (batch, head) rows whose K / V stay in L2 together: items are ordered longest first inside a group
  int items;
};

// Work item u of the launch, and the key tiles its two query tiles look at.
struct Item {
  int b, h, q0, j_lo;
  int lo0, lo1, hi0, hi1;   // per query tile: key tiles j_lo + [lo, hi)
  int n_max;
  B200_DEVICE int lo(int t) const { return t ? lo1 : lo0; }
  B200_DEVICE int hi(int t) const { return t ? hi1 : hi0; }
};
B200_DEVICE Item make_item(int u, const FwdParams& p) {
  Item it;
  const int num_pairs = (p.Sq + 2 * BQ - 1) / (2 * BQ);
  const int g = u / (p.bh_group * num_pairs), r = u - g * p.bh_group * num_pairs;
  const int gsz = min(p.bh_group, p.B * p.Hq - g * p.bh_group);
  const int pair = num_pairs - 1 - r / gsz;          // longest (latest) query tiles first
  const int bh = g * p.bh_group + r % gsz;
  it.b = bh / p.Hq;
  it.h = bh - it.b * p.Hq;
  it.q0 = pair * 2 * BQ;
  const int off = p.Skv - p.Sq;                      // causal diagonal offset (0 for self-attention)
  const int j_max = (p.Skv + BKV - 1) / BKV - 1;
  it.j_lo = 0;
  if (p.window > 0) it.j_lo = max(0, it.q0 + off - p.window + 1) / BKV;
  const int hi0 = p.causal ? min(j_max, (it.q0 + BQ - 1 + off) / BKV) : j_max;
  const int hi1 = p.causal ? min(j_max, (it.q0 + 2 * BQ - 1 + off) / BKV) : j_max;
  it.lo0 = 0;
  it.lo1 = p.window > 0 ? max(0, it.q0 + BQ + off - p.window + 1) / BKV - it.j_lo : 0;
  it.hi0 = max(hi0 - it.j_lo + 1, 0);
  it.hi1 = it.q0 + BQ < p.Sq ? max(hi1 - it.j_lo + 1, it.lo1) : it.lo1;
  it.n_max = it.hi1 > it.lo1 ? max(it.hi0, it.hi1) : it.hi0;
  return it;
}
// Items of CTA blockIdx.x: one per round of gridDim.x items, in alternating direction.
B200_DEVICE int item_of_round(int r) {
  return r * (int)gridDim.x + ((r & 1) ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x);
}

B200_DEVICE float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

B200_DEVICE void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
B200_DEVICE void tma_store_4d(const CUtensorMap* map, const void* src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map),
               "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}

template <int HD>
struct Smem {
  static constexpr int Q_TILE = BQ * HD * 2;
  static constexpr int KV_BYTES = BKV * HD * 2;
  static constexpr int STAGE_O = 32 * 128;            // per softmax warp: 32 rows x 64 output columns
  static constexpr int TOTAL = 2 * Q_TILE + 4 * KV_BYTES + 8 * STAGE_O + 1024 + 256;
};

template <int HD>
__global__ void __launch_bounds__(NTHREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                const FwdParams p) {
  b200::begin_kernel();
  using SM = Smem<HD>;
  constexpr int NB = HD / 64;  // 64-column (128-byte) blocks per head row
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                       // two tiles
  uint8_t* sK = sQ + 2 * SM::Q_TILE;        // two stages
  uint8_t* sV = sK + 2 * SM::KV_BYTES;      // two stages
  uint8_t* sO = sV + 2 * SM::KV_BYTES;      // eight warps' output staging
  uint64_t* bars = reinterpret_cast<uint64_t*>(sO + 8 * SM::STAGE_O);
  uint64_t* q_full = bars;          // 1
  uint64_t* q_empty = bars + 1;     // 1: every S of the item has been computed
  uint64_t* k_full = bars + 2;      // 2
  uint64_t* k_empty = bars + 4;     // 2
  uint64_t* v_full = bars + 6;      // 2
  uint64_t* v_empty = bars + 8;     // 2
  uint64_t* s_full = bars + 10;     // 2 (per query tile): once per key tile
  uint64_t* p_early = bars + 12;    // 2 (4 arrivals): the first PV_EARLY keys of P are in TMEM
  uint64_t* p_full = bars + 14;     // 2 (4 arrivals): all of P
  uint64_t* o_done = bars + 16;     // 2: once per item, O complete
  uint64_t* o_free = bars + 18;     // 2 (4 arrivals): once per item, O read out of TMEM
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int off = p.Skv - p.Sq;
  const int rounds = (p.items + (int)gridDim.x - 1) / (int)gridDim.x;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1); mbar_init(q_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_early[i], 4); mbar_init(&p_full[i], 4);
      mbar_init(&o_done[i], 1); mbar_init(&o_free[i], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) { tmem_alloc(tmem_holder, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  if (warp >= 8) {
    reg_dealloc<REGS_OTHER>();
    if (warp == 8 && lane == 0) {
      // ------------------------------ TMA producer ------------------------------
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
      bool ok = true;
      int kv = 0, nq = 0;                    // key tiles and items so far: stage and phase of the barriers
      for (int r = 0; r < rounds && ok; ++r) {
        const int u = item_of_round(r);
        if (u >= p.items) continue;
        const Item it = make_item(u, p);
        if (it.n_max == 0) continue;
        const int hk = it.h / (p.Hq / p.Hkv);
        if (!mbar_wait(q_empty, (nq & 1) ^ 1, abort_flag, p.status, 39)) { ok = false; break; }
        ++nq;
        mbar_expect_tx(q_full, 2 * SM::Q_TILE);
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int i = 0; i < NB; ++i)
            tma_load_4d(sQ + t * SM::Q_TILE + i * (BQ * 128), &tmQ, q_full, i * 64, it.h, it.q0 + t * BQ, it.b);
        for (int n = 0; n < it.n_max; ++n, ++kv) {
          const int j = it.j_lo + n, st = kv & 1;
          const uint32_t ph = (kv >> 1) & 1;
          if (!mbar_wait(&k_empty[st], ph ^ 1, abort_flag, p.status, 40)) { ok = false; break; }
          mbar_expect_tx(&k_full[st], SM::KV_BYTES);
#pragma unroll
          for (int i = 0; i < NB; ++i)
            tma_load_4d(sK + st * SM::KV_BYTES + i * (BKV * 128), &tmK, &k_full[st], i * 64, hk, j * BKV, it.b);
          if (!mbar_wait(&v_empty[st], ph ^ 1, abort_flag, p.status, 41)) { ok = false; break; }
          mbar_expect_tx(&v_full[st], SM::KV_BYTES);
#pragma unroll
          for (int i = 0; i < NB; ++i)
            tma_load_4d(sV + st * SM::KV_BYTES + i * (BKV * 128), &tmV, &v_full[st], i * 64, hk, j * BKV, it.b);
        }
      }
    } else if (warp == 9) {
      // ------------------------------ MMA issuer ------------------------------
      // The whole warp walks the schedule and one elected lane issues: the operands of the instructions then stay in
      // uniform registers (descriptors advance by an addition).
      const uint32_t idesc_s = umma_idesc(1, 1, 0, 0, BQ, BKV);  // Q (K-major) x K (K-major)
      const uint32_t idesc_o = umma_idesc(1, 1, 0, 1, BQ, HD);   // P (TMEM)    x V (MN-major)
      const uint64_t dQ = umma_desc_sw128(smem_u32(sQ), 16, 1024), dK = umma_desc_sw128(smem_u32(sK), 16, 1024);
      const uint64_t dV = umma_desc_sw128(smem_u32(sV), BKV * 128, 1024);
      bool ok = true;
      int kv = 0, nq = 0;
      int np[2] = {0, 0}, no[2] = {0, 0};    // P tiles consumed / items finished per query tile
      for (int r = 0; r < rounds && ok; ++r) {
        const int u = item_of_round(r);
        if (u >= p.items) continue;
        const Item it = make_item(u, p);
        if (it.n_max == 0) continue;
        if (!warp_wait_spin(q_full, nq & 1, abort_flag, p.status, 50)) { ok = false; break; }
        ++nq;
        int k_ready = -1, v_ready = -1;      // last key tile of the item whose full barrier has been observed
        int s_left = (it.hi0 - it.lo0) + (it.hi1 - it.lo1);
        // S_t(n) = Q_t K(n)^T into the S columns of tile t
        auto issue_s = [&](int t, int n) -> bool {
          const int st = (kv + n) & 1;
          while (k_ready < n) {
            ++k_ready;
            if (!warp_wait_spin(&k_full[(kv + k_ready) & 1], ((kv + k_ready) >> 1) & 1, abort_flag, p.status, 51)) return false;
          }
          // the last S that reads K(n) frees its stage: S_t(n) is issued in step n - 1 (its first one before step 0)
          const int o = 1 - t;
          const bool both = n >= it.lo(o) && n < it.hi(o);
          const int mine = n == it.lo(t) ? -1 : n - 1, theirs = n == it.lo(o) ? -1 : n - 1;
          const bool free_k = !both || mine > theirs || (mine == theirs && t == 1);
          const bool free_q = --s_left == 0;
          tc_fence_after();
          if (elect_one()) {
            const uint64_t ad = dQ + (t * SM::Q_TILE >> 4), bd = dK + (st * SM::KV_BYTES >> 4);
#pragma unroll
            for (int kk = 0; kk < HD / 16; ++kk) {
              const uint32_t o4 = ((kk / 4) * (BQ * 128) + (kk % 4) * 32) >> 4;
              tc_mma_f16_ss(tmem_base + t * 128, ad + o4, bd + o4, idesc_s, kk > 0 ? 1u : 0u);
            }
            tc_commit(&s_full[t]);
            if (free_k) tc_commit(&k_empty[st]);
            if (free_q) tc_commit(q_empty);
          }
          __syncwarp();
          return true;
        };
#pragma unroll
        for (int t = 0; t < 2; ++t)
          if (ok && it.hi(t) > it.lo(t)) ok = issue_s(t, it.lo(t));
        for (int n = 0; n < it.n_max && ok; ++n) {
          const int st = (kv + n) & 1;
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (!ok || n < it.lo(t) || n >= it.hi(t)) continue;
            const bool first = n == it.lo(t), last = n == it.hi(t) - 1;
            // O of the previous item has left TMEM
            if (first && !warp_wait_spin(&o_free[t], (no[t] & 1) ^ 1, abort_flag, p.status, 52)) { ok = false; continue; }
            while (ok && v_ready < n) {
              ++v_ready;
              ok = warp_wait_spin(&v_full[(kv + v_ready) & 1], ((kv + v_ready) >> 1) & 1, abort_flag, p.status, 54);
            }
            ok = ok && warp_wait_spin(&p_early[t], np[t] & 1, abort_flag, p.status, 53);
            if (!ok) continue;
            tc_fence_after();
            // A = P_t in TMEM: 16 bf16 keys = 8 columns per step; B = V: 16 key rows of 128 bytes
            const uint64_t bd = dV + (st * SM::KV_BYTES >> 4);
            if (elect_one()) {
#pragma unroll
              for (int kk = 0; kk < PV_EARLY / 16; ++kk)
                tc_mma_f16_ts(tmem_base + 256 + t * 128, tmem_base + t * 128 + kk * 8, bd + (kk * (16 * 128) >> 4), idesc_o,
                              (!first || kk > 0) ? 1u : 0u);
            }
            __syncwarp();
            ok = warp_wait_spin(&p_full[t], np[t] & 1, abort_flag, p.status, 55);
            if (!ok) continue;
            tc_fence_after();
            const bool free_v = (t == 1) || !(n >= it.lo1 && n < it.hi1);
            if (elect_one()) {
#pragma unroll
              for (int kk = PV_EARLY / 16; kk < BKV / 16; ++kk)
                tc_mma_f16_ts(tmem_base + 256 + t * 128, tmem_base + t * 128 + kk * 8, bd + (kk * (16 * 128) >> 4), idesc_o, 1u);
              if (last) tc_commit(&o_done[t]);
              if (free_v) tc_commit(&v_empty[st]);
            }
            __syncwarp();
            ++np[t];
            if (last) ++no[t];
            else ok = issue_s(t, n + 1);
          }
        }
        kv += it.n_max;
      }
    }
  } else {
    // ------------------------------ softmax + epilogue (one warpgroup per query tile) --------------
    reg_alloc<REGS_SOFTMAX>();
    const int t = warp >> 2;
    const int q = warp & 3;
    const int r = q * 32 + lane;           // row inside the query tile
    const uint32_t lane_base = uint32_t(q * 32) << 16;
    const uint32_t ts = tmem_base + lane_base + t * 128;        // S / P columns of this tile
    const uint32_t to = tmem_base + lane_base + 256 + t * 128;  // O columns of this tile
    uint8_t* stage = sO + warp * SM::STAGE_O;
    int ns = 0, no = 0;                    // S tiles and items so far
    bool ok = true;
    for (int round = 0; round < rounds && ok; ++round) {
      const int u = item_of_round(round);
      if (u >= p.items) continue;
      const Item it = make_item(u, p);
      if (it.hi(t) <= it.lo(t)) continue;
      const int qt0 = it.q0 + t * BQ;
      const int q_pos = qt0 + r;
      const int hi = p.causal ? min(q_pos + off, p.Skv - 1) : p.Skv - 1;         // last visible key
      const int lo = p.window > 0 ? q_pos + off - p.window + 1 : 0;              // first visible key
      float m_ref = -INFINITY, l = 0.f;
      for (int n = it.lo(t); n < it.hi(t); ++n, ++ns) {
        const int kv0 = (it.j_lo + n) * BKV;
        if (!warp_wait(&s_full[t], ns & 1, abort_flag, p.status, 60)) { ok = false; break; }
        tc_fence_after();
        const bool need_mask = (kv0 + BKV > p.Skv) || (p.causal && kv0 + BKV - 1 > qt0 + off) ||
                               (p.window > 0 && kv0 < qt0 + BQ - 1 + off - p.window + 1);
        // the whole score row (128 fp32) comes into registers with one TMEM round trip
        uint32_t v[BKV];
#pragma unroll
        for (int c = 0; c < BKV / 32; ++c) tmem_ld_32x32b_x32(ts + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&v[c * 32]));
        tc_wait_ld();
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < BKV; ++i) {
            const int kp = kv0 + i;
            if (kp > hi || kp < lo) v[i] = 0xff800000u;  // -inf
          }
        }
        float mx4[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) mx4[c] = fmaxf(__uint_as_float(v[2 * c]), __uint_as_float(v[2 * c + 1]));
#pragma unroll
        for (int i = 8; i < BKV; i += 8)
#pragma unroll
          for (int c = 0; c < 4; ++c) mx4[c] = max3(mx4[c], __uint_as_float(v[i + 2 * c]), __uint_as_float(v[i + 2 * c + 1]));
        float mx = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]);
        mx *= p.scale_log2;  // -inf stays -inf (scale > 0)
        // lazy rescale: move the reference maximum only when it grew by more than 2^8
        const bool grow = (mx > m_ref + 8.f) || (m_ref == -INFINITY && mx > -INFINITY);
        if (__any_sync(0xffffffffu, grow)) {
          const float m_new = fmaxf(m_ref, mx);
          const float alpha = (m_ref == -INFINITY) ? 0.f : ex2_approx(m_ref - m_new);
          m_ref = m_new;
          l *= alpha;
          if (n > it.lo(t)) {
            // (S of this key tile was issued after P V of the one before it and completes after it: O is complete)
#pragma unroll 1
            for (int c = 0; c < HD / 32; ++c) {
              uint32_t o[32];
              tmem_ld_32x32b_x32(to + c * 32, o);
              tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st_32x32b_x32(to + c * 32, o);
            }
            tc_wait_st();
          }
        }
        const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
        // P = exp2(S * scale - m) as bf16 pairs over the first half of the S columns; every fourth
        // pair takes the polynomial path (FMA pipe), the rest the MUFU path; -inf gives 2^-126 and 0
        const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
        const float2 nm2 = make_float2(-m_use, -m_use);
#pragma unroll
        for (int c = 0; c < BKV / 32; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int e = c * 32 + 2 * i;
            const float2 a = ffma2(make_float2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), sc2, nm2);
            float2 x;
            if ((i & POLY) == POLY) x = ex2_poly2(a);
            else x = make_float2(ex2_approx(a.x), ex2_approx(a.y));
            v[e] = __float_as_uint(x.x); v[e + 1] = __float_as_uint(x.y);
            pk[i] = pack_bf16x2(x.x, x.y);
          }
          tmem_st_32x32b_x16(ts + c * 16, pk);
          if (c == PV_EARLY / 32 - 1 || c == BKV / 32 - 1) {
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(c == BKV / 32 - 1 ? &p_full[t] : &p_early[t]);
          }
        }
        // the row sum, off the path of the MMAs
        float2 rs2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int i = 0; i < BKV / 2; ++i)
          rs2[i & 1] = fadd2(rs2[i & 1], make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])));
        l += (rs2[0].x + rs2[0].y) + (rs2[1].x + rs2[1].y);
      }
      // ------------------------------ epilogue ------------------------------
      if (!ok || !warp_wait(&o_done[t], no & 1, abort_flag, p.status, 62)) { ok = false; break; }
      ++no;
      tc_fence_after();
      if (p.sink != nullptr) {
        const float sk = p.sink[it.h] * 1.4426950408889634f;
        if (m_ref == -INFINITY) { m_ref = sk; l = 1.f; }
        else l += ex2_approx(sk - m_ref);
      }
      const float inv = l > 0.f ? 1.f / l : 0.f;
      if (q_pos < p.Sq && p.lse != nullptr)
        p.lse[((long long)it.b * p.Hq + it.h) * p.Sq + q_pos] =
            (l > 0.f) ? (m_ref + log2f(l)) * 0.6931471805599453f : -INFINITY;
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        uint32_t v[64];
        tmem_ld_32x32b_x32(to + i * 64, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
        tmem_ld_32x32b_x32(to + i * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
        tc_wait_ld();
        if (i == NB - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&o_free[t]);
        }
        if (lane == 0) tma_store_wait_read<0>();     // the previous block has left the staging buffer
        __syncwarp();
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            w[j] = pack_bf16x2(__uint_as_float(v[8 * g + 2 * j]) * inv, __uint_as_float(v[8 * g + 2 * j + 1]) * inv);
          *reinterpret_cast<uint4*>(stage + lane * 128 + ((g ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (qt0 + q * 32 < p.Sq) tma_store_4d(&tmO, stage, i * 64, it.h, qt0 + q * 32, it.b);
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait_all<0>();
  }

  __syncwarp();
  if (*abort_flag) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// tensor [B][S][H][HD] view with arbitrary row pitch: dims (inner to outer) {HD, H, S, B}
int make_qkv_map(CUtensorMap* m, const void* ptr, int HD, int H, int S, int B, long long row_stride,
                 long long batch_stride, int box_rows) {
  return b200::make_tmap_4d(m, b200::DT_BF16, ptr, HD, H, S, B, (uint64_t)HD * 2, (uint64_t)row_stride * 2,
                            (uint64_t)batch_stride * 2, 64, 1, box_rows, 1, b200::SWZ_128);
}

template <int HD>
int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to,
               const FwdParams& p, cudaStream_t stream) {
  using SM = Smem<HD>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(attn_fwd_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::TOTAL);
    if (e != cudaSuccess) cudaGetLastError();  // clear the sticky error before reporting
    if (e != cudaSuccess) return b200::fail(601, "attn_fwd: cannot set %d bytes of shared memory: %s", SM::TOTAL,
                                            cudaGetErrorString(e));
    configured[dev & 63] = true;
  }
  const int grid = p.items < b200::sm_count() ? p.items : b200::sm_count();
  b200::launch(attn_fwd_kernel<HD>, grid, NTHREADS, SM::TOTAL, stream, tq, tk, tv, to, p);
  b200::count_launch();
  return b200::check_launch("attn_fwd");
}

}  // namespace

// q: [B, Sq, Hq, HD], k/v: [B, Skv, Hkv, HD], o: [B, Sq, Hq, HD]; each with its own row pitch
// (elements between consecutive tokens) and batch pitch, heads contiguous inside a token row.
B200_API int b200_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const float* sink,
                           int B, int Sq, int Skv, int Hq, int Hkv, int HD, long long q_row, long long k_row,
                           long long v_row, long long o_row, long long q_batch, long long k_batch,
                           long long v_batch, long long o_batch, float scale, int causal, int window,
                           void* stream) {
  if (HD != 64 && HD != 128) return b200::fail(600, "attn_fwd: head dim %d not supported (64 or 128)", HD);
  if (Hq % Hkv != 0) return b200::fail(600, "attn_fwd: Hq=%d not a multiple of Hkv=%d", Hq, Hkv);
  if (causal && Skv < Sq) return b200::fail(600, "attn_fwd: causal needs Skv >= Sq");
  CUtensorMap tq, tk, tv, to;
  int r;
  if ((r = make_qkv_map(&tq, q, HD, Hq, Sq, B, q_row, q_batch, BQ))) return r;
  if ((r = make_qkv_map(&tk, k, HD, Hkv, Skv, B, k_row, k_batch, BKV))) return r;
  if ((r = make_qkv_map(&tv, v, HD, Hkv, Skv, B, v_row, v_batch, BKV))) return r;
  if ((r = make_qkv_map(&to, o, HD, Hq, Sq, B, o_row, o_batch, 32))) return r;
  FwdParams p;
  p.B = B; p.Hq = Hq; p.Hkv = Hkv; p.Sq = Sq; p.Skv = Skv;
  p.causal = causal; p.window = window;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.sink = sink; p.lse = lse;
  p.status = b200::status_ptr();
  const long long items = (long long)((Sq + 2 * BQ - 1) / (2 * BQ)) * Hq * B;
  if (items <= 0 || items > 0x3fffffff) return b200::fail(600, "attn_fwd: %lld query tile pairs", items);
  p.items = (int)items;
  // Full attention: every item costs the same, and heads go in groups whose K and V take half of the 126 MB L2, so that the
  // next group's fit beside them (16384 x 32 heads of 128: groups of 8 3828 us, all heads at once 4009; 2 x 4608 x 24, where
  // the group is more than half of the heads: 505 and 504).
  // Causal: the longest items of all heads first, whatever that does to L2.  Groups leave a tail of their own each (groups by
  // the rule above and all at once: 16384 x 32 heads of 128 2189 and 2017 us, 2 x 8192 x 32 1159 and 1067, window 1024 383 and
  // 365, 2 x 8192 x 64 heads of 64 1886 and 1733; single heads and groups of four lie between or above).
  const long long per_kv_head = (long long)Skv * HD * 4, fit = (64ll << 20) / per_kv_head;
  const long long group = (fit > 0 ? fit : 1) * (Hq / Hkv);
  p.bh_group = (int)(!causal && group < (long long)B * Hq ? group : (long long)B * Hq);
  if (HD == 128) return launch_fwd<128>(tq, tk, tv, to, p, (cudaStream_t)stream);
  return launch_fwd<64>(tq, tk, tv, to, p, (cudaStream_t)stream);
}
