// Flash-attention backward for sm_100a.  One CTA owns one (batch, kv-head, 128-key tile) and
// loops over the query heads of its GQA group and over the query tiles that see those keys:
//
//   S  = Q K^T            dP = dO V^T                   (tcgen05, accumulators in TMEM)
//   P  = exp2(S*c - lse)  dS = P * (dP - delta) * scale (softmax warps, registers)
//   dQ = dS K   (TMEM -> fp32 TMA reduce-add into a global fp32 dQ buffer)
//   dV += P^T dO          dK += dS^T Q                  (stay in TMEM for the whole CTA)
//
// The scores are computed transposed, S^T = K Q^T and dP^T = V dO^T, so a worker thread owns a key row.  P^T goes back to
// TMEM over its own scores (tcgen05.st) and is the TMEM operand of dV; only dS^T is written to shared memory, once, as a
// [key][query] bf16 tile that the tensor core reads key-major for dK and, through an MN-major descriptor, transposed for
// dQ.  The log-sum-exp and delta of the tile's queries run along the columns: they are staged in shared memory.  dK / dV
// leave as bf16 through TMA stores.
//
// 512 threads: warp 0 TMA producer, warp 1 MMA issuer, warps 4-7 dQ drain (TMEM -> registers, accumulator released,
// registers -> shared memory -> fp32 TMA reduce-add), warps 8-15 workers.  Two workers share a TMEM lane quarter (32 key
// rows): each takes half of the 128 query columns.  Every exponential is ex2.approx: a polynomial on the
// FMA pipe (relative error up to 7e-4, as the forward takes for a quarter of the keys) for a quarter of the query columns was
// neither exact nor the forward's P, and added up to 0.13 % to the errors of dQ and dK against 64 bits (6 draws of 5 shapes
// up to 2048 tokens).  On the MUFU unit alone the errors are 0.02 to 0.25 % below those of the forward's own P.  It costs nothing
// at head dim 128 (8192 x 32 / 8 1293 us with the polynomial, 1297 without; 8 x 512 x 24 full 128 and 128) and 4 to 6 % at 64,
// where the products are half as long (2000 x 64 / 8 282 and 298, 8192 x 64 / 8 with window 128 263 and 273).
// TMEM (512 columns): S^T / P^T | dP^T, then dQ | dK | dV.  Order of the MMAs of step i, Q double-buffered:
//     [P^T(i) written]  dV(i)   [dS^T(i) written]  dQ(i)  S(i+1)  dK(i)  [dQ(i) drained]  dP(i+1)
// so dQ(i) is drained and S(i+1) exponentiated while the tensor core runs dK(i) and dP(i+1).  (The drain has warps of its
// own: staged by the workers, its 64 KB a step took 3000 of their 6700 cycles, clock64 in the roles.)
// Measured with delta, clearing and launches: queries as rows, P and dS through shared memory, one Q stage -> transposed ->
// drain warps, as it is: 8192 x 32 / 8 heads of 128 causal 1990 -> 1766 -> 1310 us (1.05 PFLOP/s), 4096 x 64 / 8 1130 -> 1005
// -> 765, 4 x 2048 607 -> 550 -> 408, 2000 x 64 / 8 of 64 448 -> 378 -> 298, 8 x 512 x 24 full 175 -> 157 -> 128.
//
// The reference takes this kernel from Primus-Turbo / AITER / CK (config knobs
// llama2_sft/primus/config_MI355X_1x8x1.sh:35-39); there is no in-tree counterpart.
#include <algorithm>
#include <climits>
#include <queue>
#include <vector>

#include "common.cuh"
#include "runtime.h"

namespace {

constexpr int BQ = 128;
constexpr int BKV = 128;
constexpr int NTHREADS = 512;  // warp 0 TMA, 1 MMA (2, 3 complete the warpgroup), 4-7 dQ drain, 8-15 P / dS workers
// 4 x 128 threads launch with 128 registers each: 88 + 88 + 2 x 168
constexpr int REGS_OTHER = 88, REGS_WORKER = 168;
constexpr int STG = 4096;  // dQ staging chunk: 32 rows x 32 fp32 (two per drain warp)

constexpr int MAX_PARTS = 8, MAX_ENTRIES = 512;

struct BwdParams {
  int B, Hq, Hkv, Sq, Skv;
  int causal, window;
  float scale, scale_log2;
  const float* lse;    // [B, Hq, Sq]
  const float* delta;  // [B, Hq, Sq]  rowsum(dO * O)
  int* status;
  int bh_group;        // (batch, kv head) pairs scheduled together, longest key tiles first
  // Split schedule (cap > 0): no CTA takes more than cap steps of a key tile; the others of a tile take its next ones.
  int cap, entries;    // entries: CTAs of one (batch, kv head) pair, in `order` as (key tile << 3 | part), longest first
  int slots;           // parts of the tiles that are cut, and where in them each entry's is
  float* partial;      // fp32 [B * Hkv][slots][dK | dV][128][HD]
  uint16_t order[MAX_ENTRIES];
  uint16_t slot[MAX_ENTRIES];
};

// The key tiles that are cut, and the first slot of each.
struct CutTiles {
  int n;
  uint16_t tile[MAX_ENTRIES / 2], slot[MAX_ENTRIES / 2];
};

// (query head, query tile) steps of key tile jt and its first query tile.
__host__ __device__ inline int tile_steps(int jt, int Sq, int Skv, int group, int causal, int window, int& i_lo, int& i_hi) {
  const int kv0 = jt * BKV, off = Skv - Sq;
  i_lo = 0; i_hi = (Sq + BQ - 1) / BQ - 1;
  if (causal) {
    const int first_q = kv0 - off;  // first query position that sees key kv0
    if (first_q > 0) i_lo = first_q / BQ;
  }
  if (window > 0) {
    const int last_q = kv0 + BKV - 1 + window - 1 - off;  // last query that still sees the tile's last key
    if (last_q / BQ < i_hi) i_hi = last_q / BQ;
  }
  return i_hi >= i_lo ? (i_hi - i_lo + 1) * group : 0;
}
__host__ __device__ inline int tile_parts(int steps, int cap) { return steps > cap ? (steps + cap - 1) / cap : 1; }

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
B200_DEVICE void tma_reduce_add_4d(const CUtensorMap* map, const void* src, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map),
      "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

template <int HD>
struct Smem {
  static constexpr int T_BYTES = 128 * HD * 2;        // K, V, Q (two stages), dO tiles
  static constexpr int DS_BYTES = BQ * BKV * 2;       // dS^T tile
  static constexpr int STG_BYTES = 8 * STG;
  static constexpr int LD_BYTES = 2 * 2 * BQ * 4;     // log-sum-exp and delta of two query tiles
  // The base of dynamic shared memory is 1024-byte aligned when a kernel has no static shared memory; checked at entry
  // (at head dim 128 there is no room to align it).
  static constexpr int TOTAL = 5 * T_BYTES + DS_BYTES + STG_BYTES + LD_BYTES + 256;
};

template <int HD>
__global__ void __launch_bounds__(NTHREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                const __grid_constant__ CUtensorMap tmdQ, const __grid_constant__ CUtensorMap tmdK,
                const __grid_constant__ CUtensorMap tmdV, const __grid_constant__ BwdParams p) {
  b200::begin_kernel();
  using SM = Smem<HD>;
  constexpr int NB = HD / 64;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;
  uint8_t* sV = sK + SM::T_BYTES;
  uint8_t* sQ = sV + SM::T_BYTES;           // two stages
  uint8_t* sdO = sQ + 2 * SM::T_BYTES;
  uint8_t* sdS = sdO + SM::T_BYTES;
  uint8_t* sStg = sdS + SM::DS_BYTES;
  float* sLD = reinterpret_cast<float*>(sStg + SM::STG_BYTES);   // [stage][lse2 | delta * scale][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sLD + 4 * BQ);
  uint64_t* kv_full = bars + 0;     // K and V landed
  uint64_t* q_full = bars + 1;      // 2: Q_i landed
  uint64_t* q_empty = bars + 3;     // 2: MMAs reading Q_i finished
  uint64_t* do_full = bars + 5;     // dO_i landed
  uint64_t* do_empty = bars + 6;    // MMAs reading dO_i finished
  uint64_t* s_full = bars + 7;      // S^T complete in TMEM
  uint64_t* dp_full = bars + 8;     // dP^T complete in TMEM (and every MMA of the step before: dS^T is free)
  uint64_t* p_full = bars + 9;      // P^T written to TMEM (8 arrivals)
  uint64_t* ds_full = bars + 10;    // dS^T written to shared memory (8 arrivals)
  uint64_t* dq_full = bars + 11;    // dQ tile complete in TMEM
  uint64_t* dq_drained = bars + 12; // dQ tile copied out of TMEM (4 arrivals)
  uint64_t* ld_full = bars + 13;    // 2: the step's log-sum-exp / delta are in shared memory (8 arrivals)
  uint64_t* acc_done = bars + 15;   // every MMA of this CTA finished
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  if (smem_u32(smem) & 1023u) {             // (the same for every thread of the launch)
    if (threadIdx.x == 0) b200_report(p.status, B200_ERR_BOUNDS, 94);
    return;
  }

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int num_kt = (p.Skv + BKV - 1) / BKV;
  // early key tiles see the most queries: they are scheduled first, over all heads of a group
  const int bh_all = p.B * p.Hkv;
  int jt, bh, part = 0, e = 0;
  if (p.cap > 0) {
    e = (int)blockIdx.x / bh_all;
    bh = (int)blockIdx.x - e * bh_all;
    jt = p.order[e] >> 3;
    part = p.order[e] & 7;
  } else {
    const int per_group = p.bh_group * num_kt;
    const int grp = (int)blockIdx.x / per_group, rest = (int)blockIdx.x - grp * per_group;
    const int gsz = min(p.bh_group, bh_all - grp * p.bh_group);
    jt = rest / gsz;
    bh = grp * p.bh_group + rest % gsz;
  }
  const int b = bh / p.Hkv, hk = bh - b * p.Hkv;
  const int group = p.Hq / p.Hkv;
  const int kv0 = jt * BKV;
  const int off = p.Skv - p.Sq;
  // query tiles that see at least one key of this tile
  int i_lo, i_hi;
  const int steps = tile_steps(jt, p.Sq, p.Skv, group, p.causal, p.window, i_lo, i_hi);
  const int n_q = i_hi >= i_lo ? i_hi - i_lo + 1 : 0;
  // this CTA's steps of the tile's
  const int parts = p.cap > 0 ? tile_parts(steps, p.cap) : 1;
  const int it0 = steps * part / parts, n_iter = steps * (part + 1) / parts - it0;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1); mbar_init(do_full, 1); mbar_init(do_empty, 1); mbar_init(s_full, 1); mbar_init(dp_full, 1);
    mbar_init(p_full, 8); mbar_init(ds_full, 8); mbar_init(dq_full, 1); mbar_init(dq_drained, 4); mbar_init(acc_done, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); mbar_init(&ld_full[i], 8); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(tmem_holder, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tm_S = tmem_base;          // S^T; P^T of queries 0-63 in columns 0-31, of 64-127 in 64-95
  const uint32_t tm_dP = tmem_base + 128;   // dP^T, later dQ
  const uint32_t tm_dK = tmem_base + 256;
  const uint32_t tm_dV = tmem_base + 384;

  if (warp < 8) reg_dealloc<REGS_OTHER>();
  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    // (a key tile that no query sees loads nothing: nobody would wait for it, and the CTA must not leave with copies in flight)
    if (lane == 0 && n_iter > 0) {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO);
      mbar_expect_tx(kv_full, 2 * SM::T_BYTES);
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        tma_load_4d(sK + i * (BKV * 128), &tmK, kv_full, i * 64, hk, kv0, b);
        tma_load_4d(sV + i * (BKV * 128), &tmV, kv_full, i * 64, hk, kv0, b);
      }
      for (int it = 0; it < n_iter; ++it) {
        const int h = hk * group + (it0 + it) / n_q;
        const int q0 = (i_lo + (it0 + it) % n_q) * BQ;
        const int st = it & 1;
        if (!mbar_wait(&q_empty[st], ((it >> 1) & 1) ^ 1, abort_flag, p.status, 70)) break;
        mbar_expect_tx(&q_full[st], SM::T_BYTES);
#pragma unroll
        for (int i = 0; i < NB; ++i) tma_load_4d(sQ + st * SM::T_BYTES + i * (BQ * 128), &tmQ, &q_full[st], i * 64, h, q0, b);
        if (!mbar_wait(do_empty, (it & 1) ^ 1, abort_flag, p.status, 71)) break;
        mbar_expect_tx(do_full, SM::T_BYTES);
#pragma unroll
        for (int i = 0; i < NB; ++i) tma_load_4d(sdO + i * (BQ * 128), &tmdO, do_full, i * 64, h, q0, b);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    // The warp stays converged and one elected lane issues: operands live in uniform registers and descriptors advance by
    // an addition (rebuilt by one lane of a divergent warp they cost more than the 64 cycles an instruction runs).
    if (n_iter > 0) {
      const uint32_t id_kk = umma_idesc(1, 1, 0, 0, 128, 128);   // S^T = K Q^T, dP^T = V dO^T (both K-major)
      const uint32_t id_dv = umma_idesc(1, 1, 0, 1, 128, HD);    // dV = P^T (TMEM) x dO (MN-major)
      const uint32_t id_dk = umma_idesc(1, 1, 0, 1, 128, HD);    // dK = dS^T (K-major) x Q (MN-major)
      const uint32_t id_dq = umma_idesc(1, 1, 1, 1, 128, HD);    // dQ = dS (the tile read MN-major) x K (MN-major)
      const uint64_t kK = umma_desc_sw128(smem_u32(sK), 16, 1024), kV = umma_desc_sw128(smem_u32(sV), 16, 1024);
      const uint64_t kQ = umma_desc_sw128(smem_u32(sQ), 16, 1024), kdO = umma_desc_sw128(smem_u32(sdO), 16, 1024);
      const uint64_t kdS = umma_desc_sw128(smem_u32(sdS), 16, 1024), mdS = umma_desc_sw128(smem_u32(sdS), 128 * 128, 1024);
      const uint64_t mK = umma_desc_sw128(smem_u32(sK), 128 * 128, 1024), mQ = umma_desc_sw128(smem_u32(sQ), 128 * 128, 1024);
      const uint64_t mdO = umma_desc_sw128(smem_u32(sdO), 128 * 128, 1024);
      auto issue_s = [&](int it) -> bool {
        const int st = it & 1;
        if (!warp_wait_spin(&q_full[st], (it >> 1) & 1, abort_flag, p.status, 81)) return false;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t bd = kQ + (st * SM::T_BYTES >> 4);
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) {
            const uint32_t o = ((kk / 4) * (128 * 128) + (kk % 4) * 32) >> 4;
            tc_mma_f16_ss(tm_S, kK + o, bd + o, id_kk, kk > 0);
          }
          tc_commit(s_full);
        }
        __syncwarp();
        return true;
      };
      auto issue_dp = [&](int it) -> bool {
        if (!warp_wait_spin(do_full, it & 1, abort_flag, p.status, 82)) return false;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) {
            const uint32_t o = ((kk / 4) * (128 * 128) + (kk % 4) * 32) >> 4;
            tc_mma_f16_ss(tm_dP, kV + o, kdO + o, id_kk, kk > 0);
          }
          tc_commit(dp_full);
        }
        __syncwarp();
        return true;
      };
      bool ok = warp_wait_spin(kv_full, 0, abort_flag, p.status, 80) && issue_s(0) && issue_dp(0);
      for (int it = 0; it < n_iter && ok; ++it) {
        const uint32_t ph = it & 1;
        const int st = it & 1;
        const bool last = it == n_iter - 1;
        if (!warp_wait_spin(p_full, ph, abort_flag, p.status, 83)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          // dV += P^T dO : 16 queries = 8 TMEM columns per step, dO as 16 query rows of 128 bytes
#pragma unroll
          for (int kk = 0; kk < BQ / 16; ++kk)
            tc_mma_f16_ts(tm_dV, tm_S + (kk / 4) * 64 + (kk % 4) * 8, mdO + kk * 128, id_dv, (it > 0 || kk > 0));
          tc_commit(do_empty);
        }
        __syncwarp();
        if (!warp_wait_spin(ds_full, ph, abort_flag, p.status, 84)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          // dQ = dS K : contraction over keys, 16 key rows of the dS^T tile and of K per step
#pragma unroll
          for (int kk = 0; kk < BKV / 16; ++kk) tc_mma_f16_ss(tm_dP, mdS + kk * 128, mK + kk * 128, id_dq, kk > 0);
          tc_commit(dq_full);
        }
        __syncwarp();
        if (!last && !issue_s(it + 1)) { ok = false; break; }     // (P^T(i) was read by dV(i), issued before)
        if (elect_one()) {
          // dK += dS^T Q : contraction over queries
          const uint64_t bd = mQ + (st * SM::T_BYTES >> 4);
#pragma unroll
          for (int kk = 0; kk < BQ / 16; ++kk) {
            const uint32_t ao = ((kk / 4) * (128 * 128) + (kk % 4) * 32) >> 4;
            tc_mma_f16_ss(tm_dK, kdS + ao, bd + kk * 128, id_dk, (it > 0 || kk > 0));
          }
          tc_commit(&q_empty[st]);
          if (last) tc_commit(acc_done);
        }
        __syncwarp();
        if (!last) ok = warp_wait_spin(dq_drained, ph, abort_flag, p.status, 85) && issue_dp(it + 1);
      }
    }
  } else if (warp >= 4 && warp < 8) {
    // ------------------------------ dQ drain ------------------------------
    const int q = warp & 3;                   // TMEM lane quarter: 32 query rows
    const uint32_t lane_base = uint32_t(q * 32) << 16;
    uint8_t* stg = sStg + q * 2 * STG;
    for (int it = 0; it < n_iter; ++it) {
      const int h = hk * group + (it0 + it) / n_q;
      const int q0 = (i_lo + (it0 + it) % n_q) * BQ;
      if (!warp_wait(dq_full, it & 1, abort_flag, p.status, 95)) break;
      tc_fence_after();
#pragma unroll
      for (int c2 = 0; c2 < HD / 64; ++c2) {       // 64 columns at a time: two staging buffers
        uint32_t v[64];
        tmem_ld_32x32b_x32(tm_dP + lane_base + c2 * 64, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
        tmem_ld_32x32b_x32(tm_dP + lane_base + c2 * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
        tc_wait_ld();
        if (c2 == HD / 64 - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(dq_drained);  // the accumulator may be overwritten by the next dP
        }
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          if (lane == 0) tma_store_wait_read<1>(); // the reduce before the last has read this buffer
          __syncwarp();
          uint8_t* sb = stg + cc * STG + lane * 128;
#pragma unroll
          for (int g = 0; g < 8; ++g)
            *reinterpret_cast<uint4*>(sb + ((g ^ (lane & 7)) << 4)) =
                make_uint4(v[cc * 32 + 4 * g], v[cc * 32 + 4 * g + 1], v[cc * 32 + 4 * g + 2], v[cc * 32 + 4 * g + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (q0 + q * 32 < p.Sq) tma_reduce_add_4d(&tmdQ, stg + cc * STG, c2 * 64 + cc * 32, h, q0 + q * 32, b);
            tma_store_commit();
          }
        }
      }
    }
    if (lane == 0) tma_store_wait_all<0>();
  } else if (warp >= 8) {
    // ------------------------------ workers: P / dS ------------------------------
    reg_alloc<REGS_WORKER>();
    const int q = warp & 3;                   // TMEM lane quarter
    const int half = (warp - 8) >> 2;         // which half of the query columns
    const int r = q * 32 + lane;              // key row of the tile
    const uint32_t lane_base = uint32_t(q * 32) << 16;
    const int key = kv0 + r;
    // this thread stages one value per step: the log-sum-exp (half 0) or delta (half 1) of query r of the tile
    // (loaded a step ahead as it is and turned into what the columns need only when it is stored: used at once, it cost the
    // step a global-memory latency)
    auto fetch = [&](int h, int q_pos) -> float {
      if (q_pos >= p.Sq) return half == 0 ? -INFINITY : 0.f;
      const long long idx = ((long long)b * p.Hq + h) * p.Sq + q_pos;
      return half == 1 ? p.delta[idx] : p.lse[idx];
    };
    // a row that is not there or sees no key: P = exp2(s - inf) = 0
    auto staged = [&](float x) -> float {
      return half == 1 ? x * p.scale : (x == -INFINITY ? INFINITY : x * 1.4426950408889634f);
    };
    int h_next = hk * group + (n_iter > 0 ? it0 / n_q : 0), i_next = i_lo + (n_iter > 0 ? it0 % n_q : 0);
    bool ok = true;
    if (n_iter > 0) {
      sLD[half * BQ + r] = staged(fetch(h_next, i_next * BQ + r));
      __syncwarp();
      if (lane == 0) mbar_arrive(&ld_full[0]);
    }
    for (int it = 0; it < n_iter && ok; ++it) {
      const int q0 = i_next * BQ;
      if (++i_next > i_hi) { i_next = i_lo; ++h_next; }
      const float next = it + 1 < n_iter ? fetch(h_next, i_next * BQ + r) : 0.f;
      const bool need_mask = (kv0 + BKV > p.Skv) || (p.causal && kv0 + BKV - 1 > q0 + off) ||
                             (p.window > 0 && kv0 < q0 + BQ - 1 + off - p.window + 1);
      // visible queries of this key: columns [c_lo, c_hi)
      int c_lo = 0, c_hi = BQ;
      if (p.causal) c_lo = key - off - q0;
      if (p.window > 0) c_hi = key - off - q0 + p.window;
      if (key >= p.Skv) c_hi = c_lo = 0;
      if (!warp_wait(&ld_full[it & 1], (it >> 1) & 1, abort_flag, p.status, 89)) { ok = false; break; }
      const float* ld = sLD + (it & 1) * 2 * BQ + half * 64;
      if (!warp_wait(s_full, it & 1, abort_flag, p.status, 90)) { ok = false; break; }
      tc_fence_after();
      float pr[64];
      {
        uint32_t s[64];
        tmem_ld_32x32b_x32(tm_S + lane_base + half * 64, *reinterpret_cast<uint32_t(*)[32]>(&s[0]));
        tmem_ld_32x32b_x32(tm_S + lane_base + half * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&s[32]));
        tc_wait_ld();
        const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
          const float4 l4 = *reinterpret_cast<const float4*>(ld + i);
          const float2 a = ffma2(make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), sc2, make_float2(-l4.x, -l4.y));
          const float2 c = ffma2(make_float2(__uint_as_float(s[i + 2]), __uint_as_float(s[i + 3])), sc2, make_float2(-l4.z, -l4.w));
          pr[i] = ex2_approx(a.x); pr[i + 1] = ex2_approx(a.y); pr[i + 2] = ex2_approx(c.x); pr[i + 3] = ex2_approx(c.y);
        }
      }
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < 64; ++i) {
          const int col = half * 64 + i;
          if (col < c_lo || col >= c_hi) pr[i] = 0.f;
        }
      }
      {
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) pk[i] = pack_bf16x2(pr[2 * i], pr[2 * i + 1]);
        tmem_st_32x32b_x32(tm_S + lane_base + half * 64, pk);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
      }
      if (!warp_wait(dp_full, it & 1, abort_flag, p.status, 91)) { ok = false; break; }
      tc_fence_after();
      uint8_t* drow = sdS + half * (BKV * 128) + r * 128;       // 64 queries of key r
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t d[32];
        tmem_ld_32x32b_x32(tm_dP + lane_base + half * 64 + c * 32, d);
        tc_wait_ld();
        const float2 s2 = make_float2(p.scale, p.scale);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const float4 d0 = *reinterpret_cast<const float4*>(ld + BQ + c * 32 + g * 8);
          const float4 d1 = *reinterpret_cast<const float4*>(ld + BQ + c * 32 + g * 8 + 4);
          const float dl[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int i = g * 8 + 2 * j;
            const float2 t2 = ffma2(make_float2(__uint_as_float(d[i]), __uint_as_float(d[i + 1])), s2, make_float2(-dl[2 * j], -dl[2 * j + 1]));
            const float2 g2 = fmul2(make_float2(pr[c * 32 + i], pr[c * 32 + i + 1]), t2);
            w[j] = pack_bf16x2(g2.x, g2.y);
          }
          *reinterpret_cast<uint4*>(drow + (((c * 4 + g) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
      // the next step's staged value, into the buffer of step it - 1: every worker has left that step, since dP(it) was issued
      // after all of them had written dS(it - 1)
      if (it + 1 < n_iter) {
        sLD[((it + 1) & 1) * 2 * BQ + half * BQ + r] = staged(next);
        __syncwarp();
        if (lane == 0) mbar_arrive(&ld_full[(it + 1) & 1]);
      }
    }
    // ------------------------------ dK / dV epilogue ------------------------------
    // workers of half 0 write dK (staged in the dS tile), those of half 1 write dV (staged in the first Q stage)
    if (ok && n_iter > 0) ok = warp_wait(acc_done, 0, abort_flag, p.status, 92);
    if (ok) {
      tc_fence_after();
      uint8_t* tile = (half == 0) ? sdS : sQ;
      uint8_t* dst = tile + r * 128;
      const uint32_t src = (half == 0 ? tm_dK : tm_dV) + lane_base;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t v[32];
        if (n_iter > 0) { tmem_ld_32x32b_x32(src + c * 32, v); tc_wait_ld(); }
        else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0u;
        }
        if (parts > 1) {                        // fp32, as it is: attn_bwd_finish_kernel adds the parts up
          float4* o = reinterpret_cast<float4*>(p.partial + (((long long)bh * p.slots + p.slot[e]) * 2 + half) * BKV * HD + r * HD +
                                                c * 32);
#pragma unroll
          for (int g = 0; g < 8; ++g)
            o[g] = make_float4(__uint_as_float(v[4 * g]), __uint_as_float(v[4 * g + 1]), __uint_as_float(v[4 * g + 2]),
                               __uint_as_float(v[4 * g + 3]));
          continue;
        }
        uint8_t* blk = dst + (c / 2) * (BKV * 128);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int sw = (((c & 1) * 4 + g) ^ (r & 7)) << 4;
          *reinterpret_cast<uint4*>(blk + sw) = make_uint4(
              pack_bf16x2(__uint_as_float(v[8 * g]), __uint_as_float(v[8 * g + 1])),
              pack_bf16x2(__uint_as_float(v[8 * g + 2]), __uint_as_float(v[8 * g + 3])),
              pack_bf16x2(__uint_as_float(v[8 * g + 4]), __uint_as_float(v[8 * g + 5])),
              pack_bf16x2(__uint_as_float(v[8 * g + 6]), __uint_as_float(v[8 * g + 7])));
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && parts == 1 && kv0 + q * 32 < p.Skv) {
#pragma unroll
        for (int i = 0; i < NB; ++i)
          tma_store_4d(half == 0 ? &tmdK : &tmdV, tile + i * (BKV * 128) + q * 32 * 128, i * 64, hk, kv0 + q * 32, b);
        tma_store_commit();
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
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// dK and dV of a key tile that is cut from its parts, added in their order (no atomics: runs are bit-reproducible).
template <int HD>
__global__ void __launch_bounds__(256)
attn_bwd_finish_kernel(const float* __restrict__ partial, int cap, int slots, int Hkv, int Sq, int Skv, int group, int causal, int window,
                       const __grid_constant__ CutTiles cut, __nv_bfloat16* dk, __nv_bfloat16* dv, long long dk_row, long long dv_row,
                       long long dk_batch, long long dv_batch) {
  b200::begin_kernel();
  constexpr int VPR = HD / 8;
  const int bh = (int)blockIdx.x / cut.n, t = (int)blockIdx.x - bh * cut.n, jt = cut.tile[t];
  int i_lo, i_hi;
  const int parts = tile_parts(tile_steps(jt, Sq, Skv, group, causal, window, i_lo, i_hi), cap);
  const int b = bh / Hkv, hk = bh - b * Hkv;
  const float* src = partial + ((long long)bh * slots + cut.slot[t]) * 2 * BKV * HD;
  for (int i = blockIdx.y * 256 + threadIdx.x; i < 2 * BKV * VPR; i += gridDim.y * 256) {
    const int half = i / (BKV * VPR), r = i / VPR % BKV, c = i % VPR * 8, key = jt * BKV + r;
    if (key >= Skv) continue;
    float v[8] = {};
    for (int z = 0; z < parts; ++z) {
      const float* f = src + (long long)z * 2 * BKV * HD + i * 8;
      const float4 x = *reinterpret_cast<const float4*>(f), y = *reinterpret_cast<const float4*>(f + 4);
      v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w; v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
    }
    __nv_bfloat16* o = half == 0 ? dk + b * dk_batch + (long long)key * dk_row : dv + b * dv_batch + (long long)key * dv_row;
    *reinterpret_cast<uint4*>(o + hk * HD + c) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                                            pack_bf16x2(v[6], v[7]));
  }
}

// A CTA of one (batch, kv head) pair: a part of a key tile (tile << 3 | part), its cost in steps, and the slot of its sums.
struct Entry {
  int cost;
  uint16_t id, slot;
};

// The CTAs of one (batch, kv head) pair, longest first, and the tiles that are cut; 0 if cap cuts a tile into more than MAX_PARTS or
// there are more than MAX_ENTRIES.
int split_order(int Sq, int Skv, int group, int causal, int window, int cap, std::vector<Entry>& out, CutTiles& cut, int& slots) {
  const int num_kt = (Skv + BKV - 1) / BKV;
  out.clear();
  cut.n = slots = 0;
  for (int jt = 0; jt < num_kt; ++jt) {
    int lo, hi;
    const int steps = tile_steps(jt, Sq, Skv, group, causal, window, lo, hi), parts = tile_parts(steps, cap);
    if (parts > MAX_PARTS || (int)out.size() + parts > MAX_ENTRIES) return 0;
    if (parts > 1) {
      cut.tile[cut.n] = (uint16_t)jt;
      cut.slot[cut.n++] = (uint16_t)slots;
    }
    for (int z = 0; z < parts; ++z)
      out.push_back({steps * (z + 1) / parts - steps * z / parts + (parts > 1 ? 1 : 0), (uint16_t)(jt << 3 | z),
                     (uint16_t)(parts > 1 ? slots++ : 0)});
  }
  std::stable_sort(out.begin(), out.end(), [](const Entry& a, const Entry& b) { return a.cost > b.cost; });
  return (int)out.size();
}

// Bytes of the sums of the parts, and how many a plan may take: four times the bf16 dK and dV (two fp32 parts of every tile), or 32 MB.
// (Unbounded, a fuller chip was bought with any amount: 7168 tokens, 64 / 8 heads of 128, not causal, took 336 MB beside 28 MB of dK
// and dV for 4300 us, now 112 MB for the same 4300; 256 / 16 heads 672 MB, now none.  The shapes of split_cap's times take 6 to 24 MB,
// half of what slots for every tile took, in the same times.)
long long split_bytes(long long copies, int slots, int HD) { return copies * slots * 2 * BKV * HD * 4; }
long long split_bytes_limit(long long copies, int Skv, int HD) { return std::max(32ll << 20, 4 * copies * Skv * HD * 2 * 2); }

// Steps until the last SM is done: CTAs are taken in their order by the SM that is free first; each costs its steps and five more
// (set-up, first loads and the output: from the times of split and whole tiles at 2000 and 3000 tokens).
long long makespan(const std::vector<int>& cost, long long copies, int sms) {
  std::priority_queue<long long, std::vector<long long>, std::greater<long long>> sm;
  for (int i = 0; i < sms; ++i) sm.push(0);
  long long last = 0;
  for (int c : cost)
    for (long long i = 0; i < copies; ++i) {
      const long long t = sm.top() + c + 5;
      sm.pop();
      sm.push(t);
      if (t > last) last = t;
    }
  return last;
}

// Longest run of steps a CTA should take (0: whole key tiles).  One CTA takes a key tile's steps over all query heads of its
// group in series, so with few tiles the longest outlasts the average SM (2000 tokens, 64 / 8 heads, causal: 128 steps against 59).  Caps
// of 2/12 .. 11/12 of the longest tile are compared by the schedule they give; a split has to gain a twelfth of it.
// Backward, whole tiles -> split: 2000 x 64 / 8 heads of 64 267 -> 171 us, 800 tokens 130 -> 68; heads of 128: 3000 x 64 / 8 532 -> 433,
// 1024 x 32 / 8 103 -> 65, 2 x 1500 x 16 / 4 143 -> 106.  Parts of every tile alike (five at 2000 tokens) gained half as much, and cost
// where a part is a few steps long: 4 x 512 x 12 heads 34 -> 56, so those stay whole.
int split_cap(int B, int Sq, int Skv, int Hq, int Hkv, int HD, int causal, int window, int& slots) {
  const int num_kt = (Skv + BKV - 1) / BKV, group = Hq / Hkv, P = b200::sm_count();
  const long long copies = (long long)B * Hkv;
  if (num_kt > MAX_ENTRIES || copies * num_kt > 8 * P) return 0;
  std::vector<int> cost;
  long long longest = 0;
  for (int jt = 0; jt < num_kt; ++jt) {
    int lo, hi;
    cost.push_back(tile_steps(jt, Sq, Skv, group, causal, window, lo, hi));
    if (cost.back() > longest) longest = cost.back();
  }
  if (longest < 4 || longest * 12 > INT_MAX) return 0;
  long long best = makespan(cost, copies, P) * 11 / 12;
  int cap = 0, n;
  std::vector<Entry> order;
  CutTiles cut;
  for (int k = 2; k <= 11; ++k) {
    const int c = (int)((longest * k + 11) / 12);
    if (!split_order(Sq, Skv, group, causal, window, c, order, cut, n)) continue;
    if (split_bytes(copies, n, HD) > split_bytes_limit(copies, Skv, HD)) continue;
    cost.clear();
    for (const auto& e : order) cost.push_back(e.cost);
    const long long t = makespan(cost, copies, P) + 3;      // the launch that adds the parts up
    if (t < best) { best = t; cap = c; slots = n; }
  }
  return cap;
}

// delta[b, h, s] = sum_d O[b, s, h, d] * dO[b, s, h, d]; HD / 8 lanes per (token, head), one 16-byte load of either each (a
// warp per head with 4-byte loads: 8192 x 64 heads of 64 105 us, now 32; 32 heads of 128 58, now 33). VEC = false: rows that are not 16-byte aligned, 4 bytes
// at a time, in the same order of addition.
template <int HD, bool VEC>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout, float* __restrict__ delta, int B, int S,
                  int H, long long o_row, long long do_row, long long o_batch, long long do_batch) {
  b200::begin_kernel();
  constexpr int LANES = HD / 8;
  const long long w = (blockIdx.x * 256ll + threadIdx.x) / LANES;
  const int l = threadIdx.x % LANES;
  const long long total = (long long)B * S * H;
  const bool live = w < total;                 // (every lane takes part in the shuffles)
  const int h = live ? (int)(w % H) : 0;
  const long long t = live ? w / H : 0;
  const int s = (int)(t % S);
  const int b = (int)(t / S);
  float acc = 0.f;
  if (live) {
    const __nv_bfloat16* op = o + b * o_batch + (long long)s * o_row + h * HD + l * 8;
    const __nv_bfloat16* dp = dout + b * do_batch + (long long)s * do_row + h * HD + l * 8;
    uint32_t x[4], y[4];
    if (VEC) {
      const uint4 u = *reinterpret_cast<const uint4*>(op), v = *reinterpret_cast<const uint4*>(dp);
      x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
      y[0] = v.x; y[1] = v.y; y[2] = v.z; y[3] = v.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[j] = reinterpret_cast<const uint32_t*>(op)[j];
        y[j] = reinterpret_cast<const uint32_t*>(dp)[j];
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 p = unpack_bf16x2(x[j]), q = unpack_bf16x2(y[j]);
      acc += p.x * q.x + p.y * q.y;
    }
  }
#pragma unroll
  for (int off = LANES / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (live && l == 0) delta[((long long)b * H + h) * S + s] = acc;
}

int qkv_map(CUtensorMap* m, const void* ptr, int HD, int H, int S, int B, long long row, long long batch, int box_rows) {
  return b200::make_tmap_4d(m, b200::DT_BF16, ptr, HD, H, S, B, (uint64_t)HD * 2, (uint64_t)row * 2,
                            (uint64_t)batch * 2, 64, 1, box_rows, 1, b200::SWZ_128);
}

template <int HD>
int launch_bwd(const CUtensorMap* m, const BwdParams& p, cudaStream_t stream) {
  using SM = Smem<HD>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(attn_bwd_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::TOTAL);
    if (e != cudaSuccess) cudaGetLastError();  // clear the sticky error before reporting
    if (e != cudaSuccess) return b200::fail(611, "attn_bwd: cannot set %d bytes of shared memory: %s", SM::TOTAL,
                                            cudaGetErrorString(e));
    configured[dev & 63] = true;
  }
  const long long grid = (long long)(p.cap > 0 ? p.entries : (p.Skv + BKV - 1) / BKV) * p.Hkv * p.B;
  if (grid > 0x7fffffff) return b200::fail(612, "attn_bwd: %lld key tiles are too many", grid);
  b200::launch(attn_bwd_kernel<HD>, (unsigned)grid, NTHREADS, SM::TOTAL, stream, m[0], m[1], m[2], m[3], m[4], m[5], m[6], p);
  b200::count_launch();
  return b200::check_launch("attn_bwd");
}

}  // namespace

// delta = rowsum(O * dO), [B, H, S] fp32
B200_API int b200_attn_delta(const void* o, const void* dout, float* delta, int B, int S, int H, int HD,
                             long long o_row, long long do_row, long long o_batch, long long do_batch, void* stream) {
  const long long rows = (long long)B * S * H;
  if (rows == 0) return 0;
  if (HD != 64 && HD != 128) return b200::fail(613, "attn_delta: head dim %d (64 or 128)", HD);
  const bool vec = (((uintptr_t)o | (uintptr_t)dout) & 15) == 0 && ((o_row | do_row | o_batch | do_batch) & 7) == 0;
  const unsigned blocks = (unsigned)((rows * (HD / 8) + 255) / 256);
  auto fn = HD == 128 ? (vec ? attn_delta_kernel<128, true> : attn_delta_kernel<128, false>)
                      : (vec ? attn_delta_kernel<64, true> : attn_delta_kernel<64, false>);
  b200::launch(fn, blocks, 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta, B, S, H, o_row, do_row, o_batch,
                                               do_batch);
  b200::count_launch();
  return b200::check_launch("attn_delta");
}

// plan[0]: longest run of steps a CTA should take (0: whole key tiles); plan[1]: bytes of partial sums that this needs.
B200_API int b200_attn_bwd_plan(int B, int Sq, int Skv, int Hq, int Hkv, int HD, int causal, int window, long long* plan) {
  plan[0] = plan[1] = 0;
  if (B <= 0 || Sq <= 0 || Skv <= 0 || Hkv <= 0 || Hq <= 0 || Hq % Hkv != 0 || (HD != 64 && HD != 128)) return 0;
  try {
    int slots = 0;
    const int cap = split_cap(B, Sq, Skv, Hq, Hkv, HD, causal, window, slots);
    if (cap > 0) { plan[0] = cap; plan[1] = split_bytes((long long)B * Hkv, slots, HD); }
  } catch (const std::exception&) {
  }
  return 0;
}

// dq_acc: fp32 [B, Sq, Hq, HD] contiguous, zero-initialised by the caller (reduce-add target).
// dk / dv: bf16 [B, Skv, Hkv, HD] with their own pitches.  cap, workspace: 0 and null, or b200_attn_bwd_plan's cap and as many bytes,
// which nothing else uses until this call's work is done.
B200_API int b200_attn_bwd(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                           const float* delta, float* dq_acc, void* dk, void* dv, int B, int Sq, int Skv, int Hq,
                           int Hkv, int HD, long long q_row, long long k_row, long long v_row, long long do_row,
                           long long dk_row, long long dv_row, long long q_batch, long long k_batch,
                           long long v_batch, long long do_batch, long long dk_batch, long long dv_batch,
                           float scale, int causal, int window, int cap, void* workspace, long long workspace_bytes, void* stream) {
  if (HD != 64 && HD != 128) return b200::fail(610, "attn_bwd: head dim %d not supported (64 or 128)", HD);
  if (Hq % Hkv != 0) return b200::fail(610, "attn_bwd: Hq=%d not a multiple of Hkv=%d", Hq, Hkv);
  CUtensorMap m[7];
  int r;
  if ((r = qkv_map(&m[0], q, HD, Hq, Sq, B, q_row, q_batch, BQ))) return r;
  if ((r = qkv_map(&m[1], k, HD, Hkv, Skv, B, k_row, k_batch, BKV))) return r;
  if ((r = qkv_map(&m[2], v, HD, Hkv, Skv, B, v_row, v_batch, BKV))) return r;
  if ((r = qkv_map(&m[3], dout, HD, Hq, Sq, B, do_row, do_batch, BQ))) return r;
  if ((r = b200::make_tmap_4d(&m[4], b200::DT_F32, dq_acc, HD, Hq, Sq, B, (uint64_t)HD * 4, (uint64_t)Hq * HD * 4,
                              (uint64_t)Sq * Hq * HD * 4, 32, 1, 32, 1, b200::SWZ_128)))
    return r;
  if ((r = qkv_map(&m[5], dk, HD, Hkv, Skv, B, dk_row, dk_batch, 32))) return r;
  if ((r = qkv_map(&m[6], dv, HD, Hkv, Skv, B, dv_row, dv_batch, 32))) return r;
  BwdParams p;
  p.B = B; p.Hq = Hq; p.Hkv = Hkv; p.Sq = Sq; p.Skv = Skv;
  p.causal = causal; p.window = window;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.lse = lse; p.delta = delta;
  p.status = b200::status_ptr();
  // Causal: a key tile's work falls with its position, so all heads' early tiles go first (head after head leaves the last
  // head's longest CTAs running alone: 8192 x 32 / 8 heads of 128, delta and clearing included, 1512 us, this way 1310;
  // 4096 x 64 / 8 992 and 765; 4 x 2048 480 and 408; 3 x 1337 231 and 167).  Otherwise every tile costs the same and head after
  // head keeps that head's Q and dO in L2 (full, 8 x 512 x 24 heads 128 us, 134 the other way; 2 x 4608 x 24 1211 and 1345).
  // With a window the two are even (8192 x 64 / 8 of 64, window 128: 269 and 269; 2 x 8192 x 32, window 1024: 920 and 925).
  p.bh_group = (causal && window <= 0) ? B * Hkv : 1;
  const int group = Hq / Hkv;
  p.cap = 0; p.entries = 0; p.slots = 0; p.partial = (float*)workspace;
  CutTiles cut;
  cut.n = 0;
  if (cap > 0) {
    try {
      std::vector<Entry> order;
      p.entries = split_order(Sq, Skv, group, causal, window, cap, order, cut, p.slots);
      if (p.entries == 0 || workspace == nullptr || workspace_bytes < split_bytes((long long)B * Hkv, p.slots, HD))
        return b200::fail(613, "attn_bwd: cap %d and %lld bytes are not the plan of this shape", cap, workspace_bytes);
      for (int i = 0; i < p.entries; ++i) {
        p.order[i] = order[i].id;
        p.slot[i] = order[i].slot;
      }
    } catch (const std::exception& e) {
      return b200::fail(614, "attn_bwd: %s", e.what());
    }
    p.cap = cap;
  }
  if ((r = HD == 128 ? launch_bwd<128>(m, p, (cudaStream_t)stream) : launch_bwd<64>(m, p, (cudaStream_t)stream)) || cut.n == 0) return r;
  auto fin = HD == 128 ? attn_bwd_finish_kernel<128> : attn_bwd_finish_kernel<64>;
  b200::launch(fin, dim3((unsigned)(B * Hkv * cut.n), HD / 16), 256, 0, (cudaStream_t)stream, (const float*)p.partial, cap, p.slots, Hkv, Sq, Skv,
               group, causal, window, cut, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, dk_row, dv_row, dk_batch, dv_batch);
  b200::count_launch();
  return b200::check_launch("attn_bwd_finish");
}
