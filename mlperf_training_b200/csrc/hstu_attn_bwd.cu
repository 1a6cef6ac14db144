// Jagged HSTU attention backward for sm_100a.  With P = silu(alpha S) / N * mask and S = Q K^T:
//
//   dV += P^T dO      dP = dO V^T      dS = dP * silu'(alpha S) * alpha / N * mask
//   dQ  = dS K        dK += dS^T Q
//
// One CTA per (sequence, head, 128-key tile) loops over the query tiles that see those keys; the engine of
// attention_bwd.cu: transposed scores (a worker thread owns a key row), P^T back in TMEM as the operand of dV, dS^T once in
// shared memory for dK and dQ, Q double-buffered, warps of their own for the fp32 TMA reduce-add of dQ, and per step
//     [P^T(i) written]  dV(i)   [dS^T(i) written]  dQ(i)  S(i+1)  dK(i)  [dQ(i) drained]  dP(i+1)
// No row statistics are needed, so nothing but Q, K, V, dO is read.  Mask and jagged layout as in hstu_attn_fwd.cu.
// Measured with the clearing and conversion around it, before (queries as rows, P and dS through shared memory, drained by
// the workers) -> now: 128 users of median 512 tokens, 4 heads of 128: 1345 -> 1018 us; 12 users of median 700: 235 -> 163.
// The kernel alone, 128 users: 882 us with the mask on every tile past a sequence's end, 715 with it on the diagonal's.
//
// Math oracle: autograd of generative_recommenders/ops/pytorch/pt_hstu_attention.py:130-187; the
// reference's production kernels are generative_recommenders/ops/flydsl/hstu_bwd_dkdv.py and
// generative_recommenders/ops/triton/triton_hstu_attention.py (_hstu_attn_bwd).
#include "common.cuh"
#include "runtime.h"

namespace {

constexpr int BQ = 128;
constexpr int BKV = 128;
constexpr int NTHREADS = 512;  // warp 0 TMA, 1 MMA (2, 3 complete the warpgroup), 4-7 dQ drain, 8-15 P / dS workers
// 4 x 128 threads launch with 128 registers each: 88 + 88 + 2 x 168
constexpr int REGS_OTHER = 88, REGS_WORKER = 168;
constexpr int STG = 4096;  // dQ staging chunk: 32 rows x 32 fp32 (two per drain warp)

struct HstuBwdParams {
  int max_len, H, contextual;
  float alpha;
  const int* offsets;
  const int* num_targets;
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  long long dk_row, dv_row;
  int tiles_outer;          // grid order: 1 = key tile slowest, 0 = (sequence, head) slowest
  int num_bh, num_kt;       // (sequence, head) pairs and key tiles: the grid is their product along x, which has no 65,535 limit
  int* status;
};

B200_DEVICE float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int HD>
struct Smem {
  static constexpr int T_BYTES = 128 * HD * 2;        // K, V, Q (two stages), dO tiles
  static constexpr int DS_BYTES = BQ * BKV * 2;       // dS^T tile
  static constexpr int STG_BYTES = 8 * STG;
  static constexpr int TOTAL = 5 * T_BYTES + DS_BYTES + STG_BYTES + 1024 + 256;
};

template <int HD>
__global__ void __launch_bounds__(NTHREADS, 1)
hstu_attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                const __grid_constant__ CUtensorMap tmdQ, const HstuBwdParams p) {
  b200::begin_kernel();
  using SM = Smem<HD>;
  constexpr int NB = HD / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + SM::T_BYTES;
  uint8_t* sQ = sV + SM::T_BYTES;           // two stages
  uint8_t* sdO = sQ + 2 * SM::T_BYTES;
  uint8_t* sdS = sdO + SM::T_BYTES;
  uint8_t* sStg = sdS + SM::DS_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStg + SM::STG_BYTES);
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
  uint64_t* acc_done = bars + 13;   // every MMA of this CTA finished
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int x = (int)blockIdx.x;
  const int jt = p.tiles_outer ? x / p.num_bh : x % p.num_kt;
  const int bh = p.tiles_outer ? x % p.num_bh : x / p.num_kt;
  const int hk = bh % p.H, b = bh / p.H;
  const int row_base = p.offsets[b];
  const int len = p.offsets[b + 1] - row_base;
  const int kv0 = jt * BKV;
  if (kv0 >= len) return;     // grid is sized by the maximum length
  const int n_tgt = p.num_targets ? p.num_targets[b] : 0;
  const int ctx = p.contextual;
  const int hist_end = len - n_tgt;
  const int max_id = hist_end - (ctx > 0 ? ctx - 1 : 0);
  // query tiles that see at least one key of this tile: the causal range, plus the earlier tiles that
  // hold contextual rows (they see every history column)
  const int i_lo = kv0 / BQ, i_hi = (len - 1) / BQ;
  const int extra = min((ctx + BQ - 1) / BQ, i_lo);
  const int n_q = (i_hi - i_lo + 1) + extra;
  const int n_iter = n_q;
  auto q_tile = [&](int it) { return it < extra ? it : i_lo + it - extra; };

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1); mbar_init(do_full, 1); mbar_init(do_empty, 1); mbar_init(s_full, 1); mbar_init(dp_full, 1);
    mbar_init(p_full, 8); mbar_init(ds_full, 8); mbar_init(dq_full, 1); mbar_init(dq_drained, 4); mbar_init(acc_done, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
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
    if (lane == 0) {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO);
      mbar_expect_tx(kv_full, 2 * SM::T_BYTES);
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        tma_load_3d(sK + i * (BKV * 128), &tmK, kv_full, i * 64, hk, row_base + kv0);
        tma_load_3d(sV + i * (BKV * 128), &tmV, kv_full, i * 64, hk, row_base + kv0);
      }
      for (int it = 0; it < n_iter; ++it) {
        const int q0 = q_tile(it) * BQ;
        const int st = it & 1;
        if (!mbar_wait(&q_empty[st], ((it >> 1) & 1) ^ 1, abort_flag, p.status, 70)) break;
        mbar_expect_tx(&q_full[st], SM::T_BYTES);
#pragma unroll
        for (int i = 0; i < NB; ++i) tma_load_3d(sQ + st * SM::T_BYTES + i * (BQ * 128), &tmQ, &q_full[st], i * 64, hk, row_base + q0);
        if (!mbar_wait(do_empty, (it & 1) ^ 1, abort_flag, p.status, 71)) break;
        mbar_expect_tx(do_full, SM::T_BYTES);
#pragma unroll
        for (int i = 0; i < NB; ++i) tma_load_3d(sdO + i * (BQ * 128), &tmdO, do_full, i * 64, hk, row_base + q0);
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
      const int q0 = q_tile(it) * BQ;
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
            if (q0 + q * 32 < len) tma_reduce_add_3d(&tmdQ, stg + cc * STG, c2 * 64 + cc * 32, hk, row_base + q0 + q * 32);
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
    const int kp = kv0 + r;                   // this thread's key
    // Queries that see key kp: q >= q_begin (id(q) > id(k) is one comparison of q), q == kp, and contextual rows q < ctx_end.
    // A key past the sequence's end belongs to the next sequence: nobody sees it.
    constexpr int NONE = 0x3fffffff;
    const int id_off = ctx - (ctx > 0 ? 1 : 0);
    const int k_id = min(max(kp - id_off, 0), max_id);
    const int q_begin = (kp < len && k_id < max_id) ? k_id + 1 + id_off : NONE;
    const int ctx_end = (ctx > 0 && max_id >= 0 && kp < hist_end) ? (max_id == 0 ? NONE : id_off + 1) : 0;
    const int q_self = kp < len ? kp : -1;
    const float ha = 0.5f * p.alpha, inv_n = 1.0f / (float)p.max_len, an = p.alpha * inv_n;
    bool ok = true;
    for (int it = 0; it < n_iter && ok; ++it) {
      const int q0 = q_tile(it) * BQ;
      // a tile whose every (query, key) pair is visible needs no element mask: ids grow with the position, so it
      // is enough that the tile's first query is later than its last key, and that the query tile lies inside the sequence
      // (then its keys do)
      const int first_q_id = min(max(q0 - id_off, 0), max_id);
      const bool need_mask = !(q0 + BQ <= len && first_q_id > 0 && kv0 + BKV <= first_q_id + id_off);
      if (!warp_wait(s_full, it & 1, abort_flag, p.status, 90)) { ok = false; break; }
      tc_fence_after();
      float f[64];                            // dS / dP of this key and the half's queries
      {
        uint32_t s[64];
        tmem_ld_32x32b_x32(tm_S + lane_base + half * 64, *reinterpret_cast<uint32_t(*)[32]>(&s[0]));
        tmem_ld_32x32b_x32(tm_S + lane_base + half * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&s[32]));
        tc_wait_ld();
        const float2 ha2 = make_float2(ha, ha), an2 = make_float2(an, an), hn2 = make_float2(inv_n, inv_n);
        const float2 one = make_float2(1.f, 1.f), half2 = make_float2(0.5f, 0.5f), neg = make_float2(-1.f, -1.f);
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          // P = silu(a s) / N ; dS = dP * silu'(a s) * a / N   (sig = (1 + tanh(a s / 2)) / 2)
          const float2 hx = fmul2(make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), ha2);
          const float2 sig = ffma2(make_float2(tanh_approx(hx.x), tanh_approx(hx.y)), half2, half2);
          const float2 x = fadd2(hx, hx);
          const float2 pv = fmul2(fmul2(x, sig), hn2);
          const float2 fv = fmul2(fmul2(sig, ffma2(x, ffma2(sig, neg, one), one)), an2);
          s[i] = __float_as_uint(pv.x); s[i + 1] = __float_as_uint(pv.y);
          f[i] = fv.x; f[i + 1] = fv.y;
        }
        if (need_mask) {
          const int qc = q0 + half * 64;
          const int beg = q_begin - qc, self = q_self - qc, end = len - qc, cend = ctx_end - qc;
          if (ctx == 0) {
#pragma unroll
            for (int i = 0; i < 64; ++i)
              if ((i < beg && i != self) || i >= end) { s[i] = 0u; f[i] = 0.f; }
          } else {
#pragma unroll
            for (int i = 0; i < 64; ++i)
              if ((i < beg && i != self && i >= cend) || i >= end) { s[i] = 0u; f[i] = 0.f; }
          }
        }
        uint32_t pk[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) pk[j] = pack_bf16x2(__uint_as_float(s[2 * j]), __uint_as_float(s[2 * j + 1]));
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
        if (need_mask) {
          // (rows past the end belong to the next sequence: what it holds must not reach 0 * inf)
#pragma unroll
          for (int i = 0; i < 32; ++i) if (f[c * 32 + i] == 0.f) d[i] = 0u;
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int i = g * 8 + 2 * j;
            const float2 g2 = fmul2(make_float2(f[c * 32 + i], f[c * 32 + i + 1]), make_float2(__uint_as_float(d[i]), __uint_as_float(d[i + 1])));
            w[j] = pack_bf16x2(g2.x, g2.y);
          }
          *reinterpret_cast<uint4*>(drow + (((c * 4 + g) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
    }
    // ------------------------------ dK / dV epilogue ------------------------------
    // workers of half 0 write dK, those of half 1 write dV; guarded row stores: rows past the
    // sequence end belong to the next sequence
    if (ok && n_iter > 0) ok = warp_wait(acc_done, 0, abort_flag, p.status, 92);
    if (ok) {
      tc_fence_after();
      const int k_pos = kv0 + r;
      __nv_bfloat16* dst = (half == 0 ? p.dk : p.dv) + (long long)(row_base + k_pos) * (half == 0 ? p.dk_row : p.dv_row) + hk * HD;
      const uint32_t src = (half == 0 ? tm_dK : tm_dV) + lane_base;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(src + c * 32, v);
        tc_wait_ld();
        if (k_pos < len) {
#pragma unroll
          for (int g = 0; g < 4; ++g)
            *reinterpret_cast<uint4*>(dst + c * 32 + g * 8) = make_uint4(
                pack_bf16x2(__uint_as_float(v[8 * g]), __uint_as_float(v[8 * g + 1])),
                pack_bf16x2(__uint_as_float(v[8 * g + 2]), __uint_as_float(v[8 * g + 3])),
                pack_bf16x2(__uint_as_float(v[8 * g + 4]), __uint_as_float(v[8 * g + 5])),
                pack_bf16x2(__uint_as_float(v[8 * g + 6]), __uint_as_float(v[8 * g + 7])));
        }
      }
    }
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

template <int HD>
int launch_hstu_bwd(const CUtensorMap* m, const HstuBwdParams& p, cudaStream_t stream) {
  using SM = Smem<HD>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(hstu_attn_bwd_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::TOTAL);
    if (e != cudaSuccess) { cudaGetLastError(); return b200::fail(1211, "hstu_attn_bwd: cannot set %d bytes of shared memory: %s", SM::TOTAL, cudaGetErrorString(e)); }
    configured[dev & 63] = true;
  }
  const long long grid = (long long)p.num_bh * p.num_kt;
  if (grid > 0x7fffffff) return b200::fail(1212, "hstu_attn_bwd: %lld key tiles are too many", grid);
  b200::launch(hstu_attn_bwd_kernel<HD>, (unsigned)grid, NTHREADS, SM::TOTAL, stream, m[0], m[1], m[2], m[3], m[4], p);
  b200::count_launch();
  return b200::check_launch("hstu_attn_bwd");
}

}  // namespace

// q / k / v / dout: jagged [L, H, HD] bf16 views; dq_acc: fp32 [L, H, HD] contiguous, zeroed by the
// caller (reduce-add target); dk / dv: bf16 [L, H, HD] views (every valid row is written).
B200_API int b200_hstu_attn_bwd(const void* q, const void* k, const void* v, const void* dout, float* dq_acc, void* dk,
                                void* dv, const int* offsets, const int* num_targets, int B, long long L, int H, int HD,
                                int max_len, int contextual, long long q_row, long long k_row, long long v_row,
                                long long do_row, long long dk_row, long long dv_row, float alpha, void* stream) {
  if (HD != 64 && HD != 128) return b200::fail(1210, "hstu_attn_bwd: head dim %d not supported (64 or 128)", HD);
  if (L == 0 || B == 0) return 0;
  CUtensorMap m[5];
  int r;
  auto mk = [&](CUtensorMap* t, const void* ptr, long long row, int box) {
    return b200::make_tmap_3d(t, b200::DT_BF16, ptr, HD, H, L, (uint64_t)HD * 2, (uint64_t)row * 2, 64, 1, box, b200::SWZ_128);
  };
  if ((r = mk(&m[0], q, q_row, BQ))) return r;
  if ((r = mk(&m[1], k, k_row, BKV))) return r;
  if ((r = mk(&m[2], v, v_row, BKV))) return r;
  if ((r = mk(&m[3], dout, do_row, BQ))) return r;
  if ((r = b200::make_tmap_3d(&m[4], b200::DT_F32, dq_acc, HD, H, L, (uint64_t)HD * 4, (uint64_t)H * HD * 4, 32, 1, 32, b200::SWZ_128))) return r;
  HstuBwdParams p;
  p.max_len = max_len; p.H = H; p.contextual = contextual; p.alpha = alpha;
  p.offsets = offsets; p.num_targets = num_targets;
  p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv; p.dk_row = dk_row; p.dv_row = dv_row;
  p.status = b200::status_ptr();
  // Early key tiles see the most queries.  With few sequences their longest CTAs go first over all of them (4 heads of 128,
  // pairs slowest and tiles slowest: 12 users of median 700 171 and 163 us, 40 of median 200 165 and 144); with several chips of
  // (sequence, head) pairs one pair after the other keeps its Q and dO in L2 (128 of median 512: 1018 and 1099).  In between
  // the lengths decide, by 5 % at most: 45 of median 512 391 and 382, 60 493 and 517, 74 603 and 636, 74 of median 200 264 and
  // 256; the line lies at two chips of pairs.
  p.num_bh = H * B;
  p.num_kt = (max_len + BKV - 1) / BKV;
  p.tiles_outer = p.num_bh <= 2 * b200::sm_count() ? 1 : 0;
  if (HD == 128) return launch_hstu_bwd<128>(m, p, (cudaStream_t)stream);
  return launch_hstu_bwd<64>(m, p, (cudaStream_t)stream);
}
