// Queries, keys and values of an MMDiT block from its fused projection, in one pass each way:
//
//   forward   q = rope(rmsnorm(qkv[:, 0]) * q_scale), k = rope(rmsnorm(qkv[:, 1]) * k_scale), v = qkv[:, 2]
//             from a token's row [3][H][D] (any row pitch) to the joint [B, S, H, D] tensors the attention reads, at
//             token offset s_off of its sample (the double blocks write two streams into one sequence)
//   backward  the gradient of that row from dq, dk, dv, and the two scale gradients
//
// The chain it replaces - slice copies, two norms, concatenation, clone + rotation, and the same backwards with a
// zero-filled gradient per slice - moved each of q, k, v six to eight times.  Bound by HBM: D / 8 lanes own a head row, a
// lane holds 4 columns of either half, so the rotation pairs are its own (no exchange) and the row sum is a few shuffles.
// The normalised value and its gradient stay in fp32 between the norm and the rotation.
// Measured for 8 samples of 512 tokens, 24 heads of 128, L2 flushed: 39 us forward (75 MB read, 75 written: 3.9 TB/s) and 77 us
// backward with the scale gradients (126 MB read, 75 written: 2.6 TB/s), for about 500 us a block of slices, clones, norms and
// concatenations, both directions together.  MMDiT training pass of 8 samples
// 12.8 -> 10.9 ms, sampling pass of one 2.43 -> 2.07 ms (21 launches fewer).
//
// Reference: the fused norm + RoPE of the FLUX submission (flux1/primus/config_common.sh:84-150).
#include "common.cuh"
#include "runtime.h"

namespace {

constexpr int NT = 256;

struct Shape {
  int B, S_part, S_all, s_off, H;
  long long ld;          // row pitch of qkv in elements
};

B200_DEVICE void ld4(const __nv_bfloat16* p, float (&f)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}
B200_DEVICE void st4(__nv_bfloat16* p, const float (&f)[4]) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
}
B200_DEVICE void ldf4(const float* p, float (&f)[4]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
}
template <int LANES>
B200_DEVICE float team_sum(float v) {
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// rstd: [tokens of the part][2][H]
template <int D>
__global__ void __launch_bounds__(NT)
qk_norm_rope_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ wq,
                        const __nv_bfloat16* __restrict__ wk, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                        __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ k, __nv_bfloat16* __restrict__ v,
                        float* __restrict__ rstd, Shape sh, float eps) {
  b200::begin_kernel();
  constexpr int LANES = D / 8, HALF = D / 2;
  const int l = threadIdx.x % LANES;
  const long long items = (long long)sh.B * sh.S_part * sh.H;
  const long long step = (long long)gridDim.x * (NT / LANES);
  const long long first = blockIdx.x * (long long)(NT / LANES) + threadIdx.x / LANES;
  const long long warp_first = __shfl_sync(0xffffffffu, (int)(threadIdx.x / LANES), 0) + blockIdx.x * (long long)(NT / LANES);
  float w[2][8];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const __nv_bfloat16* p = (i == 0 ? wq : wk);
    float a[4], b[4];
    ld4(p + l * 4, a);
    ld4(p + HALF + l * 4, b);
#pragma unroll
    for (int j = 0; j < 4; ++j) { w[i][j] = a[j]; w[i][4 + j] = b[j]; }
  }
  // every lane of a warp runs the same number of steps (the shuffles name all 32)
  for (long long off = 0; warp_first + off < items; off += step) {
    const long long it = first + off;
    const bool live = it < items;
    const long long t = live ? it / sh.H : 0;
    const int h = live ? (int)(it - t * sh.H) : 0;
    const int b = (int)(t / sh.S_part), s = sh.s_off + (int)(t - (long long)b * sh.S_part);
    const __nv_bfloat16* src = qkv + t * sh.ld + h * D + l * 4;
    const long long dst = (((long long)b * sh.S_all + s) * sh.H + h) * D + l * 4;
    float x[3][8];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      float a[4], c[4];
      ld4(src + (long long)i * sh.H * D, a);
      ld4(src + (long long)i * sh.H * D + HALF, c);
#pragma unroll
      for (int j = 0; j < 4; ++j) { x[i][j] = a[j]; x[i][4 + j] = c[j]; }
    }
    float cs[4], sn[4];
    ldf4(cos_t + (long long)s * HALF + l * 4, cs);
    ldf4(sin_t + (long long)s * HALF + l * 4, sn);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float ss = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += x[i][j] * x[i][j];
      const float r = rsqrtf(team_sum<LANES>(ss) / D + eps);
      if (live) {
        if (l == 0 && rstd != nullptr) rstd[(t * 2 + i) * sh.H + h] = r;
        float lo[4], hi[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float n0 = x[i][j] * r * w[i][j], n1 = x[i][4 + j] * r * w[i][4 + j];
          lo[j] = n0 * cs[j] - n1 * sn[j];
          hi[j] = n1 * cs[j] + n0 * sn[j];
        }
        __nv_bfloat16* o = (i == 0 ? q : k) + dst;
        st4(o, lo);
        st4(o + HALF, hi);
      }
    }
    if (live) {
      float lo[4], hi[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) { lo[j] = x[2][j]; hi[j] = x[2][4 + j]; }
      st4(v + dst, lo);
      st4(v + dst + HALF, hi);
    }
  }
}

// dqkv: the rows' gradient (pitch ld_d); partial: [gridDim.x][2][D] sums of the scale gradients over the CTA's rows
template <int D>
__global__ void __launch_bounds__(NT)
qk_norm_rope_bwd_kernel(const __nv_bfloat16* __restrict__ dq, const __nv_bfloat16* __restrict__ dk,
                        const __nv_bfloat16* __restrict__ dv, const __nv_bfloat16* __restrict__ qkv,
                        const __nv_bfloat16* __restrict__ wq, const __nv_bfloat16* __restrict__ wk,
                        const float* __restrict__ cos_t, const float* __restrict__ sin_t, const float* __restrict__ rstd,
                        __nv_bfloat16* __restrict__ dqkv, long long ld_d, float* __restrict__ partial, Shape sh) {
  b200::begin_kernel();
  constexpr int LANES = D / 8, HALF = D / 2, TEAMS = NT / LANES;
  __shared__ float acc[TEAMS][D];
  const int l = threadIdx.x % LANES, team = threadIdx.x / LANES;
  const long long items = (long long)sh.B * sh.S_part * sh.H;
  const long long step = (long long)gridDim.x * TEAMS;
  const long long first = blockIdx.x * (long long)TEAMS + team;
  const long long warp_first = __shfl_sync(0xffffffffu, team, 0) + blockIdx.x * (long long)TEAMS;
  float w[2][8], dw[2][8];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const __nv_bfloat16* p = (i == 0 ? wq : wk);
    float a[4], b[4];
    ld4(p + l * 4, a);
    ld4(p + HALF + l * 4, b);
#pragma unroll
    for (int j = 0; j < 4; ++j) { w[i][j] = a[j]; w[i][4 + j] = b[j]; dw[i][j] = dw[i][4 + j] = 0.f; }
  }
  for (long long off = 0; warp_first + off < items; off += step) {
    const long long it = first + off;
    const bool live = it < items;
    const long long t = live ? it / sh.H : 0;
    const int h = live ? (int)(it - t * sh.H) : 0;
    const int b = (int)(t / sh.S_part), s = sh.s_off + (int)(t - (long long)b * sh.S_part);
    const long long src = (((long long)b * sh.S_all + s) * sh.H + h) * D + l * 4;
    const __nv_bfloat16* xr = qkv + t * sh.ld + h * D + l * 4;
    __nv_bfloat16* out = dqkv + t * ld_d + h * D + l * 4;
    float cs[4], sn[4];
    ldf4(cos_t + (long long)s * HALF + l * 4, cs);
    ldf4(sin_t + (long long)s * HALF + l * 4, sn);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const __nv_bfloat16* dp = (i == 0 ? dq : dk) + src;
      float g0[4], g1[4], x0[4], x1[4];
      ld4(dp, g0);
      ld4(dp + HALF, g1);
      ld4(xr + (long long)i * sh.H * D, x0);
      ld4(xr + (long long)i * sh.H * D + HALF, x1);
      const float r = live ? rstd[(t * 2 + i) * sh.H + h] : 0.f;
      float xn[8], g[8], s1 = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float d0 = g0[j] * cs[j] + g1[j] * sn[j], d1 = g1[j] * cs[j] - g0[j] * sn[j];   // the inverse rotation
        xn[j] = x0[j] * r;
        xn[4 + j] = x1[j] * r;
        if (live) { dw[i][j] += d0 * xn[j]; dw[i][4 + j] += d1 * xn[4 + j]; }
        g[j] = d0 * w[i][j];
        g[4 + j] = d1 * w[i][4 + j];
        s1 += g[j] * xn[j] + g[4 + j] * xn[4 + j];
      }
      s1 = team_sum<LANES>(s1) / D;
      if (live) {
        float lo[4], hi[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) { lo[j] = r * (g[j] - xn[j] * s1); hi[j] = r * (g[4 + j] - xn[4 + j] * s1); }
        st4(out + (long long)i * sh.H * D, lo);
        st4(out + (long long)i * sh.H * D + HALF, hi);
      }
    }
    if (live) {
      *reinterpret_cast<uint2*>(out + 2ll * sh.H * D) = *reinterpret_cast<const uint2*>(dv + src);
      *reinterpret_cast<uint2*>(out + 2ll * sh.H * D + HALF) = *reinterpret_cast<const uint2*>(dv + src + HALF);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) { acc[team][l * 4 + j] = dw[i][j]; acc[team][HALF + l * 4 + j] = dw[i][4 + j]; }
    __syncthreads();
    if (threadIdx.x < D) {
      float t = 0.f;
      for (int m = 0; m < TEAMS; ++m) t += acc[m][threadIdx.x];
      partial[((long long)blockIdx.x * 2 + i) * D + threadIdx.x] = t;
    }
  }
}

// out[which][c] = sum_p partial[p][which][c] in a fixed order; 32 columns per CTA, a warp takes every eighth row
__global__ void __launch_bounds__(256)
scale_grad_kernel(const float* __restrict__ partial, int nparts, int D, float* __restrict__ out) {
  b200::begin_kernel();
  __shared__ float sm[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float s = 0.f;
#pragma unroll 4
  for (int p = warp; p < nparts; p += 8) s += partial[((long long)p * 2 + blockIdx.y) * D + c];
  sm[warp][lane] = s;
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 1; k < 8; ++k) s += sm[k][lane];
    out[blockIdx.y * D + c] = s;
  }
}

int bwd_grid(long long items, int D) {
  const long long need = (items + NT / (D / 8) - 1) / (NT / (D / 8)), cap = b200::sm_count() * 4ll;
  return (int)(need < cap ? need : cap);
}

int check(const char* what, int D, long long ld, int B, int S_part, int S_all, int s_off, int H) {
  if ((D != 64 && D != 128) || ld % 8 != 0 || B < 0 || S_part < 0 || H <= 0 || s_off < 0 || s_off + S_part > S_all)
    return b200::fail(1700, "%s: D=%d (64 or 128), pitch %lld (x8), B=%d S=%d of %d at %d, H=%d", what, D, ld, B, S_part, S_all, s_off, H);
  return 0;
}

}  // namespace

// qkv: rows [B * S_part] of [3][H][D] bf16 with pitch ld; wq / wk [D] bf16; cos / sin [S_all][D / 2] fp32; q / k / v:
// [B, S_all, H, D] contiguous, tokens s_off .. s_off + S_part of every sample are written; rstd [B * S_part][2][H] or null.
B200_API int b200_qk_norm_rope_fwd(const void* qkv, long long ld, const void* wq, const void* wk, const float* cos_t,
                                   const float* sin_t, void* q, void* k, void* v, float* rstd, int B, int S_part, int S_all,
                                   int s_off, int H, int D, float eps, void* stream) {
  if (int r = check("qk_norm_rope_fwd", D, ld, B, S_part, S_all, s_off, H)) return r;
  const long long items = (long long)B * S_part * H;
  if (items == 0) return 0;
  const Shape sh{B, S_part, S_all, s_off, H, ld};
  const long long need = (items + NT / (D / 8) - 1) / (NT / (D / 8)), cap = b200::sm_count() * 16ll;
  const int grid = (int)(need < cap ? need : cap);
  auto X = (const __nv_bfloat16*)qkv; auto Q = (const __nv_bfloat16*)wq; auto K = (const __nv_bfloat16*)wk;
  auto fn = D == 128 ? qk_norm_rope_fwd_kernel<128> : qk_norm_rope_fwd_kernel<64>;
  b200::launch(fn, grid, NT, 0, (cudaStream_t)stream, X, Q, K, cos_t, sin_t, (__nv_bfloat16*)q, (__nv_bfloat16*)k, (__nv_bfloat16*)v, rstd, sh, eps);
  b200::count_launch();
  return b200::check_launch("qk_norm_rope_fwd");
}

// Floats of scratch b200_qk_norm_rope_bwd needs.
B200_API long long b200_qk_norm_rope_scratch_elems(int B, int S_part, int H, int D) {
  return D == 64 || D == 128 ? 2ll * D * bwd_grid((long long)B * S_part * H, D) : 0;
}

// dq / dk / dv [B, S_all, H, D] contiguous; dqkv: rows of [3][H][D] with pitch ld_d; dscale [2][D] fp32 (q then k).
B200_API int b200_qk_norm_rope_bwd(const void* dq, const void* dk, const void* dv, const void* qkv, long long ld, const void* wq,
                                   const void* wk, const float* cos_t, const float* sin_t, const float* rstd, void* dqkv,
                                   long long ld_d, float* dscale, float* scratch, int B, int S_part, int S_all, int s_off, int H,
                                   int D, void* stream) {
  if (int r = check("qk_norm_rope_bwd", D, ld, B, S_part, S_all, s_off, H)) return r;
  if (ld_d % 8 != 0) return b200::fail(1700, "qk_norm_rope_bwd: gradient pitch %lld (x8)", ld_d);
  const long long items = (long long)B * S_part * H;
  cudaStream_t st = (cudaStream_t)stream;
  if (items == 0) {
    cudaMemsetAsync(dscale, 0, 2ll * D * sizeof(float), st);
    return 0;
  }
  const Shape sh{B, S_part, S_all, s_off, H, ld};
  const int grid = bwd_grid(items, D);
  auto fn = D == 128 ? qk_norm_rope_bwd_kernel<128> : qk_norm_rope_bwd_kernel<64>;
  b200::launch(fn, grid, NT, 0, st, (const __nv_bfloat16*)dq, (const __nv_bfloat16*)dk, (const __nv_bfloat16*)dv, (const __nv_bfloat16*)qkv,
                          (const __nv_bfloat16*)wq, (const __nv_bfloat16*)wk, cos_t, sin_t, rstd, (__nv_bfloat16*)dqkv, ld_d, scratch, sh);
  b200::launch(scale_grad_kernel, dim3(D / 32, 2), 256, 0, st, scratch, grid, D, dscale);
  b200::count_launch(2);
  return b200::check_launch("qk_norm_rope_bwd");
}
