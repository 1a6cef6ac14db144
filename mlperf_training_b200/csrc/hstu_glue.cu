// HSTU layer glue between the jagged attention and the output projection, one pass each way:
//
//   forward   u = silu(u_raw);  n = LayerNorm(attn) * w + b;  cat = [u | attn | u * n]        ([T, 3D] bf16)
//   backward  from dcat = [du' | da' | dy]:
//             du_raw = (du' + dy * n) * silu'(u_raw)
//             dattn  = da' + LayerNorm_bwd(dy * u)
//             dw    += sum_t (dy * u) * xhat,   db += sum_t dy * u
//
// u_raw is a column block of the fused uvqk projection (row pitch given), so the kernel reads it in
// place; du_raw is written with its own pitch so it can land inside the gradient of that projection.
// D = 256, 512 or 768: forward gives a row to a warp, backward to D / 256 warps.  The weight / bias gradients are kept per
// lane in registers over all rows the warp visits, summed over the CTA's warps in a fixed order and written as one partial row
// per CTA that a second kernel adds up: no atomics, bit-reproducible.
//
// Dropout of the concatenation (rate p, survivors scaled by 1 / (1 - p)) is part of both passes: the keep
// mask comes from a Philox stream keyed by (seed, row, lane), so backward regenerates it instead of
// reading a stored mask.
//
// Replaces the chain the reference fuses as "layer norm * u (+ dropout)" before the output linear
// (generative_recommenders/ops/triton/triton_hstu_linear.py: _ln_mul_dropout_fwd / _ln_mul_dropout_bwd,
// with concat_ux) and the SiLU of u (generative_recommenders/ops/hstu_compute.py: hstu_preprocess_and_attention).
#include <curand_kernel.h>

#include "common.cuh"
#include "runtime.h"

namespace {

constexpr int GATE_CTAS = 2;   // resident CTAs an SM, either way: with three the kernels spill (forward 80 us, backward 134)
constexpr int GV = 3;   // vectors of 8 per lane -> D <= 768

B200_DEVICE void unpack8(const uint4& u, float (&f)[8]) {
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
B200_DEVICE void ld8(const __nv_bfloat16* p, float (&f)[8]) { unpack8(*reinterpret_cast<const uint4*>(p), f); }
B200_DEVICE void st8(__nv_bfloat16* p, const float (&f)[8]) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                                            pack_bf16x2(f[6], f[7]));
}
B200_DEVICE float rbf(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// Dropout of 8 adjacent elements: section (0 = u, 1 = attn, 2 = y) of vector i of this lane's row.  Every 32-bit Philox word
// decides two elements: a 16-bit half is compared with thr = round(p * 65536), so the rate is p to within 2^-17.  Block
// 3 * i + section of the stream (seed, row * 32 + lane) is drawn by itself, where its 8 elements are scaled: no generator state
// is carried and no mask assembled (which took a third of the forward's instructions).
B200_DEVICE void drop8(float (&f)[8], unsigned thr, float inv_keep, unsigned long long seed, long long row, int lane, int i,
                       int section) {
  const unsigned long long sub = (unsigned long long)row * 32 + lane;
  const uint4 r = curand_Philox4x32_10(make_uint4(3 * i + section, 0, (unsigned)sub, (unsigned)(sub >> 32)),
                                       make_uint2((unsigned)seed, (unsigned)(seed >> 32)));
  const unsigned wv[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    f[2 * k] = (wv[k] & 0xffffu) >= thr ? f[2 * k] * inv_keep : 0.f;
    f[2 * k + 1] = (wv[k] >> 16) >= thr ? f[2 * k + 1] * inv_keep : 0.f;
  }
}

// A warp per row; the next row's vectors are in flight while this one is computed: the loads' latency bounded it (40,000
// rows of 512, dropout 0.2: 88 us, now 70, without dropout 69 and 45; 32 us is what the bytes take, the random words bound it).
template <int NV>
__global__ void __launch_bounds__(256, GATE_CTAS)
gate_cat_fwd_kernel(const __nv_bfloat16* __restrict__ u_raw, long long ld_u, const __nv_bfloat16* __restrict__ attn,
                    const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
                    __nv_bfloat16* __restrict__ cat, float* __restrict__ mean_out, float* __restrict__ rstd_out, int T,
                    float eps, float p, unsigned thr, unsigned long long seed) {
  b200::begin_kernel();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int D = NV * 256;
  const float inv_keep = 1.f / (1.f - p);
  const long long step = (long long)gridDim.x * 8;
  long long row = (long long)blockIdx.x * 8 + warp;
  uint4 na[NV], nu[NV];
  if (row < T)
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      na[i] = *reinterpret_cast<const uint4*>(attn + row * D + (lane + 32 * i) * 8);
      nu[i] = *reinterpret_cast<const uint4*>(u_raw + row * ld_u + (lane + 32 * i) * 8);
    }
  for (; row < T; row += step) {
    float a[NV][8];
    uint4 uu[NV];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      unpack8(na[i], a[i]);
      uu[i] = nu[i];
    }
    if (row + step < T)
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        na[i] = *reinterpret_cast<const uint4*>(attn + (row + step) * D + (lane + 32 * i) * 8);
        nu[i] = *reinterpret_cast<const uint4*>(u_raw + (row + step) * ld_u + (lane + 32 * i) * 8);
      }
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) s += a[i][j];
    const float mean = warp_sum(s) / D;
    float var = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) { const float d = a[i][j] - mean; var += d * d; }
      }
    const float rstd = rsqrtf(warp_sum(var) / D + eps);
    if (lane == 0) { mean_out[row] = mean; rstd_out[row] = rstd; }
    __nv_bfloat16* out = cat + row * 3 * D;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = (lane + 32 * i) * 8;
        float ur[8], w8[8], b8[8], u[8], y[8];
        unpack8(uu[i], ur);
        ld8(w + c, w8);
        ld8(b + c, b8);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          u[j] = rbf(ur[j] / (1.f + __expf(-ur[j])));
          const float n = rbf((a[i][j] - mean) * rstd * w8[j] + b8[j]);
          y[j] = u[j] * n;
        }
        if (thr != 0) {
          drop8(u, thr, inv_keep, seed, row, lane, i, 0);
          drop8(a[i], thr, inv_keep, seed, row, lane, i, 1);
          drop8(y, thr, inv_keep, seed, row, lane, i, 2);
        }
        st8(out + c, u);
        st8(out + D + c, a[i]);
        st8(out + 2 * D + c, y);
      }
  }
}

template <int NV>
struct BwdShape {
  static constexpr int TEAMS = NV == 3 ? 2 : 8 / NV, THREADS = TEAMS * NV * 32;
};

// NV warps share a row, 8 columns a lane: with one warp per row the vectors, the weight gradients and the row's intermediate
// values did not fit the registers (spills, 16 warps an SM, nothing in flight ahead).  The next row is loaded while this one is
// computed; the row's two sums cross the warps through shared memory, two buffers in turn, one barrier a row.
// (40,000 rows of 512, dropout 0.2, with the sum over CTAs: 159 us, now 97, without dropout 67; 45 us is what the bytes take.)
template <int NV>
__global__ void __launch_bounds__(BwdShape<NV>::THREADS, GATE_CTAS)
gate_cat_bwd_kernel(const __nv_bfloat16* __restrict__ dcat, const __nv_bfloat16* __restrict__ u_raw, long long ld_u,
                    const __nv_bfloat16* __restrict__ attn, const __nv_bfloat16* __restrict__ w,
                    const __nv_bfloat16* __restrict__ b, const float* __restrict__ mean_in,
                    const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ du_raw, long long ld_du,
                    __nv_bfloat16* __restrict__ dattn, float* __restrict__ partial, int T, float p, unsigned thr,
                    unsigned long long seed) {
  b200::begin_kernel();
  constexpr int D = NV * 256, TEAMS = BwdShape<NV>::TEAMS;
  __shared__ float acc[TEAMS][2][D];
  __shared__ float2 red[TEAMS][2][NV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int team = warp / NV, vec = warp % NV;
  const int c = (lane + 32 * vec) * 8;
  const float inv_keep = 1.f / (1.f - p);
  const uint4 uw = *reinterpret_cast<const uint4*>(w + c), ub = *reinterpret_cast<const uint4*>(b + c);
  float gw[8] = {}, gb[8] = {};
  const long long step = (long long)gridDim.x * TEAMS;
  long long row = (long long)blockIdx.x * TEAMS + team;
  uint4 nu, na, ny, nd, nx;
  float nmean = 0.f, nrstd = 0.f;
  auto fetch = [&](long long r) {
    const __nv_bfloat16* dc = dcat + r * 3 * D + c;
    nu = *reinterpret_cast<const uint4*>(u_raw + r * ld_u + c);
    na = *reinterpret_cast<const uint4*>(attn + r * D + c);
    nd = *reinterpret_cast<const uint4*>(dc);
    nx = *reinterpret_cast<const uint4*>(dc + D);
    ny = *reinterpret_cast<const uint4*>(dc + 2 * D);
    nmean = mean_in[r];
    nrstd = rstd_in[r];
  };
  if (row < T) fetch(row);
  for (int buf = 0; row < T; row += step, buf ^= 1) {
    const float mean = nmean, rstd = nrstd;
    float ur[8], xn[8], dy[8], du[8], w8[8], b8[8], g[8], o[8];
    const uint4 ux = nx;
    unpack8(nu, ur);
    unpack8(na, xn);
    unpack8(ny, dy);
    unpack8(nd, du);
    if (row + step < T) fetch(row + step);
    unpack8(uw, w8);
    unpack8(ub, b8);
    if (thr != 0) {
      drop8(du, thr, inv_keep, seed, row, lane, vec, 0);
      drop8(dy, thr, inv_keep, seed, row, lane, vec, 2);
    }
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sg = 1.f / (1.f + __expf(-ur[j]));
      const float u = rbf(ur[j] * sg);
      xn[j] = (xn[j] - mean) * rstd;
      const float n = rbf(xn[j] * w8[j] + b8[j]);
      const float dn = dy[j] * u;
      gw[j] += dn * xn[j];
      gb[j] += dn;
      g[j] = dn * w8[j];
      s1 += g[j] * xn[j];
      s2 += g[j];
      o[j] = (du[j] + dy[j] * n) * (sg * (1.f + ur[j] * (1.f - sg)));
    }
    st8(du_raw + row * ld_du + c, o);
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (NV > 1) {
      if (lane == 0) red[team][buf][vec] = make_float2(s1, s2);
      asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(NV * 32) : "memory");
      s1 = s2 = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) { const float2 v = red[team][buf][i]; s1 += v.x; s2 += v.y; }
    }
    s1 /= D;
    s2 /= D;
    float da[8];
    unpack8(ux, da);
    if (thr != 0) drop8(da, thr, inv_keep, seed, row, lane, vec, 1);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = da[j] + rstd * (g[j] - xn[j] * s1 - s2);
    st8(dattn + row * D + c, o);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) { acc[team][0][c + j] = gw[j]; acc[team][1][c + j] = gb[j]; }
  __syncthreads();
  float* pw = partial + (long long)blockIdx.x * 2 * D;
  for (int k = threadIdx.x; k < 2 * D; k += BwdShape<NV>::THREADS) {
    float sum = 0.f;
#pragma unroll
    for (int t = 0; t < TEAMS; ++t) sum += (&acc[t][0][0])[k];
    pw[k] = sum;
  }
}

// Sum of the CTAs' partial rows: 32 of the 2 D columns a CTA, a warp every eighth row with eight in flight.  (One thread per
// column over all rows: 46 us for 296 rows of 1024, now 5.)
__global__ void __launch_bounds__(256)
gate_cat_reduce_kernel(const float* __restrict__ partial, int nparts, int D, float* __restrict__ dw, float* __restrict__ db,
                       int accumulate) {
  b200::begin_kernel();
  __shared__ float sm[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;                    // (D is a multiple of 256)
  float s = 0.f;
#pragma unroll 8
  for (int p = warp; p < nparts; p += 8) s += partial[(long long)p * 2 * D + c];
  sm[warp][lane] = s;
  __syncthreads();
  if (warp != 0) return;
  s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += sm[k][lane];
  float* out = c < D ? dw + c : db + c - D;
  *out = accumulate ? *out + s : s;
}

// Rows of [L, width] (pitch ld) that the attention does not write, set to zero: those of no sequence (before offsets[0], from
// offsets[B] on; with no sequence, B = 0, all of them) and those of a sequence past `cover` (the rows its grid reaches).  CTA b < B:
// sequence b; the others share the rest.
// (Clearing a whole output of 105,000 x 512 took 28 us a tensor, this 2.)
__global__ void __launch_bounds__(256)
zero_uncovered_rows_kernel(__nv_bfloat16* __restrict__ buf, const int* __restrict__ offsets, int B, long long L, long long ld, int vpr,
                           long long cover) {
  b200::begin_kernel();
  long long lo, hi;
  int part = 0, parts = 1;
  if ((int)blockIdx.x < B) {
    lo = offsets[blockIdx.x] + cover;
    hi = offsets[blockIdx.x + 1];
  } else {
    part = (int)blockIdx.x - B;
    parts = (int)gridDim.x - B;
    lo = offsets[B];
    hi = L;
    const long long head = offsets[0];
    for (long long i = (long long)part * 256 + threadIdx.x; i < head * vpr; i += parts * 256ll)
      *reinterpret_cast<uint4*>(buf + i / vpr * ld + i % vpr * 8) = make_uint4(0u, 0u, 0u, 0u);
  }
  for (long long i = (long long)part * 256 + threadIdx.x; i < (hi - lo) * vpr; i += parts * 256ll)
    *reinterpret_cast<uint4*>(buf + (lo + i / vpr) * ld + i % vpr * 8) = make_uint4(0u, 0u, 0u, 0u);
}

// dst[r, c] (bf16, pitch ld) = src[r, c] (fp32, dense rows of 8 vpr)
template <typename I>
__global__ void __launch_bounds__(256)
cast_rows_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, I total, I vpr, long long ld) {
  b200::begin_kernel();
  for (I i = blockIdx.x * (I)256 + threadIdx.x; i < total; i += (I)gridDim.x * 256) {
    const float4 a = *reinterpret_cast<const float4*>(src + (long long)i * 8), b = *reinterpret_cast<const float4*>(src + (long long)i * 8 + 4);
    const I r = i / vpr;
    *reinterpret_cast<uint4*>(dst + (long long)r * ld + (long long)(i - r * vpr) * 8) =
        make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
  }
}

int gate_grid(int T, int rows_per_cta) {
  const int grid = (T + rows_per_cta - 1) / rows_per_cta;
  const int cap = b200::sm_count() * GATE_CTAS;
  return grid < cap ? (grid < 1 ? 1 : grid) : cap;
}
int gate_bwd_grid(int T, int D) { return gate_grid(T, D == 256 ? BwdShape<1>::TEAMS : D == 512 ? BwdShape<2>::TEAMS : BwdShape<3>::TEAMS); }

bool gate_ok(int D, long long ld_u) { return D % 256 == 0 && D >= 256 && D <= 256 * GV && ld_u % 8 == 0; }

}  // namespace

// fp32 scratch elements b200_hstu_gate_cat_bwd needs for T rows of width D.
B200_API long long b200_hstu_gate_cat_scratch_elems(int T, int D) { return (long long)gate_bwd_grid(T, D) * 2 * D; }

// cat[T, 3D] = dropout([silu(u_raw) | attn | silu(u_raw) * LayerNorm(attn)], p);  mean / rstd [T] fp32 are kept for
// backward, which must be given the same p and seed.
B200_API int b200_hstu_gate_cat_fwd(const void* u_raw, long long ld_u, const void* attn, const void* w, const void* b,
                                    void* cat, float* mean, float* rstd, int T, int D, float eps, float p,
                                    unsigned long long seed, void* stream) {
  if (!(p >= 0.f && p < 1.f)) return b200::fail(902, "hstu_gate_cat_fwd: dropout rate %f outside [0, 1)", (double)p);
  if (!gate_ok(D, ld_u)) return b200::fail(900, "hstu_gate_cat_fwd: D=%d must be 256, 512 or 768 and the pitch %lld a multiple of 8", D, ld_u);
  if (T <= 0) return 0;
  const unsigned thr = (unsigned)lrintf(p * 65536.f);
  const float pe = (float)thr / 65536.f;   // the rate the 16-bit comparison realises
  auto U = (const __nv_bfloat16*)u_raw; auto A = (const __nv_bfloat16*)attn; auto W = (const __nv_bfloat16*)w;
  auto B = (const __nv_bfloat16*)b; auto C = (__nv_bfloat16*)cat;
  const int grid = gate_grid(T, 8);
  cudaStream_t st = (cudaStream_t)stream;
  if (D == 256) b200::launch(gate_cat_fwd_kernel<1>, grid, 256, 0, st, U, ld_u, A, W, B, C, mean, rstd, T, eps, pe, thr, seed);
  else if (D == 512) b200::launch(gate_cat_fwd_kernel<2>, grid, 256, 0, st, U, ld_u, A, W, B, C, mean, rstd, T, eps, pe, thr, seed);
  else b200::launch(gate_cat_fwd_kernel<3>, grid, 256, 0, st, U, ld_u, A, W, B, C, mean, rstd, T, eps, pe, thr, seed);
  b200::count_launch();
  return b200::check_launch("hstu_gate_cat_fwd");
}

// du_raw (row pitch ld_du) and dattn [T, D] from dcat [T, 3D]; dw / db fp32 [D] written, or added to when
// accumulate != 0.  scratch: b200_hstu_gate_cat_scratch_elems(T, D) floats.
B200_API int b200_hstu_gate_cat_bwd(const void* dcat, const void* u_raw, long long ld_u, const void* attn, const void* w,
                                    const void* b, const float* mean, const float* rstd, void* du_raw, long long ld_du,
                                    void* dattn, float* dw, float* db, float* scratch, int T, int D, int accumulate,
                                    float p, unsigned long long seed, void* stream) {
  if (!(p >= 0.f && p < 1.f)) return b200::fail(902, "hstu_gate_cat_bwd: dropout rate %f outside [0, 1)", (double)p);
  if (!gate_ok(D, ld_u) || ld_du % 8 != 0)
    return b200::fail(901, "hstu_gate_cat_bwd: D=%d must be 256, 512 or 768 and the pitches %lld / %lld multiples of 8", D, ld_u, ld_du);
  if (T <= 0) return 0;
  const int grid = gate_bwd_grid(T, D);
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned thr = (unsigned)lrintf(p * 65536.f);
  const float pe = (float)thr / 65536.f;
  auto DC = (const __nv_bfloat16*)dcat; auto U = (const __nv_bfloat16*)u_raw; auto A = (const __nv_bfloat16*)attn;
  auto W = (const __nv_bfloat16*)w; auto B = (const __nv_bfloat16*)b; auto DU = (__nv_bfloat16*)du_raw; auto DA = (__nv_bfloat16*)dattn;
  if (D == 256) b200::launch(gate_cat_bwd_kernel<1>, grid, BwdShape<1>::THREADS, 0, st, DC, U, ld_u, A, W, B, mean, rstd, DU, ld_du, DA, scratch, T, pe, thr, seed);
  else if (D == 512) b200::launch(gate_cat_bwd_kernel<2>, grid, BwdShape<2>::THREADS, 0, st, DC, U, ld_u, A, W, B, mean, rstd, DU, ld_du, DA, scratch, T, pe, thr, seed);
  else b200::launch(gate_cat_bwd_kernel<3>, grid, BwdShape<3>::THREADS, 0, st, DC, U, ld_u, A, W, B, mean, rstd, DU, ld_du, DA, scratch, T, pe, thr, seed);
  b200::count_launch();
  if (int r = b200::check_launch("hstu_gate_cat_bwd")) return r;
  b200::launch(gate_cat_reduce_kernel, 2 * D / 32, 256, 0, st, scratch, grid, D, dw, db, accumulate);
  b200::count_launch();
  return b200::check_launch("hstu_gate_cat_reduce");
}

// Zeroes the rows of buf [L, width] bf16 (pitch ld elements) that belong to no sequence of `offsets` [B + 1], and the rows of a
// sequence from `cover` on.
B200_API int b200_hstu_zero_uncovered(void* buf, const int* offsets, int B, long long L, long long ld, int width, long long cover,
                                      void* stream) {
  if (width % 8 != 0 || ld % 8 != 0 || ((uintptr_t)buf & 15) != 0)
    return b200::fail(903, "hstu_zero_uncovered: width %d and pitch %lld must be multiples of 8, the base 16-byte aligned", width, ld);
  if (L <= 0 || B < 0) return 0;          // (B < 0 is for the attention's launcher to refuse)
  b200::launch(zero_uncovered_rows_kernel, B + 16, 256, 0, (cudaStream_t)stream, (__nv_bfloat16*)buf, offsets, B, L, ld, width / 8, cover);
  b200::count_launch();
  return b200::check_launch("hstu_zero_uncovered");
}

// dst [rows, width] bf16 (pitch ld elements) = src [rows, width] fp32, dense.
B200_API int b200_cast_rows(const float* src, void* dst, long long rows, int width, long long ld, void* stream) {
  if (width % 8 != 0 || ld % 8 != 0 || (((uintptr_t)src | (uintptr_t)dst) & 15) != 0)
    return b200::fail(904, "cast_rows: width %d and pitch %lld must be multiples of 8, pointers 16-byte aligned", width, ld);
  const long long work = rows * (width / 8);
  if (work <= 0) return 0;
  const long long cap = (long long)b200::sm_count() * 16, want = (work + 255) / 256;
  const int grid = (int)(want < cap ? want : cap);
  if (work < (1ll << 31)) b200::launch(cast_rows_kernel<uint32_t>, grid, 256, 0, (cudaStream_t)stream, src, (__nv_bfloat16*)dst, (uint32_t)work, (uint32_t)(width / 8), ld);
  else b200::launch(cast_rows_kernel<long long>, grid, 256, 0, (cudaStream_t)stream, src, (__nv_bfloat16*)dst, work, width / 8, ld);
  b200::count_launch();
  return b200::check_launch("cast_rows");
}
