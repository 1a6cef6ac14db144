// RMSNorm / LayerNorm forward and backward over rows of a [T, D] bf16 matrix (fp32 math).
//
// A row stays in registers between its load and its store, so the activation is read once and
// written once.  Backward produces dx in one pass and the weight / bias gradients as per-CTA fp32
// partial rows in scratch memory (summed in registers over the CTA's rows), which a second
// fixed-order kernel sums: no atomics, so runs are bit-reproducible.
//
// All of it is bound by HBM as long as enough bytes are in flight, so the split follows the width:
//   D <= 1024   a team of 8, 16 or 32 lanes owns a row (one to four 16-byte vectors per lane), the row
//               reductions are shuffles inside the team and a warp keeps several rows in flight.  Rows of
//               a head dim (128) are the case this is for: one 256-thread CTA per such row left 240
//               threads idle and paid two barriers per 256 bytes.
//   D  > 1024   the CTA owns ROWS rows at a time: their loads are in flight together and ONE pair of
//               barriers reduces all of them (a barrier pair per row made the kernel latency-bound).
//   1024 < D <= 4096, a multiple of 256: forward and the activation's backward, a warp owns a row, for the order of its sums
//               (reasons at norm_fwd_warp_kernel).
// Backward without the activation, D > 256: the next rows' loads are in flight in a ring in shared memory (norm_bwd_ring_kernel).
// Measured (bf16 in and out, L2 flushed, launch included), one warp or CTA per row -> this split:
//   98304 x 128   forward 276 -> 16 us   backward 722 -> 30 us
//   92160 x 512   LayerNorm 116 -> 46 us;   8192 x 2880  52 -> 31 us;   4096 x 8192  50 -> 38 us
// Four rows of a 512-thread CTA instead of two of a 256-thread one lost 5 to 15 % at widths 2880 and 4096; above
// 4096 the backward takes 512 threads (with 256 its accumulators leave one CTA of 8 warps per SM: 97 us).
//
// Covers the reference's norm family: generative_recommenders/ops/triton/triton_layer_norm.py
// (_weighted_layer_norm_fwd / _bwd_dx / _layer_norm_bwd_dwdb, RMSNorm fwd/bwd, SwishLayerNorm)
// and the Primus-Turbo RMSNorm selected by small_llm_pretraining/primus/conf/
// llama3.1_8B-pretrain-fp4.yaml:122-123.
#include "common.cuh"
#include "runtime.h"

namespace {

constexpr int NT = 256;          // threads per CTA (512 for rows wider than 4096)
constexpr int MAX_D = 8192;

B200_DEVICE void unpack8(const uint4& u, float (&f)[8]) {
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
B200_DEVICE uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}
B200_DEVICE uint4 ld16(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
B200_DEVICE void st16(__nv_bfloat16* p, const uint4& u) { *reinterpret_cast<uint4*>(p) = u; }

// Sums of NV values over the threads that own a row.  G <= 32: the G lanes of a team (xor shuffles stay inside
// it); G == 0: the whole CTA, all NV values with one pair of barriers.  `red` holds NV x 16 floats.
template <int G, int NV>
B200_DEVICE void team_sum(float (&v)[NV], float* red) {
#pragma unroll
  for (int i = 0; i < NV; ++i) {
#pragma unroll
    for (int o = (G == 0 ? 16 : G / 2); o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  }
  if (G == 0) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncthreads();   // the previous use of `red` has been read
    if (l == 0)
#pragma unroll
      for (int i = 0; i < NV; ++i) red[i * 16 + w] = v[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float r = 0.f;
      for (int k = 0; k < nw; ++k) r += red[i * 16 + k];
      v[i] = r;
    }
  }
}

// Which rows and columns a thread works on.  A team (G lanes, or the CTA) takes ROWS rows per step.
template <int G, int ROWS>
struct Split {
  int t, stride, first, step;   // index inside the team, team size, first row, rows per grid step
  B200_DEVICE Split() {
    if (G == 0) {
      t = threadIdx.x; stride = blockDim.x;
      first = blockIdx.x * ROWS; step = gridDim.x * ROWS;
    } else {
      constexpr int TEAMS = NT / (G == 0 ? 1 : G);
      t = threadIdx.x % (G == 0 ? 1 : G); stride = G;
      first = (blockIdx.x * TEAMS + threadIdx.x / (G == 0 ? 1 : G)) * ROWS;
      step = gridDim.x * TEAMS * ROWS;
    }
  }
};

// MODE: 0 = RMSNorm, 1 = LayerNorm.  act: 0 = none, 1 = swish (y = x * sigmoid(norm(x))).
// Optional residual input: h = x + res is normalised and also written to h_out.
// Every lane of a warp runs the same number of steps (the shuffles name all 32): rows past T are predicated.
template <int MODE, int G, int V, int ROWS, int MAXT = NT>
__global__ void __launch_bounds__(MAXT)
norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
                __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ h_out, float* __restrict__ mean_out,
                float* __restrict__ rstd_out, int T, int D, float eps, int act) {
  b200::begin_kernel();
  __shared__ float red[ROWS * 16];
  const Split<G, ROWS> sp;
  const int nvec = D / 8;
  const float inv_d = 1.f / D;
  const int warp_first = (G == 0) ? sp.first : __shfl_sync(0xffffffffu, sp.first, 0);
  for (int off = 0; warp_first + off < T; off += sp.step) {
    const int row0 = sp.first + off;
    uint4 xv[ROWS][V];
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int vi = sp.t + i * sp.stride;
        xv[r][i] = (row0 + r < T && vi < nvec) ? ld16(x + (long long)(row0 + r) * D + vi * 8) : make_uint4(0, 0, 0, 0);
      }
    if (res != nullptr) {
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int i = 0; i < V; ++i) {
          const int vi = sp.t + i * sp.stride;
          if (row0 + r < T && vi < nvec) {
            const long long at = (long long)(row0 + r) * D + vi * 8;
            float a[8], c[8];
            unpack8(xv[r][i], a);
            unpack8(ld16(res + at), c);
#pragma unroll
            for (int j = 0; j < 8; ++j) a[j] += c[j];
            xv[r][i] = pack8(a);   // the normalised value matches the stored (rounded) sum
            if (h_out != nullptr) st16(h_out + at, xv[r][i]);
          }
        }
    }
    float sum[ROWS], mean[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        float a[8];
        unpack8(xv[r][i], a);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += (MODE == 1) ? a[j] : a[j] * a[j];
      }
      sum[r] = s;
      mean[r] = 0.f;
    }
    team_sum<G, ROWS>(sum, red);
    if (MODE == 1) {
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        mean[r] = sum[r] * inv_d;
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < V; ++i) {
          if (sp.t + i * sp.stride < nvec) {
            float a[8];
            unpack8(xv[r][i], a);
#pragma unroll
            for (int j = 0; j < 8; ++j) { const float d = a[j] - mean[r]; s += d * d; }
          }
        }
        sum[r] = s;
      }
      team_sum<G, ROWS>(sum, red);
    }
    float rstd[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      rstd[r] = rsqrtf(sum[r] * inv_d + eps);
      if (sp.t == 0 && row0 + r < T) {
        if (rstd_out != nullptr) rstd_out[row0 + r] = rstd[r];
        if (MODE == 1 && mean_out != nullptr) mean_out[row0 + r] = mean[r];
      }
    }
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int vi = sp.t + i * sp.stride;
      if (vi < nvec) {
        float w8[8], b8[8];
        if (w != nullptr) unpack8(ld16(w + vi * 8), w8);
        if (b != nullptr) unpack8(ld16(b + vi * 8), b8);
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
          if (row0 + r < T) {
            float a[8], o[8];
            unpack8(xv[r][i], a);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float n = (a[j] - mean[r]) * rstd[r];
              if (w != nullptr) n *= w8[j];
              if (b != nullptr) n += b8[j];
              o[j] = act ? a[j] * (1.f / (1.f + __expf(-n))) : n;
            }
            st16(y + (long long)(row0 + r) * D + vi * 8, pack8(o));
          }
      }
    }
  }
}

// Forward of widths that are whole vectors of a warp up to 4096: a warp per row, up to 16 vectors per lane, summed lane
// by lane in column order.  The CTA-per-row split is up to 20 % faster at 4096 (27 -> 22 us for 4011 rows) and no less exact.  It is not
// taken here yet: it adds the squares in another order, one bf16 bit in 90000 flips, and block-scaled linears behind it turn that
// into 3 % of the attention gradients over three quantisers, at the same error against 64 bits.  (The backward has taken the ring's
// order, which does the same to a step's gradients, for 73 -> 52 us at 8192 x 4096.)
constexpr int WMAXV = 16;
template <int MODE>
__global__ void __launch_bounds__(256)
norm_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                     const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
                     __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ h_out, float* __restrict__ mean_out,
                     float* __restrict__ rstd_out, int T, int D, float eps, int act) {
  b200::begin_kernel();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nv = D >> 8;  // vectors per lane
  for (int row = blockIdx.x * 8 + warp; row < T; row += gridDim.x * 8) {
    const long long base = (long long)row * D;
    uint4 xv[WMAXV];
#pragma unroll
    for (int i = 0; i < WMAXV; ++i)
      if (i < nv) xv[i] = *reinterpret_cast<const uint4*>(x + base + (lane + 32 * i) * 8);
    if (res != nullptr) {
#pragma unroll
      for (int i = 0; i < WMAXV; ++i)
        if (i < nv) {
          float a[8], r[8];
          unpack8(xv[i], a);
          unpack8(ld16(res + base + (lane + 32 * i) * 8), r);
#pragma unroll
          for (int j = 0; j < 8; ++j) a[j] += r[j];
          xv[i] = make_uint4(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]), pack_bf16x2(a[4], a[5]), pack_bf16x2(a[6], a[7]));
          if (h_out != nullptr) *reinterpret_cast<uint4*>(h_out + base + (lane + 32 * i) * 8) = xv[i];
        }
    }
    float s = 0.f, ss = 0.f;
#pragma unroll
    for (int i = 0; i < WMAXV; ++i)
      if (i < nv) {
        float a[8];
        unpack8(xv[i], a);
#pragma unroll
        for (int j = 0; j < 8; ++j) { s += a[j]; ss += a[j] * a[j]; }
      }
    float mean = 0.f, rstd;
    if (MODE == 1) {
      mean = warp_sum(s) / D;
      float var = 0.f;
#pragma unroll
      for (int i = 0; i < WMAXV; ++i)
        if (i < nv) {
          float a[8];
          unpack8(xv[i], a);
#pragma unroll
          for (int j = 0; j < 8; ++j) { const float d = a[j] - mean; var += d * d; }
        }
      rstd = rsqrtf(warp_sum(var) / D + eps);
    } else {
      rstd = rsqrtf(warp_sum(ss) / D + eps);
    }
    if (lane == 0) {
      if (rstd_out) rstd_out[row] = rstd;
      if (MODE == 1 && mean_out) mean_out[row] = mean;
    }
#pragma unroll
    for (int i = 0; i < WMAXV; ++i)
      if (i < nv) {
        const int c = (lane + 32 * i) * 8;
        float a[8], w8[8], b8[8], o[8];
        unpack8(xv[i], a);
        if (w != nullptr) unpack8(ld16(w + c), w8);
        if (b != nullptr) unpack8(ld16(b + c), b8);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float n = (a[j] - mean) * rstd;
          if (w != nullptr) n *= w8[j];
          if (b != nullptr) n += b8[j];
          o[j] = act ? a[j] * (1.f / (1.f + __expf(-n))) : n;
        }
        st16(y + base + c, pack8(o));
      }
  }
}

// dx for every row, plus per-CTA partial sums of dw (and db) in `partial` laid out [gridDim.x][2][D].
template <int MODE, int ACT, int G, int V, int ROWS, int MAXT = NT>
__global__ void __launch_bounds__(MAXT)
norm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
                const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                float* __restrict__ partial, int T, int D) {
  b200::begin_kernel();
  constexpr int NACC = (MODE == 1 || ACT) ? 2 : 1;
  constexpr int NS = (MODE == 1) ? 2 * ROWS : ROWS;
  constexpr int TEAMS = (G == 0) ? 1 : NT / (G == 0 ? 1 : G);
  __shared__ float red[G == 0 ? NS * 16 : 1];
  extern __shared__ float acc_sm[];     // G > 0: [TEAMS][D], used for dw and then for db
  const Split<G, ROWS> sp;
  const int nvec = D / 8;
  const float inv_d = 1.f / D;
  float dw_acc[V][8], db_acc[NACC == 2 ? V : 1][8];
#pragma unroll
  for (int i = 0; i < V; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) { dw_acc[i][j] = 0.f; if (NACC == 2) db_acc[NACC == 2 ? i : 0][j] = 0.f; }

  const int warp_first = (G == 0) ? sp.first : __shfl_sync(0xffffffffu, sp.first, 0);
  for (int off = 0; warp_first + off < T; off += sp.step) {
    const int row0 = sp.first + off;
    uint4 xv[ROWS][V], gv[ROWS][V];
    float rstd[ROWS], mean[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const bool live = row0 + r < T;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int vi = sp.t + i * sp.stride;
        const long long at = (long long)(row0 + r) * D + vi * 8;
        xv[r][i] = gv[r][i] = make_uint4(0, 0, 0, 0);
        if (live && vi < nvec) { xv[r][i] = ld16(x + at); gv[r][i] = ld16(dy + at); }
      }
      rstd[r] = live ? rstd_in[row0 + r] : 0.f;
      mean[r] = (MODE == 1 && live) ? mean_in[row0 + r] : 0.f;
    }
    float s[NS];
#pragma unroll
    for (int r = 0; r < NS; ++r) s[r] = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int vi = sp.t + i * sp.stride;
      if (vi < nvec) {
        float w8[8], b8[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) { w8[j] = 1.f; b8[j] = 0.f; }
        if (w != nullptr) unpack8(ld16(w + vi * 8), w8);
        if (ACT && b != nullptr) unpack8(ld16(b + vi * 8), b8);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          float x8[8], d8[8];
          unpack8(xv[r][i], x8);
          unpack8(gv[r][i], d8);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float xn = (x8[j] - mean[r]) * rstd[r];
            float dn = d8[j];   // gradient w.r.t. the affine output n = xn * w + b
            if (ACT) {
              // y = x * sigmoid(n): through n the gradient is dy * x * s * (1 - s); the direct path
              // dy * s is added to dx after the row reductions
              const float sg = 1.f / (1.f + __expf(-(xn * w8[j] + b8[j])));
              dn = d8[j] * x8[j] * sg * (1.f - sg);
            }
            dw_acc[i][j] += dn * xn;
            if (NACC == 2) db_acc[NACC == 2 ? i : 0][j] += dn;
            const float g = dn * w8[j];
            s[r] += g * xn;
            if (MODE == 1) s[ROWS * (MODE == 1) + r] += g;
          }
        }
      }
    }
    team_sum<G, NS>(s, red);
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int vi = sp.t + i * sp.stride;
      if (vi < nvec) {
        float w8[8], b8[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) { w8[j] = 1.f; b8[j] = 0.f; }
        if (w != nullptr) unpack8(ld16(w + vi * 8), w8);
        if (ACT && b != nullptr) unpack8(ld16(b + vi * 8), b8);
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
          if (row0 + r < T) {
            const long long at = (long long)(row0 + r) * D + vi * 8;
            const float s1 = s[r] * inv_d, s2 = (MODE == 1) ? s[ROWS * (MODE == 1) + r] * inv_d : 0.f;
            float x8[8], d8[8], o[8];
            unpack8(xv[r][i], x8);
            unpack8(gv[r][i], d8);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float xn = (x8[j] - mean[r]) * rstd[r];
              float dn = d8[j], direct = 0.f;
              if (ACT) {
                const float sg = 1.f / (1.f + __expf(-(xn * w8[j] + b8[j])));
                dn = d8[j] * x8[j] * sg * (1.f - sg);
                direct = d8[j] * sg;
              }
              o[j] = rstd[r] * (dn * w8[j] - xn * s1 - s2) + direct;
            }
            if (dres != nullptr) {
              float r8[8];
              unpack8(ld16(dres + at), r8);
#pragma unroll
              for (int j = 0; j < 8; ++j) o[j] += r8[j];
            }
            st16(dx + at, pack8(o));
          }
      }
    }
  }
  if (partial == nullptr) return;
  float* pw = partial + (long long)blockIdx.x * 2 * D;
  if (G == 0) {
    // a thread owns its columns for every row of the CTA
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int vi = sp.t + i * sp.stride;
      if (vi < nvec) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          pw[vi * 8 + j] = dw_acc[i][j];
          pw[D + vi * 8 + j] = NACC == 2 ? db_acc[NACC == 2 ? i : 0][j] : 0.f;
        }
      }
    }
    return;
  }
  const int team = threadIdx.x / (G == 0 ? 1 : G);
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    if (which < NACC) {
      __syncthreads();
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int vi = sp.t + i * sp.stride;
        if (vi < nvec)
#pragma unroll
          for (int j = 0; j < 8; ++j)
            acc_sm[team * D + vi * 8 + j] = which == 0 ? dw_acc[i][j] : db_acc[NACC == 2 ? i : 0][j];
      }
      __syncthreads();
    }
    for (int c = threadIdx.x; c < D; c += NT) {
      float t = 0.f;
      if (which < NACC)
        for (int k = 0; k < TEAMS; ++k) t += acc_sm[k * D + c];
      pw[which * D + c] = t;
    }
  }
}

// Backward of the same widths with the activation: a warp per row, summed lane by lane in column order as in the forward, so that the
// activation is recomputed over the same split.  dw / db accumulated per warp in shared memory (fixed lane -> column mapping, no
// atomics), summed over the CTA's warps in order and written as one partial row per CTA.
template <int MODE>
__global__ void __launch_bounds__(256)
norm_bwd_warp_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                     const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
                     const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                     const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                     float* __restrict__ partial, int T, int D, int nwarps) {
  b200::begin_kernel();
  extern __shared__ float acc[];  // [nwarps][dw | db][D]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nv = D >> 8;
  float* my_w = acc + (long long)warp * 2 * D;
  float* my_b = my_w + D;
  if (warp < nwarps)
    for (int i = lane; i < 2 * D; i += 32) my_w[i] = 0.f;
  __syncwarp();
  if (warp < nwarps) {
    for (int row = blockIdx.x * nwarps + warp; row < T; row += gridDim.x * nwarps) {
      const long long base = (long long)row * D;
      const float rstd = rstd_in[row];
      const float mean = (MODE == 1) ? mean_in[row] : 0.f;
      uint4 xv[WMAXV], gv[WMAXV];
#pragma unroll
      for (int i = 0; i < WMAXV; ++i)
        if (i < nv) {
          xv[i] = *reinterpret_cast<const uint4*>(x + base + (lane + 32 * i) * 8);
          gv[i] = *reinterpret_cast<const uint4*>(dy + base + (lane + 32 * i) * 8);
        }
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int i = 0; i < WMAXV; ++i)
        if (i < nv) {
          const int c = (lane + 32 * i) * 8;
          float x8[8], d8[8], w8[8], b8[8];
          unpack8(xv[i], x8);
          unpack8(gv[i], d8);
#pragma unroll
          for (int j = 0; j < 8; ++j) { w8[j] = 1.f; b8[j] = 0.f; }
          if (w != nullptr) unpack8(ld16(w + c), w8);
          if (b != nullptr) unpack8(ld16(b + c), b8);
          float4 a0 = *reinterpret_cast<float4*>(my_w + c), a1 = *reinterpret_cast<float4*>(my_w + c + 4);
          float aw[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
          float4 b0 = *reinterpret_cast<float4*>(my_b + c), b1 = *reinterpret_cast<float4*>(my_b + c + 4);
          float ab[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float xn = (x8[j] - mean) * rstd;
            const float n = xn * w8[j] + b8[j];
            const float sg = 1.f / (1.f + __expf(-n));
            const float dn = d8[j] * x8[j] * sg * (1.f - sg);
            aw[j] += dn * xn;
            ab[j] += dn;
            const float gj = dn * w8[j];
            s1 += gj * xn;
            s2 += gj;
          }
          *reinterpret_cast<float4*>(my_w + c) = make_float4(aw[0], aw[1], aw[2], aw[3]);
          *reinterpret_cast<float4*>(my_w + c + 4) = make_float4(aw[4], aw[5], aw[6], aw[7]);
          *reinterpret_cast<float4*>(my_b + c) = make_float4(ab[0], ab[1], ab[2], ab[3]);
          *reinterpret_cast<float4*>(my_b + c + 4) = make_float4(ab[4], ab[5], ab[6], ab[7]);
        }
      s1 = warp_sum(s1) / D;
      s2 = (MODE == 1) ? warp_sum(s2) / D : 0.f;
#pragma unroll
      for (int i = 0; i < WMAXV; ++i)
        if (i < nv) {
          const int c = (lane + 32 * i) * 8;
          float x8[8], d8[8], w8[8], b8[8], o[8];
          unpack8(xv[i], x8);
          unpack8(gv[i], d8);
#pragma unroll
          for (int j = 0; j < 8; ++j) { w8[j] = 1.f; b8[j] = 0.f; }
          if (w != nullptr) unpack8(ld16(w + c), w8);
          if (b != nullptr) unpack8(ld16(b + c), b8);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float xn = (x8[j] - mean) * rstd;
            const float n = xn * w8[j] + b8[j];
            const float sg = 1.f / (1.f + __expf(-n));
            const float dn = d8[j] * x8[j] * sg * (1.f - sg);
            o[j] = rstd * (dn * w8[j] - xn * s1 - s2) + d8[j] * sg;
          }
          if (dres != nullptr) {
            float r8[8];
            unpack8(ld16(dres + base + c), r8);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] += r8[j];
          }
          st16(dx + base + c, pack8(o));
        }
    }
  }
  __syncthreads();
  if (partial != nullptr) {
    float* pw = partial + (long long)blockIdx.x * 2 * D;
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
      float sw = 0.f, sb = 0.f;
      for (int k = 0; k < nwarps; ++k) {
        sw += acc[(long long)k * 2 * D + c];
        sb += acc[(long long)k * 2 * D + D + c];
      }
      pw[c] = sw;
      pw[D + c] = sb;
    }
  }
}

// Backward without the activation for rows of more than 256 columns: x and dy (and dres) are read and dx
// written once.  A team (G = 32: a warp, G = 0: the CTA) owns whole rows, a thread the same V vectors of columns in all of them, so the
// column sums stay in its registers.  Every thread copies its own vectors of the next S - 1 row groups into its own slots of a
// ring in shared memory (cp.async: no registers held, no barrier).  With loads of a row that started when the row before was done,
// column sums included: 8192 x 2880 64 us, now 46, 8192 x 4096 73 and 52, 4096 x 8192 85 and 64; with a residual's
// gradient 89 and 50, 114 and 58, 109 and 75; LayerNorm of 46000 x 512 46 and 46, with a residual 67 and 52.
// Bound by instructions before memory: alone it takes 34 us for 8192 x 2880 (4.1 TB/s, 0.63 of the measured copy rate) and 42 for
// 8192 x 4096 (4.8 TB/s), with 68 and 73 % of the issue slots taken by the 23 and 29 warps that 64 registers a thread leave on an SM;
// the rest waits for barriers and shared memory.  The sum over the CTAs' partial rows and the launches are the other 10 us.
template <int MODE, int G, int V, int R, int S, int MAXT>
__global__ void __launch_bounds__(MAXT, MODE == 1 && V * MAXT > 512 ? 1 : 2)
norm_bwd_ring_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                     const float* __restrict__ mean_in, const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ dres,
                     __nv_bfloat16* __restrict__ dx, float* __restrict__ partial, int T, int D) {
  b200::begin_kernel();
  constexpr int NACC = MODE == 1 ? 2 : 1, NS = R * NACC;
  extern __shared__ uint4 ring[];                    // [S][R][x | dy | dres][V][threads]
  __shared__ float red[2][NS][16];
  const int nt = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int nvec = D / 8, nin = dres != nullptr ? 3 : 2;
  const float inv_d = 1.f / D;
  const int team = G == 32 ? blockIdx.x * nw + warp : blockIdx.x, teams = G == 32 ? gridDim.x * nw : gridDim.x;
  const int first = G == 32 ? lane : tid, stride = G == 32 ? 32 : nt;
  const int groups = (T + R - 1) / R;
  auto slot = [&](int s, int r, int in, int i) { return ring + (((s * R + r) * nin + in) * V + i) * nt + tid; };
  auto copy = [&](uint4* to, const __nv_bfloat16* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(to)), "l"(from) : "memory");
  };
  auto issue = [&](int g, int s) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int row = g * R + r, vi = first + i * stride;
        if (g < groups && row < T && vi < nvec) {
          const long long at = (long long)row * D + vi * 8;
          copy(slot(s, r, 0, i), x + at);
          copy(slot(s, r, 1, i), dy + at);
          if (nin == 3) copy(slot(s, r, 2, i), dres + at);
        }
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto stats = [&](int g, float (&rs)[R], float (&mu)[R]) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = g * R + r;
      rs[r] = g < groups && row < T ? rstd_in[row] : 0.f;
      mu[r] = MODE == 1 && g < groups && row < T ? mean_in[row] : 0.f;
    }
  };
  uint4 wv[V];
  float dw_acc[V][8], db_acc[MODE == 1 ? V : 1][8];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int vi = first + i * stride;
    wv[i] = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);      // 1.0
    if (w != nullptr && vi < nvec) wv[i] = ld16(w + vi * 8);
#pragma unroll
    for (int j = 0; j < 8; ++j) { dw_acc[i][j] = 0.f; if (MODE == 1) db_acc[MODE == 1 ? i : 0][j] = 0.f; }
  }
  float rs_next[R], mu_next[R];
  stats(team, rs_next, mu_next);
#pragma unroll
  for (int k = 0; k < S - 1; ++k) issue(team + k * teams < groups ? team + k * teams : groups, k);
  int cur = 0, buf = 0;
  for (int g = team; g < groups; g += teams) {
    // the slot that this thread read in the iteration before
    const long long ahead = (long long)g + (long long)(S - 1) * teams;
    issue(ahead < groups ? (int)ahead : groups, cur == 0 ? S - 1 : cur - 1);
    float rstd[R], mean[R], s[NS];
#pragma unroll
    for (int r = 0; r < R; ++r) { rstd[r] = rs_next[r]; mean[r] = mu_next[r]; }
    stats(groups - g > teams ? g + teams : groups, rs_next, mu_next);
#pragma unroll
    for (int r = 0; r < NS; ++r) s[r] = 0.f;
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 1) : "memory");
    uint4 xv[R][V], gv[R][V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const bool in = first + i * stride < nvec;
      float w8[8];
      unpack8(wv[i], w8);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        xv[r][i] = gv[r][i] = make_uint4(0, 0, 0, 0);
        if (in && g * R + r < T) { xv[r][i] = *slot(cur, r, 0, i); gv[r][i] = *slot(cur, r, 1, i); }
        float x8[8], d8[8];
        unpack8(xv[r][i], x8);
        unpack8(gv[r][i], d8);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xn = (x8[j] - mean[r]) * rstd[r];
          dw_acc[i][j] += d8[j] * xn;
          if (MODE == 1) db_acc[MODE == 1 ? i : 0][j] += d8[j];
          const float gj = d8[j] * w8[j];
          s[r] += gj * xn;
          if (MODE == 1) s[R * (MODE == 1) + r] += gj;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < NS; ++k) s[k] = warp_sum(s[k]);
    if (G == 0) {
      if (lane == 0)
#pragma unroll
        for (int k = 0; k < NS; ++k) red[buf][k][warp] = s[k];
      __syncthreads();                               // the other buffer is free again when this is passed
#pragma unroll
      for (int k = 0; k < NS; ++k) s[k] = warp_sum(lane < nw ? red[buf][k][lane] : 0.f);
      buf ^= 1;
    }
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int vi = first + i * stride;
      float w8[8];
      unpack8(wv[i], w8);
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (vi < nvec && g * R + r < T) {
          const float s1 = s[r] * inv_d, s2 = MODE == 1 ? s[R * (MODE == 1) + r] * inv_d : 0.f;
          float x8[8], d8[8], o[8];
          unpack8(xv[r][i], x8);
          unpack8(gv[r][i], d8);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = rstd[r] * (d8[j] * w8[j] - (x8[j] - mean[r]) * rstd[r] * s1 - s2);
          if (nin == 3) {
            float r8[8];
            unpack8(*slot(cur, r, 2, i), r8);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] += r8[j];
          }
          st16(dx + (long long)(g * R + r) * D + vi * 8, pack8(o));
        }
    }
    cur = cur + 1 == S ? 0 : cur + 1;
  }
  if (partial == nullptr) return;
  float* pw = partial + (long long)blockIdx.x * 2 * D;
  if (G == 0) {
    // a thread owns its columns for every row of the CTA
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int vi = first + i * stride;
      if (vi < nvec) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float4* o = reinterpret_cast<float4*>(pw + h * D + vi * 8);
          float v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = h == 0 ? dw_acc[i][j] : (MODE == 1 ? db_acc[MODE == 1 ? i : 0][j] : 0.f);
          o[0] = make_float4(v[0], v[1], v[2], v[3]);
          o[1] = make_float4(v[4], v[5], v[6], v[7]);
        }
      }
    }
    return;
  }
  // the warps' sums, in their order, through the ring (its copies are all done)
  asm volatile("cp.async.wait_all;" ::: "memory");
  float* acc = reinterpret_cast<float*>(ring);       // [warps][D]
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (h < NACC) {
      __syncthreads();
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int vi = first + i * stride;
        if (vi < nvec)
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[warp * D + vi * 8 + j] = h == 0 ? dw_acc[i][j] : db_acc[MODE == 1 ? i : 0][j];
      }
      __syncthreads();
    }
    for (int c = tid; c < D; c += nt) {
      float t = 0.f;
      if (h < NACC)
        for (int k = 0; k < nw; ++k) t += acc[k * D + c];
      pw[h * D + c] = t;
    }
  }
}

// out[c] (+)= sum_p partial[p][which][c]: 32 columns per CTA, its 8 warps take every eighth partial row (their loads
// are independent: one thread per column walked all of them in series), summed in a fixed order.
__global__ void __launch_bounds__(256)
norm_bwd_reduce_kernel(const float* __restrict__ partial, int nparts, int D, float* __restrict__ dw,
                       float* __restrict__ db, int accumulate) {
  b200::begin_kernel();
  __shared__ float sm[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane, which = blockIdx.y;
  float* out = which == 0 ? dw : db;
  if (out == nullptr) return;
  float s = 0.f;
  if (c < D)
#pragma unroll 4
    for (int p = warp; p < nparts; p += 8) s += partial[((long long)p * 2 + which) * D + c];
  sm[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && c < D) {
#pragma unroll
    for (int k = 1; k < 8; ++k) s += sm[k][lane];
    out[c] = accumulate ? out[c] + s : s;
  }
}

struct FwdArgs {
  const __nv_bfloat16 *x, *res, *w, *b;
  __nv_bfloat16 *y, *h;
  float *mean, *rstd;
  int T, D, act;
  float eps;
  cudaStream_t st;
};
struct BwdArgs {
  const __nv_bfloat16 *dy, *x, *w, *b, *dres;
  const float *mean, *rstd;
  __nv_bfloat16* dx;
  float* partial;
  int T, D, grid;
  cudaStream_t st;
};

int block_threads(int D, int V) { return ((D / 8 + V - 1) / V + 31) / 32 * 32; }

template <int MODE, int G, int V, int ROWS, int MAXT = NT>
void run_fwd(const FwdArgs& a) {
  const int per_cta = (G == 0 ? 1 : NT / (G == 0 ? 1 : G)) * ROWS;
  const int need = (a.T + per_cta - 1) / per_cta, cap = b200::sm_count() * 8;
  b200::launch(norm_fwd_kernel<MODE, G, V, ROWS, MAXT>, need < cap ? need : cap, G == 0 ? block_threads(a.D, V) : NT, 0, a.st, 
      a.x, a.res, a.w, a.b, a.y, a.h, a.mean, a.rstd, a.T, a.D, a.eps, a.act);
}

template <int MODE>
void dispatch_fwd(const FwdArgs& a) {
  if (a.D <= 64) run_fwd<MODE, 8, 1, 4>(a);
  else if (a.D <= 128) run_fwd<MODE, 16, 1, 4>(a);
  else if (a.D <= 256) run_fwd<MODE, 32, 1, 4>(a);
  else if (a.D <= 512) run_fwd<MODE, 32, 2, 2>(a);
  else if (a.D <= 1024) run_fwd<MODE, 32, 4, 1>(a);
  else if (a.D % 256 == 0 && a.D <= 4096) {
    const int need = (a.T + 7) / 8, cap = b200::sm_count() * 8;
    b200::launch(norm_fwd_warp_kernel<MODE>, need < cap ? need : cap, 256, 0, a.st, a.x, a.res, a.w, a.b, a.y, a.h, a.mean, a.rstd, a.T,
                                                                         a.D, a.eps, a.act);
  }
  else if (a.D <= 4096) run_fwd<MODE, 0, 2, 2>(a);
  else run_fwd<MODE, 0, 4, 2>(a);
}

template <int MODE, int ACT, int G, int V, int ROWS, int MAXT = NT>
int run_bwd(const BwdArgs& a) {
  const int per_cta = (G == 0 ? 1 : NT / (G == 0 ? 1 : G)) * ROWS;
  const int need = (a.T + per_cta - 1) / per_cta;
  const int grid = need < a.grid ? need : a.grid;      // never more partial rows than the scratch holds
  const int smem = G == 0 ? 0 : NT / (G == 0 ? 1 : G) * a.D * 4;      // at most 32 KB
  b200::launch(norm_bwd_kernel<MODE, ACT, G, V, ROWS, MAXT>, grid, G == 0 ? block_threads(a.D, V) : NT, smem, a.st, 
      a.dy, a.x, a.w, a.b, a.mean, a.rstd, a.dres, a.dx, a.partial, a.T, a.D);
  return grid;
}

template <int MODE, int G, int V, int R, int S, int MAXT>
int launch_bwd_ring(const BwdArgs& a, int threads, int smem) {
  auto kern = norm_bwd_ring_kernel<MODE, G, V, R, S, MAXT>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return -b200::fail(302, "norm_bwd: cannot raise shared memory: %s", cudaGetErrorString(e));
    }
    configured[dev & 63] = true;
  }
  const int per_cta = (G == 32 ? threads / 32 : 1) * R, need = (a.T + per_cta - 1) / per_cta;
  const int grid = need < a.grid ? need : a.grid;      // never more partial rows than the scratch holds
  b200::launch(kern, grid, threads, smem, a.st, a.dy, a.x, a.w, a.mean, a.rstd, a.dres, a.dx, a.partial, a.T, a.D);
  return grid;
}

// As deep a ring as leaves room for two CTAs an SM: at most 4 stages and 104 KB (2 stages of 48 KB at 8192 columns and a residual).
template <int MODE, int G, int V, int R, int MAXT>
int run_bwd_ring(const BwdArgs& a) {
  const int threads = G == 32 ? MAXT : block_threads(a.D, V);
  const int stage = R * V * threads * 16 * (a.dres != nullptr ? 3 : 2);
  if (4 * stage <= 104 * 1024) return launch_bwd_ring<MODE, G, V, R, 4, MAXT>(a, threads, 4 * stage);
  if (3 * stage <= 104 * 1024) return launch_bwd_ring<MODE, G, V, R, 3, MAXT>(a, threads, 3 * stage);
  return launch_bwd_ring<MODE, G, V, R, 2, MAXT>(a, threads, 2 * stage);
}

template <int MODE>
int run_bwd_warp(const BwdArgs& a) {
  int nwarps = (200 * 1024) / (a.D * 4 * 2);
  if (nwarps > 8) nwarps = 8;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(norm_bwd_warp_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return -b200::fail(302, "norm_bwd: cannot raise shared memory: %s", cudaGetErrorString(e));
    }
    configured[dev & 63] = true;
  }
  const int grid = b200::sm_count() < a.grid ? b200::sm_count() : a.grid;
  b200::launch(norm_bwd_warp_kernel<MODE>, grid, 256, nwarps * 2 * a.D * 4, a.st, a.dy, a.x, a.w, a.b, a.mean, a.rstd, a.dres, a.dx,
               a.partial, a.T, a.D, nwarps);
  return grid;
}

template <int MODE, int ACT>
int dispatch_bwd(const BwdArgs& a) {
  if (a.D <= 64) return run_bwd<MODE, ACT, 8, 1, 4>(a);
  if (a.D <= 128) return run_bwd<MODE, ACT, 16, 1, 4>(a);
  if (a.D <= 256) return run_bwd<MODE, ACT, 32, 1, 4>(a);
  if constexpr (ACT == 0) {
    if (a.D <= 512) return run_bwd_ring<MODE, 32, 2, 2, 256>(a);
    if (a.D <= 1024) return run_bwd_ring<MODE, 32, 4, 1, 256>(a);
    if (a.D <= 4096) return run_bwd_ring<MODE, 0, 1, 2, 512>(a);
    return run_bwd_ring<MODE, 0, 2, 1, 512>(a);
  } else {
    if (a.D <= 512) return run_bwd<MODE, ACT, 32, 2, 2>(a);
    if (a.D <= 1024) return run_bwd<MODE, ACT, 32, 4, 1>(a);
    if (a.D % 256 == 0 && a.D <= 4096) return run_bwd_warp<MODE>(a);
    if (a.D <= 4096) return run_bwd<MODE, ACT, 0, 2, 2>(a);
    return run_bwd<MODE, ACT, 0, 2, 2, 512>(a);
  }
}

}  // namespace

// Number of fp32 elements of scratch needed by b200_norm_bwd for a [T, D] problem.
B200_API long long b200_norm_bwd_scratch_elems(int T, int D) {
  int grid = b200::sm_count() * 2;
  if (grid > T) grid = T;
  return (long long)grid * 2 * D;
}

// mode 0 RMSNorm / 1 LayerNorm.  res/h_out/b/mean/w may be null.  act=1: y = h * sigmoid(norm(h)).
B200_API int b200_norm_fwd(int mode, const void* x, const void* res, const void* w, const void* b, void* y,
                           void* h_out, float* mean, float* rstd, int T, int D, float eps, int act, void* stream) {
  if (D % 8 != 0 || D > MAX_D) return b200::fail(300, "norm_fwd: D=%d must be a multiple of 8 and <= %d", D, MAX_D);
  if (T <= 0) return 0;
  FwdArgs a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w, (const __nv_bfloat16*)b,
            (__nv_bfloat16*)y, (__nv_bfloat16*)h_out, mean, rstd, T, D, act, eps, (cudaStream_t)stream};
  if (mode == 0) dispatch_fwd<0>(a);
  else dispatch_fwd<1>(a);
  b200::count_launch();
  return b200::check_launch("norm_fwd");
}

// dx = d(norm)/dx (+ dres); dw/db fp32 [D] (written, or added to when accumulate != 0).
// `scratch` must hold b200_norm_bwd_scratch_elems(T, D) floats.
B200_API int b200_norm_bwd(int mode, const void* dy, const void* x, const void* w, const void* b, const float* mean,
                           const float* rstd, const void* dres, void* dx, float* dw, float* db, float* scratch,
                           int T, int D, int act, int accumulate, void* stream) {
  if (D % 8 != 0 || D > MAX_D) return b200::fail(301, "norm_bwd: D=%d must be a multiple of 8 and <= %d", D, MAX_D);
  if (T <= 0) return 0;
  int grid = b200::sm_count() * 2;
  if (grid > T) grid = T;
  cudaStream_t st = (cudaStream_t)stream;
  BwdArgs a{(const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)b,
            (const __nv_bfloat16*)dres, mean, rstd, (__nv_bfloat16*)dx, scratch, T, D, grid, st};
  int parts;
  if (mode == 0) parts = act ? dispatch_bwd<0, 1>(a) : dispatch_bwd<0, 0>(a);
  else parts = act ? dispatch_bwd<1, 1>(a) : dispatch_bwd<1, 0>(a);
  if (parts < 0) return -parts;
  b200::count_launch();
  if (int r = b200::check_launch("norm_bwd")) return r;
  if (scratch != nullptr && (dw != nullptr || db != nullptr)) {
    b200::launch(norm_bwd_reduce_kernel, dim3((D + 31) / 32, 2), 256, 0, st, scratch, parts, D, dw, db, accumulate);
    b200::count_launch();
    return b200::check_launch("norm_bwd_reduce");
  }
  return 0;
}
