// Bandwidth-bound elementwise kernels (bf16 storage, fp32 math, 16-byte accesses):
// rotary embedding on a packed QKV buffer, SwiGLU / GELU and their backward, embedding row
// gather and its scatter-add backward, bf16 residual add, fp32 accumulate.
//
// Reference counterparts: the fused single-QKV RoPE and fused SwiGLU selected by
// small_llm_pretraining/primus/conf/llama3.1_8B-pretrain-fp4.yaml:62,122-123 (Primus-Turbo),
// generative_recommenders/ops/triton/triton_swiglu.py (_swiglu_fwd_kernel) and the dedup-expand
// row gather of generative_recommenders/dlrm_v4/train/ec_expand_gather.py.
#include "common.cuh"
#include "runtime.h"

namespace {

B200_DEVICE void ld8(const __nv_bfloat16* p, float (&f)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
B200_DEVICE void st8(__nv_bfloat16* p, const float (&f)[8]) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]),
                                            pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

// ---------------------------------------------------------------------------------------
// RoPE ("rotate-half" convention: pairs are (i, i + hd/2)), in place on rows of
// [T, row_stride] holding n_rot_heads heads of size hd starting at column col0.
// cos/sin tables are fp32 [S, hd/2]; position of token t is pos[t] if given, else t % S.
// sign = +1 forward, -1 backward (transpose of the rotation).
// ---------------------------------------------------------------------------------------
__global__ void rope_kernel(__nv_bfloat16* __restrict__ buf, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, const int* __restrict__ pos, long long T, int S,
                            long long row_stride, int col0, int n_heads, int hd, float sign) {
  b200::begin_kernel();
  const int half = hd / 2;
  const int vec_per_head = half / 8;  // each work item rotates 8 pairs
  const long long total = T * n_heads * vec_per_head;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int v = (int)(i % vec_per_head);
    const long long r = i / vec_per_head;
    const int h = (int)(r % n_heads);
    const long long t = r / n_heads;
    const int p = pos ? pos[t] : (int)(t % S);
    __nv_bfloat16* base = buf + t * row_stride + col0 + h * hd + v * 8;
    float x1[8], x2[8], o1[8], o2[8];
    ld8(base, x1);
    ld8(base + half, x2);
    const float4* c4 = reinterpret_cast<const float4*>(cos_t + (long long)p * half + v * 8);
    const float4* s4 = reinterpret_cast<const float4*>(sin_t + (long long)p * half + v * 8);
    float c[8], s[8];
    float4 ca = c4[0], cb = c4[1], sa = s4[0], sb = s4[1];
    c[0] = ca.x; c[1] = ca.y; c[2] = ca.z; c[3] = ca.w; c[4] = cb.x; c[5] = cb.y; c[6] = cb.z; c[7] = cb.w;
    s[0] = sa.x; s[1] = sa.y; s[2] = sa.z; s[3] = sa.w; s[4] = sb.x; s[5] = sb.y; s[6] = sb.z; s[7] = sb.w;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sj = s[j] * sign;
      o1[j] = x1[j] * c[j] - x2[j] * sj;
      o2[j] = x2[j] * c[j] + x1[j] * sj;
    }
    st8(base, o1);
    st8(base + half, o2);
  }
}

// Gradients of the rotated projections, finished in one pass: head h < hq of a row comes from the attention backward's fp32
// dq [T, hq, hd], the next hkv heads (k) from `buf` itself; every one of them is rotated back and stored to `buf` as bf16.  A
// copy of dq into `buf` and the rotation in place read and wrote the q columns twice and rounded them twice (8192 tokens, 64 / 8
// heads of 64: 82 + 22 -> 34 us; 4096, 64 / 8 of 128: 80 + 24 -> 36).
template <typename I>
__global__ void __launch_bounds__(256)
rope_grad_kernel(const float* __restrict__ dq, __nv_bfloat16* __restrict__ buf, const float* __restrict__ cos_t,
                 const float* __restrict__ sin_t, I total, int S, long long row_stride, I hq, I heads, int hd) {
  b200::begin_kernel();
  const int half = hd / 2;
  const I vec_per_head = half / 8, per_row = heads * vec_per_head;
  for (I i = blockIdx.x * (I)blockDim.x + threadIdx.x; i < total; i += (I)gridDim.x * blockDim.x) {
    const I t = i / per_row, r = i - t * per_row, h = r / vec_per_head, v = r - h * vec_per_head;
    const long long at = (long long)(t % (I)S) * half + v * 8;
    __nv_bfloat16* base = buf + (long long)t * row_stride + h * hd + v * 8;
    float x1[8], x2[8], c[8], s[8], o1[8], o2[8];
    auto ldf = [](const float* p, float (&f)[8]) {
      const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
      f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    };
    if (h < hq) {
      const float* src = dq + ((long long)t * hq + h) * hd + v * 8;
      ldf(src, x1);
      ldf(src + half, x2);
    } else {
      ld8(base, x1);
      ld8(base + half, x2);
    }
    ldf(cos_t + at, c);
    ldf(sin_t + at, s);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o1[j] = x1[j] * c[j] + x2[j] * s[j];
      o2[j] = x2[j] * c[j] - x1[j] * s[j];
    }
    st8(base, o1);
    st8(base + half, o2);
  }
}

// ---------------------------------------------------------------------------------------
// SwiGLU: a[t, f] = silu(gu[t, f]) * gu[t, F + f]  (gate columns first, up columns second)
// ---------------------------------------------------------------------------------------
// One vector of SwiGLU, forward and backward (g, u: gate and up; d: gradient of the product).
B200_DEVICE void swiglu_vec(const __nv_bfloat16* g_in, const __nv_bfloat16* u_in, __nv_bfloat16* out) {
  float g[8], u[8], o[8];
  ld8(g_in, g);
  ld8(u_in, u);
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = g[j] * sigmoid(g[j]) * u[j];
  st8(out, o);
}
B200_DEVICE void swiglu_grad_vec(const __nv_bfloat16* g_in, const __nv_bfloat16* u_in, const __nv_bfloat16* d_in, __nv_bfloat16* dg_out,
                                 __nv_bfloat16* du_out) {
  float g[8], u[8], d[8], dg[8], du[8];
  ld8(g_in, g);
  ld8(u_in, u);
  ld8(d_in, d);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float sg = sigmoid(g[j]);
    const float silu = g[j] * sg;
    du[j] = d[j] * silu;
    dg[j] = d[j] * u[j] * sg * (1.f + g[j] * (1.f - sg));
  }
  st8(dg_out, dg);
  st8(du_out, du);
}
template <typename I>
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ a, I T,
                  int F) {
  b200::begin_kernel();
  const I vpr = F / 8, total = T * vpr;
  for (I i = blockIdx.x * (I)blockDim.x + threadIdx.x; i < total; i += (I)gridDim.x * blockDim.x) {
    const long long t = i / vpr;
    const int v = (int)(i - (I)t * vpr);
    swiglu_vec(gu + t * 2 * F + v * 8, gu + t * 2 * F + F + v * 8, a + t * F + v * 8);
  }
}
template <typename I>
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ da, const __nv_bfloat16* __restrict__ gu,
                                  __nv_bfloat16* __restrict__ dgu, I T, int F) {
  b200::begin_kernel();
  const I vpr = F / 8, total = T * vpr;
  for (I i = blockIdx.x * (I)blockDim.x + threadIdx.x; i < total; i += (I)gridDim.x * blockDim.x) {
    const long long t = i / vpr;
    const int v = (int)(i - (I)t * vpr);
    swiglu_grad_vec(gu + t * 2 * F + v * 8, gu + t * 2 * F + F + v * 8, da + t * F + v * 8, dgu + t * 2 * F + v * 8,
                    dgu + t * 2 * F + F + v * 8);
  }
}

// The same over the 256-row tiles of an expert-grouped buffer: a tile's rows up to the multiple of 64 behind its expert's last one,
// nothing in tiles of no expert.  (8000 pairs on 32 experts: 9000 of 16,192 rows, 90 / 86 / 78 -> 33 / 36 / 39 us for forward,
// recomputed forward and backward of 2 x 2880 columns, index divisions included.)  da == nullptr: forward.
__global__ void __launch_bounds__(256)
swiglu_tiles_kernel(const __nv_bfloat16* __restrict__ da, const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out, int F,
                    const int* __restrict__ tile_expert, const int* __restrict__ seg, const int* __restrict__ counts) {
  b200::begin_kernel();
  const int tile = blockIdx.y, e = tile_expert[tile];
  if (e < 0) return;
  const int n = min(256, (seg[e] + counts[e] - tile * 256 + 63) / 64 * 64), vpr = F / 8;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n * vpr; i += gridDim.x * 256) {
    const int r = i / vpr, v = (i - r * vpr) * 8;
    const long long t = (long long)tile * 256 + r;
    const __nv_bfloat16* g = gu + t * 2 * F + v;
    if (da == nullptr) swiglu_vec(g, g + F, out + t * F + v);
    else swiglu_grad_vec(g, g + F, da + t * F + v, out + t * 2 * F + v, out + t * 2 * F + F + v);
  }
}

// GELU (tanh approximation), used by the MMDiT MLPs: x / 2 (1 + tanh u) = x sigmoid(2 u), u = k (x + 0.044715 x^3); its
// derivative, with s = sigmoid(2 u), is s + 2 x s (1 - s) u'.  (tanhf and its branch held both kernels to half the memory rate,
// and 1 + tanh u cancels for a negative x.)
B200_DEVICE float gelu_tanh(float x) {
  const float k2 = 2.f * 0.7978845608028654f;
  return x * sigmoid(k2 * (x + 0.044715f * x * x * x));
}
B200_DEVICE float gelu_tanh_grad(float x) {
  const float k2 = 2.f * 0.7978845608028654f;
  const float s = sigmoid(k2 * (x + 0.044715f * x * x * x));
  const float c = fminf(fmaxf(x, -16.f), 16.f);      // beyond, s (1 - s) is 0 and the factor beside it must not overflow
  return s + c * s * (1.f - s) * k2 * (1.f + 3.f * 0.044715f * c * c);
}
// rows x vpr vectors of 8; pitches in elements (a plain tensor is one row)
template <typename I>
__global__ void __launch_bounds__(256) gelu_fwd_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, __nv_bfloat16* __restrict__ y, long long ldy,
                                I total, I vpr) {
  b200::begin_kernel();
  for (I i = blockIdx.x * (I)blockDim.x + threadIdx.x; i < total; i += (I)gridDim.x * blockDim.x) {
    const long long r = i / vpr, c = (long long)(i - (I)r * vpr) * 8;
    float a[8], o[8];
    ld8(x + r * ldx + c, a);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = gelu_tanh(a[j]);
    st8(y + r * ldy + c, o);
  }
}
template <typename I>
__global__ void __launch_bounds__(256) gelu_bwd_kernel(const __nv_bfloat16* __restrict__ dy, long long ldg, const __nv_bfloat16* __restrict__ x, long long ldx,
                                __nv_bfloat16* __restrict__ dx, long long ldd, I total, I vpr) {
  b200::begin_kernel();
  for (I i = blockIdx.x * (I)blockDim.x + threadIdx.x; i < total; i += (I)gridDim.x * blockDim.x) {
    const long long r = i / vpr, c = (long long)(i - (I)r * vpr) * 8;
    float a[8], d[8], o[8];
    ld8(x + r * ldx + c, a);
    ld8(dy + r * ldg + c, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = d[j] * gelu_tanh_grad(a[j]);
    st8(dx + r * ldd + c, o);
  }
}

// ---------------------------------------------------------------------------------------
// Embedding gather: out[t, :] = table[ids[t], :] (bf16, D % 8 == 0); ids < 0 give zero rows.
// ---------------------------------------------------------------------------------------
__global__ void gather_rows_kernel(const __nv_bfloat16* __restrict__ table, const long long* __restrict__ ids,
                                   __nv_bfloat16* __restrict__ out, long long T, int D, long long rows, int* status) {
  b200::begin_kernel();
  const int vpr = D / 8;
  const long long total = T * vpr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vpr;
    const int v = (int)(i % vpr);
    const long long id = ids[t];
    uint4 u = make_uint4(0, 0, 0, 0);
    if (id >= 0 && id < rows) u = *reinterpret_cast<const uint4*>(table + id * D + v * 8);
    else if (v == 0) B200_BOUNDS_REPORT(status, 401);
    *reinterpret_cast<uint4*>(out + t * D + v * 8) = u;
  }
}
// grad_table[ids[t], :] += dy[t, :]  (fp32 atomics; used for the vocabulary embedding)
__global__ void scatter_add_rows_kernel(const __nv_bfloat16* __restrict__ dy, const long long* __restrict__ ids,
                                        float* __restrict__ grad, long long T, int D, long long rows, int* status) {
  b200::begin_kernel();
  const int vpr = D / 8;
  const long long total = T * vpr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vpr;
    const int v = (int)(i % vpr);
    const long long id = ids[t];
    if (id < 0 || id >= rows) {
      if (v == 0) B200_BOUNDS_REPORT(status, 402);
      continue;
    }
    float d[8];
    ld8(dy + t * D + v * 8, d);
    float* g = grad + id * D + v * 8;
    if ((reinterpret_cast<uintptr_t>(grad) & 15) == 0) {       // two 16-byte reductions (8192 x 4096: 208 -> 74 us)
      atomicAdd(reinterpret_cast<float4*>(g), make_float4(d[0], d[1], d[2], d[3]));
      atomicAdd(reinterpret_cast<float4*>(g) + 1, make_float4(d[4], d[5], d[6], d[7]));
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) atomicAdd(g + j, d[j]);
    }
  }
}

// y = a + b (bf16)
__global__ void add_bf16_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                                __nv_bfloat16* __restrict__ y, long long n8) {
  b200::begin_kernel();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    float x[8], z[8];
    ld8(a + i * 8, x);
    ld8(b + i * 8, z);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] += z[j];
    st8(y + i * 8, x);
  }
}
// acc(fp32) += src(bf16)
__global__ void accum_f32_bf16_kernel(float* __restrict__ acc, const __nv_bfloat16* __restrict__ src, long long n8) {
  b200::begin_kernel();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    float x[8];
    ld8(src + i * 8, x);
    float4* a4 = reinterpret_cast<float4*>(acc + i * 8);
    float4 p = a4[0], q = a4[1];
    p.x += x[0]; p.y += x[1]; p.z += x[2]; p.w += x[3];
    q.x += x[4]; q.y += x[5]; q.z += x[6]; q.w += x[7];
    a4[0] = p; a4[1] = q;
  }
}

// Index type of a grid-stride loop over `work` items: 32 bits where they hold the indices (the loop steps past `work` once, by at
// most a grid); a 64-bit division per vector costs more than the vector's arithmetic.
inline bool fits32(long long work) { return work < (1ll << 31); }

inline int grid_for(long long work, int threads) {
  long long g = (work + threads - 1) / threads;
  long long cap = (long long)b200::sm_count() * 16;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace

B200_API int b200_rope(void* buf, const float* cos_t, const float* sin_t, const int* pos, long long T, int S,
                       long long row_stride, int col0, int n_heads, int hd, int backward, void* stream) {
  if (hd % 16 != 0 || row_stride % 8 != 0 || col0 % 8 != 0)
    return b200::fail(400, "rope: head dim %d must be a multiple of 16, stride/offset multiples of 8", hd);
  const long long work = T * n_heads * (hd / 16);
  if (work == 0) return 0;
  b200::launch(rope_kernel, grid_for(work, 256), 256, 0, (cudaStream_t)stream, (__nv_bfloat16*)buf, cos_t, sin_t, pos, T, S,
                                                                     row_stride, col0, n_heads, hd,
                                                                     backward ? -1.f : 1.f);
  b200::count_launch();
  return b200::check_launch("rope");
}
// dq: fp32 [T, hq, hd] contiguous; buf: bf16 rows [hq | hkv | ...] x hd (pitch row_stride) whose k columns hold dk.
B200_API int b200_rope_grad(const float* dq, void* buf, const float* cos_t, const float* sin_t, long long T, int S, long long row_stride,
                            int hq, int hkv, int hd, void* stream) {
  if (hd % 16 != 0 || row_stride % 8 != 0 || S <= 0 || (((uintptr_t)dq | (uintptr_t)buf | (uintptr_t)cos_t | (uintptr_t)sin_t) & 15) != 0)
    return b200::fail(406, "rope_grad: head dim %d must be a multiple of 16, the row pitch of 8, pointers 16-byte aligned", hd);
  const long long work = T * (hq + hkv) * (hd / 16);
  if (work == 0) return 0;
  if (fits32(work))
    b200::launch(rope_grad_kernel<uint32_t>, grid_for(work, 256), 256, 0, (cudaStream_t)stream, 
        dq, (__nv_bfloat16*)buf, cos_t, sin_t, (uint32_t)work, S, row_stride, (uint32_t)hq, (uint32_t)(hq + hkv), hd);
  else
    b200::launch(rope_grad_kernel<long long>, grid_for(work, 256), 256, 0, (cudaStream_t)stream, 
        dq, (__nv_bfloat16*)buf, cos_t, sin_t, work, S, row_stride, hq, hq + hkv, hd);
  b200::count_launch();
  return b200::check_launch("rope_grad");
}
B200_API int b200_swiglu_fwd(const void* gu, void* a, long long T, int F, void* stream) {
  if (F % 8 != 0) return b200::fail(401, "swiglu: F=%d must be a multiple of 8", F);
  if (T == 0) return 0;
  const long long work = T * (F / 8);
  if (fits32(work)) b200::launch(swiglu_fwd_kernel<uint32_t>, grid_for(work, 256), 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)gu, (__nv_bfloat16*)a, (uint32_t)T, F);
  else b200::launch(swiglu_fwd_kernel<long long>, grid_for(work, 256), 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)gu, (__nv_bfloat16*)a, T, F);
  b200::count_launch();
  return b200::check_launch("swiglu_fwd");
}
B200_API int b200_swiglu_bwd(const void* da, const void* gu, void* dgu, long long T, int F, void* stream) {
  if (F % 8 != 0) return b200::fail(401, "swiglu: F=%d must be a multiple of 8", F);
  if (T == 0) return 0;
  const long long work = T * (F / 8);
  if (fits32(work))
    b200::launch(swiglu_bwd_kernel<uint32_t>, grid_for(work, 256), 256, 0, (cudaStream_t)stream, 
        (const __nv_bfloat16*)da, (const __nv_bfloat16*)gu, (__nv_bfloat16*)dgu, (uint32_t)T, F);
  else
    b200::launch(swiglu_bwd_kernel<long long>, grid_for(work, 256), 256, 0, (cudaStream_t)stream, 
        (const __nv_bfloat16*)da, (const __nv_bfloat16*)gu, (__nv_bfloat16*)dgu, T, F);
  b200::count_launch();
  return b200::check_launch("swiglu_bwd");
}
static void run_gelu_fwd(const void* x, long long ldx, void* y, long long ldy, long long work, long long vpr, cudaStream_t st) {
  if (fits32(work)) b200::launch(gelu_fwd_kernel<uint32_t>, grid_for(work, 256), 256, 0, st, (const __nv_bfloat16*)x, ldx, (__nv_bfloat16*)y, ldy, (uint32_t)work, (uint32_t)vpr);
  else b200::launch(gelu_fwd_kernel<long long>, grid_for(work, 256), 256, 0, st, (const __nv_bfloat16*)x, ldx, (__nv_bfloat16*)y, ldy, work, vpr);
  b200::count_launch();
}
static void run_gelu_bwd(const void* dy, long long ldg, const void* x, long long ldx, void* dx, long long ldd, long long work, long long vpr,
                         cudaStream_t st) {
  if (fits32(work))
    b200::launch(gelu_bwd_kernel<uint32_t>, grid_for(work, 256), 256, 0, st, (const __nv_bfloat16*)dy, ldg, (const __nv_bfloat16*)x, ldx,
                                                                   (__nv_bfloat16*)dx, ldd, (uint32_t)work, (uint32_t)vpr);
  else
    b200::launch(gelu_bwd_kernel<long long>, grid_for(work, 256), 256, 0, st, (const __nv_bfloat16*)dy, ldg, (const __nv_bfloat16*)x, ldx,
                                                                    (__nv_bfloat16*)dx, ldd, work, vpr);
  b200::count_launch();
}
B200_API int b200_gelu_fwd(const void* x, void* y, long long n, void* stream) {
  if (n % 8 != 0) return b200::fail(402, "gelu: n=%lld must be a multiple of 8", n);
  if (n == 0) return 0;
  run_gelu_fwd(x, n, y, n, n / 8, n / 8, (cudaStream_t)stream);
  return b200::check_launch("gelu_fwd");
}
B200_API int b200_gelu_bwd(const void* dy, const void* x, void* dx, long long n, void* stream) {
  if (n % 8 != 0) return b200::fail(402, "gelu: n=%lld must be a multiple of 8", n);
  if (n == 0) return 0;
  run_gelu_bwd(dy, n, x, n, dx, n, n / 8, n / 8, (cudaStream_t)stream);
  return b200::check_launch("gelu_bwd");
}
// swiglu_tiles_kernel over n_tiles tiles of 256 rows: out [rows, F] from gu [rows, 2F], or with da [rows, F] out [rows, 2F].
B200_API int b200_swiglu_tiles(const void* da, const void* gu, void* out, int F, const int* tile_expert, const int* seg, const int* counts,
                               int n_tiles, void* stream) {
  if (F % 8 != 0) return b200::fail(401, "swiglu: F=%d must be a multiple of 8", F);
  if (n_tiles <= 0 || F <= 0) return 0;
  if (n_tiles > 65535) return b200::fail(407, "swiglu_tiles: %d tiles are too many", n_tiles);
  b200::launch(swiglu_tiles_kernel, dim3(32, n_tiles), 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)da, (const __nv_bfloat16*)gu,
                                                                           (__nv_bfloat16*)out, F, tile_expert, seg, counts);
  b200::count_launch();
  return b200::check_launch("swiglu_tiles");
}
B200_API int b200_gather_rows(const void* table, const long long* ids, void* out, long long T, int D, long long rows,
                              void* stream) {
  if (D % 8 != 0) return b200::fail(403, "gather_rows: D=%d must be a multiple of 8", D);
  if (T == 0) return 0;
  b200::launch(gather_rows_kernel, grid_for(T * (D / 8), 256), 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)table, ids,
                                                                                  (__nv_bfloat16*)out, T, D, rows, b200::status_ptr());
  b200::count_launch();
  return b200::check_launch("gather_rows");
}
B200_API int b200_scatter_add_rows(const void* dy, const long long* ids, float* grad, long long T, int D,
                                   long long rows, void* stream) {
  if (D % 8 != 0) return b200::fail(403, "scatter_add_rows: D=%d must be a multiple of 8", D);
  if (T == 0) return 0;
  b200::launch(scatter_add_rows_kernel, grid_for(T * (D / 8), 256), 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)dy, ids,
                                                                                       grad, T, D, rows, b200::status_ptr());
  b200::count_launch();
  return b200::check_launch("scatter_add_rows");
}
B200_API int b200_add_bf16(const void* a, const void* b, void* y, long long n, void* stream) {
  if (n % 8 != 0) return b200::fail(404, "add_bf16: n=%lld must be a multiple of 8", n);
  if (n == 0) return 0;
  b200::launch(add_bf16_kernel, grid_for(n / 8, 256), 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)a, (const __nv_bfloat16*)b,
                                                                         (__nv_bfloat16*)y, n / 8);
  b200::count_launch();
  return b200::check_launch("add_bf16");
}
B200_API int b200_accum_f32_bf16(float* acc, const void* src, long long n, void* stream) {
  if (n % 8 != 0) return b200::fail(405, "accum: n=%lld must be a multiple of 8", n);
  if (n == 0) return 0;
  b200::launch(accum_f32_bf16_kernel, grid_for(n / 8, 256), 256, 0, (cudaStream_t)stream, acc, (const __nv_bfloat16*)src, n / 8);
  b200::count_launch();
  return b200::check_launch("accum_f32_bf16");
}

// GELU on [rows, cols] blocks of wider matrices (pitches in elements, multiples of 8 like cols).
B200_API int b200_gelu_fwd_rows(const void* x, long long ldx, void* y, long long ldy, long long rows, long long cols, void* stream) {
  if (cols % 8 != 0 || ldx % 8 != 0 || ldy % 8 != 0) return b200::fail(402, "gelu_rows: %lld columns, pitches %lld / %lld (x8)", cols, ldx, ldy);
  if (rows == 0 || cols == 0) return 0;
  run_gelu_fwd(x, ldx, y, ldy, rows * (cols / 8), cols / 8, (cudaStream_t)stream);
  return b200::check_launch("gelu_fwd_rows");
}
B200_API int b200_gelu_bwd_rows(const void* dy, long long ldg, const void* x, long long ldx, void* dx, long long ldd, long long rows,
                                long long cols, void* stream) {
  if (cols % 8 != 0 || ldg % 8 != 0 || ldx % 8 != 0 || ldd % 8 != 0)
    return b200::fail(402, "gelu_rows: %lld columns, pitches %lld / %lld / %lld (x8)", cols, ldg, ldx, ldd);
  if (rows == 0 || cols == 0) return 0;
  run_gelu_bwd(dy, ldg, x, ldx, dx, ldd, rows * (cols / 8), cols / 8, (cudaStream_t)stream);
  return b200::check_launch("gelu_bwd_rows");
}
