// MXFP8 quantisation producers: bf16 [R, C] -> e4m3 codes + one UE8M0 scale per 32 elements
// along the contraction axis, in the layouts the block-scaled tcgen05 GEMM consumes directly.
//
// One pass over the input produces (either or both of)
//   * the row-wise copy     q_row [R, C]   scaled along C  (operand whose contraction axis is C)
//   * the column-wise copy  q_col [C, R]   scaled along R, written transposed, so that it is
//                                          again a K-major operand (contraction axis R)
// Scales are written pre-arranged for tcgen05.cp: the operand's rows are cut into tiles of
// `tile_rows` (the GEMM's M or N tile), each tile into atoms of 128 rows, and for every atom and
// every group of 4 scale columns (= 128 contraction elements) 512 bytes are stored as
//   byte[(r % 32) * 16 + (r / 32) * 4 + k],   r = row in atom, k = scale column in group,
// indexed [tile][k_group][atom].  The GEMM's TMA producer then moves whole atoms with plain bulk
// copies and the MMA warp forwards them to TMEM unchanged.
//
// Scale rule: e = ceil(log2(amax / 448)) clamped to [-127, 127], stored biased (e + 127); codes
// are round-to-nearest-even e4m3 of x * 2^-e with saturation.  amax == 0 gives scale 2^-127, codes 0.
//
// Reference counterparts: Transformer Engine's MXFP8/MXFP4 block-scaling recipes selected by
// small_llm_pretraining/primus/conf/llama3.1_8B-pretrain-fp4.yaml:108-112, the one-pass cast + amax
// kernels of generative_recommenders/ops/triton/bwd_fp8.py (_quantize_amax*), and the LN store of
// generative_recommenders/ops/hip/ln_store_mx6.cu (codes + E8M0 per 32).
#include <cuda_fp8.h>

#include "common.cuh"
#include "runtime.h"

namespace {

constexpr int TILE = 128;
// Shared-memory tile: rows of 64 words (two bf16 columns each) at a pitch of 68 words, and 4 words more every 16 rows.  Rows
// start on 16 bytes, so the row pass stores whole vectors (8 lanes cover all banks); in the column pass the eight lanes of a
// column, 16 rows apart, lie 4 banks apart and the four columns of a warp fill the banks between them.
constexpr int PITCH_W = 68;
constexpr int TILE_WORDS = TILE * PITCH_W + 8 * 4;
B200_DEVICE int tile_off(int r) { return r * PITCH_W + (r >> 4) * 4; }

// Largest magnitudes of the two columns of a word pair (bf16 values are compared as they are; a NaN loses, as with fmaxf).
B200_DEVICE uint32_t max2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmax2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
B200_DEVICE uint32_t abs2(uint32_t a) { return a & 0x7fff7fffu; }

// Biased exponent of the smallest power of two s with amax / s <= 448 = 1.75 * 2^8, amax given by its bf16 bits: its exponent
// less 8, one more where its fraction exceeds 1.75 (0x60 of 0x7f: adding 0x1f carries into the exponent).  No division; the
// limits are those of rounding amax / 448 up to a power of two in fp32: amax / 448 below the normal numbers gives 1,
// amax == 0 (or NaN alone) 0, infinity 254.
B200_DEVICE uint32_t e8m0_from_bits(uint32_t b) {
  const int e = max((int)((b + 0x1fu) >> 7) - 8, 1);
  return b >= 0x7f80u ? (b == 0x7f80u ? 254u : 0u) : (b == 0u ? 0u : (uint32_t)e);
}
B200_DEVICE float scale_inv_from_e8m0(uint32_t b) {
  // 2^-(b - 127)
  return __uint_as_float((uint32_t)(254 - (int)b) << 23);
}
B200_DEVICE uint32_t pack4_e4m3(float a, float b, float c, float d) {
  const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return (uint32_t)lo | ((uint32_t)hi << 16);
}
// byte offset of scale (row r of the operand, scale column kc) in the atom layout
B200_DEVICE long long sf_offset(long long r, int kc, int tile_rows, int atoms_per_tile, long long k_groups) {
  const long long tile = r / tile_rows;
  const int rr = (int)(r - tile * tile_rows);
  const int atom = rr >> 7, ra = rr & 127;
  return ((tile * k_groups + (kc >> 2)) * atoms_per_tile + atom) * 512 + (ra & 31) * 16 + (ra >> 5) * 4 + (kc & 3);
}

// Row quantisation of 8 values of a 32-block that four neighbouring lanes hold: codes and the block's scale byte.
B200_DEVICE uint2 quant_row8(const uint4& v, uint32_t& e) {
  uint32_t m = max2(max2(abs2(v.x), abs2(v.y)), max2(abs2(v.z), abs2(v.w)));
  m = max2(m, __shfl_xor_sync(0xffffffffu, m, 1));
  m = max2(m, __shfl_xor_sync(0xffffffffu, m, 2));
  e = e8m0_from_bits(max2(m, m >> 16) & 0xffffu);
  const float inv = scale_inv_from_e8m0(e);
  const float2 i2 = make_float2(inv, inv);
  const float2 a = fmul2(unpack_bf16x2(v.x), i2), b = fmul2(unpack_bf16x2(v.y), i2);
  const float2 c = fmul2(unpack_bf16x2(v.z), i2), d = fmul2(unpack_bf16x2(v.w), i2);
  return make_uint2(pack4_e4m3(a.x, a.y, b.x, b.y), pack4_e4m3(c.x, c.y, d.x, d.y));
}

// Column quantisation: this lane's 16 rows (sub * 16 ..) of the two columns of word `cw`; eight lanes (sub = 0 .. 7) walk the
// 128 rows.  Codes of the columns in qa / qb, scale bytes of their 32-blocks in ea / eb (equal in lanes sub and sub ^ 1).
B200_DEVICE void quant_col2(const uint32_t* tile, int sub, int cw, uint4& qa, uint4& qb, uint32_t& ea, uint32_t& eb) {
  uint32_t w[16];
  const uint32_t* t = tile + tile_off(sub * 16) + cw;
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i] = t[i * PITCH_W];
  uint32_t m = abs2(w[0]);
#pragma unroll
  for (int i = 1; i < 16; ++i) m = max2(m, abs2(w[i]));
  m = max2(m, __shfl_xor_sync(0xffffffffu, m, 1));
  ea = e8m0_from_bits(m & 0xffffu);
  eb = e8m0_from_bits(m >> 16);
  const float2 inv = make_float2(scale_inv_from_e8m0(ea), scale_inv_from_e8m0(eb));
  uint32_t a[4], b[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f0 = fmul2(unpack_bf16x2(w[4 * i]), inv), f1 = fmul2(unpack_bf16x2(w[4 * i + 1]), inv);
    const float2 f2 = fmul2(unpack_bf16x2(w[4 * i + 2]), inv), f3 = fmul2(unpack_bf16x2(w[4 * i + 3]), inv);
    a[i] = pack4_e4m3(f0.x, f1.x, f2.x, f3.x);
    b[i] = pack4_e4m3(f0.y, f1.y, f2.y, f3.y);
  }
  qa = make_uint4(a[0], a[1], a[2], a[3]);
  qb = make_uint4(b[0], b[1], b[2], b[3]);
}

B200_DEVICE void unpack8(const uint4& u, float (&f)[8]) {
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
B200_DEVICE uint4 pack8(const float (&o)[8]) {
  return make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]), pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
}

// What a launch reads and writes.  q_row / q_col may each be null; `live`: null, or the number of leading rows that count
// (a multiple of 128, read on the device): tiles past it are skipped and their outputs left as they are.
struct QuantArgs {
  const __nv_bfloat16* x;      // MODE 0: [R, C]; MODE 1, SwiGLU-backward kernel: gu [R, 2F]
  long long ldx;
  const __nv_bfloat16* aux;    // SwiGLU-backward kernel: da [R, F]
  long long ldaux;
  int R, C, F;
  uint8_t* q_row; uint8_t* sf_row; int row_tile;
  uint8_t* q_col; uint8_t* sf_col; int col_tile;
  const int* live;
};

// grid: (ceil(C / 128), R / 128); 256 threads.  R is a multiple of 128, C a multiple of 32: in the last column tile
// the columns past C read as zero and nothing is stored for them (their scale bytes are written as 0).
//   row pass:    a warp instruction covers 2 rows x 256 bytes of input (lane = 8 elements); a block of
//                32 elements is 4 lanes, so amax is two shuffles; codes leave as 2 x 128 contiguous bytes.
//   column pass: 8 lanes walk two columns (16 rows each, amax of a 32-block = one shuffle) and write each
//                column's 128 codes as one contiguous 128-byte piece of the transposed copy.
//   scales:      staged in shared memory and written as one 32-bit word per operand row.
//
// MODE selects what the tile is made of (the values are rounded to bf16 first, so the codes equal
// those of quantising the stand-alone kernel's bf16 output):
//   0  x[r, c]
//   1  SwiGLU forward   a[r, c] = silu(gu[r, c]) * gu[r, F + c],  x = gu [R, 2F], C = F
// (SwiGLU backward: quant_swiglu_bwd_kernel below.)
//
// Bound by memory as far as the instructions allow: two columns a lane, magnitudes compared as packed bf16 and a scale
// exponent without a division leave about 6 issue slots an element where 10 were.  36,900 live of 40,960 rows: 2880 columns row +
// column 91 -> 75 us (5.7 TB/s), SwiGLU of 2 x 2880 259 -> 157 us (an IEEE division an element before); 8192 x 2 x 14336 row alone
// 195 -> 145 us.
template <int MODE>
__global__ void __launch_bounds__(256, 4)
quant_mxfp8_kernel(const QuantArgs p) {
  b200::begin_kernel();
  __shared__ __align__(16) uint32_t tile[TILE_WORDS];
  __shared__ __align__(4) uint8_t sfs[2][TILE][4];     // [row pass | column pass][operand row][scale column]
  const int c0 = blockIdx.x * TILE, r0 = blockIdx.y * TILE;
  if (p.live != nullptr && r0 >= *p.live) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int sub_row = lane >> 4, chunk = lane & 15;
  const int C = p.C;
  const bool col_live = c0 + chunk * 8 < C;
  constexpr int STEP = MODE == 0 ? 8 : 4;              // vectors in flight per thread: 8 of one input, 4 of each of two
#pragma unroll
  for (int h = 0; h < 8; h += STEP) {
    uint4 v[STEP];
    {
      const __nv_bfloat16* src = p.x + (long long)(r0 + h * 16 + warp * 2 + sub_row) * p.ldx + c0 + chunk * 8;
      const long long pitch = 16 * p.ldx;
#pragma unroll
      for (int i = 0; i < STEP; ++i) v[i] = col_live ? *reinterpret_cast<const uint4*>(src + i * pitch) : make_uint4(0u, 0u, 0u, 0u);
      if constexpr (MODE == 1) {
        uint4 u[STEP];
#pragma unroll
        for (int i = 0; i < STEP; ++i)
          u[i] = col_live ? *reinterpret_cast<const uint4*>(src + p.F + i * pitch) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int i = 0; i < STEP; ++i) {
          float g[8], w[8];
          unpack8(v[i], g);
          unpack8(u[i], w);
#pragma unroll
          for (int j = 0; j < 8; ++j) g[j] = g[j] * sigmoid(g[j]) * w[j];
          v[i] = pack8(g);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < STEP; ++i) {
      const int r = (h + i) * 16 + warp * 2 + sub_row;
      if (p.q_row != nullptr) {
        uint32_t e;
        const uint2 q = quant_row8(v[i], e);
        if (col_live) *reinterpret_cast<uint2*>(p.q_row + (long long)(r0 + r) * C + c0 + chunk * 8) = q;
        if ((chunk & 3) == 0) sfs[0][r][chunk >> 2] = (uint8_t)e;
      }
      if (p.q_col != nullptr) *reinterpret_cast<uint4*>(tile + tile_off(r) + chunk * 4) = v[i];
    }
  }
  __syncthreads();
  if (p.q_row != nullptr && tid < TILE) {
    const long long o = sf_offset(r0 + tid, c0 >> 5, p.row_tile, (p.row_tile + 127) >> 7, (C + 127) >> 7);
    *reinterpret_cast<uint32_t*>(p.sf_row + o) = *reinterpret_cast<const uint32_t*>(&sfs[0][tid][0]);
  }
  if (p.q_col == nullptr) return;
  const int sub = lane & 7;                      // rows sub * 16 .. + 15 of the columns
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    const int cw = pass * 32 + warp * 4 + (lane >> 3), c = 2 * cw;
    uint4 qa, qb;
    uint32_t ea, eb;
    quant_col2(tile, sub, cw, qa, qb, ea, eb);
    if (c0 + c < C) {
      uint8_t* dst = p.q_col + (long long)(c0 + c) * p.R + r0 + sub * 16;
      *reinterpret_cast<uint4*>(dst) = qa;
      *reinterpret_cast<uint4*>(dst + p.R) = qb;
    }
    if ((sub & 1) == 0) { sfs[1][c][sub >> 1] = (uint8_t)ea; sfs[1][c + 1][sub >> 1] = (uint8_t)eb; }
  }
  __syncthreads();
  if (tid < TILE && c0 + tid < C) {
    const long long o = sf_offset(c0 + tid, r0 >> 5, p.col_tile, (p.col_tile + 127) >> 7, p.R >> 7);
    *reinterpret_cast<uint32_t*>(p.sf_col + o) = *reinterpret_cast<const uint32_t*>(&sfs[1][tid][0]);
  }
}

// SwiGLU backward quantised: dgu [R, 2F] (d gate | d up) from gu [R, 2F] and da [R, F]:
//   d gate = da * up * silu'(gate),  d up = da * silu(gate)
// grid: (ceil(F / 64), R / 128); 256 threads.  A CTA makes the 128 x 64 tiles of both halves at the same columns of F, so gate, up
// and da are read, and the sigmoid taken, once.  (A tile of either half by itself read them twice: 8192 x 2 x 8192 269 us at 2.5 TB/s,
// 8192 x 2 x 14336 484 -> 330 us; at widths that are no multiple of 128 a kernel of its own wrote dgu first, 191 + 174 -> 257 us
// for 36,900 x 2 x 2880.)  The shared tile holds d gate in its columns 0 - 63 and d up in 64 - 127.  F is a multiple of 32: the
// columns past F are neither read nor stored, and the scale bytes past 2F up to a whole word are written as 0.
__global__ void __launch_bounds__(256, 4)
quant_swiglu_bwd_kernel(const QuantArgs p) {
  b200::begin_kernel();
  __shared__ __align__(16) uint32_t tile[TILE_WORDS];
  __shared__ __align__(4) uint8_t sfr[TILE][4];        // row pass: scale columns of d gate (0, 1) and d up (2, 3)
  __shared__ __align__(4) uint8_t sfc[TILE][4];        // column pass
  const int c0 = blockIdx.x * 64, r0 = blockIdx.y * TILE;
  if (p.live != nullptr && r0 >= *p.live) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int sub_row = lane >> 3, chunk = lane & 7;     // 4 rows x 64 columns per warp instruction
  const int F = p.F, C = 2 * F;
  const bool col_live = c0 + chunk * 8 < F;
#pragma unroll
  for (int h = 0; h < 4; h += 2) {
    uint4 vg[2], vu[2], vd[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const long long row = r0 + (h + i) * 32 + warp * 4 + sub_row;
      vg[i] = vu[i] = vd[i] = make_uint4(0u, 0u, 0u, 0u);
      if (col_live) {
        vg[i] = *reinterpret_cast<const uint4*>(p.x + row * p.ldx + c0 + chunk * 8);
        vu[i] = *reinterpret_cast<const uint4*>(p.x + row * p.ldx + F + c0 + chunk * 8);
        vd[i] = *reinterpret_cast<const uint4*>(p.aux + row * p.ldaux + c0 + chunk * 8);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = (h + i) * 32 + warp * 4 + sub_row;
      float g[8], u[8], d[8];
      unpack8(vg[i], g);
      unpack8(vu[i], u);
      unpack8(vd[i], d);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float sg = sigmoid(g[j]);
        const float du = d[j] * (g[j] * sg);
        g[j] = d[j] * u[j] * sg * (1.f + g[j] * (1.f - sg));
        u[j] = du;
      }
      const uint4 o[2] = {pack8(g), pack8(u)};
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (p.q_row != nullptr) {
          uint32_t e;
          const uint2 q = quant_row8(o[s], e);
          if (col_live) *reinterpret_cast<uint2*>(p.q_row + (long long)(r0 + r) * C + s * F + c0 + chunk * 8) = q;
          if ((chunk & 3) == 0) sfr[r][s * 2 + (chunk >> 2)] = (uint8_t)e;
        }
        if (p.q_col != nullptr) *reinterpret_cast<uint4*>(tile + tile_off(r) + s * 32 + chunk * 4) = o[s];
      }
    }
  }
  __syncthreads();
  if (p.q_row != nullptr) {
    // (F may be an odd number of scale columns, so the halves of a word of d up's scales are not aligned: byte stores)
    const int r = tid & 127, s = tid >> 7;
    const int kc = (s * F + c0) >> 5, kend = ((s + 1) * F) >> 5, kpad = s == 1 ? (kend + 3) & ~3 : kend;
    const long long k_groups = (C + 127) >> 7;
    const int atoms = (p.row_tile + 127) >> 7;
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (kc + k < kend) p.sf_row[sf_offset(r0 + r, kc + k, p.row_tile, atoms, k_groups)] = sfr[r][s * 2 + k];
    if (c0 + 64 >= F)
      for (int k = kend; k < kpad; ++k) p.sf_row[sf_offset(r0 + r, k, p.row_tile, atoms, k_groups)] = 0;
  }
  if (p.q_col == nullptr) return;
  const int sub = lane & 7;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int cw = s * 32 + warp * 4 + (lane >> 3), c = 2 * (cw & 31);     // word of the tile, column of F's chunk
    uint4 qa, qb;
    uint32_t ea, eb;
    quant_col2(tile, sub, cw, qa, qb, ea, eb);
    if (c0 + c < F) {
      uint8_t* dst = p.q_col + (long long)(s * F + c0 + c) * p.R + r0 + sub * 16;
      *reinterpret_cast<uint4*>(dst) = qa;
      *reinterpret_cast<uint4*>(dst + p.R) = qb;
    }
    if ((sub & 1) == 0) { sfc[2 * cw][sub >> 1] = (uint8_t)ea; sfc[2 * cw + 1][sub >> 1] = (uint8_t)eb; }
  }
  __syncthreads();
  if (tid < TILE) {
    const int s = tid >> 6, c = c0 + (tid & 63);
    if (c < F) {
      const long long o = sf_offset(s * F + c, r0 >> 5, p.col_tile, (p.col_tile + 127) >> 7, p.R >> 7);
      *reinterpret_cast<uint32_t*>(p.sf_col + o) = *reinterpret_cast<const uint32_t*>(&sfc[tid][0]);
    }
  }
}

template <int MODE>
int launch_quant(const QuantArgs& p, cudaStream_t stream, const char* what) {
  b200::launch(quant_mxfp8_kernel<MODE>, dim3((p.C + TILE - 1) / TILE, p.R / TILE), 256, 0, stream, p);
  b200::count_launch();
  return b200::check_launch(what);
}

}  // namespace

// Bytes of the scale buffer of an operand with `rows` rows and `k` contraction elements whose rows
// are tiled by `tile_rows` in the GEMM.
B200_API long long b200_mxfp8_sf_bytes(long long rows, long long k, int tile_rows) {
  const long long tiles = (rows + tile_rows - 1) / tile_rows;
  const long long atoms = (tile_rows + 127) / 128;
  return tiles * ((k + 127) / 128) * atoms * 512;
}

// x: bf16 [R, C] with row pitch ldx (elements); R a multiple of 128, C a multiple of 32.
// q_row / sf_row (row-wise copy, rows tiled by row_tile) and q_col / sf_col (column-wise copy stored
// transposed as [C, R], rows tiled by col_tile) may each be null.  The scale bytes of an atom's rows past the operand's
// or the tile's last row are not written: the tensor core reads them for accumulator columns (rows) that nobody stores.
B200_API int b200_quant_mxfp8(const void* x, long long ldx, int R, int C, void* q_row, void* sf_row, int row_tile,
                              void* q_col, void* sf_col, int col_tile, const int* live, void* stream) {
  if (R % 128 != 0 || C % 32 != 0 || R <= 0 || C <= 0)
    return b200::fail(700, "quant_mxfp8: R=%d must be a multiple of 128 and C=%d of 32", R, C);
  if (ldx % 8 != 0 || ((uintptr_t)x & 15) != 0) return b200::fail(701, "quant_mxfp8: input must be 16-byte aligned");
  if ((q_row && (row_tile % 16 != 0 || row_tile <= 0)) || (q_col && (col_tile % 16 != 0 || col_tile <= 0)))
    return b200::fail(702, "quant_mxfp8: tile rows must be positive multiples of 16");
  const QuantArgs p = {(const __nv_bfloat16*)x, ldx, nullptr, 0, R, C, 0, (uint8_t*)q_row, (uint8_t*)sf_row, row_tile,
                       (uint8_t*)q_col, (uint8_t*)sf_col, col_tile, live};
  return launch_quant<0>(p, (cudaStream_t)stream, "quant_mxfp8");
}

// Quantised SwiGLU: the codes / scales of a = silu(gate) * up without writing a.
//   gu: bf16 [R, 2F] (gate columns first), pitch ldgu.  Outputs as b200_quant_mxfp8 for the matrix a [R, F].
B200_API int b200_quant_swiglu_mxfp8(const void* gu, long long ldgu, int R, int F, void* q_row, void* sf_row, int row_tile,
                                     void* q_col, void* sf_col, int col_tile, const int* live, void* stream) {
  if (R % 128 != 0 || F % 32 != 0 || R <= 0 || F <= 0)
    return b200::fail(710, "quant_swiglu: R=%d must be a multiple of 128 and F=%d of 32", R, F);
  if (ldgu % 8 != 0 || ((uintptr_t)gu & 15) != 0) return b200::fail(711, "quant_swiglu: input must be 16-byte aligned");
  const QuantArgs p = {(const __nv_bfloat16*)gu, ldgu, nullptr, 0, R, F, F, (uint8_t*)q_row, (uint8_t*)sf_row, row_tile,
                       (uint8_t*)q_col, (uint8_t*)sf_col, col_tile, live};
  return launch_quant<1>(p, (cudaStream_t)stream, "quant_swiglu_mxfp8");
}

// Quantised SwiGLU backward: the codes / scales of dgu [R, 2F] (d gate | d up) from da [R, F] and gu [R, 2F].
B200_API int b200_quant_swiglu_bwd_mxfp8(const void* da, long long ldda, const void* gu, long long ldgu, int R, int F,
                                         void* q_row, void* sf_row, int row_tile, void* q_col, void* sf_col, int col_tile,
                                         const int* live, void* stream) {
  if (R % 128 != 0 || F % 32 != 0 || R <= 0 || F <= 0)
    return b200::fail(712, "quant_swiglu_bwd: R=%d must be a multiple of 128 and F=%d of 32", R, F);
  if (ldgu % 8 != 0 || ldda % 8 != 0 || (((uintptr_t)gu | (uintptr_t)da) & 15) != 0)
    return b200::fail(713, "quant_swiglu_bwd: inputs must be 16-byte aligned");
  const QuantArgs p = {(const __nv_bfloat16*)gu, ldgu, (const __nv_bfloat16*)da, ldda, R, 2 * F, F, (uint8_t*)q_row,
                       (uint8_t*)sf_row, row_tile, (uint8_t*)q_col, (uint8_t*)sf_col, col_tile, live};
  b200::launch(quant_swiglu_bwd_kernel, dim3((F + 63) / 64, R / TILE), 256, 0, (cudaStream_t)stream, p);
  b200::count_launch();
  return b200::check_launch("quant_swiglu_bwd_mxfp8");
}
