// Grouped (per-expert) GEMMs of the MoE layer on the CTA-pair tcgen05 core (gemm_core.cuh), MXFP8 and bf16.  MXFP8:
// e4m3 codes with one UE8M0 scale per 32 contraction elements, block-scaled MMAs, one persistent
// launch per GEMM driven by the device-resident dispatch plan (no host read of the routing result).
//
//   rows   (forward, dgrad)  D[r, :] = A[r, :] * W[e(r)]^T      A: the padded row buffer (expert segments
//                            start at multiples of 256 rows), W: the experts' matrices stacked [(E * N), K]
//   wgrad                    D[e] += Y^T[:, seg_e] * X^T[:, seg_e]^T   both operands are the column-wise
//                            (transposed) quantised copies, so the contraction over an expert's rows is K-major
//
// bf16 (b200_gemm_grouped_pair_*) runs the same schedules on the row buffer and the weights as they are.
// Before, bf16 experts ran one CTA per 128-row tile (gemm_grouped.cu, still the path of 128-row segments), and weight
// gradients were added into cleared tensors: for block-scaled experts 3.2 GB of fp32 cleared, added into and converted per
// layer.  Layer of 32 experts of 2880 x 2880, top-4, forward + backward: 2000 tokens bf16 3.99 -> 3.25 ms, 8192 tokens
// block-scaled 8.33 -> 6.47 ms (0.25 ms of either from the attention and dense GEMMs).
//
// The reference gets this stage from its grouped GEMM / fused grouped MLP with MX-scaled operands
// (small_llm_moe_pretraining/primus/conf/gpt_oss_20B-MXFP4-deosc-mlperf-pretrain.yaml:130-167,186-222).
#include "gemm_core.cuh"

namespace {

using namespace gemmcore;

// N tile: a column tile must not straddle two experts of the stacked weight, so it has to divide N.
int grouped_bn(int N) {
  if (N % 192 == 0) return 192;
  if (N % 128 == 0) return 128;
  return 0;
}

template <int BN>
int run_grouped(const void* a_q, const void* sfa, const void* b_q, const void* sfb, void* d, const PairParams& p0,
                long long a_rows_total, long long b_rows_total, long long d_rows_total, long long lda, long long ldb,
                long long ldd, cudaStream_t stream, const char* what) {
  CUtensorMap tmA, tmB, tmSFA, tmSFB, tmD, tmDt;
  int r;
  const int K = p0.K;
  if ((r = b200::make_tmap_2d(&tmA, b200::DT_U8, a_q, K, a_rows_total, lda, 128, 128, b200::SWZ_128))) return r;
  if ((r = b200::make_tmap_2d(&tmB, b200::DT_U8, b_q, K, b_rows_total, ldb, 128, BN / 2, b200::SWZ_128))) return r;
  const int kg = (K + 127) / 128, atoms = (BN + 127) / 128;
  const long long sfa_rows = ((a_rows_total + 127) / 128) * kg;
  const long long sfb_rows = (b_rows_total / BN) * kg * atoms;
  if ((r = b200::make_tmap_2d(&tmSFA, b200::DT_I32, sfa, 128, sfa_rows, 512, 128, 2, b200::SWZ_NONE))) return r;
  if ((r = b200::make_tmap_2d(&tmSFB, b200::DT_I32, sfb, 128, sfb_rows, 512, 128, 2 * atoms, b200::SWZ_NONE))) return r;
  if ((r = make_out_tmap<BN>(&tmD, &tmDt, d, (int)d_rows_total, p0.N, ldd, p0.epi.out_f32))) return r;
  return launch_pair<KIND_MXFP8, BN, 2>(tmA, tmB, tmSFA, tmSFB, tmD, tmDt, p0, stream, what);
}

}  // namespace

// N tile the grouped kernels use for per-expert output width N (0: no tile divides N - use the bf16 path).
// The B operand's scales must be laid out with this tile height by the quantiser.
B200_API int b200_gemm_grouped_mx_bn(int N) { return grouped_bn(N); }

// a_q [rows, K] e4m3 (pitch lda bytes) with scale atoms sfa (tile rows 128); b_q [(E * N), K] (pitch ldb) with
// scale atoms sfb (tile rows b200_gemm_grouped_mx_bn(N)); d [rows, N] bf16 or fp32 (pitch ldd elements);
// tile_expert [rows / 256] on the device.  rows must be a multiple of 256, K of 32.
B200_API int b200_gemm_grouped_mx_rows(const void* a_q, const void* sfa, const void* b_q, const void* sfb, void* d,
                                       const int* tile_expert, int rows, int N, int K, int E, long long lda, long long ldb,
                                       long long ldd, int out_f32, float alpha, void* stream) {
  const int BN = grouped_bn(N);
  if (rows <= 0 || rows % 256 != 0 || K <= 0 || K % 32 != 0 || E <= 0 || BN == 0)
    return b200::fail(830, "gemm_grouped_mx_rows: rows=%d (x256) N=%d (x128 or x192) K=%d (x32) E=%d", rows, N, K, E);
  PairParams p = {};
  p.grp.mode = 1; p.grp.E = E; p.grp.tile_expert = tile_expert;
  p.M = rows; p.N = N; p.K = K;
  p.group_m = 16;               // 16 row tiles (4096 rows) stay in L2 while their experts' weight tiles stream once
  p.epi.M = rows; p.epi.N = N;
  p.epi.out_f32 = out_f32 ? 1 : 0;
  p.epi.alpha = alpha;
  p.status = b200::status_ptr();
  if (BN == 192)
    return run_grouped<192>(a_q, sfa, b_q, sfb, d, p, rows, (long long)E * N, rows, lda, ldb, ldd, (cudaStream_t)stream,
                            "gemm_grouped_mx_rows");
  return run_grouped<128>(a_q, sfa, b_q, sfb, d, p, rows, (long long)E * N, rows, lda, ldb, ldd, (cudaStream_t)stream,
                          "gemm_grouped_mx_rows");
}

// a_q [M, T] / b_q [N, T]: column-wise quantised copies (contraction over the T rows of the padded buffer; pitches
// lda / ldb bytes; scale tiles 128 / b200_gemm_grouped_mx_bn(N)); seg [E + 1] padded segment offsets (multiples of
// 256) on the device; d [E, M, N] contiguous, bf16 or fp32.  M must be a multiple of 32.  accumulate: add into d;
// otherwise all of d is written (zeros for an expert without rows).
B200_API int b200_gemm_grouped_mx_wgrad(const void* a_q, const void* sfa, const void* b_q, const void* sfb, void* d,
                                        const int* seg, int T, int M, int N, int E, long long lda, long long ldb, int out_f32,
                                        int accumulate, float alpha, void* stream) {
  const int BN = grouped_bn(N);
  if (T <= 0 || T % 256 != 0 || M <= 0 || M % 32 != 0 || E <= 0 || BN == 0)
    return b200::fail(831, "gemm_grouped_mx_wgrad: T=%d (x256) M=%d (x32) N=%d (x128 or x192) E=%d", T, M, N, E);
  PairParams p = {};
  p.grp.mode = 2; p.grp.E = E; p.grp.seg = seg;
  p.M = M; p.N = N; p.K = T;
  p.group_m = 1;
  p.epi.M = M; p.epi.N = N;
  p.epi.out_f32 = out_f32 ? 1 : 0;
  p.epi.accumulate = accumulate ? 1 : 0;
  p.epi.alpha = alpha;
  p.status = b200::status_ptr();
  if (BN == 192)
    return run_grouped<192>(a_q, sfa, b_q, sfb, d, p, M, N, (long long)E * M, lda, ldb, N, (cudaStream_t)stream,
                            "gemm_grouped_mx_wgrad");
  return run_grouped<128>(a_q, sfa, b_q, sfb, d, p, M, N, (long long)E * M, lda, ldb, N, (cudaStream_t)stream,
                          "gemm_grouped_mx_wgrad");
}

// bf16 rows: d[r, :] = a[r, :] op(b[e(r)])^T over a row buffer whose segments start at multiples of 256 rows.
// a [rows, K]; b [E, N, K] or, b_mn_major, [E, K, N] (then K must be a multiple of 64: an expert's contraction must not
// run into the next one's rows); d [rows, N] (pitch ldd elements); tile_expert [rows / 256] on the device.
B200_API int b200_gemm_grouped_pair_rows(const void* a, const void* b, void* d, const int* tile_expert, int rows, int N, int K,
                                         int E, long long lda, long long ldd, int b_mn_major, float alpha, void* stream) {
  if (rows <= 0 || rows % 256 != 0 || N <= 0 || K <= 0 || E <= 0 || (b_mn_major && K % 64 != 0))
    return b200::fail(832, "gemm_grouped_pair_rows: rows=%d (x256) N=%d K=%d (x64 when MN-major) E=%d", rows, N, K, E);
  CUtensorMap tmA, tmB, tmD, tmDt;
  int r;
  if ((r = b200::make_tmap_2d(&tmA, b200::DT_BF16, a, K, rows, lda * 2, 64, 128, b200::SWZ_128))) return r;
  if (!b_mn_major) r = b200::make_tmap_2d(&tmB, b200::DT_BF16, b, K, (uint64_t)E * N, (uint64_t)K * 2, 64, 128, b200::SWZ_128);
  else r = b200::make_tmap_2d(&tmB, b200::DT_BF16, b, N, (uint64_t)E * K, (uint64_t)N * 2, 64, 64, b200::SWZ_128);
  if (r) return r;
  if ((r = make_out_tmap<256>(&tmD, &tmDt, d, rows, N, ldd, 0))) return r;
  PairParams p = {};
  p.grp.mode = 1; p.grp.E = E; p.grp.tile_expert = tile_expert;
  p.M = rows; p.N = N; p.K = K;
  p.b_mn_major = b_mn_major ? 1 : 0;
  p.group_m = 16;
  p.epi.M = rows; p.epi.N = N; p.epi.alpha = alpha;
  p.status = b200::status_ptr();
  return launch_pair<KIND_BF16, 256, 1>(tmA, tmB, tmA, tmB, tmD, tmDt, p, (cudaStream_t)stream, "gemm_grouped_pair_rows");
}

// bf16 weight gradient: d[e] (+)= a[seg[e]:seg[e+1], :]^T b[seg[e]:seg[e+1], :]; a [rows, M], b [rows, N], d [E, M, N]
// contiguous, bf16 or fp32; segments are multiples of 256 rows, M of 32.  accumulate as above.  counts [E] or null: the contraction of
// expert e ends with its first counts[e] rows rounded up to 64 (the rows behind them are zero in a and b up to there).
B200_API int b200_gemm_grouped_pair_wgrad(const void* a, const void* b, void* d, const int* seg, const int* counts, int rows, int M, int N, int E,
                                          long long lda, long long ldb, int out_f32, int accumulate, float alpha, void* stream) {
  if (rows <= 0 || rows % 256 != 0 || M <= 0 || M % 32 != 0 || N <= 0 || E <= 0)
    return b200::fail(833, "gemm_grouped_pair_wgrad: rows=%d (x256) M=%d (x32) N=%d E=%d", rows, M, N, E);
  CUtensorMap tmA, tmB, tmD, tmDt;
  int r;
  if ((r = b200::make_tmap_2d(&tmA, b200::DT_BF16, a, M, rows, lda * 2, 64, 64, b200::SWZ_128))) return r;
  if ((r = b200::make_tmap_2d(&tmB, b200::DT_BF16, b, N, rows, ldb * 2, 64, 64, b200::SWZ_128))) return r;
  if ((r = make_out_tmap<256>(&tmD, &tmDt, d, E * M, N, N, out_f32))) return r;
  PairParams p = {};
  p.grp.mode = 2; p.grp.E = E; p.grp.seg = seg; p.grp.counts = counts;
  p.M = M; p.N = N; p.K = rows;
  p.a_mn_major = 1; p.b_mn_major = 1;
  p.group_m = 1;
  p.epi.M = M; p.epi.N = N; p.epi.alpha = alpha;
  p.epi.out_f32 = out_f32 ? 1 : 0; p.epi.accumulate = accumulate ? 1 : 0;
  p.status = b200::status_ptr();
  return launch_pair<KIND_BF16, 256, 1>(tmA, tmB, tmA, tmB, tmD, tmDt, p, (cudaStream_t)stream, "gemm_grouped_pair_wgrad");
}
