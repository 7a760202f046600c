// Launchers of the heavy kernel templates, each compiled in its own
// translation unit (oa_stats.cu, oa_gemm_simt.cu, oa_gemm_tc.cu).
#pragma once
#include "oa_common.cuh"

namespace oa {
struct StatsArgs;
struct LeanArgs;
struct SchurArgs;
cudaError_t oa_launch_snp_stats(int R, int LP, const StatsArgs& A, int grid, size_t smem, cudaStream_t st);
// spb: SNPs per CTA group, a power of two <= 8 / R; threads: 256 per CTA, or 512 with one SNP per group and
// R = 1, 2 or 4 (lean_threads_for); A.Afull: with the in-kernel projection (oa_lean_has_qx)
cudaError_t oa_launch_snp_lean(int R, int spb, const LeanArgs& A, int grid, int threads, size_t smem,
                               cudaStream_t st);
// resident CTAs of k_snp_lean per SM for this shared-memory size and thread count (0 on error)
int oa_lean_ctas_per_sm(int R, int spb, size_t smem, int ql, int threads, bool f64);
bool oa_lean_has_qx(int R, int spb, int ql, bool f64);
cudaError_t oa_launch_schur(int R, const SchurArgs& S, cudaStream_t st);
// pre-GEMM C[col * ldc + row] = sum_k X[row][k] B[col][k], col < c2 (BF16 hi / lo operands)
cudaError_t oa_launch_pre_tc(const __nv_bfloat16* Xhi, const __nv_bfloat16* Xlo, int xrows,
                             const __nv_bfloat16* Bhi, const __nv_bfloat16* Blo, int c2, int n_pad, float* C, int ldc,
                             int* err, cudaStream_t st);
// FP32-accurate product C[col * ldc + row] = rscale[row] * cscale[col] * sum_k X[row][k] B[col][k], col < cols,
// of FP16 hi / lo operands (held in 16-bit buffers): each K-block's tensor-core sum is added in FP32 registers
cudaError_t oa_launch_gemm_tcp(const __nv_bfloat16* Xhi, const __nv_bfloat16* Xlo, int xrows,
                               const __nv_bfloat16* Bhi, const __nv_bfloat16* Blo, int cols, int n_pad,
                               const float* rscale, const float* cscale, float* C, int ldc, int* err, cudaStream_t st);
// statistics of traits [j0, j0 + nt) from the stored product z (column 0 = trait j0)
cudaError_t oa_launch_test_stats(int R, const EpiArgs& E, const float* z, int ldz, int j0, int nt, cudaStream_t st);
// FP32 SIMT product with fused statistics, r = 1, 2 or 4 (zero-allocation entry point); NaN dosages -> colmean
cudaError_t oa_launch_gemm_simt(int R, const float* X, size_t ldx, int xrows, const float* Yt, size_t ldy, int t,
                                int K, const float* colmean, const int* has_nan, const EpiArgs& E, cudaStream_t st);
// variant: 1 = BK 32 x 4 stages, 2 = BK 64 x 2 stages, 3 = CTA pairs (2-SM MMA) BK 32 x 6, 4 = pairs BK 64 x 3;
// raster: 1 = trait tiles inner, 2 = SNP tiles inner
// Bound (ns of %globaltimer) of the pipeline waits of the tensor-core GEMMs and of the staging waits of the
// per-SNP statistics kernels on the current device (2 s by default); the drain waits keep 2 s
cudaError_t oa_set_wait_limit_tc(unsigned long long ns);
cudaError_t oa_set_wait_limit_stats(unsigned long long ns);
cudaError_t oa_launch_gemm_tc(int R, int variant, int raster, const __nv_bfloat16* Xhi, const __nv_bfloat16* Xlo,
                              int xrows, const __nv_bfloat16* Yhi, const __nv_bfloat16* Ylo, int t, int n_pad,
                              const EpiArgs& E, int* err, cudaStream_t st);
// Fused-operand forms: X read as FP32 (columns of ldx floats, n of them valid; ldx * 4 and X 16-byte aligned)
// and split into BF16 hi / lo in shared memory, each value taken as NaN -> fill, else x - shift, with
// shift = center ? colmean : 0 and fill = center ? 0 : colmean per row (fill only when *has_nan != 0).  oa_gemm_tc_fusable: the pipeline
// variant and trait count have a fused form (at most 128 traits, or CTA pairs); the pre-GEMM's fused form
// takes at most 128 columns.
bool oa_gemm_tc_fusable(int variant, int t);
cudaError_t oa_launch_gemm_tcf(int R, int raster, const float* X, size_t ldx, int n, int xrows, const float* colmean,
                               const int* has_nan, int center, const __nv_bfloat16* Yhi, const __nv_bfloat16* Ylo, int t, int n_pad,
                               const EpiArgs& E, int* err, cudaStream_t st);
cudaError_t oa_launch_pre_tcf(const float* X, size_t ldx, int n, int xrows, const float* colmean, const int* has_nan,
                              int center,
                              const __nv_bfloat16* Bhi, const __nv_bfloat16* Blo, int c2, int n_pad, float* C, int ldc,
                              int* err, cudaStream_t st);
}  // namespace oa
