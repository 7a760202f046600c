// Statistics of every SNP x trait test from a stored product z = X'Y~
// (k_gemm_tcp / k_gemm_tcp2, or the store form of k_gemm_tc): the arithmetic
// of the fused epilogues (oa_epilogue.cuh) in a kernel of its own.
//
// Lane = SNP, so that z (column j of the product holds trait j's z of
// consecutive SNPs), the Schur inverses and var_x are coalesced loads and no
// shuffle gathers a SNP's columns; a work item is 256 SNPs x 64 traits whose
// constants sit in shared memory.  z is read eight traits at a time before
// they are evaluated.  Bound by instruction issue (77 warp instructions per 32
// tests in full, most of them the FP64 residual sum; fewer where the FP32
// screening drops a warp's tests: 60 M tests 0.41 -> 0.23 ms): two CTAs of
// eight warps per SM keep the FP64 chain's latency covered within 128
// registers a thread.
#pragma once
#include "oa_epilogue.cuh"

namespace oa {

constexpr int TS_THREADS = 256;
constexpr int TS_TRAITS = 64;
constexpr int TS_COLS = 8;        // traits whose z is loaded together
// Record slots a warp reserves at a time.  Two CTAs of eight warps per SM: as
// many slots held back as the tensor-core epilogues' eight warps with EMIT_BLOCK.
constexpr int TS_CTAS_PER_SM = 2;
constexpr int TS_EMIT = EMIT_BLOCK * EPI_WARPS_TC / (TS_CTAS_PER_SM * (TS_THREADS / 32));

// FAST, SCREEN: as in epi_columns (oa_gemm_tc.cu).
template <int R, bool FAST, bool SCREEN>
__device__ __forceinline__ void test_stats_item(const EpiArgs& E, const float* __restrict__ z, int ldz, int j0, int jn,
                                                int i, bool live, const TraitP* tps, Emitter& em) {
    int cg = -1;            // pattern whose Schur inverse is cached
    bool csing = true;
    double S[R * R];
    float Sf[R * R];        // the same in FP32, for the screening
    float vx[R];
#pragma unroll
    for (int a = 0; a < R; ++a) vx[a] = live ? E.varx[(size_t)i * R + a] : 1.f;
    float v[TS_COLS][R], vn[TS_COLS][R];   // this and the next eight traits' z
    auto load = [&](int c0, float (&d)[TS_COLS][R]) {
#pragma unroll
        for (int q = 0; q < TS_COLS; ++q)
#pragma unroll
            for (int a = 0; a < R; ++a)
                d[q][a] = live && c0 + q < jn ? z[(size_t)(c0 + q) * ldz + (size_t)i * R + a] : 0.f;
    };
    load(0, v);
    for (int c0 = 0; c0 < jn; c0 += TS_COLS) {
        if (R <= 2) load(c0 + TS_COLS, vn);
#pragma unroll
        for (int q = 0; q < TS_COLS; ++q) {
            if (c0 + q >= jn) break;   // block-uniform
            const TraitP tp = tps[c0 + q];
            const int j = j0 + c0 + q;
            if (tp.g != cg) {          // traits are sorted by pattern: reloads are rare
                cg = tp.g;
                csing = live ? !load_schur<R>(E, cg, i, S) : true;
                if constexpr (SCREEN)
#pragma unroll
                    for (int a = 0; a < R * R; ++a) Sf[a] = csing ? 0.f : (float)S[a];
            }
            if constexpr (SCREEN)   // no lane can store a row: the usual case at high thresholds
                if (!__any_sync(0xffffffffu, live && (csing || !epi_screen<R>(E, v[q], tp, Sf, vx)))) continue;
            EpiTest<R> o;
            bool st = false;
            if (live) {
                if (csing) {
                    atomicAdd(E.n_singular, 1ull);
                    epi_dense_nan<R>(E, i, tp);
                } else {
                    st = epi_decide<R, FAST>(E, i, j, v[q], tp, S, vx, o);
                }
            }
            epi_emit_lazy<R>(E, st, em, [&](RecOf<R>* dst) { epi_write<R>(E, i, j, tp, o, dst); }, TS_EMIT);
        }
        if (R <= 2) {
#pragma unroll
            for (int q = 0; q < TS_COLS; ++q)
#pragma unroll
                for (int a = 0; a < R; ++a) v[q][a] = vn[q][a];
        } else {
            load(c0 + TS_COLS, v);
        }
    }
}

// Items with quirk terms, dense outputs or zero sets, out of line: their registers stay out of the
// usual case's.
template <int R>
__device__ __noinline__ void test_stats_rare(const EpiArgs& E, const float* __restrict__ z, int ldz, int j0, int jn,
                                             int i, bool live, const TraitP* tps, Emitter& em) {
    test_stats_item<R, false, false>(E, z, ldz, j0, jn, i, live, tps, em);
}

// Traits [j0, j0 + nt) of the block, seg (<= TS_TRAITS) of them per item; column 0 of z is trait j0's.
template <int R>
__global__ void __launch_bounds__(TS_THREADS, R <= 2 ? TS_CTAS_PER_SM : 1)
k_test_stats(EpiArgs E, const float* __restrict__ z, int ldz, int j0, int nt, int seg) {
    __shared__ TraitP tps[TS_TRAITS];
    const int sblocks = (E.mb + TS_THREADS - 1) / TS_THREADS, segs = (nt + seg - 1) / seg;
    Emitter em;
    for (int item = blockIdx.x; item < sblocks * segs; item += gridDim.x) {
        const int c0 = item / sblocks * seg, jn = min(seg, nt - c0);
        const int i = item % sblocks * TS_THREADS + (int)threadIdx.x;
        int zs = 0;
        if ((int)threadIdx.x < jn) {
            tps[threadIdx.x] = load_trait(E, j0 + c0 + threadIdx.x);
            zs = tps[threadIdx.x].zs >= 0;
        }
        const bool fast = !__syncthreads_or(zs) && !E.qK && !E.d_r2;
        const float* zc = z + (size_t)c0 * ldz;
        if (R <= 2 && fast && E.screen_t2 > 0.f)
            test_stats_item<R, true, true>(E, zc, ldz, j0 + c0, jn, i, i < E.mb, tps, em);
        else if (R <= 2 && fast)
            test_stats_item<R, true, false>(E, zc, ldz, j0 + c0, jn, i, i < E.mb, tps, em);
        else
            test_stats_rare<R>(E, zc, ldz, j0 + c0, jn, i, i < E.mb, tps, em);
        __syncthreads();   // the trait constants are read before the next item's replace them
    }
    epi_retire<R>(E, em);
}

}  // namespace oa
