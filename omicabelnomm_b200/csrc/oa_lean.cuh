// Per-SNP column statistics without covariates (k_snp_lean) and the FP64
// Schur kernel (k_schur) that combines them with the pre-GEMM output.
//
// The per-SNP quantities of the reference's corrected systems
// (Str/Sbr and their missing-row downdates, src/Algorithm.cpp:633-689,
// 1260-1315) split into
//   * X'X (r x r) over all rows and over each row set (missingness pattern
//     or zero set): k_snp_lean, from the SNP columns staged in shared memory
//     (x-only gathers, no covariate loads);
//   * Q'X and (Q o m_s)'X for every row set s: a GEMM of the SNP block with
//     the column matrix B2 = [Q | Q o m_1 | ... | Q o m_S] ("pre-GEMM", on
//     the tensor cores, in one launch with the traits where their product is
//     stored as well);
// and k_schur forms, per (pattern, SNP), the FP64 Schur complement
//     (D - D_g) - (A - A_g)' W_g (A - A_g)
// and its inverse, plus var_x from the all-rows complement D - A'A.
#pragma once
#include <type_traits>

#include "oa_stats.cuh"

namespace oa {

struct LeanArgs {
    const float* X;       // SNP block, column c at X + c*ldx
    size_t ldx;
    int padded;           // columns are 16-byte aligned and zero from row n to the next multiple of 4
    const int* xrows;     // row k of a column is X[c*ldx + xrows[k]] (a row subset), or null: X[c*ldx + k]
    int n, n_pad, mb;
    int nsets;
    const uint4* item_rows;   // rows of the sets in blocks of LEAN_BLOCK_ROWS 16-bit values (k_item_rows)
    const int2* items;        // work items, each within one set: {first block, rows}
    const int* set_item_off;  // items of set s: [set_item_off[s], set_item_off[s+1])
    const int* pass_off;      // passes over sets [pass_off[p], pass_off[p+1]) whose items fit in shared memory
    int npass;
    int items_cap;
    float* mean;          // [mb*r] column means if center, else imputation means (0 if the column had no NaN)
    int* has_nan;
    double* D;            // [mb][r*r] X'X over all rows
    float* Dset;          // [nsets][mb][r*r] X'X over each row set
    __nv_bfloat16* Xhi;   // [mb*r][n_pad] (tensor-core form) or null
    __nv_bfloat16* Xlo;
    int write_split;
    float* xscale;        // FP16 split of the columns times a power of two, 1 / scale here ([mb*r]); null: BF16 split
    __nv_bfloat16* Bhi;   // with xscale and the f64 kernels: a BF16 split as well (the mixed form's main product), or null
    __nv_bfloat16* Blo;
    int center;           // take each column relative to its mean (valid when XL holds an intercept)
    int* err;
    // all-rows covariate projection A = Q'(x - shift) of every column, summed here (short FP32
    // partial sums, FP64 across warps) instead of taken from the pre-GEMM, or null: where the
    // all-rows Schur complement D - A'A (var_x) and the pattern systems cancel a large part of D
    // (two or more columns per SNP; a SNP column near a covariate), the pre-GEMM's sums of A are
    // the largest error of the statistics (the qx kernels, l <= ql)
    const float4* Qb;     // [n_pad / 4][l] the orthonormal covariate basis (FP32) by blocks of four
                          // rows: Qb[k4 * l + q] = rows 4 k4 .. 4 k4 + 3 of covariate q (0 past n)
    int l, ql;            // covariates, and the slots for them: 4, 8 or 16
    int f64;              // the qx kernels' sums are FP64 from the thread's partial sum on
    const double* qsum;   // [l] column sums of the basis (FP64)
    double* Afull;        // [mb*R][ql]: A of column c, covariate q at Afull[c * ql + q]
};

// Threads per CTA (the template's NT): 256; groups of one SNP may also run 512 (launched where
// its columns fill so much shared memory that few CTAs fit on an SM).  Shared scratch is sized
// for 512.
constexpr int LEAN_MAX_THREADS = 512;
constexpr int LEAN_MAX_WARPS = LEAN_MAX_THREADS / 32;
constexpr int LEAN_BLOCK_ROWS = 256;    // rows of a set per index block (one 16-byte load of eight rows per lane)
constexpr int LEAN_STAGE_U = 8;         // elements per thread and step of the element-wise staging
constexpr int LEAN_QX_SUMS = 32;        // slots of the in-kernel projection: columns per group x 4, 8 or 16 covariates
constexpr int LEAN_COL_PAD = 8;         // floats after a staged column: its offset (0..3) and the pad row

// Shared memory of k_snp_lean: the group's columns (stride n_pad + LEAN_COL_PAD floats) | per-item
// partial sums | reduction scratch.
__host__ __device__ inline size_t lean_smem_bytes(int R, int n_pad, int spb, int items_cap, int ql = 0) {
    const int NC = spb * R, NU = spb * R * (R + 1) / 2;
    const int NQ = NC + NU + NC * ql;   // NU >= NC: also the NaN path's 2 NC sums
    return (size_t)NC * (n_pad + LEAN_COL_PAD) * 4 + (size_t)items_cap * NU * 4 +
           (size_t)(LEAN_MAX_WARPS + 1) * NQ * 8 + 64;
}

// Threads per CTA, from the columns' length alone (so that every tuning sums in the same order and gives the
// same bits): 512 where a SNP's columns leave an SM at most three CTAs (one column: n >= 16,384) or, with
// two or four, two; the plan then keeps one SNP per group.  Else 256: more, smaller CTAs per SM with
// cheaper block barriers.  (Statistics stage with 256 / 512 threads, two columns: 20,000 SNPs at
// n = 12,545 1.67 / 1.38 ms, n = 10,001 1.01 / 0.90, n = 9,500 0.97 / 0.98; 10,000 at n = 14,411 with 85 sets
// of 1,441 rows 4.98 / 3.97.)
inline int lean_threads_for(int R, int n_pad) {
    const size_t col = (size_t)n_pad * 4;
    const bool longc = R == 1 ? col >= 64 * 1024 : (R <= 4 && R * col >= 75 * 1024);
    return longc ? LEAN_MAX_THREADS : 256;
}

// SNPs per group where the caller asks for none (a power of two): at most four columns, as far as they fit
// the group's bytes and leave at least two groups per SM.  With one column per SNP two SNPs are worth going
// down to three CTAs per SM, four to five (50,000 SNPs, statistics stage with 1 / 2 / 4 / 8 SNPs per group:
// n = 1,000 0.29 / 0.18 / 0.16 / 0.19 ms, n = 2,000 0.33 / 0.21 / 0.20 / 0.26, n = 3,500 0.39 / 0.27 / 0.29 /
// 0.34, n = 7,000 0.65 / 0.62 / - / -, n = 10,000 1.37 / 1.46 / - / -);
// with two, the covariate basis read once per group is worth two CTAs (20,000 SNPs, n = 6,000 1.27 / 1.23).
inline int lean_auto_spb(int R, int n_pad, int ql, int snps, int sms) {
    int s = 1;
    for (;;) {
        const size_t bytes = (R > 1 ? 100 : (s == 1 ? 60 : 40)) * 1024;
        if (s * 2 * R > 4 || lean_smem_bytes(R, n_pad, s * 2, 0, ql) > bytes || snps / (s * 2) < 2 * sms) break;
        s *= 2;
    }
    return s;
}

// Rows per work item of the set pass: one block of a set where that gives the eight warps few items,
// else up to four (each item ends in a shuffle reduction, which with 150 sets of 600 rows took more of
// the shared-memory pipe than the rows themselves).
constexpr int LEAN_ITEMS_ENOUGH = 128;
inline int lean_item_rows(long long blocks) {
    return LEAN_BLOCK_ROWS * (blocks > 2 * LEAN_ITEMS_ENOUGH ? 4 : (blocks > LEAN_ITEMS_ENOUGH ? 2 : 1));
}

// The rows of every set in the order the set pass reads them, in blocks of LEAN_BLOCK_ROWS: lane l of
// step u of a block takes slot l * 8 + u (one 16-byte load of a lane covers its eight steps); slots past
// the end of a set hold the pad row n_pad.  A set's rows are taken by their rank among its rows of the same
// shared-memory bank (row % 32), then by bank, so that the 32 rows of a step fall into (nearly) as many
// banks: in ascending order random rows of a set gave 3.4 wavefronts per load, and the statistics
// kernel's shared-memory pipe was at 80 %.  One CTA of 32 warps per set, warp = bank.
static __global__ void __launch_bounds__(1024)
k_item_rows(const int* __restrict__ rows, const int* __restrict__ set_off, const int* __restrict__ set_blk_off,
            int n_pad, uint16_t* __restrict__ item_rows) {
    __shared__ int cnt[32];
    const int s = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int r0 = set_off[s], r1 = set_off[s + 1];
    uint16_t* out = item_rows + (size_t)set_blk_off[s] * LEAN_BLOCK_ROWS;
    const int slots = (set_blk_off[s + 1] - set_blk_off[s]) * LEAN_BLOCK_ROWS;
    for (int q = threadIdx.x; q < slots; q += blockDim.x) out[q] = (uint16_t)n_pad;
    int c = 0;
    for (int k0 = r0; k0 < r1; k0 += 32) {
        const int row = k0 + lane < r1 ? rows[k0 + lane] : -1;
        c += __popc(__ballot_sync(0xffffffffu, row >= 0 && row % 32 == w));
    }
    if (lane == 0) cnt[w] = c;
    __syncthreads();   // counts, and the pad rows are in place
    const int mine = cnt[lane];   // rows of bank `lane`
    int rank = 0;
    for (int k0 = r0; k0 < r1; k0 += 32) {
        const int row = k0 + lane < r1 ? rows[k0 + lane] : -1;
        unsigned m = __ballot_sync(0xffffffffu, row >= 0 && row % 32 == w);
        for (; m; m &= m - 1, ++rank) {
            const int r = __shfl_sync(0xffffffffu, row, __ffs(m) - 1);
            // rows of lower rank in every bank, then those of this rank in lower banks
            const int pos = __reduce_add_sync(0xffffffffu, min(mine, rank)) +
                            __popc(__ballot_sync(0xffffffffu, mine > rank) & ((1u << w) - 1u));
            if (lane == 0)
                out[pos / LEAN_BLOCK_ROWS * LEAN_BLOCK_ROWS + pos % 32 * 8 + pos % LEAN_BLOCK_ROWS / 32] = (uint16_t)r;
        }
    }
}

// Warp sums of the NV values of v: store(q, sum) is called for every q by one lane.  The lanes
// halve the values between them while they halve the distance (31 shuffles for 32 values where
// one butterfly per value takes 160), with the pairs, and so the bits, of a butterfly per value.
template <int NV, class Store>
__device__ __forceinline__ void warp_sums(const float (&v)[NV], Store&& store) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int base = 0; base < NV; base += 32) {
        constexpr int REST = NV % 32 == 0 ? 32 : NV % 32;
        const int cnt = NV - base >= 32 ? 32 : REST;           // values of this round (compile time)
        constexpr int PMAX = NV >= 32 ? 32 : (NV > 16 ? 32 : (NV > 8 ? 16 : (NV > 4 ? 8 : (NV > 2 ? 4 : NV))));
        float x[PMAX];
#pragma unroll
        for (int i = 0; i < PMAX; ++i) x[i] = i < cnt ? v[base + i < NV ? base + i : 0] : 0.f;
        int m = PMAX, idx = 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            if (m > 1) {
                const bool up = (lane & o) != 0;
                m /= 2;
#pragma unroll
                for (int i = 0; i < PMAX / 2; ++i)
                    if (i < m) {
                        const float keep = up ? x[i + m] : x[i], send = up ? x[i] : x[i + m];
                        x[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                idx += up ? m : 0;
            } else {
                x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
            }
        }
        if ((lane & (32 / PMAX - 1)) == 0 && idx < cnt) store(base + idx, x[0]);
    }
}

// The same in FP64, eight values at a time (18 shuffles where one butterfly per value takes 80).
template <int NV, class Store>
__device__ __forceinline__ void warp_sums_f64(const float (&v)[NV], Store&& store) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int base = 0; base < NV; base += 8) {
        double x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = base + i < NV ? (double)v[base + i < NV ? base + i : 0] : 0.0;
        int idx = 0;
#pragma unroll
        for (int m = 4, o = 16; m > 0; m /= 2, o /= 2) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < m) {
                    const double keep = up ? x[i + m] : x[i], send = up ? x[i] : x[i + m];
                    x[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            idx += up ? m : 0;
        }
        x[0] += __shfl_xor_sync(0xffffffffu, x[0], 2);
        x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
        if ((lane & 3) == 0 && base + idx < NV) store(base + idx, x[0]);
    }
}

// Block-wide sum of NV floats per thread over NW warps: FP32 (F64: FP64) within a warp, FP64 across
// warps (in warp order; the values are spread over the warps); the first NB sums are copied to out[] on
// every thread, all NV stay at red + LEAN_MAX_WARPS * NV until red is reused.
template <int NW, int NV, int NB = NV, bool F64 = false>
__device__ __forceinline__ void block_sum_fd(float (&v)[NV], double (&out)[NB], double* red /* [warps + 1][NV] */) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if constexpr (F64)
        warp_sums_f64<NV>(v, [&](int q, double sum) { red[w * NV + q] = sum; });
    else
        warp_sums<NV>(v, [&](int q, float sum) { red[w * NV + q] = (double)sum; });
    __syncthreads();
    double* bc = red + LEAN_MAX_WARPS * NV;
    constexpr int PER = 32 / NW;   // values a warp adds up at once, NW lanes each
    for (int q0 = w * PER; q0 < NV; q0 += NW * PER) {
        const int q = q0 + lane / NW;
        double s = q < NV ? red[lane % NW * NV + q] : 0.0;
#pragma unroll
        for (int o = NW / 2; o > 0; o /= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane % NW == 0 && q < NV) bc[q] = s;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NB; ++q) out[q] = bc[q];
}

// Index of the pair (a, b), a <= b, among a SNP's R (R + 1) / 2 column pairs.
template <int R>
__host__ __device__ constexpr int lean_pair(int a, int b) {
    return a * R - a * (a - 1) / 2 + (b - a);
}

// A column whose sum of squares `raw` is 8 times that of the centred column or more (1 + mean^2 / variance): the
// difference of the raw FP32 sums keeps 2^-24 times this ratio of the centred one.  Dosages of the minor
// allele stay below 3; an expression level of 8 +- 2 has 17, one of 12 +- 0.05 57,601 (n = 1,000, beta's
// error from the raw sums 1.8e-3, from the moved column's 1.6e-7).
__device__ __forceinline__ bool lean_narrow(float raw, float mean, int n) {
    return 8.f * (float)n * mean * mean > 7.f * raw;
}

// Moves the narrow columns of a group to their means in place (moved[c]: what was taken off, untouched
// elsewhere) and sums their SNPs again in FP64, into the block's sums (bc: column sums, cross products,
// Q'x with l covariates, Qb); offs: two bits of offset per column.  A constant column becomes exact zeros,
// whatever its mean was rounded to.  Called by the whole block, out of line: rare, and its code and
// registers stay out of the usual case's.
template <int R, int NC, int QL>
__device__ __noinline__ void lean_recentre(float* cols, int cs, unsigned offs, int n, int ncol, double* red, double* bc,
                                           float* moved, const float4* Qb, int l) {
    constexpr int NP = R * (R + 1) / 2, NU = NC / R * NP;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    auto column = [&](int c) { return cols + (size_t)c * cs + (offs >> (2 * c) & 3u); };
    auto block_total = [&](double v, double* out) {
        v = warp_sum(v);
        if (lane == 0) red[w] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += red[q];
            *out = s;
        }
        __syncthreads();
    };
    __syncthreads();   // the columns are swept, the sums read
#pragma unroll 1
    for (int i = 0; i < ncol; i += R) {
        int narrow = 0;
#pragma unroll
        for (int a = 0; a < R; ++a) {
            const float mean = (float)(bc[i + a] / (double)n);
            if (lean_narrow((float)bc[NC + i / R * NP + lean_pair<R>(a, a)], mean, n)) narrow |= 1 << a;
        }
        if (!narrow) continue;   // block-uniform
#pragma unroll 1
        for (int a = 0; a < R; ++a) {
            if (!(narrow >> a & 1)) continue;
            float* col = column(i + a);
            const float first = col[0], mean = (float)(bc[i + a] / (double)n);
            int differs = 0;
            for (int k = threadIdx.x; k < n; k += blockDim.x) differs |= col[k] != first;
            const float shift = __syncthreads_or(differs) ? mean : first;
            for (int k = threadIdx.x; k < n; k += blockDim.x) col[k] -= shift;
            if (threadIdx.x == 0) moved[i + a] = shift;
        }
        __syncthreads();
#pragma unroll 1
        for (int a = 0; a < R; ++a) {
            const float* xa = column(i + a);
#pragma unroll 1
            for (int b = a; b < R; ++b) {
                if (!(narrow >> a & 1) && !(narrow >> b & 1)) continue;
                const float* xb = column(i + b);
                double sum = 0.0, prod = 0.0;
                for (int k = threadIdx.x; k < n; k += blockDim.x) {
                    sum += (double)xa[k];
                    prod += (double)xa[k] * (double)xb[k];
                }
                if (b == a) block_total(sum, bc + i + a);
                block_total(prod, bc + NC + i / R * NP + lean_pair<R>(a, b));
            }
            if (QL && (narrow >> a & 1))
#pragma unroll 1
                for (int q = 0; q < l; ++q) {
                    double dot = 0.0;
                    for (int k = threadIdx.x; k < n; k += blockDim.x)
                        dot += (double)reinterpret_cast<const float*>(Qb + (size_t)(k / 4) * l + q)[k % 4] * (double)xa[k];
                    block_total(dot, bc + NC + NU + (i + a) * QL + q);
                }
        }
    }
}

// Resident CTAs the register allocation leaves room for: 64 registers a thread for groups of one or two
// columns or of four SNPs, 48 for two SNPs and 40 for a gathered one (where shared memory holds five and
// six CTAs of 256 threads), else 128.
// The projection's partial sums take their own registers.
constexpr int lean_min_ctas(int R, int SPB, bool gather, int NT, int QL) {
    if (R == 1 && QL > 0) return SPB * QL <= 16 && QL < 16 ? 1024 / NT : 512 / NT;
    if (R == 1 && SPB == 2) return 5;
    if (R == 1 && SPB == 1 && gather) return 1536 / NT;
    return R * SPB <= 2 || (R == 1 && SPB == 4) ? 1024 / NT : 512 / NT;
}

// One CTA handles SPB SNPs (SPB*R columns) per group in a persistent loop over groups:
//   staging the group's columns stream into shared memory by TMA bulk copies.  A column that does not
//           start on a 16-byte boundary (any n that is no multiple of 4) is copied from the boundary
//           below it to the one above its end and read at its offset o; the block's first and last
//           columns, whose boundaries may lie outside the block, are then copied element by element.
//           A row subset of a resident matrix (GATHER) is gathered by 4-byte cp.async copies.
//   pass 1  column sums and raw cross products from float4 reads of the
//           staged columns, one block reduction (FP64 across warps); NaN
//           propagates, so a column whose sum is NaN is counted and
//           mean-imputed in place (src/Utility.cpp:302-326) and the sweep
//           repeated - rare, dosage files seldom hold NaN.  With an
//           intercept among the covariates every later sum uses x - mean
//           (the Schur complements, X'y~ and var_x do not change; the sums
//           lose their large common part); X'X of the shifted columns
//           follows from the raw sums in FP64, and where that difference
//           would cancel (lean_narrow) the column is moved to its mean in
//           place and summed again first
//   pass 2  16-bit hi/lo split of the shifted columns
//   pass 3  X'X over each row set: work items of up to four index blocks of one set
//           (fixed per trait block) go round-robin to the warps; a warp's item
//           sum (eight row indices per 16-byte load, gathers that seldom share
//           a bank, shuffle reduction) lands in its own shared-memory slot, and
//           a set's sum adds its items in order.  No atomics: the sums are
//           bit-reproducible.
// One column buffer and as many CTAs per SM as fit: the other CTAs cover a group's copy and its block
// barriers better than a second buffer did (50,000 SNPs, statistics stage with two buffers / one:
// n = 12,348 with 3 row sets 0.94 / 0.79 ms, n = 4,834 and two columns 2.97 / 1.42 ms).  Bound by HBM
// where the row sets are few (n = 12,347: 5.9 TB/s of columns read and split written, 0.90 of a copy's
// rate); with 20 sets of 500 rows the set pass takes the shared-memory pipe to 0.6 and it runs at
// 4.8 TB/s (n = 10,000).  Unaligned columns: 0.86 ms where 4-byte copies took 1.27 (n = 12,347).
// QL: covariate slots of the in-kernel projection (0: none); F64: LeanArgs.f64.
template <int R, int SPB, bool GATHER, int QL = 0, int NT = 256, bool F64 = false>
__global__ void __launch_bounds__(NT, lean_min_ctas(R, SPB, GATHER, NT, QL))
k_snp_lean(LeanArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int NC = SPB * R;                 // columns per group
    constexpr int NP = R * (R + 1) / 2;         // column pairs per SNP
    constexpr int NU = SPB * NP;                // X'X entries per group
    constexpr int NWARP = NT / 32;
    const int n = A.n, cs = A.n_pad + LEAN_COL_PAD;
    float* cols = reinterpret_cast<float*>(smem_raw);                                    // [NC][cs]
    float* part = cols + (size_t)NC * cs;                                                // [items_cap][NU]
    double* red = reinterpret_cast<double*>(
        (reinterpret_cast<uintptr_t>(part + (size_t)A.items_cap * NU) + 7) & ~(uintptr_t)7);   // [LEAN_MAX_WARPS + 1][NQ]
    __shared__ __align__(8) uint64_t mbar;
    __shared__ int stop;
    __shared__ float moved[NC];                 // taken off the staged column (lean_recentre)
    const int ngroups = (A.mb + SPB - 1) / SPB;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // some column starts or ends off a 16-byte boundary: copies write past column ends
    const bool ragged = !GATHER && !A.padded &&
                        (((n | (int)(A.ldx & 3)) & 3) != 0 || (reinterpret_cast<uintptr_t>(A.X) & 15) != 0);

    // Offset (floats) of column c of the block below its first element, and whether the 16-byte
    // boundaries around it may lie outside the block.
    auto col_off = [&](int c) { return (int)((reinterpret_cast<uintptr_t>(A.X + (size_t)c * A.ldx) >> 2) & 3); };
    auto col_edge = [&](int c) {
        const int o = col_off(c);
        return !A.padded && ((c == 0 && o != 0) || (c == A.mb * R - 1 && ((o + n) & 3) != 0));
    };
    // thread 0: bulk copies of a group's columns
    auto issue = [&](int g) {
        const int c0 = g * SPB * R, ncol = min(SPB, A.mb - g * SPB) * R;
        uint32_t total = 0;
        for (int c = 0; c < ncol; ++c)
            if (!col_edge(c0 + c)) total += ((uint32_t)(col_off(c0 + c) + n) * 4u + 15u) & ~15u;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(st_su32(&mbar)), "r"(total)
                     : "memory");
        for (int c = 0; c < ncol; ++c) {
            if (col_edge(c0 + c)) continue;
            const int o = col_off(c0 + c);
            const float* src = A.X + (size_t)(c0 + c) * A.ldx - o;
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    st_su32(cols + (size_t)c * cs)),
                "l"(reinterpret_cast<uint64_t>(src)), "r"(((uint32_t)(o + n) * 4u + 15u) & ~15u), "r"(st_su32(&mbar))
                : "memory");
        }
    };
    // GATHER: 4-byte cp.async copies of the subset's rows, one commit group per group of columns and thread
    auto stage = [&](int g) {
        const int i0 = g * SPB;
        const int ncol = min(SPB, A.mb - i0) * R;
        for (int c = 0; c < ncol; ++c) {
            const float* src = A.X + (size_t)(i0 * R + c) * A.ldx;
            const uint32_t dst = st_su32(cols + (size_t)c * cs);
            // LEAN_STAGE_U elements per thread and step: the row indices of a step
            // are loaded together, so their latencies overlap
            for (int k0 = threadIdx.x; k0 < n; k0 += LEAN_STAGE_U * NT) {
                int kk[LEAN_STAGE_U];
#pragma unroll
                for (int u = 0; u < LEAN_STAGE_U; ++u) {
                    const int k = k0 + u * NT;
                    kk[u] = k < n ? __ldg(A.xrows + k) : -1;
                }
#pragma unroll
                for (int u = 0; u < LEAN_STAGE_U; ++u)
                    if (kk[u] >= 0)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                                         dst + 4u * (uint32_t)(k0 + u * NT)),
                                     "l"(src + kk[u])
                                     : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (GATHER && (int)blockIdx.x < ngroups) stage(blockIdx.x);

    // zero the column tails once: aligned copies and gathers write only [0, n)
    for (int q = threadIdx.x; q < NC * (cs - n); q += NT) cols[(size_t)(q / (cs - n)) * cs + n + q % (cs - n)] = 0.f;
    if (threadIdx.x == 0) {
        stop = 0;
        if (!GATHER) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(st_su32(&mbar)));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    if (!GATHER) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // own writes to the columns
    __syncthreads();
    if (!GATHER && threadIdx.x == 0 && (int)blockIdx.x < ngroups) issue(blockIdx.x);

    uint32_t par = 0;
    for (int g = blockIdx.x; g < ngroups; g += gridDim.x, par ^= 1u) {
        const int gn = g + gridDim.x;
        const int i0 = g * SPB;
        const int nsnp = min(SPB, A.mb - i0);
        const int ncol = nsnp * R;
        int off[NC];                           // offset of the column in its buffer
#pragma unroll
        for (int c = 0; c < NC; ++c)
            off[c] = ragged && c < ncol && !col_edge(i0 * R + c) ? col_off(i0 * R + c) : 0;

        if (GATHER) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        } else {
            if (ragged)
                for (int c = 0; c < ncol; ++c)
                    if (col_edge(i0 * R + c))
                        for (int k = threadIdx.x; k < n; k += NT)
                            cols[(size_t)c * cs + k] = __ldg(A.X + (size_t)(i0 * R + c) * A.ldx + k);
            if (w == 0) {
                int ok = 1;
                if (lane == 0 && !st_mbar_wait(&mbar, par)) {
                    stop = 1;
                    atomicExch(A.err, 1);
                    ok = 0;
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (ragged && ok) {   // the copies wrote up to three floats past each column
                    st_mbar_try(&mbar, par);
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        for (int k = n + lane; k < A.n_pad; k += 32) cols[(size_t)c * cs + off[c] + k] = 0.f;
                }
            }
        }
        __syncthreads();
        if (stop) break;
        if (!GATHER) st_mbar_try(&mbar, par);

        // Four consecutive rows of column c.  O: the offset of every column where it is known (0, or
        // 1..3 of a single column), -1: off[c]
        auto ld4 = [&](auto O, int c, int k4) -> float4 {
            const float4* p = reinterpret_cast<const float4*>(cols + (size_t)c * cs) + k4;
            const float4 x = p[0];
            const int o = decltype(O)::value >= 0 ? decltype(O)::value : off[c];
            if (o == 0) return x;
            const float4 y = p[1];
            if (o == 1) return make_float4(x.y, x.z, x.w, y.x);
            if (o == 2) return make_float4(x.z, x.w, y.x, y.y);
            return make_float4(x.w, y.x, y.y, y.z);
        };
        auto by_offset = [&](auto&& f) {
            if constexpr (GATHER) {
                f(std::integral_constant<int, 0>{});
            } else if constexpr (NC == 1) {
                switch (off[0]) {
                    case 0: f(std::integral_constant<int, 0>{}); break;
                    case 1: f(std::integral_constant<int, 1>{}); break;
                    case 2: f(std::integral_constant<int, 2>{}); break;
                    default: f(std::integral_constant<int, 3>{}); break;
                }
            } else {
                if (ragged) f(std::integral_constant<int, -1>{});
                else f(std::integral_constant<int, 0>{});
            }
        };

        // ---- pass 1: column sums and raw cross products in one sweep (the
        // zero tail adds nothing); NaN propagates, so a column whose sum is
        // NaN is counted and mean-imputed in place (src/Utility.cpp:302-326)
        // and the sweep is repeated - rare, dosage files seldom hold NaN
        float sh[NC];                          // subtracted from every value (centring), 0 without
        float hs[NC];                          // scale of the FP16 split
        {
            constexpr int NQX = NC * QL;
            constexpr int NV = NC + NU + NQX;  // [column sums | cross products | Q'x of the raw columns]
            constexpr int NB = NC + NU;        // sums every thread keeps (Q'x stays in shared memory)
            static_assert(NQX <= LEAN_QX_SUMS, "slots of the qx kernels");
            double tot[NB];
            const double* qxs = red + LEAN_MAX_WARPS * NV + NB;   // the block's Q'x sums after the last sweep
            bool cnan[NC];
            float cmean[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) cnan[c] = false;
            if ((int)threadIdx.x < NC) moved[threadIdx.x] = 0.f;   // before the sums' barriers
            for (int round = 0;; ++round) {
                float acc[NV];
#pragma unroll
                for (int u = 0; u < NV; ++u) acc[u] = 0.f;
                by_offset([&](auto O) {
                    for (int k4 = threadIdx.x; k4 < A.n_pad / 4; k4 += NT) {
                        float4 v[NC];
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            v[c] = c < ncol ? ld4(O, c, k4) : make_float4(0.f, 0.f, 0.f, 0.f);
                            acc[c] += (v[c].x + v[c].y) + (v[c].z + v[c].w);
                        }
                        if constexpr (QL > 0) {
                            // rows 4 k4 .. 4 k4 + 3 of each covariate: one 16-byte load per covariate
#pragma unroll
                            for (int qq = 0; qq < QL; ++qq) {
                                if (qq < A.l) {
                                    const float4 q4 = __ldg(A.Qb + (size_t)k4 * A.l + qq);
#pragma unroll
                                    for (int c = 0; c < NC; ++c) {
                                        float& a = acc[NC + NU + c * QL + qq];
                                        a = fmaf(q4.x, v[c].x, a);
                                        a = fmaf(q4.y, v[c].y, a);
                                        a = fmaf(q4.z, v[c].z, a);
                                        a = fmaf(q4.w, v[c].w, a);
                                    }
                                }
                            }
                        }
#pragma unroll
                        for (int s2 = 0; s2 < SPB; ++s2)
#pragma unroll
                            for (int a = 0; a < R; ++a)
#pragma unroll
                                for (int bb = a; bb < R; ++bb) {
                                    const float4 xa = v[s2 * R + a], xb = v[s2 * R + bb];
                                    float& d = acc[NC + s2 * NP + lean_pair<R>(a, bb)];
                                    d = fmaf(xa.x, xb.x, d);
                                    d = fmaf(xa.y, xb.y, d);
                                    d = fmaf(xa.z, xb.z, d);
                                    d = fmaf(xa.w, xb.w, d);
                                }
                    }
                });
                block_sum_fd<NWARP, NV, NB, F64>(acc, tot, red);
                if (round == 1) break;
                bool any_nan = false;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    cnan[c] = (c < ncol) && isnan(tot[c]);
                    any_nan |= cnan[c];
                    cmean[c] = (float)(tot[c] / (double)n);
                }
                if (!any_nan) break;
                // block-uniform: count and sum the observed values, impute in place
                __syncthreads();   // every thread has read the sums before the scratch is reused
                float ns[2 * NC];
                double ct[2 * NC];
#pragma unroll
                for (int u = 0; u < 2 * NC; ++u) ns[u] = 0.f;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (cnan[c]) {
                        const float* col = cols + (size_t)c * cs + off[c];
                        for (int k = threadIdx.x; k < n; k += NT) {
                            const float v = col[k];
                            if (isnan(v)) ns[NC + c] += 1.f;
                            else ns[c] += v;
                        }
                    }
                }
                block_sum_fd<NWARP, 2 * NC>(ns, ct, red);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (cnan[c]) {
                        cmean[c] = (float)(ct[c] / ((double)n - ct[NC + c]));
                        float* col = cols + (size_t)c * cs + off[c];
                        for (int k = threadIdx.x; k < n; k += NT)
                            if (isnan(col[k])) col[k] = cmean[c];
                    }
                }
                __syncthreads();
            }
            if (A.center) {
                bool narrow = false;
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    narrow |= c < ncol && lean_narrow((float)tot[NC + c / R * NP + lean_pair<R>(c % R, c % R)], cmean[c], n);
                if (narrow) {   // block-uniform
                    unsigned offs = 0;
#pragma unroll
                    for (int c = 0; c < NC; ++c) offs |= (unsigned)off[c] << (2 * c);
                    double* bc = red + LEAN_MAX_WARPS * NV;
                    lean_recentre<R, NC, QL>(cols, cs, offs, n, ncol, red, bc, moved, A.Qb, A.l);
#pragma unroll
                    for (int u = 0; u < NB; ++u) tot[u] = bc[u];
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        if (moved[c] != 0.f) cmean[c] = (float)(tot[c] / (double)n);
                }
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                sh[c] = A.center ? cmean[c] : 0.f;
                hs[c] = 1.f;
            }
            if (A.xscale) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    // sum of squares of the shifted column; the second term keeps it an upper bound
                    // where the FP32 sums cancel (a column that is constant but for its last digits)
                    const double raw = tot[NC + c / R * NP + lean_pair<R>(c % R, c % R)], s0 = sh[c];
                    const double d = raw - 2.0 * s0 * tot[c] + (double)n * s0 * s0;
                    float inv = 1.f;
                    hs[c] = half_scale(fmax(d, 0.0) + raw * 0x1p-18, &inv);
                    if (threadIdx.x == 0 && c < ncol) A.xscale[i0 * R + c] = inv;
                }
            }
            if constexpr (QL > 0) {
                // A = Q'(x - shift) = Q'x - shift * (column sums of Q), in FP64; thread u writes entry u
                // (compile-time register indices)
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    if ((int)threadIdx.x / QL == c && c < ncol) {
                        const int qq = threadIdx.x % QL;
                        A.Afull[(size_t)(i0 * R + c) * QL + qq] =
                            qq < A.l ? qxs[c * QL + qq] - (double)sh[c] * A.qsum[qq] : 0.0;
                    }
            }
            if (threadIdx.x == 0) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (c < ncol) {
                        A.mean[i0 * R + c] = A.center ? moved[c] + cmean[c] : (cnan[c] ? cmean[c] : 0.f);
                        if (cnan[c]) atomicOr(A.has_nan, 1);
                    }
                }
            }
            // X'X of the columns taken relative to sh over the n rows, pairs spread over the warps:
            // sum x_a x_b - s_a sum x_b - s_b sum x_a + n s_a s_b
#pragma unroll
            for (int s2 = 0; s2 < SPB; ++s2)
#pragma unroll
                for (int a = 0; a < R; ++a)
#pragma unroll
                    for (int bb = a; bb < R; ++bb) {
                        const int ca = s2 * R + a, cb = s2 * R + bb, u = s2 * NP + lean_pair<R>(a, bb);
                        if (lane == 0 && w == u % NWARP && s2 < nsnp) {
                            const double sa = sh[ca], sb = sh[cb];
                            const double d = tot[NC + u] - sa * tot[cb] - sb * tot[ca] + (double)n * sa * sb;
                            A.D[(size_t)(i0 + s2) * R * R + a * R + bb] = d;
                            A.D[(size_t)(i0 + s2) * R * R + bb * R + a] = d;
                        }
                    }
        }

        // ---- pass 2: 16-bit hi/lo split of the shifted columns, 4 rows per thread and step (eight
        // rows, two 16-byte loads at a 32-byte stride, cost two wavefronts for one).  The tail rows
        // [n, n_pad) are zero: the other operands of the GEMMs are too, but 0 - sh times the FP16 scale
        // (which the shifted column's norm bounds, not its mean) would overflow, and inf x 0 is NaN.
        if (A.write_split) {
            auto store = [&](int c, int k4, const float4& p) {
                uint2 h, o;
                if (A.xscale)
                    split4h(p, hs[c], h, o);
                else
                    split4(p, h, o);
                reinterpret_cast<uint2*>(A.Xhi + (size_t)(i0 * R + c) * A.n_pad)[k4] = h;
                reinterpret_cast<uint2*>(A.Xlo + (size_t)(i0 * R + c) * A.n_pad)[k4] = o;
                if constexpr (F64)
                    if (A.Bhi) {
                        split4(p, h, o);
                        reinterpret_cast<uint2*>(A.Bhi + (size_t)(i0 * R + c) * A.n_pad)[k4] = h;
                        reinterpret_cast<uint2*>(A.Blo + (size_t)(i0 * R + c) * A.n_pad)[k4] = o;
                    }
            };
            by_offset([&](auto O) {
#pragma unroll 2
                for (int k4 = threadIdx.x; k4 < n / 4; k4 += NT) {
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        if (c >= ncol) continue;
                        const float s0 = sh[c];
                        float4 p = ld4(O, c, k4);
                        p.x -= s0; p.y -= s0; p.z -= s0; p.w -= s0;
                        store(c, k4, p);
                    }
                }
            });
            // the last rows and the tail, by the last warp (n_pad - n < 64: at most 16 blocks of four rows)
            const int k4 = n / 4 + (int)threadIdx.x - (NT - 32);
            if ((int)threadIdx.x >= NT - 32 && k4 < A.n_pad / 4) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (c >= ncol) continue;
                    const float* q = cols + (size_t)c * cs + off[c] + 4 * k4;
                    store(c, k4, make_float4(4 * k4 < n ? q[0] - sh[c] : 0.f, 4 * k4 + 1 < n ? q[1] - sh[c] : 0.f,
                                             4 * k4 + 2 < n ? q[2] - sh[c] : 0.f, 0.f));
                }
            }
        }

        // ---- pass 3: X'X over each row set, by work items.  The pad row holds the column's shift,
        // so that empty slots add (x - sh)^2 = 0 (every warp writes it for itself: the same value)
        if (A.npass > 0) {
            if (lane == 0)
#pragma unroll
                for (int c = 0; c < NC; ++c) cols[(size_t)c * cs + off[c] + A.n_pad] = sh[c];
            __syncwarp();
        }
        for (int ps = 0; ps < A.npass; ++ps) {
            const int s0 = __ldg(A.pass_off + ps), s1 = __ldg(A.pass_off + ps + 1);
            const int it0 = __ldg(A.set_item_off + s0), it1 = __ldg(A.set_item_off + s1);
            for (int item = it0 + w; item < it1; item += NWARP) {
                const int2 it = __ldg(A.items + item);
                float sacc[NU];
#pragma unroll
                for (int u = 0; u < NU; ++u) sacc[u] = 0.f;
                const uint4* blk = A.item_rows + (size_t)it.x * 32 + lane;
                for (int left = it.y; left > 0; left -= LEAN_BLOCK_ROWS, blk += 32) {
                    const uint4 q = __ldg(blk);
                    const uint32_t kid[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int u = 0; u < LEAN_BLOCK_ROWS / 32; ++u) {
                        if ((u == 2 || u == 4) && left <= 32 * u) break;   // warp-uniform
                        const int k = (int)(u % 2 ? kid[u / 2] >> 16 : kid[u / 2] & 0xffffu);
                        float x[NC];
#pragma unroll
                        for (int c = 0; c < NC; ++c) x[c] = cols[(size_t)c * cs + off[c] + k] - sh[c];
#pragma unroll
                        for (int s = 0; s < SPB; ++s)
#pragma unroll
                            for (int a = 0; a < R; ++a)
#pragma unroll
                                for (int bb = a; bb < R; ++bb) {
                                    float& d = sacc[s * NP + lean_pair<R>(a, bb)];
                                    d = fmaf(x[s * R + a], x[s * R + bb], d);
                                }
                    }
                }
                warp_sums<NU>(sacc, [&](int u, float sum) { part[(size_t)(item - it0) * NU + u] = sum; });
            }
            __syncthreads();
            for (int u = threadIdx.x; u < (s1 - s0) * NU; u += NT) {
                const int set = s0 + u / NU, e = u % NU;
                const int s = e / NP, f = e % NP;
                const int a0 = __ldg(A.set_item_off + set), a1 = __ldg(A.set_item_off + set + 1);
                float sum = 0.f;
                for (int it = a0; it < a1; ++it) sum += part[(size_t)(it - it0) * NU + e];
                if (s < nsnp) {
                    int a = 0, bb = 0;
#pragma unroll
                    for (int x = 0; x < R; ++x)
                        if (f >= lean_pair<R>(x, x)) a = x;
                    bb = a + f - (a * R - a * (a - 1) / 2);
                    float* d = A.Dset + ((size_t)set * A.mb + i0 + s) * R * R;
                    d[a * R + bb] = sum;
                    if (a != bb) d[bb * R + a] = sum;
                }
            }
            if (ps + 1 < A.npass) __syncthreads();   // the partial sums are read before the next pass's
        }
        if (!GATHER) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // own writes to the columns
        __syncthreads();   // every reader of the columns is done before they are refilled
        if (!GATHER && threadIdx.x == 0 && gn < ngroups) issue(gn);
        if (GATHER && gn < ngroups) stage(gn);
    }
    if (GATHER) asm volatile("cp.async.wait_group 0;" ::: "memory");   // nothing in flight at exit
    if (!GATHER && threadIdx.x == 0 && stop) {
        st_mbar_wait(&mbar, 0, true);
        st_mbar_wait(&mbar, 1, true);
    }
}

// The pre-GEMM's column matrix B2 = [Q | Q o m_1 | ... | Q o m_S] (K-major:
// column c of B2 is row c of the c2 x n_pad array), split into 16-bit hi / lo:
// BF16, or FP16 of HALF_SCALE_Q times the value (`half`).  Step 1 writes Q and
// zeros; step 2 scatters Q's rows into the columns of every row set that
// contains them.
__device__ __forceinline__ void b2_store(float v, int half, __nv_bfloat16* hi, __nv_bfloat16* lo) {
    if (half) {
        split_half(v * HALF_SCALE_Q, *reinterpret_cast<__half*>(hi), *reinterpret_cast<__half*>(lo));
    } else {
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        *hi = h;
        *lo = __float2bfloat16_rn(v - __bfloat162float(h));
    }
}

static __global__ void k_b2_init(const float* __restrict__ Qr, int LP, int n, int n_pad, int l, int c2, int half,
                          __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= (long long)c2 * n_pad) return;
    const int c = (int)(q / n_pad), k = (int)(q % n_pad);
    b2_store((c < l && k < n) ? Qr[(size_t)k * LP + c] : 0.f, half, hi + q, lo + q);
}

static __global__ void k_b2_scatter(const float* __restrict__ Qr, int LP, int n_pad, int l, const int* __restrict__ set_off,
                             const int* __restrict__ rows, int half, __nv_bfloat16* __restrict__ hi,
                             __nv_bfloat16* __restrict__ lo) {
    const int s = blockIdx.x;
    const int r0 = set_off[s], r1 = set_off[s + 1];
    const size_t base = (size_t)(l + s * l) * n_pad;
    for (int kk = r0 + threadIdx.x; kk < r1; kk += blockDim.x) {
        const int k = rows[kk];
        for (int a = 0; a < l; ++a) {
            const size_t q = base + (size_t)a * n_pad + k;
            b2_store(Qr[(size_t)k * LP + a], half, hi + q, lo + q);
        }
    }
}

static __global__ void k_fill(float* __restrict__ p, int n, float v) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) p[q] = v;
}

struct SchurArgs {
    int l, mb, G, Z, ldc;
    int rr;                  // the caller's columns per SNP; columns [rr, R) are zero padding
    const float* C2;         // pre-GEMM output, column c of SNP column x at C2[c * ldc + x]
    const double* D;         // [mb][r*r]
    const float* Dset;       // [G+Z][mb][r*r]
    const double* W;         // [G][l][l]
    const uint8_t* pat_bad;  // [G]
    double* sinv;            // [G][mb][r*r]
    uint8_t* sing;           // [G][mb]
    float* varx;             // [mb][r]
    float* aobs;             // [G][mb][l][r] or null
    float* afull;            // [mb][l][r] or null
    double* sfinv;           // [mb][r*r] or null
    float* zA;               // [Z][mb][l][r]
    float* zD;               // [Z][mb][r][r]
    // the reference's r >= 2 downdate (quirk mode, raw uncentred columns), or null:
    float* qdel;             // [G][mb][l][r] the quirk's change of Q_obs'X
    double* qK;              // [G][mb][r][r] Gram matrix term of the quirk's RSS
    // all-rows projection A of each SNP column from k_snp_lean ([mb*r][ql]), or null: A from
    // the pre-GEMM's first l columns
    const double* Afull_lean;
    int ql;
};

// The system of (pattern g, SNP i) as the reference's r >= 2 downdate builds
// it (correct_missings_S, src/Algorithm.cpp:1370-1399, read through sposv's
// upper triangle; Sbr_corr filled only for j < min(l, r), :1300): every SNP
// column's covariate downdate Str_corr is subtracted from the first SNP
// column only, and with r > l the SNP-block downdates of rows a >= l are
// missing.  In the orthonormal covariate basis (XL = Q R, raw uncentred SNP
// columns, Str_corr = R' A_g with A_g = (Q o m_g)'X) the quirk changes the
// covariate block ao = Q_obs'X to ao + dl with
//     dl[:, 0] = -sum_{b >= 1} A_g[:, b],   dl[:, b] = A_g[:, b] (b >= 1),
// and the SNP block Dobs = X_obs'X_obs by +D_g[a][b] for min(a, b) >= l.
// The quirk's solution is the Frisch-Waugh-Lovell one of that system:
//     beta_x = Sq^-1 (z - dl' b0_j),  Sq = Dobs + dD - (ao + dl)' W_g (ao + dl),
// and the reference's explicit RSS of that beta over the observed rows is
//     RSS = RSS0_j - 2 beta_x' z + beta_x' (Schur_g + dl' W_g dl) beta_x
// (the cross terms vanish because Q_obs' y~ = 0 and Q_obs'Q_obs = W_g^-1).
// Stored per (g, i): Sq^-1 (sinv), dl (qdel), Schur_g + dl' W_g dl (qK), and
// ao + dl (aobs: the covariate fit and the rows with y == 0 use it).
template <int R>
__device__ __noinline__ void schur_quirk(const SchurArgs& S, int i, int g, size_t gi, const double* ao,
                                         const double* Dm, const double* dso, bool full_ok) {
    const int l = S.l;
    const double* Wg = S.W + (size_t)g * l * l;
    double dl[OA_MAX_L * R], aq[OA_MAX_L * R];
    for (int qq = 0; qq < l; ++qq) {
        double ag[R];
#pragma unroll
        for (int a = 0; a < R; ++a) ag[a] = (double)S.C2[(size_t)(l + g * l + qq) * S.ldc + i * R + a];
        double rest = 0.0;
#pragma unroll
        for (int b = 1; b < R; ++b) rest += ag[b];
        dl[qq * R] = -rest;
#pragma unroll
        for (int b = 1; b < R; ++b) dl[qq * R + b] = ag[b];
#pragma unroll
        for (int a = 0; a < R; ++a) aq[qq * R + a] = ao[qq * R + a] + dl[qq * R + a];
    }
    // X'W X for the three column sets this needs: (ao, ao), (aq, aq), (dl, dl)
    auto quad = [&](const double* u, double* out) {
#pragma unroll
        for (int a = 0; a < R * R; ++a) out[a] = 0.0;
        for (int qq = 0; qq < l; ++qq) {
            double wu[R];
#pragma unroll
            for (int b = 0; b < R; ++b) wu[b] = 0.0;
            for (int v = 0; v < l; ++v) {
                const double w = Wg[qq * l + v];
#pragma unroll
                for (int b = 0; b < R; ++b) wu[b] += w * u[v * R + b];
            }
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
                for (int b = 0; b < R; ++b) out[a * R + b] += u[qq * R + a] * wu[b];
        }
    };
    double Dobs[R * R], Sq[R * R], t1[R * R], t2[R * R];
#pragma unroll
    for (int u = 0; u < R * R; ++u) Dobs[u] = Dm[u] - (double)S.Dset[gi * R * R + u];
    quad(aq, t1);
#pragma unroll
    for (int a = 0; a < R; ++a)
#pragma unroll
        for (int b = 0; b < R; ++b) {
            const double dD = (a >= l && b >= l) ? (double)S.Dset[gi * R * R + a * R + b] : 0.0;
            Sq[a * R + b] = Dobs[a * R + b] + dD - t1[a * R + b];
        }
    quad(ao, t1);
    quad(dl, t2);
#pragma unroll
    for (int u = 0; u < R * R; ++u) S.qK[gi * R * R + u] = Dobs[u] - t1[u] + t2[u];
#pragma unroll
    for (int a = 0; a < R; ++a)
        if (a >= S.rr) Sq[a * R + a] = 1.0;
    const bool ok = full_ok && !S.pat_bad[g] && schur_inverse<R>(Sq, dso);
    S.sing[gi] = ok ? 0 : 1;
#pragma unroll
    for (int u = 0; u < R * R; ++u) S.sinv[gi * R * R + u] = ok ? Sq[u] : 0.0;
    for (int u = 0; u < l * R; ++u) S.qdel[gi * l * R + u] = (float)dl[u];
    if (S.aobs)
        for (int u = 0; u < l * R; ++u) S.aobs[gi * l * R + u] = (float)aq[u];
}

// All (SNP, pattern) systems of a SNP block in one persistent launch.  Slot 0 is
// the all-rows complement (var_x), slots 1..G the patterns, slots G+1..G+Z
// copy the zero-set sums; a thread takes one SNP and up to SCHUR_SLOTS
// consecutive slots, so that the SNP's projection, its all-rows complement and
// that complement's factorisation (which every slot needs) are formed once for
// them.  LC: covariates held in registers (l <= LC).  Bound by FP64 latency:
// with one slot per thread and arrays in local memory 20,000 SNPs of two
// columns x 151 slots took 415 us for 260 MB of sums and inverses (333 us now).
constexpr int SCHUR_SLOTS = 8;

template <int R, int LC>
__device__ __forceinline__ void schur_slots(const SchurArgs& S, int i, int slot0, int slot1) {
    const int l = S.l;
    constexpr int UL = R <= 4 ? LC * R : 1;   // eight columns: arrays too large for registers, rolled loops
    const int QL = R <= 4 ? LC : l;
    double a_full[LC * R];
#pragma unroll UL
    for (int qq = 0; qq < QL; ++qq)
#pragma unroll
        for (int a = 0; a < R; ++a)
            a_full[qq * R + a] = qq >= l ? 0.0
                                 : S.Afull_lean ? S.Afull_lean[((size_t)i * R + a) * S.ql + qq]
                                                : (double)S.C2[(size_t)qq * S.ldc + i * R + a];
    double Dm[R * R];
#pragma unroll
    for (int u = 0; u < R * R; ++u) Dm[u] = S.D[(size_t)i * R * R + u];
    // all-rows Schur complement D - A'A (Q orthonormal): var_x of the SNP terms (src/Algorithm.cpp:665-670)
    double Sf[R * R];
#pragma unroll
    for (int a = 0; a < R; ++a)
#pragma unroll
        for (int b = 0; b < R; ++b) {
            double v = Dm[a * R + b];
#pragma unroll UL
            for (int qq = 0; qq < QL; ++qq)
                if (qq < l) v -= a_full[qq * R + a] * a_full[qq * R + b];
            Sf[a * R + b] = v;
        }
    double dss[R];
#pragma unroll
    for (int a = 0; a < R; ++a) dss[a] = Dm[a * R + a];
    // zero padding columns (r = 3, 5, 6, 7 run as 4 or 8): their rows and columns of every sum are
    // exactly 0; an identity block keeps them out of the other columns' solution (coefficient 0)
#pragma unroll
    for (int a = 0; a < R; ++a)
        if (a >= S.rr) Sf[a * R + a] = dss[a] = 1.0;
    const bool full_ok = schur_inverse<R>(Sf, dss);
    for (int slot = slot0; slot < slot1; ++slot) {
        if (slot == 0) {
#pragma unroll
            for (int a = 0; a < R; ++a) S.varx[(size_t)i * R + a] = full_ok ? (float)Sf[a * R + a] : 0.f;
            if (S.sfinv)
#pragma unroll
                for (int u = 0; u < R * R; ++u) S.sfinv[(size_t)i * R * R + u] = full_ok ? Sf[u] : 0.0;
            if (S.afull)
#pragma unroll UL
                for (int u = 0; u < QL * R; ++u)
                    if (u < l * R) S.afull[(size_t)i * l * R + u] = (float)a_full[u];
            continue;
        }
        if (slot > S.G) {  // zero set z: its sums go to the epilogue unchanged
            const int z = slot - 1 - S.G;
            const size_t zi = (size_t)z * S.mb + i;
            for (int qq = 0; qq < l; ++qq)
#pragma unroll
                for (int a = 0; a < R; ++a)
                    S.zA[zi * l * R + qq * R + a] = S.C2[(size_t)(l + (S.G + z) * l + qq) * S.ldc + i * R + a];
#pragma unroll
            for (int u = 0; u < R * R; ++u) S.zD[zi * R * R + u] = S.Dset[((size_t)(S.G + z) * S.mb + i) * R * R + u];
            continue;
        }
        const int g = slot - 1;
        const size_t gi = (size_t)g * S.mb + i;
        double ao[LC * R];
#pragma unroll UL
        for (int qq = 0; qq < QL; ++qq)
#pragma unroll
            for (int a = 0; a < R; ++a)
                ao[qq * R + a] =
                    qq < l ? a_full[qq * R + a] - (double)S.C2[(size_t)(l + g * l + qq) * S.ldc + i * R + a] : 0.0;
        double Sg[R * R];
#pragma unroll
        for (int u = 0; u < R * R; ++u) Sg[u] = Dm[u] - (double)S.Dset[gi * R * R + u];
        double dso[R];
#pragma unroll
        for (int a = 0; a < R; ++a) dso[a] = a < S.rr ? Sg[a * R + a] : 1.0;
        const double* Wg = S.W + (size_t)g * l * l;
#pragma unroll UL
        for (int qq = 0; qq < QL; ++qq) {
            if (qq < l) {
                double wa[R];
#pragma unroll
                for (int b = 0; b < R; ++b) wa[b] = 0.0;
#pragma unroll UL
                for (int u = 0; u < QL; ++u) {
                    if (u < l) {
                        const double wq = Wg[qq * l + u];
#pragma unroll
                        for (int b = 0; b < R; ++b) wa[b] += wq * ao[u * R + b];
                    }
                }
#pragma unroll
                for (int a = 0; a < R; ++a)
#pragma unroll
                    for (int b = 0; b < R; ++b) Sg[a * R + b] -= ao[qq * R + a] * wa[b];
            }
        }
        if (S.qK) {
            double aoq[LC * R], Dq[R * R], dq[R];   // copies: the arrays above stay in registers
#pragma unroll UL
            for (int u = 0; u < QL * R; ++u) aoq[u] = ao[u];
#pragma unroll
            for (int u = 0; u < R * R; ++u) Dq[u] = Dm[u];
#pragma unroll
            for (int a = 0; a < R; ++a) dq[a] = dso[a];
            schur_quirk<R>(S, i, g, gi, aoq, Dq, dq, full_ok);
            continue;
        }
#pragma unroll
        for (int a = 0; a < R; ++a)
            if (a >= S.rr) Sg[a * R + a] = 1.0;
        const bool ok = full_ok && !S.pat_bad[g] && schur_inverse<R>(Sg, dso);
        S.sing[gi] = ok ? 0 : 1;
#pragma unroll
        for (int u = 0; u < R * R; ++u) S.sinv[gi * R * R + u] = ok ? Sg[u] : 0.0;
        if (S.aobs)
#pragma unroll UL
            for (int u = 0; u < QL * R; ++u)
                if (u < l * R) S.aobs[gi * l * R + u] = (float)ao[u];
    }
}

// Items (SNP, `per` slots) are numbered slot-major (consecutive threads take consecutive SNPs of one slot
// range), so that a warp's loads of the SNP-indexed sums (pre-GEMM columns, D, D_s) and its stores of the
// inverses are coalesced and the slot's W_g is one broadcast.
template <int R, int LC>
__global__ void __launch_bounds__(256) k_schur(SchurArgs S, int per) {
    const int slots = 1 + S.G + S.Z;
    const long long total = (long long)S.mb * ((slots + per - 1) / per);
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const int slot0 = (int)(q / S.mb) * per;
        schur_slots<R, LC>(S, (int)(q % S.mb), slot0, min(slots, slot0 + per));
    }
}

}  // namespace oa
