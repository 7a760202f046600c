// FP32-accurate contraction on the tensor cores (the plain form):
//     C[col][row] = sum_k X[row][k] B[col][k]
// with both operands split into FP16 hi + lo (each column scaled by a power
// of two, x s = hi + lo to about 2^-23 relative) and the products
//     hi lo' + lo hi' + hi hi'            (lo lo', ~2^-24, is dropped)
// accumulated in TMEM for one K-block of 64 only: the epilogue warps add
// every K-block's partial product to FP32 register sums (round to nearest).
//
// Why the partial sums leave TMEM: the tensor core's FP32 accumulation
// truncates, and over a whole column (n / 16 MMA steps of three products)
// that bias is 3e-5 of the result at n = 10,000.  In a K-block the small
// products go first (the accumulator is still ~2^-11 of its final size, so
// their truncation does not count), then four hi hi' steps: a bias of about
// 1e-7 whatever n, below the rounding of one sequential FP32 sum (measured
// against FP64: 1.2e-6 of beta at n = 10,000 with the FP32 SIMT GEMM).
//
// What bounds it: 12 tcgen05.mma per K-block and 256 x 256 pair tile, 128
// cycles each, while the drain of that K-block (128 columns of 32 lanes per
// warp: tcgen05.ld + FADD) takes about a third of them; at small column
// counts the reading of X.  Measured (60,000 SNPs x 1,084 columns, n =
// 10,000): FP32 SIMT 26.5 + 5.0 ms in two launches a chunk, this 2.87 ms =
// 1.36 PFLOP/s of FP16 products (the power-capped rate of a dense GEMM);
// error against 64 bits 1.6e-6 -> 2.7e-7 of the outputs' 2-norm.
//
// The product is stored (not evaluated in the epilogue): the register sums
// leave no registers for the statistics, and z is 4 bytes per test against
// the 4 n / t bytes per test of X; k_test_stats (oa_test_stats.cuh) reads it
// back from L2.  Stored columns can then hold the pre-GEMM's column matrix as
// well as the traits, so that one launch reads X once for both.
//
// Included by oa_gemm_tc.cu (barrier, TMA and MMA helpers).

// Pipeline shape of the promoted kernels: K-block 64 (128-byte swizzle).
// ACCS TMEM accumulators of BN columns: with narrow tiles four of them, so
// that the drain's latency stays off the MMA's path.
template <int STAGES_, int BN_, bool PAIR>
struct ShapeP {
    static constexpr int BK = 64, STAGES = STAGES_, BN = BN_;
    static constexpr int ACCS = BN <= 128 ? 4 : 2;
    static constexpr int A_BYTES = BM * BK * 2;                     // this CTA's 128 rows, one of hi / lo
    static constexpr int B_ROWS = PAIR ? BN / 2 : BN;               // this CTA's rows of B
    static constexpr int B_BYTES = B_ROWS * BK * 2;
    static constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;
    static constexpr size_t SMEM_BYTES = 1024 + (size_t)STAGES * STAGE_BYTES;
    static constexpr uint64_t LAYOUT = 2u;
    static constexpr uint32_t SBO = 1024u;
    static constexpr uint32_t TMEM_COLS = ACCS * BN;                // 256 or 512
    // kind::f16, D FP32 (bits 4-5 = 1), A and B FP16 (bits 7-9 and 10-12 = 0), K-major, N at bits 17-22, M >> 4
    static constexpr uint32_t IDESC_M = (1u << 4) | ((uint32_t)((PAIR ? 256 : 128) >> 4) << 24);
    static constexpr int GPW = BN / 64;                             // 32-column groups per epilogue warp
    static_assert(TMEM_COLS == 256 || TMEM_COLS == 512, "TMEM allocation");
    static_assert(SMEM_BYTES <= 227u * 1024u, "shared memory");
};

// The twelve MMAs of one K-block into a fresh accumulator: the eight small
// products first, then hi hi'.
template <class SH, bool PAIR>
__device__ __forceinline__ void mma_kblock(uint32_t d_tmem, uint32_t ahi, uint32_t alo, uint32_t bhi, uint32_t blo,
                                           uint32_t idesc) {
    auto mma = [&](uint32_t a, uint32_t b, uint32_t acc) {
        if constexpr (PAIR)
            mma_bf16_pair(d_tmem, smem_desc<SH>(a), smem_desc<SH>(b), idesc, acc);
        else
            mma_bf16(d_tmem, smem_desc<SH>(a), smem_desc<SH>(b), idesc, acc);
    };
#pragma unroll
    for (int kk = 0; kk < SH::BK / 16; ++kk) {
        const uint32_t off = (uint32_t)kk * 32u;   // 16 halves along K inside the swizzled row
        mma(ahi + off, blo + off, kk > 0 ? 1u : 0u);
        mma(alo + off, bhi + off, 1u);
    }
#pragma unroll
    for (int kk = 0; kk < SH::BK / 16; ++kk) mma(ahi + (uint32_t)kk * 32u, bhi + (uint32_t)kk * 32u, 1u);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Adds one K-block's accumulator to the warp's register sums.  The warp's 32
// lanes are rows; of the tile's 32-column groups it owns h, h + 2, ... (two
// warps share each TMEM lane group); groups at or past `ncols` hold nothing.
template <int GPW>
__device__ __forceinline__ void drain_kblock(uint32_t taddr, int h, int ncols, float (&sum)[GPW][32]) {
#pragma unroll
    for (int g = 0; g < GPW; ++g) {
        const int c = 32 * (2 * g + h);
        if (c < ncols) {
            // 16 columns at a time: with 128 sums a thread has no room for 32 more registers
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                uint32_t v[16];
                tmem_ld16(taddr + (uint32_t)(c + 16 * u), v);
#pragma unroll
                for (int q = 0; q < 16; ++q) sum[g][16 * u + q] += __uint_as_float(v[q]);
            }
        }
    }
}

// The tile's sums to C (transposed, lane = row: 128-byte segments), taken
// back to the columns' own scale: rs = 1 / scale of the lane's row, cscale =
// 1 / scale of each column.
template <int GPW>
__device__ __forceinline__ void store_sums(const float (&sum)[GPW][32], int h, int n0, int t, int row, int xrows,
                                           float rs, const float* __restrict__ cscale, float* __restrict__ cout,
                                           int ldc) {
#pragma unroll
    for (int g = 0; g < GPW; ++g) {
        const int c = n0 + 32 * (2 * g + h);
        if (c < t && row < xrows) {
#pragma unroll
            for (int q = 0; q < 32; ++q)
                if (c + q < t) cout[(size_t)(c + q) * ldc + row] = sum[g][q] * rs * __ldg(cscale + c + q);
        }
    }
}

// One CTA per tile of 128 rows x BN columns (column counts up to 128).
// Warps as in k_gemm_tc: 0 TMA producer, 1 MMA issuer, 2..9 drain and store.
template <class SH>
__global__ void __launch_bounds__(NUM_THREADS, 1)
k_gemm_tcp(const __grid_constant__ CUtensorMap mAhi, const __grid_constant__ CUtensorMap mAlo,
           const __grid_constant__ CUtensorMap mBhi, const __grid_constant__ CUtensorMap mBlo, int xrows, int t,
           int nk, const float* __restrict__ rscale, const float* __restrict__ cscale, float* __restrict__ cout,
           int ldc, int* err) {
    constexpr int BK = SH::BK, STAGES = SH::STAGES, BN = SH::BN, ACCS = SH::ACCS;
    constexpr int A_BYTES = SH::A_BYTES, B_BYTES = SH::B_BYTES, STAGE_BYTES = SH::STAGE_BYTES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[ACCS], acc_empty[ACCS], done_bar;
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_sh;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m_tiles = (xrows + BM - 1) / BM, n_tiles = (t + BN - 1) / BN;
    const int ntiles = m_tiles * n_tiles;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int a = 0; a < ACCS; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], EPI_WARPS);
        }
        mbar_init(&done_bar, 1);
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&tmem_base_sh)),
                     "r"(SH::TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem_base = tmem_base_sh;
    auto stage_ptr = [&](int s, int which) -> uint8_t* {
        uint8_t* b = smem + (size_t)s * STAGE_BYTES;
        return which < 2 ? b + which * A_BYTES : b + 2 * A_BYTES + (which - 2) * B_BYTES;
    };

    if (warp == 0) {
        if (lane == 0) {
            // ---------------- TMA producer ----------------
            int s = 0;
            uint32_t ph = 0;
            uint32_t pend_par[STAGES];
            bool pend[STAGES];
            for (int q = 0; q < STAGES; ++q) pend[q] = false;
            bool ok = true;
            int pt = blockIdx.x, pkb = 0;   // L2 prefetch cursor, pf_blocks<BK>() K-blocks ahead
            auto prefetch_next = [&]() {
                if (pt >= ntiles) return;
                const int pm0 = pt / n_tiles * BM;
                tma_prefetch_2d(&mAhi, pkb * BK, pm0);
                tma_prefetch_2d(&mAlo, pkb * BK, pm0);
                if (++pkb == nk) {
                    pkb = 0;
                    pt += gridDim.x;
                }
            };
            for (int q = 0; q < pf_blocks<BK>(); ++q) prefetch_next();
            for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
                const int m0 = tile / n_tiles * BM, n0 = tile % n_tiles * BN;
                for (int kb = 0; kb < nk; ++kb) {
                    if (!mbar_wait(&empty_bar[s], ph ^ 1u, &abort_sh)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&full_bar[s], STAGE_BYTES);
                    tma_load_2d(&mAhi, &full_bar[s], stage_ptr(s, 0), kb * BK, m0);
                    tma_load_2d(&mAlo, &full_bar[s], stage_ptr(s, 1), kb * BK, m0);
                    tma_load_2d(&mBhi, &full_bar[s], stage_ptr(s, 2), kb * BK, n0);
                    tma_load_2d(&mBlo, &full_bar[s], stage_ptr(s, 3), kb * BK, n0);
                    prefetch_next();
                    pend[s] = true;
                    pend_par[s] = ph;
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (!ok)  // drain our own copies before the shared memory goes away
                for (int q = 0; q < STAGES; ++q)
                    if (pend[q]) mbar_drain(&full_bar[q], pend_par[q]);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---------------- MMA issuer ----------------
            constexpr uint32_t idesc = SH::IDESC_M | ((uint32_t)(BN >> 3) << 17);
            int s = 0, acc = 0;
            uint32_t ph = 0, aph = 0;
            bool ok = true, issued = false;
            for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
                for (int kb = 0; kb < nk; ++kb) {
                    if (!mbar_wait(&acc_empty[acc], aph ^ 1u, &abort_sh) || !mbar_wait(&full_bar[s], ph, &abort_sh)) {
                        ok = false;
                        break;
                    }
                    fence_after();
                    mma_kblock<SH, false>(tmem_base + (uint32_t)(acc * BN), su32(stage_ptr(s, 0)),
                                          su32(stage_ptr(s, 1)), su32(stage_ptr(s, 2)), su32(stage_ptr(s, 3)), idesc);
                    issued = true;
                    mma_commit(&empty_bar[s]);
                    mma_commit(&acc_full[acc]);
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                    if (++acc == ACCS) {
                        acc = 0;
                        aph ^= 1u;
                    }
                }
            }
            if (issued) {  // all MMAs of this CTA complete before TMEM is freed
                mma_commit(&done_bar);
                mbar_drain(&done_bar, 0);
            }
        }
    } else {
        // ---------------- drain and store ----------------
        const int lg = warp & 3, h = (warp - 2) >> 2;
        const uint32_t tlane = tmem_base + ((uint32_t)(lg * 32) << 16);
        int acc = 0;
        uint32_t aph = 0;
        bool go = true;
        for (int tile = blockIdx.x; tile < ntiles && go; tile += gridDim.x) {
            const int m0 = tile / n_tiles * BM, n0 = tile % n_tiles * BN;
            const int row = m0 + lg * 32 + lane;
            const float rs = row < xrows ? __ldg(rscale + row) : 0.f;
            float sum[SH::GPW][32];
#pragma unroll
            for (int g = 0; g < SH::GPW; ++g)
#pragma unroll
                for (int q = 0; q < 32; ++q) sum[g][q] = 0.f;
            for (int kb = 0; kb < nk; ++kb) {
                int ok = 1;
                if (lane == 0) ok = mbar_wait(&acc_full[acc], aph, &abort_sh) ? 1 : 0;
                if (!__shfl_sync(0xffffffffu, ok, 0)) {
                    go = false;
                    break;
                }
                mbar_try(&acc_full[acc], aph);
                fence_after();
                drain_kblock<SH::GPW>(tlane + (uint32_t)(acc * BN), h, BN, sum);
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[acc]);
                if (++acc == ACCS) {
                    acc = 0;
                    aph ^= 1u;
                }
            }
            if (go) store_sums<SH::GPW>(sum, h, n0, t, row, xrows, rs, cscale, cout, ldc);
        }
    }

    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(SH::TMEM_COLS));
    }
    if (threadIdx.x == 0 && abort_sh) atomicExch(err, 1);
}

// CTA pairs (256 rows x 256 columns, tcgen05.mma.cta_group::2; barriers and
// operand halves as in k_gemm_tc2).  The last column tile runs at its own
// width (a multiple of 32), so that t = 1,084 costs 1,088 columns of MMA work
// and not 1,280.
template <class SH>
__global__ void __launch_bounds__(NUM_THREADS, 1)
k_gemm_tcp2(const __grid_constant__ CUtensorMap mAhi, const __grid_constant__ CUtensorMap mAlo,
            const __grid_constant__ CUtensorMap mBhi, const __grid_constant__ CUtensorMap mBlo, int xrows, int t,
            int nk, const float* __restrict__ rscale, const float* __restrict__ cscale, float* __restrict__ cout,
            int ldc, int* err) {
    constexpr int BK = SH::BK, STAGES = SH::STAGES, BN = SH::BN, ACCS = SH::ACCS;
    constexpr int A_BYTES = SH::A_BYTES, B_BYTES = SH::B_BYTES, STAGE_BYTES = SH::STAGE_BYTES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[ACCS], acc_empty[ACCS], done_bar;
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_sh;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const bool leader = rank == 0;
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const int m_tiles = (xrows + 2 * BM - 1) / (2 * BM), n_tiles = (t + BN - 1) / BN;
    const int ntiles = m_tiles * n_tiles;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int a = 0; a < ACCS; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 2 * EPI_WARPS);   // one arrival per epilogue warp of both CTAs (leader's copy)
        }
        mbar_init(&done_bar, 1);
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&tmem_base_sh)),
                     "r"(SH::TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    cluster_sync();       // both CTAs' barriers and TMEM exist before any remote use
    fence_after();
    const uint32_t tmem_base = tmem_base_sh;
    auto stage_ptr = [&](int s, int which) -> uint8_t* {
        uint8_t* b = smem + (size_t)s * STAGE_BYTES;
        return which < 2 ? b + which * A_BYTES : b + 2 * A_BYTES + (which - 2) * B_BYTES;
    };
    // first row, first column and column count (a multiple of 32) of a tile
    auto tile_mn = [&](int tile, int& m0, int& n0, int& nc) {
        m0 = tile / n_tiles * 2 * BM;
        n0 = tile % n_tiles * BN;
        nc = min(BN, (t - n0 + 31) & ~31);
    };

    if (warp == 0) {
        if (lane == 0) {
            // ---------------- TMA producer (both CTAs) ----------------
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            int pt = pair, pkb = 0;          // L2 prefetch cursor, pf_blocks<BK>() K-blocks ahead
            auto prefetch_next = [&]() {
                if (pt >= ntiles) return;
                const int pm0 = pt / n_tiles * 2 * BM;
                tma_prefetch_2d(&mAhi, pkb * BK, pm0 + (int)rank * BM);
                tma_prefetch_2d(&mAlo, pkb * BK, pm0 + (int)rank * BM);
                if (++pkb == nk) {
                    pkb = 0;
                    pt += npairs;
                }
            };
            for (int q = 0; q < pf_blocks<BK>(); ++q) prefetch_next();
            for (int tile = pair; tile < ntiles && ok; tile += npairs) {
                int m0, n0, nc;
                tile_mn(tile, m0, n0, nc);
                const int ma = m0 + (int)rank * BM, nb = n0 + (int)rank * (nc / 2);
                for (int kb = 0; kb < nk; ++kb) {
                    if (!mbar_wait(&empty_bar[s], ph ^ 1u, &abort_sh)) {
                        ok = false;
                        break;
                    }
                    const uint32_t fb = map_to_rank(&full_bar[s], 0);
                    if (leader) mbar_expect_tx(&full_bar[s], 2 * STAGE_BYTES);
                    tma_load_2d_pair(&mAhi, fb, stage_ptr(s, 0), kb * BK, ma);
                    tma_load_2d_pair(&mAlo, fb, stage_ptr(s, 1), kb * BK, ma);
                    tma_load_2d_pair(&mBhi, fb, stage_ptr(s, 2), kb * BK, nb);
                    tma_load_2d_pair(&mBlo, fb, stage_ptr(s, 3), kb * BK, nb);
                    prefetch_next();
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (!ok && leader)   // the leader's full barriers see both CTAs' copies: drain them
                for (int q = 0; q < STAGES; ++q) mbar_drain(&full_bar[q], 0), mbar_drain(&full_bar[q], 1);
        }
    } else if (warp == 1) {
        if (lane == 0 && leader) {
            // ---------------- MMA issuer (leader CTA) ----------------
            int s = 0, acc = 0;
            uint32_t ph = 0, aph = 0;
            bool ok = true, issued = false;
            for (int tile = pair; tile < ntiles && ok; tile += npairs) {
                int m0, n0, nc;
                tile_mn(tile, m0, n0, nc);
                const uint32_t idesc = SH::IDESC_M | ((uint32_t)(nc >> 3) << 17);
                for (int kb = 0; kb < nk; ++kb) {
                    if (!mbar_wait(&acc_empty[acc], aph ^ 1u, &abort_sh) || !mbar_wait(&full_bar[s], ph, &abort_sh)) {
                        ok = false;
                        break;
                    }
                    fence_after();
                    mma_kblock<SH, true>(tmem_base + (uint32_t)(acc * BN), su32(stage_ptr(s, 0)),
                                         su32(stage_ptr(s, 1)), su32(stage_ptr(s, 2)), su32(stage_ptr(s, 3)), idesc);
                    issued = true;
                    mma_commit_pair(&empty_bar[s]);
                    mma_commit_pair(&acc_full[acc]);
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                    if (++acc == ACCS) {
                        acc = 0;
                        aph ^= 1u;
                    }
                }
            }
            if (issued) mma_commit_pair(&done_bar);   // both CTAs learn when the last MMA has completed
        }
        if (lane == 0) mbar_drain(&done_bar, 0);      // (a CTA pair that issued nothing waits out the bound once)
    } else {
        // ---------------- drain and store (both CTAs, own 128 rows) ----------------
        const int lg = warp & 3, h = (warp - 2) >> 2;
        const uint32_t tlane = tmem_base + ((uint32_t)(lg * 32) << 16);
        int acc = 0;
        uint32_t aph = 0;
        bool go = true;
        for (int tile = pair; tile < ntiles && go; tile += npairs) {
            int m0, n0, nc;
            tile_mn(tile, m0, n0, nc);
            const int row = m0 + (int)rank * BM + lg * 32 + lane;
            const float rs = row < xrows ? __ldg(rscale + row) : 0.f;
            float sum[SH::GPW][32];
#pragma unroll
            for (int g = 0; g < SH::GPW; ++g)
#pragma unroll
                for (int q = 0; q < 32; ++q) sum[g][q] = 0.f;
            for (int kb = 0; kb < nk; ++kb) {
                int ok = 1;
                if (lane == 0) ok = mbar_wait(&acc_full[acc], aph, &abort_sh) ? 1 : 0;
                if (!__shfl_sync(0xffffffffu, ok, 0)) {
                    go = false;
                    break;
                }
                mbar_try(&acc_full[acc], aph);
                fence_after();
                drain_kblock<SH::GPW>(tlane + (uint32_t)(acc * BN), h, nc, sum);
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_drained(map_to_rank(&acc_empty[acc], 0));
                if (++acc == ACCS) {
                    acc = 0;
                    aph ^= 1u;
                }
            }
            if (go) store_sums<SH::GPW>(sum, h, n0, t, row, xrows, rs, cscale, cout, ldc);
        }
    }

    fence_before();
    __syncthreads();
    cluster_sync();       // no CTA frees TMEM or leaves while its pair may still touch it
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(SH::TMEM_COLS));
    }
    if (threadIdx.x == 0 && abort_sh) atomicExch(err, 1);
}
