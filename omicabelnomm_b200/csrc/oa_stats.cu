// Instantiations of the per-SNP statistics kernels (oa_stats.cuh, oa_lean.cuh).
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "oa_lean.cuh"
#include "oa_launch.h"

namespace oa {

template <int R, int LP>
static cudaError_t go(const StatsArgs& A, int grid, size_t smem, cudaStream_t st) {
    // TMA bulk staging needs 16-byte aligned columns whose size is a multiple of 16 bytes
    const bool bulk = (A.n % 4 == 0) && (A.ldx % 4 == 0) && ((reinterpret_cast<uintptr_t>(A.X) & 15) == 0);
    // the opt-in shared-memory size is raised once per kernel and device (no
    // attribute call while a stream is being captured into a graph)
    static int set_bulk[64], set_plain[64];
    int dev = 0;
    cudaGetDevice(&dev);
    const int d = dev & 63;
    if (bulk) {
        if (set_bulk[d] < (int)smem) {
            cudaError_t e = cudaFuncSetAttribute(k_snp_stats<R, LP, true>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024);
            if (e != cudaSuccess) return e;
            set_bulk[d] = 227 * 1024 - 1024;
        }
        k_snp_stats<R, LP, true><<<grid, OA_NTHREADS, smem, st>>>(A);
    } else {
        if (set_plain[d] < (int)smem) {
            cudaError_t e = cudaFuncSetAttribute(k_snp_stats<R, LP, false>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024);
            if (e != cudaSuccess) return e;
            set_plain[d] = 227 * 1024 - 1024;
        }
        k_snp_stats<R, LP, false><<<grid, OA_NTHREADS, smem, st>>>(A);
    }
    return cudaGetLastError();
}

cudaError_t oa_launch_snp_stats(int R, int LP, const StatsArgs& A, int grid, size_t smem, cudaStream_t st) {
    switch (R * 100 + LP) {
        case 104: return go<1, 4>(A, grid, smem, st);
        case 108: return go<1, 8>(A, grid, smem, st);
        case 116: return go<1, 16>(A, grid, smem, st);
        case 204: return go<2, 4>(A, grid, smem, st);
        case 208: return go<2, 8>(A, grid, smem, st);
        case 216: return go<2, 16>(A, grid, smem, st);
        case 404: return go<4, 4>(A, grid, smem, st);
        case 408: return go<4, 8>(A, grid, smem, st);
        case 416: return go<4, 16>(A, grid, smem, st);
        default: return cudaErrorInvalidValue;
    }
}

template <int R, int SPB, int QL, int NT, bool F64>
static cudaError_t go_lean(const LeanArgs& A, int grid, size_t smem, cudaStream_t st) {
    static int set_bulk[64], set_gather[64];
    int dev = 0;
    cudaGetDevice(&dev);
    const int d = dev & 63;
    int* done = A.xrows ? set_gather : set_bulk;
    if (done[d] < (int)smem) {
        cudaError_t e = A.xrows ? cudaFuncSetAttribute(k_snp_lean<R, SPB, true, QL, NT, F64>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024)
                                : cudaFuncSetAttribute(k_snp_lean<R, SPB, false, QL, NT, F64>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024);
        if (e != cudaSuccess) return e;
        done[d] = 227 * 1024 - 1024;
    }
    if (A.xrows)
        k_snp_lean<R, SPB, true, QL, NT, F64><<<grid, NT, smem, st>>>(A);
    else
        k_snp_lean<R, SPB, false, QL, NT, F64><<<grid, NT, smem, st>>>(A);
    return cudaGetLastError();
}

template <int R, int SPB, int QL, int NT, bool F64>
static int lean_occ(size_t smem) {
    int nb = 0;
    if (cudaFuncSetAttribute(k_snp_lean<R, SPB, false, QL, NT, F64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             227 * 1024 - 1024) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_snp_lean<R, SPB, false, QL, NT, F64>, NT, smem) !=
            cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return nb;
}

// The instantiated forms: groups of R columns x SPB SNPs, QL covariate slots of the in-kernel projection
// (0: none), threads, FP64 sums.  f(R, SPB, QL, NT, F64) as integral constants; false if there is no such form.
template <class F>
static bool lean_form(int R, int spb, int ql, int threads, bool f64, F&& f) {
    const int key = (((R * 16 + spb) * 32 + ql) * 4 + threads / 256) * 2 + (f64 ? 1 : 0);
    bool found = false;
    auto form = [&](auto r, auto s, auto q, auto nt, auto p) {
        constexpr int k = (((decltype(r)::value * 16 + decltype(s)::value) * 32 + decltype(q)::value) * 4 +
                           decltype(nt)::value / 256) * 2 + (decltype(p)::value ? 1 : 0);
        if (key == k) {
            f(r, s, q, nt, p);
            found = true;
        }
    };
    using std::integral_constant;
    constexpr std::false_type f32{};
    constexpr std::true_type dbl{};
    constexpr integral_constant<int, 0> n0{};
    constexpr integral_constant<int, 1> n1{};
    constexpr integral_constant<int, 2> n2{};
    constexpr integral_constant<int, 4> n4{};
    constexpr integral_constant<int, 8> n8{};
    constexpr integral_constant<int, 16> n16{};
    constexpr integral_constant<int, 256> t256{};
    constexpr integral_constant<int, LEAN_MAX_THREADS> t512{};
    form(n1, n1, n0, t256, f32);
    form(n1, n2, n0, t256, f32);
    form(n1, n4, n0, t256, f32);
    form(n1, n8, n0, t256, f32);
    form(n2, n1, n0, t256, f32);
    form(n2, n2, n0, t256, f32);
    form(n2, n4, n0, t256, f32);
    form(n4, n1, n0, t256, f32);
    form(n4, n2, n0, t256, f32);
    form(n8, n1, n0, t256, f32);
    form(n1, n1, n0, t512, f32);
    form(n2, n1, n0, t512, f32);
    form(n4, n1, n0, t512, f32);
    form(n2, n1, n8, t256, f32);
    form(n2, n2, n8, t256, f32);
    form(n4, n1, n8, t256, f32);
    form(n2, n1, n8, t512, f32);
    form(n4, n1, n8, t512, f32);
    // wide blocks
    form(n1, n1, n4, t256, dbl);
    form(n1, n2, n4, t256, dbl);
    form(n1, n4, n4, t256, dbl);
    form(n1, n1, n4, t512, dbl);
    form(n1, n1, n8, t256, dbl);
    form(n1, n2, n8, t256, dbl);
    form(n1, n4, n8, t256, dbl);
    form(n1, n1, n8, t512, dbl);
    form(n1, n1, n16, t256, dbl);
    form(n1, n1, n16, t512, dbl);
    form(n2, n1, n8, t256, dbl);
    form(n2, n2, n8, t256, dbl);
    form(n4, n1, n8, t256, dbl);
    form(n2, n1, n8, t512, dbl);
    form(n4, n1, n8, t512, dbl);
    return found;
}

bool oa_lean_has_qx(int R, int spb, int ql, bool f64) {
    return ql > 0 && lean_form(R, spb, ql, 256, f64, [](auto...) {});
}

int oa_lean_ctas_per_sm(int R, int spb, size_t smem, int ql, int threads, bool f64) {
    // cached per (device, R, spb, ql, smem, threads, f64): no runtime calls while a stream is captured
    static std::map<std::tuple<int, int, int, int, size_t, int, bool>, int> cache;
    static std::mutex mu;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_tuple(dev, R, spb, ql, smem, threads, f64);
    {
        std::lock_guard<std::mutex> g(mu);
        auto it = cache.find(key);
        if (it != cache.end()) return it->second;
    }
    int v = 0;
    lean_form(R, spb, ql, threads, f64, [&](auto r, auto s, auto q, auto nt, auto p) {
        v = lean_occ<decltype(r)::value, decltype(s)::value, decltype(q)::value, decltype(nt)::value,
                     decltype(p)::value>(smem);
    });
    std::lock_guard<std::mutex> g(mu);
    cache[key] = v;
    return v;
}

cudaError_t oa_launch_snp_lean(int R, int spb, const LeanArgs& A, int grid, int threads, size_t smem,
                               cudaStream_t st) {
    cudaError_t e = cudaErrorInvalidValue;
    lean_form(R, spb, A.Afull ? A.ql : 0, threads, A.Afull && A.f64, [&](auto r, auto s, auto q, auto nt, auto p) {
        e = go_lean<decltype(r)::value, decltype(s)::value, decltype(q)::value, decltype(nt)::value,
                    decltype(p)::value>(A, grid, smem, st);
    });
    return e;
}

cudaError_t oa_set_wait_limit_stats(unsigned long long ns) {
    return cudaMemcpyToSymbol(c_st_wait_ns, &ns, sizeof ns);
}

template <int R>
static void go_schur(const SchurArgs& S, int per, unsigned blocks, cudaStream_t st) {
    if constexpr (R == 8) {
        k_schur<R, 16><<<blocks, 256, 0, st>>>(S, per);
    } else if (S.l > 8) {
        k_schur<R, 16><<<blocks, 256, 0, st>>>(S, per);
    } else if (S.l > 4) {
        k_schur<R, 8><<<blocks, 256, 0, st>>>(S, per);
    } else {
        k_schur<R, 4><<<blocks, 256, 0, st>>>(S, per);
    }
}

cudaError_t oa_launch_schur(int R, const SchurArgs& S, cudaStream_t st) {
    const long long slots = 1 + S.G + S.Z;
    if (S.mb <= 0) return cudaSuccess;
    // persistent: at most 8 resident CTAs of 256 threads per SM
    static int sms[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (!sms[dev & 63]) cudaDeviceGetAttribute(&sms[dev & 63], cudaDevAttrMultiProcessorCount, dev);
    // slots per thread: as many as leave every resident thread an item
    const long long room = 8LL * sms[dev & 63] * 256;
    int per = 1;
    while (per < SCHUR_SLOTS && (long long)S.mb * ((slots + 2 * per - 1) / (2 * per)) >= room) per *= 2;
    const long long total = (long long)S.mb * ((slots + per - 1) / per);
    const unsigned blocks = (unsigned)std::min<long long>((total + 255) / 256, 8LL * sms[dev & 63]);
    switch (R) {
        case 1: go_schur<1>(S, per, blocks, st); break;
        case 2: go_schur<2>(S, per, blocks, st); break;
        case 4: go_schur<4>(S, per, blocks, st); break;
        case 8: go_schur<8>(S, per, blocks, st); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace oa
