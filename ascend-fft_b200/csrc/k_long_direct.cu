// C2C of n = 32768 and 65536 in one HBM pass without a workspace.
//
// n = N1 * 256: one thread-block cluster per row, 4096 points per CTA.  The row
// is the N1 x 256 matrix x[256*n1 + n2] of the four-step decomposition
//   X[k1 + N1*k2] = sum_n2 W_256^(n2*k2) * W_n^(n2*k1) * sum_n1 W_N1^(n1*k1) x[256*n1 + n2].
// CTA `rank` owns columns n2 in [rank*COLS, (rank+1)*COLS) for the N1-point FFTs and rows k1 in
// [16*rank, 16*rank + 16) for the 256-point FFTs.  Between the two the matrix sits in the row's own
// output: the cluster writes it there and reads it back a few microseconds later, when it is still
// in L2, so HBM sees the compulsory 16 bytes per point (ncu, n = 32768: 134 MB read for 134 MB of
// input) and no workspace is needed.  In place (in == out) is safe: a CTA's matrix writes cover
// exactly the addresses it alone has read.  Every global access is a run of at least 128 bytes
// (32-byte runs through a layout that saves an exchange measured 2545 GB/s against 3374): the
// row FFTs load with 16 threads along a row and change to 16 rows across lanes at their one
// exchange, so that the stride-N1 stores are 128-byte runs too.
// 2^26 points, one launch, GB/s at n = 32768 / 65536: 3828 / 3379 (loads ahead into L2 add nothing), against
// 2980 / 2925 for the two four-step kernels, each of which crosses HBM; exchanging through
// distributed shared memory instead of L2 3009 / 2565, 8192 points per CTA (512 threads) 3318 /
// 3104.  What bounds it: the wait for the matrix writes to reach L2 at the first cluster barrier,
// at four 64-register CTAs per SM.
#include <cuda_runtime.h>

#include <mutex>
#include <vector>

#include "backend.h"
#include "fft_kernels.cuh"
#include "launch.cuh"
#include "tma.cuh"

namespace bfly {
namespace dev {

template <int N1>
struct LongDirect {
    static constexpr int N2 = 256, E = 16, N = N1 * N2;
    static constexpr int C = N / 4096;          // CTAs per row
    static constexpr int NT = 256;
    static constexpr int COLS = N2 / C;         // columns per CTA
    static constexpr int T1 = N1 / E;           // threads per column
    static constexpr int ROWS2 = N1 / C;        // rows per CTA
    static constexpr int S1 = smem_stride<N1, E, true>();
    static constexpr int S2 = (spad(N2 - 1) + 1) | 1;   // odd: rows across lanes hit distinct banks
    static constexpr int SMEM = (COLS * S1 > ROWS2 * S2 ? COLS * S1 : ROWS2 * S2) * 8;
    static_assert(COLS * T1 == NT && ROWS2 * (N2 / E) == NT, "inconsistent cluster shape");
    // one table: Stockham twiddles of N1 and of 256, then rows of 256 values W_n^(n2 T1 j), j < 16,
    // and W_n^(n2 t), t < T1
    static constexpr int TW2 = Sched<N1, E>::TWSIZE, WT = TW2 + Sched<N2, E>::TWSIZE, TABLE = WT + (E + T1) * N2;
};

template <int N1, bool INV>
__global__ void __launch_bounds__(LongDirect<N1>::NT, min_blocks_64regs(LongDirect<N1>::NT))
k_long_direct(const float2* in, float2* out, const float2* __restrict__ table, float scale) {
    using L = LongDirect<N1>;
    constexpr int E = L::E, T1 = L::T1;
    using TA = Team<N1, E, INV, kSyncBlock>;
    using TB = Team<L::N2, E, INV, kSyncBlock>;
    extern __shared__ float2 smem[];
    pdl_wait();
    const int tid = threadIdx.x;
    const uint32_t rank = cluster_ctarank();
    const uint64_t row = blockIdx.x / L::C;
    out += row * L::N;
    float2 v[E];
    {   // columns, times W_n^(n2*k1); k1 = t1 + j T1, so the factor is W_n^(n2 t1) W_n^(n2 T1 j)
        const int c = tid % L::COLS, t1 = tid / L::COLS;
        const uint32_t n2 = rank * L::COLS + c;
        const float2* src = in + row * L::N + n2;
        TA::load_first(v, t1, [&](int i) { return ld_once_ca(src + i * L::N2); });
        TA::template passes<0>(v, smem + c * L::S1, table, t1, 0);
        const float2* wt = table + L::WT + n2;
        const float2 w0 = __ldg(wt + (E + t1) * L::N2);
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const float2 w = j == 0 ? w0 : cmul<false>(w0, __ldg(wt + j * L::N2));
            __stcg(out + n2 + (t1 + j * T1) * L::N2, cmul<INV>(v[TA::slot(j)], w));
        }
    }
    cluster_arrive();
    cluster_wait();   // the whole matrix is written
    {
        const int r = tid / TB::T, t2 = tid % TB::T;
        const float2* src = out + (rank * L::ROWS2 + r) * L::N2;
        TB::load_first(v, t2, [&](int i) { return __ldcg(src + i); });   // past L1, which may hold the input
        TB::template butterflies<0>(v, table + L::TW2, t2);
        TB::template put<0>(v, smem + r * L::S2, t2);
    }
    __syncthreads();
    cluster_arrive_relaxed();   // this CTA's rows are in shared memory: their addresses may be overwritten
    {
        const int r = tid % L::ROWS2, t2 = tid / L::ROWS2;
        TB::template get<1>(v, smem + r * L::S2, t2);
        TB::template butterflies<1>(v, table + L::TW2, t2);
        cluster_wait();
        pdl_trigger();
        float2* dst = out + rank * L::ROWS2 + r;
        TB::for_each_out(v, t2, [&](int k2, float2 x) { st_stream(dst + k2 * N1, cscale(x, scale)); });
    }
}

}  // namespace dev

namespace backend {

namespace {

// Whether the current device can hold a cluster beyond the portable size; allows the kernel that
// size.  Asked once per device and kernel.
bool wideClusterFits(const void* fn, unsigned cluster, int block, int smem) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return false;
    struct Answer {
        int device;
        const void* fn;
        bool fits;
    };
    static std::mutex mu;
    static std::vector<Answer> known;
    std::lock_guard<std::mutex> lock(mu);
    for (const Answer& a : known)
        if (a.device == device && a.fn == fn) return a.fits;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = cluster;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    const bool fits = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                      cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess && clusters > 0;
    cudaGetLastError();   // a refusal is an answer, not an error of the calls that follow
    known.push_back({device, fn, fits});
    return fits;
}

template <int N1>
size_t tableBytes() {
    using L = dev::LongDirect<N1>;
    if (L::C > 8)
        for (const void* fn : {(const void*)dev::k_long_direct<N1, false>, (const void*)dev::k_long_direct<N1, true>})
            if (!wideClusterFits(fn, L::C, L::NT, L::SMEM)) return 0;
    return L::TABLE * 8;
}

template <int N1>
int buildTable(float2* t, cudaStream_t s) {
    using L = dev::LongDirect<N1>;
    constexpr int c1 = dev::Sched<N1, L::E>::TWSIZE, c2 = dev::Sched<L::N2, L::E>::TWSIZE;
    dev::k_tw_stockham<N1, L::E><<<(c1 + 255) / 256, 256, 0, s>>>(t);
    dev::k_tw_stockham<L::N2, L::E><<<(c2 + 255) / 256, 256, 0, s>>>(t + L::TW2);
    for (int j = 0; j < L::E + L::T1; ++j)
        dev::k_tw_linear<<<1, L::N2, 0, s>>>(t + L::WT + j * L::N2, L::N2, j < L::E ? L::T1 * j : j - L::E, L::N);
    return (int)cudaGetLastError();
}

template <int N1>
int launchRows(const float2* in, float2* out, uint64_t batch, bool inverse, float scale, const float2* table,
               cudaStream_t s) {
    using L = dev::LongDirect<N1>;
    const void* fn = inverse ? (const void*)dev::k_long_direct<N1, true> : (const void*)dev::k_long_direct<N1, false>;
    if (batch > 0x7fffffffull / L::C) return (int)cudaErrorInvalidValue;
    if (L::C > 8 && !wideClusterFits(fn, L::C, L::NT, L::SMEM)) return (int)cudaErrorInvalidConfiguration;
    return (int)launchPdlCluster(fn, (unsigned)(batch * L::C), L::NT, L::SMEM, L::C, s, in, out, table, scale);
}

}  // namespace

size_t directTableBytes(uint32_t n) {
    switch (n) {
        case 32768: return tableBytes<128>();
        case 65536: return tableBytes<256>();
        default: return 0;
    }
}

int buildDirectTable(void* table, uint32_t n, void* stream) {
    float2* t = static_cast<float2*>(table);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    switch (n) {
        case 32768: return buildTable<128>(t, s);
        case 65536: return buildTable<256>(t, s);
        default: return (int)cudaErrorInvalidValue;
    }
}

int launchDirect(const void* in, void* out, uint32_t n, uint64_t batch, bool inverse, float scale,
                     const void* table, void* stream) {
    const float2* x = static_cast<const float2*>(in);
    float2* y = static_cast<float2*>(out);
    const float2* t = static_cast<const float2*>(table);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    switch (n) {
        case 32768: return launchRows<128>(x, y, batch, inverse, scale, t, s);
        case 65536: return launchRows<256>(x, y, batch, inverse, scale, t, s);
        default: return (int)cudaErrorInvalidValue;
    }
}

}  // namespace backend
}  // namespace bfly
