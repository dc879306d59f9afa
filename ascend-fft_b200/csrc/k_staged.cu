// Column FFTs of 2048 and 4096 points (k_cols' arguments), the next strip on its way while the
// current one computes.
//
// A strip of 8 columns of 2048 points or 4 of 4096 takes a whole register file (512 threads x 32
// values), so a CTA that loads, computes and stores leaves HBM idle while it computes.  Here one
// persistent CTA per SM copies its next strip into shared memory (cp.async, 128 KB) from the moment
// its current one is in registers.  The room for that comes from the exchanges, which send the real
// parts and then the imaginary parts through a buffer of half the size: the same bytes, one barrier
// more each.  2^25 points, GB/s, k_cols and this: NY = 2048: 3171 / 3573; 4096: 2073 / 2731.  At NY =
// 1024 (16 columns, 4928 / 4669) and for rows of 16384 (4350 / 3524) the strip's segments are wide
// enough for loads ahead into L2 to keep up, and the doubled shared-memory accesses lose.
#include <cuda_runtime.h>

#include "backend.h"
#include "fft_kernels.cuh"
#include "launch.cuh"

namespace bfly {
namespace dev {

// 16 bytes (the first `bytes` of them read, the rest zero) from global to shared memory.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <int N, int C>
struct Staged {
    static constexpr int E = 32, T = N / E, NT = T * C;
    // Exchange plane of one column: element i at i + i/32, columns PLANE floats apart with PLANE =
    // 32/C mod 32, so the C columns x 32/C threads of a warp hit 32 banks.
    static constexpr int LEN = N + N / 32;
    static constexpr int PLANE = LEN + (32 / C - LEN % 32 + 32) % 32;
    static constexpr int STAGE_BYTES = N * C * 8, SMEM = STAGE_BYTES + C * PLANE * 4;
    static_assert(N * C == 16384 && NT == 512, "one strip fills an SM's registers");
};

// Passes p.. of Team with its exchanges by halves through `plane`.
template <class TM, int E, int p>
__device__ __forceinline__ void staged_passes(float2 (&v)[E], float* plane, const float2* __restrict__ tw, int t) {
    using S = typename TM::S;
    TM::template butterflies<p>(v, tw, t);
    if constexpr (p < TM::P - 1) {
        constexpr int R = S::radix(p), B = E / R, Ns = S::ns(p);
        constexpr int R2 = S::radix(p + 1), B2 = E / R2, STEP2 = TM::T * B2;   // N / R2
        static_assert(R == 32 && (Ns == 1 || Ns % 32 == 0) && STEP2 % 32 == 0, "offsets add up with the padding");
        auto pad = [](int i) { return i + (i >> 5); };
        const int k = t & (Ns - 1), to = pad((t - k) * R + k), from = pad(t);
        static_assert(B == 1, "every pass but the last is one butterfly per thread");
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            if (half) __syncthreads();   // the real parts have been read
#pragma unroll
            for (int r = 0; r < R; ++r) plane[to + r * Ns + (r * Ns >> 5)] = half ? v[r].y : v[r].x;
            __syncthreads();
#pragma unroll
            for (int s = 0; s < B2; ++s)
#pragma unroll
                for (int r = 0; r < R2; ++r) {
                    const int off = s * TM::T + r * STEP2;
                    const float x = plane[from + off + (off >> 5)];
                    if (half) v[s * R2 + r].y = x;
                    else v[s * R2 + r].x = x;
                }
        }
        if constexpr (p + 1 < TM::P - 1) __syncthreads();   // the next exchange writes the plane again
        staged_passes<TM, E, p + 1>(v, plane, tw, t);
    }
}

// Strip b: columns [C (b mod colBlocks), ...) of matrix b / colBlocks.  Every row of a strip on a
// 16-byte boundary: `in` aligned, pitch and matStride even.
template <int N, int C, bool INV>
__global__ void __launch_bounds__(Staged<N, C>::NT, 1)
k_staged(const float2* in, float2* out, const float2* __restrict__ tw, uint64_t strips, uint32_t ncols, uint64_t pitch,
         uint64_t matStride, uint32_t colBlocks, float scale) {
    using G = Staged<N, C>;
    constexpr int E = G::E;
    using TM = Team<N, E, INV, kSyncBlock>;
    extern __shared__ __align__(16) unsigned char staged_smem[];
    float2* stage = reinterpret_cast<float2*>(staged_smem);
    float* plane = reinterpret_cast<float*>(staged_smem + G::STAGE_BYTES);
    pdl_wait();
    const int c = threadIdx.x % C, t = threadIdx.x / C;
    auto issue = [&](uint64_t b) {
        const uint32_t col = (uint32_t)(b % colBlocks) * C + 2 * (threadIdx.x % (C / 2));
        const int row = threadIdx.x / (C / 2);
        const int live = col + 1 < ncols ? 16 : col < ncols ? 8 : 0;
        const float2* src = in + b / colBlocks * matStride + (live ? col : 0u);
        float2* dst = stage + 2 * threadIdx.x;
#pragma unroll
        for (int i = 0; i < N; i += G::NT / (C / 2)) cp_async16(dst + i * C, src + (uint64_t)(row + i) * pitch, live);
    };
    uint64_t left = blockIdx.x;   // strip strips - 1 - left: the last matrix first, as k_cols
    if (left < strips) issue(strips - 1 - left);
    cp_async_commit();
    for (; left < strips; left += gridDim.x) {
        const uint64_t b = strips - 1 - left;
        cp_async_wait_all();
        __syncthreads();   // the strip is staged, and the last one's exchanges are over
        float2 v[E];
        TM::load_first(v, t, [&](int i) { return stage[i * C + c]; });
        __syncthreads();   // the stage is free
        if (left + gridDim.x < strips) issue(b - gridDim.x);
        cp_async_commit();
        staged_passes<TM, E, 0>(v, plane + c * G::PLANE, tw, t);
        const uint32_t col = (uint32_t)(b % colBlocks) * C + c;
        if (col < ncols) {
            float2* dst = out + b / colBlocks * matStride + col;
            TM::for_each_out(v, t, [&](int k, float2 x) { st_stream(dst + (uint64_t)k * pitch, cscale(x, scale)); });
        }
    }
}

}  // namespace dev

namespace backend {

namespace {
template <int N, int C, bool INV>
int launchStaged(const float2* in, float2* out, const float2* tw, uint64_t strips, uint32_t ncols, uint64_t pitch,
                 uint64_t matStride, uint32_t colBlocks, float scale, void* stream) {
    using G = dev::Staged<N, C>;
    auto* fn = dev::k_staged<N, C, INV>;
    if (int e = optInSharedMemory((const void*)fn, G::SMEM)) return e;
    return (int)launchPdlKernel(fn, dev::kSms, G::NT, G::SMEM, stream, in, out, tw, strips, ncols, pitch, matStride,
                                colBlocks, scale);
}
}  // namespace

// Taken from the first strip past one per SM on, with rows on 16-byte boundaries: with a second round
// most SMs have a next strip or idle through it either way.  us, k_cols of 16 values a thread and this:
// NY = 2048: 149 strips 24.1 / 21.6, 296 27.9 / 25.5, 297 36.2 / 32.3, 1100 103.7 / 89.4; 4096: 149 34.8 / 24.4,
// 296 39.5 / 28.4, 1100 156 / 108.  148 strips, k_cols both: 14.4 / 13.8 and 20.1 / 20.1.
bool launchColsStaged(const void* in, void* out, uint32_t ny, uint32_t ncols, uint64_t pitch, uint64_t matStride,
                      uint64_t mats, bool inverse, float scale, const void* tw, void* stream, int* rc) {
    if ((ny != 2048 && ny != 4096) || reinterpret_cast<uintptr_t>(in) % 16 || pitch % 2 || matStride % 2) return false;
    const uint32_t C = 16384 / ny, colBlocks = (ncols + C - 1) / C;
    const uint64_t strips = mats * colBlocks;
    if (strips <= dev::kSms) return false;
    const float2 *x = static_cast<const float2*>(in), *t = static_cast<const float2*>(tw);
    float2* y = static_cast<float2*>(out);
    static_assert(colsE(2048) == 32 && colsE(4096) == 32, "the table is that of 32 values a thread");
#define BFLY_CS(N, C, INV) launchStaged<N, C, INV>(x, y, t, strips, ncols, pitch, matStride, colBlocks, scale, stream)
    *rc = ny == 2048 ? (inverse ? BFLY_CS(2048, 8, true) : BFLY_CS(2048, 8, false))
                     : (inverse ? BFLY_CS(4096, 4, true) : BFLY_CS(4096, 4, false));
#undef BFLY_CS
    return true;
}

}  // namespace backend
}  // namespace bfly
