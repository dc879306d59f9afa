// Kernel templates of the batched FFT library (sm_100a).
//
//   k_c2c      batched C2C, one team per row, rows [batch][N] interleaved fp32.
//              Reference: Plan::run -> kfft_fwd (src/framework/butterfly.cpp:723-749,
//              src/ascendc/fft_radix2.cpp:51-481).
//   k_r2c      R2C as an N/2 complex FFT with the even/odd split fused into its epilogue;
//              writes the dense half spectrum [batch][N/2+1] complex (= [batch][N+2] floats).
//              Reference: Plan::runR2C -> kfft_fwd(n/2) + kfft_r2c_post
//              (butterfly.cpp:753-806, src/ascendc/fft_real.cpp:47-162).
//   k_c2r      C2R as an N/2 complex inverse with the Hermitian un-split fused into its
//              prologue; output includes 1/N like numpy.fft.irfft.
//              Reference: Plan::runC2R -> kfft_c2r_prep + kfft_fwd(xflip) + kfft_c2r_post
//              (butterfly.cpp:810-850, fft_real.cpp:167-267).
//   k_long_a / k_long_b
//              four-step long C2C, N = N1*N2: column FFTs of N1 with the W_N^(n2*k1) twiddle
//              fused into the store, then row FFTs of N2 with the transpose fused into the
//              store.  Reference: four-step chain of src/host/fft_check.cpp:289-308, 843-970,
//              kfft_lt_tr / kfft_lt_tw (src/ascendc/fft_long_lt_tr.inc:22-157,
//              src/ascendc/fft_long.cpp:82-140).
//   k_tw_*     twiddle tables computed in FP64 on the GPU and rounded to fp32.
#pragma once
#include "fft_core.cuh"

namespace bfly {
namespace dev {

// ------------------------------------------------------------------ C2C
// Minimum resident CTAs that keeps a kernel at <= 64 registers per thread: the budget at which
// the 512-thread single-transform kernels still fit two CTAs per SM.
__host__ __device__ constexpr int min_blocks_64regs(int threads) {
    return 65536 / (threads * 64) > 0 ? 65536 / (threads * 64) : 1;
}

// Minimum resident CTAs of a kernel with E complex values per thread: 64 registers up to E = 16,
// 128 for E = 32 (64 of them hold the values).
template <int E>
__host__ __device__ constexpr int min_blocks(int threads) {
    return E <= 16 ? min_blocks_64regs(threads) : 65536 / (threads * 128) > 0 ? 65536 / (threads * 128) : 1;
}

template <int N, int E, int ROWS, bool INV>
__global__ void __launch_bounds__((N / E) * ROWS, min_blocks<E>((N / E) * ROWS))
k_c2c(const float2* __restrict__ in, float2* __restrict__ out, const float2* __restrict__ tw,
      uint64_t batch, float scale) {
    constexpr int T = N / E;
    constexpr int S = smem_stride<N, E, false>();
    using TM = Team<N, E, INV, sync_kind(T, T * ROWS)>;
    extern __shared__ float2 smem[];
    pdl_wait();
    const int rl = threadIdx.x / T;
    const int t = threadIdx.x - rl * T;
    const uint64_t row = (uint64_t)blockIdx.x * ROWS + rl;
    const bool ok = row < batch;
    const float2* src = in + row * N;
    float2* dst = out + row * N;
    float2 v[E];
    TM::load_first(v, t, [&](int i) { return ok ? ld_once_ca(src + i) : make_float2(0.f, 0.f); });
    constexpr unsigned AHEAD = prefetch_ahead(min_blocks<E>(T * ROWS));
    // (rows of 32 fill the memory pipeline by themselves: 524288 of them 55.5 us with, 53.5 without)
    if (N > 32 && blockIdx.x + AHEAD < gridDim.x)
        prefetch_span<ROWS * N * 8, T * ROWS>(in + ((uint64_t)blockIdx.x + AHEAD) * (ROWS * N), in + batch * N);
    TM::template passes<0>(v, smem + rl * S, tw, t, rl);
    pdl_trigger();
    if (ok) TM::for_each_out(v, t, [&](int i, float2 x) { st_stream(dst + i, cscale(x, scale)); });
}

// ------------------------------------------------------------------ real split, by pairs
// x real [N] viewed as z[m] = x[2m] + i x[2m+1] (M = N/2), Z = FFT_M(z).  With b = conj(Z[M-k]),
//   e = (Z[k] + b)/2, o = (Z[k] - b)/(2i), p = W_N^k o:   X[k] = e + p, X[M-k] = conj(e - p)
// (same split as fft_real.cpp:9-14, :139-149), so bins k and M-k come from one pair of values.
__device__ __forceinline__ void r2c_pair(float2 a, float2 b, float2 w, float2& xk, float2& xm) {
    const float2 e = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y));
    const float2 o = make_float2(0.5f * (a.y + b.y), 0.5f * (b.x - a.x));
    const float2 p = cmul<false>(o, w);
    const float2 d = csub(e, p);
    xk = cadd(e, p);
    xm = make_float2(d.x, -d.y);
}
// The inverse of r2c_pair times 2 out_scale: Z[k] and Z[M-k] of
//   Z[k] = (Xk + conj Xm) + i (Xk - conj Xm) W_N^-k   (Xm = X[M-k]; k = 0 pairs X[0] with X[M]).
// Bins 0 and M: imaginary parts ignored (as in the real part extraction of kfft_c2r_post,
// fft_real.cpp:262-263), weight s_edge; the others s_int.
__device__ __forceinline__ void c2r_pair(float2 xk, float2 xm, bool edge, float2 w, float s_edge, float s_int,
                                         float out_scale, float2& zk, float2& zm) {
    if (edge) {
        xk = make_float2(xk.x * s_edge, 0.f);
        xm = make_float2(xm.x * s_edge, 0.f);
    } else {
        xk = cscale(xk, s_int);
        xm = cscale(xm, s_int);
    }
    const float2 ev = make_float2(xk.x + xm.x, xk.y - xm.y);
    // the scale rides on the twiddle and on the sums' multiply-adds
    const float2 od = cmul<true>(make_float2(xk.x - xm.x, xk.y + xm.y), cscale(w, out_scale));
    zk = make_float2(fmaf(ev.x, out_scale, -od.y), fmaf(ev.y, out_scale, od.x));
    zm = make_float2(fmaf(ev.x, out_scale, od.y), fmaf(-ev.y, out_scale, od.x));
}

// The split of one row held by a team (TM = Team<M, E, ...>), pairs (k, M-k) with k = t + j T,
// j < E/2, handled by thread t: it holds the values at k itself, and those at M-k belong to
// thread T - t, so only the upper half of the row crosses shared memory (E/2 stores and loads a
// thread in place of E and 2 E), and each pair shares its twiddle and its sums.  Every bin on its
// own / by pairs, ncu: k_istft n = 512, 60008 frames, 72.7 / 57.4 us; k_stft n = 1024, 20032
// frames, 53.7 / 48.6 us; k_c2r n = 256, 32768 rows, 18.6 / 16.3 us.
template <class TM, int M, int E>
struct RealSplit {
    static constexpr int T = M / E, H = E / 2;
    // v: a finished transform, as Team leaves it; emit(k, X[k], k is 0 or M) for every bin
    // k <= M of the team's row.  `sm` must be free once the team has synchronised.
    template <class Emit>
    static __device__ __forceinline__ void store(float2 (&v)[E], float2* sm, const float2* __restrict__ twr, int t,
                                                 int row, Emit&& emit) {
        float2 lo[H], w[H], mid;
#pragma unroll
        for (int j = 0; j < H; ++j) w[j] = __ldg(twr + t + j * T);   // in flight over the exchange
        TM::sync(row);
        TM::for_each_out(v, t, [&](int i, float2 x) {
            if (i >= t + H * T) sm[spad(i - M / 2)] = x;   // i - t is a compile-time multiple of T
        });
#pragma unroll
        for (int j = 0; j < H; ++j) lo[j] = v[TM::slot(j)];
        mid = v[TM::slot(H)];
        TM::sync(row);
        if (t == 0) emit(M / 2, cconj(mid), false);   // bin M/2 pairs with itself
#pragma unroll
        for (int j = 0; j < H; ++j) {
            const int k = t + j * T;
            const float2 b = j == 0 && t == 0 ? lo[0] : sm[spad(M / 2 - k)];
            float2 xk, xm;
            r2c_pair(lo[j], b, w[j], xk, xm);
            emit(k, xk, j == 0 && t == 0);
            emit(M - k, xm, j == 0 && t == 0);
        }
    }

    // Bins of one row as loaded (all loads in flight before the first use).
    struct Bins {
        float2 lo[H], hi[H], mid;
    };
    template <class Load>
    static __device__ __forceinline__ Bins bins(int t, Load&& load) {
        Bins x;
#pragma unroll
        for (int j = 0; j < H; ++j) x.lo[j] = load(t + j * T);
#pragma unroll
        for (int j = 0; j < H; ++j) x.hi[j] = load(M - t - j * T);
        x.mid = t == 0 ? load(M / 2) : make_float2(0.f, 0.f);
        return x;
    }
    // Z of the loaded bins into v, as pass 0 of the team wants it: element t + j T in v[j].  `sm`
    // must be free when called and is free again on return.
    static __device__ __forceinline__ void load(float2 (&v)[E], float2* sm, const float2* __restrict__ twr, int t,
                                                int row, const Bins& x, float s_edge, float s_int, float out_scale) {
        static_assert(TM::S::radix(0) == E, "pass 0 takes element t + r T in v[r]");
#pragma unroll
        for (int j = 0; j < H; ++j) {
            const int k = t + j * T;
            float2 zm;
            c2r_pair(x.lo[j], x.hi[j], j == 0 && t == 0, __ldg(twr + k), s_edge, s_int, out_scale, v[j], zm);
            if (j > 0 || t > 0) sm[spad(M / 2 - k)] = zm;
        }
        if (t == 0) {   // bin M/2 pairs with itself
            const float c = 2.f * s_int * out_scale;
            sm[0] = make_float2(c * x.mid.x, -c * x.mid.y);
        }
        TM::sync(row);
#pragma unroll
        for (int j = H; j < E; ++j) v[j] = sm[spad(t + (j - H) * T)];
        TM::sync(row);
    }
};

// ------------------------------------------------------------------ R2C
// Optional per-bin weights (WEIGHTED): X[k] *= (k==0||k==M ? s_edge : s_int); used by the
// adjoint of C2R.
template <int N, int E, int ROWS, bool WEIGHTED>
__global__ void __launch_bounds__((N / 2 / E) * ROWS, min_blocks_64regs((N / 2 / E) * ROWS))
k_r2c(const float2* __restrict__ in, float2* __restrict__ out, const float2* __restrict__ tw,
      const float2* __restrict__ twr, uint64_t batch, float s_edge, float s_int) {
    constexpr int M = N / 2;
    constexpr int T = M / E;
    constexpr int S = smem_stride<M, E, false>();
    using TM = Team<M, E, false, sync_kind(T, T * ROWS)>;
    extern __shared__ float2 smem[];
    pdl_wait();
    const int rl = threadIdx.x / T;
    const int t = threadIdx.x - rl * T;
    const uint64_t row = (uint64_t)blockIdx.x * ROWS + rl;
    const bool ok = row < batch;
    const float2* src = in + row * M;
    float2* dst = out + row * (M + 1);
    float2* sm = smem + rl * S;
    float2 v[E];
    TM::load_first(v, t, [&](int i) { return ok ? ld_stream(src + i) : make_float2(0.f, 0.f); });
    constexpr unsigned AHEAD = prefetch_ahead(min_blocks_64regs(T * ROWS));
    if (blockIdx.x + AHEAD < gridDim.x)
        prefetch_span<ROWS * M * 8, T * ROWS>(in + ((uint64_t)blockIdx.x + AHEAD) * (ROWS * M), in + batch * M);
    TM::template passes<0>(v, sm, tw, t, rl);
    pdl_trigger();
    RealSplit<TM, M, E>::store(v, sm, twr, t, rl, [&](int k, float2 X, bool edge) {
        if constexpr (WEIGHTED) X = cscale(X, edge ? s_edge : s_int);
        if (ok) st_stream(dst + k, X);
    });
}

// ------------------------------------------------------------------ C2R
// X half spectrum [M+1] (M = N/2) to Z by pairs of bins, z = IDFT_M(Z),
//   x[2m] = Re z[m], x[2m+1] = Im z[m].   out_scale = 1/N gives numpy.fft.irfft.
template <int N, int E, int ROWS>
__global__ void __launch_bounds__((N / 2 / E) * ROWS, min_blocks_64regs((N / 2 / E) * ROWS))
k_c2r(const float2* __restrict__ in, float2* __restrict__ out, const float2* __restrict__ tw,
      const float2* __restrict__ twr, uint64_t batch, float s_edge, float s_int, float out_scale) {
    constexpr int M = N / 2;
    constexpr int T = M / E;
    constexpr int S = smem_stride<M, E, false>();
    using TM = Team<M, E, true, sync_kind(T, T * ROWS)>;
    extern __shared__ float2 smem[];
    pdl_wait();
    const int rl = threadIdx.x / T;
    const int t = threadIdx.x - rl * T;
    const uint64_t row = (uint64_t)blockIdx.x * ROWS + rl;
    const bool ok = row < batch;
    const float2* src = in + row * (M + 1);
    float2* dst = out + row * M;
    float2* sm = smem + rl * S;
    using RS = RealSplit<TM, M, E>;
    const auto x = RS::bins(t, [&](int k) { return ok ? ld_stream(src + k) : make_float2(0.f, 0.f); });
    constexpr unsigned AHEAD = prefetch_ahead(min_blocks_64regs(T * ROWS));
    if (blockIdx.x + AHEAD < gridDim.x)
        prefetch_span<ROWS * (M + 1) * 8, T * ROWS>(in + ((uint64_t)blockIdx.x + AHEAD) * (ROWS * (M + 1)),
                                                    in + batch * (M + 1));
    float2 v[E];
    RS::load(v, sm, twr, t, rl, x, s_edge, s_int, out_scale);
    TM::template passes<0>(v, sm, tw, t, rl);
    pdl_trigger();
    if (ok) TM::for_each_out(v, t, [&](int i, float2 x) { st_stream(dst + i, x); });
}

// ------------------------------------------------------------------ column FFTs
// NY-point FFTs down the columns of a batch of row-major matrices:
//   in[m*matStride + i*pitch + col], i < NY, col < ncols, m < gridDim.x / colBlocks.
// Serves the column pass of a 2-D transform ([batch][ny][nx]: pitch = nx, matStride = ny*nx)
// and transforms along a middle axis of a contiguous [outer][n][inner] array (pitch = inner).
// C consecutive columns per CTA with the column index fastest across threads, so every row
// access is one C*8-byte segment; columns at or past ncols compute on zeros and store nothing.
// (Numbering the columns of all matrices through, so that only the last CTA has idle columns, gave
// nothing at 129 columns of 256 and cost 7 % at 1024 of 1024: the division delays the loads.)
// Every load precedes the CTA's first __syncthreads and every store follows its last, so
// in == out is allowed.
template <int NY, int E, int C, bool INV>
__global__ void __launch_bounds__((NY / E) * C, min_blocks<E>((NY / E) * C))
k_cols(const float2* __restrict__ in, float2* __restrict__ out, const float2* __restrict__ tw,
       uint32_t ncols, uint64_t pitch, uint64_t matStride, uint32_t colBlocks, float scale) {
    constexpr int S = smem_stride<NY, E, true>();
    using TM = Team<NY, E, INV, kSyncBlock>;
    static_assert(TM::P >= 2, "in-place safety needs a barrier between loads and stores");
    extern __shared__ float2 smem[];
    pdl_wait();
    const int c = threadIdx.x % C;
    const int t = threadIdx.x / C;
    // from the last matrix to the first: a 2-D transform's row pass has left the last ones in L2
    // (1024 x 1024 x 16: 103.6 -> 100.0 us for both passes)
    const uint32_t blk = gridDim.x - 1 - blockIdx.x;
    const uint64_t m = blk / colBlocks;
    const uint32_t col = (blk % colBlocks) * C + c;
    const bool live = col < ncols;
    const float2* src = in + m * matStride + (live ? col : 0u);
    float2* dst = out + m * matStride + col;
    float2 v[E];
    TM::load_first(v, t, [&](int i) { return live ? ld_once_ca(src + (size_t)i * pitch) : make_float2(0.f, 0.f); });
    constexpr unsigned AHEAD = prefetch_ahead(min_blocks<E>((NY / E) * C));
    if (blockIdx.x + AHEAD < gridDim.x) {   // the first line of each row segment of a later strip
        const uint32_t b = blk - AHEAD;
        const float2* next = in + (uint64_t)(b / colBlocks) * matStride + (b % colBlocks) * C;
#pragma unroll
        for (int i = 0; i < NY; i += (NY / E) * C)
            if (i + (int)threadIdx.x < NY) prefetch_l2(next + (size_t)(i + threadIdx.x) * pitch);
    }
    TM::template passes<0>(v, smem + c * S, tw, t, 0);
    pdl_trigger();
    if (live) TM::for_each_out(v, t, [&](int k, float2 x) { st_stream(dst + (size_t)k * pitch, cscale(x, scale)); });
}

// ------------------------------------------------------------------ four-step long C2C
// x[b][N2*n1 + n2] -> (pass A) y[b][N2*k1 + n2] = W_N^(n2*k1) * FFT_N1 over n1
//                  -> (pass B) X[b][k1 + N1*k2]  = FFT_N2 over n2 of y[b][N2*k1 + :]
// W_N^m for m < N is assembled from two FP64-built tables: tlo[m & 255] * thi[m >> 8].

// Pass A: C consecutive columns per CTA, column index fastest across threads so each global
// access is C consecutive complex values (C*8 bytes).
template <int N1, int E, int C, bool INV>
__global__ void __launch_bounds__((N1 / E) * C, 3)
k_long_a(const float2* __restrict__ in, float2* __restrict__ out, const float2* __restrict__ tw,
         const float2* __restrict__ tlo, const float2* __restrict__ thi, uint64_t batch, int logN2) {
    constexpr int T = N1 / E;
    constexpr int S = smem_stride<N1, E, true>();
    using TM = Team<N1, E, INV, kSyncBlock>;
    extern __shared__ float2 smem[];
    const int c = threadIdx.x % C;
    const int t = threadIdx.x / C;
    const uint32_t N2 = 1u << logN2;
    const uint32_t colBlocks = N2 / C;
    const uint64_t b = blockIdx.x / colBlocks;
    const uint32_t n2 = (blockIdx.x % colBlocks) * C + c;
    const uint64_t N = (uint64_t)N1 << logN2;
    const float2* src = in + b * N + n2;
    float2* dst = out + b * N + n2;
    (void)batch;
    float2 v[E];
    TM::run(v, smem + c * S, tw, t, 0, [&](int i) { return ld_once_ca(src + ((size_t)i << logN2)); });
    TM::for_each_out(v, t, [&](int k1, float2 x) {
        const uint32_t m = n2 * (uint32_t)k1;
        const float2 w = cmul<false>(__ldg(thi + (m >> 8)), __ldg(tlo + (m & 255u)));
        st_stream(dst + ((size_t)k1 << logN2), cmul<INV>(x, w));
    });
}

// Pass B: C consecutive rows per CTA; loads row-contiguous, FFT, then a shared-memory
// transpose so the stride-N1 output is written as C consecutive complex values per k2.
template <int N2, int E, int C, bool INV>
__global__ void __launch_bounds__((N2 / E) * C)
k_long_b(const float2* __restrict__ in, float2* __restrict__ out, const float2* __restrict__ tw,
         uint64_t batch, int logN1, float scale) {
    constexpr int T = N2 / E;
    constexpr int S = smem_stride<N2, E, false>();
    using TM = Team<N2, E, INV, sync_kind(T, T * C)>;
    extern __shared__ float2 smem[];
    const int rl = threadIdx.x / T;
    const int t = threadIdx.x - rl * T;
    const uint32_t N1 = 1u << logN1;
    const uint32_t rowBlocks = N1 / C;
    const uint64_t b = blockIdx.x / rowBlocks;
    const uint32_t k1_0 = (blockIdx.x % rowBlocks) * C;
    const uint64_t N = (uint64_t)N2 << logN1;
    const float2* src = in + b * N + (uint64_t)(k1_0 + rl) * N2;
    float2* sm = smem + rl * S;
    (void)batch;
    float2 v[E];
    TM::run(v, sm, tw, t, rl, [&](int i) { return ld_once_ca(src + i); });
    __syncthreads();
    TM::for_each_out(v, t, [&](int i, float2 x) { sm[spad(i)] = x; });
    __syncthreads();
    float2* dst = out + b * N + k1_0;
    for (int idx = threadIdx.x; idx < C * N2; idx += blockDim.x) {
        const int c = idx % C;
        const int k2 = idx / C;
        st_stream(dst + c + ((size_t)k2 << logN1), cscale(smem[c * S + spad(k2)], scale));
    }
}

// ------------------------------------------------------------------ FP64 twiddle builders
// Stockham table of Sched<N,E>: pass p >= 1 holds exp(-2*pi*i*r*k/(Ns*R)) at
// twoff(p) + (r-1)*Ns + k.  The only FP64 arithmetic in the library.
template <int N, int E>
__global__ void k_tw_stockham(float2* __restrict__ tw) {
    using Sd = Sched<N, E>;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Sd::TWSIZE) return;
    int p = 1;
    while (p + 1 < Sd::P && i >= Sd::twoff(p + 1)) ++p;
    const int rel = i - Sd::twoff(p);
    const int ns = Sd::ns(p);
    const int R = Sd::radix(p);
    const int r = rel / ns + 1;
    const int k = rel % ns;
    double s, c;
    sincospi(-2.0 * (double)(r * k) / (double)(ns * R), &s, &c);
    tw[i] = make_float2((float)c, (float)s);
}

// tw[i] = exp(-2*pi*i*(i*stride)/N), i < count.
static __global__ void k_tw_linear(float2* __restrict__ tw, int count, long long stride, long long n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const long long m = ((long long)i * stride) % n;
    double s, c;
    sincospi(-2.0 * (double)m / (double)n, &s, &c);
    tw[i] = make_float2((float)c, (float)s);
}

}  // namespace dev
}  // namespace bfly
