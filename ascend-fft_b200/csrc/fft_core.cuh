// Device core of the batched power-of-two FFT: in-register DFTs of size 2/4/8/16, the
// Stockham autosort pass schedule, and the "team" FFT in which T = N/E threads each hold
// E complex values and exchange them through padded shared memory between passes.
//
// Transform computed (forward): X[k] = sum_j x[j] * exp(-2*pi*i*j*k/N), unnormalised, the
// convention of the reference's Plan::run (src/framework/butterfly.cpp:723-749, kernel
// src/ascendc/fft_radix2.cpp:51).  INV flips the exponent sign (unnormalised inverse).
//
// Pass p of the schedule has radix R_p and Ns_p = R_0*...*R_{p-1}.  Butterfly j (0 <= j < N/R_p)
// with k = j mod Ns_p reads x[j + r*N/R_p] (r < R_p), multiplies element r by
// exp(-2*pi*i*r*k/(Ns_p*R_p)), applies DFT_{R_p} and writes y[(j-k)*R_p + k + r*Ns_p].
// Reads are unit-stride across threads in every pass, and the last pass writes
// y[j + r*N/R_last], so first-pass loads and last-pass stores are coalesced global accesses.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace bfly {
namespace dev {

// ------------------------------------------------------------------ complex helpers
// Sums, differences and real multiples of a complex value act on both halves alike, so they are
// issued as packed two-wide fp32 instructions (one per complex value; each half rounds as the
// scalar instruction does).  Products by +-i and by a general twiddle cross the halves and stay
// scalar: packing them would spend the saved instruction on register moves.
__device__ __forceinline__ float2 f2(float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.f), a); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return __fmul2_rn(a, f2(s)); }
__device__ __forceinline__ float2 cfma(float2 a, float s, float2 c) { return __ffma2_rn(a, f2(s), c); }   // s a + c
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
// a + s*d*w and a - s*d*w with w = -i (forward) or +i (INV), s a constant.
template <bool INV>
__device__ __forceinline__ void add_sub_i(float2 a, float2 d, float s, float2& plus, float2& minus) {
    const float h = INV ? -s : s;
    plus = make_float2(fmaf(h, d.y, a.x), fmaf(-h, d.x, a.y));
    minus = make_float2(fmaf(-h, d.y, a.x), fmaf(h, d.x, a.y));
}
template <bool INV>
__device__ __forceinline__ void add_sub_i(float2 a, float2 d, float2& plus, float2& minus) {
    const float2 p = make_float2(a.x + d.y, a.y - d.x), m = make_float2(a.x - d.y, a.y + d.x);
    plus = INV ? m : p;
    minus = INV ? p : m;
}
// a * w (CONJ=false) or a * conj(w) (CONJ=true)
template <bool CONJ>
__device__ __forceinline__ float2 cmul(float2 a, float2 w) {
    if (CONJ) return make_float2(fmaf(a.x, w.x, a.y * w.y), fmaf(a.y, w.x, -(a.x * w.y)));
    return make_float2(fmaf(a.x, w.x, -(a.y * w.y)), fmaf(a.x, w.y, a.y * w.x));
}

// Multiply by exp(-2*pi*i*q/16) for a compile-time q (forward direction). Exact special cases
// for multiples of pi/4; the remaining angles use correctly rounded constants.
template <int Q>
__device__ __forceinline__ float2 rot16(float2 a) {
    constexpr int q = ((Q % 16) + 16) % 16;
    constexpr float H = 0.70710678118654752440f;   // sqrt(1/2)
    constexpr float C1 = 0.92387953251128675613f;  // cos(pi/8)
    constexpr float S1 = 0.38268343236508977173f;  // sin(pi/8)
    if constexpr (q == 0) return a;
    else if constexpr (q == 4) return make_float2(a.y, -a.x);
    else if constexpr (q == 8) return make_float2(-a.x, -a.y);
    else if constexpr (q == 12) return make_float2(-a.y, a.x);
    else if constexpr (q == 2) return make_float2(H * (a.x + a.y), H * (a.y - a.x));
    else if constexpr (q == 6) return make_float2(H * (a.y - a.x), -H * (a.x + a.y));
    else if constexpr (q == 10) return make_float2(-H * (a.x + a.y), H * (a.x - a.y));
    else if constexpr (q == 14) return make_float2(H * (a.x - a.y), H * (a.x + a.y));
    else {
        // cos/sin of 2*pi*q/16 for odd q
        constexpr float c = (q == 1 || q == 15) ? C1 : (q == 3 || q == 13) ? S1
                          : (q == 5 || q == 11) ? -S1 : -C1;
        constexpr float s = (q == 1 || q == 7) ? S1 : (q == 3 || q == 5) ? C1
                          : (q == 9 || q == 15) ? -S1 : -C1;
        // a * (c - i s)
        return make_float2(fmaf(a.x, c, a.y * s), fmaf(a.y, c, -(a.x * s)));
    }
}

// a * exp(sign*2*pi*i*e/R), sign = -1 forward, +1 inverse; R divides 16.
template <int E, int R, bool INV>
__device__ __forceinline__ float2 rot(float2 a) {
    constexpr int q = (16 / R) * E;
    if constexpr (INV) return rot16<16 - (q % 16)>(a);
    else return rot16<q>(a);
}

// ------------------------------------------------------------------ in-register DFTs
// Natural order in and out: v[k] <- sum_m v[m] * exp(sign*2*pi*i*m*k/R).
template <int R, bool INV> struct DFT;

template <bool INV> struct DFT<1, INV> {
    static __device__ __forceinline__ void run(float2*) {}
};

template <bool INV> struct DFT<2, INV> {
    static __device__ __forceinline__ void run(float2* v) {
        const float2 a = v[0];
        v[0] = cadd(a, v[1]);
        v[1] = csub(a, v[1]);
    }
};

template <bool INV> struct DFT<4, INV> {
    static __device__ __forceinline__ void run(float2* v) {
        const float2 t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
        const float2 t2 = cadd(v[1], v[3]), t3 = csub(v[1], v[3]);
        v[0] = cadd(t0, t2);
        v[2] = csub(t0, t2);
        add_sub_i<INV>(t1, t3, v[1], v[3]);
    }
};

// DFT4 of (a0, w a1, w^2 a2, w^3 a3) for w = W_8: the eighth roots are a sum and a difference
// times sqrt(1/2), and that factor rides on the sums after them as a multiply-add.
template <bool INV>
__device__ __forceinline__ void dft4_w8(float2* v) {
    constexpr float H = 0.70710678118654752440f;   // sqrt(1/2)
    float2 t0, t1;
    add_sub_i<INV>(v[0], v[2], t0, t1);   // W_8^2 = -i (INV: +i)
    // H*u1 = W_8 a1, H*u3 = W_8^3 a3
    const float2 u1 = INV ? make_float2(v[1].x - v[1].y, v[1].x + v[1].y) : make_float2(v[1].x + v[1].y, v[1].y - v[1].x);
    const float2 u3 = INV ? make_float2(-v[3].x - v[3].y, v[3].x - v[3].y) : make_float2(v[3].y - v[3].x, -v[3].x - v[3].y);
    const float2 s = cadd(u1, u3), d = csub(u1, u3);
    v[0] = cfma(s, H, t0);
    v[2] = cfma(s, -H, t0);
    add_sub_i<INV>(t1, d, H, v[1], v[3]);
}

// DFT4 of (a0, w a1, w^2 a2, w^3 a3) for w = W_16^K, K = 1 or 3 (w^2 an odd eighth root).
template <int K, bool INV>
__device__ __forceinline__ void dft4_w16(float2* v) {
    constexpr float H = 0.70710678118654752440f;
    const float2 a = rot<K, 16, INV>(v[1]), b = rot<3 * K, 16, INV>(v[3]);
    const float x = v[2].x, y = v[2].y;   // H*u = W_16^(2K) a2
    const float2 u = K == 1 ? (INV ? make_float2(x - y, x + y) : make_float2(x + y, y - x))
                            : (INV ? make_float2(-x - y, x - y) : make_float2(y - x, -x - y));
    const float2 t0 = cfma(u, H, v[0]), t1 = cfma(u, -H, v[0]);
    const float2 t2 = cadd(a, b), t3 = csub(a, b);
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    add_sub_i<INV>(t1, t3, v[1], v[3]);
}

// 8 = 2 x 4 and 16 = 4 x 4 Cooley-Tukey, input n = B n1 + n2, output k = k1 + A k2; the inner
// twiddles W_R^(n2 k1) are part of the second stage's butterflies.  A DFT16 is 106 fp32
// instructions (160 with scalar sums): k_c2c n = 4096 executes 21.9 M against 29.1 M per 2^24
// points, with the constant exchange offsets of Team::at_off.
template <bool INV> struct DFT<8, INV> {
    static __device__ __forceinline__ void run(float2* v) {
        float2 a[4], b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            a[j] = cadd(v[j], v[4 + j]);
            b[j] = csub(v[j], v[4 + j]);
        }
        DFT<4, INV>::run(a);
        dft4_w8<INV>(b);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[2 * k] = a[k];
            v[2 * k + 1] = b[k];
        }
    }
};
template <bool INV>
__device__ __forceinline__ void dft16_rows(float2 (&y)[4][4], float2* v) {   // y[k1][n2]
    DFT<4, INV>::run(y[0]);
    dft4_w16<1, INV>(y[1]);
    dft4_w8<INV>(y[2]);
    dft4_w16<3, INV>(y[3]);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
        for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = y[k1][k2];
}
template <bool INV> struct DFT<16, INV> {
    static __device__ __forceinline__ void run(float2* v) {
        float2 y[4][4];
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2) {
            float2 c[4] = {v[n2], v[4 + n2], v[8 + n2], v[12 + n2]};
            DFT<4, INV>::run(c);
#pragma unroll
            for (int k1 = 0; k1 < 4; ++k1) y[k1][n2] = c[k1];
        }
        dft16_rows<INV>(y, v);
    }
};

// a * exp(-+2*pi*i*Q/32), Q compile-time.
template <int Q, bool INV>
__device__ __forceinline__ float2 rot32(float2 a) {
    if constexpr (Q % 2 == 0) {
        return rot<Q / 2, 16, INV>(a);
    } else {
        constexpr int q = Q % 32;
        constexpr int m = q % 16 > 8 ? 16 - q % 16 : q % 16;   // angle folded into the first quadrant
        constexpr float C1 = 0.98078528040323044913f, S1 = 0.19509032201612826785f;   // cos, sin of pi/16
        constexpr float C3 = 0.83146961230254523708f, S3 = 0.55557023301960222474f;   // of 3 pi/16
        constexpr float c0 = m == 1 ? C1 : m == 3 ? C3 : m == 5 ? S3 : S1;
        constexpr float s0 = m == 1 ? S1 : m == 3 ? S3 : m == 5 ? C3 : C1;
        constexpr float c = (q < 8 || q > 24) ? c0 : -c0;
        constexpr float s = (q < 16) != INV ? s0 : -s0;
        return make_float2(fmaf(a.x, c, a.y * s), fmaf(a.y, c, -(a.x * s)));
    }
}
template <int K1, bool INV, int N2 = 1>
__device__ __forceinline__ void twiddle32(float2* v) {   // v[n2] *= W_32^(K1 n2), n2 < 8
    if constexpr (N2 < 8) {
        v[N2] = rot32<K1 * N2, INV>(v[N2]);
        twiddle32<K1, INV, N2 + 1>(v);
    }
}
// 32 = 4 x 8.
template <bool INV>
__device__ __forceinline__ void dft32_rows(float2 (&y)[4][8], float2* v) {   // y[k1][n2]
    twiddle32<1, INV>(y[1]);
    twiddle32<2, INV>(y[2]);
    twiddle32<3, INV>(y[3]);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
        DFT<8, INV>::run(y[k1]);
#pragma unroll
        for (int k2 = 0; k2 < 8; ++k2) v[k1 + 4 * k2] = y[k1][k2];
    }
}
template <bool INV> struct DFT<32, INV> {
    static __device__ __forceinline__ void run(float2* v) {
        float2 y[4][8];
#pragma unroll
        for (int n2 = 0; n2 < 8; ++n2) {
            float2 c[4] = {v[n2], v[8 + n2], v[16 + n2], v[24 + n2]};
            DFT<4, INV>::run(c);
#pragma unroll
            for (int k1 = 0; k1 < 4; ++k1) y[k1][n2] = c[k1];
        }
        dft32_rows<INV>(y, v);
    }
};

// DFT of R = 16 or 32 values whose upper half is zero, whatever v holds there.
template <int R, bool INV>
__device__ __forceinline__ void dft_low(float2* v) {
    constexpr int B = R / 4;
    float2 y[4][B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
        const float2 a = v[n2], b = v[B + n2];
        y[0][n2] = cadd(a, b);
        y[2][n2] = csub(a, b);
        add_sub_i<INV>(a, b, y[1][n2], y[3][n2]);
    }
    if constexpr (R == 16) dft16_rows<INV>(y, v);
    else dft32_rows<INV>(y, v);
}

// ------------------------------------------------------------------ pass schedule
// Greedy radix schedule: radix E while it divides the remaining length, remainder last.
// Shared with the host twiddle-table builder through the same constexpr functions.
__host__ __device__ constexpr int ilog2c(int n) { return n <= 1 ? 0 : 1 + ilog2c(n >> 1); }

template <int N, int E>
struct Sched {
    static_assert((N & (N - 1)) == 0 && N >= 2, "N must be a power of two");
    static_assert(E == 2 || E == 4 || E == 8 || E == 16 || E == 32, "E must be 2,4,8,16,32");
    static_assert(N >= E, "N must be >= E");
    static constexpr int T = N / E;                      // threads per transform
    static constexpr int LOGN = ilog2c(N), LOGE = ilog2c(E);
    static constexpr int P = (LOGN + LOGE - 1) / LOGE;   // number of passes
    __host__ __device__ static constexpr int radix(int p) {
        return (p < P - 1) ? E : (1 << (LOGN - (P - 1) * LOGE));
    }
    __host__ __device__ static constexpr int ns(int p) {  // product of radices before p
        int v = 1;
        for (int q = 0; q < p; ++q) v *= radix(q);
        return v;
    }
    // float2 offset of pass p's twiddles in the table: (R_p - 1) * Ns_p entries per pass p >= 1
    __host__ __device__ static constexpr int twoff(int p) {
        int off = 0;
        for (int q = 1; q < p; ++q) off += (radix(q) - 1) * ns(q);
        return off;
    }
    static constexpr int TWSIZE = twoff(P);
};

// Shared-memory layout: one pad element per 16 (8-byte words => 16 banks of a half-warp).
__host__ __device__ constexpr int spad(int i) { return i + (i >> 4); }

// Row stride (in float2) of one transform's exchange buffer.
//  ROW_FAST=false: lanes of a half-warp are consecutive threads t of the same transform
//    (or, when T < 16, of 16/T consecutive transforms): stride = T mod 16 keeps the
//    transforms in disjoint bank groups.
//  ROW_FAST=true : lanes are consecutive transforms with the same t: an odd stride spreads
//    them over all 16 banks whatever the within-transform index.
template <int N, int E, bool ROW_FAST>
__host__ __device__ constexpr int smem_stride() {
    constexpr int base = spad(N - 1) + 1;
    constexpr int T = N / E;
    if constexpr (ROW_FAST) return base | 1;
    else if constexpr (T < 16) return base + ((T - (base % 16)) % 16 + 16) % 16;
    else return base;
}

// ------------------------------------------------------------------ synchronisation
// How the threads of one transform synchronise between passes:
//   kSyncWarp   the transform lives inside one warp (T <= 32)
//   kSyncNamed  the transform spans whole warps of a larger CTA: named barrier 1 + row, T threads
//   kSyncBlock  the transform is the whole CTA
enum SyncKind { kSyncWarp = 0, kSyncNamed = 1, kSyncBlock = 2 };

template <int SYNC>
__device__ __forceinline__ void team_sync(int row, int nthreads) {
    if constexpr (SYNC == kSyncWarp) {
        __syncwarp();
    } else if constexpr (SYNC == kSyncNamed) {
        asm volatile("bar.sync %0, %1;" ::"r"(1 + row), "r"(nthreads) : "memory");
    } else {
        __syncthreads();
    }
}

// Sync policy for a transform of T threads in a CTA of `ctaThreads`.
__host__ __device__ constexpr int sync_kind(int T, int ctaThreads) {
    return T <= 32 ? kSyncWarp : (T < ctaThreads ? kSyncNamed : kSyncBlock);
}

// ------------------------------------------------------------------ team FFT
// One transform of length N held by T = N/E threads, E complex values per thread.
// Thread t, slot s (< E/R), element r of pass p covers butterfly j = t + s*T.
// On return, v[s*R_last + r] holds output element t + s*T + r*(N/R_last) (natural order).
// `sm` is this transform's exchange buffer (smem_stride<> float2), `tw` the Stockham
// twiddle table of Sched<N,E> (TWSIZE entries, pass p at twoff(p)), `load(i)` yields input
// element i.  SYNC selects the barrier (see team_sync); `row` is the transform's index in its
// CTA (named-barrier id - 1).  ESTRIDE selects the exchange layout: 0 = element i at
// sm[spad(i)] (padded, threads of one transform across lanes); s > 0 = element i at sm[i*s]
// (transforms across lanes, e.g. the columns of a tile staged densely by TMA).
template <int N, int E, bool INV, int SYNC, int ESTRIDE = 0>
struct Team {
    using S = Sched<N, E>;
    static constexpr int T = S::T;
    static constexpr int P = S::P;

    static __device__ __forceinline__ int at(int i) {
        if constexpr (ESTRIDE == 0) return spad(i);
        else return i * ESTRIDE;
    }

    // Where at(base + off) lies, given a = at(base): the padding adds up exactly when off is a
    // multiple of 16, or base is one (16 | STEP, the divisor that the caller knows of base), so the
    // elements of a butterfly are constant offsets from one address.  Other cases recompute.
    template <int OFFSTEP, int STEP>
    static __device__ __forceinline__ int at_off(int base, int a, int off) {
        if constexpr (ESTRIDE != 0) return a + off * ESTRIDE;
        else if constexpr (OFFSTEP % 16 == 0 || STEP % 16 == 0) return a + spad(off);
        else return spad(base + off);
    }
    // Element r of butterfly j as pass p stores it, and as pass p loads it.
    template <int p>
    static __device__ __forceinline__ int out_at(int base, int a, int r) {
        return at_off<S::ns(p), S::ns(p) == 1 ? S::radix(p) : 1>(base, a, r * S::ns(p));
    }
    template <int p>
    static __device__ __forceinline__ int in_at(int j, int a, int r) {
        return at_off<N / S::radix(p), 1>(j, a, r * (N / S::radix(p)));
    }

    static __device__ __forceinline__ void sync(int row) { team_sync<SYNC>(row, T); }

    template <class Load>
    static __device__ __forceinline__ void load_first(float2 (&v)[E], int t, Load&& load) {
        constexpr int R = S::radix(0);
        constexpr int B = E / R;
#pragma unroll
        for (int s = 0; s < B; ++s)
#pragma unroll
            for (int r = 0; r < R; ++r) v[s * R + r] = load(t + s * T + r * (N / R));
    }

    // Apply f(index, value&) to every input element as load_first holds them.
    template <class F>
    static __device__ __forceinline__ void for_each_in(float2 (&v)[E], int t, F&& f) {
        constexpr int R = S::radix(0);
#pragma unroll
        for (int s = 0; s < E / R; ++s)
#pragma unroll
            for (int r = 0; r < R; ++r) f(t + s * T + r * (N / R), v[s * R + r]);
    }

    // The steps of pass p: twiddles and DFTs in registers, the results to the exchange buffer, the
    // next pass's inputs back from it.  A kernel may take them apart to hold another t after an
    // exchange than before it.
    template <int p>
    static __device__ __forceinline__ void butterflies(float2 (&v)[E], const float2* __restrict__ tw, int t) {
        constexpr int R = S::radix(p);
        constexpr int B = E / R;
        constexpr int Ns = S::ns(p);
        if constexpr (p > 0) {
            const float2* twp = tw + S::twoff(p);
#pragma unroll
            for (int s = 0; s < B; ++s) {
                const int k = (t + s * T) & (Ns - 1);
#pragma unroll
                for (int r = 1; r < R; ++r)
                    v[s * R + r] = cmul<INV>(v[s * R + r], __ldg(twp + (r - 1) * Ns + k));
            }
        }
#pragma unroll
        for (int s = 0; s < B; ++s) DFT<R, INV>::run(&v[s * R]);
    }
    template <int p>
    static __device__ __forceinline__ void put(const float2 (&v)[E], float2* sm, int t) {
        constexpr int R = S::radix(p);
        constexpr int B = E / R;
        constexpr int Ns = S::ns(p);
#pragma unroll
        for (int s = 0; s < B; ++s) {
            const int j = t + s * T;
            const int k = j & (Ns - 1);
            const int base = (j - k) * R + k, a = at(base);
#pragma unroll
            for (int r = 0; r < R; ++r) sm[out_at<p>(base, a, r)] = v[s * R + r];
        }
    }
    template <int p>
    static __device__ __forceinline__ void get(float2 (&v)[E], const float2* sm, int t) {
        constexpr int R = S::radix(p);
        constexpr int B = E / R;
#pragma unroll
        for (int s = 0; s < B; ++s) {
            const int j = t + s * T, a = at_off<T, 1>(t, at(t), s * T);
#pragma unroll
            for (int r = 0; r < R; ++r) v[s * R + r] = sm[in_at<p>(j, a, r)];
        }
    }

    template <int p>
    static __device__ __forceinline__ void passes(float2 (&v)[E], float2* sm,
                                                  const float2* __restrict__ tw, int t, int row) {
        butterflies<p>(v, tw, t);
        if constexpr (p < P - 1) {
            put<p>(v, sm, t);
            sync(row);
            get<p + 1>(v, sm, t);
            if constexpr (p + 1 < P - 1) sync(row);   // next pass writes the buffer again
            passes<p + 1>(v, sm, tw, t, row);
        }
    }

    // The transform by the transposed graph: passes P-1 .. 0, pass p a DFT_R of the elements put<p>
    // writes, then the twiddles of pass p, stored where get<p> reads.  Its input is laid out as
    // run() leaves a result and its output as run() takes an input (element t + s*T + r*N/R_0),
    // so a product of spectra goes from one transform into the next without an exchange, on the
    // same twiddle table.  `sm` may still be read by the team when called.
    template <int p = P - 1>
    static __device__ __forceinline__ void passes_transposed(float2 (&v)[E], float2* sm, const float2* __restrict__ tw,
                                                             int t, int row) {
        constexpr int R = S::radix(p);
        constexpr int B = E / R;
        constexpr int Ns = S::ns(p);
#pragma unroll
        for (int s = 0; s < B; ++s) DFT<R, INV>::run(&v[s * R]);
        if constexpr (p > 0) {
            const float2* twp = tw + S::twoff(p);
            sync(row);
#pragma unroll
            for (int s = 0; s < B; ++s) {
                const int j = t + s * T, k = j & (Ns - 1), a = at_off<T, 1>(t, at(t), s * T);
                sm[a] = v[s * R];
#pragma unroll
                for (int r = 1; r < R; ++r)
                    sm[in_at<p>(j, a, r)] = cmul<INV>(v[s * R + r], __ldg(twp + (r - 1) * Ns + k));
            }
            sync(row);
            constexpr int R2 = S::radix(p - 1);
            constexpr int B2 = E / R2;
            constexpr int Ns2 = S::ns(p - 1);
#pragma unroll
            for (int s = 0; s < B2; ++s) {
                const int j = t + s * T, k = j & (Ns2 - 1), base = (j - k) * R2 + k, a = at(base);
#pragma unroll
                for (int r = 0; r < R2; ++r) v[s * R2 + r] = sm[out_at<p - 1>(base, a, r)];
            }
            passes_transposed<p - 1>(v, sm, tw, t, row);
        }
    }

    // Element index held in v[s*R_last + r] after run().
    static __device__ __forceinline__ int out_index(int t, int s, int r) {
        constexpr int R = S::radix(P - 1);
        return t + s * T + r * (N / R);
    }

    // Where run() leaves element t + j*T (T = N/E): the slot of v with s + r*B = j.
    static __host__ __device__ constexpr int slot(int j) {
        constexpr int R = S::radix(P - 1), B = E / R;
        return (j % B) * R + j / B;
    }

    template <class Load>
    static __device__ __forceinline__ void run(float2 (&v)[E], float2* sm,
                                               const float2* __restrict__ tw, int t, int row,
                                               Load&& load) {
        load_first(v, t, load);
        passes<0>(v, sm, tw, t, row);
    }

    // Apply f(index, value&) to every output element held by this thread (in place).
    template <class F>
    static __device__ __forceinline__ void for_each_slot(float2 (&v)[E], int t, F&& f) {
        constexpr int R = S::radix(P - 1);
        constexpr int B = E / R;
#pragma unroll
        for (int s = 0; s < B; ++s)
#pragma unroll
            for (int r = 0; r < R; ++r) f(t + s * T + r * (N / R), v[s * R + r]);
    }

    // Apply f(index, value) to every output element held by this thread.
    template <class F>
    static __device__ __forceinline__ void for_each_out(float2 (&v)[E], int t, F&& f) {
        constexpr int R = S::radix(P - 1);
        constexpr int B = E / R;
#pragma unroll
        for (int s = 0; s < B; ++s)
#pragma unroll
            for (int r = 0; r < R; ++r) f(t + s * T + r * (N / R), v[s * R + r]);
    }
};

// ------------------------------------------------------------------ programmatic dependent launch
// A kernel launched with programmatic stream serialisation may start while the previous kernel
// on its stream drains: pdl_wait(), before a kernel's first global access, blocks until the
// previous grid has finished and its writes are visible, so a chain of such launches overlaps
// only launch latency, never data; pdl_trigger(), just before a CTA's final stores, lets the
// next kernel launch once every CTA of this grid has reached that point or ended (triggering at entry
// placed the next grid's CTAs beside this one's and unbalanced one-wave launches; k_pfa and the
// mixed-radix C2C kernels have no trigger).  Without
// the launch attribute both are no-ops.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ------------------------------------------------------------------ global access helpers
// Streaming (evict-first) accesses: every input and output element is touched exactly once.
__device__ __forceinline__ float2 ld_stream(const float2* p) { return __ldcs(p); }
// Input load with the default cache operator (ld.global.ca, a coherent weak load, valid for
// inputs written by a kernel that a programmatic-launch wait ordered before this one).  On the
// single-length C2C kernel it measured 2 % faster than evict-first loads with N(0,1) inputs
// (n = 4096: 0.846 -> 0.861 of the copy peak at batch 4096, 0.896 -> 0.914 at 8192), level
// with read-only (.nc) loads, which are not used because an input may be written by a kernel
// still draining when this one launches.  The two four-step passes gained too (long C2C
// n = 32768: 0.433 -> 0.455; 65536: 0.443 -> 0.446) and so did the column pass (NY = 1024:
// 0.57 -> 0.59); R2C, C2R, the mixed-radix, prime-factor, STFT and Bluestein kernels measured level.  Kernels that
// keep several twiddle tables in L1 (the ragged launch over many lengths) lost with it and keep
// ld_stream.
__device__ __forceinline__ float2 ld_once_ca(const float2* p) { return __ldca(p); }
// Arrays of the caller of which a kernel reads elements more than once (the overlapping frames of a
// signal, a window) are read by plain loads through pointers without __restrict__: coherent for the
// same reason, and free for the compiler to unroll and to issue together, which inline assembly
// (__ldca among it) is not: with that the edge envelopes of a short-time transform, chains of window
// loads, took up to seven times as long.
__device__ __forceinline__ void st_stream(float2* p, float2 v) { __stcs(p, v); }

// Loading ahead into L2: a CTA asks for the lines of the tile that the CTA `ahead` places later
// in the grid will load, so DRAM keeps working while the resident CTAs compute.  Half the CTAs the
// GPU holds at once (kSms SMs, `perSm` CTAs each) is the distance that measured best; a whole
// residency costs 1-5 % of the gain and 1.5 residencies most of it.  Plain launches, 2^25 points,
// without and with: k_c2c n = 4096: 6178 -> 6300 GB/s, 8192: 5049 -> 5433, 16384: 3755 -> 4322;
// k_cols NY = 512: 5798 -> 6410, 1024: 4002 -> 4928.  The fewer CTAs share an SM, the more it
// gives.  kSms sets this distance, and the grid and least size of k_staged: no result depends on it.
constexpr unsigned kSms = 148;
__host__ __device__ constexpr unsigned prefetch_ahead(int perSm) { return perSm * kSms / 2; }
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// The lines of [p, min(p + bytes, end)) by `threads` threads.
template <int BYTES, int THREADS>
__device__ __forceinline__ void prefetch_span(const void* p, const void* end) {
    const char* q = static_cast<const char*>(p) + threadIdx.x * 128;
#pragma unroll
    for (int i = 0; i < BYTES; i += THREADS * 128)
        if ((int)threadIdx.x * 128 + i < BYTES && q + i < static_cast<const char*>(end)) prefetch_l2(q + i);
}

}  // namespace dev
}  // namespace bfly
