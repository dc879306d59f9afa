// C2C kernel instantiations (forward).  Variant list: N in 32..16384, E in {8,16},
// CTA in {128,256,512} (1024 only for one-transform-per-CTA lengths), shared memory <= 227 KB.
#include "fft_kernels.cuh"
#include "registry.cuh"

namespace bfly {
namespace dev {

#define E_(N, E, CTA) {N, E, CTA, 0, (const void*)&k_c2c<N, E, BFLY_ROWS(N, E, CTA), false>, \
    BFLY_ROWS(N, E, CTA), BFLY_ROWS(N, E, CTA) * smem_stride<N, E, false>() * 8}
// Radix 16 served by k_long_direct.cu; listed for the candidates' limits.
#define D_(N, CTA) {N, 16, CTA, 0, nullptr, BFLY_ROWS(N, 16, CTA), BFLY_ROWS(N, 16, CTA) * smem_stride<N, 16, false>() * 8}
static const Entry kTable[] = {
    E_(32, 8, 128),
    E_(32, 8, 256),
    E_(32, 8, 512),
    E_(32, 16, 128),
    E_(32, 16, 256),
    E_(32, 16, 512),
    E_(64, 8, 128),
    E_(64, 8, 256),
    E_(64, 8, 512),
    E_(64, 16, 128),
    E_(64, 16, 256),
    E_(64, 16, 512),
    E_(128, 8, 128),
    E_(128, 8, 256),
    E_(128, 8, 512),
    E_(128, 16, 128),
    E_(128, 16, 256),
    E_(128, 16, 512),
    E_(256, 8, 128),
    E_(256, 8, 256),
    E_(256, 8, 512),
    E_(256, 16, 128),
    E_(256, 16, 256),
    E_(256, 16, 512),
    E_(512, 8, 128),
    E_(512, 8, 256),
    E_(512, 8, 512),
    E_(512, 16, 128),
    E_(512, 16, 256),
    E_(512, 16, 512),
    E_(1024, 8, 128),
    E_(1024, 8, 256),
    E_(1024, 8, 512),
    D_(1024, 128),
    D_(1024, 256),
    D_(1024, 512),
    E_(2048, 8, 256),
    E_(2048, 8, 512),
    E_(2048, 16, 128),
    E_(2048, 16, 256),
    E_(2048, 16, 512),
    E_(4096, 8, 512),
    E_(4096, 16, 256),
    E_(4096, 16, 512),
    E_(8192, 8, 1024),
    D_(8192, 512),
    D_(16384, 1024),
};
#undef D_
#undef E_

const Entry* findC2CFwd(uint32_t n, int e, int cta) {
    for (const Entry& x : kTable)
        if (x.n == n && x.e == e && x.cta == cta) return &x;
    return nullptr;
}

}  // namespace dev
}  // namespace bfly
