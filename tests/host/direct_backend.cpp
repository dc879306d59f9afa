// The fake seam (fake_backend.cpp) with the kernels it lacks: 32 values a thread at 1024, 8192 and
// 16384, and the one-pass cluster kernels of 32768 and 65536.  Records which kernel each C2C launch
// named.  Test infrastructure only.
#include "backend.h"

#define hasVariant narrowVariant
#define launchC2C narrowLaunchC2C
#define launchLongB narrowLaunchLongB
#include "fake_backend.cpp"
#undef hasVariant
#undef launchC2C
#undef launchLongB

namespace fake {
int lastE = 0, lastCta = 0;        // of the last C2C launch; -3: a cluster kernel
int directTables = 0;              // tables built for the cluster kernels
uint32_t clusterUnavailable = 0;   // a length whose cluster the device cannot hold
int longLaunches = 0;              // four-step transforms
}  // namespace fake

namespace bfly {
namespace backend {

bool hasVariant(int kind, uint32_t n, int e, int cta) {
    if (kind == kC2C && e == 32) return (n == 1024 && cta == 64) || ((n == 8192 || n == 16384) && cta == (int)n / 32);
    return narrowVariant(kind, n, e, cta);
}

int launchC2C(const void* in, void* out, uint32_t n, uint64_t batch, bool inverse, float scale, const void* tw, int e,
              int cta, void* stream) {
    fake::lastE = e;
    fake::lastCta = cta;
    if (!tw || !hasVariant(kC2C, n, e, cta)) return 1;
    if (n < 8192) return narrowLaunchC2C(in, out, n, batch, inverse, scale, tw, e, cta, stream);
    if (int r = launch()) return r;   // a direct DFT of the long lengths takes too long
    std::memcpy(out, in, (size_t)n * batch * 8);
    return 0;
}

int launchLongB(const void* in, void* out, uint32_t n1, uint32_t n2, uint64_t batch, bool, float, const void*, void*) {
    ++fake::longLaunches;
    if (int r = launch()) return r;
    std::memcpy(out, in, (size_t)n1 * n2 * batch * 8);
    return 0;
}

size_t directTableBytes(uint32_t n) {
    return (n == 32768 || n == 65536) && n != fake::clusterUnavailable ? (size_t)n : 0;
}
int buildDirectTable(void* table, uint32_t n, void*) {
    if (!table || !directTableBytes(n)) return 1;
    ++fake::directTables;
    std::memset(table, 0, directTableBytes(n));
    return launch();
}
// The first values of each row are enough to tell rows and directions apart: a direct DFT of 65536
// points takes minutes.
int launchDirect(const void* in, void* out, uint32_t n, uint64_t batch, bool inverse, float scale, const void* table,
                 void*) {
    if (!table || !directTableBytes(n)) return 1;
    fake::lastE = -3;
    if (int r = launch()) return r;
    for (uint64_t b = 0; b < batch; ++b) {
        const float* x = (const float*)in + b * 2 * n;
        float* y = (float*)out + b * 2 * n;
        for (uint32_t i = 0; i < 2 * n; ++i) y[i] = (inverse ? -1.f : 1.f) * scale * x[i];
    }
    return 0;
}

}  // namespace backend
}  // namespace bfly
