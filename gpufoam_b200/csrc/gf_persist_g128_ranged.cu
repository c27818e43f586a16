// Persistent work-queue kernels with 128 threads per cell for a range of matrix sizes.
#include "gf_persist.cuh"

namespace gf {
const void* persistent_ranged_fn_g128(int range) {
    if (range == 32) return reinterpret_cast<const void*>(&persistent_kernel<128, true, 0, 8, -32>);
    if (range == 64) return reinterpret_cast<const void*>(&persistent_kernel<128, true, 0, 8, -64>);
    if (range == 128) return reinterpret_cast<const void*>(&persistent_kernel<128, true, 0, 8, -128>);
    return nullptr;
}
#ifdef GF_PHASE_TIMERS
int phase_cycles_g128r(unsigned long long* out, int reset) { return phase_cycles_local(out, reset); }
#endif
}  // namespace gf
