// Persistent work-queue kernels with 64 threads per cell for a range of matrix sizes.
#include "gf_persist.cuh"

namespace gf {
const void* persistent_ranged_fn_g64(int range) {
    if (range == 32) return reinterpret_cast<const void*>(&persistent_kernel<64, true, 0, 8, -32>);
    if (range == 64) return reinterpret_cast<const void*>(&persistent_kernel<64, true, 0, 8, -64>);
    if (range == 128) return reinterpret_cast<const void*>(&persistent_kernel<64, true, 0, 8, -128>);
    return nullptr;
}
#ifdef GF_PHASE_TIMERS
int phase_cycles_g64r(unsigned long long* out, int reset) { return phase_cycles_local(out, reset); }
#endif
}  // namespace gf
