// Persistent work-queue kernels with 32 threads per cell for a range of matrix sizes.
#include "gf_persist.cuh"

namespace gf {
const void* persistent_ranged_fn_g32(int range, bool dense) {
    if (range != 32) return nullptr;
    return dense ? reinterpret_cast<const void*>(&persistent_kernel<32, true, 2, 8, -32>)
                 : reinterpret_cast<const void*>(&persistent_kernel<32, true, 0, 8, -32>);
}
#ifdef GF_PHASE_TIMERS
int phase_cycles_g32r(unsigned long long* out, int reset) { return phase_cycles_local(out, reset); }
#endif
}  // namespace gf
