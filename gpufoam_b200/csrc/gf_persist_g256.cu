// Persistent work-queue kernel variants with 256 thread(s) per cell.
#include "gf_persist.cuh"

namespace gf {
const void* persistent_fn_g256(bool shared, int slim) { return persistent_variant<256>(shared, slim); }
const void* persistent_ranged_fn_g256() {
    return reinterpret_cast<const void*>(&persistent_kernel<256, true, 0, 8, kAllRanges>);
}
#ifdef GF_PHASE_TIMERS
int phase_cycles_g256(unsigned long long* out, int reset) { return phase_cycles_local(out, reset); }
#endif
}  // namespace gf
