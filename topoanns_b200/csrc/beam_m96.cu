// The beam-search kernels for 96 chunks.
#include "beam_long.cuh"
#include "beam_short.cuh"

namespace tann {
BeamKernelFn PickShort96(uint32_t rounds, int kind, uint32_t list_regs) {
    switch (list_regs) {
        case 1: return PickShortOf<96, 1>(rounds, kind);
        case 2: return PickShortOf<96, 2>(rounds, kind);
        case 4: return PickShortOf<96, 4>(rounds, kind);
        default: return PickShortOf<96, 8>(rounds, kind);
    }
}
BeamKernelFn PickLong96(uint32_t rounds, int kind, bool late) { return PickLongOf<96>(rounds, kind, late); }
}  // namespace tann
