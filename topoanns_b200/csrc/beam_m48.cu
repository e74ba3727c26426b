// The beam-search kernels for 48 chunks.
#include "beam_long.cuh"
#include "beam_short.cuh"

namespace tann {
BeamKernelFn PickShort48(uint32_t rounds, int kind, uint32_t list_regs) {
    switch (list_regs) {
        case 1: return PickShortOf<48, 1>(rounds, kind);
        case 2: return PickShortOf<48, 2>(rounds, kind);
        case 4: return PickShortOf<48, 4>(rounds, kind);
        default: return PickShortOf<48, 8>(rounds, kind);
    }
}
BeamKernelFn PickLong48(uint32_t rounds, int kind, bool late) { return PickLongOf<48>(rounds, kind, late); }
}  // namespace tann
