// The beam-search kernels for 32 chunks.
#include "beam_long.cuh"
#include "beam_short.cuh"

namespace tann {
BeamKernelFn PickShort32(uint32_t rounds, int kind, uint32_t list_regs) {
    switch (list_regs) {
        case 1: return PickShortOf<32, 1>(rounds, kind);
        case 2: return PickShortOf<32, 2>(rounds, kind);
        case 4: return PickShortOf<32, 4>(rounds, kind);
        default: return PickShortOf<32, 8>(rounds, kind);
    }
}
BeamKernelFn PickLong32(uint32_t rounds, int kind, bool late) { return PickLongOf<32>(rounds, kind, late); }
}  // namespace tann
