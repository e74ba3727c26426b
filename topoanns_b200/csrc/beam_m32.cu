// The beam-search kernels for 32 chunks.
#include "beam_long.cuh"
#include "beam_short.cuh"

namespace tann {
BeamKernelFn PickShort32(uint32_t rounds, int kind, uint32_t list_regs) {
    return list_regs == 1 ? PickShortOf<32, 1>(rounds, kind) : (list_regs == 2 ? PickShortOf<32, 2>(rounds, kind) : PickShortOf<32, 4>(rounds, kind));
}
BeamKernelFn PickLong32(uint32_t rounds, int kind, bool late) { return PickLongOf<32>(rounds, kind, late); }
}  // namespace tann
