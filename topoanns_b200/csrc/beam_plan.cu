// Which beam-search kernel serves a call, and with what shared memory.
#include "beam_long.cuh"
#include "beam_short.cuh"
#include "tann_launch.h"

namespace tann {

BeamKernelFn PickShort32(uint32_t rounds, int kind, uint32_t list_regs);
BeamKernelFn PickShort48(uint32_t rounds, int kind, uint32_t list_regs);
BeamKernelFn PickShort96(uint32_t rounds, int kind, uint32_t list_regs);
BeamKernelFn PickLong32(uint32_t rounds, int kind, bool late);
BeamKernelFn PickLong48(uint32_t rounds, int kind, bool late);
BeamKernelFn PickLong96(uint32_t rounds, int kind, bool late);

static uint32_t ResidentBlocks(uint32_t smem) { return (228u * 1024u) / (smem + 1024u + 512u); }

bool PlanFast(const TannIndexView& ix, const TannBeamParams& p, FastPlan* plan) {
    *plan = FastPlan{};
    const uint32_t M = ix.num_chunks, C = p.candidate_capacity, L = p.top_l;
    const uint32_t slots = p.search_width * ix.degree;
    const bool late = p.learned_stop.enabled != 0;
    if (!(M == 32 || M == 48 || M == 96) || slots > 256u || L > 1024 || C > 1024 || ix.dim > kBloomWords) return false;
    if (p.stop_prefix != 0 && p.stop_prefix < L) return false;
    const bool sharded = ix.adjacency.num_shards > 1 || ix.codes.num_shards > 1;
    const bool nbr = ix.neighbor_codes.base[0] != nullptr;
    if ((sharded && (late || nbr)) || (nbr && ix.neighbor_codes.num_shards > 1)) return false;
    plan->kind = sharded ? 2 : (nbr ? 1 : 0);
    plan->rounds = slots > 128u ? 2u : 1u;
    plan->late = late;
    // Long form -> short form on the same index: L = 64 (M = 48) 307 -> 219 us for 500 queries, L = 256 9.74 -> 7.2 ms for 10 k.
    // Lists of 512 would need 16 register pairs per lane, whose merges bound the step: 2.7 -> 6.5 ms for 2 k queries (M = 32).
    const bool single = p.search_width <= 2 && !late && ix.num_nodes <= 0x3fffffffull;
    if (single && C >= 32 && C <= 256) {
        plan->list_regs = C / 32;
        plan->smem = ShortLayout(M, plan->rounds).total;
        return plan->smem <= 227u * 1024u - 512u;
    }
    if (single && L <= 256 && plan->rounds == 1) return false;
    plan->list_len = C;
    const uint32_t one = LongLayout(M, plan->rounds, C, false).total, two = LongLayout(M, plan->rounds, C, true).total;
    plan->two_lists = ResidentBlocks(two) == ResidentBlocks(one);
    plan->smem = plan->two_lists ? two : one;
    return plan->smem <= 227u * 1024u - 512u;
}

static cudaError_t LaunchBeamKernel(BeamKernelFn k, const BeamArgs& a, uint32_t grid, uint32_t threads, uint32_t smem, cudaStream_t stream) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<grid, threads, smem, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t LaunchFast(BeamArgs a, const FastPlan& plan, uint64_t num_queries, cudaStream_t stream) {
    const uint32_t M = a.ix.num_chunks;
    a.list_len = plan.list_len;
    a.two_lists = plan.two_lists ? 1u : 0u;
    if (plan.list_regs != 0) {
        BeamKernelFn k = M == 32   ? PickShort32(plan.rounds, plan.kind, plan.list_regs)
                         : M == 48 ? PickShort48(plan.rounds, plan.kind, plan.list_regs)
                                   : PickShort96(plan.rounds, plan.kind, plan.list_regs);
        return LaunchBeamKernel(k, a, (uint32_t)num_queries, kShortThreads, plan.smem, stream);
    }
    BeamKernelFn k = M == 32   ? PickLong32(plan.rounds, plan.kind, plan.late)
                     : M == 48 ? PickLong48(plan.rounds, plan.kind, plan.late)
                               : PickLong96(plan.rounds, plan.kind, plan.late);
    return LaunchBeamKernel(k, a, (uint32_t)num_queries, kBeamThreads, plan.smem, stream);
}

uint32_t FastBlocksPerSm(const FastPlan& plan) { return ResidentBlocks(plan.smem); }

}  // namespace tann
