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

// Which form takes a call. Below: speed relative to the general form (beam_search.cu) on 100 k x 128 uint8 (degree 32), 10 M x 128 uint8
// (degrees 32 and 64, with and without neighbour codes), 4 M x 96 float32 (64) and 1 M x 768 float32 (64), M = 32, 32, 48 and 96, batches
// of 1 to 10 000.
// Other chunk counts (16 and 64 have forms of their own there) stay with the general form: none of the configurations has them.
// * Register list (widths 1 and 2; capacities C of 32, 64, 128 and 256, without the learned stop): 1.02 to 1.78 for C of up to 128. A
//   list of 256 costs more per step, which a short search does not earn back: at width 2, C = 256 and L = 16 / 32 / 64 / 100
//   M = 32 has 0.80-0.91 / 0.87-0.99 / 0.97-1.13 / 1.01-1.16, M = 96 0.77-0.79 / 0.82-0.88 / 0.92-1.03 / 0.98-1.11, at width 1 and
//   L = 32 / 64 1.02-1.30 and 0.92-1.17. The line is at L = 32 (M = 96: 64) times the width.
//   Longer lists: 16 key registers per lane double the list warp's chain (L = 512, M = 32, 2 k queries 2.7 -> 6.5 ms).
// * Shared-memory list, steps of up to 128 slots: ahead where its one list in place of two lets one block more reside on an SM and the
//   batch needs more than one wave. M = 32, C = 512, L = 400 / 512: 1.01-1.25 / 1.02-1.34 for 600 queries and more (0.85-1.0 for 150 and
//   fewer; L of up to 128: 0.89-0.99; C = 1024, where as many blocks reside: 0.73-0.88); M = 96, C = 512 / 1024: 1.0-1.9 /
//   1.46-1.8 from 150 queries on (one query: 0.79-1.0); with the learned stop M = 32, C = 512 1.0-1.2, M = 48, C up to 128 1.11-1.22
//   for 2 k queries and more. Widths 3 and 4 lose (0.67-0.99 on a degree of 32), but for M = 96 (1.49-1.73). M = 96 with the learned
//   stop and a list that ends at top_l: 1.0-1.15 at every batch size.
// * Steps of 129 to 256 slots, which the general form takes in rounds through a sort in shared memory: the register list (degree 96,
//   width 2: 1.5 to 7.1), for M = 96 at C = 256 and L below 64 and for all other calls the shared-memory list (1.0 to 6.5; width 32
//   on a degree of 8, which selects 32 nodes one by one, 0.94 to 1.1 for batches of up to 150).
bool PlanFast(const TannIndexView& ix, const TannBeamParams& p, uint64_t num_queries, FastPlan* plan) {
    *plan = FastPlan{};
    const uint32_t M = ix.num_chunks, C = p.candidate_capacity, L = p.top_l, W = p.search_width;
    const uint32_t slots = W * ix.degree;
    const bool late = p.learned_stop.enabled != 0;
    if (!(M == 32 || M == 48 || M == 96) || slots > 256u || L > 1024 || C > 1024 || ix.dim > kBloomWords || num_queries > 0x7fffffffull) return false;
    if (p.stop_prefix != 0 && p.stop_prefix < L) return false;
    const bool sharded = ix.adjacency.num_shards > 1 || ix.codes.num_shards > 1;
    const bool nbr = ix.neighbor_codes.base[0] != nullptr;
    if ((sharded && (late || nbr)) || (nbr && ix.neighbor_codes.num_shards > 1)) return false;
    plan->kind = sharded ? 2 : (nbr ? 1 : 0);
    plan->rounds = slots > 128u ? 2u : 1u;
    plan->late = late;
    const uint32_t least_l = C < 256 ? 0u : (plan->rounds == 1 ? (M == 96 ? 64u : 32u) * W : (M == 96 ? 64u : 0u));
    const bool registers = W <= 2 && !late && ix.num_nodes <= 0x3fffffffull && C >= 32 && C <= 256 && L >= least_l;
    if (registers) {
        plan->list_regs = C / 32;
        plan->smem = ShortLayout(M, plan->rounds).total;
        return plan->smem <= 227u * 1024u - 512u;
    }
    plan->list_len = C;
    const uint32_t one = LongLayout(M, plan->rounds, C, false).total, two = LongLayout(M, plan->rounds, C, true).total;
    plan->two_lists = ResidentBlocks(two) == ResidentBlocks(one);
    plan->smem = plan->two_lists ? two : one;
    if (plan->rounds == 1) {
        const uint32_t general = (228u * 1024u) / ((uint32_t)BeamSmemBytes(M, C, 128u, L, ix.dim) + 1024u + 960u);
        const bool more_blocks = ResidentBlocks(plan->smem) > general && num_queries > (uint64_t)SmCount() * general;
        const bool ahead = (more_blocks && (M == 96 ? W <= 4 : W <= 2 && (late || (M == 32 && L > 256)))) || (M == 96 && W <= 2 && late && C < 2 * L);
        if (!ahead) return false;
    }
    return plan->smem <= 227u * 1024u - 512u;
}

static cudaError_t LaunchBeamKernel(BeamKernelFn k, const BeamArgs& a, uint32_t grid, uint32_t threads, uint32_t smem, cudaStream_t stream) {
    if (k == nullptr) return cudaErrorInvalidDeviceFunction;   // PlanFast asks for no such form
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
