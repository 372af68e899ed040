// Edge-frontier enactors: contract-expand (two O(m) edge frontiers), two-phase
// (one O(n) vertex and one O(m) edge frontier) and hybrid
// (enactor_contract_expand.cuh:61, enactor_two_phase.cuh:68,
// enactor_hybrid.cuh:64).
//
// Fused searches never write the edge frontier: a level's expansion and the
// next level's contraction are one pass of the vertex-frontier kernel
// (ec_kernel), which tests each gathered neighbour instead of storing it for
// the next pass to read -- 8 bytes per edge and one grid barrier per level less,
// and for hybrid no hand-off through the host.  R-MAT 22 contract-expand 1060
// -> 790 us, random 10^6 hybrid 340 -> 167 us.  What the caller sees is kept: labels,
// search depth, the queue total (the edges of the processed levels) and the
// overflow of a level larger than the edge frontiers' capacity.  Per-level
// launches and captured graphs run the two phases as launches of their own
// (edge_kernel).
#include "launch_common.cuh"

namespace b40c {
namespace rt {

namespace {

template <int B, bool PRED>
int enact_phases_t(b40c_bfs_problem *p, int strategy, int mode, int32_t src, int max_grid, const b40c_bfs_policy &pol,
                   int32_t depth_limit)
{
    int rc;
    const bool pingpong = strategy != B40C_TWO_PHASE;
    const int64_t ecap = cap_of(p->queue_sizing, p->edges), vcap = cap_of(p->queue_sizing, p->nodes);
    if ((rc = ensure_ef(p, 0, ecap))) return rc;
    if (pingpong && (rc = ensure_ef(p, 1, ecap))) return rc;
    if ((rc = ensure_vf(p, 0, vcap))) return rc;
    if ((rc = ensure_slots(p))) return rc;
    BfsParams k = make_params(p, pol);
    k.edge_pingpong = pingpong ? 1 : 0;
    k.vcap = (int32_t)p->vcap[0];
    k.ecap = (int32_t)(pingpong ? std::min(p->ecap[0], p->ecap[1]) : p->ecap[0]);
    const void *kern = (const void *)dev::edge_kernel<B, PRED>;
    const size_t smem = kernel_smem<dev::ExpandSmem<B, PRED>>(pol);
    int grid = 0;
    if ((rc = persistent_grid(p, kern, pol, max_grid, smem, kernel_smem_limit<B, PRED>(), &grid))) return rc;
    if ((rc = begin_enact(p, src, depth_limit))) return rc;
    if ((rc = begin_instrumented(p))) return rc;

    BfsParams kc = k, kx = k;  // contract, expand
    kc.phase_mask = 1;
    kx.phase_mask = 2;

    if (mode == B40C_ENACT_GRAPH) {
        if ((rc = mark_search_start(p))) return rc;
        KernelNode init{init_kernel_ptr<PRED>(false, true), dim3(init_grid(p, true)), dim3(kThreads), 0, k};
        KernelNode body[2] = {{kern, dim3(grid), dim3(B), smem, kc}, {kern, dim3(grid), dim3(B), smem, kx}};
        if ((rc = run_graph(p, strategy, init, body, 2))) return rc;
        return finish_timing(p);
    }
    if (mode != B40C_ENACT_ITERATIVE) return b40c::fail(B40C_ERROR_INVALID_VALUE, "unknown enact mode %d", mode);
    if ((rc = upload_source(p))) return rc;
    if ((rc = launch_init<PRED>(p, k, false, p->needs_init))) return rc;
    if ((rc = mark_search_start(p))) return rc;
    if ((rc = read_state(p))) return rc;
    while (!(p->h_st->error || p->h_st->done || qe_count(p->h_st->qe[(2 * p->h_st->cur_level) % 3]) == 0)) {
        if ((rc = launch_plain(p, kern, grid, B, smem, kc, "contract launch"))) return rc;
        if ((rc = launch_plain(p, kern, grid, B, smem, kx, "expand launch"))) return rc;
        if ((rc = read_state(p))) return rc;
    }
    return finish_timing(p);
}

}  // namespace

int enact_edge(b40c_bfs_problem *p, int strategy, int mode, int32_t src, int max_grid, const b40c_bfs_policy &pol,
               int32_t depth_limit)
{
    if (mode == B40C_ENACT_FUSED) {
        // the capacity the edge frontiers have, or would be given: a larger level
        // overflows, as it does in the per-phase launches
        const int64_t ecap = std::max<int64_t>(cap_of(p->queue_sizing, p->edges), 1);
        const int64_t first = std::max(ecap, p->ecap[0]), second = std::max(ecap, p->ecap[1]);
        const int64_t limit = strategy == B40C_TWO_PHASE ? first : std::min(first, second);
        p->queues_edges = true;
        return enact_vertex(p, mode, src, max_grid, pol, depth_limit, false,
                            (int32_t)std::min<int64_t>(limit, INT32_MAX - 1));
    }
#define B40C_EDGE(B)                                                                                \
    (p->mark_pred ? enact_phases_t<B, true>(p, strategy, mode, src, max_grid, pol, depth_limit)     \
                  : enact_phases_t<B, false>(p, strategy, mode, src, max_grid, pol, depth_limit))
    switch (pol.threads) {
    case 128: return B40C_EDGE(128);
    case 512: return B40C_EDGE(512);
    default: return B40C_EDGE(256);
    }
#undef B40C_EDGE
}

}  // namespace rt
}  // namespace b40c
