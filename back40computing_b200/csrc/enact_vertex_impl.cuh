// The expand-contract enactor's body for one CTA size (included by the
// per-size translation units enact_vertex_<B>.cu, so the kernel variants of
// each size compile in parallel).
#pragma once
#include "launch_common.cuh"

namespace b40c {
namespace rt {

template <int B, bool PRED>
int enact_ec_t(b40c_bfs_problem *p, int mode, int32_t src, int max_grid, const b40c_bfs_policy &pol,
               int32_t depth_limit, bool direction_opt, int32_t edge_limit)
{
    int rc;
    const int64_t vcap = cap_of(p->queue_sizing, p->nodes);
    VertexFrontier queue[2];
    int64_t queue_cap = 0;
    if (edge_limit != INT32_MAX) {
        if ((rc = edge_strategy_queues(p, vcap, queue, &queue_cap))) return rc;
    } else {
        for (int i = 0; i < 2; i++) {
            if ((rc = ensure_vf(p, i, vcap))) return rc;
            queue[i] = p->vf[i];
        }
        queue_cap = std::min(p->vcap[0], p->vcap[1]);
    }
    if ((rc = ensure_slots(p))) return rc;
    if (direction_opt && pol.bottom_up_hub_probes > 0 && (rc = ensure_hubs(p))) return rc;
    const bool lists = direction_opt && !PRED && pol.bottom_up_list > 0;
    if (lists && (rc = ensure_unvisited_lists(p))) return rc;
    BfsParams k = make_params(p, pol);
    k.vf[0] = queue[0];
    k.vf[1] = queue[1];
    k.vcap = (int32_t)queue_cap;
    k.direction_opt = direction_opt ? 1 : 0;
    k.edge_limit = edge_limit;
    if (!direction_opt) k.hub2 = nullptr;
    if (lists) {
        // distance searches: bottom-up levels after the first one scan the unvisited list
        k.ul[0] = p->d_ul[0];
        k.ul[1] = p->d_ul[1];
    }
    // distance searches with unvisited lists run the kernel variant that
    // carries list mode; the others keep the leaner code
    const bool lists_kernel = direction_opt && !PRED && pol.bottom_up_list > 0;
    // plain expand-contract searches (and directed graphs) never go bottom-up:
    // they run the top-down-only variants; list mode is built for 256-thread CTAs
    // only, and a sub-grid threshold asks for them too (not of the edge-frontier
    // strategies, whose policies may carry one with any CTA size)
    const bool subgrid =
        mode == B40C_ENACT_FUSED && pol.subgrid_frontier_edges > 0 && edge_limit == INT32_MAX;
    if (B != 256 && (lists_kernel || subgrid))
        return b40c::fail(B40C_ERROR_INVALID_VALUE,
                          "policy.threads %d: bottom-up list mode and the sub-grid phase need 256", B);
    const void *kern = direction_opt ? (const void *)dev::ec_kernel<B, PRED, false>
                                     : (const void *)dev::ec_kernel<B, PRED, false, false>;
    if constexpr (B == 256)
        if (lists_kernel) kern = (const void *)dev::ec_kernel<256, false, true>;
    const size_t smem = kernel_smem<dev::ExpandSmem<B, PRED>>(pol);
    int grid = 0;
    if ((rc = persistent_grid(p, kern, pol, max_grid, smem, kernel_smem_limit<B, PRED>(), &grid))) return rc;
    if ((rc = begin_enact(p, src, depth_limit, mode == B40C_ENACT_FUSED))) return rc;
    if ((rc = begin_instrumented(p))) return rc;
    if (mode == B40C_ENACT_GRAPH) {
        if ((rc = mark_search_start(p))) return rc;
        KernelNode init{init_kernel_ptr<PRED>(true, true), dim3(init_grid(p, true)), dim3(kThreads), 0, k};
        KernelNode body[1] = {{kern, dim3(grid), dim3(B), smem, k}};
        const int slot = direction_opt ? B40C_HYBRID + 1 : B40C_EXPAND_CONTRACT;
        if ((rc = run_graph(p, slot, init, body, 1))) return rc;
        return finish_timing(p);
    }
    // the source and depth limit travel as kernel arguments of the init kernel
    // (no host-to-device copy in the search's stream)
    k.src_by_value = 1;
    k.src_arg = src;
    k.depth_arg = depth_limit;
    if (mode == B40C_ENACT_FUSED) {
        // the kernel sets the search up itself: one launch less (see ec_kernel).  A
        // launch captured into a graph may be replayed, but its turn of the barrier
        // counters may not: it keeps the set-up launch, which clears the one it uses,
        // and fills the labels and the mask, which a replay finds as any search left them
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        CUDA_TRY(cudaStreamIsCapturing(p->stream, &capture), "capture query");
        const bool captured = capture != cudaStreamCaptureStatusNone;
        if (captured && (rc = launch_init<PRED>(p, k, true, true))) return rc;
        if ((rc = mark_search_start(p))) return rc;
        k.init = captured ? 0 : p->needs_init ? 2 : 1;
        k.barrier_sel = p->barrier_sel;
        k.persistent = 1;
        k.max_levels = INT32_MAX;
        k.skip_arrival_cta = injected_skip_cta();
        k.late_start_ns = injected_late_start_ns();
        if ((rc = launch_cooperative(p, kern, grid, B, smem, k, "cooperative launch of the expand-contract kernel")))
            return rc;
        if (!captured) p->barrier_sel ^= 1;  // (this launch clears the other counter)
    } else if (mode == B40C_ENACT_ITERATIVE) {
        if ((rc = launch_init<PRED>(p, k, true, p->needs_init))) return rc;
        if ((rc = mark_search_start(p))) return rc;
        // one launch per level; the host reads the next frontier's size.  On a small
        // graph one CTA per SM, but a level nearly all of whose edges meet visited
        // vertices is bound by its tests and takes what fits (us per level with one and
        // with two: R-MAT 16 x 8, 741 thousand edges with 24 thousand left, 37 and 26;
        // R-MAT 16 x 5, 344 thousand with 307 thousand left, 31 and 36)
        const bool small = B == 512 && pol.ctas_per_sm == 0 && p->edges <= kSmallGraphEdges;
        for (int level = 0;; level++) {
            if ((rc = read_state(p))) return rc;
            if (p->h_st->error || p->h_st->done) break;
            const int q = qe_count(p->h_st->qe[level % 3]), E = qe_edges(p->h_st->qe[level % 3]);
            if (q == 0) break;
            int g = std::max(1, std::min(grid, (E + dev::kChunkGrain - 1) / dev::kChunkGrain));
            const int64_t left = p->edges - (int64_t)p->h_st->visited_edges[level % 3] - E;
            if (small && E <= 8 * left) g = std::min(g, p->sms);
            if (direction_opt) g = grid;  // a bottom-up level spans every vertex
            if ((rc = launch_plain(p, kern, g, B, smem, k, "expand-contract level launch"))) return rc;
        }
    } else {
        return b40c::fail(B40C_ERROR_INVALID_VALUE, "unknown enact mode %d", mode);
    }
    return finish_timing(p);
}

// One CTA size's entry, instantiated in enact_vertex_<B>.cu.
template <int B>
int enact_vertex_b(b40c_bfs_problem *p, int mode, int32_t src, int max_grid, const b40c_bfs_policy &pol,
                   int32_t depth_limit, bool direction_optimizing, int32_t edge_limit)
{
    return p->mark_pred ? enact_ec_t<B, true>(p, mode, src, max_grid, pol, depth_limit, direction_optimizing, edge_limit)
                        : enact_ec_t<B, false>(p, mode, src, max_grid, pol, depth_limit, direction_optimizing,
                                               edge_limit);
}

}  // namespace rt
}  // namespace b40c
