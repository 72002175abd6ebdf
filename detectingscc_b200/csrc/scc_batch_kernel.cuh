// The batched kernel (see scc_batch.cu), one translation unit per CTA size:
// the units compile side by side.
#pragma once
#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include "scc_phases.cuh"
#include "scc_batch_internal.h"

using namespace sccb;

namespace {

// Runs one graph with execution policy `ex` on the scratch slice `base`
// (every CTA of the policy calls it with the same arguments).
template <bool HONG, class Ex>
__device__ void batch_one(Ex &ex, const BatchParams &p, uint32_t gi, char *base, Work &s_w)
{
    const BatchGraph bg = p.graphs[gi];
    const unsigned long long t0 = gtimer();
    if (bg.V == 0u) {
        if (ex.leader()) {
            p.res[gi] = BatchRes{0ull, 0ull, 0ull, 0, 0, 0ull};
            if (p.done) {
                __threadfence_system();
                *(volatile unsigned *)&p.done[gi] = 1u;
            }
        }
        return;
    }
    Graph g{bg.V, bg.E, p.Fr + bg.off_r, p.Fc + bg.off_c, p.Br + bg.off_r, p.Bc + bg.off_c, p.vec};
    if (threadIdx.x == 0) {
        carve_work(base, bg.V, bg.E, &s_w);
        s_w.qcap = p.qcap;
        s_w.bu_k = p.bu_k;
        s_w.pull_lane = PULL_LANE;
    }
    __syncthreads();
    const Work &w = s_w;
    ex.ctl = w.ctl;
    // fresh control block and pivot word for this graph
    {
        uint32_t *c = reinterpret_cast<uint32_t *>(w.ctl);
        for (unsigned i = ex.tid(); i < sizeof(Ctl) / 4; i += ex.nthr()) c[i] = 0u;
        if (ex.leader()) w.pivkey[0] = w.pivkey[1] = 0ull;
        ex.sync();
        if constexpr (!Ex::cluster) ex.reset_counters();   // this CTA's counter ring and error flag
        if (ex.leader()) {
            w.ctl->timeout_ns = p.timeout_ns;
            w.ctl->first_min = 0xFFFFFFFFu;
        }
        ex.sync();
    }
    ex.gl = 0u;
    Carry cy{};
    int rc = HONG ? hong_front(ex, g, w, p.t1, p.t2, p.lw, cy) : slota_front(ex, g, w, p.t1, p.lw, cy);
    if (rc == RUN_DONE) rc = peel_loop(ex, g, w, cy, 0u);
    ex.sync();   // the same error word in every CTA of the policy
    const int err = *(volatile int *)&w.ctl->error;
    if (!err) {
        uint32_t *o = p.out + bg.off_out;
        const uint32_t fm = *(volatile const uint32_t *)&w.ctl->first_min;
        for (uint32_t v = ex.tid() + 1u; v <= bg.V; v += ex.nthr()) {
            const uint32_t s = nib_of(w.nb, v);
            const uint32_t l = nib_label(s, v, fm, w.label);
            o[v - 1u] = (l & LBL_SELF) ? (l & ~LBL_SELF) : (l <= bg.V ? w.smin[l] : 0u);
        }
    }
    if (ex.leader())
        p.res[gi] = BatchRes{w.ctl->n_trim1, w.ctl->n_trim2, w.ctl->n_pivot, err, w.ctl->where, gtimer() - t0};
    if (p.done) __threadfence_system();   // labels and result reach the host before the flag
    ex.sync();   // the slice is reused by the next graph
    if (p.done && ex.leader()) *(volatile unsigned *)&p.done[gi] = 1u;
}

// The first p.nbig graphs of p.order run one at a time on a whole cluster
// (when the launch has clusters), the rest one per CTA.  Counters:
// next[0] for cluster graphs, next[1] for CTA graphs.
// CL: the variant with the cluster loop, launched only when the batch has
// cluster graphs (kept apart so the common one-CTA-per-graph kernel does
// not carry the cluster path's registers).  64 registers a thread, so that an
// SM holds 1,024 of them: spilled, bytes stored / loaded (-Xptxas -v): Slota
// 16 / 20 and with clusters 160 / 808, Hong, whose trims share the frame with
// the search and the peels, 184 / 160 and 540 / 1,712.
template <int THREADS, bool HONG, bool CL>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_scc_batch(BatchParams p)
{
    __shared__ uint32_t s_k, s_kb;
    __shared__ Work s_w;   // per-graph carving, kept in shared memory rather than local memory
    bq_init();
    char *mine = p.scratch + (size_t)blockIdx.x * p.scratch_per_cta;
    if (CL && p.nbig) {
        const unsigned cr = cluster_rank(), cn = cluster_size();
        char *lead = p.scratch + (size_t)((blockIdx.x - cr) / p.lead_div) * p.scratch_per_cta;   // 1-D clusters
        for (;;) {
            if (cr == 0 && threadIdx.x == 0) s_kb = atomicAdd(&p.next[0], 1u);
            cluster_barrier();
            const uint32_t k = *cooperative_groups::this_cluster().map_shared_rank(&s_kb, 0);
            // check mode: every graph starts from a clean software barrier
            // word (all CTAs are past the previous graph here; a graph that
            // ended on a timed-out wait can leave the word mid-count)
            if (p.cbar && cr == 0 && threadIdx.x == 0) p.cbar[(blockIdx.x - cr) / cn] = 0u;
            cluster_barrier();   // rank 0 rewrites s_kb only after every CTA has read it
            if (k >= p.nbig) break;
            ClusterExec<false> ex{nullptr, 0u, cr, cn, p.cbar ? p.cbar + (blockIdx.x - cr) / cn : nullptr,
                                  p.timeout_ns, p.pass_cap, p.cbar ? p.hold : 0u};
            batch_one<HONG>(ex, p, p.order[k], lead, s_w);
        }
    }
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_k = p.nbig + atomicAdd(&p.next[1], 1u);
        __syncthreads();
        const uint32_t k = s_k;
        if (k >= p.n) return;
        BlockExec<false> ex{nullptr, 0u, p.pass_cap};
        batch_one<HONG>(ex, p, p.order[k], mine, s_w);
    }
}

template <int THREADS>
void *batch_kernel(bool hong, bool cl)
{
    if (cl) return hong ? (void *)k_scc_batch<THREADS, true, true> : (void *)k_scc_batch<THREADS, false, true>;
    return hong ? (void *)k_scc_batch<THREADS, true, false> : (void *)k_scc_batch<THREADS, false, false>;
}

}  // namespace
