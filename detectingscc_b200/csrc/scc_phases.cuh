// Phases of the four SCC drivers (vHong / wHong, scc_WCC.cu:53-998; vSlota /
// wSlota, scc_Coloring.cu:6-701), rewritten as work-list passes over a
// persistent launch.  Each phase cites the reference kernel whose result it
// reproduces; the schedules differ (frontier queues instead of full-V
// sweeps, device-side convergence instead of a host round trip per level).
#pragma once
#include "scc_device.cuh"

namespace sccb {

// A vertex list.
struct VList {
    const uint32_t *p;
    uint32_t n;
};

// Four consecutive entries of a list for this lane (entries i0 .. i0+3): one
// 128-bit load (list buffers are 256-byte aligned).
__device__ __forceinline__ void load_list4(const VList &src, uint32_t i0, uint32_t (&v)[4], bool (&ok)[4])
{
    if (i0 + 3u < src.n) {
        const uint4 x = *reinterpret_cast<const uint4 *>(src.p + i0);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        ok[0] = ok[1] = ok[2] = ok[3] = true;
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        ok[j] = i0 + (uint32_t)j < src.n;
        v[j] = ok[j] ? src.p[i0 + (uint32_t)j] : 0u;
    }
}

template <class Ex>
__device__ __forceinline__ void count_edges(Ex &ex, unsigned warp_total)
{
    if constexpr (Ex::instr) {
        if (lane_id() == 0 && warp_total) atomicAdd(&ex.ctl->t_edges, (unsigned long long)warp_total);
    }
}
template <class Ex>
__device__ __forceinline__ void count_verts(Ex &ex, bool valid)
{
    if constexpr (Ex::instr) {
        unsigned m = __ballot_sync(FULL, valid);
        if (lane_id() == 0 && m) atomicAdd(&ex.ctl->t_verts, (unsigned long long)__popc(m));
    }
}
template <class Ex>
__device__ __forceinline__ void count_verts_n(Ex &ex, unsigned n)
{
    if constexpr (Ex::instr) {
        n = __reduce_add_sync(FULL, n);
        if (lane_id() == 0 && n) atomicAdd(&ex.ctl->t_verts, (unsigned long long)n);
    }
}

// Passes that a search or a spread of colours can take: at most V hops, each
// one pass, or two where the vertex is heavy (one cuts its list, the next
// walks the chunks).
__device__ __forceinline__ uint32_t max_levels(uint32_t V) { return 2u * V + 4u; }

// Vertices a warp takes at once from a list of n (1 << item_shift): the smallest power of two
// that still gives every warp at most one item, at most 32.  A level's time
// is the chain of dependent accesses of its longest item, so a short list is
// spread over all warps before lanes are filled.
template <class Ex>
__device__ __forceinline__ uint32_t item_shift(const Ex &ex, uint32_t n)
{
    const uint32_t nw = ex.nwarps();
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < 5; i++) s += (n + (1u << s) - 1u) >> s > nw ? 1u : 0u;
    return s;
}
template <class Ex>
__device__ __forceinline__ uint32_t item_group(const Ex &ex, uint32_t n)
{
    return 1u << item_shift(ex, n);
}

// Rounds that a warp goes on for by itself at the end of its items of a
// pass: it takes what it just appended off its own staging slice (the newest
// 32) and expands that, while the slice holds at most local_cap entries and
// it walked fewer than LOCAL_EDGES arcs.  A
// search does not depend on the order its vertices are expanded in, so a
// pass need not be one level: a high-diameter graph takes a tenth of the
// barriers, and a vertex's neighbours are expanded while their sectors are
// still cached.  A level-synchronous pass costs 6 to 7 us on the whole GPU
// whatever the frontier (queue entry, offsets, arcs, state, claim, append,
// flush, barrier), a local round 3 to 4.  701^2 grid, vHong: 125 levels in
// 0.93 ms, now 8 passes in 0.40 ms; 50,021-vertex random graph of degree 4:
// 13 levels in 88 us, now 2 passes in 48 us; 4096^2 grid: 163 levels in
// 2.95 ms, now 15 passes in 2.28 ms (bound by the latency of scattered
// sectors: DRAM and issue slots are each below 25 % busy).  Longer slices, and what is left after the last round, go
// to the global queue and are spread over all warps by the next pass.
// Until there is work for every warp (full) only short slices stay: a warp
// whose slice grows fast shares it.
constexpr uint32_t LOCAL_ROUNDS = 16, LOCAL_EDGES = 4096;   // of the first search
constexpr uint32_t PEEL_ROUNDS = 8;     // of the peels
__device__ __forceinline__ uint32_t local_cap(uint32_t qcap, bool full = false)
{
    return full && qcap > 256u ? qcap - 128u : min(96u, qcap / 2u);
}

// Where they do not (spreads): a search that grows fast has few levels to
// merge, and a warp that goes on with its finds runs past the level that would
// go bottom-up and walks, top-down and on its own, what all would share.
// fwd, bwd: arcs of the next level, if all but one arc a vertex of this one
// find a new vertex; grow: arcs a vertex less one.  A pass stays one level
// when the next is work for every warp and the one after it would be
// bottom-up (batched graphs, whose passes are cheaper: a quarter of that).
// Random graphs, 2M vertices of degree 5 and 12, vSlota: 495 -> 290 and
// 309 -> 224 us; one CTA, 8,000 of degree 8: 159 -> 98 us; 600 of up to 4,096
// of degree 12 at once: 249 -> 143 us.  grow is 2.4 on the grids and their
// passes stay long.
constexpr float SPREAD_ARCS = 256.0f;   // of a level, a warp: two steps of a walk
template <class Ex>
__device__ __forceinline__ bool spreads(const Ex &ex, float fwd, float bwd, float grow, float bottom_up)
{
    return fwd + bwd > SPREAD_ARCS * (float)ex.nwarps() &&
           fmaxf(fwd, bwd) * grow > (Ex::grid ? bottom_up : 0.25f * bottom_up);
}

// Bits 0, 4, ..., 28 of a nibble word as bits 0 .. 7.
__device__ __forceinline__ uint32_t nib8(uint32_t m)
{
    m &= NIBS;
    m = (m | m >> 3) & 0x03030303u;
    m = (m | m >> 6) & 0x000F000Fu;
    return (m | m >> 12) & 0xFFu;
}
// The live, forward- and backward-visited bits of a unit: the 32 vertices
// 32 * u .. 32 * u + 31, four nibble words (units are whole: ph_init writes
// the words past V as zero).
struct NibUnit {
    uint32_t live, fwd, bwd;
};
__device__ __forceinline__ NibUnit load_unit(const Work &w, bool in, uint32_t u)
{
    const uint4 x = in ? *reinterpret_cast<const uint4 *>(w.nb + 4u * u) : make_uint4(0u, 0u, 0u, 0u);
    auto four = [&](int k) { return nib8(x.x >> k) | nib8(x.y >> k) << 8 | nib8(x.z >> k) << 16 | nib8(x.w >> k) << 24; };
    return NibUnit{four(0), four(1), four(2)};
}
// Units a warp takes at once: all V / 32 are dealt out in as few equal rounds
// as 32 a warp allow.  Marks are walked 64 a step, and the last step of an
// item is rarely full, so few large items take fewer steps than many small
// ones.  Items of about 64 marks, R-MAT scale 21: the first bottom-up step
// 66 us, now 44; scale 22 91 and now 75 us, whole run 199 and now 184 us.
template <class Ex>
__device__ __forceinline__ uint32_t unit_group(const Ex &ex, uint32_t V)
{
    const uint32_t nu = V / 32u + 1u, nw = ex.nwarps(), rounds = (nu + 32u * nw - 1u) / (32u * nw);
    return (nu + rounds * nw - 1u) / (rounds * nw);
}

// Walks the marked vertices (mask m of each lane's unit u), 64 at a time:
// fn(ok[2], v[2], unit's lane[2]) is called by all lanes.  Marks are packed
// into full lanes, so a sparse unit costs its marks, not its width.
template <class Fn>
__device__ __forceinline__ void unit_walk2(uint32_t u, uint32_t m, Fn &&fn)
{
    const unsigned c = __popc(m), incl = warp_incl_scan(c), total = __shfl_sync(FULL, incl, 31), excl = incl - c;
    for (unsigned base = 0; base < total; base += 64u) {
        bool ok[2];
        uint32_t v[2];
        unsigned own[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const unsigned e = base + 32u * (unsigned)h + lane_id();
            unsigned lo = 0;
#pragma unroll
            for (unsigned step = 16; step >= 1; step >>= 1) {
                const unsigned x = __shfl_sync(FULL, excl, (lo + step) & 31u);
                if (lo + step < 32u && x <= e) lo += step;
            }
            uint32_t mo = __shfl_sync(FULL, m, lo), k = e - __shfl_sync(FULL, excl, lo), at = 0;
            const uint32_t uo = __shfl_sync(FULL, u, lo);
#pragma unroll
            for (unsigned b = 16; b >= 1; b >>= 1) {   // the k-th set bit
                const uint32_t n = __popc(mo & ((1u << b) - 1u));
                if (k >= n) {
                    k -= n;
                    mo >>= b;
                    at += b;
                }
            }
            ok[h] = e < total;
            v[h] = ok[h] ? uo * 32u + at : 0u;
            own[h] = lo;
        }
        fn(ok, v, own);
    }
}

// Does each of the lane's four lists hold a vertex u with (nibble(u) & m) ==
// want?  Lists 0 and 2 lie in (Br, Bc), 1 and 3 in (Fr, Fc); mr, mf are their
// masks.  Every lane keeps its four searches in flight, two entries per step,
// so it waits on one round of gathers for all of them; of a list longer than
// pull_lane the lane tests the first entries (a hit is usually among them)
// and the whole warp the rest.  Bit t of the result: list t has one.
template <class Ex>
__device__ __forceinline__ uint32_t find4(Ex &ex, const Graph &g, const Work &w, uint32_t (&pos)[4],
                                          const uint32_t (&end)[4], uint32_t mr, uint32_t mf,
                                          const uint32_t (&want)[4])
{
    unsigned scanned = 0;
    uint32_t lim[4], found = 0u, on = 0u;
    const uint32_t first = min(8u, w.pull_lane);
#pragma unroll
    for (int t = 0; t < 4; t++) {
        on |= end[t] > pos[t] ? 1u << t : 0u;
        lim[t] = end[t] - pos[t] <= w.pull_lane ? end[t] : pos[t] + first;
    }
    const uint32_t any = on;
    while (on) {
        uint32_t c0[4], c1[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const uint32_t *C = (t & 1) ? g.Fc : g.Bc;
            const bool o = (on >> t) & 1u;
            c0[t] = o ? __ldg(&C[pos[t]]) : 0u;
            c1[t] = o && pos[t] + 1u < end[t] ? __ldg(&C[pos[t] + 1u]) : 0u;
        }
#pragma unroll
        for (int t = 0; t < 4; t++) {
            if (!((on >> t) & 1u)) continue;
            const uint32_t m = (t & 1) ? mf : mr;
            const bool two = pos[t] + 1u < end[t];
            const uint32_t a = nib_of(w.nb, guard_id(c0[t], g.V, ex.ctl));
            const uint32_t b = two ? nib_of(w.nb, guard_id(c1[t], g.V, ex.ctl)) : 0u;
            if constexpr (Ex::instr) scanned += two ? 2u : 1u;
            if ((a & m) == want[t] || (two && (b & m) == want[t])) {
                found |= 1u << t;
                on &= ~(1u << t);
            } else {
                pos[t] += 2u;
                if (pos[t] >= lim[t]) on &= ~(1u << t);
            }
        }
    }
    // the rest of long lists by the whole warp, one search at a time
#pragma unroll
    for (int t = 0; t < 4; t++) {
        unsigned hm = __ballot_sync(FULL, ((any & ~found) >> t & 1u) && end[t] > pos[t]);
        const uint32_t *C = (t & 1) ? g.Fc : g.Bc;
        const uint32_t m = (t & 1) ? mf : mr;
        while (hm) {
            const unsigned j = __ffs(hm) - 1u;
            hm &= hm - 1u;
            const uint32_t bj = __shfl_sync(FULL, pos[t], j), ej = __shfl_sync(FULL, end[t], j);
            const uint32_t wj = __shfl_sync(FULL, want[t], j);
            for (uint32_t b = bj; b < ej; b += 32u) {
                const uint32_t e = b + lane_id();
                const bool hit = e < ej && (nib_of(w.nb, guard_id(__ldg(&C[e]), g.V, ex.ctl)) & m) == wj;
                if constexpr (Ex::instr) scanned += lane_id() == 0 ? min(32u, ej - b) : 0u;
                if (__ballot_sync(FULL, hit)) {
                    if (lane_id() == j) found |= 1u << t;
                    break;
                }
            }
        }
    }
    if constexpr (Ex::instr) count_edges(ex, __reduce_add_sync(FULL, scanned));
    return found;
}

// ---------------------------------------------------------------------
// init: every vertex live (the reference's cudaMemset of range and tags,
// scc_WCC.cu:630-631), or, with trim, every vertex that has an in- and an
// out-arc: with every vertex live the first trim-1 sweep is decided by the
// degrees alone (scc_kernels.cu:187-233).  Eight ids per lane, one nibble
// word: 128-bit offset loads, half a byte written per vertex.  Also checks
// the offsets (the reference layout: Fr[0] = Fr[1] = 0, non-decreasing,
// Fr[V+1] = E, load.cpp:55-77; same for Br) and sets the error before the
// barrier, so no later pass runs on a bad graph; counts the live vertices
// (C_LIST) and folds the first pivot's key over them.  What bounds it is
// reading the offsets; a trimmed vertex's label is its own id and is not
// written here (nibble 0).  R-MAT scale 22: with a state word, a label and a
// live list written per vertex 21.8 us, now 12.4 us (33.5 MB of offsets).
// ---------------------------------------------------------------------
template <class Ex>
__device__ bool ph_init(Ex &ex, const Graph &g, const Work &w, bool trim, bool stamps)
{
    return run_pass(ex, PH_INIT, [&](unsigned, unsigned nxt) {
        if (ex.leader() && (g.Fr[0] != 0u || g.Fr[1] != 0u || g.Br[0] != 0u || g.Br[1] != 0u ||
                            g.Fr[g.V + 1] != g.E || g.Br[g.V + 1] != g.E))
            set_error(ex.ctl, E_BAD_GRAPH, 62);
        unsigned long long best = 0;
        uint32_t dmax = 0, nlive = 0, ntrim = 0, nv = 0;
        bool bad = false;
        const uint32_t nwords = (g.V / 32u + 1u) * 4u;   // whole units
        for (uint32_t wd = ex.tid(); wd < nwords; wd += ex.nthr()) {
            const uint32_t i0 = wd * 8u;
            uint32_t x = 0;
            if (i0 > g.V) {
                w.nb[wd] = 0u;
                continue;
            }
#pragma unroll
            for (uint32_t q = 0; q < 2u; q++) {
                uint32_t f[5], b[5];
                load_off5(g.Fr, i0 + 4u * q, g.V, g.vec, f);
                load_off5(g.Br, i0 + 4u * q, g.V, g.vec, b);
#pragma unroll
                for (uint32_t j = 0; j < 4u; j++) {
                    const uint32_t v = i0 + 4u * q + j;
                    if (v < 1u || v > g.V) continue;
                    bad |= f[j] > f[j + 1] || b[j] > b[j + 1];
                    const uint32_t out = f[j + 1] - f[j], in = b[j + 1] - b[j];
                    dmax = max(dmax, max(out, in));
                    if (trim && (out == 0u || in == 0u)) {
                        ntrim++;
                        continue;
                    }
                    nlive++;
                    x |= NL << (16u * q + 4u * j);
                    const unsigned long long k = ((unsigned long long)(out * in) << 32) | (0xFFFFFFFFu - v);
                    best = k > best ? k : best;
                }
            }
            w.nb[wd] = x;
            if (stamps && x) {   // trim-1 work lists stamp the live vertices
                if (i0 + 7u <= g.V) {
                    *reinterpret_cast<uint4 *>(w.st + i0) = make_uint4(0u, 0u, 0u, 0u);
                    *reinterpret_cast<uint4 *>(w.st + i0 + 4u) = make_uint4(0u, 0u, 0u, 0u);
                } else {
                    for (uint32_t i = i0; i <= g.V; i++) w.st[i] = 0u;
                }
            }
            nv += min(8u, g.V + 1u - i0);
        }
        if (bad) set_error(ex.ctl, E_BAD_GRAPH, 61);
        count_verts_n(ex, nv);
        bq_add_edges(0, nlive);
        bq_add_edges(1, ntrim);
        block_max_atomic(best, &w.pivkey[0], dmax, Ex::grid ? &ex.ctl->maxdeg : nullptr);
        if (threadIdx.x == 0) {
            if (sccb_dsmem[12]) atomicAdd(&ex.lc(nxt)[C_LIST], sccb_dsmem[12]);
            if (sccb_dsmem[13]) atomicAdd(&ex.ctl->n_trim1, (unsigned long long)sccb_dsmem[13]);
            sccb_dsmem[12] = sccb_dsmem[13] = 0u;
        }
    });
}

// ---------------------------------------------------------------------
// trim1 iterated to its fixpoint (vHong / wHong, scc_WCC.cu:680-687,
// :773-780, :808-815).  Pass 0 checks every live vertex (all: by id, off the
// nibble units, n of them) or a list; a trimmed vertex queues its live neighbours of the
// same class for the next pass (stamped with the pass, so none is listed
// twice; a vertex that is being checked meanwhile is listed all the same),
// so later passes only recheck vertices that lost a neighbour.  A vertex is checked by searching both its lists for one live
// neighbour, as in a bottom-up step: the first entries usually hold one.
// Checking the live vertices instead of walking the lists of the vertices
// that the degrees trim, R-MAT scale 20 with permuted ids (602,000 of
// 1,048,576 trimmed): 58 us for the first pass,
// now 21 us.
// ---------------------------------------------------------------------
template <class Ex>
__device__ __forceinline__ void trim1_check(Ex &ex, const Graph &g, const Work &w, const bool (&in)[2],
                                            const uint32_t (&v)[2], unsigned par, unsigned nxt)
{
    uint32_t s[2], pos[4], end[4], want[4];
    bool ok[2];
#pragma unroll
    for (int h = 0; h < 2; h++) s[h] = in[h] ? nib_of(w.nb, v[h]) : 0u;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        ok[h] = (s[h] & NL) != 0u;
        pos[2 * h] = ok[h] ? __ldg(&g.Br[v[h]]) : 0u;
        end[2 * h] = ok[h] ? __ldg(&g.Br[v[h] + 1u]) : 0u;
        pos[2 * h + 1] = ok[h] ? __ldg(&g.Fr[v[h]]) : 0u;
        end[2 * h + 1] = ok[h] ? __ldg(&g.Fr[v[h] + 1u]) : 0u;
        want[2 * h] = want[2 * h + 1] = s[h] & NCLASS;
        count_verts(ex, in[h]);
    }
    const uint32_t found = find4(ex, g, w, pos, end, NCLASS, NCLASS, want);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const bool trim = ok[h] && (found >> (2 * h) & 3u) != 3u;
        const unsigned m = __ballot_sync(FULL, trim);
        if (m == 0u) continue;
        if (trim) {
            nib_kill(w.nb, v[h]);
            w.label[v[h]] = v[h] | LBL_SELF;
        }
        if (lane_id() == 0) atomicAdd(&ex.ctl->n_trim1, (unsigned long long)__popc(m));
        const uint32_t r = s[h] & NCLASS, tag = ex.gl + 1u;
        // its live neighbours lost an in- or out-neighbour: the warp walks
        // all the lists together, 64 entries per step
        auto fn2 = [&](bool v0, uint32_t u0, uint32_t r0, bool v1, uint32_t u1, uint32_t r1) {
            if (v0) u0 = guard_id(u0, g.V, ex.ctl);
            if (v1) u1 = guard_id(u1, g.V, ex.ctl);
            const bool p0 = v0 && (nib_of(w.nb, u0) & NCLASS) == r0 && stamp_claim(w.st, u0, tag);
            const bool p1 = v1 && (nib_of(w.nb, u1) & NCLASS) == r1 && stamp_claim(w.st, u1, tag);
            bq_push(0, p0, u0, w.qcap, w.Q[0][par], &ex.lc(nxt)[C_FQ], g.V, ex.ctl, 11);
            bq_push(0, p1, u1, w.qcap, w.Q[0][par], &ex.lc(nxt)[C_FQ], g.V, ex.ctl, 11);
        };
#pragma unroll
        for (int dir = 0; dir < 2; dir++) {
            const uint32_t *R = dir ? g.Br : g.Fr;
            const uint32_t *C = dir ? g.Bc : g.Fc;
            const uint32_t beg = trim ? __ldg(&R[v[h]]) : 0u;
            const uint32_t deg = trim ? __ldg(&R[v[h] + 1]) - beg : 0u;
            count_edges(ex, lbs_expand2(beg, deg, r, C, fn2));
        }
    }
}

// (all is a parameter of its own: with the choice made by the list's pointer
// the three calls share code that spills, one CTA and 1,024 vertices 104 -> 115 us)
template <class Ex>
__device__ bool ph_trim1_fix(Ex &ex, const Graph &g, const Work &w, VList src0, bool all)
{
    uint32_t nq = src0.n;
    for (unsigned it = 0;; it++) {
        if (it > g.V + 2u) { if (ex.leader()) set_error(ex.ctl, E_NOT_CONVERGED, 30); return false; }
        const bool ok = run_pass(ex, PH_TRIM1_FIX, [&](unsigned, unsigned nxt) {
            const unsigned par = ex.gl & 1u;
            if (all && it == 0u) {
                const uint32_t nu = g.V / 32u + 1u, cu = unit_group(ex, g.V), ni = (nu + cu - 1u) / cu;
                for (uint32_t i = ex.wid(); i < ni; i += ex.nwarps()) {
                    const uint32_t u = lane_id() * ni + i;
                    unit_walk2(u, load_unit(w, lane_id() < cu && u < nu, u).live,
                               [&](const bool (&in)[2], const uint32_t (&v)[2], const unsigned (&)[2]) {
                                   trim1_check(ex, g, w, in, v, par, nxt);
                               });
                }
            } else {
                const uint32_t *src = it == 0u ? src0.p : w.Q[0][par ^ 1u];
                const uint32_t gs = item_group(ex, (nq + 1u) / 2u);
                for (uint32_t base = ex.wid() * 2u * gs; base < nq; base += ex.nwarps() * 2u * gs) {
                    bool in[2];
                    uint32_t v[2];
#pragma unroll
                    for (uint32_t h = 0; h < 2u; h++) {
                        const uint32_t i = base + h * gs + lane_id();
                        in[h] = lane_id() < gs && i < nq;
                        v[h] = in[h] ? src[i] : 0u;
                    }
                    trim1_check(ex, g, w, in, v, par, nxt);
                }
            }
            bq_flush(1, w.qcap, w.Q[0][par], &ex.lc(nxt)[C_FQ], nullptr, nullptr, g.V, ex.ctl);
        });
        if (!ok) return false;
        nq = last_count(ex, C_FQ);
        if (nq == 0u) return true;
    }
}

// Up to two live neighbours of x in class r in (R, C); *first gets the first
// one (scc_kernels.cu:250-261).
__device__ __forceinline__ uint32_t count_upto2(const uint32_t *nb, const uint32_t *__restrict__ R,
                                                const uint32_t *__restrict__ C, uint32_t x,
                                                uint32_t r, uint32_t *first, uint32_t V, Ctl *ctl)
{
    uint32_t n = 0;
    for (uint32_t e = __ldg(&R[x]), end = __ldg(&R[x + 1]); e < end; e++) {
        uint32_t u = guard_id(__ldg(&C[e]), V, ctl);
        if ((nib_of(nb, u) & NCLASS) == r) {
            n++;
            if (n == 2u) break;
            if (first) *first = u;
        }
    }
    return n;
}

// trim2 decision for v (scc_kernels.cu:236-348): the partner k, possibly v
// itself through a self-loop, or 0.
__device__ __forceinline__ uint32_t trim2_partner(const Graph &g, const uint32_t *nb, uint32_t v, uint32_t r, Ctl *c)
{
    uint32_t k = 0;
    if (count_upto2(nb, g.Br, g.Bc, v, r, &k, g.V, c) == 1u) {
        for (uint32_t e = __ldg(&g.Fr[v]), end = __ldg(&g.Fr[v + 1]); e < end; e++) {
            if (__ldg(&g.Fc[e]) == k) {
                if (count_upto2(nb, g.Br, g.Bc, k, r, nullptr, g.V, c) == 1u) return k;
                break;
            }
        }
    }
    k = 0;
    if (count_upto2(nb, g.Fr, g.Fc, v, r, &k, g.V, c) == 1u) {
        for (uint32_t e = __ldg(&g.Br[v]), end = __ldg(&g.Br[v + 1]); e < end; e++) {
            if (__ldg(&g.Bc[e]) == k) {
                if (count_upto2(nb, g.Fr, g.Fc, k, r, nullptr, g.V, c) == 1u) return k;
                break;
            }
        }
    }
    return 0;
}

// ---------------------------------------------------------------------
// trim2 once, decided on the state before the pass (scc_WCC.cu:792-793,
// scc_kernels.cu:236-357).  Both members are marked; the pair counts once,
// on its smaller id.  The reference marks both members with unsynchronised
// byte writes (scc_kernels.cu:350-354) and can lose the trim2 tag.
// ---------------------------------------------------------------------
template <class Ex>
__device__ bool ph_trim2(Ex &ex, const Graph &g, const Work &w, VList src)
{
    bool ok = run_pass(ex, PH_TRIM2, [&](unsigned, unsigned nxt) {
        const unsigned par = ex.gl & 1u;
        const uint32_t gs = item_group(ex, src.n);
        for (uint32_t base = ex.wid() * gs; base < src.n; base += ex.nwarps() * gs) {
            uint32_t i = base + lane_id();
            bool valid = lane_id() < gs && i < src.n, hit = false, cnt = false;
            uint32_t v = valid ? src.p[i] : 0u;
            if (valid) {
                const uint32_t s = nib_of(w.nb, v);
                if (s & NL) {
                    uint32_t k = trim2_partner(g, w.nb, v, s & NCLASS, ex.ctl);
                    if (k) {
                        hit = true;
                        cnt = v <= k;
                        w.label[v] = (v < k ? v : k) | LBL_SELF;
                    }
                }
            }
            count_verts(ex, valid);
            unsigned m = __ballot_sync(FULL, cnt);
            if (lane_id() == 0 && m) atomicAdd(&ex.ctl->n_trim2, (unsigned long long)__popc(m));
            bq_push(0, hit, v, w.qcap, w.Q[0][par], &ex.lc(nxt)[C_LIST], g.V, ex.ctl, 12);
        }
        bq_flush(1, w.qcap, w.Q[0][par], &ex.lc(nxt)[C_LIST], nullptr, nullptr, g.V, ex.ctl);
    });
    if (!ok) return false;
    const uint32_t nT = last_count(ex, C_LIST);
    if (nT == 0u) return true;
    return run_pass(ex, PH_TRIM2_APPLY, [&](unsigned, unsigned) {
        const uint32_t *T = w.Q[0][(ex.gl & 1u) ^ 1u];
        for (uint32_t i = ex.tid(); i < nT; i += ex.nthr()) nib_kill(w.nb, T[i]);
    });
}

// ---------------------------------------------------------------------
// The first FW-BW search (fwd/bwd, scc_kernels.cu:360-445, and
// fwd_warp/bwd_warp, include/scc_kernels.h:46-105) over queues instead of
// full sweeps.  Every vertex is in one range, so an arc is decided by half a
// byte of its neighbour: live, and not yet visited in this direction; it is
// claimed with atomicOr and appended to the next frontier (warp ballot
// compaction).  At eight vertices a word the states of 16.8M vertices take
// 8.4 MB and stay in L2 (a 32-bit word each: 67 MB, most gathers a DRAM
// sector).  Vertices with more than HEAVY_T entries are cut into CH-entry
// chunks for the next pass.
//
// K arcs per lane: all gathers, then all claims are issued before any
// append.  eager (a short frontier, where a level's time is its chain of
// dependent accesses): the claim is made without looking first, and the
// offsets of the vertex are brought into L1 beside it, for the warp that goes
// on with it.  This sets visited bits on trimmed vertices too.  They mean
// nothing there: a bottom-up step takes a visited neighbour as one reached
// through live vertices, and a trimmed vertex never lies between two live ones
// (it has no live in-neighbour or no live out-neighbour, by its degrees or by
// trim-1 to its fixpoint).  The step tests the live bit all the same, which
// costs nothing.  cnt (uniform over the CTA) adds the claimed vertices'
// degrees to the pass's frontier-edge tally; a pass whose claims are not
// expected to reach the bottom-up threshold skips those offset gathers.
// ---------------------------------------------------------------------
template <int K, class Ex>
__device__ __forceinline__ void bfs_visit(Ex &ex, const Graph &g, const Work &w, int dir, const bool (&v)[K],
                                          uint32_t (&n)[K], unsigned par, unsigned nxt, bool cnt, bool eager = false)
{
    const uint32_t bit = dir ? NB : NF;
    const uint32_t *Rn = dir ? g.Br : g.Fr;
    uint32_t x[K];
    bool c[K];
#pragma unroll
    for (int j = 0; j < K; j++) {
        if (v[j]) n[j] = guard_id(n[j], g.V, ex.ctl);
        x[j] = !v[j] ? 0u : eager ? NL : nib_of(w.nb, n[j]);
    }
#pragma unroll
    for (int j = 0; j < K; j++) {
        const bool t = (x[j] & (bit | NL)) == NL;
        x[j] = t ? nib_or(w.nb, n[j], bit) : bit;
        if (t && eager) prime_l1(Rn + n[j]);
    }
#pragma unroll
    for (int j = 0; j < K; j++) c[j] = (x[j] & (bit | NL)) == NL;
    if (cnt) {   // edges the claimed vertices will expand next (direction-switch rule)
        unsigned e = 0;
#pragma unroll
        for (int j = 0; j < K; j++)
            if (c[j]) e += __ldg(&Rn[n[j] + 1]) - __ldg(&Rn[n[j]]);
        bq_add_edges((unsigned)dir, e);
    }
    bq_pushK<K>((unsigned)dir, c, n, w.qcap, w.Q[dir][par], &ex.lc(nxt)[C_FQ + dir], g.V, ex.ctl, 13);
}

template <class Ex>
__device__ __forceinline__ void bfs_visit2(Ex &ex, const Graph &g, const Work &w, int dir, bool v0, uint32_t n0,
                                           bool v1, uint32_t n1, unsigned par, unsigned nxt, bool cnt)
{
    const bool v[2] = {v0, v1};
    uint32_t n[2] = {n0, n1};
    bfs_visit<2>(ex, g, w, dir, v, n, par, nxt, cnt);
}

// Frontier vertices, one per lane.  Lists of at most LANE_DEG entries are
// walked by their own lanes, four entries a step (a low-degree frontier is
// done in one or two rounds of gathers and needs no owner search); a warp
// that holds a longer list, or at most 128 entries in all, walks the
// concatenation of its lists, 128 entries a step.
constexpr uint32_t LANE_DEG = 8;
template <class Ex>
__device__ __forceinline__ uint32_t bfs_expand_lanes(Ex &ex, const Graph &g, const Work &w, int dir, bool act,
                                                     uint32_t v, unsigned par, unsigned nxt, bool cnt, bool eager,
                                                     bool local = false)
{
    const uint32_t *R = dir ? g.Br : g.Fr;
    const uint32_t *C = dir ? g.Bc : g.Fc;
    const uint32_t beg = act ? __ldg(&R[v]) : 0u;
    uint32_t deg = act ? __ldg(&R[v + 1u]) - beg : 0u;
    count_verts(ex, act);
    const uint32_t maxd = __reduce_max_sync(FULL, deg), total = __reduce_add_sync(FULL, deg);
    if (cnt && local && lane_id() == 0) atomicSub(&sccb_dsmem[12 + dir], total);   // not in the next frontier any more
    if (maxd <= LANE_DEG && (maxd <= 4u || total > 128u)) {
        for (uint32_t k = 0; k < maxd; k += 4u) {
            bool ok[4];
            uint32_t n[4];
#pragma unroll
            for (uint32_t j = 0; j < 4u; j++) {
                ok[j] = k + j < deg;
                n[j] = ok[j] ? __ldg(&C[beg + k + j]) : 0u;
            }
            bfs_visit<4>(ex, g, w, dir, ok, n, par, nxt, cnt, eager);
        }
        count_edges(ex, total);
        return total;
    }
    if (maxd > HEAVY_T) {
        const bool heavy = deg > HEAVY_T;
        warp_push_chunks(v, heavy ? (deg + CH - 1u) / CH : 0u, w.H[dir][par], &ex.lc(nxt)[C_FH + dir], w.hcap, ex.ctl);
        if (heavy) deg = 0u;
    }
    count_edges(ex, lbs_walk4(beg, deg, C, [&](const bool (&ok)[4], uint32_t (&n)[4], const unsigned (&)[4]) {
        bfs_visit<4>(ex, g, w, dir, ok, n, par, nxt, cnt, eager);
    }));
    return total;
}

// Top-down expansion with the virtual-warp schedule (W = 1 << lw lanes per
// vertex, the reference's fwd_warp/bwd_warp), VWK frontier vertices per
// lane group in the same steps.
constexpr int VWK = 4;
template <class Ex>
__device__ __forceinline__ void bfs_expand_vwk(Ex &ex, const Graph &g, const Work &w, int dir,
                                               const uint32_t (&v)[VWK], const bool (&act)[VWK], int lw, unsigned par,
                                               unsigned nxt, bool cnt)
{
    const uint32_t *R = dir ? g.Br : g.Fr;
    const uint32_t *C = dir ? g.Bc : g.Fc;
    const bool lead = (lane_id() & ((1u << lw) - 1u)) == 0u;
    uint32_t beg[VWK], deg[VWK];
#pragma unroll
    for (int j = 0; j < VWK; j++) {
        beg[j] = act[j] ? __ldg(&R[v[j]]) : 0u;
        deg[j] = act[j] ? __ldg(&R[v[j] + 1]) - beg[j] : 0u;
    }
#pragma unroll
    for (int j = 0; j < VWK; j++) {
        const bool heavy = deg[j] > HEAVY_T;
        warp_push_chunks(v[j], heavy && lead ? (deg[j] + CH - 1u) / CH : 0u, w.H[dir][par],
                         &ex.lc(nxt)[C_FH + dir], w.hcap, ex.ctl);
        if (heavy) deg[j] = 0u;
    }
    auto fn = [&](int, bool v0, uint32_t n0, bool v1, uint32_t n1) {
        bfs_visit2(ex, g, w, dir, v0, n0, v1, n1, par, nxt, cnt);
    };
    count_edges(ex, vw_expandK<VWK>(beg, deg, (unsigned)lw, C, fn));
}

// One CH-entry chunk of a heavy vertex, expanded by the whole warp:
// fn(v0, n0, v1, n1).
template <class Ex, class Fn>
__device__ __forceinline__ void chunk_expand(Ex &ex, const uint32_t *__restrict__ R, const uint32_t *__restrict__ C,
                                             uint2 hc, Fn &&fn)
{
    uint32_t beg = __ldg(&R[hc.x]) + hc.y * CH;
    uint32_t end = min(__ldg(&R[hc.x + 1]), beg + CH);
    for (uint32_t k = lane_id(); k < CH; k += 64u) {
        const uint32_t e0 = beg + k, e1 = e0 + 32u;
        const bool v0 = e0 < end, v1 = e1 < end;
        const uint32_t n0 = v0 ? __ldg(&C[e0]) : 0u;
        const uint32_t n1 = v1 ? __ldg(&C[e1]) : 0u;
        fn(v0, n0, v1, n1);
    }
    count_edges(ex, end > beg ? end - beg : 0u);
}

// Bottom-up step over the warp's units, both directions at once: every live
// vertex still unvisited in a direction that goes bottom-up (puf forward,
// pub backward) searches its lists for a visited neighbour.  The nibbles name
// those vertices by themselves, so no scope list is kept or walked.  The live
// vertices still unvisited in some direction are tallied (C_SCOPE): the scope
// the next pass weighs its frontier against.
template <class Ex>
__device__ __forceinline__ void bfs_pull(Ex &ex, const Graph &g, const Work &w, bool puf, bool pub, uint32_t u,
                                         const NibUnit &x, unsigned par, unsigned nxt)
{
    const uint32_t wf = puf ? x.live & ~x.fwd : 0u, wb = pub ? x.live & ~x.bwd : 0u;
    uint32_t left = __popc(x.live & ~(x.fwd & x.bwd));
    unit_walk2(u, wf | wb, [&](const bool (&in)[2], const uint32_t (&v)[2], const unsigned (&own)[2]) {
        uint32_t pos[4], end[4];
        const uint32_t want[4] = {NL | NF, NL | NB, NL | NF, NL | NB};
        bool half[2];   // already visited the other way
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t b = v[h] & 31u;
            const bool nf = in[h] & (__shfl_sync(FULL, wf, own[h]) >> b);   // forward: a visited in-neighbour
            const bool nb = in[h] & (__shfl_sync(FULL, wb, own[h]) >> b);   // backward: a visited out-neighbour
            half[h] = (__shfl_sync(FULL, x.fwd | x.bwd, own[h]) >> b) & 1u;
            pos[2 * h] = nf ? __ldg(&g.Br[v[h]]) : 0u;
            end[2 * h] = nf ? __ldg(&g.Br[v[h] + 1u]) : 0u;
            pos[2 * h + 1] = nb ? __ldg(&g.Fr[v[h]]) : 0u;
            end[2 * h + 1] = nb ? __ldg(&g.Fr[v[h] + 1u]) : 0u;
        }
        const uint32_t found = find4(ex, g, w, pos, end, NL | NF, NL | NB, want);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const bool ff = found >> (2 * h) & 1u, fb = found >> (2 * h + 1) & 1u;
            if (ff || fb) {
                nib_or(w.nb, v[h], (ff ? NF : 0u) | (fb ? NB : 0u));
                if ((ff && fb) || half[h]) left--;
            }
            // frontier edges of the next level: out-degree forward, in-degree backward
            if (puf) bq_add_edges(0u, ff ? __ldg(&g.Fr[v[h] + 1u]) - __ldg(&g.Fr[v[h]]) : 0u);
            if (pub) bq_add_edges(1u, fb ? __ldg(&g.Br[v[h] + 1u]) - __ldg(&g.Br[v[h]]) : 0u);
            count_verts(ex, in[h]);
            if (puf) bq_push(0u, ff, v[h], w.qcap, w.Q[0][par], &ex.lc(nxt)[C_FQ], g.V, ex.ctl, 19);
            if (pub) bq_push(1u, fb, v[h], w.qcap, w.Q[1][par], &ex.lc(nxt)[C_BQ], g.V, ex.ctl, 19);
        }
    });
    bq_add_edges(2u, left);
}

// Forward and backward reachability from the first pivot p to closure.  Pass
// 0 flags the pivot and expands it.  Each later pass picks, per direction,
// top-down (expand the frontier queue and the heavy chunks) or bottom-up
// (scan the unvisited live vertices) when the frontier's vertices have more
// than bu_k * nscope edges to expand; nscope is the live count, and after
// the first bottom-up step what that left unvisited.  lw < 0 selects the
// warp schedule for top-down steps, lw >= 0 the virtual-warp schedule with
// W = 1 << lw.
template <class Ex>
__device__ bool ph_bfs(Ex &ex, const Graph &g, const Work &w, uint32_t p, int lw, uint32_t nscope)
{
    bool shrunk = false;
    const float degree = (float)g.E / (float)g.V, grow = fmaxf(degree - 1.0f, 0.0f);
    const bool wide = w.bu_k && 2.0f * (float)nscope * grow > SPREAD_ARCS * (float)ex.nwarps();   // spreads() can hold
    uint32_t rest = nscope;   // live vertices still unvisited in some direction, as of the last bottom-up step
    bool ok = run_pass(ex, PH_BFS0, [&](unsigned, unsigned nxt) {
        const unsigned par = ex.gl & 1u;
        if (ex.leader()) {
            nib_or(w.nb, p, NF | NB);
            atomicAdd(&ex.ctl->n_pivot, 1ull);
        }
        // the pivot is usually the largest hub: 64-entry pieces of its out-
        // and in-list, one per warp, so they spread over the whole grid in
        // one round of gathers
        const uint32_t fb = __ldg(&g.Fr[p]), fe = __ldg(&g.Fr[p + 1]);
        const uint32_t bb = __ldg(&g.Br[p]), be = __ldg(&g.Br[p + 1]);
        const uint32_t nfc = (fe - fb + 63u) / 64u, nbc = (be - bb + 63u) / 64u;
        for (uint32_t c = ex.wid(); c < nfc + nbc; c += ex.nwarps()) {
            const int dir = c < nfc ? 0 : 1;
            const uint32_t beg = dir ? bb + (c - nfc) * 64u : fb + c * 64u;
            const uint32_t end = min(beg + 64u, dir ? be : fe);
            const uint32_t *C = dir ? g.Bc : g.Fc;
            const uint32_t e0 = beg + lane_id(), e1 = e0 + 32u;
            // the pivot itself (a self-loop) is flagged by the leader alone
            const uint32_t n0 = e0 < end ? __ldg(&C[e0]) : p, n1 = e1 < end ? __ldg(&C[e1]) : p;
            bfs_visit2(ex, g, w, dir, n0 != p, n0, n1 != p, n1, par, nxt, true);
            count_edges(ex, end - beg);
        }
        bq_flush(2, w.qcap, w.Q[0][par], &ex.lc(nxt)[C_FQ], w.Q[1][par], &ex.lc(nxt)[C_BQ], g.V, ex.ctl,
                 &ex.lc(nxt)[C_FE], &ex.lc(nxt)[C_BE]);
    });
    if (!ok) return false;
    // The claims of a pass are tallied by degree (the frontier edges Beamer's
    // rule weighs) only while they could reach the bottom-up threshold: each
    // claim brings at most maxdeg edges, and a pass of one level claims at most
    // the edges of its frontier (and at most the scope).  A pass in which warps
    // go on with their own finds can claim more; it is weighed by its frontier
    // all the same, so a pass that should go bottom-up may come one pass later.
    // That is rare (such a pass is not expected to grow, see spreads) and
    // cheaper than the offset gathers: 2M random vertices of degree 8 behind a
    // path of 500, vSlota, 1,161 us, tallied in every such pass 1,210; 4096^2
    // grid 2,306 and 2,522.  Four times the frontier's edges, as a guess at what those
    // passes claim, is no better either: 400,000 random vertices of degree 3
    // 294 us, now 283; 4096^2 grid 2,438.
    // Bit d of known: the previous pass tallied direction d, so its count is
    // exact.  Whole-GPU policy only: the single-CTA and batched searches are short, and there the
    // extra registers cost more than the gathers they save.
    unsigned known = 3u;
    const uint32_t dmax32 = Ex::grid ? __ldcg(&ex.ctl->maxdeg) : 0u;
    for (unsigned lev = 1;; lev++) {
        const uint32_t nf = last_count(ex, C_FQ), nb = last_count(ex, C_BQ);
        const uint32_t nhf = last_count(ex, C_FH), nhb = last_count(ex, C_BH);
        if (nf + nb + nhf + nhb == 0u) return true;
        if (lev > max_levels(g.V)) { if (ex.leader()) set_error(ex.ctl, E_NOT_CONVERGED, 40); return false; }
        // Beamer's rule: bottom-up when the frontier has more edges to
        // expand than the scope has vertices to test (times bu_k)
        const uint32_t mf = last_count(ex, C_FE), mb = last_count(ex, C_BE);
        const bool puf = w.bu_k && (unsigned long long)mf > (unsigned long long)nscope * w.bu_k;
        const bool pub = w.bu_k && (unsigned long long)mb > (unsigned long long)nscope * w.bu_k;
        // may warps go on with their own finds?
        bool local = lw < 0;
        if (local && wide) {
            const float xf = (known & 1u ? (float)mf : (float)nf * degree) + (float)(nhf * CH);
            const float xb = (known & 2u ? (float)mb : (float)nb * degree) + (float)(nhb * CH);
            local = !spreads(ex, fminf(xf, (float)rest) * grow, fminf(xb, (float)rest) * grow, grow,
                             (float)nscope * (float)w.bu_k);
        }
        unsigned cm = 3u;   // bit d: this pass tallies direction d
        if constexpr (Ex::grid) {
            cm = 0u;
            const unsigned long long dmax = dmax32;
#pragma unroll
            for (int d = 0; d < 2; d++) {
                const bool pu = d ? pub : puf;
                const unsigned long long nfd = d ? nb : nf, mfd = d ? mb : mf, nhd = d ? nhb : nhf;
                unsigned long long xe = pu ? nscope : (((known >> d) & 1u) ? mfd : nfd * dmax) + nhd * CH;
                xe = min(xe, (unsigned long long)nscope);
                if (w.bu_k && xe * dmax > (unsigned long long)nscope * w.bu_k) cm |= 1u << d;
            }
            // a bottom-up step may shrink the scope the next pass weighs
            // against, so it tallies both directions (and its finds)
            if (puf || pub) cm = 3u;
            known = cm;
        }
        ok = run_pass(ex, (puf || pub) ? PH_BFS_PULL : PH_BFS, [&](unsigned, unsigned nxt) {
            const unsigned par = ex.gl & 1u, cp = par ^ 1u;
            if (puf || pub) {
                // a warp's units lie far apart: where ids follow degree, the
                // hubs' long lists spread over all warps (R-MAT scale 22, the
                // first step: 256 adjacent vertices a warp 122 us, spread
                // 86 us)
                const uint32_t nu = g.V / 32u + 1u, cu = unit_group(ex, g.V), ni = (nu + cu - 1u) / cu;
                for (uint32_t i = ex.wid(); i < ni; i += ex.nwarps()) {
                    const uint32_t u = lane_id() * ni + i;
                    bfs_pull(ex, g, w, puf, pub, u, load_unit(w, lane_id() < cu && u < nu, u), par, nxt);
                }
            }
            // frontier vertices a warp takes at once: 1 << gsh (a virtual-warp
            // item takes VWK = 4 groups of 32 >> lw)
            const bool full = nf + nb >= 16u * ex.nwarps();   // work for every warp
            const uint32_t gsh = lw >= 0 ? 7u - (uint32_t)lw : item_shift(ex, nf + nb);
            const uint32_t ngf = (nf + (1u << gsh) - 1u) >> gsh, ngb = (nb + (1u << gsh) - 1u) >> gsh;
            const uint32_t items_f = puf ? 0u : nhf + ngf;
            const uint32_t items_b = pub ? 0u : nhb + ngb;
            for (uint32_t it = ex.wid(); it < items_f + items_b; it += ex.nwarps()) {
                const int dir = it < items_f ? 0 : 1;
                const uint32_t k = dir ? it - items_f : it;
                const uint32_t nh = dir ? nhb : nhf;
                if (k < nh) {
                    auto fn2 = [&](bool v0, uint32_t n0, bool v1, uint32_t n1) {
                        bfs_visit2(ex, g, w, dir, v0, n0, v1, n1, par, nxt, (cm >> dir) & 1u);
                    };
                    chunk_expand(ex, dir ? g.Br : g.Fr, dir ? g.Bc : g.Fc, w.H[dir][cp][k], fn2);
                    continue;
                }
                const uint32_t n = dir ? nb : nf;
                if (lw < 0) {
                    const uint32_t i = ((k - nh) << gsh) + lane_id();
                    const bool valid = lane_id() >> gsh == 0u && i < n;
                    bfs_expand_lanes(ex, g, w, dir, valid, valid ? w.Q[dir][cp][i] : 0u, par, nxt, (cm >> dir) & 1u, !full);
                } else {
                    const bool lead = (lane_id() & ((1u << lw) - 1u)) == 0u;
                    uint32_t vk[VWK];
                    bool ak[VWK];
#pragma unroll
                    for (int j = 0; j < VWK; j++) {
                        const uint32_t ij = ((k - nh) << gsh) + (lane_id() >> lw) + (uint32_t)j * (32u >> lw);
                        ak[j] = ij < n;
                        vk[j] = ak[j] ? w.Q[dir][cp][ij] : 0u;
                        count_verts(ex, ak[j] && lead);
                    }
                    bfs_expand_vwk(ex, g, w, dir, vk, ak, lw, par, nxt, (cm >> dir) & 1u);
                }
            }
            if (local) {
                for (int dir = 0; dir < 2; dir++) {
                    if (dir ? pub : puf) continue;   // found bottom-up: left to the next pass
                    uint32_t edges = 0;
                    for (unsigned left = LOCAL_ROUNDS; left && edges < LOCAL_EDGES; left--) {
                        uint32_t v;
                        const unsigned took = bq_pop((unsigned)dir, w.qcap, full ? 24u : 1u, local_cap(w.qcap, full), v);
                        if (took == 0u) break;
                        edges += bfs_expand_lanes(ex, g, w, dir, lane_id() < took, v, par, nxt, (cm >> dir) & 1u, !full,
                                                  true);
                    }
                }
            }
            bq_flush(2, w.qcap, w.Q[0][par], &ex.lc(nxt)[C_FQ], w.Q[1][par], &ex.lc(nxt)[C_BQ], g.V, ex.ctl,
                     &ex.lc(nxt)[C_FE], &ex.lc(nxt)[C_BE], &ex.lc(nxt)[C_SCOPE]);
        });
        if (!ok) return false;
        // one shrink per search: weighing against a smaller scope again
        // would make bottom-up steps of what top-down steps do cheaper
        if (puf || pub) {
            rest = last_count(ex, C_SCOPE);
            if (!shrunk) nscope = rest;
            shrunk = true;
        }
    }
}

// ---------------------------------------------------------------------
// The end of the first FW-BW (scc_kernels.cu:124-142 for Hong,
// assignUniqueRange, :477-484, for Slota), off the nibble words in id order:
// vertices with both visited bits are the first pivot's SCC and stay as they
// are -- the label write maps them to Ctl::first_min, their smallest id,
// found here -- and every other live vertex is listed for what follows, its
// out-degree tallied.  Its class bits (forward, backward or neither) stay as
// its range: no SCC crosses them.
// ---------------------------------------------------------------------
template <class Ex>
__device__ bool ph_first_update(Ex &ex, const Graph &g, const Work &w, uint32_t *Lout)
{
    return run_pass(ex, PH_FIRST_UPDATE, [&](unsigned, unsigned nxt) {
        uint32_t mn = 0xFFFFFFFFu;
        const uint32_t nu = g.V / 32u + 1u, cu = item_group(ex, nu);
        for (uint32_t base = ex.wid() * cu; base < nu; base += ex.nwarps() * cu) {
            const uint32_t u = base + lane_id();
            const bool in = lane_id() < cu && u < nu;
            const NibUnit x = load_unit(w, in, u);
            const uint32_t both = x.live & x.fwd & x.bwd;
            if (both) mn = min(mn, u * 32u + (uint32_t)__ffs(both) - 1u);
            count_verts_n(ex, __popc(x.live & ~both));   // the listed ones: the rest cost half a byte each
            unit_walk2(u, x.live & ~both, [&](const bool (&ok)[2], const uint32_t (&v)[2], const unsigned (&)[2]) {
                bq_add_edges(0, (ok[0] ? __ldg(&g.Fr[v[0] + 1u]) - __ldg(&g.Fr[v[0]]) : 0u) +
                                    (ok[1] ? __ldg(&g.Fr[v[1] + 1u]) - __ldg(&g.Fr[v[1]]) : 0u));
                bq_pushK<2>(0, ok, v, w.qcap, Lout, &ex.lc(nxt)[C_LIST], g.V, ex.ctl, 16);
            });
        }
        block_min_atomic(mn, &ex.ctl->first_min);
        bq_flush(1, w.qcap, Lout, &ex.lc(nxt)[C_LIST], nullptr, nullptr, g.V, ex.ctl, &ex.lc(nxt)[C_FE]);
    });
}

// Hong: the vertices left after the trims, compacted, with their out-arcs
// tallied (the residual check).
template <class Ex>
__device__ bool ph_compact(Ex &ex, const Graph &g, const Work &w, VList src, uint32_t *Lout)
{
    return run_pass(ex, PH_COMPACT, [&](unsigned, unsigned nxt) {
        for (uint32_t base = ex.wid() * 128u; base < src.n; base += ex.nwarps() * 128u) {
            uint32_t v[4], s[4];
            bool ok[4];
            load_list4(src, base + 4u * lane_id(), v, ok);
#pragma unroll
            for (int j = 0; j < 4; j++) s[j] = ok[j] ? nib_of(w.nb, v[j]) : 0u;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const bool surv = (s[j] & NL) != 0u;
                bq_add_edges(0, surv ? __ldg(&g.Fr[v[j] + 1u]) - __ldg(&g.Fr[v[j]]) : 0u);
                bq_push(0, surv, v[j], w.qcap, Lout, &ex.lc(nxt)[C_LIST], g.V, ex.ctl, 18);
            }
            count_verts_n(ex, (unsigned)ok[0] + ok[1] + ok[2] + ok[3]);
        }
        bq_flush(1, w.qcap, Lout, &ex.lc(nxt)[C_LIST], nullptr, nullptr, g.V, ex.ctl, &ex.lc(nxt)[C_FE]);
    });
}

// ---------------------------------------------------------------------
// Colour peels: the SCCs of the vertices that the first FW-BW and the trims
// leave, for all four drivers (the colouring loop of scc_Coloring.cu:590-637
// and, with the same SCCs and counts, Hong's main loop scc_WCC.cu:851-930).
// A peel gives every live vertex the largest id that reaches it (its colour),
// finds the SCC of every colour's root -- the members of the colour that
// reach the root -- and leaves the colours behind as ranges: no SCC crosses
// two colours, so later peels walk no arc between them.  Peels alternate
// between the forward and the reverse CSR ("reaches" and "is reached by"),
// so both ends of a chain are cut.  The reference's loops drop the colours
// after each peel (scc_Coloring.cu:614-623) and keep the direction, or split
// each range by one pivot at a time (scc_WCC.cu:860-905): on a chain of
// 6,278 SCCs (65,000 vertices, 418,172 arcs) that is 570 colour sweeps, or
// 118 rounds with 1,450 BFS levels; kept colours need 8 peels, about 170
// sweeps and levels together, and a third of the colour loop's arcs.  What
// bounds them is the chain of dependent accesses of each level (list entry,
// offsets and colour, arcs, neighbour's pair, atomic).  That graph, before
// and now: one CTA vHong 26.5 -> 7.3 ms, vSlota 50.1 -> 6.4 ms; whole GPU
// 18.6 -> 1.22 ms and 11.7 -> 1.16 ms.
//
// A live vertex's word pair pc[v]: x the range, y = (colour << 1) | flag.
// One 8-byte gather per arc decides; a word of a vertex without colour is
// all ones.  While colours spread, the flag says that v is in a work list
// and not yet expanded (a raise finds it set and does not list v again;
// taking v off the list clears it and reads the newest colour); it is clear
// everywhere when they have settled, and then says that v reaches its root.
// ---------------------------------------------------------------------

// Word pairs of all vertices from their nibbles: the range is the class of
// the first search.
template <class Ex>
__device__ bool ph_peel_init(Ex &ex, const Graph &g, const Work &w)
{
    return run_pass(ex, PH_PEEL_INIT, [&](unsigned, unsigned) {
        for (uint32_t i0 = ex.tid() * 2u; i0 <= g.V; i0 += ex.nthr() * 2u) {
            const uint32_t x = w.nb[i0 >> 3] >> (4u * (i0 & 7u)), ca = x & NCLASS, cb = (x >> 4) & NCLASS;
            const bool la = (ca & NL) && ca != NCLASS, lb = (cb & NL) && cb != NCLASS;
            const uint4 o = make_uint4(la ? ca : FULL, la ? (i0 << 1) | 1u : FULL, lb ? cb : FULL,
                                       lb ? ((i0 + 1u) << 1) | 1u : FULL);
            if (i0 + 1u <= g.V) *reinterpret_cast<uint4 *>(w.pc + i0) = o;
            else w.pc[i0] = make_uint2(o.x, o.y);
        }
    });
}

// K arcs per lane, all gathers, then all atomics before any append: with
// RAISE the owner's colour c is offered to neighbour n in range r, else n
// joins the SCC of colour c's root.
template <bool RAISE, int K, class Ex>
__device__ __forceinline__ void peel_visit(Ex &ex, const Graph &g, const Work &w, const bool (&v)[K], uint32_t (&n)[K],
                                           const uint32_t (&r)[K], const uint32_t (&c)[K], unsigned par, unsigned nxt)
{
    uint2 a[K];
    bool push[K];
#pragma unroll
    for (int j = 0; j < K; j++) {
        if (v[j]) n[j] = guard_id(n[j], g.V, ex.ctl);
        a[j] = make_uint2(FULL, FULL);
        if (v[j] && RAISE) a[j] = w.pc[n[j]];
        if (v[j] && !RAISE) a[j].y = w.pc[n[j]].y;
    }
#pragma unroll
    for (int j = 0; j < K; j++) {
        const uint32_t wc = (c[j] << 1) | 1u;
        if (RAISE) {
            const bool t = a[j].x == r[j] && a[j].y >> 1 < c[j];   // a colourless word's range is all ones: no owner's
            a[j].y = t ? atomicMax(&w.pc[n[j]].y, wc) : FULL;
            push[j] = !(a[j].y & 1u) && a[j].y < wc;               // whoever sets the flag lists the vertex
        } else {
            const bool t = a[j].y == c[j] << 1;
            push[j] = t && !(atomicOr(&w.pc[n[j]].y, 1u) & 1u);
        }
    }
    bq_pushK<K>(0, push, n, w.qcap, w.Q[0][par], &ex.lc(nxt)[C_FQ], g.V, ex.ctl, 14);
}

// Vertices of a peel's work list, one per lane, expanded over (R, C); with
// seeds the list is the live list (JOIN: only the roots of their colours
// are expanded).  local: v comes off the warp's own slice.  A raised vertex
// can come off slices again and again within a pass, and the chunk queues
// have room for one cut of every heavy vertex; so a heavy one taken off a
// slice is not cut but goes to the next pass: its flag is set again, and
// whoever finds it clear lists the vertex.  (Left set until the degree is
// known, every vertex waits for its offsets before the newest colour is
// read: 1M-vertex chain of SCCs, vSlota, 2,713 us, now 2,659.)  JOIN takes
// every vertex once.
template <bool RAISE, class Ex>
__device__ __forceinline__ void peel_expand(Ex &ex, const Graph &g, const Work &w, const uint32_t *__restrict__ R,
                                            const uint32_t *__restrict__ C, bool valid, uint32_t v, bool seeds,
                                            unsigned par, unsigned nxt, bool local = false)
{
    uint32_t r = 0, c = 0, beg = 0, deg = 0;
    bool act = valid;
    if (valid) {
        beg = __ldg(&R[v]);
        deg = __ldg(&R[v + 1u]) - beg;
        if (RAISE) {
            r = w.pc[v].x;
            c = atomicAnd(&w.pc[v].y, ~1u) >> 1;   // off the list: the newest colour
        } else {
            const uint32_t y = w.pc[v].y;
            c = y >> 1;
            if (seeds) {   // the root of its colour?
                act = y == v << 1;
                if (act) {
                    w.pc[v].y = y | 1u;
                    w.smin[v] = v;   // v represents its SCC: the update folds the members in
                }
            }
        }
    }
    if (RAISE && local) {
        const bool later = deg > HEAVY_T;   // (deg is 0 without a vertex)
        const bool list = later && !(atomicOr(&w.pc[v].y, 1u) & 1u);
        warp_push(list, v, w.Q[0][par], &ex.lc(nxt)[C_FQ], g.V, ex.ctl, 15);
        if (later) valid = act = false;
    }
    if (!RAISE && seeds) {
        const unsigned m = __ballot_sync(FULL, act);
        if (lane_id() == 0 && m) atomicAdd(&ex.ctl->n_pivot, (unsigned long long)__popc(m));
        if (m == 0u) return;
    }
    if (!act) deg = 0u;
    const bool heavy = deg > HEAVY_T;
    warp_push_chunks(v, heavy ? (deg + CH - 1u) / CH : 0u, w.H[0][par], &ex.lc(nxt)[C_FH], w.hcap, ex.ctl);
    if (heavy) deg = 0u;
    count_verts(ex, valid);
    // 128 arcs a step: a level's time is its rounds of gather and atomic
    // (65,000-vertex chain on one CTA: 64 a step 6.8 ms, 128 6.6 ms)
    count_edges(ex, lbs_walk4(beg, deg, C, [&](const bool (&ok)[4], uint32_t (&n)[4], const unsigned (&own)[4]) {
        uint32_t rr[4], cc[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            cc[j] = __shfl_sync(FULL, c, own[j]);
            rr[j] = RAISE ? __shfl_sync(FULL, r, own[j]) : 0u;
        }
        peel_visit<RAISE, 4>(ex, g, w, ok, n, rr, cc, par, nxt);
    }));
}

// One fixpoint of a peel over (R, C): with RAISE the colours of the live
// list spread, else the roots' SCCs are searched.  Lists longer than HEAVY_T
// go through chunks, as in the first search.
template <bool RAISE, class Ex>
__device__ bool ph_peel_spread(Ex &ex, const Graph &g, const Work &w, VList L, const uint32_t *__restrict__ R,
                               const uint32_t *__restrict__ C)
{
    uint32_t nq = L.n, nh = 0;
    for (unsigned lev = 0;; lev++) {
        if (lev > max_levels(g.V)) { if (ex.leader()) set_error(ex.ctl, E_NOT_CONVERGED, RAISE ? 50 : 40); return false; }
        const bool ok = run_pass(ex, RAISE ? PH_PROP : PH_PEEL_SCC, [&](unsigned, unsigned nxt) {
            const unsigned par = ex.gl & 1u, cp = par ^ 1u;
            const uint32_t *src = lev == 0u ? L.p : w.Q[0][cp];
            const uint32_t gsh = item_shift(ex, nq), ng = (nq + (1u << gsh) - 1u) >> gsh;
            for (uint32_t it = ex.wid(); it < nh + ng; it += ex.nwarps()) {
                if (it < nh) {
                    const uint2 hc = w.H[0][cp][it];
                    const uint2 x = make_uint2(vld(&w.pc[hc.x].x), vld(&w.pc[hc.x].y));
                    const uint32_t c = x.y >> 1;
                    auto fn = [&](bool v0, uint32_t n0, bool v1, uint32_t n1) {
                        const bool ok[2] = {v0, v1};
                        uint32_t n[2] = {n0, n1};
                        const uint32_t rr[2] = {x.x, x.x}, cc[2] = {c, c};
                        peel_visit<RAISE, 2>(ex, g, w, ok, n, rr, cc, par, nxt);
                    };
                    chunk_expand(ex, R, C, hc, fn);
                    continue;
                }
                const uint32_t i = ((it - nh) << gsh) + lane_id();
                const bool valid = lane_id() >> gsh == 0u && i < nq;
                peel_expand<RAISE>(ex, g, w, R, C, valid, valid ? src[i] : 0u, lev == 0u, par, nxt);
            }
            // Rounds of the warp's own finds, where a barrier spans CTAs: on
            // one CTA it costs less than a round's lost balance.  65,000-vertex
            // chains on clusters of 1,024-thread CTAs: four CTAs 4.8 -> 4.5 and
            // 3.8 -> 3.0 ms, sixteen 2.8 -> 2.4 and 2.5 -> 1.8 ms.
            for (unsigned left = Ex::grid || Ex::cluster ? PEEL_ROUNDS : 0u; left; left--) {
                uint32_t v;
                const unsigned took = bq_pop(0, w.qcap, 1u, local_cap(w.qcap), v);
                if (took == 0u) break;
                peel_expand<RAISE>(ex, g, w, R, C, lane_id() < took, v, false, par, nxt, true);
            }
            bq_flush(1, w.qcap, w.Q[0][par], &ex.lc(nxt)[C_FQ], nullptr, nullptr, g.V, ex.ctl);
        });
        if (!ok) return false;
        nq = last_count(ex, C_FQ);
        nh = last_count(ex, C_FH);
        if (nq + nh == 0u) return true;
    }
}

// Peel end: vertices that reach their root are its SCC; the rest keep their
// colour as range, take their own id as colour and form the next live list.
template <class Ex>
__device__ bool ph_peel_update(Ex &ex, const Graph &g, const Work &w, VList src, uint32_t *Lout)
{
    return run_pass(ex, PH_PEEL_UPDATE, [&](unsigned, unsigned nxt) {
        for (uint32_t base = ex.wid() * 128u; base < src.n; base += ex.nwarps() * 128u) {
            uint32_t v[4], y[4];
            bool ok[4];
            load_list4(src, base + 4u * lane_id(), v, ok);
#pragma unroll
            for (int j = 0; j < 4; j++) y[j] = ok[j] ? w.pc[v[j]].y : 0u;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const bool scc = ok[j] && (y[j] & 1u), surv = ok[j] && !scc;
                const uint32_t c = y[j] >> 1;
                if (scc) {
                    w.pc[v[j]] = make_uint2(FULL, FULL);
                    w.label[v[j]] = c;
                }
                if (surv) w.pc[v[j]] = make_uint2(c, (v[j] << 1) | 1u);
                smin_fold(scc, c, v[j], w.smin);
                bq_add_edges(0, surv ? __ldg(&g.Fr[v[j] + 1u]) - __ldg(&g.Fr[v[j]]) : 0u);
                bq_push(0, surv, v[j], w.qcap, Lout, &ex.lc(nxt)[C_LIST], g.V, ex.ctl, 17);
            }
            count_verts_n(ex, (unsigned)ok[0] + ok[1] + ok[2] + ok[3]);
        }
        bq_flush(1, w.qcap, Lout, &ex.lc(nxt)[C_LIST], nullptr, nullptr, g.V, ex.ctl, &ex.lc(nxt)[C_FE]);
    });
}

// ---------------------------------------------------------------------
// drivers
// ---------------------------------------------------------------------
struct Carry {
    unsigned gl;
    unsigned lsel;
    uint32_t nL;
    uint32_t nE;    // out-arcs of the live vertices (tallied by the pass that listed them)
    uint32_t peels; // colour peels made so far
    bool paired;    // the word pairs are made
};

enum { RUN_DONE = 0, RUN_SWITCH = 1, RUN_RESIDUAL = 2, RUN_ERROR = -1 };

// ---------------------------------------------------------------------
// Small residuals: when the live vertices left for the main loop / the
// colouring peels are few (at most RES_MAX_V, with at most RES_MAX_E
// out-arcs), their SCCs are found on one CTA in shared memory instead of
// by further whole-GPU passes.  SCCs never contain a vertex whose SCC is
// already known, so the SCCs of the live vertices are those of the
// subgraph they induce; every SCC found here counts as a pivot SCC, as the
// reference counts each SCC its main loop / colouring finds once
// (scc_WCC.cu:933-949, scc_Coloring.cu:640-652), so the counters and the
// canonical labels are those of any complete run.
//   pass 1 (all CTAs): live vertex L[i] gets its local number i and the
//          residual flag in its nibble;
//   pass 2 (all CTAs): the arcs between live vertices, as (i << 16) | j,
//          into a work queue;
//   then one CTA loads them into shared memory and peels SCCs by colour
//   propagation (max of the local ids reachable on even peels, min on odd
//   ones, so a chain is cut from either end) and a forward search inside
//   each colour from its root, as scc_Coloring.cu:590-637 does, but with
//   __syncthreads barriers between sweeps and with the colours of a peel kept
//   as ranges of the next (3,000 vertices of a chain of SCCs: 7 to 11 peels
//   instead of 16 to 19, a third of the sweeps).
// ---------------------------------------------------------------------
constexpr uint32_t RES_MAX_V = 4096;
constexpr uint32_t RES_MAX_E = 16384;

__host__ __device__ __forceinline__ uint32_t res_al4(uint32_t x) { return (x + 3u) & ~3u; }
// shared memory of the solver: gid, off, aux (u32), col, rng (u16), flag (u8), adj (u16)
__host__ __device__ __forceinline__ uint32_t res_smem_bytes(uint32_t n, uint32_t m)
{
    return 4u * n + 4u * (n + 1u) + 4u * n + 2u * res_al4(2u * n) + res_al4(n) + res_al4(2u * m);
}

// Uniform decision (same in every thread of the launch or CTA): solve the
// live list on one CTA?  The solver uses the staging queues' shared memory.
template <class Ex>
__device__ __forceinline__ bool res_fits(const Graph &g, const Work &w, const Carry &cy)
{
    if (Ex::cluster || cy.nL == 0u || cy.nL > RES_MAX_V || cy.nE > RES_MAX_E || cy.nE > g.V + 1u) return false;
    const uint32_t avail = Ex::nbq * (blockDim.x >> 5) * w.qcap * 4u;
    return res_smem_bytes(cy.nL, cy.nE) <= avail;
}

// Block-wide exclusive prefix sum of a[0..len) in place (shared memory).
// Every thread of the CTA calls it.
__device__ __forceinline__ void block_excl_scan(uint32_t *a, uint32_t len)
{
    __shared__ uint32_t s_part[32];
    const uint32_t per = (len + blockDim.x - 1u) / blockDim.x;
    const uint32_t lo = threadIdx.x * per, hi = min(lo + per, len);
    uint32_t sum = 0;
    for (uint32_t i = lo; i < hi; i++) sum += a[i];
    const uint32_t incl = warp_incl_scan(sum);
    const unsigned wi = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane_id() == 31u) s_part[wi] = incl;
    __syncthreads();
    if (wi == 0) {
        const uint32_t x = lane_id() < nw ? s_part[lane_id()] : 0u;
        const uint32_t xs = warp_incl_scan(x);
        if (lane_id() < nw) s_part[lane_id()] = xs - x;   // exclusive offset of each warp
    }
    __syncthreads();
    uint32_t run = s_part[wi] + incl - sum;
    for (uint32_t i = lo; i < hi; i++) {
        const uint32_t x = a[i];
        a[i] = run;
        run += x;
    }
    __syncthreads();
}

// Passes 1 and 2 (every CTA of the policy).  On return the arcs are in
// Q[0][(cy.gl - 1) & 1] (the colour words lie over Q[1]) and their number in
// the pass counter C_BQ.
template <class Ex>
__device__ bool res_extract(Ex &ex, const Graph &g, const Work &w, Carry &cy)
{
    const uint32_t *L = w.L[cy.lsel];
    const uint32_t n = cy.nL;
    if (!run_pass(ex, PH_RES_TAG, [&](unsigned, unsigned) {
            for (uint32_t i = ex.tid(); i < n; i += ex.nthr()) {
                w.st[L[i]] = i;
                nib_or(w.nb, L[i], NQ);
            }
        }))
        return false;
    const bool ok = run_pass(ex, PH_RES_EXTRACT, [&](unsigned, unsigned nxt) {
        uint32_t *eb = w.Q[0][ex.gl & 1u];
        for (uint32_t base = ex.wid() * 32u; base < n; base += ex.nwarps() * 32u) {
            const uint32_t i = base + lane_id();
            const bool valid = i < n;
            const uint32_t v = valid ? L[i] : 0u;
            const uint32_t beg = valid ? __ldg(&g.Fr[v]) : 0u, deg = valid ? __ldg(&g.Fr[v + 1u]) - beg : 0u;
            const uint32_t r = !valid ? 0u : cy.peels ? w.pc[v].x : nib_of(w.nb, v) & NCLASS;
            auto fn = [&](bool ok2, uint32_t u, uint32_t own) {
                bool hit = false;
                uint32_t e = 0;
                const uint32_t src = __shfl_sync(FULL, i, own), rs = __shfl_sync(FULL, r, own);
                if (ok2) {
                    u = guard_id(u, g.V, ex.ctl);
                    const uint32_t x = nib_of(w.nb, u);
                    hit = (x & (NL | NQ)) == (NL | NQ) && (cy.peels ? w.pc[u].x : x & NCLASS) == rs;
                    if (hit) e = (src << 16) | w.st[u];
                }
                warp_push(hit, e, eb, &ex.lc(nxt)[C_BQ], RES_MAX_E, ex.ctl, 24);
            };
            count_edges(ex, lbs_walk(beg, deg, g.Fc, fn));
        }
    });
    cy.gl = ex.gl;
    return ok;
}

// The solver (every thread of one CTA).  L[0..n): the live vertices;
// eb[0..m): their arcs (i << 16) | j.  Writes every live vertex's
// canonical label (LBL_SELF: the smallest id of its SCC) and adds the SCCs
// found to n_pivot.  Each peel removes at least the root with
// the largest (or smallest) key, so at most n peels, each with at most n + 1
// sweeps per fixpoint.
// With out set the canonical labels of the residual vertices also go straight
// to out: the other CTAs are writing every other vertex's label meanwhile,
// leaving out those with the residual flag.
static __device__ __noinline__ void res_solve(const Graph &g, const Work &w, const uint32_t *L, uint32_t n, const uint32_t *eb,
                          uint32_t m, Ctl *ctl, uint32_t *out = nullptr)
{
    constexpr uint8_t ALIVE = 1, VIS = 2;
    constexpr uint16_t RNG_DONE = 0xFFFFu;   // above every local id: matches no live vertex's range
    char *sb = reinterpret_cast<char *>(&sccb_dsmem[BQ_HDR]);
    uint32_t *gid = reinterpret_cast<uint32_t *>(sb);
    uint32_t *off = gid + n;
    uint32_t *aux = off + n + 1u;                  // fill cursor, then smallest member id per root
    uint16_t *col = reinterpret_cast<uint16_t *>(aux + n);
    uint16_t *rng = reinterpret_cast<uint16_t *>(sb + 12u * n + 4u + res_al4(2u * n));   // colour of the last peel
    uint8_t *flag = reinterpret_cast<uint8_t *>(sb + 12u * n + 4u + 2u * res_al4(2u * n));
    uint16_t *adj = reinterpret_cast<uint16_t *>(sb + 12u * n + 4u + 2u * res_al4(2u * n) + res_al4(n));
    __shared__ uint32_t s_alive, s_npiv, s_peels;
    const uint32_t t = threadIdx.x, T = blockDim.x;
    for (uint32_t i = t; i < n; i += T) {
        gid[i] = L[i];
        off[i] = 0u;
        rng[i] = 0u;
        flag[i] = ALIVE;
    }
    if (t == 0) { off[n] = 0u; s_alive = n; s_npiv = 0u; s_peels = 0u; }
    __syncthreads();
    for (uint32_t k = t; k < m; k += T) atomicAdd(&off[eb[k] >> 16], 1u);
    __syncthreads();
    block_excl_scan(off, n + 1u);
    for (uint32_t i = t; i < n; i += T) aux[i] = off[i];
    __syncthreads();
    for (uint32_t k = t; k < m; k += T) {
        const uint32_t e = eb[k];
        adj[atomicAdd(&aux[e >> 16], 1u)] = (uint16_t)(e & 0xFFFFu);
    }
    __syncthreads();
    for (uint32_t i = t; i < n; i += T) aux[i] = 0xFFFFFFFFu;
    __syncthreads();
    bool failed = false;
    for (uint32_t peel = 0;; peel++) {
        if (s_alive == 0u) break;
        if (peel > n + 1u) { failed = true; break; }
        const bool up = (peel & 1u) == 0u;
        for (uint32_t i = t; i < n; i += T)
            if (flag[i] & ALIVE) col[i] = (uint16_t)(up ? i : n - 1u - i);
        __syncthreads();
        // colour = largest key reachable (scc_kernels.cu:539-564)
        for (uint32_t sweep = 0;; sweep++) {
            int ch = 0;
            for (uint32_t i = t; i < n; i += T) {
                if (!(flag[i] & ALIVE)) continue;
                uint16_t c = col[i];
                const uint16_t r = rng[i];
                for (uint32_t e = off[i]; e < off[i + 1u]; e++) {
                    const uint16_t j = adj[e];
                    if (rng[j] == r && col[j] > c) c = col[j];
                }
                if (c > col[i]) { col[i] = c; ch = 1; }
            }
            if (!__syncthreads_or(ch)) break;
            if (sweep > n + 1u) { failed = true; break; }
        }
        if (failed) break;
        // roots keep their own key; the forward search inside each colour
        // (scc_kernels.cu:567-610) marks their SCCs
        for (uint32_t i = t; i < n; i += T)
            if ((flag[i] & ALIVE) && col[i] == (up ? i : n - 1u - i)) flag[i] |= VIS;
        __syncthreads();
        for (uint32_t sweep = 0;; sweep++) {
            int ch = 0;
            for (uint32_t i = t; i < n; i += T) {
                if ((flag[i] & (ALIVE | VIS)) != (ALIVE | VIS)) continue;
                for (uint32_t e = off[i]; e < off[i + 1u]; e++) {
                    const uint16_t j = adj[e];
                    if ((flag[j] & (ALIVE | VIS)) == ALIVE && col[j] == col[i]) { flag[j] |= VIS; ch = 1; }
                }
            }
            if (!__syncthreads_or(ch)) break;
            if (sweep > n + 1u) { failed = true; break; }
        }
        if (failed) break;
        uint32_t done = 0, roots = 0;
        for (uint32_t i = t; i < n; i += T) {
            if ((flag[i] & (ALIVE | VIS)) != (ALIVE | VIS)) {
                rng[i] = (flag[i] & ALIVE) ? col[i] : RNG_DONE;
                continue;
            }
            const uint32_t r = up ? col[i] : n - 1u - col[i];
            rng[i] = RNG_DONE;
            atomicMin(&aux[r], gid[i]);
            col[i] = (uint16_t)r;   // the root, from here on
            flag[i] = 0;
            done++;
            roots += (r == i) ? 1u : 0u;
        }
        done = __reduce_add_sync(FULL, done);
        roots = __reduce_add_sync(FULL, roots);
        if (lane_id() == 0 && done) { atomicSub(&s_alive, done); atomicAdd(&s_npiv, roots); }
        if (t == 0) s_peels = peel + 1u;
        __syncthreads();
    }
    if (failed) {
        if (t == 0) set_error(ctl, E_NOT_CONVERGED, 71);
        return;
    }
    for (uint32_t i = t; i < n; i += T) {
        w.label[gid[i]] = LBL_SELF | aux[col[i]];
        if (out) out[gid[i] - 1u] = aux[col[i]];
    }
    if (t == 0) {
        atomicAdd(&ctl->n_pivot, (unsigned long long)s_npiv);
        atomicAdd(&ctl->outer, s_peels);
    }
    __syncthreads();
}

// Records the solver as one more pass in the pass trace (one CTA).
__device__ __forceinline__ void res_trace(Ctl *ctl, unsigned gl, uint32_t n)
{
    if (threadIdx.x == 0 && ctl->trace && gl < ctl->trace_cap) {
        ctl->trace[2 * gl] = gtimer();
        ctl->trace[2 * gl + 1] = (unsigned long long)PH_RES_SOLVE | ((unsigned long long)n << 8);
    }
}

// Residual path at a main-loop / peel head.  On the whole-GPU policy it
// returns RUN_RESIDUAL after the two passes (CTA 0 then solves and the
// others leave); on one CTA it also solves and returns RUN_DONE.
template <class Ex>
__device__ int residual(Ex &ex, const Graph &g, const Work &w, Carry &cy)
{
    if (!res_extract(ex, g, w, cy)) return RUN_ERROR;
    if (Ex::grid) return RUN_RESIDUAL;
    res_solve(g, w, w.L[cy.lsel], cy.nL, w.Q[0][(cy.gl - 1u) & 1u], last_count(ex, C_BQ), ex.ctl);
    res_trace(ex.ctl, ex.gl, cy.nL);
    ex.gl++;
    cy.gl = ex.gl;
    cy.nL = 0u;
    return ex.sync() ? RUN_DONE : RUN_ERROR;
}

// Colour peels until no vertex is left.  Entry: live list L[lsel] with nL
// entries, nE out-arcs, their ranges in the nibbles.
template <class Ex>
__device__ int peel_loop(Ex &ex, const Graph &g, const Work &w, Carry &cy, uint32_t tail_n)
{
    while (cy.nL > 0u) {
        if (res_fits<Ex>(g, w, cy)) return residual(ex, g, w, cy);
        // before one CTA takes over: the word pairs of all V vertices are a
        // whole-GPU pass (4.2M vertices: 8 us, on one CTA 672 us)
        if (!cy.paired && !ph_peel_init(ex, g, w)) return RUN_ERROR;
        cy.paired = true;
        if (Ex::grid && cy.nL <= tail_n) { cy.gl = ex.gl; return RUN_SWITCH; }
        if (ex.leader()) ex.ctl->outer++;
        const VList L{w.L[cy.lsel], cy.nL};
        const bool odd = (cy.peels & 1u) != 0u;
        const uint32_t *R0 = odd ? g.Br : g.Fr, *C0 = odd ? g.Bc : g.Fc;
        const uint32_t *R1 = odd ? g.Fr : g.Br, *C1 = odd ? g.Fc : g.Bc;
        if (!ph_peel_spread<true>(ex, g, w, L, R0, C0)) return RUN_ERROR;
        if (!ph_peel_spread<false>(ex, g, w, L, R1, C1)) return RUN_ERROR;
        if (!ph_peel_update(ex, g, w, L, w.L[cy.lsel ^ 1u])) return RUN_ERROR;
        cy.nL = last_count(ex, C_LIST);
        cy.nE = last_count(ex, C_FE);
        cy.lsel ^= 1u;
        cy.peels++;
        cy.gl = ex.gl;
    }
    return RUN_DONE;
}

// The pivot over the live vertices after trim1 to its fixpoint
// (pollForFirstPivot / selectFirstPivot, scc_WCC.cu:701-703), into pivkey[1]:
// run only when the pivot that the init pass found was trimmed since (else
// it is still the largest).
template <class Ex>
__device__ bool ph_first_pivot(Ex &ex, const Graph &g, const Work &w)
{
    return run_pass(ex, PH_FIRST_PIVOT, [&](unsigned, unsigned) {
        unsigned long long best = 0;
        const uint32_t nwords = g.V / 8u + 1u;
        for (uint32_t wd = ex.tid(); wd < nwords; wd += ex.nthr()) {
            for (uint32_t m = w.nb[wd] & NIBS; m; m &= m - 1u) {
                const unsigned long long k = pivot_key(g, wd * 8u + ((uint32_t)__ffs(m) - 1u) / 4u);
                best = k > best ? k : best;
            }
        }
        block_max_atomic(best, &w.pivkey[1]);
    });
}

__device__ __forceinline__ unsigned long long vld64(const unsigned long long *p)
{
    return *(const volatile unsigned long long *)p;
}

// vHong / wHong up to the peels (scc_WCC.cu:573-848): trim1*, first pivot,
// FW-BW, update, trim1*, trim2, trim1*, live list of what is left.  wHong /
// wSlota run the FW-BW with the virtual-warp schedule (scc_WCC.cu:209-317,
// scc_Coloring.cu:154-263).
template <class Ex>
__device__ int hong_front(Ex &ex, const Graph &g, const Work &w, bool t1, bool t2, int lw, Carry &cy)
{
    if (!ph_init(ex, g, w, t1, t1)) return RUN_ERROR;
    uint32_t nlive = last_count(ex, C_LIST);
    unsigned long long k = vld64(&w.pivkey[0]);
    if (t1 && nlive) {
        if (!ph_trim1_fix(ex, g, w, VList{nullptr, nlive}, true)) return RUN_ERROR;
        nlive = g.V - (uint32_t)vld64(&ex.ctl->n_trim1);
        if (nlive && !(nib_of(w.nb, key_vertex(k)) & NL)) {
            if (!ph_first_pivot(ex, g, w)) return RUN_ERROR;
            k = vld64(&w.pivkey[1]);
        }
    }
    cy.gl = ex.gl;
    if (nlive == 0u) return RUN_DONE;
    if (!ph_bfs(ex, g, w, key_vertex(k), lw, nlive)) return RUN_ERROR;
    if (!ph_first_update(ex, g, w, w.L[1])) return RUN_ERROR;
    const VList L1{w.L[1], last_count(ex, C_LIST)};
    cy.gl = ex.gl;
    if (L1.n == 0u) return RUN_DONE;   // every vertex is trimmed or in the first SCC
    cy.lsel = 1u;
    cy.nL = L1.n;
    cy.nE = last_count(ex, C_FE);
    if (t1 && !ph_trim1_fix(ex, g, w, L1, false)) return RUN_ERROR;
    if (t2 && !ph_trim2(ex, g, w, L1)) return RUN_ERROR;
    if (t1 && t2 && !ph_trim1_fix(ex, g, w, L1, false)) return RUN_ERROR;
    if (t1 || t2) {
        if (!ph_compact(ex, g, w, L1, w.L[0])) return RUN_ERROR;
        cy.lsel = 0u;
        cy.nL = last_count(ex, C_LIST);
        cy.nE = last_count(ex, C_FE);
    }
    cy.gl = ex.gl;
    return RUN_DONE;
}

// vSlota / wSlota up to the peels (scc_Coloring.cu:403-587): trim1 once,
// first pivot, FW-BW, update.  t2 is not used by the reference's Slota
// drivers.
template <class Ex>
__device__ int slota_front(Ex &ex, const Graph &g, const Work &w, bool t1, int lw, Carry &cy)
{
    if (!ph_init(ex, g, w, t1, false)) return RUN_ERROR;
    const uint32_t nlive = last_count(ex, C_LIST);
    cy.gl = ex.gl;
    if (nlive == 0u) return RUN_DONE;
    if (!ph_bfs(ex, g, w, key_vertex(vld64(&w.pivkey[0])), lw, nlive)) return RUN_ERROR;
    if (!ph_first_update(ex, g, w, w.L[1])) return RUN_ERROR;
    cy.lsel = 1u;
    cy.nL = last_count(ex, C_LIST);
    cy.nE = last_count(ex, C_FE);
    cy.gl = ex.gl;
    return RUN_DONE;
}

}  // namespace sccb
