// Device-side building blocks of the B200 SCC engine.
//
// Vertex state is half a byte per vertex, eight vertices to a word (nb):
//   bit 0  NL  live: its SCC is not known (the reference's rangeSet tag,
//              include/scc.h:36-37, inverted)
//   bit 1  NF  forward-visited  (FV, include/scc.h:24)
//   bit 2  NB  backward-visited (BV, include/scc.h:26)
//   bit 3  NQ  trimmed after the init pass (its label is written), or, on a
//              live vertex, in the residual
// Neither NL nor NQ: a vertex that the init pass trimmed.  The first search runs in one
// range, so one gather per adjacency entry tells whether the neighbour is
// live and unvisited; afterwards the three low bits are the vertex's range.
// The reference keeps uint8 tags plus a uint32 range and reads both per edge
// (scc_kernels.cu:374-377).
//
// Every phase is written once against an execution policy:
//   GridExec   all CTAs of a cooperative (co-resident) launch; passes end in
//              a grid barrier whose wait is bounded by %globaltimer;
//   BlockExec  one CTA; passes end in __syncthreads.
// The plain path runs GridExec and drops to BlockExec on CTA 0 when the live
// set gets small; the batched form runs one BlockExec per graph.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace sccb {

constexpr uint32_t NL = 1u, NF = 2u, NB = 4u, NQ = 8u;
constexpr uint32_t NCLASS = NL | NF | NB;
constexpr uint32_t NIBS = 0x11111111u;    // bit 0 of every nibble of a word
constexpr uint32_t FULL = 0xFFFFFFFFu;
constexpr uint32_t MAX_V = 0x0FFFFFFEu;   // ids fit a colour word beside its flag
// label[v] with this bit set holds v's canonical label itself (the low
// bits): a vertex that is its own SCC (trim-1, trim-2, small residual SCCs)
// needs no smin entry and no gather when the labels are written out.
constexpr uint32_t LBL_SELF = 0x80000000u;

// Load-balancing constants of the frontier expansion: a frontier vertex
// whose degree exceeds HEAVY_T is cut into CH-edge chunks that the next pass
// spreads over all warps.
constexpr uint32_t HEAVY_T = 256;
constexpr uint32_t CH = 512;

// error codes shared with the host (include/scc_b200.h)
constexpr int E_OVERFLOW = 20;
constexpr int E_NOT_CONVERGED = 21;
constexpr int E_TIMEOUT = 22;
constexpr int E_BAD_GRAPH = 23;

enum { C_FQ = 0, C_BQ = 1, C_FH = 2, C_BH = 3, C_LIST = 4, C_FE = 5, C_BE = 6, C_SCOPE = 7, NCNT = 8 };

struct __align__(128) Ctl {
    // grid barrier arrival counter and the sticky error code share one
    // 8-byte word so that a waiter polls both with one load
    unsigned bar_count;
    int error;
    int where; unsigned _p0[29];
    unsigned lc[3][NCNT];                          // per-pass counters, 3-slot ring
    unsigned maxdeg;                               // largest out- or in-degree (init sweep)
    unsigned _p3[7];
    unsigned long long n_trim1, n_trim2, n_pivot;
    unsigned long long t_edges, t_verts;           // instrumented work counters
    unsigned passes, outer;                        // passes run, peels / iterations
    unsigned long long timeout_ns;
    unsigned tail_pass;                            // pass at which CTA 0 took over (0 = never)
    unsigned nlive_tail;
    unsigned long long t_start;                    // %globaltimer at kernel entry
    unsigned long long *trace;                     // optional: 2 words per pass
    unsigned trace_cap;
    unsigned labels_done;                          // the SCC kernel wrote the canonical labels itself
    unsigned first_min;                            // smallest member of the first pivot's SCC; ~0 before
};

// A control block reset on the device (k_canon_write), as the host would
// initialise it: zero, then the fields below; pivkey: one pivot word to
// clear as well, or nullptr.
struct CtlReset {
    Ctl *next;
    unsigned long long timeout_ns;
    unsigned long long *trace;
    unsigned trace_cap;
    unsigned long long *pivkey;
};

// Phase ids recorded in the pass trace.
enum {
    PH_INIT = 1, PH_TRIM1_FIX = 4, PH_TRIM2 = 5, PH_TRIM2_APPLY = 6,
    PH_FIRST_PIVOT = 7, PH_BFS0 = 8, PH_BFS = 9, PH_PROP = 10, PH_FIRST_UPDATE = 11,
    PH_PEEL_UPDATE = 13, PH_COMPACT = 14, PH_PEEL_SCC = 15, PH_BFS_PULL = 16, PH_PEEL_INIT = 17,
    PH_RES_TAG = 18, PH_RES_EXTRACT = 19, PH_RES_SOLVE = 20
};

struct Graph {
    uint32_t V, E;
    const uint32_t *__restrict__ Fr, *__restrict__ Fc, *__restrict__ Br, *__restrict__ Bc;
    uint32_t vec;   // Fr and Br are 16-byte aligned: 128-bit offset loads allowed
};

// o[0..4] = R[i0 .. i0+4] with indices clipped to V+1 (the last offset);
// one 128-bit load plus one 32-bit load when R is 16-byte aligned (i0 is a
// multiple of 4).
__device__ __forceinline__ void load_off5(const uint32_t *__restrict__ R, uint32_t i0, uint32_t V, uint32_t vec,
                                          uint32_t (&o)[5])
{
    if (vec && i0 + 4u <= V + 1u) {
        const uint4 x = __ldg(reinterpret_cast<const uint4 *>(R + i0));
        o[0] = x.x; o[1] = x.y; o[2] = x.z; o[3] = x.w;
        o[4] = __ldg(&R[i0 + 4u]);
    } else {
#pragma unroll
        for (int j = 0; j < 5; j++) o[j] = __ldg(&R[min(i0 + (uint32_t)j, V + 1u)]);
    }
}

struct Work {
    uint32_t *nb;               // vertex states: nibble v & 7 of word v >> 3
    uint32_t *st;               // trim-1 stamps, then the local numbers of the residual's vertices
    uint32_t *label;            // of vertices whose SCC is found after the first search, or trimmed after init
    uint32_t *smin;             // smin[r] = smallest member id of the SCC represented by r; set to r
                                // when r becomes a representative (its seed pass), then folded
    uint32_t *L[2];
    uint32_t *Q[2][2];          // [direction][parity]
    uint2 *H[2][2];             // heavy chunks (vertex, chunk) [direction][parity]
    uint32_t hcap;
    uint2 *pc;                  // colour peels: (range, colour word) per vertex, over Q[1][0] and Q[1][1]
    unsigned long long *pivkey; // the first pivot's key: over init's live vertices, over the trimmed graph's
    Ctl *ctl;
    uint32_t qcap;              // entries per CTA staging queue (dynamic shared memory)
    uint32_t bu_k;              // bottom-up BFS step when frontier edges > bu_k * scope vertices (0 = never)
    uint32_t pull_lane;         // bottom-up step: lists up to this many entries are tested by their lane alone;
                                // of a longer list the lane tests the first min(8, pull_lane), the warp the rest
};

constexpr uint32_t PULL_LANE = 32;   // Work::pull_lane of the batched and no-allocation paths

// Bytes of the nibble array (words 0 .. V / 8).
__host__ __device__ constexpr size_t nib_bytes(size_t V) { return ((V / 8 + 1) * 4 + 255) / 256 * 256; }

// Carve the work arrays for a graph of V vertices and E edges out of `base`
// (nullptr: only count).  Returns the bytes used.  Same layout on host and
// device; used by the batched form, where every CTA re-carves its private
// scratch for each graph it takes.
// A chunk queue holds one cut of every vertex above HEAVY_T (at most deg / CH + 1
// chunks each): no pass may cut a vertex twice.
__host__ __device__ inline size_t carve_work(char *base, uint32_t V, uint32_t E, Work *w)
{
    const size_t n1 = (size_t)V + 1;
    const size_t hcap = (size_t)E / CH + (size_t)E / HEAVY_T + 64;
    const size_t va = (n1 * 4 + 255) / 256 * 256;       // one vertex array
    const size_t na = nib_bytes(V);
    const size_t ha = (hcap * 8 + 255) / 256 * 256;     // one chunk queue
    const size_t pa = 256;                              // the pivot words
    const size_t ca = (sizeof(Ctl) + 255) / 256 * 256;
    if (w && base) {
        w->st = (uint32_t *)(base);
        w->label = (uint32_t *)(base + va);
        w->smin = (uint32_t *)(base + 2 * va);
        w->L[0] = (uint32_t *)(base + 3 * va);
        w->L[1] = (uint32_t *)(base + 4 * va);
        w->Q[0][0] = (uint32_t *)(base + 5 * va);
        w->Q[0][1] = (uint32_t *)(base + 6 * va);
        w->Q[1][0] = (uint32_t *)(base + 7 * va);
        w->Q[1][1] = (uint32_t *)(base + 8 * va);
        w->pc = (uint2 *)w->Q[1][0];
        char *h = base + 9 * va;
        w->nb = (uint32_t *)h;
        h += na;
        w->H[0][0] = (uint2 *)(h);
        w->H[0][1] = (uint2 *)(h + ha);
        w->H[1][0] = (uint2 *)(h + 2 * ha);
        w->H[1][1] = (uint2 *)(h + 3 * ha);
        w->hcap = (uint32_t)hcap;
        w->pivkey = (unsigned long long *)(h + 4 * ha);
        w->ctl = (Ctl *)(h + 4 * ha + pa);
    }
    return 9 * va + na + 4 * ha + pa + ca;
}

// Dynamic shared memory of the SCC kernels: BQ_HDR control words, then the
// two staging queues, each split into one slice of qcap entries per warp of
// the CTA; the whole-GPU kernel has room for a third, for the residual
// solver, which takes all of it.
constexpr unsigned NBQ = 2;
constexpr unsigned BQ_WARPS = 32;                       // at most 1024 threads per CTA
constexpr unsigned BQ_CNT = 16;                         // per-warp fill counts [NBQ][BQ_WARPS]
constexpr unsigned BQ_PRE = BQ_CNT + NBQ * BQ_WARPS;    // per-warp flush offsets [NBQ][BQ_WARPS]
constexpr unsigned BQ_HDR = BQ_PRE + NBQ * BQ_WARPS;
extern __shared__ uint32_t sccb_dsmem[];

__device__ __forceinline__ uint32_t nib_of(const uint32_t *nb, uint32_t v) { return (nb[v >> 3] >> (4u * (v & 7u))) & 15u; }
// Sets bits of v's nibble; the nibble before.
__device__ __forceinline__ uint32_t nib_or(uint32_t *nb, uint32_t v, uint32_t bits)
{
    const uint32_t sh = 4u * (v & 7u);
    return (atomicOr(&nb[v >> 3], bits << sh) >> sh) & 15u;
}
// Reads *p into L1 without waiting for it.
__device__ __forceinline__ void prime_l1(const uint32_t *p)
{
    uint32_t x;
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(x) : "l"(p));
}
// Canonical label of v, or the vertex whose smin entry holds it: by its
// nibble v is its own SCC (trimmed by init), a member of the first pivot's
// SCC, or has its label written.
__device__ __forceinline__ uint32_t nib_label(uint32_t s, uint32_t v, uint32_t first_min, const uint32_t *label)
{
    return (s & (NL | NQ)) == 0u ? LBL_SELF | v : (s & NCLASS) == NCLASS ? LBL_SELF | first_min : label[v];
}
// v's SCC is known and its label written.
__device__ __forceinline__ void nib_kill(uint32_t *nb, uint32_t v)
{
    atomicOr(&nb[v >> 3], NQ << (4u * (v & 7u)));
    atomicAnd(&nb[v >> 3], ~(NL << (4u * (v & 7u))));
}

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }
__device__ __forceinline__ unsigned long long gtimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned vld(const unsigned *p) { return *(const volatile unsigned *)p; }
// The CTA's own copy of "an error was set", read by the single-CTA
// barrier instead of the control block's word (one load from L2 less per
// pass); every set_error raises it.
__device__ __forceinline__ int *cta_err()
{
    __shared__ int s_cta_err;
    return &s_cta_err;
}

__device__ __forceinline__ void set_error(Ctl *c, int code, int where)
{
    *(volatile int *)cta_err() = 1;
    if (atomicCAS(&c->error, 0, code) == 0) c->where = where;
}

// Adjacency ids must lie in [1, V].  An id outside that range is reported
// as a malformed graph and treated as vertex 0, which is permanently dead,
// so no state array is ever indexed out of bounds.
__device__ __forceinline__ uint32_t guard_id(uint32_t x, uint32_t V, Ctl *c)
{
    if (x - 1u >= V) {
        set_error(c, E_BAD_GRAPH, 60);
        return 0u;
    }
    return x;
}

// ---------------------------------------------------------------------
// execution policies
// ---------------------------------------------------------------------
// Per-CTA copy of the counters the last pass pushed (written by thread 0
// right after the pass barrier, read by every thread through last_count):
// one load per CTA instead of one per warp on the same few words, which made
// a same-address hot spot in L2 on every pass.
__device__ __forceinline__ unsigned *cnt_snap()
{
    __shared__ unsigned s_cnt[NCNT];
    return s_cnt;
}
// Pass counter ring of the single-CTA policy (BlockExec): in shared memory,
// since no other CTA reads it.
__device__ __forceinline__ unsigned (*block_lc())[NCNT]
{
    __shared__ unsigned s_lc[3][NCNT];
    return s_lc;
}

__device__ __forceinline__ void take_snap(const unsigned *c)
{
    unsigned *d = cnt_snap();
#pragma unroll
    for (int i = 0; i < NCNT; i++) d[i] = *(volatile const unsigned *)&c[i];
}

template <bool INSTR>
struct GridExec {
    static constexpr bool instr = INSTR;
    static constexpr bool grid = true;
    static constexpr bool cluster = false;
    static constexpr unsigned nbq = 3;   // staging queues the launch's shared memory has room for
    Ctl *ctl;
    unsigned gl;        // pass counter, identical in every thread
    unsigned cap = 0;   // pass cap of the run (0: none), see run_pass
    unsigned hold = 0;  // failure-detection test hook, see sync
    __device__ __forceinline__ unsigned tid() const { return blockIdx.x * blockDim.x + threadIdx.x; }
    __device__ __forceinline__ unsigned nthr() const { return gridDim.x * blockDim.x; }
    __device__ __forceinline__ unsigned wid() const { return tid() >> 5; }
    __device__ __forceinline__ unsigned nwarps() const { return nthr() >> 5; }
    __device__ __forceinline__ bool leader() const { return blockIdx.x == 0 && threadIdx.x == 0; }
    __device__ __forceinline__ unsigned *lc(unsigned slot) const { return ctl->lc[slot]; }

    // Grid barrier.  One arrival counter: CTA 0 adds 0x80000000 - (n - 1),
    // every other CTA adds 1, so bit 31 flips exactly when all n CTAs have
    // arrived.  Arrival is a release, the flip is read with acquire.  A
    // waiter leaves early when the sticky error word (polled with the
    // counter in one 8-byte load) is set, or after ctl->timeout_ns; any CTA
    // that sees an error returns, and the error stays set for the others.
    //
    // hold = k + 1 makes the last CTA withhold its arrival at pass k: the
    // failure-detection tests use it to make every wait of that barrier run
    // out (an arrival that never comes), which must end the run with
    // E_TIMEOUT and leave the context usable.
    __device__ bool sync(const unsigned *snap = nullptr)
    {
        __shared__ int s_err;
        __syncthreads();
        if (threadIdx.x == 0) {
            const unsigned nb = (blockIdx.x == 0) ? (0x80000000u - (gridDim.x - 1u)) : 1u;
            unsigned old;
            if (hold != 0u && gl + 1u == hold && blockIdx.x == gridDim.x - 1u)
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(old) : "l"(&ctl->bar_count) : "memory");
            else
                asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(&ctl->bar_count), "r"(nb) : "memory");
            int err = 0;
            unsigned long long t0 = 0;
            for (unsigned spin = 0;; spin++) {
                unsigned long long wv;
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(wv) : "l"(&ctl->bar_count) : "memory");
                err = (int)(wv >> 32);
                if ((((unsigned)wv ^ old) & 0x80000000u) != 0u || err) break;
                if ((spin & 255u) == 0u) {
                    unsigned long long t = gtimer();
                    if (spin == 0) t0 = t;
                    else if (t - t0 > ctl->timeout_ns) {
                        set_error(ctl, E_TIMEOUT, 1000);
                        err = E_TIMEOUT;
                        break;
                    }
                }
            }
            s_err = err;
            if (snap) take_snap(snap);
        }
        __syncthreads();
        return s_err == 0;
    }
};

template <bool INSTR>
struct BlockExec {
    static constexpr bool instr = INSTR;
    static constexpr bool grid = false;
    static constexpr bool cluster = false;
    static constexpr unsigned nbq = 2;
    Ctl *ctl;
    unsigned gl;
    unsigned cap = 0;
    __device__ __forceinline__ unsigned tid() const { return threadIdx.x; }
    __device__ __forceinline__ unsigned nthr() const { return blockDim.x; }
    __device__ __forceinline__ unsigned wid() const { return threadIdx.x >> 5; }
    __device__ __forceinline__ unsigned nwarps() const { return blockDim.x >> 5; }
    __device__ __forceinline__ bool leader() const { return threadIdx.x == 0; }
    __device__ __forceinline__ unsigned *lc(unsigned slot) const { return block_lc()[slot]; }
    // Counters and the error flag of a new run on this CTA (every thread calls).
    __device__ void reset_counters() const
    {
        for (unsigned i = threadIdx.x; i < 3u * NCNT; i += blockDim.x) (&block_lc()[0][0])[i] = 0u;
        if (threadIdx.x == 0) *cta_err() = *(volatile int *)&ctl->error != 0;
        __syncthreads();
    }
    __device__ bool sync(const unsigned *snap = nullptr)
    {
        __shared__ int s_err;
        __syncthreads();
        if (threadIdx.x == 0) {
            s_err = *(volatile int *)cta_err();
            if (snap) take_snap(snap);
        }
        __syncthreads();
        return s_err == 0;
    }
};

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// Hardware cluster barrier (every thread of every CTA of the cluster);
// writes before it, in any state space, are visible to the whole cluster
// after it.
__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// One graph on the CTAs of a thread-block cluster (co-scheduled by the
// hardware, so the barrier is the cluster barrier and needs no timeout).
// The error word is read between two barriers: no pass body runs while
// any CTA reads it, so every CTA takes the same branch.
//
// With `soft` set, the barrier is instead a counter in global memory (the
// grid barrier's bit-flip scheme over the cluster's CTAs) whose waits give
// up after soft_timeout_ns with E_TIMEOUT: a check mode in which a
// mismatch of barrier counts between the CTAs ends in an error status
// rather than a wait that never ends.
template <bool INSTR>
struct ClusterExec {
    static constexpr bool instr = INSTR;
    static constexpr bool grid = false;
    static constexpr bool cluster = true;
    static constexpr unsigned nbq = 2;
    Ctl *ctl;
    unsigned gl;
    unsigned rank, csize;
    unsigned *soft;   // the cluster's barrier counter, or nullptr for the hardware barrier
    unsigned long long soft_timeout_ns;
    unsigned cap = 0;
    unsigned hold = 0;  // check mode only: the last CTA withholds its arrival at pass hold - 1 (test hook)
    __device__ __forceinline__ unsigned tid() const { return rank * blockDim.x + threadIdx.x; }
    __device__ __forceinline__ unsigned nthr() const { return csize * blockDim.x; }
    __device__ __forceinline__ unsigned wid() const { return tid() >> 5; }
    __device__ __forceinline__ unsigned nwarps() const { return nthr() >> 5; }
    __device__ __forceinline__ bool leader() const { return rank == 0 && threadIdx.x == 0; }
    __device__ __forceinline__ unsigned *lc(unsigned slot) const { return ctl->lc[slot]; }
    __device__ void barrier()
    {
        if (!soft) {
            cluster_barrier();
            return;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const unsigned nb = rank == 0 ? (0x80000000u - (csize - 1u)) : 1u;
            unsigned old;
            if (hold != 0u && gl + 1u == hold && rank == csize - 1u)
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(old) : "l"(soft) : "memory");
            else
                asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(soft), "r"(nb) : "memory");
            unsigned long long t0 = 0;
            for (unsigned spin = 0;; spin++) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(soft) : "memory");
                if (((v ^ old) & 0x80000000u) != 0u) break;
                if ((spin & 255u) == 0u) {
                    const unsigned long long t = gtimer();
                    if (spin == 0) t0 = t;
                    else if (t - t0 > soft_timeout_ns) {
                        set_error(ctl, E_TIMEOUT, 1001);
                        break;
                    }
                }
            }
        }
        __syncthreads();
    }
    __device__ bool sync(const unsigned *snap = nullptr)
    {
        __shared__ int s_err;
        barrier();
        if (threadIdx.x == 0) {
            s_err = *(volatile int *)&ctl->error;
            if (snap) take_snap(snap);
        }
        barrier();
        return s_err == 0;
    }
};

// One pass: clear the counters the pass after next will push into, run the
// body with (cur, nxt) counter slots, then the barrier.  A pass pushes into
// counter slot gl%3 and buffer parity gl&1; the following pass reads them as
// its "current" slot (gl+2)%3 and parity (gl+1)&1.
//
// A run whose pass count reaches ex.cap (when set) stops with
// E_NOT_CONVERGED: the host's bound on the work of one run, on top of the
// V + 2 passes every convergence loop allows itself.
template <class Ex, class F>
__device__ __forceinline__ bool run_pass(Ex &ex, int phase, F &&body)
{
    if (ex.cap != 0u && ex.gl >= ex.cap) {
        if (ex.leader()) set_error(ex.ctl, E_NOT_CONVERGED, 70);
        ex.sync();
        ex.gl++;
        return false;
    }
    const unsigned nxt = ex.gl % 3u, clr = (ex.gl + 1u) % 3u, cur = (ex.gl + 2u) % 3u;
    if (ex.leader()) {
#pragma unroll
        for (int i = 0; i < NCNT; i++) ex.lc(clr)[i] = 0u;
    }
    body(cur, nxt);
    bool ok = ex.sync(ex.lc(nxt));
    if (ex.leader() && ex.ctl->trace && ex.gl < ex.ctl->trace_cap) {
        // pass trace: end time and (phase, items pushed) -- the reference's
        // _DEBUG per-phase event timers (scc_WCC.cu:650-672) at pass granularity
        // (instrumented runs record the running count of adjacency entries scanned instead)
        const unsigned *c = ex.lc(nxt);
        unsigned long long pushed = (unsigned long long)vld(&c[C_FQ]) + vld(&c[C_BQ]) + vld(&c[C_LIST]);
        if constexpr (Ex::instr) pushed = *(volatile unsigned long long *)&ex.ctl->t_edges;
        ex.ctl->trace[2 * ex.gl] = gtimer();
        ex.ctl->trace[2 * ex.gl + 1] = (unsigned long long)phase | (pushed << 8);
    }
    ex.gl++;
    return ok;
}

// Counter value pushed by the pass that just finished (the CTA's snapshot).
template <class Ex>
__device__ __forceinline__ unsigned last_count(const Ex &, int which)
{
    return cnt_snap()[which];
}

// ---------------------------------------------------------------------
// warp primitives
// ---------------------------------------------------------------------

// Warp-aggregated append (ballot + one atomicAdd per warp): the frontier
// compaction.  All 32 lanes must call it.
__device__ __forceinline__ void warp_push(bool pred, uint32_t val, uint32_t *q, unsigned *cnt,
                                          uint32_t cap, Ctl *ctl, int where)
{
    unsigned m = __ballot_sync(FULL, pred);
    if (m == 0u) return;
    unsigned lane = lane_id();
    unsigned ld = __ffs(m) - 1u;
    unsigned base = 0;
    if (lane == ld) base = atomicAdd(cnt, (unsigned)__popc(m));
    base = __shfl_sync(FULL, base, ld);
    if (pred) {
        unsigned pos = base + __popc(m & ((1u << lane) - 1u));
        if (pos < cap) q[pos] = val;
        else set_error(ctl, E_OVERFLOW, where);
    }
}

// Staging of queue appends in shared memory: every warp appends into its
// own slice (warp ballot, no atomics); a full slice is written out by its
// warp with one global atomicAdd per qcap entries, and bq_flush writes the
// rest of all slices with one global atomicAdd per CTA and pass.  This keeps
// the global queue tail from becoming a same-address atomic hot spot.
__device__ __forceinline__ void bq_init()
{
    for (unsigned i = threadIdx.x; i < BQ_HDR; i += blockDim.x) sccb_dsmem[i] = 0u;
    if (threadIdx.x == 0) *cta_err() = 0;
    __syncthreads();
}

__device__ __forceinline__ void bq_push(unsigned qi, bool pred, uint32_t val, uint32_t qcap, uint32_t *gq,
                                        unsigned *gcnt, uint32_t gcap, Ctl *ctl, int where)
{
    const unsigned m = __ballot_sync(FULL, pred);
    if (m == 0u) return;
    const unsigned lane = lane_id(), wi = threadIdx.x >> 5;
    uint32_t *slice = &sccb_dsmem[BQ_HDR + (qi * (blockDim.x >> 5) + wi) * qcap];
    unsigned *wc = &sccb_dsmem[BQ_CNT + qi * BQ_WARPS + wi];
    unsigned cnt = *wc;
    const unsigned n = __popc(m);
    if (cnt + n > qcap) {
        unsigned base = 0;
        if (lane == 0) base = atomicAdd(gcnt, cnt);
        base = __shfl_sync(FULL, base, 0);
        for (unsigned i = lane; i < cnt; i += 32u) {
            if (base + i < gcap) gq[base + i] = slice[i];
            else set_error(ctl, E_OVERFLOW, where);
        }
        __syncwarp();
        cnt = 0;
    }
    if (pred) slice[cnt + __popc(m & ((1u << lane) - 1u))] = val;
    __syncwarp();
    if (lane == 0) *wc = cnt + n;
    __syncwarp();
}

// K appends per lane in one go: one reading and one writing of the slice's
// fill count instead of K (a slice too small for 32 * K entries takes them
// one by one).
template <int K>
__device__ __forceinline__ void bq_pushK(unsigned qi, const bool (&pred)[K], const uint32_t (&val)[K], uint32_t qcap,
                                         uint32_t *gq, unsigned *gcnt, uint32_t gcap, Ctl *ctl, int where)
{
    if (qcap < 32u * K) {
#pragma unroll
        for (int j = 0; j < K; j++) bq_push(qi, pred[j], val[j], qcap, gq, gcnt, gcap, ctl, where);
        return;
    }
    unsigned m[K], n = 0;
#pragma unroll
    for (int j = 0; j < K; j++) {
        m[j] = __ballot_sync(FULL, pred[j]);
        n += __popc(m[j]);
    }
    if (n == 0u) return;
    const unsigned lane = lane_id(), wi = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    uint32_t *slice = &sccb_dsmem[BQ_HDR + (qi * (blockDim.x >> 5) + wi) * qcap];
    unsigned *wc = &sccb_dsmem[BQ_CNT + qi * BQ_WARPS + wi];
    unsigned cnt = *wc;
    if (cnt + n > qcap) {
        unsigned base = 0;
        if (lane == 0) base = atomicAdd(gcnt, cnt);
        base = __shfl_sync(FULL, base, 0);
        for (unsigned i = lane; i < cnt; i += 32u) {
            if (base + i < gcap) gq[base + i] = slice[i];
            else set_error(ctl, E_OVERFLOW, where);
        }
        __syncwarp();
        cnt = 0;
    }
    unsigned at = cnt;
#pragma unroll
    for (int j = 0; j < K; j++) {
        if (pred[j]) slice[at + __popc(m[j] & lt)] = val[j];
        at += __popc(m[j]);
    }
    __syncwarp();
    if (lane == 0) *wc = at;
    __syncwarp();
}

// Takes up to 32 of the newest entries off the warp's slice of queue qi, if
// it holds least to most of them; lane l < the result gets one in val.
__device__ __forceinline__ unsigned bq_pop(unsigned qi, uint32_t qcap, uint32_t least, uint32_t most,
                                           uint32_t &val)
{
    const unsigned wi = threadIdx.x >> 5, lane = lane_id();
    const uint32_t *slice = &sccb_dsmem[BQ_HDR + (qi * (blockDim.x >> 5) + wi) * qcap];
    unsigned *wc = &sccb_dsmem[BQ_CNT + qi * BQ_WARPS + wi];
    const unsigned cnt = *wc;
    if (cnt < least || cnt > most) return 0u;
    const unsigned n = min(cnt, 32u);
    val = lane < n ? slice[cnt - n + lane] : 0u;
    __syncwarp();
    if (lane == 0) *wc = cnt - n;
    __syncwarp();
    return n;
}

// Adds x to the CTA's tally qi (words 12 .. 14): the frontier edges of queues
// 0 and 1, and the scope left by a bottom-up step.
__device__ __forceinline__ void bq_add_edges(unsigned qi, unsigned x)
{
    x = __reduce_add_sync(FULL, x);
    if (lane_id() == 0 && x) atomicAdd(&sccb_dsmem[12 + qi], x);
}

// Called by every thread of the CTA at the end of a pass.  ecnt0, ecnt1 and
// scnt (optional) receive the CTA's tallies.
__device__ __forceinline__ void bq_flush(unsigned nq, uint32_t qcap, uint32_t *gq0, unsigned *gcnt0, uint32_t *gq1,
                                         unsigned *gcnt1, uint32_t gcap, Ctl *ctl, unsigned *ecnt0 = nullptr,
                                         unsigned *ecnt1 = nullptr, unsigned *scnt = nullptr)
{
    __syncthreads();
    const unsigned nw = blockDim.x >> 5;
    const unsigned wi = threadIdx.x >> 5;
    // warp q lays out queue q: the warps' fill counts scanned by shuffles,
    // one global atomicAdd for the CTA's room; the queues' atomics overlap
    for (unsigned qi = wi; qi < nq; qi += nw) {
        const unsigned ln = lane_id();
        const unsigned c = ln < nw ? sccb_dsmem[BQ_CNT + qi * BQ_WARPS + ln] : 0u;
        unsigned incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(FULL, incl, o);
            if (ln >= (unsigned)o) incl += y;
        }
        if (ln < nw) sccb_dsmem[BQ_PRE + qi * BQ_WARPS + ln] = incl - c;
        const unsigned total = __shfl_sync(FULL, incl, 31);
        if (ln == 0) {
            sccb_dsmem[8 + qi] = total ? atomicAdd(qi ? gcnt1 : gcnt0, total) : 0u;
            unsigned *ec = qi ? ecnt1 : ecnt0;
            if (ec && sccb_dsmem[12 + qi]) atomicAdd(ec, sccb_dsmem[12 + qi]);
            sccb_dsmem[12 + qi] = 0u;
            if (qi == 0) {
                if (scnt && sccb_dsmem[14]) atomicAdd(scnt, sccb_dsmem[14]);
                sccb_dsmem[14] = 0u;
            }
        }
    }
    __syncthreads();
    for (unsigned qi = 0; qi < nq; qi++) {
        uint32_t *gq = qi ? gq1 : gq0;
        const unsigned cnt = sccb_dsmem[BQ_CNT + qi * BQ_WARPS + wi];
        const unsigned base = sccb_dsmem[8 + qi] + sccb_dsmem[BQ_PRE + qi * BQ_WARPS + wi];
        const uint32_t *slice = &sccb_dsmem[BQ_HDR + (qi * nw + wi) * qcap];
        for (unsigned i = lane_id(); i < cnt; i += 32u) {
            if (base + i < gcap) gq[base + i] = slice[i];
            else set_error(ctl, E_OVERFLOW, 3);
        }
        __syncwarp();
        if (lane_id() == 0) sccb_dsmem[BQ_CNT + qi * BQ_WARPS + wi] = 0u;
    }
}

__device__ __forceinline__ unsigned warp_incl_scan(unsigned x)
{
    unsigned lane = lane_id();
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned y = __shfl_up_sync(FULL, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    return x;
}

// Append nch chunk descriptors (v, 0..nch-1) per lane.  All lanes call.
__device__ __forceinline__ void warp_push_chunks(uint32_t v, uint32_t nch, uint2 *hq, unsigned *hcnt,
                                                 uint32_t hcap, Ctl *ctl)
{
    unsigned incl = warp_incl_scan(nch);
    unsigned total = __shfl_sync(FULL, incl, 31);
    if (total == 0u) return;
    unsigned base = 0;
    if (lane_id() == 0) base = atomicAdd(hcnt, total);
    base = __shfl_sync(FULL, base, 0);
    unsigned pos = base + incl - nch;
    if (pos + nch > hcap) { if (nch) set_error(ctl, E_OVERFLOW, 2); return; }
    for (uint32_t c = 0; c < nch; c++) hq[pos + c] = make_uint2(v, c);
}

// First pusher of u for pass tag wins (stamp dedup of work lists).
__device__ __forceinline__ bool stamp_claim(uint32_t *stamp, uint32_t u, uint32_t tag)
{
    if (stamp[u] >= tag) return false;
    return atomicMax(&stamp[u], tag) < tag;
}

// Load-balanced expansion of up to 32 adjacency lists held one per lane
// (merge-path style): the warp walks the concatenation of the lists 32
// entries at a time, each lane finds its owner by a 5-step binary search
// over the exclusive scan of the degrees.  fn(valid, neighbour, owner's lane)
// is called by all lanes on every step.  Degrees must be <= HEAVY_T.
template <class Fn>
__device__ __forceinline__ unsigned lbs_walk(uint32_t beg, uint32_t deg, const uint32_t *__restrict__ C, Fn &&fn)
{
    unsigned incl = warp_incl_scan(deg);
    unsigned total = __shfl_sync(FULL, incl, 31);
    unsigned excl = incl - deg;
    unsigned lane = lane_id();
    for (unsigned base = 0; base < total; base += 32u) {
        unsigned e = base + lane;
        unsigned lo = 0;
#pragma unroll
        for (unsigned step = 16; step >= 1; step >>= 1) {
            unsigned cand = lo + step;
            unsigned x = __shfl_sync(FULL, excl, cand & 31u);
            if (cand < 32u && x <= e) lo = cand;
        }
        unsigned ex_o = __shfl_sync(FULL, excl, lo);
        unsigned beg_o = __shfl_sync(FULL, beg, lo);
        bool valid = e < total;
        uint32_t nbr = valid ? __ldg(&C[beg_o + (e - ex_o)]) : 0u;
        fn(valid, nbr, lo);
    }
    return total;
}

// Same walk, two entries per lane per step so that each lane has two
// independent gathers in flight: fn(v0, n0, lane0, v1, n1, lane1).
template <class Fn>
__device__ __forceinline__ unsigned lbs_walk2(uint32_t beg, uint32_t deg, const uint32_t *__restrict__ C, Fn &&fn)
{
    unsigned incl = warp_incl_scan(deg);
    unsigned total = __shfl_sync(FULL, incl, 31);
    unsigned excl = incl - deg;
    unsigned lane = lane_id();
    for (unsigned base = 0; base < total; base += 64u) {
        const unsigned e0 = base + lane, e1 = e0 + 32u;
        unsigned lo0 = 0, lo1 = 0;
#pragma unroll
        for (unsigned step = 16; step >= 1; step >>= 1) {
            unsigned c0 = lo0 + step, c1 = lo1 + step;
            unsigned x0 = __shfl_sync(FULL, excl, c0 & 31u);
            unsigned x1 = __shfl_sync(FULL, excl, c1 & 31u);
            if (c0 < 32u && x0 <= e0) lo0 = c0;
            if (c1 < 32u && x1 <= e1) lo1 = c1;
        }
        const unsigned x0 = __shfl_sync(FULL, excl, lo0), x1 = __shfl_sync(FULL, excl, lo1);
        const unsigned b0 = __shfl_sync(FULL, beg, lo0), b1 = __shfl_sync(FULL, beg, lo1);
        const bool v0 = e0 < total, v1 = e1 < total;
        const uint32_t n0 = v0 ? __ldg(&C[b0 + (e0 - x0)]) : 0u;
        const uint32_t n1 = v1 ? __ldg(&C[b1 + (e1 - x1)]) : 0u;
        fn(v0, n0, lo0, v1, n1, lo1);
    }
    return total;
}

// Same walk, four entries per lane per step: fn(valid[4], neighbour[4],
// owner's lane[4]).
template <class Fn>
__device__ __forceinline__ unsigned lbs_walk4(uint32_t beg, uint32_t deg, const uint32_t *__restrict__ C, Fn &&fn)
{
    const unsigned incl = warp_incl_scan(deg), total = __shfl_sync(FULL, incl, 31), excl = incl - deg;
    const uint32_t at = beg - excl;   // entry e of a list lies at C[at of its owner + e]
    for (unsigned base = 0; base < total; base += 128u) {
        bool ok[4];
        uint32_t n[4];
        unsigned own[4];
#pragma unroll
        for (unsigned j = 0; j < 4u; j++) {
            const unsigned e = base + 32u * j + lane_id();
            unsigned lo = 0;
#pragma unroll
            for (unsigned step = 16; step >= 1; step >>= 1) {
                const unsigned x = __shfl_sync(FULL, excl, (lo + step) & 31u);
                if (lo + step < 32u && x <= e) lo += step;
            }
            const uint32_t a = __shfl_sync(FULL, at, lo);
            ok[j] = e < total;
            n[j] = ok[j] ? __ldg(&C[a + e]) : 0u;
            own[j] = lo;
        }
        fn(ok, n, own);
    }
    return total;
}

// The same with one value per owner: fn(v0, n0, aux0, v1, n1, aux1).
template <class Fn>
__device__ __forceinline__ unsigned lbs_expand2(uint32_t beg, uint32_t deg, uint32_t aux,
                                                const uint32_t *__restrict__ C, Fn &&fn)
{
    return lbs_walk2(beg, deg, C, [&](bool v0, uint32_t n0, unsigned l0, bool v1, uint32_t n1, unsigned l1) {
        const uint32_t a0 = __shfl_sync(FULL, aux, l0), a1 = __shfl_sync(FULL, aux, l1);
        fn(v0, n0, a0, v1, n1, a1);
    });
}

// Fold member v into smin[rep] (the canonical label of rep's SCC): lanes
// sharing rep reduce first, one atomicMin per group, skipped when the
// stored value is already smaller.  All 32 lanes call.
__device__ __forceinline__ void smin_fold(bool valid, uint32_t rep, uint32_t v, uint32_t *smin)
{
    const unsigned vm = __ballot_sync(FULL, valid);
    if (vm == 0u) return;
    const uint32_t rep0 = __shfl_sync(FULL, rep, __ffs(vm) - 1);
    if (__all_sync(FULL, !valid || rep == rep0)) {   // one SCC for the whole warp (the common case)
        const uint32_t mn = __reduce_min_sync(FULL, valid ? v : 0xFFFFFFFFu);
        if (lane_id() == 0 && mn < vld(&smin[rep0])) atomicMin(&smin[rep0], mn);
        return;
    }
    unsigned grp = __match_any_sync(FULL, valid ? rep : 0xFFFFFFFFu);
    uint32_t mn = __reduce_min_sync(grp, valid ? v : 0xFFFFFFFFu);
    if (valid && lane_id() == (unsigned)(__ffs(grp) - 1) && mn < vld(&smin[rep])) atomicMin(&smin[rep], mn);
}

// Virtual-warp expansion: groups of W = 1 << lw lanes share a vertex and
// stride over its adjacency (the reference's fwd_warp/bwd_warp schedule,
// include/scc_kernels.h:46-105), K vertices per lane group at once: the K
// lists are walked in the same steps,
// so every lane has K gathers in flight.  fn(j, valid, nbr) per entry, in
// pairs of j; returns the entries of the warp.
template <int K, class Fn>
__device__ __forceinline__ unsigned vw_expandK(const uint32_t (&beg)[K], const uint32_t (&deg)[K], unsigned lw,
                                               const uint32_t *__restrict__ C, Fn &&fn)
{
    const unsigned W = 1u << lw;
    const unsigned sub = lane_id() & (W - 1u);
    unsigned md = 0, own = 0;
#pragma unroll
    for (int j = 0; j < K; j++) {
        md = max(md, deg[j]);
        own += deg[j];
    }
    const unsigned maxd = __reduce_max_sync(FULL, md);
    for (unsigned base = 0; base < maxd; base += W) {
        const unsigned k = base + sub;
        uint32_t n[K];
        bool v[K];
#pragma unroll
        for (int j = 0; j < K; j++) {
            v[j] = k < deg[j];
            n[j] = v[j] ? __ldg(&C[beg[j] + k]) : 0u;
        }
#pragma unroll
        for (int j = 0; j < K; j += 2) fn(j, v[j], n[j], v[j + 1], n[j + 1]);
    }
    return __reduce_add_sync(FULL, sub == 0u ? own : 0u);
}

// Minimum of x over the CTA folded into *dst with one atomicMin by thread 0
// (skipped when *dst is already smaller).  Called by every thread of the
// CTA; 0xFFFFFFFF means "nothing".  Used where every member found in a pass
// belongs to the same SCC, so its canonical label needs one atomic per CTA
// rather than one per warp on the same word.
__device__ __forceinline__ void block_min_atomic(uint32_t x, uint32_t *dst)
{
    __shared__ uint32_t s_min[32];
    const uint32_t m = __reduce_min_sync(FULL, x);
    const unsigned wi = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane_id() == 0) s_min[wi] = m;
    __syncthreads();
    if (wi == 0) {
        const uint32_t r = __reduce_min_sync(FULL, lane_id() < nw ? s_min[lane_id()] : 0xFFFFFFFFu);
        if (lane_id() == 0 && r != 0xFFFFFFFFu && r < *(volatile uint32_t *)dst) atomicMin(dst, r);
    }
    __syncthreads();
}

// 64-bit max of a pivot key over the warp, then the CTA; the CTA's thread 0
// performs one atomicMax.  With dst32 set, the 32-bit max of x goes to
// dst32 in the same two barriers.  Called by every thread of the CTA.
__device__ __forceinline__ void block_max_atomic(unsigned long long key, unsigned long long *dst, uint32_t x = 0u,
                                                 uint32_t *dst32 = nullptr)
{
    __shared__ unsigned long long s_red[32];
    __shared__ uint32_t s_x[32];
    unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    unsigned mhi = __reduce_max_sync(FULL, hi);
    unsigned mlo = __reduce_max_sync(FULL, hi == mhi ? lo : 0u);
    unsigned long long wk = ((unsigned long long)mhi << 32) | mlo;
    unsigned w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t mx = dst32 ? __reduce_max_sync(FULL, x) : 0u;
    if (lane_id() == 0) { s_red[w] = wk; s_x[w] = mx; }
    __syncthreads();
    if (w == 0) {
        const unsigned long long k = lane_id() < nw ? s_red[lane_id()] : 0ull;
        const unsigned khi = __reduce_max_sync(FULL, (unsigned)(k >> 32));
        const unsigned klo = __reduce_max_sync(FULL, (unsigned)(k >> 32) == khi ? (unsigned)k : 0u);
        const unsigned long long m = ((unsigned long long)khi << 32) | klo;
        if (lane_id() == 0 && m && m > *(volatile unsigned long long *)dst) atomicMax(dst, m);
        if (dst32) {
            const uint32_t r = __reduce_max_sync(FULL, lane_id() < nw ? s_x[lane_id()] : 0u);
            if (lane_id() == 0 && r > *(volatile uint32_t *)dst32) atomicMax(dst32, r);
        }
    }
    __syncthreads();
}

// Pivot key (scc_kernels.cu:643-656): uint32 product of full-graph out- and
// in-degree, larger wins; ties go to the smaller id.  Never 0 for v <= MAX_V.
__device__ __forceinline__ unsigned long long pivot_key(const Graph &g, uint32_t v)
{
    uint32_t prod = (__ldg(&g.Fr[v + 1]) - __ldg(&g.Fr[v])) * (__ldg(&g.Br[v + 1]) - __ldg(&g.Br[v]));
    return ((unsigned long long)prod << 32) | (unsigned long long)(0xFFFFFFFFu - v);
}
__device__ __forceinline__ uint32_t key_vertex(unsigned long long k) { return 0xFFFFFFFFu - (uint32_t)k; }

}  // namespace sccb
