// update.cu -- the batch-update kernels of the dynamic SSSP engine (sm_103a).
//
// One batch (replaces SSSPmainForUndirected.cu:196-281) is four launches on one stream:
//   k_prepare   clear the control block and the deletion set, bring the records from pinned host
//               memory and validate them
//   k_delete    the child end of a deleted tree edge is cut off and every adjacency entry
//               matching a deletion is tombstoned (binary search in the sorted row prefix +
//               scan of older appended entries); deletions also go into a device hash set
//               (replaces deleteEdge, gpuFunctions_undir.cuh:179-215)
//   k_append    insertions that no deletion of the batch removes go into row slack (atomic
//               degree bump, both directions).  The reference appends every insertion and
//               then tombstones matches (all_structure_undir.cuh:106-117 before
//               gpuFunctions_undir.cuh:201-213); skipping the removed ones gives the same graph.
//               Each surviving insertion then relaxes both ends and seeds the first frontier
//               (replaces insertEdge, gpuFunctions_undir.cuh:217-251)
//   k_update    one persistent cooperative kernel with a bounded grid barrier:
//               0. rows that the insertions overflow grow (grow.cuh)
//               A. cut-off subtrees are walked level by level from the roots (replaces
//                  filterAffectedNodes + updateNeighbors_del and its host loop,
//                  gpuFunctions_undir.cuh:125-144, 312-349, MAIN:219-239); after bfs_levels
//                  levels it switches to pointer jumping over the parent array.  The walk
//                  follows the parent words as k_append left them, so an end relaxed from a
//                  vertex that turns out to be cut off is cut off with it.
//               B. every cut-off vertex pulls its best live neighbour
//               C. frontier relaxation rounds with 64-bit atomicMin on the packed
//                  (dist, parent) word until the frontier is empty (replaces
//                  filterAllAffected + updateNeighbors and its host loop,
//                  gpuFunctions_undir.cuh:162-174, 370-433, MAIN:263-281).  With a bucket
//                  width delta > 0 the rounds are near-far ordered: a vertex whose new
//                  distance is at or above the threshold T waits in a de-duplicated far list;
//                  when the near frontier runs dry, T moves on and the far list is split
//                  again.  Small levels and rounds run as local stretches in the CTAs' queues.  High-diameter graphs then settle most
//                  vertices once instead of once per improving wave.  The result is the same
//                  fixpoint: exact distances, the same parents.
// Load balance: a vertex entering a frontier is split by degree into work items -- rows of
// at most te edges are one thread's item, longer rows up to large_deg become ceil(deg/te)
// thread items (a warp's worth for a few hundred edges), longer ones become CTA items of
// `chunk` edges -- so every round is one even wave over all threads.
#include <cuda_runtime.h>

#include "engine.cuh"

namespace dsssp {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr unsigned kSpinLimit = 1u << 20;  // polls of ~1 us: a barrier gives up after ~1 s
constexpr int kMaxWarps = 8;               // update kernel blocks have at most 256 threads
constexpr int kBuf = 176;                  // per-warp push buffer entries (16 bytes each: four
                                           // CTAs of the update kernel stay within 100 KB of
                                           // shared memory, which leaves the L1 its 156 KB)
constexpr int kListRegion = 512;           // per-warp u32 staging of the batch front kernels
constexpr int kAddsPerCheck = 32;          // entries a warp may add between two flush checks
                                           // (one add of up to 32 lanes; visit4 reserves room
                                           // for its four adds instead)
static_assert(kBuf > kAddsPerCheck, "a push buffer must take one visit's adds after a check");
constexpr int kSoloSteps = 256;            // consecutive solo steps before the grid re-syncs
constexpr unsigned kQueue = 256;           // items of a CTA's queue in a local stretch (two queues)
constexpr int kLocalTe = 16;               // thread items of more edges than this keep to the rounds
constexpr unsigned kFewHops = 16;          // an advance that buys fewer is widened (see advance)
constexpr unsigned kFarBuf = 64;           // per-warp staging of far-list pushes
constexpr int kSpill = 64;                 // per-warp staging of vertices that leave a stretch
constexpr unsigned kStretch = 256;         // steps of a local stretch at most
constexpr unsigned kShortStretch = 4, kMinRest = 8, kMaxRest = 256;  // see after_stretch
static_assert(64 * (kLocalTe / 4) <= kQueue, "a CTA's first items must fit its queue");
// a stretch keeps all of it in the push buffers: kSpill entries a warp for vertices that leave it,
// the queues (two, and a third for the walk), the far staging in the third one's place
constexpr unsigned kQueueAt = kSpill * kMaxWarps, kFarAt = kQueueAt + 2 * kQueue;
static_assert(kQueueAt + 3 * kQueue <= kBuf * kMaxWarps && kMaxWarps * kFarBuf / 4 <= kQueue && kSpill >= 2 * 32,
              "a stretch fits the push buffers");

__shared__ unsigned s_nbar;        // grid barriers this CTA has passed
__shared__ unsigned s_gen;         // barrier generation this CTA waits on next (ctl->bar_gen)
__shared__ unsigned s_ggen;        // group-barrier generation this CTA waits on next (ctl->grp_gen)
// List counters of solo steps (CTA 0 alone): (thread items, CTA items) per slot, slots used
// like the control block's three rotating counters.  Shared-memory atomics and reads save a
// global round trip each per step.
__shared__ unsigned s_solo_cnt[3][2];
__shared__ unsigned s_spin_limit;  // polls before a grid barrier gives up
__shared__ uint4 s_pbuf[kMaxWarps][kBuf];  // (vertex, degree, row start) pushed, not yet expanded
__shared__ unsigned s_done[2];             // ... where a step's items go in the walk's done list
__shared__ unsigned s_stop[2];             // ... another CTA has ended the stretch (seen in a step, read in the next)
__shared__ unsigned s_qcnt[3];             // local stretches: items of the steps' queues, rotating
__shared__ unsigned s_near[2];  // advance: the sizes of the near list
__shared__ unsigned long long s_threshold;
__shared__ unsigned long long s_width;  // near-far: the bucket width
__shared__ unsigned s_advanced;         // ... the hops as of the last advance
__shared__ unsigned long long s_lstat[8];  // ... their counters, added to the kernel's at the end
__shared__ unsigned s_wlist[kMaxWarps][kListRegion];  // k_delete / k_append list staging

// Per-thread counters (32 bits: a thread's share stays far below 2^32 in any run; the block
// sums in flush_stats are 64-bit), few registers in the register-bound update kernel.
struct LocalStats {
    unsigned edges_relax = 0, edges_inv = 0, updates = 0, dist_ovf = 0, frontier = 0, items = 0, marked = 0,
             edges_pull = 0;
};

// Grid-wide barrier for a cooperative launch.  The wait is bounded: on timeout the status
// word gets DSSSP_E_TIMEOUT (with where it happened in ctl->diag) and every CTA leaves at
// its next barrier.  Returns false when the kernel must stop (timeout or any error).  Each
// CTA tracks the generation it waits on (s_gen, read once at kernel start: no barrier can
// complete before every CTA has arrived), so arriving costs no load.  With a and b given,
// the two counters the caller needs next are read once per CTA together with the status
// word and returned in va and vb.  The chain is a fence, the arrival, the last arrival's fence and
// store, the pollers' load and fence and the load of the counters: the arrivals are counted through
// the launch, not from 0 each time, so that nothing is reset in between (a barrier 1 us less: the
// update kernel on RMAT-20 0.142 -> 0.131 ms, on 64 pooled graphs 0.402 -> 0.388 ms).  The polls
// order nothing and the fence comes once behind them: an acquiring poll throws away the L1
// of its SM each time, also for the CTAs that still work there (the walk of ER graphs of
// 10k and 300k vertices 0.073 -> 0.062 and 0.100 -> 0.090 ms).
__device__ bool grid_sync(Ctl* ctl, const unsigned* a, const unsigned* b, unsigned& va, unsigned& vb,
                          const unsigned* c, unsigned& vc) {
    __shared__ int s_go;
    __shared__ unsigned s_va, s_vb, s_vc;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned gen = s_gen;
        __threadfence();
        const unsigned arrived = atomicAdd(&ctl->bar_count, 1u);
        if (arrived + 1 == (s_nbar + 1) * gridDim.x) {
            __threadfence();
            st_relaxed(&ctl->bar_gen, gen + 1);
        } else {
            unsigned spins = 0;
            while (ld_relaxed(&ctl->bar_gen) == gen) {
                if (++spins > s_spin_limit) {
                    if (atomicCAS(&ctl->status, 0, -6 /* DSSSP_E_TIMEOUT */) == 0) {
                        ctl->diag[0] = s_nbar;
                        ctl->diag[1] = atomicAdd(&ctl->bar_count, 0u) - s_nbar * gridDim.x;
                    }
                    atomicAdd(&ctl->diag[2], 1u);
                    break;
                }
                __nanosleep(spins < 32 ? 32 : (spins < 2048 ? 200 : 1000));  // long waits: solo steps
            }
            __threadfence();
        }
        s_gen = gen + 1;
        s_nbar++;
        const int st = __ldcg(&ctl->status);
        s_va = a ? __ldcg(a) : 0u;
        s_vb = b ? __ldcg(b) : 0u;
        s_vc = c ? __ldcg(c) : 0u;
        s_go = st == 0;
    }
    __syncthreads();
    va = s_va;
    vb = s_vb;
    vc = s_vc;
    return s_go != 0;
}

__device__ __forceinline__ bool grid_sync(Ctl* ctl, const unsigned* a, const unsigned* b, unsigned& va, unsigned& vb) {
    unsigned x;
    return grid_sync(ctl, a, b, va, vb, nullptr, x);
}

// Barrier of the first G CTAs (a group running mid-size steps while the others wait at the
// next grid barrier): like grid_sync, bounded, with the counters the caller needs next read
// once per CTA after the release.  Every CTA of the group calls it the same number of times.
__device__ bool group_sync(Ctl* ctl, unsigned G, const unsigned* a, const unsigned* b, unsigned& va, unsigned& vb) {
    __shared__ int s_go;
    __shared__ unsigned s_va, s_vb;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned gen = s_ggen;
        __threadfence();
        const unsigned arrived = atomicAdd(&ctl->grp_count, 1u);
        if (arrived == G - 1) {
            atomicExch(&ctl->grp_count, 0u);
            __threadfence();
            st_release(&ctl->grp_gen, gen + 1);
        } else {
            unsigned spins = 0;
            while (ld_acquire(&ctl->grp_gen) == gen) {
                if (++spins > s_spin_limit) {
                    if (atomicCAS(&ctl->status, 0, -6 /* DSSSP_E_TIMEOUT */) == 0) {
                        ctl->diag[0] = 0x80000000u | s_nbar;  // high bit: a group barrier
                        ctl->diag[1] = atomicAdd(&ctl->grp_count, 0u);
                    }
                    atomicAdd(&ctl->diag[2], 1u);
                    break;
                }
                if (spins > 32) __nanosleep(spins < 4096 ? 64 : 1000);
            }
        }
        __threadfence();
        s_ggen = gen + 1;
        const int st = __ldcg(&ctl->status);
        s_va = __ldcg(a);
        s_vb = __ldcg(b);
        s_go = st == 0;
    }
    __syncthreads();
    va = s_va;
    vb = s_vb;
    return s_go != 0;
}

__device__ __forceinline__ bool grid_sync(Ctl* ctl) {
    unsigned x, y;
    return grid_sync(ctl, nullptr, nullptr, x, y);
}

// Offers distance nd through parent u to vertex c whose current word is cur.  Returns true
// when c's distance went down (c must then be pushed).  Zero-weight edges only replace a
// strictly larger distance, so equal-distance parent swaps can never close a cycle.  A swap
// to a smaller parent id at the same distance (the packed minimum's tie rule) is recorded in
// chg_tag, so the batch's set of changed vertices stays complete.
__device__ __forceinline__ bool relax_to(const DevGraph& g, unsigned epoch, unsigned c, unsigned long long nd,
                                         unsigned u, int w, unsigned long long cur, LocalStats& ls) {
    unsigned long long* state = g.state;
    if (nd >= kDistInf) {
        if (cur == kInfState) ls.dist_ovf++;
        return false;
    }
    const unsigned long long cand = (nd << 32) | u;
    if (cand >= cur) return false;
    if (w > 0) {
        const unsigned long long old = atomicMin(&state[c], cand);
        if ((old >> 32) > nd) {
            ls.updates++;
            return true;
        }
        if (old > cand && g.chg_tag) g.chg_tag[c] = epoch;
        return false;
    }
    while ((cur >> 32) > nd) {
        const unsigned long long prev = atomicCAS(&state[c], cur, cand);
        if (prev == cur) {
            ls.updates++;
            return true;
        }
        cur = prev;
    }
    return false;
}

// The two seed relaxations of an insertion (u, v, w) with w > 0: v is offered ndv = d(u) + w
// through u and u is offered ndu = d(v) + w through v, from the states su, sv read before.
// Both atomicMin go out before either result is used; the outcome is that of two relax_to
// calls.  pu / pv: u / v went down and must be pushed.
__device__ __forceinline__ void relax_both(const DevGraph& g, unsigned epoch, unsigned u, unsigned v,
                                           unsigned long long ndv, unsigned long long ndu, unsigned long long su,
                                           unsigned long long sv, bool& pu, bool& pv, LocalStats& ls) {
    const bool from_u = (su >> 32) != kDistInf, from_v = (sv >> 32) != kDistInf;
    if (from_u && ndv >= kDistInf && sv == kInfState) ls.dist_ovf++;
    if (from_v && ndu >= kDistInf && su == kInfState) ls.dist_ovf++;
    const unsigned long long cv = (ndv << 32) | u, cu = (ndu << 32) | v;
    const bool tv = from_u && ndv < kDistInf && cv < sv;
    const bool tu = from_v && ndu < kDistInf && cu < su;
    const unsigned long long ov = tv ? atomicMin(&g.state[v], cv) : kInfState;
    const unsigned long long ou = tu ? atomicMin(&g.state[u], cu) : kInfState;
    pv = tv && (ov >> 32) > ndv;
    pu = tu && (ou >> 32) > ndu;
    ls.updates += (pv ? 1 : 0) + (pu ? 1 : 0);
    if (g.chg_tag) {
        if (tv && !pv && ov > cv) g.chg_tag[v] = epoch;
        if (tu && !pu && ou > cu) g.chg_tag[u] = epoch;
    }
}

// Destination of pushed vertices: a thread-item list and a CTA-item list with counters.
struct Out {
    Item* tl;
    unsigned* tcnt;
    long long tcap;
    Item* cl;
    unsigned* ccnt;
    long long ccap;
};

// Work items of the entries a lane holds in a push buffer (entries lane, lane + 32, ...).
__device__ __forceinline__ void buf_counts(const uint4* buf, int count, const UpdParams& p, unsigned& nt,
                                           unsigned& nc) {
    nt = nc = 0;
    for (int e = (int)lane_id(); e < count; e += 32) {
        const int deg = (int)buf[e].y;
        if (deg > p.large_deg) nc += (unsigned)((deg + p.chunk - 1) / p.chunk);
        else if (deg > 0) nt += (unsigned)((deg + p.te - 1) / p.te);
    }
}

// Writes those items from list positions ft (thread items) and fc (CTA items) on.
__device__ __forceinline__ void buf_write(const uint4* buf, int count, const UpdParams& p, const Out& o, unsigned ft,
                                          unsigned fc) {
    for (int e = (int)lane_id(); e < count; e += 32) {
        const uint4 x = buf[e];
        const int deg = (int)x.y;
        const long long start = (long long)(((unsigned long long)x.w << 32) | x.z);
        if (deg > p.large_deg) {
            for (int k = 0; k < deg; k += p.chunk) o.cl[fc++] = make_item(x.x, start + k, (unsigned)min(p.chunk, deg - k));
        } else if (deg > 0) {
            for (int k = 0; k < deg; k += p.te) o.tl[ft++] = make_item(x.x, start + k, (unsigned)min(p.te, deg - k));
        }
    }
}

__device__ __forceinline__ unsigned warp_incl_scan(unsigned x) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(kFull, x, o);
        if (lane_id() >= (unsigned)o) x += t;
    }
    return x;
}

#include "grow.cuh"

// Per-warp shared-memory buffer of pushed (vertex, degree, row start).  Entries are split into work
// items when the buffer is nearly full (one list-counter atomic per warp for up to kBuf
// vertices) and at the end of a phase (one atomic per CTA): the list counters are single
// words that every CTA appends to, so their atomics are kept few.
struct PushBuf {
    uint4* buf;
    int count;  // warp-uniform

    // pushes v with its row (start, deg) for every lane with pred
    __device__ __forceinline__ void add(bool pred, unsigned v, const RowDesc& rd) {
        const unsigned mask = __ballot_sync(kFull, pred);
        if (pred)
            buf[count + __popc(mask & ((1u << lane_id()) - 1u))] =
                make_uint4(v, (unsigned)rd.deg, (unsigned)rd.start, (unsigned)((unsigned long long)rd.start >> 32));
        count += __popc(mask);
        __syncwarp();
    }

    // the same with the ballot of pred at hand
    __device__ __forceinline__ void add_mask(unsigned mask, bool pred, unsigned v, const RowDesc& rd) {
        if (pred)
            buf[count + __popc(mask & ((1u << lane_id()) - 1u))] =
                make_uint4(v, (unsigned)rd.deg, (unsigned)rd.start, (unsigned)((unsigned long long)rd.start >> 32));
        count += __popc(mask);
    }

    // warp-collective: expands the buffer once it could not take another kAddsPerCheck
    __device__ __forceinline__ void flush(const UpdParams& p, const Out& o, LocalStats& ls) {
        if (count <= kBuf - kAddsPerCheck) return;
        expand_all(p, o, ls);
    }

    // warp-collective: makes room for n more entries (n warp-uniform, at most kBuf)
    __device__ __forceinline__ void reserve(unsigned n, const UpdParams& p, const Out& o, LocalStats& ls) {
        if ((unsigned)count + n <= (unsigned)kBuf) return;
        expand_all(p, o, ls);
    }

    // warp-collective: splits every buffered entry into work items (one atomic per list)
    __device__ __forceinline__ void expand_all(const UpdParams& p, const Out& o, LocalStats& ls) {
        unsigned nt, nc;
        buf_counts(buf, count, p, nt, nc);
        const unsigned it = warp_incl_scan(nt), ic = warp_incl_scan(nc);
        const unsigned tt = __shfl_sync(kFull, it, 31), tc = __shfl_sync(kFull, ic, 31);
        unsigned bt = 0, bc = 0;
        if (lane_id() == 0) {
            if (tt) bt = atomicAdd(o.tcnt, tt);
            if (tc) bc = atomicAdd(o.ccnt, tc);
        }
        bt = __shfl_sync(kFull, bt, 0);
        bc = __shfl_sync(kFull, bc, 0);
        if ((long long)bt + tt > o.tcap || (long long)bc + tc > o.ccap) {
            if (lane_id() == 0) set_status(p.g.ctl, -4 /* work list capacity: internal error */);
        } else {
            buf_write(buf, count, p, o, bt + it - nt, bc + ic - nc);
        }
        ls.items += nt + nc;
        count = 0;
        __syncwarp();
    }

    // CTA-collective (every thread of the CTA): expands what every warp still holds
    __device__ void flush_cta(const UpdParams& p, const Out& o, LocalStats& ls) {
        __shared__ unsigned s_t[kMaxWarps], s_c[kMaxWarps], s_bt, s_bc, s_ok;
        const unsigned w = threadIdx.x >> 5, nw = blockDim.x >> 5;
        unsigned nt, nc;
        buf_counts(buf, count, p, nt, nc);
        const unsigned it = warp_incl_scan(nt), ic = warp_incl_scan(nc);
        if (lane_id() == 31) {
            s_t[w] = it;
            s_c[w] = ic;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned tt = 0, tc = 0;
            for (unsigned k = 0; k < nw; k++) {
                const unsigned a = s_t[k], b = s_c[k];
                s_t[k] = tt;
                s_c[k] = tc;
                tt += a;
                tc += b;
            }
            s_bt = tt ? atomicAdd(o.tcnt, tt) : 0u;
            s_bc = tc ? atomicAdd(o.ccnt, tc) : 0u;
            s_ok = (long long)s_bt + tt <= o.tcap && (long long)s_bc + tc <= o.ccap;
            if (!s_ok) set_status(p.g.ctl, -4 /* work list capacity: internal error */);
        }
        __syncthreads();
        if (s_ok) buf_write(buf, count, p, o, s_bt + s_t[w] + it - nt, s_bc + s_c[w] + ic - nc);
        ls.items += nt + nc;
        count = 0;
        __syncthreads();
    }
};

// Claims c for the next frontier; its row descriptor (for the work items) is loaded alongside
// the claim.
__device__ __forceinline__ bool claim_with_row(const UpdParams& p, bool want, unsigned c, unsigned tag, RowDesc& rd) {
    rd = RowDesc{0, 0, 0};
    if (!want) return false;
    const RowDesc r = p.g.rows[c];
    const bool won = atomicExch(&p.g.push_tag[c], tag) != tag;
    rd = r;
    return won;
}

// The row descriptor of v when pred holds (an empty row otherwise).
__device__ __forceinline__ RowDesc row_if(const UpdParams& p, bool pred, unsigned v) {
    return pred ? p.g.rows[v] : RowDesc{0, 0, 0};
}

// Near-far ordering: pushes whose new distance is at or above the threshold T go to a far
// list, each vertex at most once per list generation (far_tag).  T = ~0 turns it off.
struct Far {
    unsigned* list;
    unsigned* cnt;
    unsigned* tag;
    unsigned gen;
    unsigned cap;
    unsigned long long T;
};

// Appends c to the far list for every lane with pred (warp-collective).
__device__ __forceinline__ void far_push(const UpdParams& p, const Far& f, bool pred, unsigned c) {
    if (pred) pred = atomicExch(&f.tag[c], f.gen) != f.gen;
    const unsigned mask = __ballot_sync(kFull, pred);
    if (mask == 0) return;
    const unsigned lane = lane_id();
    const unsigned leader = __ffs(mask) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(f.cnt, (unsigned)__popc(mask));
    base = __shfl_sync(kFull, base, leader);
    if ((unsigned long long)base + __popc(mask) > f.cap) {  // cannot happen: one entry per vertex
        if (lane == leader) set_status(p.g.ctl, -4);
        return;
    }
    if (pred) f.list[base + __popc(mask & ((1u << lane) - 1u))] = c;
}

// Appends c[q] for every pred[q] of every lane to the far list with one atomic per warp
// (warp-collective; the far tags are already claimed).
__device__ __forceinline__ void far_append4(const UpdParams& p, const Far& f, const bool (&pred)[4],
                                            const unsigned (&c)[4]) {
    unsigned cnt = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) cnt += pred[q] ? 1u : 0u;
    if (!__any_sync(kFull, cnt != 0)) return;
    const unsigned incl = warp_incl_scan(cnt);
    const unsigned total = __shfl_sync(kFull, incl, 31);
    unsigned base = 0;
    if (lane_id() == 31) base = atomicAdd(f.cnt, total);
    base = __shfl_sync(kFull, base, 31);
    if ((unsigned long long)base + total > f.cap) {  // cannot happen: one entry per vertex
        if (lane_id() == 31) set_status(p.g.ctl, -4);
        return;
    }
    unsigned at = base + incl - cnt;
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (pred[q]) f.list[at++] = c[q];
}

// Warp-aggregated offers: lanes offering to the same vertex c (offer set) are grouped with
// __match_any_sync; the group's least candidate word goes to its lowest lane (lead), the only
// one that issues the atomicMin, so a vertex offered by several lanes of a warp takes one
// atomic instead of one per lane.  Warp-collective; the loop runs (largest group - 1) times.
__device__ __forceinline__ void warp_agg_min(bool offer, unsigned c, unsigned long long& best, bool& lead) {
    const unsigned lane = lane_id();
    if (!__any_sync(kFull, offer)) return;
    // lanes without an offer get keys no vertex id takes (ids are below 2^31)
    const unsigned grp = __match_any_sync(kFull, offer ? c : 0x80000000u | lane);
    unsigned rem = grp & ~(1u << lane);
    while (__any_sync(kFull, rem != 0)) {
        const int src = rem ? __ffs(rem) - 1 : (int)lane;
        const unsigned long long o = __shfl_sync(kFull, best, src);
        best = o < best ? o : best;
        rem &= rem - 1;
    }
    lead = offer && (__ffs(grp) - 1) == (int)lane;
}

// ---- per-edge operations ---------------------------------------------------------------
// visit4 handles up to four adjacency entries per lane (a, a + stride, ... while below n; none for
// n <= 0) and is called by all 32 lanes.  A busy round makes 130-150 G visits a second, one random
// access to a neighbour's state each, about half of what loads alone reach in an array of the L2
// (280 G/s), so these accesses by themselves are not its bound.  Reading the next item early and
// leaving a visit in which no lane improved anything gained (the tree of RMAT scale 22 1.39 -> 1.35
// ms); prefetching the next items' entries (1.36 -> 1.40), adjacency words read by four lanes an
// item (1.361 -> 1.360) and states through the L1 (1.35 -> 1.32 in one build, 1.36 -> 1.37 in
// another) did not.  The other half of the cost is that an entry is visited about twice: that tree
// takes 132M visits for 67M entries.
template <bool kAgg>
struct RelaxOp {
    const UpdParams* p;
    unsigned tag;
    Out out;
    PushBuf pb;
    LocalStats* ls;
    Far far;
    // Offer by atomicMin alone, without first loading the neighbour's state to skip offers
    // that cannot win: one memory latency less per item, one atomic per edge instead of per
    // winning edge.  Used for steps of at most one wave of items, which wait on latency.
    bool direct;

    __device__ __forceinline__ unsigned long long prep(unsigned v) const { return __ldcg(&p->g.state[v]) >> 32; }
    __device__ __forceinline__ bool skip(unsigned long long du) const { return du >= kDistInf; }
    __device__ __forceinline__ void begin_lane(unsigned) {}
    __device__ __forceinline__ void end_lane(unsigned, bool) {}
    __device__ __forceinline__ void begin_group(unsigned) {}
    __device__ __forceinline__ void end_group(unsigned) {}
    __device__ __forceinline__ void finish() { pb.flush_cta(*p, out, *ls); }

    __device__ __forceinline__ void visit4(unsigned u, unsigned long long du, const int2* a, int n, int stride) {
        unsigned long long* state = p->g.state;
        int2 e[4];
#pragma unroll
        for (int q = 0; q < 4; q++) e[q] = q * stride < n ? ld_stream(a + q * stride) : make_int2(0, -1);
        unsigned long long cur[4];
#pragma unroll
        for (int q = 0; q < 4; q++) cur[q] = e[q].y >= 0 && !direct ? __ldcg(&state[e[q].x]) : kInfState;
        // The lane's four offers go out before any result is used, then its claims: two
        // memory latencies for the four edges instead of two per improving edge.  The
        // adjacency loads above were issued alongside the load of du (an unreachable u offers
        // nothing).
        const bool live = du < kDistInf;
        bool push[4], later[4];
        if constexpr (!kAgg) {
            unsigned long long old[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const unsigned long long nd = du + (unsigned)e[q].y;
                const bool offer = live && e[q].y > 0 && nd < kDistInf && ((nd << 32) | u) < cur[q];
                if (live && e[q].y > 0 && nd >= kDistInf &&
                    (direct ? __ldcg(&state[e[q].x]) : cur[q]) == kInfState)
                    ls->dist_ovf++;
                old[q] = offer ? atomicMin(&state[e[q].x], (nd << 32) | u) : 0ull;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const unsigned long long nd = du + (unsigned)e[q].y;
                const unsigned long long cand = (nd << 32) | u;
                push[q] = false;
                if (live && e[q].y > 0 && nd < kDistInf && cand < cur[q]) {
                    push[q] = (old[q] >> 32) > nd;
                    if (push[q]) ls->updates++;
                    else if (old[q] > cand && p->g.chg_tag) p->g.chg_tag[e[q].x] = p->epoch;
                } else if (live && e[q].y == 0) {  // zero weight: strict improvements only (compare-and-swap)
                    push[q] = relax_to(p->g, p->epoch, (unsigned)e[q].x, nd, u, 0,
                                       direct ? __ldcg(&state[e[q].x]) : cur[q], *ls);
                }
                later[q] = push[q] && nd >= far.T;
            }
        } else {
            // the lanes' offers to one vertex are reduced in the warp first: only the group's
            // least candidate word is issued, by the group's lowest lane
            unsigned long long old[4], best[4];
            bool lead[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const unsigned long long nd = du + (unsigned)e[q].y;
                const bool offer = live && e[q].y > 0 && nd < kDistInf && ((nd << 32) | u) < cur[q];
                if (live && e[q].y > 0 && nd >= kDistInf &&
                    (direct ? __ldcg(&state[e[q].x]) : cur[q]) == kInfState)
                    ls->dist_ovf++;
                best[q] = offer ? (nd << 32) | u : kInfState;
                lead[q] = offer;
                warp_agg_min(offer, (unsigned)e[q].x, best[q], lead[q]);
                old[q] = lead[q] ? atomicMin(&state[e[q].x], best[q]) : 0ull;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const unsigned long long nd = best[q] >> 32;  // the group's least distance
                push[q] = false;
                if (lead[q]) {
                    push[q] = (old[q] >> 32) > nd;
                    if (push[q]) ls->updates++;
                    else if (old[q] > best[q] && p->g.chg_tag) p->g.chg_tag[e[q].x] = p->epoch;
                } else if (live && e[q].y == 0) {  // zero weight: strict improvements only (compare-and-swap)
                    push[q] = relax_to(p->g, p->epoch, (unsigned)e[q].x, du, u, 0,
                                       direct ? __ldcg(&state[e[q].x]) : cur[q], *ls);
                }
                later[q] = push[q] && (e[q].y == 0 ? du : nd) >= far.T;
            }
        }
        if (live) ls->edges_relax += (unsigned)(n <= 0 ? 0 : min(4, (n + stride - 1) / stride));
        if (!__any_sync(kFull, push[0] || push[1] || push[2] || push[3])) return;
        unsigned ftag[4], ctag[4];
        RowDesc rd[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const unsigned c = (unsigned)e[q].x;
            const bool want = push[q] && !later[q];
            ftag[q] = later[q] ? atomicExch(&far.tag[c], far.gen) : far.gen;
            rd[q] = row_if(*p, want, c);
            ctag[q] = want ? atomicExch(&p->g.push_tag[c], tag) : tag;
        }
        bool fl[4], doit[4];
        unsigned fc[4], m[4], nadd = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            fl[q] = later[q] && ftag[q] != far.gen;
            fc[q] = (unsigned)e[q].x;
            doit[q] = push[q] && !later[q] && ctag[q] != tag;
            m[q] = __ballot_sync(kFull, doit[q]);
            nadd += __popc(m[q]);
        }
        if (nadd) {
            pb.reserve(nadd, *p, out, *ls);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                ls->frontier += doit[q] ? 1 : 0;
                pb.add_mask(m[q], doit[q], (unsigned)e[q].x, rd[q]);
            }
            __syncwarp();
        }
        if (far.T != ~0ull) far_append4(*p, far, fl, fc);
    }
};

struct MarkOp {
    const UpdParams* p;
    Out out;
    PushBuf pb;
    LocalStats* ls;

    __device__ __forceinline__ unsigned long long prep(unsigned) const { return 0; }
    __device__ __forceinline__ bool skip(unsigned long long) const { return false; }
    __device__ __forceinline__ void begin_lane(unsigned) {}
    __device__ __forceinline__ void end_lane(unsigned, bool) {}
    __device__ __forceinline__ void begin_group(unsigned) {}
    __device__ __forceinline__ void end_group(unsigned) {}
    __device__ __forceinline__ void finish() { pb.flush_cta(*p, out, *ls); }

    __device__ __forceinline__ void visit4(unsigned x, unsigned long long, const int2* a, int n, int stride) {
        unsigned long long* state = p->g.state;
        int2 e[4];
#pragma unroll
        for (int q = 0; q < 4; q++) e[q] = q * stride < n ? ld_stream(a + q * stride) : make_int2(0, -1);
        unsigned par[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
            par[q] = e[q].y >= 0 ? __ldcg(reinterpret_cast<const unsigned*>(&state[e[q].x])) : kNone;  // low word
        ls->edges_inv += (unsigned)(n <= 0 ? 0 : min(4, (n + stride - 1) / stride));
        bool child[4];
#pragma unroll
        for (int q = 0; q < 4; q++) child[q] = e[q].y >= 0 && par[q] == x;
        // a child is cut off even when already tagged: a root that an insertion of this batch
        // re-parented onto a vertex of a cut-off subtree must lose that distance.  The four
        // tag exchanges and degree loads go out before any result is used.
        unsigned old[4];
        RowDesc rd[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const unsigned c = (unsigned)e[q].x;
            if (child[q]) state[c] = kInfState;
            old[q] = child[q] ? atomicExch(&p->g.inv_tag[c], p->epoch) : p->epoch;
            rd[q] = row_if(*p, child[q], c);
        }
        unsigned m[4], nadd = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            m[q] = __ballot_sync(kFull, old[q] != p->epoch);
            nadd += __popc(m[q]);
        }
        pb.reserve(nadd, *p, out, *ls);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const bool mark = old[q] != p->epoch;
            ls->marked += mark ? 1 : 0;
            pb.add_mask(m[q], mark, (unsigned)e[q].x, rd[q]);
        }
        __syncwarp();
    }
};

struct PullOp {
    const UpdParams* p;
    unsigned tag;
    Out out;
    PushBuf pb;
    LocalStats* ls;
    Far far;
    unsigned long long best;
    bool need;

    // pushes x (pred) to the next round or, at or above the threshold, to the far list; d is
    // x's distance when the caller knows it (its own lowering atomicMin), else kDistInf
    __device__ __forceinline__ void route(bool pred, unsigned x, unsigned long long d) {
        const bool later = pred && far.T != ~0ull && (d < kDistInf ? d : __ldcg(&p->g.state[x]) >> 32) >= far.T;
        far_push(*p, far, later, x);
        RowDesc rd;
        const bool doit = claim_with_row(*p, pred && !later, x, tag, rd);
        ls->frontier += doit ? 1 : 0;
        pb.add(doit, x, rd);
        pb.flush(*p, out, *ls);
    }

    __device__ __forceinline__ unsigned long long prep(unsigned) const { return 0; }
    __device__ __forceinline__ bool skip(unsigned long long) const { return false; }
    __device__ __forceinline__ void begin_lane(unsigned) { best = kInfState; need = false; }
    __device__ __forceinline__ void begin_group(unsigned) { best = kInfState; need = false; }
    __device__ __forceinline__ void finish() { pb.flush_cta(*p, out, *ls); }

    __device__ __forceinline__ void visit4(unsigned x, unsigned long long, const int2* a, int n, int stride) {
        unsigned long long* state = p->g.state;
        int2 e[4];
#pragma unroll
        for (int q = 0; q < 4; q++) e[q] = q * stride < n ? ld_stream(a + q * stride) : make_int2(0, -1);
        unsigned long long s[4];
#pragma unroll
        for (int q = 0; q < 4; q++) s[q] = e[q].y >= 0 ? __ldcg(&state[e[q].x]) : kInfState;
        ls->edges_pull += (unsigned)(n <= 0 ? 0 : min(4, (n + stride - 1) / stride));
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (e[q].y < 0 || s[q] == kInfState) continue;
            const unsigned long long nd = (s[q] >> 32) + (unsigned)e[q].y;
            if (nd >= kDistInf) {
                ls->dist_ovf++;
                continue;
            }
            if (e[q].y > 0) {
                const unsigned long long cand = (nd << 32) | (unsigned)e[q].x;
                best = cand < best ? cand : best;
            } else if (relax_to(p->g, p->epoch, x, nd, (unsigned)e[q].x, 0, __ldcg(&state[x]), *ls)) {
                need = true;
            }
        }
    }
    // a lane's own item
    __device__ __forceinline__ void end_lane(unsigned x, bool valid) {
        bool improved = false;
        if (valid && best != kInfState) {
            const unsigned long long old = atomicMin(&p->g.state[x], best);
            if ((old >> 32) > (best >> 32)) {
                improved = true;
                ls->updates++;
            }
        }
        route(valid && (need || improved), x, improved ? best >> 32 : kDistInf);
    }
    // an item shared by the warp (part of a CTA item)
    __device__ __forceinline__ void end_group(unsigned x) {
        const unsigned long long b = warp_min_u64(best);
        const bool nd = __any_sync(kFull, need);
        bool improved = false;
        if (lane_id() == 0 && b != kInfState) {
            const unsigned long long old = atomicMin(&p->g.state[x], b);
            if ((old >> 32) > (b >> 32)) {
                improved = true;
                ls->updates++;
            }
        }
        route(lane_id() == 0 && (nd || improved), x, improved ? b >> 32 : kDistInf);
    }
};

// A step of nt thread items and nc CTA items is small when CTA 0 alone finishes it in at most
// `solo` waves (opts.solo_waves, default 2): then it skips the grid barrier, whose cost (~2.5 us
// plus the wait for the slowest CTA) exceeds the work.  solo 0: every step runs on the grid.
__device__ __forceinline__ bool small_step(unsigned nt, unsigned nc, unsigned solo) {
    return solo > 0 && (nt + blockDim.x - 1) / blockDim.x + nc <= solo;
}

// A step is mid-size when the group (the first G CTAs) finishes it in at most p.group_waves
// waves: it runs there with the group barrier, shorter than the grid's and waiting for the
// slowest of G chains instead of all CTAs'.
__device__ __forceinline__ bool group_step(const UpdParams& p, unsigned nt, unsigned nc) {
    const unsigned G = p.group_ctas;
    if (G < 2 || G >= gridDim.x || small_step(nt, nc, p.solo_waves)) return false;
    return (unsigned long long)(nt + blockDim.x - 1) / blockDim.x + nc <= (unsigned long long)G * p.group_waves;
}

// Processes one step's work on ncta CTAs (the whole grid, or CTA 0 alone for a small step;
// this CTA is number cta of them): CTA items first (one CTA per chunk of a long row; CTA
// items cta, cta + ncta, ...), then thread items (te edges each; the list tl2 behind tl) in one
// grid-stride wave over the ncta CTAs' threads.
template <class Op>
__device__ void run_items(Op& op, const UpdParams& p, const Item* tl, unsigned nt, const Item* cl, unsigned nc,
                          unsigned cta, unsigned ncta, const Item* tl2 = nullptr, unsigned nt2 = 0) {
    const unsigned lane = lane_id();
    const unsigned gtid = cta * blockDim.x + threadIdx.x;
    const unsigned nthreads = ncta * blockDim.x;
    // CTA items, split further while they are too few for the CTAs (a hub's row alone: 93 items of
    // 1,024 edges, all of which push, took 39 us on as many CTAs, in quarters 20 us)
    const unsigned parts = nc * 4 <= ncta ? 4u : nc * 2 <= ncta ? 2u : 1u;
    for (unsigned t = cta; t < nc * parts; t += ncta) {
        Item it = __ldcg(&cl[t / parts]);
        const unsigned long long du = __shfl_sync(kFull, op.prep(it.z), 0);
        if (op.skip(du)) continue;
        if (parts > 1) {
            const unsigned len = (it.w + parts - 1) / parts, from = min(it.w, len * (t % parts));
            it = make_item(it.z, item_lo(it) + from, min(len, it.w - from));
        }
        const long long lo = item_lo(it), hi = lo + (long long)it.w;
        op.begin_group(it.z);
        for (long long b = lo; b < hi; b += 4LL * blockDim.x)
            op.visit4(it.z, du, p.g.adj + b + threadIdx.x, (int)(hi - b) - (int)threadIdx.x, (int)blockDim.x);
        op.end_group(it.z);
    }
    // thread items: the item names its slots, so the adjacency loads go out alongside the
    // load of the vertex's own state (prep)
    auto load = [&](unsigned i) {
        return i < nt + nt2 ? __ldcg(i < nt ? &tl[i] : &tl2[i - nt]) : make_uint4(0u, 0u, 0u, 0u);
    };
    Item ahead = load(gtid);
    for (unsigned base = gtid - lane; base < nt + nt2; base += nthreads) {
        const unsigned i = base + lane;
        const bool has = i < nt + nt2;
        const Item it = ahead;
        ahead = load(i + nthreads);
        const unsigned long long du = has ? op.prep(it.z) : kDistInf;
        const long long lo = item_lo(it);
        const int cnt = (int)it.w;
        op.begin_lane(it.z);
        for (int b = 0; b < p.te; b += 4)  // warp-uniform trip count (visit4 is warp-collective)
            op.visit4(it.z, du, p.g.adj + lo + b, cnt - b, 1);
        op.end_lane(it.z, has && !op.skip(du));
    }
    op.finish();
}

// ---- local stretches -------------------------------------------------------------------------
// A relaxation round of few items is one chain of dependent accesses plus a grid barrier, about
// 8 us however small it is.  A local stretch replaces a run of such rounds: every CTA takes a share
// of the round's items into a queue in shared memory and relaxes on from there for up to `kStretch`
// steps, pushing what it improves into the next step's queue, with one block barrier a step and
// no grid barrier.  Four lanes share an item of at most four entries, and the chain of a step is
// two accesses long: the entry beside the vertex's own state, then the offer beside the
// neighbour's row descriptor (which the next step needs if the offer wins).  What still waits at
// the end, rows above kLocalDeg and what does not fit the queue go to the grid's lists, claimed as
// in a round; distances at or above the near-far threshold go to the far list.  The order of
// relaxations differs from the rounds', the fixpoint does not: every strict improvement is pushed
// by the thread that made it, and an item is dropped only if its vertex has been improved again
// since (then that thread has pushed it).  The queue's pushes mark chg_tag, not push_tag, whose
// tag says "claimed for the next list".
//
// Bound: the latency of the two accesses, 1,000 and 1,200-1,400 cycles of a step's 3,300 (clock
// counts on grids of 1.6M and 16.8M vertices), then the push, the block barrier and, per stretch,
// a grid barrier with a new deal of the work.  So the push is kept short (one shared atomic a
// warp, no ranking bits unless a row takes two places), the fields of the parameter block are
// held in registers and the pushed row is prefetched: 27.0 -> 23.7 ms on the 4096^2 grid below; with
// the shorter usual push, barrier and advances 22.8 ms.
// A queue per CTA, not per warp: with one per warp a step was shorter, but a queue that grew past
// 32 entries took several steps a hop and the others waited for it (21,476 steps and 46 ms
// against 12,310 and 36 ms).  A CTA whose queue passes one and a half passes ends everybody's
// stretch (rstop), so the work is dealt out again when it is needed and not every 16 or 64 steps
// (27.1 ms against 28.6 and 36).  Measured against rounds throughout: a 4096^2 grid with 100k
// changes 95.0 -> 22.8 ms a batch, a 1021 x 1543 grid with 9k changes 23.3 -> 5.7 ms, the tree of
// a 2048^2 grid 38.0 -> 9.1 ms, ER graphs of 10k and 300k vertices 0.157 -> 0.130 and 0.264 ->
// 0.211 ms of k_update.
// A round is a local stretch when it holds thread items only, no more than one pass of every CTA:
// above that the grid is busy and the rounds' throughput counts.  (Half or a quarter of a pass:
// the same on grids and ER graphs within 2 %, 64 pooled ER graphs 0.405 -> 0.410 and 0.424 ms.)
__device__ __forceinline__ bool local_step(const UpdParams& p, unsigned nt, unsigned nc) {
    return nc == 0 && nt <= gridDim.x * (blockDim.x >> 2) && p.te <= kLocalTe && p.group_ctas == 0;
}

__device__ __forceinline__ void keep_stats(const LocalStats& ls);

// Whether relaxations may run in local stretches and far lists go whole into them.  Not under a round
// cap of the caller's that may bind: the steps of a stretch add up to more than the depth, by how
// much depends on which CTA was faster, so a cap that is enough for the rounds would stop a batch
// that converges, and not in every run.  Such a call takes the rounds it counts, each at its own
// barrier.
__device__ __forceinline__ bool stretches(const UpdParams& p) { return p.capped == 0; }

// A stretch of at most four steps that leaves work does not pay where the next ones are like it: rows above
// kLocalDeg leave it at every hop, and a barrier with a new deal of the work costs 7 us where a round
// of few items on CTA 0 alone costs 3 (small_step).  From the fourth such stretch in a row on, the
// next lists run as rounds, 8 at first and twice as many after each further one, up to 256.  A spine of
// 3,000 vertices with 60 leaves each, computation and batches 25.7 and 2.7 ms in stretches throughout,
// 12.6 and 1.9 ms so, 12.4 and 2.0 ms in rounds; 400 layers of 50 vertices with 20 edges to the next
// 4.2, 3.4 and 2.9 ms.  Not earlier: RMAT and ER graphs, a few short stretches deep in all, took up to
// 10 % more (RMAT-18 with 1,000 changes 121 -> 134 us).  Two or 8 steps for four: 4.2 and 3.4 ms on the
// layers, the rest the same.  The state is in shared memory: the loops' registers are full.
__shared__ unsigned s_rest[2];  // lists (levels) before number [0] run as rounds; [1] how many the last time

__device__ __forceinline__ void no_rest() {  // read behind the next block barrier
    if (threadIdx.x < 2) s_rest[threadIdx.x] = 0;
}

__device__ __forceinline__ void after_stretch(unsigned used, bool left, unsigned next) {
    if (threadIdx.x == 0) {
        unsigned span = 0;
        if (used <= kShortStretch && left) {
            span = s_rest[1] ? min(2 * s_rest[1], kMaxRest) : 1u;
            if (span >= kMinRest) s_rest[0] = next + span;
        }
        s_rest[1] = span;
    }
    __syncthreads();
}

// A graph of whose rows nearly all fit a stretch's queue.  On others (RMAT: one row in ten above
// kLocalDeg) a stretch soon leaves through the lists, and the phases before it are better kept
// apart: seeds, pulls and the first rounds of an RMAT-20 insertion batch 0.071 ms apart, 0.083 in one.
__device__ __forceinline__ bool short_rows(const UpdParams& p) {
    return 64ull * __ldcg(&p.g.ctl->long_rows) <= (unsigned long long)p.g.n;
}

// Pushes c (want), whose row rd has entries, into a CTA's queue: ceil(deg / 4) items, ranked in the
// warp by the bits of (items - 1).  False for rows above kLocalDeg and where the queue is full (its
// last places stay empty).  Warp-collective.
__device__ __forceinline__ bool queue_push(bool want, unsigned c, unsigned nd, const RowDesc& rd, uint4* queue,
                                           unsigned* count) {
    const unsigned lane = lane_id(), lt = (1u << lane) - 1u;
    const bool shrt = want && rd.deg <= kLocalDeg;
    const unsigned extra = shrt ? ((unsigned)rd.deg - 1u) >> 2 : 0u;
    const unsigned m = __ballot_sync(kFull, shrt), mx = __ballot_sync(kFull, extra != 0);
    if (m == 0) return false;
    unsigned rank = __popc(m & lt), total = __popc(m);
    if (mx) {
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const unsigned mb = __ballot_sync(kFull, extra & (1u << b));
            rank += __popc(mb & lt) << b;
            total += __popc(mb) << b;
        }
    }
    unsigned at = 0;
    if (lane == 0) at = atomicAdd(count, total);
    at = __shfl_sync(kFull, at, 0) + rank;
    const bool in = shrt && at + extra < kQueue;
    if (in) {
        if (extra == 0) {
            queue[at] = make_uint4(c, nd, (unsigned)rd.start,
                                   (unsigned)((unsigned long long)rd.start >> 32) | ((unsigned)rd.deg << 8));
        } else {
            long long lo = rd.start;
            for (unsigned k = 0; k <= extra; k++, lo += 4)
                queue[at + k] = make_uint4(c, nd, (unsigned)lo, (unsigned)((unsigned long long)lo >> 32) |
                                                                    (min(4u, (unsigned)rd.deg - 4 * k) << 8));
        }
    } else if (shrt) {
        for (unsigned k = at; k < kQueue; k++) queue[k] = make_uint4(0, 0, 0, 0);
    }
    return in;
}

struct Stretch {
    const UpdParams* p;
    // fields of *p in registers: a function of its own reads them through memory
    unsigned long long* state;
    const int2* adj;
    const RowDesc* rows;
    unsigned* chg;
    unsigned epoch, r, rbase, adv;  // list r is read, list r + 1 written; far list adv & 1
    unsigned long long T;
    int spilled;    // entries of the warp's spill staging
    unsigned nfar;  // ... and of its far staging
    LocalStats ls;

    __device__ __forceinline__ unsigned tag() const { return rbase + r + 2u; }
    __device__ __forceinline__ PushBuf buf() const {
        return PushBuf{&s_pbuf[0][0] + (threadIdx.x >> 5) * kSpill, spilled};
    }
    __device__ __forceinline__ Out out() const {
        const DevGraph& g = p->g;
        const bool odd = (r & 1) != 0;
        const unsigned slot = (r + 1) % 3;
        return Out{odd ? g.rt0 : g.rt1, &g.ctl->rcT[slot], g.tcap, odd ? g.rc0 : g.rc1, &g.ctl->rcC[slot], g.ccap};
    }
    __device__ __forceinline__ unsigned* lfar() const {
        return reinterpret_cast<unsigned*>(&s_pbuf[0][0] + kFarAt) + (threadIdx.x >> 5) * kFarBuf;
    }

    __device__ __forceinline__ void spill(bool pred, unsigned v, const RowDesc& rd) {
        PushBuf pb = buf();
        if (spilled + 32 > kSpill) pb.expand_all(*p, out(), ls);
        pb.add(pred, v, rd);
        spilled = pb.count;
        ls.frontier += pred ? 1 : 0;
    }

    __device__ __forceinline__ void flush_far() {
        if (nfar == 0) return;
        __syncwarp();
        const Far far{(adv & 1) ? p->g.far1 : p->g.far0, &p->g.ctl->fc[adv % 3], p->g.far_tag, rbase + adv,
                      (unsigned)p->g.n, T};
        for (unsigned b = 0; b < nfar; b += 32)
            far_push(*p, far, b + lane_id() < nfar, lfar()[(b + lane_id()) & (kFarBuf - 1)]);
        nfar = 0;
        __syncwarp();
    }

    __device__ __forceinline__ void stage_far(bool later, unsigned v) {
        const unsigned fmask = __ballot_sync(kFull, later);
        if (fmask == 0) return;
        if (nfar + __popc(fmask) > kFarBuf) flush_far();
        if (later) lfar()[nfar + __popc(fmask & ((1u << lane_id()) - 1u))] = v;
        nfar += __popc(fmask);
    }

    // v (pred) into the queue, or to the lists
    __device__ __forceinline__ void begin(bool pred, unsigned v, unsigned d, uint4* queue, unsigned* count) {
        const RowDesc rd = row_if(*p, pred, v);
        pred = pred && rd.deg > 0;
        const bool in = queue_push(pred, v, d, rd, queue, count);
        ls.frontier += in ? 1 : 0;
        if (__any_sync(kFull, pred && !in)) {
            const bool won = pred && !in && atomicExch(&p->g.push_tag[v], tag()) != tag();
            spill(won, v, rd);
        }
    }

    __device__ __forceinline__ void begin_seed(unsigned i, unsigned ns, uint4* queue, unsigned* count) {
        const unsigned v = i < ns ? __ldcg(&p->seedq[i]) : 0u;
        begin(i < ns, v, 0u, queue, count);  // distance 0: whatever the state says
    }

    // vertex i of the other far list, at the threshold before (below it: settled since)
    __device__ __forceinline__ void begin_far(unsigned i, unsigned n, unsigned long long before, uint4* queue,
                                              unsigned* count) {
        const unsigned v = i < n ? __ldcg(&((adv & 1) ? p->g.far0 : p->g.far1)[i]) : 0u;
        const unsigned long long d = i < n ? __ldcg(&state[v]) >> 32 : 0ull;
        stage_far(i < n && d >= before && d >= T, v);
        begin(i < n && d >= before && d < T, v, (unsigned)d, queue, count);
    }

    // item i of a cut-off vertex: its best live neighbour, as PullOp
    __device__ __forceinline__ void begin_pull(unsigned i, unsigned nt, unsigned nd, uint4* queue, unsigned* count) {
        const bool has = i < nt + nd;
        const Item it = has ? __ldcg(i < nt ? &p->g.it[i] : &p->g.rt1[i - nt]) : make_uint4(0u, 0u, 0u, 0u);
        const int2* a = adj + item_lo(it);
        int2 e[4];
#pragma unroll
        for (int q = 0; q < 4; q++) e[q] = q < (int)it.w ? ld_stream(a + q) : make_int2(0, -1);
        unsigned long long s[4];
#pragma unroll
        for (int q = 0; q < 4; q++) s[q] = e[q].y >= 0 ? __ldcg(&state[e[q].x]) : kInfState;
        ls.edges_pull += min(4u, it.w);
        unsigned long long best = kInfState;
        bool push = false;
        unsigned d = 0;  // of a push through a zero weight: whatever the state says
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (e[q].y < 0 || s[q] == kInfState) continue;
            const unsigned long long nd = (s[q] >> 32) + (unsigned)e[q].y;
            if (nd >= kDistInf) ls.dist_ovf++;
            else if (e[q].y > 0) best = min(best, (nd << 32) | (unsigned)e[q].x);
            else if (relax_to(p->g, epoch, it.z, nd, (unsigned)e[q].x, 0, __ldcg(&state[it.z]), ls)) push = true;
        }
        if (best != kInfState) {
            const unsigned long long old = atomicMin(&state[it.z], best);
            if ((old >> 32) > (best >> 32)) {
                if (!push) d = (unsigned)(best >> 32);
                push = true;
                ls.updates++;
            }
        }
        if (__any_sync(kFull, push)) begin(push, it.z, d, queue, count);
    }

    // One item's entry per lane (warp-collective): x = the item, (vertex, distance, slots, count)
    // of at most 4 entries (count 0: none), next = the next step's queue with its counter.
    __device__ __forceinline__ void visit(const uint4& x, uint4* next, unsigned* next_cnt) {
        const unsigned lane = lane_id(), sub = lane & 3u;
        const bool act = sub < (x.w >> 8);
        const long long j = (long long)((unsigned long long)(x.w & 0xFFu) << 32 | x.z) + sub;
        const int2 e = act ? ld_stream(&adj[j]) : make_int2(0, -1);
        const unsigned long long du = act ? __ldcg(&state[x.x]) >> 32 : kDistInf;
        const bool live = du < kDistInf && du >= x.y;  // below: improved since, and pushed again then
        const unsigned c = (unsigned)e.x;
        const unsigned long long nd = du + (unsigned)e.y;
        RowDesc rd{0, 0, 0};
        bool push = false;
        if (live && e.y >= 0) {
            rd = rows[c];
            if (e.y == 0) {
                push = relax_to(p->g, epoch, c, nd, x.x, 0, __ldcg(&state[c]), ls);
            } else if (nd < kDistInf) {
                const unsigned long long cand = (nd << 32) | x.x;
                const unsigned long long old = atomicMin(&state[c], cand);
                push = (old >> 32) > nd;
                if (push) ls.updates++;
                else if (old > cand && chg) chg[c] = epoch;
            } else if (__ldcg(&state[c]) == kInfState) {
                ls.dist_ovf++;
            }
        }
        ls.edges_relax += live ? 1 : 0;
        const unsigned pushed = __ballot_sync(kFull, push);
        if (pushed == 0) return;
        // The usual push, near vertices with one item each that all fit: one vote and one ranking
        // word (grids of 1.6M and 16.8M vertices 5.78 -> 5.57 and 22.1 -> 21.3 ms of rounds).
        if (__all_sync(kFull, !push || (nd < T && (unsigned)rd.deg - 1u < 4u))) {
            const unsigned total = __popc(pushed);
            unsigned at = 0;
            if (lane == 0) at = atomicAdd(next_cnt, total);
            at = __shfl_sync(kFull, at, 0);
            if (at + total <= kQueue) {
                if (push) {
                    next[at + __popc(pushed & ((1u << lane) - 1u))] =
                        make_uint4(c, (unsigned)nd, (unsigned)rd.start,
                                   (unsigned)((unsigned long long)rd.start >> 32) | ((unsigned)rd.deg << 8));
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(adj + rd.start));
                    if (chg) chg[c] = epoch;
                    ls.frontier++;
                }
                return;
            }
            if (at + lane < kQueue) next[at + lane] = make_uint4(0, 0, 0, 0);  // the last places stay empty
        }
        const bool later = push && nd >= T;
        const bool near = push && !later && rd.deg > 0;
        const bool in = queue_push(near, c, (unsigned)nd, rd, next, next_cnt);
        if (in) {
            // the next step reads the row: on its way while this one ends
            asm volatile("prefetch.global.L2 [%0];" ::"l"(adj + rd.start));
            if (chg) chg[c] = epoch;
            ls.frontier++;
        }
        if (__any_sync(kFull, near && !in)) {
            const bool won = near && !in && atomicExch(&p->g.push_tag[c], tag()) != tag();
            spill(won, c, rd);
        }
        stage_far(later, c);
    }
};

// CTA-collective; reads list r (nt thread items) and appends to list r + 1.  A stretch of kind kPulls
// begins at the seeds of k_append (ns of them) and the cut-off vertices' items (nt in `it`, nd in
// rt1) instead: each of these pulls the vertex's best live neighbour, and what improves is relaxed
// on at once, while other CTAs still pull.  That is exact: a neighbour that a pull reads too early
// is pushed by whoever lowers it.  One of kind kWaiting begins at the ns vertices of the other far
// list, `before` the threshold till now: what lies below T is near, the rest waits on.  A function
// of its own, with its own counters, so that the rounds keep their registers.
enum Begin { kList, kPulls, kWaiting };
__device__ __noinline__ void relax_local(const UpdParams& p, unsigned r, unsigned nt, unsigned rbase, unsigned adv,
                                         unsigned long long T, Begin kind, unsigned nd, unsigned ns,
                                         unsigned long long before) {
    Ctl* const ctl = p.g.ctl;
    const bool odd = (r & 1) != 0;
    const unsigned slot = (r + 1) % 3;
    const Item* const tl = odd ? p.g.rt1 : p.g.rt0;
    const unsigned lane = lane_id();
    const unsigned per = blockDim.x >> 2, parts = (unsigned)p.te >> 2;
    // near-far frontiers are steady, and a CTA that falls behind holds up the others; a plain one grows
    // and shrinks again (3 passes against 1.5: 300,000 vertices 0.049 -> 0.043 ms, the grid 27 -> 32 ms)
    const unsigned limit = T == ~0ull ? 3 * per : per + per / 2;
    uint4 *now = &s_pbuf[0][0] + kQueueAt, *next = now + kQueue;
    Stretch st{&p, p.g.state, p.g.adj, p.g.rows, p.g.chg_tag, p.epoch, r, rbase, adv, T, 0, 0, LocalStats{}};
    unsigned* const stopped = &ctl->rstop[slot];
    // items blockIdx, blockIdx + gridDim, ... of the list, at most `per` of them
    const unsigned mine = kind == kList && nt > blockIdx.x ? (nt - blockIdx.x - 1) / gridDim.x + 1 : 0u;
    for (unsigned i = threadIdx.x; i < mine; i += blockDim.x) {
        const Item it = __ldcg(&tl[blockIdx.x + (unsigned long long)i * gridDim.x]);
        for (unsigned k = 0; k < parts; k++) {
            const long long lo = item_lo(it) + 4 * k;
            const unsigned cnt = it.w > 4 * k ? min(4u, it.w - 4 * k) : 0u;
            now[i * parts + k] =
                make_uint4(it.z, 0u, (unsigned)lo, (unsigned)((unsigned long long)lo >> 32) | (cnt << 8));
        }
    }
    if (threadIdx.x == 0) {
        s_qcnt[0] = mine * parts;
        s_qcnt[1] = 0;
        s_stop[0] = s_stop[1] = 0;
    }
    __syncthreads();
    if (kind == kWaiting) {
        for (unsigned i0 = (threadIdx.x & ~31u); blockIdx.x + i0 * gridDim.x < ns; i0 += blockDim.x)
            st.begin_far(blockIdx.x + (i0 + lane) * gridDim.x, ns, before, now, &s_qcnt[0]);
        __syncthreads();
    }
    if (kind == kPulls) {
        for (unsigned i0 = (threadIdx.x & ~31u); blockIdx.x + i0 * gridDim.x < ns; i0 += blockDim.x)
            st.begin_seed(blockIdx.x + (i0 + lane) * gridDim.x, ns, now, &s_qcnt[0]);
        for (unsigned i0 = (threadIdx.x & ~31u); blockIdx.x + i0 * gridDim.x < nt + nd; i0 += blockDim.x)
            st.begin_pull(blockIdx.x + (i0 + lane) * gridDim.x, nt, nd, now, &s_qcnt[0]);
        __syncthreads();
    }
    unsigned k = 0, n, cur = 0, nxt = 1, old = 2;  // the steps' counters rotate
    for (;; k++) {
        n = min(s_qcnt[cur], kQueue);
        if (n == 0 || k >= kStretch || s_stop[k & 1]) break;
        if (n > limit && k > 0) {  // too much for this CTA: everybody's work is dealt out again
            if (threadIdx.x == 0) atomicExch(stopped, 1u);
            break;
        }
        if (threadIdx.x == 0) s_qcnt[old] = 0;  // read by every thread before the last barrier
        const unsigned stop = threadIdx.x == blockDim.x - 1 ? __ldcg(stopped) : 0u;
        for (unsigned b = (threadIdx.x & ~31u) >> 2; b < n; b += per) {  // warp-uniform
            const unsigned i = b + (lane >> 2);
            st.visit(i < n ? now[i] : make_uint4(0, 0, 0, 0), next, &s_qcnt[nxt]);
        }
        if (stop) s_stop[(k + 1) & 1] = 1;  // a slow warp may still read this step's word
        const unsigned t = old;
        old = cur;
        cur = nxt;
        nxt = t;
        uint4* const q = now;
        now = next;
        next = q;
        __syncthreads();
    }
    st.flush_far();
    for (unsigned b = threadIdx.x & ~31u; b < n; b += blockDim.x) {
        const uint4 x = b + lane < n ? now[b + lane] : make_uint4(0, 0, 0, 0);
        const bool has = (x.w >> 8) != 0;
        RowDesc rd;
        const bool won = claim_with_row(p, has, x.x, st.tag(), rd);  // the whole row, once
        st.spill(won, x.x, rd);
    }
    st.buf().flush_cta(p, st.out(), st.ls);
    if (threadIdx.x == 0 && k) atomicMax(&ctl->rsteps[slot], k);
    keep_stats(st.ls);
}

// The same for levels of the subtree walk: list entries [lo, lo + nt) of `it` are this stretch's first
// items, hiT and hiC where the grid's lists end.  The items of the vertices that the stretch cuts
// off and walks on from go to `done` (rt1, free during the walk), for their pull; those it does
// not reach go behind hiT, as the next level's.  With `roots` > 0 the stretch begins at the roots
// instead (at most half a pass of every CTA), without a list of them.  Three accesses a step: the entry, the neighbour's
// parent word, and for a child its tag beside its row descriptor.  A step is a level.
// Against levels on the grid and on CTA 0, the walk of ER graphs of 10k, 300k vertices and of 64
// pooled ones: 0.088 -> 0.073, 0.140 -> 0.106 and 0.166 -> 0.145 ms; a 1021 x 1543 grid's 48 levels and
// pointer jumping 0.52 -> 0.31 ms; RMAT, whose levels hold hub rows, unchanged.
__device__ __noinline__ void walk_local(const UpdParams& p, unsigned li, unsigned lo, unsigned nt, unsigned hiT,
                                        unsigned hiC, unsigned steps_max, unsigned roots) {
    Ctl* const ctl = p.g.ctl;
    const DevGraph& g = p.g;
    unsigned long long* const state = g.state;
    const unsigned slot = (li + 1) % 3, lane = lane_id(), per = blockDim.x >> 2, limit = per + per / 2;
    const unsigned warp0 = (threadIdx.x & ~31u) >> 2;
    const Out out{g.it + hiT, &ctl->ltT[slot], g.tcap - hiT, g.ic + hiC, &ctl->ltC[slot], g.ccap - hiC};
    PushBuf pb{&s_pbuf[0][0] + (threadIdx.x >> 5) * kSpill, 0};
    uint4 *now = &s_pbuf[0][0] + kQueueAt, *next = now + kQueue, *prev = next + kQueue;
    unsigned* const stopped = &ctl->lstop[slot];
    LocalStats ls;
    const unsigned mine = nt > blockIdx.x ? (nt - blockIdx.x - 1) / gridDim.x + 1 : 0u;
    for (unsigned i = threadIdx.x; i < mine; i += blockDim.x) {
        const Item it = __ldcg(&g.it[lo + blockIdx.x + (unsigned long long)i * gridDim.x]);
        now[i] = make_uint4(it.z, 0u, it.x, it.y | (it.w << 8));
    }
    if (threadIdx.x == 0) {
        s_qcnt[0] = mine;
        s_qcnt[1] = 0;
        s_stop[0] = s_stop[1] = 0;
    }
    __syncthreads();
    if (roots) {
        const unsigned share = roots > blockIdx.x ? (roots - blockIdx.x - 1) / gridDim.x + 1 : 0u;
        for (unsigned b = threadIdx.x & ~31u; b < share; b += blockDim.x) {
            const bool has = b + lane < share;
            const unsigned v = has ? __ldcg(&g.invq[blockIdx.x + (b + lane) * gridDim.x]) : 0u;
            const RowDesc rd = row_if(p, has, v);
            const bool in = queue_push(has && rd.deg > 0, v, 0u, rd, now, &s_qcnt[0]);
            if (pb.count + 32 > kSpill) pb.expand_all(p, out, ls);
            pb.add(has && !in, v, rd);
        }
        __syncthreads();
    }
    // writes n items of a queue to a list from place `at` on (thread items of at most 4 entries)
    auto keep = [&](const uint4* q, unsigned n, Item* list, long long at, long long cap) {
        if (at + n > cap) {
            if (threadIdx.x == 0) set_status(ctl, -4 /* work list capacity: internal error */);
            return;
        }
        for (unsigned i = threadIdx.x; i < n; i += blockDim.x) {
            const uint4 x = q[i];
            list[at + i] = make_uint4(x.z, x.w & 0xFFu, x.x, x.w >> 8);
        }
    };
    unsigned k = 0, n, cur = 0, nxt = 1, old = 2, nprev = 0;
    for (;; k++) {
        n = min(s_qcnt[cur], kQueue);
        if (nprev) keep(prev, nprev, g.rt1, s_done[(k + 1) & 1], g.tcap);  // the last step's items
        nprev = 0;
        if (n == 0 || k >= steps_max || s_stop[k & 1]) break;
        if (n > limit && k > 0) {
            if (threadIdx.x == 0) atomicExch(stopped, 1u);
            break;
        }
        unsigned at = 0;
        if (threadIdx.x == 0) {
            s_qcnt[old] = 0;
            if (k > 0 || roots) at = atomicAdd(&ctl->walk_done, n);  // a list's items are in `it` already
        }
        const unsigned stop = threadIdx.x == blockDim.x - 1 ? __ldcg(stopped) : 0u;
        for (unsigned b = warp0; b < n; b += per) {  // warp-uniform
            const unsigned i = b + (lane >> 2), sub = lane & 3u;
            const uint4 x = i < n ? now[i] : make_uint4(0, 0, 0, 0);
            const bool act = sub < (x.w >> 8);
            const long long j = (long long)((unsigned long long)(x.w & 0xFFu) << 32 | x.z) + sub;
            const int2 e = act ? ld_stream(&g.adj[j]) : make_int2(0, -1);
            const unsigned c = (unsigned)e.x;
            const bool child = e.y >= 0 && (unsigned)__ldcg(&state[c]) == x.x;
            RowDesc rd{0, 0, 0};
            bool mark = false;
            if (child) {  // cut off even when already tagged, as in MarkOp
                rd = g.rows[c];
                state[c] = kInfState;
                mark = atomicExch(&g.inv_tag[c], p.epoch) != p.epoch;
            }
            ls.edges_inv += act ? 1 : 0;
            if (!__any_sync(kFull, mark)) continue;
            ls.marked += mark ? 1 : 0;
            const bool in = queue_push(mark && rd.deg > 0, c, 0u, rd, next, &s_qcnt[nxt]);
            if (in) asm volatile("prefetch.global.L2 [%0];" ::"l"(g.adj + rd.start));
            if (__any_sync(kFull, mark && !in)) {
                if (pb.count + 32 > kSpill) pb.expand_all(p, out, ls);
                pb.add(mark && !in, c, rd);
            }
        }
        if (stop) s_stop[(k + 1) & 1] = 1;  // a slow warp may still read this step's word
        if (threadIdx.x == 0) s_done[k & 1] = at;
        if (k > 0 || roots) nprev = n;
        unsigned t = old;
        old = cur;
        cur = nxt;
        nxt = t;
        uint4* const q = prev;
        prev = now;
        now = next;
        next = q;
        __syncthreads();
    }
    if (n) {  // not walked: the next level's
        if (threadIdx.x == 0) s_done[k & 1] = atomicAdd(out.tcnt, n);
        __syncthreads();
        keep(now, n, g.it, (long long)hiT + s_done[k & 1], g.tcap);
    }
    pb.flush_cta(p, out, ls);
    if (threadIdx.x == 0 && k) atomicMax(&ctl->lsteps[slot], k);
    keep_stats(ls);
}

__device__ void block_max(unsigned long long* dst, unsigned long long x) {
    __shared__ unsigned long long s_max;
    __syncthreads();
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    x = warp_max_u64(x);
    if (lane_id() == 0 && x) atomicMax(&s_max, x);
    __syncthreads();
    if (threadIdx.x == 0 && s_max) atomicMax(dst, s_max);
}

// Adds a phase's counters to the CTA's (whole warps).
__device__ __forceinline__ void keep_stats(const LocalStats& ls) {
    const unsigned v[8] = {ls.edges_relax, ls.edges_inv, ls.updates, ls.dist_ovf,
                           ls.frontier, ls.items, ls.marked, ls.edges_pull};
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const unsigned x = __reduce_add_sync(kFull, v[q]);
        if (lane_id() == 0 && x) atomicAdd(&s_lstat[q], (unsigned long long)x);
    }
}

// Near-far: the near frontier is empty, nfar vertices wait in the far list.  The next threshold is
// one width on; with `least`, it is the least waiting distance plus the width, which takes a pass
// and a barrier.  0 when nothing waits or the kernel must stop.
__device__ __forceinline__ unsigned long long next_threshold(const UpdParams& p, unsigned nfar, unsigned adv,
                                                          unsigned long long T, bool least) {
    const unsigned long long width = s_width;
    if (!least) return T + width;
    Ctl* const ctl = p.g.ctl;
    const DevGraph& g = p.g;
    const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
    const unsigned* const fl = (adv & 1) ? g.far1 : g.far0;
    unsigned long long mn = ~0ull;
    for (unsigned i = gtid; i < nfar; i += nthreads) {
        const unsigned long long d = __ldcg(&g.state[__ldcg(&fl[i])]) >> 32;
        if (d >= T && d < mn) mn = d;  // below T: settled by an earlier near phase
    }
    block_max(&ctl->fmin[adv & 1], ~mn);  // max of ~d = min of d; 0 = nothing waits
    if (!grid_sync(ctl)) return 0;
    const unsigned long long fm = __ldcg(&ctl->fmin[adv & 1]);
    return fm ? ~fm + width : 0;
}

// A far list of at most one pass of the grid goes straight into a local stretch: every CTA takes its
// share of it into its queue and relaxes on, without a near list, a barrier and a deal of that in
// between.  Measured on batches of a 1021 x 1543 and a 4096^2 grid and the tree of a 2048^2 grid:
// 5.52 -> 5.35, 21.3 -> 20.9 and 9.30 -> 9.10 ms of rounds.  (A quarter of the pass: 21.05 on the
// 4096^2 grid; four passes: the same.)  Longer lists are split by the grid.
__device__ __forceinline__ bool local_advance(const UpdParams& p, unsigned nfar) {
    return nfar <= gridDim.x * blockDim.x && p.te <= kLocalTe && p.group_ctas == 0;
}

// Splits the far list, whose generation is rbase + adv, at the next threshold tn into list r (near)
// and the other far list.  False when the kernel must stop; the sizes of list r are left in s_near.
__device__ __forceinline__ bool far_advance(const UpdParams& p, unsigned r, unsigned nfar, unsigned rbase, unsigned adv,
                                         unsigned long long T, unsigned long long tn) {
    const int cf = (int)(adv & 1u);  // the list that is split; generations and lists follow the advances
    const unsigned fgen = rbase + adv;
    Ctl* const ctl = p.g.ctl;
    const DevGraph& g = p.g;
    const unsigned lane = lane_id(), gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
    const unsigned* fl = cf ? g.far1 : g.far0;
    const Far nxt{cf ? g.far0 : g.far1, &ctl->fc[(adv + 1) % 3], g.far_tag, fgen + 1, (unsigned)g.n, tn};
    const Out near{(r & 1) ? g.rt1 : g.rt0, &ctl->rcT[r % 3], g.tcap, (r & 1) ? g.rc1 : g.rc0, &ctl->rcC[r % 3], g.ccap};
    const unsigned tagr = rbase + r + 1u;  // the tag of list r
    PushBuf pb{s_pbuf[threadIdx.x >> 5], 0};
    LocalStats ls;
    for (unsigned base = gtid - lane; base < nfar; base += nthreads) {
        const unsigned i = base + lane;
        const unsigned v = i < nfar ? __ldcg(&fl[i]) : 0u;
        const unsigned long long d = i < nfar ? __ldcg(&g.state[v]) >> 32 : 0ull;
        const bool live = i < nfar && d >= T;
        far_push(p, nxt, live && d >= tn, v);
        RowDesc rd;
        const bool doit = claim_with_row(p, live && d < tn, v, tagr, rd);
        ls.frontier += doit ? 1 : 0;
        pb.add(doit, v, rd);
        pb.flush(p, near, ls);
    }
    pb.flush_cta(p, near, ls);
    keep_stats(ls);
    unsigned nt, nc;
    if (!grid_sync(ctl, &ctl->rcT[r % 3], &ctl->rcC[r % 3], nt, nc)) return false;
    if (threadIdx.x == 0) {
        s_near[0] = nt;
        s_near[1] = nc;
    }
    return true;
}

// The counters of a round's lists and of a stretch, before either writes them.
__device__ __forceinline__ void clear_slots(Ctl* ctl, unsigned slot) {
    ctl->rcT[slot] = 0;
    ctl->rcC[slot] = 0;
    ctl->rsteps[slot] = 0;
    ctl->rstop[slot] = 0;
}

// The near frontier is empty and nfar vertices wait: moves the threshold on (to s_threshold).  kSplit:
// list r is the near one, its sizes in s_near; kWhole: a stretch is to take the far list.  A
// function of its own, so that the rounds keep their registers.
enum Advance { kStop, kSplit, kWhole };
__device__ __noinline__ Advance advance(const UpdParams& p, unsigned r, unsigned nfar, unsigned rbase, unsigned adv,
                                        unsigned long long T, bool least, bool local, unsigned hops) {
    Ctl* const ctl = p.g.ctl;
    if (p.delta == 0) {
        // A plain computation that goes on near-far has a width by the mean weight alone, which says little
        // where weights differ widely: a path of 8,000 edges of 250,000 beside 3M of 1 and 2 took an
        // advance of 12 us for each edge, 98 ms against 25 ms of plain rounds.  An advance that has bought
        // few hops doubles the width: 12.5 ms.  (Grids buy about 80 hops with each and keep theirs.)
        if (threadIdx.x == 0) {
            if (adv > 0 && hops - s_advanced < kFewHops && s_width < kDistInf) s_width *= 2;
            s_advanced = hops;
        }
        __syncthreads();
    }
    const unsigned long long tn = next_threshold(p, nfar, adv, T, least);
    if (tn == 0) return kStop;
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // read by every CTA before the last barrier, written after the next
        ctl->fc[(adv + 2) % 3] = 0;
        ctl->fmin[(adv + 1) & 1] = 0;
    }
    const bool whole = local && local_advance(p, nfar);
    if (!whole && !far_advance(p, r, nfar, rbase, adv, T, tn)) return kStop;
    if (threadIdx.x == 0) s_threshold = tn;
    __syncthreads();
    return whole ? kWhole : kSplit;
}

// ---- A. cut-off subtrees (grid-wide) -----------------------------------------------------------
// Returns
// the sizes of the lists it and ic, every cut-off vertex's items (~0: the kernel must stop).
__device__ __forceinline__ unsigned long long walk(const UpdParams& p) {
    Ctl* const ctl = p.g.ctl;
    const DevGraph& g = p.g;
    const unsigned lane = lane_id(), gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
    const bool leader = gtid == 0;
    uint4* pbuf = s_pbuf[threadIdx.x >> 5];
    LocalStats ls;
    // Level L processes items [lo, hi) of the lists it/ic and appends the items of the
    // vertices it cuts off after hi through counters of its own, lt*[(li+1)%3] with li the lists
    // so far, so every CTA derives the same bounds while faster CTAs already append.  Small
    // levels are walked in CTA queues, several to a list.
    const unsigned nroots = __ldcg(&ctl->inv_count);  // written by k_delete
    unsigned loT = 0, loC = 0, hiT = 0, hiC = 0;
    int level = 0;
    unsigned li = 0;
    if (nroots == 0) return 0;
    if (leader) ls.marked += nroots;
    if (p.te == 4 && p.group_ctas == 0 && nroots <= gridDim.x * min(4u, blockDim.x >> 3) && short_rows(p)) {
        unsigned used;
        walk_local(p, li, 0, 0, 0, 0, (unsigned)p.bfs_levels, nroots);
        if (!grid_sync(ctl, &ctl->ltT[1], &ctl->ltC[1], hiT, hiC, &ctl->lsteps[1], used)) return ~0ull;
        level = (int)used;
        li = 1;
    } else {
        const Out lvl0{g.it, &ctl->ltT[0], g.tcap, g.ic, &ctl->ltC[0], g.ccap};
        PushBuf pb{pbuf, 0};
        for (unsigned base = gtid - lane; base < nroots; base += nthreads) {
            const unsigned i = base + lane;
            const unsigned v = i < nroots ? __ldcg(&g.invq[i]) : 0u;
            pb.add(i < nroots, v, row_if(p, i < nroots, v));
            pb.flush(p, lvl0, ls);
        }
        pb.flush_cta(p, lvl0, ls);
        if (!grid_sync(ctl, &ctl->ltT[0], &ctl->ltC[0], hiT, hiC)) return ~0ull;
    }
    bool need_pj = false;
    for (;;) {
        if (loT >= hiT && loC >= hiC) break;
        if (level >= p.bfs_levels) {
            need_pj = true;
            break;
        }
        if (p.te == 4 && (unsigned)level >= s_rest[0] && local_step(p, hiT - loT, hiC - loC)) {
            if (leader) {
                ctl->ltT[(li + 2) % 3] = 0;
                ctl->ltC[(li + 2) % 3] = 0;
                ctl->lsteps[(li + 2) % 3] = 0;
                ctl->lstop[(li + 2) % 3] = 0;
            }
            walk_local(p, li, loT, hiT - loT, hiT, hiC, (unsigned)(p.bfs_levels - level), 0);
            unsigned addT, addC, used;
            if (!grid_sync(ctl, &ctl->ltT[(li + 1) % 3], &ctl->ltC[(li + 1) % 3], addT, addC, &ctl->lsteps[(li + 1) % 3], used))
                return ~0ull;
            loT = hiT;
            loC = hiC;
            hiT += addT;
            hiC += addC;
            level += (int)used;
            after_stretch(used, addT != 0 || addC != 0, (unsigned)level);
            li++;
            continue;
        }
        if (small_step(hiT - loT, hiC - loC, p.solo_waves)) {
            // small levels: CTA 0 walks on alone while they stay small; the others wait
            if (blockIdx.x == 0) {
                if (threadIdx.x < 6) s_solo_cnt[threadIdx.x / 2][threadIdx.x % 2] = 0;
                __syncthreads();
                for (int steps = 0; steps < kSoloSteps; steps++) {
                    if ((loT >= hiT && loC >= hiC) || level >= p.bfs_levels || !small_step(hiT - loT, hiC - loC, p.solo_waves))
                        break;
                    unsigned* cnt = s_solo_cnt[(level + 1) % 3];
                    if (threadIdx.x == 0) {
                        s_solo_cnt[(level + 2) % 3][0] = 0;
                        s_solo_cnt[(level + 2) % 3][1] = 0;
                    }
                    MarkOp op{&p, Out{g.it + hiT, &cnt[0], g.tcap - hiT, g.ic + hiC, &cnt[1], g.ccap - hiC},
                              PushBuf{pbuf, 0}, &ls};
                    run_items(op, p, g.it + loT, hiT - loT, g.ic + loC, hiC - loC, 0, 1);
                    __syncthreads();
                    loT = hiT;
                    loC = hiC;
                    hiT += cnt[0];
                    hiC += cnt[1];
                    level++;
                    __syncthreads();  // every thread has read the counters before the next reset
                }
                if (threadIdx.x == 0) {
                    ctl->solo[0] = ((unsigned long long)hiT << 32) | loT;
                    ctl->solo[1] = ((unsigned long long)hiC << 32) | loC;
                    ctl->solo[2] = (unsigned long long)level;
                    ctl->ltT[(li + 1) % 3] = 0;  // the grid's next level appends here
                    ctl->ltC[(li + 1) % 3] = 0;
                }
            }
            if (!grid_sync(ctl)) return ~0ull;
            const unsigned long long a = __ldcg(&ctl->solo[0]), b = __ldcg(&ctl->solo[1]);
            loT = (unsigned)a;
            hiT = (unsigned)(a >> 32);
            loC = (unsigned)b;
            hiC = (unsigned)(b >> 32);
            level = (int)__ldcg(&ctl->solo[2]);
            continue;
        }
        if (leader) {
            ctl->ltT[(li + 2) % 3] = 0;
            ctl->ltC[(li + 2) % 3] = 0;
            ctl->lsteps[(li + 2) % 3] = 0;
            ctl->lstop[(li + 2) % 3] = 0;
        }
        MarkOp op{&p,
                  Out{g.it + hiT, &ctl->ltT[(li + 1) % 3], g.tcap - hiT, g.ic + hiC, &ctl->ltC[(li + 1) % 3],
                      g.ccap - hiC},
                  PushBuf{pbuf, 0}, &ls};
        run_items(op, p, g.it + loT, hiT - loT, g.ic + loC, hiC - loC, blockIdx.x, gridDim.x);
        unsigned addT, addC;
        if (!grid_sync(ctl, &ctl->ltT[(li + 1) % 3], &ctl->ltC[(li + 1) % 3], addT, addC)) return ~0ull;
        loT = hiT;
        loC = hiC;
        hiT += addT;
        hiC += addC;
        level++;
        li++;
    }
    if (leader) ctl->stat[ST_LEVELS] = (unsigned long long)level;
    if (need_pj) {
        // pointer jumping: jm[v] climbs towards the root until it meets a cut-off vertex
        // (kTagInv) or the root / an unreachable vertex (kTagOk); O(log depth) passes
        for (unsigned v = gtid; v < (unsigned)g.n; v += nthreads) {
            unsigned t;
            if (__ldcg(&g.inv_tag[v]) == p.epoch) {
                t = kTagInv;
            } else {
                const unsigned par = (unsigned)__ldcg(&g.state[v]);
                t = (par == v || par == kNone) ? kTagOk : par;  // a root, or unreachable
            }
            g.jm[v] = t;
        }
        if (!grid_sync(ctl)) return ~0ull;
        int pass = 0;
        for (;; pass++) {
            if (pass >= 64) {
                if (leader) set_status(ctl, -7 /* BAD_TREE: parent cycle */);
                grid_sync(ctl);
                return ~0ull;
            }
            if (leader) ctl->pjf[(pass + 1) % 3] = 0;
            int moving = 0;
            for (unsigned v = gtid; v < (unsigned)g.n; v += nthreads) {
                const unsigned j = __ldcg(&g.jm[v]);
                if (j < kTagInv) {
                    const unsigned jj = __ldcg(&g.jm[j]);
                    g.jm[v] = jj;
                    moving |= jj < kTagInv;
                }
            }
            moving = __syncthreads_or(moving);
            if (moving && threadIdx.x == 0) atomicOr(&ctl->pjf[pass % 3], 1u);
            if (!grid_sync(ctl)) return ~0ull;
            if (__ldcg(&ctl->pjf[pass % 3]) == 0) break;
        }
        if (leader) ctl->stat[ST_PJ] = (unsigned long long)(pass + 1);
        const Out pjo{g.it + hiT, &ctl->pjT, g.tcap - hiT, g.ic + hiC, &ctl->pjC, g.ccap - hiC};
        PushBuf pb{pbuf, 0};
        for (unsigned base = gtid - lane; base < (unsigned)g.n; base += nthreads) {
            const unsigned v = base + lane;
            bool newinv = false;
            const bool inv = v < (unsigned)g.n && __ldcg(&g.jm[v]) == kTagInv;
            if (inv && __ldcg(&g.inv_tag[v]) != p.epoch) {
                g.inv_tag[v] = p.epoch;
                newinv = true;
            }
            // also the roots: one that an insertion re-parented may hold a distance
            // through a cut-off vertex (the pull gives it its best live value again)
            if (inv) g.state[v] = kInfState;
            ls.marked += newinv ? 1 : 0;
            pb.add(newinv, v, row_if(p, newinv, v));
            pb.flush(p, pjo, ls);
        }
        pb.flush_cta(p, pjo, ls);
        if (!grid_sync(ctl)) return ~0ull;
        hiT += __ldcg(&ctl->pjT);
        hiC += __ldcg(&ctl->pjC);
    }
    keep_stats(ls);
    return ((unsigned long long)hiC << 32) | hiT;
}

// ---- B. the seeds of k_append become work items; cut-off vertices pull their best live neighbour ----
__device__ __forceinline__ void seed_and_pull(const UpdParams& p, unsigned hiT, unsigned hiC, unsigned rbase,
                                           unsigned long long T) {
    Ctl* const ctl = p.g.ctl;
    const DevGraph& g = p.g;
    const unsigned lane = lane_id(), gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
    const unsigned tag0 = rbase + 1;
    const Out relax0{g.rt0, &ctl->rcT[0], g.tcap, g.rc0, &ctl->rcC[0], g.ccap};
    uint4* pbuf = s_pbuf[threadIdx.x >> 5];
    LocalStats ls;
    {
        const unsigned ns = __ldcg(&ctl->seed_count);
        PushBuf pb{pbuf, 0};
        for (unsigned base = gtid - lane; base < ns; base += nthreads) {
            const unsigned i = base + lane;
            const unsigned v = i < ns ? __ldcg(&p.seedq[i]) : 0u;
            pb.add(i < ns, v, row_if(p, i < ns, v));
            pb.flush(p, relax0, ls);
        }
        pb.flush_cta(p, relax0, ls);
    }
    {
        PullOp op{&p, tag0, relax0, PushBuf{pbuf, 0}, &ls, Far{g.far0, &ctl->fc[0], g.far_tag, rbase, (unsigned)g.n, T}, kInfState, false};
        run_items(op, p, g.it, hiT, g.ic, hiC, blockIdx.x, gridDim.x, g.rt1, __ldcg(&ctl->walk_done));
    }
    keep_stats(ls);
}

// The CTA's counters, one atomic each.
__device__ void flush_stats(Ctl* ctl, const LocalStats& ls) {
    keep_stats(ls);
    __syncthreads();
    const int idx[8] = {ST_EDGES_RELAX, ST_EDGES_INV, ST_UPDATES, ST_DIST_OVF, ST_FRONTIER, ST_ITEMS, ST_INV,
                        ST_EDGES_PULL};
    if (threadIdx.x < 8 && s_lstat[threadIdx.x]) atomicAdd(&ctl->stat[idx[threadIdx.x]], s_lstat[threadIdx.x]);
}

// Adds a CTA's sums of N counters to stat[idx[0]], stat[idx[1]], ..., one atomic each.
template <int N>
__device__ void block_add(Ctl* ctl, const int (&idx)[N], const unsigned long long (&x)[N]) {
    __shared__ unsigned long long s_sum[N];
    if (threadIdx.x < N) s_sum[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < N; q++) {
        const unsigned long long t = warp_sum_u64(x[q]);
        if (lane_id() == 0 && t) atomicAdd(&s_sum[q], t);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < N; q++)
        if (threadIdx.x == q && s_sum[q]) atomicAdd(&ctl->stat[idx[q]], s_sum[q]);
}

// Per-warp staging of appends to a plain u32 list.  A warp writes its region of shared memory
// and appends it to the list with one atomic when the region is nearly full; at the end the
// CTA appends what its warps still hold with one atomic (flush_cta).  The list counters are
// single words that every CTA hits, so their atomics are kept few, and no CTA-wide barrier
// is needed while the warps work.
struct WarpList {
    unsigned* buf;  // this warp's region of shared memory
    int cap;        // entries in the region
    int count;      // warp-uniform

    __device__ __forceinline__ void add(bool pred, unsigned v) {
        const unsigned mask = __ballot_sync(kFull, pred);
        if (pred) buf[count + __popc(mask & ((1u << lane_id()) - 1u))] = v;
        count += __popc(mask);
        __syncwarp();
    }

    // warp-collective: appends the region once fewer than `room` entries are free
    __device__ __forceinline__ void flush(unsigned* list, unsigned* counter, unsigned list_cap, int room, Ctl* ctl) {
        if (count + room <= cap) return;
        unsigned b = 0;
        if (lane_id() == 0) b = atomicAdd(counter, (unsigned)count);
        b = __shfl_sync(kFull, b, 0);
        if ((unsigned long long)b + (unsigned)count > list_cap) {
            if (lane_id() == 0) set_status(ctl, -4 /* list capacity: internal error */);
        } else {
            for (int j = (int)lane_id(); j < count; j += 32) list[b + j] = buf[j];
        }
        count = 0;
        __syncwarp();
    }

    // CTA-collective (every thread of the CTA)
    __device__ void flush_cta(unsigned* list, unsigned* counter, unsigned list_cap, Ctl* ctl) {
        __shared__ unsigned s_off[kMaxWarps], s_base, s_ok;
        const unsigned w = threadIdx.x >> 5, nw = blockDim.x >> 5;
        if (lane_id() == 0) s_off[w] = (unsigned)count;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned t = 0;
            for (unsigned k = 0; k < nw; k++) {
                const unsigned c = s_off[k];
                s_off[k] = t;
                t += c;
            }
            s_base = t ? atomicAdd(counter, t) : 0u;
            s_ok = (unsigned long long)s_base + t <= list_cap;
            if (!s_ok) set_status(ctl, -4 /* list capacity: internal error */);
        }
        __syncthreads();
        if (s_ok)
            for (int j = (int)lane_id(); j < count; j += 32) list[s_base + s_off[w] + j] = buf[j];
        count = 0;
        __syncthreads();
    }
};

// ---- row search and the deletion set -------------------------------------------------------

// Inserts (pair, w) into the open-addressing deletion set.  Probing depends only on the pair;
// a slot whose pair matches but whose weight is taken by another weight is skipped.
__device__ bool hash_insert(const UpdParams& p, unsigned long long pair, int w) {
    unsigned long long h = dmix64(pair) & p.hmask;
    for (unsigned long long probe = 0; probe <= p.hmask; probe++) {
        DelSlot* slot = &p.hset[h];
        const unsigned long long old = atomicCAS(&slot->pair, kHashEmpty, pair);
        if (old == kHashEmpty || old == pair) {
            const int ow = atomicCAS(&slot->w, kHashNoWeight, w);
            if (ow == kHashNoWeight || ow == w) return true;
        }
        h = (h + 1) & p.hmask;
    }
    return false;
}

__device__ bool hash_contains(const UpdParams& p, unsigned long long pair, int w) {
    unsigned long long h = dmix64(pair) & p.hmask;
    for (unsigned long long probe = 0; probe <= p.hmask; probe++) {
        const DelSlot slot = p.hset[h];
        if (slot.pair == kHashEmpty) return false;
        if (slot.pair == pair && slot.w == w) return true;
        h = (h + 1) & p.hmask;
    }
    return false;
}

// Tombstones a reverse entry, slot t.  A twin word outside the adjacency is an internal error: it is
// reported in the status word and the access is skipped.
__device__ __forceinline__ void tombstone_twin(const UpdParams& p, unsigned t) {
    if ((long long)t < p.g.cap_total) p.g.adj[t].y = -1;
    else set_status(p.g.ctl, -4 /* twin index out of range: internal error */);
}

// Tombstones one matching entry; the compare-and-swap makes the count exact when a batch
// deletes one line twice.  Returns the entries tombstoned (2 with the twin).
__device__ __forceinline__ unsigned tombstone_at(const UpdParams& p, long long j, int w, bool with_twin) {
    if (w < 0) return 0;  // a negative weight matches no live entry (tombstones hold -1)
    const unsigned t = with_twin ? p.g.twin[j] : 0u;  // on its way with the compare-and-swap
    if (atomicCAS(&p.g.adj[j].y, w, -1) != w) return 0;
    if (with_twin) tombstone_twin(p, t);
    return with_twin ? 2u : 1u;
}

// Tombstones every live entry (col, w) in the neighbour-sorted prefix [lo, sl) of a row: binary search
// down to four entries, then four loads in flight at a time.  With the twin index the reverse
// entries are tombstoned too.  Returns the number of entries examined; `dead` counts the entries
// tombstoned.
__device__ __forceinline__ unsigned tombstone_prefix(const UpdParams& p, long long lo, long long sl, int col, int w,
                                                     bool with_twin, unsigned& dead) {
    const int2* adj = p.g.adj;
    for (long long hi = sl; hi - lo > 4;) {  // the first entry of col or above lies in [lo, hi]
        const long long mid = lo + ((hi - lo) >> 1);
        if (adj[mid].x < col) lo = mid + 1;
        else hi = mid;
    }
    unsigned probed = 1;
    for (bool more = lo < sl; more; lo += 4) {
        int2 e[4];
#pragma unroll
        for (int k = 0; k < 4; k++) e[k] = lo + k < sl ? adj[lo + k] : make_int2(0x7FFFFFFF, -1);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (e[k].x != col) continue;
            probed++;
            if (e[k].y == w) dead += tombstone_at(p, lo + k, w, with_twin);
        }
        more = e[3].x <= col && lo + 4 < sl;
    }
    return probed;
}

// The whole row: the sorted prefix, then the unsorted tail (the entries appended since the row was
// laid out) by this thread.
__device__ unsigned long long tombstone_row(const UpdParams& p, const RowDesc& rd, int sorted_len, int col, int w,
                                            bool with_twin, unsigned& dead) {
    const int2* adj = p.g.adj;
    const long long sl = rd.start + sorted_len, end = rd.start + rd.deg;
    unsigned long long probed = tombstone_prefix(p, rd.start, sl, col, w, with_twin, dead);
    probed += (unsigned long long)(end > sl ? end - sl : 0);
    for (long long j = sl; j < end; j += 4) {  // four loads in flight
        int2 e[4];
#pragma unroll
        for (int k = 0; k < 4; k++) e[k] = j + k < end ? adj[j + k] : make_int2(-1, -1);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (e[k].x == col && e[k].y == w) dead += tombstone_at(p, j + k, w, with_twin);
    }
    return probed;
}

// Unsorted tails of rows.  Under sustained insertion and deletion they grow until the row is compacted
// or the adjacency is repacked, on hub rows to thousands of entries.  A deletion's lane scans up
// to kShortTail of them itself (four loads in flight); the warp scans its 32 deletions' longer ones
// together, their entries side by side, 128 in flight; a tail above kLongTail goes to the batch's
// list in chunks, which k_append's warps scan (its appends lie behind every tail).  Bound: the
// latency of the loads, so many are kept in flight, and the longest tail, so it is cut up.  RMAT
// scale 22, a stream of 10^6 changes with 2.5 * 10^7 tail entries a batch: k_delete 0.36 -> 0.27 ms
// against the tails of a warp one after the other, 32 entries at a time (0.14 without tails).
// kShortTail 8 or 32: the same there, 64 pooled ER graphs 0.101 and 0.085 ms of the front kernels
// against 0.085 at 16; 6 CTAs per SM (40 registers) against 4: 0.30 -> 0.27 ms.
constexpr int kShortTail = 16;
constexpr int kLongTail = 512;
constexpr unsigned kTailChunk = 1024;
constexpr unsigned kNoPair = 0x80000000u;  // in a tail's weight: leave the twins alone (weights are below 2^31)

// One tail per lane (len 0: none), scanned by the warp; w carries kNoPair.  Returns the entries
// this lane tombstoned.
__device__ __forceinline__ unsigned scan_tails(const UpdParams& p, long long lo, unsigned len, int col, unsigned w) {
    const unsigned lane = lane_id();
    const unsigned incl = warp_incl_scan(len), total = __shfl_sync(kFull, incl, 31);
    unsigned dead = 0;
    for (unsigned b = 0; b < total; b += 128) {
        long long j[4];
        int2 e[4];
        unsigned own[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const unsigned pos = b + 32 * k + lane;
            unsigned o = 0;  // the first lane whose tails end behind pos
#pragma unroll
            for (int s = 16; s > 0; s >>= 1)
                if (__shfl_sync(kFull, incl, o + s - 1) <= pos) o += s;
            own[k] = o & 31u;
            j[k] = __shfl_sync(kFull, lo, own[k]) + (pos - (__shfl_sync(kFull, incl, own[k]) - __shfl_sync(kFull, len, own[k])));
            e[k] = pos < total ? p.g.adj[j[k]] : make_int2(-1, -1);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int c = __shfl_sync(kFull, col, own[k]);
            const unsigned x = __shfl_sync(kFull, w, own[k]);
            if (e[k].x == c && (unsigned)e[k].y == (x & ~kNoPair))
                dead += tombstone_at(p, j[k], (int)(x & ~kNoPair), (x & kNoPair) == 0);
        }
    }
    return dead;
}

// Lists a long tail in chunks; false when the list is full (its last places stay empty chunks).
__device__ __forceinline__ bool list_tail(const UpdParams& p, long long lo, unsigned len, int col, unsigned w) {
    const unsigned n = (len + kTailChunk - 1) / kTailChunk;
    const unsigned at = atomicAdd(&p.g.ctl->tail_count, n);
    const bool fits = at < p.tail_cap && n <= p.tail_cap - at;
    for (unsigned k = 0; k < n && at < p.tail_cap && k < p.tail_cap - at; k++, lo += kTailChunk)
        p.tail_list[at + k] = make_uint4((unsigned)lo, (unsigned)((unsigned long long)lo >> 32) |
                                         (fits ? min(kTailChunk, len - k * kTailChunk) << 8 : 0u), (unsigned)col, w);
    return fits;
}

}  // namespace

// ---- kernels -----------------------------------------------------------------------------

// Clears the control block and the batch's deletion set and validates the records, which it brings
// from pinned host memory if they lie there (a copy and two memset nodes before it cost a batch of 17
// changes 8 us; for 16 MB the link is the bound either way).  A refusal is told under the batch's epoch (line 0 of the control block), so
// that no word needs clearing before any of this.
__global__ void k_prepare(UpdParams p) {
    Ctl* ctl = p.g.ctl;
    if (blockIdx.x == 0) {  // line 1 on
        unsigned* w = reinterpret_cast<unsigned*>(&ctl->status);
        const unsigned words = (unsigned)((sizeof(Ctl) - offsetof(Ctl, status)) / sizeof(unsigned));
        for (unsigned i = threadIdx.x; i < words; i += blockDim.x) w[i] = 0;
    }
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    static_assert(sizeof(DelSlot) == sizeof(uint4), "a deletion-set slot is one store");
    uint4* const set = reinterpret_cast<uint4*>(p.hset);
    for (unsigned long long i = (unsigned long long)tid; i <= p.hmask; i += (unsigned long long)nthreads)
        set[i] = make_uint4(kNone, kNone, kNone, kNone);
    unsigned refused = 0;
    for (long long i = tid; i < p.k; i += nthreads) {
        const int4 c = p.chg_src ? __ldcs(&p.chg_src[i]) : p.chg[i];
        if (p.chg_src) p.chg[i] = c;
        if (c.w == 1 || c.w == 0) {
            if (c.x < 0 || c.x >= p.g.n || c.y < 0 || c.y >= p.g.n) refused = kRefusedVertex;
            else if (c.w == 1 && c.z < 0) refused = max(refused, kRefusedWeight);
        }
    }
    if (refused) atomicMax(&ctl->refused, ((unsigned long long)p.epoch << 32) | refused);
}

// Deletions: cut off the child end of a deleted tree edge, tombstone every matching entry,
// record the deletion in the batch's deletion set.
// kTails: rows may hold unsorted tails (entries appended since the last layout); without, every tail
// is scanned by its deletion's lane (the host picks this form after a layout, a repack or a
// compaction, until a batch appends again: the long-tail path alone costs the kernel a few
// percent).
template <bool kTails>
__global__ void __launch_bounds__(256, 5) k_delete(UpdParams p) {
    Ctl* ctl = p.g.ctl;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const long long base0 = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane;
    auto load = [&](long long i) { return i < p.k ? p.chg[i] : make_int4(0, 0, 0, -1); };
    int4 next = load(base0 + lane);
    const unsigned long long refused = __ldcg(&ctl->refused);  // by k_prepare: same for every thread
    if (refused >> 32 == p.epoch) {
        if (blockIdx.x == 0 && threadIdx.x == 0)
            set_status(ctl, (unsigned)refused == kRefusedVertex ? -3 /* BAD_VERTEX */ : -10 /* BAD_WEIGHT */);
        return;
    }
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    unsigned long long probed = 0;
    unsigned roots = 0, dead = 0;
    WarpList roots_list{s_wlist[warp], kListRegion, 0};
    for (long long base = base0; base < p.k; base += nthreads) {
        const long long i = base + lane;
        const int4 c = next;
        next = load(i + nthreads);
        unsigned cutv = 0, was = p.epoch;
        long long tlo = 0;  // this lane's tail for the warp to scan
        unsigned tlen = 0, tw = 0;
        int tcol = 0;
        if (c.w == 0) {
            const unsigned a = (unsigned)c.x, b = (unsigned)c.y;
            // All accesses that wait for the record alone go out together, the next record is on its way
            // meanwhile, and the cut mark and the deletion set's answer are looked at behind the search:
            // fewer accesses one after the other.  RMAT-22 with 500,000 deletions 0.270 -> 0.253 ms (with 5
            // CTAs an SM; 6 take 0.266, 4 take 0.266), small batches 2 us less.
            const unsigned pb = (unsigned)__ldcg(&p.g.state[b]), pa = (unsigned)__ldcg(&p.g.state[a]);
            const RowDesc ra = p.g.rows[a], rb = p.g.rows[b];
            const unsigned long long pair = dpair_key(a, b);
            DelSlot* const slot = &p.hset[dmix64(pair) & p.hmask];
            const unsigned long long had = c.z >= 0 ? atomicCAS(&slot->pair, kHashEmpty, pair) : 0ull;
            // gpuFunctions_undir.cuh:189-198: the child end is checked as b first, then as a.
            // A self-loop never cuts: its only parent relation is a root's (parent == itself),
            // and roots are never cut off.
            if (a != b && (pb == a || pa == b)) {
                cutv = pb == a ? b : a;
                was = atomicExch(&p.g.inv_tag[cutv], p.epoch);
            }
            const bool mine = c.z >= 0 && (had == kHashEmpty || had == pair);
            const int weight = mine ? atomicCAS(&slot->w, kHashNoWeight, c.z) : kHashNoWeight;
            if (p.g.twin) {
                // search the shorter row; each match's reverse entry is found through twin[].  Of rows
                // of equal degree the lower vertex's, whichever end the record names first: records of
                // one line then meet at one entry, whose compare-and-swap one of them wins (at an end
                // each, both won, and the line's two entries were counted twice)
                const bool use_a = ra.deg < rb.deg || (ra.deg == rb.deg && a <= b);
                const RowDesc& rs = use_a ? ra : rb;
                const int sl = p.g.sorted_len[use_a ? a : b];
                const int col = (int)(use_a ? b : a);
                // a self-loop's two entries lie in the one row: the search meets both, each is
                // counted by its own compare-and-swap (by the other's twin store as well, a loop
                // deleted by two records of a batch was counted twice)
                const bool both = a != b;
                if (!kTails || rs.deg - sl <= kShortTail) {
                    probed += tombstone_row(p, rs, sl, col, c.z, both, dead);
                } else {
                    tlo = rs.start + sl;
                    probed += tombstone_prefix(p, rs.start, tlo, col, c.z, both, dead);
                    tcol = col;
                    tw = (unsigned)c.z | (both ? 0u : kNoPair);
                    if (c.z >= 0) tlen = (unsigned)(rs.deg - sl);  // a negative weight matches nothing
                    probed += tlen;
                    if (tlen > (unsigned)kLongTail && list_tail(p, tlo, tlen, tcol, tw)) tlen = 0;
                }
            } else {
                probed += tombstone_row(p, ra, p.g.sorted_len[a], (int)b, c.z, false, dead);
                probed += tombstone_row(p, rb, p.g.sorted_len[b], (int)a, c.z, false, dead);
            }
            // not in the first place: search from there on
            if (c.z >= 0 && !(mine && (weight == kHashNoWeight || weight == c.z)) && !hash_insert(p, pair, c.z))
                set_status(ctl, -4 /* deletion set full */);
        }
        const bool cut = was != p.epoch;
        if (cut) p.g.state[cutv] = kInfState;
        if constexpr (kTails) dead += scan_tails(p, tlo, tlen, tcol, tw);
        roots_list.add(cut, cutv);
        roots += cut ? 1 : 0;
        roots_list.flush(p.g.invq, &ctl->inv_count, (unsigned)p.g.n, 32, ctl);
    }
    roots_list.flush_cta(p.g.invq, &ctl->inv_count, (unsigned)p.g.n, ctl);
    block_add<3>(ctl, {ST_ROOTS, ST_DEL_PROBED, ST_TOMBS}, {roots, probed, dead});
}

// Insertions that no deletion of the batch removes go into row slack, both directions.  An end that
// does not fit is listed with its row, and k_update grows the row first.  Every surviving insertion then relaxes both of its ends
// (replaces insertEdge, gpuFunctions_undir.cuh:217-251); an improved end is claimed for the
// first frontier and listed in seedq (k_update splits it into work items once every row has
// its final degree) or, in near-far mode, put in the far list.  Doing this before the
// subtree walk is exact: k_delete has already cut off the roots (their distance is
// infinite, so nothing relaxes from them), an end relaxed from a vertex that the walk later
// cuts off takes that vertex as its parent and is cut off with it, and every other relaxed
// distance is the length of a live path.
// 5 CTAs per SM (48 registers) against 4: 0.146 -> 0.141 ms on RMAT scale 22 with 10^6 changes.
__global__ void __launch_bounds__(256, 5) k_append(UpdParams p) {
    Ctl* ctl = p.g.ctl;
    DevGraph& g = p.g;
    const unsigned lane = lane_id();
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    unsigned long long n_del = 0, n_ign = 0;
    if (__ldcg(&ctl->status) < 0) {  // refused (same for every thread): only counted
        unsigned long long n_ins = 0;
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.k; i += nthreads) {
            const int op = p.chg[i].w;
            n_ins += op == 1 ? 1 : 0;
            n_del += op == 0 ? 1 : 0;
            n_ign += op != 0 && op != 1 ? 1 : 0;
        }
        block_add<3>(ctl, {ST_INS, ST_DEL, ST_IGN}, {n_ins, n_del, n_ign});
        return;
    }
    const unsigned rbase = __ldcg(&ctl->round_base);
    const unsigned tag0 = rbase + 1;
    // near-far: a batch starts with threshold 0, so every seed waits in the far list
    const bool nf = p.delta != 0 && g.far0 != nullptr && g.far1 != nullptr && g.far_tag != nullptr;
    const unsigned long long T = nf ? 0ull : ~0ull;
    // seeds are staged per warp (half of the warp's staging region each for near and far)
    unsigned* region = s_wlist[threadIdx.x >> 5];
    WarpList near_list{region, kListRegion / 2, 0}, far_list{region + kListRegion / 2, kListRegion / 2, 0};
    const unsigned seed_cap = (unsigned)min(2 * p.k, (long long)g.n);  // distinct claimed ends
    LocalStats ls;
    unsigned long long killed = 0, ovf = 0, live_ins = 0;
    const unsigned tails = min(__ldcg(&ctl->tail_count), p.tail_cap);
    if (tails) {  // the long tails that k_delete listed, a chunk per warp at a time
        unsigned dead = 0;
        for (unsigned c = (unsigned)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5); c < tails;
             c += (unsigned)(nthreads >> 5)) {
            const uint4 x = __ldcg(&p.tail_list[c]);
            const long long lo = (long long)((unsigned long long)(x.y & 0xFFu) << 32 | x.x);
            const unsigned len = x.y >> 8;
            for (unsigned b = 0; b < len; b += 256) {
                int2 e[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const unsigned o = b + 32 * k + lane;
                    e[k] = o < len ? ld_stream(&g.adj[lo + o]) : make_int2(-1, -1);
                }
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (e[k].x == (int)x.z && (unsigned)e[k].y == (x.w & ~kNoPair))
                        dead += tombstone_at(p, lo + b + 32 * k + lane, e[k].y, (x.w & kNoPair) == 0);
            }
        }
        block_add<1>(ctl, {ST_TOMBS}, {dead});
    }
    for (long long base = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane; base < p.k; base += nthreads) {
        const long long i = base + lane;
        const int4 c = i < p.k ? p.chg[i] : make_int4(0, 0, 0, -1);
        n_del += i < p.k && c.w == 0 ? 1 : 0;
        n_ign += i < p.k && c.w != 0 && c.w != 1 ? 1 : 0;
        // Independent accesses of one record go out together (states, rows and the deletion-set
        // probe; both degree bumps; both seed relaxations; both claims).
        int alive = 0;
        unsigned long long sa = kInfState, sb = kInfState;
        RowDesc rx{0, 0, 0}, ry{0, 0, 0};
        int pos0 = 0, pos1 = 0;
        bool ov0 = false, ov1 = false;
        if (c.w == 1) {
            sa = __ldcg(&g.state[c.x]);
            sb = __ldcg(&g.state[c.y]);
            rx = g.rows[c.x], ry = g.rows[c.y];  // start and cap are fixed in this kernel
            if (hash_contains(p, dpair_key((unsigned)c.x, (unsigned)c.y), c.z)) {
                killed++;
            } else {
                alive = 1;
                live_ins++;
                pos0 = atomicAdd(&g.rows[c.x].deg, 1);
                pos1 = atomicAdd(&g.rows[c.y].deg, 1);
                ov0 = pos0 >= rx.cap;
                ov1 = pos1 >= ry.cap;
                if (!ov0) g.adj[rx.start + pos0] = make_int2(c.y, c.z);
                if (!ov1) g.adj[ry.start + pos1] = make_int2(c.x, c.z);
                if (g.twin) {  // an overflowed end is placed (and paired) by the row growth
                    if (!ov0) g.twin[rx.start + pos0] = ov1 ? kNoTwin : (unsigned)(ry.start + pos1);
                    if (!ov1) g.twin[ry.start + pos1] = ov0 ? kNoTwin : (unsigned)(rx.start + pos0);
                }
                ovf += (ov0 ? 1 : 0) + (ov1 ? 1 : 0);
            }
        }
        list_overflow(p, i, c, rx, ry, pos0, pos1, ov0, ov1, rx.start + pos0, ry.start + pos1);
        // seed: relax both ends through the new edge
        bool pa = false, pbv = false;
        const unsigned long long ndb = (sa >> 32) + (unsigned)c.z, nda = (sb >> 32) + (unsigned)c.z;
        if (alive) {
            if (c.z > 0) {
                relax_both(g, p.epoch, (unsigned)c.x, (unsigned)c.y, ndb, nda, sa, sb, pa, pbv, ls);
            } else {  // zero weight: strict improvements only (compare-and-swap)
                if ((sa >> 32) != kDistInf) pbv = relax_to(g, p.epoch, (unsigned)c.y, ndb, (unsigned)c.x, c.z, sb, ls);
                if ((sb >> 32) != kDistInf)
                    pa = relax_to(g, p.epoch, (unsigned)c.x, nda, (unsigned)c.y, c.z, __ldcg(&g.state[c.x]), ls);
            }
            ls.edges_relax += 2;
        }
        // claim: far-list tag for an end at or above the threshold, frontier tag otherwise
        const bool lb = pbv && ndb >= T, la = pa && nda >= T;
        unsigned* tb = lb ? g.far_tag + c.y : g.push_tag + c.y;
        unsigned* ta = la ? g.far_tag + c.x : g.push_tag + c.x;
        const unsigned vb = lb ? rbase : tag0, va = la ? rbase : tag0;
        const unsigned ob = pbv ? atomicExch(tb, vb) : vb;
        const unsigned oa = pa ? atomicExch(ta, va) : va;
        const bool fb = lb && ob != vb, db = pbv && !lb && ob != vb;
        const bool fa = la && oa != va, da = pa && !la && oa != va;
        ls.frontier += (db ? 1 : 0) + (da ? 1 : 0) + (fb ? 1 : 0) + (fa ? 1 : 0);
        near_list.add(db, (unsigned)c.y);  // claimed: one entry per vertex
        near_list.add(da, (unsigned)c.x);
        far_list.add(fb, (unsigned)c.y);  // far-tagged: one entry per vertex
        far_list.add(fa, (unsigned)c.x);
        near_list.flush(p.seedq, &ctl->seed_count, seed_cap, 64, ctl);
        far_list.flush(g.far0, &ctl->fc[0], (unsigned)g.n, 64, ctl);
    }
    near_list.flush_cta(p.seedq, &ctl->seed_count, seed_cap, ctl);
    far_list.flush_cta(g.far0, &ctl->fc[0], (unsigned)g.n, ctl);
    // the seeds' counters are kept apart from k_update's
    block_add<9>(ctl, {ST_SEED_UPD, ST_SEED_FRONT, ST_DIST_OVF, ST_OVF, ST_LIVE_INS, ST_KILLED, ST_INS, ST_DEL, ST_IGN},
                 {ls.updates, ls.frontier, ls.dist_ovf, ovf, live_ins, killed, live_ins + killed, n_del, n_ign});
}

// grid-wide; true when the kernel may go on
__device__ __forceinline__ bool grow_rows(const UpdParams& p) { return __ldcg(&p.g.ctl->ovf_count) == 0 || grow(p); }

// The last phase of a growth once more, for a batch whose update kernel gave up at a grid barrier
// while that phase may have been running.
__global__ void k_grow_finish(UpdParams p) {
    const unsigned long long list = p.g.ctl->grow_list;
    grow_finish(p, GrowTeam{blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x}, (unsigned)list,
                (unsigned)(list >> 32), (unsigned)p.g.ctl->ovf_count);
}

// Whether a distance does not fit below 2^32-1: a vertex has none at the fixpoint although an entry
// joins a reachable one to it.  Run only after offers that did not fit have been counted: such an
// offer alone says nothing, a shorter path may come behind it, and which comes first depends on how
// far the CTAs' queues are (in rounds it was the path of fewer hops).
__global__ void k_dist_check(DevGraph g) {
    const unsigned lane = lane_id();
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    bool over = false;
    for (long long v = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < g.n; v += warps) {
        if (g.state[v] == kInfState) continue;
        const RowDesc rd = g.rows[v];
        for (int j = (int)lane; j < rd.deg; j += 32) {
            const int2 e = g.adj[rd.start + j];
            over |= e.y >= 0 && g.state[e.x] == kInfState;
        }
    }
    if (__any_sync(kFull, over) && lane == 0) g.ctl->dist_over = 1;
}

template <bool kAgg>
__device__ void update_body(const UpdParams& p);

// 3 CTAs of 256 threads per SM: 80 registers a thread (2 CTAs: the tree of RMAT-22 1.354 -> 1.749 ms;
// 4: 1.430 ms, a grid batch 6.1 -> 7.3 ms).  Every walk level and
// relaxation round waits on its slowest CTA's chain of dependent accesses, so shorter chains
// and fewer CTAs at each barrier beat more resident warps here (4 CTAs per SM with 64
// registers and spills was slower on every workload but the throughput-bound 256-graph batch).
// kAgg: warp-aggregated distance offers (opts.warp_agg), compiled as its own kernel so that
// the default kernel keeps its register allocation.
template <bool kAgg>
__global__ void __launch_bounds__(256, 3) k_update(const __grid_constant__ UpdParams p) {
    if (threadIdx.x < 8) s_lstat[threadIdx.x] = 0;
    no_rest();
    if (threadIdx.x == 0) {
        s_nbar = 0;
        s_width = p.delta ? p.delta : p.late_delta;
        s_advanced = 0;
        s_gen = ld_acquire(&p.g.ctl->bar_gen);
        s_ggen = ld_acquire(&p.g.ctl->grp_gen);
        const unsigned lim = __ldcg(&p.g.ctl->spin_limit);
        s_spin_limit = lim ? lim : kSpinLimit;
    }
    __syncthreads();
    update_body<kAgg>(p);
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(&p.g.ctl->diag[3], s_nbar);
        atomicMax(&p.g.ctl->diag[4], 0xFFFFFFFFu - s_nbar);
    }
}

template <bool kAgg>
__device__ void update_body(const UpdParams& p) {
    Ctl* ctl = p.g.ctl;
    const DevGraph& g = p.g;
    __shared__ int s_skip;
    if (threadIdx.x == 0) s_skip = __ldcg(&ctl->status) != 0;  // set before launch: same for every CTA
    __syncthreads();
    if (s_skip) return;
    const unsigned stall_us = __ldcg(&ctl->stall_us);
    if (stall_us && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        // test hook (failure detection): arrive late at the first barrier so that the others
        // run out of polls; a bounded wait (at most 2^21 sleeps of 1 us).  One launch only: the
        // hook clears itself, so a recomputation after the failed batch runs normally.
        const unsigned long long t0 = globaltimer();
        for (unsigned i = 0; i < (1u << 21) && globaltimer() - t0 < 1000ull * stall_us; i++) __nanosleep(1000);
        ctl->stall_us = 0;
    }
    const unsigned lane = lane_id();
    const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned nthreads = gridDim.x * blockDim.x;
    const bool leader = gtid == 0;
    uint4* pbuf = s_pbuf[threadIdx.x >> 5];
    LocalStats ls;
    if (!grow_rows(p)) return;
    if (leader) ctl->ts[0] = globaltimer();

    unsigned rbase = __ldcg(&ctl->round_base);
    if (rbase > 0xF0000000u) {  // push and far tags would wrap: clear them
        for (unsigned v = gtid; v < (unsigned)g.n; v += nthreads) {
            g.push_tag[v] = 0;
            if (g.far_tag) g.far_tag[v] = 0;
        }
        if (!grid_sync(ctl)) return;
        rbase = 1;
    }
    const unsigned tag0 = rbase + 1;
    const Out relax0{g.rt0, &ctl->rcT[0], g.tcap, g.rc0, &ctl->rcC[0], g.ccap};
    // Near-far state (identical in every thread).  A batch update starts with T = 0, so every
    // seed waits in the far list and the first advance picks the threshold; a computation
    // from scratch starts with the sources (distance 0) near and T = delta.  Far generations
    // of this call are rbase, rbase + 1, ... (at most one per round, so below the next
    // call's round base).
    bool nf = p.delta != 0 && g.far0 != nullptr && g.far1 != nullptr && g.far_tag != nullptr;
    unsigned long long T = nf ? (p.mode == 1 ? p.delta : 0ull) : ~0ull;
    unsigned adv = 0;     // advances: far list adv & 1 takes this near phase's far pushes, generation rbase + adv
    bool sparse = false;  // an advance by one width has found nothing
    auto far_now = [&]() {
        return Far{(adv & 1) ? g.far1 : g.far0, &ctl->fc[adv % 3], g.far_tag, rbase + adv, (unsigned)g.n, T};
    };

    unsigned nT = 0, nC = 0;  // the sizes of the next relaxation round's lists
    // r counts the lists (a round or a local stretch each), hops the rounds and the steps of
    // the stretches, the most of any CTA: at least the depth of the dependent relaxations.  The cap
    // is on r.  A list relaxes every vertex that waits in it, so after r of them all shortest paths
    // of r edges are found, as after r rounds, and in a plain computation r stays below n + 2.  A
    // near-far phase settles a vertex at least for each of its lists: below 2n + 16 in all.
    unsigned r = 0, hops = 0;
    if (p.mode == 1) {
        PushBuf pb{pbuf, 0};
        for (unsigned base = gtid - lane; base < (unsigned)p.nsrc; base += nthreads) {
            const unsigned i = base + lane;
            const unsigned v = i < (unsigned)p.nsrc ? (unsigned)p.srcs[i] : 0u;
            if (i < (unsigned)p.nsrc) g.push_tag[v] = tag0;
            pb.add(i < (unsigned)p.nsrc, v, row_if(p, i < (unsigned)p.nsrc, v));
            pb.flush(p, relax0, ls);
            ls.frontier += i < (unsigned)p.nsrc ? 1 : 0;
        }
        pb.flush_cta(p, relax0, ls);
        if (!grid_sync(ctl, &ctl->rcT[0], &ctl->rcC[0], nT, nC)) return;
    } else {
        unsigned hiT, hiC;
        const unsigned long long ends = walk(p);
        if (ends == ~0ull) return;
        hiT = (unsigned)ends;
        hiC = (unsigned)(ends >> 32);
        if (leader) ctl->ts[1] = globaltimer();

        const unsigned ns = __ldcg(&ctl->seed_count), nd = __ldcg(&ctl->walk_done);
        if (!kAgg && !nf && p.te == 4 && stretches(p) && local_step(p, ns + hiT + nd, hiC) && short_rows(p)) {
            // few enough for one stretch: its list is number 2 (rt0; rt1 holds items of the walk)
            if (leader) ctl->ts[2] = ctl->ts[1];
            relax_local(p, 1, hiT, rbase, 0, T, kPulls, nd, ns, 0);
            if (!grid_sync(ctl, &ctl->rcT[2], &ctl->rcC[2], nT, nC, &ctl->rsteps[2], hops)) return;
            r = 2;
        } else {
            seed_and_pull(p, hiT, hiC, rbase, T);
            if (!grid_sync(ctl, &ctl->rcT[0], &ctl->rcC[0], nT, nC)) return;
            if (leader) ctl->ts[2] = globaltimer();
        }
    }
    if (leader && p.mode == 1) ctl->ts[2] = globaltimer();

    // ---- C. relaxation rounds ---------------------------------------------------------------
    no_rest();  // ... of the walk: behind a barrier as well
    __syncthreads();
    for (;; r++) {
        // nT, nC: the sizes of round r's lists (read at the barrier before)
        if (!nf && p.late_delta != 0 && hops >= p.late_after) {
            // A plain computation has turned out deep: what it pushes from here on waits, and the
            // first advance picks a threshold.  (Switching after 256, 512, 1024, 2048 rounds, the first
            // tree of a 2048^2 grid: 9.2, 9.2, 11.7, 27.6 ms; never: 61 ms.)
            nf = true;
            T = 0;
        }
        Begin kind = kList;
        const bool local = !kAgg && stretches(p) && r >= s_rest[0];
        bool least = true;
        unsigned nfar = 0;
        unsigned long long before = 0;
        if (nT == 0 && nC == 0) {
            if (!nf) break;
            // near frontier empty: advance the threshold past the least waiting distance
            nfar = __ldcg(&ctl->fc[adv % 3]);
            if (nfar == 0) break;
            least = T == 0 || sparse || !stretches(p);
            before = T;
            const Advance got = advance(p, r, nfar, rbase, adv, T, least, local, hops);
            if (got == kStop) break;
            T = s_threshold;
            adv++;
            if (got == kWhole) {
                kind = kWaiting;
            } else {
                nT = s_near[0];
                nC = s_near[1];
                if (!least && nT == 0 && nC == 0) {  // nothing within one width: look for the least
                    sparse = true;
                    r--;
                    continue;
                }
            }
        }
        if (r >= p.max_rounds) {
            if (leader) set_status(ctl, -5 /* NO_CONVERGENCE */);
            break;
        }
        if (local && (kind == kWaiting || local_step(p, nT, nC))) {
            if (leader) clear_slots(ctl, (r + 2) % 3);
            relax_local(p, r, nT, rbase, adv, T, kind, 0, nfar, before);
            unsigned t2, used;
            if (!grid_sync(ctl, &ctl->rcT[(r + 1) % 3], &ctl->rcC[(r + 1) % 3], t2, nC, &ctl->rsteps[(r + 1) % 3], used))
                break;
            nT = t2;
            hops += used;
            after_stretch(used, nT != 0 || nC != 0, r + 1);
            if (!least && used == 0 && nT == 0 && nC == 0) sparse = true;
            continue;
        }
        if (small_step(nT, nC, p.solo_waves)) {
            // small rounds: CTA 0 relaxes on alone while they stay small; the others wait.  An
            // empty frontier goes back to the grid (near-far advance or the end).
            if (blockIdx.x == 0) {
                unsigned rr = r;
                unsigned t = nT, c = nC;
                if (threadIdx.x < 6) s_solo_cnt[threadIdx.x / 2][threadIdx.x % 2] = 0;
                __syncthreads();
                for (int steps = 0; steps < kSoloSteps; steps++) {
                    if ((t == 0 && c == 0) || !small_step(t, c, p.solo_waves) || rr >= p.max_rounds) break;
                    unsigned* cnt = s_solo_cnt[(rr + 1) % 3];
                    if (threadIdx.x == 0) {
                        s_solo_cnt[(rr + 2) % 3][0] = 0;
                        s_solo_cnt[(rr + 2) % 3][1] = 0;
                    }
                    const bool odd = (rr & 1) != 0;
                    RelaxOp<kAgg> op{&p, rbase + rr + 2u,
                               Out{odd ? g.rt0 : g.rt1, &cnt[0], g.tcap, odd ? g.rc0 : g.rc1, &cnt[1], g.ccap},
                               PushBuf{pbuf, 0}, &ls, far_now(), true};
                    run_items(op, p, odd ? g.rt1 : g.rt0, t, odd ? g.rc1 : g.rc0, c, 0, 1);
                    __syncthreads();
                    rr++;
                    t = cnt[0];
                    c = cnt[1];
                    __syncthreads();  // every thread has read the counters before the next reset
                }
                if (threadIdx.x == 0) {
                    ctl->solo[3] = (unsigned long long)rr;
                    ctl->solo_n[0] = t;
                    ctl->solo_n[1] = c;
                    ctl->rcT[rr % 3] = t;  // round rr's lists (the near-far advance appends here when empty)
                    ctl->rcC[rr % 3] = c;
                    ctl->rcT[(rr + 1) % 3] = 0;  // the grid's round rr appends here
                    ctl->rcC[(rr + 1) % 3] = 0;
                    ctl->rsteps[(rr + 1) % 3] = 0;
                    ctl->rstop[(rr + 1) % 3] = 0;
                }
            }
            if (!grid_sync(ctl, &ctl->solo_n[0], &ctl->solo_n[1], nT, nC)) break;
            const unsigned rr = (unsigned)__ldcg(&ctl->solo[3]);
            hops += rr - r;
            r = rr - 1;  // the loop steps to the first round left
            continue;
        }
        if (group_step(p, nT, nC)) {
            // mid-size rounds: the group relaxes on with its own barrier while they stay
            // mid-size (at most kSoloSteps); the others wait at the next grid barrier.  Lists and
            // counters are the grid's, so the hand-over is the same as after solo rounds.
            const unsigned G = p.group_ctas;
            if (blockIdx.x < G) {
                unsigned rr = r;
                unsigned t = nT, c = nC;
                for (int steps = 0; steps < kSoloSteps; steps++) {
                    if ((t == 0 && c == 0) || !group_step(p, t, c) || rr >= p.max_rounds) break;
                    if (blockIdx.x == 0 && threadIdx.x == 0) {
                        ctl->rcT[(rr + 2) % 3] = 0;
                        ctl->rcC[(rr + 2) % 3] = 0;
                    }
                    const bool odd = (rr & 1) != 0;
                    RelaxOp<kAgg> op{&p, rbase + rr + 2u,
                                     Out{odd ? g.rt0 : g.rt1, &ctl->rcT[(rr + 1) % 3], g.tcap, odd ? g.rc0 : g.rc1,
                                         &ctl->rcC[(rr + 1) % 3], g.ccap},
                                     PushBuf{pbuf, 0}, &ls, far_now(),
                                     (unsigned long long)t + (unsigned long long)c * blockDim.x <=
                                         (unsigned long long)G * blockDim.x};
                    run_items(op, p, odd ? g.rt1 : g.rt0, t, odd ? g.rc1 : g.rc0, c, blockIdx.x, G);
                    unsigned t2, c2;
                    const bool go = group_sync(ctl, G, &ctl->rcT[(rr + 1) % 3], &ctl->rcC[(rr + 1) % 3], t2, c2);
                    rr++;
                    t = t2;
                    c = c2;
                    if (!go) break;
                }
                if (blockIdx.x == 0 && threadIdx.x == 0) {
                    ctl->solo[3] = (unsigned long long)rr;
                    ctl->solo_n[0] = t;
                    ctl->solo_n[1] = c;
                    ctl->rcT[rr % 3] = t;  // round rr's lists (the near-far advance appends here when empty)
                    ctl->rcC[rr % 3] = c;
                    ctl->rcT[(rr + 1) % 3] = 0;  // the grid's round rr appends here
                    ctl->rcC[(rr + 1) % 3] = 0;
                    ctl->rsteps[(rr + 1) % 3] = 0;
                    ctl->rstop[(rr + 1) % 3] = 0;
                }
            }
            if (!grid_sync(ctl, &ctl->solo_n[0], &ctl->solo_n[1], nT, nC)) break;
            const unsigned rr = (unsigned)__ldcg(&ctl->solo[3]);
            hops += rr - r;
            r = rr - 1;  // the loop steps to the first round left
            continue;
        }
        if (leader) clear_slots(ctl, (r + 2) % 3);
        const bool odd = (r & 1) != 0;
        RelaxOp<kAgg> op{&p, rbase + r + 2u,
                   Out{odd ? g.rt0 : g.rt1, &ctl->rcT[(r + 1) % 3], g.tcap, odd ? g.rc0 : g.rc1,
                       &ctl->rcC[(r + 1) % 3], g.ccap},
                   PushBuf{pbuf, 0}, &ls, far_now(),
                   (unsigned long long)nT + (unsigned long long)nC * blockDim.x <= (unsigned long long)nthreads};
        run_items(op, p, odd ? g.rt1 : g.rt0, nT, odd ? g.rc1 : g.rc0, nC, blockIdx.x, gridDim.x);
        if (!grid_sync(ctl, &ctl->rcT[(r + 1) % 3], &ctl->rcC[(r + 1) % 3], nT, nC)) break;
        hops++;
    }
    flush_stats(ctl, ls);
    if (leader) {
        ctl->stat[ST_ROUNDS] = (unsigned long long)hops;
        ctl->stat[ST_ADVANCES] = (unsigned long long)adv;
        ctl->round_base = rbase + r + 4u;
        ctl->ts[3] = globaltimer();
    }
}

}  // namespace dsssp

// ---- host launch wrappers (the kernels above are launched only through these) -----------
namespace dsssp {

void count_launch(int n);

// after_prepare / after_delete: events recorded between the kernels (nullptr = none)
cudaError_t launch_front(const UpdParams& p, int grid, cudaStream_t s, cudaEvent_t after_prepare,
                         cudaEvent_t after_delete) {
    if (p.k <= 0) return cudaSuccess;
    const long long need = (p.k + 255) / 256;
    const unsigned g = (unsigned)(need < grid ? need : grid);
    k_prepare<<<g, 256, 0, s>>>(p);
    if (after_prepare) cudaEventRecord(after_prepare, s);
    if (p.tails) k_delete<true><<<g, 256, 0, s>>>(p);
    else k_delete<false><<<g, 256, 0, s>>>(p);
    if (after_delete) cudaEventRecord(after_delete, s);
    k_append<<<g, 256, 0, s>>>(p);
    count_launch(3);
    return cudaGetLastError();
}

cudaError_t launch_grow_finish(const UpdParams& p, int grid, cudaStream_t s) {
    UpdParams copy = p;
    void* args[] = {&copy};
    count_launch(1);
    return cudaLaunchKernel((const void*)k_grow_finish, dim3((unsigned)grid), dim3(256), args, 0, s);
}

cudaError_t launch_dist_check(const DevGraph& g, int grid, cudaStream_t s) {
    DevGraph copy = g;
    void* args[] = {&copy};
    count_launch(1);
    return cudaLaunchKernel((const void*)k_dist_check, dim3((unsigned)grid), dim3(256), args, 0, s);
}

// Loads the kernel, so that its first launch allocates nothing.
cudaError_t load_dist_check() {
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, (const void*)k_dist_check);
}

// The batch kernels as graph-node functions: k_prepare, k_delete, k_append, k_update.
void batch_kernels(const void* fns[4]) {
    fns[0] = (const void*)k_prepare;
    fns[1] = (const void*)k_delete<true>;
    fns[2] = (const void*)k_append;
    fns[3] = (const void*)k_update<false>;
}

const void* delete_kernel(bool tails) {
    return tails ? (const void*)k_delete<true> : (const void*)k_delete<false>;
}

const void* update_kernel(bool warp_agg) {
    return warp_agg ? (const void*)k_update<true> : (const void*)k_update<false>;
}

cudaError_t update_occupancy(int block, int* blocks_per_sm) {
    int a = 0, b = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_update<false>, block, 0);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_update<true>, block, 0);
    *blocks_per_sm = a < b ? a : b;
    return e;
}

cudaError_t launch_update(const UpdParams& p, int grid, int block, cudaStream_t s) {
    UpdParams copy = p;
    void* args[] = {&copy};
    cudaError_t e = cudaLaunchCooperativeKernel(update_kernel(p.warp_agg != 0), dim3((unsigned)grid),
                                                dim3((unsigned)block), args, 0, s);
    count_launch(1);
    return e;
}

}  // namespace dsssp
