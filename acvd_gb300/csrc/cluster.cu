// Clustering kernels: the deterministic parallel form of the reference's
// boundary-swap loop (Common/vtkUniformClustering.h:833-995), the per-cluster
// statistics (ReComputeStatistics :376-403), connectivity cleaning
// (CleanClustering :406-549) and hole filling (FillHolesInClustering :552-633).
//
// Schedule: the items are coloured once (no two adjacent items share a colour).
// One step handles one colour class: `eval` proposes, for every boundary item of
// the class, the move to a neighbouring cluster with the most negative energy
// change; each proposal claims its source and destination clusters with a
// 64-bit atomicMin; `apply` commits the proposals that hold both claims.  No
// cluster takes part in two commits of one step, so every committed energy
// change is exact and the result does not depend on thread timing.
#include <algorithm>

#include "primitives.cuh"
#include "state.cuh"

namespace acvd {

// ---------------------------------------------------------------------------
// item and cluster records
// ---------------------------------------------------------------------------
// relative margin an energy decrease must exceed to be proposed (about 100 float32 ulps)
constexpr float kAcceptTol = 1e-5f;

// A load issued here, not sunk to where its value is used (behind a branch that most of
// the loads' latency would then follow).
ACVD_DEV float2 load_now(const float2* p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
ACVD_DEV float4 load_now(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
ACVD_DEV int4 load_now(const int4* p) {
    int4 v;
    asm volatile("ld.global.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
ACVD_DEV uint2 load_now(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
ACVD_DEV int load_now(const int* p) {
    int v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
ACVD_DEV double load_now(const double* p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

struct ItemRec {
    float x[3];
    float w;
    float A[6];
    float T[6];
};

template <int M>
ACVD_DEV void load_item(const DevState& st, int i, ItemRec& it) {
    const float4 a = st.xw[i];
    it.x[0] = a.x; it.x[1] = a.y; it.x[2] = a.z; it.w = a.w;
    if (M != kIso) {
        const float4 q = st.qa[i];
        const float2 r = st.qb[i];
        it.A[0] = q.x; it.A[1] = q.y; it.A[2] = q.z; it.A[3] = q.w; it.A[4] = r.x; it.A[5] = r.y;
    }
    if (M == kAniso) {
        const float4 t = st.ta[i];
        const float2 u = st.tb[i];
        it.T[0] = t.x; it.T[1] = t.y; it.T[2] = t.z; it.T[3] = t.w; it.T[4] = u.x; it.T[5] = u.y;
    }
}

struct EvalRec {
    float m[3], W;
    float d[3], P;
    float r[3];
    float A[6];
    float T[6];
    float g[3];
    float anc;      // QEM: nonzero for an anchored cluster, whose m is the anchor vertex
    int anc_item;   // ... and the anchor's item
};

// Cluster k's anchor item (QEM Cluster::AnchorItem), -1 for none
template <int M>
ACVD_DEV int anchor_of(const DevState& st, int64_t k) {
    return (M == kQEM && st.anchor) ? st.anchor[k] : -1;
}

template <int M>
ACVD_DEV void load_eval(const DevState& st, int k, EvalRec& e) {
    const float4* p = st.ev + (int64_t)k * Layout<M>::ev;
    const float4 e0 = p[0];
    e.m[0] = e0.x; e.m[1] = e0.y; e.m[2] = e0.z; e.W = e0.w;
    e.anc = 0.0f;
    e.anc_item = -1;
    if (M != kIso) {
        const float4 e1 = p[1], e2 = p[2], e3 = p[3], e4 = p[4];
        e.d[0] = e1.x; e.d[1] = e1.y; e.d[2] = e1.z; e.P = e1.w;
        e.r[0] = e2.x; e.r[1] = e2.y; e.r[2] = e2.z;
        e.A[0] = e3.x; e.A[1] = e3.y; e.A[2] = e3.z; e.A[3] = e3.w; e.A[4] = e4.x; e.A[5] = e4.y;
        if (M == kQEM) {
            e.anc = e4.z;
            e.anc_item = __float_as_int(e4.w);
        }
    }
    if (M == kAniso) {
        const float4 e5 = p[5], e6 = p[6], e7 = p[7];
        e.T[0] = e5.x; e.T[1] = e5.y; e.T[2] = e5.z; e.T[3] = e5.w; e.T[4] = e6.x; e.T[5] = e6.y;
        e.g[0] = e6.z; e.g[1] = e6.w; e.g[2] = e7.x;
    }
}

// symmetric 3x3 (compact) times vector
ACVD_DEV void sym_mul(const double a[6], const double v[3], double o[3]) {
    o[0] = a[0] * v[0] + a[1] * v[1] + a[2] * v[2];
    o[1] = a[1] * v[0] + a[3] * v[1] + a[4] * v[2];
    o[2] = a[2] * v[0] + a[4] * v[1] + a[5] * v[2];
}
ACVD_DEV void sym_mul(const float a[6], const float v[3], float o[3]) {
    o[0] = dot3(a[0], v[0], a[1], v[1], a[2], v[2]);
    o[1] = dot3(a[1], v[0], a[3], v[1], a[4], v[2]);
    o[2] = dot3(a[4], v[1], a[2], v[0], a[5], v[2]);
}

// ---------------------------------------------------------------------------
// Energy changes in float32, in forms built from local differences only
// (x - m, m' - m, the residual r = b - A m) so that no large cancelling terms
// appear.  E_iso = -|S|^2 / W; the QEM energy with the placed vertex c = m + delta
// is W |delta|^2 - |S|^2 / W; the anisotropic energy is c^T T c - 2 c.u.
// ---------------------------------------------------------------------------

// Cluster X after removing (sgn = -1) or adding (sgn = +1) the item: weight,
// centroid shift dm = m' - m and placement delta' (relative to m').
template <int M>
ACVD_DEV void modified_cluster(const EvalRec& c, const ItemRec& it, float sgn, int level, float thr,
                               float& Wn, float dm[3], float dn[3]) {
    // (a product by sgn = +-1 is exact)
    Wn = __fadd_rn(c.W, sgn * it.w);
    const float xm[3] = {it.x[0] - c.m[0], it.x[1] - c.m[1], it.x[2] - c.m[2]};
    const float f = sgn * it.w / Wn;
#pragma unroll
    for (int j = 0; j < 3; j++) dm[j] = __fmul_rn(f, xm[j]);
    float An[6];
#pragma unroll
    for (int j = 0; j < 6; j++) An[j] = __fadd_rn(c.A[j], sgn * it.A[j]);
    float Aix[3], And[3];
    sym_mul(it.A, xm, Aix);
    sym_mul(An, dm, And);
    float rn[3];
#pragma unroll
    for (int j = 0; j < 3; j++) rn[j] = __fsub_rn(__fadd_rn(c.r[j], sgn * Aix[j]), And[j]);
    pinv_apply<float>(An, rn, dn, level, thr, 8);
}

// Energy change of cluster X (anisotropic metric) when its placed vertex moves by
// e, ignoring the item's own term: -2 e.g + e^T T e.
ACVD_DEV float aniso_shift(const EvalRec& c, const float e[3]) {
    float Te[3];
    sym_mul(c.T, e, Te);
    return __fmaf_rn(-2.0f, dot3(e[0], c.g[0], e[1], c.g[1], e[2], c.g[2]),
                     dot3(e[0], Te[0], e[1], Te[1], e[2], Te[2]));
}

ACVD_DEV float item_quad(const float T[6], const float v[3]) {
    float Tv[3];
    sym_mul(T, v, Tv);
    return dot3(v[0], Tv[0], v[1], Tv[1], v[2], Tv[2]);
}

// The isotropic part of a change, a quotient times a squared distance, and that of the
// placed vertex added: v + (W' |delta'|^2 - P).
ACVD_DEV float iso_part(float num, float den, float d2) { return __fmul_rn(__fdiv_rn(num, den), d2); }
ACVD_DEV float with_placement(float v, float Wn, const float dn[3], float P) {
    return __fadd_rn(v, __fmaf_rn(Wn, dot3(dn[1], dn[1], dn[0], dn[0], dn[2], dn[2]), -P));
}

// Removing its anchor item from a QEM cluster breaks the anchor, which the reference
// prices at 1e100 (vtkQEMetricForClustering.h:194-200, 259): such a move is never taken.
constexpr float kBrokenAnchor = 1e30f;

template <int M>
ACVD_DEV bool is_anchor_item(const EvalRec& eL, int i) {
    return M == kQEM && eL.anc != 0.0f && eL.anc_item == i;
}

// Part of the energy change that depends on the source cluster L only.
template <int M>
ACVD_DEV float remove_part(const EvalRec& eL, const ItemRec& it, const RunFlags& fl, float cprime[3]) {
    const float xm[3] = {it.x[0] - eL.m[0], it.x[1] - eL.m[1], it.x[2] - eL.m[2]};
    const float d2 = dot3(xm[0], xm[0], xm[1], xm[1], xm[2], xm[2]);
    if (M == kIso) return iso_part(__fmul_rn(-it.w, eL.W), __fsub_rn(eL.W, it.w), d2);
    if (M == kQEM) {
        if (eL.anc != 0.0f) return __fmul_rn(-it.w, d2);   // placed vertex fixed at the anchor: -w |x - p|^2
        const float v = iso_part(__fmul_rn(-it.w, eL.W), __fsub_rn(eL.W, it.w), d2);
        if (!(fl.constrained && fl.level > 0)) return v;
        float Wn, dm[3], dn[3];
        modified_cluster<M>(eL, it, -1.0f, fl.level, fl.thr, Wn, dm, dn);
        return with_placement(v, Wn, dn, eL.P);
    }
    // anisotropic: shift of L's placed vertex, minus the item's own term at L'
    float Wn, dm[3], dn[3], e[3];
    modified_cluster<M>(eL, it, -1.0f, fl.level, fl.thr, Wn, dm, dn);
#pragma unroll
    for (int j = 0; j < 3; j++) {
        e[j] = __fsub_rn(__fadd_rn(dm[j], dn[j]), eL.d[j]);
        cprime[j] = __fsub_rn(__fsub_rn(xm[j], dm[j]), dn[j]);
    }
    return __fsub_rn(aniso_shift(eL, e), item_quad(it.T, cprime));
}

template <int M>
ACVD_DEV float add_part(const EvalRec& eB, const ItemRec& it, const RunFlags& fl) {
    const float xm[3] = {it.x[0] - eB.m[0], it.x[1] - eB.m[1], it.x[2] - eB.m[2]};
    const float d2 = dot3(xm[0], xm[0], xm[1], xm[1], xm[2], xm[2]);
    if (M == kIso) return iso_part(__fmul_rn(it.w, eB.W), __fadd_rn(eB.W, it.w), d2);
    if (M == kQEM) {
        if (eB.anc != 0.0f) return __fmul_rn(it.w, d2);
        const float v = iso_part(__fmul_rn(it.w, eB.W), __fadd_rn(eB.W, it.w), d2);
        if (!(fl.constrained && fl.level > 0)) return v;
        float Wn, dm[3], dn[3];
        modified_cluster<M>(eB, it, 1.0f, fl.level, fl.thr, Wn, dm, dn);
        return with_placement(v, Wn, dn, eB.P);
    }
    float Wn, dm[3], dn[3], e[3], xc[3];
    modified_cluster<M>(eB, it, 1.0f, fl.level, fl.thr, Wn, dm, dn);
#pragma unroll
    for (int j = 0; j < 3; j++) {
        e[j] = __fsub_rn(__fadd_rn(dm[j], dn[j]), eB.d[j]);
        xc[j] = __fsub_rn(__fsub_rn(xm[j], dm[j]), dn[j]);
    }
    return __fadd_rn(aniso_shift(eB, e), item_quad(it.T, xc));
}

// ---------------------------------------------------------------------------
// local connectivity (vtkVerticesProcessing.h:168-237): the ring members of the
// item that carry label L must stay connected through edges among themselves.
// ---------------------------------------------------------------------------
ACVD_DEV bool ring_connected(const DevState& st, int p0, int p1, int L) {
    const int d = p1 - p0;
    if (d > 32) return false;
    unsigned msk = 0u;
    for (int q = 0; q < d; q++)
        if (st.label[st.col[p0 + q]] == L) msk |= 1u << q;
    if (msk == 0u) return true;
    unsigned vis = msk & (0u - msk);
    unsigned front = vis;
    while (front) {
        unsigned nxt = 0u;
        unsigned f = front;
        while (f) {
            const int q = __ffs(f) - 1;
            f &= f - 1u;
            nxt |= st.adj[p0 + q];
        }
        nxt &= msk & ~vis;
        vis |= nxt;
        front = nxt;
    }
    return vis == msk;
}

// An item changed cluster: it and its ring may now lie on a boundary, and their
// cached screens (bflag 2) no longer hold.
ACVD_DEV void mark_ring(const DevState& st, int i) {
    st.bflag[i] = 1;
    for (int p = st.row[i]; p < st.row[i + 1]; p++) st.bflag[st.col[p]] = 1;
}

ACVD_DEV void warp_count(unsigned long long* ctr, unsigned v) {
    const unsigned tot = __reduce_add_sync(kFull, v);
    if ((threadIdx.x & 31) == 0 && tot) atomicAdd(ctr, (unsigned long long)tot);
}

// ---------------------------------------------------------------------------
// eval: proposals for one colour class
//
// An item is skipped when neither its own cluster nor any cluster around it
// changed since it was last evaluated without result (the reference skips an
// edge when neither cluster was modified in the previous loop,
// vtkUniformClustering.h:912-920).  Proposals go to a compact per-step list.
// ---------------------------------------------------------------------------
constexpr int kRingPref = 8;   // ring slots whose labels phase A loads up front
constexpr int kMaxTgt = 8;     // destination clusters per item on the task path
constexpr int kTaskRemove = 15;  // task code of an item's remove part
constexpr int kScrCached = 1 << 30;  // screen list entry: the item's screen is cached (bflag 2)

// Local connectivity of an item with d <= 8 neighbours, from their labels and adjacency: the
// slots labelled L that the first of them reaches.  All in registers: read from the rings'
// CSR instead (its bounds, then a word for each slot reached), the test put two or three more
// dependent loads on the evaluation's chain (2047 x 1801 anisotropic solve: 45.8 ms against
// 45.4 now, 1024 x 1024: 23.2 against 23.1, 1024 x 512 quadric torus: 9.63 against 9.57).
ACVD_DEV bool ring_connected8(uint2 near, int d, int L, const int* lb) {
    unsigned msk = 0u;
#pragma unroll
    for (int q = 0; q < 8; q++)
        if (q < d && lb[q] == L) msk |= 1u << q;
    unsigned vis = msk & (0u - msk);
    for (unsigned front = vis; front;) {
        // the adjacency bytes of the slots in front, or-ed: bit q of front spread to byte q
        const unsigned lo = (((front & 15u) * 0x00204081u) & 0x01010101u) * 255u & near.x;
        const unsigned hi = (((front >> 4) * 0x00204081u) & 0x01010101u) * 255u & near.y;
        unsigned m = lo | hi;
        m |= m >> 16;
        m |= m >> 8;
        front = m & msk & ~vis;
        vis |= front;
    }
    return vis == msk;
}

// Local connectivity with the first kRingPref ring labels already loaded.
ACVD_DEV bool ring_connected_pref(const DevState& st, int p0, int p1, int L, const int* lb) {
    const int d = p1 - p0;
    if (d > 32) return false;
    unsigned msk = 0u;
#pragma unroll
    for (int q = 0; q < kRingPref; q++)
        if (q < d && lb[q] == L) msk |= 1u << q;
    for (int q = kRingPref; q < d; q++)
        if (st.label[st.col[p0 + q]] == L) msk |= 1u << q;
    if (msk == 0u) return true;
    unsigned vis = msk & (0u - msk);
    unsigned front = vis;
    while (front) {
        unsigned nxt = 0u;
        unsigned f = front;
        while (f) {
            const int q = __ffs(f) - 1;
            f &= f - 1u;
            nxt |= st.adj[p0 + q];
        }
        nxt &= msk & ~vis;
        vis |= nxt;
        front = nxt;
    }
    return vis == msk;
}

// Items per tile when `blocks` blocks of TB threads share `count` items: whole warps, no more
// than TB.  An item on a boundary makes about 2.4 energy tasks, which the block's threads
// share, so a block with TB items runs two rounds of them while other SMs idle.
template <int TB>
__host__ __device__ inline int spread_items(int64_t count, int64_t blocks) {
    const int64_t n = (count + 32 * blocks - 1) / (32 * blocks) * 32;
    return (int)(n < 32 ? 32 : (n > TB ? TB : n));
}

// A new evaluation sweep for an item whose screen record c is valid (bflag 2): into
// the record, or, beyond the sweeps a record holds, the item is screened in full next.
ACVD_DEV void set_cached_ev(const DevState& st, int i, int4 c, int ev) {
    if (ev < kCacheSweeps) st.tcache[i] = screen_with_ev(c, ev);
    else st.bflag[i] = 1;
}

// One tile of `per` items of a colour class (blockDim.x == TB; every thread of the
// block calls it).  Arrays written during a sweep are read through plain
// pointers: the persistent sweep kernel reads them after other blocks wrote them.
//
// Phase A (one item per thread): skip test, boundary test, size guard and local
// connectivity, with the ring's labels loaded up front; a movable item joins the
// block's work list with its distinct destination clusters.  Phase B1: the energy
// tests -- one task per (item, destination) plus one per item for the part that
// depends on its own cluster -- spread over all threads of the block.  Phase B2
// (one work item per thread): the best destination, the acceptance margin, the
// proposal and its claims.  Unassigned items and items with more than kMaxTgt
// destinations run the whole test in B2.
//
// List mode (entries != nullptr): the tile's items are entries[0 .. n_entries), the
// colour-list positions a screen_kernel pass forwarded (see below); they were
// counted as visited there.
template <int M, int TB = 256>
ACVD_DEV void eval_tile(const DevState& st, int item0, int64_t count, int color, int claims, int64_t tile, int per,
                        const int* entries = nullptr, int n_entries = 0) {
    __shared__ int s_idx[TB];                 // work item -> colour-list position
    __shared__ int s_tgt[TB][kMaxTgt];        // work item -> destination clusters (ring order)
    __shared__ float s_val[TB][kMaxTgt + 1];  // energy parts: [j] add to s_tgt[j], [kMaxTgt] remove
    __shared__ signed char s_nt[TB];          // destinations; -1: the whole test runs in B2
    __shared__ unsigned short s_task[TB * kMaxTgt];   // add tasks: (work item << 4) | destination
    __shared__ unsigned char s_rem[TB];                // work items whose remove part B1 computes
    __shared__ int s_scr[TB];                 // flagged items of the tile (colour-list positions)
    __shared__ unsigned char s_rec[TB];       // work item -> its screen record is valid (bflag 2)
    __shared__ int4 s_scn[TB];                // ... and that record (its evaluation sweep aside)
    __shared__ int s_lab[TB];                 // work item -> its cluster
    __shared__ unsigned s_nwork, s_ntask, s_nrem, s_nscr, s_nfull;
    __syncthreads();                     // the previous tile is done with the shared arrays
    if (threadIdx.x == 0) {
        s_nwork = 0u;
        s_ntask = 0u;
        s_nrem = 0u;
        s_nfull = 0u;
        s_nscr = 0u;
    }
    __syncthreads();
    const int epoch = color * kRounds;   // claim epoch of this step's first matching round
    const bool listed = entries != nullptr;
    const bool in = (int)threadIdx.x < (listed ? n_entries : per) && (listed || tile * per + threadIdx.x < count);
    const int64_t idx_t = listed ? (in ? (int64_t)entries[threadIdx.x] : 0) : tile * per + threadIdx.x;
    const SweepState sw = *st.sweep;
    const RunFlags fl = *st.flags;
    unsigned n_slots = 0, n_bnd = 0, n_tgt = 0, n_cand = 0, n_scr = 0, n_cached = 0;
    // A0: only items that may lie on a boundary go on to the ring screen, packed
    // so that warps without one issue nothing: cached screens from the front of the
    // list, full screens from its back, so that a warp runs one kind
    {
        const unsigned char bf = in ? st.bflag[item0 + idx_t] : (unsigned char)0;
        const int lane = threadIdx.x & 31;
        const unsigned below = (1u << lane) - 1u;
        const unsigned bal_c = __ballot_sync(kFull, bf == 2);
        const unsigned bal_f = __ballot_sync(kFull, bf == 1);
        if (bal_c) {
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(&s_nscr, (unsigned)__popc(bal_c));
            base = __shfl_sync(kFull, base, 0);
            if (bf == 2) s_scr[base + __popc(bal_c & below)] = (int)idx_t | kScrCached;
        }
        if (bal_f) {
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(&s_nfull, (unsigned)__popc(bal_f));
            base = __shfl_sync(kFull, base, 0);
            if (bf == 1) s_scr[TB - 1 - (base + __popc(bal_f & below))] = (int)idx_t;
        }
    }
    __syncthreads();
    if (threadIdx.x < s_nscr || threadIdx.x >= (unsigned)TB - s_nfull) {
        const int code = s_scr[threadIdx.x];
        const int64_t idx = code & ~kScrCached;
        const int i = item0 + (int)idx;
        n_scr = 1;
        // a cached screen's record holds the item's cluster and evaluation sweep too; a full
        // screen starts from the item's label, evaluation sweep and ring, loaded together
        const bool cached = (code & kScrCached) != 0;
        int4 c = make_int4(0, 0, 0, 0), ra = c, rb = c;
        uint2 near = make_uint2(0u, 0u);
        int lab_i = 0, evald_i = 0;
        if (cached) {
            c = load_now(st.tcache + i);
        } else {
            lab_i = load_now(st.label + i);
            evald_i = load_now(st.evald + i);
            ra = load_now(st.ring8 + 2 * (int64_t)i);
            rb = load_now(st.ring8 + 2 * (int64_t)i + 1);
            if (fl.connexity) near = load_now(st.near8 + i);
        }
        const Screen sc = unpack_screen(c);
        const int L = cached ? sc.L : lab_i;
        int ev_i = cached ? sc.ev : evald_i;
        if (cached) ACVD_VALID(st, L == st.label[i] && ev_i == st.evald[i]);
        bool screened = !ACVD_VALID(st, L >= 0 && L <= st.k);   // a bad label is skipped
        if (cached && !screened) {
            // the ring kept its labels since the last full screen: its distinct
            // neighbour clusters and the connectivity test are in the cache
            const int n = sc.n;
            const bool conn_known = sc.conn_known, conn_ok = sc.conn_ok;
            // the size and every stamp in one go (unused targets are cluster 0)
            const int tg[3] = {sc.t[0], sc.t[1], sc.t[2]};
            const int size = load_now(st.size + L), stamp = load_now(st.stamp + L);
            const int st0 = load_now(st.stamp + tg[0]), st1 = load_now(st.stamp + tg[1]),
                      st2 = load_now(st.stamp + tg[2]);
            const bool may_move = size > 1 && !(st.frozen && st.frozen[L]);
            if (!(fl.connexity && may_move && !conn_known)) {
                screened = true;
                n_cached = 1;
                const bool fresh = ev_i <= sw.floor || stamp >= ev_i || (n > 0 && st0 >= ev_i) ||
                                   (n > 1 && st1 >= ev_i) || (n > 2 && st2 >= ev_i);
                if (fresh) {
                    n_bnd = 1;
                    if (may_move && (!fl.connexity || conn_ok)) {
                        const int w = (int)atomicAdd(&s_nwork, 1u);
                        s_idx[w] = (int)idx;
                        s_lab[w] = L;
                        s_rec[w] = 1;
                        s_scn[w] = c;
                        int nt = 0;
#pragma unroll
                        for (int q = 0; q < 3; q++)
                            if (q < n && !(st.frozen && st.frozen[tg[q]])) s_tgt[w][nt++] = tg[q];
                        s_nt[w] = (signed char)nt;
                        n_tgt += (unsigned)nt;
                        if (nt > 0) {
                            const unsigned base = atomicAdd(&s_ntask, (unsigned)nt);
                            for (int j = 0; j < nt; j++) s_task[base + j] = (unsigned short)((w << 4) | j);
                            s_rem[atomicAdd(&s_nrem, 1u)] = (unsigned char)w;
                        }
                    } else {
                        st.evald[i] = sw.sweep;   // evaluated: nothing it may do
                        set_cached_ev(st, i, c, sw.sweep);
                    }
                }
            }
        }
        if (!screened) {
        if (cached) {   // its connectivity test is not known yet: the full screen after all
            ra = st.ring8[2 * (int64_t)i];
            rb = st.ring8[2 * (int64_t)i + 1];
            near = st.near8[i];
        }
        int lb[kRingPref] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
        const bool longer = lb[7] == -2;   // ring longer than 8: bounds and tail from the CSR
        int deg = 0;
        if (longer) {
            deg = st.row[i + 1] - st.row[i];
            lb[7] = st.col[st.row[i] + 7];
        } else {
#pragma unroll
            for (int q = 0; q < kRingPref; q++) deg += lb[q] >= 0;
        }
#pragma unroll
        for (int q = 0; q < kRingPref; q++) lb[q] = lb[q] >= 0 ? load_now(st.label + lb[q]) : L;
        // every stamp in one go (stamp[k], the null label's, exists and is not used)
        int sb[kRingPref];
        const int stamp = load_now(st.stamp + L), size = load_now(st.size + L);
#pragma unroll
        for (int q = 0; q < kRingPref; q++) sb[q] = lb[q] != L ? load_now(st.stamp + lb[q]) : 0;
        bool fresh = ev_i <= sw.floor || (L < st.k && stamp >= ev_i);
        n_slots = (unsigned)deg;
        bool boundary = false;
#pragma unroll
        for (int q = 0; q < kRingPref; q++) {
            const int B = lb[q];
            if (B != L) {
                boundary = true;
                if (B < st.k && sb[q] >= ev_i) fresh = true;
            }
        }
        if (longer) {
            const int p0 = st.row[i];
            for (int q = kRingPref; q < deg; q++) {
                const int B = st.label[st.col[p0 + q]];
                if (B != L) {
                    boundary = true;
                    if (B < st.k && st.stamp[B] >= ev_i) fresh = true;
                }
            }
        }
        if (!boundary) st.bflag[i] = 0;   // interior until a commit touches its ring
        const bool may_move = L < st.k && size > 1 && !(st.frozen && st.frozen[L]);
        int conn = -1;   // the local connectivity test, evaluated at most once
        // cache a boundary screen of a ring of at most 8 with at most 3 neighbour
        // clusters: they hold until a commit touches the ring (mark_ring).  The record
        // is written below, with the evaluation sweep this screen leaves.
        bool cache_it = false;
        int4 rec = make_int4(0, 0, 0, 0);
        if (boundary && !longer && L < st.k && st.k <= kCacheClusters) {
            int tg[3] = {0, 0, 0};
            int n = 0;
#pragma unroll
            for (int q = 0; q < kRingPref; q++) {
                const int B = lb[q];
                if (B == L || B >= st.k) continue;
                bool dup = false;
#pragma unroll
                for (int r = 0; r < q; r++) dup |= lb[r] == B;
                if (dup) continue;
                if (n < 3) tg[n] = B;
                n++;
            }
            if (n <= 3) {
                int meta = n;
                if (fl.connexity && may_move) {
                    conn = ring_connected8(near, deg, L, lb) ? 1 : 0;
                    meta |= 4 | (conn ? 8 : 0);
                }
                rec = pack_screen(L, tg[0], tg[1], tg[2], meta, 0);
                cache_it = true;
            }
        }
        if (boundary && fresh) {
            n_bnd = 1;
            if (fl.connexity && may_move && conn < 0)
                conn = (longer ? ring_connected_pref(st, st.row[i], st.row[i] + deg, L, lb)
                               : ring_connected8(near, deg, L, lb)) ? 1 : 0;
            const bool movable = L >= st.k || (may_move && (!fl.connexity || conn == 1));
            if (movable) {
                const int w = (int)atomicAdd(&s_nwork, 1u);
                s_idx[w] = (int)idx;
                s_lab[w] = L;
                s_rec[w] = cache_it ? 1 : 0;
                s_scn[w] = rec;
                int nt = 0;
                bool all = L < st.k && deg <= kRingPref;
#pragma unroll
                for (int q = 0; q < kRingPref; q++) {
                    const int B = lb[q];
                    if (!all || B == L || B >= st.k || (st.frozen && st.frozen[B])) continue;
                    bool dup = false;
#pragma unroll
                    for (int r = 0; r < q; r++) dup |= lb[r] == B;
                    if (dup) continue;
                    if (nt == kMaxTgt) {
                        all = false;
                        continue;
                    }
                    s_tgt[w][nt++] = B;
                }
                if (all) {
                    s_nt[w] = (signed char)nt;
                    n_tgt += (unsigned)nt;
                    if (nt > 0) {
                        const unsigned base = atomicAdd(&s_ntask, (unsigned)nt);
                        for (int j = 0; j < nt; j++) s_task[base + j] = (unsigned short)((w << 4) | j);
                        s_rem[atomicAdd(&s_nrem, 1u)] = (unsigned char)w;
                    }
                } else {
                    s_nt[w] = -1;
                }
            } else {
                st.evald[i] = sw.sweep;   // evaluated: nothing it may do
                ev_i = sw.sweep;
            }
        }
        if (cache_it) {
            if (ev_i < kCacheSweeps) {
                st.tcache[i] = screen_with_ev(rec, ev_i);
                st.bflag[i] = 2;
            } else {
                st.bflag[i] = 1;   // beyond the sweeps a record holds: screened in full
            }
        }
        }
    }
    __syncthreads();
    // B1: energy parts -- the remove parts first, then the add parts, so that a warp
    // runs one kind
    const unsigned nrem = s_nrem, ntask = nrem + s_ntask;
    for (unsigned t = threadIdx.x; t < ntask; t += TB) {
        const unsigned code = t < nrem ? ((unsigned)s_rem[t] << 4) | (unsigned)kTaskRemove : s_task[t - nrem];
        const int w = (int)(code >> 4), j = (int)(code & 15u);
        const int i = item0 + s_idx[w];
        ItemRec it;
        load_item<M>(st, i, it);
        if (j == kTaskRemove) {
            EvalRec eL;
            load_eval<M>(st, s_lab[w], eL);
            float xc[3];
            s_val[w][kMaxTgt] = is_anchor_item<M>(eL, i) ? kBrokenAnchor : remove_part<M>(eL, it, fl, xc);
        } else {
            EvalRec eB;
            load_eval<M>(st, s_tgt[w][j], eB);
            s_val[w][j] = add_part<M>(eB, it, fl);
        }
    }
    __syncthreads();
    // B2: decision
    int4 my_cand = make_int4(-1, -1, -1, 0);   // x = -1: no proposal
    if (threadIdx.x < s_nwork) {
        const int w = threadIdx.x;
        const int widx = s_idx[w];
        const int i = item0 + widx;
        const int L = s_lab[w];
        const int nt = s_nt[w];
        int best = -1;
        unsigned pr = 0u;
        if (nt >= 0) {
            if (nt > 0) {
                const float rem = s_val[w][kMaxTgt];
                float bde = 0.0f, badd = 0.0f;
                for (int j = 0; j < nt; j++) {
                    const int B = s_tgt[w][j];
                    const float add = s_val[w][j];
                    const float de = rem + add;
                    if (de < bde || (de == bde && best >= 0 && B < best)) { best = B; bde = de; badd = add; }
                }
                // a move must gain more than the float32 error of its own test
                // (two near-tie moves could otherwise both test negative and
                // alternate); the reference keeps an item on ties (:960)
                if (best >= 0 && !(bde < -kAcceptTol * (fabsf(rem) + fabsf(badd)))) best = -1;
                if (best >= 0) pr = prio_of_delta(bde);
            }
        } else {
            const int p0 = st.row[i], p1 = st.row[i + 1];
            ItemRec it;
            load_item<M>(st, i, it);
            if (L >= st.k) {
                // unassigned item: joins the neighbouring cluster it is cheapest to join
                float bv = 0.0f;
                for (int p = p0; p < p1; p++) {
                    const int B = st.label[st.col[p]];
                    if (B >= st.k) continue;
                    const float4 e0 = st.ev[(int64_t)B * Layout<M>::ev];
                    const float dx = it.x[0] - e0.x, dy = it.x[1] - e0.y, dz = it.x[2] - e0.z;
                    const float v = it.w * e0.w / (e0.w + it.w) * (dx * dx + dy * dy + dz * dz);
                    n_tgt++;
                    if (best < 0 || v < bv || (v == bv && B < best)) { best = B; bv = v; }
                }
            } else {
                EvalRec eL;
                load_eval<M>(st, L, eL);
                float xc[3];
                const float rem = is_anchor_item<M>(eL, i) ? kBrokenAnchor : remove_part<M>(eL, it, fl, xc);
                float bde = 0.0f, badd = 0.0f;
                for (int p = p0; p < p1; p++) {
                    const int B = st.label[st.col[p]];
                    if (B == L || B >= st.k || (st.frozen && st.frozen[B])) continue;
                    bool dup = false;
                    for (int q = p0; q < p; q++) dup |= (st.label[st.col[q]] == B);
                    if (dup) continue;
                    EvalRec eB;
                    load_eval<M>(st, B, eB);
                    const float add = add_part<M>(eB, it, fl);
                    const float de = rem + add;
                    n_tgt++;
                    if (de < bde || (de == bde && best >= 0 && B < best)) { best = B; bde = de; badd = add; }
                }
                if (best >= 0 && !(bde < -kAcceptTol * (fabsf(rem) + fabsf(badd)))) best = -1;
                if (best >= 0) pr = prio_of_delta(bde);
            }
        }
        if (best >= 0) {
            if (claims) {
                const unsigned long long c = make_claim((unsigned)epoch, pr, (unsigned)widx);
                if (L < st.k) atomicMin(&st.claim[L], c);
                atomicMin(&st.claim[best], c);
            } else if (L < st.k) {
                atomicAdd(&st.out_cnt[L], 1);   // relaxed step: proposals leaving L
            }
            n_cand = 1;
            my_cand = make_int4(widx, best, L, (int)pr);
            st.evald[i] = -1;
            if (s_rec[w]) set_cached_ev(st, i, s_scn[w], -1);
        } else {
            st.evald[i] = sw.sweep;
            if (s_rec[w]) set_cached_ev(st, i, s_scn[w], sw.sweep);
        }
    }
    // block-aggregated append to the compact proposal list and block totals of the
    // counters: one atomic per block and counter (tens of thousands of warps would
    // otherwise serialise on the class's count and the counter stripes)
    {
        constexpr int kNC = 7;
        constexpr int kW = TB / 32;
        __shared__ unsigned s_wc[kW], s_base, s_cnt[kW][kNC];
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const unsigned bal = __ballot_sync(kFull, my_cand.x >= 0);
        const unsigned v[kNC] = {(in && !listed) ? 1u : 0u, n_scr - n_cached, n_cached, n_slots, n_bnd, n_tgt,
                                 n_cand};
#pragma unroll
        for (int c = 0; c < kNC; c++) {
            const unsigned t = __reduce_add_sync(kFull, v[c]);
            if (lane == 0) s_cnt[wid][c] = t;
        }
        if (lane == 0) s_wc[wid] = (unsigned)__popc(bal);
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned tot = 0;
            for (int w = 0; w < kW; w++) {
                const unsigned c = s_wc[w];
                s_wc[w] = tot;
                tot += c;
            }
            s_base = tot ? atomicAdd(&st.cand_count[color], tot) : 0u;
        } else if (threadIdx.x >= 32 && threadIdx.x < 32 + kNC) {
            const int c = threadIdx.x - 32;
            const int which = c == 0 ? kCntVisited : c == 1 ? kCntScreened : c == 2 ? kCntCached
                            : c == 3 ? kCntSlots : c == 4 ? kCntBoundary : c == 5 ? kCntTargets : kCntCand;
            unsigned t = 0;
            for (int w = 0; w < kW; w++) t += s_cnt[w][c];
            if (t) atomicAdd(ctr(st.counters, which), (unsigned long long)t);
        }
        __syncthreads();
        if (my_cand.x >= 0) st.cand_list[s_base + s_wc[wid] + __popc(bal & ((1u << lane) - 1u))] = my_cand;
    }
}

// TB: threads (and items) per block.  A block is the unit that waits at the tile's
// barriers, so smaller blocks at the same threads per SM (B * 256 / TB blocks of TB)
// let more of them be in different phases of their tiles: the default is 128 threads, 8
// blocks per SM (64 registers a thread), for every metric.  Blocks of 256 are compiled for
// 3, 4 and 5 per SM (80, 64 and 48 registers: fewer spill less of the energy tests, more
// hide more latency); launch_eval takes the context's eval_blocks and eval_threads
// (ACVD_EVAL_BLOCKS, ACVD_EVAL_THREADS; the autotuner times the choices).  Converged solves in
// ms, 256 threads at 3 / 4 / 5 blocks, 128 threads: 1024 x 512 quadric torus 11.13 / 10.95 / 11.01,
// 10.64 to 10.94; 4096^2 anisotropic heightfield 181.0 / 171.4 / 177.1, 173.2; batch of 256 quadric
// meshes 100.2 / 96.5 / 96.2, 97.1.
template <int M, int B, int TB = 256>
__global__ void __launch_bounds__(TB, B * 256 / TB) eval_kernel(DevState st, int item0, int64_t count, int color,
                                                                int claims, int per) {
    eval_tile<M, TB>(st, item0, count, color, claims, blockIdx.x, per);
}

// blocks of 256 per SM where only ACVD_EVAL_THREADS=256 was asked for: the fused evaluation 4
// (isotropic, QEM) and 5 (the quadric-anisotropic metric, by which it was faster when every
// class ran it), the work-list evaluation 4
constexpr int default_eval_blocks(int metric) { return metric == kAniso ? 5 : 4; }
constexpr int kDefaultListBlocks = 4;

// ---------------------------------------------------------------------------
// Split evaluation of a large colour class: screen_kernel streams the class and
// settles every item whose screen decides it does nothing -- interior items
// (boundary flag 0) and cached screens whose clusters did not change since the
// item's last evaluation, or that cannot move -- exactly as eval_tile's cached
// path would; the other items (full screens, fresh movable cached screens) are
// appended to a work list that eval_list_kernel runs through eval_tile.  Each item
// takes the same decisions as in the fused kernel, so the clustering is the same
// bit for bit; the screen pass is a plain stream at high occupancy with several
// items' loads in flight per thread, where the fused kernel's per-tile barriers
// and energy-test registers left the cached screens latency-bound.
//
// Work-list layout: kWorkStripes stripes, block b of the screen pass appends to
// stripe b % kWorkStripes (one atomic per block, spread over the stripes' counters);
// stripe s holds its entries at work[s * cap ...], cap = work_cap(count).
// ---------------------------------------------------------------------------
constexpr int kScreenFlags = kScreenTile / 256;   // boundary flags each thread loads per tile
constexpr int kScreenBatch = 4;                    // cached screens each thread resolves at once

// Cached screen of item i: forward it (energy test to run, or its connectivity test is
// not cached), or settle it here -- counted as cached, and when fresh but unable to
// move marked evaluated -- exactly as eval_tile's cached path decides.
template <int M>
__global__ void __launch_bounds__(256, 4) screen_kernel(DevState st, int item0, int64_t count, int color, int* work,
                                                        unsigned* work_count) {
    __shared__ int s_cached[kScreenTile];   // tile positions with a cached screen
    __shared__ int s_fwd[kScreenTile];      // tile positions forwarded to the work list
    __shared__ unsigned s_nc, s_nf, s_base, s_cnt[8][3];
    const SweepState sw = *st.sweep;
    const RunFlags fl = *st.flags;
    const int64_t cap = work_cap(count);
    const int64_t ntiles = (count + kScreenTile - 1) / kScreenTile;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned n_visit = 0, n_cached = 0, n_bnd = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        if (threadIdx.x == 0) {
            s_nc = 0u;
            s_nf = 0u;
        }
        __syncthreads();
        const int64_t t0 = tile * kScreenTile;
        // stage 1: every flag of the tile in one burst (coalesced, kScreenFlags loads in
        // flight per thread), then the cached items compacted, full screens forwarded
        unsigned char bf[kScreenFlags];
#pragma unroll
        for (int u = 0; u < kScreenFlags; u++) {
            const int64_t idx = t0 + u * 256 + threadIdx.x;
            bf[u] = idx < count ? st.bflag[item0 + idx] : (unsigned char)0;
            n_visit += idx < count ? 1u : 0u;
        }
#pragma unroll
        for (int u = 0; u < kScreenFlags; u++) {
            const int pos = u * 256 + (int)threadIdx.x;
            if (bf[u] == 2) s_cached[atomicAdd(&s_nc, 1u)] = pos;
            else if (bf[u] == 1) s_fwd[atomicAdd(&s_nf, 1u)] = pos;
        }
        __syncthreads();
        // stage 2: the cached screens, kScreenBatch per thread with all their loads
        // issued before any is used
        const int nc = (int)s_nc;
        for (int j0 = 0; j0 < nc; j0 += 256 * kScreenBatch) {
            // one 16-byte record per cached screen: cluster, targets, evaluation sweep
            int pos[kScreenBatch], size[kScreenBatch], stamp[kScreenBatch][4];
            int4 c[kScreenBatch];
#pragma unroll
            for (int u = 0; u < kScreenBatch; u++) {
                const int j = j0 + u * 256 + (int)threadIdx.x;
                pos[u] = j < nc ? s_cached[j] : -1;
                c[u] = pos[u] >= 0 ? st.tcache[item0 + (int)(t0 + pos[u])] : make_int4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < kScreenBatch; u++) {
                const Screen sc = unpack_screen(c[u]);
                const bool known = pos[u] >= 0 && sc.L <= st.k;
                size[u] = known ? load_now(st.size + sc.L) : 0;
                stamp[u][0] = known ? load_now(st.stamp + sc.L) : 0;
#pragma unroll
                for (int q = 0; q < 3; q++) stamp[u][q + 1] = known ? load_now(st.stamp + sc.t[q]) : 0;
            }
#pragma unroll
            for (int u = 0; u < kScreenBatch; u++) {
                const Screen sc = unpack_screen(c[u]);
                const int L = sc.L, ev_i = sc.ev;
                if (pos[u] >= 0) {
                    const int i = item0 + (int)(t0 + pos[u]);
                    ACVD_VALID(st, L == st.label[i] && ev_i == st.evald[i]);
                }
                if (pos[u] < 0 || !ACVD_VALID(st, L >= 0 && L <= st.k)) continue;
                const int n = sc.n;
                const bool may_move = size[u] > 1 && !(st.frozen && st.frozen[L]);
                bool fwd = fl.connexity && may_move && !sc.conn_known;   // connectivity not cached: full screen
                if (!fwd) {
                    bool fresh = ev_i <= sw.floor || stamp[u][0] >= ev_i;
#pragma unroll
                    for (int q = 0; q < 3; q++)
                        if (q < n && stamp[u][q + 1] >= ev_i) fresh = true;
                    if (fresh && may_move && (!fl.connexity || sc.conn_ok)) {
                        fwd = true;   // an energy test to run
                    } else {
                        n_cached++;
                        if (fresh) {
                            n_bnd++;
                            const int i = item0 + (int)(t0 + pos[u]);
                            st.evald[i] = sw.sweep;   // nothing it may do
                            set_cached_ev(st, i, c[u], sw.sweep);
                        }
                    }
                }
                if (fwd) s_fwd[atomicAdd(&s_nf, 1u)] = pos[u];
            }
        }
        __syncthreads();
        // the tile's forwarded items: one atomic per tile, on the stripe's counter
        const int stripe = (int)(tile % kWorkStripes);
        if (threadIdx.x == 0) s_base = s_nf ? atomicAdd(&work_count[color * kWorkStripes + stripe], s_nf) : 0u;
        __syncthreads();
        int* out = work + stripe * cap + s_base;
        const int nf = (int)s_nf;
        for (int j = threadIdx.x; j < nf; j += 256) out[j] = (int)t0 + s_fwd[j];
    }
    const unsigned v[3] = {n_visit, n_cached, n_bnd};
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const unsigned t = __reduce_add_sync(kFull, v[q]);
        if (lane == 0) s_cnt[wid][q] = t;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int q = threadIdx.x;
        const int which = q == 0 ? kCntVisited : (q == 1 ? kCntCached : kCntBoundary);
        unsigned t = 0;
        for (int w = 0; w < 8; w++) t += s_cnt[w][q];
        if (t) atomicAdd(ctr(st.counters, which), (unsigned long long)t);
    }
}

// The work list of a screen_kernel pass through eval_tile, TB entries per tile,
// grid-stride over (stripe, tile) pairs.
template <int M, int B, int TB = 256>
__global__ void __launch_bounds__(TB, B * 256 / TB) eval_list_kernel(DevState st, int item0, int64_t count,
                                                                     int color, int claims, const int* work,
                                                                     const unsigned* work_count) {
    __shared__ unsigned s_cnt[kWorkStripes];
    if (threadIdx.x < kWorkStripes) s_cnt[threadIdx.x] = work_count[color * kWorkStripes + threadIdx.x];
    __syncthreads();
    unsigned mx = 0, total = 0;
    for (int q = 0; q < kWorkStripes; q++) {
        mx = max(mx, s_cnt[q]);
        total += s_cnt[q];
    }
    const int n = spread_items<TB>(total, gridDim.x);   // entries per tile
    const int64_t per = (mx + n - 1) / n;               // tiles of the fullest stripe
    const int64_t cap = work_cap(count);
    for (int64_t t = blockIdx.x; t < per * kWorkStripes; t += gridDim.x) {
        const int q = (int)(t % kWorkStripes);
        const int64_t j = t / kWorkStripes;
        const int64_t have = (int64_t)s_cnt[q] - j * n;
        if (have <= 0) continue;   // block-uniform
        eval_tile<M, TB>(st, item0, count, color, claims, t, n, work + q * cap + j * n,
                         have < n ? (int)have : n);
    }
}

// ---------------------------------------------------------------------------
// accumulators
// ---------------------------------------------------------------------------
// Adds sgn * (contribution of item i) to a cluster accumulator (double-float):
// S += w x, W += w, A += A_i, b += A_i x, T += T_i, u += T_i x, with the
// products formed exactly (TwoProd) so that b and u stay consistent with A, T, x.
template <int M>
ACVD_DEV void accumulate_item(df* acc, const ItemRec& it, float sgn) {
    auto addp = [&](int j, float a, float b) {
        const df p = two_prod(a, b);
        acc[j] = df_add(acc[j], sgn > 0 ? p : df_neg(p));
    };
    auto addf = [&](int j, float a) { acc[j] = df_add_f(acc[j], sgn * a); };
    addp(0, it.w, it.x[0]);
    addp(1, it.w, it.x[1]);
    addp(2, it.w, it.x[2]);
    addf(3, it.w);
    if (M == kIso) return;
#pragma unroll
    for (int j = 0; j < 6; j++) addf(4 + j, it.A[j]);
    const int rowi[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
#pragma unroll
    for (int c = 0; c < 3; c++) {
        addp(10 + c, it.A[rowi[c][0]], it.x[0]);
        addp(10 + c, it.A[rowi[c][1]], it.x[1]);
        addp(10 + c, it.A[rowi[c][2]], it.x[2]);
    }
    if (M == kQEM) return;
#pragma unroll
    for (int j = 0; j < 6; j++) addf(13 + j, it.T[j]);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        addp(19 + c, it.T[rowi[c][0]], it.x[0]);
        addp(19 + c, it.T[rowi[c][1]], it.x[1]);
        addp(19 + c, it.T[rowi[c][2]], it.x[2]);
    }
}

// Per-cluster evaluation record and energy from the compensated accumulators, in
// float32 and double-float arithmetic only: the incremental path after committed
// moves (float64 throughput on this part is a small fraction of float32).  Same
// formulas as the FP64 full recompute below (ComputeClusterCentroid +
// ComputeClusterEnergy of the metric plugins): m = S / W, residual r = b - A m,
// placement delta = pinv(A) r in float32 (the evaluation kernel's), P = W |delta|^2.
// Writes the record to ev[0 .. Layout<M>::ev) and returns the energy.  anc: the
// anchor vertex of an anchored QEM cluster (null: none) and anc_item its item.
template <int M>
ACVD_DEV double cluster_record_df(const df* a, const RunFlags& fl, float4* ev, const double* anc, int anc_item) {
    const df W = a[3];
    if (!(W.hi > 0.0f)) {
#pragma unroll
        for (int j = 0; j < Layout<M>::ev; j++) ev[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        return 0.0;
    }
    const df m[3] = {df_div(a[0], W), df_div(a[1], W), df_div(a[2], W)};
    ev[0] = make_float4(m[0].hi, m[1].hi, m[2].hi, W.hi);
    // |S|^2 / W = S . m
    const df S2W = df_add(df_add(df_mul(a[0], m[0]), df_mul(a[1], m[1])), df_mul(a[2], m[2]));
    if (M == kIso) return -df_to_d(S2W);
    const df* A = a + 4;    // a00 a01 a02 a11 a12 a22
    const df* b = a + 10;
    if (M == kQEM && anc) {
        // the placed vertex is the anchor p (ComputeClusterCentroid,
        // vtkQEMetricForClustering.h:268-275): E = W |p|^2 - 2 p.S = W |p - m|^2 - |S|^2 / W
        const df q[3] = {df_sub(df_from_d(anc[0]), m[0]), df_sub(df_from_d(anc[1]), m[1]),
                         df_sub(df_from_d(anc[2]), m[2])};
        const df qq = df_add(df_add(df_mul(q[0], q[0]), df_mul(q[1], q[1])), df_mul(q[2], q[2]));
        ev[0] = make_float4((float)anc[0], (float)anc[1], (float)anc[2], W.hi);
        ev[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        ev[2] = make_float4(0.f, 0.f, 0.f, 0.f);
        ev[3] = make_float4(A[0].hi, A[1].hi, A[2].hi, A[3].hi);
        ev[4] = make_float4(A[4].hi, A[5].hi, 1.0f, __int_as_float(anc_item));
        return df_to_d(df_sub(df_mul(W, qq), S2W));
    }
    const int rowi[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    df r[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const df Am = df_add(df_add(df_mul(A[rowi[c][0]], m[0]), df_mul(A[rowi[c][1]], m[1])),
                             df_mul(A[rowi[c][2]], m[2]));
        r[c] = df_sub(b[c], Am);
    }
    float d[3] = {0.f, 0.f, 0.f};
    const bool place = (M == kAniso) || (fl.constrained && fl.level > 0);
    if (place) {
        const float Af[6] = {A[0].hi, A[1].hi, A[2].hi, A[3].hi, A[4].hi, A[5].hi};
        const float rf[3] = {r[0].hi, r[1].hi, r[2].hi};
        pinv_apply<float>(Af, rf, d, fl.level, fl.thr, 8);
    }
    const df dd = df_add(df_add(two_prod(d[0], d[0]), two_prod(d[1], d[1])), two_prod(d[2], d[2]));
    const df P = df_mul(W, dd);
    ev[1] = make_float4(d[0], d[1], d[2], P.hi);
    ev[2] = make_float4(r[0].hi, r[1].hi, r[2].hi, 0.f);
    ev[3] = make_float4(A[0].hi, A[1].hi, A[2].hi, A[3].hi);
    ev[4] = make_float4(A[4].hi, A[5].hi, 0.f, 0.f);
    if (M == kQEM) return df_to_d(df_sub(P, S2W));
    const df* T = a + 13;
    const df* u = a + 19;
    const df c[3] = {df_add_f(m[0], d[0]), df_add_f(m[1], d[1]), df_add_f(m[2], d[2])};
    df Tc[3];
#pragma unroll
    for (int q = 0; q < 3; q++)
        Tc[q] = df_add(df_add(df_mul(T[rowi[q][0]], c[0]), df_mul(T[rowi[q][1]], c[1])), df_mul(T[rowi[q][2]], c[2]));
    const df g[3] = {df_sub(u[0], Tc[0]), df_sub(u[1], Tc[1]), df_sub(u[2], Tc[2])};
    ev[5] = make_float4(T[0].hi, T[1].hi, T[2].hi, T[3].hi);
    ev[6] = make_float4(T[4].hi, T[5].hi, g[0].hi, g[1].hi);
    ev[7] = make_float4(g[2].hi, 0.f, 0.f, 0.f);
    const df cTc = df_add(df_add(df_mul(c[0], Tc[0]), df_mul(c[1], Tc[1])), df_mul(c[2], Tc[2]));
    const df cu = df_add(df_add(df_mul(c[0], u[0]), df_mul(c[1], u[1])), df_mul(c[2], u[2]));
    return df_to_d(df_sub(cTc, df_add(cu, cu)));
}

// Record and energy of cluster k.  FULL: the quadric placement with the
// reference's thresholded pseudo-inverse in FP64 (full recompute, final
// results), the placed vertex in cent[0 .. 2] when that is given (an output vertex of the
// coarse mesh).  Otherwise the double-float path above.
template <int M, bool FULL>
ACVD_DEV void update_cluster(const DevState& st, int k, double* cent = nullptr) {
    const df* a = st.acc + (int64_t)k * Layout<M>::acc;
    float4* ev = st.ev + (int64_t)k * Layout<M>::ev;
    if (!FULL) {
        df al[Layout<M>::acc];
#pragma unroll
        for (int q = 0; q < Layout<M>::acc; q++) al[q] = a[q];
        float4 el[Layout<M>::ev];
        const int ak = anchor_of<M>(st, k);
        const double e =
            cluster_record_df<M>(al, *st.flags, el, ak >= 0 ? st.anchor_xyz + 3 * (int64_t)k : nullptr, ak);
#pragma unroll
        for (int q = 0; q < Layout<M>::ev; q++) ev[q] = el[q];
        st.energy[k] = e;
        return;
    }
    const double W = df_to_d(a[3]);
    const double S[3] = {df_to_d(a[0]), df_to_d(a[1]), df_to_d(a[2])};
    if (!(W > 0.0)) {
        ev[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (M != kIso) for (int j = 1; j < Layout<M>::ev; j++) ev[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        st.energy[k] = 0.0;
        const int ak = anchor_of<M>(st, k);
        for (int j = 0; cent && j < 3; j++) cent[j] = ak >= 0 ? st.anchor_xyz[3 * (int64_t)k + j] : S[j] / W;
        return;
    }
    const double m[3] = {S[0] / W, S[1] / W, S[2] / W};
    if (cent) { cent[0] = m[0]; cent[1] = m[1]; cent[2] = m[2]; }
    ev[0] = make_float4((float)m[0], (float)m[1], (float)m[2], (float)W);
    const double S2W = (S[0] * S[0] + S[1] * S[1] + S[2] * S[2]) / W;
    if (M == kIso) {
        st.energy[k] = -S2W;
        return;
    }
    const RunFlags fl = *st.flags;
    double A[6], b[3];
    for (int j = 0; j < 6; j++) A[j] = df_to_d(a[4 + j]);
    for (int j = 0; j < 3; j++) b[j] = df_to_d(a[10 + j]);
    const int ak = anchor_of<M>(st, k);
    if (M == kQEM && ak >= 0) {
        // anchored: the vertex itself, and ComputeClusterEnergy's expression
        // (vtkQEMetricForClustering.h:194-208) as written
        const double* c = st.anchor_xyz + 3 * (int64_t)k;
        ev[0] = make_float4((float)c[0], (float)c[1], (float)c[2], (float)W);
        ev[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        ev[2] = make_float4(0.f, 0.f, 0.f, 0.f);
        ev[3] = make_float4((float)A[0], (float)A[1], (float)A[2], (float)A[3]);
        ev[4] = make_float4((float)A[4], (float)A[5], 1.0f, __int_as_float(ak));
        st.energy[k] = (c[0] * c[0] + c[1] * c[1] + c[2] * c[2]) * W - 2.0 * (c[0] * S[0] + c[1] * S[1] + c[2] * S[2]);
        if (cent) { cent[0] = c[0]; cent[1] = c[1]; cent[2] = c[2]; }
        return;
    }
    double Am[3];
    sym_mul(A, m, Am);
    const double r[3] = {b[0] - Am[0], b[1] - Am[1], b[2] - Am[2]};
    double d[3] = {0.0, 0.0, 0.0};
    const bool place = (M == kAniso) || (fl.constrained && fl.level > 0);
    if (place) pinv_apply<double>(A, r, d, fl.level, (double)fl.thr, 32);
    if (cent) { cent[0] = m[0] + d[0]; cent[1] = m[1] + d[1]; cent[2] = m[2] + d[2]; }
    const double P = W * (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    ev[1] = make_float4((float)d[0], (float)d[1], (float)d[2], (float)P);
    ev[2] = make_float4((float)r[0], (float)r[1], (float)r[2], 0.f);
    ev[3] = make_float4((float)A[0], (float)A[1], (float)A[2], (float)A[3]);
    if (M == kQEM) {
        ev[4] = make_float4((float)A[4], (float)A[5], 0.f, 0.f);
        st.energy[k] = P - S2W;
        return;
    }
    double T[6], u[3];
    for (int j = 0; j < 6; j++) T[j] = df_to_d(a[13 + j]);
    for (int j = 0; j < 3; j++) u[j] = df_to_d(a[19 + j]);
    const double c[3] = {m[0] + d[0], m[1] + d[1], m[2] + d[2]};
    double Tc[3];
    sym_mul(T, c, Tc);
    const double g[3] = {u[0] - Tc[0], u[1] - Tc[1], u[2] - Tc[2]};
    ev[4] = make_float4((float)A[4], (float)A[5], 0.f, 0.f);
    ev[5] = make_float4((float)T[0], (float)T[1], (float)T[2], (float)T[3]);
    ev[6] = make_float4((float)T[4], (float)T[5], (float)g[0], (float)g[1]);
    ev[7] = make_float4((float)g[2], 0.f, 0.f, 0.f);
    st.energy[k] = (c[0] * Tc[0] + c[1] * Tc[1] + c[2] * Tc[2]) - 2.0 * (c[0] * u[0] + c[1] * u[1] + c[2] * u[2]);
}

// ---------------------------------------------------------------------------
// Committing a step's proposals.  The list's length is known on the device only, and it
// is short next to the class: 5 to 10,000 proposals.  Both commit kernels are a chain of
// dependent loads and one record update per proposal, so they give a proposal to a lane
// (pair) of warp j % W, W the grid's warps: a short list spreads over every SM, one or two
// proposals to a warp.  (With consecutive proposals in one block of 256, a list of 4,800 ran
// on 19 SMs: 8-11 us a launch at the 1024 x 512 torus.)  A proposal's record carries its
// clusters and priority, and is read beside the length, so that only one load separates the
// launch from the clusters' records.
// ---------------------------------------------------------------------------
constexpr int kCommitThreads = 128;
constexpr int kCommitWarps = kCommitThreads / 32;

template <int M>
ACVD_DEV void load_item_now(const DevState& st, int i, ItemRec& it) {
    const float4 a = load_now(st.xw + i);
    it.x[0] = a.x; it.x[1] = a.y; it.x[2] = a.z; it.w = a.w;
    if (M != kIso) {
        const float4 q = load_now(st.qa + i);
        const float2 r = load_now(st.qb + i);
        it.A[0] = q.x; it.A[1] = q.y; it.A[2] = q.z; it.A[3] = q.w; it.A[4] = r.x; it.A[5] = r.y;
    }
    if (M == kAniso) {
        const float4 t = load_now(st.ta + i);
        const float2 u = load_now(st.tb + i);
        it.T[0] = t.x; it.T[1] = t.y; it.T[2] = t.z; it.T[3] = t.w; it.T[4] = u.x; it.T[5] = u.y;
    }
}

// mark_ring with the first 8 neighbours already loaded
ACVD_DEV void mark_ring8(const DevState& st, int i, int4 a, int4 b) {
    if (b.w == -2) {   // a longer ring
        mark_ring(st, i);
        return;
    }
    st.bflag[i] = 1;
    const int nb[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int q = 0; q < 8; q++)
        if (nb[q] >= 0) st.bflag[nb[q]] = 1;
}

// ---------------------------------------------------------------------------
// apply: commit the proposals that hold both claims.  warp / nwarps: this warp's
// position among those that walk the list (count: the class's items, the list's
// capacity).  A lane pair handles one proposal: the even lane the destination
// cluster B, the odd lane the source cluster L; the pair exchanges the two new
// energies and both take the same decision.  The records a winner updates are loaded
// with the claims that decide whether it wins.
// ---------------------------------------------------------------------------
template <int M>
ACVD_DEV void apply_range(const DevState& st, int item0, int64_t count, int color, int round, unsigned warp,
                          unsigned nwarps) {
    constexpr int NA = Layout<M>::acc;
    const unsigned lane = threadIdx.x & 31u;
    const int role = (int)(lane & 1u);
    const unsigned pair_mask = 3u << (lane & ~1u);
    unsigned j = warp + (lane >> 1) * nwarps;
    int4 e = j < (unsigned)count ? load_now(st.cand_list + j) : make_int4(0, -1, 0, 0);
    const unsigned n = st.cand_count[color];
    const unsigned epoch = (unsigned)(color * kRounds + round);
    unsigned won_total = 0;
    while (j < n) {
        const unsigned at = j;
        const int idx = e.x, B = e.y, L = e.z;
        const unsigned prio = (unsigned)e.w;
        j += 16u * nwarps;
        if (j < n) e = st.cand_list[j];
        if (B < 0) continue;                     // committed or dropped in an earlier round
        const int i = item0 + idx;
        if (!ACVD_VALID(st, B < st.k && L >= 0 && L <= st.k && L == st.label[i])) continue;
        const unsigned long long key = make_claim(epoch, prio, (unsigned)idx);
        const int C = role && L < st.k ? L : B;  // the cluster of this lane
        const unsigned long long claim_b = st.claim[B], claim_l = st.claim[L < st.k ? L : B];
        ItemRec it;
        load_item_now<M>(st, i, it);
        const int4 ra = load_now(st.ring8 + 2 * (int64_t)i), rb = load_now(st.ring8 + 2 * (int64_t)i + 1);
        df* aC = st.acc + (int64_t)C * NA;
        const double e_mine = load_now(st.energy + C);
        const int size = load_now(st.size + C);
        df nC[NA];
#pragma unroll
        for (int q = 0; q < NA; q++) {
            const float2 v = load_now(reinterpret_cast<const float2*>(aC) + q);
            nC[q] = {v.x, v.y};
        }
        if (claim_b != key || (L < st.k && claim_l != key)) continue;
        __syncwarp(pair_mask);                   // both lanes have read the claims and the proposal
        const int now = st.sweep->sweep;
        if (L >= st.k) {
            // unassigned item joining a cluster: always committed
            if (role == 0) {
                st.claim[B] = claim_taken(color);   // taken for the rest of this step
                st.cand_list[at].y = -1;
                won_total++;
                st.label[i] = B;
                mark_ring8(st, i, ra, rb);
                st.size[B] = size + 1;
                st.stamp[B] = now;
                accumulate_item<M>(st.acc + (int64_t)B * Layout<M>::acc, it, 1.0f);
                update_cluster<M, false>(st, B);
            }
            continue;
        }
        // the new records are built in registers and written only if the tracked
        // energy of the pair strictly decreases (the float32 test can disagree with
        // the updated records, e.g. when a pseudo-inverse eigenvalue sits at the
        // threshold), so the minimisation descends monotonically and terminates
        float4* eC = st.ev + (int64_t)C * Layout<M>::ev;
        const RunFlags fl = *st.flags;
        accumulate_item<M>(nC, it, role ? -1.0f : 1.0f);
        float4 rC[Layout<M>::ev];
        const int anc = anchor_of<M>(st, C);
        const double en_mine =
            cluster_record_df<M>(nC, fl, rC, anc >= 0 ? st.anchor_xyz + 3 * (int64_t)C : nullptr, anc);
        const double e_other = __shfl_xor_sync(pair_mask, e_mine, 1);
        const double en_other = __shfl_xor_sync(pair_mask, en_mine, 1);
        // energy of the pair in the order B + L on both lanes
        const double e_old = role ? e_other + e_mine : e_mine + e_other;
        const double e_new = role ? en_other + en_mine : en_mine + en_other;
        if (e_new < e_old) {
#pragma unroll
            for (int q = 0; q < NA; q++) aC[q] = nC[q];
#pragma unroll
            for (int q = 0; q < Layout<M>::ev; q++) eC[q] = rC[q];
            st.energy[C] = en_mine;
            st.size[C] = size + (role ? -1 : 1);
            st.stamp[C] = now;
            st.claim[C] = claim_taken(color);   // taken for the rest of this step
            if (role == 0) {
                won_total++;
                st.label[i] = B;
                mark_ring8(st, i, ra, rb);
                st.cand_list[at].y = -1;
            }
        } else {
            st.claim[C] = claim_taken(color);
            if (role == 0) {
                st.cand_list[at].y = -1;
                atomicAdd(ctr(st.counters, kCntReverted), 1ull);
            }
        }
    }
    // every thread of the grid reaches this point: warp-aggregated count
    warp_count(ctr(st.counters, kCntMoves), won_total);
}

template <int M>
__global__ void __launch_bounds__(kCommitThreads) apply_kernel(DevState st, int item0, int64_t count, int color,
                                                               int round) {
    apply_range<M>(st, item0, count, color, round, blockIdx.x * kCommitWarps + (threadIdx.x >> 5),
                   gridDim.x * kCommitWarps);
}

// Next matching round of a step: a proposal whose two clusters were not touched
// by this step's commits still carries an exact energy change and claims again
// with a newer epoch; one that lost a cluster to a commit is dropped (its item
// is evaluated again next sweep).
ACVD_DEV void reclaim_range(const DevState& st, int item0, int color, int round, unsigned gtid, unsigned gstride) {
    const unsigned n = st.cand_count[color];
    const unsigned epoch = (unsigned)(color * kRounds + round);
    for (unsigned j = gtid; j < n; j += gstride) {
        const int4 e = st.cand_list[j];
        const int B = e.y, L = e.z;
        if (B < 0) continue;
        const unsigned long long taken = claim_taken(color);
        if (st.claim[B] == taken || (L < st.k && st.claim[L] == taken)) {
            st.cand_list[j].y = -1;
            continue;
        }
        const unsigned long long key = make_claim(epoch, (unsigned)e.w, (unsigned)e.x);
        if (L < st.k) atomicMin(&st.claim[L], key);
        atomicMin(&st.claim[B], key);
    }
}

__global__ void reclaim_kernel(DevState st, int item0, int color, int round) {
    reclaim_range(st, item0, color, round, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// ---------------------------------------------------------------------------
// relaxed step (phases without the connectivity constraint): every proposal of
// the colour class commits at once, except that a cluster is never emptied.
// Items of one colour are never adjacent.  The committed moves' contributions are
// summed per cluster in 64-bit fixed point -- exact, so the atomics' order does
// not matter -- and folded into the compensated accumulators by fx_finalize.
// ---------------------------------------------------------------------------

// item contribution j (the accumulate_item components) as a double-float: the
// products w x, A x and T x are formed exactly (TwoProd) and summed compensated
template <int M>
ACVD_DEV df contrib_df(const ItemRec& it, int j) {
    const int rowi[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    if (j < 3) return two_prod(it.w, it.x[j]);
    if (j == 3) return df_make(it.w);
    if (j < 10) return df_make(it.A[j - 4]);
    if (j < 13) {
        const int c = j - 10;
        return df_add(df_add(two_prod(it.A[rowi[c][0]], it.x[0]), two_prod(it.A[rowi[c][1]], it.x[1])),
                      two_prod(it.A[rowi[c][2]], it.x[2]));
    }
    if (j < 19) return df_make(it.T[j - 13]);
    const int c = j - 19;
    return df_add(df_add(two_prod(it.T[rowi[c][0]], it.x[0]), two_prod(it.T[rowi[c][1]], it.x[1])),
                  two_prod(it.T[rowi[c][2]], it.x[2]));
}

// Fixed-point units of component q: the scale is a power of two 2^e held as two
// float factors (x, y; inverses in z, w), so both conversions are exact scalings.
ACVD_DEV long long to_fixed(df v, float4 p) {
    const float h = __fmul_rn(__fmul_rn(v.hi, p.x), p.y);
    const float l = __fmul_rn(__fmul_rn(v.lo, p.x), p.y);
    return __float2ll_rn(h) + __float2ll_rn(l);
}

ACVD_DEV df from_fixed(long long d, float4 p) {
    const float h = __ll2float_rn(d);
    const float l = __ll2float_rn(d - __float2ll_rn(h));
    return df_renorm(__fmul_rn(__fmul_rn(h, p.z), p.w), __fmul_rn(__fmul_rn(l, p.z), p.w));
}

// The fixed-point sums of a proposal, added by a group of lanes: its contributions are
// staged in shared memory (lane p's proposal in s_v[p]), then GROUP lanes add the
// components of one cluster side by side, so that the atomics of a cluster fall in one or
// two 128-byte lines instead of one each.
template <int M>
struct CommitStage {
    static constexpr int NA = Layout<M>::acc;
    static constexpr int GROUP = M == kIso ? 4 : (M == kQEM ? 16 : 32);
    alignas(16) long long v[32][NA];
    int cl[32][2];   // destination and source; -1: none
};

template <int M>
ACVD_DEV void relaxed_commit_range(const DevState& st, int item0, int64_t count, int color, unsigned warp,
                                   unsigned nwarps, CommitStage<M>& s) {
    constexpr int NA = Layout<M>::acc;
    constexpr int GROUP = CommitStage<M>::GROUP;
    const unsigned lane = threadIdx.x & 31u;
    // up to 32 proposals per warp: lane l takes proposal warp + l * nwarps; longer lists go
    // by runs of 32 consecutive proposals, whose items lie near one another
    unsigned j = warp + lane * nwarps;
    int4 e = j < (unsigned)count ? load_now(st.cand_list + j) : make_int4(0, 0, 0, 0);
    const unsigned n = st.cand_count[color];
    const bool runs = n > 32u * nwarps;
    const unsigned step = 32u * nwarps;
    unsigned first = warp;                        // lane 0's proposal
    if (runs) {
        first = warp * 32u;
        j = first + lane;
        if (j < n) e = st.cand_list[j];
    }
    unsigned won = 0;
    const int now = st.sweep->sweep;
    for (; first < n; first += step, j += step) {
        if (j >= step && j < n) e = st.cand_list[j];
        bool live = j < n;
        const int i = item0 + e.x, B = e.y, L = e.z;
        if (live && !ACVD_VALID(st, B >= 0 && B < st.k && L >= 0 && L <= st.k && L == st.label[i])) live = false;
        const bool from = live && L < st.k;
        int4 ra = make_int4(-1, -1, -1, -1), rb = ra;
        int size = 0, out = 0;
        ItemRec it;
        if (live) {
            load_item_now<M>(st, i, it);
            ra = load_now(st.ring8 + 2 * (int64_t)i);
            rb = load_now(st.ring8 + 2 * (int64_t)i + 1);
            if (from) {
                size = load_now(st.size + L);
                out = load_now(st.out_cnt + L);
            }
        }
        // sizes are untouched until fx_finalize: a cluster whose every member would
        // leave keeps them all
        if (from && size - out < 1) live = false;
        s.cl[lane][0] = live ? B : -1;
        s.cl[lane][1] = live && from ? L : -1;
        if (live) {
            won++;
            st.label[i] = B;
            mark_ring8(st, i, ra, rb);
            atomicAdd(&st.in_done[B], 1);
            st.stamp[B] = now;
            if (from) {
                atomicAdd(&st.out_done[L], 1);
                st.stamp[L] = now;
            }
#pragma unroll
            for (int q = 0; q < NA; q++) s.v[lane][q] = to_fixed(contrib_df<M>(it, q), st.fx_pow[q]);
        }
        const unsigned have = 32u - (unsigned)__clz((int)__ballot_sync(kFull, live));   // lanes in use
        __syncwarp();
        const unsigned g = lane / GROUP, q = lane % GROUP;
        for (unsigned t = g; t < 2u * have; t += 32u / GROUP) {
            const unsigned p = t >> 1, side = t & 1u;
            const int c = s.cl[p][side];
            if (c < 0 || q >= (unsigned)NA) continue;
            const long long v = s.v[p][q];
            atomicAdd((unsigned long long*)&st.fx_delta[(int64_t)c * NA + q], (unsigned long long)(side ? -v : v));
        }
        __syncwarp();
    }
    warp_count(ctr(st.counters, kCntMoves), won);
}

template <int M>
__global__ void __launch_bounds__(kCommitThreads) relaxed_commit_kernel(DevState st, int item0, int64_t count,
                                                                        int color) {
    __shared__ CommitStage<M> s[kCommitWarps];
    relaxed_commit_range<M>(st, item0, count, color, blockIdx.x * kCommitWarps + (threadIdx.x >> 5),
                            gridDim.x * kCommitWarps, s[threadIdx.x >> 5]);
}

// Finalisation: 32 consecutive clusters to a warp.  Their sums lie in one stretch of memory,
// which the lanes read and write side by side, a component each, by way of shared memory; the
// record of a cluster is then one lane's work.  (A lane that walked its own cluster's sums
// touched 32 lines with every load: 19.0 us a launch against 13.6 now on the anisotropic
// 2047 x 1801 heightfield, 6.4 against 6.2 on the 1024 x 512 quadric torus, where the chain of
// one record is what is left.)  At least 6 blocks to an SM: the anisotropic record takes 208
// registers otherwise, and the 2047 x 1801 solve was 1 % slower; at 8 and 10 it spills.
template <int M>
ACVD_DEV void fx_finalize_range(const DevState& st, unsigned warp, unsigned nwarps, CommitStage<M>& s) {
    constexpr int NA = Layout<M>::acc, NE = Layout<M>::ev;
    const unsigned lane = threadIdx.x & 31u;
    float2* sums = reinterpret_cast<float2*>(&s.v[0][0]);
    float4* recs = reinterpret_cast<float4*>(&s.v[0][0]);
    static_assert(sizeof(s.v) >= 32 * NE * sizeof(float4), "the records take the sums' place");
    for (int64_t k0 = 32 * (int64_t)warp; k0 < st.k; k0 += 32 * (int64_t)nwarps) {
        const int64_t k = k0 + lane;
        int in = 0, out = 0;
        if (k < st.k) {
            in = st.in_done[k];
            out = st.out_done[k];
            st.out_cnt[k] = 0;
        }
        const bool touched = in != 0 || out != 0;
        const unsigned mask = __ballot_sync(kFull, touched);
        if (!mask) continue;
        df* a = st.acc + k0 * NA;
        long long* d = st.fx_delta + k0 * NA;
        // every load first (independent), then the arithmetic, then the stores
        df al[NA];
        long long dl[NA];
#pragma unroll
        for (int t = 0; t < NA; t++) {
            const unsigned e = lane + 32u * t;
            al[t] = df_make(0.0f);
            dl[t] = 0;
            if (mask >> (e / NA) & 1u) {
                al[t] = a[e];
                dl[t] = d[e];
            }
        }
        if (touched) {
            st.in_done[k] = 0;
            st.out_done[k] = 0;
            st.size[k] += in - out;
        }
#pragma unroll
        for (int t = 0; t < NA; t++) {
            const unsigned e = lane + 32u * t;
            const df v = df_add(al[t], from_fixed(dl[t], st.fx_pow[e % NA]));
            sums[e] = make_float2(v.hi, v.lo);
            if (mask >> (e / NA) & 1u) {
                a[e] = v;
                d[e] = 0;
            }
        }
        __syncwarp();
        float4 el[NE];
        if (touched) {
            df mine[NA];
#pragma unroll
            for (int q = 0; q < NA; q++) {
                const float2 v = sums[lane * NA + q];
                mine[q] = {v.x, v.y};
            }
            const int ak = anchor_of<M>(st, k);
            st.energy[k] = cluster_record_df<M>(mine, *st.flags, el, ak >= 0 ? st.anchor_xyz + 3 * k : nullptr, ak);
        }
        __syncwarp();
        if (touched) {
#pragma unroll
            for (int q = 0; q < NE; q++) recs[lane * NE + q] = el[q];
        }
        __syncwarp();
        float4* ev = st.ev + k0 * NE;
#pragma unroll
        for (int t = 0; t < NE; t++) {
            const unsigned e = lane + 32u * t;
            if (mask >> (e / NE) & 1u) ev[e] = recs[e];
        }
        __syncwarp();
    }
}

constexpr int kFinalizeThreads = 64;   // small blocks: every SM gets some

template <int M>
__global__ void __launch_bounds__(kFinalizeThreads, 6) fx_finalize_kernel(DevState st) {
    __shared__ CommitStage<M> s[kFinalizeThreads / 32];
    const unsigned w = threadIdx.x >> 5;
    fx_finalize_range<M>(st, blockIdx.x * (kFinalizeThreads / 32) + w, gridDim.x * (kFinalizeThreads / 32), s[w]);
}

// per accumulator component: the largest |contribution| over the items (as float
// bits, monotone for non-negative values), from which the fixed-point scales follow
template <int M>
__global__ void __launch_bounds__(256) fx_maxabs_kernel(DevState st, unsigned* __restrict__ maxbits) {
    constexpr int NA = Layout<M>::acc;
    __shared__ unsigned s_mx[NA];
    if (threadIdx.x < NA) s_mx[threadIdx.x] = 0u;
    __syncthreads();
    float mx[NA];
#pragma unroll
    for (int q = 0; q < NA; q++) mx[q] = 0.f;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < st.n; i += (int64_t)gridDim.x * blockDim.x) {
        ItemRec it;
        load_item<M>(st, (int)i, it);
#pragma unroll
        for (int q = 0; q < NA; q++) mx[q] = fmaxf(mx[q], fabsf(contrib_df<M>(it, q).hi));
    }
    // warp, then block maxima; one global atomic per block and component
#pragma unroll
    for (int q = 0; q < NA; q++) {
        float v = mx[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
        if ((threadIdx.x & 31) == 0) atomicMax(&s_mx[q], __float_as_uint(v));
    }
    __syncthreads();
    if (threadIdx.x < NA) atomicMax(&maxbits[threadIdx.x], s_mx[threadIdx.x]);
}

// The start of a sweep, by one block: the sweep counter, the proposal and work-list counts
// and this sweep's moves.
ACVD_DEV void start_sweep(const DevState& st, int ncolors) {
    const int t = threadIdx.x;
    if (t == 0) st.sweep->sweep += 1;
    for (int j = t; j < ncolors; j += blockDim.x) st.cand_count[j] = 0u;
    if (st.work_count)
        for (int j = t; j < ncolors * kWorkStripes; j += blockDim.x) st.work_count[j] = 0u;
    for (int j = t; j < kStripes; j += blockDim.x) st.counters[j * kNumCounters + kCntMoves] = 0ull;
}

ACVD_DEV void reset_claims(const DevState& st) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k <= st.k; k += (int64_t)gridDim.x * blockDim.x)
        st.claim[k] = ~0ull;
}

__global__ void begin_sweep_kernel(DevState st, int ncolors, int claims) {
    if (blockIdx.x == 0) start_sweep(st, ncolors);
    if (claims) reset_claims(st);
}

// ---------------------------------------------------------------------------
// Persistent sweep kernel: the sweeps between two convergence events in one
// cooperative launch.  Each phase of a sweep (claim reset, evaluation, commit
// steps, finalisation, energy sum) is a grid-stride pass over the same device
// functions as the per-phase kernels, in the same order, with a grid barrier
// between phases.  The operations of the float32 energy tests are named one by one
// (dot3 and its like), so its clusterings are the per-phase schedule's bit for bit.  Block 0
// takes the host loop's after-sweep decisions (relaxed -> exact switch, move
// count, convergence test, sweep cap); the other blocks read them after the
// sweep's last barrier.
// ---------------------------------------------------------------------------
constexpr long long kBarrierSpins = 1ll << 24;   // about 1-2 s of 64 ns naps

ACVD_DEV unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

ACVD_DEV unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Every thread of every block calls it.  Writes made by any thread before the
// barrier are visible to every thread after it (release fence before the
// arrival, acquire load of the generation, fence after).  A wait that runs out
// of spins sets the error flag; every later call then returns false and the
// kernel ends.
ACVD_DEV bool grid_barrier(GridBar* b, long long max_spins = kBarrierSpins) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned g = ld_acquire(&b->gen);
        __threadfence();
        const unsigned arrived = atomicAdd(&b->count, 1u) + 1u;
        int ok = 1;
        if (arrived == gridDim.x) {
            atomicExch(&b->count, 0u);
            __threadfence();
            atomicAdd(&b->gen, 1u);
        } else {
            long long spins = 0;
            while (ld_acquire(&b->gen) == g) {
                if (*(volatile int*)&b->err) {   // another block gave up already
                    ok = 0;
                    break;
                }
                if (++spins > max_spins) {
                    atomicExch(&b->err, 1);
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
        if (*(volatile int*)&b->err) ok = 0;
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Self-check of the barrier's wait limit: block 1 never arrives, so block 0's wait
// runs out after max_spins naps, sets the error flag and returns.
__global__ void barrier_wait_limit_kernel(GridBar* bar, long long max_spins) {
    if (blockIdx.x == 1) return;
    grid_barrier(bar, max_spins);
}

cudaError_t launch_barrier_wait_limit(GridBar* bar, long long max_spins, cudaStream_t s) {
    ++g_launches;
    barrier_wait_limit_kernel<<<2, 32, 0, s>>>(bar, max_spins);
    return cudaGetLastError();
}

// The barrier of a thread-block cluster: every CTA's earlier writes are visible after it.
ACVD_DEV void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// CLUSTER: the grid is one thread-block cluster and its hardware barrier takes the grid
// barrier's place (a.bar is not used).  Small meshes run this way: see kClusterCtas.
template <int M, bool CLUSTER>
__global__ void __launch_bounds__(256, CLUSTER ? 1 : 2) sweep_run_kernel(SweepRun a) {
    const DevState& st = a.st;
    const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned gstride = gridDim.x * blockDim.x;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    volatile LoopState* vls = a.ls;
    extern __shared__ __align__(16) char stage_mem[];   // 8 warps' commit stages
    CommitStage<M>* stage = reinterpret_cast<CommitStage<M>*>(stage_mem);
    auto barrier = [&]() {
        if (!CLUSTER) return grid_barrier(a.bar);
        cluster_barrier();
        return true;
    };
    for (int run = 0;; run++) {
        const bool relaxed = vls->relaxed_ok && !st.flags->connexity;
        if (blockIdx.x == 0) start_sweep(st, a.nclasses);
        if (!relaxed) reset_claims(st);   // once per sweep: a taken cluster keeps a marker per step
        if (!barrier()) return;
        for (int c = 0; c < a.nclasses; c++) {
            const long long o0 = a.off[c];
            const int64_t cnt = a.off[c + 1] - o0;
            if (cnt == 0) continue;
            const int item0 = (int)o0;
            const unsigned long long t0 = lead ? global_ns() : 0ull;
            const int per = spread_items<256>(cnt, gridDim.x);
            const int64_t ntiles = (cnt + per - 1) / per;
            for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x)
                eval_tile<M>(st, item0, cnt, c, relaxed ? 0 : 1, t, per);
            if (!barrier()) return;
            if (lead) a.ls->eval_ns += global_ns() - t0;
            if (relaxed) {
                relaxed_commit_range<M>(st, item0, cnt, c, gtid >> 5, gstride >> 5, stage[threadIdx.x >> 5]);
                if (!barrier()) return;
                // neighbouring warps of clusters on different SMs
                fx_finalize_range<M>(st, (threadIdx.x >> 5) * gridDim.x + blockIdx.x, gstride >> 5,
                                     stage[threadIdx.x >> 5]);
                if (!barrier()) return;
            } else {
                apply_range<M>(st, item0, cnt, c, 0, gtid >> 5, gstride >> 5);
                if (!barrier()) return;
                for (int r = 1; r < a.match_rounds; r++) {
                    reclaim_range(st, item0, c, r, gtid, gstride);
                    if (!barrier()) return;
                    apply_range<M>(st, item0, cnt, c, r, gtid >> 5, gstride >> 5);
                    if (!barrier()) return;
                }
            }
        }
        double e_now = 0.0;
        if (relaxed) {
            // the energy after the sweep, in sum_f64's tree
            const int64_t per = (int64_t)kSumThreads * kSumPer;
            int64_t nb = ((int64_t)st.k + per - 1) / per;
            if (nb < 1) nb = 1;
            double* pa = a.esum;
            double* pb = a.esum + nb + 1;
            for (int64_t ch = blockIdx.x; ch < nb; ch += gridDim.x) sum_f64_chunk(st.energy, st.k, ch, pa);
            if (!barrier()) return;
            const double* cur = pa;
            int64_t m = nb;
            double* dst = pb;
            double* other = pa;
            while (m > 1) {
                const int64_t mb = (m + per - 1) / per;
                for (int64_t ch = blockIdx.x; ch < mb; ch += gridDim.x) sum_f64_chunk(cur, m, ch, dst);
                if (!barrier()) return;
                cur = dst;
                m = mb;
                double* t = dst;
                dst = other;
                other = t;
            }
            if (lead) e_now = *(volatile const double*)cur;
        }
        if (lead) {
            LoopState* L = a.ls;
            long long mods = 0;
            for (int q = 0; q < kStripes; q++)
                mods += (long long)*(volatile unsigned long long*)(st.counters + q * kNumCounters + kCntMoves);
            if (relaxed) {
                if (L->have_prev && !(e_now < L->e_prev)) L->relaxed_ok = 0;
                L->e_prev = e_now;
                L->have_prev = 1;
                L->relaxed_run += 1;
            }
            if (L->sweeps < a.log_cap) {
                SweepLog& g = a.log[L->sweeps];
                g.moves = mods;
                g.energy = e_now;
                g.relaxed = relaxed ? 1 : 0;
            }
            L->sweeps += 1;
            L->run += 1;
            L->moves += mods;
            L->last_moves = mods;
            if (mods == 0 || L->sweeps > L->max_loops || (mods <= L->early / 1000 && L->convergences <= 1))
                L->status = 1;
        }
        if (!barrier()) return;
        if (vls->status != 0 || run + 1 >= a.max_run) return;
    }
}

// ---------------------------------------------------------------------------
// Device-side sweep loop: a CUDA-graph WHILE node repeats an IF / ELSE of the
// relaxed and the exact sweep, and the kernel that ends a sweep takes, on the device,
// the decisions the host loop takes after each sweep (the same ones as block 0 of
// the persistent kernel), so the sweeps between two convergence events run without
// returning to the host.
//
// One kernel ends a sweep and starts the next (each launch of a graph costs 2-3.5 us here,
// whatever it does; ending a relaxed sweep with two launches of the energy sum, a copy, a
// decision and a start kernel took 12 us of 180 at the 1024 x 512 torus): every block
// resets its part of the claims; a relaxed sweep's blocks each add a chunk of the energies,
// and the last one to finish adds the chunks (sum_f64's tree, so the same bits), decides
// and, if the loop goes on, starts the next sweep.
// ---------------------------------------------------------------------------
constexpr int kEndThreads = 256;
static_assert(kEndThreads == kSumThreads, "a block of sweep_end_kernel adds one chunk of sum_f64");

__global__ void __launch_bounds__(kEndThreads) loop_start_kernel(DevState st, LoopState* L, int ncolors,
                                                                 cudaGraphConditionalHandle h_loop,
                                                                 cudaGraphConditionalHandle h_mode) {
    reset_claims(st);
    if (blockIdx.x != 0) return;
    start_sweep(st, ncolors);
    if (threadIdx.x == 0) {
        L->done = 0u;
        cudaGraphSetConditional(h_loop, 1u);
        cudaGraphSetConditional(h_mode, (L->relaxed_ok && !st.flags->connexity) ? 1u : 0u);
    }
}

// partial: a double per chunk of 2,048 clusters (the grid of a relaxed sweep's end), and one more
template <bool RELAXED>
__global__ void __launch_bounds__(kEndThreads) sweep_end_kernel(DevState st, LoopState* L, double* partial,
                                                                int ncolors, cudaGraphConditionalHandle h_loop,
                                                                cudaGraphConditionalHandle h_mode) {
    __shared__ int s_last, s_go;
    reset_claims(st);
    double e = 0.0;
    if (RELAXED) {
        sum_f64_chunk(st.energy, st.k, blockIdx.x, partial);
        if (threadIdx.x == 0) {
            __threadfence();
            s_last = atomicAdd(&L->done, 1u) == gridDim.x - 1u;
            __threadfence();
        }
        __syncthreads();
        if (!s_last) return;
        if (gridDim.x > 1) sum_f64_chunk(partial, gridDim.x, 0, partial + gridDim.x);
        if (threadIdx.x == 0) e = gridDim.x > 1 ? partial[gridDim.x] : partial[0];   // its own write
    } else if (blockIdx.x != 0) {
        return;
    }
    if (threadIdx.x < 32) {
        static_assert(kStripes == 32, "a lane per stripe");
        unsigned long long v = st.counters[threadIdx.x * kNumCounters + kCntMoves];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
        const long long mods = (long long)v;
        if (threadIdx.x == 0) {
            if (RELAXED) {
                if (L->have_prev && !(e < L->e_prev)) L->relaxed_ok = 0;
                L->e_prev = e;
                L->have_prev = 1;
                L->relaxed_run += 1;
                L->done = 0u;
            }
            L->sweeps += 1;
            L->run += 1;
            L->moves += mods;
            L->last_moves = mods;
            const bool stop =
                mods == 0 || L->sweeps > L->max_loops || (mods <= L->early / 1000 && L->convergences <= 1);
            if (stop) L->status = 1;
            s_go = !stop;
            cudaGraphSetConditional(h_loop, stop ? 0u : 1u);
            cudaGraphSetConditional(h_mode, (L->relaxed_ok && !st.flags->connexity) ? 1u : 0u);
        }
    }
    __syncthreads();
    if (s_go) start_sweep(st, ncolors);
}

// ---------------------------------------------------------------------------
// full recompute of the accumulators: items sorted by cluster, one warp per
// cluster, fixed-order butterfly reduction (deterministic).  20,000 clusters of 26 items
// took 33.5 us with 65 double-float additions per lane in the butterfly, 18.5 us with
// its components spread over the lanes.
// ---------------------------------------------------------------------------
__global__ void cluster_keys_kernel(DevState st, uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st.n) return;
    int L = st.label[i];
    if (L < 0 || L > st.k) L = st.k;
    keys[i] = (uint32_t)L;
    vals[i] = (uint32_t)i;
}

// Sum over a warp of C components per lane, in the order of the butterfly that adds every
// component on every lane (lane and lane ^ 16, then ^ 8, ...; the lower lane's value
// first), with half the components handed to the partner at each step: 7 + 4 + 2 + 1 + 1
// additions per lane for 13 components instead of 65.  Component `at` of the total ends in
// acc[0] of the one lane with have > 0.
template <int C, int O>
ACVD_DEV void warp_sum_spread(df* acc, int lane, int& at, int& have) {
    constexpr int H = (C + 1) / 2;
    const bool up = (lane & O) != 0;
#pragma unroll
    for (int j = 0; j < H; j++) {
        const df lower = acc[j], upper = H + j < C ? acc[H + j] : df{0.f, 0.f};
        df t;
        t.hi = __shfl_xor_sync(kFull, up ? lower.hi : upper.hi, O);
        t.lo = __shfl_xor_sync(kFull, up ? lower.lo : upper.lo, O);
        acc[j] = up ? df_add(t, upper) : df_add(lower, t);
    }
    at += up ? H : 0;
    have = up ? have - H : min(have, H);
    if constexpr (O > 1) warp_sum_spread<H, O / 2>(acc, lane, at, have);
}

template <int M>
__global__ void __launch_bounds__(256) reduce_clusters_kernel(DevState st, const uint32_t* __restrict__ sorted,
                                                              const uint32_t* __restrict__ seg_off) {
    constexpr int NA = Layout<M>::acc;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= st.k) return;
    const uint32_t off = seg_off[w], cnt = seg_off[w + 1] - off;
    df acc[NA];
#pragma unroll
    for (int j = 0; j < NA; j++) acc[j] = {0.f, 0.f};
    for (uint32_t j = lane; j < cnt; j += 32) {
        ItemRec it;
        load_item<M>(st, (int)sorted[off + j], it);
        accumulate_item<M>(acc, it, 1.0f);
    }
    int at = 0, have = NA;
    warp_sum_spread<NA, 16>(acc, lane, at, have);
    if (have > 0) st.acc[w * NA + at] = acc[0];
    if (lane == 0) st.size[w] = (int)cnt;
}

// The FP64 decompositions of the quadric metrics bound it (2 FP64 lanes per SM and cycle):
// one warp per block, so that the SMs differ by one warp at most (20,000 clusters in 157
// blocks of 128 put a second block on 5 of 152 SMs and took 63 us; 46 us so).  What
// acvd_get_clusters returns is written along: the placed vertex needs no second
// decomposition.
constexpr int kUpdateThreads = 32;

template <int M>
__global__ void __launch_bounds__(kUpdateThreads) update_all_kernel(DevState st, ClusterOut out) {
    const int64_t k = (int64_t)blockIdx.x * kUpdateThreads + threadIdx.x;
    if (k >= st.k) return;
    double c[3];
    update_cluster<M, true>(st, (int)k, out.centroid ? c : nullptr);
    const df* a = st.acc + k * Layout<M>::acc;
    if (out.centroid)
        for (int j = 0; j < 3; j++) out.centroid[3 * k + j] = c[j];
    if (out.S)
        for (int j = 0; j < 3; j++) out.S[3 * k + j] = df_to_d(a[j]);
    if (out.W) out.W[k] = df_to_d(a[3]);
    if (out.Q) {
        // the reference's compact quadric: A entries and -b in slots 3, 6, 8
        double q[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        if (M != kIso) {
            q[0] = df_to_d(a[4]); q[1] = df_to_d(a[5]); q[2] = df_to_d(a[6]); q[3] = -df_to_d(a[10]);
            q[4] = df_to_d(a[7]); q[5] = df_to_d(a[8]); q[6] = -df_to_d(a[11]); q[7] = df_to_d(a[9]);
            q[8] = -df_to_d(a[12]);
        }
        for (int j = 0; j < 9; j++) out.Q[9 * k + j] = q[j];
    }
}

// ---------------------------------------------------------------------------
// connectivity cleaning: min-id label propagation over same-cluster edges with
// pointer jumping; each cluster keeps its largest component (ties -> the one
// containing the smallest item id), the rest become unassigned
// ---------------------------------------------------------------------------
// Components carry the smallest ORIGINAL vertex id among their items (the
// tie-break between equally large components follows the reference's item
// order, not the internal one); inv maps such an id back to its item.
__global__ void comp_init_kernel(DevState st, int* __restrict__ comp) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st.n) return;
    comp[i] = st.label[i] < st.k ? st.orig[i] : -1;
}

__global__ void comp_step_kernel(DevState st, int* __restrict__ comp) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st.n) return;
    const int L = st.label[i];
    if (L >= st.k) return;
    const int cur = comp[i];
    int m = cur;
    for (int p = st.row[i]; p < st.row[i + 1]; p++) {
        const int j = st.col[p];
        if (st.label[j] == L) m = min(m, comp[j]);
    }
    for (int hop = 0; hop < 64; hop++) {
        const int mm = comp[st.inv[m]];
        if (mm >= m) break;
        m = mm;
    }
    if (m < cur) {
        comp[i] = m;
        atomicAdd(ctr(st.counters, kCntChanged), 1ull);
    }
}

// The same components by union-find in one pass over the ring CSR (the result equals
// the propagation's: every component ends as the smallest original id of its items).
// parent[] links items; a root is linked only under a root of smaller original id, so
// ids decrease along every chain and each set's root is its smallest-id item.  Concurrent
// links race through atomicCAS on the root's slot; a failed CAS retries from the new
// roots.  Finding a root halves the path (writes of an ancestor, benign under races).

__device__ __forceinline__ int uf_root(int* parent, int x) {
    for (;;) {
        const int p = parent[x];
        if (p == x) return x;
        const int g = parent[p];
        if (g != p) parent[x] = g;
        x = p;
    }
}

__global__ void uf_init_kernel(DevState st, int* __restrict__ parent) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < st.n) parent[i] = (int)i;
}

__global__ void uf_link_kernel(DevState st, int* parent, int tries) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st.n) return;
    const int L = st.label[i];
    if (L >= st.k) return;
    unsigned gave_up = 0;
    for (int p = st.row[i]; p < st.row[i + 1]; p++) {
        const int j = st.col[p];
        if (j <= (int)i || st.label[j] != L) continue;   // each same-cluster edge once
        int a = uf_root(parent, (int)i), b = uf_root(parent, j);
        int t = 0;
        for (; t < tries && a != b; t++) {
            if (st.orig[a] > st.orig[b]) {
                const int x = a;
                a = b;
                b = x;
            }
            // b (larger original id) goes under a
            const int old = atomicCAS(&parent[b], b, a);
            if (old == b) break;
            a = uf_root(parent, a);
            b = uf_root(parent, old);
        }
        gave_up += a != b && t == tries;
    }
    if (gave_up) atomicAdd(ctr(st.counters, kCntChanged), (unsigned long long)gave_up);
}

__global__ void uf_flatten_kernel(DevState st, int* parent, int* __restrict__ comp) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st.n) return;
    comp[i] = st.label[i] < st.k ? st.orig[uf_root(parent, (int)i)] : -1;
}

__global__ void comp_size_kernel(DevState st, const int* __restrict__ comp, int* __restrict__ csize) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st.n) return;
    const int L = st.label[i];
    if (L >= st.k) return;
    // the component holding the cluster's fixed item outweighs any other
    // (vtkUniformClustering.h:439-447)
    const bool fixed_item = L < st.nfixed && st.fixed[L] == (int)i;
    atomicAdd(&csize[comp[i]], fixed_item ? 1000000000 : 1);
}

__global__ void comp_best_kernel(DevState st, const int* __restrict__ comp, const int* __restrict__ csize,
                                 unsigned long long* __restrict__ best) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st.n) return;
    const int L = st.label[i];
    const int o = st.orig[i];
    if (L >= st.k || comp[i] != o) return;
    const unsigned long long key = ((unsigned long long)(unsigned)csize[o] << 32) | (0xffffffffull - (uint32_t)o);
    atomicMax(&best[L], key);
}

__global__ void comp_reset_kernel(DevState st, const int* __restrict__ comp,
                                  const unsigned long long* __restrict__ best, int* __restrict__ multi) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st.n) return;
    const int L = st.label[i];
    if (L >= st.k) return;
    const uint32_t root = 0xffffffffu - (uint32_t)(best[L] & 0xffffffffull);
    if ((uint32_t)comp[i] != root) {
        st.label[i] = st.k;
        if (atomicExch(&multi[L], 1) == 0) atomicAdd(ctr(st.counters, kCntDisconnected), 1ull);
    }
}

// ---------------------------------------------------------------------------
// hole filling, one colour class at a time: an unassigned item joins the
// cluster of its first assigned ring neighbour (ring order); with the
// connectivity constraint on, only if the unassigned ring members stay
// connected without it (the reference applies the same local test to the null
// cluster, Common/vtkUniformClustering.h:606-607)
// ---------------------------------------------------------------------------
// The rounds run over lists of the unassigned items: fill_collect_kernel lists them
// per colour class (class c at list[off[c] ...], items being numbered by class); a
// round then runs the classes in order over their lists.  Items of one class are never
// ring neighbours, so the order inside a class list does not matter.
__global__ void fill_collect_kernel(DevState st, const int64_t* __restrict__ off, int ncolors, int* __restrict__ list,
                                    unsigned* __restrict__ cnt) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st.n || st.label[i] < st.k) return;
    int c = 0;
    while (c + 1 < ncolors && off[c + 1] <= i) c++;
    list[off[c] + atomicAdd(&cnt[c], 1u)] = (int)i;
}

__global__ void fill_list_kernel(DevState st, const int* __restrict__ list, const unsigned* __restrict__ cnt) {
    const unsigned n = *cnt;
    unsigned done = 0;
    for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const int i = list[j];
        if (st.label[i] < st.k) continue;   // filled in an earlier round
        const int p0 = st.row[i], p1 = st.row[i + 1];
        int B = -1;
        for (int p = p0; p < p1 && B < 0; p++) {
            const int l = st.label[st.col[p]];
            if (l < st.k) B = l;
        }
        if (B >= 0 && (!st.flags->connexity || ring_connected(st, p0, p1, st.k))) {
            st.label[i] = B;
            done++;
        }
    }
    warp_count(ctr(st.counters, kCntAssigned), done);
}

// Every round over short lists in one block: the classes in order with a block barrier
// between them (the items of one class read only labels of other classes), rounds until
// one assigns nothing.  *err is set when the round bound runs out.
constexpr int kFillRounds = 1 << 20;

__global__ void __launch_bounds__(1024) fill_block_kernel(DevState st, const int* __restrict__ list,
                                                          const int64_t* __restrict__ off, int ncolors,
                                                          const unsigned* __restrict__ cnt, unsigned* err,
                                                          unsigned max_items) {
    __shared__ int s_changed;
    // lists longer than max_items: *err = 2 and nothing done (the host runs the rounds
    // one launch per class instead)
    unsigned total = 0;
    for (int c = 0; c < ncolors; c++) total += cnt[c];
    if (total > max_items) {
        if (threadIdx.x == 0) *err = 2u;
        return;
    }
    unsigned done = 0;
    int round = 0;
    for (; round < kFillRounds; round++) {
        if (threadIdx.x == 0) s_changed = 0;
        __syncthreads();
        for (int c = 0; c < ncolors; c++) {
            const int* lc = list + off[c];
            const unsigned n = cnt[c];
            for (unsigned j = threadIdx.x; j < n; j += blockDim.x) {
                const int i = lc[j];
                if (st.label[i] < st.k) continue;
                const int p0 = st.row[i], p1 = st.row[i + 1];
                int B = -1;
                for (int p = p0; p < p1 && B < 0; p++) {
                    const int l = st.label[st.col[p]];
                    if (l < st.k) B = l;
                }
                if (B >= 0 && (!st.flags->connexity || ring_connected(st, p0, p1, st.k))) {
                    st.label[i] = B;
                    done++;
                    s_changed = 1;
                }
            }
            __syncthreads();   // the next class reads this class's labels
        }
        const bool again = s_changed != 0;
        __syncthreads();
        if (!again) break;
    }
    if (round == kFillRounds && threadIdx.x == 0) *err = 1u;
    warp_count(ctr(st.counters, kCntAssigned), done);
}

__global__ void compact_kernel(const uint32_t* __restrict__ flags, const uint32_t* __restrict__ pos, int64_t n,
                               int* __restrict__ out) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n && flags[j]) out[pos[j]] = (int)j;
}

// ---------------------------------------------------------------------------
// ACVD's quadric post-placement (DiscreteRemeshing/Examples/ACVD.cxx:217-291), FP64.
// (1) per vertex: the unweighted plane quadrics (vtkQuadricTools::AddTriangleQuadric,
// FullQuadric = false, Common/vtkQuadricTools.cxx:56-79) of its faces, in increasing
// face id; (2) per cluster: the sum over its items in increasing vertex id, then the
// output vertex moved by ComputeRepresentativePoint (.cxx:83-177): P + pinv(A)(b - A P),
// A = (Q0 Q1 Q2 / Q4 Q5 / Q7), b = -(Q3, Q6, Q8), `level` singular values above
// 1e-3 of the largest.
// ---------------------------------------------------------------------------
__global__ void vertex_quadric_kernel(const double* __restrict__ xyz, const int* __restrict__ tri,
                                      const uint32_t* __restrict__ vf_row, const uint32_t* __restrict__ vf_face,
                                      int64_t nv, double* __restrict__ qv) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    double q[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t t = vf_row[v]; t < vf_row[v + 1]; t++) {
        const int f = (int)vf_face[t];
        const int a = tri[3 * f], b = tri[3 * f + 1], c = tri[3 * f + 2];
        const double x1[3] = {xyz[3 * a], xyz[3 * a + 1], xyz[3 * a + 2]};
        const double e1[3] = {xyz[3 * b] - x1[0], xyz[3 * b + 1] - x1[1], xyz[3 * b + 2] - x1[2]};
        const double e2[3] = {xyz[3 * c] - x1[0], xyz[3 * c + 1] - x1[1], xyz[3 * c + 2] - x1[2]};
        double n[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
        const double len = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
        if (len > 0.0) { n[0] /= len; n[1] /= len; n[2] /= len; } else { n[0] = n[1] = n[2] = 0.0; }
        const double d = -(n[0] * x1[0] + n[1] * x1[1] + n[2] * x1[2]);
        q[0] += n[0] * n[0]; q[1] += n[0] * n[1]; q[2] += n[0] * n[2]; q[3] += n[0] * d;
        q[4] += n[1] * n[1]; q[5] += n[1] * n[2]; q[6] += n[1] * d;
        q[7] += n[2] * n[2]; q[8] += n[2] * d;
    }
    for (int j = 0; j < 9; j++) qv[9 * v + j] = q[j];
}

__global__ void first_nonempty_kernel(const uint32_t* __restrict__ seg_off, int k, int* __restrict__ first) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    // most clusters hold items: one atomic per warp
    const unsigned some = __ballot_sync(kFull, c < k && seg_off[c + 1] > seg_off[c]);
    if (some && (threadIdx.x & 31) == __ffs(some) - 1) atomicMin(first, (int)c);
}

// start: the output vertices (3K, the metric's cluster centroids); sorted: items
// by cluster (original ids), cluster c's at seg_off[c] .. seg_off[c + 1]
__global__ void post_place_kernel(const double* __restrict__ qv, const uint32_t* __restrict__ sorted,
                                  const uint32_t* __restrict__ seg_off, const int* __restrict__ first,
                                  const double* __restrict__ start, int k, int level, double* __restrict__ out) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= k) return;
    double q[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const uint32_t s0 = seg_off[c], s1 = seg_off[c + 1];
    for (uint32_t t = s0; t < s1; t++) {
        const uint32_t v = sorted[t];
        for (int j = 0; j < 9; j++) q[j] += qv[9 * (int64_t)v + j];
    }
    const int64_t src = s1 > s0 ? c : (int64_t)(*first < k ? *first : 0);
    const double P[3] = {start[3 * src], start[3 * src + 1], start[3 * src + 2]};
    const double A[6] = {q[0], q[1], q[2], q[4], q[5], q[7]};
    double AP[3];
    sym_mul(A, P, AP);
    const double r[3] = {-q[3] - AP[0], -q[6] - AP[1], -q[8] - AP[2]};
    double d[3];
    pinv_apply<double>(A, r, d, level, 1e-3, 32);
    out[3 * c] = P[0] + d[0];
    out[3 * c + 1] = P[1] + d[1];
    out[3 * c + 2] = P[2] + d[2];
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static inline unsigned nblk(int64_t n, int b = 256) { return (unsigned)((n + b - 1) / b); }

#define ACVD_DISPATCH(metric, KERNEL, grid, block, stream, ...)                         \
    do {                                                                                \
        ++g_launches;                                                                   \
        if ((metric) == kIso) KERNEL<kIso><<<grid, block, 0, stream>>>(__VA_ARGS__);     \
        else if ((metric) == kQEM) KERNEL<kQEM><<<grid, block, 0, stream>>>(__VA_ARGS__); \
        else KERNEL<kAniso><<<grid, block, 0, stream>>>(__VA_ARGS__);                     \
    } while (0)

static int64_t sm_count();

// (metric, blocks per SM) -> the instantiation; blocks outside 3..5 take `dflt`
#define ACVD_DISPATCH_B(metric, blocks, dflt, KERNEL, grid, block, stream, ...)                               \
    do {                                                                                                    \
        ++g_launches;                                                                                       \
        const int b_ = ((blocks) >= 3 && (blocks) <= 5) ? (blocks) : (dflt);                                \
        if ((metric) == kIso) {                                                                             \
            if (b_ == 3) KERNEL<kIso, 3><<<grid, block, 0, stream>>>(__VA_ARGS__);                          \
            else if (b_ == 4) KERNEL<kIso, 4><<<grid, block, 0, stream>>>(__VA_ARGS__);                     \
            else KERNEL<kIso, 5><<<grid, block, 0, stream>>>(__VA_ARGS__);                                  \
        } else if ((metric) == kQEM) {                                                                      \
            if (b_ == 3) KERNEL<kQEM, 3><<<grid, block, 0, stream>>>(__VA_ARGS__);                          \
            else if (b_ == 4) KERNEL<kQEM, 4><<<grid, block, 0, stream>>>(__VA_ARGS__);                     \
            else KERNEL<kQEM, 5><<<grid, block, 0, stream>>>(__VA_ARGS__);                                  \
        } else {                                                                                            \
            if (b_ == 3) KERNEL<kAniso, 3><<<grid, block, 0, stream>>>(__VA_ARGS__);                        \
            else if (b_ == 4) KERNEL<kAniso, 4><<<grid, block, 0, stream>>>(__VA_ARGS__);                   \
            else KERNEL<kAniso, 5><<<grid, block, 0, stream>>>(__VA_ARGS__);                                \
        }                                                                                                   \
    } while (0)

// metric -> the 128-thread instantiation with B = 4 (the threads per SM of four
// 256-thread blocks)
#define ACVD_DISPATCH_128(metric, KERNEL, grid, stream, ...)                                                    \
    do {                                                                                                        \
        ++g_launches;                                                                                           \
        if ((metric) == kIso) KERNEL<kIso, 4, 128><<<grid, 128, 0, stream>>>(__VA_ARGS__);                      \
        else if ((metric) == kQEM) KERNEL<kQEM, 4, 128><<<grid, 128, 0, stream>>>(__VA_ARGS__);                 \
        else KERNEL<kAniso, 4, 128><<<grid, 128, 0, stream>>>(__VA_ARGS__);                                     \
    } while (0)

// Resident blocks per SM of the 128-thread eval_list_kernel instantiation
template <int M>
static int list_occupancy_128() {
    int nb = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, eval_list_kernel<M, 4, 128>, 128, 0);
    return (e == cudaSuccess && nb > 0) ? nb : 1;
}

static int eval_list_blocks_per_sm_128(int metric) {
    if (metric == kIso) return list_occupancy_128<kIso>();
    if (metric == kQEM) return list_occupancy_128<kQEM>();
    return list_occupancy_128<kAniso>();
}

// Resident blocks per SM of an eval_list_kernel instantiation (its grid strides over
// the work list).
template <int M, int B>
static int list_occupancy() {
    int nb = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, eval_list_kernel<M, B>, 256, 0);
    return (e == cudaSuccess && nb > 0) ? nb : 1;
}

static int eval_list_blocks_per_sm(int metric, int blocks) {
    const int b = (blocks >= 3 && blocks <= 5) ? blocks : kDefaultListBlocks;
    if (metric == kIso)
        return b == 3 ? list_occupancy<kIso, 3>() : b == 4 ? list_occupancy<kIso, 4>() : list_occupancy<kIso, 5>();
    if (metric == kQEM)
        return b == 3 ? list_occupancy<kQEM, 3>() : b == 4 ? list_occupancy<kQEM, 4>() : list_occupancy<kQEM, 5>();
    return b == 3 ? list_occupancy<kAniso, 3>() : b == 4 ? list_occupancy<kAniso, 4>() : list_occupancy<kAniso, 5>();
}

// Blocks per SM of screen_kernel (its grid strides over the class's tiles).
static int screen_blocks_per_sm(int metric) {
    int nb = 0;
    cudaError_t e;
    if (metric == kIso) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, screen_kernel<kIso>, 256, 0);
    else if (metric == kQEM) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, screen_kernel<kQEM>, 256, 0);
    else e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, screen_kernel<kAniso>, 256, 0);
    return (e == cudaSuccess && nb > 0) ? nb : 1;
}

cudaError_t launch_eval(int metric, const DevState& st, int item0, int64_t count, int color, bool claims, bool split,
                        int blocks, int threads, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    if (threads == 128) {
        // 128-thread blocks, as many threads per SM as four blocks of 256
        if (!split) {
            const int per = spread_items<128>(count, 8 * sm_count());
            ACVD_DISPATCH_128(metric, eval_kernel, nblk(count, per), s, st, item0, count, color, claims ? 1 : 0, per);
            return cudaGetLastError();
        }
        const unsigned sgrid =
            (unsigned)std::min<int64_t>(nblk(count, kScreenTile), sm_count() * screen_blocks_per_sm(metric));
        ACVD_DISPATCH(metric, screen_kernel, sgrid, 256, s, st, item0, count, color, st.work, st.work_count);
        const int64_t tiles = kWorkStripes * (work_cap(count) / 128);
        const unsigned grid = (unsigned)std::min<int64_t>(tiles, sm_count() * eval_list_blocks_per_sm_128(metric));
        ACVD_DISPATCH_128(metric, eval_list_kernel, grid, s, st, item0, count, color, claims ? 1 : 0, (const int*)st.work, (const unsigned*)st.work_count);
        return cudaGetLastError();
    }
    if (!split) {
        const int dflt = default_eval_blocks(metric), b = blocks >= 3 && blocks <= 5 ? blocks : dflt;
        const int per = spread_items<256>(count, b * sm_count());
        ACVD_DISPATCH_B(metric, blocks, dflt, eval_kernel, nblk(count, per), 256, s, st, item0, count, color,
                        claims ? 1 : 0, per);
        return cudaGetLastError();
    }
    const unsigned sgrid = (unsigned)std::min<int64_t>(nblk(count, kScreenTile), sm_count() * screen_blocks_per_sm(metric));
    ACVD_DISPATCH(metric, screen_kernel, sgrid, 256, s, st, item0, count, color, st.work, st.work_count);
    const int64_t tiles = kWorkStripes * (work_cap(count) / 256);
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, sm_count() * eval_list_blocks_per_sm(metric, blocks));
    ACVD_DISPATCH_B(metric, blocks, kDefaultListBlocks, eval_list_kernel, grid, 256, s, st, item0, count, color,
                    claims ? 1 : 0, (const int*)st.work, (const unsigned*)st.work_count);
    return cudaGetLastError();
}

static int64_t sm_count() {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

static unsigned list_grid(int64_t count) {
    // the proposal count is only known on the device: a grid of 2 blocks per SM
    // strides over the list
    return (unsigned)std::min<int64_t>(nblk(count), 2 * sm_count());
}

// Blocks of the commit kernels: a warp for every 32 items of the class, at most 16 warps
// to an SM (2,432 on a 152-SM GB300; more proposals than that take further lanes of them)
static unsigned commit_grid(int64_t count) {
    return (unsigned)std::min<int64_t>(nblk(count, kCommitThreads), 4 * sm_count());
}

cudaError_t launch_apply(int metric, const DevState& st, int item0, int64_t count, int color, int round,
                         cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    ACVD_DISPATCH(metric, apply_kernel, commit_grid(count), kCommitThreads, s, st, item0, count, color, round);
    return cudaGetLastError();
}

cudaError_t launch_reclaim(const DevState& st, int item0, int64_t count, int color, int round, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    ++g_launches;
    reclaim_kernel<<<list_grid(count), 256, 0, s>>>(st, item0, color, round);
    return cudaGetLastError();
}

cudaError_t launch_relaxed_step(int metric, const DevState& st, int item0, int64_t count, int color,
                                cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    ACVD_DISPATCH(metric, relaxed_commit_kernel, commit_grid(count), kCommitThreads, s, st, item0, count, color);
    ACVD_DISPATCH(metric, fx_finalize_kernel, nblk(st.k, kFinalizeThreads), kFinalizeThreads, s, st);
    return cudaGetLastError();
}

cudaError_t launch_fx_scale(int metric, const DevState& st, unsigned* maxbits, cudaStream_t s) {
    if (st.n == 0) return cudaSuccess;
    ACVD_DISPATCH(metric, fx_maxabs_kernel, list_grid(st.n), 256, s, st, maxbits);
    return cudaGetLastError();
}

// blocks that reset the claims of k clusters
static unsigned claim_grid(int64_t k) { return (unsigned)std::min<int64_t>(nblk(k + 1, kEndThreads), 2 * sm_count()); }

cudaError_t launch_begin_sweep(const DevState& st, int ncolors, bool claims, cudaStream_t s) {
    ++g_launches;
    begin_sweep_kernel<<<claims ? claim_grid(st.k) : 1u, kEndThreads, 0, s>>>(st, ncolors, claims ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_loop_start(const DevState& st, LoopState* ls, int ncolors, cudaGraphConditionalHandle h_loop,
                              cudaGraphConditionalHandle h_mode, cudaStream_t s) {
    ++g_launches;
    loop_start_kernel<<<claim_grid(st.k), kEndThreads, 0, s>>>(st, ls, ncolors, h_loop, h_mode);
    return cudaGetLastError();
}

int64_t sweep_end_partials(int64_t k) {
    const int64_t per = (int64_t)kSumThreads * kSumPer;
    return std::max<int64_t>(1, (k + per - 1) / per) + 1;
}

cudaError_t launch_sweep_end(const DevState& st, LoopState* ls, double* partial, int ncolors, bool relaxed,
                             cudaGraphConditionalHandle h_loop, cudaGraphConditionalHandle h_mode, cudaStream_t s) {
    ++g_launches;
    if (relaxed)
        sweep_end_kernel<true><<<(unsigned)(sweep_end_partials(st.k) - 1), kEndThreads, 0, s>>>(st, ls, partial, ncolors,
                                                                                                h_loop, h_mode);
    else
        sweep_end_kernel<false><<<claim_grid(st.k), kEndThreads, 0, s>>>(st, ls, partial, ncolors, h_loop, h_mode);
    return cudaGetLastError();
}

template <bool CLUSTER>
static const void* sweep_run_fn(int metric) {
    return metric == kIso ? (const void*)sweep_run_kernel<kIso, CLUSTER>
         : metric == kQEM ? (const void*)sweep_run_kernel<kQEM, CLUSTER>
                          : (const void*)sweep_run_kernel<kAniso, CLUSTER>;
}

static size_t sweep_run_stage_bytes(int metric) {
    return 8 * (metric == kIso ? sizeof(CommitStage<kIso>)
              : metric == kQEM ? sizeof(CommitStage<kQEM>) : sizeof(CommitStage<kAniso>));
}

int sweep_run_blocks_per_sm(int metric) {
    int nb = 0;
    cudaError_t e;
    const int sm = (int)sweep_run_stage_bytes(metric);
    const void* fn = sweep_run_fn<false>(metric);
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, 256, sm);
    return e == cudaSuccess ? nb : 0;
}

cudaError_t launch_sweep_run(int metric, const SweepRun& a, int grid, cudaStream_t s) {
    ++g_launches;
    SweepRun arg = a;
    void* args[] = {(void*)&arg};
    return cudaLaunchCooperativeKernel(sweep_run_fn<false>(metric), dim3((unsigned)grid), dim3(256), args,
                                       sweep_run_stage_bytes(metric), s);
}

// One cluster of kClusterCtas CTAs of 256 threads, one to an SM.
static void cluster_config(int metric, cudaStream_t s, cudaLaunchConfig_t& cfg, cudaLaunchAttribute& at) {
    at = cudaLaunchAttribute{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kClusterCtas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(kClusterCtas);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = sweep_run_stage_bytes(metric);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
}

bool sweep_cluster_available(int metric) {
    const void* fn = sweep_run_fn<true>(metric);
    const int sm = (int)sweep_run_stage_bytes(metric);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    cluster_config(metric, nullptr, cfg, at);
    int n = 0;
    const bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) == cudaSuccess &&
                    cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n > 0;
    if (!ok) cudaGetLastError();
    return ok;
}

cudaError_t launch_sweep_cluster(int metric, const SweepRun& a, cudaStream_t s) {
    ++g_launches;
    SweepRun arg = a;
    void* args[] = {(void*)&arg};
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    cluster_config(metric, s, cfg, at);
    return cudaLaunchKernelExC(&cfg, sweep_run_fn<true>(metric), args);
}

cudaError_t launch_update_all(int metric, const DevState& st, const ClusterOut& out, cudaStream_t s) {
    if (st.k == 0) return cudaSuccess;
    ACVD_DISPATCH(metric, update_all_kernel, nblk(st.k, kUpdateThreads), kUpdateThreads, s, st, out);
    return cudaGetLastError();
}

cudaError_t launch_cluster_keys(const DevState& st, uint32_t* keys, uint32_t* vals, cudaStream_t s) {
    if (st.n == 0) return cudaSuccess;
    ++g_launches;
    cluster_keys_kernel<<<nblk(st.n), 256, 0, s>>>(st, keys, vals);
    return cudaGetLastError();
}

cudaError_t launch_reduce_clusters(int metric, const DevState& st, const uint32_t* sorted_items,
                                   const uint32_t* seg_off, cudaStream_t s) {
    if (st.k == 0) return cudaSuccess;
    ACVD_DISPATCH(metric, reduce_clusters_kernel, nblk((int64_t)st.k * 32), 256, s, st, sorted_items, seg_off);
    return cudaGetLastError();
}

cudaError_t launch_comp_init(const DevState& st, int* comp, cudaStream_t s) {
    ++g_launches;
    comp_init_kernel<<<nblk(st.n), 256, 0, s>>>(st, comp);
    return cudaGetLastError();
}

cudaError_t launch_comp_step(const DevState& st, int* comp, cudaStream_t s) {
    ++g_launches;
    comp_step_kernel<<<nblk(st.n), 256, 0, s>>>(st, comp);
    return cudaGetLastError();
}

cudaError_t launch_comp_union(const DevState& st, int* comp, int* parent, int tries, cudaStream_t s) {
    g_launches += 3;
    uf_init_kernel<<<nblk(st.n), 256, 0, s>>>(st, parent);
    uf_link_kernel<<<nblk(st.n), 256, 0, s>>>(st, parent, tries);
    uf_flatten_kernel<<<nblk(st.n), 256, 0, s>>>(st, parent, comp);
    return cudaGetLastError();
}

cudaError_t launch_comp_finish(const DevState& st, const int* comp, int* csize, unsigned long long* best,
                               int* multi, cudaStream_t s) {
    ++g_launches;
    comp_size_kernel<<<nblk(st.n), 256, 0, s>>>(st, comp, csize);
    ++g_launches;
    comp_best_kernel<<<nblk(st.n), 256, 0, s>>>(st, comp, csize, best);
    ++g_launches;
    comp_reset_kernel<<<nblk(st.n), 256, 0, s>>>(st, comp, best, multi);
    return cudaGetLastError();
}


cudaError_t launch_fill_collect(const DevState& st, const int64_t* off, int ncolors, int* list, unsigned* cnt,
                                cudaStream_t s) {
    ++g_launches;
    fill_collect_kernel<<<nblk(st.n), 256, 0, s>>>(st, off, ncolors, list, cnt);
    return cudaGetLastError();
}

cudaError_t launch_fill_list(const DevState& st, const int* list, const unsigned* cnt, int64_t cap, cudaStream_t s) {
    if (cap == 0) return cudaSuccess;
    ++g_launches;
    const unsigned grid = (unsigned)std::min<int64_t>(nblk(cap), 2 * sm_count());
    fill_list_kernel<<<grid, 256, 0, s>>>(st, list, cnt);
    return cudaGetLastError();
}

cudaError_t launch_fill_block(const DevState& st, const int* list, const int64_t* off, int ncolors,
                              const unsigned* cnt, unsigned* err, unsigned max_items, cudaStream_t s) {
    ++g_launches;
    fill_block_kernel<<<1, 1024, 0, s>>>(st, list, off, ncolors, cnt, err, max_items);
    return cudaGetLastError();
}

cudaError_t launch_compact(const uint32_t* flags, const uint32_t* pos, int64_t n, int* out, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    ++g_launches;
    compact_kernel<<<nblk(n), 256, 0, s>>>(flags, pos, n, out);
    return cudaGetLastError();
}

}  // namespace acvd

namespace acvd {

cudaError_t launch_vertex_quadrics(const double* xyz, const int* tri, const uint32_t* vf_row, const uint32_t* vf_face,
                                   int64_t nv, double* qv, cudaStream_t s) {
    if (nv == 0) return cudaSuccess;
    ++g_launches;
    vertex_quadric_kernel<<<nblk(nv), 256, 0, s>>>(xyz, tri, vf_row, vf_face, nv, qv);
    return cudaGetLastError();
}

cudaError_t launch_post_place(const double* qv, const uint32_t* sorted, const uint32_t* seg_off, int* first,
                              const double* start, int k, int level, double* out, cudaStream_t s) {
    if (k == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(first, 0x7f, sizeof(int), s);
    if (e != cudaSuccess) return e;
    g_launches += 2;
    first_nonempty_kernel<<<nblk(k), 256, 0, s>>>(seg_off, k, first);
    post_place_kernel<<<nblk(k, 128), 128, 0, s>>>(qv, sorted, seg_off, first, start, k, level, out);
    return cudaGetLastError();
}

}  // namespace acvd
