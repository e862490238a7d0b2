// sopb_resident.cuh — the replica-resident Langevin step kernel.
//
// A cluster of one to sixteen CTAs owns one job for a whole launch of
// `nsteps` steps.  Coordinates, Hybrid Taus states and the temperature
// accumulator sit in shared memory; every updater of the reference loop
// (indentation tip, force-ramp cantilever, possible pairs, temperature reset,
// Verlet pairlist, heating) runs inside the kernel at its step, so there is
// no host round trip and no launch per step (the reference launches 4-6
// kernels per step and copies all coordinates to the host every `stride`
// steps for pulling, src/Potentials/pulling.cu:152-165).
//
// Neighbour lists.  The possible-pairs list of a job is a bitmask over its
// beads (n <= 2048, so at most 64 words a row), with bonded/native
// exclusions as a precomputed bitmask.  The Verlet list is kept per pair of
// consecutive beads (2p, 2p + 1), as one row of u16 entries in three
// sections: the partners of both beads, of the first alone, of the second
// alone, each in increasing j (86 % of the entries' two slots are used on
// globular chains of 100 to 2000 beads).  One gather of a partner's
// coordinates then serves both beads, which halves the shared-memory
// wavefronts of the pair loop, and a rebuild reads and writes one row where
// two were.  The rows of a launch sit in shared memory, allocated one after
// another; rows that do not fit stay in global memory.
//
// One step is two phases.  Forces: a group of lanes takes a pair of beads,
// strides over the shared section together, then each half of the group goes
// on with one bead's own section and its covalent and native entries;
// xor-shuffles combine the partial forces.  Warps that have no more pairs
// draw the step's noise, 32 beads at a time, which fills the phase's end.
// Integration: one thread per bead moves the bead.  A bead's arithmetic
// depends only on the job and on lpb, never on which group or CTA computed it
// or on where its row is kept.
//
// Clusters.  With C CTAs per job, CTA r owns the pairs [r P / C, (r + 1) P / C):
// their lists, forces and integration.  Every CTA holds all coordinates,
// double-buffered by step parity; after integrating, it sends its beads' new
// coordinates to the other CTAs with st.async, whose byte counts complete the
// receivers' mbarriers (one per parity), so a step costs one message latency
// and no cluster barrier.  A sender that runs ahead writes the other buffer
// and the other mbarrier, and it can run no more than one step ahead, since
// it needs this CTA's coordinates too.  Scalar updaters are computed by every
// CTA from the same coordinates; CTA 0 writes them back and logs.
#pragma once

#include "sopb_device.cuh"

namespace sopb {

// shared memory per bead that every resident job holds: coordinates, RNG
// state, force and noise (16 B each), temperature (4 B), pulling flag (1 B)
// and the pair's row header (8 B per two beads)
constexpr int kResidentSmemPerBead = 73;

__host__ __device__ inline int job_pairs(int n) { return (n + 1) >> 1; }
// CTA r's first pair of C CTAs
__host__ __device__ inline int pair_begin(int n, int r, int C) { return (int)((int64_t)job_pairs(n) * r / C); }
// Most beads a CTA of C owns.
__host__ __device__ inline int local_beads_max(int n, int C) {
    const int m = 2 * ((job_pairs(n) + C - 1) / C);
    return m < n ? m : n;
}

// Shared-memory layout of a CTA of a resident launch (byte offsets, 16-B
// aligned arrays).  The coordinates are followed by two far-away dummy beads
// (the second bead of the last pair of an odd job; the beads of a lane group
// past the last pair), the headers of rows and of bonded maps by a warp's
// worth of empty ones, so that a group past the end needs no tests.  The bonded maps of the
// CTA's beads (covalent and native rows with parameters) are copied in when
// `bonded` is set; the Verlet rows take `cache` u16 entries.
constexpr int kClusterBlock = 512;   // largest CTA of a cluster
constexpr int kPadPairs = 16;   // a warp's pairs with two lanes each
struct ResidentLayout {
    size_t x, F, N, sd, nat_par, cov_par, bh, hd, order, xref, Ts, nat_j, flags, nbr, total;
};
__host__ __device__ inline size_t align16(size_t v) { return (v + 15) & ~(size_t)15; }
__host__ __device__ inline ResidentLayout resident_layout(int n, int C, int ncov, int nnat, int bonded, int cache) {
    ResidentLayout L;
    const size_t b = bonded ? 1 : 0, cl = C > 1 ? 1 : 0, nb = (size_t)local_beads_max(n, C);
    size_t o = 0;
    L.x = o;        o = align16(o + (1 + cl) * (size_t)(n + 2) * 16);
    L.F = o;        o = align16(o + nb * 16);
    L.N = o;        o = align16(o + cl * nb * 16);
    L.sd = o;       o = align16(o + nb * 16);
    L.nat_par = o;  o = align16(o + b * (size_t)nnat * 8);
    L.cov_par = o;  o = align16(o + b * (size_t)ncov * 8);
    L.bh = o;       o = align16(o + b * (nb + 2 * kPadPairs) * 8);
    L.hd = o;       o = align16(o + ((nb + 1) / 2 + kPadPairs) * 8);
    L.order = o;    o = align16(o + (1 - cl) * ((nb + 1) / 2 + kPadPairs) * 2);
    L.xref = o;     o = align16(o + cl * (size_t)n * 16);
    L.Ts = o;       o = align16(o + nb * 4);
    L.nat_j = o;    o = align16(o + b * (size_t)nnat * 2);
    L.flags = o;    o = align16(o + nb);
    L.nbr = o;      o = align16(o + (size_t)cache * 2);
    L.total = o;
    return L;
}

struct StepScalars {
    float var;
    float pullF[3];
    float cant[3];
    IndentGeom ig;
    float chip[3];
    float V, dx;
    float fav[4];
    int32_t err;
    int32_t nr_valid;   // the job's near list is usable (written back at the end)
    uint32_t log_head;  // event-log rows appended (written back at the end)
    float plane_displ, plane_cant;   // pulling plane (written back at the end)
};

// Cooperative copy of a job descriptor into shared memory (read by every
// thread as a broadcast instead of per-thread register copies).
template <int BLOCK>
__device__ __forceinline__ void load_job(JobDev& dst, const JobDev* src) {
    static_assert(sizeof(JobDev) % 4 == 0, "JobDev must be word sized");
    const int* s = reinterpret_cast<const int*>(src);
    int* d = reinterpret_cast<int*>(&dst);
    for (int w = threadIdx.x; w < (int)(sizeof(JobDev) / 4); w += BLOCK) d[w] = s[w];
}

__device__ __forceinline__ void load_job(JobDev& dst, const JobDev* src) {
    const int* s = reinterpret_cast<const int*>(src);
    int* d = reinterpret_cast<int*>(&dst);
    for (int w = threadIdx.x; w < (int)(sizeof(JobDev) / 4); w += blockDim.x) d[w] = s[w];
}

// Sum over a lane group; `mask` names the lanes taking part (the whole
// warp, or just the group when groups of a warp run independently).
__device__ __forceinline__ float3 group_reduce(float3 f, int lpb, unsigned mask = 0xffffffffu) {
    for (int o = lpb >> 1; o > 0; o >>= 1) {
        f.x += __shfl_xor_sync(mask, f.x, o);
        f.y += __shfl_xor_sync(mask, f.y, o);
        f.z += __shfl_xor_sync(mask, f.z, o);
    }
    return f;
}

// Covalent then native terms of bead i, strided over lanes
// (the reference sums its kernels' contributions in this order,
// src/gsop.cu:80-85).
__device__ __forceinline__ void bonded_partial(const JobDev& J, const float4* __restrict__ xs, int i, float4 xi, int l, int lpb,
                                               float3& f) {
    const int c0 = J.cov_off[i], c1 = J.cov_off[i + 1];
    const int n0 = J.nat_off[i], n1 = J.nat_off[i + 1];
    for (int k = c0 + l; k < c1; k += lpb) fene_term(xi, xs[J.cov_j[k]], J.cov_r0[k], J.ks, J.R2, f);
    for (int k = n0 + l; k < n1; k += lpb) native_term(xi, xs[J.nat_j[k]], J.nat_par[k], f);
}

// Verlet-pair terms of bead i from its index row, lane l of lpb taking
// entries l, l+lpb, ... in that order.  Four entries are fetched per
// iteration so four gathers are in flight; the per-lane summation order is
// unchanged.
template <typename Idx>
__device__ __forceinline__ void pair_run(const JobDev& J, const float4* __restrict__ xs, const Idx* __restrict__ r,
                                         int cnt, float4 xi, int l, int lpb, float3& f) {
    const float c8 = J.c8, cut2 = J.cut2;
    int k = l;
    for (; k + 3 * lpb < cnt; k += 4 * lpb) {
        const int j0 = r[k], j1 = r[k + lpb], j2 = r[k + 2 * lpb], j3 = r[k + 3 * lpb];
        const float4 x0 = xs[j0], x1 = xs[j1], x2 = xs[j2], x3 = xs[j3];
        pair_term(xi, x0, c8, cut2, f);
        pair_term(xi, x1, c8, cut2, f);
        pair_term(xi, x2, c8, cut2, f);
        pair_term(xi, x3, c8, cut2, f);
    }
    for (; k < cnt; k += lpb) pair_term(xi, xs[r[k]], c8, cut2, f);
}

// ---- Verlet rows of bead pairs -------------------------------------------------
// A CTA's part of a job during a launch: its pairs [p0, p1) and beads
// [b0, b1), the coordinates of all beads, and the rows in shared memory.
// `hd` null (a list rebuild outside a launch): headers and rows go to global
// memory.
struct PartView {
    int p0, p1, b0, b1;
    int rank, C;
    uint2* hd;          // row headers (RowHead), by local pair
    uint16_t* nbr;      // rows
    int cap;            // entries of nbr
    uint16_t* order;    // local pairs, longest row first (null in a cluster)
    float4* xref;       // coordinates the near list was built at, all beads
    const int64_t* gave_up;   // step at which a chunk of steps that some CTA gave up ends
};

// A pair's row: `start` in the CTA's shared rows, or kRowGlobal for the
// pair's row in global memory; nf entries for both beads, then n0 for the
// first alone, then n1 for the second.  An entry is 16 j, the byte offset of
// the partner's coordinates.
constexpr uint32_t kRowGlobal = 0xfffffu;
struct RowHead {
    uint32_t start;
    int nf, n0, n1;
};
__device__ __forceinline__ uint2 pack_head(const RowHead& h) {
    return make_uint2(h.start | ((uint32_t)h.n1 << 20), (uint32_t)h.nf | ((uint32_t)h.n0 << 16));
}
__device__ __forceinline__ RowHead unpack_head(uint2 v) {
    return {v.x & kRowGlobal, (int)(v.y & 0xffffu), (int)(v.y >> 16), (int)(v.x >> 20)};
}
static_assert(kMaxResidentBeads <= 2048, "row counts of 12 bits, byte offsets of 16");

__device__ __forceinline__ float4 bead_at(const char* xb, uint32_t off) { return *reinterpret_cast<const float4*>(xb + off); }

// ---- the forces of a pair of beads ---------------------------------------------
// The order of a bead's sum is that of V = 4 lpb (at most 32) lanes per pair
// of beads, whatever the number of lanes that compute it:
//   both-section: lane v sums entries v, v + V, ...; then the sums of lanes v
//     and v ^ V/2, then u and u ^ V/4 are added, which leaves V/4 sums S[w];
//   a bead's own section and its bonded maps: lane w of V/4 sums entries w,
//     w + V/4, ..., which gives O[w];
//   then c8 S[w] + O[w] is summed over w by a butterfly.
// A narrow group of G = V/2 lanes keeps two both-section sums per lane, for
// lanes l and l + G of V; a wide one of V lanes keeps one (and the upper half
// of each bead's lanes has no part in the bead's own entries).  Launches that
// fill the GPU are bound by issue slots and take narrow groups, which spend
// the instructions around the loops once for twice the beads; clusters, where
// a step is bound by latency, take wide ones (200 beads on eight CTAs: 3.1 us
// a step wide, 4.0 narrow).
template <bool WIDE>
struct PairGroup {
    int G, H;          // lanes per pair, per bead
    int l, h, lh;      // lane of the group, its bead of the pair, lane of the bead's half
    __device__ __forceinline__ PairGroup(int lpb, int lane, int G_) {
        G = G_ ? G_ : (lpb < 8 ? 4 * lpb : 32) / (WIDE ? 1 : 2);
        H = G >> 1;
        l = lane & (G - 1);
        h = l >= H ? 1 : 0;
        lh = l & (H - 1);
    }
    __device__ __forceinline__ int own_lanes() const { return WIDE ? H >> 1 : H; }
    __device__ __forceinline__ bool owns() const { return !WIDE || 2 * lh < H; }
};

__device__ __forceinline__ void add3(float3& a, float3 b) {
    a.x += b.x;
    a.y += b.y;
    a.z += b.z;
}
__device__ __forceinline__ float3 shfl3_xor(float3 f, int o) {
    return make_float3(__shfl_xor_sync(0xffffffffu, f.x, o), __shfl_xor_sync(0xffffffffu, f.y, o),
                       __shfl_xor_sync(0xffffffffu, f.z, o));
}

// S[w] of the lane's bead from the lanes' both-section sums: a of lane l, b
// (narrow) of lane l + G.  All lanes of the warp take part.
template <bool WIDE>
__device__ __forceinline__ float3 pair_sum(const PairGroup<WIDE>& g, float3 a0, float3 a1, float3 b0, float3 b1) {
    __syncwarp();
    float3 s;
    if (WIDE) {
        add3(a0, shfl3_xor(a0, g.H));
        add3(a1, shfl3_xor(a1, g.H));
        s = g.h ? a1 : a0;
        add3(s, shfl3_xor(s, g.H >> 1));
    } else {
        add3(a0, b0);
        add3(a1, b1);
        s = g.h ? a1 : a0;
        add3(s, shfl3_xor(g.h ? a0 : a1, g.H));
    }
    return s;
}

// The both-section: unscaled sums of d / r^8 (an empty row where a group has
// no pair).
template <bool WIDE, typename Entry>
__device__ __forceinline__ float3 row_both(const Entry* __restrict__ row, int cnt, const PairGroup<WIDE>& g,
                                           const char* xb, float4 x0, float4 x1, float cut2) {
    float3 a0 = make_float3(0.f, 0.f, 0.f), a1 = a0, b0 = a0, b1 = a0;
    int k = g.l;
    for (; k + g.G < cnt; k += 2 * g.G) {
        const int o0 = row[k], o1 = row[k + g.G];
        const float4 q0 = bead_at(xb, o0), q1 = bead_at(xb, o1);
        pair_term8(x0, q0, cut2, a0);
        pair_term8(x1, q0, cut2, a1);
        pair_term8(x0, q1, cut2, WIDE ? a0 : b0);
        pair_term8(x1, q1, cut2, WIDE ? a1 : b1);
    }
    if (k < cnt) {
        const float4 q = bead_at(xb, row[k]);
        pair_term8(x0, q, cut2, a0);
        pair_term8(x1, q, cut2, a1);
    }
    return pair_sum(g, a0, a1, b0, b1);
}

// A bead's own section, its bonded maps and its surface beads, over the V/4
// lanes of its half of the group.
template <bool WIDE, typename Entry>
__device__ __forceinline__ float3 row_own(const Entry* __restrict__ row, int cnt, const PairGroup<WIDE>& g, const char* xb,
                                          float4 xi, float cut2, float c8) {
    float3 f = make_float3(0.f, 0.f, 0.f);
    const int step = g.own_lanes();
    if (g.owns()) {
        int k = g.lh;
        for (; k + step < cnt; k += 2 * step) {
            const int o0 = row[k], o1 = row[k + step];
            const float4 q0 = bead_at(xb, o0), q1 = bead_at(xb, o1);
            pair_term8(xi, q0, cut2, f);
            pair_term8(xi, q1, cut2, f);
        }
        if (k < cnt) pair_term8(xi, bead_at(xb, row[k]), cut2, f);
    }
    return make_float3(f.x * c8, f.y * c8, f.z * c8);
}

// Bonded terms of bead i from the global maps.
template <bool WIDE>
__device__ __forceinline__ void bonded_global(const JobDev& J, const float4* __restrict__ xs, int i, float4 xi,
                                              const PairGroup<WIDE>& g, float3& f) {
    if (g.owns()) bonded_partial(J, xs, i, xi, g.lh, g.own_lanes(), f);
}

// The bead's total on every lane that takes part in its own entries: s from
// row_both, f the lane's own entries.
template <bool WIDE>
__device__ __forceinline__ float3 pair_total(float3 s, float3 f, float c8, const PairGroup<WIDE>& g) {
    __syncwarp();
    float3 t = make_float3(fmaf(c8, s.x, f.x), fmaf(c8, s.y, f.y), fmaf(c8, s.z, f.z));
    for (int m = g.own_lanes() >> 1; m > 0; m >>= 1) add3(t, shfl3_xor(t, m));
    return t;
}

// Bead i's partners in its global row, one after another (observables).
template <typename Visit>
__device__ __forceinline__ void for_partners(const JobDev& J, int i, Visit visit) {
    if (J.mask) {
        const RowHead hd = unpack_head(J.vh[i >> 1]);
        const uint16_t* row = J.vr + (size_t)(i >> 1) * J.cap_u;
        for (int k = 0; k < hd.nf; ++k) visit(row[k] >> 4);
        const uint16_t* own = row + hd.nf + ((i & 1) ? hd.n0 : 0);
        for (int k = 0; k < ((i & 1) ? hd.n1 : hd.n0); ++k) visit(own[k] >> 4);
    } else if (J.gvr) {
        const int4 hd = J.gvh[i >> 1];
        const int32_t* row = J.gvr + (size_t)((i >> 1) / J.tile) * J.tile * J.cap_u + hd.w;
        for (int k = 0; k < hd.x; ++k) visit((int)((uint32_t)row[k] >> 4));
        const int32_t* own = row + hd.x + ((i & 1) ? hd.y : 0);
        for (int k = 0; k < ((i & 1) ? hd.z : hd.y); ++k) visit((int)((uint32_t)own[k] >> 4));
    } else {
        const int32_t* row = J.pl_j + (size_t)i * J.cap_pl;
        for (int k = 0; k < J.pl_cnt[i]; ++k) visit(row[k]);
    }
}

// generate_possiblepairs (src/Updaters/possiblepairlist_kernel.cu:18-71):
// every q of the job with |r| < pairs_threshold that is neither i nor a
// covalent or native partner, as a bitmask row (the CTA's beads).  A warp takes one bead;
// lane b tests bead 32w+b of word w and a ballot forms the word.  More than
// max_possiblePairs sets err (the reference writes past its rows there).
__device__ __noinline__ void build_possible(const JobDev& J, const PartView& V, const float4* __restrict__ xs, int& err) {
    const int n = J.n, W = J.W, lane = threadIdx.x & 31;
    for (int i = V.b0 + (threadIdx.x >> 5); i < V.b1; i += blockDim.x >> 5) {
        const float4 xi = xs[i];
        const uint32_t* ex = J.ex_mask + (size_t)i * W;
        uint32_t* row = J.pp_mask + (size_t)i * W;
        int cnt = 0;
        for (int w = 0; w < W; ++w) {
            const int q = 32 * w + lane;
            const bool ok = q < n && within_cutoff(xi, xs[q < n ? q : 0], J.pp_t);
            const uint32_t bits = __ballot_sync(0xffffffffu, ok) & ~__ldg(&ex[w]);
            if (lane == 0) row[w] = bits;
            cnt += __popc(bits);
        }
        if (lane == 0 && cnt > J.max_pp) err = SOPB_STATUS_CAPACITY;
    }
}

// generate_pairs (src/Updaters/pairlist_kernel.cu:33-76): the possible pairs
// with |r| < pairlist_cutoff, as one row per pair of beads.  A warp takes a
// pair.  The lane's candidates of round u (32 candidates in increasing j per
// round) are e[u] for the first kKeptRounds rounds, which cover nearly every
// row, and far(u) after them: 16 q, bit 0 when the first bead may pair with q
// and bit 1 when the second may; 0 for none.  Ballots give each hit its place
// in its section (in increasing j; kept in a register for the first rounds)
// and the sections' lengths; then lane 0 takes room for the row in the CTA's
// shared rows, or the pair's global row where none is left, and the hits are
// stored.  More than max_pairs partners of a bead sets err;
// a row beyond its storage is cut off.
constexpr int kKeptRounds = 8;
__device__ __forceinline__ int row_hit(const JobDev& J, const char* xb, float4 x0, float4 x1, int e) {
    const float4 q = bead_at(xb, e & 0xfff0);
    return ((dist2_rn(x0, q) < J.pl_t ? 1 : 0) | (dist2_rn(x1, q) < J.pl_t ? 2 : 0)) & e;
}
template <typename Far>
__device__ __forceinline__ void build_row(const JobDev& J, const PartView& V, int* alloc, int p,
                                          const float4* __restrict__ xs, int rounds, const int (&e)[kKeptRounds], Far far,
                                          int& err) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u, all = 0xffffffffu;
    const float4 x0 = xs[2 * p], x1 = xs[2 * p + 1 < J.n ? 2 * p + 1 : 2 * p];
    const char* xb = reinterpret_cast<const char*>(xs);
    // one round's hits: their numbers so far per section, and the lane's
    // verdict and place in its section beside its candidate
    int cf = 0, c0 = 0, c1 = 0;
    auto round = [&](int c) {
        const int hit = row_hit(J, xb, x0, x1, c);
        const unsigned mf = __ballot_sync(all, hit == 3), m0 = __ballot_sync(all, hit == 1), m1 = __ballot_sync(all, hit == 2);
        const int at = (hit == 3 ? cf : (hit == 1 ? c0 : c1)) +
                       __popc((hit == 3 ? mf : (hit == 1 ? m0 : m1)) & below);
        cf += __popc(mf);
        c0 += __popc(m0);
        c1 += __popc(m1);
        return (c & 0xfff0) | hit | (at << 16);
    };
    unsigned w[kKeptRounds];
#pragma unroll
    for (int u = 0; u < kKeptRounds; ++u) w[u] = u < rounds ? (unsigned)round(e[u]) : 0u;
    const int kf = cf, k0 = c0, k1 = c1;
    for (int u = kKeptRounds; u < rounds; ++u) round(far(u));
    RowHead hd{kRowGlobal, cf, c0, c1};
    if (max(hd.n0, hd.n1) + hd.nf > J.cap_pl) {
        err = SOPB_STATUS_CAPACITY;
        hd.nf = min(hd.nf, J.cap_u);
        hd.n0 = min(hd.n0, J.cap_u - hd.nf);
        hd.n1 = min(hd.n1, J.cap_u - hd.nf - hd.n0);
    }
    const int len = hd.nf + hd.n0 + hd.n1;
    if (V.hd) {
        int at = 0;
        if (lane == 0) at = atomicAdd(alloc, len);
        at = __shfl_sync(all, at, 0);
        if (at + len <= V.cap) hd.start = (uint32_t)at;
        if (lane == 0) V.hd[p - V.p0] = pack_head(hd);
    } else if (lane == 0) {
        J.vh[p] = pack_head(hd);
    }
    auto store = [&](uint16_t* dst, unsigned v) {
        const int hit = v & 3, at = (int)(v >> 16) + (hit == 3 ? 0 : (hit == 1 ? hd.nf : hd.nf + hd.n0));
        if (hit && at < len) dst[at] = (uint16_t)(v & 0xfff0);
    };
    auto store_all = [&](uint16_t* dst) {
#pragma unroll
        for (int u = 0; u < kKeptRounds; ++u)
            if (u < rounds) store(dst, w[u]);
        if (rounds > kKeptRounds) {
            cf = kf;
            c0 = k0;
            c1 = k1;
            for (int u = kKeptRounds; u < rounds; ++u) store(dst, (unsigned)round(far(u)));
        }
    };
    if (hd.start != kRowGlobal) store_all(V.nbr + hd.start);
    else store_all(J.vr + (size_t)p * J.cap_u);
}

// The rows from the possible pairs of both beads, and with them the near
// rows: the possible pairs within pairlist_cutoff + skin of either bead, as
// candidates (16 q and which bead they are near to) for the cheaper rebuilds
// that follow (build_verlet_near).  The two beads' mask words are held two
// per lane each (W <= 64); lane b tests candidate 32 u + b of round u.  A
// near row longer than its capacity sets *near_over.
__device__ __noinline__ void build_verlet(const JobDev& J, const PartView& V, int* alloc, const float4* __restrict__ xs,
                                          int& err, int* near_over) {
    static_assert(kMaxResidentBeads <= 64 * 32, "two mask words per lane");
    const int n = J.n, W = J.W, lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    for (int p = V.p0 + (threadIdx.x >> 5); p < V.p1; p += blockDim.x >> 5) {
        const uint32_t* pm = J.pp_mask + (size_t)(2 * p) * W;
        const bool two = 2 * p + 1 < n;
        const uint32_t a0 = lane < W ? pm[lane] : 0u, a1 = lane + 32 < W ? pm[lane + 32] : 0u;
        const uint32_t d0 = two && lane < W ? pm[W + lane] : 0u, d1 = two && lane + 32 < W ? pm[W + lane + 32] : 0u;
        auto cand = [&](int u) {
            const uint32_t m = __shfl_sync(0xffffffffu, u < 32 ? a0 : a1, u & 31);
            const uint32_t d = __shfl_sync(0xffffffffu, u < 32 ? d0 : d1, u & 31);
            const int c = (int)((m >> lane) & 1u) | (int)(((d >> lane) & 1u) << 1);
            return c ? (32 * u + lane) * 16 | c : 0;
        };
        if (J.drift2 > 0.f) {
            const float4 x0 = xs[2 * p], x1 = xs[two ? 2 * p + 1 : 2 * p];
            uint16_t* nrow = J.nr_j + (size_t)p * J.cap_nr;
            int cnt = 0;
            for (int u = 0; u < W; ++u) {
                int e = cand(u);
                const float4 q = bead_at(reinterpret_cast<const char*>(xs), e & 0xfff0);
                if (!((e & 1) && dist2_rn(x0, q) < J.nr_t)) e &= ~1;
                if (!((e & 2) && dist2_rn(x1, q) < J.nr_t)) e &= ~2;
                const unsigned hit = __ballot_sync(0xffffffffu, e & 3);
                const int pos = cnt + __popc(hit & below);
                if ((e & 3) && pos < J.cap_nr) nrow[pos] = (uint16_t)e;
                cnt += __popc(hit);
            }
            if (lane == 0) {
                if (cnt > J.cap_nr) atomicOr(near_over, 1);
                J.nr_cnt[p] = cnt < J.cap_nr ? cnt : J.cap_nr;
            }
        }
        int e[kKeptRounds];
#pragma unroll
        for (int u = 0; u < kKeptRounds; ++u) e[u] = u < W ? cand(u) : 0;
        build_row(J, V, alloc, p, xs, W, e, cand, err);
    }
}

// The Verlet rows from the near rows: while no bead moved more than half the
// skin since they were built, every pair now closer than pairlist_cutoff was
// closer than pairlist_cutoff + skin then, so filtering the near rows
// (increasing j) with the same exact test gives the same rows as the full
// scan.  A warp per pair; it fetches its next pair's row length while it
// filters the current row, and a row's first kKeptRounds x 32 entries are
// loaded before any of them is tested, so a row costs one global round trip.
__device__ __forceinline__ void build_verlet_near(const JobDev& J, const PartView& V, int* alloc,
                                                  const float4* __restrict__ xs, int& err) {
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    int p = V.p0 + (threadIdx.x >> 5);
    int ncnt = p < V.p1 ? J.nr_cnt[p] : 0;
    for (; p < V.p1; p += warps) {
        const int cnt = ncnt;
        ncnt = p + warps < V.p1 ? J.nr_cnt[p + warps] : 0;
        const uint16_t* nrow = J.nr_j + (size_t)p * J.cap_nr;
        int e[kKeptRounds];
#pragma unroll
        for (int u = 0; u < kKeptRounds; ++u) e[u] = 32 * u + lane < cnt ? nrow[32 * u + lane] : 0;
        auto far = [&](int u) { return 32 * u + lane < cnt ? (int)nrow[32 * u + lane] : 0; };
        build_row(J, V, alloc, p, xs, (cnt + 31) >> 5, e, far, err);
    }
}

// ---- clusters ---------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_nctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
    cluster_arrive();
    cluster_wait();
}
// The address of CTA `rank`'s copy of this CTA's shared address `a`.
__device__ __forceinline__ uint32_t map_rank(uint32_t a, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// Stores v to a CTA's shared memory and counts its 16 bytes on that CTA's
// mbarrier (both cluster addresses).
__device__ __forceinline__ void send16(uint32_t addr, float4 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
                 "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)),
                 "r"(bar)
                 : "memory");
}
constexpr uint32_t kPeerWaitLimit = 1u << 20;   // try_wait suspends for a while itself
__device__ __forceinline__ bool peers_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t it = 0; it < kPeerWaitLimit; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred P1;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P1;\n\t}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// A cluster gives up as a whole.  A CTA whose wait for its peers runs out
// writes into every CTA's `gave_up` the step at which its chunk of steps ends,
// arrives at its last cluster barrier and leaves.  The barrier that pairs with
// it is the first one of an updater boundary at that step or later, or the last
// one: a CTA there finds the step of its boundary reached and leaves as well,
// without another barrier or a store into a peer, which may be gone.  A CTA
// that gives up after the boundary writes a later step, so every thread that
// looks sees the same, however late.  None writes its state back: the job keeps
// the one it had at the launch (its lists may be newer), with the status
// SOPB_ERR_TIMEOUT.
constexpr int64_t kNeverStep = INT64_MAX;
__device__ __forceinline__ int64_t gave_up_at(const int64_t* word) { return *(const volatile int64_t*)word; }
__device__ __forceinline__ void give_up(int64_t* word, int C, int64_t step) {
    if ((int)threadIdx.x < C) {
        const uint32_t a = map_rank((uint32_t)__cvta_generic_to_shared(word), threadIdx.x);
        asm volatile("st.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(step) : "memory");
    }
}
// A boundary's first cluster barrier; false when a peer gave up before it.
__device__ __forceinline__ bool peers_meet(const PartView& V, int64_t step) {
    cluster_sync_all();
    return gave_up_at(V.gave_up) > step;
}

// Verlet rebuild of a resident job: from the near rows when they are valid
// and no bead drifted more than half the skin from where they were built,
// else a full scan that also renews the near rows at the current
// coordinates.  The CTAs of a cluster decide alike: each looks at every bead
// (its own copy of the coordinates and of x_ref), and after a full scan the
// near rows count as valid when no CTA's overflowed.  False when a peer gave up.
template <bool CL>
__device__ bool rebuild_verlet(const JobDev& J, const PartView& V, const float4* __restrict__ xs, int& valid,
                               bool possible_changed, int64_t step, int& err) {
    __shared__ int drift_bits, near_over, alloc;
    const int tid = threadIdx.x, n = J.n;
    if (tid == 0) {
        drift_bits = 0;
        near_over = 0;
        alloc = 0;
    }
    __syncthreads();
    if (valid && !possible_changed) {
        float d2 = 0.f;
        for (int i = tid; i < n; i += blockDim.x) {
            const float e = dist2_rn(V.xref[i], xs[i]);
            d2 = fmaxf(d2, isfinite(e) ? e : INFINITY);   // fmaxf drops a NaN: count it as an infinite drift
        }
        // non-negative floats order as ints
        const int m = __reduce_max_sync(0xffffffffu, __float_as_int(d2));
        if ((tid & 31) == 0 && m > 0) atomicMax(&drift_bits, m);
    }
    __syncthreads();
    if (valid && !possible_changed && __int_as_float(drift_bits) < J.drift2) {
        build_verlet_near(J, V, &alloc, xs, err);
        return true;
    }
    if (CL && !peers_meet(V, step)) return false;   // every CTA has cleared near_over
    build_verlet(J, V, &alloc, xs, err, &near_over);
    for (int i = tid; i < n; i += blockDim.x) V.xref[i] = xs[i];
    __syncthreads();
    if (CL) {
        if (near_over && tid < V.C) {
            const uint32_t a = map_rank((uint32_t)__cvta_generic_to_shared(&near_over), (uint32_t)tid);
            asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(1) : "memory");
        }
        cluster_sync_all();
    }
    valid = near_over || !(J.drift2 > 0.f) ? 0 : 1;   // drift2 0: the job keeps no near list
    return true;
}

// Deterministic CTA sum of a float3 (fixed tree for a given BLOCK).
template <int BLOCK>
__device__ float3 block_sum3(float3 v, float (*red)[4]) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        v.z += __shfl_xor_sync(0xffffffffu, v.z, o);
    }
    __syncthreads();
    if (lane == 0) { red[w][0] = v.x; red[w][1] = v.y; red[w][2] = v.z; }
    __syncthreads();
    float3 s = make_float3(0.f, 0.f, 0.f);
    for (int q = 0; q < BLOCK / 32; ++q) { s.x += red[q][0]; s.y += red[q][1]; s.z += red[q][2]; }
    return s;
}

// Sum of the job's per-bead tip forces, by the tree of a CTA of J.block
// threads whatever the launch's CTA size (so that it does not depend on the
// cluster): virtual warp v of it sums beads 32 v + lane, + J.block, ...
__device__ __noinline__ float3 tip_sum(const JobDev& J, float (*red)[4]) {
    const int lane = threadIdx.x & 31, vb = J.block;
    for (int v = threadIdx.x >> 5; v < vb / 32; v += blockDim.x >> 5) {
        float3 p = make_float3(0.f, 0.f, 0.f);
        for (int i = 32 * v + lane; i < J.n; i += vb) {
            const float4 t = __ldcg(&J.tipF[i]);
            p.x += t.x; p.y += t.y; p.z += t.z;
        }
        for (int o = 16; o > 0; o >>= 1) {
            p.x += __shfl_xor_sync(0xffffffffu, p.x, o);
            p.y += __shfl_xor_sync(0xffffffffu, p.y, o);
            p.z += __shfl_xor_sync(0xffffffffu, p.z, o);
        }
        if (lane == 0) { red[v][0] = p.x; red[v][1] = p.y; red[v][2] = p.z; }
    }
    __syncthreads();
    float3 s = make_float3(0.f, 0.f, 0.f);
    for (int q = 0; q < vb / 32; ++q) { s.x += red[q][0]; s.y += red[q][1]; s.z += red[q][2]; }
    return s;
}

// Appends one row to the job's event-log ring (sopb_log_row layout: kind,
// pad, step, twelve floats); the host drains it with sopb_job_log.
__device__ __forceinline__ void log_row(const JobDev& J, uint32_t& head, int32_t kind, int64_t step, const float* v) {
    if (J.log_cap <= 0) return;
    float* r = J.log + (size_t)(head & (uint32_t)(J.log_cap - 1)) * 16;
    reinterpret_cast<int32_t*>(r)[0] = kind;
    reinterpret_cast<int32_t*>(r)[1] = 0;
    *reinterpret_cast<int64_t*>(r + 2) = step;
    for (int k = 0; k < 12; ++k) r[4 + k] = v[k];
    ++head;
}

// PullingPotential::savePullingData (src/Potentials/pulling.cu:167-190): the
// end-to-end distance, its projection and the applied force along the pull
// vector, from the coordinates of this step and the force just computed.
// The reference evaluates it on the host (IEEE, no contraction).
__device__ __noinline__ void log_pull(const JobDev& J, StepScalars& sc, float4 xp, float4 xf, int64_t step) {
    const float e[3] = {__fsub_rn(xp.x, xf.x), __fsub_rn(xp.y, xf.y), __fsub_rn(xp.z, xf.z)};
    auto dot3 = [](const float* a, const float* b) {
        return __fadd_rn(__fadd_rn(__fmul_rn(a[0], b[0]), __fmul_rn(a[1], b[1])), __fmul_rn(a[2], b[2]));
    };
    const float v[12] = {__fsqrt_rn(dot3(e, e)), dot3(e, J.pullvec), dot3(sc.pullF, J.pullvec),
                         sc.pullF[0], sc.pullF[1], sc.pullF[2], 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    log_row(J, sc.log_head, SOPB_LOG_PULL, step, v);
}

// PullingPlaneUpdater::update (src/Potentials/pulling_plane.cu:183-258), run
// every stride by one thread: the cantilever moves by deltax per update
// period; the plane takes one overdamped step of update-period length under
// the cantilever spring and the beads' springs, summed in bead order from
// the forces of the last step; every output period one log line with the
// distance between the centroids of the fixed and the pulled beads.  Host
// arithmetic in the reference: explicit _rn operations.
__device__ __noinline__ void plane_update(const JobDev& J, StepScalars& sc, const float4* __restrict__ xs, int64_t step) {
    const float xt = __fdiv_rn(__fmul_rn(J.plane_deltax, (float)step), (float)J.plane_freq);
    sc.plane_cant = xt;
    const int32_t* fixed = J.plane_idx;
    const int32_t* pulled = J.plane_idx + J.nplane_fixed;
    float ext = 0.0f;
    for (int k = 0; k < J.nplane_pulled; ++k) ext = __fadd_rn(ext, __ldcg(&J.plane_f[pulled[k]]));
    const float cant = __fmul_rn(__fsub_rn(xt, sc.plane_displ), J.plane_kscant);
    const float mult = __fdiv_rn(__fmul_rn((float)J.plane_freq, J.h), J.plane_zeta);
    sc.plane_displ = __fadd_rn(sc.plane_displ, __fmul_rn(mult, __fsub_rn(cant, ext)));
    if (step % J.plane_ofreq == 0) {
        float cf[3] = {0.f, 0.f, 0.f}, cp[3] = {0.f, 0.f, 0.f};
        for (int k = 0; k < J.nplane_fixed; ++k) {
            const float4 q = xs[fixed[k]];
            cf[0] = __fadd_rn(cf[0], q.x); cf[1] = __fadd_rn(cf[1], q.y); cf[2] = __fadd_rn(cf[2], q.z);
        }
        for (int k = 0; k < J.nplane_pulled; ++k) {
            const float4 q = xs[pulled[k]];
            cp[0] = __fadd_rn(cp[0], q.x); cp[1] = __fadd_rn(cp[1], q.y); cp[2] = __fadd_rn(cp[2], q.z);
        }
        float d[3];
        for (int c = 0; c < 3; ++c)
            d[c] = __fsub_rn(__fdiv_rn(cp[c], (float)J.nplane_pulled), __fdiv_rn(cf[c], (float)J.nplane_fixed));
        const float e2e = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1])), __fmul_rn(d[2], d[2])));
        const float v[12] = {sc.plane_displ, xt, cant, ext, e2e, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        log_row(J, sc.log_head, SOPB_LOG_PLANE, step, v);
    }
}

// Discrete surface at a tip update: the surface beads follow dx when the
// surface moves (IndentationTipUpdater::update, indentation.cu:446-455), then
// every bead's list of surface beads within the cutoff is rebuilt
// (generateMicaList_kernel, indentation_kernel.cu:182-201) as a bitmask row,
// a warp per bead and a ballot per 32 surface beads.
template <bool CL>
__device__ __noinline__ void build_mica(const JobDev& J, const PartView& V, const float4* __restrict__ xs, float dx) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (J.moveSurface) {
        for (int q = V.rank * blockDim.x + tid; q < J.nsurf; q += V.C * blockDim.x) {
            const float4 s0 = J.surf0[q];
            J.surf[q] = make_float4(__fadd_rn(s0.x, __fmul_rn(J.dir[0], dx)), __fadd_rn(s0.y, __fmul_rn(J.dir[1], dx)),
                                    __fadd_rn(s0.z, __fmul_rn(J.dir[2], dx)), 0.f);
        }
        if (CL) cluster_sync_all();
        else __syncthreads();
    }
    for (int i = V.b0 + w; i < V.b1; i += blockDim.x >> 5) {
        const float4 xi = xs[i];
        uint32_t* row = J.mica + (size_t)i * J.Wm;
        for (int wd = 0; wd < J.Wm; ++wd) {
            const int q = 32 * wd + lane;
            bool in = false;
            if (q < J.nsurf) in = dist2_rn(xi, J.surf[q]) < J.mica_cut2;
            const uint32_t m = __ballot_sync(0xffffffffu, in);
            if (lane == 0) row[wd] = m;
        }
    }
    __syncthreads();
}

// IndentationTipUpdater::update (src/Potentials/indentation.cu:414-550) for
// the continuous surface, run by thread 0 after the CTA summed the tip force.
// Host-side arithmetic of the reference is IEEE without contraction, hence
// the explicit _rn intrinsics.
__device__ __noinline__ void tip_update(const JobDev& J, StepScalars& sc, float3 fsum, int64_t step) {
    const float inv = (float)J.nav;
    float f[3] = {__fdiv_rn(fsum.x, inv), __fdiv_rn(fsum.y, inv), __fdiv_rn(fsum.z, inv)};
    sc.dx = __fmul_rn((float)(step / J.nav), sc.V);
    if (J.moveSurface) {
        for (int c = 0; c < 3; ++c) sc.ig.micaR[c] = __fadd_rn(J.micaR0[c], __fmul_rn(J.dir[c], sc.dx));
    } else {
        for (int c = 0; c < 3; ++c) sc.chip[c] = __fadd_rn(J.chip0[c], __fmul_rn(J.dir[c], sc.dx));
    }
    float df[3], dr[3];
    for (int c = 0; c < 3; ++c) dr[c] = __fsub_rn(sc.chip[c], sc.ig.tip[c]);
    const float drw = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dr[0], dr[0]), __fmul_rn(dr[1], dr[1])), __fmul_rn(dr[2], dr[2])));
    for (int c = 0; c < 3; ++c) df[c] = __fadd_rn(-f[c], __fmul_rn(dr[c], J.cantKs));
    const float mult = __fdiv_rn(__fmul_rn(J.h, (float)J.nav), J.tipZeta);
    if (J.fixTrans) {
        float ct = __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(mult, df[0]), J.dir[0]), __fmul_rn(__fmul_rn(mult, df[1]), J.dir[1])),
                             __fmul_rn(__fmul_rn(mult, df[2]), J.dir[2]));
        for (int c = 0; c < 3; ++c) sc.ig.tip[c] = __fadd_rn(sc.ig.tip[c], __fmul_rn(ct, J.dir[c]));
    } else {
        for (int c = 0; c < 3; ++c) sc.ig.tip[c] = __fadd_rn(sc.ig.tip[c], __fmul_rn(mult, df[c]));
    }
    sc.fav[0] = f[0];
    sc.fav[1] = f[1];
    sc.fav[2] = f[2];
    sc.fav[3] = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(f[0], f[0]), __fmul_rn(f[1], f[1])), __fmul_rn(f[2], f[2])));
    const float v[12] = {sc.fav[0], sc.fav[1], sc.fav[2], sc.fav[3], drw, sc.dx,
                         sc.ig.tip[0], sc.ig.tip[1], sc.ig.tip[2], sc.chip[0], sc.chip[1], sc.chip[2]};
    log_row(J, sc.log_head, SOPB_LOG_TIP, step, v);
}

// The CTA's pairs ordered by the length of their rows, longest first (a
// counting sort by fours), so that the pairs of a warp take alike long and
// the warps end together: without it the longest of a warp's rows is 1.4
// times their mean on chains of 200 to 600 beads.  The order inside a bucket
// is arbitrary; no result depends on it.
__device__ __noinline__ void order_rows(const PartView& V) {
    __shared__ int hist[64];
    const int tid = threadIdx.x, npl = V.p1 - V.p0;
    auto bucket = [&](int pl) {
        const RowHead hd = unpack_head(V.hd[pl]);
        return max(0, 63 - ((hd.nf + max(hd.n0, hd.n1)) >> 2));
    };
    if (tid < 64) hist[tid] = 0;
    __syncthreads();
    for (int pl = tid; pl < npl; pl += blockDim.x) atomicAdd(&hist[bucket(pl)], 1);
    __syncthreads();
    if (tid < 32) {
        const int a = hist[2 * tid], b = hist[2 * tid + 1];
        int incl = a + b;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (tid >= o) incl += t;
        }
        hist[2 * tid] = incl - a - b;
        hist[2 * tid + 1] = incl - b;
    }
    __syncthreads();
    for (int pl = tid; pl < npl; pl += blockDim.x) V.order[atomicAdd(&hist[bucket(pl)], 1)] = (uint16_t)pl;
}

// The rows of the CTA's pairs from global memory into its shared rows (at a
// launch's start) and back (at its end).
__device__ __noinline__ void load_rows(const JobDev& J, const PartView& V) {
    __shared__ int alloc;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) alloc = 0;
    __syncthreads();
    for (int p = V.p0 + (threadIdx.x >> 5); p < V.p1; p += blockDim.x >> 5) {
        RowHead hd = unpack_head(J.vh[p]);
        const int len = hd.nf + hd.n0 + hd.n1;
        int at = 0;
        if (lane == 0) at = atomicAdd(&alloc, len);
        at = __shfl_sync(0xffffffffu, at, 0);
        hd.start = at + len <= V.cap ? (uint32_t)at : kRowGlobal;
        if (lane == 0) V.hd[p - V.p0] = pack_head(hd);
        if (hd.start != kRowGlobal) {
            const uint16_t* src = J.vr + (size_t)p * J.cap_u;
            for (int k = lane; k < len; k += 32) V.nbr[at + k] = src[k];
        }
    }
    __syncthreads();
}
__device__ __noinline__ void store_rows(const JobDev& J, const PartView& V) {
    const int lane = threadIdx.x & 31;
    for (int p = V.p0 + (threadIdx.x >> 5); p < V.p1; p += blockDim.x >> 5) {
        RowHead hd = unpack_head(V.hd[p - V.p0]);
        if (hd.start != kRowGlobal) {
            const int len = hd.nf + hd.n0 + hd.n1;
            uint16_t* dst = J.vr + (size_t)p * J.cap_u;
            for (int k = lane; k < len; k += 32) dst[k] = V.nbr[hd.start + k];
        }
        hd.start = kRowGlobal;
        if (lane == 0) J.vh[p] = pack_head(hd);
    }
}

// The updaters of one `stride` boundary in the reference order
// (creation order in src/gsop.cu:80-101; loop in src/gsop.cu:129-133).
// Returns 1 when the Verlet list was rebuilt, -1 when a peer gave up.
template <bool CL>
__device__ __noinline__ int run_updaters(const JobDev& J, const PartView& V, StepScalars& sc, const float4* __restrict__ xs,
                                         float* Ts, float (*red)[4], int64_t step, int& err) {
    const int tid = threadIdx.x, nb = V.b1 - V.b0;
    // the tip's and the plane's per-bead forces of the other CTAs' beads
    if (CL && (J.indent || J.plane) && !peers_meet(V, step)) return -1;
    if (J.indent) {
        if (tid == 0 && step == J.retraction_step) sc.V = -sc.V;
        if (step % J.nav == 0) {
            const float3 s = tip_sum(J, red);
            if (CL) cluster_sync_all();
            else __syncthreads();
            for (int i = V.b0 + tid; i < V.b1; i += blockDim.x) {
                const float4 t = J.tipF[i];
                J.tipF[i] = make_float4(0.f, 0.f, 0.f, t.w);
            }
            if (tid == 0) tip_update(J, sc, s, step);
            if (J.discrete) {
                __syncthreads();
                build_mica<CL>(J, V, xs, sc.dx);
            }
        }
    }
    if (J.pulling && J.ramp && tid == 0) {
        // PullingUpdater::update runs every stride (src/Potentials/pulling.cu:198-204)
        const float xt = __fmul_rn(J.deltax, (float)(step / J.pull_freq));
        const float4 xe = xs[J.pulledEnd];
        const float xe3[3] = {xe.x, xe.y, xe.z};
        for (int c = 0; c < 3; ++c) sc.pullF[c] = __fmul_rn(J.k_trans, __fsub_rn(sc.cant[c], xe3[c]));
        for (int c = 0; c < 3; ++c) sc.cant[c] = __fadd_rn(J.cant0[c], __fmul_rn(xt, J.pullvec[c]));
        if (step % J.pull_freq == 0) log_pull(J, sc, xe, xs[J.fixedEnd], step);
    }
    if (J.plane && tid == 0) plane_update(J, sc, xs, step);
    const bool pp = step % J.pp_freq == 0;
    if (pp) build_possible(J, V, xs, err);
    if (step % J.nav == 0)
        for (int i = tid; i < nb; i += blockDim.x) Ts[i] = 0.0f;   // output_manager.cu:125-127
    const bool verlet = step % J.pairs_freq == 0;
    if (pp && !verlet && tid == 0) sc.nr_valid = 0;   // the near list no longer matches the possible pairs
    if (verlet) {
        if (pp) __syncthreads();
        int valid = sc.nr_valid;
        if (!rebuild_verlet<CL>(J, V, xs, valid, pp, step, err)) return -1;
        if (tid == 0) sc.nr_valid = valid;
        if (!CL) {
            __syncthreads();
            order_rows(V);
        }
    }
    if (J.heating && tid == 0 && step % J.temp_freq == 0) {
        // TemperatureUpdater (src/Integrators/langevin.cu:129-135, 44-48)
        const float temp = __fadd_rn(J.initialT, __fmul_rn((float)(step / J.temp_freq), J.deltaT));
        sc.var = __fsqrt_rn(__fdiv_rn(__fmul_rn(__fmul_rn(2.0f, temp), J.zeta), J.h));
    }
    // a plane's forces are read above by every CTA before any writes new ones
    if (CL && J.plane) cluster_sync_all();
    else __syncthreads();
    return verlet ? 1 : 0;
}

// What bounds it, and what it measured (B200, 200 steps).  One CTA per job:
// issue slots (77-78 % busy) beside the shared-memory pipe, and within
// them the pair terms; 512 replicas of 60 to 600 beads 5.1 ms, 6.95 ms with
// a row per bead.  Clusters: the dependent chain of a step (about 1200 cycles
// without any list, the exchange 250 to 900 of them); one job of 200 beads
// 0.66 ms (1.63 on one CTA), of 1733 beads 1.36 ms (14.2).
//
// One CTA per job (CL false; up to 1024 threads and 64 registers, so that an
// SM holds 1024 threads of resident CTAs) or a cluster (CL true).  G_: lanes
// per pair of beads for the usual four lanes per bead (8, or 16 wide), 0 when
// it follows from the job.
template <bool CL, bool WIDE, int G_>
__global__ void __launch_bounds__(CL ? kClusterBlock : 1024, 1)
k_resident_steps(JobDev* __restrict__ jobs, const int32_t* __restrict__ ids, const int64_t* __restrict__ steps) {
    const int C = CL ? (int)cluster_nctarank() : 1, rank = CL ? (int)cluster_ctarank() : 0;
    const int entry = CL ? blockIdx.x / C : blockIdx.x;
    const int64_t nsteps = steps[entry];   // each job its own number of steps
    JobDev* Jp = &jobs[ids[entry]];
    __shared__ JobDev Js;
    load_job(Js, Jp);
    __syncthreads();
    const JobDev& J = Js;
    if (J.status != 0) return;             // the same for a job's CTAs: written after their last barrier
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ StepScalars sc;
    __shared__ PartView Vs;                // read as a broadcast, not held in registers
    __shared__ float red[32][4];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ int64_t gave_up;
    __shared__ int next_task[2];           // per-step task counters, double buffered
    const int n = J.n, tid = threadIdx.x, lane = tid & 31, nt = blockDim.x;
    const int lc = 31 - __clz(C);          // C is a power of two
    const int bonded = J.bsm[lc];
    const ResidentLayout lay = resident_layout(n, C, J.lcov[lc], J.lnat[lc], bonded, J.lcache[lc]);
    float4* xs = reinterpret_cast<float4*>(smem + lay.x);
    float4* F = reinterpret_cast<float4*>(smem + lay.F);
    float4* N = reinterpret_cast<float4*>(smem + lay.N);
    uint4* sd = reinterpret_cast<uint4*>(smem + lay.sd);
    float* Ts = reinterpret_cast<float*>(smem + lay.Ts);
    uint8_t* fl = smem + lay.flags;
    const uint16_t* nbr = reinterpret_cast<const uint16_t*>(smem + lay.nbr);
    const uint2* cov_par = reinterpret_cast<const uint2*>(smem + lay.cov_par);
    const float2* nat_par = reinterpret_cast<const float2*>(smem + lay.nat_par);
    const uint16_t* nat_j = reinterpret_cast<const uint16_t*>(smem + lay.nat_j);
    const ushort4* bh = reinterpret_cast<const ushort4*>(smem + lay.bh);
    const int p0 = pair_begin(n, rank, C), p1 = pair_begin(n, rank + 1, C), npl = p1 - p0;
    const int b0 = 2 * p0, b1 = min(n, 2 * p1), nb = b1 - b0;
    for (int i = tid; i < n; i += nt) xs[i] = J.x[i];
    if (tid < 2) {
        xs[n + tid] = make_float4(1.0e18f, 1.0e18f, 1.0e18f, 0.f);
        if (CL) xs[2 * n + 2 + tid] = make_float4(1.0e18f, 1.0e18f, 1.0e18f, 0.f);
    }
    for (int b = tid; b < nb; b += nt) {
        const int i = b0 + b;
        sd[b] = J.seeds[i];
        Ts[b] = J.T[i];
        fl[b] = J.pulling ? J.flags[i] : (uint8_t)FLAG_FREE;
    }
    uint2* hdw = reinterpret_cast<uint2*>(smem + lay.hd);
    uint16_t* order = CL ? nullptr : reinterpret_cast<uint16_t*>(smem + lay.order);
    for (int p = tid; p < npl + kPadPairs; p += nt) {
        hdw[p] = make_uint2(0u, 0u);
        if (!CL) order[p] = (uint16_t)p;     // past the last pair: empty rows
    }
    if (CL && J.nr_valid) {
        float4* xr = reinterpret_cast<float4*>(smem + lay.xref);
        for (int i = tid; i < n; i += nt) xr[i] = J.x_ref[i];
    }
    if (bonded) {
        // the maps of the CTA's beads are constant for the launch
        ushort4* bhw = reinterpret_cast<ushort4*>(smem + lay.bh);
        uint2* cw = reinterpret_cast<uint2*>(smem + lay.cov_par);
        float2* nw = reinterpret_cast<float2*>(smem + lay.nat_par);
        uint16_t* njw = reinterpret_cast<uint16_t*>(smem + lay.nat_j);
        const int c0 = J.cov_off[b0], n0 = J.nat_off[b0], nc = J.cov_off[b1] - c0, nn = J.nat_off[b1] - n0;
        for (int b = tid; b < 2 * (npl + kPadPairs); b += nt)
            bhw[b] = b < nb ? make_ushort4((unsigned short)(J.cov_off[b0 + b] - c0), (unsigned short)(J.cov_off[b0 + b + 1] - c0),
                                           (unsigned short)(J.nat_off[b0 + b] - n0), (unsigned short)(J.nat_off[b0 + b + 1] - n0))
                            : make_ushort4(0, 0, 0, 0);
        for (int k = tid; k < nc; k += nt) cw[k] = make_uint2(__float_as_uint(J.cov_r0[c0 + k]), 16u * (uint32_t)J.cov_j[c0 + k]);
        for (int k = tid; k < nn; k += nt) { nw[k] = J.nat_par[n0 + k]; njw[k] = (uint16_t)(16 * J.nat_j[n0 + k]); }
    }
    if (tid == 0) {
        sc.var = J.var;
        for (int c = 0; c < 3; ++c) {
            sc.pullF[c] = J.pullF[c];
            sc.cant[c] = J.cant[c];
            sc.ig.tip[c] = J.tip[c];
            sc.ig.micaR[c] = J.micaR[c];
            sc.ig.micaN[c] = J.micaN[c];
            sc.chip[c] = J.chip[c];
        }
        sc.ig.tipR = J.tipR; sc.ig.tipAp = J.tipAp; sc.ig.tipBp = J.tipBp;
        sc.ig.surfAp = J.surfAp; sc.ig.surfBp = J.surfBp;
        sc.V = J.V; sc.dx = J.dx;
        for (int c = 0; c < 4; ++c) sc.fav[c] = J.fav[c];
        sc.err = 0;
        sc.nr_valid = J.nr_valid;
        sc.log_head = J.log_head;
        sc.plane_displ = J.plane_displ;
        sc.plane_cant = J.plane_cant;
        Vs = PartView{p0, p1, b0, b1, rank, C, hdw, reinterpret_cast<uint16_t*>(smem + lay.nbr), J.lcache[lc], order,
                      CL ? reinterpret_cast<float4*>(smem + lay.xref) : J.x_ref, &gave_up};
        gave_up = kNeverStep;
        if (CL) {
            for (int q = 0; q < 2; ++q)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(&bars[q])), "r"(1));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            if (rank != 0) Js.log_cap = 0;   // CTA 0 logs
        }
    }
    __syncthreads();
    if (CL) cluster_sync_all();              // the CTAs' mbarriers are ready
    const PartView& V = Vs;
    int64_t step = J.step;
    const int64_t last = step + nsteps;
    int phase = (int)(step % J.stride);      // steps since the last updater pass
    if (phase != 0 || step % J.pairs_freq != 0) {   // else the first step builds them
        load_rows(J, V);
        if (!CL) order_rows(V);
    }

    // a warp's tasks of a step: `per` pairs each, then the noise of 32 beads each
    const PairGroup<WIDE> g(J.lpb, lane, G_);
    const int per = 32 / g.G, group = lane / g.G;
    const int tpairs = (npl + per - 1) / per, tasks = tpairs + (CL && !J.minimization ? (nb + 31) >> 5 : 0);
    const int warps = nt >> 5;
    const bool more = tasks > warps;         // the warps' first tasks are not all of them
    const bool extra = J.indent || J.plane || J.discrete;
    int err = 0;
    bool built = false;
    bool late = false, left = false;         // this CTA gave up; a peer did, and the last barrier is behind
    if (tid < 2) next_task[tid] = warps;
    __syncthreads();
    uint32_t s = 0;                          // steps of this launch, for the buffers' and mbarriers' parity
    while (step < last) {
        if (phase == 0) {
            const int r = run_updaters<CL>(J, V, sc, xs, Ts, red, step, err);
            if (CL && r < 0) {
                left = true;
                break;
            }
            if (r) built = true;
        }
        int m = (int)min((int64_t)(J.stride - phase), last - step);   // steps to the next updater pass or the end
        step += m;
        phase = phase + m == J.stride ? 0 : phase + m;
        for (; m > 0; --m, ++s) {
            float4* xn = CL ? reinterpret_cast<float4*>(smem + lay.x) + (((s + 1) & 1) ? n + 2 : 0) : xs;
            const uint32_t bar = CL ? (uint32_t)__cvta_generic_to_shared(&bars[s & 1]) : 0u;
            if (CL && tid == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(16u * (uint32_t)(n - nb))
                             : "memory");
            int* counter = &next_task[s & 1];
            const char* xb = reinterpret_cast<const char*>(xs);
            // forces: a warp's first task is its own, the next ones it claims
            // from a shared counter (the claim in flight during the task before)
            for (int task = tid >> 5; task < tasks;) {
                int claim = tasks;
                if (more && lane == 0) claim = atomicAdd(counter, 1);
                if (task < tpairs) {
                    const int slot = task * per + group;
                    const int pl = CL ? slot : order[slot], bead = 2 * pl + g.h;   // local pair and bead
                    const RowHead hd = unpack_head(hdw[pl]);
                    const float4* xp = xs + (pl < npl ? b0 + 2 * pl : n);
                    const float4 x0 = xp[0], x1 = xp[1], xi = g.h ? x1 : x0;
                    const int o_own = hd.nf + (g.h ? hd.n0 : 0), n_own = g.h ? hd.n1 : hd.n0;
                    float3 fs, f;
                    if (__any_sync(0xffffffffu, hd.start == kRowGlobal)) {
                        const uint16_t* row = hd.start == kRowGlobal ? J.vr + (size_t)(p0 + pl) * J.cap_u : nbr + hd.start;
                        fs = row_both(row, hd.nf, g, xb, x0, x1, J.cut2);
                        f = row_own(row + o_own, n_own, g, xb, xi, J.cut2, J.c8);
                    } else {
                        fs = row_both(nbr + hd.start, hd.nf, g, xb, x0, x1, J.cut2);
                        f = row_own(nbr + hd.start + o_own, n_own, g, xb, xi, J.cut2, J.c8);
                    }
                    if (bonded) {
                        const ushort4 m = bh[bead];
                        const int step = g.own_lanes();
                        if (g.owns()) {
                            for (int k = m.x + g.lh; k < m.y; k += step) {
                                const uint2 c = cov_par[k];
                                fene_term(xi, bead_at(xb, (int)c.y), __uint_as_float(c.x), J.ks, J.R2, f);
                            }
                            for (int k = m.z + g.lh; k < m.w; k += step) native_term(xi, bead_at(xb, nat_j[k]), nat_par[k], f);
                        }
                    } else if (bead < nb) {
                        bonded_global(J, xs, b0 + bead, xi, g, f);
                    }
                    if (extra && J.discrete && bead < nb && g.owns()) mica_partial(J, b0 + bead, xi, g.lh, g.own_lanes(), f);
                    f = pair_total(fs, f, J.c8, g);
                    if (g.lh == 0 && bead < nb) {
                        if (extra) {
                            const int i = b0 + bead;
                            if (J.indent) {
                                float3 tf;
                                if (J.discrete) tip_term(xi, sc.ig, f, tf);
                                else indentation_term(xi, sc.ig, f, tf);
                                float4 t = J.tipF[i];
                                t.x += tf.x; t.y += tf.y; t.z += tf.z;
                                J.tipF[i] = t;
                            }
                            if (J.plane) {
                                const int mask = J.plane_mask[i];
                                if (mask) J.plane_f[i] = plane_term(J, sc.plane_displ, mask, xi, J.plane_r0[i], f);
                            }
                        }
                        F[bead] = make_float4(f.x, f.y, f.z, 0.f);
                    }
                } else if (CL) {
                    const int b = 32 * (task - tpairs) + lane;
                    if (b < nb) {
                        uint4 st = sd[b];
                        N[b] = gaussian4(st);
                        sd[b] = st;
                    }
                }
                task = more ? __shfl_sync(0xffffffffu, claim, 0) : tasks;
            }
            __syncthreads();
            if (tid == 0) *counter = warps;      // reused two steps from now, after a barrier
            // integrateLangevin_kernel (src/Integrators/langevin_kernel.cu:17-58),
            // one thread per bead: every force of the step is final
            for (int b = tid; b < nb; b += nt) {
                const float4 f4 = F[b];
                float3 f = make_float3(f4.x, f4.y, f4.z);
                if (!J.minimization) {
                    float4 gg;
                    if (CL) {
                        gg = N[b];
                    } else {
                        uint4 st = sd[b];
                        gg = gaussian4(st);
                        sd[b] = st;
                    }
                    const float var = sc.var;
                    f.x += gg.x * var;
                    f.y += gg.y * var;
                    f.z += gg.z * var;
                }
                const uint8_t fi = fl[b];
                if (fi == FLAG_FIXED) f = make_float3(0.f, 0.f, 0.f);
                if (fi == FLAG_PULLED) { f.x += sc.pullF[0]; f.y += sc.pullF[1]; f.z += sc.pullF[2]; }
                const float4 xi = xs[b0 + b];
                const float dx = J.hOverZeta * f.x, dy = J.hOverZeta * f.y, dz = J.hOverZeta * f.z;
                const float4 xw = make_float4(xi.x + dx, xi.y + dy, xi.z + dz, xi.w);
                xn[b0 + b] = xw;
                if (CL) {
                    const uint32_t a = (uint32_t)__cvta_generic_to_shared(&xn[b0 + b]);
                    for (int k = 1; k < C; ++k) {
                        const uint32_t r = (uint32_t)((rank + k) & (C - 1));
                        send16(map_rank(a, r), xw, map_rank(bar, r));
                    }
                }
                Ts[b] += J.tempNorm * (dx * dx + dy * dy + dz * dz);
            }
            if (CL) {
                xs = xn;
                if (!__syncthreads_and(peers_wait(bar, (s >> 1) & 1))) {
                    late = true;
                    break;
                }
            } else {
                __syncthreads();
            }
        }
        if (CL && late) break;
    }
    if (CL && late) give_up(&gave_up, C, step);
    if (CL && !left) cluster_arrive();
    if (built) store_rows(J, V);
    if (CL) {
        if (!left) cluster_wait();           // none sends any more
        if (gave_up_at(&gave_up) != kNeverStep) {
            // the bytes of the step that was given up land before the shared memory is released
            if (late) peers_wait((uint32_t)__cvta_generic_to_shared(&bars[s & 1]), (s >> 1) & 1);
            if (tid == 0 && rank == 0) Jp->nr_valid = 0;   // near rows may have been renewed
            if (tid == 0) atomicMax(&Jp->status, SOPB_ERR_TIMEOUT);
            return;
        }
    }
    for (int b = tid; b < nb; b += nt) {
        const int i = b0 + b;
        const float4 v = xs[i];
        if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) err = max(err, SOPB_STATUS_NONFINITE);
        J.x[i] = v;
        J.seeds[i] = sd[b];
        J.T[i] = Ts[b];
        if (CL && built && sc.nr_valid) J.x_ref[i] = V.xref[i];
    }
    if (err) atomicMax(&sc.err, err);
    __syncthreads();
    if (tid == 0) {
        if (rank == 0) {
            Jp->step = step;
            Jp->var = sc.var;
            for (int c = 0; c < 3; ++c) {
                Jp->pullF[c] = sc.pullF[c];
                Jp->cant[c] = sc.cant[c];
                Jp->tip[c] = sc.ig.tip[c];
                Jp->micaR[c] = sc.ig.micaR[c];
                Jp->chip[c] = sc.chip[c];
            }
            Jp->V = sc.V;
            Jp->dx = sc.dx;
            for (int c = 0; c < 4; ++c) Jp->fav[c] = sc.fav[c];
            Jp->nr_valid = sc.nr_valid;
            Jp->log_head = sc.log_head;
            Jp->plane_displ = sc.plane_displ;
            Jp->plane_cant = sc.plane_cant;
        }
        if (sc.err) atomicMax(&Jp->status, sc.err);
    }
}

// Potential forces only (SOPPotential::compute of every potential, no
// integrator) at the job's current coordinates and Verlet rows, with the
// step kernel's lane split; does not touch the tip accumulator.  blockIdx.y
// shares a job's beads.
__global__ void __launch_bounds__(1024, 1)
k_forces_only(const JobDev* __restrict__ jobs, const int32_t* __restrict__ ids, float4* __restrict__ out) {
    __shared__ JobDev Js;
    load_job(Js, &jobs[ids[blockIdx.x]]);
    __syncthreads();
    const JobDev& J = Js;
    const int n = J.n, tid = threadIdx.x;
    // rows per pair of beads: a lane group per pair; others: lpb lanes per bead
    const bool pairs = J.mask || J.gvr;
    const PairGroup<false> pg(J.lpb, tid & 31, 0);
    const int G = pairs ? pg.G : J.lpb, ng = blockDim.x / G, tasks = pairs ? job_pairs(n) : n;
    const int lh = pairs ? pg.lh : tid % G, h = pairs ? pg.h : 0;
    IndentGeom ig;
    for (int c = 0; c < 3; ++c) { ig.tip[c] = J.tip[c]; ig.micaR[c] = J.micaR[c]; ig.micaN[c] = J.micaN[c]; }
    ig.tipR = J.tipR; ig.tipAp = J.tipAp; ig.tipBp = J.tipBp; ig.surfAp = J.surfAp; ig.surfBp = J.surfBp;
    for (int base = blockIdx.y * ng; base < tasks; base += gridDim.y * ng) {
        const int t = base + tid / G, i = pairs ? 2 * t + h : t;
        const bool act = i < n;
        const float4 xi = J.x[act ? i : 0];
        float3 f = make_float3(0.f, 0.f, 0.f);
        if (pairs) {
            const int p = t < tasks ? t : 0;
            int nf = 0, n0 = 0, n1 = 0, start = 0;
            if (t < tasks && J.mask) {
                const RowHead hd = unpack_head(J.vh[p]);
                nf = hd.nf;
                n0 = hd.n0;
                n1 = hd.n1;
            } else if (t < tasks) {
                const int4 hd = J.gvh[p];
                nf = hd.x;
                n0 = hd.y;
                n1 = hd.z;
                start = hd.w;
            }
            const float4 x0 = J.x[2 * p], x1 = J.x[2 * p + 1 < n ? 2 * p + 1 : 2 * p];
            const char* xb = reinterpret_cast<const char*>(J.x);
            float3 fs;
            auto sums = [&](auto* row) {
                fs = row_both(row, nf, pg, xb, x0, x1, J.cut2);
                f = row_own(row + nf + (h ? n0 : 0), h ? n1 : n0, pg, xb, xi, J.cut2, J.c8);
            };
            if (J.mask) sums(J.vr + (size_t)p * J.cap_u);
            else sums(J.gvr + (size_t)(p / J.tile) * J.tile * J.cap_u + start);
            if (act) {
                bonded_global(J, J.x, i, xi, pg, f);
                if (J.discrete) mica_partial(J, i, xi, lh, pg.own_lanes(), f);
            }
            f = pair_total(fs, f, J.c8, pg);
        } else {
            if (act) {
                bonded_partial(J, J.x, i, xi, lh, G, f);
                pair_run(J, J.x, J.pl_j + (size_t)i * J.cap_pl, J.pl_cnt[i], xi, lh, G, f);
                if (J.discrete) mica_partial(J, i, xi, lh, G, f);
            }
            __syncwarp();
            f = group_reduce(f, G);
        }
        if (act && lh == 0) {
            if (J.indent) {
                float3 tf;
                if (J.discrete) tip_term(xi, ig, f, tf);
                else indentation_term(xi, ig, f, tf);
            }
            if (J.plane) {
                const int mask = J.plane_mask[i];
                if (mask) plane_term(J, J.plane_displ, mask, xi, J.plane_r0[i], f);
            }
            out[i] = make_float4(f.x, f.y, f.z, 0.f);
        }
    }
}

// Rebuilds the possible-pairs and/or Verlet lists of a job now, without the step
// gate: a cluster of CTAs with a share of its pairs each.  Bound by latency: a
// call that renews the Verlet rows of 600 beads takes 59 us, of 2000 beads 285
// (130 and 945 with one CTA and a row per bead; 200 and 2010 with one CTA).
__host__ __device__ inline int rebuild_ctas(int n) { return n >= 256 ? 8 : (n >= 64 ? 4 : 1); }
__global__ void __launch_bounds__(1024, 1)
k_rebuild_lists(JobDev* __restrict__ jobs, const int32_t* __restrict__ ids, int possible, int verlet) {
    const int C = (int)cluster_nctarank(), rank = (int)cluster_ctarank();
    JobDev* Jp = &jobs[ids[blockIdx.x / C]];
    __shared__ JobDev Js;
    load_job(Js, Jp);
    const JobDev& J = Js;
    __shared__ int errs;
    __shared__ int64_t gave_up;
    cluster_arrive();                        // this CTA has begun: its shared memory may be written
    if (threadIdx.x == 0) {
        errs = 0;
        gave_up = kNeverStep;
    }
    __syncthreads();
    int err = 0;
    const int p0 = pair_begin(J.n, rank, C), p1 = pair_begin(J.n, rank + 1, C);
    const PartView V{p0, p1, 2 * p0, min(J.n, 2 * p1), rank, C, nullptr, nullptr, 0, nullptr, J.x_ref, &gave_up};
    if (possible) build_possible(J, V, J.x, err);
    __syncthreads();
    cluster_wait();
    int valid = 0;
    if (verlet) rebuild_verlet<true>(J, V, J.x, valid, true, 0, err);   // a full scan, which also renews the near list
    // (without it the near list no longer matches the possible pairs)
    if ((verlet || possible) && rank == 0 && threadIdx.x == 0) Jp->nr_valid = valid;
    if (err) atomicMax(&errs, err);
    __syncthreads();
    if (threadIdx.x == 0 && errs) Jp->status = errs;
}

}  // namespace sopb
