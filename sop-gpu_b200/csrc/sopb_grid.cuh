// sopb_grid.cuh — the grid path: per-step kernels for jobs too large for one
// CTA (n > 2048 beads, e.g. a 198k-bead capsid shell) and for jobs with
// hydrodynamic interactions, whose O(N^2) sums need the whole GPU.
//
// One step of a job without hydrodynamics is one kernel (potentials, noise and
// move, from one coordinate buffer into the other); with them, a forces kernel
// followed by the integrator's.  Every `stride` steps the updater kernels run
// first; each reads the job's step counter on the device and returns at once
// when its frequency does not divide it, so a whole stride chunk is one fixed
// launch sequence that the host captures once in a CUDA graph and replays.  The
// step counter moves by `stride` in the chunk's last launch.
//
// Lists are index rows in global memory.  Verlet rows are per bead for jobs
// with hydrodynamics, per pair of beads without; possible pairs are per bead,
// for large jobs from a cell list (cells no smaller than pairs_threshold,
// 27-cell search, exact distance test) whose rows are then sorted, so that
// they equal the reference's brute-force rows
// (src/Updaters/possiblepairlist_kernel.cu:18-71) entry for entry.
#pragma once

#include "sopb_resident.cuh"

namespace sopb {

constexpr int kGridBlock = 256;
constexpr int kGridLpb = 4;      // lanes per bead of the observables' sums
constexpr int kForceLpb = 16;    // lanes per bead of k_g_forces
constexpr int kCellMax = 1 << 22;
constexpr int kSortCap = 2048;   // rows up to this length are sorted in registers

struct GridAux {
    int32_t n;           // beads
    // per-bead buffers of the grid path
    float4* F;           // potential forces of the current step (HI), or the second coordinate buffer
    // hydrodynamics (TEA / Cholesky)
    float4* rf;          // rho * g (random force)
    float4* mf;          // molecular force (+ pulling), then D F for Cholesky
    float4* xc;          // coordinate copy read during the O(N^2) sums
    float4* ci4;         // sum of squared normalised tensor rows (x,y,z), sum of entries (w)
    float* eps;          // per-bead epsilon share
    double* beta;        // beta' of the job (TEA), FP64
    float* tensor;       // Cholesky: (3n)^2 matrix, row-major
    int32_t ld;          // leading dimension of `tensor`
    float* linv;         // blocked Cholesky: inverses of the last two diagonal tiles' factors, 2 x 128 x 128
    float* plane_hi;     // blocked Cholesky: the solved tiles of the last two outer panels split into
    float* plane_lo;     //   TF32 hi and lo (bit patterns), [2 * plane_rows][plane_ld], by panel parity
    int32_t plane_rows;  // tile rows x 128
    int32_t plane_ld;    // outer-panel width in columns
    // reductions
    float4* part;        // per-CTA partial sums
    int32_t npart;
    // cell list
    int32_t* cell_count; // [kCellMax + 1]
    int32_t* cell_start; // [kCellMax + 1]
    int32_t* cell_beads; // [n]
    int32_t* bead_cell;  // [n]
    float* cell_geo;     // origin[3], size, dims[3] (as float), ncell
    int32_t use_cells;
    // near list of the Verlet rebuilds (null: none, every rebuild filters
    // the possible rows)
    int32_t* nr_j;       // [n * cap_nr] possible pairs within pairlist_cutoff + skin
    int32_t* nr_cnt;     // [n]
    float4* x_ref;       // coordinates it was built at
    int32_t* near;       // [4] drift bits, overflow, usable, not tried again
    int32_t cap_nr;
    // Verlet rows per pair of beads of a job without hydrodynamics (whose near
    // rows are per pair as well: nr_j and nr_cnt by pair)
    int4* vh;            // [ceil(n/2)] partners of both beads, of the first alone, of the second alone; start
    int32_t* vr;         // [tiles * tile * cap_u] the three sections of each row: 16 j.  The rows of a tile of
                         //   pairs lie one after another, each from its start on (tile 1: start 0)
    int32_t* vtot;       // [tiles] entries of a tile's rows
    int32_t cap_u, tile;
    // constants of a step
    float cut2, c8, ks, R2, hOverZeta, tempNorm;
    int32_t minimization, pulling, indent;
    const int32_t *cov_off, *cov_j, *nat_off, *nat_j;
    const float* cov_r0;
    const float2* nat_par;
};


__device__ __forceinline__ int64_t job_step(const JobDev* Jp) { return *(volatile const int64_t*)&Jp->step; }

// ---- potentials ------------------------------------------------------------
// Verlet-pair terms of bead i from its row (16-byte aligned), a group of
// kForceLpb lanes: lane l takes four entries with one 16-byte load, and the
// next block's indices are fetched before this block's four gathers, so the
// row load overlaps the coordinate gathers.  16 lanes, since only jobs with
// hydrodynamics come here, which rarely fill the GPU: k_g_forces takes 9.0 us
// at 517 beads and 9.5 at 4000 (14.4 and 16.1 with 4 lanes).
__device__ __forceinline__ void pair_row_v4(const JobDev& J, const float4* __restrict__ xs,
                                            const int32_t* __restrict__ row, int cnt, float4 xi, int l, float3& f) {
    const float c8 = J.c8, cut2 = J.cut2;
    const int4* __restrict__ r4 = reinterpret_cast<const int4*>(row);
    int k = 4 * l;
    int4 nx = make_int4(0, 0, 0, 0);
    if (k < cnt) nx = __ldg(r4 + l);
    for (; k < cnt; k += 4 * kForceLpb) {
        const int4 cur = nx;
        if (k + 4 * kForceLpb < cnt) nx = __ldg(r4 + (k >> 2) + kForceLpb);
        if (k + 3 < cnt) {
            const float4 x0 = xs[cur.x], x1 = xs[cur.y], x2 = xs[cur.z], x3 = xs[cur.w];
            pair_term(xi, x0, c8, cut2, f);
            pair_term(xi, x1, c8, cut2, f);
            pair_term(xi, x2, c8, cut2, f);
            pair_term(xi, x3, c8, cut2, f);
        } else {
            pair_term(xi, xs[cur.x], c8, cut2, f);
            if (k + 1 < cnt) pair_term(xi, xs[cur.y], c8, cut2, f);
            if (k + 2 < cnt) pair_term(xi, xs[cur.z], c8, cut2, f);
        }
    }
}

// integrateTea_prepare (bdhitea_kernel.cu:33-65): the random force rho g, the
// molecular force with pulling applied and a copy of the coordinates.
__device__ __forceinline__ void hi_prepare(const JobDev& J, const GridAux& aux, int i, float4 xi, float3 f) {
    uint4 st = J.seeds[i];
    float4 g = gaussian4(st);
    J.seeds[i] = st;
    g.x *= J.var;
    g.y *= J.var;
    g.z *= J.var;
    aux.rf[i] = g;
    if (J.pulling) {
        const uint8_t fl = J.flags[i];
        if (fl == FLAG_FIXED) f.x = f.y = f.z = 0.f;
        if (fl == FLAG_PULLED) { f.x += J.pullF[0]; f.y += J.pullF[1]; f.z += J.pullF[2]; }
    }
    aux.mf[i] = make_float4(f.x, f.y, f.z, 0.f);
    aux.xc[i] = xi;
}

// The tip's and the plane's terms of bead i (and the tip's share accumulated
// per bead, indentation_kernel.cu:71-128).
template <bool EXT>
__device__ __forceinline__ void external_terms(const JobDev& J, int i, float4 xi, float3& f) {
    if (J.indent) {
        // read from the shared copy here, not held in registers over the pair loop
        IndentGeom ig;
        for (int c = 0; c < 3; ++c) { ig.tip[c] = J.tip[c]; ig.micaR[c] = J.micaR[c]; ig.micaN[c] = J.micaN[c]; }
        ig.tipR = J.tipR; ig.tipAp = J.tipAp; ig.tipBp = J.tipBp; ig.surfAp = J.surfAp; ig.surfBp = J.surfBp;
        float3 tf;
        if (EXT && J.discrete) tip_term(xi, ig, f, tf);
        else indentation_term(xi, ig, f, tf);
        float4 t = J.tipF[i];
        t.x += tf.x; t.y += tf.y; t.z += tf.z;
        J.tipF[i] = t;
    }
    if (EXT && J.plane) {
        const int mask = J.plane_mask[i];
        if (mask) J.plane_f[i] = plane_term(J, J.plane_displ, mask, xi, J.plane_r0[i], f);
    }
}

// All potentials of every bead of a job with hydrodynamics at the current
// coordinates, into aux.F or (PREP) prepared for the O(N^2) sums.
// EXT: the job has a discrete surface or a pulling plane (a separate
// instantiation, so the common one keeps its register budget).
template <bool EXT, bool PREP>
__global__ void __launch_bounds__(kGridBlock)
k_g_forces(JobDev* __restrict__ Jp, GridAux aux) {
    __shared__ JobDev Js;
    load_job<kGridBlock>(Js, Jp);
    __syncthreads();
    const JobDev& J = Js;
    if (J.status) return;
    const int lpb = kForceLpb, l = threadIdx.x % lpb;
    const int groups = gridDim.x * (kGridBlock / lpb);
    const int g0 = blockIdx.x * (kGridBlock / lpb) + threadIdx.x / lpb;
    for (int base = 0; base < J.n; base += groups) {
        const int i = base + g0;
        const bool act = i < J.n;
        const float4 xi = J.x[act ? i : 0];
        float3 f = make_float3(0.f, 0.f, 0.f);
        if (act) {
            bonded_partial(J, J.x, i, xi, l, lpb, f);
            if ((J.cap_pl & 3) == 0) pair_row_v4(J, J.x, J.pl_j + (size_t)i * J.cap_pl, J.pl_cnt[i], xi, l, f);
            else pair_run(J, J.x, J.pl_j + (size_t)i * J.cap_pl, J.pl_cnt[i], xi, l, lpb, f);
            if (EXT && J.discrete) mica_partial(J, i, xi, l, lpb, f);
        }
        f = group_reduce(f, lpb);
        if (act && l == 0) {
            external_terms<EXT>(J, i, xi, f);
            if (PREP) hi_prepare(J, aux, i, xi, f);
            else aux.F[i] = make_float4(f.x, f.y, f.z, 0.f);
        }
    }
}

// ---- one step without hydrodynamics -----------------------------------------
// All potentials and the Langevin move (langevin_kernel.cu:17-58) from `xin`
// into `xout`.  A lane group per pair of beads, in the resident kernel's order
// of sums: the partners of both beads by the whole group, each bead's own by
// its half, with its covalent and native terms; then a thread per bead draws
// the noise and moves the bead.  One gather serves two beads.
//
// Bound by the latency of the chain header -> entries -> coordinates, not by
// bytes: the gathers hit L1 and L2.  Wide groups (16 lanes a pair) shorten a
// lane's chain and fetch the entries ahead, before the header is there; narrow
// groups (8 lanes) do less work per pair, and their CTA's rows, which lie one
// after another, arrive in shared memory by one bulk copy while the bonded
// terms are computed.
//
// Wide CTAs take 32 beads, and three of them fit an SM (80 registers): up to
// 148 x 3 x 32 = 14208 beads they run in one wave.  Above, narrow steps are
// faster (per step of 200, rebuilds included; clamped globules, 20 A lists):
// 12000 beads 10.7 us wide, 14.3 narrow; 18000 beads 15.6 and 13.4, a shell of
// 18000 beads 15.8 and 10.9; 24000 beads 17.2 and 15.1.  With a lane group per
// bead and the integrator as a kernel of its own: 14.4, 15.8, 14.8 and 18.5.
// A clamped chain of 5011 beads takes 10.5 us per step, 14.0 before; a
// 198000-bead shell 102 us, 126 before (88 + 6 us under the profiler, now 70).
constexpr int kWideStepBeads = 14208;
__host__ __device__ constexpr int step_pairs(bool wide) { return kGridBlock / (wide ? 16 : 8); }   // pairs per CTA
// Row entries per pair that a CTA has shared memory for: four CTAs' share of an
// SM.  A tile whose rows are longer reads them from global memory (40000 beads
// with 26 and 32 A lists: 15.1 and 21.9 us per step, 20.0 and 32.5 with a lane
// group per bead).
constexpr int kStepRow = 192;
constexpr uint32_t kStepWaitLimit = 1u << 20;

// Entries [k0 + l, k1) of a row in steps of G, four gathers in flight:
// term(u, coordinates) for the u-th of four.
template <typename Term>
__device__ __forceinline__ void gather4(const int32_t* row, int k, int k1, int G, const char* xb, Term term) {
    for (; k + 3 * G < k1; k += 4 * G) {
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = bead_at(xb, row[k + u * G]);
#pragma unroll
        for (int u = 0; u < 4; ++u) term(u, q[u]);
    }
    float4 q[3];
#pragma unroll
    for (int u = 0; u < 3; ++u)
        if (k + u * G < k1) q[u] = bead_at(xb, row[k + u * G]);
#pragma unroll
    for (int u = 0; u < 3; ++u)
        if (k + u * G < k1) term(u, q[u]);
}

template <bool EXT, bool WIDE>
__global__ void __launch_bounds__(kGridBlock, WIDE ? 3 : 4)
k_g_step(JobDev* __restrict__ Jp, const GridAux aux, const float4* __restrict__ xin, float4* __restrict__ xout) {
    constexpr int G = WIDE ? 16 : 8, kPairs = step_pairs(WIDE);
    __shared__ float4 Fs[2 * kPairs];
    __shared__ __align__(128) int32_t rows_s[WIDE ? 4 : kPairs * kStepRow];
    __shared__ __align__(8) uint64_t bar_s;
    __shared__ int in_smem;
    const int tid = threadIdx.x, n = aux.n;
    const int p0 = blockIdx.x * kPairs, p = p0 + tid / G;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&bar_s);
    const int32_t* rows_g = aux.vr + (size_t)(WIDE ? p : p0) * aux.cap_u;
    // the CTA's rows into shared memory with one bulk copy, if they fit
    if (!WIDE && tid == 0) {
        const int total = aux.vtot[blockIdx.x];
        in_smem = total <= kPairs * kStepRow;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        const uint32_t bytes = in_smem ? 4u * (uint32_t)total : 0u;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        if (bytes)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(rows_s)),
                         "l"(rows_g), "r"(bytes), "r"(bar)
                         : "memory");
    }
    const PairGroup<WIDE> g(4, tid & 31, G);
    const int i = 2 * p + g.h;
    const bool act = i < n;
    const char* xb = reinterpret_cast<const char*>(xin);
    const int own = g.own_lanes();
    // meanwhile the row's header, the two beads and the bead's maps
    const int status = Jp->status;
    int4 hd = make_int4(0, 0, 0, 0);
    float4 x0 = make_float4(1.0e18f, 1.0e18f, 1.0e18f, 0.f), x1 = x0;
    int c0 = 0, c1 = 0, n0 = 0, n1 = 0;
    int pre[WIDE ? 4 : 1];
    if (WIDE)                              // readable whatever the row's length
#pragma unroll
        for (int u = 0; u < 4; ++u) pre[u] = 2 * p < n ? rows_g[min(g.l + u * G, aux.cap_u - 1)] : 0;
    if (2 * p < n) {
        hd = aux.vh[p];
        x0 = xin[2 * p];
        if (2 * p + 1 < n) x1 = xin[2 * p + 1];
    }
    if (act && g.owns()) {
        c0 = aux.cov_off[i] + g.lh;
        c1 = aux.cov_off[i + 1];
        n0 = aux.nat_off[i] + g.lh;
        n1 = aux.nat_off[i + 1];
    }
    const float4 xi = g.h ? x1 : x0;
    const int k_own = hd.x + (g.h ? hd.y : 0) + g.lh, e_own = hd.x + hd.y + (g.h ? hd.z : 0);
    int w[WIDE ? 4 : 1];
    if (WIDE)
#pragma unroll
        for (int u = 0; u < 4; ++u) w[u] = g.owns() && k_own + u * own < e_own ? rows_g[k_own + u * own] : -1;
    // the first bond and the first two contacts of the lane
    int cj = 0, nj0 = 0, nj1 = 0;
    float cr = 0.f;
    float2 np0 = make_float2(0.f, 0.f), np1 = np0;
    if (c0 < c1) {
        cj = aux.cov_j[c0];
        cr = aux.cov_r0[c0];
    }
    if (n0 < n1) {
        nj0 = aux.nat_j[n0];
        np0 = aux.nat_par[n0];
    }
    if (n0 + own < n1) {
        nj1 = aux.nat_j[n0 + own];
        np1 = aux.nat_par[n0 + own];
    }
    float3 fb = make_float3(0.f, 0.f, 0.f);
    auto bonded = [&] {
        const float4 qc = xin[cj], q0 = xin[nj0], q1 = xin[nj1];
        if (c0 < c1) fene_term(xi, qc, cr, aux.ks, aux.R2, fb);
        if (n0 < n1) native_term(xi, q0, np0, fb);
        if (n0 + own < n1) native_term(xi, q1, np1, fb);
        for (int k = c0 + own; k < c1; k += own) fene_term(xi, xin[aux.cov_j[k]], aux.cov_r0[k], aux.ks, aux.R2, fb);
        for (int k = n0 + 2 * own; k < n1; k += own) native_term(xi, xin[aux.nat_j[k]], aux.nat_par[k], fb);
    };
    if (!WIDE) bonded();                   // they do not need the rows
    if (EXT && act && g.owns() && Jp->discrete) mica_partial(*Jp, i, xi, g.lh, own, fb);
    if (!WIDE) {
        __syncthreads();                       // the barrier is set up
        bool there = false;
        for (uint32_t it = 0; it < kStepWaitLimit && !there; ++it) {
            uint32_t ok;
            asm volatile(
                "{\n\t.reg .pred P1;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], 0;\n\t"
                "selp.b32 %0, 1, 0, P1;\n\t}\n"
                : "=r"(ok)
                : "r"(bar)
                : "memory");
            there = ok;
        }
        if (!__syncthreads_and(there && !status)) {
            if (!there) atomicMax(&Jp->status, SOPB_ERR_TIMEOUT);   // the copy did not arrive
            return;
        }
    }
    // a narrow CTA voted, since another one may set the status meanwhile; no
    // CTA of a wide step does, nor anything beside it on the job's stream
    if (WIDE && status) return;
    const float cut2 = aux.cut2;
    const float3 zero = make_float3(0.f, 0.f, 0.f);
    float3 a0 = zero, a1 = zero, b0 = zero, b1 = zero, f = zero;
    auto both = [&](int u, float4 q) {
        pair_term8(x0, q, cut2, WIDE || u % 2 == 0 ? a0 : b0);
        pair_term8(x1, q, cut2, WIDE || u % 2 == 0 ? a1 : b1);
    };
    auto single = [&](int, float4 q) { pair_term8(xi, q, cut2, f); };
    if (WIDE) {
        // four entries of the lane at a time, the next ones fetched before
        // these ones' gathers are used
        for (int k = g.l; k < hd.x; k += 4 * G) {
            int o[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) o[u] = k + u * G < hd.x ? pre[u] : -1;
            if (k + 4 * G < hd.x) {
#pragma unroll
                for (int u = 0; u < 4; ++u) pre[u] = rows_g[min(k + (4 + u) * G, aux.cap_u - 1)];
            }
            float4 q[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (o[u] >= 0) q[u] = bead_at(xb, o[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (o[u] >= 0) both(u, q[u]);
        }
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (w[u] >= 0) q[u] = bead_at(xb, w[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (w[u] >= 0) single(u, q[u]);
        if (g.owns()) gather4(rows_g, k_own + 4 * own, e_own, own, xb, single);
        bonded();
    } else {
        auto sums = [&](const int32_t* row) {
            gather4(row, g.l, hd.x, G, xb, both);
            gather4(row, k_own, e_own, own, xb, single);
        };
        if (in_smem) sums(rows_s + hd.w);
        else sums(rows_g + hd.w);
    }
    const float3 fs = pair_sum(g, a0, a1, b0, b1);
    f = make_float3(fmaf(aux.c8, f.x, fb.x), fmaf(aux.c8, f.y, fb.y), fmaf(aux.c8, f.z, fb.z));
    f = pair_total(fs, f, aux.c8, g);
    if (g.lh == 0 && act) {
        if (EXT || aux.indent) external_terms<EXT>(*Jp, i, xi, f);
        Fs[i - 2 * p0] = make_float4(f.x, f.y, f.z, 0.f);
    }
    __syncthreads();
    const int b = 2 * p0 + tid;
    if (tid < 2 * kPairs && b < n) {
        f = make_float3(Fs[tid].x, Fs[tid].y, Fs[tid].z);
        if (!aux.minimization) {
            uint4 st = Jp->seeds[b];
            const float var = Jp->var;
            const float4 gg = gaussian4(st);
            Jp->seeds[b] = st;
            f.x += gg.x * var;
            f.y += gg.y * var;
            f.z += gg.z * var;
        }
        if (aux.pulling) {
            const uint8_t fl = Jp->flags[b];
            if (fl == FLAG_FIXED) f = make_float3(0.f, 0.f, 0.f);
            if (fl == FLAG_PULLED) { f.x += Jp->pullF[0]; f.y += Jp->pullF[1]; f.z += Jp->pullF[2]; }
        }
        const float4 xi0 = xin[b];
        const float dx = aux.hOverZeta * f.x, dy = aux.hOverZeta * f.y, dz = aux.hOverZeta * f.z;
        xout[b] = make_float4(xi0.x + dx, xi0.y + dy, xi0.z + dz, xi0.w);
        Jp->T[b] += aux.tempNorm * (dx * dx + dy * dy + dz * dz);
    }
}

// The coordinates after an odd number of steps, back into the job's own buffer
// (a failed job's steps wrote nothing: it keeps its coordinates).
__global__ void __launch_bounds__(kGridBlock)
k_g_copy_back(JobDev* __restrict__ Jp, const float4* __restrict__ x) {
    const JobDev& J = *Jp;
    if (J.status) return;
    for (int i = blockIdx.x * kGridBlock + threadIdx.x; i < J.n; i += gridDim.x * kGridBlock) J.x[i] = x[i];
}

// ---- updaters ----------------------------------------------------------------
// Tip force: per-CTA partial sums of the per-bead accumulators (zeroed).
__global__ void __launch_bounds__(kGridBlock)
k_g_tip_partial(JobDev* __restrict__ Jp, GridAux aux) {
    __shared__ float red[kGridBlock / 32][4];
    const int64_t step = job_step(Jp);
    const JobDev& J = *Jp;
    if (!J.indent || J.status || step % J.stride != 0 || step % J.nav != 0) return;
    float3 p = make_float3(0.f, 0.f, 0.f);
    for (int i = blockIdx.x * kGridBlock + threadIdx.x; i < J.n; i += gridDim.x * kGridBlock) {
        float4 t = J.tipF[i];
        p.x += t.x; p.y += t.y; p.z += t.z;
        J.tipF[i] = make_float4(0.f, 0.f, 0.f, t.w);
    }
    const float3 s = block_sum3<kGridBlock>(p, red);
    if (threadIdx.x == 0) aux.part[blockIdx.x] = make_float4(s.x, s.y, s.z, 0.f);
}

// One thread: the remaining host-side updaters of the reference in order
// (indentation tip, force-ramp cantilever, heating), reading their state
// from and writing it back to the descriptor.
__global__ void k_g_scalar_updaters(JobDev* __restrict__ Jp, GridAux aux) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    JobDev& J = *Jp;
    const int64_t step = job_step(Jp);
    if (J.status || step % J.stride != 0) return;
    StepScalars sc;
    sc.var = J.var;
    for (int c = 0; c < 3; ++c) {
        sc.pullF[c] = J.pullF[c]; sc.cant[c] = J.cant[c]; sc.chip[c] = J.chip[c];
        sc.ig.tip[c] = J.tip[c]; sc.ig.micaR[c] = J.micaR[c]; sc.ig.micaN[c] = J.micaN[c];
    }
    sc.V = J.V;
    sc.dx = J.dx;
    for (int c = 0; c < 4; ++c) sc.fav[c] = J.fav[c];
    sc.log_head = J.log_head;
    sc.plane_displ = J.plane_displ;
    sc.plane_cant = J.plane_cant;
    if (J.indent) {
        if (step == J.retraction_step) sc.V = -sc.V;
        if (step % J.nav == 0) {
            float3 s = make_float3(0.f, 0.f, 0.f);
            for (int b = 0; b < aux.npart; ++b) { float4 q = aux.part[b]; s.x += q.x; s.y += q.y; s.z += q.z; }
            tip_update(J, sc, s, step);
        }
    }
    if (J.pulling && J.ramp) {
        const float xt = __fmul_rn(J.deltax, (float)(step / J.pull_freq));
        const float4 xe = J.x[J.pulledEnd];
        const float xe3[3] = {xe.x, xe.y, xe.z};
        for (int c = 0; c < 3; ++c) sc.pullF[c] = __fmul_rn(J.k_trans, __fsub_rn(sc.cant[c], xe3[c]));
        for (int c = 0; c < 3; ++c) sc.cant[c] = __fadd_rn(J.cant0[c], __fmul_rn(xt, J.pullvec[c]));
        if (step % J.pull_freq == 0) log_pull(J, sc, xe, J.x[J.fixedEnd], step);
    }
    if (J.plane) plane_update(J, sc, J.x, step);
    if (J.heating && step % J.temp_freq == 0) {
        const float temp = __fadd_rn(J.initialT, __fmul_rn((float)(step / J.temp_freq), J.deltaT));
        sc.var = __fsqrt_rn(__fdiv_rn(__fmul_rn(__fmul_rn(2.0f, temp), J.zeta), J.h));
    }
    J.var = sc.var;
    for (int c = 0; c < 3; ++c) {
        J.pullF[c] = sc.pullF[c]; J.cant[c] = sc.cant[c]; J.chip[c] = sc.chip[c];
        J.tip[c] = sc.ig.tip[c]; J.micaR[c] = sc.ig.micaR[c];
    }
    J.V = sc.V;
    J.dx = sc.dx;
    for (int c = 0; c < 4; ++c) J.fav[c] = sc.fav[c];
    J.log_head = sc.log_head;
    J.plane_displ = sc.plane_displ;
    J.plane_cant = sc.plane_cant;
}

// Discrete surface at a tip update (after k_g_scalar_updaters moved dx):
// the surface beads follow dx when the surface moves (indentation.cu:446-455).
__global__ void __launch_bounds__(kGridBlock)
k_g_surf_move(JobDev* __restrict__ Jp) {
    const int64_t step = job_step(Jp);
    const JobDev& J = *Jp;
    if (!J.indent || !J.discrete || !J.moveSurface || J.status || step % J.stride != 0 || step % J.nav != 0) return;
    const float dx = J.dx;
    for (int q = blockIdx.x * kGridBlock + threadIdx.x; q < J.nsurf; q += gridDim.x * kGridBlock) {
        const float4 s0 = J.surf0[q];
        J.surf[q] = make_float4(__fadd_rn(s0.x, __fmul_rn(J.dir[0], dx)), __fadd_rn(s0.y, __fmul_rn(J.dir[1], dx)),
                                __fadd_rn(s0.z, __fmul_rn(J.dir[2], dx)), 0.f);
    }
}

// Every bead's surface-bead list (generateMicaList_kernel,
// indentation_kernel.cu:182-201) as a bitmask row, a warp per bead.
__global__ void __launch_bounds__(kGridBlock)
k_g_mica(JobDev* __restrict__ Jp) {
    const int64_t step = job_step(Jp);
    const JobDev& J = *Jp;
    if (!J.indent || !J.discrete || J.status || step % J.stride != 0 || step % J.nav != 0) return;
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (kGridBlock / 32);
    for (int i = blockIdx.x * (kGridBlock / 32) + (threadIdx.x >> 5); i < J.n; i += warps) {
        const float4 xi = J.x[i];
        uint32_t* row = J.mica + (size_t)i * J.Wm;
        for (int wd = 0; wd < J.Wm; ++wd) {
            const int q = 32 * wd + lane;
            const bool in = q < J.nsurf && dist2_rn(xi, J.surf[q]) < J.mica_cut2;
            const uint32_t m = __ballot_sync(0xffffffffu, in);
            if (lane == 0) row[wd] = m;
        }
    }
}

// Temperature-accumulator reset at nav (output_manager.cu:125-127).
__global__ void k_g_treset(JobDev* __restrict__ Jp) {
    const int64_t step = job_step(Jp);
    const JobDev& J = *Jp;
    if (J.status || step % J.stride != 0 || step % J.nav != 0) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < J.n; i += gridDim.x * blockDim.x) J.T[i] = 0.f;
}

// Possible pairs by brute force, one group of lanes per bead, order kept by
// ballot compaction (possiblepairlist_kernel.cu:18-71).
__global__ void __launch_bounds__(kGridBlock)
k_g_possible_brute(JobDev* __restrict__ Jp, int force) {
    __shared__ JobDev Js;
    load_job<kGridBlock>(Js, Jp);
    __syncthreads();
    const JobDev& J = Js;
    const int64_t step = J.step;
    if (J.status || (!force && (step % J.stride != 0 || step % J.pp_freq != 0))) return;
    const int lpb = 32, l = threadIdx.x % 32, n = J.n;
    int err = 0;
    for (int i = blockIdx.x * (kGridBlock / 32) + threadIdx.x / 32; i < n; i += gridDim.x * (kGridBlock / 32)) {
        const float4 xi = J.x[i];
        int32_t* row = J.pp_j + (size_t)i * J.cap_pp;
        int cnt = 0;
        const int c0 = J.cov_off[i], c1 = J.cov_off[i + 1], n0 = J.nat_off[i], n1 = J.nat_off[i + 1];
        for (int qb = 0; qb < n; qb += lpb) {
            const int q = qb + l;
            bool ok = q < n && q != i && within_cutoff(xi, J.x[q < n ? q : 0], J.pp_t);
            if (ok) {
                for (int k = c0; k < c1 && ok; ++k) ok = J.cov_j[k] != q;
                for (int k = n0; k < n1 && ok; ++k) ok = J.nat_j[k] != q;
            }
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            if (ok) {
                const int pos = cnt + __popc(m & ((1u << l) - 1u));
                if (pos < J.cap_pp) row[pos] = q;
                else err = SOPB_STATUS_CAPACITY;
            }
            cnt += __popc(m);
        }
        if (l == 0) J.pp_cnt[i] = cnt < J.cap_pp ? cnt : J.cap_pp;
    }
    if (err) atomicMax(&Jp->status, err);
}

// ---- cell list (large systems) ------------------------------------------------
__global__ void __launch_bounds__(kGridBlock)
k_cl_bounds(JobDev* __restrict__ Jp, GridAux aux, int force) {
    __shared__ float red[6][kGridBlock / 32];
    const JobDev& J = *Jp;
    const int64_t step = job_step(Jp);
    if (J.status || (!force && (step % J.stride != 0 || step % J.pp_freq != 0))) return;
    float mn[3] = {3.4e38f, 3.4e38f, 3.4e38f}, mx[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
    for (int i = blockIdx.x * kGridBlock + threadIdx.x; i < J.n; i += gridDim.x * kGridBlock) {
        const float4 x = J.x[i];
        const float v[3] = {x.x, x.y, x.z};
        for (int c = 0; c < 3; ++c) { mn[c] = fminf(mn[c], v[c]); mx[c] = fmaxf(mx[c], v[c]); }
    }
    for (int o = 16; o > 0; o >>= 1)
        for (int c = 0; c < 3; ++c) {
            mn[c] = fminf(mn[c], __shfl_xor_sync(0xffffffffu, mn[c], o));
            mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], o));
        }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int c = 0; c < 3; ++c) { red[c][w] = mn[c]; red[3 + c][w] = mx[c]; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 1; q < kGridBlock / 32; ++q)
            for (int c = 0; c < 3; ++c) { red[c][0] = fminf(red[c][0], red[c][q]); red[3 + c][0] = fmaxf(red[3 + c][0], red[3 + c][q]); }
        aux.part[blockIdx.x] = make_float4(red[0][0], red[1][0], red[2][0], 0.f);
        aux.part[gridDim.x + blockIdx.x] = make_float4(red[3][0], red[4][0], red[5][0], 0.f);
    }
}

// Cell geometry: cells no smaller than the threshold (slightly enlarged so a
// pair closer than the threshold is never two cells apart), at most kCellMax.
// One warp: its lanes share the partial bounds (13 us for 198000 beads; 113
// when one thread read them all).
__global__ void k_cl_geometry(JobDev* __restrict__ Jp, GridAux aux, int nparts, int force) {
    const JobDev& J = *Jp;
    const int64_t step = job_step(Jp);
    if (J.status || (!force && (step % J.stride != 0 || step % J.pp_freq != 0))) return;
    float mn[3] = {3.4e38f, 3.4e38f, 3.4e38f}, mx[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
    for (int b = threadIdx.x; b < nparts; b += 32) {
        const float4 a = aux.part[b], z = aux.part[nparts + b];
        mn[0] = fminf(mn[0], a.x); mn[1] = fminf(mn[1], a.y); mn[2] = fminf(mn[2], a.z);
        mx[0] = fmaxf(mx[0], z.x); mx[1] = fmaxf(mx[1], z.y); mx[2] = fmaxf(mx[2], z.z);
    }
    for (int o = 16; o > 0; o >>= 1)
        for (int c = 0; c < 3; ++c) {
            mn[c] = fminf(mn[c], __shfl_xor_sync(0xffffffffu, mn[c], o));
            mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], o));
        }
    if (threadIdx.x != 0) return;
    float size = J.pp_thr * 1.0001f + 1e-3f;
    int dims[3] = {1, 1, 1};
    bool ok = true;
    for (int c = 0; c < 3; ++c) ok = ok && isfinite(mn[c]) && isfinite(mx[c]) && mx[c] >= mn[c];
    if (!ok) {   // non-finite coordinates: one cell; the job is flagged after the step
        atomicMax(&Jp->status, SOPB_STATUS_NONFINITE);
        for (int c = 0; c < 3; ++c) mn[c] = 0.f;
    } else {
        for (int it = 0; it < 200; ++it) {   // bounded: each round grows the cells by 25%
            double tot = 1.0;
            for (int c = 0; c < 3; ++c) {
                dims[c] = (int)fminf(floorf((mx[c] - mn[c]) / size) + 1.0f, (float)kCellMax);
                tot *= dims[c];
            }
            if (tot <= (double)kCellMax) break;
            size *= 1.25f;
        }
        double tot = (double)dims[0] * dims[1] * dims[2];
        if (tot > (double)kCellMax) { dims[0] = dims[1] = dims[2] = 1; size = 3.0e38f; }
    }
    for (int c = 0; c < 3; ++c) aux.cell_geo[c] = mn[c];
    aux.cell_geo[3] = size;
    for (int c = 0; c < 3; ++c) aux.cell_geo[4 + c] = (float)dims[c];
    aux.cell_geo[7] = (float)(dims[0] * dims[1] * dims[2]);
}

__device__ __forceinline__ int cell_coord(float v, float o, float size, int dim) {
    int c = (int)floorf((v - o) / size);
    return c < 0 ? 0 : (c >= dim ? dim - 1 : c);
}

__global__ void __launch_bounds__(kGridBlock)
k_cl_count(JobDev* __restrict__ Jp, GridAux aux, int force) {
    const JobDev& J = *Jp;
    const int64_t step = job_step(Jp);
    if (J.status || (!force && (step % J.stride != 0 || step % J.pp_freq != 0))) return;
    const float o0 = aux.cell_geo[0], o1 = aux.cell_geo[1], o2 = aux.cell_geo[2], sz = aux.cell_geo[3];
    const int d0 = (int)aux.cell_geo[4], d1 = (int)aux.cell_geo[5], d2 = (int)aux.cell_geo[6];
    for (int i = blockIdx.x * kGridBlock + threadIdx.x; i < J.n; i += gridDim.x * kGridBlock) {
        const float4 x = J.x[i];
        const int c = (cell_coord(x.z, o2, sz, d2) * d1 + cell_coord(x.y, o1, sz, d1)) * d0 + cell_coord(x.x, o0, sz, d0);
        aux.bead_cell[i] = c;
        atomicAdd(&aux.cell_count[c], 1);
    }
}

// Exclusive scan of the cell counts (one CTA); cell_count becomes the fill
// cursor.
__global__ void __launch_bounds__(1024)
k_cl_scan(JobDev* __restrict__ Jp, GridAux aux, int force) {
    __shared__ int32_t tot[1024];
    const JobDev& J = *Jp;
    const int64_t step = job_step(Jp);
    if (J.status || (!force && (step % J.stride != 0 || step % J.pp_freq != 0))) return;
    const int nc = (int)aux.cell_geo[7];
    const int per = (nc + 1023) / 1024;
    const int b0 = threadIdx.x * per, b1 = min(nc, b0 + per);
    int32_t s = 0;
    for (int c = b0; c < b1; ++c) s += aux.cell_count[c];
    tot[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int32_t run = 0;
        for (int t = 0; t < 1024; ++t) { const int32_t v = tot[t]; tot[t] = run; run += v; }
        aux.cell_start[nc] = run;
    }
    __syncthreads();
    int32_t run = tot[threadIdx.x];
    for (int c = b0; c < b1; ++c) {
        const int32_t v = aux.cell_count[c];
        aux.cell_start[c] = run;
        aux.cell_count[c] = run;
        run += v;
    }
}

__global__ void __launch_bounds__(kGridBlock)
k_cl_fill(JobDev* __restrict__ Jp, GridAux aux, int force) {
    const JobDev& J = *Jp;
    const int64_t step = job_step(Jp);
    if (J.status || (!force && (step % J.stride != 0 || step % J.pp_freq != 0))) return;
    for (int i = blockIdx.x * kGridBlock + threadIdx.x; i < J.n; i += gridDim.x * kGridBlock) {
        const int pos = atomicAdd(&aux.cell_count[aux.bead_cell[i]], 1);
        aux.cell_beads[pos] = i;
    }
}

// Candidates from the 27 neighbouring cells with the exact test, appended
// unordered; one warp per bead.  Cells side by side in x hold their beads in
// one run of the array, so there are nine runs to walk (1.59 ms for the
// 198000-bead shell, 1.87 cell by cell).
__global__ void __launch_bounds__(kGridBlock)
k_cl_possible(JobDev* __restrict__ Jp, GridAux aux, int force) {
    __shared__ JobDev Js;
    load_job<kGridBlock>(Js, Jp);
    __syncthreads();
    const JobDev& J = Js;
    const int64_t step = J.step;
    if (J.status || (!force && (step % J.stride != 0 || step % J.pp_freq != 0))) return;
    const int l = threadIdx.x & 31;
    const float o0 = aux.cell_geo[0], o1 = aux.cell_geo[1], o2 = aux.cell_geo[2], sz = aux.cell_geo[3];
    const int d0 = (int)aux.cell_geo[4], d1 = (int)aux.cell_geo[5], d2 = (int)aux.cell_geo[6];
    int err = 0;
    for (int i = blockIdx.x * (kGridBlock / 32) + threadIdx.x / 32; i < J.n; i += gridDim.x * (kGridBlock / 32)) {
        const float4 xi = J.x[i];
        const int cx = cell_coord(xi.x, o0, sz, d0), cy = cell_coord(xi.y, o1, sz, d1), cz = cell_coord(xi.z, o2, sz, d2);
        const int c0 = J.cov_off[i], c1 = J.cov_off[i + 1], n0 = J.nat_off[i], n1 = J.nat_off[i + 1];
        int32_t* row = J.pp_j + (size_t)i * J.cap_pp;
        int cnt = 0;
        for (int dz = -1; dz <= 1; ++dz) {
            const int z = cz + dz;
            if (z < 0 || z >= d2) continue;
            for (int dy = -1; dy <= 1; ++dy) {
                const int y = cy + dy;
                if (y < 0 || y >= d1) continue;
                const int c = (z * d1 + y) * d0;
                const int s0 = aux.cell_start[c + max(cx - 1, 0)], s1 = aux.cell_start[c + min(cx + 1, d0 - 1) + 1];
                for (int kb = s0; kb < s1; kb += 32) {
                    const int k = kb + l;
                    int q = -1;
                    bool ok = false;
                    if (k < s1) {
                        q = aux.cell_beads[k];
                        ok = q != i && within_cutoff(xi, J.x[q], J.pp_t);
                        for (int t = c0; t < c1 && ok; ++t) ok = J.cov_j[t] != q;
                        for (int t = n0; t < n1 && ok; ++t) ok = J.nat_j[t] != q;
                    }
                    const unsigned m = __ballot_sync(0xffffffffu, ok);
                    if (ok) {
                        const int pos = cnt + __popc(m & ((1u << l) - 1u));
                        if (pos < J.cap_pp) row[pos] = q;
                        else err = SOPB_STATUS_CAPACITY;
                    }
                    cnt += __popc(m);
                }
            }
        }
        if (l == 0) J.pp_cnt[i] = cnt < J.cap_pp ? cnt : J.cap_pp;
    }
    if (err) atomicMax(&Jp->status, err);
}

// Sorts 32 R keys of a warp, R to a lane, ascending in blocked order (lane l
// ends with the ranks R l to R l + R - 1): Batcher's bitonic network in the
// form whose every comparator points up, since each merge starts with the
// mirrored partner.  Partners up to R - 1 apart are in the same lane.
template <int R, int STRIDE>
__device__ __forceinline__ void sort_strides(int32_t (&v)[R], int l) {
    if constexpr (STRIDE >= R) {
        const bool low = (l & (STRIDE / R)) == 0;
#pragma unroll
        for (int a = 0; a < R; ++a) {
            const int32_t o = __shfl_xor_sync(0xffffffffu, v[a], STRIDE / R);
            v[a] = low ? min(v[a], o) : max(v[a], o);
        }
    } else if constexpr (STRIDE > 0) {
#pragma unroll
        for (int a = 0; a < R; ++a)
            if ((a & STRIDE) == 0) {
                const int32_t lo = min(v[a], v[a | STRIDE]);
                v[a | STRIDE] = max(v[a], v[a | STRIDE]);
                v[a] = lo;
            }
    }
    if constexpr (STRIDE > 1) sort_strides<R, STRIDE / 2>(v, l);
}

template <int R, int SIZE = 2>
__device__ __forceinline__ void sort_keys(int32_t (&v)[R], int l) {
    if constexpr (SIZE <= R) {
#pragma unroll
        for (int a = 0; a < R; ++a)
            if ((a ^ (SIZE - 1)) > a) {
                const int32_t lo = min(v[a], v[a ^ (SIZE - 1)]);
                v[a ^ (SIZE - 1)] = max(v[a], v[a ^ (SIZE - 1)]);
                v[a] = lo;
            }
    } else {
        // the lane mirrored within SIZE / R lanes, the register from the other end
        const bool low = (l & (SIZE / R >> 1)) == 0;
#pragma unroll
        for (int a = 0; a < R / 2; ++a) {
            const int32_t oa = __shfl_xor_sync(0xffffffffu, v[R - 1 - a], SIZE / R - 1);
            const int32_t ob = __shfl_xor_sync(0xffffffffu, v[a], SIZE / R - 1);
            v[a] = low ? min(v[a], oa) : max(v[a], oa);
            v[R - 1 - a] = low ? min(v[R - 1 - a], ob) : max(v[R - 1 - a], ob);
        }
    }
    if constexpr (SIZE > 2) sort_strides<R, SIZE / 4>(v, l);
    if constexpr (SIZE < 32 * R) sort_keys<R, SIZE * 2>(v, l);
}

template <int R>
__device__ __forceinline__ void sort_row(int32_t* row, int cnt, int32_t* sb, int l) {
    int32_t v[R];
#pragma unroll
    for (int a = 0; a < R; ++a) v[a] = 32 * a + l < cnt ? row[32 * a + l] : 0x7fffffff;
    sort_keys(v, l);
    // through shared memory (a word of padding in 32) back into rows of 32
#pragma unroll
    for (int a = 0; a < R; ++a) sb[R * l + a + ((R * l + a) >> 5)] = v[a];
    __syncwarp();
#pragma unroll
    for (int a = 0; a < R; ++a)
        if (32 * a + l < cnt) row[32 * a + l] = sb[33 * a + l];
    __syncwarp();
}

// Sorts every possible-pairs row ascending (the brute-force order); one warp
// per row: the keys in registers and the comparators as shuffles for rows up
// to kSortCap entries, odd-even transposition in place for longer rows.
// Bound by instruction issue: 1.33 ms for a 198000-bead shell (3 capsids of 60 x 1100
// beads), 9.2 ms with the keys and every comparator in shared memory.  128
// registers (16 warps per SM) cover the longest class without a spill.
__global__ void __launch_bounds__(128, 4)
k_cl_sort_rows(JobDev* __restrict__ Jp, int force) {
    extern __shared__ int32_t buf[];   // 4 warps x kSortCap / 32 * 33
    const JobDev& J = *Jp;
    const int64_t step = job_step(Jp);
    if (J.status || (!force && (step % J.stride != 0 || step % J.pp_freq != 0))) return;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    int32_t* sb = buf + w * (kSortCap / 32 * 33);
    for (int i = blockIdx.x * 4 + w; i < J.n; i += gridDim.x * 4) {
        const int cnt = J.pp_cnt[i];
        int32_t* row = J.pp_j + (size_t)i * J.cap_pp;
        if (cnt <= 128) sort_row<4>(row, cnt, sb, l);
        else if (cnt <= 256) sort_row<8>(row, cnt, sb, l);
        else if (cnt <= 512) sort_row<16>(row, cnt, sb, l);
        else if (cnt <= 1024) sort_row<32>(row, cnt, sb, l);
        else if (cnt <= kSortCap) sort_row<64>(row, cnt, sb, l);
        else {
            for (int pass = 0; pass < cnt; ++pass) {
                for (int k = 2 * l + (pass & 1); k + 1 < cnt; k += 64) {
                    const int32_t a = row[k], b = row[k + 1];
                    if (a > b) { row[k] = b; row[k + 1] = a; }
                }
                __syncwarp();
            }
        }
    }
}
static_assert(kSortCap == 2048, "k_cl_sort_rows handles rows up to 32 x 64 keys in registers");

// Near list of the Verlet rebuilds (a grid job with a skin): the possible
// pairs within pairlist_cutoff + skin, in the order of the possible rows,
// with the coordinates it was built at.  While no bead has moved more than
// half the skin since, every possible pair now closer than pairlist_cutoff
// was closer than pairlist_cutoff + skin then, so filtering the near rows with
// the same exact test gives the rows a filter of the possible rows gives.
// aux.near: [0] largest squared drift (float bits), [1] a near row overflowed
// its capacity, [2] the near list is usable, [3] it overflowed since the
// possible pairs are what they are: it would again, and rebuilds filter the
// possible rows without trying (jobs without hydrodynamics).  [0] and [1] are
// cleared by k_g_near_commit, the last kernel of every rebuild.
__device__ __forceinline__ bool verlet_from_near(const JobDev& J, const GridAux& a, int64_t step, int force) {
    return !force && a.nr_j && a.near[2] && step % J.pp_freq != 0 && __int_as_float(a.near[0]) < J.drift2;
}

// Whether a rebuild that is not from the near rows renews them.
__device__ __forceinline__ bool near_renewed(const JobDev& J, const GridAux& a, int64_t step, int force) {
    return a.nr_j && (force || !a.vh || !a.near[3] || step % J.pp_freq == 0);
}

// Largest squared displacement since the near list was built, at a Verlet
// step that may reuse it.
__global__ void __launch_bounds__(kGridBlock)
k_g_drift(JobDev* __restrict__ Jp, GridAux a) {
    const JobDev& J = *Jp;
    const int64_t step = job_step(Jp);
    if (J.status || step % J.stride != 0 || step % J.pairs_freq != 0 || step % J.pp_freq == 0 || !a.near[2]) return;
    float d2 = 0.f;
    for (int i = blockIdx.x * kGridBlock + threadIdx.x; i < J.n; i += gridDim.x * kGridBlock) {
        const float e = dist2_rn(a.x_ref[i], J.x[i]);
        d2 = fmaxf(d2, isfinite(e) ? e : INFINITY);   // fmaxf drops a NaN: count it as an infinite drift
    }
    for (int o = 16; o > 0; o >>= 1) d2 = fmaxf(d2, __shfl_xor_sync(0xffffffffu, d2, o));
    if ((threadIdx.x & 31) == 0 && d2 > 0.f) atomicMax(&a.near[0], __float_as_int(d2));   // non-negative floats order as ints
}

// Exclusive prefix sum over the warp's lanes, and the warp total.
__device__ __forceinline__ int warp_excl_scan(int v, int l, int& total) {
    int s = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, s, o);
        if (l >= o) s += t;
    }
    total = __shfl_sync(0xffffffffu, s, 31);
    return s - v;
}

// Appends the candidates of `hits` (bit u: q[u]) to a row in entry order:
// lane l holds entries 4l..4l+3 of the warp's 128, so its first hit goes
// after the hits of the lanes below.  Returns 1 when the row overflowed.
__device__ __forceinline__ int append_hits(int32_t* row, int cap, int& cnt, unsigned hits, const int (&q)[4], int l) {
    int total;
    int pos = cnt + warp_excl_scan(__popc(hits), l, total);
    int over = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if ((hits >> u) & 1u) {
            if (pos < cap) row[pos] = q[u];
            else over = 1;
            ++pos;
        }
    cnt += total;
    return over;
}

// Verlet rows (pairlist_kernel.cu:33-76) of a job with hydrodynamics, per
// bead, order kept: a warp per bead, each
// lane testing four consecutive candidates of the warp's 128 (four gathers in
// flight), an order-preserving warp scan placing the hits.  From the near
// rows when they are usable and no bead drifted too far; else from the
// possible rows, renewing the near rows at the current coordinates.
__global__ void __launch_bounds__(kGridBlock)
k_g_verlet(JobDev* __restrict__ Jp, GridAux a, int force) {
    __shared__ JobDev Js;
    load_job<kGridBlock>(Js, Jp);
    __syncthreads();
    const JobDev& J = Js;
    const int64_t step = J.step;
    if (J.status || (!force && (step % J.stride != 0 || step % J.pairs_freq != 0))) return;
    const bool near = verlet_from_near(J, a, step, force);
    const bool renew = !near && a.nr_j;
    const int srcw = near ? a.cap_nr : J.cap_pp;
    const bool vec = (srcw & 3) == 0;      // 16-byte aligned source rows
    const int l = threadIdx.x & 31;
    int err = 0, over = 0;
    for (int i = blockIdx.x * (kGridBlock / 32) + threadIdx.x / 32; i < J.n; i += gridDim.x * (kGridBlock / 32)) {
        const float4 xi = J.x[i];
        const int src = near ? a.nr_cnt[i] : J.pp_cnt[i];
        const int32_t* srow = near ? a.nr_j + (size_t)i * a.cap_nr : J.pp_j + (size_t)i * J.cap_pp;
        int32_t* row = J.pl_j + (size_t)i * J.cap_pl;
        int32_t* nrow = renew ? a.nr_j + (size_t)i * a.cap_nr : nullptr;
        int cnt = 0, ncnt = 0;
        for (int kb = 0; kb < src; kb += 128) {
            const int k = kb + 4 * l;
            int q[4] = {0, 0, 0, 0};
            if (vec && k + 3 < src) {
                const int4 v = __ldg(reinterpret_cast<const int4*>(srow + k));
                q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (k + u < src) q[u] = __ldg(srow + k + u);
            }
            float r2[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) r2[u] = k + u < src ? dist2_rn(xi, J.x[q[u]]) : 0.f;
            unsigned hits = 0u, nhits = 0u;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool cand = k + u < src;
                if (cand && r2[u] < J.pl_t) hits |= 1u << u;
                if (cand && r2[u] < J.nr_t) nhits |= 1u << u;
            }
            if (append_hits(row, J.cap_pl, cnt, hits, q, l)) err = SOPB_STATUS_CAPACITY;
            if (renew) over |= append_hits(nrow, a.cap_nr, ncnt, nhits, q, l);
        }
        if (l == 0) {
            J.pl_cnt[i] = cnt < J.cap_pl ? cnt : J.cap_pl;
            if (renew) {
                a.nr_cnt[i] = ncnt < a.cap_nr ? ncnt : a.cap_nr;
                a.x_ref[i] = xi;
            }
        }
    }
    if (err) atomicMax(&Jp->status, err);
    if (over) atomicOr(&a.near[1], 1);
}

// Verlet rows (pairlist_kernel.cu:33-76) of a job without hydrodynamics, per
// pair of beads (2p, 2p + 1): the partners of both, of the first alone, of the
// second alone, each in increasing j.  A warp per pair.
// A bead's partners are its possible partners (increasing j) within the cutoff.
// The warp filters both beads' possible rows into shared memory, a part at a
// time, and merges the two: what both lists hold is a partner of both.  The near
// rows are merged in the same way from what is within pairlist_cutoff + skin,
// as 8 q with bit 0 when q is near the first bead and bit 1 when it is near the
// second; a rebuild from them tests their entries alone.  Either way a row's
// sections come out in increasing j.
// As in the resident kernel, ballots give each hit its place in its section,
// then the hits are stored.  More than max_pairs partners of a bead sets err.
// A CTA takes a tile of pairs at a time and gives their rows consecutive places
// (any order: a header holds its row's start), four rounds' gathers in flight.
// Bound by latency: 169 us from the near rows of a 198000-bead shell, 566 when
// they are renewed (192 and 552 with a row per bead, which the step then gathers
// twice; 1600 when a near entry was searched for in the other bead's row).  200
// steps of 6000 beads without near rows 2.0 ms, 2.6 with a row per bead (3.3 with
// searches; 32 when the possible rows hold all beads).  Eight warps: a tile's 32
// pairs four deep (18000 beads without near rows 3.1 ms, 3.8 with four warps);
// three CTAs per SM: 80 registers without a spill (64 slow the near rebuilds).
constexpr int kPairWarps = 8;      // warps per CTA
constexpr int kPairBuf = 512;      // entries of a filtered possible row kept in shared memory
constexpr int kMaxPairBeads = 1 << 28;   // entries 16 j of 32 bits
static_assert(16ull * kMaxPairBeads <= 1ull << 32, "row entries");

// The possible partners of a bead within the root of t, increasing, from
// `o` to `n` of a warp's buffer; the row's entries from k on are still to come.
struct Filtered {
    const int32_t* row;
    int cnt, k, o, n;
    int32_t* buf;
    float4 x;
};
// At least 32 entries or all there are.
__device__ __forceinline__ void refill(Filtered& f, const float4* __restrict__ x, float t) {
    if (f.k >= f.cnt || f.n - f.o >= 32) return;
    const int l = threadIdx.x & 31, left = f.n - f.o;
    const unsigned below = (1u << l) - 1u;
    const int keep = l < left ? f.buf[f.o + l] : 0;
    __syncwarp();
    if (l < left) f.buf[l] = keep;
    int n = left, k = f.k, nq[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) nq[u] = f.row[min(k + 32 * u + l, f.cnt - 1)];
    for (; k < f.cnt && n + 128 <= kPairBuf; k += 128) {
        int q[4];
        float4 xq[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            q[u] = nq[u];
            xq[u] = x[q[u]];
        }
        // the next entries while these ones' coordinates are on the way
#pragma unroll
        for (int u = 0; u < 4; ++u) nq[u] = f.row[min(k + 128 + 32 * u + l, f.cnt - 1)];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool in = k + 32 * u + l < f.cnt && dist2_rn(f.x, xq[u]) < t;
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (in) f.buf[n + __popc(m & below)] = q[u];
            n += __popc(m);
        }
    }
    f.o = 0;
    f.n = n;
    f.k = k;
    __syncwarp();
}
// Entries of the warp's sorted window (a lane each) below v.
__device__ __forceinline__ int window_rank(int w, int v) {
    int r = 0;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
        if (__shfl_sync(0xffffffffu, w, r + s - 1) < v) r += s;
    return r + (__shfl_sync(0xffffffffu, w, r) < v ? 1 : 0);
}
// Merges two filtered rows, up to 32 entries of each at a time: visit(a, bits
// of a, b, bits of b, a's rank in the second window, the second window's
// entries that are in the first).  Bits 3 for an entry of both (once, as a), 1
// and 2 for one of the first or second alone, 0 for none.
template <typename Visit>
__device__ __forceinline__ void merge_rows(Filtered& A, Filtered& B, const float4* __restrict__ x, float t, Visit visit) {
    const int l = threadIdx.x & 31;
    const unsigned all = 0xffffffffu;
    constexpr int kEnd = 0x7fffffff;
    for (;;) {
        refill(A, x, t);
        refill(B, x, t);
        const int na = A.n - A.o, nb = B.n - B.o;
        if (na + nb == 0) break;
        const int a = l < na ? A.buf[A.o + l] : kEnd, b = l < nb ? B.buf[B.o + l] : kEnd;
        // as far as both windows are complete
        const int enda = na > 32 || A.k < A.cnt ? __shfl_sync(all, a, 31) : kEnd;
        const int endb = nb > 32 || B.k < B.cnt ? __shfl_sync(all, b, 31) : kEnd;
        const int end = min(enda, endb);
        const bool ta = l < na && a <= end, tb = l < nb && b <= end;
        const int r = window_rank(b, a);
        const bool both = __shfl_sync(all, b, r & 31) == a && ta && r < 32;
        const unsigned dup = __reduce_or_sync(all, both ? 1u << r : 0u);
        visit(a, ta ? (both ? 3 : 1) : 0, b, tb && !((dup >> l) & 1u) ? 2 : 0, r, dup);
        A.o += __popc(__ballot_sync(all, ta));
        B.o += __popc(__ballot_sync(all, tb));
    }
}

// Room for pair p's row and its header: sections of nf, n0 and n1 entries, cut
// off where a bead has more than max_pairs partners.
struct PairRow {
    int32_t* dst;
    int nf, n0, n1;
    __device__ __forceinline__ void store(int hit, int pos, uint32_t entry) const {
        pos += hit == 3 ? 0 : (hit == 1 ? nf : nf + n0);
        if (hit && pos < nf + n0 + n1) dst[pos] = (int32_t)entry;
    }
};
__device__ __forceinline__ PairRow place_row(const JobDev& J, const GridAux& a, int p, int nf, int n0, int n1, int* alloc, int& err) {
    const int l = threadIdx.x & 31, cap = a.cap_u & ~3;
    if (max(n0, n1) + nf > J.cap_pl) {
        err = SOPB_STATUS_CAPACITY;
        nf = min(nf, cap);
        n0 = min(n0, cap - nf);
        n1 = min(n1, cap - nf - n0);
    }
    int start = 0;
    if (a.tile > 1) {
        if (l == 0) start = atomicAdd(alloc, (nf + n0 + n1 + 3) & ~3);
        start = __shfl_sync(0xffffffffu, start, 0);
    }
    if (l == 0) a.vh[p] = make_int4(nf, n0, n1, start);
    return {a.vr + (size_t)(p / a.tile) * a.tile * a.cap_u + start, nf, n0, n1};
}

// Pair p's row from its near row.
__device__ __forceinline__ void row_from_near(const JobDev& J, const GridAux& a, int p, float4 x0, float4 x1, const int32_t* nrow,
                                              int count, int* alloc, int& err) {
    const int l = threadIdx.x & 31, rounds = (count + 31) >> 5;
    const unsigned below = (1u << l) - 1u, all = 0xffffffffu;
    int cf = 0, c0 = 0, c1 = 0;
    auto cand = [&](int u) { return 32 * u + l < count ? (uint32_t)nrow[32 * u + l] : 0u; };
    auto take = [&](float4 q, uint32_t e, int& at) {
        const int hit = ((dist2_rn(x0, q) < J.pl_t ? 1 : 0) | (dist2_rn(x1, q) < J.pl_t ? 2 : 0)) & (int)e;
        const unsigned mf = __ballot_sync(all, hit == 3), m0 = __ballot_sync(all, hit == 1), m1 = __ballot_sync(all, hit == 2);
        at = (hit == 3 ? cf : (hit == 1 ? c0 : c1)) + __popc((hit == 3 ? mf : (hit == 1 ? m0 : m1)) & below);
        cf += __popc(mf);
        c0 += __popc(m0);
        c1 += __popc(m1);
        return (e & ~7u) | (uint32_t)hit;
    };
    uint32_t w[kKeptRounds];
    int place[kKeptRounds];
#pragma unroll
    for (int u = 0; u < kKeptRounds; ++u) w[u] = u < rounds ? cand(u) : 0u;
#pragma unroll
    for (int u = 0; u < kKeptRounds; u += 4)
        if (u < rounds) {
            // four rounds' gathers in flight; an entry 0 hits nothing
            float4 q[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) q[v] = bead_at(reinterpret_cast<const char*>(J.x), 2 * (w[u + v] & ~7u));
#pragma unroll
            for (int v = 0; v < 4; ++v) w[u + v] = take(q[v], w[u + v], place[u + v]);
        }
    const int kf = cf, k0 = c0, k1 = c1;
    int at;
    for (int u = kKeptRounds; u < rounds; ++u) {
        const uint32_t e = cand(u), j = e >> 3;
        take(J.x[j], e, at);
    }
    const PairRow row = place_row(J, a, p, cf, c0, c1, alloc, err);
#pragma unroll
    for (int u = 0; u < kKeptRounds; ++u)
        if (u < rounds) row.store(w[u] & 3, place[u], 2 * (w[u] & ~7u));      // 16 j
    cf = kf;
    c0 = k0;
    c1 = k1;
    for (int u = kKeptRounds; u < rounds; ++u) {
        const uint32_t e = cand(u), j = e >> 3, v = take(J.x[j], e, at);
        row.store(v & 3, at, 2 * (v & ~7u));
    }
}

// Pair p's row from the possible rows of its beads.
__device__ __forceinline__ void row_from_possible(const JobDev& J, const GridAux& a, int p, const Filtered& A0, const Filtered& B0,
                                                  int* alloc, int& err) {
    const unsigned below = (1u << (threadIdx.x & 31)) - 1u, all = 0xffffffffu;
    int cf = 0, c0 = 0, c1 = 0;
    auto pass = [&](Filtered A, Filtered B, auto store) {
        cf = c0 = c1 = 0;
        merge_rows(A, B, J.x, J.pl_t, [&](int qa, int ba, int qb, int bb, int, unsigned) {
            const unsigned mf = __ballot_sync(all, ba == 3), m0 = __ballot_sync(all, ba == 1), m1 = __ballot_sync(all, bb);
            store(ba, (ba == 3 ? cf + __popc(mf & below) : c0 + __popc(m0 & below)), 16u * (uint32_t)qa);
            store(bb, c1 + __popc(m1 & below), 16u * (uint32_t)qb);
            cf += __popc(mf);
            c0 += __popc(m0);
            c1 += __popc(m1);
        });
    };
    Filtered A = A0, B = B0;
    refill(A, J.x, J.pl_t);
    refill(B, J.x, J.pl_t);
    const bool whole = A.k >= A.cnt && B.k >= B.cnt;    // both stay as they are for the second pass
    pass(A, B, [](int, int, uint32_t) {});
    const PairRow row = place_row(J, a, p, cf, c0, c1, alloc, err);
    pass(whole ? A : A0, whole ? B : B0, [&](int hit, int pos, uint32_t entry) { row.store(hit, pos, entry); });
}

// The near row of pair p; its length, also beyond its capacity.
__device__ __forceinline__ int build_near_row(const JobDev& J, int32_t* nrow, int cap, Filtered A, Filtered B) {
    const int l = threadIdx.x & 31;
    const unsigned below = (1u << l) - 1u, all = 0xffffffffu;
    int count = 0;
    merge_rows(A, B, J.x, J.nr_t, [&](int qa, int ba, int qb, int bb, int r, unsigned dup) {
        const unsigned ma = __ballot_sync(all, ba), mb = __ballot_sync(all, bb);
        // before a: the lanes below and the second row's own entries below its rank
        const unsigned lower = r < 32 ? (1u << r) - 1u : all;
        const int pa = count + l + __popc(mb & lower);
        if (ba && pa < cap) nrow[pa] = (int32_t)(8u * (uint32_t)qa + (uint32_t)ba);
        const int pb = count + __popc(mb & below) + window_rank(qa, qb);
        if (bb && pb < cap) nrow[pb] = (int32_t)(8u * (uint32_t)qb + 2u);
        count += __popc(ma) + __popc(mb);
    });
    return count;
}

__global__ void __launch_bounds__(32 * kPairWarps, 3)
k_g_pair_rows(JobDev* __restrict__ Jp, GridAux a, int force) {
    __shared__ JobDev Js;
    __shared__ int32_t buf[kPairWarps][2][kPairBuf];
    __shared__ int alloc;
    load_job<32 * kPairWarps>(Js, Jp);
    __syncthreads();
    const JobDev& J = Js;
    const int64_t step = J.step;
    if (J.status || (!force && (step % J.stride != 0 || step % J.pairs_freq != 0))) return;
    const bool near = verlet_from_near(J, a, step, force), renew = !near && near_renewed(J, a, step, force);
    const int l = threadIdx.x & 31, wp = threadIdx.x >> 5, np = (J.n + 1) >> 1;
    const int group = max(a.tile, kPairWarps), groups = (np + group - 1) / group;
    int err = 0, over = 0;
    for (int t = blockIdx.x; t < groups; t += gridDim.x) {
        if (threadIdx.x == 0) alloc = 0;
        __syncthreads();
        for (int p = t * group + wp; p < min(np, (t + 1) * group); p += kPairWarps) {
            const bool two = 2 * p + 1 < J.n;
            const float4 x0 = J.x[2 * p], x1 = J.x[two ? 2 * p + 1 : 2 * p];
            int32_t* nrow = a.nr_j ? a.nr_j + (size_t)p * a.cap_nr : nullptr;
            int count = near ? a.nr_cnt[p] : 0;
            bool from_near = near;
            Filtered A, B;
            if (!near) {
                const int32_t* r0 = J.pp_j + (size_t)(2 * p) * J.cap_pp;
                A = {r0, J.pp_cnt[2 * p], 0, 0, 0, buf[wp][0], x0};
                B = {r0 + J.cap_pp, two ? J.pp_cnt[2 * p + 1] : 0, 0, 0, 0, buf[wp][1], x1};
            }
            if (renew) {
                count = build_near_row(J, nrow, a.cap_nr, A, B);
                if (l == 0) {
                    a.nr_cnt[p] = min(count, a.cap_nr);
                    a.x_ref[2 * p] = x0;
                    if (two) a.x_ref[2 * p + 1] = x1;
                }
                if (count > a.cap_nr) over = 1;
                else from_near = true;
                __syncwarp();
            }
            if (from_near) row_from_near(J, a, p, x0, x1, nrow, count, &alloc, err);
            else row_from_possible(J, a, p, A, B, &alloc, err);
            __syncwarp();
        }
        __syncthreads();
        if (threadIdx.x == 0 && a.tile > 1) a.vtot[t] = alloc;
        __syncthreads();
    }
    if (err) atomicMax(&Jp->status, err);
    if (over) atomicOr(&a.near[1], 1);
}

// Closes a rebuild: the near list is usable after a rebuild that renewed it
// without overflow, unusable after new possible pairs without a Verlet
// rebuild, unchanged otherwise.  possible/verlet: an explicit rebuild (-1 in
// a run, where the step decides).
__global__ void k_g_near_commit(JobDev* __restrict__ Jp, GridAux a, int possible, int verlet) {
    if (threadIdx.x != 0 || blockIdx.x != 0 || !a.nr_j) return;
    const JobDev& J = *Jp;
    const int64_t step = job_step(Jp);
    const bool force = verlet >= 0;
    if (!force) {
        const bool at = step % J.stride == 0;
        possible = at && step % J.pp_freq == 0;
        verlet = at && step % J.pairs_freq == 0;
    }
    if (J.status) {
        a.near[2] = 0;
    } else if (verlet && !verlet_from_near(J, a, step, force ? 1 : 0)) {
        const bool renewed = near_renewed(J, a, step, force ? 1 : 0);
        a.near[2] = renewed && !a.near[1] ? 1 : 0;
        if (renewed) a.near[3] = a.near[1] ? 1 : 0;
    } else if (possible && !verlet) {
        a.near[2] = 0;
        a.near[3] = 0;
    }
    a.near[0] = 0;
    a.near[1] = 0;
}

// Advances the job's step counter by `by` (last launch of a chunk) and flags
// non-finite coordinates.
__global__ void k_g_advance(JobDev* __restrict__ Jp, int by) {
    if (threadIdx.x == 0 && blockIdx.x == 0) Jp->step += by;
}

__global__ void __launch_bounds__(kGridBlock)
k_g_check_finite(JobDev* __restrict__ Jp) {
    const JobDev& J = *Jp;
    for (int i = blockIdx.x * kGridBlock + threadIdx.x; i < J.n; i += gridDim.x * kGridBlock) {
        const float4 v = J.x[i];
        if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) atomicMax(&Jp->status, SOPB_STATUS_NONFINITE);
    }
}

}  // namespace sopb
