// sopb_hi.cuh — hydrodynamic interactions on the grid path.
//
// TEA (Geyer & Winter 2009, the reference's BDHI-TEA integrator,
// src/Integrators/bdhitea_kernel.cu:192-515): the O(N^2) sums over all bead
// pairs of a job, the step's (k_tea_step, which also moves the beads) and the
// updater's (k_tea_eps), are taken by a cluster of CTAs per 32 or 64 beads, in
// an order that does not depend on scheduling.  The per-job epsilon and beta'
// are reduced on the device in FP64, as the reference's host does
// (src/Integrators/bdhitea.cu:133-176).
//
// Exact HI for jobs up to 128 beads (3n <= 384, the reference's CHOLSIZE,
// src/Integrators/bdhitea.h:24): the normalised RPY tensor D is assembled,
// factorised and applied to the random forces by one cluster of CTAs
// (k_hi_small, B = L); or, for parity with the reference's noise matrix, by
// its own algorithm (L below, L^T above the diagonal, as
// integrateCholesky_decompose leaves it) and its symmetrised upper 3x3 blocks
// (integrateCholesky_L).
#pragma once

#include <type_traits>

#include "sopb_grid.cuh"

namespace sopb {

constexpr int kHiTile = 128;

struct Blk6 {
    float xx, xy, xz, yy, yz, zz;
};

// RPY block normalised by D_ii (bdhitea_kernel.cu:67-87): (ex,ey,ez) unit
// vector from i to j, r the distance, a the hydrodynamic radius.
__device__ __forceinline__ Blk6 rpy_block(float ex, float ey, float ez, float r, float a) {
    const float ra = r / a;
    float crr, cii;
    if (ra > 2.f) {
        crr = 0.75f / ra * (1.f - 2.f / ra / ra);
        cii = 0.75f / ra * (1.f + 2.f / 3.f / ra / ra);
    } else {
        crr = 3.f * ra / 32.f;
        cii = 1.f - 9.f * ra / 32.f;
    }
    return {ex * ex * crr + cii, ex * ey * crr, ex * ez * crr, ey * ey * crr + cii, ey * ez * crr, ez * ez * crr + cii};
}

__device__ __forceinline__ Blk6 rpy_between(float4 xi, float4 xj, float a) {
    float dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
    const float r = sqrtf(dx * dx + dy * dy + dz * dz);
    dx /= r;
    dy /= r;
    dz /= r;
    return rpy_block(dx, dy, dz, r, a);
}

// The same block for the per-step O(n^2) sums, with one reciprocal square
// root per pair: e = d rsqrt(r^2), u = a / r = a rsqrt(r^2), and the far
// field (r > 2a) tested as r^2 > 4a^2; both branches are formed and one is
// selected, so a warp does not diverge on the pair distance.
__device__ __forceinline__ Blk6 rpy_fast(float4 xi, float4 xj, float a, float inv_a) {
    const float dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
    const float r2 = dx * dx + dy * dy + dz * dz;
    const float ir = rsqrtf(r2);
    const float ex = dx * ir, ey = dy * ir, ez = dz * ir;
    const float u = a * ir, u2 = u * u, ra = r2 * ir * inv_a;
    const bool far = r2 > 4.f * a * a;
    const float crr = far ? 0.75f * u * (1.f - 2.f * u2) : (3.f / 32.f) * ra;
    const float cii = far ? 0.75f * u * (1.f + (2.f / 3.f) * u2) : 1.f - (9.f / 32.f) * ra;
    return {ex * ex * crr + cii, ex * ey * crr, ex * ez * crr, ey * ey * crr + cii, ey * ez * crr, ez * ez * crr + cii};
}

// integrateTea_epsilon_local (bdhitea_kernel.cu:192-210): squared row sums
// (x, y, z) and the sum of all nine entries (w).
__device__ __forceinline__ void eps_stats(float4 xi, float4 xj, float a, float4& s) {
    const Blk6 d = rpy_between(xi, xj, a);
    s.w += d.xx + 2 * d.xy + 2 * d.xz + d.yy + 2 * d.yz + d.zz;
    s.x += d.xx * d.xx + d.xy * d.xy + d.xz * d.xz;
    s.y += d.xy * d.xy + d.yy * d.yy + d.yz * d.yz;
    s.z += d.xz * d.xz + d.yz * d.yz + d.zz * d.zz;
}

// integrateTea_force (bdhitea_kernel.cu:252-301): D_ij F with F = F_j + beta
// C_i o g_j, as cii F + (crr / r^2) (d . F) d for the separation d: one
// reciprocal square root, no unit vector and no block.
struct TeaConst {
    float far2, u1, c1, c2, n0, n1;
    __device__ __forceinline__ explicit TeaConst(float a)
        : far2(4.f * a * a), u1(0.75f * a), c1((2.f / 3.f) * a * a), c2(-2.f * a * a), n0((3.f / 32.f) / a), n1((-9.f / 32.f) / a) {}
};
__device__ __forceinline__ void tea_pair(float4 xi, float4 xj, float4 mj, float4 rj, float3 bci, const TeaConst& c, float3& f) {
    const float dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float ir = rsqrtf(r2), ir2 = ir * ir;
    const bool far = r2 > c.far2;
    const float u = c.u1 * ir;
    const float cii = far ? u * fmaf(c.c1, ir2, 1.f) : fmaf(c.n1 * r2, ir, 1.f);
    const float crr = far ? u * ir2 * fmaf(c.c2, ir2, 1.f) : c.n0 * ir;
    const float f0 = fmaf(rj.x, bci.x, mj.x), f1 = fmaf(rj.y, bci.y, mj.y), f2 = fmaf(rj.z, bci.z, mj.z);
    const float s = crr * fmaf(dx, f0, fmaf(dy, f1, dz * f2));
    f.x = fmaf(cii, f0, fmaf(s, dx, f.x));
    f.y = fmaf(cii, f1, fmaf(s, dy, f.y));
    f.z = fmaf(cii, f2, fmaf(s, dz, f.z));
}

__device__ __forceinline__ bool tea_eps_due(const JobDev& J, int64_t step) {
    return step % J.stride == 0 && step % J.eps_freq == 0;
}

// ---- TEA epsilon (updater) --------------------------------------------------
// The split of k_tea_step with a bead per lane.
constexpr int kTeaCtas = 8, kTeaWarps = 8, kTeaChunk = 256;

// The updater's sums.  Bound by FP32 issue for large jobs (a square root and
// divisions per pair): 43 us at 4000 beads, 6.7 at 517 (latency); 47 + 10.5
// and 20 + 5.2 as tiles of 128 x 128 beads and a second kernel that added the
// slices.
__global__ void __launch_bounds__(32 * kTeaWarps)
k_tea_eps(JobDev* __restrict__ Jp, GridAux aux, int force) {
    __shared__ float4 xs[kTeaChunk], part[kTeaWarps][32], sums[kTeaCtas][32];
    const JobDev& J = *Jp;
    const int64_t step = job_step(Jp);
    if (J.status || (!force && !tea_eps_due(J, step))) return;
    cluster_arrive();                                      // this CTA has begun: its shared memory may be written
    const int tid = threadIdx.x, l = tid & 31, w = tid >> 5, rank = blockIdx.x % kTeaCtas, i0 = blockIdx.x / kTeaCtas * 32;
    const int n = J.n, i = i0 + l;
    const float4 xi = J.x[min(i, n - 1)];
    const float a = J.hi_a;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (J.hi_unlisted) {
        const int span = (n + kTeaCtas - 1) / kTeaCtas, j0 = rank * span, j1 = min(n, j0 + span);
        for (int t0 = j0; t0 < j1; t0 += kTeaChunk) {
            const int cnt = min(kTeaChunk, j1 - t0);
            __syncthreads();
            if (tid < cnt) xs[tid] = J.x[t0 + tid];
            __syncthreads();
            if (t0 < i0 + 32 && i0 < t0 + cnt) {       // some of the CTA's own beads
                for (int k = w; k < cnt; k += kTeaWarps)
                    if (t0 + k != i) eps_stats(xi, xs[k], a, acc);
            } else {
#pragma unroll 4
                for (int k = w; k < cnt; k += kTeaWarps) eps_stats(xi, xs[k], a, acc);
            }
        }
    } else if (i < n) {
        // integrateTea_epsilon: covalent, native and Verlet partners
        const int first = rank * kTeaWarps + w, by = kTeaCtas * kTeaWarps;
        for (int k = J.cov_off[i] + first; k < J.cov_off[i + 1]; k += by) eps_stats(xi, J.x[J.cov_j[k]], a, acc);
        for (int k = J.nat_off[i] + first; k < J.nat_off[i + 1]; k += by) eps_stats(xi, J.x[J.nat_j[k]], a, acc);
        const int32_t* row = J.pl_j + (size_t)i * J.cap_pl;
        for (int k = first; k < J.pl_cnt[i]; k += by) eps_stats(xi, J.x[row[k]], a, acc);
    }
    part[w][l] = acc;
    __syncthreads();
    cluster_wait();
    auto add4 = [](float4& t, float4 p) { t.x += p.x; t.y += p.y; t.z += p.z; t.w += p.w; };
    if (tid < 32) {
        float4 t = part[0][l];
        for (int q = 1; q < kTeaWarps; ++q) add4(t, part[q][l]);
        const uint32_t to = map_rank((uint32_t)__cvta_generic_to_shared(&sums[rank][l]), 0);
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to), "f"(t.x), "f"(t.y), "f"(t.z), "f"(t.w) : "memory");
    }
    cluster_sync_all();
    if (rank != 0 || tid >= 32 || i >= n) return;
    float4 t = sums[0][l];
    for (int q = 1; q < kTeaCtas; ++q) add4(t, sums[q][l]);
    aux.ci4[i] = t;
    aux.eps[i] = t.w;
}

// TeaUpdater::update's host arithmetic (bdhitea.cu:143-169) in FP64: the
// average off-diagonal coupling epsilon, the capricious checks, and
// beta' = (1 - sqrt(1 - a)) / a with a = (3N-1) eps^2 - (3N-2) eps.
__global__ void __launch_bounds__(256)
k_tea_beta(JobDev* __restrict__ Jp, GridAux aux, int force) {
    __shared__ double red[256];
    JobDev& J = *Jp;
    const int64_t step = job_step(Jp);
    if (J.status || (!force && !tea_eps_due(J, step))) return;
    const int n = J.n;
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += 256) s += (double)aux.eps[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        double eps = red[0];
        if (n > 1) eps /= 3. * n * (3. * n - 3.);
        int st = 0;
        if (eps > 1.0) {
            if (J.hi_capricious) st = SOPB_ERR_HI;
            eps = 1.0;
        }
        if (eps > J.hi_epsmax) st = SOPB_ERR_HI;
        const double a = (3. * n - 1.) * eps * eps - (3. * n - 2.) * eps;
        double beta;
        if (fabs(a) < 1e-7) {
            beta = 0.5;
            if (J.hi_capricious && J.hi_a > 0.0f) st = SOPB_ERR_HI;
        } else {
            beta = (1. - sqrt(1. - a)) / a;
        }
        J.beta = (float)beta;
        J.epsilon = (float)eps;
        if (st) J.status = st;
    }
}

// ---- TEA integration step ----------------------------------------------------
__device__ __forceinline__ float3 tea_bci(const JobDev& J, const GridAux& aux, int i, float3* ci_out) {
    const float4 c = aux.ci4[i];
    const float b2 = J.beta * J.beta;
    const float3 ci = make_float3(1.f / sqrtf(1.f + b2 * c.x), 1.f / sqrtf(1.f + b2 * c.y), 1.f / sqrtf(1.f + b2 * c.z));
    if (ci_out) *ci_out = ci;
    return make_float3(ci.x * J.beta, ci.y * J.beta, ci.z * J.beta);
}

// The sums and the move of a step.  A cluster of kTeaCtas CTAs takes 32 B
// beads, each CTA a share of the partners (staged in shared memory kTeaChunk at
// a time), each warp every eighth of those; a lane sums B beads, so the staged
// operands are read once for B.  The partial sums go to the first CTA through
// distributed shared memory and are added there in a fixed order (warps, then
// CTAs), and that CTA moves the beads.
// Bound by FP32 issue for large jobs: 31 us at 4000 beads (16 M pairs, 34
// instructions each); 43 + 11 as tiles of 128 x 128 beads with the partial sums
// in global memory and a second kernel that added them.  Below a thousand
// beads one bead per lane gives every SM a CTA: 7.3 us at 517 beads, most of it
// latency, where the tiles (25 CTAs) took 17 + 5.6.
constexpr int kTeaOneBead = 1024;   // up to this size a lane sums one bead, above it two

template <int B>
__global__ void __launch_bounds__(32 * kTeaWarps)
k_tea_step(JobDev* __restrict__ Jp, GridAux aux) {
    __shared__ float4 stage[3][kTeaChunk > 32 * B * kTeaWarps / 3 ? kTeaChunk : 32 * B * kTeaWarps / 3 + 1];
    __shared__ float4 sums[kTeaCtas][32 * B];
    const JobDev& J = *Jp;
    if (J.status) return;
    cluster_arrive();                                      // this CTA has begun: its shared memory may be written
    const int tid = threadIdx.x, l = tid & 31, w = tid >> 5, rank = blockIdx.x % kTeaCtas, i0 = blockIdx.x / kTeaCtas * (32 * B);
    const int n = J.n;
    float4 xi[B];
    float3 bci[B], f[B];
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const int i = min(i0 + 32 * b + l, n - 1);
        xi[b] = aux.xc[i];
        bci[b] = tea_bci(J, aux, i, nullptr);
        f[b] = make_float3(0.f, 0.f, 0.f);
    }
    const TeaConst c(J.hi_a);
    if (J.hi_unlisted) {
        const int span = (n + kTeaCtas - 1) / kTeaCtas, j0 = rank * span, j1 = min(n, j0 + span);
        for (int t0 = j0; t0 < j1; t0 += kTeaChunk) {
            const int cnt = min(kTeaChunk, j1 - t0);
            __syncthreads();
            for (int k = tid; k < cnt; k += 32 * kTeaWarps) {
                stage[0][k] = aux.xc[t0 + k];
                stage[1][k] = aux.mf[t0 + k];
                stage[2][k] = aux.rf[t0 + k];
            }
            __syncthreads();
            if (t0 < i0 + 32 * B && i0 < t0 + cnt) {   // some of the CTA's own beads
                for (int k = w; k < cnt; k += kTeaWarps) {
                    const float4 xj = stage[0][k], mj = stage[1][k], rj = stage[2][k];
#pragma unroll
                    for (int b = 0; b < B; ++b)
                        if (t0 + k != i0 + 32 * b + l) tea_pair(xi[b], xj, mj, rj, bci[b], c, f[b]);
                }
            } else {
#pragma unroll 4
                for (int k = w; k < cnt; k += kTeaWarps) {
                    const float4 xj = stage[0][k], mj = stage[1][k], rj = stage[2][k];
#pragma unroll
                    for (int b = 0; b < B; ++b) tea_pair(xi[b], xj, mj, rj, bci[b], c, f[b]);
                }
            }
        }
    } else {
        // integrateTea_kernel: covalent, native and Verlet partners, every
        // 64th of a list to a warp
        const int first = rank * kTeaWarps + w, by = kTeaCtas * kTeaWarps;
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int i = i0 + 32 * b + l;
            if (i >= n) continue;
            auto pair = [&](int q) { tea_pair(xi[b], aux.xc[q], aux.mf[q], aux.rf[q], bci[b], c, f[b]); };
            for (int k = J.cov_off[i] + first; k < J.cov_off[i + 1]; k += by) pair(J.cov_j[k]);
            for (int k = J.nat_off[i] + first; k < J.nat_off[i + 1]; k += by) pair(J.nat_j[k]);
            const int32_t* row = J.pl_j + (size_t)i * J.cap_pl;
            for (int k = first; k < J.pl_cnt[i]; k += by) pair(row[k]);
        }
    }
    // the warps' sums, then the CTAs'
    __syncthreads();
    float4* part = &stage[0][0];
#pragma unroll
    for (int b = 0; b < B; ++b) part[w * (32 * B) + 32 * b + l] = make_float4(f[b].x, f[b].y, f[b].z, 0.f);
    __syncthreads();
    cluster_wait();
    if (tid < 32 * B) {
        float4 t = part[tid];
        for (int q = 1; q < kTeaWarps; ++q) {
            const float4 p = part[q * (32 * B) + tid];
            t.x += p.x; t.y += p.y; t.z += p.z;
        }
        const uint32_t to = map_rank((uint32_t)__cvta_generic_to_shared(&sums[rank][tid]), 0);
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to), "f"(t.x), "f"(t.y), "f"(t.z), "f"(t.w) : "memory");
    }
    cluster_sync_all();
    const int i = i0 + tid;
    if (rank != 0 || tid >= 32 * B || i >= n) return;
    float3 ci;
    tea_bci(J, aux, i, &ci);
    const float4 m = aux.mf[i], r = aux.rf[i], xc = aux.xc[i];
    float3 F = make_float3(m.x + r.x * ci.x, m.y + r.y * ci.y, m.z + r.z * ci.z);
    for (int q = 0; q < kTeaCtas; ++q) {
        const float4 p = sums[q][tid];
        F.x += p.x; F.y += p.y; F.z += p.z;
    }
    if (J.pulling && J.flags[i] == FLAG_FIXED) F = make_float3(0.f, 0.f, 0.f);
    const float dx = J.hOverZeta * F.x, dy = J.hOverZeta * F.y, dz = J.hOverZeta * F.z;
    J.x[i] = make_float4(xc.x + dx, xc.y + dy, xc.z + dz, xc.w);
    J.T[i] += J.tempNorm * (dx * dx + dy * dy + dz * dz);
}

// ---- exact HI, n <= 128 ---------------------------------------------------------
// integrateCholesky_D (bdhitea_kernel.cu:89-152): bead i's block column of
// D (identity diagonal blocks; written when the factor is refreshed) and
// D F with every bead reading the prepared forces (the reference reads them
// while other threads overwrite them).
__global__ void __launch_bounds__(kGridBlock)
k_chol_D(JobDev* __restrict__ Jp, GridAux aux, int assemble) {
    const JobDev& J = *Jp;
    if (J.status) return;
    const int n = J.n, ld = aux.ld;
    for (int i = blockIdx.x * kGridBlock + threadIdx.x; i < n; i += gridDim.x * kGridBlock) {
        const float4 xi = J.x[i];
        float4 f = aux.mf[i];
        for (int q = 0; q < n; ++q) {
            float* r0 = aux.tensor + (size_t)(3 * q) * ld + 3 * i;
            float* r1 = r0 + ld;
            float* r2 = r1 + ld;
            if (q == i) {
                if (assemble) {
                    r0[0] = 1.f; r0[1] = 0.f; r0[2] = 0.f;
                    r1[0] = 0.f; r1[1] = 1.f; r1[2] = 0.f;
                    r2[0] = 0.f; r2[1] = 0.f; r2[2] = 1.f;
                }
                continue;
            }
            const Blk6 d = rpy_between(xi, J.x[q], J.hi_a);
            if (assemble) {
                r0[0] = d.xx; r0[1] = d.xy; r0[2] = d.xz;
                r1[0] = d.xy; r1[1] = d.yy; r1[2] = d.yz;
                r2[0] = d.xz; r2[1] = d.yz; r2[2] = d.zz;
            }
            const float4 fq = aux.mf[q];
            f.x += d.xx * fq.x + d.xy * fq.y + d.xz * fq.z;
            f.y += d.xy * fq.x + d.yy * fq.y + d.yz * fq.z;
            f.z += d.xz * fq.x + d.yz * fq.y + d.zz * fq.z;
        }
        aux.F[i] = f;   // D F (the potential forces are no longer needed)
    }
}

// integrateCholesky_decompose (bdhitea_kernel.cu:154-190): one CTA of 3n
// threads, one column per round.
__global__ void __launch_bounds__(384)
k_chol_factor_small(JobDev* __restrict__ Jp, GridAux aux) {
    __shared__ float row[384];
    __shared__ float diag;
    const JobDev& J = *Jp;
    if (J.status) return;
    const int m = 3 * J.n, ld = aux.ld, t = threadIdx.x;
    float* M = aux.tensor;
    for (int j = 0; j < m; ++j) {
        if (t < m) row[t] = M[(size_t)j * ld + t];
        __syncthreads();
        float val = t < m ? row[t] : 0.f;
        if (t < m && t >= j)
            for (int k = 0; k < j; ++k) val -= M[(size_t)k * ld + t] * row[k];
        if (t == j) diag = sqrtf(val);
        __syncthreads();
        if (t < m && t >= j) {
            val = val / diag;
            M[(size_t)t * ld + j] = val;
            M[(size_t)j * ld + t] = val;
        }
        __syncthreads();
    }
}

// integrateCholesky_L (bdhitea_kernel.cu:303-361) with the reference's noise
// matrix: f_i = (D F)_i + sum_{q<=i} B_iq (rho g)_q, B the symmetrised upper
// 3x3 blocks, then the fixed beads and the Ermak-McCammon move.
__global__ void __launch_bounds__(kGridBlock)
k_chol_apply(JobDev* __restrict__ Jp, GridAux aux) {
    const JobDev& J = *Jp;
    if (J.status) return;
    const int n = J.n, ld = aux.ld;
    const float* M = aux.tensor;
    for (int i = blockIdx.x * kGridBlock + threadIdx.x; i < n; i += gridDim.x * kGridBlock) {
        const float4 dfi = aux.F[i];
        float3 f = make_float3(dfi.x, dfi.y, dfi.z);
        for (int q = 0; q <= i; ++q) {
            const float4 g = aux.rf[q];
            const float* L0 = M + (size_t)(3 * q) * ld + 3 * i;
            const float bxx = L0[0], bxy = L0[1], bxz = L0[2], byy = L0[ld + 1], byz = L0[ld + 2], bzz = L0[2 * ld + 2];
            f.x += bxx * g.x + bxy * g.y + bxz * g.z;
            f.y += bxy * g.x + byy * g.y + byz * g.z;
            f.z += bxz * g.x + byz * g.y + bzz * g.z;
        }
        if (J.pulling && J.flags[i] == FLAG_FIXED) f = make_float3(0.f, 0.f, 0.f);
        const float4 xc = aux.xc[i];
        const float dx = J.hOverZeta * f.x, dy = J.hOverZeta * f.y, dz = J.hOverZeta * f.z;
        J.x[i] = make_float4(xc.x + dx, xc.y + dy, xc.z + dz, xc.w);
        J.T[i] = J.T[i] + J.tempNorm * (dx * dx + dy * dy + dz * dz);
    }
}

// ---- exact HI with the true factor (B = L), n <= 128: one kernel per step --------
// integrateTea_prepare, integrateCholesky_D, _decompose and _L
// (bdhitea_kernel.cu:33-65, 89-190, 303-361) in one cluster of up to eight
// CTAs that holds the 3n x 3n matrix in shared memory from its assembly to
// the product with the noise.
//   Rows are dealt to the CTAs in blocks of 32 (block b to CTA b mod C).
//   Right-looking in panels of 32 columns: four warps of the diagonal block's
//   owner factor the 32 x 32 tile (in registers, four lanes per row; its 8 x 8
//   blocks by every lane for itself, so nothing but arithmetic sits between
//   their pivots) and send the tile to every CTA; each CTA solves its rows
//   below (four lanes per row) and sends them; each updates its own trailing
//   tiles (a warp per 32 x 32 tile, a row per lane).  The next diagonal tile is
//   updated first, by eight of its owner's warps, and factored while the other
//   warps update the rest.
//   All in FP32; a pivot's reciprocal root is an estimate with one Newton step,
//   the root and the quotients by it are corrected by their residuals.
// Then D F (a warp per bead), L g (a warp per row), the fixed beads and the
// Ermak-McCammon move.  Between refreshes L is read from the tensor.
// Bound: the serial chain of 3n/32 panels (factor 9000 cycles, solve and send
// 5000, two cluster barriers).  90 beads, a new factor every step: 79 us a
// step with the forces, 231 us with a one-CTA factor that kept the matrix in
// L2 and took two barriers per column.
constexpr int kSmallPanel = 32;
constexpr int kSmallThreads = 512;
constexpr int kSmallMaxCtas = 8;
constexpr int kSmallLdp = kSmallPanel + 4;                 // floats: rows of a panel, 16-byte aligned, no bank conflicts
struct SmallLayout {                                       // in floats
    int ldr, rows, P, Dg, dinv, S, x, mf, df, sd, g, total;
};
__host__ __device__ inline int small_blocks(int n) { return (3 * n + kSmallPanel - 1) / kSmallPanel; }
__host__ __device__ inline int small_ctas(int n) {
    const int T = small_blocks(n);
    return T >= 8 ? 8 : (T >= 4 ? 4 : (T >= 2 ? 2 : 1));
}
__host__ __device__ inline SmallLayout small_layout(int n, int C) {
    const int T = small_blocks(n), mp = kSmallPanel * T;
    SmallLayout L;
    L.ldr = mp + 4;
    int o = 0;
    L.rows = o; o += (T + C - 1) / C * kSmallPanel * L.ldr;
    L.P = o;    o += mp * kSmallLdp;
    L.Dg = o;   o += kSmallPanel * kSmallLdp;
    L.dinv = o; o += kSmallPanel;
    L.S = o;    o += 64;
    L.x = o;    o += 4 * n;
    L.mf = o;   o += 4 * n;
    L.df = o;   o += 4 * n;
    L.sd = o;   o += 4 * n;
    L.g = o;    o += mp;
    L.total = o;
    return L;
}

// 1 / sqrt(p): the hardware estimate and one Newton-Raphson step; d = sqrt(p)
// by one residual correction (P. Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", 1990); each within an ulp.
__device__ __forceinline__ float rsqrt_newton(float p, float& d) {
    float y = rsqrtf(p);
    y = fmaf(0.5f * y, fmaf(-p * y, y, 1.0f), y);
    d = p * y;
    d = fmaf(fmaf(-d, d, p), 0.5f * y, d);
    return y;
}
// a / d from r ~ 1 / d, corrected by the quotient's residual (Markstein): within
// an ulp
__device__ __forceinline__ float quotient(float a, float d, float r) {
    const float q = a * r;
    return fmaf(fmaf(-q, d, a), r, q);
}

__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
// A row's eight entries of a lower-triangular solve against the 8 x 8 factor
// block d8: x L^T = a.
__device__ __forceinline__ void solve8(float (&a)[8], const float (&d8)[8][8], const float (&dinv)[8]) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        float v = a[c];
#pragma unroll
        for (int q = 0; q < c; ++q) v = fmaf(-a[q], d8[c][q], v);
        a[c] = quotient(v, d8[c][c], dinv[c]);
    }
}
// a[k] -= x . l_k, l_k the eight entries at L + k kSmallLdp
__device__ __forceinline__ void rank8(float (&a)[8], const float (&x)[8], const float* L) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float l[8];
        load8(L + k * kSmallLdp, l);
#pragma unroll
        for (int c = 0; c < 8; ++c) a[k] = fmaf(-x[c], l[c], a[k]);
    }
}
__device__ __forceinline__ void store8(float* p, const float (&v)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void send8(uint32_t addr, const float (&v)[8]) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr + 16), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

// A warp's eight rows, four lanes per row: lane 8 t + r holds entries 8 t ..
// 8 t + 7 of row r (so a step's chain is eight entries long, not 32).  Both
// functions walk the 8-column blocks s: the lanes t = s solve, hand the result
// to the row's other lanes, and those beyond s take it off their entries.

// Rows below the diagonal tile, solved against it (Dg, dinv).
__device__ __forceinline__ void small_solve(float (&a)[8], const float* Dg, const float* dinv) {
    const int lane = threadIdx.x & 31, t = lane >> 3, r = lane & 7;
    for (int s = 0; s < kSmallPanel / 8; ++s) {
        if (t == s) {
            float d8[8][8], r8[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) load8(Dg + (8 * s + i) * kSmallLdp + 8 * s, d8[i]);
            load8(dinv + 8 * s, r8);
            solve8(a, d8, r8);
        }
        __syncwarp();
        float x[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) x[c] = __shfl_sync(0xffffffffu, a[c], 8 * s + r);
        if (t > s) rank8(a, x, Dg + 8 * t * kSmallLdp + 8 * s);
    }
}

// Factors the diagonal tile at `tile` (row stride ldr) with the CTA's first
// four warps and sends it and its pivots' reciprocals to every CTA.  S: 8 x 8
// floats of scratch.
constexpr int kSmallDiagWarps = 4;
__device__ __noinline__ void small_diag(float* tile, int ldr, float* Dg, float* dinv, float* S, int C, int rank) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, t = lane >> 3, r = lane & 7, row = 8 * w + r;
    // the four warps' barrier: counted by threads (barrier, not bar, whose
    // warps have to arrive converged), after the lanes of the branches above
    auto sync = [] {
        __syncwarp();
        asm volatile("barrier.sync 1, 128;" ::: "memory");
    };
    float a[8];
    load8(tile + row * ldr + 8 * t, a);
    for (int s = 0; s < kSmallPanel / 8; ++s) {
        if (w == s && t == s) store8(S + 8 * r, a);
        sync();
        if (t == s && w >= s) {
            float d8[8][8], r8[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) load8(S + 8 * i, d8[i]);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                float d;
                r8[c] = rsqrt_newton(d8[c][c], d);
                d8[c][c] = d;
#pragma unroll
                for (int i = c + 1; i < 8; ++i) d8[i][c] = quotient(d8[i][c], d, r8[c]);
#pragma unroll
                for (int i = c + 1; i < 8; ++i)
#pragma unroll
                    for (int k = c + 1; k <= i; ++k) d8[i][k] = fmaf(-d8[i][c], d8[k][c], d8[i][k]);
            }
            solve8(a, d8, r8);               // rows of the block itself get their rows of the factor
            store8(Dg + row * kSmallLdp + 8 * s, a);
            if (w == s && r == 0) store8(dinv + 8 * s, r8);
        }
        sync();
        float x[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) x[c] = __shfl_sync(0xffffffffu, a[c], 8 * s + r);
        if (t > s && t <= w) rank8(a, x, Dg + 8 * t * kSmallLdp + 8 * s);
    }
    store8(tile + row * ldr + 8 * t, a);
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(Dg + row * kSmallLdp + 8 * t);
    const uint32_t inv = (uint32_t)__cvta_generic_to_shared(dinv + 8 * r);
    float v[8];
    load8(dinv + 8 * (r & 3), v);
    for (int k = 1; k < C; ++k) {
        const uint32_t to = (uint32_t)((rank + k) % C);
        if (t <= w) send8(map_rank(mine, to), a);
        if (w == 0 && lane < kSmallPanel / 8) send8(map_rank(inv, to), v);
    }
}

// Columns [32 cb + 4 j0, 32 cb + 4 j1) of the tile of 32 rows at `rows` (row 0 of it
// is row 32 gb): minus the panel's rank-32 product, a row per lane.
__device__ __forceinline__ void small_tile(float* rows, int ldr, const float* P, int gb, int cb, int j0, int j1) {
    const int lane = threadIdx.x & 31;
    float x[kSmallPanel];
#pragma unroll
    for (int q = 0; q < kSmallPanel; q += 8) {
        float v[8];
        load8(P + (kSmallPanel * gb + lane) * kSmallLdp + q, v);
#pragma unroll
        for (int t = 0; t < 8; ++t) x[q + t] = v[t];
    }
    for (int j = j0; j < j1; ++j) {
        const float* p = P + (kSmallPanel * cb + 4 * j) * kSmallLdp;
        float acc[4] = {};
#pragma unroll
        for (int q = 0; q < kSmallPanel; q += 4)
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float4 b = *reinterpret_cast<const float4*>(p + t * kSmallLdp + q);
                acc[t] = fmaf(x[q], b.x, acc[t]);
                acc[t] = fmaf(x[q + 1], b.y, acc[t]);
                acc[t] = fmaf(x[q + 2], b.z, acc[t]);
                acc[t] = fmaf(x[q + 3], b.w, acc[t]);
            }
        float4* dst = reinterpret_cast<float4*>(rows + lane * ldr + kSmallPanel * cb + 4 * j);
        float4 v = *dst;
        v.x -= acc[0];
        v.y -= acc[1];
        v.z -= acc[2];
        v.w -= acc[3];
        *dst = v;
    }
}

__global__ void __launch_bounds__(kSmallThreads, 1)
k_hi_small(JobDev* __restrict__ Jp, GridAux aux, int refresh) {
    extern __shared__ __align__(16) float sm[];
    const JobDev& J = *Jp;
    if (J.status) return;                                   // the same for the whole cluster
    cluster_arrive();                                       // this CTA has begun: its shared memory may be written
    const int C = (int)cluster_nctarank(), rank = (int)cluster_ctarank();
    const int n = J.n, m = 3 * n, T = small_blocks(n), ld = aux.ld;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kWarps = kSmallThreads / 32;
    const SmallLayout lay = small_layout(n, C);
    const int ldr = lay.ldr;
    float *rows = sm + lay.rows, *P = sm + lay.P, *Dg = sm + lay.Dg, *dinv = sm + lay.dinv, *S = sm + lay.S, *g = sm + lay.g;
    float4 *xs = reinterpret_cast<float4*>(sm + lay.x), *mf = reinterpret_cast<float4*>(sm + lay.mf),
           *df = reinterpret_cast<float4*>(sm + lay.df);
    uint4* sd = reinterpret_cast<uint4*>(sm + lay.sd);
    // integrateTea_prepare (bdhitea_kernel.cu:33-65), by every CTA
    for (int q = tid; q < n; q += kSmallThreads) {
        xs[q] = J.x[q];
        uint4 st = J.seeds[q];
        const float4 gg = gaussian4(st);
        sd[q] = st;
        g[3 * q] = gg.x * J.var;
        g[3 * q + 1] = gg.y * J.var;
        g[3 * q + 2] = gg.z * J.var;
        float4 f = aux.F[q];
        if (J.pulling) {
            const uint8_t fl = J.flags[q];
            if (fl == FLAG_FIXED) f.x = f.y = f.z = 0.f;
            if (fl == FLAG_PULLED) { f.x += J.pullF[0]; f.y += J.pullF[1]; f.z += J.pullF[2]; }
        }
        mf[q] = f;
    }
    __syncthreads();
    const float a = J.hi_a;
    float* M = aux.tensor;
    if (refresh) {
        // D's rows of this CTA, lower triangle; rows past 3n are the identity's
        for (int lb = 0, gb = rank; gb < T; ++lb, gb += C) {
            const int r0 = kSmallPanel * gb, i0 = r0 / 3, i1 = min(n - 1, (r0 + kSmallPanel - 1) / 3);
            float* R = rows + lb * kSmallPanel * ldr;
            for (int e = tid; e < (i1 - i0 + 1) * (i1 + 1); e += kSmallThreads) {
                const int i = i0 + e / (i1 + 1), q = e % (i1 + 1);
                if (q > i) continue;
                Blk6 d{1.f, 0.f, 0.f, 1.f, 0.f, 1.f};
                if (q < i) d = rpy_between(xs[i], xs[q], a);
                const float b[3][3] = {{d.xx, d.xy, d.xz}, {d.xy, d.yy, d.yz}, {d.xz, d.yz, d.zz}};
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    const int r = 3 * i + u - r0;
                    if (r >= 0 && r < kSmallPanel)
#pragma unroll
                        for (int v = 0; v < 3; ++v) R[r * ldr + 3 * q + v] = b[u][v];
                }
            }
            for (int e = tid; e < (r0 + kSmallPanel - max(m, r0)) * (r0 + kSmallPanel); e += kSmallThreads) {
                const int r = max(m, r0) + e / (r0 + kSmallPanel), c = e % (r0 + kSmallPanel);
                R[(r - r0) * ldr + c] = r == c ? 1.f : 0.f;
            }
        }
        __syncthreads();
    }
    // no CTA stores into another one that has not begun (the assembly hides the wait)
    cluster_wait();
    if (refresh) {
        if (rank == 0 && warp < kSmallDiagWarps) small_diag(rows, ldr, Dg, dinv, S, C, rank);
        for (int p = 0; p < T; ++p) {
            cluster_sync_all();                            // the factored tile is everywhere
            const int lb0 = (p + C - rank) / C;            // this CTA's first block below p
            const int nlb = (T - rank + C - 1) / C - lb0;  // and their number
            for (int t = warp; t < kSmallPanel / 8 * nlb; t += kWarps) {
                const int lb = lb0 + t / (kSmallPanel / 8), r = 8 * (t % (kSmallPanel / 8)) + (lane & 7), c = 8 * (lane >> 3);
                float* src = rows + (lb * kSmallPanel + r) * ldr + kSmallPanel * p + c;
                float x[8];
                load8(src, x);
                small_solve(x, Dg, dinv);
                store8(src, x);
                const uint32_t to =
                    (uint32_t)__cvta_generic_to_shared(P + (kSmallPanel * (lb * C + rank) + r) * kSmallLdp + c);
                for (int k = 0; k < C; ++k) send8(map_rank(to, (uint32_t)((rank + k) % C)), x);
            }
            cluster_sync_all();                            // the panel is everywhere
            if (p + 1 == T) break;
            const bool next = rank == (p + 1) % C;         // owner of the next diagonal tile
            float* R1 = rows + (p + 1) / C * kSmallPanel * ldr;
            if (next) {
                if (warp < 8) small_tile(R1, ldr, P, p + 1, p + 1, warp, warp + 1);
                __syncthreads();
                if (warp < kSmallDiagWarps) small_diag(R1 + kSmallPanel * (p + 1), ldr, Dg, dinv, S, C, rank);
            }
            // the other tiles: block gb's columns p + 1 .. gb
            if (!next || warp >= kSmallDiagWarps) {
                int t = next ? warp - kSmallDiagWarps : warp;
                for (int lb = lb0; lb < lb0 + nlb; ++lb) {
                    const int gb = lb * C + rank, first = gb == p + 1 ? gb + 1 : p + 1;
                    const int count = gb - first + 1;
                    for (; t < count; t += next ? kWarps - kSmallDiagWarps : kWarps)
                        small_tile(rows + lb * kSmallPanel * ldr, ldr, P, gb, first + t, 0, kSmallPanel / 4);
                    t -= count;
                }
            }
            __syncthreads();
        }
        for (int lb = 0, gb = rank; gb < T; ++lb, gb += C)
            for (int r = warp; r < kSmallPanel; r += kWarps) {
                const int gr = kSmallPanel * gb + r;
                if (gr < m)
                    for (int c = lane; c <= gr; c += 32) M[(size_t)gr * ld + c] = rows[(lb * kSmallPanel + r) * ldr + c];
            }
    }
    // (L g)_r, a warp per row, and (D F)_i, a warp per bead
    float* y = reinterpret_cast<float*>(aux.part);
    for (int lb = 0, gb = rank; gb < T; ++lb, gb += C)
        for (int r = warp; r < kSmallPanel; r += kWarps) {
            const int gr = kSmallPanel * gb + r;
            if (gr >= m) continue;
            const float* Lr = refresh ? rows + (lb * kSmallPanel + r) * ldr : M + (size_t)gr * ld;
            float s = 0.f;
            for (int c = lane; c <= gr; c += 32) s = fmaf(Lr[c], g[c], s);
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) y[gr] = s;
        }
    for (int i = rank + C * warp; i < n; i += C * kWarps) {
        const float4 xi = xs[i];
        float3 f = make_float3(0.f, 0.f, 0.f);
        for (int q = lane; q < n; q += 32)
            if (q != i) {
                const Blk6 d = rpy_fast(xi, xs[q], a, 1.f / a);
                const float4 fq = mf[q];
                f.x += d.xx * fq.x + d.xy * fq.y + d.xz * fq.z;
                f.y += d.xy * fq.x + d.yy * fq.y + d.yz * fq.z;
                f.z += d.xz * fq.x + d.yz * fq.y + d.zz * fq.z;
            }
        f = group_reduce(f, 32);
        if (lane == 0) df[i] = make_float4(mf[i].x + f.x, mf[i].y + f.y, mf[i].z + f.z, 0.f);
    }
    __syncthreads();
    cluster_sync_all();                                    // y is complete, every CTA has read the job's state
    for (int i = rank + C * tid; i < n; i += C * kSmallThreads) {
        float3 f = make_float3(df[i].x + __ldcg(y + 3 * i), df[i].y + __ldcg(y + 3 * i + 1), df[i].z + __ldcg(y + 3 * i + 2));
        if (J.pulling && J.flags[i] == FLAG_FIXED) f = make_float3(0.f, 0.f, 0.f);
        const float4 xc = xs[i];
        const float dx = J.hOverZeta * f.x, dy = J.hOverZeta * f.y, dz = J.hOverZeta * f.z;
        J.x[i] = make_float4(xc.x + dx, xc.y + dy, xc.z + dz, xc.w);
        J.T[i] = J.T[i] + J.tempNorm * (dx * dx + dy * dy + dz * dz);
        J.seeds[i] = sd[i];
    }
}

}  // namespace sopb
