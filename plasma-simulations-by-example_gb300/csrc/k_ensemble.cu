/*
 * k_ensemble.cu -- a batched ensemble of independent grounded boxes (the ch2
 * box of ch2/Main.cpp:14-75, one per ensemble member) stepped together on one
 * GPU.  Boxes differ in node counts, particle counts, species weights and
 * densities.  Compiled with -fmad=false: the float64 density, charge and E
 * arithmetic is the one of k_fp64.cu (World::computeChargeDensity,
 * ch2/World.cpp:46-54; PotentialSolver::computeEF, ch2/PotentialSolver.cpp:
 * 70-110), so a box of the ensemble reproduces the same box run as a World.
 *
 * Layout in HBM: node fields of all boxes concatenated (box b owns nodes
 * [node0_b, node0_b + nn_b)): phi, rho (f64), ef4 (float4), the SOR
 * correction and residual (f32), and one int64 fixed-point accumulator per
 * species; particles of all (box, species) segments concatenated in the
 * mixed form (cell key, f32 offsets, f32 velocity), each segment starting on
 * a 64-particle boundary.
 *
 * A step is two persistent launches, captured once in a CUDA graph:
 *  1. k_ens_push (k_mixed.cu): push + deposit over a flattened work list of
 *     particle chunks; the walls reflect, so counts never change and the
 *     work list is built once on the host;
 *  2. k_ens_solve: thread-block clusters (1 to 8 CTAs on as many SMs) claim
 *     boxes, largest first, from an atomic counter; per box: rho from the
 *     accumulators (which it clears), the red-black SOR of
 *     PotentialSolver::solve (ch2/PotentialSolver.cpp:11-67) as float32
 *     correction sweeps under a float64 residual, then E, every pass split
 *     over the cluster's CTAs between cluster barriers.
 *
 * The SOR: the residual R = rho/eps0 + L phi of the reference
 * (ch2/PotentialSolver.cpp:44-61, L2 = sqrt(sum R^2 / (ni nj nk))) is formed
 * in float64; while L2 >= tol, 25 red-black sweeps solve L e = -R for a
 * float32 correction e (e = 0 on the walls) and phi += e.  The float64
 * residual bounds the error of phi, the float32 sweeps do the work.  Its
 * sum is taken plane by plane in a fixed order, so results do not depend on
 * the launch shape the autotuner picks.
 */
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include <cooperative_groups.h>

#include "espic.h"
#include "espic_world.h"

namespace cg = cooperative_groups;

int espic_internal_fail(int code, const char *msg);

namespace espic {

#define ENS_EPS_0 8.85418782e-12
constexpr int ENS_VW = 1024;      /* virtual width of the deterministic reductions */
constexpr int ENS_SWEEPS = 25;    /* float32 sweeps between float64 residual checks */

/* sum of part[0..ENS_VW) in a fixed tree; every thread gets the total */
__device__ double ens_tree_sum(double *part) {
    __syncthreads();
    for (int w = ENS_VW / 2; w > 0; w >>= 1) {
        for (int v = threadIdx.x; v < w; v += blockDim.x) part[v] += part[v + w];
        __syncthreads();
    }
    double t = part[0];
    __syncthreads();
    return t;
}

__device__ __forceinline__ double ens_node_volume(const Geo &g, int i, int j, int k) {
    double V = g.dh[0] * g.dh[1] * g.dh[2];
    if (i == 0 || i == g.ni - 1) V *= 0.5;
    if (j == 0 || j == g.nj - 1) V *= 0.5;
    if (k == 0 || k == g.nk - 1) V *= 0.5;
    return V;
}

/* d / node_vol: node_vol = V0 2^-h (h boundary halvings), so the quotient is
 * the correctly rounded d / V0 scaled by 2^h, exactly */
__device__ __forceinline__ double ens_per_volume(const Geo &g, int i, int j, int k, double d, double V0,
                                                 double yV0) {
    double scale = 1.0;
    if (i == 0 || i == g.ni - 1) scale *= 2.0;
    if (j == 0 || j == g.nj - 1) scale *= 2.0;
    if (k == 0 || k == g.nk - 1) scale *= 2.0;
    return div_rcp(d, V0, yV0) * scale;
}

/* reciprocals of 2 dh per axis: the divisors of the E differences */
struct EfRcp {
    double d2[3], y2[3];
};

__device__ __forceinline__ EfRcp ef_rcp(const Geo &g) {
    EfRcp r;
    for (int d = 0; d < 3; d++) {
        r.d2[d] = 2 * g.dh[d];
        r.y2[d] = 1.0 / r.d2[d];
    }
    return r;
}

/* E at node u = (i, j, k) of a box, the differences of k_efield (the same
 * numerators; the division by 2 dh correctly rounded through div_rcp) */
__device__ __forceinline__ void ens_efield(const Geo &g, const EfRcp &rc, const double *phi, int64_t u, int i, int j,
                                           int k, double &e0, double &e1, double &e2) {
    const int64_t sy = g.ni, sz = (int64_t)g.ni * g.nj;
    double n0, n1, n2;
    if (i == 0)
        n0 = -(-3 * phi[u] + 4 * phi[u + 1] - phi[u + 2]);
    else if (i == g.ni - 1)
        n0 = -(phi[u - 2] - 4 * phi[u - 1] + 3 * phi[u]);
    else
        n0 = -(phi[u + 1] - phi[u - 1]);
    if (j == 0)
        n1 = -(-3 * phi[u] + 4 * phi[u + sy] - phi[u + 2 * sy]);
    else if (j == g.nj - 1)
        n1 = -(phi[u - 2 * sy] - 4 * phi[u - sy] + 3 * phi[u]);
    else
        n1 = -(phi[u + sy] - phi[u - sy]);
    if (k == 0)
        n2 = -(-3 * phi[u] + 4 * phi[u + sz] - phi[u + 2 * sz]);
    else if (k == g.nk - 1)
        n2 = -(phi[u - 2 * sz] - 4 * phi[u - sz] + 3 * phi[u]);
    else
        n2 = -(phi[u + sz] - phi[u - sz]);
    e0 = div_rcp(n0, rc.d2[0], rc.y2[0]);
    e1 = div_rcp(n1, rc.d2[1], rc.y2[1]);
    e2 = div_rcp(n2, rc.d2[2], rc.y2[2]);
}

/* cluster barrier between passes that exchange global memory across the
 * cluster's SMs: barrier.cluster.arrive (release) + wait (acquire) orders
 * every CTA's global writes before the other CTAs' later reads */
__device__ __forceinline__ void cluster_sync_global(cg::cluster_group &cl) { cl.sync(); }

/* Division of the planes of a box among a cluster's CTAs: CTA r of `parts`
 * owns interior planes first(r) .. first(r + 1) - 1 (0-based). */
struct EnsPlanes {
    int planes, parts;
    __host__ __device__ int first(int r) const { return planes * r / parts; }
    __host__ __device__ int owner(int p) const { return ((p + 1) * parts - 1) / planes; }
    __host__ __device__ int most() const { return (planes + parts - 1) / parts; }
};

__host__ __device__ inline EnsPlanes ens_planes(int nk, int C) {
    const int P = nk - 2;
    return {P, C < P ? C : P};
}

constexpr int64_t ENS_SLAB_MAX = 200 * 1024; /* beside 9 KB of static shared memory */
constexpr int ENS_PLANE_WARPS = 8; /* virtual warps of a plane's residual sum */

/* slots of a row of one colour: half the nodes, in whole float4 */
__host__ __device__ inline int ens_slots(int ni) { return ((ni + 1) / 2 + 3) & ~3; }

/* floats of a CTA's correction (with a halo plane on either side) and of its
 * right-hand side: two colours, planes of nj rows of slots */
__host__ __device__ inline int64_t ens_slab_e(int ni, int nj, int nk, int C) {
    return 2ll * (ens_planes(nk, C).most() + 2) * nj * ens_slots(ni);
}
__host__ __device__ inline int64_t ens_slab_r(int ni, int nj, int nk, int C) {
    return 2ll * ens_planes(nk, C).most() * nj * ens_slots(ni);
}

/* whether a box is swept in a launch's shared memory: its correction fits, its
 * planes' sums fit their arrays, a colour fits a work array, and div_small's
 * range holds whatever the axes */
__host__ __device__ inline bool ens_has_slab(int ni, int nj, int nk, int C, int64_t slab_bytes) {
    const int64_t nn = (int64_t)ni * nj * nk;
    return nn < (1 << 24) && 4 * ens_slab_e(ni, nj, nk, C) <= slab_bytes &&
           ens_planes(nk, C).most() <= ENS_VW / ENS_PLANE_WARPS && (int64_t)(nk - 2) * nj * ens_slots(ni) <= nn;
}

/* Pieces of the residual's sum, whose bits depend on neither the cluster nor
 * the block size: a plane's nodes in ENS_PLANE_WARPS virtual warps (ens_warp_sum
 * of each), their sums in order (ens_plane_sum), and the planes' sums over the
 * lanes of a warp (ens_planes_total; get(p) is plane p's, all lanes get the
 * total). */
__device__ __forceinline__ double ens_warp_sum(double x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}
__device__ __forceinline__ double ens_plane_sum(const double *part) {
    double s = 0;
    for (int w = 0; w < ENS_PLANE_WARPS; w++) s += part[w];
    return s;
}
template <class F>
__device__ __forceinline__ double ens_planes_total(int planes, F get) {
    double s = 0;
    for (int p = (int)(threadIdx.x & 31); p < planes; p += 32) s += get(p);
    return ens_warp_sum(s);
}

struct EnsSolved {
    int sweeps, converged;
    double residual;
};

/* The sweeps of one box with the correction in shared memory.  Each CTA owns
 * a run of planes; its float32 correction e, and its right-hand side R where
 * that fits too (else R lies in global memory in the same order, a colour
 * in each of the box's two work arrays), lie split by colour, rows of
 * consecutive slots (node i of a row in slot i / 2), so that a thread takes
 * four nodes with 16-byte loads and no bank conflicts.  A new value on an outer plane is also
 * written into the neighbouring CTA's halo plane (distributed shared
 * memory), and a half sweep costs one cluster barrier and no memory latency:
 * with e and R in global memory a half sweep read six neighbours through L2
 * and found its nodes by integer divisions.  Boxes of 16 to 64 nodes an
 * axis, 8 CTAs: a half sweep 1.9 us on average, a step's solve of 64 boxes
 * 5.2 ms before, 2.9 ms now; what is left is a third float64 residuals (14
 * instructions a node).  The residual's sum is taken as in k_ens_solve, the
 * planes' sums from the CTAs' shared memory. */
__device__ __forceinline__ EnsSolved ens_sor_slab(const EnsBox &B, double *ph, const double *__restrict__ rh,
                                                  float *R0, float *R1, int max_it, double tol, bool r_shared,
                                                  float *slab, double *part, double *plane_sum, double *total,
                                                  int *err) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), C = (int)cl.num_blocks();
    const Geo &g = B.g;
    const int ni = g.ni, nj = g.nj, nk = g.nk, sy = ni, sz = ni * nj;
    const EnsPlanes pl = ens_planes(nk, C);
    const bool on = rank < pl.parts;
    const int ka = on ? 1 + pl.first(rank) : 1, np = on ? pl.first(rank + 1) - pl.first(rank) : 0;
    const int hs = ens_slots(ni), plane = nj * hs, most = pl.most();
    const int ecol = (most + 2) * plane;
    float *E = slab; /* [2][most + 2][plane] */
    /* the own planes' right-hand side of each colour */
    float *R[2];
    R[0] = r_shared ? slab + 2 * ecol : R0 + (ka - 1) * plane;
    R[1] = r_shared ? slab + 2 * ecol + most * plane : R1 + (ka - 1) * plane;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const double idx2 = 1.0 / (g.dh[0] * g.dh[0]);
    const double idy2 = 1.0 / (g.dh[1] * g.dh[1]);
    const double idz2 = 1.0 / (g.dh[2] * g.dh[2]);
    const double D = 2 * idx2 + 2 * idy2 + 2 * idz2;
    const float fcx = (float)idx2, fcy = (float)idy2, fcz = (float)idz2, fiD = (float)(1.0 / D);
    const double yeps = 1.0 / ENS_EPS_0;
    const float fw = (float)B.omega;
    const uint32_t rows = (uint32_t)(nj - 2), inner = (uint32_t)(ni - 2);
    const uint32_t quads = (uint32_t)hs / 4;
    const float inv_quads = 1.f / (float)quads, inv_rows = 1.f / (float)rows, inv_inner = 1.f / (float)inner;
    float *below = rank > 0 && on ? cl.map_shared_rank(E, rank - 1) : nullptr;
    float *above = on && rank + 1 < pl.parts ? cl.map_shared_rank(E, rank + 1) : nullptr;
    const int below_top = rank > 0 && on ? (pl.first(rank) - pl.first(rank - 1) + 1) * plane : 0;
    for (int t = tid; t < 2 * ecol; t += nt) E[t] = 0.f;
    __syncthreads();
    int sweeps = 0, conv = 0;
    double L2 = 0;
    /* with R in shared memory the work arrays hold the halves of rho / eps0,
     * written in the first residual pass */
    int *b_hi = (int *)R0, *b_lo = (int *)R1;
    for (;;) {
        /* float64 residual of the own planes, e = 0 on them */
        for (int task = warp; task < np * ENS_PLANE_WARPS; task += nw) {
            const int kk = task / ENS_PLANE_WARPS, vw = task % ENS_PLANE_WARPS, k = ka + kk;
            double acc2 = 0;
            for (uint32_t t = (uint32_t)(vw * 32 + lane); t < inner * rows; t += 32 * ENS_PLANE_WARPS) {
                const uint32_t r = div_small(t, inner, inv_inner);
                const int i = 1 + (int)(t - r * inner), j = 1 + (int)r;
                const int u = (k * nj + j) * ni + i;
                double b;
                if (r_shared && sweeps) {
                    b = __hiloint2double(b_hi[u], b_lo[u]);
                } else {
                    b = div_rcp(rh[u], ENS_EPS_0, yeps);
                    if (r_shared) {
                        b_hi[u] = __double2hiint(b);
                        b_lo[u] = __double2loint(b);
                    }
                }
                const double Ru = -ph[u] * D + b + idx2 * (ph[u - 1] + ph[u + 1]) + idy2 * (ph[u - sy] + ph[u + sy]) +
                                  idz2 * (ph[u - sz] + ph[u + sz]);
                const int c = (i + j + k) & 1, o = j * hs + (i >> 1);
                R[c][kk * plane + o] = (float)Ru;
                E[c * ecol + (kk + 1) * plane + o] = 0.f;
                acc2 += Ru * Ru;
            }
            acc2 = ens_warp_sum(acc2);
            if (lane == 0) part[task] = acc2;
        }
        if (sweeps) /* the halo planes: what the neighbours wrote */
            for (int t = tid; t < plane; t += nt)
                for (int c = 0; c < 2; c++) E[c * ecol + t] = E[c * ecol + (np + 1) * plane + t] = 0.f;
        __syncthreads();
        for (int kk = tid; kk < np; kk += nt) plane_sum[kk] = ens_plane_sum(part + kk * ENS_PLANE_WARPS);
        cluster_sync_global(cl);
        if (warp == 0) {
            const double s = ens_planes_total(pl.planes, [&](int p) {
                const int o = pl.owner(p);
                return *cl.map_shared_rank(plane_sum + (p - pl.first(o)), o);
            });
            if (lane == 0) *total = s;
        }
        __syncthreads();
        L2 = sqrt(*total / ((double)ni * nj * nk));
        if (!isfinite(L2)) {
            if (rank == 0 && tid == 0) atomicOr(err, DERR_NONFINITE);
            break;
        }
        if (L2 < tol) {
            conv = 1;
            break;
        }
        if (sweeps >= max_it) break;
        /* ENS_SWEEPS float32 sweeps of L e = -R */
        const int ns = max_it - sweeps < ENS_SWEEPS ? max_it - sweeps : ENS_SWEEPS;
        const uint32_t entries = (uint32_t)np * rows * quads;
        for (int s = 0; s < ns; s++) {
#pragma unroll
            for (int c = 0; c < 2; c++) {
                float *Ec = E + c * ecol;
                const float *Eo = E + (1 - c) * ecol;
                for (uint32_t t = tid; t < entries; t += nt) {
                    const uint32_t r = div_small(t, quads, inv_quads);
                    const uint32_t kk = div_small(r, rows, inv_rows);
                    const int slot = 4 * (int)(t - r * quads), j = 1 + (int)(r - kk * rows), k = ka + (int)kk;
                    const int par = (c + j + k) & 1; /* node of slot q: i = 2 q + par */
                    const int oc = (int)kk * plane + j * hs + slot, o = oc + plane;
                    const float4 rv = *(const float4 *)(R[c] + oc), ev = *(const float4 *)(Ec + o),
                                 xv = *(const float4 *)(Eo + o), ym = *(const float4 *)(Eo + o - hs),
                                 yp = *(const float4 *)(Eo + o + hs), zm = *(const float4 *)(Eo + o - plane),
                                 zp = *(const float4 *)(Eo + o + plane);
                    /* nodes i - 1 and i + 1 lie in slots q - 1 + par and q +
                     * par: the quad's own four and one beside it */
                    const float side = Eo[par ? o + 4 : o - 1];
                    const float xs[5] = {par ? xv.x : side, par ? xv.y : xv.x, par ? xv.z : xv.y,
                                         par ? xv.w : xv.z, par ? side : xv.w};
                    const float rr[4] = {rv.x, rv.y, rv.z, rv.w}, eo[4] = {ev.x, ev.y, ev.z, ev.w};
                    const float y0[4] = {ym.x, ym.y, ym.z, ym.w}, y1[4] = {yp.x, yp.y, yp.z, yp.w};
                    const float z0[4] = {zm.x, zm.y, zm.z, zm.w}, z1[4] = {zp.x, zp.y, zp.z, zp.w};
                    float v[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float sum = rr[q] + fcx * (xs[q] + xs[q + 1]) + fcy * (y0[q] + y1[q]) +
                                          fcz * (z0[q] + z1[q]);
                        const float en = sum * fiD;
                        const int i = 2 * (slot + q) + par;
                        v[q] = i >= 1 && i <= ni - 2 ? eo[q] + fw * (en - eo[q]) : 0.f; /* 0 on the walls */
                    }
                    const float4 nv = make_float4(v[0], v[1], v[2], v[3]);
                    *(float4 *)(Ec + o) = nv;
                    if (kk == 0 && below) *(float4 *)(below + c * ecol + below_top + (oc - (int)kk * plane)) = nv;
                    if ((int)kk == np - 1 && above) *(float4 *)(above + c * ecol + (oc - (int)kk * plane)) = nv;
                }
                cluster_sync_global(cl);
            }
        }
        sweeps += ns;
        for (uint32_t t = tid; t < (uint32_t)np * rows * inner; t += nt) {
            const uint32_t r = div_small(t, inner, inv_inner);
            const uint32_t kk = div_small(r, rows, inv_rows);
            const int i = 1 + (int)(t - r * inner), j = 1 + (int)(r - kk * rows), k = ka + (int)kk;
            ph[(k * nj + j) * ni + i] +=
                (double)E[((i + j + k) & 1) * ecol + ((int)kk + 1) * plane + j * hs + (i >> 1)];
        }
        cluster_sync_global(cl);
    }
    cluster_sync_global(cl); /* plane_sum and the halo planes are free again */
    return {sweeps, conv, L2};
}

/* The sweeps of one box whose slab does not fit the launch's shared memory:
 * e and R in global memory, every half sweep's nodes an even share of each
 * CTA.  psum: the planes' sums, one double a plane of the box. */
__device__ __forceinline__ EnsSolved ens_sor_global(const EnsBox &B, double *ph, const double *__restrict__ rh,
                                                    float *R, float *e, int max_it, double tol, double *psum,
                                                    double *part, double *total, int *err) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), C = (int)cl.num_blocks();
    const Geo &g = B.g;
    const int ni = g.ni, nj = g.nj, nk = g.nk, sy = ni, sz = ni * nj;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const double idx2 = 1.0 / (g.dh[0] * g.dh[0]);
    const double idy2 = 1.0 / (g.dh[1] * g.dh[1]);
    const double idz2 = 1.0 / (g.dh[2] * g.dh[2]);
    const double D = 2 * idx2 + 2 * idy2 + 2 * idz2;
    const float fcx = (float)idx2, fcy = (float)idy2, fcz = (float)idz2, fiD = (float)(1.0 / D);
    const double yeps = 1.0 / ENS_EPS_0;
    const float fw = (float)B.omega;
    const int hx = (ni - 2 + 1) / 2;
    const int count = hx * (nj - 2) * (nk - 2);
    const int interior = (ni - 2) * (nj - 2) * (nk - 2);
    const int c0 = (int)((int64_t)count * rank / C), c1 = (int)((int64_t)count * (rank + 1) / C);
    const int i0 = (int)((int64_t)interior * rank / C), i1 = (int)((int64_t)interior * (rank + 1) / C);
    constexpr int PLANES = ENS_VW / ENS_PLANE_WARPS; /* planes that part holds */
    const EnsPlanes pl = ens_planes(nk, C);
    const int pa = rank < pl.parts ? pl.first(rank) : 0, pb = rank < pl.parts ? pl.first(rank + 1) : 0;
    const uint32_t in_row = (uint32_t)(ni - 2), in_plane = in_row * (uint32_t)(nj - 2);
    int sweeps = 0, conv = 0;
    double L2 = 0;
    for (;;) {
        for (int p0 = pa; p0 < pb; p0 += PLANES) {
            const int np = pb - p0 < PLANES ? pb - p0 : PLANES;
            for (int task = warp; task < np * ENS_PLANE_WARPS; task += nw) {
                const int k = 1 + p0 + task / ENS_PLANE_WARPS, vw = task % ENS_PLANE_WARPS;
                double acc2 = 0;
                /* two nodes at once, all loads before any store */
                for (uint32_t t0 = (uint32_t)(vw * 32 + lane); t0 < in_plane; t0 += 64 * ENS_PLANE_WARPS) {
                    int uq[2];
                    double Rq[2];
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const uint32_t t = t0 + q * 32 * ENS_PLANE_WARPS, r = t / in_row;
                        uq[q] = t < in_plane ? (k * nj + 1 + (int)r) * ni + 1 + (int)(t - r * in_row) : -1;
                        const int u = uq[q] < 0 ? (k * nj + 1) * ni + 1 : uq[q];
                        Rq[q] = -ph[u] * D + div_rcp(rh[u], ENS_EPS_0, yeps) + idx2 * (ph[u - 1] + ph[u + 1]) +
                                idy2 * (ph[u - sy] + ph[u + sy]) + idz2 * (ph[u - sz] + ph[u + sz]);
                    }
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        if (uq[q] < 0) continue;
                        R[uq[q]] = (float)Rq[q];
                        e[uq[q]] = 0.f;
                        acc2 += Rq[q] * Rq[q];
                    }
                }
                acc2 = ens_warp_sum(acc2);
                if (lane == 0) part[task] = acc2;
            }
            __syncthreads();
            for (int kk = tid; kk < np; kk += nt) psum[p0 + kk] = ens_plane_sum(part + kk * ENS_PLANE_WARPS);
            __syncthreads();
        }
        cluster_sync_global(cl);
        if (warp == 0) {
            const double t = ens_planes_total(pl.planes, [&](int p) { return __ldcg(psum + p); });
            if (lane == 0) *total = t;
        }
        __syncthreads();
        L2 = sqrt(*total / ((double)ni * nj * nk));
        if (!isfinite(L2)) {
            if (rank == 0 && tid == 0) atomicOr(err, DERR_NONFINITE);
            break;
        }
        if (L2 < tol) {
            conv = 1;
            break;
        }
        if (sweeps >= max_it) break;
        /* ENS_SWEEPS float32 sweeps of L e = -R, then phi += e and the
         * float64 residual decides again */
        const int ns = max_it - sweeps < ENS_SWEEPS ? max_it - sweeps : ENS_SWEEPS;
        for (int s = 0; s < ns; s++) {
            for (int c = 0; c < 2; c++) {
                /* four independent nodes of colour c per thread: all
                 * loads before any store */
                for (int tb = c0 + tid; tb < c1; tb += 4 * nt) {
                    int uq[4];
                    float eo[4], sum[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int t = tb + q * nt;
                        uq[q] = -1;
                        eo[q] = 0.f;
                        sum[q] = 0.f;
                        if (t >= c1) continue;
                        const int i2 = t % hx;
                        const int r = t / hx;
                        const int j = 1 + r % (nj - 2);
                        const int k = 1 + r / (nj - 2);
                        const int i = 1 + 2 * i2 + ((1 + j + k + c) & 1);
                        if (i > ni - 2) continue;
                        const int u = (k * nj + j) * ni + i;
                        uq[q] = u;
                        eo[q] = e[u];
                        sum[q] = R[u] + fcx * (e[u - 1] + e[u + 1]) + fcy * (e[u - sy] + e[u + sy]) +
                                 fcz * (e[u - sz] + e[u + sz]);
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (uq[q] < 0) continue;
                        const float en = sum[q] * fiD;
                        e[uq[q]] = eo[q] + fw * (en - eo[q]);
                    }
                }
                cluster_sync_global(cl);
            }
        }
        sweeps += ns;
        for (int t = i0 + tid; t < i1; t += nt) {
            const int i = 1 + t % (ni - 2);
            const int r = t / (ni - 2);
            const int j = 1 + r % (nj - 2);
            const int k = 1 + r / (nj - 2);
            const int u = (k * nj + j) * ni + i;
            ph[u] += (double)e[u];
        }
        cluster_sync_global(cl);
    }
    cluster_sync_global(cl); /* psum is free again */
    return {sweeps, conv, L2};
}

__device__ __noinline__ EnsSolved ens_sor_global_call(const EnsBox &B, double *ph, const double *rh, float *R, float *e,
                                                      int max_it, double tol, double *psum, double *part,
                                                      double *total, int *err) {
    return ens_sor_global(B, ph, rh, R, e, max_it, tol, psum, part, total, err);
}

/* One box per thread-block cluster of C CTAs (C = 1, 2, 4 or 8, chosen at
 * launch): the CTAs split every node pass and every half sweep into
 * contiguous slices and meet at cluster barriers.  Boxes whose slabs fit the
 * launch's shared memory are swept there (ens_sor_slab), the others here.  The
 * box a cluster works on is claimed by CTA 0 and read by the others from its
 * shared memory.  The residual is summed plane by plane on both routes (see
 * ens_planes_total), here with the planes' sums in global memory, so the
 * solve's outcome depends on neither C nor the block size, nor on whether
 * these let the box's slab fit.  ROUTES: those of the launch's
 * boxes.  The shared-memory sweeps are inlined (64 boxes of 16 to 64 nodes
 * with 8 CTAs, five steps: 22.1 ms, as a call 22.8), the others a call where
 * they are alone (24 boxes of 80 to 120 nodes an axis with single CTAs of
 * 1024 threads, three steps: 887 ms, inlined 987) and inlined beside them
 * (512 boxes, 4 CTAs: 27.2 ms a step, as calls 27.5). */
enum { ENS_SLAB = 1, ENS_GLOBAL = 2 };

template <int ROUTES>
__global__ void __launch_bounds__(1024) k_ens_solve(const EnsBox *__restrict__ boxes, const EnsSeg *__restrict__ segs,
                                                    int nsp, const int *__restrict__ order, int nbox, int *counter,
                                                    double *phi, double *rho, float *ecor, float *res, float4 *ef4,
                                                    unsigned long long *acc, int64_t total_nodes, int max_it,
                                                    double tol, int solve, EnsStat *stat, int slab_bytes, int *err) {
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) float ens_slab[];
    const int C = (int)cl.num_blocks();
    const int rank = (int)cl.block_rank();
    __shared__ double part[ENS_VW];
    __shared__ double plane_sum[ENS_VW / ENS_PLANE_WARPS];
    __shared__ double total;
    __shared__ int sb;
    const int tid = threadIdx.x, nt = blockDim.x;
    for (;;) {
        if (rank == 0 && tid == 0) sb = atomicAdd(counter, 1);
        cluster_sync_global(cl);
        const int b = *cl.map_shared_rank(&sb, 0);
        cluster_sync_global(cl);
        if (b >= nbox) break;
        const int bid = order[b];
        const EnsBox B = boxes[bid];
        const Geo g = B.g;
        const int ni = g.ni, nj = g.nj, nk = g.nk;
        const int64_t nn = B.nn;
        double *ph = phi + B.node0;
        double *rh = rho + B.node0;
        float *e = ecor + B.node0;
        float *R = res + B.node0;
        const int64_t n0 = nn * rank / C, n1 = nn * (rank + 1) / C;
        /* 1. rho = sum_s q_s den_s, den_s = counts * unit_s / node_vol; the
         *    accumulators are cleared for the next deposit */
        const double V0 = g.dh[0] * g.dh[1] * g.dh[2];
        const double yV0 = 1.0 / V0;
        const float inv_ni = 1.f / (float)ni, inv_nj = 1.f / (float)nj;
        const bool small = nn < (1 << 24); /* div_small's range, whatever the axes */
        const int64_t slab_e = 4 * ens_slab_e(ni, nj, nk, C), slab_r = 4 * ens_slab_r(ni, nj, nk, C);
        const bool slab = ROUTES == ENS_SLAB || ((ROUTES & ENS_SLAB) && ens_has_slab(ni, nj, nk, C, slab_bytes));
        for (int64_t u = n0 + tid; u < n1; u += nt) {
            int i, j, k;
            if (small) {
                const uint32_t row = div_small((uint32_t)u, (uint32_t)ni, inv_ni);
                k = (int)div_small(row, (uint32_t)nj, inv_nj);
                i = (int)((uint32_t)u - row * (uint32_t)ni);
                j = (int)(row - (uint32_t)k * (uint32_t)nj);
            } else {
                i = (int)(u % ni), j = (int)((u / ni) % nj), k = (int)(u / ((int64_t)ni * nj));
            }
            double r = 0;
            const int faces = (i == 0 || i == ni - 1) + (j == 0 || j == nj - 1) + (k == 0 || k == nk - 1);
            const double halved = __hiloint2double((1023 + faces) << 20, 0); /* 2^faces */
            for (int s = 0; s < nsp; s++) {
                const EnsSeg &sg = segs[bid * nsp + s];
                unsigned long long *A = acc + (int64_t)s * total_nodes + B.node0;
                /* the halvings of the volume multiply the unit, exactly */
                const double d = __ll2double_rn((long long)A[u]) * (sg.unit * halved);
                A[u] = 0ull;
                if (sg.q != 0) r += div_rcp(d, V0, yV0) * sg.q;
            }
            rh[u] = r;
            if (!slab) e[u] = 0.f;
        }
        cluster_sync_global(cl);
        /* 2. red-black SOR: float32 correction sweeps under the float64
         *    residual */
        const int sy = ni, sz = ni * nj;
        EnsSolved done = {0, 0, 0.0};
        if (solve && slab)
            done = ens_sor_slab(B, ph, rh, R, e, max_it, tol, slab_e + slab_r <= slab_bytes, ens_slab, part, plane_sum,
                                &total, err);
        else if (solve) /* the planes' sums where the box's E will be written */
            done = ROUTES == ENS_GLOBAL
                       ? ens_sor_global_call(boxes[bid], ph, rh, R, e, max_it, tol, (double *)(ef4 + B.node0), part,
                                             &total, err)
                       : ens_sor_global(B, ph, rh, R, e, max_it, tol, (double *)(ef4 + B.node0), part, &total, err);
        /* 3. E = -grad phi, float32 copy for the push */
        /* interior nodes first, the face nodes in passes of their own: a
         * row of at most 64 nodes puts a face lane into every warp, and the
         * warp would issue the one-sided formulas for all its nodes */
        const EfRcp rc = ef_rcp(g);
        if (small) {
            const uint32_t in_i = (uint32_t)(ni - 2), in_j = (uint32_t)(nj - 2), in_k = (uint32_t)(nk - 2);
            const uint32_t nin = in_i * in_j * in_k;
            const uint32_t a0 = (uint32_t)((int64_t)nin * rank / C), a1 = (uint32_t)((int64_t)nin * (rank + 1) / C);
            const float inv_i = 1.f / (float)in_i, inv_j = 1.f / (float)in_j;
            for (uint32_t t = a0 + tid; t < a1; t += nt) {
                const uint32_t row = div_small(t, in_i, inv_i), kk = div_small(row, in_j, inv_j);
                const int u = ((1 + (int)kk) * nj + 1 + (int)(row - kk * in_j)) * ni + 1 + (int)(t - row * in_i);
                const double e0 = div_rcp(-(ph[u + 1] - ph[u - 1]), rc.d2[0], rc.y2[0]);
                const double e1 = div_rcp(-(ph[u + sy] - ph[u - sy]), rc.d2[1], rc.y2[1]);
                const double e2 = div_rcp(-(ph[u + sz] - ph[u - sz]), rc.d2[2], rc.y2[2]);
                ef4[B.node0 + u] = make_float4((float)e0, (float)e1, (float)e2, 0.f);
            }
            /* k faces, j faces, i faces, each node once */
            const uint32_t fk = (uint32_t)(ni * nj), fj = (uint32_t)ni * in_k, fi = in_j * in_k;
            const uint32_t nf = 2 * (fk + fj + fi);
            const uint32_t b0 = (uint32_t)((int64_t)nf * rank / C), b1 = (uint32_t)((int64_t)nf * (rank + 1) / C);
            for (uint32_t t = b0 + tid; t < b1; t += nt) {
                uint32_t q = t >> 1;
                const bool far = t & 1;
                int i, j, k;
                if (q < fk) {
                    j = (int)div_small(q, (uint32_t)ni, inv_ni);
                    i = (int)q - j * ni;
                    k = far ? nk - 1 : 0;
                } else if ((q -= fk) < fj) {
                    k = (int)div_small(q, (uint32_t)ni, inv_ni);
                    i = (int)q - k * ni;
                    k += 1;
                    j = far ? nj - 1 : 0;
                } else {
                    q -= fj;
                    k = (int)div_small(q, in_j, inv_j);
                    j = 1 + (int)(q - (uint32_t)k * in_j);
                    k += 1;
                    i = far ? ni - 1 : 0;
                }
                const int64_t u = ((int64_t)k * nj + j) * ni + i;
                double e0, e1, e2;
                ens_efield(g, rc, ph, u, i, j, k, e0, e1, e2);
                ef4[B.node0 + u] = make_float4((float)e0, (float)e1, (float)e2, 0.f);
            }
        }
        for (int64_t u = n0 + tid; u < n1 && !small; u += nt) {
            const int i = (int)(u % ni), j = (int)((u / ni) % nj), k = (int)(u / ((int64_t)ni * nj));
            double e0, e1, e2;
            ens_efield(g, rc, ph, u, i, j, k, e0, e1, e2);
            ef4[B.node0 + u] = make_float4((float)e0, (float)e1, (float)e2, 0.f);
        }
        if (rank == 0 && tid == 0) {
            stat[bid].sweeps = done.sweeps;
            stat[bid].converged = done.converged;
            stat[bid].residual = done.residual;
        }
        cluster_sync_global(cl);
    }
}

/* float64 E of one box (for reading) */
__global__ void k_ens_efield64(Geo g, const double *__restrict__ phi, double *ef) {
    int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t nn = (int64_t)g.ni * g.nj * g.nk;
    if (u >= nn) return;
    const int i = (int)(u % g.ni), j = (int)((u / g.ni) % g.nj), k = (int)(u / ((int64_t)g.ni * g.nj));
    double e0, e1, e2;
    ens_efield(g, ef_rcp(g), phi, u, i, j, k, e0, e1, e2);
    ef[3 * u] = e0;
    ef[3 * u + 1] = e1;
    ef[3 * u + 2] = e2;
}

/* den of one species of one box from its accumulator (for reading) */
__global__ void k_ens_density(Geo g, const unsigned long long *__restrict__ acc, double unit, double *den) {
    int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t nn = (int64_t)g.ni * g.nj * g.nk;
    if (u >= nn) return;
    const int i = (int)(u % g.ni), j = (int)((u / g.ni) % g.nj), k = (int)(u / ((int64_t)g.ni * g.nj));
    const double V0 = g.dh[0] * g.dh[1] * g.dh[2];
    const double d = __ll2double_rn((long long)acc[u]) * unit;
    den[u] = ens_per_volume(g, i, j, k, d, V0, 1.0 / V0);
}

/* loadParticlesBox (ch2/Species.cpp:74-97) into a segment: x = x1 + U (x2 -
 * x1) per axis from Philox stream `stream` (uniforms 3p, 3p+1, 3p+2), v = 0
 * (the half-step rewind of addParticle with the zero field of a new box) */
__global__ void k_ens_load(Geo g, double3 x1, double3 x2, int64_t n, uint64_t seed, uint64_t stream, int64_t first,
                           int32_t *cell, float *off, float *vel, int64_t stride) {
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const double a[3] = {x1.x, x1.y, x1.z}, b[3] = {x2.x, x2.y, x2.z};
    const int nmax[3] = {g.ni, g.nj, g.nk};
    int c[3];
    for (int d = 0; d < 3; d++) {
        const double x = a[d] + philox_uniform(seed, stream, 3 * (uint64_t)p + d) * (b[d] - a[d]);
        const double lc = (x - g.x0[d]) / g.dh[d];
        int i = (int)lc;
        if (i < 0) i = 0;
        if (i > nmax[d] - 2) i = nmax[d] - 2;
        c[d] = i;
        off[d * stride + first + p] = (float)(lc - i);
        vel[d * stride + first + p] = 0.f;
    }
    cell[first + p] = c[0] | (c[1] << 10) | (c[2] << 20);
}

/* per box: kinetic energy of every species (0.5 m mpw0 sum v^2, getKE of
 * ch2/Species.cpp:144-168) and the field energy 0.5 eps0 sum E^2 dV
 * (World::getPE, ch2/World.cpp:72-84); one block per box, fixed order */
__global__ void __launch_bounds__(256) k_ens_diag(const EnsBox *__restrict__ boxes, const EnsSeg *__restrict__ segs,
                                                  int nsp, const double *__restrict__ mass, const double *mpw,
                                                  const double *__restrict__ phi, const float *__restrict__ vel,
                                                  int64_t stride, double *out) {
    __shared__ double part[ENS_VW];
    const int bid = blockIdx.x;
    const EnsBox B = boxes[bid];
    const Geo g = B.g;
    const int ncol = nsp + 1;
    for (int s = 0; s < nsp; s++) {
        const EnsSeg sg = segs[bid * nsp + s];
        for (int v = threadIdx.x; v < ENS_VW; v += blockDim.x) {
            double a = 0;
            for (int64_t q = v; q < sg.n; q += ENS_VW) {
                const int64_t p = sg.p0 + q;
                const double vx = vel[p], vy = vel[stride + p], vz = vel[2 * stride + p];
                a += vx * vx + vy * vy + vz * vz;
            }
            part[v] = a;
        }
        const double t = ens_tree_sum(part);
        if (threadIdx.x == 0) out[bid * ncol + s] = 0.5 * mass[s] * mpw[bid * nsp + s] * t;
    }
    const double *ph = phi + B.node0;
    const EfRcp rc = ef_rcp(g);
    for (int v = threadIdx.x; v < ENS_VW; v += blockDim.x) {
        double a = 0;
        for (int64_t u = v; u < B.nn; u += ENS_VW) {
            const int i = (int)(u % g.ni), j = (int)((u / g.ni) % g.nj), k = (int)(u / ((int64_t)g.ni * g.nj));
            double e0, e1, e2;
            ens_efield(g, rc, ph, u, i, j, k, e0, e1, e2);
            a += (e0 * e0 + e1 * e1 + e2 * e2) * ens_node_volume(g, i, j, k);
        }
        part[v] = a;
    }
    const double t = ens_tree_sum(part);
    if (threadIdx.x == 0) out[bid * ncol + nsp] = 0.5 * ENS_EPS_0 * t;
}

}  // namespace espic

/* ======================================================================== */
/* C-ABI                                                                    */
using namespace espic;

struct espic_ensemble {
    int nbox = 0, nsp = 0, device = 0, sm_count = 0;
    cudaStream_t stream = nullptr;
    double dt = 0;
    uint64_t seed = 0x5eed;
    std::vector<EnsBox> boxes;
    std::vector<int32_t> box_id; /* the id that keys each box's random streams (default: its index) */
    std::vector<EnsSeg> segs; /* [box][species] */
    std::vector<double> mass, charge, mpw0;
    int64_t total_nodes = 0, total_cap = 0;
    EnsBox *d_boxes = nullptr;
    EnsSeg *d_segs = nullptr;
    double *d_mass = nullptr, *d_mpw = nullptr;
    double *phi = nullptr, *rho = nullptr;
    float4 *ef4 = nullptr;
    float *ecor = nullptr, *res = nullptr;
    unsigned long long *acc = nullptr;
    int32_t *cell = nullptr;
    float *off = nullptr, *vel = nullptr;
    int4 *d_work = nullptr;
    int nwork = 0;
    bool work_valid = false;
    int *d_order = nullptr, *d_counter = nullptr, *d_err = nullptr;
    EnsStat *d_stat = nullptr;
    double *d_scratch = nullptr;
    size_t scratch_bytes = 0;
    int max_it = 10000;
    double tol = 1e-4, omega_req = 0;
    int chunk = 4096, push_threads = 256, solve_threads = 1024, cluster = 8;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int64_t nlaunch = 0, steps = 0;
};

static int efail(int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    return espic_internal_fail(code, buf);
}

#define ECK(call)                                                                                       \
    do {                                                                                                \
        cudaError_t e_ = (call);                                                                        \
        if (e_ != cudaSuccess) return efail(ESPIC_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_));   \
    } while (0)

#define ENSEMBLE(h)                                                        \
    if (!(h)) return efail(ESPIC_ERR_ARG, "null ensemble handle");         \
    espic_ensemble &E = *(h);                                              \
    if (cudaSetDevice(E.device) != cudaSuccess) return efail(ESPIC_ERR_CUDA, "cudaSetDevice failed")

template <typename T>
static cudaError_t ens_alloc(T **p, size_t count) {
    cudaError_t e = cudaMalloc((void **)p, count * sizeof(T) + 16);
    if (e == cudaSuccess) e = cudaMemset(*p, 0, count * sizeof(T) + 16);
    return e;
}

static void ens_free(espic_ensemble *e) {
    if (e->exec) cudaGraphExecDestroy(e->exec);
    if (e->graph) cudaGraphDestroy(e->graph);
    void *ptrs[] = {e->d_boxes, e->d_segs, e->d_mass, e->d_mpw, e->phi, e->rho, e->ef4, e->ecor, e->res, e->acc,
                    e->cell, e->off, e->vel, e->d_work, e->d_order, e->d_counter, e->d_err, e->d_stat,
                    e->d_scratch};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    if (e->stream) cudaStreamDestroy(e->stream);
    delete e;
}

/* optimal red-black SOR factor of the Dirichlet 7-point Laplacian on a box
 * (Young): rho_J = sum c_d cos(pi / (n_d - 1)) / sum c_d */
static double omega_opt(const Geo &g) {
    double c[3], num = 0, den = 0;
    int n[3] = {g.ni, g.nj, g.nk};
    for (int d = 0; d < 3; d++) {
        c[d] = 1.0 / (g.dh[d] * g.dh[d]);
        num += c[d] * cos(3.14159265358979323846 / (n[d] - 1));
        den += c[d];
    }
    double rj = num / den;
    return 2.0 / (1.0 + sqrt(1.0 - rj * rj));
}

static void ens_set_omega(espic_ensemble &E) {
    for (EnsBox &b : E.boxes) b.omega = E.omega_req > 0 ? E.omega_req : omega_opt(b.g);
}

static int ens_upload_tables(espic_ensemble &E) {
    ECK(cudaMemcpyAsync(E.d_boxes, E.boxes.data(), E.boxes.size() * sizeof(EnsBox), cudaMemcpyHostToDevice,
                        E.stream));
    ECK(cudaMemcpyAsync(E.d_segs, E.segs.data(), E.segs.size() * sizeof(EnsSeg), cudaMemcpyHostToDevice,
                        E.stream));
    ECK(cudaStreamSynchronize(E.stream));
    return ESPIC_OK;
}

static void ens_drop_graph(espic_ensemble &E) {
    if (E.exec) cudaGraphExecDestroy(E.exec);
    if (E.graph) cudaGraphDestroy(E.graph);
    E.exec = nullptr;
    E.graph = nullptr;
}

/* the flattened work list: chunks of at most E.chunk particles, each inside
 * one segment, the largest segments first */
static int ens_build_work(espic_ensemble &E) {
    std::vector<int> sidx(E.segs.size());
    for (size_t i = 0; i < sidx.size(); i++) sidx[i] = (int)i;
    std::stable_sort(sidx.begin(), sidx.end(), [&](int a, int b) { return E.segs[a].n > E.segs[b].n; });
    std::vector<int4> work;
    for (int si : sidx) {
        const EnsSeg &s = E.segs[si];
        for (int64_t st = 0; st < s.n; st += E.chunk) {
            int64_t c = s.n - st < E.chunk ? s.n - st : E.chunk;
            work.push_back(make_int4(si, (int)st, (int)c, 0));
        }
    }
    if (E.d_work) cudaFree(E.d_work);
    E.d_work = nullptr;
    E.nwork = (int)work.size();
    if (E.nwork) {
        ECK(cudaMalloc(&E.d_work, work.size() * sizeof(int4)));
        ECK(cudaMemcpy(E.d_work, work.data(), work.size() * sizeof(int4), cudaMemcpyHostToDevice));
    }
    E.work_valid = true;
    return ESPIC_OK;
}

static int ens_push_blocks(espic_ensemble &E) {
    int64_t b = (int64_t)E.sm_count * (2048 / E.push_threads);
    return (int)(E.nwork < b ? (E.nwork > 0 ? E.nwork : 1) : b);
}

/* Shared memory of the solve launch: for the largest slab that fits
 * (correction and right-hand side, or the correction alone), or none.  A
 * launch with slabs leaves little L1, and the slower of its two forms, to the
 * boxes that do not fit: they take 15% longer (64 boxes of 16 to 64 nodes an
 * axis with single CTAs of 256 threads, where the largest boxes decide: 114 ms
 * without slabs, 131 with), the others half as long (8 CTAs of 1024 threads:
 * 15.5 and 7.7 ms; 512 such boxes with 4 CTAs, of which the largest do not
 * fit: 39 and 27 ms a step).
 * A box's time goes as its nodes and, through the sweeps, its longest axis;
 * the launch's is that of the largest box or the sum over the clusters. */
static int64_t ens_slab_launch(const espic_ensemble &E) {
    int64_t bytes = 0;
    double with = 0, without = 0, sum_with = 0, sum_without = 0;
    for (const EnsBox &b : E.boxes) {
        const int64_t e = 4 * ens_slab_e(b.g.ni, b.g.nj, b.g.nk, E.cluster);
        const int64_t er = e + 4 * ens_slab_r(b.g.ni, b.g.nj, b.g.nk, E.cluster);
        const bool fits = ens_has_slab(b.g.ni, b.g.nj, b.g.nk, E.cluster, ENS_SLAB_MAX);
        if (fits) bytes = std::max(bytes, er <= ENS_SLAB_MAX ? er : e);
        const double t = (double)b.nn * std::max(b.g.ni, std::max(b.g.nj, b.g.nk));
        const double t_with = fits ? 0.5 * t : 1.15 * t;
        with = std::max(with, t_with);
        without = std::max(without, t);
        sum_with += t_with;
        sum_without += t;
    }
    const double clusters = std::max(1, E.sm_count / E.cluster);
    return std::max(with, sum_with / clusters) <= std::max(without, sum_without / clusters) ? bytes : 0;
}

/* the solve launch: clusters of E.cluster CTAs, as many as can be resident
 * (one box each at a time), at most one per box */
static cudaError_t ens_launch_solve(espic_ensemble &E, int solve) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = E.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(E.solve_threads);
    const int64_t bytes = ens_slab_launch(E);
    int routes = 0;
    for (const EnsBox &b : E.boxes)
        routes |= ens_has_slab(b.g.ni, b.g.nj, b.g.nk, E.cluster, bytes) ? ENS_SLAB : ENS_GLOBAL;
    auto *fn = routes == ENS_SLAB     ? k_ens_solve<ENS_SLAB>
               : routes == ENS_GLOBAL ? k_ens_solve<ENS_GLOBAL>
                                      : k_ens_solve<ENS_SLAB | ENS_GLOBAL>;
    /* the limit belongs to the kernel, not to this ensemble: always the same
     * value, or another thread's ensemble could lower it before the launch */
    cudaError_t fe = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ENS_SLAB_MAX);
    if (fe != cudaSuccess) return fe;
    cfg.dynamicSmemBytes = (size_t)bytes;
    cfg.stream = E.stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(E.cluster);
    int ncl = 0;
    cudaError_t ce = cudaOccupancyMaxActiveClusters(&ncl, (void *)fn, &cfg);
    if (ce != cudaSuccess || ncl < 1) ncl = E.sm_count / E.cluster > 0 ? E.sm_count / E.cluster : 1;
    if (ncl > E.nbox) ncl = E.nbox;
    cfg.gridDim = dim3(ncl * E.cluster);
    return cudaLaunchKernelEx(&cfg, fn, (const EnsBox *)E.d_boxes, (const EnsSeg *)E.d_segs, E.nsp,
                              (const int *)E.d_order, E.nbox, E.d_counter, E.phi, E.rho, E.ecor, E.res, E.ef4, E.acc,
                              E.total_nodes, E.max_it, E.tol, solve, E.d_stat, (int)bytes, E.d_err);
}

/* enqueue one phase sequence: [push +] deposit, then rho / solve / E */
static int ens_enqueue(espic_ensemble &E, bool push, bool solve) {
    if (!E.work_valid) {
        int rc = ens_build_work(E);
        if (rc) return rc;
    }
    launch_ens_push(E.stream, push, ens_push_blocks(E), E.push_threads, E.d_boxes, E.d_segs, E.d_work, E.nwork,
                    E.ef4, E.cell, E.off, E.vel, E.total_cap, E.acc, E.total_nodes, E.d_err);
    ECK(cudaMemsetAsync(E.d_counter, 0, sizeof(int), E.stream));
    ECK(ens_launch_solve(E, solve ? 1 : 0));
    E.nlaunch += E.nwork ? 2 : 1;
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return efail(ESPIC_ERR_CUDA, "ensemble launch: %s", cudaGetErrorString(le));
    return ESPIC_OK;
}

static int ens_take_errors(espic_ensemble &E) {
    int bits = 0;
    ECK(cudaMemcpyAsync(&bits, E.d_err, sizeof(int), cudaMemcpyDeviceToHost, E.stream));
    ECK(cudaStreamSynchronize(E.stream));
    if (bits) ECK(cudaMemsetAsync(E.d_err, 0, sizeof(int), E.stream));
    if (bits & DERR_NONFINITE) return efail(ESPIC_ERR_NONFINITE, "non-finite value in the ensemble step");
    return ESPIC_OK;
}

extern "C" int espic_ensemble_create(int nbox, const int32_t *nodes, const double *x0, const double *xm,
                                     int nspecies, const double *mass, const double *charge, const double *mpw0,
                                     const int64_t *capacity, double dt, espic_ensemble **out) {
    if (!out || !nodes || !x0 || !xm || !mass || !charge || !mpw0 || !capacity)
        return efail(ESPIC_ERR_ARG, "null argument");
    *out = nullptr;
    if (nbox < 1 || nspecies < 1 || nspecies > 8) return efail(ESPIC_ERR_ARG, "need nbox >= 1 and 1..8 species");
    if (!(dt > 0)) return efail(ESPIC_ERR_ARG, "dt must be positive");
    espic_ensemble *e = new espic_ensemble();
    espic_ensemble &E = *e;
    E.nbox = nbox;
    E.nsp = nspecies;
    E.dt = dt;
    cudaGetDevice(&E.device);
    cudaDeviceGetAttribute(&E.sm_count, cudaDevAttrMultiProcessorCount, E.device);
    E.mass.assign(mass, mass + nspecies);
    E.charge.assign(charge, charge + nspecies);
    E.mpw0.assign(mpw0, mpw0 + (size_t)nbox * nspecies);
    int64_t node0 = 0, p0 = 0;
    for (int b = 0; b < nbox; b++) {
        EnsBox bx{};
        int n3[3] = {nodes[3 * b], nodes[3 * b + 1], nodes[3 * b + 2]};
        for (int d = 0; d < 3; d++) {
            if (n3[d] < 3 || n3[d] > 1024) {
                ens_free(e);
                return efail(ESPIC_ERR_ARG, "box %d: node counts must be in [3, 1024]", b);
            }
            if (!(xm[3 * b + d] > x0[3 * b + d])) {
                ens_free(e);
                return efail(ESPIC_ERR_ARG, "box %d: xm must exceed x0", b);
            }
        }
        bx.g.ni = n3[0];
        bx.g.nj = n3[1];
        bx.g.nk = n3[2];
        for (int d = 0; d < 3; d++) {
            bx.g.x0[d] = x0[3 * b + d];
            bx.g.xm[d] = xm[3 * b + d];
            bx.g.dh[d] = (xm[3 * b + d] - x0[3 * b + d]) / (n3[d] - 1);
            bx.dtdh[d] = (float)(dt / bx.g.dh[d]);
        }
        bx.nn = (int64_t)n3[0] * n3[1] * n3[2];
        bx.node0 = node0;
        node0 += (bx.nn + 63) / 64 * 64;
        E.boxes.push_back(bx);
        for (int s = 0; s < nspecies; s++) {
            int64_t cap = capacity[(size_t)b * nspecies + s];
            if (cap < 0 || cap > 0x7fffffffLL) {
                ens_free(e);
                return efail(ESPIC_ERR_ARG, "capacity must be in [0, 2^31)");
            }
            EnsSeg sg{};
            sg.box = b;
            sg.sp = s;
            sg.p0 = p0;
            sg.n = 0;
            sg.cap = cap;
            sg.unit = mpw0[(size_t)b * nspecies + s] / 8388608.0;
            sg.q = charge[s];
            sg.qmdt = (float)(charge[s] / mass[s] * dt);
            p0 += (cap + 63) / 64 * 64;
            E.segs.push_back(sg);
        }
    }
    E.total_nodes = node0;
    E.total_cap = p0 > 0 ? p0 : 64;
    ens_set_omega(E);
    cudaError_t ce = cudaStreamCreateWithFlags(&E.stream, cudaStreamNonBlocking);
    const int64_t TN = E.total_nodes, TC = E.total_cap;
    if (ce == cudaSuccess) ce = ens_alloc(&E.d_boxes, (size_t)nbox);
    if (ce == cudaSuccess) ce = ens_alloc(&E.d_segs, E.segs.size());
    if (ce == cudaSuccess) ce = ens_alloc(&E.d_mass, (size_t)nspecies);
    if (ce == cudaSuccess) ce = ens_alloc(&E.d_mpw, E.mpw0.size());
    if (ce == cudaSuccess) ce = ens_alloc(&E.phi, (size_t)TN);
    if (ce == cudaSuccess) ce = ens_alloc(&E.rho, (size_t)TN);
    if (ce == cudaSuccess) ce = ens_alloc(&E.ef4, (size_t)TN);
    if (ce == cudaSuccess) ce = ens_alloc(&E.ecor, (size_t)TN);
    if (ce == cudaSuccess) ce = ens_alloc(&E.res, (size_t)TN);
    if (ce == cudaSuccess) ce = ens_alloc(&E.acc, (size_t)TN * nspecies);
    if (ce == cudaSuccess) ce = ens_alloc(&E.cell, (size_t)TC);
    if (ce == cudaSuccess) ce = ens_alloc(&E.off, (size_t)TC * 3);
    if (ce == cudaSuccess) ce = ens_alloc(&E.vel, (size_t)TC * 3);
    if (ce == cudaSuccess) ce = ens_alloc(&E.d_order, (size_t)nbox);
    if (ce == cudaSuccess) ce = ens_alloc(&E.d_counter, 1);
    if (ce == cudaSuccess) ce = ens_alloc(&E.d_err, 1);
    if (ce == cudaSuccess) ce = ens_alloc(&E.d_stat, (size_t)nbox);
    if (ce != cudaSuccess) {
        ens_free(e);
        return efail(ESPIC_ERR_CUDA, "ensemble allocation: %s", cudaGetErrorString(ce));
    }
    /* boxes in decreasing node count: the solve claims big boxes first */
    std::vector<int> order(nbox);
    for (int b = 0; b < nbox; b++) order[b] = b;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return E.boxes[a].nn > E.boxes[b].nn; });
    cudaMemcpy(E.d_order, order.data(), nbox * sizeof(int), cudaMemcpyHostToDevice);
    cudaMemcpy(E.d_mass, E.mass.data(), nspecies * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(E.d_mpw, E.mpw0.data(), E.mpw0.size() * sizeof(double), cudaMemcpyHostToDevice);
    int rc = ens_upload_tables(E);
    if (rc) {
        ens_free(e);
        return rc;
    }
    *out = e;
    return ESPIC_OK;
}

extern "C" void espic_ensemble_destroy(espic_ensemble *e) {
    if (!e) return;
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    ens_free(e);
}

#define SEG(box, sp)                                                                              \
    if ((box) < 0 || (box) >= E.nbox || (sp) < 0 || (sp) >= E.nsp)                               \
        return efail(ESPIC_ERR_ARG, "box %d / species %d out of range", (int)(box), (int)(sp));  \
    EnsSeg &S = E.segs[(size_t)(box)*E.nsp + (sp)];                                               \
    const EnsBox &BX = E.boxes[(box)]

extern "C" int espic_ensemble_set_particles(espic_ensemble *h, int box, int sp, const double *P, int64_t stride,
                                            int64_t n) {
    ENSEMBLE(h);
    SEG(box, sp);
    if (n < 0 || (n > 0 && (!P || stride < n))) return efail(ESPIC_ERR_ARG, "bad particle block");
    if (n > S.cap) return efail(ESPIC_ERR_CAPACITY, "%lld particles exceed the capacity", (long long)n);
    if (n > 0) {
        size_t bytes = (size_t)7 * n * sizeof(double);
        if (E.scratch_bytes < bytes) {
            if (E.d_scratch) cudaFree(E.d_scratch);
            E.d_scratch = nullptr;
            E.scratch_bytes = 0;
            ECK(cudaMalloc(&E.d_scratch, bytes));
            E.scratch_bytes = bytes;
        }
        ECK(cudaMemcpy2DAsync(E.d_scratch, n * sizeof(double), P, stride * sizeof(double), n * sizeof(double), 7,
                              cudaMemcpyHostToDevice, E.stream));
        launch_to_mixed_raw(E.stream, BX.g, E.d_scratch, n, n, S.p0, E.cell, E.off, E.vel, E.total_cap);
        E.nlaunch++;
        ECK(cudaGetLastError());
        ECK(cudaStreamSynchronize(E.stream));
    }
    S.n = n;
    E.work_valid = false;
    ens_drop_graph(E);
    return ens_upload_tables(E);
}

extern "C" int espic_ensemble_load_box(espic_ensemble *h, int box, int sp, const double x1[3], const double x2[3],
                                       int64_t num_mp) {
    ENSEMBLE(h);
    SEG(box, sp);
    if (!x1 || !x2) return efail(ESPIC_ERR_ARG, "null argument");
    if (num_mp < 0 || num_mp > S.cap) return efail(ESPIC_ERR_CAPACITY, "num_mp exceeds the capacity");
    for (int d = 0; d < 3; d++)
        if (x1[d] < BX.g.x0[d] || x2[d] > BX.g.xm[d] || !(x2[d] > x1[d]))
            return efail(ESPIC_ERR_ARG, "load region must lie inside the box");
    const uint64_t id = E.box_id.empty() ? (uint64_t)box : (uint64_t)E.box_id[box];
    uint64_t stream = ((uint64_t)(0x40000 + id * E.nsp + sp)) << 32;
    if (num_mp > 0) {
        k_ens_load<<<blocks_for(num_mp, 256), 256, 0, E.stream>>>(BX.g, make_double3(x1[0], x1[1], x1[2]),
                                                                  make_double3(x2[0], x2[1], x2[2]), num_mp, E.seed,
                                                                  stream, S.p0, E.cell, E.off, E.vel, E.total_cap);
        E.nlaunch++;
        ECK(cudaGetLastError());
    }
    S.n = num_mp;
    E.work_valid = false;
    ens_drop_graph(E);
    return ens_upload_tables(E);
}

extern "C" int espic_ensemble_set_box_ids(espic_ensemble *h, const int32_t *ids) {
    ENSEMBLE(h);
    if (!ids) {
        E.box_id.clear();
        return ESPIC_OK;
    }
    for (int b = 0; b < E.nbox; b++)
        if (ids[b] < 0 || ids[b] >= (1 << 24)) return efail(ESPIC_ERR_ARG, "box id %d out of range", ids[b]);
    E.box_id.assign(ids, ids + E.nbox);
    return ESPIC_OK;
}

extern "C" int espic_partition_boxes(int nbox, const double *work, int nparts, int32_t *owner, double *load) {
    if (nbox < 0 || nparts < 1 || (nbox > 0 && (!work || !owner)))
        return efail(ESPIC_ERR_ARG, "bad partition arguments");
    for (int b = 0; b < nbox; b++)
        if (!(work[b] >= 0)) return efail(ESPIC_ERR_ARG, "box %d: work must be finite and >= 0", b);
    /* largest work first (ties by box index), each to the least loaded part
     * (ties to the lowest part): deterministic on every rank */
    std::vector<int> order(nbox);
    for (int b = 0; b < nbox; b++) order[b] = b;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return work[a] > work[b]; });
    std::vector<double> L(nparts, 0.0);
    for (int b : order) {
        int best = 0;
        for (int r = 1; r < nparts; r++)
            if (L[r] < L[best]) best = r;
        owner[b] = best;
        L[best] += work[b];
    }
    if (load)
        for (int r = 0; r < nparts; r++) load[r] = L[r];
    return ESPIC_OK;
}

extern "C" int espic_ensemble_set_seed(espic_ensemble *h, uint64_t seed) {
    ENSEMBLE(h);
    E.seed = seed;
    return ESPIC_OK;
}

extern "C" int espic_ensemble_get_particles(espic_ensemble *h, int box, int sp, double *P, int64_t stride,
                                            int64_t cap, int64_t *n_out) {
    ENSEMBLE(h);
    SEG(box, sp);
    if (n_out) *n_out = S.n;
    if (S.n == 0 || !P) return ESPIC_OK; /* P = NULL: count only */
    if (cap < S.n || stride < S.n) return efail(ESPIC_ERR_ARG, "buffer smaller than the particle count");
    size_t bytes = (size_t)7 * S.n * sizeof(double);
    if (E.scratch_bytes < bytes) {
        if (E.d_scratch) cudaFree(E.d_scratch);
        E.d_scratch = nullptr;
        E.scratch_bytes = 0;
        ECK(cudaMalloc(&E.d_scratch, bytes));
        E.scratch_bytes = bytes;
    }
    launch_from_mixed_raw(E.stream, BX.g, E.cell, E.off, E.vel, E.total_cap, S.p0, S.n, E.mpw0[(size_t)box * E.nsp + sp],
                          E.d_scratch, S.n);
    E.nlaunch++;
    ECK(cudaGetLastError());
    ECK(cudaMemcpy2DAsync(P, stride * sizeof(double), E.d_scratch, S.n * sizeof(double), S.n * sizeof(double), 7,
                          cudaMemcpyDeviceToHost, E.stream));
    ECK(cudaStreamSynchronize(E.stream));
    return ESPIC_OK;
}

extern "C" int espic_ensemble_set_solver(espic_ensemble *h, int max_it, double tol, double omega) {
    ENSEMBLE(h);
    if (max_it < 0 || !(tol > 0) || omega < 0 || omega >= 2) return efail(ESPIC_ERR_ARG, "bad solver controls");
    E.max_it = max_it;
    E.tol = tol;
    E.omega_req = omega;
    ens_set_omega(E);
    ens_drop_graph(E);
    return ens_upload_tables(E);
}

extern "C" int espic_ensemble_set_launch(espic_ensemble *h, int chunk, int push_threads, int solve_threads,
                                         int cluster) {
    ENSEMBLE(h);
    bool okp = push_threads == 128 || push_threads == 256 || push_threads == 512;
    bool oks = solve_threads == 256 || solve_threads == 512 || solve_threads == 1024;
    bool okc = cluster == 1 || cluster == 2 || cluster == 4 || cluster == 8;
    if (chunk < 256 || chunk > (1 << 24) || !okp || !oks || !okc) return efail(ESPIC_ERR_ARG, "bad launch shape");
    if (chunk != E.chunk) E.work_valid = false;
    E.chunk = chunk;
    E.push_threads = push_threads;
    E.solve_threads = solve_threads;
    E.cluster = cluster;
    ens_drop_graph(E);
    return ESPIC_OK;
}

extern "C" int espic_ensemble_get_launch(espic_ensemble *h, int *chunk, int *push_threads, int *solve_threads,
                                         int *cluster) {
    ENSEMBLE(h);
    if (chunk) *chunk = E.chunk;
    if (push_threads) *push_threads = E.push_threads;
    if (solve_threads) *solve_threads = E.solve_threads;
    if (cluster) *cluster = E.cluster;
    return ESPIC_OK;
}

/* the state before the first step of ch2/Main.cpp: deposit, charge density,
 * solve, E */
extern "C" int espic_ensemble_prepare(espic_ensemble *h) {
    ENSEMBLE(h);
    int rc = ens_enqueue(E, false, true);
    if (rc) return rc;
    return ens_take_errors(E);
}

/* nsteps steps (push + deposit, charge, solve, E), each one launch of the
 * step's CUDA graph; asynchronous unless an error must be reported */
extern "C" int espic_ensemble_step(espic_ensemble *h, int nsteps) {
    ENSEMBLE(h);
    if (nsteps < 0) return efail(ESPIC_ERR_ARG, "nsteps must be >= 0");
    if (!E.work_valid) {
        int rc = ens_build_work(E);
        if (rc) return rc;
    }
    if (!E.exec) {
        ECK(cudaStreamBeginCapture(E.stream, cudaStreamCaptureModeThreadLocal));
        int64_t before = E.nlaunch;
        int rc = ens_enqueue(E, true, true);
        cudaGraph_t g = nullptr;
        cudaError_t ce = cudaStreamEndCapture(E.stream, &g);
        if (rc) {
            if (g) cudaGraphDestroy(g);
            return rc;
        }
        if (ce != cudaSuccess) return efail(ESPIC_ERR_CUDA, "graph capture: %s", cudaGetErrorString(ce));
        E.nlaunch = before;
        E.graph = g;
        ECK(cudaGraphInstantiate(&E.exec, g, 0));
    }
    for (int s = 0; s < nsteps; s++) {
        ECK(cudaGraphLaunch(E.exec, E.stream));
        E.nlaunch += E.nwork ? 2 : 1;
        E.steps++;
    }
    return ESPIC_OK;
}

/* the same step as direct launches (no graph) */
extern "C" int espic_ensemble_step_direct(espic_ensemble *h, int nsteps) {
    ENSEMBLE(h);
    for (int s = 0; s < nsteps; s++) {
        int rc = ens_enqueue(E, true, true);
        if (rc) return rc;
        E.steps++;
    }
    return ESPIC_OK;
}

extern "C" int espic_ensemble_sync(espic_ensemble *h) {
    ENSEMBLE(h);
    return ens_take_errors(E);
}

extern "C" void *espic_ensemble_stream(espic_ensemble *h) { return h ? (void *)h->stream : nullptr; }

extern "C" int espic_ensemble_launches(espic_ensemble *h, int64_t *n) {
    ENSEMBLE(h);
    if (n) *n = E.nlaunch;
    return ESPIC_OK;
}

extern "C" int espic_ensemble_status(espic_ensemble *h, int32_t *sweeps, int32_t *converged, double *residual) {
    ENSEMBLE(h);
    std::vector<EnsStat> st(E.nbox);
    ECK(cudaMemcpyAsync(st.data(), E.d_stat, E.nbox * sizeof(EnsStat), cudaMemcpyDeviceToHost, E.stream));
    ECK(cudaStreamSynchronize(E.stream));
    for (int b = 0; b < E.nbox; b++) {
        if (sweeps) sweeps[b] = st[b].sweeps;
        if (converged) converged[b] = st[b].converged;
        if (residual) residual[b] = st[b].residual;
    }
    return ens_take_errors(E);
}

/* field of one box: ESPIC_FIELD_PHI, RHO, EF ([nn][3]) or DEN of species sp
 * (deposited from the current particles) */
extern "C" int espic_ensemble_read(espic_ensemble *h, int box, int field, int sp, double *out) {
    ENSEMBLE(h);
    if (box < 0 || box >= E.nbox || !out) return efail(ESPIC_ERR_ARG, "bad box or null output");
    const EnsBox &B = E.boxes[box];
    size_t nn = (size_t)B.nn;
    if (field == ESPIC_FIELD_PHI || field == ESPIC_FIELD_RHO) {
        const double *src = (field == ESPIC_FIELD_PHI ? E.phi : E.rho) + B.node0;
        ECK(cudaMemcpyAsync(out, src, nn * sizeof(double), cudaMemcpyDeviceToHost, E.stream));
        ECK(cudaStreamSynchronize(E.stream));
        return ESPIC_OK;
    }
    size_t need = (field == ESPIC_FIELD_EF ? 3 : 1) * nn * sizeof(double);
    if (E.scratch_bytes < need) {
        if (E.d_scratch) cudaFree(E.d_scratch);
        E.d_scratch = nullptr;
        E.scratch_bytes = 0;
        ECK(cudaMalloc(&E.d_scratch, need));
        E.scratch_bytes = need;
    }
    if (field == ESPIC_FIELD_EF) {
        k_ens_efield64<<<blocks_for((int64_t)nn, 256), 256, 0, E.stream>>>(B.g, E.phi + B.node0, E.d_scratch);
        E.nlaunch++;
    } else if (field == ESPIC_FIELD_DEN) {
        if (sp < 0 || sp >= E.nsp) return efail(ESPIC_ERR_ARG, "species out of range");
        /* deposit every box into the (clear) accumulators, convert this one,
         * clear them again */
        if (!E.work_valid) {
            int rc = ens_build_work(E);
            if (rc) return rc;
        }
        launch_ens_push(E.stream, false, ens_push_blocks(E), E.push_threads, E.d_boxes, E.d_segs, E.d_work,
                        E.nwork, E.ef4, E.cell, E.off, E.vel, E.total_cap, E.acc, E.total_nodes, E.d_err);
        const EnsSeg &S = E.segs[(size_t)box * E.nsp + sp];
        k_ens_density<<<blocks_for((int64_t)nn, 256), 256, 0, E.stream>>>(
            B.g, E.acc + (int64_t)sp * E.total_nodes + B.node0, S.unit, E.d_scratch);
        E.nlaunch += 2;
        ECK(cudaGetLastError());
        ECK(cudaMemsetAsync(E.acc, 0, (size_t)E.total_nodes * E.nsp * sizeof(unsigned long long), E.stream));
    } else {
        return efail(ESPIC_ERR_ARG, "field %d cannot be read from an ensemble", field);
    }
    ECK(cudaGetLastError());
    ECK(cudaMemcpyAsync(out, E.d_scratch, need, cudaMemcpyDeviceToHost, E.stream));
    ECK(cudaStreamSynchronize(E.stream));
    return ESPIC_OK;
}

/* out[box][0..nsp) kinetic energy per species, out[box][nsp] field energy */
extern "C" int espic_ensemble_diag(espic_ensemble *h, double *out) {
    ENSEMBLE(h);
    if (!out) return efail(ESPIC_ERR_ARG, "null output");
    size_t need = (size_t)E.nbox * (E.nsp + 1) * sizeof(double);
    if (E.scratch_bytes < need) {
        if (E.d_scratch) cudaFree(E.d_scratch);
        E.d_scratch = nullptr;
        E.scratch_bytes = 0;
        ECK(cudaMalloc(&E.d_scratch, need));
        E.scratch_bytes = need;
    }
    k_ens_diag<<<E.nbox, 256, 0, E.stream>>>(E.d_boxes, E.d_segs, E.nsp, E.d_mass, E.d_mpw, E.phi, E.vel,
                                            E.total_cap, E.d_scratch);
    E.nlaunch++;
    ECK(cudaGetLastError());
    ECK(cudaMemcpyAsync(out, E.d_scratch, need, cudaMemcpyDeviceToHost, E.stream));
    ECK(cudaStreamSynchronize(E.stream));
    return ens_take_errors(E);
}

/* Autotuner: times every candidate launch shape on real steps (results do not
 * depend on the shape: per-particle pushes, integer deposits, colour-ordered
 * sweeps, fixed-width reductions) with CUDA events around the two phases, and
 * keeps the fastest chunk / push block for the push phase and the fastest
 * cluster size / solve block for the solve phase.  Consumes 27 steps. */
extern "C" int espic_ensemble_autotune(espic_ensemble *h, int *chunk, int *push_threads, int *solve_threads,
                                       double *push_ms, double *solve_ms) {
    ENSEMBLE(h);
    const int chunks[] = {1024, 2048, 4096, 8192, 16384};
    const int pts[] = {128, 256, 512};
    const int sts[] = {256, 512, 1024};
    const int cls[] = {1, 2, 4, 8};
    cudaEvent_t a, b, c;
    ECK(cudaEventCreate(&a));
    ECK(cudaEventCreate(&b));
    ECK(cudaEventCreate(&c));
    float best_push = 1e30f, best_solve = 1e30f;
    int bc = E.chunk, bp = E.push_threads, bs = E.solve_threads;
    for (int ci = 0; ci < 5; ci++)
        for (int pi = 0; pi < 3; pi++) {
            E.chunk = chunks[ci];
            E.push_threads = pts[pi];
            E.work_valid = false;
            int rc = ens_build_work(E);
            if (rc) return rc;
            ECK(cudaEventRecord(a, E.stream));
            launch_ens_push(E.stream, true, ens_push_blocks(E), E.push_threads, E.d_boxes, E.d_segs, E.d_work,
                            E.nwork, E.ef4, E.cell, E.off, E.vel, E.total_cap, E.acc, E.total_nodes, E.d_err);
            ECK(cudaEventRecord(b, E.stream));
            ECK(cudaMemsetAsync(E.d_counter, 0, sizeof(int), E.stream));
            ECK(ens_launch_solve(E, 1));
            E.nlaunch += 2;
            E.steps++;
            ECK(cudaGetLastError());
            ECK(cudaEventSynchronize(b));
            float ms = 0;
            ECK(cudaEventElapsedTime(&ms, a, b));
            if (ms < best_push) {
                best_push = ms;
                bc = E.chunk;
                bp = E.push_threads;
            }
        }
    E.chunk = bc;
    E.push_threads = bp;
    E.work_valid = false;
    int rc = ens_build_work(E);
    if (rc) return rc;
    int bcl = E.cluster;
    for (int ki = 0; ki < 4; ki++)
        for (int si = 0; si < 3; si++) {
            E.cluster = cls[ki];
            E.solve_threads = sts[si];
            launch_ens_push(E.stream, true, ens_push_blocks(E), E.push_threads, E.d_boxes, E.d_segs, E.d_work,
                            E.nwork, E.ef4, E.cell, E.off, E.vel, E.total_cap, E.acc, E.total_nodes, E.d_err);
            ECK(cudaMemsetAsync(E.d_counter, 0, sizeof(int), E.stream));
            ECK(cudaEventRecord(b, E.stream));
            ECK(ens_launch_solve(E, 1));
            ECK(cudaEventRecord(c, E.stream));
            E.nlaunch += 2;
            E.steps++;
            ECK(cudaGetLastError());
            ECK(cudaEventSynchronize(c));
            float ms = 0;
            ECK(cudaEventElapsedTime(&ms, b, c));
            if (ms < best_solve) {
                best_solve = ms;
                bs = E.solve_threads;
                bcl = E.cluster;
            }
        }
    E.solve_threads = bs;
    E.cluster = bcl;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaEventDestroy(c);
    ens_drop_graph(E);
    if (chunk) *chunk = E.chunk;
    if (push_threads) *push_threads = E.push_threads;
    if (solve_threads) *solve_threads = E.solve_threads;
    if (push_ms) *push_ms = best_push;
    if (solve_ms) *solve_ms = best_solve;
    return ens_take_errors(E);
}

extern "C" int espic_ensemble_steps_taken(espic_ensemble *h, int64_t *steps) {
    ENSEMBLE(h);
    if (steps) *steps = E.steps;
    return ESPIC_OK;
}
