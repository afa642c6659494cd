/*
 * k_pcg.cu -- matrix-free Newton / Jacobi-PCG solve of the Boltzmann-electron
 * Poisson problem of ch3/ver2 (PotentialSolver::solveNRPCG,
 * ch3/ver2/PotentialSolver.cpp:225-331), in one cooperative launch.
 *
 * The discrete problem is the one whose fixed point solveGS
 * (ch3/ver2/PotentialSolver.cpp:334-430) converges to.  Unknowns are the
 * interior nodes with object_id == 0.  With c = 1/dh^2 per axis,
 *   F_u = sum_{nb unknown or Dirichlet} c (phi_u - phi_nb)
 *         + (qe n0/eps0) exp((phi_u - phi0)/Te) - rho_u/eps0
 * (a Neumann boundary neighbour of an interior node always copies that node,
 * so it contributes nothing), and J = L + diag((qe n0/(eps0 Te)) e^...) is
 * symmetric positive definite.  The reference's own matrix has first-order,
 * non-symmetric Neumann rows on which CG breaks down.
 *
 * Newton residual F, the update of phi and the stopping test RMS(y) < nr_tol
 * (the reference's vec::norm, ch3/ver2/PotentialSolver.cpp:114-121) are
 * float64.  The inner PCG runs in T = double or float: with float it is the
 * inner solve of an iterative refinement whose outer residual is float64.
 * Dot products are reduced per block and summed by every block in block
 * order, so every block takes the same branch.  The inner PCG stops when
 * |r| <= pcg_tol |F|, or earlier once the RMS of the preconditioned residual
 * z = M r (an estimate of the error left in the Newton update y) is below
 * nr_tol / 2 (nr_tol / 10 in linear mode): the Newton test RMS(y) < nr_tol
 * cannot then depend on more inner accuracy, and the last Newton step stops
 * needing a full solve; when the first V-cycle's z is already that small,
 * z itself is the update.
 *
 * Preconditioner: an aggregation multigrid V-cycle.  Level l+1 groups the
 * level-l unknowns in 2x2x2 blocks of the structured index space; its
 * operator is the Galerkin product P^T A_l P with piecewise-constant P
 * (a 7-point stencil again, with per-node weights), built once per geometry
 * by a deterministic gather.  Smoothing is red-black Gauss-Seidel (red then
 * black before the coarse correction, black then red after), restriction is
 * P^T, prolongation P scaled by a constant.  The first level with at most
 * World::mg_dense_max nodes (default 1024) is the coarsest and is solved by
 * its dense inverse (computed once per geometry by k_gauss_jordan), every
 * level above it on the whole grid.  With mg_dense_max 0 (or a singular
 * coarse operator) the coarsest level gets symmetric sweeps instead and
 * levels with fewer than World::mg_block_nodes nodes (default 4096) run on
 * block 0 alone between two grid barriers.  Either way the preconditioner
 * is symmetric, as CG requires.  Without levels, it is Jacobi.
 */
#include <cooperative_groups.h>

#include "dfloat.h"
#include "espic_world.h"

namespace cg = cooperative_groups;

namespace espic {

#define PCG_EPS_0 8.85418782e-12
#define PCG_QE 1.602176565e-19

enum : uint16_t { SELF = 1u << 12, BLACK = 1u << 13 };

/* neighbour m: 0 -x, 1 +x, 2 -y, 3 +y, 4 -z, 5 +z.  bit m: unknown; bit 6+m:
 * Dirichlet; SELF: the node is an unknown. */
__global__ void k_pcg_codes(Geo g, const int32_t *__restrict__ obj, uint16_t *code) {
    int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t nn = (int64_t)g.ni * g.nj * g.nk;
    if (u >= nn) return;
    int i = (int)(u % g.ni), j = (int)((u / g.ni) % g.nj), k = (int)(u / ((int64_t)g.ni * g.nj));
    uint16_t c = 0;
    bool interior = i > 0 && j > 0 && k > 0 && i < g.ni - 1 && j < g.nj - 1 && k < g.nk - 1;
    if (interior && obj[u] == 0) {
        c |= SELF;
        if ((i + j + k) & 1) c |= BLACK;
        int64_t sy = g.ni, sz = (int64_t)g.ni * g.nj;
        int64_t nb[6] = {u - 1, u + 1, u - sy, u + sy, u - sz, u + sz};
        int ii[6] = {i - 1, i + 1, i, i, i, i}, jj[6] = {j, j, j - 1, j + 1, j, j},
            kk[6] = {k, k, k, k, k - 1, k + 1};
        for (int m = 0; m < 6; m++) {
            if (obj[nb[m]] > 0) {
                c |= (uint16_t)(1u << (6 + m));
            } else {
                bool in = ii[m] > 0 && jj[m] > 0 && kk[m] > 0 && ii[m] < g.ni - 1 && jj[m] < g.nj - 1 &&
                          kk[m] < g.nk - 1;
                if (in) c |= (uint16_t)(1u << m);
            }
        }
    }
    code[u] = c;
}

/* Grid-wide sums of NV per-thread values of type T: block partials, one grid
 * barrier, then every block sums the partials with its first warp (lane l
 * takes partials l, l+32, ... in order; a fixed shuffle tree combines the
 * lanes).  Every block computes bit-identical totals, so all blocks take the
 * same branches.  Floats are added in float within a warp; the warps' sums,
 * the blocks' partials and the total are float64.  Doubles go through shared
 * memory, 128 threads per value adding blockDim / 128 of them first: a
 * shuffle tree would issue five full-warp float64 additions per warp and
 * value, half of a pass over a small grid.  The partials of up to 160 blocks
 * are loaded at once (loaded in a rolled loop, they cost two L2 latencies
 * per value). */
template <int NV, typename T>
__device__ __forceinline__ void grid_sum(cg::grid_group &grid, const T (&v)[NV], double (&out)[NV], double *partials,
                                         int &round) {
    __shared__ double shw[NV][32];
    __shared__ double tot[NV];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int nw = (int)(blockDim.x >> 5); /* entries of shw per value */
    if (sizeof(T) == sizeof(double)) {
        __shared__ double all[NV][1024];
#pragma unroll
        for (int q = 0; q < NV; q++) all[q][threadIdx.x] = (double)v[q];
        __syncthreads();
        if ((int)threadIdx.x < 128 * NV) {
            const int q = threadIdx.x >> 7, t = threadIdx.x & 127;
            double x = all[q][t];
            for (int b = t + 128; b < (int)blockDim.x; b += 128) x += all[q][b];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if (lane == 0) shw[q][wid & 3] = x;
        }
        nw = 4;
    } else {
#pragma unroll
        for (int q = 0; q < NV; q++) {
            T x = v[q];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) shw[q][wid] = (double)x;
        }
    }
    __syncthreads();
    double *slot = partials + (size_t)(round & 1) * gridDim.x * NV;
    if (wid == 0) {
        double x[NV];
#pragma unroll
        for (int q = 0; q < NV; q++) x[q] = lane < nw ? shw[q][lane] : 0.0;
#pragma unroll
        for (int o = sizeof(T) == sizeof(double) ? 2 : 16; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < NV; q++) x[q] += __shfl_xor_sync(0xffffffffu, x[q], o);
        if (lane == 0)
#pragma unroll
            for (int q = 0; q < NV; q++) slot[(size_t)blockIdx.x * NV + q] = x[q];
    }
    round++;
    grid.sync();
    if (wid == 0) {
        double x[NV];
#pragma unroll
        for (int q = 0; q < NV; q++) x[q] = 0;
        /* once for up to 160 blocks: unrolled by the compiler, the passes past
         * the last block would add zeros in float64 */
#pragma unroll 1
        for (unsigned b0 = lane; b0 < gridDim.x; b0 += 160) {
            double t[5][NV];
#pragma unroll
            for (int i = 0; i < 5; i++)
#pragma unroll
                for (int q = 0; q < NV; q++)
                    t[i][q] = b0 + 32 * i < gridDim.x ? __ldcg(slot + (size_t)(b0 + 32 * i) * NV + q) : 0.0;
#pragma unroll
            for (int i = 0; i < 5; i++)
#pragma unroll
                for (int q = 0; q < NV; q++) x[q] += t[i][q];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < NV; q++) x[q] += __shfl_xor_sync(0xffffffffu, x[q], o);
        if (lane == 0)
#pragma unroll
            for (int q = 0; q < NV; q++) tot[q] = x[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; q++) out[q] = tot[q];
}

/* Whether the inner type takes the cheaper sweeps.  The float64 inner solve
 * is bound by the narrow float64 pipe, and its last bits reach phi far below
 * any tolerance, so it multiplies by stored reciprocal diagonals and leaves
 * out terms that cancel.  The float inner solve keeps the arithmetic of the
 * plain formulas (its last bits reach the particles' float E). */
template <typename T>
constexpr bool LIGHT = sizeof(T) == sizeof(double);

constexpr int MG_MAX = 12;
/* threads per block of the cooperative solve (one block per SM): 1024 for
 * large grids, whose passes live on loads in flight (256x256x512 float: 20
 * ms against 28 with 512 threads), 512 for small ones, whose passes are a
 * chain of latencies that the 64 registers of 1024 threads lengthen by
 * spills (33x29x65 float solve: 0.75 ms with 1024, 0.63 with 512; 64x64x128
 * float64: 7.5 and 6.8 ms a cold solve) */
constexpr int PCG_THREADS = 1024, PCG_THREADS_SMALL = 512;
constexpr int GJ_ROWS = 64;                /* rows of the dense inversion per block */
constexpr size_t GJ_SMEM_MAX = 200 * 1024; /* and the shared memory they may take */
constexpr size_t PCG_SMEM_MAX = 160 * 1024; /* shared memory for block 0's coarse levels */

template <typename T>
struct MgLevel {
    int nx, ny, nz;
    int merge; /* MERGE_PRE | MERGE_POST: half sweeps of the whole grid in one phase */
    int64_t n;
    T *diag, *w, *b, *e; /* w: 6 weights per node, [m][n] */
    T *f;                /* the level's final correction: its own array with MERGE_POST, else e */
    T *id;               /* 1 / diag, 0 where diag is 0 (an aggregate without unknowns) */
};

/* MERGE_PRE: the black half sweep before the restriction runs inside the
 * restriction (restrict_through); MERGE_POST: the two half sweeps after the
 * prolongation run as one (coarse_post).  Neighbouring work items then
 * relax the same black nodes again, which costs little where a level has
 * fewer nodes than the grid has threads, and saves a phase, that is a grid
 * barrier (1.29 us) and an L2 latency. */
enum { MERGE_PRE = 1, MERGE_POST = 2 };

template <typename T>
struct MgArgs {
    int fine_pre;    /* MERGE_PRE for the node grid */
    int nlev;        /* coarse levels (0: Jacobi preconditioner) */
    int grid_levels; /* coarse levels 1..grid_levels-1 run on the whole grid */
    int nu_coarse;   /* sweeps each way on the coarsest level */
    T scale;         /* coarse-correction scale */
    int smem_from;   /* block 0 keeps levels L[smem_from..] in shared memory (-1: none) */
    int dense_n;     /* nodes of the coarsest level when it is solved by its dense inverse */
    T *dense;        /* that inverse, row-major (null: smoothing sweeps on the coarsest level) */
    const int *dense_ok; /* 0 when the inversion met a vanishing pivot (a singular coarse operator,
                            e.g. without Dirichlet nodes): the coarsest level is smoothed instead */
    MgLevel<T> L[MG_MAX];
};

/* bytes of one level's arrays (diag or 1 / diag, 6 weights, b, e) in shared memory */
template <typename T>
__host__ __device__ inline size_t level_smem_bytes(int64_t n) {
    return ((size_t)n * sizeof(T) + 15) / 16 * 16 * 9;
}

/* everything the level-0 (node grid) operations need */
template <typename T>
struct Coef3 {
    T c[3];
};

template <typename T>
struct Fine {
    Geo g;
    const uint16_t *code;
    T ct[3];
    uint32_t nn;
    T *dg, *r, *z; /* dg: the Boltzmann part of the Jacobian diagonal (LIGHT: the whole of it) */
    T *id;         /* LIGHT: 1 / the diagonal on the unknowns, 0 elsewhere */
    uint32_t ncolour; /* entries of a colour's enumeration */
};

/* What the passes of a solve share, kept once per block in shared memory: the
 * passes are functions of their own (not inlined) that read it there, so
 * that each has the block's registers to itself.  Inlined into one kernel,
 * 1024 threads of 64 registers spilled in the node loops (256x256x512 float:
 * the black post-smoothing half took 262 us against 116 us for the same half
 * without the prolongation). */
template <typename T>
struct SolveShared {
    Fine<T> F;
    MgArgs<T> A; /* the levels in global memory */
    MgArgs<T> B; /* block 0's view of the levels it works alone: shared-memory copies of L[smem_from..] */
};

template <typename T>
__device__ __forceinline__ SolveShared<T> &shared_of() {
    __shared__ SolveShared<T> st;
    return st;
}

/* fills the shared state; block 0 also copies the diagonals (or their
 * reciprocals, what the sweeps read) and weights of the levels it works alone
 * into shared memory, once per launch */
template <typename T>
__device__ __forceinline__ void shared_init(const Fine<T> &F, const MgArgs<T> &A, unsigned char *base) {
    SolveShared<T> &st = shared_of<T>();
    const bool staged = A.smem_from >= 0 && A.nlev > 0 && blockIdx.x == 0;
    if (threadIdx.x == 0) {
        st.F = F;
        st.A = A;
        st.B = A;
        size_t off = 0;
        for (int i = A.smem_from; staged && i < A.nlev; i++) {
            const size_t a = ((size_t)A.L[i].n * sizeof(T) + 15) / 16 * 16;
            st.B.L[i].diag = st.B.L[i].id = (T *)(base + off); /* the one that the sweeps read */
            st.B.L[i].w = (T *)(base + off + a);
            st.B.L[i].b = (T *)(base + off + 7 * a);
            st.B.L[i].e = st.B.L[i].f = (T *)(base + off + 8 * a);
            off += 9 * a;
        }
    }
    __syncthreads();
    for (int i = A.smem_from; staged && i < A.nlev; i++) {
        const int64_t n = st.A.L[i].n;
        for (int64_t t = threadIdx.x; t < n; t += blockDim.x)
            st.B.L[i].diag[t] = LIGHT<T> ? st.A.L[i].id[t] : st.A.L[i].diag[t];
        for (int64_t t = threadIdx.x; t < 6 * n; t += blockDim.x) st.B.L[i].w[t] = st.A.L[i].w[t];
    }
    __syncthreads();
}

/* A thread's share of count work items: t, t + step, ... below end (grids
 * have at most 2^31 nodes). */
struct Span {
    uint32_t t, end, step;
};

/* The block alone (whole = false), or the whole grid: with more items than
 * threads a grid stride (all blocks near each other, so that the neighbour
 * planes stay in L2); with fewer, one contiguous range of whole warps per
 * block.  A grid stride over a small count leaves it to the first few blocks
 * (a colour of 31,000 nodes on 31 of 152 SMs, whose narrow float64 pipes
 * then work alone); even ranges use every SM.  Up to one item per thread,
 * both give a warp the same 32 items, so the float warp sums of the dot
 * products do not depend on the rule. */
__device__ __forceinline__ Span span(bool whole, uint32_t count) {
    if (!whole) return {threadIdx.x, count, blockDim.x};
    const uint32_t all = gridDim.x * blockDim.x;
    if (count > all) return {blockIdx.x * blockDim.x + threadIdx.x, count, all};
    const uint32_t per = ((count + gridDim.x - 1) / gridDim.x + 31u) & ~31u;
    const uint32_t t0 = blockIdx.x * per;
    return {t0 + threadIdx.x, t0 + per < count ? t0 + per : count, blockDim.x};
}

/* Full Jacobian diagonal of an unknown: its Boltzmann part plus c per
 * unknown or Dirichlet neighbour. */
template <typename T>
__device__ __forceinline__ T full_diag(uint16_t cc, T dB, const T ct[3]) {
    T d = dB;
#pragma unroll
    for (int m = 0; m < 6; m++) d += (cc & ((1u << m) | (1u << (6 + m)))) ? ct[m >> 1] : (T)0;
    return d;
}

/* J x at an unknown in difference form, dB x_u + sum_unknown c (x_u - x_nb)
 * + sum_Dirichlet c x_u: no term is the difference of two large products,
 * so float keeps full relative accuracy on the smooth modes, where the
 * equivalent diag x_u - sum c x_nb loses most of its digits at fine spacing */
template <typename T>
__device__ __forceinline__ T jacobian_apply(uint16_t cc, T dB, const T ct[3], T xu, const T xn[6]) {
    T s = dB * xu;
#pragma unroll
    for (int m = 0; m < 6; m++)
        s += (cc & (1u << m)) ? ct[m >> 1] * (xu - xn[m]) : ((cc & (1u << (6 + m))) ? ct[m >> 1] * xu : (T)0);
    return s;
}

/* a node index clamped into the grid (loads of a boundary node's missing
 * neighbours, whose values are never used) */
__device__ __forceinline__ int64_t clamp_node(int64_t v, int64_t nn) { return v < 0 ? 0 : (v >= nn ? nn - 1 : v); }

/* Red-black Gauss-Seidel pieces.  A Gauss-Seidel update never reads the
 * node's own old value, which allows three fusions: the first red half
 * sweep from a zero guess is pointwise (e = b / diag) and is done by whoever
 * produces b; the prolongation of the coarse correction is applied on the
 * fly to the red neighbours read by the following black half sweep (the red
 * nodes are overwritten next anyway); and the dot products r.z and z.z are
 * accumulated by the last two half sweeps, which produce the final z. */
/* Keeps a loaded value where it was loaded: without it the compiler moves a
 * pass's loads behind the test of the code word, and each pass waits for two
 * memory latencies instead of one. */
__device__ __forceinline__ void pin(float &x) { asm volatile("" : "+f"(x)); }
__device__ __forceinline__ void pin(double &x) { asm volatile("" : "+d"(x)); }
template <typename T, int N>
__device__ __forceinline__ void pin(T (&x)[N]) {
#pragma unroll
    for (int m = 0; m < N; m++) pin(x[m]);
}

/* The six neighbours of u in order -x, +x, -y, +y, -z, +z */
template <typename T>
__device__ __forceinline__ void load_neighbours(const T *__restrict__ x, uint32_t u, int32_t sy, int32_t sz, T xn[6]) {
    const T *p = x + u;
    xn[0] = p[-1];
    xn[1] = p[1];
    xn[2] = p[-sy];
    xn[3] = p[sy];
    xn[4] = p[-sz];
    xn[5] = p[sz];
}

/* Red-black half sweep of a colour on the node grid, z = (r + sum c z_nb) /
 * diag; POST_* return the thread's sums of r*z and z*z over the nodes it
 * updated.  POST_BLACK reads the red neighbours with the coarse correction
 * added.  LIGHT: z is 0 on every node that is not an unknown, so a Dirichlet
 * or Neumann neighbour adds nothing without a look at the code, and id, the
 * reciprocal diagonal written once per Newton step, is 0 there, which marks
 * the nodes to skip (9 float64 instructions a node; ~25 with the diagonal
 * summed from the code word and a division).  Each thread takes PER entries
 * of the colour's enumeration per pass and issues every load of theirs before
 * any store (a padding entry reads the interior node (1,1,1) and stores
 * nothing).  Entry t is node i = 1 + 2 i2 + ((1+j+k+c)&1) of interior row
 * (j, k), with i2 = t mod hx. */
enum { PRE_BLACK = 0, POST_BLACK = 1, POST_RED = 2 };

template <typename T>
struct Dots {
    T rz, zz;
};

template <typename T, int MODE, int PER>
__device__ __forceinline__ Dots<T> fine_half() {
    const Fine<T> &F = shared_of<T>().F;
    constexpr int c = MODE == POST_RED ? 0 : 1;
    T rz = 0, zz = 0;
    T *__restrict__ z = F.z;
    const T *__restrict__ r = F.r;
    const T *__restrict__ dd = LIGHT<T> ? F.id : F.dg;
    const uint16_t *__restrict__ code = F.code;
    const T ct[3] = {F.ct[0], F.ct[1], F.ct[2]};
    const int32_t ni = F.g.ni, sz = F.g.ni * F.g.nj;
    const uint32_t hx = (uint32_t)((ni - 1) / 2), rj = (uint32_t)(F.g.nj - 2);
    const float inv_hx = 1.f / (float)hx, inv_rj = 1.f / (float)rj;
    const Span S = span(true, F.ncolour);
#pragma unroll 1
    for (uint32_t t = S.t; t < S.end; t += PER * S.step) {
        uint32_t u[PER];
        bool ok[PER];
        T ru[PER], du[PER], zn[PER][6], ea[PER], en[PER][3];
        uint16_t cc[PER];
        int par[PER];
#pragma unroll
        for (int q = 0; q < PER; q++) {
            const bool in = t + q * S.step < S.end;
            const uint32_t tt = in ? t + q * S.step : 0u;
            const uint32_t row = div_small(tt, hx, inv_hx);
            const uint32_t kk = div_small(row, rj, inv_rj);
            int j = 1 + (int)(row - kk * rj), k = 1 + (int)kk;
            int i = 1 + 2 * (int)(tt - row * hx) + ((1 + j + k + c) & 1);
            ok[q] = in && i <= ni - 2;
            if (!ok[q]) i = j = k = 1;
            u[q] = (uint32_t)k * (uint32_t)sz + (uint32_t)(j * ni + i);
            /* interior node: all six neighbours are in bounds, so their loads
             * do not wait for the code word, which only selects */
            ru[q] = r[u[q]];
            du[q] = dd[u[q]];
            if (MODE == POST_BLACK || !LIGHT<T>) cc[q] = code[u[q]];
            load_neighbours(z, u[q], ni, sz, zn[q]);
            if (MODE == POST_BLACK) {
                /* the coarse correction at the six neighbours: for each axis
                 * one neighbour shares the node's aggregate, the other is
                 * the next aggregate on the side of the node's parity */
                const MgLevel<T> &C = shared_of<T>().A.L[0];
                const int32_t cy = C.nx, cz = C.nx * C.ny;
                const T *e = C.f + ((k >> 1) * cz + (j >> 1) * cy + (i >> 1));
                par[q] = (i & 1) | ((j & 1) << 1) | ((k & 1) << 2);
                ea[q] = e[0];
                en[q][0] = e[(i & 1) ? 1 : -1];
                en[q][1] = e[(j & 1) ? cy : -cy];
                en[q][2] = e[(k & 1) ? cz : -cz];
            }
        }
#pragma unroll
        for (int q = 0; q < PER; q++) {
            pin(ru[q]);
            pin(du[q]);
            pin(zn[q]);
            if (MODE == POST_BLACK) {
                pin(ea[q]);
                pin(en[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < PER; q++) {
            if (MODE == POST_BLACK) {
                const T scale = shared_of<T>().A.scale;
#pragma unroll
                for (int m = 0; m < 6; m++) {
                    /* the neighbour inside the aggregate? */
                    const bool own = (bool)(par[q] & (1 << (m >> 1))) != (bool)(m & 1);
                    const T cor = scale * (own ? ea[q] : en[q][m >> 1]);
                    if (LIGHT<T>)
                        zn[q][m] += (cc[q] & (1u << m)) ? cor : (T)0;
                    else
                        zn[q][m] += cor;
                }
            }
            T zu, s = ru[q];
            if (LIGHT<T>) {
                if (!ok[q] || du[q] == (T)0) continue;
#pragma unroll
                for (int a = 0; a < 3; a++) s += ct[a] * (zn[q][2 * a] + zn[q][2 * a + 1]);
                zu = s * du[q];
            } else {
                if (!ok[q] || !(cc[q] & SELF)) continue;
#pragma unroll
                for (int m = 0; m < 6; m++) s += (cc[q] & (1u << m)) ? ct[m >> 1] * zn[q][m] : (T)0;
                zu = s / full_diag(cc[q], du[q], ct);
            }
            z[u[q]] = zu;
            if (MODE != PRE_BLACK) {
                rz += ru[q] * zu;
                zz += zu * zu;
            }
        }
    }
    return {rz, zz};
}

/* A node of a coarse level: all loads first (a missing neighbour reads a
 * clamped node; its zero weight deselects it), then its relaxation, (b + sum
 * w e_nb) / diag.  POST reads the neighbours with the next level's correction
 * added (per axis one neighbour shares the node's aggregate, the other is in
 * the next one). */
template <typename T, bool POST>
struct CoarseNode {
    T d, s, wm[6], en[6];
    __device__ __forceinline__ void load_self(const MgLevel<T> &L, int32_t I) {
        d = LIGHT<T> ? L.id[I] : L.diag[I];
        s = L.b[I];
#pragma unroll
        for (int m = 0; m < 6; m++) wm[m] = L.w[m * L.n + I];
    }
    __device__ __forceinline__ void load(const MgArgs<T> &A, int l, int i, int j, int k) {
        const MgLevel<T> &L = A.L[l];
        const int32_t offs[6] = {-1, 1, -L.nx, L.nx, -L.nx * L.ny, L.nx * L.ny};
        const int32_t I = (k * L.ny + j) * L.nx + i;
        load_self(L, I);
#pragma unroll
        for (int m = 0; m < 6; m++) {
            int32_t nb = I + offs[m];
            nb = nb < 0 ? 0 : (nb >= (int32_t)L.n ? (int32_t)L.n - 1 : nb);
            en[m] = L.e[nb];
        }
        if (POST) {
            const MgLevel<T> &C = A.L[l + 1];
            const T scale = A.scale;
            const int g = ((k >> 1) * C.ny + (j >> 1)) * C.nx + (i >> 1);
            /* the next aggregate along each axis; a neighbour off the level
             * has weight 0 and may read the node's own */
            const int ax = (i & 1) ? (i + 1 < L.nx ? g + 1 : g) : (i > 0 ? g - 1 : g);
            const int ay = (j & 1) ? (j + 1 < L.ny ? g + C.nx : g) : (j > 0 ? g - C.nx : g);
            const int az = (k & 1) ? (k + 1 < L.nz ? g + C.nx * C.ny : g) : (k > 0 ? g - C.nx * C.ny : g);
            const T ea = C.f[g];
            const T ex[3] = {C.f[ax], C.f[ay], C.f[az]};
            const bool odd[3] = {(bool)(i & 1), (bool)(j & 1), (bool)(k & 1)};
#pragma unroll
            for (int m = 0; m < 6; m++) en[m] += scale * (odd[m >> 1] != (bool)(m & 1) ? ea : ex[m >> 1]);
        }
        pin(s);
        pin(wm);
        pin(en);
    }
    __device__ __forceinline__ T relax() const {
        T t = s;
#pragma unroll
        for (int m = 0; m < 6; m++) t += (wm[m] != (T)0) ? wm[m] * en[m] : (T)0;
        return LIGHT<T> ? t * d : t / d;
    }
};

/* entry t of the x pairs of a level's rows (hx of them a row) */
__device__ __forceinline__ void pair_coords(uint32_t t, uint32_t hx, uint32_t ny, float inv_hx, float inv_ny, int &i2,
                                            int &j, int &k) {
    const uint32_t rr = div_small(t, hx, inv_hx);
    const uint32_t kk = div_small(rr, ny, inv_ny);
    i2 = (int)(t - rr * hx);
    j = (int)(rr - kk * ny);
    k = (int)kk;
}

/* one half sweep of colour c on level l (0: the first coarse one), by the
 * grid or by block 0 on its own view */
template <typename T, bool POST>
__device__ __forceinline__ void coarse_half(int l, int c, bool whole) {
    const MgArgs<T> &A = whole ? shared_of<T>().A : shared_of<T>().B;
    const MgLevel<T> &L = A.L[l];
    const int hx = (L.nx + 1) / 2;
    const float inv_hx = 1.f / (float)hx, inv_ny = 1.f / (float)L.ny;
    const Span S = span(whole, (uint32_t)(hx * L.ny * L.nz));
#pragma unroll 1
    for (uint32_t t = S.t; t < S.end; t += S.step) {
        int i2, j, k;
        pair_coords(t, (uint32_t)hx, (uint32_t)L.ny, inv_hx, inv_ny, i2, j, k);
        const int i = 2 * i2 + ((j + k + c) & 1);
        if (i >= L.nx) continue;
        CoarseNode<T, POST> x;
        x.load(A, l, i, j, k);
        if (x.d == (T)0) continue;
        L.e[(k * L.ny + j) * L.nx + i] = x.relax();
    }
}

/* Both half sweeps after the prolongation, black then red, by the whole grid
 * (MERGE_POST).  Eight lanes take an x pair of nodes: six relax the black
 * neighbours of its red node, which they hand to the first, and one of them
 * is the pair's black node.  The results go to f, since other lanes still
 * read the red values of e. */
template <typename T>
__device__ __forceinline__ void coarse_post(int l) {
    const MgArgs<T> &A = shared_of<T>().A;
    const MgLevel<T> &L = A.L[l];
    const uint32_t hx = (uint32_t)(L.nx + 1) / 2;
    const float inv_hx = 1.f / (float)hx, inv_ny = 1.f / (float)L.ny;
    const uint32_t total = 8 * hx * (uint32_t)(L.ny * L.nz);
    const int m0 = (int)(threadIdx.x & 7);
    const int step = (m0 & 1) ? 1 : -1;
    const Span S = span(true, (total + 31u) & ~31u);
#pragma unroll 1
    for (uint32_t t = S.t; t < S.end; t += S.step) {
        const bool valid = t < total;
        int i2, j, k;
        pair_coords(valid ? t >> 3 : 0u, hx, (uint32_t)L.ny, inv_hx, inv_ny, i2, j, k);
        const int odd = (j + k) & 1;
        const int i = 2 * i2 + odd; /* the red node */
        const int bi = i + (m0 < 2 ? step : 0), bj = j + (m0 == 2 || m0 == 3 ? step : 0),
                  bk = k + (m0 == 4 || m0 == 5 ? step : 0);
        const bool in = valid && m0 < 6 && bi >= 0 && bj >= 0 && bk >= 0 && bi < L.nx && bj < L.ny && bk < L.nz;
        const bool red = valid && m0 == 0 && i < L.nx;
        CoarseNode<T, true> x;
        CoarseNode<T, false> y;
        const int32_t I = red ? (k * L.ny + j) * L.nx + i : 0;
        y.load_self(L, I);
        x.load(A, l, in ? bi : 0, in ? bj : 0, in ? bk : 0);
        const bool on = in && x.d != (T)0;
        const T v = on ? x.relax() : (T)0;
        if (on && m0 == 1 - odd) L.f[(bk * L.ny + bj) * L.nx + bi] = v;
#pragma unroll
        for (int m = 0; m < 6; m++) y.en[m] = __shfl_sync(0xffffffffu, v, m, 8);
        if (red && y.d != (T)0) L.f[I] = y.relax();
    }
}

/* The red children of a coarse node (its 2x2x2 block), in the order in which
 * their residuals are summed: offsets dx | dy<<1 | dz<<2 with dx+dy+dz even
 * (black residuals are zero after the black half sweep).  LIGHT: a red
 * child's residual r - J z is sum c z over its black neighbours, because its
 * own value is r / diag from the first red half sweep: neither r nor the
 * diagonal is read. */
__device__ __forceinline__ int red_child(int q) { return q == 0 ? 0 : (q == 1 ? 3 : (q == 2 ? 5 : 6)); }

/* Coordinates of coarse node I. */
template <typename T>
__device__ __forceinline__ void coarse_coords(const MgLevel<T> &C, uint32_t I, float inv_nx, float inv_ny, int &ci,
                                              int &cj, int &ck) {
    const uint32_t cr = div_small(I, (uint32_t)C.nx, inv_nx);
    const uint32_t ckk = div_small(cr, (uint32_t)C.ny, inv_ny);
    ci = (int)(I - cr * (uint32_t)C.nx);
    cj = (int)(cr - ckk * (uint32_t)C.ny);
    ck = (int)ckk;
}

/* The sum of four lanes' residuals (lanes 4g..4g+3, in lane order) into
 * b of the coarse node, and the fused first red half sweep (e = b / diag; d:
 * the node's diagonal, or LIGHT its reciprocal).  Every lane of the warp
 * calls it. */
template <typename T>
__device__ __forceinline__ void restrict_store(const MgLevel<T> &C, bool valid, uint32_t I, int ci, int cj, int ck,
                                               T res, T d) {
    const T r1 = __shfl_down_sync(0xffffffffu, res, 1);
    const T r2 = __shfl_down_sync(0xffffffffu, res, 2);
    const T r3 = __shfl_down_sync(0xffffffffu, res, 3);
    if (!valid || (threadIdx.x & 3)) return;
    T sum = 0;
    sum += res;
    sum += r1;
    sum += r2;
    sum += r3;
    C.b[I] = sum;
    if (((ci + cj + ck) & 1) == 0 && d != (T)0) C.e[I] = LIGHT<T> ? sum * d : sum / d;
}

/* A red child of the node grid: what its residual needs, loaded at once, and
 * the residual (0 for a node that is not an unknown, or not interior). */
template <typename T>
struct FineChild {
    T id, r, dg, z, zn[6];
    uint16_t cc;
    __device__ __forceinline__ void load_self(const Fine<T> &F, uint32_t u, bool in) {
        if (LIGHT<T>) {
            id = in ? F.id[u] : (T)0;
        } else {
            cc = in ? F.code[u] : (uint16_t)0;
            r = F.r[u];
            dg = F.dg[u];
            z = F.z[u];
        }
    }
    __device__ __forceinline__ void load(const Fine<T> &F, int32_t sy, int32_t sz, uint32_t u, bool in) {
        load_self(F, u, in);
        load_neighbours<T>(F.z, u, sy, sz, zn);
    }
    __device__ __forceinline__ void hold() {
        if (LIGHT<T>) {
            pin(id);
        } else {
            pin(r);
            pin(dg);
            pin(z);
        }
        pin(zn);
    }
    __device__ __forceinline__ T residual(const Fine<T> &F) const {
        if (LIGHT<T>) {
            T res = 0;
#pragma unroll
            for (int a = 0; a < 3; a++) res += F.ct[a] * (zn[2 * a] + zn[2 * a + 1]);
            return id != (T)0 ? res : (T)0;
        }
        return (cc & SELF) ? r - jacobian_apply(cc, dg, F.ct, z, zn) : (T)0;
    }
};

/* interior node of the grid (i, j, k), or the interior node (1,1,1) */
__device__ __forceinline__ uint32_t interior_or_safe(const Geo &g, int i, int j, int k, bool &in) {
    in = in && i > 0 && j > 0 && k > 0 && i < g.ni - 1 && j < g.nj - 1 && k < g.nk - 1;
    const uint32_t ii = in ? (uint32_t)i : 1u, jj = in ? (uint32_t)j : 1u, kk = in ? (uint32_t)k : 1u;
    return (kk * (uint32_t)g.nj + jj) * (uint32_t)g.ni + ii;
}

/* b of level 1 = sum of the node-grid children's residuals (r - J z).  When
 * the level has fewer nodes than the grid has threads (latency-bound),
 * four consecutive threads take the four red children of a coarse node,
 * each issuing all its loads at once (neighbour indices clamped into the
 * grid; a child that is not an unknown contributes zero); otherwise
 * (bandwidth-bound) a thread takes a coarse node and its four children, so
 * that a warp's loads of one child cover consecutive nodes of a row. */
template <typename T>
__device__ __forceinline__ void restrict_fine() {
    const Fine<T> &F = shared_of<T>().F;
    const MgLevel<T> &C = shared_of<T>().A.L[0];
    const Geo g = F.g;
    const int32_t sy = g.ni, sz = g.ni * g.nj;
    const float inv_nx = 1.f / (float)C.nx, inv_ny = 1.f / (float)C.ny;
    const T *__restrict__ diag = LIGHT<T> ? C.id : C.diag;
    const uint32_t n = (uint32_t)C.n;
    if (n > gridDim.x * blockDim.x) {
        const Span S = span(true, n);
#pragma unroll 1
        for (uint32_t I = S.t; I < S.end; I += S.step) {
            int ci, cj, ck;
            coarse_coords(C, I, inv_nx, inv_ny, ci, cj, ck);
            const T cd = diag[I];
            T sum = 0;
            /* all children's loads at once (256x256x512 float: 130 us, in two
             * pairs 161) */
            constexpr int PER = LIGHT<T> ? 2 : 4;
#pragma unroll
            for (int q0 = 0; q0 < 4; q0 += PER) {
                FineChild<T> ch[PER];
#pragma unroll
                for (int q = 0; q < PER; q++) {
                    const int d = red_child(q0 + q);
                    bool in = true;
                    const uint32_t u =
                        interior_or_safe(g, 2 * ci + (d & 1), 2 * cj + ((d >> 1) & 1), 2 * ck + (d >> 2), in);
                    ch[q].load(F, sy, sz, u, in);
                }
#pragma unroll
                for (int q = 0; q < PER; q++) ch[q].hold();
#pragma unroll
                for (int q = 0; q < PER; q++) sum += ch[q].residual(F);
            }
            C.b[I] = sum;
            if (((ci + cj + ck) & 1) == 0 && cd != (T)0) C.e[I] = LIGHT<T> ? sum * cd : sum / cd;
        }
        return;
    }
    const uint32_t total = 4 * n;
    const Span S = span(true, (total + 31u) & ~31u);
#pragma unroll 1
    for (uint32_t t = S.t; t < S.end; t += S.step) {
        const bool valid = t < total;
        const uint32_t I = valid ? (t >> 2) : 0;
        int ci, cj, ck;
        coarse_coords(C, I, inv_nx, inv_ny, ci, cj, ck);
        const int d = red_child((int)(t & 3));
        bool in = valid;
        const uint32_t u = interior_or_safe(g, 2 * ci + (d & 1), 2 * cj + ((d >> 1) & 1), 2 * ck + (d >> 2), in);
        FineChild<T> ch;
        T cd = diag[I];
        ch.load(F, sy, sz, u, in);
        ch.hold();
        pin(cd);
        restrict_store(C, valid, I, ci, cj, ck, ch.residual(F), cd);
    }
}

/* b of level l+1 from level l, laid out like restrict_fine (an aggregate
 * without unknowns has no weights and contributes 0) */
template <typename T>
__device__ __forceinline__ T coarse_residual(T bu, T dd, T eu, const T (&wm)[6], const T (&en)[6]) {
    T res = LIGHT<T> ? (T)0 : bu - dd * eu;
#pragma unroll
    for (int m = 0; m < 6; m++) res += (wm[m] != (T)0) ? wm[m] * en[m] : (T)0;
    return res;
}

template <typename T>
__device__ __forceinline__ T coarse_child_residual(const MgLevel<T> &L, int i, int j, int k, bool in) {
    const int32_t offs[6] = {-1, 1, -L.nx, L.nx, -L.nx * L.ny, L.nx * L.ny};
    in = in && i < L.nx && j < L.ny && k < L.nz;
    const int32_t u = in ? (k * L.ny + j) * L.nx + i : 0;
    T wm[6], en[6];
    const T dd = LIGHT<T> ? (T)1 : L.diag[u], bu = LIGHT<T> ? (T)0 : L.b[u], eu = LIGHT<T> ? (T)0 : L.e[u];
#pragma unroll
    for (int m = 0; m < 6; m++) {
        int32_t nb = u + offs[m];
        nb = nb < 0 ? 0 : (nb >= (int32_t)L.n ? (int32_t)L.n - 1 : nb);
        wm[m] = L.w[m * L.n + u];
        en[m] = L.e[nb];
    }
    pin(wm);
    pin(en);
    if (!in || dd == (T)0) return (T)0;
    return coarse_residual(bu, dd, eu, wm, en);
}

template <typename T>
__device__ __forceinline__ void restrict_coarse(int l, bool whole) {
    const MgArgs<T> &A = whole ? shared_of<T>().A : shared_of<T>().B;
    const MgLevel<T> &L = A.L[l], &C = A.L[l + 1];
    const float inv_nx = 1.f / (float)C.nx, inv_ny = 1.f / (float)C.ny;
    const T *__restrict__ diag = LIGHT<T> ? C.id : C.diag;
    const uint32_t n = (uint32_t)C.n;
    if (n > (whole ? gridDim.x : 1u) * blockDim.x) {
        const Span S = span(whole, n);
#pragma unroll 1
        for (uint32_t I = S.t; I < S.end; I += S.step) {
            int ci, cj, ck;
            coarse_coords(C, I, inv_nx, inv_ny, ci, cj, ck);
            const T cd = diag[I];
            T sum = 0;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int d = red_child(q);
                sum += coarse_child_residual(L, 2 * ci + (d & 1), 2 * cj + ((d >> 1) & 1), 2 * ck + (d >> 2), true);
            }
            C.b[I] = sum;
            if (((ci + cj + ck) & 1) == 0 && cd != (T)0) C.e[I] = LIGHT<T> ? sum * cd : sum / cd;
        }
        return;
    }
    const uint32_t total = 4 * n;
    const Span S = span(whole, (total + 31u) & ~31u);
#pragma unroll 1
    for (uint32_t t = S.t; t < S.end; t += S.step) {
        const bool valid = t < total;
        const uint32_t I = valid ? (t >> 2) : 0;
        int ci, cj, ck;
        coarse_coords(C, I, inv_nx, inv_ny, ci, cj, ck);
        const int d = red_child((int)(t & 3));
        T cd = diag[I];
        pin(cd);
        const T res =
            coarse_child_residual(L, 2 * ci + (d & 1), 2 * cj + ((d >> 1) & 1), 2 * ck + (d >> 2), valid);
        restrict_store(C, valid, I, ci, cj, ck, res, cd);
    }
}

/* The black half sweep and the restriction in one phase (MERGE_PRE), by the
 * whole grid: sixteen lanes take a coarse node and relax the sixteen black
 * nodes around its four red children (four in its 2x2x2 block, twelve just
 * outside), which the first four lanes then read as their red child's
 * neighbours.  Nothing else reads the black values of this half sweep (the
 * black half after the prolongation overwrites them), so they are not
 * stored. */
struct Block16 {
    int dx, dy, dz; /* this lane's black node, -1..2 from the block's corner */
    int red;        /* red child of lanes 0..3 (bits dx | dy << 1 | dz << 2) */
    int src[6];     /* lanes of that child's neighbours */
};

__device__ __forceinline__ Block16 block16() {
    Block16 B;
    const int lane = (int)(threadIdx.x & 15);
    if (lane < 4) {
        const int mask = lane == 3 ? 7 : 1 << lane;
        B.dx = mask & 1;
        B.dy = (mask >> 1) & 1;
        B.dz = mask >> 2;
    } else {
        const int mask = red_child((lane - 4) / 3), a = (lane - 4) % 3;
        B.dx = mask & 1;
        B.dy = (mask >> 1) & 1;
        B.dz = mask >> 2;
        if (a == 0) B.dx = B.dx ? 2 : -1;
        if (a == 1) B.dy = B.dy ? 2 : -1;
        if (a == 2) B.dz = B.dz ? 2 : -1;
    }
    const int q = lane & 3;
    B.red = red_child(q);
#pragma unroll
    for (int m = 0; m < 6; m++) {
        const int a = m >> 1, bit = (B.red >> a) & 1, inner = B.red ^ (1 << a);
        B.src[m] = (m & 1) != bit ? (inner == 7 ? 3 : inner >> 1) : 4 + 3 * q + a;
    }
    return B;
}

template <typename T>
__device__ __forceinline__ void restrict_through(int l) {
    const MgArgs<T> &A = shared_of<T>().A;
    const MgLevel<T> &L = A.L[l], &C = A.L[l + 1];
    const float inv_nx = 1.f / (float)C.nx, inv_ny = 1.f / (float)C.ny;
    const T *__restrict__ diag = LIGHT<T> ? C.id : C.diag;
    const Block16 B = block16();
    const uint32_t total = 16 * (uint32_t)C.n;
    const Span S = span(true, (total + 31u) & ~31u);
#pragma unroll 1
    for (uint32_t t = S.t; t < S.end; t += S.step) {
        const bool valid = t < total;
        const uint32_t I = valid ? (t >> 4) : 0;
        int ci, cj, ck;
        coarse_coords(C, I, inv_nx, inv_ny, ci, cj, ck);
        const int i = 2 * ci + B.dx, j = 2 * cj + B.dy, k = 2 * ck + B.dz;
        const bool in = i >= 0 && j >= 0 && k >= 0 && i < L.nx && j < L.ny && k < L.nz;
        const int ri = 2 * ci + (B.red & 1), rj = 2 * cj + ((B.red >> 1) & 1), rk = 2 * ck + (B.red >> 2);
        const bool rin = (threadIdx.x & 12) == 0 && ri < L.nx && rj < L.ny && rk < L.nz;
        const int32_t u = rin ? (rk * L.ny + rj) * L.nx + ri : 0;
        CoarseNode<T, false> x;
        T wm[6], nb[6], cd = diag[I];
        const T dd = LIGHT<T> ? (T)1 : L.diag[u], bu = LIGHT<T> ? (T)0 : L.b[u], eu = LIGHT<T> ? (T)0 : L.e[u];
#pragma unroll
        for (int m = 0; m < 6; m++) wm[m] = L.w[m * L.n + u];
        x.load(A, l, in ? i : 0, in ? j : 0, in ? k : 0);
        pin(wm);
        pin(cd);
        const T v = in && x.d != (T)0 ? x.relax() : (T)0;
#pragma unroll
        for (int m = 0; m < 6; m++) nb[m] = __shfl_sync(0xffffffffu, v, B.src[m], 16);
        const T res = rin && dd != (T)0 ? coarse_residual(bu, dd, eu, wm, nb) : (T)0;
        restrict_store(C, valid && (threadIdx.x & 15) == 0, I, ci, cj, ck, res, cd);
    }
}

template <typename T>
__device__ __forceinline__ void restrict_through_fine() {
    const Fine<T> &F = shared_of<T>().F;
    const MgLevel<T> &C = shared_of<T>().A.L[0];
    const Geo g = F.g;
    const int32_t sy = g.ni, sz = g.ni * g.nj;
    const float inv_nx = 1.f / (float)C.nx, inv_ny = 1.f / (float)C.ny;
    const T *__restrict__ diag = LIGHT<T> ? C.id : C.diag;
    const T *__restrict__ dv = LIGHT<T> ? F.id : F.dg;
    const Block16 B = block16();
    const uint32_t total = 16 * (uint32_t)C.n;
    const Span S = span(true, (total + 31u) & ~31u);
#pragma unroll 1
    for (uint32_t t = S.t; t < S.end; t += S.step) {
        const bool valid = t < total;
        const uint32_t I = valid ? (t >> 4) : 0;
        int ci, cj, ck;
        coarse_coords(C, I, inv_nx, inv_ny, ci, cj, ck);
        bool in = true, rin = (threadIdx.x & 12) == 0;
        const uint32_t u = interior_or_safe(g, 2 * ci + B.dx, 2 * cj + B.dy, 2 * ck + B.dz, in);
        const uint32_t ur = interior_or_safe(g, 2 * ci + (B.red & 1), 2 * cj + ((B.red >> 1) & 1), 2 * ck + (B.red >> 2),
                                             rin);
        FineChild<T> ch;
        T cd = diag[I], ru = F.r[u], du = dv[u], zn[6];
        const uint16_t cc = LIGHT<T> ? (uint16_t)0 : F.code[u];
        load_neighbours(F.z, u, sy, sz, zn);
        ch.load_self(F, ur, rin);
        pin(cd);
        pin(ru);
        pin(du);
        pin(zn);
        T v = 0, s = ru;
        if (LIGHT<T>) {
#pragma unroll
            for (int a = 0; a < 3; a++) s += F.ct[a] * (zn[2 * a] + zn[2 * a + 1]);
            if (in) v = s * du;
        } else if (in && (cc & SELF)) {
#pragma unroll
            for (int m = 0; m < 6; m++) s += (cc & (1u << m)) ? F.ct[m >> 1] * zn[m] : (T)0;
            v = s / full_diag(cc, du, F.ct);
        }
#pragma unroll
        for (int m = 0; m < 6; m++) ch.zn[m] = __shfl_sync(0xffffffffu, v, B.src[m], 16);
        restrict_store(C, valid && (threadIdx.x & 15) == 0, I, ci, cj, ck, ch.residual(F), cd);
    }
}

/* e = A^-1 b on the coarsest level by its dense inverse, on the whole grid:
 * block b takes a contiguous range of rows, eight at a time, four warps per
 * row, each warp a quarter of the columns (lanes in a fixed order, a fixed
 * shuffle tree); the four quarter sums are added in order.  Every thread of
 * every block calls it (blocks of 128 threads or a multiple). */
template <typename T>
__device__ __forceinline__ void dense_apply() {
    __shared__ T part[32];
    const MgLevel<T> L = shared_of<T>().A.L[shared_of<T>().A.nlev - 1];
    const T *__restrict__ Ainv = shared_of<T>().A.dense;
    const int n = shared_of<T>().A.dense_n;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr int WPR = 4; /* warps per row */
    const int RPP = (int)(blockDim.x >> 5) / WPR; /* rows per pass */
    const int64_t rpb = ((int64_t)n + gridDim.x - 1) / gridDim.x;
    const int64_t r0 = (int64_t)blockIdx.x * rpb;
    const int64_t r1 = r0 + rpb < n ? r0 + rpb : n;
    for (int64_t rb = r0; rb < r1; rb += RPP) {
        const int64_t r = rb + wid / WPR;
        const int q = wid % WPR;
        T acc = 0;
        if (r < r1) {
            const int64_t c0 = (int64_t)q * n / WPR, c1 = (int64_t)(q + 1) * n / WPR;
            const T *row = Ainv + r * n;
#pragma unroll 8
            for (int64_t j = c0 + lane; j < c1; j += 32) acc += row[j] * L.b[j];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) part[wid] = acc;
        __syncthreads();
        if (threadIdx.x < RPP && rb + threadIdx.x < r1) {
            T sum = 0;
#pragma unroll
            for (int k = 0; k < WPR; k++) sum += part[threadIdx.x * WPR + k];
            L.e[rb + threadIdx.x] = sum;
        }
        __syncthreads();
    }
}

/* The passes as calls (CALL) or inlined.  On large grids with 1024 threads the
 * call gives a pass the 64 registers to itself (see SolveShared); with 512
 * nothing spills, and inlining is quicker. */
template <typename T, int MODE>
__device__ __noinline__ Dots<T> fine_half_call() {
    return fine_half<T, MODE, 2>();
}
template <typename T, bool POST>
__device__ __noinline__ void coarse_half_call(int l, int c, bool whole) {
    coarse_half<T, POST>(l, c, whole);
}
template <typename T>
__device__ __noinline__ void restrict_fine_call() {
    restrict_fine<T>();
}
template <typename T>
__device__ __noinline__ void restrict_coarse_call(int l, bool whole) {
    restrict_coarse<T>(l, whole);
}
template <typename T>
__device__ __noinline__ void dense_apply_call() {
    dense_apply<T>();
}
template <typename T>
__device__ __noinline__ void coarse_post_call(int l) {
    coarse_post<T>(l);
}
template <typename T>
__device__ __noinline__ void restrict_through_call(int l) {
    restrict_through<T>(l);
}

template <typename T, bool CALL>
struct Pass {
    template <int MODE>
    static __device__ __forceinline__ Dots<T> fine() {
        return CALL ? fine_half_call<T, MODE>() : fine_half<T, MODE, 2>();
    }
    template <bool POST>
    static __device__ __forceinline__ void coarse(int l, int c, bool whole) {
        if (CALL)
            coarse_half_call<T, POST>(l, c, whole);
        else
            coarse_half<T, POST>(l, c, whole);
    }
    static __device__ __forceinline__ void restrict_to_first() {
        if (CALL)
            restrict_fine_call<T>();
        else
            restrict_fine<T>();
    }
    static __device__ __forceinline__ void restrict_from(int l, bool whole) {
        if (CALL)
            restrict_coarse_call<T>(l, whole);
        else
            restrict_coarse<T>(l, whole);
    }
    static __device__ __forceinline__ void through_from(int l) {
        if (CALL)
            restrict_through_call<T>(l);
        else
            restrict_through<T>(l);
    }
    static __device__ __forceinline__ void post(int l) {
        if (CALL)
            coarse_post_call<T>(l);
        else
            coarse_post<T>(l);
    }
    static __device__ __forceinline__ void dense() {
        if (CALL)
            dense_apply_call<T>();
        else
            dense_apply<T>();
    }
};

/* The V-cycle z = M r after its first red half sweep on the node grid
 * (done by the caller, fused with the CG update of r).  Every block executes
 * the same grid barriers; returns the grid-wide r.z of the final z and puts
 * z.z in zz (the last barrier is the one of that reduction). */
template <typename T, bool CALL>
__device__ __forceinline__ double vcycle_rest(cg::grid_group &grid, double *partials, int &round, double &zz) {
    using P = Pass<T, CALL>;
    const MgArgs<T> &A = shared_of<T>().A;
    const Fine<T> &F = shared_of<T>().F;
    const int NL = A.nlev;
    if (NL == 0) { /* Jacobi: the caller computed z on every node */
        T rz = 0, z2 = 0;
        int64_t nn = (int64_t)F.g.ni * F.g.nj * F.g.nk;
        const Span S = span(true, (uint32_t)nn);
        for (int64_t u = S.t; u < S.end; u += S.step)
            if (F.code[u] & SELF) {
                T zu = F.z[u];
                rz += F.r[u] * zu;
                z2 += zu * zu;
            }
        const T vt[2] = {rz, z2};
        double v[2];
        grid_sum<2, T>(grid, vt, v, partials, round);
        zz = v[1];
        return v[0];
    }
    const int GL = A.grid_levels;
    if (!CALL && A.fine_pre) {
        restrict_through_fine<T>();
    } else {
        P::template fine<PRE_BLACK>();
        grid.sync();
        P::restrict_to_first();
    }
    grid.sync();
    int l = 1; /* level l lives in A.L[l-1] and its red half was fused */
    for (; l < GL && l < NL; l++) {
        if (A.L[l - 1].merge & MERGE_PRE) {
            P::through_from(l - 1);
        } else {
            P::template coarse<false>(l - 1, 1, true);
            grid.sync();
            P::restrict_from(l - 1, true);
        }
        grid.sync();
    }
    const int lblock = l;
    const bool coarsest_whole = NL < GL;
    const int nuc = A.nu_coarse;
    if (!coarsest_whole) {
        if (blockIdx.x == 0) {
            /* with shared-memory levels, stage b and e of the first one */
            const MgArgs<T> &B = shared_of<T>().B;
            const bool staged = B.smem_from >= 0 && B.smem_from == lblock - 1;
            if (staged) {
                const MgLevel<T> &G0 = A.L[lblock - 1], &S0 = B.L[lblock - 1];
                for (int64_t t = threadIdx.x; t < G0.n; t += blockDim.x) {
                    S0.b[t] = G0.b[t];
                    S0.e[t] = G0.e[t];
                }
                __syncthreads();
            }
            for (int b = lblock; b < NL; b++) {
                P::template coarse<false>(b - 1, 1, false);
                __syncthreads();
                P::restrict_from(b - 1, false);
                __syncthreads();
            }
            for (int s = 0; s < nuc; s++) {
                if (s) {
                    P::template coarse<false>(NL - 1, 0, false);
                    __syncthreads();
                }
                P::template coarse<false>(NL - 1, 1, false);
                __syncthreads();
            }
            for (int s = 0; s < nuc; s++) {
                P::template coarse<false>(NL - 1, 1, false);
                __syncthreads();
                P::template coarse<false>(NL - 1, 0, false);
                __syncthreads();
            }
            for (int b = NL - 1; b >= lblock; b--) {
                P::template coarse<true>(b - 1, 1, false);
                __syncthreads();
                P::template coarse<false>(b - 1, 0, false);
                __syncthreads();
            }
            if (staged) {
                const MgLevel<T> &G0 = A.L[lblock - 1], &S0 = B.L[lblock - 1];
                for (int64_t t = threadIdx.x; t < G0.n; t += blockDim.x) G0.e[t] = S0.e[t];
            }
        }
        grid.sync();
    } else if (A.dense && *A.dense_ok) {
        P::dense();
        grid.sync();
    } else {
        for (int s = 0; s < nuc; s++) {
            if (s) {
                P::template coarse<false>(NL - 1, 0, true);
                grid.sync();
            }
            P::template coarse<false>(NL - 1, 1, true);
            grid.sync();
        }
        for (int s = 0; s < nuc; s++) {
            P::template coarse<false>(NL - 1, 1, true);
            grid.sync();
            P::template coarse<false>(NL - 1, 0, true);
            grid.sync();
        }
    }
    const int top = coarsest_whole ? NL - 1 : lblock - 1;
    for (int b = top; b >= 1; b--) {
        if (A.L[b - 1].merge & MERGE_POST) {
            P::post(b - 1);
        } else {
            P::template coarse<true>(b - 1, 1, true);
            grid.sync();
            P::template coarse<false>(b - 1, 0, true);
        }
        grid.sync();
    }
    const Dots<T> db = P::template fine<POST_BLACK>();
    grid.sync();
    const Dots<T> dr = P::template fine<POST_RED>();
    const T vt[2] = {db.rz + dr.rz, db.zz + dr.zz};
    double v[2];
    grid_sum<2, T>(grid, vt, v, partials, round);
    zz = v[1];
    return v[0];
}



/* The pairs of phi and rho / eps0 at every node, once per solve, with the
 * predictor folded in.  phi_prev holds two rows, the potentials of the last
 * two solves before this one (p1 = phi_prev, p2 = phi_prev + nn); phi is
 * the last solve's.  predict 1: p1 = phi; 2: also start each unknown from
 * 2 phi - p1 (linear extrapolation in time), and p2 = p1; 3: start from
 * 3 phi - 3 p1 + p2 (quadratic), and p2 = p1.  In double-float. */
__device__ __noinline__ void df_prepass(const double *__restrict__ phi, const double *__restrict__ rho, float2 *phf,
                                        float2 *rhf, const uint16_t *__restrict__ code, double *phi_prev,
                                        int predict, dfl d_inv_eps0, int64_t nn, Span S) {
    /* four nodes a pass, every load before any store (the pass is bound by
     * the loads in flight) */
    for (uint32_t u0 = S.t; u0 < S.end; u0 += 4 * S.step) {
        double cur[4], prev[4], prev2[4], rh[4];
        uint16_t c[4];
        bool on[4];
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const uint32_t u = u0 + h * S.step;
            on[h] = u < S.end;
            const uint32_t v = on[h] ? u : 0;
            cur[h] = phi[v];
            rh[h] = rho[v];
            c[h] = predict >= 2 ? code[v] : (uint16_t)0;
            prev[h] = predict >= 2 ? phi_prev[v] : 0.0;
            prev2[h] = predict == 3 ? phi_prev[nn + v] : 0.0;
        }
#pragma unroll
        for (int h = 0; h < 4; h++) {
            if (!on[h]) continue;
            const uint32_t u = u0 + h * S.step;
            dfl x = df_split(cur[h]);
            if (predict) {
                if (predict >= 2 && (c[h] & SELF)) {
                    const dfl p1 = df_split(prev[h]);
                    if (predict == 2) {
                        x = df_add({2.f * x.h, 2.f * x.l}, df_neg(p1));
                    } else {
                        const dfl d = df_add(x, df_neg(p1));
                        x = df_add({3.f * d.h, 3.f * d.l}, df_split(prev2[h]));
                    }
                }
                if (predict >= 2) phi_prev[nn + u] = prev[h];
                phi_prev[u] = cur[h];
            }
            phf[u] = df_pack(x);
            rhf[u] = df_pack(df_mul(df_split(rh[h]), d_inv_eps0));
        }
    }
}

/* The Newton update phi -= y on the pairs of the unknowns; returns the
 * thread's sum of y^2 */
template <typename T>
__device__ __noinline__ float df_update(const uint16_t *__restrict__ code, const T *__restrict__ yv, float2 *phf,
                                        Span S) {
    float yys = 0.f;
    /* four nodes a pass, every load before any store */
    for (uint32_t u0 = S.t; u0 < S.end; u0 += 4 * S.step) {
        uint16_t c[4];
        float yu[4];
        float2 x[4];
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const uint32_t u = u0 + h * S.step;
            const uint32_t v = u < S.end ? u : 0;
            c[h] = u < S.end ? code[v] : (uint16_t)0;
            yu[h] = (float)yv[v];
            x[h] = phf[v];
        }
#pragma unroll
        for (int h = 0; h < 4; h++) {
            if (!(c[h] & SELF)) continue;
            phf[u0 + h * S.step] = df_pack(df_add(df_unpack(x[h]), {-yu[h], 0.f}));
            yys = __fmaf_rn(yu[h], yu[h], yys);
        }
    }
    return yys;
}

/* phi of the unknowns from their pairs (hi + lo rounded once), four nodes
 * a pass with every load before any store */
__device__ __noinline__ void df_rebuild(const uint16_t *__restrict__ code, const float2 *__restrict__ phf,
                                        double *phi, Span S) {
    for (uint32_t u0 = S.t; u0 < S.end; u0 += 4 * S.step) {
        uint16_t c[4];
        float2 x[4];
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const uint32_t u = u0 + h * S.step;
            c[h] = u < S.end ? code[u] : (uint16_t)0;
            x[h] = phf[u < S.end ? u : 0];
        }
#pragma unroll
        for (int h = 0; h < 4; h++)
            if (c[h] & SELF) phi[u0 + h * S.step] = (double)x[h].x + (double)x[h].y;
    }
}

/* Neumann boundary nodes take the value at the end of their chain (the
 * chains end at unknowns or Dirichlet nodes, which this pass does not
 * write), four nodes a pass */
__device__ __noinline__ void neumann_copies(const int32_t *__restrict__ target, double *phi, Span S) {
    for (uint32_t u0 = S.t; u0 < S.end; u0 += 4 * S.step) {
        int32_t t[4];
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const uint32_t u = u0 + h * S.step;
            t[h] = u < S.end ? target[u] : -1;
        }
#pragma unroll
        for (int h = 0; h < 4; h++)
            if (t[h] >= 0) phi[u0 + h * S.step] = phi[t[h]];
    }
}

/* The Newton residual pass of the float-inner nonlinear solve in
 * double-float arithmetic (per axis c (2 x_u - x_w - x_e), a missing link
 * reading x_u; the Boltzmann factor as expf of the leading part times a
 * first-order factor for the rest; rho / eps0 from its pair), with the
 * Jacobian's Boltzmann diagonal and the first red smoothing half sweep.
 * Returns the thread's sum of r^2.  Not inlined: the call spills the
 * solver's live state once, and the loop gets the registers (inlined, the
 * loop ran 4x slower).  An unknown is an interior node, so its neighbours
 * need no clamp (s1, s2: the y and z strides). */
template <typename T>
__device__ __noinline__ float df_residual(const uint16_t *__restrict__ code, const float2 *__restrict__ phf,
                                          const float2 *__restrict__ rhf, T *z, T *dg, T *r, T *y, Span S,
                                          int32_t s1, int32_t s2, const T ct[3],
                                          const float cl[3], dfl d_phi0, dfl d_inv_te0, dfl d_A0, float A0_te0,
                                          bool jacobi) {
    float ffs = 0.f;
    /* two nodes a pass, every load before the arithmetic; a node that is
     * not an unknown reads the interior node safe_u and stores nothing */
    const int64_t safe_u = (int64_t)s2 + s1 + 1;
    for (uint32_t u0 = S.t; u0 < S.end; u0 += 2 * S.step) {
        uint16_t cq[2];
        int64_t uq[2];
        float2 xq[2], pq[2][6], bq[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t u = u0 + h * S.step;
            cq[h] = u < S.end ? code[u] : (uint16_t)0;
            uq[h] = (cq[h] & SELF) ? u : safe_u;
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float2 *pu = phf + uq[h];
            xq[h] = pu[0];
            pq[h][0] = pu[-1];
            pq[h][1] = pu[1];
            pq[h][2] = pu[-s1];
            pq[h][3] = pu[s1];
            pq[h][4] = pu[-s2];
            pq[h][5] = pu[s2];
            bq[h] = rhf[uq[h]];
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint16_t c = cq[h];
            if (!(c & SELF)) continue;
            const int64_t u = uq[h];
            const float2 xu = xq[h];
            const dfl x = df_unpack(xu);
            dfl L = {0.f, 0.f};
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const unsigned mw = (1u << (2 * a)) | (1u << (6 + 2 * a));
                const unsigned me = (1u << (2 * a + 1)) | (1u << (7 + 2 * a));
                const dfl pw = df_unpack((c & mw) ? pq[h][2 * a] : xu);
                const dfl pe = df_unpack((c & me) ? pq[h][2 * a + 1] : xu);
                const dfl d = df_add(df_add({2.f * x.h, 2.f * x.l}, df_neg(pw)), df_neg(pe));
                L = df_add(L, df_mul(d, {(float)ct[a], cl[a]}));
            }
            const dfl xa = df_mul(df_add(x, df_neg(d_phi0)), d_inv_te0);
            const float ef = expf(xa.h);
            const dfl e = df_fast2(ef, ef * xa.l);
            const dfl Fd = df_add(df_add(L, df_mul(d_A0, e)), df_neg(df_unpack(bq[h])));
            const float rv = Fd.h + Fd.l;
            const float dBt = A0_te0 * ef;
            if (jacobi || !(c & BLACK)) z[u] = (T)(rv / full_diag(c, (T)dBt, ct));
            dg[u] = (T)dBt;
            r[u] = (T)rv;
            y[u] = 0;
            ffs = __fmaf_rn(rv, rv, ffs);
        }
    }
    return ffs;
}

/* p = z + beta p (on the fly at the node and its neighbours) and q = J p;
 * returns the thread's sum of p q.  old: there is a previous p.  LIGHT: J p
 * = J z + beta J p_old, the last q instead of p's neighbours (10 float64
 * instructions a node, 28 with p formed at seven nodes).  PER nodes per pass,
 * every load before any store; the loads do not wait for the code word (a
 * plane of padding around the vectors takes a boundary node's missing
 * neighbours, a node past the end reads node 0); a node that is not an
 * unknown stores nothing. */
template <typename T, int PER>
__device__ __forceinline__ T pcg_direction(const T *__restrict__ pold, T *__restrict__ pnew, T *__restrict__ q,
                                           T beta, bool old) {
    const Fine<T> &F = shared_of<T>().F;
    const uint16_t *__restrict__ code = F.code;
    const T *__restrict__ z = F.z, *__restrict__ dg = F.dg;
    const T ct[3] = {F.ct[0], F.ct[1], F.ct[2]};
    const int32_t sy = F.g.ni, sz = F.g.ni * F.g.nj;
    const Span S = span(true, F.nn);
    T pq = 0;
#pragma unroll 1
    for (uint32_t t = S.t; t < S.end; t += PER * S.step) {
        uint32_t u[PER];
        uint16_t c[PER];
        T zc[PER], pc[PER], dB[PER], zn[PER][6], pn[PER][6];
#pragma unroll
        for (int h = 0; h < PER; h++) {
            const bool in = t + h * S.step < S.end;
            u[h] = in ? t + h * S.step : 0u;
            c[h] = in ? code[u[h]] : (uint16_t)0;
            zc[h] = z[u[h]];
            dB[h] = dg[u[h]];
            load_neighbours(z, u[h], sy, sz, zn[h]);
            pc[h] = old ? pold[u[h]] : (T)0;
            if (LIGHT<T>) {
                pn[h][0] = old ? q[u[h]] : (T)0;
            } else if (old) {
                load_neighbours(pold, u[h], sy, sz, pn[h]);
            } else {
#pragma unroll
                for (int m = 0; m < 6; m++) pn[h][m] = (T)0;
            }
        }
#pragma unroll
        for (int h = 0; h < PER; h++) {
            if (!(c[h] & SELF)) continue;
            const T pu = zc[h] + beta * pc[h];
            T s;
            if (LIGHT<T>) {
                s = dB[h] * zc[h];
#pragma unroll
                for (int a = 0; a < 3; a++) s -= ct[a] * (zn[h][2 * a] + zn[h][2 * a + 1]);
                s += beta * pn[h][0];
            } else {
#pragma unroll
                for (int m = 0; m < 6; m++) pn[h][m] = zn[h][m] + beta * pn[h][m];
                s = jacobian_apply(c[h], dB[h], ct, pu, pn[h]);
            }
            pnew[u[h]] = pu;
            q[u[h]] = s;
            pq += pu * s;
        }
    }
    return pq;
}

/* y += alpha p, r -= alpha q, and the first red half sweep of the
 * preconditioner; returns the thread's sum of r^2 */
template <typename T>
__device__ __forceinline__ T pcg_update(T *__restrict__ y, const T *__restrict__ p, const T *__restrict__ q, T alpha) {
    const Fine<T> &F = shared_of<T>().F;
    const uint16_t *__restrict__ code = F.code;
    T *__restrict__ z = F.z, *__restrict__ r = F.r;
    const T *__restrict__ dd = LIGHT<T> ? F.id : F.dg;
    const T ct[3] = {F.ct[0], F.ct[1], F.ct[2]};
    const bool jacobi = shared_of<T>().A.nlev == 0;
    const Span S = span(true, F.nn);
    T rr = 0;
#pragma unroll 1
    for (uint32_t t = S.t; t < S.end; t += 2 * S.step) {
        uint32_t u[2];
        uint16_t c[2];
        T yv[2], pv[2], rv[2], qv[2], dv[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const bool in = t + h * S.step < S.end;
            u[h] = in ? t + h * S.step : 0u;
            c[h] = in ? code[u[h]] : (uint16_t)0;
            yv[h] = y[u[h]];
            pv[h] = p[u[h]];
            rv[h] = r[u[h]];
            qv[h] = q[u[h]];
            dv[h] = dd[u[h]];
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            pin(yv[h]);
            pin(pv[h]);
            pin(rv[h]);
            pin(qv[h]);
            pin(dv[h]);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (!(c[h] & SELF)) continue;
            y[u[h]] = yv[h] + alpha * pv[h];
            const T ru = rv[h] - alpha * qv[h];
            r[u[h]] = ru;
            rr += ru * ru;
            if (jacobi || !(c[h] & BLACK))
                z[u[h]] = LIGHT<T> ? ru * dv[h] : ru / full_diag(c[h], dv[h], ct);
        }
    }
    return rr;
}

template <typename T>
__device__ __noinline__ T pcg_direction_call(const T *pold, T *pnew, T *q, T beta, bool old) {
    return pcg_direction<T, 2>(pold, pnew, q, beta, old);
}
template <typename T>
__device__ __noinline__ T pcg_update_call(T *y, const T *p, const T *q, T alpha) {
    return pcg_update<T>(y, p, q, alpha);
}

template <typename T, int THREADS, bool CALL>
__global__ void __launch_bounds__(THREADS, 1) k_newton_pcg(Geo g, double *phi, const double *__restrict__ rho,
                                                        const uint16_t *__restrict__ code,
                                                        const int32_t *__restrict__ target, double phi0,
                                                        double te0, double n0, int nr_max, double nr_tol,
                                                        int pcg_max, double pcg_tol, T *y, T *r, T *z, T *p0,
                                                        T *p1, T *q, T *dg, T *id, MgArgs<T> mg, double *partials, SolveStatus *st, int *err,
                                                        double *lin_y, const double *__restrict__ lin_b,
                                                        int gs_max, double gs_tol, float2 *dfbuf, double *phi_prev,
                                                        int predict, Coef3<T> ctp) {
    cg::grid_group grid = cg::this_grid();
    extern __shared__ __align__(16) unsigned char pcg_smem[];
    __shared__ T bc_alpha, bc_beta;
    __shared__ int bc_stop;
    const int64_t nn = (int64_t)g.ni * g.nj * g.nk;
    const int64_t sy = g.ni, sz = (int64_t)g.ni * g.nj;
    const int64_t off[6] = {-1, 1, -sy, sy, -sz, sz};
    const int64_t safe = sz + sy + 1; /* the interior node (1,1,1) */
    const double cd[3] = {1.0 / (g.dh[0] * g.dh[0]), 1.0 / (g.dh[1] * g.dh[1]), 1.0 / (g.dh[2] * g.dh[2])};
    /* (T)cd from the host: derived here from cd, the compiler re-derived it
     * inside the node loops (a float64-to-float conversion each time, on the
     * narrow float64 pipe) instead of holding it */
    const bool tf = sizeof(T) == sizeof(float);
    const T ct[3] = {tf ? ctp.c[0] : (T)cd[0], tf ? ctp.c[1] : (T)cd[1], tf ? ctp.c[2] : (T)cd[2]};
    const double A0 = PCG_QE * n0 / PCG_EPS_0;
    const double inv_te0 = 1.0 / te0, A0_te0 = A0 / te0, inv_eps0 = 1.0 / PCG_EPS_0;
    const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const Span S = span(true, (uint32_t)nn); /* this thread's nodes */
    const bool jacobi = mg.nlev == 0;
    Fine<T> F;
    F.g = g;
    F.code = code;
    for (int m = 0; m < 3; m++) F.ct[m] = ct[m];
    F.nn = (uint32_t)nn;
    F.dg = dg;
    F.id = id;
    F.r = r;
    F.z = z;
    F.ncolour = (uint32_t)((g.ni - 1) / 2) * (uint32_t)(g.nj - 2) * (uint32_t)(g.nk - 2);
    shared_init(F, mg, pcg_smem);
    int round = 0, nr, conv = 0, inner = 0, fallback = 0;
    double norm = 0;
    /* linear mode (lin_y != null): Newton on F(y) = J y - b with J frozen at
     * phi solves J y = b; the stopping test is relative to the first update */
    const bool linear = lin_y != nullptr;
    /* float inner solve of the nonlinear problem: the Newton residual and
     * update run in double-float arithmetic on the float pipes (the float64
     * pipe of this GPU is narrow) from phi and rho / eps0 split once into
     * (hi, lo) pairs here; phi is rebuilt from its pairs after the last
     * update */
    const bool dfm = sizeof(T) == sizeof(float) && !linear && dfbuf != nullptr;
    float2 *phf = dfbuf, *rhf = dfbuf ? dfbuf + nn : nullptr;
    const dfl d_phi0 = df_of(phi0), d_inv_te0 = df_of(inv_te0), d_A0 = df_of(A0), d_inv_eps0 = df_of(inv_eps0);
    if (dfm) {
        df_prepass(phi, rho, phf, rhf, code, phi_prev, predict, d_inv_eps0, nn, S);
        grid.sync();
    }
    const float cl[3] = {(float)(cd[0] - (double)ct[0]), (float)(cd[1] - (double)ct[1]),
                         (float)(cd[2] - (double)ct[2])};
    double nr_scale = linear ? 0.0 : 1.0;
    double zz_stop = nr_tol * nr_tol / 4.0 * (double)nn * nr_scale;
    for (nr = 0; nr < nr_max; nr++) {
        /* Newton residual (float64) and the Boltzmann part of the Jacobian
         * diagonal; the first red smoothing half sweep (or Jacobi) of the
         * preconditioner rides along */
        double ff = 0;
        const double *XR = linear ? lin_y : phi;
        if (dfm) {
            /* the residual of the float-inner form below, in double-float:
             * per axis c (2 x_u - x_w - x_e) (a missing link reads x_u), the
             * Boltzmann factor as expf of the leading part times a
             * first-order factor for the rest, rho / eps0 from its pair */
            const float ffs = df_residual<T>(code, phf, rhf, z, dg, r, y, S, (int32_t)sy, (int32_t)sz, ct, cl,
                                             d_phi0, d_inv_te0, d_A0, (float)A0_te0, jacobi);
            ff = (double)ffs;
        } else
        /* two nodes per pass, every load before any store; the loads do not
         * wait for the code word (neighbour indices are clamped into the
         * grid, a node past the end reads the interior node (1,1,1)), and
         * a node that is not an unknown stores nothing */
        for (uint32_t u0 = S.t; u0 < S.end; u0 += 2 * S.step) {
            const int64_t uq[2] = {u0, u0 + S.step};
            bool onq[2];
            uint16_t c[2];
            int64_t u[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                c[h] = uq[h] < S.end ? code[uq[h]] : (uint16_t)0;
                onq[h] = c[h] & SELF;
                u[h] = uq[h] < S.end ? uq[h] : safe;
            }
            double xu[2], pn[2][6], ph[2], bv[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                xu[h] = XR[u[h]];
#pragma unroll
                for (int m = 0; m < 6; m++) pn[h][m] = XR[clamp_node(u[h] + off[m], nn)];
                ph[h] = phi[u[h]];
                bv[h] = linear ? lin_b[u[h]] : rho[u[h]];
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (!onq[h]) continue;
                double Fv;
                T rv, dBt;
                if (sizeof(T) == sizeof(float)) {
                    /* the float-inner form spends fewer float64 operations
                     * (the float64 pipe is narrow here): per axis
                     * c (2 x_u - x_w - x_e) with a missing link reading x_u
                     * itself; the Boltzmann factor as the float exponential of
                     * the leading part of the argument times a first-order
                     * factor for the rest (relative error ~1e-7, which moves
                     * phi by ~Te 1e-7, far below the Newton tolerance); the
                     * Jacobian's Boltzmann diagonal in float */
                    double L = 0;
#pragma unroll
                    for (int a = 0; a < 3; a++) {
                        const unsigned mw = (1u << (2 * a)) | (1u << (6 + 2 * a));
                        const unsigned me = (1u << (2 * a + 1)) | (1u << (7 + 2 * a));
                        const double pw = (c[h] & mw) ? pn[h][2 * a] : xu[h];
                        const double pe = (c[h] & me) ? pn[h][2 * a + 1] : xu[h];
                        L = fma(cd[a], fma(2.0, xu[h], -(pw + pe)), L);
                    }
                    const double xa = (ph[h] - phi0) * inv_te0;
                    const float xh = (float)xa;
                    const float ef = expf(xh);
                    const double e = fma((double)ef, xa - (double)xh, (double)ef);
                    if (linear) {
                        const double dB = A0_te0 * e;
                        Fv = fma(dB, xu[h], L) - bv[h];
                        dBt = (T)dB;
                    } else {
                        Fv = fma(-bv[h], inv_eps0, fma(A0, e, L));
                        dBt = (T)((float)A0_te0 * ef);
                    }
                    rv = (T)Fv;
                    if (jacobi || !(c[h] & BLACK)) z[u[h]] = rv / full_diag(c[h], dBt, ct);
                } else {
                    double L = 0, dL = 0;
#pragma unroll
                    for (int m = 0; m < 6; m++) {
                        const bool on = c[h] & ((1u << m) | (1u << (6 + m)));
                        L += on ? cd[m >> 1] * (xu[h] - pn[h][m]) : 0.0;
                        dL += on ? cd[m >> 1] : 0.0;
                    }
                    const double e = exp((ph[h] - phi0) * inv_te0);
                    const double dB = A0_te0 * e;
                    Fv = linear ? L + dB * xu[h] - bv[h] : L + A0 * e - bv[h] * inv_eps0;
                    rv = (T)Fv;
                    dBt = (T)(dL + dB); /* the whole diagonal (LIGHT) */
                    const T iv = (T)(1.0 / (dL + dB));
                    if (jacobi || !(c[h] & BLACK)) z[u[h]] = rv * iv;
                    id[u[h]] = iv;
                }
                dg[u[h]] = dBt;
                r[u[h]] = rv;
                y[u[h]] = 0;
                ff += Fv * Fv;
            }
        }
        const double t1[1] = {ff};
        double s1[1];
        grid_sum<1, double>(grid, t1, s1, partials, round);
        double FF = s1[0];
        if (!isfinite(FF)) {
            if (gtid == 0) atomicOr(err, DERR_NONFINITE);
            break;
        }
        bool take_z = false;
        if (FF > 0) {
            const double stop2 = pcg_tol * pcg_tol * FF;
            double ZZ;
            double RZ = vcycle_rest<T, CALL>(grid, partials, round, ZZ);
            /* the first preconditioned residual already estimates an update
             * below the inner stop: it is the update */
            take_z = ZZ < zz_stop;
            bool inner_ok = take_z;
            T beta = 0;
            T *pold = p0, *pnew = p1;
            for (int it = 0; it < pcg_max && !take_z; it++) {
                const T pq = CALL ? pcg_direction_call<T>(pold, pnew, q, beta, it > 0)
                                  : pcg_direction<T, 2>(pold, pnew, q, beta, it > 0);
                const T t3[1] = {pq};
                double s3[1];
                grid_sum<1, T>(grid, t3, s3, partials, round);
                /* block-uniform scalars are computed by one thread and
                 * broadcast: 32 warps each dividing in float64 would queue
                 * on the narrow float64 pipe */
                if (threadIdx.x == 0) bc_alpha = (T)(RZ / s3[0]);
                __syncthreads();
                const T alpha = bc_alpha;
                const T rr = CALL ? pcg_update_call<T>(y, pnew, q, alpha) : pcg_update<T>(y, pnew, q, alpha);
                const T t4[1] = {rr};
                double s4[1];
                grid_sum<1, T>(grid, t4, s4, partials, round);
                inner++;
                if (threadIdx.x == 0) bc_stop = !(s4[0] > stop2); /* also leaves on NaN */
                __syncthreads();
                if (bc_stop) {
                    inner_ok = true;
                    break;
                }
                double RZn = vcycle_rest<T, CALL>(grid, partials, round, ZZ);
                /* z = M r estimates the remaining error of y: once its RMS is
                 * below half the Newton tolerance, further inner
                 * iterations cannot change the outcome of the Newton test */
                if (threadIdx.x == 0) {
                    bc_stop = ZZ < zz_stop;
                    bc_beta = (T)(RZn / RZ);
                }
                __syncthreads();
                if (bc_stop) {
                    inner_ok = true;
                    break;
                }
                beta = bc_beta;
                RZ = RZn;
                T *tp = pold;
                pold = pnew;
                pnew = tp;
            }
            /* The reference's fallback when the linear PCG fails
             * (ch3/ver2/PotentialSolver.cpp:270-271, solveGSLinear :433-461):
             * Gauss-Seidel (omega 1) on the same linear system from the
             * inner solve's last iterate, the residual's RMS checked every
             * 25 sweeps (from the first) against the solver tolerance, at
             * most gs_max sweeps.  Here the sweeps are red-black and act on
             * the correction, J e = r from e = 0 (r = F - J y is the PCG's
             * residual), then y += e. */
            if (!inner_ok && gs_max > 0) {
                for (int64_t u = S.t; u < S.end; u += S.step) z[u] = (T)0;
                grid.sync();
                for (int sw = 0; sw < gs_max; sw++) {
                    for (int col = 0; col < 2; col++) {
                        for (int64_t u = S.t; u < S.end; u += S.step) {
                            const uint16_t cc = code[u];
                            if (!(cc & SELF) || ((cc & BLACK) ? 1 : 0) != col) continue;
                            T acc = r[u];
#pragma unroll
                            for (int m = 0; m < 6; m++)
                                if (cc & (1u << m)) acc += ct[m >> 1] * z[u + off[m]];
                            z[u] = LIGHT<T> ? acc * id[u] : acc / full_diag(cc, dg[u], ct);
                        }
                        grid.sync();
                    }
                    fallback++;
                    if (sw % 25 == 0) {
                        T rr2 = 0;
                        for (int64_t u = S.t; u < S.end; u += S.step) {
                            const uint16_t cc = code[u];
                            if (!(cc & SELF)) continue;
                            T xn[6];
#pragma unroll
                            for (int m = 0; m < 6; m++) xn[m] = (cc & (1u << m)) ? z[u + off[m]] : (T)0;
                            T Jz;
                            if (LIGHT<T>) {
                                Jz = dg[u] * z[u];
#pragma unroll
                                for (int a = 0; a < 3; a++) Jz -= ct[a] * (xn[2 * a] + xn[2 * a + 1]);
                            } else {
                                Jz = jacobian_apply(cc, dg[u], ct, z[u], xn);
                            }
                            const T R = r[u] - Jz;
                            rr2 += R * R;
                        }
                        const T t5[1] = {rr2};
                        double s5[1];
                        grid_sum<1, T>(grid, t5, s5, partials, round);
                        if (threadIdx.x == 0) bc_stop = sqrt(s5[0] / (double)nn) < gs_tol;
                        __syncthreads();
                        if (bc_stop) break;
                    }
                }
                for (int64_t u = S.t; u < S.end; u += S.step)
                    if (code[u] & SELF) y[u] += z[u];
                grid.sync();
            }
        }
        /* Newton update */
        double yy = 0;
        double *X = linear ? lin_y : phi;
        if (dfm) {
            yy = (double)df_update<T>(code, take_z ? z : y, phf, S);
        } else
        /* two nodes per pass, loads ahead of the code test and the stores */
        for (uint32_t u0 = S.t; u0 < S.end; u0 += 2 * S.step) {
            const int64_t uq[2] = {u0, u0 + S.step};
            int64_t u[2];
            uint16_t c[2];
            T yv[2];
            double xv[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                u[h] = uq[h] < S.end ? uq[h] : safe;
                c[h] = uq[h] < S.end ? code[u[h]] : (uint16_t)0;
                yv[h] = take_z ? z[u[h]] : y[u[h]];
                xv[h] = X[u[h]];
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (!(c[h] & SELF)) continue;
                const double yu = (double)yv[h];
                X[u[h]] = xv[h] - yu;
                yy += yu * yu;
            }
        }
        const double t6[1] = {yy};
        double s6[1];
        grid_sum<1, double>(grid, t6, s6, partials, round);
        norm = sqrt(s6[0] / (double)nn);
        if (!isfinite(norm)) {
            if (gtid == 0) atomicOr(err, DERR_NONFINITE);
            break;
        }
        if (linear && nr == 0) {
            nr_scale = norm;
            zz_stop = 0.01 * nr_tol * nr_tol * norm * norm * (double)nn;
        }
        if (norm < nr_tol * nr_scale || (linear && norm == 0.0)) {
            conv = 1;
            nr++;
            break;
        }
    }
    if (dfm) {
        df_rebuild(code, phf, phi, S);
        grid.sync();
    }
    if (!linear) neumann_copies(target, phi, S);
    if (gtid == 0) {
        st->converged = conv;
        st->iterations = nr;
        st->inner_iterations = inner;
        st->fallback_sweeps = fallback;
        st->residual = norm;
        st->solves += 1;
        st->outer_total += nr;
        st->inner_total += inner;
    }
}

/* Galerkin coarse operator of level l+1 from level l (deterministic gather:
 * one thread per coarse node, children and their links in a fixed order).
 * Level 0 is the node grid with the operator L (Dirichlet links kept on the
 * diagonal); the Boltzmann diagonal term is left to the fine smoother. */
template <typename T>
__global__ void k_mg_setup(Geo g, const uint16_t *__restrict__ code, MgLevel<T> Lf, MgLevel<T> C, int from_fine) {
    int64_t I = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= C.n) return;
    int ci = (int)(I % C.nx);
    int cj = (int)((I / C.nx) % C.ny);
    int ck = (int)(I / ((int64_t)C.nx * C.ny));
    const double cd[3] = {1.0 / (g.dh[0] * g.dh[0]), 1.0 / (g.dh[1] * g.dh[1]), 1.0 / (g.dh[2] * g.dh[2])};
    double diag = 0, w[6] = {0, 0, 0, 0, 0, 0};
    int nx = from_fine ? g.ni : Lf.nx, ny = from_fine ? g.nj : Lf.ny, nz = from_fine ? g.nk : Lf.nz;
    int64_t offs[6] = {-1, 1, -(int64_t)nx, nx, -(int64_t)nx * ny, (int64_t)nx * ny};
    const int di[6] = {-1, 1, 0, 0, 0, 0}, dj[6] = {0, 0, -1, 1, 0, 0}, dk[6] = {0, 0, 0, 0, -1, 1};
    for (int d = 0; d < 8; d++) {
        int i = 2 * ci + (d & 1), j = 2 * cj + ((d >> 1) & 1), k = 2 * ck + (d >> 2);
        if (i >= nx || j >= ny || k >= nz) continue;
        int64_t u = ((int64_t)k * ny + j) * nx + i;
        if (from_fine) {
            uint16_t c = code[u];
            if (!(c & SELF)) continue;
            for (int m = 0; m < 6; m++)
                if (c & ((1u << m) | (1u << (6 + m)))) diag += cd[m >> 1];
            for (int m = 0; m < 6; m++) {
                if (!(c & (1u << m))) continue;
                bool inside = ((i + di[m]) >> 1) == ci && ((j + dj[m]) >> 1) == cj && ((k + dk[m]) >> 1) == ck;
                if (inside)
                    diag -= cd[m >> 1];
                else
                    w[m] += cd[m >> 1];
            }
        } else {
            double dd = (double)Lf.diag[u];
            if (dd == 0) continue;
            diag += dd;
            for (int m = 0; m < 6; m++) {
                double wm = (double)Lf.w[m * Lf.n + u];
                if (wm == 0) continue;
                bool inside = ((i + di[m]) >> 1) == ci && ((j + dj[m]) >> 1) == cj && ((k + dk[m]) >> 1) == ck;
                if (inside)
                    diag -= wm;
                else
                    w[m] += wm;
            }
        }
        (void)offs;
    }
    C.diag[I] = (T)diag;
    C.id[I] = diag != 0 ? (T)(1.0 / diag) : (T)0;
    for (int m = 0; m < 6; m++) C.w[m * C.n + I] = (T)w[m];
}

/* The coarsest level's operator as a dense float64 matrix (A e = diag e -
 * sum_m w_m e_nb(m)); an aggregate without unknowns (diag 0) gets an
 * identity row. */
template <typename T>
__global__ void k_dense_build(MgLevel<T> L, double *M, double *diag0) {
    const int64_t n = L.n;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * n) return;
    const int64_t i = t / n, j = t - i * n;
    const double di = (double)L.diag[i];
    double v = 0;
    if (di == 0) {
        v = i == j ? 1.0 : 0.0;
    } else if (i == j) {
        v = di;
    } else if ((double)L.diag[j] != 0) {
        const int xi = (int)(i % L.nx), yi = (int)((i / L.nx) % L.ny), zi = (int)(i / ((int64_t)L.nx * L.ny));
        const int xj = (int)(j % L.nx), yj = (int)((j / L.nx) % L.ny), zj = (int)(j / ((int64_t)L.nx * L.ny));
        const int dx = xj - xi, dy = yj - yi, dz = zj - zi;
        int m = -1;
        if (dy == 0 && dz == 0 && (dx == -1 || dx == 1)) m = dx < 0 ? 0 : 1;
        if (dx == 0 && dz == 0 && (dy == -1 || dy == 1)) m = dy < 0 ? 2 : 3;
        if (dx == 0 && dy == 0 && (dz == -1 || dz == 1)) m = dz < 0 ? 4 : 5;
        if (m >= 0) v = -(double)L.w[m * n + i];
    }
    M[t] = v;
    if (i == j) diag0[i] = v;
}

/* Row k of the inversion, divided by its pivot, for every block to read, and
 * its place in row: 1 / pivot in column k.  One thread divides 1 by the pivot
 * and the block's threads multiply (div_rcp; a division where an operand is
 * too small for it).  A pivot that vanished against the original diagonal (a
 * singular operator) clears *ok. */
__device__ __forceinline__ void gj_publish(const double *row, int n, int k, double diag0, double *out, int *ok) {
    __shared__ double piv, rpiv;
    if (threadIdx.x == 0) {
        double p = row[k];
        if (!(p > 1e-9 * diag0)) {
            *ok = 0;
            p = 1.0;
        }
        piv = p;
        rpiv = 1.0 / p;
    }
    __syncthreads();
    const double p = piv, y = rpiv;
    const bool normal = p > 1e-100 && p < 1e100;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const double a = j == k ? 1.0 : row[j];
        out[j] = normal && (fabs(a) > 1e-150 || a == 0.0) && fabs(a) < 1e150 ? div_rcp(a, p, y) : a / p;
    }
}

/* In-place Gauss-Jordan inversion without pivoting (the operator is
 * symmetric positive definite), in one cooperative launch.  A block keeps
 * every gridDim.x-th row, in shared memory when they fit (staged), else where
 * they lie.  For each k it reads the scaled row k and eliminates column k
 * from its rows, the owner of row k + 1 that one first, so that it publishes
 * the next scaled row while the others still work: one grid barrier a pivot
 * and only a row of traffic.  With two barriers, a column buffer and the
 * matrix in global memory 1024 rows took 13.1 ms; 6.6 ms now, of which the
 * barriers and the row's way through L2 are the most.  pub: two rows of n. */
__global__ void __launch_bounds__(1024, 1) k_gauss_jordan(double *M, int n, double *pub,
                                                          const double *__restrict__ diag0, int *ok, int staged) {
    cg::grid_group grid = cg::this_grid();
    extern __shared__ __align__(16) double gj_rows[];
    __shared__ double col[GJ_ROWS];
    const int G = (int)gridDim.x, b = (int)blockIdx.x;
    const int cnt = (n - b + G - 1) / G; /* rows b, b + G, ...; G <= n */
    double *S = staged ? gj_rows : M + (int64_t)b * n;
    const int64_t ld = staged ? n : (int64_t)G * n;
    if (staged) {
        for (int m = 0; m < cnt; m++)
            for (int j = threadIdx.x; j < n; j += blockDim.x) S[m * ld + j] = M[((int64_t)b + (int64_t)m * G) * n + j];
        __syncthreads();
    }
    if (b == 0) gj_publish(S, n, 0, diag0[0], pub, ok);
    grid.sync();
    for (int k = 0; k < n; k++) {
        const double *R = pub + (k & 1) * n;
        double r[4]; /* n <= 4096 */
#pragma unroll
        for (int q = 0; q < 4; q++) r[q] = threadIdx.x + 1024 * q < n ? __ldcg(R + threadIdx.x + 1024 * q) : 0.0;
        for (int m = threadIdx.x; m < cnt; m += blockDim.x) col[m] = S[m * ld + k];
        __syncthreads();
        const int next = k + 1 < n && (k + 1) % G == b ? (k + 1) / G : -1;
        for (int t = next >= 0 ? -1 : 0; t < cnt; t++) {
            const int m = t < 0 ? next : t;
            if (t >= 0 && t == next) continue;
            const double f = col[m];
            const bool own = b + m * G == k;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int j = threadIdx.x + 1024 * q;
                if (j >= n) break;
                const double x = j == k ? 0.0 : S[m * ld + j];
                S[m * ld + j] = own ? r[q] : x - f * r[q];
            }
            if (t < 0) {
                __syncthreads();
                gj_publish(S + m * ld, n, k + 1, diag0[k + 1], pub + ((k + 1) & 1) * n, ok);
            }
        }
        grid.sync();
    }
    if (staged)
        for (int m = 0; m < cnt; m++)
            for (int j = threadIdx.x; j < n; j += blockDim.x) M[((int64_t)b + (int64_t)m * G) * n + j] = S[m * ld + j];
}

/* the inverse in T, symmetrised; rows and columns of aggregates without
 * unknowns are zero */
template <typename T>
__global__ void k_dense_store(MgLevel<T> L, const double *__restrict__ M, T *out) {
    const int64_t n = L.n;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * n) return;
    const int64_t i = t / n, j = t - i * n;
    const bool live = (double)L.diag[i] != 0 && (double)L.diag[j] != 0;
    out[t] = live ? (T)(0.5 * (M[t] + M[j * n + i])) : (T)0;
}

/* ======================================================================== */
template <typename T>
static size_t mg_layout(World &w, MgArgs<T> &A, char *base) {
    size_t off = 0;
    int nx = (w.g.ni + 1) / 2, ny = (w.g.nj + 1) / 2, nz = (w.g.nk + 1) / 2;
    int nlev = 0, grid_levels = 1;
    while (nlev < MG_MAX) {
        MgLevel<T> &L = A.L[nlev];
        L.nx = nx;
        L.ny = ny;
        L.nz = nz;
        L.merge = 0;
        L.n = (int64_t)nx * ny * nz;
        size_t bytes = ((L.n * sizeof(T) + 255) / 256) * 256;
        L.diag = (T *)(base ? base + off : nullptr);
        off += bytes;
        L.id = (T *)(base ? base + off : nullptr);
        off += bytes;
        L.w = (T *)(base ? base + off : nullptr);
        off += 6 * bytes;
        L.b = (T *)(base ? base + off : nullptr);
        off += bytes;
        L.e = (T *)(base ? base + off : nullptr);
        off += bytes;
        L.f = (T *)(base ? base + off : nullptr);
        off += bytes;
        nlev++;
        if (L.n >= w.mg_block_nodes) grid_levels = nlev + 1;
        if (L.n <= 64 || (nx <= 2 && ny <= 2 && nz <= 2)) break;
        nx = (nx + 1) / 2;
        ny = (ny + 1) / 2;
        nz = (nz + 1) / 2;
    }
    A.nlev = w.mg_levels_max < nlev ? w.mg_levels_max : nlev;
    /* the first level with at most mg_dense_max nodes becomes the coarsest,
     * solved by its dense inverse on the whole grid (every level above it
     * runs on the whole grid too); the float64 work matrix of the inversion,
     * its two published rows and the diagonal follow the levels */
    A.dense = nullptr;
    A.dense_n = 0;
    if (w.mg_dense_max > 0)
        for (int i = 0; i < A.nlev; i++)
            if (A.L[i].n <= w.mg_dense_max) {
                A.nlev = i + 1;
                A.dense_n = (int)A.L[i].n;
                grid_levels = A.nlev + 1;
                break;
            }
    if (A.dense_n > 0) {
        const size_t nsq = (size_t)A.dense_n * A.dense_n;
        A.dense = (T *)(base ? base + off : nullptr);
        off += (nsq * sizeof(T) + 255) / 256 * 256;
        off += (nsq * sizeof(double) + 255) / 256 * 256 + 3 * (((size_t)A.dense_n * sizeof(double) + 255) / 256 * 256);
        A.dense_ok = (const int *)(base ? base + off : nullptr);
        off += 256;
    } else {
        A.dense_ok = nullptr;
    }
    A.grid_levels = grid_levels;
    A.nu_coarse = 2;
    A.scale = (T)w.mg_scale;
    /* block 0 works levels lblock-1 .. nlev-1 alone (lblock = min(grid
     * levels, nlev)); keep them in its shared memory when they fit */
    A.smem_from = -1;
    const int lblock = grid_levels < A.nlev ? grid_levels : A.nlev;
    if (A.nlev > 0 && A.nlev >= grid_levels) {
        size_t bytes = 0;
        for (int i = lblock - 1; i < A.nlev; i++) bytes += level_smem_bytes<T>(A.L[i].n);
        if (bytes <= PCG_SMEM_MAX) A.smem_from = lblock - 1;
    }
    return off;
}

template <typename T>
static int run_pcg(World &w) {
    /* node indices fit 32 bits, and a row index 2^21 (div_small) */
    if (w.g.ni > 1024 || w.g.nj > 1024 || w.g.nk > 2048) return (int)cudaErrorInvalidValue;
    size_t es = sizeof(T);
    /* a plane of padding on both sides of each vector, so that reads of a
     * boundary node's neighbours need no clamp */
    const size_t pad = (((size_t)w.g.ni * w.g.nj * es + 255) / 256) * 256;
    size_t vec = ((w.nn * es + 255) / 256) * 256 + 2 * pad;
    size_t codeb = ((w.nn * sizeof(uint16_t) + 255) / 256) * 256;
    MgArgs<T> A;
    size_t mgb = mg_layout<T>(w, A, nullptr);
    /* float inner solves: the (hi, lo) pairs of phi and rho / eps0 */
    size_t dfb = sizeof(T) == sizeof(float) ? 2 * (((size_t)w.nn * sizeof(float2) + 255) / 256) * 256 : 0;
    size_t need = 8 * vec + codeb + mgb + dfb;
    if (w.pcg_bytes < need || w.pcg_elem != (int)es) {
        if (w.pcg_buf) {
            cudaStreamSynchronize(w.stream);
            cudaFree(w.pcg_buf);
        }
        w.pcg_buf = nullptr;
        w.pcg_bytes = 0;
        if (cudaMalloc(&w.pcg_buf, need) != cudaSuccess) return (int)cudaErrorMemoryAllocation;
        cudaMemsetAsync(w.pcg_buf, 0, need, w.stream);
        w.pcg_bytes = need;
        w.pcg_elem = (int)es;
        w.pcg_codes_valid = false;
    }
    char *base = (char *)w.pcg_buf;
    uint16_t *code = (uint16_t *)(base + 8 * vec);
    mg_layout<T>(w, A, base + 8 * vec + codeb);
    if (!w.pcg_codes_valid) {
        /* the sweeps rely on zeros off the unknowns, which just changed */
        cudaMemsetAsync(base, 0, 8 * vec, w.stream);
        k_pcg_codes<<<blocks_for(w.nn, 256), 256, 0, w.stream>>>(w.g, w.obj, code);
        w.nlaunch++;
        for (int l = 0; l < A.nlev; l++) {
            MgLevel<T> prev = l ? A.L[l - 1] : A.L[0];
            k_mg_setup<T><<<blocks_for(A.L[l].n, 256), 256, 0, w.stream>>>(w.g, code, prev, A.L[l], l == 0);
            w.nlaunch++;
        }
        if (A.dense) {
            const int n = A.dense_n;
            const int64_t nsq = (int64_t)n * n;
            double *M = (double *)((char *)A.dense + (nsq * sizeof(T) + 255) / 256 * 256);
            double *pub = (double *)((char *)M + (nsq * sizeof(double) + 255) / 256 * 256);
            double *diag0 = pub + (2 * (size_t)n * sizeof(double) + 255) / 256 * 256 / sizeof(double);
            int *ok = (int *)A.dense_ok;
            const int one = 1;
            cudaMemcpyAsync(ok, &one, sizeof(int), cudaMemcpyHostToDevice, w.stream);
            const MgLevel<T> &Lc = A.L[A.nlev - 1];
            k_dense_build<T><<<blocks_for(nsq, 256), 256, 0, w.stream>>>(Lc, M, diag0);
            /* one block per SM; its share of the rows (n <= 4096 of at least
             * 64 SMs) */
            const int gj_grid = w.sm_count < n ? w.sm_count : n;
            const size_t gj_bytes = (size_t)((n + gj_grid - 1) / gj_grid) * n * sizeof(double);
            if ((n + gj_grid - 1) / gj_grid > GJ_ROWS) return (int)cudaErrorInvalidValue;
            int nn_ = n, staged = gj_bytes <= GJ_SMEM_MAX;
            cudaFuncSetAttribute(k_gauss_jordan, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GJ_SMEM_MAX);
            void *gj_args[] = {&M, &nn_, &pub, &diag0, &ok, &staged};
            cudaLaunchCooperativeKernel((const void *)k_gauss_jordan, gj_grid, 1024, gj_args, staged ? gj_bytes : 0,
                                        w.stream);
            k_dense_store<T><<<blocks_for(nsq, 256), 256, 0, w.stream>>>(Lc, M, A.dense);
            w.nlaunch += 3;
        }
        w.pcg_codes_valid = true;
    }
    /* float: up to one node per thread, where both give a warp the same
     * nodes and so the same dot products; float64: up to 2^20 nodes
     * (102x102x100, just below: 21.2 ms a cold solve with 512 threads, 25.0
     * with 1024 and calls; 96x96x192, above: 13.8 and 14.4; 128x128x192: 29.8
     * either way) */
    bool small = sizeof(T) == sizeof(float) ? w.nn <= (int64_t)PCG_THREADS_SMALL * w.sm_count : w.nn <= 1 << 20;
    /* Solves of several worlds run beside each other when each takes a part
     * of the SMs, which a small grid hardly misses.  Float solves in ms, one
     * alone and per solve with three worlds in flight: 17x17x33 1.24 and 1.17
     * on every SM, 1.24 and 0.42 on a third; 24x24x48 1.22 and 1.17, on half
     * of them 1.31 and 0.64; 28x28x56 1.43 and 1.38, on a third with 1024
     * threads 1.64 and 0.55 (with a block per 1024 nodes: 2.16 and 0.73, 2.17
     * and 0.73, 2.30 and 0.80).  A float grid still has one node per thread,
     * see span.  Float64: 17x17x33 1.41 and 1.32, on half 1.39 and 0.67;
     * above 512 nodes an SM of a third, the SMs' float64 pipes count. */
    const int64_t third = w.sm_count / 3, half = w.sm_count / 2;
    int at_once = 1;
    if (w.nn <= PCG_THREADS_SMALL * third) {
        at_once = sizeof(T) == sizeof(float) ? 3 : 2;
    } else if (sizeof(T) == sizeof(float) && w.nn <= PCG_THREADS_SMALL * half) {
        at_once = 2;
    } else if (sizeof(T) == sizeof(float) && w.nn <= PCG_THREADS * third) {
        at_once = 3;
        small = false;
    }
    const int threads = small ? PCG_THREADS_SMALL : PCG_THREADS;
    const void *fn = (const void *)k_newton_pcg<T, PCG_THREADS, true>;
    if (small) fn = (const void *)k_newton_pcg<T, PCG_THREADS_SMALL, false>;
    /* between: the passes inlined (a cold solve of 128x128x127 nodes, just
     * below the line: 10.3 ms, 10.8 as calls; above it the calls are not yet
     * ahead: 128x128x129 10.5 and 11.0, 160x160x320 16.2 and 16.4; 256x256x512
     * sphere step: 25.7 ms inlined, 24.9 as calls) */
    if constexpr (sizeof(T) == sizeof(float))
        if (!small && w.nn <= 1 << 21) fn = (const void *)k_newton_pcg<T, PCG_THREADS, false>;
    size_t dyn = 0;
    if (A.smem_from >= 0)
        for (int i = A.smem_from; i < A.nlev; i++) dyn += level_smem_bytes<T>(A.L[i].n);
    /* the kernel's limit, not this world's need: another thread's world must
     * not lower it before the launch */
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PCG_SMEM_MAX);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, dyn);
    if (per_sm < 1) per_sm = 1;
    int64_t maxb = (int64_t)per_sm * (w.sm_count / at_once);
    /* every SM (of the share) as soon as there is a warp of nodes for each:
     * the phases of a small grid are bound by the instructions and float64
     * operations that one SM issues between two barriers, and a barrier of
     * 152 blocks costs what one of 16 does (1.29 and 1.30 us) */
    int64_t needb = (w.nn + 31) / 32;
    int grid = (int)(needb < maxb ? needb : maxb);
    if (grid > w.partial_slots / 4) grid = w.partial_slots / 4;
    if (w.solver_blocks > 0 && grid > w.solver_blocks) grid = w.solver_blocks;
    /* Half sweeps are merged where the lanes of the merged pass fill the grid
     * once, and in float the pass before a restriction up to twice: 33x29x65
     * float sphere run, 20 steps: 16.8 ms unmerged, 14.7 with one, 14.2 with
     * two; 64x64x128 float: 20.8, 19.7, 19.8 (the post pass of its first
     * level; 21.8 with all up to eight times).  The float64 pipe, which all
     * lanes' relaxations queue on, ends the gain earlier: 64x64x128 float64
     * solve 5.53 ms unmerged, 5.44 with one, 5.78 with two; 32x32x96
     * differentiable run 193, 180, 188. */
    const int64_t most = (int64_t)grid * threads, pre_most = sizeof(T) == sizeof(float) ? 2 * most : most;
    const int whole = A.grid_levels < A.nlev ? A.grid_levels : A.nlev; /* levels 0..whole-2 are the grid's */
    A.fine_pre = A.nlev > 0 && 16 * A.L[0].n <= pre_most;
    for (int l = 0; l < A.nlev; l++) {
        MgLevel<T> &L = A.L[l];
        L.merge = 0;
        if (l + 1 < whole) {
            if (16 * A.L[l + 1].n <= pre_most) L.merge |= MERGE_PRE;
            if (8 * (int64_t)((L.nx + 1) / 2) * L.ny * L.nz <= most) L.merge |= MERGE_POST;
        }
        if (!(L.merge & MERGE_POST)) L.f = L.e;
    }
    Geo g = w.g;
    double *phi = w.phi;
    const double *rho = w.rho;
    const int32_t *tg = w.target;
    const uint16_t *cc = code;
    double phi0 = w.phi0, te0 = w.te0, n0 = w.n0, nr_tol = w.nr_tol, pcg_tol = w.pcg_tol;
    int nr_max = w.nr_max, pcg_max = w.pcg_max;
    T *v[8];
    for (int i = 0; i < 8; i++) v[i] = (T *)(base + i * vec + pad);
    double *part = w.d_partials;
    SolveStatus *st = w.d_status;
    int *err = w.d_err;
    double *ly = w.lin_y;
    const double *lb = w.lin_b;
    int gs_max = w.gs_fallback ? w.max_it : 0;
    double gs_tol = w.tol;
    /* the pairs hold nn float2 each, the second array 256-byte aligned */
    float2 *dfp = dfb ? (float2 *)(base + 8 * vec + codeb + mgb) : nullptr;
    /* the predictor rides on the pairs' pass (the caller skipped k_predict) */
    double *pp = w.phi_prev;
    int predict = dfp && !ly ? w.predict_mode : 0;
    w.predict_mode = 0;
    /* the axis coefficients 1 / dh^2 rounded to T, as the kernel's cd */
    Coef3<T> ctp;
    for (int a = 0; a < 3; a++) ctp.c[a] = (T)(1.0 / (g.dh[a] * g.dh[a]));
    void *args[] = {&g,    &phi,  &rho,  &cc,   &tg,   &phi0, &te0, &n0,  &nr_max, &nr_tol, &pcg_max, &pcg_tol,
                    &v[0], &v[1], &v[2], &v[3], &v[4], &v[5], &v[6], &v[7], &A,  &part,   &st,      &err,
                    &ly,   &lb,   &gs_max, &gs_tol, &dfp,  &pp,   &predict, &ctp};
    w.nlaunch++;
    return (int)cudaLaunchCooperativeKernel(fn, grid, threads, args, dyn, w.stream);
}

int launch_newton_pcg(World &w, bool fp32) { return fp32 ? run_pcg<float>(w) : run_pcg<double>(w); }

/* y = J^-1 b on the unknowns, J the Jacobian of the Boltzmann problem at the
 * current phi (the adjoint solve: J is symmetric); y must be zero off the
 * unknowns.  Outer iterations until the update's RMS is below rel_tol times
 * the first one's. */
int launch_pcg_linear(World &w, bool fp32, const double *b, double *y, double rel_tol, int max_outer) {
    double keep_tol = w.nr_tol;
    int keep_max = w.nr_max;
    w.lin_b = b;
    w.lin_y = y;
    w.nr_tol = rel_tol;
    w.nr_max = max_outer;
    int rc = fp32 ? run_pcg<float>(w) : run_pcg<double>(w);
    w.lin_b = nullptr;
    w.lin_y = nullptr;
    w.nr_tol = keep_tol;
    w.nr_max = keep_max;
    return rc;
}

}  // namespace espic
