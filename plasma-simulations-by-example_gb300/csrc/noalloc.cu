/*
 * noalloc.cu -- espic_deposit_noalloc: the fixed-point CIC charge deposit of
 * Species::computeNumberDensity for callers that may not allocate device
 * memory (see include/espic.h for who they are).
 *
 * The deposit needs an int64 accumulator the size of the node grid.  Here it
 * is a file-scope __device__ array of ESPIC_NOALLOC_MAX_NODES entries
 * (8 MiB), so the call itself allocates nothing: every GPU that loads
 * libespic holds those 8 MiB until the process exits.  Host code may not
 * hand the array's name to a kernel (on the host it is only a stand-in), so
 * the device address is fetched with cudaGetSymbolAddress once per device,
 * with that device current, on the first call made on it; the kernels
 * receive that address.  All calls share the one array and leave their sums
 * in it, so each call clears the part it uses first, and calls that overlap
 * on the GPU (different streams, or different host threads on one device)
 * race on it.  Particles the fixed-point sum cannot take (a weight beyond
 * weight_bound, a non-finite position) are skipped and reported in the
 * caller's flag word, the counterpart of the allocating path's
 * ESPIC_ERR_FIXED and ESPIC_ERR_NONFINITE.
 *
 * The arithmetic is the float64 deposit of k_fp64.cu: corner weights
 * value*(1-di)*(1-dj)*(1-dk) in the reference's corner order (Field_::scatter,
 * ch2/Field.h:164-183), each rounded once to a count of 1/fx, then
 * den = count/fx / node_volume (World::computeNodeVolumes,
 * ch2/World.cpp:58-69).  Built with -fmad=false like k_fp64.cu.
 */
#include <math.h>
#include <stdio.h>

#include <mutex>

#include "cic64.h"
#include "espic.h"

namespace {

__device__ __align__(256) unsigned long long g_noalloc_acc[ESPIC_NOALLOC_MAX_NODES];

struct NaGeo {
    int ni, nj, nk;
    double x0[3], dh[3], rdh[3]; /* rdh = RN(1 / dh) */
    double V, rV;                /* an inner node's volume dh dh dh and RN(1 / V) */
};

__device__ __forceinline__ int na_clamp(int i, int n) { return i < 0 ? 0 : (i > n - 2 ? n - 2 : i); }

/* The three kernels of a call are launched so that each may start while the
 * one before drains (programmatic dependent launch): the waits hide the
 * launches and, in the deposit, the particle's arithmetic.  next_may_start
 * lets the next kernel be scheduled once every block of this one runs;
 * wait_for_previous returns when the kernel before has finished and its
 * writes are visible. */
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__global__ void __launch_bounds__(256) k_na_clear(unsigned long long *acc, uint32_t nn, int *flags) {
    next_may_start();
    const uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u < nn) acc[u] = 0ull;
    if (u == 0 && flags) *flags = 0;
}

/* A particle whose position is not finite, or whose weight is not within
 * [-weight_bound, weight_bound] (so that its corner counts could wrap the
 * int64 sums), deposits nothing and sets a bit of the flags.  Bound by the
 * float64 pipe and the integer work of scatter8 alike: float64 are the three
 * differences, nine operations of the quotients by dh and seven products (6M
 * particles on 97x89x117 nodes, the whole call: 869 us with divisions and a
 * conversion per weight, 401 us now). */
__global__ void __launch_bounds__(256) k_na_deposit(NaGeo g, const double *__restrict__ P, int64_t stride, int64_t n,
                                                    double fx, double weight_bound, unsigned long long *acc,
                                                    int *flags) {
    next_may_start();
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int nn3[3] = {g.ni, g.nj, g.nk};
    double off[3] = {0, 0, 0}, rest[3] = {1, 1, 1}, value = 0;
    int c[3] = {0, 0, 0};
    bool unit = true, finite = true, in_range = true;
    const bool there = p < n;
    if (there) {
        double lc[3];
        for (int d = 0; d < 3; d++) lc[d] = espic::div_rcp(P[d * stride + p] - g.x0[d], g.dh[d], g.rdh[d]);
        value = P[6 * stride + p];
        finite = espic::finite_bits(lc[0]) && espic::finite_bits(lc[1]) && espic::finite_bits(lc[2]);
        /* false for NaN, whose key lies beyond infinity's */
        in_range = espic::order_key(fabs(value)) <= espic::order_key(weight_bound);
        if (finite && in_range)
#pragma unroll
            for (int d = 0; d < 3; d++)
                if (!espic::cell_of(lc[d], nn3[d], c[d], off[d], rest[d])) {
                    c[d] = na_clamp((int)lc[d], nn3[d]);
                    off[d] = lc[d] - c[d];
                    rest[d] = 1 - off[d];
                    unit = false;
                }
    }
    wait_for_previous();
    if (!(finite && in_range) && flags)
        atomicOr(flags, (finite ? 0 : ESPIC_NOALLOC_NONFINITE) | (in_range ? 0 : ESPIC_NOALLOC_RANGE));
    const int64_t sy = g.ni, sz = (int64_t)g.ni * g.nj;
    espic::scatter8(acc, (uint32_t)(c[2] * sz + c[1] * sy + c[0]), sy, sz, off, rest, value, fx,
                    unit, there && finite && in_range);
}

__global__ void __launch_bounds__(256) k_na_density(NaGeo g, const unsigned long long *acc, double unit, double *den) {
    wait_for_previous();
    const uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= (uint32_t)(g.ni * g.nj * g.nk)) return;
    const uint32_t row = u / (uint32_t)g.ni;
    const int i = (int)(u - row * (uint32_t)g.ni), j = (int)(row % (uint32_t)g.nj), k = (int)(row / (uint32_t)g.nj);
    /* each face halves the volume: d / (V / 2) = 2 d / V exactly */
    double s = unit;
    if (i == 0 || i == g.ni - 1) s *= 2;
    if (j == 0 || j == g.nj - 1) s *= 2;
    if (k == 0 || k == g.nk - 1) s *= 2;
    const double d = __ll2double_rn((long long)acc[u]) * s;
    den[u] = g.rV != 0 ? espic::div_rcp(d, g.V, g.rV) : (g.V != 0 ? d / g.V : 0.0);
}

std::mutex g_na_mutex;
constexpr int NA_MAX_DEVICES = 64;
void *g_na_addr[NA_MAX_DEVICES] = {nullptr};

}  // namespace

int espic_internal_fail(int code, const char *msg);

/* The device address of g_noalloc_acc for the current device, looked up once
 * per device with that device current. */
static int na_scratch(unsigned long long **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return espic_internal_fail(ESPIC_ERR_CUDA, "espic_deposit_noalloc: no current device");
    if (dev < 0 || dev >= NA_MAX_DEVICES)
        return espic_internal_fail(ESPIC_ERR_ARG, "espic_deposit_noalloc: device index out of range");
    std::lock_guard<std::mutex> lock(g_na_mutex);
    if (!g_na_addr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_acc);
        if (e != cudaSuccess || !p) {
            char buf[256];
            snprintf(buf, sizeof buf, "espic_deposit_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
            return espic_internal_fail(ESPIC_ERR_CUDA, buf);
        }
        g_na_addr[dev] = p;
    }
    *out = (unsigned long long *)g_na_addr[dev];
    return ESPIC_OK;
}

/* a launch that may overlap the tail of the kernel before it on the stream
 * (the kernel itself waits for its results) */
template <class... P, class... A>
static cudaError_t launch_early(unsigned blocks, unsigned threads, cudaStream_t st, void (*fn)(P...), A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.stream = st;
    cudaLaunchAttribute early;
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &early;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, args...);
}

extern "C" int espic_deposit_noalloc(const double *d_P, int64_t stride, int64_t n, int ni, int nj, int nk,
                                     const double x0[3], const double xm[3], double weight_bound, double *d_den,
                                     int *d_flags, void *stream) {
    if (!x0 || !xm || !d_den || (n > 0 && !d_P))
        return espic_internal_fail(ESPIC_ERR_ARG, "espic_deposit_noalloc: null argument");
    if (ni < 3 || nj < 3 || nk < 3)
        return espic_internal_fail(ESPIC_ERR_ARG, "espic_deposit_noalloc: need at least 3 nodes per axis");
    /* bound each factor before multiplying, so that no product can wrap */
    if (ni > ESPIC_NOALLOC_MAX_NODES || nj > ESPIC_NOALLOC_MAX_NODES || nk > ESPIC_NOALLOC_MAX_NODES ||
        (int64_t)ni * nj > ESPIC_NOALLOC_MAX_NODES / nk) {
        char buf[240];
        snprintf(buf, sizeof buf,
                 "espic_deposit_noalloc: a %d x %d x %d grid exceeds its fixed scratch of %d nodes; use "
                 "espic_deposit",
                 ni, nj, nk, ESPIC_NOALLOC_MAX_NODES);
        return espic_internal_fail(ESPIC_ERR_ARG, buf);
    }
    const int64_t nn = (int64_t)ni * nj * nk;
    if (n < 0 || stride < n) return espic_internal_fail(ESPIC_ERR_ARG, "espic_deposit_noalloc: bad particle count");
    if (!(weight_bound > 0)) return espic_internal_fail(ESPIC_ERR_ARG, "espic_deposit_noalloc: weight_bound <= 0");
    for (int d = 0; d < 3; d++)
        if (!(xm[d] > x0[d])) return espic_internal_fail(ESPIC_ERR_ARG, "espic_deposit_noalloc: xm <= x0");
    unsigned long long *acc = nullptr;
    int rc = na_scratch(&acc);
    if (rc != ESPIC_OK) return rc;
    NaGeo g;
    g.ni = ni;
    g.nj = nj;
    g.nk = nk;
    int nn3[3] = {ni, nj, nk};
    for (int d = 0; d < 3; d++) {
        g.x0[d] = x0[d];
        g.dh[d] = (xm[d] - x0[d]) / (nn3[d] - 1);
        g.rdh[d] = 1.0 / g.dh[d];
    }
    g.V = g.dh[0] * g.dh[1] * g.dh[2];
    /* 0: a volume or reciprocal outside the range where the quotient by the
     * reciprocal is exact */
    g.rV = g.V > 1e-280 && g.V < 1e280 ? 1.0 / g.V : 0.0;
    /* the fixed-point scale of a species of capacity n with this weight bound */
    int64_t cap = n < 1 ? 1 : n;
    double lim = ldexp(1.0, 62) / ((double)cap * weight_bound);
    int ex;
    frexp(lim, &ex);
    int S = ex - 1 > 52 ? 52 : ex - 1;
    double fx = ldexp(1.0, S);
    cudaStream_t st = (cudaStream_t)stream;
    /* small blocks for few particles (4096 an SM of 152): an even share of
     * float64 work per SM */
    const unsigned nt = n < 600000 ? 64 : 256;
    k_na_clear<<<(unsigned)((nn + 255) / 256), 256, 0, st>>>(acc, (uint32_t)nn, d_flags);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && n > 0)
        e = launch_early((unsigned)((n + nt - 1) / nt), nt, st, k_na_deposit, g, d_P, stride, n, fx, weight_bound, acc, d_flags);
    if (e == cudaSuccess)
        e = launch_early((unsigned)((nn + 255) / 256), 256, st, k_na_density, g, (const unsigned long long *)acc, 1.0 / fx,
                         d_den);
    if (e != cudaSuccess) {
        char buf[200];
        snprintf(buf, sizeof buf, "espic_deposit_noalloc: launch: %s", cudaGetErrorString(e));
        return espic_internal_fail(ESPIC_ERR_CUDA, buf);
    }
    return ESPIC_OK;
}
