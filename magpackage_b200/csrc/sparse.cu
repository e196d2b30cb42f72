// Sparse linear algebra around the assembled CSR: y = A x, the reference's
// Dirichlet elimination, and a preconditioned conjugate-gradient solve that
// stands in for the reference's MUMPS call (LinearSolver.m:22-46) in the
// transient Newton driver.
//
// Every reduction runs over a fixed grid in a fixed order, so a solve is
// bitwise reproducible. The CG iterations run in one cooperative kernel, up to
// kPcgChunk iterations per launch; the host reads the solver's state once per
// launch.
#include <cstdint>
#include <new>

#include "common.cuh"
#include "sparse.cuh"

namespace mag {

namespace {

constexpr int kThreads = 256;
constexpr int kLanes = 8;  // lanes per CSR row in y = A x
constexpr int kPcgChunk = 256;

struct Csr {
    const int64_t *rp;
    const int32_t *ci;
    const double *v;
    int64_t n;
};

// Row i of A x with kLanes lanes; the value is valid in the group's lane 0.
__device__ __forceinline__ double row_dot(const Csr &A, int64_t i, int lane, const double *__restrict__ x) {
    double s = 0.0;
    if (i < A.n) {
        const int64_t a = A.rp[i], b = A.rp[i + 1];
        for (int64_t k = a + lane; k < b; k += kLanes) s = s + A.v[k] * __ldg(x + A.ci[k]);
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) s = s + __shfl_down_sync(0xffffffffu, s, o, kLanes);
    return s;
}

// Fixed-order block sum of one value per thread; result valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) t = t + sh[i];
    return t;
}

// Row loops over groups of kLanes threads run a block-uniform number of passes,
// so every lane reaches the shuffles in row_dot.
#define MAG_ROW_LOOP(n)                                                                                      \
    for (int64_t i = blockIdx.x * (int64_t)(kThreads / kLanes) + threadIdx.x / kLanes;                       \
         i - (threadIdx.x / kLanes) < (n); i += (int64_t)gridDim.x * (kThreads / kLanes))

__global__ void __launch_bounds__(kThreads) k_spmv(Csr A, const double *__restrict__ x, double *__restrict__ y) {
    const int lane = threadIdx.x % kLanes;
    MAG_ROW_LOOP(A.n) {
        double s = row_dot(A, i, lane, x);
        if (lane == 0 && i < A.n) y[i] = s;
    }
}

// M_free A M_free + M_fixed in place (BoundaryCondition.m:81-112), rhs[fixed] = 0.
__global__ void k_dirichlet(int64_t n, const int64_t *__restrict__ rp, const int32_t *__restrict__ ci,
                            double *__restrict__ v, const uint8_t *__restrict__ fixed, double *__restrict__ rhs) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bool fi = fixed[i] != 0;
    for (int64_t k = rp[i]; k < rp[i + 1]; k++) {
        const int64_t j = ci[k];
        if (fi) v[k] = j == i ? 1.0 : 0.0;
        else if (fixed[j]) v[k] = 0.0;
    }
    if (rhs && fi) rhs[i] = 0.0;
}

// ---- preconditioned CG --------------------------------------------------------------

struct PcgState {
    double rz, alpha, beta, rr, bb, tol2;
    int done;  // 0 running, 1 converged, 2 iteration limit, 3 breakdown (p.Ap <= 0 or not finite)
    int iters, max_iter;
};

struct PcgBufs {
    double *x, *r, *r2, *p, *q, *z, *dinv, *part;  // r, r2: before even and odd iterations
    PcgState *st;
    unsigned *bar;  // arrivals at the grid barriers; the word after it: a barrier gave up
    int nb;
};

// Auxiliary gradient space of the preconditioner: z = D^-1 r + G (D_N^-1 (G^T r)),
// G the (free edge x interior node) incidence of the discrete gradient and D_N the
// diagonal of G^T A G. The curl-curl part of A vanishes on gradients, so without this
// term the gradient modes are held only by the small regularisation and Jacobi-CG
// needs tens of thousands of iterations (a Hiptmair-type additive correction).
struct Aux {
    int64_t ni;
    const int64_t *g_rp;   // G   [n x ni]
    const int32_t *g_ci;
    const double *g_v;
    const int64_t *gt_rp;  // G^T [ni x n]
    const int32_t *gt_ci;
    const double *gt_v;
    const double *dn_inv;  // [ni]
    double *w;             // [ni] scratch
};

__global__ void __launch_bounds__(kThreads) k_aux_gt(Aux a, const double *__restrict__ r) {
    for (int64_t j = blockIdx.x * (int64_t)kThreads + threadIdx.x; j < a.ni; j += (int64_t)gridDim.x * kThreads) {
        double s = 0.0;
        for (int64_t k = a.gt_rp[j]; k < a.gt_rp[j + 1]; k++) s = s + a.gt_v[k] * r[a.gt_ci[k]];
        a.w[j] = a.dn_inv[j] * s;
    }
}

// Before the first iteration: z = D^-1 r (+ G w with the auxiliary space), p = z, and the
// partials of (r.z, r.r, b.b) with stride 3.
template <bool AUX>
__global__ void __launch_bounds__(kThreads) k_pcg_precond(int64_t n, PcgBufs B, Aux a, const double *__restrict__ b) {
    __shared__ double sh[kThreads / 32];
    double rz = 0.0, rr = 0.0, bb = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
        double r = B.r[i];
        double z = B.dinv[i] * r;
        if (AUX)
            for (int64_t k = a.g_rp[i]; k < a.g_rp[i + 1]; k++) z = z + a.g_v[k] * a.w[a.g_ci[k]];
        B.p[i] = z;
        bb = bb + b[i] * b[i];
        rz = rz + r * z;
        rr = rr + r * r;
    }
    double t0 = block_sum(rz, sh), t1 = block_sum(rr, sh), t2 = block_sum(bb, sh);
    if (threadIdx.x == 0) {
        B.part[3 * blockIdx.x] = t0;
        B.part[3 * blockIdx.x + 1] = t1;
        B.part[3 * blockIdx.x + 2] = t2;
    }
}

// x = x0, r = b - A x0, dinv = 1/diag(A) (1 where the diagonal is missing or not positive)
__global__ void __launch_bounds__(kThreads) k_pcg_setup(Csr A, const double *__restrict__ b,
                                                        const double *__restrict__ x0, PcgBufs B) {
    const int lane = threadIdx.x % kLanes;
    MAG_ROW_LOOP(A.n) {
        double s = row_dot(A, i, lane, x0);
        if (lane == 0 && i < A.n) {
            double d = 0.0;
            for (int64_t k = A.rp[i]; k < A.rp[i + 1]; k++)
                if (A.ci[k] == i) d = A.v[k];
            B.dinv[i] = d > 0.0 ? 1.0 / d : 1.0;
            B.r[i] = b[i] - s;
            B.x[i] = x0[i];
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_pcg_init_reduce(PcgBufs B, double rtol, int max_iter) {
    __shared__ double sh[kThreads / 32];
    double a = 0.0, c = 0.0, d = 0.0;
    for (int i = threadIdx.x; i < B.nb; i += kThreads) {
        a = a + B.part[3 * i];
        c = c + B.part[3 * i + 1];
        d = d + B.part[3 * i + 2];
    }
    double rz = block_sum(a, sh), rr = block_sum(c, sh), bb = block_sum(d, sh);
    if (threadIdx.x == 0) {
        PcgState s{};
        s.rz = rz;
        s.rr = rr;
        s.bb = bb;
        s.tol2 = rtol * rtol * bb;
        s.max_iter = max_iter;
        s.iters = 0;
        s.done = rr <= s.tol2 ? 1 : 0;
        *B.st = s;
    }
}

// ---- the iterations, one cooperative kernel ----------------------------------------
//
// A CG iteration at 233,700 unknowns moves 45 MB of matrix out of L2 (5 us) but ran 39 us as
// seven launches, two of them one-CTA reductions. Here one CTA per SM (1024 threads) keeps the
// solve and the phases of an iteration are separated by four grid barriers:
//   S  q = A p, partials of p.q                         | barrier
//   X  alpha; x += alpha p; r' = r - alpha q (the other of two r buffers, so that w can be
//      formed in the same phase from r and q of any row); w = D_N^-1 G^T r'   | barrier
//   Z  z = D^-1 r' + G w, partials of (r'.z, r'.r')     | barrier
//   P  beta; p = z + beta p                             | barrier
// Every CTA reduces the partials itself, in the same order, instead of waiting for one that
// does. The sums keep the order of kThreads-thread blocks on grids of grid_for(8 n) (rows) and
// grid_for(n) (vectors): a CTA holds kPcgSub such blocks. Measured on the E-core problem at
// 40 x 40 x 20 (233,700 unknowns, 15,600 iterations): 39 us an iteration as launches, 30 us so;
// of those the rows' product takes 13 us, each barrier 1.6 us, the rest 2 to 4 us each. The
// product is bound by the load/store unit (8 lanes a row; by count 60 of its cycles per warp and
// pass), not by latency or L2. With the column indices kept in shared memory, 485 ms for the
// problem's step against 487; with p gathered from shared memory by per-pass lists of distinct
// columns, one pass ahead 571 ms, three ahead by cp.async 581 ms.
constexpr int kPcgSub = 4;
constexpr int kPcgThreads = kPcgSub * kThreads;
constexpr int kPcgRows = 2;     // rows of one lane group in flight
constexpr int kPcgAhead = 3;    // entries per lane and row loaded ahead (8 lanes: rows of <= 24)
constexpr int kPcgKeep = 2;     // elements of r' and z a thread keeps between phases
constexpr int kPcgGtLanes = 4;  // lanes per row of G^T, and entries each loads ahead
constexpr int kPcgGtAhead = 4;
constexpr long long kPcgSpin = 1LL << 24;  // polls before a grid barrier gives up, unless set

struct PcgShared {
    double part[kPcgThreads / 32][2];
    double bc[3];
    int fail;
};

// Bounded grid barrier (all CTAs are co-resident: cooperative launch). target counts arrivals
// since the launch. The caller has passed a __syncthreads after its last global write, except
// for writes of warp 0, which the __syncwarp orders; the release and the acquire of thread 0
// carry the CTA's writes and reads with them. L1 is not read stale: the acquire invalidates it.
__device__ __forceinline__ bool pcg_barrier(PcgShared &S, unsigned *bar, unsigned &target, int *err, long long spin) {
    target += gridDim.x;
    if (threadIdx.x < 32) {
        __syncwarp();
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
            unsigned v = 0;
            long long i = 0;
            for (; i < spin; i++) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
                if ((int)(v - target) >= 0) break;
            }
            if (i == spin) {
                S.fail = 1;
                atomicExch(err, 1);
            }
        }
    }
    __syncthreads();
    return S.fail == 0;
}

// One value per thread and lane-group sum order of block_sum: warp trees, then the warps of a
// kThreads block in order. Leaves block b's sums in dst[2 b + c] (c < M).
template <int M>
__device__ __forceinline__ void pcg_block_sums(PcgShared &S, double v0, double v1, int block, int nblocks, double *dst) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v0 = v0 + __shfl_down_sync(0xffffffffu, v0, o);
        if (M > 1) v1 = v1 + __shfl_down_sync(0xffffffffu, v1, o);
    }
    if ((threadIdx.x & 31) == 0) {
        S.part[threadIdx.x >> 5][0] = v0;
        if (M > 1) S.part[threadIdx.x >> 5][1] = v1;
    }
    __syncthreads();
    if (threadIdx.x < kPcgSub * M) {
        const int sub = threadIdx.x / M, c = threadIdx.x % M, b = block + sub;
        if (b < nblocks) {
            double t = 0.0;
            for (int i = 0; i < kThreads / 32; i++) t = t + S.part[sub * (kThreads / 32) + i][c];
            dst[M * b + c] = t;
        }
    }
}

// The sums of n partials with stride M by the CTA's first kThreads threads (the order of a
// one-block reduction); valid in thread 0.
template <int M>
__device__ __forceinline__ void pcg_reduce(PcgShared &S, const double *part, int n, double out[2]) {
    double v[2] = {0.0, 0.0};
    if (threadIdx.x < kThreads) {
        for (int i = threadIdx.x; i < n; i += kThreads)
#pragma unroll
            for (int c = 0; c < M; c++) v[c] = v[c] + part[M * i + c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < M; c++) v[c] = v[c] + __shfl_down_sync(0xffffffffu, v[c], o);
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int c = 0; c < M; c++) S.part[threadIdx.x >> 5][c] = v[c];
    }
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int c = 0; c < M; c++) {
            out[c] = 0.0;
            for (int i = 0; i < kThreads / 32; i++) out[c] = out[c] + S.part[i][c];
        }
}

// Matrix entries are read once per iteration: loads that leave L1 to the gathers of p.
// Predicated, so that a group's loads are all in flight together.
__device__ __forceinline__ double ld_entry(bool in, const double *p) {
    double v = 0.0;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q ld.global.nc.L1::no_allocate.f64 %0, [%1];\n\t}"
        : "+d"(v)
        : "l"(p), "r"((int)in));
    return v;
}
__device__ __forceinline__ int ld_entry(bool in, const int32_t *p) {
    int v = -1;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q ld.global.nc.L1::no_allocate.s32 %0, [%1];\n\t}"
        : "+r"(v)
        : "l"(p), "r"((int)in));
    return v;
}

// r[0], r[1]: the residual before even and odd iterations. gs, gv: blocks of the row and of
// the vector sums. part: [gs] then [2 gv].
struct PcgLoop {
    Csr A;
    Aux aux;
    double *x, *r[2], *p, *q, *z;
    const double *dinv;
    double *part;
    PcgState *st;
    unsigned *bar;
    int *err;
    int gs, gv;
    long long spin;
};

// SPIN_SET: the barriers' poll limit is L.spin. (The default, a constant: as a value of L it took 1 %
// of the time.)
template <bool SPIN_SET>
__global__ void __launch_bounds__(kPcgThreads, 1) k_pcg_iterate(PcgLoop L) {
    __shared__ PcgShared S;
    const Csr &A = L.A;
    const int64_t n = A.n;
    const int sub = threadIdx.x / kThreads, ltid = threadIdx.x % kThreads, lane = ltid % kLanes;
    const int b0 = blockIdx.x * kPcgSub, vb = b0 + sub;
    const int64_t vstep = (int64_t)L.gv * kThreads, vfirst = vb < L.gv ? (int64_t)vb * kThreads + ltid : n;
    const int64_t rstep = (int64_t)L.gs * (kThreads / kLanes);
    const int64_t rfirst = (int64_t)vb * (kThreads / kLanes) + ltid / kLanes;
    double *part_rz = L.part + L.gs;
    double rz = L.st->rz, rr = L.st->rr, al = L.st->alpha, be = L.st->beta;
    const double tol2 = L.st->tol2;
    const int max_iter = L.st->max_iter;
    int done = L.st->done, iters = L.st->iters;
    unsigned target = 0;
    if (threadIdx.x == 0) S.fail = 0;
    __syncthreads();
    for (int it = 0; it < kPcgChunk && !done; it++) {
        // S: rows of this group, kPcgRows at a time, in ascending order
        double acc = 0.0;
        if (vb < L.gs)
            // (a block-uniform number of passes: every lane reaches the shuffles)
            for (int64_t i0 = rfirst; i0 - ltid / kLanes < n; i0 += kPcgRows * rstep) {
                int64_t ka[kPcgRows], kb[kPcgRows];
#pragma unroll
                for (int u = 0; u < kPcgRows; u++) {
                    const int64_t i = i0 + u * rstep;
                    ka[u] = i < n ? __ldg(A.rp + i) + lane : 0;
                    kb[u] = i < n ? __ldg(A.rp + i + 1) : 0;
                }
                double v[kPcgRows][kPcgAhead];
                int c[kPcgRows][kPcgAhead];
#pragma unroll
                for (int u = 0; u < kPcgRows; u++)
#pragma unroll
                    for (int j = 0; j < kPcgAhead; j++) {
                        const int64_t k = ka[u] + j * kLanes;
                        c[u][j] = ld_entry(k < kb[u], A.ci + k);  // -1: no entry
                        v[u][j] = ld_entry(k < kb[u], A.v + k);
                    }
                double s[kPcgRows];
#pragma unroll
                for (int u = 0; u < kPcgRows; u++) {
                    s[u] = 0.0;
#pragma unroll
                    for (int j = 0; j < kPcgAhead; j++)
                        if (c[u][j] >= 0) s[u] = fma(v[u][j], L.p[c[u][j]], s[u]);
                    for (int64_t k = ka[u] + kPcgAhead * kLanes; k < kb[u]; k += kLanes)
                        s[u] = fma(A.v[k], L.p[A.ci[k]], s[u]);
                }
#pragma unroll
                for (int o = kLanes / 2; o > 0; o >>= 1)
#pragma unroll
                    for (int u = 0; u < kPcgRows; u++) s[u] = s[u] + __shfl_down_sync(0xffffffffu, s[u], o, kLanes);
                if (lane == 0)
#pragma unroll
                    for (int u = 0; u < kPcgRows; u++) {
                        const int64_t i = i0 + u * rstep;
                        if (i < n) {
                            L.q[i] = s[u];
                            acc = fma(L.p[i], s[u], acc);
                        }
                    }
            }
        pcg_block_sums<1>(S, acc, 0.0, b0, L.gs, L.part);
        if (!pcg_barrier(S, L.bar, target, L.err, SPIN_SET ? L.spin : kPcgSpin)) return;
        // alpha
        {
            double pq[2];
            pcg_reduce<1>(S, L.part, L.gs, pq);
            if (threadIdx.x == 0) {
                S.bc[0] = pq[0];
                S.bc[1] = rz / pq[0];
            }
            __syncthreads();
            if (!(S.bc[0] > 0.0) || !isfinite(S.bc[0])) {
                done = 3;
                break;
            }
            al = S.bc[1];
        }
        // X
        const double *rin = L.r[iters & 1];
        double *rout = L.r[(iters + 1) & 1];
        double rk[kPcgKeep], zk[kPcgKeep];  // this thread's first elements of r' and z
#pragma unroll
        for (int m = 0; m < kPcgKeep; m++) {
            const int64_t i = vfirst + m * vstep;
            rk[m] = 0.0;
            if (i < n) {
                L.x[i] = fma(al, L.p[i], L.x[i]);
                rk[m] = fma(-al, L.q[i], rin[i]);
                rout[i] = rk[m];
            }
        }
        for (int64_t i = vfirst + kPcgKeep * vstep; i < n; i += vstep) {
            L.x[i] = fma(al, L.p[i], L.x[i]);
            rout[i] = fma(-al, L.q[i], rin[i]);
        }
        if (L.aux.ni > 0) {
            // rows of G^T, a contiguous share per CTA, kPcgGtLanes lanes per row: the lanes
            // load a row's entries side by side, its first lane adds them in row order
            const Aux &a = L.aux;
            const int64_t share = (a.ni + gridDim.x - 1) / gridDim.x, j0 = share * blockIdx.x;
            const int64_t j1 = j0 + share < a.ni ? j0 + share : a.ni;
            const int gl = threadIdx.x % kPcgGtLanes;
            for (int64_t jb = j0; jb < j1; jb += kPcgThreads / kPcgGtLanes) {
                const int64_t j = jb + threadIdx.x / kPcgGtLanes;
                const int64_t k0 = j < j1 ? __ldg(a.gt_rp + j) : 0, k1 = j < j1 ? __ldg(a.gt_rp + j + 1) : 0;
                double s = 0.0;
                for (int64_t kc = k0; __any_sync(0xffffffffu, kc < k1); kc += kPcgGtLanes * kPcgGtAhead) {
                    double v[kPcgGtAhead], t[kPcgGtAhead];
                    int c[kPcgGtAhead];
#pragma unroll
                    for (int m = 0; m < kPcgGtAhead; m++) {
                        const int64_t k = kc + m * kPcgGtLanes + gl;
                        c[m] = ld_entry(k < k1, a.gt_ci + k);
                        v[m] = ld_entry(k < k1, a.gt_v + k);
                    }
#pragma unroll
                    for (int m = 0; m < kPcgGtAhead; m++) t[m] = c[m] >= 0 ? fma(-al, L.q[c[m]], rin[c[m]]) : 0.0;
#pragma unroll
                    for (int m = 0; m < kPcgGtAhead; m++)
#pragma unroll
                        for (int l = 0; l < kPcgGtLanes; l++) {
                            const double vv = __shfl_sync(0xffffffffu, v[m], l, kPcgGtLanes);
                            const double tt = __shfl_sync(0xffffffffu, t[m], l, kPcgGtLanes);
                            if (kc + m * kPcgGtLanes + l < k1) s = fma(vv, tt, s);
                        }
                }
                if (gl == 0 && j < j1) a.w[j] = __ldg(a.dn_inv + j) * s;
            }
            __syncthreads();
            if (!pcg_barrier(S, L.bar, target, L.err, SPIN_SET ? L.spin : kPcgSpin)) return;
        }
        // Z (each thread reads its own r', and w of any node)
        double zr = 0.0, zz = 0.0;
        auto precond = [&](int64_t i, double r) {
            double z = L.dinv[i] * r;
            if (L.aux.ni > 0) {
                const int64_t k1 = __ldg(L.aux.g_rp + i + 1);
                for (int64_t k = __ldg(L.aux.g_rp + i); k < k1; k++)
                    z = fma(__ldg(L.aux.g_v + k), L.aux.w[__ldg(L.aux.g_ci + k)], z);
            }
            zr = fma(r, z, zr);
            zz = fma(r, r, zz);
            return z;
        };
#pragma unroll
        for (int m = 0; m < kPcgKeep; m++) {
            const int64_t i = vfirst + m * vstep;
            zk[m] = i < n ? precond(i, rk[m]) : 0.0;
        }
        for (int64_t i = vfirst + kPcgKeep * vstep; i < n; i += vstep) L.z[i] = precond(i, rout[i]);
        pcg_block_sums<2>(S, zr, zz, b0, L.gv, part_rz);
        if (!pcg_barrier(S, L.bar, target, L.err, SPIN_SET ? L.spin : kPcgSpin)) return;
        // beta and the stopping test
        {
            double t[2];
            pcg_reduce<2>(S, part_rz, L.gv, t);
            if (threadIdx.x == 0) {
                S.bc[0] = t[0];
                S.bc[1] = t[1];
                S.bc[2] = t[0] / rz;
            }
            __syncthreads();
            iters++;
            rr = S.bc[1];
            be = S.bc[2];
            rz = S.bc[0];
            if (rr <= tol2) done = 1;
            else if (!isfinite(rr)) done = 3;
            else if (iters >= max_iter) done = 2;
        }
        if (done) break;
        // P
#pragma unroll
        for (int m = 0; m < kPcgKeep; m++) {
            const int64_t i = vfirst + m * vstep;
            if (i < n) L.p[i] = fma(be, L.p[i], zk[m]);
        }
        for (int64_t i = vfirst + kPcgKeep * vstep; i < n; i += vstep) L.p[i] = fma(be, L.p[i], L.z[i]);
        __syncthreads();
        if (!pcg_barrier(S, L.bar, target, L.err, SPIN_SET ? L.spin : kPcgSpin)) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        PcgState &st = *L.st;
        st.rz = rz;
        st.rr = rr;
        st.alpha = al;
        st.beta = be;
        st.iters = iters;
        st.done = done;
    }
}

int grid_for(int64_t threads) {
    static int nsm = 0;
    if (!nsm) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (nsm <= 0) nsm = 1;
    }
    int64_t want = (threads + kThreads - 1) / kThreads;
    int64_t cap = 4LL * nsm;
    return (int)(want < 1 ? 1 : (want < cap ? want : cap));
}

}  // namespace

struct PcgSolver {
    int64_t n = 0;
    PcgBufs B{};
    Aux aux{};
    double *w = nullptr;
    int64_t w_cap = 0;
    cudaStream_t s = nullptr;
    PcgState *h_st = nullptr;  // pinned; the barrier words after it
    long long spin = kPcgSpin;
};

int csr_spmv(int64_t n, const int64_t *rp, const int32_t *ci, const double *v, const double *x, double *y,
             cudaStream_t s) {
    Csr A{rp, ci, v, n};
    k_spmv<<<grid_for(n * kLanes), kThreads, 0, s>>>(A, x, y);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}

int csr_dirichlet(int64_t n, const int64_t *rp, const int32_t *ci, double *v, const uint8_t *fixed, double *rhs,
                  cudaStream_t s) {
    k_dirichlet<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, rp, ci, v, fixed, rhs);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}

int pcg_create(int64_t n, PcgSolver **out) {
    *out = nullptr;
    PcgSolver *P = new (std::nothrow) PcgSolver();
    if (!P) return MAG_E_NOMEM;
    P->n = n;
    const int gs = grid_for(n * kLanes), gv = grid_for(n);
    P->B.nb = gs > gv ? gs : gv;
    size_t vb = (size_t)n * sizeof(double);
    double **bufs[] = {&P->B.x, &P->B.r, &P->B.r2, &P->B.p, &P->B.q, &P->B.z, &P->B.dinv};
    bool ok = true;
    for (double **b : bufs) ok = ok && cudaMalloc(b, vb) == cudaSuccess;
    ok = ok && cudaMalloc(&P->B.part, (size_t)3 * P->B.nb * sizeof(double)) == cudaSuccess;
    ok = ok && cudaMalloc(&P->B.st, sizeof(PcgState) + 2 * sizeof(unsigned)) == cudaSuccess;
    ok = ok && cudaMallocHost(&P->h_st, sizeof(PcgState) + 2 * sizeof(unsigned)) == cudaSuccess;
    if (ok) P->B.bar = reinterpret_cast<unsigned *>(P->B.st + 1);
    ok = ok && cudaStreamCreateWithFlags(&P->s, cudaStreamNonBlocking) == cudaSuccess;
    if (!ok) {
        pcg_destroy(P);
        return MAG_E_NOMEM;
    }
    *out = P;
    return MAG_OK;
}

void pcg_destroy(PcgSolver *P) {
    if (!P) return;
    if (P->s) cudaStreamSynchronize(P->s);
    double *bufs[] = {P->B.x, P->B.r, P->B.r2, P->B.p, P->B.q, P->B.z, P->B.dinv, P->B.part, P->w};
    for (double *b : bufs)
        if (b) cudaFree(b);
    if (P->B.st) cudaFree(P->B.st);
    if (P->h_st) cudaFreeHost(P->h_st);
    if (P->s) cudaStreamDestroy(P->s);
    delete P;
}

void pcg_set_spin_limit(PcgSolver *P, int64_t polls) { P->spin = polls > 0 ? (long long)polls : kPcgSpin; }

int pcg_set_aux(PcgSolver *P, int64_t ni, const int64_t *g_rp, const int32_t *g_ci, const double *g_v,
                const int64_t *gt_rp, const int32_t *gt_ci, const double *gt_v, const double *dn_inv) {
    if (ni <= 0) {
        P->aux = Aux{};
        return MAG_OK;
    }
    if (ni > P->w_cap) {
        if (P->w) cudaFree(P->w);
        P->w = nullptr;
        P->w_cap = 0;
        if (cudaMalloc(&P->w, (size_t)ni * sizeof(double)) != cudaSuccess) {
            P->aux = Aux{};
            return MAG_E_NOMEM;
        }
        P->w_cap = ni;
    }
    P->aux = Aux{ni, g_rp, g_ci, g_v, gt_rp, gt_ci, gt_v, dn_inv, P->w};
    return MAG_OK;
}

namespace {

PcgBufs bufs_with(const PcgSolver *P, int nb) {
    PcgBufs b = P->B;
    b.nb = nb;
    return b;
}

// Up to kPcgChunk iterations; the state says whether more are needed.
cudaError_t launch_iterations(PcgSolver *P, const Csr &A, cudaStream_t s) {
    const PcgBufs &B = P->B;
    const int gs = grid_for(P->n * kLanes), gv = grid_for(P->n);
    PcgLoop L{A, P->aux, B.x, {B.r, B.r2}, B.p, B.q, B.z, B.dinv, B.part, B.st, B.bar,
              reinterpret_cast<int *>(B.bar + 1), gs, gv, P->spin};
    cudaError_t e = cudaMemsetAsync(B.bar, 0, 2 * sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    void *args[] = {&L};
    const auto kern = P->spin == kPcgSpin ? k_pcg_iterate<false> : k_pcg_iterate<true>;
    return cudaLaunchCooperativeKernel((const void *)kern, dim3((gs + kPcgSub - 1) / kPcgSub),
                                       dim3(kPcgThreads), args, 0, s);
}

}  // namespace

int pcg_solve(PcgSolver *P, const int64_t *rp, const int32_t *ci, const double *v, const double *b, double *x,
              double rtol, int max_iter, int *iters, double *relres, int *status, cudaStream_t caller) {
    Csr A{rp, ci, v, P->n};
    cudaStream_t s = P->s;
    cudaEvent_t ev;
    MAG_CUDA_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    cudaEventRecord(ev, caller);
    cudaStreamWaitEvent(s, ev, 0);
    const int gs = grid_for(P->n * kLanes), gv = grid_for(P->n);
    const PcgBufs Bv = bufs_with(P, gv);
    k_pcg_setup<<<gs, kThreads, 0, s>>>(A, b, x, P->B);
    if (P->aux.ni > 0) {
        k_aux_gt<<<grid_for(P->aux.ni), kThreads, 0, s>>>(P->aux, P->B.r);
        k_pcg_precond<true><<<gv, kThreads, 0, s>>>(P->n, Bv, P->aux, b);
    } else {
        k_pcg_precond<false><<<gv, kThreads, 0, s>>>(P->n, Bv, P->aux, b);
    }
    k_pcg_init_reduce<<<1, kThreads, 0, s>>>(Bv, rtol, max_iter);
    cudaError_t le = cudaPeekAtLastError();
    if (le != cudaSuccess) {
        cudaEventDestroy(ev);
        set_error("pcg setup launch: %s", cudaGetErrorString(le));
        return MAG_E_CUDA;
    }
    const size_t state_bytes = sizeof(PcgState) + 2 * sizeof(unsigned);
    bool gave_up = false;
    for (bool first = true;; first = false) {
        cudaError_t e = first ? cudaSuccess : launch_iterations(P, A, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(P->h_st, P->B.st, state_bytes, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            cudaEventDestroy(ev);
            set_error("pcg iterations: %s", cudaGetErrorString(e));
            return MAG_E_CUDA;
        }
        gave_up = !first && reinterpret_cast<const unsigned *>(P->h_st + 1)[1] != 0;
        if (P->h_st->done || gave_up) break;
    }
    if (gave_up) {
        cudaEventDestroy(ev);
        set_error("pcg: a grid barrier gave up waiting");
        return MAG_E_TIMEOUT;
    }
    MAG_CUDA_TRY(cudaMemcpyAsync(x, P->B.x, (size_t)P->n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    cudaEventRecord(ev, s);
    cudaStreamWaitEvent(caller, ev, 0);
    cudaEventDestroy(ev);
    const PcgState &h = *P->h_st;
    if (iters) *iters = h.iters;
    if (relres) *relres = h.bb > 0 ? sqrt(h.rr / h.bb) : sqrt(h.rr);
    if (status) *status = h.done;
    if (h.done == 3) {
        set_error("pcg breakdown after %d iterations (matrix not positive definite on the Krylov space)", h.iters);
        return MAG_E_GEOMETRY;
    }
    return MAG_OK;
}

}  // namespace mag
