// Harmonic-balance (HBFEM) assembly, FP64 (sm_100a).
//
// Element phase restates assemble_hbfem_kernel_mex.cpp:108-226
// operation for operation: the signed harmonic edge values, per quadrature point the
// physical curls, per time sample t the edge values A(t) = sum_h (Re A_h Re D(t,h) -
// Im A_h Im D(t,h)), B(t), nu(|B(t)|^2) from the B-H table (with the coefficient offsets
// the reference gateway forgets to set), H = nu B, and the harmonic residual
// R_h += w (C_i . H) P(h,t); the Jacobian block is w nu_dc C_r . C_c with nu_dc the
// time average of nu. Two kernels: k_hbfem_std, six threads per element, for the standard curl
// table with equal weights, and k_hbfem_elems, one thread per element, for any table, weights and
// sample count. Per (element, local row) they write the 2K residual entries into a workspace that
// k_rows_reduce_harm sums per CSR row, in ascending element order, as MATLAB's sparse() does with
// the gateway's triplets. The DC block is one tile assembly from k_hbfem_std's nu_dc, or block rows
// in the common element scratch (reduced by k_rows_reduce).
#include "assemble.cuh"
#include "common.cuh"
#include "element.cuh"
#include "hbfem.cuh"

namespace mag {

namespace {

using namespace elem;

struct HbArgs {
    ElemData m;
    const double *sr, *si;  // [K][ndof] harmonic solution (si may be NULL)
    const double *dr, *di;  // [K][N]: D(t, h) at h * N + t (di may be NULL)
    const double *pr, *pi;  // [N][K]: P(h, t) at t * K + h (pi may be NULL)
    int K, N;
    int64_t ndof;
    QuadParams qp;
    MaterialParams mp;
    double *scratch;  // [Ne][6][kScratchStride] block rows (NULL: residual only)
    double *rscr;     // [Ne][6][2K] residual entries (re | im)
    double *nu_dc;    // [Ne] time-averaged reluctivity (NULL: not wanted; k_hbfem_std only)
};

// Index of (r, c), r <= c, in the upper triangle of a 6 x 6 block stored row by row.
__host__ __device__ constexpr int kb_at(int r, int c) { return r * 6 - r * (r - 1) / 2 + (c - r); }

// General form, one thread per element: any curl table, any weights, any sample count. KC: the
// harmonic count as a compile-time constant, so that the harmonic loops unroll and their arrays are
// registers (up to 255, two CTAs per SM); 0: A.K at run time, arrays sized for kMaxHarm in local
// memory. Measured, ms, residual and DC block of 384,000 elements with run-time / constant count: 3
// harmonics, 256 samples 24.4 / 11.0, 32 samples with unequal weights 3.25 / 1.89; 1 harmonic, 256
// samples 9.03 / 4.68.
template <bool CALCJ, int KC>
__global__ void __launch_bounds__(128, KC > 0 ? 2 : 3) k_hbfem_elems(HbArgs A) {
    constexpr int KA = KC > 0 ? KC : kMaxHarm;
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= A.m.ne) return;
    const int K = KC > 0 ? KC : A.K, N = A.N;
    const int4 tt = A.m.tet[e];
    int d[6];
    load_dofs(A.m.dofs, e, d);
    const unsigned sb = A.m.signbits ? A.m.signbits[e] : derived_signs(tt);
    const int tag = A.m.tags[e];
    Geo g;
    geometry(A.m.xyz, tt, g);
    double ar[6][KA], ai[6][KA];
    for (int k = 0; k < 6; k++)
        for (int h = 0; h < K; h++) {
            const bool has = d[k] >= 0;
            const double xr = has ? __ldg(A.sr + h * A.ndof + d[k]) : 0.0;
            const double xi = has && A.si ? __ldg(A.si + h * A.ndof + d[k]) : 0.0;
            ar[k][h] = flip(xr, (sb >> k) & 1);
            ai[k][h] = flip(xi, (sb >> k) & 1);
        }
    double rr[6][KA], ri[6][KA];
    for (int k = 0; k < 6; k++)
        for (int h = 0; h < K; h++) {
            rr[k][h] = 0.0;
            ri[k][h] = 0.0;
        }
    // The DC block is symmetric bit for bit (C_r . C_c and C_c . C_r are the same products
    // summed in the same order), so only its upper triangle is accumulated: kb[r][c], r <= c,
    // at kb_at(r, c).
    double kb[21];
#pragma unroll
    for (int i = 0; i < 21; i++) kb[i] = 0.0;
    const bool imag_a = A.si && A.di;
    for (int q = 0; q < A.qp.nq; q++) {
        const double w = A.qp.qw[q] * g.adet;
        double C[6][3];
        curls_generic(g, A.qp.curl_ref, q, C);
        double sum_nu = 0.0;
        for (int t = 0; t < N; t++) {
            double at[6];
            for (int k = 0; k < 6; k++) {
                double acc = 0.0;
                for (int h = 0; h < K; h++) {
                    double term = ar[k][h] * __ldg(A.dr + h * N + t);
                    if (imag_a) term = term - ai[k][h] * __ldg(A.di + h * N + t);
                    acc = acc + term;
                }
                at[k] = acc;
            }
            double B[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int i = 0; i < 6; i++)
#pragma unroll
                for (int c = 0; c < 3; c++) B[c] = B[c] + C[i][c] * at[i];
            const double bsq = B[0] * B[0] + B[1] * B[1] + B[2] * B[2];
            double nu, dnu;
            material_eval(A.mp, tag, bsq, nu, dnu);
            sum_nu = sum_nu + nu;
            const double H[3] = {nu * B[0], nu * B[1], nu * B[2]};
            for (int h = 0; h < K; h++) {
                const double p_r = __ldg(A.pr + t * K + h);
                const double p_i = A.pi ? __ldg(A.pi + t * K + h) : 0.0;
#pragma unroll
                for (int i = 0; i < 6; i++) {
                    const double dot = C[i][0] * H[0] + C[i][1] * H[1] + C[i][2] * H[2];
                    rr[i][h] = rr[i][h] + w * dot * p_r;
                    if (A.pi) ri[i][h] = ri[i][h] + w * dot * p_i;
                }
            }
        }
        if (CALCJ) {
            const double nu_dc = sum_nu / (double)N;
#pragma unroll
            for (int c = 0; c < 6; c++)
#pragma unroll
                for (int r = 0; r <= c; r++) {
                    const double dot = C[r][0] * C[c][0] + C[r][1] * C[c][1] + C[r][2] * C[c][2];
                    kb[kb_at(r, c)] = kb[kb_at(r, c)] + w * nu_dc * dot;
                }
        }
    }
    double *rdst = A.rscr + (int64_t)e * 6 * 2 * K;
#pragma unroll
    for (int i = 0; i < 6; i++) {
        const unsigned si = (sb >> i) & 1;
        for (int h = 0; h < K; h++) {
            rdst[i * 2 * K + h] = flip(rr[i][h], si);
            rdst[i * 2 * K + K + h] = flip(ri[i][h], si);
        }
        if (CALCJ) {
            double row[6];
#pragma unroll
            for (int j = 0; j < 6; j++) row[j] = flip(kb[i <= j ? kb_at(i, j) : kb_at(j, i)], si ^ ((sb >> j) & 1));
            store_row(A.scratch + e * kScratchPerElem + i * kScratchStride, row, 0.0);
        }
    }
}

// ---- constant curls, equal weights: six threads per element ------------------------
//
// With the standard curl table and equal weights every quadrature point repeats the same
// curls C_i, flux density B(t), nu(t) and weight w, so the time loop runs once per element,
// not once per point. What cannot be merged is the order of the residual's sum: the
// reference adds (w C_i . H(t)) P(h,t) over points, then samples, and its rounding needs all
// nq N additions one after another. The products repeat, though, so each thread forms the N
// products of one (edge, harmonic, part) once, in registers, and adds them nq times.
//
// A CTA of six warps takes kHbElems = 32 elements, lane = element:
//   1. warp i loads the harmonic values of local edge i; warp 0 the geometry (curls with the
//      edge signs folded in: negation commutes with rounding);
//   2. warp i evaluates samples i, i + 6, ...: A(t), B(t), nu(t), H(t), kHbSamples at a time
//      (one load of a harmonic value serves them all, and their spline searches run side by
//      side: the lookup is a chain of dependent loads). NT > 0: it has the curls of all six
//      edges in registers, so it leaves v(t) = w C_i . H(t) of every edge in shared memory,
//      where H would be read and multiplied again by six threads, and keeps nu in registers
//      until the harmonic values' place is free;
//   3. warp i sums the 2K residual entries of edge i. NT > 0: N <= NT samples, padded with
//      zeros (adding +0 changes no sum, which starts from +0 and so is never -0); v(t) is read
//      from the thread's own column of shared memory, so that only the products are held in
//      registers and three CTAs fit an SM. NT = 0: any N, kHbGroup sums at a time, H from
//      shared memory and v(t) formed in the loop.
// Work per element, without FMA (parity): 2 K 6 N (nq + 1) operations for the sums, N (24 K +
// 75) for the fields; at 40^3 (384,000 elements), K = 3, N = 32 that is 0.24 ms of the FP64
// pipe. Measured there, whole call: one thread per element with the time loop inside the point
// loop 1687 us; this split with v in registers (160 of them, two CTAs per SM, one sample at a
// time) 736 us; with v in shared memory, formed from H by step 3, and three CTAs 624 us (two
// CTAs: 721 us); with v formed by step 2, 602 us (two CTAs, nothing spilled: 662 us). Latency
// of the sums' dependent additions and of the spline lookups bounds it now.
constexpr int kHbElems = 32;
constexpr int kHbThreads = 6 * kHbElems;
constexpr int kHbSamples = 3;
constexpr int kHbGroup = 8;

// Shared memory: curls and weight [19][32]; harmonic values [6][2K][32], reused for nu (NT > 0)
// and the results; D and P [4K][np]; then v [np][6][32] (NT > 0) or H [np][3][32] and nu [np][32].
size_t hb_smem_bytes(int K, int N, int NT) {
    const int np = NT > 0 ? NT : N, held = NT > 0 && 12 * K < np ? np : 12 * K;
    return sizeof(double) * ((size_t)kHbElems * (19 + held) + (size_t)4 * K * np +
                             (size_t)kHbElems * np * (NT > 0 ? 6 : 4));
}

// nu of one material at M values of s = |B|^2: material_eval's arithmetic, the M searches in
// step.
template <int M>
__device__ __forceinline__ void material_nu(const MaterialParams &mp, int tag, const double s[M], double nu[M]) {
    const int m = tag - 1;
    const double nu0 = __ldg(mp.lin + m);
    if (__ldg(mp.is_non + m) == 0.0) {
#pragma unroll
        for (int j = 0; j < M; j++) nu[j] = nu0;
        return;
    }
    const double smax = __ldg(mp.max_bsq + m);
    const double *b = mp.breaks + __ldg(mp.start + m);
    const double *coefs = mp.coefs + __ldg(mp.coef_start + m);
    const int pieces = __ldg(mp.count + m);
    const double scale = mp.bucket ? __ldg(mp.bucket_geom + 2 * m + 1) : 0.0;
    double x[M];
    int k[M], lo[M], hi[M];
#pragma unroll
    for (int j = 0; j < M; j++) {
        x[j] = s[j] > smax ? smax : s[j];
        k[j] = 0;
        lo[j] = 0;
        hi[j] = pieces - 1;
    }
    if (scale > 0.0) {
        const double origin = __ldg(mp.bucket_geom + 2 * m);
#pragma unroll
        for (int j = 0; j < M; j++) {
            const double f = (x[j] - origin) * scale;
            const int i = !(f >= 0.0) ? 0 : (f >= (double)(kMatBuckets - 1) ? kMatBuckets - 1 : (int)f);
            const int *w = mp.bucket + 2 * kMatBuckets * m + i;
            lo[j] = __ldg(w);
            hi[j] = __ldg(w + kMatBuckets);
            k[j] = lo[j];
        }
    }
    for (;;) {
        bool more = false;
#pragma unroll
        for (int j = 0; j < M; j++)
            if (lo[j] <= hi[j]) {
                const int mid = lo[j] + (hi[j] - lo[j]) / 2;
                if (x[j] >= __ldg(b + mid)) {
                    k[j] = mid;
                    lo[j] = mid + 1;
                } else {
                    hi[j] = mid - 1;
                }
                more = true;
            }
        if (!more) break;
    }
#pragma unroll
    for (int j = 0; j < M; j++) {
        int kk = k[j];
        if (kk >= pieces) kk = pieces - 1;
        if (kk < 0) kk = 0;
        const double *c = coefs + 4 * kk;
        const double q0 = __ldg(c), q1 = __ldg(c + 1), q2 = __ldg(c + 2), q3 = __ldg(c + 3);
        const double t = x[j] - __ldg(b + kk);
        double v = ((q0 * t + q1) * t + q2) * t + q3;
        const double dv = (3.0 * q0 * t + 2.0 * q1) * t + q2;
        if (s[j] > smax) v = v + dv * (s[j] - smax);
        if (v > nu0 || v < 1e-7) v = nu0;
        nu[j] = v;
    }
}

template <int NT>
__global__ void __launch_bounds__(kHbThreads, NT > 0 ? 3 : 1) k_hbfem_std(HbArgs A) {
    extern __shared__ __align__(16) double hb_smem[];
    const int K = A.K, N = A.N, NP = NT > 0 ? NT : A.N, W = 2 * K;
    double *sC = hb_smem;                    // [18][32] signed curls
    double *sw = sC + 18 * kHbElems;         // [32] weight
    double *sa = sw + kHbElems;              // [6][2K][32] harmonic values; the results at the end
    double *sd = sa + (NT > 0 && 6 * W < NP ? NP : 6 * W) * kHbElems;  // [2K][NP] D re | im
    double *sp = sd + W * NP;                // [2K][NP] P re | im
    double *sH = sp + W * NP;                // [NP][3][32]; NT > 0: v [NP][6][32]
    double *snu = NT > 0 ? sa : sH + 3 * NP * kHbElems;  // [NP][32]
    const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t e0 = (int64_t)blockIdx.x * kHbElems, e = e0 + lane;
    const bool valid = e < A.m.ne;
    const bool imag_a = A.si && A.di;
    for (int i = threadIdx.x; i < W * NP; i += kHbThreads) {
        const int c = i / NP, t = i - c * NP, h = c < K ? c : c - K;
        const bool in = t < N;
        sd[i] = !in ? 0.0 : c < K ? __ldg(A.dr + h * N + t) : imag_a ? __ldg(A.di + h * N + t) : 0.0;
        sp[i] = !in ? 0.0 : c < K ? __ldg(A.pr + t * K + h) : A.pi ? __ldg(A.pi + t * K + h) : 0.0;
    }
    {
        const int d = valid ? __ldg(A.m.dofs + 6 * e + wi) : -1;
        for (int h = 0; h < K; h++) {
            sa[(wi * W + h) * kHbElems + lane] = d >= 0 ? __ldg(A.sr + h * A.ndof + d) : 0.0;
            if (imag_a) sa[(wi * W + K + h) * kHbElems + lane] = d >= 0 ? __ldg(A.si + h * A.ndof + d) : 0.0;
        }
    }
    const int tag = valid ? A.m.tags[e] : 0;
    if (wi == 0 && valid) {
        const int4 tt = A.m.tet[e];
        const unsigned sb = A.m.signbits ? A.m.signbits[e] : derived_signs(tt);
        Geo g;
        geometry(A.m.xyz, tt, g);
        double C[6][3];
        curls_standard(g, C);
#pragma unroll
        for (int i = 0; i < 6; i++)
#pragma unroll
            for (int r = 0; r < 3; r++) sC[(3 * i + r) * kHbElems + lane] = flip(C[i][r], (sb >> i) & 1);
        sw[lane] = A.qp.qw[0] * g.adet;
    }
    __syncthreads();
    constexpr int kPasses = NT > 0 ? (NT + 6 * kHbSamples - 1) / (6 * kHbSamples) : 1;
    double nuk[kPasses][kHbSamples];  // NT > 0: nu of this thread's samples
    if (valid) {
        double C[6][3];
        const double wq = sw[lane];
#pragma unroll
        for (int i = 0; i < 6; i++)
#pragma unroll
            for (int r = 0; r < 3; r++) C[i][r] = sC[(3 * i + r) * kHbElems + lane];
        auto samples = [&](int t, double (&nu)[kHbSamples]) {
            int ts[kHbSamples];
            double at[kHbSamples][6], B[kHbSamples][3], s[kHbSamples];
#pragma unroll
            for (int u = 0; u < kHbSamples; u++) {  // past the end: the first sample again
                ts[u] = t + 6 * u < N ? t + 6 * u : t;
#pragma unroll
                for (int k = 0; k < 6; k++) at[u][k] = 0.0;
            }
            for (int h = 0; h < K; h++) {
                double dr[kHbSamples], di[kHbSamples];
#pragma unroll
                for (int u = 0; u < kHbSamples; u++) {
                    dr[u] = sd[h * NP + ts[u]];
                    if (imag_a) di[u] = sd[(K + h) * NP + ts[u]];
                }
#pragma unroll
                for (int k = 0; k < 6; k++) {
                    const double xr = sa[(k * W + h) * kHbElems + lane];
                    const double xi = imag_a ? sa[(k * W + K + h) * kHbElems + lane] : 0.0;
#pragma unroll
                    for (int u = 0; u < kHbSamples; u++) {
                        double term = xr * dr[u];
                        if (imag_a) term = term - xi * di[u];
                        at[u][k] = at[u][k] + term;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < kHbSamples; u++) {
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    B[u][c] = 0.0;
#pragma unroll
                    for (int k = 0; k < 6; k++) B[u][c] = B[u][c] + C[k][c] * at[u][k];
                }
                s[u] = B[u][0] * B[u][0] + B[u][1] * B[u][1] + B[u][2] * B[u][2];
            }
            material_nu<kHbSamples>(A.mp, tag, s, nu);
#pragma unroll
            for (int u = 0; u < kHbSamples; u++) {
                const double H[3] = {nu[u] * B[u][0], nu[u] * B[u][1], nu[u] * B[u][2]};
                if constexpr (NT > 0) {
#pragma unroll
                    for (int i = 0; i < 6; i++)
                        sH[(6 * ts[u] + i) * kHbElems + lane] =
                            wq * (C[i][0] * H[0] + C[i][1] * H[1] + C[i][2] * H[2]);
                } else {
                    snu[ts[u] * kHbElems + lane] = nu[u];
#pragma unroll
                    for (int c = 0; c < 3; c++) sH[(3 * ts[u] + c) * kHbElems + lane] = H[c];
                }
            }
        };
        if constexpr (NT > 0) {
#pragma unroll
            for (int p = 0; p < kPasses; p++)
                if (wi + 6 * kHbSamples * p < N) samples(wi + 6 * kHbSamples * p, nuk[p]);
        } else {
            for (int t = wi; t < N; t += 6 * kHbSamples) samples(t, nuk[0]);
        }
    }
    if constexpr (NT > 0)
        for (int t = N; t < NT; t++) sH[(6 * t + wi) * kHbElems + lane] = 0.0;
    __syncthreads();
    const double c0 = sC[(3 * wi) * kHbElems + lane], c1 = sC[(3 * wi + 1) * kHbElems + lane],
                 c2 = sC[(3 * wi + 2) * kHbElems + lane], w = sw[lane];  // (not read for an invalid lane)
    const int nq = A.qp.nq;
    if (NT > 0 && (A.scratch || A.nu_dc)) {  // the harmonic values are used up
        if (valid)
#pragma unroll
            for (int p = 0; p < kPasses; p++)
#pragma unroll
                for (int u = 0; u < kHbSamples; u++) {
                    const int t = wi + 6 * kHbSamples * p + 6 * u;
                    if (t < N) snu[t * kHbElems + lane] = nuk[p][u];
                }
        __syncthreads();
    }
    if (valid && (A.scratch || (A.nu_dc && wi == 5))) {
        double sum_nu = 0.0;
        for (int t = 0; t < N; t++) sum_nu = sum_nu + snu[t * kHbElems + lane];
        const double nu_dc = sum_nu / (double)N;
        if (A.nu_dc && wi == 5) A.nu_dc[e] = nu_dc;
        if (A.scratch) {  // row wi of the DC block, w nu_dc (C_r . C_c) summed over the points
            double row[6];
#pragma unroll
            for (int j = 0; j < 6; j++) {
                const double dot = c0 * sC[(3 * j) * kHbElems + lane] + c1 * sC[(3 * j + 1) * kHbElems + lane] +
                                   c2 * sC[(3 * j + 2) * kHbElems + lane];
                const double v = w * nu_dc * dot;
                double acc = v;
                for (int q = 1; q < nq; q++) acc = acc + v;
                row[j] = acc;
            }
            store_row(A.scratch + e * kScratchPerElem + wi * kScratchStride, row, 0.0);
        }
    }
    double *out = sa + (lane * 6 + wi) * W;  // the harmonic values are used up
    if constexpr (NT > 0) {
        const double *sv = sH + threadIdx.x;  // [NT][6][32], this thread's column
        if (A.scratch || A.nu_dc) __syncthreads();  // nu is used up
        if (valid)
#pragma unroll 1
            for (int c = 0; c < W; c++) {
                double u[NT], acc = 0.0;
#pragma unroll
                for (int t = 0; t < NT; t++) {
                    u[t] = sv[t * kHbThreads] * sp[c * NP + t];
                    acc = acc + u[t];
                }
#pragma unroll 1
                for (int q = 1; q < nq; q++)
#pragma unroll
                    for (int t = 0; t < NT; t++) acc = acc + u[t];
                out[c] = acc;
            }
    } else if (valid) {
        for (int cb = 0; cb < W; cb += kHbGroup) {
            double acc[kHbGroup];
#pragma unroll
            for (int j = 0; j < kHbGroup; j++) acc[j] = 0.0;
            for (int q = 0; q < nq; q++)
                for (int t = 0; t < N; t++) {
                    const double *H = sH + 3 * t * kHbElems + lane;
                    const double v = w * (c0 * H[0] + c1 * H[kHbElems] + c2 * H[2 * kHbElems]);
#pragma unroll
                    for (int j = 0; j < kHbGroup; j++)
                        if (cb + j < W) acc[j] = acc[j] + v * sp[(cb + j) * NP + t];
                }
#pragma unroll
            for (int j = 0; j < kHbGroup; j++)
                if (cb + j < W) out[cb + j] = acc[j];
        }
    }
    __syncthreads();
    const int64_t left = A.m.ne - e0;
    const int count = (int)(left < kHbElems ? left : kHbElems) * 6 * W;
    double *dst = A.rscr + e0 * 6 * W;
    for (int i = threadIdx.x; i < count; i += kHbThreads) dst[i] = sa[i];
}

// out_re[h][row], out_im[h][row]: per CSR row and residual component, the incidences'
// entries summed from zero in ascending element order. parts: the residual components to sum (2K, or
// K without Im P: the imaginary residual is then zero whatever the entries hold, 0 x infinity is NaN).
__global__ void __launch_bounds__(128) k_rows_reduce_harm(RowPlan rp, const double *__restrict__ rscr, int K, int parts,
                                                          double *__restrict__ out_re, double *__restrict__ out_im) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int W = 2 * K;
    if (idx >= rp.ndof * W) return;
    const int64_t a = idx / W;
    const int c = (int)(idx % W);
    double r = 0.0;
    const int32_t t1 = c < parts ? rp.inc_ptr[a + 1] : 0;
    for (int32_t t = rp.inc_ptr[a]; t < t1; t++) {
        const uint32_t ew = rp.inc_elem[t];
        r = r + __ldg(rscr + ((int64_t)(ew & 0x1FFFFFFFu) * 6 + (ew >> 29)) * W + c);
    }
    if (c < K) out_re[(int64_t)c * rp.ndof + a] = r;
    else out_im[(int64_t)(c - K) * rp.ndof + a] = r;
}

}  // namespace

namespace {

template <int NT>
int launch_hb_std(const HbArgs &A, size_t smem, cudaStream_t s) {
    auto kern = k_hbfem_std<NT>;
    if (!allow_max_smem((const void *)kern)) return MAG_E_CUDA;
    kern<<<(unsigned)((A.m.ne + kHbElems - 1) / kHbElems), 6 * kHbElems, smem, s>>>(A);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}

}  // namespace

// Whether the general kernel, compiled for up to four harmonics, is the faster one although the
// constant-curl kernel could serve. With more samples than the register forms hold, k_hbfem_std<0> forms
// v(t) again for every group of sums: with one or two harmonics the general kernel then wins once its
// one thread per element fills the GPU. Measured, us, constant-curl / general kernel, four points: 1
// harmonic, 64 samples, residual and DC block at 29,478 elements 166 / 235, 48,000 252 / 252, 82,944
// 401 / 346, 384,000 1825 / 1440, residual alone at 29,478 155 / 212, 48,000 239 / 225; 2 harmonics,
// residual alone, 33 samples at 82,944 elements 252 / 287, 196,608 599 / 552, 663,552 2025 / 1751,
// 160 samples there 7257 / 7159; with the DC block, 64 samples, 3428 / 3502.
// A single point leaves no repeated work to merge: 64 samples at 48,000 and 384,000 elements, with the
// DC block, 1 harmonic 127 / 100 and 775 / 535, 2 harmonics 145 / 123 and 1061 / 797, 3 harmonics 170 / 184
// and 1224 / 1156; 3 harmonics, residual alone, 146 / 140 and 1160 / 869. Residuals alone with few samples
// (the constant-curl kernel takes them 18 at a time): 1 harmonic at 384,000, 8 samples 188 / 137, 16
// 186 / 168, 24 252 / 200, 32 260 / 238, but 196,608 elements 16 samples 89 / 109, 32 133 / 146; 2 harmonics,
// 8 samples 256 / 227, 16 259 / 287.
static bool hb_general_faster(int nq, int K, int N, int64_t ne, bool dc) {
    if (nq == 1) {
        if (ne < 45000) return false;
        if (N > 32) return K <= 2 || (K == 3 && !dc && ne >= 150000);
        return !dc && K <= 2 && (N <= 8 || (K == 1 && N > 16 && N <= 24));
    }
    if (N <= 32) return false;
    return (K == 1 && ne >= (dc ? 60000 : 45000)) || (K == 2 && !dc && N <= 128 && ne >= 190000);
}

bool hbfem_constant_curls(const QuadParams &qp, int K, int N, int64_t ne, bool dc) {
    const int nt = N <= 16 ? 16 : N <= 24 ? 24 : N <= 32 ? 32 : 0;
    return qp.standard_curl && qp.uniform_w && hb_smem_bytes(K, N, nt) <= (size_t)kMaxDynSmem &&
           !hb_general_faster(qp.nq, K, N, ne, dc);
}

namespace {

template <int KC>
void launch_hb_elems(const HbArgs &A, bool rows, cudaStream_t s) {
    const unsigned g = (unsigned)((A.m.ne + 127) / 128);
    if (rows) k_hbfem_elems<true, KC><<<g, 128, 0, s>>>(A);
    else k_hbfem_elems<false, KC><<<g, 128, 0, s>>>(A);
}

}  // namespace

int launch_hbfem(const ElemData &m, const RowPlan &rp, int max_row, const double *sr, const double *si, int K,
                 const double *dr, const double *di, const double *pr, const double *pi, int N,
                 const QuadParams &qp, const MaterialParams &mp, double *scratch, double *rscr, double *nu_dc,
                 double *vals, double *out_re, double *out_im, cudaStream_t s) {
    const bool rows = vals && !nu_dc;  // DC block rows through the element scratch
    HbArgs A{m, sr, si, dr, di, pr, pi, K, N, rp.ndof, qp, mp, rows ? scratch : nullptr, rscr, nu_dc};
    if (hbfem_constant_curls(qp, K, N, m.ne, vals != nullptr)) {
        const int nt = N <= 16 ? 16 : N <= 24 ? 24 : N <= 32 ? 32 : 0;
        const size_t smem = hb_smem_bytes(K, N, nt);
        MAG_TRY(nt == 16   ? launch_hb_std<16>(A, smem, s)
                : nt == 24 ? launch_hb_std<24>(A, smem, s)
                : nt == 32 ? launch_hb_std<32>(A, smem, s)
                           : launch_hb_std<0>(A, smem, s));
    } else {
        switch (K) {
            case 1: launch_hb_elems<1>(A, rows, s); break;
            case 2: launch_hb_elems<2>(A, rows, s); break;
            case 3: launch_hb_elems<3>(A, rows, s); break;
            case 4: launch_hb_elems<4>(A, rows, s); break;
            default: launch_hb_elems<0>(A, rows, s);
        }
        if (cudaPeekAtLastError() != cudaSuccess) return MAG_E_CUDA;
    }
    const int64_t nt = rp.ndof * 2 * K;
    k_rows_reduce_harm<<<(unsigned)((nt + 127) / 128), 128, 0, s>>>(rp, rscr, K, pi ? 2 * K : K, out_re, out_im);
    if (cudaPeekAtLastError() != cudaSuccess) return MAG_E_CUDA;
    if (rows) return launch_rows_reduce(rp, max_row, scratch, vals, nullptr, s);
    return MAG_OK;
}

}  // namespace mag
