// Tile-block Newton-Jacobian assembly (FP64, sm_100a): one launch, no scratch in HBM,
// each element evaluated by one thread, about 1.5 times per assembly.
//
// Rows (edges) are grouped by the spatial tile of their lower node: nodes are binned
// into coordinate layers along x, y and z, and 4 x 4 x 4 layers make a tile, on small meshes
// 3 x 3 x 3 or 4 x 2 x 2 (a CTA block holds at most kTileMaxNnz nonzeros, kTileMaxInc
// incidences and kTileMaxRows rows; larger tiles are cut). A CTA takes one block: its CSR
// rows, and every element incident to them.
//   colour phases -- one thread per element evaluates geometry, the six curls, B and
//              nu(|B|^2) once (the reference's arithmetic), then, for each of its local
//              rows that belongs to the block, the row of the 6x6 tangent and the
//              residual entry. Off-diagonal entries go straight into the block's
//              shared-memory copy of its CSR values as slot = slot + v. An
//              off-diagonal entry has at most two contributions (the two tetrahedra
//              that share a face) and (0 + a) + b equals (0 + b) + a bit for bit, so
//              the order does not matter, only that the two updates never overlap:
//              the plan colours the block's elements so that no two elements of a
//              colour share an entry (the face-adjacency graph of a Kuhn mesh is
//              bipartite: two colours), and the colours run one after another.
//              Diagonal entries and residual entries go to per-incidence slots.
//   row phase -- one thread per row sums its diagonal and residual contributions in
//              ascending element order (the reference's sparse() order).
//   store phase -- the block's rows form runs of consecutive rows, contiguous in the
//              CSR; warps store them in chunks, coalesced.
// No floating-point atomics; results equal the reference's MEX + sparse() bit for bit.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "element.cuh"
#include "tile.cuh"

namespace mag {

namespace {

using namespace elem;

struct TileArgs {
    const TileBlock *blocks;
    const uint2 *rows;
    const uint2 *chunks;
    const uint4 *recs;
    int64_t nrec;
    const double4 *xyz;
    const double *sol;
    const double *nu_e;    // K(nu): per-element reluctivity
    const double *bscale;  // seeded Jacobian: per-element flux-density scale of the tangent
    QuadParams qp;
    MaterialParams mp;
    double *vals;
    double *res;
    int *err;
    int64_t nnz_total, ndof;
    int smem_nnz;  // doubles reserved for the block's values (even)
    int smem_inc, smem_rows, smem_chunks;  // incidence slots, row-table and chunk entries reserved
};

// Sum over the quadrature points of v * w_q (w_q = qw_q |det J|) from zero, in point
// order. Q4: four equal weights, u = v w_0; the reference's ((u + u) + u) + u equals
// (3 u) + u because u + u is exact, so 3 u rounds like (u + u) + u.
template <bool Q4>
__device__ __forceinline__ double qsum4(double v, const QuadParams &qp, double w0, double adet) {
    const double u = v * w0;
    if (Q4) {
        const double t = 3.0 * u;
        return t + u;
    }
    double acc = u;
    if (qp.uniform_w) {
        for (int q = 1; q < qp.nq; q++) acc = acc + u;
    } else {
        for (int q = 1; q < qp.nq; q++) acc = acc + v * (qp.qw[q] * adet);
    }
    return acc;
}

// The sum of nq equal terms u from zero, in order (Q4: nq = 4, as above).
template <bool Q4>
__device__ __forceinline__ double qsum_equal(double u, int nq) {
    if (Q4) return 3.0 * u + u;
    double acc = u;
    for (int q = 1; q < nq; q++) acc = acc + u;
    return acc;
}

__device__ __forceinline__ void flag(int *err) { atomicOr(err, 1); }

// A record plane is read once: with PASS it does not displace the coordinates, solution and tables
// in L1 (records_pass says when that pays).
template <bool PASS = true>
__device__ __forceinline__ uint4 ld_record(const uint4 *p) {
    if (!PASS) return __ldg(p);
    uint4 v;
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

enum TileMode { kJacobian = 0, kStiffness = 1, kSeeded = 2, kHarmonicDc = 3 };

// One element of the block: record i. Returns the element's id.
//   kJacobian: residual and tangent at the element's state (assemble_jacobian_kernel_mex.cpp:92-131);
//   kStiffness: K(nu) with the element's given nu (assemble_curl_curl_kernel_mex.cpp:94-101), no residual;
//   kHarmonicDc: the harmonic-balance DC block, K(nu_dc) in that kernel's operation order
//            (w nu) (Ci.Cj) (assemble_hbfem_kernel_mex.cpp:211-226), no residual;
//   kSeeded: residual at B, tangent at the seeded state beta B:
//            nu(|beta B|^2) Ci.Cj + 2 nu'(|beta B|^2) (beta B.Ci)(beta B.Cj), the operation order of
//            the two-pass seeded kernel.
// FIRST: the block's first colour class. Its slots are all still +0 (no element of the
// class shares one), so an entry is stored rather than added: slot = v instead of
// slot = 0 + v, the same value up to the sign of an exact zero, which the store phase
// normalises (x + 0 turns -0 into +0 and leaves every other value unchanged).
template <bool CALCJ, bool Q4, int MODE, bool PASS, bool FIRST = false>
__device__ __forceinline__ uint32_t tile_element(const TileArgs &A, int64_t i, double *__restrict__ slot,
                                             double2 *__restrict__ incv, int bnnz, int binc) {
    const int64_t n = A.nrec;
    const uint4 p0 = ld_record<PASS>(A.recs + i), p1 = ld_record<PASS>(A.recs + n + i),
                p2 = ld_record<PASS>(A.recs + 2 * n + i), p3 = ld_record<PASS>(A.recs + 3 * n + i),
                p4 = ld_record<PASS>(A.recs + 4 * n + i), p5 = ld_record<PASS>(A.recs + 5 * n + i);
    const int4 tt = make_int4((int)p0.x, (int)p0.y, (int)p0.z, (int)p0.w);
    const unsigned sb = (p2.w >> 8) & 0x3Fu;
    const unsigned pos[6] = {p3.x, p3.y, p3.z, p3.w, p4.x, p4.y};
    const unsigned sl[6] = {p4.z, p4.w, p5.x, p5.y, p5.z, p5.w};
    Geo g;
    geometry(A.xyz, tt, g);
    double C[6][3];
    curls_standard(g, C);
    // Orientation signs folded into the curls (C_j s_j): negation is exact and commutes with
    // rounding to nearest, so B = sum a_j C_j is the same bits with unsigned edge values, and
    // every entry below comes out as s_l s_j times the unsigned one, which is how the
    // reference signs its finished entries. Only the sign of an exact zero can differ, and
    // every sum these entries enter starts from +0, which absorbs it.
#pragma unroll
    for (int j = 0; j < 6; j++)
        if ((sb >> j) & 1u) {
            C[j][0] = -C[j][0];
            C[j][1] = -C[j][1];
            C[j][2] = -C[j][2];
        }
    constexpr bool STIFF = MODE == kStiffness || MODE == kHarmonicDc;
    double nu, g2 = 0.0, b[6];
    double nut = 0.0, be = 1.0;  // seeded tangent: nu(|beta B|^2), beta
    if (STIFF) {
        nu = __ldg(A.nu_e + p2.z);
#pragma unroll
        for (int j = 0; j < 6; j++) b[j] = 0.0;
    } else {
        const int d[6] = {(int)p1.x, (int)p1.y, (int)p1.z, (int)p1.w, (int)p2.x, (int)p2.y};
        double a[6];
#pragma unroll
        for (int k = 0; k < 6; k++) a[k] = d[k] >= 0 ? __ldg(A.sol + d[k]) : 0.0;  // signs in C
        double B[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            double v = a[0] * C[0][c];
#pragma unroll
            for (int k = 1; k < 6; k++) v = v + a[k] * C[k][c];
            B[c] = v;
        }
        double dnu;
        material_eval(A.mp, (int)(p2.w & 0xFFu), dot3(B, B), nu, dnu);
#pragma unroll
        for (int j = 0; j < 6; j++) b[j] = dot3(B, C[j]);
        g2 = 2.0 * dnu;
        if (MODE == kSeeded && CALCJ) {
            be = __ldg(A.bscale + p2.z);
            double dnut;
            material_eval(A.mp, (int)(p2.w & 0xFFu), (be * be) * dot3(B, B), nut, dnut);
            g2 = 2.0 * dnut;
        }
    }
    const double adet = g.adet, w0 = A.qp.qw[0] * adet;
    // A warp that holds both kinds of element takes one path, not one after the other.
    const bool linear = g2 == 0.0;
    const bool linear_warp = MODE == kJacobian && CALCJ ? __all_sync(__activemask(), linear) != 0 : true;
#pragma unroll
    for (int l = 0; l < 6; l++) {
        const unsigned s = sl[l];
        if (s == kTileAbsent) continue;
        const int nzb = (int)(s & 0xFFFFu), is = (int)(s >> 16);
        // One check per row: the slot region has kTileSlotPad doubles beyond the largest
        // block, so nzb < bnnz keeps every nzb + p (p <= 30) inside it.
        if (nzb >= bnnz) {
            flag(A.err);
            continue;
        }
        const double rv = STIFF ? 0.0 : qsum4<Q4>(nu * b[l], A.qp, w0, adet);  // signed through C
        double dv = 0.0;
        if (CALCJ) {
            // the row's six entries first, then its five off-diagonal updates (the six
            // independent chains of arithmetic overlap; placing each entry as it is formed
            // measured slower)
            double v[6];
            if (MODE == kHarmonicDc) {  // the weight times nu first, then the product with each dot
                const double wn = w0 * nu;
#pragma unroll
                for (int j = 0; j < 6; j++) v[j] = qsum_equal<Q4>(wn * dot3(C[l], C[j]), A.qp.nq);
            } else if (MODE == kSeeded) {
                const double gl = g2 * (be * b[l]);
#pragma unroll
                for (int j = 0; j < 6; j++)
                    v[j] = qsum4<Q4>(nut * dot3(C[l], C[j]) + gl * (be * b[j]), A.qp, w0, adet);
            } else if (linear_warp) {
#pragma unroll
                for (int j = 0; j < 6; j++) v[j] = qsum4<Q4>(nu * dot3(C[l], C[j]), A.qp, w0, adet);
            } else {  // a linear element's second term is +0 (adding it changes at most the sign of a zero)
                const double gl = g2 * b[l];
#pragma unroll
                for (int j = 0; j < 6; j++) {
                    const double t = linear ? 0.0 : gl * b[j];
                    v[j] = qsum4<Q4>(nu * dot3(C[l], C[j]) + t, A.qp, w0, adet);
                }
            }
            dv = v[l];
#pragma unroll
            for (int j = 0; j < 6; j++) {
                if (j == l) continue;
                const int k = nzb + (int)((pos[l] >> (5 * j)) & 31u);  // absent column: the diagonal
                if (FIRST) slot[k] = v[j];
                else slot[k] = slot[k] + v[j];
            }
        }
        if (is < binc) {
            incv[is] = make_double2(rv, dv);
        } else {
            flag(A.err);
        }
    }
    return p2.z;
}

// L2 prefetch of [p, p + bytes) (16-byte aligned start and length; the plan's arrays are
// padded so that the rounded range stays inside them).
__device__ __forceinline__ void l2_prefetch(const void *p, size_t bytes) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uintptr_t lo = a & ~uintptr_t(15), hi = (a + bytes + 15) & ~uintptr_t(15);
    if (hi > lo)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lo), "r"((uint32_t)(hi - lo)) : "memory");
}

// What a block's next CTA visit will read first: its descriptor, records (six planes), rows
// and chunks.
__device__ __forceinline__ void prefetch_block(const TileArgs &A, int b) {
    const TileBlock *Bp = A.blocks + b;
    l2_prefetch(Bp, sizeof(TileBlock));
    const int rec0 = Bp->rec0, nrec = Bp->nrec;
    for (int k = 0; k < 6; k++) l2_prefetch(A.recs + (int64_t)k * A.nrec + rec0, (size_t)nrec * sizeof(uint4));
    l2_prefetch(A.rows + Bp->row0, (size_t)Bp->nrows * sizeof(uint2));
    l2_prefetch(A.chunks + Bp->chunk0, (size_t)Bp->nchunks * sizeof(uint2));
}

// 8-byte asynchronous global -> shared copies (both addresses 8-byte aligned).
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One CTA per block. The CTA of block b prefetches into L2 the records of block b + ahead
// (ahead = the CTAs resident at once), the block the hardware starts about when b ends.
// The block's row table and store chunks are copied into shared memory while its
// elements run, so the row and store phases start without a global round trip.
template <int BT, int MINB, bool CALCJ, bool Q4, int MODE, bool PASS>
__global__ void __launch_bounds__(BT, MINB) k_tile(TileArgs A, int nblocks, int ahead) {
    constexpr bool STIFF = MODE == kStiffness || MODE == kHarmonicDc;
    extern __shared__ __align__(16) double tile_smem[];
    double *slot = tile_smem;
    double2 *incv = reinterpret_cast<double2 *>(tile_smem + A.smem_nnz);
    uint2 *srows = reinterpret_cast<uint2 *>(incv + A.smem_inc);
    uint2 *schunks = srows + A.smem_rows;
    const int tid = threadIdx.x;
    {
        const int blk = blockIdx.x;
        if (tid == 0 && blk + ahead < nblocks) prefetch_block(A, blk + ahead);
        const TileBlock *Bp = A.blocks + blk;
        const int nrows = Bp->nrows, row0 = Bp->row0, rec0 = Bp->rec0, nrec = Bp->nrec;
        const int nnz = Bp->nnz, ninc = Bp->ninc, ncolors = Bp->ncolors;
        const int chunk0 = Bp->chunk0, nchunks = Bp->nchunks;
        if (nrows > A.smem_rows || nchunks > A.smem_chunks || nnz > A.smem_nnz - kTileSlotPad || ninc > A.smem_inc) {
            if (tid == 0) flag(A.err);  // the whole CTA leaves before its first barrier
            return;
        }
        for (int i = tid; i < nrows; i += BT) cp_async8(srows + i, A.rows + row0 + i);
        if (CALCJ)
            for (int i = tid; i < nchunks; i += BT) cp_async8(schunks + i, A.chunks + chunk0 + i);
        cp_async_commit();
        if (CALCJ) {
            for (int i = tid; i < (nnz + 1) / 2; i += BT)  // 16-byte stores; an odd tail's pair ends in the pad
        reinterpret_cast<double2 *>(slot)[i] = make_double2(0.0, 0.0);
            __syncthreads();
            int c0 = 0;
            for (int c = 0; c < ncolors; c++) {
                const int c1 = Bp->col_end[c];
                if (c == 0)
                    for (int i = c0 + tid; i < c1; i += BT)
                        tile_element<CALCJ, Q4, MODE, PASS, true>(A, (int64_t)rec0 + i, slot, incv, nnz, ninc);
                else
                    for (int i = c0 + tid; i < c1; i += BT)
                        tile_element<CALCJ, Q4, MODE, PASS>(A, (int64_t)rec0 + i, slot, incv, nnz, ninc);
                c0 = c1;
                if (c + 1 == ncolors) cp_async_wait_all();
                __syncthreads();
            }
            if (ncolors == 0) {
                cp_async_wait_all();
                __syncthreads();
            }
        } else {
            for (int i = tid; i < nrec; i += BT)
                tile_element<CALCJ, Q4, MODE, PASS>(A, (int64_t)rec0 + i, slot, incv, nnz, ninc);
            cp_async_wait_all();
            __syncthreads();
        }
        // rows: diagonal and residual in ascending element order
        for (int r = tid; r < nrows; r += BT) {
            const uint2 rw = srows[r];
            const int nzb = (int)(rw.y & 0x1FFFu), incb = (int)((rw.y >> 13) & 0xFFFu);
            const int diag = (int)((rw.y >> 25) & 31u);
            int ince = r + 1 < nrows ? (int)((srows[r + 1].y >> 13) & 0xFFFu) : ninc;
            if (ince > ninc) ince = ninc;
            double racc = 0.0, dacc = 0.0;
            for (int k = incb; k < ince; k++) {
                const double2 v = incv[k];
                racc = racc + v.x;
                if (CALCJ) dacc = dacc + v.y;
            }
            if (!STIFF) {
                if ((int64_t)rw.x < A.ndof) A.res[rw.x] = racc;
                else flag(A.err);
            }
            if (CALCJ && ince > incb) {
                if (nzb + diag < nnz) slot[nzb + diag] = dacc;
                else flag(A.err);
            }
        }
        __syncthreads();
        if (CALCJ) {
            const int warp = tid >> 5, lane = tid & 31;
            for (int c = warp; c < nchunks; c += BT / 32) {
                const uint2 ch = schunks[c];
                const int sb0 = (int)(ch.x & 0xFFFFu), len = (int)(ch.x >> 16);
                const int64_t g = (int64_t)ch.y;
                if (sb0 + len > nnz || g + len > A.nnz_total) {
                    if (lane == 0) flag(A.err);
                    continue;
                }
                for (int i = lane; i < len; i += 32) A.vals[g + i] = slot[sb0 + i] + 0.0;  // -0 -> +0
            }
        }
    }
}

// ---- batched complex assembly: K(nu) + j omega M(sigma) over many meshes ------------

struct TileComplexInstance {
    TileArgs a;              // the mesh's plan, coordinates, nu (nu_e), quadrature, error word
    const double *sigma;     // [Ne] or NULL (sigma = 1)
    const double *val_ref;   // [18 * nq] reference basis values, entry (i, c, q) at i + 6c + 18q
    double omega;
    double *cvals;           // complex128 [nnz] as (re, im)
};

// The sigma-mass rows of one element of the block (assemble_mass_kernel_mex.cpp:186-230):
// m_lj = sum_q ((N_l . N_j) sigma) w_q with N = J^{-T} N_ref at each point. The element's
// matrix is symmetric bit for bit (the same products in the same order), so its upper triangle
// is accumulated once, point by point, and each of the block's rows picks its six entries,
// signed: off-diagonal ones into their nonzeros' slots, the diagonal into the incidence slot's
// x. Elements with |sigma| <= 1e-12 add nothing (the reference skips them; a skipped
// contribution and a +0 one give the same sums).
// FIRST: the block's first colour class, whose slots are all still +0: stored, not added.
template <bool FIRST>
__device__ __forceinline__ void tile_mass_element(const TileArgs &A, const double *__restrict__ sigma_e, int64_t i,
                                                  double *__restrict__ slot, double2 *__restrict__ incv, int bnnz,
                                                  int binc, const double *__restrict__ sval) {
    const int64_t n = A.nrec;
    const uint4 p2 = ld_record<>(A.recs + 2 * n + i);
    const double sigma = sigma_e ? __ldg(sigma_e + p2.z) : 1.0;
    if (!(fabs(sigma) > 1e-12)) return;
    const uint4 p0 = ld_record<>(A.recs + i);
    const int4 tt = make_int4((int)p0.x, (int)p0.y, (int)p0.z, (int)p0.w);
    const unsigned sb = (p2.w >> 8) & 0x3Fu;
    double M[21];  // row by row from the diagonal
#pragma unroll
    for (int k = 0; k < 21; k++) M[k] = 0.0;
    {
        Geo g;
        geometry(A.xyz, tt, g);
        double iv[3][3];
        inverse3(g, iv);
        const int nq = A.qp.nq;
#pragma unroll 1
        for (int q = 0; q < nq; q++) {
            const double w = A.qp.qw[q] * g.adet;
            const double *r = sval + 18 * q;
            double N[6][3];
#pragma unroll
            for (int j = 0; j < 6; j++) {
                const double r0 = r[j], r1 = r[j + 6], r2 = r[j + 12];
#pragma unroll
                for (int c = 0; c < 3; c++) N[j][c] = iv[0][c] * r0 + iv[1][c] * r1 + iv[2][c] * r2;
            }
            int k = 0;
#pragma unroll
            for (int l = 0; l < 6; l++)
#pragma unroll
                for (int j = l; j < 6; j++, k++) M[k] = M[k] + dot3(N[l], N[j]) * sigma * w;
        }
    }
    const uint4 p3 = ld_record<>(A.recs + 3 * n + i), p4 = ld_record<>(A.recs + 4 * n + i), p5 = ld_record<>(A.recs + 5 * n + i);
    const unsigned pos[6] = {p3.x, p3.y, p3.z, p3.w, p4.x, p4.y};
    const unsigned sl[6] = {p4.z, p4.w, p5.x, p5.y, p5.z, p5.w};
#pragma unroll
    for (int l = 0; l < 6; l++) {
        const unsigned s = sl[l];
        if (s == kTileAbsent) continue;
        const int nzb = (int)(s & 0xFFFFu), is = (int)(s >> 16);
        if (nzb >= bnnz) {  // one check per row (kTileSlotPad)
            flag(A.err);
            continue;
        }
        const unsigned si = (sb >> l) & 1u;
#pragma unroll
        for (int j = 0; j < 6; j++) {
            if (j == l) continue;
            const int a = l < j ? l : j, b = l < j ? j : l;
            const int k = nzb + (int)((pos[l] >> (5 * j)) & 31u);  // absent column: the diagonal
            const double v = flip(M[a * 6 - a * (a - 1) / 2 + (b - a)], si ^ ((sb >> j) & 1u));
            if (FIRST) slot[k] = v;
            else slot[k] = slot[k] + v;
        }
        if (is < binc) incv[is].x = M[l * 6 - l * (l - 1) / 2];  // the diagonal: si ^ si = 0, no flip
        else flag(A.err);
    }
}

// Sums each row's diagonal contributions (incidence slots, component x or y) in ascending
// element order into the row's diagonal nonzero.
template <int BT, bool COMP_Y>
__device__ __forceinline__ void tile_rows_diag(const uint2 *srows, int nrows, const double2 *incv, int ninc,
                                               double *slot, int nnz, int *err) {
    for (int r = threadIdx.x; r < nrows; r += BT) {
        const uint2 rw = srows[r];
        const int nzb = (int)(rw.y & 0x1FFFu), incb = (int)((rw.y >> 13) & 0xFFFu);
        const int diag = (int)((rw.y >> 25) & 31u);
        int ince = r + 1 < nrows ? (int)((srows[r + 1].y >> 13) & 0xFFFu) : ninc;
        if (ince > ninc) ince = ninc;
        double dacc = 0.0;
        for (int k = incb; k < ince; k++) dacc = dacc + (COMP_Y ? incv[k].y : incv[k].x);
        if (ince > incb) {
            if (nzb + diag < nnz) slot[nzb + diag] = dacc;
            else flag(err);
        }
    }
}

// One CTA per (mesh, block) item: the tile kernel's K(nu) elements (incidence slots get (0, K
// diagonal)), row sums, (K, omega * 0) pairs stored in one coalesced pass. A block that holds a
// conducting element goes onto the list of k_tile_complex_mass, which then stores its imaginary
// parts. (Both passes in one kernel needed the registers of the M pass everywhere.)
// Values equal (K_ab, omega * M_ab) of MATLAB's K + 1j*omega*M (FrequencySolver.m:131).
template <int BT, int MINB, bool Q4>
__global__ void __launch_bounds__(BT, MINB)
    k_tile_complex(const TileComplexInstance *__restrict__ inst, const int2 *__restrict__ items, int nitems,
                   int ahead, int smem_nnz, int smem_inc, int smem_rows, int smem_chunks, int *__restrict__ list) {
    extern __shared__ __align__(16) double tile_smem[];
    double *slot = tile_smem;
    double2 *incv = reinterpret_cast<double2 *>(tile_smem + smem_nnz);
    uint2 *srows = reinterpret_cast<uint2 *>(incv + smem_inc);
    uint2 *schunks = srows + smem_rows;
    const int tid = threadIdx.x;
    const int it = blockIdx.x;
    if (tid == 0 && it + ahead < nitems) {
        const int2 nx = items[it + ahead];
        prefetch_block(inst[nx.x].a, nx.y);
    }
    const int2 w = items[it];
    const TileComplexInstance &I = inst[w.x];
    const TileArgs &A = I.a;
    const TileBlock *Bp = A.blocks + w.y;
    const int nrows = Bp->nrows, row0 = Bp->row0, rec0 = Bp->rec0;
    const int nnz = Bp->nnz, ninc = Bp->ninc, ncolors = Bp->ncolors;
    const int chunk0 = Bp->chunk0, nchunks = Bp->nchunks;
    if (nrows > smem_rows || nchunks > smem_chunks || nnz > smem_nnz - kTileSlotPad || ninc > smem_inc) {
        if (tid == 0) flag(A.err);  // the whole CTA leaves before its first barrier
        return;
    }
    for (int i = tid; i < nrows; i += BT) cp_async8(srows + i, A.rows + row0 + i);
    for (int i = tid; i < nchunks; i += BT) cp_async8(schunks + i, A.chunks + chunk0 + i);
    cp_async_commit();
    for (int i = tid; i < (nnz + 1) / 2; i += BT)  // 16-byte stores; an odd tail's pair ends in the pad
        reinterpret_cast<double2 *>(slot)[i] = make_double2(0.0, 0.0);
    __syncthreads();
    // the barrier after the last colour also tells whether any element of the block conducts
    int conducting = 0;
    int c0 = 0;
    bool any_m = false;
    for (int c = 0; c < ncolors; c++) {
        const int c1 = Bp->col_end[c];
        for (int i = c0 + tid; i < c1; i += BT) {
            const int64_t r = (int64_t)rec0 + i;
            const uint32_t e = c == 0 ? tile_element<true, Q4, kStiffness, true, true>(A, r, slot, incv, nnz, ninc)
                                      : tile_element<true, Q4, kStiffness, true>(A, r, slot, incv, nnz, ninc);
            if (!conducting) conducting = fabs(I.sigma ? __ldg(I.sigma + e) : 1.0) > 1e-12;
        }
        c0 = c1;
        if (c + 1 == ncolors) {
            cp_async_wait_all();
            any_m = __syncthreads_or(conducting) != 0;
        } else {
            __syncthreads();
        }
    }
    if (ncolors == 0) {
        cp_async_wait_all();
        __syncthreads();
    }
    if (tid == 0 && any_m) list[1 + atomicAdd(list, 1)] = it;
    tile_rows_diag<BT, true>(srows, nrows, incv, ninc, slot, nnz, A.err);
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    double2 *cv2 = reinterpret_cast<double2 *>(I.cvals);
    const double im = I.omega * 0.0;
    for (int c = warp; c < nchunks; c += BT / 32) {
        const uint2 ch = schunks[c];
        const int sb0 = (int)(ch.x & 0xFFFFu), len = (int)(ch.x >> 16);
        const int64_t g = (int64_t)ch.y;
        if (sb0 + len > nnz || g + len > A.nnz_total) {
            if (lane == 0) flag(A.err);
            continue;
        }
        // (+ 0.0: -0 -> +0, the first colour stores its entries)
        for (int i = lane; i < len; i += 32) cv2[g + i] = make_double2(slot[sb0 + i] + 0.0, im);
    }
}

// The sigma-mass values of one block: slots and incidence slots zeroed, the conducting elements'
// rows colour by colour, diagonals in element order, then each stored value through `store(nonzero,
// value)`. Uniform over the CTA; ends without a barrier.
struct TileSmem {
    double *slot;
    double2 *incv;
    uint2 *rows, *chunks;
    double *val;  // [18 nq] reference basis values
    int nnz, inc, nrows, nchunks;
};

__device__ __forceinline__ TileSmem tile_smem_layout(double *base, int nnz, int inc, int rows, int chunks) {
    TileSmem S;
    S.slot = base;
    S.incv = reinterpret_cast<double2 *>(base + nnz);
    S.rows = reinterpret_cast<uint2 *>(S.incv + inc);
    S.chunks = S.rows + rows;
    S.val = reinterpret_cast<double *>(S.chunks + chunks);
    S.nnz = nnz;
    S.inc = inc;
    S.nrows = rows;
    S.nchunks = chunks;
    return S;
}

template <int BT, typename Store>
__device__ __forceinline__ void tile_mass_block(const TileArgs &A, const TileSmem &S, const TileBlock *Bp,
                                                const double *__restrict__ sigma, const double *__restrict__ val_ref,
                                                Store store) {
    const int tid = threadIdx.x;
    const int nrows = Bp->nrows, row0 = Bp->row0, rec0 = Bp->rec0;
    const int nnz = Bp->nnz, ninc = Bp->ninc, ncolors = Bp->ncolors;
    const int chunk0 = Bp->chunk0, nchunks = Bp->nchunks;
    const int nq = A.qp.nq;
    if (nrows > S.nrows || nchunks > S.nchunks || nnz > S.nnz - kTileSlotPad || ninc > S.inc || nq > kMaxQuad) {
        if (tid == 0) flag(A.err);  // the whole CTA skips the block
        return;
    }
    for (int i = tid; i < nrows; i += BT) cp_async8(S.rows + i, A.rows + row0 + i);
    for (int i = tid; i < nchunks; i += BT) cp_async8(S.chunks + i, A.chunks + chunk0 + i);
    cp_async_commit();
    for (int i = tid; i < 18 * nq; i += BT) S.val[i] = __ldg(val_ref + i);
    for (int i = tid; i < (nnz + 1) / 2; i += BT)  // 16-byte stores; an odd tail's pair ends in the pad
        reinterpret_cast<double2 *>(S.slot)[i] = make_double2(0.0, 0.0);
    for (int i = tid; i < ninc; i += BT) S.incv[i] = make_double2(0.0, 0.0);  // no sigma: nothing written
    __syncthreads();
    int c0 = 0;
    for (int c = 0; c < ncolors; c++) {
        const int c1 = Bp->col_end[c];
        if (c == 0)
            for (int i = c0 + tid; i < c1; i += BT)
                tile_mass_element<true>(A, sigma, (int64_t)rec0 + i, S.slot, S.incv, nnz, ninc, S.val);
        else
            for (int i = c0 + tid; i < c1; i += BT)
                tile_mass_element<false>(A, sigma, (int64_t)rec0 + i, S.slot, S.incv, nnz, ninc, S.val);
        c0 = c1;
        if (c + 1 == ncolors) cp_async_wait_all();
        __syncthreads();
    }
    if (ncolors == 0) {
        cp_async_wait_all();
        __syncthreads();
    }
    tile_rows_diag<BT, false>(S.rows, nrows, S.incv, ninc, S.slot, nnz, A.err);
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    for (int c = warp; c < nchunks; c += BT / 32) {
        const uint2 ch = S.chunks[c];
        const int sb0 = (int)(ch.x & 0xFFFFu), len = (int)(ch.x >> 16);
        const int64_t g = (int64_t)ch.y;
        if (sb0 + len > nnz || g + len > A.nnz_total) {
            if (lane == 0) flag(A.err);
            continue;
        }
        for (int i = lane; i < len; i += 32) store(g + i, S.slot[sb0 + i] + 0.0);  // -0 -> +0
    }
}

// 256 threads x 2 CTAs per SM: 128 registers hold the element's upper triangle and six basis
// vectors (at 320 x 2, 96 registers, they spill).
constexpr int kMassBT = 256;

// M(sigma) of one mesh, one CTA per block. 613,000 elements, a tenth of them conducting: 295 us
// with element blocks through HBM scratch and row sums, 60 us here.
template <int BT, int MINB>
__global__ void __launch_bounds__(BT, MINB)
    k_tile_mass(TileArgs A, const double *__restrict__ sigma, const double *__restrict__ val_ref, int nblocks, int ahead) {
    extern __shared__ __align__(16) double tile_smem[];
    const TileSmem S = tile_smem_layout(tile_smem, A.smem_nnz, A.smem_inc, A.smem_rows, A.smem_chunks);
    const int blk = blockIdx.x;
    if (threadIdx.x == 0 && blk + ahead < nblocks) prefetch_block(A, blk + ahead);
    double *vals = A.vals;
    tile_mass_block<BT>(A, S, A.blocks + blk, sigma, val_ref, [&](int64_t k, double v) { vals[k] = v; });
}

// The imaginary parts omega * M of the listed items (list[0] of them), resident CTAs striding.
__global__ void __launch_bounds__(kMassBT, 2)
    k_tile_complex_mass(const TileComplexInstance *__restrict__ inst, const int2 *__restrict__ items, int smem_nnz,
                        int smem_inc, int smem_rows, int smem_chunks, const int *__restrict__ list) {
    extern __shared__ __align__(16) double tile_smem[];
    const TileSmem S = tile_smem_layout(tile_smem, smem_nnz, smem_inc, smem_rows, smem_chunks);
    const int count = list[0];
    for (int k = blockIdx.x; k < count; k += gridDim.x) {
        const int2 w = items[list[1 + k]];
        const TileComplexInstance &I = inst[w.x];
        double *im = I.cvals + 1;
        const double omega = I.omega;
        tile_mass_block<kMassBT>(I.a, S, I.a.blocks + w.y, I.sigma, I.val_ref,
                                 [&](int64_t k, double v) { im[2 * k] = omega * v; });
        __syncthreads();  // the block's values are read out of shared memory
    }
}

// 320 threads: a colour class of an interior 4x4x4 tile holds about 288 elements, so each
// colour phase runs in one pass (256 threads left a second pass with one warp busy).
constexpr int kTileBT = 320;
constexpr int kTileMinB = 2;
// Small blocks (tiles of 4x2x2 or 3x3x3 layers, a colour class of 90 to 135 elements): each colour
// phase in one pass. A tile that holds more than its layers' share (graded meshes, layers that nodes
// of different depth fall into) is cut at a block's limits instead; its classes take two passes and
// more of 160 threads, so that the plan says which shape suits. Jacobian, us, 160 x 3 / 320 x 2: 8^3
// hexahedra 9.3 / 9.7, graded 20^3 21.6 / 17.5, 1 x 1 x 4000 16.5 / 11.1, two cubes far apart 19.7 / 14.7.
constexpr int kSmallBT = kTileSmallThreads;
constexpr int kSmallMinB = 3;

}  // namespace

namespace {

// A block at every limit of the plan (a chunk has a row that owns it, or lies inside one), with the
// mass kernels' basis values, fits a CTA.
static_assert((kTileMaxNnz + 1 + kTileSlotPad) * 8 + kTileMaxInc * 16 +
                      (2 * kTileMaxRows + kTileMaxNnz / kTileChunk + 1) * 8 + 18 * kMaxQuad * 8 <= kMaxDynSmem,
              "a block's shared memory");

// Shared memory of one CTA: the block's values (an even count of doubles), the incidence
// slots (double2), then the block's row table and store chunks (uint2 each).
size_t tile_smem_bytes(const TilePlan &tp, TileArgs *a) {
    a->smem_nnz = ((tp.max_nnz + 1) & ~1) + kTileSlotPad;
    a->smem_inc = tp.max_inc;
    a->smem_rows = tp.max_rows;
    a->smem_chunks = tp.max_chunks;
    return (size_t)a->smem_nnz * sizeof(double) + (size_t)a->smem_inc * sizeof(double2) +
           (size_t)(a->smem_rows + a->smem_chunks) * sizeof(uint2);
}

// Allows the kernel its shared memory and gives the CTAs resident at once on the device (how
// far ahead a CTA prefetches).
int resident_ctas(const void *kern, int threads, size_t smem, int *out) {
    int dev = 0, nsm = 0, per = 0;
    if (!allow_max_smem(kern) || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem) != cudaSuccess || per < 1)
        return MAG_E_CUDA;
    *out = per * nsm;
    return MAG_OK;
}

// Whether the records pass L1 by: below these sizes loads that go through it are faster. Measured, us,
// through L1 / by: Jacobian at 20^3 hexahedra (72,000 records) 14.8 / 14.9, shuffled 26^3 (163,000) 27.7 /
// 29.7, 34^3 (354,000) 37.8 / 38.2, 36^3 (420,000) 47.6 / 45.0, 40^3 65.2 / 62.5, 60^3 191 / 190; residual
// alone at 26^3 shuffled 17.8 / 18.4, 40^3 (576,000) 28.1 / 28.9, 44^3 (767,000) 38.6 / 37.8, 48^3 53.1 /
// 47.2. CTAs of the small shape have few records and each SM three of them: Jacobian at 8^3 9.24 / 9.06,
// residual at 17^3 7.2 / 6.8, always by. So does the harmonic-balance DC block, which follows the
// harmonic kernel's stores: the whole call at 24^3 with 4 harmonics, 64 samples 544 / 534.
template <bool CALCJ>
bool records_pass(const TilePlan &tp) {
    return tp.nrec >= (CALCJ ? 380000 : 650000);
}

template <bool CALCJ, bool Q4, int MODE, int BT, int MINB>
int launch_shape(const TileArgs &a, const TilePlan &tp, size_t smem, cudaStream_t s) {
    auto kern = k_tile<BT, MINB, CALCJ, Q4, MODE, true>;
    if constexpr (BT != kSmallBT && MODE != kHarmonicDc)
        if (!records_pass<CALCJ>(tp)) kern = k_tile<BT, MINB, CALCJ, Q4, MODE, false>;
    int resident = 0;
    MAG_TRY(resident_ctas((const void *)kern, BT, smem, &resident));
    // (ahead >= nblocks: no CTA prefetches)
    const int ahead = tp.prefetch_waves > 0 ? resident * tp.prefetch_waves : tp.nblocks;
    kern<<<tp.nblocks, BT, smem, s>>>(a, tp.nblocks, ahead);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}

// The shape of the plan's blocks.
template <bool CALCJ, bool Q4, int MODE>
int launch(const TileArgs &a, const TilePlan &tp, size_t smem, cudaStream_t s) {
    return tp.small_blocks ? launch_shape<CALCJ, Q4, MODE, kSmallBT, kSmallMinB>(a, tp, smem, s)
                          : launch_shape<CALCJ, Q4, MODE, kTileBT, kTileMinB>(a, tp, smem, s);
}

TileArgs make_args(const TilePlan &tp, const ElemData &m, const QuadParams &qp, int *err) {
    TileArgs a{};
    a.blocks = tp.blocks;
    a.rows = tp.rows;
    a.chunks = tp.chunks;
    a.recs = tp.recs;
    a.nrec = tp.nrec;
    a.xyz = m.xyz;
    a.qp = qp;
    a.err = err;
    a.ndof = tp.nrows;
    return a;
}

}  // namespace

int launch_tile_jacobian(const TilePlan &tp, const ElemData &m, const double *sol, const QuadParams &qp,
                         const MaterialParams &mp, int calc_j, double *vals, double *res, int *err,
                         cudaStream_t s) {
    if (!tp.ok || !qp.standard_curl) return MAG_E_UNSUPPORTED;
    TileArgs a = make_args(tp, m, qp, err);
    a.sol = sol;
    a.mp = mp;
    a.vals = vals;
    a.res = res;
    a.nnz_total = tp.nnz;
    size_t smem = tile_smem_bytes(tp, &a);
    const bool q4 = qp.nq == 4 && qp.uniform_w;
    if (calc_j && q4) {  // the launch shape of the Newton Jacobian (threads per CTA x CTAs per SM)
        switch (tp.variant) {
            case 1: return launch_shape<true, true, kJacobian, 288, 2>(a, tp, smem, s);
            case 2: return launch_shape<true, true, kJacobian, 256, 2>(a, tp, smem, s);
            case 3: return launch_shape<true, true, kJacobian, 512, 1>(a, tp, smem, s);
            default: return launch<true, true, kJacobian>(a, tp, smem, s);
        }
    }
    if (calc_j) return launch<true, false, kJacobian>(a, tp, smem, s);
    return q4 ? launch<false, true, kJacobian>(a, tp, smem, s) : launch<false, false, kJacobian>(a, tp, smem, s);
}

const char *tile_variant_name(int v) {
    static const char *names[kTileVariants] = {"320 threads x 2 CTAs/SM (small blocks: 160 x 3)", "288 threads x 2 CTAs/SM",
                                               "256 threads x 2 CTAs/SM", "512 threads x 1 CTA/SM"};
    return v >= 0 && v < kTileVariants ? names[v] : "";
}

int launch_tile_stiffness(const TilePlan &tp, const ElemData &m, const double *nu, const QuadParams &qp,
                          double *vals, int *err, cudaStream_t s) {
    if (!tp.ok || !qp.standard_curl) return MAG_E_UNSUPPORTED;
    TileArgs a = make_args(tp, m, qp, err);
    a.nu_e = nu;
    a.vals = vals;
    a.nnz_total = tp.nnz;
    size_t smem = tile_smem_bytes(tp, &a);
    const bool q4 = qp.nq == 4 && qp.uniform_w;
    return q4 ? launch<true, true, kStiffness>(a, tp, smem, s) : launch<true, false, kStiffness>(a, tp, smem, s);
}

int launch_tile_mass(const TilePlan &tp, const ElemData &m, const double *sigma, const QuadParams &qp, double *vals,
                     int *err, cudaStream_t s) {
    if (!tp.ok || qp.nq > kMaxQuad) return MAG_E_UNSUPPORTED;
    TileArgs a = make_args(tp, m, qp, err);
    a.vals = vals;
    a.nnz_total = tp.nnz;
    const size_t smem = tile_smem_bytes(tp, &a) + (size_t)18 * qp.nq * sizeof(double);
    const auto kern = tp.small_blocks ? k_tile_mass<kSmallBT, kSmallMinB> : k_tile_mass<kMassBT, 2>;
    const int threads = tp.small_blocks ? kSmallBT : kMassBT;
    int resident = 0;
    MAG_TRY(resident_ctas((const void *)kern, threads, smem, &resident));
    const int ahead = tp.prefetch_waves > 0 ? resident * tp.prefetch_waves : tp.nblocks;
    kern<<<tp.nblocks, threads, smem, s>>>(a, sigma, qp.val_ref, tp.nblocks, ahead);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}

int launch_tile_harmonic_dc(const TilePlan &tp, const ElemData &m, const double *nu_dc, const QuadParams &qp,
                            double *vals, int *err, cudaStream_t s) {
    if (!tp.ok || !qp.standard_curl || !qp.uniform_w) return MAG_E_UNSUPPORTED;
    TileArgs a = make_args(tp, m, qp, err);
    a.nu_e = nu_dc;
    a.vals = vals;
    a.nnz_total = tp.nnz;
    size_t smem = tile_smem_bytes(tp, &a);
    return qp.nq == 4 ? launch<true, true, kHarmonicDc>(a, tp, smem, s) : launch<true, false, kHarmonicDc>(a, tp, smem, s);
}

int launch_tile_seeded(const TilePlan &tp, const ElemData &m, const double *sol, const double *bscale,
                       const QuadParams &qp, const MaterialParams &mp, double *vals, double *res, int *err,
                       cudaStream_t s) {
    if (!tp.ok || !qp.standard_curl) return MAG_E_UNSUPPORTED;
    TileArgs a = make_args(tp, m, qp, err);
    a.sol = sol;
    a.bscale = bscale;
    a.mp = mp;
    a.vals = vals;
    a.res = res;
    a.nnz_total = tp.nnz;
    size_t smem = tile_smem_bytes(tp, &a);
    const bool q4 = qp.nq == 4 && qp.uniform_w;
    return q4 ? launch<true, true, kSeeded>(a, tp, smem, s) : launch<true, false, kSeeded>(a, tp, smem, s);
}

namespace {

using ComplexKernel = void (*)(const TileComplexInstance *, const int2 *, int, int, int, int, int, int, int *);

ComplexKernel complex_kernel(int variant, bool q4) {
    if (q4) return variant == 1 ? k_tile_complex<288, 2, true> : k_tile_complex<320, 2, true>;
    return variant == 1 ? k_tile_complex<288, 2, false> : k_tile_complex<320, 2, false>;
}
constexpr int kComplexThreads[kTileComplexVariants] = {320, 288};

}  // namespace

int build_tile_complex(const std::vector<TileComplexInput> &in, TileComplexBatch *b, cudaStream_t s) {
    *b = TileComplexBatch{};
    if (in.empty()) return MAG_OK;
    std::vector<TileComplexInstance> hi(in.size());
    int q4 = 1;
    for (size_t i = 0; i < in.size(); i++) {
        const TilePlan &tp = *in[i].tp;
        if (!tp.ok || !in[i].qp.standard_curl || in[i].qp.nq > kMaxQuad) return MAG_OK;
        TileComplexInstance &t = hi[i];
        t = TileComplexInstance{};
        t.a = make_args(tp, in[i].m, in[i].qp, in[i].err);
        t.a.nu_e = in[i].nu;
        t.a.nnz_total = tp.nnz;
        t.sigma = in[i].sigma;
        t.val_ref = in[i].qp.val_ref;
        t.omega = in[i].omega;
        t.cvals = in[i].vals;
        b->smem_nnz = std::max(b->smem_nnz, ((tp.max_nnz + 1) & ~1) + kTileSlotPad);
        b->smem_inc = std::max(b->smem_inc, tp.max_inc);
        b->smem_rows = std::max(b->smem_rows, tp.max_rows);
        b->smem_chunks = std::max(b->smem_chunks, tp.max_chunks);
        q4 &= (in[i].qp.nq == 4 && in[i].qp.uniform_w) ? 1 : 0;
    }
    // items: larger meshes first (a short tail), each mesh's blocks in plan order
    std::vector<int> order(in.size());
    for (size_t i = 0; i < in.size(); i++) order[i] = (int)i;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return in[x].tp->nrec > in[y].tp->nrec; });
    std::vector<int2> items;
    for (int i : order)
        for (int k = 0; k < in[i].tp->nblocks; k++) items.push_back(make_int2(i, k));
    if (items.empty() || items.size() >= (size_t)INT32_MAX) return MAG_OK;
    b->q4 = q4;
    b->smem = (size_t)b->smem_nnz * sizeof(double) + (size_t)b->smem_inc * sizeof(double2) +
              (size_t)(b->smem_rows + b->smem_chunks) * sizeof(uint2);
    b->smem_mass = b->smem + (size_t)18 * kMaxQuad * sizeof(double);
    bool fits = resident_ctas((const void *)k_tile_complex_mass, kMassBT, b->smem_mass, &b->mass_ctas) == MAG_OK;
    for (int v = 0; v < kTileComplexVariants; v++)
        fits = fits && resident_ctas((const void *)complex_kernel(v, q4 != 0), kComplexThreads[v], b->smem,
                                     &b->ahead[v]) == MAG_OK;
    if (!fits || cudaMalloc(&b->inst, hi.size() * sizeof(TileComplexInstance)) != cudaSuccess ||
        cudaMalloc(&b->items, items.size() * sizeof(int2)) != cudaSuccess ||
        cudaMalloc(&b->list, (items.size() + 1) * sizeof(int)) != cudaSuccess) {
        cudaGetLastError();
        free_tile_complex(b);
        return MAG_OK;  // the blocks do not fit: the other batch variants remain
    }
    b->mass_ctas = std::min(b->mass_ctas, (int)items.size());
    MAG_CUDA_TRY(cudaMemcpyAsync(b->inst, hi.data(), hi.size() * sizeof(TileComplexInstance), cudaMemcpyHostToDevice, s));
    MAG_CUDA_TRY(cudaMemcpyAsync(b->items, items.data(), items.size() * sizeof(int2), cudaMemcpyHostToDevice, s));
    MAG_CUDA_TRY(cudaStreamSynchronize(s));
    b->nitems = (int)items.size();
    b->ok = 1;
    return MAG_OK;
}

int launch_tile_complex(const TileComplexBatch &b, int variant, cudaStream_t s) {
    if (!b.ok || variant < 0 || variant >= kTileComplexVariants) return MAG_E_UNSUPPORTED;
    const TileComplexInstance *inst = static_cast<const TileComplexInstance *>(b.inst);
    if (cudaMemsetAsync(b.list, 0, sizeof(int), s) != cudaSuccess) return MAG_E_CUDA;
    complex_kernel(variant, b.q4 != 0)<<<b.nitems, kComplexThreads[variant], b.smem, s>>>(
        inst, b.items, b.nitems, b.ahead[variant], b.smem_nnz, b.smem_inc, b.smem_rows, b.smem_chunks, b.list);
    k_tile_complex_mass<<<b.mass_ctas, kMassBT, b.smem_mass, s>>>(
        inst, b.items, b.smem_nnz, b.smem_inc, b.smem_rows, b.smem_chunks, b.list);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}

const char *tile_complex_variant_name(int v) {
    static const char *names[kTileComplexVariants] = {"tile blocks, 320 threads x 2 CTAs/SM",
                                                      "tile blocks, 288 threads x 2 CTAs/SM"};
    return v >= 0 && v < kTileComplexVariants ? names[v] : "";
}

void free_tile_complex(TileComplexBatch *b) {
    if (b->inst) cudaFree(b->inst);
    if (b->items) cudaFree(b->items);
    if (b->list) cudaFree(b->list);
    *b = TileComplexBatch{};
}

}  // namespace mag
