// One-time integer work on the GPU: edge numbering (Mesh.generateEdges), the CSR
// pattern of the dof coupling, the per-row incidence plan used by the
// fixed-order value reduction, and MATLAB-style zero dropping.
//
// Sorting uses CUB's stable radix sort (header library shipped with the CUDA
// toolkit). Stability is what makes every row's incidence list come out in
// ascending element order, which fixes the summation order of the assembly.
#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_reduce.cuh>
#include <cub/device/device_scan.cuh>

#include "common.cuh"
#include "internal.h"

namespace mag {

namespace {

int bits_for(uint64_t n) {
    int b = 1;
    while (b < 64 && (uint64_t(1) << b) <= n) b++;
    return b;
}

constexpr int kBlock = 256;
inline unsigned grid_for(int64_t n, int block = kBlock) {
    return (unsigned)((n + block - 1) / block);
}

// ---- edges --------------------------------------------------------------

__global__ void k_edge_keys(const int32_t *__restrict__ T, int64_t ne, int64_t nn, int nb,
                            uint64_t *__restrict__ keys, uint32_t *__restrict__ slots,
                            int8_t *__restrict__ sign, int *__restrict__ err) {
    int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= 6 * ne) return;
    int64_t e = s / 6;
    int k = (int)(s - 6 * e);
    int32_t a = T[4 * e + edge_a(k)], b = T[4 * e + edge_b(k)];
    if (a < 0 || b < 0 || a >= nn || b >= nn || a == b) {
        atomicExch(err, 1);
        a = b = 0;
    }
    uint64_t lo = (uint64_t)(a < b ? a : b), hi = (uint64_t)(a < b ? b : a);
    keys[s] = (lo << nb) | hi;
    slots[s] = (uint32_t)s;
    // +1 iff the local start node carries the smaller global id (Mesh.m:134-135)
    sign[s] = (int8_t)(a < b ? 1 : -1);
}

__global__ void k_head_flags(const uint64_t *__restrict__ keys, int64_t n, int32_t *__restrict__ f) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    f[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

__global__ void k_edge_scatter(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ slots,
                               const int32_t *__restrict__ flags, const int32_t *__restrict__ ids,
                               int64_t n, int nb, int32_t *__restrict__ edges,
                               int32_t *__restrict__ t2e) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    int32_t id = ids[i] - 1;
    t2e[slots[i]] = id;
    if (flags[i]) {
        uint64_t k = keys[i];
        edges[2 * (int64_t)id] = (int32_t)(k >> nb);
        edges[2 * (int64_t)id + 1] = (int32_t)(k & ((uint64_t(1) << nb) - 1));
    }
}

// ---- pattern ------------------------------------------------------------

__global__ void k_inc_keys(const int32_t *__restrict__ dofs, int64_t ne, int64_t ndof,
                           uint32_t *__restrict__ keys, uint32_t *__restrict__ vals,
                           int32_t *__restrict__ cnt, int *__restrict__ err) {
    int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= 6 * ne) return;
    int64_t e = s / 6;
    int k = (int)(s - 6 * e);
    int32_t d = dofs[s];
    if (d >= ndof || d < -1) {
        atomicExch(err, 1);
        d = -1;
    }
    keys[s] = d < 0 ? (uint32_t)ndof : (uint32_t)d;  // dof-less slots sort to the end
    vals[s] = (uint32_t)e | ((uint32_t)k << 29);
    if (d >= 0) atomicAdd(&cnt[d], 1);
}

// Sorted unique insert into a small per-thread list; returns false on overflow.
__device__ inline bool insert_sorted(int32_t *list, int &n, int cap, int32_t v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (list[mid] < v) lo = mid + 1; else hi = mid;
    }
    if (lo < n && list[lo] == v) return true;
    if (n >= cap) return false;
    for (int t = n; t > lo; t--) list[t] = list[t - 1];
    list[lo] = v;
    n++;
    return true;
}

__device__ inline int find_sorted(const int32_t *list, int n, int32_t v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (list[mid] < v) lo = mid + 1; else hi = mid;
    }
    return lo;
}

constexpr int kRowCap = 256;

// Pass 1 (fill == false): count each row's distinct columns.
// Pass 2 (fill == true): write col_idx and every incidence's six in-row positions.
template <bool FILL>
__global__ void k_rows(const int32_t *__restrict__ dofs, const int32_t *__restrict__ inc_ptr,
                       const uint32_t *__restrict__ inc_elem, int64_t ndof,
                       int32_t *__restrict__ row_nnz, const int32_t *__restrict__ row_ptr,
                       int32_t *__restrict__ col_idx, uint32_t *__restrict__ inc_pos, int wide,
                       int *__restrict__ err) {
    int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (a >= ndof) return;
    int32_t list[kRowCap];
    int n = 0;
    int32_t t0 = inc_ptr[a], t1 = inc_ptr[a + 1];
    for (int32_t t = t0; t < t1; t++) {
        uint32_t e = inc_elem[t] & 0x1FFFFFFFu;
        for (int j = 0; j < 6; j++) {
            int32_t d = dofs[6 * (int64_t)e + j];
            if (d < 0) continue;
            if (!insert_sorted(list, n, kRowCap, d)) {
                atomicExch(err, 2);
                return;
            }
        }
    }
    if (!FILL) {
        row_nnz[a] = n;
        return;
    }
    int32_t base = row_ptr[a];
    for (int i = 0; i < n; i++) col_idx[base + i] = list[i];
    for (int32_t t = t0; t < t1; t++) {
        uint32_t e = inc_elem[t] & 0x1FFFFFFFu;
        if (!wide) {
            uint32_t w = 0;
            for (int j = 0; j < 6; j++) {
                int32_t d = dofs[6 * (int64_t)e + j];
                uint32_t p = d < 0 ? (uint32_t)kCompactMaxRow : (uint32_t)find_sorted(list, n, d);
                w |= p << (5 * j);
            }
            inc_pos[t] = w;
        } else {
            uint32_t w0 = 0, w1 = 0;
            for (int j = 0; j < 6; j++) {
                int32_t d = dofs[6 * (int64_t)e + j];
                uint32_t p = d < 0 ? (uint32_t)kWideMaxRow : (uint32_t)find_sorted(list, n, d);
                if (j < 4) w0 |= p << (8 * j); else w1 |= p << (8 * (j - 4));
            }
            inc_pos[2 * (int64_t)t] = w0;
            inc_pos[2 * (int64_t)t + 1] = w1;
        }
    }
}

// ---- zero dropping --------------------------------------------------------
//
// Three launches: the rows' counts and their sums within a CTA, the sums of the CTAs, the entries
// to their places. A warp takes kDropAhead rows at a time, a lane per entry (rows of a Nedelec
// matrix have 13 to 19, so a row is one coalesced load and its rank one vote), steps such groups
// one after another; CTAs of short rows take a thread per row. One thread per row walking its entries took
// 6.3 us to count and 10.4 us to copy at 28,000 rows (460,000 entries), with a device-wide scan of 7.7 us
// between them: 6.2, 7.6 and 5.6 us here. The call, with its copy back, at 60^3 hexahedra (25 M entries):
// 565 to 350 us. Without the bound on its CTAs the copying kernel takes 68 registers, three CTAs an SM: 3
// million rows of 18 entries 760 against 606 us.
constexpr int kDropThreads = 256;
constexpr int kDropAhead = 4;
constexpr int kDropStep = kDropThreads / 32 * kDropAhead;  // rows of a CTA's step
constexpr int kDropMaxSteps = kDropThreads / kDropStep;    // at most a row per thread
// A CTA of kDropMaxSteps steps with at most this many entries a row takes a thread per row: most lanes of
// a row's load would be idle. Measured, us, the call with a lane per entry / a thread per row, no zeros and
// 30 %: 3 million rows of 5 entries 553, 546 / 236, 209; of 14 628, 616 / 632, 481; of 16 653, 640 / 838, 629;
// 400,000 rows of 5 entries 89, 88 / 52, 47; of 14 111, 110 / 113, 89. (Before the lanes came, with its
// device-wide scan, one thread per row took 241, 208; 804, 575; 103, 102; 167, 141.)
constexpr int kDropShort = 14;
// Many rows: more of them per CTA, so that the sums of the CTAs (one CTA adds them) stay few.
inline int drop_steps(int64_t nrows) { return nrows < 200000 ? 1 : kDropMaxSteps; }

// COPY false: rp_out[r + 1] = nonzeros of the CTA's rows up to r. (The last of them is the CTA's
// total, at the place of the next CTA's start: k_drop_scan turns these into the starts.)
// COPY true: the start of the CTA's first row is final; the others' are added up, and the rows'
// nonzeros go to their places.
template <bool COPY>
__global__ void __launch_bounds__(kDropThreads, COPY ? 4 : 6) k_drop(const int64_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                                       const double *__restrict__ v, int64_t nrows, int steps,
                                                       int64_t *__restrict__ rp_out, int32_t *__restrict__ ci_out,
                                                       double *__restrict__ v_out) {
    using Scan = cub::BlockScan<int, kDropThreads>;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ int cnt[kDropThreads];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t r0 = blockIdx.x * (int64_t)steps * kDropStep;
    const int64_t off = COPY ? rp_out[r0] : 0;
    const int64_t r1 = r0 + (int64_t)steps * kDropStep < nrows ? r0 + (int64_t)steps * kDropStep : nrows;
    const bool short_rows = steps == kDropMaxSteps && rp[r1] - rp[r0] <= kDropShort * (r1 - r0);  // of the CTA
    if (short_rows) {
        const int64_t r = r0 + threadIdx.x, b = r < nrows ? rp[r + 1] : 0;
        int64_t o = COPY && r < nrows ? (r == r0 ? 0 : rp_out[r]) + off : 0;
        if (COPY && threadIdx.x > 0 && r < nrows) rp_out[r] = o;
        int n = 0;
        for (int64_t k = r < nrows ? rp[r] : 0; k < b; k++) {
            const double x = v[k];
            if (x != 0.0) {
                if (COPY) {
                    ci_out[o] = ci[k];
                    v_out[o] = x;
                    o++;
                }
                n++;
            }
        }
        if (!COPY) cnt[threadIdx.x] = n;
    }
    for (int st = 0; st < steps && !short_rows; st++) {
        const int i0 = st * kDropStep + warp * kDropAhead;  // row of the CTA
        int64_t a[kDropAhead], b[kDropAhead], o[kDropAhead];
        double x[kDropAhead];
        int c[kDropAhead];
#pragma unroll
        for (int u = 0; u < kDropAhead; u++) {
            const int64_t r = r0 + i0 + u;
            a[u] = r < nrows ? rp[r] : 0;
            b[u] = r < nrows ? rp[r + 1] : 0;
            o[u] = COPY && r < nrows ? (r == r0 ? 0 : rp_out[r]) + off : 0;
        }
#pragma unroll
        for (int u = 0; u < kDropAhead; u++) {
            x[u] = a[u] + lane < b[u] ? v[a[u] + lane] : 0.0;
            c[u] = COPY && a[u] + lane < b[u] ? ci[a[u] + lane] : 0;
        }
#pragma unroll
        for (int u = 0; u < kDropAhead; u++) {
            int n = 0;
            for (int64_t k = a[u];;) {  // one pass unless the row has more than 32 entries
                const unsigned m = __ballot_sync(0xffffffffu, x[u] != 0.0);
                if (COPY && x[u] != 0.0) {
                    const int64_t d = o[u] + n + __popc(m & ((1u << lane) - 1u));
                    ci_out[d] = c[u];
                    v_out[d] = x[u];
                }
                n += __popc(m);
                k += 32;
                if (k >= b[u]) break;
                x[u] = k + lane < b[u] ? v[k + lane] : 0.0;
                if (COPY) c[u] = k + lane < b[u] ? ci[k + lane] : 0;
            }
            if (!COPY && lane == 0) cnt[i0 + u] = n;
            if (COPY && lane == 0 && i0 + u > 0 && r0 + i0 + u < nrows) rp_out[r0 + i0 + u] = o[u];
        }
    }
    if (!COPY) {
        __syncthreads();
        const bool mine = (int)threadIdx.x < steps * kDropStep;
        int upto;
        Scan(tmp).InclusiveSum(mine ? cnt[threadIdx.x] : 0, upto);
        if (mine && r0 + threadIdx.x < nrows) rp_out[r0 + threadIdx.x + 1] = upto;
        if (blockIdx.x == 0 && threadIdx.x == 0) rp_out[0] = 0;
    }
}

// The totals of the nb CTAs of `rows` rows, at the starts of their successors, summed in place.
__global__ void __launch_bounds__(1024) k_drop_scan(int64_t *__restrict__ rp_out, int64_t nb, int64_t rows, int64_t nrows) {
    using Scan = cub::BlockScan<int64_t, 1024>;
    __shared__ typename Scan::TempStorage tmp;
    int64_t carry = 0;
    for (int64_t i0 = 0; i0 < nb; i0 += 1024) {
        const int64_t i = i0 + threadIdx.x, at = (i + 1) * rows < nrows ? (i + 1) * rows : nrows;
        int64_t x = i < nb ? rp_out[at] : 0, sum;
        Scan(tmp).InclusiveSum(x, x, sum);
        if (i < nb) rp_out[at] = carry + x;
        carry += sum;
        __syncthreads();
    }
}

// Device scratch that frees itself on every return path.
struct DevBuf {
    void *p = nullptr;
    cudaStream_t s = nullptr;
    explicit DevBuf(cudaStream_t st) : s(st) {}
    ~DevBuf() {
        if (p) cudaFreeAsync(p, s);
    }
    cudaError_t alloc(size_t bytes) { return cudaMallocAsync(&p, bytes ? bytes : 16, s); }
    template <class T> T *as() const { return static_cast<T *>(p); }
};

int read_flag(const int *d_err, cudaStream_t s, int *out) {
    MAG_CUDA_TRY(cudaMemcpyAsync(out, d_err, sizeof(int), cudaMemcpyDeviceToHost, s));
    MAG_CUDA_TRY(cudaStreamSynchronize(s));
    return MAG_OK;
}

}  // namespace

int generate_edges(const int32_t *d_T, int64_t ne, int64_t nn, int32_t *d_edges, int32_t *d_t2e,
                   int8_t *d_sign, int64_t *E_out, cudaStream_t s) {
    if (ne <= 0 || nn <= 0 || !d_T || !d_edges || !d_t2e || !d_sign || !E_out) {
        set_error("generate_edges: bad arguments");
        return MAG_E_ARG;
    }
    if (6 * ne >= (int64_t(1) << 32) || nn >= (int64_t(1) << 31)) {
        set_error("generate_edges: mesh too large");
        return MAG_E_UNSUPPORTED;
    }
    int64_t n = 6 * ne;
    int nb = bits_for((uint64_t)nn);
    DevBuf keys(s), keys2(s), slots(s), slots2(s), flags(s), ids(s), err(s), tmp(s);
    MAG_CUDA_TRY(keys.alloc(n * 8));
    MAG_CUDA_TRY(keys2.alloc(n * 8));
    MAG_CUDA_TRY(slots.alloc(n * 4));
    MAG_CUDA_TRY(slots2.alloc(n * 4));
    MAG_CUDA_TRY(flags.alloc(n * 4));
    MAG_CUDA_TRY(ids.alloc(n * 4));
    MAG_CUDA_TRY(err.alloc(4));
    MAG_CUDA_TRY(cudaMemsetAsync(err.p, 0, 4, s));
    k_edge_keys<<<grid_for(n), kBlock, 0, s>>>(d_T, ne, nn, nb, keys.as<uint64_t>(),
                                               slots.as<uint32_t>(), d_sign, err.as<int>());
    size_t tb = 0, tb2 = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tb, keys.as<uint64_t>(), keys2.as<uint64_t>(),
                                    slots.as<uint32_t>(), slots2.as<uint32_t>(), (int64_t)n, 0,
                                    2 * nb, s);
    cub::DeviceScan::InclusiveSum(nullptr, tb2, flags.as<int32_t>(), ids.as<int32_t>(), (int64_t)n, s);
    MAG_CUDA_TRY(tmp.alloc(tb > tb2 ? tb : tb2));
    MAG_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp.p, tb, keys.as<uint64_t>(), keys2.as<uint64_t>(),
                                                 slots.as<uint32_t>(), slots2.as<uint32_t>(),
                                                 (int64_t)n, 0, 2 * nb, s));
    k_head_flags<<<grid_for(n), kBlock, 0, s>>>(keys2.as<uint64_t>(), n, flags.as<int32_t>());
    tb2 = tb > tb2 ? tb : tb2;
    MAG_CUDA_TRY(cub::DeviceScan::InclusiveSum(tmp.p, tb2, flags.as<int32_t>(), ids.as<int32_t>(),
                                               (int64_t)n, s));
    k_edge_scatter<<<grid_for(n), kBlock, 0, s>>>(keys2.as<uint64_t>(), slots2.as<uint32_t>(),
                                                  flags.as<int32_t>(), ids.as<int32_t>(), n, nb,
                                                  d_edges, d_t2e);
    MAG_CUDA_TRY(cudaGetLastError());
    int32_t last = 0;
    MAG_CUDA_TRY(cudaMemcpyAsync(&last, ids.as<int32_t>() + (n - 1), 4, cudaMemcpyDeviceToHost, s));
    int eflag = 0;
    MAG_TRY(read_flag(err.as<int>(), s, &eflag));
    if (eflag) {
        set_error("generate_edges: node id out of range or repeated node in an element");
        return MAG_E_RANGE;
    }
    *E_out = last;
    return MAG_OK;
}

int build_pattern(const int32_t *d_dofs, int64_t ne, int64_t ndof, PatternBuffers *out,
                  cudaStream_t s) {
    *out = PatternBuffers{};
    if (ne <= 0 || ndof <= 0 || !d_dofs) {
        set_error("build_pattern: bad arguments");
        return MAG_E_ARG;
    }
    if (ne >= (int64_t(1) << 29) || ndof >= (int64_t(1) << 31) - 2) {
        set_error("build_pattern: mesh too large (elements < 2^29, dofs < 2^31 supported)");
        return MAG_E_UNSUPPORTED;
    }
    int64_t n = 6 * ne;
    int nb = bits_for((uint64_t)ndof + 1);
    DevBuf keys(s), keys2(s), vals2(s), cnt(s), err(s), tmp(s), rownnz(s), maxrow(s);
    MAG_CUDA_TRY(keys.alloc(n * 4));
    MAG_CUDA_TRY(keys2.alloc(n * 4));
    MAG_CUDA_TRY(vals2.alloc(n * 4));
    MAG_CUDA_TRY(cnt.alloc((ndof + 1) * 4));
    MAG_CUDA_TRY(err.alloc(4));
    MAG_CUDA_TRY(rownnz.alloc((ndof + 1) * 4));
    MAG_CUDA_TRY(maxrow.alloc(4));
    MAG_CUDA_TRY(cudaMemsetAsync(err.p, 0, 4, s));
    MAG_CUDA_TRY(cudaMemsetAsync(cnt.p, 0, (ndof + 1) * 4, s));
    MAG_CUDA_TRY(cudaMemsetAsync(rownnz.p, 0, (ndof + 1) * 4, s));

    MAG_CUDA_TRY(cudaMallocAsync((void **)&out->inc_ptr, (ndof + 1) * 4, s));
    MAG_CUDA_TRY(cudaMallocAsync((void **)&out->row_ptr, (ndof + 1) * 4, s));
    MAG_CUDA_TRY(cudaMallocAsync((void **)&out->inc_elem, n * 4, s));

    k_inc_keys<<<grid_for(n), kBlock, 0, s>>>(d_dofs, ne, ndof, keys.as<uint32_t>(),
                                              out->inc_elem, cnt.as<int32_t>(), err.as<int>());
    // Stable sort by dof: each row's incidences stay in ascending element order.
    size_t tb = 0, tb2 = 0, tb3 = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tb, keys.as<uint32_t>(), keys2.as<uint32_t>(),
                                    out->inc_elem, vals2.as<uint32_t>(), (int64_t)n, 0, nb, s);
    cub::DeviceScan::ExclusiveSum(nullptr, tb2, cnt.as<int32_t>(), out->inc_ptr, (int64_t)ndof + 1, s);
    cub::DeviceReduce::Max(nullptr, tb3, rownnz.as<int32_t>(), maxrow.as<int32_t>(), (int64_t)ndof, s);
    size_t tbm = tb > tb2 ? tb : tb2;
    tbm = tbm > tb3 ? tbm : tb3;
    MAG_CUDA_TRY(tmp.alloc(tbm));
    MAG_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp.p, tb, keys.as<uint32_t>(), keys2.as<uint32_t>(),
                                                 out->inc_elem, vals2.as<uint32_t>(), (int64_t)n, 0,
                                                 nb, s));
    MAG_CUDA_TRY(cudaMemcpyAsync(out->inc_elem, vals2.p, n * 4, cudaMemcpyDeviceToDevice, s));
    tb2 = tbm;
    MAG_CUDA_TRY(cub::DeviceScan::ExclusiveSum(tmp.p, tb2, cnt.as<int32_t>(), out->inc_ptr,
                                               (int64_t)ndof + 1, s));
    int32_t ninc = 0;
    MAG_CUDA_TRY(cudaMemcpyAsync(&ninc, out->inc_ptr + ndof, 4, cudaMemcpyDeviceToHost, s));
    int eflag = 0;
    MAG_TRY(read_flag(err.as<int>(), s, &eflag));
    if (eflag) {
        set_error("build_pattern: dof index out of range");
        return MAG_E_RANGE;
    }
    out->ninc = ninc;

    k_rows<false><<<grid_for(ndof, 128), 128, 0, s>>>(d_dofs, out->inc_ptr, out->inc_elem, ndof,
                                                       rownnz.as<int32_t>(), nullptr, nullptr,
                                                       nullptr, 0, err.as<int>());
    tb3 = tbm;
    MAG_CUDA_TRY(cub::DeviceReduce::Max(tmp.p, tb3, rownnz.as<int32_t>(), maxrow.as<int32_t>(),
                                        (int64_t)ndof, s));
    // row_nnz has a zero at index ndof, so the exclusive scan ends with nnz.
    tb2 = tbm;
    MAG_CUDA_TRY(cub::DeviceScan::ExclusiveSum(tmp.p, tb2, rownnz.as<int32_t>(),
                                               out->row_ptr, (int64_t)ndof + 1, s));
    int32_t nnz = 0, mx = 0;
    MAG_CUDA_TRY(cudaMemcpyAsync(&nnz, out->row_ptr + ndof, 4, cudaMemcpyDeviceToHost, s));
    MAG_CUDA_TRY(cudaMemcpyAsync(&mx, maxrow.p, 4, cudaMemcpyDeviceToHost, s));
    MAG_TRY(read_flag(err.as<int>(), s, &eflag));
    if (eflag) {
        set_error("build_pattern: a row couples more than %d dofs", kRowCap);
        return MAG_E_UNSUPPORTED;
    }
    if (mx > kWideMaxRow) {
        set_error("build_pattern: a row has %d entries (at most %d supported)", mx, kWideMaxRow);
        return MAG_E_UNSUPPORTED;
    }
    out->nnz = nnz;
    out->max_row = mx;
    out->wide = mx > kCompactMaxRow ? 1 : 0;
    MAG_CUDA_TRY(cudaMallocAsync((void **)&out->col_idx, (size_t)nnz * 4 + 16, s));
    MAG_CUDA_TRY(cudaMallocAsync((void **)&out->inc_pos, (size_t)ninc * 4 * (out->wide ? 2 : 1) + 16, s));
    k_rows<true><<<grid_for(ndof, 128), 128, 0, s>>>(d_dofs, out->inc_ptr, out->inc_elem, ndof,
                                                      nullptr, out->row_ptr, out->col_idx,
                                                      out->inc_pos, out->wide, err.as<int>());
    MAG_CUDA_TRY(cudaGetLastError());
    MAG_CUDA_TRY(cudaStreamSynchronize(s));
    return MAG_OK;
}

void free_pattern(PatternBuffers *p, cudaStream_t s) {
    void *ptrs[] = {p->row_ptr, p->col_idx, p->inc_ptr, p->inc_elem, p->inc_pos};
    for (void *q : ptrs)
        if (q) cudaFreeAsync(q, s);
    *p = PatternBuffers{};
}

int csr_drop_zeros(const int64_t *rp, const int32_t *ci, const double *v, int64_t nrows,
                   int64_t *rp_out, int32_t *ci_out, double *v_out, int64_t *nnz_out,
                   cudaStream_t s) {
    if (nrows <= 0 || !rp || !ci || !v || !rp_out || !ci_out || !v_out || !nnz_out) {
        set_error("csr_drop_zeros: bad arguments");
        return MAG_E_ARG;
    }
    const int steps = drop_steps(nrows), rows = steps * kDropStep;
    const int64_t nb = (nrows + rows - 1) / rows;
    k_drop<false><<<(unsigned)nb, kDropThreads, 0, s>>>(rp, ci, v, nrows, steps, rp_out, nullptr, nullptr);
    k_drop_scan<<<1, 1024, 0, s>>>(rp_out, nb, rows, nrows);
    k_drop<true><<<(unsigned)nb, kDropThreads, 0, s>>>(rp, ci, v, nrows, steps, rp_out, ci_out, v_out);
    MAG_CUDA_TRY(cudaGetLastError());
    MAG_CUDA_TRY(cudaMemcpyAsync(nnz_out, rp_out + nrows, 8, cudaMemcpyDeviceToHost, s));
    MAG_CUDA_TRY(cudaStreamSynchronize(s));
    return MAG_OK;
}

}  // namespace mag
