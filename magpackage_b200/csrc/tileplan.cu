// Tile plan of a mesh (tile.cuh), built on the GPU from its incidence plan.
//
//   layers   the node coordinates of each axis, sorted; a layer ends where consecutive values
//            lie more than 0.3 h apart or it would span more than h, h = (volume / Nn)^(1/3)
//   rows     the tile of a row is that of its edge's lower node; rows sorted by tile (stable),
//            tiles cut into blocks of at most kTileMaxNnz nonzeros, kTileMaxInc incidences and
//            kTileMaxRows rows
//   records  the incidences sorted by (block, element): one record per group
//   colours  per block, one CTA: which records share an off-diagonal slot, a two-colouring of
//            that graph by label propagation (smallest record of the component, parity of the
//            distance to it), or, where the graph is not bipartite, the smallest free colour in
//            element order
//   fill     records by colour, then element, into the six planes
//
// The host planner this replaces downloaded the mesh and ran on the host threads: 62 to 80 ms at
// 40^3 hexahedra, 230 to 300 ms at 60^3 and 1.7 s at 110^3 on 16 threads; here 1.9, 3.5 and 11 ms.
#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "tile.cuh"

namespace mag {

namespace {

constexpr int kPB = 256;         // threads of the per-block kernels
constexpr int kLayerB = 1024;    // threads of the layer walk
// Node layers per tile: the first of these forms whose tiles, and the blocks they are cut into, are
// few enough, the last one otherwise. A block's time is latency: where blocks would leave SMs idle (148 on the GPU),
// smaller ones finish sooner although they evaluate more elements twice (4x2x2 up to 1.9 times an
// element, 3x3x3 1.67, 4x4x4 1.5). Measured on the device alone, us, with 4x4x4 / as chosen here:
// Jacobian at 8^3 hexahedra (4x2x2) 14.9 / 10.3, 14^3 (3x3x3) 15.5 / 11.4, 16^3 15.7 / 12.5; M(1)
// 18.6 / 10.5, 18.8 / 13.0, 19.0 / 14.9; at 20^3, where 4x4x4 stays, 3x3x3 has Jacobian 14.5
// against 16.3 but at 24^3 23.3 against 20.0. Where tiles hold so many rows that a colour class is
// more than kTileSmallThreads elements, a block is no small one, and one wave of them is the limit:
// graded 16^3 (136 blocks) 11.5 against 14.2, 20^3 (232) 17.5 against 18.1 but M(1) 28.3 against 27.2,
// 24^3 (335) 24.5 against 19.9.
struct TileForm {
    int l[3];
    int64_t most;
};
constexpr int kOneWave = 148;
constexpr int kNumForms = 3;
constexpr TileForm kTileForms[kNumForms] = {{{4, 2, 2}, kOneWave}, {{3, 3, 3}, 2 * kOneWave}, {{4, 4, 4}, INT64_MAX}};
constexpr uint32_t kNone16 = 0xFFFFu;

unsigned grid1(int64_t n, int b = 256) { return (unsigned)((n + b - 1) / b); }

int bits_of(uint64_t n) {  // bits that hold 0 .. n - 1
    int b = 1;
    while (b < 64 && (uint64_t(1) << b) < n) b++;
    return b;
}

// Stats and flags the host reads.
struct PlanInfo {
    unsigned long long lo[3], hi[3];  // coordinate bounds as ordered integers
    int last_layer[3];
    int unused_rows;   // rows without incidences
    int fail;          // the mesh does not suit the schedule
    int nblocks, nchunks, nrec;
    int max_nnz, max_inc, max_colors, max_rows, max_chunks, max_class;
};

__host__ __device__ inline unsigned long long ordered(double x) {
    unsigned long long b;
    memcpy(&b, &x, 8);
    return (b >> 63) ? ~b : b | (1ull << 63);
}
double unordered(unsigned long long k) {
    const unsigned long long b = (k >> 63) ? k & ~(1ull << 63) : ~k;
    double x;
    memcpy(&x, &b, 8);
    return x;
}

// Workspace: pieces of one device range, and stream-ordered allocations beyond it.
class Arena {
public:
    Arena(void *base, size_t bytes, cudaStream_t s) : p_(static_cast<char *>(base)), left_(base ? bytes : 0), s_(s) {}
    ~Arena() {
        for (void *p : more_) cudaFreeAsync(p, s_);
    }
    template <typename T>
    bool get(T **out, size_t n) {
        const size_t b = (std::max<size_t>(n, 1) * sizeof(T) + 255) & ~size_t(255);
        if (b <= left_) {
            *out = reinterpret_cast<T *>(p_);
            p_ += b;
            left_ -= b;
            return true;
        }
        void *q = nullptr;
        if (cudaMallocAsync(&q, b, s_) != cudaSuccess) return false;
        more_.push_back(q);
        *out = static_cast<T *>(q);
        return true;
    }

private:
    char *p_;
    size_t left_;
    cudaStream_t s_;
    std::vector<void *> more_;
};

// ---- layers -------------------------------------------------------------------------

// Coordinates by axis and their bounds.
__global__ void k_axes(const double4 *__restrict__ xyz, int64_t nn, double *__restrict__ c, PlanInfo *__restrict__ info) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    unsigned long long lo[3], hi[3];
    const double4 p = i < nn ? xyz[i] : xyz[0];
    const double v[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        if (i < nn) c[a * nn + i] = v[a];
        lo[a] = hi[a] = ordered(v[a]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long l = __shfl_xor_sync(0xffffffffu, lo[a], o), h = __shfl_xor_sync(0xffffffffu, hi[a], o);
            lo[a] = l < lo[a] ? l : lo[a];
            hi[a] = h > hi[a] ? h : hi[a];
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&info->lo[a], lo[a]);
            atomicMax(&info->hi[a], hi[a]);
        }
    }
}

// One CTA per axis walks the sorted coordinates: thr[axis][k] is the first coordinate of layer
// k + 1. The rule looks at the start of the running layer, so layers follow one another; within
// a layer the CTA looks at kLayerB coordinates at a time.
__global__ void __launch_bounds__(kLayerB) k_layers(const double *__restrict__ sorted, int64_t nn, double h,
                                                    double *__restrict__ thr, PlanInfo *__restrict__ info) {
    __shared__ int first;
    const double *x = sorted + blockIdx.x * nn;
    double *out = thr + blockIdx.x * nn;
    double start = x[0];
    int layers = 0;
    for (int64_t base = 1; base < nn;) {
        const int64_t i = base + threadIdx.x;
        if (threadIdx.x == 0) first = kLayerB;
        __syncthreads();
        if (i < nn) {
            const double v = x[i];
            if (v - x[i - 1] > 0.3 * h || v - start > h) atomicMin(&first, (int)threadIdx.x);
        }
        __syncthreads();
        const int f = first;
        __syncthreads();
        if (f == kLayerB) {
            base += kLayerB;
        } else {
            start = x[base + f];
            if (threadIdx.x == 0) out[layers] = start;
            layers++;
            base += f + 1;
        }
    }
    if (threadIdx.x == 0) info->last_layer[blockIdx.x] = layers;
}

// ---- rows and blocks ----------------------------------------------------------------

struct TileGrid {
    int n[3];  // tiles per axis
    int l[3];  // node layers per tile
};

__device__ __forceinline__ int layer_of(const double *__restrict__ thr, int n, double x) {
    int lo = 0, hi = n;  // layers started at or before x
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (thr[mid] <= x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__global__ void k_node_tiles(const double4 *__restrict__ xyz, int64_t nn, const double *__restrict__ thr,
                             const PlanInfo *__restrict__ info, TileGrid g, uint32_t *__restrict__ tile) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nn) return;
    const double4 p = xyz[i];
    const double v[3] = {p.x, p.y, p.z};
    int t[3];
#pragma unroll
    for (int a = 0; a < 3; a++) t[a] = layer_of(thr + a * nn, info->last_layer[a], v[a]) / g.l[a];
    tile[i] = (uint32_t)(t[0] + g.n[0] * (t[1] + g.n[1] * t[2]));
}

// Tile of each row; last[r] = r, or -1 for a row without incidences (it joins the tile of the
// row before it).
__global__ void k_row_tiles(TilePlanInput in, const uint32_t *__restrict__ node_tile, uint32_t *__restrict__ tile,
                            uint32_t *__restrict__ row, int *__restrict__ last, PlanInfo *__restrict__ info) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= in.ndof) return;
    const int32_t i0 = in.inc_ptr[r], i1 = in.inc_ptr[r + 1];
    uint32_t t = 0;
    if (i1 > i0) {
        const uint32_t ew = in.inc_elem[i0];
        const int l = (int)(ew >> 29);
        const int4 q = in.tet[ew & 0x1FFFFFFFu];
        const int n[4] = {q.x, q.y, q.z, q.w};
        int na = 0, nb = 0;
#pragma unroll
        for (int k = 0; k < 6; k++)
            if (k == l) {
                na = n[edge_a(k)];
                nb = n[edge_b(k)];
            }
        t = node_tile[na < nb ? na : nb];
    } else {
        atomicAdd(&info->unused_rows, 1);
    }
    if (in.row_ptr[r + 1] - in.row_ptr[r] > kCompactMaxRow || i1 - i0 > kCompactMaxRow) info->fail = 1;
    tile[r] = t;
    row[r] = (uint32_t)r;
    last[r] = i1 > i0 ? (int)r : -1;
}

struct MaxOp {
    __device__ __forceinline__ int operator()(int a, int b) const { return a > b ? a : b; }
};

__global__ void k_join_unused(int64_t ndof, const int *__restrict__ last, uint32_t *__restrict__ tile) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= ndof || last[r] == (int)r) return;
    tile[r] = last[r] < 0 ? 0u : tile[last[r]];  // (the tile of a used row is not written here)
}

// An element with a repeated dof would update a diagonal slot or one slot twice.
__global__ void k_repeated_dofs(const int32_t *__restrict__ dofs, int64_t ne, PlanInfo *__restrict__ info) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= ne) return;
    const int2 *p = reinterpret_cast<const int2 *>(dofs + 6 * e);
    const int2 a = p[0], b = p[1], c = p[2];
    const int d[6] = {a.x, a.y, b.x, b.y, c.x, c.y};
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
        for (int j = i + 1; j < 6; j++)
            if (d[i] >= 0 && d[i] == d[j]) info->fail = 1;
}

// Nonzeros and incidences of the rows in tile order (scanned afterwards; zero at the end).
__global__ void k_row_sizes(TilePlanInput in, const uint32_t *__restrict__ order, int *__restrict__ nn, int *__restrict__ ni) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k > in.ndof) return;
    const int64_t r = k < in.ndof ? order[k] : 0;
    nn[k] = k < in.ndof ? in.row_ptr[r + 1] - in.row_ptr[r] : 0;
    ni[k] = k < in.ndof ? in.inc_ptr[r + 1] - in.inc_ptr[r] : 0;
}

__device__ __forceinline__ int64_t lower_bound_u32(const uint32_t *__restrict__ a, int64_t n, uint32_t v) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The blocks of each tile: as many rows as fit, in order. pn, pi: nonzeros and incidences before
// a row. WRITE: start rows at off[tile]; else their number.
template <bool WRITE>
__global__ void k_cut_tiles(int64_t ntiles, int64_t ndof, const uint32_t *__restrict__ sorted_tile,
                            const int *__restrict__ pn, const int *__restrict__ pi, int *__restrict__ cnt,
                            const int *__restrict__ off, int *__restrict__ bstart) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t > ntiles) return;
    if (t == ntiles) {
        if (WRITE) bstart[off[ntiles]] = (int)ndof;
        else cnt[t] = 0;
        return;
    }
    int64_t k = lower_bound_u32(sorted_tile, ndof, (uint32_t)t);
    const int64_t k1 = t + 1 < ntiles ? lower_bound_u32(sorted_tile, ndof, (uint32_t)t + 1) : ndof;
    int n = 0;
    while (k < k1) {
        if (WRITE) bstart[off[t] + n] = (int)k;
        n++;
        int64_t lo = k + 1, hi = k1;  // the last end that fits (one row always does)
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) >> 1;
            if (pn[mid] - pn[k] <= kTileMaxNnz && pi[mid] - pi[k] <= kTileMaxInc && mid - k <= kTileMaxRows) lo = mid;
            else hi = mid - 1;
        }
        k = lo;
    }
    if (!WRITE) cnt[t] = n;
}

// One CTA per block: the row table, the sort keys (block, element) and slot words of its
// incidences, and the number of its store chunks. A chunk starts where a run of consecutive rows
// starts and every kTileChunk nonzeros after that; the row that holds a chunk's first nonzero
// owns it. WRITE_CHUNKS: the chunks themselves at chunk0[b] instead.
template <bool WRITE_CHUNKS>
__global__ void __launch_bounds__(kPB) k_block_rows(TilePlanInput in, const uint32_t *__restrict__ order,
                                                    const int *__restrict__ bstart, const int *__restrict__ pn,
                                                    const int *__restrict__ pi, int elem_bits, uint2 *__restrict__ rows,
                                                    uint64_t *__restrict__ keys, uint32_t *__restrict__ inc,
                                                    uint32_t *__restrict__ slotw, int *__restrict__ nchunks,
                                                    const int *__restrict__ chunk0, uint2 *__restrict__ chunks,
                                                    PlanInfo *__restrict__ info) {
    using Scan = cub::BlockScan<int, kPB>;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ int run_carry, own_carry;
    const int b = blockIdx.x, k0 = bstart[b], k1 = bstart[b + 1];
    const int n0 = pn[k0], i0 = pi[k0], bnnz = pn[k1] - n0;
    if (threadIdx.x == 0) {
        run_carry = 0;
        own_carry = 0;
    }
    __syncthreads();
    for (int kb = k0; kb < k1; kb += kPB) {
        const int k = kb + threadIdx.x;
        const bool in_block = k < k1;
        const uint32_t r = in_block ? order[k] : 0;
        const int bn = in_block ? pn[k] - n0 : 0, rn = in_block ? pn[k + 1] - n0 - bn : 0;
        // start (in the block's nonzeros) of the run of consecutive rows this row belongs to
        const bool head = in_block && (k == k0 || order[k - 1] + 1 != r);
        int run;
        Scan(tmp).InclusiveScan(head ? bn : 0, run, MaxOp());
        run = run > run_carry ? run : run_carry;
        __syncthreads();
        const int o = bn - run;
        const int own = (o + rn + kTileChunk - 1) / kTileChunk - (o + kTileChunk - 1) / kTileChunk;
        int before, total;
        Scan(tmp).ExclusiveSum(in_block ? own : 0, before, total);
        before += own_carry;
        __syncthreads();
        if (threadIdx.x == kPB - 1) run_carry = run;
        if (threadIdx.x == 0) own_carry += total;
        if (WRITE_CHUNKS) {
            for (int j = 0; in_block && j < own; j++) {
                const int s = run + ((o + kTileChunk - 1) / kTileChunk + j) * kTileChunk;  // in the block
                chunks[chunk0[b] + before + j] = make_uint2((uint32_t)s, (uint32_t)(in.row_ptr[r] + (s - bn)));
            }
        } else if (in_block) {
            const int bi = pi[k] - i0;
            const int32_t t0 = in.inc_ptr[r], t1 = in.inc_ptr[r + 1];
            uint32_t diag = 0;
            for (int32_t t = t0; t < t1; t++) {
                const uint32_t ew = in.inc_elem[t];
                if (t == t0) diag = (in.inc_pos[t] >> (5 * (ew >> 29))) & 31u;
                keys[t] = ((uint64_t)b << elem_bits) | (ew & 0x1FFFFFFFu);
                inc[t] = (uint32_t)t;
                slotw[t] = (uint32_t)bn | ((uint32_t)(bi + (t - t0)) << 16);
            }
            rows[k] = make_uint2(r, (uint32_t)bn | ((uint32_t)bi << 13) | (diag << 25));
        }
        __syncthreads();
    }
    if (WRITE_CHUNKS) {  // lengths: the chunks tile the block's nonzeros
        const int nc = own_carry, c0 = chunk0[b];
        __syncthreads();
        for (int cb = 0; cb < nc; cb += kPB) {
            const int c = cb + threadIdx.x;
            uint2 ch = make_uint2(0, 0);
            uint32_t end = 0;
            if (c < nc) {
                ch = chunks[c0 + c];
                end = c + 1 < nc ? chunks[c0 + c + 1].x & 0xFFFFu : (uint32_t)bnnz;
            }
            __syncthreads();
            if (c < nc) chunks[c0 + c].x = ch.x | ((end - ch.x) << 16);
            __syncthreads();
        }
    } else if (threadIdx.x == 0) {
        nchunks[b] = own_carry;
        atomicMax(&info->max_chunks, own_carry);
        atomicMax(&info->max_rows, k1 - k0);
        atomicMax(&info->max_nnz, bnnz);
        atomicMax(&info->max_inc, pi[k1] - i0);
    }
}

// ---- records ------------------------------------------------------------------------

__global__ void k_record_heads(const uint64_t *__restrict__ keys, int64_t n, int *__restrict__ head) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) head[i] = i == 0 || keys[i] != keys[i - 1] ? 1 : 0;
}

// rec[i] = record of sorted incidence i, plus one (inclusive sum of the heads).
__global__ void k_record_starts(const uint64_t *__restrict__ keys, int64_t n, const int *__restrict__ rec,
                                const uint32_t *__restrict__ inc, const uint32_t *__restrict__ inc_elem,
                                int *__restrict__ start, PlanInfo *__restrict__ info) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (i == 0 || keys[i] != keys[i - 1]) start[rec[i] - 1] = (int)i;
    if (i + 1 == n) {
        start[rec[i]] = (int)n;
        info->nrec = rec[i];
    }
    // one element twice in a row's incidences at the same local row
    const uint32_t l = inc_elem[inc[i]] >> 29;
    for (int64_t j = i - 1; j >= 0 && i - j < 7 && keys[j] == keys[i]; j--)
        if ((inc_elem[inc[j]] >> 29) == l) info->fail = 1;
}

struct ColorSmem {
    uint32_t own[kTileMaxNnz + 1];  // records of a slot: first | second << 16 (kNone16: none)
    uint32_t label[kTileMaxInc + 1];  // smallest record of the component << 1 | parity of the distance
    uint32_t comp[kTileMaxInc + 1];   // per component: records of parity 0 | of parity 1 << 16; then its flip
    uint8_t color[kTileMaxInc + 1];
    int col_end[kTileMaxColors];
    int ncolors, bad;
};

// One CTA per block: colours of its records, their places (pos: record -> place in the planes)
// and the block's descriptor.
__global__ void __launch_bounds__(kPB) k_color_blocks(TilePlanInput in, const int *__restrict__ bstart,
                                                      const int *__restrict__ pn, const int *__restrict__ pi,
                                                      const int *__restrict__ rec, const int *__restrict__ rec_start,
                                                      const uint32_t *__restrict__ inc, const uint32_t *__restrict__ slotw,
                                                      const int *__restrict__ nchunks, const int *__restrict__ chunk0,
                                                      TileBlock *__restrict__ blocks, int *__restrict__ pos,
                                                      PlanInfo *__restrict__ info) {
    extern __shared__ __align__(16) unsigned char plan_smem[];
    ColorSmem &S = *reinterpret_cast<ColorSmem *>(plan_smem);
    using Scan = cub::BlockScan<int, kPB>;
    __shared__ typename Scan::TempStorage tmp;
    const int b = blockIdx.x, tid = threadIdx.x, k0 = bstart[b], k1 = bstart[b + 1];
    const int i0 = pi[k0], i1 = pi[k1], nnz = pn[k1] - pn[k0];
    const int rec0 = i1 > i0 ? rec[i0] - 1 : i0 > 0 ? rec[i0 - 1] : 0;
    const int nr = i1 > i0 ? rec[i1 - 1] - rec0 : 0;
    for (int i = tid; i < nnz; i += kPB) S.own[i] = kNone16 | (kNone16 << 16);
    for (int i = tid; i < nr; i += kPB) {
        S.label[i] = (uint32_t)i << 1;
        S.comp[i] = 0;
        S.color[i] = 0xFF;
    }
    if (tid == 0) {
        S.ncolors = 2;
        S.bad = 0;
    }
    __syncthreads();
    // the records of each off-diagonal slot: at most two
    for (int i = i0 + tid; i < i1; i += kPB) {
        const uint32_t t = inc[i], ew = in.inc_elem[t], pw = in.inc_pos[t], base = slotw[t] & 0xFFFFu;
        const uint32_t me = (uint32_t)(rec[i] - 1 - rec0);
        const int l = (int)(ew >> 29);
        for (int j = 0; j < 6; j++) {
            const uint32_t p = (pw >> (5 * j)) & 31u;
            if (j == l || p == (uint32_t)kCompactMaxRow) continue;
            const uint32_t sl = base + p;
            if (sl >= (uint32_t)nnz) {
                S.bad = 1;
                continue;
            }
            uint32_t old = atomicCAS(&S.own[sl], kNone16 | (kNone16 << 16), me | (kNone16 << 16));
            if (old != (kNone16 | (kNone16 << 16))) {
                if ((old >> 16) != kNone16 || atomicCAS(&S.own[sl], old, (old & 0xFFFFu) | (me << 16)) != old) S.bad = 1;
            }
        }
    }
    __syncthreads();
    if (S.bad) {  // a third contribution: the schedule does not suit (no colours needed)
        if (tid == 0) info->fail = 1;
        return;
    }
    // labels to the smallest of each component
    for (;;) {
        int changed = 0;
        for (int i = tid; i < nnz; i += kPB) {
            const uint32_t w = S.own[i], a = w & 0xFFFFu, c = w >> 16;
            if (c == kNone16) continue;
            const uint32_t la = S.label[a], lc = S.label[c];
            if ((la ^ 1u) < lc) {
                atomicMin(&S.label[c], la ^ 1u);
                changed = 1;
            } else if ((lc ^ 1u) < la) {
                atomicMin(&S.label[a], lc ^ 1u);
                changed = 1;
            }
        }
        if (!__syncthreads_or(changed)) break;
    }
    int odd = 0;
    for (int i = tid; i < nnz; i += kPB) {
        const uint32_t w = S.own[i], a = w & 0xFFFFu, c = w >> 16;
        if (c != kNone16 && ((S.label[a] ^ S.label[c]) & 1u) == 0) odd = 1;
    }
    const bool two = !__syncthreads_or(odd);
    if (two) {  // components flipped, in order, to balance the classes
        for (int i = tid; i < nr; i += kPB) atomicAdd(&S.comp[S.label[i] >> 1], (S.label[i] & 1u) ? 0x10000u : 1u);
        __syncthreads();
        if (tid < 32) {
            int diff = 0;  // records of colour 0 minus records of colour 1 so far
            for (int ib = 0; ib < nr; ib += 32) {
                const int i = ib + tid;
                const int d = i < nr ? (int)(S.comp[i] & 0xFFFFu) - (int)(S.comp[i] >> 16) : 0;
                unsigned roots = __ballot_sync(0xffffffffu, i < nr && S.comp[i] != 0);
                unsigned flips = 0;
                while (roots) {
                    const int j = __ffs(roots) - 1;
                    roots &= roots - 1;
                    const int dj = __shfl_sync(0xffffffffu, d, j);
                    const bool f = abs(diff - dj) < abs(diff + dj);
                    flips |= (f ? 1u : 0u) << j;
                    diff += f ? -dj : dj;
                }
                __syncwarp();
                if (i < nr) S.comp[i] = (flips >> tid) & 1u;
            }
        }
        __syncthreads();
        for (int i = tid; i < nr; i += kPB) S.color[i] = (uint8_t)((S.label[i] & 1u) ^ S.comp[S.label[i] >> 1]);
    } else if (tid < 32) {  // one warp: the smallest colour none of the sharing records has, in element order
        int ncol = 0;
        for (int u = 0; u < nr; u++) {
            const int q0 = rec_start[rec0 + u], q1 = rec_start[rec0 + u + 1];
            unsigned used = 0;
            for (int x = tid; x < 5 * (q1 - q0); x += 32) {
                const uint32_t t = inc[q0 + x / 5];
                const int l = (int)(in.inc_elem[t] >> 29), jj = x % 5, j = jj < l ? jj : jj + 1;
                const uint32_t p = (in.inc_pos[t] >> (5 * j)) & 31u;
                if (p == (uint32_t)kCompactMaxRow) continue;
                const uint32_t w = S.own[(slotw[t] & 0xFFFFu) + p];
                const uint32_t other = (w & 0xFFFFu) == (uint32_t)u ? w >> 16 : w & 0xFFFFu;
                if (other != kNone16 && S.color[other] < 32) used |= 1u << S.color[other];
            }
            used = __reduce_or_sync(0xffffffffu, used);
            const int c = used == 0xFFFFFFFFu ? 32 : __ffs(~used) - 1;
            if (tid == 0) S.color[u] = (uint8_t)c;
            ncol = c + 1 > ncol ? c + 1 : ncol;
            __syncwarp();
        }
        if (tid == 0) S.ncolors = ncol;
    }
    __syncthreads();
    const int ncol = S.ncolors;
    if (ncol > kTileMaxColors) {
        if (tid == 0) info->fail = 1;
        return;
    }
    // places: by colour, then record (ascending element)
    int base = 0;
    for (int c = 0; c < kTileMaxColors; c++) {
        if (c < ncol) {
            for (int ib = 0; ib < nr; ib += kPB) {
                const int i = ib + tid;
                const int mine = i < nr && S.color[i] == c;
                int before, total;
                Scan(tmp).ExclusiveSum(mine, before, total);
                if (mine) pos[rec0 + i] = rec0 + base + before;
                base += total;
                __syncthreads();
            }
        }
        if (tid == 0) S.col_end[c] = c < ncol ? base : 0;
    }
    __syncthreads();
    if (tid == 0) {
        TileBlock B{};
        B.row0 = k0;
        B.nrows = k1 - k0;
        B.rec0 = rec0;
        B.nrec = nr;
        B.chunk0 = chunk0[b];
        B.nchunks = nchunks[b];
        B.nnz = nnz;
        B.ninc = i1 - i0;
        B.ncolors = ncol;
        int most = 0;
        for (int c = 0; c < kTileMaxColors; c++) {
            B.col_end[c] = S.col_end[c];
            if (c < ncol) most = max(most, S.col_end[c] - (c > 0 ? S.col_end[c - 1] : 0));
        }
        blocks[b] = B;
        atomicMax(&info->max_colors, ncol);
        atomicMax(&info->max_class, most);
    }
}

// The records' six planes. An absent column (a dof of -1) of a row points at the row's own
// diagonal nonzero: the kernels add its discarded value there without a test, and the row phase
// overwrites that slot with the diagonal's element-ordered sum afterwards.
__global__ void k_fill_records(TilePlanInput in, int64_t nrec, const int *__restrict__ rec_start,
                               const uint64_t *__restrict__ keys, uint64_t elem_mask, const uint32_t *__restrict__ inc,
                               const uint32_t *__restrict__ slotw, const int *__restrict__ pos, uint4 *__restrict__ recs) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nrec) return;
    const int q0 = rec_start[i], q1 = rec_start[i + 1];
    const int64_t e = (int64_t)(keys[q0] & elem_mask);
    const int4 tt = in.tet[e];
    const int2 *dp = reinterpret_cast<const int2 *>(in.dofs + 6 * e);
    const int2 d0 = dp[0], d1 = dp[1], d2 = dp[2];
    unsigned sb = 0;
    if (in.signbits) {
        sb = in.signbits[e];
    } else {
        const int n[4] = {tt.x, tt.y, tt.z, tt.w};
#pragma unroll
        for (int k = 0; k < 6; k++) sb |= (n[edge_a(k)] < n[edge_b(k)] ? 0u : 1u) << k;
    }
    uint32_t pw[6] = {0, 0, 0, 0, 0, 0}, sl[6];
#pragma unroll
    for (int l = 0; l < 6; l++) sl[l] = kTileAbsent;
    for (int q = q0; q < q1; q++) {
        const uint32_t t = inc[q];
        const int l = (int)(in.inc_elem[t] >> 29);
        uint32_t w = in.inc_pos[t];
        const uint32_t diag = (w >> (5 * l)) & 31u;
#pragma unroll
        for (int j = 0; j < 6; j++)
            if (((w >> (5 * j)) & 31u) == (uint32_t)kCompactMaxRow) w = (w & ~(31u << (5 * j))) | (diag << (5 * j));
        const uint32_t s = slotw[t];
#pragma unroll
        for (int k = 0; k < 6; k++)
            if (k == l) {
                pw[k] = w;
                sl[k] = s;
            }
    }
    uint4 *dst = recs + pos[i];
    dst[0] = make_uint4((uint32_t)tt.x, (uint32_t)tt.y, (uint32_t)tt.z, (uint32_t)tt.w);
    dst[nrec] = make_uint4((uint32_t)d0.x, (uint32_t)d0.y, (uint32_t)d1.x, (uint32_t)d1.y);
    dst[2 * nrec] = make_uint4((uint32_t)d2.x, (uint32_t)d2.y, (uint32_t)e, (uint32_t)in.tags[e] | (sb << 8));
    dst[3 * nrec] = make_uint4(pw[0], pw[1], pw[2], pw[3]);
    dst[4 * nrec] = make_uint4(pw[4], pw[5], sl[0], sl[1]);
    dst[5 * nrec] = make_uint4(sl[2], sl[3], sl[4], sl[5]);
}

int read_info(const PlanInfo *d, PlanInfo *h, cudaStream_t s) {
    MAG_CUDA_TRY(cudaMemcpyAsync(h, d, sizeof(PlanInfo), cudaMemcpyDeviceToHost, s));
    MAG_CUDA_TRY(cudaStreamSynchronize(s));
    return MAG_OK;
}

// CUB's two-call form with a shared temporary buffer.
struct CubTemp {
    void *p = nullptr;
    size_t bytes = 0;
    bool need(Arena &a, size_t b) {
        if (b <= bytes) return true;
        char *q = nullptr;
        if (!a.get(&q, b)) return false;
        p = q;
        bytes = b;
        return true;
    }
};
#define MAG_CUB(call)                                                  \
    do {                                                               \
        size_t cub_bytes = 0;                                          \
        {                                                              \
            void *cub_p = nullptr;                                     \
            MAG_CUDA_TRY(call);                                        \
        }                                                              \
        if (!temp.need(arena, cub_bytes)) return MAG_E_NOMEM;          \
        cub_bytes = temp.bytes;                                        \
        {                                                              \
            void *cub_p = temp.p;                                      \
            MAG_CUDA_TRY(call);                                        \
        }                                                              \
    } while (0)
#define MAG_GET(ptr, n) \
    do {                \
        if (!arena.get(&ptr, n)) return MAG_E_NOMEM; \
    } while (0)

// The plan with the first form from *form on whose tiles are few enough. p->ok stays 0 where the mesh
// does not suit the schedule (*form is then kNumForms) or where the form's blocks turn out too many or
// too large (*form is the next one to try).
int build(const TilePlanInput &in, void *work, size_t work_bytes, int *form, TilePlan *p, cudaStream_t s) {
    int k = *form;
    *form = kNumForms;
    Arena arena(work, work_bytes, s);
    CubTemp temp;
    const int64_t nn = in.nn, ne = in.ne, ndof = in.ndof, ninc = in.ninc;
    PlanInfo *info = nullptr, hi{};
    MAG_GET(info, 1);
    for (int a = 0; a < 3; a++) hi.lo[a] = ~0ull;
    MAG_CUDA_TRY(cudaMemcpyAsync(info, &hi, sizeof hi, cudaMemcpyHostToDevice, s));
    double *coord = nullptr, *sorted = nullptr;
    MAG_GET(coord, 3 * nn);
    MAG_GET(sorted, 3 * nn);
    k_repeated_dofs<<<grid1(ne), 256, 0, s>>>(in.dofs, ne, info);
    k_axes<<<grid1(nn), 256, 0, s>>>(in.xyz, nn, coord, info);
    for (int a = 0; a < 3; a++)
        MAG_CUB(cub::DeviceRadixSort::SortKeys(cub_p, cub_bytes, coord + a * nn, sorted + a * nn, nn, 0, 64, s));
    MAG_TRY(read_info(info, &hi, s));
    double vol = 1.0, ext_max = 0.0;
    for (int a = 0; a < 3; a++) {
        const double ext = unordered(hi.hi[a]) - unordered(hi.lo[a]);
        vol *= ext;
        ext_max = std::max(ext_max, ext);
    }
    double h = vol > 0.0 ? std::cbrt(vol / (double)nn) : ext_max / std::max(1.0, std::cbrt((double)nn));
    if (!(h > 0.0)) h = 1.0;
    double *thr = coord;  // the unsorted coordinates are used up
    k_layers<<<3, kLayerB, 0, s>>>(sorted, nn, h, thr, info);
    MAG_TRY(read_info(info, &hi, s));
    if (hi.fail) return MAG_OK;
    TileGrid g;
    int64_t tiles = 1;
    for (;; k++) {
        const TileForm &f = kTileForms[k];
        tiles = 1;
        for (int a = 0; a < 3; a++) {
            g.l[a] = f.l[a];
            g.n[a] = hi.last_layer[a] / f.l[a] + 1;
            tiles *= g.n[a];
            if (tiles >= (int64_t(1) << 31)) return MAG_OK;
        }
        if (tiles <= f.most) break;
    }
    const bool small = k + 1 < kNumForms;
    uint32_t *node_tile = nullptr, *tile = nullptr, *tile_s = nullptr, *row = nullptr, *order = nullptr;
    int *last = nullptr, *pn = nullptr, *pi = nullptr;
    MAG_GET(node_tile, nn);
    MAG_GET(tile, ndof);
    MAG_GET(tile_s, ndof);
    MAG_GET(row, ndof);
    MAG_GET(order, ndof);
    MAG_GET(last, ndof);
    MAG_GET(pn, ndof + 1);
    MAG_GET(pi, ndof + 1);
    k_node_tiles<<<grid1(nn), 256, 0, s>>>(in.xyz, nn, thr, info, g, node_tile);
    k_row_tiles<<<grid1(ndof), 256, 0, s>>>(in, node_tile, tile, row, last, info);
    MAG_TRY(read_info(info, &hi, s));
    if (hi.fail) return MAG_OK;
    if (hi.unused_rows) {
        MAG_CUB(cub::DeviceScan::InclusiveScan(cub_p, cub_bytes, last, last, MaxOp(), ndof, s));
        k_join_unused<<<grid1(ndof), 256, 0, s>>>(ndof, last, tile);
    }
    MAG_CUB(cub::DeviceRadixSort::SortPairs(cub_p, cub_bytes, tile, tile_s, row, order, ndof, 0, bits_of((uint64_t)tiles), s));
    k_row_sizes<<<grid1(ndof + 1), 256, 0, s>>>(in, order, pn, pi);
    MAG_CUB(cub::DeviceScan::ExclusiveSum(cub_p, cub_bytes, pn, pn, ndof + 1, s));
    MAG_CUB(cub::DeviceScan::ExclusiveSum(cub_p, cub_bytes, pi, pi, ndof + 1, s));
    int *tcnt = nullptr, *bstart = nullptr;
    MAG_GET(tcnt, tiles + 1);
    k_cut_tiles<false><<<grid1(tiles + 1, 128), 128, 0, s>>>(tiles, ndof, tile_s, pn, pi, tcnt, nullptr, nullptr);
    MAG_CUB(cub::DeviceScan::ExclusiveSum(cub_p, cub_bytes, tcnt, tcnt, tiles + 1, s));
    int nb = 0;
    MAG_CUDA_TRY(cudaMemcpyAsync(&nb, tcnt + tiles, sizeof(int), cudaMemcpyDeviceToHost, s));
    MAG_CUDA_TRY(cudaStreamSynchronize(s));
    if (nb > kTileForms[k].most) {
        *form = k + 1;
        return MAG_OK;
    }
    MAG_GET(bstart, nb + 1);
    k_cut_tiles<true><<<grid1(tiles + 1, 128), 128, 0, s>>>(tiles, ndof, tile_s, pn, pi, nullptr, tcnt, bstart);
    // rows padded by 16 bytes, like the chunks: the kernels' L2 prefetches round to 16 bytes
    const size_t b_rows = (size_t)ndof * sizeof(uint2) + 16, b_blk = (size_t)nb * sizeof(TileBlock);
    if (cudaMalloc(&p->rows, b_rows) != cudaSuccess || cudaMalloc(&p->blocks, b_blk) != cudaSuccess) return MAG_E_NOMEM;
    const int eb = bits_of((uint64_t)ne), bb = bits_of((uint64_t)nb);
    uint64_t *keys = nullptr, *keys_s = nullptr;
    uint32_t *inc = nullptr, *inc_s = nullptr, *slotw = nullptr;
    int *rec = nullptr, *nch = nullptr, *ch0 = nullptr;
    MAG_GET(keys, ninc);
    MAG_GET(keys_s, ninc);
    MAG_GET(inc, ninc);
    MAG_GET(inc_s, ninc);
    MAG_GET(slotw, ninc);
    MAG_GET(rec, ninc);
    MAG_GET(nch, nb + 1);
    MAG_GET(ch0, nb + 1);
    MAG_CUDA_TRY(cudaMemsetAsync(nch + nb, 0, sizeof(int), s));
    k_block_rows<false><<<nb, kPB, 0, s>>>(in, order, bstart, pn, pi, eb, p->rows, keys, inc, slotw, nch, nullptr, nullptr,
                                           info);
    MAG_CUB(cub::DeviceScan::ExclusiveSum(cub_p, cub_bytes, nch, ch0, nb + 1, s));
    int *start = nullptr;
    if (ninc > 0) {
        MAG_CUB(cub::DeviceRadixSort::SortPairs(cub_p, cub_bytes, keys, keys_s, inc, inc_s, ninc, 0, eb + bb, s));
        k_record_heads<<<grid1(ninc), 256, 0, s>>>(keys_s, ninc, rec);
        MAG_CUB(cub::DeviceScan::InclusiveSum(cub_p, cub_bytes, rec, rec, ninc, s));
        start = reinterpret_cast<int *>(keys);  // the unsorted keys are used up; 2 ninc ints hold ninc + 1
        k_record_starts<<<grid1(ninc), 256, 0, s>>>(keys_s, ninc, rec, inc_s, in.inc_elem, start, info);
    }
    int nchunks = 0;
    MAG_CUDA_TRY(cudaMemcpyAsync(&nchunks, ch0 + nb, sizeof(int), cudaMemcpyDeviceToHost, s));
    MAG_TRY(read_info(info, &hi, s));
    if (hi.fail) return MAG_OK;
    const int64_t nrec = hi.nrec;
    const size_t b_ch = (size_t)std::max(nchunks, 1) * sizeof(uint2) + 16,
                 b_rec = (size_t)std::max<int64_t>(6 * nrec, 1) * sizeof(uint4);
    if (cudaMalloc(&p->chunks, b_ch) != cudaSuccess || cudaMalloc(&p->recs, b_rec) != cudaSuccess) return MAG_E_NOMEM;
    k_block_rows<true><<<nb, kPB, 0, s>>>(in, order, bstart, pn, pi, eb, nullptr, nullptr, nullptr, nullptr, nullptr, ch0,
                                          p->chunks, info);
    int *pos = reinterpret_cast<int *>(inc);  // the unsorted incidences are used up
    MAG_CUDA_TRY(cudaFuncSetAttribute(k_color_blocks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ColorSmem)));
    k_color_blocks<<<nb, kPB, sizeof(ColorSmem), s>>>(in, bstart, pn, pi, rec, start, inc_s, slotw, nch, ch0, p->blocks, pos,
                                                     info);
    MAG_TRY(read_info(info, &hi, s));
    if (hi.fail) return MAG_OK;
    if (small && hi.max_class > kTileSmallThreads && nb > kOneWave) {
        *form = k + 1;
        return MAG_OK;
    }
    if (nrec > 0)
        k_fill_records<<<grid1(nrec, 128), 128, 0, s>>>(in, nrec, start, keys_s, (uint64_t(1) << eb) - 1, inc_s, slotw, pos,
                                                       p->recs);
    MAG_CUDA_TRY(cudaGetLastError());
    MAG_CUDA_TRY(cudaStreamSynchronize(s));
    p->nblocks = nb;
    p->nrows = ndof;
    p->nchunks = nchunks;
    p->nrec = nrec;
    p->nnz = in.nnz;
    p->max_nnz = hi.max_nnz;
    p->max_inc = hi.max_inc;
    p->max_colors = hi.max_colors;
    p->max_rows = hi.max_rows;
    p->max_chunks = hi.max_chunks;
    p->small_tiles = small ? 1 : 0;
    p->small_blocks = small && hi.max_class <= kTileSmallThreads ? 1 : 0;
    p->evals_per_elem = (double)nrec / (double)ne;
    p->bytes = (int64_t)(b_blk + b_rows + b_ch + b_rec);
    p->ok = 1;
    return MAG_OK;
}

}  // namespace

void free_tile_plan(TilePlan *p) {
    void *q[] = {p->blocks, p->rows, p->chunks, p->recs};
    for (void *x : q)
        if (x) cudaFree(x);
    *p = TilePlan{};
}

int build_tile_plan(const TilePlanInput &in, void *work, size_t work_bytes, TilePlan *plan, cudaStream_t s, bool large) {
    *plan = TilePlan{};
    if (in.wide || in.ne <= 0 || in.ndof <= 0 || in.nn <= 0 || in.nnz >= (int64_t(1) << 32)) return MAG_OK;
    const auto t0 = std::chrono::steady_clock::now();
    TilePlan p;
    int rc = MAG_OK;
    for (int form = large ? kNumForms - 1 : 0; form < kNumForms && !p.ok;) {
        rc = build(in, work, work_bytes, &form, &p, s);
        if (rc != MAG_OK || !p.ok) free_tile_plan(&p);
        if (rc != MAG_OK) break;
    }
    if (rc != MAG_OK || !p.ok) {
        if (rc != MAG_E_NOMEM) return rc;
        cudaGetLastError();
        return MAG_OK;  // no room: the other schedules remain
    }
    p.build_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    *plan = p;
    return MAG_OK;
}

}  // namespace mag
