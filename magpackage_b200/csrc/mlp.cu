// Per-element reluctivity predictor: a 4 -> 64 -> 64 -> 64 -> 1 MLP with SiLU
// activations, BF16 tensor-core GEMMs (tcgen05, FP32 accumulators in TMEM) and
// FP32 master weights. Forward (inference and training) and backward kernels.
//
// Tile = 128 rows (elements). Forward: 128 threads a tile, thread t owns row t, and warp w reads
// TMEM lanes 32w..32w+31 (accumulator row m lives in lane m for M=128); inference runs two tiles
// in a CTA, which share the weights. Backward: 256 threads a tile, 32 columns a thread.
// Operands live in shared memory in the no-swizzle K-major "core matrix"
// layout: 8 rows x 16 bytes per core matrix, K-adjacent core matrices 128 B
// apart (leading byte offset), 8-row groups K*16 B apart (stride byte offset).
// One elected thread issues the MMAs (M=128, N=64, K=16 each) and commits them
// to an mbarrier; all threads wait with a bounded spin and read the
// accumulators with tcgen05.ld.
//
// Rounding points (mirrored by oracle/mlp_ref.py): layer inputs are rounded to
// BF16 before each MMA; accumulation, biases, activations, the last (64 -> 1)
// layer and all gradients are FP32: dX takes dZ rounded to BF16 as its MMA's input, dW all of dZ as
// three BF16 parts. Inference halves W1..W3 and b1..b3 (exact), so that its accumulators hold z/2
// and SiLU takes one FMA after the tanh.
#include <cuda_bf16.h>

#include <cstdint>

#include "mlp.cuh"

namespace mag {

namespace {

constexpr int kRows = 128;
constexpr int kH = 64;
constexpr long long kMbarSpin = 1LL << 24;

// ---- parameter layout (floats) -------------------------------------------------
// W1[64][4] b1[64] W2[64][64] b2[64] W3[64][64] b3[64] w4[64] b4
constexpr int oW1 = 0, ob1 = oW1 + kH * 4, oW2 = ob1 + kH, ob2 = oW2 + kH * kH, oW3 = ob2 + kH,
              ob3 = oW3 + kH * kH, ow4 = ob3 + kH, ob4 = ow4 + kH;
static_assert(ob4 + 1 == kMlpParams, "parameter layout");

// ---- bf16 operand images (core-matrix K-major), element offsets -----------------
// W1p[64 out][16 in], W2[64][64], W3[64][64], W2T[64 in][64 out], W3T[64][64]
constexpr int kW1pElems = kH * 16, kWElems = kH * kH;
constexpr int bW1p = 0, bW2 = bW1p + kW1pElems, bW3 = bW2 + kWElems, bW2T = bW3 + kWElems,
              bW3T = bW2T + kWElems;
static_assert(bW3T + kWElems == kMlpOperandElems, "operand layout");

__host__ __device__ constexpr int core_off(int r, int k, int K) {
    // element offset of (row r, column k) in a K-major core-matrix image of width K
    return (r >> 3) * (K * 8) + (k >> 3) * 64 + (r & 7) * 8 + (k & 7);
}

// sigmoid(z) = (1 + tanh(z/2)) / 2 with the hardware tanh approximation (one MUFU
// operation; relative error about 2^-11, below the BF16 rounding every layer input gets).
__device__ __forceinline__ float sigmoid_fast(float z) {
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * z));
    return 0.5f + 0.5f * t;
}
__device__ __forceinline__ float silu(float z) { return z * sigmoid_fast(z); }
__device__ __forceinline__ float dsilu(float z) {
    float s = sigmoid_fast(z);
    return s * (1.0f + z * (1.0f - s));
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ uint64_t smem_desc(const void *p, uint32_t lbo, uint32_t sbo) {
    uint64_t a = smem_u32(p);
    return ((a >> 4) & 0x3FFFull) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);  // version 1, no swizzle
}

// kind::f16 instruction descriptor: F32 accumulate, BF16 A and B, both K-major.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kH >> 3) << 17) |
                            ((uint32_t)(kRows >> 4) << 24);

__device__ __forceinline__ void mbar_init(uint64_t *bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Bounded wait on phase `parity`; returns false if it gave up. limit = 0: kMbarSpin
// polls of the potentially blocking try_wait; limit > 0: that many polls of the
// non-blocking test_wait (a caller-set limit, small in tests, that really runs out).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, long long limit = 0) {
    uint32_t done = 0;
    if (limit > 0) {
        for (long long i = 0; i < limit; i++) {
            asm volatile(
                "{\n\t.reg .pred P1;\n\t"
                "mbarrier.test_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
                "selp.b32 %0, 1, 0, P1;\n\t}"
                : "=r"(done)
                : "r"(smem_u32(bar)), "r"(parity)
                : "memory");
            if (done) return true;
        }
        return false;
    }
    for (long long i = 0; i < kMbarSpin; i++) {
        asm volatile(
            "{\n\t.reg .pred P1;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P1;\n\t}"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[128 x 64] (TMEM) = A[128 x K] * B[64 x K]^T, issued by one thread, completion on bar.
__device__ __forceinline__ void mma_issue(uint32_t tmem, const __nv_bfloat16 *A, const __nv_bfloat16 *B, int K,
                                          uint64_t *bar) {
    const uint32_t sbo = (uint32_t)K * 16;
    for (int kk = 0; kk < K / 16; kk++) {
        uint64_t ad = smem_desc(A + kk * 128, 128, sbo);  // 2 core matrices (256 B) per K=16 step
        uint64_t bd = smem_desc(B + kk * 128, 128, sbo);
        uint32_t acc = kk > 0 ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem), "l"(ad), "l"(bd), "r"(kIdesc), "r"(acc));
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// Columns c..c+15 of this thread's accumulator row from TMEM.
__device__ __forceinline__ void tmem_cols16(uint32_t tmem, int c, float out[16]) {
    const uint32_t lane_base = (uint32_t)(((threadIdx.x >> 5) & 3) * 32) << 16;
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(tmem + lane_base + (uint32_t)c));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) out[i] = __uint_as_float(r[i]);
}

// 16 pre-activations of one row: whole 32-byte sectors where the rows start on 16 bytes (vec).
__device__ __forceinline__ void store_z16(float *dst, const float z[16], bool vec) {
    if (vec) {
#pragma unroll
        for (int i = 0; i < 16; i += 4)
            *reinterpret_cast<float4 *>(dst + i) = make_float4(z[i], z[i + 1], z[i + 2], z[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; i++) dst[i] = z[i];
    }
}

// A hidden layer's epilogue, 16 columns at a time (few live registers): z = acc + b,
// h = SiLU(z) as BF16 into the next layer's input image; z kept for training.
__device__ __forceinline__ void hidden_epilogue(uint32_t tmem, const float *bias, __nv_bfloat16 *img, int row_t,
                                                float *z_row, bool vec) {
#pragma unroll
    for (int c = 0; c < kH; c += 16) {
        float z[16];
        tmem_cols16(tmem, c, z);
        __align__(16) __nv_bfloat162 hp[8];
#pragma unroll
        for (int i = 0; i < 16; i++) z[i] += bias[c + i];
#pragma unroll
        for (int i = 0; i < 8; i++) hp[i] = __floats2bfloat162_rn(silu(z[2 * i]), silu(z[2 * i + 1]));
        *reinterpret_cast<uint4 *>(img + core_off(row_t, c, kH)) = *reinterpret_cast<uint4 *>(hp);
        *reinterpret_cast<uint4 *>(img + core_off(row_t, c + 8, kH)) = *reinterpret_cast<uint4 *>(hp + 4);
        if (z_row) store_z16(z_row + c, z, vec);
    }
}

// ---- inference epilogue: packed FP32 pairs (f32x2) ---------------------------------

__device__ __forceinline__ uint64_t pk2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk2(uint64_t v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// SiLU of a hidden pair from its halved pre-activations h = z/2, packed as BF16 (z0's
// value in the low half). The inference kernel halves W1..W3 and b1..b3 (exact: a power of
// two), so the accumulators hold h, and z sigmoid(z) = h (1 + tanh h) = h + h tanh h: one
// single-precision tanh.approx per value and one packed FMA per pair.
// (A half-precision tanh of the pair, one MUFU operation for two values, was measured: 4 %
// faster at 8M rows, but its forward error, 6.7e-3 of max|y|, is above the 5.6e-3 bound.)
__device__ __forceinline__ uint32_t silu2h_bf16(uint64_t h) {
    float h0, h1, t0, t1;
    upk2(h, h0, h1);
    asm("tanh.approx.f32 %0, %1;" : "=f"(t0) : "f"(h0));
    asm("tanh.approx.f32 %0, %1;" : "=f"(t1) : "f"(h1));
    float p0, p1;
    upk2(fma2(h, pk2(t0, t1), h), p0, p1);
    uint32_t out;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out) : "f"(p1), "f"(p0));
    return out;
}

// Inference form of hidden_epilogue: the same image, packed arithmetic on the halved
// accumulators and biases (h = z/2).
__device__ __forceinline__ void hidden_epilogue_infer(uint32_t tmem, const float *bias, __nv_bfloat16 *img,
                                                      int row_t) {
#pragma unroll
    for (int c = 0; c < kH; c += 16) {
        float z[16];
        tmem_cols16(tmem, c, z);
        __align__(16) uint32_t hp[8];
#pragma unroll
        for (int i = 0; i < 8; i += 2) {  // one 16-byte shared load of biases per two pairs
            const float4 b = *reinterpret_cast<const float4 *>(bias + c + 2 * i);
            hp[i] = silu2h_bf16(add2(pk2(z[2 * i], z[2 * i + 1]), pk2(b.x, b.y)));
            hp[i + 1] = silu2h_bf16(add2(pk2(z[2 * i + 2], z[2 * i + 3]), pk2(b.z, b.w)));
        }
        *reinterpret_cast<uint4 *>(img + core_off(row_t, c, kH)) = *reinterpret_cast<uint4 *>(hp);
        *reinterpret_cast<uint4 *>(img + core_off(row_t, c + 8, kH)) = *reinterpret_cast<uint4 *>(hp + 4);
    }
}

// The backward kernel's images and barrier.
struct Smem {
    __nv_bfloat16 act[kRows * kH];  // dZ image of the running layer
    __nv_bfloat16 w[2 * kWElems];   // W2T | W3T
    uint64_t bar;
    uint32_t tmem;
    int fail;
};

__device__ __forceinline__ void load_ops(__nv_bfloat16 *w, const __nv_bfloat16 *ops, int first, int count) {
    const uint4 *src = reinterpret_cast<const uint4 *>(ops + first);
    uint4 *dst = reinterpret_cast<uint4 *>(w);
    for (int i = threadIdx.x; i < count / 8; i += blockDim.x) dst[i] = src[i];
}

// load_ops with every weight halved (a power-of-two scale: exact for every weight above
// 2^-125 in magnitude, where BF16 values are normal).
__device__ __forceinline__ void load_ops_halved(__nv_bfloat16 *w, const __nv_bfloat16 *ops, int first, int count) {
    const uint4 *src = reinterpret_cast<const uint4 *>(ops + first);
    uint4 *dst = reinterpret_cast<uint4 *>(w);
    const __nv_bfloat162 half2 = __floats2bfloat162_rn(0.5f, 0.5f);
    for (int i = threadIdx.x; i < count / 8; i += blockDim.x) {
        uint4 v = src[i];
        __nv_bfloat162 *p = reinterpret_cast<__nv_bfloat162 *>(&v);
#pragma unroll
        for (int j = 0; j < 4; j++) p[j] = __hmul2(p[j], half2);
        dst[i] = v;
    }
}

__device__ __forceinline__ void tmem_alloc(uint32_t *addr, uint32_t cols) {
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(addr)), "r"(cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        tc_fence_before();  // the allocated address is read by every thread after the next barrier
    }
}

__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols));
    }
}

// The forward kernel's shared memory: the weights, and per tile in flight an image and a
// completion barrier.
template <int TILES>
struct FwdSmem {
    __nv_bfloat16 act[TILES][kRows * kH];
    __nv_bfloat16 w[2 * kWElems + kW1pElems];
    float vec[4 * kH + 1];  // b1 | b2 | b3 | w4 | b4
    uint64_t bar[TILES];
    uint32_t tmem;
    int fail;
};

// OR over the kRows threads of named barrier ID.
template <int ID>
__device__ __forceinline__ bool named_barrier_or(bool v) {
    uint32_t any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %1, 0;\n\tbar.red.or.pred p, %2, %3, q;\n\tselp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(any)
        : "r"((uint32_t)v), "n"(ID), "n"(kRows)
        : "memory");
    return any != 0;
}

// The barrier of tile `id` (0 or 1) of the CTA; the branch is uniform over the tile's warps.
__device__ __forceinline__ bool tile_barrier_or(int id, bool v) {
    return id == 0 ? named_barrier_or<1>(v) : named_barrier_or<2>(v);
}

// One layer of one tile: one barrier of the tile's threads per layer. The barrier before the
// MMA issue also settles whether any thread's previous wait gave up (`ok` is this
// thread's outcome of its last wait): then every thread leaves the tile loop together.
// A wait that gives up drains first: the issued MMAs still read shared memory and write TMEM,
// so the kernel waits for their commit (default bound) before it leaves the tile loop.
__device__ __forceinline__ bool run_layer_fwd(int tile_id, uint32_t tmem, const __nv_bfloat16 *act, const __nv_bfloat16 *W,
                                              int K, uint64_t *bar, int *fail, uint32_t &phase, long long limit, bool &ok) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // smem writes -> tensor core
    tc_fence_before();
    const bool issuer = threadIdx.x % kRows == 0;
    if (tile_barrier_or(tile_id, !ok)) {
        if (issuer) *fail = 1;
        return false;
    }
    if (issuer) {
        tc_fence_after();
        mma_issue(tmem, act, W, K, bar);
    }
    ok = mbar_wait(bar, phase, limit);
    if (!ok) mbar_wait(bar, phase);
    phase ^= 1u;
    tc_fence_after();
    return true;
}

// ---- forward ---------------------------------------------------------------------

// INFER: no pre-activations kept (prediction); the epilogues use the packed forms above.
// TILES tiles run in a CTA, each with its kRows threads, image, TMEM columns and barriers; they
// share the weights, so that 32 warps fit an SM instead of 24: 14.8 to 12.8 us at 100,000 rows; at 8M
// rows 445 and 444 us: the transcendental unit is busy 81 % of the active cycles there, and the queue
// it shares with shared memory (MIO throttle) is the longest stall.
template <bool INFER, int TILES>
__global__ void __launch_bounds__(TILES * kRows, TILES == 2 ? 4 : 6) k_mlp_forward(MlpForwardArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    FwdSmem<TILES> &S = *reinterpret_cast<FwdSmem<TILES> *>(smem_raw);
    const int ct = threadIdx.x, t = ct % kRows, id = ct / kRows;
    if (t == 0) mbar_init(&S.bar[id]);
    if (ct == 0) S.fail = 0;
    // all weight images: W1p | W2 | W3 (contiguous in the operand buffer). Inference halves
    // W1..W3 and b1..b3 (exact), so that the accumulators hold z/2 (silu2h_bf16).
    const float hs = INFER ? 0.5f : 1.0f;
    if (INFER) load_ops_halved(S.w, a.ops, bW1p, kW1pElems + 2 * kWElems);
    else load_ops(S.w, a.ops, bW1p, kW1pElems + 2 * kWElems);
    for (int i = ct; i < kH; i += TILES * kRows) {
        S.vec[i] = hs * a.params[ob1 + i];
        S.vec[kH + i] = hs * a.params[ob2 + i];
        S.vec[2 * kH + i] = hs * a.params[ob3 + i];
        S.vec[3 * kH + i] = a.params[ow4 + i];
    }
    if (ct == 0) S.vec[4 * kH] = a.params[ob4];
    tmem_alloc(&S.tmem, TILES * kH);
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem + (uint32_t)(id * kH);  // this tile's accumulator columns
    __nv_bfloat16 *act = S.act[id];
    const int stride = (int)gridDim.x * TILES;
    const __nv_bfloat16 *W1 = S.w, *W2 = S.w + kW1pElems, *W3 = S.w + kW1pElems + kWElems;
    const float *sb1 = S.vec, *sb2 = S.vec + kH, *sb3 = S.vec + 2 * kH, *sw4 = S.vec + 3 * kH;
    const bool zvec = ((uintptr_t)a.z_out & 15) == 0;
    uint32_t phase = 0;
    bool ok = true;  // this thread's last tensor-core wait completed
    // The next tile's feature row (one 16-byte load: feature rows are 16 bytes, the buffer
    // 16-byte aligned) and output index are loaded one tile ahead, so their DRAM latency
    // overlaps the current tile's layers.
    const float4 *feats4 = reinterpret_cast<const float4 *>(a.feats);
    float4 f_next = make_float4(0.f, 0.f, 0.f, 0.f);
    int64_t dst_next = 0;
    {
        const int64_t r0 = ((int64_t)blockIdx.x * TILES + id) * kRows + t;
        if (r0 < a.n) {
            f_next = __ldg(feats4 + r0);
            dst_next = a.rows ? (int64_t)__ldg(a.rows + r0) : r0;
        }
    }
    for (int64_t tile = (int64_t)blockIdx.x * TILES + id; tile * kRows < a.n; tile += stride) {
        const int64_t row = tile * kRows + t;
        const bool valid = row < a.n;
        const float4 f = f_next;
        const int64_t dst = dst_next;
        {
            const int64_t rn = row + (int64_t)stride * kRows;
            if (rn < a.n) {
                f_next = __ldg(feats4 + rn);
                dst_next = a.rows ? (int64_t)__ldg(a.rows + rn) : rn;
            }
        }
        float x[4] = {0, 0, 0, 0};
        if (valid) {
            x[0] = f.x;
            x[1] = f.y;
            x[2] = f.z;
            x[3] = f.w;
        }
        {  // input image, K = 16 (features 4..15 are zero)
            __align__(16) __nv_bfloat16 v[16];
            for (int i = 0; i < 16; i++) v[i] = __float2bfloat16_rn(i < 4 ? x[i] : 0.0f);
            *reinterpret_cast<uint4 *>(act + core_off(t, 0, 16)) = *reinterpret_cast<uint4 *>(v);
            *reinterpret_cast<uint4 *>(act + core_off(t, 8, 16)) = *reinterpret_cast<uint4 *>(v + 8);
        }
        float *zr = (a.z_out && valid) ? a.z_out + row * 3 * kH : nullptr;
        // layer 1
        // (a completed MMA has read its input image; the next layer's issue barrier orders
        // every thread's TMEM reads and image writes before the next MMA, also across tiles:
        // the next tile's first MMA is issued after its own barrier)
        if (!run_layer_fwd(id, tmem, act, W1, 16, &S.bar[id], &S.fail, phase, a.spin_limit, ok)) break;
        if (INFER) hidden_epilogue_infer(tmem, sb1, act, t);
        else hidden_epilogue(tmem, sb1, act, t, zr, zvec);
        // layer 2
        if (!run_layer_fwd(id, tmem, act, W2, kH, &S.bar[id], &S.fail, phase, a.spin_limit, ok)) break;
        if (INFER) hidden_epilogue_infer(tmem, sb2, act, t);
        else hidden_epilogue(tmem, sb2, act, t, zr ? zr + kH : nullptr, zvec);
        // layer 3 and the 64 -> 1 output, 16 columns at a time
        if (!run_layer_fwd(id, tmem, act, W3, kH, &S.bar[id], &S.fail, phase, a.spin_limit, ok)) break;
        float y = 0.0f;
        if (INFER) {  // pairs of halved pre-activations: single-precision tanh (the output is not rounded to BF16)
            uint64_t yacc = pk2(0.0f, 0.0f);
#pragma unroll
            for (int c = 0; c < kH; c += 16) {
                float z[16];
                tmem_cols16(tmem, c, z);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    // biases and output weights by 16-byte shared loads, two pairs each
                    float4 b4, w4;
                    if ((i & 1) == 0) {
                        b4 = *reinterpret_cast<const float4 *>(sb3 + c + 2 * i);
                        w4 = *reinterpret_cast<const float4 *>(sw4 + c + 2 * i);
                    }
                    const float2 b = (i & 1) ? make_float2(b4.z, b4.w) : make_float2(b4.x, b4.y);
                    const float2 w = (i & 1) ? make_float2(w4.z, w4.w) : make_float2(w4.x, w4.y);
                    const uint64_t hh = add2(pk2(z[2 * i], z[2 * i + 1]), pk2(b.x, b.y));  // z/2
                    float h0, h1, t0, t1;
                    upk2(hh, h0, h1);
                    asm("tanh.approx.f32 %0, %1;" : "=f"(t0) : "f"(h0));
                    asm("tanh.approx.f32 %0, %1;" : "=f"(t1) : "f"(h1));
                    yacc = fma2(pk2(w.x, w.y), fma2(hh, pk2(t0, t1), hh), yacc);  // w4 silu(z)
                }
            }
            float y0, y1;
            upk2(yacc, y0, y1);
            y = y0 + y1;
        } else {
#pragma unroll
            for (int c = 0; c < kH; c += 16) {
                float z[16];
                tmem_cols16(tmem, c, z);
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    z[i] += sb3[c + i];
                    y += sw4[c + i] * silu(z[i]);
                }
                if (zr) store_z16(zr + 2 * kH + c, z, zvec);
            }
        }
        y += S.vec[4 * kH];
        if (valid && ok) {  // (after a wait that gave up, the kernel reports a timeout instead)
            if (a.y_out) a.y_out[row] = y;
            if (a.nu_out) {  // nu = exp(y * scale + shift), clamped to [nu_min, nu_max]
                double v = exp((double)y * a.y_scale + a.y_shift);
                v = v < a.nu_min ? a.nu_min : (v > a.nu_max ? a.nu_max : v);
                a.nu_out[dst] = v;
            }
        }
    }
    if (!ok) S.fail = 1;  // a wait of the last layer gave up
    tmem_free(S.tmem, TILES * kH);  // (its barrier makes S.fail visible to thread 0)
    if (ct == 0 && S.fail && a.err) atomicExch(a.err, 1);
}

// ---- backward --------------------------------------------------------------------
//
// 256 threads per 128-row tile: warp w serves rows 32 (w & 3) .. + 31 (the TMEM lanes it can
// read), columns 32 (w >> 2) .. + 31. The weight gradients dW = dZ^T H contract over the tile's
// rows: dZ is FP32 and H has BF16 values, so dZ is split into three BF16 parts that add up to it
// exactly (8 + 8 + 8 bits) and each part's products with H, which are exact, are summed by the
// tensor cores in FP32. They run beside the tcgen05 MMA that forms the next layer's dZ W; these
// operands lie row by row in shared memory, the transposed form mma.sync takes by ldmatrix
// (16 x 32 outputs a warp). Bias and output gradients are sums over rows by a shuffle tree.
// Measured at 32,768 rows: 130 us with one thread per row and 32 outputs a thread read from shared
// memory one by one; 43 us as FP32 outer products, 4 x 4 outputs a thread (bound by 8 words of
// shared memory per 16 products); 30 us so. The gradient then differs from the FP32 sums by 3e-7 in norm,
// and its error against 64 bits (7e-3, the BF16 layer inputs) is the same.
constexpr int kBwd = 256;
constexpr int kLd = kH + 8;  // row stride of the BF16 tiles: eight rows of an 8x8 matrix fall into different banks

struct BwdSmem {
    Smem s;
    alignas(16) __nv_bfloat16 dz[3][kRows * kLd];  // current layer's dZ: leading, middle, trailing part
    alignas(16) __nv_bfloat16 hin[kRows * kLd];    // current layer's input
    float sum[4][kH];                              // column sums of the four groups of 32 rows
    float dy[4];
};

// 32 consecutive pre-activations.
__device__ __forceinline__ void load_z32(const float *src, bool valid, bool vec, float z[32]) {
    if (valid && vec) {
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(src + i));
            z[i] = v.x;
            z[i + 1] = v.y;
            z[i + 2] = v.z;
            z[i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; i++) z[i] = valid ? __ldg(src + i) : 0.0f;
    }
}

// 32 columns c0.. of one row as BF16 into a K=64 core-matrix image.
__device__ __forceinline__ void put_bf16_32(__nv_bfloat16 *img, int row, int c0, const float v[32]) {
#pragma unroll
    for (int kb = 0; kb < 4; kb++) {
        __align__(16) __nv_bfloat162 t[4];
#pragma unroll
        for (int i = 0; i < 4; i++) t[i] = __floats2bfloat162_rn(v[kb * 8 + 2 * i], v[kb * 8 + 2 * i + 1]);
        *reinterpret_cast<uint4 *>(img + core_off(row, c0 + kb * 8, kH)) = *reinterpret_cast<uint4 *>(t);
    }
}

// 32 BF16 values (bits) to a tile row.
__device__ __forceinline__ void put_bits32(__nv_bfloat16 *dst, const uint32_t v[16]) {
#pragma unroll
    for (int i = 0; i < 16; i += 4) *reinterpret_cast<uint4 *>(dst + 2 * i) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
}

// The three parts of 32 FP32 values: each the leading 8 bits of what the parts before leave, so
// that they add up exactly (but for bits below 2^-133, the last of a BF16). Infinities and NaN stay
// in the leading part. An input that rounds to an infinity meets a dZ that is NaN in its whole row
// (dsilu of the next layer's infinite or NaN pre-activations), so 0 x infinity of a zero part adds
// no NaN that FP32 products would not have.
__device__ __forceinline__ void put_split32(BwdSmem &B, int row, int c0, const float v[32]) {
    float x[32];
#pragma unroll
    for (int i = 0; i < 32; i++) x[i] = v[i];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const uint32_t a = __float_as_uint(x[2 * i]) & 0xFFFF0000u, b = __float_as_uint(x[2 * i + 1]) & 0xFFFF0000u;
            w[i] = (a >> 16) | b;
            x[2 * i] = (a & 0x7F800000u) == 0x7F800000u ? 0.0f : x[2 * i] - __uint_as_float(a);
            x[2 * i + 1] = (b & 0x7F800000u) == 0x7F800000u ? 0.0f : x[2 * i + 1] - __uint_as_float(b);
        }
        put_bits32(B.dz[k] + row * kLd + c0, w);
    }
}

// BF16 of 32 values to a tile row.
__device__ __forceinline__ void put_input32(BwdSmem &B, int row, int c0, const float v[32]) {
    uint32_t w[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const __nv_bfloat162 t = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t *>(&t);
    }
    put_bits32(B.hin + row * kLd + c0, w);
}

// Sums over a warp's 32 rows (lanes) of 32 columns: lane c gets column c's.
__device__ __forceinline__ float warp_columns(const float v[32]) {
    float x[16];
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const float keep = lane & 16 ? v[i + 16] : v[i], send = lane & 16 ? v[i] : v[i + 16];
        x[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; i++) {
            const float keep = lane & o ? x[i + o] : x[i], send = lane & o ? x[i] : x[i + o];
            x[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    return x[0];
}

__device__ __forceinline__ void ldm_x4_trans(uint32_t r[4], const __nv_bfloat16 *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_u32(p))
                 : "memory");
}

__device__ __forceinline__ void mma_16816(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void add_to(float *g, float v, bool first) { *g = first ? v : *g + v; }

// gW[o][i] += sum_r dz[r][o] hin[r][i] (64 x 64): warp w the outputs o in 16 (w & 3) .. + 15,
// i in 32 (w >> 2) .. + 31; the smaller parts first.
__device__ __forceinline__ void weight_grads(const BwdSmem &B, float *gW, bool first) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, m0 = (w & 3) * 16, n0 = (w >> 2) * 32;
    const int ar = (lane & 7) + (lane >> 4) * 8, ac = m0 + ((lane >> 3) & 1) * 8;
    const int br = (lane & 7) + ((lane >> 3) & 1) * 8, bc = n0 + (lane >> 4) * 8;
    float acc[4][4];
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[n][j] = 0.0f;
#pragma unroll 2
    for (int k0 = 0; k0 < kRows; k0 += 16) {
        uint32_t b[2][4];
        ldm_x4_trans(b[0], B.hin + (k0 + br) * kLd + bc);
        ldm_x4_trans(b[1], B.hin + (k0 + br) * kLd + bc + 16);
#pragma unroll
        for (int p = 2; p >= 0; p--) {
            uint32_t a[4];
            ldm_x4_trans(a, B.dz[p] + (k0 + ar) * kLd + ac);
#pragma unroll
            for (int n = 0; n < 4; n++) mma_16816(acc[n], a, b[n >> 1][2 * (n & 1)], b[n >> 1][2 * (n & 1) + 1]);
        }
    }
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float2 *dst = reinterpret_cast<float2 *>(gW + (m0 + (lane >> 2) + 8 * h) * kH + n0 + 8 * n + 2 * (lane & 3));
            float2 v = make_float2(acc[n][2 * h], acc[n][2 * h + 1]);
            if (!first) {
                const float2 p = *dst;
                v = make_float2(p.x + v.x, p.y + v.y);
            }
            *dst = v;
        }
}

// The same for the first layer: four inputs, in the first eight columns of the input tile.
__device__ __forceinline__ void weight_grads4(const BwdSmem &B, float *gW, bool first) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, m0 = (w & 3) * 16;
    if (w >= 4) return;
    const int ar = (lane & 7) + (lane >> 4) * 8, ac = m0 + ((lane >> 3) & 1) * 8;
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int k0 = 0; k0 < kRows; k0 += 32) {
        uint32_t b[4];  // rows k0 .. k0 + 31 of the eight columns
        ldm_x4_trans(b, B.hin + (k0 + lane) * kLd);
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int p = 2; p >= 0; p--) {
                uint32_t a[4];
                ldm_x4_trans(a, B.dz[p] + (k0 + 16 * h + ar) * kLd + ac);
                mma_16816(acc, a, b[2 * h], b[2 * h + 1]);
            }
    }
    if ((lane & 3) < 2)
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int j = 0; j < 2; j++)
                add_to(gW + (m0 + (lane >> 2) + 8 * h) * 4 + 2 * (lane & 3) + j, acc[2 * h + j], first);
}

// Column sums over the tile from the warps' (after a barrier), by 64 threads.
__device__ __forceinline__ void tile_columns(const BwdSmem &B, float *g, bool first) {
    if (threadIdx.x < kH) {
        const int o = threadIdx.x;
        add_to(g + o, (B.sum[0][o] + B.sum[1][o]) + (B.sum[2][o] + B.sum[3][o]), first);
    }
}

// The two halves of a layer: the MMA on the image every thread has written, and the wait for
// it; work that touches neither the image nor TMEM goes between. finish() is block-uniform.
__device__ __forceinline__ void layer_issue(Smem &S, const __nv_bfloat16 *W) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // smem writes -> tensor core
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) {
        tc_fence_after();
        mma_issue(S.tmem, S.act, W, kH, &S.bar);
    }
}

__device__ __forceinline__ bool layer_finish(Smem &S, uint32_t &phase, long long limit) {
    bool ok = mbar_wait(&S.bar, phase, limit);
    if (!ok) mbar_wait(&S.bar, phase);  // the issued MMAs still read shared memory: drain
    phase ^= 1u;
    tc_fence_after();
    const bool any_fail = __syncthreads_or(ok ? 0 : 1) != 0;
    if (any_fail && threadIdx.x == 0) S.fail = 1;
    return !any_fail;
}

// Columns c0 .. c0 + 31 of this thread's accumulator row.
__device__ __forceinline__ void tmem_cols32(uint32_t tmem, int c0, float out[32]) {
    const uint32_t base = tmem + ((uint32_t)(((threadIdx.x >> 5) & 3) * 32) << 16) + (uint32_t)c0;
    uint32_t r[32];
#pragma unroll
    for (int c = 0; c < 32; c += 16)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[c + 0]), "=r"(r[c + 1]), "=r"(r[c + 2]), "=r"(r[c + 3]), "=r"(r[c + 4]), "=r"(r[c + 5]),
              "=r"(r[c + 6]), "=r"(r[c + 7]), "=r"(r[c + 8]), "=r"(r[c + 9]), "=r"(r[c + 10]), "=r"(r[c + 11]),
              "=r"(r[c + 12]), "=r"(r[c + 13]), "=r"(r[c + 14]), "=r"(r[c + 15])
            : "r"(base + (uint32_t)c));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) out[i] = __uint_as_float(r[i]);
    tc_fence_before();  // ordered before the next MMA by the barrier that precedes its issue
}

__global__ void __launch_bounds__(kBwd, 2) k_mlp_backward(MlpBackwardArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    BwdSmem &B = *reinterpret_cast<BwdSmem *>(smem_raw);
    Smem &S = B.s;
    const int t = threadIdx.x;
    const int lr = ((t >> 5) & 3) * 32 + (t & 31), c0 = (t >> 7) * 32;  // row in the tile, first column
    if (t == 0) {
        mbar_init(&S.bar);
        S.fail = 0;
    }
    load_ops(S.w, a.ops, bW2T, 2 * kWElems);  // W2T | W3T
    tmem_alloc(&S.tmem, kH);
    __syncthreads();
    tc_fence_after();
    const __nv_bfloat16 *W2T = S.w, *W3T = S.w + kWElems;
    float *G = a.grad_partial + (size_t)blockIdx.x * kMlpPartial;  // this CTA's partial gradient
    const bool zvec = ((uintptr_t)a.z & 15) == 0;
    float *my_sum = B.sum[(t >> 5) & 3] + c0 + (t & 31);  // where this lane's column sum goes
    uint32_t phase = 0;
    bool first = true;
    for (int tile = blockIdx.x; tile * kRows < a.n; tile += gridDim.x, first = false) {
        const int64_t row = (int64_t)tile * kRows + lr;
        const bool valid = row < a.n;
        const float *zr = a.z + (valid ? row : 0) * 3 * kH + c0;
        float z[32], v[32], dz[32];
        load_z32(zr + 2 * kH, valid, zvec, z);
        const float dy = valid ? (a.y[row] - a.target[row]) * a.loss_scale : 0.0f;
        // last layer: dz3, and the sums of dy h3 (dw4) and dy (db4)
#pragma unroll
        for (int o = 0; o < 32; o++) {
            dz[o] = dy * __ldg(a.params + ow4 + c0 + o) * dsilu(z[o]);
            v[o] = dy * silu(z[o]);
        }
        load_z32(zr + kH, valid, zvec, z);
        put_bf16_32(S.act, lr, c0, dz);
        *my_sum = warp_columns(v);
        if (c0 == 0) {
            float d = dy;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
            if ((t & 31) == 0) B.dy[t >> 5] = d;
        }
        layer_issue(S, W3T);  // dh2 = dz3 W3
        tile_columns(B, G + ow4, first);
        if (t == 0) add_to(G + ob4, (B.dy[0] + B.dy[1]) + (B.dy[2] + B.dy[3]), first);
        put_split32(B, lr, c0, dz);
#pragma unroll
        for (int o = 0; o < 32; o++) v[o] = silu(z[o]);
        put_input32(B, lr, c0, v);
        const float sum3 = warp_columns(dz);
        __syncthreads();
        *my_sum = sum3;
        // layer 3: dW3 += dz3^T h2
        weight_grads(B, G + oW3, first);
        if (!layer_finish(S, phase, a.spin_limit)) break;
        tile_columns(B, G + ob3, first);
        tmem_cols32(S.tmem, c0, v);
#pragma unroll
        for (int o = 0; o < 32; o++) dz[o] = v[o] * dsilu(z[o]);
        // layer 2: dW2 += dz2^T h1, dh1 = dz2 W2
        load_z32(zr, valid, zvec, z);
        put_bf16_32(S.act, lr, c0, dz);
        put_split32(B, lr, c0, dz);
        const float sum2 = warp_columns(dz);
#pragma unroll
        for (int o = 0; o < 32; o++) v[o] = silu(z[o]);
        put_input32(B, lr, c0, v);
        layer_issue(S, W2T);
        *my_sum = sum2;
        weight_grads(B, G + oW2, first);
        if (!layer_finish(S, phase, a.spin_limit)) break;
        tile_columns(B, G + ob2, first);
        tmem_cols32(S.tmem, c0, v);
#pragma unroll
        for (int o = 0; o < 32; o++) dz[o] = v[o] * dsilu(z[o]);
        // layer 1: dW1 += dz1^T x
        put_split32(B, lr, c0, dz);
        const float sum1 = warp_columns(dz);
        if (c0 == 0) {
            uint32_t w[4] = {0, 0, 0, 0};
            if (valid) {
                const float *f = a.feats + row * 4;
                const __nv_bfloat162 f01 = __floats2bfloat162_rn(f[0], f[1]), f23 = __floats2bfloat162_rn(f[2], f[3]);
                w[0] = *reinterpret_cast<const uint32_t *>(&f01);
                w[1] = *reinterpret_cast<const uint32_t *>(&f23);
            }
            *reinterpret_cast<uint4 *>(B.hin + lr * kLd) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        __syncthreads();
        *my_sum = sum1;
        weight_grads4(B, G + oW1, first);
        __syncthreads();
        tile_columns(B, G + ob1, first);
        __syncthreads();
    }
    if (t == 0 && S.fail && a.err) atomicExch(a.err, 1);
    tmem_free(S.tmem, kH);
}

// grad[p] = sum over CTAs (fixed order) of the partials. A CTA of eight warps takes 32
// parameters: the warps load kRedChunk partials side by side into shared memory, the first one
// adds them in order. (One thread per parameter loading as it adds: 13 us at 256 partials, a
// chain of loads; 6.8 us so.)
constexpr int kRedChunk = 256;
__global__ void __launch_bounds__(256) k_mlp_reduce(const float *__restrict__ partial, int nparts, float *__restrict__ grad) {
    __shared__ float sh[kRedChunk][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, p = blockIdx.x * 32 + lane;
    float s = 0.0f;
    for (int c0 = 0; c0 < nparts; c0 += kRedChunk) {
        const int m = nparts - c0 < kRedChunk ? nparts - c0 : kRedChunk;
        float v[kRedChunk / 8];
#pragma unroll
        for (int j = 0; j < kRedChunk / 8; j++)
            v[j] = w + 8 * j < m && p < kMlpParams ? __ldg(partial + (size_t)(c0 + w + 8 * j) * kMlpPartial + p) : 0.0f;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kRedChunk / 8; j++) sh[w + 8 * j][lane] = v[j];
        __syncthreads();
        if (w == 0) {
#pragma unroll 16
            for (int c = 0; c < m; c++) s += sh[c][lane];
        }
    }
    if (w == 0 && p < kMlpParams) grad[p] = s;
}

// Adam step on the FP32 master weights.
__global__ void k_mlp_adam(float *__restrict__ params, const float *__restrict__ grad, float *__restrict__ m,
                           float *__restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kMlpParams) return;
    float g = grad[p];
    float mm = b1 * m[p] + (1.0f - b1) * g;
    float vv = b2 * v[p] + (1.0f - b2) * g * g;
    m[p] = mm;
    v[p] = vv;
    params[p] -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
}

// BF16 operand images from the FP32 master weights.
__global__ void k_mlp_pack(const float *__restrict__ P, __nv_bfloat16 *__restrict__ ops) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < kH * 16) {  // W1p [64 out][16 in], inputs 4..15 zero
        int o = idx / 16, i = idx % 16;
        ops[bW1p + core_off(o, i, 16)] = __float2bfloat16_rn(i < 4 ? P[oW1 + o * 4 + i] : 0.0f);
    }
    if (idx < kH * kH) {
        int o = idx / kH, i = idx % kH;
        ops[bW2 + core_off(o, i, kH)] = __float2bfloat16_rn(P[oW2 + o * kH + i]);
        ops[bW3 + core_off(o, i, kH)] = __float2bfloat16_rn(P[oW3 + o * kH + i]);
        // transposed images: row = input feature i, column = output feature o
        ops[bW2T + core_off(i, o, kH)] = __float2bfloat16_rn(P[oW2 + o * kH + i]);
        ops[bW3T + core_off(i, o, kH)] = __float2bfloat16_rn(P[oW3 + o * kH + i]);
    }
}

__global__ void k_mlp_gather(const float4 *__restrict__ feats, const float *__restrict__ target,
                             const int64_t *__restrict__ perm, int64_t off, int64_t b, float4 *__restrict__ xb,
                             float *__restrict__ tb) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= b) return;
    const int64_t r = perm[off + i];
    xb[i] = feats[r];
    tb[i] = target[r];
}

// One CTA of 1024 threads: strided partial sums, then a fixed tree over the shared array.
__global__ void __launch_bounds__(1024) k_mlp_sqerr(const float *__restrict__ y, const float *__restrict__ t,
                                                    int64_t b, float *__restrict__ acc) {
    __shared__ float part[1024];
    float v = 0.0f;
    for (int64_t i = threadIdx.x; i < b; i += 1024) {
        const float d = y[i] - t[i];
        v += d * d;
    }
    part[threadIdx.x] = v;
    __syncthreads();
    for (int w = 512; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) part[threadIdx.x] += part[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *acc += part[0];
}

}  // namespace

int mlp_gather(const float *feats, const float *target, const int64_t *perm, int64_t off, int64_t b, float *xb,
               float *tb, cudaStream_t s) {
    k_mlp_gather<<<(unsigned)((b + 255) / 256), 256, 0, s>>>(reinterpret_cast<const float4 *>(feats), target, perm,
                                                            off, b, reinterpret_cast<float4 *>(xb), tb);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}

int mlp_sqerr(const float *y, const float *t, int64_t b, float *acc, cudaStream_t s) {
    k_mlp_sqerr<<<1, 1024, 0, s>>>(y, t, b, acc);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}


int mlp_pack(const float *params, __nv_bfloat16 *ops, cudaStream_t s) {
    k_mlp_pack<<<(kH * kH + 255) / 256, 256, 0, s>>>(params, ops);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}

namespace {

template <bool INFER, int TILES>
int launch_forward(const MlpForwardArgs &a, int tiles, cudaStream_t s) {
    constexpr size_t sm = sizeof(FwdSmem<TILES>);
    auto kern = k_mlp_forward<INFER, TILES>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    // The CTAs loop over tiles; launching several waves of them (about 9 tiles each at 8M rows)
    // lets SMs that finish early take more CTAs, which evens out the tail (measured at 7.99M rows
    // with one tile per CTA at a time: 8 CTAs per SM 0.514 ms, 24 0.474, 48 0.467, 96 0.470, one
    // tile per CTA 0.654: the per-CTA weight load and TMEM allocation then dominate).
#ifndef MAG_MLP_TILES_PER_SM
#define MAG_MLP_TILES_PER_SM 48
#endif
    int grid = (tiles + TILES - 1) / TILES, dev = 0, nsm = 0;
    constexpr int most = MAG_MLP_TILES_PER_SM / TILES;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
        nsm > 0 && grid > most * nsm)
        grid = most * nsm;
    kern<<<grid, TILES * kRows, sm, s>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}

}  // namespace

int mlp_forward(const MlpForwardArgs &a, int tiles, cudaStream_t s) {
    return a.z_out ? launch_forward<false, 1>(a, tiles, s) : launch_forward<true, 2>(a, tiles, s);
}

int mlp_backward(const MlpBackwardArgs &a, int grid, cudaStream_t s) {
    size_t sm = sizeof(BwdSmem);
    cudaFuncSetAttribute(k_mlp_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_mlp_backward<<<grid, kBwd, sm, s>>>(a);
    if (cudaPeekAtLastError() != cudaSuccess) return MAG_E_CUDA;
    k_mlp_reduce<<<(kMlpParams + 31) / 32, 256, 0, s>>>(a.grad_partial, grid, a.grad);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}

int mlp_adam(float *params, const float *grad, float *m, float *v, float lr, float b1, float b2, float eps,
             int step, cudaStream_t s) {
    float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
    k_mlp_adam<<<(kMlpParams + 255) / 256, 256, 0, s>>>(params, grad, m, v, lr, b1, b2, eps, c1, c2);
    return cudaPeekAtLastError() == cudaSuccess ? MAG_OK : MAG_E_CUDA;
}

}  // namespace mag
