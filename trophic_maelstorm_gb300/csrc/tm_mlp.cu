// tm_mlp.cu -- the sweep surrogate: a 3-128-128-128-2 GELU network with BF16
// weights, trained and evaluated on the 5th-generation tensor cores.
//
// The reference has no learned part; the network, its rounding points and its
// optimiser are specified in include/tm.h (tm_mlp_*).  One CTA owns a tile of
// 128 samples (sample t = TMEM lane t) and runs the whole forward and backward
// pass of that tile with 32 warps: warp w reads TMEM lane quarter w % 4 (the
// quarter a warp may access) and handles column slice w / 4, so a thread does
// 16 of the 128 columns of its sample; sums over 128 columns or samples are formed
// from four parts of 32 terms:
//   * the two 128x128 layers and the four GEMMs of their backward pass are
//     tcgen05.mma (kind::f16, BF16 x BF16 -> FP32, M = N = K = 128), issued by
//     one thread, with both operands in shared memory in the K-major
//     no-swizzle core-matrix layout and the accumulators in TMEM;
//   * the 3-wide input layer, the 2-wide output layer, GELU and its derivative
//     run on the CUDA cores between the MMAs, reading accumulators back with
//     tcgen05.ld;
//   * each CTA writes its partial gradient; a second kernel sums the partials
//     in tile order (no atomics: the result does not depend on scheduling) and
//     applies Adam to the FP32 master weights, refreshing their BF16 copies.
// Bound by one tile's serial chain (phases of a few thousand cycles between barriers), not
// by arithmetic: 12,000 samples are 94 tiles on 152 SMs.  Measured per training step:
// 53.3 us with everything unrolled (waiting for instructions), tanh evaluated twice and
// 2-byte transposed stores; 36.4 us with loops, gelu' kept in TMEM, matrix-load
// transposes, 16-byte constant loads, one polling warp, and both kernels' prologues overlapping
// their predecessors' ends (programmatic dependent launch: 43 -> 36).  512 or 1024 threads made
// no difference before the shared-memory work went down.
// Every wait on an MMA completion is bounded: on timeout the CTA records an
// error, waits once more (again bounded) for the MMAs it issued, frees its
// TMEM and returns; the update kernel then leaves the parameters unchanged.
#include "tm_kernels.cuh"
#include "../../include/tm.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <new>

namespace {

constexpr int TS = 128;              // samples per tile = TMEM lanes
constexpr int NT = 1024;             // threads per CTA: 8 column slices x 128 samples
constexpr int CW = 128 / (NT / TS);  // columns of a thread's slice
constexpr int NS = 4;                // parts of 32 terms that each sum over 128 is formed from
constexpr int OFF_W1 = 0, OFF_B1 = 384, OFF_W2 = 512, OFF_B2 = 16896, OFF_W3 = 17024, OFF_B3 = 33408,
              OFF_W4 = 33536, OFF_B4 = 33792, NP = 33794;
static_assert(NP == TM_MLP_NPARAMS, "parameter layout");
constexpr int PS = 33808;            // per-tile stride of the partial gradients (rows stay 32-byte aligned)
static_assert(PS % 8 == 0 && OFF_W2 % 8 == 0 && OFF_W3 % 8 == 0, "32-byte aligned gradient rows");

// shared memory map
constexpr int BUF = 32768;           // one 128 x 128 BF16 operand tile
constexpr int SM_W1 = 6 * BUF;
constexpr int SM_B = SM_W1 + 1536;   // b1 | b2 | b3
constexpr int SM_W4 = SM_B + 1536;
constexpr int SM_B4 = SM_W4 + 1024;
constexpr int SM_X = SM_B4 + 16;
constexpr int SM_DY = SM_X + 1536;
constexpr int SM_LOSS = SM_DY + 1024;
constexpr int SM_RED = SM_LOSS + 512;       // [NS][128][3] FP32 partial sums
constexpr int SM_BAR = SM_RED + NS * TS * 3 * 4;
constexpr int SM_TMEM = SM_BAR + 8;
constexpr int SM_TOTAL = SM_TMEM + 8;
constexpr int FPAD = 129;            // row stride (floats) of the FP32 column-sum scratch over buffers 0-2
static_assert(TS * FPAD * 4 <= 3 * BUF, "scratch fits buffers 0-2");
static_assert(SM_BAR % 8 == 0, "mbarrier alignment");

constexpr int kWaitLimit = 1 << 22;  // polls of an MMA completion before the CTA gives up (~0.3 s)
constexpr int kProbeWaitLimit = 1 << 16;  // the same under TM_PROBE_MLP_WAIT (nothing in flight)

// byte offset of element (row r, k) of a 128-row operand in the K-major,
// no-swizzle canonical layout: 8 x 16-byte core matrices, 128 B apart along K
// (leading byte offset) and 2048 B apart along the rows (stride byte offset)
__device__ __forceinline__ uint32_t cm(int r, int k)
{
    return (uint32_t)((r >> 3) * 2048 + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: start >> 4, LBO = 128 B, SBO = 2048 B,
// fixed 0b001 at bits 46-48, no swizzle
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t a)
{
    return (uint64_t)((a & 0x3FFFFu) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(2048 >> 4) << 32) |
           (1ull << 46);
}

// instruction descriptor, kind::f16: D FP32 (bits 4-5 = 1), A and B BF16 (bits 7-9, 10-12 = 1),
// both K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 3) << 17) |
                            ((uint32_t)(128 >> 4) << 24);

// D[128 x 128] (TMEM columns d..d+127) = A[128 x 128] * B[128 x 128]^T, both K-major in shared memory
__device__ __forceinline__ void mma_128(uint32_t d, uint32_t a, uint32_t b)
{
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
        const uint64_t da = desc_kmajor(a + kk * 256), db = desc_kmajor(b + kk * 256);
        const uint32_t acc = kk > 0 ? 1u : 0u;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                     :: "r"(d), "l"(da), "l"(db), "r"(kIdesc), "r"(acc));
    }
}

__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, int limit)
{
    for (int i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if (i > 32) __nanosleep(64);
    }
    return false;
}

// 8 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v)
{
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float* v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 :: "r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
                    "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
                    "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7]))
                 : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

constexpr float kGeluC = 0.7978845608028654f;   // sqrt(2/pi)
constexpr float kGeluK = 0.044715f;

__device__ __forceinline__ float gelu(float a)
{
    const float th = tanhf(kGeluC * (a + kGeluK * (a * a * a)));
    return 0.5f * a * (1.0f + th);
}

__device__ __forceinline__ float gelu_grad(float a)
{
    const float th = tanhf(kGeluC * (a + kGeluK * (a * a * a)));
    return 0.5f * (1.0f + th) + 0.5f * a * (1.0f - th * th) * kGeluC * (1.0f + 3.0f * kGeluK * (a * a));
}

// both from one tanh
__device__ __forceinline__ float gelu_and_grad(float a, float& grad)
{
    const float th = tanhf(kGeluC * (a + kGeluK * (a * a * a)));
    grad = 0.5f * (1.0f + th) + 0.5f * a * (1.0f - th * th) * kGeluC * (1.0f + 3.0f * kGeluK * (a * a));
    return 0.5f * a * (1.0f + th);
}

// 128 x 128 BF16 row-major matrix (global) -> K-major core-matrix tile (shared)
__device__ __forceinline__ void load_tile(unsigned char* dst, const __nv_bfloat16* src)
{
    const uint4* s = reinterpret_cast<const uint4*>(src);
    for (int c = threadIdx.x; c < 2048; c += NT) *reinterpret_cast<uint4*>(dst + cm(c >> 4, (c & 15) * 8)) = s[c];
}

// sum over k in [32 p, 32 p + 32) of row r of a K-major BF16 tile, k ascending
__device__ __forceinline__ float row_sum_part(const unsigned char* buf, int r, int p)
{
    float s = 0.0f;
    for (int g = 4 * p; g < 4 * p + 4; ++g) {
        const uint4 q = *reinterpret_cast<const uint4*>(buf + cm(r, g * 8));
        const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&q);
#pragma unroll
        for (int i = 0; i < 8; ++i) s = s + __bfloat162float(h[i]);
    }
    return s;
}

__device__ __forceinline__ void store8(unsigned char* buf, int r, int k0, const __nv_bfloat16* h)
{
    *reinterpret_cast<uint4*>(buf + cm(r, k0)) = *reinterpret_cast<const uint4*>(h);
}

// The transpose of a warp's 32 rows x CW columns (rows r0.., columns k0.. of `from`, just
// stored by this warp) into rows k0.., columns r0.. of `to`: an 8 x 8 block is 128
// contiguous bytes in either tile, so four blocks go by one transposing matrix load and
// one matrix store (2-byte stores took 4 bank cycles each, 16 of them a thread).
__device__ __forceinline__ void transpose_warp(const unsigned char* from, unsigned char* to, int r0, int k0)
{
    const int lane = threadIdx.x & 31, blk = lane >> 3, i = lane & 7;
    __syncwarp();
#pragma unroll
    for (int c = 0; c < CW; c += 8) {
        uint32_t m0, m1, m2, m3;
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(m0), "=r"(m1), "=r"(m2), "=r"(m3) : "r"(saddr(from + cm(r0 + blk * 8 + i, k0 + c))) : "memory");
        asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};"
                     :: "r"(saddr(to + cm(k0 + c + i, r0 + blk * 8))), "r"(m0), "r"(m1), "r"(m2), "r"(m3) : "memory");
    }
}

// 8 consecutive floats of shared memory (16-byte aligned)
__device__ __forceinline__ void lds8(const float* p, float* v)
{
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// 8 floats to a 32-byte aligned global address in one instruction
__device__ __forceinline__ void stg8(float* p, const float* v)
{
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 :: "l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}

// z1 = W1 x + b1 of columns j .. j + 7 (j a multiple of 8)
__device__ __forceinline__ void layer1(const float* W1s, const float* bs, int j, float x0, float x1, float x2, float* z)
{
    float w[24], b[8];
    lds8(W1s + 3 * j, w);
    lds8(W1s + 3 * j + 8, w + 8);
    lds8(W1s + 3 * j + 16, w + 16);
    lds8(bs + j, b);
#pragma unroll
    for (int i = 0; i < 8; ++i) z[i] = ((w[3 * i] * x0 + w[3 * i + 1] * x1) + w[3 * i + 2] * x2) + b[i];
}

struct MlpArgs {
    const float* x;                  // n x 3 features
    const float* y;                  // n x 2 targets (training)
    const float* w;                  // n x 2 loss weights (training)
    int n;
    float inv_norm;
    const float* p;                  // FP32 master parameters
    const __nv_bfloat16 *W2, *W2T, *W3, *W3T;   // BF16 copies, [out][in] and transposed
    float* grad_part;                // [tiles][PS] partial gradients (training)
    float* loss_part;                // [tiles] partial losses (training)
    float* y_out;                    // n x 2 outputs (inference)
    int* err;                        // set to 1 when an MMA wait ran out
    int wait_limit;                  // polls of one MMA completion
    int probe_no_mma;                // TM_PROBE_MLP_WAIT: the first GEMM is not issued, so its wait runs out
};

template <bool TRAIN>
__global__ void __launch_bounds__(NT, 1) mlp_tile_kernel(MlpArgs a)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    unsigned char* B0 = sm;
    unsigned char* B1 = sm + BUF;
    unsigned char* B2 = sm + 2 * BUF;
    unsigned char* B3 = sm + 3 * BUF;
    unsigned char* B4 = sm + 4 * BUF;
    unsigned char* B5 = sm + 5 * BUF;
    float* F = reinterpret_cast<float*>(sm);           // FP32 scratch [128][FPAD] over B0..B2
    float* W1s = reinterpret_cast<float*>(sm + SM_W1);
    float* bs = reinterpret_cast<float*>(sm + SM_B);
    float* W4s = reinterpret_cast<float*>(sm + SM_W4);
    float* b4s = reinterpret_cast<float*>(sm + SM_B4);
    float* xs = reinterpret_cast<float*>(sm + SM_X);
    float* dys = reinterpret_cast<float*>(sm + SM_DY);
    float* ls = reinterpret_cast<float*>(sm + SM_LOSS);
    float* red = reinterpret_cast<float*>(sm + SM_RED);    // [NS][TS][3]
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + SM_BAR);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + SM_TMEM);

    const int tid = threadIdx.x, warp = tid >> 5;
    const int q = warp & 3, cs = warp >> 2;            // TMEM lane quarter, column slice
    const int t = q * 32 + (tid & 31);                 // this thread's sample (= TMEM lane)
    const int c0 = cs * CW;                            // first column of this thread's slice
    const int up = tid >> 9, sj = tid & 127, sp = (tid >> 7) & 3;   // sums: half of the block, row or column, part
    const int tile = blockIdx.x;
    const long long s = (long long)tile * TS + t;
    const bool valid = s < a.n;
    const uint32_t bar_a = saddr(bar);

    // what the update kernel does not write comes before the wait for it
    float x0 = 0.0f, x1 = 0.0f, x2 = 0.0f;
    if (valid) {
        x0 = a.x[3 * s];
        x1 = a.x[3 * s + 1];
        x2 = a.x[3 * s + 2];
    }
    if (cs == 0) {
        xs[3 * t] = x0;
        xs[3 * t + 1] = x1;
        xs[3 * t + 2] = x2;
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar_a) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(saddr(tslot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tmg::pdl_wait();
    load_tile(B0, a.W2);
    load_tile(B1, a.W3);
    for (int i = tid; i < 384; i += NT) W1s[i] = bf16r(a.p[OFF_W1 + i]);
    for (int i = tid; i < 128; i += NT) {
        bs[i] = a.p[OFF_B1 + i];
        bs[128 + i] = a.p[OFF_B2 + i];
        bs[256 + i] = a.p[OFF_B3 + i];
    }
    for (int i = tid; i < 256; i += NT) W4s[i] = bf16r(a.p[OFF_W4 + i]);
    if (tid < 2) b4s[tid] = a.p[OFF_B4 + tid];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t lane = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;   // this warp's lanes and slice
    float* gp = TRAIN ? a.grad_part + (size_t)tile * PS : nullptr;
    uint32_t phase = 0;
    bool failed = false;
    __align__(16) __nv_bfloat16 hb[8];
    float v[8], dg[8], cv[8];
    // The passes over a thread's columns take 8 at a time in loops that stay loops: a
    // CTA runs this code once, so what it waited for most was instructions (4.6 of 12
    // stall cycles per issue with everything unrolled).

    do {
        // ---- layer 1 (CUDA cores): h1 = bf16(gelu(W1 x + b1)) -> B2 (A operand); h1^T -> B3
#pragma unroll 1
        for (int g = 0; g < CW / 8; ++g) {
            const int j = c0 + g * 8;
            layer1(W1s, bs, j, x0, x1, x2, v);
#pragma unroll
            for (int i = 0; i < 8; ++i) hb[i] = __float2bfloat16_rn(gelu(v[i]));
            store8(B2, t, j, hb);
        }
        if (TRAIN) transpose_warp(B2, B3, q * 32, c0);
        fence_async_smem();
        __syncthreads();
        if (tid == 0 && !a.probe_no_mma) {
            tc_fence_after();
            mma_128(tmem + 0, saddr(B2), saddr(B0));          // a2 - b2 -> TMEM cols 0..127
            mma_commit(bar_a);
        }
        failed = __syncthreads_or(warp == 0 && !bar_wait(bar_a, phase, a.wait_limit));
        phase ^= 1;
        if (failed) break;
        tc_fence_after();

        // ---- layer 2 epilogue: h2 = bf16(gelu(a2)) -> B2 (A operand); h2^T -> B4;
        //      gelu'(a2) takes the place of a2 - b2 in TMEM
#pragma unroll 1
        for (int g = 0; g < CW / 8; ++g) {
            tmem_ld8(lane + g * 8, v);
            lds8(bs + 128 + c0 + g * 8, cv);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float z = v[i] + cv[i];
                hb[i] = __float2bfloat16_rn(TRAIN ? gelu_and_grad(z, dg[i]) : gelu(z));
            }
            store8(B2, t, c0 + g * 8, hb);
            if (TRAIN) tmem_st8(lane + g * 8, dg);
        }
        if (TRAIN) transpose_warp(B2, B4, q * 32, c0);
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            mma_128(tmem + 128, saddr(B2), saddr(B1));        // a3 - b3 -> TMEM cols 128..255
            mma_commit(bar_a);
        }
        failed = __syncthreads_or(warp == 0 && !bar_wait(bar_a, phase, a.wait_limit));
        phase ^= 1;
        if (failed) break;
        tc_fence_after();

        // ---- layer 3 epilogue and output layer: y = W4 gelu(a3) + b4, h3 in FP32 in F (also for
        //      dW4), in four parts of 32 columns summed in order
#pragma unroll 1
        for (int g = 0; g < CW / 8; ++g) {
            tmem_ld8(lane + 128 + g * 8, v);
            lds8(bs + 256 + c0 + g * 8, cv);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float z = v[i] + cv[i];
                F[(c0 + g * 8 + i) * FPAD + t] = TRAIN ? gelu_and_grad(z, dg[i]) : gelu(z);
            }
            if (TRAIN) tmem_st8(lane + 128 + g * 8, dg);     // gelu'(a3)
        }
        __syncthreads();
        {
            // output `up` of sample sj over columns 32 sp .. 32 sp + 31
            float y = 0.0f;
#pragma unroll 1
            for (int j = 32 * sp; j < 32 * sp + 32; j += 8) {
                lds8(W4s + 128 * up + j, cv);
#pragma unroll
                for (int i = 0; i < 8; ++i) y = y + cv[i] * F[(j + i) * FPAD + sj];
            }
            red[(sp * TS + sj) * 3 + up] = y;
        }
        __syncthreads();
        float dy0 = 0.0f, dy1 = 0.0f;
        if (cs == 0) {
            float y0 = 0.0f, y1 = 0.0f;
            for (int p = 0; p < NS; ++p) {
                y0 = y0 + red[(p * TS + t) * 3];
                y1 = y1 + red[(p * TS + t) * 3 + 1];
            }
            y0 = y0 + b4s[0];
            y1 = y1 + b4s[1];
            if (!TRAIN) {
                if (valid) {
                    a.y_out[2 * s] = y0;
                    a.y_out[2 * s + 1] = y1;
                }
            } else {
                // loss and output-layer gradient of this sample
                float e0 = 0.0f, e1 = 0.0f, w0 = 0.0f, w1 = 0.0f;
                if (valid) {
                    e0 = y0 - a.y[2 * s];
                    e1 = y1 - a.y[2 * s + 1];
                    w0 = a.w[2 * s];
                    w1 = a.w[2 * s + 1];
                }
                ls[t] = w0 * e0 * e0 + w1 * e1 * e1;
                dys[2 * t] = ((2.0f * w0) * e0) * a.inv_norm;
                dys[2 * t + 1] = ((2.0f * w1) * e1) * a.inv_norm;
            }
        }
        if (!TRAIN) break;
        __syncthreads();
        dy0 = dys[2 * t];
        dy1 = dys[2 * t + 1];
        {
            // gW4[o][j] = sum_u dy_o[u] h3[u][j]: output `up`, column sj, samples 32 sp ..
            float g = 0.0f;
#pragma unroll 8
            for (int u = 32 * sp; u < 32 * sp + 32; ++u) g = g + dys[2 * u + up] * F[sj * FPAD + u];
            red[(sp * TS + sj) * 3 + up] = g;
        }
        __syncthreads();
        if (tid < 128) {
            float g0 = 0.0f, g1 = 0.0f;
            for (int p = 0; p < NS; ++p) {
                g0 = g0 + red[(p * TS + tid) * 3];
                g1 = g1 + red[(p * TS + tid) * 3 + 1];
            }
            gp[OFF_W4 + tid] = g0;
            gp[OFF_W4 + 128 + tid] = g1;
        }
        // the three sums over samples, in sample order, on three other warps
        if (tid == 128 || tid == 160 || tid == 192) {
            const float* from = tid == 128 ? dys : (tid == 160 ? dys + 1 : ls);
            const int step = tid == 192 ? 1 : 2;
            float sum = 0.0f;
#pragma unroll 16
            for (int u = 0; u < TS; ++u) sum = sum + from[step * u];
            if (tid == 192) a.loss_part[tile] = sum * a.inv_norm;
            else gp[OFF_B4 + (tid == 160)] = sum;
        }
        __syncthreads();                                      // F (B0..B2) and red free again

        // ---- dz3 = bf16((dy W4) * gelu'(a3)) -> B2 (A operand of dH2); dz3^T -> B5 (A operand of dW3)
        load_tile(B1, a.W3T);
#pragma unroll 1
        for (int g = 0; g < CW / 8; ++g) {
            tmem_ld8(lane + 128 + g * 8, dg);
            lds8(W4s + c0 + g * 8, cv);
            lds8(W4s + 128 + c0 + g * 8, v);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float dh = dy0 * cv[i] + dy1 * v[i];
                hb[i] = __float2bfloat16_rn(dh * dg[i]);
            }
            store8(B2, t, c0 + g * 8, hb);
        }
        transpose_warp(B2, B5, q * 32, c0);
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            mma_128(tmem + 256, saddr(B2), saddr(B1));        // dH2 = dz3 W3      -> cols 256..383
            mma_128(tmem + 384, saddr(B5), saddr(B4));        // gW3 = dz3^T h2    -> cols 384..511
            mma_commit(bar_a);
        }
        if (up == 0) red[(sp * TS + sj) * 3 + 2] = row_sum_part(B5, sj, sp);   // gb3 partial: row sj of dz3^T, samples 32 sp..
        failed = __syncthreads_or(warp == 0 && !bar_wait(bar_a, phase, a.wait_limit));
        phase ^= 1;
        if (failed) break;
        tc_fence_after();
        if (tid < 128) {
            float sb = 0.0f;
            for (int p = 0; p < NS; ++p) sb = sb + red[(p * TS + tid) * 3 + 2];
            gp[OFF_B3 + tid] = sb;
        }

        // ---- gW3 rows; dz2 = bf16(dH2 * gelu'(a2)) -> B2; dz2^T -> B5
        load_tile(B0, a.W2T);
#pragma unroll 1
        for (int g = 0; g < CW / 8; ++g) {
            tmem_ld8(lane + 384 + g * 8, v);
            stg8(gp + OFF_W3 + t * 128 + c0 + g * 8, v);
            tmem_ld8(lane + 256 + g * 8, v);
            tmem_ld8(lane + g * 8, dg);
#pragma unroll
            for (int i = 0; i < 8; ++i) hb[i] = __float2bfloat16_rn(v[i] * dg[i]);
            store8(B2, t, c0 + g * 8, hb);
        }
        transpose_warp(B2, B5, q * 32, c0);
        fence_async_smem();
        tc_fence_before();
        __syncthreads();                                      // also: every gb3 read of red is done
        if (tid == 0) {
            tc_fence_after();
            mma_128(tmem + 128, saddr(B2), saddr(B0));        // dH1 = dz2 W2      -> cols 128..255
            mma_128(tmem + 0, saddr(B5), saddr(B3));          // gW2 = dz2^T h1    -> cols 0..127
            mma_commit(bar_a);
        }
        if (up == 0) red[(sp * TS + sj) * 3 + 2] = row_sum_part(B5, sj, sp);   // gb2 partial
        failed = __syncthreads_or(warp == 0 && !bar_wait(bar_a, phase, a.wait_limit));
        phase ^= 1;
        if (failed) break;
        tc_fence_after();
        if (tid < 128) {
            float sb = 0.0f;
            for (int p = 0; p < NS; ++p) sb = sb + red[(p * TS + tid) * 3 + 2];
            gp[OFF_B2 + tid] = sb;
        }

        // ---- gW2 rows; dz1 = dH1 * gelu'(z1) (FP32) -> F; gW1, gb1 by column sums
#pragma unroll 1
        for (int g = 0; g < CW / 8; ++g) {
            tmem_ld8(lane + g * 8, v);
            stg8(gp + OFF_W2 + t * 128 + c0 + g * 8, v);
            tmem_ld8(lane + 128 + g * 8, v);
            layer1(W1s, bs, c0 + g * 8, x0, x1, x2, dg);
#pragma unroll
            for (int i = 0; i < 8; ++i) F[(c0 + g * 8 + i) * FPAD + t] = v[i] * gelu_grad(dg[i]);
        }
        __syncthreads();                                      // F complete; every gb2 read of red is done
        {
            // gW1[j][k] = sum_u dz1[u][j] x[u][k], k = 0, 1 by the lower half, 2 by the upper
            float g0 = 0.0f, g1 = 0.0f;
#pragma unroll 8
            for (int u = 32 * sp; u < 32 * sp + 32; ++u) {
                const float d = F[sj * FPAD + u];
                g0 = g0 + d * xs[3 * u + 2 * up];
                if (up == 0) g1 = g1 + d * xs[3 * u + 1];
            }
            red[(sp * TS + sj) * 3 + 2 * up] = g0;
            if (up == 0) red[(sp * TS + sj) * 3 + 1] = g1;
        }
        if (tid >= NT - 128) {                                // gb1, in sample order
            float gb = 0.0f;
#pragma unroll 16
            for (int u = 0; u < TS; ++u) gb = gb + F[sj * FPAD + u];
            gp[OFF_B1 + sj] = gb;
        }
        __syncthreads();
        if (tid < 128) {
            float g0 = 0.0f, g1 = 0.0f, g2 = 0.0f;
            for (int p = 0; p < NS; ++p) {
                g0 = g0 + red[(p * TS + tid) * 3];
                g1 = g1 + red[(p * TS + tid) * 3 + 1];
                g2 = g2 + red[(p * TS + tid) * 3 + 2];
            }
            gp[OFF_W1 + 3 * tid] = g0;
            gp[OFF_W1 + 3 * tid + 1] = g1;
            gp[OFF_W1 + 3 * tid + 2] = g2;
        }
    } while (false);

    if (failed) {
        // the wait on the phase just toggled past ran out: give the MMAs issued
        // for it one more bounded wait before their TMEM is freed
        if (tid == 0) atomicExch(a.err, 1);
        (void)bar_wait(bar_a, phase ^ 1u, a.wait_limit);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem) : "memory");
}

// Sum the partial gradients in tile order, optionally apply Adam, and refresh
// the BF16 copies of W2 and W3 (row-major and transposed).
struct AdamArgs {
    const float* part;
    int n_tiles;
    const float* loss_part;
    double* loss_out;                // sum of the partial losses (may be null)
    float* p;
    float* m;
    float* v;
    float* grad_out;                 // summed gradient (may be null)
    int update;
    float lr, b1, b2, eps, c1, c2;
    __nv_bfloat16 *W2, *W2T, *W3, *W3T;
    const int* err;                  // a tile kernel's wait ran out: the partials are invalid, change nothing
};

// A block's 64 parameters: its 256 threads bring 128 tiles' partials into shared memory
// at a time, all loads in flight together, and one thread per parameter adds them in
// tile order.  (One thread per parameter loading its own 94 partials waited for memory
// six times over: 9.6 us, 7.3 now, the serial FP64 loss sum included.)
constexpr int kAdamParams = 64, kAdamThreads = 256, kAdamTiles = 128;
constexpr int kAdamGrid = (NP + kAdamParams - 1) / kAdamParams + 1;      // the last block sums the loss

__global__ void __launch_bounds__(kAdamThreads) mlp_adam_kernel(AdamArgs a)
{
    __shared__ float part[kAdamTiles][kAdamParams];
    tmg::pdl_wait();
    if (a.err != nullptr && *a.err != 0) return;
    const int tid = threadIdx.x;
    if (blockIdx.x == gridDim.x - 1) {
        // FP64 sum of the FP32 losses: lanes take every 32nd tile, then a butterfly
        if (a.loss_out && tid < 32) {
            double sl = 0.0;
            for (int k = tid; k < a.n_tiles; k += 32) sl += (double)a.loss_part[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sl += __shfl_xor_sync(0xffffffffu, sl, o);
            if (tid == 0) *a.loss_out = sl;
        }
        return;
    }
    const int p0 = blockIdx.x * kAdamParams, i = p0 + tid;
    float g = 0.0f, pv = 0.0f, m0 = 0.0f, v0 = 0.0f;
    if (tid < kAdamParams && i < NP) {
        pv = a.p[i];
        if (a.update) {
            m0 = a.m[i];
            v0 = a.v[i];
        }
    }
    for (int k0 = 0; k0 < a.n_tiles; k0 += kAdamTiles) {
        const int nk = min(kAdamTiles, a.n_tiles - k0);
        const int c = tid % kAdamParams;
        if (k0 > 0) __syncthreads();
        // PS > NP: the columns beyond the last parameter are allocated, and not used
#pragma unroll 16
        for (int k = tid / kAdamParams; k < nk; k += kAdamThreads / kAdamParams)
            part[k][c] = p0 + c < PS ? a.part[(size_t)(k0 + k) * PS + p0 + c] : 0.0f;
        __syncthreads();
        if (tid < kAdamParams) {
#pragma unroll 16
            for (int k = 0; k < nk; ++k) g = g + part[k][tid];
        }
    }
    if (tid < kAdamParams && i < NP) {
        if (a.n_tiles > 0) {
            if (a.grad_out) a.grad_out[i] = g;
            if (a.update) {
                const float mv = a.b1 * m0 + (1.0f - a.b1) * g;
                const float vv = a.b2 * v0 + (1.0f - a.b2) * (g * g);
                pv = pv - a.lr * (mv * a.c1) / (sqrtf(vv * a.c2) + a.eps);
                a.m[i] = mv;
                a.v[i] = vv;
                a.p[i] = pv;
            }
        }
        if (i >= OFF_W2 && i < OFF_W2 + 16384) {
            const int r = (i - OFF_W2) >> 7, c = (i - OFF_W2) & 127;
            const __nv_bfloat16 h = __float2bfloat16_rn(pv);
            a.W2[r * 128 + c] = h;
            a.W2T[c * 128 + r] = h;
        } else if (i >= OFF_W3 && i < OFF_W3 + 16384) {
            const int r = (i - OFF_W3) >> 7, c = (i - OFF_W3) & 127;
            const __nv_bfloat16 h = __float2bfloat16_rn(pv);
            a.W3[r * 128 + c] = h;
            a.W3T[c * 128 + r] = h;
        }
    }
}

template <typename P>
cudaError_t dalloc(P** p, size_t n)
{
    *p = nullptr;
    return cudaMalloc(reinterpret_cast<void**>(p), n * sizeof(P));
}

}  // namespace

struct tm_mlp {
    tm_ctx* ctx = nullptr;
    float *p = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr;
    __nv_bfloat16 *W2 = nullptr, *W2T = nullptr, *W3 = nullptr, *W3T = nullptr;
    float *x = nullptr, *y = nullptr, *w = nullptr;   // training set
    int n = 0;
    float* part = nullptr;                             // [tiles][PS]
    float* loss_part = nullptr;
    int tiles_cap = 0;
    double* loss_dev = nullptr;
    int loss_cap = 0;
    float *px = nullptr, *py = nullptr;                // prediction buffers
    int pcap = 0;
    int* err = nullptr;
    long long step = 0;
};

namespace {

#define MLP_CUDA(call)                     \
    do {                                   \
        cudaError_t e__ = (call);          \
        if (e__ != cudaSuccess) {          \
            (void)cudaGetLastError();      \
            return TM_ERR_CUDA;            \
        }                                  \
    } while (0)

int grow_tiles(tm_mlp* m, int tiles)
{
    if (tiles <= m->tiles_cap) return TM_OK;
    cudaFree(m->part);
    cudaFree(m->loss_part);
    m->part = nullptr;
    m->loss_part = nullptr;
    m->tiles_cap = 0;
    if (dalloc(&m->part, (size_t)tiles * PS) != cudaSuccess || dalloc(&m->loss_part, (size_t)tiles) != cudaSuccess) {
        (void)cudaGetLastError();
        return TM_ERR_NOMEM;
    }
    m->tiles_cap = tiles;
    return TM_OK;
}

void launch_adam(const AdamArgs& a, cudaStream_t s)
{
    (void)tmg::launch_pdl(mlp_adam_kernel, dim3(kAdamGrid), dim3(kAdamThreads), 0, s, a);   // finish() reports errors
}

cudaError_t set_smem_attr()
{
    cudaError_t e = cudaFuncSetAttribute(mlp_tile_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_TOTAL);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(mlp_tile_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_TOTAL);
}

AdamArgs adam_args(tm_mlp* m, int n_tiles, double* loss_out, float* grad_out, int update, float lr, float b1,
                   float b2, float eps, float c1, float c2)
{
    AdamArgs a;
    a.part = m->part;
    a.n_tiles = n_tiles;
    a.loss_part = m->loss_part;
    a.loss_out = loss_out;
    a.p = m->p;
    a.m = m->m;
    a.v = m->v;
    a.grad_out = grad_out;
    a.update = update;
    a.lr = lr;
    a.b1 = b1;
    a.b2 = b2;
    a.eps = eps;
    a.c1 = c1;
    a.c2 = c2;
    a.W2 = m->W2;
    a.W2T = m->W2T;
    a.W3 = m->W3;
    a.W3T = m->W3T;
    a.err = m->err;
    return a;
}

MlpArgs tile_args(tm_mlp* m, const float* x, int n, float inv_norm, float* y_out)
{
    MlpArgs a;
    a.x = x;
    a.y = m->y;
    a.w = m->w;
    a.n = n;
    a.inv_norm = inv_norm;
    a.p = m->p;
    a.W2 = m->W2;
    a.W2T = m->W2T;
    a.W3 = m->W3;
    a.W3T = m->W3T;
    a.grad_part = m->part;
    a.loss_part = m->loss_part;
    a.y_out = y_out;
    a.err = m->err;
    a.probe_no_mma = (m->ctx->probe & TM_PROBE_MLP_WAIT) ? 1 : 0;
    a.wait_limit = a.probe_no_mma ? kProbeWaitLimit : kWaitLimit;
    return a;
}

int finish(tm_mlp* m)
{
    int herr = 0;
    MLP_CUDA(cudaGetLastError());
    MLP_CUDA(cudaMemcpyAsync(&herr, m->err, sizeof(int), cudaMemcpyDeviceToHost, m->ctx->stream));
    MLP_CUDA(cudaStreamSynchronize(m->ctx->stream));
    if (herr) {
        (void)cudaMemsetAsync(m->err, 0, sizeof(int), m->ctx->stream);
        (void)cudaStreamSynchronize(m->ctx->stream);
        return TM_ERR_TIMEOUT;
    }
    return TM_OK;
}

int upload_params(tm_mlp* m, const float* params)
{
    cudaStream_t s = m->ctx->stream;
    MLP_CUDA(cudaMemcpyAsync(m->p, params, NP * sizeof(float), cudaMemcpyHostToDevice, s));
    MLP_CUDA(cudaMemsetAsync(m->m, 0, NP * sizeof(float), s));
    MLP_CUDA(cudaMemsetAsync(m->v, 0, NP * sizeof(float), s));
    AdamArgs a = adam_args(m, 0, nullptr, nullptr, 0, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f);
    launch_adam(a, s);
    m->step = 0;
    return finish(m);
}

}  // namespace

extern "C" {

int tm_mlp_create(tm_ctx* ctx, const float* params, tm_mlp** out)
{
    if (!ctx || !params || !out) return TM_ERR_INVALID;
    *out = nullptr;
    tm_mlp* m = new (std::nothrow) tm_mlp();
    if (!m) return TM_ERR_NOMEM;
    m->ctx = ctx;
    if (cudaSetDevice(ctx->device) != cudaSuccess || set_smem_attr() != cudaSuccess) {
        (void)cudaGetLastError();
        delete m;
        return TM_ERR_CUDA;
    }
    if (dalloc(&m->p, NP) != cudaSuccess || dalloc(&m->m, NP) != cudaSuccess || dalloc(&m->v, NP) != cudaSuccess ||
        dalloc(&m->grad, NP) != cudaSuccess || dalloc(&m->W2, 16384) != cudaSuccess ||
        dalloc(&m->W2T, 16384) != cudaSuccess || dalloc(&m->W3, 16384) != cudaSuccess ||
        dalloc(&m->W3T, 16384) != cudaSuccess || dalloc(&m->err, 1) != cudaSuccess ||
        cudaMemset(m->err, 0, sizeof(int)) != cudaSuccess) {
        (void)cudaGetLastError();
        tm_mlp_destroy(m);
        return TM_ERR_NOMEM;
    }
    const int rc = upload_params(m, params);
    if (rc != TM_OK) {
        tm_mlp_destroy(m);
        return rc;
    }
    *out = m;
    return TM_OK;
}

int tm_mlp_destroy(tm_mlp* m)
{
    if (!m) return TM_ERR_INVALID;
    if (m->ctx) cudaSetDevice(m->ctx->device);
    void* ptrs[] = {m->p, m->m, m->v, m->grad, m->W2, m->W2T, m->W3, m->W3T, m->x, m->y, m->w,
                    m->part, m->loss_part, m->loss_dev, m->px, m->py, m->err};
    for (void* q : ptrs) cudaFree(q);
    (void)cudaGetLastError();
    delete m;
    return TM_OK;
}

int tm_mlp_set_params(tm_mlp* m, const float* params)
{
    if (!m || !params) return TM_ERR_INVALID;
    MLP_CUDA(cudaSetDevice(m->ctx->device));
    return upload_params(m, params);
}

int tm_mlp_get_params(tm_mlp* m, float* params)
{
    if (!m || !params) return TM_ERR_INVALID;
    MLP_CUDA(cudaSetDevice(m->ctx->device));
    MLP_CUDA(cudaMemcpyAsync(params, m->p, NP * sizeof(float), cudaMemcpyDeviceToHost, m->ctx->stream));
    MLP_CUDA(cudaStreamSynchronize(m->ctx->stream));
    return TM_OK;
}

int tm_mlp_set_data(tm_mlp* m, const float* x, const float* y, const float* w, int n)
{
    if (!m || !x || !y || !w || n < 1) return TM_ERR_INVALID;
    MLP_CUDA(cudaSetDevice(m->ctx->device));
    if (n > m->n) {
        cudaFree(m->x);
        cudaFree(m->y);
        cudaFree(m->w);
        m->x = m->y = m->w = nullptr;
        m->n = 0;
        if (dalloc(&m->x, (size_t)n * 3) != cudaSuccess || dalloc(&m->y, (size_t)n * 2) != cudaSuccess ||
            dalloc(&m->w, (size_t)n * 2) != cudaSuccess) {
            (void)cudaGetLastError();
            return TM_ERR_NOMEM;
        }
    }
    const int rc = grow_tiles(m, (n + TS - 1) / TS);
    if (rc != TM_OK) return rc;
    cudaStream_t s = m->ctx->stream;
    MLP_CUDA(cudaMemcpyAsync(m->x, x, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice, s));
    MLP_CUDA(cudaMemcpyAsync(m->y, y, (size_t)n * 2 * sizeof(float), cudaMemcpyHostToDevice, s));
    MLP_CUDA(cudaMemcpyAsync(m->w, w, (size_t)n * 2 * sizeof(float), cudaMemcpyHostToDevice, s));
    MLP_CUDA(cudaStreamSynchronize(s));
    m->n = n;
    return TM_OK;
}

int tm_mlp_loss_grad(tm_mlp* m, float inv_norm, double* loss, float* grad)
{
    if (!m || m->n < 1) return !m ? TM_ERR_INVALID : TM_ERR_STATE;
    MLP_CUDA(cudaSetDevice(m->ctx->device));
    if (m->loss_cap < 1) {
        if (dalloc(&m->loss_dev, 64) != cudaSuccess) return TM_ERR_NOMEM;
        m->loss_cap = 64;
    }
    cudaStream_t s = m->ctx->stream;
    const int tiles = (m->n + TS - 1) / TS;
    (void)tmg::launch_pdl(mlp_tile_kernel<true>, dim3(tiles), dim3(NT), SM_TOTAL, s, tile_args(m, m->x, m->n, inv_norm, nullptr));
    AdamArgs a = adam_args(m, tiles, m->loss_dev, m->grad, 0, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f);
    launch_adam(a, s);
    const int rc = finish(m);
    if (rc != TM_OK) return rc;
    if (grad) MLP_CUDA(cudaMemcpy(grad, m->grad, NP * sizeof(float), cudaMemcpyDeviceToHost));
    if (loss) MLP_CUDA(cudaMemcpy(loss, m->loss_dev, sizeof(double), cudaMemcpyDeviceToHost));
    return TM_OK;
}

int tm_mlp_train(tm_mlp* m, int steps, float lr, float beta1, float beta2, float eps, float inv_norm,
                 double* loss_hist)
{
    if (!m || steps < 0 || !(lr >= 0.f) || !(beta1 >= 0.f && beta1 < 1.f) || !(beta2 >= 0.f && beta2 < 1.f))
        return TM_ERR_INVALID;
    if (m->n < 1) return TM_ERR_STATE;
    MLP_CUDA(cudaSetDevice(m->ctx->device));
    if (steps > m->loss_cap) {
        cudaFree(m->loss_dev);
        m->loss_dev = nullptr;
        m->loss_cap = 0;
        if (dalloc(&m->loss_dev, (size_t)steps) != cudaSuccess) return TM_ERR_NOMEM;
        m->loss_cap = steps;
    }
    cudaStream_t s = m->ctx->stream;
    const int tiles = (m->n + TS - 1) / TS;
    for (int k = 0; k < steps; ++k) {
        const long long st = m->step + 1 + k;
        const float c1 = (float)(1.0 / (1.0 - std::pow((double)beta1, (double)st)));
        const float c2 = (float)(1.0 / (1.0 - std::pow((double)beta2, (double)st)));
        (void)tmg::launch_pdl(mlp_tile_kernel<true>, dim3(tiles), dim3(NT), SM_TOTAL, s, tile_args(m, m->x, m->n, inv_norm, nullptr));
        AdamArgs a = adam_args(m, tiles, m->loss_dev + k, nullptr, 1, lr, beta1, beta2, eps, c1, c2);
        launch_adam(a, s);
    }
    const int rc = finish(m);
    if (rc != TM_OK) return rc;
    m->step += steps;
    if (loss_hist && steps > 0)
        MLP_CUDA(cudaMemcpy(loss_hist, m->loss_dev, (size_t)steps * sizeof(double), cudaMemcpyDeviceToHost));
    return TM_OK;
}

int tm_mlp_predict(tm_mlp* m, const float* x, int n, float* y)
{
    if (!m || !x || !y || n < 0) return TM_ERR_INVALID;
    if (n == 0) return TM_OK;
    MLP_CUDA(cudaSetDevice(m->ctx->device));
    if (n > m->pcap) {
        cudaFree(m->px);
        cudaFree(m->py);
        m->px = m->py = nullptr;
        m->pcap = 0;
        if (dalloc(&m->px, (size_t)n * 3) != cudaSuccess || dalloc(&m->py, (size_t)n * 2) != cudaSuccess) {
            (void)cudaGetLastError();
            return TM_ERR_NOMEM;
        }
        m->pcap = n;
    }
    cudaStream_t s = m->ctx->stream;
    MLP_CUDA(cudaMemcpyAsync(m->px, x, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice, s));
    mlp_tile_kernel<false><<<(n + TS - 1) / TS, NT, SM_TOTAL, s>>>(tile_args(m, m->px, n, 0.f, m->py));
    const int rc = finish(m);
    if (rc != TM_OK) return rc;
    MLP_CUDA(cudaMemcpy(y, m->py, (size_t)n * 2 * sizeof(float), cudaMemcpyDeviceToHost));
    return TM_OK;
}

}  // extern "C"
