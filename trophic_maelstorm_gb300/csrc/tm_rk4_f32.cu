// tm_rk4_f32.cu -- RK4 of the Rietkerk three-field right-hand side in FP32, fused in
// one pass over a shared-memory tile.
//
// Rietkerk (rietkerk_bjork_FKE.cpp:2363-2444 stochastic remainder f_2Dor,
// :1760-1856 noise-off f_2D): the W and O tendencies carry 5-point Laplacians (P's
// too when the noise is off), so stage s needs stage s-1 values one site further
// out.  A CTA copies a (64+8) x (32+8) region of [P*, W, O] (halo 4, periodic wrap)
// into shared memory and runs all four stages there, stage s only on the region inset
// by s+1 cells, so the 64 x 32 interior comes out exact after stage 4.  Stage inputs
// ping-pong between two shared buffers, so each stage needs one barrier; the weighted
// stage sums of the interior stay in registers (fixed thread mapping).
//
// A thread evaluates two neighbouring cells at once with 8-byte shared-memory accesses.
// The region is 36 pairs wide; pairs that stick out of a stage's inset compute a cell
// nobody reads.  The reciprocals are the FP32 estimate and one fused Newton step (neg_rcp);
// a pair whose residuals show an argument outside that method's range takes __frcp_rn.
// Measured at 2048^2: 83.5 us a step one cell at a time with __frcp_rn and every warp
// polling for the copies, 73 us now; bound by the stages' barriers and the issue slots
// (58 %) in turns.  Slower: three CTAs of 64 x 20 tiles (2 %), four of 64 x 12 (4 %), one
// of 1024 threads (18 %), the whole state in registers with rows exchanged through shared
// memory (one CTA per SM: 60 %).  Packed add/mul/fma.f32x2 saved a tenth of the
// instructions and 4 % of the time, but the compiler contracts packed products with
// packed sums whatever their rounding says.
//
// Tile rows by bulk copy: where the lattice's rows are multiples of 16 bytes and at
// least a region wide, each halo row is one contiguous segment (two where it wraps)
// starting on a 16-byte boundary, so one thread per row and field issues it as
// cp.async.bulk copies completing on an mbarrier; other tiles use per-thread loads.
// The copies of the next tile start when a tile's second buffer is free, before its
// last stage.
// Every wait on the copies is bounded (RK4Args::wait_limit polls, about 0.3 s at
// the default): a CTA whose copies do not complete marks the instances of its
// current and remaining tiles with TM_STATUS_WAIT_BIT (their fields are invalid
// after this step, and the host call returns TM_ERR_TIMEOUT), waits once more,
// again bounded, for copies still in flight into its shared memory, and exits.
// Under TM_PROBE_TILE_WAIT the CTA issues no copy and arms nothing, so the
// first wait runs out with nothing in flight (the test of this path).
#include "tm_device.cuh"
#include "tm_kernels.cuh"

namespace tmg {

namespace {

__device__ __forceinline__ float2 ld2(const float* p) { return *reinterpret_cast<const float2*>(p); }

// c + s x for a power of two s: s x is exact, so the fused form rounds once, as the
// separate multiply and add do -- the same bits in one instruction.
__device__ __forceinline__ float add_pow2_times(float c, float s, float x) { return fmaf(s, x, c); }

// the five-point Laplacians of the pair at float offset c (even): ((north + south) +
// west) + east - 4 x
__device__ __forceinline__ float2 laplacian(const float* S, int c, float2 x)
{
    const float2 n = ld2(S + c - RK_RX), s = ld2(S + c + RK_RX);
    return make_float2(add_pow2_times(((n.x + s.x) + S[c - 1]) + x.y, -4.0f, x.x),
                       add_pow2_times(((n.y + s.y) + x.x) + S[c + 2], -4.0f, x.y));
}

struct Tend {
    float P, W, O;
};

// Right-hand side of one cell (f_2Dor, or f_2D when DET) from its values, its
// Laplacians and the negated reciprocals of W + k1 and P + k2.  The constants those
// multiply are negated too (a product's rounding is symmetric).
template <bool DET>
__device__ __forceinline__ Tend rhs_cell(const RK4Args<float>& A, float R, float P, float W, float O, float lapP, float lapW,
                                         float lapO, float n_iwk, float n_ipk)
{
    const float infil = (((-A.alpha) * (P + A.k2W0)) * n_ipk) * O;
    Tend f;
    f.P = (((-A.cgmax) * W) * P) * n_iwk;
    const float upt = (((-A.gmax) * W) * P) * n_iwk;
    if (DET) f.P = (f.P - A.d * P) + A.DPx * lapP;
    f.W = ((infil - upt) - A.rW * W) + A.DWx * lapW;
    f.O = (R - infil) + A.DOx * lapO;
    return f;
}

// Tendencies of the pair at region offset c of S.
template <bool DET>
__device__ __forceinline__ void rhs_pair(const RK4Args<float>& A, const float* S, int c, float R, Tend& f0, Tend& f1)
{
    const float2 P = ld2(S + c), W = ld2(S + RK_RN + c), O = ld2(S + 2 * RK_RN + c);
    const float2 lapW = laplacian(S + RK_RN, c, W), lapO = laplacian(S + 2 * RK_RN, c, O);
    float2 lapP = make_float2(0.0f, 0.0f);
    if (DET) lapP = laplacian(S, c, P);
    const float wk0 = W.x + A.k1, wk1 = W.y + A.k1, pk0 = P.x + A.k2, pk1 = P.y + A.k2;
    bool ok = true;
    float iw0 = neg_rcp(wk0, ok), iw1 = neg_rcp(wk1, ok), ip0 = neg_rcp(pk0, ok), ip1 = neg_rcp(pk1, ok);
    if (!ok) {
        iw0 = -__frcp_rn(wk0); iw1 = -__frcp_rn(wk1);
        ip0 = -__frcp_rn(pk0); ip1 = -__frcp_rn(pk1);
    }
    f0 = rhs_cell<DET>(A, R, P.x, W.x, O.x, lapP.x, lapW.x, lapO.x, iw0, ip0);
    f1 = rhs_cell<DET>(A, R, P.y, W.y, O.y, lapP.y, lapW.y, lapO.y, iw1, ip1);
}

__device__ __forceinline__ uint32_t rk_saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool rk_bar_wait(uint32_t bar, uint32_t parity, int limit)
{
    for (int i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if (i > 16) __nanosleep(32);
    }
    return false;
}

__device__ __forceinline__ void bulk_copy(uint32_t to, const float* from, int n, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(to), "l"(from), "r"((uint32_t)(n * sizeof(float))), "r"(bar) : "memory");
}

// Whether a tile's region comes by bulk copies: rows of whole 16-byte units and at least
// a region wide, fields 16-byte aligned (their offsets and strides are multiples of 32
// elements).
template <bool DET>
__device__ __forceinline__ bool by_copies(const RK4Args<float>& A, int L)
{
    return ((L & 3) == 0 && L >= RK_RX && (((uintptr_t)A.in | (uintptr_t)(DET ? A.in : A.pstar)) & 15u) == 0) ||
           A.probe_no_copy;
}

// Starts the copies of task tk's region into X (3 x RK_RY rows, one thread each); they
// complete on the barrier, armed by thread 0 (the phase cannot end before its arrival).
template <bool DET>
__device__ __forceinline__ void start_copies(const RK4Args<float>& A, const int4 tk, float* X, uint32_t bar)
{
    constexpr int kRows = 3 * RK_RY;
    if (A.probe_no_copy) return;
    if (threadIdx.x == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                     :: "r"(bar), "r"((uint32_t)(kRows * RK_RX * sizeof(float))) : "memory");
    if (threadIdx.x < kRows) {
        const int L = A.it.L[tk.x];
        const int f = threadIdx.x / RK_RY, ry = threadIdx.x - f * RK_RY;
        int gy = (tk.z - RK_H + ry) % L;
        if (gy < 0) gy += L;
        const int gx = tk.y < RK_H ? tk.y - RK_H + L : tk.y - RK_H;
        const int n1 = min(RK_RX, L - gx);
        const float* src = (f == 0 && !DET ? A.pstar : A.in + f * A.it.fstride[tk.x]) + A.it.off[tk.x] + (long long)gy * L;
        const uint32_t to = rk_saddr(X + threadIdx.x * RK_RX);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        bulk_copy(to, src + gx, n1, bar);
        if (n1 < RK_RX) bulk_copy(to + (uint32_t)(n1 * sizeof(float)), src, RK_RX - n1, bar);
    }
}

// Waits for tile t's copies.  False when they did not complete: this tile's and every
// later tile's instances are flagged, copies still in flight get one more bounded wait,
// and the block returns.
__device__ __forceinline__ bool wait_copies(const RK4Args<float>& A, int t, uint32_t bar, uint32_t& phase)
{
    // one warp polls: 16 polling warps took a fifth of the issue slots
    const bool ok = threadIdx.x >= 32 || rk_bar_wait(bar, phase, A.wait_limit);
    phase ^= 1u;
    if (!__syncthreads_or(!ok)) return true;
    for (int t2 = t + (int)threadIdx.x * (int)gridDim.x; t2 < A.n_tasks; t2 += RK_THREADS * (int)gridDim.x)
        atomicOr(A.it.status + A.tasks[t2].x, TM_STATUS_WAIT_BIT);
    (void)rk_bar_wait(bar, phase ^ 1u, A.wait_limit);
    return false;
}

// The region of a tile by per-thread loads.
template <bool DET>
__device__ __forceinline__ void load_region(const RK4Args<float>& A, const int4 tk, float* X)
{
    const int L = A.it.L[tk.x];
    const long long off = A.it.off[tk.x], fs = A.it.fstride[tk.x];
    for (int c = threadIdx.x; c < RK_RN; c += RK_THREADS) {
        const int ry = c / RK_RX, rx = c - ry * RK_RX;
        int gy = (tk.z - RK_H + ry) % L, gx = (tk.y - RK_H + rx) % L;
        if (gy < 0) gy += L;
        if (gx < 0) gx += L;
        const long long gi = off + (long long)gy * L + gx;
        X[c] = (DET ? A.in : A.pstar)[gi];
        X[RK_RN + c] = A.in[gi + fs];
        X[2 * RK_RN + c] = A.in[gi + 2 * fs];
    }
    __syncthreads();
}

}  // namespace

// One CTA per tile (persistent over tiles), two CTAs per SM.
template <bool DET>
__global__ void __launch_bounds__(RK_THREADS, RK_CTAS) rk4_tile_kernel(const RK4Args<float> A)
{
    extern __shared__ __align__(16) unsigned char rk_smem[];
    __shared__ __align__(8) uint64_t tile_bar;
    float* X0 = reinterpret_cast<float*>(rk_smem);                // [3][RK_RN] stage-0 input
    float* MA = X0 + 3 * RK_RN;                                     // [3][RK_RN] stage inputs (ping)
    float* MB = MA + 3 * RK_RN;                                     // [3][RK_RN] (pong)
    constexpr int kPer = RK_TX * RK_TY / 2 / RK_THREADS;            // interior pairs per thread
    static_assert(RK_TX * RK_TY % (2 * RK_THREADS) == 0 && RK_TX == 64, "a warp owns one interior row");
    const int tid = threadIdx.x;
    const uint32_t bar = rk_saddr(&tile_bar);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_wait();
    __syncthreads();
    uint32_t phase = 0;
    if ((int)blockIdx.x < A.n_tasks && by_copies<DET>(A, A.it.L[A.tasks[blockIdx.x].x]))
        start_copies<DET>(A, A.tasks[blockIdx.x], X0, bar);
    // this thread's interior pairs: rows w, w + 16 of the tile, columns 2 lane, 2 lane + 1
    const int c_in = ((tid >> 5) + RK_H) * RK_RX + RK_H + 2 * (tid & 31);
    constexpr int kStep = RK_THREADS / 32 * RK_RX;
    for (int t = blockIdx.x; t < A.n_tasks; t += gridDim.x) {
        const int4 tk = A.tasks[t];
        const int k = tk.x;
        const int L = A.it.L[k];
        const long long off = A.it.off[k];
        const long long fs = A.it.fstride[k];
        const float R = (float)A.it.R[k];
        const int x0 = tk.y, y0 = tk.z;
        if (by_copies<DET>(A, L)) {
            if (!wait_copies(A, t, bar, phase)) return;
        } else {
            load_region<DET>(A, tk, X0);
        }
        float2 acc[3][kPer];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const float* S = (s == 0) ? X0 : ((s & 1) ? MA : MB);
            float* D = (s & 1) ? MB : MA;
            const float coef = (s == 2) ? A.dt : A.dt2;
            auto advance = [&](int c, const Tend& f0, const Tend& f1) {
                auto put = [&](int o, float k0, float k1) {
                    const float2 x = ld2(X0 + o);
                    *reinterpret_cast<float2*>(D + o) = make_float2(x.x + coef * k0, x.y + coef * k1);
                };
                put(c, f0.P, f1.P);
                put(c + RK_RN, f0.W, f1.W);
                put(c + 2 * RK_RN, f0.O, f1.O);
            };
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int c = c_in + j * kStep;
                Tend f0, f1;
                rhs_pair<DET>(A, S, c, R, f0, f1);
                auto sum = [&](float2& a, float k0, float k1) {
                    if (s == 0) a = make_float2(k0, k1);
                    else if (s == 3) a = make_float2(a.x + k0, a.y + k1);
                    else a = make_float2(add_pow2_times(a.x, 2.0f, k0), add_pow2_times(a.y, 2.0f, k1));
                };
                sum(acc[0][j], f0.P, f1.P);
                sum(acc[1][j], f0.W, f1.W);
                sum(acc[2][j], f0.O, f1.O);
                if (s < 3) advance(c, f0, f1);
            }
            if (s < 3) {
                // pairs of the inset outside the interior: th rows above and below, np pairs
                // each from pair p0 on, and ns pairs a row left and right of the interior
                constexpr int kAll = RK_RX / 2;
                const int th = 3 - s, p0 = s == 0 ? 0 : 1, np = kAll - 2 * p0, ns = 2 - p0;
                const int nband = th * np, nside = RK_TY * ns;
                for (int q = tid; q < 2 * nband + 2 * nside; q += RK_THREADS) {
                    int ry, px;
                    if (q < 2 * nband) {
                        const int qb = q < nband ? q : q - nband;
                        ry = (q < nband ? s + 1 : RK_H + RK_TY) + qb / np;
                        px = p0 + qb % np;
                    } else {
                        const int qs = q - 2 * nband;
                        const int qq = qs < nside ? qs : qs - nside;
                        ry = RK_H + qq / ns;
                        px = (qs < nside ? p0 : kAll - 2) + qq % ns;
                    }
                    // the region's first and last value have no neighbour: any will do there
                    const int c = ry * RK_RX + 2 * px;
                    Tend f0, f1;
                    rhs_pair<DET>(A, S, c, R, f0, f1);
                    advance(c, f0, f1);
                }
            }
            if (s == 3) break;
            __syncthreads();
            if (s == 2) {
                // nobody reads MB any more: the next tile's region goes there
                const int tn = t + (int)gridDim.x;
                if (tn < A.n_tasks && by_copies<DET>(A, A.it.L[A.tasks[tn].x])) start_copies<DET>(A, A.tasks[tn], MB, bar);
            }
        }
        unsigned top = 0;
        const int gx = x0 + 2 * (tid & 31);
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int gy = y0 + (tid >> 5) + j * (RK_THREADS / 32);
            const int c = c_in + j * kStep;
            if (gy < L && gx < L) {
                const long long gi = off + (long long)gy * L + gx;
                const bool two = gx + 1 < L;
                // fields start on multiples of 32 elements, so one parity serves all three
                const bool wide = two && (((uintptr_t)(A.out + gi)) & 7u) == 0;
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                    const float2 x = ld2(X0 + f * RK_RN + c);
                    float a = x.x + A.dt6 * acc[f][j].x, b = x.y + A.dt6 * acc[f][j].y;
                    if (a < A.ceps && a >= A.clo) a = 0.0f;
                    if (b < A.ceps && b >= A.clo) b = 0.0f;
                    // The status bits by the largest bit pattern: NaN, Inf and signs lie
                    // above the finite values, and what was stored is looked at again then
                    // (a test per value took 8 % of the tile's instructions; 4096 x 4096,
                    // 24 steps: 11.61 ms with it, 11.36 without).
                    top = max(top, __float_as_uint(a));
                    if (two) top = max(top, __float_as_uint(b));
                    float* out = A.out + gi + f * fs;
                    if (wide) {
                        *reinterpret_cast<float2*>(out) = make_float2(a, b);
                    } else {
                        out[0] = a;
                        if (two) out[1] = b;
                    }
                }
            }
        }
        if (top >= 0x7f800000u) {
            unsigned st = 0;
#pragma unroll 1
            for (int j = 0; j < kPer; ++j) {
                const int gy = y0 + (tid >> 5) + j * (RK_THREADS / 32);
                if (gy >= L || gx >= L) continue;
                for (int f = 0; f < 3; ++f) {
                    const float* out = A.out + off + (long long)gy * L + gx + f * fs;
                    st |= value_status(out[0]);
                    if (gx + 1 < L) st |= value_status(out[1]);
                }
            }
            if (st) atomicOr(A.it.status + k, st);
        }
        // the buffers rotate; MA and X0 are not written before the next tile's first barrier
        float* const next = MB;
        MB = X0;
        X0 = next;
    }
}

template <>
cudaError_t launch_rk4<float>(const RK4Args<float>& a, bool det, int grid, cudaStream_t s)
{
    if (a.n_tasks <= 0) return cudaSuccess;
    const size_t smem = 9 * (size_t)RK_RN * sizeof(float);
    static PerDevice allowed[2];
    const auto kernel = det ? rk4_tile_kernel<true> : rk4_tile_kernel<false>;
    const cudaError_t e = allow_smem(allowed[det ? 1 : 0], kernel, smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(kernel, dim3(grid), dim3(RK_THREADS), smem, s, a);
}

}  // namespace tmg
