// tm_rk4.cu -- RK4 of the Rietkerk three-field right-hand side in FP64, fused in one
// pass over a shared-memory tile (tm_rk4_f32.cu: FP32), and the noise-off DP step's tiles.
//
// Rietkerk (rietkerk_bjork_FKE.cpp:2363-2444 stochastic remainder f_2Dor,
// :1760-1856 noise-off f_2D): the W and O tendencies carry 5-point
// Laplacians, so stage s needs stage s-1 values one site further out.  A CTA
// loads a region of [P*, W, O] with a halo of 4 (periodic wrap) into shared memory
// and runs all four stages there, stage s only on the region inset by s+1 cells, so
// the interior (64 columns by 24 or 12 rows) comes out exact after stage 4.
// The state is read and written once per step (plus the halo re-read, which
// hits L2); the K1..K4 temporaries the reference keeps as full lattices
// never leave the SM.
#include "tm_device.cuh"
#include "tm_kernels.cuh"

namespace tmg {

// c + s * x for a power of two s: s * x is exact, so the fused form rounds once,
// as the separate multiply and add do -- the same bits in one instruction.
template <typename T>
__device__ __forceinline__ T add_pow2_times(T c, T s, T x)
{
    return Tr<T>::fma_(s, x, c);
}

// One CTA per tile (persistent over tiles).  Stage s (0..3) is evaluated on
// the region inset by s+1 cells -- exactly the cells whose stage-s value an
// interior cell depends on -- so the interior is exact after stage 3.  Stage
// inputs ping-pong between two shared buffers, so each stage needs one barrier.
// Tile rows by bulk copy: for a tile that does not wrap in x on a lattice whose rows
// are multiples of 16 bytes, each of the halo rows is a contiguous segment of RK_RX
// values starting on a 16-byte boundary (instance offsets and field strides are
// multiples of 32 elements), so one thread per row and field issues it as a cp.async.bulk copy
// completing on an mbarrier instead of every thread loading values.
// Every wait on the copies is bounded (RK4Args::wait_limit polls, about 0.3 s at
// the default): a CTA whose copies do not complete marks the instances of its
// current and remaining tiles with TM_STATUS_WAIT_BIT (their fields are invalid
// after this step, and the host call returns TM_ERR_TIMEOUT), waits once more,
// again bounded, for copies still in flight into its shared memory, and exits.
// Under TM_PROBE_TILE_WAIT the CTA issues no copy and arms nothing, so the
// first wait runs out with nothing in flight (the test of this path).

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

// The region of tile t (RK_RX columns x ry_n rows of P, W, O, periodic) into X0.  False
// when its copies did not complete: the instances are flagged and the block returns.
__device__ __forceinline__ bool load_tile(const RK4Args<double>& A, double* X0, int ry_n, const double* __restrict__ P0,
                                          const double* __restrict__ W0, const double* __restrict__ O0, int L, int x0, int y0, int t,
                                          uint32_t bar, uint32_t& phase)
{
    const int tid = threadIdx.x, rn = RK_RX * ry_n;
    __syncthreads();  // previous tile done with shared memory
    // halo coordinates lie within RK_H of [0, L + tile), so one wrap is enough
    // once L covers the tile and its halo; smaller lattices take the modulo
    const bool one_wrap = L >= ry_n && L >= RK_RX;
    // one halo row per thread (3 x ry_n rows): the block takes the bulk path only if
    // every row start is 16-byte aligned
    const int n_rows = 3 * ry_n;
    const bool shape = (one_wrap && (L * sizeof(double)) % 16 == 0 && x0 >= RK_H && x0 + RK_TX + RK_H <= L) || A.probe_no_copy;
    const double* src = nullptr;
    bool aligned = true;
    if (shape && !A.probe_no_copy && tid < n_rows) {
        const int f = tid / ry_n, ry = tid - f * ry_n;
        int gy = y0 - RK_H + ry;
        gy = gy < 0 ? gy + L : (gy >= L ? gy - L : gy);
        src = (f == 0 ? P0 : (f == 1 ? W0 : O0)) + (long long)gy * L + (x0 - RK_H);
        aligned = ((uintptr_t)src & 15u) == 0;
    }
    if (shape && __syncthreads_and(aligned)) {
        if (!A.probe_no_copy) {
            constexpr uint32_t row_bytes = RK_RX * sizeof(double);
            static_assert(row_bytes % 16 == 0, "bulk rows");
            if (tid == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                             :: "r"(bar), "r"((uint32_t)n_rows * row_bytes) : "memory");
            __syncthreads();
            if (tid < n_rows) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
                             "[%0], [%1], %2, [%3];"
                             :: "r"(rk_saddr(X0 + tid * RK_RX)), "l"(src), "r"(row_bytes), "r"(bar)
                             : "memory");
            }
        }
        const bool ok = rk_bar_wait(bar, phase, A.wait_limit);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
            // copies did not complete: flag this tile's and every later tile's
            // instance, give copies still in flight one more bounded wait, stop
            for (int t2 = t + tid * (int)gridDim.x; t2 < A.n_tasks; t2 += (int)blockDim.x * (int)gridDim.x)
                atomicOr(A.it.status + A.tasks[t2].x, TM_STATUS_WAIT_BIT);
            (void)rk_bar_wait(bar, phase ^ 1u, A.wait_limit);
            return false;
        }
    } else {
#pragma unroll 2
        for (int c = tid; c < rn; c += (int)blockDim.x) {
            const int ry = c / RK_RX, rx = c - ry * RK_RX;
            int gy = y0 - RK_H + ry, gx = x0 - RK_H + rx;
            if (one_wrap) {
                gy = gy < 0 ? gy + L : (gy >= L ? gy - L : gy);
                gx = gx < 0 ? gx + L : (gx >= L ? gx - L : gx);
            } else {
                gy %= L; if (gy < 0) gy += L;
                gx %= L; if (gx < 0) gx += L;
            }
            const long long gi = (long long)gy * L + gx;
            X0[c] = P0[gi];
            X0[rn + c] = W0[gi];
            X0[2 * rn + c] = O0[gi];
        }
        __syncthreads();
    }
    return true;
}

// ---- the same step in FP64
// The FP64 pipe takes one warp instruction per 64-76 cycles, so the products run on the
// integer pipe and the quotients are exact integer divisions, the two by W + k1 sharing
// its reciprocal (tm_f64.cuh): 22 FP64 instructions per cell and stage, all of them
// additions, where the plain expressions took 58.  An evaluation is then some 900
// instructions long, so the code has one copy of it: one loop over the interior and
// ring cells of a stage, the stage a loop variable, and the weighted stage sums of a
// thread's interior cells rotating through fixed registers.  Tiles are 64 columns x
// tk.w rows (rk64_tile_rows, tm_capi.cu).
// Bound by the FP64 and the integer pipe taking turns (61 % and 46 % busy, 41 % of the
// issue slots): 768 threads (6 warps per scheduler, 76 registers) took 9.3 ms for 20 steps
// of 16 lattices of 256^2, 512 threads 10.1 and 1024 9.7; with some products back on the
// FP64 pipe 9.6 to 10.0.  The plain expressions took 15.2 ms (both with the draw of P*).
__device__ __forceinline__ double clamp_zero(double v, double clo, double ceps)
{
    // not below ceps if positive with larger bits (a NaN neither)
    const long long vb = __double_as_longlong(v);
    if (!(vb >= 0 && vb >= __double_as_longlong(ceps)) && vb != 0) {
        if (tmf::hw_in_range(v, clo, ceps)) return 0.0;
    }
    return v;
}

template <bool DET>
__device__ __forceinline__ void rk_rhs_cell64(const RK4Args<double>& A, const double* S, int rn, int c, double R, double& fP,
                                              double& fW, double& fO)
{
    const int cn = c - RK_RX, cs = c + RK_RX, cw = c - 1, ce = c + 1;
    const double* SP = S;
    const double* SW = S + rn;
    const double* SO = S + 2 * rn;
    const double Pc = SP[c], Wc = SW[c], Oc = SO[c];
    const double wk = Wc + A.k1;
    const uint32_t rw = tmf::recip_of(wk);
    fP = tmf::div_by(tmf::mul(tmf::mul(A.cgmax, Wc), Pc), wk, rw);
    const double upt = tmf::div_by(tmf::mul(tmf::mul(A.gmax, Wc), Pc), wk, rw);
    const double infil = tmf::mul(tmf::div(tmf::mul(A.alpha, Pc + A.k2W0), Pc + A.k2), Oc);
    const double lapW = add_pow2_times(((SW[cn] + SW[cs]) + SW[cw]) + SW[ce], -4.0, Wc);
    const double lapO = add_pow2_times(((SO[cn] + SO[cs]) + SO[cw]) + SO[ce], -4.0, Oc);
    if (DET) {
        const double lapP = add_pow2_times(((SP[cn] + SP[cs]) + SP[cw]) + SP[ce], -4.0, Pc);
        fP = (fP - tmf::mul(A.d, Pc)) + tmf::mul(A.DPx, lapP);
    }
    fW = ((infil - upt) - tmf::mul(A.rW, Wc)) + tmf::mul(A.DWx, lapW);
    fO = (R - infil) + tmf::mul(A.DOx, lapO);
}

template <bool DET>
__global__ void __launch_bounds__(RK64_THREADS, 1) rk4_tile64_kernel(const RK4Args<double> A)
{
    extern __shared__ __align__(16) unsigned char rk_smem[];
    constexpr int kMax = RK_TX * RK64_TY / RK64_THREADS;        // interior cells per thread in the tallest tile
    __shared__ __align__(8) uint64_t tile_bar;
    const int tid = threadIdx.x;
    const uint32_t bar = rk_saddr(&tile_bar);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_wait();
    __syncthreads();
    uint32_t phase = 0;
    for (int t = blockIdx.x; t < A.n_tasks; t += gridDim.x) {
        const int4 tk = A.tasks[t];
        const int k = tk.x;
        const int L = A.it.L[k];
        const long long off = A.it.off[k];
        const long long fs = A.it.fstride[k];
        const double R = A.it.R[k];
        const int x0 = tk.y, y0 = tk.z, ty = tk.w;
        const int ry_n = ty + 2 * RK_H, rn = RK_RX * ry_n;
        const int per = RK_TX * ty / RK64_THREADS;
        double* const X0 = reinterpret_cast<double*>(rk_smem);   // [3][rn] stage-0 input
        double* const MA = X0 + 3 * rn;                            // [3][rn] stage inputs (ping)
        double* const MB = MA + 3 * rn;                            // [3][rn] (pong)
        const double* __restrict__ P0 = (DET ? A.in : A.pstar) + off;
        const double* __restrict__ W0 = A.in + off + fs;
        const double* __restrict__ O0 = A.in + off + 2 * fs;
        if (!load_tile(A, X0, ry_n, P0, W0, O0, L, x0, y0, t, bar, phase)) return;
        double acc[3][kMax];
#pragma unroll
        for (int j = 0; j < kMax; ++j) acc[0][j] = acc[1][j] = acc[2][j] = 0.0;
#pragma unroll 1
        for (int s = 0; s < 4; ++s) {
            const double* S = (s == 0) ? X0 : ((s & 1) ? MA : MB);
            double* D = (s & 1) ? MB : MA;
            const double coef = (s == 2) ? A.dt : A.dt2;
            const double weight = (s == 0 || s == 3) ? 1.0 : 2.0;
            // the interior (per cells of this thread), then the ring between the region
            // inset by s + 1 and the interior: top and bottom bands (th rows of the
            // inset's width w), left and right bands (ty rows, th columns)
            const int in = s + 1, th = 3 - s, w = RK_RX - 2 * in;
            const int nband = th * w, nside = ty * th, nring = 2 * nband + 2 * nside;
#pragma unroll 1
            for (int q = 0; q < per || tid + (q - per) * RK64_THREADS < nring; ++q) {
                int rx, ry;
                const bool inner = q < per;
                if (inner) {
                    const int a = tid + q * RK64_THREADS;
                    ry = a / RK_TX + RK_H;
                    rx = a % RK_TX + RK_H;
                } else {
                    const int a = tid + (q - per) * RK64_THREADS;
                    if (a < 2 * nband) {
                        const int b = a < nband ? a : a - nband;
                        ry = (a < nband ? in : RK_H + ty) + b / w;
                        rx = in + b % w;
                    } else {
                        const int b = a - 2 * nband, b2 = b < nside ? b : b - nside;
                        ry = RK_H + b2 / th;
                        rx = (b < nside ? in : RK_H + RK_TX) + b2 % th;
                    }
                }
                const int c = ry * RK_RX + rx;
                double k0, k1, k2;
                rk_rhs_cell64<DET>(A, S, rn, c, R, k0, k1, k2);
                if (inner) {
                    // sums of K (weights 1, 2, 2, 1: each fused add rounds once, as k + 2 k'
                    // does); the front moves to the back
                    const double n0 = fma(weight, k0, acc[0][0]), n1 = fma(weight, k1, acc[1][0]),
                                 n2 = fma(weight, k2, acc[2][0]);
#pragma unroll
                    for (int j = 0; j + 1 < kMax; ++j) {
                        acc[0][j] = acc[0][j + 1]; acc[1][j] = acc[1][j + 1]; acc[2][j] = acc[2][j + 1];
                    }
                    acc[0][kMax - 1] = n0; acc[1][kMax - 1] = n1; acc[2][kMax - 1] = n2;
                }
                if (s < 3) {
                    D[c] = X0[c] + tmf::mul(coef, k0);
                    D[rn + c] = X0[rn + c] + tmf::mul(coef, k1);
                    D[2 * rn + c] = X0[2 * rn + c] + tmf::mul(coef, k2);
                }
            }
            for (int q = per; q < kMax; ++q) {               // shorter tiles: bring the first cell to the front
                const double n0 = acc[0][0], n1 = acc[1][0], n2 = acc[2][0];
#pragma unroll
                for (int j = 0; j + 1 < kMax; ++j) {
                    acc[0][j] = acc[0][j + 1]; acc[1][j] = acc[1][j + 1]; acc[2][j] = acc[2][j + 1];
                }
                acc[0][kMax - 1] = n0; acc[1][kMax - 1] = n1; acc[2][kMax - 1] = n2;
            }
            __syncthreads();
        }
        unsigned st = 0;
#pragma unroll
        for (int j = 0; j < kMax; ++j) {
            const int a = tid + j * RK64_THREADS;
            const int ly = a / RK_TX, lx = a % RK_TX;
            const int gy = y0 + ly, gx = x0 + lx;
            if (j < per && gy < L && gx < L) {
                const int c = (ly + RK_H) * RK_RX + lx + RK_H;
                const long long gi = off + (long long)gy * L + gx;
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                    const double v = clamp_zero(X0[f * rn + c] + A.dt6 * acc[f][j], A.clo, A.ceps);
                    st |= value_status(v);
                    A.out[gi + f * fs] = v;
                }
            }
        }
        if (st) atomicOr(A.it.status + k, st);
    }
}

template <>
cudaError_t launch_rk4<double>(const RK4Args<double>& a, bool det, int grid, cudaStream_t s)
{
    if (a.n_tasks <= 0) return cudaSuccess;
    const size_t smem = 9 * (size_t)RK_RX * (RK64_TY + 2 * RK_H) * sizeof(double);   // of the tallest tile
    static PerDevice allowed[2];
    const auto kernel = det ? rk4_tile64_kernel<true> : rk4_tile64_kernel<false>;
    const cudaError_t e = allow_smem(allowed[det ? 1 : 0], kernel, smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(kernel, dim3(grid), dim3(RK64_THREADS), smem, s, a);
}

// ---- noise-off DP: drho/dt = a rho - b rho^2 - c rho^3 + D Lap(rho) ---------------
// percNoDiff_2D (stochasticSPDP.cpp:549-662) with the 5-point Laplacian or the
// 4th-order cross of fP_2D (:516-529), written as f = react - D/(12 dx^2)
// (o2 - 16 o1 + 60 rho).  One CTA per 64 x 32 tile (persistent over the tiles of
// every instance), all stages in shared memory as in rk4_tile_kernel: a stencil of
// radius RAD makes stage s need stage s-1 values RAD sites further out, so the tile
// loads a halo of NST * RAD sites and evaluates stage s on the region inset by
// (s+1) RAD.  The reference keeps K1..K4 and the stage input as full lattices
// (:594-626); here they never leave the SM, and one launch per step covers the
// whole batch.
template <typename T, int RAD>
__device__ __forceinline__ T dp_det_rhs(const DetTileArgs<T>& A, const T* S, int c, int rx, T a)
{
    const T r = S[c];
    T f = (a * r) - ((A.b * r) * r);
    if (A.cubic) f = f - ((A.c * r) * r) * r;
    if constexpr (RAD == 1) {
        const T lap = add_pow2_times(((S[c - rx] + S[c + rx]) + S[c - 1]) + S[c + 1], T(-4), r);
        f = f + A.dlap * lap;
    } else {
        const T o2 = ((S[c - 2 * rx] + S[c + 2 * rx]) + S[c - 2]) + S[c + 2];
        const T o1 = ((S[c - rx] + S[c + rx]) + S[c - 1]) + S[c + 1];
        const T sm = add_pow2_times(o2, T(-16), o1) + T(60) * r;
        f = f - A.dk12 * sm;
    }
    return f;
}

template <typename T, int RAD, int NST>
__global__ void __launch_bounds__(RK_THREADS, 1) dp_det_tile_kernel(const DetTileArgs<T> A)
{
    constexpr int H = RAD * NST, RX = RK_TX + 2 * H, RY = RK_TY + 2 * H, RN = RX * RY;
    constexpr int kPer = RK_TX * RK_TY / RK_THREADS;
    extern __shared__ __align__(16) unsigned char det_smem[];
    T* const X0 = reinterpret_cast<T*>(det_smem);
    T* const MA = X0 + RN;
    T* const MB = MA + RN;
    const int tid = threadIdx.x;
    pdl_wait();
    for (int t = blockIdx.x; t < A.n_tasks; t += gridDim.x) {
        const int4 tk = A.tasks[t];
        const int k = tk.x;
        const int L = A.it.L[k];
        const long long off = A.it.off[k];
        const T a = (T)A.it.R[k];
        const int x0 = tk.y, y0 = tk.z;
        const T* __restrict__ src = A.in + off;
        __syncthreads();  // previous tile done with shared memory
        const bool one_wrap = L >= RY && L >= RX;
        for (int c = tid; c < RN; c += RK_THREADS) {
            const int ry = c / RX, rx = c - ry * RX;
            int gy = y0 - H + ry, gx = x0 - H + rx;
            if (one_wrap) {
                gy = gy < 0 ? gy + L : (gy >= L ? gy - L : gy);
                gx = gx < 0 ? gx + L : (gx >= L ? gx - L : gx);
            } else {
                gy %= L; if (gy < 0) gy += L;
                gx %= L; if (gx < 0) gx += L;
            }
            X0[c] = src[(long long)gy * L + gx];
        }
        __syncthreads();
        T acc[kPer];
#pragma unroll
        for (int s = 0; s < NST; ++s) {
            const T* S = (s == 0) ? X0 : ((s & 1) ? MA : MB);
            T* D = (s & 1) ? MB : MA;
            const T coef = (s == 2) ? A.dt : A.dt2;
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int q = tid + j * RK_THREADS;
                const int c = ((q / RK_TX) + H) * RX + (q % RK_TX) + H;
                const T kv = dp_det_rhs<T, RAD>(A, S, c, RX, a);
                if (s == 0) acc[j] = kv;
                else if (s == NST - 1) acc[j] = acc[j] + kv;
                else acc[j] = add_pow2_times(acc[j], T(2), kv);
                if (s < NST - 1) D[c] = X0[c] + coef * kv;
            }
            if (s < NST - 1) {
                // ring between the region inset by (s+1) RAD and the interior: top and
                // bottom bands (tt rows of the inset's width w), left and right bands
                const int in = (s + 1) * RAD, tt = H - in, w = RX - 2 * in;
                const int nband = tt * w, nside = RK_TY * tt;
                for (int q = tid; q < 2 * nband + 2 * nside; q += RK_THREADS) {
                    int ry, rx;
                    if (q < 2 * nband) {
                        const int qb = q < nband ? q : q - nband;
                        ry = (q < nband ? in : H + RK_TY) + qb / w;
                        rx = in + qb % w;
                    } else {
                        const int qs = q - 2 * nband;
                        const int qq = qs < nside ? qs : qs - nside;
                        ry = H + qq / tt;
                        rx = (qs < nside ? in : H + RK_TX) + qq % tt;
                    }
                    const int c = ry * RX + rx;
                    D[c] = X0[c] + coef * dp_det_rhs<T, RAD>(A, S, c, RX, a);
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int q = tid + j * RK_THREADS;
            const int ly = q / RK_TX, lx = q % RK_TX;
            const int gy = y0 + ly, gx = x0 + lx;
            if (gy < L && gx < L) {
                const int c = (ly + H) * RX + lx + H;
                const T v = (NST == 4) ? X0[c] + A.dt6 * acc[j] : X0[c] + acc[j] * A.dt;
                A.out[off + (long long)gy * L + gx] = v;
            }
        }
    }
}

template <typename T, int RAD, int NST>
cudaError_t launch_det_t(const DetTileArgs<T>& a, int grid, cudaStream_t s)
{
    constexpr int H = RAD * NST;
    const size_t smem = 3 * (size_t)(RK_TX + 2 * H) * (RK_TY + 2 * H) * sizeof(T);
    static PerDevice allowed;
    const cudaError_t e = allow_smem(allowed, dp_det_tile_kernel<T, RAD, NST>, smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(dp_det_tile_kernel<T, RAD, NST>, dim3(grid), dim3(RK_THREADS), smem, s, a);
}

template <typename T>
cudaError_t launch_dp_det(const DetTileArgs<T>& a, int stencil, int rk4, int grid, cudaStream_t s)
{
    if (a.n_tasks <= 0) return cudaSuccess;
    if (stencil == 5) return rk4 ? launch_det_t<T, 1, 4>(a, grid, s) : launch_det_t<T, 1, 1>(a, grid, s);
    if (stencil == 9) return rk4 ? launch_det_t<T, 2, 4>(a, grid, s) : launch_det_t<T, 2, 1>(a, grid, s);
    return cudaErrorInvalidValue;
}
template cudaError_t launch_dp_det<float>(const DetTileArgs<float>&, int, int, int, cudaStream_t);
template cudaError_t launch_dp_det<double>(const DetTileArgs<double>&, int, int, int, cudaStream_t);

}  // namespace tmg
