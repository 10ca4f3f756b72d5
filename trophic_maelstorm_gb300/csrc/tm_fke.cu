// tm_fke.cu -- FKE advection-diffusion of a consumer field, as separable gathers.
//
// The reference moves its consumer species with advdiff_FKE_MultiSp
// (simulations/Rietkerk_FPE/rietkerk_bjork_FKE.cpp:3614-3695) and, on the GPU,
// with updateMovement (kernel_advdiff_FKE2D.cu:92-180): every source site with
// rho >= eps scatters its mass through four separable Gaussian stencils
// (diffusion around the site, advection around the site shifted by
// round(v * pref), and the two mixed products), the reference kernel with FP64
// atomicAdd.  Here the four terms are grouped by their row stencil and
// gathered in two passes, with no atomics (the result does not depend on
// scheduling):
//   pass 1, along rows:  A_D[r][q] = sum over the sources of row r of
//                                    wDD gD(q - cj) + wDV gV(q - muy)
//                        A_V[r][q] = the same sum over the sources whose
//                                    shifted row mux is r, of wDV gD(q - cj) + wVV gV(q - muy)
//   pass 2, down columns: out[p][q] = sum_r gD(p - r) A_D[r][q] + gV(p - r) A_V[r][q]
// with wDD = gamma^2 rho, wDV = gamma (1 - gamma) rho, wVV = (1 - gamma)^2 rho,
// and gD, gV the stencils wrapped onto the periodic lattice (summed over every
// image, so lattices narrower than a stencil are exact).  A site costs about 10
// FP64 instructions for its weights and shift, a few additions where weights land on
// one site, and 3 (2 RD + 1) + 3 (2 RV + 1) fused multiply-adds.
#include "tm_f64.cuh"
#include "tm_kernels.cuh"
#include "../../include/tm.h"

#include <cuda_runtime.h>

#include <stdint.h>
#include <vector>

namespace {

__device__ __forceinline__ int pmod(int p, int L)
{
    const int r = p % L;
    return r < 0 ? r + L : r;
}

// round(t), halves away from 0, as an int.  FP64: from the bits (its round() is several
// FP64 instructions); values beyond an int take the library's.
__device__ __forceinline__ int round_int(float t) { return (int)round(t); }
__device__ __forceinline__ int round_int(double t)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(t);
    const int e = (int)((u >> 52) & 0x7ff) - 1023;
    if (e < -1) return 0;
    if (e > 29) return (int)round(t);
    const unsigned long long m = (u & tmf::kFrac) | tmf::kOne;
    const int v = (int)((m + (1ULL << (51 - e))) >> (52 - e));
    return (long long)u < 0 ? -v : v;
}

__device__ __forceinline__ float prod(float a, float b) { return a * b; }
__device__ __forceinline__ double prod(double a, double b) { return tmf::mul(a, b); }

__device__ __forceinline__ bool is_zero(float a) { return a == 0.0f; }
__device__ __forceinline__ bool is_zero(double a) { return tmf::is_zero(a); }
__device__ __forceinline__ float to_float(int n, float) { return (float)n; }
__device__ __forceinline__ double to_float(int n, double) { return tmf::from_u31((uint32_t)n); }
// a < b; FP64: positive values compare by their bits
__device__ __forceinline__ bool below(float a, float b) { return a < b; }
__device__ __forceinline__ bool below(double a, double b)
{
    const long long ua = __double_as_longlong(a), ub = __double_as_longlong(b);
    if (ua >= 0 && ub >= 0 && ub <= 0x7ff0000000000000LL) return ua < ub;
    return tmf::hw_less(a, b);
}

// Per source: its mass (0 below eps) and the row and column its shifted centre falls on,
// 16 bits each (L <= 46340; kNowhere for a source without mass), and the largest shift.
constexpr uint32_t kNowhere = 0xffffffffu;

// How far t lies from c.  From L on the sources of a whole axis are looked at, so L stands
// for more: an infinite velocity rounds to the largest int, and windows of that many
// sites overflow.
__device__ __forceinline__ int reach(int t, int c, int L)
{
    const long long d = (long long)t - c;
    return (int)min(d < 0 ? -d : d, (long long)L);
}

template <typename T>
__global__ void fke_prep_kernel(const T* rho, const T* vx, const T* vy, int L, T pref, T eps, T* w, uint32_t* to, int* smax)
{
    const int n = L * L;
    int local = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int ci = i / L, cj = i - ci * L;
        const T rv = rho[i];
        const bool dead = below(rv, eps) || is_zero(rv);
        w[i] = dead ? T(0) : rv;
        const int tx = round_int(to_float(ci, T(0)) + prod(vx[i], pref));
        const int ty = round_int(to_float(cj, T(0)) + prod(vy[i], pref));
        to[i] = dead ? kNowhere : ((uint32_t)pmod(tx, L) << 16) | (uint32_t)pmod(ty, L);
        if (!dead) local = max(local, max(reach(tx, ci, L), reach(ty, cj, L)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local = max(local, __shfl_xor_sync(0xffffffffu, local, o));
    if ((threadIdx.x & 31) == 0) atomicMax(smax, local);
}

// A source's weights from its mass and gamma.
template <typename T>
__device__ __forceinline__ T weight_dd(T w, T g) { return w == T(0) ? T(0) : prod(prod(g, g), w); }
template <typename T>
__device__ __forceinline__ T weight_dv(T w, T g) { return prod(g - prod(g, g), w); }
template <typename T>
__device__ __forceinline__ T weight_vv(T w, T g)
{
    const T h = T(1) - g;
    return prod(prod(h, h), w);
}

// offsets o of a window [-R, R] taken mod L: each residue once (all of them when 2R+1 >= L)
__device__ __forceinline__ void window(int R, int L, int& lo, int& hi)
{
    if (2 * R + 1 >= L) { lo = 0; hi = L - 1; }
    else { lo = -R; hi = R; }
}

// Stencils passed by value.
constexpr int kMaxRadius = TM_FKE_WS_MAX_RADIUS;
struct FkeStencils {
    double gD[kMaxRadius + 1];
    double gV[kMaxRadius + 1];
    int RD, RV;
};

// Passes 1 and 2 for stencils of any width (those wider than kMaxRadius or than the
// lattice, which only the allocating entry point takes): one (row, column) per thread.
template <typename T>
__global__ void fke_rows_wide_kernel(const T* w, const T* gam, const uint32_t* to, const int* smax, int L, const T* gDw,
                                     const T* gVw, int RD, int RV, T* AD, T* AV)
{
    const int n = L * L;
    const int S = *smax;
    int wlo, whi, slo, shi;
    window(max(RD, RV + S), L, wlo, whi);
    window(S, L, slo, shi);
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int r = t / L, q = t - r * L;
        T ad = T(0), av = T(0);
        for (int o = wlo; o <= whi; ++o) {
            const int cj = pmod(q - o, L);
            const int j = r * L + cj;
            if (to[j] == kNowhere) continue;
            ad = fma(weight_dd(w[j], gam[j]), gDw[pmod(q - cj, L)], ad);
            ad = fma(weight_dv(w[j], gam[j]), gVw[pmod(q - (int)(to[j] & 0xffffu), L)], ad);
        }
        for (int so = slo; so <= shi; ++so) {
            const int ci = pmod(r - so, L);
            for (int o = wlo; o <= whi; ++o) {
                const int cj = pmod(q - o, L);
                const int j = ci * L + cj;
                if ((to[j] >> 16) != (uint32_t)r) continue;
                av = fma(weight_dv(w[j], gam[j]), gDw[pmod(q - cj, L)], av);
                av = fma(weight_vv(w[j], gam[j]), gVw[pmod(q - (int)(to[j] & 0xffffu), L)], av);
            }
        }
        AD[t] = ad;
        AV[t] = av;
    }
}

template <typename T>
__global__ void fke_cols_wide_kernel(const T* AD, const T* AV, int L, const T* gDw, const T* gVw, int RD, int RV, T* out)
{
    const int n = L * L;
    int dlo, dhi, vlo, vhi;
    window(RD, L, dlo, dhi);
    window(RV, L, vlo, vhi);
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int p = t / L, q = t - p * L;
        T acc = T(0);
        for (int d = dlo; d <= dhi; ++d) acc = fma(gDw[pmod(d, L)], AD[pmod(p - d, L) * L + q], acc);
        for (int d = vlo; d <= vhi; ++d) acc = fma(gVw[pmod(d, L)], AV[pmod(p - d, L) * L + q], acc);
        out[t] = acc;
    }
}

// Pass 1: A_D and A_V of kCols columns of one row.
//
// The sources' weights are first gathered where they land -- F_DV at the shifted
// column, F_VD at the shifted row, F_VV at both -- so that each of the four stencils is
// a plain convolution along the row, 2 R + 1 fused multiply-adds, instead of a visit to
// every source that might reach the column.  The FP64 pipe bounds the pass (one warp
// instruction per 64-76 cycles whatever its lanes), so a cell lists its sources by their
// coordinates first (a bit each) and then adds them: the first needs no addition, and
// the warp executes as many additions as its fullest cell has sources.  Measured at
// 1024^2, RD = 5, RV = 2, S = 1: 47 FP64 instructions a site, 32 of them the stencils,
// 113 us (917 us when every column visited its (2 W + 1)(2 S + 2) sources).
constexpr int kCols = 256;
constexpr int kMaxListed = 3;              // largest shift whose (2 S + 1)^2 candidates fit 8 x 8 bits

template <typename T>
__device__ __forceinline__ void land(T& f, bool& any, T w)
{
    f = any ? f + w : w;
    any = true;
}

template <typename T>
__global__ void __launch_bounds__(kCols) fke_rows_kernel(const T* __restrict__ w, const T* __restrict__ gam,
                                                         const uint32_t* __restrict__ to, const int* __restrict__ smax, int L,
                                                         const __grid_constant__ FkeStencils st, T* AD, T* AV)
{
    const int RD = st.RD, RV = st.RV;
    extern __shared__ __align__(16) unsigned char fke_smem[];
    T* const fDD = reinterpret_cast<T*>(fke_smem);        // kCols + 2 RD
    T* const fVD = fDD + kCols + 2 * RD;
    T* const fDV = fVD + kCols + 2 * RD;                  // kCols + 2 RV
    T* const fVV = fDV + kCols + 2 * RV;
    T* const gD = fVV + kCols + 2 * RV;                   // 2 RD + 1, by offset
    T* const gV = gD + 2 * RD + 1;
    const int segs = (L + kCols - 1) / kCols;
    const int r = blockIdx.x / segs, q0 = (blockIdx.x - r * segs) * kCols;
    const int nc = min(kCols, L - q0);
    const int S = *smax;
    int slo, shi;
    window(S, L, slo, shi);
    const int ns = shi - slo + 1;
    const bool listed = S <= kMaxListed;
    for (int i = threadIdx.x; i <= 2 * RD; i += kCols) gD[i] = (T)st.gD[abs(i - RD)];
    for (int i = threadIdx.x; i <= 2 * RV; i += kCols) gV[i] = (T)st.gV[abs(i - RV)];
    for (int c = threadIdx.x; c < nc + 2 * RD; c += kCols) {
        int col = q0 - RD + c;
        col = col < 0 ? col + L : (col >= L ? col - L : col);
        fDD[c] = weight_dd(w[r * L + col], gam[r * L + col]);
        T f = T(0);
        bool any = false;
        auto add = [&](int j) { land(f, any, weight_dv(w[j], gam[j])); };
        if (listed) {
            unsigned m = 0;
            for (int s = 0; s < ns; ++s) m |= (unsigned)((to[pmod(r - slo - s, L) * L + col] >> 16) == (uint32_t)r) << s;
            for (; m; m &= m - 1) add(pmod(r - slo - (__ffs(m) - 1), L) * L + col);
        } else {
            for (int s = 0; s < ns; ++s) {
                const int j = pmod(r - slo - s, L) * L + col;
                if ((to[j] >> 16) == (uint32_t)r) add(j);
            }
        }
        fVD[c] = f;
    }
    for (int c = threadIdx.x; c < nc + 2 * RV; c += kCols) {
        int col = q0 - RV + c;
        col = col < 0 ? col + L : (col >= L ? col - L : col);
        const uint32_t here = ((uint32_t)r << 16) | (uint32_t)col;
        T f = T(0), h = T(0);
        bool any = false, anyh = false;
        auto add = [&](int j) { land(f, any, weight_dv(w[j], gam[j])); };
        auto addh = [&](int j) { land(h, anyh, weight_vv(w[j], gam[j])); };
        if (listed) {
            unsigned m = 0;
            unsigned long long m2 = 0;
            for (int s = 0; s < ns; ++s) {
                const int row = pmod(r - slo - s, L) * L;
                for (int o = 0; o < ns; ++o) {
                    int cj = col - slo - o;
                    cj = cj < 0 ? cj + L : (cj >= L ? cj - L : cj);
                    const uint32_t t = to[row + cj];
                    if (slo + s == 0) m |= (unsigned)((t & 0xffffu) == (uint32_t)col) << o;
                    m2 |= (unsigned long long)(t == here) << (8 * s + o);
                }
            }
            for (; m; m &= m - 1) add(r * L + pmod(col - slo - (__ffs(m) - 1), L));
            for (; m2; m2 &= m2 - 1) {
                const int b = __ffsll((long long)m2) - 1;
                addh(pmod(r - slo - (b >> 3), L) * L + pmod(col - slo - (b & 7), L));
            }
        } else {
            for (int o = 0; o < ns; ++o) {
                const int j = r * L + pmod(col - slo - o, L);
                if ((to[j] & 0xffffu) == (uint32_t)col) add(j);
            }
            for (int s = 0; s < ns; ++s)
                for (int o = 0; o < ns; ++o) {
                    const int j = pmod(r - slo - s, L) * L + pmod(col - slo - o, L);
                    if (to[j] == here) addh(j);
                }
        }
        fDV[c] = f;
        fVV[c] = h;
    }
    __syncthreads();
    const int q = threadIdx.x;
    if (q < nc) {
        T ad = T(0), av = T(0);
        for (int i = 0; i <= 2 * RD; ++i) {
            ad = fma(gD[i], fDD[q + 2 * RD - i], ad);
            av = fma(gD[i], fVD[q + 2 * RD - i], av);
        }
        for (int i = 0; i <= 2 * RV; ++i) {
            ad = fma(gV[i], fDV[q + 2 * RV - i], ad);
            av = fma(gV[i], fVV[q + 2 * RV - i], av);
        }
        AD[r * L + q0 + q] = ad;
        AV[r * L + q0 + q] = av;
    }
}

// Pass 2: out[p][q] = sum_d gD(d) A_D[p - d][q] + gV(d) A_V[p - d][q], two rows a thread.
template <typename T>
__global__ void __launch_bounds__(kCols) fke_cols_kernel(const T* __restrict__ AD, const T* __restrict__ AV, int L,
                                                         const __grid_constant__ FkeStencils st, T* out)
{
    const int RD = st.RD, RV = st.RV;
    __shared__ T gD[2 * kMaxRadius + 1], gV[2 * kMaxRadius + 1];
    for (int i = threadIdx.x; i <= 2 * RD; i += kCols) gD[i] = (T)st.gD[abs(i - RD)];
    for (int i = threadIdx.x; i <= 2 * RV; i += kCols) gV[i] = (T)st.gV[abs(i - RV)];
    __syncthreads();
    const int segs = (L + kCols - 1) / kCols;
    const int p0 = (int)(blockIdx.x / segs) * 2, q = (int)(blockIdx.x % segs) * kCols + threadIdx.x;
    if (q >= L) return;
    T a0 = T(0), a1 = T(0);
    // rows p0 - R .. p0 + 1 + R: row y adds offset d = p0 - y to the first sum, d + 1 to the second
    auto sum = [&](const T* __restrict__ A, const T* g, int R) {
        int y = p0 - R;
        if (y < 0) y += L;
        for (int i = 2 * R; i >= -1; --i) {              // offset index of the first sum
            const T v = A[y * L + q];
            if (i >= 0) a0 = fma(g[i], v, a0);
            if (i < 2 * R) a1 = fma(g[i + 1], v, a1);
            y = y + 1 == L ? 0 : y + 1;
        }
    };
    sum(AD, gD, RD);
    sum(AV, gV, RV);
    out[p0 * L + q] = a0;
    if (p0 + 1 < L) out[(p0 + 1) * L + q] = a1;
}

// Workspace of one call (each region 256-byte aligned): w, A_D, A_V (T, L^2 each), the
// landing sites (4 bytes, L^2), a region of the same size that is not used -- callers
// allocate by the size tm_fke_workspace_bytes has always given -- the wrapped stencils gDw,
// gVw (T, L each), smax (int).
struct FkeLayout {
    size_t w, AD, AV, to, spare, gD, gV, smax, end;
};
inline size_t al256(size_t v) { return (v + 255) / 256 * 256; }
inline FkeLayout fke_layout(size_t esize, int L)
{
    const size_t n = (size_t)L * L;
    FkeLayout y;
    y.w = 0;
    y.AD = al256(y.w + n * esize);
    y.AV = al256(y.AD + n * esize);
    y.to = al256(y.AV + n * esize);
    y.spare = al256(y.to + n * sizeof(uint32_t));
    y.gD = al256(y.spare + n * sizeof(uint32_t));
    y.gV = al256(y.gD + (size_t)L * esize);
    y.smax = al256(y.gV + (size_t)L * esize);
    y.end = y.smax + 256;
    return y;
}

// The stencils wrapped onto the lattice: residue i gets every g[|d|] with
// d = i (mod L), |d| <= R, added in increasing d in FP64 and rounded once --
// the same sums the host forms for the allocating entry point.
template <typename T>
__global__ void fke_wrap_kernel(const FkeStencils st, int L, T* gDw, T* gVw)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L; i += gridDim.x * blockDim.x) {
        double sd = 0.0, sv = 0.0;
        for (int d = -st.RD; d <= st.RD; ++d)
            if (pmod(d, L) == i) sd += st.gD[d < 0 ? -d : d];
        for (int d = -st.RV; d <= st.RV; ++d)
            if (pmod(d, L) == i) sv += st.gV[d < 0 ? -d : d];
        gDw[i] = (T)sd;
        gVw[i] = (T)sv;
    }
}

// Queues one movement on a workspace of fke_layout's size; `wrapped` queues what puts
// the wrapped stencils there, which only the wide passes read.  Nothing waits.
template <typename T, typename Wrapped>
cudaError_t enqueue_passes(const void* rho, const void* gam, const void* vx, const void* vy, int L, double pref,
                           double eps, const double* gD, int RD, const double* gV, int RV, void* out, unsigned char* ws,
                           cudaStream_t s, const Wrapped& wrapped)
{
    const FkeLayout y = fke_layout(sizeof(T), L);
    T* w = (T*)(ws + y.w);
    T* AD = (T*)(ws + y.AD);
    T* AV = (T*)(ws + y.AV);
    uint32_t* to = (uint32_t*)(ws + y.to);
    int* smax = (int*)(ws + y.smax);
    const size_t n = (size_t)L * L;
    cudaError_t e = cudaMemsetAsync(smax, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
    const int grid = (int)((n + 255) / 256 < 8192 ? (n + 255) / 256 : 8192);
    fke_prep_kernel<T><<<grid, 256, 0, s>>>((const T*)rho, (const T*)vx, (const T*)vy, L, (T)pref, (T)eps, w, to, smax);
    if (RD <= kMaxRadius && RV <= kMaxRadius && 2 * (RD > RV ? RD : RV) + 1 <= L) {
        FkeStencils st;
        for (int d = 0; d <= kMaxRadius; ++d) {
            st.gD[d] = d <= RD ? gD[d] : 0.0;
            st.gV[d] = d <= RV ? gV[d] : 0.0;
        }
        st.RD = RD;
        st.RV = RV;
        const int segs = (L + kCols - 1) / kCols;
        const size_t smem = (4 * (size_t)kCols + 6 * (size_t)RD + 6 * (size_t)RV + 2) * sizeof(T);
        fke_rows_kernel<T><<<L * segs, kCols, smem, s>>>(w, (const T*)gam, to, smax, L, st, AD, AV);
        fke_cols_kernel<T><<<(L + 1) / 2 * segs, kCols, 0, s>>>(AD, AV, L, st, (T*)out);
    } else {
        e = wrapped((T*)(ws + y.gD), (T*)(ws + y.gV));
        if (e != cudaSuccess) return e;
        const T* dgD = (const T*)(ws + y.gD);
        const T* dgV = (const T*)(ws + y.gV);
        fke_rows_wide_kernel<T><<<grid, 256, 0, s>>>(w, (const T*)gam, to, smax, L, dgD, dgV, RD, RV, AD, AV);
        fke_cols_wide_kernel<T><<<grid, 256, 0, s>>>(AD, AV, L, dgD, dgV, RD, RV, (T*)out);
    }
    return cudaGetLastError();
}

template <typename T>
int run(const void* rho, const void* gam, const void* vx, const void* vy, int L, double pref, double eps,
        const double* gD, int RD, const double* gV, int RV, void* out, cudaStream_t s)
{
    std::vector<T> hd, hv;
    // the stencils wrapped onto the lattice: every image d = delta (mod L) of |d| <= R summed
    auto wrapped = [&](T* dD, T* dV) {
        std::vector<double> wd(L, 0.0), wv(L, 0.0);
        for (int d = -RD; d <= RD; ++d) wd[((d % L) + L) % L] += gD[d < 0 ? -d : d];
        for (int d = -RV; d <= RV; ++d) wv[((d % L) + L) % L] += gV[d < 0 ? -d : d];
        hd.assign(wd.begin(), wd.end());
        hv.assign(wv.begin(), wv.end());
        const cudaError_t e = cudaMemcpyAsync(dD, hd.data(), L * sizeof(T), cudaMemcpyHostToDevice, s);
        return e != cudaSuccess ? e : cudaMemcpyAsync(dV, hv.data(), L * sizeof(T), cudaMemcpyHostToDevice, s);
    };
    unsigned char* ws = nullptr;
    int rc = TM_OK;
    if (cudaMalloc(&ws, fke_layout(sizeof(T), L).end) != cudaSuccess) {
        rc = TM_ERR_NOMEM;
    } else if (enqueue_passes<T>(rho, gam, vx, vy, L, pref, eps, gD, RD, gV, RV, out, ws, s, wrapped) != cudaSuccess ||
               cudaStreamSynchronize(s) != cudaSuccess) {
        rc = TM_ERR_CUDA;
    }
    cudaFree(ws);
    (void)cudaGetLastError();
    return rc;
}

template <typename T>
int run_ws(const void* rho, const void* gam, const void* vx, const void* vy, int L, double pref, double eps,
           const double* gD, int RD, const double* gV, int RV, void* out, void* ws, cudaStream_t s)
{
    auto wrapped = [&](T* dD, T* dV) {
        FkeStencils st;
        for (int d = 0; d <= kMaxRadius; ++d) {
            st.gD[d] = d <= RD ? gD[d] : 0.0;
            st.gV[d] = d <= RV ? gV[d] : 0.0;
        }
        st.RD = RD;
        st.RV = RV;
        fke_wrap_kernel<T><<<(L + 255) / 256, 256, 0, s>>>(st, L, dD, dV);
        return cudaGetLastError();
    };
    if (enqueue_passes<T>(rho, gam, vx, vy, L, pref, eps, gD, RD, gV, RV, out, (unsigned char*)ws, s, wrapped) !=
        cudaSuccess) {
        (void)cudaGetLastError();
        return TM_ERR_CUDA;
    }
    return TM_OK;
}

}  // namespace

extern "C" size_t tm_fke_workspace_bytes(int precision, int L)
{
    if ((precision != TM_FP64 && precision != TM_FP32) || L < 1 || L > 46340) return 0;
    return fke_layout(precision == TM_FP64 ? 8 : 4, L).end;
}

extern "C" int tm_fke_advdiff_device_ws(const void* dev_rho, const void* dev_gamma, const void* dev_vx,
                                        const void* dev_vy, int precision, int L, double pref, double eps,
                                        const double* gD, int RD, const double* gV, int RV, void* dev_out,
                                        void* dev_workspace, size_t workspace_bytes, void* stream)
{
    if (!dev_rho || !dev_gamma || !dev_vx || !dev_vy || !dev_out || !dev_workspace || !gD || !gV || L < 1 ||
        L > 46340 || RD < 0 || RV < 0 || RD > TM_FKE_WS_MAX_RADIUS || RV > TM_FKE_WS_MAX_RADIUS ||
        ((uintptr_t)dev_workspace & 255u) != 0)
        return TM_ERR_INVALID;
    const size_t need = tm_fke_workspace_bytes(precision, L);
    if (need == 0 || workspace_bytes < need) return TM_ERR_INVALID;
    if (precision == TM_FP64)
        return run_ws<double>(dev_rho, dev_gamma, dev_vx, dev_vy, L, pref, eps, gD, RD, gV, RV, dev_out, dev_workspace,
                              (cudaStream_t)stream);
    return run_ws<float>(dev_rho, dev_gamma, dev_vx, dev_vy, L, pref, eps, gD, RD, gV, RV, dev_out, dev_workspace,
                         (cudaStream_t)stream);
}

extern "C" int tm_fke_advdiff_device(const void* dev_rho, const void* dev_gamma, const void* dev_vx,
                                     const void* dev_vy, int precision, int L, double pref, double eps,
                                     const double* gD, int RD, const double* gV, int RV, void* dev_out, void* stream)
{
    if (!dev_rho || !dev_gamma || !dev_vx || !dev_vy || !dev_out || !gD || !gV || L < 1 || L > 46340 || RD < 0 ||
        RV < 0 || RD > (1 << 20) || RV > (1 << 20))
        return TM_ERR_INVALID;
    if (precision == TM_FP64)
        return run<double>(dev_rho, dev_gamma, dev_vx, dev_vy, L, pref, eps, gD, RD, gV, RV, dev_out,
                           (cudaStream_t)stream);
    if (precision == TM_FP32)
        return run<float>(dev_rho, dev_gamma, dev_vx, dev_vy, L, pref, eps, gD, RD, gV, RV, dev_out,
                          (cudaStream_t)stream);
    return TM_ERR_INVALID;
}
