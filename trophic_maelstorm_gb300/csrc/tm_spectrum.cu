// tm_spectrum.cu -- radially averaged power spectrum of a lattice on the GPU.
//
// Semantics of gen_FFT_PowerSpectra (simulations/Utilities/glow_up.py:752-827),
// the reference's pattern-wavelength estimator: the field is divided by its
// maximum (unless that is 0), transformed by a 2-D FFT in double precision,
// |F(k)|^2 is averaged over annuli k in [e_b, e_{b+1}) with e_b = 1 - w/2 + b w
// (the last bin closed, as numpy.histogram), and each bin mean is multiplied by
// the annulus area pi (e_{b+1}^2 - e_b^2).  Empty bins are 0 (the reference
// turns them into NaN afterwards).  The wavelength is L / k at the peak.
//
// The FFT is cuFFT's D2Z (half spectrum); columns with a mirror image count
// twice.  k^2 is a whole number, so each annulus is a range of whole numbers
// [T_b, T_b+1) found once on the host, and a block sums one annulus straight from the
// spectrum: a row's columns in it are one interval.  (Listing every element of every
// annulus on the host took most of a call's time.)  Rows go to threads in order and
// their sums combine in a fixed tree: the result does not depend on scheduling.
// Plans and buffers live in a SpectrumWork, which a batch keeps for its next call.
#include "tm_f64.cuh"
#include "tm_kernels.cuh"
#include "../../include/tm.h"

#include <cuda_runtime.h>
#include <cufft.h>
#include <cmath>
#include <new>
#include <vector>

namespace {

__device__ __forceinline__ double wsum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <typename T>
__global__ void max_partial_kernel(const T* f, long long n, double* part)
{
    __shared__ double red[32];
    double m = -INFINITY;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        m = fmax(m, (double)f[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : -INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) part[blockIdx.x] = m;
    }
}

__global__ void max_final_kernel(double* part, int n)
{
    double m = -INFINITY;
    for (int i = threadIdx.x; i < n; i += 32) m = fmax(m, part[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) part[0] = (m != 0.0) ? m : 1.0;
}

template <typename T>
__global__ void normalise_kernel(const T* f, long long n, const double* mx, double* out)
{
    const double m = *mx;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = tmf::div((double)f[i], m);
}

// largest x >= 0 with x x <= n, for 0 <= n < 2^33
__device__ __forceinline__ int isqrt(long long n)
{
    int r = (int)sqrtf((float)n);
    while ((long long)r * r > n) --r;
    while ((long long)(r + 1) * (r + 1) <= n) ++r;
    return r;
}

constexpr int kBinThreads = 128;

// one block per annulus: mean of |F|^2 over the modes with lim[b] <= k^2 < lim[b + 1],
// times its area
__global__ void __launch_bounds__(kBinThreads) bin_kernel(const cufftDoubleComplex* F, int L, const long long* lim,
                                                          const double* area, double* power)
{
    __shared__ double red[kBinThreads / 32];
    __shared__ unsigned long long cred[kBinThreads / 32];
    const int b = blockIdx.x, nx = L / 2 + 1;
    const long long lo = lim[b], hi = lim[b + 1] - 1;         // k^2 in [lo, hi]
    const int fmax = (L - 1) / 2, fmin = -(L / 2);              // row frequencies
    const int R = hi < 0 ? -1 : isqrt(hi);
    double s = 0.0;
    unsigned long long c = 0;
    for (int fy = max(fmin, -R) + (int)threadIdx.x; fy <= min(fmax, R); fy += kBinThreads) {
        const long long f2 = (long long)fy * fy;
        const int x1 = min(nx - 1, isqrt(hi - f2));
        const int x0 = lo - f2 <= 0 ? 0 : isqrt(lo - f2 - 1) + 1;
        const cufftDoubleComplex* row = F + (long long)(fy < 0 ? fy + L : fy) * nx;
        for (int x = x0; x <= x1; ++x) {
            const cufftDoubleComplex z = row[x];
            const double p = fma(z.x, z.x, z.y * z.y);
            const bool twice = x >= 1 && x <= (L - 1) / 2;     // the mirror column's mode
            s = twice ? fma(2.0, p, s) : s + p;
            c += twice ? 2 : 1;
        }
    }
    s = wsum(s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = s;
        cred[threadIdx.x >> 5] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kBinThreads / 32; ++w) {
            s += red[w];
            c += cred[w];
        }
        power[b] = c ? (s / (double)c) * area[b] : 0.0;
    }
}

// Annuli of a lattice: centres, areas, and the limits of k^2: lim[b] is the least whole
// n with sqrt(n) >= e_b, the last one the least with sqrt(n) > e_nbins (that bin is closed).
struct Annuli {
    int nbins = 0;
    std::vector<double> kvals, area;
    std::vector<long long> lim;
};

// Their number without listing them; more than an int holds counts as the largest int.
int count_annuli(int L, double bw)
{
    const double start = 1.0 - bw / 2.0, stop = (double)(L / 2 + 1);
    const double n = std::ceil((stop - start) / bw) - 1.0;    // numpy.arange's length, less one
    return n >= 1.0 ? (n < 2147483647.0 ? (int)n : 2147483647) : 0;
}

void make_annuli(int L, double bw, Annuli& p)
{
    // edges: numpy.arange(1 - bw/2, L//2 + 1, bw)
    p.nbins = count_annuli(L, bw);
    std::vector<double> e(p.nbins ? (size_t)p.nbins + 1 : 0);
    const double start = 1.0 - bw / 2.0;
    for (size_t i = 0; i < e.size(); ++i) e[i] = start + (double)i * bw;
    p.kvals.resize(p.nbins);
    p.area.resize(p.nbins);
    for (int b = 0; b < p.nbins; ++b) {
        p.kvals[b] = 0.5 * (e[b + 1] + e[b]);
        p.area[b] = M_PI * (e[b + 1] * e[b + 1] - e[b] * e[b]);
    }
    p.lim.clear();
    for (size_t i = 0; i < e.size() && p.nbins; ++i) {
        if (e[i] <= 0.0) { p.lim.push_back(0); continue; }
        const bool last = i + 1 == e.size();
        auto below = [&](long long n) { return last ? std::sqrt((double)n) <= e[i] : std::sqrt((double)n) < e[i]; };
        long long n = (long long)(e[i] * e[i]);
        while (n > 0 && !below(n - 1)) --n;
        while (below(n)) ++n;
        p.lim.push_back(n);
    }
}

#define SPEC_CUDA(call)                                        \
    do {                                                       \
        if ((call) != cudaSuccess) {                           \
            (void)cudaGetLastError();                          \
            return TM_ERR_CUDA;                                \
        }                                                      \
    } while (0)

}  // namespace

// Device buffers and FFT plan for one lattice side and bin width.
struct SpectrumWork {
    int L = 0;
    double bw = 0.0;
    Annuli ann;
    bool have_plan = false;
    cufftHandle plan = 0;
    double *img = nullptr, *part = nullptr, *area = nullptr, *power = nullptr;
    long long* lim = nullptr;
    cufftDoubleComplex* F = nullptr;
    static constexpr int kBlocks = 304;

    ~SpectrumWork()
    {
        if (have_plan) cufftDestroy(plan);
        for (void* q : {(void*)img, (void*)part, (void*)area, (void*)power, (void*)lim, (void*)F}) cudaFree(q);
        (void)cudaGetLastError();
    }

    // Plan and buffers.
    int prepare(cudaStream_t s)
    {
        const size_t n = (size_t)L * L;
        SPEC_CUDA(cudaMalloc(&img, n * sizeof(double)));
        SPEC_CUDA(cudaMalloc(&F, (size_t)L * (L / 2 + 1) * sizeof(cufftDoubleComplex)));
        SPEC_CUDA(cudaMalloc(&part, kBlocks * sizeof(double)));
        SPEC_CUDA(cudaMalloc(&area, ann.nbins * sizeof(double)));
        SPEC_CUDA(cudaMalloc(&power, ann.nbins * sizeof(double)));
        SPEC_CUDA(cudaMalloc(&lim, ann.lim.size() * sizeof(long long)));
        SPEC_CUDA(cudaMemcpyAsync(area, ann.area.data(), ann.nbins * sizeof(double), cudaMemcpyHostToDevice, s));
        SPEC_CUDA(cudaMemcpyAsync(lim, ann.lim.data(), ann.lim.size() * sizeof(long long), cudaMemcpyHostToDevice, s));
        if (cufftPlan2d(&plan, L, L, CUFFT_D2Z) != CUFFT_SUCCESS) return TM_ERR_CUDA;
        have_plan = true;
        return cufftSetStream(plan, s) == CUFFT_SUCCESS ? TM_OK : TM_ERR_CUDA;
    }

    template <typename T>
    int run(const T* field, cudaStream_t s, double* kvals, double* out)
    {
        const long long n = (long long)L * L;
        max_partial_kernel<T><<<kBlocks, 256, 0, s>>>(field, n, part);
        max_final_kernel<<<1, 32, 0, s>>>(part, kBlocks);
        normalise_kernel<T><<<kBlocks, 256, 0, s>>>(field, n, part, img);
        SPEC_CUDA(cudaGetLastError());
        if (cufftExecD2Z(plan, img, F) != CUFFT_SUCCESS) return TM_ERR_CUDA;
        bin_kernel<<<ann.nbins, kBinThreads, 0, s>>>(F, L, lim, area, power);
        SPEC_CUDA(cudaGetLastError());
        SPEC_CUDA(cudaMemcpyAsync(out, power, ann.nbins * sizeof(double), cudaMemcpyDeviceToHost, s));
        SPEC_CUDA(cudaStreamSynchronize(s));
        for (int b = 0; b < ann.nbins; ++b) kvals[b] = ann.kvals[b];
        return TM_OK;
    }
};

void spectrum_work_destroy(SpectrumWork* w) { delete w; }

// Spectrum of a device field; *keep (may be null) is a SpectrumWork of an earlier call, used
// when side and bin width are the same and replaced otherwise.  One host thread and one
// stream at a time, as its owner's.
int power_spectrum(const void* dev_field, int precision, int L, double binwidth, cudaStream_t s, double* kvals,
                   double* power, int max_bins, int* n_bins, SpectrumWork** keep)
{
    if (!dev_field || L < 2 || !(binwidth > 0) || !kvals || !power || !n_bins || max_bins < 0) return TM_ERR_INVALID;
    if (precision != TM_FP64 && precision != TM_FP32) return TM_ERR_INVALID;
    SpectrumWork* w = keep ? *keep : nullptr;
    if (!w || w->L != L || w->bw != binwidth) {
        *n_bins = count_annuli(L, binwidth);
        if (*n_bins > max_bins) return TM_ERR_INVALID;
        if (*n_bins == 0) return TM_OK;
        SpectrumWork* fresh = new (std::nothrow) SpectrumWork;
        if (!fresh) return TM_ERR_NOMEM;
        fresh->L = L;
        fresh->bw = binwidth;
        try {
            make_annuli(L, binwidth, fresh->ann);
        } catch (const std::bad_alloc&) {
            delete fresh;
            return TM_ERR_NOMEM;
        }
        if (keep) {
            delete w;                       // first, so that both never hold memory together
            *keep = nullptr;
        }
        const int rc = fresh->prepare(s);
        if (rc != TM_OK) {
            delete fresh;
            return rc;
        }
        w = fresh;
        if (keep) *keep = w;
    }
    *n_bins = w->ann.nbins;
    int rc = TM_ERR_INVALID;
    if (w->ann.nbins <= max_bins)
        rc = precision == TM_FP64 ? w->run((const double*)dev_field, s, kvals, power)
                                  : w->run((const float*)dev_field, s, kvals, power);
    if (!keep) delete w;
    return rc;
}

extern "C" int tm_power_spectrum_device(const void* dev_field, int precision, int L, double binwidth, void* stream,
                                        double* kvals, double* power, int max_bins, int* n_bins)
{
    return power_spectrum(dev_field, precision, L, binwidth, (cudaStream_t)stream, kvals, power, max_bins, n_bins, nullptr);
}
