// tm_measure.cu -- observables in FP64 with a fixed reduction order.
//
// mean_of_vector / occupied_sites_of_vector (stochasticSPDP.cpp:123-154) for
// every instance of a batch: one warp per task sums its strip (lanes own
// columns, rows in order), a butterfly of shuffles combines the lanes, and
// the warp that finishes an instance last sums its per-task partials -- in one
// order whoever that is, so a given state always gives the same bits.  Up to
// 512 tasks are summed at once; above, groups of 256 or more, about as many as each
// holds, are summed by the warps that finish them last and the groups' sums by the
// last of those.
//
// A measurement is short beside its launches and round trips.  With a second kernel of
// one warp per instance for the sums, 64 spreading FP64 lattices of 101 x 101 took 18.7 us
// to measure, 12.8 us with the sums in the same launch (and no additions for rows of
// zeros), 8.6 us with one-field code of its own (64 registers instead of 102); on a 4096 x
// 4096 FP32 Rietkerk lattice that one warp walked 65,536 partials, 613 us of a run of 24
// steps and one measurement that went from 12.31 to 11.75 ms.
//
// GB300's FP64 rate is a small fraction of its FP32 rate, so the per-site work
// avoids FP64: active sites are counted with ballots, and an FP32 lane keeps
// the sum of its column's values (at most 16) as an unevaluated pair hi + lo
// by Knuth's TwoSum, which is exact up to the rounding of lo (relative 2^-48).
// The lanes' pairs are combined the same way through the shuffle butterfly
// (the values are non-negative, so nothing cancels), and lane 0 converts the
// task's pair to FP64.
#include "tm_device.cuh"
#include "tm_kernels.cuh"

namespace tmg {

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// hi + lo += v with hi the rounded sum and its error carried in lo (TwoSum; the
// kernels are built without contraction of multiply-adds, so every step rounds)
__device__ __forceinline__ void two_sum_add(float& hi, float& lo, float v)
{
    const float s = hi + v;
    const float bp = s - hi;
    const float e = (hi - (s - bp)) + (v - bp);
    hi = s;
    lo = lo + e;
}

template <typename T>
struct ColSum {
    T s = T(0);
    __device__ __forceinline__ void add(T v) { s += v; }
    __device__ __forceinline__ double warp_total() const { return warp_sum((double)s); }
};
template <>
struct ColSum<float> {
    float hi = 0.0f, lo = 0.0f;
    __device__ __forceinline__ void add(float v) { two_sum_add(hi, lo, v); }
    // sum over the warp, valid in lane 0
    __device__ __forceinline__ double warp_total() const
    {
        float h = hi, l = lo;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ho = __shfl_down_sync(0xffffffffu, h, o);
            const float lo2 = __shfl_down_sync(0xffffffffu, l, o);
            two_sum_add(h, l, ho);
            l = l + lo2;
        }
        return (double)h + (double)l;
    }
};

// x > 0; FP64 by the bits (a comparison costs as much as an addition there)
__device__ __forceinline__ bool positive(float x) { return x > 0.0f; }
__device__ __forceinline__ bool positive(double x)
{
    const long long u = __double_as_longlong(x);
    return u > 0 && u <= 0x7ff0000000000000LL;
}

__device__ __forceinline__ bool nonzero(float) { return true; }
__device__ __forceinline__ bool nonzero(double x) { return (__double_as_longlong(x) << 1) != 0; }

constexpr int kChunk = 8;   // rows whose loads a warp issues together

// Sums of n rows of four by one warp, valid in every lane; the rows were written by
// other SMs within this launch.  Active sites are whole numbers below 2^53, so they add
// as integers; sums that a measurement does not have are not formed.
struct Sum4 {
    double s0, s1, s2;
    long long active;
};
__device__ __forceinline__ Sum4 sum_rows(const double* rows, int n, bool has1, bool has2)
{
    const double2* const p = reinterpret_cast<const double2*>(rows);
    Sum4 r = {0.0, 0.0, 0.0, 0};
#pragma unroll 4
    for (int t = (int)(threadIdx.x & 31); t < n; t += 32) {
        const double2 a = __ldcg(p + 2LL * t), b = __ldcg(p + 2LL * t + 1);
        r.s0 += a.x;
        if (has1) r.s1 += a.y;
        if (has2) r.s2 += b.x;
        r.active += (long long)b.y;
    }
    r.s0 = warp_sum(r.s0);
    if (has1) r.s1 = warp_sum(r.s1);
    if (has2) r.s2 = warp_sum(r.s2);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r.active += __shfl_xor_sync(0xffffffffu, r.active, o);
    return r;
}

// `count` more rows of a sum of `total` are written (by lane 0); true in the warp that
// wrote the last of them, for which all are then readable.  The counter is left at 0.
__device__ __forceinline__ bool arrive(int* counter, int count, int total)
{
    int last = 0;
    if ((threadIdx.x & 31) == 0) {
        __threadfence();
        last = atomicAdd(counter, count) + count == total;
        if (last) {
            *counter = 0;
            __threadfence();
        }
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    __syncwarp();
    return last != 0;
}

// obs_row[k*W + f], W = 2 (DP: mean, active), 3 (DP spreading: mean, active, summed
// squared distance) or 4 (Rietkerk: mean P, W, O, active P).  With dp_extinction, an
// instance seen with no active site is marked extinct (stochasticSPDP.cpp:1021-1022):
// by its last warp, when all its tasks have read the mark.
template <typename T>
__device__ __forceinline__ void observe(const MeasureArgs<T>& A, int k, const Sum4& r)
{
    const double ac = (double)r.active;
    const bool dead = A.it.alive != nullptr && A.it.alive[k] == 0;
    const double n = (double)A.it.L[k] * (double)A.it.L[k];
    if (A.nf == 1 && A.spread) {
        A.obs_row[3LL * k + 0] = dead ? 0.0 : r.s0 / n;
        A.obs_row[3LL * k + 1] = dead ? 0.0 : ac;
        A.obs_row[3LL * k + 2] = dead ? 0.0 : r.s1;
    } else if (A.nf == 1) {
        A.obs_row[2LL * k + 0] = dead ? 0.0 : r.s0 / n;
        A.obs_row[2LL * k + 1] = dead ? 0.0 : ac;
    } else {
        A.obs_row[4LL * k + 0] = r.s0 / n;
        A.obs_row[4LL * k + 1] = r.s1 / n;
        A.obs_row[4LL * k + 2] = r.s2 / n;
        A.obs_row[4LL * k + 3] = ac;
    }
    if (A.dp_extinction && A.it.alive != nullptr && ac == 0.0) A.it.alive[k] = 0;
}

// A warp takes a run of consecutive tasks, so that it reports a stretch of rows at a time.
// NF fields: one field's code needs half the registers of three.
template <typename T, int NF>
__global__ void __launch_bounds__(256) measure_kernel(const MeasureArgs<T> A)
{
    const int lane = threadIdx.x & 31;
    const long long gw = (long long)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int nw = (int)((gridDim.x * blockDim.x) >> 5);
    pdl_wait();
    const int spread = A.spread;
    const bool has1 = NF == 3 || spread, has2 = NF == 3;
    const long long run = ((long long)A.n_tasks + nw - 1) / nw;
    const int end = (int)min((long long)A.n_tasks, (gw + 1) * run);
    int written = 0;                       // rows not reported yet
    for (int t = (int)min((long long)A.n_tasks, gw * run); t < end; ++t) {
        const int4 tk = A.tasks[t];
        const int k = tk.x;
        const int L = A.it.L[k];
        const int b0 = A.begin[k], b1 = A.begin[k + 1];
        const int x = tk.y + lane;
        ColSum<T> c0, c1, c2;
        int ac = 0;
        long long sq = 0;
        bool any = false;                  // a value that changes the sum
        const bool on = A.it.alive == nullptr || A.it.alive[k] != 0;   // warp-uniform
        if (on) {
            const T* base = A.state + A.it.off[k];
            const long long fs = A.it.fstride[k];
            const bool in = x < L;
            const long long cx = A.scx < 0 ? L / 2 : A.scx, cy = A.scy < 0 ? L / 2 : A.scy;
            // rows in chunks of kChunk: every load of a chunk is issued before the
            // sums use them (the state streams from HBM once; the sums keep row order)
            for (int r0 = 0; r0 < tk.w; r0 += kChunk) {
                T v0[kChunk], v1[kChunk], v2[kChunk];
#pragma unroll
                for (int j = 0; j < kChunk; ++j) {
                    const bool ok = in && r0 + j < tk.w;
                    const long long i = (long long)(tk.z + r0 + j) * L + x;
                    v0[j] = ok ? base[i] : T(0);
                    v1[j] = (NF == 3 && ok) ? base[i + fs] : T(0);
                    v2[j] = (NF == 3 && ok) ? base[i + 2 * fs] : T(0);
                }
#pragma unroll
                for (int j = 0; j < kChunk; ++j) {
                    if (r0 + j >= tk.w) break;
                    if (NF == 3) {
                        c0.add(v0[j]);
                        any = true;
                        if (in) {
                            c1.add(v1[j]);
                            c2.add(v2[j]);
                        }
                    } else if (__any_sync(0xffffffffu, nonzero(v0[j]))) {
                        c0.add(v0[j]);     // rows of zeros, most of a spreading run's, cost FP64 no addition
                        any = true;
                    }
                    ac += __popc(__ballot_sync(0xffffffffu, positive(v0[j])));
                    if (spread && positive(v0[j])) {
                        const long long dy = (long long)(tk.z + r0 + j) - cy, dx = (long long)x - cx;
                        sq += dy * dy + dx * dx;
                    }
                }
            }
        }
        const double s0 = any ? c0.warp_total() : 0.0;
        double s1 = 0.0, s2 = 0.0;
        if (NF == 3) { s1 = c1.warp_total(); s2 = c2.warp_total(); }
        if (spread && ac) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
            s1 = (double)sq;
        }
        if (lane == 0) {
            reinterpret_cast<double2*>(A.partial)[2LL * t] = make_double2(s0, s1);
            reinterpret_cast<double2*>(A.partial)[2LL * t + 1] = make_double2(s2, (double)ac);
        }
        ++written;
        const int nt = b1 - b0, at = t + 1 - b0;
        const bool grouped = nt > kMeasureOnce;
        const int sh = measure_group_shift(nt);
        if (t + 1 != end && at != nt && !(grouped && (at & ((1 << sh) - 1)) == 0)) continue;
        // the stretch ends: with the run, the instance or the group
        if (!grouped) {
            if (arrive(A.arrived + k, written, nt)) {
                const Sum4 r = sum_rows(A.partial + 4LL * b0, nt, has1, has2);
                if (lane == 0) observe(A, k, r);
            }
        } else {
            const int g = (at - 1) >> sh, n_g = ((nt - 1) >> sh) + 1;
            const int first = b0 + (g << sh), n = min(1 << sh, b1 - first);
            const int base = measure_group_base(b0, k);
            if (arrive(A.arrived + A.n_inst + base + g, written, n)) {
                const Sum4 r = sum_rows(A.partial + 4LL * first, n, has1, has2);
                if (lane == 0) {
                    double2* const q = reinterpret_cast<double2*>(A.group_sums) + 2LL * (base + g);
                    q[0] = make_double2(r.s0, r.s1);
                    q[1] = make_double2(r.s2, (double)r.active);
                }
                if (arrive(A.arrived + k, 1, n_g)) {
                    const Sum4 a = sum_rows(A.group_sums + 4LL * base, n_g, has1, has2);
                    if (lane == 0) observe(A, k, a);
                }
            }
        }
        written = 0;
    }
}

template <typename T>
cudaError_t launch_measure(const MeasureArgs<T>& a, int grid, int block, cudaStream_t s)
{
    if (a.n_tasks <= 0) return cudaSuccess;
    if (a.nf == 3) return launch_pdl(measure_kernel<T, 3>, dim3(grid), dim3(block), 0, s, a);
    return launch_pdl(measure_kernel<T, 1>, dim3(grid), dim3(block), 0, s, a);
}
template cudaError_t launch_measure<float>(const MeasureArgs<float>&, int, int, cudaStream_t);
template cudaError_t launch_measure<double>(const MeasureArgs<double>&, int, int, cudaStream_t);

// Spreading runs stop once activity reaches the lattice's edge (theborderwall,
// stochasticSPDP.cpp:380-390, checked before every step at :1206-1213): one warp
// per live instance scans its four border rows/columns and marks it stopped
// (alive = 0, so later steps skip it and its later measurements are 0).
template <typename T>
__global__ void border_stop_kernel(const T* state, const InstTables it, int n_inst)
{
    const int lane = threadIdx.x & 31;
    const int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    pdl_wait();
    if (k >= n_inst || it.alive[k] == 0) return;
    const int L = it.L[k];
    const T* base = state + it.off[k];
    bool hit = false;
    // all loads of an unrolled trip in flight together
#pragma unroll 4
    for (int i = lane; i < L; i += 32) {
        const T a = base[i], b = base[(long long)i * L], c = base[(long long)(L - 1) * L + i], d = base[(long long)i * L + L - 1];
        hit = hit | positive(a) | positive(b) | positive(c) | positive(d);
    }
    if (__any_sync(0xffffffffu, hit) && lane == 0) it.alive[k] = 0;
}

template <typename T>
cudaError_t launch_border_stop(const T* state, const InstTables& it, int n_inst, cudaStream_t s)
{
    if (n_inst <= 0) return cudaSuccess;
    return launch_pdl(border_stop_kernel<T>, dim3((n_inst + 1) / 2), dim3(64), 0, s, state, it, n_inst);
}
template cudaError_t launch_border_stop<float>(const float*, const InstTables&, int, cudaStream_t);
template cudaError_t launch_border_stop<double>(const double*, const InstTables&, int, cudaStream_t);

// Status bits of an uploaded state, per instance: TM_STATUS_NAN_BIT for a NaN or
// Inf and TM_STATUS_NEG_BIT for a negative value in any field -- the checks the
// reference runs on every new state (multiSPDP.cpp:2949-2955, 3237-3255;
// rietkerk_bjork_FKE.cpp:4352-4370), applied to the state a caller uploads.
template <typename T>
__global__ void __launch_bounds__(256) validate_kernel(const T* state, const InstTables it, const int4* tasks,
                                                       int n_tasks, int nf)
{
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int nw = (int)((gridDim.x * blockDim.x) >> 5);
    for (int t = gw; t < n_tasks; t += nw) {
        const int4 tk = tasks[t];
        const int k = tk.x;
        const int L = it.L[k];
        const int x = tk.y + lane;
        unsigned st = 0;
        if (x < L) {
            const T* base = state + it.off[k];
            const long long fs = it.fstride[k];
            for (int f = 0; f < nf; ++f)
                for (int r0 = 0; r0 < tk.w; r0 += kChunk) {
                    T v[kChunk];
#pragma unroll
                    for (int j = 0; j < kChunk; ++j)
                        v[j] = r0 + j < tk.w ? base[f * fs + (long long)(tk.z + r0 + j) * L + x] : T(0);
#pragma unroll
                    for (int j = 0; j < kChunk; ++j) st |= value_status(v[j]);
                }
        }
        st = __reduce_or_sync(0xffffffffu, st);
        if (lane == 0 && st) atomicOr(it.status + k, st);
    }
}

template <typename T>
cudaError_t launch_validate(const T* state, const InstTables& it, const int4* tasks, int n_tasks, int nf, int grid,
                            cudaStream_t s)
{
    if (n_tasks <= 0) return cudaSuccess;
    validate_kernel<T><<<grid, 256, 0, s>>>(state, it, tasks, n_tasks, nf);
    return cudaGetLastError();
}
template cudaError_t launch_validate<float>(const float*, const InstTables&, const int4*, int, int, int, cudaStream_t);
template cudaError_t launch_validate<double>(const double*, const InstTables&, const int4*, int, int, int,
                                             cudaStream_t);

// Upload of a state from page-locked host memory: the device reads it over the host
// link, 16 bytes per load, grid-stride.  On GB300 machines the copy engines' host-to-device
// rate dropped from 211 to 18-30 GB/s in some copies after compute phases, while these
// loads of the same buffer held 212 GB/s.
__global__ void __launch_bounds__(512) copy_in_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst,
                                                      long long n16)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += stride) dst[i] = src[i];
}

cudaError_t launch_copy_in(const void* src, void* dst, size_t bytes, int grid, cudaStream_t s)
{
    if (bytes == 0) return cudaSuccess;
    if (((uintptr_t)src | (uintptr_t)dst | (uintptr_t)bytes) & 15u) return cudaErrorInvalidValue;
    copy_in_kernel<<<grid, 512, 0, s>>>((const uint4*)src, (uint4*)dst, (long long)(bytes / 16));
    return cudaGetLastError();
}

}  // namespace tmg
