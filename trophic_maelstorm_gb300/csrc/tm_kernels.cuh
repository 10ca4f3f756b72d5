// tm_kernels.cuh -- kernel parameter blocks and launchers shared by the
// kernel translation units and the C ABI implementation.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "tm_per_device.h"

// A context: one device and the stream every call on it launches on (tm_create).
struct tm_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    int num_sms = 0;
    unsigned probe = 0;            // TM_PROBE_* flags for objects created from now on (tests)
};

// tm_spectrum.cu: plan and buffers of a power spectrum, kept by their batch
struct SpectrumWork;
void spectrum_work_destroy(SpectrumWork* w);
int power_spectrum(const void* dev_field, int precision, int L, double binwidth, cudaStream_t s, double* kvals,
                   double* power, int max_bins, int* n_bins, SpectrumWork** keep);

namespace tmg {

// Programmatic dependent launch: a kernel launched by launch_pdl may start while the last
// blocks of its predecessor on the stream end, and waits for that end (and its writes) in
// pdl_wait(), which every block of such a kernel calls before it touches memory that
// another kernel writes.  Its prologue -- tables, barriers, the launch itself -- then
// overlaps the predecessor's tail.  No kernel lets its successor start any earlier
// (griddepcontrol.launch_dependents): blocks waiting in slots that the predecessor's own
// blocks could use made the dilute DP step 17 % and the 8 x 256^2 Rietkerk step 16 %
// slower than this.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... Params, typename... Args>
cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, const Args&... args)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute a;
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<Params>(args)...);
}

// Lets `kernel` take `bytes` of dynamic shared memory on the current device; `done` is the
// kernel's own.
template <typename Kernel>
cudaError_t allow_smem(PerDevice& done, Kernel kernel, size_t bytes)
{
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    return done.run(device, [&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); });
}

// Dornic constants of one instance: lambda e^{beta dt}, 1/lambda, e^{beta dt}, (e^{beta dt}-1)/beta
struct __align__(16) Dc4 { double x, y, z, w; };

// Per-instance tables in device memory (structure of arrays).
struct InstTables {
    const long long* off;          // element offset of the instance's first field
    const long long* fstride;      // elements between fields of one instance
    const int* L;
    const unsigned long long* seed;
    const double* R;               // Rietkerk rainfall (per instance)
    const Dc4* consts;         // Dornic constants: (lambda e^{beta dt}, 1/lambda, e^{beta dt}, (e^{beta dt}-1)/beta)
    int* alive;                    // DP extinction flags (nullptr: never skip)
    unsigned* status;              // TM_STATUS_* bits
};

// Warp task: 32 columns x `rows` rows of one instance: (inst, x0, y0, rows).
// Block task (RK4 tile): (inst, x0, y0, tile rows).

template <typename T>
struct DornicArgs {
    const T* in;                   // state (field 0 is read)
    T* out;                        // field-0 slots receive the result
    InstTables it;
    const int4* tasks;
    int n_tasks;
    const long long* step_base;    // device step counter (graph replays) or nullptr
    long long step_off;            // step = (*step_base) + step_off
    T dcoef, two_s2, b, c, dt, dt2, dt6, clo, ceps;
    int sampler;                   // 0 exact, 1 Gaussian above 100, 2 mean (noise off)
    int cubic;
    int rows_cap;                  // rows of the largest task (<= kMaxRowsPerTask)
    const T* site_b;               // per-site loss coefficient b_v (packed like the state) or nullptr
    int zero_fixed;                // a +0 draw finishes as +0, no status bit (finite b, c, dt; no site_b)
    int cap1;                      // TM_PROBE_SAMPLER_CAP1: rejection loops stop after one attempt
    uint4* dlist;                  // FP32: deferred sites (instance, site, Poisson mean, Gamma shape bits),
                                   // one segment of seg_cap entries per warp of the step kernel's grid
    unsigned* dcnt;                // FP32: entries in each warp's segment (written by the step kernel)
    long long seg_cap;             // entries per segment (all sites of one warp's tasks)
    long long dlist_cap;           // entries the list holds
    long long max_seg;             // segments dcnt holds
};

template <typename T>
struct RK4Args {
    const T* in;                   // [P|W|O] state
    const T* pstar;                // P after the Dornic draw (field-0 slots); nullptr when deterministic
    T* out;
    InstTables it;
    const int4* tasks;             // block tasks
    int n_tasks;
    T alpha, k2, k2W0, gmax, cgmax, k1, rW, d, DPx, DWx, DOx, dt2, dt6, dt, clo, ceps;
    int wait_limit;                // polls of a tile's copy barrier before the CTA gives up
    int probe_no_copy;             // TM_PROBE_TILE_WAIT: issue no copy, so the bounded wait runs out
};

// Measurements.  partial[t*4 + f] of task t: f = 0..nf-1 field sums, 3 = sites with field
// 0 > 0.  With spread (DP), f = 1 is the sum over occupied sites of the squared distance
// (row - cy)^2 + (col - cx)^2 from the seed site (meansq_spread_of_vector,
// stochasticSPDP.cpp:156-170), summed as integers; scx, scy < 0 mean L/2.
constexpr int kMeasureOnce = 512;      // an instance with more tasks is summed in groups
constexpr int kMeasureGroupShift = 8;  // groups of 256 tasks at least
__host__ __device__ inline int measure_group_shift(int nt)
{
    int sh = kMeasureGroupShift;
    while ((1LL << (2 * sh)) < nt) ++sh;
    return sh;
}
// First group of instance k, whose tasks start at b0: up to floor(n / 256) + 1 groups of
// its n tasks end before the next instance's first.
__host__ __device__ inline int measure_group_base(int b0, int k) { return (b0 >> kMeasureGroupShift) + k; }
template <typename T>
struct MeasureArgs {
    const T* state;
    InstTables it;
    const int4* tasks;
    const int* begin;              // first task of each instance, and n_tasks
    int n_tasks, n_inst, nf;
    int spread, scx, scy;
    int dp_extinction;
    double* partial;               // 4 per task
    double* group_sums;            // 4 per group
    int* arrived;                  // per instance, then per group: rows written so far; 0 between launches
    double* obs_row;
};

template <typename T>
struct DetTileArgs {               // noise-off DP step over 64 x 32 tiles of every instance (a = it.R[k])
    const T* in;
    T* out;
    InstTables it;
    const int4* tasks;             // block tasks
    int n_tasks;
    T b, c, dlap, dk12, dt, dt2, dt6;
    int cubic;
};

// launchers (defined in the kernel translation units)
template <typename T>
cudaError_t launch_dornic(const DornicArgs<T>& a, int rem, int grid, int block, cudaStream_t s);
template <>   // tm_step.cu
cudaError_t launch_dornic<float>(const DornicArgs<float>& a, int rem, int grid, int block, cudaStream_t s);
template <>   // tm_step64.cu
cudaError_t launch_dornic<double>(const DornicArgs<double>& a, int rem, int grid, int block, cudaStream_t s);
template <typename T>
cudaError_t launch_rk4(const RK4Args<T>& a, bool det, int grid, cudaStream_t s);
template <>
cudaError_t launch_rk4<float>(const RK4Args<float>& a, bool det, int grid, cudaStream_t s);
template <>
cudaError_t launch_rk4<double>(const RK4Args<double>& a, bool det, int grid, cudaStream_t s);
template <typename T>
cudaError_t launch_measure(const MeasureArgs<T>& a, int grid, int block, cudaStream_t s);
template <typename T>
cudaError_t launch_border_stop(const T* state, const InstTables& it, int n_inst, cudaStream_t s);
template <typename T>
cudaError_t launch_validate(const T* state, const InstTables& it, const int4* tasks, int n_tasks, int nf, int grid,
                            cudaStream_t s);
cudaError_t launch_consts(const double* a0, const double* astep, int n, int n_steps, double diff4, double sigma2, double dt,
                          const long long* step_base, long long step_off, Dc4* out, cudaStream_t s);
cudaError_t launch_set_step(long long* d_step, long long v, cudaStream_t s);
cudaError_t launch_copy_in(const void* src, void* dst, size_t bytes, int grid, cudaStream_t s);
template <typename T>
cudaError_t launch_box_means(const T* field, int L, int box, double* out, cudaStream_t s);
template <typename T>
cudaError_t launch_dp_det(const DetTileArgs<T>& a, int stencil, int rk4, int grid, cudaStream_t s);

constexpr int kMaxRowsPerTask = 16;
constexpr int RK_TX = 64, RK_TY = 32, RK_H = 4;
constexpr int RK_RX = RK_TX + 2 * RK_H, RK_RY = RK_TY + 2 * RK_H, RK_RN = RK_RX * RK_RY;
constexpr int RK_THREADS = 512;
constexpr int RK64_THREADS = 768;          // FP64 RK4 tiles: threads, and rows of the tallest tile
constexpr int RK64_UNIT = RK64_THREADS / RK_TX, RK64_TY = 32 / RK64_UNIT * RK64_UNIT;
constexpr int RK_CTAS = 2;                 // resident FP32 RK4 tile CTAs per SM

}  // namespace tmg
