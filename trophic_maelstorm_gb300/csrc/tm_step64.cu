// tm_step64.cu -- the fused Dornic step in FP64.
//
// The step is the one of tm_step.cu: the same streams, the same operations in the
// same order, the same bits.  What differs is what GB300 does cheaply.  One FP64
// warp instruction occupies its scheduler's FP64 pipe for 64-76 cycles, however
// many lanes it has, so the kernel is written around how few of them a site needs:
//   * absorbing sites are found by the bits of the five values (row masks from
//     ballots), without an FP64 operation;
//   * the Poisson search, the squeeze, the ziggurat's wedge test and the log test
//     only decide something.  They run in FP32 with an error bound, and the FP32
//     answer is taken where the bound proves that the FP64 comparison has the same
//     outcome; the rest (two in 10^4 of the searches) do the FP64 comparison;
//   * divisions, square roots and some products are rounded exactly on the integer
//     pipe (tm_f64.cuh).
// The whole warp runs the straight-line draw together (lanes without a site repeat
// one): lanes that left the search one by one made the rest of the draw run twice.
// Measured, 16 lattices of 256^2, 32 steps of a decaying run: RK4 remainder 20.2 ->
// 3.9 ms; general sampler for every site 319 FP64 instructions per 32 sites, now about 30
// (Euler-exact remainder).  Bound by the FP64 pipe (60-65 % busy) and the integer
// pipe together.  Two CTAs of 8 warps per SM: three (80 registers, small spills) took
// the same time, four 13 % more.
//
// Sites the straight-line draw cannot finish are carried in three lists per warp
// and drawn 32 at a time, so that a rare path runs with full lanes: the whole
// general sampler (list 0), the general Gamma draw with its shape known (list 1)
// and the boost U^(1/k) of shapes below 1 (list 2).  A draw depends only on (seed,
// site, step), so it may run in any later pass of the same warp.
#include "tm_draw64.cuh"
#include "tm_kernels.cuh"

namespace tmg {

namespace {

constexpr int kWarps = 8;
constexpr int kListCap = 64;                // carried entries of one list: up to 31, and 32 new ones

struct ListEntry {                          // 24 bytes
    int k;                                  // instance
    uint32_t site;
    double a, b;
};

__host__ __device__ __forceinline__ size_t warp_bytes(int rows_cap)
{
    return 3 * kListCap * sizeof(ListEntry) + (size_t)rows_cap * 32 * sizeof(unsigned short);
}

// -b x^2 (- c x^3)
template <bool CUBIC>
__device__ __forceinline__ double rem_f64(double x, double b, double c)
{
    double f = tmf::mul((-b) * x, x);
    if (CUBIC) f = f - tmf::mul(tmf::mul(c * x, x), x);
    return f;
}
template <bool CUBIC>
__device__ __forceinline__ double rem_rk4(const DornicArgs<double>& A, double rs, double bi)
{
    const double k1 = rem_f64<CUBIC>(rs, bi, A.c);
    const double k2 = rem_f64<CUBIC>(rs + A.dt2 * k1, bi, A.c);
    const double k3 = rem_f64<CUBIC>(rs + A.dt2 * k2, bi, A.c);
    const double k4 = rem_f64<CUBIC>(rs + A.dt * k3, bi, A.c);
    return rs + A.dt6 * (fma(2.0, k3, fma(2.0, k2, k1)) + k4);
}

// Remainder, clamp and status bits of one site after its draw (finish_site of
// tm_step.cu, with the comparisons on bits).
template <int REM>
__device__ __forceinline__ double finish64(const DornicArgs<double>& A, double rs, double bi, unsigned& st)
{
    double res;
    if (REM == 0) {
        res = tmf::div(rs, 1.0 + (bi * rs) * A.dt);
    } else if (REM == 1) {
        res = A.cubic ? rem_rk4<true>(A, rs, bi) : rem_rk4<false>(A, rs, bi);
    } else {
        res = rs;
    }
    if (REM != 2) {
        // not below ceps if positive with larger bits (a NaN neither)
        const long long rb = __double_as_longlong(res);
        if (!(rb >= 0 && rb >= __double_as_longlong(A.ceps)) && rb != 0) {
            if (tmf::hw_in_range(res, A.clo, A.ceps)) res = 0.0;
        }
        st |= value_status(res);
    }
    return res;
}

struct SiteMean {
    double cur, alpha, m, mu1;
};

// Value, neighbour coupling, Poisson mean and Gamma shape of a site.
__device__ __forceinline__ SiteMean site_mean(const DornicArgs<double>& A, const double* __restrict__ src, int L, int y,
                                              int x, double pm)
{
    const int yn = (y == 0) ? L - 1 : y - 1, ys = (y == L - 1) ? 0 : y + 1;
    const int xw = (x == 0) ? L - 1 : x - 1, xe = (x == L - 1) ? 0 : x + 1;
    SiteMean s;
    s.cur = src[(long long)y * L + x];
    const double n = src[(long long)yn * L + x], so = src[(long long)ys * L + x];
    const double w = src[(long long)y * L + xw], e = src[(long long)y * L + xe];
    s.alpha = A.dcoef * (((n + so) + w) + e);
    s.m = tmf::mul(pm, s.cur);
    s.mu1 = tmf::mul(s.alpha, A.two_s2);
    return s;
}

// Finish a drawn site and store it.
template <int REM>
__device__ __forceinline__ void store_site(const DornicArgs<double>& A, int k, uint32_t site, double rs, unsigned st)
{
    const long long o = A.it.off[k] + (long long)site;
    double res = rs;
    if (!(A.zero_fixed && __double_as_longlong(rs) == 0))
        res = finish64<REM>(A, rs, A.site_b ? A.site_b[o] : A.b, st);
    A.out[o] = res;
    if (st) atomicOr(A.it.status + k, st);
}

// One carried entry of list `which`.
template <int REM, int SAMP, int CAP>
__device__ __forceinline__ void draw_general(const DornicArgs<double>& A, const Tab64& tab, long long step, bool whole,
                                             const ListEntry& e)
{
    Stream<double> g;
    g.init(A.it.seed[e.k], e.site, step);
    double k = e.a;
    bool gauss = false;
    if (whole) {
        const int L = A.it.L[e.k];
        const int y = (int)(e.site / (uint32_t)L), x = (int)(e.site - (uint32_t)y * (uint32_t)L);
        const SiteMean s = site_mean(A, A.in + A.it.off[e.k], L, y, x, A.it.consts[e.k].x);
        double n = 0.0;
        if (s.m > 0.0) {
            if (SAMP == 1 && s.m > 100.0) {
                const double z = normal64<CAP>(g, tab);
                n = trunc(z * tmf::sqrt(s.m) + s.m);
            } else {
                n = s.m < 32.0 ? poisson_exact<CAP>(g, s.m, (const SmemTab<double>&)tab) : ptrs64<CAP>(g, s.m, tab);
            }
        }
        k = s.mu1 + n;
        gauss = SAMP == 1 && k > 100.0;
    } else if (e.b != 0.0) {
        (void)g.u32();                       // the word the count took
    }
    double gv;
    if (gauss) {
        const double z = normal64<CAP>(g, tab);
        gv = z * tmf::sqrt(k) + k;
    } else {
        gv = gamma64<CAP>(g, k, tab);
    }
    store_site<REM>(A, e.k, e.site, gv * A.it.consts[e.k].y, g.status);
}

// The boost of a shape below 1: entry a = shape, b = the Gamma(shape + 1) draw,
// negative where the site took no Poisson word.
template <int REM>
__device__ __forceinline__ void draw_boost(const DornicArgs<double>& A, long long step, const ListEntry& e)
{
    const unsigned long long seed = A.it.seed[e.k];
    const uint32_t slo = (uint32_t)(unsigned long long)step, shi = (uint32_t)((unsigned long long)step >> 32);
    const bool drew = (int32_t)hi32(e.b) >= 0;
    const U4 r1 = philox4x32_10(e.site, slo, 1u, shi, (uint32_t)seed, (uint32_t)(seed >> 32));
    uint32_t w1 = r1.x, w2 = r1.y;
    if (!drew) {
        const U4 r0 = philox4x32_10(e.site, slo, 0u, shi, (uint32_t)seed, (uint32_t)(seed >> 32));
        w1 = r0.w;
        w2 = r1.x;
    }
    const double u = tmf::open_unit(((unsigned long long)w1 << 21) | (unsigned long long)(w2 >> 11));
    const double res = tmf::abs_bits(e.b) * tm_exp(tmf::div(tm_log_pos(u), e.a));
    store_site<REM>(A, e.k, e.site, res * A.it.consts[e.k].y, 0u);
}

}  // namespace

template <int REM, int SAMP, int CAP>
__global__ void __launch_bounds__(256, 2) dornic_step64_kernel(const DornicArgs<double> A)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ Tab64 tab;
    __shared__ int left[kWarps][3];
    tab.fill_all();
    pdl_wait();
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    unsigned char* const wbase = smem_raw + warp * warp_bytes(A.rows_cap);
    ListEntry* const lists = reinterpret_cast<ListEntry*>(wbase);
    unsigned short* const Wq = reinterpret_cast<unsigned short*>(lists + 3 * kListCap);
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    // consecutive tasks go to different blocks, so that few tasks still spread over the SMs
    const int gw = warp * (int)gridDim.x + (int)blockIdx.x;
    const int nw = (int)gridDim.x * kWarps;
    const long long step = (A.step_base ? *A.step_base : 0LL) + A.step_off;
    int cnt[3] = {0, 0, 0};
    // one more trip after the last task empties the lists of the whole block together
    int4 next = A.tasks[gw < A.n_tasks ? gw : 0];
    for (int t = gw;; t += nw) {
        const bool more = t < A.n_tasks;
        // the next task is asked for a trip ahead, its instance's tables in one round
        const int4 tk = next;
        const int k = tk.x, x0 = tk.y, y0 = tk.z, rows = tk.w;
        const int L = A.it.L[k], alive = A.it.alive ? A.it.alive[k] : 1;
        const long long off = A.it.off[k];
        if (t + nw < A.n_tasks) next = A.tasks[t + nw];
        int nq = 0;
        if (more && alive != 0) {
            const double* __restrict__ src = A.in + off;
            const int w = min(32, L - x0);
            const int x = x0 + lane;
            const bool act = lane < w;
            // pass 1: a site is absorbing when it and its neighbours are zero, which row
            // masks of non-zero values tell; absorbing sites are finished here
            const bool erow = lane < rows;
            const int xw = (x0 == 0) ? L - 1 : x0 - 1;
            const int xe = (x0 + w == L) ? 0 : x0 + w;
            const int yn = (y0 == 0) ? L - 1 : y0 - 1;
            // Every load of the pass is issued before the first vote waits for one: each vote
            // in between cost a round trip to the L2, and an empty task 4.6k cycles instead
            // of 2.7k (64 spreading lattices of 101^2, 200 steps: 6.20 -> 5.19 ms).
            const double vw = erow ? src[(long long)(y0 + lane) * L + xw] : 0.0;
            const double ve = erow ? src[(long long)(y0 + lane) * L + xe] : 0.0;
            const double vn = act ? src[(long long)yn * L + x] : 0.0;
            const double vc = act ? src[(long long)y0 * L + x] : 0.0;
            double v[8];
            const auto load8 = [&](int r0) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    int y = y0 + r0 + j + 1;
                    if (y >= L) y -= L;
                    v[j] = (act && r0 + j < rows) ? src[(long long)y * L + x] : 0.0;
                }
            };
            load8(0);
            const unsigned wm = __ballot_sync(0xffffffffu, !tmf::is_zero(vw));
            const unsigned em = __ballot_sync(0xffffffffu, !tmf::is_zero(ve));
            const unsigned actm = __ballot_sync(0xffffffffu, act);
            unsigned mn = __ballot_sync(0xffffffffu, !tmf::is_zero(vn));
            unsigned mc = __ballot_sync(0xffffffffu, !tmf::is_zero(vc));
            unsigned st = 0;
            for (int r0 = 0; r0 < rows; r0 += 8) {
                if (r0 > 0) load8(r0);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int r = r0 + j;
                    if (r >= rows) break;
                    const unsigned ms = __ballot_sync(0xffffffffu, !tmf::is_zero(v[j]));
                    unsigned lm = mn | mc | ms | (mc << 1) | (mc >> 1) | ((wm >> r) & 1u) | (((em >> r) & 1u) << (w - 1));
                    if (SAMP == 2) lm = 0xffffffffu;
                    lm &= actm;
                    if ((lm >> lane) & 1u) {
                        Wq[nq + __popc(lm & lt_mask)] = (unsigned short)(r * 32 + lane);
                    } else if (act) {
                        const long long o = off + (long long)(y0 + r) * L + x;
                        double res = 0.0;
                        if (!A.zero_fixed) res = finish64<REM>(A, 0.0, A.site_b ? A.site_b[o] : A.b, st);
                        A.out[o] = res;
                    }
                    nq += __popc(lm);
                    mn = mc;
                    mc = ms;
                }
            }
            if (st) atomicOr(A.it.status + k, st);
            __syncwarp();
        }
        const unsigned long long seed = A.it.seed[k];
        const Dc4 cs = A.it.consts[k];
        // pass 2: the queued sites, 32 at a time, straight line and with the whole warp
        // (lanes without a site draw the last one again); then whatever list is full
        int base = 0;
        do {
            int outcome = -1;                  // -1 done, 0..2: the list that draws it
            ListEntry en;
            en.k = k;
            if (base < nq) {
                const bool has = base + lane < nq;
                const int li = Wq[has ? base + lane : nq - 1];
                const int y = y0 + (li >> 5), x = x0 + (li & 31);
                const uint32_t site = (uint32_t)y * (uint32_t)L + (uint32_t)x;
                en.site = site;
                const SiteMean s = site_mean(A, A.in + off, L, y, x, cs.x);
                double rs = 0.0;               // also where the neighbours cancel or their sum underflows
                if (SAMP == 2) {
                    rs = cs.z * s.cur + cs.w * s.alpha;
                } else {
                    const U4 r = philox4x32_10(site, (uint32_t)(unsigned long long)step, 0u,
                                               (uint32_t)((unsigned long long)step >> 32), (uint32_t)seed,
                                               (uint32_t)(seed >> 32));
                    const uint32_t hm = hi32(s.m), hmu = hi32(s.mu1);
                    const bool live = !(tmf::is_zero(s.alpha) && tmf::is_zero(s.cur));
                    const bool draw = !tmf::is_zero(s.m);
                    // above 100 by the high word: 100 itself has it too, and takes list 0
                    const bool gauss = SAMP == 1 && live && hmu < 0x7ff00000u && hm >= 0x40590000u && hm < 0x7ff00000u;
                    // m < 32 (not negative, not NaN), shape not negative, Inf or NaN
                    const bool small = live && hmu < 0x7ff00000u && hm < 0x40400000u;
                    if (live && !small) outcome = 0;
                    const int n = search_count(small && draw, small ? tmf::trunc_f32(s.m) : 0.0f, r.x, tab.rcpf + 3);
                    if (small && draw && n < 0) outcome = 0;
                    if (SAMP == 1 && __any_sync(0xffffffffu, gauss)) {
                        // Gaussian approximations of both draws: one ziggurat word each
                        if (gauss && s.m > 100.0) {
                            const int32_t h1 = zig_value(r.x), h2 = zig_value(r.y);
                            const ZigLayer<double> l1 = tab.zig[zig_layer(r.x)], l2 = tab.zig[zig_layer(r.y)];
                            const uint32_t a1 = (uint32_t)(h1 < 0 ? -h1 : h1), a2 = (uint32_t)(h2 < 0 ? -h2 : h2);
                            const double kk = s.mu1 + trunc(tmf::mul(signed_mul(h1, l1.w), tmf::sqrt(s.m)) + s.m);
                            if (a1 < l1.k && a2 < l2.k && kk > 100.0) {
                                rs = (tmf::mul(signed_mul(h2, l2.w), tmf::sqrt(kk)) + kk) * cs.y;
                                outcome = -1;
                            }
                        }
                        __syncwarp();
                    }
                    const bool gamma = small && outcome < 0;
                    if (__any_sync(0xffffffffu, gamma)) {
                        const double kg = gamma ? s.mu1 + tmf::from_u31(draw ? (uint32_t)n : 0u) : 1.0;
                        const uint32_t hk = hi32(kg);
                        const uint32_t wz = draw ? r.y : r.x, wu = draw ? r.z : r.y;
                        const bool boost = hk < 0x3ff00000u;
                        const double d = (kg + (boost ? 1.0 : 0.0)) - 1.0 / 3.0;
                        const double c = Tr<double>::inv_sqrt(9.0 * d);
                        const int32_t hz = zig_value(wz);
                        const uint32_t az = (uint32_t)(hz < 0 ? -hz : hz);
                        const ZigLayer<double> lz = tab.zig[zig_layer(wz)];
                        const double xz = signed_mul(hz, lz.w);
                        const double v = 1.0 + c * xz;
                        const float vf = tmf::trunc_f32(v), xf = tmf::trunc_f32(tmf::abs_bits(xz)), x2f = xf * xf;
                        // squeeze with room for the FP32 roundings; 1 - u is at least ~wu 2^-32
                        const float lhs = ((float)(~wu) * 0x1p-32f) * ((108.0f * tmf::trunc_f32(d)) * (vf < 1.0f ? vf : 1.0f));
                        const bool ok = az < lz.k && (int32_t)hi32(v) > 0 && lhs > (x2f * x2f) * 1.0001f;
                        const double res = tmf::mul_normal(d, tmf::mul_normal(tmf::mul_normal(v, v), v));
                        if (gamma && !tmf::is_zero(kg)) {              // Gamma(0) = 0
                            if (SAMP == 1 && hk >= 0x40590000u) {
                                outcome = 0;
                            } else if (!ok) {
                                outcome = 1;
                                en.b = draw ? 1.0 : 0.0;
                            } else if (boost) {
                                outcome = 2;
                                en.b = tmf::with_sign(res, !draw);
                            } else {
                                rs = res * cs.y;
                            }
                            en.a = kg;
                        }
                        __syncwarp();
                    }
                }
                if (!has) outcome = 3;
                if (outcome < 0) store_site<REM>(A, k, site, rs, 0u);
                __syncwarp();
            }
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                const unsigned bal = __ballot_sync(0xffffffffu, outcome == l);
                if (outcome == l) lists[l * kListCap + cnt[l] + __popc(bal & lt_mask)] = en;
                cnt[l] += __popc(bal);
            }
            __syncwarp();
            // full lists are drawn 32 entries at a time.  On the last trip what the block's
            // warps still carry is joined, so that it takes as few passes as it can and
            // the passes run on different warps.
            if (!more) {
                if (lane < 3) left[warp][lane] = lane == 0 ? cnt[0] : (lane == 1 ? cnt[1] : cnt[2]);
                __syncthreads();
            }
            for (int job = warp;; job += kWarps) {
                int l, at = 0;
                const ListEntry* e = lists;
                bool on = true;
                if (more) {
                    l = cnt[2] >= 32 ? 2 : (cnt[0] >= 32 ? 0 : 1);
                    at = (l == 2 ? cnt[2] : (l == 0 ? cnt[0] : cnt[1])) - 32;
                    if (at < 0) break;
                    if (l == 2) cnt[2] = at;
                    else if (l == 0) cnt[0] = at;
                    else cnt[1] = at;
                    e += l * kListCap + at + lane;
                } else {
                    // job -> list and 32 of the joined entries: the general draws first
                    int j = job;
                    for (l = 0; l < 3; ++l) {
                        int n = 0;
                        for (int w = 0; w < kWarps; ++w) n += left[w][l];
                        const int passes = (n + 31) / 32;
                        if (j < passes) break;
                        j -= passes;
                    }
                    if (l == 3) break;
                    int i = j * 32 + lane;
                    on = false;
                    for (int w = 0; w < kWarps; ++w) {
                        const int n = left[w][l];
                        if (!on && i < n) {
                            on = true;
                            e = reinterpret_cast<const ListEntry*>(smem_raw + w * warp_bytes(A.rows_cap)) + l * kListCap + i;
                        }
                        i -= n;
                    }
                }
                if (l == 2) {
                    if (on) draw_boost<REM>(A, step, *e);
                } else {
                    if (on) draw_general<REM, SAMP, CAP>(A, tab, step, l == 0, *e);
                }
                __syncwarp();
            }
            base += 32;
        } while (base < nq);
        if (!more) break;
        __syncwarp();
    }
}

namespace {

template <int REM, int SAMP, int CAP = kSamplerCap>
cudaError_t launch64_t(const DornicArgs<double>& a, int grid, int block, cudaStream_t s)
{
    static PerDevice allowed;
    const cudaError_t e = allow_smem(allowed, dornic_step64_kernel<REM, SAMP, CAP>, warp_bytes(kMaxRowsPerTask) * kWarps);
    if (e != cudaSuccess) return e;
    return launch_pdl(dornic_step64_kernel<REM, SAMP, CAP>, dim3(grid), dim3(block), warp_bytes(a.rows_cap) * kWarps, s, a);
}

template <int REM>
cudaError_t launch64_r(const DornicArgs<double>& a, int grid, int block, cudaStream_t s)
{
    if (a.cap1) {  // the sampler-cap probe: DP, Euler-exact remainder, exact sampler only
        if (REM == 0 && a.sampler == 0) return launch64_t<0, 0, 1>(a, grid, block, s);
        return cudaErrorInvalidValue;
    }
    if (a.sampler == 0) return launch64_t<REM, 0>(a, grid, block, s);
    if (a.sampler == 1) return launch64_t<REM, 1>(a, grid, block, s);
    if (a.sampler == 2) return launch64_t<REM, 2>(a, grid, block, s);
    return cudaErrorInvalidValue;
}

}  // namespace

template <>
cudaError_t launch_dornic<double>(const DornicArgs<double>& a, int rem, int grid, int block, cudaStream_t s)
{
    if (a.n_tasks <= 0) return cudaSuccess;
    if (block != 32 * kWarps || a.rows_cap < 1 || a.rows_cap > kMaxRowsPerTask) return cudaErrorInvalidValue;
    if (rem == 0) return launch64_r<0>(a, grid, block, s);
    if (rem == 1) return launch64_r<1>(a, grid, block, s);
    if (rem == 2) return launch64_r<2>(a, grid, block, s);
    return cudaErrorInvalidValue;
}

}  // namespace tmg
