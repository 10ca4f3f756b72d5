// Device arithmetic and draws against the hardware's own operations and the FP64 methods,
// exhaustively where the argument is one FP32 value.  Built and called by
// test_gpu_device_checks.py; every entry returns 0 or a CUDA error and fills a Result.
#include "tm_draw64.cuh"

#include <cuda_runtime.h>
#include <math.h>

using namespace tmg;

struct Result {
    unsigned long long n, bad, aux;   // compared, different, per check
    unsigned worst;                   // largest ratio seen, as the bits of a float >= 0
    unsigned where;                   // some argument that differed
};

namespace {

constexpr int kGrid = 152 * 8, kBlock = 256;

__device__ void note(Result* r, unsigned long long n, unsigned long long bad, unsigned long long aux, unsigned where)
{
    atomicAdd(&r->n, n);
    if (bad) { atomicAdd(&r->bad, bad); r->where = where; }
    if (aux) atomicAdd(&r->aux, aux);
}
__device__ unsigned long long index0() { return blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; }
__device__ unsigned long long stride() { return (unsigned long long)gridDim.x * blockDim.x; }

__device__ unsigned long long mix(unsigned long long x)   // splitmix64
{
    x += 0x9e3779b97f4a7c15ULL;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
    return x ^ (x >> 31);
}
__device__ double unit(unsigned long long h) { return (double)(h >> 11) * 0x1p-53; }

template <typename K>
int run(Result* out, K kernel, unsigned long long a, unsigned long long b)
{
    Result* d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(Result));
    if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(Result));
    if (e == cudaSuccess) {
        kernel<<<kGrid, kBlock>>>(d, a, b);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d, sizeof(Result), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}

// ---- every FP32 value
// aux: values between 2^-100 and 2^100 that neg_rcp hands on
__global__ void k_reciprocals(Result* r, unsigned long long, unsigned long long)
{
    unsigned long long n = 0, bad = 0, aux = 0;
    unsigned where = 0;
    for (unsigned long long i = index0(); i < (1ULL << 32); i += stride()) {
        const float x = __uint_as_float((unsigned)i), ax = fabsf(x), want = __frcp_rn(x);
        bool ok = true;
        const float v = neg_rcp(x, ok);
        bool wrong = ok && __float_as_uint(v) != __float_as_uint(-want);
        const bool plain = ax >= 0x1p-100f && ax <= 0x1p100f;
        if (plain) {
            wrong = wrong || __float_as_uint(rcp_newton(x)) != __float_as_uint(want);
            aux += !ok;
        }
        n += ok;
        bad += wrong;
        if (wrong) where = (unsigned)i;
    }
    note(r, n, bad, aux, where);
}
__global__ void k_inv_sqrt(Result* r, unsigned long long, unsigned long long)
{
    unsigned long long n = 0, bad = 0;
    unsigned where = 0;
    for (unsigned long long i = 0x3f800000ULL + index0(); i < 0x7f800000ULL; i += stride(), ++n) {
        const float x = __uint_as_float((unsigned)i);
        if (__float_as_uint(Tr<float>::inv_sqrt_normal(x)) != __float_as_uint(__frsqrt_rn(x))) { ++bad; where = (unsigned)i; }
    }
    note(r, n, bad, 0, where);
}
// the logarithm's quotient for every mantissa in (sqrt(1/2), sqrt(2)]
__global__ void k_log_quotient(Result* r, unsigned long long, unsigned long long)
{
    unsigned long long n = 0, bad = 0;
    unsigned where = 0;
    for (unsigned long long i = 0x3f3504f3ULL + index0(); i <= 0x3fb504f4ULL; i += stride(), ++n) {
        const float f = __uint_as_float((unsigned)i) - 1.0f;
        if (__float_as_uint(quot_normal(f, 2.0f + f)) != __float_as_uint(__fdiv_rn(f, 2.0f + f))) { ++bad; where = (unsigned)i; }
    }
    note(r, n, bad, 0, where);
}

// ---- quotients next to the middle of two numbers: for every divisor mantissa b and every
// |e| <= 32 the dividends a and odd 25-bit M with 2^k a = M b + e (k = 24 where a >= b,
// else 25), that is every a / b within 32 / (2 b) ulp of such a middle
__global__ void k_quotient_middles(Result* r, unsigned long long, unsigned long long)
{
    unsigned long long n = 0, bad = 0;
    unsigned where = 0;
    for (unsigned long long b = (1ULL << 23) + index0(); b < (1ULL << 24); b += stride()) {
        const int s = __ffsll((long long)b) - 1;
        const unsigned long long odd = b >> s;
        unsigned long long inv = odd;
        for (int i = 0; i < 6; ++i) inv *= 2 - odd * inv;
        for (int k = 24; k <= 25; ++k)
            for (int e = -32; e <= 32; ++e) {
                // M is odd exactly if e has b's power of two
                if (e == 0 || __ffs(e) - 1 != s) continue;
                const unsigned long long mod = 1ULL << (k - s);
                const unsigned long long M0 = ((unsigned long long)(-(long long)(e >> s)) * inv) & (mod - 1);
                for (unsigned long long M = (1ULL << 24) + ((M0 - (1ULL << 24)) & (mod - 1)); M < (1ULL << 25); M += mod) {
                    const unsigned long long t = M * b + (long long)e;
                    const unsigned long long a = t >> k;
                    if ((t & ((1ULL << k) - 1)) || a < (1ULL << 23) || a >= (1ULL << 24) || (k == 24) != (a >= b)) continue;
                    const float fa = -(float)a * 0x1p-20f, fb = (float)b * 0x1p-60f;
                    ++n;
                    if (__float_as_uint(quot_normal(fa, fb)) != __float_as_uint(__fdiv_rn(fa, fb))) { ++bad; where = (unsigned)b; }
                }
            }
    }
    note(r, n, bad, 0, where);
}
// the boost's quotient log(u) / k: every u the draw can see, `per` shapes k each
__global__ void k_boost_quotient(Result* r, unsigned long long per, unsigned long long seed)
{
    unsigned long long n = 0, bad = 0;
    unsigned where = 0;
    for (unsigned long long i = index0(); i < per << 24; i += stride(), ++n) {
        const float l = tm_log_pos(((float)(i & 0xffffffu) + 0.5f) * 0x1p-24f);
        const unsigned long long h = mix(seed + i);
        // k in (2^-60, 1), its exponent 0..59 below 1
        const float k = __uint_as_float(((127u - 1u - (unsigned)((h >> 32) % 60)) << 23) | (unsigned)(h & 0x7fffffu));
        if (!(k > 0x1p-60f)) continue;
        if (__float_as_uint(quot_normal(l, k)) != __float_as_uint(__fdiv_rn(l, k))) { ++bad; where = (unsigned)i; }
    }
    note(r, n, bad, 0, where);
}

// ---- FP64 on the integer pipe, with the device's estimates
__device__ double operand(unsigned long long h, unsigned long long spread)
{
    unsigned long long m = mix(h) & tmf::kFrac;
    const int kind = (int)(h % 5), cut = (int)((h >> 8) % 52);
    if (kind == 0) m |= (1ULL << cut) - 1;
    if (kind == 1) m &= ~((1ULL << cut) - 1);
    if (kind == 2) m = tmf::kFrac - (m & 3);
    const unsigned long long w = mix(h ^ 0xabcdefULL);
    const unsigned long long e = spread ? 1023 - spread + w % (2 * spread + 1) : w % 2048;
    return __longlong_as_double((long long)(((w >> 60) & 1) << 63 | e << 52 | m));
}
__device__ bool same(double a, double b)
{
    return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
}
__global__ void k_f64(Result* r, unsigned long long n_pairs, unsigned long long spread)
{
    unsigned long long n = 0, bad = 0;
    for (unsigned long long i = index0(); i < n_pairs; i += stride(), ++n) {
        const double a = operand(mix(2 * i + 1), spread), b = operand(mix(2 * i + 2), spread);
        bad += !same(tmf::mul(a, b), __dmul_rn(a, b));
        bad += !same(tmf::div(a, b), __ddiv_rn(a, b));
        bad += !same(tmf::sqrt(a), __dsqrt_rn(a));
    }
    note(r, n, bad, 0, 0);
}
// recip31 for every leading 32 bits of the divisor, with the lowest and the highest rest:
// below 2^31 / (mb 2^-53) by at most 16
__global__ void k_recip31(Result* r, unsigned long long, unsigned long long)
{
    unsigned long long n = 0, bad = 0;
    unsigned where = 0;
    for (unsigned long long dh = (1ULL << 31) + index0(); dh < (1ULL << 32); dh += stride())
        for (int hi = 0; hi < 2; ++hi, ++n) {
            const unsigned long long mb = (dh << 21) | (hi ? (1ULL << 21) - 1 : 0);
            const unsigned __int128 top = (unsigned __int128)1 << 84, R = tmf::recip31(mb);
            if (!(R * mb <= top && (R + 16) * mb >= top)) { ++bad; where = (unsigned)dh; }
        }
    note(r, n, bad, 0, where);
}
// square roots for every argument of the FP32 estimate, 16 rests each
__global__ void k_sqrt(Result* r, unsigned long long, unsigned long long)
{
    unsigned long long n = 0, bad = 0;
    for (unsigned long long i = index0(); i < (1ULL << 28); i += stride(), ++n) {
        const unsigned long long head = i >> 4, odd = head >> 23;
        unsigned long long rest = mix(i) & ((1ULL << 29) - 1);
        if ((i & 15) == 0) rest = 0;
        if ((i & 15) == 1) rest = (1ULL << 29) - 1;
        const double x = __longlong_as_double((long long)((1023 + odd) << 52 | (head & 0x7fffff) << 29 | rest));
        bad += !same(tmf::sqrt(x), __dsqrt_rn(x));
    }
    note(r, n, bad, 0, 0);
}
__global__ void k_open_unit(Result* r, unsigned long long, unsigned long long)
{
    unsigned long long n = 0, bad = 0;
    for (unsigned long long i = index0(); i < (1ULL << 26); i += stride(), ++n) {
        const unsigned long long x = (i < 4096 ? i : (i < 8192 ? (1ULL << 53) - 1 - (i - 4096) : mix(i) >> (11 + i % 53)));
        bad += !same(tmf::open_unit(x), ((double)x + 0.5) * 0x1p-53);
    }
    note(r, n, bad, 0, 0);
}

// unit_f32 against the FP64 uniform of the same words and of their complements; worst is
// the largest relative difference in units of 2^-23
__global__ void k_unit(Result* r, unsigned long long n_words, unsigned long long)
{
    unsigned long long n = 0, bad = 0;
    float worst = 0.0f;
    for (unsigned long long i = index0(); i < n_words; i += stride(), ++n) {
        const unsigned long long h = mix(i);
        // leading words 0 to 7, all ones, and of every length
        const uint32_t w1 = i < (1u << 20) ? (uint32_t)(i & 7) : (i < (2u << 20) ? ~(uint32_t)(i & 7) : (uint32_t)(h >> 32) >> (i & 31));
        const uint32_t w2 = (i & 64) ? (uint32_t)h >> ((h >> 40) & 31) : (uint32_t)h;
        const double u = tmf::open_unit(((unsigned long long)w1 << 21) | (w2 >> 11));
        const float share = (float)(fabs((double)unit_f32(w1, w2) - u) / u * 0x1p23);
        worst = fmaxf(worst, share);
        bad += !(share <= 1.0f + 0x1p-20f);
    }
    note(r, n, bad, 0, 0);
    atomicMax(&r->worst, __float_as_uint(worst));
}

// ---- decisions in FP32 against the FP64 method
__device__ double mean_below_32(unsigned long long h)
{
    return (h & 1) ? 32.0 * unit(mix(h)) : 32.0 * exp2(-30.0 * unit(mix(h)));
}
// near: 0 the search on the stream's own word; 1 on words within two bounds of a tail.
// aux: undecided.
__global__ void k_search(Result* r, unsigned long long n_draws, unsigned long long near)
{
    __shared__ Tab64 tab;
    tab.fill_all();
    __syncthreads();
    unsigned long long n = 0, bad = 0, aux = 0;
    unsigned where = 0;
    for (unsigned long long i = index0(); i < n_draws; i += stride(), ++n) {     // whole warps: n_draws is a multiple of 32
        const double m = mean_below_32(mix(i));
        Stream<double> g;
        g.init(mix(i) | 1, (uint32_t)i, 7);
        Stream<double> at = g;
        uint32_t w = at.u32();
        double want;
        if (near) {
            // u on the grid of the words, within 2 search_eps of a tail of the FP64 search
            double p = m < 0.25 ? 0.0 : tm_exp(-m), q = m < 0.25 ? tm_negexpm1(m) : 1.0 - p;
            if (m < 0.25) p = tm_exp(-m);
            const int stop = (int)(mix(i ^ 5) % (2 + (unsigned)(2 * m)));
            double pt = p, qt = q;
            for (int k = 1; k <= stop; ++k) { pt = (pt * m) * tab.rcp[k]; qt = qt - pt; }
            const double off = (4.0 * unit(mix(i ^ 6)) - 2.0) * search_eps((float)m);
            const long long at_tail = (long long)((qt + off) * 0x1p32);
            w = (uint32_t)(at_tail < 0 ? 0 : (at_tail > 0xffffffffLL ? 0xffffffffLL : at_tail));
            const double u = (double)w * 0x1p-32;
            int k = 0;
            while (u < q && k < 200) { ++k; p = (p * m) * tab.rcp[k]; q = q - p; }
            want = (double)k;
        } else {
            want = poisson_exact<kSamplerCap>(g, m, (const SmemTab<double>&)tab);
        }
        __syncwarp();
        const int got = search_count(true, tmf::trunc_f32(m), w, tab.rcpf + 3);
        __syncwarp();
        if (got < 0) ++aux;
        else if ((double)got != want) { ++bad; where = (unsigned)i; }
    }
    note(r, n, bad, aux, where);
}
// the tails themselves: worst is the largest |FP32 - FP64| as a share of search_eps
__global__ void k_search_tails(Result* r, unsigned long long n_means, unsigned long long)
{
    __shared__ Tab64 tab;
    tab.fill_all();
    __syncthreads();
    unsigned long long n = 0, bad = 0;
    float worst = 0.0f;
    for (unsigned long long i = index0(); i < n_means; i += stride(), ++n) {
        const double m = mean_below_32(mix(i ^ 77));
        const float mf = tmf::trunc_f32(m);
        double p = tm_exp(-m), q = m < 0.25 ? tm_negexpm1(m) : 1.0 - p;
        float pf = tm_exp_neg_small(-mf), qf = mf < 0.25f ? tm_negexpm1(mf) : 1.0f - pf;
        for (int k = 0; k < kSearch; ++k) {
            const float share = (float)fabs(q - (double)qf) / search_eps(mf);
            worst = fmaxf(worst, share);
            bad += !(share < 1.0f);
            p = (p * m) * tab.rcp[k + 1];
            q = q - p;
            pf = (pf * mf) * tab.rcpf[3 + k + 1];
            qf = qf - pf;
        }
    }
    note(r, n, bad, 0, 0);
    atomicMax(&r->worst, __float_as_uint(worst));
}

template <typename F, typename W>
__device__ void compare_draws(Result* r, unsigned long long n_draws, F fast, W want)
{
    unsigned long long n = 0, bad = 0;
    unsigned where = 0;
    for (unsigned long long i = index0(); i < n_draws; i += stride(), ++n) {
        Stream<double> a;
        a.init(mix(i ^ 99), (uint32_t)mix(i), (int64_t)(i >> 20));
        Stream<double> b = a;
        const double x = fast(a, i), y = want(b, i);
        // value, status, and the place in the stream
        if (!same(x, y) || a.status != b.status || a.call != b.call || a.avail != b.avail) { ++bad; where = (unsigned)i; }
    }
    note(r, n, bad, 0, where);
}
__device__ double large_mean(unsigned long long i)
{
    const unsigned long long h = mix(i ^ 13);
    const double m = 32.0 * exp2(7.1 * unit(h));                     // 32 .. 4390
    return (h & 3) == 0 ? floor(m) : m;
}
template <int CAP>
__global__ void k_ptrs(Result* r, unsigned long long n_draws, unsigned long long)
{
    __shared__ Tab64 tab;
    tab.fill_all();
    __syncthreads();
    compare_draws(r, n_draws, [&](Stream<double>& g, unsigned long long i) { return ptrs64<CAP>(g, large_mean(i), tab); },
                  [&](Stream<double>& g, unsigned long long i) { return poisson_exact<CAP>(g, large_mean(i), (const SmemTab<double>&)tab); });
}
template <int CAP>
__global__ void k_normal(Result* r, unsigned long long n_draws, unsigned long long)
{
    __shared__ Tab64 tab;
    tab.fill_all();
    __syncthreads();
    compare_draws(r, n_draws, [&](Stream<double>& g, unsigned long long) { return normal64<CAP>(g, tab); },
                  [&](Stream<double>& g, unsigned long long) { return g.template normal<CAP>((const SmemTab<double>&)tab); });
}
template <int CAP>
__global__ void k_gamma(Result* r, unsigned long long n_draws, unsigned long long)
{
    __shared__ Tab64 tab;
    tab.fill_all();
    __syncthreads();
    const auto shape = [](unsigned long long i) { return exp2(-10.0 + 33.0 * unit(mix(i ^ 21))); };   // 10^-3 .. 8 10^6
    compare_draws(r, n_draws, [&](Stream<double>& g, unsigned long long i) { return gamma64<CAP>(g, shape(i), tab); },
                  [&](Stream<double>& g, unsigned long long i) { return gamma_mt<CAP, double>(g, shape(i), (const SmemTab<double>&)tab); });
}

}  // namespace

#define CHECK(NAME, KERNEL) \
    extern "C" int chk_##NAME(Result* out, unsigned long long a, unsigned long long b) { return run(out, KERNEL, a, b); }
CHECK(reciprocals, k_reciprocals)
CHECK(inv_sqrt, k_inv_sqrt)
CHECK(log_quotient, k_log_quotient)
CHECK(quotient_middles, k_quotient_middles)
CHECK(boost_quotient, k_boost_quotient)
CHECK(f64, k_f64)
CHECK(recip31, k_recip31)
CHECK(f64_sqrt, k_sqrt)
CHECK(open_unit, k_open_unit)
CHECK(unit, k_unit)
CHECK(search, k_search)
CHECK(search_tails, k_search_tails)
CHECK(ptrs, k_ptrs<kSamplerCap>)
CHECK(ptrs_cap, k_ptrs<1>)
CHECK(normal, k_normal<kSamplerCap>)
CHECK(normal_cap, k_normal<1>)
CHECK(gamma, k_gamma<kSamplerCap>)
CHECK(gamma_cap, k_gamma<1>)
