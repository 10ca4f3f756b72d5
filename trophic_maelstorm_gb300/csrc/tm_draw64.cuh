// tm_draw64.cuh -- the FP64 draws whose decisions are taken in FP32 where an error bound
// allows (tm_step64.cu says why): the Poisson search, the transformed rejection, the
// ziggurat's wedge and the two tests of the Gamma draw.  Each gives the bits of the FP64
// method in tm_device.cuh from the same stream; the tests compare the two on the GPU.
#pragma once
#include "tm_device.cuh"

namespace tmg {

constexpr int kSearch = 96;                 // terms of the FP32 Poisson search (multiple of 4)

struct Tab64 : SmemTab<double> {
    __align__(16) float rcpf[kSearch + 8];  // rcpf[3 + n] = 1/n: the search reads n = 4 i + 1 .. 4 i + 4 at once
    __device__ __forceinline__ void fill_all()
    {
        fill();
        for (int i = threadIdx.x; i < kSearch + 8; i += blockDim.x) rcpf[i] = i > 3 ? 1.0f / (float)(i - 3) : 0.0f;
    }
};

// h w of a ziggurat value h (below 2^24) and its layer's width, rounded once
__device__ __forceinline__ double signed_mul(int32_t h, double w)
{
    return tmf::with_sign(tmf::from_u31((uint32_t)(h < 0 ? -h : h)), h < 0) * w;
}

__device__ __forceinline__ uint32_t hi32(double x) { return (uint32_t)__double2hiint(x); }

// Upper bound of |FP32 search's tail - FP64 search's tail| for a mean below 32.
// The rounding of m (relative 2^-23) moves a tail by at most m 2^-23 max p <= 0.4
// m 2^-23; a term p_i carries 3 i + 4 roundings, which sum to (3 m + 4) 2^-24, and the
// differences q - p another m 2^-24: (4 m + 8) 2^-24 in all.  The largest
// difference seen over 2.7 10^8 means is 0.22 of this bound; 0.02 % of the searches with
// means up to 32 are left to FP64.
__device__ __forceinline__ float search_eps(float m) { return (m + 4.0f) * 0x1p-22f; }

// Poisson count for the mean m < 32 and the 32-bit uniform w of the lanes with
// `need`, by the search of poisson_exact in FP32; -1 where a tail lies within the
// bound of u.  The whole warp runs it: lanes that leave a search loop one by one
// would drag the rest of the draw through the pipe in pieces.
__device__ __forceinline__ int search_count(bool need, float m, uint32_t w, const float* rcp)
{
    const float eps = search_eps(m);
    const float u = (float)w * 0x1p-32f;
    const float up = u + eps, dn = u - eps;
    float p = tm_exp_neg_small(-m);
    float q = (m < 0.25f) ? tm_negexpm1(m) : 1.0f - p;
    bool run = need && up < q;
    int n = q <= dn ? 0 : -1;
    for (int it = 0; it < kSearch && __any_sync(0xffffffffu, run); it += 4) {
        // four terms per trip; the tails only decrease, so those certainly above u form a prefix
        const float4 r4 = *reinterpret_cast<const float4*>(rcp + it + 1);
        const float p1 = (p * m) * r4.x, q1 = q - p1;
        const float p2 = (p1 * m) * r4.y, q2 = q1 - p2;
        const float p3 = (p2 * m) * r4.z, q3 = q2 - p3;
        p = (p3 * m) * r4.w;
        q = q3 - p;
        const bool a1 = up < q1, a2 = up < q2, a3 = up < q3;
        const float first = a2 ? (a3 ? q : q3) : (a1 ? q2 : q1);     // the first tail not certainly above u
        const int c = a2 ? (a3 ? 4 : 3) : (a1 ? 2 : 1);
        if (run && !(up < q)) {
            n = first <= dn ? it + c : -1;
            run = false;
        }
    }
    return run ? -1 : n;
}

// FP32 value of the uniform that Stream<double>::open forms of two words, (x + 1/2) 2^-53
// with x the 53 leading bits: within 2^-23 relative, whatever the words (the roundings of
// w1 and of the sum; the low part is exact).
__device__ __forceinline__ float unit_f32(uint32_t w1, uint32_t w2)
{
    return fmaf((float)w1, 0x1p-32f, ((float)(w2 >> 11) + 0.5f) * 0x1p-53f);
}

// poisson_exact for m >= 32 (PTRS) with its floor and its tests decided in FP32 where the
// error bounds allow: the candidate k is taken when the FP32 value lies further from a
// whole number than its error, a comparison when the two sides differ by more than theirs.
// Anything closer runs the FP64 method from the same counter; beyond 4096 that would be
// most draws.  The FP64 method is six divisions, a root and up to six logs on a pipe that
// takes a warp instruction every 64 cycles: with it the list of general draws was 30 % of
// the whole kernel on a Rietkerk run (means up to 100); 16 lattices of 256^2, 20 steps:
// 9.24 ms before, 8.79 ms with this.
//
// The errors, in units of e = 2^-24 (one rounding); a log's is |log| + 3:
//   mf 1 m;  slam 1.5 slam;  b 4.5 b;  a 9 a (its terms cancel by 1.19 at b = 15);
//   us 2 us (unit_f32), U 2;  2 a / us 12, scale 13 scale;  scale U 9 scale (|U| <= 1/2)
//   x: 9 scale + m, and the two sums' scale + 2 m + 1: 10 scale + 3 m + 1, where err is
//     16 scale + 32 m + 32 (so us below 2^-19, where scale passes 2^19, is never sure)
//   us and V against 0.07, vr and 0.013: 2 of each and 30 for vr (3.6 / (b - 2) at b = 15),
//     where the bands are 1e-4, 1e-5 and 1e-6, 16 at least
//   lhs: log V 2 + |log V| + 3;  loginvalpha 7;  log(a / us^2 + b) 17 + |log| + 3;  the two
//     sums |lhs| each: below 33 + 3 |lhs|, as |log V| and the last log add up to |lhs| + 0.2
//   rhs, k < 16: k (log m + 4) + 4 (k log m + m + log k!): below 60 + 5 size
//   rhs, else: an error of m or d moves d - k log1p(d/m) by itself times |k - m|/m or 1/z
//     only; the quotient |d|, the log1p 15 |kl| (below -0.29 and above 0.41: the rounding
//     of 1 + x and the log's, where |l| > 0.34; else 4 |kl|), the product and the sums |kl| +
//     2 |d| + |log z| + 4, the dropped term of corr 6e-10: below 16 |kl| + 3 |d| + 20
//   tol is 32 (size + m/4 + |lhs| + 16) + 67: twice their sum or more.
template <int CAP>
__device__ __forceinline__ double ptrs64(Stream<double>& g, double m, const Tab64& tb)
{
    if (m < 4096.0) {
        const Stream<double> at = g;             // where the FP64 method would start
        const float mf = (float)m;
        const float slam = sqrtf(mf), loglam = tm_log_pos(mf);
        const float b = 0.931f + 2.53f * slam, a = -0.059f + 0.02483f * b;
        const float invalpha = 1.1239f + 1.1328f / (b - 3.4f), vr = 0.9277f - 3.6224f / (b - 2.0f);
        const float loginvalpha = tm_log_pos(invalpha);
        bool sure = true;
        for (int it = 0; it < CAP; ++it) {
            const uint32_t u1 = g.u32(), u2 = g.u32(), v1 = g.u32(), v2 = g.u32();
            // U = open() - 0.5 by its distance from the nearer end: us = 0.5 - |U|
            const bool low = u1 < 0x80000000u;
            const float us = low ? unit_f32(u1, u2) : unit_f32(~u1, ~u2);
            const float U = low ? us - 0.5f : 0.5f - us;
            const float V = unit_f32(v1, v2);
            const float scale = 2.0f * a / us + b, x = scale * U + mf + 0.43f;
            const float err = 0x1p-20f * (scale + 2.0f * mf + 2.0f);
            const float kf = floorf(x);
            if (!(x - kf >= err && kf + 1.0f - x >= err)) { sure = false; break; }
            const double k = (double)kf;
            if (us >= 0.0701f && V <= vr - 1e-4f) return k;
            const bool maybe_fast = us >= 0.0699f && V <= vr + 1e-4f;
            if (kf < 0.0f) {
                if (maybe_fast) { sure = false; break; }
                continue;
            }
            if (maybe_fast || fabsf(us - 0.013f) < 1e-5f || (us < 0.013f && fabsf(V - us) < 1e-6f)) { sure = false; break; }
            if (us < 0.013f && V > us) continue;
            const float lhs = (tm_log_pos(V) + loginvalpha) - tm_log_pos(a / (us * us) + b);
            float rhs, size;
            if (kf < 16.0f) {
                const float lf = (float)logfact_small((int)kf);
                rhs = (kf * loglam - mf) - lf;
                size = kf * loglam + mf + lf;
            } else {
                const float z = kf + 1.0f, d = z - mf, iz = 1.0f / z;
                const float corr = iz * ((1.0f / 12.0f) - (iz * iz) * (1.0f / 360.0f));
                const float l = tm_log1p(d / mf), kl = kf * l;
                rhs = ((d - kl) - 0.5f * tm_log_pos(z)) - (0.9189385f + corr);
                size = fabsf(d) + fabsf(kl) + 8.0f;
            }
            const float gap = rhs - lhs, tol = 0x1p-19f * (size + 4.0f * mf * 0x1p-4f + fabsf(lhs) + 16.0f) + 4e-6f;
            if (gap > tol) return k;
            if (gap < -tol) continue;
            sure = false;
            break;
        }
        if (sure) {
            g.status |= TM_STATUS_CAP_BIT;
            return floor(m);
        }
        g = at;
    }
    return poisson_exact<CAP>(g, m, (const SmemTab<double>&)tb);
}

// Stream<double>::normal with the wedge test decided in FP32 where its error
// (below 2^-20 on values up to 1) allows.
template <int CAP>
__device__ __forceinline__ double normal64(Stream<double>& g, const Tab64& tb)
{
    for (int it = 0; it < CAP; ++it) {
        const uint32_t w = g.u32();
        const int iz = zig_layer(w);
        const int32_t hz = zig_value(w);
        const uint32_t az = (uint32_t)(hz < 0 ? -hz : hz);
        const ZigLayer<double> zl = tb.zig[iz];
        const double x = signed_mul(hz, zl.w);
        if (az < zl.k) return x;
        if (iz == 0) {
            for (int jt = 0; jt < CAP; ++jt) {
                const double xt = -tm_log_pos(g.open()) * (1.0 / kZigR);
                const double yt = -tm_log_pos(g.open());
                if (yt + yt >= xt * xt) {
                    const double r = kZigR + xt;
                    return hz < 0 ? -r : r;
                }
            }
            break;
        }
        const double fb = tb.zf[iz], ft = tb.zf[iz + 1];
        const double u = g.open();
        const float xf = (float)x;
        const float lhs = (float)fb + (float)u * ((float)ft - (float)fb);
        const float diff = tm_exp(-0.5f * (xf * xf)) - lhs;
        if (diff > 0x1p-18f) return x;
        if (diff < -0x1p-18f) continue;
        if (fb + u * (ft - fb) < tm_exp(-0.5 * (x * x))) return x;
    }
    g.status |= TM_STATUS_CAP_BIT;
    return 0.0;
}

// gamma_mt with its two acceptance tests decided in FP32 where their error bounds
// allow.
template <int CAP>
__device__ __forceinline__ double gamma64(Stream<double>& g, double k, const Tab64& tb)
{
    if (!(k > 0.0)) return 0.0;
    const double kk = (k < 1.0) ? k + 1.0 : k;
    const double d = kk - 1.0 / 3.0;
    const double c = Tr<double>::inv_sqrt(9.0 * d);
    double res = kk;
    bool done = false;
    for (int it = 0; it < CAP && !done; ++it) {
        double x = 0.0, v = 0.0;
        bool ok = false;
        for (int jt = 0; jt < CAP; ++jt) {
            x = normal64<CAP>(g, tb);
            v = 1.0 + c * x;
            if (v > 0.0) { ok = true; break; }
        }
        if (!ok) break;
        const double mm = (v < 1.0) ? v : 1.0;
        v = (v * v) * v;
        const double u = g.open();
        const float xf = (float)x, df = (float)d, vf = (float)v, uf = (float)u;
        const float x2f = xf * xf;
        if (vf > 1e-30f && uf < 0.999f && df < 1e6f) {
            // squeeze: relative error of either side below 2^-20 (1 - u from u < 0.999: 2^-14)
            const float lhs = (1.0f - uf) * ((108.0f * df) * (float)mm), rhs = x2f * x2f;
            if (lhs > rhs * 1.001f) { res = d * v; done = true; break; }
            // log test: absolute error below the margin
            const float lu = tm_log_pos(uf), lv = tm_log_pos(vf);
            const float margin = 0x1p-18f * ((2.0f + fabsf(lu)) + x2f + df * ((1.0f + vf) + fabsf(lv)));
            const float gap = (0.5f * x2f + df * ((1.0f - vf) + lv)) - lu;
            if (lhs < rhs * 0.999f) {
                if (gap > margin) { res = d * v; done = true; break; }
                if (gap < -margin) continue;
            } else if (gap > margin) {      // either test accepts
                res = d * v; done = true; break;
            }
        }
        const double x2 = x * x;
        if ((1.0 - u) * ((108.0 * d) * mm) > x2 * x2) { res = d * v; done = true; break; }
        if (tm_log_pos(u) < 0.5 * x2 + d * ((1.0 - v) + tm_log(v))) { res = d * v; done = true; break; }
    }
    if (!done) g.status |= TM_STATUS_CAP_BIT;
    if (k < 1.0) {
        const double u = g.open();
        res = res * tm_exp(tmf::div(tm_log_pos(u), k));
    }
    return res;
}

}  // namespace tmg
