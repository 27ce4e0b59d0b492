// swb_f64.cuh -- Float64 arithmetic of the cell kernels.
//
// Every operation rounds as the reference's does, so results equal the
// oracle bit for bit; what changes is the unit that computes it.  GB300 has
// one Float64 result per 64 FP32 ones (a warp instruction every 64 cycles on
// each SM quarter), so Float64 kernels are bound by their count of Float64
// instructions, and 30 integer instructions are cheaper than one division.
#pragma once
#include "swb_internal.h"

namespace swb {

__device__ __forceinline__ uint32_t hi64(double v) { return (uint32_t)__double2hiint(v); }
__device__ __forceinline__ uint32_t lo64(double v) { return (uint32_t)__double2loint(v); }
__device__ __forceinline__ bool finite64(double v) { return (hi64(v) & 0x7ff00000u) != 0x7ff00000u; }

// An approximation y of 1 / b: the hardware's seed (about 2^-20) and one
// cubic step y (1 + e + e^2), e = 1 - b y, whose own error is e^3; y is then
// within about half an ulp of 1 / b.
__device__ __forceinline__ double recip64(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = __fma_rn(-b, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}

// a / b rounded to nearest from y = recip64(b): q = a y is within two ulp, and
// the integer remainder R = A 2^s - B Q of the 53-bit significands (exact
// modulo 2^64, and |R| < 2^56) says by how many ulp q is off, because q is
// the nearest iff 2 |R| < B (a quotient of doubles is never half-way between
// two doubles).  One Float64 instruction instead of about nine.  Sets `hard`
// where that does not hold: exponents near the ends of the range, a q whose
// neighbours may lie across a power of two, zero or non-finite b; the caller
// then divides.  A zero a is exact as it is.
__device__ __forceinline__ double quot64(double a, double b, double y, double nzero, bool &hard) {
    const double q = __fma_rn(a, y, nzero);
    const uint32_t ah = hi64(a), al = lo64(a), bh = hi64(b), bl = lo64(b), qh = hi64(q), ql = lo64(q);
    const uint32_t ea = (ah >> 20) & 0x7ff, eb = (bh >> 20) & 0x7ff, eq = (qh >> 20) & 0x7ff;
    const bool zero = ((ah << 1) | al) == 0;
    const uint32_t Bh = (bh & 0xfffff) | 0x100000, Qh = (qh & 0xfffff) | 0x100000;
    // s is 52 or 53, so the low word of A 2^s is zero and its high word is
    // A's low word shifted by s - 32
    const uint32_t s = (ea - eb - eq + 1023 + 20) & 31;
    const uint64_t bq = (uint64_t)bl * ql;
    const uint32_t Rh = (al << s) - (uint32_t)(bq >> 32) - Bh * ql - bl * Qh;
    const int64_t R = (int64_t)(((uint64_t)Rh << 32) - (uint32_t)bq);
    const int64_t B = (int64_t)(((uint64_t)Bh << 32) | bl);
    const int64_t T = 2 * (R < 0 ? -R : R);
    int k = (T > B ? 1 : 0) + (T > 3 * B ? 1 : 0);
    if (R < 0) k = -k;
    const bool edge = (Qh == 0x1fffffu) | ((Qh == 0x100000u) & (ql < 4u));
    const bool range = (ea - 64u < 1919u) & (eq - 64u < 1919u);
    hard |= (eb - 64u >= 1919u) | (!zero & (edge | !range));
    if (zero) k = 0;
    return __longlong_as_double(__double_as_longlong(q) + k);
}

// The general division, out of line: its expansion stays out of the kernels.
static __device__ __noinline__ double div64(double a, double b) { return a / b; }

// x^m and x^n by repeated multiplication as power_broad does
// (src/pressure.jl:363-369); n > m >= 1, so x^m is met on the way to x^n.
// 1 * x is x.
__device__ __forceinline__ void powers64(const Fma64 &f, double x, int n, int m, double &pn, double &pm) {
    if (n == 9 && m == 3) {
        const double x2 = f.mul(x, x);
        pm = f.mul(x2, x);
        double t = pm;
#pragma unroll
        for (int i = 3; i < 9; ++i) t = f.mul(t, x);
        pn = t;
    } else {
        double t = x;
        pm = x;
        for (int i = 1; i < n; ++i) {
            t = f.mul(t, x);
            if (i == m - 1) pm = t;
        }
        pn = t;
    }
}

// moments! (src/moments.jl:43-51), left to right.
__device__ __forceinline__ void moments64(const Fma64 &f, const double p[9], double &h, double &jx,
                                          double &jy) {
    // 0 + f0: f0, with -0 made +0
    double s = (hi64(p[0]) == 0x80000000u && lo64(p[0]) == 0u) ? 0.0 : p[0];
#pragma unroll
    for (int q = 1; q < 9; ++q) s = f.add(s, p[q]);
    h = s;
    jx = f.add(f.sub(f.sub(f.add(f.sub(p[1], p[3]), p[5]), p[6]), p[7]), p[8]);
    jy = f.sub(f.sub(f.add(f.add(f.sub(p[2], p[4]), p[5]), p[6]), p[7]), p[8]);
}

// u = j / h.
__device__ __forceinline__ void velocity64(const Fma64 &f, double h, double jx, double jy, double &ux,
                                           double &uy) {
    const double y = recip64(h);
    bool hard = false;
    ux = quot64(jx, h, y, f.nzero, hard);
    uy = quot64(jy, h, y, f.nzero, hard);
    if (hard) {
        ux = div64(jx, h);
        uy = div64(jy, h);
    }
}

// filmpressure! of one cell (src/pressure.jl:141-153); names as in pressure_cell.
__device__ __forceinline__ double pressure64(const Fma64 &f, double h, double ip, double jp, double im,
                                             double jm, double ipjp, double imjp, double imjm,
                                             double ipjm, double kap, double gamma, double hmin,
                                             double hcrit, int n, int m) {
    const double d = f.add(h, hcrit);
    bool hard = false;
    double x = quot64(hmin, d, recip64(d), f.nzero, hard);
    if (hard) x = div64(hmin, d);
    double pn, pm;
    powers64(f, x, n, m, pn, pm);
    const double p = f.mul(-gamma, f.mul(kap, f.sub(pn, pm)));
    const double near = f.mul(2.0 / 3.0, f.add(f.add(f.add(jp, ip), im), jm));
    const double diag = f.mul(1.0 / 6.0, f.add(f.add(f.add(ipjp, imjp), imjm), ipjm));
    const double lap = f.sub(f.add(near, diag), f.mul(10.0 / 3.0, h));
    return f.sub(p, f.mul(gamma, lap));
}

// Gradient stencil of h∇p! (src/forcing.jl:181-184).
__device__ __forceinline__ void grad64(const Fma64 &f, double ip, double jp, double im, double jm,
                                       double ipjp, double imjp, double imjm, double ipjm, double &gx,
                                       double &gy) {
    gx = f.sub(f.mul(-1.0 / 3.0, f.sub(ip, im)),
               f.mul(1.0 / 12.0, f.add(f.sub(f.sub(ipjp, imjp), imjm), ipjm)));
    gy = f.sub(f.mul(-1.0 / 3.0, f.sub(jp, jm)),
               f.mul(1.0 / 12.0, f.sub(f.sub(f.add(ipjp, imjp), imjm), ipjm)));
}

// slippage! (src/forcing.jl:43-44): (6 μ h u) / (2 h^2 + 6 δ h + 3 δ^2).
// 2 (h h) is exact, so it joins the sum in one rounding.
__device__ __forceinline__ void slippage64(const Fma64 &f, double h, double ux, double uy, double mu6,
                                           double delta6, double delta3sq, double &sx, double &sy) {
    const double den = f.add(__fma_rn(2.0, f.mul(h, h), f.mul(delta6, h)), delta3sq);
    const double mh = f.mul(mu6, h), nx = f.mul(mh, ux), ny = f.mul(mh, uy), y = recip64(den);
    bool hard = false;
    sx = quot64(nx, den, y, f.nzero, hard);
    sy = quot64(ny, den, y, f.nzero, hard);
    if (hard) {
        sx = div64(nx, den);
        sy = div64(ny, den);
    }
}

// equilibrium! (src/equilibrium.jl:67-114); g56 = 5/6 g, g15 = 1.5 g.  G0: no gravity.  Then g h is an
// exact zero for a finite h and 0 + x is x (a zero x only ever meets another
// term), so those operations are left out; a non-finite h gives NaN in every
// population either way.
template <bool G0>
__device__ __forceinline__ void feq64(const Fma64 &f, double h, double ux, double uy, double g56,
                                      double g15, double fe[9]) {
    const double hh = (!G0 || finite64(h)) ? h : __longlong_as_double(0x7ff8000000000000LL);
    const double xx = f.mul(ux, ux), yy = f.mul(uy, uy), vsq = f.add(xx, yy);
    const double v15 = f.mul(1.5, vsq), v23 = f.mul(2.0 / 3.0, vsq);
    if (G0)
        fe[0] = f.mul(hh, f.sub(1.0, v23));
    else
        fe[0] = f.mul(hh, f.sub(f.sub(1.0, f.mul(g56, hh)), v23));
    const double gh = G0 ? 0.0 : f.mul(g15, hh);
    const double s = f.add(ux, uy), d = f.sub(uy, ux);
    const double cu[4] = {ux, uy, s, d};
    const double cc[4] = {xx, yy, f.mul(s, s), f.mul(d, d)};
    // q and its opposite: 1/3, 2/4, 5/7, 6/8
    constexpr int qp[4] = {1, 2, 5, 6}, qm[4] = {3, 4, 7, 8};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double w = f.mul(k < 2 ? 1.0 / 9.0 : 1.0 / 36.0, hh);
        const double c3 = f.mul(3.0, cu[k]), c45 = f.mul(4.5, cc[k]);
        const double tp = G0 ? c3 : f.add(gh, c3), tm = G0 ? -c3 : f.sub(gh, c3);
        fe[qp[k]] = f.mul(w, f.sub(f.add(tp, c45), v15));
        fe[qm[k]] = f.mul(w, f.sub(f.add(tm, c45), v15));
    }
}

// ------------------------------------------------------------ exact sums
// A Float64 value as an integer in units of 2^-96, split into four chunks of
// 27 bits and a signed top chunk, so that a warp adds each chunk with one
// 32-bit reduction: sums of these are exact and do not depend on their order.
// Values from 2^30 on (and non-finite ones) are not held (false); bits below
// 2^-96 are dropped.
__device__ __forceinline__ bool chunks64(double v, uint32_t c[kChunks]) {
    const int e = (int)((hi64(v) >> 20) & 0x7ff) - 979;  // v = m 2^e in units of 2^-96
    if (e > 73) return false;
    const uint64_t m = e > -979 ? (__double_as_longlong(v) & 0xfffffffffffffull) | 0x10000000000000ull : 0ull;
    unsigned __int128 u = e >= 0 ? (unsigned __int128)m << e : (unsigned __int128)(e > -64 ? m >> -e : 0);
    if (hi64(v) & 0x80000000u) u = ~u + 1;
#pragma unroll
    for (int i = 0; i < kChunks - 1; ++i) c[i] = (uint32_t)(u >> (27 * i)) & 0x7ffffffu;
    c[kChunks - 1] = (uint32_t)(int32_t)((__int128)u >> 108);
    return true;
}
// The value of chunk sums (each the sum of up to 2^31 chunks).
__device__ __forceinline__ double value64(const long long c[kChunks]) {
    long long d[kChunks], carry = 0;
#pragma unroll
    for (int i = 0; i < kChunks - 1; ++i) {
        d[i] = (c[i] + carry) & 0x7ffffffLL;
        carry = (c[i] + carry) >> 27;
    }
    d[kChunks - 1] = c[kChunks - 1] + carry;
    // 127 bits hold a sum below 2^30 whole; of a larger one the lower chunks
    // are only a sticky last bit
    const bool whole = d[4] < (1 << 18) && d[4] >= -(1 << 18);
    const __int128 low = ((__int128)d[1] << 27) | d[0], mid = ((__int128)d[3] << 27) | d[2];
    const __int128 u = whole ? ((__int128)d[4] << 108) + (mid << 54) + low
                             : ((__int128)d[4] << 54) + (mid | (low ? 1 : 0));
    const double v = (double)(long long)(u >> 64) * 0x1p64 + (double)(unsigned long long)u;
    return v * (whole ? 0x1p-96 : 0x1p-42);
}

// Order-preserving keys for unsigned 64-bit maxima; 0 stands for no cell and
// for NaN, which maximum and minimum leave out.
__device__ __forceinline__ unsigned long long order64(double v) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double unorder64(unsigned long long o) {
    return __longlong_as_double((long long)((o >> 63) ? (o & 0x7fffffffffffffffull) : ~o));
}

}  // namespace swb
