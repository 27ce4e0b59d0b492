// swb_f64.cuh -- Float64 arithmetic of the cell kernels.
//
// Every operation rounds as the reference's does, so results equal the
// oracle bit for bit; what changes is the unit that computes it.  GB300 has
// one Float64 result per 64 FP32 ones: a Float64 warp instruction occupies its
// SM quarter's unit for 64 cycles or more, in which the quarter can issue some
// forty integer instructions.  So the products and the quotients, half of a
// cell's operations, are computed with integers while the Float64 unit does the
// sums (Fast64).  Measured: products alone 15 cycles per SM and
// warp, sums alone 16.5 to 19, one of each 19 together.
#pragma once
#include "swb_internal.h"

namespace swb {

__device__ __forceinline__ uint32_t hi64(double v) { return (uint32_t)__double2hiint(v); }
__device__ __forceinline__ uint32_t lo64(double v) { return (uint32_t)__double2loint(v); }
__device__ __forceinline__ bool finite64(double v) { return (hi64(v) & 0x7ff00000u) != 0x7ff00000u; }

__device__ __forceinline__ bool zero64(double v) { return ((hi64(v) & 0x7fffffffu) | lo64(v)) == 0; }
// v / 2 by its exponent, on the Float64 unit only where that is not enough (an asm
// statement, which is not computed beside the other case and then selected).
__device__ __forceinline__ double half64(double v) {
    if (((hi64(v) >> 20) & 0x7ff) - 2u <= 2044u) return __hiloint2double((int)(hi64(v) - 0x100000u), (int)lo64(v));
    asm volatile("mul.rn.f64 %0, %0, 0d3FE0000000000000;" : "+d"(v));
    return v;
}

// v, but where v / 2 is rounded (v below 2^-1021) the number twice as large as
// that, and where 2 v overflows infinity: 0.5 even64(v) + b and 2 large64(v) + b
// as one fused operation round as the two they stand for.  (Selections of a few
// integer instructions; a branch costs a warp alone on its SM quarter 20 to 70 ns.)
__device__ __forceinline__ double even64(double v) {
    const uint32_t h = hi64(v), l = lo64(v);
    const long long odd = ((h & 0x7fe00000u) == 0u && (l & 1u)) ? (long long)(int)(l & 2u) - 1 : 0;
    return __longlong_as_double(__double_as_longlong(v) + odd);
}
__device__ __forceinline__ double large64(double v) {
    const bool big = (hi64(v) & 0x7ff00000u) == 0x7fe00000u;
    return __hiloint2double((int)(big ? (hi64(v) | 0x7ff00000u) & 0xfff00000u : hi64(v)),
                            (int)(big ? 0u : lo64(v)));
}

// a b rounded to nearest, of normal numbers or (ZERO) zeros, in integers: the
// 106-bit product of the significands, its upper 62 or 63 bits with a sticky
// last bit, rounded half to even at bit 10.  Sets `bad` where an operand or
// the result is neither: the caller then computes the cell again (Plain64).
template <bool ZERO>
__device__ __forceinline__ double mul64(double a, double b, bool &bad) {
    const uint32_t ah = hi64(a), bh = hi64(b);
    // significands with their leading ones at bits 63 and 62
    const uint32_t Ah = __funnelshift_l(lo64(a), (ah & 0xfffff) | 0x100000, 11), Al = lo64(a) << 11;
    const uint32_t Bh = __funnelshift_l(lo64(b), (bh & 0xfffff) | 0x100000, 10), Bl = lo64(b) << 10;
    const uint64_t p0 = (uint64_t)Al * Bl;
    const uint64_t p1 = (uint64_t)Ah * Bl + (p0 >> 32);
    const uint64_t p2 = (uint64_t)Al * Bh + (uint32_t)p1;
    const uint64_t p = (uint64_t)Ah * Bh + (p1 >> 32) + (p2 >> 32);
    const uint32_t sticky = (uint32_t)p0 | (uint32_t)p2;
    uint32_t h = (uint32_t)(p >> 32), l = (uint32_t)p;
    const uint32_t ea = (ah >> 20) & 0x7ff, eb = (bh >> 20) & 0x7ff;
    uint32_t e = ea + eb - 1024;  // biased exponent less one
    if (h & 0x40000000u) {
        e += 1;
    } else {
        h = __funnelshift_l(l, h, 1);
        l <<= 1;
    }
    l |= sticky ? 1u : 0u;
    const uint64_t r = ((uint64_t)h << 32 | l) + (0x1ff + ((l >> 10) & 1));
    uint32_t rl = __funnelshift_r((uint32_t)r, (uint32_t)(r >> 32), 10);
    uint32_t rh = (uint32_t)(r >> 42) + (e << 20);  // the leading one adds the one e lacks
    const bool zero = ZERO && (zero64(a) || zero64(b));
    const bool off = (ea - 1u >= 2046u) | (eb - 1u >= 2046u) | (e >= 2045u);
    if (zero) rl = rh = 0;
    bad |= ZERO ? (off && !(zero && ea != 2047 && eb != 2047)) : off;
    return __hiloint2double((int)(rh | ((ah ^ bh) & 0x80000000u)), (int)rl);
}

// r ~ 2^115 / B for the 53-bit significand B of b, within 6 units: the FP32
// reciprocal (2^-22) and two Newton steps r (1 + e), e = 1 - r B, in fixed
// point, the first with e to 2^-51, the second to 2^-60.
__device__ __forceinline__ uint64_t recip64(double b) {
    const uint32_t bh = hi64(b), bl = lo64(b);
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;"
        : "=f"(y)
        : "f"(__uint_as_float(0x3f800000u | __funnelshift_l(bl, bh & 0xfffffu, 3))));
    y = fminf(y, 0x1.fffffep-1f);
    const uint32_t r0 = ((__float_as_uint(y) & 0x7fffffu) | 0x800000u) << 7;
    // B 2^11 in two words
    const uint32_t Bh = __funnelshift_l(bl, (bh & 0xfffffu) | 0x100000u, 11), Bl = bl << 11;
    const int64_t e = (int64_t)(0x4000000000000000ull - (uint64_t)r0 * Bh - __umulhi(r0, Bl));
    const int64_t r1 = (int64_t)((uint64_t)r0 << 32) + (((int64_t)(int32_t)r0 * (int32_t)(e >> 11)) >> 19);
    const uint32_t rh = (uint32_t)(r1 >> 32), rl = (uint32_t)r1;
    const int32_t e1 = -(int32_t)(rh * Bh + __umulhi(rh, Bl) + __umulhi(rl, Bh));
    return (uint64_t)(r1 + (((int64_t)(int32_t)rh * e1) >> 30));
}

// a / b rounded to nearest from r = recip64(b): Q = A r / 2^115, rounded to 53
// bits, is within 0.52 of the quotient of the significands, and the integer
// remainder R = A 2^s - B Q (exact modulo 2^64) says whether it is the nearest:
// that is so iff 2 |R| < B, because a quotient of doubles is never half-way
// between two doubles.  No Float64 instruction instead of about nine.  Sets
// `bad` where that does not hold: operands or a quotient that are not normal,
// a Q at the bottom of a binade with a smaller quotient (the doubles below lie
// closer).  A zero a is exact.
__device__ __forceinline__ double quot64(double a, double b, uint64_t r, bool &bad) {
    const uint32_t ah = hi64(a), al = lo64(a), bh = hi64(b), bl = lo64(b);
    const uint32_t Ah = __funnelshift_l(al, (ah & 0xfffffu) | 0x100000u, 11), Al = al << 11;
    const uint32_t rh = (uint32_t)(r >> 32), rl = (uint32_t)r;
    const uint64_t m1 = (uint64_t)Ah * rl, m2 = (uint64_t)Al * rh;
    uint64_t q = (uint64_t)Ah * rh + (m1 >> 32) + (m2 >> 32);  // A / B 2^62, within 9
    const uint32_t ea = (ah >> 20) & 0x7ff, eb = (bh >> 20) & 0x7ff;
    const bool up = (uint32_t)(q >> 32) >= 0x40000000u;  // A >= B
    const uint32_t e = ea - eb + (up ? 1022 : 1021);     // biased exponent less one
    if (!up) q += q;
    q = (q + 512) >> 10;
    const uint32_t Qh = (uint32_t)(q >> 32), Ql = (uint32_t)q, Bh = (bh & 0xfffffu) | 0x100000u;
    // s is 52 or 53: the low word of A 2^s is zero, its high word A's low
    // word shifted by s - 32
    const uint64_t bq = (uint64_t)bl * Ql;
    const uint32_t Rh = (al << (up ? 20 : 21)) - (uint32_t)(bq >> 32) - Bh * Ql - bl * Qh;
    const int64_t R = (int64_t)(((uint64_t)Rh << 32) - (uint32_t)bq);
    const int64_t B = (int64_t)(((uint64_t)Bh << 32) | bl);
    const int k = (2 * R > B ? 1 : 0) - (2 * R < -B ? 1 : 0);
    const bool zero = zero64(a);
    bad |= (eb - 1u >= 2046u) |
           (!zero & ((ea - 1u >= 2046u) | (e >= 2045u) | ((Qh == 0x100000u) & (Ql < 2u) & (R < 0))));
    const uint64_t v = zero ? 0 : q + ((uint64_t)e << 52) + (int64_t)k;
    return __longlong_as_double((long long)(v | ((uint64_t)((ah ^ bh) & 0x80000000u) << 32)));
}

// The operations of a cell.  mul: operands that may be zero; muln: operands
// that are not (a zero is then computed again); twice_plus: 2 a + b, rounded
// once either way because 2 a is exact (or, beyond large64, infinite).
struct Fast64 {
    Fma64 f;
    bool bad;
    __device__ __forceinline__ explicit Fast64(const Fma64 &g) : f(g.in_registers()), bad(false) {}
    __device__ __forceinline__ double add(double a, double b) const { return f.add(a, b); }
    __device__ __forceinline__ double sub(double a, double b) const { return f.sub(a, b); }
    __device__ __forceinline__ double mul(double a, double b) { return mul64<true>(a, b, bad); }
    __device__ __forceinline__ double muln(double a, double b) { return mul64<false>(a, b, bad); }
    __device__ __forceinline__ double twice_plus(double a, double b) const { return __fma_rn(2.0, a, b); }
    __device__ __forceinline__ uint64_t recip(double b) const { return recip64(b); }
    __device__ __forceinline__ double quot(double a, double b, uint64_t r) { return quot64(a, b, r, bad); }
};
struct Plain64 {
    __device__ __forceinline__ double add(double a, double b) const { return a + b; }
    __device__ __forceinline__ double sub(double a, double b) const { return a - b; }
    __device__ __forceinline__ double mul(double a, double b) const { return a * b; }
    __device__ __forceinline__ double muln(double a, double b) const { return a * b; }
    __device__ __forceinline__ double twice_plus(double a, double b) const { return 2.0 * a + b; }
    __device__ __forceinline__ uint64_t recip(double) const { return 0; }
    __device__ __forceinline__ double quot(double a, double b, uint64_t) const { return a / b; }
};

// x^m and x^n by repeated multiplication as power_broad does
// (src/pressure.jl:363-369); n > m >= 1, so x^m is met on the way to x^n.
// 1 * x is x.
template <class O>
__device__ __forceinline__ void powers64(O &o, double x, int n, int m, double &pn, double &pm) {
    if (n == 9 && m == 3) {
        const double x2 = o.muln(x, x);
        pm = o.muln(x2, x);
        double t = pm;
#pragma unroll
        for (int i = 3; i < 9; ++i) t = o.muln(t, x);
        pn = t;
    } else {
        double t = x;
        pm = x;
#pragma unroll 1
        for (int i = 1; i < n; ++i) {
            t = o.muln(t, x);
            if (i == m - 1) pm = t;
        }
        pn = t;
    }
}

// moments! (src/moments.jl:43-51), left to right: h and the momenta.
template <class O>
__device__ __forceinline__ void moments64(O &o, const double p[9], double &h, double &jx, double &jy) {
    // 0 + f0: f0, with -0 made +0
    double s = (hi64(p[0]) == 0x80000000u && lo64(p[0]) == 0u) ? 0.0 : p[0];
#pragma unroll
    for (int q = 1; q < 9; ++q) s = o.add(s, p[q]);
    h = s;
    jx = o.add(o.sub(o.sub(o.add(o.sub(p[1], p[3]), p[5]), p[6]), p[7]), p[8]);
    jy = o.sub(o.sub(o.add(o.add(o.sub(p[2], p[4]), p[5]), p[6]), p[7]), p[8]);
}

// The neighbours of a cell, named as in the reference: ip = v[i-1, j],
// jp = v[i, j-1], im = v[i+1, j], jm = v[i, j+1], ...
struct Near64 {
    double ip, jp, im, jm, ipjp, imjp, imjm, ipjm;
};

// filmpressure! of one cell (src/pressure.jl:141-153).
template <class O>
__device__ __forceinline__ double pressure64(O &o, double h, const Near64 &v, double kap, double gamma,
                                             double hmin, double hcrit, int n, int m) {
    const double d = o.add(h, hcrit);
    const double x = o.quot(hmin, d, o.recip(d));
    double pn, pm;
    powers64(o, x, n, m, pn, pm);
    const double p = o.mul(-gamma, o.mul(kap, o.sub(pn, pm)));
    const double near = o.muln(2.0 / 3.0, o.add(o.add(o.add(v.jp, v.ip), v.im), v.jm));
    const double diag = o.muln(1.0 / 6.0, o.add(o.add(o.add(v.ipjp, v.imjp), v.imjm), v.ipjm));
    const double lap = o.sub(o.add(near, diag), o.muln(10.0 / 3.0, h));
    return o.sub(p, o.mul(gamma, lap));
}

// Gradient stencil of h∇p! (src/forcing.jl:181-184).
template <class O>
__device__ __forceinline__ void grad64(O &o, const Near64 &v, double &gx, double &gy) {
    gx = o.sub(o.mul(-1.0 / 3.0, o.sub(v.ip, v.im)),
               o.mul(1.0 / 12.0, o.add(o.sub(o.sub(v.ipjp, v.imjp), v.imjm), v.ipjm)));
    gy = o.sub(o.mul(-1.0 / 3.0, o.sub(v.jp, v.jm)),
               o.mul(1.0 / 12.0, o.sub(o.sub(o.add(v.ipjp, v.imjp), v.imjm), v.ipjm)));
}

// slippage! (src/forcing.jl:43-44): (6 μ h u) / (2 h^2 + 6 δ h + 3 δ^2).
template <class O>
__device__ __forceinline__ void slip64(O &o, double h, double ux, double uy, double mu6, double delta6,
                                       double delta3sq, double &sx, double &sy) {
    const double den = o.add(o.twice_plus(o.muln(h, h), o.mul(delta6, h)), delta3sq);
    const uint64_t r = o.recip(den);
    const double mh = o.mul(mu6, h);
    sx = o.quot(o.mul(mh, ux), den, r);
    sy = o.quot(o.mul(mh, uy), den, r);
}

// equilibrium! (src/equilibrium.jl:67-114); g56 = 5/6 g, g15 = 1.5 g.  G0: no
// gravity.  Then g h is an exact zero for a finite h and 0 + x is x (a zero x
// only ever meets another term), so those operations are left out; a
// non-finite h gives NaN in every population either way.
template <bool G0, class O>
__device__ __forceinline__ void feq64(O &o, double h, double ux, double uy, double g56, double g15,
                                      double fe[9]) {
    const double hh = (!G0 || finite64(h)) ? h : __longlong_as_double(0x7ff8000000000000LL);
    const double xx = o.mul(ux, ux), yy = o.mul(uy, uy), vsq = o.add(xx, yy);
    const double v15 = o.mul(1.5, vsq), v23 = o.mul(2.0 / 3.0, vsq);
    if (G0)
        fe[0] = o.muln(hh, o.sub(1.0, v23));
    else
        fe[0] = o.muln(hh, o.sub(o.sub(1.0, o.mul(g56, hh)), v23));
    const double gh = G0 ? 0.0 : o.mul(g15, hh);
    const double s = o.add(ux, uy), d = o.sub(uy, ux);
    const double cu[4] = {ux, uy, s, d};
    const double cc[4] = {xx, yy, o.mul(s, s), o.mul(d, d)};
    // q and its opposite: 1/3, 2/4, 5/7, 6/8
    constexpr int qp[4] = {1, 2, 5, 6}, qm[4] = {3, 4, 7, 8};
    const double w[2] = {o.muln(1.0 / 9.0, hh), o.muln(1.0 / 36.0, hh)};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double c3 = o.mul(3.0, cu[k]), c45 = o.mul(4.5, cc[k]);
        const double tp = G0 ? c3 : o.add(gh, c3), tm = G0 ? -c3 : o.sub(gh, c3);
        fe[qp[k]] = o.mul(w[k / 2], o.sub(o.add(tp, c45), v15));
        fe[qm[k]] = o.mul(w[k / 2], o.sub(o.add(tm, c45), v15));
    }
}

// BGKandStream!'s collision (src/collide.jl:76-89): relaxation towards fe and
// the sources of the force; fq (the streamed populations) only for τ != 1.
template <bool TAU1, class O>
__device__ __forceinline__ void relax64(O &o, const double fe[9], const double fq[9], double omeg,
                                        double invtau, double Fx, double Fy, double out[9]) {
    const double S[4] = {o.mul(1.0 / 3.0, Fx), o.mul(1.0 / 3.0, Fy), o.mul(1.0 / 24.0, o.add(Fx, Fy)),
                         o.mul(1.0 / 24.0, o.sub(Fy, Fx))};
    constexpr int qp[4] = {1, 2, 5, 6}, qm[4] = {3, 4, 7, 8};
#pragma unroll
    for (int q = 0; q < 9; ++q) out[q] = TAU1 ? fe[q] : o.add(o.mul(omeg, fq[q]), o.mul(invtau, fe[q]));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        out[qp[k]] = o.add(out[qp[k]], S[k]);
        out[qm[k]] = o.sub(out[qm[k]], S[k]);
    }
}

// ------------------------------------------------------------ exact sums
// A Float64 value as an integer in units of 2^-96, split into four chunks of
// 27 bits and a signed top chunk, so that a warp adds each chunk with one
// 32-bit reduction: sums of these are exact and do not depend on their order.
// Held are zeros and values from 2^-44 (whose last bit is 2^-96) up to 2^30;
// of others the result is false.
__device__ __forceinline__ bool chunks64(double v, uint32_t c[kChunks]) {
    const int e = (int)((hi64(v) >> 20) & 0x7ff) - 979;  // v = m 2^e in units of 2^-96
    const bool in = (uint32_t)e <= 73u;
    if (!in && !zero64(v)) return false;
    const uint64_t m = (__double_as_longlong(v) & 0xfffffffffffffull) | 0x10000000000000ull;
    unsigned __int128 u = in ? (unsigned __int128)m << e : (unsigned __int128)0;
    if (hi64(v) & 0x80000000u) u = ~u + 1;
#pragma unroll
    for (int i = 0; i < kChunks - 1; ++i) c[i] = (uint32_t)(u >> (27 * i)) & 0x7ffffffu;
    c[kChunks - 1] = (uint32_t)(int32_t)((__int128)u >> 108);
    return true;
}
// An integer as a double, rounded once.
__device__ __forceinline__ double round128(__int128 u) {
    const unsigned __int128 m = u < 0 ? -(unsigned __int128)u : (unsigned __int128)u;
    const uint64_t h = (uint64_t)(m >> 64), l = (uint64_t)m;
    double v = (double)l;
    if (h) {  // the upper 64 bits, the last one sticky
        const int s = 64 - __clzll((long long)h);
        v = (double)((uint64_t)(m >> s) | ((m & (((unsigned __int128)1 << s) - 1)) ? 1u : 0u));
        v *= __longlong_as_double((long long)(1023 + s) << 52);
    }
    return u < 0 ? -v : v;
}
// The value of chunk sums (each the sum of up to 2^31 chunks), rounded once.
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
    return round128(u) * (whole ? 0x1p-96 : 0x1p-42);
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
