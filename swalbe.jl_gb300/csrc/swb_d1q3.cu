// swb_d1q3.cu -- the one-dimensional thin-film solver (D1Q3), GPU side.
//
// One iteration is the reference's 1D time loop body (src/simulate.jl:98-179):
//   filmpressure!  p = -γ κ (x^n - x^m) - γ (h[i-1] - 2h + h[i+1])   (src/pressure.jl:231-256)
//   h∇p!           h (-1/2) (p[i-1] - p[i+1])                       (src/forcing.jl:189-198)
//   slippage!      6μ h u / (2h^2 + 6δh + 3δ^2)                      (src/forcing.jl:68-71)
//   force          F = -h∇p - slip (- ∇γ with a γ field, src/simulate.jl:548)
//   equilibrium!   D1Q3 feq                                          (src/equilibrium.jl:169-181)
//   BGKandStream!  collision + streaming f1 -> i+1, f2 -> i-1          (src/collide.jl:179-201)
//   moments!       h = f0 + f1 + f2, u = (f1 - f2) / h                (src/moments.jl:54-62)
// in the reference's operation order (this unit is compiled with
// --fmad=false), so Float64 results equal the oracle's bit for bit, at the ends
// of the exponent range and for heights that are not finite as well.
//
// An SM's Float64 units take about 2 us for a Float64 iteration of 128 cells,
// whatever else is done, so the cells of a lattice are spread over the SMs: a CTA
// of 64 or 128 cells, one or two threads each, runs K iterations in registers
// and shared memory on its own cells and a halo of 3 K cells on either side (an
// iteration reaches 3 cells: pressure, force, streaming), recomputing the halo
// instead of exchanging it, and writes its own cells to the other set of
// buffers.  (One CTA for a whole lattice took 26.8 us per Float64 iteration of
// 1024 cells; this takes 1.62, with records 1.95.)  No CTA waits for another, and a launch is paid
// once per K iterations.  Lattices of at most that many cells fit one CTA with
// no halo.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "swb_f64.cuh"
#include "swb_lattice.h"
#include "swb_step_impl.cuh"

namespace swb {

// Cells of a CTA, halo included: kD1Cells, or half as many where that spreads a
// Float64 lattice over more SMs (one warp per SM quarter, see D1Ops64).
constexpr int kD1Cells = 128;

struct D1Args {
    int L;
    int n, m;
    double gamma, hmin, hcrit, delta, mu, g, kap, omeg, invtau;
    void *f[2], *h[2], *u[2];  // streamed populations (the reference's fout, 3 planes of L) and fields,
                               // read from one set and written to the other by every launch
    void *p;                   // pressure of the last iteration
    const void *kapF;          // θ field: κ per cell (or null)
    const void *gamF;          // γ field (or null)
    const void *dgF;           // ∇γ of the γ field (or null)
    Record *rec;               // per-iteration measures (ring of rec_cap, or null)
    int rec_cap;
    int chunk0, chunks;        // this lattice's entries of the chunk table
    int *nan_flag;
};

// The cells [x0, x0 + w) of a lattice, owned by one CTA.
struct D1Chunk {
    int lattice, x0, w;
};

// Measures of one warp's own cells at the start of one iteration.
struct D1Part {
    uint32_t mass[kChunks], wet;
    unsigned long long kmax, kmin;
    double big;
};

namespace {

// A cell's constants, and its slippage and equilibrium.
template <class R>
struct D1Cell {
    R kap, gam, dg;  // κ, surface tension and ∇γ of the cell
    R mu6, delta6, delta3sq, omeg, invtau, g, g25, g50;
    bool grad, tau1;
};
template <class R>
struct D1Mid {
    R slip, half, fe[3];  // slippage, h / 2, equilibrium
};

// One cell's operations, Float64: rounded as the reference's.  With g = 0 and
// τ = 1 the products with 0 are left out, which are zeros unless a factor is not
// finite: such cells are computed again with Plain64, which leaves nothing out.
template <class O>
struct D1Cell64 {
    static constexpr bool kPlain = std::is_same<O, Plain64>::value;
    O o;
    __device__ __forceinline__ static double or_nan(double v, double factor) {
        return finite64(factor) ? v : __longlong_as_double(0x7ff8000000000000LL);
    }
    __device__ __forceinline__ double quot(double a, double b) { return o.quot(a, b, o.recip(b)); }
    __device__ __forceinline__ double pressure(const D1Args &a, const D1Cell<double> &c, double h, double hip,
                                               double him) {
        double pn, pm;
        powers64(o, quot(a.hmin, o.add(h, a.hcrit)), a.n, a.m, pn, pm);
        const double p = o.mul(-c.gam, o.mul(c.kap, o.sub(pn, pm)));
        return o.sub(p, o.mul(c.gam, o.add(o.twice_plus(large64(-h), hip), him)));
    }
    // slippage and equilibrium, which need only the cell's own fields
    __device__ __forceinline__ void local(const D1Cell<double> &c, double h, double u, const double fo[3],
                                          D1Mid<double> &m) {
        const double den = o.add(o.twice_plus(large64(o.muln(h, h)), o.mul(c.delta6, h)), c.delta3sq);
        m.slip = quot(o.mul(o.mul(c.mu6, h), u), den);
        m.half = half64(h);
        const double uu = o.mul(u, u), u2 = half64(u), uu2 = half64(uu);
        if (c.g == 0.0 && !kPlain) {
            m.fe[0] = o.muln(h, o.sub(1.0, uu));
            m.fe[1] = o.mul(h, o.add(u2, uu2));
            m.fe[2] = o.mul(h, o.sub(uu2, u2));
        } else {
            const double gh = o.muln(c.g25, h);
            m.fe[0] = o.muln(h, o.sub(o.sub(1.0, o.muln(c.g50, h)), uu));
            m.fe[1] = o.mul(h, o.add(o.add(gh, u2), uu2));
            m.fe[2] = o.mul(h, o.add(o.sub(gh, u2), uu2));
        }
        if (c.tau1 && kPlain)  // 0 fo
#pragma unroll
            for (int q = 0; q < 3; ++q) m.fe[q] = or_nan(m.fe[q], fo[q]);
    }
    __device__ __forceinline__ void second(const D1Cell<double> &c, const D1Mid<double> &m, double pm, double pp,
                                           const double fo[3], double out[3]) {
        double F = o.sub(o.mul(m.half, o.sub(pm, pp)), m.slip);
        if (c.grad) F = o.sub(F, c.dg);
        double fe[3] = {m.fe[0], m.fe[1], m.fe[2]};
        if (!c.tau1)
#pragma unroll
            for (int q = 0; q < 3; ++q) fe[q] = o.add(o.mul(c.omeg, fo[q]), o.mul(c.invtau, fe[q]));
        F = even64(F);
        out[0] = fe[0];
        out[1] = __fma_rn(0.5, F, fe[1]);
        out[2] = __fma_rn(-0.5, F, fe[2]);
    }
    __device__ __forceinline__ void moments(const double f[3], double &h, double &u) {
        h = o.add(o.add(f[0], f[1]), f[2]);
        u = quot(o.sub(f[1], f[2]), h);
    }
};
// The parts of an iteration with the integer unit's help, each computed again
// out of line where that met a number it does not hold.
__device__ __noinline__ double d1_pressure_again(const D1Args &a, const D1Cell<double> &c, double h, double hip,
                                                 double him) {
    return D1Cell64<Plain64>{}.pressure(a, c, h, hip, him);
}
__device__ __noinline__ void d1_local_again(const D1Cell<double> &c, double h, double u, const double *fo,
                                            D1Mid<double> *m) {
    D1Cell64<Plain64>{}.local(c, h, u, fo, *m);
}
__device__ __noinline__ void d1_second_again(const D1Cell<double> &c, const D1Mid<double> &m, double pm, double pp,
                                             const double *fo, double *out) {
    D1Cell64<Plain64>{}.second(c, m, pm, pp, fo, out);
}
__device__ __noinline__ void d1_moments_again(const double *f, double *h, double *u) {
    D1Cell64<Plain64>{}.moments(f, *h, *u);
}
// Products in integers (Fast64), or with FAST = D1Direct64 on the Float64 unit:
// alone on an SM quarter a warp waits 64 cycles for a Float64 product and 113
// for one in integers (64 cells per CTA: 1.75 and 2.34 us per iteration; 128
// cells, two warps per quarter: 2.6 either way).
struct D1Direct64 : Fast64 {
    using Fast64::Fast64;
    __device__ __forceinline__ double mul(double a, double b) const { return a * b; }
    __device__ __forceinline__ double muln(double a, double b) const { return a * b; }
};
template <class FAST>
struct D1Ops64 {
    Fma64 f;
    __device__ __forceinline__ double pressure(const D1Args &a, const D1Cell<double> &c, double h, double hip,
                                               double him) const {
        D1Cell64<FAST> k{FAST(f)};
        const double p = k.pressure(a, c, h, hip, him);
        if (!k.o.bad) return p;
        const D1Cell<double> cc = c;
        return d1_pressure_again(a, cc, h, hip, him);
    }
    // odd: the height or a population is not finite
    __device__ __forceinline__ void local(const D1Cell<double> &c, double h, double u, const double fo[3], bool odd,
                                          D1Mid<double> &m) const {
        D1Cell64<FAST> k{FAST(f)};
        k.local(c, h, u, fo, m);
        if (k.o.bad | odd) {
            const D1Cell<double> cc = c;
            const double in[3] = {fo[0], fo[1], fo[2]};
            D1Mid<double> again;
            d1_local_again(cc, h, u, in, &again);
            m = again;
        }
    }
    __device__ __forceinline__ void second(const D1Cell<double> &c, double, const D1Mid<double> &m, double pm,
                                           double pp, const double fo[3], double out[3]) const {
        D1Cell64<FAST> k{FAST(f)};
        k.second(c, m, pm, pp, fo, out);
        if (k.o.bad) {
            const D1Cell<double> cc = c;
            const D1Mid<double> mm = m;
            const double in[3] = {fo[0], fo[1], fo[2]};
            double again[3];
            d1_second_again(cc, mm, pm, pp, in, again);
#pragma unroll
            for (int q = 0; q < 3; ++q) out[q] = again[q];
        }
    }
    __device__ __forceinline__ void moments(const double fo[3], double &h, double &u) const {
        D1Cell64<FAST> k{FAST(f)};
        k.moments(fo, h, u);
        if (k.o.bad) {
            const double in[3] = {fo[0], fo[1], fo[2]};
            double ha, ua;
            d1_moments_again(in, &ha, &ua);
            h = ha;
            u = ua;
        }
    }
};

// The same in FP32, operation by operation.
struct D1Ops32 {
    Fma64 f;  // (of Float64 states)
    __device__ __forceinline__ static float pow_n(float x, int n) {  // power_broad (src/pressure.jl:363-369)
        float t = 1.0f;
        for (int i = 0; i < n; ++i) t *= x;
        return t;
    }
    __device__ __forceinline__ float pressure(const D1Args &a, const D1Cell<float> &c, float h, float hip,
                                              float him) const {
        const float x = float(a.hmin) / (h + float(a.hcrit));
        const float p = -c.gam * (c.kap * (pow_n(x, a.n) - pow_n(x, a.m)));
        return p - c.gam * ((hip - 2.0f * h) + him);
    }
    __device__ __forceinline__ void local(const D1Cell<float> &c, float h, float u, const float *, bool,
                                          D1Mid<float> &m) const {
        m.slip = (c.mu6 * h * u) / ((2.0f * (h * h) + c.delta6 * h) + c.delta3sq);
        const float uu = u * u;
        m.fe[0] = h * ((1.0f - (0.5f * c.g) * h) - uu);
        m.fe[1] = h * (((0.25f * c.g) * h + 0.5f * u) + 0.5f * uu);
        m.fe[2] = h * (((0.25f * c.g) * h - 0.5f * u) + 0.5f * uu);
    }
    __device__ __forceinline__ void second(const D1Cell<float> &c, float h, const D1Mid<float> &m, float pm,
                                           float pp, const float fo[3], float out[3]) const {
        const float hgp = (h * -0.5f) * (pm - pp);
        float F = -hgp - m.slip;
        if (c.grad) F = F - c.dg;
        out[0] = c.omeg * fo[0] + c.invtau * m.fe[0];
        out[1] = c.omeg * fo[1] + c.invtau * m.fe[1] + 0.5f * F;
        out[2] = c.omeg * fo[2] + c.invtau * m.fe[2] - 0.5f * F;
    }
    __device__ __forceinline__ void moments(const float o[3], float &h, float &u) const {
        h = (o[0] + o[1]) + o[2];
        u = (o[1] - o[2]) / h;
    }
};

__device__ __forceinline__ bool finite(double v) { return finite64(v); }
__device__ __forceinline__ bool finite(float v) { return isfinite(v); }

// A warp's measures of its own cells' heights.
__device__ __forceinline__ void d1_measure(D1Part *out, bool own, double h, bool wet) {
    uint32_t c[kChunks] = {};
    bool held = true;
    if (own) held = chunks64(h, c);
    const unsigned long long o = own && h == h ? order64(h) : 0ull, o2 = o ? ~o : 0ull;
    D1Part p;
    p.big = 0.0;
    if (__any_sync(0xffffffffu, !held)) {
        double b = held ? 0.0 : h;
        if (!held)
#pragma unroll
            for (int q = 0; q < kChunks; ++q) c[q] = 0;
        for (int k = 16; k; k >>= 1) b += __shfl_xor_sync(0xffffffffu, b, k);
        p.big = b;
    }
#pragma unroll
    for (int q = 0; q < kChunks; ++q) p.mass[q] = __reduce_add_sync(0xffffffffu, c[q]);
    p.wet = __popc(__ballot_sync(0xffffffffu, own && wet));
    const uint32_t xh = __reduce_max_sync(0xffffffffu, (uint32_t)(o >> 32));
    const uint32_t xl = __reduce_max_sync(0xffffffffu, (uint32_t)(o >> 32) == xh ? (uint32_t)o : 0u);
    const uint32_t nh = __reduce_max_sync(0xffffffffu, (uint32_t)(o2 >> 32));
    const uint32_t nl = __reduce_max_sync(0xffffffffu, (uint32_t)(o2 >> 32) == nh ? (uint32_t)o2 : 0u);
    p.kmax = (unsigned long long)xh << 32 | xl;
    p.kmin = (unsigned long long)nh << 32 | nl;
    if ((threadIdx.x & 31) == 0) *out = p;
}

// n iterations of the cells of chunk blockIdx.x, from the buffers `from` to the
// others.  part: this launch's measures, [n][gridDim.x][NT / 32] (or null).
// Float64 has two threads per cell: the first NT compute pressures (and the
// measures) while the others compute slippage and equilibrium, the two long
// chains of an iteration, and then collide and stream (2.82 -> 2.58 us per
// iteration; FP32, whose chains are short, 0.94 -> 0.97 and so one thread).
template <class R>
constexpr int kD1Halves = sizeof(R) == 8 ? 2 : 1;
template <class R, class Ops, int NT>
__global__ void __launch_bounds__(kD1Halves<R> * NT) d1q3_run_kernel(const D1Args *__restrict__ args,
                                                         const D1Chunk *__restrict__ table, const Ops op,
                                                         int from, int n, D1Part *part) {
    __shared__ D1Args a;
    __shared__ R sh[NT], sp[NT], s1[NT], s2[NT];
    const D1Chunk ck = table[blockIdx.x];
    if (threadIdx.x == 0) a = args[ck.lattice];
    __syncthreads();
    grid_dep_wait();
    grid_dep_launch();
    const int t = threadIdx.x & (NT - 1), L = a.L;
    const bool first = threadIdx.x < NT;  // computes pressures (whole warps)
    const bool second = kD1Halves<R> == 1 || !first;  // holds the cell's state
    const bool whole = ck.w == L && L <= NT;  // periodic within the CTA
    const int halo = whole ? 0 : 3 * n, span = ck.w + 2 * halo;
    const bool in = t < span, own = t >= halo && t < halo + ck.w;
    int g = ck.x0 - halo + t;  // halo < L
    g = g < 0 ? g + L : (g >= L ? g - L : g);
    if (!in) g = 0;
    // neighbours; at the ends of a span with halos their values do not matter
    const int tm = t == 0 ? (whole ? span - 1 : 0) : t - 1;
    const int tp = t >= span - 1 ? (whole ? 0 : span - 1) : t + 1;
    D1Cell<R> c;
    c.mu6 = R(6) * R(a.mu);
    c.delta6 = R(6) * R(a.delta);
    c.delta3sq = R(3) * (R(a.delta) * R(a.delta));
    c.omeg = R(a.omeg);
    c.invtau = R(a.invtau);
    c.tau1 = a.omeg == 0.0 && a.invtau == 1.0;
    c.g = R(a.g);
    c.g25 = R(0.25) * c.g;
    c.g50 = R(0.5) * c.g;
    c.kap = a.kapF ? reinterpret_cast<const R *>(a.kapF)[g] : R(a.kap);
    c.gam = a.gamF ? reinterpret_cast<const R *>(a.gamF)[g] : R(a.gamma);
    c.dg = a.dgF ? reinterpret_cast<const R *>(a.dgF)[g] : R(0);
    c.grad = a.dgF != nullptr;
    const bool rec = part != nullptr && a.rec;
    const R *ff = reinterpret_cast<const R *>(a.f[from]);
    R h = reinterpret_cast<const R *>(a.h[from])[g], u = reinterpret_cast<const R *>(a.u[from])[g];
    R fo[3] = {ff[g], ff[L + g], ff[2 * L + g]}, p = R(0);
    bool odd = !(finite(h) && finite(fo[0]) && finite(fo[1]) && finite(fo[2]));
    int bad = 0;
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        if (second) sh[t] = h;
        __syncthreads();
        D1Mid<R> m;
        if (first) {
            const R hc = sh[t];
            if (in) {
                p = op.pressure(a, c, hc, sh[tm], sh[tp]);
                sp[t] = p;
            }
            if (rec)
                d1_measure(part + ((size_t)k * gridDim.x + blockIdx.x) * (NT / 32) + (t >> 5), own, (double)hc,
                           hc > R(0.055));
        }
        if (second && in) {
            op.local(c, h, u, fo, odd, m);
        }
        __syncthreads();
        R o[3];
        if (second && in) {
            op.second(c, h, m, sp[tm], sp[tp], fo, o);
            s1[t] = o[1];
            s2[t] = o[2];
        }
        __syncthreads();
        if (second && in) {
            fo[0] = o[0];
            fo[1] = s1[tm];
            fo[2] = s2[tp];
            op.moments(fo, h, u);
            odd = !finite(h);  // as it is where a population is not
            if (own && odd) bad = 1;
        }
    }
    if (!own) return;
    if (first) reinterpret_cast<R *>(a.p)[g] = p;
    if (!second) return;
    R *fn = reinterpret_cast<R *>(a.f[from ^ 1]);
    reinterpret_cast<R *>(a.h[from ^ 1])[g] = h;
    reinterpret_cast<R *>(a.u[from ^ 1])[g] = u;
#pragma unroll
    for (int q = 0; q < 3; ++q) fn[q * L + g] = fo[q];
    if (bad) *a.nan_flag = 1;
}

// The records of n iterations after t0 from their warps' measures: one warp
// per lattice (blockIdx.x, of which there may be more than 65535) and iteration.
__global__ void __launch_bounds__(128) d1q3_record_kernel(const D1Args *__restrict__ args,
                                                          const D1Part *__restrict__ part, int nchunks,
                                                          int warps, int n, long long t0) {
    const D1Args &a = args[blockIdx.x];
    const int k = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (k >= n || !a.rec || n - k > a.rec_cap) return;  // only the newest the ring holds
    long long c[kChunks] = {};
    unsigned long long mx = 0, mn = 0;
    int wet = 0;
    double big = 0.0;
    const D1Part *pp = part + ((size_t)k * nchunks + a.chunk0) * warps;
    for (int i = lane; i < a.chunks * warps; i += 32) {
#pragma unroll
        for (int q = 0; q < kChunks; ++q)
            c[q] += q == kChunks - 1 ? (long long)(int32_t)pp[i].mass[q] : (long long)pp[i].mass[q];
        wet += (int)pp[i].wet;
        mx = max(mx, pp[i].kmax);
        mn = max(mn, pp[i].kmin);
        big += pp[i].big;
    }
    for (int o = 16; o; o >>= 1) {
#pragma unroll
        for (int q = 0; q < kChunks; ++q) c[q] += __shfl_xor_sync(0xffffffffu, c[q], o);
        wet += __shfl_xor_sync(0xffffffffu, wet, o);
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        mn = max(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        big += __shfl_xor_sync(0xffffffffu, big, o);
    }
    if (lane == 0) {
        const long long t = t0 + k + 1;
        Record &r = a.rec[(t - 1) % a.rec_cap];
        r.t = t;
        r.mass = value64(c) + big;
        r.wetted = (double)wet;
        r.hmax = mx ? unorder64(mx) : -INFINITY;
        r.hmin = mn ? unorder64(~mn) : INFINITY;
        r.area = 0.0;
        r.cos_sum = 0.0;
    }
}

// ∇γ = -3/2 (γ[i-1] - γ[i+1]) / 2 (src/forcing.jl:423-432), once per γ field.
template <class R>
__global__ void d1q3_gradgamma_kernel(const R *gam, R *dg, int L) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L; i += gridDim.x * blockDim.x)
        dg[i] = R(-3.0 / 2.0) * ((gam[i == 0 ? L - 1 : i - 1] - gam[i == L - 1 ? 0 : i + 1]) / R(2.0));
}

}  // namespace
}  // namespace swb

using swb::D1Args;
using swb::Record;

namespace {
thread_local std::string d1_err;
int d1fail(std::string *slot, int code, const std::string &m) {
    if (slot) *slot = m;
    d1_err = m;
    swb::set_global_error(m.c_str());
    return code;
}
}  // namespace

struct swb1d {
    int count = 0, precision = SWB_F64, rb = 8;
    std::vector<swb_params> params;
    std::vector<D1Args> args;
    std::vector<char *> mem;  // one block per lattice
    D1Args *d_args = nullptr;
    int *d_flags = nullptr;
    int rec_cap = 0;
    int cur = 0;               // buffers that hold the fields and populations
    long long t = 0;           // iterations done
    swb::D1Chunk *d_chunks = nullptr;
    int nchunks = 0;
    int per_launch = 0;        // iterations a launch may run
    int cells = swb::kD1Cells;  // cells of a CTA, halo included
    swb::D1Part *d_part = nullptr;
    int part_steps = 0;        // iterations d_part holds
    bool args_dirty = true;
    cudaStream_t stream = nullptr;
    std::string err;
    ~swb1d() {
        if (stream) cudaStreamSynchronize(stream);
        for (char *q : mem) cudaFree(q);
        cudaFree(d_args);
        cudaFree(d_flags);
        cudaFree(d_chunks);
        cudaFree(d_part);
        if (stream) cudaStreamDestroy(stream);
    }
};

#define D1_TRY(b, expr)                                                                        \
    do {                                                                                       \
        cudaError_t e_ = (expr);                                                               \
        if (e_ != cudaSuccess)                                                                 \
            return d1fail(&(b)->err, e_ == cudaErrorMemoryAllocation ? SWB_ERR_OOM : SWB_ERR_CUDA, \
                          std::string(#expr) + ": " + cudaGetErrorString(e_));                 \
    } while (0)

namespace {
// Bytes of one lattice's block: two sets of populations (3L), h and u, then
// p, κ, γ, ∇γ (L each) and the measure ring.
size_t d1_bytes(int L, int rb, int rec_cap) {
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    return 2 * al((size_t)3 * L * rb) + 8 * al((size_t)L * rb) + al((size_t)rec_cap * sizeof(Record));
}

int layout(swb1d *b, int i, char *base) {
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const int L = b->params[i].Lx, rb = b->rb;
    D1Args &a = b->args[i];
    size_t o = 0;
    for (int k = 0; k < 2; ++k) {
        a.f[k] = base + o; o += al((size_t)3 * L * rb);
        a.h[k] = base + o; o += al((size_t)L * rb);
        a.u[k] = base + o; o += al((size_t)L * rb);
    }
    a.p = base + o; o += al((size_t)L * rb);
    o += 3 * al((size_t)L * rb);  // κ, γ, ∇γ: addressed through field_ptr
    a.rec = b->rec_cap ? reinterpret_cast<Record *>(base + o) : nullptr;
    a.rec_cap = b->rec_cap;
    return SWB_OK;
}

char *field_ptr(swb1d *b, int i, int which) {  // 0 κ, 1 γ, 2 ∇γ (allocated slots)
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const int L = b->params[i].Lx, rb = b->rb;
    return b->mem[i] + 2 * al((size_t)3 * L * rb) + (5 + which) * al((size_t)L * rb);
}

int upload(swb1d *b, void *dst, const double *host, int L) {
    if (b->rb == 8) {
        D1_TRY(b, cudaMemcpyAsync(dst, host, (size_t)L * 8, cudaMemcpyHostToDevice, b->stream));
    } else {
        std::vector<float> tmp(host, host + L);
        D1_TRY(b, cudaMemcpyAsync(dst, tmp.data(), (size_t)L * 4, cudaMemcpyHostToDevice, b->stream));
        D1_TRY(b, cudaStreamSynchronize(b->stream));
    }
    return SWB_OK;
}

int download(swb1d *b, const void *src, double *host, size_t n) {
    if (b->rb == 8) {
        D1_TRY(b, cudaMemcpyAsync(host, src, n * 8, cudaMemcpyDeviceToHost, b->stream));
        D1_TRY(b, cudaStreamSynchronize(b->stream));
    } else {
        std::vector<float> tmp(n);
        D1_TRY(b, cudaMemcpyAsync(tmp.data(), src, n * 4, cudaMemcpyDeviceToHost, b->stream));
        D1_TRY(b, cudaStreamSynchronize(b->stream));
        for (size_t k = 0; k < n; ++k) host[k] = tmp[k];
    }
    return SWB_OK;
}

__global__ void fill1(void *p, int L, int rb, double v) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L; i += gridDim.x * blockDim.x) {
        if (rb == 8)
            reinterpret_cast<double *>(p)[i] = v;
        else
            reinterpret_cast<float *>(p)[i] = (float)v;
    }
}

constexpr int kBurst = 4096;                  // iterations between records
constexpr size_t kPartBytes = (size_t)64 << 20;  // of measures a burst keeps

// Cuts the lattices into chunks of one CTA each and returns the iterations K
// of a launch.  A launch of c CTAs per SM lasts about K max(1, c / r) t + t0 + c l:
// Float64 t = 2.5 us with CTAs of 128 cells and 1.75 with 64, r = 1 (one CTA keeps
// an SM's Float64 units busy), FP32 t = 0.9 us and r = 6.25 (it leaves them idle),
// t0 = 2 us, l = 0.15 us (FP32; for its loads and stores, 4 % of a Float64 CTA's
// time); larger K need more CTAs, because 6 K of their cells are halo.  With FP32 the
// K this gives are within 2 % of the best of 1 to 20 for 1 to 3000 lattices of 130
// to 2M cells (2000 of 1000 cells: K = 4 26.9 us per iteration; 2 30.8, 8 30.5).
int split_lattices(swb1d *b, std::vector<swb::D1Chunk> &out) {
    int sms = 1, dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) sms = 1;
    const bool f64 = b->rb == 8;
    auto pieces = [](int L, int cells, int K) {
        const int w = cells - 6 * K;
        return L <= cells ? 1 : (L + w - 1) / w;
    };
    int best = 1, cells = swb::kD1Cells;
    double cost = 1e300;
    for (int nt : {swb::kD1Cells, swb::kD1Cells / 2}) {
        if (nt != swb::kD1Cells && !f64) break;
        const double t = !f64 ? 0.9 : (nt == swb::kD1Cells ? 2.5 : 1.75), r = f64 ? 1.0 : 6.25;
        for (int K = 1; 6 * K + 8 <= nt; ++K) {
            long long n = 0;
            for (const swb_params &p : b->params) n += pieces(p.Lx, nt, K);
            const double us = std::max(1.0, std::ceil((double)n / sms) / r) * t +
                              (2.0 + (f64 ? 0.0 : 0.15) * (double)n / sms) / K;
            if (us < cost) {
                cost = us;
                best = K;
                cells = nt;
            }
        }
    }
    b->cells = cells;
    bool small = true;
    for (const swb_params &p : b->params) small = small && p.Lx <= cells;
    for (int i = 0; i < b->count; ++i) {
        const int L = b->params[i].Lx, k = pieces(L, cells, best);
        b->args[i].chunk0 = (int)out.size();
        b->args[i].chunks = k;
        for (int j = 0; j < k; ++j) {
            const int x0 = (int)((long long)L * j / k), x1 = (int)((long long)L * (j + 1) / k);
            out.push_back({i, x0, x1 - x0});
        }
    }
    return small ? kBurst : best;  // without halos a launch may run any number of iterations
}
}  // namespace

extern "C" {

int swb1d_create(const swb_params *params, int count, int precision, int rec_cap, swb1d **out) {
    if (!out || !params || count < 1 || rec_cap < 0)
        return d1fail(nullptr, SWB_ERR_ARG, "bad arguments");
    *out = nullptr;
    if (precision != SWB_F64 && precision != SWB_F32)
        return d1fail(nullptr, SWB_ERR_ARG, "1D precision must be SWB_F64 or SWB_F32");
    for (int i = 0; i < count; ++i) {
        const swb_params &p = params[i];
        if (p.Lx < 3 || p.Ly != 1 || 3LL * p.Lx >= (1LL << 31) || !(p.tau > 0) || p.n <= p.m ||
            p.m < 1 || !(p.hmin > 0))
            return d1fail(nullptr, SWB_ERR_ARG, "invalid 1D params for lattice " + std::to_string(i) +
                                                    " (L = Lx >= 3, Ly = 1)");
        if (p.kbt != 0.0)
            return d1fail(nullptr, SWB_ERR_UNSUPPORTED, "1D thermal fluctuations are not supported");
    }
    swb1d *b = new swb1d();
    b->count = count;
    b->precision = precision;
    b->rb = precision == SWB_F64 ? 8 : 4;
    b->rec_cap = rec_cap;
    b->params.assign(params, params + count);
    b->args.resize(count);
    auto bad = [&](int code) {
        std::string m = b->err;
        delete b;
        d1_err = m;
        swb::set_global_error(m.c_str());
        return code;
    };
#define C1_TRY(expr)                                                                       \
    do {                                                                                   \
        cudaError_t e_ = (expr);                                                           \
        if (e_ != cudaSuccess) {                                                           \
            b->err = std::string(#expr) + ": " + cudaGetErrorString(e_);                   \
            return bad(e_ == cudaErrorMemoryAllocation ? SWB_ERR_OOM : SWB_ERR_CUDA);      \
        }                                                                                  \
    } while (0)
    C1_TRY(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
    C1_TRY(cudaMalloc((void **)&b->d_flags, sizeof(int) * count));
    C1_TRY(cudaMemsetAsync(b->d_flags, 0, sizeof(int) * count, b->stream));
    C1_TRY(cudaMalloc((void **)&b->d_args, sizeof(D1Args) * count));
    for (int i = 0; i < count; ++i) {
        const swb_params &p = params[i];
        char *m = nullptr;
        const size_t bytes = d1_bytes(p.Lx, b->rb, rec_cap);
        C1_TRY(cudaMalloc((void **)&m, bytes));
        b->mem.push_back(m);
        C1_TRY(cudaMemsetAsync(m, 0, bytes, b->stream));  // populations 0 (Sys(), src/initialize.jl:587-599)
        D1Args &a = b->args[i];
        a = D1Args{};
        a.L = p.Lx;
        a.n = p.n;
        a.m = p.m;
        a.gamma = p.gamma;
        a.hmin = p.hmin;
        a.hcrit = p.hcrit;
        a.delta = p.delta;
        a.mu = p.mu;
        a.g = p.g;
        a.kap = swb::host_kappa_shared(p.theta, p.n, p.m, p.hmin);
        a.omeg = 1.0 - 1.0 / p.tau;
        a.invtau = 1.0 / p.tau;
        layout(b, i, m);
        a.nan_flag = b->d_flags + i;
        fill1<<<(p.Lx + 255) / 256, 256, 0, b->stream>>>(a.h[0], p.Lx, b->rb, 1.0);  // height = 1
        swb::count_launches(1);
        C1_TRY(cudaGetLastError());
    }
    std::vector<swb::D1Chunk> chunks;
    b->per_launch = split_lattices(b, chunks);
    b->nchunks = (int)chunks.size();
    C1_TRY(cudaMalloc((void **)&b->d_chunks, sizeof(swb::D1Chunk) * chunks.size()));
    C1_TRY(cudaMemcpyAsync(b->d_chunks, chunks.data(), sizeof(swb::D1Chunk) * chunks.size(),
                           cudaMemcpyHostToDevice, b->stream));
    C1_TRY(cudaStreamSynchronize(b->stream));
#undef C1_TRY
    *out = b;
    return SWB_OK;
}

int swb1d_destroy(swb1d *b) {
    delete b;
    return SWB_OK;
}

int swb1d_set_field(swb1d *b, int idx, int field, const double *host) {
    if (!b || idx < 0 || idx >= b->count) return d1fail(b ? &b->err : nullptr, SWB_ERR_ARG, "bad arguments");
    D1Args &a = b->args[idx];
    const int L = a.L;
    switch (field) {
        case SWB_FIELD_HEIGHT:
        case SWB_FIELD_VELX:
            if (!host) return d1fail(&b->err, SWB_ERR_ARG, "NULL field");
            return upload(b, field == SWB_FIELD_HEIGHT ? a.h[b->cur] : a.u[b->cur], host, L);
        case SWB1D_FIELD_THETA: {
            if (!host) {
                a.kapF = nullptr;
                b->args_dirty = true;
                return SWB_OK;
            }
            std::vector<double> kap(L);
            const swb_params &p = b->params[idx];
            for (int i = 0; i < L; ++i)  // (fields are often constant over long stretches)
                kap[i] = i > 0 && host[i] == host[i - 1]
                             ? kap[i - 1]
                             : swb::host_kappa_shared(host[i], p.n, p.m, p.hmin);
            char *dst = field_ptr(b, idx, 0);
            int rc = upload(b, dst, kap.data(), L);
            if (rc) return rc;
            a.kapF = dst;
            b->args_dirty = true;
            return SWB_OK;
        }
        case SWB1D_FIELD_GAMMA: {
            if (!host) {
                a.gamF = a.dgF = nullptr;
                b->args_dirty = true;
                return SWB_OK;
            }
            char *g = field_ptr(b, idx, 1), *dg = field_ptr(b, idx, 2);
            int rc = upload(b, g, host, L);
            if (rc) return rc;
            if (b->rb == 8)
                swb::d1q3_gradgamma_kernel<double><<<(L + 255) / 256, 256, 0, b->stream>>>(
                    (const double *)g, (double *)dg, L);
            else
                swb::d1q3_gradgamma_kernel<float><<<(L + 255) / 256, 256, 0, b->stream>>>(
                    (const float *)g, (float *)dg, L);
            swb::count_launches(1);
            D1_TRY(b, cudaGetLastError());
            a.gamF = g;
            a.dgF = dg;
            b->args_dirty = true;
            return SWB_OK;
        }
        default:
            return d1fail(&b->err, SWB_ERR_ARG, "1D fields: height, vel, theta, gamma");
    }
}

int swb1d_get_field(swb1d *b, int idx, int field, double *host) {
    if (!b || !host || idx < 0 || idx >= b->count)
        return d1fail(b ? &b->err : nullptr, SWB_ERR_ARG, "bad arguments");
    D1Args &a = b->args[idx];
    switch (field) {
        case SWB_FIELD_HEIGHT: return download(b, a.h[b->cur], host, (size_t)a.L);
        case SWB_FIELD_VELX: return download(b, a.u[b->cur], host, (size_t)a.L);
        case SWB_FIELD_PRESSURE: return download(b, a.p, host, (size_t)a.L);
        case SWB_FIELD_FOUT: return download(b, a.f[b->cur], host, (size_t)3 * a.L);
        default: return d1fail(&b->err, SWB_ERR_ARG, "1D fields: height, vel, pressure, fout");
    }
}

int swb1d_step(swb1d *b, int64_t nsteps) {
    if (!b || nsteps < 0) return d1fail(b ? &b->err : nullptr, SWB_ERR_ARG, "bad arguments");
    if (b->args_dirty) {
        D1_TRY(b, cudaMemcpyAsync(b->d_args, b->args.data(), sizeof(D1Args) * b->count,
                                  cudaMemcpyHostToDevice, b->stream));
        b->args_dirty = false;
    }
    // bursts of launches, then the burst's records
    const int warps = b->cells / 32;
    const size_t row = sizeof(swb::D1Part) * warps * (size_t)b->nchunks;
    while (nsteps > 0) {
        int burst = (int)std::min<int64_t>(nsteps, kBurst);
        if (b->rec_cap) {
            burst = (int)std::min<size_t>((size_t)burst, std::max<size_t>(1, kPartBytes / row));
            if (burst > b->part_steps) {
                D1_TRY(b, cudaStreamSynchronize(b->stream));
                cudaFree(b->d_part);
                b->d_part = nullptr;
                b->part_steps = 0;
                D1_TRY(b, cudaMalloc((void **)&b->d_part, row * (size_t)burst));
                b->part_steps = burst;
            }
        }
        for (int done = 0; done < burst;) {
            const int n = std::min(b->per_launch, burst - done);
            swb::D1Part *part =
                b->rec_cap ? b->d_part + (size_t)done * b->nchunks * warps : nullptr;
            const swb::Fma64 f{1.0};
            auto run = [&](auto *kern, int halves, auto ops) {
                return swb::launch_step(kern, b->nchunks, halves * b->cells, b->stream, b->d_args, b->d_chunks, ops,
                                        b->cur, n, part);
            };
            using Split = swb::D1Ops64<swb::Fast64>;
            using Direct = swb::D1Ops64<swb::D1Direct64>;
            constexpr int C = swb::kD1Cells;
            const cudaError_t e =
                b->rb == 4       ? run(swb::d1q3_run_kernel<float, swb::D1Ops32, C>, swb::kD1Halves<float>, swb::D1Ops32{f})
                : b->cells == C ? run(swb::d1q3_run_kernel<double, Split, C>, swb::kD1Halves<double>, Split{f})
                                : run(swb::d1q3_run_kernel<double, Direct, C / 2>, swb::kD1Halves<double>, Direct{f});
            D1_TRY(b, e);
            swb::count_launches(1);
            b->cur ^= 1;
            done += n;
        }
        if (b->rec_cap) {
            swb::d1q3_record_kernel<<<dim3((unsigned)b->count, (unsigned)((burst + 3) / 4)), 128, 0, b->stream>>>(
                b->d_args, b->d_part, b->nchunks, warps, burst, b->t);
            swb::count_launches(1);
            D1_TRY(b, cudaGetLastError());
        }
        b->t += burst;
        nsteps -= burst;
    }
    return SWB_OK;
}

int swb1d_sync(swb1d *b) {
    if (!b) return d1fail(nullptr, SWB_ERR_ARG, "NULL");
    D1_TRY(b, cudaStreamSynchronize(b->stream));
    std::vector<int> flags(b->count);
    D1_TRY(b, cudaMemcpy(flags.data(), b->d_flags, sizeof(int) * b->count, cudaMemcpyDeviceToHost));
    for (int i = 0; i < b->count; ++i)
        if (flags[i]) return d1fail(&b->err, SWB_ERR_NAN, "non-finite height in 1D lattice " + std::to_string(i));
    return SWB_OK;
}

int swb1d_get_measures(swb1d *b, int idx, swb_measure *out, int64_t cap, int64_t *count) {
    if (!b || !count || idx < 0 || idx >= b->count || (cap > 0 && !out))
        return d1fail(b ? &b->err : nullptr, SWB_ERR_ARG, "bad arguments");
    *count = 0;
    const D1Args &a = b->args[idx];
    if (!a.rec) return SWB_OK;
    const long long t = b->t;
    D1_TRY(b, cudaStreamSynchronize(b->stream));
    long long n = t < a.rec_cap ? t : a.rec_cap;
    if (n > cap) n = cap;
    std::vector<Record> r((size_t)a.rec_cap);
    D1_TRY(b, cudaMemcpy(r.data(), a.rec, sizeof(Record) * a.rec_cap, cudaMemcpyDeviceToHost));
    for (long long k = 0; k < n; ++k) {  // the newest n iterations, oldest first
        const Record &x = r[(size_t)((t - n + k) % a.rec_cap)];
        out[k].t = x.t;
        out[k].mass = x.mass;
        out[k].wetted = (int64_t)x.wetted;
        out[k].hmax = x.hmax;
        out[k].hmin = x.hmin;
        out[k].area = 0.0;
        out[k].energy = 0.0;
    }
    *count = n;
    return SWB_OK;
}

}  // extern "C"
