// swb_step_f64.cu -- Float64 kernels.  Compiled with --fmad=false so that no
// a*b+c is contracted into an FMA: the reference (Julia broadcasts) rounds
// every operation, and this translation unit reproduces it bit for bit.
//
// Contents: the cell kernels of single lattices, the strips of batched and
// served ones (literal arithmetic), θ fields, the plain
// one-kernel-per-reference-op path, and the standalone measure reduction.
#include "swb_step_impl.cuh"
#include "swb_f64.cuh"

namespace swb {

// ------------------------------------------------------------ fused, Float64
#define DISPATCH_NT(nt, ...)                       \
    do {                                           \
        if ((nt) == 64) {                          \
            constexpr int NT = 64;                 \
            __VA_ARGS__;                           \
        } else if ((nt) == 256) {                  \
            constexpr int NT = 256;                \
            __VA_ARGS__;                           \
        } else {                                   \
            constexpr int NT = 128;                \
            __VA_ARGS__;                           \
        }                                          \
    } while (0)

// One iteration of a single Float64 lattice is three kernels of one cell per
// thread: the film pressure of the fields, forces and collision into the
// post-collision populations, and the moments of those populations back into
// the fields (so h and u are always those of the iteration that comes next).
//
// Why not the strips of the FP32 states: the step is bound by the Float64
// units (a warp instruction per 64 cycles and SM quarter), so what counts is
// the number of Float64 instructions per cell and an even share of them for
// every SM quarter; memory and the extra launches hide behind them.  A
// strip recomputes the moments and pressures of its halo and leaves lanes
// idle where the lattice is no multiple of it; one cell per thread does
// neither, and needs no barrier.  Against strips with the plain operations
// (302 Float64 instructions per cell; here 145, and with the products in
// integers 94): 600 iterations of a 256² droplet 41.1 -> 16.0 -> 12.6 ms, 60 of a
// 1000 x 1030 film 34.3 -> 17.1 -> 13.2 ms (upload and download included), 512²
// 141 -> 77 -> 57 us per iteration; with the reciprocals in integers as well
// (80 instructions) 52 us, and 1000 x 1030 195 -> 181.  A 56 x 40 film, one warp per SM quarter, is
// bound by latency: 43.7 -> 10.7 -> 11.1 us.  (One kernel of 8 x 4 tiles with
// recomputed halos: 9.4 there, but 12.4 at 128 x 96 and 104 at 512².)
constexpr int kCellNT = 128;

namespace {

struct Cell {
    int i, j, im, ip, jm, jp;  // column, row, and the periodic neighbours
};
__device__ __forceinline__ Cell cell_at(int c, int Lx, int Ly) {
    Cell g;
    g.j = c / Lx;
    g.i = c - g.j * Lx;
    g.im = g.i == 0 ? Lx - 1 : g.i - 1;
    g.ip = g.i == Lx - 1 ? 0 : g.i + 1;
    g.jm = (g.j == 0 ? Ly - 1 : g.j - 1) * Lx;
    g.jp = (g.j == Ly - 1 ? 0 : g.j + 1) * Lx;
    g.j *= Lx;  // rows as offsets
    return g;
}

// Index into a θ field moved by (sx, sy), of column i and row offset j.
__device__ __forceinline__ int field_at(const StepArgs &a, int i, int j, int sx, int sy) {
    return (j - sy * a.Lx < 0 ? j + (a.Ly - sy) * a.Lx : j - sy * a.Lx) + (i - sx < 0 ? i - sx + a.Lx : i - sx);
}

// κ and cospi(θ) of every column for iteration step_base + k + 1 of the θ wave.
__global__ void __launch_bounds__(kCellNT) cell_wave_kernel(const StepArgs a, const Cell64 x, int k) {
    grid_dep_wait();
    grid_dep_launch();
    const int i = blockIdx.x * kCellNT + threadIdx.x;
    if (i >= a.Lx) return;
    const KapCos<double> w = wave_at<double>(a, i, a.ctl->step_base + k + 1);
    x.wave[i] = w.kap;
    x.wave[a.Lx + i] = w.cs;
}

__device__ __forceinline__ Near64 near_cell(const double *v, const Cell &g) {
    return {v[g.j + g.im],  v[g.jm + g.i],  v[g.j + g.ip],  v[g.jp + g.i],
            v[g.jm + g.im], v[g.jm + g.ip], v[g.jp + g.ip], v[g.jp + g.im]};
}

// A cell whose integer arithmetic met a number it does not hold, again in
// Float64 operations (out of line).
__device__ __noinline__ double cell_pressure_again(double h, const Near64 &v, double kap, double gamma,
                                                   double hmin, double hcrit, int n, int m) {
    Plain64 o;
    return pressure64(o, h, v, kap, gamma, hmin, hcrit, n, m);
}
__device__ __forceinline__ double cell_pressure(const StepArgs &a, const Cell64 &x, double h, const Near64 &v,
                                                double kap) {
    Fast64 o(x.f);
    const double p = pressure64(o, h, v, kap, a.gamma, a.hmin, a.hcrit, a.n, a.m);
    if (!o.bad) return p;
    const Near64 w = v;
    return cell_pressure_again(h, w, kap, a.gamma, a.hmin, a.hcrit, a.n, a.m);
}

template <int MODE>
__global__ void __launch_bounds__(kCellNT) cell_pressure_kernel(const StepArgs a, const Cell64 x, int k) {
    const int c = blockIdx.x * kCellNT + threadIdx.x;
    const int cc = c < a.Lx * a.Ly ? c : 0;
    const Cell g = cell_at(cc, a.Lx, a.Ly);
    grid_dep_wait();
    grid_dep_launch();
    if (c != cc) return;
    const double *h = reinterpret_cast<const double *>(a.hF);
    double kap = a.kap;
    if (MODE == THETA_WAVE) kap = x.wave[g.i];
    if (MODE == THETA_FIELD) {
        int sx, sy;
        substrate_shift(a, a.ctl->step_base + k + 1, &sx, &sy);
        kap = reinterpret_cast<const double *>(a.kapF)[field_at(a, g.i, g.j, sx, sy)];
    }
    x.p[c] = cell_pressure(a, x, h[c], near_cell(h, g), kap);
}

// Sums of values that chunks64 does not hold, over the whole range of Float64:
// limb i of a sum counts units of 2^(32 i - 1074) in 64 bits, so that it takes
// 2^31 values before it has to pass anything on, and the sum is exact and free
// of order like the other.  (Rare, so one atomic per limb and value will do.)
__device__ __forceinline__ void wide_add(unsigned long long *w, double v) {
    const int e = (int)((hi64(v) >> 20) & 0x7ff), p = e ? e - 1 : 0;
    const uint64_t m = (__double_as_longlong(v) & 0xfffffffffffffull) | (e ? 0x10000000000000ull : 0ull);
    const unsigned __int128 u = (unsigned __int128)m << (p & 31);
    const bool neg = hi64(v) & 0x80000000u;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const unsigned long long l = (uint32_t)(u >> (32 * i));
        if (l) atomicAdd(w + p / 32 + i, neg ? 0ull - l : l);
    }
}
// The value of the limbs w and chunk sums c together, rounded once; clears w.
// One thread, with nobody else at w.
__device__ __noinline__ double wide_value(unsigned long long *w, const long long *c) {
    auto at = [&](int i) { return i < 0 ? 0ll : (long long)__ldcg(w + i); };
    for (int i = 0; i < kChunks; ++i) {  // chunk i counts units of 2^(27 i - 96)
        const int p = 27 * i + 1074 - 96;
        const __int128 v = (__int128)c[i] << (p & 31);
        w[p / 32] = (unsigned long long)(at(p / 32) + (long long)(uint32_t)v);
        w[p / 32 + 1] = (unsigned long long)(at(p / 32 + 1) + (long long)(uint32_t)(v >> 32));
        w[p / 32 + 2] = (unsigned long long)(at(p / 32 + 2) + (long long)(v >> 64));
    }
    long long carry = 0;
    for (int i = 0; i < kWide64; ++i) {
        const long long v = at(i) + carry;
        w[i] = (uint32_t)v;
        carry = v >> 32;
    }
    const bool neg = carry < 0;
    if (neg) {  // the magnitude
        carry = 1;
        for (int i = 0; i < kWide64; ++i) {
            const long long v = (long long)(uint32_t)~(uint32_t)at(i) + carry;
            w[i] = (uint32_t)v;
            carry = v >> 32;
        }
    }
    int n = kWide64 - 1;
    while (n >= 0 && !at(n)) --n;
    double v = 0.0;
    if (n >= 0) {  // the upper 64 bits, the last one sticky
        const uint64_t h = (uint64_t)at(n) << 32 | (uint64_t)at(n - 1), l = (uint64_t)at(n - 2) << 32;
        const int z = __clzll((long long)h);
        uint64_t top = z ? h << z | l >> (64 - z) : h;
        bool rest = (l << z) != 0;
        for (int i = n - 3; i >= 0; --i) rest |= at(i) != 0;
        if (rest) top |= 1;
        v = ldexp((double)top, 32 * (n - 1) - z - 1074);
    }
    for (int i = 0; i < kWide64; ++i) w[i] = 0ull;
    return neg ? -v : v;
}

__device__ __noinline__ void cell_measure_outside(unsigned long long *acc, int at, double v) {
    unsigned long long *out = acc + kOut64;
    out[0] = 1ull;
    if (finite64(v))
        wide_add(out + 4 + at * kWide64, v);
    else
        atomicAdd(reinterpret_cast<double *>(out) + 1 + at, v);
}

// The measures of an iteration's height: every warp adds its cells' values
// as integers (chunks64: exact, in any order), the block its warps', and one
// atomic per value adds the block's to lane blockIdx % kLanes64.  Values that
// chunks64 does not hold are added one by one, exactly as well.
template <int NT>
__device__ __forceinline__ void cell_measures(const StepArgs &a, const Cell64 &x, int par, bool in,
                                              double h, double area, double cs, bool wet) {
    __shared__ uint32_t sh[NT / 32][kSums64 + 4];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool with_area = a.meas_mask & SWB_MEAS_AREA;
    unsigned long long *acc = x.acc + (size_t)par * kAcc64;
    uint32_t ch[kChunks];
    auto add = [&](double v, bool on, int at) {
#pragma unroll
        for (int q = 0; q < kChunks; ++q) ch[q] = 0;
        if (on && !chunks64(v, ch)) {
#pragma unroll
            for (int q = 0; q < kChunks; ++q) ch[q] = 0;
            cell_measure_outside(acc, at, v);
        }
#pragma unroll
        for (int q = 0; q < kChunks; ++q) {
            const uint32_t s = __reduce_add_sync(0xffffffffu, ch[q]);
            if (lane == 0) sh[w][at * kChunks + q] = s;
        }
    };
    add(h, in, 0);
    if (with_area) {
        add(area, wet, 1);
        add(cs, wet, 2);
    }
    const uint32_t nwet = __popc(__ballot_sync(0xffffffffu, wet));
    const unsigned long long o = in && h == h ? order64(h) : 0ull, o2 = o ? ~o : 0ull;
    const uint32_t xh = __reduce_max_sync(0xffffffffu, (uint32_t)(o >> 32));
    const uint32_t xl = __reduce_max_sync(0xffffffffu, (uint32_t)(o >> 32) == xh ? (uint32_t)o : 0u);
    const uint32_t nh = __reduce_max_sync(0xffffffffu, (uint32_t)(o2 >> 32));
    const uint32_t nl = __reduce_max_sync(0xffffffffu, (uint32_t)(o2 >> 32) == nh ? (uint32_t)o2 : 0u);
    if (lane == 0) {
        sh[w][kSums64 - 1] = nwet;
        sh[w][kSums64] = xl;
        sh[w][kSums64 + 1] = xh;
        sh[w][kSums64 + 2] = nl;
        sh[w][kSums64 + 3] = nh;
    }
    __syncthreads();
    const int t = threadIdx.x, l = blockIdx.x % kLanes64;
    if (t < kSums64) {
        if (t >= kChunks && t < 3 * kChunks && !with_area) return;
        const bool top = t < 3 * kChunks && t % kChunks == kChunks - 1;  // the signed chunk
        long long s = 0;
#pragma unroll
        for (int q = 0; q < NT / 32; ++q) s += top ? (long long)(int32_t)sh[q][t] : (long long)sh[q][t];
        atomicAdd(acc + t * kLanes64 + l, (unsigned long long)s);
    } else if (t < kSums64 + 2) {
        const int q0 = kSums64 + 2 * (t - kSums64);
        unsigned long long m = 0;
#pragma unroll
        for (int q = 0; q < NT / 32; ++q)
            m = max(m, (unsigned long long)sh[q][q0 + 1] << 32 | sh[q][q0]);
        atomicMax(acc + t * kLanes64 + l, m);
    }
}

// Reads, clears and sums the accumulators of iteration s and writes its
// record: one block, beside a later kernel.
template <int NT>
__device__ void cell_reduce(const StepArgs &a, const Cell64 &x, long long s) {
    __shared__ long long sum[kSums64];
    __shared__ unsigned long long mx[2];
    unsigned long long *acc = x.acc + (size_t)(s & 1) * kAcc64;
    const int lane = threadIdx.x & (kLanes64 - 1), grp = threadIdx.x / kLanes64;
    constexpr int G = NT / kLanes64;  // fields handled at a time
    static_assert(kLanes64 == 16 && (kSums64 + 2) % 2 == 0, "half-warp reductions");
#pragma unroll
    for (int f0 = 0; f0 < kSums64 + 2; f0 += G) {
        const int f = f0 + grp;
        const bool on = f < kSums64 + 2;
        unsigned long long v = on ? __ldcg(acc + f * kLanes64 + lane) : 0ull;
        if (on) acc[f * kLanes64 + lane] = 0ull;
#pragma unroll
        for (int o = kLanes64 / 2; o; o >>= 1) {
            const unsigned long long w = __shfl_down_sync(0xffffffffu, v, o, kLanes64);
            v = f < kSums64 ? v + w : max(v, w);
        }
        if (on && lane == 0) {
            if (f < kSums64)
                sum[f] = (long long)v;
            else
                mx[f - kSums64] = v;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double v[3];
        unsigned long long *out = acc + kOut64;
        if (__ldcg(out)) {
            double *inf = reinterpret_cast<double *>(out) + 1;
            for (int q = 0; q < 3; ++q) {
                v[q] = wide_value(out + 4 + q * kWide64, sum + q * kChunks) + __ldcg(inf + q);
                inf[q] = 0.0;
            }
            out[0] = 0ull;
        } else {
            for (int q = 0; q < 3; ++q) v[q] = value64(sum + q * kChunks);
        }
        finish_step(a, s, v[0], (double)sum[kSums64 - 1], mx[0] ? unorder64(mx[0]) : -INFINITY,
                    mx[1] ? unorder64(~mx[1]) : INFINITY, v[1], v[2]);
    }
}

// Forces, equilibrium and collision of one cell (slippage!, h∇p!, the force
// sum, thermal!, inclination!, equilibrium!, BGKandStream!'s collision).
struct CollideIn {
    double h, ux, uy;
    Near64 p;
    double kx, ky, ix, iy;  // thermal! and inclination! forces (GEN)
    double fq[9];           // streamed populations (τ != 1)
};
template <bool TAU1, bool G0, bool GEN, class O>
__device__ __forceinline__ void collide64(O &o, const StepArgs &a, const Cell64 &x, const CollideIn &v,
                                          double out[9]) {
    double gx, gy, sx, sy, fe[9];
    grad64(o, v.p, gx, gy);
    slip64(o, v.h, v.ux, v.uy, x.mu6, x.delta6, x.delta3sq, sx, sy);
    // the force sum (src/simulate.jl:18-19)
    double Fx = o.sub(-o.mul(v.h, gx), sx), Fy = o.sub(-o.mul(v.h, gy), sy);
    if (GEN && a.thermal) {  // Fx .= -h∇px .- slipx .- kbtx (scripts/Rivulet_stability.jl:123)
        Fx = o.sub(Fx, v.kx);
        Fy = o.sub(Fy, v.ky);
    }
    if (GEN && a.incl) {  // inclination! (src/forcing.jl:364-365)
        Fx = o.add(Fx, v.ix);
        Fy = o.add(Fy, v.iy);
    }
    feq64<G0>(o, v.h, v.ux, v.uy, x.g56, x.g15, fe);
    relax64<TAU1>(o, fe, v.fq, a.omeg, a.invtau, Fx, Fy, out);
}
template <bool TAU1, bool G0, bool GEN>
__device__ __noinline__ void cell_collide_again(const StepArgs &a, const Cell64 &x, const CollideIn &v,
                                                double out[9]) {
    Plain64 o;
    collide64<TAU1, G0, GEN>(o, a, x, v, out);
}

// Collides cell c (its fields, pressures and streamed populations in v) in
// iteration tt and stores the nine populations.
template <bool TAU1, bool G0, bool GEN>
__device__ __forceinline__ void cell_collide(const StepArgs &a, const Cell64 &x, CollideIn &v, int c,
                                             long long tt, void *dst) {
    if (GEN && a.thermal) thermal_force<true, double>(a.seed, (long long)c, tt, a.k6, v.h, a.delta, &v.kx, &v.ky);
    if (GEN && a.incl) {
        const double fac = a.incl_loop_time
                               ? 0.5 + 0.5 * tanh((double)(tt - a.incl_tstart) / (double)a.incl_tsmooth)
                               : a.incl_fixed;
        v.ix = (v.h * a.ax) * fac;
        v.iy = (v.h * a.ay) * fac;
    }
    double out[9];
    Fast64 o(x.f);
    collide64<TAU1, G0, GEN>(o, a, x, v, out);
    if (o.bad) {
        const CollideIn w = v;
        double again[9];
        cell_collide_again<TAU1, G0, GEN>(a, x, w, again);
#pragma unroll
        for (int q = 0; q < 9; ++q) out[q] = again[q];
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) StoreF64::st(dst, (int)a.pitch, q, c, out[q]);
    if (!finite64(v.h)) a.ctl->nan_flag = 1;
}

// The surface element of a wetted cell and its cos θ.
template <bool GEN>
__device__ __forceinline__ void cell_area(const StepArgs &a, const Cell64 &x, const Near64 &h, int i, int j,
                                          long long tt, double &area, double &cs) {
    Plain64 o;
    double gx, gy;
    grad64(o, h, gx, gy);
    area = sqrt(gx * gx + gy * gy + 1.0);
    if (GEN && a.theta_mode == THETA_FIELD) {
        int sx, sy;
        substrate_shift(a, tt, &sx, &sy);
        cs = reinterpret_cast<const double *>(a.cosF)[field_at(a, i, j, sx, sy)];
    } else if (GEN && a.theta_mode == THETA_WAVE) {
        cs = x.wave[a.Lx + i];
    }
}

// Seven blocks per SM (72 registers, a little spill) instead of the four that the
// compiler's 106 registers leave: with six, 256² 24.9 -> 19.9 us per iteration and
// 1000 x 1030 208 -> 195; seven against six, 1000 x 1030 183 -> 181.
template <bool TAU1, bool G0, bool GEN>
__global__ void __launch_bounds__(kCellNT, 7) cell_collide_kernel(const __grid_constant__ StepArgs a,
                                                               const __grid_constant__ Cell64 x, int k) {
    const int c = blockIdx.x * kCellNT + threadIdx.x, N = a.Lx * a.Ly;
    const int cc = c < N ? c : 0;
    const Cell g = cell_at(cc, a.Lx, a.Ly);
    // the sequence's step_base was written before the pressure kernel began
    const long long done = __ldcg(&a.ctl->step_base) + k, tt = done + 1;
    void *dst = (done & 1) ? a.fa : a.fb;
    grid_dep_wait();
    grid_dep_launch();
    const bool in = c == cc;
    double h = 0.0, area = 0.0, cs = 0.0;
    bool wet = false;
    if (in) {
        const double *hf = reinterpret_cast<const double *>(a.hF);
        CollideIn v;
        h = v.h = hf[c];
        v.ux = reinterpret_cast<const double *>(a.uxF)[c];
        v.uy = reinterpret_cast<const double *>(a.uyF)[c];
        v.p = near_cell(x.p, g);
        if (!TAU1)
            pull9<StoreF64>((done & 1) ? a.fb : a.fa, (int)a.pitch, 1, g.i, g.j, g.im, g.ip, g.jm, g.jp, v.fq);
        cell_collide<TAU1, G0, GEN>(a, x, v, c, tt, dst);
        wet = h == h && order64(h) > x.thr_key;  // h > threshold, on the integer unit
        if ((a.meas_mask & SWB_MEAS_AREA) && wet) cell_area<GEN>(a, x, near_cell(hf, g), g.i, g.j, tt, area, cs);
    }
    if (a.meas_mask) cell_measures<kCellNT>(a, x, (int)(tt & 1), in, h, area, cs, wet);
}

// u = j / h of a cell whose quotients the integers do not hold.
__device__ __noinline__ void cell_velocity_again(double h, double jx, double jy, double *ux, double *uy) {
    *ux = jx / h;
    *uy = jy / h;
}
__device__ __forceinline__ void cell_velocity(const Cell64 &x, double h, double jx, double jy, double &ux,
                                              double &uy) {
    Fast64 o(x.f);
    const uint64_t r = o.recip(h);
    ux = o.quot(jx, h, r);
    uy = o.quot(jy, h, r);
    if (o.bad) {
        double vx, vy;
        cell_velocity_again(h, jx, jy, &vx, &vy);
        ux = vx;
        uy = vy;
    }
}

// moments! of the populations the iteration wrote, pulled; the last block
// reduces the iteration's measures.
__global__ void __launch_bounds__(kCellNT) cell_moments_kernel(const StepArgs a, const Cell64 x, int k) {
    const int c = blockIdx.x * kCellNT + threadIdx.x, N = a.Lx * a.Ly;
    const int cc = c < N ? c : 0;
    const Cell g = cell_at(cc, a.Lx, a.Ly);
    const long long done = __ldcg(&a.ctl->step_base) + k;
    const void *src = (done & 1) ? a.fa : a.fb;
    grid_dep_wait();
    grid_dep_launch();
    if (a.meas_mask && blockIdx.x == gridDim.x - 1) {
        cell_reduce<kCellNT>(a, x, done + 1);
        return;
    }
    if (c != cc) return;
    double ft[9], h, jx, jy, ux, uy;
    pull9<StoreF64>(src, (int)a.pitch, 1, g.i, g.j, g.im, g.ip, g.jm, g.jp, ft);
    Fast64 o(x.f);
    moments64(o, ft, h, jx, jy);
    cell_velocity(x, h, jx, jy, ux, uy);
    reinterpret_cast<double *>(a.hF)[c] = h;
    reinterpret_cast<double *>(a.uxF)[c] = ux;
    reinterpret_cast<double *>(a.uyF)[c] = uy;
}

template <class F>
void by_kind(const StepArgs &a, F f) {  // f(TAU1, G0, GEN)
    const bool gen = step_general(a), g0 = a.g == 0.0;
    using T = std::true_type;
    using N = std::false_type;
    auto go = [&](auto t, auto g) { gen ? f(t, g, T{}) : f(t, g, N{}); };
    if (!a.tau_is_one)
        go(N{}, N{});
    else
        g0 ? go(T{}, T{}) : go(T{}, N{});
}

}  // namespace

cudaError_t launch_cell_step(const StepArgs &a, const Cell64 &x, int k, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kern, int blocks) {
        if (e != cudaSuccess) return;
        e = launch_step(kern, blocks, kCellNT, st, a, x, k);
        count_launches(1);
    };
    const int grid = (int)(((long long)a.Lx * a.Ly + kCellNT - 1) / kCellNT);
    if (a.theta_mode == THETA_WAVE) {
        go(cell_wave_kernel, (a.Lx + kCellNT - 1) / kCellNT);
        go(cell_pressure_kernel<THETA_WAVE>, grid);
    } else if (a.theta_mode == THETA_FIELD) {
        go(cell_pressure_kernel<THETA_FIELD>, grid);
    } else {
        go(cell_pressure_kernel<THETA_SCALAR>, grid);
    }
    by_kind(a, [&](auto t, auto g, auto gen) {
        go(cell_collide_kernel<decltype(t)::value, decltype(g)::value, decltype(gen)::value>, grid);
    });
    go(cell_moments_kernel, grid + (a.meas_mask ? 1 : 0));
    return e;
}

cudaError_t launch_advance(const StepArgs &a, int n, cudaStream_t st) {
    count_launches(1);
    return launch_step(advance_kernel<128>, 1, 128, st, a, n);
}

cudaError_t launch_batch_advance(const StepArgs *d_args, int count, int n, cudaStream_t st) {
    count_launches(1);
    return launch_step(batch_advance_kernel<128>, count, 128, st, d_args, n);
}

static int grid_for(long long n, int threads) {
    long long b = (n + threads - 1) / threads;
    if (b > 152LL * 32) b = 152LL * 32;
    return (int)(b < 1 ? 1 : b);
}

cudaError_t launch_moments_f64(const StepArgs &a, cudaStream_t st) {
    moments_kernel<StoreF64><<<grid_for((long long)a.Lx * a.Ly, 256), 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_fout_f64(const StepArgs &a, double *out, cudaStream_t st) {
    fout_kernel<StoreF64><<<grid_for((long long)a.Lx * a.Ly, 256), 256, 0, st>>>(a, out);
    return cudaGetLastError();
}

cudaError_t launch_thermal_field_f64(const StepArgs &a, long long t, double *fx, double *fy,
                                     cudaStream_t st) {
    thermal_field_kernel<StoreF64><<<grid_for((long long)a.Lx * a.Ly, 256), 256, 0, st>>>(a, t, fx, fy);
    return cudaGetLastError();
}

cudaError_t launch_pressure_now_f64(const StepArgs &a, double *out, cudaStream_t st) {
    pressure_now_kernel<StoreF64><<<grid_for((long long)a.Lx * a.Ly, 256), 256, 0, st>>>(a, out);
    return cudaGetLastError();
}

cudaError_t launch_batch_step_f64(int nt, bool gen, const StepArgs *d_args, const TileRef *d_tiles,
                                  int ntiles, int grid, int k, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    if (gen)
        DISPATCH_NT(nt, e = launch_step(batch_step_kernel<StoreF64, NT, true>, grid, NT, st, d_args, d_tiles, ntiles, k));
    else
        DISPATCH_NT(nt, e = launch_step(batch_step_kernel<StoreF64, NT, false>, grid, NT, st, d_args, d_tiles, ntiles, k));
    return e;
}

int batch_blocks_per_sm_f64(int nt) {
    int n = 0;
    DISPATCH_NT(nt, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_step_kernel<StoreF64, NT, false>, NT, 0));
    return n < 1 ? 1 : n;
}

// ------------------------------------------------------------ θ fields
// cospi(θ) and κ of a θ field.  The host's cosine runs in long double, which
// is 128-bit software arithmetic on Arm hosts: 0.4 us per value, 65 ms for a
// 301 x 257 field, more than the 400 iterations that follow (12 ms with this
// kernel, 79 ms with the host's loop).  Here every cell's cosine is a
// Taylor series in pairs of Float64 (about 2^-100) after an exact reduction of
// θ to [0, 1/4], rounded once.  Where the rounding could depend on the last
// bits of either evaluation, *hard is set and the host computes the field.
namespace {

struct DD {
    double h, l;
};
__device__ __forceinline__ DD fast_sum(double a, double b) {  // |a| >= |b|
    const double s = a + b;
    return {s, b - (s - a)};
}
__device__ __forceinline__ DD dd_mul(DD a, DD b) {
    const double p = a.h * b.h;
    double e = __fma_rn(a.h, b.h, -p);
    e = __fma_rn(a.h, b.l, e);
    return fast_sum(p, __fma_rn(a.l, b.h, e));
}
__device__ __forceinline__ DD dd_add(DD a, DD b) {  // accurate sum (two_sum on both words)
    double s, e, t, r;
    two_sum(a.h, b.h, s, e);
    two_sum(a.l, b.l, t, r);
    const DD u = fast_sum(s, e + t);
    return fast_sum(u.h, u.l + r);
}

// (-1)^k / (2k)! and (-1)^k / (2k + 1)!, as pairs: the next terms are below
// 2^-117 of the sum for arguments up to π/4
constexpr int kTerms = 15;
__constant__ DD kCosTerm[kTerms] = {
    {1.0, 0.0},
    {-0x1.0000000000000p-1, 0.0},
    {0x1.5555555555555p-5, 0x1.5555555555555p-59},
    {-0x1.6c16c16c16c17p-10, 0x1.f49f49f49f49fp-65},
    {0x1.a01a01a01a01ap-16, 0x1.a01a01a01a01ap-76},
    {-0x1.27e4fb7789f5cp-22, -0x1.cbbc05b4fa99ap-76},
    {0x1.1eed8eff8d898p-29, -0x1.2aec959e14c06p-83},
    {-0x1.93974a8c07c9dp-37, -0x1.05d6f8a2efd1fp-92},
    {0x1.ae7f3e733b81fp-45, 0x1.1d8656b0ee8cbp-101},
    {-0x1.6827863b97d97p-53, -0x1.eec01221a8b0bp-107},
    {0x1.e542ba4020225p-62, 0x1.ea72b4afe3c2fp-120},
    {-0x1.0ce396db7f853p-70, 0x1.aebcdbd20331cp-124},
    {0x1.f2cf01972f578p-80, -0x1.9ada5fcc1ab14p-135},
    {-0x1.88e85fc6a4e5ap-89, 0x1.71c37ebd16540p-143},
    {0x1.0a18a2635085dp-98, 0x1.b9e2e28e1aa54p-153},
};
__constant__ DD kSinTerm[kTerms] = {
    {1.0, 0.0},
    {-0x1.5555555555555p-3, -0x1.5555555555555p-57},
    {0x1.1111111111111p-7, 0x1.1111111111111p-63},
    {-0x1.a01a01a01a01ap-13, -0x1.a01a01a01a01ap-73},
    {0x1.71de3a556c734p-19, -0x1.c154f8ddc6c00p-73},
    {-0x1.ae64567f544e4p-26, 0x1.c062e06d1f209p-80},
    {0x1.6124613a86d09p-33, 0x1.f28e0cc748ebep-87},
    {-0x1.ae7f3e733b81fp-41, -0x1.1d8656b0ee8cbp-97},
    {0x1.952c77030ad4ap-49, 0x1.ac981465ddc6cp-103},
    {-0x1.2f49b46814157p-57, -0x1.2650f61dbdcb4p-112},
    {0x1.71b8ef6dcf572p-66, -0x1.d043ae40c4647p-120},
    {-0x1.761b41316381ap-75, 0x1.3423c7d91404fp-130},
    {0x1.3f3ccdd165fa9p-84, -0x1.58ddadf344487p-139},
    {-0x1.d1ab1c2dccea3p-94, -0x1.054d0c78aea14p-149},
    {0x1.259f98b4358adp-103, 0x1.eaf8c39dd9bc5p-157},
};

__device__ double cospi_rounded(double x, bool &hard) {
    double r = fmod(fabs(x), 2.0);  // exact, as are the reductions below
    if (r > 1.0) r = 2.0 - r;
    if (r == 0.0) return 1.0;
    if (r == 1.0) return -1.0;
    if (r == 0.5) return 0.0;
    const bool neg = r > 0.5;
    if (neg) r = 1.0 - r;
    const bool sine = r > 0.25;
    if (sine) r = 0.5 - r;
    // y = π r, π in three words (the third only rounds the second product)
    const double ph = 0x1.921fb54442d18p+1, pl = 0x1.1a62633145c07p-53, pll = -0x1.f1976b7ed8fbcp-109;
    const double q = ph * r;
    const DD y = fast_sum(q, __fma_rn(ph, r, -q) + __fma_rn(pl, r, pll * r));
    const DD z = dd_mul(y, y);
    const DD *c = sine ? kSinTerm : kCosTerm;
    DD s = c[kTerms - 1];
    for (int k = kTerms - 2; k >= 0; --k) s = dd_add(c[k], dd_mul(s, z));
    if (sine) s = dd_mul(s, y);
    // the nearest double unless 2^-98 of the value, or the long double's own
    // argument error (2^-112, taken 2^-108), could carry it over a midpoint
    const double e = fmax(fabs(s.h) * 0x1p-98, 0x1p-108);
    if (!(s.h + (s.l + e) == s.h && s.h + (s.l - e) == s.h)) hard = true;
    return neg ? -s.h : s.h;
}

template <class R>
__global__ void __launch_bounds__(128) theta_field_kernel(const double *theta, R *kap, R *cs, long long N,
                                                          int n, int m, double hmin, int *hard) {
    const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (c >= N) return;
    bool bad = false;
    const double co = cospi_rounded(theta[c], bad);
    // κ left to right (src/pressure.jl:141-147)
    double k = 1.0 - co;
    k = k * (double)(n - 1);
    k = k * (double)(m - 1);
    kap[c] = (R)(k / ((double)(n - m) * hmin));
    cs[c] = (R)co;
    if (bad) *hard = 1;
}

}  // namespace

cudaError_t launch_theta_field(const double *theta, void *kap, void *cs, bool is_double, long long N, int n,
                               int m, double hmin, int *hard, cudaStream_t st) {
    const unsigned blocks = (unsigned)((N + 127) / 128);
    count_launches(1);
    if (is_double)
        theta_field_kernel<double><<<blocks, 128, 0, st>>>(theta, (double *)kap, (double *)cs, N, n, m, hmin, hard);
    else
        theta_field_kernel<float><<<blocks, 128, 0, st>>>(theta, (float *)kap, (float *)cs, N, n, m, hmin, hard);
    return cudaGetLastError();
}

// ------------------------------------------------------------ plain path
// One kernel per reference function, Float64, same per-element operations.
// Neighbour (i±1, j±1) indexing replaces the reference's circshift! copies.
#define PLAIN_LOOP(s)                                                              \
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < (s).N; \
         c += (long long)gridDim.x * blockDim.x)

struct Nb {
    long long c, ip, im, jp, jm, ipjp, imjp, imjm, ipjm;  // reference names
};
__device__ __forceinline__ Nb neighbours(long long c, int Lx, int Ly) {
    const int i = (int)(c % Lx), j = (int)(c / Lx);
    const int im1 = i == 0 ? Lx - 1 : i - 1, ip1 = i == Lx - 1 ? 0 : i + 1;
    const int jm1 = j == 0 ? Ly - 1 : j - 1, jp1 = j == Ly - 1 ? 0 : j + 1;
    Nb n;
    n.c = c;
    n.ip = (long long)j * Lx + im1;      // h[i-1, j]
    n.im = (long long)j * Lx + ip1;      // h[i+1, j]
    n.jp = (long long)jm1 * Lx + i;      // h[i, j-1]
    n.jm = (long long)jp1 * Lx + i;      // h[i, j+1]
    n.ipjp = (long long)jm1 * Lx + im1;  // h[i-1, j-1]
    n.imjp = (long long)jm1 * Lx + ip1;  // h[i+1, j-1]
    n.imjm = (long long)jp1 * Lx + ip1;  // h[i+1, j+1]
    n.ipjm = (long long)jp1 * Lx + im1;  // h[i-1, j+1]
    return n;
}

__device__ __forceinline__ Near64 near_of(const double *v, const Nb &b) {
    return {v[b.ip], v[b.jp], v[b.im], v[b.jm], v[b.ipjp], v[b.imjp], v[b.imjm], v[b.ipjm]};
}

// An op's cell with the integer unit's help (Fast64), and out of line again in
// Float64 where that met a number it does not hold.  f(o, r): the op with
// operations o and results r[0 .. K).
template <int K, class F>
__device__ __noinline__ void plain_again(const F &f, double *r) {
    Plain64 o;
    f(o, r);
}
template <int K, class F>
__device__ __forceinline__ void plain_cell(const Fma64 &g, const F &f, double (&r)[K]) {
    Fast64 o(g);
    f(o, r);
    if (o.bad) {
        const F copy = f;
        double again[K];
        plain_again<K>(copy, again);
#pragma unroll
        for (int q = 0; q < K; ++q) r[q] = again[q];
    }
}

// (sx, sy): offset of a moving θ field (0 for a fixed one)
__global__ void k_filmpressure(PlainState s, Fma64 g, const double *kapF, double kap, double gamma,
                               int n, int m, double hmin, double hcrit, int sx, int sy) {
    grid_dep_wait();
    grid_dep_launch();
    PLAIN_LOOP(s) {
        const Nb b = neighbours(c, s.Lx, s.Ly);
        double k = kap;
        if (kapF) {
            int i = (int)(c % s.Lx) - sx, j = (int)(c / s.Lx) - sy;
            if (i < 0) i += s.Lx;
            if (j < 0) j += s.Ly;
            k = kapF[(long long)j * s.Lx + i];
        }
        const double h = s.h[c];
        const Near64 v = near_of(s.h, b);
        double r[1];
        plain_cell<1>(g, [=](auto &o, double *p) { p[0] = pressure64(o, h, v, k, gamma, hmin, hcrit, n, m); }, r);
        s.p[c] = r[0];
    }
}

__global__ void k_hgradp(PlainState s, Fma64 g) {
    grid_dep_wait();
    grid_dep_launch();
    PLAIN_LOOP(s) {
        const Near64 v = near_of(s.p, neighbours(c, s.Lx, s.Ly));
        const double h = s.h[c];
        double r[2];
        plain_cell<2>(g, [=](auto &o, double *q) {
            double gx, gy;
            grad64(o, v, gx, gy);
            q[0] = o.mul(h, gx);
            q[1] = o.mul(h, gy);
        }, r);
        s.hgx[c] = r[0];
        s.hgy[c] = r[1];
    }
}

__global__ void k_slippage(PlainState s, Fma64 g, double delta6, double delta3sq, double mu6) {
    grid_dep_wait();
    grid_dep_launch();
    PLAIN_LOOP(s) {
        const double h = s.h[c], ux = s.ux[c], uy = s.uy[c];
        double r[2];
        plain_cell<2>(g, [=](auto &o, double *q) { slip64(o, h, ux, uy, mu6, delta6, delta3sq, q[0], q[1]); }, r);
        s.sx[c] = r[0];
        s.sy[c] = r[1];
    }
}

__global__ void k_force_sum(PlainState s, Fma64) {
    grid_dep_wait();
    grid_dep_launch();
    PLAIN_LOOP(s) {
        s.Fx[c] = -s.hgx[c] - s.sx[c];
        s.Fy[c] = -s.hgy[c] - s.sy[c];
    }
}

// Fx .-= kbtx, Fy .-= kbty with thermal!'s forces of iteration t
// (src/forcing.jl:297-311; the force sum of scripts/Rivulet_stability.jl:123).
__global__ void k_thermal(PlainState s, Fma64, double k6, double delta, unsigned long long seed,
                          long long t) {
    grid_dep_wait();
    grid_dep_launch();
    PLAIN_LOOP(s) {
        double kx, ky;
        thermal_force<true, double>(seed, c, t, k6, s.h[c], delta, &kx, &ky);
        s.Fx[c] = s.Fx[c] - kx;
        s.Fy[c] = s.Fy[c] - ky;
    }
}

__global__ void k_inclination(PlainState s, Fma64, double ax, double ay, double fac) {
    grid_dep_wait();
    grid_dep_launch();
    PLAIN_LOOP(s) {
        s.Fx[c] = s.Fx[c] + (s.h[c] * ax) * fac;
        s.Fy[c] = s.Fy[c] + (s.h[c] * ay) * fac;
    }
}

template <bool G0>
__global__ void k_equilibrium(PlainState s, Fma64 g, double g56, double g15) {
    grid_dep_wait();
    grid_dep_launch();
    PLAIN_LOOP(s) {
        const double h = s.h[c], ux = s.ux[c], uy = s.uy[c];
        double r[10];
        plain_cell<10>(g, [=](auto &o, double *q) {
            double fe[9];
            feq64<G0>(o, h, ux, uy, g56, g15, fe);
            for (int k = 0; k < 9; ++k) q[k] = fe[k];
            q[9] = o.add(o.mul(ux, ux), o.mul(uy, uy));
        }, r);
        s.vsq[c] = r[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) s.feq[q * s.N + c] = r[q];
    }
}

// BGKandStream! in one pass: the collision of every cell, each population
// stored where it streams to (circshift!(ft_q, fo_q, c_q)).  The reference's
// ftemp equals its fout between ops, so the other buffer takes the result
// and the two are exchanged, or (after a capture) the result is copied back.
__global__ void k_bgk_stream(PlainState s, Fma64 g, double omeg, double invtau) {
    const int CX[9] = {0, 1, 0, -1, 0, 1, -1, -1, 1};
    const int CY[9] = {0, 0, 1, 0, -1, 1, 1, -1, -1};
    grid_dep_wait();
    grid_dep_launch();
    PLAIN_LOOP(s) {
        const double Fx = s.Fx[c], Fy = s.Fy[c];
        struct {
            double f[9], fe[9];
        } v;
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            v.f[q] = s.fout[q * s.N + c];
            v.fe[q] = s.feq[q * s.N + c];
        }
        double r[9];
        plain_cell<9>(g, [=](auto &o, double *out) {
            double w[9];
            relax64<false>(o, v.fe, v.f, omeg, invtau, Fx, Fy, w);
            for (int q = 0; q < 9; ++q) out[q] = w[q];
        }, r);
        const int i = (int)(c % s.Lx), j = (int)(c / s.Lx);
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const int di = wrapc(i + CX[q], s.Lx), dj = wrapc(j + CY[q], s.Ly);
            s.ftemp[q * s.N + (long long)dj * s.Lx + di] = r[q];
        }
    }
}

__global__ void k_copy_streamed(PlainState s) {
    grid_dep_wait();
    grid_dep_launch();
    PLAIN_LOOP(s) {
#pragma unroll
        for (int q = 0; q < 9; ++q) s.fout[q * s.N + c] = s.ftemp[q * s.N + c];
    }
}

__global__ void k_moments(PlainState s, Fma64 g) {
    grid_dep_wait();
    grid_dep_launch();
    PLAIN_LOOP(s) {
        struct {
            double f[9];
        } v;
#pragma unroll
        for (int q = 0; q < 9; ++q) v.f[q] = s.fout[q * s.N + c];
        double r[3];
        plain_cell<3>(g, [=](auto &o, double *q) {
            double h, jx, jy;
            moments64(o, v.f, h, jx, jy);
            const uint64_t r = o.recip(h);
            q[0] = h;
            q[1] = o.quot(jx, h, r);
            q[2] = o.quot(jy, h, r);
        }, r);
        s.h[c] = r[0];
        s.ux[c] = r[1];
        s.uy[c] = r[2];
    }
}

// Blocks of 64 threads: a lattice of 128 x 96 cells then has a warp for every SM
// quarter, where blocks of 256 kept two thirds of the SMs idle.  The launches
// overlap (launch_step): an op's kernel after another takes 4.1 us without
// that, however short it is.
constexpr int kPlainNT = 64;
#define PLAIN_LAUNCH(kernel, s, st, ...)                                                               \
    do {                                                                                               \
        count_launches(1);                                                                             \
        return launch_step(kernel, grid_for((s).N, kPlainNT), kPlainNT, st, s, Fma64{1.0}, ##__VA_ARGS__); \
    } while (0)

cudaError_t plain_filmpressure(const PlainState &s, const double *kapF, double kap, double gamma,
                               int n, int m, double hmin, double hcrit, int sx, int sy,
                               cudaStream_t st) {
    PLAIN_LAUNCH(k_filmpressure, s, st, kapF, kap, gamma, n, m, hmin, hcrit, sx, sy);
}
cudaError_t plain_hgradp(const PlainState &s, cudaStream_t st) { PLAIN_LAUNCH(k_hgradp, s, st); }
cudaError_t plain_slippage(const PlainState &s, double delta, double mu, cudaStream_t st) {
    PLAIN_LAUNCH(k_slippage, s, st, 6.0 * delta, 3.0 * (delta * delta), 6.0 * mu);
}
cudaError_t plain_force_sum(const PlainState &s, cudaStream_t st) {
    PLAIN_LAUNCH(k_force_sum, s, st);
}
cudaError_t plain_thermal(const PlainState &s, double k6, double delta, unsigned long long seed,
                          long long t, cudaStream_t st) {
    PLAIN_LAUNCH(k_thermal, s, st, k6, delta, seed, t);
}
cudaError_t plain_inclination(const PlainState &s, double ax, double ay, double fac,
                              cudaStream_t st) {
    PLAIN_LAUNCH(k_inclination, s, st, ax, ay, fac);
}
cudaError_t plain_equilibrium(const PlainState &s, double g, cudaStream_t st) {
    auto *const kern = g == 0.0 ? k_equilibrium<true> : k_equilibrium<false>;
    PLAIN_LAUNCH(kern, s, st, (5.0 / 6.0) * g, 1.5 * g);
}
// A captured op that uses fout is replayed with the address of its capture, any
// number of times and with calls outside the graph in between, so from the first
// such op on fout is not exchanged any more.
static cudaError_t note_capture(bool &captured, cudaStream_t st) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (captured) return cudaSuccess;
    const cudaError_t e = cudaStreamIsCapturing(st, &cap);
    captured = e == cudaSuccess && cap != cudaStreamCaptureStatusNone;
    return e;
}
cudaError_t plain_bgk_stream(PlainState &s, bool &captured, double omeg, double invtau, cudaStream_t st) {
    cudaError_t e = note_capture(captured, st);
    if (e != cudaSuccess) return e;
    count_launches(1);
    e = launch_step(k_bgk_stream, grid_for(s.N, kPlainNT), kPlainNT, st, s, Fma64{1.0}, omeg, invtau);
    if (e != cudaSuccess) return e;
    if (captured) {  // the result goes back to where it was read
        count_launches(1);
        return launch_step(k_copy_streamed, grid_for(s.N, kPlainNT), kPlainNT, st, s);
    }
    double *f = s.fout;
    s.fout = s.ftemp;
    s.ftemp = f;
    return e;
}
cudaError_t plain_moments(const PlainState &s, bool &captured, cudaStream_t st) {
    const cudaError_t e = note_capture(captured, st);
    if (e != cudaSuccess) return e;
    PLAIN_LAUNCH(k_moments, s, st);
}

// ------------------------------------------------------------ measures
// Grid-stride partials per block, then the last block (ticket) reduces the
// partials in a fixed order and writes one Record.  Per-cell values are
// computed in the height's type R (as the fused step computes them); the
// block sums are Float64 for every R.  cos θ of a wetted cell comes from the
// θ source `cs`: a scalar, a (possibly moving) field, or the θ wave, with the
// fused step's formulas for its iteration cs.t.
template <class R>
__device__ __forceinline__ R cos_of_cell(const CosSrc &cs, long long c, int Lx, int Ly) {
    const int i = (int)(c % Lx), j = (int)(c / Lx);
    if (cs.mode == THETA_FIELD) {
        const int fi = cs.sx ? (i - cs.sx < 0 ? i - cs.sx + Lx : i - cs.sx) : i;
        const int fj = cs.sy ? (j - cs.sy < 0 ? j - cs.sy + Ly : j - cs.sy) : j;
        return reinterpret_cast<const R *>(cs.cosF)[(long long)fj * Lx + fi];
    }
    return wave_kap_cos<R>(R(cs.theta0), R(cs.dtheta), R(cs.wave_v), i, cs.t, Lx, 2, 1, R(1)).cs;
}

template <class R>
__global__ void __launch_bounds__(256) measure_kernel(const R *h, int Lx, int Ly, R thr,
                                                      const CosSrc cs, double *scratch,
                                                      unsigned int *ticket, Record *rec,
                                                      long long t) {
    __shared__ PartT<double> red[8];
    __shared__ int last;
    const long long N = (long long)Lx * Ly;
    const bool percell = cs.mode != THETA_SCALAR;
    PartT<double> p;
    part_init(p);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N;
         c += (long long)gridDim.x * blockDim.x) {
        const R v = h[c];
        mass_add(p, (double)v);
        const bool wet = v > thr;
        p.wet += wet ? 1 : 0;
        p.hmax = fmax(p.hmax, (double)v);
        p.hmin = fmin(p.hmin, (double)v);
        if (wet) {
            const Nb b = neighbours(c, Lx, Ly);
            R gx, gy;
            grad9<R>(h[b.ip], h[b.jp], h[b.im], h[b.jm], h[b.ipjp], h[b.imjp], h[b.imjm],
                     h[b.ipjm], gx, gy);
            p.area += (double)R(sqrt(gx * gx + gy * gy + R(1)));
            if (percell) p.cossum += (double)cos_of_cell<R>(cs, c, Lx, Ly);
        }
    }
    PartT<double> tot = block_reduce<256>(p, red);
    if (threadIdx.x == 0) {
        double *pp = scratch + (size_t)blockIdx.x * kNPart;
        pp[0] = tot.mhi + tot.mlo;
        pp[1] = (double)tot.wet;
        pp[2] = tot.hmax;
        pp[3] = tot.hmin;
        pp[4] = tot.area;
        pp[5] = tot.cossum;
        __threadfence();
        last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    PartT<double> acc;
    part_init(acc);
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
        const double *pp = scratch + (size_t)b * kNPart;
        PartT<double> q;
        q.mhi = __ldcg(pp + 0);
        q.mlo = 0.0;
        q.wet = (int)__ldcg(pp + 1);
        q.hmax = __ldcg(pp + 2);
        q.hmin = __ldcg(pp + 3);
        q.area = __ldcg(pp + 4);
        q.cossum = __ldcg(pp + 5);
        part_merge(acc, q);
    }
    acc = block_reduce<256>(acc, red);
    if (threadIdx.x == 0) {
        rec->t = t;
        rec->mass = acc.mhi + acc.mlo;
        rec->wetted = (double)acc.wet;
        rec->hmax = acc.hmax;
        rec->hmin = acc.hmin;
        rec->area = acc.area;
        rec->cos_sum = percell ? acc.cossum : (double)acc.wet * cs.cos_theta;
        *ticket = 0u;
    }
}

int measure_blocks(long long N) {
    long long b = (N + 255) / 256;
    if (b > 1024) b = 1024;
    return (int)(b < 1 ? 1 : b);
}

cudaError_t launch_measure(const void *h, int is_double, int Lx, int Ly, double hthresh,
                           const CosSrc &cs, double *scratch, unsigned int *ticket, Record *rec,
                           long long t, cudaStream_t st) {
    const int blocks = measure_blocks((long long)Lx * Ly);
    count_launches(1);
    if (is_double)
        measure_kernel<double><<<blocks, 256, 0, st>>>((const double *)h, Lx, Ly, hthresh, cs,
                                                       scratch, ticket, rec, t);
    else
        measure_kernel<float><<<blocks, 256, 0, st>>>((const float *)h, Lx, Ly, (float)hthresh,
                                                      cs, scratch, ticket, rec, t);
    return cudaGetLastError();
}

cudaError_t launch_measure(const void *h, int is_double, int Lx, int Ly, double hthresh,
                           const void *cosF, double cos_theta, double *scratch, unsigned int *ticket,
                           Record *rec, long long t, cudaStream_t st) {
    CosSrc cs{};
    cs.mode = cosF ? THETA_FIELD : THETA_SCALAR;
    cs.cosF = cosF;
    cs.cos_theta = cos_theta;
    return launch_measure(h, is_double, Lx, Ly, hthresh, cs, scratch, ticket, rec, t, st);
}

}  // namespace swb
