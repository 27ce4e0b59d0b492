// swb_lattice.h -- device memory of one lattice inside a batch or a server:
// layout, initialisation and host<->device field transfer.  Internal.
#pragma once
#include <cuda_fp16.h>

#include <cmath>
#include <string>
#include <unordered_map>
#include <utility>
#include <vector>

#include "swb_internal.h"

namespace swb {

double host_cospi_shared(double x);
double host_kappa_shared(double theta, int n, int m, double hmin);

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
inline long long pitch_for(long long N) { return (N + 63) / 64 * 64; }
inline int real_bytes_of(int precision) { return precision == SWB_F64 ? 8 : 4; }
inline size_t fbuf_bytes_of(int precision, long long pitch) {
    switch (precision) {
        case SWB_F64: return (size_t)9 * pitch * 8;
        case SWB_F32: return (size_t)9 * pitch * 4;
        default: return (size_t)pitch * 4 + (size_t)8 * pitch * 2;
    }
}

// Byte offsets of one lattice's buffers inside a contiguous block.
struct LatticeLayout {
    size_t fa, fb, h, ux, uy, partials, ctl, total;
};

inline LatticeLayout lattice_layout(const swb_params &p, int precision) {
    const long long N = (long long)p.Lx * p.Ly, pitch = pitch_for(N);
    const long long tiles = max_tiles(p.Lx, p.Ly);
    LatticeLayout L{};
    size_t o = 0;
    const size_t fb = align256(fbuf_bytes_of(precision, pitch));
    const size_t fld = align256((size_t)N * real_bytes_of(precision));
    L.fa = o; o += fb;
    L.fb = o; o += fb;
    L.h = o; o += fld;
    L.ux = o; o += fld;
    L.uy = o; o += fld;
    L.partials = o; o += align256((size_t)2 * tiles * kNPart * 8);
    L.ctl = o; o += align256(sizeof(Control));
    L.total = o;
    return L;
}

// Strip rows of batched and served lattices: the batch has parallelism from
// its many lattices, so strips can be tall (fewer halo rows re-pulled; on
// GB300 the ensemble ran 26 GLUPS at 124x4 strips, 45 GLUPS at 60x32).
constexpr int kBatchRows = 32;

// Rows of the strips that cover Ly rows with as few strips of at most `cap` rows
// as that takes, all about equally high.
inline int balanced_rows(int Ly, int cap) {
    const int strips = (Ly + cap - 1) / cap;
    return (Ly + strips - 1) / strips;
}
// Lattices (Lx, Ly) cut into strips of w columns, by height: (Ly, column strips of
// all lattices that high).  An estimate is made for each of up to 126 strip sizes
// whenever a server's resident set changes, and takes a pass over the heights
// instead of the lattices (a server's 3000 requests of 32 to 64 columns and rows
// that join and leave: 0.51 s with passes over the lattices, 0.32 s so).
using StripColumns = std::vector<std::pair<int, double>>;
inline StripColumns strip_columns(const std::vector<std::pair<int, int>> &sizes, int w) {
    std::unordered_map<int, double> of;
    for (const auto &p : sizes) of[p.second] += (double)((p.first + w - 1) / w);
    return StripColumns(of.begin(), of.end());
}
// Columns of the pair strips of geometry nt.
inline int pair_columns(int nt) { return -2 * nt - 4; }
// Estimated time of an iteration of many lattices on pair strips of geometry nt
// and at most cap rows, balanced: launch and drain, then waves of
// up to `slots` CTAs per SM, each as long as a march over the tallest strip.
// c CTAs of 64 threads (or 2 c of 32) on an SM take 0.655 us per row up to
// c = 1.4 and 0.11 us more for each further one.  Measured on GB300 with the θ
// wave: 64 to 4M cells in 1 to 32 lattices, 18 geometries each; the estimate is
// within 20 % of all, and the strips it picks within 15 % of the best.  E.g. a
// 1024² lattice 50.7 us with 64 rows, 21.0 with 8; eight of 32k to 147k cells
// 51.1 and 17.7 (60 columns, 6 rows).
inline double pair_iteration_us(const StripColumns &columns, int nt, int cap, int sms, int slots) {
    double strips = 0.0;
    int tallest = 0;
    for (const auto &p : columns) {
        const int h = balanced_rows(p.first, cap);
        tallest = h > tallest ? h : tallest;
        strips += p.second * (double)((p.first + h - 1) / h);
    }
    const double c = strips / sms, waves = std::floor(c / slots), rest = c - slots * waves;
    auto row = [nt](double c) { return 0.655 * (1.0 + 0.17 * std::fmax(0.0, c * (-nt / 64.0) - 1.4)); };
    return 4.7 + (tallest + 4) * (waves * row(slots) + (rest > 0.0 ? row(rest) : 0.0));
}

// Step arguments of a lattice whose buffers start at `base`; strips of
// nt threads and `rows` rows (capped at the lattice height).
inline StepArgs lattice_args(const swb_params &p, int precision, char *base, const LatticeLayout &L,
                             int nt = kBatchNT, int rows = kBatchRows) {
    StepArgs a{};
    a.Lx = p.Lx;
    a.Ly = p.Ly;
    a.pitch = pitch_for((long long)p.Lx * p.Ly);
    a.fa = base + L.fa;
    a.fb = base + L.fb;
    a.hF = base + L.h;
    a.uxF = base + L.ux;
    a.uyF = base + L.uy;
    a.partials = (double *)(base + L.partials);
    a.part_stride = (int)max_tiles(p.Lx, p.Ly);
    a.ctl = (Control *)(base + L.ctl);
    a.gamma = p.gamma;
    a.hmin = p.hmin;
    a.hcrit = p.hcrit;
    a.delta = p.delta;
    a.mu = p.mu;
    a.g = p.g;
    a.invtau = 1.0 / p.tau;
    a.omeg = 1.0 - 1.0 / p.tau;
    a.tau_is_one = (p.tau == 1.0);
    a.n = p.n;
    a.m = p.m;
    a.theta_mode = THETA_SCALAR;
    a.kap = host_kappa_shared(p.theta, p.n, p.m, p.hmin);
    a.cos_theta = host_cospi_shared(p.theta);
    int h = rows < p.Ly ? rows : p.Ly;  // one CTA width serves every lattice of a batch
    if (h < kMinRows) h = kMinRows;
    set_geometry(a, nt, h);
    a.hthresh = 0.055;
    a.thermal = p.kbt > 0.0 ? 1 : 0;
    a.k6 = ((2.0 * p.kbt) * p.mu) * 6.0;  // src/forcing.jl:300-302, left to right
    a.seed = 0;
    a.mass_fixed = (precision == SWB_F32 || precision == SWB_F16) ? 1 : 0;
    a.mass_corr = (precision == SWB_F16) ? 1 : 0;
    a.records = nullptr;
    a.rec_cap = 0;
    a.meas_mask = 0;
    a.stop_at = 0x7fffffffffffffffLL;  // runs until told otherwise
    return a;
}

inline void set_wave(StepArgs &a, double theta0, double dtheta, double v) {
    if (dtheta == 0.0 && v == 0.0) {
        a.theta_mode = THETA_SCALAR;
        a.kap = host_kappa_shared(theta0, a.n, a.m, a.hmin);
        a.cos_theta = host_cospi_shared(theta0);
    } else {
        a.theta_mode = THETA_WAVE;
        a.theta0 = theta0;
        a.dtheta = dtheta;
        a.wave_v = v;
    }
}

// Zero populations, h = 1 (or h0), u = 0, fresh control block.  Async on st.
cudaError_t lattice_init(const StepArgs &a, int precision, const LatticeLayout &L,
                         const double *h0_host, cudaStream_t st);
// Upload a host Float64 height into the field (converted to the compute type)
// and mark the lattice fresh.  Async on st; `staging` must stay alive until
// the stream passes this point (pinned or synchronised by the caller).
cudaError_t lattice_upload_height(const StepArgs &a, int precision, const double *h_host,
                                  void *staging, cudaStream_t st);
// Height of the lattice into host memory (runs the moments kernel first
// unless the fields are the current source).  Synchronises st.
cudaError_t lattice_download_height(const StepArgs &a, int precision, bool fields_current,
                                    double *h_host, cudaStream_t st);

}  // namespace swb
