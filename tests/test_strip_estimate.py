"""The estimate that strip geometries of many lattices are chosen by (host code):
it is that of a sum over the lattices, and trying every strip size takes about as
long as looking at the lattices once (no GPU)."""
import subprocess
import sys

import pytest

import swalbe_gb300  # noqa: F401  (its build module is hidden by the function of that name)

B = sys.modules["swalbe_gb300.build"]

SOURCE = r"""
#include <chrono>
#include <cstdio>
#include "swb_lattice.h"
using namespace swb;
static double over_lattices(const std::vector<std::pair<int, int>> &sizes, int nt, int cap, int sms, int slots) {
    const int w = -2 * nt - 4;
    double strips = 0.0;
    int tallest = 0;
    for (const auto &p : sizes) {
        const int h = balanced_rows(p.second, cap);
        tallest = h > tallest ? h : tallest;
        strips += (double)((p.first + w - 1) / w) * (double)((p.second + h - 1) / h);
    }
    const double c = strips / sms, waves = std::floor(c / slots), rest = c - slots * waves;
    auto row = [nt](double c) { return 0.655 * (1.0 + 0.17 * std::fmax(0.0, c * (-nt / 64.0) - 1.4)); };
    return 4.7 + (tallest + 4) * (waves * row(slots) + (rest > 0.0 ? row(rest) : 0.0));
}
static double seconds() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}
int main(int argc, char **argv) {
    unsigned n = (unsigned)atoi(argv[1]), x = 1;
    std::vector<std::pair<int, int>> sizes;
    for (unsigned i = 0; i < n; ++i) {
        x = x * 1664525u + 1013904223u;
        sizes.push_back({2 + (int)(x >> 22), 1 + (int)(x >> 8) % 300});
    }
    int wrong = 0;
    double sum = 0.0, t0 = seconds();
    for (int nt : {-64, -32}) sum += pair_iteration_us(strip_columns(sizes, pair_columns(nt)), nt, 64, 152, 9);
    const double once = seconds() - t0;
    t0 = seconds();
    for (int nt : {-64, -32}) {
        const StripColumns columns = strip_columns(sizes, pair_columns(nt));
        for (int cap = 64; cap >= 2; --cap) sum += pair_iteration_us(columns, nt, cap, 152, 9);
    }
    const double all = seconds() - t0;
    for (int nt : {-64, -32})
        for (int cap : {64, 33, 17, 2})
            wrong += pair_iteration_us(strip_columns(sizes, pair_columns(nt)), nt, cap, 152, 9) !=
                     over_lattices(sizes, nt, cap, 152, 9);
    printf("%d %.9f %.9f %g\n", wrong, once, all, sum);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("strips")
    (d / "e.cu").write_text(SOURCE)
    subprocess.check_call([B.nvcc(), *B.ARCH, *B.COMMON, "-I", B.CSRC, "-o", str(d / "e"), str(d / "e.cu")])
    return str(d / "e")


@pytest.mark.parametrize("n", [1, 2, 37, 5000])
def test_the_sum_over_the_lattices(program, n):
    assert subprocess.check_output([program, str(n)]).split()[0] == b"0"


def test_all_sizes_take_about_as_long_as_one(program):
    _, once, every, _ = (float(v) for v in subprocess.check_output([program, "200000"]).split())
    assert every < 20 * once  # 63 with a pass over the lattices for each
