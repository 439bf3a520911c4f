"""The screening's table look-ups on the CPU: the device functions of radial.cuh compiled as host code with
undefined-behaviour checks, over the tables of tables.cpp, every read checked against their bounds.

libgrpp's quotient of two Bessel functions is 0/0 for orders l >= 6 at 1e-7 < x < 0.005, so the fixed
point, the arguments k r and 1/(k r) may be NaN or infinite. A row number is never formed from those
without a limit, an undefined r0 gives an undefined estimate, r0 = inf one of 0, and a triple whose
coefficient is not finite is not dropped."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "libgrpp_b200", "csrc")
CUDA = "/usr/local/cuda/include"

PROGRAM = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <utility>
#include <vector>
#include <cuda_runtime.h>
using std::max;
using std::min;
static std::vector<std::pair<const char *, const char *>> g_tabs;
template <typename T> static T __ldg(const T *p)
{
    for (auto &t : g_tabs)
        if ((const char *)p >= t.first && (const char *)(p + 1) <= t.second) return *p;
    std::printf("read outside the tables\n");
    std::exit(2);
}
// as the PTX conversion: saturating, most significant bit for NaN
static unsigned __double2uint_rz(double x)
{
    if (x != x) return 0x80000000u;
    return x <= 0 ? 0u : (x >= 4294967295.0 ? 0xffffffffu : (unsigned)x);
}
#define __logf logf
#define __noinline__
static int __clz(unsigned x) { return __builtin_clz(x); }
static double __dmul_rn(double x, double y) { return x * y; }
static double __dadd_rn(double x, double y) { return x + y; }
static double __fma_rn(double x, double y, double z) { return std::fma(x, y, z); }
static double __shfl_sync(unsigned, double x, int, int) { return x; }
static void __syncthreads() {}
static struct { unsigned x; } threadIdx, blockIdx, blockDim, gridDim;
#define GRPP_RADIAL_TABLES_ONLY
#define GRPP_NO_RADIAL_TABLE_KERNELS
#include "radial.cuh"
#include "tables.h"
using namespace grpp;
#define REQUIRE(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main()
{
    HostTables h;
    build_host_tables(h);
    c_tab.bessel = h.bessel.data();
    c_tab.rfun = h.rfun.data();
    c_tab.dfact = h.dfact.data();
    c_tab.ratio = h.ratio.data();
    c_tab.ratio_y = h.ratio_y.data();
    c_tab.bes_t = h.bes_t.data();
    c_tab.bes_y = h.bes_y.data();
    for (auto *v : {&h.bessel, &h.rfun, &h.dfact, &h.ratio, &h.ratio_y, &h.bes_t, &h.bes_y})
        g_tabs.push_back({(const char *)v->data(), (const char *)(v->data() + v->size())});
    const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    std::vector<double> xs = {0.0, 1e-320, 1e-8, 1e-7, 2e-7, 1e-3, 4.9e-3, 0.1, 1.2499999, 1.25, 3.0, 15.994, 15.999, 16.0, 16.0000001, 17.0,
                              300.0, 1e9, 1e300, inf, nan, -1.0, -1e9, -inf};
    for (int l = 0; l <= kRadMaxLam; l++)
        for (double x : xs)
            for (double ix : {1.0 / x, 0.0, 1.0 / 16, inf, -inf, nan, -1.0}) {
                const double t = scr_t(l, x, ix), m = scr_m(l, x, ix);
                if (x != x) REQUIRE(t != t && (ix == ix || m != m));
            }
    for (int l1 = 0; l1 <= kRadMaxLam; l1 += 3)
        for (int l2 = 0; l2 <= kRadMaxLam; l2 += 4)
            for (double k1 : {0.0, 1e-320, 1e-3, 7.0})
                for (double k2 : {0.0, 1e-3, 1e4})
                    for (double eta : {0.0, 2.0}) {
                        const double p = 1.5 + eta;
                        auto env = [&](double r0) {
                            return scr_envelope(l1, l2, 3, 1.0, 2.0, 0.5, 1.0, eta, p, k1, k2, 1 / k1, 1 / k2, r0, std::sqrt(kPi / p), std::sqrt(p));
                        };
                        REQUIRE(std::isnan(env(nan)));
                        REQUIRE(eta == 0.0 ? std::isnan(env(inf)) : env(inf) == 0.0);
                        for (double r0 : {1e-320, 1e-9, 0.3, 5.0, 40.0}) env(r0);
                        env(0.0);
                    }
    // a far, tight triple is dropped, unless its coefficient is not finite
    for (double c : {0.0, 1.0, -1e3, 1e-300}) REQUIRE(scr_dead(3.0, 4.0, 50.0, 60.0, 20.0, c, 0, 2, 2, 0, 2));
    for (double c : {nan, inf, -inf}) REQUIRE(!scr_dead(3.0, 4.0, 50.0, 60.0, 20.0, c, 0, 2, 2, 0, 2));
    REQUIRE(!scr_dead(3.0, 4.0, nan, 60.0, 20.0, 1.0, 0, 2, 2, 0, 2));
    std::printf("ok\n");
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="needs g++ and the CUDA headers")
def test_lookups_stay_in_their_tables(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    cmd = ["g++", "-std=c++17", "-O1", "-fsanitize=undefined,float-cast-overflow", "-fno-sanitize-recover=all", "-I", CSRC, "-I", CUDA,
           str(src), os.path.join(CSRC, "tables.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), r.stdout[-2000:] + r.stderr[-2000:]
