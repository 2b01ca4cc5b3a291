"""The FP64 background means' |theta| and |phi| (abs_phi_theta), the device
function itself: its text is taken from the kernels' sources and compiled for
the host, with the CUDA intrinsics it uses written in C++, and compared with
long double arithmetic."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "axion-strings_gb300", "csrc")

PROLOGUE = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <cstdint>
#include <random>
using std::max; using std::min;
#define __device__
#define __forceinline__ inline
#define __noinline__
template <class To, class From> static To as(From v) { static_assert(sizeof(To) == sizeof(From)); To t; memcpy(&t, &v, sizeof t); return t; }
static int __double2hiint(double x) { return (int)(as<uint64_t>(x) >> 32); }
static int __double2loint(double x) { return (int)(uint32_t)as<uint64_t>(x); }
static double __hiloint2double(int h, int l) { return as<double>((uint64_t)(uint32_t)h << 32 | (uint32_t)l); }
static float __uint_as_float(unsigned u) { return as<float>(u); }
static unsigned __float_as_uint(float f) { return as<unsigned>(f); }
static int __float2int_rn(float f) { return (int)lrintf(f); }
static float __frcp_rn(float f) { return 1.0f / f; }
static float g_off = 1.0f;   // __fdividef is within 2 ulp: the quotient times g_off
static float __fdividef(float a, float b) { return a / b * g_off; }
"""

MAIN = r"""
int main() {
    for (int k = -kRot; k <= kRot; ++k) {
        const double t = (double)k * (3.141592653589793 / kRot);
        g_theta_rot[k + kRot] = ThetaRot{cos(t), sin(t), fabs(t), 0.0};
    }
    std::mt19937_64 g(7);
    std::normal_distribution<double> nrm;
    std::uniform_real_distribution<double> uni(-1.0, 1.0);
    long double worst_small = 0, worst_angle = 0, worst_mod = 0;
    const double edge = 3.141592653589793 / kRot;
    for (int n = 0; n < 3000000; ++n) {
        g_off = 1.0f + 1.1920929e-7f * (float)(n % 5 - 2);
        double a, b;
        if (n % 3 == 0) {   // any direction, components up to e^24 apart
            a = nrm(g) * exp(12 * uni(g));
            b = nrm(g) * exp(12 * uni(g));
        } else if (n % 3 == 1) {   // angles around the edges between two table entries
            const double t = (std::uniform_int_distribution<int>(-kRot, kRot)(g) + 0.5) * edge * (1 + 1e-6 * uni(g)), r = exp(2 * uni(g));
            a = r * sin(t);
            b = r * cos(t);
        } else {   // the first entry: theta below pi / 1024, the reciprocal's float residual at its largest
            b = ldexp(1.0 + ldexp(std::uniform_int_distribution<int>(0, 3)(g), -23) + ldexp(1.0 - 1e-6 * (1 + uni(g)), -23), n % 7);
            a = b * uni(g) * (n % 2 ? 3e-3 : exp(-20 * fabs(uni(g))) * 3e-3);
        }
        if (a == 0 || b == 0) continue;
        double phi, th;
        abs_phi_theta(a, b, phi, th);
        const long double wt = fabsl(atan2l(a, b)), wm = sqrtl((long double)a * a + (long double)b * b);
        worst_angle = max(worst_angle, fabsl(th - wt));
        worst_mod = max(worst_mod, fabsl(phi - wm) / wm);
        if (wt < 0.999L * edge / 2) worst_small = max(worst_small, fabsl(th - wt) / wt);
    }
    printf("%.17Lg %.17Lg %.17Lg\n", worst_small, worst_angle, worst_mod);
    printf("%.17g\n", tan(edge / 2 + 9e-7));
}
"""


def test_fp64_angle_and_modulus_of_the_kernel(tmp_path):
    """Angles of the first table entry (no table term to add to): three roundings of 2^-53, relative to themselves. Any
    angle: within 4 ulp of pi, the modulus within 4 ulp (the rotation's and the table's roundings)."""
    an = open(os.path.join(CSRC, "axs_analysis.cu")).read()
    internal = open(os.path.join(CSRC, "axs_internal.h")).read()

    def cut(text, start, end):
        i = text.index(start)
        return text[i:text.index(end, i)]

    def function(text, head):
        i = text.index(head)
        return text[i:text.index("\n}\n", i) + 3]

    parts = [PROLOGUE, function(internal, "__device__ __forceinline__ float float_bits"),
             function(internal, "__device__ __forceinline__ double double_bits"),
             cut(an, "__device__ constexpr float kAtanC", "// The string finder's angle"),
             function(an, "__device__ __forceinline__ float fast_atan2"),
             cut(an, "static constexpr int kRot", "// the rotation table of abs_phi_theta"), MAIN]
    src = tmp_path / "angle.cpp"
    src.write_text("\n".join(parts))
    exe = str(tmp_path / "angle")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", str(src), "-o", exe], check=True)
    out = re.split(r"\s+", subprocess.run([exe], check=True, capture_output=True, text=True).stdout.strip())
    small, angle, mod, tan_edge = map(float, out)
    assert tan_edge < 0.00307   # the quotient the two series are made for
    assert small <= 3.1 * 2.0 ** -53, small
    assert angle <= 4 * 2.0 ** -51, angle
    assert mod <= 4 * 2.0 ** -52, mod
