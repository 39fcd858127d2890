"""Compile-time coefficients of the folded lines (wtd_circ.cuh) against their defining sums in
80-bit arithmetic, on the CPU.

A coefficient is a combination of the operator's kernel t(d) on N points, with the doubles k_q and
k_q^2 of the transforms' tables as its symbol.  It is rounded once, so it lies within half a unit in
the last place (2^-53 relative) of the exact value; the mean of N terms in 80 bits is good to
N 2^-64 max |symbol|, which is added to the bound.
"""
import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "wslda_b200", "csrc")
NVCC = "/usr/local/cuda/bin/nvcc"

MAIN = r"""
#include <cstdio>
#include <cmath>
#include <utility>
#define NX 12
#define NY 20
#define NZ 48
#define DX 1.15
#define DY 1.0
#define DZ 0.7
#define LX (DX*NX)
#define LY (DY*NY)
#define LZ (DZ*NZ)
#include "wtd_circ.cuh"
typedef long double Q;
static const Q PIQ = 3.14159265358979323846264338327950288L;
static double worst = 0.0;
static int count = 0;

/* (1/N) sum_q of the operator's symbol times e^{2 pi i q d/N}, Nyquist mode zeroed in the derivative */
static double k0;      /* 2 pi / L of the axis */
static Q exact_t(int op, int N, int d)
{
    Q s = 0;
    for (int q = -N / 2; q < N / 2; q++) {
        const Q a = 2 * PIQ * (((Q)q * d) - N * roundl((Q)q * d / N)) / N;
        const double k = k0 * (double)q, k2 = k * k;
        if (op == circ::LAP) s -= (Q)k2 * cosl(a);
        else if (q != -N / 2) s -= (Q)k * sinl(a);
    }
    return s / N;
}
/* block of n points: 2^-l sum over the shifts by n, alternating in the last fold where skew */
static Q exact_b(int op, int N, int n, bool skew, int d)
{
    Q s = 0;
    const int step = skew ? 2 * n : n;
    for (int k = 0; k < N / step; k++) s += exact_t(op, N, d + k * step) - (skew ? exact_t(op, N, d + n + k * step) : 0);
    return s * n / N;
}
template <int OP, int AX, int N, int n, bool SKEW, bool EV, int j, int k> static void one()
{
    k0 = 2.0 * 3.14159265358979323846 / (AX == 0 ? LX : AX == 1 ? LY : LZ);
    const Q a = exact_b(OP, N, n, SKEW, j - k), b = exact_b(OP, N, n, SKEW, j + k);
    const bool self = EV ? circ::self_even(n, SKEW, k) : circ::self_odd(n, SKEW, k);
    const Q want = self ? a : EV ? (a + b) / 2 : (a - b) / 2, kmax = k0 * N / 2;
    const Q bound = fabsl(want) * 0x1p-53L + N * 0x1p-64L * (OP == circ::LAP ? kmax * kmax : kmax);
    const double got = circ::Coef<OP, AX, N, n, SKEW, EV, j, k>::value;
    const double e = (double)(fabsl((Q)got - want) / bound);
    if (!(e <= worst)) worst = e;
    count++;
}
template <int OP, int AX, int N, int n, bool SKEW, bool EV, int j, int... K> static void row(std::integer_sequence<int, K...>)
{
    (one<OP, AX, N, n, SKEW, EV, j, K + (EV ? 0 : 1)>(), ...);
}
template <int OP, int AX, int N, int n, bool SKEW, bool EV, int... J> static void rows(std::integer_sequence<int, J...>)
{
    constexpr bool OV = OP == circ::LAP ? EV : !EV;
    (row<OP, AX, N, n, SKEW, EV, J + (OV ? 0 : 1)>(std::make_integer_sequence<int, EV ? circ::n_even(n, SKEW) : circ::n_odd(n, SKEW)>()), ...);
}
/* the blocks that half<> applies to a line of N points */
template <int OP, int AX, int N, int n, bool EV> static void block()
{
    constexpr bool OV = OP == circ::LAP ? EV : !EV;
    if constexpr (n % 2 == 0 && n >= 4) {
        constexpr int h = n / 2;
        rows<OP, AX, N, h, true, EV>(std::make_integer_sequence<int, OV ? circ::n_even(h, true) : circ::n_odd(h, true)>());
        block<OP, AX, N, h, EV>();
    } else
        rows<OP, AX, N, n, false, EV>(std::make_integer_sequence<int, OV ? circ::n_even(n, false) : circ::n_odd(n, false)>());
}
template <int AX, int N> static void line()
{
    block<circ::LAP, AX, N, N, true>();
    block<circ::LAP, AX, N, N, false>();
    block<circ::DER, AX, N, N, true>();
    block<circ::DER, AX, N, N, false>();
}
int main()
{
    line<0, 2>(); line<0, 4>(); line<0, 12>(); line<1, 18>(); line<1, 20>(); line<1, 22>(); line<0, 32>(); line<2, 48>();
    line<2, 50>(); line<2, 64>();
    printf("%d %.4f\n", count, worst);
    return 0;
}
"""


def test_coefficients_are_rounded_once(tmp_path):
    src, exe = tmp_path / "m.cu", tmp_path / "m"
    src.write_text(MAIN)
    subprocess.run([NVCC, "-std=c++17", "-w", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-DCODEDIM=3", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    count, worst = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert int(count) > 1000
    assert float(worst) <= 1.0, worst     # in units of the bound
