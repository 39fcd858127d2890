"""The regularised coupling of the local functionals (reg_lambda in wtd_functional.cuh): the real
form against the complex one over every sign of its arguments, on the CPU.

With kc = sqrt(k2) real and |p0| = sqrt(|m2|) below it both forms evaluate the same expression; the
real one takes sqrt, log or atan of real numbers.  Each is good to a few units in the last place of
kc, and for real p0 the rounding of kc and p0 (half a unit each) enters the logarithm's argument
through kc - p0: a relative error of up to eps kc/(kc - p0) in each form, times R1 p0 <= kc/2 in
lambda; for imaginary p0 the terms are kc and 2 R1 |p0| atan <= 1.6 |p0|.  So lambda / (R0 (kc +
|p0|)) agrees to eps (16 + 2 kc/(kc - p0)), eps = 2.2e-16.
Arguments outside (kc imaginary, or p0 beyond a fixed cut-off) must be left to the complex form.
"""
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "wslda_b200", "csrc")
NVCC = "/usr/local/cuda/bin/nvcc"

MAIN = r"""
#include "predefines.h"
#include "wtd_settings.h"
#include "wtd_surface.h"
#include "problem-definition.h"
#include "wtd_functional.cuh"
int main()
{
    double worst = 0.0;
    int real = 0, general = 0, wrong = 0;
    const double grid[] = {0.0, 1e-14, 1e-9, 1e-5, 0.01, 0.3, 1.0, 2.7, 8.0, 23.9, 24.0, 24.1, 60.0, 1e4};
    const int n = sizeof(grid) / sizeof(grid[0]);
    for (int a = -n + 1; a < n; a++)
        for (int b = -n + 1; b < n; b++) {
            const double m2 = a < 0 ? -grid[-a] : grid[a], k2 = b < 0 ? -grid[-b] : grid[b];
            const RegLambda f = reg_lambda(m2, k2), g = reg_lambda_complex(m2, k2);
#ifdef USE_CUBIC_CUTOFF
            const double kk = (M_PI / DX) * (M_PI / DX);
#else
            const double kk = k2;
#endif
            if (f.real != (kk > 0.0 && m2 < kk)) wrong++;
            if (!f.real) { general++; continue; }
            real++;
            const double kc = sqrt(kk), bound = 2.2e-16 * (16 + (m2 > 0.0 ? 2 * kc / (kc - sqrt(m2)) : 2));
            const double d = fabs(f.lam.real() - g.lam.real()) / (REG_COEFF_R0 * (kc + sqrt(fabs(m2)))) / bound;
            const double e = fabs(f.p0 - g.p0) / kc / bound;
            if (!(d <= worst)) worst = d;
            if (!(e <= worst)) worst = e;
        }
    const RegLambda q = reg_lambda(0.0 / 0.0 * 1.0, 1.0), i = reg_lambda(-1.0 / 0.0 * 1.0, 1.0);
    printf("%d %d %d %.3e %d %d\n", real, general, wrong, worst, (int)q.real, (int)i.real);
    return 0;
}
"""


@pytest.mark.parametrize("project,dim", [("t2d_slda", 2), ("t1d_sldae_a1", 1)])   # spherical and cubic cut-off
def test_real_form_matches_complex_form(tmp_path, project, dim):
    src, exe = tmp_path / "m.cu", tmp_path / "m"
    src.write_text(MAIN)
    subprocess.run([NVCC, "-std=c++17", "-w", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    f"-DCODEDIM={dim}", f"-I{REPO}/wslda_b200/projects/{project}", f"-I{CSRC}/surface", f"-I{CSRC}",
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    real, general, wrong, worst, nan_real, inf_real = int(out[0]), int(out[1]), int(out[2]), float(out[3]), int(out[4]), int(out[5])
    assert real > 100 and general > 50 and wrong == 0 and nan_real == 0 and inf_real == 0
    assert worst < 1.0, worst     # in units of the bound
