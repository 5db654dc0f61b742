"""Scalars of the corrected CG: the step length is the FP64 quotient's rounding, and the dot products keep FP64's digits
beyond the few terms of a chunk that FP32 adds."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "light-field-remote-vision_gb300" / "csrc"

SRC = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "cg_scalars.h"
int main() {
    std::mt19937_64 rng(5);
    std::uniform_real_distribution<double> mant(1.0, 2.0);
    double worst = 0.0, plain = 0.0;
    long exact = 0;
    for (long i = 0; i < 4000000; ++i) {
        // exponents inside the FP32 form's range, at its ends and beyond
        const int ea = (int)(rng() % 220) - 110, eb = (int)(rng() % 220) - 110;
        const double a = std::ldexp(mant(rng), ea), b = std::ldexp(mant(rng), eb), q = a / b;
        if (!(q > 1e-37 && q < 1e38)) continue;
        const float got = lfrv::cg_quotient(a, b);
        int e;
        std::frexp(q, &e);
        const double ulp = std::ldexp(1.0, e - 24);
        worst = std::fmax(worst, std::fabs((double)got - q) / ulp);
        plain = std::fmax(plain, std::fabs((double)((float)a / (float)b) - q) / ulp);
        exact += got == (float)q;
    }
    std::printf("%.9f %.9f %ld\n", worst, plain, exact);
    return 0;
}
"""


def test_step_length_is_the_rounded_fp64_quotient(tmp_path):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "scalars.cpp", tmp_path / "scalars"
    src.write_text(SRC)
    subprocess.run([cc, "-std=c++17", "-O2", "-ffp-contract=off", f"-I{CSRC}", "-o", str(exe), str(src)], check=True)
    worst, plain, exact = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert float(worst) <= 0.5 + 2.0 ** -18
    assert float(plain) > 1.0  # the quotient of the rounded operands, which is not enough
    assert int(exact) > 3000000


@pytest.mark.gpu
def test_dot_products_of_tall_units(ctx):
    """One step from 0 on a residual of +-c: the step length is r . r / r . A r, whose terms are all c^2 and 5 c^2 (3 c^2 in
    the outer columns), so FP32 chains round one way. c has 21 bits, so r and A r are exact; a chain of 8 equal terms errs by
    at most (2 + ... + 8) / 8 halves of 2^-23, the step length and the step round once each: (2 * 35/8 + 2) 2^-24. c is
    the value for which a chain of 28 terms, a unit's rows at this size, is off most."""
    H, W = 1008, 1024
    c = np.float32(1876087 / 2.0 ** 20)
    gx = np.zeros((H, W), np.float32)
    gx[:, 0::2] = c
    out, it, _ = ctx.stage_cg(gx, np.zeros_like(gx), np.zeros((3, H, W), np.float32), False, 1, 0.0)
    assert it == 1
    alpha = np.abs(out.astype(np.float64)) / float(c)
    exact = W / (5.0 * (W - 2) + 3.0 * 2)
    assert np.max(np.abs(alpha / exact - 1.0)) <= (2 * 35 / 8 + 2) * 2.0 ** -24
