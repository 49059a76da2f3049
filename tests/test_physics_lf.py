"""The FP64 Lax-Friedrichs flux of the face kernels (flux_lax_friedrichs_sq, which picks
the larger wave speed by its square) beside the one with both speeds rooted
(flux_lax_friedrichs_fast), on the host (CPU only): the same values to rounding on
ordinary states, and the same values, infinities and NaN where squares over- or underflow,
a state is at rest, or a density or pressure is negative -- a NaN flux is how a trace with
a negative pressure is noticed.  Bar: the two differ by a few roundings of terms that are
at most the flux's largest, 1e-14 of it (1e-16 per operation, some thirty of them)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

PROBE = r"""
#include "dg_physics.cuh"
#include <cstdio>
int main()
{
    double ul[5], ur[5];
    const double n[3] = {0.36, 0.48, 0.8}, nm = 0.7;
    while (std::scanf("%lf %lf %lf %lf %lf %lf %lf %lf %lf %lf", ul, ul + 1, ul + 2, ul + 3, ul + 4, ur, ur + 1, ur + 2, ur + 3,
                      ur + 4) == 10) {
        double F[2][5];
        dgp::flux_lax_friedrichs_fast<double>(1.4, ul, ur, n, nm, F[0]);
        dgp::flux_lax_friedrichs_sq(1.4, ul, ur, n, nm, F[1]);
        for (int k = 0; k < 2; ++k)
            for (int s = 0; s < 5; ++s) std::printf("%.17g ", F[k][s]);
        std::printf("\n");
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("lf")
    (d / "probe.cpp").write_text(PROBE)
    subprocess.run([cxx, "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "dg-mpi_b200", "csrc"), "-o", str(d / "probe"),
                    str(d / "probe.cpp")], check=True, capture_output=True)

    def run(rows):
        text = "\n".join(" ".join(repr(float(x)) for x in r) for r in rows) + "\n"
        out = subprocess.run([str(d / "probe")], input=text, check=True, capture_output=True, text=True).stdout
        return np.array([[float(x) for x in l.split()] for l in out.splitlines()]).reshape(-1, 2, 5)

    return run


def state(rho, u, P):
    u = np.asarray(u, float)
    with np.errstate(all="ignore"):
        return [rho, *(rho * u), P / 0.4 + 0.5 * rho * (u @ u)]


def agree(F):
    with np.errstate(all="ignore"):
        scale = np.abs(np.where(np.isfinite(F), F, 0.0)).max(axis=(1, 2))
        close = np.abs(F[:, 0] - F[:, 1]) <= 1e-14 * scale[:, None]
    return np.where(np.isfinite(F[:, 0]), close, (F[:, 0] == F[:, 1]) | (np.isnan(F[:, 0]) & np.isnan(F[:, 1])))


def test_ordinary_states(probe):
    rng = np.random.default_rng(3)
    rows = []
    for _ in range(2000):
        c = 10.0 ** rng.uniform(-3, 3)
        rows.append([x for _ in "LR" for x in state(rng.uniform(0.2, 3), c * 10.0 ** rng.uniform(-3, 1) * rng.standard_normal(3),
                                                    c * c * rng.uniform(0.2, 3))])
    F = probe(rows)
    assert np.isfinite(F).all() and agree(F).all()


good = state(1.0, [0.3, -0.2, 0.5], 1.2)
ODD = {
    "left at rest with negative pressure": (state(1.0, [0, 0, 0], -0.1), good),
    "right at rest with negative pressure": (good, state(1.0, [0, 0, 0], -0.1)),
    "both at rest with negative pressure": (state(1.0, [0, 0, 0], -0.1), state(2.0, [0, 0, 0], -3.0)),
    "left moving with negative pressure": (state(1.0, [0.1, 0, 0], -0.1), good),
    "right moving with negative pressure": (good, state(1.0, [0.1, 0, 0], -0.1)),
    "both at rest": (state(1.0, [0, 0, 0], 1.0), state(0.5, [0, 0, 0], 2.0)),
    "no pressure": (state(1.0, [0.1, 0.2, 0], 0.0), good),
    "speeds of 1e80": (state(1.0, [1e80, 0, 0], 1e160), state(1.0, [2e80, 0, 0], 3e160)),
    "speeds of 1e-80": (state(1.0, [1e-80, 0, 0], 1e-160), state(1.0, [2e-80, 0, 0], 3e-160)),
    "speeds of 1e-140": (state(1.0, [1e-140, 0, 0], 1e-280), state(1.0, [2e-140, 0, 0], 3e-280)),
    "left density and pressure negative": (state(-1.0, [0.2, 0.1, 0], -1.0), good),
    "right density and pressure negative": (good, state(-1.0, [0.2, 0.1, 0], -1.0)),
    "no density": ([0.0, 0.1, 0.0, 0.0, 1.0], good),
    "left NaN": ([float("nan")] * 5, good),
    "right NaN": (good, [float("nan")] * 5),
    "left infinite energy": ([1.0, 0.1, 0.0, 0.0, float("inf")], good),
    "right infinite energy": (good, [1.0, 0.1, 0.0, 0.0, float("inf")]),
}


@pytest.mark.parametrize("name", ODD)
def test_odd_states(probe, name):
    left, right = ODD[name]
    F = probe([[*left, *right]])
    assert agree(F).all(), F
