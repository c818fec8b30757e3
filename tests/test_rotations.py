"""The host tables of the FP64 translations by rotations (rotations.cpp), compiled here with g++: the
blocks against projections of the rotated harmonics onto the harmonics by quadrature, in extended
precision, the time that the first state of an order waits for them, and the CTAs of the translations that an SM holds.

Bar: the tables are rounded once from extended precision, entries are at most 2 in magnitude (half an ulp
is 2⁻⁵³ below 2), and the quadrature's own error stays below 1e-17, so 1.2e-16.
"""
import os
import re
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flexiblefmm.jl_b200", "csrc")
MAIN = r"""
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include "m2l_rot.h"
using namespace fmmb;
int main(int, char** v) {
  const int p = atoi(v[1]);
  printf("fit %d %zu\n", rot_resident(p, 3, 1, 99), rot_smem(p, 3, 1));
  const HostOperators op = build_operators(p, 1.0);
  const auto t0 = std::chrono::steady_clock::now();
  const auto h = rotation_tables(p, op);
  printf("ms %.17g\n", std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
  for (int c = 0; c <= NCLASS; ++c) {
    if (c < NCLASS) printf("class %d %d %d\n", op.reps_off[3 * c], op.reps_off[3 * c + 1], op.reps_off[3 * c + 2]);
    else printf("class 1 1 1\n");
    for (int l = 0; l <= p; ++l)
      for (int part = 0; part < 2; ++part)
        for (int j = part; j <= l; ++j)
          for (int k = part; k <= l; ++k)
            printf("%.17g\n", h->d[(size_t)c * 32 * h->layout.nd + h->layout.rot_at(l, part, j, k)]);
  }
}
"""


@pytest.fixture(scope="module")
def tables(tmp_path_factory):
    d = tmp_path_factory.mktemp("rotations")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I/usr/local/cuda/include", "-I" + CSRC, str(d / "main.cpp"),
                    os.path.join(CSRC, "rotations.cpp"), os.path.join(CSRC, "operators.cpp"), "-o", str(d / "main")],
                   check=True)

    def run(p):
        out = subprocess.run([str(d / "main"), str(p)], check=True, capture_output=True, text=True).stdout
        fit, out = out.split("\n", 1)
        ms, *parts = re.split(r"^class ", out, flags=re.M)
        classes = []
        for part in parts:
            head, *vals = part.strip().split("\n")
            classes.append((tuple(map(int, head.split())), np.array(vals, np.float64)))
        return float(ms.split()[1]), classes, tuple(map(int, fit.split()[1:]))

    return run


def harmonics(x, y, z, p):
    """Re and Im of the Schmidt harmonics by (n, m), longdouble, at unit vectors."""
    v = {}
    s = np.ones_like(x) + 0j
    for m in range(p + 1):
        if m:
            s = -np.sqrt(np.longdouble(2 * m - 1) / (2 * m)) * (x + 1j * y) * s
        prev, cur = np.zeros_like(s), s
        v[m, m] = s
        for n in range(m + 1, p + 1):
            c = np.sqrt(np.longdouble((n - m) * (n + m)))
            prev, cur = cur, (2 * n - 1) / c * z * cur - np.sqrt(np.longdouble((n - m - 1) * (n + m - 1))) / c * prev
            v[n, m] = cur
    return v


def legendre(n):
    t = np.polynomial.legendre.leggauss(n)[0].astype(np.longdouble)
    for _ in range(3):
        p0, p1 = np.ones_like(t), t
        for k in range(2, n + 1):
            p0, p1 = p1, ((2 * k - 1) * t * p1 - (k - 1) * p0) / k
        d = n * (t * p1 - p0) / (t * t - 1)
        t = t - p1 / d
    return t, 2 / ((1 - t * t) * d * d)


@pytest.mark.parametrize("p", [1, 2, 5, 9])
def test_blocks_are_the_projections(tables, p):
    _, classes, _ = tables(p)
    assert len(classes) == 35
    t, wt = legendre(p + 1)
    nph = 2 * p + 2
    pi = np.arctan(np.longdouble(1)) * 4
    ph = (np.arange(nph) + np.longdouble(0.5)) * (2 * pi / nph)
    st = np.sqrt(1 - t * t)
    x, y, z = np.outer(st, np.cos(ph)).ravel(), np.outer(st, np.sin(ph)).ravel(), np.repeat(t, nph)
    w = np.repeat(wt, nph) * (2 * pi / nph)
    base = harmonics(x, y, z, p)
    for (ox, oy, oz), got in classes:
        r = np.sqrt(np.longdouble(ox * ox + oy * oy + oz * oz))
        ct, s = oz / r, np.sqrt(np.longdouble(ox * ox + oy * oy)) / r
        rot = harmonics(ct * x - s * z, y, s * x + ct * z, p)
        want = []
        for l in range(p + 1):
            for part in (np.real, np.imag):
                f = 1 if part is np.imag else 0
                if f > l:
                    continue
                R = np.array([part(rot[l, j]) for j in range(f, l + 1)])
                B = np.array([part(base[l, k]) * w * (2 * l + 1) / (4 * pi if k == 0 else 2 * pi) for k in range(f, l + 1)])
                want.append((R @ B.T).ravel())
        assert np.max(np.abs(np.concatenate(want) - got)) <= 1.2e-16, (ox, oy, oz)


def test_first_state_does_not_wait_for_the_tables(tables):
    """They cost less than the dense operators that a cache builds anyway: 5 ms at the largest order (84 ms the
    operators), 292 by quadrature; the bar leaves room for a loaded machine."""
    assert min(tables(20)[0] for _ in range(3)) < 60


def test_ctas_that_fit_an_sm(tables):
    """The launches count on four CTAs an SM up to p = 10 and on three at p = 11 (chunks of 24 pairs)."""
    fits = {p: tables(p)[2] for p in (1, 10, 11, 12, 15)}
    for p, (fit, smem) in fits.items():
        assert fit * (smem + 1024) <= 228 * 1024 < (fit + 1) * (smem + 1024)
    assert fits[1][0] >= 4 and fits[10][0] == 4 and fits[11][0] == 3 and fits[12][0] == fits[15][0] == 2
