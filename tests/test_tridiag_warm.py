"""TridiagLowest (pyqcm_gb300/csrc/qcmg_tridiag.cpp): called after every step
of a Lanczos run, past convergence and through copies of the lowest
eigenvalue, it returns the same eigenvalue and vector as a call from scratch,
bit for bit."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "pyqcm_gb300", "csrc")

DRIVER = r"""
#include "qcmg_tridiag.h"
#include <cstdio>
#include <vector>
int main() {
  int n;
  while (std::scanf("%d", &n) == 1) {
    std::vector<double> a, b, z, zc;
    qcmg::TridiagLowest lowest;
    int bad = 0;
    for (int i = 0; i < n; ++i) {
      double x, y;
      if (std::scanf("%la %la", &x, &y) != 2) return 1;
      a.push_back(x);
      b.push_back(y);
      const double l = lowest(a, b, z), lc = qcmg::tridiag_lowest(a, b, zc);
      if (l != lc || z != zc) ++bad;
    }
    std::printf("%d\n", bad);
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("tridiag")
    (d / "driver.cpp").write_text(DRIVER)
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, str(d / "driver.cpp"),
                    os.path.join(CSRC, "qcmg_tridiag.cpp"), "-o", str(d / "driver")], check=True)
    return str(d / "driver")


def _lanczos(ev, steps, rng):
    r, q, a, b = rng.normal(size=len(ev)), np.zeros(len(ev)), [], []
    r /= np.linalg.norm(r)
    for j in range(steps):
        if j:
            r, q = q / b[-1], -b[-1] * r
        q = q + ev * r
        a.append(float(q @ r))
        q = q - a[-1] * r
        b.append(float(np.linalg.norm(q)))
    return a, b


@pytest.mark.parametrize("kind", ["wide", "narrow", "offset", "pair", "few", "flat"])
def test_one_row_more_each_call(driver, kind):
    rng = np.random.default_rng(7)
    ev = {"wide": rng.normal(size=800) * 5, "narrow": rng.normal(size=800) * 1e-3, "offset": 1e3 + rng.normal(size=800),
          "pair": np.concatenate([[-30.0, -30.0 + 1e-7], rng.normal(size=500) * 5]), "few": np.repeat([-3.0, 1.0, 2.0], 60),
          "flat": np.full(50, 2.5)}[kind]
    a, b = _lanczos(ev, 160, rng)
    text = f"{len(a)}\n" + "\n".join(f"{x.hex()} {y.hex()}" for x, y in zip(a, b)) + "\n"
    out = subprocess.run([driver], input=text, capture_output=True, text=True, check=True).stdout
    assert out.split() == ["0"]
