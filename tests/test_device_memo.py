"""DeviceMemo (pyqcm_gb300/csrc/qcmg_memo.h): a property found out for one
device, or before a device reset, is not taken for another's.  The on-chip
Lanczos asks in this way whether clusters of sixteen CTAs run; the consent
given while asking holds for one device's context only."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "pyqcm_gb300", "csrc")

DRIVER = r"""
#include "qcmg_memo.h"
#include <cstdio>
#include <stdexcept>
int main() {
  qcmg::DeviceMemo<bool> memo;
  int asked[3] = {0, 0, 0};
  auto get = [&](int dev, unsigned long long ctx) { return memo.get(dev, ctx, [&] { return ++asked[dev], dev != 1; }); };
  bool ok = get(0, 1) && get(0, 1) && asked[0] == 1;  // once per device
  ok = ok && !get(1, 2) && !get(1, 2) && asked[1] == 1;  // a second device asks for itself
  ok = ok && get(0, 1) && asked[0] == 1;
  ok = ok && get(0, 3) && asked[0] == 2;  // and so does a new context
  try {  // a question that failed is asked again
    memo.get(2, 1, [&]() -> bool { throw std::runtime_error("no device"); });
    ok = false;
  } catch (const std::runtime_error&) {
  }
  ok = ok && get(2, 1) && asked[2] == 1;
  std::puts(ok ? "ok" : "bad");
}
"""


def test_asked_once_per_device_and_context(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    (tmp_path / "driver.cpp").write_text(DRIVER)
    exe = str(tmp_path / "driver")
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", "-I", CSRC, str(tmp_path / "driver.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split() == ["ok"]


def test_no_cluster_size_is_kept_for_the_whole_process():
    """What clusters_run answers is kept nowhere but in a DeviceMemo: a plain
    static of the process would hand one device's answer to all."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            for line in f:
                if "clusters_run(" in line:
                    assert "static" not in line, (name, line)
