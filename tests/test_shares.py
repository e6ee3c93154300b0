"""run_shares (pyqcm_gb300/csrc/qcmg_shares.h), the host threads of a batched
on-chip Lanczos: every share is done, and the program goes on, when the system
gives fewer threads than asked for or none; a share's exception comes out of
the call after all shares are over."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "pyqcm_gb300", "csrc")

DRIVER = r"""
#include "qcmg_shares.h"
#include <atomic>
#include <cstdio>
#include <stdexcept>
#include <string>
struct Limited {  // a system that gives `left` threads
  int left;
  template <class F>
  std::thread operator()(F&& f) {
    if (left-- <= 0) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
    return std::thread(std::forward<F>(f));
  }
};
int main() {
  int bad = 0;
  for (int n : {1, 2, 8})
    for (int give = 0; give <= n; ++give)
      for (int fail = -1; fail < n; ++fail) {
        std::atomic<int> done[8] = {};
        int caught = -1;
        try {
          qcmg::run_shares(n, [&](int t) {
            ++done[t];
            if (t == fail) throw std::out_of_range(std::to_string(t));
          }, Limited{give});
        } catch (const std::out_of_range& e) {
          caught = std::stoi(e.what());
        }
        bad += caught != fail;
        for (int t = 0; t < n; ++t) bad += done[t] != 1;
      }
  std::printf("%d\n", bad);
}
"""


def test_every_share_is_done_whatever_threads_there_are(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    (tmp_path / "driver.cpp").write_text(DRIVER)
    exe = str(tmp_path / "driver")
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", "-I", CSRC, str(tmp_path / "driver.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split() == ["0"]


def test_batched_solves_start_their_threads_there():
    """A bare thread that cannot be started would end the caller's program:
    the unwinding destroys the joinable threads before it."""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cpp", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                assert "std::vector<std::thread>" not in f.read(), name
