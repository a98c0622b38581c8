"""The threads that compile the generated kernels' units: a thread that cannot be started and an
exception inside a unit leave an error or a result, never a terminated process."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "reseact", "esm_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <atomic>
#include <stdexcept>
#include <system_error>
#include "rs_units.h"
int main(int, char** argv) {
  const int mode = argv[1][0] - '0', n = 8;  // 1: no thread starts, 2: every second, 3: parts throw
  std::vector<int> done(n, 0);
  std::vector<std::string> err;
  std::atomic<int> started{0};
  auto work = [&](int u) {
    if (mode == 3 && u % 3 == 0) throw std::runtime_error("part " + std::to_string(u));
    if (mode == 3 && u == 4) throw 4;
    done[u] = u + 1;
  };
  auto start = [&](auto f) {
    if (mode == 1 || (mode == 2 && ++started % 2)) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
    return std::thread(f);
  };
  if (mode == 0) rs::run_units(n, work, &err);
  else rs::run_units(n, work, &err, start);
  for (int u = 0; u < n; ++u) std::printf("%d:%s ", done[u], err[u].c_str());
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("units")
    (d / "p.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(d / "p.cpp"), "-o", str(d / "p")], check=True)
    return str(d / "p")


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_every_unit_ends_in_a_result_or_an_error(program, mode):
    r = subprocess.run([program, str(mode)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.returncode
    want = ["%d:" % (u + 1) for u in range(8)]
    if mode == 3:
        for u in (0, 3, 6):
            want[u] = "0:part %d" % u
        want[4] = "0:exception"
    assert r.stdout.rstrip(" ") == " ".join(want)


def test_the_compiler_starts_no_threads_of_its_own():
    assert "std::thread" not in open(os.path.join(CSRC, "rs_jit.cu")).read()
