"""Tables built on first use (csrc/once.hpp): a build that fails half way is
made again by the next call, a complete one is not."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "once.hpp"
#include <cstdio>
enum status { OK = 0, FAILED = 2 };
int main() {
  bool built = false;
  int first = 0, second = 0, fail_at = 1, calls = 0;
  // two fake allocations and a launch, of which step `fail_at` fails
  auto make = [&]() -> status {
    ++calls;
    first = 1;
    if (fail_at == 1) return FAILED;
    second = 1;
    if (fail_at == 2) return FAILED;
    return OK;
  };
  if (build_once(built, make) != FAILED || built || second) return 1;
  fail_at = 2;
  if (build_once(built, make) != FAILED || built) return 2;
  fail_at = 0;
  if (build_once(built, make) != OK || !built || calls != 3) return 3;
  if (build_once(built, make) != OK || calls != 3) return 4;
  return 0;
}
"""


def test_a_failed_build_is_made_again(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "rbc3d_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_influence_tables_use_it():
    """Both precisions' influence tables are behind such a flag, not behind
    the pointer of their first allocation."""
    with open(os.path.join(ROOT, "rbc3d_gb300", "csrc", "pme.cu")) as f:
        text = f.read()
    for bits in ("32", "64"):
        assert f"build_once(P.infl{bits}_built" in text and f"!P.infl{bits}.p" not in text
