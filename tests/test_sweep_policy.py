"""Contexts of a sweep that share a device give up the factorisation's second
stream from eight on; contexts on other devices do not count."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "for90-mom2_b200", "csrc")
MAIN = """
#include <cstdio>
#include <cstdlib>
#include "sweep_policy.h"
int main(int argc, char **argv) {
  int d[64];
  bool c[64];
  for (int i = 1; i < argc; i++) d[i - 1] = std::atoi(argv[i]);
  mom::crowded_contexts(argc - 1, d, c);
  for (int i = 1; i < argc; i++) std::putchar(c[i - 1] ? '1' : '0');
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("policy")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", str(d / "main"), str(d / "main.cpp")], check=True)
    return str(d / "main")


@pytest.mark.parametrize("devices,crowded", [
    ([0], "0"), ([0] * 7, "0" * 7), ([0] * 8, "1" * 8), (list(range(8)), "0" * 8), ([0] * 8 + [1] * 7, "1" * 8 + "0" * 7),
    ([0, 1] * 8, "1" * 16), ([0] * 7 + [-1] * 9, "0" * 16)])
def test_crowded_contexts(program, devices, crowded):
    r = subprocess.run([program] + [str(d) for d in devices], capture_output=True, text=True, check=True)
    assert r.stdout == crowded
