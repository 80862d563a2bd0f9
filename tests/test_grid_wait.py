"""The arithmetic of the meeting of a kernel's CTAs (csrc/grid_wait.h), on the
CPU: a run may meet more often than 31 or 32 bits count, and a CTA that gave up
ends every other CTA's wait."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "grid_wait.h"
using namespace kites_internal;
int main(int argc, char **argv) {
  const unsigned long long first = strtoull(argv[1], nullptr, 10);
  const uint32_t ctas = (uint32_t)atoi(argv[2]);
  grid_word word = (grid_word)((first - 1) * ctas);
  for (unsigned long long met = first; met < first + 8; ++met) {
    for (uint32_t c = 0; c < ctas; ++c) {
      if (grid_met(word, met, ctas)) return printf("meeting %llu early at %u\n", met, c), 1;
      if (grid_failed(word)) return printf("meeting %llu failed at %u\n", met, c), 1;
      word += 1;
    }
    if (!grid_met(word, met, ctas)) return printf("meeting %llu missed\n", met), 1;
    if (grid_failed(word)) return printf("meeting %llu failed\n", met), 1;
    const grid_word gave_up = (grid_word)(word - 1) | kGridGaveUp;
    if (!grid_met(gave_up, met, ctas) || !grid_failed(gave_up) || !grid_failed(gave_up + 1))
      return printf("meeting %llu hides a CTA that gave up\n", met), 1;
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("grid_wait")
    (d / "p.cpp").write_text(PROGRAM)
    exe = str(d / "p")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "kites_b200", "csrc"),
                    "-o", exe, str(d / "p.cpp")], check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("ctas", [1, 2, 147, 148])
@pytest.mark.parametrize("bits", [0, 31, 32, 40])
def test_meetings(program, ctas, bits):
    """Eight meetings around the one at which the arrivals reach 2^bits."""
    first = max(1, 2**bits // ctas - 3)
    r = subprocess.run([program, str(first), str(ctas)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
