"""The grid barrier's word (csrc/qedf_barrier_word.h) over more arrivals than 32
bits count, compiled for the host: the count does not read as an error, and an
error stays one whatever arrives after it."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "qed_fermion_b200", "csrc")
PROGRAM = """
#include "qedf_barrier_word.h"
int main() {
  const unsigned long long blocks = %d;
  // barriers around the 2^32nd arrival, the first ones and the last of 10^9 iterations
  const unsigned long long wrap = (1ull << 32) / blocks, at[] = {0, 1, wrap - 1, wrap, wrap + 1, 2 * wrap + 3, 2000000000ull};
  for (unsigned long long n : at) {
    const unsigned int target = (unsigned int)((n + 1) * blocks);
    unsigned long long word = n * blocks;  // every block passed barrier n
    for (unsigned long long k = 0; k < blocks; ++k, ++word)
      if (qedf::bar_error(word) != 0 || qedf::bar_reached(word, target)) return 1;
    if (qedf::bar_error(word) != 0 || !qedf::bar_reached(word, target)) return 2;
    for (unsigned int code = 1; code < 8; ++code)
      if (qedf::bar_error((word | qedf::bar_error_bits(code)) + blocks) != code) return 3;
  }
  return 0;
}
"""


@pytest.mark.parametrize("blocks", [1, 148, 592])
def test_count_keeps_out_of_the_error(blocks, tmp_path):
    cc = shutil.which("g++") or shutil.which("c++")
    assert cc, "no C++ compiler (nvcc needs one too)"
    src = tmp_path / "word.cpp"
    src.write_text(PROGRAM % blocks)
    exe = tmp_path / "word"
    subprocess.run([cc, "-std=c++17", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
