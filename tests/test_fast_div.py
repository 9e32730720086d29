"""The divisions by numbers that the host knows (``FastDiv``), on the CPU: every kind of divisor and dividend of 32 bits."""

import subprocess

from kohakufa_b200 import build

PROGRAM = """
#include <cstdio>
#include <random>
#include "kfa_ptx.cuh"

int main() {
  std::mt19937 gen(1);
  unsigned edges[] = {1u, 2u, 3u, 5u, 127u, 128u, 129u, 148u, 65535u, 65536u, 65537u, 0x7ffffffeu, 0x7fffffffu, 0x80000000u, 0x80000001u,
                      0xfffffffeu, 0xffffffffu};
  long long wrong = 0, looked = 0;
  auto look = [&](unsigned n, const kfa::FastDiv& by) {
    ++looked;
    if (by.div(n) != n / by.d && wrong++ == 0) std::printf("%u / %u\\n", n, by.d);
  };
  auto divisor = [&](unsigned d) {
    const kfa::FastDiv by = kfa::FastDiv::by(d);
    look(0, by);
    for (unsigned n : edges) look(n, by);
    for (int i = 0; i < 40; ++i) {
      const unsigned n = gen() >> (gen() % 32), m = n / d * d;
      look(n, by);
      look(m, by);
      look(m - 1, by);
    }
  };
  for (unsigned d : edges) divisor(d);
  for (unsigned d = 1; d < 20000; ++d) divisor(d);
  for (int i = 0; i < 20000; ++i) {
    const unsigned d = gen() >> (gen() % 32);
    divisor(d ? d : 1);
  }
  std::printf("%lld wrong of %lld\\n", wrong, looked);
  return wrong != 0;
}
"""


def test_fast_division(tmp_path):
    (tmp_path / "t.cu").write_text(PROGRAM)
    cmd = [build.nvcc_path(), "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{build.CSRC}", "-o", str(tmp_path / "t")]
    subprocess.run([*cmd, str(tmp_path / "t.cu")], check=True, capture_output=True)
    run = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout.startswith("0 wrong of 5"), run.stdout
