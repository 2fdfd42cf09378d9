"""Host-side rules of the pulsed update and arithmetic that its kernels share with the host, compiled and run on the
CPU: the longest train of an update, the count of an implicit pair of lines, places in the pool of Gaussians."""

import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SOURCE = r"""
#include "pulse_common.cuh"
#include <cstdio>
#include <cstdlib>
using namespace ab200;
int main(int argc, char **argv) {
  if (argv[1][0] == 'l') { // desired_bl fixed_bl update_bl_management lr dw_min
    UpEff up{};
    up.desired_bl = atoi(argv[2]);
    up.fixed_bl = atoi(argv[3]);
    up.update_bl_management = atoi(argv[4]);
    printf("%d\n", longestTrain(up, strtof(argv[5], nullptr), strtof(argv[6], nullptr)));
  } else if (argv[1][0] == 'c') { // short_train values...
    for (int i = 3; i < argc; i++) {
      printf("%d\n", implicitPulses(strtof(argv[i], nullptr), argv[2][0] == '1'));
    }
  } else { // the largest place that any lane looks at in a pool's row, and the length of the row
    int largest = 0;
    uint32_t takers = 1u;
    for (int turn = 0; turn < 2000; turn++) {
      takers = turn == 0 ? 0u : (turn == 1 ? 0xffffffffu : takers * 1664525u + 1013904223u);
      const int n = __builtin_popcount(takers);
      for (int pos = 0; pos + n <= kNoisePool; pos++) {
        for (int lane = 0; lane < 32; lane++) {
          largest = std::max(largest, noisePoolSlot(pos, takers, lane));
        }
      }
    }
    printf("%d %d\n", largest, kNoisePoolRow);
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("needs nvcc")
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cu").write_text(SOURCE)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-I" + os.path.join(ROOT, "aihwkit_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                    str(d / "rules.cu"), "-o", str(d / "rules")], check=True)

    def run(*args):
        out = subprocess.run([str(d / "rules"), *map(str, args)], check=True, capture_output=True, text=True).stdout
        return [int(v) for v in out.split()]

    return run


@pytest.mark.parametrize("desired,fixed,managed,lr,dw_min,want", [
    (31, 1, 0, 1.0, 1e-3, 31),             # the length is fixed
    (31, 0, 1, 1.0, 1e-3, 31),             # or the most that update management takes
    (31, 0, 0, 0.02, 1e-3, 31),            # one train of the wanted length reaches lr
    (31, 0, 0, 0.5, 1e-3, 500),            # it does not: as many slots as lr takes
    (8, 0, 0, 1.0, 2.0 ** -22, 1 << 22),
    (8, 0, 0, 1.0, 2.0 ** -25, 1 << 25),
    (8, 0, 0, 1.0, 1e-30, 2 ** 31 - 1),
    (8, 0, 0, 1.0, 0.0, 2 ** 31 - 1),
])
def test_longest_train(rules, desired, fixed, managed, lr, dw_min, want):
    assert rules("l", desired, fixed, managed, repr(lr), repr(dw_min)) == [want]


def test_counts_of_implicit_pulses(rules):
    rng = np.random.default_rng(0)
    small = np.concatenate([[0.0, 0.49999997, 0.5, 0.50000006, 1.5, 2.5, 1048575.5, 1048576.0],
                            rng.uniform(0, 40, 200), rng.uniform(0, 2 ** 20, 200)]).astype(np.float32)
    large = np.concatenate([small, [2.0 ** 22 + 0.5, 2.0 ** 23 - 0.5, 2.0 ** 24 + 2, 2.0 ** 30]]).astype(np.float32)
    for short, values in (("1", small), ("0", large)):
        for sign in (1, -1):
            got = rules("c", short, *(repr(float(sign * v)) for v in values))
            assert got == [int(v) for v in np.rint(values)]
        assert rules("c", short, "nan") == [0]
    assert rules("c", "0", "1e12", "-inf") == [2 ** 31 - 1] * 2


def test_no_lane_looks_past_its_pool(rules):
    largest, row = rules("p")
    assert largest < row
