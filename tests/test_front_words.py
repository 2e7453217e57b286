"""The words of the front-end launch (csrc/front_words.h) are zero behind every launch, in whatever order
its groups of blocks end: a block that waits for a row gives up after a while, so that a row may be announced
when the gate's blocks and the linears' are through.  Runs on the CPU."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "nemotron-inference_b200", "csrc")

DRIVER = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "front_words.h"
using namespace nmoe;

// argv: rows, linears.  Goes through the orders in which the groups end; each announces its row, if it has
// one, just before.
int main(int argc, char** argv) {
  (void)argc;
  const int rows = std::atoi(argv[1]), linears = std::atoi(argv[2]);
  std::vector<int> order(front_groups(rows, linears));
  for (size_t i = 0; i < order.size(); ++i) order[i] = static_cast<int>(i);
  FrontWords words{};
  long orders = 0;
  do {
    for (int group : order) {
      if (group < rows) words.row_known[group] = 1;
      else if (group < rows + linears) words.row_rounded[group - rows] = 1;
      front_group_through(&words, rows, linears, [](int32_t* word) { return (*word)++; });
    }
    const int32_t* all = reinterpret_cast<const int32_t*>(&words);
    for (size_t i = 0; i < sizeof(words) / sizeof(int32_t); ++i) {
      if (all[i] != 0) {
        std::printf("word %zu is %d behind the order", i, all[i]);
        for (int group : order) std::printf(" %d", group);
        return 1;
      }
    }
    ++orders;
  } while (std::next_permutation(order.begin(), order.end()));
  std::printf("%ld orders", orders);
  return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    folder = tmp_path_factory.mktemp("front_words")
    source, binary = folder / "driver.cpp", folder / "driver"
    source.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(source), "-o",
                    str(binary)], check=True)
    return str(binary)


@pytest.mark.parametrize("rows,linears", [(1, 0), (2, 0), (8, 0), (1, 1), (1, 2)])
def test_words_are_zero_behind_a_launch(driver, rows, linears):
    done = subprocess.run([driver, str(rows), str(linears)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
