"""The 32-bit slots in which the sampling loops put samples aside (compiled by g++ from the library's
header): each gives back its 64-bit sample index up to the last round of a loop that uses them, and one
more round is refused."""
import os
import subprocess

import pytest

from test_host_arith import ROOT, _cuda_include

SOURCE = """
#include <stdio.h>
#include "zg_internal.cuh"
int main() {
  const uint64_t strides[] = {256, 155648, 4194304};
  for (uint64_t stride : strides) {
    const uint64_t most = ZG_QUEUE_ROUNDS * stride, starts[] = {0, 96, most, most + 96};
    const uint64_t rounds[] = {0, 1, (1u << 26) + 5, ZG_QUEUE_ROUNDS - 2, ZG_QUEUE_ROUNDS - 1};
    printf("hold %d %d %d\\n", zg_slots_hold(stride + 1, stride), zg_slots_hold(most, stride), zg_slots_hold(most + 1, stride));
    for (uint64_t start : starts)
      for (uint64_t k : rounds)
        for (uint32_t lane = 0; lane < 32; lane += 31)
          printf("slot %llu %llu\\n", (unsigned long long)(start + k * stride + lane),
                 (unsigned long long)zg_slot_sample(start, stride, zg_slot((uint32_t)k, lane)));
  }
  return 0;
}
"""


def test_slots_give_back_their_samples(tmp_path):
    inc = _cuda_include()
    if not inc:
        pytest.skip("the CUDA headers are missing")
    src, exe = tmp_path / "slots.cpp", str(tmp_path / "slots")
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", inc, "-I", os.path.join(ROOT, "sampling-graph-mining_gb300", "csrc"),
                    str(src), "-o", exe], check=True)
    rows = [ln.split() for ln in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]
    hold, slots = [r[1:] for r in rows if r[0] == "hold"], [r[1:] for r in rows if r[0] == "slot"]
    assert hold == [["1", "1", "0"]] * 3
    assert len(slots) == 3 * 4 * 5 * 2 and all(want == got for want, got in slots)
