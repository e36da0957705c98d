"""The timing of the forms of the plain iterations (plain_form_tuner) on the CPU, against events that
are counted: every event that a solve takes is destroyed with its tuner, also where the form is decided,
or the solve ends, while a timed cycle is open."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include "plain_form.hpp"
#include <cstdio>
#include <cstring>
static int live = 0;
extern "C" cudaError_t cudaEventCreate(cudaEvent_t* e) { ++live; *e = (cudaEvent_t)new int; return cudaSuccess; }
extern "C" cudaError_t cudaEventDestroy(cudaEvent_t e) { --live; delete (int*)e; return cudaSuccess; }
extern "C" cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
extern "C" cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
extern "C" cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return ""; }
int main(int, char** argv)
{
  using cuopt_b200::plain_form_tuner;
  const bool avail[3] = {true, true, false};
  int chosen = -1;
  {
    plain_form_tuner t;
    for (int solve = 0; solve < 3; ++solve) {
      t.reset(-1, -1, avail);
      // The samples of a cycle are collected while the next one is open, as where checks are read after
      // the iterations that follow them have been launched.
      for (int c = 0; c < 2 * plain_form_tuner::kSamples + 1 && !t.decided(); ++c) {
        const int form = t.next();
        t.begin(nullptr);
        t.collect();
        if (!std::strcmp(argv[1], "unfinished") && c == 3) break;  // the solve ends here
        t.end(nullptr, form, 10, false);
      }
      chosen = t.chosen();
    }
  }
  std::printf("%d %d", live, chosen);
}
"""


@pytest.mark.parametrize("case,chosen", [("decided", 0), ("unfinished", -1)])
def test_events_of_open_cycles_are_released(tmp_path, case, chosen):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT / 'cuopt_b200' / 'csrc'}",
                    "-I/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), case], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", str(chosen)]
