"""CPU test of the FFT convolutions' cache keys (csrc/rgf_fft_cache.h): scratch
and cuFFT plans follow their own device, whichever form of the transforms ran
in between."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "rgf_fft_cache.h"
#include <cassert>
int main() {
  rgf::FftKeys k;
  const rgf::FftPlanKey on0{0, 2, 2, 16384, 7, 3}, on1{1, 2, 2, 16384, 7, 3};
  assert(!k.scratch_fits(0, 1) && !k.plans_fit(on0) && !k.plans_fit(rgf::FftPlanKey()));
  k.set_scratch(0, 100);      // plans and scratch on device 0
  k.set_plans(on0);
  assert(k.scratch_fits(0, 100) && !k.scratch_fits(0, 101) && !k.scratch_fits(1, 1));
  k.set_scratch(1, 200);      // the own transforms on device 1: scratch alone
  assert(k.scratch_fits(1, 200) && !k.scratch_fits(0, 100));
  assert(!k.plans_fit(on1));  // the plans are still device 0's
  assert(k.plans_fit(on0));
  k.set_plans(on1);
  assert(k.plans_fit(on1) && !k.plans_fit(on0));
  rgf::FftPlanKey other = on1;
  other.tail = 0;
  assert(!k.plans_fit(other));
  k.drop_plans();
  assert(!k.plans_fit(on1));
  return 0;
}
"""


def test_scratch_and_plans_have_their_own_device(tmp_path):
    src, exe = tmp_path / "keys.cpp", tmp_path / "keys"
    src.write_text(PROGRAM)
    inc = os.path.join(ROOT, "liteqt_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", inc, str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True)
