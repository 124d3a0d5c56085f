"""The dealing of a call's steps to persistent launches (``csrc/step_form.h``),
compiled for the host: each step is issued once and in order, and where the
runtime refuses a launch the rest is left to the launched step, on the history
side it belongs to."""

import shutil
import subprocess

import pytest

from sand_atlas_dem_gb300 import native

MAIN = r"""
#include <cstdio>
#include "step_form.h"
int main() {
    const uint32_t sizes[] = {0, 1, 63, 64, 65, 128, 200};
    for (uint32_t steps : sizes)
        for (int refuse = -1; refuse < 5; ++refuse) {
            uint32_t issued = 0, launches = 0;
            bool refused = false;
            uint32_t done = sdg::runSteps(steps, [&](uint32_t n) {
                if (n == 0 || n > sdg::RUN_STEPS || issued % 2 != 0) return std::puts("bad launch"), false;
                if (int(launches++) == refuse) { refused = true; return false; }
                issued += n;
                return true;
            });
            if (done != issued || done > steps || (!refused && done != steps) || (refused && done % 2 != 0))
                return std::printf("steps %u refuse %d done %u\n", steps, refuse, done), 1;
            if (refuse == 0 && steps && done != 0) return 1;
        }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host C++ compiler")
def test_steps_are_issued_once_and_a_refusal_leaves_the_rest(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    program = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", str(native.CSRC), str(tmp_path / "main.cpp"), "-o",
                    str(program)], check=True)
    result = subprocess.run([str(program)], capture_output=True, text=True)
    assert result.returncode == 0, result.stdout

