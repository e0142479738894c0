"""The stopping decision of a launch that carries the previous launch's check:
one CTA may set the flag while the others read it, so whether a tile runs must
not depend on which of the two values a warp sees (a CTA whose warps disagree
would reach its barriers with a part of them).  Host code of csrc/common.cuh."""
import os
import shutil
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ccpi-regularisation-toolkit_gb300",
                    "csrc")

PROGRAM = r"""
#include <cstdio>
#include "common.cuh"
int main() {
    int bad = 0;
    for (int riding = 0; riding <= 9; riding++)      // the check reduced in this launch; 0: none
        for (int fired = 0; fired < (riding ? riding : 9); fired++) {  // set by an earlier check; 0: not yet
            const bool before = cilreg::tile_runs(fired, riding);
            const bool after = cilreg::tile_runs(fired == 0 && riding ? riding : fired, riding);
            if (before != after || before != (fired == 0)) bad++;
        }
    printf("%d\n", bad);
    return bad != 0;
}
"""


def test_a_tile_runs_whichever_value_of_the_flag_it_sees(tmp_path):
    src, exe = tmp_path / "stop.cu", tmp_path / "stop"
    src.write_text(PROGRAM)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC, "-o", str(exe),
                    str(src)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.strip() == "0"
