"""The persistent solve's FP32 rows compile for every lane count that the colour
kernels' tuning defines accept, and their index words fit the words that a lane
reads (CPU; nvcc cross-compiles)."""
import os
import subprocess

import pytest

from cpfem_code_b200 import build

SRC = """
#include "fas_sor_flow.cuh"
using namespace fasdev;
template <typename T, int S> constexpr bool fits()
{
    using L = FlowRow<T, S>;
    // a row held in registers: a lane's columns, on one lane the header in the last one's place, in at most 8 words
    return L::SPL <= L::MW && (!L::AHEAD || L::MW <= 8) && L::LPR <= 32;
}
static_assert(fits<float, SLOTS>() && fits<float, SLOTS20>() && fits<double, SLOTS>() && fits<double, SLOTS20>(), "words");
"""


@pytest.mark.parametrize("defines", [{}, dict(FAS_TMA_LPR32=2, FAS_TMA_ROWS32=16), dict(FAS_TMA_LPR32=1, FAS_TMA_ROWS32=32),
                                     dict(FAS_TMA_LPR32=32), dict(FAS_TMA_LPR81_32=4), dict(FAS_TMA_LPR81_32=2),
                                     dict(FAS_TMA_LPR81_32=32, FAS_TMA_ROWS81_32=4)],
                         ids=lambda d: "-".join(f"{k[8:]}{v}" for k, v in d.items()) or "default")
def test_lane_counts(tmp_path, defines):
    src = tmp_path / "shape.cu"
    src.write_text(SRC)
    cmd = [build.nvcc(), *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", build.SRC, "-O0", "-Xptxas=-O0",
           *[f"-D{k}={v}" for k, v in defines.items()], "-c", "-o", os.devnull, str(src)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
