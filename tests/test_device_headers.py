"""The arithmetic headers compile for the device without a diagnostic (a value
read before it is set, an order of evaluation that C++ does not fix)."""
import subprocess
import sys
from pathlib import Path

import pytest

PKG = Path(__file__).resolve().parent.parent / "cahn-hilliard_gb300"
SOURCE = r"""
#include "common.cuh"
#include "bfp.cuh"
#include "fxsum.cuh"
__global__ void k(chgb::ModelDev m, chgb::MobilityDev md, const double *x, double *y) {
    const chgb::SwCell c = chgb::sw_cell(m, x[0]);
    y[0] = c.der + c.rhoXv + chgb::saleh_log_X(m.dAA, m.sv0, x[0], m.half, x[1], m.logtab) + chgb::gel_exp(md, x[2]);
}
"""


def test_no_diagnostics(tmp_path):
    sys.path.insert(0, str(PKG))
    try:
        import build
        nvcc = build.nvcc()
    except FileNotFoundError:
        pytest.skip("no nvcc")
    finally:
        sys.path.remove(str(PKG))
    src = tmp_path / "headers.cu"
    src.write_text(SOURCE)
    r = subprocess.run([nvcc, *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-fmad=false", "-Werror", "all-warnings", f"-I{PKG / 'csrc'}",
                        "-c", str(src), "-o", str(tmp_path / "headers.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
