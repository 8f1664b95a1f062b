"""Shared-memory layouts of the column march for every allowed ring depth (the
build setting MHD3D_NRAW): the mbarriers of all slots lie in front of the
reduction area.  Static assertions in a translation unit that includes the
kernels; a last assertion that always fails ends the compilation before code
is generated."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SOURCE = """
#include "%s"
using namespace mhd3d::fast;
#define FITS(MAG, S) static_assert(Lay<MAG, S>::BAR_OFF + Lay<MAG, S>::NR + NZS <= Lay<MAG, S>::RED_OFF, "stage " #S);
FITS(true, 0) FITS(true, 1) FITS(true, 2) FITS(true, 3)
FITS(false, 0) FITS(false, 1) FITS(false, 2) FITS(false, 3)
static_assert(NRAW < 0, "end of the checks");
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
@pytest.mark.parametrize("nraw", [3, 4, 5, 6])
def test_barriers_fit(tmp_path, nraw):
    src = tmp_path / "layout.cu"
    src.write_text(SOURCE % os.path.join(PKG, "csrc", "stage_fast.cu"))
    r = subprocess.run([NVCC, "-arch=compute_100a", "-std=c++17", f"-DMHD3D_NRAW={nraw}", "-I", os.path.join(ROOT, "include"),
                        "-fatbin", str(src), "-o", str(tmp_path / "layout.fatbin")], capture_output=True, text=True)
    out = r.stdout + r.stderr
    errors = [line for line in out.splitlines() if "error:" in line]
    assert len(errors) == 1 and "end of the checks" in errors[0], out
