"""The FP64 engine is a template over the number of species; the library
instantiates it for the shipped mechanism's nine.  A program that adds another
count needs every kernel of the step to compile for it."""
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.parametrize("cfg", ["2, 1, 10", "1, 0, 7"])
def test_the_engine_compiles_for_another_species_count(tmp_path, cfg):
    from openstc_b200.build import ARCH, _nvcc

    src = tmp_path / "engine.cu"
    src.write_text(f'#include "device/engine_impl.cuh"\nnamespace ostc {{\ntemplate class EngineT<Cfg<{cfg}>>;\n}}\n')
    res = subprocess.run([_nvcc(), *ARCH, "-std=c++20", "--expt-relaxed-constexpr", "-Xcicc", "-O0", "-Xptxas", "-O0", "-I",
                          str(ROOT / "include"), "-I", str(ROOT / "openstc_b200" / "csrc"), "-c", str(src), "-o",
                          str(tmp_path / "engine.o")], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
