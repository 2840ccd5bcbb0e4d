"""The host units build and link without OpenMP: every use of its runtime is guarded."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "fierro_gb300", "csrc")


@pytest.mark.parametrize("unit", ["sgh_host.cpp", "sgh_capi.cpp", "sgh_batch.cpp", "sgh_adjoint.cpp", "sgh_output.cpp",
                                  "sgh_rz.cpp"])
def test_no_openmp_symbols(tmp_path, unit):
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    obj = str(tmp_path / "unit.o")
    subprocess.run(["g++", "-O0", "-std=c++17", "-Wno-unknown-pragmas", "-I", cuda, "-I", os.path.join(ROOT, "include"),
                    "-I", CSRC, "-c", os.path.join(CSRC, unit), "-o", obj], check=True)
    undefined = subprocess.run(["nm", "-u", obj], check=True, capture_output=True, text=True).stdout
    assert "omp_" not in undefined and "GOMP" not in undefined, undefined
