"""The float-float forms of the re-evaluation and the Fisher pass
(``csrc/pes_ff.cuh``), compiled for the host and checked against long double: the
unrenormalised multiply-add and dot product, the tabulated sine and cosine up to the
argument that the general function's wrap is good for, and a chain of multiply-adds.

Bounds: an operation's, the sine's and cosine's and the wrap's as for the
renormalised forms; a chain's tails grow with its cancellations, and its users
narrow the result to 24 bits (6e-8): a thousandth of 2^-30."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
BOUNDS = {"mad": 3e-14, "dot2": 3e-14, "chain": 1e-12, "tab_1e3": 3e-14, "tab_1e4": 3e-14, "tab_2e18": 1e-12}


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("ff") / "ff_forms_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-w", "-o", exe,
                    os.path.join(HERE, "native", "ff_forms_check.cu")], check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {k: float(v) for k, v in (line.split() for line in out.strip().splitlines())}


@pytest.mark.parametrize("name", sorted(BOUNDS))
def test_form_error_bound(errors, name):
    assert errors[name] <= BOUNDS[name], (name, errors[name])
