"""The integer operations that stand for float64 ones in the cloud-in-cell
kernels (csrc/cic64.h), compiled as host code with g++: cells and offsets,
products rounded to counts, counts to float64, quotients by a rounded
reciprocal, order and finiteness, each bit for bit the plain expression's over
millions of drawn cases and the edges of their ranges."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not found")
    tmp = tmp_path_factory.mktemp("cic64host")
    (tmp / "cuda_runtime.h").write_text("")
    out = str(tmp / "libcic64host.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(tmp), "-I",
                    os.path.join(ROOT, "plasma-simulations-by-example_gb300", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "cic64_host.cpp")], check=True, capture_output=True)
    return C.CDLL(out)


def count(f, *args):
    f.restype = C.c_longlong
    return f(C.c_longlong(3_000_000), *args)


@pytest.mark.parametrize("n", [2, 3, 21, 1024, 1 << 20])
def test_cells_and_offsets(host, n):
    assert count(host.cic_cells, C.c_int(n)) == 0


@pytest.mark.parametrize("name", ["cic_products", "cic_counts", "cic_quotients", "cic_keys"])
def test_formulas(host, name):
    assert count(getattr(host, name)) == 0
