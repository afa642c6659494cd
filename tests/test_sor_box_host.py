"""The linear box solver's enumeration of a colour (csrc/sor_box.h), compiled
as host code with nvcc: on every grid it takes the 32-bit route or the 64-bit
one and finds the nodes that plain division finds.  Thin boxes with millions
of short rows, where the float-estimated division of the 32-bit route would
miss, the last box of that route, and one of more than 2^31 nodes."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    out = str(tmp_path_factory.mktemp("sorhost") / "libsorhost.so")
    csrc = os.path.join(ROOT, "plasma-simulations-by-example_gb300", "csrc")
    subprocess.run([nvcc, "-shared", "-Xcompiler", "-fPIC", "-Xcompiler", "-ffp-contract=off", "-O2", "-std=c++17",
                    "-I", csrc, "-gencode", "arch=compute_103a,code=sm_103a", "-o", out,
                    os.path.join(ROOT, "tests", "sor_box_host.cu")], check=True, capture_output=True)
    lib = C.CDLL(out)
    lib.sor_host_misplaced.restype = C.c_int64
    lib.sor_host_misplaced.argtypes = 3 * [C.c_int] + 2 * [C.c_int64]
    return lib


@pytest.mark.parametrize("nodes,brief", [
    ((3, 3, 3), 1), ((21, 21, 21), 1), ((26, 25, 23), 1), ((256, 256, 512), 1), ((5, 2050, 2049), 1),
    ((5, 2898, 2898), 1), ((5, 2899, 2899), 0), ((21, 2050, 2049), 1), ((21, 2100, 2100), 0), ((7, 3402, 3402), 0),
    ((3, 5800, 5800), 0), ((13, 3500, 3500), 0)])
def test_every_entry_finds_its_node(host, nodes, brief):
    assert host.sor_host_short(*nodes) == brief
    assert host.sor_host_misplaced(*nodes, 0, 1) == 0


@pytest.mark.parametrize("nodes", [(1290, 1290, 1290), (1291, 1291, 1291), (1025, 1024, 2048), (3, 46400, 23200)])
def test_grids_of_two_to_the_31_nodes(host, nodes):
    assert host.sor_host_misplaced(*nodes, 7, 1009) == 0
    count = (nodes[0] - 1) // 2 * (nodes[1] - 2) * (nodes[2] - 2)
    assert host.sor_host_misplaced(*nodes, count - 100_000, 1) == 0
