"""Kernels that may be resident while the kernel before them still writes (launch_early): only kernels
that are launched so wait for the grids before them (grid_wait), and they treat no argument as constant:
no __restrict__ parameter and no read-only load (__ldg), whose data the compiler and the hardware may
take to be unchanged for the kernel's whole life."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ark-cpp-mpi_gb300", "csrc")


def sources():
    """(file, text without comments) of the kernels' sources."""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(CSRC, name)) as f:
                yield name, re.sub(r"//[^\n]*", "", f.read())


def functions_with_wait():
    """(file, name, parameter list, body) of each function whose body calls grid_wait()."""
    for name, text in sources():
        # a function ends with a brace in the first column (this code's layout) and starts after the last one
        for part in text.split("\n}"):
            if re.search(r"\bgrid_wait\(\);", part):
                m = re.search(r"\b(k_\w+|\w+_body)\s*\(([^{]*)\)\s*\{(?P<body>.*)", part, re.S)
                yield name, m.group(1), m.group(2), m.group("body")


FOUND = list(functions_with_wait())


def test_only_kernels_launched_early_wait():
    names = {n for _, n, _, _ in FOUND}
    assert names == {"k_mlp_grad", "k_mlp_update", "phase1_tma_body", "k_step_begin", "k_sweep_y_seams", "k_sweeps"}
    never = [f for f, text in sources() if re.search(r"\blaunch_early\(\s*false\b", text)]
    assert not never


@pytest.mark.parametrize("file,name,params,body", FOUND, ids=[f[1] for f in FOUND])
def test_no_argument_is_taken_to_be_constant(file, name, params, body):
    assert "__restrict__" not in params, (file, name)
    assert "__ldg" not in body, (file, name)
