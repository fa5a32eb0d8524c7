"""Host rules of the SCC-resident solver (`csrc/scc_plan.h`), compiled here without CUDA."""
import ctypes as C
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "scc_plan.h"
using namespace esl;
extern "C" {
uint32_t own_rows(int j, uint32_t even, uint32_t odd) { return scc_own_rows(j, even, odd); }
int own_a() { return kOwnA; }
int own_w() { return kOwnW; }
int own_iq() { return kOwnIQ; }
int own_count() { return kOwnCount; }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("scc_plan")
    src, lib = d / "plan.cpp", d / "plan.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(REPO, "paraexastolog_b200", "csrc"),
                    str(src), "-o", str(lib)], check=True)
    return C.CDLL(str(lib))


@pytest.mark.parametrize("even,odd", [(158272, 158269), (24577, 24576), (3, 10), (1, 0), (0, 1)])
def test_vectors_hold_every_row_that_indexes_them(plan, even, odd):
    # the operator's input is indexed by odd rows and, in the setup, by even rows
    for j in range(plan.own_count()):
        rows = plan.own_rows(j, even, odd)
        need = even if j in (plan.own_w(), plan.own_iq()) else max(even, odd) if j == plan.own_a() else odd
        assert rows >= max(need, 1), j
