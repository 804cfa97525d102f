"""Kernels of a chain (chain_wait, csrc/hd_common.cuh) begin while the kernels before
them still write, so they read nothing but the caller's sets through the read-only
path: no __ldg and no const __restrict__ parameter for anything else."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "hausdorffdistance_gb300", "csrc")
# The caller's sets by the names that kernels give them.
INPUT_PARAMS = {"A", "B"}
INPUT_LOADS = {"a4", "b4"}


def source(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


def chained_kernels(text):
    """(name, parameters, body) of every kernel that calls chain_wait."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, start = text[m.end():i - 1], text.index("{", i)
        depth, j = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        if "chain_wait()" in text[start:j]:
            yield m.group(1), params, text[start:j]


def ldg_pointers(body):
    return set(re.findall(r"__ldg\(\s*&?(\w+)", body)) | (
        {"?"} if re.search(r"__ldg\(\s*[^\w&\s]", body) else set())


FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")))


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_chained_kernels_read_the_inputs_alone_as_constant(path):
    for name, params, body in chained_kernels(source(path)):
        constant = set(re.findall(r"const[^,]*?__restrict__\s+(\w+)", params))
        assert constant <= INPUT_PARAMS, (name, constant)
        assert ldg_pointers(body) <= INPUT_LOADS, (name, ldg_pointers(body))


def test_helpers_of_the_cell_filter():
    """Its device functions are inlined into chained kernels.  (The collection is
    not chained: the marks it looks up are constant by then.)"""
    text = source(os.path.join(CSRC, "hd_cells.cu"))
    assert ldg_pointers(text) <= {"any", "dq", "dt"}
    assert ldg_pointers(text[:text.index("k_cell_collect(")]) == set()
    assert re.search(r"launch_next\(c\.stream, false, k_cell_collect<", text)
    assert set(re.findall(r"__restrict__\s+(\w+)", text)) <= INPUT_PARAMS


def test_the_kernels_are_found():
    found = {n for p in FILES for n, _, _ in chained_kernels(source(p))}
    assert {"k_cell_occ", "k_cell_near", "k_cell_mark", "k_eb_pack", "k_eb_main", "k_eb_heavy",
            "k_argmin", "k_finalize"} <= found
