"""Rules that the CUDA sources keep and no run on a GPU shows to be broken.

A kernel that is launched with programmatic serialization is resident while the
launch before it still writes.  The read-only load path (`__ldg`) is allowed only
for memory that nothing writes while the kernel lives, and a load through a
`__restrict__` argument may be moved above the wait: so an earlier launch's data
is read with plain loads through pointers that went through `pdl_fresh`."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "kapsel_old_b200", "csrc")


def _sources():
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        yield os.path.basename(f), re.sub(r"//[^\n]*", "", open(f).read())


def _block(src, at):
    """The text between the brace at or after `at` and its partner."""
    b = src.index("{", at)
    depth = 0
    for i in range(b, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[b:i + 1]
    raise AssertionError("unbalanced braces")


def kernels():
    """(file, name, parameter list, body) of every __global__ definition."""
    for f, src in _sources():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", src):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(src[i], 0)
                i += 1
            if src[i:].lstrip().startswith("{"):
                yield f, m.group(1), src[m.end():i - 1], _block(src, i)


CHAINED = [k for k in kernels() if "pdl_begin()" in k[3]]


def test_the_chained_kernels_are_found():
    names = {k[1] for k in CHAINED}
    assert {"k_particles_hydro_velocity", "k_particles_scatter", "k_zw_c2r", "k_yzw_c2r", "k_xw_advect", "k_zw_flux",
            "k_obl_to_cart", "k_cell_scan", "k_y_pass", "k_z_c2r"} <= names
    assert len(names) > 40


def test_read_only_loads_are_of_the_constant_offset_table():
    for f, src in _sources():
        for m in re.finditer(r"__ldg\s*\(|ld\.global\.nc", src):
            fn = src.rfind("Cell load_cell(const", 0, m.start())
            assert fn >= 0 and m.start() < fn + len(_block(src, fn)) + src[fn:].index("{"), \
                f"{f}: {src[m.start():m.start() + 40]}"


@pytest.mark.parametrize("k", CHAINED, ids=lambda k: k[1])
def test_earlier_launches_data_is_read_through_fresh_pointers(k):
    _, name, params, body = k
    assert re.match(r"\s*(?:(?:using|constexpr|extern|__shared__|typename)\b[^;]*;\s*|\w+ \w+\[[^;]*;\s*)*pdl_begin\(\);",
                    body[1:]), f"{name}: pdl_begin is not the first statement"
    for p in params.split(","):
        m = re.search(r"\*\s*(?:__restrict__\s*)?(\w+)\s*(?:=.*)?$", p.strip())
        if not m or m.group(1) == "cells" or not ("const" in p or "DPart" in p):
            continue
        assert re.search(rf"pdl_fresh\({m.group(1)}\)", body), f"{name}: {m.group(1)}"


def test_kernels_of_planned_block_sizes_stride_by_the_block_they_run_in():
    """zplan launches fewer warps than the template's NW where shared memory does
    not hold them: a kernel that strode by NW would then leave rows out."""
    src = dict(_sources())["kapsel_gpu.cu"]
    planned = set(re.findall(r"zplan\((k_\w+)<", src))
    assert {"k_zw_products", "k_zw_c2r", "k_zw_cross", "k_zw_flux"} <= planned
    for _, name, _, body in kernels():
        if name in planned:
            assert "blockDim.x >> 5" in body and not re.search(r"\bNW\b", body), name
