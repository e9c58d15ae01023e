"""Kernels that may be resident while their producer still writes (programmatic
dependent launches) read what the chain writes by plain loads: read-only loads
(__restrict__ parameters that the compiler turns into them, __ldg,
ld.global.nc) promise data that nobody writes while the kernel runs."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pyfstat_gb300",
                    "csrc")
# what the chain's kernels leave for each other
CHAIN = {"T", "atoms8", "P", "G", "parts", "results", "maps", "rowsum", "colsum"}


def read(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def kernels(src):
    """(name, parameters, body) of every __global__ function."""
    for m in re.finditer(r"__global__.*?\s(\w+)\s*\(([^()]*)\)\s*\{", src, re.S):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[i], 0)
            i += 1
        yield m.group(1), m.group(2), src[m.end():i]


def test_dependent_kernels_take_the_chains_data_by_plain_loads():
    found = set()
    for name, params, body in kernels(read("tcw_kernels.cu")):
        if "pdl_begin()" not in body:
            continue
        found.add(name)
        for p in params.split(","):
            if p.split()[-1].lstrip("*") in CHAIN and p.split()[0] == "const":
                assert "__restrict__" not in p, (name, p)
        for line in body.splitlines():
            args = re.findall(r"__ldg\((.*)", line)
            if args and "kChained ?" not in line:
                assert not CHAIN & set(re.findall(r"\w+", args[0])), (name, line)
    assert found >= {"exp_seg_kernel", "map_kernel", "finalize_kernel", "finalize_block_kernel",
                     "post_sums_kernel", "post_argmax_kernel"}


def test_single_maps_take_rows_by_plain_loads():
    """Read-only row loads stand behind a template argument that only the plans'
    warp-scheduled tiles and listed segments set."""
    src = read("tcw_kernels.cu")
    assert "ld.global.nc" not in src
    one = next(b for n, _, b in kernels(src) if n == "map_kernel")
    one = one[one.index("pdl_begin()"):]
    assert "rect_tile<kWrite, kPrec, false>" in one
    assert "exp_tile<kWrite, kPrec, kChunks, false>" in one
    assert "exp_column2<kPrec == kPrecFF_F64Det, kWarp>" in src
    assert "ExpColumn<kPrec == kPrecFF_F64Det, true, false, kWarp>" in src
    seg = next(b for n, _, b in kernels(src) if n == "exp_seg_kernel")
    assert "ExpColumn<false, true, false, kList>" in seg
    for name in ("tcw_kernels.cu", "tcw_cell.h", "tcw_exp_walk.cuh"):
        for line in read(name).splitlines():
            if re.search(r"__ldg\((a8|atoms8|P_all|seg|nz)", line):
                assert "kReadOnly ?" in line, (name, line)
