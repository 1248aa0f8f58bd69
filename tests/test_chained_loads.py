"""The EDT's chained launches (csrc/edt_search.cu): a kernel of the chain may begin while the one before it still
writes, so what the chain itself writes is read by ordinary loads after the wait.  The read-only path (__ldg, or a
const __restrict__ parameter) is for data that nothing writes while the kernel lives.  Checked in the source: a kernel
that broke the rule could give the right bits on every run of a test."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-voxels_b200", "csrc", "edt_search.cu")
KERNELS = ("near_kernel", "search_y_kernel", "search_x_kernel", "near_batch_kernel", "search_y_batch_kernel",
           "search_x_batch_kernel")


def _code():
    with open(SRC) as f:
        return re.sub(r"/\*.*?\*/", "", re.sub(r"//[^\n]*", "", f.read()), flags=re.S)


def test_read_only_loads_never_take_what_the_chain_writes():
    taken = set(re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?\s*(\w+)", _code()))
    assert taken and taken <= {"xyz", "vox", "prefix"}  # clouds, the filled map and the batch's tables


def test_chained_kernels_have_no_read_only_parameters_but_tables():
    code = _code()
    assert set(re.findall(r"launch_next\((\w+)", code)) == {"void", "near", *KERNELS[1:]}  # near: near_kernel of some height
    for name in KERNELS:
        params = re.search(r"%s\(([^)]*)\)\s*\{(.*?)\n\}" % name, code, re.S)
        for p in params.group(1).split(","):
            assert "__restrict__" not in p or re.match(r"\s*const (BatchMap|long long)\* __restrict__ (maps|prefix)\s*$", p), (name, p)
        assert "*skip" not in params.group(2) and "*other_flag" not in params.group(2)
    for name in ("item_y", "item_x", "near_column"):
        assert "__restrict__" not in re.search(r"void %s\(([^)]*)\)" % name, code).group(1)
