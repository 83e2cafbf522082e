"""The mixed-precision H-LU rounds to FP32 what its recompression cores work on,
and nothing before: the products W = B_ik' A_kj and A_ik W of the trailing
update are FP64 sums of the FP64 factors (what they are subtracted from cancels).
The loss shows only as a somewhat larger error of the same order as the core's,
so the types are checked in the source."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir, "hmatrix.jl_b200", "csrc", "hm_lu_pair.cuh")


def body(name):
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    m = re.search(r"__global__[^;{]*\b%s\s*\([^{;]*\)\s*\{" % name, text)
    depth, i = 1, m.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[m.end():i]


def test_products_of_the_update_are_fp64():
    # up to where the cores begin
    pair = body("lu_pair_kernel").split("const int ok =")[0]
    core = body("lu_tile_core_kernel").split("CoreJob J")[0]
    assert re.search(r"__shared__\s+double\s+sW\[", pair) and re.search(r"double\s*\*\s*sw\s*=", core)
    # factors and weights are not narrowed, the sums they enter are FP64
    assert not re.search(r"\(TS\)\s*-?(p\[|v\.|sW)", pair)
    assert not re.search(r"\(TS\)\s*-?(v\.Aik|v\.Bik|v\.Akj|sw\[)", core)
    assert not re.search(r"\bTS\s+(t|d|w|y)\b", pair)
    assert not re.search(r"\bTS\s+s\b", core) and not re.search(r"sw\[e\]\s*=\s*\(TS\)", core)
