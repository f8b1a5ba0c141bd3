"""Bounded waits of whole warps: whether one ran out is found by each lane for itself, so lanes may disagree, and what stands behind it (shuffles,
warp barriers, tcgen05.ld) has to be reached by all of them or by none. The kernels vote. Shown on the source: a wait that runs out needs
a copy or a product that never comes, which no test brings about."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "src")


def _code(*parts):
    with open(os.path.join(SRC, *parts)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_rows_of_the_norm():
    code = _code("contrib", "devapi_samples.cu")
    kernel = code[code.index("rmsNormRowsKernel(const"):code.index("struct RowPlan")]
    waits = re.findall(r"[^\n]*\bwait\(&fullBar[^\n]*", kernel)
    assert len(waits) == 1 and re.search(r"const bool ok = __all_sync\(0xffffffffu, wait\(&fullBar\[s\], phase\)\);", waits[0])


@pytest.mark.parametrize("name", ["gemm_fp8_sm100.cu", "gemm_split_sm100.cu", "gemm_sm100.cu", "gemm_pair_sm100.cu"])
def test_accumulators(name):
    code = _code("tp", name)
    waits = re.findall(r"[^\n]*\bmbarWait\(smemAddr\(&accFull[^\n]*", code)
    assert waits and all(re.search(r"__all_sync\((0xffffffffu|~0u), mbarWait\(smemAddr\(&accFull", w) for w in waits)
    # the word that ends a kernel early, where whole warps go from tile to tile: the loops behind those of the single threads that load and multiply
    loops = re.findall(r"for \(int t = [^\n]*", code)
    assert len(loops) == (0 if "split" in name else 3)
    for loop in loops[2:]:
        body = code[code.rindex(loop):]
        assert body[:body.index("accFull")].count("*abortFlag") == body[:body.index("accFull")].count("__any_sync(0xffffffffu, *abortFlag)") == 1
