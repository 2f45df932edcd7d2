"""Rules of dependent launch (csrc/torch/pdl.cuh) that the compiler does not check, read from the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "csrc"


def _kernels(text):
    """(name, template and parameter list, body) of every __global__ function; bodies end at the first brace in column 0."""
    for m in re.finditer(r"__global__", text):
        head_end = text.index(") {", m.start())
        head = text[m.start():head_end]
        yield re.findall(r"(\w+)\(", head)[-1], head, text[head_end:text.index("\n}\n", head_end)]


SOURCES = {p.name: p.read_text() for p in sorted(CSRC.rglob("*.cu"))}
KERNELS = {name: (head, body) for text in SOURCES.values() for name, head, body in _kernels(text)}
LAUNCHED = {n for text in SOURCES.values() for n in re.findall(r"launchPdl\((\w+)", text)}


def test_the_sources_were_understood():
    assert {"lnBwdFusedKernel", "colSumFoldKernel", "quantActKernel", "fcxGemmPairKernel", "moeGroupKernel"} <= set(KERNELS)
    assert {"lnParamFoldKernel", "adamwKernel", "gemmFp8PairKernel"} <= LAUNCHED


@pytest.mark.parametrize("name", sorted(n for n, (_, body) in KERNELS.items() if "pdlWait" in body))
def test_no_load_of_a_predecessors_memory_may_take_the_read_only_path(name):
    head, body = KERNELS[name]
    assert "__restrict__" not in head and "__ldg" not in body and "ld.global.nc" not in body


@pytest.mark.parametrize("name", sorted(n for n, (_, body) in KERNELS.items() if "tcgen05.alloc" in body and "pdlRelease" in body))
def test_successors_come_up_only_after_the_tmem_allocation(name):
    body = KERNELS[name][1]
    assert body.index("pdlRelease") > body.index("tcgen05.alloc")


@pytest.mark.parametrize("name", sorted(LAUNCHED & set(KERNELS)))
def test_every_kernel_launched_that_way_waits_for_its_predecessor(name):
    assert "pdlWait()" in KERNELS[name][1]
