"""Kernels launched dependently through a wrapper or with attributes keep the rules of csrc/torch/pdl.cuh, too: whatever releases its
successor early waits for its predecessor itself, before it touches global memory."""
import re

import pytest

from tests.test_dependent_launch_source_cpu import KERNELS, SOURCES

RELEASING = sorted(n for n, (_, body) in KERNELS.items() if "pdlRelease" in body)


def _launched():
    """Kernels named in a call of launchPdl, launchPdlAttr or launchPdlCluster, or in the arguments of a wrapper that makes one."""
    names = set()
    for text in SOURCES.values():
        for call in re.findall(r"launchPdl(?:Attr|Cluster)?\(([^;]*);", text):
            names |= set(re.findall(r"\w*Kernel\b", call))
        for m in re.finditer(r"auto (\w+) = \[&\]\(auto kernel[^;]*?\{.*?launchPdl(?:Attr|Cluster)?\(kernel", text, re.S):
            for call in re.findall(r"\b%s\(([^;]*);" % m.group(1), text[m.end():]):
                names |= set(re.findall(r"\w*Kernel\b", call))
    return names


def test_kernels_behind_wrappers_and_attributes_are_seen():
    assert {"embFwdKernel", "embBwdKernel", "moeDispatchLocalKernel", "gemmFp8Kernel", "gemmFp8PairKernel", "adamwKernel"} <= _launched()


@pytest.mark.parametrize("name", sorted(_launched() & set(KERNELS)))
def test_launched_kernels_wait(name):
    assert "pdlWait()" in KERNELS[name][1]


@pytest.mark.parametrize("name", RELEASING)
def test_kernels_that_release_wait(name):
    assert "pdlWait()" in KERNELS[name][1]
