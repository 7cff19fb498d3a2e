"""Barriers and tensor-memory allocations written as inline PTX are the aligned forms: every lane of a
warp has to execute them together.  A warp whose lanes left a branch or a loop at different trips is not
converged by itself, so each of them directly follows a __syncwarp()."""
import glob
import os
import re

import pytest

from tests.conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "jaxns_gb300", "csrc", "*.cu*")))
ALIGNED = r'asm volatile\(\s*"(?:bar\.sync|barrier\.cluster\.arrive|tcgen05\.alloc)'
CONVERGED = r'__syncwarp\(\);(?:\s|//[^\n]*\n)*(?:if \(warp == 0\) \{\s*)?' + ALIGNED


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_aligned_barriers_follow_a_warp_barrier(path):
    src = open(path).read()
    assert len(re.findall(ALIGNED, src)) == len(re.findall(CONVERGED, src))


def test_the_barriers_are_found():
    assert sum(len(re.findall(ALIGNED, open(p).read())) for p in SOURCES) >= 8
