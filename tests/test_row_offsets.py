"""Grid rows hold 16 j, the byte offset of a partner's coordinates, in 32 bits.  As
signed numbers they would turn negative from 2^27 beads on, and gathers would
fault; unsigned they reach 2^28 beads, and a larger job without hydrodynamics is
refused.  Read from the sources on the CPU: such a job does not fit a test."""
import os
import re

import numpy as np
import pytest

from conftest import REPO

CSRC = os.path.join(REPO, "sop-gpu_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_offsets_are_unsigned():
    dev, grid, api = source("sopb_resident.cuh"), source("sopb_grid.cuh"), source("sopb_api.cu")
    assert re.search(r"bead_at\(const char\* xb, uint32_t off\)", dev)
    # no signed shift of a row's or near row's entry, no signed product 16 j
    assert not re.search(r"(?<!\(uint32_t\))\b(?:row|own)\[k\] >> 4", dev.split("J.gvr) {")[1].split("} else {")[0])
    assert "16 * q" not in grid and not re.search(r"\[e >> 3\]|\[w\[u \+ v\] >> 3\]", grid)
    assert re.search(r"kMaxPairBeads = 1 << 28", dev + grid)
    assert re.search(r"!p\.hi_on && n > kMaxPairBeads\) return SOPB_ERR_UNSUPPORTED", api)


@pytest.mark.parametrize("j", [2 ** 27 - 1, 2 ** 27, 2 ** 28 - 1])
def test_an_entry_holds_its_bead(j):
    e = np.uint32(16 * j)
    assert int(e) >> 4 == j and int(np.uint32(8 * j + 3)) >> 3 == j
    assert (int(e.astype(np.int32)) < 0) == (j >= 2 ** 27)      # what a signed entry would be
