"""Instructions marked ``.aligned`` must be executed by a converged warp. Reads the helpers that every kernel issues them through:
each brings the warp together itself, whatever its callers did before (guarded stores of ragged rows, loops of unequal trip
counts)."""
import re

import pytest

from scirust_b200 import _build

HELPERS = re.findall(r"__device__ __forceinline__ \w+ (\w+)\([^)]*\) \{(.*?)\n?\}\n", (_build.CSRC / "sm100_ptx.cuh").read_text(),
                     re.S)
# a wait directly follows its load or store; the callers of a `_converged` form answer for their warp
ALIGNED = [(n, body) for n, body in HELPERS if re.search(r"\.aligned|_converged\(", body) and not n.endswith(("_wait", "_converged"))]


def test_the_helpers_are_found():
    assert {"cluster_sync_all", "tmem_alloc", "tmem_dealloc", "tmem_dealloc_pair", "tmem_ld_32x32", "tmem_st_32x32"} <= {
        n for n, _ in ALIGNED}


@pytest.mark.parametrize("name,body", ALIGNED, ids=[n for n, _ in ALIGNED])
def test_aligned_instructions_follow_a_warp_barrier(name, body):
    assert "__syncwarp();" in re.split(r"\.aligned|_converged\(", body)[0]


def test_kernels_issue_them_through_the_helpers():
    for src in sorted(_build.CSRC.glob("*.cu")):
        for line in src.read_text().splitlines():
            assert not re.search(r"(tcgen05|barrier\.cluster)[\w.:]*\.aligned", line), (src.name, line)
