"""Tensor memory of a CTA pair is allocated by both CTAs together, and nothing says that an allocation waits for a CTA that does not run
yet: in both kernels it stands behind a cluster barrier."""
import re
from pathlib import Path

import pytest

GEMM = Path(__file__).resolve().parent.parent / "csrc" / "gemm"


@pytest.mark.parametrize("name,kernel,alloc", [("gemm_pair.cu", "gemm_pair_kernel", "tmem_alloc_pair("),
                                               ("gemm_cluster.cu", "gemm_cluster_kernel", "tcgen05.alloc.cta_group::2")])
def test_a_pair_allocates_behind_a_cluster_barrier(name, kernel, alloc):
    text = (GEMM / name).read_text()
    body = re.search(r"__global__[^;{]*?\b" + kernel + r"\(", text)
    assert body is not None
    before = text[body.end():].split(alloc)
    assert len(before) == 2, "one allocation in the kernel"
    assert re.search(r"\bcluster_(wait|sync|sync_all)\(\)", before[0])
