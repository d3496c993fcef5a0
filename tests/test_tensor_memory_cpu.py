"""Sources of the kernels of CTA pairs: tensor memory is released for both CTAs, so neither may still be reading it."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "create_llm_by_cupy_b200" / "ops" / "csrc"


def kernels():
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        for part in re.split(r"__global__", text)[1:]:
            body = part.split("\n}\n", 1)[0]
            if "tmem_dealloc_pair(" in body:
                yield pytest.param(body, id=f"{f.name}:{re.search(r'(\w+_kernel)', body).group(1)}")


def test_there_are_some():
    assert len(list(kernels())) >= 2


@pytest.mark.parametrize("body", list(kernels()))
def test_a_cluster_barrier_between_the_last_access_and_the_release(body):
    release = body.index("tmem_dealloc_pair(")
    assert body.count("tmem_dealloc_pair(") == 1
    last = max(m.start() for m in re.finditer(r"\b(tmem_ld|tmem_st|umma)_\w+\(", body))
    assert last < release, "tensor memory is read behind its release"
    between = body[last:release]
    # loads have arrived and are ordered before the barrier that both CTAs pass
    assert re.search(r"tmem_ld_wait\(\).*tc_fence_before\(\).*__syncthreads\(\).*cluster_sync_all\(\)",
                     body[body.rindex("tmem_ld_32x32b", 0, release):release], re.S)
    assert "cluster_sync_all()" in between
