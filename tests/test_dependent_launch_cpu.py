"""Sources of the kernels that start before their predecessor has finished: nothing in them can be read ahead of the wait."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "create_llm_by_cupy_b200" / "ops" / "csrc"


def kernels():
    """(file, text from the parameter list to the end) of every kernel that waits for its predecessor."""
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        parts = re.split(r"__global__", text)
        for part in parts[1:]:
            body = part.split("\n}\n", 1)[0]
            if "pdl_wait()" in body:
                yield pytest.param(body, id=f"{f.name}:{re.search(r'(\w+_kernel)', body).group(1)}")


@pytest.mark.parametrize("body", list(kernels()))
def test_no_load_can_pass_the_wait(body):
    params = body[:body.index("{\n")]
    assert not re.search(r"const\s+[\w:]+\s*\*\s*__restrict__", params)
    assert not re.search(r"__ld(g|cs|cg|ca|lu)\s*\(|ld\.global\.nc", body)
    # in front of the wait: parameters and shared memory; of global memory only prefetches (and the status of a failure)
    ahead = body[len(params):body.index("pdl_wait()")]
    assert not re.search(r"p\.(?!status)\w+\[|checked_index\(|ld\.global", ahead)


def test_shared_device_code_has_no_invariant_loads():
    for f in CSRC.glob("*.cuh"):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        assert not re.search(r"__ldg\s*\(|ld\.global\.nc|const\s+[\w:]+\s*\*\s*__restrict__", text), f.name


def test_launched_kernels_wait():
    """Whatever goes through launch_pdl is a kernel that waits (or a variable that holds one)."""
    for f in CSRC.glob("*.cu"):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        waiting = {re.search(r"(\w+_kernel)", k.split("\n}\n", 1)[0]).group(1)
                   for k in re.split(r"__global__", text)[1:] if "pdl_wait()" in k.split("\n}\n", 1)[0]}
        for name in re.findall(r"launch_pdl\(\(?[^;]*?(\w+_kernel)", text):
            assert name in waiting, (f.name, name)
