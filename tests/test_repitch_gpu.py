"""Copies between pitches: every alignment of source and destination, remainders of a 16-byte block, padding, segments."""
import pytest
import torch

from create_llm_by_cupy_b200.ops.gemm import repitch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 5, 300])
@pytest.mark.parametrize("cols,pad", [(1, 7), (2, 0), (7, 1), (8, 0), (9, 7), (15, 8), (33, 7), (257, 7), (2730, 6), (2730, 0)])
def test_repitch(rows, cols, pad):
    g = torch.Generator().manual_seed(rows + cols)
    width = cols + pad
    for s0 in range(8):
        for d0 in range(8):
            nseg, extra = 1 + (s0 + d0) % 2, (3 * s0 + d0) % 5
            src = torch.randint(-2 ** 15, 2 ** 15, (rows, nseg * cols + s0 + extra), generator=g, dtype=torch.int16).cuda()
            dst = torch.full((rows, nseg * width + d0 + extra), 77, dtype=torch.int16, device="cuda")
            want = dst.clone()
            for k in range(nseg):
                want[:, d0 + k * width:d0 + k * width + cols] = src[:, s0 + k * cols:s0 + (k + 1) * cols]
                want[:, d0 + k * width + cols:d0 + (k + 1) * width] = 0
            repitch(src[:, s0:].view(torch.bfloat16), dst[:, d0:].view(torch.bfloat16), cols, width, nseg, cols, width)
            assert torch.equal(dst, want)
