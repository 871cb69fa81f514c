"""mxfp4_unpack at block counts where its last thread block is cut."""
import numpy as np
import pytest
import torch

import gpt_oss_amd_b200 as pkg
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,G", [(1, 1), (3, 7), (255, 1), (257, 4), (1025, 3)])
def test_unpack_ragged(rows, G):
    """Block counts around the kernel's 1024 words per thread block, every scale byte."""
    g = torch.Generator().manual_seed(rows)
    blocks = torch.randint(0, 256, (rows, G, 16), generator=g, dtype=torch.uint8)
    scales = torch.randint(0, 256, (rows, G), generator=g, dtype=torch.uint8)
    out = pkg.mxfp4_unpack(blocks.cuda(), scales.cuda()).cpu().numpy().view(np.uint16)
    assert np.array_equal(out, oracle.mxfp4_dequant_bf16(blocks.numpy(), scales.numpy()))
