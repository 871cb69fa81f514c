"""Calls queued back to back, each kernel a programmatic dependent of the one before, give the
bits of the same calls made one at a time."""
import pytest
import torch

import gpt_oss_amd_b200 as pkg
from gpt_oss_amd_b200 import synth

pytestmark = pytest.mark.gpu

SHAPE = pkg.MoEShape(hidden=576, intermediate=320, n_experts=20, top_k=4)
LAYERS = 3
# the front end's sizes, the separate kernels, both small-batch GEMM forms, the CTA-pair GEMM
SIZES = [1, 16, 17, 64, 400, 700]


@pytest.fixture(scope="module")
def engine():
    with pkg.MoEEngine(SHAPE, n_layers=LAYERS, max_tokens=max(SIZES)) as eng:
        for layer in range(LAYERS):
            eng.load_layer(layer, synth.make_layer(SHAPE, seed=40 + layer))
        yield eng


def queue(eng, jobs, wait):
    """jobs: (layer, x, out).  out = MoE(x) for bf16 rows, x += MoE(rmsnorm(x)) for fp32 ones."""
    w = torch.linspace(0.5, 1.5, SHAPE.hidden, device="cuda")
    for layer, x, out in jobs:
        if x.dtype == torch.float32:
            eng.forward_norm(layer, x, w, out=x, accumulate=True)
        else:
            eng.forward(layer, x, out=out)
        if wait:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    assert eng.device_status() == 0


@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("order", ["mixed", "one size"])
def test_queued_calls_equal_single_calls(engine, order, norm):
    g = torch.Generator().manual_seed(5)

    def make_jobs():
        g.manual_seed(5)
        jobs = []
        for T in SIZES:
            x = torch.randn(T, SHAPE.hidden, generator=g).cuda()
            for layer in range(LAYERS):  # norm: the layers of one size are a chain on one stream x
                rows = x if norm else (x * (layer + 1.0) + layer).to(torch.bfloat16)
                jobs.append((layer, rows, torch.empty(T, SHAPE.hidden, device="cuda")))
        if order == "mixed":  # successive calls differ in size, so their plans do too
            jobs = [jobs[i] for layer in range(LAYERS) for i in range(layer, len(jobs), LAYERS)]
        return jobs

    single = make_jobs()
    queue(engine, single, wait=True)
    for _ in range(20):
        queued = make_jobs()
        torch.cuda.synchronize()
        queue(engine, queued, wait=False)
        for (layer, x1, o1), (_, x2, o2) in zip(single, queued):
            assert torch.equal(x1, x2) if norm else torch.equal(o1, o2), (layer, x1.shape)
