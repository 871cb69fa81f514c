"""GPU parity of the one-launch front end (up to 16 tokens), at the sizes where its dispatch
changes or its K split is uneven.  The oracle and its tolerances are those of
test_gpu_parity.py."""
import numpy as np
import pytest
import torch

import gpt_oss_amd_b200 as pkg
from gpt_oss_amd_b200 import capi, synth
from oracle import oracle
from parity_util import compare, oracle_case, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,I,E,K,T", [
    (64, 64, 4, 1, 1),       # one chunk of K: seven of the eight CTAs of the cluster have none
    (576, 64, 20, 4, 15),    # nine chunks: CTA 0 has two
    (128, 64, 33, 8, 16),    # the most tokens; E just above an expert tile
    (192, 64, 100, 2, 7),
    (1088, 64, 200, 4, 16),  # eight expert tiles
    (576, 64, 20, 4, 17),    # one token more: the separate kernels
])
@pytest.mark.parametrize("form", ["bf16", "f32", "norm"])
def test_front_end(H, I, E, K, T, form):
    shape = pkg.MoEShape(hidden=H, intermediate=I, n_experts=E, top_k=K)
    lw = synth.make_layer(shape, seed=H + E + T)
    if form != "norm":
        x_bits = synth.make_tokens(T, H, seed=T)
        ref = oracle_case(lw, x_bits)
        res = run_gpu(shape, lw, x_bits, capi.GEMM_TCGEN05, dtype=form)
    else:
        g = torch.Generator().manual_seed(T)
        x = (3.0 * torch.randn(T, H, generator=g)).float()
        w = (1.0 + 0.2 * torch.randn(H, generator=g)).float()
        x_bits = synth.bf16_bits(torch.from_numpy(oracle.rmsnorm(x.numpy(), w.numpy())))
        ref = oracle_case(lw, x_bits)
        with pkg.MoEEngine(shape, max_tokens=T) as eng:
            eng.load_layer(0, lw)
            out, sc, ti, tw = eng.forward_norm(0, x.cuda(), w.cuda(), side=True)
            h = eng.last_intermediate(T)
            torch.cuda.synchronize()
            assert eng.device_status() == 0
            res = {"out": out.cpu().numpy(), "score": sc.cpu().numpy(), "topk_i": ti.cpu().numpy(),
                   "topk_w": tw.cpu().numpy(), "h_bits": h.cpu().numpy().view(np.uint16),
                   "counts": eng.last_expert_counts()}
    compare(res, ref, K, f"{(H, I, E, K, T, form)}")
    assert np.abs(res["score"] - ref["router_score"]).max() < 1e-5
    assert list(np.bincount(ref["topk_i"].reshape(-1), minlength=E)) == res["counts"]
